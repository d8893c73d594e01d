"""Host paths that a GPU shows only when a device call fails or threads meet: the built library on a CUDA runtime of host
memory (fake_cudart.cpp), where any call can be made to fail and every launch and its arguments can be looked at. A
scenario runs in a process of its own, whose loader finds that runtime instead of the real one."""
import ctypes as C
import os
import subprocess
import sys
from contextlib import closing

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SCENARIOS = {}


def scenario(f):
    SCENARIOS[f.__name__] = f
    return f


@pytest.fixture(scope="session")
def fake_runtime(tmp_path_factory, pkg):
    if not os.path.exists(pkg.LIB_PATH):
        import mynah_asr_b200.build as b
        b.build()
    out = tmp_path_factory.mktemp("fake_cudart")
    (out / "versions").write_text("libcudart.so.12 { global: *; };\n")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", os.path.join(cuda, "include"), os.path.join(HERE, "fake_cudart.cpp"),
                    "-o", str(out / "libcudart.so.12"), "-Wl,-soname,libcudart.so.12", "-Wl,--version-script," + str(out / "versions")], check=True)
    return str(out)


@pytest.mark.parametrize("name", [
    "vad_allocation_fails", "vad_gives_back", "error_is_reported_once", "failed_call_waits", "launches_of_other_threads", "qmat_workspace_is_shared",
    "foreign_capture_survives", "chain_table_copy_fails", "chain_graph_reads_its_own_table",
    "copies_by_pieces", "copies_on_few_cores", "copies_of_other_classes", "copies_under_a_quota", "waits_of_copies_end_in_sleep", "copies_leave_others_alone", "small_copies_go_the_drivers_way", "ragged_audio_arrives_whole",
])
def test_host_path(fake_runtime, name):
    env = dict(os.environ, LD_LIBRARY_PATH=fake_runtime + ":" + os.environ.get("LD_LIBRARY_PATH", ""), OMP_NUM_THREADS="1")
    if name == "copies_under_a_quota":
        env["LD_PRELOAD"] = _quota_shim(fake_runtime)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), name], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def _quota_shim(folder):
    """A control group of this process's own: its cpu.max is the file beside the shim."""
    src, lib = os.path.join(folder, "quota.c"), os.path.join(folder, "quota.so")
    with open(src, "w") as f:
        f.write("""#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <string.h>
FILE *fopen(const char *path, const char *mode) {
    FILE *(*real)(const char *, const char *) = dlsym(RTLD_NEXT, "fopen");
    return real(strcmp(path, "/sys/fs/cgroup/cpu.max") ? path : "%s/cpu.max", mode);
}
""" % folder)
    subprocess.run(["gcc", "-O1", "-fPIC", "-shared", src, "-o", lib, "-ldl"], check=True)
    return lib


# ------------------------------------------------------------------------------------------- in the child process
def _fake():
    L = C.CDLL("libcudart.so.12")
    for f in ("fake_device_bytes", "fake_device_peak", "fake_room"):
        getattr(L, f).restype = C.c_size_t
    L.fake_calls.restype = L.fake_broken_captures.restype = C.c_longlong
    L.fake_calls.argtypes = [C.c_char_p]
    L.fake_fail.argtypes = [C.c_char_p, C.c_longlong]
    L.fake_slow.argtypes = [C.c_longlong, C.c_int]
    L.fake_room.argtypes = [C.c_void_p]
    return L


LAUNCH = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.c_void_p), C.c_int)
HOOK = C.CFUNCTYPE(None)


def _arg(args, i, kind):
    return C.cast(args[i], C.POINTER(kind)).contents.value


@scenario
def vad_allocation_fails(pkg, synth, fake):
    """Whatever allocation of a longer signal fails, the calls after it run on buffers of their own size."""
    cfg, tensors = synth.make_vad()
    frame = cfg["vad"]["frame_samples"]
    seen = []

    def look(name, args, recorded):
        if b"vad_lstm_kernel" in name:                   # (v, xz, f0, f1, hist, c_state, status)
            seen.append((_arg(args, 3, C.c_int), fake.fake_room(_arg(args, 4, C.c_void_p))))
        if b"vad_head_kernel" in name:                   # (v, hist, frames, probs)
            seen.append((_arg(args, 2, C.c_int), fake.fake_room(_arg(args, 1, C.c_void_p))))
            assert fake.fake_room(_arg(args, 3, C.c_void_p)) >= 4 * _arg(args, 2, C.c_int)

    cb = LAUNCH(look)
    fake.fake_on_launch(cb)
    for nth in (1, 2, 3):                                # audio, states, probabilities
        with closing(pkg.Vad(cfg["vad"], tensors)) as v:
            v.probs(np.zeros(100 * frame, np.float32))
            fake.fake_fail(b"cudaMalloc", nth)
            try:
                v.probs(np.zeros(200 * frame, np.float32))
                raise AssertionError("the allocation did not fail")
            except pkg.BackendError:
                assert fake.fake_failed()
            seen.clear()
            for frames in (50, 100, 150, 200):
                assert len(v.probs(np.zeros(frames * frame, np.float32))) == frames
            assert seen and all(room >= 512 * frames for frames, room in seen), seen


@scenario
def vad_gives_back(pkg, synth, fake):
    """What a handle keeps is bounded by the lines of its buffers, not by the longest signal it ever saw."""
    cfg, tensors = synth.make_vad()
    frame, keep = cfg["vad"]["frame_samples"], 256 << 20
    with closing(pkg.Vad(cfg["vad"], tensors)) as v:
        v.probs(np.zeros(frame, np.float32))
        small = fake.fake_device_bytes()
        line = np.zeros(keep // 4, np.float32)                   # the longest signal whose buffers stay
        v.probs(line)
        kept = fake.fake_device_bytes()
        assert kept - small > line.size * 4
        v.probs(line)
        assert fake.fake_device_bytes() == kept
        v.probs(np.zeros(keep // 4 + 64 * frame, np.float32))
        assert fake.fake_device_bytes() <= small
        assert fake.fake_device_peak() > kept
        v.probs(np.zeros(3 * frame, np.float32))
        # frames of few samples: the states have their own line
    with closing(pkg.Vad(dict(cfg["vad"], frame_samples=64, context_samples=512), tensors)) as v:
        before = fake.fake_device_bytes()
        v.probs(np.zeros(64 * 140000, np.float32))
        assert fake.fake_device_bytes() - before < (48 << 20)
    assert fake.fake_device_bytes() == 0


def _small_calls(pkg, synth):
    """Calls that between them reach the front end's groups, the decoder's lanes, the attention decoder and the streams."""
    import cases
    rng = np.random.default_rng(0)
    audio = [rng.standard_normal(16000 * s).astype(np.float32) for s in (2, 61, 1)]      # two groups of the front end
    feats = [rng.standard_normal((t, 80), dtype=np.float32) for t in (200, 6100, 90)]
    models = {}
    for name in ("tdt_q4", "ctc_q8", "aed_same", "rnnt_kq"):
        cfg, tensors = cases.build(synth, name)
        models[name] = cases.device_model(pkg, synth, cfg, tensors, **({"aed_heads": cfg.aed_heads} if name == "aed_same" else {}))

    def stream():
        with closing(models["rnnt_kq"].stream_open(2, 5, 1)) as g:
            for i in range(8):
                g.step_decode(np.zeros((2, g.need(), 128), np.float32))

    return {
        "transcribe": lambda: models["tdt_q4"].transcribe_batch(audio * 6),              # two decoder groups
        "encoder": lambda: models["ctc_q8"].encoder_forward_batch(feats),
        "aed": lambda: models["aed_same"].transcribe_batch_aed(audio[:1], cases.AED_PROMPT, -1, 5),
        "stream": stream,
    }


def _each_failure(pkg, synth, fake, functions, after):
    """Every call with the first, some and the last of its calls of each device function failing; after(what) follows."""
    for what, call in _small_calls(pkg, synth).items():
        call()                                                                           # streams, events, attributes
        for f in functions:
            fake.fake_reset()
            call()
            n = fake.fake_calls(f)
            for nth in sorted({1, 2, 3, 5, 8, n // 2, n - 1, n} & set(range(1, n + 1))):
                fake.fake_fail(f, nth)
                try:
                    call()
                    raise AssertionError((what, f, nth, "did not fail"))
                except pkg.BackendError:
                    assert fake.fake_failed()
                after((what, f, nth), call)


ASYNC = (b"cudaMemcpyAsync", b"cudaMemsetAsync", b"cudaEventRecord", b"cudaLaunchKernel")


@scenario
def error_is_reported_once(pkg, synth, fake):
    """The error of a failed device call is that call's: the next call on the thread does not find it again."""
    _each_failure(pkg, synth, fake, ASYNC, lambda what, call: call())
    import cases
    cfg, tensors = cases.build(synth, "ctc_q8")
    with closing(cases.device_model(pkg, synth, cfg, tensors)) as m:
        for f in (b"cudaMalloc", b"cudaMallocHost", b"cudaStreamCreate"):                # workspace, tables, copy stream
            fake.fake_fail(f, 1)
            try:
                m.transcribe_batch([np.zeros(16000, np.float32)], decoder=1)
                raise AssertionError((f, "did not fail"))
            except pkg.BackendError:
                assert fake.fake_failed()
        m.transcribe_batch([np.zeros(16000, np.float32)], decoder=1)


@scenario
def failed_call_waits(pkg, synth, fake):
    """A call returns with nothing in flight, also one that fails on the way: neither copies out of the caller's memory nor
    kernels on the workspace that the next call lays out anew."""
    def idle(what, call):
        assert fake.fake_pending() == 0, what
        call()
        assert fake.fake_pending() == 0, what

    _each_failure(pkg, synth, fake, ASYNC, idle)


@scenario
def launches_of_other_threads(pkg, synth, fake):
    """A thread that records a graph takes its own launches out of the count, not those of the threads beside it."""
    import threading
    import cases
    w = np.ones((64, 128), np.float32)
    x = np.ones((3, 128), np.float32)
    beside = pkg.QMat(pkg.F32, w, 64, 128)
    beside.mul(x)

    def count(call, during=0):
        hits = []

        def hook():
            t = threading.Thread(target=lambda: [beside.mul(np.ones((100, 128), np.float32)) for _ in range(during)])
            t.start()
            t.join()
            hits.append(1)

        cb = HOOK(hook)
        fake.fake_on_capture(cb)
        before = pkg.launch_count()
        call()
        fake.fake_on_capture(HOOK(0))
        assert hits, "nothing was recorded"
        return pkg.launch_count() - before

    before = pkg.launch_count()
    beside.mul(np.ones((100, 128), np.float32))
    one = pkg.launch_count() - before
    assert one > 0

    def products():
        with closing(pkg.QMat(pkg.F32, w, 64, 128)) as q:
            for _ in range(4):
                q.mul(x)

    calls = _small_calls(pkg, synth)
    cfg = synth.config("aed_f32", **dict(cases.AED["aed_same"], wtype="f32"))            # no tiles: a graph per position
    aed = cases.device_model(pkg, synth, cfg, synth.make_model(cfg, seed=1), aed_heads=cfg.aed_heads)
    for call in (products, calls["stream"], lambda: aed.aed_decode(np.ones((9, 128), np.float32), (1, 2), -1, 9)):
        call()                                                                           # buffers
        assert count(call, 3) == count(call) + 3 * one


@scenario
def qmat_workspace_is_shared(pkg, synth, fake):
    """Handles share the workspace of their products: the first product of a handle allocates nothing that another handle
    has allocated, memory does not grow with the handles that were used, and the last handle gives it back. Products that
    may overlap on the device have blocks of their own, or wait for one another there."""
    n, k, rows = 128, 512, 600                               # 2.7 MB of rows, planes and results
    w = np.ones((n, k), np.float32)
    x = np.ones((rows, k), np.float32)
    handles = [pkg.QMat(pkg.F32, w, n, k) for _ in range(12)]
    created = fake.fake_device_bytes()
    handles[0].mul(x)
    handles[0].mul(x[:2])
    used = fake.fake_device_bytes() - created
    fake.fake_reset()
    for q in handles[1:]:
        q.mul(x)
        q.mul(x[:2])                                         # (a small call, the first with these rows: not a graph yet)
    assert fake.fake_device_bytes() - created == used <= 4 << 20
    for f in (b"cudaMalloc", b"cudaFree", b"cudaHostAlloc"):
        assert fake.fake_calls(f) == 0, f

    planes = []
    cb = LAUNCH(lambda name, args, recorded: planes.append(_arg(args, 1, C.c_void_p)) if b"split" in name else None)
    fake.fake_on_launch(cb)
    L = pkg.lib()
    L.mynah_b200_qmat_mul_device.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int]
    xd, od = np.ones((rows, k), np.float32), np.ones((rows, n), np.float32)

    def device(q):
        fake.fake_reset()
        assert L.mynah_b200_qmat_mul_device(q.h, xd.ctypes.data, od.ctypes.data, rows, 0) == 0
        return planes[-1], fake.fake_calls(b"cudaStreamWaitEvent")

    busy = set()
    for q in handles[:8]:                                    # nothing waits for them on the host
        block, waits = device(q)
        assert block not in busy or waits, "a block in use was handed to another stream without a wait"
        busy.add(block)
    assert 1 < len(busy) <= 4
    block, waits = device(handles[7])                        # its own work is in order on its stream
    assert block in busy and not waits
    assert fake.fake_device_bytes() - created <= 4 * (4 << 20)
    for q in handles[:8]:
        assert L.mynah_b200_qmat_sync(q.h) == 0
    for q in handles:
        q.mul(x)
    for i, q in enumerate(handles):
        q.close()
    assert fake.fake_device_bytes() == 0


@scenario
def foreign_capture_survives(pkg, synth, fake):
    """Queries of events and streams, allocations and frees end a recording that another thread of the process makes in the
    global mode. Calls whose buffers are there already issue none that would, and neither does a product that has to grow."""
    calls = _small_calls(pkg, synth)
    calls = {k: v for k, v in calls.items() if k != "stream"}    # (opening a group allocates)
    import cases
    cfg, tensors = cases.build(synth, "ctc_q8")
    m = cases.device_model(pkg, synth, cfg, tensors)
    calls["log_mel"] = lambda: m.log_mel(np.zeros(16000, np.float32))
    handles = [pkg.QMat(pkg.F32, np.ones((128, 512), np.float32), 128, 512) for _ in range(3)]
    calls["products"] = lambda: [q.mul(np.ones((600, 512), np.float32)) for q in handles]
    for what, call in calls.items():
        call()
        fake.fake_foreign_capture(1)
        call()
        assert fake.fake_broken_captures() == 0, what
        fake.fake_foreign_capture(0)
    fake.fake_foreign_capture(1)
    handles[0].mul(np.ones((3000, 512), np.float32))
    assert fake.fake_broken_captures() == 0
    fake.fake_foreign_capture(0)


def _chain_model(pkg, synth):
    """A streaming model whose layers run as the persistent few-row chain."""
    import cases
    cfg = synth.config("chain", d_model=128, n_layers=2, n_heads=1, ffn_dim=256, n_mels=80, decoder="rnnt", vocab=33, pred_hidden=32, pred_layers=1,
                       causal=True, normalize=False, wtype="q8_0")
    return cases.device_model(pkg, synth, cfg, synth.make_model(cfg, seed=3))


class ChainArgs(C.Structure):                                # the head of FrArgs and of FrOp (fewrow.h)
    _fields_ = [("ops", C.c_void_p), ("n_ops", C.c_int)]


OP_BYTES = 256


def _table(args):
    a = C.cast(args[0], C.POINTER(ChainArgs)).contents
    return a.ops, C.string_at(a.ops, a.n_ops * OP_BYTES)


@scenario
def chain_table_copy_fails(pkg, synth, fake):
    """If the table of a chain did not reach the device, the next step copies it again: its kernel never reads a table that
    was not written."""
    m = _chain_model(pkg, synth)
    seen = []

    def look(name, args, recorded):
        if b"fr_kernel" in name:
            table = np.frombuffer(_table(args)[1], np.int32).reshape(-1, OP_BYTES // 4)
            seen.append(bool((table[:, 0] <= 3).all() and (table.any(axis=1)).all() and (table[0, 4:6] > 0).all()))

    cb = LAUNCH(look)
    fake.fake_on_launch(cb)
    for nth in range(1, 9):
        with closing(m.stream_open(2, 5, 0)) as g:
            fake.fake_reset()
            fake.fake_fail(b"cudaMemcpyAsync", nth)
            for i in range(4):
                try:
                    g.step(np.zeros((2, g.need(), 80), np.float32))
                except pkg.BackendError:
                    pass
    assert len(seen) > 16 and all(seen), seen


@scenario
def chain_graph_reads_its_own_table(pkg, synth, fake):
    """A step of another size lays the buffers of the chain out anew. A graph recorded before it must not be replayed over the
    other table: its buffers would overlap."""
    m = _chain_model(pkg, synth)
    recorded_table, replays = {}, []

    def look(name, args, recorded):
        if b"fr_kernel" in name and recorded:
            recorded_table["now"] = _table(args)
        if name == b"" and recorded_table:
            at, table = recorded_table["now"]
            replays.append(C.string_at(at, len(table)) == table)

    cb = LAUNCH(look)
    fake.fake_on_launch(cb)
    with closing(m.stream_open(2, 8, 3)) as g:
        for step in range(16):
            last = step == 10                                # a short chunk that ends an utterance; the stream goes on
            g.step(np.zeros((2, 9 if last else g.need(), 80), np.float32), last)
    assert len(replays) >= 8 and all(replays), replays


@scenario
def copies_by_pieces(pkg, synth, fake):
    """Rows and results of more pieces than there are places for arrive whole, from several threads at once, while calls of
    the transfers fail, and after the last handle has given threads and pieces back."""
    import threading
    if len(os.sched_getaffinity(0)) < 2:                     # no pieces on one core
        return
    n, k, rows = 640, 1024, 1500                             # 6.1 MB in, 3.8 MB out
    rng = np.random.default_rng(0)
    seen, errors = [], []

    def look(name, args, recorded):                          # the split reads the product's input
        if b"split_kernel" in name and _arg(args, 3, C.c_size_t) == rows * k // 4:
            at = _arg(args, 0, C.c_void_p)
            got = np.ctypeslib.as_array(C.cast(at, C.POINTER(C.c_float)), shape=(rows, k))
            seen.append(any(np.array_equal(got, x) for x in xs))

    xs = [rng.standard_normal((rows, k)).astype(np.float32) for _ in range(4)]

    def guarded(name, args, recorded):
        try:
            look(name, args, recorded)
        except BaseException as e:
            errors.append(repr(e))

    cb = LAUNCH(guarded)
    fake.fake_on_launch(cb)
    w = np.ones((n, k), np.float32)
    for life in range(2):
        handles = [pkg.QMat(pkg.F32, w, n, k) for _ in xs]
        failed = 0
        for f in (b"cudaMemcpyAsync", b"cudaEventRecord", b"cudaHostAlloc"):
            for at in (1, 2, 7, 13, 16, 20):
                fake.fake_fail(f, at)
                try:
                    handles[0].mul(xs[0])
                except pkg.BackendError:
                    failed += 1
                fake.fake_fail(b"", 0)
                handles[1].mul(xs[1])
        assert failed >= 8, failed

        def many(i):
            for _ in range(20):
                handles[i].mul(xs[i])

        threads = [threading.Thread(target=many, args=(i,)) for i in range(len(xs))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for q in handles:
            q.close()
    assert len(seen) > 160 and all(seen) and not errors, (len(seen), sum(seen), errors[:3])


def _product(pkg, fake):
    """A product of 6.1 MB in and 3.8 MB out: () -> (threads that the process has gained since now, copies of one call)."""
    def threads():
        return len(os.listdir("/proc/self/task"))

    q = pkg.QMat(pkg.F32, np.ones((640, 1024), np.float32), 640, 1024)
    x = np.ones((1500, 1024), np.float32)
    before = threads()

    def call():
        q.mul(x)
        fake.fake_reset()
        q.mul(x)
        return threads() - before, fake.fake_calls(b"cudaMemcpyAsync")

    call.close = q.close
    return call


@scenario
def copies_on_few_cores(pkg, synth, fake):
    """Helpers are counted by the cores that the process may use: on one core none, and no pieces."""
    cores = sorted(os.sched_getaffinity(0))
    os.sched_setaffinity(0, cores[:1])
    call = _product(pkg, fake)
    threads, copies = call()
    assert threads == 0 and copies <= 3, (threads, copies)
    for n in (2, 3, 4, 5):
        if len(cores) >= n:
            os.sched_setaffinity(0, cores[:n])
            threads, copies = call()
            assert threads == min(n - 1, 3) and copies > 16, (n, threads, copies)
    os.sched_setaffinity(0, cores[:1])
    assert call()[1] <= 3


@scenario
def copies_of_other_classes(pkg, synth, fake):
    """A real-time or idle thread starts no helpers, which would inherit its class, and waits for none."""
    for policy, priority in ((os.SCHED_IDLE, 0), (os.SCHED_FIFO, 1), (os.SCHED_RR, 1)):
        with closing(_product(pkg, fake)) as call:
            try:
                os.sched_setscheduler(0, policy, os.sched_param(priority))
            except PermissionError:
                continue
            threads, copies = call()
            assert threads == 0 and copies <= 3, (policy, threads, copies)
            try:
                os.sched_setscheduler(0, os.SCHED_OTHER, os.sched_param(0))
            except PermissionError:                          # out of the idle class
                break


@scenario
def copies_under_a_quota(pkg, synth, fake):
    """A control group's share of processor time counts as its cores."""
    cores = len(os.sched_getaffinity(0))
    for text, want in (("150000 100000", 1), ("50000 100000", 1), ("max 100000", cores), ("200000 100000", 2), ("350000 100000", 3)):
        with open(os.path.join(os.path.dirname(os.environ["LD_PRELOAD"]), "cpu.max"), "w") as f:
            f.write(text + "\n")
        with closing(_product(pkg, fake)) as call:           # (read when the first handle comes)
            threads, copies = call()
            want = min(want, cores, 4)
            assert threads == want - 1 and (copies > 16 if want > 1 else copies <= 3), (text, threads, copies)


@scenario
def waits_of_copies_end_in_sleep(pkg, synth, fake):
    """Helpers and the caller that wait for one another, or for the device, give up their core: a result that takes its time
    costs no processor time, and calls on one or two cores stay within a few plain copies of their bytes. (This runtime copies on the
    caller's core where a device has its link: two copies a call are its due.)"""
    import time
    cores = sorted(os.sched_getaffinity(0))
    q = pkg.QMat(pkg.F32, np.ones((1024, 4096), np.float32), 1024, 4096)
    x = np.ones((1500, 4096), np.float32)                    # 24.6 MB in, 6.1 MB out
    to = np.zeros((1500, 5120), np.float32)

    def copy():
        to[:, :4096] = x
        to[:, 4096:] = 0

    def timed(call, n=25):
        wall, cpu = [], time.process_time()
        for _ in range(n):
            time.sleep(0.002)
            t = time.perf_counter()
            call()
            wall.append(time.perf_counter() - t)
        return np.median(wall), (time.process_time() - cpu) / n

    for n in (1, 2):
        os.sched_setaffinity(0, cores[:n])
        q.mul(x)
        one = min(timed(copy) for _ in range(2))
        call = min(timed(lambda: q.mul(x)) for _ in range(3))
        assert call[0] < 2.5 * one[0] and call[1] < 4 * one[1], (n, call, one)

    os.sched_setaffinity(0, cores)
    q.mul(x)
    for at in (1, 2, 13, 14, 24):                            # waits for pieces on their way in, for the result and its pieces
        fake.fake_reset()
        fake.fake_slow(at, 300)
        cpu, t = time.process_time(), time.perf_counter()
        q.mul(x)
        cpu, t = time.process_time() - cpu, time.perf_counter() - t
        assert t > 0.3, (at, t)
        assert cpu < 0.15, (at, cpu, t)


@scenario
def copies_leave_others_alone(pkg, synth, fake):
    """While a product is being computed whose result is large, other threads make and free handles, and copy by pieces."""
    import threading
    import time
    if len(os.sched_getaffinity(0)) < 2:
        return
    slow = pkg.QMat(pkg.F32, np.ones((4096, 64), np.float32), 4096, 64)
    x = np.ones((400, 64), np.float32)                       # 0.1 MB in, 6.5 MB out
    slow.mul(x)
    with closing(_product(pkg, fake)) as call:
        threads, copies = call()
        fake.fake_slow(1, 600)                               # the first wait of the product
        done = []
        thread = threading.Thread(target=lambda: (slow.mul(x), done.append(1)))
        thread.start()
        time.sleep(0.1)
        t = time.perf_counter()
        pkg.QMat(pkg.F32, np.ones((64, 64), np.float32), 64, 64).close()
        beside = call()[1]
        t = time.perf_counter() - t
        assert not done and t < 0.4 and beside == copies > 16, (done, t, beside, copies)
        thread.join()


@scenario
def small_copies_go_the_drivers_way(pkg, synth, fake):
    """Pieces from 640 KB of rows and 512 KB of results on: below, waking the helpers costs more than they save."""
    if len(os.sched_getaffinity(0)) < 2:
        return
    for n, k, rows, copies in ((64, 1024, 159, 2), (64, 1024, 160, 3), (64, 1024, 257, 4),        # rows, and result with status
                               (1024, 64, 127, 3), (1024, 64, 128, 3), (1024, 64, 129, 4)):       # rows, status, result
        with closing(pkg.QMat(pkg.F32, np.ones((n, k), np.float32), n, k)) as q:
            x = np.ones((rows, k), np.float32)
            q.mul(x)
            fake.fake_reset()
            q.mul(x)
            assert fake.fake_calls(b"cudaMemcpyAsync") == copies, (n, k, rows, fake.fake_calls(b"cudaMemcpyAsync"))


@scenario
def ragged_audio_arrives_whole(pkg, synth, fake):
    """Signals of every length modulo the 64 bytes that a copy past the caches moves at once, from any address, and signals that
    end with a piece or a part."""
    import cases
    cfg, tensors = cases.build(synth, "ctc_q8")
    m = cases.device_model(pkg, synth, cfg, tensors)
    rng = np.random.default_rng(3)
    signal = rng.standard_normal(700000).astype(np.float32)
    seen = []

    def look(name, args, recorded):
        if b"mel_frame_kernel" in name:
            item = C.cast(_arg(args, 19, C.c_void_p), C.POINTER(C.c_void_p * 2)).contents     # (audio, n_samples, ..)
            seen.append(np.ctypeslib.as_array(C.cast(item[0], C.POINTER(C.c_float)), shape=(item[1],)).copy())

    cb = LAUNCH(look)
    fake.fake_on_launch(cb)
    for n in [163840 + i for i in range(17)] + [262143, 262144, 262145, 278528, 655359]:
        x = signal[n % 7:n % 7 + n]
        m.transcribe_batch([x], decoder=1)
        assert len(seen) == 1 and np.array_equal(seen.pop(), x), n


if __name__ == "__main__":
    sys.path.insert(0, HERE)
    import conftest
    package = conftest.load_package()
    import mynah_asr_b200.synth as synth_module
    runtime = _fake()
    assert package.available()
    SCENARIOS[sys.argv[1]](package, synth_module, runtime)
