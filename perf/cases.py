"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values: `kind` names the entry point, the rest its sizes and options.

  qmat        one product of a resident quantised weight with host rows (QMat.mul), what a host program that keeps
              its own encoder calls for every linear
  transcribe  audio in, token ids out (Model.transcribe_batch): the offline path of the CTC, TDT and RNNT models
  encoder     features in, encoder frames out (Model.encoder_forward_batch), in the two numerics that a caller can
              choose instead of the default: one fp16 product per term ("fast") and int8 activations ("a8")
  aed         audio in, token ids out through the attention decoder (Model.transcribe_batch_aed)
  stream      one chunk of every stream of a group: the encoder step (StreamGroup.step), for a program that decodes
              itself, or the step and greedy decoding (StreamGroup.step_decode)
  plan        cutting a long recording where nobody speaks (plan_segments with the voice activity network)

Models have the architectures of this repository's configurations with seeded random weights. A program loads its
model once, so a model is made once per process and shared by the states that use it.
"""
import importlib.util
import os
import sys

import numpy as np

ROOT = os.getcwd()


def _package():
    if "mynah_asr_b200" not in sys.modules:
        folder = os.path.join(ROOT, "mynah-asr_b200")
        spec = importlib.util.spec_from_file_location("mynah_asr_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        sys.modules["mynah_asr_b200"] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules["mynah_asr_b200"])
    return sys.modules["mynah_asr_b200"]


pkg = _package()
import mynah_asr_b200.synth as synth  # noqa: E402

RATE, HOP = 16000, 160
PROMPT, EOS, DELTA = (3, 4, 5, 6, 7), 2, 50           # start tokens, end token and allowance beyond the encoder frames
# blank bias of the transducer heads: the greedy stream then has a few tokens per second, as speech has
BLANK_BIAS = {"cfg1": 1.2, "cfg2": 3.1, "cfg3": 2.4}
BYTES = {"f32": 4.0, "q8_0": 34 / 32, "q4_0": 18 / 32, "q4_k": 144 / 256, "q6_k": 210 / 256}


def listed():
    return [
        # a single activation row through one linear: the smallest call there is, latency alone
        dict(name="qmat_row", kind="qmat", rows=1, fmt="q4_0", n=4096, k=1024),
        # the rows of a 15 s utterance through a down projection, many-row kernel and host copies both ways
        dict(name="qmat_rows", kind="qmat", rows=187, fmt="q8_0", n=1024, k=4096),
        # a voice command: one short utterance through the small CTC model
        dict(name="ctc_short", kind="transcribe", model="cfg0", items=1, min_s=3.7, max_s=3.7),
        # a server's batch of ragged requests on the small model, single-product numerics
        dict(name="encoder_fast", kind="encoder", model="cfg0", mode="fast", items=12, min_s=2.0, max_s=31.0),
        # one minute of audio, one user waiting for it
        dict(name="tdt_one", kind="transcribe", model="cfg1", items=1, min_s=60.0, max_s=60.0),
        # the benchmark's step: a full batch of one-minute recordings
        dict(name="tdt_batch", kind="transcribe", model="cfg1", items=16, min_s=60.0, max_s=60.0),
        # a ragged batch with int8 activations on natively quantised weights
        dict(name="encoder_a8", kind="encoder", model="cfg1", mode="a8", items=8, min_s=5.0, max_s=30.0),
        # bulk transcription of recordings of every length on the deepest model, K-quants: the largest case
        dict(name="rnnt_ragged", kind="transcribe", model="cfg2", items=32, min_s=5.0, max_s=120.0),
        # live captioning of one speaker
        dict(name="stream_one", kind="stream", streams=1, right=0, decode=False),
        # a captioning server: 64 speakers in lock step
        dict(name="stream_group", kind="stream", streams=64, right=0, decode=True),
        # sentences through the attention decoder
        dict(name="aed_batch", kind="aed", model="cfg4", items=8, min_s=7.0, max_s=13.0),
        # a five-minute recording cut into segments before it is transcribed
        dict(name="plan", kind="plan", seconds=300.0, segment=30.0),
    ]


def draw(rng):
    def log(lo, hi):
        return lo * (hi / lo) ** rng.random()

    def spread(lo, hi):                                  # two lengths, in order
        a, b = sorted((round(log(lo, hi), 3), round(log(lo, hi), 3)))
        return dict(min_s=a, max_s=b)

    kind = rng.choice(("qmat", "transcribe", "transcribe", "encoder", "stream", "stream", "aed", "plan"))
    if kind == "qmat":
        n, k = rng.choice(((4096, 1024), (1024, 4096), (1024, 1024), (2048, 1024), (2048, 512), (512, 2048), (512, 512)))
        return dict(kind=kind, rows=int(log(1, 600)), fmt=rng.choice(("q4_0", "q8_0", "q4_k", "q6_k")), n=n, k=k)
    if kind == "transcribe":
        model = rng.choice(("cfg0", "cfg1", "cfg2"))
        return dict(kind=kind, model=model, items=int(log(1, 17)), **spread(1.0, 60.0))
    if kind == "encoder":
        model, mode = rng.choice((("cfg0", "fast"), ("cfg1", "a8")))
        return dict(kind=kind, model=model, mode=mode, items=int(log(1, 13)), **spread(1.5, 40.0))
    if kind == "stream":
        n = int(log(1, 513))                             # few streams rarely say a token in one chunk
        return dict(kind=kind, streams=n, right=rng.choice((0, 0, 1)), decode=n >= 32 and rng.random() < 0.5)
    if kind == "aed":
        return dict(kind=kind, model="cfg4", items=int(log(1, 13)), **spread(2.0, 15.0))
    return dict(kind=kind, seconds=round(log(20.0, 600.0), 2), segment=rng.choice((15.0, 30.0, 60.0)))


# ------------------------------------------------------------------------------------------------------- models
_models = {}


def _config(name):
    return synth.config(name, blank_bias=BLANK_BIAS.get(name, 0.0))


def _tensors(cfg, native_int8):
    """The architecture's tensors. The generator makes one encoder layer; the others are that layer with the rows of
    every matrix in another order, so that no two layers are alike and a model is ready in a second or two. Linears
    have a deviation under which the signal still varies over time behind the last layer."""
    layers = cfg.n_layers
    cfg.n_layers = 1
    if native_int8:
        cfg.wtype, cfg.wtype_out = "f32", ""
    first = synth.make_model(cfg, seed=0, weight_std=0.32 / float(np.sqrt(cfg.d_model)))
    if native_int8:
        first = synth.to_native_int8(first, lambda kind, raw: raw.view(np.float32))
    cfg.n_layers = layers
    out = dict(first)
    head = "encoder.layers.0."
    for name, t in first.items():
        if not name.startswith(head):
            continue
        for li in range(1, layers):
            raw = t.raw
            if ".weight" in name and (len(t.shape) == 2 or name.endswith(".scales")) and t.shape[0] > 1:
                raw = np.roll(raw.reshape(t.shape[0], -1), 37 * li, axis=0)
            to = "encoder.layers.%d.%s" % (li, name[len(head):])
            out[to] = synth.Tensor(to, t.ggml_type, t.shape, raw)
    return out


def _model(name, mode="strict"):
    if (name, mode) not in _models:
        cfg = _config(name)
        _models[name, mode] = cfg, pkg.Model(
            _tensors(cfg, mode == "a8"), n_mels=cfg.n_mels, mel_fb=synth.mel_filterbank(cfg.n_mels), window=synth.hann_window(),
            causal=int(cfg.causal), normalize=cfg.normalize, left=cfg.left, right=cfg.right, blank=cfg.vocab - 1,
            max_symbols=cfg.max_symbols, durations=tuple(cfg.durations), strict=mode != "fast", aed_heads=cfg.aed_heads,
            a8=mode == "a8")
    return _models[name, mode]


def _vad():
    if "vad" not in _models:
        cfg, tensors = synth.make_vad()
        _models["vad"] = pkg.Vad(cfg["vad"], tensors)
    return _models["vad"]


# ------------------------------------------------------------------------------------------------------- inputs
def _samples(case):
    """Samples of each utterance of a batch: spread evenly at random between the case's two lengths."""
    r = np.random.default_rng([case["items"], int(case["min_s"] * 1000), int(case["max_s"] * 1000)])
    return [int(s * RATE) for s in r.uniform(case["min_s"], case["max_s"], case["items"])]


def _frames(cfg, samples):
    t = samples // HOP
    for _ in range(3):
        t = (t + (3 if cfg.causal else 2) - 3) // 2 + 1
    return t


def _audio(rng, n):
    """Noise under a 4 Hz envelope, 16-bit samples as floats: the level and the modulation of speech."""
    env = np.float32(1500.0) * (1.0 + np.sin(np.arange(n, dtype=np.float32) * np.float32(8.0 * np.pi / RATE)))
    return np.rint(np.clip(rng.standard_normal(n, dtype=np.float32) * env, -32768, 32767)) / np.float32(32768.0)


def _mel(rng, *shape):
    """Log-mel features [..., frames, bands], neighbouring frames alike."""
    x = rng.standard_normal(shape, dtype=np.float32)
    x[..., 1:, :] = np.float32(0.8) * x[..., 1:, :] + np.float32(0.6) * x[..., :-1, :]
    return x


def _blocks(rng, fmt, n, k):
    return synth.QUANTIZERS[synth.GGML_NAMES[fmt]](rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))


class _Streams:
    """A group of streams in the middle of its life: the caches are full."""

    def __init__(self, case, seed):
        cfg, model = _model("cfg3")
        rng = np.random.default_rng(seed)
        self.group = model.stream_open(case["streams"], cfg.left, case["right"])
        self.symbols, self.q = cfg.max_symbols, case["right"] + 1
        first = _mel(rng, case["streams"], self.group.need(), cfg.n_mels) - np.float32(6.0)
        self.group.step(first)
        need = self.group.need()
        self.chunks = [_mel(rng, case["streams"], need, cfg.n_mels) - np.float32(6.0) for _ in range(8)]
        self.at = 0
        for _ in range(cfg.left // self.q + 4):
            self.group.step(self.next())
        self.frame = 0                                    # frames decoded so far

    def next(self):
        self.at += 1
        return self.chunks[self.at % len(self.chunks)]

    def __del__(self):
        self.group.close()


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "qmat":
        fmt = {"q4_0": pkg.GGML_Q4_0, "q8_0": pkg.GGML_Q8_0, "q4_k": pkg.GGML_Q4_K, "q6_k": pkg.GGML_Q6_K}[case["fmt"]]
        w = pkg.QMat(fmt, _blocks(rng, case["fmt"], case["n"], case["k"]), case["n"], case["k"])
        return dict(case=case, w=w, x=rng.standard_normal((case["rows"], case["k"]), dtype=np.float32))
    if kind == "stream":
        return dict(case=case, streams=_Streams(case, seed))
    if kind == "plan":
        return dict(case=case, vad=_vad(), audio=synth.speech_like_audio(case["seconds"], seed=seed))
    cfg, model = _model(case["model"], case.get("mode", "strict"))
    samples = _samples(case)
    state = dict(case=case, cfg=cfg, model=model, frames=[_frames(cfg, n) for n in samples])
    if kind == "encoder":
        state["mel"] = [_mel(rng, n // HOP, cfg.n_mels) for n in samples]
    else:
        state["audio"] = [_audio(rng, n) for n in samples]
    return state


# --------------------------------------------------------------------------------------------------------- runs
def _by_frame(results, frames, symbols, first=0):
    """Token ids where they were spoken: [all frames, symbols per frame], -1 where there is none."""
    out = np.full((sum(frames), symbols), -1, np.int32)
    base = 0
    for (tokens, at), n in zip(results, frames):
        if tokens:
            at = np.asarray(at) - first
            rank = np.arange(at.size) - np.searchsorted(at, at)           # the how-manieth of its frame
            out[base + at, rank] = tokens
        base += n
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "qmat":
        return state["w"].mul(state["x"])
    if kind == "transcribe":
        cfg = state["cfg"]
        got = state["model"].transcribe_batch(state["audio"], 1 if cfg.decoder == "ctc" else 0)
        return _by_frame(got, state["frames"], 1 if cfg.decoder == "ctc" else cfg.max_symbols)
    if kind == "encoder":
        return state["model"].encoder_forward_batch(state["mel"])
    if kind == "aed":
        got = state["model"].transcribe_batch_aed(state["audio"], PROMPT, EOS, DELTA)
        out = np.full((len(got), max(state["frames"]) + DELTA), -1, np.int32)
        for row, tokens in zip(out, got):
            row[:len(tokens)] = tokens
        return out
    if kind == "stream":
        s = state["streams"]
        if not case["decode"]:
            return s.group.step(s.next())
        got = s.group.step_decode(s.next())
        s.frame += s.q
        return _by_frame(got, [s.q] * s.group.n, s.symbols, s.frame - s.q)
    got = pkg.plan_segments(state["audio"], RATE, case["segment"], state["vad"])
    out = np.full((int(case["seconds"]) + 2, 2), -1, np.int64)            # no more segments than seconds
    out[:len(got)] = got
    return out


# --------------------------------------------------------------------------------------------------------- work
def _front(cfg, samples):
    """(flops, parameters) of the mel and subsampling stages for one utterance."""
    C, t, f, flops = cfg.channels, samples // HOP, cfg.n_mels, 0.0
    flops += t * 5.0 * 512 * 9
    for stage in range(3):
        t, f = ((v + (3 if cfg.causal else 2) - 3) // 2 + 1 for v in (t, f))
        flops += 2.0 * t * f * C * (9 + (C if stage else 0))
    return flops + 2.0 * t * f * C * cfg.d_model, 27 * C + 2 * C * C + f * C * cfg.d_model


def _layers(cfg, frames, keys):
    """(flops, bytes of the stored weights) of the encoder stack over `frames` rows that each see `keys` keys."""
    d, F = cfg.d_model, cfg.ffn_dim
    linears = 4 * d * F + 7 * d * d
    flops = cfg.n_layers * frames * (2.0 * linears + 6.0 * keys * d + 2.0 * cfg.conv_k * d)
    return flops, cfg.n_layers * (linears * BYTES[cfg.wtype] + 4.0 * d * d)


def _head(cfg, frames, seconds):
    """(flops, bytes of the stored weights) of the decoder: three tokens a second where nothing else is known."""
    H, V, tokens = cfg.pred_hidden, cfg.vocab + len(cfg.durations), 3.0 * seconds
    if cfg.decoder == "ctc":
        return 2.0 * frames * V * cfg.d_model, V * cfg.d_model * BYTES[cfg.wtype]
    lstm = cfg.pred_layers * 8 * H * H + H * H
    steps = tokens + frames / (max(cfg.durations) if cfg.durations else 1)
    return 2.0 * frames * cfg.d_model * H + 2.0 * tokens * lstm + 2.0 * steps * V * H, \
        4.0 * (lstm + cfg.d_model * H) + V * H * BYTES[cfg.wtype]


def work(case):
    kind = case["kind"]
    if kind == "qmat":
        r, n, k = case["rows"], case["n"], case["k"]
        return dict(bytes=n * k * BYTES[case["fmt"]] + 4.0 * r * (n + k), flops=2.0 * r * n * k)
    if kind == "plan":                                   # 0.55 MFLOP of the voice activity network per 512 samples
        n = case["seconds"] * RATE
        return dict(bytes=4.0 * n, flops=0.55e6 * n / 512)
    if kind == "stream":
        cfg = _config("cfg3")
        q, s = case["right"] + 1, case["streams"]
        flops, weights = _layers(cfg, s * q, cfg.left + q)
        f2, front = _front(cfg, 8 * q * HOP)
        f3, head = _head(cfg, s * q, 0.08 * q * s)
        caches = cfg.n_layers * s * cfg.left * 2 * cfg.d_model * 2.0
        if not case["decode"]:                           # the projector alone
            f3, head = 2.0 * s * q * cfg.d_model * cfg.pred_hidden, 4.0 * cfg.d_model * cfg.pred_hidden
        moved = 4.0 * s * q * (8 * cfg.n_mels + (0 if case["decode"] else cfg.pred_hidden))
        return dict(bytes=weights + 4.0 * front + head + caches + moved, flops=flops + s * f2 + f3)
    cfg = _config(case["model"])
    if case.get("mode") == "a8":
        cfg.wtype = "q8_0"
    samples = _samples(case)
    frames = [_frames(cfg, n) for n in samples]
    flops = sum(_layers(cfg, t, t)[0] + _front(cfg, n)[0] for t, n in zip(frames, samples))
    moved = _layers(cfg, 1, 1)[1] + 4.0 * _front(cfg, HOP * 100)[1]
    if kind == "encoder":
        width = cfg.d_out
        flops += 2.0 * sum(frames) * cfg.d_model * (width if width != cfg.d_model else 0)
        return dict(flops=flops, bytes=moved + 4.0 * sum(n // HOP * cfg.n_mels for n in samples) + 4.0 * sum(frames) * width)
    moved += 4.0 * sum(samples)
    if kind == "transcribe":
        f, b = _head(cfg, sum(frames), sum(samples) / RATE)
        return dict(flops=flops + f, bytes=moved + b)
    D, V = cfg.aed_d, cfg.vocab                          # positions one after the other, each over the whole decoder
    per = cfg.aed_layers * (6 * D * D + 2 * D * cfg.aed_ffn) + V * D
    steps = [t + DELTA + len(PROMPT) for t in frames]
    flops += 2.0 * sum(t * cfg.aed_layers * 2 * D * D for t in frames)
    flops += sum(s * (2.0 * per + cfg.aed_layers * 4.0 * D * (t + s / 2)) for s, t in zip(steps, frames))
    return dict(flops=flops, bytes=moved + BYTES[cfg.wtype] * (per + cfg.aed_layers * 2 * D * D))


def tolerance(case):
    kind = case["kind"]
    if kind == "qmat":
        return dict(rel=1e-5)                            # f32-grade products and sums
    if kind == "encoder":
        # one fp16 product per term through every layer; int8 activations, where a value at a rounding boundary may
        # go either way and a step is 1/127 of a row's largest value
        return dict(rel=2e-3) if case["mode"] == "fast" else dict(rel=2.5e-2)
    if kind == "plan":
        return "exact"
    if kind == "stream" and not case["decode"]:
        return dict(rel=1e-4)                            # 24 layers, keys and values rounded to fp16 in each
    return dict(differ=0.01)                             # ties between two logits
