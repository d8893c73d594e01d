"""The attention decoder as launches: where its linears have no tiles for the persistent kernel (other formats than Q8_0 and
Q4_0) or the batch has more than 128 utterances, positions are replayed from a graph of the few-row contraction
(csrc/gemm_skinny.cu) and the attention and selection kernels of csrc/decoder_aed.cu. The same weights as f32 hold the
reference's tokens for these models (tests/golden/ref_aed_*.npz); 128 is a width with LayerNorms inside the contractions
and one launch between positions, 64 one without."""
import os
from contextlib import closing

import numpy as np
import pytest

import cases
from oracle import mynah_oracle as O, model_io

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


@pytest.fixture(scope="module", params=list(cases.AED))
def as_f32(request, gpu_pkg, synth):
    cfg, tensors = cases.build(synth, request.param)
    plain = {n: synth.Tensor(n, 0, tensors[n].shape, np.ascontiguousarray(w, np.float32).reshape(-1).view(np.uint8))
             for n, w in model_io.effective_f32(tensors).items()}
    dm = cases.device_model(gpu_pkg, synth, cfg, plain, aed_heads=cfg.aed_heads)
    yield gpu_pkg, dm, model_io.oracle_model(cfg, plain)["aed"], np.load(os.path.join(GOLD, f"ref_{request.param}.npz"))
    dm.close()


def _launched(pkg, call, positions):
    before = pkg.launch_count()
    out = call()
    assert pkg.launch_count() - before > 8 * positions           # every position is launches: the path this file is about
    return out


def test_decoder_on_reference_encoder_output(as_f32):
    pkg, dm, A, g = as_f32
    for i in range(2):
        enc = g[f"enc{i}"]
        got = _launched(pkg, lambda: dm.aed_decode(enc, cases.AED_PROMPT, -1, cases.AED_CAP), cases.AED_CAP)
        assert got.tolist() == g[f"tokens{i}"].tolist()
        assert dm.aed_decode(enc, cases.AED_PROMPT, int(g[f"eos{i}"]), cases.AED_CAP).tolist() == g[f"tokens_eos{i}"].tolist()
        assert dm.aed_decode(enc, cases.AED_PROMPT[:1], -1, cases.AED_CAP).tolist() == g[f"tokens_start{i}"].tolist()


@pytest.mark.parametrize("batch", [2, 3, 9, 17])
def test_batch_equals_single_and_oracle(as_f32, batch):
    """Different lengths, prompts and budgets in lock step; one utterance runs into the end of the position table."""
    pkg, dm, A, g = as_f32
    rng = np.random.default_rng(batch)
    encs = [rng.standard_normal((3 + 5 * i, g["enc0"].shape[1]), dtype=np.float32) for i in range(batch)]
    prompts = [cases.AED_PROMPT[:1 + i % 4] for i in range(batch)]
    limits = [1000 if i == 1 else 4 + i for i in range(batch)]
    eos = int(g["eos1"])
    got = _launched(pkg, lambda: dm.aed_decode_batch(encs, prompts, eos, limits), 4)
    for i in {0, 1, batch // 2, batch - 1}:
        assert list(got[i]) == dm.aed_decode(encs[i], prompts[i], eos, limits[i]).tolist() == O.aed_decode(A, encs[i], prompts[i], eos, limits[i]).tolist()


def test_more_utterances_than_the_persistent_kernel_takes(gpu_pkg, synth):
    cfg, tensors = cases.build(synth, "aed_same")
    A = model_io.oracle_model(cfg, tensors)["aed"]
    rng = np.random.default_rng(1)
    encs = [rng.standard_normal((3 + i % 7, cfg.d_model), dtype=np.float32) for i in range(129)]
    with closing(cases.device_model(gpu_pkg, synth, cfg, tensors, aed_heads=cfg.aed_heads)) as dm:
        got = _launched(gpu_pkg, lambda: dm.aed_decode_batch(encs, [cases.AED_PROMPT[:2]] * 129, -1, [12] * 129), 12)
        before = gpu_pkg.launch_count()
        fewer = dm.aed_decode_batch(encs[:128], [cases.AED_PROMPT[:2]] * 128, -1, [12] * 128)
        assert gpu_pkg.launch_count() - before < 60              # one launch for all positions
        for i in (0, 64, 127, 128):
            assert list(got[i]) == O.aed_decode(A, encs[i], cases.AED_PROMPT[:2], -1, 12).tolist()
            assert i == 128 or list(fewer[i]) == list(got[i])
