"""Kernels and dispatch branches at the sizes where they change over: row tiles of 64 and 128, repeated calls and growing
buffers of a resident weight, the vector widths of the int8 row quantiser, batched front ends, q | k | v as one
contraction, and the pieces in which a signal goes through the voice activity network."""
from contextlib import closing

import numpy as np
import pytest

import cases
from oracle import mynah_oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("n,k", [(1024, 4096), (40, 64), (320, 192)])
def test_product_rows(gpu_pkg, synth, n, k):
    """Every row count at the edges of the tiles, in an order that makes the buffers grow between calls, three calls each
    (the third repeats what the second one recorded) on different inputs."""
    rng = np.random.default_rng(n)
    raw = synth.QUANTIZERS[synth.GGML_NAMES["q8_0"]](rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.05))
    w = O.ggml_dequant(synth.GGML_NAMES["q8_0"], raw).reshape(n, k).astype(np.float64)
    q = gpu_pkg.QMat(gpu_pkg.GGML_Q8_0, raw, n, k)
    for rows in (1, 2, 8, 9, 17, 63, 64, 65, 128, 129, 257, 64, 1, 700, 9):
        for again in range(3):
            x = rng.standard_normal((rows, k), dtype=np.float32)
            assert rel(q.mul(x), x.astype(np.float64) @ w.T) < 2e-5, (rows, again)
    q.close()


@pytest.mark.parametrize("k", [512, 1024, 2048, 4096, 256, 1536])
def test_int8_rows(gpu_pkg, k):
    """Quantised activation rows, bit for bit, at every vector width and at row counts that leave warps idle."""
    rng = np.random.default_rng(k)
    q8, s8 = O.quantize_int8(rng.uniform(-1, 1, (128, k)).astype(np.float32))
    q = gpu_pkg.QMat(gpu_pkg.MYNAH_Q8, q8, 128, k, scales=s8)
    for rows in (17, 18, 19, 33, 135):
        x = (rng.standard_normal((rows, k)) * rng.uniform(0.1, 30, (rows, 1))).astype(np.float32)
        x[rows // 2] = 0.0
        assert np.array_equal(q.mul(x, gpu_pkg.A8), O.qmat_mul_a8_q8(x, q8, s8)), rows
    q.close()


@pytest.mark.parametrize("items", [2, 17, 33])
def test_ragged_batches(gpu_pkg, synth, items):
    """Utterances from a few frames up, more than one group of them: the same bits as each alone, tokens too."""
    cfg, tensors = cases.build(synth, "tdt_q4")
    with closing(cases.device_model(gpu_pkg, synth, cfg, tensors)) as dm:
        audio = [synth.synth_audio(0.1 + 0.13 * ((7 * i) % 19), seed=i) for i in range(items)]
        got = dm.transcribe_batch(audio, 0)
        feats = [dm.log_mel(a) for a in audio]
        feats = [f[:v] for f, v in feats]
        outs = dm.encoder_forward_batch(feats)
        for i in sorted({0, 1, items // 2, items - 1}):
            assert np.array_equal(outs[i], dm.encoder_forward(feats[i])), i
            one = dm.transcribe_batch(audio[i:i + 1], 0)[0]
            assert list(got[i][0]) == list(one[0]) and list(got[i][1]) == list(one[1]), i


@pytest.mark.parametrize("frames", [1, 15, 16, 17, 255, 256, 257, 511, 513, 1279, 1280, 1281])
def test_voice_activity_pieces(gpu_pkg, synth, frames):
    """The network is causal: a prefix has the first probabilities of the whole signal, wherever the pieces end."""
    cfg, tensors = synth.make_vad()
    a = synth.speech_like_audio(1300 * 512 / 16000, seed=2)
    with closing(gpu_pkg.Vad(cfg["vad"], tensors)) as v:
        whole = v.probs(a)
        got = v.probs(a[:frames * 512])
        assert got.shape == (frames,) and np.abs(got - whole[:frames]).max() < 1e-6
        assert np.array_equal(v.probs(a[:frames * 512]), got)
