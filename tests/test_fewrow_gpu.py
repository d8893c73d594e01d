"""The persistent few-row kernel (csrc/fewrow.cu) where its tiles end: one row, the largest rows with fused LayerNorms,
a tile and one row more, several tiles; slabs of K (one partial, one whole, two); a depthwise width without a register
path. Streams against the numpy oracle, attention-decoder batches against each utterance alone and the oracle."""
from contextlib import closing

import numpy as np
import pytest

import cases
from oracle import mynah_oracle as O, model_io

pytestmark = pytest.mark.gpu

SHAPES = {
    "partial_slab": dict(d_model=192, n_heads=6, ffn_dim=448, wtype="q8_0", use_bias=True),
    "two_slabs": dict(d_model=128, n_heads=1, ffn_dim=2048, wtype="q4_0", conv_k=5),
    "whole_slab": dict(d_model=1024, n_heads=8, ffn_dim=1024, wtype="q8_0"),
}


@pytest.mark.parametrize("shape,streams,right", [
    ("partial_slab", 1, 0), ("partial_slab", 4, 0), ("partial_slab", 5, 0), ("partial_slab", 17, 0), ("partial_slab", 64, 1),
    ("two_slabs", 1, 2), ("two_slabs", 3, 1), ("two_slabs", 33, 0), ("whole_slab", 2, 0), ("whole_slab", 9, 0)])
def test_streams(gpu_pkg, synth, shape, streams, right):
    cfg = synth.config(shape, n_layers=2, n_mels=80, decoder="rnnt", vocab=33, pred_hidden=32, pred_layers=1, causal=True,
                       normalize=False, **SHAPES[shape])
    tensors = synth.make_model(cfg, seed=3)
    with closing(cases.device_model(gpu_pkg, synth, cfg, tensors)) as dm:
        mels = np.random.default_rng(streams).standard_normal((streams, 96, 80), dtype=np.float32) - 5.0
        g, outs, pos = dm.stream_open(streams, 5, right), [], 0
        while pos < 96:
            n = min(g.need(), 96 - pos)
            outs.append(g.step(mels[:, pos:pos + n], pos + n >= 96))
            pos += n
        g.close()
        out = np.concatenate(outs, axis=1)
    M = model_io.oracle_model(cfg, tensors)
    for s in {0, streams // 2, streams - 1}:
        ref = O.stream_encode(M, mels[s], 5, right)
        assert out[s].shape == ref.shape and np.linalg.norm(out[s] - ref) < 1e-3 * np.linalg.norm(ref)


@pytest.mark.parametrize("batch", [1, 2, 4, 5, 16, 17])
def test_attention_decoder(gpu_pkg, synth, batch):
    cfg, tensors = cases.build(synth, "aed_proj")
    A = model_io.oracle_model(cfg, tensors)["aed"]
    rng = np.random.default_rng(batch)
    encs = [rng.standard_normal((3 + 5 * i, cfg.d_model), dtype=np.float32) for i in range(batch)]
    with closing(cases.device_model(gpu_pkg, synth, cfg, tensors, aed_heads=cfg.aed_heads)) as dm:
        got = dm.aed_decode_batch(encs, [cases.AED_PROMPT[:1 + i % 3] for i in range(batch)], -1, [12] * batch)
        for i in {0, batch // 2, batch - 1}:
            p = cases.AED_PROMPT[:1 + i % 3]
            assert list(got[i]) == dm.aed_decode(encs[i], p, -1, 12).tolist() == O.aed_decode(A, encs[i], p, -1, 12).tolist()


def test_streams_go_on_after_a_short_chunk(gpu_pkg, synth):
    """A short last chunk lays the buffers of the chain out anew; the graph of the steady step before it must not run over
    that layout. The same steps with spans on, which keeps graphs away, give the same bits."""
    cfg = synth.config("chain", n_layers=2, n_mels=80, decoder="rnnt", vocab=33, pred_hidden=32, pred_layers=1, causal=True,
                       normalize=False, **SHAPES["partial_slab"])
    tensors = synth.make_model(cfg, seed=3)
    mels = np.random.default_rng(5).standard_normal((6, 400, 80), dtype=np.float32) - 5.0
    outs = []
    with closing(cases.device_model(gpu_pkg, synth, cfg, tensors)) as dm:
        for graphs in (True, False):
            if not graphs:
                dm.profile_begin()
            got, pos = [], 0
            with closing(dm.stream_open(6, 8, 3)) as g:
                for step in range(12):
                    n = 9 if step == 7 else g.need()
                    got.append(g.step(mels[:, pos:pos + n], step == 7))
                    pos += n
            outs.append(got)
    assert outs[0][7].shape[1] < outs[0][6].shape[1]
    assert all(np.array_equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("d", [128, 192])
def test_layernorm_of_rows_far_from_zero(gpu_pkg, synth, d):
    """Rows of one large value c with as many elements one step above it as below: their mean is c. Squares take 48 bits, the
    sum of K of them more than the 53 of a double, so K c^2 is lost to the last units, and the variance of 2 / K or 6 / K
    steps^2 with it (d = 128: sums of squares give 0 and 8 / K) unless the sums are of differences."""
    cfg = synth.config("far", d_model=128, n_layers=1, n_heads=4, ffn_dim=256, n_mels=80, decoder="aed", vocab=211, aed_d=d,
                       aed_layers=2, aed_heads=2, aed_ffn=256, aed_max_seq=48, wtype="q8_0")
    tensors = synth.make_model(cfg, seed=4)
    tables = {n: tensors[n].raw.view(np.float32).reshape(tensors[n].shape).copy() for n in ("aed.embedding.weight", "aed.pos_enc")}
    emb, pos = tables.values()
    prompt = (3, 4, 5, 6)
    for tok, c, pairs in zip(prompt, (16777214.0, 16777213.0, 16777214.0 * 128, -16777212.0), (1, 3, 1, 3)):
        step = abs(c) - np.float64(np.nextafter(np.float32(abs(c)), np.float32(0)))
        emb[tok] = c
        for i in range(pairs):
            emb[tok, (7 * i) % d] = c + step                 # (the row's first value is one of them)
            emb[tok, d - 2 - 11 * i] = c - step
    pos[:len(prompt)] = 0
    for n, a in tables.items():
        tensors[n] = synth.Tensor(n, tensors[n].ggml_type, tensors[n].shape, a.reshape(-1).view(np.uint8))
    A = model_io.oracle_model(cfg, tensors)["aed"]
    enc = np.random.default_rng(2).standard_normal((11, cfg.d_model), dtype=np.float32)
    with closing(cases.device_model(gpu_pkg, synth, cfg, tensors, aed_heads=cfg.aed_heads)) as dm:
        for n in range(1, 5):
            for p in (prompt[:n], prompt[n - 1:n]):
                assert dm.aed_decode(enc, p, -1, 12).tolist() == O.aed_decode(A, enc, p, -1, 12).tolist(), p
