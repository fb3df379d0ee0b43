"""Edges of the kernels that serve few rows: the f32 and int4 GEMVs (column and row tiles, K slices, splits over a
cluster, a LayerNorm taken along), the split-context decode attention (stages, splits, clusters) and the int4 GEMM's
epilogues.  Each is compared with float64 of the same operands; sums of n f32 terms may differ from it by
n * 2^-24 of the terms' magnitudes at most, and the bounds below are a fraction of that for the longest sum.
"""
import time

import numpy as np
import pytest

import b200nn
import np_ref
import test_gpu_vivezen as vivezen
import test_gpu_zufilorn as zufilorn
from b200nn import Gpt2Config, Gpt2Model, GpuTensor, Int4Gpt2Model, Int4Linear, Int4TransformerBlock, Linear, TransformerBlock, ops, synth
from oracle import oracle
from test_gpu_block import _int4_oracle, _slices

pytestmark = pytest.mark.gpu


def _close(got, ref, mag):
    """f32 sums in another order: within 2e-6 of the sum of the terms' magnitudes."""
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) <= 2e-6 * mag + 1e-30).all(), np.max(np.abs(got - ref) / mag)


@pytest.mark.parametrize("m", [1, 2, 3, 4])
# activations staged in pieces, with and without a K split; the last weight of 32-column tiles and the first of 128-column ones
# (148 SMs)
@pytest.mark.parametrize("k,n", [(1, 1), (63, 33), (64, 32), (65, 31), (768, 2304), (3072, 770), (20000, 40), (100, 50257), (100000, 64), (10500, 2401),
                                 (97, 14208), (97, 14209), (1, 14336), (800, 14401)])
def test_f32_linear_few_rows(reg, m, k, n):
    rng = np.random.default_rng(k * 7 + n + m)
    w, b, x = (rng.standard_normal(s).astype(np.float32) for s in ((n, k), (n,), (m, k)))
    ref, mag = x.astype(np.float64) @ w.T + b, np.abs(x).astype(np.float64) @ np.abs(w).T + np.abs(b)
    _close(Linear(w, b, k, n, reg).forward(GpuTensor.from_host(x, (m, k), reg)).to_host(), ref, mag)
    # a matrix product takes the weight as it is: rows that need not start on 16 bytes
    got = ops.matmul(GpuTensor.from_host(x, (m, k), reg), GpuTensor.from_host(np.ascontiguousarray(w.T), (k, n), reg), reg).to_host()
    _close(got, ref - b, mag)


def _seconds(reg, f, n=20):
    """A call's time, the best of five rounds."""
    f()
    best = []
    for _ in range(5):
        reg.synchronize()
        t = time.perf_counter()
        for _ in range(n):
            f()
        reg.synchronize()
        best.append((time.perf_counter() - t) / n)
    return min(best)


def _linear_seconds(reg, k, n, m):
    layer = Linear(np.ones((n, k), np.float32), None, k, n, reg)
    x = GpuTensor.from_host(np.ones((m, k), np.float32), (m, k), reg)
    return _seconds(reg, lambda: layer.forward(x))


def test_f32_linear_of_very_long_rows_keeps_its_pace(reg):
    """1.7 times the bytes; on the tiled kernel the longer one took 400 times as long."""
    assert _linear_seconds(reg, 100000, 64, 1) < 6 * _linear_seconds(reg, 60000, 64, 1)


def test_f32_linear_of_long_rows_and_many_columns(reg):
    """Wide tiles whose activations are staged in pieces."""
    import torch

    k, n, m = 10300, 14212, 4
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    w, x = torch.randn(n, k, generator=g, device="cuda"), torch.randn(m, k, generator=g, device="cuda")
    ref, mag = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    got = Linear(w.cpu().numpy(), None, k, n, reg).forward(GpuTensor.from_host(x.cpu().numpy(), (m, k), reg)).to_host()
    _close(got, ref.cpu().numpy(), mag.cpu().numpy())


def test_f32_output_matrix_of_four_rows_keeps_its_pace(reg):
    """The weight's bytes bound it: four rows took 2.3 times as long as one while a block per SM was all their registers left."""
    assert _linear_seconds(reg, 768, 50257, 4) < 1.9 * _linear_seconds(reg, 768, 50257, 1)


def _int4(rng, k, n, group):
    q = rng.integers(-8, 8, (k, n))
    s = (rng.random(((k + group - 1) // group, n)) * 0.015 + 0.005).astype(np.float16).astype(np.float32)
    packed = ((q + 8).reshape(k // 8, 8, n).astype(np.uint64) << (4 * np.arange(8, dtype=np.uint64)).reshape(1, 8, 1)).sum(1).astype(np.uint32)
    return q * np.repeat(s.astype(np.float64), group, 0)[:k], packed, s


@pytest.mark.parametrize("m", [1, 2, 3, 4, 7])
# one block of K, ragged rows, K split over a cluster, the last weight of 32-row blocks and the first of 128-row ones
@pytest.mark.parametrize("k,n,group", [(64, 1, 64), (128, 33, 128), (1600, 1600, 128), (6400, 130, 128), (3072, 768, 64),
                                       (1088, 9472, 64), (128, 9473, 128), (64, 50257, 64)])
def test_int4_linear_few_rows(reg, m, k, n, group):
    rng = np.random.default_rng(k + n + m)
    w, packed, s = _int4(rng, k, n, group)
    x, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    reg.set_tuning("gemv_max_rows", 8)
    try:
        got = Int4Linear(packed, s, b, k, n, group, reg).forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    finally:
        reg.set_tuning("gemv_max_rows", -1)
    _close(got, x.astype(np.float64) @ w + b, np.abs(x).astype(np.float64) @ np.abs(w) + np.abs(b))


@pytest.mark.parametrize("m", [3, 32, 33, 65, 130, 300])
@pytest.mark.parametrize("k,n", [(128, 128), (192, 132), (1600, 257), (64, 19000)])
def test_int4_linear_epilogues(reg, m, k, n):
    """Rows that leave in 16-byte pieces and rows that start anywhere, with and without splits; fp16 operands, so the reference
    multiplies the rounded ones."""
    rng = np.random.default_rng(m * 31 + n)
    w, packed, s = _int4(rng, k, n, 64)
    x, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    got = Int4Linear(packed, s, b, k, n, 64, reg).forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    xh, wh = x.astype(np.float16).astype(np.float64), w.astype(np.float16).astype(np.float64)
    _close(got, xh @ wh + b, np.abs(xh) @ np.abs(wh) + np.abs(b))


@pytest.mark.parametrize("d", [128, 768, 1600, 2048, 2112])
@pytest.mark.parametrize("int4", [False, True])
def test_block_with_a_layernorm_taken_along(reg, int4, d):
    """One to four new rows on cached ones, the LayerNorms applied by the GEMV behind them up to 2048 columns (int4: one and two
    rows), against float64."""
    cfg = Gpt2Config(n_layer=1, n_embd=d, n_head=d // 64, vocab_size=64, n_positions=32)
    w = synth.gpt2_weights(cfg, base_seed=d, std=1.5 / d ** 0.5, random_ln=True)
    blk = Int4TransformerBlock(*_slices(w), cfg, reg, group_size=64) if int4 else TransformerBlock(*_slices(w), cfg, reg)
    om = oracle.Model(cfg.as_dict(), _int4_oracle(w, cfg, 64) if int4 else w)
    x = np.random.default_rng(d).standard_normal((12, d)).astype(np.float32)
    ref = om.block_forward(0, x, flags=oracle.KV_FP16)[0]
    for n in (1, 2) if int4 else (1, 2, 3, 4): # (more int4 rows go to the tensor cores)
        past = 12 - n
        _, k0, v0 = blk.forward_cached(GpuTensor.from_host(x[:past], (past, d), reg), None, None, 0)
        got = blk.forward_cached(GpuTensor.from_host(x[past:], (n, d), reg), k0, v0, past)[0].to_host()
        for i in range(n):
            assert np_ref.rel_rms(got[i], ref[past + i]) < 1e-3, (n, i, np_ref.rel_rms(got[i], ref[past + i]))


def test_rows_after_rows(reg):
    """Blocks of one to four f32 rows one after another: every kernel is resident before its input is written, so an old line
    of the residual stream or of the buffers that the calls share would show."""
    d = 192
    cfg = Gpt2Config(n_layer=1, n_embd=d, n_head=d // 64, vocab_size=64, n_positions=64)
    w = synth.gpt2_weights(cfg, base_seed=5, std=0.06, random_ln=True)
    blk, om = TransformerBlock(*_slices(w), cfg, reg), oracle.Model(cfg.as_dict(), w)
    for turn, n in enumerate((1, 2, 3, 4, 4, 3, 4, 1, 4)):
        x = np.random.default_rng(turn).standard_normal((20, d)).astype(np.float32)
        ref = om.block_forward(0, x, flags=oracle.KV_FP16)[0]
        past = 20 - n
        _, k0, v0 = blk.forward_cached(GpuTensor.from_host(x[:past], (past, d), reg), None, None, 0)
        got = blk.forward_cached(GpuTensor.from_host(x[past:], (n, d), reg), k0, v0, past)[0].to_host()
        for i in range(n):
            assert np_ref.rel_rms(got[i], ref[past + i]) < 1e-3, (turn, n, i)


def test_layer_norm_of_parameters_just_computed(reg):
    """Scale and shift that the calls before it make: a LayerNorm that is given tensors must not read them ahead of its wait."""
    k, d = 16384, 256
    rng = np.random.default_rng(8)
    w = GpuTensor.from_host(np.ones((k, d), np.float32), (k, d), reg)
    x = rng.standard_normal((3, d)).astype(np.float32)
    xd = GpuTensor.from_host(x, (3, d), reg)
    plain = oracle.layer_norm(x, np.ones(d, np.float32), np.zeros(d, np.float32), 1e-5).reshape(3, d)
    rows = [GpuTensor.from_host(np.full((1, k), v, np.float32), (1, k), reg) for v in (2.0 ** -10, 2.0 ** -12, 2.0 ** -14)]
    for i in range(12):
        gamma, beta = ops.matmul(rows[i % 3], w, reg), ops.matmul(rows[(i + 1) % 3], w, reg)
        got = ops.layer_norm(xd, gamma, beta, 1e-5, reg).to_host()
        g, b = (16.0, 4.0, 1.0)[i % 3], (16.0, 4.0, 1.0)[(i + 1) % 3]
        assert np.abs(got - (plain * g + b)).max() < 1e-5 * 40, i


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("family", [vivezen, zufilorn])
def test_rows_after_rows_of_hybrid_models(reg, family, dtype):
    """The same of the hybrid decoders: steps of one to four requests' single tokens, with that family's tolerances."""
    reqs = {k: family.tokens("small", 40 + k, k) for k in range(4)}
    rb = b200nn.RequestBatch(family.model(reg, "small", dtype), 4, 64)
    got = {k: list(rb.step([(k, t[:10 + k], range(10 + k))])) for k, t in reqs.items()}
    for turn in range(24):
        live = [(turn + j) % 4 for j in range((1, 2, 3, 4, 4, 3, 4, 1)[turn % 8])]
        for k, row in zip(live, rb.step([(k, [reqs[k][len(got[k])]], [0]) for k in live])):
            got[k].append(row)
    for k, rows in got.items():
        ref = family.reference("small", reqs[k][:len(rows)])
        family.check(np.stack(rows), ref, family.TOL[dtype] if family is vivezen else dtype, f"request {k}")


@pytest.mark.parametrize("int4", [False, True])
def test_greedy_pick_of_a_vocabulary_between_tiles(reg, int4):
    """The pick of one row reads the entries of whole 32-feature groups only: a model of 256 tokens with large logits has left
    its entries in the buffers that a model of 130 then uses."""
    for vocab, scale in ((256, 50.0), (130, 1.0), (256, 50.0), (97, 1.0), (14300, 1.0)):
        cfg = Gpt2Config(n_layer=1, n_embd=64, n_head=1, vocab_size=vocab, n_positions=16)
        w = synth.gpt2_weights(cfg, base_seed=vocab, std=0.02)
        w["wte"] = w["wte"] * scale
        m = Int4Gpt2Model(w, cfg, reg, flags=b200nn.QUANT_LM_HEAD, group_size=64) if int4 else Gpt2Model.from_weights(w, cfg, reg)
        prompt = np.array([1, 2, 3], dtype=np.uint32)
        got = m.generate(prompt, 6, flags=0)
        reg.set_tuning("fused_argmax", 0)
        try:
            ref = m.generate(prompt, 6, flags=0)
        finally:
            reg.set_tuning("fused_argmax", 1)
        assert np.array_equal(got, ref) and got.max() < vocab
        del m


# one row, a stage's edge, a split's edge, the most splits, and the pairs around which the split count changes
@pytest.mark.parametrize("batch,heads,ctx,cap", [(1, 1, 1, 1), (1, 1, 64, 64), (1, 2, 65, 65), (1, 1, 129, 300), (1, 3, 1024, 1024),
                                                 (1, 1, 5000, 5000), (37, 3, 513, 520), (37, 12, 200, 256), (37, 13, 77, 128), (74, 12, 130, 130),
                                                 (75, 12, 131, 131),
                                                 # blocks of 16 warps, of 8 (by rows, by blocks), and of 4 again
                                                 (1, 1, 4089, 4100), (1, 1, 4088, 4088), (1, 2, 2041, 2041), (1, 2, 2040, 2050), (1, 18, 4100, 4100),
                                                 (1, 19, 4100, 4101), (1, 37, 2049, 2049), (1, 38, 2049, 2049)])
def test_decode_attention_splits(reg, batch, heads, ctx, cap):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(ctx * 100 + batch)
    q = torch.randn(batch, heads * 64, generator=g, device="cuda").half()
    k, v = (torch.randn(batch, heads, cap, 64, generator=g, device="cuda").half() for _ in range(2))
    k[:, :, ctx:], v[:, :, ctx:] = float("nan"), float("nan")  # rows past the context are not looked at
    out = torch.zeros_like(q)
    torch.cuda.synchronize()
    ops.decode_attention_f16(q.data_ptr(), k.data_ptr(), v.data_ptr(), batch, heads, cap, ctx, out.data_ptr(), reg)
    reg.synchronize()
    s = torch.einsum("bhd,bhnd->bhn", q.double().reshape(batch, heads, 64), k[:, :, :ctx].double()) / 8
    ref = torch.einsum("bhn,bhnd->bhd", torch.softmax(s, -1), v[:, :, :ctx].double()).reshape(batch, heads * 64)
    # the result is rounded to fp16: 2^-11 of a value, and f32 sums below that
    assert ((out.double() - ref).abs() <= 2.0 ** -10 * ref.abs() + 2e-5).all()
