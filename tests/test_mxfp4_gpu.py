"""MXFP4 on the GPU: the activation quantizer against the CPU oracle bit for bit (and the reference's golden vectors),
the GEMM against the dequantized product within 1e-3 relative Frobenius error (the reference's own test allows 2e-3,
tests/test_mxfp4.py:54-85), both epilogues, batch invariance (tests/test_mxfp4.py:88-102)."""
import os

import numpy as np
import pytest
import torch

import oracle
from prism_b200 import mxfp4, synth
from util import np_bits, same

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")


def quant_gpu(x, dev, inv=None):
    n, k = x.shape
    q = torch.zeros(n, k // 2, dtype=torch.uint8, device=dev)
    s = torch.zeros(n, k // 32, dtype=torch.uint8, device=dev)
    if inv is None:
        mxfp4.quantize_act(x.to(dev), q, s)
    else:
        mxfp4.quantize_act_scaled(x.to(dev), inv.to(dev), q, s)
    return q, s


def test_quantize_act_golden(dev):
    g = np.load(os.path.join(G, "mxfp4.npz"))
    xb = torch.from_numpy(g["act_bf16"].view(np.int16)).view(torch.bfloat16)
    q, s = quant_gpu(xb, dev)
    assert same(q, g["act_q_bf16"]) and same(s, g["act_s_bf16"])
    q, s = quant_gpu(torch.from_numpy(g["act_f32"]), dev)
    assert same(q, g["act_q_f32"]) and same(s, g["act_s_f32"])
    q, s = quant_gpu(xb, dev, torch.from_numpy(g["act_inv"]))
    assert same(q, g["act_q_scaled"]) and same(s, g["act_s_scaled"])


@pytest.mark.parametrize("n,k", [(7, 256), (33, 512), (128, 4096), (16, 5120), (3, 17408)])
def test_quantize_act_oracle(dev, n, k):
    x = synth.activations(n, k, seed=n + k)
    rq, rs = oracle.mxfp4_quant(np_bits(x))
    q, s = quant_gpu(x, dev)
    assert same(q, rq) and same(s, rs)
    dq = mxfp4.dequant_packed(q.cpu(), s.cpu())
    rel = (dq - x.float()).norm() / x.float().norm()
    assert rel < 0.2                                      # tests/test_mxfp4.py:41-51


def quant_by_thresholds(x, inv):
    """The quantizer's definition in numpy: a block's exponent from its largest magnitude (a NaN does not count), magnitude codes by
    strict thresholds, the sign bit where v < 0."""
    v = x * inv if inv is not None else x
    b = v.reshape(x.shape[0], -1, 32)
    amax = np.maximum(np.where(np.isnan(b), 0, np.abs(b)).max(2), np.float32(1e-30)).astype(np.float32)
    bits = amax.view(np.uint32)
    e = np.clip((bits >> 23).astype(np.int32) - np.where((bits & 0x7fffff) <= 0x400000, 129, 128), -127, 127)
    with np.errstate(all="ignore"):
        a = np.abs(b) * np.ldexp(np.float32(1), -e).astype(np.float32)[..., None]
        c = sum((a > t).astype(np.uint8) for t in (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0)) | np.where(b < 0, 8, 0).astype(np.uint8)
    c = c.reshape(x.shape)
    return c[:, ::2] | (c[:, 1::2] << 4), (e + 127).astype(np.uint8)


@pytest.mark.parametrize("n", [3, 601])                   # one vector a thread, four vectors a thread
@pytest.mark.parametrize("kind", ["bf16", "f32", "scaled"])
def test_quantize_act_edges(dev, n, kind):
    """Halfway values and their neighbours on both sides, both zeros, values far below the block's largest, infinities and
    NaN, in every block position."""
    k = 8192
    g = np.random.default_rng(n)
    half = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0, 0.5, 1.0, 3.0, 0.0, -0.0, 1e-38, 2.0 ** -140], np.float32)
    near = np.concatenate([half, np.nextafter(half, np.float32(9)), np.nextafter(half, np.float32(-9))])
    near = np.concatenate([near, half * np.float32(1 + 2.0 ** -7), half * np.float32(1 - 2.0 ** -8)])
    v = g.choice(np.concatenate([near, -near]).astype(np.float32), (n, k // 32, 32))
    v[:, :, 0] = 6.0                                      # the block's scale is 2^e
    v = v * np.ldexp(np.float32(1), g.integers(-40, 40, (n, k // 32, 1))).astype(np.float32)
    v[g.random(v.shape) < 2e-4] = np.nan
    v[g.random(v.shape) < 1e-4] = np.inf
    v[g.random(v.shape) < 1e-4] = -np.inf
    v = torch.from_numpy(g.permuted(v, axis=2).reshape(n, k))
    inv = torch.from_numpy(g.choice(np.array([1, 0.5, 1.1, 3], np.float32), k)) if kind == "scaled" else None
    x = v if kind == "f32" else v.bfloat16()
    q, s = quant_gpu(x, dev, inv)
    rq, rs = quant_by_thresholds(x.float().numpy(), None if inv is None else inv.numpy())
    assert same(s, rs) and same(q, rq)


def rel_fro(got, ref):
    return float(np.linalg.norm(got.astype(np.float64) - ref) / np.linalg.norm(ref))


def bf16_within_one_step(out, ref64):
    """A bf16 output against the float64 product rounded to bf16 (round to nearest even): equal, or its neighbour (fp32
    accumulation in another order can move a value across a rounding boundary).  The output's own rounding alone is
    1.1e-3 relative Frobenius error, so the bound on the bf16 path is this one, not a Frobenius figure."""
    want = torch.from_numpy(np.ascontiguousarray(ref64)).to(torch.bfloat16)
    got = out.detach().cpu()
    gi, wi = got.view(torch.int16).int(), want.view(torch.int16).int()
    tiny = (got.float().abs() < 1e-30) & (want.float().abs() < 1e-30)
    return bool((((gi - wi).abs() <= 1) | tiny).all())


@pytest.mark.parametrize("M,N,K", [(32, 512, 256), (257, 1024, 512), (16, 5120, 5120), (300, 1000, 2560),
                                   (1024, 4096, 4096), (1024, 4808, 512), (1000, 4664, 768), (2048, 5120, 1024)])
def test_gemm(dev, M, N, K):
    w = mxfp4.pack(synth.weights(N, K, seed=N + K))
    x = synth.activations(M, K, seed=M)
    q, s = quant_gpu(x, dev)
    wd = mxfp4.prepare(mxfp4.MX4(w.q.to(dev), w.s.to(dev), N, K))
    _, ref = oracle.mxfp4_gemm(q.cpu().numpy(), s.cpu().numpy(), w.q.numpy(), w.s.numpy())
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q, s, wd, out, M, epi=0)
    err0 = rel_fro(out.float().cpu().numpy(), ref)
    assert err0 < 2e-3, err0                              # the reference's own bound; the output's bf16 rounding dominates
    assert bf16_within_one_step(out, ref)                 # ... and every value is the rounded exact product or its neighbour
    h0 = torch.randn(M, N, generator=torch.Generator().manual_seed(1))
    h = h0.to(dev)
    mxfp4.gemm(q, s, wd, h, M, epi=1)
    err1 = rel_fro(h.cpu().numpy() - h0.numpy(), ref)
    assert err1 < 1e-3, err1                              # the fp32 accumulators against the float64 product


@pytest.mark.parametrize("M,N,K", [(16, 5120, 5120), (1, 1000, 2560), (64, 384, 4352), (100, 256, 1024)])
def test_gemm_k_split(dev, M, N, K):
    """K slices per tile, added in slice order by the tile's last CTA: the same tolerances as the unsplit product, the
    same bits on every run (a poisoned workspace in between), counters left zeroed."""
    from prism_b200 import w8a8
    w = mxfp4.pack(synth.weights(N, K, seed=N + K))
    q, s = quant_gpu(synth.activations(M, K, seed=M), dev)
    wd = mxfp4.prepare(mxfp4.MX4(w.q.to(dev), w.s.to(dev), N, K))
    _, ref = oracle.mxfp4_gemm(q.cpu().numpy(), s.cpu().numpy(), w.q.numpy(), w.s.numpy())
    ws, counters = w8a8._workspace(dev)
    for split in (2, 3, 5, "auto"):
        h0 = torch.randn(M, N, generator=torch.Generator().manual_seed(1))
        runs = []
        for rep in range(2):
            ws.fill_(0x7f)
            h = h0.to(dev)
            mxfp4.gemm(q, s, wd, h, M, epi=1, split=split)
            runs.append(h)
        assert same(runs[0], runs[1]), split
        assert rel_fro(runs[0].cpu().numpy() - h0.numpy(), ref) < 1e-5, split
        out = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
        mxfp4.gemm(q, s, wd, out, M, epi=0, split=split)
        assert rel_fro(out.float().cpu().numpy(), ref) < 2e-3, split
        assert int(counters.abs().sum()) == 0


@pytest.mark.parametrize("M,N,K", [(1, 5120, 5120), (2, 1000, 2560), (1, 133, 256), (2, 34816, 512), (4, 7168, 1024),
                                   (3, 300, 768)])
def test_gemv_rows(dev, M, N, K):
    """One to four rows on the CUDA-core kernel (exact integer block products, fp32 over the blocks) against the
    float64 product, both epilogues; deterministic; rows past M and columns past N untouched."""
    w = mxfp4.pack(synth.weights(N, K, seed=N + K))
    q, s = quant_gpu(synth.activations(M, K, seed=M + 7, outliers=K // 64), dev)
    wd = mxfp4.prepare(mxfp4.MX4(w.q.to(dev), w.s.to(dev), N, K))
    _, ref = oracle.mxfp4_gemm(q.cpu().numpy(), s.cpu().numpy(), w.q.numpy(), w.s.numpy())
    h0 = torch.randn(M + 1, N + 3, generator=torch.Generator().manual_seed(1))
    runs = []
    for rep in range(2):
        h = h0.to(dev)
        mxfp4.gemv(q, s, wd, h[:M, :N], M, epi=1)
        runs.append(h)
    assert same(runs[0], runs[1])
    got = runs[0].cpu().numpy()
    assert rel_fro(got[:M, :N] - h0.numpy()[:M, :N], ref) < 1e-5
    assert np.array_equal(got[M:], h0.numpy()[M:]) and np.array_equal(got[:, N:], h0.numpy()[:, N:])
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemv(q, s, wd, out, M, epi=0)
    assert rel_fro(out.float().cpu().numpy(), ref) < 2e-3 and bf16_within_one_step(out, ref)
    if M == 1:                                            # split="auto" routes one row against few weight rows here
        auto = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
        mxfp4.gemm(q, s, wd, auto, M, epi=0, split="auto")
        assert rel_fro(auto.float().cpu().numpy(), ref) < 2e-3
    # and close to the tensor-core kernel's bits: the same exact block products, another order of fp32 additions
    out_tc = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q, s, wd, out_tc, M, epi=0)
    assert rel_fro(out.float().cpu().numpy(), out_tc.float().cpu().numpy().astype(np.float64)) < 2e-3


def test_gemm_fp32_path_tight(dev):
    """Against the float64 product the fp32-accumulated result is within 1e-5 (no operand rounding happens inside the
    MMA: e2m1 products and power-of-two scales are exact; only the fp32 sums round)."""
    M, N, K = 64, 256, 1024
    w = mxfp4.pack(synth.weights(N, K, seed=3))
    q, s = quant_gpu(synth.activations(M, K, seed=4), dev)
    wd = mxfp4.prepare(mxfp4.MX4(w.q.to(dev), w.s.to(dev), N, K))
    _, ref = oracle.mxfp4_gemm(q.cpu().numpy(), s.cpu().numpy(), w.q.numpy(), w.s.numpy())
    h = torch.zeros(M, N, device=dev)
    mxfp4.gemm(q, s, wd, h, M, epi=1)
    assert rel_fro(h.cpu().numpy(), ref) < 1e-5


def test_batch_invariance(dev):
    M, N, K = 64, 1024, 512
    w = mxfp4.pack(synth.weights(N, K, seed=5))
    wd = mxfp4.prepare(mxfp4.MX4(w.q.to(dev), w.s.to(dev), N, K))
    q, s = quant_gpu(synth.activations(M, K, seed=6), dev)
    out64 = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q, s, wd, out64, M)
    out32 = torch.zeros(32, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q[:32].contiguous(), s[:32].contiguous(), wd, out32, 32)
    assert same(out64[:32].contiguous(), out32)
    big = torch.zeros(300, N, dtype=torch.bfloat16, device=dev)
    q3 = torch.cat([q] * 5)[:300].contiguous()
    s3 = torch.cat([s] * 5)[:300].contiguous()
    mxfp4.gemm(q3, s3, wd, big, 300)
    assert same(big[:64].contiguous(), out64) and same(big[256:300].contiguous(), out64[:44].contiguous())


def test_wide_tiles_same_bits(dev):
    """Enough tiles for the 128 x 256 kernel (at least one per SM): every row's bits equal the 128 x 128 kernel's (which
    runs when the same rows come in a small batch) - one accumulator over all of K either way."""
    M, N, K = 2048, 5120, 1024
    w = mxfp4.pack(synth.weights(N, K, seed=3))
    wd = mxfp4.prepare(mxfp4.MX4(w.q.to(dev), w.s.to(dev), N, K))
    q, s = quant_gpu(synth.activations(M, K, seed=4), dev)
    big = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q, s, wd, big, M)
    for r0 in (0, 900, 1984):
        small = torch.zeros(64, N, dtype=torch.bfloat16, device=dev)
        mxfp4.gemm(q[r0:r0 + 64].contiguous(), s[r0:r0 + 64].contiguous(), wd, small, 64)
        assert same(big[r0:r0 + 64].contiguous(), small)


@pytest.mark.parametrize("M,N,K", [(1, 40, 256), (15, 1000, 2304), (16, 132, 8704), (17, 9500, 512), (33, 4800, 1280), (48, 20000, 768),
                                   (63, 2500, 4352), (64, 19072, 256)])
def test_few_rows(dev, M, N, K):
    """The decode kernel: row counts around its steps of 16, weight tiles whole, halved and quartered over CTAs and ending inside a
    part, K shorter and longer than its stages, out a column slice.  The bits of the many-rows kernel."""
    g = torch.Generator().manual_seed(M + N)
    w = mxfp4.MX4(torch.randint(0, 256, (N, K // 2), generator=g, dtype=torch.uint8).to(dev),
                  torch.randint(110, 124, (N, K // 32), generator=g, dtype=torch.uint8).to(dev), N, K)
    wd = mxfp4.prepare(w)
    q, s = quant_gpu(synth.activations(M + 65, K, seed=M + 7), dev)
    want = torch.zeros(M + 65, N, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q, s, wd, want, M + 65)
    h0 = torch.randn(M + 2, N + 4, generator=g).to(dev)
    h, ref = h0.clone(), torch.zeros(M + 65, N, device=dev)
    ref[:M] = h0[:M, 1:1 + N]
    mxfp4.gemm(q, s, wd, ref, M + 65, epi=1)
    out = torch.full((M + 2, N + 4), 3.0, dtype=torch.bfloat16, device=dev)
    mxfp4.gemm(q[:M], s[:M], wd, out[:M, 3:3 + N], M)
    mxfp4.gemm(q[:M], s[:M], wd, h[:M, 1:1 + N], M, epi=1)
    assert same(out[:M, 3:3 + N].contiguous(), want[:M].contiguous())
    assert same(h[:M, 1:1 + N].contiguous(), ref[:M].contiguous())
    assert bool((out[M:] == 3).all()) and bool((out[:, :3] == 3).all()) and bool((out[:, 3 + N:] == 3).all())
    assert same(h[M:], h0[M:]) and same(h[:, :1], h0[:, :1]) and same(h[:, 1 + N:], h0[:, 1 + N:])
