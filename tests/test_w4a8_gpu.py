"""W4A8 on the GPU against the CPU oracle (the restatement of the reference's gemm_ref), bit for bit: Q4_K and Q6_K,
bf16 stores and fp32 residual adds, several row counts and live counts (padded buckets), a fused mixed-kind projection
(tests/test_w4a8.py:45-75).  Activations: N(0, 1) with k / 64 outlier channels x20 (tests/test_w4a8.py:26-30)."""
import numpy as np
import pytest
import torch

import oracle
from prism_b200 import quant, synth, w4a8
from util import bf16_from_bits, first_diff, n_rows, np_bits, same

pytestmark = pytest.mark.gpu


def weights(kind, n, k, seed):
    w = synth.weights(n, k, seed)
    return w4a8.repack(synth.q4_k(w) if kind == "q4k" else synth.q6_k(w)), w


def ref_gemm(xq, a, xs, w, epi, live, out=None):
    g = lambda t: None if t is None else t.numpy()          # noqa: E731
    return oracle.w4a8_gemm(xq, a, xs, w.kind, g(w.q), g(w.sc), g(w.mn), g(w.d), g(w.dm), epi=epi, live=live, out=out)


@pytest.mark.parametrize("kind", ["q4k", "q6k"])
@pytest.mark.parametrize("m,live,n,k", [(1, 1, 256, 512), (7, 7, 320, 2560), (64, 50, 1024, 5120), (300, 300, 192, 1024),
                                        (130, 127, 4100, 512), (17, 17, 1000, 1024), (48, 33, 132, 768),
                                        (16, 16, 5120, 5120), (2, 2, 1000, 1024), (4, 3, 4100, 2560), (3, 3, 132, 768),
                                        (4, 4, 100, 512), (1, 1, 5120, 5120), (8, 8, 1000, 1024), (6, 5, 320, 2560),
                                        (8, 8, 5120, 5120), (5, 5, 132, 768)])
def test_gemm_bits(dev, kind, m, live, n, k):
    w, wf = weights(kind, n, k, seed=n + k)
    x = synth.activations(m, k, seed=m, outliers=k // 64)
    xq, a, xs = oracle.quant_g(np_bits(x))
    ref0 = ref_gemm(xq, a, xs, w, 0, live)
    base = torch.randn(m, n, generator=torch.Generator().manual_seed(4))
    ref1 = ref_gemm(xq, a, xs, w, 1, live, out=base.numpy())
    wd = w.to(dev)
    nr = n_rows(live, dev)
    xqd, ad, xsd = (torch.from_numpy(t).to(dev) for t in (xq, a, xs))
    out = torch.zeros(m, n, dtype=torch.bfloat16, device=dev)
    w4a8.gemm(xqd, ad, xsd, wd, out, nr, epi=0)
    assert same(out, bf16_from_bits(ref0)), first_diff(np_bits(out), ref0)
    res = base.to(dev)
    w4a8.gemm(xqd, ad, xsd, wd, res, nr, epi=1)
    assert same(res, ref1), first_diff(res.cpu().numpy(), ref1)
    if m <= 16:
        # cfg is accepted for signature parity and changes nothing: K is split over a CTA's warps at most
        for cfg in (1, 2, 5):
            out = torch.zeros(m, n, dtype=torch.bfloat16, device=dev)
            w4a8.gemm(xqd, ad, xsd, wd, out, nr, epi=0, cfg=cfg)
            assert same(out, bf16_from_bits(ref0)), (cfg, first_diff(np_bits(out), ref0))
            res = base.to(dev)
            w4a8.gemm(xqd, ad, xsd, wd, res, nr, epi=1, cfg=cfg)
            assert same(res, ref1), (cfg, first_diff(res.cpu().numpy(), ref1))
    # the quantized product stays close to the unquantized one (tests/test_w4a8.py:73-75: a few per cent)
    kq = synth.q4_k(wf) if kind == "q4k" else synth.q6_k(wf)
    true = x[:live].float() @ kq.dequant().T
    got = oracle.bf16_to_f32(ref0)[:live]
    assert np.linalg.norm(got - true.numpy()) / np.linalg.norm(true.numpy()) < 0.05


def random_weights(kind, n, k, seed):
    """Random packed words and scales over their whole ranges (no encoder: large shapes are quick)."""
    g = torch.Generator().manual_seed(seed)
    u8 = lambda *s, hi: torch.randint(0, hi, s, generator=g, dtype=torch.uint8)          # noqa: E731
    f = lambda: torch.rand(k // 256, n, generator=g) * 1e-3                              # noqa: E731
    if kind == "q4k":
        return w4a8.W4(kind, u8(n, k // 2, hi=256), u8(k // 256, n, 8, hi=64), u8(k // 256, n, 8, hi=64), f(), f(), n, k), g
    return w4a8.W4(kind, torch.randint(-32, 32, (n, k), generator=g, dtype=torch.int8),
                   torch.randint(-128, 128, (k // 256, n, 16), generator=g, dtype=torch.int8), None, f(), None, n, k), g


@pytest.mark.parametrize("kind", ["q4k", "q6k"])
@pytest.mark.parametrize("m,live,n,k", [(3, 3, 20, 256), (9, 8, 36, 1280), (17, 17, 2500, 768), (31, 30, 68, 2304),
                                        (33, 33, 1024, 512), (64, 64, 2052, 512), (8, 8, 18948, 512), (16, 13, 18948, 512),
                                        (32, 32, 18948, 512)])
def test_gemm_bits_decode_tiles(dev, kind, m, live, n, k):
    """The decode kernels' edges: weight rows that end inside a tile of 16, 32 or 64, super-blocks that do not fill a round
    of the warps, row counts just above a block of 8, 16 or 32, and both sides of the rule on the weight rows."""
    w, g = random_weights(kind, n, k, n + k + m)
    xq, a, xs = oracle.quant_g(np_bits(synth.activations(m, k, seed=m, outliers=k // 64)))
    base = torch.randn(m, n, generator=g)
    ref0, ref1 = ref_gemm(xq, a, xs, w, 0, live), ref_gemm(xq, a, xs, w, 1, live, out=base.numpy().copy())
    xqd, ad, xsd = (torch.from_numpy(t).to(dev) for t in (xq, a, xs))
    out, res = torch.zeros(m, n, dtype=torch.bfloat16, device=dev), base.to(dev)
    w4a8.gemm(xqd, ad, xsd, w.to(dev), out, n_rows(live, dev))
    w4a8.gemm(xqd, ad, xsd, w.to(dev), res, n_rows(live, dev), epi=1)
    assert same(out, bf16_from_bits(ref0)), first_diff(np_bits(out), ref0)
    assert same(res, ref1), first_diff(res.cpu().numpy(), ref1)


@pytest.mark.parametrize("kind,m,live,n,k", [("q4k", 8, 8, 40, 6656), ("q4k", 8, 7, 14300, 2304), ("q4k", 16, 16, 36, 4608),
                                             ("q4k", 24, 23, 200, 4608), ("q4k", 13, 13, 14300, 1792), ("q4k", 30, 30, 7200, 2304),
                                             ("q4k", 5, 5, 7200, 2048), ("q4k", 12, 12, 9000, 1024), ("q6k", 8, 8, 100, 8704),
                                             ("q6k", 7, 7, 4100, 8704), ("q6k", 24, 24, 100, 6656), ("q6k", 8, 6, 4800, 4608),
                                             ("q6k", 16, 16, 2500, 4608), ("q6k", 32, 31, 2500, 2304), ("q6k", 64, 64, 1024, 6656)])
def test_gemm_bits_long_k(dev, kind, m, live, n, k):
    """A K that takes each decode tile more than twice around its ring of rounds and ends inside a round, either side of the
    lines in the weight rows; out a column slice at an odd offset.  First, last and 150 other weight rows, bit for bit."""
    w, g = random_weights(kind, n, k, n + k + m)
    at = torch.cat([torch.arange(min(n, 70)), torch.randint(0, n, (150,), generator=g), torch.arange(max(n - 70, 0), n)])
    pick = lambda t: None if t is None else t[:, at].contiguous()                        # noqa: E731
    part = w4a8.W4(kind, w.q[at].contiguous(), pick(w.sc), pick(w.mn), pick(w.d), pick(w.dm), len(at), k)
    xq, a, xs = oracle.quant_g(np_bits(synth.activations(m, k, seed=m, outliers=k // 64)))
    base = torch.randn(m, n + 6, generator=g)
    wd, nr = w.to(dev), n_rows(live, dev)
    xqd, ad, xsd = (torch.from_numpy(t).to(dev) for t in (xq, a, xs))
    out, res = torch.full((m, n + 6), 3.0, dtype=torch.bfloat16, device=dev), base.to(dev)
    w4a8.gemm(xqd, ad, xsd, wd, out[:, 3:3 + n], nr)
    w4a8.gemm(xqd, ad, xsd, wd, res[:, 1:1 + n], nr, epi=1)
    out, res = out.cpu(), res.cpu()
    ref0 = ref_gemm(xq, a, xs, part, 0, live)
    ref1 = ref_gemm(xq, a, xs, part, 1, live, out=base[:, 1 + at].numpy())
    assert np.array_equal(np_bits(out[:live, 3 + at]), ref0[:live]), first_diff(np_bits(out[:live, 3 + at]), ref0[:live])
    assert same(res[:, 1 + at], ref1), first_diff(res[:, 1 + at].numpy(), ref1)
    assert bool((out[live:] == 3).all()) and bool((out[:, :3] == 3).all()) and bool((out[:, 3 + n:] == 3).all())


@pytest.mark.parametrize("kind,m,live,n,k", [("q4k", 40, 33, 19000, 512), ("q4k", 200, 199, 5000, 768), ("q4k", 150, 129, 4996, 2304),
                                             ("q4k", 300, 300, 13000, 512), ("q6k", 200, 193, 4900, 1280), ("q6k", 300, 290, 9900, 512),
                                             ("q6k", 64, 49, 18940, 256)])
def test_gemm_bits_tensor_memory_operand(dev, kind, m, live, n, k):
    """Sizes that run with the expanded weights in tensor memory: one and two units of 64 rows a tile and part of one, a tile or more
    per SM, weight rows that end inside a tile, K below and above its three stages."""
    w, g = random_weights(kind, n, k, n + k + m)
    at = torch.cat([torch.arange(140), torch.randint(0, n, (200,), generator=g), torch.arange(n - 140, n)])
    pick = lambda t: None if t is None else t[:, at].contiguous()                        # noqa: E731
    part = w4a8.W4(kind, w.q[at].contiguous(), pick(w.sc), pick(w.mn), pick(w.d), pick(w.dm), len(at), k)
    xq, a, xs = oracle.quant_g(np_bits(synth.activations(m, k, seed=m, outliers=k // 64)))
    base = torch.randn(m, n + 6, generator=g)
    wd, nr = w.to(dev), n_rows(live, dev)
    xqd, ad, xsd = (torch.from_numpy(t).to(dev) for t in (xq, a, xs))
    out, res = torch.full((m, n + 6), 3.0, dtype=torch.bfloat16, device=dev), base.to(dev)
    w4a8.gemm(xqd, ad, xsd, wd, out[:, 3:3 + n], nr)
    w4a8.gemm(xqd, ad, xsd, wd, res[:, 1:1 + n], nr, epi=1)
    out, res = out.cpu(), res.cpu()
    ref0 = ref_gemm(xq, a, xs, part, 0, live)
    ref1 = ref_gemm(xq, a, xs, part, 1, live, out=base[:, 1 + at].numpy())
    assert np.array_equal(np_bits(out[:live, 3 + at]), ref0[:live]), first_diff(np_bits(out[:live, 3 + at]), ref0[:live])
    assert same(res[:, 1 + at], ref1), first_diff(res[:, 1 + at].numpy(), ref1)
    assert bool((out[live:] == 3).all()) and bool((out[:, :3] == 3).all()) and bool((out[:, 3 + n:] == 3).all())


@pytest.mark.parametrize("kind,n,k", [("q4k", 1000, 1024), ("q4k", 8200, 768), ("q6k", 1000, 1024), ("q6k", 5000, 768)])
def test_batch_invariance_across_kernels(dev, kind, n, k):
    """A row's bits do not depend on how many rows are multiplied with it, although 1, 2, 8, 9, 17, 33 and 100 rows run on
    different kernels and tiles."""
    w, _ = random_weights(kind, n, k, n + k)
    wd = w.to(dev)
    xq, a, xs = (torch.from_numpy(t).to(dev) for t in oracle.quant_g(np_bits(synth.activations(100, k, seed=k, outliers=4))))
    want = torch.empty(100, n, dtype=torch.bfloat16, device=dev)
    w4a8.gemm(xq, a, xs, wd, want, n_rows(100, dev))
    for m in (1, 2, 3, 8, 9, 16, 17, 32, 33, 64):
        got = torch.empty(m, n, dtype=torch.bfloat16, device=dev)
        w4a8.gemm(xq[:m], a[:, :m].contiguous(), xs[:, :m].contiguous(), wd, got, n_rows(m, dev))
        assert same(got, want[:m].contiguous()), m


def test_fused_mixed_projection(dev):
    """q | k as Q4_K and v as Q6_K in one output buffer (the Q4_K_M convention), through rows_g on the GPU."""
    k, m = 1024, 20
    wq = synth.weights(384, k, 1)
    wv = synth.weights(128, k, 2)
    kqs = [synth.q4_k(wq[:256]), synth.q4_k(wq[256:]), synth.q6_k(wv)]
    segs = w4a8.segments(kqs, dev)
    assert [(s[0].kind, s[0].n, s[1]) for s in segs] == [("q4k", 384, 0), ("q6k", 128, 384)]
    assert w4a8.seg_width(segs) == 512
    x = synth.activations(m, k, seed=9, outliers=16)
    nr = n_rows(m, dev)
    q = torch.empty(m, k, dtype=torch.int8, device=dev)
    a = torch.empty(k // 256, m, device=dev)
    xs = torch.empty(k // 256, m, 16, dtype=torch.int8, device=dev)
    quant.rows_g(x.to(dev), q, a, xs, nr, m)
    out = torch.zeros(m, 512, dtype=torch.bfloat16, device=dev)
    w4a8.gemm_segs(q, a, xs, segs, out, nr)
    rq, ra, rxs = oracle.quant_g(np_bits(x))
    for (w, off) in segs:
        ref = ref_gemm(rq, ra, rxs, w.to("cpu"), 0, m)
        assert same(out[:, off:off + w.n].contiguous(), bf16_from_bits(ref)), w.kind
    sub = w4a8.seg_rows(segs, 300, 450)
    assert [(s[0].kind, s[0].n, s[1]) for s in sub] == [("q4k", 84, 0), ("q6k", 66, 84)]
