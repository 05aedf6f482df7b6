"""Host-side logic on the CPU: weight containers and encoders against gguf-py and the golden vectors, weight
preparation, sharding indices, the C-ABI library's exported symbols (no kernel is launched)."""
import ctypes
import os
import re
import types

import numpy as np
import pytest
import torch

from prism_b200 import _lib, gguf_weights as GW, synth, tp, w8a8

G = os.path.join(os.path.dirname(__file__), "golden")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def load(name):
    return np.load(os.path.join(G, name))


def test_library_exports_every_declared_symbol(lib):
    header = open(os.path.join(ROOT, "include", "prism_b200.h")).read()
    declared = set(re.findall(r"\b(pb_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in include/prism_b200.h but not exported"
    assert declared == set(_lib.declared_symbols())
    assert lib.pb_version() >= 1
    assert b"ok" == lib.pb_status_string(0)


def test_operators_refuse_cpu_tensors(lib):
    a = torch.zeros(4, 64, dtype=torch.int8)
    with pytest.raises(RuntimeError, match="no CPU path"):
        w8a8.gemm(a, torch.ones(4), a, torch.ones(4), torch.zeros(4, 4, dtype=torch.bfloat16),
                  torch.tensor([4], dtype=torch.int32), 64)


def test_pdl_switch_belongs_to_its_thread(lib):
    """Two threads that each save, set and put back the switch around a pass, one inside the other's: neither sees the
    other's setting, and nothing stays on."""
    import threading
    seen = []
    assert lib.pb_set_pdl(1) == 0
    try:
        t = threading.Thread(target=lambda: seen.extend([lib.pb_set_pdl(1), lib.pb_set_pdl(0), lib.pb_set_pdl(0)]))
        t.start()
        t.join()
        assert seen == [0, 1, 0]
    finally:
        assert lib.pb_set_pdl(0) == 1
    assert lib.pb_set_pdl(0) == 0


def test_one_row_chain_takes_its_own_table_entry(monkeypatch, tmp_path):
    """A chained one-row product uses the entry that was measured for it, the next larger row count when there is none, and
    never the CUDA-core kernel's; nothing else sees the chained entry."""
    import json

    from prism_b200 import tune
    e = {m: {"split": i + 1, "defer": False, "us": 1.0} for i, m in enumerate(("1", "8", "64", "1p"))}
    path = tmp_path / "table.json"
    path.write_text(json.dumps({"table": {"256x512": e, "256x1024": {m: e[m] for m in ("1", "8", "64")}}}))
    monkeypatch.setattr(w8a8, "_TABLE", tune.load_table(str(path)))
    split = lambda M, K, chained: w8a8._choice(M, 256, K, False, chained)["split"]          # noqa: E731
    assert (split(1, 512, False), split(1, 512, True), split(1, 1024, True)) == (1, 4, 2)
    assert (split(2, 512, False), split(2, 512, True), split(60, 512, True)) == (2, 2, 3)


class _Recorder:
    """The library with every launch replaced by a note of its arguments."""

    def __init__(self, real):
        self.real, self.gemms = real, []

    def __getattr__(self, name):
        if name.endswith(("_bytes", "_counters")) or name == "pb_set_pdl":
            return getattr(self.real, name)

        def launch(*args):
            if name == "pb_w8a8_gemm":
                self.gemms.append(args)
            return 0
        return launch


class _Weights:
    """A weight matrix's shape: no memory is touched."""

    def __init__(self, n, k):
        self.shape, self.dtype = (n, k), torch.int8

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 4096


def test_one_row_chain_needs_weights_to_hide(lib):
    """One row: a chain of dependent launches where a layer's weights are worth prefetching, plain launches (the CUDA-core
    GEMM) below that; more rows: always a chain."""
    from prism_b200 import linear_stack as LS

    def chained(M, hid, kv, ffn):
        shapes = {"qkv": (hid + 2 * kv, hid), "o": (hid, hid), "gate_up": (2 * ffn, hid), "down": (hid, ffn)}
        layer = {name: (_Weights(n, k), torch.ones(n)) for name, (n, k) in shapes.items()}
        return LS.LinearStack([layer], M, torch.device("cpu"), None, hid, hid, kv, ffn).pdl
    assert chained(1, 5120, 1024, 17408) and chained(1, 1792, 256, 4864)
    assert not chained(1, 1024, 256, 2816) and not chained(1, 1536, 256, 4096)
    assert chained(2, 1024, 256, 2816) and chained(64, 512, 128, 1408) and not chained(65, 5120, 1024, 17408)


@pytest.mark.parametrize("M", [1, 2, 16, 64])
def test_few_row_stacks_share_no_workspace(lib, monkeypatch, M):
    """Two stacks of the 27B shapes may have their passes in flight on two streams: a product that splits K inside the
    kernel must be given partial sums and counters that belong to its own stack, with room for it."""
    from prism_b200 import linear_stack as LS
    rec = _Recorder(lib)
    monkeypatch.setattr(_lib, "lib", lambda: rec)
    monkeypatch.setattr(_lib, "need_cuda", lambda *t: None)
    monkeypatch.setattr(_lib, "stream", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(w8a8, "_WORKSPACE", {})

    shapes = {"qkv": (7168, 5120), "o": (5120, 5120), "gate_up": (34816, 5120), "down": (5120, 17408)}
    layers = [{name: (_Weights(n, k), torch.ones(n)) for name, (n, k) in shapes.items()}]
    used = []
    for _ in range(2):
        stack = LS.LinearStack(layers, M, torch.device("cpu"))
        rec.gemms.clear()
        stack(torch.zeros(M, 5120))
        assert len(rec.gemms) == 4
        ws = [(g[14], g[16]) for g in rec.gemms if g[14] is not None]
        for g in rec.gemms:
            m, n, epi, split = g[7], g[8], g[11], g[12]
            if split > 1 and epi != w8a8.EPI_I32:
                assert g[15] >= lib.pb_w8a8_workspace_bytes(m, n, split) and g[17] >= lib.pb_w8a8_counters(m, n)
        used.append((stack, ws))
    assert used[0][1], "q|k|v splits K inside the kernel at every few-row count"
    assert not set(used[0][1]) & set(used[1][1]) and not w8a8._WORKSPACE
    # what a kernel that gave up leaves behind is cleared there as well
    scratch = used[0][0].scratch
    scratch.counters.fill_(1)
    w8a8.reset_workspace()
    assert not scratch.counters.any()


def test_argument_checks_without_gpu(lib):
    """Bad arguments are refused before any CUDA call."""
    assert lib.pb_w8a8_gemm(None, None, None, None, None, 0, None, 1, 1, 16, 16, 0, 1, 0, None, 0, None, 0, 0, None) == 1
    buf = (ctypes.c_char * 4096)()
    p = ctypes.addressof(buf)
    p16 = (p + 15) & ~15
    assert lib.pb_w8a8_gemm(p16, p16, p16, p16, p16, 8, p16, 4, 8, 24, 24, 0, 1, 0, None, 0, None, 0, 0, None) == 2  # K % 16
    assert lib.pb_w8a8_gemm(p16 + 1, p16, p16, p16, p16, 8, p16, 4, 8, 32, 32, 0, 1, 0, None, 0, None, 0, 0, None) == 1
    assert lib.pb_quant_rows(p16, 0, 32, None, p16, p16, p16, 4, 64, 64, 1, None, None) == 1   # mode 1 without amax
    assert lib.pb_w8a8_workspace_bytes(16, 5120, 4) == 4 * 40 * 16 * 128 * 4
    assert lib.pb_w8a8_counters(64, 7168) == 56
    # row blocks of the scattered int32 output: whole tiles, at most eight, covering every row
    blocks = (ctypes.c_void_p * 8)(*([p16] * 8))
    assert lib.pb_w8a8_gemm_scatter(p16, p16, blocks, 2, 100, 64, p16, 200, 64, 128, None) == 2      # block rows % 128
    assert lib.pb_w8a8_gemm_scatter(p16, p16, blocks, 9, 128, 64, p16, 256, 64, 128, None) == 1      # more than 8 blocks
    assert lib.pb_w8a8_gemm_scatter(p16, p16, blocks, 2, 128, 64, p16, 512, 64, 128, None) == 1      # rows not covered
    assert lib.pb_w8a8_gemm_scatter(p16, p16, blocks, 1, 128, 64, p16, 64, 64, 128, None) == 2       # few rows
    # MXFP4: split needs its workspace; the CUDA-core kernel takes up to four rows
    assert lib.pb_mxfp4_gemm_split(p16, p16, p16, p16, p16, 128, 16, 128, 2048, 0, 2, None, 0, None, 0, None) == 1
    assert lib.pb_mxfp4_workspace_bytes(16, 5120, 3) == 40 * 3 * 128 * 128 * 4 and lib.pb_mxfp4_counters(16, 5120) == 40
    assert lib.pb_mxfp4_gemv(p16, p16, p16, p16, p16, 128, 5, 128, 256, 0, None) == 2
    assert lib.pb_mxfp4_gemv(p16, p16, p16, p16, p16, 128, 1, 128, 128, 0, None) == 2                # K % 256


def _run_row_ring(where, groups, stages, rows, rng):
    """The row quantizers' loop over a CTA's rows with copies that land in any order and groups that run at any speed: `where(row)` is
    (slot, barrier, parity).  Returns what went wrong, or None.  A wait is true when the barrier's phase has the other parity."""
    slots, phase, armed, flying = [None] * stages, {}, set(), []
    at, waiting = list(range(groups)), [True] * groups

    def issue(i):
        slot, bar, _ = where(i)
        if bar in armed:
            return f"row {i} arms a barrier whose copy is still in flight"
        armed.add(bar)
        slots[slot] = ("copy in flight", i)
        flying.append(i)

    for i in range(min(stages, rows)):
        issue(i)
    for _ in range(100 * rows):
        g = rng.randrange(groups + 1)
        if g == groups:                                   # a copy lands
            if flying:
                i = flying.pop(rng.randrange(len(flying)))
                slot, bar, _ = where(i)
                slots[slot] = ("row", i)
                armed.discard(bar)
                phase[bar] = phase.get(bar, 0) + 1
        elif at[g] < rows:
            slot, bar, parity = where(at[g])
            if waiting[g]:
                if phase.get(bar, 0) & 1 != parity:
                    waiting[g] = False                    # it reads from here on
                    if slots[slot] != ("row", at[g]):
                        return f"row {at[g]} read while its slot holds {slots[slot]}"
            else:
                wrong = issue(at[g] + stages) if at[g] + stages < rows else None
                if wrong:
                    return wrong
                at[g] += groups
                waiting[g] = True
    return None if min(at) >= rows else f"stuck at {at}"


@pytest.mark.parametrize("groups,stages", [(1, 2), (1, 3), (1, 8), (2, 2), (2, 3), (2, 4)])
def test_row_ring_waits_for_its_own_copy(lib, groups, stages):
    """Whatever order the copies land in, a row is read after its own copy, and no barrier is armed twice.  One barrier per
    slot does not give that when the slots are not a multiple of the groups, which the model has to see."""
    import random

    def where(i):
        out = [ctypes.c_int() for _ in range(3)]
        assert lib.pb_test_row_ring(groups, stages, i, *(ctypes.addressof(x) for x in out)) == 0
        return tuple(x.value for x in out)

    per_slot = lambda i: (i % stages, i % stages, (i // stages) & 1)                         # noqa: E731
    rows = [where(i) for i in range(64)]
    assert all(0 <= s < stages and 0 <= b < 8 for s, b, _ in rows)
    for seed in range(300):
        assert _run_row_ring(rows.__getitem__, groups, stages, 40 + seed % 20, random.Random(seed)) is None
    seen = any(_run_row_ring(per_slot, groups, stages, 60, random.Random(seed)) for seed in range(300))
    assert seen == (stages % groups != 0)
    n = ctypes.addressof(ctypes.c_int())
    assert lib.pb_test_row_ring(2, 5, 0, n, n, n) == 1 and lib.pb_test_row_ring(1, 9, 0, n, n, n) == 1


def test_pair_tiles_are_shapes_of_the_mma(lib):
    """Row tiles of the CTA-pair kernel are N of an int8 MMA of two CTAs, which exists in steps of 32 up to 256 (0: the tile kernel
    runs)."""
    for n, k in ((7168, 5120), (5120, 17408), (34816, 5120), (512, 2048), (40, 144), (100000, 4096)):
        for m in [*range(65, 1200), 2047, 2048, 4097, 8191, 8192, 16400, 100000]:
            for epi in (0, 1):
                nt = lib.pb_w8a8_pair_rows(m, n, k, epi)
                assert nt % 32 == 0 and 0 <= nt <= 256, (m, n, k, nt)
    assert lib.pb_w8a8_pair_rows(333, 34816, 5120, 0) == 192 and lib.pb_w8a8_pair_rows(8192, 34816, 5120, 0) == 256
    # few weight rows: tiles small enough that the pairs fill the GPU (22 of 74 with 192 rows a tile)
    assert lib.pb_w8a8_pair_rows(2048, 512, 5120, 0) == 64
    # one wave of the tile kernel, whose copy engine makes the residual add
    assert lib.pb_w8a8_pair_rows(333, 5120, 17408, 1) == 0 and lib.pb_w8a8_pair_rows(333, 5120, 5120, 1) == 0
    assert lib.pb_w8a8_pair_rows(64, 5120, 5120, 0) == 0 and lib.pb_w8a8_pair_rows(333, 5120, 5120, 3) == 0


def test_split_rules_of_the_other_formats():
    from prism_b200 import mxfp4, w4a8
    # few-rows W4A8: time goes as waves / slices; Q6_K's 80 tiles of the down projection take 7 slices (4 waves)
    assert w4a8.pick_split(8, 5120, 5120, 128) == 3 and w4a8.pick_split(8, 34816, 5120, 128) == 1
    assert w4a8.pick_split(8, 5120, 17408, 64) == 7 and w4a8.pick_split(17, 5120, 17408, 64) == 1
    # MXFP4: only where one row tile's tiles leave most SMs idle
    assert mxfp4.pick_split(16, 5120, 5120) == 3 and mxfp4.pick_split(16, 34816, 5120) == 1
    assert mxfp4.pick_split(300, 5120, 5120) == 1 and mxfp4.pick_split(1, 5120, 512) == 1


def test_split_rule():
    assert w8a8.effective_split(256, 4) == 2 and w8a8.effective_split(5120, 7) == 7
    assert w8a8.effective_split(17408, 8) == 8 and w8a8.effective_split(640, 4) == 3   # 5 blocks: 2 + 2 + 1
    assert w8a8.pick_split(16, 5120, 5120) == 7 and w8a8.pick_split(16, 34816, 5120) == 1
    assert w8a8.pick_split(8192, 5120, 5120) == 1


def test_q8_and_weight_from_q8_match_reference():
    g = load("w8a8.npz")
    q8 = GW.Q8(torch.from_numpy(g["qs"]), torch.from_numpy(g["d"]))
    assert np.array_equal(q8.dequant().numpy(), g["dequant"])
    sm = torch.from_numpy(g["smooth"])
    for gk, s, tag in ((32, None, "gk32"), (64, None, "gk64"), (256, None, "gk256"), (256, sm, "gk256s"),
                       (32, sm, "gk32s")):
        q, sc = w8a8.weight_from_q8(q8, gk, s)
        assert np.array_equal(q.numpy(), g[f"q_{tag}"]) and np.array_equal(sc.numpy(), g[f"s_{tag}"]), tag
    gu = w8a8.interleave_gate_up(torch.from_numpy(g["gate"]), torch.from_numpy(g["up"]), 16)
    assert np.array_equal(gu.numpy(), g["gu16"])


def test_kquant_dequant_matches_reference_and_gguf_py():
    g = load("kquant.npz")
    from gguf.constants import GGMLQuantizationType as T
    from gguf.quants import dequantize
    for tag, typ, gt in (("4", GW.GGML_Q4_K, T.Q4_K), ("6", GW.GGML_Q6_K, T.Q6_K)):
        kq = GW.KQuant(torch.from_numpy(g[f"raw{tag}"]), typ, 512)
        got = kq.dequant().numpy()
        assert np.array_equal(got, g[f"deq{tag}"])
        assert np.array_equal(got, dequantize(g[f"raw{tag}"].reshape(24, -1), gt).reshape(24, 512))
        q8 = kq.as_q8()
        assert np.array_equal(q8.qs.numpy(), g[f"q8_{tag}_qs"]) and np.array_equal(q8.d.numpy(), g[f"q8_{tag}_d"])
    sc, mn = GW.scale_min_k4(torch.from_numpy(g["raw4"]).reshape(-1, 144)[:, 4:16])
    assert np.array_equal(sc.numpy(), g["sc"].astype(np.int32)) and np.array_equal(mn.numpy(), g["mn"].astype(np.int32))


def test_encoders_are_valid_blocks():
    """Seeded inputs: Q8_0 byte-for-byte as gguf-py quantizes; Q4_K / Q6_K blocks dequantize identically under gguf-py
    and stay close to the source weights; Q5_K dequantizes as gguf-py on random bytes."""
    from gguf.constants import GGMLQuantizationType as T
    from gguf.quants import dequantize, quantize
    w = synth.weights(32, 1024, 5)
    q8 = synth.q8_0(w)
    ref = quantize(w.numpy(), T.Q8_0).reshape(32, 32, 34)
    assert np.array_equal(ref[..., 2:].copy().view(np.int8).reshape(32, 1024), q8.qs.numpy())
    assert np.array_equal(ref[..., :2].copy().view(np.float16).reshape(32, 32), q8.d.numpy())
    assert np.array_equal(GW.Q8.from_blocks(torch.from_numpy(ref.reshape(-1)), 32, 1024).qs.numpy(), q8.qs.numpy())
    for enc, gt, tol in ((synth.q4_k, T.Q4_K, 0.12), (synth.q6_k, T.Q6_K, 0.04)):
        kq = enc(w)
        d = kq.dequant().numpy()
        assert np.array_equal(d, dequantize(kq.raw.numpy().reshape(32, -1), gt).reshape(32, 1024))
        assert np.linalg.norm(d - w.numpy()) / np.linalg.norm(w.numpy()) < tol
    raw = torch.randint(0, 256, (8, 2, 176), dtype=torch.uint8, generator=torch.Generator().manual_seed(0))
    raw[..., 1] = 0x2c                      # keep the fp16 d / dmin finite
    raw[..., 3] = 0x2c
    k5 = GW.KQuant(raw, GW.GGML_Q5_K, 512)
    assert np.array_equal(k5.dequant().numpy(), dequantize(raw.numpy().reshape(8, -1), T.Q5_K).reshape(8, 512))


def test_shard_index_matches_reference():
    g = load("tp.npz")
    cfg = types.SimpleNamespace(n_head=20, n_kv_head=4, head_dim=128, k_heads=16, v_heads=48, gdn_dim=128, ffn=17408)
    for n in (2, 4):
        for r in range(n):
            for k, v in tp.shard_index(cfg, n, r).items():
                assert np.array_equal(v.numpy(), g[f"n{n}_r{r}_{k}"]), (n, r, k)


def test_linear_shards_partition():
    for n in (1, 2, 4, 8):
        seen = {k: [] for k in ("qkv", "o", "gu", "down")}
        for r in range(n):
            for k, v in tp.linear_shards(5120, 1024, 17408, n, r).items():
                seen[k].append(v)
        assert torch.equal(torch.cat(seen["qkv"]).sort().values, torch.arange(7168))
        assert torch.equal(torch.cat(seen["o"]), torch.arange(5120))
        assert torch.equal(torch.cat(seen["gu"]).sort().values, torch.arange(34816))
        assert torch.equal(torch.cat(seen["down"]), torch.arange(17408))
    with pytest.raises(ValueError):
        tp.linear_shards(5120, 1024, 17408, 3, 0)
    assert tp.parts_elems(64, 5120) == 4 * 64 * 5120 and tp.parts_elems(8192, 5120) == 8192 * 5120


def test_w4a8_repack_matches_reference():
    from prism_b200 import w4a8
    g, k = load("w4a8.npz"), load("kquant.npz")
    w = w4a8.repack(GW.KQuant(torch.from_numpy(k["raw4"]), GW.GGML_Q4_K, 512))
    assert w.kind == "q4k" and (w.n, w.k) == (24, 512)
    for f in ("q", "sc", "mn", "d", "dm"):
        assert np.array_equal(getattr(w, f).numpy(), g[f + "4"]), f
    w6 = w4a8.repack(GW.KQuant(torch.from_numpy(k["raw6"]), GW.GGML_Q6_K, 512))
    for f in ("q", "sc", "d"):
        assert np.array_equal(getattr(w6, f).numpy(), g[f + "6"]), f
    assert w6.mn is None and w6.dm is None
    both = w4a8.concat([w, w])
    assert both.n == 48 and both.sc.shape == (2, 48, 8) and both.q.shape == (48, 256)
    part = both.rows(10, 30)
    assert part.n == 20 and np.array_equal(part.d.numpy(), np.concatenate([g["d4"], g["d4"]], 1)[:, 10:30])
    with pytest.raises(ValueError):
        w4a8.concat([w, w6])


def test_mxfp4_pack_matches_reference():
    from prism_b200 import mxfp4
    g = load("mxfp4.npz")
    w = torch.from_numpy(g["w"])
    for mode in ("max", "mse"):
        m = mxfp4.pack(w, mode)
        assert np.array_equal(m.q.numpy(), g[f"q_{mode}"]) and np.array_equal(m.s.numpy(), g[f"s_{mode}"]), mode
        assert np.array_equal(mxfp4.dequant_packed(m.q, m.s).numpy(), g[f"deq_{mode}"])
    m = mxfp4.pack(torch.from_numpy(g["grid"]))                   # tests/test_mxfp4.py:34-38: exact-grid values survive
    assert np.array_equal(m.q.numpy(), g["grid_q"]) and np.array_equal(m.s.numpy(), g["grid_s"])
    assert float((mxfp4.dequant_packed(m.q, m.s) - torch.from_numpy(g["grid"])).abs().max()) < 1e-6
    assert mxfp4.MX4(m.q, m.s, 1, 32).rows(0, 1).shape == (1, 32)
