"""GPU parity tests: every kernel, called through the C ABI, against the CPU oracle on the same seeded
inputs. Shapes, seeds and tolerances restate the reference's own kernel tests
(reference tests/gpu/test_kernels.cu); cases the reference does not cover (ragged B > 1, GQA with 4 KV
heads, several layers in the pools, shuffled page tables, 27B-sized matrices) are added."""

import ctypes as C

import numpy as np
import pytest
import torch

import q38_testlib as tl
from q38_testlib import bq, pkg

pytestmark = pytest.mark.gpu


def K():
    return pkg.kernels()


def sync_ok():
    torch.cuda.synchronize()
    assert K().q38_device_error(1) == 0


# ---------------------------------------------------------------------------------------------------
# BQ decode: bit-exact dequantised weights
# ---------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("bits", [4, 5, 6, 8])
def test_dequantised_weights_are_bit_exact(bits):
    gold = np.load(tl.ROOT / "tests" / "golden" / "bq_golden.npz")
    cases = [bq.Packed(bits, 128, 192, gold[f"lo{bits}"].tobytes(), gold[f"hi{bits}"].tobytes(),
                       gold[f"sc{bits}"].tobytes()),
             tl.make_bq(256, 320, bits, seed=40 + bits)]
    for p in cases:
        w = tl.DeviceBQ(p)
        out = torch.empty((p.n, p.k), dtype=torch.bfloat16, device="cuda")
        pkg.check(K().q38_bq_dequant(C.byref(w.desc), pkg.ptr(out), None))
        sync_ok()
        want = tl.oracle().dequant(p)
        assert np.array_equal(out.float().cpu().numpy(), want)


# ---------------------------------------------------------------------------------------------------
# qgemm
# ---------------------------------------------------------------------------------------------------
def run_gemm_f32(a_dev, m, w, ws, config, sync=True):
    out = torch.empty((m, w.packed.n), dtype=torch.float32, device="cuda")
    ep = pkg.GemmEpilogue(pkg.EPI_STORE_F32, pkg.ptr(out), w.packed.n, 0, None, None, None, None, 0, 1e-6)
    pkg.check(K().q38_qgemm(pkg.ptr(a_dev), m, C.byref(w.desc), C.byref(ep), C.byref(ws) if ws else None, None, config))
    if sync:
        torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("bits", [4, 5, 6, 8])
def test_qgemm_matches_oracle_all_configs(bits):
    rng = np.random.default_rng(42)
    ws = tl.Workspace()
    for (n, k) in ((256, 256), (1536, 192), (384, 1024)):
        p = tl.make_bq(n, k, bits, seed=bits * 100 + n, std=0.05, fast=(n > 256))
        w = tl.DeviceBQ(p)
        wd = tl.oracle().dequant(p)
        for m in (1, 3, 16, 17, 40, 64, 130, 300, 512):
            a = tl.bf16_round(rng.standard_normal((m, k)))
            a_dev = tl.to_dev_bf16(a)
            want = np.zeros((m, n), np.float32)
            tl.oracle().qgemm(a, wd, None, 3, out=want, ldo=n)
            mag = np.abs(a).astype(np.float64) @ np.abs(wd).astype(np.float64).T
            for cfg in range(K().q38_qgemm_num_configs()):
                if bits == 8 and K().q38_qgemm_config_name(cfg) == b"umma_t512":
                    with pytest.raises(pkg.KernelError):  # not built: shared memory cannot hold two raw stages
                        run_gemm_f32(a_dev, m, w, ws.desc, cfg)
                    continue
                for use_ws in (True, False):
                    got = run_gemm_f32(a_dev, m, w, ws.desc if use_ws else None, cfg)
                    err = np.abs(got.cpu().numpy().astype(np.float64) - want)
                    bad = err > 1e-6 + 2e-3 * mag
                    assert not bad.any(), (bits, n, k, m, cfg, use_ws, float(err.max()))
                    again = run_gemm_f32(a_dev, m, w, ws.desc if use_ws else None, cfg)
                    assert torch.equal(got, again), "second run is not bit-identical"
    sync_ok()
    assert int(ws.counters.abs().sum()) == 0, "tile counters must reset themselves"


def _epilogue_case(m, H, I, n_in, n_store, seed, bits=(5, 4, 6), rows=None):
    """Inputs and oracle results of the three fused epilogues for one token count (with `rows`: the results of those tokens)."""
    rng = np.random.default_rng(seed)
    o = tl.oracle()
    residual = tl.bf16_round(rng.standard_normal((m, H)) * 3)
    xbf = tl.bf16_round(residual)
    partials = np.stack([o.norm_partials(residual[i]) for i in range(m)])
    rs = np.array([o.norm_row_scale(partials[i], H, 1e-6) for i in range(m)], np.float32)
    c = {"m": m, "H": H, "I": I, "n_in": n_in, "n_store": n_store, "residual": residual, "partials": partials,
         "xbf_dev": tl.to_dev_bf16(xbf), "part_dev": torch.from_numpy(partials).cuda(), "rows": rows}
    pick = slice(None) if rows is None else rows
    n_pick = m if rows is None else len(rows)
    xbf, rs = xbf[pick], rs[pick]
    # StoreBF16 + folded-norm row scale, with padded rows trimmed by n_store
    p = tl.make_bq(n_in, H, bits[0], seed=seed + 1, std=0.05, fast=True)
    c["w_store"], wd = tl.DeviceBQ(p, rows=n_store), o.dequant(p)
    c["want_store"] = np.zeros((n_pick, n_in), np.float32)
    o.qgemm(xbf, wd, rs, 0, out=c["want_store"], ldo=n_in)
    # SwiGLU on interleaved gate/up columns
    p = tl.make_bq(2 * I, H, bits[1], seed=seed + 2, std=0.05, fast=True)
    c["w_swiglu"], wd = tl.DeviceBQ(p), o.dequant(p)
    c["want_swiglu"] = np.zeros((n_pick, I), np.float32)
    o.qgemm(xbf, wd, rs, 1, out=c["want_swiglu"], ldo=I)
    # Residual: residual += C, xbf == bf16(residual) exactly, next-norm partials
    p = tl.make_bq(H, I, bits[2], seed=seed + 3, std=0.05, fast=True)
    c["w_res"], wd = tl.DeviceBQ(p), o.dequant(p)
    act = tl.bf16_round(rng.standard_normal((m, I)) * 0.5)
    c["act_dev"] = tl.to_dev_bf16(act)
    c["res_want"] = residual[pick].copy()
    c["xbf_want"], c["part_want"] = np.zeros_like(c["res_want"]), np.zeros_like(partials[pick])
    o.qgemm(act[pick], wd, None, 2, residual=c["res_want"], xbf=c["xbf_want"], partials=c["part_want"])
    return c


def _check_epilogues(c, ws, config):
    m, H, I, n_in, n_store = c["m"], c["H"], c["I"], c["n_in"], c["n_store"]
    pick = slice(None) if c["rows"] is None else c["rows"]
    tag = (m, K().q38_qgemm_config_name(config) if config >= 0 else "auto")
    out = torch.full((m, n_in), 7.0, dtype=torch.bfloat16, device="cuda")
    ep = pkg.GemmEpilogue(pkg.EPI_STORE_BF16, pkg.ptr(out), n_in, n_store, None, None, None, pkg.ptr(c["part_dev"]), H, 1e-6)
    pkg.check(K().q38_qgemm(pkg.ptr(c["xbf_dev"]), m, C.byref(c["w_store"].desc), C.byref(ep), C.byref(ws.desc), None, config))
    got, want = out.float().cpu().numpy(), c["want_store"]
    results = [out]
    assert np.all(got[:, n_store:] == 7.0), ("columns beyond n_store must not be written", tag)
    got = got[pick]
    assert np.all(np.abs(got[:, :n_store] - want[:, :n_store]) <= 1e-3 + 2e-2 * np.abs(want[:, :n_store])), tag

    out = torch.empty((m, I), dtype=torch.bfloat16, device="cuda")
    ep = pkg.GemmEpilogue(pkg.EPI_SWIGLU, pkg.ptr(out), I, 0, None, None, None, pkg.ptr(c["part_dev"]), H, 1e-6)
    pkg.check(K().q38_qgemm(pkg.ptr(c["xbf_dev"]), m, C.byref(c["w_swiglu"].desc), C.byref(ep), C.byref(ws.desc), None, config))
    results.append(out)
    got, want = out.float().cpu().numpy()[pick], c["want_swiglu"]
    assert np.all(np.abs(got - want) <= 2e-2 * (np.abs(want) + 1e-3 * np.abs(want).max())), tag

    res_dev = torch.from_numpy(c["residual"].copy()).cuda()
    xbf_out = torch.empty((m, H), dtype=torch.bfloat16, device="cuda")
    part_out = torch.empty((m, H // 128), dtype=torch.float32, device="cuda")
    ep = pkg.GemmEpilogue(pkg.EPI_RESIDUAL, None, 0, 0, pkg.ptr(res_dev), pkg.ptr(xbf_out), pkg.ptr(part_out), None, 0, 1e-6)
    pkg.check(K().q38_qgemm(pkg.ptr(c["act_dev"]), m, C.byref(c["w_res"].desc), C.byref(ep), C.byref(ws.desc), None, config))
    sync_ok()
    res_got = res_dev.cpu().numpy()
    assert np.all(np.abs(res_got[pick] - c["res_want"]) <= 1e-3 + 1e-3 * np.abs(c["res_want"])), tag
    assert np.array_equal(xbf_out.float().cpu().numpy(), tl.bf16_round(res_got)), tag
    assert np.all(np.abs(part_out.cpu().numpy()[pick] - c["part_want"]) <= 1e-3 + 1e-4 * np.abs(c["part_want"])), tag
    return results + [res_dev, xbf_out, part_out]


@pytest.mark.parametrize("m", [1, 5, 16, 17, 33, 64, 77, 130, 257, 300])
def test_qgemm_epilogues(m):
    """StoreBF16 (+ n_store trimming), SwiGLU and Residual through the dispatcher's own choice and through every
    tile configuration of both kernels (a configuration smaller than m is applied to row blocks)."""
    c = _epilogue_case(m, H=512, I=1024, n_in=1152, n_store=1100, seed=7)
    ws = tl.Workspace()
    for config in range(-1, K().q38_qgemm_num_configs()):
        _check_epilogues(c, ws, config)
    assert int(ws.counters.abs().sum()) == 0


@pytest.mark.parametrize("m", [33, 64])
def test_qgemm_epilogues_27b_width(m):
    """The epilogues at the 27B hidden size (40 weight tiles for the Residual projections, the cut of every tile over
    three CTAs) and a 4-bit gate/up block of 68 tiles, decode-batch token counts."""
    c = _epilogue_case(m, H=5120, I=4352, n_in=2048, n_store=2000, seed=11)
    ws = tl.Workspace()
    names = {K().q38_qgemm_config_name(i).decode(): i for i in range(K().q38_qgemm_num_configs())}
    for config in (-1, names["tmem_t64"], names["tmem_t128"], names["umma_t64"], names["stream_m16"]):
        _check_epilogues(c, ws, config)
    assert int(ws.counters.abs().sum()) == 0


@pytest.mark.parametrize("m", [300, 513, 769, 1531])
def test_qgemm_epilogues_of_several_token_blocks(m):
    """More than 256 tokens: all 256-token blocks in one launch, two to six of them, 80 k-groups per tile. Where the last wave of
    (tile, block) items is uneven enough they are cut over all SMs and pieces meet in the workspace (on 148 SMs: SwiGLU at 300, 769
    and 1531 tokens, all three products at 769), elsewhere a CTA has whole items. Both operand paths, the same bits on a second call,
    counters back at zero; and the whole-item path of a workspace with too few counters, with too few floats, and of none.
    The oracle has the tokens at the edges of the blocks and a few more."""
    rows = sorted({r for b in range(0, m, 256) for r in (b, b + 127, b + 255) if r < m} | {m - 1, m // 2, m // 3})
    c = _epilogue_case(m, H=5120, I=5120, n_in=5120, n_store=5100, seed=17, rows=rows)
    names = {K().q38_qgemm_config_name(i).decode(): i for i in range(K().q38_qgemm_num_configs())}
    ws = tl.Workspace()
    first = _check_epilogues(c, ws, -1)
    for config in (-1, names["tmem_t256x2"], names["umma_t256x2"]):
        for a, b in zip(first, _check_epilogues(c, ws, config)):
            assert torch.equal(a, b), config
    assert int(ws.counters.abs().sum()) == 0
    for small in (tl.Workspace(counters=40), tl.Workspace(floats=2 * 148 * 128 * 128)):
        _check_epilogues(c, small, -1)
        assert int(small.counters.abs().sum()) == 0


@pytest.mark.parametrize("m", [1, 8, 9, 16])
def test_qgemm_allreduce_epilogue_of_tiles_split_over_a_cluster(m):
    """One rank's shard of the 27B down-projection (40 tiles, 34 k-groups: three CTAs per tile): the all-reduce epilogue gathers
    a tile's rows in one CTA of the cluster, the Residual epilogue spreads them over all. With a world of one the sums are
    the same ones, so the results have the same bits. Four calls in a row use both receive buffers twice."""
    n, k = 5120, 2176
    w = tl.DeviceBQ(tl.make_bq(n, k, 5, seed=3, std=0.05, fast=True))
    ws = tl.Workspace()
    gen = torch.Generator(device="cuda").manual_seed(m)
    zeros = lambda count: torch.zeros(count, dtype=torch.int32, device="cuda")
    recv, flags, seq = torch.zeros(2 * 16 * n, device="cuda"), zeros(n // 128), zeros(n // 128)
    ar = pkg.PeerAllreduce()
    ar.world, ar.rank = 1, 0
    ar.recv[0], ar.flags[0], ar.seq = pkg.ptr(recv), pkg.ptr(flags), pkg.ptr(seq)
    for call in range(4):
        a = torch.randn((m, k), generator=gen, device="cuda").to(torch.bfloat16)
        old = torch.randn((m, n), generator=gen, device="cuda")
        got = []
        for kind in (pkg.EPI_RESIDUAL, pkg.EPI_ALLREDUCE_RESIDUAL):
            res, xbf = old.clone(), torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
            part = torch.empty((m, n // 128), device="cuda")
            ep = pkg.GemmEpilogue(kind, None, 0, 0, pkg.ptr(res), pkg.ptr(xbf), pkg.ptr(part), None, 0, 1e-6,
                                  C.pointer(ar) if kind == pkg.EPI_ALLREDUCE_RESIDUAL else None)
            pkg.check(K().q38_qgemm(pkg.ptr(a), m, C.byref(w.desc), C.byref(ep), C.byref(ws.desc), None, -1))
            sync_ok()
            got.append((res, xbf, part))
        assert all(torch.equal(x, y) for x, y in zip(*got)), call
        assert not torch.equal(got[0][0], old)
    assert (seq == 4).all()


@pytest.mark.parametrize("n,k,bits", [(34816, 5120, 4), (5120, 17408, 6)])
def test_qgemm_27b_shapes(n, k, bits):
    """Full-size projection matrices; the oracle is evaluated on a seeded subset of output columns."""
    g = torch.Generator(device="cuda").manual_seed(n)
    wt = torch.randn((n, k), generator=g, device="cuda") * 0.02
    codes, scales = bq.quantize_absmax(wt, bits)
    p = bq.pack(codes.cpu(), scales.cpu(), bits)
    w = tl.DeviceBQ(p)
    ws = tl.Workspace()
    rng = np.random.default_rng(5)
    cols = np.sort(rng.choice(n, size=192, replace=False))
    wd = bq.dequantize(codes[cols].cpu(), scales[cols].cpu()).numpy()
    # whole-matrix dequant check against the python definition (bit-exact)
    deq = torch.empty((n, k), dtype=torch.bfloat16, device="cuda")
    pkg.check(K().q38_bq_dequant(C.byref(w.desc), pkg.ptr(deq), None))
    assert torch.equal(deq[cols].float().cpu(), torch.from_numpy(wd))
    for m in (1, 8, 64, 300):  # streaming kernel, tcgen05 kernel with the weights in TMEM, two 256-token blocks per launch
        a = tl.bf16_round(rng.standard_normal((m, k)))
        want = np.zeros((m, len(cols)), np.float32)
        tl.oracle().qgemm(a, wd, None, 3, out=want, ldo=len(cols))
        mag = np.abs(a).astype(np.float64) @ np.abs(wd).astype(np.float64).T
        a_dev = tl.to_dev_bf16(a)
        got = run_gemm_f32(a_dev, m, w, ws.desc, -1)
        err = np.abs(got[:, cols].cpu().numpy().astype(np.float64) - want)
        assert not (err > 1e-6 + 2e-3 * mag).any(), (m, float(err.max()))
        assert torch.equal(got, run_gemm_f32(a_dev, m, w, ws.desc, -1))
    sync_ok()


@pytest.mark.parametrize("bits", [5, 8])
def test_qgemm_even_cut_over_all_sms(bits):
    """More than four tiles per SM (the LM head's regime): the tcgen05 kernel cuts the list of (tile, k-group) evenly
    over the SMs, so segments begin and end anywhere inside a tile - partial stages, units of one k-group, segments
    of a single unit - and the tiles' pieces meet in the workspace. 11 k-groups per tile make every remainder occur.
    Each configuration against the oracle on a seeded subset of columns, both operand paths bit-identical, and twenty
    launches back to back (each overlapping the tail of the one before) equal to a launch on its own."""
    n, k = 76800, 704
    g = torch.Generator(device="cuda").manual_seed(bits)
    wt = torch.randn((n, k), generator=g, device="cuda") * 0.02
    codes, scales = bq.quantize_absmax(wt, bits)
    p = bq.pack(codes, scales, bits)
    w = tl.DeviceBQ(p)
    ws = tl.Workspace()
    names = {K().q38_qgemm_config_name(c).decode(): c for c in range(K().q38_qgemm_num_configs())}
    rng = np.random.default_rng(bits)
    cols = np.sort(rng.choice(n, size=160, replace=False))
    wd = bq.dequantize(codes[cols].cpu(), scales[cols].cpu()).numpy()
    for m, tok in ((24, 32), (64, 64), (100, 128)):
        a = tl.bf16_round(rng.standard_normal((m, k)))
        want = np.zeros((m, len(cols)), np.float32)
        tl.oracle().qgemm(a, wd, None, 3, out=want, ldo=len(cols))
        mag = np.abs(a).astype(np.float64) @ np.abs(wd).astype(np.float64).T
        a_dev = tl.to_dev_bf16(a)
        outs = {}
        for name in (f"tmem_t{tok}", f"umma_t{tok}"):
            got = run_gemm_f32(a_dev, m, w, ws.desc, names[name])
            err = np.abs(got[:, cols].cpu().numpy().astype(np.float64) - want)
            assert not (err > 1e-6 + 2e-3 * mag).any(), (bits, m, name, float(err.max()))
            outs[name] = got
        assert torch.equal(outs[f"tmem_t{tok}"], outs[f"umma_t{tok}"]), (bits, m)
        for name in (f"tmem_t{tok}", f"umma_t{tok}"):
            for _ in range(20):
                last = run_gemm_f32(a_dev, m, w, ws.desc, names[name], sync=False)
            assert torch.equal(last, outs[name]), (bits, m, name, "back-to-back launches")
    sync_ok()
    assert int(ws.counters.abs().sum()) == 0, "tile counters must reset themselves"


@pytest.mark.parametrize("bits", [4, 5, 8])
def test_qgemm_operand_paths_give_the_same_bits(bits):
    """The tcgen05 kernel hands the decoded weights to the MMA either through shared memory (umma_*) or through
    tensor memory (tmem_*); the MMAs, their order over k and the epilogue are the same, so the outputs must be
    bit-identical, cut over k (with a workspace) or not."""
    names = {K().q38_qgemm_config_name(c).decode(): c for c in range(K().q38_qgemm_num_configs())}
    rng = np.random.default_rng(bits)
    ws = tl.Workspace()
    p = tl.make_bq(2048, 1536, bits, seed=40 + bits, std=0.05, fast=True)
    w = tl.DeviceBQ(p)
    for m, pairs in ((20, [("umma_t32", "tmem_t32")]), (64, [("umma_t64", "tmem_t64")]), (100, [("umma_t128", "tmem_t128")]),
                     (300, [("umma_t256", "tmem_t256"), ("umma_t256x2", "tmem_t256x2")])):
        a_dev = tl.to_dev_bf16(tl.bf16_round(rng.standard_normal((m, 1536))))
        for smem_cfg, tmem_cfg in pairs:
            for use_ws in (True, False):
                x = run_gemm_f32(a_dev, m, w, ws.desc if use_ws else None, names[smem_cfg])
                y = run_gemm_f32(a_dev, m, w, ws.desc if use_ws else None, names[tmem_cfg])
                assert torch.equal(x, y), (bits, m, smem_cfg, tmem_cfg, use_ws)
    sync_ok()


@pytest.mark.parametrize("bits", [4, 5, 6, 8])
def test_quantiser_on_gpu_equals_cpu(bits):
    """The MSE-search quantiser (reference tools/bqpack.py:40-102) is plain tensor arithmetic: run on the GPU it must
    give the codes and scales of the CPU run (which the golden fixtures pin to the reference's bytes)."""
    g = torch.Generator().manual_seed(100 + bits)
    w = torch.randn((384, 1024), generator=g) * 0.02
    w[5, 64:128] = 0.0          # a dead group
    w[7, 0] = 3.0               # an outlier
    c_cpu, s_cpu = bq.quantize_matrix(w, bits)
    c_gpu, s_gpu = bq.quantize_matrix(w.cuda(), bits)
    assert torch.equal(s_gpu.cpu(), s_cpu)
    assert torch.equal(c_gpu.cpu(), c_cpu)


# ---------------------------------------------------------------------------------------------------
# embed, ragged packing
# ---------------------------------------------------------------------------------------------------
def test_embed_matches_oracle():
    H, V = 512, 1024
    g = torch.Generator().manual_seed(1)
    table = (torch.randn((V, H), generator=g)).to(torch.bfloat16)
    tokens = torch.tensor([0, 5, 1023, 17, 17, 400], dtype=torch.int32)
    m = len(tokens)
    # device table and mapped pinned host table (zero-copy)
    host_table = table.clone().pin_memory()
    for tab in (table.cuda(), host_table):
        res = torch.empty((m, H), dtype=torch.float32, device="cuda")
        xbf = torch.empty((m, H), dtype=torch.bfloat16, device="cuda")
        part = torch.empty((m, H // 128), dtype=torch.float32, device="cuda")
        tok_d = tokens.cuda()
        pkg.check(K().q38_embed(pkg.ptr(tab), pkg.ptr(tok_d), m, H, pkg.ptr(res), pkg.ptr(xbf), pkg.ptr(part), None))
        sync_ok()
        rows = table[tokens.long()].float().numpy()
        assert np.array_equal(res.cpu().numpy(), rows)
        assert np.array_equal(xbf.float().cpu().numpy(), rows)
        want = np.stack([tl.oracle().norm_partials(rows[i]) for i in range(m)])
        assert np.all(np.abs(part.cpu().numpy() - want) <= 1e-4 + 1e-5 * np.abs(want))


def test_pack_ragged_matches_host_loops():
    rng = np.random.default_rng(3)
    for nseq in (1, 4, 64, 1500):
        counts = rng.integers(0, 9, size=nseq).astype(np.int32)
        counts[0] = max(counts[0], 1)
        pos0 = rng.integers(0, 5000, size=nseq).astype(np.int32)
        total = int(counts.sum())
        d = lambda a: torch.from_numpy(a).cuda()
        seq_start = torch.empty(nseq + 1, dtype=torch.int32, device="cuda")
        tok_pos = torch.empty(max(total, 1), dtype=torch.int32, device="cuda")
        tok_seq = torch.empty(max(total, 1), dtype=torch.int32, device="cuda")
        counts_d, pos0_d = d(counts), d(pos0)
        pkg.check(K().q38_pack_ragged(pkg.ptr(counts_d), pkg.ptr(pos0_d), nseq, total, pkg.ptr(seq_start),
                                      pkg.ptr(tok_pos), pkg.ptr(tok_seq), None))
        sync_ok()
        want_start = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
        assert np.array_equal(seq_start.cpu().numpy(), want_start)
        want_pos = np.concatenate([pos0[b] + np.arange(counts[b]) for b in range(nseq)]).astype(np.int32)
        want_seq = np.concatenate([np.full(counts[b], b) for b in range(nseq)]).astype(np.int32)
        assert np.array_equal(tok_pos.cpu().numpy()[:total], want_pos)
        assert np.array_equal(tok_seq.cpu().numpy()[:total], want_seq)


# ---------------------------------------------------------------------------------------------------
# attention
# ---------------------------------------------------------------------------------------------------
def run_attention_chunk(pool, layer, nq, nkv, proj, batch, qn_dev, kn_dev, decode, split_rows=4):
    n = batch.num_tokens
    ld = proj.shape[1]
    proj_dev = tl.to_dev_bf16(proj)
    q16 = torch.empty((n, nq, 256), dtype=torch.float16, device="cuda")
    out = torch.empty((n, nq * 256), dtype=torch.bfloat16, device="cuda")
    qp = pkg.QkNormRopeParams(pkg.ptr(proj_dev), ld, pkg.ptr(qn_dev), pkg.ptr(kn_dev), 1e-6, 1e7, nq, nkv, pkg.ptr(q16), layer)
    pkg.check(K().q38_qk_norm_rope_append(C.byref(qp), C.byref(batch.desc), C.byref(pool.desc), None))
    scratch_rows = max(split_rows, batch.desc.num_seqs)
    max_splits = 64 if scratch_rows <= 64 else 16
    split = torch.empty(scratch_rows * nq * max_splits * 258, dtype=torch.float32, device="cuda")
    ap = pkg.AttentionParams(pkg.ptr(q16), pkg.ptr(proj_dev) + nq * 256 * 2, ld, pkg.ptr(out), nq, nkv, layer,
                             pkg.ptr(split), max_splits, scratch_rows)
    fn = K().q38_attention_decode if decode else K().q38_attention_prefill
    pkg.check(fn(C.byref(ap), C.byref(batch.desc), C.byref(pool.desc), None))
    sync_ok()
    return q16.float().cpu().numpy().reshape(n, nq * 256), out.float().cpu().numpy()


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("prefix", [0, 1, 63, 64, 300, 2100])
def test_attention_matches_oracle(dtype, prefix):
    """One sequence: chunked prefill up to `prefix`, then two decode tokens (6 q heads / 1 kv head)."""
    nq, nkv = 6, 1
    ld = 2 * nq * 256 + 2 * nkv * 256
    rng = np.random.default_rng(11 + prefix)
    r3 = np.random.default_rng(3)
    qn, kn = (1 + 0.2 * r3.standard_normal(256)).astype(np.float32), (1 + 0.2 * r3.standard_normal(256)).astype(np.float32)
    qn_dev, kn_dev = torch.from_numpy(qn).cuda(), torch.from_numpy(kn).cuda()
    pool = tl.KvPool(nkv, layers=2, num_pages=64, slots=4, max_pages_per_seq=64, dtype=dtype)
    perm = np.random.default_rng(5).permutation(64).astype(np.int32)
    pool.table[2] = torch.from_numpy(perm).cuda()
    chunks, pos = [], 0
    sizes = (37, 64, 90, 211)
    while pos < prefix:
        n = min(sizes[len(chunks) % 4], prefix - pos)
        chunks.append((pos, n))
        pos += n
    chunks += [(prefix, 1), (prefix + 1, 1)]
    o = tl.oracle()
    okv = tl.OracleKv(o, nkv, prefix + 2)
    got_all, want_all = [], []
    layer = 1
    for pos0, n in chunks:
        proj = tl.bf16_round(rng.standard_normal((n, ld)))
        batch = tl.Batch([(2, pos0, n)])
        q_got, out_got = run_attention_chunk(pool, layer, nq, nkv, proj, batch, qn_dev, kn_dev, decode=(n == 1))
        kd, vd = pool.read_sequence(layer, 2, pos0 + n)
        for i in range(n):
            q_ref = okv.append(nq, 1e-6, 1e7, proj[i], pos0 + i, qn, kn, 2 if dtype == 0 else 1)
            assert np.all(np.abs(q_got[i] - q_ref) <= 2e-3 + 2e-3 * np.abs(q_ref)), (pos0 + i)
            # K written by the kernel vs the oracle's quantisation: at most one int8 step apart
            for h in range(nkv):
                diff = np.abs(kd[h, pos0 + i] - okv.k[h, pos0 + i]).max()
                assert diff <= np.abs(okv.k[h, pos0 + i]).max() / 100.0 + 1e-3
        # attention over the cache contents the kernel actually wrote
        seen = tl.OracleKv(o, nkv, pos0 + n)
        seen.k[:], seen.v[:] = kd, vd
        for i in range(n):
            want_all.append(seen.attend(nq, q_got[i], proj[i, nq * 256:2 * nq * 256], pos0 + i))
            got_all.append(out_got[i])
    got, want = np.stack(got_all), np.stack(want_all)
    assert np.all(np.abs(got - want) <= 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max()))


def test_attention_ragged_batch_gqa4_long_context():
    """B = 5 sequences decoded together, 8 q / 4 kv heads (group 2) and 24 / 4 (group 6), contexts up to 9000,
    shuffled page table, attention layer 2 of 3."""
    rng = np.random.default_rng(21)
    o = tl.oracle()
    for nq, nkv in ((8, 4), (24, 4)):
        ld = 2 * nq * 256 + 2 * nkv * 256
        qn = (1 + 0.2 * rng.standard_normal(256)).astype(np.float32)
        kn = (1 + 0.2 * rng.standard_normal(256)).astype(np.float32)
        qn_dev, kn_dev = torch.from_numpy(qn).cuda(), torch.from_numpy(kn).cuda()
        ctx = [1, 64, 130, 4100, 9000]
        pages_needed = sum((c + 64) // 64 + 1 for c in ctx)
        pool = tl.KvPool(nkv, layers=3, num_pages=pages_needed + 3, slots=8, max_pages_per_seq=160, dtype=0)
        perm = np.random.default_rng(5).permutation(pages_needed + 3).astype(np.int32)
        used = 0
        slots = [6, 0, 3, 1, 5]
        for s, c in zip(slots, ctx):
            need = (c + 64) // 64 + 1
            pool.table[s, :need] = torch.from_numpy(perm[used:used + need]).cuda()
            used += need
        layer = 2
        # fill the caches by prefill chunks of 512 through the append kernel (K/V only matter here)
        for s, c in zip(slots, ctx):
            for p0 in range(0, c - 1, 512):
                n = min(512, c - 1 - p0)
                proj = tl.bf16_round(rng.standard_normal((n, ld)))
                batch = tl.Batch([(s, p0, n)])
                q16 = torch.empty((n, nq, 256), dtype=torch.float16, device="cuda")
                proj_d = tl.to_dev_bf16(proj)
                qp = pkg.QkNormRopeParams(pkg.ptr(proj_d), ld, pkg.ptr(qn_dev), pkg.ptr(kn_dev), 1e-6, 1e7,
                                          nq, nkv, pkg.ptr(q16), layer)
                pkg.check(K().q38_qk_norm_rope_append(C.byref(qp), C.byref(batch.desc), C.byref(pool.desc), None))
        # one decode step for all five
        proj = tl.bf16_round(rng.standard_normal((len(ctx), ld)))
        batch = tl.Batch([(s, c - 1, 1) for s, c in zip(slots, ctx)])
        q_got, out_got = run_attention_chunk(pool, layer, nq, nkv, proj, batch, qn_dev, kn_dev, decode=True, split_rows=8)
        for b, (s, c) in enumerate(zip(slots, ctx)):
            kd, vd = pool.read_sequence(layer, s, c)
            seen = tl.OracleKv(o, nkv, c)
            seen.k[:], seen.v[:] = kd, vd
            want = seen.attend(nq, q_got[b], proj[b, nq * 256:2 * nq * 256], c - 1)
            assert np.all(np.abs(out_got[b] - want) <= 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max())), (nq, b)
        # the same tokens as a ragged "prefill" batch of single-token chunks must agree as well
        _, out_pf = run_attention_chunk(pool, layer, nq, nkv, proj, batch, qn_dev, kn_dev, decode=False, split_rows=8)
        assert np.all(np.abs(out_pf - out_got) <= 2e-2 * (np.abs(out_got) + 0.02 * np.abs(out_got).max()))


def fill_kv_random(pool, layer, nq, nkv, slot, upto, qn_dev, kn_dev, gen):
    """Appends `upto` tokens of N(0, 1) projections (drawn on the device) to a sequence's cache, 512 at a time."""
    ld = 2 * nq * 256 + 2 * nkv * 256
    for p0 in range(0, upto, 512):
        n = min(512, upto - p0)
        proj_d = torch.randn((n, ld), generator=gen, device="cuda").to(torch.bfloat16)
        batch = tl.Batch([(slot, p0, n)])
        q16 = torch.empty((n, nq, 256), dtype=torch.float16, device="cuda")
        qp = pkg.QkNormRopeParams(pkg.ptr(proj_d), ld, pkg.ptr(qn_dev), pkg.ptr(kn_dev), 1e-6, 1e7, nq, nkv, pkg.ptr(q16), layer)
        pkg.check(K().q38_qk_norm_rope_append(C.byref(qp), C.byref(batch.desc), C.byref(pool.desc), None))


def test_attention_decode_16_sequences_up_to_32768():
    """The decode step of a 16-sequence ragged batch, 24 q / 4 kv heads, contexts log-uniform in 128..32768 (seed 3)
    with the longest forced to 32768, page ids from a seeded shuffle."""
    nq, nkv, layer = 24, 4, 0
    ld = 2 * nq * 256 + 2 * nkv * 256
    r3 = np.random.default_rng(3)
    ctx = [int(round(np.exp(u))) for u in r3.uniform(np.log(128), np.log(32768), size=16)]
    ctx[5] = 32768
    qn = (1 + 0.2 * r3.standard_normal(256)).astype(np.float32)
    kn = (1 + 0.2 * r3.standard_normal(256)).astype(np.float32)
    qn_dev, kn_dev = torch.from_numpy(qn).cuda(), torch.from_numpy(kn).cuda()
    need = [(c + 63) // 64 for c in ctx]
    pool = tl.KvPool(nkv, layers=1, num_pages=sum(need) + 5, slots=16, max_pages_per_seq=max(need), dtype=0)
    perm = np.random.default_rng(5).permutation(sum(need) + 5).astype(np.int32)
    used = 0
    for s, pages in enumerate(need):
        pool.table[s, :pages] = torch.from_numpy(perm[used:used + pages]).cuda()
        used += pages
    gen = torch.Generator(device="cuda").manual_seed(33)
    for s, c in enumerate(ctx):
        fill_kv_random(pool, layer, nq, nkv, s, c - 1, qn_dev, kn_dev, gen)
    proj = tl.bf16_round(np.random.default_rng(34).standard_normal((16, ld)))
    batch = tl.Batch([(s, c - 1, 1) for s, c in enumerate(ctx)])
    q_got, out_got = run_attention_chunk(pool, layer, nq, nkv, proj, batch, qn_dev, kn_dev, decode=True, split_rows=64)
    o = tl.oracle()
    for s, c in enumerate(ctx):
        kd, vd = pool.read_sequence(layer, s, c)
        seen = tl.OracleKv(o, nkv, c)
        seen.k[:], seen.v[:] = kd, vd
        want = seen.attend(nq, q_got[s], proj[s, nq * 256:2 * nq * 256], c - 1)
        assert np.all(np.abs(out_got[s] - want) <= 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max())), (s, c)


@pytest.mark.parametrize("dtype", [0, 1], ids=["int8", "bf16"])
@pytest.mark.parametrize("nq,nkv,split_rows", [(24, 4, 4), (3, 1, 800)])
def test_attention_prefill_ragged_chunks_at_long_prefixes(nq, nkv, split_rows, dtype):
    """One ragged prefill step of three sequences: a 512-token chunk behind an 8,200-token prefix, a 200-token chunk
    behind 300 tokens and a 65-token chunk at position 0 (query tiles that start inside a page, end inside a page and
    span pages). 24 q / 4 kv heads is the 27B layer (21 tokens x six heads per tile); 3 q / 1 kv head is one rank of
    the 8-way tensor-parallel layout, where the few tiles cut their keys over several CTAs and the merge kernel
    finishes (the scratch is sized per token for it). Both cache types: int8 pages go through staging, bf16 pages land in the
    operand slots and are converted in place, by asynchronous copies into the same fp16 tiles. The oracle attends over the cache as the kernel wrote it, on a
    sample of the prompt tokens (every position of the short chunks, every 29th and the ends of the long one)."""
    ld = 2 * nq * 256 + 2 * nkv * 256
    r3 = np.random.default_rng(3)
    qn = (1 + 0.2 * r3.standard_normal(256)).astype(np.float32)
    kn = (1 + 0.2 * r3.standard_normal(256)).astype(np.float32)
    qn_dev, kn_dev = torch.from_numpy(qn).cuda(), torch.from_numpy(kn).cuda()
    prefix, chunk, slots, layer = [8200, 300, 0], [512, 200, 65], [2, 0, 1], 1
    need = [(a + c + 63) // 64 for a, c in zip(prefix, chunk)]
    pool = tl.KvPool(nkv, layers=2, num_pages=sum(need) + 3, slots=3, max_pages_per_seq=max(need), dtype=dtype)
    perm = np.random.default_rng(5).permutation(sum(need) + 3).astype(np.int32)
    used = 0
    for s, pages in zip(slots, need):
        pool.table[s, :pages] = torch.from_numpy(perm[used:used + pages]).cuda()
        used += pages
    gen = torch.Generator(device="cuda").manual_seed(44)
    for s, a in zip(slots, prefix):
        fill_kv_random(pool, layer, nq, nkv, s, a, qn_dev, kn_dev, gen)
    n = sum(chunk)
    proj = tl.bf16_round(np.random.default_rng(45).standard_normal((n, ld)))
    batch = tl.Batch([(s, a, c) for s, a, c in zip(slots, prefix, chunk)])
    q_got, out_got = run_attention_chunk(pool, layer, nq, nkv, proj, batch, qn_dev, kn_dev, decode=False,
                                         split_rows=split_rows)
    o = tl.oracle()
    row0 = 0
    got_rows, want_rows, where = [], [], []
    for s, a, c in zip(slots, prefix, chunk):
        kd, vd = pool.read_sequence(layer, s, a + c)
        picks = sorted(set(range(c)) if c <= 200 else set(range(0, c, 29)) | {1, 63, 64, c - 2, c - 1})
        for i in picks:
            pos = a + i
            seen = tl.OracleKv(o, nkv, pos + 1)
            seen.k[:], seen.v[:] = kd[:, :pos + 1], vd[:, :pos + 1]
            want_rows.append(seen.attend(nq, q_got[row0 + i], proj[row0 + i, nq * 256:2 * nq * 256], pos))
            got_rows.append(out_got[row0 + i])
            where.append((s, i, pos))
        row0 += c
    # the reference's bound (tests/gpu/test_kernels.cu:486-492): |got - want| <= 2e-2 (|want| + 0.02 max|want|) with the
    # maximum taken over the whole run
    got, want = np.stack(got_rows), np.stack(want_rows)
    bad = np.abs(got - want) > 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max())
    assert not bad.any(), [where[r] for r in np.nonzero(bad.any(axis=1))[0][:5]]


@pytest.mark.parametrize("seqs", [12, 16, 20, 40])
@pytest.mark.parametrize("dtype", [0, 1], ids=["int8", "bf16"])
def test_attention_decode_merge_of_many_splits(seqs, dtype):
    """The merge takes eight, four, two or one warp per (row, head), by the number of rows and of splits (24 / 4 heads on 148 SMs: up
    to 64, 37, 30 and 15 splits). Contexts with one live split, with a few (a round of loads that is not full) and with all."""
    nq, nkv, layer = 24, 4, 0
    ld = 2 * nq * 256 + 2 * nkv * 256
    rng = np.random.default_rng(seqs)
    ctx = [int(c) for c in rng.choice([1, 64, 700, 1500, 2500, 4500], size=seqs)]
    ctx[:3] = [4500, 1, 2111]
    need = [(c + 63) // 64 for c in ctx]
    pool = tl.KvPool(nkv, layers=1, num_pages=sum(need), slots=seqs, max_pages_per_seq=max(need), dtype=dtype)
    perm, used = rng.permutation(sum(need)).astype(np.int32), 0
    one = torch.ones(256, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(seqs)
    for s, n in enumerate(need):
        pool.table[s, :n] = torch.from_numpy(perm[used:used + n]).cuda()
        used += n
        fill_kv_random(pool, layer, nq, nkv, s, ctx[s] - 1, one, one, gen)
    proj = tl.bf16_round(rng.standard_normal((seqs, ld)))
    batch = tl.Batch([(s, c - 1, 1) for s, c in enumerate(ctx)])
    q_got, out_got = run_attention_chunk(pool, layer, nq, nkv, proj, batch, one, one, decode=True, split_rows=seqs)
    for s in range(0, seqs, 1 if seqs <= 16 else 3):
        seen = tl.OracleKv(tl.oracle(), nkv, ctx[s])
        seen.k[:], seen.v[:] = pool.read_sequence(layer, s, ctx[s])
        want = seen.attend(nq, q_got[s], proj[s, nq * 256:2 * nq * 256], ctx[s] - 1)
        assert np.all(np.abs(out_got[s] - want) <= 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max())), (s, ctx[s])


def write_sequence(pool, layer, slot, k, v):
    """K, V [kv_heads][length][256] into a sequence's pages, as the append kernel lays them out."""
    H, length, _ = k.shape
    table = pool.table[slot].cpu().numpy()
    for p in range((length + 63) // 64):
        page, n = np.zeros(pool.page_bytes, np.uint8), min(64, length - 64 * p)
        for which, x in enumerate((k, v)):
            x = np.pad(x[:, 64 * p:64 * p + n], ((0, 0), (0, 64 - n), (0, 0))).astype(np.float32)
            if pool.dtype == 0:
                g = x.reshape(H, 64, 4, 64)
                scale = (np.abs(g).max(-1) / 127.0).astype(np.float16)
                q = np.rint(g / np.maximum(scale.astype(np.float32), 1e-8)[..., None]).clip(-127, 127).astype(np.int8)
                at, sc_at = which * H * 64 * 256, 2 * H * 64 * 256 + which * H * 64 * 8
                page[at:at + H * 64 * 256] = q.reshape(-1).view(np.uint8)
                page[sc_at:sc_at + H * 64 * 8] = scale.reshape(-1).view(np.uint8)
            else:
                at = which * H * 64 * 512
                page[at:at + H * 64 * 512] = torch.from_numpy(x).to(torch.bfloat16).view(torch.uint8).numpy().reshape(-1)
        base = layer * pool.layer_stride + int(table[p]) * pool.page_bytes
        pool.pool[base:base + pool.page_bytes] = torch.from_numpy(page).cuda()


def run_prefill(pool, layer, nq, nkv, q16, gate, batch, scratch, max_splits, scratch_rows):
    n = batch.num_tokens
    out = torch.empty((n, nq * 256), dtype=torch.bfloat16, device="cuda")
    ap = pkg.AttentionParams(pkg.ptr(q16), pkg.ptr(gate), nq * 256, pkg.ptr(out), nq, nkv, layer, pkg.ptr(scratch), max_splits,
                             scratch_rows)
    pkg.check(K().q38_attention_prefill(C.byref(ap), C.byref(batch.desc), C.byref(pool.desc), None))
    sync_ok()
    return out


@pytest.mark.parametrize("dtype", [0, 1], ids=["int8", "bf16"])
@pytest.mark.parametrize("nq,nkv,cuts", [(24, 4, False), (24, 4, True), (3, 1, True)])
def test_attention_prefill_rising_scores(nq, nkv, cuts, dtype):
    """Keys along single query rows, longer from block to block of 128, so that a row's reference maximum has to move in the middle
    of its tile and the accumulator is rescaled: in consecutive blocks (both score buffers) and in the last one, for some lanes
    of a warp and not for others, by rises on both sides of the 2^8 below which the maximum stays. One tile per CTA and keys
    cut over several. A dropped or doubled factor would be one of at least 2^8."""
    prefix, n, layer, slot = 4400, 70, 1, 1
    rng = np.random.default_rng(12)
    total = prefix + n
    q = rng.standard_normal((n, nq, 256)).astype(np.float16)
    k = 0.3 * rng.standard_normal((nkv, total, 256))
    v = rng.standard_normal((nkv, total, 256))
    blocks = [1, 2, 3, (prefix - 1) // 128 - 1, prefix // 128]
    for j in range(40):
        i, h = (7 * j) % n, (5 * j) % nq
        for t, (b, grow) in enumerate(zip(blocks, (1.0, 2.1, 3.3, 4.6, 6.0))):
            if (j + t) % 4 == 3:
                continue
            pos = 128 * b + 3 * j if b < prefix // 128 else prefix - 41 + j
            # q . k / 16 = 5 ... 9 times `grow`: rises of 7 ... 13 powers of two
            k[h // (nq // nkv), pos] = q[i, h].astype(np.float64) * (16.0 * (5 + 0.1 * j) * grow / (q[i, h].astype(np.float64) ** 2).sum())
    pages = (total + 63) // 64
    pool = tl.KvPool(nkv, layers=2, num_pages=pages + 2, slots=2, max_pages_per_seq=pages, dtype=dtype)
    pool.table[slot] = torch.from_numpy(np.random.default_rng(5).permutation(pages + 2).astype(np.int32)[:pages]).cuda()
    write_sequence(pool, layer, slot, k, v)
    gate = tl.bf16_round(rng.standard_normal((n, nq * 256)))
    scratch = torch.full((n * nq * 16 * 258,), float("nan"), device="cuda")
    got = run_prefill(pool, layer, nq, nkv, torch.from_numpy(q).cuda(), tl.to_dev_bf16(gate), tl.Batch([(slot, prefix, n)]), scratch, 16,
                      n if cuts else 0).float().cpu().numpy()
    seen = tl.OracleKv(tl.oracle(), nkv, total)
    seen.k[:], seen.v[:] = pool.read_sequence(layer, slot, total)
    want = np.stack([seen.attend(nq, q[i].astype(np.float32), gate[i], prefix + i) for i in range(n)])
    assert np.all(np.abs(got - want) <= 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max()))


@pytest.mark.parametrize("nq,nkv,n,prefix", [(3, 1, 512, 2048), (24, 4, 64, 4096), (24, 4, 64, 300), (3, 1, 512, 0), (6, 1, 2, 255)])
def test_attention_prefill_few_tiles_are_cut_over_idle_sms(nq, nkv, n, prefix):
    """With fewer (tile, kv head) pairs than SMs every pair's keys are cut as far as there are SMs for the cuts, down to two blocks of
    128 keys: no cut has more blocks than that asks for. The states that the cuts leave in the scratch (a row maximum of -inf
    where a cut has no keys) count them; results against the oracle, among them tiles that one cut finishes by itself."""
    rng = np.random.default_rng(n + prefix)
    total, layer, slot, max_splits = prefix + n, 0, 0, 16
    pages = (total + 63) // 64
    pool = tl.KvPool(nkv, layers=1, num_pages=pages, slots=1, max_pages_per_seq=pages, dtype=0)
    pool.table[slot] = torch.from_numpy(rng.permutation(pages).astype(np.int32)).cuda()
    k, v = rng.standard_normal((2, nkv, total, 256))
    write_sequence(pool, layer, slot, k, v)
    q = rng.standard_normal((n, nq, 256)).astype(np.float16)
    gate = tl.bf16_round(rng.standard_normal((n, nq * 256)))
    scratch = torch.full((n, nq, max_splits, 258), float("nan"), device="cuda")
    got = run_prefill(pool, layer, nq, nkv, torch.from_numpy(q).cuda(), tl.to_dev_bf16(gate), tl.Batch([(slot, prefix, n)]), scratch, max_splits, n)
    maxima, sums = scratch[..., 256].cpu().numpy(), scratch[..., 257].cpu().numpy()
    live = np.isfinite(maxima) & np.isfinite(sums) | (sums < 0)
    tq = 128 // (nq // nkv)
    room = max(1, min(max_splits, K().q38_num_sms() // (((n + tq - 1) // tq) * nkv)))
    for first in range(0, n, tq):
        blocks = (prefix + min(n, first + tq) + 127) // 128
        per = max(2, -(-blocks // room))
        cuts = live[first:first + tq].any(axis=(0, 1)).sum()  # (a row that sees none of a cut's keys leaves -inf as well)
        assert cuts >= -(-blocks // per), (first, cuts, blocks, per)
    seen = tl.OracleKv(tl.oracle(), nkv, total)
    seen.k[:], seen.v[:] = pool.read_sequence(layer, slot, total)
    picks = sorted(set(range(0, n, 23)) | {n - 1, n // 2, n - 2})
    want = np.stack([seen.attend(nq, q[i].astype(np.float32), gate[i], prefix + i) for i in picks])
    assert np.all(np.abs(got.float().cpu().numpy()[picks] - want) <= 2e-2 * (np.abs(want) + 0.02 * np.abs(want).max()))


# ---------------------------------------------------------------------------------------------------
# Gated DeltaNet
# ---------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("lens", [[1, 1, 1], [5, 1, 2], [1, 2, 300, 3], [255, 1]], ids=str)
def test_gdn_conv_by_vectors_and_at_any_alignment(lens):
    """The same inputs at aligned addresses (four channels per lane) and one element off with an odd row stride (a channel per
    thread): the same taps and products in the same order; the norm of a head is summed in another order, 128 fp32 squares,
    so a value moves by a few units of 2^-24. The state is moved, not computed: the same bytes."""
    nk, nv, slots, layers = 2, 3, 6, 2
    conv_dim = (2 * nk + nv) * 128
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    m = sum(lens)
    x = torch.randn((m, conv_dim), generator=gen, device="cuda").to(torch.bfloat16)
    w = 0.4 * torch.randn((conv_dim, 4), generator=gen, device="cuda")
    state = torch.randn((slots, layers, 3, conv_dim), generator=gen, device="cuda").to(torch.bfloat16)
    batch = tl.Batch([(len(lens) - i, 7, n) for i, n in enumerate(lens)])
    got = []
    for shift, ld in ((0, conv_dim + 8), (1, conv_dim + 3)):
        buf = torch.zeros(m * ld + 8, dtype=torch.bfloat16, device="cuda")
        proj = buf[shift:shift + m * ld].view(m, ld)
        proj[:, :conv_dim] = x
        conv, qkv = state.clone(), torch.full((m, conv_dim), float("nan"), device="cuda")
        cp = pkg.GdnConvParams(pkg.ptr(proj), pkg.ptr(w), pkg.ptr(qkv), 1)
        dims, st = pkg.GdnDims(nk, nv, conv_dim, ld), pkg.GdnStateDesc(pkg.ptr(w), pkg.ptr(conv), layers)
        pkg.check(K().q38_gdn_conv(C.byref(cp), C.byref(dims), C.byref(batch.desc), C.byref(st), None))
        sync_ok()
        got.append((qkv, conv))
    assert torch.equal(got[0][1], got[1][1]) and not torch.equal(got[0][1], state)
    scale = got[1][0].view(m, -1, 128).abs().amax(-1, keepdim=True)
    assert ((got[0][0] - got[1][0]).view(m, -1, 128).abs() <= 2.0 ** -20 * scale).all()


@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("nk,nv,H", [(2, 6, 512), (2, 2, 512), (16, 32, 5120), (16, 48, 5120)])
def test_gdn_matches_oracle(nk, nv, H, chunked):
    """Chunk lengths {37, 64, 1, 1, 100, 1, 17, 300} on slot 1 of 3, GDN layer 1 of 2; a second sequence runs in
    the same ragged batch on slot 2 with its own lengths. Head counts: small ones, 16 key / 32 value heads (value
    heads share a key head in pairs) and the 27B model's 16 / 48 at its hidden size 5120."""
    rng = np.random.default_rng(5)
    o = tl.oracle()
    conv_dim = 2 * nk * 128 + nv * 128
    ld = conv_dim + nv * 128
    layers, layer, slots = 2, 1, 3
    w_ab = tl.bf16_round(rng.standard_normal((2 * nv, H)) / np.sqrt(H))
    conv_w = (0.4 * rng.standard_normal((conv_dim, 4))).astype(np.float32)
    A = (-rng.uniform(0.5, 8, nv)).astype(np.float32)
    dt = (0.5 * rng.standard_normal(nv)).astype(np.float32)
    nw = (1 + 0.2 * rng.standard_normal(128)).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    w_ab_d, conv_w_d, A_d, dt_d, nw_d = tl.to_dev_bf16(w_ab), dev(conv_w), dev(A), dev(dt), dev(nw)
    rec = torch.zeros((slots, layers, nv, 128, 128), dtype=torch.float32, device="cuda")
    conv = torch.zeros((slots, layers, 3, conv_dim), dtype=torch.bfloat16, device="cuda")
    st = pkg.GdnStateDesc(pkg.ptr(rec), pkg.ptr(conv), layers)
    dims = pkg.GdnDims(nk, nv, conv_dim, ld)
    ref_state = {1: (np.zeros(nv * 128 * 128, np.float32), np.zeros(3 * conv_dim, np.float32)),
                 2: (np.zeros(nv * 128 * 128, np.float32), np.zeros(3 * conv_dim, np.float32))}
    pos = {1: 0, 2: 0}
    for n1, n2 in zip((37, 64, 1, 1, 100, 1, 17, 300), (1, 2, 3, 70, 1, 1, 1, 129)):
        seqs = [(1, pos[1], n1), (2, pos[2], n2)]
        batch = tl.Batch(seqs)
        n = n1 + n2
        proj = tl.bf16_round(rng.standard_normal((n, ld)))
        x = tl.bf16_round(rng.standard_normal((n, H)))
        partials = np.stack([o.norm_partials(x[i]) for i in range(n)])
        ab = torch.empty((n, 2 * nv), dtype=torch.float32, device="cuda")
        qkv = torch.empty((n, conv_dim), dtype=torch.float32, device="cuda")
        out = torch.empty((n, nv * 128), dtype=torch.bfloat16, device="cuda")
        proj_d = tl.to_dev_bf16(proj)
        x_d, part_d = tl.to_dev_bf16(x), dev(partials)
        pkg.check(K().q38_gdn_ab(pkg.ptr(x_d), n, H, pkg.ptr(w_ab_d), 2 * nv, pkg.ptr(part_d), 1e-6, pkg.ptr(ab), None))
        cp = pkg.GdnConvParams(pkg.ptr(proj_d), pkg.ptr(conv_w_d), pkg.ptr(qkv), layer)
        pkg.check(K().q38_gdn_conv(C.byref(cp), C.byref(dims), C.byref(batch.desc), C.byref(st), None))
        rp = pkg.GdnRecurrenceParams(pkg.ptr(qkv), pkg.ptr(ab), pkg.ptr(A_d), pkg.ptr(dt_d), pkg.ptr(proj_d) + conv_dim * 2,
                                     ld, pkg.ptr(nw_d), 1e-6, pkg.ptr(out), layer)
        if chunked:  # the 64-token chunked form, also for the short runs (they are padded to a chunk)
            need = K().q38_gdn_chunk_scratch_floats(n, len(seqs), nv)
            scratch = torch.empty(need, dtype=torch.float32, device="cuda")
            pkg.check(K().q38_gdn_recurrence_chunked(C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st),
                                                     pkg.ptr(scratch), need, None))
        else:
            pkg.check(K().q38_gdn_recurrence(C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st), None))
        sync_ok()
        ab_got = ab.cpu().numpy()
        rs = np.array([o.norm_row_scale(partials[i], H, 1e-6) for i in range(n)], np.float32)
        ab_ref = np.zeros((n, 2 * nv), np.float32)
        o.qgemm(x, w_ab, rs, 3, out=ab_ref, ldo=2 * nv)
        assert np.all(np.abs(ab_got - ab_ref) <= 1e-3 + 1e-3 * np.abs(ab_ref))
        got = out.float().cpu().numpy()
        row = 0
        for slot, _, cnt in seqs:
            s, cs = ref_state[slot]
            for i in range(cnt):
                want = o.gdn_token(nk, nv, 1e-6, proj[row], ab_got[row], conv_w, A, dt, nw, s, cs)
                assert np.all(np.abs(got[row] - want) <= 2e-2 * (np.abs(want) + 0.05)), (slot, pos[slot] + i)
                row += 1
            pos[slot] += cnt
    for slot in (1, 2):
        s_got = rec[slot, layer].cpu().numpy().reshape(-1)
        assert np.all(np.abs(s_got - ref_state[slot][0]) <= 1e-3 + 1e-2 * np.abs(ref_state[slot][0]))
        c_got = conv[slot, layer].float().cpu().numpy().reshape(-1)
        assert np.array_equal(c_got, ref_state[slot][1])
    assert float(rec[0].abs().sum()) == 0 and float(rec[:, 0].abs().sum()) == 0, "other slots / layers untouched"


@pytest.mark.parametrize("tensor_cores", [0, 1])
@pytest.mark.parametrize("seqs", [2, 30])
def test_gdn_chunked_matches_sequential_kernel(seqs, tensor_cores):
    """The chunked form against the token-sequential kernel on the same inputs. Few sequences: one value head per CTA of the
    preparation, and the fp32 scan with two CTAs per head and the separate norm kernel. Many: three heads per CTA, the fp32 scan with
    one CTA per head and the norm inside. The scan on the tensor cores has one CTA per (head, sequence) and the separate norm
    kernel with either, fewer CTAs than SMs and more. Both forms of the scan's products (fp32 on the CUDA cores; three bf16 terms a
    factor, six MMAs per product, on the tensor cores) must agree with the sequential kernel to fp32-like rounding."""
    K().q38_gdn_set_chunk_scan_tensor_cores(tensor_cores)
    rng = np.random.default_rng(31)
    nk, nv, layers, layer = 2, 6, 1, 0
    conv_dim = 2 * nk * 128 + nv * 128
    ld = conv_dim + nv * 128
    lens = [int(x) for x in rng.integers(1, 150, size=seqs)]
    n = sum(lens)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A_d = dev((-rng.uniform(0.5, 8, nv)).astype(np.float32))
    dt_d = dev((0.5 * rng.standard_normal(nv)).astype(np.float32))
    nw_d = dev((1 + 0.2 * rng.standard_normal(128)).astype(np.float32))
    qkv_np = rng.standard_normal((n, conv_dim)).astype(np.float32)
    for h in range(2 * nk):  # q and k heads normalised as the conv kernel leaves them
        blk = qkv_np[:, h * 128:(h + 1) * 128]
        blk /= np.sqrt((blk * blk).sum(axis=1, keepdims=True) + 1e-6)
    qkv = dev(qkv_np)
    ab = dev(rng.standard_normal((n, 2 * nv)).astype(np.float32))
    proj_d = tl.to_dev_bf16(tl.bf16_round(rng.standard_normal((n, ld))))
    rec0 = dev((0.1 * rng.standard_normal((seqs, layers, nv, 128, 128))).astype(np.float32))
    batch = tl.Batch([(b, 0, lens[b]) for b in range(seqs)])
    dims = pkg.GdnDims(nk, nv, conv_dim, ld)
    res = []
    for chunked in (False, True):
        rec = rec0.clone()
        conv = torch.zeros((seqs, layers, 3, conv_dim), dtype=torch.bfloat16, device="cuda")
        st = pkg.GdnStateDesc(pkg.ptr(rec), pkg.ptr(conv), layers)
        out = torch.zeros((n, nv * 128), dtype=torch.bfloat16, device="cuda")
        rp = pkg.GdnRecurrenceParams(pkg.ptr(qkv), pkg.ptr(ab), pkg.ptr(A_d), pkg.ptr(dt_d), pkg.ptr(proj_d) + conv_dim * 2,
                                     ld, pkg.ptr(nw_d), 1e-6, pkg.ptr(out), layer)
        if chunked:
            need = K().q38_gdn_chunk_scratch_floats(n, seqs, nv)
            scratch = torch.empty(need, dtype=torch.float32, device="cuda")
            pkg.check(K().q38_gdn_recurrence_chunked(C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st),
                                                     pkg.ptr(scratch), need, None))
        else:
            pkg.check(K().q38_gdn_recurrence(C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st), None))
        sync_ok()
        res.append((out.float().cpu().numpy(), rec.cpu().numpy()))
    K().q38_gdn_set_chunk_scan_tensor_cores(1)
    (o_seq, s_seq), (o_chk, s_chk) = res
    assert np.all(np.abs(o_chk - o_seq) <= 2e-2 * (np.abs(o_seq) + 0.05))
    err = np.abs(s_chk - s_seq)
    assert np.all(err <= 1e-4 + 1e-3 * np.abs(s_seq)), float((err / (1e-4 + 1e-3 * np.abs(s_seq))).max())


def _both_recurrences(nk, nv, lens, ab, A, seed, z_shift=0, spoil=None):
    """(outputs, states) of the token-sequential and of the chunked kernel on the same inputs: one run per sequence."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    conv_dim, n, seqs = (2 * nk + nv) * 128, sum(lens), len(lens)
    ld = conv_dim + nv * 128 + z_shift
    qkv = torch.randn((n, conv_dim), generator=gen, device="cuda")
    qk = qkv[:, :2 * nk * 128].view(n, 2 * nk, 128)
    qk /= qk.norm(dim=-1, keepdim=True)
    if spoil:
        spoil(qkv)
    dt = torch.zeros(nv, device="cuda")
    nw = 1 + 0.2 * torch.randn(128, generator=gen, device="cuda")
    proj = torch.randn((n, ld), generator=gen, device="cuda").to(torch.bfloat16)
    rec0 = 0.1 * torch.randn((seqs, 1, nv, 128, 128), generator=gen, device="cuda")
    batch, dims = tl.Batch([(b, 0, c) for b, c in enumerate(lens)]), pkg.GdnDims(nk, nv, conv_dim, ld)
    res = []
    for chunked in (False, True):
        rec, conv = rec0.clone(), torch.zeros((seqs, 1, 3, conv_dim), dtype=torch.bfloat16, device="cuda")
        st = pkg.GdnStateDesc(pkg.ptr(rec), pkg.ptr(conv), 1)
        out = torch.zeros((n, nv * 128), dtype=torch.bfloat16, device="cuda")
        rp = pkg.GdnRecurrenceParams(pkg.ptr(qkv), pkg.ptr(ab), pkg.ptr(A), pkg.ptr(dt), pkg.ptr(proj) + (conv_dim + z_shift) * 2, ld,
                                     pkg.ptr(nw), 1e-6, pkg.ptr(out), 0)
        args = C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st)
        if chunked:
            need = K().q38_gdn_chunk_scratch_floats(n, seqs, nv)
            scratch = torch.empty(need, device="cuda")
            pkg.check(K().q38_gdn_recurrence_chunked(*args, pkg.ptr(scratch), need, None))
        else:
            pkg.check(K().q38_gdn_recurrence(*args, None))
        sync_ok()
        res.append((out.float(), rec))
    return res


@pytest.mark.parametrize("z_shift", [0, 1])
@pytest.mark.parametrize("lens", [[2], [63], [64], [65], [1, 128, 129, 64], [700]])
def test_gdn_chunk_scan_edges(lens, z_shift):
    """Runs that end on, before and behind a chunk of the scan, one chunk to eleven; gates at an aligned place and rows, and at odd
    ones. Bounds as in test_gdn_chunked_matches_sequential_kernel."""
    nk, nv = 2, 6
    gen = torch.Generator(device="cuda").manual_seed(sum(lens))
    ab = torch.randn((sum(lens), 2 * nv), generator=gen, device="cuda")
    (o_seq, s_seq), (o_chk, s_chk) = _both_recurrences(nk, nv, lens, ab, -0.5 - 7.5 * torch.rand(nv, generator=gen, device="cuda"), 3, z_shift)
    assert ((o_chk - o_seq).abs() <= 2e-2 * (o_seq.abs() + 0.05)).all()
    assert ((s_chk - s_seq).abs() <= 1e-4 + 1e-3 * s_seq.abs()).all()


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("what", ["key", "value"])
@pytest.mark.parametrize("at", [15, 37, 64, 101, 127, 150])
def test_gdn_chunked_rows_that_are_not_finite(at, what, bad):
    """A bad key or value row of a token spoils what follows it in its run, as in the sequential kernel; ahead of its block of sixteen
    tokens, in the other run and (value) in the other heads every output keeps its bits."""
    nk, nv, lens = 2, 6, [170, 70]
    gen = torch.Generator(device="cuda").manual_seed(at)
    ab = torch.randn((sum(lens), 2 * nv), generator=gen, device="cuda")
    A = -0.5 - 7.5 * torch.rand(nv, generator=gen, device="cuda")
    column = (nk + 1) * 128 + 5 if what == "key" else (2 * nk + 4) * 128 + 77  # key head 1 (value heads 3, 4, 5); value head 4

    def spoil(qkv):
        qkv[at, column] = bad

    (_, _), (clean, clean_s) = _both_recurrences(nk, nv, lens, ab, A, 9)
    (seq, seq_s), (got, got_s) = _both_recurrences(nk, nv, lens, ab, A, 9, spoil=spoil)
    heads = [3, 4, 5] if what == "key" else [4]
    got, clean, seq = (x.view(-1, nv, 128) for x in (got, clean, seq))
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[at // 16 * 16:lens[0], heads] = True
    assert torch.equal(got[~hit], clean[~hit])
    for x in (seq, got):  # every later row of the heads, in some of its values at least
        assert not torch.isfinite(x[at:lens[0], heads]).all(-1).any()
    others = [h for h in range(nv) if h not in heads]
    assert torch.equal(got_s[0, :, others], clean_s[0, :, others]) and torch.equal(got_s[1], clean_s[1])
    assert not torch.isfinite(seq_s[0, 0, heads]).all() and not torch.isfinite(got_s[0, 0, heads]).all()


@pytest.mark.parametrize("tensor_cores", [0, 1])
@pytest.mark.parametrize("slow", [False, True])
def test_gdn_chunked_against_float64(slow, tensor_cores):
    """Final states and outputs against the recurrence token by token in float64, with decays as models have them and with ones of at most 1 % a
    token, behind which errors add up longest. States: four times the largest relative error measured (2-norm, 4.7e-7 over 1531
    tokens); outputs: their rounding to bf16, at most 2^-8 each."""
    nk, nv, lens = 2, 6, [333, 129]
    gen = torch.Generator(device="cuda").manual_seed(17)
    rand = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    conv_dim, n = (2 * nk + nv) * 128, sum(lens)
    ld = conv_dim + nv * 128
    qkv, ab, proj, rec0 = rand(n, conv_dim), rand(n, 2 * nv), rand(n, ld).to(torch.bfloat16), 0.1 * rand(2, 1, nv, 128, 128)
    qk = qkv[:, :2 * nk * 128].view(n, 2 * nk, 128)
    qk /= qk.norm(dim=-1, keepdim=True)
    u = torch.rand(nv, generator=gen, device="cuda")
    A, dt, nw = -(0.001 + 0.009 * u if slow else 0.5 + 7.5 * u), torch.zeros(nv, device="cuda"), 1 + 0.2 * rand(128)
    batch, dims, rec, conv = tl.Batch([(0, 0, lens[0]), (1, 0, lens[1])]), pkg.GdnDims(nk, nv, conv_dim, ld), rec0.clone(), torch.zeros((2, 1, 3, conv_dim), dtype=torch.bfloat16, device="cuda")
    need = K().q38_gdn_chunk_scratch_floats(n, 2, nv)
    scratch, out = torch.empty(need, device="cuda"), torch.zeros((n, nv * 128), dtype=torch.bfloat16, device="cuda")
    st = pkg.GdnStateDesc(pkg.ptr(rec), pkg.ptr(conv), 1)
    rp = pkg.GdnRecurrenceParams(pkg.ptr(qkv), pkg.ptr(ab), pkg.ptr(A), pkg.ptr(dt), pkg.ptr(proj) + conv_dim * 2, ld, pkg.ptr(nw), 1e-6, pkg.ptr(out), 0)
    K().q38_gdn_set_chunk_scan_tensor_cores(tensor_cores)
    try:
        pkg.check(K().q38_gdn_recurrence_chunked(C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st), pkg.ptr(scratch), need, None))
        sync_ok()
    finally:
        K().q38_gdn_set_chunk_scan_tensor_cores(1)
    q, k = (qk[:, h * nk:(h + 1) * nk].double().repeat_interleave(nv // nk, 1) for h in (0, 1))
    v, beta = qkv[:, 2 * nk * 128:].double().view(n, nv, 128), torch.sigmoid(ab[:, :nv].double())
    decay = torch.exp(A.double() * torch.nn.functional.softplus(ab[:, nv:].double()))
    want, at = torch.empty((n, nv, 128), dtype=torch.float64, device="cuda"), 0
    for b, length in enumerate(lens):
        s = rec0[b, 0].double()
        for t in range(at, at + length):
            s = s * decay[t, :, None, None]
            s = s + (beta[t, :, None] * (v[t] - torch.einsum("hvk,hk->hv", s, k[t])))[:, :, None] * k[t, :, None, :]
            want[t] = torch.einsum("hvk,hk->hv", s, q[t])
        assert (rec[b, 0].double() - s).norm() < 2e-6 * s.norm()
        at += length
    z = proj[:, conv_dim:].double().view(n, nv, 128)
    want = want / (want.square().mean(-1, keepdim=True) + 1e-6).sqrt() * nw.double() * z * torch.sigmoid(z)
    got = out.double().view(n, nv, 128)
    assert ((got - want).abs() <= want.abs() / 256 + 1e-4 * want.square().mean().sqrt()).all()


@pytest.mark.parametrize("tensor_cores", [0, 1])
@pytest.mark.parametrize("lead", [1, 37, 200])
def test_gdn_chunked_part_of_a_step(lead, tensor_cores):
    """Runs behind the rows of another sequence, with the scratch that their own tokens need: the same bits as by themselves."""
    nk, nv, lens, ld = 2, 6, [170, 70], 22 * 128
    conv_dim, n = (2 * nk + nv) * 128, sum(lens)
    gen = torch.Generator(device="cuda").manual_seed(lead)
    rand = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    qkv, ab, proj, rec0 = rand(lead + n, conv_dim), rand(lead + n, 2 * nv), rand(lead + n, ld).to(torch.bfloat16), 0.1 * rand(3, 1, nv, 128, 128)
    qk = qkv[:, :2 * nk * 128].view(lead + n, 2 * nk, 128)
    qk /= qk.norm(dim=-1, keepdim=True)
    A, dt, nw = -0.5 - 7.5 * torch.rand(nv, generator=gen, device="cuda"), torch.zeros(nv, device="cuda"), 1 + 0.2 * rand(128)
    whole, alone = tl.Batch([(0, 0, lead), (1, 0, lens[0]), (2, 0, lens[1])]), tl.Batch([(1, 0, lens[0]), (2, 0, lens[1])])
    part = pkg.BatchDesc(2, n, max(lens), *[pkg.ptr(t) + 4 * k for t, k in ((whole.seq_start, 1), (whole.seq_slot, 1), (whole.seq_pos0, 1),
                                                                          (whole.tok_pos, lead), (whole.tok_seq, lead))])
    need = K().q38_gdn_chunk_scratch_floats(n, 2, nv)
    dims, res = pkg.GdnDims(nk, nv, conv_dim, ld), []
    K().q38_gdn_set_chunk_scan_tensor_cores(tensor_cores)
    try:
        for first, desc in ((lead, alone.desc), (0, part)):
            x, g, z = qkv[first:], ab[first:], proj[first:]
            rec, conv = rec0.clone(), torch.zeros((3, 1, 3, conv_dim), dtype=torch.bfloat16, device="cuda")
            scratch = torch.full((need + 64,), 7.0, device="cuda")
            out = torch.zeros((lead + n - first, nv * 128), dtype=torch.bfloat16, device="cuda")
            st = pkg.GdnStateDesc(pkg.ptr(rec), pkg.ptr(conv), 1)
            rp = pkg.GdnRecurrenceParams(pkg.ptr(x), pkg.ptr(g), pkg.ptr(A), pkg.ptr(dt), pkg.ptr(z) + conv_dim * 2, ld, pkg.ptr(nw), 1e-6, pkg.ptr(out), 0)
            pkg.check(K().q38_gdn_recurrence_chunked(C.byref(rp), C.byref(dims), C.byref(desc), C.byref(st), pkg.ptr(scratch), need, None))
            sync_ok()
            assert (scratch[need:] == 7.0).all()
            res.append((out, rec))
    finally:
        K().q38_gdn_set_chunk_scan_tensor_cores(1)
    assert (res[1][0][:lead] == 0).all() and torch.equal(res[1][0][lead:], res[0][0]) and torch.equal(res[1][1], res[0][1])


@pytest.mark.parametrize("nk,nv", [(2, 10), (1, 7), (2, 8), (3, 3)])
def test_gdn_chunked_head_ratios(nk, nv):
    """Value heads per key head that the CTAs of the chunk preparation do not divide (five as three and two, seven as three, three
    and one), two CTAs of two, and one each; enough chunks that several heads share a CTA. Bounds as in
    test_gdn_chunked_matches_sequential_kernel."""
    lens = [int(x) for x in np.random.default_rng(nv).integers(1, 150, size=48)]
    gen = torch.Generator(device="cuda").manual_seed(nv)
    ab = torch.randn((sum(lens), 2 * nv), generator=gen, device="cuda")
    (o_seq, s_seq), (o_chk, s_chk) = _both_recurrences(nk, nv, lens, ab, -0.5 - 7.5 * torch.rand(nv, generator=gen, device="cuda"), nv)
    assert ((o_chk - o_seq).abs() <= 2e-2 * (o_seq.abs() + 0.05)).all()
    assert ((s_chk - s_seq).abs() <= 1e-4 + 1e-3 * s_seq.abs()).all()


@pytest.mark.parametrize("seqs", [1, 60])
def test_gdn_chunked_strong_decays(seqs):
    """Sums of the log decays of up to 10^6, then tokens that hardly decay: the factor between two of those is 1, but a difference of
    two sums that were not rounded in the same order is off by an ulp of the sums, 2^-4 here. One value head per CTA and
    several. The sequential kernel multiplies the factors one by one, 0 and 1; bounds as above."""
    nk, nv, n = 1, 6, 64
    gen = torch.Generator(device="cuda").manual_seed(seqs)
    ab = torch.randn((seqs * n, 2 * nv), generator=gen, device="cuda")
    decay = torch.full((seqs, n, nv), -40.0, device="cuda")  # softplus: 4e-18
    decay[:, 2:13] = 2000 + 4000 * torch.rand((seqs, 11, nv), generator=gen, device="cuda")
    ab[:, nv:] = decay.view(seqs * n, nv)
    (o_seq, s_seq), (o_chk, s_chk) = _both_recurrences(nk, nv, [n] * seqs, ab, torch.full((nv,), -16.0, device="cuda"), 5)
    assert ((s_chk - s_seq).abs() <= 1e-4 + 1e-3 * s_seq.abs()).all()
    assert ((o_chk - o_seq).abs() <= 2e-2 * (o_seq.abs() + 0.05)).all()


def test_gdn_decode_kernel_equals_general_kernel():
    """Batches in which every sequence advances by one token take the persistent state-streaming kernel; it must
    reproduce the general kernel bit for bit (outputs and states), also with an empty sequence in the batch and
    with more (sequence, head) items than SMs."""
    rng = np.random.default_rng(21)
    nk, nv, layers, layer, slots = 2, 4, 2, 1, 70
    conv_dim = 2 * nk * 128 + nv * 128
    ld = conv_dim + nv * 128
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A_d = dev((-rng.uniform(0.5, 8, nv)).astype(np.float32))
    dt_d = dev((0.5 * rng.standard_normal(nv)).astype(np.float32))
    nw_d = dev((1 + 0.2 * rng.standard_normal(128)).astype(np.float32))
    rec0 = torch.from_numpy(rng.standard_normal((slots, layers, nv, 128, 128)).astype(np.float32) * 0.1).cuda()
    seqs = [(slot, 5, 0 if slot == 17 else 1) for slot in range(2, 66)]
    n = sum(c for _, _, c in seqs)
    dims = pkg.GdnDims(nk, nv, conv_dim, ld)
    results = []
    for force_general in (False, True):
        rec = rec0.clone()
        conv = torch.zeros((slots, layers, 3, conv_dim), dtype=torch.bfloat16, device="cuda")
        st = pkg.GdnStateDesc(pkg.ptr(rec), pkg.ptr(conv), layers)
        outs = []
        step_rng = np.random.default_rng(22)
        for step in range(3):
            batch = tl.Batch(seqs)
            if force_general:
                batch.desc.max_tokens_per_seq = 2
            qkv = dev(step_rng.standard_normal((n, conv_dim)).astype(np.float32) * 0.3)
            ab = dev(step_rng.standard_normal((n, 2 * nv)).astype(np.float32))
            proj_d = tl.to_dev_bf16(tl.bf16_round(step_rng.standard_normal((n, ld))))
            out = torch.zeros((n, nv * 128), dtype=torch.bfloat16, device="cuda")
            rp = pkg.GdnRecurrenceParams(pkg.ptr(qkv), pkg.ptr(ab), pkg.ptr(A_d), pkg.ptr(dt_d),
                                         pkg.ptr(proj_d) + conv_dim * 2, ld, pkg.ptr(nw_d), 1e-6, pkg.ptr(out), layer)
            pkg.check(K().q38_gdn_recurrence(C.byref(rp), C.byref(dims), C.byref(batch.desc), C.byref(st), None))
            sync_ok()
            outs.append(out.view(torch.int16).cpu().numpy())
        results.append((outs, rec.cpu().numpy()))
    for a, b in zip(results[0][0], results[1][0]):
        assert np.array_equal(a, b)
    assert np.array_equal(results[0][1], results[1][1])
    assert np.array_equal(results[0][1][17], rec0[17].cpu().numpy()), "the empty sequence's state is untouched"
    assert not np.array_equal(results[0][1][2, layer], rec0[2, layer].cpu().numpy())


# ---------------------------------------------------------------------------------------------------
# sampling
# ---------------------------------------------------------------------------------------------------
def run_sampler(logits, params, step, history=None, hist_len=None, cap=16):
    B, V = logits.shape
    lg = torch.from_numpy(logits.copy()).cuda()
    prm = (pkg.SamplingParamsDev * B)(*params)
    prm_dev = torch.frombuffer(bytearray(bytes(prm)), dtype=torch.uint8).cuda()
    slot = torch.arange(B, dtype=torch.int32, device="cuda")
    steps = torch.full((B,), step, dtype=torch.int32, device="cuda")
    hl = torch.zeros(B, dtype=torch.int32, device="cuda") if hist_len is None else torch.tensor(hist_len, dtype=torch.int32, device="cuda")
    hist = torch.zeros((B, cap), dtype=torch.int32, device="cuda") if history is None else torch.tensor(history, dtype=torch.int32, device="cuda")
    out = torch.empty(B, dtype=torch.int32, device="cuda")
    lp = torch.empty(B, dtype=torch.float32, device="cuda")
    a = pkg.SamplingArgs(pkg.ptr(lg), V, V, pkg.ptr(prm_dev), pkg.ptr(slot), pkg.ptr(hist), pkg.ptr(hl), cap,
                         pkg.ptr(steps), pkg.ptr(out), pkg.ptr(lp))
    pkg.check(K().q38_sample(C.byref(a), B, None))
    torch.cuda.synchronize()
    return out.cpu().numpy(), lp.cpu().numpy(), lg.cpu().numpy(), hl.cpu().numpy(), hist.cpu().numpy()


def P(t=0.0, k=0, p=1.0, minp=0.0, pres=0.0, rep=1.0, seed=1):
    return pkg.SamplingParamsDev(t, k, p, minp, pres, rep, seed)


def test_sampling_filters_and_determinism():
    V, B = 248320, 4
    rng = np.random.default_rng(9)
    logits = (2.0 * rng.standard_normal((B, V))).astype(np.float32)
    logits[3] = -1e4
    toks, lps = [10, 20, 30, 40, 50], [0.0, -0.5, -1.0, -2.0, -8.0]
    for t, l in zip(toks, lps):
        logits[3, t] = l
    logits[1, 77] = logits[1].max() + 1.0
    logits[1, 50000] = logits[1, 77]  # a tie: the lowest id wins
    argmax = logits.argmax(axis=1)
    assert argmax[1] == 77
    got, lp, _, hl, hist = run_sampler(logits, [P()] * B, 0)
    assert np.array_equal(got, argmax) and np.all(lp == 0.0)
    assert np.all(hl == 1) and np.array_equal(hist[:, 0], argmax), "the sampled token is appended to the history"
    got, *_ = run_sampler(logits, [P(t=1.0, k=1)] * B, 0)
    assert np.array_equal(got, argmax)
    # top-p 0.9 on row 3: nucleus {10, 20, 30}
    counts, trials = {}, 1500
    for s in range(trials):
        t = int(run_sampler(logits, [P(t=1.0, p=0.9, seed=1234)] * B, s)[0][3])
        counts[t] = counts.get(t, 0) + 1
    assert set(counts) <= {10, 20, 30}
    z = sum(np.exp(l) for l in lps[:3])
    for t, l in zip(toks[:3], lps[:3]):
        expect = np.exp(l) / z * trials
        assert abs(counts.get(t, 0) - expect) < 5 * np.sqrt(expect)
    for s in range(200):  # min_p 0.3 keeps logits >= log 0.3
        assert int(run_sampler(logits, [P(t=1.0, minp=0.3, seed=99)] * B, s)[0][3]) in (10, 20, 30)
    a = run_sampler(logits, [P(t=0.8, k=50, p=0.95, seed=777)] * B, 5)[0]
    b = run_sampler(logits, [P(t=0.8, k=50, p=0.95, seed=777)] * B, 5)[0]
    assert np.array_equal(a, b)
    # penalties: each distinct history token is penalised once
    history = np.zeros((B, 16), np.int32)
    history[0, :3] = [argmax[0], argmax[0], 5]
    _, _, lg_after, _, _ = run_sampler(logits, [P(pres=0.5, rep=2.0)] * B, 0, history=history.tolist(), hist_len=[3, 0, 0, 0])
    l0 = logits[0, argmax[0]]
    assert np.isclose(lg_after[0, argmax[0]], (l0 / 2.0 if l0 > 0 else l0 * 2.0) - 0.5)
    l5 = logits[0, 5]
    assert np.isclose(lg_after[0, 5], (l5 / 2.0 if l5 > 0 else l5 * 2.0) - 0.5)


def test_sampler_draws_equal_the_cpu_restatement():
    """The stochastic sampler against its CPU restatement (oracle/q38_oracle.cpp): sampled token ids must be
    identical, draw for draw, on the 27B vocabulary (248,320 logits) for top-k, top-p, min-p, their combinations and
    penalties: 10,240 draws = 10 parameter sets x 4 logit rows x 256 (seed, step) pairs. Both sides compute the
    fixed-point masses and thresholds with the same IEEE operations, so there is no tolerance on the ids; the reported
    log-probability goes through a library log and is compared to 1e-5."""
    V, D = 248320, 256
    rng = np.random.default_rng(90)
    o = tl.oracle()
    rows = [(2.0 * rng.standard_normal(V)).astype(np.float32),            # flat: thousands of candidates
            (6.0 * rng.standard_normal(V)).astype(np.float32),            # peaked
            np.round(3.0 * rng.standard_normal(V)).astype(np.float32),    # heavy ties (integer logits)
            (0.02 * rng.standard_normal(V)).astype(np.float32) * 70.0]    # the range of a random-weight model
    psets = [dict(t=1.0, k=50), dict(t=0.7, k=0, p=0.9), dict(t=1.3, minp=0.05), dict(t=0.8, k=20, p=0.95),
             dict(t=1.0, k=1000, p=0.5, minp=0.001), dict(t=0.6), dict(t=2.5, p=0.99), dict(t=1.0, k=40, pres=0.7, rep=1.3),
             dict(t=0.9, p=0.8, pres=-0.5, rep=0.8), dict(t=1.0, k=5, minp=0.2, rep=2.0)]
    cap = 64
    mism = 0
    for pi, ps in enumerate(psets):
        for ri, row in enumerate(rows):
            seeds = rng.integers(1, 2 ** 63, size=D, dtype=np.uint64)
            steps = rng.integers(0, 5000, size=D).astype(np.int32)
            order = np.argsort(row)
            hist = np.concatenate([order[-20:], order[-5:], rng.integers(0, V, size=cap - 25)]).astype(np.int32)
            assert hist.shape == (cap,)  # the kernel addresses history rows of exactly `cap` entries
            use_hist = ("pres" in ps) or ("rep" in ps)
            prm = [P(t=ps["t"], k=ps.get("k", 0), p=ps.get("p", 1.0), minp=ps.get("minp", 0.0), pres=ps.get("pres", 0.0),
                     rep=ps.get("rep", 1.0), seed=int(sd)) for sd in seeds]
            lg = torch.from_numpy(row).cuda().repeat(D, 1).contiguous()
            prm_dev = torch.frombuffer(bytearray(bytes((pkg.SamplingParamsDev * D)(*prm))), dtype=torch.uint8).cuda()
            slot = torch.arange(D, dtype=torch.int32, device="cuda")
            steps_d = torch.from_numpy(steps).cuda()
            hl = torch.full((D,), len(hist) if use_hist else 0, dtype=torch.int32, device="cuda")
            hist_d = torch.from_numpy(np.tile(hist, (D, 1))).cuda().contiguous()
            out = torch.full((D,), -1, dtype=torch.int32, device="cuda")
            lp = torch.empty(D, dtype=torch.float32, device="cuda")
            a = pkg.SamplingArgs(pkg.ptr(lg), V, V, pkg.ptr(prm_dev), pkg.ptr(slot), pkg.ptr(hist_d), pkg.ptr(hl), cap,
                                 pkg.ptr(steps_d), pkg.ptr(out), pkg.ptr(lp))
            pkg.check(K().q38_sample(C.byref(a), D, None))
            sync_ok()
            pen = o.sample_penalties(row, hist if use_hist else [], ps.get("pres", 0.0), ps.get("rep", 1.0), cap)
            assert np.array_equal(lg[0].cpu().numpy(), pen), "penalised logits differ"
            want, want_lp = o.sample_draws(pen, ps["t"], ps.get("k", 0), ps.get("p", 1.0), ps.get("minp", 0.0), seeds, steps)
            got = out.cpu().numpy()
            mism += int((got != want).sum())
            assert np.array_equal(got, want), (pi, ri, int((got != want).sum()), got[:8], want[:8])
            assert np.allclose(lp.cpu().numpy(), want_lp, atol=1e-5, rtol=1e-5), (pi, ri)
            assert len(np.unique(got)) > 1 or ps.get("k", 0) == 1
    assert mism == 0


@pytest.mark.parametrize("V,ld,D", [(9, 9, 2), (1024, 1024, 40), (1027, 1031, 3), (16383, 16384, 150), (131077, 131077, 5), (248320, 248320, 1)])
def test_sampler_split_over_a_cluster_equals_the_cpu_restatement(V, ld, D):
    """Rows divided over 1 ... 8 CTAs, rows that do not start on 16 bytes, and the edges of the short-list path: its largest
    top_k and one more, ties that overflow the lists (all logits equal), candidates in one CTA's part, -inf logits. Integer
    masses leave no tolerance on the ids."""
    rng = np.random.default_rng(V + D)
    o = tl.oracle()
    clump = rng.standard_normal(V).astype(np.float32)
    clump[:max(1, V // 16)] += 9.0
    holes = (4.0 * rng.standard_normal(V)).astype(np.float32)
    holes[rng.random(V) < 0.9] = -np.inf
    holes[V // 2] = 3.0
    for row in (clump, holes, np.zeros(V, np.float32), np.round(rng.standard_normal(V)).astype(np.float32)):
        for ps in (dict(k=20, p=0.95), dict(k=1), dict(k=256, p=0.7), dict(k=257, minp=0.01), dict(k=V - 1, p=0.5), dict(k=V),
                   dict(p=0.9), dict(minp=0.2), dict()):
            seeds = rng.integers(1, 2 ** 63, size=D, dtype=np.uint64)
            steps = rng.integers(0, 5000, size=D).astype(np.int32)
            prm = [P(t=0.9, k=ps.get("k", 0), p=ps.get("p", 1.0), minp=ps.get("minp", 0.0), seed=int(sd)) for sd in seeds]
            lg = torch.full((D, ld), 50.0, device="cuda")  # columns behind the vocabulary must not be read
            lg[:, :V] = torch.from_numpy(row).cuda()
            prm_dev = torch.frombuffer(bytearray(bytes((pkg.SamplingParamsDev * D)(*prm))), dtype=torch.uint8).cuda()
            out, lp = torch.full((D,), -1, dtype=torch.int32, device="cuda"), torch.empty(D, device="cuda")
            steps_d = torch.from_numpy(steps).cuda()
            a = pkg.SamplingArgs(pkg.ptr(lg), ld, V, pkg.ptr(prm_dev), None, None, None, 0, pkg.ptr(steps_d), pkg.ptr(out), pkg.ptr(lp))
            pkg.check(K().q38_sample(C.byref(a), D, None))
            sync_ok()
            want, want_lp = o.sample_draws(row, 0.9, ps.get("k", 0), ps.get("p", 1.0), ps.get("minp", 0.0), seeds, steps)
            assert np.array_equal(out.cpu().numpy(), want), ps
            assert np.allclose(lp.cpu().numpy(), want_lp, atol=1e-5, rtol=1e-5), ps  # the log of a double: one fp32 rounding


@pytest.mark.parametrize("first_zero", [0.0, -0.0])
@pytest.mark.parametrize("V", [640, 4096, 30001])
def test_sampler_with_zero_maxima_and_nan(V, first_zero):
    """Maxima of zero with both signs (the first one's decides) and NaN of both signs among the logits: a NaN is no maximum and has no
    mass, but a positive one counts as one of the top k; where nothing with a mass is left, the maximum, in a row without a number token 0. As in
    the test above, ids leave no tolerance."""
    D = 6
    rng = np.random.default_rng(V)
    o = tl.oracle()
    zeros = -np.abs(rng.standard_normal(V)).astype(np.float32)
    at = np.sort(rng.choice(V, 9, replace=False))
    zeros[at] = [first_zero] + [0.0, -0.0] * 4
    nans = (3.0 * rng.standard_normal(V)).astype(np.float32)
    at = rng.choice(np.arange(1, V), 8, replace=False)
    nans[at] = np.array([0x7fc00000, 0x7f800001, 0xffc00000, 0xffffffff] * 2, np.uint32).view(np.float32)
    both = zeros.copy()
    both[at] = nans[at]
    both[0] = first_zero
    none = np.full(V, -np.inf, np.float32)
    none[at] = nans[at]
    few = np.full(V, np.float32(np.nan))
    few[at[:5]] = [-7.0, 2.0, 1.0, 2.0, -3.0]
    for row in (zeros, nans, both, none, few):
        for ps in (dict(k=1), dict(k=4), dict(k=20, p=0.95), dict(k=5), dict(k=8, minp=1.0), dict(k=256, p=0.7), dict(k=300, p=0.9), dict(p=0.9), dict(minp=1.0), dict(), dict(t=0.0)):
            seeds = rng.integers(1, 2 ** 63, size=D, dtype=np.uint64)
            steps = rng.integers(0, 5000, size=D).astype(np.int32)
            prm = [P(t=ps.get("t", 0.9), k=ps.get("k", 0), p=ps.get("p", 1.0), minp=ps.get("minp", 0.0), seed=int(sd)) for sd in seeds]
            lg = torch.from_numpy(np.tile(row, (D, 1))).cuda()
            prm_dev = torch.frombuffer(bytearray(bytes((pkg.SamplingParamsDev * D)(*prm))), dtype=torch.uint8).cuda()
            out, lp = torch.full((D,), -1, dtype=torch.int32, device="cuda"), torch.empty(D, device="cuda")
            steps_d = torch.from_numpy(steps).cuda()
            a = pkg.SamplingArgs(pkg.ptr(lg), V, V, pkg.ptr(prm_dev), None, None, None, 0, pkg.ptr(steps_d), pkg.ptr(out), pkg.ptr(lp))
            pkg.check(K().q38_sample(C.byref(a), D, None))
            sync_ok()
            want, want_lp = o.sample_draws(row, ps.get("t", 0.9), ps.get("k", 0), ps.get("p", 1.0), ps.get("minp", 0.0), seeds, steps)
            assert np.array_equal(out.cpu().numpy(), want), ps
            assert np.allclose(lp.cpu().numpy(), want_lp, atol=1e-5, rtol=1e-5), ps


@pytest.mark.parametrize("V,D", [(131077, 5), (131077, 60), (131077, 120), (131077, 150), (40000, 3)])
def test_sampler_penalties_reach_every_cta_of_a_row(V, D):
    """One CTA of a row's cluster (eight, four, two; two with more rows than SMs; eight of a smaller vocabulary) changes the logits of the history, the others
    read them behind the barrier: ids in every CTA's part, the largest logits among them, so that a stale one would be drawn."""
    rng = np.random.default_rng(V + D)
    o, cap = tl.oracle(), 96
    row = (3.0 * rng.standard_normal(V)).astype(np.float32)
    top = np.argsort(row)[::-1]
    hist = np.concatenate([top[:40], np.arange(16) * (V // 16) + 5, rng.integers(0, V, size=cap - 56)]).astype(np.int32)
    row[hist[40:56]] = row[top[0]] + 0.5  # one per sixteenth of the row
    for ps in (dict(t=0.0), dict(t=0.9, k=20, p=0.95), dict(t=0.8, k=256), dict(t=0.9, p=0.9), dict(t=0.7, k=300, minp=0.01), dict(t=0.5)):
        pres, rep = 1.5, 1.7
        seeds = rng.integers(1, 2 ** 63, size=D, dtype=np.uint64)
        steps = rng.integers(0, 5000, size=D).astype(np.int32)
        prm = [P(t=ps["t"], k=ps.get("k", 0), p=ps.get("p", 1.0), minp=ps.get("minp", 0.0), pres=pres, rep=rep, seed=int(sd)) for sd in seeds]
        lg = torch.from_numpy(row).cuda().repeat(D, 1).contiguous()
        prm_dev = torch.frombuffer(bytearray(bytes((pkg.SamplingParamsDev * D)(*prm))), dtype=torch.uint8).cuda()
        hl = torch.full((D,), cap, dtype=torch.int32, device="cuda")
        hist_d, steps_d = torch.from_numpy(np.tile(hist, (D, 1))).cuda().contiguous(), torch.from_numpy(steps).cuda()
        out, lp = torch.full((D,), -1, dtype=torch.int32, device="cuda"), torch.empty(D, device="cuda")
        a = pkg.SamplingArgs(pkg.ptr(lg), V, V, pkg.ptr(prm_dev), None, pkg.ptr(hist_d), pkg.ptr(hl), cap, pkg.ptr(steps_d), pkg.ptr(out),
                             pkg.ptr(lp))
        pkg.check(K().q38_sample(C.byref(a), D, None))
        sync_ok()
        pen = o.sample_penalties(row, hist, pres, rep, cap)
        assert pen.argmax() not in hist and row.argmax() in hist
        if ps["t"] == 0.0:
            want = np.full(D, pen.argmax())
        else:
            want, want_lp = o.sample_draws(pen, ps["t"], ps.get("k", 0), ps.get("p", 1.0), ps.get("minp", 0.0), seeds, steps)
            assert np.allclose(lp.cpu().numpy(), want_lp, atol=1e-5, rtol=1e-5), ps
        assert np.array_equal(out.cpu().numpy(), want), ps
        assert (hl == cap + 1).all() and np.array_equal(hist_d[:, 0].cpu().numpy(), want)


def test_target_logprobs_matches_oracle():
    rng = np.random.default_rng(2)
    V, rows = 4096, 5
    logits = (3 * rng.standard_normal((rows, V))).astype(np.float32)
    targets = rng.integers(0, V, size=rows).astype(np.int32)
    out = torch.empty(rows, dtype=torch.float32, device="cuda")
    lg_d, tg_d = torch.from_numpy(logits).cuda(), torch.from_numpy(targets).cuda()
    pkg.check(K().q38_target_logprobs(pkg.ptr(lg_d), V, V, pkg.ptr(tg_d), rows, pkg.ptr(out), None))
    torch.cuda.synchronize()
    lib = tl.oracle().fn("target_logprob", C.c_float)
    want = [lib(logits[i].ctypes.data_as(C.c_void_p), C.c_int(V), C.c_int(int(targets[i]))) for i in range(rows)]
    assert np.allclose(out.cpu().numpy(), np.array(want, np.float32), atol=1e-5)


def test_launchers_reject_bad_arguments_without_launching():
    p = tl.make_bq(128, 64, 4, seed=1, fast=True)
    w = tl.DeviceBQ(p)
    a = torch.zeros((1, 64), dtype=torch.bfloat16, device="cuda")
    out = torch.zeros((1, 128), dtype=torch.float32, device="cuda")
    ep = pkg.GemmEpilogue(pkg.EPI_STORE_F32, pkg.ptr(out), 128, 0, None, None, None, None, 0, 1e-6)
    assert K().q38_qgemm(pkg.ptr(a), 0, C.byref(w.desc), C.byref(ep), None, None, -1) == -1
    assert b"m must be positive" in K().q38_last_error()
    bad = pkg.BQWeight(w.desc.lo, None, w.desc.scales, 7, 128, 64, 128)
    assert K().q38_qgemm(pkg.ptr(a), 1, C.byref(bad), C.byref(ep), None, None, -1) == -1
    assert K().q38_embed(None, None, 0, 128, None, None, None, None) == 0  # m == 0 is a no-op
    # the all-reduce epilogue: its peer description is required, it serves up to 16 tokens, and only the streaming kernel
    res = torch.zeros((32, 128), dtype=torch.float32, device="cuda")
    xbf = torch.zeros((32, 128), dtype=torch.bfloat16, device="cuda")
    part = torch.zeros((32, 1), dtype=torch.float32, device="cuda")
    ep = pkg.GemmEpilogue(pkg.EPI_ALLREDUCE_RESIDUAL, None, 0, 0, pkg.ptr(res), pkg.ptr(xbf), pkg.ptr(part), None, 0, 1e-6)
    assert K().q38_qgemm(pkg.ptr(a), 1, C.byref(w.desc), C.byref(ep), None, None, -1) == -1
    assert b"peer description" in K().q38_last_error()
    ar = pkg.PeerAllreduce()
    ar.world, ar.rank = 1, 0
    buf = torch.zeros(2 * 16 * 128, dtype=torch.float32, device="cuda")
    words = torch.zeros(8, dtype=torch.int32, device="cuda")
    ar.recv[0], ar.flags[0], ar.seq = pkg.ptr(buf), pkg.ptr(words), pkg.ptr(words) + 16
    ep = pkg.GemmEpilogue(pkg.EPI_ALLREDUCE_RESIDUAL, None, 0, 0, pkg.ptr(res), pkg.ptr(xbf), pkg.ptr(part), None, 0, 1e-6,
                          C.pointer(ar))
    a32 = torch.zeros((32, 64), dtype=torch.bfloat16, device="cuda")
    assert K().q38_qgemm(pkg.ptr(a32), 17, C.byref(w.desc), C.byref(ep), None, None, -1) == -1
    assert b"up to 16 tokens" in K().q38_last_error()
    names = {K().q38_qgemm_config_name(c).decode(): c for c in range(K().q38_qgemm_num_configs())}
    assert K().q38_qgemm(pkg.ptr(a32), 8, C.byref(w.desc), C.byref(ep), None, None, names["tmem_t32"]) == -1
    assert b"streaming kernel only" in K().q38_last_error()
    ar.world = 9
    assert K().q38_qgemm(pkg.ptr(a), 1, C.byref(w.desc), C.byref(ep), None, None, -1) == -1
