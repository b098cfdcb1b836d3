"""The places where the kernels' branches meet: tile edges, remainders, half-way codes, the smallest and largest sizes.

Everything is compared with the CPU oracle; integer results and dequantized values bit for bit.
"""
import numpy as np
import pytest

import nuvec_b200 as nv
import oracle
from cuda_backend import CudaBackend, host
from test_qmm_plan import SHAPES

pytestmark = pytest.mark.gpu

CODE = {"f32": oracle.F32, "f16": oracle.F16, "bf16": oracle.BF16}
NVC = {"f32": nv.F32, "f16": nv.F16, "bf16": nv.BF16}


@pytest.fixture(scope="module")
def be():
    return CudaBackend()


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
def test_quantize_codes_at_half_way_points(be, bits, dt):
    """Values of few bits put many quotients exactly on, or a rounding away from, a half-way point between two codes."""
    rng = np.random.default_rng(bits)
    for gs in (32, 64, 128):
        grid = rng.integers(-200, 201, (24, 3 * gs)).astype(np.float32) * 2.0 ** rng.integers(-9, 3, (24, 1)).astype(np.float32)
        grid[0], grid[1, :gs], grid[2, ::2] = 0.0, 1e-30, np.float32(-0.0)
        w = oracle.from_f32(grid, CODE[dt])
        got = be.quantize(w, NVC[dt], oracle.AFFINE, gs, bits)
        want = oracle.quantize(w, CODE[dt], oracle.AFFINE, gs, bits)
        for g, o in zip(got, want):
            assert np.array_equal(np.asarray(g).view(np.uint8), np.asarray(o).view(np.uint8)), (bits, gs, dt)


@pytest.mark.parametrize("dt", ["bf16", "f32"])
def test_rms_norm_where_the_sums_rounding_is_in_doubt(be, dt):
    """Sums of squares exactly half-way between two float32: the reference's own order has to decide."""
    for d in (8, 24, 4096, 20000):
        x = np.zeros((3, d), np.float32)
        x[:, 0], x[0, 1], x[1, d - 1], x[2, d // 2] = 1.0, 2.0 ** -12, 2.0 ** -12, -(2.0 ** -12)
        xs = oracle.from_f32(x, CODE[dt])
        got = host(nv.rms_norm(be.up(xs, NVC[dt]), None, 0.0))
        assert np.array_equal(got.view(np.uint8), np.ascontiguousarray(oracle.rms_norm(xs, CODE[dt], eps=0.0)).view(np.uint8)), d


@pytest.mark.parametrize("experts,k", [(1, 1), (31, 31), (33, 8), (128, 32), (129, 33), (1000, 32), (1024, 5)])
def test_route_sort_at_the_forms_edges(be, experts, k):
    rng = np.random.default_rng(experts)
    for rows in (1, 5, 130):
        p = rng.integers(-6, 7, (rows, experts)).astype(np.float32) / 4  # ties, zeros of both signs
        p[p == 0] *= rng.choice([1.0, -1.0], (p == 0).sum()).astype(np.float32)
        if experts > 30:
            p[0, 3], p[0, 17] = np.nan, np.nan
        idx, sc = nv.moe_route(be.up(p, nv.F32), k, normalize=False)
        want = np.argsort(p, axis=1, kind="stable")[:, experts - k:]
        assert np.array_equal(idx.to_numpy(), want), (rows, experts, k)
        assert np.array_equal(sc.to_numpy(), np.take_along_axis(p, want, 1), equal_nan=True)
        flat = rng.integers(0, experts, rows * k).astype(np.uint32)
        order, restore, tokens, srt, off = (a.to_numpy() for a in nv.moe_sort(be.up(flat.reshape(rows, k), nv.U32), experts))
        w = np.argsort(flat, kind="stable")
        assert np.array_equal(order, w) and np.array_equal(restore, np.argsort(w, kind="stable"))
        assert np.array_equal(tokens, w // k) and np.array_equal(srt, flat[w])
        assert np.array_equal(off, np.searchsorted(flat[w], np.arange(experts)))


@pytest.mark.parametrize("mode", [oracle.MXFP4, oracle.MXFP8, oracle.NVFP4])
def test_fp_codecs_with_extreme_values(be, mode):
    gs, bits = (16, 4) if mode == oracle.NVFP4 else (32, 8 if mode == oracle.MXFP8 else 4)
    rng = np.random.default_rng(5)
    w = rng.standard_normal((40, 3 * gs)).astype(np.float32) * 10.0 ** rng.integers(-38, 38, (40, 1)).astype(np.float32)
    w[0], w[1, 5], w[2, 7], w[3, :gs] = 0.0, np.nan, np.inf, 1e-42
    got = be.quantize(w, nv.F32, mode, gs, bits)
    want = oracle.quantize(w, oracle.F32, mode, gs, bits)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    for dt in ("f32", "bf16", "f16"):
        d = be.dequantize(got[0], got[1], None, NVC[dt], mode, gs, bits)
        o = oracle.dequantize(want[0], want[1], None, CODE[dt], mode, gs, bits)
        d, o = np.asarray(d).reshape(-1), np.asarray(o).reshape(-1)
        nan = np.isnan(oracle.to_f32(o, CODE[dt]))  # (which NaN a conversion to 16 bits writes is its own: any NaN will do)
        assert np.array_equal(np.isnan(oracle.to_f32(d, CODE[dt])), nan) and nan.sum() <= 2 * gs, dt
        assert np.array_equal(d[~nan].view(np.uint8), o[~nan].view(np.uint8)), dt


# ── many-row products: unit rows return columns of the dequantized matrix bit for bit ───────
FORMATS = [(oracle.AFFINE, b, g, dt) for b, g, dt in ((4, 64, "f16"), (4, 32, "bf16"), (8, 128, "f16"), (2, 64, "bf16"), (3, 64, "bf16"), (3, 32, "f16"),
                                                      (6, 64, "bf16"), (6, 128, "f16"), (8, 64, "bf16"))]
FORMATS += [(oracle.MXFP4, 4, 32, "bf16"), (oracle.MXFP8, 8, 32, "bf16"), (oracle.NVFP4, 4, 16, "bf16")]


def packed(rng, rows, K, fmt):
    mode, bits, gs, dt = fmt
    w = oracle.from_f32((rng.standard_normal((rows, K)) * 0.02).astype(np.float32), CODE[dt])
    q = oracle.quantize(w, CODE[dt], mode, gs, bits)
    c, s, b = (*q, None)[:3]
    return c, s, b, oracle.dequantize(c, s, b, CODE[dt], mode, gs, bits)


def unit(rng, M, K, dt):
    ks = rng.integers(0, K, M)
    x = np.zeros((M, K), np.float32)
    x[np.arange(M), ks] = 1.0
    return oracle.from_f32(x, CODE[dt]), ks


def same(got, want, dt):
    """Equal values (a weight of -0, which the floating-point codes have, sums with the row's zeros to +0)."""
    return np.array_equal(oracle.to_f32(got, CODE[dt]), oracle.to_f32(np.ascontiguousarray(want), CODE[dt]))


@pytest.mark.parametrize("fmt", FORMATS)
def test_many_rows_at_the_tiles_edges(be, fmt):
    """Around every token tile, one to 21 k-blocks (an odd number leaves half a stage), rows of scales on no boundary, N no
    multiple of 128, tiles cut along K, pairs of blocks."""
    mode, bits, gs, dt = fmt
    rng = np.random.default_rng(bits + gs)
    for M, N, K in ((9, 128, 128), (32, 130, 192), (33, 8, 1344), (64, 136, 4224), (65, 257, 128), (129, 260, 320), (160, 128, 1344), (161, 390, 576),
                    (193, 1160, 192), (300, 520, 2176), (1601, 2460, 1088), (2100, 2440, 64)):
        if K % gs:
            K = (K // gs + 1) * gs
        c, s, b, dense = packed(rng, N, K, fmt)
        x, ks = unit(rng, M, K, dt)
        got = be.quantized_matmul(x, c, s, b, CODE[dt], mode, gs, bits, True)
        assert same(got, dense[:, ks].T, dt), (M, N, K)


@pytest.mark.parametrize("fmt,shape", [(f, s) for f in FORMATS for s in SHAPES if s[2] % f[2] == 0 and s[0] * s[1] * s[2] < 10 ** 10])
def test_many_rows_in_every_plan(be, fmt, shape):
    """Every token tile, single blocks and pairs (198 x 9490: the last pair has weight rows for its first block only)."""
    mode, bits, gs, dt = fmt
    M, N, K = shape
    assert nv.Device.shared(0).info()["multiprocessors"] == 148  # (the plans of these shapes, see test_qmm_plan.py)
    rng = np.random.default_rng(bits + gs + M)
    c, s, b, dense = packed(rng, N, K, fmt)
    x, ks = unit(rng, M, K, dt)
    assert same(be.quantized_matmul(x, c, s, b, CODE[dt], mode, gs, bits, True), dense[:, ks].T, dt)


@pytest.mark.parametrize("fmt", [FORMATS[0], FORMATS[4], *FORMATS[-4:]])
def test_grouped_rows_at_the_schedules_edges(be, fmt):
    """Experts without rows, with one, with a tile and one more; fewer and more tiles than multiprocessors; more experts than the table holds."""
    mode, bits, gs, dt = fmt
    rng = np.random.default_rng(bits)
    for counts, N, K in (([0, 1, 129, 40, 300], 200, 192), ([700, 0, 0, 3], 1160, 320), ([33] * 40 + [0] * 24, 520, 128), ([2] * 600, 136, 64),
                         ([1] * 511 + [90], 128, 64)):
        if K % gs:
            K = (K // gs + 1) * gs
        E = len(counts)
        c, s, b, dense = packed(rng, E * N, K, fmt)
        dense = dense.reshape(E, N, K)
        rhs = np.repeat(np.arange(E), counts).astype(np.uint32)
        x, ks = unit(rng, len(rhs), K, dt)
        got = be.gather_qmm(x[:, None, :], c.reshape(E, N, -1), s.reshape(E, N, -1), b if b is None else b.reshape(E, N, -1), None, rhs, CODE[dt], mode, gs, bits,
                            True, None, True)
        assert same(got[:, 0], dense[rhs, :, ks], dt), (counts[:5], N, K)


@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_swiglu_of_every_16_bit_gate(be, dt):
    """The approximate sigmoid may only be used where it rounds like the exact one."""
    gate = np.arange(65536, dtype=np.uint16)
    if dt == "f16":
        gate = gate.view(np.float16)
    one = oracle.from_f32(np.ones(65536, np.float32), CODE[dt])
    for oai in (False, True):
        got = (nv.swiglu_oai if oai else nv.swiglu)(be.up(gate, NVC[dt]), be.up(one, NVC[dt])).to_numpy()
        g, w = (oracle.to_f32(a, CODE[dt]) for a in (np.asarray(got).view(np.uint16), np.asarray(oracle.swiglu(gate, one, CODE[dt], oai=oai)).view(np.uint16)))
        # (the host's and the device's expf may differ by 2^-23, which moves one float16 rounding in 2^11 at most: 32 of these)
        other = np.flatnonzero((g != w) & ~(np.isnan(g) & np.isnan(w)))
        assert len(other) <= (32 if dt == "f16" else 0), (oai, other[:8])
        assert np.all(np.abs(g[other] - w[other]) <= 2.0 ** -9 * np.abs(w[other]) + 2.0 ** -23), other[:8]


# ── few-row products: the staging of the activations, both block sizes ──────────────────────
@pytest.mark.parametrize("fmt", [f for f in FORMATS if f[3] == "bf16"])
def test_few_rows_staged_across_rows(be, fmt):
    """Every number of rows, K from one iteration to where a second block's activations no longer fit, rows on no 16-byte boundary."""
    mode, bits, gs, dt = fmt
    rng = np.random.default_rng(bits + gs)
    for N, K in ((33, 128), (16, 640), (250, 2048), (40, 6144)):
        c, s, b, dense = packed(rng, N, K, fmt)
        for M in (2, 3, 5, 8):
            x, ks = unit(rng, M, K, dt)
            got = be.quantized_matmul(x, c, s, b, CODE[dt], mode, gs, bits, True)
            assert same(got, dense[:, ks].T, dt), (M, N, K)
        flat = be.up(np.concatenate([np.zeros(3, x.dtype), x.reshape(-1)]), NVC[dt])  # the same rows, 6 bytes into an allocation
        got = host(nv.quantized_matmul(flat[3:].reshape(M, K), be.quantized(c, s, b, NVC[dt], mode, gs, bits)))
        assert same(got, dense[:, ks].T, dt), (N, K)


# ── reads ahead of the wait for the kernel in front ─────────────────────────────────────────
@pytest.mark.parametrize("path", ["few rows", "many rows", "gather", "grouped", "attention", "attention rows"])
def test_operands_that_the_kernels_in_front_have_just_written(be, path):
    """Weights, scales, lists and caches come from launches directly in front or one kernel further, into blocks that held
    other values a moment ago: the results are those with an idle stream before every launch, eagerly and recorded."""
    rng = np.random.default_rng(3)
    N, K, E = 96, 512, 8
    quant = nv.Quant.affine(64, 4)
    table = nv.quantize(be.up(oracle.from_f32(rng.standard_normal((8 * N, K)).astype(np.float32), oracle.BF16), nv.BF16), quant)
    picks = [be.up(rng.permutation(8 * N)[:4 * N].astype(np.uint32), nv.U32) for _ in range(6)]
    x = be.up(oracle.from_f32(rng.standard_normal((40, K)).astype(np.float32), oracle.BF16), nv.BF16)
    rows = 4 if path == "attention rows" else 1

    def step(pick, pause, between):
        parts = []
        for a in (table.scales, table.biases, table.weight):
            parts.append(nv.take_rows(a, pick))
            pause()
        q = nv.Quantized(parts[2], parts[0], parts[1], quant)
        h = x[:40 if path in ("many rows", "grouped") else 4]
        if between:  # a kernel that lets the product start before it has waited itself
            h = nv.rms_norm(h)
            pause()
        if path in ("few rows", "many rows"):
            y = nv.quantized_matmul(h, q)
        elif path in ("gather", "grouped"):
            experts = nv.Quantized(*(a.reshape(E, -1, a.shape[-1]) for a in (q.weight, q.scales, q.biases)), quant)
            probs = nv.quantized_matmul(h, nv.Quantized(q.weight[:E], q.scales[:E], q.biases[:E], quant))
            pause()
            idx, _ = nv.moe_route(probs, 2)
            pause()
            if path == "gather":
                y = nv.gather_qmm(h.reshape(4, 1, K), experts, lhs, idx)
            else:
                order, _, tokens, ids, offs = nv.moe_sort(idx, E)
                pause()
                mine = nv.take_rows(h, tokens)
                pause()
                y = nv.gather_qmm(mine.reshape(80, 1, K), experts, None, ids, nv.GatherQmm(sorted_indices=True), offs)
        else:
            heads = 2 if path == "attention" else 1  # 1536 or 3072 keys of 64
            k = nv.Quantized(*(a.reshape(1, heads, -1, a.shape[-1] // 8) for a in (q.weight, q.scales, q.biases)), quant)
            y = nv.quantized_attention(h[:rows].reshape(1, 8, rows, 64), k, k, 0.125)
        pause()
        return y, parts

    lhs = be.up(np.repeat(np.arange(4, dtype=np.uint32), 2).reshape(4, 2), nv.U32)
    for between in (False, True):
        want = [host(step(p, be.dev.synchronize, between)[0]) for p in picks]
        for _ in range(3):
            kept = [step(p, lambda: None, between) for p in picks]
            for (g, _), w in zip(kept, want):
                assert np.array_equal(host(g), w), (path, between, "eager")
        kept = []  # (the blocks go back to the pool, which cannot grow while recording)
        graph = be.dev.record(lambda: kept.extend(step(p, lambda: None, between) for p in picks))
        for _ in range(3):
            graph.launch()
            for (g, _), w in zip(kept, want):
                assert np.array_equal(host(g), w), (path, between, "recorded")
