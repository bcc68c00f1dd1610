"""Newton-Schulz GEMMs (tcgen05/TMEM/TMA) against the oracle with the same operand rounding.

Tolerances: intermediates after one GEMM differ only by FP32 accumulation order, so 16-bit
results may differ by one unit in the last place on a small fraction of entries; the full
single iteration is held to relative L2 <= 2e-3.  Over five iterations with the fixed
coefficient triple the map amplifies perturbations (|p'(s)| is about 1.6 inside the band the
singular values oscillate in), so two BF16 implementations that round at identical points but
accumulate in a different order already differ by about 1e-2: the five-iteration bound is
relative L2 <= 2e-2 (the stated tolerance of the path), with a loose sanity bound of 1e-1 of the
peak entry on the largest single-entry difference.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import llmini_b200 as b2
from llmini_b200 import _ffi
from oracle import oracle as o
from tests import _util as U
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
F = np.float32


def _x0(rng, rows, cols, fmt):
    x = (rng.standard_normal((rows, cols))).astype(F)
    x = x / (np.linalg.norm(x) * 1.01)
    return o.round_bf16(x) if fmt == b2.OPERAND_BF16 else x.astype(np.float16).astype(F)


def _run(shapes, fmt, iterations, coeffs, tile_n, xs, schedule=b2.NS_PER_PHASE):
    opt = b2.OptimizerModule()
    plan = b2.MuonPlan(shapes, operand_format=fmt, scale_layout=b2.SCALES_RAW, tile_n=tile_n, max_iterations=iterations,
                       ns_schedule=schedule)
    for i, x in enumerate(xs):
        t = plan.scratch(i, 0)
        t.copy_(dev(x).to(t.dtype))
    opt.muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=iterations, coefficients=coeffs))
    torch.cuda.synchronize()
    assert plan.status() == 0
    return plan


@pytest.mark.parametrize("schedule", [b2.NS_CHAINED, b2.NS_PER_PHASE, b2.NS_FUSED_GRAM_POLY])
@pytest.mark.parametrize("tile_n", [128, 256, 512])  # 512 = two-CTA 256 x 256 tiles
@pytest.mark.parametrize("fmt", [b2.OPERAND_BF16, b2.OPERAND_F16])
@pytest.mark.parametrize("rows,cols", [(64, 256), (256, 64), (128, 128), (96, 160), (160, 96), (320, 832), (832, 320)])
def test_single_iteration_intermediates(rows, cols, fmt, tile_n, schedule):
    rng = np.random.default_rng(rows * 7 + cols)
    x = _x0(rng, rows, cols, fmt)
    co = o.polar_express_coefficients(1) if fmt == b2.OPERAND_F16 else o.fixed_coefficients(1)
    plan = _run([(rows, cols)], fmt, 1, co, tile_n, [x], schedule)
    mode = o.ROUND_BF16 if fmt == b2.OPERAND_BF16 else o.ROUND_F16
    rnd = (lambda a: o.round_bf16(a)) if fmt == b2.OPERAND_BF16 else (lambda a: np.asarray(a, F).astype(np.float16).astype(F))
    xs = x if rows <= cols else np.ascontiguousarray(x.T)   # polar orientation [n][m]
    n = min(rows, cols)
    G = (xs.astype(np.float64) @ xs.T.astype(np.float64)).astype(F)
    g16 = host(plan.scratch(0, 5).float())
    ulp = 2.0 ** (-7 if fmt == b2.OPERAND_BF16 else -10)  # one unit in the last place of the 16-bit type
    tiny = 0.0 if fmt == b2.OPERAND_BF16 else 2.0 ** -24   # binary16 subnormal spacing
    assert np.all(np.abs(g16 - rnd(G)) <= 1.01 * ulp * np.abs(G) + 1e-6 * np.max(np.abs(G)) + tiny)
    assert np.mean(g16 != rnd(G)) < 0.02
    a, b, c = (F(v) for v in co[0])
    Gr = rnd(G).astype(np.float64)
    Q = (c * (Gr @ Gr) + b * G.astype(np.float64) + a * np.eye(n)).astype(F)
    q16 = host(plan.scratch(0, 6).float())
    assert np.all(np.abs(q16 - rnd(Q)) <= 3 * ulp * np.abs(Q) + 2e-5 * np.max(np.abs(Q)))
    want = o.polar(x, 1, co, round_mode=mode)
    got = host(plan.scratch(0, 1))
    assert U.rel_l2(got, want) <= 2e-3 and U.max_rel_to_peak(got, want) <= 2e-2
    plan.close()


@pytest.mark.parametrize("schedule", [b2.NS_CHAINED, b2.NS_PER_PHASE, b2.NS_FUSED_GRAM_POLY])
@pytest.mark.parametrize("tile_n", [0, 256])
@pytest.mark.parametrize("shapes", [
    [(768, 768), (768, 3072), (3072, 768), (2304, 768)],
    [(1600, 1600), (1600, 320), (48, 1600)],
])
def test_five_iterations_multi_slot(shapes, tile_n, schedule):
    rng = np.random.default_rng(len(shapes) * 97 + shapes[0][0])
    xs = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in shapes]
    co = o.fixed_coefficients(5)
    plan = _run(shapes, b2.OPERAND_BF16, 5, co, tile_n, xs, schedule)
    for i, x in enumerate(xs):
        want = o.polar(x, 5, co, round_mode=o.ROUND_BF16)
        got = host(plan.scratch(i, 1))
        assert np.isfinite(got).all()
        r2, mx = U.rel_l2(got, want), U.max_rel_to_peak(got, want)
        print(f"slot {shapes[i]}: rel_l2 {r2:.3e} max/peak {mx:.3e}")
        assert r2 <= 2e-2 and mx <= 1e-1
        # orthogonality sanity: the bulk of the singular values sits in the Newton-Schulz band
        sv = np.linalg.svd(got.astype(np.float64), compute_uv=False)
        assert sv.max() < 1.6 and np.median(sv) > 0.5
    plan.close()


@pytest.mark.parametrize("tile_n", [0, 128, 256])
@pytest.mark.parametrize("shapes", [
    [(768, 768), (768, 3072), (3072, 768), (2304, 768), (0, 0), (768, 768)],
    [(1600, 1600), (1600, 320), (48, 1600), (4800, 1600)],
    [(64, 64)],
    # 13 x 13 pair tiles = 91 Gram tiles, more than the device runs CTA pairs at once: the fused form must step
    # aside (a pair waiting for tiles that no resident pair can take would wait for ever)
    [(3328, 3328), (256, 512)],
])
def test_chained_launch_equals_the_per_phase_launches_bit_for_bit(shapes, tile_n):
    # The chained launch runs the same tiles with the same k order as the fifteen per-phase launches; only the
    # ordering between tiles differs (per-matrix progress counts instead of launch boundaries), so every
    # intermediate and the result must be identical, and its progress words must be zero again afterwards.
    rng = np.random.default_rng(31 + len(shapes))
    xs = [_x0(rng, r, c, b2.OPERAND_BF16) if r * c else np.zeros((0, 0), F) for r, c in shapes]
    co = o.fixed_coefficients(5)
    live = [(i, x) for i, x in enumerate(xs) if x.size]

    def run(schedule):
        opt = b2.OptimizerModule()
        plan = b2.MuonPlan(shapes, scale_layout=b2.SCALES_RAW, tile_n=tile_n, ns_schedule=schedule)
        for i, x in live:
            t = plan.scratch(i, 0)
            t.copy_(dev(x).to(t.dtype))
        for _ in range(2):   # twice: the second run starts from the words the first one left
            for i, x in live:
                t = plan.scratch(i, 0)
                t.copy_(dev(x).to(t.dtype))
            opt.muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=5, coefficients=co))
        torch.cuda.synchronize()
        assert plan.status() == 0
        assert not host(plan.scratch(0, 11)).any()
        out = [[host(plan.scratch(i, w).float()).copy() for w in (1, 5, 6, 7)] for i, _ in live]
        plan.close()
        return out

    b = run(b2.NS_PER_PHASE)
    # (the fused Gram + polynomial form draws its tiles the same way and keeps the FP32 Gram tile in tensor memory
    # instead of reading it back: the same arithmetic again)
    for schedule in (b2.NS_CHAINED, b2.NS_FUSED_GRAM_POLY):
        a = run(schedule)
        for (i, _), ra, rb in zip(live, a, b):
            for w, ta, tb in zip(("U", "Gram", "Q", "X1"), ra, rb):
                assert np.array_equal(ta, tb), (schedule, shapes[i], w)


def test_steps_with_fewer_iterations_take_the_per_phase_launches():
    # a plan made for five iterations asked for three: the chained list does not apply, the result must not change
    rng = np.random.default_rng(5)
    shapes = [(256, 512), (512, 256)]
    xs = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in shapes]
    co = o.fixed_coefficients(3)
    plan = _run(shapes, b2.OPERAND_BF16, 3, co, 0, xs, b2.NS_CHAINED)                     # max_iterations = 3: chained
    plan5 = b2.MuonPlan(shapes, scale_layout=b2.SCALES_RAW, ns_schedule=b2.NS_CHAINED)     # made for 5: per phase for 3
    for i, x in enumerate(xs):
        t = plan5.scratch(i, 0)
        t.copy_(dev(x).to(t.dtype))
    b2.OptimizerModule().muon_polar(plan5, b2.MuonMegaUpdateArgs(iterations=3, coefficients=co))
    torch.cuda.synchronize()
    for i in range(len(shapes)):
        assert torch.equal(plan.scratch(i, 1), plan5.scratch(i, 1))
    plan.close()
    plan5.close()


SMALL = [(16, 16), (64, 64), (128, 128), (128, 512), (512, 128), (100, 112), (129, 128), (127, 144), (512, 16), (16, 512),
         (1, 496), (384, 80), (65, 64), (128, 48), (80, 448)]   # one SM holds each of them


@pytest.mark.parametrize("fmt", [b2.OPERAND_BF16, b2.OPERAND_F16])
@pytest.mark.parametrize("iterations,deferred,update16", [(1, False, False), (2, False, True), (5, False, False), (5, True, True)])
def test_one_cta_loop_equals_the_per_phase_launches_bit_for_bit(fmt, iterations, deferred, update16):
    """Plans whose matrices all fit one SM take the one-CTA loop; a forced tile shape keeps the launches per phase."""
    if deferred and fmt == b2.OPERAND_F16:   # an un-normalised update can leave F16's range
        with pytest.raises(b2.B2Error):
            b2.MuonPlan(SMALL, operand_format=fmt, scale_layout=b2.SCALES_RAW, normalize_mode=b2.NORMALIZE_DEFERRED)
        return
    rng = np.random.default_rng(iterations)
    shapes = SMALL[:7] + [(0, 0)] + SMALL[7:]
    live = [(i, s) for i, s in enumerate(shapes) if s[0]]
    xs = {i: _x0(rng, r, c, fmt) for i, (r, c) in live}
    co = o.polar_express_coefficients(iterations) if fmt == b2.OPERAND_F16 else o.fixed_coefficients(iterations)
    results = []
    for tile_n in (0, 128):
        plan = b2.MuonPlan(shapes, operand_format=fmt, scale_layout=b2.SCALES_RAW, tile_n=tile_n, max_iterations=iterations,
                           normalize_mode=b2.NORMALIZE_DEFERRED if deferred else b2.NORMALIZE_TWO_PASS,
                           update_input=b2.UPDATE_16BIT if update16 else b2.UPDATE_F32)
        for i, (r, c) in live:
            for w in (0, 1, 5, 6, 7):
                plan.scratch(i, w).zero_()
            plan.scratch(i, 0).copy_(dev(xs[i]).to(plan.scratch(i, 0).dtype))
            plan.scratch(i, 2).view(torch.float32).fill_(0.75)   # read by a one-pass plan only
        b2.OptimizerModule().muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=iterations, coefficients=co))
        torch.cuda.synchronize()
        assert plan.status() == 0
        results.append([[host(plan.scratch(i, w).float()).copy() for w in (0, 1, 5, 6, 7)] for i, _ in live])
    for (_, shape), a, b in zip(live, *results):
        for w, u, v in zip(("operand 0", "U", "G", "Q", "operand 1"), a, b):
            assert np.array_equal(u, v), (shape, w, float(np.abs(u - v).max()))


@pytest.mark.parametrize("fmt,update16", [(b2.OPERAND_BF16, False), (b2.OPERAND_F16, True)])
def test_one_cta_loop_at_the_edges_of_its_units(fmt, update16):
    """G and Q in units of 32 x 32, results in blocks of 128: one and two units, three, a row beyond, a last block of 16."""
    shapes = [(32, 32), (33, 64), (96, 96), (31, 160), (257, 112), (400, 32), (48, 384), (64, 272), (112, 512), (512, 96)]
    rng = np.random.default_rng(4)
    xs = [_x0(rng, r, c, fmt) for r, c in shapes]
    results = []
    for tile_n in (0, 128):
        plan = b2.MuonPlan(shapes, operand_format=fmt, scale_layout=b2.SCALES_RAW, tile_n=tile_n, max_iterations=4,
                           update_input=b2.UPDATE_16BIT if update16 else b2.UPDATE_F32)
        for i, x in enumerate(xs):
            plan.scratch(i, 0).copy_(dev(x).to(plan.scratch(i, 0).dtype))
        b2.OptimizerModule().muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=4, coefficients=o.fixed_coefficients(4)))
        torch.cuda.synchronize()
        assert plan.status() == 0
        results.append([[host(plan.scratch(i, w).float()).copy() for w in ((0, 5, 6, 7) if update16 else (1, 5, 6, 7))] for i in range(len(shapes))])
        plan.close()
    for shape, a, b in zip(shapes, *results):
        for u, v in zip(a, b):
            assert np.array_equal(u, v), shape



@pytest.mark.parametrize("fmt", [b2.OPERAND_BF16, b2.OPERAND_F16])
@pytest.mark.parametrize("kind", ["nan", "inf", "overflow"])
def test_one_cta_loop_treats_non_finite_values_as_the_per_phase_launches_do(kind, fmt):
    rng = np.random.default_rng(1)
    xs = [_x0(rng, r, c, fmt) for r, c in SMALL]
    for x in xs:
        if kind == "overflow":
            x *= F(3e4 if fmt == b2.OPERAND_F16 else 1e30)   # the Gram matrix leaves the operand type's range
        else:
            x[x.shape[0] // 2, x.shape[1] // 2] = F(kind)
    for iterations in (1, 2):
        a, b = (_run(SMALL, fmt, iterations, o.fixed_coefficients(iterations), tile_n, xs) for tile_n in (0, 128))
        for i, shape in enumerate(SMALL):
            for w, name in (1, "U"), (5, "G"), (6, "Q"):
                assert np.array_equal(host(a.scratch(i, w).float()), host(b.scratch(i, w).float()), equal_nan=True), (shape, name)
        a.close()
        b.close()


def test_tile_choice_agrees_with_the_oracle_on_both_sides_of_the_line():
    """One layer of width 512 takes 128 x 128 tiles, three of width 768 take pairs; mixed with odd row counts."""
    rng = np.random.default_rng(3)
    for shapes in ([(1536, 512), (333, 512)], [(2304, 768)] * 9 + [(701, 768)]):
        xs = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in shapes]
        plan = _run(shapes, b2.OPERAND_BF16, 1, o.fixed_coefficients(1), 0, xs)
        for i in (0, len(shapes) - 1):
            x = xs[i].astype(np.float64)
            n_major = x if shapes[i][0] <= shapes[i][1] else x.T
            a, b, c = (float(v) for v in o.fixed_coefficients(1)[0])
            g = n_major @ n_major.T
            u = (a * np.eye(len(g)) + b * g + c * g @ g) @ n_major
            u = u if shapes[i][0] <= shapes[i][1] else u.T
            got = host(plan.scratch(i, 1)).reshape(shapes[i])
            # G, Q and X are BF16 operands (2^-9 relative each); Q is dominated by its rounded diagonal
            assert np.linalg.norm(got - u) <= 4.0 * 2.0 ** -9 * np.linalg.norm(u)


@pytest.mark.parametrize("deferred", [False, True])
@pytest.mark.parametrize("shapes", [
    [(3072, 768)],                              # 36 Gram tiles of 128 x 128, each 48 k-blocks
    [(77, 1040), (1999, 64), (130, 16)],        # ragged everywhere
    [(200, 1536)],                              # wide, tiles clipped in both directions
])
def test_few_gram_tiles_with_a_long_k(shapes, deferred):
    """One iteration of 128 x 128 tiles, launch after launch, against FP64: every phase from the operands it has read."""
    rng = np.random.default_rng(17)
    xs = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in shapes]
    s = 0.75 if deferred else 1.0
    ca, cb, cc = (float(v) for v in o.fixed_coefficients(1)[0])
    plan = b2.MuonPlan(shapes, scale_layout=b2.SCALES_RAW, tile_n=128, max_iterations=1,
                       normalize_mode=b2.NORMALIZE_DEFERRED if deferred else b2.NORMALIZE_TWO_PASS)
    first = None
    for _ in range(3):
        for i, x in enumerate(xs):
            plan.scratch(i, 0).copy_(dev(x).to(torch.bfloat16))
            plan.scratch(i, 2).view(torch.float32).fill_(0.75)   # read by a one-pass plan only
            plan.scratch(i, 5).zero_()
        b2.OptimizerModule().muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=1, coefficients=o.fixed_coefficients(1)))
        torch.cuda.synchronize()
        assert plan.status() == 0
        got = [[host(plan.scratch(i, w).float()).copy() for w in (5, 6, 1)] for i in range(len(shapes))]
        if first is not None:   # every launch gives the same bits
            assert all(np.array_equal(u, v) for a, b in zip(first, got) for u, v in zip(a, b))
        first = got
    half_ulp, eps = 2.0 ** -8, 2.0 ** -24   # one rounding to BF16: half a unit in the last place, 2^-9 .. 2^-8 relative
    for x, (r, c), (g16, q16, u) in zip(xs, shapes, got):
        n = min(r, c)
        xd = (x if r <= c else x.T).astype(np.float64)
        G = xd @ xd.T * s * s
        g16, q16 = (v.reshape(n, -1)[:, :n].astype(np.float64) for v in (g16, q16))
        # FP32 sums of max(r, c) products, the scaling included
        g_sum = (max(r, c) + 2) * eps * s * s * (np.abs(xd) @ np.abs(xd).T)
        assert np.all(np.abs(g16 - G) <= half_ulp * np.abs(G) + g_sum)
        # Q = c G16 G16 + b G + a I: FP32 sums of n products and two fused multiply-adds, then one rounding to BF16
        Q = cc * (g16 @ g16) + cb * G + ca * np.eye(n)
        q_sum = (n + 4) * eps * (abs(cc) * (np.abs(g16) @ np.abs(g16)) + abs(cb) * np.abs(G) + abs(ca)) + abs(cb) * g_sum
        assert np.all(np.abs(q16 - Q) <= half_ulp * (np.abs(Q) + q_sum) + q_sum)
        want = s * (q16 @ xd)
        got_u = (u.reshape(r, c) if r <= c else u.reshape(r, c).T).astype(np.float64)
        assert np.all(np.abs(got_u - want) <= (n + 2) * eps * s * (np.abs(q16) @ np.abs(xd)))


@pytest.mark.parametrize("fmt,deferred", [(b2.OPERAND_BF16, True), (b2.OPERAND_F16, False)])
@pytest.mark.parametrize("shapes", [
    [(130, 528)],                                        # K of 9 and 3 k-blocks: the last stage of two is half full
    [(129, 144), (144, 256), (2000, 16)],                # one row or 16 columns into the second tile; one k-block
    [(1000, 1040), (77, 1040), (200, 208), (48, 1600)],  # rows no multiple of 8, 16 or 64; columns not of 64
    [(960, 320), (320, 320), (1280, 320), (320, 1280)],  # MN-major on one side, K-major on the other
    [(768, 768)] * 3 + [(3072, 768)],                    # 144 tiles, just within one wave of CTAs; Apply in 256 x 256
])
def test_small_pair_tiles_equal_one_cta_tiles_bit_for_bit(shapes, fmt, deferred):
    """Plans of few tiles take the pairs' 128 x 128 for Gram and polynomial, and some for Apply; a sum runs over K in the
    same order in every shape."""
    rng = np.random.default_rng(sum(r for r, _ in shapes))
    xs = [_x0(rng, r, c, fmt) for r, c in shapes]
    results = []
    for tile_n in (0, 128):
        plan = b2.MuonPlan(shapes, operand_format=fmt, scale_layout=b2.SCALES_RAW, tile_n=tile_n, max_iterations=3,
                           normalize_mode=b2.NORMALIZE_DEFERRED if deferred else b2.NORMALIZE_TWO_PASS)
        for i, x in enumerate(xs):
            plan.scratch(i, 0).copy_(dev(x).to(plan.scratch(i, 0).dtype))
            plan.scratch(i, 2).view(torch.float32).fill_(0.75)   # read by a one-pass plan only
        b2.OptimizerModule().muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=3, coefficients=o.fixed_coefficients(3)))
        torch.cuda.synchronize()
        assert plan.status() == 0
        results.append([[host(plan.scratch(i, w).float()).copy() for w in (5, 6, 7, 1)] for i in range(len(shapes))])
        plan.close()
    for shape, a, b in zip(shapes, *results):
        for w, u, v in zip(("Gram", "Q", "X1", "U"), a, b):
            assert np.isfinite(u).all() and np.array_equal(u, v), (shape, w)


def _tiles(shapes, tile_n, fmt):
    """(tile of Gram and polynomial, by a pair of CTAs, triangle of tiles, tile of Apply, by a pair) that a plan takes."""
    n = len(shapes)
    opt = _ffi.MuonOptions(fmt, b2.SCALES_RAW, 0, 3, tile_n)
    out = (C.c_uint32 * 7)()
    rows, cols = (C.c_uint32 * n)(*[r for r, _ in shapes]), (C.c_uint32 * n)(*[c for _, c in shapes])
    assert b2.lib().b2_debug_muon_tiles(rows, cols, n, C.byref(opt), out) == 0
    return (out[0], out[1]), bool(out[2]), bool(out[3]), (out[4], out[5]), bool(out[6])


@pytest.mark.parametrize("fmt", [b2.OPERAND_BF16, b2.OPERAND_F16])
@pytest.mark.parametrize("shapes,apply", [
    ([(1920, 640), (640, 640), (2560, 640), (640, 2560)], ((128, 128), True)),      # whole tiles
    ([(650, 656)] * 3, ((128, 128), False)),                                        # ten rows into the last tile, no multiple of 8
    ([(1001, 1040), (700, 1200)], ((128, 128), False)),                             # an odd row count: G and Q have padding columns
    ([(645, 656), (1300, 656), (645, 1312), (2000, 656)], ((256, 256), True)),      # both sides ragged
])
def test_triangles_of_small_pair_tiles_equal_full_one_cta_tiles_bit_for_bit(shapes, apply, fmt):
    """Beyond one wave the pairs' 128 x 128 tiles leave out what lies below the diagonal and store it as transposes, 64 rows a
    CTA with their columns in two halves of the lanes."""
    assert _tiles(shapes, 0, fmt) == ((128, 128), True, True, *apply)
    assert _tiles(shapes, 128, fmt) == ((128, 128), False, False, (128, 128), False)
    rng = np.random.default_rng(sum(r for r, _ in shapes))
    xs = [_x0(rng, r, c, fmt) for r, c in shapes]
    results = []
    for tile_n in (0, 128):
        plan = b2.MuonPlan(shapes, operand_format=fmt, scale_layout=b2.SCALES_RAW, tile_n=tile_n, max_iterations=3)
        for i, x in enumerate(xs):
            plan.scratch(i, 0).copy_(dev(x).to(plan.scratch(i, 0).dtype))
        b2.OptimizerModule().muon_polar(plan, b2.MuonMegaUpdateArgs(iterations=3, coefficients=o.fixed_coefficients(3)))
        torch.cuda.synchronize()
        assert plan.status() == 0
        results.append([[host(plan.scratch(i, w).float()).copy() for w in (5, 6, 7, 1)] for i in range(len(shapes))])
        plan.close()
    for shape, a, b in zip(shapes, *results):
        for w, u, v in zip(("Gram", "Q", "X1", "U"), a, b):
            assert np.isfinite(u).all() and np.array_equal(u, v), (shape, w)


@pytest.mark.parametrize("company", [
    [(512, 256), (256, 256), (256, 1024), (384, 128)],   # few more tiles of 128 x 128
    [(64, 64)],
    [(768, 768)] * 5,
    [(2304, 768)] * 9,                                   # two-CTA tiles
])
@pytest.mark.parametrize("shape", [(768, 256), (512, 256), (384, 128), (3072, 768), (200, 1536), (77, 1040)])
def test_result_of_a_matrix_does_not_depend_on_its_company(shape, company):
    """A rank of a sharded run and a single GPU compute the same bits: whatever tiles a plan takes for the matrices it
    holds, every sum runs over K in one order."""
    rng = np.random.default_rng(shape[0])
    x = _x0(rng, *shape, b2.OPERAND_BF16)
    others = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in company]
    results = []
    for at, shapes, xs in ((0, [shape], [x]), (0, [shape] + company, [x] + others), (len(company), company + [shape], others + [x])):
        plan = _run(shapes, b2.OPERAND_BF16, 5, o.fixed_coefficients(5), 0, xs)
        results.append([host(plan.scratch(at, w).float()).copy() for w in (1, 5, 6, 7)])
        plan.close()
    for other in results[1:]:
        for w, a, b in zip(("U", "Gram", "Q", "X1"), results[0], other):
            assert np.array_equal(a, b), (w, float(np.abs(a - b).max()))


def test_one_cta_loop_with_more_matrices_than_sms():
    rng = np.random.default_rng(9)
    shapes = [(64, 96), (96, 64), (128, 256)] * 110   # 330 CTAs, more than two waves of one per SM
    xs = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in shapes[:3]]
    results = []
    for tile_n in (0, 128):
        plan = _run(shapes, b2.OPERAND_BF16, 5, o.fixed_coefficients(5), tile_n, [xs[i % 3] for i in range(len(shapes))])
        results.append([host(plan.scratch(i, 1)).copy() for i in range(len(shapes))])
    for i, (a, b) in enumerate(zip(*results)):
        assert np.array_equal(a, b) and np.array_equal(a, results[0][i % 3]), i


def test_a_plan_made_later_leaves_an_earlier_one_working():
    """Plans of the one-CTA loop need 116 to 193 KB of shared memory; the kernel's limit is one for all of them."""
    rng = np.random.default_rng(2)
    shapes = [(128, 512), (64, 64)]
    xs = [_x0(rng, r, c, b2.OPERAND_BF16) for r, c in shapes]
    args = b2.MuonMegaUpdateArgs(coefficients=o.fixed_coefficients(5))
    plans = [b2.MuonPlan([s], scale_layout=b2.SCALES_RAW) for s in shapes]   # the largest first, both alive
    for plan, x, s in zip(plans, xs, shapes):
        plan.scratch(0, 0).copy_(dev(x).to(torch.bfloat16))
        b2.OptimizerModule().muon_polar(plan, args)
        torch.cuda.synchronize()
        assert plan.status() == 0
        alone = _run([s], b2.OPERAND_BF16, 5, o.fixed_coefficients(5), 128, [x])   # per phase
        assert torch.equal(plan.scratch(0, 1), alone.scratch(0, 1))
