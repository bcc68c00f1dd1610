"""NVFP4 quantiser on the GPU against the oracle: bit-exact codes, block scales, tensor scale."""
import numpy as np
import pytest
import torch

import llmini_b200 as b2
from oracle import oracle as o
from tests import _util as U
from tests.gpu_util import dev, host, rcp_table

pytestmark = pytest.mark.gpu
F = np.float32


def _quantize_gpu(x, layout, rows=None, k=None):
    q = b2.Nvfp4QuantModule()
    n = x.size
    xd = dev(x)
    chunk = torch.zeros((n + 2047) // 2048, device="cuda")
    amax = torch.zeros(1, device="cuda")
    q.tensor_amax_f32(xd, chunk, amax, n)
    fp4 = torch.zeros(n // 2, dtype=torch.uint8, device="cuda")
    if layout == b2.SCALES_CSF:
        scales = b2.zero_scales(rows, k)
    else:
        scales = torch.zeros(n // 16, dtype=torch.uint8, device="cuda")
    gs = torch.zeros(1, device="cuda")
    q.fp32_to_nvfp4_four_six(xd, amax, fp4, scales, gs, n // 16, layout)
    torch.cuda.synchronize()
    return host(fp4), host(scales), host(gs)[0], host(amax)[0], host(chunk)


def test_abi_handshake():
    b2.OptimizerModule().verify_storage_layout()


def test_known_sixteen_values():
    # crates/cuda-kernels/tests/nvfp4_quant.rs:21-53
    x = np.array([-3.25, -2.0, -1.25, -0.5, -0.125, 0.0, 0.25, 0.75, 1.0, 1.5, 2.25, 3.0, 4.0, 5.0, 6.5, 8.0], F)
    fp4, scales, gs, amax, _ = _quantize_gpu(x, b2.SCALES_RAW)
    assert amax == 8.0 and abs(gs - F(8.0) / F(1536.0)) <= 1e-8
    assert fp4.any() and scales.any()
    codes, sc, ogs, _ = o.nvfp4_quantize(x, rcp_table=rcp_table(gs))
    assert np.array_equal(fp4, codes) and np.array_equal(scales, sc) and gs == ogs


def test_negative_underflow_keeps_sign_nibble():
    # values that round to zero keep their sign bit (code 0x8), as the oracle assumes
    x = np.zeros(16, F)
    x[0], x[1], x[2], x[3], x[15] = -1e-9, -0.0, 1e-9, -0.2, 6.0
    fp4, scales, gs, _, _ = _quantize_gpu(x, b2.SCALES_RAW)
    codes, sc, _, _ = o.nvfp4_quantize(x, rcp_table=rcp_table(gs))
    assert np.array_equal(fp4, codes), (fp4, codes)
    assert np.array_equal(scales, sc)


@pytest.mark.parametrize("rows,k,layout", [
    (256, 4096, b2.SCALES_CSF), (1024, 4096, b2.SCALES_CSF), (3072, 768, b2.SCALES_CSF),
    (129, 256, b2.SCALES_CSF), (1, 4096, b2.SCALES_CSF), (1, 128, b2.SCALES_CSF),
    (7, 48, b2.SCALES_RAW), (1600, 1600, b2.SCALES_RAW), (1, 16, b2.SCALES_RAW), (4096, 4096, b2.SCALES_CSF),
])
def test_flat_quantiser_bit_exact(rows, k, layout):
    rng = np.random.default_rng(rows * 131 + k)
    x = U.with_outliers(rng, U.weights(rng, rows * k))
    fp4, scales, gs, amax, chunk = _quantize_gpu(x, layout, rows, k)
    assert amax == np.max(np.abs(x))
    want_chunks = np.array([np.max(np.abs(x[i:i + 2048])) for i in range(0, x.size, 2048)], F)
    assert np.array_equal(chunk, want_chunks)
    codes, raw, ogs, misses = o.nvfp4_quantize(x, amax=amax, rcp_table=rcp_table(gs))
    assert misses == 0 and gs == ogs
    assert np.array_equal(fp4, codes)
    got_raw = scales if layout == b2.SCALES_RAW else o.csf_decode_matrix(scales, rows, k)
    assert np.array_equal(got_raw, raw)
    if layout == b2.SCALES_CSF:  # whole storage, header and padding included
        assert np.array_equal(scales, o.csf_encode(raw, rows, k))
    # the optimised kernel equals the literal one-thread-per-group transcription bit for bit
    q = b2.Nvfp4QuantModule()
    l4, ls, lg = q.debug_quantize_literal(dev(x), dev(np.array([amax], F)))
    assert np.array_equal(host(l4), fp4) and np.array_equal(host(ls), raw) and host(lg)[0] == gs
    # The oracle on its own, with the correctly rounded reciprocal in place of the device's `rcp.approx.ftz`:
    # a result can differ only where v * inv sits within an ulp of an E2M1 rounding boundary, or the block
    # maximum within an ulp of an E4M3 tie.  Measured: 1 code in 16.7 M values, no scale byte.  Held here at
    # two codes per 2^24 values (rounded up to a whole value for small tensors) and no scale byte.
    c2, r2, _, _ = o.nvfp4_quantize(x, amax=amax)
    code_diff = int(np.count_nonzero((c2 & 0xF) != (codes & 0xF)) + np.count_nonzero((c2 >> 4) != (codes >> 4)))
    scale_diff = int(np.count_nonzero(r2 != raw))
    print(f"exact-rcp mismatches: codes {code_diff} scales {scale_diff} of {x.size}")
    assert code_diff <= 2 * -(-x.size // (1 << 24)) and scale_diff == 0


def test_all_zero_tensor_and_empty():
    x = np.zeros(4096, F)
    fp4, scales, gs, amax, _ = _quantize_gpu(x, b2.SCALES_RAW)
    assert gs == 1.0 and amax == 0.0 and not fp4.any() and not scales.any()
    q = b2.Nvfp4QuantModule()
    g = torch.zeros(1, device="cuda")
    q.fp32_to_nvfp4_four_six(dev(x), dev(np.zeros(1, F)), torch.zeros(8, dtype=torch.uint8, device="cuda"),
                             torch.zeros(8, dtype=torch.uint8, device="cuda"), g, 0, b2.SCALES_RAW)
    torch.cuda.synchronize()
    assert host(g)[0] == 1.0


def test_materialize_master_and_schedule_free():
    rng = np.random.default_rng(5)
    rows, k = 384, 1024
    n = rows * k
    z, x = U.weights(rng, n), U.weights(rng, n)
    opt = b2.OptimizerModule()
    t = b2.Nvfp4Tensor.empty(rows, k)
    amax, chunk = torch.zeros(1, device="cuda"), torch.zeros(n // 2048, device="cuda")
    opt.materialize_master(t.bytes, t.scales, t.global_scale, dev(x), amax, chunk, n)
    torch.cuda.synchronize()
    gs = host(t.global_scale)[0]
    codes, raw, ogs, _ = o.nvfp4_quantize(x, rcp_table=rcp_table(gs))
    assert gs == ogs and np.array_equal(host(t.bytes), codes)
    assert np.array_equal(host(t.scales), o.csf_encode(raw, rows, k))

    beta = 0.4
    y, am = o.schedule_free_values(z, x, beta)
    t2 = b2.Nvfp4Tensor.empty(rows, k)
    amax2 = torch.full((1,), 123.0, device="cuda")
    kw = dict(bytes=t2.bytes, scales=t2.scales, global_scale=t2.global_scale, z_master=dev(z), x_master=dev(x),
              amax=amax2, len=n, scale_rows=rows, scale_k=k, beta=beta)
    opt.materialize_schedule_free(**kw)
    torch.cuda.synchronize()
    assert host(amax2)[0] == am
    gs2 = host(t2.global_scale)[0]
    codes2, raw2, ogs2, _ = o.nvfp4_quantize(y, amax=am, rcp_table=rcp_table(gs2))
    assert gs2 == ogs2 and np.array_equal(host(t2.bytes), codes2)
    assert np.array_equal(host(t2.scales), o.csf_encode(raw2, rows, k))
    # precomputed values + cached amax (the production per-step requant): same bits
    t3 = b2.Nvfp4Tensor.empty(rows, k)
    kw.update(bytes=t3.bytes, scales=t3.scales, global_scale=t3.global_scale, precomputed_values=dev(y))
    opt.materialize_schedule_free_precomputed(**kw)
    torch.cuda.synchronize()
    assert np.array_equal(host(t3.bytes), codes2) and np.array_equal(host(t3.scales), host(t2.scales))
    # on-the-fly values from z, x with the cached amax
    t4 = b2.Nvfp4Tensor.empty(rows, k)
    kw.update(bytes=t4.bytes, scales=t4.scales, global_scale=t4.global_scale, precomputed_values=None)
    opt.materialize_schedule_free_precomputed(**kw)
    torch.cuda.synchronize()
    assert np.array_equal(host(t4.bytes), codes2)
    with pytest.raises(b2.B2Error):   # a negative SymExpLin beta is an argument error
        kw.update(symexp_lin_beta=-0.5)
        opt.materialize_schedule_free(**kw)
    # SymExpLin with explicit scale scalars against its definition (symexp_lin.rs:8-26); exp() here is
    # the exact one, the device uses ex2.approx: values agree to a few ulp, so compare dequantised
    kw.update(symexp_lin_beta=4.0)
    one = lambda v: torch.full((1,), v, device="cuda")
    sc = [one(1.25), one(0.75), one(0.5), one(1.5), one(2.0), one(1.0)]   # (z, x) of exponential, linear, curvature
    kw.update(symexp_lin_scales=sc)
    opt.materialize_schedule_free(**kw)
    torch.cuda.synchronize()
    e_, l_, c_ = [zz + beta * (xx - zz) for zz, xx in ((1.25, 0.75), (0.5, 1.5), (2.0, 1.0))]
    y64 = y.astype(np.float64)
    want = np.sign(y64) * (e_ * (np.exp(4.0 * c_ * np.abs(y64)) - 1.0) / 4.0 + l_ * y64 / 4.0)
    assert abs(host(amax2)[0] - np.max(np.abs(want))) <= 1e-5 * np.max(np.abs(want))
    deq = o.nvfp4_dequantize(host(t4.bytes), o.csf_decode_matrix(host(t4.scales), rows, k), host(t4.global_scale)[0])
    assert np.max(np.abs(deq - want)) <= 0.26 * np.max(np.abs(want))   # an E2M1 step at the top of the range
    assert np.corrcoef(deq, want)[0, 1] > 0.99


def test_quantise_round_trip_property_large():
    # size-independent property at a bandwidth-sweep shape: |dequant - x| <= half a code step
    rows, k = 16384, 4096
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(rows * k, device="cuda", generator=g) * 0.02
    q = b2.Nvfp4QuantModule()
    chunk, amax = torch.zeros(rows * k // 2048, device="cuda"), torch.zeros(1, device="cuda")
    q.tensor_amax_f32(x, chunk, amax, rows * k)
    t = b2.Nvfp4Tensor.empty(rows, k, b2.SCALES_RAW)
    q.fp32_to_nvfp4_four_six(x, amax, t.bytes, t.scales, t.global_scale, rows * k // 16, b2.SCALES_RAW)
    torch.cuda.synchronize()
    assert amax.item() == x.abs().max().item()
    lut = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, -0., -.5, -1, -1.5, -2, -3, -4, -6], device="cuda")
    codes = torch.stack([t.bytes & 15, t.bytes >> 4], dim=1).reshape(-1).long()
    sc = t.scales.view(torch.float8_e4m3fn).float().repeat_interleave(16)
    deq = lut[codes] * sc * t.global_scale
    # per element: error at most half the largest code gap (2 at the top of the grid) times its scale,
    # plus the E4M3 rounding of the block scale (relative 2^-4) on the block maximum
    bound = sc * t.global_scale * 1.0 + 1e-12
    blockmax = x.abs().view(-1, 16).max(dim=1).values.repeat_interleave(16)
    assert bool(((deq - x).abs() <= bound + blockmax * 0.07).all())


def test_long_tensors_in_interleaved_runs_bit_exact():
    """Where a CTA's share is 64 chunks or more it takes runs of 16 chunks, interleaved with the others': 16 CTAs (of 128
    threads, more never fit) on every SM have 64 each here, and the last runs are uneven and end in a part of a chunk."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (sms * 16 * 64 + 5) * 2048 + 48
    x = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).mul_(0.02)
    q = b2.Nvfp4QuantModule()
    amax = x.abs().max().reshape(1)
    got = [torch.full((s,), 255, dtype=torch.uint8, device="cuda") for s in (n // 2, n // 16)] + [torch.zeros(1, device="cuda")]
    q.fp32_to_nvfp4_four_six(x, amax, *got, n // 16, b2.SCALES_RAW)
    want = q.debug_quantize_literal(x, amax)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b.view_as(a))


@pytest.mark.parametrize("chunks,tail", [(1, 0), (0, 16), (1, 48), (1279, 2032), (1280, 16), (6143, 2032), (6144, 16)])
def test_one_tensor_calls_equal_their_parts(chunks, tail):
    """Maximum and encode of one tensor as a chain of launches, up to 1280 chunks of 2048 values (schedule-free pairs up to 6144,
    with the transform all): the same bits as the maximum and the quantiser called one after the other."""
    n = chunks * 2048 + tail
    gen = torch.Generator(device="cuda").manual_seed(n)
    z, x = (torch.randn(n, device="cuda", generator=gen).mul_(0.02) for _ in range(2))
    opt, q, beta = b2.OptimizerModule(), b2.Nvfp4QuantModule(), 0.7

    def buffers():
        return [torch.full((n // 2,), 255, dtype=torch.uint8, device="cuda"), torch.full((n // 16,), 255, dtype=torch.uint8, device="cuda"),
                torch.full((1,), -1.0, device="cuda")], torch.full((1,), 7.0, device="cuda"), torch.full(((n + 2047) // 2048,), 7.0, device="cuda")

    for source in ("master", "schedule", "transform"):
        got, amax, chunk = buffers()
        want, want_amax, want_chunk = buffers()
        if source == "master":
            opt.materialize_master(got[0], got[1], got[2], x, amax, chunk, n, b2.SCALES_RAW)
            q.tensor_amax_f32(x, want_chunk, want_amax, n)
            q.fp32_to_nvfp4_four_six(x, want_amax, *want, n // 16, b2.SCALES_RAW)
            assert torch.equal(chunk, want_chunk)
        else:
            kw = dict(z_master=z, x_master=x, len=n, scale_rows=n // 16, scale_k=16, beta=beta, scale_layout=b2.SCALES_RAW,
                      symexp_lin_beta=12.5 if source == "transform" else 0.0)
            opt.materialize_schedule_free(bytes=got[0], scales=got[1], global_scale=got[2], amax=amax, **kw)
            y = z + (x - z) * beta
            if source == "schedule":
                q.tensor_amax_f32(y, want_chunk, want_amax, n)
            else:   # (the maximum: test_transformed_maximum_over_many_chunks)
                want_amax.copy_(amax)
            opt.materialize_schedule_free_precomputed(bytes=want[0], scales=want[1], global_scale=want[2], amax=want_amax,
                                                      precomputed_values=y if source == "schedule" else None, **kw)
        torch.cuda.synchronize()
        assert torch.equal(amax, want_amax), source
        for a, b in zip(got, want):
            assert torch.equal(a, b), source


@pytest.mark.parametrize("symexp", [12.5, 0.37, 1.0 / 3.0, 2.0 ** -20, 1.9999999])
def test_transform_divides_as_the_division_does(symexp):
    """Four values that are all far from the ends of the range are divided by multiplication with the reciprocal and two
    remainder steps, correctly rounded; a zero among them sends the four to the division.  The maximum shows the value itself."""
    rng = np.random.default_rng(11)
    values = (np.exp(rng.uniform(np.log(1e-7), np.log(3.0 / max(symexp, 0.1)), 150)) * rng.choice([-1.0, 1.0], 150)).astype(F)
    opt = b2.OptimizerModule()
    t = b2.Nvfp4Tensor.empty(1, 16, b2.SCALES_RAW)
    out = torch.zeros(2, len(values), device="cuda")
    for i, v in enumerate(values):
        for way, four in enumerate(([v, v, v, v], [v, v, v, 0.0])):
            x = dev(np.array(four * 4, F))
            opt.materialize_schedule_free(bytes=t.bytes, scales=t.scales, global_scale=t.global_scale, amax=out[way, i:i + 1], z_master=x,
                                          x_master=x, len=16, scale_rows=1, scale_k=16, beta=0.5, scale_layout=b2.SCALES_RAW,
                                          symexp_lin_beta=symexp)
    torch.cuda.synchronize()
    a, b = host(out)
    assert np.array_equal(a, b) and len(np.unique(a)) > 100


@pytest.mark.parametrize("chunks,tail", [(0, 16), (1, 48), (3, 0), (1279, 2032), (6144, 16)])
@pytest.mark.parametrize("at", ["first", "between", "last"])
def test_transformed_maximum_over_many_chunks(chunks, tail, at):
    """The transform with positive scales grows with |y|, so the maximum of a tensor is the transform of its largest value, which a
    call on 16 values shows alone; it stands out by a third, which no rounding of the transform turns round."""
    n = chunks * 2048 + tail
    where = {"first": 0, "between": n // 2 + 5, "last": n - 1}[at]
    gen = torch.Generator(device="cuda").manual_seed(n + where)
    z, x = (torch.rand(n, device="cuda", generator=gen).sub_(0.5).mul_(0.3) for _ in range(2))
    z[where] = -0.21
    x[where] = -0.2
    opt, scales = b2.OptimizerModule(), [torch.full((1,), v, device="cuda") for v in (1.1, 0.9, 0.8, 1.3, 1.2, 1.0)]
    amax = torch.full((2,), 7.0, device="cuda")
    outs = []
    for i, (zz, xx) in enumerate(((z, x), (z[where:where + 1].repeat(16), x[where:where + 1].repeat(16)))):
        m = zz.numel()
        q = dict(bytes=torch.full((m // 2,), 255, dtype=torch.uint8, device="cuda"), scales=torch.full((m // 16,), 255, dtype=torch.uint8, device="cuda"),
                 global_scale=torch.zeros(1, device="cuda"))
        opt.materialize_schedule_free(**q, amax=amax[i:i + 1], z_master=zz, x_master=xx, len=m, scale_rows=m // 16, scale_k=16, beta=0.5,
                                      scale_layout=b2.SCALES_RAW, symexp_lin_beta=12.5, symexp_lin_scales=scales)
        outs.append(q)
    torch.cuda.synchronize()
    assert float(torch.max((z + (x - z) * 0.5).abs())) == float((z + (x - z) * 0.5)[where].abs()) and float(amax[0]) > 0.1
    assert float(amax[0]) == float(amax[1])
    assert torch.equal(outs[0]["global_scale"], outs[1]["global_scale"])
    group = where // 16
    assert outs[0]["scales"][group] == outs[1]["scales"][0]
