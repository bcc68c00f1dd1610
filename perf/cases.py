"""Performance cases of the optimizer and requantisation path.

What a training program has this library do, through the entry points it calls: the matrix step as one call
(`OptimizerModule.muon_mega_update`), the matrix step in the trainer's order of separate calls with the per-step
variants, schedule-free AdamW on what is not a matrix, requantisation of single tensors, and the global gradient
norm.  Sizes are those of the GPT-2 configurations in bench.py, of the fixtures in tests/ and of the [R, 4096]
bandwidth sweep; `draw` gives other sizes and option combinations of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import llmini_b200 as b2

DEVICE = "cuda"
STEP = dict(mu=0.95, grad_scale=1.0, learning_rate=1.0e-4, weight_decay=0.025, average_coefficient=0.5,
            schedule_beta=0.2, iterations=5)
ADAM = dict(grad_scale=1.0, learning_rate=2.0e-4, weight_decay=0.005, beta1=0.9, beta2=0.95, beta1_correction=0.1,
            beta2_correction=0.05, eps=1.0e-10, average_coefficient=0.5, schedule_beta=0.2)
FIXED_TRIPLE = (3.4445, -4.7750, 2.0315)
LAYOUTS = {"csf": b2.SCALES_CSF, "raw": b2.SCALES_RAW, "sm100": b2.SCALES_SM100}
PAD = 256  # values between the tensors of an arena: every tensor starts on a 256-byte boundary or better


def _layer(d):
    """The four weight matrices of a transformer layer as [out, in]: qkv, attention projection, fc, MLP projection."""
    return f"{3 * d}x{d} {d}x{d} {4 * d}x{d} {d}x{4 * d}"


def _step(name, shapes, layers=1, operands="bf16", prepare="one pass", scales="csf", quantise="x"):
    return {"name": name, "path": "step", "shapes": shapes, "layers": layers, "operands": operands,
            "prepare": prepare, "scales": scales, "quantise": quantise}


def _trainer(name, shapes, layers=1, operands="bf16", scales="csf", finish="normuon", variance=False, clip=False):
    return {"name": name, "path": "trainer", "shapes": shapes, "layers": layers, "operands": operands,
            "prepare": "two passes", "scales": scales, "finish": finish, "variance": variance, "clip": clip}


def listed():
    return [
        # The smallest matrix step: the 64-wide matrices of the reference's fixtures, F16 operands and the default
        # coefficient table.  A toy model in a test or a first integration; launches and latency are all there is.
        _step("step, 64-wide fixture", "64x64 64x32 32x64", operands="f16", prepare="two passes", scales="raw"),
        # One MLP matrix of GPT-2 small with the plan's defaults (the reference's rounding point).
        _step("step, one 3072x768", "3072x768", prepare="two passes"),
        # The six matrices that one of eight GPUs owns of GPT-2 small: the step of a sharded run.
        _step("step, GPT-2 small / 8", "2304x768 2304x768 3072x768 3072x768 768x3072 768x768"),
        # All 48 matrices of GPT-2 small: the headline workload of bench.py.
        _step("step, GPT-2 small", _layer(768), layers=12),
        # All 192 matrices of GPT-2 XL, 1.47 G weights: the largest configuration.  1600 is no multiple of 128.
        _step("step, GPT-2 XL", _layer(1600), layers=48, scales="raw"),
        # GPT-2 medium in the order of the reference's trainer: adaptive-variance momentum, Newton-Schulz in F16 with
        # the default table, NorMuon and qk-clip in the update, then the training weights y as NVFP4.
        _trainer("trainer, GPT-2 medium", _layer(1024), layers=24, operands="f16", variance=True, clip=True),
        # Odd matrices in one plan (tall, wide, clipped at every tile edge) with the Hyperball finish.
        _trainer("trainer, ragged Hyperball", "1600x320 48x1600 200x208 1000x1040 77x512", scales="raw",
                 finish="hyperball"),
        # Embeddings (requantised), LayerNorm and bias values of GPT-2 small through one pointer table.
        {"name": "AdamW, GPT-2 small table", "path": "adamw", "rows": 50304, "d": 768, "vector": 102144,
         "mode": "requantise", "scales": "csf"},
        # One LayerNorm gain of GPT-2 small by itself: the smallest call there is.
        {"name": "AdamW, one 768 vector", "path": "vector", "len": 768},
        # A square weight of GPT-2 XL materialised from its schedule-free pair, with the SymExpLin transform.
        {"name": "schedule-free, 1600x1600", "path": "quantise", "source": "schedule", "rows": 1600, "k": 1600,
         "scales": "raw", "symexp": 12.5},
        # A large tensor requantised from its master: a row of the bandwidth sweep.
        {"name": "requantise, 65536x4096", "path": "quantise", "source": "master", "rows": 65536, "k": 4096,
         "scales": "csf", "symexp": 0.0},
        # The global gradient norm over every matrix of GPT-2 small in 4096-value chunks; the scale stays on the device.
        {"name": "gradient clip, GPT-2 small", "path": "clip", "shapes": _layer(768), "layers": 12, "apply": False},
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(v) // step * step))


def _draw_shapes(rng, budget):
    """-> (shapes, layers): whole transformer layers, or one to eight unrelated matrices with odd row counts."""
    if rng.random() < 0.65:
        d = _log_int(rng, 64, 1600, 16 if rng.random() < 0.5 else 64)
        return _layer(d), _log_int(rng, 1, max(1, min(48, int(budget // (12 * d * d)))))
    dims = []
    for _ in range(rng.randint(1, 8)):
        dims.append(f"{_log_int(rng, 16, 4096)}x{_log_int(rng, 16, 4096, 16)}")
    return " ".join(dims), 1


def _draw_layout(rng, columns):
    names = ["raw", "sm100"] + (["csf", "csf"] if all(c % 128 == 0 for c in columns) else [])
    return rng.choice(names)


def draw(rng):
    path = rng.choice(["step", "step", "step", "trainer", "trainer", "adamw", "vector", "quantise", "quantise", "clip"])
    if path == "step":
        shapes, layers = _draw_shapes(rng, 1.4e9)
        operands = rng.choice(["bf16", "bf16", "f16"])
        c = _step("", shapes, layers, operands, "two passes" if operands == "f16" else rng.choice(["one pass", "two passes"]),
                  _draw_layout(rng, [k for _, k in _shapes(shapes, 1)]), rng.choice(["x", "y"]))
    elif path == "trainer":
        shapes, layers = _draw_shapes(rng, 7.0e8)
        c = _trainer("", shapes, layers, rng.choice(["bf16", "f16"]), _draw_layout(rng, [k for _, k in _shapes(shapes, 1)]),
                     rng.choice(["plain", "normuon", "hyperball", "sign"]), rng.random() < 0.5, rng.random() < 0.5)
    elif path == "adamw":
        d = _log_int(rng, 64, 1600, 16)
        c = {"path": path, "rows": _log_int(rng, 128, 50304), "d": d, "vector": _log_int(rng, 100, 1000000),
             "mode": rng.choice(["requantise", "deferred"]), "scales": "csf" if d % 128 == 0 else "raw"}
    elif path == "vector":
        c = {"path": path, "len": _log_int(rng, 16, 4000000)}
    elif path == "quantise":
        k = _log_int(rng, 16, 8192, 16 if rng.random() < 0.5 else 128)
        k = max(k, 16)
        c = {"path": path, "source": rng.choice(["master", "schedule"]), "rows": _log_int(rng, 1, min(262144, int(3.0e8 // k))),
             "k": k, "scales": "csf" if k % 128 == 0 and rng.random() < 0.7 else "raw",
             "symexp": rng.choice([0.0, 0.0, 12.5])}
    else:
        shapes, layers = _draw_shapes(rng, 1.4e9)
        c = {"path": path, "shapes": shapes, "layers": layers, "apply": rng.random() < 0.5}
    c.pop("name", None)
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------
def _shapes(text, layers):
    return [tuple(int(v) for v in s.split("x")) for s in text.split()] * layers


def _arena_offsets(sizes):
    at, offsets = 0, []
    for n in sizes:
        offsets.append(at)
        at += (n + PAD - 1) // PAD * PAD
    return offsets, at


def _weights(gen, n):
    return torch.randn(n, device=DEVICE, generator=gen).mul_(0.02)


def _gradients(gen, n):
    """N(0, 1e-3) with one value in a thousand fifty times as large."""
    g = torch.randn(n, device=DEVICE, generator=gen).mul_(1.0e-3)
    k = max(1, n // 1000)
    g[torch.randint(0, n, (k,), device=DEVICE, generator=gen)] *= 50.0
    return g


def _scale_storage(rows, cols, layout):
    """Initial block-scale storage of one tensor: a CSF header in front where the layout has one."""
    if layout == b2.SCALES_CSF:
        return b2.zero_scales(rows, cols, DEVICE)
    size = b2.sm100_scales_bytes(rows, cols) if layout == b2.SCALES_SM100 else rows * cols // 16
    return torch.zeros(size, dtype=torch.uint8, device=DEVICE)


def _matrices(case, gen):
    """Every matrix of the model in one arena per kind of buffer, as a trainer holds them."""
    shapes = _shapes(case["shapes"], case["layers"])
    layout = LAYOUTS[case["scales"]]
    offsets, total = _arena_offsets([r * c for r, c in shapes])
    stores = {s: _scale_storage(*s, layout) for s in set(shapes)}
    s_offsets, s_total = _arena_offsets([stores[s].numel() for s in shapes])
    out = {"grad": _gradients(gen, total), "momentum": (torch.randn(total, device=DEVICE, generator=gen) * 1.0e-3).to(torch.bfloat16),
           "z": _weights(gen, total), "x": _weights(gen, total),
           "amax": torch.zeros(len(shapes), device=DEVICE), "codes": torch.zeros(total // 2, dtype=torch.uint8, device=DEVICE),
           "scales": torch.zeros(s_total, dtype=torch.uint8, device=DEVICE),
           "global_scale": torch.zeros(len(shapes), device=DEVICE)}
    variance, finish = case.get("variance", False), case.get("finish", "plain")
    if variance:
        out["variance"] = (torch.rand(total, device=DEVICE, generator=gen) * 2.0e-6).to(torch.bfloat16)
    if finish in ("normuon", "hyperball"):
        n_offsets, n_total = _arena_offsets([max(r, c) for r, c in shapes])
        out["second_momentum"] = torch.rand(n_total, device=DEVICE, generator=gen).mul_(2.0e-3).add_(1.0e-4)
    slots, heads = [], 0
    for i, (r, c) in enumerate(shapes):
        at, n = offsets[i], r * c
        part = lambda key: out[key][at:at + n].view(r, c)
        s = b2.MuonSlot(part("grad"), part("momentum"), part("z"), part("x"), out["amax"][i:i + 1],
                        out["codes"][at // 2:(at + n) // 2], out["scales"][s_offsets[i]:s_offsets[i] + stores[(r, c)].numel()],
                        out["global_scale"][i:i + 1], r, c)
        s.scales.copy_(stores[(r, c)])
        if variance:
            s.variance = part("variance")
        if finish in ("normuon", "hyperball"):
            s.second_momentum = out["second_momentum"][n_offsets[i]:n_offsets[i] + max(r, c)]
        if case.get("clip", False) and r == 3 * c:   # fused qkv: 64-wide heads, the last one narrower where c is odd
            s.qk_clip_factor_offset, s.qk_clip_head_dim = heads, 64
            heads += (c + 63) // 64
        slots.append(s)
    factors = None
    if heads:   # most heads are below the logit threshold in a given step
        factors = torch.where(torch.rand(heads, device=DEVICE, generator=gen) < 0.875, 1.0, 0.95)
    return shapes, slots, out, factors


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    state = {"case": case, "opt": b2.OptimizerModule()}
    path = case["path"]
    if path in ("step", "trainer"):
        shapes, slots, out, factors = _matrices(case, gen)
        f16 = case["operands"] == "f16"
        state["plan"] = b2.MuonPlan(shapes, operand_format=b2.OPERAND_F16 if f16 else b2.OPERAND_BF16,
                                    scale_layout=LAYOUTS[case["scales"]],
                                    quantize_target=b2.QUANTIZE_Y if case.get("quantise") == "y" else b2.QUANTIZE_X,
                                    normalize_mode=b2.NORMALIZE_DEFERRED if case["prepare"] == "one pass" else b2.NORMALIZE_TWO_PASS)
        state["slots"], state["table"], state["out"] = slots, b2.slot_table(slots), out
        extra = {}
        if path == "trainer":
            extra = dict(variance_adaptive=case["variance"], bias_correction_inv=1.5 if case["variance"] else 1.0,
                         qk_clip_factors=factors, normuon=case["finish"] == "normuon")
        coefficients = None if f16 else np.tile(np.asarray(FIXED_TRIPLE, np.float32), (5, 1))
        state["args"] = b2.MuonMegaUpdateArgs(coefficients=coefficients, **STEP, **extra)
    elif path == "adamw":
        layout, tensors, out = LAYOUTS[case["scales"]], [], []
        mode = {"requantise": 2, "deferred": 1}[case["mode"]]
        # token embedding, position embedding, then every LayerNorm and bias value as one plain FP32 tensor
        for rows, cols, m in ((case["rows"], case["d"], mode), (1024, case["d"], mode), (1, case["vector"], 0)):
            t = _adam_tensor(gen, rows * cols)
            if m:
                t.update(bytes=torch.zeros(rows * cols // 2, dtype=torch.uint8, device=DEVICE),
                         scales=_scale_storage(rows, cols, layout), global_scale=torch.zeros(1, device=DEVICE),
                         amax=torch.zeros(1, device=DEVICE), scale_layout=layout)
            tensors.append(dict(t, mode=m, len=rows * cols))
            out.append({k: v for k, v in t.items() if torch.is_tensor(v) and (k != "grad" or m == 1)})
        state["tensors"], state["out"] = tensors, out
        state["table"] = state["opt"].adamw_table(tensors)
    elif path == "vector":
        state["tensor"] = _adam_tensor(gen, case["len"])
        state["out"] = {k: v for k, v in state["tensor"].items() if k != "grad"}
    elif path == "quantise":
        rows, k = case["rows"], case["k"]
        n, layout = rows * k, LAYOUTS[case["scales"]]
        q = dict(bytes=torch.zeros(n // 2, dtype=torch.uint8, device=DEVICE), scales=_scale_storage(rows, k, layout),
                 global_scale=torch.zeros(1, device=DEVICE), amax=torch.zeros(1, device=DEVICE))
        state["out"] = q
        z = _weights(gen, n)
        if case["source"] == "master":
            state["call"] = dict(bytes_=q["bytes"], scales=q["scales"], global_scale=q["global_scale"], master=z, amax=q["amax"],
                                 chunk_amax=torch.zeros((n + 2047) // 2048, device=DEVICE), len_=n, scale_layout=layout)
        else:
            state["call"] = dict(q, z_master=z, x_master=_weights(gen, n), len=n, scale_rows=rows, scale_k=k, beta=0.7,
                                 symexp_lin_beta=case["symexp"], scale_layout=layout)
    else:
        shapes = _shapes(case["shapes"], case["layers"])
        offsets, total = _arena_offsets([r * c for r, c in shapes])
        grad = _gradients(gen, total)
        cuts = [(grad.data_ptr() + 4 * (o + a), min(4096, r * c - a)) for o, (r, c) in zip(offsets, shapes)
                for a in range(0, r * c, 4096)]
        # what other tensors contribute (summed where they were computed) keeps the norm above the limit
        extra = torch.rand(8, device=DEVICE, generator=gen).add_(1.0)
        one = lambda: torch.zeros(1, device=DEVICE)
        state["out"] = {"scale": one(), "norm": one(), "chunk_sums": torch.zeros(len(cuts), device=DEVICE)}
        if case["apply"]:
            state["out"]["grad"] = grad
        state["grad"] = grad
        state["call"] = dict(chunk_ptrs=torch.tensor([p for p, _ in cuts], dtype=torch.int64, device=DEVICE),
                             chunk_lens=torch.tensor([n for _, n in cuts], dtype=torch.int32, device=DEVICE),
                             chunk_sums=state["out"]["chunk_sums"], extra_sums=extra, scale=state["out"]["scale"],
                             norm=state["out"]["norm"], chunk_count=len(cuts), extra_sum_count=extra.numel(), max_norm=3.0,
                             apply=case["apply"])
    return state


def _adam_tensor(gen, n):
    randn = lambda std: torch.randn(n, device=DEVICE, generator=gen).mul_(std)
    return dict(z_master=randn(0.02), x_master=randn(0.02), grad=_gradients(gen, n), first_moment=randn(1.0e-4),
                second_moment=torch.rand(n, device=DEVICE, generator=gen).mul_(2.0e-6))


# ---- one pass -------------------------------------------------------------------------------------------------
def run(state):
    case, opt = state["case"], state["opt"]
    path = case["path"]
    if path == "step":
        opt.muon_mega_update(state["plan"], state["table"], state["args"])
    elif path == "trainer":
        plan, table, args = state["plan"], state["table"], state["args"]
        if case["finish"] == "sign":
            opt.muon_tma_sign_update_deferred_quantization(plan, table, args)
        else:
            opt.muon_tma_prepare_polar(plan, table, args)
            opt.muon_polar(plan, args)
            if case["finish"] == "hyperball":
                opt.muon_tma_finish_hyperball_update_deferred_quantization(plan, table, args)
            else:
                opt.muon_tma_finish_update_deferred_quantization(plan, table, args)
        opt.muon_materialize_training_weights(plan, table)
    elif path == "adamw":
        table, count, chunks = state["table"]
        opt.apply_adamw_update_multi(table, count, chunks, **ADAM)
        if case["mode"] == "deferred":
            opt.adamw_materialize_training_weights(table, count, chunks, ADAM["schedule_beta"])
    elif path == "vector":
        opt.apply_fp32_adamw_update(len=case["len"], **state["tensor"], **ADAM)
    elif path == "quantise":
        if case["source"] == "master":
            opt.materialize_master(**state["call"])
        else:
            opt.materialize_schedule_free(**state["call"])
    else:
        opt.clip_gradients(**state["call"])
    return state["out"]


# ---- what a pass cannot do without ----------------------------------------------------------------------------
def work(case):
    path = case["path"]
    packed = 0.5 + 1.0 / 16.0     # codes and block scales of one value
    if path in ("step", "trainer"):
        shapes = _shapes(case["shapes"], case["layers"])
        n = sum(r * c for r, c in shapes)
        # gradient read and overwritten by y, momentum, z and x read and written
        bpe = 8.0 + 4.0 + 8.0 + 8.0 + packed + (4.0 if case.get("variance") else 0.0)
        flops = 0.0
        if case.get("finish") != "sign":
            # an iteration: half of the symmetric X X^T and of its square, and the product with X
            for r, c in shapes:
                lo, hi = min(r, c), max(r, c)
                flops += 5.0 * (3.0 * lo * lo * hi + lo ** 3)
        return {"bytes": n * bpe, "flops": flops + 30.0 * n}
    if path == "adamw":
        e = (case["rows"] + 1024) * case["d"]
        deferred = case["mode"] == "deferred"
        return {"bytes": e * (36.0 + packed + (4.0 if deferred else 0.0)) + case["vector"] * 36.0,
                "flops": 25.0 * (e + case["vector"])}
    if path == "vector":
        return {"bytes": case["len"] * 36.0, "flops": 20.0 * case["len"]}
    if path == "quantise":
        n = case["rows"] * case["k"]
        return {"bytes": n * ((4.0 if case["source"] == "master" else 8.0) + packed), "flops": 4.0 * n}
    n = sum(r * c for r, c in _shapes(case["shapes"], case["layers"]))
    return {"bytes": n * (8.0 if case["apply"] else 4.0), "flops": 2.0 * n}


def tolerance(case):
    path = case["path"]
    if path == "quantise":
        return "exact"            # a maximum and roundings: no order of operations to choose
    if path in ("step", "trainer"):
        # The orthogonalised direction is a BF16 / F16 result (1e-2); a step moves the weights by a thousandth of their
        # size, so the masters are good to 1e-5, the BF16 momentum to one unit in the last place here and there, and
        # a code or scale byte flips where a value sits on a rounding boundary.  Hyperball moves them by lr times
        # their norm, NorMuon divides by a root of a second moment: the same order.
        return {"rel": 2.0e-4, "max": 2.0e-2, "differ": 3.0e-3}
    if path in ("adamw", "vector"):
        return {"rel": 1.0e-6, "max": 1.0e-4, "differ": 1.0e-4}
    return {"rel": 1.0e-5, "max": 1.0e-5}
