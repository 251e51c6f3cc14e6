"""Performance cases of the GCOO sparse x dense multiply.

A case is one call (or one short call sequence) that a user of this library
makes through its Python entry points, at a size its configurations, tests or
benchmark use:

  mulby      GcooHandle.multiply_by: the sparse operand arrives dense and new
             with every call, so each pass converts it and multiplies (the
             plugin's mutiplyBy).
  spdm       GcooHandle.spdm on a handle built once, FP32 (the plugin's
             build + runKernelTest).
  form       the same with a reduced-precision form: BF16, split-BF16 or
             FP8-B, on block-clustered or on unstructured matrices.
  irregular  spdm on a power-law matrix ingested from COO triplets.
  left       GcooHandle.spdm_left: C = D x A (the plugin's mutiply).
  view       conversion into caller-owned arrays and the multiply straight
             from those arrays (convert_count, convert_scatter, spdm_view).
  batch      GcooBatch.run: many small multiplies of uneven shape at once.
"""
import math

import torch

import gcoospdm_gb300 as g
from gcoospdm_gb300 import datagen

DEV = "cuda"


def listed():
    return [
        # the reference's README example, the smallest call: launches and host time count
        {"name": "mulby_800", "kind": "mulby", "m": 800, "k": 800, "n": 800, "density": 0.1, "mask": "random"},
        # the headline workload: convert + multiply at 1 % density
        {"name": "mulby_8192", "kind": "mulby", "m": 8192, "k": 8192, "n": 8192, "density": 0.01, "mask": "random"},
        # sizes as real data brings them: no dimension a multiple of anything
        {"name": "mulby_ragged", "kind": "mulby", "m": 4001, "k": 3999, "n": 2047, "density": 0.02, "mask": "random"},
        # the largest and sparsest point of the n x sparsity sweep, one conversion kept
        {"name": "spdm_16384", "kind": "spdm", "m": 16384, "k": 16384, "n": 16384, "density": 0.001, "mask": "random"},
        # a block-clustered operand in plain FP32 (block-pruned weights, FEM matrices)
        {"name": "spdm_block", "kind": "spdm", "m": 8192, "k": 8192, "n": 1024, "density": 0.25, "mask": "block"},
        # the same operand in the reduced-precision forms that the tensor cores serve
        {"name": "bf16_block", "kind": "form", "prec": "bf16", "m": 8192, "k": 8192, "n": 1024, "density": 0.25,
         "mask": "block"},
        {"name": "split_block", "kind": "form", "prec": "split_bf16", "m": 8192, "k": 8192, "n": 1024,
         "density": 0.25, "mask": "block"},
        # an FP8 dense operand against an unstructured matrix
        {"name": "fp8_random", "kind": "form", "prec": "fp8_b", "m": 4096, "k": 4096, "n": 4096, "density": 0.02,
         "mask": "random"},
        # a graph-like matrix: Zipf row lengths up to 4096 entries
        {"name": "irregular", "kind": "irregular", "m": 65536, "k": 65536, "n": 256, "nnz": 1200000},
        # the other orientation: a batch of 1024 activations times a sparse weight
        {"name": "left_8192", "kind": "left", "m": 8192, "k": 8192, "n": 1024, "density": 0.01, "mask": "random"},
        # a caller that keeps the GCOO arrays in its own memory
        {"name": "view_4096", "kind": "view", "m": 4096, "k": 4096, "n": 2048, "density": 0.01, "mask": "count"},
        # 512 small multiplies of uneven shape as one launch
        {"name": "batch_512", "kind": "batch", "prec": "fp32", "count": 512, "shapes": 30},
    ]


def _size(rng, lo, hi, multiple=1):
    """Log-uniform in [lo, hi]; for multiple 1 half of the sizes are round."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if multiple == 1 and rng.random() < 0.5:
        multiple = 32
    return max(lo, min(hi, v // multiple * multiple if v >= multiple else multiple))


def _density(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 5)


def draw(rng):
    kind = rng.choice(["mulby", "mulby", "spdm", "spdm", "form", "form", "irregular", "left", "view", "batch"])
    if kind == "batch":
        return {"kind": kind, "prec": rng.choice(["fp32", "bf16"]), "count": _size(rng, 32, 512), "shapes": rng.randrange(1 << 20)}
    if kind == "irregular":
        m = _size(rng, 8192, 65536)
        return {"kind": kind, "m": m, "k": m, "n": _size(rng, 32, 256), "nnz": int(m * rng.uniform(6.0, 18.0))}
    while True:
        mask = "random"
        if kind == "form":
            prec = rng.choice(["bf16", "split_bf16", "fp8_b"])
            mask = rng.choice(["block", "random"])
            if mask == "block":
                m, k, n = _size(rng, 1024, 8192), _size(rng, 1024, 8192), _size(rng, 64, 1024, 16)
                density = _density(rng, 0.1, 0.25)
            else:
                m, k, n = _size(rng, 1024, 8192), _size(rng, 1024, 8192), _size(rng, 128, 4096, 16)
                density = _density(rng, 0.001, 0.05)
            c = {"kind": kind, "prec": prec}
        elif kind == "spdm":
            mask = rng.choice(["block", "random", "random"])
            c = {"kind": kind}
            if mask == "block":
                m, k, n = _size(rng, 1024, 8192), _size(rng, 1024, 8192), _size(rng, 64, 1024)
                density = _density(rng, 0.1, 0.25)
            else:
                m, k, n = (_size(rng, 800, 16384) for _ in range(3))
                density = _density(rng, 0.001, 0.1)
        elif kind == "mulby":
            c = {"kind": kind}
            m, k, n = (_size(rng, 800, 8192) for _ in range(3))
            density = _density(rng, 0.001, 0.1)
        else:
            c = {"kind": kind}
            if kind == "view":
                mask = "count"
            m, k, n = _size(rng, 800, 8192), _size(rng, 800, 8192), _size(rng, 128, 2048)
            density = _density(rng, 0.001, 0.05)
        c.update(m=m, k=k, n=n, density=density, mask=mask)
        # no more work than the largest listed case of its sort
        limit = 3.4e10 if mask == "block" else 1.4e9 if kind in ("left", "view") else 1.1e10
        if work(c)["flops"] <= limit:
            return c


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _pm1(gen, rows, cols):
    """U(-1, 1), never 0 (odd multiples of 2^-24)."""
    u = torch.randint(0, 1 << 24, (rows, cols), generator=gen, device=DEV, dtype=torch.int32)
    return (2 * u + (1 - (1 << 24))).to(torch.float32) * 2.0 ** -24


def _operand(gen, m, k, density, mask):
    """The sparse operand as the dense buffer with zeros that the handle takes."""
    vals = _pm1(gen, m, k)
    if mask == "block":  # 16 x 16 blocks, each active with the density's probability and dense inside
        on = torch.rand((m + 15) // 16, (k + 15) // 16, generator=gen, device=DEV) < density
        on = on.repeat_interleave(16, 0)[:m].repeat_interleave(16, 1)[:, :k]
    elif mask == "count":  # the same number of entries whatever the seed
        on = torch.zeros(m * k, dtype=torch.bool, device=DEV)
        on[torch.randperm(m * k, generator=gen, device=DEV)[:round(density * m * k)]] = True
        on = on.view(m, k)
    else:
        on = torch.rand(m, k, generator=gen, device=DEV) < density
    return vals.masked_fill_(~on, 0.0)


def _zipf(case, seed):
    rows, cols, vals = datagen.zipf_coo(seed, case["m"], case["k"], case["nnz"], alpha=2.0, cap=4096)
    to = lambda a, t: torch.from_numpy(a).to(DEV, t)  # noqa: E731
    return to(rows, torch.int32), to(cols, torch.int32), to(vals, torch.float32)


def _inputs(case, seed):
    gen = _gen(seed)
    if case["kind"] == "batch":
        shapes = datagen.batched_shapes(case["shapes"], case["count"])
        return [(_operand(gen, m, k, 1.0 - s, "random"), _pm1(gen, k, n)) for m, k, n, s in shapes]
    if case["kind"] == "irregular":
        B = torch.randn(case["k"], case["n"], generator=gen, device=DEV)
        return _zipf(case, seed), B
    A = _operand(gen, case["m"], case["k"], case["density"], case["mask"])
    if case["kind"] == "left":
        return A, _pm1(gen, case["n"], case["m"])
    return A, _pm1(gen, case["k"], case["n"])


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        problems = _inputs(case, seed)
        # the results side by side in one buffer, each 256-byte aligned
        sizes = [(A.shape[0], B.shape[1]) for A, B in problems]
        steps = [(m * n + 63) // 64 * 64 for m, n in sizes]
        s["C"] = torch.zeros(sum(steps), device=DEV)
        outs = [c[:m * n].view(m, n) for c, (m, n) in zip(s["C"].split(steps), sizes)]
        s["batch"] = g.GcooBatch([(g.GcooHandle(A).build(), B, C) for (A, B), C in zip(problems, outs)],
                                 prec=case["prec"])
        return s
    if kind == "irregular":
        coo, s["B"] = _inputs(case, seed)
        s["handle"] = g.GcooHandle.from_coo(*coo, m=case["m"], k=case["k"]).build()
        s["C"] = torch.empty(case["m"], case["n"], device=DEV)
        return s
    A, s["B"] = _inputs(case, seed)
    if kind == "view":
        s["A"] = A
        s["C"] = torch.empty(case["m"], case["n"], device=DEV)
        return s
    s["handle"] = g.GcooHandle(A)
    if kind == "left":
        s["C"] = torch.empty(case["n"], case["k"], device=DEV)
    else:
        s["C"] = torch.empty(case["m"], case["n"], device=DEV)
    if kind != "mulby":
        s["handle"].build()
    if kind == "form":
        s["prec"] = case["prec"]
        s["handle"].prepare(case["n"], case["prec"])
    return s


def run(state):
    kind = state["kind"]
    if kind == "mulby":
        return state["handle"].multiply_by(state["B"], state["C"])
    if kind in ("spdm", "irregular"):
        return state["handle"].spdm(state["B"], state["C"])
    if kind == "form":
        return state["handle"].spdm(state["B"], state["C"], prec=state["prec"])
    if kind == "left":
        return state["handle"].spdm_left(state["B"], state["C"])
    if kind == "batch":
        state["batch"].run()
        return state["C"]
    A = state["A"]
    group_index, nnz_per_group, nnz = g.convert_count(A)
    vals, rows, cols = g.convert_scatter(A, group_index, nnz)
    C = g.spdm_view(A.shape[0], A.shape[1], 4, group_index, nnz_per_group, vals, rows, cols, state["B"], state["C"])
    return {"group_index": group_index, "nnz_per_group": nnz_per_group, "vals": vals, "rows": rows, "cols": cols,
            "C": C}


def work(case):
    """Every input read once and every output written once; two operations per entry and output column."""
    kind = case["kind"]
    if kind == "batch":
        # shapes uniform in [256, 4096], n in {32, 64, 128}, density uniform in [0.001, 0.1]
        m = k = 2176.0
        nnz, n = m * k * 0.0505, 224.0 / 3.0
        one = {"bytes": 8 * nnz + 4 * (m + 1) + 4 * n * (k + m), "flops": 2 * nnz * n}
        return {key: v * case["count"] for key, v in one.items()}
    m, k, n = case["m"], case["k"], case["n"]
    nnz = case["nnz"] if kind == "irregular" else case["density"] * m * k
    dense = 4 * k * n + 4 * m * n
    if kind == "left":
        dense = 4 * n * m + 4 * n * k
    if kind == "mulby":
        moved = 4 * m * k  # the operand as it arrives
    elif kind == "view":
        moved = 4 * m * k + 12 * nnz + 8 * (m // 4 + 1)  # and the caller's arrays written
    else:
        moved = 8 * nnz + 4 * (m + 1)  # a column and a value per entry, the row offsets
    return {"bytes": moved + dense, "flops": 2 * nnz * n}


def exact(case, seed):
    """The products in 64 bits; the conversion's values are copies, its indices whole numbers."""
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for A, B in _inputs(case, seed):
            C = (A.double() @ B.double()).flatten()
            parts += [C, C.new_zeros(-C.numel() % 64)]
        return torch.cat(parts)
    if kind == "irregular":
        (rows, cols, vals), B = _inputs(case, seed)
        C = torch.zeros(case["m"], case["n"], dtype=torch.float64, device=DEV)
        for at in range(0, rows.numel(), 1 << 20):
            part = slice(at, at + (1 << 20))
            C.index_add_(0, rows[part], vals[part].double()[:, None] * B[cols[part]].double())
        return C
    A, B = _inputs(case, seed)
    if kind == "left":
        return B.double() @ A.double()
    C = A.double() @ B.double()
    if kind != "view":
        return C
    none = dict.fromkeys(("group_index", "nnz_per_group", "vals", "rows", "cols"))
    return {**none, "C": C}
