"""The work that users of this framework have it do, as cases that can be prepared, run and compared.

A case is a plain dict: what is asked (`kind`), the matrix (`family` and its sizes), the value type and the logical
width of the dense operand.  `listed()` names the standing cases, `draw(rng)` gives more of the same ranges.

Kinds:
  spmm    the steady state of a solver, an eigenvalue iteration or a graph network: the matrix is converted and tuned
          once, then multiplied again and again with operands that stay on the GPU (`TileMatrix.spmm`);
  once    a matrix that is multiplied once: conversion of a CSR already on the GPU and one product;
  once_host  the same for a CSR in host memory, with the threshold model in front -- the whole sequence of the
          command-line driver: features, model, conversion, product;
  host    one blocking product with operands in ordinary host memory (`TileMatrix.spmm_host`);
  stream  several right-hand sides from and to pinned host memory through the two staging slots
          (`tsp_spmm_host_async` / `tsp_spmm_host_wait`).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from tilespmm_b200 import api, synth

PRECISION = {"fp16": 0, "tf32": 1}
DTYPE = {"fp16": torch.float16, "tf32": torch.float32}
STREAM_STEPS = 4   # right-hand sides of one pass of a `stream` case


# ---------------------------------------------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest call: 4096^2 with 16 entries a row and a 32-column operand; latency and launches count
        {"name": "spmm_fixed_4096_fp16", "kind": "spmm", "family": "fixed", "precision": "fp16", "rows": 4096, "cols": 4096, "per_row": 16, "colB": 32},
        # a small rectangular matrix with clustered rows, odd sizes and a width that needs padding: several tile classes in one product
        {"name": "spmm_clustered_4099_tf32", "kind": "spmm", "family": "clustered", "precision": "tf32", "rows": 4099, "cols": 9000, "colB": 100},
        # the benchmark's headline: a 27-point stencil on 64^3 (a PDE operator times a block of vectors)
        {"name": "spmm_stencil_64_tf32", "kind": "spmm", "family": "stencil", "precision": "tf32", "grid": 64, "colB": 128},
        # a power-law graph times node features (graph networks)
        {"name": "spmm_rmat_20_fp16", "kind": "spmm", "family": "rmat", "precision": "fp16", "scale": 20, "values": "one", "colB": 64},
        # dense blocks in a few panels, almost empty rows elsewhere, a wide operand larger than the L2
        {"name": "spmm_mixed_524288_tf32", "kind": "spmm", "family": "mixed", "precision": "tf32", "rows": 524288, "colB": 256},
        # block-diagonal weights, the tall tiles' home ground, at a width that is no multiple of 128
        {"name": "spmm_blocks_65536_fp16", "kind": "spmm", "family": "blocks", "precision": "fp16", "rows": 65536, "block": 64, "density": 0.5, "colB": 192},
        # the largest: 130 million entries, nothing fits the L2
        {"name": "spmm_rmat_22_fp16", "kind": "spmm", "family": "rmat", "precision": "fp16", "scale": 22, "values": "u01", "colB": 128},
        # a small matrix that changes on every call (a sampled sub-graph)
        {"name": "once_fixed_4096_fp16", "kind": "once", "family": "fixed", "precision": "fp16", "rows": 4096, "cols": 4096, "per_row": 16, "colB": 32},
        # a graph that changes on every call (an epoch's sparsified adjacency)
        {"name": "once_rmat_18_fp16", "kind": "once", "family": "rmat", "precision": "fp16", "scale": 18, "values": "u01", "colB": 64},
        # what the command-line driver does with a matrix it has just read
        {"name": "once_host_stencil_40_tf32", "kind": "once_host", "family": "stencil", "precision": "tf32", "grid": 40, "colB": 128},
        # one product for a caller whose arrays are ordinary numpy arrays
        {"name": "host_stencil_48_tf32", "kind": "host", "family": "stencil", "precision": "tf32", "grid": 48, "colB": 128},
        # many right-hand sides for a caller with pinned buffers
        {"name": "stream_stencil_48_tf32", "kind": "stream", "family": "stencil", "precision": "tf32", "grid": 48, "colB": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmm"] * 7 + ["once", "once", "once_host", "host", "stream"])
    small = kind != "spmm"   # the other kinds stay within the cost of their listed cases
    family = rng.choice(["fixed", "clustered", "stencil", "rmat", "mixed", "blocks", "banded"])
    case = {"kind": kind, "family": family, "precision": rng.choice(["fp16", "tf32"])}
    case["colB"] = rng.choice([32, 64, 128, 256]) if rng.random() < 0.5 else rng.randint(1, 256 if small or family == "rmat" else 320)
    if family == "fixed":
        case["rows"] = _log_int(rng, 500, 40_000 if small else 300_000)
        case["cols"] = max(64, int(case["rows"] * rng.uniform(0.5, 1.5 if small else 2.0)))
        case["per_row"] = min(_log_int(rng, 4, 256), case["cols"] // 2, max(4, (3_000_000 if small else 20_000_000) // case["rows"]))
    elif family == "clustered":
        case["rows"] = _log_int(rng, 300, 40_000 if small else 200_000)
        case["cols"] = max(512, int(case["rows"] * rng.uniform(0.7, 1.5 if small else 2.2)))
    elif family == "stencil":
        case["grid"] = _log_int(rng, 10, 36 if small else 72)
    elif family == "rmat":
        case["scale"] = rng.randint(11, 20 if not small else (17 if kind.startswith("once") else 15))
        case["values"] = rng.choice(["one", "u01"])
    elif family == "mixed":
        case["rows"] = 64 * _log_int(rng, 64, 750 if small else 8192)
    elif family == "blocks":
        case["block"] = rng.choice([32, 64, 128])
        case["density"] = rng.choice([0.2, 0.3, 0.5, 0.8])
        case["rows"] = case["block"] * _log_int(rng, 32, (40_000 if small else 130_000) // case["block"])
    else:
        case["rows"] = _log_int(rng, 1000, 50_000 if small else 260_000)
        case["half"] = _log_int(rng, 4, 40)
    return case


# ---------------------------------------------------------------------------------------------------------------
# matrices, made on the GPU from a seed: CSR of int32 row pointers, int32 columns and float32 values

def _csr(rows, cols, shape, gen, shuffle=False):
    """Row pointers and columns of the distinct (row, col) pairs; columns sorted within rows, or in random order."""
    keys = torch.unique(rows * shape[1] + cols)
    r = torch.div(keys, shape[1], rounding_mode="floor")
    c = keys - r * shape[1]
    if shuffle:
        c = c[torch.argsort(r.double() + torch.rand(r.numel(), generator=gen, device="cuda", dtype=torch.float64))]
    ptr = torch.zeros(shape[0] + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=shape[0]), 0)
    return ptr.to(torch.int32), c.to(torch.int32)


def _normal(n, gen):
    return torch.randn(n, generator=gen, device="cuda")


def _fixed(case, gen):
    n, m, k = case["rows"], case["cols"], case["per_row"]
    rows = torch.arange(n, device="cuda").repeat_interleave(k)
    cols = torch.randint(0, m, (n * k,), generator=gen, device="cuda")
    ptr, ci = _csr(rows, cols, (n, m), gen, shuffle=True)      # stored in generation order, unsorted
    return ptr, ci, torch.rand(ci.numel(), generator=gen, device="cuda") * 2 - 1, (n, m)


CLUSTER_RUNS, CLUSTER_POOL = (8, 16, 24, 64, 72, 128), 32


def _clustered(case, gen):
    """Runs of neighbouring rows; a run's rows share most of their columns, share none, or share a few of them."""
    n, m = case["rows"], case["cols"]
    lengths = torch.tensor(CLUSTER_RUNS, device="cuda")[torch.randint(0, len(CLUSTER_RUNS), (n // CLUSTER_RUNS[0] + 1,), generator=gen, device="cuda")]
    run = torch.searchsorted(torch.cumsum(lengths, 0), torch.arange(n, device="cuda"), right=True)
    runs = int(lengths.numel())
    style = torch.randint(0, 3, (runs,), generator=gen, device="cuda")[run]
    base = torch.randint(0, m - 200, (runs,), generator=gen, device="cuda")
    pool = torch.topk(torch.rand((runs, 200), generator=gen, device="cuda"), CLUSTER_POOL, dim=1).indices + base[:, None]
    shared = torch.where(style[:, None] == 0, torch.rand((n, CLUSTER_POOL), generator=gen, device="cuda") < 0.8,
                         (style[:, None] == 2) & (torch.arange(CLUSTER_POOL, device="cuda")[None, :] < 6))
    r0, q = torch.nonzero(shared, as_tuple=True)
    alone = torch.tensor([0, 6, 3], device="cuda")[style]
    r1 = torch.arange(n, device="cuda").repeat_interleave(alone)
    c1 = torch.randint(0, m, (r1.numel(),), generator=gen, device="cuda")
    ptr, ci = _csr(torch.cat([r0, r1]), torch.cat([pool[run[r0], q], c1]), (n, m), gen, shuffle=True)
    return ptr, ci, _normal(ci.numel(), gen), (n, m)


def _stencil(case, gen):
    """27-point stencil on grid^3, x fastest, neighbours outside dropped; 26 on the diagonal, -1 elsewhere, with jitter."""
    g = case["grid"]
    n = g ** 3
    i = torch.arange(n, device="cuda")[:, None]
    o = torch.arange(27, device="cuda")[None, :]
    dx, dy, dz = o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1
    x, y, z = i % g + dx, i // g % g + dy, i // (g * g) + dz
    ok = (x >= 0) & (x < g) & (y >= 0) & (y < g) & (z >= 0) & (z < g)
    ci = (x + y * g + z * g * g)[ok].to(torch.int32)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(ok.sum(1), 0)
    v = torch.where((o == 13).expand(n, 27)[ok], 26.0, -1.0)
    return ptr.to(torch.int32), ci, v + (torch.rand(v.numel(), generator=gen, device="cuda") * 2 - 1) * 1e-3, (n, n)


def _mixed(case, gen):
    """A tenth of the 64-row panels hold four half-full 64x64 blocks; every other row has four entries anywhere."""
    n = case["rows"]
    panels = n // 64
    order = torch.randperm(panels, generator=gen, device="cuda")
    dense = order[:max(1, round(panels / 10))]
    sparse = torch.ones(panels, dtype=torch.bool, device="cuda")
    sparse[dense] = False
    rs = torch.nonzero(sparse.repeat_interleave(64)).reshape(-1).repeat_interleave(4)
    cs = torch.randint(0, n, (rs.numel(),), generator=gen, device="cuda")
    at = torch.randint(0, panels, (dense.numel(), 4), generator=gen, device="cuda")
    p, b, r, c = torch.nonzero(torch.rand((dense.numel(), 4, 64, 64), generator=gen, device="cuda") < 0.5, as_tuple=True)
    ptr, ci = _csr(torch.cat([rs, dense[p] * 64 + r]), torch.cat([cs, at[p, b] * 64 + c]), (n, n), gen)
    return ptr, ci, _normal(ci.numel(), gen), (n, n)


def _blocks(case, gen):
    n, k = case["rows"], case["block"]
    b, r, c = torch.nonzero(torch.rand((n // k, k, k), generator=gen, device="cuda") < case["density"], as_tuple=True)
    ptr, ci = _csr(b * k + r, b * k + c, (n, n), gen)
    return ptr, ci, _normal(ci.numel(), gen), (n, n)


def _banded(case, gen):
    n, h = case["rows"], case["half"]
    keep = torch.rand((n, 2 * h + 1), generator=gen, device="cuda") < 0.6
    keep[:, h] = True
    r, d = torch.nonzero(keep, as_tuple=True)
    c = r + d - h
    ok = (c >= 0) & (c < n)
    ptr, ci = _csr(r[ok], c[ok], (n, n), gen)
    return ptr, ci, _normal(ci.numel(), gen), (n, n)


def _matrix(case, seed):
    if case["family"] == "rmat":
        return synth.rmat_symmetric_device(case["scale"], 16, 1003 + seed, values=case["values"])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1003 + seed)
    return {"fixed": _fixed, "clustered": _clustered, "stencil": _stencil, "mixed": _mixed, "blocks": _blocks, "banded": _banded}[case["family"]](case, gen)


def _rhs(case, cols, width, seed):
    """Dense operand on the GPU: U[-1, 1] for FP16, N(0, 1) for TF32; the columns beyond the logical width are zero."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7 + seed)
    if case["precision"] == "fp16":
        b = torch.rand((cols, width), generator=gen, device="cuda") * 2 - 1
    else:
        b = torch.randn((cols, width), generator=gen, device="cuda")
    b[:, case["colB"]:] = 0
    return b.to(DTYPE[case["precision"]])


# ---------------------------------------------------------------------------------------------------------------

def _thresholds(precision, shape, rowptr, colB):
    major, minor = torch.cuda.get_device_capability()
    return api.predict(precision, api.features_from_csr(rowptr, shape, major + minor / 10.0, colB))


def _host(t):
    """Ordinary (pageable) numpy array of a GPU tensor; FP16 as bit patterns, as the host entry points take it."""
    a = t.cpu().numpy()
    return a.view(np.uint16) if a.dtype == np.float16 else a


def prepare(case, seed):
    precision, width = PRECISION[case["precision"]], api.padded_width(case["colB"])
    ptr, ci, v, shape = _matrix(case, seed)
    v = v.to(DTYPE[case["precision"]])
    m = api.TileMatrix(precision, torch.cuda.current_device())
    s = {"kind": case["kind"], "m": m, "shape": shape, "width": width, "colB": case["colB"], "precision": precision,
         "stream": torch.cuda.current_stream().cuda_stream}
    c_rows = (shape[0] + 64) // 64 * 64
    if case["kind"] == "once_host":
        s["csr"] = tuple(_host(t) for t in (ptr, ci, v))
    else:
        s["thresholds"] = _thresholds(precision, shape, ptr.cpu().numpy(), case["colB"])
    if case["kind"] == "once":
        s["csr"] = (ptr, ci, v)
    if case["kind"] in ("spmm", "host", "stream"):
        m.convert_device(shape, ptr, ci, v, ci.numel(), *s["thresholds"])
        m.info()
    if case["kind"] in ("spmm", "once", "once_host"):
        s["b"] = _rhs(case, shape[1], width, seed)
        s["c"] = torch.empty((c_rows, width), dtype=torch.float32, device="cuda")
    if case["kind"] == "spmm":
        m.tune(s["b"], s["c"], width)
    elif case["kind"] == "host":
        s["b"] = _host(_rhs(case, shape[1], width, seed))
    elif case["kind"] == "stream":
        s["b"] = [_rhs(case, shape[1], width, seed + 101 * k).cpu().pin_memory() for k in range(2)]
        s["c"] = [torch.empty((shape[0], width), dtype=torch.float32).pin_memory() for _ in range(STREAM_STEPS)]
    return s


def _stream(s):
    m, slots = s["m"], 2
    for i in range(STREAM_STEPS):
        if i >= slots:
            api._check(m.L.tsp_spmm_host_wait(m.h, i % slots), "tsp_spmm_host_wait")
        api._check(m.L.tsp_spmm_host_async(m.h, ctypes.c_void_p(s["b"][i % 2].data_ptr()), ctypes.c_void_p(s["c"][i].data_ptr()), s["width"], i % slots),
                   "tsp_spmm_host_async")
    for slot in range(slots):
        api._check(m.L.tsp_spmm_host_wait(m.h, slot), "tsp_spmm_host_wait")
    return s["c"]


def run(s):
    m, rows, kind = s["m"], s["shape"][0], s["kind"]
    if kind == "host":
        return m.spmm_host(s["b"], s["width"])
    if kind == "stream":
        return _stream(s)
    if kind == "spmm":
        m.spmm(s["b"], s["c"], s["width"], s["stream"])
        return s["c"][:rows]
    if kind == "once":
        ptr, ci, v = s["csr"]
        m.convert_device(s["shape"], ptr, ci, v, ci.numel(), *s["thresholds"])
    else:
        ptr, ci, v = s["csr"]
        m.convert_host(s["shape"], ptr, ci, v, *_thresholds(s["precision"], s["shape"], ptr, s["colB"]))
    m.spmm(s["b"], s["c"], s["width"], s["stream"])
    return {"tiles": m.info(), "c": s["c"][:rows]}


# ---------------------------------------------------------------------------------------------------------------

def _shape_and_entries(case):
    """(rows, cols, expected number of stored entries) without making the matrix."""
    f = case["family"]
    if f == "fixed":
        n, m, k = case["rows"], case["cols"], case["per_row"]
        return n, m, n * m * -math.expm1(k * math.log1p(-1.0 / m))
    if f == "clustered":
        return case["rows"], case["cols"], case["rows"] * (0.8 * CLUSTER_POOL + 6 + 9) / 3
    if f == "stencil":
        g = case["grid"]
        return g ** 3, g ** 3, (3 * g - 2) ** 3
    if f == "rmat":
        # distinct symmetrised pairs of 16 * 2^scale samples: cells grouped by how often each quadrant was taken
        s, a, b, d, total = case["scale"], 0.57, 0.19, 0.05, 0.0
        for i in range(s + 1):
            for j in range(1, s + 1 - i):   # j = 0 is the diagonal, which is dropped
                cells = math.comb(s, i) * math.comb(s - i, j) * 2.0 ** j
                total += cells * -math.expm1(-2.0 * 16 * 2.0 ** s * a ** i * b ** j * d ** (s - i - j))
        return 1 << s, 1 << s, total
    if f == "mixed":
        n = case["rows"]
        dense = max(1, round(n // 64 / 10))
        return n, n, dense * 4 * 2048 + (n - dense * 64) * 4
    if f == "blocks":
        return case["rows"], case["rows"], case["rows"] * case["block"] * case["density"]
    n, h = case["rows"], case["half"]
    return n, n, n * (1 + 1.2 * h) - 0.6 * h * (h + 1)


def work(case):
    rows, cols, nnz = _shape_and_entries(case)
    width, size = api.padded_width(case["colB"]), 2 if case["precision"] == "fp16" else 4
    a, b, c = nnz * (4 + size) + (rows + 1) * 4, cols * width * size, rows * width * 4
    flops = 2.0 * nnz * width
    if case["kind"] == "stream":   # the matrix stays on the GPU; operands and results move once per right-hand side
        return {"bytes": float(STREAM_STEPS * (a + b + c)), "flops": STREAM_STEPS * flops}
    return {"bytes": float(a + b + c), "flops": flops}


def tolerance(case):
    """Products of FP16 or TF32-truncated inputs are exact in FP32; what differs is the order of the 32-bit sums (the
    largest rows of a power-law graph add up 10^4 - 10^5 terms)."""
    return {"rel": 1e-5}
