"""The work that users of this package have it do, as cases that can be timed.

Almost all of it is the SpMM C = A * B of a handle that was built once from a
sparse matrix (a graph, a banded or stencil operator, a block-pruned weight)
with dense right-hand sides that change from call to call; around it stand the
grouped launch of many small matrices, the call on host buffers and the
merged-tile build on the GPU. Every case goes through the public entry points.

Matrices are drawn on the GPU from the seed and handed over as host CSR arrays,
as a program that has read a file or built a graph holds them.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "sptc-smat_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "sptc-smat_gb300"))

import smat  # noqa: E402

DEV = "cuda:0"
FORMS = {"f16": smat.FORM_F16, "bf16": smat.FORM_BF16, "fp8": smat.FORM_FP8, "split": smat.FORM_SPLIT_BF16}
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest operator somebody multiplies with in a loop: a narrow band, eight
        # right-hand sides (the width at which the reference reports its band results);
        # launches and host time count
        {"name": "band_1k_n8", "kind": "spmm", "family": "band", "rows": 1024, "half": 16, "N": 8, "form": "f16",
         "b": "f16", "layout": "row", "c": "f32"},
        # the small band workload: 4096 rows, half-bandwidth 64, 64 right-hand sides
        {"name": "band_4k_n64", "kind": "spmm", "family": "band", "rows": 4096, "half": 64, "N": 64, "form": "f16",
         "b": "f16", "layout": "row", "c": "f32"},
        # the scale-free workload: 2^16 rows, 2M entries, 30 % of the blocks exactly 2:4, rows
        # brought into a good order by a permutation, B column-major as the reference has it
        {"name": "rmat_64k_n128", "kind": "spmm", "family": "rmat", "scale": 16, "nnz": 2000000, "force24": 0.3,
         "N": 128, "form": "f16", "b": "f16", "layout": "col", "c": "f32", "perm": True, "keep": True},
        # a plain graph (nothing rewritten) times node features in BF16: graph aggregation,
        # rows in the order of the file
        {"name": "graph_32k_n256_bf16", "kind": "spmm", "family": "rmat", "scale": 15, "nnz": 600000, "force24": 0.0,
         "N": 256, "form": "bf16", "b": "bf16", "layout": "row", "c": "f32", "perm": False, "keep": True},
        # the three precision forms on the 27-point stencil operator (a block of FP32 vectors
        # through a discretised PDE): the full 64^3 grid in FP16 ...
        {"name": "stencil_64_n256", "kind": "spmm", "family": "stencil", "nx": 64, "ny": 64, "nz": 64, "N": 256,
         "form": "f16", "b": "f32", "layout": "row", "c": "f32", "keep": True},
        # ... near-FP32 by the split form on a grid of odd sides and a ragged width ...
        {"name": "stencil_odd_split_n100", "kind": "spmm", "family": "stencil", "nx": 47, "ny": 39, "nz": 53, "N": 100,
         "form": "split", "b": "f32", "layout": "row", "c": "f32"},
        # ... and FP8 blocks with scales
        {"name": "stencil_48_fp8_n256", "kind": "spmm", "family": "stencil", "nx": 48, "ny": 48, "nz": 48, "N": 256,
         "form": "fp8", "b": "f32", "layout": "row", "c": "f32"},
        # a block-pruned rectangular weight on a ragged batch of activations, FP16 in and out,
        # 32 x 16 blocks
        {"name": "blocks_ragged_n200", "kind": "spmm", "family": "blocks", "rows": 5003, "cols": 7001, "density": 0.08,
         "fill": 0.9, "N": 200, "form": "f16", "b": "f16", "layout": "row", "c": "f16", "bh": 32},
        # a 2:4-pruned block-sparse weight on the structured-sparse path
        {"name": "pruned24_n128", "kind": "spmm", "family": "blocks24", "rows": 8192, "cols": 8192, "density": 0.12,
         "N": 128, "form": "f16", "b": "f16", "layout": "col", "c": "f32", "use24": 1},
        # many uneven matrices in one grouped launch (band / R-MAT / random blocks in turn)
        {"name": "group_24", "kind": "group", "count": 24, "lo": 1024, "hi": 8192},
        # the call on page-locked host buffers, B in and C out over the CPU-GPU link
        {"name": "host_16k_n128", "kind": "host", "family": "rmat", "scale": 14, "nnz": 400000, "force24": 0.0,
         "N": 128, "form": "f16", "b": "f16", "layout": "row", "c": "f32", "perm": False},
        # the merged 4 x 4-block tiles of a graph's BCSR, built on the GPU
        {"name": "tiles_8k", "kind": "tiles", "family": "rmat", "scale": 13, "nnz": 120000, "force24": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any family, form, type and layout at any size up to the listed ones'."""
    kind = rng.choice(["spmm"] * 9 + ["group", "host", "tiles"])
    if kind == "group":
        lo = _log(rng, 512, 2048)
        return {"kind": "group", "count": rng.randint(4, 24), "lo": lo, "hi": min(8192, lo * rng.choice([2, 4, 8]))}
    family = "rmat" if kind == "tiles" else rng.choice(["band", "rmat", "rmat", "stencil", "blocks"])
    c = {"kind": kind, "family": family}
    if family == "band":
        c["rows"] = _log(rng, 700, 40000)
        c["half"] = _log(rng, 4, 256)
    elif family == "rmat":
        c["scale"] = rng.randint(10, 13 if kind == "tiles" else 15)
        c["nnz"] = int((1 << c["scale"]) * _log(rng, 4, 30))
        c["force24"] = rng.choice([0.0, 0.0, 0.0, 0.3])
        c["perm"] = kind != "tiles" and rng.random() < 0.5
    elif family == "stencil":
        c["nx"], c["ny"], c["nz"] = (_log(rng, 9, 56) for _ in range(3))
    else:
        c["rows"], c["cols"] = _log(rng, 500, 9000), _log(rng, 500, 9000)
        c["density"] = round(math.exp(rng.uniform(math.log(0.01), math.log(0.3))), 4)
        c["fill"] = round(rng.uniform(0.3, 1.0), 3)
    if kind == "tiles":
        return c
    form = rng.choice(["f16", "f16", "f16", "bf16", "bf16", "split", "fp8"])
    c["form"] = form
    c["b"] = rng.choice(["f32", form]) if form in ("f16", "bf16") else "f32"
    if kind == "host":
        c["form"] = form = rng.choice(["f16", "split"])
        c["b"] = rng.choice(["f32", "f16"]) if form == "f16" else "f32"
    c["N"] = _log(rng, 4, 320)
    c["layout"] = rng.choice(["row", "col"]) if kind != "host" else "row"
    c["c"] = rng.choice(["f32", "f32", "f16"])
    if form in ("f16", "bf16") and rng.random() < 0.15:
        c["bh"] = 32
    return c


# ------------------------------------------------------------------ matrices
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _band(n, half, g):
    d = torch.arange(-half, half + 1, device=DEV)
    r = torch.arange(n, device=DEV).repeat_interleave(d.numel())
    k = r + d.repeat(n)
    ok = (k >= 0) & (k < n)
    r, k = r[ok], k[ok]
    v = torch.rand(r.numel(), generator=g, device=DEV) * 2 - 1
    return n, n, r * n + k, v.half()


def _stencil(nx, ny, nz, g):
    n = nx * ny * nz
    i = torch.arange(n, device=DEV)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    keys = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz)
                r = i[ok]
                keys.append(r * n + r + (dz * ny + dy) * nx + dx)
    key = torch.sort(torch.cat(keys)).values
    v = 1.0 + 0.1 * torch.randn(key.numel(), generator=g, device=DEV)
    diag = key // n == key % n
    return n, n, key, torch.where(diag, 27.0 + (v - 1.0) * 10.0, v)


def _rmat(scale, nnz, force24, g):
    n = 1 << scale
    keys = torch.zeros(0, dtype=torch.int64, device=DEV)
    while keys.numel() < nnz:
        m = int((nnz - keys.numel()) * 1.3) + 1024
        r = torch.zeros(m, dtype=torch.int64, device=DEV)
        c = torch.zeros(m, dtype=torch.int64, device=DEV)
        for _ in range(scale):  # quadrants a, b, c, d = 0.57, 0.19, 0.19, 0.05
            u = torch.rand(m, generator=g, device=DEV)
            r = 2 * r + (u >= 0.76)
            c = 2 * c + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
        keys = torch.unique(torch.cat([keys, r * n + c]))
    keys = keys[torch.randperm(keys.numel(), generator=g, device=DEV)[:nnz]].sort().values
    if force24:
        nbc = (n + 15) // 16
        blk = (keys // n // 16) * nbc + (keys % n) // 16
        ub = torch.unique(blk)
        chosen = ub[torch.randperm(ub.numel(), generator=g, device=DEV)[: int(force24 * ub.numel())]]
        hit = torch.zeros(nbc * nbc, dtype=torch.bool, device=DEV)
        hit[chosen] = True
        keys = torch.cat([keys[~hit[blk]], _pairs24(chosen // nbc, chosen % nbc, n, g)]).sort().values
    return n, n, keys, torch.randn(keys.numel(), generator=g, device=DEV).half()


def _pairs24(br, bc, cols, g):
    """Keys of two entries in every aligned group of four columns of every row of the given 16 x 16 blocks."""
    two = torch.tensor([(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)], device=DEV)
    pick = two[torch.randint(0, 6, (br.numel(), 16, 4), generator=g, device=DEV)]
    row = br[:, None, None, None] * 16 + torch.arange(16, device=DEV)[None, :, None, None]
    col = bc[:, None, None, None] * 16 + torch.arange(4, device=DEV)[None, None, :, None] * 4 + pick
    return (row * cols + col).reshape(-1)


def _blocks(rows, cols, density, fill, pruned, g):
    nbr, nbc = (rows + 15) // 16, (cols + 15) // 16
    at = torch.randperm(nbr * nbc, generator=g, device=DEV)[: max(1, int(nbr * nbc * density))]
    br, bc = at // nbc, at % nbc
    if pruned:
        key = _pairs24(br, bc, cols, g)
    else:
        share = fill * (0.8 + 0.4 * torch.rand(at.numel(), 1, 1, generator=g, device=DEV))
        m = torch.rand(at.numel(), 16, 16, generator=g, device=DEV) < share
        k, rr, cc = m.nonzero(as_tuple=True)
        r, c = br[k] * 16 + rr, bc[k] * 16 + cc
        ok = (r < rows) & (c < cols)
        key = r[ok] * cols + c[ok]
    key = key.sort().values
    return rows, cols, key, torch.randn(key.numel(), generator=g, device=DEV).half()


def _coo(case, g):
    f = case["family"]
    if f == "band":
        return _band(case["rows"], case["half"], g)
    if f == "stencil":
        return _stencil(case["nx"], case["ny"], case["nz"], g)
    if f == "rmat":
        return _rmat(case["scale"], case["nnz"], case["force24"], g)
    return _blocks(case["rows"], case["cols"], case["density"], case.get("fill", 1.0), f == "blocks24", g)


class _Matrix:
    """A of a case: sorted row * cols + column keys and values on the GPU, and the host CSR. With `perm`, the
    rows of the CSR are shuffled and `row_perm` leads back to the order they were made in."""

    def __init__(self, case, g):
        if case.get("kind") == "tiles":  # one graph, other values: the number of tiles is the graph's
            rows, cols, key, val = _coo(case, _gen(1))
            val = torch.randn(key.numel(), generator=g, device=DEV).half()
        else:
            rows, cols, key, val = _coo(case, g)
        self.row_perm = None
        if case.get("perm"):
            place = torch.randperm(rows, generator=g, device=DEV)  # row r of the good order is row place[r] of the CSR
            key, by = torch.sort(place[key // cols] * cols + key % cols)
            val = val[by]
            self.row_perm = place.cpu().numpy()
        self.rows, self.cols, self.key, self.val = rows, cols, key, val

    def csr(self):
        ptr = torch.searchsorted(self.key, torch.arange(self.rows + 1, device=DEV) * self.cols)
        return smat.Csr(self.rows, self.cols, ptr.cpu().numpy(), (self.key % self.cols).int().cpu().numpy(),
                        self.val.cpu().numpy())

    def times(self, B):
        """A * B in 64 bits."""
        ptr = torch.searchsorted(self.key, torch.arange(self.rows + 1, device=DEV) * self.cols)
        return torch.sparse_csr_tensor(ptr, self.key % self.cols, self.val.double(),
                                       size=(self.rows, self.cols)) @ B.double()


def _dense(case, rows, g):
    B = torch.randn(rows, case["N"], generator=g, device=DEV).to(DTYPES[case["b"]])
    return B.t().contiguous().t() if case["layout"] == "col" else B


def _members(case):
    """The matrices of a grouped case, their sizes spread evenly over the range (by the case alone)."""
    out = []
    for i in range(case["count"]):
        u, w = (i * 0.6180339887) % 1.0, (i * 0.7548776662) % 1.0
        rows = int(case["lo"] * (case["hi"] / case["lo"]) ** u)
        if i % 3 == 0:
            m = {"family": "band", "rows": rows, "half": int(8 * 32 ** w)}
        elif i % 3 == 1:
            scale = max(9, int(math.log2(rows)))
            m = {"family": "rmat", "scale": scale, "nnz": int((8 + 40 * w) * (1 << scale)), "force24": 0.0}
        else:
            m = {"family": "blocks", "rows": rows, "cols": rows, "density": 0.01 + 0.04 * w, "fill": 0.65}
        form = "f16" if i % 2 == 0 else "bf16"
        m.update(N=(32, 64, 128)[int(((i * 0.5698402910) % 1.0) * 3)], b=form, c="f32", layout="row", form=form)
        out.append(m)
    return out


class _Ints:
    """A device array that the package owns, for torch to look at in place; keeps its owner alive."""

    def __init__(self, owner, addr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (addr, False), "version": 3}


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "group":
        probs = []
        for m in _members(case):
            A = _Matrix(m, g)
            M = smat.Bcsr(A.csr(), forms=(FORMS[m["form"]],))
            B = _dense(m, A.cols, g)
            probs.append((M, FORMS[m["form"]], B, torch.zeros(A.rows, m["N"], device=DEV)))
        return {"kind": "group", "group": smat.Group(probs), "out": [p[3] for p in probs]}
    A = _Matrix(case, g)
    if case["kind"] == "tiles":
        rp, ci, v = smat.csr_to_bcsr_host(A.csr())
        return {"kind": "tiles", "rows": A.rows, "cols": A.cols, "rp": torch.from_numpy(rp).to(DEV),
                "ci": torch.from_numpy(ci).to(DEV), "v": torch.from_numpy(v.reshape(-1)).to(DEV)}
    form = FORMS[case["form"]]
    M = smat.Bcsr(A.csr(), block=(case.get("bh", 16), 16), forms=(form,), row_perm=A.row_perm,
                  use_24=case.get("use24", 0))
    B = _dense(case, A.cols, g)
    s = {"kind": case["kind"], "M": M, "form": form, "B": B, "c": DTYPES[case["c"]]}
    if case["kind"] == "host":
        s["Bh"] = B.cpu().pin_memory()
        s["Ch"] = torch.zeros(A.rows, case["N"], dtype=s["c"]).pin_memory()
    elif case.get("keep"):
        b = {"f16": smat.F16, "bf16": smat.BF16, "f32": smat.F32}[case["b"]]
        s["ws"] = torch.empty(M.workspace_size(form, b, case["N"]), dtype=torch.uint8, device=DEV)
        s["out"] = torch.empty(A.rows, case["N"], dtype=s["c"], device=DEV)
    return s


def run(state):
    kind = state["kind"]
    if kind == "group":
        state["group"].run(stream=torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "tiles":
        T = smat.Tiles(state["rows"], state["cols"], 16, state["rp"], state["ci"], state["v"])
        d, (tr, tc) = T.desc, T.grid
        return {name: torch.as_tensor(_Ints(T, addr, shape, typ), device=DEV) for name, addr, shape, typ in (
            ("values", d.values, (T.n_tiles * 4096,), "<i2"), ("row_ptr", d.row_ptr, (T.n_rowptr,), "<i4"),
            ("col_idx", d.col_idx, (T.n_tiles,), "<i4"), ("block_info", d.block_info, (tr * tc,), "<i4"),
            ("rel_map", d.rel_map, (tr * tc,), "<i4"), ("tile_info", d.tile_info, (T.n_tiles * 16,), "<i4"))}
    if kind == "host":
        state["M"].spmm_host(state["Bh"].numpy(), form=state["form"], out=state["Ch"].numpy(),
                             stream=torch.cuda.current_stream().cuda_stream)
        return state["Ch"]
    return state["M"].spmm(state["B"], form=state["form"], out=state.get("out"), out_dtype=state["c"],
                           workspace=state.get("ws"))


# ------------------------------------------------------------------ what a pass cannot do without
def _nnz_of(case):
    """(rows, columns, expected entries) of a case's matrix."""
    f = case["family"]
    if f == "band":
        n, h = case["rows"], min(case["half"], case["rows"] - 1)
        return n, n, n * (2 * h + 1) - h * (h + 1)
    if f == "stencil":
        n = case["nx"] * case["ny"] * case["nz"]
        return n, n, (3 * case["nx"] - 2) * (3 * case["ny"] - 2) * (3 * case["nz"] - 2)
    if f == "rmat":
        n = 1 << case["scale"]
        # a rewritten block holds 128 entries; about 0.4 nonzero blocks per entry of these graphs
        return n, n, int(case["nnz"] * (1 + case["force24"] * 50))
    blocks = ((case["rows"] + 15) // 16) * ((case["cols"] + 15) // 16) * case["density"]
    return case["rows"], case["cols"], int(blocks * 256 * (0.5 if f == "blocks24" else case["fill"]))


def _work_one(case):
    rows, cols, nnz = _nnz_of(case)
    N = case["N"]
    a = {"f16": 2, "bf16": 2, "fp8": 1, "split": 4}[case["form"]]
    b, c = (4 if case["b"] == "f32" else 2), (2 if case.get("c") == "f16" else 4)
    # A as CSR (value and 32-bit column of each entry, a pointer of each row), B in, C out
    return nnz * (a + 4) + rows * 4 + cols * N * b + rows * N * c, 2 * nnz * N


def work(case):
    if case["kind"] == "group":
        each = [_work_one(m) for m in _members(case)]
        return {"bytes": sum(e[0] for e in each), "flops": sum(e[1] for e in each)}
    if case["kind"] == "tiles":
        rows, _, nnz = _nnz_of(case)
        blocks = 0.7 * nnz  # nonzero 16 x 16 blocks, 512 bytes in; tiles of 8 KB out, about two blocks in each
        return {"bytes": blocks * (512 + 4) + blocks / 2 * (8192 + 68), "flops": 0}
    b, f = _work_one(case)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ what it computes, in 64 bits
def exact(case, seed):
    g = _gen(seed)
    if case["kind"] == "tiles":
        return None  # a rearrangement of bytes
    if case["kind"] == "group":
        out = []
        for m in _members(case):
            A = _Matrix(m, g)
            out.append(A.times(_dense(m, A.cols, g)))
        return out
    A = _Matrix(case, g)
    C = A.times(_dense(case, A.cols, g))
    return C.cpu() if case["kind"] == "host" else C
