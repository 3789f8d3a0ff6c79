"""GPU: gathered blocks (sparse blocks taken apart into columns) against FP64,
at the sizes where they can go wrong: N around the 64-column halves and
128-column tiles of the packed B, every form, both block heights, every panel
height, B in both layouts, hub rows and split panels, 256-column passes and a
short pipeline; and the NaNs and infinities that a block's stored zeros make
of such values in B, against the product of the exported blocks.

Tolerances (relative Frobenius, as the other GPU tests): FP16 1e-3, BF16 1e-2,
split 1e-4, FP8 1e-5 against its own codes and scales."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch.device("cuda", 0)


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def matrix(smat, kind, rows, cols, seed):
    """graph: scattered entries and a few hub rows; mixed: one block in five dense, the rest nearly empty."""
    rng = np.random.default_rng(seed)
    d = np.full((rows, cols), 0.006)
    if kind == "graph":
        d[rng.integers(0, rows, 3)] = 0.5
    else:
        d[((np.arange(rows)[:, None] // 16) + (np.arange(cols)[None, :] // 16)) % 5 == 0] = 0.5
    m = rng.random((rows, cols)) < d
    rp = np.concatenate([[0], np.cumsum(m.sum(1))])
    return smat.Csr(rows, cols, rp, np.nonzero(m)[1].astype(np.int32), rng.standard_normal(rp[-1]).astype(np.float32))


def dense(A):
    D = np.zeros((A.rows, A.cols))
    D[np.repeat(np.arange(A.rows), np.diff(A.row_ptr)), A.col_idx] = A.values
    return D


def blocks_product(M, B):
    """C of the exported blocks in FP64: every stored zero takes part."""
    rp, ci, v, _ = M.export()
    bh, i = v.shape[1], M.info
    Bp = np.zeros((i["cols_padded"], B.shape[1]))
    Bp[: B.shape[0]] = B
    out = np.zeros((i["rows_padded"], B.shape[1]))
    with np.errstate(all="ignore"):
        for r in range(len(rp) - 1):
            for k in range(rp[r], rp[r + 1]):
                out[r * bh:(r + 1) * bh] += v[k].astype(np.float64) @ Bp[ci[k]: ci[k] + 16]
    return out[: i["rows"]]


@pytest.mark.parametrize("N", [1, 63, 64, 65, 129, 200])
@pytest.mark.parametrize("form,tol", [("F16", 1e-3), ("BF16", 1e-2), ("SPLIT_BF16", 1e-4), ("FP8", 1e-5)])
@pytest.mark.parametrize("kind", ["graph", "mixed"])
def test_forms_and_widths(dev, smat_mod, kind, form, tol, N):
    f = getattr(smat_mod, "FORM_" + form)
    A = matrix(smat_mod, kind, 517, 1203, 3)
    M = smat_mod.Bcsr(A, forms=(f,))
    Bh = np.random.default_rng(N).standard_normal((A.cols, N)).astype(np.float32)
    B = torch.from_numpy(Bh).to(dev)
    if N % 2:
        B = B.t().contiguous().t()
    Cm = M.spmm(B, form=f).cpu().numpy()
    M.check_device_error()
    if form == "F16":
        ref = dense(A).astype(np.float16).astype(np.float64) @ Bh.astype(np.float16).astype(np.float64)
    elif form == "FP8":
        n = M.info["nnzb"]
        codes, scales = np.zeros(n * 256, np.uint8), np.zeros(n, np.float32)
        smat_mod.lib().smat_bcsr_export_fp8(M.handle, C.c_void_p(codes.ctypes.data), C.c_void_p(scales.ctypes.data))
        val = torch.from_numpy(codes).view(torch.float8_e4m3fn).float().numpy().reshape(n, 16, 16)
        val = (val * scales[:, None, None]).astype(np.float16).astype(np.float64)
        rp, ci, _, _ = M.export()
        Bp = np.zeros((M.info["cols_padded"], N))
        Bp[: A.cols] = Bh.astype(np.float16)
        ref = np.zeros((M.info["rows_padded"], N))
        for r in range(len(rp) - 1):
            for k in range(rp[r], rp[r + 1]):
                ref[r * 16:(r + 1) * 16] += val[k] @ Bp[ci[k]: ci[k] + 16]
        ref = ref[: A.rows]
    else:
        ref = dense(A) @ Bh.astype(np.float64)
    assert rel(Cm, ref) <= tol, rel(Cm, ref)


@pytest.mark.parametrize("bh,R,ntc,frac,depth", [(16, 4, 0, 0.0, 0), (16, 8, 256, 0.0, 0), (16, 8, 0, 0.05, 2),
                                                (16, 16, 0, 0.05, 0), (32, 4, 0, 0.0, 2), (32, 8, 0, 0.05, 0)])
@pytest.mark.parametrize("kind", ["graph", "mixed"])
def test_panels_splits_and_depths(dev, smat_mod, kind, bh, R, ntc, frac, depth):
    A = matrix(smat_mod, kind, 1500, 2100, 5)
    M = smat_mod.Bcsr(A, block=(bh, 16), panel_rows=R, n_tile_cols=ntc, split_frac=frac, pipeline_depth=depth)
    Bh = np.random.default_rng(R).uniform(-1, 1, (A.cols, 321)).astype(np.float16)
    ref = dense(A).astype(np.float16).astype(np.float64) @ Bh.astype(np.float64)
    B = torch.from_numpy(Bh).to(dev)
    one = M.spmm(B).cpu().numpy()
    two = M.spmm(B).cpu().numpy()
    M.check_device_error()
    assert rel(one, ref) <= 1e-3, rel(one, ref)
    assert np.array_equal(one, two)


@pytest.mark.parametrize("form", ["F16", "BF16", "SPLIT_BF16"])
@pytest.mark.parametrize("frac", [0.0, 0.05])
@pytest.mark.parametrize("layout", ["row", "col"])
def test_infinite_and_nan_b(dev, smat_mod, form, frac, layout):
    f = getattr(smat_mod, "FORM_" + form)
    A = matrix(smat_mod, "graph", 700, 1900, 11)
    M = smat_mod.Bcsr(A, forms=(f,), split_frac=frac)
    N = 150
    rng = np.random.default_rng(2)
    Bh = rng.uniform(-1, 1, (A.cols, N)).astype(np.float32)
    for q in range(8):
        Bh[rng.integers(0, A.cols), rng.integers(0, N)] = [np.inf, -np.inf, np.nan][q % 3]
    B = torch.from_numpy(Bh).to(dev)
    if layout == "col":
        B = B.t().contiguous().t()
    Cm = M.spmm(B, form=f).cpu().numpy()
    M.check_device_error()
    ref = blocks_product(M, Bh.astype(np.float64))
    bad = ~np.isfinite(ref)
    assert bad.any() and not bad.all()
    if form == "SPLIT_BF16":  # hi - lo of an infinity is NaN: any non-finite value will do
        assert np.array_equal(~np.isfinite(Cm), bad)
    else:
        assert np.array_equal(np.isnan(Cm), np.isnan(ref))
        assert np.array_equal(Cm[np.isinf(ref)], ref[np.isinf(ref)])
    assert rel(Cm[~bad], ref[~bad]) <= 1e-2
    # the same handle on finite values again
    Bh = np.nan_to_num(Bh, nan=0.0, posinf=0.0, neginf=0.0)
    Cm = M.spmm(torch.from_numpy(Bh).to(dev), form=f).cpu().numpy()
    assert np.isfinite(Cm).all()
