"""GPU: matrices whose blocks are all on the 2:4 path, which then writes C
itself (no dense kernel before it): block rows and whole groups of eight of
them without a block, C full of NaN before the call and wider than N, rows
permuted, groups whole and split, both entry points; against FP64.

Tolerances (relative Frobenius, as the other GPU tests): FP32 C 1e-3, FP16 C
2e-3; rows without a block are exactly zero, also where B is infinite."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch.device("cuda", 0)


def matrix(rng, rows, cols):
    D = np.zeros((rows, cols), np.float16)
    for q in range(0, cols, 4):                  # two of four in every group of columns
        pick = rng.integers(0, 2, rows)
        D[np.arange(rows), q + pick] = rng.standard_normal(rows)
        D[np.arange(rows), q + 2 + pick] = rng.standard_normal(rows)
    D[16:32] = 0                                 # a block row
    D[256:400] = 0                               # a group and a block row (where there are so many)
    return D


@pytest.mark.parametrize("N", [1, 100, 128, 130])
@pytest.mark.parametrize("c_dt,tol", [("float32", 1e-3), ("float16", 2e-3)])
@pytest.mark.parametrize("rows,cols", [(1000, 512), (200, 6000)])
def test_all_blocks_24(dev, smat_mod, rows, cols, c_dt, tol, N):
    rng = np.random.default_rng(11)
    D = matrix(rng, rows, cols)
    perm = rng.permutation(rows) if N == 130 else None
    E = np.zeros_like(D)
    if perm is None:
        E = D
    else:                                        # new row r = old row perm[r]
        E[perm] = D
    m = E != 0
    A = smat_mod.Csr(rows, cols, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32), E[m])
    M = smat_mod.Bcsr(A, use_24=1, row_perm=perm)
    assert M.info["n_blocks_24"] == M.info["nnzb"]
    Bh = rng.uniform(-1, 1, (cols, N)).astype(np.float16)
    ref = E.astype(np.float64) @ Bh.astype(np.float64)
    empty = ~m.any(1)
    code = smat_mod.F32 if c_dt == "float32" else smat_mod.F16
    n = M.workspace_size(smat_mod.FORM_F16, smat_mod.F16, N)
    ws = torch.empty(n, dtype=torch.uint8, device=dev)
    B = torch.from_numpy(Bh).to(dev)
    sp = torch.cuda.current_stream().cuda_stream
    for packed in (False, True):
        out = torch.full((rows, N + 3), float("nan"), dtype=getattr(torch, c_dt), device=dev)
        if packed:
            M.pack_b(smat_mod.FORM_F16, B, smat_mod.F16, smat_mod.ROW_MAJOR, N, N, ws, n, sp)
            M.spmm_packed(smat_mod.FORM_F16, ws, N, out, code, N + 3, sp)
        else:
            M.spmm_raw(smat_mod.FORM_F16, B, smat_mod.F16, smat_mod.ROW_MAJOR, N, out, code, N + 3, N, ws, n, sp)
        got = out.cpu().numpy()
        assert np.isnan(got[:, N:]).all()
        assert np.linalg.norm(got[:, :N].astype(np.float64) - ref) <= tol * np.linalg.norm(ref)
        assert (got[empty, :N] == 0).all()
    B[0, :] = float("inf")
    M.spmm_raw(smat_mod.FORM_F16, B, smat_mod.F16, smat_mod.ROW_MAJOR, N, out, code, N + 3, N, ws, n, sp)
    M.check_device_error()
    assert (out.cpu().numpy()[empty, :N] == 0).all()
