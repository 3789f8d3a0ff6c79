"""GPU: work split over CTAs. The 2:4 path's groups cut into parts (few groups,
many windows) against FP64 at widths around a column tile, with FP32 and FP16
C, bit-identical on repetition; and the static scratch when the partial sums
of split panels do not fit beside the packed B (panels then stay whole).

Tolerances (relative Frobenius, as the other GPU tests): FP16 1e-3, BF16 1e-2."""
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


def csr(smat, D):
    m = D != 0
    return smat.Csr(D.shape[0], D.shape[1], np.concatenate([[0], np.cumsum(m.sum(1))]),
                    np.nonzero(m)[1].astype(np.int32), D[m])


@pytest.mark.parametrize("N", [1, 100, 128, 130])
@pytest.mark.parametrize("form,tol,c_dt", [("F16", 1e-3, "float32"), ("F16", 2e-3, "float16"), ("BF16", 1e-2, "float32")])
def test_split_24_groups(dev, smat_mod, form, tol, c_dt, N):
    rng = np.random.default_rng(7)
    rows, cols = 200, 6000                       # two groups of 128 rows, 188 windows each
    D = np.zeros((rows, cols), np.float16)
    for q in range(0, cols, 4):                  # two of four in every group of columns
        pick = rng.integers(0, 2, rows)
        D[np.arange(rows), q + pick] = rng.standard_normal(rows)
        D[np.arange(rows), q + 2 + pick] = rng.standard_normal(rows)
    f = getattr(smat_mod, "FORM_" + form)
    A = csr(smat_mod, D)
    M = smat_mod.Bcsr(A, forms=(f,), use_24=1)
    assert M.info["n_blocks_24"] == M.info["nnzb"]
    Bh = rng.uniform(-1, 1, (cols, N)).astype(np.float32)
    B = torch.from_numpy(Bh).to(dev)
    one = M.spmm(B, form=f, out_dtype=getattr(torch, c_dt)).cpu().numpy()
    two = M.spmm(B, form=f, out_dtype=getattr(torch, c_dt)).cpu().numpy()
    M.check_device_error()
    ref = D.astype(np.float64) @ (Bh.astype(np.float16) if form == "F16" else Bh).astype(np.float64)
    assert rel(one, ref) <= tol, rel(one, ref)
    assert np.array_equal(one, two)


def test_static_scratch_without_room_for_partial_sums(dev, smat_mod):
    rng = np.random.default_rng(3)
    rows, cols, N = 1024, 2048, 4096
    D = np.where(rng.random((rows, cols)) < 0.3, rng.standard_normal((rows, cols)), 0.0).astype(np.float16)
    M = smat_mod.Bcsr(csr(smat_mod, D), split_frac=0.02)
    assert M.workspace_size(smat_mod.FORM_F16, smat_mod.F16, N) > (32 << 20)   # 16 MiB of it are B
    B = torch.from_numpy(rng.uniform(-1, 1, (cols, N)).astype(np.float16)).to(dev)
    out = torch.full((rows, N), float("nan"), dtype=torch.float32, device=dev)
    ref = D.astype(np.float64) @ B.cpu().numpy().astype(np.float64)
    L = smat_mod.lib()
    st = L.smat_spmm_static_scratch(M.handle, smat_mod.FORM_F16, C.c_void_p(B.data_ptr()), smat_mod.F16,
                                    smat_mod.ROW_MAJOR, N, C.c_void_p(out.data_ptr()), smat_mod.F32, N, N,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, L.smat_last_error().decode()
    torch.cuda.synchronize()
    M.check_device_error()
    assert rel(out.cpu().numpy(), ref) <= 1e-3
    assert rel(M.spmm(B).cpu().numpy(), ref) <= 1e-3
