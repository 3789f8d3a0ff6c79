"""GPU: a launcher of the reference's harness whose partial sums do not fit in the
static scratch beside the packed B runs with split panels in a workspace of its
own, as smat_spmm does with one: the same bits (FP32 sums in another order would
round to another FP16 somewhere), and within 1e-3 of FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch.device("cuda", 0)


def heavy(smat, rng, rows, cols):
    d = np.full((rows, cols), 0.0005)
    d[:1024] = 0.3
    m = rng.random((rows, cols)) < d
    v = rng.uniform(-1, 1, int(m.sum())).astype(np.float16).astype(np.float32)
    return smat.Csr(rows, cols, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32), v)


def test_shim_splits_panels(dev, smat_mod):
    import scipy.sparse as sps
    from smat import _lib
    rng = np.random.default_rng(2)
    A = heavy(smat_mod, rng, 4096, 8192)
    N = 1024
    M = smat_mod.Bcsr(A)
    assert M.workspace_size(smat_mod.FORM_F16, smat_mod.F16, N) > (32 << 20)    # 16 MiB of it are B
    rp, ci, v = smat_mod.csr_to_bcsr_host(A, block=(16, 16))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    dv, drp, dci = t(v.reshape(-1).view(np.int16)).view(torch.float16), t(rp), t(ci)
    Bh = rng.uniform(-1, 1, (A.cols, N)).astype(np.float16)
    Bc = torch.from_numpy(Bh).to(dev).t().contiguous()
    out = torch.zeros((A.rows, N), dtype=torch.float16, device=dev)
    _lib.ref_shim("mmaOBTKernel")(dv.data_ptr(), drp.data_ptr(), dci.data_ptr(), Bc.data_ptr(), out.data_ptr(), A.rows, N,
                                  A.cols, len(ci), None, None)
    torch.cuda.synchronize()
    one = M.spmm(Bc.t(), out_dtype=torch.float16)
    assert torch.equal(out, one)
    ref = sps.csr_matrix((A.values.astype(np.float64), A.col_idx, A.row_ptr), shape=(A.rows, A.cols)) @ Bh.astype(np.float64)
    assert np.linalg.norm(out.cpu().numpy().astype(np.float64) - ref) <= 1e-3 * np.linalg.norm(ref)
