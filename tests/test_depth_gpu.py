"""GPU: the pipeline depth changes when a stage is copied, never what is
computed: every form gives the same bits with two and three stages in flight as
with all that fit (three; four for FP8, whose two sets of converter warps take
every other slot), over long and short units, hub rows and a ragged width."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch.device("cuda", 0)


@pytest.mark.parametrize("form", ["F16", "BF16", "FP8", "SPLIT_BF16"])
@pytest.mark.parametrize("rows,cols,density,N", [(300, 9000, 0.05, 100), (3000, 2000, 0.02, 130)])
def test_depth_gives_the_same_bits(dev, smat_mod, form, rows, cols, density, N):
    rng = np.random.default_rng(rows)
    D = np.where(rng.random((rows, cols)) < density, rng.standard_normal((rows, cols)), 0.0).astype(np.float32)
    D[5:8] = rng.standard_normal((3, cols))     # hub rows
    m = D != 0
    A = smat_mod.Csr(rows, cols, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32), D[m])
    B = torch.from_numpy(rng.uniform(-1, 1, (cols, N)).astype(np.float32)).to(dev)
    f = getattr(smat_mod, "FORM_" + form)
    ref = None
    for depth in (0, 2, 3):
        M = smat_mod.Bcsr(A, forms=(f,), panel_rows=8, pipeline_depth=depth)
        for _ in range(3):
            C = M.spmm(B, form=f).cpu()
            ref = C if ref is None else ref
            assert torch.equal(C, ref), depth
        M.check_device_error()
