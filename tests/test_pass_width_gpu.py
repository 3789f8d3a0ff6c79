"""GPU: 256-column passes are for the panel heights that a caller names (8 block rows or
fewer): without one the handle runs 128 columns a pass, whatever height the number
of panels leads to, and holds one copy of A."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1000, 180000])
@pytest.mark.parametrize("bh", [16, 32])
def test_width_with_and_without_a_panel_height(smat_mod, rows, bh):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from smat import generators as G
    smat_mod.lib().smat_autotune_clear()
    A = G.band(rows, 3, seed=1)
    B = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (A.cols, 200)).astype(np.float16)).cuda()
    M = smat_mod.Bcsr(A, block=(bh, 16), n_tile_cols=256)
    assert M.info["n_tile_cols"] == 128
    one = M.spmm(B)
    W = smat_mod.Bcsr(A, block=(bh, 16), n_tile_cols=256, panel_rows=8)
    assert W.info["n_tile_cols"] == (256 if bh == 16 else 128)
    two = W.spmm(B)
    torch.cuda.synchronize()
    assert float((one - two).norm() / one.norm()) <= 1e-5
