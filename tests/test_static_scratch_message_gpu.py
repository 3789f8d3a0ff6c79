"""GPU: what the static scratch says when the packed B itself does not fit: the bytes
that it would need, without the partial sums of split panels, which may be left out."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_static_scratch_says_how_much_it_lacks(smat_mod):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(2)
    d = np.full((2048, 8192), 0.0005)
    d[:1024] = 0.3                                       # eight heavy panels: split, with partial sums
    m = rng.random(d.shape) < d
    v = rng.uniform(-1, 1, int(m.sum())).astype(np.float32)
    M = smat_mod.Bcsr(smat_mod.Csr(*d.shape, np.concatenate([[0], np.cumsum(m.sum(1))]),
                                   np.nonzero(m)[1].astype(np.int32), v))
    N = 2176                                             # K * N * 2 = 34 MiB, 36 MiB of tiles
    B = torch.zeros((8192, N), dtype=torch.float16, device=dev)
    out = torch.zeros((2048, N), dtype=torch.float32, device=dev)
    L = smat_mod.lib()
    st = L.smat_spmm_static_scratch(M.handle, smat_mod.FORM_F16, C.c_void_p(B.data_ptr()), smat_mod.F16,
                                    smat_mod.ROW_MAJOR, N, C.c_void_p(out.data_ptr()), smat_mod.F32, N, N,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st != 0
    # what it needs is the packed B (and the counter), not the partial sums that may be left out
    assert f"needs {36 * (1 << 20) + 256} bytes" in L.smat_last_error().decode()
