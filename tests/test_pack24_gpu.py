"""GPU: the 2:4 path's copy of B. A 64-column half of a tile without a column below
N is not packed, so its part of the copy is zeros, not what the workspace held,
and a tile without a column below N (packed tiles come in pairs) is not copied."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [40, 64, 65, 128, 170, 300])
def test_copy_holds_b_and_zeros(smat_mod, N):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    K, rows = 80, 64
    rng = np.random.default_rng(N)
    D = np.zeros((rows, K), np.float32)
    D[:, ::4] = 1                                        # 2:4 throughout
    m = D != 0
    A = smat_mod.Csr(rows, K, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32), D[m])
    M = smat_mod.Bcsr(A, use_24=1)
    assert M.info["n_blocks_24"] == M.info["nnzb"]
    Bh = rng.uniform(-1, 1, (K, N)).astype(np.float16)
    B = torch.from_numpy(Bh).cuda()
    n = M.workspace_size(smat_mod.FORM_F16, smat_mod.F16, N)
    ws = torch.full((n,), 0xff, dtype=torch.uint8, device="cuda")
    M.pack_b(smat_mod.FORM_F16, B, smat_mod.F16, smat_mod.ROW_MAJOR, N, N, ws, n,
             torch.cuda.current_stream().cuda_stream)
    nt = (N + 127) // 128
    packed = nt if nt == 1 else (nt + 1) // 2 * 2        # tiles of packed B
    kbs, kw = 5, 3                                       # k-blocks, windows of two
    at = (kbs * packed * 4096 + 255) // 256 * 256
    copy = ws[at:at + kw * packed * 8192].cpu().numpy().view(np.uint16).reshape(packed, kw, 128, 4, 8)
    want = np.zeros((nt * 128, kw * 32), np.float16)     # [n][k]
    want[:N, :K] = Bh.T
    want = want.view(np.uint16).reshape(nt, 128, kw, 4, 8).transpose(0, 2, 1, 3, 4)
    row = np.arange(128)
    for c in range(4):                                   # 16-byte chunk c of row n lies at c ^ ((n >> 1) & 3)
        assert np.array_equal(copy[:nt, :, row, c ^ ((row >> 1) & 3)], want[:, :, :, c])
    assert (copy[nt:] == 0xffff).all()
