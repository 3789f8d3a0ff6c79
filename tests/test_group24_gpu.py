"""GPU: groups whose handles keep exact-2:4 blocks for the structured-sparse
path (use_24): every problem against FP64, in a group with plain handles, with
blocks of both kinds and all on that path, groups of block rows cut into parts
(6,000 columns), FP16 and BF16 forms, FP32 and FP16 C wider than N; repeated,
and replayed from a CUDA graph.

Tolerances (relative Frobenius, as the other GPU tests): FP16 1e-3, BF16 1e-2,
one more rounding for FP16 C (2e-3)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def csr(smat, D):
    m = D != 0
    return smat.Csr(*D.shape, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32), D[m])


def matrix(rng, rows, cols, all24):
    D = np.zeros((rows, cols), np.float32)
    for q in range(0, cols, 4):                  # two of four in every group of columns
        pick = rng.integers(0, 2, rows)
        D[np.arange(rows), q + pick] = rng.standard_normal(rows)
        D[np.arange(rows), q + 2 + pick] = rng.standard_normal(rows)
    D[rng.random(D.shape) < 0.3] = 0
    D[32:48] = 0                                 # a block row without a block
    if not all24:
        D[: rows // 2, : cols // 2] = rng.standard_normal((rows // 2, cols // 2))
    return D.astype(np.float16).astype(np.float32)


@pytest.mark.parametrize("N", [1, 100, 200])
def test_groups_of_24_handles(smat_mod, N):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(N)
    probs, refs = [], []
    for i, (rows, cols, all24, use24) in enumerate([(500, 640, False, 1), (200, 6000, True, 1), (700, 320, False, 0),
                                                    (300, 330, True, 4), (130, 512, False, 4), (96, 64, True, 1)]):
        D = matrix(rng, rows, cols - cols % 4, all24)
        form, dt = [(smat_mod.FORM_F16, torch.float16), (smat_mod.FORM_BF16, torch.bfloat16)][i % 2]
        M = smat_mod.Bcsr(csr(smat_mod, D), forms=(form,), use_24=use24)
        assert (M.info["n_blocks_24"] > 0) == (use24 > 0)
        B = torch.from_numpy(rng.uniform(-1, 1, (D.shape[1], N)).astype(np.float32)).cuda().to(dt)
        C = torch.full((rows, N + 5), float("nan"), dtype=[torch.float32, torch.float16][i // 2 % 2], device="cuda")
        probs.append((M, form, B, C[:, :N]))
        refs.append(D.astype(np.float64) @ B.float().cpu().numpy().astype(np.float64))
    g = smat_mod.Group(probs)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g.run(s.cuda_stream)
    s.synchronize()
    g.check_device_error()
    first = [C.clone() for *_, C in probs]
    for (M, form, B, C), ref in zip(probs, refs):
        err = float(np.linalg.norm(C.float().cpu().numpy().astype(np.float64) - ref) / np.linalg.norm(ref))
        tol = 1e-2 if form == smat_mod.FORM_BF16 else (2e-3 if C.dtype == torch.float16 else 1e-3)
        assert err <= tol, (M.info["rows"], M.info["cols"], err)
        assert torch.isnan(C._base[:, N:]).all()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        g.run(s.cuda_stream)
    for *_, C in probs:
        C.fill_(float("nan"))
    torch.cuda.synchronize()
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    g.check_device_error()
    for a, (*_, C) in zip(first, probs):
        assert torch.equal(a, C)
    g.close()
