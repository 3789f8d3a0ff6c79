"""GPU: infinite and NaN values of B. A block's stored zeros count, so such a value
in B's rows 16 k .. 16 k + 15 makes C infinite or NaN in every row of every block row
with a block there, and nowhere else; gathering leaves all-zero columns out, and
the kernels look them up for such a B. Through every launch that does: each
form, both block heights, passes of 256 columns, permuted columns, packed B used
twice, the static scratch, groups, whole and split panels. And that it costs no
more than the call itself: many long block rows under a short wait limit, and a
call with one such value against one without.

Tolerance for the finite part (relative Frobenius): 1e-2, as the other tests with
such values."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch.device("cuda", 0)


def graph(smat, rows, cols, seed, hubs=3):
    rng = np.random.default_rng(seed)
    d = np.full((rows, cols), 0.004)
    d[rng.integers(0, rows, hubs)] = 0.4
    m = rng.random((rows, cols)) < d
    rp = np.concatenate([[0], np.cumsum(m.sum(1))])
    return smat.Csr(rows, cols, rp, np.nonzero(m)[1].astype(np.int32), rng.uniform(0.5, 1, rp[-1]).astype(np.float32))


def dense(A):
    D = np.zeros((A.rows, A.cols))
    D[np.repeat(np.arange(A.rows), np.diff(A.row_ptr)), A.col_idx] = A.values
    return D


def b_matrix(rng, K, N, many):
    B = rng.uniform(-1, 1, (K, N)).astype(np.float32)
    for q in range(many):
        B[rng.integers(0, K), rng.integers(0, N)] = [np.inf, -np.inf, np.nan][q % 3]
    return B


def expect(A, B, bh):
    """(C of B with zeros for such values, where C is not finite)."""
    D = dense(A)
    pad = lambda x, m: np.pad(x, ((0, -x.shape[0] % m), (0, 0)))
    has = pad(pad(D != 0, bh).T, 16).T.reshape(-(-A.rows // bh), bh, -(-A.cols // 16), 16).any((1, 3))
    odd = pad(~np.isfinite(B), 16).reshape(has.shape[1], 16, -1).any(1)
    bad = np.repeat(has.astype(np.int32) @ odd.astype(np.int32) > 0, bh, 0)[: A.rows]
    return D @ np.where(np.isfinite(B), B, 0).astype(np.float64), bad


def check(got, A, B, bh):
    ref, bad = expect(A, B, bh)
    assert bad.any() and not bad.all()
    assert np.array_equal(~np.isfinite(got), bad)
    assert np.linalg.norm(got[~bad] - ref[~bad]) <= 1e-2 * np.linalg.norm(ref[~bad])


@pytest.mark.parametrize("form", ["F16", "BF16", "SPLIT_BF16", "FP8"])
@pytest.mark.parametrize("bh,R,ntc,N,frac", [(16, 8, 0, 150, 0.0), (16, 16, 0, 70, 0.05), (32, 4, 0, 129, -1.0),
                                             (32, 8, 0, 97, 0.05), (16, 8, 256, 300, 0.05), (16, 4, 256, 257, -1.0)])
@pytest.mark.parametrize("out", ["float32", "float16"])
def test_forms_and_shapes(dev, smat_mod, form, bh, R, ntc, N, frac, out):
    if form == "FP8" and bh == 32:
        pytest.skip("FP8 takes blocks of 16 rows")
    A = graph(smat_mod, 900, 2300, 4)
    M = smat_mod.Bcsr(A, forms=(getattr(smat_mod, "FORM_" + form),), block=(bh, 16), panel_rows=R, n_tile_cols=ntc,
                      split_frac=frac)
    for many in (1, 9):
        Bh = b_matrix(np.random.default_rng(many), A.cols, N, many)
        got = M.spmm(torch.from_numpy(Bh).to(dev), form=getattr(smat_mod, "FORM_" + form),
                     out_dtype=getattr(torch, out)).float().cpu().numpy()
        M.check_device_error()
        # 8-bit values are further off, so only where they are finite
        if form == "FP8":
            assert np.array_equal(~np.isfinite(got), expect(A, Bh, bh)[1])
        else:
            check(got, A, Bh, bh)


@pytest.mark.parametrize("route", ["columns", "packed", "static"])
def test_routes(dev, smat_mod, route):
    A = graph(smat_mod, 700, 1900, 8)
    N = 130
    Bh = b_matrix(np.random.default_rng(3), A.cols, N, 5)
    B = torch.from_numpy(Bh).to(dev)
    F, s = smat_mod.FORM_F16, torch.cuda.current_stream().cuda_stream
    perm = np.random.default_rng(1).permutation(A.cols) if route == "columns" else None
    M = smat_mod.Bcsr(A, col_perm=perm)
    C = torch.empty((A.rows, N), dtype=torch.float32, device=dev)
    if route == "columns":
        got = M.spmm(B).cpu().numpy()
        D = dense(A)[:, perm]
        m = D != 0
        A2 = smat_mod.Csr(A.rows, A.cols, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32),
                          D[m].astype(np.float32))
        check(got, A2, Bh[perm], 16)
        return
    if route == "static":
        smat_mod._lib.check(smat_mod.lib().smat_spmm_static_scratch(
            M.handle, F, B.data_ptr(), smat_mod.F32, smat_mod.ROW_MAJOR, N, C.data_ptr(), smat_mod.F32, N, N, s))
        check(C.cpu().numpy(), A, Bh, 16)
        return
    n = M.workspace_size(F, smat_mod.F32, N)
    ws = torch.empty(n, dtype=torch.uint8, device=dev)
    M.pack_b(F, B, smat_mod.F32, smat_mod.ROW_MAJOR, N, N, ws, n, s)
    for _ in range(2):
        C.fill_(1.0)
        M.spmm_packed(F, ws, N, C, smat_mod.F32, N, s)
        check(C.cpu().numpy(), A, Bh, 16)


def test_groups(dev, smat_mod):
    """One variant, several problems; such values in some Bs only, in different column tiles."""
    probs, data = [], []
    for i in range(6):
        A = graph(smat_mod, 400 + 90 * i, 1100 + 230 * i, 20 + i)
        Bh = b_matrix(np.random.default_rng(i), A.cols, 200, 3 * (i % 2))
        M = smat_mod.Bcsr(A, split_frac=0.05)
        B = torch.from_numpy(Bh).to(dev)
        C = torch.empty((A.rows, 200), dtype=torch.float32, device=dev)
        probs.append((M, smat_mod.FORM_F16, B, C))
        data.append((A, Bh))
    g = smat_mod.Group(probs)
    g.run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    g.check_device_error()
    for (A, Bh), (*_, C) in zip(data, probs):
        got = C.cpu().numpy()
        if np.isfinite(Bh).all():
            assert np.isfinite(got).all()
        else:
            check(got, A, Bh, 16)


def long_rows(smat, panels, blocks, cols):
    """Panels of eight block rows, each with one entry in each of `blocks` blocks of its first row."""
    rng = np.random.default_rng(5)
    nbr = panels * 8
    ci = np.empty((nbr, blocks), np.int32)
    for r in range(nbr):
        ci[r] = np.sort(rng.choice(cols // 16, blocks, replace=False)) * 16 + rng.integers(0, 16, blocks)
    rp = np.zeros(nbr * 16 + 1, np.int64)
    rp[1:] = np.repeat(np.arange(1, nbr + 1) * blocks, 16)
    return smat.Csr(nbr * 16, cols, rp, ci.reshape(-1), rng.uniform(0.5, 1, ci.size).astype(np.float32)), ci


@pytest.mark.parametrize("frac", [-1.0, 0.0])
def test_long_rows_under_a_short_wait_limit(dev, smat_mod, frac):
    """Four units a CTA, with 500 left-out entries to look up in each block row: the
    MMAs wait for the accumulators no longer than without such a value, within 1 ms,
    and the call takes at most four times as long."""
    A, ci = long_rows(smat_mod, 4 * 152, 500, 16000)
    M = smat_mod.Bcsr(A, panel_rows=8, split_frac=frac)
    M.set_wait_limit(1_000_000)
    N = 128
    Bh = np.random.default_rng(0).uniform(-1, 1, (A.cols, N)).astype(np.float16)
    rows = np.random.default_rng(1).choice(A.cols, 5, replace=False)

    def timed(B):
        t = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            C = M.spmm(B)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        M.check_device_error()
        return C.cpu().numpy(), sorted(t)[2]

    clean, t0 = timed(torch.from_numpy(Bh).to(dev))
    Bh[rows, [1, 40, 41, 90, 127]] = np.inf
    got, t1 = timed(torch.from_numpy(Bh).to(dev))
    print(f"split_frac {frac}: {t0 * 1e3:.0f} us, with infinities {t1 * 1e3:.0f} us")
    bad = np.zeros(got.shape, bool)
    for k, n in zip(rows, [1, 40, 41, 90, 127]):
        bad[np.repeat((ci // 16 == k // 16).any(1), 16), n] = True
    assert bad.any()
    assert np.array_equal(~np.isfinite(got), bad)
    assert np.array_equal(got[~bad], clean[~bad])
    assert t1 <= 4 * t0, (t0, t1)


def test_more_units_than_a_cta_notes(dev, smat_mod):
    """One panel and so many column tiles that every CTA of 152 has more than 512
    units; such values in the first and in the last tiles."""
    N = 128 * 152 * 516
    rng = np.random.default_rng(3)
    D = np.zeros((16, 32), np.float32)
    D[0, [1, 7]] = D[3, 20] = D[15, 1] = 1.5         # sparse blocks: gathered
    m = D != 0
    A = smat_mod.Csr(16, 32, np.concatenate([[0], np.cumsum(m.sum(1))]), np.nonzero(m)[1].astype(np.int32), D[m])
    M = smat_mod.Bcsr(A, panel_rows=4)
    B = torch.ones((32, N), dtype=torch.float16, device=dev)
    at = np.concatenate([rng.integers(0, 128 * 152, 40), rng.integers(N - 128 * 152 * 3, N, 200)])
    B[torch.from_numpy(rng.integers(0, 32, at.size)).to(dev), torch.from_numpy(at).to(dev)] = float("inf")
    out = torch.empty((16, N), dtype=torch.float16, device=dev)
    M.spmm(B, out=out)
    M.check_device_error()
    bad = ~torch.isfinite(B).reshape(2, 16, N).all(1)
    assert torch.equal(~torch.isfinite(out), bad.any(0)[None].expand(16, N))
    good = torch.isfinite(B).all(0)
    ref = torch.from_numpy(D.sum(1)).to(dev).half()[:, None]
    assert torch.equal(torch.where(good[None], out, ref), ref.expand(16, N))
