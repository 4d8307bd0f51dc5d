"""The triangular inverse at the edges of its 32-row blocks, and the FP64 <->
float-pair conversions over the exponent range.

Inverse: against numpy's solve in FP64 on triangles with a dominant diagonal
(off-diagonal row sums at most half the diagonal), whose condition number is
below 10: a substitution of length n carries at most about n rounding errors, so
element-wise 4 n 2^-53 relative to the largest entry bounds both sides.

Conversions: A <- A - Y Z with Y = [I; 0] and A's top rows zero leaves the rest
of A as its float pair, fl(x) + fl(x - fl(x)), which numpy forms the same way:
equal bits, not close ones.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cm():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import candmc_gb300 as cm
    cm.lib()
    return cm


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.T)).cuda().t()


def triangle(n, lower, seed):
    g = np.random.default_rng(seed)
    X = g.uniform(-1, 1, (n, n)) / (2.0 * n)
    X[np.diag_indices(n)] = g.uniform(0.5, 2.0, n) * np.where(g.random(n) < 0.5, -1.0, 1.0)
    return np.tril(X) if lower else np.triu(X)


@pytest.mark.parametrize("n", [1, 3, 31, 32, 33, 64, 100, 127, 128, 129, 255, 300])
def test_triangular_inverse(cm, n):
    tol = 4 * n * 2.0 ** -53
    # upper: invT = -W^-T Y1
    W, Y1 = triangle(n, False, n), triangle(n, True, n + 1)
    got = cm.compute_invT_from_W(dev(W), dev(Y1)).cpu().numpy()
    want = -np.linalg.solve(W.T, Y1)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
    if n > 256:
        return
    # lower and unit lower: A - Y T^T (Y^T A) with T^T = W^-1, and with T^T = -Y1^-1 W^T
    g = np.random.default_rng(n + 2)
    m = n + 40
    Y = np.tril(g.uniform(-1, 1, (m, n)) / (2.0 * n), -1) + np.eye(m, n)
    A = g.standard_normal((m, 5))
    for lower, top in ((True, lambda W: np.linalg.inv(W)), (False, lambda W: -np.linalg.solve(Y[:n], W.T))):
        W = triangle(n, lower, n + 3)
        dA = dev(A)
        cm.upd_A(dev(Y), dA, W=dev(W), W_is_T=lower)
        want = A - Y @ (top(W) @ (Y.T @ A))
        assert np.abs(dA.cpu().numpy() - want).max() <= 4 * (n + m) * 2.0 ** -53 * np.abs(want).max() * 4


@pytest.mark.parametrize("m,n,ld", [(200, 3, 200), (2500, 70, 2501), (1024 + 128, 1, 1300)])
@pytest.mark.parametrize("lo,hi", [(-10, 10), (-140, -60), (60, 120)])
def test_float_pair_round_trip(cm, m, n, ld, lo, hi):
    g = np.random.default_rng(m + n)
    b = 64
    x = np.ldexp(g.uniform(-1, 1, (m, n)), g.integers(lo, hi, (m, n)))
    x[g.random((m, n)) < 0.05] = 0.0
    x[b:b + 8] = np.ldexp(1.0, hi - 1) * np.array([1, -1, 1 + 2.0 ** -24, 1 - 2.0 ** -25, 2 - 2.0 ** -52,
                                                   1 + 2.0 ** -52, 1 + 2.0 ** -23, -(2 - 2.0 ** -25)])[:, None]
    x[:b] = 0.0
    buf = torch.zeros(n, ld, dtype=torch.float64, device="cuda")
    A = buf.t()[:m]
    A.copy_(torch.from_numpy(x).cuda())
    cm.upd_A(dev(np.eye(m, b)), A, precision="ozaki")
    with np.errstate(under="ignore"):
        h = x.astype(np.float32)
        l = (x - h.astype(np.float64)).astype(np.float32)
    want = h.astype(np.float64) + l.astype(np.float64)
    assert np.array_equal(A.cpu().numpy(), want)
    assert not buf.t()[m:].any()


# products beyond the small-product kernel (2e7 multiplications): tile and
# column-block remainders of the split-row product (8 x 4 lane blocks, 64 x 64
# tiles, one or four column groups) and of the row-per-lane product (4-column
# groups, 64-deep stages), Y dense or read under its unit-lower mask
@pytest.mark.parametrize("m,nb,n", [(20011, 50, 49), (9001, 33, 70), (70001, 100, 3), (30011, 97, 8), (33333, 64, 9),
                                    (5003, 129, 65), (2501, 256, 40), (40007, 7, 75), (1700, 64, 300)])
@pytest.mark.parametrize("masked", [False, True])
def test_fp64_products(cm, m, nb, n, masked):
    """Y^T C and C - Y Z against numpy in FP64.  A sum of k products in any
    order is within k 2^-53 sum |x||y| of the exact one, so two of them are
    within twice that; Z carries the first product's difference through T = 2 I
    and |Y|."""
    g = np.random.default_rng(m + nb + n)
    Y = g.standard_normal((m, nb)) / np.sqrt(m)
    C = g.standard_normal((m, n))
    E = np.tril(Y, -1) + np.eye(m, nb) if masked else Y
    u = 2.0 ** -53
    aZ = np.abs(E).T @ np.abs(C)
    if not masked:
        got = cm.compute_invT_from_Y2(dev(Y), dev(C)).cpu().numpy()
        assert (np.abs(got - E.T @ C) <= 2 * m * u * aZ).all()
    dC = dev(C)
    W = dev(0.5 * np.eye(nb))          # T^-T = I / 2
    if masked:
        cm.update_A(dev(Y), dC, nb, W=W, W_is_T=True)
    else:
        cm.upd_A(dev(Y), dC, W=W, W_is_T=True)
    want = C - E @ (2 * (E.T @ C))
    bound = 2 * u * (np.abs(C) + (m + nb + 2) * (np.abs(E) @ (2 * aZ)))
    assert (np.abs(dC.cpu().numpy() - want) <= bound).all()


# many column tiles, where the row split balances the rounds: one tile more than a
# round of SMs, odd chunks, chunks of the smallest length
@pytest.mark.parametrize("m,nb,n", [(1111, 65, 4900), (900, 128, 2500), (256, 70, 9800), (2050, 33, 3300)])
def test_fp64_products_wide(cm, m, nb, n):
    test_fp64_products(cm, m, nb, n, False)


def invert_upper(W):
    """Column by column back substitution: element (i, c) from rows and columns i..c."""
    n = len(W)
    X = np.zeros((n, n))
    for c in range(n):
        x = np.zeros(c + 1)
        x[c] = 1.0
        for k in range(c, -1, -1):
            x[k] /= W[k, k]
            x[:k] -= W[:k, k] * x[k]
        X[:c + 1, c] = x
    return X


# What stays finite: the rows of -W^-T Y1 whose columns of the inverse do not reach the
# odd entry.  Where all stay finite, the substitution's bound |W^-1| |W| |W^-1| n 2^-53.
@pytest.mark.parametrize("kind", ["zero pivot", "nan", "inf", "small pivot", "large pivot", "tiny pivot",
                                  "small entry", "quotient"])
@pytest.mark.parametrize("n", [2, 5, 32, 33, 64, 100, 300])
def test_triangular_inverse_extremes(cm, n, kind):
    W, Y1 = triangle(n, False, n), triangle(n, True, n + 1)
    q = n // 2
    if kind == "zero pivot":
        W[q, q] = 0.0
    elif kind == "nan":
        W[0, q] = np.nan
    elif kind == "inf":
        W[0, q] = np.inf
    elif kind == "small pivot":
        W[q, q] = 2.0 ** -600
    elif kind == "large pivot":
        W[q, q] = 2.0 ** 1000
    elif kind == "tiny pivot":   # its reciprocal overflows
        W[q, q] = 2.0 ** -1060
    elif kind == "small entry":   # W[0, q] / W[q, q] underflows
        W[0, q], W[q, q] = 2.0 ** -700, 2.0 ** 400
    else:   # W[0, q] / W[q, q] overflows
        W[0, q], W[q, q] = 2.0 ** 700, 2.0 ** -400
    got = cm.compute_invT_from_W(dev(W), dev(Y1)).cpu().numpy()
    with np.errstate(all="ignore"):
        Wi = invert_upper(W)
        up = np.triu(np.ones((n, n), dtype=bool))
        cols = np.isfinite(np.where(up, Wi, 0.0)).all(axis=0)
        assert np.isfinite(got[cols]).all() and not np.isfinite(got[~cols]).all(axis=1).any()
        if kind not in ("small pivot", "large pivot", "small entry"):
            assert not cols.all() and cols[:q].all()
        V = Wi[:, cols]
        fin = lambda a: np.abs(np.where(np.isfinite(a), a, 0.0))
        bound = 4 * n * 2.0 ** -53 * (fin(Wi) @ (fin(W) @ np.abs(V))).T @ np.abs(Y1)
        assert (np.abs(got[cols] + V.T @ Y1) <= bound).all()


# short products wider than a launch grid of 16-column tiles (65535 of them); each
# output is a sum of m products on both sides, m 2^-53 sum |x||y| apiece
@pytest.mark.parametrize("m,b1,n", [(1, 18, 1100000), (4, 4, 1048561), (4, 4, 1048560)])
def test_short_wide_products(cm, m, b1, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    Y1 = torch.randn(b1, m, dtype=torch.float64, device="cuda", generator=g).t()
    Y2 = torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g).t()
    got = cm.compute_invT_from_Y2(Y1, Y2)
    want, size = Y1.t() @ Y2, Y1.t().abs() @ Y2.abs()
    assert bool(((got - want).abs() <= 2 * m * 2.0 ** -53 * size).all())
