"""The emulated-FP64 contractions at the edges of their tiles, K groups, K
splits and scale exponents.

C - Y (Y^T C) / 2 (the operator is the inverse of W = 2 I) against numpy in
FP64.  The bound is worked out from the
format, per element.  An operand entry is its digits to half a unit of the
last one, 2^-57 of its scale, which is at most twice its row's largest entry;
the slice products left out come to less than 2^-55 of both scales: together
less than 2^-52 max|x| max|y| per product.  Float pairs, the exact combine of
the accumulators and the pair additions round at 2^-46, which over a sum is
taken as 2^-44 of sum |x||y|.  A float pair resolves 2^-149.  The reference's
own k-term sums are within k 2^-53 sum |x||y|.
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
    return torch.from_numpy(np.asfortranarray(a)).cuda().t().contiguous().t()


def product_bound(X, Y, dX, dY):
    """|error| of the emulated X Y for operands with errors dX, dY."""
    k = X.shape[1]
    a = np.abs(X) @ np.abs(Y)
    scales = np.abs(X).max(axis=1, keepdims=True) * np.abs(Y).max(axis=0, keepdims=True)
    return k * 2.0 ** -52 * scales + (2.0 ** -44 + k * 2.0 ** -53) * a + dX @ np.abs(Y) + np.abs(X) @ dY


def check_update(cm, m, nb, n, scales, store):
    g = np.random.default_rng(m + nb + n)
    Y = g.standard_normal((m, nb)) / np.sqrt(m)
    C = np.ldexp(g.standard_normal((m, n)), np.resize(scales, n)[None, :])
    if n > 2:
        C[:, 2] = 0.0
    out = store(C)
    cm.upd_A(dev(Y), out, W=dev(2.0 * np.eye(nb)), W_is_T=True, precision="ozaki")
    tiny = 2.0 ** -148
    zero = lambda a: np.zeros_like(a)
    Z = Y.T @ C
    dZ = product_bound(Y.T, C, zero(Y.T), np.full_like(C, tiny)) + tiny
    T = 0.5 * np.eye(nb)
    Z2 = T @ Z
    dZ2 = product_bound(T, Z, zero(T), dZ) + tiny
    want = C - Y @ Z2
    bound = product_bound(Y, Z2, zero(Y), dZ2) + 2.0 ** -46 * (np.abs(C) + np.abs(Y @ Z2)) + 4 * tiny
    got = out.cpu().numpy()
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


# rows: one group of 128, one more or less, 16-row blocks, many K splits (157
# groups); columns: 96-column tiles, below and from 1024 columns (the operator
# product on the tensor cores); panel widths: 8-row core matrices, 16-deep K steps
@pytest.mark.parametrize("m,nb,n", [(1, 1, 1), (128, 16, 96), (129, 17, 97), (127, 8, 95), (255, 128, 193),
                                    (656, 9, 1100), (1000, 100, 1024), (20000, 128, 30), (20090, 33, 289)])
@pytest.mark.parametrize("scales", [(0,), (0, -60, 60, -112)])
def test_update_edges(cm, m, nb, n, scales):
    check_update(cm, m, nb, n, scales, dev)


# C as rows of a larger matrix: columns aligned to 16 bytes with an odd number of
# rows, and columns at every 8-byte boundary; what lies around C stays
@pytest.mark.parametrize("m,nb,n", [(129, 17, 97), (1003, 64, 200), (20001, 32, 40)])
@pytest.mark.parametrize("off,extra", [(0, 1), (2, 5), (1, 3), (1, 2)])
def test_update_within_matrix(cm, m, nb, n, off, extra):
    buf = torch.full((n, m + extra), 3.0, dtype=torch.float64, device="cuda")

    def store(C):
        A = buf.t()[off:off + m]
        A.copy_(torch.from_numpy(C).cuda())
        return A

    check_update(cm, m, nb, n, (0,), store)
    assert (buf[:, :off] == 3.0).all() and (buf[:, off + m:] == 3.0).all()


def product_bound_f32(X, Y, dX, dY):
    """The same for the three-slice form.  An operand entry is its digits to half a
    unit of the last one, 2^-25 of its scale, which is at most twice its row's largest
    entry: 2^-24 max|x| on each side.  The slice products left out (1, 2), (2, 1) and
    (2, 2) come to at most 2^-25 of both scales, four times the largest entries:
    2^-23.  Together 2^-22 max|x| max|y| per product; twice that is taken for the parts
    that cancel between the levels.  The levels' exact sums over 128 rows are added in
    FP32, as are the groups: 2^-24 sum |x||y| a piece, two per group and four more."""
    k = X.shape[1]
    a = np.abs(X) @ np.abs(Y)
    scales = np.abs(X).max(axis=1, keepdims=True) * np.abs(Y).max(axis=0, keepdims=True)
    return k * 2.0 ** -21 * scales + (2 * (k // 128 + 1) + 4) * 2.0 ** -24 * a + dX @ np.abs(Y) + np.abs(X) @ dY


# the three-slice kernels at the same edges; the operator product runs on them too from
# 1024 columns on.  C takes part as the FP32 sum of its pair and is rounded once more.
@pytest.mark.parametrize("m,nb,n,off,extra", [(1, 1, 1, 0, 0), (128, 16, 96, 0, 0), (129, 17, 97, 0, 0),
                                              (127, 8, 95, 0, 0), (255, 128, 193, 0, 0), (656, 9, 1100, 0, 0),
                                              (1000, 100, 1024, 0, 0), (20090, 33, 289, 0, 0), (129, 17, 97, 0, 1),
                                              (1003, 64, 200, 2, 5), (1003, 64, 200, 1, 3), (20001, 32, 40, 1, 2)])
@pytest.mark.parametrize("scales", [(0,), (0, -60, 30, -80)])
def test_update_edges_fp32(cm, m, nb, n, off, extra, scales):
    g = np.random.default_rng(m + nb + n)
    Y = g.standard_normal((m, nb)) / np.sqrt(m)
    C = np.ldexp(g.standard_normal((m, n)), np.resize(scales, n)[None, :])
    if n > 2:
        C[:, 2] = 0.0
    buf = torch.full((n, m + extra), 3.0, dtype=torch.float64, device="cuda")
    out = buf.t()[off:off + m]
    out.copy_(torch.from_numpy(C).cuda())
    cm.upd_A(dev(Y), out, W=dev(2.0 * np.eye(nb)), W_is_T=True, precision="fp32")
    tiny = 2.0 ** -148 * (m // 128 + 2)
    zero = lambda a: np.zeros_like(a)
    Z = Y.T @ C
    dZ = product_bound_f32(Y.T, C, zero(Y.T), np.full_like(C, tiny)) + tiny
    T = 0.5 * np.eye(nb)
    Z2 = T @ Z
    dZ2 = product_bound_f32(T, Z, zero(T), dZ) + tiny
    want = C - Y @ Z2
    bound = product_bound_f32(Y, Z2, zero(Y), dZ2) + 2.0 ** -23 * (np.abs(C) + np.abs(Y @ Z2)) + 4 * tiny
    got = out.cpu().numpy()
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()
    assert (buf[:, :off] == 3.0).all() and (buf[:, off + m:] == 3.0).all()
