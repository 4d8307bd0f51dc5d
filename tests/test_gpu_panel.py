"""The TSQR-HR kernels at the edges of their row slots, widths and ranges.

Inputs are Gaussian panels scaled by a power of two: the reflectors, T and the
signs do not depend on the scale and R carries it exactly, so one oracle run
serves every scale.  Beyond 2^+-30 the squares leave the range of the
reflector's FP32 seeds and the scaled form of the reflector runs.  Tolerance:
the element-wise bar of the parity tests, 2e-12 max(1, b / 16) relative to the
largest entry (a few ulps times the panel width).
"""
import numpy as np
import pytest

from oracle import candmc_oracle as co
from oracle import fixtures as fx
from oracle import lapack_restated as lp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cm():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import candmc_gb300 as cm
    cm.lib()
    return cm


# leaves of 1, 2, 3, 4 and more than 4 row slots; one leaf, a pass-through
# node, nodes of 2, 3 and 4 children, two and three levels; widths 1 to 32
@pytest.mark.parametrize("m,b,leaf", [(32, 32, 32), (33, 1, 32), (63, 2, 64), (96, 31, 96), (97, 32, 96),
                                      (128, 32, 128), (129, 9, 256), (256, 32, 256), (160, 32, 32), (545, 17, 32),
                                      (700, 32, 64), (2100, 32, 32), (5000, 25, 256)])
@pytest.mark.parametrize("exp", [0, 40, -700, 480])
def test_panel_steps(cm, m, b, leaf, exp):
    A = fx.gaussian(m, b, 31 * m + b)
    YRo, Wo = co.hh_recon_qr(A, b)
    To = co.T_from_W(Wo, lp.unit_lower(YRo, b)[:b])
    tol = 2e-12 * max(1.0, b / 16)
    dA = torch.from_numpy(np.ldexp(A, exp)).cuda().t().contiguous().t()
    for pipe in (1, 0):
        d = dA.t().clone().t()
        try:
            cm.set_tuning("leaf_rows", leaf)
            cm.set_tuning("pipe_tree", pipe)
            W, T = cm.hh_recon_qr(d)
            torch.cuda.synchronize()
        finally:
            cm.set_tuning("pipe_tree", 1)
            cm.set_tuning("leaf_rows", 128)
        YR = d.cpu().numpy()
        up = np.triu_indices(b)
        YR[up] = np.ldexp(YR[up], -exp)
        assert np.abs(YR - YRo).max() <= tol * max(1.0, np.abs(YRo).max())
        assert np.abs(W.cpu().numpy() - Wo).max() <= tol
        assert np.abs(T.cpu().numpy() - To).max() <= tol


def test_panel_empty_tails_and_non_finite(cm):
    """Columns with empty tails keep the sign-flip reflector (tau = 2) exactly,
    and a NaN stays a NaN instead of hanging or vanishing."""
    A = np.zeros((300, 16))
    A[:16] = np.diag(np.arange(1.0, 17.0))
    d = torch.from_numpy(A).cuda().t().contiguous().t()
    W, T = cm.hh_recon_qr(d)
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy(), -A)
    assert np.array_equal(T.diagonal().cpu().numpy(), np.full(16, 2.0))
    A = fx.gaussian(600, 24, 5)
    A[410, 7] = np.nan
    d = torch.from_numpy(A).cuda().t().contiguous().t()
    cm.hh_recon_qr(d)
    torch.cuda.synchronize()
    assert np.isnan(d.cpu().numpy()[:24, 7:]).any()


# T from two halves' factors (T12 = -T11 G T22): halves of 16 to 128 columns, even
# and odd, FP64 products and, from 16 row splits on, the emulated ones
@pytest.mark.parametrize("m,b,oz", [(300, 33, 0), (300, 47, 0), (700, 64, 0), (333, 65, 0), (600, 100, 0), (520, 128, 0),
                                    (600, 255, 0), (2500, 96, 1), (2049, 50, 1), (1900, 128, 1)])
def test_merged_factors(cm, m, b, oz):
    A = fx.gaussian(m, b, 7 * m + b)
    YRo, Wo = co.hh_recon_qr(A, b)
    To = co.T_from_W(Wo, lp.unit_lower(YRo, b)[:b])
    tol = 2e-12 * max(1.0, b / 16)
    d = torch.from_numpy(np.asfortranarray(A)).cuda().t().contiguous().t()
    if oz:   # one panel; T enters through the next half's update only
        try:
            cm.set_tuning("panel_oz_min_rows", 1024)
            cm.QR_2D(d, b, precision="ozaki")
            torch.cuda.synchronize()
        finally:
            cm.set_tuning("panel_oz_min_rows", 8192)
    else:
        W, T = cm.hh_recon_qr(d)
        torch.cuda.synchronize()
        assert np.abs(T.cpu().numpy() - To).max() <= tol
        assert np.array_equal(np.tril(T.cpu().numpy(), -1), np.zeros((b, b)))
    assert np.abs(d.cpu().numpy() - YRo).max() <= tol * max(1.0, np.abs(YRo).max())


def test_widest_panel(cm):
    """513 columns, the widest panel: halves of 256 and 257; 514 is refused."""
    m, b = 700, 513
    A = fx.gaussian(m, b, 11)
    YRo, Wo = co.hh_recon_qr(A, b)
    To = co.T_from_W(Wo, lp.unit_lower(YRo, b)[:b])
    tol = 2e-12 * max(1.0, b / 16)
    d = torch.from_numpy(A).cuda().t().contiguous().t()
    W, T = cm.hh_recon_qr(d)
    torch.cuda.synchronize()
    assert np.abs(d.cpu().numpy() - YRo).max() <= tol * max(1.0, np.abs(YRo).max())
    assert np.abs(W.cpu().numpy() - Wo).max() <= tol
    assert np.abs(T.cpu().numpy() - To).max() <= tol
    d = torch.zeros((514, m), dtype=torch.float64, device="cuda").t()
    with pytest.raises(cm.CandmcError):
        cm.hh_recon_qr(d)


@pytest.mark.parametrize("b", [1, 2, 20, 31, 32, 40, 70])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_last_column(cm, b, bad):
    """The last reflector of a square panel has an empty tail, whatever its column
    holds: a non-finite entry there stays in that column of R."""
    A = fx.gaussian(b, b, b)
    out = []
    for v in (A[b // 2, -1], bad):
        A[b // 2, -1] = v
        d = torch.from_numpy(A).cuda().t().contiguous().t()
        W, T = cm.hh_recon_qr(d)
        torch.cuda.synchronize()
        out.append((d.cpu().numpy(), W.cpu().numpy(), T.cpu().numpy()))
    (YR, W, T), (YR2, W2, T2) = out
    assert np.array_equal(YR[:, :-1], YR2[:, :-1]) and np.array_equal(W, W2) and np.array_equal(T, T2)
    assert np.isfinite(YR).all() and not np.isfinite(YR2[:, -1]).all()


# the widths at which the leaves' Gram matrices and triangular inverses change size
@pytest.mark.parametrize("b", [7, 8, 9, 15, 16, 17])
@pytest.mark.parametrize("pipe", [1, 0])
def test_narrow_widths(cm, b, pipe):
    A = fx.gaussian(1300, b, b)
    YRo, Wo = co.hh_recon_qr(A, b)
    To = co.T_from_W(Wo, lp.unit_lower(YRo, b)[:b])
    tol = 2e-12 * max(1.0, b / 16)
    d = torch.from_numpy(A).cuda().t().contiguous().t()
    try:
        cm.set_tuning("pipe_tree", pipe)
        W, T = cm.hh_recon_qr(d)
        torch.cuda.synchronize()
    finally:
        cm.set_tuning("pipe_tree", 1)
    assert np.abs(d.cpu().numpy() - YRo).max() <= tol * max(1.0, np.abs(YRo).max())
    assert np.abs(W.cpu().numpy() - Wo).max() <= tol
    assert np.abs(T.cpu().numpy() - To).max() <= tol


def test_leaves_cost_by_their_width(cm):
    """One column takes less than a fifth of the time of 32 (a tenth as measured; 0.27
    when the leaves worked all 32 columns at every width)."""
    def best(b):
        P = torch.randn(b, 400000, dtype=torch.float64, device="cuda").t()
        A = torch.empty_like(P)
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ms = []
        for _ in range(8):
            A.copy_(P)
            e[0].record()
            cm.hh_recon_qr(A)
            e[1].record()
            torch.cuda.synchronize()
            ms.append(e[0].elapsed_time(e[1]))
        return min(ms)

    assert best(1) < 0.2 * best(32)
