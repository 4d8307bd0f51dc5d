"""The bounded waits of the kernels: one that runs out makes the call return
CANDMC_ERR_TIMEOUT (the limits are lowered from the host; nothing is left
waiting), and the next call with the usual limits is right again.
"""
import numpy as np
import pytest

from oracle import candmc_oracle as co
from oracle import fixtures as fx

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

POLLS = 1 << 22
TIMEOUT, NUMERIC = 4, 5


@pytest.fixture(scope="module")
def cm():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import candmc_gb300 as cm
    cm.lib()
    return cm


def status_of(cm, f):
    try:
        f()
    except cm.CandmcError as e:
        return e.status
    return 0


# one leaf (only its publishing warp and the root's solver wait), a node of three
# leaves, two levels of nodes with a pass-through one
@pytest.mark.parametrize("knob", ["panel_smem_polls", "panel_polls"])
@pytest.mark.parametrize("m,b", [(60, 20), (180, 32), (1100, 32)])
def test_panel_waits(cm, knob, m, b):
    A = fx.gaussian(m, b, m + b)
    try:
        cm.set_tuning(knob, 1)
        assert status_of(cm, lambda: cm.hh_recon_qr(np.asfortranarray(A.copy()))) == TIMEOUT
    finally:
        cm.set_tuning(knob, POLLS)
    YR = np.asfortranarray(A.copy())
    W, T = cm.hh_recon_qr(YR)
    YRo, Wo = co.hh_recon_qr(A, b)
    tol = 2e-12 * max(1.0, b / 16)
    assert np.abs(YR - YRo).max() <= tol * max(1.0, np.abs(YRo).max())
    assert np.abs(W - Wo).max() <= tol


@pytest.mark.parametrize("first", ["nan", "wait"])
def test_first_failure_is_reported(cm, first):
    """Of two batched calls that fail, one for a NaN and one for a wait, the status
    word has the first one's failure."""
    def call(what):
        A = fx.gaussian(200, 16, 3)
        if what == "nan":
            A[100, 3] = np.nan
        else:
            cm.set_tuning("panel_smem_polls", 1)
        dA = torch.from_numpy(A).cuda().t().contiguous().t()
        db = torch.ones((200, 1), dtype=torch.float64, device="cuda")
        try:
            cm.batched_ls([dA], [db])
            torch.cuda.synchronize()
        finally:
            cm.set_tuning("panel_smem_polls", POLLS)

    assert status_of(cm, cm.batched_status) == 0
    call(first)
    call("wait" if first == "nan" else "nan")
    assert status_of(cm, cm.batched_status) == (NUMERIC if first == "nan" else TIMEOUT)
    assert status_of(cm, cm.batched_status) == 0


# the contractions: float pairs (Y^T C sliced on the way, C -= Y Z) and a panel's own
# FP64 columns, in the seven- and three-slice forms.  With few polls a wait may or may
# not run out, at any place: the call reports it, or its result is the usual one.
@pytest.mark.parametrize("precision", ["ozaki", "fp32"])
@pytest.mark.parametrize("m,n,b,min_rows", [(300, 200, 32, 8192), (1500, 1300, 64, 1024)])
def test_contraction_waits(cm, precision, m, n, b, min_rows):
    A = np.asfortranarray(fx.gaussian(m, n, m))

    def run():
        d = A.copy(order="F")
        return status_of(cm, lambda: cm.QR_2D(d, b, precision=precision)), d

    try:
        cm.set_tuning("panel_oz_min_rows", min_rows)
        st, want = run()
        assert st == 0
        for polls in (0, 1, 2, 4, 16):
            cm.set_tuning("oz_polls", polls)
            st, got = run()
            assert st == TIMEOUT if polls == 0 else st in (0, TIMEOUT), polls
            assert st == TIMEOUT or np.array_equal(got, want), polls
        cm.set_tuning("oz_polls", POLLS)
        st, got = run()
        assert st == 0 and np.array_equal(got, want)
    finally:
        cm.set_tuning("oz_polls", POLLS)
        cm.set_tuning("panel_oz_min_rows", 8192)


def test_wait_limits_are_checked(cm):
    for knob, bad in (("panel_smem_polls", 0), ("panel_polls", 0), ("oz_polls", -1)):
        with pytest.raises(cm.CandmcError):
            cm.set_tuning(knob, bad)
