"""The leaf heights that panels take by themselves: on both sides of each line of the
rule, equal bits with the height set by hand, and the oracle's result (tolerance of
the parity tests, 2e-12 max(1, b / 16) relative to the largest entry)."""
import numpy as np
import pytest

from oracle import candmc_oracle as co
from oracle import fixtures as fx

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def cm():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import candmc_gb300 as cm
    cm.set_tuning("leaf_rows", 0)
    cm.set_tuning("pipe_leaf_rows", 0)
    yield cm
    cm.set_tuning("leaf_rows", 0)
    cm.set_tuning("pipe_leaf_rows", 0)


def short_limit():
    """The tallest panel with 64-row leaves: p of them, p parts of Y and the tree's
    nodes (p / 3 + 4 covers them) have a multiprocessor each."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p = max(p for p in range(1, sms) if 2 * p + p // 3 + 4 <= sms)
    return 64 * p


@pytest.mark.parametrize("entry", ["panel", "pipe"])
@pytest.mark.parametrize("at", ["short", "above short", "below tall", "tall"])
def test_default_heights(cm, entry, at):
    m, leaf = {"short": (short_limit(), 64), "above short": (short_limit() + 1, 128), "below tall": (32767, 128),
               "tall": (32768, 256)}[at]
    n, knob = (32, "leaf_rows") if entry == "panel" else (64, "pipe_leaf_rows")
    A = fx.gaussian(m, n, m)
    YRo, _ = co.hh_recon_qr(A, n)

    def run():
        d = torch.from_numpy(A).cuda().t().contiguous().t()
        if entry == "panel":
            cm.hh_recon_qr(d)
        else:
            cm.QR_2D_pipe(d, n)
        torch.cuda.synchronize()
        return d.cpu().numpy()

    auto = run()
    assert np.abs(auto - YRo).max() <= 2e-12 * max(1.0, n / 16) * max(1.0, np.abs(YRo).max())
    if entry == "panel":
        cm.set_tuning(knob, leaf)
        assert np.array_equal(run(), auto)
        cm.set_tuning(knob, 0)
        assert np.array_equal(run(), auto)


def test_default_heights_above_the_pipelined_tree(cm):
    """More than 4096 thread blocks of 256-row leaves: the level-by-level tree."""
    m, b = 800001, 4
    A = fx.gaussian(m, b, 5)
    YRo, Wo = co.hh_recon_qr(A, b)
    d = torch.from_numpy(A).cuda().t().contiguous().t()
    W, T = cm.hh_recon_qr(d)
    torch.cuda.synchronize()
    assert np.abs(d.cpu().numpy() - YRo).max() <= 2e-12 * max(1.0, np.abs(YRo).max())
    assert np.abs(W.cpu().numpy() - Wo).max() <= 2e-12
