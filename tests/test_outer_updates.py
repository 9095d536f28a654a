"""The one-launch OC updates and the tiled cone filter at the sizes where their splits can go wrong:
grids that end inside a 32 x 8 x 4 tile or an 8-row chunk, tap tables inside and beyond the tile form's
radius and capacity, against the oracle's restatement.

Bounds: filtered fields are sums of positive terms (relative error about taps * 2^-53, 1e-13 is ample);
the designs pass through a power or a square root and a clip, 1e-12 absolute on values below 1.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


def fields(n, seed):
    rng = np.random.default_rng([n, seed])
    return rng.uniform(0.05, 0.95, (n, n, n)), rng.uniform(0.1, 2.0, (n, n, n))


@pytest.mark.parametrize("n,rmin", [(2, 1.5), (5, 3.9), (9, 2.0), (31, 3.0), (33, 3.5), (40, 1.2), (12, 5.3), (10, 7.0)])
def test_paper_update(pkg, oracle, n, rmin):
    x, e = fields(n, 1)
    po = pkg.PaperOuter(n, 0.3, rmin=rmin, emin=1e-6)
    po.set_initial(x)
    po.evaluate()
    hs = oracle.cone_filter(np.ones_like(x), rmin)
    t = oracle.cone_filter(x, rmin)
    assert np.abs(po.t.cpu().numpy() / t - 1).max() < 1e-13
    ph, dp, _ = oracle.paper_physical(t, hs, emin=1e-6)
    po.step(torch.tensor(-e, device="cuda"))
    new, steps, change = oracle.paper_oc(x, -e, ph, dp, hs, rmin, 0.3, emin=1e-6)
    assert po.steps == steps
    assert np.abs(po.new.cpu().numpy() - new).max() < 1e-12
    assert abs(float(po.change) - change) < 1e-12


@pytest.mark.parametrize("n,beta", [(2, 1.0), (5, 8.0), (11, 4.0), (32, 2.0), (33, 4.0), (45, 4.0)])
def test_study1_update(pkg, oracle, n, beta):
    x, e = fields(n, 2)
    ro = pkg.ResidentOuter(n)
    ro.set_initial(x)
    ro.evaluate(beta)
    ph, dp = oracle.study1_physical(x, beta)
    assert np.abs(ro.ph.cpu().numpy() - ph).max() < 1e-13
    ro.step(torch.tensor(e, device="cuda"))
    gradient = oracle.study1_filter(dp * 3 * (1 - 1e-4) * ph ** 2 * e)
    new = oracle.study1_oc(x, gradient, oracle.study1_filter(dp), beta)
    assert np.abs(ro.new.cpu().numpy() - new).max() < 1e-12
    assert abs(float(ro.change) - np.abs(new - x).max()) < 1e-12
