"""Study I updates with filters wider than the grid, on both sides of the shared memory limit of the one-launch update
(54 with radius 108 takes 98.7 KB of 100; 56 with radius 112 goes through the separate passes), against the oracle with the
same filter as circulant matrices.

A filtered value sums 2 radius + 1 positive terms three times: relative error below 3 x 225 x 2^-53 = 8e-14; the design
passes through a square root and a clip, 1e-12 absolute on values below 1 (as in test_outer_updates.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


@pytest.mark.parametrize("n,radius", [(10, 20), (54, 108), (56, 112)])
def test_study1_update_with_a_wide_filter(pkg, oracle, n, radius, monkeypatch):
    k = np.arange(-radius, radius + 1)
    w = 1.0 / (1.0 + (k / 3.0) ** 2)
    w /= w.sum()
    matrix = np.zeros((n, n))
    for i in range(n):
        np.add.at(matrix[i], (i + k) % n, w)
    monkeypatch.setattr(oracle, "study1_filter", lambda x: np.einsum("ai,bj,ck,ijk->abc", matrix, matrix, matrix, x,
                                                                     optimize=True))
    rng = np.random.default_rng(n)
    x, e, beta = rng.uniform(0.05, 0.95, (n, n, n)), rng.uniform(0.1, 2.0, (n, n, n)), 4.0
    ro = pkg.ResidentOuter(n)
    ro.weights, ro.radius = torch.tensor(w, device="cuda"), radius
    ro.set_initial(x)
    ro.evaluate(beta)
    ph, dp = oracle.study1_physical(x, beta)
    assert np.abs(ro.ph.cpu().numpy() - ph).max() < 1e-12
    ro.step(torch.tensor(e, device="cuda"))
    gradient = oracle.study1_filter(dp * 3 * (1 - 1e-4) * ph ** 2 * e)
    new = oracle.study1_oc(x, gradient, oracle.study1_filter(dp), beta)
    assert np.abs(ro.new.cpu().numpy() - new).max() < 1e-12
    assert abs(float(ro.change) - np.abs(new - x).max()) < 1e-12
