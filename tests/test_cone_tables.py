"""The cone filter on tap tables that PaperOuter does not build: offsets far outside the grid, anisotropic and long
tables, and weights that are not finite, against the sum over the taps whose neighbour lies inside the grid; and design
updates with wide filters, at grids of each tile depth of the general loop (bounds as in test_outer_updates.py).

Taps are summed in table order with one fused multiply-add each; the reference sums products, so a cell's difference is
below (taps + 1) x 2^-53 times the sum of |w x|. Cells that a non-finite weight reaches agree in kind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


def reference(x, offsets, weights):
    n = x.shape[0]
    y, size = np.zeros_like(x), np.zeros_like(x)
    with np.errstate(invalid="ignore"):
        for (dx, dy, dz), w in zip(offsets, weights):
            at = [slice(max(0, -d), n - max(0, d)) for d in (dz, dy, dx)]
            of = [slice(max(0, d), n + min(0, d)) for d in (dz, dy, dx)]
            if all(s.start < s.stop for s in at):
                y[tuple(at)] += w * x[tuple(of)]
                size[tuple(at)] += np.abs(w * x[tuple(of)])
    return y, size


def tables():
    rng = np.random.default_rng(3)
    yield "line", [[k, 0, 0] for k in range(-5, 6)], np.linspace(-1, 1, 11)
    yield "far", [[100, 0, 0], [0, -300, 2], [0, 0, 0], [4, 0, -4]], [1.0, 2.0, 3.0, 4.0]
    yield "long", rng.integers(-3, 4, (700, 3)), rng.standard_normal(700)
    yield "wide", rng.integers(-7, 8, (515, 3)), rng.standard_normal(515)
    yield "inf", [[0, 0, 0], [1, 0, 0], [0, 2, -1]], [1.0, np.inf, 2.0]
    yield "nan", [[0, 0, 0], [0, 0, 3]], [1.0, np.nan]


@pytest.mark.parametrize("n", [2, 5, 33, 64])
def test_general_tables(pkg, n):
    x = np.random.default_rng(n).uniform(0.1, 1.0, (n, n, n))
    xd = torch.tensor(x, device="cuda")
    y = torch.empty_like(xd)
    for name, offsets, weights in tables():
        off = torch.tensor(np.asarray(offsets), dtype=torch.int32, device="cuda")
        w = torch.tensor(np.asarray(weights, dtype=np.float64), device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        assert pkg._lib.lib().pgj_cone_filter(n, off.data_ptr(), w.data_ptr(), len(weights), xd.data_ptr(),
                                              y.data_ptr(), stream) == 0
        got = y.cpu().numpy()
        want, size = reference(x, np.asarray(offsets), np.asarray(weights))
        fin = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fin), name
        assert np.array_equal(np.isposinf(got), np.isposinf(want)), name
        assert np.all(np.abs(got - want)[fin] <= (len(weights) + 1) * 2.0 ** -53 * size[fin]), name


@pytest.mark.parametrize("n,rmin", [(9, 4.2), (40, 4.6), (50, 4.6)])
def test_paper_update_with_a_wide_filter(pkg, oracle, n, rmin):
    rng = np.random.default_rng(n)
    x, e = rng.uniform(0.05, 0.95, (n, n, n)), rng.uniform(0.1, 2.0, (n, n, n))
    po = pkg.PaperOuter(n, 0.3, rmin=rmin, emin=1e-6)
    po.set_initial(x)
    po.evaluate()
    hs, t = oracle.cone_filter(np.ones_like(x), rmin), oracle.cone_filter(x, rmin)
    assert np.abs(po.t.cpu().numpy() / t - 1).max() < 1e-13
    ph, dp, _ = oracle.paper_physical(t, hs, emin=1e-6)
    po.step(torch.tensor(-e, device="cuda"))
    new, steps, change = oracle.paper_oc(x, -e, ph, dp, hs, rmin, 0.3, emin=1e-6)
    assert po.steps == steps
    assert np.abs(po.new.cpu().numpy() - new).max() < 1e-12
    assert abs(float(po.change) - change) < 1e-12
