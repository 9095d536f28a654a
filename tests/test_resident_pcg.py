"""Cluster-resident PCG (one launch per attempt, one thread-block cluster per load) against the
step-by-step kernels, on every grid it is built for: block boundaries along z, y tiles of the operator,
odd numbers of real slabs, z-pass columns that do not fill the last block, one to six loads.

Both forms solve to a relative residual of 1e-11. The displacements of two such solutions differ by the
residual times the conditioning of K restricted to the load, for which 1e3 is ample at a weak-material
ratio of 1e-4 (the same bound as between the device and a dense solve elsewhere in these tests).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)

GRIDS = (8, 10, 12, 16, 18, 20, 24, 30, 32, 36, 40, 48)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", GRIDS)
def test_resident_matches_step_by_step(pkg, n, precision):
    loads = (1, 3, 6)[GRIDS.index(n) % 3]
    a = torch.tensor(pkg.baseline_design(n, seed=n, emin=1e-4), device="cuda")
    macros = np.eye(6)[6 - loads:]
    out = {}
    for fused in (False, True):
        op = pkg.Operator(n, loads, *pkg.PAPER_MEDIUM, precision=precision)
        op.set_fused_iteration(fused)
        op.set_material(a)
        op.set_alpha(0.5)
        u = torch.zeros((loads, 3 * n ** 3), dtype=torch.float64, device="cuda")
        infos, st = op.solve(macros, 1e-11, u)
        assert st == 0, infos
        out[fused] = (u, np.array([i["iterations"] for i in infos]), op.energies(u, macros))
        again = torch.zeros_like(u)
        op.solve(macros, 1e-11, again)
        assert torch.equal(again, u)  # fixed summation order: the same bits every time
    (u0, i0, e0), (u1, i1, e1) = out[False], out[True]
    assert float((u1 - u0).norm() / u0.norm()) < 1e-8
    assert float((e1 - e0).norm() / e0.norm()) < 1e-8
    if precision == "fp64":  # (an FP32 recurrence's count also depends on where its replacements fall)
        assert np.all(np.abs(i1 - i0) <= np.maximum(2, np.ceil(0.02 * i0))), (i0, i1)


def test_resident_warm_start_and_failure(pkg):
    """A certified warm start takes no iteration; a non-finite density fails certification and leaves
    the context usable."""
    n = 20
    a = torch.tensor(pkg.baseline_design(n, seed=1, emin=1e-4), device="cuda")
    for precision in ("fp64", "mixed"):
        op = pkg.Operator(n, 6, *pkg.PAPER_MEDIUM, precision=precision)
        u = torch.zeros((6, 3 * n ** 3), dtype=torch.float64, device="cuda")
        bad = a.clone()
        bad[1, 2, 3] = float("nan")
        op.set_material(bad)
        op.set_alpha(0.5)
        _, st = op.solve(np.eye(6), 1e-8, u)
        assert st == pkg._lib.PGJ_ERR_CERTIFICATION
        op.set_material(a)
        op.set_alpha(0.5)
        _, st = op.solve(np.eye(6), 1e-8, u.zero_())
        assert st == 0
        infos, st = op.solve(np.eye(6), 1e-8, u)
        assert st == 0 and all(i["iterations"] == 0 for i in infos)
