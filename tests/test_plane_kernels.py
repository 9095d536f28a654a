"""The four-kernel PCG iteration (plane transform kernels) against the step-by-step kernels, on every
line length it is built for: grids that fill neither a block's threads nor the last chunk of z columns,
one and two blocks per SM, and grids beyond those the step-by-step form may be exchanged with.

Both forms solve to a relative residual of 1e-11; as for the resident kernels, 1e3 times that bounds the
difference of the displacements at a weak-material ratio of 1e-4.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [4, 6, 8, 18, 30, 40, 48, 50, 54, 60, 64, 72, 80, 90, 100, 108, 120])
def test_plane_kernels_match_step_by_step(pkg, n, precision, monkeypatch):
    if precision == "fp64" and n > 108:
        pytest.skip("beyond the built FP64 grids")
    monkeypatch.setenv("PGJ_RESIDENT", "0")
    loads = 1 if n >= 72 else (2, 6)[n % 4 == 0]
    a = torch.tensor(pkg.baseline_design(n, seed=n, emin=1e-4), device="cuda")
    macros = np.eye(6)[:loads]
    out = []
    for four in (False, True):
        op = pkg.Operator(n, loads, *pkg.PAPER_MEDIUM, precision=precision)
        if not four:
            op.set_fused_iteration(False)
        op.set_material(a)
        op.set_alpha(0.5)
        u = torch.zeros((loads, 3 * n ** 3), dtype=torch.float64, device="cuda")
        infos, st = op.solve(macros, 1e-11, u)
        assert st == 0, infos
        out.append((u, op.energies(u, macros)))
        if four:
            again = torch.zeros_like(u)
            op.solve(macros, 1e-11, again)
            assert torch.equal(again, u)
    (u0, e0), (u1, e1) = out
    assert float((u1 - u0).norm() / u0.norm()) < 1e-8
    assert float((e1 - e0).norm() / e0.norm()) < 1e-8


def test_flexible_update_and_sweeps_on_plane_kernels(pkg):
    """The options that keep the separate kernels on small grids: flexible direction, FP64 arithmetic on
    FP32 vectors, refinement sweeps. Tensors agree with FP64 to the mixed tolerance of these tests, 1e-7."""
    n = 20
    a = torch.tensor(pkg.baseline_design(n, seed=4, emin=1e-6), device="cuda")

    def tensor(precision, configure):
        op = pkg.Operator(n, 6, *pkg.PAPER_MEDIUM, precision=precision)
        configure(op)
        op.set_material(a)
        op.set_alpha(0.6)
        u = torch.zeros((6, 3 * n ** 3), dtype=torch.float64, device="cuda")
        _, st = op.solve(np.eye(6), 1e-8, u)
        assert st == 0
        return op.effective_tensor(u)

    ref = tensor("fp64", lambda op: None)
    for configure in (lambda op: op.set_flexible_beta(True), lambda op: op.set_mixed_operator(True),
                      lambda op: op.set_mixed_mode("sweeps")):
        assert float((tensor("mixed", configure) - ref).norm() / ref.norm()) < 1e-7
