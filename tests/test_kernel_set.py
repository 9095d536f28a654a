"""The kernel set of the PCG iteration: what is reported can be written back, on grids without a choice too, and the
plane kernels of those grids against the step-by-step kernels, which only new contexts can be told to run there.

Solves to a relative residual of 1e-11; 1e3 times that bounds the difference of the displacements at a weak-material
ratio of 1e-4 (the condition of the scaled operator)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


def operator(pkg, n, precision):
    op = pkg.Operator(n, 1, *pkg.PAPER_MEDIUM, precision=precision)
    op.set_material(torch.tensor(pkg.baseline_design(n, seed=n, emin=1e-4), device="cuda"))
    op.set_alpha(0.5)
    return op


@pytest.mark.parametrize("n,precision,kernels", [(96, "fp64", 4), (108, "fp64", 4), (120, "mixed", 4), (64, "fp64", 4),
                                                 (24, "mixed", 4), (120, "fp64", 8)])
def test_reported_kernel_set_can_be_written_back(pkg, n, precision, kernels):
    op = operator(pkg, n, precision)
    for _ in range(2):
        assert len(op.profile_iteration(np.eye(6)[:1], reps=1)) == kernels
        assert op.tile_shapes()["fused"] == (kernels == 4)
        op.set_fused_iteration(op.fused_iteration)
    if op.fused_iteration:  # the choice, there and back
        op.set_fused_iteration(False)
        assert len(op.profile_iteration(np.eye(6)[:1], reps=1)) == 8 and not op.tile_shapes()["fused"]
        op.set_fused_iteration(True)
        assert len(op.profile_iteration(np.eye(6)[:1], reps=1)) == 4


@pytest.mark.parametrize("n,precision", [(90, "fp64"), (100, "fp64"), (108, "fp64"), (120, "mixed"), (128, "mixed")])
def test_plane_kernels_without_a_choice_match_step_by_step(pkg, n, precision, monkeypatch):
    out = []
    for unfused in (True, False):
        if unfused:
            monkeypatch.setenv("PGJ_UNFUSED", "1")
        else:
            monkeypatch.delenv("PGJ_UNFUSED")
        op = operator(pkg, n, precision)
        assert op.tile_shapes()["fused"] != unfused
        u = torch.zeros((1, 3 * n ** 3), dtype=torch.float64, device="cuda")
        infos, st = op.solve(np.eye(6)[:1], 1e-11, u)
        assert st == 0, infos
        out.append(u)
    assert float((out[1] - out[0]).norm() / out[0].norm()) < 1e-8
