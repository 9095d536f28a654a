"""A second attempt of a solve iterates, in each form of the FP64 iteration.

The solve starts from random displacements 1e3 times too large: when the recurrence's residual falls below the 1e-11 asked
for, it has drifted from the true one by rounding of the first residual's size, so the certificate refuses, and the second
attempt starts from the true residual and passes. (Far larger starts leave a mean in the residual, which the projection
keeps out of the corrections, above the threshold: no form of the solve certifies those.)
Both starts end with a relative residual of 1e-11, and 1e3 times that bounds the difference of the displacements at this
weak-material ratio."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


@pytest.mark.parametrize("n,fused", [(12, True), (24, True), (48, True), (64, True), (30, False), (48, False)])
def test_second_attempt_iterates(pkg, n, fused):
    op = pkg.Operator(n, 3, *pkg.PAPER_MEDIUM, precision="fp64")
    op.set_fused_iteration(fused)
    op.set_material(torch.tensor(pkg.baseline_design(n, seed=3, emin=1e-3), device="cuda"))
    op.set_alpha(0.5)
    macros = np.eye(6)[3:]
    zero = torch.zeros((3, 3 * n ** 3), dtype=torch.float64, device="cuda")
    infos, st = op.solve(macros, 1e-11, zero)
    assert st == 0
    first = max(i["iterations"] for i in infos)
    far = 1e3 * torch.randn(zero.shape, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda",
                            dtype=torch.float64) * zero.abs().max()
    infos, st = op.solve(macros, 1e-11, far)
    assert st == 0 and all(i["converged"] for i in infos), infos
    assert max(i["restarts"] for i in infos) >= 1, infos
    assert max(i["iterations"] for i in infos) > first
    assert float((far - zero).norm() / zero.norm()) < 1e-8
