"""pgj_precondition on vectors with a large mean, which the projection P takes out: the plane kernels against the
step-by-step passes.

Both forms subtract the same mean (summed in the same order) before the transforms, so the bound of the two forms on
vectors without a mean holds for any mean: 64 x 1.1e-16 in the norm (a value is rounded less than 64 times on its way
through six line transforms and the symbol). Left to the transforms, a mean of 2^20 would leave 1e-10."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


@pytest.mark.parametrize("alpha", [0.0, 0.7])
@pytest.mark.parametrize("n,loads", [(4, 6), (16, 2), (50, 1), (64, 6), (80, 2)])
def test_precondition_takes_the_mean_out_exactly(pkg, n, loads, alpha):
    gen = torch.Generator(device="cuda").manual_seed(n)
    r = torch.rand((loads, n ** 3, 3), generator=gen, device="cuda", dtype=torch.float64) - 0.5
    r += 2.0 ** 20 * torch.tensor([1.0, -0.75, 0.5], device="cuda", dtype=torch.float64)
    r = r.reshape(loads, -1)
    op = pkg.Operator(n, loads, *pkg.PAPER_MEDIUM)
    op.set_material(torch.tensor(pkg.baseline_design(n, seed=n, emin=1e-6), device="cuda"))
    op.set_alpha(alpha)
    op.set_fused_iteration(False)
    want = op.apply_precond(r)
    op.set_fused_iteration(True)
    assert float((op.apply_precond(r) - want).norm()) <= 64 * 1.1e-16 * float(want.norm())
