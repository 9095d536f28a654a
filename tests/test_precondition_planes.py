"""pgj_precondition on the plane kernels against the step-by-step passes: every kind of line length, few and many
loads, vectors that start at an odd value, and the result written over the input.

Tolerance: each form rounds a value less than 64 times on its way through six line transforms (at most 7 levels
each) and the symbol; 64 x 1.1e-16 bounds the difference in the norm."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


@pytest.mark.parametrize("n,loads", [(4, 6), (6, 1), (18, 2), (30, 6), (48, 3), (50, 1), (64, 6), (80, 2)])
def test_precondition_on_plane_kernels(pkg, n, loads):
    a = torch.tensor(pkg.baseline_design(n, seed=n, emin=1e-6), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(n)
    size = loads * 3 * n ** 3
    store = torch.rand(size + 1, generator=gen, device="cuda", dtype=torch.float64) - 0.3
    r = store[1:].view(loads, -1)
    op = pkg.Operator(n, loads, *pkg.PAPER_MEDIUM)
    op.set_material(a)
    op.set_alpha(0.7)
    op.set_fused_iteration(False)
    want = op.apply_precond(r)
    op.set_fused_iteration(True)
    z = op.apply_precond(r)
    assert float((z - want).norm()) <= 64 * 1.1e-16 * float(want.norm())
    stream = torch.cuda.current_stream().cuda_stream
    assert pkg._lib.lib().pgj_precondition(op._ctx, loads, r.data_ptr(), r.data_ptr(), stream) == 0
    assert torch.equal(r, z)
