"""Element energies and homogenized tensor (columns of elements marched along z) where the columns and chunks end
unevenly: planes of 9 to 2500 elements (blocks hold 32 and 128), chunks of four planes and of whole columns, one to
six loads, and the odd grids that the allocation-free entry point takes, against element matrices in FP64.

Tolerance: an energy sums 24 x 24 products; 128 roundings of the largest bound it and the tensor's mean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


def element_fields(u, macro, n):
    """(N, 8, 3) corner values of u plus the affine field of an engineering Voigt strain."""
    xx, yy, zz, yz, xz, xy = macro
    strain = torch.tensor([[xx, xy / 2, xz / 2], [xy / 2, yy, yz / 2], [xz / 2, yz / 2, zz]], dtype=u.dtype, device=u.device)
    v = u.reshape(n, n, n, 3)
    out = []
    for b in range(8):
        k = torch.tensor([b & 1, b >> 1 & 1, b >> 2 & 1], dtype=u.dtype, device=u.device)
        out.append(torch.roll(v, (-(b >> 2 & 1), -(b >> 1 & 1), -(b & 1)), (0, 1, 2)) + strain @ k / n)
    return torch.stack(out, dim=3).reshape(-1, 24)


@pytest.mark.parametrize("n,loads", [(3, 6), (5, 6), (7, 6), (4, 1), (6, 6), (12, 3), (18, 6), (30, 2), (50, 6)])
def test_energies_and_tensor(pkg, oracle, n, loads):
    lam, mu = pkg.PAPER_MEDIUM
    gen = torch.Generator(device="cuda").manual_seed(n)
    u = (torch.rand((loads, 3 * n ** 3), generator=gen, device="cuda", dtype=torch.float64) - 0.5) / n
    a = 10.0 ** (-6 * torch.rand(n ** 3, generator=gen, device="cuda", dtype=torch.float64))
    ke = torch.tensor(oracle.element_stiffness(n, lam, mu), device="cuda")
    rows = np.eye(6)[:loads]
    v = torch.stack([element_fields(u[k], rows[k], n) for k in range(loads)])
    tol = 128 * 1.1e-16
    if n % 2 == 0:
        op = pkg.Operator(n, loads, lam, mu)
        op.set_material(a)
        want = torch.einsum("lei,ij,lej->le", v, ke, v) * n ** 3
        assert float((op.energies(u, rows) - want).abs().max()) <= tol * float(want.abs().max())
    if loads == 6:
        want = torch.einsum("iep,pq,jeq,e->ij", v, ke, v, a)
        tensors = []
        if n % 2 == 0:
            tensors.append(op.effective_tensor(u))
        out = torch.empty((6, 6), dtype=torch.float64, device="cuda")
        assert pkg._lib.lib().pgj_effective_tensor_noalloc(n, lam, mu, a.data_ptr(), u.data_ptr(), out.data_ptr(),
                                                           torch.cuda.current_stream().cuda_stream) == 0
        tensors.append(out)
        for got in tensors:
            assert float((got - want).abs().max()) <= tol * float(want.abs().max())
            assert torch.equal(got, got.T)
