"""The operator (two elements of a row per thread) at the sizes where its tiles can go wrong: a thread row of 2
to 128 pairs, tiles that overhang the grid, chunks that end short, a single tile row, several blocks per SM,
vectors that are not aligned to a pair of values, and inactive loads, against K(a) u summed in FP64.

Tolerance: a node sums 8 elements x 24 terms, and the modal form adds a few additions; 64 roundings of the
largest term bound the error, 64 x 1.1e-16 and 64 x 6e-8 relative to the largest |q|.
"""
import itertools

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)


def dense(oracle, a, u, n, lam, mu):
    """sum over elements of a_e Ke u_e, one corner pair at a time."""
    ke = torch.tensor(oracle.element_stiffness(n, lam, mu), device="cuda").reshape(8, 3, 8, 3)
    v, a = u.reshape(n, n, n, 3), a.reshape(n, n, n, 1)
    out = torch.zeros_like(v)
    corner = [(b >> 2 & 1, b >> 1 & 1, b & 1) for b in range(8)]
    for i in range(8):
        f = sum(torch.roll(v, [-k for k in corner[j]], (0, 1, 2)) @ ke[i, :, j, :].T for j in range(8))
        out += torch.roll(a * f, corner[i], (0, 1, 2))
    return out.reshape(-1)


@pytest.mark.parametrize("n,loads", [(4, 1), (6, 6), (10, 3), (16, 6), (30, 2), (50, 6), (64, 6), (90, 1), (128, 2),
                                     (250, 1), (256, 1)])
def test_row_operator(pkg, oracle, n, loads):
    lam, mu = pkg.PAPER_MEDIUM
    gen = torch.Generator(device="cuda").manual_seed(n)
    a = 10.0 ** (-4 * torch.rand(n ** 3, generator=gen, device="cuda", dtype=torch.float64))
    u = torch.rand((loads, 3 * n ** 3), generator=gen, device="cuda", dtype=torch.float64) - 0.5
    op = pkg.Operator(n, loads, lam, mu, precision="mixed")
    op.set_material(a)
    lib, stream = pkg._lib.lib(), torch.cuda.current_stream().cuda_stream
    mask = torch.ones(loads, dtype=torch.int32, device="cuda")
    mask[loads // 2] = 0 if loads > 1 else 1
    for (dtype, fn, eps), shift in itertools.product(
            ((torch.float64, lib.pgj_apply, 1.1e-16), (torch.float32, lib.pgj_apply_f32, 6e-8)), (0, 1)):
        p = torch.empty(u.numel() + 2, dtype=dtype, device="cuda")[shift:shift + u.numel()].view_as(u)
        q = torch.full((u.numel() + 2,), 7.0, dtype=dtype, device="cuda")
        p.copy_(u)
        w = q[shift:shift + u.numel()].view_as(u)
        assert fn(op._ctx, loads, p.data_ptr(), mask.data_ptr(), w.data_ptr(), stream) == 0
        for load in range(loads):
            want = dense(oracle, a, p[load].double(), n, lam, mu) * float(mask[load])
            assert float((w[load].double() - want).abs().max()) <= 64 * eps * float(want.abs().max())
        rest = torch.cat([q[:shift], q[shift + u.numel():]])
        assert torch.equal(rest, torch.full_like(rest, 7.0))
