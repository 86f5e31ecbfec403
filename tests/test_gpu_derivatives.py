"""The marching FP64 products (csrc/deriv.cu mirror_kernel, csrc/stencil_ops.cuh even8_march) against the forms that
take any stencil."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _nearly(c):
    """The stencils with 1e-13 of their largest coefficient moved (c(d) up, c(-d) down): odd to 1e-12, so the pair
    kernels take them, but not mirror symmetric to 1e-15, so the marching kernels do not."""
    c = np.array(c, dtype=np.float64).reshape(-1, 27)
    e = 1e-13 * np.abs(c).max()
    c[:, 3] += e
    c[:, 23] -= e
    return c, e


# tiles that end inside the grid, one-row and one-column remainders, planes split unevenly, the shortest axes
@pytest.mark.parametrize("dims", [(33, 50, 61), (3, 200, 140), (150, 3, 190), (200, 140, 3), (47, 46, 45),
                                  (64, 40, 33)])
def test_marching_products_match_the_pair_kernels(dims):
    """A moved coefficient changes each output by at most 2 e max|x| per stencil it enters (e = 1e-13 of the largest
    coefficient); rounding adds less than 1e-14 of the largest output."""
    from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
    from cupymag_gb300.utils.stencil_derivatives import StencilCoupling, StencilDerivatives
    from cupymag_gb300.workloads import hex_params
    cell = SimulationOperators(hex_params(6, 1, True, True), device="cuda")
    fx, fy, fz = cell.stencil_derivatives().coef
    fel = cell.stencil_coupling().coef
    n = dims[0] * dims[1] * dims[2]
    (gx, ex), (gy, ey), (gz, ez) = (_nearly(f) for f in (fx, fy, fz))
    gel, eel = _nearly(fel)
    D, D2 = StencilDerivatives(*dims, fx, fy, fz), StencilDerivatives(*dims, gx, gy, gz)
    F, F2 = StencilCoupling(*dims, fel), StencilCoupling(*dims, gel.reshape(-1))
    rng = np.random.default_rng(sum(dims))
    dev = lambda *s: torch.as_tensor(rng.normal(size=s), device="cuda")  # noqa: E731
    new = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")  # noqa: E731

    def close(a, b, bound, what):
        assert float((a - b).abs().max()) <= bound + 1e-14 * float(b.abs().max()), what

    U, m, avg, u, E0 = dev(n), dev(n, 3), dev(3), dev(3 * n), dev(6 * n)
    big = lambda x: float(x.abs().max())  # noqa: E731
    close(D.hd_into(U, new(n, 3)), D2.hd_into(U, new(n, 3)), 2 * max(ex, ey, ez) * big(U), "Hd")
    a, b = D.demag_rhs_into(m, avg, new(n), pin=5), D2.demag_rhs_into(m, avg, new(n), pin=5)
    close(a, b, 2 * (ex + ey + ez) * big(m), "right-hand side")
    assert float(a[5]) == 0.0
    R = torch.as_tensor(np.linalg.qr(rng.normal(size=(3, 3)))[0], device="cuda")
    for rot in (None, R):
        # at most 6 derivatives enter a rotated component, each times at most 1
        close(D.compute_E_from_u(n, u, rot), D2.compute_E_from_u(n, u, rot), 12 * max(ex, ey, ez) * big(u), "strain")
    a, b = F.spmv(E0), F2.spmv(E0)
    close(a, b, 12 * eel * big(E0), "F_el E0")
    assert float(a[0]) == float(a[n]) == float(a[2 * n]) == 0.0


@pytest.mark.parametrize("dims", [(3, 3, 3), (17, 4, 5), (16, 33, 3), (35, 9, 31), (5, 40, 64)])
@pytest.mark.parametrize("nvec", [1, 3])
def test_marching_scalar_product_matches_the_per_node_form(dims, nvec):
    """Identity, empty and excluded rows among the flags; planes that the marches split unevenly.  One coefficient
    moved by 1e-13 of the largest keeps the per-node form: at most 1e-13 max|c| max|x| per output apart from
    rounding (27 terms)."""
    from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
    from cupymag_gb300.utils.stencil_operator import COL_EXCLUDED, ROW_IDENTITY, ROW_ZERO, StencilOperator
    from cupymag_gb300.workloads import hex_params
    so = SimulationOperators(hex_params(6, 1, False, False), device="cuda").stencil_operators()
    rng = np.random.default_rng(sum(dims) + nvec)
    n = dims[0] * dims[1] * dims[2]
    flags = np.zeros(n, dtype=np.uint8)
    flags[rng.integers(0, n, 3)] = ROW_IDENTITY | COL_EXCLUDED
    flags[rng.integers(0, n, 2)] = ROW_ZERO
    x = torch.as_tensor(rng.normal(size=(n, nvec) if nvec == 3 else n), device="cuda")
    for name in ("F1", "A1", "A_demag"):
        c = so[name].coef_host
        moved = c.copy()
        moved[5] += 1e-13 * np.abs(c).max()
        a = StencilOperator(*dims, c, flags).spmv(x, alpha=-2.0)
        b = StencilOperator(*dims, moved, flags).spmv(x, alpha=-2.0)
        big = float(x.abs().max())
        bound = 2 * (1e-13 * np.abs(c).max() + 54 * 2.0 ** -53 * np.abs(c).sum()) * big
        assert float((a - b).abs().max()) <= bound, name


# grids on both sides of the rule that picks the marching form, per product: small, flat and long ones
@pytest.mark.parametrize("dims", [(5, 7, 9), (6, 6, 7), (20, 21, 19), (44, 45, 43), (50, 45, 39), (130, 20, 33),
                                  (9, 130, 90), (256, 4, 70), (64, 150, 5)])
def test_products_match_on_both_sides_of_the_marching_rule(dims):
    test_marching_products_match_the_pair_kernels(dims)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_coefficients_that_are_not_finite_reach_the_result(bad):
    """A coefficient outside the mirror form's pattern (dx = 0 in F_x) that is not finite is no rounding of zero: the
    products with that stencil are not finite anywhere, on grids that otherwise march."""
    from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
    from cupymag_gb300.utils.stencil_derivatives import StencilCoupling, StencilDerivatives
    from cupymag_gb300.workloads import hex_params
    cell = SimulationOperators(hex_params(6, 1, True, True), device="cuda")
    fx, fy, fz = (f.copy() for f in cell.stencil_derivatives().coef)
    fel = cell.stencil_coupling().coef.copy()
    dims = (44, 45, 43)
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(1)
    dev = lambda *s: torch.as_tensor(rng.normal(size=s), device="cuda")  # noqa: E731
    fx[12] = bad       # offset (0, 0, -1)
    D = StencilDerivatives(*dims, fx, fy, fz)
    H = D.hd_into(dev(n), torch.empty((n, 3), dtype=torch.float64, device="cuda"))
    assert not torch.isfinite(H[:, 0]).any() and torch.isfinite(H[:, 1:]).all()
    b = D.demag_rhs_into(dev(n, 3), None, torch.empty(n, dtype=torch.float64, device="cuda"), pin=0)
    assert not torch.isfinite(b[1:]).any()
    fel[12 * 1 + 27 * 2] = bad   # block (0, 2)
    r = StencilCoupling(*dims, fel).spmv(dev(6 * n)).reshape(3, n)
    assert not torch.isfinite(r[0, 1:]).any() and torch.isfinite(r[1:]).all()
