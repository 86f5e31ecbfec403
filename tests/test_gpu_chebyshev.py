"""The Chebyshev iteration of the projection solves (A1, A2) against the CG form and the assembled matrices."""
import numpy as np
import pytest
import torch

from . import _golden as G

pytestmark = pytest.mark.gpu

# smallest eigenvalue of the free-node operators (the symbol's minimum, material of the golden case): a residual
# of tol ||b|| leaves ||x - x*|| <= tol ||b|| / sigma, so two solves differ by at most twice that
TOL = 1e-10


def _case(dims, defect):
    from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
    p = G.params(G.load("hex_me_rot")).with_(Nx=dims[0], Ny=dims[1], Nz=dims[2], Ndx=defect, Ndy=defect, Ndz=defect)
    S = SimulationOperators(p)
    return S, S.stencil_operators(), S.host_operators()


def _sigma(op):
    c = op.coef_host.reshape(3, 3, 3)
    return min(np.einsum("abc,a,b,c->", c, *[np.array([u, 1.0, u]) for u in (x, y, z)])
               for x in (1, -1) for y in (1, -1) for z in (1, -1))


def _solve(op, b, x0=None, form=0, maxiter=20000, precision="IR"):
    from cupymag_gb300.solvers.linear_solvers import CGSolver, decode_info, new_info
    bd = torch.as_tensor(b, device="cuda").contiguous()
    x = torch.zeros_like(bd) if x0 is None else torch.as_tensor(x0, device="cuda").clone().contiguous()
    info = new_info(1)
    CGSolver().launch(op, bd, x, info[0], tol=TOL, maxiter=maxiter, precision=precision, inner_tol=1e-5, form=form,
                      use_init=x0 is not None)
    return x.cpu().numpy(), decode_info(info[0].cpu().numpy())


# z-lines of 3 .. 130: quads with 1 to 4 unknowns, lines shorter and longer than a warp's run of 128
@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 3, 4), (4, 6, 5), (9, 10, 31), (6, 5, 33), (3, 9, 126), (4, 3, 128),
                                  (5, 4, 130), (33, 12, 11)])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_chebyshev_solves_match_cg(dims, nrhs):
    """Cold and warm, with a defect where one fits: the FP64 stopping test holds on the host, the solution is the
    CG form's within 2 tol ||b|| / sigma, pinned DOFs are exact, and the steps are the schedule's (cold: the same
    for every grid, far below CG's maximum)."""
    S, so, csr = _case(dims, 1 if min(dims) >= 5 else 0)
    rng = np.random.default_rng(sum(dims) + nrhs)
    for name in ("A1", "A2"):
        A, op = csr[name], so[name]
        n = A.shape[0]
        b = rng.normal(size=(n, nrhs)) if nrhs == 3 else rng.normal(size=n)
        if nrhs == 3:
            b[:, 1] *= 1e-9   # right-hand sides of very different size are scaled one by one
        x0 = rng.normal(size=b.shape)
        for warm in (None, x0):
            xc, ic = _solve(op, b, warm)
            xg, ig = _solve(op, b, warm, form=1)
            assert ic["status"] == 0 and ig["status"] == 0, (name, ic, ig)
            bb, cc, gg = b.reshape(n, -1), xc.reshape(n, -1), xg.reshape(n, -1)
            for r in range(nrhs):
                nb = np.linalg.norm(bb[:, r])
                assert np.linalg.norm(bb[:, r] - A @ cc[:, r]) <= TOL * nb, (name, r)
                assert np.linalg.norm(cc[:, r] - gg[:, r]) <= 2 * TOL * nb / _sigma(op), (name, r)
            assert np.array_equal(cc[S.DefDOF], bb[S.DefDOF])


def test_chebyshev_zero_and_tiny_right_hand_sides():
    """A zero column returns zeros (also from a warm start), one of norm 1e-30 is solved all the same."""
    S, so, csr = _case((8, 7, 9), 2)
    A, op = csr["A1"], so["A1"]
    rng = np.random.default_rng(3)
    b = rng.normal(size=(A.shape[0], 3))
    b[:, 1] = 0.0
    for x0 in (None, rng.normal(size=b.shape)):
        x, inf = _solve(op, b, x0)
        assert inf["status"] == 0 and inf["iters"][1] == 0 and not x[:, 1].any()
    b[:, 1] = rng.normal(size=A.shape[0]) * 1e-30
    x, inf = _solve(op, b)
    assert inf["status"] == 0
    for r in range(3):
        assert np.linalg.norm(b[:, r] - A @ x[:, r]) <= TOL * np.linalg.norm(b[:, r])


def test_rows_that_are_not_pinned_and_small_maxiter_keep_cg():
    """An empty row among the flags (not a pinned DOF) and a maxiter near the iteration counts run the CG form."""
    from cupymag_gb300 import _native as N
    from cupymag_gb300.utils.stencil_operator import COL_EXCLUDED, ROW_IDENTITY, StencilOperator
    S, so, csr = _case((8, 9, 10), 2)
    op = so["A1"]
    f = np.zeros(op.n, dtype=np.uint8)
    f[17] = ROW_IDENTITY                       # its column stays in the other rows
    f[300] = ROW_IDENTITY | COL_EXCLUDED
    odd = StencilOperator(op.nx, op.ny, op.nz, op.coef_host, f)
    b = np.random.default_rng(5).normal(size=op.n)
    b[17] = 0.0
    x, inf = _solve(odd, b)
    assert inf["status"] == 0, inf
    r = b - odd.spmv(torch.as_tensor(x, device="cuda")).cpu().numpy()
    assert np.linalg.norm(r) <= TOL * np.linalg.norm(b)
    b = np.random.default_rng(6).normal(size=op.n)
    for cap in (3, 50):
        _, inf = _solve(op, b, maxiter=cap)
        _, ref = _solve(op, b, maxiter=cap, form=N.CG_FORM_THREE_BARRIER)
        assert inf["iters"] == ref["iters"] and inf["status"] == ref["status"]


@pytest.mark.parametrize("nrhs", [1, 3])
def test_batched_chebyshev_is_the_same_alone_and_in_a_mix(nrhs):
    """Systems of one batch that run Chebyshev steps (different grids, one with a zero right-hand side) beside ones
    left to CG (a row that is not pinned; a maxiter below the rule): bit for bit the same alone and in the mix, the
    stopping test holds, and the Chebyshev systems give the single solver's steps."""
    from cupymag_gb300.serving.blockdiag import BlockDiagPlan, BlockSystem, work_bytes
    from cupymag_gb300.solvers.linear_solvers import decode_info, new_info
    from cupymag_gb300.utils.stencil_operator import COL_EXCLUDED, ROW_IDENTITY, StencilOperator
    rng = np.random.default_rng(nrhs)
    coef = _case((6, 6, 6), 0)[1]["A1"].coef_host
    ops = []
    for dims in ((7, 9, 11), (16, 16, 16), (5, 30, 33), (24, 20, 22), (8, 8, 8), (9, 9, 9)):
        f = np.zeros(dims[0] * dims[1] * dims[2], dtype=np.uint8)
        f[rng.integers(0, f.size, 5)] = ROW_IDENTITY | COL_EXCLUDED
        if dims == (8, 8, 8):
            f[100] = ROW_IDENTITY     # its column stays: CG
        ops.append(StencilOperator(*dims, coef, f))
    caps = [20000, 20000, 20000, 20000, 20000, 100]
    bs = [rng.normal(size=(o.n, nrhs)) if nrhs == 3 else rng.normal(size=o.n) for o in ops]
    bs[4].reshape(ops[4].n, -1)[100] = 0.0
    bs[3].reshape(ops[3].n, -1)[:, 0] = 0.0

    def solve(which):
        systems = []
        for i in which:
            b = torch.as_tensor(bs[i], device="cuda").contiguous()
            work = torch.empty(work_bytes((ops[i].nx, ops[i].ny, ops[i].nz), 1, nrhs, "IR"), dtype=torch.uint8,
                               device="cuda")
            systems.append(BlockSystem(ops[i], b, torch.zeros_like(b), new_info(1)[0], work, TOL, caps[i]))
        plan = BlockDiagPlan(systems, "IR", inner_tol=1e-5)
        plan.launch()
        first = [s.x.clone() for s in systems]
        plan.launch()   # a plan is launched many times
        out = [(s.x.cpu().numpy(), decode_info(s.info.cpu().numpy())) for s in systems]
        assert all(torch.equal(a, s.x) for a, s in zip(first, systems))
        return out

    mix = solve(range(len(ops)))
    for i, op in enumerate(ops):
        (x, inf), = solve([i])
        assert np.array_equal(x, mix[i][0]) and inf == mix[i][1], i
        assert inf["status"] == 0, (i, inf)
        b2, x2 = bs[i].reshape(op.n, -1), x.reshape(op.n, -1)
        for r in range(b2.shape[1]):
            y = op.spmv(torch.as_tensor(np.ascontiguousarray(x2[:, r]), device="cuda")).cpu().numpy()
            assert np.linalg.norm(b2[:, r] - y) <= 1.001 * TOL * np.linalg.norm(b2[:, r]), (i, r)
        if i < 4:
            _, ref = _solve(op, bs[i])
            assert ref["iters"] == inf["iters"] and inf["df_updates"] == ref["df_updates"], (i, inf, ref)
