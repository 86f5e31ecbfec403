"""Where the Chebyshev iteration of the projection solves hands over, decides and ends."""
import numpy as np
import pytest
import torch

from . import _golden as G

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _case(dims, defect):
    from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
    p = G.params(G.load("hex_me_rot")).with_(Nx=dims[0], Ny=dims[1], Nz=dims[2], Ndx=defect, Ndy=defect, Ndz=defect)
    S = SimulationOperators(p)
    return S, S.stencil_operators(), S.host_operators()


def _solve(op, b, x0=None, form=0, maxiter=20000, tol=TOL, solver=None):
    from cupymag_gb300.solvers.linear_solvers import CGSolver, decode_info, new_info
    bd = torch.as_tensor(b, device="cuda").contiguous()
    x = torch.zeros_like(bd) if x0 is None else torch.as_tensor(x0, device="cuda").clone().contiguous()
    info = new_info(1)
    (solver or CGSolver()).launch(op, bd, x, info[0], tol=tol, maxiter=maxiter, precision="IR", inner_tol=1e-5,
                                  form=form, use_init=x0 is not None)
    return x.cpu().numpy(), decode_info(info[0].cpu().numpy())


@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("dims", [(5, 4, 3), (12, 13, 14), (40, 33, 37)])
def test_hand_over_to_cg_gives_the_same_bits_every_time(dims, nrhs):
    """Systems with a flagged row that is not pinned run CG behind the Chebyshev start of the same launch: the
    stopping test holds and every repetition gives the same bits and the same record."""
    from cupymag_gb300.solvers.linear_solvers import CGSolver
    from cupymag_gb300.utils.stencil_operator import COL_EXCLUDED, ROW_IDENTITY, StencilOperator
    op = _case(dims, 0)[1]["A1"]
    f = np.zeros(op.n, dtype=np.uint8)
    f[17] = ROW_IDENTITY                       # its column stays in the other rows
    f[41] = ROW_IDENTITY | COL_EXCLUDED
    odd = StencilOperator(*dims, op.coef_host, f)
    rng = np.random.default_rng(8)
    b = rng.normal(size=(op.n, 3) if nrhs == 3 else op.n)
    b[17] = 0.0
    solver = CGSolver()
    for x0 in (None, 0.1 * rng.normal(size=b.shape)):
        if x0 is not None:
            x0[17] = 0.0
        x, inf = _solve(odd, b, x0, solver=solver)
        assert inf["status"] == 0, inf
        r = b - odd.spmv(torch.as_tensor(x, device="cuda")).cpu().numpy()
        assert np.all(np.linalg.norm(r.reshape(op.n, -1), axis=0) <=
                      1.001 * TOL * np.linalg.norm(b.reshape(op.n, -1), axis=0))
        for _ in range(40):
            y, other = _solve(odd, b, x0, solver=solver)
            assert np.array_equal(x, y) and inf == other


@pytest.mark.parametrize("nrhs", [1, 3])
def test_values_beyond_floats_end_as_in_cg(nrhs):
    """A warm start or a right-hand side that is not finite in floats: the status is the CG form's, and the next
    solve on the same workspace is sound."""
    from cupymag_gb300 import _native as N
    from cupymag_gb300.solvers.linear_solvers import CGSolver
    op = _case((9, 8, 10), 2)[1]["A2"]
    rng = np.random.default_rng(2)
    b = rng.normal(size=(op.n, 3) if nrhs == 3 else op.n)
    x0 = np.zeros_like(b)
    x0[5] = 1e200
    bad = b.copy()
    bad[3] = np.inf
    solver = CGSolver()
    ref, good = _solve(op, b, solver=solver)
    assert good["status"] == 0
    for rhs, start in ((b, x0), (bad, None)):
        _, inf = _solve(op, rhs, start, solver=solver)
        _, cg = _solve(op, rhs, start, form=N.CG_FORM_THREE_BARRIER)
        assert inf["status"] == cg["status"] != 0, (inf, cg)
        again, inf = _solve(op, b, solver=solver)
        assert np.array_equal(again, ref) and inf == good


@pytest.mark.parametrize("name", ["A1", "A2"])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_fp64_residuals_decide_where_they_are_asked_for(name, nrhs):
    """df_residual = False: every cycle of a cold solve ends with an FP64 residual of the x that is returned (the
    default form proves the last one in FP32).  The residual reported is then that of x to the rounding of an FP64
    product, 64 * 2^-53 sum|c| ||x||, relative to a residual near tol ||b||."""
    from cupymag_gb300.solvers.linear_solvers import CGSolver
    S, so, csr = _case((12, 11, 13), 3)
    A, op = csr[name], so[name]
    rng = np.random.default_rng(7)
    b = rng.normal(size=(op.n, 3) if nrhs == 3 else op.n)
    solver = CGSolver()
    _, fast = _solve(op, b, solver=solver)
    solver.df_residual = False
    x, inf = _solve(op, b, solver=solver)
    assert inf["status"] == 0 and inf["df_updates"] == 0 and fast["df_updates"] == fast["outer"] >= 1
    assert inf["iters"] == fast["iters"] and inf["outer"] == fast["outer"] + 1, (inf, fast)
    bb, xx = b.reshape(op.n, -1), x.reshape(op.n, -1)
    for r in range(nrhs):
        res = np.linalg.norm(bb[:, r] - A @ xx[:, r])
        tol = 64 * 2.0 ** -53 * np.abs(op.coef_host).sum() * np.linalg.norm(xx[:, r])
        assert res <= TOL * np.linalg.norm(bb[:, r])
        assert abs(inf["resid"][r] - res) <= tol, (inf["resid"][r], res, tol)


def test_residual_norm_that_decides_is_summed_in_fp64():
    """b = 1 without pinned DOFs: every node holds the same residual, and a loose tolerance with a warm start of
    1.2e6 half tolerances ends on a double-float residual after one cycle.  Its norm is that of x to the double-float
    bound, 128 * 2^-48 sum|c| max|x| per node, and 512 roundings of FP64 sums (256 equal squares per thread in FP32
    would be off by 1e-7)."""
    from fractions import Fraction
    from cupymag_gb300.utils.stencil_operator import StencilOperator
    coef = _case((4, 4, 4), 0)[1]["A1"].coef_host
    op = StencilOperator(256, 280, 280, coef)
    tol = 1e-2
    b = np.ones(op.n)
    x, inf = _solve(op, b, np.full(op.n, 1.0 + 1.2e6 * 0.5 * tol), tol=tol)
    assert inf["status"] == 0 and inf["outer"] == inf["df_updates"] == 1, inf
    assert np.all(x == x[0])
    r = abs(float(1 - sum(Fraction(float(c)) for c in coef) * Fraction(float(x[0]))))
    assert 0.1 * tol < r <= tol
    err = 128 * 2.0 ** -48 * np.abs(coef).sum() * abs(x[0]) / r + 512 * 2.0 ** -53
    assert abs(inf["resid"][0] / (r * np.sqrt(op.n)) - 1) <= err, (inf["resid"][0], r * np.sqrt(op.n), err)


def _residuals(A, b, x):
    n = b.shape[0]
    bb, xx = b.reshape(n, -1), x.reshape(n, -1)
    return [np.linalg.norm(bb[:, r] - A @ xx[:, r]) / np.linalg.norm(bb[:, r]) for r in range(bb.shape[1])]


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -200, 2.0 ** 300])
@pytest.mark.parametrize("df", [True, False])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_warm_start_far_from_the_solution_takes_several_cycles(nrhs, df, scale):
    """Three and more cycles (corrections beyond the pair of a cold start), in both residual forms and with
    right-hand sides that are scaled down and up; pinned DOFs are exact."""
    from cupymag_gb300.solvers.linear_solvers import CGSolver
    S, so, csr = _case((9, 12, 7), 2)
    A, op = csr["A2"], so["A2"]
    rng = np.random.default_rng(11)
    b = rng.normal(size=(op.n, 3) if nrhs == 3 else op.n)
    x0 = 1e4 * rng.normal(size=b.shape)
    solver = CGSolver()
    solver.df_residual = df
    x, inf = _solve(op, scale * b, scale * x0, solver=solver)
    assert inf["status"] == 0 and inf["outer"] >= 2, inf
    assert max(_residuals(A, b, x / scale)) <= TOL
    assert np.array_equal(x[S.DefDOF], scale * b[S.DefDOF])
    y, _ = _solve(op, b, x0, solver=solver)
    assert np.array_equal(scale * y, x)


@pytest.mark.parametrize("nz", [5, 8])
@pytest.mark.parametrize("ratio", [0.02, 0.0158])
def test_wide_spectrum(ratio, nz):
    """Condition numbers of 50 and 63 (a cycle's FP32 rounding leaves more for the next): the stopping test holds,
    cold and warm, with either residual."""
    from cupymag_gb300.solvers.linear_solvers import CGSolver
    from cupymag_gb300.utils.stencil_operator import StencilOperator
    t = (1 - ratio ** (1 / 3)) / 4   # symbol of the tensor product: (1 - 2 t + 2 t cos)^3, between 1 and `ratio`
    one = np.array([t, 1 - 2 * t, t])
    op = StencilOperator(11, 6, nz, np.einsum("a,b,c->abc", one, one, one).reshape(27))
    rng = np.random.default_rng(1)
    b = rng.normal(size=op.n)
    for df in (True, False):
        solver = CGSolver()
        solver.df_residual = df
        for x0 in (None, rng.normal(size=op.n)):
            x, inf = _solve(op, b, x0, tol=1e-9, solver=solver)
            r = b - op.spmv(torch.as_tensor(x, device="cuda")).cpu().numpy()
            assert inf["status"] == 0 and np.linalg.norm(r) <= 1e-9 * np.linalg.norm(b), inf


@pytest.mark.parametrize("name,steps", [("A1", 40), ("A2", 60)])
def test_the_default_form_runs_the_schedule(name, steps):
    """Cold solves to 1e-10 take the iteration's own step count (one less or more by the sizes of the two cycles) on
    every grid, with double-float residuals, where CG's count depends on the grid and the right-hand side."""
    for dims in ((8, 9, 10), (21, 5, 33), (30, 28, 26)):
        op = _case(dims, 2)[1][name]
        for nrhs in (1, 3):
            b = np.random.default_rng(dims[2]).normal(size=(op.n, 3) if nrhs == 3 else op.n)
            _, inf = _solve(op, b)
            _, cg = _solve(op, b, form=1)
            assert inf["status"] == 0 and abs(inf["iters"][0] - steps) <= 1, inf
            assert inf["iters"][:nrhs] == inf["iters"][:1] * nrhs and inf["outer"] == inf["df_updates"] == 1, inf
            assert cg["iters"][0] < steps - 2, cg


@pytest.mark.parametrize("dims,nrhs", [((672, 672, 672), 1), ((3, 1500, 1500), 3), ((1200, 330, 260), 3)])
def test_large_grids_run_the_schedule(dims, nrhs):
    """Grids whose residual passes are cut by what the partial sums hold, and the flattest planes: the schedule's steps
    and the stopping test against an FP64 product."""
    from cupymag_gb300 import _native as N
    from cupymag_gb300.solvers.linear_solvers import CGSolver, decode_info, new_info
    from cupymag_gb300.utils.stencil_operator import StencilOperator
    n = dims[0] * dims[1] * dims[2]
    free, _ = torch.cuda.mem_get_info()
    if free < 70 * n * nrhs + (8 << 30):
        pytest.skip("not enough device memory")
    op = StencilOperator(*dims, _case((4, 4, 4), 0)[1]["A1"].coef_host)
    steps = N.lib().cpm_stencil_cheb_steps(op.struct(), nrhs, TOL, 20000)
    g = torch.Generator(device="cuda").manual_seed(5)
    b = torch.randn((n, 3) if nrhs == 3 else n, dtype=torch.float64, device="cuda", generator=g)
    x, info = torch.zeros_like(b), new_info(1)
    CGSolver().launch(op, b, x, info[0], tol=TOL, maxiter=20000, precision="IR")
    inf = decode_info(info[0].cpu().numpy())
    assert inf["status"] == 0 and steps == 40 and abs(inf["iters"][0] - steps) <= 1, inf
    r = torch.linalg.norm(b - op.spmv(x), dim=0)
    assert bool((r <= 1.001 * TOL * torch.linalg.norm(b, dim=0)).all())
    del b, x, r
    torch.cuda.empty_cache()


@pytest.mark.parametrize("maxiter", [0, 1, 2, 5])
@pytest.mark.parametrize("tol", [0.5, 1.9, 2.0, 40.0])
def test_loose_tolerances_respect_a_small_maxiter(tol, maxiter):
    """A tolerance that x = 0 meets already, with fewer iterations allowed than four cycles: CG's record (one
    iteration at least)."""
    from cupymag_gb300 import _native as N
    op = _case((8, 7, 9), 2)[1]["A1"]
    b = np.random.default_rng(3).normal(size=op.n)
    _, inf = _solve(op, b, tol=tol, maxiter=maxiter)
    _, cg = _solve(op, b, tol=tol, maxiter=maxiter, form=N.CG_FORM_THREE_BARRIER)
    assert inf["iters"][0] <= max(maxiter, 1) and inf["status"] == cg["status"] and inf["iters"] == cg["iters"], (inf, cg)


@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("nz", [7, 8])
def test_workspaces_aligned_to_8_bytes_are_solved(nz, nrhs):
    """A workspace of the full size that starts 8 bytes off a 16-byte boundary runs CG on scalar loads (it is compared
    with the aligned one only in what both promise: status, stopping test and pinned rows)."""
    import ctypes as C
    from cupymag_gb300 import _native as N
    from cupymag_gb300.solvers.linear_solvers import decode_info, new_info
    S, so, csr = _case((9, 8, nz), 2)
    A, op = csr["A1"], so["A1"]
    b = np.random.default_rng(nz).normal(size=(op.n, 3) if nrhs == 3 else op.n)
    bd = torch.as_tensor(b, device="cuda").contiguous()
    L = N.lib()
    nbytes = int(L.cpm_cg_stencil_workspace(op.struct(), nrhs, 1))
    mem = torch.zeros(nbytes + 64, dtype=torch.uint8, device="cuda")
    for off in (0, 8):
        ws = mem[off:off + nbytes]
        assert ws.data_ptr() % 16 == off
        x, info = torch.zeros_like(bd), new_info(1)
        o = N.CGOpts()
        o.tol, o.maxiter, o.precision, o.inner_tol, o.barrier_timeout_s = TOL, 20000, 1, 1e-5, 2.0
        assert L.cpm_cg_solve_stencil(op.struct(), bd.data_ptr(), x.data_ptr(), nrhs, C.byref(o), ws.data_ptr(), nbytes,
                                      info[0].data_ptr(), N.stream_ptr()) == N.CPM_OK
        inf = decode_info(info[0].cpu().numpy())
        assert inf["status"] == 0 and (inf["iters"][0] >= 39) == (off == 0), inf
        xs = x.cpu().numpy()
        assert max(_residuals(A, b, xs)) <= TOL
        assert np.array_equal(xs[S.DefDOF], b[S.DefDOF])


@pytest.mark.parametrize("dims,name", [((120, 100, 3), "A1"), ((130, 80, 4), "A2"), ((90, 60, 8), "A1"),
                                       ((500, 800, 12), "A1"), ((60, 50, 16), "A2")])
def test_cold_solves_of_one_vector_on_short_lines_keep_cg(dims, name):
    """One right-hand side from a cold start runs CG on grids of short z-lines, three right-hand sides and warm starts
    (nz = 4 below a million nodes) the Chebyshev schedule; both meet the stopping test."""
    from cupymag_gb300.utils.stencil_operator import StencilOperator
    op = StencilOperator(*dims, _case((4, 4, 4), 0)[1][name].coef_host)
    rng = np.random.default_rng(dims[2])
    b = rng.normal(size=(op.n, 3))
    one = np.ascontiguousarray(b[:, 0])
    product = lambda v: op.spmv(torch.as_tensor(v, device="cuda")).cpu().numpy()  # noqa: E731
    for rhs, x0, cheb in ((one, None, False), (b, None, True), (one, rng.normal(size=op.n), True)):
        x, inf = _solve(op, rhs, x0)
        _, cg = _solve(op, rhs, x0, form=1)
        assert inf["status"] == 0 and (inf["iters"] != cg["iters"]) == cheb, (inf, cg)
        r = np.linalg.norm((rhs - product(x)).reshape(op.n, -1), axis=0)
        assert np.all(r <= 1.001 * TOL * np.linalg.norm(rhs.reshape(op.n, -1), axis=0))
