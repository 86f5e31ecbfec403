"""What a user of this package has it do, as cases that can be timed and checked.

A case is a dict of plain values.  Its ``kind`` says which public entry points it goes through:

* ``step``    one Gauss-Seidel-projection LLG step (LLGSolver.step) from a given magnetisation;
* ``gs``      a projection solve A1 x = b or A2 x = b of the step (CGSolver.launch, or solve_cg as a
              script of the reference calls it), one or three right-hand sides, cold or warm;
* ``field``   an elastic or demag equilibrium solve in the precision form (CGSolver.launch, FFT solver);
* ``products``  the derivative products of a step: b_el = F_el E0, the strain of a displacement, the demag
              right-hand side b = -div(m - <m>) and H = -grad U;
* ``batch``   the projection solves of several served runs of different sizes in one launch;
* ``tet``     a CSR solve on an unstructured tetrahedral mesh.

Material, time step, tolerance and sweep are those of the package's own workloads.  ``exact`` computes the
same results in 64 bits with NumPy and torch alone, from the raw material constants and the element
integrals (trilinear hex, linear tet).
"""
import math

import numpy as np
import torch

MU0, GAMMA = 1.25663706127e-6, 1.76e11
DEV = "cuda"
TOL, MAXITER = 1e-10, 20000
F64 = torch.float64


# ---------------------------------------------------------------------------------------- the cases
def _grid(nx, ny, nz, defect):
    return {"nx": nx, "ny": ny, "nz": nz, "defect": defect}


def listed():
    return [
        # the headline run: 128^3 magnetoelastic hysteresis sweep, precision form, matrix-free operators
        {"name": "step_me_128", "kind": "step", **_grid(128, 128, 128, 16), "ME": True, "precision": "IR",
         "operators": "stencil"},
        # a mid-sized magnetoelastic film cell with odd edges, as a parameter study steps it
        {"name": "step_me_48", "kind": "step", **_grid(50, 45, 39, 10), "ME": True, "precision": "IR",
         "operators": "stencil"},
        # the small plain run in the package's default form: FP64 on CSR operators
        {"name": "step_plain_32_dp", "kind": "step", **_grid(32, 32, 32, 4), "ME": False, "precision": "DP",
         "operators": "csr"},
        # the same default accuracy (FP64) on matrix-free operators, with coupling: the parity runs
        {"name": "step_me_40_dp", "kind": "step", **_grid(40, 40, 40, 6), "ME": True, "precision": "DP",
         "operators": "stencil"},
        # first projection solve of a large step (g1, g2, g3 together), cold
        {"name": "gs_a1x3_112", "kind": "gs", **_grid(112, 96, 90, 14), "op": "A1", "nrhs": 3, "warm": False,
         "api": "solver"},
        # last projection solve of a large plain run near its equilibrium: warm-started
        {"name": "gs_a2x3_176", "kind": "gs", **_grid(176, 160, 168, 24), "op": "A2", "nrhs": 3, "warm": True,
         "api": "solver"},
        # the smallest call: one scalar projection solve through the drop-in solve_cg
        {"name": "gs_a1_20", "kind": "gs", **_grid(20, 20, 20, 4), "op": "A1", "nrhs": 1, "warm": False,
         "api": "solve_cg"},
        # elastic equilibrium of a ragged grid, and the demag potential of a large plain run
        {"name": "elastic_90", "kind": "field", **_grid(96, 81, 90, 12), "op": "A_el", "warm": False},
        {"name": "demag_192", "kind": "field", **_grid(192, 192, 180, 24), "op": "A_demag", "warm": False},
        # the coupling and gradient products of a large run
        {"name": "products_110", "kind": "products", **_grid(110, 112, 105, 16)},
        # the solves of a serving step: runs of 16^3 to 54^3 batched
        {"name": "batch_a1x3_8", "kind": "batch", "op": "A1", "nrhs": 3, "count": 8, "lo": 16, "hi": 54, "pick": 3},
        # the demag potential on a jittered tetrahedral mesh with an ellipsoidal defect, FP64
        {"name": "tet_demag_22", "kind": "tet", "n": 22, "op": "A_demag", "nrhs": 1, "precision": "DP"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng, lo, hi):
    e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = [min(hi, max(lo, int(round(e * rng.uniform(0.85, 1.15))))) for _ in range(3)]
    return _grid(*n, rng.randint(0, min(n) // 5))


def draw(rng):
    kind = rng.choice(["step", "step", "gs", "gs", "gs", "field", "products", "batch", "tet"])
    if kind == "step":
        dp = rng.random() < 0.3
        ops = rng.choice(["csr", "stencil"]) if dp else "stencil"
        hi = 120 if not dp else 30 if ops == "csr" else 38
        return {"kind": kind, **_draw_grid(rng, 12, hi), "ME": rng.random() < (0.4 if dp else 0.7),
                "precision": "DP" if dp else "IR", "operators": ops}
    if kind == "gs":
        return {"kind": kind, **_draw_grid(rng, 12, 160), "op": rng.choice(["A1", "A2"]), "nrhs": rng.choice([1, 3]),
                "warm": rng.random() < 0.4, "api": rng.choice(["solver", "solver", "solve_cg"])}
    if kind == "field":
        op = rng.choice(["A_el", "A_demag"])
        return {"kind": kind, **_draw_grid(rng, 16, 110 if op == "A_el" else 180), "op": op,
                "warm": rng.random() < 0.3}
    if kind == "products":
        return {"kind": kind, **_draw_grid(rng, 12, 128)}
    if kind == "batch":
        return {"kind": kind, "op": rng.choice(["A1", "A2"]), "nrhs": rng.choice([1, 3]), "count": rng.randint(2, 12),
                "lo": 16, "hi": _log_int(rng, 20, 64), "pick": rng.randint(0, 10 ** 6)}
    op = rng.choice(["A_demag", "A1"])
    return {"kind": kind, "n": _log_int(rng, 8, 24), "op": op, "nrhs": 1 if op == "A_demag" else 3,
            "precision": rng.choice(["DP", "IR"])}


# ------------------------------------------------------------------- material and element integrals
class _Mat:
    """The workloads' material, nondimensional."""
    ms, ld, ad = 1.2e6, 10.0e-9, 0.1
    psi0 = MU0 * ms ** 2
    K1 = 2.0e4 / psi0
    dt = 1e-12 * (MU0 * GAMMA) * ms / (1 + ad ** 2)
    alpha = 2 * (1.5e-11 / psi0) / ld ** 2 * dt
    c11, c12, c44 = 196.0e9 / psi0, 156.0e9 / psi0, 123.0e9 / psi0
    l100, l111 = 2.0e-4, -2.0e-5
    s0 = -50.0e6 / psi0
    H = (0.1 / MU0 / ms, 0.0, 0.0)


_G = 0.57735026919
_CORN = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                  [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=np.float64)
_OFF = ((_CORN + 1) // 2).astype(int)
_GP = [(a, b, c) for a in (-_G, _G) for b in (-_G, _G) for c in (-_G, _G)]


def _hex_N(q):
    return np.prod(1 + _CORN * np.asarray(q), axis=1) / 8.0


def _hex_dN(q):
    f = 1 + _CORN * np.asarray(q)
    return np.stack([_CORN[:, 0] * f[:, 1] * f[:, 2] / 8, _CORN[:, 1] * f[:, 0] * f[:, 2] / 8,
                     _CORN[:, 2] * f[:, 0] * f[:, 1] / 8], axis=1)


def _rot():
    i2, i3, i6 = 1 / math.sqrt(2), 1 / math.sqrt(3), 1 / math.sqrt(6)
    s2, s3 = math.sqrt(2), math.sqrt(3)
    R = np.array([[i3, i3, i3], [-i2, i2, 0], [-i6, -i6, 2 * i6]])
    M = np.array([[1 / 3, 1 / 3, 1 / 3, 2 / 3, 2 / 3, 2 / 3], [1 / 2, 1 / 2, 0, 0, 0, -1.0],
                  [1 / 6, 1 / 6, 2 / 3, -2 / 3, -2 / 3, 1 / 3], [s3 / 6, -s3 / 6, 0, s3 / 3, -s3 / 3, 0],
                  [-s2 / 6, -s2 / 6, s2 / 3, s2 / 6, s2 / 6, -s2 / 3], [-i6, i6, 0, i6, -i6, 0]])
    return R, M


def _stencil(Ke, r=1, c=1):
    S = np.zeros((r, c, 3, 3, 3))
    for a in range(8):
        for b in range(8):
            d = _OFF[b] - _OFF[a] + 1
            S[:, :, d[0], d[1], d[2]] += Ke[a * r:(a + 1) * r, b * c:(b + 1) * c]
    return S


def _stencils():
    """27-point stencils of the unit cell's operators: K, M, F (3), Kel (3x3), Fel (3x6); [..., dx, dy, dz].
    The shape tables are rounded to 12 decimals, as the assembled operators' are."""
    xe = _OFF.astype(float)
    _, Mr = _rot()
    C = np.zeros((6, 6))
    C[:3, :3] = _Mat.c12
    np.fill_diagonal(C[:3, :3], _Mat.c11)
    C[3, 3] = C[4, 4] = C[5, 5] = _Mat.c44
    C = Mr @ C @ Mr.T
    K, M, F = np.zeros((8, 8)), np.zeros((8, 8)), np.zeros((3, 8, 8))
    Kel, Fel = np.zeros((24, 24)), np.zeros((24, 48))
    for q in _GP:
        dN, Nv = np.round(_hex_dN(q), 12), np.round(_hex_N(q), 12)
        J = xe.T @ dN
        w, g = np.linalg.det(J), (np.linalg.inv(J) @ dN.T).T
        K += g @ g.T * w
        M += np.outer(Nv, Nv) * w
        for i in range(3):
            F[i] += np.outer(Nv, g[:, i]) * w
        B = np.zeros((6, 8, 3))
        for row, comp, dr in ((0, 0, 0), (1, 1, 1), (2, 2, 2), (3, 0, 1), (3, 1, 0), (4, 1, 2), (4, 2, 1), (5, 0, 2),
                              (5, 2, 0)):
            B[row, :, comp] = g[:, dr]
        B = B.reshape(6, 24)
        Kel += B.T @ C @ B * w
        Fel += ((B.T @ C)[:, None, :] * Nv[None, :, None]).reshape(24, 48) * w
    return {"K": _stencil(K)[0, 0], "M": _stencil(M)[0, 0], "F": [_stencil(f)[0, 0] for f in F],
            "Kel": _stencil(Kel, 3, 3), "Fel": _stencil(Fel, 3, 6)}


def _gs_coef(st, op):
    return st["K"] * (_Mat.alpha if op == "A1" else _Mat.alpha * _Mat.ad) + st["M"]


def _apply(S, x):
    """sum_d S[d] x(p + d) on the periodic grid; x (nx, ny, nz)."""
    y = torch.zeros_like(x)
    for a in range(3):
        xa = torch.roll(x, 1 - a, 0)
        for b in range(3):
            xb = torch.roll(xa, 1 - b, 1)
            for c in range(3):
                if S[a, b, c] != 0.0:
                    y.add_(torch.roll(xb, 1 - c, 2), alpha=float(S[a, b, c]))
    return y


def _defect(dims, nd):
    """Defect DOFs of a centred cube of nd^3 cells, as a boolean (nx, ny, nz) tensor."""
    ax = []
    for N in dims:
        c = np.arange(N) + 0.5
        ax.append((c >= N / 2 - nd / 2) & (c < N / 2 + nd / 2))
    cells = torch.as_tensor(ax[0][:, None, None] & ax[1][None, :, None] & ax[2][None, None, :], device=DEV)
    mark = torch.zeros_like(cells)
    for i in (0, 1):
        for j in (0, 1):
            for k in (0, 1):
                mark |= torch.roll(cells, (i, j, k), (0, 1, 2))
    return mark


def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _m0(dims, mark, seed):
    """normalise((1, 0, 0) + N(0, 1e-3)), zero on the defect: (n, 3)."""
    m = torch.randn((*dims, 3), generator=_rng(seed), device=DEV, dtype=F64) * 1e-3
    m[..., 0] += 1.0
    m /= m.norm(dim=-1, keepdim=True)
    m[mark] = 0.0
    return m.reshape(-1, 3).contiguous()


def _E0(m):
    """Eigenstrain (n, 6) in the [111] frame."""
    R, M = (torch.as_tensor(a, device=DEV, dtype=F64) for a in _rot())
    x, y, z = (m @ R).unbind(1)
    a, b = 1.5 * _Mat.l100, 3.0 * _Mat.l111
    e = torch.stack([a * (x * x - 1 / 3), a * (y * y - 1 / 3), a * (z * z - 1 / 3), b * x * y, b * y * z, b * x * z], 1)
    return e @ M.T


def _fel(st, E0, dims):
    b = torch.stack([sum(_apply(st["Fel"][a, v], E0[:, v].reshape(dims)) for v in range(6)) for a in range(3)])
    b[:, 0, 0, 0] = 0.0
    return b.reshape(-1)


def _div(st, m, dims):
    b = -sum(_apply(st["F"][i], m[:, i].reshape(dims)) for i in range(3))
    b[0, 0, 0] = 0.0
    return b.reshape(-1)


def _grad(st, U, dims):
    return torch.stack([-_apply(st["F"][i], U.reshape(dims)).reshape(-1) for i in range(3)], 1)


def _strain(st, u, dims):
    R = _rot()[0]
    u = u.reshape(3, *dims)
    d = [[_apply(st["F"][i], u[c]).reshape(-1) for c in range(3)] for i in range(3)]
    t = [[sum(R[i, a] * d[i][c] for i in range(3)) for c in range(3)] for a in range(3)]
    return torch.stack([t[0][0], t[1][1], t[2][2], t[1][0] + t[0][1], t[2][1] + t[1][2], t[2][0] + t[0][2]], 1)


# ---------------------------------------------------------------------------- 64-bit reference solves
def _cg64(apply, b):
    """CG to 1e-14 of ||b|| on (n,) or (n, k) with one set of scalars per column."""
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), (r * r).sum(0)
    stop = 1e-28 * rr
    for k in range(20000):
        q = apply(p)
        den = (p * q).sum(0)
        al = torch.where(den > 0, rr / den, torch.zeros_like(rr))
        x += al * p
        r -= al * q
        new = (r * r).sum(0)
        if k % 8 == 7 and bool((new <= stop).all()):
            break
        p = r + torch.where(rr > 0, new / rr, torch.zeros_like(rr)) * p
        rr = new
    return x


def _gs64(S, b, dims, mark):
    """Projection solve with the defect DOFs pinned at b; b (n,) or (n, k)."""
    free = (~mark).reshape(-1).to(F64)
    f = free if b.dim() == 1 else free[:, None]

    def ap(p):
        cols = [p] if p.dim() == 1 else list(p.unbind(1))
        y = [_apply(S, c.reshape(dims)).reshape(-1) for c in cols]
        return f * (y[0] if p.dim() == 1 else torch.stack(y, 1))

    return _cg64(ap, b * f) + b * (1 - f)


def _circ64(S, b, dims):
    """The anchored circulant solve: node 0 pinned at b = 0, S (nc, nc, 3, 3, 3); b (nc n,)."""
    nc = S.shape[0]
    t = b.reshape(nc, *dims).clone()
    for c in range(nc):
        t[c, 0, 0, 0] -= t[c].sum()
    ker = torch.zeros((nc, nc, *dims), dtype=F64, device=DEV)
    for a in range(3):
        for e in range(3):
            for g in range(3):
                ker[:, :, (1 - a) % dims[0], (1 - e) % dims[1], (1 - g) % dims[2]] += torch.as_tensor(
                    S[:, :, a, e, g], device=DEV)
    sym = torch.fft.rfftn(ker, dim=(2, 3, 4)).permute(2, 3, 4, 0, 1).contiguous()
    th = torch.fft.rfftn(t, dim=(1, 2, 3)).permute(1, 2, 3, 0).unsqueeze(-1)
    sym[0, 0, 0] = torch.eye(nc, dtype=sym.dtype, device=DEV)
    th[0, 0, 0] = 0
    if nc == 1:
        eh = th / sym
    else:  # explicit inverse by cofactors: symbols are Hermitian 3x3
        m = [[sym[..., i, j] for j in range(3)] for i in range(3)]
        cof = lambda i, j: (m[(i + 1) % 3][(j + 1) % 3] * m[(i + 2) % 3][(j + 2) % 3]  # noqa: E731
                            - m[(i + 1) % 3][(j + 2) % 3] * m[(i + 2) % 3][(j + 1) % 3])
        co = [[cof(i, j) for j in range(3)] for i in range(3)]
        det = sum(m[0][j] * co[0][j] for j in range(3))
        eh = torch.stack([sum(co[j][i] * th[..., j, 0] for j in range(3)) / det for i in range(3)], -1).unsqueeze(-1)
    e = torch.fft.irfftn(eh.squeeze(-1).permute(3, 0, 1, 2), s=dims, dim=(1, 2, 3))
    e -= e[:, :1, :1, :1].clone()
    return e.reshape(-1)


def _avg_weights(dims):
    """Per-DOF weights of the volume average: the Jacobian is taken from coordinates looked up by DOF id, as the
    reference does (volume_average.py:76,108)."""
    nx, ny, nz = dims
    ar = lambda n: torch.arange(n, device=DEV)  # noqa: E731
    i, j, k = (v.reshape(-1) for v in torch.meshgrid(ar(nx), ar(ny), ar(nz), indexing="ij"))
    dof = [((i + a) % nx) * ny * nz + ((j + b) % ny) * nz + (k + c) % nz for a, b, c in _OFF.tolist()]
    node = lambda d: torch.stack([d // ((ny + 1) * (nz + 1)), d // (nz + 1) % (ny + 1), d % (nz + 1)], -1)  # noqa: E731
    xe = [node(d).to(F64) for d in dof]
    w, vol = torch.zeros(nx * ny * nz, dtype=F64, device=DEV), 0.0
    for q in _GP:
        dN, Nv = _hex_dN(q), _hex_N(q)
        J = [sum(xe[c] * float(dN[c, r]) for c in range(8)) for r in range(3)]
        det = (J[0] * torch.linalg.cross(J[1], J[2])).sum(1).abs()
        for c in range(8):
            w.index_add_(0, dof[c], det * float(Nv[c]))
        vol += float(det.sum())
    return w, vol


def _field64(m, E, Ht, avg, R):
    c = _Mat
    C1 = 2 * c.c44 * (1.5 * c.l111 ** 2) - (c.c11 - c.c12) * (1.5 * c.l100) ** 2
    C2, C3 = -1.5 * c.l100 * (c.c11 - c.c12), -6.0 * c.l111 * c.c44
    y = m if R is None else m @ R
    s = y * y
    o = s.sum(1, keepdim=True) - s
    v = -2 * c.K1 * y * o
    if E is not None:
        x0, x1, x2 = y.unbind(1)
        v = v - 2 * C1 * y * o - 2 * C2 * (E[:, :3] - c.l100) * y - C3 * torch.stack(
            [E[:, 3] * x1 + E[:, 5] * x2, E[:, 4] * x2 + E[:, 3] * x0, E[:, 5] * x0 + E[:, 4] * x1], 1)
    v = v if R is None else v @ R.T
    return v - avg / 6 + 0.5 * Ht + torch.tensor(c.H, dtype=F64, device=DEV)


def _step64(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    st, c = _stencils(), _Mat
    mark = _defect(dims, case["defect"])
    m = _m0(dims, mark, seed)
    w, vol = _avg_weights(dims)
    avg = lambda f: (w @ f) / vol  # noqa: E731
    am, ME = avg(m), case["ME"]
    R, M = (torch.as_tensor(a, device=DEV, dtype=F64) for a in _rot())
    E = None
    if ME:
        u = _circ64(st["Kel"], _fel(st, _E0(m), dims), dims)
        E = _strain(st, u, dims)
        a0, a1, a2 = (am @ R).tolist()
        den = c.c11 ** 2 + c.c11 * c.c12 - 2 * c.c12 ** 2
        s11, s12 = (c.c11 + c.c12) / den, -c.c12 / den
        eb = torch.tensor([1.5 * c.l100 * (a0 * a0 - 1 / 3) + s11 * c.s0, 1.5 * c.l100 * (a1 * a1 - 1 / 3) + s12 * c.s0,
                           1.5 * c.l100 * (a2 * a2 - 1 / 3) + s12 * c.s0, 3 * c.l111 * a0 * a1, 3 * c.l111 * a1 * a2,
                           3 * c.l111 * a0 * a2], dtype=F64, device=DEV)
        E = (E - avg(E) + M @ eb) @ torch.linalg.inv(M).T
    U = _circ64(st["K"][None, None], _div(st, m - am, dims), dims)
    Ht = _grad(st, U, dims)
    rot = R if ME else None
    f = _field64(m, E, Ht, am, rot)
    free = (~mark).reshape(-1).to(F64)
    F1 = lambda t: free * _apply(st["M"], t.reshape(dims)).reshape(-1)  # noqa: E731
    solve = lambda op, t: _gs64(_gs_coef(st, op), F1(t), dims, mark)  # noqa: E731
    t = f * c.dt + m
    g = [solve("A1", t[:, i]) for i in range(3)]
    m1 = m[:, 0] + g[1] * m[:, 2] - g[2] * m[:, 1]
    g1 = solve("A1", f[:, 0] * c.dt + m1)
    m2 = m[:, 1] + g[2] * m1 - g1 * m[:, 2]
    g2 = solve("A1", f[:, 1] * c.dt + m2)
    m3 = m[:, 2] + g1 * m2 - g2 * m1
    ms = torch.stack([m1, m2, m3], 1)
    h = _field64(ms, E, Ht, am, rot) * (c.dt * c.ad) + ms
    mm = torch.stack([solve("A2", h[:, i]) for i in range(3)], 1)
    mag = mm.norm(dim=1, keepdim=True)
    m = torch.where(mag < 1e-14, torch.zeros_like(mm), mm / mag) * free[:, None]
    out = {"m": m, "avg": avg(m), "Ht": Ht}
    if ME:
        out["E"] = E
    return out


# ------------------------------------------------------------------------------------- tet meshes
def _tet_mesh(n, seed):
    """A cube of n^3 cells cut into six tetrahedra each, interior nodes jittered by +-0.2."""
    g = np.arange(n + 1, dtype=np.float64)
    co = np.stack([v.ravel() for v in np.meshgrid(g, g, g, indexing="ij")], 1)
    inner = np.all((co > 0) & (co < n), axis=1)
    co[inner] += np.random.default_rng(seed).uniform(-0.2, 0.2, (int(inner.sum()), 3))
    cells = np.stack([v.ravel() for v in np.meshgrid(*[np.arange(n)] * 3, indexing="ij")], 1)
    node = lambda c: (c[:, 0] * (n + 1) + c[:, 1]) * (n + 1) + c[:, 2]  # noqa: E731
    tets = []
    for perm in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        c, vs = cells.copy(), [node(cells)]
        for ax in perm:
            c[:, ax] += 1
            vs.append(node(c))
        tets.append(np.stack(vs, 1))
    t = np.concatenate(tets)
    e = co[t]
    neg = np.linalg.det(e[:, 1:] - e[:, :1]) < 0
    t[neg, 1], t[neg, 2] = t[neg, 2].copy(), t[neg, 1].copy()
    return co, t


_AXES = (0.15, 0.10, 0.08)  # the defect's semi-axes as fractions of the edge


def _tet_b(gid, n_dof, seed, nrhs):
    b = torch.randn((n_dof, nrhs) if nrhs > 1 else (n_dof,), generator=_rng(seed), device=DEV, dtype=F64)
    return b


def _tet_exact(case, seed):
    n = case["n"]
    co, t = _tet_mesh(n, seed)
    w = np.where(np.abs(co - n) < 1e-12, 0.0, co)
    _, first, inv = np.unique(np.round(w, 12), axis=0, return_index=True, return_inverse=True)
    rank = np.empty(len(first), dtype=np.int64)
    rank[np.argsort(first, kind="stable")] = np.arange(len(first))
    gid = rank[inv.ravel()]
    nd = len(first)
    e = co[t]
    J = e[:, 1:] - e[:, :1]                      # rows: edge vectors
    vol = np.linalg.det(J) / 6
    ref = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    gr = np.einsum("eij,aj->eai", np.linalg.inv(J), ref)
    K = np.einsum("eai,ebi,e->eab", gr, gr, vol)
    Nt = np.full((4, 4), 0.1381966)
    np.fill_diagonal(Nt, 0.5854102)
    A = K if case["op"] == "A_demag" else K * _Mat.alpha + (Nt.T @ Nt)[None] * (vol / 4)[:, None, None]
    d = gid[t]
    pinned = np.zeros(nd, bool)
    if case["op"] == "A_demag":
        pinned[0] = True
    else:
        q = (e.mean(1) - n / 2) / (np.array(_AXES) * n)
        pinned[np.unique(d[(q * q).sum(1) <= 1.0])] = True
    rows = torch.as_tensor(np.repeat(d, 4, 1).ravel(), device=DEV)
    cols = torch.as_tensor(np.tile(d, (1, 4)).ravel(), device=DEV)
    S = torch.sparse_coo_tensor(torch.stack([rows, cols]), torch.as_tensor(A.ravel(), device=DEV), (nd, nd)).coalesce()
    S = S.to_sparse_csr()
    b = _tet_b(gid, nd, seed, case["nrhs"])
    f = torch.as_tensor(~pinned, device=DEV).to(F64)
    f = f if b.dim() == 1 else f[:, None]
    if case["op"] == "A_demag":
        b[0] = 0.0
    pin = b * (1 - f)
    mul = lambda v: S @ v if v.dim() > 1 else (S @ v[:, None])[:, 0]  # noqa: E731
    return _cg64(lambda p: f * mul(p), f * b) + pin


# --------------------------------------------------------------------------------------- preparation
def _flags(op, mark):
    """Row and column flags of a stencil operator: the anchor node 0, or the defect DOFs, pinned."""
    from cupymag_gb300.utils.stencil_operator import COL_EXCLUDED, ROW_IDENTITY
    f = np.zeros(mark.numel(), dtype=np.uint8)
    if op in ("A_demag", "A_el"):
        f[0] = ROW_IDENTITY | COL_EXCLUDED
    else:
        f[mark.reshape(-1).cpu().numpy()] = ROW_IDENTITY | COL_EXCLUDED
    return f if f.any() else None


def _operator(op, dims, mark, st):
    from cupymag_gb300.utils.stencil_operator import StencilOperator
    coef = {"A_demag": lambda: st["K"], "A_el": lambda: st["Kel"]}.get(op, lambda: _gs_coef(st, op))()
    return StencilOperator(*dims, np.asarray(coef).reshape(-1), _flags(op, mark), torch.device(DEV, 0))


def _gs_inputs(dims, mark, st, seed, nrhs):
    """t = m + f dt of a step (m and a small smooth field) and b = F1 t; columns (n, nrhs) or (n,)."""
    m = _m0(dims, mark, seed)
    g = _rng(seed + 1)
    f = torch.randn(3, generator=g, device=DEV, dtype=F64) * 0.05 + 0.02 * m.roll(1, 0)
    t = (m + _Mat.dt * f) if nrhs == 3 else (m[:, 0] + _Mat.dt * f[:, 0])
    free = (~mark).reshape(-1).to(F64)
    cols = [free * _apply(st["M"], c.reshape(dims)).reshape(-1) for c in (t.unbind(1) if nrhs == 3 else [t])]
    b = torch.stack(cols, 1).contiguous() if nrhs == 3 else cols[0]
    x0 = (t * (free[:, None] if nrhs == 3 else free)).contiguous()
    return b, x0


def _field_b(op, dims, mark, st, seed):
    m = _m0(dims, mark, seed)
    return _fel(st, _E0(m), dims) if op == "A_el" else _div(st, m - m.mean(0), dims)


def _batch_grids(case):
    r = np.random.default_rng(case["pick"])
    e = np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))
    e[-1] = case["hi"]
    return [((int(round(v)),) * 3, int(r.integers(0, int(round(v)) // 4 + 1))) for v in e]


def _product_inputs(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    mark = _defect(dims, case["defect"])
    m, g = _m0(dims, mark, seed), _rng(seed + 2)
    n = m.shape[0]
    u = torch.randn(3 * n, generator=g, device=DEV, dtype=F64) * 1e-4
    return dims, m, _E0(m).reshape(-1).contiguous(), u, torch.randn(n, generator=g, device=DEV, dtype=F64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tet":
        return _prepare_tet(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    dims = (case["nx"], case["ny"], case["nz"])
    if kind == "step":
        from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
        from cupymag_gb300.physics.llg import LLGSolver
        from cupymag_gb300.workloads import hex_params
        d = case["defect"]
        p = hex_params(dims[0], d, case["ME"], case["ME"]).with_(Nx=dims[0], Ny=dims[1], Nz=dims[2])
        S = SimulationOperators(p)
        L = LLGSolver(S, p, precision=case["precision"], operators=case["operators"])
        return {"kind": kind, "solver": L, "m0": _m0(dims, _defect(dims, d), seed), "ME": case["ME"], "H": _Mat.H}
    st = _stencils()
    if kind == "products":
        from cupymag_gb300.utils.stencil_derivatives import StencilCoupling, StencilDerivatives
        _, m, E0, u, U = _product_inputs(case, seed)
        n = m.shape[0]
        return {"kind": kind, "m": m, "avg": m.mean(0), "E0": E0, "u": u, "U": U,
                "D": StencilDerivatives(*dims, *st["F"], DEV),
                "F": StencilCoupling(*dims, st["Fel"].reshape(-1), True, DEV),
                "R9": torch.as_tensor(_rot()[0].reshape(-1), device=DEV, dtype=F64),
                "out": [torch.empty(sh, dtype=F64, device=DEV) for sh in ((3 * n,), (n, 6), (n,), (n, 3))]}
    from cupymag_gb300.physics.llg import INNER_TOL
    from cupymag_gb300.solvers.linear_solvers import CGSolver, new_info
    mark = _defect(dims, case["defect"])
    s = {"kind": kind, "api": case.get("api", "solver"), "A": _operator(case["op"], dims, mark, st),
         "warm": case["warm"], "solver": CGSolver(), "info": new_info(1)}
    if kind == "gs":
        s["b"], s["x0"] = _gs_inputs(dims, mark, st, seed, case["nrhs"])
        s["inner"], s["precond"] = INNER_TOL[2 if case["op"] == "A1" else 5], None
    else:
        s["b"] = _field_b(case["op"], dims, mark, st, seed)
        s["x0"] = 0.9 * _circ64(st["Kel"] if case["op"] == "A_el" else st["K"][None, None], s["b"], dims) \
            if case["warm"] else torch.zeros_like(s["b"])
        s["inner"], s["precond"] = None, "fft"
        s["A"].fft_plan()
    s["x"] = torch.zeros_like(s["b"])
    return s


def _prepare_batch(case, seed):
    from cupymag_gb300.physics.llg import INNER_TOL
    from cupymag_gb300.serving.blockdiag import BlockDiagPlan, BlockSystem, work_bytes
    from cupymag_gb300.solvers.linear_solvers import new_info
    st, systems = _stencils(), []
    for i, (dims, nd) in enumerate(_batch_grids(case)):
        mark = _defect(dims, nd)
        b, _ = _gs_inputs(dims, mark, st, seed * 31 + i, case["nrhs"])
        work = torch.empty(work_bytes(dims, 1, case["nrhs"], "IR"), dtype=torch.uint8, device=DEV)
        systems.append(BlockSystem(_operator(case["op"], dims, mark, st), b, torch.zeros_like(b), new_info(1)[0], work,
                                   TOL, MAXITER))
    plan = BlockDiagPlan(systems, "IR", inner_tol=INNER_TOL[2 if case["op"] == "A1" else 5])
    return {"kind": "batch", "plan": plan, "systems": systems}


def _prepare_tet(case, seed):
    from cupymag_gb300.core.assemble_simulation_operators import SimulationOperators
    from cupymag_gb300.mesh.grids import TetraGrid
    from cupymag_gb300.solvers.linear_solvers import CGSolver, new_info
    from cupymag_gb300.utils.defect_shapes import get_defect_shape_function
    from cupymag_gb300.workloads import MAGNETIC, SimParams
    n = case["n"]
    co, t = _tet_mesh(n, seed)
    axes = tuple(a * n for a in _AXES)
    p = SimParams(**MAGNETIC)
    p.grid_type, p.defect_shape, p.defect_parameters = "Tet", "Ellipsoid", axes
    S = SimulationOperators(p.finalize(), mesh=TetraGrid(
        coords=co, tets=t, defect_shape=get_defect_shape_function("RotatedEllipsoid", (axes, np.eye(3)))))
    A = S.csr_demag_and_deriv()[0] if case["op"] == "A_demag" else S.csr_GS()[0]
    b = _tet_b(None, S.n_dof, seed, case["nrhs"])
    if case["op"] == "A_demag":
        b[0] = 0.0
    if case["precision"] == "IR":
        A.ensure_fp32()
    return {"kind": "tet", "api": "solver", "A": A, "b": b, "x": torch.zeros_like(b), "warm": False, "x0": None,
            "solver": CGSolver(), "info": new_info(1), "inner": 1e-3, "precond": None,
            "precision": case["precision"]}


# ------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "step":
        L = s["solver"]
        L.set_magnetization(s["m0"])
        L.step(s["H"])
        out = {"m": L.m, "avg": L.avg_m, "Ht": L.Ht}
        if s["ME"]:
            out["E"] = L.E
        return out
    if kind == "products":
        b_el, E, b, H = s["out"]
        s["F"].spmv(s["E0"], out=b_el)
        s["D"].strain_into(s["u"], E, s["R9"])
        s["D"].demag_rhs_into(s["m"], s["avg"], b, pin=0)
        s["D"].hd_into(s["U"], H)
        return s["out"]
    if kind == "batch":
        s["plan"].launch()
        return [y.x for y in s["systems"]]
    if s["api"] == "solve_cg":
        from cupymag_gb300.solvers.linear_solvers import solve_cg
        return solve_cg(s["A"], s["b"], x0=s["x0"], tol=TOL, maxiter=MAXITER, use_init=s["warm"], precision="IR")
    if s["warm"]:
        s["x"].copy_(s["x0"])
    s["solver"].launch(s["A"], s["b"], s["x"], s["info"][0], tol=TOL, maxiter=MAXITER, use_init=s["warm"],
                       precision=s.get("precision", "IR"), inner_tol=s["inner"], precond=s["precond"])
    return s["x"]


# --------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "tet":
        n = case["n"] ** 3
        return {"bytes": n * (15 * 12 + 16 * case["nrhs"]), "flops": n * 15 * 2 * case["nrhs"]}
    if kind == "batch":
        n = sum(d[0] * d[1] * d[2] for d, _ in _batch_grids(case))
        return {"bytes": n * (16 * case["nrhs"] + 1), "flops": n * 54 * case["nrhs"]}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "step":
        # m in and out, weights; Ht (and E) out; one product of each operator the step applies
        return {"bytes": n * (24 + 24 + 24 + 8 + 1 + (48 if case["ME"] else 0)),
                "flops": n * 54 * (20 + (9 + 18 + 9 if case["ME"] else 0))}
    if kind == "gs":
        return {"bytes": n * case["nrhs"] * (24 if case["warm"] else 16) + n, "flops": n * 54 * case["nrhs"]}
    if kind == "field":
        nc = 3 if case["op"] == "A_el" else 1
        return {"bytes": n * nc * (24 if case["warm"] else 16), "flops": n * 54 * nc * nc}
    return {"bytes": n * 8 * (9 + 9 + 4 + 4), "flops": n * 54 * (18 + 9 + 6)}


# ------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "tet":
        return _tet_exact(case, seed)
    if kind == "step":
        return _step64(case, seed)
    st = _stencils()
    if kind == "batch":
        out = []
        for i, (dims, nd) in enumerate(_batch_grids(case)):
            mark = _defect(dims, nd)
            b, _ = _gs_inputs(dims, mark, st, seed * 31 + i, case["nrhs"])
            out.append(_gs64(_gs_coef(st, case["op"]), b, dims, mark))
        return out
    if kind == "products":
        dims, m, E0, u, U = _product_inputs(case, seed)
        return [_fel(st, E0.reshape(-1, 6), dims), _strain(st, u, dims), _div(st, m - m.mean(0), dims),
                _grad(st, U, dims)]
    dims = (case["nx"], case["ny"], case["nz"])
    mark = _defect(dims, case["defect"])
    if kind == "gs":
        b, _ = _gs_inputs(dims, mark, st, seed, case["nrhs"])
        return _gs64(_gs_coef(st, case["op"]), b, dims, mark)
    b = _field_b(case["op"], dims, mark, st, seed)
    return _circ64(st["Kel"] if case["op"] == "A_el" else st["K"][None, None], b, dims)
