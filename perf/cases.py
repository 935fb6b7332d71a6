"""Timed cases of the hot path: semi-Lagrangian advection, the operator apply,
the Helmholtz/Poisson solves and the step that joins them.

Every case goes through the public classes of ``se_b200`` as a time loop does.
A case's ``kind`` names the path:

  sl     ``Advector.Advect`` (first or second order, 1 or 2 components)
  apply  ``HelmholtzEqn.apply`` / ``apply_low`` on device vectors, what a
         caller with its own Krylov loop runs
  helm   ``HelmholtzEqn.Solve`` / ``PoissonEqn.Solve``: Jacobi CG (the
         drop-in) or fast diagonalization
  step   advection, then the asynchronous Helmholtz solve of the result
  batch  ``solve_batch`` over an uneven ensemble

Meshes are the repository's configurations (16x16 p=6, 64x64 p=8, the 128x64
p=6 channel, 768x768 p=8 for the apply, the ensemble's 8..64 elements at p = 4,
6, 8) and others of the same ranges: orders 3 to 12, odd element counts, walls
in y or on all sides. ``exact`` gives the 64-bit result from dense 1-D
matrices and product-form Lagrange interpolation, without the library.
"""
import math

import numpy as np
import torch

import se_b200 as S

WALLS = ("none", "y", "all")  # doubly periodic, channel, box
RTOL = 1e-10


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # one advection of a small test mesh: launch latency
        {"name": "sl1_16x16_p6", "kind": "sl", "ex": 16, "ey": 16, "p": 6, "walls": "none",
         "order": 1, "dofs": 1, "courant": 2.0},
        # the advection of the 200-step tracer run
        {"name": "sl1_64x64_p8", "kind": "sl", "ex": 64, "ey": 64, "p": 8, "walls": "none",
         "order": 1, "dofs": 1, "courant": 2.0},
        # a Navier-Stokes velocity advecting itself between walls, odd order
        {"name": "sl1_vec_117x83_p7_walls", "kind": "sl", "ex": 117, "ey": 83, "p": 7,
         "walls": "all", "order": 1, "dofs": 2, "courant": 1.0},
        # the second-order PV advection of the two-layer channel
        {"name": "sl2_128x64_p6_channel", "kind": "sl", "ex": 128, "ey": 64, "p": 6,
         "walls": "y", "order": 2, "dofs": 1, "courant": 1.5},
        # FP64 operator apply larger than L2
        {"name": "apply_768x768_p8", "kind": "apply", "ex": 768, "ey": 768, "p": 8,
         "walls": "none", "type": "fp64"},
        # a ragged high-order channel, as a p-refinement study runs it
        {"name": "apply_151x203_p10_channel", "kind": "apply", "ex": 151, "ey": 203, "p": 10,
         "walls": "y", "type": "fp64"},
        # the reduced-precision apply
        {"name": "apply_768x768_p8_bf16", "kind": "apply", "ex": 768, "ey": 768, "p": 8,
         "walls": "none", "type": "bf16"},
        # the plain Helmholtz configuration, Jacobi CG
        {"name": "cg_16x16_p6", "kind": "helm", "ex": 16, "ey": 16, "p": 6, "walls": "none",
         "lam": 1.0, "method": "cg", "mode": "exact", "precision": "fp64"},
        # the drop-in solve of the benchmark step
        {"name": "cg_64x64_p8", "kind": "helm", "ex": 64, "ey": 64, "p": 8, "walls": "none",
         "lam": 1.0, "method": "cg", "mode": "exact", "precision": "fp64"},
        # the PV inversion of the channel by fast diagonalization
        {"name": "fdm_128x64_p6_channel", "kind": "helm", "ex": 128, "ey": 64, "p": 6,
         "walls": "y", "lam": 40.0, "method": "fdm", "mode": "exact", "precision": "fp64"},
        # the benchmark step: advection and fast-diagonalization solve
        {"name": "step_64x64_p8", "kind": "step", "ex": 64, "ey": 64, "p": 8, "walls": "none",
         "lam": 1.0, "courant": 2.0},
        # an uneven ensemble solved by CG in one call
        {"name": "batch_24_cg", "kind": "batch", "count": 24, "lo": 8, "hi": 40, "spec": 2024,
         "method": "cg"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _mesh_draw(rng, p, lo, hi):
    """Element counts of about lo..hi unknowns (log-uniform), aspect 1/2 to 2."""
    unknowns = _log(rng, lo, hi)
    ne = max(4.0, unknowns / (p * p))
    aspect = _log(rng, 0.5, 2.0)
    return (max(2, round(math.sqrt(ne * aspect))), max(2, round(math.sqrt(ne / aspect))))


def draw(rng):
    kind = rng.choices(["sl", "apply", "cg", "fdm", "step", "batch"], [8, 5, 4, 4, 2, 1])[0]
    walls = rng.choices(WALLS, [3, 2, 1])[0]
    if kind == "sl":
        p = rng.randint(3, 10)
        ex, ey = _mesh_draw(rng, p, 5e3, 6e5)
        return {"kind": "sl", "ex": ex, "ey": ey, "p": p, "walls": walls,
                "order": rng.randint(1, 2), "dofs": rng.choice([1, 1, 2]),
                "courant": round(_log(rng, 0.4, 4.0), 3)}
    if kind == "apply":
        t = rng.choices(["fp64", "bf16", "fp16"], [4, 1, 1])[0]
        p = rng.randint(3, 12) if t == "fp64" else rng.randint(4, 8)
        ex, ey = _mesh_draw(rng, p, 2e4, 3e7)
        return {"kind": "apply", "ex": ex, "ey": ey, "p": p, "walls": walls, "type": t}
    if kind == "step":
        p = rng.randint(4, 8)
        ex, ey = _mesh_draw(rng, p, 1e4, 4e5)
        if rng.random() < 0.5:  # element counts of the serving stream
            ex = ey = rng.choice([8, 16, 32, 64])
        return {"kind": "step", "ex": ex, "ey": ey, "p": p, "walls": "none",
                "lam": round(_log(rng, 1.0, 100.0), 3), "courant": round(_log(rng, 0.4, 4.0), 3)}
    if kind == "batch":
        method = rng.choice(["cg", "fdm"])
        return {"kind": "batch", "count": rng.randint(8, 24), "lo": 8,
                "hi": rng.randint(20, 36 if method == "cg" else 64),
                "spec": rng.randint(1, 10 ** 6), "method": method}
    if kind == "cg":
        p = rng.randint(3, 8)
        ex, ey = _mesh_draw(rng, p, 2e3, 2e5)
        precision = "fp64"
    else:
        p = rng.randint(4, 8)
        ex, ey = _mesh_draw(rng, p, 1e4, 5e5)
        precision = rng.choice(["fp64", "fp64", "fp64", "mixed"])
    mode = rng.choice(["exact", "reference"]) if walls != "none" else "exact"
    return {"kind": "helm", "ex": ex, "ey": ey, "p": p, "walls": walls,
            "lam": round(_log(rng, 1.0, 100.0), 3), "method": kind, "mode": mode,
            "precision": precision}


# ----------------------------------------------------- the mesh, in numpy ----
def _gll(p):
    """GLL nodes and weights and the derivative matrix D[i][j] = l_j'(x_i)."""
    leg = np.polynomial.legendre.Legendre.basis(p)
    d1, d2 = leg.deriv(), leg.deriv(2)
    x = np.sort(d1.roots().real)
    for _ in range(3):
        x = x - d1(x) / d2(x)
    x = np.concatenate([[-1.0], x, [1.0]])
    x = 0.5 * (x - x[::-1])
    w = 2.0 / (p * (p + 1) * leg(x) ** 2)
    lam = np.array([1.0 / np.prod(x[j] - np.delete(x, j)) for j in range(p + 1)])
    D = np.zeros((p + 1, p + 1))
    for i in range(p + 1):
        for j in range(p + 1):
            if i != j:
                D[i, j] = lam[j] / lam[i] / (x[i] - x[j])
        D[i, i] = -D[i].sum()
    return x, w, lam, D


def _extent(case):
    """The domain: unit elements' aspect kept near 1, height 1."""
    return case["ex"] / case["ey"] if case["walls"] == "y" else 1.0, 1.0


def _periodic(case):
    return {"none": (True, True), "y": (True, False), "all": (False, False)}[case["walls"]]


def _axis(ne, p, length):
    x = _gll(p)[0]
    d = length / ne
    t = np.arange(ne * p + 1)
    e = t // p
    return e * d + (x[t - e * p] + 1.0) / 2.0 * d


def _grid(case):
    """Vertex coordinates normalised to [0, 1], shaped [nVerts y][nVerts x]."""
    lx, ly = _extent(case)
    x = _axis(case["ex"], case["p"], lx) / lx
    y = _axis(case["ey"], case["p"], ly) / ly
    return np.meshgrid(x, y)


def _velocity(case, seed, shift=0.0):
    """Taylor-Green vortex with seeded shear on the periodic directions; no
    flow through walls. [nVertsTotal][2]"""
    rng = np.random.default_rng(seed)
    X, Y = _grid(case)
    a = 1.0 + 0.1 * rng.standard_normal() - 0.02 * shift
    px, py = _periodic(case)
    b = 0.2 * rng.standard_normal(2)
    ph = rng.uniform(0, 2 * np.pi, 2)
    lx, ly = _extent(case)
    u = -a * np.sin(np.pi * X) ** 2 * np.sin(2 * np.pi * Y)
    v = a * np.sin(np.pi * Y) ** 2 * np.sin(2 * np.pi * X)
    if px:
        u = u + b[0] * np.cos(2 * np.pi * Y + ph[0])
    if py:
        v = v + b[1] * np.cos(2 * np.pi * X + ph[1])
    return np.stack([u.ravel(), v.ravel()], 1)


def _tracer(case, seed):
    """Four seeded Gaussian blobs of width 0.05."""
    rng = np.random.default_rng(seed + 7)
    X, Y = _grid(case)
    phi = np.zeros_like(X)
    for cx, cy in rng.uniform(0.1, 0.9, size=(4, 2)):
        phi += np.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / 0.05 ** 2)
    return phi.ravel()


def _rhs(case, seed):
    """Eight seeded Fourier modes with wavenumbers 1..6; between walls also
    the seeded 1e-3 perturbation of the channel's PV."""
    rng = np.random.default_rng(seed + 13)
    X, Y = _grid(case)
    f = np.zeros_like(X)
    for _ in range(8):
        kx, ky = rng.integers(1, 7, size=2)
        a, b = rng.standard_normal(2)
        arg = 2 * np.pi * (kx * X + ky * Y)
        f += a * np.cos(arg) + b * np.sin(arg)
    if case["walls"] != "none":
        f += 1e-3 * rng.standard_normal(f.shape)
        if case["walls"] == "y":
            f[:, -1] = f[:, 0]
    return f.ravel()


def _wall_values(case, seed):
    """The solution field before the solve: its Dirichlet values on walls."""
    if case["walls"] == "none":
        return np.zeros((case["ex"] * case["p"] + 1) * (case["ey"] * case["p"] + 1))
    rng = np.random.default_rng(seed + 17)
    X, Y = _grid(case)
    a = rng.standard_normal(3)
    return (a[0] + a[1] * Y + 0.3 * a[2] * np.cos(2 * np.pi * X)).ravel()


def _dt(case, vel):
    lx, ly = _extent(case)
    d = min(lx / case["ex"], ly / case["ey"])
    return float(case["courant"] * d / np.sqrt((vel ** 2).sum(1).max()))


# --------------------------------------------------------------- the state ----
class _DeviceArray:
    """A field's device memory for torch; keeps the field (and with it the
    memory) alive for as long as a tensor made from it."""

    def __init__(self, field, shape):
        self.field = field
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "version": 3,
                                         "data": (field.device_ptr(), False), "strides": None}


def _view(field):
    """A torch view of a field's values on the GPU."""
    n = field.mesh.nVertsTotal
    shape = (n,) if field.nDofs == 1 else (n, field.nDofs)
    return torch.as_tensor(_DeviceArray(field, shape), device="cuda")


def _mesh(case):
    lx, ly = _extent(case)
    px, py = _periodic(case)
    return S.Mesh("mesh", [case["ex"], case["ey"]], "legendre", case["p"], [0.0, 0.0], [lx, ly],
                  [px, py])


def _bcs(case, mesh):
    wy, wx = case["walls"] != "none", case["walls"] == "all"
    return S.BCs(wy, wy, wx, wx, mesh)


def _field(mesh, dofs, bcs, vals, name="f"):
    f = S.Field(name, mesh, dofs, bcs)
    f.vals = vals
    return f


def _opts(case):
    prec = {"fp64": S.PREC_FP64, "mixed": S.PREC_MIXED}[case.get("precision", "fp64")]
    return S.solver_opts(rtol=RTOL, max_it=20000, precision=prec,
                         mode=S.MODE_REFERENCE if case.get("mode") == "reference" else S.MODE_EXACT,
                         method=S.METHOD_FDM if case["method"] == "fdm" else S.METHOD_CG)


def _members(case):
    """The ensemble's systems: mesh size, order and lambda of each."""
    rng = np.random.default_rng(case["spec"])
    out = []
    for _ in range(case["count"]):
        ne = int(rng.integers(case["lo"], case["hi"] + 1))
        out.append({"kind": "helm", "ex": ne, "ey": ne, "p": int(rng.choice([4, 6, 8])),
                    "walls": "none", "lam": float(10 ** rng.uniform(0, 2)),
                    "method": case["method"], "mode": "exact", "precision": "fp64"})
    return out


def _helm(case, seed):
    m = _mesh(case)
    bc = _bcs(case, m)
    u = _field(m, 1, bc, _wall_values(case, seed), "u")
    rhs = _field(m, 1, bc, _rhs(case, seed), "rhs")
    ls = S.HelmholtzEqn(u, rhs, -case["lam"], -1.0, 1.0, 0, _opts(case))
    ls.Assemble()
    return {"system": ls, "u": u, "out": _view(u)}


def _apply_input(case, seed, n):
    """A search direction: white noise, as late Krylov directions are."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(n, dtype=torch.float64 if case["type"] == "fp64" else torch.float32,
                    device="cuda", generator=g)
    return x if case["type"] == "fp64" else x.to(
        torch.bfloat16 if case["type"] == "bf16" else torch.float16)


def prepare(case, seed):
    torch.cuda.init()
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("sl", "step"):
        m = _mesh(case)
        bc = _bcs(case, m)
        vel = _velocity(case, seed)
        st["dt"] = _dt(case, vel)
        st["vel"] = _field(m, 2, None, vel, "vel")
        second = case.get("order", 1) == 2
        if case.get("dofs", 1) == 2:
            st["phi"] = st["vel"]
        else:
            st["phi"] = _field(m, 1, bc, _tracer(case, seed), "phi")
        if second:
            velm = _velocity(case, seed, 1.0)
            st["velm"] = _field(m, 2, None, velm, "velm")
            st["phim"] = (st["velm"] if case["dofs"] == 2 else
                          _field(m, 1, bc, 0.97 * _tracer(case, seed), "phim"))
            st["adv"] = S.Advector(st["phi"], st["vel"], st["phim"], st["velm"])
        else:
            st["adv"] = S.Advector(st["phi"], st["vel"])
        st["out"] = _view(st["adv"].fieldSL)
        if kind == "step":
            st["u"] = S.Field("u", m, 1, bc)
            st["system"] = S.HelmholtzEqn(st["u"], st["adv"].fieldSL, -case["lam"], -1.0, 1.0, 0,
                                          _opts({"method": "fdm"}))
            st["system"].Assemble()
            st["uout"] = _view(st["u"])
    elif kind == "apply":
        m = _mesh(case)
        u = S.Field("u", m, 1, _bcs(case, m))
        ls = S.HelmholtzEqn(u, None, -1.0, -1.0, 1.0, 0,
                            S.solver_opts(rtol=RTOL, mode=S.MODE_EXACT))
        x = _apply_input(case, seed, ls.vecSize)
        st.update(u=u, system=ls, x=x, xp=x.data_ptr())
        st["y"] = torch.empty(ls.vecSize, device="cuda",
                              dtype=torch.float64 if case["type"] == "fp64" else torch.float32)
        st["yp"] = st["y"].data_ptr()
    elif kind == "helm":
        st.update(_helm(case, seed))
    else:
        st["members"] = [_helm(c, seed + 101 * k) for k, c in enumerate(_members(case))]
        st["systems"] = [h["system"] for h in st["members"]]
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind == "sl":
        st["adv"].Advect(st["dt"])
        return st["out"]
    if kind == "apply":
        t = st["case"]["type"]
        if t == "fp64":
            st["system"].apply(st["xp"], st["yp"])
        else:
            st["system"].apply_low(st["xp"], st["yp"], S.PREC_BF16 if t == "bf16" else S.PREC_FP16)
        return st["y"]
    if kind == "helm":
        st["system"].Solve("helm_")
        return st["out"]
    if kind == "step":
        st["adv"].Advect(st["dt"])
        st["system"].solve_async()
        st["system"].solve_finish()
        return [st["out"], st["uout"]]
    S.solve_batch(st["systems"])
    return [h["out"] for h in st["members"]]


# ------------------------------------------------------------------- work ----
def _iterations(case):
    """Jacobi-CG iterations to RTOL: the square root of the condition number."""
    return max(case["ex"], case["ey"]) * case["p"] ** 1.5


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [work(c) for c in _members(case)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    p, n = case["p"], case["ex"] * case["ey"] * case["p"] ** 2
    gather = (p + 1) ** 2 + (p + 1)  # multiply-adds of one interpolated component
    if kind == "sl":
        d, o = case["dofs"], case["order"]
        # velocity and field in (both levels at second order), field out
        fields = 2 * o + (d * o if d == 1 else 0) + d
        return {"bytes": 8.0 * n * fields, "flops": 2.0 * n * gather * (2 * (3 if o == 2 else 1) + d * o)}
    if kind == "apply":
        return {"bytes": n * (16.0 if case["type"] == "fp64" else 6.0), "flops": n * (4.0 * (p + 2) + 6)}
    if kind == "step":
        return {"bytes": 8.0 * n * 5, "flops": 2.0 * n * gather * 3 + n * 4.0 * (p + 2)}
    flops = n * (4.0 * (p + 2) + 6)
    if case["method"] == "cg":
        flops = _iterations(case) * n * (4.0 * (p + 2) + 20)
    return {"bytes": 16.0 * n, "flops": flops}


# ------------------------------------------------------------------ exact ----
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _assembled(ne, p, periodic, dirichlet):
    """1-D assembled stiffness and weights, and the unknown vertices' range."""
    _, w, _, D = _gll(p)
    Kh = D.T @ np.diag(w) @ D
    nv = ne * p + 1
    K, W = np.zeros((nv, nv)), np.zeros(nv)
    for e in range(ne):
        K[e * p:e * p + p + 1, e * p:e * p + p + 1] += Kh
        W[e * p:e * p + p + 1] += w
    if periodic:
        K[0] += K[-1]
        K[:, 0] += K[:, -1]
        W[0] += W[-1]
        return K, W, 0, nv - 1
    return K, W, int(dirichlet), nv - int(dirichlet)


def _operator(case, c, mode):
    lx, ly = _extent(case)
    hx, hy = lx / case["ex"], ly / case["ey"]
    alpha = c * hx * hy / 4
    if mode == "reference":
        bx, by = -4.0 / hx ** 2, -4.0 / hy ** 2
    else:
        bx, by = -hy / hx, -hx / hy
    px, py = _periodic(case)
    dx, dy = (_assembled(case["ex"], case["p"], px, not px),
              _assembled(case["ey"], case["p"], py, not py))
    return alpha, bx, by, dx, dy, hx * hy / 4


def _solve_exact(case, u0, rhs):
    """The discrete solution through the 1-D generalised eigenproblems; the
    field with its Dirichlet values and periodic copies, [nVertsTotal]."""
    alpha, bx, by, (Kx, Wx, x0, x1), (Ky, Wy, y0, y1), detj = _operator(
        case, -case["lam"], case["mode"])
    nvx, nvy = case["ex"] * case["p"] + 1, case["ey"] * case["p"] + 1
    U = u0.reshape(nvy, nvx).copy()
    px, py = _periodic(case)
    mx = np.zeros(nvx, bool)
    my = np.zeros(nvy, bool)
    mx[x0:x1] = True
    my[y0:y1] = True
    # Dirichlet data alone (nothing on unknowns or periodic duplicates)
    UD = U.copy()
    UD[np.ix_(my, mx)] = 0.0
    if px:
        UD[:, -1] = 0.0
    if py:
        UD[-1, :] = 0.0
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=_dev())  # noqa: E731
    tKx, tKy, tWx, tWy, tUD = t(Kx), t(Ky), t(Wx), t(Wy), t(UD)
    AU = (alpha * tWy[:, None] * tWx * tUD + bx * tWy[:, None] * (tUD @ tKx.T)
          + by * tWx * (tKy @ tUD))
    F = detj * tWy[:, None] * tWx * t(rhs.reshape(nvy, nvx)) - AU
    F = F[y0:y1, x0:x1]

    def eig(K, W, a, b):
        s = 1.0 / np.sqrt(W[a:b])
        lam, V = np.linalg.eigh(s[:, None] * K[a:b, a:b] * s)
        return t(lam), t(s[:, None] * V)

    lx, Vx = eig(Kx, Wx, x0, x1)
    ly, Vy = eig(Ky, Wy, y0, y1)
    Z = (Vy.T @ F @ Vx) / (alpha + bx * lx + by * ly[:, None])
    sol = Vy @ Z @ Vx.T
    out = t(U)
    out[y0:y1, x0:x1] = sol
    if px:
        out[:, -1] = out[:, 0]
    if py:
        out[-1, :] = out[0, :]
    return out.reshape(-1)


def _apply_exact(case, x):
    """y = A x from the element matrix, row by row of the tensor product."""
    alpha, bx, by, _, _, _ = _operator(case, -1.0, "exact")
    px, py = _periodic(case)
    _, w, _, D = _gll(case["p"])
    Kh = torch.as_tensor(D.T @ np.diag(w) @ D, device=x.device)
    wt = torch.as_tensor(w, device=x.device)
    p = case["p"]

    def lo(per):
        return 0 if per else 1

    nvx, nvy = case["ex"] * p + 1, case["ey"] * p + 1
    gx, gy = nvx - (1 if px else 2), nvy - (1 if py else 2)
    full = torch.zeros(nvy, nvx, dtype=torch.float64, device=x.device)
    full[lo(py):lo(py) + gy, lo(px):lo(px) + gx] = x.double().reshape(gy, gx)
    if px:
        full[:, -1] = full[:, 0]
    if py:
        full[-1, :] = full[0, :]

    def weights(ne, per):
        W = torch.zeros(ne * p + 1, dtype=torch.float64, device=x.device)
        idx = (torch.arange(ne, device=x.device)[:, None] * p
               + torch.arange(p + 1, device=x.device)).reshape(-1)
        W.index_add_(0, idx, wt.repeat(ne))
        if per:
            W[0] = W[-1] = W[0] + W[-1]
        return W

    def stiff(v, ne, per):
        """K v along the last dimension."""
        out = torch.zeros_like(v)
        E = v.unfold(-1, p + 1, p) @ Kh.T
        out[..., :-1] += E[..., :-1].reshape(*v.shape[:-1], ne * p)
        out[..., p::p] += E[..., -1]
        if per:
            s = out[..., 0] + out[..., -1]
            out[..., 0] = s
            out[..., -1] = s
        return out

    wx, wy = weights(case["ex"], px), weights(case["ey"], py)
    y = alpha * wy[:, None] * wx * full
    y += bx * wy[:, None] * stiff(full, case["ex"], px)
    y += by * wx * stiff(full.T.contiguous(), case["ey"], py).T
    return y[lo(py):lo(py) + gy, lo(px):lo(px) + gx].reshape(-1).clone()


class _Interp:
    """Field values at points, by product-form Lagrange polynomials."""

    def __init__(self, case):
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=_dev())  # noqa: E731
        self.case, self.L = case, _extent(case)
        x, _, lam, _ = _gll(case["p"])
        self.x, self.lam = t(x), t(lam)

    def weights(self, c, d):
        ne = self.case["ex" if d == 0 else "ey"]
        h = self.L[d] / ne
        e = torch.clamp(torch.floor(c / h), 0, ne - 1)
        loc = torch.clamp((c - e * h) * (2.0 / h) - 1.0, -1.0, 1.0)
        diff = loc[:, None] - self.x
        out = torch.empty_like(diff)
        for j in range(diff.shape[1]):
            keep = [k for k in range(diff.shape[1]) if k != j]
            out[:, j] = self.lam[j] * diff[:, keep].prod(1)
        return e.long(), out

    def __call__(self, vals, X, Y):
        p = self.case["p"]
        nvx = self.case["ex"] * p + 1
        out = torch.empty(len(X), vals.shape[1], dtype=torch.float64, device=X.device)
        a = torch.arange(p + 1, device=X.device)
        for b in range(0, len(X), 1 << 17):
            s = slice(b, b + (1 << 17))
            ex, cx = self.weights(X[s], 0)
            ey, cy = self.weights(Y[s], 1)
            idx = ((ey[:, None] * p + a) * nvx)[:, :, None] + (ex[:, None] * p + a)[:, None, :]
            out[s] = torch.einsum("qj,qi,qjid->qd", cy, cx, vals[idx])
        return out


def _advect_exact(case, seed, dt):
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=_dev())  # noqa: E731
    two = case.get("dofs", 1) == 2
    second = case.get("order", 1) == 2
    vel = t(_velocity(case, seed))
    phi = vel if two else t(_tracer(case, seed))[:, None]
    L, per = _extent(case), _periodic(case)
    X, Y = (t(g.ravel()) * s for g, s in zip(_grid(case), L))
    at = _Interp(case)

    def wrap(c, d):
        if per[d]:
            c = torch.where(c < 0, c + L[d], c)
            return torch.where(c > L[d], c - L[d], c)
        return torch.clamp(c, 0.0, L[d])

    def back(x, y, u, s):
        return wrap(x - s * u[:, 0], 0), wrap(y - s * u[:, 1], 1)

    if not second:
        u = at(vel, *back(X, Y, vel, 0.5 * dt))
        out = at(phi, *back(X, Y, u, dt))
    else:
        velm = t(_velocity(case, seed, 1.0))
        phim = velm if two else 0.97 * phi
        u = at(1.5 * vel - 0.5 * velm, *back(X, Y, 2.0 * vel - velm, 0.5 * dt))
        x1, y1 = back(X, Y, u, dt)
        u = at(0.5 * vel + 0.5 * velm, *back(x1, y1, at(vel, x1, y1), 0.5 * dt))
        out = 2.0 * at(phi, x1, y1) - 0.5 * at(phim, *back(x1, y1, u, dt))
    nvx, nvy = case["ex"] * case["p"] + 1, case["ey"] * case["p"] + 1
    out = out.reshape(nvy, nvx, -1)
    if per[0]:
        out[:, -1] = out[:, 0]
    if per[1]:
        out[-1, :] = out[0, :]
    return out.reshape(nvy * nvx) if not two else out.reshape(nvy * nvx, 2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sl":
        return _advect_exact(case, seed, _dt(case, _velocity(case, seed)))
    if kind == "apply":
        px, py = _periodic(case)
        n = ((case["ex"] * case["p"] + 1 - (1 if px else 2))
             * (case["ey"] * case["p"] + 1 - (1 if py else 2)))
        return _apply_exact(case, _apply_input(case, seed, n))
    if kind == "helm":
        return _solve_exact(case, _wall_values(case, seed), _rhs(case, seed))
    if kind == "step":
        a = _advect_exact(case, seed, _dt(case, _velocity(case, seed)))
        full = dict(case, mode="exact")
        return [a, _solve_exact(full, _wall_values(case, seed), a.cpu().numpy())]
    return [_solve_exact(c, _wall_values(c, seed + 101 * k), _rhs(c, seed + 101 * k))
            for k, c in enumerate(_members(case))]
