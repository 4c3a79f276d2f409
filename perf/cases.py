"""Timed workloads of the TURBINS time step on one GPU.

Each case is work that a program built on this package has it do, through the
entry points such a program calls:

* ``step``: whole TVD-RK2 steps (``Context.step``) from a state handed over in
  page-locked host arrays and read back into page-locked host arrays -- the
  lock exchange, the turbidity current over one bump and the two-fraction
  current over sixteen bumps of ``turbins_gb300.workload``;
* ``predict``: the momentum and concentration predictor driven routine by
  routine, as a host program that keeps its own loop calls it;
* ``poisson``: one pressure solve from a zero pressure and its projection;
* ``forward`` / ``gradient``: the pressure-guess network's forward pass, and
  a forward and backward pass that returns the parameter gradients.

Initial states are developed currents: a lock that has collapsed into a layer
with a wavy front, a discretely divergence-free velocity field of a few large
modes, a hydrostatic pressure gradient and a small last pressure increment.
"""
import functools

import numpy as np
import torch

from turbins_gb300 import api as A
from turbins_gb300 import net as N
from turbins_gb300 import workload as W

DT = {"lock": 1.0e-3, "bump": 5.0e-4, "multi": 2.5e-4}


def listed():
    return [
        # the smallest grid the quick checks run: a step is all launches and
        # waits for scalars
        dict(name="step_lock_32x16x16", kind="step", flow="lock", nx=32, ny=16, nz=16, steps=4, plain=False),
        # the lock-exchange configuration, solved throughout in FP64
        dict(name="step_lock_64x32x32_plain", kind="step", flow="lock", nx=64, ny=32, nz=32, steps=2, plain=True),
        # a parameter study's grid, not a power of two in any direction
        dict(name="step_bump_160x96x48", kind="step", flow="bump", nx=160, ny=96, nz=48, steps=2, plain=False),
        # the grid the training snapshots of the sixteen-bump flow come from
        dict(name="step_multi_128x64x64", kind="step", flow="multi", nx=128, ny=64, nz=64, steps=2, plain=False),
        # the single-bump configuration
        dict(name="step_bump_256x128x128", kind="step", flow="bump", nx=256, ny=128, nz=128, steps=2, plain=False),
        # the full two-fraction configuration
        dict(name="step_multi_512x256x256", kind="step", flow="multi", nx=512, ny=256, nz=256, steps=1, plain=False),
        # the predictor routine by routine: ENO-3 and implicit diffusion on a
        # ragged stretched box
        dict(name="predict_192x96x64", kind="predict", nx=192, ny=96, nz=64, stretch=1.5),
        # pressure solves alone, of the two grids they are reported on
        dict(name="poisson_128x128x128", kind="poisson", nx=128, ny=128, nz=128, lx=1.0, ly=1.0, lz=1.0, stretch=0.0,
             plain=False),
        dict(name="poisson_256x128x128_plain", kind="poisson", nx=256, ny=128, nz=128, lx=16.0, ly=2.0, lz=2.0,
             stretch=1.5, plain=True),
        # the pressure-guess network at inference and in training
        dict(name="forward_64x32x32", kind="forward", nx=64, ny=32, nz=32),
        dict(name="forward_256x128x128", kind="forward", nx=256, ny=128, nz=128),
        dict(name="gradient_128x64x64", kind="gradient", nx=128, ny=64, nz=64),
    ]


def _sizes(rng, most):
    """cell counts b 2^a whose hierarchy ends on few cells; at most `most`"""
    while True:
        a = rng.randint(3, 6)
        n = (rng.choice((4, 5, 6, 7, 8)) << a, rng.choice((2, 3, 4)) << a, rng.choice((2, 3, 4)) << a)
        if n[0] * n[1] * n[2] <= most and min(n) >= 16:
            return dict(zip(("nx", "ny", "nz"), n))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "predict", "poisson", "forward", "gradient"))
    if kind == "step":
        flow = rng.choice(("lock", "bump", "multi"))
        return dict(kind=kind, flow=flow, steps=rng.randint(1, 3), plain=rng.random() < 0.25, **_sizes(rng, 5 << 20))
    if kind == "predict":
        return dict(kind=kind, stretch=rng.choice((0.0, 1.2, 1.5)), **_sizes(rng, 8 << 20))
    if kind == "poisson":
        return dict(kind=kind, lx=16.0, ly=2.0, lz=2.0, stretch=rng.choice((0.0, 1.5)), plain=rng.random() < 0.4,
                    **_sizes(rng, 8 << 20))
    if kind == "forward":
        return dict(kind=kind, **_sizes(rng, 8 << 20))
    # training grids: powers of two, so that every level fills the weight gradient's voxel tiles
    return dict(kind=kind, nx=32 << rng.randint(0, 3), ny=16 << rng.randint(0, 2), nz=16 << rng.randint(0, 2))


# ---- inputs ------------------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _flow_case(flow, nx, ny, nz):
    """grid, immersed boundary and parameters: the same for every seed"""
    make = {"lock": W.lock_exchange_case, "bump": W.turbidity_bump_case, "multi": W.multi_bump_case}[flow]
    c = make(nx, ny, nz)
    c.state = None
    return c


@functools.lru_cache(maxsize=2)
def _box_case(nx, ny, nz, lx, ly, lz, stretch):
    """closed box without an immersed body, one settling fraction"""
    c = W.poisson_case(nx, ny, nz, (lx, ly, lz), stretch or None)
    p = c.params
    p.eno_order, p.ctype, p.vs0 = 3, [W.PARTICLE], [-0.02]
    c.state = None
    return c


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _modes(rng, x, y, z, lo, length, count, cosine=False):
    """sum of `count` products of sines (zero on the walls) or cosines"""
    f = np.cos if cosine else np.sin
    out = torch.zeros(len(z), len(y), len(x), dtype=torch.float64, device="cuda")
    for _ in range(count):
        k = rng.integers(1, (7, 4, 4))
        ex, ey, ez = (_t(f(np.pi * k[a] * (np.asarray(q) - lo[a]) / length[a])) for a, q in enumerate((x, y, z)))
        out += (rng.standard_normal() / np.sqrt(float((k * k).sum()))) * ez[:, None, None] * ey[:, None] * ex
    return out


def _developed(grid, nconc, seed):
    """state arrays (torch, GPU) of a developed current on `grid`"""
    rng = np.random.Generator(np.random.PCG64([seed, grid.nx, grid.ny, grid.nz]))
    xc, yc, zc, xu, yv, zw = grid.xc, grid.yc, grid.zc, grid.xu, grid.yv, grid.zw
    lo, ln = (xu[0], yv[0], zw[0]), (xu[-1] - xu[0], yv[-1] - yv[0], zw[-1] - zw[0])
    dx, dy, dz = _t(np.diff(xu)), _t(np.diff(yv))[:, None], _t(np.diff(zw))[:, None, None]
    ax = _modes(rng, xc, yv, zw, lo, ln, 6)
    ay = _modes(rng, xu, yc, zw, lo, ln, 6)
    az = _modes(rng, xu, yv, zc, lo, ln, 6)
    shape = grid.shape
    s = {k: torch.zeros(shape, dtype=torch.float64, device="cuda") for k in ("u", "v", "w", "phi", "dpx", "dpy", "dpz")}
    s["u"][:-1, :-1, 1:-1] = ((az.diff(dim=1) / dy)[:-1] - (ay.diff(dim=0) / dz)[:, :-1])[:, :, 1:-1]
    s["v"][:-1, 1:-1, :-1] = ((ax.diff(dim=0) / dz)[:, :, :-1] - (az.diff(dim=2) / dx)[:-1])[:, 1:-1]
    s["w"][1:-1, :-1, :-1] = ((ay.diff(dim=2) / dx)[:, :-1] - (ax.diff(dim=1) / dy)[:, :, :-1])[1:-1]
    top = max(float(s[q].abs().max()) for q in "uvw")
    for q in "uvw":
        s[q] *= 0.3 / top
    X, Y, Z = _t(xc), _t(yc)[:, None], _t(zc)[:, None, None]
    front = 0.3 * ln[0] + 0.02 * ln[0] * torch.sin(2 * np.pi * Z / ln[2] + rng.uniform(0, 6.0))
    layer = 0.25 * (1 - torch.tanh((X - front) / (0.02 * ln[0]))) * (1 - torch.tanh((Y - 0.6 * ln[1]) / (0.1 * ln[1])))
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 77)
    total = torch.zeros(shape, dtype=torch.float64, device="cuda")
    dead = _status(grid, "c", (W.BOUNDARY, W.SOLID))
    for i in range(nconc):
        c = layer + 2e-3 * (torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen) - 0.5)
        c = torch.where(layer > 1e-6, c, layer).clamp_(0.0, 1.0)
        c[dead] = 0.0
        s["c%d" % i] = c
        total += c / nconc
    # hydrostatic pressure of the layer, and the last step's small increment
    hyd = (layer * _t(np.gradient(yc))[:, None]).flip(1).cumsum(1).flip(1)
    s["dpx"][:, :, 1:] = hyd.diff(dim=2) / _t(np.diff(xc))
    s["dpy"][:, 1:] = hyd.diff(dim=1) / _t(np.diff(yc))[:, None]
    s["dpz"][1:] = hyd.diff(dim=0) / _t(np.diff(zc))[:, None, None]
    s["phi"][:-1, :-1, :-1] = 1e-3 * _modes(rng, xc, yc, zc, lo, ln, 6, cosine=True)[:-1, :-1, :-1]
    for q, k in (("u", "dpx"), ("v", "dpy"), ("w", "dpz")):
        s[k][_status(grid, q, (W.BOUNDARY,))] = 0.0
    return s


def _status(grid, q, codes):
    st = torch.as_tensor(grid.status[q], device="cuda")
    m = st == codes[0]
    for c in codes[1:]:
        m |= st == c
    return m


FIELD = dict(u=A.F_U, v=A.F_V, w=A.F_W, phi=A.F_PHI, dpx=A.F_DPX, dpy=A.F_DPY, dpz=A.F_DPZ, c0=A.F_C0, c1=A.F_C0 + 1,
             conv_u=A.F_CONV_U, conv_v=A.F_CONV_V, conv_w=A.F_CONV_W, conv_c=A.F_CCONV0)


def _pinned(arrays):
    """[(field, page-locked host copy)]"""
    out = []
    for k, t in arrays.items():
        h = A.host_empty(tuple(t.shape))
        torch.from_numpy(h).copy_(t)
        out.append((FIELD[k], h))
    return out


class _State:
    """a context, its inputs and its outputs in page-locked host memory"""

    def __init__(self, case, inputs, outputs):
        self.case = case
        self.ctx = A.Context(case.grid, case.params)
        self.inputs = _pinned(inputs)
        self.out = {k: A.host_empty(case.grid.shape) for k in outputs}
        self.outputs = [(FIELD[k], a) for k, a in self.out.items()]


def _velocity(case, seed):
    """random Fourier velocity of the pressure solves (not divergence-free)"""
    return {k: torch.from_numpy(a) for k, a in W.fourier_velocity(case.grid, int(seed)).items()}


# the network's layers (channels in, channels out) and its parameter vector:
# per layer W[27][out][in] and b[out], then 16 head weights and the head bias
LAYERS = ((16, 16), (16, 32), (32, 64), (64, 128), (128, 128), (128, 64), (64, 64), (64, 32), (32, 32), (32, 16), (16, 16))


def _net_inputs(case, seed):
    n = (case["nz"], case["ny"], case["nx"])
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    parts = []
    for cin, cout in LAYERS:
        parts += [rng.standard_normal(27 * cin * cout) * np.sqrt(2.0 / (27 * cin)), 0.05 * rng.standard_normal(cout)]
    parts += [rng.standard_normal(16) * 0.25, 0.05 * rng.standard_normal(1)]
    x = torch.randn((3,) + n, device="cuda", generator=gen)
    g = 1.0 + 0.5 * torch.randn(n, device="cuda", generator=gen)   # a loss gradient with a common part
    return np.concatenate(parts).astype(np.float32), x, g


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        p, x, g = _net_inputs(case, seed)
        net = N.Net(case["nx"], case["ny"], case["nz"], train=kind == "gradient")
        net.set_params(p)
        return dict(case=case, net=net, x=x, g=g, out=torch.zeros_like(g))
    if kind == "step":
        c = _flow_case(case["flow"], case["nx"], case["ny"], case["nz"])
        s = _developed(c.grid, c.params.nconc, seed)
        st = _State(c, s, list(s))
        if case["plain"]:
            st.ctx.set_pressure_mode(A.PMODE_FP64)
            st.ctx.set_helmholtz_mode(A.HMODE_FP64)
    elif kind == "predict":
        c = _box_case(case["nx"], case["ny"], case["nz"], 16.0, 2.0, 2.0, case["stretch"])
        s = _developed(c.grid, 1, seed)
        s.pop("phi")
        st = _State(c, s, ["u", "v", "w", "c0", "conv_u", "conv_v", "conv_w", "conv_c"])
    else:
        c = _box_case(case["nx"], case["ny"], case["nz"], case["lx"], case["ly"], case["lz"], case["stretch"])
        s = _velocity(c, seed)
        s["phi"] = torch.zeros(c.grid.shape, dtype=torch.float64)
        st = _State(c, s, ["u", "v", "w", "phi"])
        if case["plain"]:
            st.ctx.set_pressure_mode(A.PMODE_FP64)
    return dict(case=case, st=st)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        state["net"].forward(state["x"], state["out"])
        if kind == "forward":
            return state["out"]
        state["net"].backward(state["g"])
        return [state["out"], state["net"].get_grads()]
    st = state["st"]
    ctx = st.ctx
    ctx.upload_many(st.inputs)
    if kind == "step":
        ctx.reset_pressure_history()
        for _ in range(case["steps"]):
            ctx.step(st.case.dt)
    elif kind == "predict":
        dt = DT["bump"]
        ctx.Velocity_cell_center()
        for q in "uvw":
            ctx.Velocity_convective_terms(q)
        ctx.Conc_convective_terms(0)
        for q in "uvw":
            ctx.Velocity_set_RHS(q, dt)
            ctx.Velocity_solve(q, dt)
        ctx.Conc_set_RHS(0, dt)
        ctx.Conc_solve(0, dt)
    else:
        ctx.Pressure_set_RHS(1.0)
        ctx.Pressure_solve()
        ctx.Pressure_project_velocity(1.0)
    ctx.download_many(st.outputs)
    return st.out


def work(case):
    """bytes: inputs read and outputs written once; flops: the least a pass
    computes (per node and routine, iterations of the solvers not counted)"""
    n = float(case["nx"] * case["ny"] * case["nz"])
    kind = case["kind"]
    if kind == "forward":
        return {"bytes": 16.0 * n, "flops": 2.0 * 25920 * n}
    if kind == "gradient":
        return {"bytes": 20.0 * n, "flops": 6.0 * 25920 * n}
    if kind == "step":
        nq = 3 + (2 if case["flow"] == "multi" else 1)
        return {"bytes": 16.0 * (nq + 4) * n, "flops": case["steps"] * 2.0 * (nq * 75.0 + 60.0) * n}
    if kind == "predict":
        return {"bytes": 8.0 * (7 + 8) * n, "flops": 4 * 75.0 * n}
    return {"bytes": 8.0 * (3 + 4) * n, "flops": 30.0 * n}


# ---- the same in 64 bits, in plain numpy and torch -----------------------------

def _ghosts(q, pos, axis, r, lo, hi):
    """line buffers with r ghost nodes at each end: lo, hi = (on the wall,
    wall coordinate, multiple of the end node's value the ghosts take)"""
    P = np.concatenate([np.zeros(r), pos, np.zeros(r)])
    nb = len(P)
    first, last = q.narrow(axis, 0, 1), q.narrow(axis, q.shape[axis] - 1, 1)
    a, b = [], []
    for e in range(r):
        wall, at, m = lo
        end = wall and e == r - 1
        P[e] = at if end else 2 * at - P[2 * r - e - (2 if wall else 1)]
        a.append(first * (0.0 if end else m))
        wall, at, m = hi
        end = wall and e == r - 1
        P[nb - 1 - e] = at if end else 2 * at - P[nb - 2 * r + e + (1 if wall else 0)]
        b.insert(0, last * (0.0 if end else m))
    return torch.cat(a + [q] + b, axis), P


def _eno3(q, vel, pos, axis, lo, hi):
    """vel * dq/dx along an axis, third-order ENO"""
    r = 3
    D0, P = _ghosts(q, pos, axis, r, lo, hi)
    sh = [1, 1, 1]
    sh[axis] = -1

    def over(a, h):
        return a / _t(h).reshape(sh)

    n = q.shape[axis]
    D1 = over(D0.diff(dim=axis), np.diff(P))                 # D1[b] between b, b+1
    D2 = over(D1.diff(dim=axis), P[2:] - P[:-2])             # D2[t] at buffer index t + 1
    D3 = over(D2.diff(dim=axis), P[3:] - P[:-3])             # D3[t] at buffer index t + 1

    def at(D, shift):                                        # value at node c + shift, c = r .. r + n - 1
        return D.narrow(axis, r + shift, n)

    x = P
    c = np.arange(r, r + n)
    up = vel > 0
    d1 = torch.where(up, at(D1, -1), at(D1, 0))
    a, b = torch.where(up, at(D2, -2), at(D2, -1)), torch.where(up, at(D2, -1), at(D2, 0))
    left = a.abs() <= b.abs()
    g0 = _t((x[c] - x[c - 1]) + (x[c] - x[c])).reshape(sh)
    g1 = _t((x[c] - x[c]) + (x[c] - x[c + 1])).reshape(sh)
    d = d1 + torch.where(left, a, b) * torch.where(up, g0, g1)
    ks = torch.where(up, -1, 0) + torch.where(left, -1, 0)   # -2, -1, 0: first node of the third difference
    out = torch.zeros_like(d)
    for t in (-2, -1, 0):
        e, f = at(D3, t - 1), at(D3, t)
        p, s, w = x[c + t], x[c + t + 1], x[c + t + 2]
        g = _t((x[c] - p) * (x[c] - s) + (x[c] - s) * (x[c] - w) + (x[c] - p) * (x[c] - w)).reshape(sh)
        out = torch.where(ks == t, torch.where(e.abs() <= f.abs(), e, f) * g, out)
    return vel * (d + out)


def _between(f, axis, to, x0, x1):
    """the two-point means of the transposed velocities: weight |to - x0| /
    (x1 - x0) on the lower node, the rest on the upper"""
    sh = [1, 1, 1]
    sh[axis] = -1
    w = _t(np.abs((to - x0) / (x1 - x0))).reshape(sh)
    n = f.shape[axis]
    return f.narrow(axis, 0, n - 1) * w + f.narrow(axis, 1, n - 1) * (1 - w)


def _diffuse(b, dt, coef, kinds, robin):
    """(1/dt - coef Laplacian)^-1 b on a box by the eigenvectors of the three
    one-dimensional operators; kinds: (node widths, distances to the nodes
    before and after, Dirichlet) per axis of b; robin: factor folded at the end
    of the y axis"""
    lam, back = [], b
    basis = []
    for axis, (w, f, wall) in enumerate(kinds):
        n = len(w)
        T = np.zeros((n, n))
        for i in range(n):
            for j, d in ((i - 1, f[i]), (i + 1, f[i + 1])):
                a = 1.0 / d
                if 0 <= j < n:
                    T[i, i] += a
                    T[i, j] -= a
                elif wall:
                    T[i, i] += a
                elif axis == 1 and j == n:
                    T[i, i] += a * (1 - robin)
        s = 1.0 / np.sqrt(w)
        val, V = np.linalg.eigh(s[:, None] * T * s[None, :])
        lam.append(val)
        basis.append((_t((V.T) / s[None, :]), _t(s[:, None] * V)))
    for axis, (fw, _) in enumerate(basis):
        back = torch.tensordot(fw, back, dims=([1], [axis])).movedim(0, axis)
    z, y, x = (_t(v) for v in lam)
    back = back / (1.0 / dt + coef * (z[:, None, None] + y[:, None] + x))
    for axis, (_, bw) in enumerate(basis):
        back = torch.tensordot(bw, back, dims=([1], [axis])).movedim(0, axis)
    return back


def _exact_predict(case, seed):
    c = _box_case(case["nx"], case["ny"], case["nz"], 16.0, 2.0, 2.0, case["stretch"])
    g, p, dt = c.grid, c.params, DT["bump"]
    s = _developed(g, 1, seed)
    X, Y, Z = (g.xc[:-1], g.xu), (g.yc[:-1], g.yv), (g.zc[:-1], g.zw)
    u, v, w, cc = (s[k] for k in ("u", "v", "w", "c0"))
    U, V, Wv = u[:-1, :-1, :], v[:-1, :, :-1], w[:, :-1, :-1]      # with both walls
    C = cc[:-1, :-1, :-1]
    faces = {"x": X[1], "y": Y[1], "z": Z[1]}
    mir = {a: (False, faces[a][0], 1.0) for a in "xyz"}
    mir2 = {a: (False, faces[a][-1], 1.0) for a in "xyz"}
    # cell-centre velocities
    ub = U[..., :-1] + U.diff(dim=2) * _t((X[0] - X[1][:-1]) / np.diff(X[1]))
    vb = V[:, :-1] + V.diff(dim=1) * _t((Y[0] - Y[1][:-1]) / np.diff(Y[1]))[:, None]
    wb = Wv[:-1] + Wv.diff(dim=0) * _t((Z[0] - Z[1][:-1]) / np.diff(Z[1]))[:, None, None]
    ax = {"x": (2, X), "y": (1, Y), "z": (0, Z)}

    def to_face(f, a):     # centre-spaced along a -> inner faces of a
        i, (ce, fa) = ax[a]
        return _between(f, i, fa[1:-1], ce[:-1], ce[1:])

    def to_centre(f, a):   # face-spaced along a -> centres of a
        i, (ce, fa) = ax[a]
        return _between(f, i, ce, fa[:-1], fa[1:])

    ui, vi, wi = U[:, :, 1:-1], V[:, 1:-1], Wv[1:-1]
    cv = {}
    cv["u"] = _eno3(ui, ui, X[1][1:-1], 2, (True, X[1][0], -1.0), (True, X[1][-1], 0.0)) \
        + _eno3(ui, to_centre(to_face(V, "x"), "y"), Y[0], 1, mir["y"], mir2["y"]) \
        + _eno3(ui, to_centre(to_face(Wv, "x"), "z"), Z[0], 0, mir["z"], mir2["z"])
    cv["v"] = _eno3(vi, to_face(to_centre(U, "x"), "y"), X[0], 2, mir["x"], mir2["x"]) \
        + _eno3(vi, vi, Y[1][1:-1], 1, (True, Y[1][0], 0.0), (True, Y[1][-1], 0.0)) \
        + _eno3(vi, to_face(to_centre(Wv, "z"), "y"), Z[0], 0, mir["z"], mir2["z"])
    cv["w"] = _eno3(wi, to_face(to_centre(U, "x"), "z"), X[0], 2, mir["x"], mir2["x"]) \
        + _eno3(wi, to_centre(to_face(V, "z"), "y"), Y[0], 1, mir["y"], mir2["y"]) \
        + _eno3(wi, wi, Z[1][1:-1], 0, (True, Z[1][0], 0.0), (True, Z[1][-1], 0.0))
    half = 2.0 * (Y[1][-1] - Y[0][-1])
    b, vs = 2.0 / (p.pe[0] * half), abs(p.vs0[0])
    robin = (b - vs) / (b + vs)
    cv["c"] = _eno3(C, ub, X[0], 2, mir["x"], mir2["x"]) \
        + _eno3(C, vb + p.vs0[0], Y[0], 1, mir["y"], (False, Y[1][-1], robin)) \
        + _eno3(C, wb, Z[0], 0, mir["z"], mir2["z"])

    def centre(a):
        _, (ce, fa) = ax[a]
        d = np.concatenate([[2 * (ce[0] - fa[0])], np.diff(ce), [2 * (fa[-1] - ce[-1])]])
        return np.diff(fa), d, False

    def face(a):
        _, (ce, fa) = ax[a]
        return np.diff(ce), np.diff(fa), True

    out = {}
    kinds = {"u": (centre("z"), centre("y"), face("x")), "v": (centre("z"), face("y"), centre("x")),
             "w": (face("z"), centre("y"), centre("x")), "c": (centre("z"), centre("y"), centre("x"))}
    at = {"u": np.s_[:-1, :-1, 1:-1], "v": np.s_[:-1, 1:-1, :-1], "w": np.s_[1:-1, :-1, :-1], "c": np.s_[:-1, :-1, :-1]}
    buoy = C[:, :-1] + C.diff(dim=1) * _t((Y[1][1:-1] - Y[0][:-1]) / np.diff(Y[0]))[:, None]
    for q, f in (("u", ui), ("v", vi), ("w", wi), ("c", C)):
        rhs = f / dt - cv[q]
        if q != "c":
            rhs = rhs - s["dp" + "xyz"["uvw".index(q)]][at[q]]
        if q == "v":
            rhs = rhs - buoy
        sol = _diffuse(rhs, dt, 1.0 / (p.pe[0] if q == "c" else p.re), kinds[q], robin if q == "c" else 1.0)
        for k, val in (("c0" if q == "c" else q, sol), ("conv_" + q, cv[q])):
            full = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
            full[at[q]] = val
            out[k] = full
    return out


def _exact_poisson(case, seed):
    c = _box_case(case["nx"], case["ny"], case["nz"], case["lx"], case["ly"], case["lz"], case["stretch"])
    g = c.grid
    s = {k: _t(a) for k, a in _velocity(c, seed).items()}
    U, V, Wv = s["u"][:-1, :-1], s["v"][:-1, :, :-1], s["w"][:, :-1, :-1]
    wx, wy, wz = np.diff(g.xu), np.diff(g.yv), np.diff(g.zw)
    div = U.diff(dim=2) / _t(wx) + V.diff(dim=1) / _t(wy)[:, None] + Wv.diff(dim=0) / _t(wz)[:, None, None]
    vol = _t(wz)[:, None, None] * _t(wy)[:, None] * _t(wx)
    # eigenvectors of W^-1/2 K W^-1/2 per direction
    lam, fwd, bwd = [], [], []
    for w, ce in ((wz, g.zc), (wy, g.yc), (wx, g.xc)):
        n = len(w)
        d = 1.0 / np.diff(ce[:n])
        K = np.diag(np.concatenate([d, [0]]) + np.concatenate([[0], d])) - np.diag(d, 1) - np.diag(d, -1)
        r = 1.0 / np.sqrt(w)
        val, vec = np.linalg.eigh(r[:, None] * K * r[None, :])
        val[0] = 0.0
        lam.append(val)
        fwd.append(_t(vec.T / r[None, :]))
        bwd.append(_t(r[:, None] * vec))
    rhs = -div                                     # dt = 1
    rhs = rhs - (rhs * vol).sum() / vol.sum()
    for axis in range(3):
        rhs = torch.tensordot(fwd[axis], rhs, dims=([1], [axis])).movedim(0, axis)
    den = _t(lam[0])[:, None, None] + _t(lam[1])[:, None] + _t(lam[2])
    den[0, 0, 0] = 1.0
    rhs = rhs / den
    rhs[0, 0, 0] = 0.0
    for axis in range(3):
        rhs = torch.tensordot(bwd[axis], rhs, dims=([1], [axis])).movedim(0, axis)
    phi = rhs - rhs[-1, -1, -1]                    # the corner cell's level is pinned to the (zero) net source
    out = {k: s[k].clone() for k in "uvw"}
    out["u"][:-1, :-1, 1:-1] -= phi.diff(dim=2) / _t(np.diff(g.xc[:-1]))
    out["v"][:-1, 1:-1, :-1] -= phi.diff(dim=1) / _t(np.diff(g.yc[:-1]))[:, None]
    out["w"][1:-1, :-1, :-1] -= phi.diff(dim=0) / _t(np.diff(g.zc[:-1]))[:, None, None]
    full = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    full[:-1, :-1, :-1] = phi
    out["phi"] = full
    return out


def _exact_net(case, seed):
    F = torch.nn.functional
    p, x, g = _net_inputs(case, seed)
    p = torch.from_numpy(p).double().cuda().requires_grad_(True)
    at, Ws, bs = 0, [], []
    for cin, cout in LAYERS:
        Ws.append(p[at:at + 27 * cin * cout].reshape(27, cout, cin))
        at += 27 * cin * cout
        bs.append(p[at:at + cout])
        at += cout

    def conv(i, a):
        ap = F.pad(a, (1, 1, 1, 1, 1, 1))
        n = a.shape[1:]
        out = bs[i][:, None].expand(-1, a[0].numel())
        for t in range(27):
            dx, dy, dz = t % 3, (t // 3) % 3, t // 9
            out = out + Ws[i][t] @ ap[:, dz:dz + n[0], dy:dy + n[1], dx:dx + n[2]].reshape(a.shape[0], -1)
        return out.reshape((-1,) + tuple(n))

    def down(a):
        return F.avg_pool3d(a[None], 2)[0]

    def up(a):
        return a.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    relu = torch.relu
    x0 = torch.cat([x.double(), torch.zeros((13,) + tuple(x.shape[1:]), dtype=torch.float64, device="cuda")])
    with torch.set_grad_enabled(case["kind"] == "gradient"):
        a0 = relu(conv(0, x0))
        a1 = relu(conv(1, down(a0)))
        a2 = relu(conv(2, down(a1)))
        b3 = relu(conv(4, relu(conv(3, down(a2)))))
        b2 = relu(conv(6, relu(up(conv(5, b3)) + a2)))
        b1 = relu(conv(8, relu(up(conv(7, b2)) + a1)))
        b0 = relu(conv(10, relu(up(conv(9, b1)) + a0)))
        out = (p[at:at + 16, None, None, None] * b0).sum(0) + p[at + 16]
    if case["kind"] == "forward":
        return out
    out.backward(g.double())
    return [out.detach(), p.grad.cpu()]


def exact(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "predict":
        return _exact_predict(case, seed)
    if kind == "poisson":
        return _exact_poisson(case, seed)
    if kind in ("forward", "gradient"):
        return _exact_net(case, seed) if n <= 1 << 20 else None
    return None          # whole steps: the solvers of every routine above, twice a step
