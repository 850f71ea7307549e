"""The workloads whose speed is followed: one pass of each through the public Python interface.

What each kind of case stands for in use:

  step    one simulation (Navier2D.new / new_periodic): `steps` updates, then its five spectral fields are read back,
          as a run does between two save points.  FP64 is the default precision, mixed the tensor-core option.
  batch   independent simulations advanced together (Batch): `steps` updates, then the whole state in one copy.
  field   a field's transforms and derivatives (Space2 on device arrays): forward, backward and both first derivatives.
  solve   the Helmholtz (HholtzAdi, or Hholtz on a Fourier axis) and Poisson solves of a field's right-hand side.
  lanes   1-D transforms and solves of many lanes (Lanes on device arrays).

`exact` evaluates the same discrete equations with dense 64-bit matrices along each axis.
"""
import ctypes
import math

import numpy as np
import torch

import rustpde_gb300 as R
from rustpde_gb300.ensemble import draw_ensemble

KINDS = {"adiabatic": R.BOX_ADIABATIC, "conducting": R.BOX_CONDUCTING, "periodic": R.PERIODIC}
FIELDS = (R.TEMP, R.UX, R.UY, R.PRES, R.PSEUDO_PRES)
PREC = {"fp64": R.PREC_FP64, "mixed": R.PREC_MIXED}


def _step(kind, nx, ny, ra, steps, prec="fp64", pr=1.0, aspect=1.0):
    return {"do": "step", "kind": kind, "nx": nx, "ny": ny, "ra": ra, "pr": pr, "aspect": aspect,
            "dt": min(0.02, 2.0 / math.sqrt(ra)), "steps": steps, "prec": prec}


def listed():
    return [
        # the smallest configured box: latency and launches count
        dict(_step("adiabatic", 64, 64, 1e5, 20), name="box64"),
        # the solver benchmark's sizes: 129 (2^p + 1), 264 (263 is a prime) and 513, its largest
        dict(_step("adiabatic", 129, 129, 1e6, 10), name="box129"),
        dict(_step("conducting", 264, 264, 1e7, 5, pr=0.7), name="box264"),
        dict(_step("adiabatic", 513, 513, 1e7, 5), name="box513"),
        # the configured periodic channel, in both precisions
        dict(_step("periodic", 512, 257, 1e7, 10, aspect=2.0), name="periodic512x257"),
        dict(_step("periodic", 512, 257, 1e7, 10, "mixed", aspect=2.0), name="periodic512x257 mixed"),
        # the ensemble benchmark (uneven sizes, both kinds), and a small ensemble in the default precision
        {"name": "ensemble256 mixed", "do": "batch", "cases": 256, "draw": 2024, "steps": 5, "prec": "mixed"},
        {"name": "ensemble16", "do": "batch", "cases": 16, "draw": 5, "steps": 5, "prec": "fp64"},
        # one field's transforms, at sizes with and without a power of two
        {"name": "field264x265", "do": "field", "base0": "dirichlet", "n0": 264, "base1": "dirichlet", "n1": 265},
        # the implicit solves of a field
        {"name": "solve257x256", "do": "solve", "base0": "dirichlet", "n0": 257, "base1": "dirichlet", "n1": 256},
        # the lane benchmark: 4096 lanes, the largest length mixed and the smallest in FP64
        {"name": "lanes512 mixed", "do": "lanes", "base": "dirichlet", "n": 512, "lanes": 4096, "prec": "mixed"},
        {"name": "lanes128", "do": "lanes", "base": "dirichlet", "n": 128, "lanes": 4096, "prec": "fp64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["step", "step", "step", "batch", "field", "solve", "lanes"])
    if do == "step":
        prec = rng.choice(["fp64", "fp64", "mixed"])
        kind = rng.choice(list(KINDS))
        nx = _log(rng, 24, 513 if kind != "periodic" else 600)
        ny = rng.choice([_log(rng, 24, 300), 2 ** rng.randint(5, 8) + 1])
        if kind != "periodic":
            ny = max(24, min(513, ny + (nx - ny) // 2))
        ra = float("%.3g" % 10 ** rng.uniform(4.0, 7.0))
        return _step(kind, nx, ny, ra, rng.randint(4, 8), prec, rng.choice([0.7, 1.0, 7.0]),
                     round(rng.uniform(1.0, 2.0), 3))
    if do == "batch":
        prec = rng.choice(["mixed", "fp64"])
        return {"do": "batch", "cases": _log(rng, 2, 96 if prec == "mixed" else 24), "draw": rng.randint(1, 10**6),
                "steps": rng.randint(3, 6), "prec": prec}
    if do == "lanes":
        return {"do": "lanes", "base": rng.choice(["dirichlet", "neumann"]), "n": _log(rng, 16, 512),
                "lanes": _log(rng, 64, 4096), "prec": rng.choice(["fp64", "mixed"])}
    bases = ["dirichlet", "neumann"] if do == "field" else ["dirichlet"]
    return {"do": do, "base0": rng.choice(bases + ["fourier"]), "n0": _log(rng, 16, 400), "base1": rng.choice(bases),
            "n1": rng.choice([_log(rng, 16, 400), 2 ** rng.randint(4, 8) + 1])}


# --------------------------------------------------------------------------------------------------------- the passes
class DevBuf:
    """A torch tensor as the device buffer that the library's *_dev calls take."""

    def __init__(self, t):
        self.t = t
        self.ptr = ctypes.c_void_p(t.data_ptr())


BASES = {"chebyshev": R.chebyshev, "dirichlet": R.cheb_dirichlet, "neumann": R.cheb_neumann, "fourier": R.fourier_r2c}


def _modes(rng):
    """Smooth large-scale initial fields: amplitude and wave numbers of the velocity and the temperature."""
    return (float(rng.uniform(0.1, 0.3)), int(rng.integers(1, 3)), int(rng.integers(1, 3)),
            float(rng.uniform(0.1, 0.3)), int(rng.integers(1, 3)), int(rng.integers(1, 3)))


def _initial(sim, modes):
    sim.set_velocity(*modes[:3])
    sim.set_temperature(*modes[3:])


def _normal(shape, seed, cplx=False):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.complex128 if cplx else torch.float64)


def _decay(shape, seed, cplx):
    """Spectral coefficients of a resolved field: random, falling off with the mode number."""
    k = [torch.arange(n, device="cuda", dtype=torch.float64) / n for n in shape]
    return _normal(shape, seed, cplx) * torch.exp(-8.0 * (k[0][:, None] + k[1][None, :]))


def _field_inputs(case, seed):
    """Physical values, spectral shape, whether spectral data is complex."""
    fourier = case["base0"] == "fourier"
    m0 = case["n0"] // 2 + 1 if fourier else case["n0"] - 2
    return _normal((case["n0"], case["n1"]), seed), (m0, case["n1"] - 2), fourier


def _solve_inputs(case, seed):
    fourier = case["base0"] == "fourier"
    o0 = case["n0"] // 2 + 1 if fourier else case["n0"]
    return _decay((o0, case["n1"]), seed, fourier)


def _solve_coefs(case):
    return (5e-4, 3e-4), (1.0, 0.8)


def _lane_inputs(case, seed):
    n = case["n"]
    m = n if case["base"] == "chebyshev" else n - 2
    phys, spec = _normal((case["lanes"], n), seed), _normal((case["lanes"], m), seed + 1)
    return phys, spec * torch.exp(-4.0 * torch.arange(m, device="cuda", dtype=torch.float64) / m)


LANE_OPS = ((R.OP_FORWARD, 0), (R.OP_BACKWARD, 1), (R.OP_FROM_ORTHO, 0), (R.OP_HHOLTZ, 0))
LANE_C = 5e-4


def prepare(case, seed):
    do = case["do"]
    if do == "step":
        sim = R.Navier2D(case["nx"], case["ny"], case["ra"], case["pr"], case["dt"], case["aspect"],
                         KINDS[case["kind"]], PREC[case["prec"]])
        _initial(sim, _modes(np.random.default_rng(seed)))
        sim.synchronize()
        return do, sim, case["steps"]
    if do == "batch":
        params = draw_ensemble(case["cases"], case["draw"])
        b = R.Batch(params, precision=PREC[case["prec"]])
        rng = np.random.default_rng(seed)
        for c in b.cases:
            _initial(c, _modes(rng))
        b.synchronize()
        return do, b, case["steps"], torch.empty(b.state_bytes() // 8, dtype=torch.float64, pin_memory=True)
    if do == "lanes":
        L = R.Lanes(BASES[case["base"]](case["n"]), PREC[case["prec"]], hholtz_c=LANE_C)
        ins = [DevBuf(t) for t in _lane_inputs(case, seed)]
        outs = [DevBuf(torch.empty((case["lanes"], L.lengths(op)[1]), device="cuda", dtype=torch.float64))
                for op, _ in LANE_OPS]
        torch.cuda.synchronize()
        return do, L, ins, outs, case["lanes"]
    space = R.Space2(BASES[case["base0"]](case["n0"]), BASES[case["base1"]](case["n1"]))
    dt = torch.complex128 if space.is_complex else torch.float64
    new = lambda shape, d=dt: DevBuf(torch.empty(shape, device="cuda", dtype=d))  # noqa: E731
    if do == "field":
        phys, _, _ = _field_inputs(case, seed)
        st = (do, space, DevBuf(phys), new(space.spectral), new(space.physical, torch.float64),
              new(space.ortho), new(space.ortho))
    else:
        ch, cp = _solve_coefs(case)
        H = R.Hholtz(space, ch) if space.is_complex else R.HholtzAdi(space, ch)
        st = (do, H, R.Poisson(space, cp), DevBuf(_solve_inputs(case, seed)), new(space.spectral), new(space.spectral))
    torch.cuda.synchronize()
    return st


def run(state):
    do = state[0]
    if do == "step":
        _, sim, steps = state
        sim.update(steps)
        return [sim.get(f) for f in FIELDS]
    if do == "batch":
        _, b, steps, host = state
        b.update(steps)
        b.get_state_all(host.numpy())
        return host
    if do == "lanes":
        _, L, ins, outs, lanes = state
        for (op, which), out in zip(LANE_OPS, outs):
            L.apply_dev(op, ins[which], out, lanes)
        return [o.t for o in outs]
    if do == "field":
        _, space, phys, spec, back, gx, gy = state
        space.forward_dev(phys, spec)
        space.backward_dev(spec, back)
        space.gradient_dev(spec, gx, (1, 0), (2.0, 1.0))
        space.gradient_dev(spec, gy, (0, 1), (2.0, 1.0))
        return [spec.t, back.t, gx.t, gy.t]
    _, H, P, rhs, a, b = state
    H.solve_dev(rhs, a)
    P.solve_dev(rhs, b)
    return [a.t, b.t]


# ------------------------------------------------------------------------------------------------------ work, at least
def _dct(n):
    """Flops of one real fast cosine (or half a complex Fourier) transform of length n."""
    return 2.5 * n * math.log2(n)


def _step_work(nx, ny, periodic, steps):
    mx = nx // 2 + 1 if periodic else nx - 2
    cells = mx * (2 if periodic else 1)
    state = 8 * cells * (4 * (ny - 2) + ny)
    rows, cols = cells, ny
    # nine inverse and three forward transforms along each axis, some 60 flops of solves per value and field
    flops = 9 * (rows * _dct(ny) + cols * _dct(nx)) + 3 * (nx * _dct(ny) + cols * _dct(nx)) + 3 * 60 * cells * ny
    if not periodic:
        flops += 2 * 2 * mx * mx * ny  # the two eigenbasis products of the Poisson solve
    return 2 * state, steps * flops


def work(case):
    do = case["do"]
    if do == "step":
        b, f = _step_work(case["nx"], case["ny"], case["kind"] == "periodic", case["steps"])
    elif do == "batch":
        ws = [_step_work(p[0], p[1], p[6] == R.PERIODIC, case["steps"]) for p in draw_ensemble(case["cases"], case["draw"])]
        b, f = sum(w[0] for w in ws), sum(w[1] for w in ws)
    elif do == "lanes":
        b = 8 * case["lanes"] * case["n"] * 2 * len(LANE_OPS)
        f = case["lanes"] * (2 * _dct(case["n"]) + 20 * case["n"])
    else:
        n0, n1 = case["n0"], case["n1"]
        pts = n0 * n1
        if do == "field":
            b, f = 8 * pts * (1 + 1 + 1 + 2), 2 * (n0 * _dct(n1) + n1 * _dct(n0)) + 30 * pts
        else:
            b, f = 8 * pts * 3, 60 * pts + (0 if case["base0"] == "fourier" else 4 * n0 * n0 * n1)
    return {"bytes": float(b), "flops": float(f)}


# --------------------------------------------------------------------------------- the same equations, dense, in 64 bits
class Axis:
    """One axis: matrices between physical values, orthogonal and composite coefficients (x' = M x along it)."""

    def __init__(self, base, n):
        self.fourier = base == "fourier"
        if self.fourier:
            self.n, self.m = n, n // 2 + 1
            self.k = np.arange(self.m, dtype=np.float64)
            self.A, self.B, self.P = np.eye(self.m), np.diag(-self.k**2), None
            return
        self.n = n
        j = np.arange(n)
        cos = np.cos(np.pi * (np.outer(j, j) % (2 * (n - 1))) / (n - 1))
        sign = np.where(j % 2, -1.0, 1.0)
        end = np.where((j == 0) | (j == n - 1), 0.5, 1.0)
        self.Bk = cos * sign[None, :]                                   # coefficients -> values
        self.Fw = cos * (2.0 / (n - 1) * sign * end)[:, None] * end[None, :]  # values -> coefficients
        p, q = np.meshgrid(j, j, indexing="ij")
        self.D = np.where((q > p) & ((p + q) % 2 == 1), 2.0 * q, 0.0)
        self.D[0] *= 0.5
        if base == "chebyshev":
            self.S = np.eye(n)
        else:
            k = np.arange(n - 2, dtype=np.float64)
            self.S = np.eye(n, n - 2) + np.eye(n, n - 2, -2) * (-1.0 if base == "dirichlet" else -(k**2) / (k + 2) ** 2)
        self.m = self.S.shape[1]
        self.Si = np.linalg.solve(self.S.T @ self.S, self.S.T) if self.m < n else np.eye(n)
        li = np.zeros((n, n))
        i = np.arange(3, n)
        li[2, 0] = 0.25
        li[i, i - 2] = 1.0 / (4.0 * i * (i - 1))
        i = np.arange(2, n - 2)
        li[i, i] = -1.0 / (2.0 * (i * i - 1.0))
        i = np.arange(2, n - 4)
        li[i, i + 2] = 1.0 / (4.0 * i * (i + 1))
        S = self.S[:, 2:] if base == "chebyshev" else self.S
        self.P = li[2:]
        self.A, self.B = self.P @ S, S[2:]


def _ax(M, a, axis):
    return M @ a if axis == 0 else a @ M.T


class Grid:
    """Two axes; every operation takes and gives 2-D arrays."""

    def __init__(self, x, y):
        self.x, self.y = x, y

    def forward(self, v):
        a = _ax(self.y.Si @ self.y.Fw, v, 1)
        return np.fft.rfft(a, axis=0) if self.x.fourier else _ax(self.x.Si @ self.x.Fw, a, 0)

    def to_ortho(self, c):
        a = _ax(self.y.S, c, 1)
        return a if self.x.fourier else _ax(self.x.S, a, 0)

    def from_ortho(self, o):
        a = _ax(self.y.Si, o, 1)
        return a if self.x.fourier else _ax(self.x.Si, a, 0)

    def grad(self, o, d, scale):
        """First derivative of orthogonal coefficients along axis d."""
        if d:
            return _ax(self.y.D, o, 1) / scale[1]
        return (1j * self.x.k[:, None] * o if self.x.fourier else _ax(self.x.D, o, 0)) / scale[0]

    def values(self, o):
        a = _ax(self.y.Bk, o, 1)
        return np.fft.irfft(a, n=self.x.n, axis=0) if self.x.fourier else _ax(self.x.Bk, a, 0)

    def coefs(self, v):
        a = _ax(self.y.Fw, v, 1)
        return np.fft.rfft(a, axis=0) if self.x.fourier else _ax(self.x.Fw, a, 0)

    def rhs(self, o):
        a = _ax(self.y.P, o, 1)
        return a if self.x.fourier else _ax(self.x.P, a, 0)


def _rows(lam, A, B, cA, rhs):
    """Solve (cA_i A + B) x_i = rhs_i for every row i."""
    return np.linalg.solve(cA(lam)[:, None, None] * A[None] + B[None], rhs[:, :, None])[:, :, 0]


def _hholtz_adi(g, c):
    ix, iy = (np.linalg.inv(a.A - c[d] * a.B) for d, a in ((0, g.x), (1, g.y)))
    return lambda o: _ax(iy, _ax(ix, g.rhs(o), 0), 1)


def _inv_rows(lam, A, B):
    return np.linalg.inv(lam[:, None, None] * A[None] + B[None])


def _hholtz(g, c):
    inv = _inv_rows(1.0 + c[0] * g.x.k**2, g.y.A, -c[1] * g.y.B)
    return lambda o: np.einsum("iab,ib->ia", inv, g.rhs(o))


def _poisson(g, c):
    if g.x.fourier:
        lam, Q, Qi = -c[0] * g.x.k**2, None, None
    else:
        lam, Q = np.linalg.eig(np.linalg.solve(g.x.A, c[0] * g.x.B))
        at = np.argsort(-lam.real)
        lam, Q = lam.real[at], Q.real[:, at]
        Qi = np.linalg.inv(Q) @ np.linalg.inv(g.x.A)
    if abs(lam[0]) < 1e-10:
        lam = lam - 1e-10
    inv = _inv_rows(lam, g.y.A, c[1] * g.y.B)

    def solve(o):
        r = g.rhs(o)
        r = r if Q is None else Qi @ r
        r = np.einsum("iab,ib->ia", inv, r)
        return r if Q is None else Q @ r
    return solve


_axes = {}


def _axis(base, n):
    if (base, n) not in _axes:
        _axes[base, n] = Axis(base, n)
    return _axes[base, n]


def _exact_step(nx, ny, ra, pr, dt, aspect, kind, steps, modes):
    per = kind == R.PERIODIC
    ax = lambda b, n: _axis(b, n)  # noqa: E731
    y, X = ax("dirichlet", ny), (lambda b: ax("fourier" if per else b, nx))
    gu, gt = Grid(X("dirichlet"), y), Grid(X("neumann" if kind == R.BOX_ADIABATIC else "dirichlet"), y)
    gp, go = Grid(X("neumann"), ax("neumann", ny)), Grid(X("chebyshev"), ax("chebyshev", ny))
    nu, ka = math.sqrt(pr / (ra / 8.0)), math.sqrt(1.0 / (ra / 8.0 * pr))
    s = (aspect, 1.0)
    make = _hholtz if per else _hholtz_adi
    su = make(gu, [dt * nu / q**2 for q in s])
    st = make(gt, [dt * ka / q**2 for q in s])
    sp = _poisson(gp, [1.0 / q**2 for q in s])
    xs = np.arange(nx) / (nx - 1.0) if per else (1.0 - np.cos(np.pi * np.arange(nx) / (nx - 1))) / 2.0
    ys = (1.0 - np.cos(np.pi * np.arange(ny) / (ny - 1))) / 2.0
    wave = lambda f, h, m, n: f(np.pi * m * xs)[:, None] * h(np.pi * n * ys)[None, :]  # noqa: E731
    a, m, n, b, k, l = modes
    ux, uy = gu.forward(a * wave(np.sin, np.cos, m, n)), gu.forward(-a * wave(np.cos, np.sin, m, n))
    t = gt.forward(-b * wave(np.cos, np.sin, k, l))
    ot = gt.to_ortho(t)
    p0, p1 = np.zeros_like(ot), None
    bc = np.zeros_like(ot)
    bc[0, 1] = -0.5 * (nx if per else 1.0)  # the conduction profile
    cut = (np.arange(ot.shape[0])[:, None] < ot.shape[0] * 2 // 3) & (np.arange(ny)[None, :] < ny * 2 // 3)
    for _ in range(steps):
        ou, ov, ot = gu.to_ortho(ux), gu.to_ortho(uy), gt.to_ortho(t)
        u, v = go.values(ou), go.values(ov)
        conv = [cut * go.coefs(u * go.values(go.grad(o, 0, s)) + v * go.values(go.grad(o, 1, s))) for o in (ou, ov, ot + bc)]
        ux = su(ou - dt * go.grad(p0, 0, s) - dt * conv[0])
        uy = su(ov - dt * go.grad(p0, 1, s) + dt * (ot + bc) - dt * conv[1])
        div = go.grad(gu.to_ortho(ux), 0, s) + go.grad(gu.to_ortho(uy), 1, s)
        p1 = sp(div)
        p1[0, 0] = 0.0
        o1 = gp.to_ortho(p1)
        ux = ux - gu.from_ortho(go.grad(o1, 0, s))
        uy = uy - gu.from_ortho(go.grad(o1, 1, s))
        p0 = p0 - nu * div + o1 / dt
        t = st(ot - dt * conv[2])
    return [t, ux, uy, p0, p1]


def exact(case, seed):
    do = case["do"]
    if do == "step":
        return _exact_step(case["nx"], case["ny"], case["ra"], case["pr"], case["dt"], case["aspect"],
                           KINDS[case["kind"]], case["steps"], _modes(np.random.default_rng(seed)))
    if do == "batch":
        return None  # one value per case of many: over the time allowed; single cases are held to it above
    if do == "lanes":
        a = _axis(case["base"], case["n"])
        phys, spec = (t.cpu().numpy() for t in _lane_inputs(case, seed))
        H = np.linalg.solve(a.A - LANE_C * a.B, a.P)
        ops = {R.OP_FORWARD: a.Si @ a.Fw, R.OP_BACKWARD: a.Bk @ a.S, R.OP_FROM_ORTHO: a.Si, R.OP_HHOLTZ: H}
        return [(spec if which else phys) @ ops[op].T for op, which in LANE_OPS]
    g = Grid(_axis(case["base0"], case["n0"]), _axis(case["base1"], case["n1"]))
    if do == "field":
        phys = _field_inputs(case, seed)[0].cpu().numpy()
        spec = g.forward(phys)
        o = g.to_ortho(spec)
        return [spec, g.values(o), g.grad(o, 0, (2.0, 1.0)), g.grad(o, 1, (2.0, 1.0))]
    o = _solve_inputs(case, seed).cpu().numpy()
    ch, cp = _solve_coefs(case)
    return [(_hholtz if g.x.fourier else _hholtz_adi)(g, ch)(o), _poisson(g, cp)(o)]
