"""The work that programs have this integrator do, as cases that can be timed.

Every case is one call sequence through the package's public entry points: a
single step, propagations to a time or over a grid (double and single
precision, shared-memory, global-memory and team kernels), an ensemble over
many small integrators, terminal events, continuous output, first-order
variational equations and a differentiable propagation with its backward pass.
Systems and distributions are the package's own workloads (``hyk.workloads``:
pendulum, Kepler orbits, circular restricted three-body problem near L4,
Sun with five planets); batch sizes go from 4 lanes to 2^20.

The 64-bit values of ``exact`` are computed here: Kepler orbits from the
closed-form two-body solution (its state-transition matrix by forward-mode
differentiation of it), the others with a Gauss-Legendre collocation
integrator of 8 stages (order 16) with compensated summation.
"""

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("heyoka.py_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

# Per system: equations, flops of one Taylor step at the default order (the
# recurrences' convolutions, the polynomial of the state and the step size)
# and the mean number of steps per unit of time of the package's workloads.
_SYSTEMS = {
    "pendulum": {"n_eq": 2, "n_pars": 0, "flops": 1077, "rate": 9.4},
    "kepler": {"n_eq": 6, "n_pars": 0, "flops": 3194, "rate": 4.15},
    "kepler_f32": {"n_eq": 6, "n_pars": 0, "flops": 959, "rate": 4.31},
    "kepler_var": {"n_eq": 42, "n_pars": 0, "flops": 33418, "rate": 4.87},
    "cr3bp": {"n_eq": 6, "n_pars": 1, "flops": 5264, "rate": 1.094},
    "oss": {"n_eq": 36, "n_pars": 0, "flops": 48444, "rate": 0.003},
}


def listed():
    return [
        # One step of a batch as wide as a CPU's vector unit, from a loop that
        # looks at the state after every step: latency and launches only.
        {"name": "step_pendulum_4", "kind": "step", "system": "pendulum", "lanes": 4},
        # 1024 integrators of 4 lanes as one ensemble (the reference's
        # ensemble_propagate_until_batch with a generator of initial states).
        {"name": "ensemble_pendulum_1024x4", "kind": "ensemble", "system": "pendulum", "iters": 1024, "batch": 4,
         "lanes": 4096, "t": 100.0},
        # An ordinary small batch of an odd size: a few orbits of 1003 bodies,
        # far fewer lanes than the GPU has threads.
        {"name": "until_kepler_1003", "kind": "until", "system": "kepler", "lanes": 1003, "t": 50.0},
        # The headline workload: 2^20 Kepler orbits, one tenth of t = 200.
        {"name": "until_kepler_2p20", "kind": "until", "system": "kepler", "lanes": 1 << 20, "t": 20.0},
        # The same ensemble in single precision (fp_type=numpy.float32).
        {"name": "until_kepler_f32_2p20", "kind": "until", "system": "kepler_f32", "lanes": 1 << 20, "t": 20.0},
        # Dense output of an uneven number of CR3BP trajectories at 41 times.
        {"name": "grid_cr3bp_20011", "kind": "grid", "system": "cr3bp", "lanes": 20011, "t": 50.0, "points": 41},
        # Gradients through a propagation: final states and the gradients with
        # respect to the initial states and the mass parameter.
        {"name": "flow_cr3bp_16384", "kind": "flow", "system": "cr3bp", "lanes": 16384, "t": 50.0},
        # A large ensemble of a large system, end times from 1e3 to 1e5 days.
        {"name": "grid_oss_65536", "kind": "grid", "system": "oss", "lanes": 65536, "t": 1e5, "points": 25},
        # A small ensemble of the same system (a parameter scan of 331 members).
        {"name": "until_oss_331", "kind": "until", "system": "oss", "lanes": 331, "t": 2e4},
        # Propagation to each lane's first upward crossing of the vertical
        # (a Poincare section: a terminal event without a callback).
        {"name": "event_pendulum_10007", "kind": "event", "system": "pendulum", "lanes": 10007, "t": 20.0},
        # Continuous output of 2003 orbits, evaluated at 16 times afterwards.
        {"name": "coutput_kepler_2003", "kind": "coutput", "system": "kepler", "lanes": 2003, "t": 6.0, "points": 16},
        # State-transition matrices: first-order variational equations of
        # Kepler orbits (42 equations).
        {"name": "var_kepler_3001", "kind": "until", "system": "kepler_var", "lanes": 3001, "t": 10.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["step", "ensemble", "kepler", "kepler", "kepler_f32", "cr3bp", "flow", "oss_grid", "oss",
                       "event", "coutput", "var"])
    if kind == "step":
        return {"kind": "step", "system": rng.choice(["pendulum", "kepler"]), "lanes": int(_log(rng, 1, 4096))}
    if kind == "ensemble":
        it, b = int(_log(rng, 16, 1024)), rng.choice([1, 2, 4])
        return {"kind": "ensemble", "system": "pendulum", "iters": it, "batch": b, "lanes": it * b,
                "t": rng.uniform(10.0, 100.0)}
    if kind in ("kepler", "kepler_f32"):
        return {"kind": "until", "system": kind, "lanes": int(_log(rng, 100, 1 << 20)), "t": rng.uniform(5.0, 20.0)}
    if kind == "cr3bp":
        return {"kind": "grid", "system": "cr3bp", "lanes": int(_log(rng, 500, 60000)), "t": rng.uniform(10.0, 50.0),
                "points": rng.randint(5, 60)}
    if kind == "flow":
        return {"kind": "flow", "system": "cr3bp", "lanes": int(_log(rng, 500, 16384)), "t": rng.uniform(10.0, 50.0)}
    if kind == "oss_grid":
        return {"kind": "grid", "system": "oss", "lanes": int(_log(rng, 2000, 32768)), "t": 1e5,
                "points": rng.randint(5, 25)}
    if kind == "oss":
        return {"kind": "until", "system": "oss", "lanes": int(_log(rng, 32, 2000)), "t": rng.uniform(5e3, 2e4)}
    if kind == "event":
        return {"kind": "event", "system": "pendulum", "lanes": int(_log(rng, 64, 100000)), "t": 20.0}
    if kind == "coutput":
        return {"kind": "coutput", "system": "kepler", "lanes": int(_log(rng, 32, 4000)), "t": rng.uniform(3.0, 6.0),
                "points": rng.randint(4, 20)}
    return {"kind": "until", "system": "kepler_var", "lanes": int(_log(rng, 100, 6000)), "t": rng.uniform(3.0, 10.0)}


def _steps(case):
    """The mean number of Taylor steps per lane."""
    r = _SYSTEMS[case["system"]]["rate"]
    if case["kind"] == "step":
        return 1.0
    if case["kind"] == "event":
        return 1.0 * r  # the first upward crossing comes 0.3 to 1.8 time units after the start
    if case["system"] == "oss" and case["kind"] == "grid":
        return r * (1e5 - 1e3) / math.log(1e2)  # end times log-uniform in [1e3, 1e5]
    return r * case["t"]


def work(case):
    s, n = _SYSTEMS[case["system"]], case["lanes"]
    size = 4 if case["system"] == "kepler_f32" else 8
    rows = s["n_eq"] + s["n_pars"]
    b = size * n * (rows + s["n_eq"])
    fl = s["flops"] * _steps(case) * n
    if case["kind"] in ("grid", "coutput"):
        # the times in, the rows out
        b += size * n * case["points"] * (1 + s["n_eq"])
        fl += 2.0 * 19 * s["n_eq"] * n * case["points"]
    if case["kind"] == "flow":
        # the gradient of the final state in, those of the state and the
        # parameter out; the reverse sweep's chains have two terms for every
        # term of the step, and the step's coefficients come first
        b += size * n * (2 * s["n_eq"] + s["n_pars"])
        fl *= 4.0
    return {"bytes": float(b), "flops": float(fl)}


# ---------------------------------------------------------------- inputs
def _host_inputs(case, seed):
    """(initial states, parameters or None, end times or None) as NumPy arrays."""
    from hyk import workloads as W

    n = case["lanes"]
    if case["system"] == "pendulum":
        return W.pendulum_ics(n, seed=seed), None, None
    if case["system"] in ("kepler", "kepler_var"):
        return W.kepler_ics(n, seed=seed), None, None
    if case["system"] == "kepler_f32":
        return W.kepler_ics(n, seed=seed).astype(np.float32), None, None
    if case["system"] == "cr3bp":
        st, mu = W.cr3bp_ics(n, seed=seed)
        return st, mu, None
    st, t_end = W.oss_ics(n, seed=seed)
    return st, None, t_end


def _grid(case, t_end):
    """The time grid of a grid case, shape (points, lanes)."""
    u = np.linspace(0.0, 1.0, case["points"]).reshape(-1, 1)
    return u * (t_end if t_end is not None else np.full(case["lanes"], case["t"])).reshape(1, -1)


def _tm(case):
    """The evaluation times of a continuous-output case, shape (points, lanes)."""
    u = (np.arange(case["points"]).reshape(-1, 1) + 0.37) / case["points"]
    return u * np.linspace(0.9, 1.0, case["lanes"]).reshape(1, -1) * case["t"]


def _weights(case, seed):
    """The gradient of a loss with respect to the final states."""
    return np.random.default_rng([seed, 17]).normal(size=(6, case["lanes"]))


def prepare(case, seed):
    import hyk
    from hyk import workloads as W

    st, pars, t_end = _host_inputs(case, seed)
    dev = torch.device("cuda")
    s = {"case": case, "x0": torch.tensor(st, device=dev)}
    if case["kind"] == "flow":
        s["sys"] = W.cr3bp_sys()
        s["x0"].requires_grad_(True)
        s["pars"] = torch.tensor(pars, device=dev, requires_grad=True)
        s["w"] = torch.tensor(_weights(case, seed), device=dev)
        return s
    tol = 0.0
    if case["system"] == "pendulum":
        sys_, tol = W.pendulum_sys(), 2.2e-16
    elif case["system"] == "kepler":
        sys_, tol = W.kepler_sys(), 1e-15
    elif case["system"] == "kepler_f32":
        sys_ = W.kepler_sys()
    elif case["system"] == "kepler_var":
        from hyk import var

        sys_, tol = var.var_ode_sys(W.kepler_sys(), var.var_args.vars, order=1), 1e-15
        # the matrix part starts from the identity
        s["x0"] = torch.cat([s["x0"], torch.eye(6, dtype=torch.float64, device=dev).reshape(36, 1).expand(36, st.shape[1])])
    elif case["system"] == "cr3bp":
        sys_, tol = W.cr3bp_sys(), 1e-15
    else:
        sys_, tol = W.oss_sys(), 1e-15
    kw = {"tol": tol}
    if case["system"] == "kepler_f32":
        kw["fp_type"] = np.float32
    if case["kind"] == "event":
        x = sys_[0][0]
        kw["t_events"] = [hyk.t_event_batch(x, direction=hyk.event_direction.positive)]
    if case["kind"] == "ensemble":
        b = case["batch"]
        s["ta"] = hyk.taylor_adaptive_batch(sys_, np.ascontiguousarray(st[:, :b]), **kw)
        s["ics"] = [np.ascontiguousarray(st[:, i * b:(i + 1) * b]) for i in range(case["iters"])]
        del s["x0"]
        return s
    s["ta"] = hyk.taylor_adaptive_batch(sys_, st, pars=pars, **kw)
    if case["kind"] == "grid":
        s["grid"] = torch.tensor(_grid(case, t_end), device=dev)
    if case["kind"] == "coutput":
        s["tm"] = _tm(case)
    return s


def _plain(t):
    return t.as_subclass(torch.Tensor)


def run(s):
    import hyk
    from hyk.adjoint import taylor_flow

    case = s["case"]
    kind = case["kind"]
    if kind == "flow":
        x, _ = taylor_flow(s["sys"], s["x0"], case["t"], pars=s["pars"], tol=1e-15)
        gx, gp = torch.autograd.grad(x, (s["x0"], s["pars"]), s["w"])
        return [x.detach(), gx, gp]
    ta = s["ta"]
    if kind == "ensemble":
        ics = s["ics"]

        def gen(tac, i):
            tac.set_time(0.0)
            tac.state[:] = ics[i]
            return tac

        ret = hyk.ensemble_propagate_until_batch(ta, case["t"], case["iters"], gen)
        return [torch.stack([_plain(r[0].state) for r in ret])]
    ta.set_time(0.0)
    ta.state[:] = s["x0"]
    if kind == "step":
        ta.step()
        return [_plain(ta.state), ta.time]
    if kind == "until":
        ta.propagate_until(case["t"])
        return [_plain(ta.state)]
    if kind == "grid":
        out = ta.propagate_grid_tensor(s["grid"])
        return [out]
    if kind == "event":
        ta.reset_cooldowns()
        ta.propagate_until(case["t"])
        return [_plain(ta.state), ta.time]
    co, _ = ta.propagate_until(case["t"], c_output=True)
    return [co(s["tm"])]


# ---------------------------------------------------------------- 64-bit values
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _kepler_flow(x0, t):
    """The two-body state (mu = 1) a time t after x0 ((6, n) rows, t
    broadcastable), by Lagrange's f and g in the eccentric anomaly."""
    x, y, z, vx, vy, vz = x0
    r0 = (x * x + y * y + z * z).sqrt()
    v2 = vx * vx + vy * vy + vz * vz
    rv = x * vx + y * vy + z * vz
    al = 2.0 / r0 - v2
    sa = al.sqrt()
    ec, es = 1.0 - r0 * al, rv * sa
    m = t * al * sa
    k = torch.floor(m.detach() / (2.0 * math.pi))
    m = m - k * (2.0 * math.pi)
    d = m.detach().clone()
    with torch.no_grad():
        for _ in range(40):
            f = d - ec * torch.sin(d) + es * (1.0 - torch.cos(d)) - m
            fp = 1.0 - ec * torch.cos(d) + es * torch.sin(d)
            d = d - torch.clamp(f / fp, -1.0, 1.0)
    for _ in range(2):  # the last iterations carry the derivatives
        f = d - ec * torch.sin(d) + es * (1.0 - torch.cos(d)) - m
        d = d - f / (1.0 - ec * torch.cos(d) + es * torch.sin(d))
    sd, od = torch.sin(d), 2.0 * torch.sin(0.5 * d) ** 2  # od = 1 - cos d
    a = 1.0 / al
    r = a * (1.0 - ec * (1.0 - od) + es * sd)
    f = 1.0 - a / r0 * od
    g = r0 * sd / sa + a * rv * od
    fd = -sd / (sa * r * r0)
    gd = 1.0 - a / r * od
    return torch.stack([f * x + g * vx, f * y + g * vy, f * z + g * vz,
                        fd * x + gd * vx, fd * y + gd * vy, fd * z + gd * vz])


def _rhs_pendulum(s):
    return torch.stack([s[1], -9.8 * torch.sin(s[0])])


def _cr3bp_terms(s, mu):
    x, y, z = s[0], s[1], s[2]
    a, b = x - mu, x - mu + 1.0
    q = y * y + z * z
    r1, r2 = a * a + q, b * b + q
    return a, b, r1, r2, r1 ** -1.5, r2 ** -1.5


def _rhs_cr3bp(mu):
    def f(s):
        a, b, _, _, w1, w2 = _cr3bp_terms(s, mu)
        c = (1.0 - mu) * w1 + mu * w2
        return torch.stack([s[3] + s[1], s[4] - s[0], s[5], s[4] - (1.0 - mu) * w1 * a - mu * w2 * b,
                            -s[3] - c * s[1], -c * s[2]])
    return f


def _rhs_cr3bp_adjoint(mu):
    """State (6), its adjoint (6) and the gradient of the parameter (1)."""
    def f(s):
        a, b, r1, r2, w1, w2 = _cr3bp_terms(s, mu)
        m1 = 1.0 - mu
        y, z = s[1], s[2]
        c = m1 * w1 + mu * w2
        u1, u2 = -3.0 * m1 * w1 / r1, -3.0 * mu * w2 / r2  # d(m w)/d(r^2) * 2
        l0, l1, l2, l3, l4, l5 = s[6], s[7], s[8], s[9], s[10], s[11]
        # force F = (F3, F4, F5); its Jacobian with respect to (x, y, z) is symmetric
        fxx = -c - u1 * a * a - u2 * b * b
        fxy = -(u1 * a + u2 * b) * y
        fxz = -(u1 * a + u2 * b) * z
        fyy = -c - (u1 + u2) * y * y
        fyz = -(u1 + u2) * y * z
        fzz = -c - (u1 + u2) * z * z
        # dF/dmu: a and b decrease with mu, the masses change
        e = w2 - w1 - u1 * a - u2 * b  # dc/dmu
        fm3 = w1 * a + c - w2 * b + u1 * a * a + u2 * b * b
        fm4, fm5 = -e * y, -e * z
        return torch.stack([
            s[3] + y, s[4] - s[0], s[5], s[4] - m1 * w1 * a - mu * w2 * b, -s[3] - c * y, -c * z,
            l1 - (fxx * l3 + fxy * l4 + fxz * l5),
            -l0 - (fxy * l3 + fyy * l4 + fyz * l5),
            -(fxz * l3 + fyz * l4 + fzz * l5),
            -l0 + l4, -l1 - l3, -l2,
            -(fm3 * l3 + fm4 * l4 + fm5 * l5),
        ])
    return f


def _rhs_oss():
    from hyk import workloads as W

    gm = [W.OSS_G * m for m in W.OSS_MASSES]
    nb = len(gm)

    def f(s):
        p = [s[6 * i:6 * i + 3] for i in range(nb)]
        out = torch.empty_like(s)
        for i in range(nb):
            out[6 * i:6 * i + 3] = s[6 * i + 3:6 * i + 6]
            out[6 * i + 3:6 * i + 6] = 0.0
        for i in range(nb):
            for j in range(i + 1, nb):
                d = p[j] - p[i]
                r2 = (d * d).sum(dim=0)
                t = d / (r2 * r2.sqrt())
                out[6 * i + 3:6 * i + 6] += gm[j] * t
                out[6 * j + 3:6 * j + 6] -= gm[i] * t
        return out
    return f


def _gauss_tables(s=8):
    c, w = np.polynomial.legendre.leggauss(s)
    c, w = 0.5 * (c + 1.0), 0.5 * w
    bw = np.array([1.0 / np.prod([c[i] - c[j] for j in range(s) if j != i]) for i in range(s)])

    def lagrange(u):  # rows: points, columns: basis polynomials
        d = u.reshape(-1, 1) - c.reshape(1, -1)
        full = np.array([[np.prod([u[k] - c[j] for j in range(s) if j != i]) for i in range(s)] for k in range(len(u))])
        del d
        return full * bw.reshape(1, -1)

    a = np.array([ci * (w @ lagrange(ci * c)) for ci in c])
    return torch.tensor(a), torch.tensor(w), torch.tensor(lagrange(1.0 + c))


class _Gauss:
    """Gauss-Legendre collocation for x' = f(x), lanes in the last dimension;
    the state is carried as an unevaluated sum of two doubles."""

    def __init__(self, f, x, iters=60):
        self.f, self.hi, self.lo = f, x.clone(), torch.zeros_like(x)
        self.a, self.w, self.ext = (t.to(x.device) for t in _gauss_tables())
        self.k = None
        self.iters = iters

    def stages(self, h, guess=None):
        s = self.a.shape[0]
        ne, b = self.hi.shape
        x = self.hi.unsqueeze(1)
        lo = self.lo.unsqueeze(1)
        # (ne, s, B)
        k = guess if guess is not None else self.f(self.hi).unsqueeze(1).expand(ne, s, b)
        last = math.inf
        for _ in range(self.iters):
            y = x + (lo + h * torch.matmul(self.a, k))
            kn = self.f(y)
            e = float(((kn - k).abs().amax(dim=(1, 2)) / kn.abs().amax(dim=(1, 2)).clamp(min=1e-300)).max())
            k = kn
            if e < 1e-15 or (e < 1e-12 and e >= last):
                break
            last = e
        return k

    def increment(self, h, k):
        return h * torch.einsum("s,nsb->nb", self.w, k)

    def step(self, h, keep=None):
        guess = None if self.k is None else torch.matmul(self.ext, self.k)
        k = self.stages(h, guess)
        self.k = k
        d = self.increment(h, k) + self.lo
        s = self.hi + d
        bb = s - self.hi
        lo = (self.hi - (s - bb)) + (d - bb)
        if keep is not None:  # lanes that have stopped stay
            s, lo = torch.where(keep, self.hi, s), torch.where(keep, self.lo, lo)
        self.hi, self.lo = s, lo

    def advance(self, h, n):
        for _ in range(n):
            self.step(h)
        return self.hi


_FREQ = {"pendulum": 3.2, "cr3bp": 1.5, "oss": 1.46e-3}  # fastest angular frequency, sets the substep


def _substeps(system, t):
    return max(1, int(math.ceil(t * _FREQ[system] / 0.5)))


def _pendulum_step_size(x, v, order=20):
    """Jorba and Zou's step size from the Taylor coefficients of orders 0, p - 1 and p."""
    n_l = x.shape[0]
    xs, vs = np.zeros((order + 1, n_l)), np.zeros((order + 1, n_l))
    s, c = np.zeros((order + 1, n_l)), np.zeros((order + 1, n_l))
    xs[0], vs[0], s[0], c[0] = x, v, np.sin(x), np.cos(x)
    for n in range(order):
        xs[n + 1] = vs[n] / (n + 1)
        vs[n + 1] = -9.8 * s[n] / (n + 1)
        j = np.arange(1, n + 2).reshape(-1, 1)
        s[n + 1] = (j * xs[1:n + 2] * c[n::-1][:n + 1]).sum(axis=0) / (n + 1)
        c[n + 1] = -(j * xs[1:n + 2] * s[n::-1][:n + 1]).sum(axis=0) / (n + 1)
    m = [np.maximum(np.abs(xs[o]), np.abs(vs[o])) for o in (0, order - 1, order)]
    num = np.maximum(m[0], 1.0)
    rho = np.minimum((num / m[1]) ** (1.0 / (order - 1)), (num / m[2]) ** (1.0 / order))
    return rho * math.exp(-2.0 - 0.7 / (order - 1))


def exact(case, seed):
    st, pars, t_end = _host_inputs(case, seed)
    d = _dev()
    kind, system = case["kind"], case["system"]
    x0 = torch.tensor(st.astype(np.float64), device=d)
    if kind == "step":
        if system != "pendulum":
            return None  # the step size of another system: no closed form at hand
        h = _pendulum_step_size(st[0], st[1])
        g = _Gauss(_rhs_pendulum, x0)
        g.advance(torch.tensor(h / 4.0, device=d), 4)
        return [g.hi, h]
    if system in ("kepler", "kepler_f32"):
        if kind == "coutput":
            return [torch.stack([_kepler_flow(x0, t) for t in torch.tensor(_tm(case), device=d)]).cpu().numpy()]
        return [_kepler_flow(x0, case["t"])]
    if system == "kepler_var":
        cols = []
        x = None
        for j in range(6):
            e = torch.zeros_like(x0)
            e[j] = 1.0
            x, dx = torch.func.jvp(lambda s: _kepler_flow(s, case["t"]), (x0,), (e,))
            cols.append(dx)
        return [torch.cat([x, torch.stack(cols, dim=1).reshape(36, -1)])]
    if kind == "ensemble":
        g = _Gauss(_rhs_pendulum, x0)
        n = _substeps(system, case["t"])
        x = g.advance(case["t"] / n, n)
        return [x.reshape(2, case["iters"], case["batch"]).permute(1, 0, 2).contiguous()]
    if kind == "event":
        # march until x crosses zero upwards, then Newton's method on the crossing time
        g = _Gauss(_rhs_pendulum, x0)
        h, n = 0.1, int(round(case["t"] / 0.1))
        stop = torch.zeros(x0.shape[1], dtype=torch.bool, device=d)
        t0 = torch.full((x0.shape[1],), float(case["t"]), dtype=torch.float64, device=d)
        at = x0.clone()
        for i in range(n):
            bh, bl = g.hi, g.lo
            g.step(torch.full_like(t0, h), keep=stop)
            hit = ~stop & (bh[0] < 0.0) & (g.hi[0] >= 0.0)
            t0 = torch.where(hit, torch.full_like(t0, i * h), t0)
            g.hi, g.lo = torch.where(hit, bh, g.hi), torch.where(hit, bl, g.lo)
            stop = stop | hit
            g.k = None
            if bool(stop.all()):
                break
        tau = torch.where(stop, -g.hi[0] / g.hi[1].clamp(min=0.1), torch.zeros_like(t0)).clamp(0.0, h)
        for _ in range(8):
            at = g.hi + (g.lo + g.increment(tau, g.stages(tau)))
            tau = torch.where(stop, tau - at[0] / at[1], tau)
        at = g.hi + (g.lo + g.increment(tau, g.stages(tau)))
        return [at, (t0 + tau).cpu().numpy()]
    if kind == "flow":
        mu = torch.tensor(pars[0], device=d)
        n = _substeps(system, case["t"])
        g = _Gauss(_rhs_cr3bp(mu), x0)
        x = g.advance(case["t"] / n, n)
        w = torch.tensor(_weights(case, seed), device=d)
        b = _Gauss(_rhs_cr3bp_adjoint(mu), torch.cat([x, w, torch.zeros_like(w[:1])]))
        b.lo[:6] = g.lo
        y = b.advance(-case["t"] / n, n)
        return [x, y[6:12], y[12:13]]
    f = _rhs_oss() if system == "oss" else _rhs_cr3bp(torch.tensor(pars[0], device=d))
    g = _Gauss(f, x0)
    if kind == "grid":
        grid = torch.tensor(_grid(case, t_end), device=d)
        rows = [x0]
        for i in range(1, grid.shape[0]):
            dt = grid[i] - grid[i - 1]
            n = _substeps(system, float(dt.max()))
            rows.append(g.advance(dt / n, n))
        return [torch.stack(rows)]
    n = _substeps(system, case["t"])
    return [g.advance(case["t"] / n, n)]
