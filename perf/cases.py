"""The work that a user of this package has it do, as timed cases through its public entry points.

Kinds of work:

* ``rhs``   one evaluation of the semi-discrete operator on a state (``DGFlux.semi_discrete_rhs``),
            as a caller with its own time integrator or a diagnostic of the operator makes it
* ``field`` the diagnostics of a state: density, spectral Poisson solve, field energy
            (``Distribution.moment_zero``, ``Elliptic.poisson2``, ``Elliptic.electric_energy``)
* ``step``  one nonlinear SSP-RK3 step at a time (``Stepper.nonlinear_ssp_rk``), the loop body of
            the reference's driver
* ``run``   a block of steps with its energy and time histories (``Stepper.run_steps``)
* ``loop``  a run to a final time (``Stepper.main_loop``)
* ``ens``   a block of steps of a heterogeneous ensemble (``Ensemble.run_steps``)
* ``train`` one epoch of the closure network's training with its validation
            (``closure.train``: forward, backward, Adam; ``closure.evaluate``: inference)

Sizes come from the repository's benchmark (32 x 50 x 50 elements of order 8, 64^3 of order 9, the
seeded ensemble), its small 16^3 configuration, the coarse grid of the closure experiment, and odd
grids whose rows are not multiples of 16 bytes.  FP64 is the plain form; FP32 the mixed form with
the background split (``run``, ``step``, ``loop``) or the plain FP32 state (``rhs``, ``field``,
``ens``).

``exact`` evaluates the same mathematics in 64 bits with plain torch, from the initial state.
"""
import math

import numpy as np
import torch

import vlasov1d2v_b200.closure as closure
from vlasov1d2v_b200 import problem
from vlasov1d2v_b200.ensemble import Ensemble, build_members, sample_members
from vlasov1d2v_b200.timestep import get_max_speeds


def _case(name, kind, res, n, prec="fp64", steps=1):
    return {"name": name, "kind": kind, "nx": res[0], "nu": res[1], "nv": res[2], "n": n, "prec": prec,
            "steps": steps}


def listed():
    return [
        # the smallest call: the operator on a toy grid, all launch and call overhead
        _case("rhs_f64_8x12x12_n4", "rhs", (8, 12, 12), 4),
        # the operator on an odd grid: ragged last v tile, rows of an odd number of values
        _case("rhs_f64_24x31x33_n7", "rhs", (24, 31, 33), 7),
        # diagnostics of the benchmark's state
        _case("field_f64_32x50x50_n8", "field", (32, 50, 50), 8),
        # the reference driver's loop body on the small validated configuration
        _case("step_f64_16x16x16_n8", "step", (16, 16, 16), 8),
        # a run to a final time on a coarse grid (about 100 short steps)
        _case("loop_f64_16x20x20_n6", "loop", (16, 20, 20), 6, steps=100),
        # the benchmark: blocks of steps in both precisions
        _case("run_f64_32x50x50_n8", "run", (32, 50, 50), 8, steps=10),
        _case("run_f32_32x50x50_n8", "run", (32, 50, 50), 8, "fp32", 10),
        # the largest configuration in both precisions
        _case("run_f64_64x64x64_n9", "run", (64, 64, 64), 9, steps=2),
        _case("run_f32_64x64x64_n9", "run", (64, 64, 64), 9, "fp32", 2),
        # FP32 on an odd grid
        _case("run_f32_20x27x29_n7", "run", (20, 27, 29), 7, "fp32", 8),
        # many small heterogeneous runs at once (orders 6 to 9)
        {"name": "ens_f32_24_members", "kind": "ens", "members": 24, "grid_seed": 0, "steps": 8},
        # the closure network: an epoch of 16 minibatches and a validation pass
        {"name": "train_131072_b8192", "kind": "train", "samples": 131072, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


_MAX_DOF = 48.0e6          # of a drawn grid
_MAX_DOF_STEPS = 191.0e6   # of a drawn case (the largest listed case: twice this)


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "field", "step", "step", "loop", "run", "run", "run", "run", "ens", "train"])
    if kind == "ens":
        return {"kind": "ens", "members": rng.randint(3, 24), "grid_seed": rng.randint(1, 10 ** 6),
                "steps": rng.randint(2, 8)}
    if kind == "train":
        batch = rng.randint(8, 128) * 64
        return {"kind": "train", "samples": batch * rng.randint(2, 16) + rng.randint(0, 63), "batch": batch}
    while True:
        n = rng.choice([3, 4, 5, 6, 6, 7, 8, 8, 8, 9, 9])
        res = (_log_int(rng, 4, 64), _log_int(rng, 6, 72), _log_int(rng, 6, 72))
        dof = res[0] * res[1] * res[2] * n ** 3
        if dof > _MAX_DOF or res[0] * n > 576:
            continue
        steps = 1 if kind in ("rhs", "field", "step") else rng.randint(2, 10) if kind == "run" else rng.randint(33, 120)
        if dof * steps > _MAX_DOF_STEPS:
            continue
        c = _case("", kind, res, n, rng.choice(["fp64", "fp32"]), steps)
        del c["name"]
        return c


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------
def _rng(seed):
    return np.random.default_rng([17, int(seed)])


def _build(case, seed):
    rng = _rng(seed)
    split = case["kind"] in ("step", "run", "loop")
    return problem.build((case["nx"], case["nu"], case["nv"]), case["n"], perturbation="cos",
                         amp=float(rng.uniform(2.0e-3, 8.0e-3)), noise=1.0e-4, seed=int(rng.integers(1 << 31)),
                         precision=case["prec"], batch_steps=max(case["steps"], 1) if case["kind"] == "run" else 32,
                         background_split=split)


def _members(case, seed):
    rng = _rng(seed)
    params = sample_members(case["members"], seed=case["grid_seed"])
    for q in params:
        q["amp"] = float(10 ** rng.uniform(-3.0, -2.0))
    return params


def _initial_dt(p):
    st = p.stepper
    st.adapt_time_step(max_speeds=get_max_speeds(p.grids, p.elliptic, p.refs), dx=p.grids.x.dx, du=p.grids.u.dx,
                       dv=p.grids.v.dx)
    return st.dt


def _train_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = case["samples"]

    def features(rows):
        X = torch.randn((rows, closure.IN), device="cuda", generator=g)
        X[:, 88:] = 0.0
        return X

    A = torch.randn((closure.IN, closure.NOUT), device="cuda", generator=g) / 10.0
    X, Xv = features(n), features(max(n // 8, 64))
    return X, torch.tanh(X @ A).contiguous(), Xv, torch.tanh(Xv @ A).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, T, Xv, Tv = _train_inputs(case, seed)
        return {"case": case, "seed": int(seed), "mlp": closure.MLP(seed=int(seed)), "X": X, "T": T, "Xv": Xv, "Tv": Tv}
    if kind == "ens":
        probs = build_members(_members(case, seed), precision="fp32", seed=int(seed), batch_steps=case["steps"])
        return {"case": case, "ens": Ensemble(probs, batch_steps=case["steps"])}
    p = _build(case, seed)
    if kind == "step":
        _initial_dt(p)
    elif kind == "loop":   # a final time between two steps
        p.stepper.final_time = (case["steps"] - 0.5) * _initial_dt(p)
        p.stepper.dt = None
    return {"case": case, "p": p}


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------
def _plain(t):
    return t.as_subclass(torch.Tensor)


def _fields(p, prec):
    """E and phi, in the precision that the state gives them."""
    E, phi = _plain(p.elliptic.electric_field), _plain(p.elliptic.potential)
    return (E, phi) if prec == "fp64" else (E.float(), phi.float())


def _history(a, prec):
    return np.asarray(a, dtype=np.float64 if prec == "fp64" else np.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        mlp = state["mlp"]
        hist = closure.train(mlp, state["X"], state["T"], epochs=1, batch=case["batch"], seed=state["seed"],
                             val=(state["Xv"], state["Tv"]))
        return {"w": mlp.master_w, "b": mlp.master_b, "val": hist[-1]["val_loss"]}
    if kind == "ens":
        ens = state["ens"]
        for p in ens.problems:   # a program that writes each block out and goes on
            st = p.stepper
            st.time_array, st.field_energy = st.time_array[-1:], st.field_energy[-1:]
        ens.run_steps(case["steps"])
        return {"f": [_plain(p.f.arr) for p in ens.problems],
                "energy": np.concatenate([_history(p.stepper.field_energy[1:], "fp32") for p in ens.problems])}
    p, prec = state["p"], case["prec"]
    if kind == "rhs":
        return _plain(p.flux.semi_discrete_rhs(p.f.arr, p.elliptic, p.basis, p.grids))
    if kind == "field":
        n0 = p.f.moment_zero()
        p.elliptic.poisson2(charge_density=n0 - torch.mean(n0), grid=p.grids.x, basis=p.basis.b1)
        energy = _plain(p.elliptic.electric_energy(grid=p.grids.x))
        E, phi = _fields(p, prec)
        return {"rho": _plain(n0), "E": E, "phi": phi, "energy": energy if prec == "fp64" else energy.float()}
    st = p.stepper
    args = (p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs)
    if kind == "step":
        st.nonlinear_ssp_rk(*args)
        E, phi = _fields(p, prec)
        return {"f": _plain(p.f.arr), "E": E, "phi": phi, "dt": _history([st.dt], prec)}
    if kind == "loop":
        st.time, st.steps_counter, st.write_counter = 0.0, 0, 1
        st.time_array, st.field_energy = np.array([0.0]), np.array([])
        st.main_loop(*args, None)
        done = st.steps_counter
    else:
        st.time_array, st.field_energy = st.time_array[-1:], st.field_energy[-1:]
        st.run_steps(*args, case["steps"])
        done = case["steps"]
    E, phi = _fields(p, prec)
    return {"f": _plain(p.f.arr), "E": E, "phi": phi, "energy": _history(st.field_energy[-done:], prec),
            "time": _history(st.time_array[-done:], prec)}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def _weights_count():
    return sum(k * n for k, n in closure.MLP.LAYERS)


def work(case):
    """Bytes: a right-hand side reads the state and writes its result; a step is eight passes over
    the state (three stages, each of which needs the field of the one before: 2 + 3 + 3).  Flops: per
    value and stage three contractions of n terms, their upwind terms and the combination."""
    kind = case["kind"]
    if kind == "train":
        n, v, w = case["samples"], max(case["samples"] // 8, 64), _weights_count()
        return {"bytes": 4.0 * (n + v) * (closure.IN + closure.NOUT), "flops": 6.0 * w * n + 2.0 * w * v}
    if kind == "ens":
        bytes_, flops = 0.0, 0.0
        for q in _members(case, 0):
            dof = q["res"][0] * q["res"][1] * q["res"][2] * q["order"] ** 3
            bytes_ += 32.0 * dof * case["steps"]
            flops += 3.0 * dof * (6 * q["order"] + 26) * case["steps"]
        return {"bytes": bytes_, "flops": flops}
    n = case["n"]
    dof = case["nx"] * case["nu"] * case["nv"] * n ** 3
    es = 8.0 if case["prec"] == "fp64" else 4.0
    if kind == "field":
        return {"bytes": es * dof, "flops": 2.0 * dof}
    if kind == "rhs":
        return {"bytes": 2 * es * dof, "flops": float(dof) * (6 * n + 20)}
    return {"bytes": 8 * es * dof * case["steps"], "flops": 3.0 * dof * (6 * n + 26) * case["steps"]}


# ----------------------------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ----------------------------------------------------------------------------------------------
def _lgl(n):
    """LGL nodes and weights: the roots of P'_{n-1}, polished by Newton steps in extended precision."""
    c = np.zeros(n)
    c[-1] = 1.0
    x = np.sort(np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c)).real).astype(np.longdouble)
    for _ in range(6):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(1, n - 1):
            p0, p1 = p1, ((2 * k + 1) * x * p1 - k * p0) / (k + 1)
        m = n - 1
        d = m * (p0 - x * p1) / (1 - x * x)                        # P'_m
        d2 = (2 * x * d - m * (m + 1) * p1) / (1 - x * x)          # P''_m
        x = x - d / d2
    x = np.concatenate([[-1.0], ((x - x[::-1]) / 2).astype(np.float64), [1.0]])
    w = 2.0 / (n * (n - 1) * np.polynomial.legendre.legval(x, c) ** 2)
    return x, w


class _Plain:
    """The discrete system of one problem in 64 bits: tables built here, on torch tensors."""

    def __init__(self, res, n, lows, highs, accel, bfield, kappa):
        leg = np.polynomial.legendre
        nodes, w = _lgl(n)
        P = np.array([leg.legval(nodes, np.eye(n)[s]) for s in range(n)])                    # P_s(x_i)
        D = np.array([leg.legval(nodes, leg.legder(np.eye(n)[s])) if s else 0 * nodes for s in range(n)])
        half = (2.0 * np.arange(n) + 1.0) / 2.0
        up = np.einsum("s,si,sj,j->ij", half, P, D, w)
        invm = np.diag(1.0 / w) + (n / 2.0) * np.outer(P[n - 1], P[n - 1])
        dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        self.n, self.res, self.accel, self.bfield, self.kappa = n, res, accel, bfield, kappa
        self.up, self.xl, self.xr = dev(up), dev(invm[:, 0]), dev(invm[:, -1])
        self.dx = [(highs[d] - lows[d]) / res[d] for d in range(3)]
        axes = [(np.linspace(lows[d] - self.dx[d], highs[d], res[d] + 2)[:, None] + self.dx[d] * (nodes + 1) / 2)
                for d in range(3)]
        self.u, self.v = dev(axes[1]), dev(axes[2])
        self.umax, self.vmax = float(np.abs(axes[1]).max()), float(np.abs(axes[2]).max())
        self.w = dev(w)
        # high-order DFT: exact transforms of the nodal basis (Gauss quadrature) and node phases
        L = highs[0] - lows[0]
        modes = np.arange(1, int(2.5 * L // self.dx[0]))
        k = 2.0 * np.pi / L * np.concatenate([-modes[::-1], modes])
        gx, gw = leg.leggauss(48)
        ev = np.append(half[:-1], (n - 1) / 2.0)
        vinv = ev[:, None] * P * w[None, :]                                                # [s, j]
        lag = vinv.T @ np.array([leg.legval(gx, np.eye(n)[s]) for s in range(n)])         # l_j at the points
        ell = (lag * gw) @ np.exp(-0.5j * self.dx[0] * np.multiply.outer(gx, k)) / 2.0     # [j, m]
        xs = axes[0][1:-1]
        mid = 0.5 * (xs[:, 0] + xs[:, -1])
        T = np.exp(-1j * np.multiply.outer(mid, k))[:, None, :] * ell[None]
        self.T = dev(T.reshape(-1, len(k))) * (self.dx[0] / L)
        self.Pk = dev(np.exp(1j * np.multiply.outer(xs.reshape(-1), k)))
        self.k = dev(k)

    def _lift(self, F, pos, ea, na):
        """up F minus the lifted upwind traces along element axis ea, node axis na."""
        d = torch.movedim(torch.tensordot(self.up, F, dims=([1], [na])), 0, na)
        last, first = F.select(na, self.n - 1), F.select(na, 0)
        left = torch.where(pos, torch.roll(last, 1, ea), first)
        right = torch.where(pos, last, torch.roll(first, -1, ea))
        shape = [1] * F.dim()
        shape[na] = self.n
        d += left.unsqueeze(na) * self.xl.view(shape)
        d -= right.unsqueeze(na) * self.xr.view(shape)
        return d

    def rhs(self, f, E):
        """On the interior elements; f with ghost elements."""
        a, B = self.accel, self.bfield
        inner = f[:, :, 1:-1, :, 1:-1, :]
        u = self.u[1:-1]
        out = self._lift(inner, (u >= 0)[None, :, :, None, None], 0, 1)[1:-1]
        out *= (2.0 / self.dx[0]) * u[None, None, :, :, None, None]
        f = f[1:-1]
        su = a * (E[1:-1, :, None, None] + B * self.v[None, None])
        part = self._lift(f[..., 1:-1, :] * su[:, :, None, None, 1:-1, :], (su >= 0)[:, :, None, 1:-1, :], 2, 3)
        out += (2.0 / self.dx[1]) * part[:, :, 1:-1]
        sv = a * (-B * u)
        part = self._lift(f[:, :, 1:-1], (sv >= 0)[None, None, :, :, None], 4, 5)
        out += (2.0 / self.dx[2]) * sv[None, None, :, :, None, None] * part[..., 1:-1, :]
        return out

    def density(self, f):
        jw = self.w * (self.dx[1] / 2.0), self.w * (self.dx[2] / 2.0)
        inner = f[1:-1, :, 1:-1, :, 1:-1, :]
        return torch.einsum("j,k,eiajbk->ei", jw[0], jw[1], inner)

    def poisson(self, charge):
        c = (self.kappa * charge).reshape(-1).to(torch.complex128) @ self.T
        E = torch.real(self.Pk @ (1j * c / self.k)).reshape(self.res[0], self.n)
        phi = torch.real(self.Pk @ (-c / self.k ** 2)).reshape(self.res[0], self.n)
        return torch.cat([E[-1:], E, E[:1]]), phi

    def energy(self, E):
        return 0.5 * float((E[1:-1] ** 2 @ self.w).sum())

    def dt(self, E, courant):
        a, B = self.accel, self.bfield
        s = (self.umax, float((a * E).abs().max()) + abs(a * B * self.vmax), abs(a * B * self.umax))
        return courant / sum(v / d for v, d in zip(s, self.dx))

    def step(self, f, dt, courant):
        """One SSP-RK3 step of f in place; E and phi of the last solve, the next dt."""
        inner = (slice(1, -1), slice(None)) * 3
        f[0], f[-1] = f[-2], f[1]
        s = f.clone()
        for c0, c1, c2 in ((0.0, 1.0, 1.0), (3 / 4, 1 / 4, 1 / 4), (1 / 3, 2 / 3, 2 / 3)):
            rho = self.density(s)
            E, phi = self.poisson(rho.mean() - rho)
            r = self.rhs(s, E)
            s[inner] = c0 * f[inner] + c1 * s[inner] + (c2 * dt) * r
            s[0], s[-1] = s[-2], s[1]
        f[inner] = s[inner]
        return E, phi, self.dt(E, courant)


def _plain_of(p, n):
    return _Plain(tuple(int(r) for r in p.resolutions), n, [float(v) for v in p.lows], [float(v) for v in p.highs],
                  float(p.refs.electron_acceleration_multiplier), float(p.elliptic.magnetic_field),
                  float(p.elliptic.poisson_coefficient))


def _march(p, n, steps=None, final_time=None):
    """The problem's state advanced in 64 bits: the state (less the background of the split), E, phi,
    energies, times, the next dt."""
    z = _plain_of(p, n)
    f = _plain(p.f.arr).double()
    f0 = None
    if getattr(p.f, "background_split", False):
        f0 = torch.as_tensor(p.f.background, device="cuda")
        f += f0
    else:
        f = f.clone()
    courant = float(p.stepper.courant)
    dt, t, energies, times = z.dt(_plain(p.elliptic.electric_field).double(), courant), 0.0, [], []
    while len(times) < steps if final_time is None else t < final_time:
        E, phi, dt = z.step(f, dt, courant)
        t += dt
        energies.append(z.energy(E))
        times.append(t)
    return (f if f0 is None else f - f0), E, phi, np.array(energies), np.array(times), dt


def _exact_train(case, seed):
    X, T, Xv, Tv = (t.double() for t in _train_inputs(case, seed))
    mlp = closure.MLP(seed=int(seed))
    w = [v.double().clone() for v in mlp.layer_views(mlp.master_w)]
    cut = np.cumsum([0] + [n for _, n in mlp.LAYERS])
    b = [mlp.master_b[cut[i]:cut[i + 1]].double().clone() for i in range(len(w))]
    params = [v.requires_grad_(True) for v in w + b]
    k = len(w)

    def net(x):
        for i in range(k - 1):
            x = torch.nn.functional.gelu(x @ params[i] + params[k + i])
        return (x @ params[k - 1] + params[2 * k - 1])[:, :closure.NOUT]

    m1, m2 = [torch.zeros_like(v) for v in params], [torch.zeros_like(v) for v in params]
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    batch = case["batch"]
    perm = torch.randperm(case["samples"], device="cuda", generator=g)
    total = max(case["samples"] // batch, 1)
    for s in range(total):
        idx = perm[s * batch:(s + 1) * batch]
        grads = torch.autograd.grad(((net(X[idx]) - T[idx]) ** 2).mean(), params)
        lr = 2e-3 * 0.5 * (1.0 + math.cos(math.pi * s / total))
        with torch.no_grad():
            for v, d, a, c in zip(params, grads, m1, m2):
                a.mul_(0.9).add_(d, alpha=0.1)
                c.mul_(0.999).addcmul_(d, d, value=0.001)
                v -= lr * (a / (1 - 0.9 ** (s + 1))) / ((c / (1 - 0.999 ** (s + 1))).sqrt() + 1e-8)
    with torch.no_grad():
        val = float(((net(Xv) - Tv) ** 2).mean())
        return {"w": torch.cat([v.reshape(-1) for v in params[:k]]), "b": torch.cat(params[k:]), "val": val}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "ens":
        probs = build_members(_members(case, seed), precision="fp32", seed=int(seed), batch_steps=case["steps"])
        got = [_march(p, int(p.orders[0]), steps=case["steps"]) for p in probs]
        return {"f": [g[0] for g in got], "energy": np.concatenate([g[3] for g in got])}
    p, n = _build(case, seed), case["n"]
    if kind in ("rhs", "field"):
        z = _plain_of(p, n)
        f = _plain(p.f.arr).double()
        if kind == "rhs":
            out = torch.zeros_like(f)
            out[1:-1, :, 1:-1, :, 1:-1, :] = z.rhs(f, _plain(p.elliptic.electric_field))
            return out
        rho = z.density(f)
        E, phi = z.poisson(rho - rho.mean())
        return {"rho": rho, "E": E, "phi": phi, "energy": torch.tensor(z.energy(E), dtype=torch.float64)}
    if kind == "loop":
        f, E, phi, energy, time, dt = _march(p, n, final_time=(case["steps"] - 0.5) * _initial_dt(p))
    else:
        f, E, phi, energy, time, dt = _march(p, n, steps=case["steps"])
    if kind == "step":
        return {"f": f, "E": E, "phi": phi, "dt": np.array([dt])}
    return {"f": f, "E": E, "phi": phi, "energy": energy, "time": time}
