"""The work this library is measured on, through its public entry points.

Twelve listed cases cover the calls a chemistry host model makes, from a box model's 64 cells
to half a million resident cells; draw() gives more cases of the same ranges.

  host       per-cell host arrays in, one 600 s step, host states out (the reference driver's flow)
  wrf        WRF fields in, converted, one step, host states out
  resident   states kept on the GPU, several operator-split steps replayed as one CUDA graph
  pipeline   radm2_rosenbrock_host: page-locked host arrays, copies overlapped with the solve
  noalloc    radm2_rosenbrock_noalloc on the caller's device arrays
  mechanism  the batched Fun / Jac / Decomp + Solve calls on host arrays
  gradients  loss and gradient of the step-seeding network on one batch

Every pass starts from the same inputs, so a pass can be repeated.  exact() restates the method
in 64-bit torch (dense LU with pivoting) from the mechanism tables.
"""
import ctypes
import json
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "radm2-solver-multi-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
from radm2b200 import inputs, lib, seeding  # noqa: E402

DT = 600.0
SCHEDULES = {"static": lib.SCHED_STATIC, "persistent": lib.SCHED_PERSISTENT}
PLACEMENTS = {"global": lib.PLACE_GLOBAL, "tmem": lib.PLACE_LU_TMEM, "tmem-wide": lib.PLACE_LU_TMEM_WIDE}
DEFAULTS = {"workload": "plain", "night": 0.0, "rtol": 1.0e-3, "atol": 1.0, "schedule": "static", "placement": "global",
            "block": 0, "fp32lu": False, "parity": False, "learned": False, "nsplit": 1, "spinup": 0, "nchunk": 8}


def _case(kind, n, **more):
    c = dict(DEFAULTS, kind=kind, n=n)
    c.update(more)
    return c


def listed():
    wide = {"workload": "mixed", "night": 0.4, "schedule": "persistent", "placement": "tmem-wide", "block": 128, "learned": True}
    cases = {
        # A box model or a short column: the smallest call, bound by one cell's chain of steps.
        "box-64": _case("host", 64),
        # The reference workload: 4,096 independent cells, one step, library defaults.
        "plain-4k": _case("host", 4096),
        # The reference's own WRF domain (39 x 19 x 39 window): conversion, rates, integration, states back.
        "wrf-domain": _case("wrf", 28899),
        # One simulated hour of a medium resident batch, persistent schedule, default launch shape.
        "hour-64k": _case("resident", 65536, night=0.3, schedule="persistent", nsplit=6),
        # The headline method (learned seeding, the autotuner's launch shape) from a cold start.
        "mixed-256k": _case("resident", 262144, nsplit=4, **wide),
        # The same method in a running model: states already spun up, few steps per cell; ragged size.
        "later-500k": _case("resident", 500009, nsplit=2, spinup=6, **wide),
        # End to end from page-locked host arrays, chunked; ragged size.
        "pipeline-200k": _case("pipeline", 200003, **wide),
        # Reference arithmetic (parity = 1): what a user validates against the reference with; ragged.
        "parity-8k": _case("host", 8191, workload="mixed", night=0.4, parity=True),
        # FP32 Jacobian and LU with one refinement sweep.
        "fp32lu-16k": _case("resident", 16384, schedule="persistent", fp32lu=True),
        # A host framework that may not allocate: the statically sized area; ragged.
        "noalloc-10k": _case("noalloc", 10007, night=0.3),
        # The reference's host wrappers Fun(), Jac(), Decomp(), Solve() on caller arrays.
        "mechanism-8k": _case("mechanism", 8192),
        # One training batch of the step-seeding network, forward and backward.
        "gradients-16k": _case("gradients", 16384),
    }
    return [dict(c, name=k) for k, c in cases.items()]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.5 else n))


def draw(rng):
    kind = rng.choice(["host", "host", "host", "wrf", "resident", "resident", "resident", "resident", "pipeline", "noalloc",
                       "mechanism", "gradients"])
    mixed = rng.random() < 0.5
    c = _case(kind, 0, workload="mixed" if mixed else "plain", night=0.4 if mixed else rng.choice([0.0, 0.3]))
    if kind == "host":
        c["n"] = _size(rng, 1, 16384)
        c["parity"] = rng.random() < 0.25
        c["rtol"] = rng.choice([1.0e-3, 1.0e-3, 1.0e-4])
        c["schedule"] = rng.choice(["static", "persistent"])
    elif kind == "wrf":
        c["n"] = _size(rng, 500, 28899)  # rounded to whole columns of 19 levels
        c["n"] = max(1, c["n"] // 19) * 19
    elif kind == "resident":
        c["schedule"] = rng.choice(["static", "persistent", "persistent"])
        c["block"] = rng.choice([0, 64, 128])
        c["nsplit"] = rng.randint(1, 4)
        c["spinup"] = rng.choice([0, 0, 3])
        c["n"] = _size(rng, 1024, 131072)
        if c["schedule"] == "persistent":
            c["learned"] = rng.random() < 0.5
            c["placement"] = rng.choice(["global", "tmem", "tmem-wide", "tmem-wide"])
        if c["placement"] != "global":
            c["block"] = 128 if c["placement"] == "tmem-wide" else rng.choice([128, 256])
        elif rng.random() < 0.2:
            c["fp32lu"], c["n"] = True, min(c["n"], 32768)
    elif kind == "pipeline":
        c["n"] = _size(rng, 4096, 131072)
        c["nchunk"] = rng.choice([4, 8])
        c["schedule"] = "persistent"
        if rng.random() < 0.7:
            c["placement"], c["block"], c["learned"] = "tmem-wide", 128, True
    elif kind == "noalloc":
        c["n"] = _size(rng, 32, 20000)
    elif kind == "mechanism":
        c["n"] = _size(rng, 64, 8192)
    else:
        c["n"] = _size(rng, 256, 16384)
    return c


# ---------------------------------------------------------------- inputs

_nets = {}


def _net():
    if "seed" not in _nets:
        _nets["seed"] = seeding.load_net(seeding.DEFAULT_NET)
    return _nets["seed"]


def _cells(c, seed):
    return inputs.make_cells(c["n"], seed, c["workload"], c["night"])


def _wrf_grid(c):
    """(ni, nk, nj, i0, k0, j0, wi, wk, wj): the reference's domain, or a strip of c["n"] / 19 columns of it."""
    if c["n"] == 28899:
        return (48, 20, 48, 4, 0, 4, 39, 19, 39)
    col = c["n"] // 19
    wi = min(39, col)
    while col % wi:
        wi -= 1
    wj = col // wi
    return (wi + 6, 20, wj + 4, 4, 0, 2, wi, 19, wj)


def _wrf_fields(c, seed):
    g = _wrf_grid(c)
    return inputs.make_wrf_fields(seed, g[0], g[1], g[2])


def _solver(c):
    return lib.Solver(precision=lib.PREC_FP32LU if c["fp32lu"] else lib.PREC_FP64, schedule=SCHEDULES[c["schedule"]],
                      block_threads=c["block"], placement=PLACEMENTS[c["placement"]], parity=1 if c["parity"] else 0)


def _tol(c):
    return np.full(lib.NVAR, c["atol"]), np.full(lib.NVAR, c["rtol"])


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def _mechanism_inputs(c, seed):
    """States, rate constants and a matrix 1/(h gamma) I - J with a right-hand side."""
    cells = _cells(c, seed)
    with lib.Solver() as s:
        s.set_cells(cells)
        rct = s.get_rconst()
        jac = s.jac(cells["VAR"], cells["FIX"], rct)
        rhs = s.fun(cells["VAR"], cells["FIX"], rct)
    g = -jac
    g[:, _tables()["diag"]] += 1.0 / (6.0 * 0.43586652150845899941601945119356)
    return cells, rct, g, rhs


def _batch(c, seed):
    r = np.random.RandomState(seed % (1 << 32))
    x = (r.randn(c["n"], lib.NFEAT) * 2.0 + 5.0).astype(np.float32)
    t = r.randn(c["n"], 2).astype(np.float32)
    p = (r.randn(lib.load().radm2_mlp_nparams()) * 0.08).astype(np.float32)
    norm = (np.full(lib.NFEAT, 5.0, np.float32), np.full(lib.NFEAT, 2.0, np.float32), np.zeros(2, np.float32), np.ones(2, np.float32))
    return x, t, p, norm


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    kind, n = c["kind"], c["n"]
    st = {"c": c, "tol": _tol(c)}
    if kind == "mechanism":
        cells, rct, g, rhs = _mechanism_inputs(c, seed)
        st.update(solver=lib.Solver(), V=cells["VAR"], FIX=cells["FIX"], RCT=rct, G=g, X=rhs)
    elif kind == "gradients":
        x, t, p, norm = _batch(c, seed)
        m = lib.Mlp(seed=0)
        m.set_params(p)
        m.set_norm(*norm)
        st.update(net=m, x=x, t=t)
    elif kind == "wrf":
        st.update(solver=_solver(c), fields=_wrf_fields(c, seed), grid=_wrf_grid(c), out=np.empty((n, lib.NVAR)))
    elif kind == "noalloc":
        cells = _cells(c, seed)
        dev = {k: torch.from_numpy(np.ascontiguousarray(cells[k].T)).cuda() for k in ("VAR", "FIX", "TEMP", "RC_N2O5", "JV")}
        st.update(dev=dev, var=torch.empty_like(dev["VAR"]), status=torch.empty(n, dtype=torch.int32, device="cuda"))
    elif kind == "pipeline":
        cells = _cells(c, seed)
        host = {k: _pinned(v) for k, v in cells.items() if k != "cls"}
        s = _solver(c)
        s.set_cells(cells)
        if c["learned"]:
            s.attach_mlp(_net())
        st.update(solver=s, host=host, var=torch.empty_like(host["VAR"]).pin_memory())
    else:
        cells = _cells(c, seed)
        s = _solver(c)
        st.update(solver=s)
        if kind == "host":
            st.update(cells=cells, out=np.empty((n, lib.NVAR)))
        else:
            s.set_cells(cells)
            if c["learned"]:
                s.attach_mlp(_net())
            if c["spinup"]:
                ipar, rpar = lib.default_params()
                s.run_split(c["spinup"], DT, *st["tol"], rpar, ipar)
            st.update(start=torch.empty((lib.NVAR, n), dtype=torch.float64, device="cuda"),
                      out=torch.empty((lib.NVAR, n), dtype=torch.float64, device="cuda"))
            torch.cuda.synchronize()
            s.get_state_device(st["start"].data_ptr(), n)
            s.synchronize()
    return st


# ---------------------------------------------------------------- one pass


def _result(state, ierr, ipar):
    # IPAR[10..16]: Nfun, Njac, Nstp, Nacc, Nrej, Ndec, Nsol
    return {"state": state, "ierr": int(ierr), "counters": np.array(ipar[10:17])}


def run(st):
    c = st["c"]
    kind, n, s = c["kind"], c["n"], st.get("solver")
    if kind == "mechanism":
        f = s.fun(st["V"], st["FIX"], st["RCT"])
        j = s.jac(st["V"], st["FIX"], st["RCT"])
        g, x, sing = s.decomp_solve(st["G"], st["X"])
        return {"fun": f, "jac": j, "lu": g, "x": x, "sing": sing}
    if kind == "gradients":
        g, loss = st["net"].gradients(st["x"], st["t"])
        return {"grad": g, "loss": np.float32(loss)}
    atol, rtol = st["tol"]
    if kind == "resident":
        ipar, rpar = lib.default_params()
        s.set_state_device(st["start"].data_ptr(), n)
        ierr = s.run_split(c["nsplit"], DT, atol, rtol, rpar, ipar)
        s.get_state_device(st["out"].data_ptr(), n)
        s.synchronize()
        return _result(st["out"], ierr, ipar)
    ipar, rpar = lib.default_params(hstart=0.01 * DT)
    if kind == "pipeline":
        h = {k: v.numpy() for k, v in st["host"].items()}
        st["var"].copy_(st["host"]["VAR"])
        ierr = s.rosenbrock_host(st["var"].numpy(), h["FIX"], h["TEMP"], h["RC_N2O5"], h["JV"], 0.0, DT, atol, rtol, rpar, ipar,
                                 nchunk=c["nchunk"])
        return _result(st["var"], ierr, ipar)
    if kind == "noalloc":
        d = st["dev"]
        st["var"].copy_(d["VAR"])
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
        ierr = lib.load().radm2_rosenbrock_noalloc(
            n, n, ptr(st["var"]), ptr(d["FIX"]), ptr(d["TEMP"]), ptr(d["RC_N2O5"]), ptr(d["JV"]), 0.0, DT, dp(atol), dp(rtol),
            dp(rpar), ipar.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), ptr(st["status"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return dict(_result(st["var"], ierr, ipar), status=st["status"])
    if kind == "wrf":
        s.convert_wrf(st["fields"], st["grid"])
    else:
        s.set_cells(st["cells"])
    ierr = s.rosenbrock(0.0, DT, atol, rtol, rpar, ipar)
    return _result(s.get_state(st["out"]), ierr, ipar)


# ---------------------------------------------------------------- what a pass cannot do without

FLOP_ATTEMPT, FLOP_FUN = 11197, 1085  # Jacobian, LU, three solves, stage-2 RHS, vector work; Fcn0 once per accepted step


def _attempts(c):
    """Step attempts per cell of one pass, as counted on these distributions: 84 (plain) or 78 (mixed) on the first
    600 s from the initial state, 67 with seeded first steps; 10, 6, 5, then 3 on later splits."""
    first = 67 if c["learned"] else 84 if c["workload"] == "plain" else 78
    per = [first, 10, 6, 5] + [3] * 16
    k = sum(per[c["spinup"]:c["spinup"] + c["nsplit"]])
    return k * (1.9 if c["rtol"] < 5.0e-4 else 1.0)


def work(case):
    c = dict(DEFAULTS, **case)
    n = c["n"]
    if c["kind"] == "mechanism":
        words = 2 * (59 + 2 + 156) + 59 + 659 + (659 + 59) * 2 + 0.5
        return {"bytes": 8 * words * n, "flops": (1085 + 1272 + 3588 + 1259) * n}
    if c["kind"] == "gradients":
        params = 84 * 128 + 2 * 128 * 128 + 128 * 2
        return {"bytes": 4 * (86 * n + 2 * params), "flops": 6 * params * n}
    words = (105 if c["kind"] == "wrf" else 59 + 2 + 1 + 1 + 28) + 59
    return {"bytes": 8 * words * n, "flops": _attempts(c) * (FLOP_ATTEMPT + FLOP_FUN) * n}


# ---------------------------------------------------------------- the same in 64-bit torch

_tab = {}


def _poly(t):
    """A tree of sums and products as {(sorted factor refs): coefficient}."""
    op = t[0]
    if op == "num":
        return {(): float(t[1])}
    if op == "ref":
        return {((t[1], t[2]),): 1.0}
    if op == "neg":
        return {k: -v for k, v in _poly(t[1]).items()}
    a, b = _poly(t[2]), _poly(t[3])
    out = {}
    if t[1] == "*":
        for k, v in a.items():
            for q, w in b.items():
                m = tuple(sorted(k + q))
                out[m] = out.get(m, 0.0) + v * w
        return out
    for p, sign in ((a, 1.0), (b, -1.0 if t[1] == "-" else 1.0)):
        for k, v in p.items():
            out[k] = out.get(k, 0.0) + sign * v
    return out


def _products(trees):
    """(rate constant index, coefficient, three factor indices) per product; factors index [V, F, 1]."""
    rc, co, fa = [], [], []
    for t in trees:
        (refs, v), = _poly(t).items()
        r = [i for kind, i in refs if kind == "RCT"]
        f = [i if kind == "V" else 59 + i for kind, i in refs if kind != "RCT"]
        rc.append(r[0])
        co.append(v)
        fa.append(f + [61] * (3 - len(f)))
    return torch.tensor(rc), torch.tensor(co, dtype=torch.float64), torch.tensor(fa)


def _sums(trees, index):
    m = torch.zeros(len(trees), len(index), dtype=torch.float64)
    for i, t in enumerate(trees):
        for refs, v in _poly(t).items():
            if refs:
                m[i, index[refs[0][1]]] += v
    return m


def _tables():
    if not _tab:
        with open(os.path.join(_PKG, "mech", "radm2_mech.json")) as f:
            m = json.load(f)
        _tab.update(diag=m["lu"]["diag"], rconst=m["rconst"], ros=m["ros3"],
                    row=torch.tensor(m["lu"]["irow"]), col=torch.tensor(m["lu"]["icol"]),
                    A=_products(m["rates"]), S=_sums(m["vdot"], {i: i for i in range(156)}),
                    B=_products(list(m["bvals"].values())),
                    J=_sums(m["jvs"], {int(k): i for i, k in enumerate(m["bvals"])}))
    return _tab


def _law(name, a):
    exp, pw = torch.exp, torch.pow
    if name == "exp":
        return exp(a[0])
    if name == "pow":
        return pw(torch.as_tensor(a[0], dtype=torch.float64), a[1])
    if name == "ARR2":  # a0 exp(-b0 / T)
        return a[0] * exp(-a[1] / a[2])
    if name == "THERMAL_T2":
        return a[2] ** 2 * a[0] * exp(-a[1] / a[2])
    if name in ("TROE", "TROEE"):
        pre = 1.0 if name == "TROE" else a[0] * exp(-a[1] / a[6])
        k0_300, n, kinf_300, m, temp, cair = a if name == "TROE" else a[2:]
        zt = 300.0 / temp
        k0, kinf = k0_300 * pw(zt, n) * cair, kinf_300 * pw(zt, m)
        r = k0 / kinf
        return pre * (k0 / (1.0 + r) * pw(torch.full_like(r, 0.6), 1.0 / (1.0 + torch.log10(r) ** 2)))
    if name == "k46":
        cair, temp = a
        k3 = 1.9e-33 * exp(725.0 / temp) * cair
        return 7.2e-15 * exp(785.0 / temp) + k3 / (1.0 + k3 / (4.1e-16 * exp(1440.0 / temp)))
    raise ValueError(name)


def _rates(cells):
    """RCONST[n][156] from the rate expressions."""
    T = cells["TEMP"]

    def ev(t):
        if t[0] == "num":
            return float(t[1])
        if t[0] == "ref":
            return cells["JV"][:, t[2]]
        if t[0] == "var":
            return {"TEMP": T, "C_M": cells["FIX"][:, 1], "rc_n2o5": cells["RC_N2O5"]}[t[1]]
        if t[0] == "neg":
            return -ev(t[1])
        if t[0] == "call":
            return _law(t[1], [ev(x) for x in t[2]])
        a, b = ev(t[2]), ev(t[3])
        return a * b if t[1] == "*" else a / b if t[1] == "/" else a + b if t[1] == "+" else a - b

    return torch.stack([torch.as_tensor(ev(t), dtype=torch.float64, device=T.device).expand_as(T) for t in _tables()["rconst"]], 1)


class _Method:
    """RHS, Jacobian and ROS-3 steps on a batch, in 64-bit torch."""

    def __init__(self, device):
        t = _tables()
        move = lambda v: tuple(x.to(device) for x in v) if isinstance(v, tuple) else v.to(device)  # noqa: E731
        self.A, self.B, self.S, self.J, self.row, self.col = (move(t[k]) for k in ("A", "B", "S", "J", "row", "col"))
        r = t["ros"]
        num = lambda k: [float(v) for v in r[k]]  # noqa: E731
        self.a, self.cc = num("ros_A"), num("ros_C")
        self.m, self.e = ([float(np.float32(v)) for v in num(k)] for k in ("ros_M", "ros_E"))
        self.gamma = num("ros_Gamma")[0]

    @staticmethod
    def _prod(tab, y, fix, rc):
        idx, co, fa = tab
        z = torch.cat([y, fix, torch.ones_like(y[:, :1])], 1)
        return rc[:, idx] * co * z[:, fa[:, 0]] * z[:, fa[:, 1]] * z[:, fa[:, 2]]

    def fun(self, y, fix, rc):
        return self._prod(self.A, y, fix, rc) @ self.S.T

    def jvs(self, y, fix, rc):
        return self._prod(self.B, y, fix, rc) @ self.J.T

    def dense(self, slots):
        g = torch.zeros(slots.shape[0], 59, 59, dtype=torch.float64, device=slots.device)
        g[:, self.row, self.col] = slots
        return g

    def integrate(self, y, fix, rc, hstart, atol, rtol):
        n, dev = y.shape[0], y.device
        out, live = y.clone(), torch.arange(n, device=dev)
        T = torch.zeros(n, dtype=torch.float64, device=dev)
        H = torch.full_like(T, min(hstart, DT))
        last = torch.zeros(n, dtype=torch.bool, device=dev)
        more, fresh = last.clone(), ~last
        eye = torch.eye(59, dtype=torch.float64, device=dev)
        f0 = torch.zeros_like(y)
        eps = 2.220446049250313e-16
        while live.numel():
            go = ~fresh | ((T - DT) + eps <= 0.0)
            if not bool(go.all()):
                out[live[~go]] = y[~go]
                live, y, fix, rc, T, H, last, more, fresh, f0 = (v[go] for v in (live, y, fix, rc, T, H, last, more, fresh, f0))
                if not live.numel():
                    break
            H = torch.where(fresh, torch.minimum(H, (DT - T).abs()), H)
            f0 = torch.where(fresh[:, None], self.fun(y, fix, rc), f0)
            lu, piv = torch.linalg.lu_factor(eye / (H * self.gamma)[:, None, None] - self.dense(self.jvs(y, fix, rc)))
            solve = lambda b: torch.linalg.lu_solve(lu, piv, b[:, :, None])[:, :, 0]  # noqa: E731
            h = H[:, None]
            k1 = solve(f0)
            f = self.fun(y + self.a[0] * k1, fix, rc)
            k2 = solve(f + k1 * (self.cc[0] / h))
            k3 = solve(f + k1 * (self.cc[1] / h) + k2 * (self.cc[2] / h))
            new = self.m[0] * k1 + self.m[1] * k2 + self.m[2] * k3 + y
            ye = self.e[0] * k1 + self.e[1] * k2 + self.e[2] * k3
            err = ((ye / (atol + rtol * torch.maximum(y.abs(), new.abs()))) ** 2).sum(1).div(59.0).sqrt()
            hn = H * torch.clamp(0.9 / err.pow(1.0 / 3.0), 0.2, 6.0)
            ok = err <= 1.0
            hn = torch.where(ok & last, torch.minimum(hn, H), hn)
            hn = torch.where(~ok & more, H * 0.1, hn)
            T = torch.where(ok, T + H, T)
            y = torch.where(ok[:, None], new, y)
            more, last, fresh, H = ~ok & last, ~ok, ok, hn
        return out


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _on_device(cells):
    return {k: torch.from_numpy(np.ascontiguousarray(v)).to(_device()) for k, v in cells.items() if k != "cls"}


def _exact_gradients(c, seed):
    x, t, p, norm = _batch(c, seed)
    dev = _device()
    w = torch.from_numpy(p).double().to(dev).requires_grad_()
    shapes = [(96, 128), (128,), (128, 128), (128,), (128, 128), (128,), (128, 8), (8,)]  # padded to 96 inputs, 8 outputs
    at, q = 0, []
    for s in shapes:
        k = int(np.prod(s))
        q.append(w[at:at + k].reshape(s))
        at += k
    h = torch.nn.functional.pad((torch.from_numpy(x).double().to(dev) - 5.0) / 2.0, (0, 12))
    for i in range(0, 6, 2):
        h = torch.nn.functional.gelu(h @ q[i] + q[i + 1])
    loss = (((h @ q[6] + q[7])[:, :2] - torch.from_numpy(t).double().to(dev)) ** 2).mean()
    loss.backward()
    return {"grad": w.grad, "loss": loss.detach()}


def exact(case, seed):
    c = dict(DEFAULTS, **case)
    if c["kind"] == "gradients":
        return _exact_gradients(c, seed)
    # a learned first step comes from a 16-bit network; large batches take too long
    if c["learned"] or c["n"] * c["nsplit"] > 17000 or c["spinup"]:
        return None
    m = _Method(_device())
    if c["kind"] == "mechanism":
        cells, rct, g, rhs = _mechanism_inputs(c, seed)
        V, F, R, G, X = (torch.from_numpy(v).to(_device()) for v in (cells["VAR"], cells["FIX"], rct, g, rhs))
        lu = m.dense(G)
        for k in range(58):  # pivot-free, as the fixed pattern needs
            lu[:, k + 1:, k] /= lu[:, k, k, None]
            lu[:, k + 1:, k + 1:] -= lu[:, k + 1:, k, None] * lu[:, k, None, k + 1:]
        return {"fun": m.fun(V, F, R), "jac": m.jvs(V, F, R), "lu": lu[:, m.row, m.col], "x": torch.linalg.solve(m.dense(G), X),
                "sing": None}
    if c["kind"] == "wrf":
        with lib.Solver() as s:  # the conversion's outputs are this path's inputs
            s.convert_wrf(_wrf_fields(c, seed), _wrf_grid(c))
            d = _on_device(s.get_inputs())
    else:
        d = _on_device(_cells(c, seed))
    y, rc = d["VAR"], _rates(d)
    for _ in range(c["nsplit"]):
        y = m.integrate(y, d["FIX"], rc, 0.01 * DT, c["atol"], c["rtol"])
    soa = c["kind"] in ("resident", "noalloc")
    out = {"state": y.T.contiguous() if soa else y, "ierr": None, "counters": None}
    return dict(out, status=None) if c["kind"] == "noalloc" else out
