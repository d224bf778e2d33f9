"""Performance cases of the pseudo-time solver and of its learned warm start.

Each case is one call sequence that a user's program makes through the package's public entry
points:

* "routines": a driver that keeps its own loop calls solve_U, solve_V, solve_P, solve_Z, solve_C
  on host arrays, one pseudo-iteration per pass;
* "loop": a driver hands the state of one case or of a batch over, advances it by physical steps
  on the device and takes iteration counts, errors and fields back.  Steps are capped at `cap`
  pseudo-iterations (itc_max), far from their tolerance, so a pass has the same work every time;
* "forward" / "gradient": the warm start's network on a batch of canvases: inference, and one
  minibatch's loss and parameter gradients.

Sizes: 51 x 84 is the reference driver's mesh, 51 x 51, 102 x 102, 153 x 153, 1024 x 512 and the
mixed batch are the configurations of `configs.py`, 160 x 160 is the canvas of the shipped network.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.getcwd()


def _package():
    """The package directory `solver-cfd_b200`, imported as `solver_cfd_b200`."""
    name = "solver_cfd_b200"
    if name not in sys.modules:
        where = os.path.join(ROOT, "solver-cfd_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(where, "__init__.py"),
                                                      submodule_search_locations=[where])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# fields a driver hands over before a run, and those it takes back for output and restart files
STATE_IN = ("um", "vm", "um_tau", "vm_tau", "p", "pn", "T", "T_tau", "C", "C_tau")
STATE_OUT = ("um", "vm", "p", "T", "C")
SIZES_MIXED = (51, 102, 153, 204)


def _loop(name, flow, nx, ny, arith, engine, steps, cap, cases=1, mixed=False):
    return {"name": name, "kind": "loop", "flow": flow, "nx": nx, "ny": ny, "arith": arith, "engine": engine,
            "steps": steps, "cap": cap, "cases": cases, "mixed": mixed}


def listed():
    return [
        # the drop-in that changes nothing else in the driver: five routine calls on host arrays
        {"name": "routines_exact_51x84", "kind": "routines", "flow": "reference", "nx": 51, "ny": 84, "arith": "exact"},
        # the reference driver's own case through acs_physical_steps with every default (exact
        # arithmetic, cluster engine): about the pseudo-iterations of its mean physical step
        _loop("reference_exact_51x84", "reference", 51, 84, "exact", "cluster", 1, 1200),
        # plain method (upwind, no scalars): the smallest configuration, one case, default engine
        _loop("plain_fast_51x51", "plain", 51, 51, "fast", "cluster", 2, 500),
        # full equation set on one case, default engine, fast arithmetic
        _loop("full_fast_102x102", "full", 102, 102, "fast", "cluster", 2, 400),
        # the same physics where bit-identity with the driver is wanted: a small parameter study
        _loop("full_exact_8x153x153", "full", 153, 153, "exact", "cluster", 2, 100, cases=8),
        # the last cases of a batch still iterating: few cases on the tile engine, odd sizes
        _loop("tail_tile_3x101x147", "full", 101, 147, "fast", "tile", 2, 300, cases=3),
        # the benchmark's workload: 64 full-physics cases at 153 x 153
        _loop("batch_tile_64x153x153", "full", 153, 153, "fast", "tile", 2, 300, cases=64),
        # the batched configuration: 256 cases of mixed sizes
        _loop("batch_tile_256_mixed", "full", 204, 204, "fast", "tile", 2, 150, cases=256, mixed=True),
        # the combined configuration's single large case
        _loop("large_tile_1024x512", "large", 1024, 512, "fast", "tile", 2, 300),
        # the warm start's network between physical steps: one case, and the benchmark's 64 cases
        {"name": "forward_1x160x160", "kind": "forward", "batch": 1, "H": 160, "W": 160},
        {"name": "forward_64x160x160", "kind": "forward", "batch": 64, "H": 160, "W": 160},
        # its training: gradients of one minibatch of 16 snapshots
        {"name": "gradient_16x160x160", "kind": "gradient", "batch": 16, "H": 160, "W": 160},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges: sizes log-uniform, odd ones included."""
    kind = rng.choice(("loop", "loop", "loop", "loop", "loop", "routines", "forward", "gradient"))
    if kind == "routines":
        nx = _log_int(rng, 16, 120)
        return {"kind": kind, "flow": "reference", "nx": nx, "ny": _reference_jmax(nx), "arith": rng.choice(("exact", "exact", "fast"))}
    if kind in ("forward", "gradient"):
        H, W = 16 * rng.randint(2, 13), 32 * rng.randint(1, 6)  # the network takes 8-divisible pixel counts at all levels
        most = 64 if kind == "forward" else 16
        return {"kind": kind, "batch": max(1, min(most, _log_int(rng, 1, most))), "H": H, "W": W}
    flow = rng.choice(("reference", "plain", "full", "full"))
    arith = rng.choice(("exact", "fast", "fast"))
    engine = "cluster" if arith == "exact" else rng.choice(("cluster", "tile", "tile"))
    cases = rng.choice((1, 1, _log_int(rng, 2, 48)))
    nx = _log_int(rng, 20, 300 if cases > 1 else 700)
    ny = _reference_jmax(nx) if flow == "reference" else _log_int(rng, 20, 260 if cases > 1 else 500)
    # as many pseudo-iterations as keep a pass within the listed ones' cost
    cap = max(12, min(400, int(4.0e7 / (nx * ny * cases + 2.0e4))))
    return {"kind": "loop", "flow": flow, "nx": nx, "ny": ny, "arith": arith, "engine": engine,
            "steps": rng.choice((1, 2, 3)), "cap": cap, "cases": cases, "mixed": False}


def _reference_jmax(imax):
    return _package().reference_jmax(imax)


def _items(case, seed):
    """(params, mesh, state, itc) of every case of a workload, made from the seed."""
    pkg = _package()
    cfg = pkg.configs
    arith = pkg.ARITH_EXACT if case["arith"] == "exact" else pkg.ARITH_FAST
    kw = dict(arith=arith)
    if case.get("cap"):
        kw["itc_max"] = case["cap"]
    n = case.get("cases", 1)
    if case["flow"] == "reference":
        out = []
        for c in range(n):
            prm, mesh, st, itc, _ = cfg.reference_case(case["nx"], **kw)
            rng = np.random.default_rng([seed, c])
            for f in ("um", "vm"):  # a disturbed start: seeded noise of 1e-3 of the inflow
                st[f][2:-2, 2:-2] += 1.0e-3 * prm.v_in * rng.uniform(-1.0, 1.0, st[f][2:-2, 2:-2].shape)
                st[f + "_tau"][:] = st[f]
            out.append((prm, mesh, st, itc))
        return out
    if case["flow"] == "plain":
        return [cfg.channel_case(case["nx"], case["ny"], seed=seed, case_id=c, Re=100.0, scheme=pkg.SCHEME_UPWIND, **kw)
                for c in range(n)]
    if case["flow"] == "large":
        return [cfg.cfg_large(case["nx"], case["ny"], seed=seed, **kw)[:4]]
    out = []
    for c in range(n):
        q = cfg.batch_case_params(c, seed)
        nx, ny = case["nx"], case["ny"]
        if case["mixed"]:  # the sizes of the configuration's own cases, the physics from the seed
            size = cfg.batch_case_params(c, 0, SIZES_MIXED)
            nx, ny = size["nx"], size["ny"]
        out.append(cfg.channel_case(nx, ny, seed=seed, case_id=c, Re=q["Re"], scheme=pkg.SCHEME_QUICK,
                                    block=q["block"], porosity=q["porosity"], Da=q["Da"], Cf=0.55, Ri=q["Ri"],
                                    scalars=True, **kw))
    return out


def _net_inputs(case, seed, with_target):
    """Inputs as the warm start's features have them: 11 normalised channels per canvas node."""
    pkg = _package()
    ws = importlib.import_module(pkg.__name__ + ".warmstart")
    net, _, _, _, _ = ws.load(os.path.join(ROOT, "solver-cfd_b200", "unet", "weights", "ws_153.npz"))
    B, H, W = case["batch"], case["H"], case["W"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    st = {"net": net, "B": B, "H": H, "W": W,
          "x": torch.randn(B * H * W * net.cin, device="cuda", generator=g).to(torch.bfloat16)}
    if with_target:
        t = torch.randn(B * H * W, 8, device="cuda", generator=g)
        w = (torch.rand(B * H * W, 8, device="cuda", generator=g) < 0.9).float()
        t[:, net.cout:] = 0.0
        w[:, net.cout:] = 0.0
        st.update(t=t.reshape(-1), w=w.reshape(-1), inv=1.0 / float(w.sum()))
    return st


def prepare(case, seed):
    pkg = _package()
    if case["kind"] in ("forward", "gradient"):
        return {"kind": case["kind"], **_net_inputs(case, seed, case["kind"] == "gradient")}
    items = _items(case, seed)
    if case["kind"] == "routines":
        prm, mesh, st, _ = items[0]
        return {"kind": "routines", "case": pkg.Case(prm, mesh), "s": st}
    # host arrays in pinned memory, as a driver that moves them every step keeps them
    host, views_in, views_out = [], [], []
    out = {}
    for name, into in (("in", views_in), ("out", views_out)):
        for c in range(len(items)):
            into.append({})
        for f in (STATE_IN if name == "in" else STATE_OUT):
            shapes = [pkg.field_shape(f, x[0].imax, x[0].jmax) for x in items]
            flat = torch.zeros(sum(a * b for a, b in shapes), dtype=torch.float64, pin_memory=True).numpy()
            host.append(flat)
            o = 0
            for c, (a, b) in enumerate(shapes):
                v = flat[o:o + a * b].reshape((a, b), order="F")
                if name == "in":
                    v[:] = items[c][2][f]
                into[c][f] = v
                o += a * b
            if name == "out":
                out[f] = flat
    batch = pkg.Batch([x[0] for x in items], [x[1] for x in items])
    batch.set_option(pkg.OPT_ENGINE, {"cluster": pkg.ENGINE_CLUSTER, "graph": pkg.ENGINE_GRAPH,
                                      "tile": pkg.ENGINE_TILE}[case["engine"]])
    return {"kind": "loop", "batch": batch, "itc": np.array([x[3] for x in items], np.int32), "steps": case["steps"],
            "in": views_in, "out": views_out, "flat": out, "host": host}


def run(state):
    if state["kind"] == "forward":
        return state["net"].forward(state["B"], state["H"], state["W"], state["x"])
    if state["kind"] == "gradient":
        net = state["net"]
        y = net.forward(state["B"], state["H"], state["W"], state["x"])
        loss = net.loss(state["t"], state["w"], state["inv"])
        net.backward()
        return {"y": y, "loss": loss, "grad": net.grad}
    if state["kind"] == "routines":
        c, s = state["case"], state["s"]
        ru = c.solve_U(s["um"], s["vm"], None, s["um_tau"], s["vm_tau"], s["um_n_tau"], s["p"])
        rv = c.solve_V(s["um"], s["vm"], None, s["um_tau"], s["vm_tau"], s["vm_n_tau"], s["p"], s["T"])
        rp = c.solve_P(s["p"], s["um_n_tau"], s["vm_n_tau"], s["pn"])
        c.solve_Z(s["um_n_tau"], s["vm_n_tau"], s["T"], s["T_n_tau"], s["T_tau"])
        c.solve_C(s["um_n_tau"], s["vm_n_tau"], s["C"], s["C_n_tau"], s["C_tau"])
        return {"residuals": np.array([ru, rv, rp]), "um_n_tau": s["um_n_tau"], "vm_n_tau": s["vm_n_tau"],
                "pn": s["pn"], "T_n_tau": s["T_n_tau"], "C_n_tau": s["C_n_tau"]}
    b = state["batch"]
    for c, fields in enumerate(state["in"]):
        b.set_state(c, fields)
    itc, iters, err, status = b.run(state["steps"], state["itc"])
    for c in range(b.n):
        b.get_state(c, STATE_OUT, out=state["out"][c])
    return {"itc": itc, "iters": iters, "err": err, "status": status, **state["flat"]}


# ---- work ------------------------------------------------------------------------------------
# floating-point operations of one cell's pseudo-iteration: three stages of u and v (about 75 and
# 80 with QUICK, 55 each with upwind), p, three stages of two scalars at about 30
FLOPS_FULL, FLOPS_PLAIN = 650, 340


def _cells(case):
    if case.get("mixed"):
        cfg = _package().configs
        return sum(q["nx"] * q["ny"] for q in (cfg.batch_case_params(c, 0, SIZES_MIXED) for c in range(case["cases"])))
    return case["nx"] * case["ny"] * case.get("cases", 1)


def work(case):
    if case["kind"] in ("forward", "gradient"):
        un = importlib.import_module(_package().__name__ + ".unet")
        pix = case["batch"] * case["H"] * case["W"]
        flops = case["batch"] * un.conv_flops(case["H"], case["W"])
        if case["kind"] == "forward":
            return {"bytes": pix * (11 * 2 + 8 * 4) + 2 * 1.93e6, "flops": flops}
        return {"bytes": pix * (11 * 2 + 3 * 8 * 4) + 8 * 1.93e6, "flops": 3 * flops}
    n = _cells(case)
    scalars = case["flow"] != "plain"
    per = FLOPS_FULL if scalars else FLOPS_PLAIN
    if case["kind"] == "routines":
        return {"bytes": 8.0 * n * 22, "flops": float(per * n)}
    iters = case["steps"] * case["cap"]
    return {"bytes": 8.0 * n * (len(STATE_IN) + len(STATE_OUT)), "flops": float(per) * n * iters}


# ---- the same results in plain 64-bit torch --------------------------------------------------
class _Plain:
    """The discretisation on one case, as torch tensors [j, i] (0-based)."""

    def __init__(self, p, mesh, dev):
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.p, self.nx, self.ny = p, p.imax, p.jmax
        x, y, xm, ym = t(mesh["x"]), t(mesh["y"]), t(mesh["xm"]), t(mesh["ym"])
        self.dx, self.dy = (x[1:] - x[:-1])[None, :], (y[1:] - y[:-1])[:, None]      # [i] = x(i+2) - x(i+1), 1-based
        self.dxm, self.dym = (xm[1:] - xm[:-1])[None, :], (ym[1:] - ym[:-1])[:, None]
        self.eps, self.liga = t(mesh["eps"].T), t(mesh["liga"].T)

    @staticmethod
    def _adv(f, w2, w, e, e2, quick):
        """Value carried over a face by the flux f from the near and far nodes on both sides."""
        up = torch.where(f > 0, w, e)
        hi = torch.where(f > 0, 0.75 * w + 0.375 * e - 0.125 * w2, 0.75 * e + 0.375 * w - 0.125 * e2)
        return torch.where(quick, hi, up)

    def _convdiff(self, a, r0, r1, c0, c1, fw, fe, fs, fn, quick):
        z = torch.nn.functional.pad(a, (1, 1, 1, 1))
        n = lambda di, dj: z[r0 + dj + 1:r1 + dj + 1, c0 + di + 1:c1 + di + 1]
        P, W, E, S, N = n(0, 0), n(-1, 0), n(1, 0), n(0, -1), n(0, 1)
        adv = (fw * self._adv(fw, n(-2, 0), W, P, E, quick) - fe * self._adv(fe, W, P, E, n(2, 0), quick)
               + fs * self._adv(fs, n(0, -2), S, P, N, quick) - fn * self._adv(fn, S, P, N, n(0, 2), quick))
        return adv, P, W, E, S, N

    def ru(self, u, v, p):
        q, nx, ny = self.p, self.nx, self.ny
        r0, r1, c0, c1 = 1, ny - 1, 2, nx - 1
        e, lg = self.eps[r0:r1, c0:c1], self.liga[r0:r1, c0:c1]
        ax, ay = self.dx[:, c0 - 1:c1 - 1], self.dym[r0:r1]
        V = lambda di, dj: v[r0 + dj:r1 + dj, c0 + di:c1 + di]
        U = lambda di: u[r0:r1, c0 + di:c1 + di]
        fn, fs = 0.5 * (V(0, 1) + V(-1, 1)) * ax / e, 0.5 * (V(0, 0) + V(-1, 0)) * ax / e
        fe, fw = 0.5 * (U(1) + U(0)) * ay / e, 0.5 * (U(0) + U(-1)) * ay / e
        j = torch.arange(r0 + 1, r1 + 1, device=u.device)[:, None]
        quick = ((j >= 3) & (j <= ny - 2) & (q.scheme == 0)).expand_as(fn)
        adv, P, W, E, S, N = self._convdiff(u, r0, r1, c0, c1, fw, fe, fs, fn, quick)
        diff = e / q.Re * (ax * ((N - P) / self.dy[r0:r1] - (P - S) / self.dy[r0 - 1:r1 - 1])
                           + ay * ((E - P) / self.dxm[:, c0:c1] - (P - W) / self.dxm[:, c0 - 1:c1 - 1]))
        r = (adv + diff) / ax / self.dy[r0 - 1:r1 - 1] - e * (p[r0:r1, c0:c1] - p[r0:r1, c0 - 1:c1 - 1]) / ax
        vP = V(0, 0)
        drag = P / (q.Re * q.Da) + q.Cf / torch.sqrt(e * q.Da) * P * torch.sqrt(P * P + vP * vP)
        return r - e * drag * lg - q.g * e

    def rv(self, u, v, p, T):
        q, nx, ny = self.p, self.nx, self.ny
        r0, r1, c0, c1 = 2, ny - 1, 1, nx - 1
        e, lg = self.eps[r0:r1, c0:c1], self.liga[r0:r1, c0:c1]
        ax, ay = self.dxm[:, c0:c1], self.dy[r0 - 1:r1 - 1]
        U = lambda di, dj: u[r0 + dj:r1 + dj, c0 + di:c1 + di]
        V = lambda dj: v[r0 + dj:r1 + dj, c0:c1]
        fn, fs = 0.5 * (V(0) + V(1)) * ax / e, 0.5 * (V(0) + V(-1)) * ax / e
        fe, fw = 0.5 * (U(1, 0) + U(1, -1)) * ay / e, 0.5 * (U(0, 0) + U(0, -1)) * ay / e
        i = torch.arange(c0 + 1, c1 + 1, device=u.device)[None, :]
        quick = ((i >= 3) & (i <= nx - 2) & (q.scheme == 0)).expand_as(fn)
        adv, P, W, E, S, N = self._convdiff(v, r0, r1, c0, c1, fw, fe, fs, fn, quick)
        diff = e / q.Re * (ax * ((N - P) / self.dym[r0:r1] - (P - S) / self.dym[r0 - 1:r1 - 1])
                           + ay * ((E - P) / self.dx[:, c0:c1] - (P - W) / self.dx[:, c0 - 1:c1 - 1]))
        r = (adv + diff) / self.dx[:, c0 - 1:c1 - 1] / ay - e * (p[r0:r1, c0:c1] - p[r0 - 1:r1 - 1, c0:c1]) / ay
        if q.InvFr2 != 0.0:
            r = r + q.InvFr2 * (1.0 - 2.0 / (T[r0:r1, c0:c1] + T[r0 - 1:r1 - 1, c0:c1]))
        uP = U(0, 0)
        drag = P / (q.Re * q.Da) + q.Cf / torch.sqrt(e * q.Da) * P * torch.sqrt(uP * uP + P * P)
        return r - e * drag * lg

    def rs(self, u, v, z, is_c):
        q, nx, ny = self.p, self.nx, self.ny
        k = 1.0 / q.Re / q.Sc if is_c else 1.0 / q.Pe
        n = lambda di, dj: z[1 + dj:ny - 1 + dj, 1 + di:nx - 1 + di]
        P, E, W, N, S = n(0, 0), n(1, 0), n(-1, 0), n(0, 1), n(0, -1)
        ax, ay = self.dxm[:, 1:nx - 1], self.dym[1:ny - 1]
        conv = (0.5 * (E + P) * u[1:ny - 1, 2:nx] * ay - 0.5 * (W + P) * u[1:ny - 1, 1:nx - 1] * ay
                + 0.5 * (N + P) * v[2:ny, 1:nx - 1] * ax - 0.5 * (S + P) * v[1:ny - 1, 1:nx - 1] * ax)
        diff = k * (ay * ((E - P) / self.dx[:, 1:nx - 1] - (P - W) / self.dx[:, 0:nx - 2])
                    + ax * ((N - P) / self.dy[1:ny - 1] - (P - S) / self.dy[0:ny - 2]))
        lg, e = self.liga[1:ny - 1, 1:nx - 1], self.eps[1:ny - 1, 1:nx - 1]
        cap = lg * (e - 1.0) + 1.0
        return (diff - conv / cap) / ax / ay if is_c else (diff - (1.0 - lg) * conv) / cap / ax / ay

    def bc_u(self, u):
        if self.p.bc == 0:
            u[0, 1:-1] = 0.0
            u[-1, 1:-1] = u[-2, 1:-1]
            u[:, :2] = 0.0
            u[:, -2:] = 0.0
        else:
            u[:, :2] = self.p.v_in
            u[:, -2] = u[:, -3]
            u[:, -1] = u[:, -2]
            u[0] = -u[1]
            u[-1] = -u[-2]

    def bc_v(self, v):
        if self.p.bc == 0:
            v[:2] = self.p.v_in
            v[-2, 1:] = 2.0 * v[-4, 1:] - v[-3, 1:]
            v[-1, 1:] = 2.0 * v[-3, 1:] - v[-2, 1:]
            v[:, 0] = v[:, 1]
            v[1:-1, -1] = v[1:-1, -2]
        else:
            v[:, 0] = -v[:, 1]
            v[:, -1] = v[:, -2]
            v[1] = 0.0
            v[-2] = 0.0
            v[0] = -v[2]
            v[-1] = -v[-3]

    def bc_cell(self, z, zin=None):
        if self.p.bc == 0:
            z[0] = z[1] if zin is None else zin
            z[-1] = 2.0 * z[-2] - z[-3]
            z[:, 0] = z[:, 1]
            z[:, -1] = z[:, -2]
        else:
            z[:, 0] = z[:, 1] if zin is None else zin
            z[:, -1] = 2.0 * z[:, -2] - z[:, -3]
            z[0] = z[1]
            z[-1] = z[-2]

    def _rk3(self, phys, tau, rhs, bc, region):
        """Three stages of one unknown: (its new pseudo-iterate, max |increment| of the last stage)."""
        q = self.p
        s = tau
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            r = ((phys[region] - tau[region]) + rhs(s) * q.dt) * q.dtau
            new = s.clone()
            new[region] = a * tau[region] + b * (s[region] + r)
            bc(new)
            s = new
        return s, r.abs().max()

    # the boundary routine after each stage of one velocity also rewrites the other's tau array
    def solve_u(self, um, ut, vt, p):
        return self._rk3(um, ut, lambda s: self.ru(s, vt, p), lambda s: (self.bc_u(s), self.bc_v(vt)),
                         (slice(1, self.ny - 1), slice(2, self.nx - 1)))

    def solve_v(self, vm, ut, vt, p, T):
        return self._rk3(vm, vt, lambda s: self.rv(ut, s, p, T), lambda s: (self.bc_v(s), self.bc_u(ut)),
                         (slice(2, self.ny - 1), slice(1, self.nx - 1)))

    def solve_p(self, p, un, vn):
        q, ny, nx = self.p, self.ny, self.nx
        ax, ay = self.dxm[:, 1:nx - 1], self.dym[1:ny - 1]
        rp = -((un[1:ny - 1, 2:nx] - un[1:ny - 1, 1:nx - 1]) * ay + (vn[2:ny, 1:nx - 1] - vn[1:ny - 1, 1:nx - 1]) * ax)
        if q.continuity == 1:
            rp = rp / (ay * ax)
        r = q.dtau * rp * q.beta
        new = p.clone()
        new[1:ny - 1, 1:nx - 1] += r
        self.bc_cell(new)
        return new, r.abs().max()

    def solve_s(self, z, zt, un, vn, is_c):
        zin = self.p.C_in if is_c else self.p.T_in
        return self._rk3(z, zt, lambda s: self.rs(un, vn, s, is_c), lambda a: self.bc_cell(a, zin),
                         (slice(1, self.ny - 1), slice(1, self.nx - 1)))[0]

    def run(self, s, steps, itc):
        """The driver's loop; `s`: its state.  Returns (itc, iterations, errors)."""
        q = self.p
        iters, errs = [], []
        for _ in range(steps):
            k = 0
            while True:
                un, a = self.solve_u(s["um"], s["um_tau"], s["vm_tau"], s["pn"])
                vn, b = self.solve_v(s["vm"], s["um_tau"], s["vm_tau"], s["pn"], s["T"])
                pn, c = self.solve_p(s["p"], un, vn)
                new = {"um": un, "vm": vn}
                if q.solve_scalars:
                    new["T"] = self.solve_s(s["T"], s["T_tau"], un, vn, False)
                    new["C"] = self.solve_s(s["C"], s["C_tau"], un, vn, True)
                e = float(torch.stack((a, b, c)).max())
                k += 1
                s["pn"] = pn
                if itc != 1 and e < q.eps:
                    break
                for f, v in new.items():
                    s[f + "_tau"] = v
                s["p"] = pn
                itc += 1
                if itc >= q.itc_max:
                    break
            for f, v in new.items():
                s[f] = v.clone()
            itc = 0
            iters.append(k)
            errs.append(e)
        return itc, iters, errs


def _tensors(st, dev):
    return {k: torch.tensor(np.ascontiguousarray(a.T), dtype=torch.float64, device=dev) for k, a in st.items()}


def _flat(t):
    return t.cpu().numpy().reshape(-1)  # [j, i] row-major is the driver's column-major order


def _exact_net(case, seed):
    st = _net_inputs(case, seed, case["kind"] == "gradient")
    net, B, H, W = st["net"], st["B"], st["H"], st["W"]
    F = torch.nn.functional
    grad = case["kind"] == "gradient"
    # weights as the network computes with them: BF16 copies, biases in 32 bits
    flat = net.master.double()
    used = net.master.to(torch.bfloat16).double()
    for L in net.convs:
        used[L.off_b:L.off_b + L.cout] = flat[L.off_b:L.off_b + L.cout]
    used.requires_grad_(grad)

    def forward(x):
        def conv(name, t):
            L = net.by_name[name]
            w = used[L.off_w:L.off_w + L.kp * L.cout].view(L.kp, L.cout)[:9 * L.cin]
            w = w.reshape(3, 3, L.cin, L.cout).permute(3, 2, 0, 1)
            t = F.conv2d(t, w, used[L.off_b:L.off_b + L.cout], padding=1)
            return torch.relu(t) if L.relu else t

        skips, t = [], x
        for l in range(net.levels):
            t = conv(f"enc{l}b", conv(f"enc{l}a", t))
            if l + 1 < net.levels:
                skips.append(t)
                t = F.avg_pool2d(t, 2)
        for l in range(net.levels - 2, -1, -1):
            t = torch.cat([F.interpolate(t, scale_factor=2, mode="nearest"), skips[l]], dim=1)
            t = conv(f"dec{l}b", conv(f"dec{l}a", t))
        return conv("head", t).permute(0, 2, 3, 1)

    x = st["x"].double().view(B, H, W, net.cin).permute(0, 3, 1, 2)
    ys, loss = [], 0.0
    with torch.set_grad_enabled(grad):
        for b in range(B):  # one canvas at a time: 64-bit activations of a whole batch are large
            y = forward(x[b:b + 1])
            ys.append(y.detach().reshape(-1))
            if grad:
                n = H * W * 8
                t, w = st["t"][b * n:(b + 1) * n].double(), st["w"][b * n:(b + 1) * n].double()
                part = (w * (y.reshape(-1) - t) ** 2).sum() * st["inv"]
                part.backward()
                loss += float(part)
    y = torch.cat(ys)
    return {"y": y, "loss": torch.tensor([loss], dtype=torch.float64), "grad": used.grad} if grad else y


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] in ("forward", "gradient"):
        if case["batch"] * case["H"] * case["W"] > 1_700_000:
            return None  # over the time allowed on one card in 64 bits
        return _exact_net(case, seed)
    # about 10 ms of small tensor operations per pseudo-iteration of one case
    if case["kind"] == "loop" and case["cases"] * case["steps"] * case["cap"] > 1300:
        return None
    done = []
    for prm, mesh, st, itc in _items(case, seed):
        done.append((_Plain(prm, mesh, dev), _tensors(st, dev), itc))
    if case["kind"] == "routines":
        c, s, _ = done[0]
        un, ru = c.solve_u(s["um"], s["um_tau"], s["vm_tau"], s["p"])
        vn, rv = c.solve_v(s["vm"], s["um_tau"], s["vm_tau"], s["p"], s["T"])
        pn, rp = c.solve_p(s["p"], un, vn)
        T, C = c.solve_s(s["T"], s["T_tau"], un, vn, False), c.solve_s(s["C"], s["C_tau"], un, vn, True)
        t = lambda a: a.cpu().numpy().T
        # vm(imax, jmax+1) keeps what was there before the boundary passes: no value of its own
        return {"residuals": np.array([float(ru), float(rv), float(rp)]), "um_n_tau": t(un), "vm_n_tau": None,
                "pn": t(pn), "T_n_tau": t(T), "C_n_tau": t(C)}
    got = [c.run(s, case["steps"], itc) for c, s, itc in done]
    out = {"itc": None, "iters": None, "status": None, "err": np.array([g[2] for g in got])}
    for f in STATE_OUT:
        out[f] = np.concatenate([_flat(s[f]) for _, s, _ in done])
    if case["flow"] == "reference":
        out["vm"] = None  # as above
    return out
