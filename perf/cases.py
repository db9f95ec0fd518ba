"""The work a user has this library do, as cases that can be timed.

Every case integrates a batch of independent systems through one of the public
entry points (``wind_b200.lib``): the drop-in ``cudaIntegrateSystem`` on
float32 host arrays, ``integrate`` on host arrays or on CUDA tensors,
``integrate_output_steps`` and ``integrate_batch``.  Networks, intervals and
tolerances are those of the repository's workloads (``wind_b200.networks``),
tests and benchmark:

* tolerance presets: ``loose`` 5e-3 / 5e-3 (the Katz96 runs of the tiling
  sweep), ``serve`` 1e-6 / 1e-4 (the serving requests), ``tight`` 1e-8 / 1e-6
  (the benchmark);
* solvers: ``gje_f64`` is the default of every entry point, ``auto`` what the
  benchmark and the serving loop ask for, ``lu_f64`` the plain FP64 path;
* controllers: ``device`` is the default, ``gold`` the benchmark's.

A case's fields: ``net`` (katz96, nr, tiles, mass, dense, batch), ``n_eq``
(species; for ``tiles`` the copies of Katz96 per system), ``nsys``, ``call``
(dropin, host, device, outputs, batch), ``method``, ``solver``,
``controller``, ``tol``, ``dt``, ``n_out``.
"""
import ctypes as C
import math

import numpy as np
import torch

from wind_b200 import lib, networks as W

TOL = {"loose": (5e-3, 5e-3), "serve": (1e-6, 1e-4), "tight": (1e-8, 1e-6)}


def _case(name, net, n_eq, nsys, call, tol, dt, solver="gje_f64", controller="device",
          method="sie", n_out=1):
    return dict(name=name, net=net, n_eq=n_eq, nsys=nsys, call=call, method=method, solver=solver,
                controller=controller, tol=tol, dt=dt, n_out=n_out)


def listed():
    return [
        # one cell of a chemistry grid through the drop-in: pure latency
        _case("katz96_one_cell", "katz96", 5, 1, "dropin", "loose", 1e10),
        # the reference's 20^3 cell grid, one call per output interval
        _case("katz96_grid_dropin", "katz96", 5, 8000, "dropin", "loose", 1e13),
        # 65,536 cells resident on the GPU at the benchmark's tolerances
        _case("katz96_cells_auto", "katz96", 5, 65536, "device", "tight", 1e13, "auto"),
        # explicit RK2 over a short interval, host arrays, an odd cell count
        _case("katz96_cells_rk2", "katz96", 5, 20011, "host", "serve", 1e6, method="rk2"),
        # the stiff linear test: 1024 systems, 100 stored output intervals
        _case("nr_outputs", "nr", 2, 1024, "outputs", "tight", 1.0, n_out=100),
        # the tiling sweep's 20 copies of Katz96 in one 100-equation system
        _case("katz96_tiles", "tiles", 20, 1000, "host", "loose", 1e13),
        # small reaction networks at the serving tolerances, host arrays
        _case("mass5_host_auto", "mass", 5, 3001, "host", "serve", 1e-4, "auto"),
        # the reference's own elimination (the default solver) at 16 species
        _case("mass16_default", "mass", 16, 1000, "device", "loose", 1e-3),
        # the benchmark's dense 32-species network over a short interval
        _case("dense32_auto", "dense", 32, 3000, "device", "serve", 1e-3, "auto", "gold"),
        # large networks, one CTA per system: two per SM, and one
        _case("mass64_auto", "mass", 64, 600, "device", "loose", 1e-3, "auto", "gold"),
        _case("mass157_auto", "mass", 157, 200, "device", "loose", 1e-3, "auto", "gold"),
        # the five size classes in their benchmark proportions, one call
        _case("mixed_sizes_batch", "batch", 0, 1000, "batch", "loose", 1e-3, "auto", "gold"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["katz96", "katz96", "rk2", "nr", "tiles", "mass", "mass", "dense", "large", "large", "batch"])
    ctrl = rng.choice(["device", "gold"])
    if kind == "katz96":
        call = rng.choice(["dropin", "host", "device"])
        solver = "gje_f64" if call == "dropin" else rng.choice(["gje_f64", "auto", "lu_f64"])
        tol = rng.choice(["loose", "serve"])
        return _drawn(net="katz96", n_eq=5, nsys=_log_int(rng, 1, 65536), call=call, tol=tol,
                      dt=rng.choice([1e10, 1e13]), solver=solver,
                      controller="device" if call == "dropin" else ctrl)
    if kind == "rk2":
        return _drawn(net="katz96", n_eq=5, nsys=_log_int(rng, 1, 65536), method="rk2",
                      call=rng.choice(["host", "device"]), tol=rng.choice(["loose", "serve"]), dt=1e6,
                      controller=ctrl)
    if kind == "nr":
        return _drawn(net="nr", n_eq=2, nsys=_log_int(rng, 1, 1024), call="outputs",
                      tol=rng.choice(["loose", "serve", "tight"]), dt=1.0, controller=ctrl,
                      solver=rng.choice(["gje_f64", "auto"]), n_out=_log_int(rng, 1, 100))
    if kind == "tiles":
        return _drawn(net="tiles", n_eq=_log_int(rng, 2, 50), nsys=_log_int(rng, 1, 400), call="host",
                      tol="loose", dt=rng.choice([1e10, 1e13]), controller=ctrl,
                      solver=rng.choice(["gje_f64", "auto"]))
    if kind == "mass":
        solver = rng.choice(["gje_f64", "auto", "auto"])
        n = rng.randint(3, 32)
        if solver == "gje_f64":
            return _drawn(net="mass", n_eq=n, nsys=_log_int(rng, 1, 1000), call=rng.choice(["host", "device"]),
                          tol="loose", dt=1e-3, solver=solver, controller=ctrl)
        return _drawn(net="mass", n_eq=n, nsys=_log_int(rng, 1, 2000), call=rng.choice(["host", "device"]),
                      tol=rng.choice(["loose", "serve"]), dt=1e-4, solver=solver, controller=ctrl)
    if kind == "dense":
        return _drawn(net="dense", n_eq=rng.randint(4, 32), nsys=_log_int(rng, 1, 2000), call="device",
                      tol=rng.choice(["loose", "serve"]), dt=1e-3, solver="auto", controller=ctrl)
    if kind == "large":
        n = _log_int(rng, 33, 200)
        most = int(150 * (157.0 / n) ** 2)
        return _drawn(net="mass", n_eq=n, nsys=_log_int(rng, 1, min(most, 1000)), call=rng.choice(["host", "device"]),
                      tol="loose", dt=rng.choice([1e-4, 1e-3]), solver=rng.choice(["auto", "auto", "lu_f64"]),
                      controller=ctrl)
    return _drawn(net="batch", n_eq=0, nsys=_log_int(rng, 20, 1000), call="batch", tol="loose",
                  dt=rng.choice([1e-4, 1e-3]), solver="auto", controller=ctrl)


def _drawn(**kw):
    c = _case("", kw.pop("net"), kw.pop("n_eq"), kw.pop("nsys"), kw.pop("call"), kw.pop("tol"), kw.pop("dt"), **kw)
    del c["name"]
    return c


# ---- inputs ----------------------------------------------------------------
def _log_uniform(rng, lo, hi, size):
    return np.exp(rng.uniform(np.log(lo), np.log(hi), size))


def _mass(rng, n, nsys):
    """A size class of the mixed-size batch: 10N two-body reactions."""
    return W.random_mass_action(rng, nsys, n, 10 * n, 1e-4, 1e4), rng.uniform(0.0, 1.0, (nsys, n))


def _inputs(case, seed):
    """[(network, y0)] of the case, made from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    net, n, nsys = case["net"], case["n_eq"], case["nsys"]
    if net in ("katz96", "tiles"):
        # temperature, density and UV field of the cells, hydrogen fully ionised
        k = W.katz96_rates(_log_uniform(rng, 1e2, 1e8, nsys), _log_uniform(rng, 1e-4, 1e4, nsys),
                           _log_uniform(rng, 1e-15, 1e-11, nsys))
        y0 = np.tile(np.array([0.0, 1.0, 0.0, W.Y_HELIUM, 0.0]), (nsys, 1))
        nw = W.Network(W.NET_KATZ96, 5, nsys, constants=np.ascontiguousarray(k))
        if net == "tiles":
            nw = W.tile_network(nw, n)
            y0 = np.ascontiguousarray(np.tile(y0, (1, n)))
        return [(nw, y0)]
    if net == "nr":
        return [(W.nr_test(nsys), rng.uniform(0.5, 1.5, (nsys, 2)))]
    if net == "dense":
        nw = W.random_mass_action(rng, nsys, n, 2 * n, 1e-3, 1e1)
        nw.linear = W.dense_linear(rng, nsys, n, 1e-2, 1e6)
        return [(nw, rng.uniform(0.0, 1.0, (nsys, n)))]
    if net == "mass":
        return [_mass(rng, n, nsys)]
    return [_mass(rng, m, c) for m, c in zip(W.MIXED_SIZES, W.mixed_counts(nsys)) if c > 0]


def prepare(case, seed):
    groups = _inputs(case, seed)
    atol, rtol = TOL[case["tol"]]
    nw, y0 = groups[0]
    s = {"case": case, "net": nw, "y0": y0, "atol": atol, "rtol": rtol}
    if case["call"] == "device":
        s["arrays"] = {k: torch.from_numpy(np.ascontiguousarray(getattr(nw, k))).cuda()
                       for k in ("constants", "rates", "species", "linear") if getattr(nw, k) is not None}
        s["y0"] = torch.from_numpy(np.ascontiguousarray(y0)).cuda()
        s["y"] = torch.empty_like(s["y0"])
    elif case["call"] == "dropin":
        s["fn"] = lib.legacy("katz96", case["method"])
        s["constants"] = np.ascontiguousarray(nw.constants.astype(np.float32))
        s["y0"] = np.ascontiguousarray(y0.astype(np.float32))
    elif case["call"] == "batch":
        s["workloads"] = [W.Workload(g, y, 0.0, case["dt"], atol, rtol) for g, y in groups]
    return s


# ---- one pass --------------------------------------------------------------
def run(s):
    c = s["case"]
    if c["call"] == "dropin":
        y = s["y0"].copy()
        total = s["fn"](0.0, c["dt"], 1, s["constants"].ctypes.data, y.ctypes.data, y.shape[0], y.shape[1],
                        s["atol"], s["rtol"])
        return {"y": y, "total": total}
    if c["call"] == "outputs":
        y = s["y0"].copy()
        out, steps = lib.integrate_output_steps(s["net"], y, 0.0, c["dt"], s["atol"], s["rtol"], c["n_out"],
                                                method=c["method"], solver=c["solver"],
                                                controller=c["controller"])
        return {"y": y, "out": out, "steps": steps}
    if c["call"] == "batch":
        got = lib.integrate_batch(s["workloads"], c["method"], c["solver"], c["controller"])
        return [{"y": y, "status": st, "nsteps": n} for y, st, n in got]
    if c["call"] == "device":
        y = s["y"]
        y.copy_(s["y0"])
        total, status, nsteps = lib.integrate(s["net"], y, 0.0, c["dt"], s["atol"], s["rtol"], c["method"],
                                              c["solver"], c["controller"], device_arrays=s["arrays"])
    else:
        y = s["y0"].copy()
        total, status, nsteps = lib.integrate(s["net"], y, 0.0, c["dt"], s["atol"], s["rtol"], c["method"],
                                              c["solver"], c["controller"])
    return {"y": y, "total": total, "status": status, "nsteps": nsteps}


# ---- work ------------------------------------------------------------------
# Mean substeps per system (the reference's counter) of each network and
# tolerance, measured with the CPU oracle on a few hundred systems.
_KATZ = {("sie", "loose"): 154, ("sie", "serve"): 4184, ("sie", "tight"): 18426,
         ("rk2", "loose"): 21, ("rk2", "serve"): 331, ("rk2", "tight"): 3936}
_NR = {"loose": 900, "serve": 32000, "tight": 275000}
_MASS = {("loose", 1e-3): ([3, 8, 16, 32, 64, 157], [336, 643, 826, 982, 1364, 1624]),
         ("loose", 1e-4): ([3, 8, 16, 32, 64, 157], [43, 103, 134, 191, 254, 274]),
         ("serve", 1e-4): ([3, 8, 16, 32], [5917, 10872, 14030, 18192])}
_DENSE = {"loose": ([8, 32], [1500, 2015]), "serve": ([8, 20, 32], [14727, 20101, 21569])}


def _substep_flops(n, react, lin, method):
    f = 5.0 * react + (2.0 * n * n if lin else 0.0)
    if method == "rk2":
        return f + 2.0 * n
    return 2.0 / 3.0 * n ** 3 + 4.0 * n * n + f + 8.0 * react


def work(case):
    net, nsys, tol = case["net"], case["nsys"], case["tol"]
    esz = 4 if case["call"] == "dropin" else 8
    if net in ("katz96", "tiles"):
        tiles = case["n_eq"] if net == "tiles" else 1
        per = 40.0 + 10.0 if case["method"] == "rk2" else 243.0
        return {"bytes": nsys * esz * (10.0 + 10.0 * tiles),
                "flops": nsys * tiles * per * _KATZ[case["method"], tol]}
    if net == "nr":
        return {"bytes": nsys * 8.0 * (4 + 2 + 2 * (case["n_out"] + 1)), "flops": nsys * 32.0 * _NR[tol]}
    if net == "batch":
        groups = list(zip(W.MIXED_SIZES, W.mixed_counts(nsys)))
    else:
        groups = [(case["n_eq"], nsys)]
    b = f = 0.0
    for n, cnt in groups:
        lin = net == "dense"
        react = 2 * n if lin else 10 * n
        steps = np.interp(n, *(_DENSE[tol] if lin else _MASS[tol, case["dt"]]))
        b += cnt * (16.0 * n + 16.0 * react + (4.0 * n * n if lin else 0.0) + 12.0)
        f += cnt * steps * _substep_flops(n, react, lin, case["method"])
    return {"bytes": b, "flops": f}


# ---- the same results from plain torch in 64 bits --------------------------
def _katz_rhs_jac(k, y, want_jac=True):
    """f [S,T,5] and J[s,t,j,i] = d f_j / d y_i of Katz96 tiles; the electron
    density is tile 0's and the helium Jacobian keeps the reference's sign."""
    ne = (y[:, :1, 1] + y[:, :1, 3] + 2.0 * y[:, :1, 4])
    c = [k[:, i:i + 1] for i in range(10)]
    h0, hp, he0, hep, hepp = (y[:, :, i] for i in range(5))
    ih, ia, ib, r1, r2 = c[0] * ne + c[1], c[3] * ne + c[4], c[5] * ne + c[6], (c[7] + c[8]) * ne, c[9] * ne
    rh = c[2] * ne
    a, b, d, e = rh * hp - ih * h0, r1 * hep - ia * he0, ib * hep - r2 * hepp, None
    f = torch.stack([a, -a, b, -b - d, d], -1)
    if not want_jac:
        return f, None
    J = y.new_zeros(y.shape[0], y.shape[1], 5, 5)
    for j, i, v in ((0, 0, -ih), (1, 0, ih), (1, 1, -rh), (0, 1, rh), (2, 2, -ia), (3, 2, -ia),
                    (4, 3, ib), (2, 3, r1), (3, 3, -r1 - ib), (4, 4, -r2), (3, 4, r2)):
        J[:, :, j, i] = v
    return f, J


def _model(case, nw, dev):
    """rhs_jac(index, y [S,T,n]) of the network, T independent blocks of n."""
    if nw.kind == W.NET_KATZ96:
        c32 = nw.constants.astype(np.float32).astype(np.float64) if case["call"] == "dropin" else nw.constants
        k = torch.from_numpy(c32).to(dev)
        return nw.ntile, 5, lambda ix, y, jac: _katz_rhs_jac(k[ix], y, jac)
    if nw.kind == W.NET_NR_TEST:
        A = torch.from_numpy(nw.constants.reshape(-1, 2, 2).copy()).to(dev)
        return 1, 2, lambda ix, y, jac: ((A[ix][:, None] @ y[..., None])[..., 0], A[ix][:, None])
    n = nw.n_eq
    rates = torch.from_numpy(nw.rates).to(dev)
    sp = torch.from_numpy(nw.species.astype(np.int64)).to(dev)
    L = None if nw.linear is None else torch.from_numpy(nw.linear.astype(np.float64)).to(dev)
    sign = (-1.0, -1.0, 1.0, 1.0)

    def fn(ix, y, jac):
        v, q, k = y[:, 0], sp[ix], rates[ix]
        ya, yb = v.gather(1, q[:, :, 0]), v.gather(1, q[:, :, 1])
        f = v.new_zeros(v.shape) if L is None else (L[ix] @ v[..., None])[..., 0]
        J = None
        if jac:
            J = v.new_zeros(v.shape[0], n * n) if L is None else L[ix].reshape(-1, n * n).clone()
        for t in range(4):
            f = f.scatter_add(1, q[:, :, t], sign[t] * k * ya * yb)
            if jac:
                J.scatter_add_(1, q[:, :, t] * n + q[:, :, 0], sign[t] * k * yb)
                J.scatter_add_(1, q[:, :, t] * n + q[:, :, 1], sign[t] * k * ya)
        return f[:, None], None if J is None else J.view(-1, 1, n, n)
    return 1, n, fn


def _exact_group(case, nw, y0, t0, t1, atol, rtol, dev):
    """Step doubling with the reference's controllers, every system at its own
    pace: one loop turn is one attempt of each unfinished system."""
    tiles, n, fn = _model(case, nw, dev)
    gold, rk2 = case["controller"] == "gold", case["method"] == "rk2"
    cap = 20 if rk2 and not gold else 10
    y = y0.reshape(-1, tiles, n).clone()
    out = y.clone()
    ix = torch.arange(y.shape[0], device=dev)
    t = torch.full((y.shape[0],), t0, dtype=torch.float64, device=dev)
    h = torch.full_like(t, t1 - t0)
    bad = torch.zeros_like(ix)
    eye = torch.eye(n, dtype=torch.float64, device=dev)

    def substep(ix, v, h):
        f, J = fn(ix, v, not rk2)
        hh = h[:, None, None]
        if rk2:
            return v + hh * f
        x = torch.linalg.solve_ex(eye - hh[..., None] * J, f[..., None])[0][..., 0]
        return v + hh * x

    while ix.numel():
        h = torch.minimum(t1 - t, h)
        te = t + h
        full, half = te - t, (te - t) * 0.5
        y1 = substep(ix, y, full)
        y2 = substep(ix, y, half)
        y2 = substep(ix, y2, half if gold else torch.minimum(te - (t + half), half))
        d = (y2 - y1).abs()
        den = 2.0 * y2 - y1 + 1e-12 if rk2 else y2 + 1e-12
        re, big = (d / den).abs(), (y1.abs() > atol) & (y2.abs() > atol)
        e = ((d >= atol) | ((re >= rtol) & big)) if gold else ((d > atol) | ((re > rtol) & big))
        take = ~(e.flatten(1).any(1) & (bad < cap))
        y = torch.where(take[:, None, None], 2.0 * y2 - y1 if rk2 else y2, y)
        stuck = take & (t + h == t)
        t = torch.where(take, t + h, t)
        h = torch.where(take, h * 2.0 if rk2 else t1 - t, h / 2.0)
        bad = torch.where(take, torch.zeros_like(bad), bad + 1)
        done = ~(t < t1) | stuck
        if bool(done.any()):
            out[ix[done]] = y[done]
            keep = ~done
            ix, y, t, h, bad = ix[keep], y[keep], t[keep], h[keep], bad[keep]
    return out.reshape(y0.shape)


def exact(case, seed):
    # attempts of the slowest system bound the time: tens of thousands at the
    # tighter tolerances of the implicit method
    if case["method"] == "sie" and case["tol"] != "loose":
        return None
    if case["net"] in ("mass", "batch") and case["n_eq"] * case["nsys"] > 45000:
        return None
    dev = torch.device("cuda", torch.cuda.current_device())
    atol, rtol = TOL[case["tol"]]
    if case["call"] == "dropin":
        atol, rtol = (C.c_float(v).value for v in (atol, rtol))
        t1 = C.c_float(case["dt"]).value
    else:
        t1 = case["dt"]
    got = []
    for nw, y0 in _inputs(case, seed):
        if case["call"] == "dropin":
            y0 = y0.astype(np.float32).astype(np.float64)
        y = torch.from_numpy(np.ascontiguousarray(y0)).to(dev)
        if case["call"] == "outputs":
            out, t, dt = [y], 0.0, t1 / case["n_out"]
            for _ in range(case["n_out"]):
                out.append(_exact_group(case, nw, out[-1], t, t + dt, atol, rtol, dev))
                t += dt
            return {"y": out[-1].cpu().numpy(), "out": torch.stack(out).cpu().numpy(), "steps": None}
        y = _exact_group(case, nw, y, 0.0, t1, atol, rtol, dev)
        got.append(y)
    if case["call"] == "batch":
        return [{"y": y.cpu().numpy(), "status": None, "nsteps": None} for y in got]
    if case["call"] == "dropin":
        return {"y": got[0].cpu().numpy(), "total": None}
    y = got[0] if case["call"] == "device" else got[0].cpu().numpy()
    return {"y": y, "total": None, "status": None, "nsteps": None}
