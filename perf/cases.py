"""The work that programs built on this package have it do, as cases that can be timed.

Every kind goes through an entry point that such a program calls:

* ``rhs``          one mode-averaged right-hand side on device pointers (an integrator of the
                   caller's own): ``luna_b200_rhs_device``;
* ``solve``        one propagation in a gas-filled capillary: ``plan.solve_precon``;
* ``gnlse``        one propagation of an envelope with the GNLSE: ``plan.solve_precon``;
* ``scan``         a parameter scan as one batch, inputs in and saved spectra out:
                   ``plan.Batch``;
* ``radial_rhs``   one radially symmetric right-hand side on device pointers:
                   ``luna_b200_radial_rhs_device``;
* ``radial_solve`` one radially symmetric propagation: ``RadialPlan.solve``;
* ``modal_rhs``    one multimode right-hand side on device pointers:
                   ``luna_b200_modal_rhs_device``;
* ``predict``      surrogate queries: ``surrogate.predict``;
* ``train``        one training step of the surrogate ensemble: ``Ensemble.train_step``.

The propagations start at the step ``dz`` and are limited to it (``max_dt``, Luna.run's
max_dz): where the error estimate is far below the tolerance an unlimited controller follows
its rounding, and its results could not be compared.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import luna_b200_loader

luna_b200_loader.load()

from luna_b200 import _lib, fields, ionisation, modal, modal_plan, modes, physdata, plan, radial_plan, scan, surrogate  # noqa: E402
from luna_b200.grid import RealGrid  # noqa: E402
from luna_b200.interface import prop_capillary_args, prop_gnlse_args  # noqa: E402
from luna_b200.nonlinear import Kerr_field, PlasmaCumtrapz  # noqa: E402
from luna_b200.radial import prop_radial_args  # noqa: E402

PREC = {"fp64": _lib.PREC_FP64, "mixed": _lib.PREC_MIXED}


def listed():
    return [
        # the smallest call: helium in a 125 um fibre, 0.25 ps (the quick-start sizes), Kerr and
        # PPT plasma; a caller's own integrator makes it thousands of times
        dict(name="rhs_he", kind="rhs", gas="He", pressure=1.0, energy=120e-6, trange=0.25e-12, fill="constant"),
        # the same call on the longest grids of the scan family, with a Raman-active gas
        dict(name="rhs_h2_long", kind="rhs", gas="H2", pressure=1.0, energy=100e-6, trange=2e-12, fill="constant"),
        # the drop-in use: one capillary run (1 ps, 150 nm - 4 um) from host arrays to saved spectra
        dict(name="solve_ar", kind="solve", gas="Ar", pressure=1.0, energy=90e-6, trange=1e-12, flength=0.02, dz=5e-4),
        # the runs that set a scan's makespan: hydrogen on the 32768-point grid
        dict(name="solve_h2_long", kind="solve", gas="H2", pressure=1.0, energy=100e-6, trange=2e-12, flength=0.01,
             dz=5e-4),
        # supercontinuum in a nonlinear fibre (12.5 ps, 835 nm, 10 kW), envelope and Raman response
        dict(name="solve_gnlse", kind="gnlse", power=10e3, trange=12.5e-12, flength=0.006, dz=6e-5, raman=True),
        # the benchmark's parameter scan over the first centimetre, in the precision it is run in
        dict(name="scan_fp64", kind="scan", n=96, flength=0.01, dz=5e-4, precision="fp64"),
        # the same scan in mixed precision, as training data for the surrogate are generated
        dict(name="scan_mixed", kind="scan", n=48, flength=0.01, dz=5e-4, precision="mixed"),
        # free-space focusing at the benchmark's size, QDHT on the tensor cores
        dict(name="radial_rhs_mixed", kind="radial_rhs", Nr=256, trange=0.5e-12, precision="mixed"),
        # a small radial run in full precision (the size of the radial tests)
        dict(name="radial_solve", kind="radial_solve", Nr=64, trange=0.2e-12, energy=20e-6, flength=0.004, dz=2e-4),
        # the multimode benchmark: HE11 in a 13 um fibre, adaptive radial integral
        dict(name="modal_rhs", kind="modal_rhs", nmodes=1, plasma=False, trange=1e-12),
        # a screen of candidate parameters by the surrogate
        dict(name="predict", kind="predict", n=262144),
        # one training step at the batch size of the benchmark
        dict(name="train_step", kind="train", batch=4096),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["rhs", "rhs", "solve", "gnlse", "scan", "radial_rhs", "radial_solve", "modal_rhs", "predict", "train"])
    gas = rng.choice(["He", "Ar", "H2"])
    gp = dict(gas=gas, pressure=round(rng.uniform(0.5, 2.0), 3), energy=round(rng.uniform(50e-6, 90e-6 if gas == "Ar" else 150e-6), 8))
    if kind == "rhs":
        return dict(gp, kind=kind, trange=round(log(0.25e-12, 2e-12), 16), fill=rng.choice(["constant", "constant", "gradient"]))
    if kind == "solve":
        return dict(gp, kind=kind, trange=round(log(0.25e-12, 2e-12), 16), flength=round(rng.uniform(0.004, 0.01), 5), dz=5e-4)
    if kind == "gnlse":
        return dict(kind=kind, power=round(rng.uniform(2e3, 10e3), 1), trange=round(log(3e-12, 12.5e-12), 16),
                    flength=round(rng.uniform(0.002, 0.006), 6), dz=6e-5, raman=rng.random() < 0.7)
    if kind == "scan":
        return dict(kind=kind, n=rng.randint(12, 48), flength=round(rng.uniform(0.003, 0.01), 5), dz=5e-4,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "radial_rhs":
        prec = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, Nr=64 * rng.randint(1, 4) if prec == "mixed" else rng.randint(40, 200),
                    trange=round(log(0.2e-12, 0.5e-12), 16), precision=prec)
    if kind == "radial_solve":
        return dict(kind=kind, Nr=rng.randint(40, 90), trange=0.2e-12, energy=round(rng.uniform(10e-6, 20e-6), 8),
                    flength=round(rng.uniform(0.002, 0.004), 5), dz=2e-4)
    if kind == "modal_rhs":
        return dict(kind=kind, nmodes=rng.randint(1, 2), plasma=rng.random() < 0.5, trange=round(log(0.3e-12, 1e-12), 16))
    if kind == "predict":
        return dict(kind=kind, n=int(log(300, 262144)))
    return dict(kind=kind, batch=128 * rng.randint(4, 32))


# ----------------------------------------------------------------------------- problems
def _capillary(c, rng):
    L = c.get("flength", 0.05)
    p = c["pressure"] if c.get("fill", "constant") == "constant" else (2 * c["pressure"], 0.2 * c["pressure"])
    return prop_capillary_args(125e-6, L, c["gas"], p, λ0=800e-9, τfwhm=10e-15, energy=c["energy"] * rng.uniform(0.95, 1.05),
                               λlims=(150e-9, 4e-6), trange=c["trange"], ϕ=(rng.uniform(0, 6.28),), saveN=5)


def _gnlse(c, rng):
    return prop_gnlse_args(0.11, c["flength"], [0.0, 0.0, -11.83e-27, 8.1e-41], λ0=835e-9, τfwhm=50e-15,
                           power=c["power"] * rng.uniform(0.95, 1.05), pulseshape="sech", λlims=(500e-9, 2400e-9),
                           trange=c["trange"], raman=c["raman"], ϕ=(rng.uniform(0, 6.28),), saveN=5)


@functools.lru_cache(maxsize=None)
def _instances(n):
    """The first n of the benchmark's draws in He, Ar and H2 (the rate table of neon alone takes
    ten seconds of host set-up), with the energy limited where the gas would be fully ionised
    within the pulse: there one ulp decides which steps are accepted."""
    out = [p for p in scan.draw_instances(4 * n) if p["gas"] != "Ne"][:n]
    most = {"He": 3e18, "Ar": 0.6e18, "H2": 2e18}  # J/(s m^2)
    return [dict(p, energy=min(p["energy"], most[p["gas"]] * p["τfwhm"] * p["radius"] ** 2)) for p in out]


def _scan(c, rng):
    args = [dict(p, flength=c["flength"], energy=p["energy"] * rng.uniform(0.95, 1.05)) for p in _instances(c["n"])]
    return args, [scan.build_problem(p, saveN=5) for p in args]


def _radial(c, rng):
    # the benchmark's focused beam at its grid, or the tests' collimated one
    if c["kind"] == "radial_rhs":
        kw = dict(R=3e-3, trange=c["trange"], τfwhm=30e-15, energy=0.5e-3, w0=1e-3, focal_length=1.0, pressure=1.0)
    else:
        kw = dict(R=1e-3, trange=c["trange"], τfwhm=20e-15, energy=c["energy"], w0=40e-6, pressure=1.2)
    kw["energy"] *= rng.uniform(0.95, 1.05)
    p = prop_radial_args("Ar", N=c["Nr"], flength=c.get("flength", 2.0), λ0=800e-9, λlims=(400e-9, 2000e-9), saveN=5, **kw)
    p.Eω = p.Eω * np.exp(1j * rng.uniform(0, 6.28))
    return p


def _modal(c, rng):
    a, gas, pres, energy = (50e-6, "Ar", 1.0, 20e-6) if c["plasma"] else (13e-6, "Ar", 5.0, 1e-6)
    ms = tuple(modes.MarcatiliMode(a, gas, pres, n=1, m=m + 1, kind="HE", loss=False) for m in range(c["nmodes"]))
    grid = RealGrid(5e-2, 800e-9, (160e-9, 3000e-9), c["trange"])
    resp = [Kerr_field(physdata.gamma3_gas(gas))]
    if c["plasma"]:
        resp.append(PlasmaCumtrapz(grid.to, grid.to, ionisation.ionrate_PPTaccel(gas, 800e-9),
                                   physdata.ionisation_potential(gas)))
    E, t = modal.setup_modal(grid, physdata.density(gas, pres), resp,
                             fields.GaussField(800e-9, 30e-15, energy=energy * rng.uniform(0.95, 1.05)), ms, "y")
    E = E * np.exp(1j * rng.uniform(0, 6.28))
    for m in range(1, c["nmodes"]):
        E[:, m] = rng.uniform(0.2, 0.4) * E[:, 0]
    return grid, E, t


def _device(E):
    """A host field on the device as the C entry points take it (column-major, interleaved)."""
    return torch.from_numpy(np.ascontiguousarray(E.T).view(np.float64)).cuda()


def _vp(x):
    return ctypes.c_void_p(x.data_ptr())


def _surrogate(c, rng):
    """Inputs as the standardised features are distributed: uniform, the gas as indicators."""
    n = c["n"] if c["kind"] == "predict" else c["batch"]
    x = (rng.uniform(size=(n, surrogate.NFEAT)) - 0.5) * math.sqrt(12)
    gas = rng.integers(0, 4, n)
    for j in range(3):
        x[:, 5 + j] = ((gas == j + 1) - 0.25) / math.sqrt(0.1875)
    return x.astype(np.float32)


def prepare(case, seed):
    c, rng = case, np.random.default_rng([seed, 7])
    k = c["kind"]
    if k == "rhs":
        p = _capillary(c, rng)
        E = _device(p.Eω)
        return dict(kind=k, plan=plan.Plan.from_transform(p.transform), E=E, out=torch.zeros_like(E), z=0.01)
    if k in ("solve", "gnlse"):
        return dict(kind=k, p=_capillary(c, rng) if k == "solve" else _gnlse(c, rng), dz=c["dz"])
    if k == "scan":
        args, probs = _scan(c, rng)
        plans = [plan.Plan.from_transform(q.transform, PREC[c["precision"]]) for q in probs]
        b = plan.Batch(plans, 5, np.linspace(0.0, c["flength"], 5))
        b.set_priority([scan.schedule_priority(a, q) for a, q in zip(args, probs)])
        n = len(probs)
        # pinned, as a program that moves gigabytes of spectra keeps its buffers
        saves = [torch.zeros(5, len(q.Eω), dtype=torch.complex128, pin_memory=True).numpy() for q in probs]
        ys = [torch.zeros(len(q.Eω), dtype=torch.complex128, pin_memory=True).numpy() for q in probs]
        return dict(kind=k, b=b, inputs=([q.linop for q in probs], [q.Eω for q in probs], [0.0] * n, [c["dz"]] * n,
                                         [c["flength"]] * n, None, [c["dz"]] * n), saves=saves, ys=ys)
    if k == "radial_rhs":
        p = _radial(c, rng)
        E = _device(p.Eω)
        return dict(kind=k, plan=radial_plan.RadialPlan.from_transform(p.transform, PREC[c["precision"]]), E=E,
                    out=torch.zeros_like(E))
    if k == "radial_solve":
        p = _radial(c, rng)
        return dict(kind=k, p=p, plan=radial_plan.RadialPlan.from_transform(p.transform), dz=c["dz"], flength=c["flength"])
    if k == "modal_rhs":
        grid, E, t = _modal(c, rng)
        E = _device(E)
        return dict(kind=k, plan=modal_plan.ModalPlan.from_transform(t), E=E, out=torch.zeros_like(E))
    x = torch.from_numpy(_surrogate(c, rng)).cuda()
    model = surrogate.Ensemble(members=4, seed=11, batch=c.get("batch", 4096))
    if k == "predict":
        return dict(kind=k, model=model, x=x)
    T = torch.from_numpy(rng.standard_normal((c["batch"], surrogate.NOUT)).astype(np.float32)).cuda()
    return dict(kind=k, model=model, x=x, T=T)


def run(s):
    k = s["kind"]
    if k in ("rhs", "radial_rhs", "modal_rhs"):
        lib = _lib.load()
        f = {"rhs": lib.luna_b200_rhs_device, "radial_rhs": lib.luna_b200_radial_rhs_device,
             "modal_rhs": lib.luna_b200_modal_rhs_device}[k]
        _lib.check(f(s["plan"].handle, _vp(s["out"]), _vp(s["E"]), s.get("z", 0.0),
                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s["out"]
    if k in ("solve", "gnlse"):
        p = s["p"]
        r = plan.solve_precon(p.transform, p.linop, p.Eω, 0.0, s["dz"], p.grid.zmax, saveN=p.saveN, max_dt=s["dz"])
        return {"saves": r.Eω, "y": r.y}
    if k == "scan":
        b = s["b"]
        b.upload(*s["inputs"])
        b.run()
        saves, ys, _ = b.download(s["saves"], s["ys"])
        return {"saves": np.concatenate([x.ravel() for x in saves]), "y": np.concatenate(ys)}
    if k == "radial_solve":
        r = s["plan"].solve(s["p"].linop, s["p"].Eω, 0.0, s["dz"], s["flength"], saveN=5, max_dt=s["dz"])
        return {"saves": r.Eω, "y": r.y}
    m = s["model"]
    if k == "predict":
        mean, spread = surrogate.predict(m, s["x"])
        return {"mean": mean, "spread": spread}
    loss = m.train_step(s["x"], s["T"])
    return {"loss": loss, "gW": list(m.gW), "gb": list(m.gb), "W": list(m.W), "b": list(m.b)}


# ----------------------------------------------------------------------------- work
def _rhs_flops(No, raman=False, env=False):
    """Two real transforms (complex ones for an envelope) of No points, four of 2 No for a Raman
    response, and the responses per sample."""
    t = 2.5 * No * math.log2(No) * (2 if env else 1)
    return 2 * t + 49 * No + (2 * 2.5 * 2 * No * math.log2(2 * No) if raman else 0)


@functools.lru_cache(maxsize=None)
def _sizes(key):
    """(Nw, No) of a case's grid."""
    c = dict(key)
    rng = np.random.default_rng(0)
    if c["kind"] in ("rhs", "solve"):
        g = _capillary(dict(c, gas="H2", fill="constant"), rng).grid
    elif c["kind"] == "gnlse":
        g = _gnlse(c, rng).grid
    elif c["kind"] in ("radial_rhs", "radial_solve"):
        g = RealGrid(1.0, 800e-9, (400e-9, 2000e-9), c["trange"])
    else:
        g = RealGrid(5e-2, 800e-9, (160e-9, 3000e-9), c["trange"])
    return len(g.ω), g.No


def work(case):
    c = {q: v for q, v in case.items() if q != "name"}
    k = c["kind"]
    if k == "scan":
        byts = flops = 0
        for p in _instances(c["n"]):
            g = RealGrid(1.0, 800e-9, (p["λmin"], p["λmax"]), p["trange"])
            byts += 16 * len(g.ω) * 8
            flops += 6 * math.ceil(c["flength"] / c["dz"]) * _rhs_flops(g.No, p["gas"] == "H2")
        return {"bytes": byts, "flops": flops}
    if k in ("predict", "train"):
        W = list(zip(surrogate.WIDTHS[:-1], surrogate.WIDTHS[1:]))
        macs = sum(a * b for a, b in W)
        n = c["n"] if k == "predict" else c["batch"]
        if k == "predict":
            return {"bytes": n * (8 + surrogate.NOUT + 1) * 4 + 4 * macs * 2, "flops": 8.0 * macs * n}
        # forward, backward weights, backward data of all but the first layer; Adam reads and
        # writes the weights and both moments
        return {"bytes": n * (8 + surrogate.NOUT) * 4 + 4 * macs * 28,
                "flops": 8.0 * n * (3 * macs - W[0][0] * W[0][1])}
    Nw, No = _sizes(tuple(sorted(c.items())))
    if k == "rhs":
        return {"bytes": 48.0 * Nw, "flops": _rhs_flops(No, c["gas"] == "H2")}
    if k in ("solve", "gnlse"):
        raman = c["gas"] == "H2" if k == "solve" else c["raman"]
        return {"bytes": 16.0 * Nw * 8, "flops": 6 * math.ceil(c["flength"] / c["dz"]) * _rhs_flops(No, raman, k == "gnlse")}
    if k == "modal_rhs":  # at least the nine points of the first two levels
        return {"bytes": 32.0 * Nw * c["nmodes"], "flops": c["nmodes"] * 5.0 * No * math.log2(No) + 9 * 49 * No}
    Nr = c["Nr"]
    rhs = Nr * _rhs_flops(No) + 2 * 4.0 * Nw * Nr * Nr
    if k == "radial_rhs":
        return {"bytes": 48.0 * Nw * Nr, "flops": rhs}
    return {"bytes": 16.0 * Nw * Nr * 8, "flops": 6 * math.ceil(c["flength"] / c["dz"]) * rhs}


# ----------------------------------------------------------------------------- 64-bit values
EPS0, C0, E_RATIO = 8.854187817620389e-12, 299792458.0, 1.6021766208e-19 ** 2 / 9.10938356e-31


def _cumtrapz(y, dt):
    out = np.zeros_like(y)
    np.cumsum(0.5 * (y[:-1] + y[1:]) * dt, axis=0, out=out[1:])
    return out


def _rate(r, E):
    a, out = np.abs(E), np.zeros_like(E)
    if r.kind == "adk":
        m = a >= r.thr
        x = r.w_t_prefac * a[m]
        out[m] = r.w_p * r.cn_sq * (4 * r.w_p / x) ** (2 * r.nstar - 1) * np.exp(-4 / 3 * r.w_p / x)
        return out
    m = a >= r.x[0]
    x = a[m]
    i = np.clip(np.ceil((x - r.x[0]) / (r.x[-1] - r.x[0]) * (len(r.x) - 1)).astype(np.int64), 1, len(r.x) - 1)
    t, y1, y0, D1, D0 = (x - r.x[i - 1]) / (r.x[i] - r.x[i - 1]), r.y[i], r.y[i - 1], r.D[i], r.D[i - 1]
    out[m] = np.exp(y0 + D0 * t + (3 * (y1 - y0) - 2 * D0 - D1) * t ** 2 + (2 * (y0 - y1) + D0 + D1) * t ** 3)
    return out


def _polarisation(E, resp, rho):
    """The responses on samples E [n] or [n, columns]."""
    P = np.zeros_like(E)
    for r in resp:
        if r.kind == "kerr_field":
            P += rho * EPS0 * r.γ3 * E ** 3
        elif r.kind == "kerr_env":
            P += 0.75 * rho * EPS0 * r.γ3 * np.abs(E) ** 2 * E
        elif r.kind == "plasma":
            w = _rate(r.ratefunc, E)
            f = r.preionfrac + 1 - np.exp(-_cumtrapz(w, r.δt))
            J = _cumtrapz(f * E_RATIO * E, r.δt)
            nz = np.abs(E) > 0
            J[nz] += r.ionpot * w[nz] * (1 - f[nz]) / E[nz]
            P += rho * _cumtrapz(J, r.δt)
        else:  # Raman: convolution of E^2 (1/2 |E|^2 of an envelope) with the response
            q, n = r.r, len(E)
            h = q.w * sum(hp * np.exp(-q.tt / tau) for hp, tau in zip(q.hpres, q.tau2s(rho)))
            E2 = E ** 2 if r.kind == "raman_field" else 0.5 * np.abs(E) ** 2
            P += rho * E * np.fft.irfft(np.fft.rfft(h, 2 * n) * np.fft.rfft(E2, 2 * n) * q.dt, 2 * n)[:n]
    return P


def _to_time(g, Ew):
    if g.kind == "real":
        X = np.zeros((g.No // 2 + 1,) + Ew.shape[1:], dtype=complex)
        X[:len(Ew)] = Ew
        return np.fft.irfft(X, g.No, axis=0) * (g.No // 2) / (len(Ew) - 1)
    X, h = np.zeros(g.No, dtype=complex), len(Ew) // 2
    X[:h], X[g.No - h:] = Ew[:h], Ew[h:]
    return np.fft.ifft(X) * g.No / len(Ew)


def _to_freq(g, P, Nw):
    if g.kind == "real":
        return np.fft.rfft(P, axis=0)[:Nw] * (Nw - 1) / (g.No // 2)
    X, h = np.fft.fft(P), Nw // 2
    return np.concatenate([X[:h], X[g.No - h:]]) * Nw / g.No


def _mode_avg(t, Ew, z):
    g = t.grid
    zdep = hasattr(t, "densityfun")
    aeff, rho = (t.aefffun(z), t.densityfun(z)) if zdep else (t.aeff, t.density)
    E = _to_time(g, Ew) / math.sqrt(EPS0 * C0 / 2 * aeff)
    nl = _to_freq(g, _polarisation(E, t.resp, rho) * g.towin, len(Ew))
    s = g.sidx
    nl[s] *= t.norm_factor(z)[s] if zdep else t.norm.pre[s] * math.sqrt(aeff) * g.ωwin[s]
    return nl


def _radial_transform(t, Ew):
    g, q = t.grid, t.q
    E = _to_time(g, Ew) @ q.Mi.T
    P = (_polarisation(E, t.resp, t.density) * g.towin[:, None]) @ q.Mf.T
    return _to_freq(g, P, len(Ew)) * (g.ωwin * (-1j * g.ω))[:, None] / (2 * t.normfun)


def _modal_transform(t, Ew):
    """The radial integral of the projected polarisation by nested Clenshaw-Curtis rules, each
    compared with the one before."""
    g = t.grid
    ems, wts, wlow = t.tables()
    ems = np.asarray(ems).reshape(len(ems), -1)
    of = (g.ωwin * t.norm)[:, None]
    Et = _to_time(g, Ew)
    G, prev = [], None
    for level in range(len(wts)):
        for e in ems[len(G):(2 << level) - 1]:
            P = _polarisation(Et @ e, t.resp, t.density) * g.towin
            G.append(_to_freq(g, P, len(Ew))[:, None] * e[None, :] * of)
        if prev is None:
            prev = wlow * G[0]
        val = sum(w * x for w, x in zip(wts[level], G))
        err = np.linalg.norm(val - prev)
        if err <= t.atol or err <= t.rtol * np.linalg.norm(val):
            break
        prev = val
    return val


A = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
     [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
     [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
     [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
NODES = [1 / 5, 3 / 10, 4 / 5, 8 / 9, 1, 1]
B5 = [5179 / 57600, 0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40]
B4 = A[5] + [0]
DENSE = np.array([[1, 0, 0, 0, 0, 0, 0],
                  [-183 / 64, 0, 1500 / 371, -125 / 32, 9477 / 3392, -11 / 7, 3 / 2],
                  [37 / 12, 0, -1000 / 159, 125 / 12, -729 / 106, 11 / 3, -4],
                  [-145 / 128, 0, 1000 / 371, -375 / 64, 25515 / 6784, -55 / 28, 5 / 2]])


def _propagate(f, L, y, grid, zmax, dz, saveN, rtol=1e-6):
    """Dormand-Prince in the interaction picture with the PI controller, the window filter and
    the dense output at the save points."""
    col = (lambda v: v) if y.ndim == 1 else (lambda v: v[:, None])
    fwd, inv = ((np.fft.rfft, lambda Y: np.fft.irfft(Y, grid.N, axis=0)) if grid.kind == "real" else
                (np.fft.fft, lambda Y: np.fft.ifft(Y, axis=0)))
    z, dt, last, saves, zs = 0.0, dz, 0.0, [], np.linspace(0.0, zmax, saveN)
    k = [f(y)] + [None] * 6
    while z <= zmax:
        for i in range(6):
            p = np.exp(L * (NODES[i] * dt))
            k[i + 1] = f(p * (y + dt * sum(a * q for a, q in zip(A[i], k)))) / p
        yn = y + dt * sum(b * q for b, q in zip(B5, k))
        err = dt * np.linalg.norm(sum((b - a) * q for b, a, q in zip(B5, B4, k))) / rtol / max(
            np.linalg.norm(y), np.linalg.norm(yn))
        if err > 1:
            dt = min(dz, dt * max(0.1, 0.9 * err ** -0.2))
            continue
        p = np.exp(L * dt)
        yn = fwd(inv(yn * p * col(grid.ωwin)) * col(grid.twin), axis=0)
        while len(saves) < saveN and zs[len(saves)] <= z + dt:
            s = (zs[len(saves)] - z) / dt
            if s == 0 or zs[len(saves)] == z + dt:
                saves.append(yn if s else y)
                continue
            b = np.array([s, s ** 2, s ** 3, s ** 4]) @ DENSE
            kk = [k[6]] + k[1:]
            saves.append((y + dt * sum(bj * q for bj, q in zip(b, kk))) * np.exp(L * (s * dt)))
        z, y, k[0] = z + dt, yn, k[6] * p
        last = last or err
        dt, last = min(dz, dt * 0.9 * (0.8 / err) ** 0.12 * (0.8 / last) ** -0.04), err
    return {"saves": np.array(saves), "y": y}


def _network(model, x, T=None):
    """The ensemble's forward pass, and the gradients of the mean squared error, in 64 bits on
    the weights that the tensor cores are given."""
    x = x.double()
    F = model.fourier.double()
    a = 2 * math.pi * x @ F.T
    X0 = torch.cat([x, torch.sin(a), torch.cos(a)], dim=1)
    out, losses, gW, gb = [], [], [], []
    for z in range(model.members):
        W, b = [w[z].double() for w in model.Wb], [v[z].double() for v in model.b]
        X, Z = [X0], []
        for n, (w, v) in enumerate(zip(W, b)):
            Z.append(X[-1] @ w.T + v)
            X.append(Z[-1] * torch.sigmoid(Z[-1]) if n < len(W) - 1 else Z[-1])
        out.append(X[-1])
        if T is None:
            continue
        d = X[-1] - T.double()
        losses.append((d ** 2).mean())
        d = 2 * d / d.numel()
        g, h = [None] * len(W), [None] * len(W)
        for n in range(len(W) - 1, -1, -1):
            g[n], h[n] = d.T @ X[n], d.sum(0)
            if n:
                s = torch.sigmoid(Z[n - 1])
                d = (d @ W[n]) * (s * (1 + Z[n - 1] * (1 - s)))
        gW.append(g)
        gb.append(h)
    if T is None:
        return torch.stack(out)
    return torch.stack(losses), *([torch.stack([m[n] for m in q]) for n in range(len(gW[0]))] for q in (gW, gb))


def exact(case, seed):
    c, rng = case, np.random.default_rng([seed, 7])
    k = c["kind"]
    if k == "rhs":
        p = _capillary(c, rng)
        return _mode_avg(p.transform, p.Eω, 0.01).view(np.float64)
    if k in ("solve", "gnlse"):
        p = _capillary(c, rng) if k == "solve" else _gnlse(c, rng)
        return _propagate(lambda y: _mode_avg(p.transform, y, 0.0), p.linop, p.Eω, p.grid, p.grid.zmax, c["dz"], 5)
    if k == "scan":  # minutes of host time
        return None
    if k in ("radial_rhs", "radial_solve"):
        p = _radial(c, rng)
        if k == "radial_rhs":
            return np.ascontiguousarray(_radial_transform(p.transform, p.Eω).T).view(np.float64)
        return _propagate(lambda y: _radial_transform(p.transform, y), p.linop, p.Eω, p.grid, c["flength"], c["dz"], 5)
    if k == "modal_rhs":
        _, E, t = _modal(c, rng)
        return np.ascontiguousarray(_modal_transform(t, E).T).view(np.float64)
    s = prepare(case, seed)
    m = s["model"]
    if k == "predict":
        mean, spread = [], []
        for x in s["x"].split(16384):
            Y = _network(m, x)
            mean.append(Y.mean(0))
            spread.append(Y[:, :, :surrogate.NSPEC].std(dim=0, unbiased=False).amax(1))
        return {"mean": torch.cat(mean), "spread": torch.cat(spread)}
    loss, gW, gb = _network(m, s["x"], s["T"])

    def adam(p, g):  # the first step: the bias-corrected moments are g and g^2
        return p.double() - m.lr * g / (g.abs() + 1e-8)

    return {"loss": loss, "gW": gW, "gb": gb, "W": [adam(p, g) for p, g in zip(m.W, gW)],
            "b": [adam(p, g) for p, g in zip(m.b, gb)]}
