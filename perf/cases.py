"""The work that users of this framework have it do, as timed cases.

Every case goes through the Python entry points a program calls: mcd.run for
one simulation, mcd.Batch (alone or captured in autotune.BatchGraph) for many,
stream.EventStream for every event of a run, adjoint.exit_histogram for
gradients, detector.project for EBSD images and tables.DeviceTable for the
sampled-loss tables of a new parameter set.  Sizes and parameters are those
of the benchmark's configurations, of the tests and of the driver.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mc-discrete_gb300"))

from mcd import _lib, adjoint, autotune, detector, engine, stream, tables  # noqa: E402

DEV = "cuda"
SPECIES = ("Al", "Si", "Cu", "Au")
PI_EFOUR = 6.51408491409531e-14   # cm^2 eV^2

# Z, density, atomic weight, valence electrons, Joy-Luo k and the outermost
# shell (binding energy, occupancy), with the number of shells
_DATA = {"Al": (13, 2.70, 26.98154, 3, 0.815, 73.5, 6, 3), "Si": (14, 2.33, 28.085, 4, 0.822, 100.0, 6, 3),
         "Cu": (29, 8.96, 63.546, 11, 0.83, 74.0, 6, 4), "Au": (79, 19.30, 196.967, 11, 0.851, 54.0, 4, 8)}


def listed():
    return [
        # the small parity run: FP64 transport of 1000 electrons with its
        # table, one blocking call (the plain Si 10 keV configuration)
        dict(name="run Si fp64 1k", kind="run", material="Si", E0=10e3, Emin=1e3, tilt=0.0, Wc=100.0, tol=1e-3,
             mode="DS", bethe="classical", n=1000, precision="fp64", tabulated=True, rows=True),
        # the smallest calls: a worker's job of a few electrons, as the
        # reference's pool hands them out, with its per-electron rows
        dict(name="run Au fp32 37", kind="run", material="Au", E0=20e3, Emin=1e3, tilt=45.0, Wc=100.0, tol=1e-3,
             mode="DS", bethe="classical", n=37, precision="fp32", tabulated=True, rows=True),
        # an ordinary FP32 run with its rows, every cross section evaluated
        # per event (mcd.run's defaults)
        dict(name="run Cu fp32 20k", kind="run", material="Cu", E0=20e3, Emin=1e3, tilt=45.0, Wc=100.0, tol=1e-3,
             mode="DS", bethe="classical", n=20011, precision="fp32", tabulated=False, rows=True),
        # the driver's chunk size: 1e5 electrons of Au at tight tolerance,
        # tables larger than L2, with rows
        dict(name="run Au fp32 100k", kind="run", material="Au", E0=30e3, Emin=500.0, tilt=70.0, Wc=50.0, tol=1e-4,
             mode="DS", bethe="classical", n=100000, precision="fp32", tabulated=True, rows=True),
        # the continuous-slowing-down histograms: 1e6 electrons, no rows
        dict(name="run Cu cont JL 1M", kind="run", material="Cu", E0=20e3, Emin=1e3, tilt=70.0, Wc=100.0, tol=1e-3,
             mode="cont", bethe="JL", n=1000000, precision="fp32", tabulated=False, rows=False),
        # the parameter study: 64 uneven simulations in one persistent,
        # graph-captured launch
        dict(name="batch 64 graph", kind="batch", mix="grid", sims=64, lo=3.0, hi=6.0, layout=0, graph=True, rows=False),
        # a few unlike simulations at once with rows and channel counts: a
        # diffracting film, other elastic models, continuous members
        dict(name="batch mixed 6 rows", kind="batch", mix="mixed", sims=6, lo=3.0, hi=4.7, layout=3, graph=False,
             rows=True),
        # every event of a run to the host through the device rings
        dict(name="stream Au 120k", kind="stream", material="Au", E0=30e3, Emin=500.0, tilt=70.0, Wc=50.0, tol=1e-4,
             n=120000, chunk=40000),
        # fitting J: soft exit-energy bins of 1e6 electrons and their gradient
        dict(name="adjoint exit 1M", kind="adjoint", material="Al", E0=15e3, Emin=1e3, tilt=70.0, bethe="classical",
             n=1000000, quantity="exit_E"),
        # ... and of the deepest z, whose density gradient does not vanish
        dict(name="adjoint depth 300k", kind="adjoint", material="Al", E0=15e3, Emin=1e3, tilt=70.0, bethe="classical",
             n=300001, quantity="max_depth"),
        # exit directions of a large run onto the detector; the number that
        # leaves the sample is any number, not a multiple of a vector
        dict(name="project 50M ragged", kind="project", n=50000003, dtype="float32"),
        # the sampled-loss tables of a new parameter set at tight tolerance
        dict(name="tables Au tol 1e-4", kind="tables", material="Au", E0=30e3, Emin=500.0, Wc=50.0, nE_m=20000,
             nW_m=500, nE_g=100000, nW_g=600),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "batch", "batch", "adjoint", "project", "tables", "stream"))
    mat = rng.choice(SPECIES)
    E0 = float(round(rng.uniform(5e3, 30e3)))
    tilt = float(round(rng.uniform(0.0, 75.0), 1))
    if kind == "run":
        cont = rng.random() < 0.35
        fp64 = rng.random() < 0.3
        c = dict(kind="run", material=mat, E0=E0, Emin=rng.choice((500.0, 1e3, 2e3)), tilt=tilt,
                 Wc=rng.choice((50.0, 100.0)), tol=1e-3, mode="cont" if cont else "DS",
                 bethe=rng.choice(("classical", "JL", "explicit")) if cont else "classical",
                 n=_log_int(rng, 4, 1e4 if fp64 else (1e6 if cont else 3e5)), precision="fp64" if fp64 else "fp32",
                 tabulated=not cont and rng.random() < 0.6, rows=rng.random() < 0.6)
        return c
    if kind == "batch":
        if rng.random() < 0.5:
            return dict(kind="batch", mix="grid", sims=rng.randint(2, 64), lo=2.0, hi=round(rng.uniform(3.0, 5.5), 2),
                        layout=rng.randint(1, 10 ** 6), graph=rng.random() < 0.5, rows=False)
        return dict(kind="batch", mix="mixed", sims=rng.randint(1, 6), lo=2.0, hi=round(rng.uniform(3.0, 5.0), 2),
                    layout=rng.randint(1, 10 ** 6), graph=False, rows=True)
    if kind == "adjoint":
        q = rng.choice(("exit_E", "max_depth"))
        return dict(kind="adjoint", material=mat, E0=E0, Emin=1e3, tilt=tilt, bethe=rng.choice(("classical", "JL")),
                    n=_log_int(rng, 3e4, 1e6 if q == "exit_E" else 5e5), quantity=q)
    if kind == "project":
        return dict(kind="project", n=_log_int(rng, 1e3, 5e7), dtype=rng.choice(("float32", "float32", "float64")))
    if kind == "tables":
        return dict(kind="tables", material=mat, E0=E0, Emin=1e3, Wc=100.0, nE_m=rng.choice((500, 1000, 2000)),
                    nW_m=rng.choice((80, 90, 200)), nE_g=_log_int(rng, 1000, 100000),
                    nW_g=rng.choice((100, 200, 300, 600)))
    n = _log_int(rng, 2e4, 1.2e5)
    return dict(kind="stream", material=mat, E0=E0, Emin=1e3, tilt=tilt, Wc=100.0, tol=1e-3, n=n,
                chunk=max(1, n // rng.randint(1, 4)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _input(c, n=None):
    return dict(material=c["material"], E0=c["E0"], Emin=c["Emin"], s_tilt=c["tilt"], Wc=c.get("Wc", 100.0),
                tol_E=c.get("tol", 1e-3), tol_W=c.get("tol", 1e-3), mode=c.get("mode", "DS"),
                Bethe_model=c.get("bethe", "classical"), num_el=int(c["n"] if n is None else n))


def _sims(c):
    rng = np.random.default_rng(int(c["layout"]))
    out = []
    if c["mix"] == "grid":
        for m in SPECIES:
            for E0 in (5e3, 10e3, 20e3, 30e3):
                for t in (0.0, 20.0, 45.0, 70.0):
                    n = int(round(10 ** rng.uniform(c["lo"], c["hi"])))
                    out.append(dict(material=m, E0=E0, Emin=1e3, s_tilt=t, Wc=100.0, tol_E=1e-3, tol_W=1e-3,
                                    mode="DS", num_el=n))
        if c["sims"] < len(out):
            out = [out[i] for i in sorted(rng.permutation(len(out))[:int(c["sims"])])]
        return out
    kinds = (dict(material="Si", E0=15e3, thickness=3000.0, diffMFP=True), dict(material="Au", E0=30e3, Emin=500.0),
             dict(material="Cu", E0=20e3, mode="cont", Bethe_model="JL"),
             dict(material="Al", E0=10e3, elastic="Ruth_nigram"), dict(material="Cu", E0=5e3, elastic="Ruth_nigram_wDefl"),
             dict(material="Al", E0=15e3, mode="cont", Bethe_model="explicit"))
    for k in range(int(c["sims"])):
        n = int(round(10 ** rng.uniform(c["lo"], c["hi"])))
        out.append(dict(dict(Emin=1e3, s_tilt=float(rng.choice((0.0, 45.0, 70.0))), Wc=100.0, tol_E=1e-3, tol_W=1e-3,
                             mode="DS", num_el=n), **kinds[k]))
    return out


def _directions(c, seed):
    """Unit vectors of electrons that leave through the surface (z < 0)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    d = torch.randn((3, c["n"]), generator=g, device=DEV, dtype=getattr(torch, c["dtype"]))
    d /= d.norm(dim=0, keepdim=True)
    d[2].abs_().neg_()
    return d


def _grids(c, seed):
    """The W and E grids of the Moller and outer-shell tables of a beam energy
    that the seed moves a little: the float32 spacings the grid search uses."""
    E0 = c["E0"] * (1.0 + 0.01 * np.random.default_rng(seed).random())
    Eb = _DATA[c["material"]][5]
    wmax = (E0 - _fermi(c["material"])) * 0.5
    lin = lambda n: np.linspace(c["Emin"], E0, num=n, dtype=np.float32)  # noqa: E731
    geo = lambda w, n: np.geomspace(w, wmax, num=n, dtype=np.float32)    # noqa: E731
    return (geo(c["Wc"], c["nW_m"]), lin(c["nE_m"])), (geo(Eb, c["nW_g"]), lin(c["nE_g"]))


FIELDS = _lib.EV_PATHL | _lib.EV_W | _lib.EV_C2 | _lib.EV_POS | _lib.EV_PACKED_HEAD


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "run":
        p = _input(c)
        if c["mode"] == "DS":   # built once per parameter set and kept by the package's cache
            tables.ds_tables(_lib.material(c["material"]), p["E0"], p["Emin"], p["Wc"], p["tol_E"], p["tol_W"], DEV)
        return dict(c, p=p, seed=seed)
    if kind == "batch":
        b = engine.Batch(_sims(c), seed=seed, device=DEV, tally_channels=c["rows"], electrons=c["rows"])
        # the shape the autotuner picks on the 64-simulation workload
        g = autotune.BatchGraph(b, _lib.Tune(576, 0, 1, 1, 0)) if c["graph"] else None
        return dict(c, batch=b, graph=g)
    if kind == "stream":
        s = stream.EventStream(_input(c), chunk=c["chunk"], seed=seed, device=DEV, fields=FIELDS,
                               events_per_electron=1000.0, piece_bytes=1 << 28)
        return dict(c, stream=s)
    if kind == "adjoint":
        depth = c["quantity"] == "max_depth"
        kw = dict(quantity="max_depth", lo=0.0, hi=20000.0, sigma=300.0) if depth else {}
        m = adjoint.ExitEnergyModel(dict(_input(c), mode="cont"), c["n"], seed=seed, device=DEV, **kw)
        t, _, _ = m.forward(1.1, 1.0)
        return dict(c, model=m, target=torch.from_numpy(t.copy()))
    if kind == "project":
        return dict(c, dirs=_directions(c, seed))
    m, g = _grids(c, seed)
    return dict(c, mat=_lib.material(c["material"]), moller=m, gryz=g)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "run":
        r = engine.run(s["p"], seed=s["seed"], precision=s["precision"], electrons=s["rows"],
                       tabulated=s["tabulated"], device=DEV)
        return {"tally": r.tally, "status": r.status, "rows": r.electrons}
    if kind == "batch":
        b = s["batch"]
        if s["graph"] is not None:
            s["graph"].replay()
        else:
            b.run()
        t = b.tallies.view(torch.int64)   # the mcd_tally words: counts, four FP64 sums, histograms
        out = {"counts": t[:, :30], "sums": t[:, 30:33].view(torch.float64), "hists": t[:, 34:], "status": b.status}
        if s["rows"]:
            out["rows"] = b.el
        return out
    if kind == "stream":
        seen = [0] * s["stream"].nchunks

        def consumer(rec, chunk):   # a program reduces or writes the records here
            seen[chunk] += rec.size

        r = s["stream"].run(consumer)
        return {"seen": np.array(seen), "events": r["events"], "events_tallied": r["events_tallied"],
                "bytes": r["bytes"], "tallies": r["tallies"][-1],
                "outcomes": np.array([[t[k] for k in _lib.OUTCOME_NAMES] for t in r["tallies"]])}
    if kind == "adjoint":
        scales = torch.tensor([1.0, 1.0], requires_grad=True)
        h, mean = adjoint.exit_histogram(scales[0], scales[1], s["model"])
        loss = ((h - s["target"]) ** 2).sum()
        loss.backward()
        return {"h": h.detach(), "mean": mean.detach(), "loss": loss.detach(), "grad": scales.grad}
    if kind == "project":
        return detector.project(s["dirs"])
    out = {}
    for name, kd in (("moller", "Moller"), ("gryz", "Gryz")):
        Ws, Es = s[name]
        t = tables.DeviceTable(kd, s["mat"], Ws, Es, DEV)
        out[name] = {"cdf": t.cdf, "nvalid": t.nvalid, "guide": t.guide}
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _consts(mat):
    Z, rho, A, nv, k, Eb, nsh, shells = _DATA[mat]
    n = rho * 6.02214076e23 / A * 1e6                # atoms per m^3
    J = 1e-3 * (9.76 * Z + 58.5 / Z ** 0.19) * 1e3   # mean ionisation energy, eV
    if Z < 13:
        J = 11.5 * Z
    return Z, n, J, k


def _fermi(mat):
    """Fermi energy of the valence electrons, eV (3 pi^2 n)^(2/3) hbar^2 / 2m."""
    _, rho, A, nv = _DATA[mat][:4]
    n = nv * rho * 6.02214076e23 / A * 1e6
    hbar, me, e = 1.0545718176461565e-34, 9.1093837139e-31, 1.602176634e-19
    return hbar ** 2 * (3.0 * math.pi ** 2 * n) ** (2.0 / 3.0) / (2.0 * me) / e


def _events(mat, E0, Emin, tilt, cont=False):
    """Mean scatter events of an electron, about: elastic events along the
    continuous slowing-down range, less for beams that leave early, more in
    discrete mode, whose light elements lose energy in fewer events."""
    Z, n, J, k = _consts(mat)
    E = np.geomspace(Emin, E0, 200)
    a0 = 3.4 * Z ** 0.666667
    sig = 5.21e-21 * 1e6 * 4 * math.pi * Z * Z / a0 * n * 1e-14 * ((E + 511e3) / (E + 1024e3)) ** 2 / (E + a0)
    S = 2 * PI_EFOUR * n * 1e-14 * Z / E * np.log(1.166 * (E + k * J) / J)
    f = sig / S
    full = float(np.sum(0.5 * (f[1:] + f[:-1]) * np.diff(E)))
    return full * (0.75 - 0.45 * (tilt / 90.0) ** 2) * (0.8 if Z > 40 else 1.0) * (1.0 if cont else 2.45 * (14.0 / Z) ** 0.35)


def _run_flops(mat, cont, events):
    return events * (110.0 if cont else 176.0 + 18.0 * _DATA[mat][7])


def work(case):
    c = case
    kind = c["kind"]
    if kind == "run":
        ev = c["n"] * _events(c["material"], c["E0"], c["Emin"], c["tilt"], c["mode"] == "cont")
        w = 8 if c["precision"] == "fp64" else 4
        return {"bytes": 3760.0 + c["n"] * (6.0 + 8.0 * w if c["rows"] else 0.0),
                "flops": _run_flops(c["material"], c["mode"] == "cont", ev)}
    if kind == "batch":
        b = fl = 0.0
        for p in _sims(c):
            ev = p["num_el"] * _events(p["material"], p["E0"], p["Emin"], p["s_tilt"], p["mode"] == "cont")
            if p.get("thickness"):
                ev *= 0.3
            b += 3760.0 + (p["num_el"] * 38.0 if c["rows"] else 0.0)
            fl += _run_flops(p["material"], p["mode"] == "cont", ev)
        return {"bytes": b, "flops": fl}
    if kind == "stream":
        ev = c["n"] * _events(c["material"], c["E0"], c["Emin"], c["tilt"])
        return {"bytes": 28.0 * ev, "flops": _run_flops(c["material"], False, ev)}
    if kind == "adjoint":
        ev = c["n"] * _events(c["material"], c["E0"], c["Emin"], c["tilt"], True)
        return {"bytes": 8.0 * c["n"], "flops": 1.5 * _run_flops(c["material"], True, ev)}
    if kind == "project":
        return {"bytes": 5.0 * c["n"] * (4 if c["dtype"] == "float32" else 8), "flops": 5.0 * c["n"]}
    cells = c["nE_m"] * (c["nW_m"] - 1.0) + c["nE_g"] * (c["nW_g"] - 1.0)
    return {"bytes": 4.0 * cells + (c["nE_m"] + c["nE_g"]) * (4.0 + 2.0 * 257.0),
            "flops": 25.0 * c["nE_m"] * c["nW_m"] + 100.0 * c["nE_g"] * c["nW_g"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _philox(step, elec, sim_id, seed):
    """Philox4x32-10 words of (step, electron, sim id), as int64 tensors."""
    def wide(m, x):   # high and low words of a 32 x 32 bit product
        lo16, hi16 = x & 0xffff, x >> 16
        a, b = lo16 * m, hi16 * m
        low = (a + ((b & 0xffff) << 16))
        return (b >> 16) + (low >> 32), low & 0xffffffff

    c = [torch.full_like(elec, step), elec & 0xffffffff, elec >> 32, torch.full_like(elec, sim_id)]
    k0, k1 = seed & 0xffffffff, (seed >> 32) & 0xffffffff
    for r in range(10):
        h0, l0 = wide(0xD2511F53, c[0])
        h1, l1 = wide(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ ((k0 + r * 0x9E3779B9) & 0xffffffff), l1, h0 ^ c[3] ^ ((k1 + r * 0xBB67AE85) & 0xffffffff), l0]
    return c


def _continuous(c, seed, J_scale, tangents):
    """Continuous-mode transport of every electron in FP64, with the tangents
    of the per-electron results along (J, density) where asked: a dict of
    outcome masks, exit energies and deepest z, each with d/dJ and d/dn."""
    import torch.autograd.forward_ad as fwad
    Z, n_at, J0, k = _consts(c["material"])
    a0, t = 3.4 * Z ** 0.666667, math.radians(c["tilt"])
    n = c["n"]
    f64 = dict(dtype=torch.float64, device=DEV)
    one = torch.ones(n, **f64)
    res = {}
    for which in (("J", "n") if tangents else ("",)):
        with fwad.dual_level():
            def dual(v, d):
                return fwad.make_dual(v, torch.full_like(v, d))
            ids = torch.arange(n, device=DEV)
            Js = dual(J_scale * one, 1.0 if which == "J" else 0.0) if which else J_scale * one
            ns = dual(one.clone(), 1.0 if which == "n" else 0.0) if which else one.clone()
            E = c["E0"] * one
            d = [-math.sin(t) * one, 0.0 * one, math.cos(t) * one]
            y = [0.0 * one, one.clone(), 0.0 * one]
            z, maxz = 0.0 * one, 0.0 * one
            if which:
                E, z, maxz = (dual(v, 0.0) for v in (E, z, maxz))
                d, y = [dual(v, 0.0) for v in d], [dual(v, 0.0) for v in y]
            bks = torch.zeros(n, dtype=torch.bool, device=DEV)
            out = {q: torch.zeros(n, **f64) for q in ("E", "dE", "z", "dz", "steps")}
            step = 0
            while ids.numel():
                w = _philox(step, ids, 0, seed)
                u = [(x.to(torch.float64) + 0.5) * 2.0 ** -32 for x in w]
                nat = n_at * ns
                sig = (5.21e-21 * 1e6 * 4 * math.pi * Z * Z / a0 * 1e-14) * nat * ((E + 511e3) / (E + 1024e3)) ** 2 / (E + a0)
                s = -torch.log(u[1]) / sig
                J = J0 * Js
                if c["bethe"] == "JL":
                    S = 2 * PI_EFOUR * 1e-14 * Z * nat / E * torch.log(1.166 * (E + k * J) / J)
                else:
                    S = 2 * PI_EFOUR * 1e-14 * Z * nat / E * torch.log(1.166 * E / J)
                nz = z + s * d[2]
                left = nz <= 0
                z = torch.where(left, z, nz)
                maxz = torch.where(z > maxz, z, maxz)
                En = E - s * S
                done = left | (En <= c["Emin"])
                ev, zv = (fwad.unpack_dual(v) if which else (v, None) for v in (E, maxz))
                ex, zx = (ev.primal, zv.primal) if which else (ev[0], zv[0])
                i = ids[done]
                bks[i] = left[done]
                out["E"][i], out["z"][i], out["steps"][i] = ex[done], zx[done], float(step + 1)
                if which:
                    for name, v in (("dE", ev), ("dz", zv)):
                        if v.tangent is not None:
                            out[name][i] = v.tangent[done]
                a = a0 / E
                s2 = a * u[2] / (a + (1.0 - u[2]))
                cph, sph = torch.cos(2 * math.pi * u[3]), torch.sin(2 * math.pi * u[3]).abs()
                cth, sth = 1 - 2 * s2, 2 * torch.sqrt(s2 * (1 - s2))
                x = [y[1] * d[2] - y[2] * d[1], y[2] * d[0] - y[0] * d[2], y[0] * d[1] - y[1] * d[0]]
                nd = [d[q] * cth + sth * (x[q] * cph + y[q] * sph) for q in range(3)]
                ny = [y[q] * cph - x[q] * sph for q in range(3)]
                rd = torch.rsqrt(nd[0] ** 2 + nd[1] ** 2 + nd[2] ** 2)
                ry = torch.rsqrt(ny[0] ** 2 + ny[1] ** 2 + ny[2] ** 2)
                go = ~done
                E, z, maxz, Js, ns, ids = En[go], z[go], maxz[go], Js[go], ns[go], ids[go]
                d, y = [(v * rd)[go] for v in nd], [(v * ry)[go] for v in ny]
                step += 1
        res[which] = dict(out, bks=bks)
    return res


def _soft_bins(q, lo, hi, sigma, nbins=64):
    centers = lo + (torch.arange(nbins, dtype=torch.float64, device=DEV) + 0.5) * (hi - lo) / nbins
    return torch.exp(-(q[:, None] - centers) ** 2 / (2.0 * sigma ** 2)), centers


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "project":
        x = _directions(c, seed).double()
        ca, sa = math.cos(math.radians(detector.ALPHA)), math.sin(math.radians(detector.ALPHA))
        xp, yp = detector.XY_PC
        return torch.stack([x[0] - xp, ca * x[1] + sa * x[2] - yp])
    if kind == "tables":
        out = {}
        nv, Eb, nsh = (_DATA[c["material"]][i] for i in (3, 5, 6))
        Ef = np.float32(_fermi(c["material"]))
        for name, (Ws, Es) in zip(("moller", "gryz"), _grids(c, seed)):
            W = torch.from_numpy(Ws).to(DEV).double()
            ok_w = torch.from_numpy(Ws[1:]).to(DEV)
            dW = torch.from_numpy(Ws[1:] - Ws[:-1]).to(DEV).double()
            cdf = torch.empty((len(Es), len(Ws) - 1), dtype=torch.float64, device=DEV)
            for a in range(0, len(Es), 4096):
                E32 = torch.from_numpy(Es[a:a + 4096]).to(DEV)[:, None]
                E = E32.double()
                eps = W / E
                if name == "moller":
                    f = nv * PI_EFOUR * (1 / eps ** 2 + 1 / (1 - eps) ** 2 - 1 / (eps * (1 - eps))) / E ** 3
                else:
                    eb = Eb / E
                    f = (nsh * PI_EFOUR * eps * (1 + eb) ** -1.5 * (1 - eps).clamp_min(0) ** (eb / (eb + eps)) *
                         ((1 - eb) + 4 * eb * torch.log(2.7 + torch.sqrt((1 - eps).clamp_min(0) / eb)) / (3 * eps)) / W ** 3)
                part = torch.where(ok_w <= (E32 - float(Ef)) * 0.5, dW * (f[:, 1:] + f[:, :-1]) / 2, 0.0)
                run_ = torch.cumsum(torch.nan_to_num(part), dim=1)
                cdf[a:a + 4096] = torch.where(part > 0, (run_ / run_[:, -1:]).clamp_max(1.0), 0.0)
            out[name] = {"cdf": cdf, "nvalid": None, "guide": None}
        return out
    if kind == "adjoint":
        # FP32 trajectories part from the 64-bit ones at a few events of a few
        # electrons; the binned sums over many electrons are what compares
        depth = c["quantity"] == "max_depth"
        lo, hi, sg = (0.0, 20000.0, 300.0) if depth else (c["Emin"], c["E0"], 50.0)
        q = "z" if depth else "E"
        r = _continuous(c, seed, 1.1, False)[""]
        target = _soft_bins(r[q][r["bks"]], lo, hi, sg)[0].sum(0) / c["n"]
        hs, grad = {}, []
        for _, r in _continuous(c, seed, 1.0, True).items():
            v, dv = r[q][r["bks"]], r["d" + q][r["bks"]]
            K, centers = _soft_bins(v, lo, hi, sg)
            h = K.sum(0) / c["n"]
            dh = (K * (-(v[:, None] - centers) / sg ** 2) * dv[:, None]).sum(0) / c["n"]
            grad.append(float((2 * (h - target) * dh).sum()))
            hs = {"h": h, "mean": v.mean(), "loss": ((h - target) ** 2).sum()}
        return dict(hs, grad=torch.tensor(grad, dtype=torch.float64))
    # Discrete trajectories branch on every draw: an FP32 run has no 64-bit
    # counterpart electron by electron, and whole counts are compared as such
    return None
