"""The calls that a user of this framework makes, over the sizes they are made at.

The largest share of a user's time is a whole model evaluation (build a semi-analytic model and its
hardening model, call ``gwb()``), alone or as one sample of a library.  The other cases are the
stages of that evaluation through their own entry points, and the learned emulator's query and
training step.  Sizes are those of the framework's workloads: a 30^3 grid with 20 frequencies, the
default 91 x 81 x 101 grid with 40, the 181 x 161 x 201 grid with 100, library samples with 40 to 91
edges per axis; 100 to 1000 realizations; a 6 -> 4 x 256 -> 160 network with 4 members.

A case's ``kind`` says which call it is; ``draw`` spreads each kind over its range.
"""

import numpy as np
import torch

import holodeck_gb300 as H
from holodeck_gb300 import constants as C
from holodeck_gb300 import emulator as E
from holodeck_gb300.librarian import PS_Classic_Phenom_Uniform, batch
from holodeck_gb300.sams import sam_cyutils

DUR = 16.0 * C.YR          # frequencies are harmonics of 1 / 16 yr
SAMPLE_LO, SAMPLE_HI = 40, 91     # edges per axis of a library sample
WIDTH, DEPTH, MEMBERS = 256, 4, 4


def listed():
    return [
        # a quick look at one model on a coarse grid: launches and latency count
        dict(name="gwb_small", kind="gwb", m=30, q=30, z=30, nfreq=20, nreal=100, nloud=5, precision="fp64",
             params=False),
        # the default grid with 40 frequencies and 1000 realizations in the production precision
        dict(name="gwb_default", kind="gwb", m=91, q=81, z=101, nfreq=40, nreal=1000, nloud=10, precision="fp32",
             params=False),
        # the high-resolution grid (with fewer realizations than its production run, to stay short)
        dict(name="gwb_highres", kind="gwb", m=181, q=161, z=201, nfreq=100, nreal=200, nloud=10, precision="fp32",
             params=False),
        # source parameters of the loudest binaries, asked for on small grids
        dict(name="gwb_params", kind="gwb", m=41, q=31, z=37, nfreq=20, nreal=100, nloud=5, precision="fp64",
             params=True),
        # a stretch of a parameter library: every sample on its own grid, single sources and second-pass GWB
        dict(name="library_8", kind="library", nsamples=8, nfreq=40, nloud=10, reals_lo=100, reals_hi=1000,
             grid_seed=3, gwb=True, precision="fp32"),
        # the density of a new model on the default grid, M-Mbulge scatter included
        dict(name="density_default", kind="density", m=91, q=81, z=101, scatter=0.28),
        # the hardening normalisation of every (mtot, mrat) cell
        dict(name="norm_default", kind="norm", m=91, q=81, gamma_inner=-1.0),
        # differential binary number in the parity precision, two-power-law hardening
        dict(name="dbn_default", kind="dbn", m=91, q=81, z=101, nfreq=40, gamma_inner=-1.0),
        # the same for GW-only hardening, on an odd-sized grid
        dict(name="dbn_gw_odd", kind="dbn_gw", m=61, q=47, z=53, nfreq=37),
        # integration over the bins and strain of every bin, on an odd-sized grid
        dict(name="cells_odd", kind="cells", m=67, q=59, z=83, nfreq=37),
        # one parameter vector through the trained emulator: the smallest call
        dict(name="query_1", kind="query", batch=1),
        # one training step of the emulator at its default batch
        dict(name="train_512", kind="train", batch=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["gwb", "gwb", "library", "density", "norm", "dbn", "dbn_gw", "cells", "query", "train"])
    axis = lambda: _log_int(rng, 24, 101)  # noqa: E731
    if kind == "gwb":
        params = rng.random() < 0.25
        top = 40 if params else 91
        return dict(kind=kind, m=_log_int(rng, 20, top), q=_log_int(rng, 20, top), z=_log_int(rng, 20, top),
                    nfreq=rng.randint(5, 40), nreal=_log_int(rng, 20, 200 if params else 1000),
                    nloud=rng.randint(1, 10), precision=rng.choice(["fp64", "fp32"]), params=params)
    if kind == "library":
        return dict(kind=kind, nsamples=rng.randint(3, 8), nfreq=rng.randint(10, 40), nloud=rng.randint(1, 10),
                    reals_lo=100, reals_hi=_log_int(rng, 150, 1000), grid_seed=rng.randint(10, 10 ** 6),
                    gwb=rng.random() < 0.5, precision=rng.choice(["fp64", "fp32"]))
    if kind == "density":
        return dict(kind=kind, m=axis(), q=axis(), z=axis(), scatter=round(rng.uniform(0.1, 0.6), 3))
    if kind == "norm":
        return dict(kind=kind, m=axis(), q=axis(), gamma_inner=rng.choice([-1.0, -0.5, round(rng.uniform(-1.5, 0.0), 3)]))
    if kind == "dbn":
        return dict(kind=kind, m=axis(), q=axis(), z=axis(), nfreq=rng.randint(5, 40),
                    gamma_inner=rng.choice([-1.0, -0.5, round(rng.uniform(-1.5, 0.0), 3)]))
    if kind in ("dbn_gw", "cells"):
        return dict(kind=kind, m=axis(), q=axis(), z=axis(), nfreq=rng.randint(5, 60))
    if kind == "query":
        return dict(kind=kind, batch=rng.choice([rng.randint(2, 16), _log_int(rng, 17, 2048)]))
    return dict(kind=kind, batch=_log_int(rng, 64, 1024))


# ---- inputs

def _settings(seed, case):
    """Physical settings of one model, inside the ranges that libraries are drawn from."""
    rng = np.random.default_rng([int(seed), 17])
    return dict(phi0=rng.uniform(-3.0, -2.5), mchar=rng.uniform(11.0, 11.5), mamp=rng.uniform(8.4, 8.9),
                time=rng.uniform(1.0, 6.0) * C.GYR, rchar=100.0 * C.PC, gi=float(case.get("gamma_inner", -1.0)),
                go=2.5, key=int(rng.integers(1, 2 ** 62)))


def _sam(case, s, scatter):
    return H.sams.Semi_Analytic_Model(gsmf=H.sams.GSMF_Schechter(phi0=s["phi0"], mchar0_log10=s["mchar"]),
                                      gpf=H.sams.GPF_Power_Law(), gmt=H.sams.GMT_Power_Law(),
                                      mmbulge=H.host_relations.MMBulge_KH2013(mamp_log10=s["mamp"],
                                                                              scatter_dex=scatter),
                                      shape=(case["m"], case["q"], case["z"]))


def _hard(sam, s):
    return H.hardening.Fixed_Time_2PL_SAM(sam, s["time"], rchar=s["rchar"], gamma_inner=s["gi"], gamma_outer=s["go"])


def _edges(case):
    return (np.logspace(*np.log10([1e4 * C.MSOL, 1e12 * C.MSOL]), case["m"]), np.logspace(-3.0, 0.0, case["q"]),
            np.logspace(-3.0, 1.0, case["z"]) if "z" in case else None)


def prepare(case, seed):
    kind = case["kind"]
    s = _settings(seed, case)
    st = dict(case=case, s=s)
    if "nfreq" in case:
        cents, edges = H.utils.pta_freqs(DUR, case["nfreq"])
        st.update(cents=cents, edges=edges)
    if kind == "library":
        space = PS_Classic_Phenom_Uniform(nsamples=case["nsamples"], sam_shape=None, seed=int(seed) % (1 << 30))
        shapes, reals = batch.random_shapes(case["nsamples"], SAMPLE_LO, SAMPLE_HI, case["reals_lo"],
                                            case["reals_hi"], seed=case["grid_seed"])
        st.update(space=space, shapes=shapes, reals=reals)
    elif kind == "norm":
        mt, mr, _ = _edges(case)
        mt, mr = np.meshgrid(mt, mr, indexing="ij")
        st.update(mt=torch.as_tensor(mt.ravel(), device="cuda"), mr=torch.as_tensor(mr.ravel(), device="cuda"))
    elif kind in ("dbn", "dbn_gw"):
        # the model and its hardening are in hand; their density and normalisation are computed once
        sam = _sam(case, s, 0.0)
        sam.static_binary_density
        hard = _hard(sam, s) if kind == "dbn" else H.hardening.Hard_GW()
        st.update(sam=sam, hard=hard, fobs=torch.as_tensor(st["cents"] / 2.0, device="cuda"))
    elif kind == "cells":
        st.update(_cells_inputs(case, seed, st["edges"]))
    elif kind in ("query", "train"):
        emu = E.Emulator(PS_Classic_Phenom_Uniform(nsamples=2, seed=0), nfreqs=40, members=MEMBERS, width=WIDTH,
                         depth=DEPTH, seed=int(seed) % (1 << 30))
        rng = np.random.default_rng([int(seed), 23])
        emu.mu = rng.uniform(-16.0, -14.0, emu.n_out)
        emu.sd = rng.uniform(0.2, 0.8, emu.n_out)
        rows = emu.lo + (emu.hi - emu.lo) * rng.random((case["batch"], emu.lo.size))
        st.update(emu=emu, rows=rows)
        if kind == "query":
            st["ask"] = emu.native(case["batch"]) if case["batch"] <= 16 else emu.graphed(case["batch"])
        else:
            y = rng.standard_normal((case["batch"], emu.n_pad)).astype(np.float32)
            st.update(x=emu.inputs(rows), y=torch.as_tensor(y, device="cuda"))
    return st


def _cells_inputs(case, seed, gw_edges):
    """dnum and redz_final as the differential-number stage leaves them: redshifts that fall with
    frequency-independent scatter below the starting one, and a region of cells that reach no target
    frequency before z = 0 (-1 and 0)."""
    mt, mr, rz = _edges(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
    shape = (case["m"], case["q"], case["z"], case["nfreq"])
    u = torch.rand(shape, dtype=torch.float64, device="cuda", generator=g)
    z0 = torch.as_tensor(rz, device="cuda")[None, None, :, None]
    tm = torch.linspace(0.0, 1.0, case["m"], dtype=torch.float64, device="cuda")[:, None, None, None]
    tq = torch.linspace(0.0, 1.0, case["q"], dtype=torch.float64, device="cuda")[None, :, None, None]
    lag = 0.15 + 0.5 * (1.0 - tm) + 0.25 * tq
    z = z0 * (1.0 - lag * (0.9 + 0.05 * u)) - 0.02 * lag
    gone = z <= 0.0
    lam = torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    tz = torch.log10(1.0 + z0)
    dnum = 10.0 ** (4.0 - 10.0 * tm - 3.0 * tz + 0.3 * lam)
    return dict(mt=mt, mr=mr, rz=rz, fe=gw_edges / 2.0, redz_final=torch.where(gone, -1.0, z).contiguous(),
                dnum=torch.where(gone, 0.0, dnum).contiguous())


def run(state):
    case, s = state["case"], state["s"]
    kind = case["kind"]
    if kind == "gwb":
        sam = _sam(case, s, 0.28)
        hard = _hard(sam, s)
        return sam.gwb(state["edges"], hard=hard, realize=case["nreal"], loudest=case["nloud"], params=case["params"],
                       seed=s["key"], precision=case["precision"])
    if kind == "library":
        res = batch.run_library(state["space"], shapes=state["shapes"], nreals=state["reals"], nfreqs=case["nfreq"],
                                nloudest=case["nloud"], seed=s["key"], gwb_flag=case["gwb"], workers=8, waves=12,
                                precision=case["precision"])
        keys = ("hc_ss", "hc_bg", "gwb") if case["gwb"] else ("hc_ss", "hc_bg")
        return [{k: r[k] for k in keys} for r in res]
    if kind == "density":
        return _sam(case, s, case["scatter"]).static_binary_density
    if kind == "norm":
        return sam_cyutils.find_2pwl_hardening_norm(s["time"], state["mt"], state["mr"], 1e3 * C.PC, s["rchar"],
                                                    s["gi"], s["go"], 300)
    if kind in ("dbn", "dbn_gw"):
        return sam_cyutils.dynamic_binary_number_at_fobs(state["fobs"], state["sam"], state["hard"])
    if kind == "cells":
        edges = [state["mt"], state["mr"], state["rz"], state["fe"]]
        return (sam_cyutils.integrate_differential_number_3dx1d(edges, state["dnum"]),
                H.gravwaves.char_strain_sq_from_bin_edges_redz(edges, state["redz_final"]))
    if kind == "query":
        return state["ask"](state["rows"])
    net = state["emu"].net
    loss = net.train_step(state["x"], state["y"], 1e-3)
    return loss, net.grad, net.params


# ---- what a pass cannot do without: inputs once, outputs once, and the arithmetic that the
# definitions ask for (a draw counts as 2 operations for its product and sum; a transcendental as 10)

def work(case):
    kind = case["kind"]
    if kind == "gwb":
        return _gwb_work(case["m"], case["q"], case["z"], case["nfreq"], case["nreal"], case["nloud"],
                         11 if case["params"] else 0)
    if kind == "library":
        shapes, reals = batch.random_shapes(case["nsamples"], SAMPLE_LO, SAMPLE_HI, case["reals_lo"],
                                            case["reals_hi"], seed=case["grid_seed"])
        parts = [_gwb_work(*shp, case["nfreq"], nr, case["nloud"], 0) for shp, nr in zip(shapes, reals)]
        more = 2 if case["gwb"] else 1
        return {"bytes": sum(p["bytes"] for p in parts), "flops": more * sum(p["flops"] for p in parts)}
    if kind == "density":
        pts = case["m"] * case["q"] * case["z"]
        return {"bytes": 8.0 * pts, "flops": pts * (60.0 + 4.0 * 4 * case["m"])}
    if kind == "norm":
        n = case["m"] * case["q"]
        return {"bytes": 24.0 * n, "flops": n * 301.0 * (40 + 12 * 4)}
    if kind in ("dbn", "dbn_gw"):
        pts = case["m"] * case["q"] * case["z"]
        return {"bytes": 8.0 * pts * (2 + 2 * case["nfreq"]), "flops": pts * case["nfreq"] * 60.0}
    if kind == "cells":
        pts = case["m"] * case["q"] * case["z"] * case["nfreq"]
        return {"bytes": 32.0 * pts, "flops": 45.0 * pts}
    n_out = 160
    par = MEMBERS * (16 * WIDTH + (DEPTH - 1) * WIDTH ** 2 + WIDTH * n_out + DEPTH * WIDTH + n_out)
    if kind == "query":
        return {"bytes": 2.0 * par + case["batch"] * (48 + 8 * n_out), "flops": 2.0 * par * case["batch"]}
    return {"bytes": 4.0 * par * 8 + case["batch"] * (32 + 4 * n_out), "flops": 6.0 * par * case["batch"]}


def _gwb_work(m, q, z, nfreq, nreal, nloud, npar):
    elems = float((m - 1) * (q - 1) * (z - 1)) * nfreq
    out = nfreq * nreal * (nloud + 1) * 8.0
    # about four tenths of the (bin, frequency) pairs hold binaries that have to be drawn
    return {"bytes": out + nfreq * nreal * 8.0 * npar, "flops": elems * 105.0 + 0.4 * elems * nreal * 2.0}


# ---- 64-bit values

def exact(case, seed):
    kind = case["kind"]
    if kind == "cells":
        return _exact_cells(case, seed)
    if kind == "norm":
        mt, mr, _ = _edges(case)
        mt, mr = (torch.as_tensor(x.ravel(), device="cuda") for x in np.meshgrid(mt, mr, indexing="ij"))
        return _exact_norm(_settings(seed, case), mt, mr)[0]
    if kind in ("dbn", "dbn_gw"):
        return _exact_dbn(case, seed)
    if kind == "query":
        st = prepare(case, seed)
        emu = st["emu"]
        x = torch.as_tensor(2.0 * (st["rows"] - emu.lo) / (emu.hi - emu.lo) - 1.0)
        with torch.no_grad():
            out = torch.stack([_exact_forward(p, x)[0] for p in emu.net.params.double().cpu()])
        out = out[..., :emu.n_out].mean(dim=0).numpy() * emu.sd + emu.mu
        return out.reshape(len(x), emu.nfreqs, 4)
    if kind == "train":
        return _exact_train(case, seed)
    return None   # random draws (gwb, library), or scipy's interpolant in between (density)


# constants of the reference's compiled kernels (an older set than the Python stages')
CY_G, CY_C, CY_MPC, CY_SCHW = 6.6742999e-08, 29979245800.0, 3.08567758e+24, 1.4852320538237328e-28
H0, OM0 = 0.6933 * 100.0 * 1.0e5 / C.MPC, 0.2880
OL0 = 1.0 - OM0


def _dcom(z):
    """Comoving distance [cm] by 32-point Gauss-Legendre quadrature in u = sqrt(a)."""
    x, w = np.polynomial.legendre.leggauss(32)
    s = torch.sqrt(1.0 + z)
    u0 = 1.0 / s
    half = 0.5 * z / (s * (s + 1.0))   # (1 - u0) / 2 without cancellation
    tot = torch.zeros_like(z)
    for xi, wi in zip(x, w):
        u = 0.5 * (1.0 + u0) + half * xi
        tot += wi * 2.0 / torch.sqrt(OM0 + OL0 * u ** 6)
    return C.SPLC / H0 * half * tot


def _mid(x, axis):
    n = x.shape[axis]
    return 0.5 * (x.narrow(axis, 1, n - 1) + x.narrow(axis, 0, n - 1))


def _exact_cells(case, seed):
    _, edges = H.utils.pta_freqs(DUR, case["nfreq"])
    i = _cells_inputs(case, seed, edges)
    dev = [torch.as_tensor(x, device="cuda") for x in (i["mt"], i["mr"], i["rz"], i["fe"])]
    mt, mr, rz, fe = dev
    num = i["dnum"]
    for axis in range(3):
        num = _mid(num, axis)
    vol = torch.diff(torch.log10(mt))[:, None, None] * torch.diff(mr)[None, :, None] * torch.diff(rz)[None, None, :]
    num = num * vol[..., None] * torch.diff(torch.log(fe))
    z = i["redz_final"]
    for axis in range(3):
        z = _mid(z, axis)
    fc, df = _mid(fe, 0), torch.diff(fe)
    mc = _mid(mt, 0)[:, None] * _mid(mr, 0) ** 0.6 / (1.0 + _mid(mr, 0)) ** 1.2
    h2 = torch.zeros_like(z)
    for m in range(z.shape[0]):   # a slab at a time bounds the memory
        ok = z[m] > 0.0
        zz = torch.where(ok, z[m], 1.0)
        mm = mc[m][:, None, None]
        hs = C.GW_SRC_CONST * mm * (2.0 * mm * fc * (1.0 + zz)) ** (2.0 / 3.0) / _dcom(zz)
        h2[m] = torch.where(ok, hs ** 2 * fc / df, 0.0)
    return num, h2


def _rate(s, mt, mr, sepa, norm):
    """Hardening rate da/dt of the two-power-law model with GW emission (all positive here: -da/dt)."""
    x = sepa / s["rchar"]
    return (norm * (1.0 + x) ** (s["gi"] - s["go"]) / x ** (s["gi"] - 1.0) +
            64.0 * CY_G ** 3 / 5.0 / CY_C ** 5 * mt ** 3 * mr / sepa ** 3 / (1.0 + mr) ** 2)


def _nodes(mt, sepa_init, steps):
    lo = torch.log10(3.0 * CY_SCHW * mt)
    k = torch.arange(steps + 1, dtype=torch.float64, device=mt.device)
    return 10.0 ** (np.log10(sepa_init) - (np.log10(sepa_init) - lo)[:, None] / steps * k)


def _exact_norm(s, mt, mr, sepa_init=1e3 * C.PC, steps=300):
    """Brent's root (1973, ch. 4) of the lifetime in log10(norm) on [-20, 20], every cell at once, with
    the tolerance (1e-3 + 1e-5 |x|) / 2 of the reference: the iterate is part of the definition."""
    sepa = _nodes(mt, sepa_init, steps)

    def f(x):
        v = _rate(s, mt[:, None], mr[:, None], sepa, 10.0 ** x[:, None])
        return (2.0 * (sepa[:, :-1] - sepa[:, 1:]) / (v[:, :-1] + v[:, 1:])).sum(dim=1) - s["time"]

    xa, xb = torch.full_like(mt, -20.0), torch.full_like(mt, 20.0)
    fa, fb = f(xa), f(xb)
    none = fa * fb > 0.0
    root = torch.zeros_like(mt)
    done = none.clone()
    xc, fc, d = xa.clone(), fa.clone(), xb - xa
    e = d.clone()
    for _ in range(100):
        same = fb * fc > 0.0
        xc, fc = torch.where(same, xa, xc), torch.where(same, fa, fc)
        d, e = torch.where(same, xb - xa, d), torch.where(same, xb - xa, e)
        swap = fc.abs() < fb.abs()
        xa, xb, xc = torch.where(swap, xb, xa), torch.where(swap, xc, xb), torch.where(swap, xb, xc)
        fa, fb, fc = torch.where(swap, fb, fa), torch.where(swap, fc, fb), torch.where(swap, fb, fc)
        tol, m = 0.5 * (1e-3 + 1e-5 * xb.abs()), 0.5 * (xc - xb)
        stop = ((fb == 0.0) | (m.abs() < tol)) & ~done
        root = torch.where(stop, xb, root)
        done |= stop
        if bool(done.all()):
            break
        sec = -fb * (xb - xa) / (fb - fa)
        da, dc = (fa - fb) / (xa - xb), (fc - fb) / (xc - xb)
        quad = -fb * (fc * dc - fa * da) / (dc * da * (fc - fa))
        t = torch.where(xa == xc, sec, quad)
        good = (e.abs() > tol) & (fb.abs() < fa.abs()) & (2.0 * t.abs() < torch.minimum(e.abs(), 3.0 * m.abs() - tol))
        e, d = torch.where(good, d, m), torch.where(good, t, m)
        xa, fa = xb, fb
        xb = xb + torch.where(d.abs() > tol, d, torch.where(m > 0.0, tol, -tol))
        fb = f(xb)
    return root, sepa


def _tables():
    zg = np.concatenate([np.logspace(4.0, -4.0, 199), [0.0]])
    z = torch.as_tensor(zg, device="cuda")
    age = 2.0 / (3.0 * H0 * np.sqrt(OL0)) * torch.asinh(np.sqrt(OL0 / OM0) * (1.0 + z) ** -1.5)
    return z, age, _dcom(z)


def _lookup(x, xs, *ys):
    """Linear interpolation in the bracket of x in the increasing table xs, extrapolated at its ends."""
    i = (torch.searchsorted(xs, x.contiguous()) - 1).clamp(0, xs.numel() - 2)
    t = (x - xs[i]) / (xs[i + 1] - xs[i])
    return [y[i] + (y[i + 1] - y[i]) * t for y in ys]


def _exact_dbn(case, seed):
    s = _settings(seed, case)
    mt, mr, rz = (torch.as_tensor(x, device="cuda") for x in _edges(case))
    cents, _ = H.utils.pta_freqs(DUR, case["nfreq"])
    fobs = torch.as_tensor(cents / 2.0, device="cuda")
    # static density (no scatter): GSMF_Schechter, GPF_Power_Law, GMT_Power_Law and MMBulge_KH2013 defaults
    gsmf, gpf, gmt = H.sams.GSMF_Schechter(phi0=s["phi0"], mchar0_log10=s["mchar"]), H.sams.GPF_Power_Law(), \
        H.sams.GMT_Power_Law()
    mmb = H.host_relations.MMBulge_KH2013(mamp_log10=s["mamp"])
    bf, amp, ref, pl = mmb._bulge_frac.bulge_frac(), mmb._mamp, mmb._mref, mmb._mplaw
    M, Q, Z = mt[:, None, None], mr[None, :, None], rz[None, None, :]
    m1 = M / (1.0 + Q)
    pri, sec = (ref * (x / amp) ** (1.0 / pl) / bf for x in (m1, M - m1))
    rat, tot = sec / pri, sec + pri
    mchar, alpha = gsmf._mchar0 + gsmf._mcharz * Z, gsmf._alpha0 + gsmf._alphaz * Z
    x = pri / mchar
    dens = np.log(10.0) * 10.0 ** (gsmf._phi0 + gsmf._phiz * Z) * x ** (1.0 + alpha) * torch.exp(-x)
    g = [getattr(gpf, n) for n in ("_frac_norm", "_mref", "_malpha", "_zbeta", "_qgamma", "_max_frac")]
    frac = (g[0] * (pri / g[1]) ** g[2] * (1.0 + Z) ** g[3] * rat ** g[4]).clamp(max=g[5])
    gtime = gmt._time_norm * (pri / gmt._mref) ** gmt._malpha * (1.0 + Z) ** gmt._zbeta * rat ** gmt._qgamma
    dens = dens * frac / gtime / (H0 * (1.0 + Z) * torch.sqrt(OM0 * (1.0 + Z) ** 3 + OL0))
    jac = (pri * bf) / (pl * amp * (pri * bf / ref) ** pl) / bf * (1.0 + rat) / (1.0 + Q) / (pl * rat ** (pl - 1.0))
    dens = dens * (M / tot) * jac
    age = 2.0 / (3.0 * H0 * np.sqrt(OL0)) * torch.asinh(np.sqrt(OL0 / OM0) * (1.0 + Z) ** -1.5) + gtime
    t0 = 2.0 / (3.0 * H0 * np.sqrt(OL0)) * np.arcsinh(np.sqrt(OL0 / OM0))
    zp = torch.where(age < t0, (np.sqrt(OL0 / OM0) / torch.sinh(1.5 * H0 * np.sqrt(OL0) * age)) ** (2.0 / 3.0) - 1.0,
                     -1.0)
    dens = torch.where(zp < 0.0, 0.0, dens)
    zg, ag, dg = _tables()
    shape = tuple(dens.shape) + (case["nfreq"],)
    redz, dnum = torch.full(shape, -1.0, dtype=torch.float64, device="cuda"), torch.zeros(
        shape, dtype=torch.float64, device="cuda")
    kfreq, ksepa = np.sqrt(CY_G) / (2.0 * np.pi), CY_G ** (1.0 / 3.0) / (2.0 * np.pi) ** (2.0 / 3.0)
    fourpi = 4.0 * np.pi * CY_C / CY_MPC
    if case["kind"] == "dbn_gw":
        live = zp > 0.0
        zz = torch.where(live, zp, 1.0)
        dc, = _lookup(zz, zg.flip(0), dg.flip(0))
        redz[:] = torch.where(live, zp, -1.0)[..., None]
        frst = fobs * (1.0 + zz[..., None])
        isco = kfreq * torch.sqrt(M) / (3.0 * CY_SCHW * M) ** 1.5
        sepa = ksepa * (M ** (1.0 / 3.0))[..., None] / frst ** (2.0 / 3.0)
        rate = 64.0 * CY_G ** 3 / 5.0 / CY_C ** 5 * (M ** 3 * Q / (1.0 + Q) ** 2)[..., None] / sepa ** 3
        tres = 2.0 / 3.0 * sepa / rate
        val = dens[..., None] * tres * fourpi * (1.0 + zz[..., None]) * (dc[..., None] / CY_MPC) ** 2
        dnum[:] = torch.where(live[..., None] & (frst <= isco[..., None]), val, 0.0)
        return redz, dnum
    steps = 300
    cm, cq = (x.reshape(-1) for x in torch.meshgrid(mt, mr, indexing="ij"))
    root, sepa = _exact_norm(s, cm, cq)
    norm = 10.0 ** root
    frst = kfreq * torch.sqrt(cm)[:, None] / sepa ** 1.5
    v = _rate(s, cm[:, None], cq[:, None], sepa, norm[:, None])
    dts = 2.0 * (sepa[:, :-1] - sepa[:, 1:]) / (v[:, :-1] + v[:, 1:])
    tevo = torch.cumsum(dts, dim=1)
    start, = _lookup(rz, zg.flip(0), ag.flip(0))
    start = gtime.expand(dens.shape).reshape(len(cm), -1) + start    # (cells, redz)
    when = torch.zeros((len(cm), len(rz), case["nfreq"]), dtype=torch.float64, device="cuda")
    hit = torch.zeros_like(when, dtype=torch.bool)
    for k in range(steps):
        if float(frst[:, k].min()) > float(fobs.max()) * (1.0 + float(rz.max())) or \
                float(frst[:, k + 1].max()) < float(fobs.min()):
            continue
        tr = start + tevo[:, k, None]
        tl = tr - dts[:, k, None]
        zl, = _lookup(tl, ag, zg)
        zr, = _lookup(tr, ag, zg)
        ok = (tl <= ag[-1]) & (zl >= 0.0)
        fl = frst[:, k, None] / (1.0 + zl)
        fr = frst[:, k + 1, None] / (1.0 + zr.clamp(min=0.0))
        t = tl[..., None] + (tr - tl)[..., None] * (fobs - fl[..., None]) / (fr - fl)[..., None]
        new = ok[..., None] & (fobs >= fl[..., None]) & (fobs <= fr[..., None]) & (t <= ag[-1])
        when = torch.where(new, t, when)
        hit |= new
    norm, cm, cq = norm[:, None, None], cm[:, None, None], cq[:, None, None]
    redz, dnum = redz.reshape(when.shape), dnum.reshape(when.shape)
    zz, dc = _lookup(torch.where(hit, when, ag[100]), ag, zg, dg)
    sep = ksepa * cm ** (1.0 / 3.0) / (fobs * (1.0 + zz)) ** (2.0 / 3.0)
    tres = 2.0 / 3.0 * sep / _rate(s, cm, cq, sep, norm)
    val = dens.reshape(when.shape[:2])[..., None] * tres * fourpi * (1.0 + zz) * (dc / CY_MPC) ** 2
    return (torch.where(hit, zz, redz).reshape(shape), torch.where(hit, val, dnum).reshape(shape))


def _layers(p):
    dims, off = [16] + [WIDTH] * DEPTH + [160], 0
    for k, n in zip(dims[:-1], dims[1:]):
        yield p[off:off + n * k].reshape(n, k), p[off + n * k:off + n * k + n]
        off += n * k + n


def _exact_forward(p, x):
    """One member's outputs, and its parameters as the leaves that they were computed from."""
    h = torch.zeros((x.shape[0], 16), dtype=torch.float64, device=x.device)
    h[:, :x.shape[1]] = x
    layers = [(w.clone().requires_grad_(), b.clone().requires_grad_()) for w, b in _layers(p)]
    for ii, (w, b) in enumerate(layers):
        h = h @ w.T + b
        if ii + 1 < len(layers):
            h = torch.nn.functional.silu(h)
    return h, layers


def _exact_train(case, seed):
    st = prepare(case, seed)
    params = st["emu"].net.params.double()
    x, y = st["x"].double(), st["y"].double()
    losses, grads = [], []
    with torch.enable_grad():
        for p in params:
            out, layers = _exact_forward(p, x)
            loss = ((out - y) ** 2).mean()
            loss.backward()
            losses.append(loss.detach())
            grads.append(torch.cat([t.grad.reshape(-1) for wb in layers for t in wb]))
    g = torch.stack(grads)
    # AdamW, first step: m / (1 - b1) = g and v / (1 - b2) = g^2
    return torch.stack(losses), g, params - 1e-3 * (g / (g.abs() + 1e-8) + 1e-4 * params)
