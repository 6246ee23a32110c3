"""The work whose speed this repository watches: calls that a user's program
makes, through the package's public entry points, at the sizes it makes them.

``listed()`` names the cases, ``draw(rng)`` gives others of the same ranges,
``prepare(case, seed)`` makes what the program holds before the call (on the
GPU unless the path works on host arrays), ``run(state)`` is one call,
``work(case)`` the bytes and flop-equivalents it cannot do without, and
``exact(case, seed)`` the same outputs in plain 64-bit torch.

Columns follow gitm_b200.synthetic (Bates temperatures, species in diffusive
equilibrium, smooth wind profiles, Chapman ion layers on the stretched
100-600 km grid); the blocks of the horizontal cases follow
gitm_b200.horizontal.synthetic_blocks.  Both are made here with torch on the
GPU so that a globe takes milliseconds.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from gitm_b200 import abi, adjoint, horizontal, synthetic, vertical
from gitm_b200._lib import lib

DT = 2.0        # s, the vertical step of the reference's default run
DT_HOST = 0.05  # s, where the host arrays go on from call to call
DT_HZ = 1.0     # s, keeps the polar cells of the finest blocks inside their CFL limit
NS, NI, NADV = abi.NSPECIES, abi.NIONS - 1, abi.NIONS_ADVECT
STATE = adjoint.STATE
F64 = torch.float64


def listed():
    return [
        # GITM's default run: 2 x 2 blocks of 9 x 9 columns, one step per call from a state the
        # program sets (an assimilation cycle): the smallest call, latency and launches
        dict(name="default_run_step", kind="steps", cols=324, n_alts=50, solver="rusanov", threads=0, steps=1),
        # a whole globe at 1 degree, 16 steps resident in one launch: the headline workload
        dict(name="globe_1deg_resident", kind="steps", cols=64800, n_alts=50, solver="rusanov", threads=512, steps=16),
        # an ensemble of uneven resolutions and altitude counts in one launch, with heating
        dict(name="ensemble_uneven", kind="ensemble", members="50x2592 75x10368 100x2592 75x2592 50x10368 100x16200",
             steps=2),
        # the AUSM solver on the 2.5 degree globe
        dict(name="ausm_2.5deg", kind="steps", cols=10368, n_alts=50, solver="ausm", threads=384, steps=4),
        # advance_vertical_all on device arrays, one call per step, at 5 degrees
        dict(name="dropin_5deg", kind="dropin", cols=2592, n_alts=50),
        # the Fortran host's call: 4 x 8 blocks of 9 x 9 columns in GITM's own arrays on the GPU
        dict(name="fortran_5deg", kind="fortran", n_lons=9, n_lats=9, blocks=32, n_alts=50),
        # the host-pointer call of a GITM that lives in host memory, at 2.5 degrees
        dict(name="host_2.5deg", kind="host", cols=10368, n_alts=50),
        # one step forward and backward (sensitivities of a 5 degree globe)
        dict(name="adjoint_5deg", kind="adjoint", cols=2592, n_alts=50),
        # a checkpointed rollout of the 2.5 degree globe, O/N2 at 400 km
        dict(name="rollout_2.5deg", kind="rollout", cols=10368, n_alts=50, steps=4, every=2),
        # the horizontal advance of a 2 degree globe of 9 x 9 blocks
        dict(name="horizontal_2deg", kind="hz", n_lons=9, n_lats=9, n_alts=50, blocks_lon=20, blocks_lat=10),
        # the whole horizontal step (exchange, advance, exchange) of a 5 degree globe
        dict(name="horizontal_step_5deg", kind="hz_step", n_lons=9, n_lats=9, n_alts=50, blocks_lon=8, blocks_lat=4),
        # calc_timestep_vertical on a 1 degree globe
        dict(name="timestep_1deg", kind="cfl", cols=64800, n_alts=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _n_alts(rng):
    """GITM's 50 altitudes most often, else any count a user may configure."""
    return 50 if rng.random() < 0.4 else rng.randint(20, 100)


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "ensemble", "ausm", "dropin", "fortran", "host", "adjoint",
                       "rollout", "hz", "hz_step", "cfl"])
    na = _n_alts(rng)
    if kind == "steps":
        steps = rng.choice([1, 1, 2, 5, 16])
        cols = _log_int(rng, 60, 30000)
        return dict(kind="steps", cols=cols, n_alts=na, solver="rusanov",
                    threads=0 if steps == 1 else rng.choice([0, 512]), steps=steps)
    if kind == "ausm":
        return dict(kind="steps", cols=_log_int(rng, 60, 10000), n_alts=na, solver="ausm",
                    threads=384 if na == 50 else 0, steps=rng.choice([1, 2, 4]))
    if kind == "ensemble":
        m = " ".join("%dx%d" % (rng.choice([50, 75, 100, _n_alts(rng)]), _log_int(rng, 200, 8000))
                     for _ in range(rng.randint(2, 8)))
        return dict(kind="ensemble", members=m, steps=rng.choice([1, 2, 4]))
    if kind == "fortran":
        return dict(kind="fortran", n_lons=rng.randint(5, 12), n_lats=rng.randint(5, 12), blocks=rng.randint(1, 32),
                    n_alts=na)
    if kind in ("hz", "hz_step"):
        return dict(kind=kind, n_lons=rng.randint(5, 13), n_lats=rng.randint(5, 13), n_alts=rng.randint(20, 60),
                    blocks_lon=2 * rng.randint(2, 6), blocks_lat=rng.randint(2, 6))
    if kind == "rollout":
        return dict(kind="rollout", cols=_log_int(rng, 300, 6000), n_alts=na, steps=rng.randint(2, 5),
                    every=rng.randint(1, 3))
    hi = {"dropin": 20000, "host": 10000, "adjoint": 6000, "cfl": 60000}[kind]
    return dict(kind=kind, cols=_log_int(rng, 100, hi), n_alts=na)


# ------------------------------------------------------------------ columns
@functools.lru_cache(maxsize=None)
def _grid(n_alts):
    alt = synthetic.make_altitude_grid(n_alts)
    dalt, inv_r, grav = synthetic.grid_geometry(alt)
    return alt, dalt, inv_r, grav


def _gen(seed, *more):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.SeedSequence([seed, *more]).generate_state(1, np.uint64)[0] >> 2))
    return g


def _columns(n_cols, n_alts, seed, member=0, shift=0.0):
    """The arrays of one member (names as GitmColumnBatch), float64 CUDA tensors [field, cell, column]."""
    g = _gen(seed, member)
    alt, dalt, inv_r, grav = (torch.as_tensor(a, device="cuda", dtype=F64) for a in _grid(n_alts))
    G = n_alts + 4

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=F64)

    def nrm(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=F64)

    def smooth(n):
        """n random profiles with unit variance and a correlation length of about 120 km."""
        z = ((alt - alt[0]) / 120.0e3)[None, :, None]
        out = torch.zeros(n, G, n_cols, device="cuda", dtype=F64)
        for _ in range(6):
            out += nrm(n, 1, n_cols) * torch.cos(uni(0.5, 2.0, n, 1, n_cols) * z + uni(0, 2 * math.pi, n, 1, n_cols))
        return out * math.sqrt(2.0 / 6)

    tinf = torch.clamp(uni(700.0, 1500.0, n_cols) + shift, min=400.0)
    z = alt[:, None]
    T = tinf - (tinf - 190.0) * torch.exp(-0.02 * torch.clamp(z / 1000.0 - 100.0, min=0.0))
    gz = synthetic.GC * (synthetic.RBODY / (synthetic.RBODY + z)) ** 2
    base = torch.as_tensor(synthetic.BASE_DENSITY, device="cuda", dtype=F64)[:, None] * 10.0 ** uni(-0.3, 0.3, NS, n_cols)
    mass = torch.as_tensor(synthetic.MASS, device="cuda", dtype=F64)[:, None, None]
    inv_h = mass * gz / (synthetic.KB * T)
    seg = 0.5 * (inv_h[:, 1:] + inv_h[:, :-1]) * (alt[1:] - alt[:-1])[None, :, None]
    integ = torch.cat([torch.zeros_like(seg[:, :1]), torch.cumsum(seg, 1)], 1)
    nd = base[:, None] * (T[2] / T) * torch.exp(-(integ - integ[:, 2:3]))
    lay = torch.as_tensor(synthetic.ION_LAYERS, device="cuda", dtype=F64)
    zeta = (z[None] / 1000.0 - (lay[:, 1, None, None] + uni(-20.0, 20.0, NI, 1, n_cols))) / lay[:, 2, None, None]
    pk = lay[:, 0, None, None] * 10.0 ** uni(-0.3, 0.3, NI, 1, n_cols)
    ion = torch.clamp(pk * torch.exp(0.5 * (1.0 - zeta - torch.exp(-zeta))), min=1.0)
    m = {"ndensity_s": nd, "idensity_s": torch.cat([ion, ion.sum(0, keepdim=True)]),
         "velocity": torch.cat([50.0 * smooth(2), 2.0 * smooth(1)]), "vert_vel": smooth(NS),
         "ivel_up": 20.0 * smooth(1), "rho": (mass * nd).sum(0, keepdim=True)}
    mmm = (mass * nd).sum(0) / (nd.sum(0) + 1.0)
    m["temperature"] = (T / (mmm / synthetic.KB))[None]
    p = m["temperature"] * m["rho"]
    kc = synthetic.EDDY_COEF * torch.exp(0.3 * nrm(n_cols))
    p0, p1 = synthetic.EDDY_P0, synthetic.EDDY_P1
    m["eddy"] = torch.where(p > p0, kc, torch.where(p > p1, kc * (p - p1) / (p0 - p1), torch.zeros_like(p)))
    m["cos_lat"] = torch.cos(uni(-89.0, 89.0, n_cols) * (math.pi / 180.0))
    m["sza"] = uni(0.0, math.pi, n_cols)
    m["mlat"] = uni(-90.0, 90.0, n_cols)
    m.update(altitude=alt, gravity=grav, dalt_c=dalt, inv_r=inv_r)
    # EUV heating: 1e-8 K/s at 100 km scaled by density, in the units of Temperature
    m["heating"] = 1.0e-8 * m["rho"][:, 2:3] / m["rho"] / (mmm / synthetic.KB)[None]
    m["heating_scale"] = torch.exp(0.3 * nrm(n_cols))
    return {k: v.contiguous() for k, v in m.items()}


def _device_member(m, heating=False, outputs=False):
    t = {k: v for k, v in m.items() if heating or not k.startswith("heating")}
    if outputs:
        t["log_ns"], t["ndensity"] = torch.zeros_like(t["ndensity_s"]), torch.zeros_like(t["rho"])
    return vertical.DeviceMember(t["rho"].shape[1] - 4, t["rho"].shape[2], t)


def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["members"].split()]


# ------------------------------------------------------------------ blocks
def _blocks(case, seed):
    """HzBlocks of CUDA tensors: blocks_lon x blocks_lat blocks tiling the globe, ghost cells filled."""
    nl, nt, na, nbl, nbt = (case[k] for k in ("n_lons", "n_lats", "n_alts", "blocks_lon", "blocks_lat"))
    g, nb = _gen(seed, 77), nbl * nbt
    NI_, NJ, NK = nl + 4, nt + 4, na + 4
    dlon, dlat = 2 * math.pi / (nbl * nl), math.pi / (nbt * nt)

    def d(a):
        return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=F64)

    b = np.arange(nb)
    lon = d(((b % nbl) * nl)[:, None] + np.arange(-1, nl + 3) - 0.5) * dlon
    lat = d(((b // nbl) * nt)[:, None] + np.arange(-1, nt + 3) - 0.5) * dlat - math.pi / 2
    LON, LAT = lon[:, None, None, :], lat[:, None, :, None]

    def mod(amp, *lead):
        """Smooth fields on the sphere, one for each of `lead`: low-order modes with random phases."""
        a = 2 * math.pi * torch.rand(*lead, 4, generator=g, device="cuda", dtype=F64)
        a = a.reshape(1, *lead, 1, 1, 1, 4)
        lo, la = (x.reshape(nb, *([1] * len(lead)), 1, *x.shape[2:]) for x in (LON, LAT))
        p = (torch.cos(la) * torch.cos(lo + a[..., 0]) + 0.6 * torch.sin(2 * la) * torch.sin(2 * lo + a[..., 1]) +
             0.3 * torch.cos(3 * la) * torch.cos(3 * lo + a[..., 2]) + 0.2 * torch.sin(la + a[..., 3]))
        return amp * p.expand(nb, *lead, NK, NJ, NI_)

    col = _columns(1, na, seed, member=78)

    def prof(x):
        x = x[..., 0]
        return (x[0] if x.shape[0] == 1 else x).reshape(1, *(x.shape[:1] if x.shape[0] > 1 else ()), NK, 1, 1)

    A = {"temperature": prof(col["temperature"]) * (1 + mod(0.05))}
    nd = torch.full((nb, abi.NSPECIES_TOTAL, NK, NJ, NI_), 1e10, device="cuda", dtype=F64)
    nd[:, :NS] = prof(col["ndensity_s"]) * (1 + mod(0.2, NS))
    A["ndensity_s"] = nd
    mass = d(synthetic.MASS)
    A["rho"] = (nd[:, :NS] * mass[:, None, None, None]).sum(1)
    A["velocity"] = torch.cat([mod(60.0, 1), mod(40.0, 1), prof(col["velocity"])[:, 2:3] + mod(2.0, 1)], 1)
    A["vert_vel"] = prof(col["vert_vel"]) + mod(1.0, NS)
    ion = prof(col["idensity_s"][:NI]) * (1 + mod(0.3, NI))
    A["idensity_s"] = torch.cat([ion, ion.sum(1, keepdim=True)], 1)
    n1 = col["ndensity_s"]
    inv_vib = d(1.0 / (synthetic.VIBRATION - 2))[:, None, None]
    A["gamma"] = prof((n1 * inv_vib).sum(0, keepdim=True) * 2.0 / n1.sum(0, keepdim=True) + 1) * (1 + mod(0.005))
    A["ivelocity"] = torch.cat([mod(150.0, 1), mod(100.0, 1), mod(20.0, 1)], 1)
    A["ivelocity_par"] = torch.cat([mod(30.0, 1), mod(30.0, 1), mod(40.0, 1)], 1)
    cs = torch.sqrt(A["gamma"] * A["temperature"])
    A["cmax"] = (A["velocity"].abs() + cs[:, None])[:, :, 1:-1, 1:-1, 1:-1]
    R = (synthetic.RBODY + col["altitude"])[None, :, None, None].expand(nb, NK, NJ, NI_)
    A["radial_distance"], A["inv_radial_distance"] = R, 1 / R
    A["latitude"], A["cos_latitude"] = lat, torch.cos(lat)
    A["tan_latitude"] = torch.clamp(torch.tan(lat).abs(), max=100.0) * torch.sign(lat)
    cmx = torch.clamp(torch.cos(lat).abs(), min=0.01)
    cmx[:, 0], cmx[:, -1] = cmx[:, 1], cmx[:, -2]
    east, north = dlon * R * cmx[:, None, :, None], dlat * R
    for k, v in (("lon", east), ("lat", north)):
        A[f"inv_d{k}_dist_gb"], A[f"inv_d{k}_dist_fb"], A[f"d{k}_dist_fb"] = 1 / v, 1 / v, v
    for k, n, h in (("lon", nl, dlon), ("lat", nt, dlat)):  # uniform spacing h
        one = torch.ones(nb, n, device="cuda", dtype=F64)
        A[f"grad_{k}_m"], A[f"grad_{k}_0"], A[f"grad_{k}_p"] = -0.5 / h * one, 0 * one, 0.5 / h * one
    A["temp_source"] = torch.zeros(nb, na, nt, nl, device="cuda", dtype=F64)
    A["itemperature"] = A["temperature"] * (1.1 + mod(0.02))
    A["etemperature"] = A["temperature"] * (1.5 + mod(0.05))
    return horizontal.HzBlocks(nl, nt, na, nb, {k: v.clone(memory_format=torch.contiguous_format) for k, v in A.items()},
                               nbl, nbt)


# ------------------------------------------------------------------ GITM's own arrays
# (extra field extent, lower bounds) of the halo'd ModGITM arrays; a tensor of shape
# (block[, k], alt, lat, lon) holds the Fortran array (lon, lat, alt[, k], block)
_HALO = {"ndensity_s": 11, "idensity_s": 10, "velocity": 3, "ivelocity": 3, "vertical_velocity": 6, "log_ns": 6,
         "species_density": 20, "species_density_old": 20, "rho": 0, "temperature": 0, "ndensity": 0, "gamma": 0,
         "altitude": 0, "gravity": 0, "dalt": 0, "inv_r": 0, "mlatitude": 0, "mean_major_mass": 0, "temp_unit": 0}
_FORTRAN_OUT = ("ndensity_s", "idensity_s", "rho", "temperature", "velocity", "vertical_velocity", "log_ns", "ndensity",
                "species_density", "species_density_old")


def _fortran_columns(case, seed):
    """The columns of the blocks (lon fastest, then lat, then block); CosLatitude is one value per latitude row."""
    nl, nt, nb = case["n_lons"], case["n_lats"], case["blocks"]
    m = _columns(nl * nt * nb, case["n_alts"], seed)
    m["cos_lat"] = m["cos_lat"].reshape(nb, nt, nl)[:, :, :1].expand(nb, nt, nl).reshape(-1).contiguous()
    return m


def _producers(m):
    """Gamma, MeanMajorMass, TempUnit and cMax, as calc_pressure, calc_rates and calc_timestep leave them."""
    nd, N = m["ndensity_s"], m["ndensity_s"].sum(0, keepdim=True)
    w = torch.as_tensor(1.0 / (synthetic.VIBRATION - 2), device="cuda", dtype=F64)[:, None, None]
    mass = torch.as_tensor(synthetic.MASS, device="cuda", dtype=F64)[:, None, None]
    gamma = (nd * w).sum(0, keepdim=True) * 2.0 / N + 1
    mmm = (nd * mass).sum(0, keepdim=True) / (N + 1.0)
    cmax = m["vert_vel"].abs().max(0, keepdim=True).values + torch.sqrt(gamma * m["temperature"])
    return gamma, mmm, mmm / synthetic.KB, cmax


def _to_blocks(x, case):
    """[field, cell, column] -> (block, field, cell, lat, lon)."""
    f, G, _ = x.shape
    return x.reshape(f, G, case["blocks"], case["n_lats"], case["n_lons"]).permute(2, 0, 1, 3, 4)


def _fortran_arrays(case, seed):
    nl, nt, nb, na = case["n_lons"], case["n_lats"], case["blocks"], case["n_alts"]
    G, m = na + 4, _fortran_columns(case, seed)
    gamma, mmm, tu, cmax = _producers(m)
    A = {k: torch.zeros(nb, *([n] if n else []), G, nt + 4, nl + 4, device="cuda", dtype=F64) for k, n in _HALO.items()}
    for k, src, f0 in (("ndensity_s", m["ndensity_s"], 0), ("idensity_s", m["idensity_s"], 0), ("velocity", m["velocity"], 0),
                       ("vertical_velocity", m["vert_vel"], 0), ("ivelocity", m["ivel_up"], 2)):
        A[k][:, f0:f0 + src.shape[0], :, 2:-2, 2:-2] = _to_blocks(src, case)
    for k, src in (("rho", m["rho"]), ("temperature", m["temperature"]), ("gamma", gamma), ("mean_major_mass", mmm),
                   ("temp_unit", tu)):
        A[k][:, :, 2:-2, 2:-2] = _to_blocks(src, case)[:, 0]
    for k, src in (("altitude", "altitude"), ("gravity", "gravity"), ("dalt", "dalt_c"), ("inv_r", "inv_r")):
        A[k][:] = m[src][None, :, None, None]
    A["mlatitude"][:, na + 1, 2:-2, 2:-2] = m["mlat"].reshape(nb, nt, nl)
    A["cmax"] = torch.zeros(nb, 3, na + 2, nt + 2, nl + 2, device="cuda", dtype=F64)
    A["cmax"][:, 2, :, 1:-1, 1:-1] = _to_blocks(cmax, case)[:, 0, 1:-1]
    A["kappa_eddy"] = _to_blocks(m["eddy"], case)[:, 0].contiguous()
    A["cos_latitude"] = torch.ones(nb, nt + 4, device="cuda", dtype=F64)
    A["cos_latitude"][:, 2:-2] = m["cos_lat"].reshape(nb, nt, nl)[:, :, 0]
    A["sza"] = m["sza"].reshape(nb, nt, nl).contiguous()
    return A


def _fortran_struct(case, A):
    st = abi.GitmFortranState()
    st.n_lons, st.n_lats, st.n_alts, st.n_blocks = case["n_lons"], case["n_lats"], case["n_alts"], case["blocks"]
    for name in abi.FORTRAN_ARRAYS:
        t, fa = A[name], abi.GitmFArray()
        fa.data, s = abi.dptr(t.data_ptr()), t.stride()
        if name == "cos_latitude":
            strides, lower = (0, 1, 0, 0, s[0]), (1, -1, 1, 1, 1)
        elif name == "sza":
            strides, lower = (1, s[1], 0, 0, s[0]), (1, 1, 1, 1, 1)
        else:
            strides = (1, s[-2], s[-3], s[1] if t.dim() == 5 else 0, s[0])
            lower = {"cmax": (0, 0, 0, 1, 1), "kappa_eddy": (1, 1, -1, 1, 1)}.get(name, (-1, -1, -1, 1, 1))
        fa.stride[:], fa.lower[:] = strides, lower
        setattr(st, name, fa)
    return st


# ------------------------------------------------------------------ prepare and run
def _params(case):
    ausm = case.get("solver") == "ausm"
    return abi.default_params(solver=abi.SOLVER_AUSM if ausm else abi.SOLVER_RUSANOV)


def _hz_written(case, A):
    names = [k for k in horizontal.OUTPUTS if k != "temp_source"]
    return names + (["ivelocity_par", "itemperature", "etemperature"] if case["kind"] == "hz_step" else [])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "ctx": vertical.VerticalContext(_params(case))}
    if kind in ("steps", "ensemble"):
        sizes = _sizes(case) if kind == "ensemble" else [(case["n_alts"], case["cols"])]
        rng = np.random.default_rng(seed)
        cols = [_columns(n, a, seed, j, 0.0 if kind == "steps" else 100.0 * rng.standard_normal())
                for j, (a, n) in enumerate(sizes)]
        s["start"] = [c[k] for c in cols for k in STATE]
        s["members"] = [_device_member({k: v.clone() if k in STATE else v for k, v in c.items()}, heating=kind == "ensemble")
                        for c in cols]
        s["now"] = [m.tensors[k] for m in s["members"] for k in STATE]
        s["plan"] = vertical.Plan(s["ctx"], s["members"])
        if kind == "ensemble":
            s["plan"].set_config(threads=512, steps_per_launch=case["steps"])
        elif case["threads"]:
            s["plan"].set_config(threads=case["threads"], steps_per_launch=case["steps"])
        elif case["steps"] > 1:
            s["plan"].set_config(steps_per_launch=case["steps"])
    elif kind == "dropin":
        m = _columns(case["cols"], case["n_alts"], seed)
        s["start"] = [m[k].clone() for k in STATE]
        s["member"] = _device_member(m, outputs=True)
        s["now"] = [m[k] for k in STATE]
    elif kind == "fortran":
        s["arrays"] = _fortran_arrays(case, seed)
        s["names"] = ("ndensity_s", "idensity_s", "rho", "temperature", "velocity", "vertical_velocity")
        s["start"] = [s["arrays"][k].clone() for k in s["names"]]
        s["now"] = [s["arrays"][k] for k in s["names"]]
        s["struct"] = _fortran_struct(case, s["arrays"])
    elif kind == "host":
        m = _columns(case["cols"], case["n_alts"], seed)
        gamma, mmm, tu, cmax = _producers(m)
        host = {k: v.cpu().pin_memory().numpy() for k, v in m.items() if not k.startswith("heating")}
        host.update(gamma=gamma.cpu().numpy(), mean_major_mass=mmm.cpu().numpy(), temp_unit=tu.cpu().numpy(),
                    cmax=cmax.cpu().numpy())
        s["member"] = synthetic.Member(n_alts=case["n_alts"], n_cols=case["cols"], **host)
        for k in synthetic.Member.COEFFS:  # formed on the device, not passed
            setattr(s["member"], k, None)
    elif kind in ("adjoint", "rollout"):
        m = _columns(case["cols"], case["n_alts"], seed)
        s["state"] = {k: m[k].clone() for k in STATE}
        s["eddy"], s["scale"] = m["eddy"].clone(), m["heating_scale"].clone()
        s["runner"] = adjoint.StepRunner(s["ctx"], _device_member(m, heating=True), DT)
        s["bars"], s["level"] = _bars(case, m, seed)
    elif kind in ("hz", "hz_step"):
        s["blocks"] = _blocks(case, seed)
        A = s["blocks"].arrays
        s["now"] = [A[k] for k in _hz_written(case, A)]
        s["start"] = [t.clone() for t in s["now"]]
    elif kind == "cfl":
        m = _columns(case["cols"], case["n_alts"], seed)
        m["gamma"], m["cmax"] = _producers(m)[0], torch.zeros_like(m["rho"])
        s["member"] = _device_member(m)
    return s


def _bars(case, m, seed):
    """The step's output adjoints: unit-variance noise on each field's scale (adjoint), or the column weights of
    the O/N2 objective and its level (rollout)."""
    g = _gen(seed, 99)
    if case["kind"] == "rollout":
        w = torch.rand(case["cols"], generator=g, device="cuda", dtype=F64)
        return w, adjoint.level_of(m["altitude"].cpu(), 400e3)
    return [torch.randn(m[k].shape, generator=g, device="cuda", dtype=F64) / m[k].abs().mean(-1, keepdim=True).clamp_min(1.0e-30)
            for k in STATE], 0


def _differentiate(step, s_state, eddy, scale, bars, level, rollout):
    x = {k: v.detach().requires_grad_() for k, v in s_state.items()}
    e, h = eddy.detach().requires_grad_(), scale.detach().requires_grad_()
    out = step(x, e, h)
    wrt = [x[k] for k in STATE] + [e, h]
    if rollout:
        grads = torch.autograd.grad(adjoint.o_n2_objective(out["ndensity_s"], bars, level), wrt)
    else:
        grads = torch.autograd.grad([out[k] for k in STATE], wrt, bars)
    return {"out": {k: out[k].detach() for k in STATE},
            "grad": dict(zip((*STATE, "eddy", "heating_scale"), grads))}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("steps", "ensemble"):
        torch._foreach_copy_(s["now"], s["start"])
        s["plan"].advance(DT, case["steps"])
        return s["now"]
    if kind == "dropin":
        torch._foreach_copy_(s["now"], s["start"])
        vertical.advance_vertical_all(s["ctx"], s["member"], DT)
        t = s["member"].tensors
        return {k: t[k] for k in (*STATE, "log_ns", "ndensity")}
    if kind == "fortran":
        torch._foreach_copy_(s["now"], s["start"])
        rc = lib().gitm_vert_advance_fortran(s["ctx"].handle, C.byref(s["struct"]), 1, case["blocks"], DT, 1)
        if rc != abi.OK:
            raise vertical.GitmError(s["ctx"].last_error())
        return {k: s["arrays"][k] for k in _FORTRAN_OUT}
    if kind == "host":
        vertical.advance_vertical_all_host(s["ctx"], s["member"], DT_HOST)
        return {k: getattr(s["member"], k) for k in STATE}
    if kind == "adjoint":
        return _differentiate(lambda x, e, h: adjoint.vertical_step(s["runner"], x, e, h), s["state"], s["eddy"],
                              s["scale"], s["bars"], s["level"], False)
    if kind == "rollout":
        return _differentiate(lambda x, e, h: adjoint.rollout(s["runner"], x, case["steps"], case["every"], e, h),
                              s["state"], s["eddy"], s["scale"], s["bars"], s["level"], True)
    if kind in ("hz", "hz_step"):
        torch._foreach_copy_(s["now"], s["start"])
        if kind == "hz_step":
            horizontal.exchange_messages(s["ctx"], s["blocks"])
        horizontal.advance_horizontal(s["ctx"], s["blocks"], DT_HZ)
        if kind == "hz_step":
            horizontal.exchange_messages(s["ctx"], s["blocks"])
        return {k: s["blocks"].arrays[k] for k in (*_hz_written(case, None), "temp_source")}
    dt = vertical.calc_timestep_vertical(s["ctx"], s["member"])
    return {"dt": dt, "cmax": s["member"].tensors["cmax"]}


# ------------------------------------------------------------------ work
# flop-equivalents of one column-step at 50 altitudes (add, mul, div, sqrt = 1, exp, log, pow = 20), counted with
# the reference's statements; the other figures are counts of the same kind
_FLOPS_STEP = {"rusanov": 616627.0, "ausm": 1391515.0}
_FLOPS_HZ_CELL = 4 * (19 * 2 * 45.0 + 250.0)


def work(case):
    kind = case["kind"]
    if kind in ("hz", "hz_step"):
        planes = case["blocks_lon"] * case["blocks_lat"] * case["n_alts"]
        cells, ghosts = case["n_lons"] * case["n_lats"], (case["n_lons"] + 4) * (case["n_lats"] + 4)
        # state 19 fields + metrics and inputs 14 in, 20 interior fields out; the exchange moves 32 fields of the ring
        by = planes * 8.0 * (33 * ghosts + 21 * cells + (2 * 2 * 32 * (ghosts - cells) if kind == "hz_step" else 0))
        return {"bytes": by, "flops": planes * cells * _FLOPS_HZ_CELL}
    sizes = _sizes(case) if kind == "ensemble" else [(case["n_alts"], case["cols"] if "cols" in case else
                                                      case["n_lons"] * case["n_lats"] * case["blocks"])]
    cells = sum((a + 4.0) * n for a, n in sizes)
    if kind == "cfl":
        return {"bytes": 8.0 * cells * 10, "flops": 25.0 * cells}
    steps = case.get("steps", 1)
    flops = sum(_FLOPS_STEP[case.get("solver", "rusanov")] * a / 50.0 * n for a, n in sizes) * steps
    if kind in ("adjoint", "rollout"):
        # forward and reverse: twice the forward's operations again; state, its adjoint and the inputs in and out
        return {"bytes": 8.0 * cells * 27 * 4 * steps, "flops": 3.0 * flops}
    fields = 27 + 2 + 27 + (7 if kind == "dropin" else 0) + (4 + 4 + 7 + 30 if kind == "fortran" else 0)
    return {"bytes": 8.0 * cells * fields, "flops": flops}


# ------------------------------------------------------------------ the same in plain torch
_KB = 1.3807e-23
_AMU = 1.6726e-27
_MASS = [16 * _AMU, 32 * _AMU, 28 * _AMU, 14 * _AMU, 30 * _AMU, 4 * _AMU]
_D0 = [[0.000, 0.969, 0.969, 0.969, 0.715, 3.440], [0.969, 0.000, 0.715, 0.969, 0.715, 3.208],
       [0.969, 0.715, 0.000, 0.969, 0.527, 2.939], [0.969, 0.969, 0.969, 0.000, 0.969, 2.939],
       [0.715, 0.715, 0.527, 0.969, 0.000, 2.939], [3.440, 3.208, 2.939, 2.939, 2.939, 0.000]]
_DE = [[0, .774, .774, .774, .750, .749], [.774, 0, .750, .774, .750, .710], [.774, .750, 0, .774, .810, .718],
       [.774, .774, .774, 0, .774, .718], [.750, .750, .810, .774, 0, .718], [.749, .710, .718, .718, .718, 0]]
_PHOTO = (3, 4)
_THERMAL = [0, 0, 0, 0, 0, -0.38]
_OMEGA = 2.0 * math.pi / 86400.0
_F1, _F2 = 0.6250000, 0.0416667
# rows of the stage state: LogNS 0-5, VertVel 6-11, Temp, Vel east / north / up, ions 16-24, LogRho 25
_W, _T, _VE, _VN, _VU, _I, _LR = 6, 12, 13, 14, 15, 16, 25


def _col(v, like):
    return torch.as_tensor(v, device=like.device, dtype=F64)


class _Mesh:
    """Grid coefficients of one member."""

    def __init__(self, m):
        alt = m["altitude"].cpu().numpy()
        G = alt.shape[0]
        nA = self.nA = G - 4
        d = np.empty(G)
        d[1:] = np.diff(alt)
        d[0] = d[1]
        self.d = d
        one = np.vectorize(lambda i: d[i + 1])
        mc = np.zeros((5, nA))
        i = np.arange(1, nA + 1)
        h1, h2, h3, h4 = one(i - 1), one(i), one(i + 1), one(i + 2)
        H2, H3, H4 = h1 + h2, h1 + h2 + h3, h1 + h2 + h3 + h4
        mc[0] = h2 * h3 * (h3 + h4) / (h1 * H2 * H3 * H4)
        mc[1] = -H2 * h3 * (h3 + h4) / (h1 * h2 * (h2 + h3) * (h2 + h3 + h4))
        mc[2] = (h2 * h3 * (h3 + h4) + H2 * h3 * (h3 + h4) - H2 * h2 * (h3 + h4) - H2 * h2 * h3) / (H2 * h2 * h3 * (h3 + h4))
        mc[3] = H2 * h2 * (h4 + h3) / (H3 * (h2 + h3) * h3 * h4)
        mc[4] = -H2 * h2 * h3 / (H4 * (h2 + h3 + h4) * (h3 + h4) * h4)

        def onesided(h, sign):
            a, b, c, e = h
            M1, M2, M3, M4 = a, a + b, a + b + c, a + b + c + e
            return [sign * v for v in (-(M2 * M3 * M4 + M1 * M3 * M4 + M1 * M2 * M4 + M1 * M2 * M3) / (M1 * M2 * M3 * M4),
                                       M2 * M3 * M4 / (a * b * (b + c) * (b + c + e)), -M1 * M3 * M4 / (M2 * b * c * (c + e)),
                                       M1 * M2 * M4 / (M3 * (c + b) * c * e), -M1 * M2 * M3 / (M4 * (b + c + e) * (c + e) * e))]

        self.lo = [onesided(d[3 - k:7 - k], 1.0) for k in (0, 1)]
        self.up = [onesided(d[nA + 1 + k - np.arange(4)], -1.0) for k in (0, 1)]
        t = m["rho"]
        self.dA, self.mc = _col(d, t)[:, None], _col(mc, t)[:, :, None]
        self.invr, self.grav, self.dc = m["inv_r"][:, None], m["gravity"][:, None], m["dalt_c"][:, None]
        self.R, self.alt = 1.0 / self.invr, m["altitude"][:, None]
        self.mass = _col(_MASS, t)[:, None, None]


def _mc(u, d, beta=2.0):
    m = torch.minimum(torch.minimum((beta * u).abs(), (beta * d).abs()), ((u + d) * 0.5).abs())
    z = torch.zeros_like(m)
    return torch.where((u > 0) & (d > 0), m, torch.where((u <= 0) & (d < 0), -m, z))


def _slopes2(v, g):
    """2nd-order limited slopes on cells 0..nAlts+1 (last axes: cell -1..nAlts+2, column)."""
    d = (v[..., 1:, :] - v[..., :-1, :]) / g.dA[1:]
    return _mc(d[..., 1:, :], d[..., :-1, :])


def _slopes4(v, g):
    """The same with the 4th-order differences on interior cells."""
    d = v[..., 1:, :] - v[..., :-1, :]
    d4 = 2.0 / g.dA[2:-1] * (_F1 * d[..., 1:-1, :] - _F2 * (v[..., 3:, :] - v[..., :-3, :]))
    d2 = d / g.dA[1:]
    e0, e1 = _mc(d2[..., 1:2, :], d2[..., 0:1, :]), _mc(d2[..., -1:, :], d2[..., -2:-1, :])
    return torch.cat([e0, _mc(d4[..., 1:, :], d4[..., :-1, :]), e1], -2)


def _faces(v, sl, g):
    """Left and right states at faces 1..nAlts+1 (face i lies between cells i-1 and i)."""
    h = 0.5 * g.dA[2:-1]
    return v[..., 1:-2, :] + sl[..., :-1, :] * h, v[..., 2:-1, :] - sl[..., 1:, :] * h


def _rusanov(v, sl, g, cm):
    L, R = _faces(v, sl, g)
    idc = 1.0 / g.dc[2:-2]
    fl = 0.5 * torch.maximum(cm[1:-2], cm[2:-1]) * (R - L)
    s = L + R
    return 0.5 * (s[..., 1:, :] - s[..., :-1, :]) * idc, (fl[..., 1:, :] - fl[..., :-1, :]) * idc


def _boundaries(X, pre, g, co):
    """set_vertical_bcs with the default switches: X [26, G, columns] with its interior cells set; `pre` holds the
    ghost values before the call."""
    nA, d = g.nA, g.d
    x = X[:, 2:-2]
    T0 = pre[_T, 1]
    zero = torch.zeros_like(T0)

    def one_sided(c, v):
        return sum(c[q] * v[q] for q in range(5))

    eg = g.grav + co["cent"] * g.R
    lo0, lo1, up1, up2 = {}, {}, {}, {}
    for s in range(NS):
        if s in _PHOTO:
            prev = [x[s, q] for q in range(5)]
            for k, to in ((0, lo0), (1, lo1)):
                gr = one_sided(g.lo[k], prev)
                v = torch.where(gr <= 0, prev[0], prev[0] - d[2 - k] * gr)
                v = torch.where(v < prev[0] - 0.333, prev[0] - 0.333, v) if s == 4 else v
                to[s] = v
                prev = [v] + prev[:4]
        else:
            lo0[s] = pre[s, 1]
            ish = -0.5 * (eg[0] + eg[1]) * (0.5 * (co["mmm"][0] + co["mmm"][1])) / (T0 * _KB)
            lo1[s] = pre[s, 1] if s == 0 else pre[s, 1] + ish * d[0]
        prev = [x[_W + s, q] for q in range(5)]
        for k, to in ((0, lo0), (1, lo1)):
            v = prev[0] - d[2 - k] * one_sided(g.lo[k], prev)
            to[_W + s] = v
            prev = [v] + prev[:4]
        den = x[_T, -1] * _KB
        up1[s] = x[s, -1] + 0.5 * (eg[nA + 1] + eg[nA + 2]) * _MASS[s] / den * d[nA + 2]
        up2[s] = up1[s] + 0.5 * (eg[nA + 2] + eg[nA + 3]) * _MASS[s] / den * d[nA + 3]
        wn = x[_W + s, -1]
        flip = wn < 0 if s in _PHOTO else torch.zeros_like(wn, dtype=torch.bool)
        up1[_W + s], up2[_W + s] = torch.where(flip, -wn, wn), torch.where(flip, -x[_W + s, -2], wn)
    for lo in (lo0, lo1):
        ms = [_MASS[s] * torch.exp(lo[s]) for s in range(NS)]
        lo[_LR], lo[_VU] = torch.log(sum(ms)), sum(ms[s] * lo[_W + s] for s in range(NS)) / sum(ms)
        lo[_T], lo[_VE], lo[_VN] = T0, zero, zero
    for s in _PHOTO:
        flip = x[_W + s, 0] > 0
        for lo in (lo0, lo1):
            lo[_W + s] = torch.where(flip, -x[_W + s, 0], lo[_W + s])
    tec = (_col(d[2:-2], T0)[:, None] * x[_I]).sum(0)
    hold = (tec / 1e16 < 2.0) & co["plasma"]
    for s in range(NI):
        r = _I + s
        lo0[r] = lo1[r] = x[r, 0]
        n = [torch.log(x[r, nA - 1 - q]) for q in range(5)]
        old = [torch.log(pre[r, -2]), torch.log(pre[r, -1])]
        for k, to in ((0, up1), (1, up2)):
            gr = one_sided(g.up[k], n)
            gr = torch.minimum(gr, -(0.001 * old[k] / d[nA + 1]))
            y = n[0] + gr * d[nA + 2 + k]
            to[r] = torch.where(hold, pre[r, -2 + k], torch.exp(y))
            n = [torch.where(hold, old[k], y)] + n[:4]
    for up in (up1, up2):
        up[_T], up[_VE], up[_VN], up[_VU] = x[_T, -1], x[_VE, -1], x[_VN, -1], x[_VU, -1].abs()
        up[_LR] = torch.log(sum(_MASS[s] * torch.exp(up[s]) for s in range(NS)))
    rows = [torch.stack([v[f] for f in range(26)])[:, None] for v in (lo1, lo0, up1, up2)]
    return torch.cat([*rows[:2], x, *rows[2:]], 1)


def _friction(dt, ns, T, eddy, glc, w):
    lt = torch.log(T)
    a = [[None] * NS for _ in range(NS)]
    for r in range(NS):
        c = [None if q == r else dt * (1e-2 * _KB / (_MASS[r] * 1e17 * _D0[r][q])) * ns[q] * torch.exp((1 - _DE[r][q]) * lt)
             for q in range(NS)]
        for q in range(NS):
            a[r][q] = 1.0 + sum(v for v in c if v is not None) if q == r else -c[q]
    w = list(w)
    for p in range(NS):
        for r in range(p + 1, NS):
            l = a[r][p] / a[p][p]
            for q in range(p + 1, NS):
                a[r][q] = a[r][q] - l * a[p][q]
            w[r] = w[r] - l * w[p]
    for r in reversed(range(NS)):
        w[r] = (w[r] - sum(a[r][q] * w[q] for q in range(r + 1, NS))) / a[r][r] if r < NS - 1 else w[r] / a[r][r]
    return torch.stack(w) - eddy * glc


def _grad_log_cons(X, g):
    lc = torch.log(g.mass) + X[:NS] - X[_LR]
    return sum(g.mc[q] * lc[:, q:q + g.nA] for q in range(5))


def _stage(X, g, co, dt):
    """New - state on the interior cells: [26, nAlts, columns] (the passive ions stay)."""
    i = slice(2, -2)
    x = X[:, i]
    gr, df = _rusanov(X[:18], _slopes4(X[:18], g), g, co["cmax"])
    T, VE, VN, VU = x[_T], x[_VE], x[_VN], x[_VU]
    invr, km = g.invr[i], _KB / g.mass
    vel = -dt * VU * gr[_VE:_VU] + dt * df[_VE:_VU]
    dT = -dt * (VU * gr[_T] + (co["gamma"][i] - 1.0) * T * (gr[_VU] + 2 * VU * invr)) + dt * df[_T]
    ion = -dt * co["ivup"][i] * gr[_I:] + dt * df[_I:]
    Ws, gL, gW = x[_W:_T], gr[:NS], gr[_W:_T]
    dl = -dt * (gW + 2 * Ws * invr + Ws * gL) + dt * df[:NS]
    nlr = torch.log((g.mass * torch.exp(x[:NS] + dl)).sum(0))
    w = Ws - dt * (Ws * gW - (VN * VN + VE * VE) * invr + T * gL * km + gr[_T] * km - g.grav[i]) + dt * df[_W:_T] - Ws * 1e-9
    w = w + dt * (co["cent"] * g.R[i] + co["cori"] * VE) - dt * (_col(_THERMAL, T)[:, None, None] * km) * gr[_T]
    ns = torch.exp(x[:NS])
    w = torch.clamp(_friction(dt, ns, T, co["eddy"][i], _grad_log_cons(X, g), w), -1000.0, 1000.0)
    vu = (w * g.mass * ns).sum(0) * torch.exp(-x[_LR])
    return torch.cat([dl, w - Ws, dT[None], vel, (vu - VU)[None], ion, torch.zeros_like(x[_I + NADV:_LR]), (nlr - x[_LR])[None]])


def _ausm_stage(X, g, co, dt):
    """The AUSM stage: New - state on the interior cells."""
    i, nA = slice(2, -2), g.nA
    x = X[:, i]
    T, VE, VN, VU = x[_T], x[_VE], x[_VN], x[_VU]
    gr, df = _rusanov(X[_T:18], _slopes4(X[_T:18], g), g, co["cmax"])
    ion = -dt * co["ivup"][i] * gr[_I - _T:] + dt * df[_I - _T:]
    lT = torch.log(X[_T])
    eg = g.grav + co["cent"] * g.R
    # the hydrostatic background: log HydroNS(i) T(i) above cell 0, and below it from the mean major mass
    q = (g.dA[2:] * 0.5 * (eg[2:] + eg[1:-1]) / (_KB * 0.5 * (X[_T, 2:] + X[_T, 1:-1]))).cumsum(0)
    below = g.dA[0] * -0.5 * (co["mmm"][0] + co["mmm"][1]) * 0.5 * (eg[0] + eg[1]) / (_KB * 0.5 * (X[_T, 0] + X[_T, 1]))
    z = torch.zeros_like(below)[None, None]
    hq = torch.cat([below[None, None].expand(NS, -1, -1), z.expand(NS, -1, -1), g.mass * q], 1)
    base = X[:NS, 1:2] + lT[1]

    def face(v):
        sl = _slopes2(v, g)
        return v[..., 1:-2, :] + sl[..., :-1, :] * (0.5 * g.dA[1:-2]), v[..., 2:-1, :] - sl[..., 1:, :] * (0.5 * g.dA[2:-1])

    logk = math.log(_KB)
    rho = [torch.exp(torch.log(g.mass) + v) for v in face(X[:NS])]
    ps = [torch.exp(logk + v) for v in face(X[:NS] + lT)]
    hp = [torch.exp(base + logk + v) for v in face(hq)]
    ws, E, N, gam = face(X[_W:_T]), face(X[_VE]), face(X[_VN]), face(co["gamma"])
    RHO, P = [v.sum(0) for v in rho], [v.sum(0) for v in ps]
    U = [(rho[k] * ws[k]).sum(0) / RHO[k] for k in (0, 1)]
    K = [U[k] ** 2 + E[k] ** 2 + N[k] ** 2 for k in (0, 1)]
    ss = [torch.sqrt(2.0 * (gam[k] - 1.0) / (gam[k] + 1.0) * (0.5 * K[k] + gam[k] / (gam[k] - 1.0) * P[k] / RHO[k]))
          for k in (0, 1)]
    cs = torch.minimum(ss[0] ** 2 / torch.maximum(ss[0], U[0]), ss[1] ** 2 / torch.maximum(ss[1], -U[1]))
    R_lo, R_hi = 0.5 * (g.R[i] + g.R[1:-3]), 0.5 * (g.R[i] + g.R[3:-1])
    A_lo, A_hi, vol = R_lo ** 2, R_hi ** 2, (R_hi ** 3 - R_lo ** 3) / 3.0
    th = torch.tanh((g.alt[i] - 160.0e3) / 15.0e3)

    def between(lo, hi):
        return torch.exp(math.log(lo) + 0.5 * (math.log(hi) - math.log(lo)) * (1.0 + th))

    kp, ku, dc = between(1e-19, 1e-9), between(0.25, 0.50), g.dc[i]
    ns = torch.exp(x[:NS])
    rs = g.mass * ns
    dev = rs - g.mass * torch.exp(base - lT[i] + hq[:, i])
    sub = ~((dev.abs() / rs) > 1.0)

    def flux(f):
        """Species fluxes at one face of each cell (its lower or upper one), with the cell's own coefficients."""
        rl, rr, pl, pr, hl, hr, wl, wr = (v[k][:, f] for v in (rho, ps, hp, ws) for k in (0, 1))
        c = cs[f]
        Ml, Mr = wl / c, wr / c
        M2 = 0.5 * (Ml * Ml + Mr * Mr)
        M0 = torch.sqrt(torch.clamp(M2, 1e-19, 1.0))
        fa = M0 * (2.0 - M0)
        pos = torch.where(Ml.abs() >= 1, 0.5 * (Ml + Ml.abs()), 0.25 * (Ml + 1) ** 2 * (1.0 + 0.5 * (Ml - 1) ** 2))
        neg = torch.where(Mr.abs() >= 1, 0.5 * (Mr - Mr.abs()), -0.25 * (Mr - 1) ** 2 * (1.0 + 0.5 * (Mr + 1) ** 2))
        dp = torch.where(sub, (pr - hr) - (pl - hl), pr - pl)
        mp = kp * torch.clamp(1.0 - M2, min=0.0) * dp / (0.5 * (rl + rr) * c * (fa * c + dc / dt))
        nv = c * (pos + neg - mp)
        pn = torch.where(sub, 0.5 * (pl + pr) - 0.5 * (hl + hr), 0.5 * (pl + pr)) - 0.5 * ku * c * (rr * wr - rl * wl)
        up = nv >= 0
        rf = torch.where(up, rl, rr) * nv
        bulk = ((rl + rr) * nv / (RHO[0][f] + RHO[1][f])).sum(0)

        def pick(a, b):
            return torch.where(bulk >= 0, a, b)

        r, p_, kk, gg = (pick(v[0][f], v[1][f]) for v in (RHO, P, K, gam))
        return (rf, torch.where(up, wl, wr) * rf, pn, (p_ / (gg - 1.0) + 0.5 * r * kk + p_) * bulk,
                r * pick(E[0][f], E[1][f]) * bulk, r * pick(N[0][f], N[1][f]) * bulk)

    lo, hi = flux(slice(0, nA)), flux(slice(1, nA + 1))
    div = [(A_hi * b - A_lo * a) / vol for a, b in zip(lo, hi)]
    nrs = rs - dt * div[0]
    mom = rs * x[_W:_T] - dt * (div[1] + (hi[2] - lo[2]) / dc) + dt * torch.where(sub, dev, rs) * eg[i]
    w = mom / nrs + dt * (VN * VN + VE * VE) * g.invr[i] + dt * co["cori"] * VE
    w = w - dt * _col(_THERMAL, T)[:, None, None] * _KB * gr[0] / g.mass
    nns, nrho = nrs / g.mass, nrs.sum(0)
    w = torch.clamp(_friction(dt, nns, T, co["eddy"][i], _grad_log_cons(X, g), w), -1000.0, 1000.0)
    vu = (w * nrs).sum(0) / nrho
    R0 = torch.exp(x[_LR])
    damp = 0.35 * torch.exp(-(g.alt[i] - g.alt[1]) / 45.0e3)
    ve = (R0 * VE - dt * div[4]) / nrho + damp * dt * df[1]
    vn = (R0 * VN - dt * div[5]) / nrho + damp * dt * df[2]
    gm1 = co["gamma"][i] - 1.0
    en = ns.sum(0) * _KB * T / gm1 + 0.5 * R0 * (VU * VU + VN * VN + VE * VE) - dt * div[3] + dt * R0 * VU * eg[i]
    t = (en - 0.5 * nrho * (vu * vu + vn * vn + ve * ve)) * gm1 / (_KB * nns.sum(0))
    new = torch.cat([torch.log(nns), w, torch.stack([t, ve, vn, vu])])
    return torch.cat([new - x[:_I], ion, torch.zeros_like(x[_I + NADV:_LR]), (torch.log(nrho) - x[_LR])[None]])


def _step(m, g, dt, ausm=False, heating=False):
    """One step of every column: the new state arrays."""
    nd, ww, temp = m["ndensity_s"], m["vert_vel"], m["temperature"][0]
    n = nd.sum(0)
    gamma = (nd * _col([1 / 3, 1 / 5, 1 / 5, 1 / 3, 1 / 5, 1 / 3], nd)[:, None, None]).sum(0) * 2.0 / n + 1
    mmm = (g.mass * nd).sum(0) / (n + 1.0)
    tu = mmm / _KB
    cl = m["cos_lat"]
    night = (m["sza"] > math.pi / 2) & (((m["mlat"] > 30) & (m["mlat"] < 70)) | ((m["mlat"] > -60) & (m["mlat"] < -30)))
    co = {"gamma": gamma, "mmm": mmm, "cmax": ww.abs().max(0).values + torch.sqrt(gamma * temp), "ivup": m["ivel_up"][0],
          "eddy": m["eddy"][0], "cent": (cl * _OMEGA) ** 2, "cori": 2 * cl * _OMEGA, "plasma": night}
    X = torch.cat([torch.log(nd), ww, (temp * tu)[None], m["velocity"], m["idensity_s"][:NI], torch.log(m["rho"])])
    O = X = _boundaries(X, X, g, co)
    lo, hi, x = O[:, :2], O[:, -2:], O[:, 2:-2]

    def at(inner):
        Y = torch.cat([lo, inner, hi], 1)
        return _boundaries(Y, Y, g, co)

    if ausm:
        Y = [x]
        for f in (0.5, 0.5, 1.0):
            Y.append(x + _ausm_stage(X, g, co, f * dt))
            X = at(Y[-1])
        X = at((-Y[0] + Y[1] + 2 * Y[2] + Y[3] + _ausm_stage(X, g, co, 0.5 * dt)) / 3.0)
    else:
        acc = 0
        for wt, f in ((1, 0.5), (2, 0.5), (2, 1.0), (1, None)):
            K = _stage(X, g, co, dt)
            acc = acc + wt * K
            X = at(x + (f * K if f else acc / 6.0))
    t = X[_T] / tu
    if heating:
        add = dt * m["heating_scale"] * m["heating"][0]
        t = t + torch.cat([torch.zeros_like(add[:2]), add[2:-2], torch.zeros_like(add[:2])])
    ion = X[_I:_LR]
    ion = torch.cat([ion[:, :2], torch.clamp(ion[:, 2:-2], min=1.0), ion[:, -2:]], 1)
    return {"ndensity_s": torch.exp(X[:NS]), "idensity_s": torch.cat([ion, ion.sum(0, keepdim=True)]),
            "rho": torch.exp(X[_LR:]), "temperature": t[None], "velocity": X[_VE:_I], "vert_vel": X[_W:_T],
            "log_ns": X[:NS]}


def _steps(m, n, dt, **kw):
    g = _Mesh(m)
    out = {}
    for _ in range(n):
        out = _step(m, g, dt, **kw)
        m = {**m, **{k: out[k] for k in STATE}}
    return out


def _hz_sweep(V, IF, DF, CM, inv, axis):
    """Gradient and Rusanov diffusion along one axis (0: lon, 1: lat) at the interior cells; V [.., lat, lon]."""
    def sw(a):
        return a.transpose(-1, -2) if axis else a

    V, IF, DF, CM, inv = sw(V), sw(IF), sw(DF), sw(CM), sw(inv)
    V, IF, DF, CM = V[..., 2:-2, :], IF[..., 2:-2, :], DF[..., 2:-2, :], CM[..., 1:-1, :]
    d = V[..., 1:] - V[..., :-1]
    d2 = d * IF[..., 1:]
    d4 = 2 * IF[..., 2:-1] * (_F1 * d[..., 1:-1] - _F2 * (V[..., 3:] - V[..., :-3]))
    up, dn = torch.cat([d4, d2[..., -1:]], -1), torch.cat([d2[..., :1], d4], -1)
    sl = _mc(up, dn)
    L, R = V[..., 1:-2] + 0.5 * sl[..., :-1] * DF[..., 2:-1], V[..., 2:-1] - 0.5 * sl[..., 1:] * DF[..., 2:-1]
    fl = 0.5 * torch.maximum(CM[..., :-1], CM[..., 1:]) * (R - L)
    s = L + R
    return sw(0.5 * (s[..., 1:] - s[..., :-1]) * inv), sw((fl[..., 1:] - fl[..., :-1]) * inv)


def _hz_advance(A, dt):
    """advance_horizontal on every block, in place."""
    k = slice(2, -2)
    c = (slice(None), slice(None), k, k, k)

    def p(a):
        return a[:, None, k] if a.dim() == 4 else a[:, :, k]

    S = torch.cat([p(A["rho"]), p(A["temperature"]), p(A["velocity"]), p(A["ndensity_s"])[:, :NS], p(A["vert_vel"]),
                   p(A["idensity_s"])[:, :NADV]], 1)
    O, new, acc = S[..., 2:-2, 2:-2].clone(), None, 0
    inner = [a[:, None][c] for a in (A["gamma"], A["inv_radial_distance"], A["radial_distance"])]
    gamma, invr, rr = (a[:, 0] for a in inner)
    sin, cos, tan = (a[:, None, 2:-2, None] for a in (torch.sin(A["latitude"]), A["cos_latitude"], A["tan_latitude"]))
    met = {}
    for ax, n in ((0, "lon"), (1, "lat")):
        met[ax] = [p(A[f"inv_d{n}_dist_fb"]), p(A[f"d{n}_dist_fb"]), A["cmax"][:, ax:ax + 1, 1:-1],
                   A[f"inv_d{n}_dist_gb"][:, None][c]]
    IE, IN = A["ivelocity"][c][:, 0:1], A["ivelocity"][c][:, 1:2]
    for wt, f in ((1, 0.5), (2, 0.5), (2, 1.0), (1, None)):
        gE, dE = _hz_sweep(S, *met[0], 0)
        gN, dN = _hz_sweep(S, *met[1], 1)
        x = S[..., 2:-2, 2:-2]
        r, T, VE, VN, VU = (x[:, q] for q in range(5))
        div = gN[:, 3] + gE[:, 2] - tan * VN * invr
        adv = (VN[:, None] * gN + VE[:, None] * gE)
        rhs = adv.clone()
        rhs[:, 0] += r * div
        rhs[:, 1] += (gamma - 1) * T * div
        rhs[:, 2] += VE * (VU - tan * VN) * invr + gE[:, 1] + gE[:, 0] * T / r - (sin * 2 * _OMEGA * VN - cos * 2 * _OMEGA * VU)
        rhs[:, 3] += ((VN * VU + tan * VE * VE) * invr + gN[:, 1] + gN[:, 0] * T / r +
                      _OMEGA ** 2 * cos * sin * rr + sin * 2 * _OMEGA * VE)
        rhs[:, 5:5 + NS] += x[:, 5:5 + NS] * div[:, None]
        rhs[:, 5 + 2 * NS:] = gN[:, 5 + 2 * NS:] * IN + gE[:, 5 + 2 * NS:] * IE
        K = -dt * rhs + dt * (dE + dN)
        acc = acc + wt * K
        new = O + (f * K if f else acc / 6.0)
        S = S.clone()
        S[..., 2:-2, 2:-2] = new
    A["temp_source"].copy_(new[:, 1] - O[:, 1])
    A["rho"][:, k, k, k], A["temperature"][:, k, k, k] = new[:, 0], new[:, 1]
    A["velocity"][c], A["vert_vel"][c] = new[:, 2:5], new[:, 5 + NS:5 + 2 * NS]
    A["ndensity_s"][:, :NS][c] = new[:, 5:5 + NS]
    # the divergence of the parallel ion flow
    V = A["ivelocity_par"]
    glo, gla = ([A[f"grad_{n}_{q}"][:, None] for q in "m0p"] for n in ("lon", "lat"))
    E, N, U = (V[:, q] for q in range(3))
    D = sum(glo[q][:, :, None, :] * E[:, k, k, 1 + q:E.shape[-1] - 3 + q] for q in range(3)) * invr / torch.clamp(cos, min=0.17)
    D = D + sum(gla[q][:, :, :, None] * N[:, k, 1 + q:N.shape[-2] - 3 + q, k] for q in range(3)) * invr
    D = D - torch.clamp(tan, -5.0, 5.0) * N[:, k, k, k] * invr
    R = A["radial_distance"][:, :, k, k]
    up, dn = R[:, 3:-1] - R[:, 2:-2], R[:, 2:-2] - R[:, 1:-3]
    q2, Uc = (dn / up) ** 2, U[:, :, k, k]
    D = D + (q2 * Uc[:, 3:-1] - Uc[:, 1:-3] - (q2 - 1) * Uc[:, 2:-2]) / (dn * (1 + dn / up)) + 2 * Uc[:, 2:-2] * invr
    D = (D * cos)[:, None]
    A["idensity_s"][:, :NADV][c] = torch.clamp(new[:, 5 + 2 * NS:], min=1.0e2) / (1 + dt * D)
    A["idensity_s"][:, NI] = A["idensity_s"][:, :NI].sum(1)


def _hz_exchange(A, case):
    """exchange_messages_sphere with both poles connected, in place."""
    nl, nt, nbl, nbt = (case[k] for k in ("n_lons", "n_lats", "blocks_lon", "blocks_lat"))
    nb, NL, NT = nbl * nbt, nl * nbl, nt * nbt
    b, j, i = np.meshgrid(np.arange(nb), np.arange(-1, nt + 3), np.arange(-1, nl + 3), indexing="ij")
    gi, gj = (b % nbl) * nl + i, (b // nbl) * nt + j
    over = (gj < 1) | (gj > NT)
    gj = np.where(gj < 1, 1 - gj, np.where(gj > NT, 2 * NT + 1 - gj, gj))
    gi = (gi + np.where(over, NL // 2, 0) - 1) % NL
    sb = ((gj - 1) // nt) * nbl + gi // nl
    sj, si = (gj - 1) % nt + 2, gi % nl + 2
    sb, sj, si = (torch.as_tensor(v, device="cuda") for v in (sb, sj, si))
    k = slice(2, -2)
    for name, n in (("rho", 0), ("velocity", 3), ("vert_vel", NS), ("ndensity_s", NS), ("temperature", 0),
                    ("itemperature", 0), ("etemperature", 0), ("idensity_s", NI + 1), ("ivelocity_par", 3)):
        a = A[name] if n else A[name][:, None]
        for f in range(max(n, 1)):
            src = a[:, f, k].permute(0, 2, 3, 1).contiguous()
            a[:, f, k] = src[sb, sj, si].permute(0, 3, 1, 2)
    for a in (A["velocity"], A["ivelocity_par"]):
        a[:nbl, :2, :, :2] *= -1
        a[-nbl:, :2, :, -2:] *= -1


def exact(case, seed):
    kind = case["kind"]
    if kind in ("adjoint", "rollout"):
        return _exact_gradients(case, seed)
    with torch.no_grad():
        if kind in ("steps", "ensemble"):
            sizes = _sizes(case) if kind == "ensemble" else [(case["n_alts"], case["cols"])]
            rng, out = np.random.default_rng(seed), []
            for j, (a, n) in enumerate(sizes):
                m = _columns(n, a, seed, j, 0.0 if kind == "steps" else 100.0 * rng.standard_normal())
                o = _steps(m, case["steps"], DT, ausm=case.get("solver") == "ausm", heating=kind == "ensemble")
                out += [o[k] for k in STATE]
            return out
        if kind in ("dropin", "host"):
            o = _steps(_columns(case["cols"], case["n_alts"], seed), 1, DT if kind == "dropin" else DT_HOST)
            if kind == "host":
                return {k: o[k].cpu().numpy() for k in STATE}
            return {**{k: o[k] for k in (*STATE, "log_ns")}, "ndensity": o["ndensity_s"].sum(0, keepdim=True)}
        if kind == "fortran":
            return _exact_fortran(case, seed)
        if kind in ("hz", "hz_step"):
            A = _blocks(case, seed).arrays
            if kind == "hz_step":
                _hz_exchange(A, case)
            _hz_advance(A, DT_HZ)
            if kind == "hz_step":
                _hz_exchange(A, case)
            return {k: A[k] for k in (*_hz_written(case, None), "temp_source")}
        m = _columns(case["cols"], case["n_alts"], seed)
        gamma = _producers(m)[0][0]
        snd = torch.sqrt(gamma * m["temperature"][0])
        cm = m["vert_vel"].abs().max(0).values + snd
        dz = m["dalt_c"][2:-2, None]
        fast = torch.maximum((cm[2:-2] / dz).max(), ((m["ivel_up"][0].abs() + snd)[2:-2] / dz).max())
        cmax = torch.zeros_like(m["rho"])
        cmax[0, 1:-1] = cm[1:-1]
        return {"dt": float(0.75 / fast), "cmax": cmax}


def _exact_fortran(case, seed):
    A, m = _fortran_arrays(case, seed), _fortran_columns(case, seed)
    o = _steps(m, 1, DT)
    A["species_density_old"][:, :NS, :, 2:-2, 2:-2] = _to_blocks(m["ndensity_s"], case)
    A["species_density_old"][:, 11:20, :, 2:-2, 2:-2] = _to_blocks(m["idensity_s"][:NI], case)
    for k, src, f0 in (("ndensity_s", "ndensity_s", 0), ("idensity_s", "idensity_s", 0), ("velocity", "velocity", 0),
                       ("vertical_velocity", "vert_vel", 0), ("log_ns", "log_ns", 0), ("species_density", "ndensity_s", 0)):
        A[k][:, f0:f0 + o[src].shape[0], :, 2:-2, 2:-2] = _to_blocks(o[src], case)
    A["species_density"][:, 11:20, :, 2:-2, 2:-2] = _to_blocks(o["idensity_s"][:NI], case)
    for k, v in (("rho", o["rho"]), ("temperature", o["temperature"]), ("ndensity", o["ndensity_s"].sum(0, keepdim=True))):
        A[k][:, :, 2:-2, 2:-2] = _to_blocks(v, case)[:, 0]
    return {k: A[k] for k in _FORTRAN_OUT}


def _exact_gradients(case, seed):
    """Autograd through the plain step, a slice of columns at a time (they are independent)."""
    m = _columns(case["cols"], case["n_alts"], seed)
    bars, level = _bars(case, m, seed)
    rollout, parts, width = case["kind"] == "rollout", [], 1500
    for c0 in range(0, case["cols"], width):
        c = slice(c0, c0 + width)
        part = {k: v[..., c].contiguous() if v.shape[-1] == case["cols"] and k not in ("altitude", "gravity", "dalt_c", "inv_r")
                else v for k, v in m.items()}

        def step(x, e, h):
            return _steps({**part, **x, "eddy": e, "heating_scale": h}, case.get("steps", 1), DT, heating=True)

        parts.append(_differentiate(step, {k: part[k] for k in STATE}, part["eddy"], part["heating_scale"],
                                    bars[c] if rollout else [b[..., c] for b in bars], level, rollout))
    return {k: {f: torch.cat([p[k][f] for p in parts], -1) for f in parts[0][k]} for k in parts[0]}
