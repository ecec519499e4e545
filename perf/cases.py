"""The work that is timed: whole steps of melting cases and the routines a host calls one by one.

A user of this library has a host program that owns the registered arrays, attaches a case once
(registration, device mirrors, initial tagging) and then runs the time loop through the C-ABI: cfl, dt,
forcing and the RK3 step per iteration, reading the fields back every few steps.  That is what the "step"
cases do, from the small grids of parameter sweeps to the 256^3 configuration, in the FP64 and in the
precision form, with the body held, melting or free.  "batch" advances many small cases together, "loop"
is a host that also writes its own arrays back every step.  The other cases are single parts of the step
as a host that takes over one routine at a time calls them: the pressure projection, the factored line
solves, the immersed-boundary forcing and heat flux, and the line solve on device memory of the caller's own.

Sizes come from melt_ibm_gb300/workloads.py, the batched and serving configurations (48^3 to 256^3) and the
grids the library accepts (2^a 3^b).  Shapes are the library's defaults (no autotuner run).  A state is stepped
hundreds of times: on the small grids the latent heat is large enough, and the free body heavy enough, that the body
is still there at the end.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from melt_ibm_gb300 import abi
from melt_ibm_gb300 import build as mbuild
from melt_ibm_gb300.batch import BatchRunner
from melt_ibm_gb300.case import Case, CaseConfig
from melt_ibm_gb300.mesh import icosphere
from melt_ibm_gb300.serve import resolved_level

FLOW = (abi.MIBM_F_VX, abi.MIBM_F_VY, abi.MIBM_F_VZ, abi.MIBM_F_TEMP, abi.MIBM_F_PR)
FLOW_MASK = sum(1 << f for f in FLOW)
XYZ_MASK = 1 << (32 + abi.MIBM_M_XYZV)
GRIDS = (32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256)
TWO_PI = 2.0 * math.pi


@functools.lru_cache(maxsize=None)
def _lib() -> abi.Lib:
    return abi.Lib(mbuild.build())


@functools.lru_cache(maxsize=None)
def _mesh(level: int):
    return icosphere(level)


def listed():
    return [
        # a small case of a parameter sweep: 48^3 FP64, fixed melting sphere; launches and latency count
        dict(name="step_f64_48", kind="step", n=48, n3=48, level=3, rad=0.5, nu=0.01, lat=8.0, body="melt",
             forcing=0, gz=0.0, form="f64", steps=4, dtmax=2e-3),
        # a grid that is no power of two and no cube: solid body in ABC-forced flow, unequal spacings
        dict(name="step_f64_108x72", kind="step", n=108, n3=72, level=3, rad=0.5, nu=0.01, lat=1.0, body="solid",
             forcing=2, gz=0.0, form="f64", steps=2, dtmax=4e-3),
        # the 128^3 configuration: free melting body, linear forcing
        dict(name="step_f64_128_free", kind="step", n=128, n3=128, level=4, rad=0.4, nu=0.005, lat=1.0, body="free",
             forcing=3, gz=0.0, form="f64", steps=2, dtmax=1e-2),
        # the 256^3 configuration, FP64: melting spheroid, stochastic forcing, Boussinesq coupling
        dict(name="step_f64_256", kind="step", n=256, n3=256, level=5, rad=1.0, nu=0.0025, lat=0.5, body="spheroid",
             forcing=1, gz=0.1, form="f64", steps=3, dtmax=1e-2),
        # the two configurations in the precision form
        dict(name="step_mixed_128_free", kind="step", n=128, n3=128, level=4, rad=0.4, nu=0.005, lat=1.0, body="free",
             forcing=3, gz=0.0, form="mixed", steps=2, dtmax=1e-2),
        dict(name="step_mixed_256", kind="step", n=256, n3=256, level=5, rad=1.0, nu=0.0025, lat=0.5, body="spheroid",
             forcing=1, gz=0.1, form="mixed", steps=3, dtmax=1e-2),
        # many independent cases per step, the grids of the batched configuration, precision form
        dict(name="batch_mixed", kind="batch", n48=6, n64=4, n96=2, form="mixed", steps=2, dtmax=2e-3),
        # a host that uploads and reads back its arrays every step
        dict(name="loop_f64_96", kind="loop", n=96, n3=96, level=3, rad=0.4, nu=0.01, lat=8.0, body="melt",
             forcing=0, gz=0.0, form="f64", steps=1, dtmax=2e-3),
        # pressure projection alone: divg, phcalc, updvp, prcalc
        dict(name="project_f64_192", kind="project", n=192, n3=192, steps=4),
        # the factored line solves of one component alone, on a right-hand side the host supplies
        dict(name="adi_f64_144x96", kind="adi", n=144, n3=96, beta=0.02),
        # the immersed-boundary routines alone: cages, MLS weights, forcing, heat flux
        dict(name="markers_f64_128", kind="markers", n=128, n3=128, level=4, rad=0.4, nu=0.005, lat=1.0, body="melt",
             forcing=0, gz=0.0, form="f64", dtmax=1e-2),
        # x-line solves on a device array of the caller's own
        dict(name="lines_f64_96", kind="lines", n=96, n2=96, n3=64, beta=0.05),
    ]


def _grid(rng, lo, hi):
    """A grid length, even over the logarithm of [lo, hi]."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((g for g in GRIDS if lo <= g <= hi), key=lambda g: abs(math.log(g / want)))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "loop", "batch", "project", "adi", "markers", "lines"))
    if kind == "batch":
        return dict(kind=kind, n48=rng.randint(1, 8), n64=rng.randint(0, 5), n96=rng.randint(0, 3),
                    form=rng.choice(("f64", "mixed")), steps=rng.randint(1, 3), dtmax=2e-3)
    if kind == "project":
        return dict(kind=kind, n=_grid(rng, 32, 216), n3=_grid(rng, 32, 216), steps=rng.randint(1, 4))
    if kind == "adi":
        return dict(kind=kind, n=_grid(rng, 32, 216), n3=_grid(rng, 32, 216),
                    beta=round(math.exp(rng.uniform(math.log(1e-3), math.log(2.0))), 4))
    if kind == "lines":
        return dict(kind=kind, n=_grid(rng, 32, 256), n2=rng.randint(8, 256), n3=rng.randint(4, 128),
                    beta=round(math.exp(rng.uniform(math.log(1e-3), math.log(2.0))), 4))
    form = "f64" if kind == "markers" else rng.choice(("f64", "mixed"))
    n = _grid(rng, 36, 128 if kind == "loop" else 192)
    n3 = rng.choice((n, n, rng.choice([g for g in GRIDS if 2 * n <= 3 * g <= 4 * n])))
    body = rng.choice(("melt", "free", "solid", "spheroid" if n >= 96 else "melt"))
    rad = 1.0 if body == "spheroid" else round(rng.uniform(0.35, 0.6), 3)
    level = resolved_level(max(n, n3), 0.6 if body == "spheroid" else rad)
    return dict(kind=kind, n=n, n3=n3, level=level, rad=rad,
                nu=round(rng.uniform(0.005, 0.02), 4), lat=round(rng.uniform(6.0, 16.0), 2), body=body,
                forcing=rng.choice((0, 0, 1, 2, 3)), gz=rng.choice((0.0, 0.1)), form=form, steps=rng.randint(1, 3),
                dens=4.0, dtmax=2e-3)


# ------------------------------------------------------------------ inputs
def _random_flow(n, n3, seed):
    """Random-phase velocity of unit rms, |k| <= 8, free of discrete divergence, as (3, n, n, n3) on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.randn((3, n, n, n3), generator=gen, device="cuda", dtype=torch.float64)
    spec = torch.fft.rfftn(noise, dim=(1, 2, 3))
    f = lambda m: torch.fft.fftfreq(m, d=1.0 / m, device="cuda", dtype=torch.float64)
    k = [f(n)[:, None, None], f(n)[None, :, None],
         torch.fft.rfftfreq(n3, d=1.0 / n3, device="cuda", dtype=torch.float64)[None, None, :]]
    kk = torch.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
    spec = spec * torch.where((kk > 0) & (kk <= 8), kk * torch.exp(-(kk / 2) ** 2), 0.0)
    step = [(torch.exp(2j * math.pi * k[d] / m) - 1) * (m / TWO_PI) for d, m in enumerate((n, n, n3))]
    lap = sum(s.abs() ** 2 for s in step)
    lap[0, 0, 0] = 1.0
    phi = -sum(step[d] * spec[d] for d in range(3)) / lap
    for d in range(3):
        spec[d] += step[d].conj() * phi
    vel = torch.fft.irfftn(spec, s=(n, n, n3), dim=(1, 2, 3))
    return (vel / vel.square().mean().sqrt()).cpu().numpy()


def _case(c, seed, autostart=True):
    """A case attached to the library, its initial flow drawn from the seed, its arrays page-locked."""
    lib = _lib()
    n, n3 = c["n"], c["n3"]
    body = c.get("body", "none")
    cfg = CaseConfig(n=n, n3=n3, ren=1.0 / c.get("nu", 0.01), latheat=c.get("lat", 1.0), betagz=c.get("gz", 0.0),
                     dt=min(1e-2, c.get("dtmax", 1e-2)), dtmax=c.get("dtmax", 1e-2), imlsfor=0 if body == "none" else 1,
                     imlsstr=1 if body == "free" else 0, imelt=0 if body in ("solid", "none") else 1,
                     dens_ratio=c.get("dens", 2.0) if body == "free" else 1.0, forcing=1 if c.get("forcing", 0) else 0,
                     which_hit=c.get("forcing", 0) or 1, c_hit=0.25 if c.get("forcing") == 3 else 0.1, hit_seed=seed,
                     mesh=_mesh(c.get("level", 2)), rad_p=c.get("rad", 0.5), v_on_ve=0.0, velocity="rest",
                     axes=(0.6, 0.3, 0.3) if body == "spheroid" else (1.0, 1.0, 1.0))
    case = Case(cfg)
    vel = _random_flow(n, n3, seed)
    for f, v in zip(FLOW[:3], vel):
        case.interior(f)[...] = v
        case.fill_ghosts(f)
    case.attach(lib)
    lib.mibm_pin_host_(abi.ref_int(1))
    lib.check("pin_host")
    if c.get("form") == "mixed":
        lib.mibm_set_precision_(abi.ref_int(1), abi.ref_int(2))
        lib.check("set_precision")
    return case


class _State:
    """What the program keeps between passes; its contexts go with it."""

    def __init__(self, kind):
        self.kind, self.cases, self.runner, self.nt = kind, [], None, 0

    def __del__(self):
        if self.runner is not None:
            self.runner.close()
        for case in self.cases:
            case.detach(_lib())


def prepare(case, seed):
    s = _State(case["kind"])
    s.case = case
    if s.kind == "lines":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        s.src = torch.randn((case["n3"], case["n2"], case["n"]), generator=gen, device="cuda", dtype=torch.float64)
        s.buf = torch.empty_like(s.src)
        return s
    if s.kind == "batch":
        rng = np.random.default_rng(seed)
        for n, count in ((48, case["n48"]), (64, case["n64"]), (96, case["n96"])):
            for q in range(count):
                rad = 0.35 + 0.25 * q / max(1, count - 1)
                s.cases.append(_case(dict(n=n, n3=n, level=resolved_level(n, rad), rad=rad, body="melt",
                                          nu=float(rng.uniform(0.005, 0.02)), lat=float(rng.uniform(6.0, 16.0)),
                                          form=case["form"], dtmax=case["dtmax"]), int(rng.integers(1 << 30))))
        s.runner = BatchRunner(_lib(), s.cases)
        return s
    one = _case(case, seed)
    s.cases.append(one)
    if s.kind in ("project", "adi", "markers"):
        # the scalars a host sets before it calls a routine of the first substep
        al = 8.0 / 15.0
        one.set_S(abi.MIBM_S_AL, al)
        one.set_S(abi.MIBM_S_GA, al)
        one.set_S(abi.MIBM_S_RO, 0.0)
        one.set_S(abi.MIBM_S_DT, 5e-3)
        one.set_S(abi.MIBM_S_BETA, 5e-3 / one.S(abi.MIBM_S_REN) * 0.5)
    if s.kind == "project":
        # a flow that the projection has to correct: the divergence-free one plus a gradient and noise
        vel, pr = _unprojected(case, seed)
        for f, v in zip(FLOW[:3], vel):
            one.interior(f)[...] = v
            one.fill_ghosts(f)
        one.interior(abi.MIBM_F_PR)[...] = pr
        one.fill_ghosts(abi.MIBM_F_PR)
        one.sync_from_host(_lib(), FLOW_MASK)
    if s.kind == "adi":
        one.interior(abi.MIBM_F_RHS)[...] = _rhs(case, seed)
    return s


def _unprojected(case, seed):
    n, n3 = case["n"], case["n3"]
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    vel = _random_flow(n, n3, seed)
    extra = 0.05 * torch.randn((4, n, n, n3), generator=gen, device="cuda", dtype=torch.float64).cpu().numpy()
    return vel + extra[:3], extra[3]


def _rhs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    return 1e-2 * torch.randn((case["n"], case["n"], case["n3"]), generator=gen, device="cuda",
                              dtype=torch.float64).cpu().numpy()


# ------------------------------------------------------------------ one pass
def _fields(case, ids):
    return [case.interior(f) for f in ids]


def run(s):
    lib, c = _lib(), s.case
    if s.kind == "lines":
        s.buf.copy_(s.src)
        st = lib.mibm_solxi_noalloc(s.buf.data_ptr(), c["n"], c["n2"], c["n3"], c["n"], c["beta"],
                                    torch.cuda.current_stream().cuda_stream)
        if st != 0:
            raise RuntimeError(f"mibm_solxi_noalloc: status {st}")
        return s.buf
    if s.kind == "batch":
        for _ in range(c["steps"]):
            s.runner.step()
        for one in s.cases:
            one.sync_to_host(lib, FLOW_MASK | XYZ_MASK)
        big = [i for i, one in enumerate(s.cases) if i in (0, len(s.cases) - 1)]
        return [_fields(s.cases[i], FLOW) + [s.cases[i].mesh_arrays[abi.MIBM_M_XYZV]] for i in big] + \
            [one.interior(abi.MIBM_F_VX) for i, one in enumerate(s.cases) if i not in big]
    one = s.cases[0]
    if s.kind in ("step", "loop"):
        for _ in range(c["steps"]):
            if s.kind == "loop":
                one.sync_from_host(lib, FLOW_MASK | XYZ_MASK)
            s.nt += 1
            one.step(lib, s.nt)
            if s.kind == "loop":
                one.sync_to_host(lib, FLOW_MASK | XYZ_MASK)
        if s.kind == "step":
            one.sync_to_host(lib, FLOW_MASK | XYZ_MASK)
        return _fields(one, FLOW) + [one.mesh_arrays[abi.MIBM_M_XYZV], one.sc[abi.MIBM_S_POS_CM, :3],
                                     one.sc[abi.MIBM_S_VEL_CM, :3], one.S(abi.MIBM_S_DT)]
    one.bind(lib)
    if s.kind == "project":
        for _ in range(c["steps"]):
            lib.divg_()
            lib.phcalc_()
            lib.updvp_()
            lib.prcalc_()
        lib.check("projection")
        one.sync_to_host(lib, sum(1 << f for f in (FLOW[0], FLOW[1], FLOW[2], FLOW[4])))
        return _fields(one, (FLOW[0], FLOW[1], FLOW[2], FLOW[4]))
    if s.kind == "adi":
        one.sync_from_host(lib, 1 << abi.MIBM_F_RHS)
        vz = one.fields[abi.MIBM_F_VZ]
        plane1 = vz.ctypes.data + vz.strides[2]
        beta = abi.ref_double(c["beta"])
        lib.solxi_(beta)
        lib.solxj_(beta)
        lib.solxk_(C.c_void_p(plane1), beta)
        lib.check("line solves")
        one.sync_to_host(lib, 1 << abi.MIBM_F_VZ)
        return one.interior(abi.MIBM_F_VZ)
    # markers
    lib.findcentroidindices_()
    lib.mlsweight_()
    lib.mlsforce_()
    lib.velforce_()
    lib.tempforce_()
    lib.findprobeindices_()
    lib.mls_heatflux_()
    lib.check("markers")
    m = (abi.MIBM_M_PTXAB_Q1, abi.MIBM_M_PTXAB_TEMP, abi.MIBM_M_QW_O, abi.MIBM_M_QW_I, abi.MIBM_M_QW_OVERT)
    one.sync_to_host(lib, sum(1 << f for f in FLOW[:4]) | sum(1 << (32 + i) for i in m))
    return _fields(one, FLOW[:4]) + [one.mesh_arrays[i] for i in m]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: the prognostic fields (and history) in and out of every substep, the routine's own fields for
    the single parts.  Operations: about 1.4 thousand per cell and step, as counted for the reference's routines."""
    kind = case["kind"]
    if kind == "lines":
        cells = case["n"] * case["n2"] * case["n3"]
        return {"bytes": 16.0 * cells, "flops": 7.0 * cells}
    if kind == "batch":
        cells = case["n48"] * 48 ** 3 + case["n64"] * 64 ** 3 + case["n96"] * 96 ** 3
    else:
        cells = case["n"] ** 2 * case["n3"]
    if kind in ("step", "batch", "loop"):
        return {"bytes": case["steps"] * cells * 3 * 10 * 8.0, "flops": case["steps"] * 1400.0 * cells}
    if kind == "project":
        return {"bytes": case["steps"] * cells * 8 * 8.0, "flops": case["steps"] * 150.0 * cells}
    if kind == "adi":
        return {"bytes": cells * 3 * 8.0, "flops": 21.0 * cells}
    faces = 20 * 4 ** case["level"]
    return {"bytes": cells * 8 * 8.0 + faces * 27 * 8 * 8.0, "flops": faces * 4.0e4 + 10.0 * cells}


# ------------------------------------------------------------------ the same in 64 bits, without the library
def _wave(m):
    """Eigenvalues of minus the periodic second difference with unit spacing."""
    return 2.0 - 2.0 * torch.cos(2 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / m)


def _line_solve(x, beta, dim):
    """(1 + 2 beta) x_i - beta (x_{i-1} + x_{i+1}) = rhs_i, periodic along dim, refined once in 64 bits."""
    shape = [1] * x.dim()
    shape[dim] = x.shape[dim]
    den = 1.0 + beta * _wave(x.shape[dim]).reshape(shape)
    inv = lambda r: torch.fft.ifft(torch.fft.fft(r, dim=dim) / den, dim=dim).real
    y = inv(x)
    res = x - ((1.0 + 2.0 * beta) * y - beta * (torch.roll(y, 1, dim) + torch.roll(y, -1, dim)))
    return y + inv(res)


def exact(case, seed):
    kind = case["kind"]
    if kind == "lines":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn((case["n3"], case["n2"], case["n"]), generator=gen, device="cuda", dtype=torch.float64)
        return _line_solve(x, case["beta"], 2)
    if kind == "adi":
        x = torch.from_numpy(_rhs(case, seed)).cuda()
        w = torch.from_numpy(_random_flow(case["n"], case["n3"], seed)[2]).cuda()
        for dim in range(3):
            x = _line_solve(x, case["beta"], dim)
        return w + x
    if kind == "project":
        vel, pr = _unprojected(case, seed)
        vel, pr = torch.from_numpy(vel).cuda(), torch.from_numpy(pr).cuda()
        n, n3 = case["n"], case["n3"]
        dx = [n / TWO_PI, n / TWO_PI, n3 / TWO_PI]
        nu, dt, al = 0.01, 5e-3, 8.0 / 15.0
        lam = (_wave(n)[:, None, None] * dx[0] ** 2 + _wave(n)[None, :, None] * dx[1] ** 2
               + _wave(n3)[None, None, :] * dx[2] ** 2)
        lam[0, 0, 0] = 1.0
        for _ in range(case["steps"]):
            div = sum((torch.roll(vel[d], -1, d) - vel[d]) * dx[d] for d in range(3)) / (dt * al)
            spec = torch.fft.fftn(div) / -lam
            spec[0, 0, 0] = 0
            phi = torch.fft.ifftn(spec).real
            for d in range(3):
                vel[d] -= (phi - torch.roll(phi, 1, d)) * dx[d] * dt * al
            lap = sum((torch.roll(phi, 1, d) - 2 * phi + torch.roll(phi, -1, d)) * dx[d] ** 2 for d in range(3))
            pr = pr + phi - al * dt * nu * 0.5 * lap
        return [vel[0], vel[1], vel[2], pr]
    return None
