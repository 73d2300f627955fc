"""What the time-step engine is timed on: whole calls of its public entry points.

A pass is what a user's program does with a solver it holds: some time steps
(or gradients, or plane transforms) and the results read back to the host.
The sizes are those of this repository's benchmark, tests and sample
configurations: grids of 32^3 to 256^3, volume fractions of 0.01 to 0.4,
sphere diameters of 8 to 24 cells.  All arithmetic is FP64, the only type
the engine has.

Fields of a case:

  kind    "run"      Solver.run(steps): graph-replayed steps, then the state
          "loop"     the reference driver's loop: step(rks) and get_particles()
                     after every step (driver.Run without its files)
          "host"     a host program that owns the state: pibm_set_state from
                     pinned memory, one step, pibm_get_state, `steps` times
          "batch"    Batch.run(steps) of several realizations
          "adjoint"  Solver.adjoint(steps): objective, gradients, final state
          "planes"   pibm_ff2cr_noalloc on device planes, on torch's stream
  my      nodes per direction;  dia: sphere diameter in cells;  phi: volume
          fraction of the spheres (one sphere at least)
"""
import ctypes
import math

import numpy as np
import torch

import pureibm_ps2d_fd1d_b200 as pk
from pureibm_ps2d_fd1d_b200 import abi, config

GRIDS = (32, 64, 96, 128, 256)


def listed():
    return [
        # 10 steps of the driver's loop on the smallest grid: latency, launches
        # and read-backs, no kernel fills the GPU
        dict(name="driver_loop_32", kind="loop", my=32, dia=8.0, phi=0.1, re=20.0, steps=10),
        # one sphere in a box, the drag-law calibration run
        dict(name="single_sphere_64", kind="run", my=64, dia=16.0, phi=0.008, re=20.0, steps=50),
        # a fixed bed with the three-stage Runge-Kutta scheme and the limiter
        dict(name="array_rk3_96", kind="run", my=96, dia=15.0, phi=0.1, re=30.0, rk3=True, limiter="minmod", steps=10),
        # the benchmark's fixed random array, 128^3 with 100 spheres
        dict(name="array_128", kind="run", my=128, dia=20.0, phi=0.2, re=50.0, steps=40),
        # the same array with a passive scalar, its field read back too
        dict(name="array_scalar_128", kind="run", my=128, dia=20.0, phi=0.2, re=50.0, scalar=True, steps=40),
        # a host program with its own arrays: the state crosses PCIe both ways
        # in every step
        dict(name="host_state_128", kind="host", my=128, dia=20.0, phi=0.2, re=50.0, steps=2),
        # a small freely evolving suspension with collisions
        dict(name="suspension_64", kind="run", my=64, dia=12.0, phi=0.15, re=20.0, moving=True, steps=20),
        # the largest: a moving suspension of about 1200 spheres with scalar
        # transport on 256^3, one output interval
        dict(name="suspension_scalar_256", kind="run", my=256, dia=20.0, phi=0.3, re=20.0, moving=True, scalar=True, steps=10),
        # ensembles of independent realizations: many small grids, and mixed
        # ones as the statistics of a fixed bed are collected
        dict(name="ensemble_16x32", kind="batch", grids="32 32 32 32 32 32 32 32 32 32 32 32 32 32 32 32", dia=8.0, phi=0.15, re=20.0, steps=20),
        dict(name="ensemble_mixed", kind="batch", grids="64 64 64 96 96 96 128 128", dia=14.0, phi=0.25, re=30.0, steps=10),
        # gradient of the mean drag over 40 steps of a 96^3 fixed bed
        dict(name="adjoint_96", kind="adjoint", my=96, dia=16.0, phi=0.073, re=20.0, steps=40, checkpoint=20),
        # spectral planes of a 3-component 128^3 field to real space
        dict(name="planes_128", kind="planes", my=128, planes=384),
    ]


def _reynolds(rng, dia):
    """A Reynolds number that `dia` cells across a sphere resolve: with more
    than about 4 per cell a long run blows up, as under-resolved runs do."""
    return round(math.exp(rng.uniform(math.log(5.0), math.log(2.2 * dia))), 2)


def draw(rng):
    """One more case of the same ranges.  Steps shrink with the grid so that
    a pass costs at most what the largest listed case does."""
    kind = rng.choice(["run", "run", "run", "run", "loop", "host", "batch", "adjoint", "planes", "planes"])
    if kind == "planes":
        my = rng.choice([32, 64, 96, 128])
        return dict(kind=kind, my=my, planes=max(1, int(round(math.exp(rng.uniform(0.0, math.log(1000.0)))))))
    case = dict(kind=kind, dia=round(rng.uniform(8.0, 24.0), 2))
    if kind == "batch":
        grids = sorted(rng.choice([32, 64, 96, 128]) for _ in range(rng.randint(2, 12)))
        case.update(grids=" ".join(str(g) for g in grids), phi=round(rng.uniform(0.05, 0.35), 3), steps=rng.randint(3, 12))
        case["dia"] = min(case["dia"], 14.0)
        case["re"] = _reynolds(rng, case["dia"] / 1.5)
        return case
    if kind == "adjoint":
        case.update(my=rng.choice([32, 64, 96]), phi=round(rng.uniform(0.02, 0.2), 3), steps=rng.randint(3, 24),
                    checkpoint=rng.choice([0, 3, 5, 10]))
        case["dia"] = min(case["dia"], round(case["my"] / 3.0, 2))
        case["re"] = _reynolds(rng, case["dia"])
        return case
    my = rng.choice(GRIDS if kind == "run" else GRIDS[:4])
    case.update(my=my, dia=min(case["dia"], round(my / 3.0, 2)), phi=round(math.exp(rng.uniform(math.log(0.01), math.log(0.4))), 4))
    case["re"] = _reynolds(rng, case["dia"])
    if kind == "host":
        case["steps"] = rng.randint(1, 3)
        return case
    most = {32: 60, 64: 50, 96: 30, 128: 20, 256: 4}[my]
    case["steps"] = rng.randint(max(1, most // 4), most) if kind == "run" else rng.randint(1, max(2, most // 5))
    case["scheme"] = rng.choice(["upwind", "upwind", "center"])
    case["limiter"] = rng.choice(["none", "minmod"])
    case["rk3"] = rng.random() < 0.3
    case["moving"] = rng.random() < 0.3 and my >= 64
    case["scalar"] = rng.random() < 0.3
    case["meanflux"] = rng.random() < 0.2
    if case["moving"]:
        case["phi"] = min(case["phi"], 0.3)
        case["rk3"] = False
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _spheres(my, dia, phi, rng):
    """Non-overlapping sphere centres: random sites of the densest lattice of
    the box, then hard-sphere Monte Carlo moves."""
    k = max(1, int(math.floor(my / (dia * math.sqrt(2.0)) + 1e-12)))
    n = max(1, min(int(round(phi * my ** 3 / (math.pi / 6.0 * dia ** 3))), 4 * k ** 3))
    if 2 * n < k ** 3:   # dilute: any place in the box
        pts = config.random_sequential_addition(n, float(my), dia, rng)
    else:
        pts = config.fcc_subset(n, float(my), dia, rng)
        pts = 1.0 + np.mod(pts - 1.0 + rng.uniform(0.0, my, size=3), float(my))
    return config.hard_sphere_mc(pts, float(my), dia, rng, min(1000, 10 * n), 0.1 * dia)[0]


def _params(case, my):
    prm = config.default_params()
    prm.update(my=my, lybyd=my / case["dia"], dbydx=case["dia"], re=case["re"], vis=0.012, cfl=0.1, cfl_max=0.5,
               discr_scheme=case.get("scheme", "upwind"), limiter=case.get("limiter", "none"), rk3=case.get("rk3", False),
               include_frmeanfluid=case.get("meanflux", False), initialize_zero=not case.get("scalar"), dobnd=False,
               ramp_frac_steps=0)
    if case.get("scalar"):   # hot spheres in a cold stream when they move, the reverse when fixed
        hot = 1.0 if case.get("moving") else 0.0
        prm.update(iscalon=1, pr_or_sc_nu=0.7, phisurf=hot, phistream=1.0 - hot)
    if case.get("moving"):
        prm.update(imove=1, collision_type="softsphere", rhos=100.0, rhof=1.0, coeff_rest=0.9)
    if case["kind"] == "adjoint":
        uchar = case["re"] * 0.012
        prm.update(set_mpg=True, adaptive=False)
        prm["umean0"] = (uchar, 0.0, 0.0)
    return prm


def _check(rc):
    if rc != 0:
        raise RuntimeError("pibm error %d: %s" % (rc, pk.load_library().pibm_last_error().decode()))


class _Buffers:
    """Pinned host arrays in the reference layout that a solver's state is read
    into (and set from), kept by the program for the run."""

    def __init__(self, s, scalar):
        nu, np_ = 3 * s.mz * s.my2 * (s.nx + 1), s.mz * s.my2 * s.nx
        n = [2 * nu, 2 * nu, 2 * np_] + ([2 * (nu // 3)] if scalar else [])
        self.all = torch.zeros(sum(n), dtype=torch.float64).pin_memory()
        at = np.cumsum([0] + n)
        part = [self.all[at[k]:at[k + 1]] for k in range(len(n))]
        self.u, self.nl, self.p = part[:3]
        self.phi = part[3] if scalar else None
        self.view = abi.pibm_state_view()
        ptr = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
        self.view.u, self.view.nl, self.view.p = ptr(self.u), ptr(self.nl), ptr(self.p)
        self.phi_ptr = ptr(self.phi) if scalar else None
        self.flux, self.ratios = np.zeros(max(s.nbody, 1)), np.zeros(3)

    def read(self, s):
        lib = pk.load_library()
        _check(lib.pibm_get_state(s.h, ctypes.byref(self.view)))
        if self.phi is not None:
            dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
            _check(lib.pibm_get_scalar(s.h, self.phi_ptr, dp(self.flux), dp(self.ratios)))

    def out(self):
        """The fields (the program's own buffers) and the mean quantities."""
        v = self.view
        d = dict(u=self.u, nl=self.nl, p=self.p,
                 means=np.array(v.umean[:] + v.mpg[:] + v.ufmean[:] + [v.t, v.dt, v.cf]))
        if self.phi is not None:
            d.update(phi=self.phi, flux=self.flux.copy(), ratios=self.ratios.copy())
        return d


#: Report entries that are sums or means of the step's fields.  The largest
#: divergence left by the projection and the drag change are rounding-level
#: differences, so they are not compared.
REPORT = ("dt", "t", "umax", "norm_drag", "pres_drag", "visc_drag", "total_drag", "mixmeanslipmod")


def _report(r):
    return np.array([r[k] for k in REPORT] + list(r["ufmean"]) + list(r["mpg"]) + list(r["pres_total"]) + list(r["visc_total"]))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = {"case": case}
    if case["kind"] == "planes":
        my, n = case["my"], case["planes"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # spectra that fall off with the wavenumber, as velocity fields' do
        ky = torch.arange(my // 2 + 1, device="cuda", dtype=torch.float64)
        kz = torch.fft.fftfreq(my, 1.0 / my, device="cuda", dtype=torch.float64)
        decay = 1.0 / (1.0 + ky[None, :] ** 2 + kz[:, None] ** 2)
        st["a"] = torch.randn(n, my, my // 2 + 1, dtype=torch.complex128, device="cuda", generator=g) * decay
        st["b"] = torch.empty(n, my, my, dtype=torch.float64, device="cuda")
        return st
    if case["kind"] == "batch":
        members = []
        for q, my in enumerate(int(m) for m in case["grids"].split()):
            # Reynolds numbers and volume fractions spread over the ensemble
            c = dict(case, re=case["re"] * (0.5 + 0.25 * (q % 5)), dia=min(case["dia"], my / 3.0), phi=case["phi"] * (0.8 + 0.1 * (q % 5)))
            members.append((_params(c, my), _spheres(my, c["dia"], c["phi"], rng)))
        st["batch"] = pk.Batch(members)
        st["batch"].run(4)   # a developing flow, not the fluid at rest
        st["buffers"] = [_Buffers(m, False) for m in st["batch"].members]
        return st
    my, dia = case["my"], case["dia"]
    xc = _spheres(my, dia, case["phi"], rng)
    prm, vel = _params(case, my), None
    if case.get("moving"):
        vel = rng.normal(0.0, 0.1 * case["re"] * 0.012, size=xc.shape)
        vel -= vel.mean(axis=0, keepdims=True)
    if case["kind"] == "adjoint":   # imposed pressure gradient of about the array's Stokes drag
        prm["mpg"] = (-xc.shape[0] * 3.0 * math.pi * 0.012 * prm["umean0"][0] * 2.0 / (my / dia) ** 3, 0.0, 0.0)
    s = st["solver"] = pk.Solver(config.make_params(prm), xc, vel)
    st["buffers"] = _Buffers(s, bool(case.get("scalar")))
    if case["kind"] == "adjoint":
        init = s.get_state()
        init["umean"] = np.array(prm["umean0"])
        s.set_state(init)
    s.run(4)
    if case["kind"] == "host":
        st["buffers"].read(s)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "planes":
        a, b = state["a"], state["b"]
        _check(pk.load_library().pibm_ff2cr_noalloc(case["my"], case["my"], case["planes"],
                                                   ctypes.cast(a.data_ptr(), ctypes.POINTER(ctypes.c_double)),
                                                   ctypes.cast(b.data_ptr(), ctypes.POINTER(ctypes.c_double)),
                                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return b
    if kind == "batch":
        state["batch"].run(case["steps"])
        out = []
        for m, buf in zip(state["batch"].members, state["buffers"]):
            buf.read(m)
            out.append(dict(state=buf.all, means=buf.out()["means"], particles=np.stack(m.get_particles()[:3])))
        return out
    s, buf = state["solver"], state["buffers"]
    if kind == "adjoint":
        g = s.adjoint(case["steps"], (1.0, 0.0, 0.0), case["checkpoint"])
        buf.read(s)
        return dict(buf.out(), J=g["J"], g_xc=g["g_xc"], g_mpg=g["g_mpg"])
    records = []
    if kind == "run":
        rep = s.run(case["steps"])
        records.append(_report(rep))
        records.append(np.concatenate([a.ravel() for a in s.get_particles()]))
        buf.read(s)
    elif kind == "loop":
        for _ in range(case["steps"]):
            for rks in range(1, 4 if case.get("rk3") else 2):
                rep = s.step(rks)
            records.append(_report(rep))
            records.append(np.concatenate([a.ravel() for a in s.get_particles()]))
        records = [np.concatenate(records)]
        buf.read(s)
    else:
        lib, rep = pk.load_library(), abi.pibm_step_report()
        for _ in range(case["steps"]):
            _check(lib.pibm_set_state(s.h, ctypes.byref(buf.view)))
            _check(lib.pibm_step(s.h, 1, ctypes.byref(rep)))
            _check(lib.pibm_get_state(s.h, ctypes.byref(buf.view)))
        records.append(_report(rep.as_dict()))
    return dict(buf.out(), records=records)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _grid_work(my, steps, stages=1, scalar=False):
    """Bytes and operations of `steps` steps on a my^3 grid: every stage reads
    and writes u, p and the nonlinear term (7 complex fields; 2 more with the
    scalar) once; 25 plane transforms (8 more with the scalar) of 2.5 n log2 n
    operations for n real points and 5 (6) pairs of transforms along x."""
    cells, half = my ** 3, my * my * (my // 2 + 1)
    fields, planes, lines = (9, 33, 6) if scalar else (7, 25, 5)
    flops = planes * my * 2.5 * my * my * 2 * math.log2(my) + lines * 2 * (half // my) * 5 * my * math.log2(my) + 200 * cells
    return 2 * fields * half * 16 * steps * stages, flops * steps * stages


def work(case):
    kind = case["kind"]
    if kind == "planes":
        my, n = case["my"], case["planes"]
        return {"bytes": n * (my * (my // 2 + 1) * 16 + my * my * 8), "flops": n * 2.5 * my * my * 2 * math.log2(my)}
    grids = [int(m) for m in case["grids"].split()] if kind == "batch" else [case["my"]]
    stages, scalar = (3 if case.get("rk3") else 1), bool(case.get("scalar"))
    total = [0, 0]
    for my in grids:
        half = my * my * (my // 2 + 1) * 16
        b, f = _grid_work(my, case["steps"], stages, scalar)
        if kind == "adjoint":   # the reverse of a step reads its fields and costs about the step again
            b, f = 2 * b, 2 * f
        reads = case["steps"] * 2 if kind == "host" else 1   # the state to the host (and back)
        total[0] += b + reads * (8 if scalar else 7) * half
        total[1] += f
    return {"bytes": total[0], "flops": total[1]}


def tolerance(case):
    """FP64 throughout.  A change of the start's velocity by its last bit
    shows as up to 2e-14 (2-norm) in u, nl, p and the gradients after two
    passes, 6e-13 at single values, and 2e-12 in the surface fluxes of spheres
    whose sum nearly cancels; a transform differs from another by 3e-16."""
    if case["kind"] == "planes":
        return {"rel": 2e-15, "max": 1e-13}
    return {"rel": 1e-11, "max": 1e-9}


def exact(case, seed):
    """The plane transforms from numpy.  The time step has no short
    restatement: its geometry, forcing and DEM together are a program of
    their own."""
    if case["kind"] != "planes":
        return None
    a = prepare(case, seed)["a"].cpu().numpy()
    # the z transform, then the y transform of its Hermitian part
    return np.fft.irfft2(a, s=(case["my"], case["my"]), norm="forward")
