"""Full time steps of the CUDA engine against the CPU oracle.

Parity bar (floating point): relative difference <= 1e-10 in velocity,
pressure, nonlinear term and per-particle drag after the stated number of
steps; set-up integer data (active reversal points, solid mask) bit-exact.
"""
import numpy as np
import pytest

import pureibm_ps2d_fd1d_b200 as pk
from pureibm_ps2d_fd1d_b200 import config
import oracle_ctypes as oc

TOL = 1e-10


def rel(a, b):
    d = np.max(np.abs(np.asarray(a) - np.asarray(b)))
    s = np.max(np.abs(np.asarray(b)))
    return d / s if s > 0 else d


def make_pair(prm, xc):
    P = config.make_params(prm)
    parts = config.Particles(xc)
    gpu = pk.Solver(P, xc)
    cpu = oc.OracleSolver(P, parts.struct)
    cpu._parts = parts
    return gpu, cpu


def compare(gpu, cpu, tol=TOL):
    sg, sc = gpu.get_state(), cpu.get_state()
    out = {k: rel(sg[k], sc[k]) for k in ("u", "p", "nl")}
    out["umean"] = rel(sg["umean"], sc["umean"])
    out["mpg"] = rel(sg["mpg"], sc["mpg"])
    if gpu.nbody:
        pg, vg, fg, _, _ = gpu.get_particles()
        pc, vc, fc, _, _ = cpu.get_particles()
        out["pres"], out["visc"], out["force"] = rel(pg, pc), rel(vg, vc), rel(fg, fc)
    assert abs(sg["t"] - sc["t"]) <= tol * abs(sc["t"])
    bad = {k: v for k, v in out.items() if not v <= tol}
    assert not bad, out
    return out


@pytest.mark.gpu
def test_setup_geometry_bit_exact():
    prm, xc = config.random_array(my=64, dia_cells=12, nbody=12, seed=7, mc_moves=200)
    gpu, cpu = make_pair(prm, xc)
    assert gpu.nbnd == cpu.nbnd
    assert gpu.info.count_solid == cpu.info.count_solid
    assert np.array_equal(gpu.get_if_rev(), cpu.get_if_rev())
    assert np.array_equal(gpu.get_fluid_mask(), cpu.get_fluid_mask())
    assert gpu.info.dt == cpu.info.dt


@pytest.mark.gpu
@pytest.mark.parametrize("scheme,limiter", [("upwind", "none"), ("upwind", "minmod"), ("center", "none")])
def test_single_sphere_32_steps(scheme, limiter):
    prm, xc = config.single_sphere(my=32, dia_cells=8)
    prm.update(discr_scheme=scheme, limiter=limiter)
    gpu, cpu = make_pair(prm, xc)
    for _ in range(10):
        rg, rc = gpu.step(), cpu.step()
    compare(gpu, cpu)
    assert abs(rg["divmax"]) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("my,re,width", [(32, 0.05, 4), (32, 20.0, 8), (64, 0.05, 8), (64, 20.0, 4), (96, 0.05, 4), (96, 20.0, 8),
                                         (128, 0.05, 4), (128, 0.05, 8), (256, 0.05, 4), (256, 20.0, 8)])
def test_line_solves_of_a_rough_state(my, re, width):
    """Two steps from a random state with every (ky,kz) line and x mode excited,
    the (0,0) line included: at Re 0.05 (nu dt/dx^2 of order 100) the viscous
    systems couple a whole line, at Re 20 a few planes.  Bound: the pressure
    lines' condition number, up to (N/pi)^2 = 7e3 at 256, times a few roundings."""
    prm, xc = config.single_sphere(my=my, dia_cells=8.0, re=re)
    gpu, cpu = make_pair(prm, xc)
    gpu.set_tuning(width)
    rng, uchar = np.random.default_rng(my), re * prm["vis"]
    st = gpu.get_state()
    for k in ("u", "nl", "p"):
        shp = st[k].shape
        a = rng.standard_normal(shp) + 1j * rng.standard_normal(shp)
        if k != "p":
            a[..., -1] = a[..., 0]      # the periodic image plane
        st[k] = a * (uchar / my * (0.1 if k == "u" else 0.01))
    real = np.fft.rfft2(np.fft.irfft2(np.moveaxis(st["u"], 3, 1), s=(my, my)))   # the spectra of real fields
    st["u"] = np.ascontiguousarray(np.moveaxis(real, 1, 3))
    real = np.fft.rfft2(np.fft.irfft2(np.moveaxis(st["nl"], 3, 1), s=(my, my)))
    st["nl"] = np.ascontiguousarray(np.moveaxis(real, 1, 3))
    gpu.set_state(st)
    cpu.set_state(st)
    for _ in range(2):
        gpu.step()
        cpu.step()
    # the solved fields; the mpg controller is cf = -1/dt times a difference of
    # means of the random field, in which the two summation orders' last bits
    # (2e-16 x 16 M terms) show as 5e-10
    sg, sc = gpu.get_state(), cpu.get_state()
    assert max(rel(sg[k], sc[k]) for k in ("u", "p", "nl")) <= TOL


@pytest.mark.gpu
def test_single_sphere_64_100_steps():
    """Single fixed sphere, 64^3, d=16, Re=20, fluid at rest, 100 steps."""
    prm, xc = config.single_sphere(my=64, dia_cells=16, re=20.0)
    gpu, cpu = make_pair(prm, xc)
    for _ in range(100):
        gpu.step(); cpu.step()
    compare(gpu, cpu)


@pytest.mark.gpu
def test_random_array_64_10_spheres_100_steps():
    """Reduced random array: 64^3, 10 spheres of d=12, 100 steps."""
    prm, xc = config.random_array(my=64, dia_cells=12, nbody=10, re=50.0, seed=1234, mc_moves=1000)
    gpu, cpu = make_pair(prm, xc)
    for _ in range(100):
        gpu.step(); cpu.step()
    compare(gpu, cpu)


@pytest.mark.gpu
def test_graph_run_equals_step_loop_bitwise():
    prm, xc = config.random_array(my=32, dia_cells=8, nbody=4, seed=3, mc_moves=100)
    a = pk.Solver(config.make_params(prm), xc)
    b = pk.Solver(config.make_params(prm), xc)
    for _ in range(7):
        a.step()
    b.run(7)
    sa, sb = a.get_state(), b.get_state()
    for k in ("u", "p", "nl"):
        assert np.array_equal(sa[k], sb[k]), k


@pytest.mark.gpu
def test_state_round_trip_and_restart():
    prm, xc = config.single_sphere(my=32, dia_cells=8)
    a = pk.Solver(config.make_params(prm), xc)
    a.run(5)
    st = a.get_state()
    b = pk.Solver(config.make_params(prm), xc)
    b.set_state(st)
    a.run(3); b.run(3)
    sa, sb = a.get_state(), b.get_state()
    for k in ("u", "p", "nl"):
        assert np.array_equal(sa[k], sb[k]), k


@pytest.mark.gpu
def test_deterministic_rerun():
    prm, xc = config.random_array(my=32, dia_cells=8, nbody=4, seed=5, mc_moves=100)
    outs = []
    for _ in range(2):
        s = pk.Solver(config.make_params(prm), xc)
        s.run(5)
        outs.append(s.get_state()["u"])
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.gpu
def test_random_array_256_two_steps():
    """256^3 grid (8-CTA plane clusters, 4-line x tiles), 6 spheres of d=20:
    two steps against the oracle."""
    prm, xc = config.random_array(my=256, dia_cells=20, nbody=6, seed=3, mc_moves=20)
    gpu, cpu = make_pair(prm, xc)
    for _ in range(2):
        gpu.step()
        cpu.step()
    compare(gpu, cpu)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["fixed", "rk3", "scalar", "moving"])
def test_repeated_steps_equal_run_across_new_states_and_plans(kind):
    """Single steps are replayed from recorded launches after the first 24 and
    where run() has recorded them, and launched directly again after a change of
    the line tiles: with a state set and the tiles changed in between they still
    end at the bits of the same steps as one run, and a state with its scalar
    field read back and set elsewhere continues alike."""
    prm, xc = config.random_array(my=32, dia_cells=8, nbody=3, seed=3, mc_moves=50)
    if kind == "rk3":
        prm.update(rk3=True)
    if kind == "scalar":
        prm.update(iscalon=1, pr_or_sc_nu=0.7, phisurf=0.0, phistream=1.0, initialize_zero=False)
    if kind == "moving":
        prm.update(imove=1, collision_type="softsphere", rhos=100.0, rhof=1.0, coeff_rest=0.9, initialize_zero=True)
    P = config.make_params(prm)

    def step(solver):
        for r in (1, 2, 3) if kind == "rk3" else (1,):
            solver.step(r)

    a, b, c = (pk.Solver(P, xc) for _ in range(3))
    for _ in range(27):
        step(a)
    b.run(27)
    scal = a.get_scalar() if kind == "scalar" else None
    if kind != "moving":   # a moving run's particle state is part of its restart, not of its fields
        st = a.get_state()
        c.set_state(st)
        if scal is not None:
            c.set_scalar(scal["phif"], scal["nlphif"], scal["heat_ratio"], scal["heat_ratio_old"])
    for _ in range(4):
        step(a)
    a.set_tuning(4)
    b.set_tuning(4)
    for _ in range(27):
        step(a)
    b.run(31)
    solvers = [b]
    if kind != "moving":
        c.run(4)
        c.set_tuning(4)
        for _ in range(27):
            step(c)
        solvers.append(c)
    want = a.get_state()
    for s in solvers:
        got = s.get_state()
        for k in ("u", "p", "nl"):
            assert np.array_equal(got[k], want[k]), k
        assert got["t"] == want["t"]
        if scal is not None:
            x, y = a.get_scalar(), s.get_scalar()
            assert np.array_equal(x["phif"], y["phif"]) and x["heat_ratio"] == y["heat_ratio"]


@pytest.mark.gpu
@pytest.mark.parametrize("scheme,limiter,nbody,scalar", [("upwind", "minmod", 0, False), ("center", "none", 2, False), ("upwind", "none", 2, True)])
def test_sweeps_at_256(scheme, limiter, nbody, scalar):
    """256^3, where fields, nonlinear term and forcing are transformed by column
    and row sweeps and a scalar steps after the flow on its stream: two steps
    against the oracle, and two members of a batch bitwise against them."""
    prm, xc = config.random_array(my=256, dia_cells=20, nbody=max(nbody, 1), seed=3, mc_moves=20)
    xc = xc[:nbody]
    prm.update(discr_scheme=scheme, limiter=limiter)
    if scalar:
        prm.update(iscalon=1, pr_or_sc_nu=0.7, phisurf=0.0, phistream=1.0, initialize_zero=False)
    gpu, cpu = make_pair(prm, xc)
    for _ in range(2):
        gpu.step()
        cpu.step()
    if not scalar:
        compare(gpu, cpu)
    else:
        # Only fields: this run starts at its desired mean, so mpg has the
        # rounding of that mean (1e-16 of it) over dt beside the drag of two
        # spheres in 256^3, about 1e-9 of it.
        sg, sc, fg, fc = gpu.get_scalar(), oc.get_scalar(cpu), gpu.get_state(), cpu.get_state()
        out = {k: rel(fg[k], fc[k]) for k in ("u", "p", "nl")}
        out.update({k: rel(sg[k], sc[k]) for k in ("phif", "flux_body")})
        assert max(out.values()) <= TOL, out
    b = pk.Batch([(prm, xc)] * 2)
    b.run(2)
    want = gpu.get_state()
    for m in b.members:
        got = m.get_state()
        for k in ("u", "p", "nl"):
            assert np.array_equal(got[k], want[k]), k
