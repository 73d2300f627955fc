"""The host's path through the entry points, without a GPU: the engine runs in
a child process on a preloaded CUDA runtime (fake_cudart.c) whose kernels do
nothing and whose calls are counted, so what a call allocates, captures and
launches is known exactly."""
import os
import subprocess
import sys
import textwrap

import pytest

from pureibm_ps2d_fd1d_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
PRELUDE = """
import ctypes as C
import numpy as np
import pureibm_ps2d_fd1d_b200 as pk
from pureibm_ps2d_fd1d_b200 import config
fake = C.CDLL(FAKE)
fake.fake_count.argtypes, fake.fake_count.restype = [C.c_char_p], C.c_long
fake.fake_fail_launch.argtypes, fake.fake_fail_launch.restype = [C.c_long], None
count = lambda what: fake.fake_count(what.encode())
lib = pk.load_library()
def solver(**kw):
    prm, xc = config.random_array(my=32, dia_cells=8, nbody=3, seed=1, mc_moves=20)
    prm.update(kw)
    return pk.Solver(config.make_params(prm), xc)
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    build.build()
    so = str(tmp_path_factory.mktemp("fake") / "libfakecudart.so")
    subprocess.run(["gcc", "-O1", "-std=c99", "-w", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "fake_cudart.c")], check=True)

    def run(body):
        env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=os.path.dirname(HERE))
        src = "FAKE = %r\n" % so + PRELUDE + textwrap.dedent(body)
        p = subprocess.run([sys.executable, "-c", src], env=env, capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stdout + p.stderr
    return run


def test_first_read_back_of_the_particles_pins_nothing(host):
    """get_particles() stages through memory pinned with the handle: mapping a
    chunk of pinned memory costs 1 to 4 ms, fifty times the read-back."""
    host("""
    s = solver()
    s.step()
    before = count("HostAlloc"), count("HostRegister")
    pres, visc, force, xc, vel = s.get_particles()
    assert (count("HostAlloc"), count("HostRegister")) == before
    assert xc.shape == (3, 3) and not pres.any()
    for my in (1, 2):   # created and closed again
        t = solver()
        t.get_particles()
        t.close()
    assert count("HostAlloc") == 0
    """)


def test_step_captures_only_what_a_long_loop_replays(host):
    """A capture costs what a dozen replays save: short loops, and loops that
    change the run between steps (which drops the graphs), launch directly; long
    ones replay each stage and parity from one capture, RK3 by time steps and not by stages."""
    host("""
    means = np.array([1e-3, 0.0, 0.0])
    dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    for rk3 in (False, True):
        stages = 3 if rk3 else 1
        def steps(s, n):
            for _ in range(n):
                for rks in range(1, stages + 1):
                    s.step(rks)
        base = count("Instantiate")
        s = solver(rk3=rk3)
        steps(s, 20)
        assert count("Instantiate") == base
        for _ in range(60):   # each drops the graphs
            assert lib.pibm_set_desired_means(s.h, dp(means), dp(means)) == 0
            steps(s, 1)
        assert count("Instantiate") == base
        steps(s, 60)
        made, launched = count("Instantiate"), count("Launch")
        assert made == base + 2 * stages
        steps(s, 60)          # replayed: no direct launch, no further capture
        assert (count("Instantiate"), count("Launch")) == (made, launched)
        assert lib.pibm_set_tuning(s.h, s.tuning()["lines_per_cta"]) == 0
        steps(s, 20)
        assert count("Instantiate") == made and count("Launch") > launched
        s.close()
        t = solver(rk3=rk3)   # an AB2 step is the graph that pibm_run has captured
        t.run(2)
        assert count("Instantiate") == made + 2
        launched = count("Launch")
        steps(t, 3)
        assert count("Instantiate") == made + 2 and (count("Launch") == launched) == (not rk3)
        t.close()
    """)


def test_launch_that_fails_within_a_capture_is_reported(host):
    """A launch that fails while a step is captured fails the call, and the graph
    without it is not kept: the next call captures a whole one."""
    host("""
    def fails(call):
        try:
            call()
        except pk.PibmError as e:
            assert e.code == -8, e
            return
        raise AssertionError("the failed launch was not reported")
    s = solver()
    fake.fake_fail_launch(3)
    fails(lambda: s.run(2))
    assert count("Instantiate") == 0 and count("GraphLaunch") == 0
    per_step = s.info.kernels_per_step
    before = count("Capture")
    s.run(2)
    assert count("Instantiate") == 2 and count("GraphLaunch") == 2
    assert count("Capture") - before == 2 * per_step
    s.close()

    t = solver(rk3=True)
    for _ in range(24):
        for rks in (1, 2, 3):
            t.step(rks)
    made, replayed = count("Instantiate"), count("GraphLaunch")
    fake.fake_fail_launch(2)
    fails(lambda: t.step(1))
    assert (count("Instantiate"), count("GraphLaunch")) == (made, replayed)
    t.step(1)
    assert (count("Instantiate"), count("GraphLaunch")) == (made + 1, replayed + 1)
    t.close()

    prm, xc = config.random_array(my=32, dia_cells=8, nbody=3, seed=1, mc_moves=20)
    b = pk.Batch([(dict(prm), xc)] * 2 + [(dict(prm, iscalon=1, pr_or_sc_nu=0.7, phisurf=1.0, phistream=0.0,
                                                initialize_zero=False), xc)])
    made = count("Instantiate")
    fake.fake_fail_launch(5)
    fails(lambda: b.run(1))
    assert count("Instantiate") == made
    b.run(1)
    assert count("Instantiate") == made + 2
    """)


def test_dem_in_one_launch_where_its_sub_steps_pay_for_it(host):
    """Launches per step of soft-sphere runs: one for all sub-steps up to 256
    spheres, and 32 more for each sub-step after the first up to 512; else
    three per sub-step."""
    host("""
    def launches(n, rhos):
        prm, _ = config.single_sphere(my=64, dia_cells=6.0, re=20.0)
        prm.update(imove=1, collision_type="softsphere", rhos=rhos, rhof=1.0, coeff_rest=0.9, initialize_zero=True)
        s = pk.Solver(config.make_params(prm), config.fcc_subset(n, 64.0, 6.0, np.random.default_rng(n)))
        before = count("Launch")
        s.step()
        made = count("Launch") - before
        assert made == s.info.kernels_per_step
        s.close()
        return made
    one = launches(1, 1e2)
    assert [launches(n, 1e2) for n in (256, 257, 512)] == [one] * 3     # 82 sub-steps
    assert launches(513, 1e2) > one + 3 * 50
    assert launches(256, 1e9) == one                                    # one sub-step
    assert [launches(n, 1e9) for n in (257, 512, 513)] == [one + 2] * 3
    """)
