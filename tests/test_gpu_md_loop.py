"""The MD loop that reads a step's sums after its last step, launched or replayed as CUDA graphs,
against the loop that reads them at every step: constraints, thermostats and metals."""
import ctypes

import numpy as np
import pytest

from dlpoly_gb300 import systems
from test_metal_oracle import poly_tables, two_atoms

pytestmark = pytest.mark.gpu

RUNS = {
    "water": (lambda: systems.spce_water(8), 0, "nve", 1e-12),
    "water_mixed_nose_hoover": (lambda: systems.spce_water(8), 1, "nose-hoover", 1e-12),
    "water_berendsen": (lambda: systems.spce_water(8), 0, "berendsen", 1e-12),
    "nacl_langevin": (lambda: systems.nacl_melt(16), 0, "langevin", 1e-12),
    "eam": (lambda: systems.eam_alloy(8), 0, "nve", 1e-9),  # FP64 atomics: their order varies
}
FIELDS = ("engcpe_rc", "vircpe_rc", "engcpe_rl", "vircpe_rl", "engcpe_ex", "vircpe_ex", "engvdw", "virvdw", "engke",
          "vircon", "consv", "engmet", "virmet")


@pytest.mark.parametrize("name", RUNS)
def test_deferred_loop_matches_per_step_readback(gpu_lib, monkeypatch, name):
    make, precision, ens, tol = RUNS[name]
    s = make()
    out = []
    for defer, graphs in (("0", "0"), ("1", "0"), ("1", "1")):
        monkeypatch.setenv("GB_MD_DEFER", defer)
        monkeypatch.setenv("GB_GRAPHS", graphs)
        gpu_lib.init(s, precision=precision)
        if ens != "nve":
            gpu_lib.set_ensemble(ens, temp=300.0, tau_t=0.05, chi=5.0)
        gpu_lib.start()
        st = gpu_lib.md_vv(9)
        met = gpu_lib.metal_energies() if s.eam else {}
        out.append((st, gpu_lib.download(), gpu_lib.thermostat_state(), met))
    monkeypatch.delenv("GB_MD_DEFER")
    monkeypatch.delenv("GB_GRAPHS")
    sa, a, ta, ma = out[0]
    for sb, b, tb, mb in out[1:]:
        for k in a:
            assert np.abs(a[k] - b[k]).max() <= tol * np.abs(a[k]).max(), k
        for x, y in zip(sa, sb):
            assert (x.list_rebuilt, x.shake_iters, x.rattle_iters) == (y.list_rebuilt, y.shake_iters, y.rattle_iters)
            for f in FIELDS:
                scale = max(abs(getattr(x, f)), 1e-3 * abs(x.engke))
                assert abs(getattr(x, f) - getattr(y, f)) <= 10 * tol * scale, f
            for f in ("stress", "strkin", "strcon"):
                u, v = np.array(getattr(x, f)[:]), np.array(getattr(y, f)[:])
                assert np.abs(u - v).max() <= 10 * tol * max(np.abs(u).max(), 1e-30), f
        for k in ta:
            assert abs(ta[k] - tb[k]) <= 10 * tol * max(abs(ta[k]), 1e-30), k
        for k in ma:
            assert mb[k] == pytest.approx(ma[k], rel=10 * tol), k


def test_failing_step_ends_the_call_with_its_code(gpu_lib):
    """SHAKE beyond its sweeps ends a run of several steps with 105; the steps before it are reported."""
    s = systems.spce_water(8)
    gpu_lib.init(s, shake_maxit=20)
    gpu_lib.start()
    with pytest.raises(Exception) as e:
        gpu_lib.md_vv(5)
    assert getattr(e.value, "code", None) == 105
    gpu_lib.init(s)
    gpu_lib.start()
    assert all(x.shake_iters > 20 for x in gpu_lib.md_vv(5))


def _colliding_water():
    """64 molecules, one of which reaches another's oxygen in two steps: RATTLE of the second
    step then has velocities that need more sweeps than it is given."""
    s = systems.spce_water(4, box=24.0, rcut=7.0, kmax=32)
    s.tstep = 2e-5
    for v in (s.vx, s.vy, s.vz):
        v[:] = 0.0
    s.vx[:3] = (s.x[48] - s.x[0] - 1.8) / (2.0 * s.tstep)
    for c in (s.y, s.z):
        c[:3] += c[48] - c[0]
    return s


def _closing_metal():
    """Two atoms that come closer than their tables' first point in the second step."""
    s = two_atoms(1.02)
    s.eam = poly_tables()
    s.vx[:] = (4.0, -4.0)
    return s


FAILURES = {
    "rattle_nve": (_colliding_water, dict(shake_maxit=22), "nve", 515, 1),
    "rattle_langevin": (_colliding_water, dict(shake_maxit=22), "langevin", 515, 1),
    "metal_nve": (_closing_metal, {}, "nve", 506, 1),
    "metal_nose_hoover": (_closing_metal, {}, "nose-hoover", 506, 1),
}


@pytest.mark.parametrize("graphs", ["0", "1"])
@pytest.mark.parametrize("steps", ["last", "more"])
@pytest.mark.parametrize("name", FAILURES)
def test_failed_step_leaves_its_own_state(gpu_lib, monkeypatch, name, steps, graphs):
    """A step that fails in its forces or in stage 2 leaves the state, the thermostat and the
    step counter (which keys Langevin's noise) of that step, and reports the steps before it."""
    make, over, ens, code, good = FAILURES[name]
    n = good + 1 if steps == "last" else good + 4
    out = []
    for defer in ("0", "1"):
        monkeypatch.setenv("GB_MD_DEFER", defer)
        monkeypatch.setenv("GB_GRAPHS", graphs)
        s = make()
        gpu_lib.init(s, **over)
        if ens != "nve":
            gpu_lib.set_ensemble(ens, temp=300.0, tau_t=0.5, chi=0.01)
        gpu_lib.start()
        arr = (systems.GbStepStats * n)()
        for x in arr:
            x.engke = -1.0
        assert gpu_lib.fn["md_run"](n, arr) == code
        state = gpu_lib.download()
        th = gpu_lib.thermostat_state()
        again = {}
        if ens == "langevin":
            s = make()
            for v in (s.vx, s.vy, s.vz):
                v[:] = 0.0
            gpu_lib.upload(s.x, s.y, s.z, s.vx, s.vy, s.vz)
            gpu_lib.start()
            gpu_lib.md_vv(1)
            again = gpu_lib.download()
        out.append((state, th, [x.engke for x in arr], again))
    monkeypatch.delenv("GB_MD_DEFER")
    monkeypatch.delenv("GB_GRAPHS")
    (a, ta, ka, ga), (b, tb, kb, gb) = out
    for k in a:
        assert np.abs(a[k] - b[k]).max() <= 1e-12 * np.abs(a[k]).max(), k
    for k in ta:
        assert abs(ta[k] - tb[k]) <= 1e-12 * max(abs(ta[k]), 1e-30), k
    assert [k == -1.0 for k in ka] == [k == -1.0 for k in kb] == [k >= good for k in range(n)]
    for k in ga:
        assert np.abs(ga[k] - gb[k]).max() <= 1e-12 * np.abs(ga[k]).max(), k


@pytest.mark.parametrize("graphs", ["0", "1"])
@pytest.mark.parametrize("name", ["water", "water_mixed_nose_hoover", "nacl_langevin", "eam", "nacl"])
def test_region_timings_of_a_run(gpu_lib, monkeypatch, name, graphs):
    """gb_last_timings: the regions of every run but plain NVE, which has the total alone."""
    make, precision, ens, _ = RUNS.get(name, (lambda: systems.nacl_melt(16), 0, "nve", 0.0))
    monkeypatch.setenv("GB_GRAPHS", graphs)
    gpu_lib.init(make(), precision=precision)
    monkeypatch.delenv("GB_GRAPHS")
    if ens != "nve":
        gpu_lib.set_ensemble(ens, temp=300.0, tau_t=0.05, chi=5.0)
    gpu_lib.start()
    read = gpu_lib._opt("last_timings", ctypes.c_int, [ctypes.POINTER(ctypes.c_double), ctypes.c_int])
    for steps in (6, 3, 1):
        gpu_lib.md_vv(steps)
        t = (ctypes.c_double * 6)()
        assert read(t, 6) == 0
        listed, forces, spme, integ, total, span = t
        assert 0.0 < total <= 1.02 * span and spme == 0.0
        if name == "nacl":
            assert listed == forces == integ == 0.0
        else:
            assert min(listed, forces, integ) > 0.0
            assert listed + forces + integ == pytest.approx(total, rel=1e-6)
            assert total >= 0.5 * span


def test_runs_longer_than_the_ring(gpu_lib, monkeypatch):
    """4,100 steps in one call, of which the loop keeps 4,096 at a time: statistics and state of
    every step as the loop that reads them at each step has them."""
    out = []
    for defer in ("0", "1"):
        monkeypatch.setenv("GB_MD_DEFER", defer)
        s = systems.lj_pair(eps=100.0, sigma=2.0, r=2.4)
        gpu_lib.init(s)
        gpu_lib.start()
        out.append((gpu_lib.md_vv(4100), gpu_lib.download()))
    monkeypatch.delenv("GB_MD_DEFER")
    (sa, a), (sb, b) = out
    for f in ("engke", "engvdw", "list_rebuilt"):
        u, v = (np.array([getattr(x, f) for x in st]) for st in (sa, sb))
        assert np.abs(u - v).max() <= 1e-12 * max(np.abs(u).max(), 1.0), f
    assert sa[-1].engke != sa[0].engke
    for k in a:
        assert np.abs(a[k] - b[k]).max() <= 1e-12 * max(np.abs(a[k]).max(), 1.0), k
