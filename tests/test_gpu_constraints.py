"""SHAKE/RATTLE on clusters of every kind that the scalar-form kernel takes (one, two and
three constraints, frozen atoms), on clusters beyond it, and on more clusters than threads."""
import ctypes

import numpy as np
import pytest

from dlpoly_gb300 import systems

pytestmark = pytest.mark.gpu

REL = 1e-9  # the trajectory bar of the other constraint tests


def _mixed_clusters(tied):
    """Water whose molecules keep 3, 2, 1 or no constraints; every 16th has a frozen oxygen.
    tied: a molecule's oxygen is tied to another one's, a cluster of 4 atoms and 4 constraints."""
    s = systems.spce_water(8)
    lc = s.listcon.reshape(-1, 3, 3)
    keep = {0: (0, 1, 2), 1: (0, 1), 2: (0,), 3: ()}
    rows = [lc[m, k] for m in range(lc.shape[0]) for k in keep[m % 4]]
    s.lfrzn = np.zeros(s.natms, np.int32)
    s.lfrzn[0::3][8::16] = 1
    frozen = s.lfrzn != 0
    for v in (s.vx, s.vy, s.vz):
        v[frozen] = 0.0
    if tied:
        o = 3 * 3  # the oxygen of molecule 3 (no constraints of its own), tied to molecule 0
        pos = np.stack([s.x, s.y, s.z], 1)
        d = pos[0] - pos[o]
        d -= s.cell[0] * np.round(d / s.cell[0])
        s.prmcon = np.append(s.prmcon, np.linalg.norm(d))
        rows.append(np.array([3, 1, o + 1], np.int32))
    s.listcon = np.concatenate(rows).astype(np.int32)
    return s


@pytest.mark.parametrize("tied", [False, True])
def test_cluster_kinds_match_oracle(gpu_lib, oracle_lib, tied):
    s = _mixed_clusters(tied)
    out = []
    for lib in (gpu_lib, oracle_lib):
        lib.init(s)
        lib.start()
        out.append((lib.md_vv(3), lib.download()))
    (sd, a), (sr, b) = out
    assert [x.shake_iters for x in sd] == [x.shake_iters for x in sr]
    assert [x.rattle_iters for x in sd] == [x.rattle_iters for x in sr]
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.abs(a[k] - b[k]).max() <= REL * np.abs(b[k]).max(), k
    for x, y in zip(sd, sr):
        cs = np.abs(y.strcon[:]).max()
        assert np.abs(np.array(x.strcon[:]) - np.array(y.strcon[:])).max() <= 1e-8 * cs


def test_more_clusters_than_threads(gpu_lib, monkeypatch):
    """64,000 molecules: a thread runs several clusters and keeps their scalars between chunks."""
    s = systems.spce_water(40, kmax=128)
    out = []
    for glob in ("1", "0"):
        monkeypatch.setenv("GB_SHAKE_GLOBAL", glob)
        gpu_lib.init(s)
        gpu_lib.start()
        out.append((gpu_lib.md_vv(1), gpu_lib.download()))
    (sg, a), (sc, b) = out
    assert (sg[0].shake_iters, sg[0].rattle_iters) == (sc[0].shake_iters, sc[0].rattle_iters)
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.abs(a[k] - b[k]).max() <= REL * np.abs(a[k]).max(), k


def test_native_form_by_fp64_instructions(gpu_lib, oracle_lib, monkeypatch):
    """The form that checks the others runs the FP64 cluster kernel: its SHAKE takes the launches of
    the per-sweep FP64 kernels (the scalar-form kernel is a single one), also when it is chosen after gb_init."""
    s = systems.spce_water(8)
    n = {}
    launches = gpu_lib._opt("kernel_launches", ctypes.c_int64, [])
    prec = gpu_lib._opt("set_precision", ctypes.c_int, [ctypes.c_int])
    for name, glob, at_init, then in (("fp64", "0", 0, 0), ("native", "0", 2, 2), ("later", "0", 0, 2),
                                      ("global", "1", 2, 2)):
        monkeypatch.setenv("GB_SHAKE_GLOBAL", glob)
        gpu_lib.init(s, precision=at_init)
        assert prec(then) == 0
        gpu_lib.start()
        k = launches()
        gpu_lib.constraints_tags()
        gpu_lib.apply_shake()
        n[name] = launches() - k
        if name in ("native", "later"):
            oracle_lib.init(s)
            oracle_lib.start()
            (x,), (y,) = gpu_lib.md_vv(1), oracle_lib.md_vv(1)
            assert (x.shake_iters, x.rattle_iters) == (y.shake_iters, y.rattle_iters)
    monkeypatch.delenv("GB_SHAKE_GLOBAL")
    assert n["native"] == n["later"] == n["global"] > n["fp64"]


@pytest.mark.parametrize("factor", [1.2, 2.0, 3.0, 4.0, 6.0])
def test_shake_of_stretched_molecules(gpu_lib, factor):
    """Molecules whose bonds start far from their lengths: every constraint ends within its
    tolerance, after the sweeps and with the stress of the FP64 cluster kernel."""
    out = []
    for precision in (0, 2):
        s = systems.spce_water(6, box=19.7, rcut=7.0, kmax=32)
        s.shake_tol = 1e-9
        for v in (s.x, s.y, s.z):
            o = np.repeat(v[0::3], 3)
            v[:] = o + factor * (v - o)
        gpu_lib.init(s, precision=precision)
        gpu_lib.constraints_tags()
        r = gpu_lib.apply_shake()
        d = gpu_lib.download()
        lc = s.listcon.reshape(-1, 3)
        pos = np.stack([d[k] for k in "xyz"], 1)
        b = pos[lc[:, 1] - 1] - pos[lc[:, 2] - 1]
        d0 = s.prmcon[lc[:, 0] - 1]
        # |b^2 - d0^2| / 2 < tol d0, and the rounding of coordinates below 32 A (2^-48 A each)
        assert (np.abs((b ** 2).sum(1) - d0 ** 2) / (2.0 * d0)).max() < s.shake_tol + 1e-13 * factor
        out.append((r["iters"], r["strcon"], pos))
    (ia, sa, pa), (ib, sb, pb) = out
    assert ia == ib
    assert np.abs(sa - sb).max() <= 1e-9 * np.abs(sb).max()
    assert np.abs(pa - pb).max() <= 1e-9
