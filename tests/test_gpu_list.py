"""Verlet list, bit for bit, where its kernels take other branches: frozen and excluded
atoms moved to the end of the lists, and halo exports longer than a block's registers hold."""
import ctypes

import numpy as np
import pytest

from dlpoly_gb300 import systems

pytestmark = pytest.mark.gpu


def _lists(gpu_lib, oracle_lib, s):
    out = []
    for lib in (gpu_lib, oracle_lib):
        lib.init(s)
        lib.relocate()
        out.append(lib.link_cell_pairs())
    return out


def _same(a, b):
    """list(-3:0) and the listed entries, with the frozen and excluded ones beyond list(0)."""
    assert np.array_equal(a[:, :4], b[:, :4])
    k = np.arange(a.shape[1] - 4)[None, :]
    used = k < b[:, 1:2]  # list(-2): before the reordering
    assert np.array_equal(np.where(used, a[:, 4:], 0), np.where(used, b[:, 4:], 0))


@pytest.mark.parametrize("frozen", [0, 1, 2, 40, "many"])
def test_frozen_and_excluded_entries(gpu_lib, oracle_lib, frozen):
    s = systems.spce_water(8)
    s.lfrzn = np.zeros(s.natms, np.int32)
    if frozen == "many":
        s.lfrzn[np.arange(s.natms) % 3 != 0] = 1
    else:
        s.lfrzn[:3 * frozen:3] = 1
    _same(*_lists(gpu_lib, oracle_lib, s))


@pytest.mark.parametrize("blocks", [1, 2, 7])
def test_halo_runs_longer_than_a_pass(gpu_lib, oracle_lib, monkeypatch, blocks):
    monkeypatch.setenv("GB_HALO_BLOCKS", str(blocks))
    _same(*_lists(gpu_lib, oracle_lib, systems.nacl_melt(16)))
    monkeypatch.delenv("GB_HALO_BLOCKS")


@pytest.mark.parametrize("make", [lambda: systems.nacl_melt(10, kmax=30), lambda: systems.eam_alloy(5),
                                  lambda: systems.nacl_melt(22, kmax=64)])
def test_small_and_ragged_boxes(gpu_lib, oracle_lib, make):
    _same(*_lists(gpu_lib, oracle_lib, make()))


@pytest.mark.parametrize("molecules", [11, 15, 21])
def test_lanes_per_atom(gpu_lib, oracle_lib, molecules):
    """3,993, 10,125 and 27,783 atoms: each number of lanes per atom, with a last warp that has
    fewer atoms than the others."""
    _same(*_lists(gpu_lib, oracle_lib, systems.spce_water(molecules, kmax=64)))


def test_tiles_above_their_capacity(gpu_lib, oracle_lib, monkeypatch):
    monkeypatch.setenv("GB_TILE_CAP", "64")
    _same(*_lists(gpu_lib, oracle_lib, systems.spce_water(8)))
    monkeypatch.delenv("GB_TILE_CAP")


def test_halo_overflow_in_a_run_keeps_the_last_list(gpu_lib):
    """A cluster of ions flying out of the middle of its box: in the second step its images
    exceed mxatms, which ends the run with 56 before the list is built again."""
    s = systems.nacl_melt(8)
    s.cell = np.array([60.0, 0, 0, 0, 60.0, 0, 0, 0, 60.0])
    s.kmax = (64, 64, 64)
    s.vx[:] = 3000.0
    s.vy[:] = s.vz[:] = 0.0
    found = []  # the candidates that the builds since gb_init decided in FP64
    for steps in (1, 4):
        gpu_lib.init(s, max_list=512, mxatms=s.natms + 100)
        gpu_lib.start()
        st = gpu_lib.fn["md_run"](steps, (systems.GbStepStats * steps)())
        assert st == (0 if steps == 1 else 56)
        found.append(gpu_lib.pair_counts()[2])
    assert found[0] > 0 and found[1] == found[0]


def test_phase_timings_of_a_rebuild(gpu_lib):
    """Every phase's event pair is complete when the build's wait resolves the timings."""
    gpu_lib.init(systems.nacl_melt(16))
    L = gpu_lib._opt("profile", ctypes.c_int, [ctypes.c_int])
    read = gpu_lib._opt("profile_read", ctypes.c_int, [ctypes.c_char_p, ctypes.POINTER(ctypes.c_double),
                                                      ctypes.POINTER(ctypes.c_int64), ctypes.c_int])
    L(1)
    for _ in range(2):
        gpu_lib.relocate()
        gpu_lib.link_cell_pairs()
    names, ms, n = ctypes.create_string_buffer(32 * 32), (ctypes.c_double * 32)(), (ctypes.c_int64 * 32)()
    k = read(names, ms, n, 32)
    L(0)
    got = {names.raw[32 * i:32 * i + 32].split(b"\0")[0].decode(): (ms[i], n[i]) for i in range(k)}
    for phase in ("halo", "bin_sort", "list_pairs"):
        assert got[phase][1] == 2 and got[phase][0] > 0.0, phase
