"""Tabulated EAM metals on the GPU (gb_metal.cu) against the oracle's restatement of
metal_ld_compute / metal_forces, through the C-ABI."""
import numpy as np
import pytest

from conftest import force_dev
from dlpoly_gb300 import systems
from test_metal_oracle import kat_check, poly_tables, two_atoms

pytestmark = pytest.mark.gpu


def test_eam_known_answers_on_gpu(gpu_lib):
    for r in (1.3, 2.7183, 5.9):
        kat_check(gpu_lib, r=r)


@pytest.mark.parametrize("n_side,listed", [(8, None), (10, (1, 0, 1))])
def test_eam_forces_match_oracle(gpu_lib, oracle_lib, n_side, listed):
    s = systems.eam_alloy(n_side)
    if listed is not None:        # the Cu-Ni pair not listed in FIELD 'metal': no cross force
        s.metal_listed = np.array(listed, np.int32)
    for lib in (gpu_lib, oracle_lib):
        lib.init(s)
        lib.start()
    a, b = gpu_lib.download(), oracle_lib.download()
    assert force_dev(a, b) < 1e-10
    ea, eb = gpu_lib.metal_energies(), oracle_lib.metal_energies()
    for k in ("engmet", "engden"):
        assert ea[k] == pytest.approx(eb[k], rel=1e-10), k
    # the virial sums pair repulsion against embedding attraction: cancellation leaves
    # it ~100x smaller than its terms, so its bar is 1e-9
    assert ea["virmet"] == pytest.approx(eb["virmet"], rel=1e-9)
    np.testing.assert_allclose(gpu_lib.metal_rho(), oracle_lib.metal_rho(), rtol=1e-11)


def test_eam_md_matches_oracle(gpu_lib, oracle_lib):
    s = systems.eam_alloy(8)
    for lib in (gpu_lib, oracle_lib):
        lib.init(s)
        lib.start()
    sd, sr = gpu_lib.md_vv(12), oracle_lib.md_vv(12)
    assert [x.list_rebuilt for x in sd] == [x.list_rebuilt for x in sr]
    for x, y in zip(sd, sr):
        assert x.engmet == pytest.approx(y.engmet, rel=1e-10)
        assert x.virmet == pytest.approx(y.virmet, rel=1e-9)
        assert x.engke == pytest.approx(y.engke, rel=1e-10)
    a, b = gpu_lib.download(), oracle_lib.download()
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.abs(a[k] - b[k]).max() <= 1e-9 * np.abs(b[k]).max(), k


def test_eam_error_statuses_on_gpu(gpu_lib):
    s = two_atoms(0.9)
    s.eam = poly_tables()
    gpu_lib.init(s)
    with pytest.raises(Exception, match="506"):
        gpu_lib.start()
    s = two_atoms(2.0)
    tabs = poly_tables()
    tabs[2] = dict(tabs[2], start=5.0, finish=10.0)
    s.eam = tabs
    gpu_lib.init(s)
    with pytest.raises(Exception, match="507"):
        gpu_lib.start()
    kat_check(gpu_lib)             # the context is still usable


@pytest.mark.parametrize("side", [-1, 1])
@pytest.mark.parametrize("off", [2e-9, 1e-8, 2.5e-8, 1e-6])
def test_eam_pairs_next_to_a_midpoint(gpu_lib, oracle_lib, side, off):
    """Separations a small fraction of an interval from the middle of two table points, where
    the three-point interpolant jumps (here by 1e-5 of the force): the nearer point is taken."""
    ng = 100
    r = np.linspace(1.0, 6.0, ng)
    rho = np.linspace(0.0, 10.0, ng)
    dr = 5.0 / (ng - 1)
    for k in (23, 40, 61):
        s = two_atoms(1.0 + (k + 0.5 + side * off) * dr)
        s.eam = [{"kind": "pair", "types": (1, 1), "start": 1.0, "finish": 6.0, "values": r ** -3},
                 {"kind": "dens", "types": (1, 1), "start": 1.0, "finish": 6.0, "values": r ** -2},
                 {"kind": "embe", "types": (1, 1), "start": 0.0, "finish": 10.0, "values": 0.01 * rho ** 2}]
        out = []
        for lib in (gpu_lib, oracle_lib):
            lib.init(s)
            lib.start()
            out.append((lib.download()["fx"], lib.metal_rho()))
        (fa, ra), (fb, rb) = out
        assert np.abs(fa - fb).max() <= 1e-10 * np.abs(fb).max()
        np.testing.assert_allclose(ra, rb, rtol=1e-10)


def test_eam_distance_to_the_last_bits(gpu_lib):
    """Isolated pairs under V = (r - 2.5)^2 / 2, whose force r - 2.5 shows the error of r itself:
    1e-14 of the root and 0.4e-14 of r^2 (48 bits), relative to r, and as much of the force."""
    n, step = 12, 16.0
    rng = np.random.default_rng(11)
    g = np.arange(n) * step - 0.5 * n * step + 0.5 * step
    at = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    d = rng.standard_normal(at.shape)
    d *= (rng.uniform(2.2, 2.8, len(at)) / np.linalg.norm(d, axis=1))[:, None]
    d = np.round(d * 2.0 ** 30) / 2.0 ** 30  # (coordinates and separations without rounding)
    s = two_atoms(2.0, box=n * step)
    pos = np.empty((2 * len(at), 3))
    pos[0::2], pos[1::2] = at, at + d
    m = len(pos)
    s.ltype, s.chge, s.weight = np.ones(m, np.int32), np.zeros(m), np.full(m, 60.0)
    s.lfrzn = np.zeros(m, np.int32)
    s.x, s.y, s.z = (pos[:, k].copy() for k in range(3))
    s.vx, s.vy, s.vz = (np.zeros(m) for _ in range(3))
    r = np.linspace(1.0, 6.0, 401)
    rho = np.linspace(0.0, 10.0, 401)
    s.eam = [{"kind": "pair", "types": (1, 1), "start": 1.0, "finish": 6.0, "values": 0.5 * (r - 2.5) ** 2},
             {"kind": "dens", "types": (1, 1), "start": 1.0, "finish": 6.0, "values": 1.0 + 0.0 * r},
             {"kind": "embe", "types": (1, 1), "start": 0.0, "finish": 10.0, "values": 0.0 * rho}]
    gpu_lib.init(s)
    gpu_lib.start()
    f = gpu_lib.download()
    ld = d.astype(np.longdouble)
    dist = np.sqrt((ld ** 2).sum(1))
    along = sum(f[k][0::2] * ld[:, c] for c, k in enumerate(("fx", "fy", "fz"))) / dist
    err = np.abs(along - (dist - np.longdouble(2.5)))
    bound = 1.4e-14 * dist + 1.4e-14 * np.abs(dist - 2.5) + 2e-15  # (2e-15: the table's differences)
    print(float((err / dist).max()), float(np.sqrt(((err / dist) ** 2).mean())))
    assert (err <= bound).all()
