"""Charge spreading where a brick holds more atoms than its slots: the atoms of a box drawn
together into one corner, against the oracle's reciprocal sum."""
import numpy as np
import pytest

from conftest import force_dev
from dlpoly_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(0, 1e-10), (2, 1e-10), (1, 5e-5)])
@pytest.mark.parametrize("shrink", [0.25, 0.12])
def test_crowded_bricks(gpu_lib, oracle_lib, precision, tol, shrink):
    s = systems.nacl_melt(16)
    for k in ("x", "y", "z"):
        v = getattr(s, k)
        setattr(s, k, (v + 0.5 * s.cell[0]) * shrink - 0.45 * s.cell[0])
    gpu_lib.init(s, precision=precision, mxatms=12 * s.natms)  # every atom has up to 7 images
    oracle_lib.init(s, mxatms=12 * s.natms)
    gpu_lib.relocate()
    oracle_lib.relocate()
    ed, er = gpu_lib.ewald_spme_forces(), oracle_lib.ewald_spme_forces()
    assert ed[0] == pytest.approx(er[0], rel=max(tol, 1e-10))
    assert force_dev(gpu_lib.download(), oracle_lib.download()) <= tol
