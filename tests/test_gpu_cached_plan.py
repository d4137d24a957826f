"""powder_average and powder_scan keep a plan per system and sizes and point it
at each call's inputs.  Its scratch depends on the time grid (uniform grids take
the Fourier form of the phase sum, one that does not start at 0 with sine terms),
so a call must get the scratch of its own grid whatever ran before it."""

import ctypes

import numpy as np
import pytest

from muspinsim_gb300 import _lib, powder
from muspinsim_gb300.spinsys import MuonSpinSystem
from oracle import port
from tests.helpers import oracle_system

pytestmark = pytest.mark.gpu

SPINS = ["mu", "e", "H"]
A = [np.diag([40.0, 55.0, 70.0]), np.diag([-20.0, 10.0, 35.0])]
COUPLINGS = [("hyperfine", {"i": 1, "j": 2}, A[0]), ("hyperfine", {"i": 3, "j": 2}, A[1])]
TOL = {"fp64": 1e-10, "mixed": 1e-6}
N, T = 1500, 1000
GRIDS = {
    "zero": np.linspace(0.0, 10.0, T),
    "late": np.linspace(0.5, 10.0, T),
    "log": np.concatenate([[0.0], np.geomspace(1e-3, 10.0, T - 1)]),
}


def _system():
    sy = MuonSpinSystem(SPINS)
    sy.add_hyperfine_term(0, A[0], 1)
    sy.add_hyperfine_term(2, A[1], 1)
    return sy


def _rows():
    rng = np.random.default_rng(7)
    return np.stack([np.arccos(rng.uniform(-1, 1, N)), rng.uniform(0, 2 * np.pi, N)], axis=1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", ["zero log late", "log late zero", "late zero log", "zero late log"])
def test_grid_changes_on_a_kept_plan(order, precision):
    sy, rows, B = _system(), _rows(), np.array([0.0, 0.0, 0.02])
    powder._PLANS.clear()
    at = [0, 1, T // 3, T - 1]
    for name in order.split():
        got = powder.powder_average(sy, rows, B, (0.0, 0.0, 1.0), GRIDS[name], precision=precision)
        ref = port.powder_average(oracle_system(SPINS, COUPLINGS), rows, B, np.array([0.0, 0.0, 1.0]),
                                  np.inf, GRIDS[name][at])
        assert np.abs(got[at] - ref).max() <= TOL[precision]
        (plan,) = powder._PLANS.values()
        need = ctypes.c_size_t(0)
        assert _lib.load().msp_powder_workspace(ctypes.byref(plan.args), ctypes.byref(need)) == 0
        assert plan.args.workspace_bytes >= need.value  # the form of this grid, not a lesser one


def test_grid_changes_on_a_kept_scan():
    sy = _system()
    grid = powder.OrientationGrid("zcw", 400)
    fields = np.linspace(0.01, 0.04, 4)
    for name in ("zero", "log", "late"):
        powder._PLANS.clear()
        fresh = powder.powder_scan(sy, grid, fields, (0.0, 0.0, 1.0), GRIDS[name])
        powder._PLANS.clear()
        for other in GRIDS:
            powder.powder_scan(sy, grid, fields, (0.0, 0.0, 1.0), GRIDS[other])
        kept = powder.powder_scan(sy, grid, fields, (0.0, 0.0, 1.0), GRIDS[name])
        assert np.abs(kept - fresh).max() <= 1e-12  # the same sums up to rounding
