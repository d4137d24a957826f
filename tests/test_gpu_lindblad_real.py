"""The real form of the dissipative evolution (uniform grids, n^2 <= 64) at its
edges: every superoperator size up to 64, sample counts around the giant-step
chunks, an offset start, no dissipation left at T = 0, a strongly damped spin.

Oracle: numpy's eig of the superoperator; it and the scaled exponential are
good to a few 1e-13 on these norms (2 pi |L| t ~ 1e3), so 1e-10 as elsewhere."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels, workloads
from muspinsim_gb300 import quaternion as Q
from muspinsim_gb300.orientations import orientation_rows_to_quats, zcw_gen
from oracle import port
from tests.helpers import oracle_system

pytestmark = pytest.mark.gpu


def _compare(spins, diss, times, temperature, prec=_lib.PREC_FP64, orient=3, scale=10.0):
    rng = np.random.default_rng(len(times))
    coup = [("hyperfine", {"i": i + 1}, workloads.random_hyperfine(rng, scale))
            for i, s in enumerate(spins) if s != "e" and "e" in spins]
    grid = zcw_gen(orient)
    wl = workloads.Workload("l", spins, coup, grid, np.array([[0.0, 0.0, 0.003]]),
                            np.array([0.0, 0.0, 1.0]), times, temperature)
    sy = wl.system()
    qs, _ = orientation_rows_to_quats(grid)
    B, p = Q.rotate(qs, wl.fields[0]), Q.rotate(qs, wl.polarization)
    n = int(np.prod(sy.dimension))
    ops = np.array([[sy.operator({i: ax}).matrix.toarray() for ax in "xyz"]
                    for i in range(len(spins))], dtype=complex)
    out, st = kernels.lindblad_run(
        n, sy.hamiltonian_matrix(), sy.zeeman_operators(), ops, list(sy.dimension),
        sy.muon_index, sy.gammas, diss, B, p, np.full(orient, 1 / orient),
        np.zeros(orient, np.int32), 1, times, temperature=temperature, precision=prec)
    assert int(st.max().item()) == 0
    ref = port.powder_average(oracle_system(spins, coup), grid, wl.fields[0], wl.polarization,
                              temperature, times, dissipation=diss)
    return np.abs(out.cpu().numpy()[0] - ref).max()


# n = 2, 4, 6, 8: N = 4, 16, 36, 64 (all 16-row bands); the muon anywhere
@pytest.mark.parametrize("spins,diss", [(["mu"], {0: 0.4}), (["mu", "e"], {1: 2.0}),
                                        (["mu", "N"], {1: 0.7}), (["e", "mu", "H"], {0: 1.0, 2: 0.2}),
                                        (["mu", "e", "H"], {0: 0.1, 1: 2.0, 2: 0.3})])
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_sizes(spins, diss, prec):
    assert _compare(spins, diss, np.linspace(0.0, 6.0, 90), 5.0, prec) <= 1e-10


# one sample, one step, either side of a giant step and of a chunk of them
@pytest.mark.parametrize("nt", [1, 2, 7, 8, 9, 63, 64, 65, 1024, 1025, 4097])
@pytest.mark.parametrize("t0", [0.0, 0.25])
def test_sample_counts(nt, t0):
    assert _compare(["mu", "e"], {1: 2.0}, t0 + 0.004 * np.arange(nt), 20.0) <= 1e-10


# few samples of long steps: up to five squarings of the step are left out
@pytest.mark.parametrize("spins,diss", [(["mu", "e"], {1: 2.0}), (["mu", "N"], {1: 0.7}),
                                        (["mu", "e", "H"], {0: 0.1, 2: 0.3})])
@pytest.mark.parametrize("nt", [2, 3, 5, 9, 17, 33, 40])
@pytest.mark.parametrize("t0", [0.0, 0.6])
def test_long_steps(spins, diss, nt, t0):
    assert _compare(spins, diss, t0 + 0.3 * np.arange(nt), 20.0) <= 1e-10


@pytest.mark.parametrize("temperature", [np.inf, 0.0])
@pytest.mark.parametrize("rate", [0.0, 50.0])
def test_rates_and_temperatures(temperature, rate):
    assert _compare(["mu", "e", "H"], {1: rate}, np.linspace(0.0, 4.0, 120), temperature) <= 1e-10


@pytest.mark.parametrize("bad", ["field", "pol"])
def test_vectors_of_the_wrong_length_are_refused(bad):
    sy = workloads.Workload("l", ["mu"], [], zcw_gen(1), np.zeros((1, 3)), np.array([0.0, 0.0, 1.0]),
                            np.zeros(1), 5.0).system()
    ops = np.array([[sy.operator({0: ax}).matrix.toarray() for ax in "xyz"]], dtype=complex)
    vec = {"field": np.zeros((2, 3)), "pol": np.ones((2, 3)), bad: np.ones(7)}
    with pytest.raises(RuntimeError):
        kernels.lindblad_run(2, sy.hamiltonian_matrix(), sy.zeeman_operators(), ops, [2], 0, sy.gammas,
                             {0: 0.1}, vec["field"], vec["pol"], np.ones(2), np.zeros(2, np.int32), 1,
                             np.linspace(0, 1, 5))
