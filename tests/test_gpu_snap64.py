"""FP64 eigenpairs from FP32 vectors and one FP64 step (msp_snap64.cu), at
the sizes where its buffers, thread groups and first stage change, and on
spectra that take its cluster and Jacobi branches.

Tolerances: backward stable eigenpairs have residuals and deviations from
orthonormality of a few n^(1/2) units of rounding per entry; 16 n eps of the
norm bounds both, and the levels by Weyl's inequality (numpy's own error
included)."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels, workloads
from muspinsim_gb300 import quaternion as Q
from muspinsim_gb300.orientations import orientation_rows_to_quats, zcw_gen
from tests.helpers import oracle_powder, random_hermitian

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _check(H):
    n = H.shape[-1]
    e, v, st = (x.cpu().numpy() for x in kernels.eigh(H))
    assert (st == 0).all()
    for k in range(len(H)):
        norm = max(np.linalg.norm(H[k], 2), 1e-300)
        tol = 16 * n * EPS
        assert np.linalg.norm(H[k] @ v[k] - v[k] * e[k]) <= tol * norm * np.sqrt(n)
        assert np.linalg.norm(v[k].conj().T @ v[k] - np.eye(n)) <= tol * np.sqrt(n)
        assert np.abs(e[k] - np.linalg.eigvalsh(H[k])).max() <= tol * norm


@pytest.mark.parametrize("n", [2, 3, 5, 8, 13, 24, 31, 32, 33, 48, 63, 64])
def test_random(n):
    rng = np.random.default_rng(n)
    _check(np.array([random_hermitian(rng, n) for _ in range(5)]))


# 1e-20 and 1e20 leave the range of the FP32 stages (FP64 Jacobi); 1e-9 and
# 1e9 do not
@pytest.mark.parametrize("scale", [1e-20, 1e-9, 1e9, 1e20])
@pytest.mark.parametrize("n", [4, 24, 40])
def test_scales(n, scale):
    rng = np.random.default_rng(n)
    _check(scale * np.array([random_hermitian(rng, n) for _ in range(3)]))


# one rotation: any scale, diagonal and degenerate matrices, one snapshot and many
@pytest.mark.parametrize("scale", [1e-100, 1e-20, 1.0, 1e20, 1e100])
@pytest.mark.parametrize("n", [1, 2])
def test_two_levels(n, scale):
    rng = np.random.default_rng(n)
    H = np.array([random_hermitian(rng, n) for _ in range(300)])
    H[0] = np.diag(np.arange(n))
    H[1] = np.eye(n)
    H[2, -1, 0] *= 1e-9
    H[2, 0, -1] = np.conj(H[2, -1, 0])
    _check(scale * H)
    H[3, 0, -1] = H[3, -1, 0] = np.nan
    st = kernels.eigh(scale * H)[2].cpu().numpy()
    assert st[3] == 1 and st.sum() == 1


@pytest.mark.parametrize("n", [4, 8, 24, 32, 64])
def test_degenerate_and_clustered(n):
    rng = np.random.default_rng(n)
    out = [np.zeros((n, n), dtype=complex), np.eye(n, dtype=complex),
           np.kron(np.eye(2), random_hermitian(rng, n // 2))]
    for gap in (0.0, 1e-13, 1e-10, 1e-7, 1e-4):
        w = np.repeat(rng.normal(0, 100, n // 4), 4) * (1 + gap * rng.normal(size=n))
        q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
        H = (q * w) @ q.conj().T
        out.append(0.5 * (H + H.conj().T))
    _check(np.array(out))


# dim 2 has no warp stage, 4,100 snapshots take the Householder + QL stage
@pytest.mark.parametrize("spins,orient", [(["mu"], 5), (["mu", "e"], 7), (["mu", "F", "F"], 33),
                                          (["mu", "e", "N"], 4100), (["mu", "e", "H", "H", "H"], 9),
                                          (["mu", "e", "H", "H", "N"], 3)])
@pytest.mark.parametrize("temperature", [np.inf, 2.0])
def test_snapshots_match_oracle(spins, orient, temperature):
    rng = np.random.default_rng(orient)
    coup = []
    for i, s in enumerate(spins, start=1):
        if "e" in spins and s != "e":
            coup.append(("hyperfine", {"i": i}, workloads.random_hyperfine(rng)))
        elif i > 1:
            coup.append(("dipolar", {"i": 1, "j": i}, workloads.random_vector(rng, 1.0, 2.0)))
    grid = zcw_gen(orient)
    wl = workloads.Workload("s", spins, coup, grid, np.array([[0.0, 0.0, 0.01]]),
                            np.array([0.0, 0.0, 1.0]), np.linspace(0.0, 10.0, 50), temperature)
    sy = wl.system()
    qs, _ = orientation_rows_to_quats(grid)
    B, p = Q.rotate(qs, wl.fields[0]), Q.rotate(qs, wl.polarization)
    n = int(np.prod(sy.dimension))
    mode = _lib.MODE_FAST if np.isinf(temperature) else _lib.MODE_EVOLVE
    out, st = kernels.powder_run(
        n, sy.hamiltonian_matrix(), sy.zeeman_operators(), B, p, np.full(orient, 1 / orient),
        np.zeros(orient, np.int32), 1, wl.times, mode=mode, dims=list(sy.dimension), mu_index=0,
        gammas=sy.gammas, temperature=None if np.isinf(temperature) else temperature)
    assert int(st.max().item()) == 0
    assert np.abs(out.cpu().numpy()[0] - oracle_powder(wl)).max() <= 1e-10


# rho0 in its closed forms: T = inf, ground state and thermal snapshots of one
# launch, a polarisation that is not a unit vector, the muon not first
@pytest.mark.parametrize("prec,tol", [(_lib.PREC_FP64, 1e-10), (_lib.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("mode", [_lib.MODE_EVOLVE, _lib.MODE_INTEGRAL])
@pytest.mark.parametrize("length", [1.0, 0.5])
def test_temperatures_of_one_launch(prec, tol, mode, length):
    rng = np.random.default_rng(3)
    spins = ["e", "mu", "N"]
    coup = [("hyperfine", {"i": 2}, workloads.random_hyperfine(rng)),
            ("hyperfine", {"i": 3}, workloads.random_hyperfine(rng))]
    temps = np.array([np.inf, 2.0, 0.0, np.inf, 40.0])
    times = np.linspace(0.0, 10.0, 40)
    B = rng.normal(size=(5, 3)) * 0.05
    B[3] = 0.0
    p = rng.normal(size=(5, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    wl = workloads.Workload("s", spins, coup, np.zeros((1, 3)), B[:1], p[0], times)
    sy = wl.system()
    out, st = kernels.powder_run(
        12, sy.hamiltonian_matrix(), sy.zeeman_operators(), B, length * p, np.ones(5),
        np.arange(5, dtype=np.int32), 5, times, mode=mode, precision=prec,
        dims=list(sy.dimension), mu_index=1, gammas=sy.gammas, temperature=temps, tau=2.197)
    assert int(st.max().item()) == 0
    from oracle import port
    from tests.helpers import oracle_system

    osy = oracle_system(spins, coup)
    Z = osy.zeeman_operators()
    for k in range(5):
        H = osy.hamiltonian() + np.einsum("a,aij->ij", B[k], Z)
        rho = port.rho0(osy, B[k], p[k], temps[k])
        op = osy.muon_operator(length * p[k])
        ref = (port.evolve(H, rho, times, [op])[:, 0].real if mode == _lib.MODE_EVOLVE
               else port.integrate_decaying(H, rho, 2.197, [op])[:1].real / 2.197)
        assert np.abs(out[k].cpu().numpy() - ref).max() <= tol


# thermal states of one larger spin per launch, a warp's work: I = 1 ... 9/2
@pytest.mark.parametrize("prec,tol", [(_lib.PREC_FP64, 1e-10), (_lib.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("nucleus", ["N", "Cu", "Al", "V", "Nb"])
def test_thermal_states_of_large_spins(prec, tol, nucleus):
    from oracle import port
    from tests.helpers import oracle_system

    rng = np.random.default_rng(7)
    spins, coup = ["mu", nucleus], [("dipolar", {"i": 1, "j": 2}, workloads.random_vector(rng, 1.0, 2.0))]
    temps = np.array([2e-5, 1e-4, 0.0, 3.0, 1e-6, np.inf])
    S, times = len(temps), np.linspace(0.0, 10.0, 30)
    B = rng.normal(size=(S, 3)) * 0.05
    B[3] = 0.0
    p = rng.normal(size=(S, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    sy = workloads.Workload("s", spins, coup, np.zeros((1, 3)), B[:1], p[0], times).system()
    out, st = kernels.powder_run(
        int(np.prod(sy.dimension)), sy.hamiltonian_matrix(), sy.zeeman_operators(), B, p, np.ones(S),
        np.arange(S, dtype=np.int32), S, times, mode=_lib.MODE_EVOLVE, precision=prec,
        dims=list(sy.dimension), mu_index=0, gammas=sy.gammas, temperature=temps)
    assert int(st.max().item()) == 0
    osy = oracle_system(spins, coup)
    Z = osy.zeeman_operators()
    for k in range(S):
        H = osy.hamiltonian() + np.einsum("a,aij->ij", B[k], Z)
        ref = port.evolve(H, port.rho0(osy, B[k], p[k], temps[k]), times, [osy.muon_operator(p[k])])
        assert np.abs(out[k].cpu().numpy() - ref[:, 0].real).max() <= tol
