"""Celio's fixed-point tensor path (every factor unitary, D <= 16) where its
tiles, packings and rules change: every factor dimension up to 16, partly
filled columns and tiles, merged single-spin factors before and after their
pair, both state forms, and states it must hand back.

The oracle applies the factors one after the other in FP64 numpy.  Its own
rounding is ~n_ops^(1/2) eps of the norm (3e-15 for 200 products); the fixed
point adds 2^-58 per product: 1e-13."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu


def _unitary(rng, D):
    lam, v = np.linalg.eigh(random_hermitian(rng, D, 1.0))
    return (v * np.exp(-1j * lam)) @ v.conj().T


def _apply(U, digits, dims, psi):
    """U on the digits (in the factor's own order) of psi."""
    on = [d for d in digits if d >= 0]
    t = psi.reshape(dims)
    u = U.reshape([dims[d] for d in on] * 2)
    t = np.tensordot(u, t, axes=(list(range(len(on), 2 * len(on))), on))
    return np.moveaxis(t, list(range(len(on))), on).reshape(-1)


def _pure(dims, factors, k, T, states=2, prec=_lib.PREC_FP64, scale=1.0, seed=0):
    rng = np.random.default_rng(seed)
    mats = [scale * _unitary(rng, int(np.prod([dims[d] for d in f if d >= 0]))) for f in factors]
    off = np.cumsum([0] + [m.size for m in mats])
    half = int(np.prod(dims)) // 2
    ph = rng.random((1, states, half))
    n = rng.normal(size=3)
    n /= np.linalg.norm(n)
    sig = np.array([[n[2], n[0] - 1j * n[1]], [n[0] + 1j * n[1], -n[2]]])
    mu = np.linalg.eigh(sig)[1][:, 1]
    block = np.concatenate([m.reshape(-1) for m in mats])
    got, _ = kernels.celio_run(_lib.CELIO_PURE, dims, factors, off[:-1], block[None], False, 1,
                               states, k, T, mu_psi=mu[None], sigma=sig[None], phases=ph,
                               precision=prec, path=1)
    got = got.cpu().numpy()[0]
    ref = np.empty((states, T))
    for a in range(states):
        psi = np.kron(mu, np.exp(2j * np.pi * ph[0, a]) / np.sqrt(half))
        for t in range(T):
            x = psi.reshape(2, half)
            ref[a, t] = np.einsum("ih,ij,jh->", x.conj(), sig, x).real
            for _ in range(k if t + 1 < T else 0):
                for f, m in zip(factors, mats):
                    psi = _apply(m, f, dims, psi)
    return np.abs(got - ref).max()


# D = 2 d for d = 2 .. 8 (packed, padded and full columns), alone and as merged
# products with single-spin factors of every side
@pytest.mark.parametrize("d", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_factor_dimensions(d, prec):
    dims = [2, d, 3, d]
    factors = [(0, 1), (0, 3), (0, 2), (1, -1), (2, -1), (3, -1)]
    assert _pure(dims, factors, 3, 6, prec=prec, seed=d) <= 1e-13


@pytest.mark.parametrize("factors", [
    [(1, -1), (0, 1)], [(1, -1), (1, -1), (0, 1), (1, -1)], [(1, 0), (0, -1), (2, 0), (1, -1)],
    [(0, -1)], [(2, -1), (1, -1)], [(2, 1), (0, -1), (1, 2), (2, -1)], [(1, 2)],
    [(0, 1), (0, -1), (0, 2), (1, -1), (0, -1)]])
def test_merging(factors):
    assert _pure([2, 4, 3], factors, 4, 5, seed=len(factors)) <= 1e-13


@pytest.mark.parametrize("dims", [[2, 2], [2, 3], [2, 2, 3], [2, 8, 8, 8], [2, 8, 8, 8, 8]])
def test_state_sizes(dims):
    factors = [(0, q) for q in range(1, len(dims))] + [(q, -1) for q in range(1, len(dims))]
    assert _pure(dims, factors, 2, 4, states=1 if len(dims) > 4 else 3) <= 1e-13


def test_not_unitary_is_left_to_fp64():
    """Factors that change the norm would leave the fixed-point range: the FP64
    kernel takes the state (norm 1.3^24)."""
    err = _pure([2, 4, 3], [(0, 1), (0, 2)], 3, 5, scale=1.3)
    assert err <= 1e-13 * 1.3 ** 48


def test_density_form():
    rng = np.random.default_rng(4)
    dims = [2, 3]
    D = 6
    U = [_unitary(rng, 6), _unitary(rng, 3)]
    A = rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D))
    rho = A @ A.conj().T
    rho /= np.trace(rho).real
    W = rng.normal(size=(2, D, D)) + 1j * rng.normal(size=(2, D, D))
    digits, mats = [], []
    for u, f in zip(U, [(0, 1), (1, -1)]):
        digits += [f, tuple(2 + q if q >= 0 else -1 for q in f)]
        mats += [u.conj().T, u.T]
    off = np.cumsum([0] + [m.size for m in mats])
    block = np.concatenate([m.reshape(-1) for m in mats])
    got, _ = kernels.celio_run(_lib.CELIO_DENSITY, dims + dims, digits, off[:-1], block[None], False,
                               1, 1, 3, 5, rho0=rho[None], meas=W[None], path=1)
    got = got.cpu().numpy()[0]
    full = [U[0], np.kron(np.eye(2), U[1])]
    for t in range(5):
        assert np.abs(got[t] - np.einsum("ij,oij->o", rho, W)).max() <= 1e-13 * 10
        for _ in range(3):
            for u in full:
                rho = u.conj().T @ rho @ u


def _digits_sum(d2, d3, d4, d5):
    """Integers with the given balanced ten-bit digits, lowest two zero."""
    return [sum(int(v) << 10 * s if v >= 0 else -(int(-v) << 10 * s)
                for s, v in ((2, a), (3, b), (4, c), (5, d)))
            for a, b, c, d in zip(d2, d3, d4, d5)]


def _aligned_row_and_state():
    """A unit row u and a state x (16 complex entries as 32 integers of 2^-58, real
    parts first) whose digits 3 and 4 are all +-511 with the signs aligned: Re u . x
    sums them to 1.04 x 2^24 before the products with the top digits take it back
    below 2^24."""
    rng = np.random.default_rng(0)
    im = np.arange(32) >= 16
    sx = rng.choice([-1, 1], 32)
    x5 = sx * rng.integers(34, 42, 32)
    u2 = 511 * sx * np.where(im, -1, 1)
    u3 = np.full(32, -511)
    u3[31] = -510  # an odd total
    u4 = np.full(32, -511)
    frac = u4 / 2**10 + u3 / 2**20 + u2 / 2**30
    while True:
        u5 = rng.choice([-1, 1], 32) * rng.integers(38, 52, 32)
        # the last two entries give the sum and the sum of squares a unit row needs
        A, B = 16 - u5[:30].sum(), 65544 - (u5[:30] ** 2).sum()
        root = int(round(max(2 * B - A * A, 0) ** 0.5))
        if root * root != 2 * B - A * A or (A + root) % 2:
            continue
        u5[30], u5[31] = (A + root) // 2, (A - root) // 2
        if np.abs(((u5 + frac) ** 2).sum() / 65536 - 1) < 7e-10:
            break
    x2 = 511 * np.sign(u5) * np.where(im, 1, -1)
    x3 = np.where(im, 511, -511)
    return _digits_sum(u2, u3, u4, u5), _digits_sum(x2, x3, x3, x5)


def test_aligned_digits():
    """Digits that align beyond what an FP32 accumulator holds exactly: the state
    goes to the FP64 kernel (an entry is a sum of 32 products of a unit row and a
    state of norm below 1: 2^-48), it does not lose the 2^-46 that a rounded sum
    would."""
    u, x = _aligned_row_and_state()
    rng = np.random.default_rng(1)
    row = (np.array(u[:16], float) + 1j * np.array(u[16:], float)) * 2.0**-58
    q = np.linalg.qr(np.concatenate([row[None], rng.normal(size=(15, 16)) + 0j]).conj().T)[0]
    M = q.conj().T
    M[0] = row
    psi = (np.array(x[:16], float) + 1j * np.array(x[16:], float)) * 2.0**-58
    pick = np.zeros((1, 16))
    pick[0, 0] = 1.0
    got, _ = kernels.celio_run(_lib.CELIO_DENSITY, [4, 4], [(0, 1)], [0], M.reshape(1, -1), False, 1,
                               1, 1, 2, rho0=psi[None], meas=pick[None], path=1)
    got = got.cpu().numpy()[0, 1, 0]
    exact = (sum(a * b for a, b in zip(u[:16], x[:16])) - sum(a * b for a, b in zip(u[16:], x[16:])),
             sum(a * b for a, b in zip(u[:16], x[16:])) + sum(a * b for a, b in zip(u[16:], x[:16])))
    assert abs(got.real - exact[0] / 2**116) <= 2.0**-47.5
    assert abs(got.imag - exact[1] / 2**116) <= 2.0**-47.5


# a spin of I = 0 has one state, and its digit the stride of the digit before it
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("dims", [[2, 1, 5], [2, 1, 1, 3], [2, 3, 1]])
def test_digits_of_dimension_one(dims, prec):
    last = len(dims) - 1
    factors = [(0, 1), (1, 0), (0, last), (last, 1), (1, -1)] + [(1, 2)] * (last > 1)
    # 36 products of 2^-40 each in double-words
    tol = 1e-13 if prec == _lib.PREC_FP64 else 1e-10
    assert _pure(dims, factors, 2, 4, prec=prec, seed=last) <= tol


# the integer form of small factors where its lanes per group and its rounds change:
# one group, a lane per row, rows shared by fewer lanes, more groups than threads
@pytest.mark.parametrize("d", [1, 2, 3, 4])
@pytest.mark.parametrize("groups", [1, 7, 31, 32, 33, 64, 65, 128, 129, 255, 257])
def test_small_factors(d, groups):
    dims, factors = [2, d, groups], [(0, 1), (0, -1)] + ([(1, -1)] if d > 1 else [])
    assert _pure(dims, factors, 2, 4, seed=groups + d) <= 1e-13
