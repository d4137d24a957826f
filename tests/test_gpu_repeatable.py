"""FP64 results repeat bit for bit: every sum has a fixed order, whatever the order
in which blocks and warps come to it.  Sizes on both sides of n = 64, one to
eight CTAs per snapshot, close levels, all three modes."""

import numpy as np
import pytest
import torch

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu


def _matrices(n, seed):
    rng = np.random.default_rng(seed)
    H = random_hermitian(rng, n)
    lam, U = np.linalg.eigh(H)
    lam[n // 2] = lam[n // 2 - 1] + 1e-9  # a pair that is nearly degenerate
    H = (U * lam) @ U.conj().T
    Z = np.array([1e-3 * random_hermitian(rng, n) for _ in range(3)])
    return 0.5 * (H + H.conj().T), Z, rng


@pytest.mark.parametrize("n,S", [(4, 3000), (12, 1000), (24, 500), (32, 300), (48, 200), (64, 100),
                                 (66, 40), (96, 1), (96, 60), (192, 20), (256, 4)])
@pytest.mark.parametrize("mode", [_lib.MODE_FAST, _lib.MODE_EVOLVE, _lib.MODE_INTEGRAL])
def test_powder(n, S, mode):
    H, Z, rng = _matrices(n, n)
    p = rng.normal(size=(S, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    dims = _primes(n)
    kw = dict(dims=dims, mu_index=0, gammas=[135.5] + [40.0] * (len(dims) - 1)) if mode else {}
    plan = kernels.PowderPlan(n, H, Z, rng.normal(size=(S, 3)), p, np.ones(S),
                              np.arange(S, dtype=np.int32), S, np.linspace(0.0, 3.0, 65), mode=mode,
                              rho_fac=_uniform(dims, S) if mode and max(dims) > 10 else None, **kw)
    first = plan.run().clone()
    for _ in range(8):
        assert torch.equal(plan.run(), first)


def _primes(n):
    d, out = 2, []
    while n > 1:
        while n % d == 0:
            out.append(d)
            n //= d
        d += 1
    return out


def _uniform(dims, S):
    fac = [np.diag([1.0, 0.0]).ravel()] + [np.eye(d).ravel() / d for d in dims[1:]]
    return np.tile(np.concatenate(fac).astype(complex), (S, 1))


@pytest.mark.parametrize("n", [3, 8, 24, 33, 64, 70])
def test_eigh(n):
    H = np.array([_matrices(n, 100 * n + k)[0] for k in range(40)])
    first = [x.clone() for x in kernels.eigh(H)]
    for _ in range(8):
        assert all(torch.equal(a, b) for a, b in zip(kernels.eigh(H), first))
