"""FP32 reductions to tridiagonal form of matrices with columns whose squares
underflow: a block beside another one that is 1e-21 of its size (the two do not
couple), and columns left over as rounding errors of rounding errors.  n = 24 and
32 in a batch that takes the warp reduction, 192 with the matrix in shared
memory, 258 in panels.

Reference: numpy's eigenpairs, as in tests/test_gpu_large.py.  The small block's
levels move P(t) by less than 2 pi 1e-19, so the bound is MIXED's 1e-6."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian
from tests.test_gpu_sparse_rows import _signal, TIMES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(24, 4200), (32, 4200), (192, 2), (258, 2)])
@pytest.mark.parametrize("form", ["blocks", "classes"])
def test_tiny_columns(n, S, form):
    rng = np.random.default_rng(n)
    H = 0.02 * random_hermitian(rng, n)
    i = np.arange(n)
    if form == "blocks":
        small = i >= n // 2
        H = np.where(small[:, None] == small, H, 0.0) * np.where(small, 1e-21, 1.0)
    else:
        H = np.where((i * i[:, None]) % 5 == 1, H, 0.0)
    p = np.array([0.6, 0.0, 0.8])
    out, st = kernels.powder_run(n, H, np.zeros((3, n, n), dtype=complex), np.zeros((S, 3)),
                                 np.tile(p, (S, 1)), np.full(S, 1.0 / S), np.zeros(S, dtype=np.int32),
                                 1, TIMES, precision=_lib.PREC_MIXED)
    assert int(st.max().item()) == 0
    assert np.abs(out.cpu().numpy()[0] - _signal(H, p)).max() <= 1e-6
