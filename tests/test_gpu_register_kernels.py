"""Edges of the register kernels' dispatch: the two sides of the Boys table's
end, per class, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from jax_examples_b200 import eri_prim_quartets

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("cls", [(0, 0, 0, 0), (1, 0, 0, 0), (1, 0, 1, 0), (1, 1, 1, 0), (1, 1, 1, 1), (2, 1, 1, 1),
                                 (2, 2, 1, 1)])
def test_primitive_blocks_at_the_end_of_the_boys_table(cls):
    """Both pairs on one centre each (K = 1, no cancellation in P - Q) and all
    exponents 1, so T = |PQ|^2: grid points, midpoints and both sides of every
    switch between table and closed form.  Tolerance: 2e-14 of the largest
    element (the oracle's Boys bound) times (2L-1)!!, the growth of rounding in
    the alternating Hermite recursion."""
    L = sum(cls)
    ends = [36.0] + [42.0 + 3 * m for m in range(1, 7)]
    T = np.array([0.0, 1e-12, 1 / 32, 1 / 16, 0.99, 17.03125]
                 + [e + d for e in ends for d in (-0.04, -1e-9, 1e-9, 0.04)] + [100.0, 2000.0])
    rng = np.random.default_rng(3)
    u = rng.standard_normal((len(T), 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    ctr = np.zeros((len(T), 4, 3))
    ctr[:, 2] = ctr[:, 3] = u * np.sqrt(T)[:, None]
    ex = np.ones((len(T), 4))
    got = eri_prim_quartets(cls, torch.tensor(ex, device=DEV), torch.tensor(ctr, device=DEV)).cpu().numpy()
    tol = 2e-14 * float(np.prod(np.arange(1, 2 * L, 2)))
    for q in range(len(T)):
        ref = oracle.primitive_eri(1.0, ctr[q, 0], cls[0], 1.0, ctr[q, 1], cls[1], 1.0, ctr[q, 2], cls[2],
                                   1.0, ctr[q, 3], cls[3], mode=1)
        np.testing.assert_allclose(got[q], ref, rtol=0, atol=tol * np.abs(ref).max(), err_msg=f"T={T[q]!r}")
