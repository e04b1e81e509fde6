"""Edges of the quartet kernels' dispatch against the oracle: the two sides of
the Boys table's end, ragged batches of the high-L primitive blocks, short
work lists split over the primitives."""

from __future__ import annotations

import ctypes
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

import oracle
from jax_examples_b200 import DirectERI, _abi, eri_prim_quartets
from jax_examples_b200 import basis as pb
from jax_examples_b200.grad import grad_two_electron

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


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("cls", [(2, 2, 2, 1), (2, 2, 2, 2)])
def test_high_l_primitive_blocks_ragged(cls, n, aligned):
    """Blocks of eight quartets: remainders, and an output array that is only
    8-byte aligned (a C caller's).  Tolerance of the target, 1e-10 of the
    largest element; nothing is written beyond the last block."""
    rng = np.random.default_rng(100 * n + cls[3])
    ex = 10 ** rng.uniform(-1, 1, (n, 4))
    ctr = rng.uniform(0, 2.5, (n, 4, 3))
    shape = (6, 6, 6, 6 if cls[3] == 2 else 3)
    size = n * int(np.prod(shape))
    buf = torch.full((size + 3,), 7.25, dtype=torch.float64, device=DEV)
    out = buf[0 if aligned else 1:][:size]
    e, c = (torch.tensor(x, device=DEV) for x in (ex, ctr))
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _abi.call("jqc_eri_prim_quartets", *cls, n, ptr(e), ptr(c), ptr(out),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    got = out.cpu().numpy().reshape((n,) + shape)
    for q in range(n):
        args = [x for k in range(4) for x in (ex[q, k], ctr[q, k], cls[k])]
        ref = oracle.primitive_eri(*args, mode=1)
        np.testing.assert_allclose(got[q], ref, rtol=0, atol=1e-10 * np.abs(ref).max())
    rest = torch.cat([buf[: 0 if aligned else 1], buf[(0 if aligned else 1) + size:]])
    assert bool((rest == 7.25).all())


@pytest.mark.parametrize("basis,lane_prims", [("sto-3g", 1), ("6-31g*", 7), ("6-31g*", 16), ("6-31g**", 256)])
def test_short_lists_split_over_primitives(basis, lane_prims):
    """Lists cut into tasks of few primitives (and the limit itself, which takes
    16 at these sizes) give the J/K and the gradient of the largest tasks to
    1e-12: the same integrals, summed in another order."""
    mol = pb.water_cluster(1, seed=2, noise_angstrom=0.05)
    bs = pb.build_basis_set(mol, basis)
    rng = np.random.default_rng(5)
    n = bs.n_basis
    a = rng.standard_normal((2, n, n)) * 0.1
    D = torch.tensor(a + a.transpose(0, 2, 1), device=DEV)
    res = []
    for engine, lanes in ((0, lane_prims), (2, 256)):  # (2: the warp engine of the gradient)
        eng = DirectERI(bs, mol, device=0, schwarz_tau=0.0)
        cfg = np.zeros(84, dtype=np.int32)
        _abi.call("jqc_get_tuning", eng._ctx, cfg.ctypes.data_as(_abi._ip))
        cfg.reshape(21, 4)[:, 1] = lanes
        _abi.call("jqc_set_tuning", eng._ctx, cfg.ctypes.data_as(_abi._ip))
        if engine:
            for q in range(21):
                _abi.call("jqc_set_grad_engine", eng._ctx, q, engine)
        J, K = eng.jk(D)
        res.append((J, K, grad_two_electron(eng, list(D), 1.0, 1.0)))
        eng.close()
    for x, y in zip(*res):
        scale = float(y.abs().max())
        assert float((x - y).abs().max()) < 1e-12 * max(1.0, scale)


@pytest.mark.parametrize("threads", [1, 4])
def test_contexts_made_and_destroyed_share_side_streams(threads):
    """Side streams outlive their context: contexts created, used and destroyed
    one after another and in several threads at once, each thread on a stream of
    its own, give the J/K of a fresh context (1e-12; the order of the atomics
    differs)."""
    mol = pb.water_cluster(2, seed=3)
    bs = pb.build_basis_set(mol, "6-31g*")
    n = bs.n_basis
    a = np.random.default_rng(1).standard_normal((n, n)) * 0.1
    D = torch.tensor(a + a.T, device=DEV)
    eng = DirectERI(bs, mol, device=0)
    J0, K0 = eng.jk(D)
    torch.cuda.synchronize()

    def work(_):
        with torch.cuda.stream(torch.cuda.Stream(DEV)):
            worst = 0.0
            for _ in range(5):
                e = DirectERI(bs, mol, device=0)
                J, K = e.jk(D)
                e.close()
                worst = max(worst, float((J - J0).abs().max()), float((K - K0).abs().max()))
            return worst

    with ThreadPoolExecutor(threads) as ex:
        assert max(ex.map(work, range(threads))) < 1e-12
    eng.close()
