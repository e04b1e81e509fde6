"""What a J/K build of a context launches and keeps: the autotuner's lists and
accumulators, the launch count of the statistics, the accumulator copies of
several densities and of matrix sizes on both sides of their limits."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch
from cuda.bindings import runtime as rt

from jax_examples_b200 import DirectERI, _abi
from jax_examples_b200 import basis as pb

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _engine(waters, basis, seed=4, **kw):
    mol = pb.water_cluster(waters, seed=seed, noise_angstrom=0.05)
    return DirectERI(pb.build_basis_set(mol, basis), mol, device=0, **kw)


def _densities(eng, n_dens, seed=0):
    n = eng.packed.n_cart
    a = np.random.default_rng(seed).standard_normal((n_dens, n, n)) * 0.1
    return torch.tensor(a + a.transpose(0, 2, 1), device=DEV)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _captured_nodes(eng, D):
    """(kernels, memsets) of a build captured into a graph."""
    J, K = torch.empty_like(D), torch.empty_like(D)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        _abi.call("jqc_jk", eng._ctx, len(D), _ptr(D), _ptr(J), _ptr(K), 0, 0.0, 0.0,
                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    raw = rt.cudaGraph_t(g.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(raw)
    err, nodes, count = rt.cudaGraphGetNodes(raw, count)
    kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes[:count]]
    return (sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds),
            sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeMemset for k in kinds))


def _autotune(eng, D, path=b""):
    J, K, hit = torch.empty_like(D), torch.empty_like(D), ctypes.c_int()
    _abi.call("jqc_autotune", eng._ctx, len(D), _ptr(D), _ptr(J), _ptr(K), 0, 0.0, 0.0, path, ctypes.byref(hit),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return hit.value


def test_autotune_times_the_builds_that_follow(tmp_path):
    """On a list too short for lane_prims to matter the value stays at its
    default; the accumulator copies are there (one memset, not J's and K's); a
    cache line of another version is not taken."""
    path = str(tmp_path / "tune").encode()
    eng = _engine(1, "6-31g*")
    D = _densities(eng, 1)
    assert _autotune(eng, D, path) == 0
    cfg = np.zeros(84, dtype=np.int32)
    _abi.call("jqc_get_tuning", eng._ctx, cfg.ctypes.data_as(_abi._ip))
    assert set(cfg.reshape(21, 4)[:, 1]) == {256}
    assert _captured_nodes(eng, D)[1] == 1
    assert _autotune(eng, D, path) == 1
    text = open(path).read()
    open(path, "w").write(text.replace("jqc-tune2", "jqc-tune1"))
    assert _autotune(eng, D, path) == 0
    eng.close()


@pytest.mark.parametrize("copies", [True, False])
@pytest.mark.parametrize("basis", ["sto-3g", "6-31g*"])
def test_launch_count_of_the_statistics(basis, copies):
    """launches_per_jk is the number of kernels in a captured build, with
    accumulator copies and (two densities, captured before any build of two)
    without them."""
    eng = _engine(2, basis)
    D = _densities(eng, 1 if copies else 2)
    eng.jk(_densities(eng, 1))
    kernels, memsets = _captured_nodes(eng, D)
    assert memsets == (1 if copies else 2)
    assert kernels == eng.stats("fp64")["launches_per_jk"]
    eng.close()


def _tune(eng, lane_prims=None, engine=None):
    cfg = np.zeros(84, dtype=np.int32)
    _abi.call("jqc_get_tuning", eng._ctx, cfg.ctypes.data_as(_abi._ip))
    if lane_prims is not None:
        cfg.reshape(21, 4)[:, 1] = lane_prims
    if engine is not None:
        cfg.reshape(21, 4)[:, 3] = engine
    _abi.call("jqc_set_tuning", eng._ctx, cfg.ctypes.data_as(_abi._ip))


@pytest.mark.parametrize("waters,lane_prims", [(2, 5), (4, 5), (12, 5), (12, 256)])
def test_lists_of_several_host_threads(waters, lane_prims):
    """Lists of one, four and sixteen host threads, cut with remainders on both
    sides of a quartet (5 of 9 and 36 primitive pairs), give the J/K of the
    runtime-class engine, whose tasks have one ket each (same integrals in
    another order: 1e-12 of the largest element)."""
    eng = _engine(waters, "6-31g*", schwarz_tau=1e-10)
    D = _densities(eng, 1)
    _tune(eng, engine=2)
    J0, K0 = eng.jk(D)
    tasks = eng.stats("fp64")["tasks"]
    eng.close()
    eng = _engine(waters, "6-31g*", schwarz_tau=1e-10)
    _tune(eng, lane_prims=lane_prims)
    J, K = eng.jk(D)
    st = eng.stats("fp64")
    assert st["tasks"] != tasks
    assert (st["kept_pairs"] >= 512) == (waters >= 4) and (st["kept_pairs"] >= 4096) == (waters >= 12)
    for x, y in ((J, J0), (K, K0)):
        assert float((x - y).abs().max()) < 1e-12 * float(y.abs().max())
    eng.close()
