"""What a J/K build of a context launches and keeps: the autotuner's lists and
accumulators, the launch count of the statistics, the accumulator copies of
several densities and of matrix sizes on both sides of their limits."""

from __future__ import annotations

import ctypes
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from jax_examples_b200 import DirectERI, _abi
from jax_examples_b200 import basis as pb
from jax_examples_b200.grad import grad_two_electron

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


def _capture(eng, D):
    """A build captured into a graph, and its J and K."""
    J, K = torch.empty_like(D), torch.empty_like(D)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        _abi.call("jqc_jk", eng._ctx, len(D), _ptr(D), _ptr(J), _ptr(K), 0, 0.0, 0.0,
                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return g, J, K


def _captured_nodes(eng, D):
    """(kernels, memsets) of a build captured into a graph."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    g, _, _ = _capture(eng, D)
    raw = rt.cudaGraph_t(g.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(raw)
    err, nodes, count = rt.cudaGraphGetNodes(raw, count)
    kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes[:count]]
    return (sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds),
            sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeMemset for k in kinds))


def _zeroed_bytes(eng, D):
    """Bytes that a captured build sets to zero first."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    g, _, _ = _capture(eng, D)
    raw = rt.cudaGraph_t(g.raw_cuda_graph())
    _, _, count = rt.cudaGraphGetNodes(raw)
    _, nodes, count = rt.cudaGraphGetNodes(raw, count)
    total = 0
    for x in nodes[:count]:
        if rt.cudaGraphNodeGetType(x)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeMemset:
            p = rt.cudaGraphMemsetNodeGetParams(x)[1]
            total += p.elementSize * p.width * max(1, p.height)
    return total


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


@pytest.mark.parametrize("dens_tau", [0.0, 1e-9])
def test_captured_gradient_on_the_side_streams(dens_tau):
    """A gradient captured into a graph forks to the side streams and back: replays
    follow the density in the captured buffer and agree with calls (1e-12 of the
    largest component)."""
    eng = _engine(3, "6-31g*")
    D = _densities(eng, 1)
    g0 = grad_two_electron(eng, list(D), 1.0, 0.5, dens_tau=dens_tau)
    out = torch.zeros_like(g0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _abi.call("jqc_grad2e_ex", eng._ctx, 1, _ptr(D), 1.0, 0.5, dens_tau, _ptr(out),
                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    for seed in (0, 7):
        D.copy_(_densities(eng, 1, seed))
        ref = grad_two_electron(eng, list(D), 1.0, 0.5, dens_tau=dens_tau)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert float((out - ref).abs().max()) < 1e-12 * max(1.0, float(ref.abs().max()))
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


@pytest.mark.parametrize("waters,n_dens,copies", [(2, 3, 4), (2, 4, 4), (22, 4, 4), (23, 4, 2), (32, 4, 2), (33, 4, 1)])
def test_builds_of_several_densities(waters, n_dens, copies):
    """Three and four densities at once, with matrix sizes on both sides of each
    change of the accumulator copies (48 MB), against one density at a time and
    against a build captured and replayed before the copies are there."""
    eng = _engine(waters, "6-31g*", schwarz_tau=1e-7)
    n = eng.packed.n_cart
    assert n == 19 * waters
    D = _densities(eng, n_dens)
    one = [eng.jk(d) for d in D]  # brings the list, and the copies of one density
    g, Jg, Kg = _capture(eng, D)
    g.instantiate()
    g.replay()
    J, K = eng.jk(D)
    assert _zeroed_bytes(eng, D) == copies * 2 * n_dens * n * n * 8
    torch.cuda.synchronize()
    for k in range(n_dens):
        for x, ref in ((J[k], one[k][0]), (K[k], one[k][1]), (Jg[k], one[k][0]), (Kg[k], one[k][1])):
            assert float((x - ref).abs().max()) < 1e-12 * float(ref.abs().max())
    eng.close()


def _uncontracted(basis):
    """The primitives of a basis as shells of their own, and the matrix (n,
    n_primitive) of the contractions."""
    shells, rows, n = [], [], 0
    for s in basis.shells:
        l, m = s.angular_momentum, (s.angular_momentum + 1) * (s.angular_momentum + 2) // 2
        rows.append((n, m, list(s.coefficients)))
        for x in s.exponents:
            shells.append(SimpleNamespace(angular_momentum=l, exponents=[x], coefficients=[1.0], center=s.center,
                                          atom_index=s.atom_index))
            n += m
    T = np.zeros((sum(m for _, m, _ in rows), n))
    at = 0
    for first, m, coefs in rows:
        for k, c in enumerate(coefs):
            T[at:at + m, first + k * m:first + (k + 1) * m] = c * np.eye(m)
        at += m
    return SimpleNamespace(shells=shells), torch.tensor(T, device=DEV)


@pytest.mark.parametrize("basis", ["sto-3g", "6-31g*", "6-31g**"])
def test_split_lists_against_single_primitives(basis):
    """A contracted density's J, K and gradient against those of its primitives as
    shells of their own, whose quartets have nothing to split: lane limits 1, 7
    and 16 (three lists), the limits above it (the list of 16 at this size), and
    every gradient engine code of every class.  1e-12 of the largest element, the
    forces 1e-11: the same integrals summed in another order, forces of steep
    primitives cancel to a tenth."""
    mol = pb.water_cluster(1, seed=2, noise_angstrom=0.05)
    bs = pb.build_basis_set(mol, basis)
    flat, T = _uncontracted(bs)
    eng = DirectERI(bs, mol, device=0, schwarz_tau=0.0, prim_tau=0.0)
    D = _densities(eng, 2)
    ref = DirectERI(flat, mol, device=0, schwarz_tau=0.0, prim_tau=0.0)
    J0, K0 = (T @ x @ T.T for x in ref.jk(T.T @ D @ T))
    g0 = grad_two_electron(ref, list(T.T @ D @ T), 1.0, 1.0)
    ref.close()
    tasks = {}
    for lanes in (1, 7, 16, 64, 256):
        _tune(eng, lane_prims=lanes)
        J, K = eng.jk(D)
        tasks[lanes] = eng.stats("fp64")["tasks"]
        for x, y in ((J, J0), (K, K0)):
            assert float((x - y).abs().max()) < 1e-12 * float(y.abs().max())
    assert tasks[1] > tasks[7] > tasks[16] == tasks[64] == tasks[256]
    eng.close()
    for code in (None, 0, 1, 2, 3):
        e = DirectERI(bs, mol, device=0, schwarz_tau=0.0, prim_tau=0.0)
        for q in range(21):
            L, bra = sum(_CLASS[q]), _CLASS[q][:2]
            ok = {0: L <= 4, 3: L <= 4, 1: bra == (2, 1) and L >= 4 or bra == (2, 2), 2: True}.get(code, False)
            if ok:
                _abi.call("jqc_set_grad_engine", e._ctx, q, code)
            elif code is not None:
                with pytest.raises(ValueError, match="engine"):
                    _abi.call("jqc_set_grad_engine", e._ctx, q, code)
        g = grad_two_electron(e, list(D), 1.0, 1.0)
        assert float((g - g0).abs().max()) < 1e-11 * float(g0.abs().max()), code
        e.close()


_PAIRS = [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]
_CLASS = [_PAIRS[i] + _PAIRS[j] for i in range(6) for j in range(i + 1)]
