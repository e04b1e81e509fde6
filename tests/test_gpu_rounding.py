"""Rounding of the quartet kernels over the full exponent range, against the
closed forms of s-type integrals in 80-bit arithmetic.  Every tolerance is the
sum of the roundings on the path in units of u = 2^-53 (a library root: 2 u)."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from jax_examples_b200 import DirectERI, eri_prim_quartets

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
U = 2.0 ** -53
LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")


def _ssss(exps, centres):
    return eri_prim_quartets((0, 0, 0, 0), torch.tensor(exps, device=DEV),
                             torch.tensor(centres, device=DEV)).cpu().numpy().reshape(-1)


def _exponents(rng, n, binades):
    return rng.uniform(1.0, 2.0, (n, 4)) * 2.0 ** rng.integers(-binades, binades + 1, (n, 4))


@pytest.mark.parametrize("binades", [1, 12, 150])
def test_root_of_the_exponent_sum(binades):
    """One centre: (ss|ss) = 2 pi^{5/2} / (p q sqrt(p+q)).  Exponent sums 1 u a side,
    in 1/p, 1/q and the root 3 u; quotients and their products 2 x 2 u and the
    constant's 1.1 u; product of the sides 1 u, root 2 u, last product 1 u."""
    rng = np.random.default_rng(binades)
    ex = _exponents(rng, 4096, binades)
    p, q = LD(1) * ex[:, 0] + ex[:, 1], LD(1) * ex[:, 2] + ex[:, 3]
    ref = 2 * PI ** 2 * np.sqrt(PI) / (p * q * np.sqrt(p + q))
    got = _ssss(ex, np.zeros((len(ex), 4, 3)))
    err = (got - ref) / ref
    assert float(np.abs(err).max()) < 12.1 * U


@pytest.mark.parametrize("binades", [1, 12, 60])
@pytest.mark.parametrize("spread", [0.0, 0.25])
def test_root_of_the_separation_and_pair_quotients(binades, spread):
    """Pairs so far apart that F_0 is its closed form: (ss|ss) = pi^3 K_ab K_cd /
    ((pq)^{3/2} |PQ|).  As above without the root of p+q (11 u), half the 8 u of pq
    |PQ|^2 in its place, two more products 2 u; with the centres of a pair apart,
    P and Q 2 x 4 u, and for each pair 10 u times the exponent x of its K = e^{-x} (5 u
    for |AB|^2, 4 u for alpha beta / p, their product) and 2 u for the exponential."""
    rng = np.random.default_rng(17 + binades)
    n = 4096
    ex = _exponents(rng, n, binades)
    p, q = ex[:, 0] + ex[:, 1], ex[:, 2] + ex[:, 3]
    R = np.sqrt(2.0 ** rng.uniform(10, 30, n) / np.minimum(p, q))
    unit = rng.standard_normal((3, n, 3))
    unit /= np.linalg.norm(unit, axis=2)[:, :, None]
    ctr = np.zeros((n, 4, 3))
    ctr[:, 2] = ctr[:, 3] = unit[0] * R[:, None]
    if spread:
        for k, (i, j) in enumerate(((0, 1), (2, 3))):
            mu = ex[:, i] * ex[:, j] / (ex[:, i] + ex[:, j])
            d = np.minimum(np.sqrt(rng.uniform(0, 300, n) / mu), spread * R)
            ctr[:, j] = ctr[:, i] + unit[1 + k] * d[:, None]
    e, c = LD(1) * ex, LD(1) * ctr
    p, q = e[:, 0] + e[:, 1], e[:, 2] + e[:, 3]
    P = (e[:, :1] * c[:, 0] + e[:, 1:2] * c[:, 1]) / p[:, None]
    Q = (e[:, 2:3] * c[:, 2] + e[:, 3:] * c[:, 3]) / q[:, None]
    r2 = ((P - Q) ** 2).sum(1)
    assert float((p * q / (p + q) * r2).min()) > 45.0
    xab = e[:, 0] * e[:, 1] / p * ((c[:, 0] - c[:, 1]) ** 2).sum(1)
    xcd = e[:, 2] * e[:, 3] / q * ((c[:, 2] - c[:, 3]) ** 2).sum(1)
    ref = PI ** 3 * np.exp(-xab - xcd) / ((p * q) * np.sqrt(p * q * r2))
    err = (_ssss(ex, ctr) - ref) / ref
    tol = (11 + 4 + 2 + (0 if not spread else 8 + 10 * (xab + xcd) + 4)) * U
    assert float((np.abs(err) / tol).max()) < 1.0


@pytest.mark.parametrize("path", ["blocks", "tensor"])
def test_no_rounding_common_to_all_integrals(path):
    """The mean signed error of many one-centre (ss|ss) is the error that they
    share: 0.2 u of the constant 8 pi^{5/2}, and 0.15 u for the scatter left by the
    mean (five standard errors of about 0.5 u a pair over 820 pairs, 1.2 u a
    quartet over 4096 quartets)."""
    rng = np.random.default_rng(8)
    if path == "blocks":
        ex = _exponents(rng, 4096, 6)
        got = _ssss(ex, np.zeros((len(ex), 4, 3)))
        p, q = LD(1) * ex[:, 0] + ex[:, 1], LD(1) * ex[:, 2] + ex[:, 3]
    else:
        ex = _exponents(rng, 10, 6).reshape(-1)
        shells = [SimpleNamespace(angular_momentum=0, exponents=[x], coefficients=[1.0], center=[0.3, -0.1, 0.2],
                                  atom_index=0) for x in ex]
        eng = DirectERI(SimpleNamespace(shells=shells), device=0, schwarz_tau=0.0, prim_tau=0.0)
        got = eng.eri_tensor().cpu().numpy()
        eng.close()
        p = (LD(1) * ex[:, None] + ex[None, :])[:, :, None, None]
        q = p.reshape(1, 1, len(ex), len(ex))
    ref = 2 * PI ** 2 * np.sqrt(PI) / (p * q * np.sqrt(p + q))
    assert abs(float(((got - ref) / ref).mean())) < 0.35 * U
