"""Treecode sums through cells (many points per epsilon) against the oracle's
treecode: leaves of two cells and of dozens, positions on both sides of 0,
several periods, clusters with deep leaves, one species' lattice columns."""
import numpy as np
import pytest

import oracle as O
import multi_species_b200 as M

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("L,eps,n,leaf,mac,deg,kind", [
    (20 * np.pi, 0.02, 60000, 2000, 0.7, 8, "uniform"),
    (20 * np.pi, 0.02, 60000, 100, 0.7, 8, "positive"),
    (4 * np.pi, 0.05, 30001, 500, 0.5, 6, "uniform"),
    (4 * np.pi, 0.05, 30001, 1500, 0.7, 8, "cluster"),
    (2 * np.pi, 0.05, 20000, 2000, 0.7, 8, "lattice"),
    (4 * np.pi, 0.05, 20000, 30000, 0.7, 4, "uniform"),   # one leaf: the root
])
def test_fp64_matches_the_oracle(L, eps, n, leaf, mac, deg, kind):
    """To rounding (1e-12 of E) in a long box; in a short one a cluster term seen
    from a cell across the half period adds up to 24 (eps h)^2 / L^4 / 16^2 of a
    cluster's ninth, 2e-12 of the whole charge at L = 125 epsilon."""
    rng = np.random.default_rng(n + leaf)
    if kind == "uniform":
        x = rng.uniform(-1.5 * L, 1.5 * L, n)
    elif kind == "positive":
        x = rng.uniform(0, L, n)
    elif kind == "cluster":
        x = np.concatenate([rng.normal(0.3 * L, 0.002 * L, n // 2), rng.uniform(-L, L, n - n // 2)])
    else:
        x = rng.integers(-100, 100, n) / 100 * L + 1e-3 * rng.integers(0, 5, n)
    q = -np.abs(rng.normal(size=n)) * (L / n)
    e = M.E_MQ_Treecode_B200(L, eps, mac, deg, leaf, precision="fp64").evaluate(x, x, q)
    ref = O.treecode(L, eps, mac, deg, leaf, x, q)
    if L / eps > 1000:
        assert _rel(e, ref) < 1e-12
    assert np.max(np.abs(e - ref)) < 2e-12 * np.sum(np.abs(q))


def test_fp32c_takes_the_same_sums():
    """At 128 points per epsilon and more both precisions go through cells; they
    differ in how the moments' quotients are formed."""
    rng = np.random.default_rng(4)
    L, n = 2 * np.pi, 20000
    x = rng.uniform(-L, L, n)
    q = -np.abs(rng.normal(size=n)) * (L / n)
    e32 = M.E_MQ_Treecode_B200(L, 0.05, 0.7, 8, 500, precision="fp32c").evaluate(x, x, q)
    e64 = M.E_MQ_Treecode_B200(L, 0.05, 0.7, 8, 500, precision="fp64").evaluate(x, x, q)
    assert np.max(np.abs(e32 - e64)) < 1e-12 * np.sum(np.abs(q))
