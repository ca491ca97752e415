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


@pytest.mark.parametrize("n,kind,precision", [
    (1, "spread", "fp64"), (2, "crowd", "fp32c"), (3000, "pairs", "fp64"), (20000, "crowd", "fp64"),
    (20000, "crowd", "fp32c"), (60000, "crowds", "fp64"), (60000, "crowds", "fp32c"),
    (1 << 18, "spread", "fp64"), ((1 << 18) + 1, "crowd", "fp64"), (400_000, "crowds", "fp32c")])
def test_the_points_order_does_not_matter(n, kind, precision):
    """Points with distinct positions are summed in the order of x, however close
    together they are and however they come: the same bits in every order."""
    rng = np.random.default_rng(n)
    L = 4 * np.pi
    if kind == "spread":
        x = rng.uniform(-L, L, n)
    elif kind == "pairs":     # neighbours 1e-13 apart
        c = rng.uniform(0, L, n // 2)
        x = np.r_[c, c + 1e-13]
    elif kind == "crowd":     # 1,500 within 1e-10
        x = rng.uniform(-L, L, n)
        m = min(n, 1500)
        x[:m] = 1.7 + 1e-10 * np.arange(m) / m
    else:                     # groups of 2 .. 70 within 1e-11
        x, k = np.empty(0), 2
        while len(x) < n:
            x = np.r_[x, rng.uniform(-0.9 * L, 0.9 * L) + 1e-11 * np.arange(k) / k]
            if len(x) > 5000:
                x = np.r_[x, rng.uniform(-L, L, n)]
            k = 2 + (k + 31) % 69
        x = x[:n]
    x = np.unique(x)
    q = rng.normal(size=len(x)) / n
    eng = M.E_MQ_Treecode_B200(L, 0.05, 0.7, 8, 2000, precision=precision)
    e = eng.evaluate(x, x, q)
    for order in (rng.permutation(len(x)), np.arange(len(x))[::-1]):
        assert np.array_equal(eng.evaluate(x[order], x[order], q[order]), e[order])
    if len(x) <= 60000:
        ref = O.treecode(L, 0.05, 0.7, 8, 2000, x, q)
        assert np.max(np.abs(e - ref)) < (2e-12 if precision == "fp64" else 1e-8) * np.sum(np.abs(q))


@pytest.mark.parametrize("where", ["position", "charge"])
@pytest.mark.parametrize("n", [1500, 1900])
def test_nan_reaches_every_target(n, where):
    """One leaf (n < 2000) through cells, its points in the upper half of the box."""
    L = 4 * np.pi
    x = np.linspace(0.5 * L, 0.9 * L, n)
    q = np.full(n, -L / n)
    (x if where == "position" else q)[n // 3] = np.nan
    e = M.E_MQ_Treecode_B200(L, 0.2, 0.7, 8, 2000, precision="fp64").evaluate(x, x, q)
    assert np.all(np.isnan(e))


def test_a_large_sessions_step_is_the_fields_rk4():
    """1,577,475 points: the stage epilogue runs apart from the field.  One step
    against RK4 on the host through the same treecode, to rounding."""
    from multi_species_b200 import decks
    d = decks.bump_on_tail(h=8)
    d["remesh_period"] = 100
    s = M.Simulation(d, "treecode32c")
    st = s.state()
    n, dt, L = s.n, d["dt"], d["xmax"]
    x, p, q = st["xs"], st["ps"], st["q_ws"]
    qm = np.repeat([sp["q"] / sp["m"] for sp in d["species_list"]], n // 3)
    f = M.E_MQ_Treecode_B200(L, d["greens_epsilon"], d["mac"], d["degree"], d["max_source"], precision="fp32c")
    a1 = qm * st["es"]
    p2 = p + 0.5 * dt * a1
    x2 = x + 0.5 * dt * p
    a2 = qm * f.evaluate(x2, x2, q)
    p3 = p + 0.5 * dt * a2
    x3 = x + 0.5 * dt * p2
    a3 = qm * f.evaluate(x3, x3, q)
    p4 = p + dt * a3
    x4 = x + dt * p3
    a4 = qm * f.evaluate(x4, x4, q)
    s.step(1)
    out = s.state()
    assert _rel(out["xs"], x + dt / 6 * (p + 2 * p2 + 2 * p3 + p4)) < 1e-14
    assert _rel(out["ps"], p + dt / 6 * (a1 + 2 * a2 + 2 * a3 + a4)) < 1e-14


@pytest.mark.parametrize("n", [1, 5, 129, 2001, 23_999, 24_000, 24_003])
def test_fp64_pair_by_pair(n):
    """Below 16 points per epsilon: targets shared by a warp or by eight lanes, to
    rounding (as above)."""
    rng = np.random.default_rng(n)
    L = 20 * np.pi
    x = rng.uniform(-L, L, n)
    m = min(n // 8, 900)                        # fewer coincident points than a leaf holds
    x[:m] = x[0]
    x[m: 2 * m] = np.mod(x[0], L) - L / 2       # half a period apart
    q = rng.normal(size=n) / n
    e = M.E_MQ_Treecode_B200(L, 0.02, 0.7, 8, 2000, precision="fp64").evaluate(x, x, q)
    assert np.max(np.abs(e - O.treecode(L, 0.02, 0.7, 8, 2000, x, q))) < 2e-12 * np.sum(np.abs(q))


def test_fp64_pair_by_pair_with_a_vanishing_epsilon():
    """epsilon^2 underflows: a point's own pair still adds nothing."""
    x = np.linspace(0.0, 1.0, 300, endpoint=False)
    q = np.full(300, -1.0 / 300)
    e = M.E_MQ_Treecode_B200(1.0, 1e-200, 0.7, 8, 2000, precision="fp64").evaluate(x, x, q)
    assert np.max(np.abs(e - O.treecode(1.0, 1e-200, 0.7, 8, 2000, x, q))) < 2e-12


@pytest.mark.parametrize("where", ["inside", "last", "first"])
def test_subnormal_positions_left_of_0(where):
    """x / L underflows to -0 there: a leaf's cells still rise with x, and such a
    point has its neighbours' cell.  Bound as above."""
    rng = np.random.default_rng(7)
    L, n = 4 * np.pi, 12000
    tiny = -5e-324 * np.arange(1, 6)
    if where == "inside":
        rest = rng.uniform(-0.9 * L, 0.9 * L, n)
    elif where == "last":       # the tree's last points
        rest = rng.uniform(-0.9 * L, -1e-3, n)
    else:                       # a leaf begins with them
        rest = np.r_[rng.uniform(-0.9 * L, -0.4 * L, n // 2), rng.uniform(0.3 * L, 0.9 * L, n - n // 2)]
    x = np.r_[rest, tiny]
    q = rng.normal(size=len(x)) / n
    q[n:] = 1.0
    e = M.E_MQ_Treecode_B200(L, L / 700, 0.7, 8, 2000, precision="fp64").evaluate(x, x, q)
    ref = O.treecode(L, L / 700, 0.7, 8, 2000, x, q)
    assert np.max(np.abs(e - ref)) < 2e-12 * np.sum(np.abs(q))


@pytest.mark.parametrize("ratio", [33.0, 64.0, 100.0, 251.3, 500.0, 639.0, 641.0])
@pytest.mark.parametrize("parts", [8, 3, 0])
def test_fp64_charges_half_a_period_apart(ratio, parts):
    """All charge in two places half a period apart, where the kernel's second
    derivative jumps, with several leaves and with one.  Bound: n additions of
    terms of at most |q| / 2 on either side."""
    L, n = 4 * np.pi, int(20 * ratio)
    rng = np.random.default_rng(n + parts)
    x = 0.1 * L + rng.uniform(0, L / 512, n) + 0.5 * L * (np.arange(n) % 2)
    q = -rng.uniform(0.5, 1.5, n) * L / n
    leaf = n // parts if parts else 2 * n
    e = M.E_MQ_Treecode_B200(L, L / ratio, 0.7, 8, leaf, precision="fp64").evaluate(x, x, q)
    ref = O.treecode(L, L / ratio, 0.7, 8, leaf, x, q)
    assert np.max(np.abs(e - ref)) <= n * 2.0 ** -53 * np.sum(np.abs(q))


@pytest.mark.parametrize("h,ph,backend", [(6, 1, "treecode64"), (8, 0, "treecode32c")])
def test_a_session_sums_each_field_once(h, ph, backend):
    """Two steps in one call launch what two calls of one step launch."""
    from multi_species_b200 import decks
    d = decks.bump_on_tail(h=h, ph=ph)
    d["remesh_period"] = 100
    s = M.Simulation(d, backend)
    s.step(1)
    n = [M.kernel_launches()]
    for k in (1, 2):
        s.step(k)
        n.append(M.kernel_launches())
    assert n[2] - n[1] == 2 * (n[1] - n[0])
