"""The FP32-compensated direct sum through cell expansions (L between 32 and
5120 epsilon) against the oracle's FP64 pairwise sum, and the sessions whose
stage fields go through it."""
import numpy as np
import pytest

import oracle as O
import multi_species_b200 as M
from multi_species_b200 import decks

pytestmark = pytest.mark.gpu


def _points(kind, n, L, rng):
    if kind == "cell":      # all in one cell, away from its middle
        return rng.uniform(0.2, 0.21, n) * 0.6 * L / 5120
    if kind == "cluster":   # half in a few cells, the rest over several periods
        return np.concatenate([rng.normal(L / 3, 0.003 * L, n // 2), rng.uniform(-2 * L, 3 * L, n - n // 2)])
    if kind == "lattice":   # coincident points, half-period partners, cell edges
        return (rng.integers(0, 64, n) / 64 + rng.integers(-2, 3, n)) * L
    return rng.uniform(-L, 2 * L, n)


@pytest.mark.parametrize("ratio,n,nt,kind", [
    (32.5, 620_000, 200, "uniform"), (63.0, 320_001, 300, "lattice"), (251.3, 80_015, 301, "uniform"),
    (251.3, 80_016, 1, "cell"), (251.3, 80_017, 300, "cluster"), (1570.8, 12_801, 0, "uniform"),
    (1570.8, 13_056, 513, "lattice"), (1570.8, 20_000, 0, "cell"), (5119.0, 3_920, 0, "cluster"),
    (5119.0, 5_000, 33, "uniform"),
    # just outside on either side and just too few points: the pairwise kernel
    (32.0, 630_000, 20, "uniform"), (5121.0, 5_000, 0, "uniform"), (251.3, 70_000, 100, "cluster"), (1570.8, 2, 7, "uniform")])
def test_cells_match_the_fp64_sum(ratio, n, nt, kind):
    """16 Chebyshev terms on cells of epsilon / 1.6 leave (6.5)^-16 = 1e-13 of a
    pair's charge; below L = 64 epsilon the cell pair across the half period adds
    up to 0.06 (epsilon / L)^2 / 256^3 = 4e-12 of the charge.  The pairwise kernel
    is held to its own 1e-9 of the band charge."""
    rng = np.random.default_rng(n + int(ratio))
    L = 4 * np.pi
    eps = L / ratio
    s = _points(kind, n, L, rng)
    q = rng.normal(size=n) / n
    t = _points(kind, nt, L, rng) if nt else s
    e = M.E_MQ_DirectSum_B200(L, eps, "fp32c").evaluate(t, s, q)
    ref = O.direct_sum(L, eps, t, s, q)
    cells = 32 < ratio <= 5120 and n * ratio >= 2e7
    tol = 2e-9 if not cells else (1e-11 if ratio < 64 else 1e-12)
    assert np.max(np.abs(e - ref)) <= tol * np.sum(np.abs(q))


def test_nan_charge_reaches_every_target():
    L = 4 * np.pi
    for n in (100, 90_000):
        x = np.linspace(0, L, n, endpoint=False)
        q = np.full(n, 0.1)
        q[17] = np.nan
        assert np.all(np.isnan(M.E_MQ_DirectSum_B200(L, 0.05, "fp32c").evaluate(x[:100] + 0.01, x, q)))


def test_session_is_the_same_however_its_steps_are_called():
    """Stage fields through cells, E handed out summed pairwise after a call's
    last step: four steps in one call and one by one agree bit for bit, with
    and without a remesh among them."""
    for h, period in ((4, 3), (6, 3), (6, 100)):
        d = decks.two_stream(h=h, ph=1, remesh_period=period)
        a, b = M.Simulation(d, "direct32c"), M.Simulation(d, "direct32c")
        a.step(4)
        for _ in range(4):
            b.step(1)
            b.state()
        sa, sb = a.state(), b.state()
        for k in ("xs", "ps", "fs", "q_ws", "es"):
            assert np.array_equal(sa[k], sb[k]), (h, period, k)


def test_imported_field_is_the_next_steps_first():
    d = decks.two_stream(h=6, ph=0, remesh_period=100)
    a, b = M.Simulation(d, "direct32c"), M.Simulation(d, "direct64")
    es = np.sin(0.2 * a.state()["xs"])
    for s in (a, b):
        s.step(2)
        s.import_xp(es=es)
        assert np.array_equal(s.state()["es"], es)
        s.step(1)
    sa, sb = a.state(), b.state()
    for k in ("xs", "ps"):
        assert np.linalg.norm(sa[k] - sb[k]) <= 1e-8 * np.linalg.norm(sb[k]), k


@pytest.mark.parametrize("ratio,kind", [
    (600.0, "uniform"), (1570.8, "uniform"), (1570.8, "cell"), (1570.8, "cluster"), (1570.8, "lattice"),
    (5119.0, "uniform"), (640.0, "uniform"), (640.0, "cluster"), (2500.0, "ends")])
def test_exported_field_of_a_large_session(ratio, kind):
    """E handed out of a session of 66,049 points (pairs within a window of cells,
    the rest through cells; at 600 epsilon, and where a block of targets spans
    more than two groups, all pairs): the pairwise kernel's 1e-9 of the band
    charge, as above."""
    rng = np.random.default_rng(int(ratio))
    d = decks.two_stream(h=7, ph=0, remesh_period=100)
    L = d["xmax"]
    d.update(greens_epsilon=L / ratio, dt=1e-3)
    s = M.Simulation(d, "direct32c")
    n = s.n
    x = L * (1 - rng.beta(0.1, 0.1, n)) if kind == "ends" else _points(kind, n, L, rng)
    s.import_xp(xs=x, ps=np.zeros(n))
    s.step(1)
    st = s.state()
    t = np.argsort(np.mod(st["xs"], L))[np.unique(np.r_[0, n - 1, rng.integers(0, n, 300)])]
    ref = O.direct_sum(L, L / ratio, st["xs"][t], st["xs"], st["q_ws"])
    assert np.max(np.abs(st["es"][t] - ref)) <= 2e-9 * np.sum(np.abs(st["q_ws"]))


@pytest.mark.parametrize("h,ph,backend", [(6, 1, "direct32c"), (7, 0, "direct32c"), (3, 1, "direct32c"),
                                          (5, 0, "direct64"), (6, 1, "treecode32c"), (7, 1, "treecode32c")])
def test_an_exported_state_goes_on_bit_for_bit(h, ph, backend):
    """Positions, velocities and field of a session imported into a fresh one, and
    into itself, continue as the undisturbed session does."""
    deck = decks.bump_on_tail if backend.startswith("tree") else decks.two_stream
    d = deck(h=h, ph=ph)
    d["remesh_period"] = 100
    a, b, c = (M.Simulation(d, backend) for _ in range(3))
    for s in (a, b):
        s.step(3)
    st = b.state()
    for s in (b, c):
        s.import_xp(st["xs"], st["ps"], st["es"])
    for _ in range(2):
        for s in (a, b, c):
            s.step(2)
        sa = a.state()
        for s in (b, c):
            got = s.state()
            for k in ("xs", "ps", "es"):
                assert np.array_equal(got[k], sa[k]), k


def test_a_remeshed_state_imported_goes_on_bit_for_bit():
    d = decks.two_stream(h=6, ph=1, remesh_period=3)
    a, b = M.Simulation(d, "direct32c"), M.Simulation(d, "direct32c")
    for s in (a, b):
        s.step(3)
    st = b.state()
    b.import_xp(st["xs"], st["ps"], st["es"])
    for s in (a, b):
        s.step(4)
    sa, sb = a.state(), b.state()
    for k in ("xs", "ps", "fs", "q_ws", "es"):
        assert np.array_equal(sa[k], sb[k]), k
