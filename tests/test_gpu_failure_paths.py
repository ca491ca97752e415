"""Failure paths driven without a GPU fault: the bounds of the device waits are
lowered through the test hook fs_debug_set_wait_limits so that a bounded wait
runs out, the call returns its error status, and the next call on the same
object works.  Nothing traps and no wait is unbounded: with zero polls every
tile wait gives up at once, and the kernel still lets its own copies land
(bounded) before its CTAs exit."""
import numpy as np
import pytest

import oracle as O
import multi_species_b200 as M
from multi_species_b200 import decks

pytestmark = pytest.mark.gpu

FS_ERR_WALK, FS_ERR_TIMEOUT = 4, 6
FS_ERR_TREE = 9


@pytest.fixture(autouse=True)
def _default_limits():
    yield
    M.debug_set_wait_limits(0)


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def test_pair_kernel_wait_timeout_then_recovers():
    rng = np.random.default_rng(3)
    L = 4 * np.pi
    x = rng.uniform(-L, 2 * L, 20000)
    q = rng.normal(size=20000) * 1e-3
    f = M.E_MQ_DirectSum_B200(L, 0.05, "fp32c")
    ref = O.direct_sum(L, 0.05, x, x, q)
    assert rel(f.evaluate(x, x, q), ref) < 1e-6
    M.debug_set_wait_limits(0, mbar_polls=0)
    with pytest.raises(M.FsError) as e:
        f.evaluate(x, x, q)
    assert e.value.code == FS_ERR_TIMEOUT
    M.debug_set_wait_limits(0)
    for _ in range(2):
        assert rel(f.evaluate(x, x, q), ref) < 1e-6
    f.close()


def test_session_fp32c_timeout_is_reported():
    """A session step whose field wait runs out returns FS_ERR_TIMEOUT; a new
    session on the same device then steps normally."""
    d = decks.two_stream(h=4, ph=1, steps=4, remesh_period=5)
    g = M.Simulation(d, "direct32c")
    M.debug_set_wait_limits(0, mbar_polls=0)
    with pytest.raises(M.FsError) as e:
        g.step(1)
    assert e.value.code == FS_ERR_TIMEOUT
    M.debug_set_wait_limits(0)
    g.close()
    a, b = M.Simulation(d, "direct32c"), M.Simulation(d, "direct64")
    a.step(2)
    b.step(2)
    assert rel(a.state()["es"], b.state()["es"]) < 1e-6


def test_remesh_walk_limit_then_recovers():
    """The step that remeshes fails with FS_ERR_WALK when walks may visit only
    one panel; the state is left as the step's RK4 made it, and a remesh with
    the default bound on the same session gives the state of an undisturbed
    session bit for bit."""
    d = decks.two_stream(h=4, ph=1, steps=10, remesh_period=5)
    g, ref = M.Simulation(d, "direct64"), M.Simulation(d, "direct64")
    g.step(4)
    ref.step(5)
    M.debug_set_wait_limits(0, walk_panels=1)
    with pytest.raises(M.FsError) as e:
        g.step(1)
    assert e.value.code == FS_ERR_WALK
    st = g.state()
    assert not np.array_equal(st["xs"], ref.state()["xs"])  # not remeshed: still the moved points
    M.debug_set_wait_limits(0)
    g.remesh()
    a, b = g.state(), ref.state()
    for k in ("xs", "ps", "fs", "q_ws", "es"):
        assert np.array_equal(a[k], b[k]), k
    g.step(2)
    ref.step(2)
    for k in ("xs", "ps", "fs", "q_ws", "es"):
        assert np.array_equal(g.state()[k], ref.state()[k]), k


def test_failed_remesh_leaves_the_last_steps_field():
    """The same in an FP32c session whose stage fields go through cells, the failing
    step the last of five in one call: E is the fourth step's, to the FP32c sum's
    error, and the next step starts from it."""
    d = decks.two_stream(h=6, ph=1, steps=10, remesh_period=5)
    g, ref = M.Simulation(d, "direct32c"), M.Simulation(d, "direct64")
    before = M.Simulation(d, "direct64")
    before.step(4)
    M.debug_set_wait_limits(0, walk_panels=1)
    for s in (g, ref):
        with pytest.raises(M.FsError) as e:
            s.step(5)
        assert e.value.code == FS_ERR_WALK
    M.debug_set_wait_limits(0)
    assert np.array_equal(ref.state()["es"], before.state()["es"])
    assert rel(g.state()["es"], ref.state()["es"]) < 1e-8
    g.step(1)
    ref.step(1)
    for k in ("xs", "ps"):
        assert rel(g.state()[k], ref.state()[k]) < 1e-8, k


@pytest.mark.parametrize("h", [6, 8])
def test_a_step_without_a_tree_leaves_the_points(h):
    """More coincident points than a leaf may hold: the tree cannot be split, the
    step fails and the positions and velocities stay as they were (at h = 8,
    1,577,475 points, the stage epilogue is a launch of its own)."""
    d = decks.bump_on_tail(h=h)
    g = M.Simulation(d, "treecode32c")
    st = g.state()
    x, p = st["xs"].copy(), st["ps"].copy()
    x[:5000], p[:5000] = 1.0, 0.0       # coincident at the second stage
    g.import_xp(xs=x, ps=p)
    with pytest.raises(M.FsError) as e:
        g.step(1)
    assert e.value.code == FS_ERR_TREE
    after = g.state()
    assert np.array_equal(after["xs"], x) and np.array_equal(after["ps"], p)
    g.import_xp(xs=st["xs"], ps=st["ps"])
    g.step(1)
    assert np.all(np.isfinite(g.state()["xs"]))


@pytest.mark.parametrize("n", [90_000, 200_000])
def test_cell_wait_timeout_then_recovers(n):
    """The bounded waits of the sums between cells (n L / epsilon above 2e7)."""
    rng = np.random.default_rng(n)
    L = 4 * np.pi
    x = rng.uniform(-L, 2 * L, n)
    q = rng.normal(size=n) / n
    f = M.E_MQ_DirectSum_B200(L, 0.05, "fp32c")
    ref = f.evaluate(x, x, q)
    M.debug_set_wait_limits(0, mbar_polls=0)
    with pytest.raises(M.FsError) as e:
        f.evaluate(x, x, q)
    assert e.value.code == FS_ERR_TIMEOUT
    M.debug_set_wait_limits(0)
    for _ in range(2):
        assert np.array_equal(f.evaluate(x, x, q), ref)
    f.close()


@pytest.mark.parametrize("steps", [1, 3])
def test_large_session_timeout_is_reported(steps):
    """A session of 66,049 points: stage fields through cells, the field handed out
    from windows of pairs.  The failed call is reported, the state can still be
    read, and given back what it was the session steps as an undisturbed one."""
    d = decks.two_stream(h=7, ph=0, remesh_period=100)
    g, ref = M.Simulation(d, "direct32c"), M.Simulation(d, "direct32c")
    st = g.state()
    M.debug_set_wait_limits(0, mbar_polls=0)
    with pytest.raises(M.FsError) as e:
        g.step(steps)
    assert e.value.code == FS_ERR_TIMEOUT
    g.state()
    M.debug_set_wait_limits(0)
    g.import_xp(st["xs"], st["ps"], st["es"])
    g.step(2)
    ref.step(2)
    a, b = g.state(), ref.state()
    for k in ("xs", "ps", "fs", "q_ws", "es"):
        assert np.array_equal(a[k], b[k]), k
