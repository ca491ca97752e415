"""FP64 direct sum: bit-identical to the oracle at the edges of its tiles and
rounds, for periods its division handles as a product and one it does not, and
for values that take the IEEE operations."""
import numpy as np
import pytest

import oracle as O
import multi_species_b200 as M

pytestmark = pytest.mark.gpu

# a period one of whose quotients the two-part product rounds wrongly
ODD_L = float.fromhex("0x1.f6dd22369359bp+0")


@pytest.mark.parametrize("L", [4 * np.pi, 2.0, ODD_L])
@pytest.mark.parametrize("ns,nt", [(1, 1), (7, 33), (64, 31), (65, 32), (127, 0), (129, 0), (511, 5), (513, 0),
                                   (1025, 64), (65, 9472), (513, 9473)])
def test_sizes(L, ns, nt):
    rng = np.random.default_rng(ns + nt)
    s = rng.uniform(-L, 2 * L, ns)
    s[rng.random(ns) < 0.2] = 0.25 * L              # coincident sources
    t = rng.uniform(-L, 2 * L, nt) if nt else s
    if nt:
        t[rng.random(nt) < 0.2] = 0.75 * L          # half a period from them
    q = rng.normal(size=ns) * 1e-3
    e = M.E_MQ_DirectSum_B200(L, 0.02, "fp64").evaluate(t, s, q)
    assert np.array_equal(e, O.direct_sum(L, 0.02, t, s, q))


@pytest.mark.parametrize("case", ["tiny", "subnormal", "huge charge", "infinite charge", "nan charge", "far", "nan point",
                                  "small eps", "small box"])
def test_values_outside_the_products_range(case):
    rng = np.random.default_rng(5)
    L, eps, n = 4 * np.pi, 0.05, 700
    x = rng.uniform(0, L, n)
    q = rng.normal(size=n)
    if case == "tiny":
        x[::3] = rng.uniform(-1, 1, len(x[::3])) * 1e-290
    elif case == "subnormal":
        x[:] = rng.integers(-9, 9, n) * 5e-324
    elif case == "huge charge":
        q[5], q[600] = 1e300, -1e300
    elif case == "infinite charge":
        q[600], x[600] = np.inf, x[0] + 0.5 * L
    elif case == "nan charge":
        q[3] = np.nan
    elif case == "far":
        x = x * 1e18
    elif case == "nan point":
        x[9] = np.nan
    elif case == "small eps":
        eps = 1e-70
    else:
        L, eps = 1e-70, 1e-72
        x = x * 1e-70
    e = M.E_MQ_DirectSum_B200(L, eps, "fp64").evaluate(x, x, q)
    assert np.array_equal(e, O.direct_sum(L, eps, x, x, q), equal_nan=True)
