"""The FP32-compensated direct sum of few points (at most 16,384 targets and
sources, four launches) at the edges of its warps, tiles and sort blocks, against
the oracle's FP64 pairwise sum."""
import numpy as np
import pytest

import oracle as O
import multi_species_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nt", [
    (1, 0), (2, 1), (31, 0), (32, 33), (33, 0), (255, 257), (256, 0), (257, 1), (2047, 0), (2048, 31), (2049, 0),
    (4095, 0), (4096, 4097), (4097, 0), (8192, 5), (1, 16384), (16383, 0), (16384, 16384), (16384, 16385),
    (16385, 100)])
@pytest.mark.parametrize("ratio", [20.0, 251.3])
def test_few_points_match_the_fp64_sum(ns, nt, ratio):
    """The pairwise FP32c kernels' 1e-9 of the band charge, doubled; n L / epsilon
    is below 2e7 throughout, so nothing goes through cells."""
    rng = np.random.default_rng(ns + 7 * nt)
    L = 4 * np.pi
    eps = L / ratio
    s = rng.uniform(-L, 2 * L, ns)
    s[: ns // 4] = s[0]             # coincident points
    q = rng.normal(size=ns) / ns
    t = rng.uniform(-L, 2 * L, nt) if nt else s
    e = M.E_MQ_DirectSum_B200(L, eps, "fp32c").evaluate(t, s, q)
    assert np.max(np.abs(e - O.direct_sum(L, eps, t, s, q))) <= 2e-9 * np.sum(np.abs(q))
