"""Edges of the kernels' shortened arithmetic, bit for bit against the oracle
or IEEE arithmetic (imex_gpu_point_eval): inputs on both sides of each range
that decides between a short path and the general one."""
import numpy as np
import pytest

from imex_sflow2d_v2_b200.solver import point_eval
from oracle import ipow_n

pytestmark = pytest.mark.gpu


def _around(values, steps=200):
    """Each value with its `steps` nearest doubles on either side."""
    v = np.abs(np.asarray(values, np.float64)).view(np.int64)
    return (v[:, None] + np.arange(-steps, steps + 1)[None, :]).ravel().view(np.float64)


@pytest.mark.parametrize("y", [0.5, 0.687, 1.5, 2.4, 4.65, 5.0, np.nextafter(5.0, 6.0), 1e-300])
def test_ipow_common_range_edges(y):
    rng = np.random.default_rng(3)
    # the ends of the common range, the window around 1 that it leaves out,
    # every table row's ends in the binades beside 1 and at the far ones
    edges = [2.0 ** -200, 2.0 ** 200, 1.0 - 2.0 ** -8, 1.0 + 2.0 ** -7, 1.0]
    rows = (1.0 + np.arange(129) / 128.0)[:, None] * 2.0 ** np.array([-199, -30, -2, -1, 0, 1, 9, 198])
    x = np.concatenate([_around(edges), _around(rows.ravel(), 3),
                        np.exp(rng.uniform(np.log(1e-60), np.log(1e60), 200000))])
    g, o = point_eval("ipow", x, np.full(x.size, y)), ipow_n(x, np.full(x.size, y))
    bad = np.flatnonzero(g.view(np.uint64) != o.view(np.uint64))
    assert bad.size == 0, [(x[i], y, g[i], o[i]) for i in bad[:5]]
