"""Particles taken in cell order (grids from 126^3 on, no bonds, the Verlet
list) against the same instance on the cell-list path, whose spread has an
order of its own: the fixed-point sums do not depend on the order, the forces
agree to FP64 rounding.  Large steps, so that the list (and with it the order)
is rebuilt in between, and positions replaced from the host."""
import os

import numpy as np
import pytest

from helpers import rel_inf, uniform_positions

pytestmark = pytest.mark.gpu


def _make(fsl, verlet, q):
    old = os.environ.get("FLUAMSL_VERLET")
    os.environ["FLUAMSL_VERLET"] = verlet
    try:
        return fsl.StokesLimit(fsl.make_config((128,) * 3, (128.0,) * 3, eta=1.0, kT=0.5, dt=0.02, cutoff=1.5, kernel=3, pair=fsl.PAIR_SOFT,
                                               seed=2), q)
    finally:
        if old is None:
            del os.environ["FLUAMSL_VERLET"]
        else:
            os.environ["FLUAMSL_VERLET"] = old


def test_cell_order_equals_cell_list_path(fsl):
    L = (128.0,) * 3
    q = uniform_positions(20001, L, 3)
    a, b = _make(fsl, "1", q), _make(fsl, "0", q)
    for k in range(2):
        for g in (a, b):
            g.step(10)
            g.sync()
        assert rel_inf(a.positions() - q, b.positions() - q) < 1e-9
        q2 = uniform_positions(20001, L, 10 + k)
        for g in (a, b):
            g.set_positions(q2)
        q = q2
    a.close()
    b.close()


@pytest.mark.parametrize("n", [9472, 9473])  # one warp per particle up to here, quads from there on
def test_spread_before_any_list(fsl, n):
    """The spread on its own needs no list: before a step it gives the bits
    of the cell-list path's instance, and its own after one."""
    L = (128.0,) * 3
    q = uniform_positions(n, L, 5)
    F = np.random.default_rng(6).standard_normal(q.shape)
    a, b = _make(fsl, "1", q), _make(fsl, "0", q)
    want = b.spread(F)
    np.testing.assert_array_equal(a.spread(F), want)
    a.step(1)
    a.set_positions(q)
    np.testing.assert_array_equal(a.spread(F), want)
    a.close()
    b.close()
