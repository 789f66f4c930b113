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


def test_cell_order_equals_cell_list_path(fsl):
    m, L = (128, 128, 128), (128.0,) * 3
    q = uniform_positions(20001, L, 3)

    def make(verlet):
        old = os.environ.get("FLUAMSL_VERLET")
        os.environ["FLUAMSL_VERLET"] = verlet
        try:
            return fsl.StokesLimit(fsl.make_config(m, L, eta=1.0, kT=0.5, dt=0.02, cutoff=1.5, kernel=3, pair=fsl.PAIR_SOFT, seed=2), q)
        finally:
            if old is None:
                del os.environ["FLUAMSL_VERLET"]
            else:
                os.environ["FLUAMSL_VERLET"] = old

    a, b = make("1"), make("0")
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
