"""A server slot serves requests of every pair potential of its size class:
the one slot that the budget allows is used without a Verlet list (no pair
force), then with one, then for the Lennard-Jones table; every result equals
the same request run alone."""
import numpy as np
import pytest

from helpers import uniform_positions

pytestmark = pytest.mark.gpu


def test_slot_serves_every_pair_potential(fsl):
    m, L = (16, 16, 16), (16.0, 16.0, 16.0)
    q = uniform_positions(60, L, 3)
    pairs = (fsl.PAIR_NONE, fsl.PAIR_SOFT, fsl.PAIR_TABLE_LJ, fsl.PAIR_SOFT, fsl.PAIR_NONE)
    cfgs = [fsl.make_config(m, L, eta=1.0, kT=1e-4 if p == fsl.PAIR_TABLE_LJ else 0.01, dt=1e-3, cutoff=1.5, kernel=3, pair=p, seed=9)
            for p in pairs]
    srv = fsl.Server(hbm_budget=2 << 20)  # one slot of this class, not two
    for c in cfgs:
        rid = srv.submit(c, q, 3)
        info = srv.wait(rid, timeout=60)
        assert info["state"] == fsl._lib.REQ_DONE, info
        qs, Fs = srv.result(rid)
        g = fsl.StokesLimit(c, q)
        g.step(3)
        g.sync()
        np.testing.assert_array_equal(qs, g.positions())
        np.testing.assert_array_equal(Fs, g.forces())
        g.close()
    assert srv.stats()["slots"] == 1
    srv.close()
