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


def test_slots_hold_a_list_only_where_it_is_used(fsl, monkeypatch):
    """A request without pair forces is admitted under the budget that its own
    buffers take, without 284 bytes a particle for a Verlet list; so is one
    with the Lennard-Jones table, whose forces then come from the cell list."""
    m, L, n = (16, 16, 16), (16.0, 16.0, 16.0), 7 ** 3
    q = (np.stack(np.meshgrid(*[np.arange(7)] * 3)).reshape(3, -1) + 0.5) * (16.0 / 7) - 8.0
    cfg = {p: fsl.make_config(m, L, eta=1.0, kT=1e-4, dt=1e-3, cutoff=2.5, kernel=3, pair=p, seed=9)
           for p in (fsl.PAIR_NONE, fsl.PAIR_SOFT, fsl.PAIR_TABLE_LJ)}

    def serve(pair, **kw):
        with fsl.Server(**kw) as srv:
            rid = srv.submit(cfg[pair], q, 3)
            info = srv.wait(rid, timeout=60)
            done = info["state"] == fsl._lib.REQ_DONE
            return info, srv.stats()["bytes_held"], srv.result(rid) if done else None

    none, soft = (serve(p)[1] for p in (fsl.PAIR_NONE, fsl.PAIR_SOFT))
    assert none + 284 * n <= soft
    assert serve(fsl.PAIR_NONE, hbm_budget=none)[2] is not None
    assert serve(fsl.PAIR_SOFT, hbm_budget=none)[2] is None
    got = serve(fsl.PAIR_TABLE_LJ, hbm_budget=none)[2]
    monkeypatch.setenv("FLUAMSL_VERLET", "0")
    with fsl.StokesLimit(cfg[fsl.PAIR_TABLE_LJ], q) as g:
        g.step(3)
        g.sync()
        np.testing.assert_array_equal(got[0], g.positions())
        np.testing.assert_array_equal(got[1], g.forces())
