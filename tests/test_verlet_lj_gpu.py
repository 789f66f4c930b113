"""The Lennard-Jones table through the Verlet list (the default below 40
expected neighbours) against the cell-list kernel (FLUAMSL_VERLET=0) and the
FP64 oracle: forces of the same pairs to FP64 rounding, except where that
rounding moves a pair by one step of the table's 8-bit filter; and steps with
rebuilds, host position changes and a list that overflows."""
import os
import time

import numpy as np
import pytest

from helpers import rel_inf

pytestmark = pytest.mark.gpu


def lattice(n, L, seed, jitter=0.2):
    rng = np.random.default_rng(seed)
    per = int(L // 3)
    sites = rng.permutation(per ** 3)[:n]
    s = np.stack([sites % per, sites // per % per, sites // per ** 2])
    return (s + 0.5) * (L / per) - 0.5 * L + rng.uniform(-jitter, jitter, s.shape)


def make(fsl, m, q, verlet=None, **kw):
    args = dict(eta=1.0, kT=0.02, dt=0.01, cutoff=5.0, kernel=3, pair=fsl.PAIR_TABLE_LJ, seed=4)
    args.update(kw)
    old = os.environ.get("FLUAMSL_VERLET")
    if verlet is not None:
        os.environ["FLUAMSL_VERLET"] = verlet
    try:
        return fsl.StokesLimit(fsl.make_config((m,) * 3, (float(m),) * 3, **args), q)
    finally:
        if verlet is not None:
            if old is None:
                del os.environ["FLUAMSL_VERLET"]
            else:
                os.environ["FLUAMSL_VERLET"] = old


@pytest.mark.parametrize("n", [1, 2, 65, 700])
@pytest.mark.parametrize("scheme", ["SCHEME_MIDPOINT", "SCHEME_FIRST_ORDER"])
def test_steps_against_cell_list_and_oracle(fsl, oracle, n, scheme):
    m = 30
    q = lattice(n, m, n)
    a = make(fsl, m, q, scheme=getattr(fsl, scheme))
    b = make(fsl, m, q, verlet="0", scheme=getattr(fsl, scheme))
    o = oracle.Oracle(m, m, m, m, m, m, q, eta=1.0, kT=0.02, dt=0.01, cutoff=5.0, kernel=3, pair=oracle.PAIR_TABLE_LJ, seed=4,
                      scheme=getattr(oracle, scheme))
    Fa, Fb = a.compute_forces(), b.compute_forces()
    # a pair within FP64 rounding of a filter step changes by 2^-8 of a table
    # interval (2e-6 of the force seen)
    assert rel_inf(Fa, Fb) < 1e-5
    for _ in range(3):
        for x in (a, b, o):
            x.step(1)
    for x in (a, b):
        x.sync()
        assert rel_inf(x.positions() - q, o.positions() - q) < 1e-5
    a.close()
    b.close()


def test_rebuilds_and_host_moves(fsl):
    """Large steps (a rebuild every few) and positions replaced from the host."""
    m, q = 24, lattice(400, 24, 7)
    a, b = make(fsl, m, q, kT=0.3, dt=0.02), make(fsl, m, q, verlet="0", kT=0.3, dt=0.02)
    for k in range(4):
        for x in (a, b):
            x.step(10)
            x.sync()
        assert rel_inf(a.compute_forces(), b.compute_forces()) < 1e-4, k
        q = lattice(400, 24, 100 + k)
        for x in (a, b):
            x.set_positions(q)
        assert rel_inf(a.compute_forces(), b.compute_forces()) < 1e-5, k
    a.close()
    b.close()


def test_overflow(fsl):
    """A cluster with more than 64 neighbours a particle: the list gives way to
    the cells of each evaluation."""
    m = 24
    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(6)] * 3)).reshape(3, -1) * 2.2 - 5.5
    q = g + rng.uniform(-0.05, 0.05, g.shape)
    a, b = make(fsl, m, q, dt=1e-3, cutoff=5.5), make(fsl, m, q, verlet="0", dt=1e-3, cutoff=5.5)
    for _ in range(2):
        assert rel_inf(a.compute_forces(), b.compute_forces()) < 1e-5
        for x in (a, b):
            x.step(3)
            x.sync()
    assert rel_inf(a.positions() - q, b.positions() - q) < 1e-5
    a.close()
    b.close()


def test_fast_particles_take_the_cells(fsl):
    """Particles that outrun the list at every evaluation: the forces come
    from the cell list, at its speed and with its values."""
    m, q = 64, lattice(9261, 64, 9)
    a, b = make(fsl, m, q, kT=1.0, dt=0.1), make(fsl, m, q, verlet="0", kT=1.0, dt=0.1)
    us = []
    for x in (a, b):
        x.step(20)
        x.sync()
        t = []
        for _ in range(3):
            t0 = time.perf_counter()
            x.step(40)
            x.sync()
            t.append(time.perf_counter() - t0)
        us.append(min(t) / 40 * 1e6)
    # a build at every evaluation took eight times the cell list's step
    assert us[0] < 1.5 * us[1], us
    for _ in range(3):
        q = a.positions()
        b.set_positions(q)
        b.set_step(a.status()["step"])
        for x in (a, b):
            x.step(1)
            x.sync()
        assert rel_inf(a.positions() - q, b.positions() - q) < 1e-5
    a.close()
    b.close()


def test_list_tried_again(fsl):
    """Past the steps after which the list is tried again: an instance alone
    and in a batch beside slow and soft ones, bit for bit, and the values of
    the cell list on the way."""
    m = 24
    args = dict(eta=1.0, cutoff=5.0, kernel=3, seed=4)
    cfg = [fsl.make_config((m,) * 3, (24.0,) * 3, kT=kT, dt=dt, pair=p, **args)
           for kT, dt, p in [(0.5, 0.05, fsl.PAIR_TABLE_LJ), (0.01, 0.01, fsl.PAIR_TABLE_LJ), (0.5, 0.05, fsl.PAIR_SOFT)]]
    qs = [lattice(400, m, 20 + i) for i in range(3)]
    batch = fsl.Batch(cfg, qs)
    alone = [fsl.StokesLimit(c, q) for c, q in zip(cfg, qs)]
    b = make(fsl, m, qs[0], verlet="0", kT=0.5, dt=0.05)
    for n in (5, 251, 1, 1, 1, 6, 255, 30):
        batch.step(n)
        batch.sync()
        for i, a in enumerate(alone):
            a.step(n)
            a.sync()
            np.testing.assert_array_equal(batch.positions(i), a.positions(), err_msg=f"{n} {i}")
        # the fast instance's next step against the cell list's
        q = alone[0].positions()
        b.set_positions(q)
        b.set_step(alone[0].status()["step"])
        for x in (alone[0], b, batch):
            x.step(1)
            x.sync()
        for a in alone[1:]:
            a.step(1)
        assert rel_inf(alone[0].positions() - q, b.positions() - q) < 1e-5, n
    for x in alone + [b, batch]:
        x.close()
