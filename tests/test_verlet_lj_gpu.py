"""The Lennard-Jones table through the Verlet list (the default below 40
expected neighbours) against the cell-list kernel (FLUAMSL_VERLET=0) and the
FP64 oracle: forces of the same pairs to FP64 rounding, except where that
rounding moves a pair by one step of the table's 8-bit filter; and steps with
rebuilds, host position changes and a list that overflows."""
import os

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
