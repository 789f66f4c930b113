"""The spread and the interpolation of launches with few particles (one warp
per particle) give the bits of the quad kernels: instances alone take the
former, a batch of enough of them the latter.  Particle counts around the
blocks of both (8 and 64 particles), both kernels, both RFD modes, both
integrators, extra mobility, bonds, the cell-list path's order and the
float-atomic form (whose sums depend on the order of its atomics)."""
import numpy as np
import pytest

from helpers import chains, rel_inf, uniform_positions

pytestmark = pytest.mark.gpu

CASES = {
    "3pt": dict(kernel=3),
    "4pt_paper": dict(kernel=4, rfd="RFD_PAPER"),
    "3pt_paper_extra": dict(kernel=3, rfd="RFD_PAPER", extra_mobility=0.3),
    "4pt_extra": dict(kernel=4, extra_mobility=0.3),
    "4pt_first": dict(kernel=4, scheme="SCHEME_FIRST_ORDER"),
    "3pt_first_extra": dict(kernel=3, scheme="SCHEME_FIRST_ORDER", extra_mobility=0.3),
    "4pt_none": dict(kernel=4, pair="PAIR_NONE"),
    "3pt_dense": dict(kernel=3, box=0.4),
    "4pt_float_atomic": dict(kernel=4, precision=1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_batch_equals_alone(fsl, name):
    kw = dict(CASES[name])
    for k in ("rfd", "scheme", "pair"):
        if k in kw:
            kw[k] = getattr(fsl, kw[k])
    scale = kw.pop("box", 1.0)
    kw.setdefault("pair", fsl.PAIR_SOFT)
    m, L = (24, 24, 24), (24.0, 24.0, 24.0)
    counts = [1, 7, 8, 9, 63, 64, 65, 255, 256, 257] + [640] * 8  # more than the quad kernels' least launch
    cfgs = [fsl.make_config(m, L, eta=1.0, kT=0.01, dt=0.01, cutoff=1.5, seed=100 + i, **kw) for i in range(len(counts))]
    qs = [uniform_positions(n, L, 50 + i) * scale for i, n in enumerate(counts)]
    q, bi, bj = chains(40, 16, L, 5)
    qs[-1] = q
    bonds = (bi, bj, np.full(len(bi), 10.0), np.ones(len(bi)))
    b = fsl.Batch(cfgs, qs)
    b.load_bonds(len(qs) - 1, *bonds)
    b.step(3)
    b.sync()
    for i, (c, q) in enumerate(zip(cfgs, qs)):
        g = fsl.StokesLimit(c, q)
        if i == len(qs) - 1:
            g.load_bonds(*bonds)
        g.step(3)
        g.sync()
        if kw.get("precision"):
            assert rel_inf(b.positions(i) - q, g.positions() - q) < 1e-5
        else:
            np.testing.assert_array_equal(b.positions(i), g.positions())
            np.testing.assert_array_equal(b.forces(i), g.forces())
        g.close()
    b.close()


@pytest.mark.parametrize("cutoff", [3.2, 5.0, 6.0])
def test_lennard_jones_lists(fsl, cutoff):
    """Lists of a few, a few dozen and (with the cells of a box of 24) nearly
    64 entries, whose forces a warp takes entry by entry."""
    m, L = (24, 24, 24), (24.0, 24.0, 24.0)
    rng = np.random.default_rng(1)
    counts = [1, 2, 33, 400] + [512] * 10
    qs = []
    for n in counts:
        sites = rng.permutation(512)[:n]
        s = np.stack([sites % 8, sites // 8 % 8, sites // 64])
        qs.append((s + 0.5) * 3.0 - 12.0 + rng.uniform(-0.2, 0.2, s.shape))
    cfgs = [fsl.make_config(m, L, eta=1.0, kT=0.01, dt=0.01, cutoff=cutoff, kernel=3, pair=fsl.PAIR_TABLE_LJ, seed=i) for i in range(len(qs))]
    b = fsl.Batch(cfgs, qs)
    b.step(3)
    b.sync()
    for i, (c, q) in enumerate(zip(cfgs, qs)):
        g = fsl.StokesLimit(c, q)
        g.step(3)
        g.sync()
        np.testing.assert_array_equal(b.positions(i), g.positions())
        np.testing.assert_array_equal(b.forces(i), g.forces())
        g.close()
    b.close()
