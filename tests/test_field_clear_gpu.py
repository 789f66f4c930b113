"""The spread field is cleared whole between spreads for every cell count: odd
counts end in half a 16-byte group (fixed point) or in part of one (float
sums).  Particles sit around the field's last cells; a value left there would
come back as a force in the next solve.  Against the FP64 oracle."""
import numpy as np
import pytest

from helpers import rel_inf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fixed64", "float_atomic"])
@pytest.mark.parametrize("m", [(15, 9, 21), (9, 7, 10), (25, 15, 27)])
def test_last_cells(fsl, oracle, m, precision):
    L = tuple(float(e) for e in m)
    rng = np.random.default_rng(3)
    q = 0.5 * np.asarray(L)[:, None] - rng.uniform(0.0, 2.0, (3, 12))
    kw = dict(eta=1.0, kT=1e-4, dt=0.01, cutoff=1.5, kernel=4, seed=6)
    g = fsl.StokesLimit(fsl.make_config(m, L, pair=fsl.PAIR_SOFT, precision=precision, **kw), q)
    o = oracle.Oracle(*m, *L, q, pair=oracle.PAIR_SOFT, **kw)
    for _ in range(6):
        g.step(1)
        o.step(1)
    g.sync()
    assert rel_inf(g.positions() - q, o.positions() - q) < 1e-5
    assert rel_inf(g.velocity64(), o.velocity().reshape((3,) + m[::-1])) < 1e-4
    g.close()
