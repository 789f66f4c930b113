"""The transforms of extents without compiled passes (fsl_fft_g.cu): every
stage count (one to four), odd extents, primes, planes that fit shared memory
and planes that do not, in FP32 and FP64, alone and in a batch, against the
FP64 oracle.

FP32: the suite's 1e-5 of the solve.  FP64: a line transform of n points
rounds at most about 5 eps log2(n) relative, six of them follow each other on
each side: 12 x 5 x 1.1e-16 x 10 < 7e-14; 1e-12 is asked for.
"""
import numpy as np
import pytest

from helpers import rel_inf, uniform_positions

pytestmark = pytest.mark.gpu

# planes in shared memory; x, y, z with three and four stages; planes too
# large for shared memory; one thread a line (3, 7, 11)
GRIDS = [(3, 4, 5), (7, 11, 9), (11, 7, 45), (60, 18, 25), (15, 20, 125), (125, 14, 3), (12, 147, 5), (625, 4, 3), (3, 875, 4),
         (252, 250, 3), (224, 225, 4), (10, 9, 588), (64, 64, 44), (48, 50, 64)]


@pytest.mark.parametrize("m", GRIDS)
def test_solve_fp32(fsl, oracle, m):
    L = tuple(float(e) * s for e, s in zip(m, (1.0, 1.25, 0.8)))
    cfg = fsl.make_config(m, L, eta=0.7, kT=0.01, dt=0.01, cutoff=1.5, pair=fsl.PAIR_NONE, seed=3)
    g = fsl.StokesLimit(cfg, np.zeros((3, 0)))
    o = oracle.Oracle(*m, *L, np.zeros((3, 0)), eta=0.7, kT=0.01, dt=0.01, cutoff=1.5, pair=oracle.PAIR_NONE, seed=3)
    W = np.random.default_rng(5).standard_normal((3,) + m[::-1])
    assert rel_inf(g.solve(W), o.solve(W).reshape(W.shape)) < 1e-5
    g.close()


@pytest.mark.parametrize("m", [(16, 16, 16), (33, 20, 21), (125, 14, 9), (12, 147, 10), (10, 12, 189), (176, 180, 6), (64, 48, 32)])
def test_step_fp64(fsl, oracle, m):
    L = tuple(float(e) for e in m)
    q = uniform_positions(40, L, 2)
    kw = dict(eta=1.3, kT=0.01, dt=0.01, cutoff=1.5, kernel=4, seed=11)
    cfg = fsl.make_config(m, L, pair=fsl.PAIR_SOFT, precision=2, **kw)
    g = fsl.StokesLimit(cfg, q)
    o = oracle.Oracle(*m, *L, q, pair=oracle.PAIR_SOFT, **kw)
    g.step(1)
    o.step(1)
    g.sync()
    assert rel_inf(g.velocity64(), o.velocity().reshape((3,) + m[::-1])) < 1e-12
    g.close()


@pytest.mark.parametrize("m", [(16, 16, 16), (9, 22, 15), (125, 12, 8), (14, 8, 125)])
def test_incompressible(fsl, oracle, m):
    L = tuple(float(e) for e in m)
    v = 0.1 * np.random.default_rng(4).standard_normal((3,) + m[::-1])
    kw = dict(eta=1.1, kT=0.02, dt=0.05, seed=5, density=0.9)
    g = fsl.StokesLimit(fsl.make_config(m, L, scheme=fsl.SCHEME_INCOMPRESSIBLE, **kw), np.zeros((3, 0)))
    o = oracle.Oracle(*m, *L, np.zeros((3, 0)), scheme=oracle.SCHEME_INCOMPRESSIBLE, **kw)
    g.set_velocity64(v)
    o.set_velocity(v)
    g.step(2)
    o.step(2)
    g.sync()
    assert rel_inf(g.velocity64(), o.velocity().reshape(v.shape)) < 1e-11
    g.close()


@pytest.mark.parametrize("scheme", ["SCHEME_QUASI2D", "SCHEME_STOKES2D"])
@pytest.mark.parametrize("m", [(33, 25), (24, 21), (21, 40), (256, 12), (250, 147)])
def test_quasi2d(fsl, oracle, m, scheme):
    L = (float(m[0]), float(m[1]), 4.0)
    q = uniform_positions(60, L, 8)
    kw = dict(eta=0.9, kT=0.05, dt=0.01, cutoff=1.5, seed=21, radius=1.0, predictor_corrector=1)
    g = fsl.StokesLimit(fsl.make_config(m + (1,), L, scheme=getattr(fsl, scheme), pair=fsl.PAIR_SOFT, **kw), q)
    o = oracle.Oracle(*m, 1, *L, q, scheme=getattr(oracle, scheme), pair=oracle.PAIR_SOFT, **kw)
    g.step(2)
    o.step(2)
    g.sync()
    assert rel_inf(g.positions() - q, o.positions() - q) < 1e-9
    g.close()


@pytest.mark.parametrize("precision", [0, 2])
def test_batch_equals_alone(fsl, precision):
    m, L = (20, 18, 22), (20.0, 18.0, 22.0)
    cfgs = [fsl.make_config(m, L, eta=e, kT=0.01, dt=0.01, cutoff=1.5, pair=fsl.PAIR_SOFT, seed=s, precision=precision)
            for e, s in ((1.0, 3), (0.6, 4), (1.7, 5))]
    qs = [uniform_positions(n, L, n) for n in (50, 1, 130)]
    b = fsl.Batch(cfgs, qs)
    b.step(3)
    b.sync()
    for i, (c, q) in enumerate(zip(cfgs, qs)):
        g = fsl.StokesLimit(c, q)
        g.step(3)
        g.sync()
        # the FP64 form spreads with FP64 atomics, whose order varies
        if precision == 0:
            np.testing.assert_array_equal(b.positions(i), g.positions())
        else:
            assert rel_inf(b.positions(i) - q, g.positions() - q) < 1e-10
        g.close()
    b.close()
