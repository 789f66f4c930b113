"""fsl_step_io: one step with its positions in from and out to host memory
gives the bits of fsl_set_positions + fsl_step(1) + fsl_get_positions.

With page-locked buffers both copies are nodes of the step's graph and the
copy in runs beside the noise; with pageable buffers the three calls run.
Between steps the host moves the particles (some by more than half the
Verlet skin, so the moved check inside the graph requests list rebuilds),
as a caller coupling the step to host-side work would.
"""
import numpy as np
import pytest

from helpers import uniform_positions

pytestmark = pytest.mark.gpu


def _config(fsl):
    return fsl.make_config((48, 48, 48), (48.0,) * 3, kT=0.01, dt=0.01, cutoff=1.5, kernel=4,
                           pair=fsl.PAIR_SOFT, seed=41)


def _host_moves(q, rng, k):
    """Small moves every step, a few large ones every third step."""
    q += rng.normal(0.0, 0.01, q.shape)
    if k % 3 == 2:
        idx = rng.choice(q.shape[1], 20, replace=False)
        q[:, idx] += rng.normal(0.0, 0.5, (3, 20))


@pytest.mark.parametrize("pinned", [True, False], ids=["pinned", "pageable"])
def test_step_io_equals_set_step_get(fsl, pinned):
    import torch
    cfg = _config(fsl)
    q0 = uniform_positions(6000, (48, 48, 48), 7)
    a = fsl.StokesLimit(cfg, q0)
    b = fsl.StokesLimit(cfg, q0)
    if pinned:
        buf = torch.empty((3, q0.shape[1]), dtype=torch.float64).pin_memory()
        qa = buf.numpy()
    else:
        qa = np.empty_like(q0)
    qa[...] = q0
    qb = q0.copy()
    rng_a, rng_b = np.random.default_rng(3), np.random.default_rng(3)
    for k in range(9):
        a.step_io(qa, qa)
        b.set_positions(qb)
        b.step(1)
        qb = b.positions()
        np.testing.assert_array_equal(qa, qb)
        _host_moves(qa, rng_a, k)
        _host_moves(qb, rng_b, k)
    np.testing.assert_array_equal(a.forces(), b.forces())
    np.testing.assert_array_equal(a.velocity(), b.velocity())
    sa, sb = a.status(), b.status()
    assert sa["step"] == sb["step"] == 9 and sa["error_bits"] == sb["error_bits"] == 0
    if pinned:
        assert sa["graph"]
    a.close()
    b.close()


def test_step_io_then_plain_steps(fsl):
    """Alternating the input/output step with plain steps (each change of
    step kind captures its graph again) keeps the bits of the plain calls."""
    import torch
    cfg = _config(fsl)
    q0 = uniform_positions(3000, (48, 48, 48), 8)
    a = fsl.StokesLimit(cfg, q0)
    b = fsl.StokesLimit(cfg, q0)
    buf = torch.empty((3, q0.shape[1]), dtype=torch.float64).pin_memory()
    qa = buf.numpy()
    qa[...] = q0
    rng = np.random.default_rng(5)
    for k in range(4):
        q_in = qa.copy()
        a.step_io(qa, qa)
        a.step(2)
        b.set_positions(q_in)
        b.step(3)
        np.testing.assert_array_equal(a.positions(), b.positions())
        qa[...] = a.positions() + rng.normal(0.0, 0.01, qa.shape)
    a.close()
    b.close()


def _follow(fsl, cfg, q0):
    """step_io on a pinned buffer against set_positions, step and positions,
    with host moves in between (2-D instances: in the plane)."""
    import torch
    a, b = fsl.StokesLimit(cfg, q0), fsl.StokesLimit(cfg, q0)
    buf = torch.empty(q0.shape, dtype=torch.float64).pin_memory()
    qa = buf.numpy()
    qa[...] = q0
    rng = np.random.default_rng(12)
    for k in range(5):
        qb = qa.copy()
        a.step_io(qa, qa)
        b.set_positions(qb)
        b.step(1)
        yield qa, b.positions()
        qa[:2] += rng.normal(0.0, 0.01, (2, q0.shape[1]))
        if k % 2:
            idx = rng.choice(q0.shape[1], 20, replace=False)
            qa[:2, idx] += rng.normal(0.0, 0.5, (2, 20))
    sa = a.status()
    assert sa["step"] == 5 and sa["error_bits"] == 0 and sa["graph"]
    a.close()
    b.close()


@pytest.mark.parametrize("n", [16384, 16385])
def test_step_io_kernels_and_copy_nodes(fsl, n):
    """Page-locked buffers up to 16,384 particles by kernels, from there on
    by copy nodes and the moved check in the step's graph."""
    for got, want in _follow(fsl, _config(fsl), uniform_positions(n, (48, 48, 48), 7)):
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n", [300, 17000])
@pytest.mark.parametrize("scheme", ["SCHEME_FIRST_ORDER", "SCHEME_QUASI2D", "SCHEME_STOKES2D"])
def test_step_io_other_schemes(fsl, scheme, n):
    two_d = scheme != "SCHEME_FIRST_ORDER"
    m = (48, 48, 1) if two_d else (48, 48, 48)
    L = (48.0, 48.0, 4.0) if two_d else (48.0,) * 3
    q0 = uniform_positions(n, L, 8)
    if two_d:
        q0[2] = 0.0
    cfg = fsl.make_config(m, L, kT=0.01, dt=0.01, cutoff=1.5, kernel=3, pair=fsl.PAIR_SOFT, seed=42, radius=1.0,
                          extra_mobility=0.0 if two_d else 0.2, scheme=getattr(fsl, scheme))
    for got, want in _follow(fsl, cfg, q0):
        if two_d:  # FP64 atomics: sums in any order, rounding of a thousand terms
            np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 * 48)
        else:
            np.testing.assert_array_equal(got, want)


def test_step_io_without_particles(fsl):
    """The incompressible fluid has no positions: the step alone."""
    import torch
    cfg = fsl.make_config((16, 16, 16), (16.0,) * 3, kT=0.01, dt=0.05, seed=3, scheme=fsl.SCHEME_INCOMPRESSIBLE)
    a, b = fsl.StokesLimit(cfg, np.zeros((3, 0))), fsl.StokesLimit(cfg, np.zeros((3, 0)))
    buf = torch.empty(8, dtype=torch.float64).pin_memory()
    for _ in range(3):
        a.step_io(buf.data_ptr(), buf.data_ptr())
    b.step(3)
    np.testing.assert_array_equal(a.velocity64(), b.velocity64())
    assert a.status()["step"] == 3
    a.close()
    b.close()


def test_step_io_unaligned_buffer(fsl):
    """Page-locked doubles at an address that is no multiple of 8 (or of 4):
    taken by copies, which have no alignment."""
    import torch
    cfg = _config(fsl)
    q0 = uniform_positions(100, (48, 48, 48), 9)
    a, b = fsl.StokesLimit(cfg, q0), fsl.StokesLimit(cfg, q0)
    raw = torch.empty(q0.nbytes + 8, dtype=torch.uint8).pin_memory()
    for off in (4, 1, 0):
        view = raw.numpy()[off:off + q0.nbytes]
        view[:] = np.frombuffer(q0.tobytes(), np.uint8)
        a.step_io(raw.data_ptr() + off, raw.data_ptr() + off)
        b.set_positions(q0)
        b.step(1)
        q0 = b.positions()
        np.testing.assert_array_equal(np.frombuffer(view.tobytes()).reshape(q0.shape), q0)
    a.close()
    b.close()


@pytest.mark.parametrize("pinned", [True, False], ids=["pinned", "pageable"])
def test_batch_step_io_equals_set_step_get(fsl, pinned):
    """The batched form: every instance of a batch over three size classes
    (one instance empty) bit for bit as the packed set, step and get."""
    import torch
    rng = np.random.default_rng(9)
    cfgs, qs = [], []
    for i in range(9):
        m = (16, 24, 32)[i % 3]
        n = 0 if i == 4 else 200 + 150 * i
        cfgs.append(fsl.make_config((m, m, m), (float(m),) * 3, kT=0.01, dt=0.01, cutoff=1.5,
                                    kernel=3 + i % 2, pair=fsl.PAIR_SOFT, seed=60 + i))
        qs.append(uniform_positions(n, (m, m, m), 20 + i))
    a = fsl.Batch(cfgs, qs)
    b = fsl.Batch(cfgs, qs)
    n = int(a.offsets[-1])
    if pinned:
        buf = torch.empty(n, dtype=torch.float64).pin_memory()
        qa = buf.numpy()
    else:
        qa = np.empty(n)
    a.positions_packed(qa)
    qb = qa.copy()
    for k in range(6):
        a.step_io(qa, qa)
        b.set_positions_packed(qb)
        b.step(1)
        b.positions_packed(qb)
        np.testing.assert_array_equal(qa, qb)
        moves = rng.normal(0.0, 0.01, n)
        qa += moves
        qb += moves
    for i in range(len(cfgs)):
        np.testing.assert_array_equal(a.forces(i), b.forces(i))
        assert a.status(i)["error_bits"] == b.status(i)["error_bits"] == 0
    a.close()
    b.close()
