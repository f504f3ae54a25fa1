"""The ends of steps: the counters, sums and factors that a step leaves for the next one."""
import numpy as np
import pytest

from tests.test_gpu_at_size import _noise_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,nodes", [(2, 128, (25, 14, 10, 40)), (2, 100, (17, 10, 8, 25)), (3, 32, (6, 4, 3, 12))])
@pytest.mark.parametrize("substeps", [2, 3])
def test_substeps_of_a_step_match_steps_of_their_own(dim, n, nodes, substeps):
    """A step of K sub-steps is K steps of dt / K whose rows between are left out: the same
    launches, so the same bits.  Border sets of several hundred terms, which several blocks
    sum up, and many steps, because what is tested is the order of those blocks."""
    import qsf_gb300 as Q
    steps, dt = 48, 0.06
    psi0 = _noise_state(dim, n, 0.3, n)
    rows = np.zeros((steps * substeps, 3))
    rows[:, :dim] = 0.2 * np.random.default_rng(1).standard_normal((steps * substeps, 1))
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT, borders=Q.ZOA_FLUX_2D if dim == 2 else Q.ZOA_FLUX_3D)
    g = Q.Grid(dim, n, 0.3, nCAP=n // 10, Ncharge=float(dim), n_fields=1, border_nodes=nodes)
    g.upload(psi0)
    each, _ = g.step(Q.MODE_RE, dt / substeps, steps * substeps, rows, **kw)
    psi = g.download()
    assert np.abs(each[:, 3:]).max() > 0
    for _ in range(8):
        g.upload(psi0)
        got, done = g.step(Q.MODE_RE, dt, steps, rows, substeps=substeps, **kw)
        assert done == steps
        assert np.array_equal(got, each[substeps - 1::substeps])
        assert np.array_equal(g.download(), psi)
    g.close()


@pytest.mark.parametrize("dim,n", [(2, 128), (3, 32)])
def test_substeps_under_normalize_match_one_step_per_call(dim, n):
    """Normalize takes its factor from those sums: 2e-13 is the rounding of 64 steps at the
    (2 dim log2(n) + 10) eps a step of a correct run."""
    import qsf_gb300 as Q
    steps, dt = 32, 0.02
    psi0 = _noise_state(dim, n, 0.3, n)
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT, normalize=True, substeps=2,
              borders=Q.ZOA_FLUX_2D if dim == 2 else Q.ZOA_FLUX_3D)
    g = Q.Grid(dim, n, 0.3, nCAP=n // 10, Ncharge=float(dim), border_nodes=(25, 14, 10, 40) if dim == 2 else (6, 4, 3, 12))
    g.upload(psi0)
    each = np.concatenate([g.step(Q.MODE_IM, dt, 1, **kw)[0] for _ in range(steps)])
    ref = g.download()
    for _ in range(8):
        g.upload(psi0)
        got, done = g.step(Q.MODE_IM, dt, steps, **kw)
        assert done == steps
        np.testing.assert_allclose(got[:, :2], each[:, :2], rtol=4 * 2e-13, atol=0)
        assert np.linalg.norm(g.download() - ref) < 2e-13 * np.linalg.norm(ref)
    g.close()


@pytest.mark.parametrize("n", [96, 1536, 1021])
@pytest.mark.parametrize("substeps", [1, 3])
def test_line_normalize_keeps_psi_in_range(n, substeps):
    """300 large imaginary-time steps in one call: the raw norm grows by exp(2 |E| dt), about
    18, a step, past the range of a double within the 256 sub-steps of a launch.  Against
    calls of one step; the bound is that of the oracle comparison of these lines."""
    import math

    import qsf_gb300 as Q
    steps, dt = 300, 1.0
    psi0 = _noise_state(1, n, 0.2, n)
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT, normalize=True, substeps=substeps)
    g = Q.Grid(1, n, 0.2, nCAP=n // 10, Ncharge=2.0)
    g.upload(psi0)
    got, done = g.step(Q.MODE_IM, dt, steps, **kw)
    psi = g.download()
    assert done == steps
    g.upload(psi0)
    each = np.concatenate([g.step(Q.MODE_IM, dt, 1, **kw)[0] for _ in range(steps)])
    assert np.prod(each[-256:, 0], dtype=np.longdouble) > np.finfo(np.float64).max
    tol = steps * substeps * (2 * math.log2(n) + 10) * 2.2e-16
    np.testing.assert_allclose(got[:, :2], each[:, :2], rtol=4 * tol, atol=0)
    assert np.linalg.norm(psi - g.download()) < tol * np.linalg.norm(psi)
    g.close()


@pytest.mark.parametrize("dim,n", [(1, 96), (1, 1021), (2, 64), (2, 100)])
@pytest.mark.parametrize("steps", [60, 200])
def test_rows_after_a_converged_step_are_zero(dim, n, steps):
    """Calls whose rows travel with the control words (up to 256 values) and longer ones.  A
    full run goes before, so that the memory of the rows has held something."""
    import qsf_gb300 as Q
    psi0 = _noise_state(dim, n, 0.3, n)
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN, normalize=True, energy_after_normalize=3)
    g = Q.Grid(dim, n, 0.3, nCAP=n // 10, Ncharge=float(dim))
    g.upload(psi0)
    full, done = g.step(Q.MODE_IM, 0.05, steps, **kw)
    assert done == steps and full.all()
    g.upload(psi0)
    rows, done = g.step(Q.MODE_IM, 0.05, steps, state_accuracy=0.05, **kw)
    assert 1 < done < steps
    assert np.array_equal(rows[:done, :2], full[:done, :2])
    assert not rows[done:].any()
    g.close()


@pytest.mark.parametrize("dim,n", [(1, 96), (1, 1536), (1, 1021), (2, 64), (2, 100)])
@pytest.mark.parametrize("substeps,every,accuracy", [(1, 1, 0.05), (1, 1, 1e-4), (3, 1, 0.05), (1, 7, 0.05), (2, 4, 1e-3),
                                                     (1, 0, 0.02)])
def test_convergence_stop(dim, n, substeps, every, accuracy):
    """The stop comes after the first step whose energy (with E_kin every so often: among the
    steps that have it) is within the accuracy of the one before, one step later; that last
    step has E_kin, and psi is that of a call of as many steps.  every = 0: no E_kin."""
    import qsf_gb300 as Q
    steps, dt = 400, 0.05
    psi0 = _noise_state(dim, n, 0.3, n)
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT | (Q.OBS_EKIN if every else 0), normalize=True, energy_after_normalize=3,
              substeps=substeps, ekin_interval=max(every, 1))
    g = Q.Grid(dim, n, 0.3, nCAP=n // 10, Ncharge=float(dim))
    g.upload(psi0)
    full, _ = g.step(Q.MODE_IM, dt, steps, **kw)
    energy = (full[:, 1] + full[:, 2]) / full[:, 0]
    at = [s for s in range(steps) if every == 0 or (s + 1) % every == 0]
    last = next(s for before, s in zip([None] + at, at)
                if abs(energy[s] - (energy[before] if before is not None else 0.0)) <= accuracy) + 1
    assert 1 < last < steps - 1
    g.upload(psi0)
    rows, done = g.step(Q.MODE_IM, dt, steps, state_accuracy=accuracy, **kw)
    psi = g.download()
    assert done == last + 1
    assert np.array_equal(rows[:last], full[:last])
    g.upload(psi0)
    ref, _ = g.step(Q.MODE_IM, dt, done, **kw)
    assert np.array_equal(rows[:done], ref) and np.array_equal(psi, g.download())
    assert every == 0 or rows[last, 2] > 0
    g.close()


def test_batch_with_normalize_and_ekin_matches_alone():
    """Imaginary-time members, E_kin every step or every few, several groups, and a batch that
    advances in runs that end inside a member's period: the bits of each solve run alone."""
    import qsf_gb300 as Q
    specs = [(2, 48, 1, 60), (2, 64, 3, 50), (2, 64, 1, 40), (2, 128, 0, 45), (1, 256, 4, 60), (1, 1536, 1, 33),
             (3, 16, 5, 50), (3, 32, 0, 20)]
    made, alone = [], []
    for dim, n, every, steps in specs:
        nodes = (25, 14, 10, 40) if dim == 1 or n == 128 else (6, 4, 3, 12)
        psi0 = _noise_state(dim, n, 0.3, n + steps)
        g = Q.Grid(dim, n, 0.3, nCAP=n // 10, Ncharge=float(dim), border_nodes=nodes)
        kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT | (Q.OBS_EKIN if every else 0), normalize=True, ekin_interval=max(every, 1),
                  borders=[] if dim == 1 else Q.ZOA_FLUX_2D if dim == 2 else Q.ZOA_FLUX_3D)
        g.upload(psi0)
        rows, _ = g.step(Q.MODE_IM, 0.05, steps, **kw)
        alone.append((rows, g.download()))
        g.upload(psi0)
        made.append((g, steps, kw))
    b = Q.Batch()
    slots = [b.add(g, Q.MODE_IM, 0.05, steps, **kw) for g, steps, kw in made]
    while b.run(11):
        pass
    for (g, steps, _), slot, (rows, psi) in zip(made, slots, alone):
        got, done = b.result(slot)
        assert done == steps and np.array_equal(got, rows)
        b.remove(slot)
        assert np.array_equal(g.download(), psi)
    b.close()
