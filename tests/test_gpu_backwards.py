"""Steps backwards in time (dt < 0) with an absorber, whose factors are then above 1."""
import math

import numpy as np
import pytest

from tests import cases as C
from tests.test_gpu_at_size import _noise_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(1, 96), (1, 1021), (1, 1536), (2, 48), (2, 100), (2, 320), (3, 21), (3, 24)])
@pytest.mark.parametrize("absorber", ["cap", "cos8"])
def test_backwards_steps_match_oracle(dim, n, absorber):
    """Built lengths and convolutions, five steps of -dt in one call (opening, merged and closing X
    halves).  Tolerance: (2 dim log2(n) + 10) eps a step, times sqrt(n) for the oracle's direct
    DFT passes of a large prime factor, as in the comparisons forwards in time."""
    import qsf_gb300 as Q
    from oracle import oracle as O
    steps, dt, ncap = 5, -0.05, max(2, n // 10)
    psi0 = _noise_state(dim, n, 0.3, n)
    og = O.Grid(dim, n, 0.3, nCAP=ncap, pot=O.POT_EBERLY, Ncharge=float(dim), coupling=O.Coupling(O.GAUGE_VELOCITY, []))
    args = {}
    if absorber == "cos8":
        og.set_absorber(O.ABS_COS8, 0.05)
        args = dict(absorber=Q.ABS_COS8, mask_dt=0.05)
    og.psi[...] = psi0
    prop = O.Propagator(O.MODE_RE, dt, steps, og, ["norm", "epot"])
    for _ in range(steps):
        prop.make_step()
        prop.compute_each()
    g = Q.Grid(dim, n, 0.3, nCAP=ncap, Ncharge=float(dim), **args)
    g.upload(psi0)
    out, done = g.step(Q.MODE_RE, dt, steps, obs=Q.OBS_NORM | Q.OBS_EPOT)
    assert done == steps and out[-1, 0] > 1.0
    tol = steps * (2 * dim * math.log2(n) + 10) * 2.2e-16 * math.sqrt(n)
    assert C.rel_l2(g.download(), og.psi) < tol
    for s, r in enumerate(prop.rows):
        np.testing.assert_allclose(out[s, :2], [r["norm"], r["epot"]], rtol=4 * tol, atol=0)
    g.close()


@pytest.mark.parametrize("dim,n", [(1, 96), (1, 777), (2, 64), (2, 100), (3, 20)])
def test_time_steps_without_a_finite_factor_are_refused(dim, n):
    """A dt that is not a number, or whose imaginary-time factors no double holds, is an invalid
    argument, and the grid can be used afterwards."""
    import qsf_gb300 as Q
    g = Q.Grid(dim, n, 0.3, nCAP=2)
    for dt in (float("nan"), 1e6, -1e9):
        g.add_gaussian()
        with pytest.raises(Q.QsfError) as e:
            g.step(Q.MODE_IM, dt, 2)
        assert e.value.code == 1
    g.normalize()
    rows, done = g.step(Q.MODE_IM, 0.01, 2, normalize=True)
    assert done == 2 and np.isfinite(rows).all()
    g.close()
