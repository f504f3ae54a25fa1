"""The fused 2D and 3D passes against the oracle at every line plan (qsf_lines.cuh): one
length per radix set and per way a line sits in warps (whole lines inside a warp, lines
ending inside one, lines of several warps), edges that are not a multiple of a column
block, both gauges, real and imaginary time.

Tolerance: the oracle's FP64 transforms err by about log2(m) eps per component and its
phase products by about 10 eps per step, both forward and back, so (2 log2(m) + 10) eps a
step bounds the relative L2 distance of a correct run.
"""
import math

import numpy as np
import pytest

from tests import cases as C
from tests.test_gpu_at_size import _fused_vs_oracle, _noise_state

pytestmark = pytest.mark.gpu
EPS = 2.2e-16


def _tol(dim, n, steps):
    return steps * (2 * dim * math.log2(n) + 10) * EPS


@pytest.mark.parametrize("dim,n", [(2, n) for n in (8, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256, 320,
                                                    384, 512, 640, 768, 1280, 1536)] +
                         [(3, n) for n in (8, 12, 20, 24, 40, 48, 64)])
@pytest.mark.parametrize("gauge", ["velocity", "length"])
def test_fused_steps_match_oracle(dim, n, gauge):
    import qsf_gb300 as Q
    pulse = dict(field=0.1, omega=1.1, ncycles=1.0)
    g = Q.GAUGE_LENGTH if gauge == "length" else Q.GAUGE_VELOCITY
    steps = 5 if n < 512 else 2
    got, ref, psi, opsi = _fused_vs_oracle(dim, n, 0.3, float(dim), g, steps, pulse, seed=n)
    tol = _tol(dim, n, steps)
    assert C.rel_l2(psi, opsi) < tol
    # the last step's sums over the oracle's psi, added pairwise (the oracle adds one by one)
    x = [np.reshape((np.arange(n) - (n - 1) / 2.0) * 0.3, [-1 if k == d else 1 for k in range(dim)]) for d in range(dim)]
    V = sum(-float(dim) / np.sqrt(c * c + 1.0) for c in x)
    V = V + sum(1.0 / np.sqrt((x[a] - x[b]) ** 2 + 1.0) for a in range(dim) for b in range(a))
    rho = np.abs(opsi) ** 2 * 0.3 ** dim
    np.testing.assert_allclose(got[-1, :2], [rho.sum(), (V * rho).sum()], rtol=2 * tol, atol=0)
    # a flux is a sum of products of neighbouring points: its error scales with the largest
    np.testing.assert_allclose(got[:, 2:], ref[:, 2:], rtol=0, atol=1e-12 * max(1e-30, np.abs(ref[:, 2:]).max()))


@pytest.mark.parametrize("dim,n,gauge,fields", [(2, 48, "velocity", 0), (2, 320, "length", 0), (3, 24, "velocity", 0),
                                                (2, 64, "length", 1)])
def test_imaginary_time_matches_oracle(dim, n, gauge, fields):
    """Normalize and E_kin every second step; with a length-gauge field the X halves change
    |psi|, so the closing and the next opening half do not merge."""
    import qsf_gb300 as Q
    from oracle import oracle as O
    steps, dt, axis = 6, 0.01, {2: 3, 3: 7}[dim]
    psi0 = _noise_state(dim, n, 0.3, n)
    lg = gauge == "length"
    pulse = dict(field=0.1, omega=1.1, ncycles=1.0)
    oc = O.Coupling(O.GAUGE_LENGTH if lg else O.GAUGE_VELOCITY, [O.Field(axis, [O.Pulse(**pulse)])] if fields else [])
    og = O.Grid(dim, n, 0.3, nCAP=n // 10, pot=O.POT_EBERLY, Ncharge=float(dim), coupling=oc)
    og.psi[...] = psi0
    prop = O.Propagator(O.MODE_IM, dt, steps, og, ["norm", "normalize", "epot", "ekin"])
    for _ in range(steps):
        prop.make_step()
        prop.compute_each()
    g = Q.Grid(dim, n, 0.3, nCAP=n // 10, Ncharge=float(dim), gauge=Q.GAUGE_LENGTH if lg else Q.GAUGE_VELOCITY,
               n_fields=fields)
    g.upload(psi0)
    qc = Q.Coupling(Q.GAUGE_LENGTH if lg else Q.GAUGE_VELOCITY, [Q.Field(axis, [Q.Pulse(**pulse)])] if fields else [])
    from qsf_gb300.propagator import coupling_schedule
    rows = coupling_schedule(qc, dt, steps)[0] if fields else None
    out, _ = g.step(Q.MODE_IM, dt, steps, rows, obs=Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN, normalize=True, ekin_interval=2)
    tol = _tol(dim, n, steps)
    assert C.rel_l2(g.download(), og.psi) < tol
    for s, r in enumerate(prop.rows):
        assert out[s, 0] == pytest.approx(r["norm"], rel=4 * tol)
        assert out[s, 1] / out[s, 0] == pytest.approx(r["epot"], rel=4 * tol)
        if s % 2:
            assert out[s, 2] / out[s, 0] == pytest.approx(r["ekin"], rel=4 * tol)
    g.close()
