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


@pytest.mark.parametrize("substeps,n", [(1, 64), (2, 64), (3, 64), (1, 100)])
def test_normalize_in_one_call_matches_one_step_per_call(substeps, n):
    """The powers of two that Normalize takes out reach psi two sub-steps later: a long
    call against calls of one step, where none is pending.  The noise state loses most of
    its norm in each of the first steps."""
    import qsf_gb300 as Q
    steps, dt = 40, 0.05
    psi0 = _noise_state(2, n, 0.3, n)
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT, normalize=True, substeps=substeps)
    g = Q.Grid(2, n, 0.3, nCAP=n // 10, Ncharge=2.0)
    g.upload(psi0)
    one, _ = g.step(Q.MODE_IM, dt, steps, **kw)
    psi = g.download()
    g.upload(psi0)
    each = np.concatenate([g.step(Q.MODE_IM, dt, 1, **kw)[0] for _ in range(steps)])
    tol = _tol(2, n, steps * substeps)
    assert C.rel_l2(psi, g.download()) < tol
    np.testing.assert_allclose(one[:, :2], each[:, :2], rtol=4 * tol, atol=0)
    g.close()


@pytest.mark.parametrize("every,substeps", [(1, 1), (3, 1), (20, 1), (5, 2), (70, 1)])
def test_ekin_interval_in_one_call_matches_one_step_per_call(every, substeps):
    """Whole periods of passes in a graph (shorter and longer than the tables of one
    launch, and too long for a graph), with steps left over."""
    import qsf_gb300 as Q
    n, steps, dt = 64, 73, 0.01
    psi0 = _noise_state(2, n, 0.3, n)
    obs = Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN
    g = Q.Grid(2, n, 0.3, nCAP=n // 10, Ncharge=2.0)
    g.upload(psi0)
    one, _ = g.step(Q.MODE_IM, dt, steps, obs=obs, normalize=True, substeps=substeps, ekin_interval=every)
    psi = g.download()
    g.upload(psi0)
    each = np.concatenate([g.step(Q.MODE_IM, dt, 1, obs=obs, normalize=True, substeps=substeps)[0] for _ in range(steps)])
    tol = _tol(2, n, steps * substeps)
    assert C.rel_l2(psi, g.download()) < tol
    np.testing.assert_allclose(one[:, :2], each[:, :2], rtol=4 * tol, atol=0)
    at = [s for s in range(steps) if (s + 1) % every == 0 or s + 1 == steps]
    np.testing.assert_allclose(one[at, 2], each[at, 2], rtol=8 * tol, atol=0)
    assert not np.delete(one[:, 2], at).any()
    g.close()


# lines run as convolutions: shorter and longer than a box of the strided copies, ragged last
# column blocks and boxes, plans of exactly 2 n - 1 + 1 points and with spare ones
@pytest.mark.parametrize("dim,n", [(2, n) for n in (3, 7, 33, 63, 65, 100, 127, 129, 250, 513)] + [(3, n) for n in (5, 21, 50, 66)])
@pytest.mark.parametrize("gauge,mode", [("velocity", "real"), ("length", "real"), ("velocity", "imaginary")])
def test_convolution_steps_match_oracle(dim, n, gauge, mode):
    """sqrt(n): the oracle's direct DFT passes of a large prime factor add up to n terms."""
    import qsf_gb300 as Q
    from oracle import oracle as O
    from qsf_gb300.propagator import coupling_schedule
    real, lg, steps = mode == "real", gauge == "length", 4
    dt, axis = (0.05 if real else 0.01), {2: 3, 3: 7}[dim]
    psi0 = _noise_state(dim, n, 0.3, n)
    pulse = dict(field=0.1, omega=1.1, ncycles=1.0)
    og_g, qg = (O.GAUGE_LENGTH, Q.GAUGE_LENGTH) if lg else (O.GAUGE_VELOCITY, Q.GAUGE_VELOCITY)
    oc = O.Coupling(og_g, [O.Field(axis, [O.Pulse(**pulse)])] if real else [])
    og = O.Grid(dim, n, 0.3, nCAP=max(1, n // 10), pot=O.POT_EBERLY, Ncharge=float(dim), coupling=oc)
    og.psi[...] = psi0
    outs = ["norm", "epot"] if real else ["norm", "normalize", "epot", "ekin"]
    prop = O.Propagator(O.MODE_RE if real else O.MODE_IM, dt, steps, og, outs)
    for _ in range(steps):
        prop.make_step()
        prop.compute_each()
    g = Q.Grid(dim, n, 0.3, nCAP=max(1, n // 10), Ncharge=float(dim), gauge=qg, n_fields=1 if real else 0)
    g.upload(psi0)
    if real:
        rows = coupling_schedule(Q.Coupling(qg, [Q.Field(axis, [Q.Pulse(**pulse)])]), dt, steps)[0]
        out, done = g.step(Q.MODE_RE, dt, steps, rows, obs=Q.OBS_NORM | Q.OBS_EPOT)
    else:
        out, done = g.step(Q.MODE_IM, dt, steps, obs=Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN, normalize=True, ekin_interval=2)
    assert done == steps
    tol = _tol(dim, n, steps) * math.sqrt(n)
    assert C.rel_l2(g.download(), og.psi) < tol
    for s, r in enumerate(prop.rows):
        f = 1.0 if real else out[s, 0]
        assert out[s, 0] == pytest.approx(r["norm"], rel=4 * tol)
        assert out[s, 1] / f == pytest.approx(r["epot"], rel=4 * tol)
        if not real and s % 2:
            assert out[s, 2] / f == pytest.approx(r["ekin"], rel=8 * tol)
    g.close()


def _line_oracle(n, lg, mode, steps, dt, psi0, pulse, outs):
    from oracle import oracle as O
    oc = O.Coupling(O.GAUGE_LENGTH if lg else O.GAUGE_VELOCITY, [O.Field(1, [O.Pulse(**pulse)])] if pulse else [])
    og = O.Grid(1, n, 0.2, nCAP=max(1, n // 10), pot=O.POT_EBERLY, Ncharge=1.0, coupling=oc)
    og.psi[...] = psi0
    prop = O.Propagator(O.MODE_RE if mode == "real" else O.MODE_IM, dt, steps, og, outs)
    for _ in range(steps):
        prop.make_step()
        prop.compute_each()
    return og.psi, prop.rows


# one length per geometry of the 1D kernels: one line in a CTA (its lanes filling warps or
# not), N1 x N2 over 1, 2, 4 and 8 CTAs with 4 and 8 points per thread, every radix family,
# and convolution lengths for n at the edges of their ranges
LINES = [8, 12, 20, 40, 96, 160, 256, 320, 384, 640, 512, 768, 1024, 1280, 1536, 2048, 2560, 3072, 4096, 5120, 6144, 8192,
         10240, 12288, 16384, 7, 255, 257, 383, 1025, 4095, 5003, 8191, 10239, 12289, 16383]


@pytest.mark.parametrize("n", LINES)
@pytest.mark.parametrize("mode,gauge", [("real", "velocity"), ("real", "length"), ("imaginary", "velocity")])
def test_line_steps_match_oracle(n, mode, gauge):
    """Whole 1D steps: psi, norm, E_pot, E_kin (imaginary time, every second step, with
    Normalize) and the BOX flux."""
    import qsf_gb300 as Q
    from oracle import oracle as O
    from qsf_gb300.propagator import coupling_schedule
    real, lg, steps = mode == "real", gauge == "length", 6
    dt = 0.05 if real else 0.01
    psi0 = _noise_state(1, n, 0.2, n)
    pulse = dict(field=0.1, omega=1.1, ncycles=1.0) if real else None
    box = n // 4
    outs = ["norm", "epot", ("flux", ["BOX"], box)] if real else ["norm", "normalize", "epot", "ekin"]
    O.set_border_nodes(25, 14, 10, 40)
    opsi, orows = _line_oracle(n, lg, mode, steps, dt, psi0, pulse, outs)
    g = Q.Grid(1, n, 0.2, nCAP=max(1, n // 10), Ncharge=1.0, gauge=Q.GAUGE_LENGTH if lg else Q.GAUGE_VELOCITY,
               n_fields=1 if real else 0)
    g.upload(psi0)
    rows = None
    if real:
        c = Q.Coupling(Q.GAUGE_LENGTH if lg else Q.GAUGE_VELOCITY, [Q.Field(1, [Q.Pulse(**pulse)])])
        rows = coupling_schedule(c, dt, steps)[0]
        out, done = g.step(Q.MODE_RE, dt, steps, rows, obs=Q.OBS_NORM | Q.OBS_EPOT, borders=["BOX"], box_size=box)
    else:
        out, done = g.step(Q.MODE_IM, dt, steps, obs=Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN, normalize=True, ekin_interval=2)
    assert done == steps
    # lengths with a large prime factor: the oracle's direct DFT passes add up to n terms
    tol = _tol(1, n, steps) * (1 if n in LINES[:25] else math.sqrt(n))
    assert C.rel_l2(g.download(), opsi) < tol
    for s, r in enumerate(orows):
        f = 1.0 if real else out[s, 0]
        assert out[s, 0] == pytest.approx(r["norm"], rel=4 * tol)
        assert out[s, 1] / f == pytest.approx(r["epot"], rel=4 * tol)
        if real:
            assert out[s, 3] == pytest.approx(r["flux"][0], abs=8 * tol * np.abs(psi0).max() ** 2 / 0.2)
        elif s % 2:
            assert out[s, 2] / f == pytest.approx(r["ekin"], rel=8 * tol)
    g.close()


@pytest.mark.parametrize("n", [96, 1536, 4096, 1021])
def test_line_run_does_not_depend_on_its_launches(n):
    """One call of 7 steps, seven calls of one step, and psi taken out and put back between
    them give the same bits."""
    import qsf_gb300 as Q
    psi0 = _noise_state(1, n, 0.2, 3)
    rng = np.random.default_rng(4)
    rows = 0.1 * rng.standard_normal((7, 6))
    kw = dict(obs=Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN, borders=["BOX"], box_size=n // 4)
    g = Q.Grid(1, n, 0.2, nCAP=n // 10, gauge=Q.GAUGE_LENGTH, n_fields=1)
    g.upload(psi0)
    whole, _ = g.step(Q.MODE_RE, 0.05, 7, rows, **kw)
    psi = g.download()
    g.upload(psi0)
    parts = []
    for s in range(7):
        parts.append(g.step(Q.MODE_RE, 0.05, 1, rows[s:s + 1], **kw)[0].copy())
        g.upload(g.download())
    assert np.array_equal(np.concatenate(parts), whole) and np.array_equal(g.download(), psi)
    g.close()
