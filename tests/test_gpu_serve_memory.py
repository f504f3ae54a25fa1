"""Admission of 1D solves: what it counts covers what they hold."""
import time

import numpy as np
import pytest

from tests.test_gpu_at_size import _noise_state

pytestmark = pytest.mark.gpu
N, STEPS, ROUND, COUNT, BUDGET = 16384, 256, 16, 64, 300e6


@pytest.mark.parametrize("gauge", ["velocity", "length"])
def test_line_solves_stay_within_the_reserve(gauge):
    """64 solves of 256 steps on 16384 points do not fit a budget of 300 MB at once, so some
    wait; the free memory must not fall below the reserve (32 MB for the granularity of the
    allocations).  Every solve is the same one, of several rounds, and has to end as it
    does alone in one call."""
    import torch

    import qsf_gb300 as Q
    from qsf_gb300.serve import Server, grid_desc
    lg = gauge == "length"
    gg = Q.GAUGE_LENGTH if lg else Q.GAUGE_VELOCITY
    rows = 0.05 * np.random.default_rng(2).standard_normal((STEPS, 6 if lg else 3))
    psi0 = _noise_state(1, N, 0.2, 7)
    args = dict(nCAP=N // 10, Ncharge=1.0, gauge=gg, n_fields=1)
    obs = dict(obs=Q.OBS_NORM | Q.OBS_EPOT, borders=["BOX"], box_size=N // 4)
    g = Q.Grid(1, N, 0.2, **args)
    g.upload(psi0)
    alone, done = g.step(Q.MODE_RE, 0.05, STEPS, rows, **obs)
    assert done == STEPS
    g.close()
    d = grid_desc(1, N, 0.2, **args)
    warm = Server(max_slots=1, steps_per_round=ROUND)  # loads the kernels and the shared tables
    warm.wait(warm.submit(d, Q.MODE_RE, 0.05, STEPS, rows, psi0, **obs))
    warm.stop()
    free0, _ = torch.cuda.mem_get_info()
    reserve = free0 - BUDGET
    srv = Server(max_slots=COUNT, hbm_reserve_gb=reserve / 1e9, steps_per_round=ROUND)
    try:
        tickets = [srv.submit(d, Q.MODE_RE, 0.05, STEPS, rows, psi0, **obs) for _ in range(COUNT)]
        least = free0
        end = time.monotonic() + 60
        while srv.stats()["completed"] < COUNT:
            assert time.monotonic() < end, "solves that fit stay queued"
            least = min(least, torch.cuda.mem_get_info()[0])
        res = [srv.wait(t, 300) for t in tickets]
    finally:
        srv.stop()
    assert least < free0 - 50e6  # several were resident at once
    assert least > reserve - 32e6
    for r in res:
        assert r["status"] == 0 and r["steps"] == STEPS
        assert r["final_norm"] == alone[-1, 0] and r["final_epot"] == alone[-1, 1]
        assert r["flux_integral"][0] == pytest.approx(0.05 * alone[:, 3].sum(), rel=1e-12, abs=1e-12 * np.abs(alone[:, 3]).sum())
