"""The steps' graph, whose stages start before the stage ahead has ended, against
the same stages launched one by one, bit for bit: small meshes (all of a stage
resident beside the next), several tiles per CTA, and one CTA for all."""
import numpy as np
import pytest

from bbwadg_b200 import RK4A, RK4B, WaveSolver, make_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [(1, 3), (2, 8), (3, 3), (3, 8), (4, 3), (4, 11), (5, 3), (5, 12),
                                 (8, 2)])
@pytest.mark.parametrize("limit", [0, 1])
def test_steps_match_single_stages(cuda, N, n, limit):
    if limit and n > 8:
        n = 4
    p = make_problem(N, n, c2="sine", c2_jitter=0.5, seed=N)
    rng = np.random.default_rng(N)
    Q = (p.Q0 + 0.1 * rng.standard_normal(p.Q0.shape)).astype(np.float32)
    out = []
    for graph in (True, False):
        s = WaveSolver(p)
        s.set_grid_limit(limit)
        s.set_data(Q)
        if graph:
            s.steps(p.dt, 4)
        else:
            for _ in range(4):
                for a, b in zip(RK4A, RK4B):
                    s.rk_stage(np.float32(a), np.float32(b), p.dt, 0.0)
        out.append((s.get_data(), s.get_residual()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
