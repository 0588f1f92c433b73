"""Sources, receivers and batched shots on the warp-matrix stages, pinned, and the
split-FP16 instances of the one-warp form, against the C restatement run one
shot at a time (1e-5 relative L2 on states, 1e-4 on traces, the bars of the other
shot tests)."""
import numpy as np
import pytest
from conftest import golden, rel_l2

from bbwadg_b200 import WaveSolver, _lib, make_problem
from bbwadg_b200.problem import receiver_weights

pytestmark = pytest.mark.gpu
TOL = 1e-5
SINGLE = 8 | 1 << 8 | 1 << 10 | 1 << 11
GROUP = 8 | 1 << 8 | 1 << 10 | 1 << 12


def problem(N, n):
    kw = {}
    if N >= 3:
        g = golden("ops_N%d.npz" % N)
        m = int(g["Nfq"][0])
        kw = dict(cubature=(g["rq"], g["sq"], g["tq"], g["wq"]),
                  tri_cubature=(g["rfq"][:m], g["sfq"][:m], g["wfqFace"]))
    return make_problem(N, n, c2="sine", c2_jitter=0.3, seed=N, **kw)


def sources(p, S, seed):
    """Per shot a random vector in the first element, in neighbouring tiles (15, 16,
    17, 31, 32), in one of the middle and in the last element of the ragged tile."""
    rng = np.random.default_rng(seed)
    elem = np.array([0, 15, 16, 17, 31, 32, p.K // 2, p.K - 1])
    dense = np.zeros((S, p.K, p.Np), np.float32)
    for s in range(S):
        dense[s, elem] = rng.standard_normal((len(elem), p.Np)).astype(np.float32)
    shot = np.repeat(np.arange(S), len(elem)).astype(np.int32)
    return dense, shot, np.tile(elem, S).astype(np.int32), dense[:, elem].reshape(-1, p.Np)


@pytest.mark.parametrize("N,code", [(1, SINGLE), (2, SINGLE), (3, SINGLE), (4, SINGLE), (4, GROUP),
                                    (5, GROUP), (6, GROUP)])
@pytest.mark.parametrize("stage_times,limit", [(False, 1), (True, 2), (True, 0)])
def test_shots_with_sources_match_restatement(cuda, N, code, stage_times, limit):
    """3^3 x 6 elements (a ragged last tile of two), three shots: one or two CTAs walk
    tiles across shot boundaries, or the whole grid one tile each."""
    from oracle import Oracle
    p = problem(N, 3)
    S, nsteps = 3, 4
    dense, shot, elem, vec = sources(p, S, N)
    el, w = receiver_weights(p, np.array([[0.05, 0.0, 0.1], [-0.3, 0.4, 0.5], [0.9, 0.9, 0.9]]))
    s = WaveSolver(p)
    _lib.call("bbw_set_config", s._h, code)
    s.set_shots(S)
    s.set_grid_limit(limit)
    s.set_sources(shot, elem, vec, f0=10.0, amplitude=1e4, stage_times=stage_times)
    s.set_receivers(el, w, nsteps)
    s.set_time(0.05)
    s.steps(p.dt, nsteps)
    traces, Q = s.get_traces(), s.get_data().reshape(S, -1)
    s.close()
    orc = Oracle(N, p.K, p.ops_dict(), p.geo_dict())
    for i in range(S):
        q, _, tr = orc.run(np.zeros(p.K * 4 * p.Np, np.float32), np.float32(p.dt), 5 * nsteps, t0=0.05,
                           source=dict(fsrc=dense[i], f0=10.0, tR=0.1, amp=1e4, stage_times=stage_times),
                           receivers=(el, w))
        assert rel_l2(Q[i], q) < TOL, i
        assert rel_l2(traces[i], tr) < 1e-4, i


@pytest.mark.parametrize("N,code", [(3, SINGLE), (4, SINGLE), (5, GROUP)])
def test_windows_with_sources_equal_the_whole_stage(cuda, N, code):
    """Windows that start inside a 16-element tile and inside a 32-element block of
    the source table."""
    p = problem(N, 3)
    _, shot, elem, vec = sources(p, 1, N)
    out = []
    for windows in ([(0, p.K)], [(0, 7), (7, 16), (16, 37), (37, 100), (100, p.K)]):
        s = WaveSolver(p)
        _lib.call("bbw_set_config", s._h, code)
        s.set_sources(shot, elem, vec, f0=10.0, amplitude=1e4)
        s.set_data(p.Q0)
        s.set_time(0.05)
        for k0, k1 in windows:
            s.stage_part(0.0, 0.5, p.dt, k0, k1)
        s.stage_commit()
        out.append((s.get_data(), s.get_residual()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("N,n,S", [(2, 10, 1), (3, 10, 1), (4, 6, 8)])
def test_split_fp16_one_warp_form_matches_restatement(cuda, N, n, S):
    """The sizes from which split FP16 takes one warp per tile: 375 tiles, and 648
    over eight shots at N = 4."""
    from oracle import Oracle
    p = problem(N, n)
    rng = np.random.default_rng(N)
    Q0 = np.stack([p.Q0 * (1 - 0.1 * i) + 0.01 * rng.standard_normal(p.Q0.size)
                   for i in range(S)]).astype(np.float32)
    s = WaveSolver(p, precision="f16x3")
    s.set_shots(S)
    s.set_data(Q0)
    s.steps(p.dt, 1)
    out = s.get_data().reshape(S, -1)
    s.close()
    orc = Oracle(N, p.K, p.ops_dict(), p.geo_dict())
    for i in {0, S - 1}:
        q, _ = orc.run(Q0[i].copy(), p.dt, 5)
        assert rel_l2(out[i], q) < TOL, i
