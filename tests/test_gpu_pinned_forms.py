"""The CTA-wide stages stay reachable where the time loop runs on the warp-matrix
stages: pinned by bbw_set_config, steps() gives forward()'s bits, and in
split-FP16 solvers it is the tcgen05 stage, against the restatement (1e-5, its bar
elsewhere) and beside the warp-matrix stage."""
import numpy as np
import pytest
from conftest import golden, rel_l2

from bbwadg_b200 import WaveSolver, make_problem
from bbwadg_b200.problem import gaussian_source, receiver_weights, source_entries

pytestmark = pytest.mark.gpu
TOL = 1e-5
CTA = (8, True, False)


def problem(N, n, **kw):
    g = golden("ops_N%d.npz" % N)
    m = int(g["Nfq"][0])
    return make_problem(N, n, c2="sine", c2_jitter=0.5, seed=N,
                        cubature=(g["rq"], g["sq"], g["tq"], g["wq"]),
                        tri_cubature=(g["rfq"][:m], g["sfq"][:m], g["wfqFace"]), **kw)


@pytest.mark.parametrize("N,n,prec", [(3, 10, "fp32"), (4, 4, "fp32"), (5, 3, "fp32"),
                                      (4, 4, "f16x3"), (5, 3, "f16x3")])
def test_pinned_steps_equal_the_forward_pass(cuda, N, n, prec):
    """Traces and state of steps() and forward() bit for bit: the misfit at the
    medium that made the data is zero."""
    p = problem(N, n)
    el, w = receiver_weights(p, np.array([[0.05, 0.0, 0.1], [-0.3, 0.4, 0.5]]))
    out = []
    for tape in (False, True):
        s = WaveSolver(p, precision=prec)
        s.set_config(*CTA)
        s.set_sources(*source_entries(gaussian_source(p, (0.1, 0.2, 0.0), a=5.0)), f0=10.0)
        s.set_receivers(el, w, 4)
        s.set_data(p.Q0)
        if tape:
            s.forward(p.dt, 4).free()
        else:
            s.steps(p.dt, 4)
        out.append((s.get_traces(), s.get_data(), s.get_residual()))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("N,n,limit", [(4, 3, 0), (4, 3, 1), (5, 3, 0), (5, 10, 0), (5, 10, 3)])
def test_both_split_fp16_stages_match_restatement(cuda, N, n, limit):
    """A partial last tile, one CTA that walks every tile, many tiles per CTA; one
    tile below the range of a per-tile power-of-two scale, one exactly zero."""
    from oracle import Oracle
    p = problem(N, n)
    Q = p.Q0.reshape(p.K, 4, p.Np).copy()
    Q[:, 0] += 0.1
    Q[32:64] = 1e-39 * np.sign(Q[32:64] + 0.5)
    Q[96:128] = 0.0
    Q = Q.ravel().astype(np.float32)
    ref, _ = Oracle(N, p.K, p.ops_dict(), p.geo_dict()).run(Q.copy(), p.dt, 10)
    got = []
    for config in (CTA, (8, True, "group", 16)):
        s = WaveSolver(p, precision="f16x3")
        s.set_config(*config)
        s.set_grid_limit(limit)
        s.set_data(Q)
        s.steps(p.dt, 2)
        s.check()
        got.append(s.get_data())
        s.close()
        assert rel_l2(got[-1], ref) < TOL, config
    assert not np.array_equal(*got)  # two different kernels ran
