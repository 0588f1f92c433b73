"""The curved elements' stage on warp-level matrix instructions, at the smallest
balls that take it, against the FP64 restatement (1e-5 relative L2, the FP32
bar of the curvilinear path), and the device-side state permutation."""
import numpy as np
import pytest
from conftest import golden, rel_l2

from bbwadg_b200.curved import CurvedSolver, make_curved_problem

pytestmark = pytest.mark.gpu
TOL = 1e-5


def problem(N, n, rule):
    kw = {}
    if rule == "table":
        g = golden("ops_N%d.npz" % N)
        m = int(g["Nfq"][0])
        kw = dict(cubature=(g["rq"], g["sq"], g["tq"], g["wq"]),
                  tri_cubature=(g["rfq"][:m], g["sfq"][:m], g["wfqFace"]))
    return make_curved_problem(N, n, c2=lambda x, y, z: 1.0 + 0.4 * np.sin(3 * x) * np.cos(y + z), **kw)


@pytest.mark.parametrize("N,n,rule", [(1, 16, "default"), (2, 12, "default"), (3, 8, "table"),
                                      (3, 8, "default"), (3, 16, "table"), (4, 6, "table"),
                                      (5, 6, "table"), (5, 6, "default")])
def test_matrix_stage_matches_restatement(cuda, N, n, rule):
    from curved import CurvedOracle
    p = problem(N, n, rule)
    rng = np.random.default_rng(N)
    Q = (p.Q0 + 0.05 * rng.standard_normal(p.Q0.size)).astype(np.float32)
    s = CurvedSolver(p)
    s.set_data(Q)
    s.steps(p.dt, 1)
    got, res = s.get_data(), s.get_residual()
    s.close()
    ref, rref = CurvedOracle(N, p.K, p.Nq, p.Nfq, p.desc_arrays()).run(Q, p.dt, 5)
    assert rel_l2(got, ref) < TOL
    assert rel_l2(res, rref) < 1e-4


def test_state_round_trip_between_stages(cuda):
    """The permutation goes through the next state's buffer: reading the state
    or the residual changes neither."""
    p = problem(3, 8, "table")
    a, b = CurvedSolver(p), CurvedSolver(p)
    for s in (a, b):
        s.set_data(p.Q0)
        assert np.array_equal(s.get_data(), p.Q0.astype(np.float32))
    for i in range(3):
        a.rk_stage(-0.3, 0.5, p.dt)
        b.rk_stage(-0.3, 0.5, p.dt)
        a.get_data(), a.get_residual()
    assert np.array_equal(a.get_data(), b.get_data())
    assert np.array_equal(a.get_residual(), b.get_residual())


@pytest.mark.parametrize("N,n", [(3, 8), (5, 6)])
def test_pressure_and_velocity_of_different_size(cuda, N, n):
    """Pressure 2^24 times the velocity (p ~ c u in the caller's units) and the
    other way round, both continuous, the pressure zero on the wall: each field's
    right-hand side on the curved elements is as far from 64 bits as with equal
    sizes, since every field has its own power-of-two scale (half as much again
    is left for the sums of both in the fluxes)."""
    from curved import CurvedOracle
    p = problem(N, n, "default")
    a = p.desc_arrays()
    kc = np.asarray(a["KlistCurved"])
    x, y, z = (np.asarray(p.mesh[c], np.float64).reshape(p.K, p.Np) for c in "xyz")
    Q0 = np.stack([(1 - x * x - y * y - z * z) * np.cos(x + 2 * y - z), np.sin(2 * x + y),
                   np.cos(y - z), np.sin(z + x * y)], 1)
    err = []
    for kp, ku in ((0, 0), (24, 0), (0, 24)):
        Q = Q0 * np.array([2.0 ** kp] + 3 * [2.0 ** ku])[:, None]
        Q = np.ascontiguousarray(Q, np.float32).ravel()
        s = CurvedSolver(p)
        s.set_data(Q)
        s.rk_stage(0.0, 0.0, p.dt)
        res = s.get_residual().reshape(p.K, 4, p.Np)
        s.close()
        _, ref = CurvedOracle(N, p.K, p.Nq, p.Nfq, a).run(Q, p.dt, 1)
        ref = np.asarray(ref).reshape(p.K, 4, p.Np)
        err.append([rel_l2(res[kc, c], ref[kc, c]) for c in range(4)])
    assert (np.array(err[1:]) <= 1.5 * np.array(err[0])).all(), err


@pytest.mark.parametrize("N,n", [(2, 10), (4, 6), (4, 8)])
def test_planar_and_curved_forms_beside_each_other(cuda, N, n):
    """Thread-per-output curved kernel beside the CTA-wide planar stage (N = 2, ball 10:
    3840 planar elements of 6000; N = 4, ball 6) and matrix form beside the group
    form (N = 4, ball 8)."""
    from curved import CurvedOracle
    p = problem(N, n, "table" if N >= 3 else "default")
    rng = np.random.default_rng(N + n)
    Q = (p.Q0 + 0.05 * rng.standard_normal(p.Q0.size)).astype(np.float32)
    s = CurvedSolver(p)
    s.set_data(Q)
    s.steps(p.dt, 1)
    got = s.get_data()
    s.close()
    ref, _ = CurvedOracle(N, p.K, p.Nq, p.Nfq, p.desc_arrays()).run(Q, p.dt, 5)
    assert rel_l2(got, ref) < TOL
