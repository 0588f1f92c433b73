"""The stages on warp-level matrix instructions (one warp, or a group of warps,
per 16-element tile), pinned by their configuration codes, against the C
restatement and against each other.  Tolerance against the restatement:
1e-5 relative L2, the FP32 bar of the other stages."""
import numpy as np
import pytest
from conftest import golden, rel_l2

from bbwadg_b200 import WaveSolver, _lib, make_problem
from bbwadg_b200._lib import BBWError

pytestmark = pytest.mark.gpu
TOL = 1e-5
SINGLE = 8 | 1 << 8 | 1 << 10 | 1 << 11
GROUP = 8 | 1 << 8 | 1 << 10 | 1 << 12


def problem(N, n, variant="nodal", rule="table"):
    kw = {}
    if rule == "table" and N >= 3:
        g = golden("ops_N%d.npz" % N)
        m = int(g["Nfq"][0])
        kw = dict(cubature=(g["rq"], g["sq"], g["tq"], g["wq"]),
                  tri_cubature=(g["rfq"][:m], g["sfq"][:m], g["wfqFace"]))
    return make_problem(N, n, variant=variant, c2="sine", c2_jitter=0.5, seed=N, **kw)


def run(p, code, Q, steps=2, bc="pressure_release", limit=0):
    s = WaveSolver(p, bc=bc)
    _lib.call("bbw_set_config", s._h, code)
    s.set_grid_limit(limit)
    s.set_data(Q)
    s.steps(p.dt, steps)
    out = s.get_data(), s.get_residual()
    s.close()
    return out


FORMS = [(N, SINGLE) for N in (1, 2, 3, 4)] + [(N, GROUP) for N in (4, 5, 6, 7)]


@pytest.mark.parametrize("N,code", FORMS)
@pytest.mark.parametrize("variant,bc", [("nodal", "pressure_release"), ("nodal", "rigid"),
                                        ("bb", "pressure_release")])
def test_forms_match_restatement(cuda, N, code, variant, bc):
    """3^3 x 6 tets: ten full tiles and a ragged one of two elements; on the
    full grid and on one CTA that walks all of them."""
    from oracle import Oracle
    p = problem(N, 3, variant)
    rng = np.random.default_rng(N)
    Q = (p.Q0 + 0.1 * rng.standard_normal(p.Q0.size)).astype(np.float32)
    ref, _ = Oracle(N, p.K, p.ops_dict(), p.geo_dict(), variant=variant,
                    bc=1 if bc == "rigid" else 0).run(Q.copy(), p.dt, 10)
    a, ra = run(p, code, Q, bc=bc)
    b, rb = run(p, code, Q, bc=bc, limit=1)
    assert rel_l2(a, ref) < TOL
    assert np.array_equal(a, b) and np.array_equal(ra, rb)


@pytest.mark.parametrize("rule", ["table", "default"])
def test_single_warp_and_group_agree_bit_for_bit(cuda, rule):
    """N = 4 has both forms; the 125-point rule leaves a ragged last chunk."""
    p = problem(4, 3, rule=rule)
    rng = np.random.default_rng(4)
    Q = rng.standard_normal(p.Q0.size).astype(np.float32)
    (a, ra), (b, rb) = run(p, SINGLE, Q), run(p, GROUP, Q)
    assert np.array_equal(a, b) and np.array_equal(ra, rb)


@pytest.mark.parametrize("N,code", [(2, SINGLE), (3, SINGLE), (4, GROUP), (5, GROUP), (7, GROUP)])
def test_power_of_two_scaling_is_exact(cuda, N, code):
    """Every operand is scaled by a power of two per element, so a state times
    2^k gives the result times 2^k, bit for bit."""
    p = problem(N, 2)
    rng = np.random.default_rng(N)
    Q = rng.standard_normal(p.Q0.size).astype(np.float32)
    a, _ = run(p, code, Q)
    for k in (-40, 60):
        b, _ = run(p, code, np.ldexp(Q, k).astype(np.float32))
        assert np.array_equal(np.ldexp(a, k).astype(np.float32), b)


@pytest.mark.parametrize("N,code", [(3, SINGLE), (4, SINGLE), (4, GROUP), (5, GROUP), (6, GROUP)])
def test_windows_equal_whole_stage(cuda, N, code):
    """Element windows that start inside a tile advance the same elements as
    one whole-mesh stage, bit for bit."""
    p = problem(N, 3)
    a, b = WaveSolver(p), WaveSolver(p)
    for s in (a, b):
        _lib.call("bbw_set_config", s._h, code)
        s.set_data(p.Q0)
    a.rk_stage(0.0, 0.5, p.dt, 0.0)
    for k0, k1 in ((0, 37), (37, 100), (100, p.K)):
        b.stage_part(0.0, 0.5, p.dt, k0, k1)
    b.stage_commit()
    assert np.array_equal(a.get_data(), b.get_data())
    assert np.array_equal(a.get_residual(), b.get_residual())


def test_forms_outside_their_orders_are_refused(cuda):
    for N, code in ((5, SINGLE), (3, GROUP), (8, SINGLE), (8, GROUP)):
        s = WaveSolver(make_problem(N, 1))
        with pytest.raises(BBWError):
            _lib.call("bbw_set_config", s._h, code)
        s.close()


@pytest.mark.parametrize("N", [5, 6])
def test_non_finite_values_stay_in_reach(cuda, N):
    """An infinity in one element reaches that element and its neighbours in
    one stage, as in the CTA-wide stage, and no other element of the tile."""
    p = problem(N, 3)
    Q = p.Q0.reshape(p.K, 4, p.Np).copy()
    Q[40, 0, 3] = np.inf
    got = []
    for code in (GROUP, 8 | 1 << 10):
        s = WaveSolver(p)
        _lib.call("bbw_set_config", s._h, code)
        s.set_data(Q.ravel())
        s.rk_stage(0.0, 0.5, p.dt, 0.0)
        got.append(np.isfinite(s.get_data().reshape(p.K, -1)).all(axis=1))
        s.close()
    reach = set(p.mesh["EToE"][40]) | {40}
    for ok in got:
        assert set(np.nonzero(~ok)[0]) <= reach
    assert not got[0][40]
