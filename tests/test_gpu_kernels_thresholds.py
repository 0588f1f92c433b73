"""rk_volume, rk_surface and rk_update_WADG on both sides of the element counts
from which they take their matrix forms, against the C restatement (1e-5
relative L2, FP32): one tile and a ragged second one, and the smallest meshes
above each count that leave a ragged last tile."""
import numpy as np
import pytest
from conftest import rel_l2
from test_gpu_kernels_matrix import TOL, problem, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [(3, 1), (4, 1), (5, 1), (2, 18), (3, 13), (5, 6), (6, 7), (7, 6),
                                 (7, 9)])
def test_both_forms_match_restatement(cuda, N, n):
    from oracle import Oracle
    p = problem(N, n)
    rng = np.random.default_rng(N + n)
    Q, rhs0, res0 = (rng.standard_normal(p.K * 4 * p.Np).astype(np.float32) for _ in range(3))
    Jq = (0.5 + rng.random(p.K * p.Nq)).astype(np.float32)
    vol, sur, res, Qn = run(p, 0, Q, rhs0, res0, Jq)
    orc = Oracle(N, p.K, p.ops_dict(), dict(p.geo_dict(), Jq=Jq), variant="nodal", bc=0)
    r, s, q, rr = np.zeros_like(Q), rhs0.copy(), Q.copy(), res0.copy()
    orc.rk_volume(Q, r)
    orc.rk_surface(Q, s)
    orc.rk_update_wadg(-0.4, 0.3, 0.01, s, rr, q)
    for got, ref in ((vol, r), (sur, s), (res, rr), (Qn, q)):
        assert rel_l2(got, ref) < TOL
