"""Matrix forms of rk_volume, rk_surface and rk_update_WADG at the smallest
meshes that take them and with a ragged last tile, against the C
restatement, and the scalar forms for pointers that are not 16-byte aligned.
Tolerance: 1e-5 relative L2 (FP32), as for the other kernel-level tests."""
import numpy as np
import pytest
from conftest import golden, rel_l2

from bbwadg_b200 import _lib, make_problem

pytestmark = pytest.mark.gpu
TOL = 1e-5


def problem(N, n):
    g = golden("ops_N%d.npz" % N) if N >= 3 else None
    kw = {}
    if g is not None:
        m = int(g["Nfq"][0])
        kw = dict(cubature=(g["rq"], g["sq"], g["tq"], g["wq"]),
                  tri_cubature=(g["rfq"][:m], g["sfq"][:m], g["wfqFace"]))
    return make_problem(N, n, c2="sine", c2_jitter=0.5, seed=N, **kw)


def run(p, bc, Q, rhs0, res0, Jq, offset=0):
    """The three kernels on seeded inputs; every vector starts `offset` floats
    past an aligned address."""
    import torch

    def dev(a):
        a = np.ascontiguousarray(a)
        t = torch.zeros(a.size + 4, dtype=torch.int32 if a.dtype == np.int32 else torch.float32,
                        device="cuda")
        t[offset:offset + a.size] = torch.from_numpy(a.ravel()).cuda()
        return t[offset:offset + a.size]

    o, g = p.ops_dict(), p.geo_dict()
    a = {k: dev(o[k]) for k in ("Dr", "Ds", "Dt", "LIFT", "Vq", "Pq", "Fmask")}
    a.update({k: dev(g[k]) for k in ("vgeo", "fgeo", "vmapP", "c2q")})
    a.update(Jq=dev(Jq), Q=dev(Q), rhs=dev(np.zeros_like(Q)), sur=dev(rhs0), res=dev(res0), Qn=dev(Q))
    P = {k: t.data_ptr() for k, t in a.items()}
    _lib.call("bbw_rk_volume", p.N, p.K, P["vgeo"], P["Dr"], P["Ds"], P["Dt"], P["Q"], P["rhs"], None)
    _lib.call("bbw_rk_surface", p.N, p.K, bc, P["fgeo"], P["Fmask"], P["vmapP"], P["LIFT"], P["Q"],
              P["sur"], None)
    _lib.call("bbw_rk_update_wadg", p.N, p.K, p.Nq, P["Vq"], P["Pq"], P["Jq"], P["c2q"], -0.4, 0.3,
              0.01, P["sur"], P["res"], P["Qn"], None)
    torch.cuda.synchronize()
    return [a[k].cpu().numpy() for k in ("rhs", "sur", "res", "Qn")]


# one element below a multiple of 16 never occurs on these meshes (K = 6 n^3):
# n = 7 and 15 leave 10 of 16 rows in the last tile
@pytest.mark.parametrize("N,n", [(2, 15), (3, 11), (3, 15), (4, 7), (5, 7), (6, 9), (7, 7)])
@pytest.mark.parametrize("bc", [0, 1])
def test_matrix_kernels_match_restatement(cuda, N, n, bc):
    from oracle import Oracle
    p = problem(N, n)
    rng = np.random.default_rng(N)
    Q, rhs0, res0 = (rng.standard_normal(p.K * 4 * p.Np).astype(np.float32) for _ in range(3))
    Jq = (0.5 + rng.random(p.K * p.Nq)).astype(np.float32)
    vol, sur, res, Qn = run(p, bc, Q, rhs0, res0, Jq)
    geo = dict(p.geo_dict(), Jq=Jq)
    orc = Oracle(N, p.K, p.ops_dict(), geo, variant="nodal", bc=bc)
    r = np.zeros_like(Q)
    orc.rk_volume(Q, r)
    assert rel_l2(vol, r) < TOL
    s = rhs0.copy()
    orc.rk_surface(Q, s)
    assert rel_l2(sur, s) < TOL
    q, rr = Q.copy(), res0.copy()
    orc.rk_update_wadg(-0.4, 0.3, 0.01, s, rr, q)
    assert rel_l2(res, rr) < TOL
    assert rel_l2(Qn, q) < TOL


@pytest.mark.parametrize("N,n", [(4, 7), (5, 7)])
def test_unaligned_pointers_take_the_scalar_forms(cuda, N, n):
    p = problem(N, n)
    rng = np.random.default_rng(N)
    Q, rhs0, res0 = (rng.standard_normal(p.K * 4 * p.Np).astype(np.float32) for _ in range(3))
    Jq = np.ones(p.K * p.Nq, np.float32)
    for x, y in zip(run(p, 0, Q, rhs0, res0, Jq), run(p, 0, Q, rhs0, res0, Jq, offset=1)):
        assert rel_l2(x, y) < TOL
