"""Device memory of the solvers: contexts are still created where there is no
room for the matrix stages' own data, and the curved solver keeps its point data
once."""
import numpy as np
import pytest
from conftest import golden

from bbwadg_b200 import WaveSolver, make_problem
from bbwadg_b200.curved import CurvedSolver, make_curved_problem

pytestmark = pytest.mark.gpu


def rule(N):
    g = golden("ops_N%d.npz" % N)
    m = int(g["Nfq"][0])
    return dict(cubature=(g["rq"], g["sq"], g["tq"], g["wq"]),
                tri_cubature=(g["rfq"][:m], g["sfq"][:m], g["wfqFace"]))


def free():
    import gc

    import torch
    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision", ["fp32", "f16x3"])
def test_context_without_room_for_the_matrix_stages(cuda, precision):
    """N = 5, 24^3 x 6: the padded medium takes 32 MB beyond what the CTA-wide stages
    need.  With half of that missing the context is created all the same and runs
    those, bit for bit as when they are pinned.  (In a long process the driver may
    hold back enough from contexts that were closed for the medium to fit; then
    the context runs its default form.)"""
    import torch
    p = make_problem(5, 24, c2="sine", c2_jitter=0.5, seed=1, **rule(5))
    extra = p.K * ((p.Nq + 15) // 16 * 16 + 1) * 4
    out = []
    for config in (None, (8, True, False)):
        a = free()
        s = WaveSolver(p, precision=precision)
        used = a - free()
        if config:
            s.set_config(*config)
        s.set_data(p.Q0)
        s.steps(p.dt, 1)
        out.append(s.get_data())
        s.close()
    fill = torch.empty(free() - (used - extra // 2), dtype=torch.uint8, device=cuda)
    try:
        s = WaveSolver(p, precision=precision)
        del fill
        torch.cuda.empty_cache()
        s.set_data(p.Q0)
        s.steps(p.dt, 1)
        got = s.get_data()
        s.set_c2q(p.c2q)
        s.close()
    finally:
        fill = None
        torch.cuda.empty_cache()
    assert np.array_equal(got, out[1]) or np.array_equal(got, out[0])


def test_curved_point_data_is_kept_once(cuda):
    """N = 5, ball 10: 2160 of 6000 elements curved.  State, next state and residual,
    the planar context's arrays and one copy of the point data, with a
    quarter for padding to 16 points and 16 elements and the allocator's blocks."""
    p = make_curved_problem(5, 10, **rule(5))
    a = p.desc_arrays()
    kc, Nfp = len(a["KlistCurved"]), 21
    point = 4 * kc * (10 * p.Nq + 16 * p.Nfq + 2 * p.Nq)
    whole = 4 * p.K * (3 * 4 * p.Np + 25 + 28 + 4 + 4 * Nfp + 2 * p.Nq + 16)
    before = free()
    s = CurvedSolver(p)
    used = before - free()
    s.steps(p.dt, 1)
    s.close()
    assert used < 1.25 * (point + whole) + (4 << 20), (used, point, whole)
