"""Slab decomposition of a mesh whose stage runs on the matrix units while its
parts, by their own size, would not: the owned elements must equal the
single-context run bit for bit (bbw_set_whole_mesh)."""
import numpy as np
import pytest

from bbwadg_b200 import RK4A, RK4B, WaveSolver, make_problem
from bbwadg_b200._lib import BBWError
from bbwadg_b200.decomp import LocalExchange, local_solver, local_state, run_decomposed, slab_partition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,shots,overlap", [(1, 1, False), (2, 1, True), (3, 1, False), (3, 2, True)])
def test_parts_of_a_large_mesh_equal_one_context(cuda, N, shots, overlap):
    """6000 elements (375 tiles, above the two per SM from which N <= 3 takes the
    matrix units)
    in three parts of 2000 and their halos; with two shots 3072 in three of 1024."""
    p = make_problem(N, 10 if shots == 1 else 8, c2="sine", c2_jitter=0.5, seed=N)
    rng = np.random.default_rng(N)
    Q0 = rng.standard_normal((shots, p.K, 4 * p.Np)).astype(np.float32)
    ref = WaveSolver(p)
    ref.set_shots(shots)
    ref.set_data(Q0)
    for i in range(5):
        ref.rk_stage(np.float32(RK4A[i]), np.float32(RK4B[i]), p.dt, 0.0)
    full = ref.get_data().reshape(shots, p.K, -1)
    ref.close()
    parts = slab_partition(p, 3, interface_first=overlap)
    solvers = []
    for part in parts:
        s = local_solver(p, part)
        s.set_shots(shots)
        s.set_data(np.stack([local_state(p, part, q) for q in Q0]))
        solvers.append(s)
    run_decomposed(solvers, LocalExchange(parts, solvers), p.dt, 1, overlap=overlap)
    for part, s in zip(parts, solvers):
        q = s.get_data().reshape(shots, part.K, -1)[:, :part.Kc]
        assert np.array_equal(q, full[:, part.owned])
        s.close()


def test_whole_mesh_size_is_validated(cuda):
    s = WaveSolver(make_problem(2, 1))
    with pytest.raises(BBWError):
        s.set_whole_mesh(0)
    s.close()
