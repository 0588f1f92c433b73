"""Small meshes at N <= 3: the stage on 16-element tiles that a context takes by
itself against the pinned 32-element one, bit for bit."""
import numpy as np
import pytest

from bbwadg_b200 import WaveSolver, _lib, make_problem

pytestmark = pytest.mark.gpu
WIDE = 8 | 1 << 8  # 32-element tiles, operators in shared memory


def run(p, code, shots):
    s = WaveSolver(p)
    if shots > 1:
        s.set_shots(shots)
    if code:
        _lib.call("bbw_set_config", s._h, code)
    rng = np.random.default_rng(shots)
    Q = 0.1 * rng.standard_normal((shots, p.Q0.size)) + p.Q0.ravel()
    Q = Q.astype(np.float32)
    s.set_data(Q.reshape(p.Q0.shape) if shots == 1 else Q.reshape((shots,) + p.Q0.shape))
    s.steps(p.dt, 3)
    out = s.get_data(), s.get_residual()
    s.close()
    return out


# 162 elements: ten full 16-element tiles and one of two; 2058: 129 tiles, the
# most a cube mesh has below one per SM; three shots of 750: 141
@pytest.mark.parametrize("N", [1, 2, 3])
@pytest.mark.parametrize("variant", ["nodal", "bb"])
@pytest.mark.parametrize("n,shots", [(1, 1), (3, 1), (7, 1), (5, 3)])
def test_narrow_tiles_agree_with_wide(cuda, N, variant, n, shots):
    p = make_problem(N, n, variant=variant, c2="sine", c2_jitter=0.5, seed=N)
    a, ra = run(p, 0, shots)
    b, rb = run(p, WIDE, shots)
    assert np.array_equal(a, b) and np.array_equal(ra, rb)
