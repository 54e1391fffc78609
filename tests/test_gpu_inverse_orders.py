"""The bottom level's plain inverse (csrc/inverse.cu) beyond the wide panels."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu


def test_panels_of_sixteen_columns():
    """An order above 6400, where a panel is 16 columns wide."""
    import stzpp_gb300 as sg
    dims, per = (13, 13, 13), (False, False, False)
    m, n, o = dims
    h = P.grid_spacing(m, n, o, per, h=1.0 / 8)
    A = np.array(P.elastic_stencil_points(np.ones((o, n, m)), 2 * np.ones((o, n, m)), *h, per)).reshape(o, n, m, 27, 3, 3)
    A[..., 13, :, :] += A[..., 13, :, :] * np.eye(3)   # the condition is below 100
    b = np.random.default_rng(6).standard_normal((o, n, m, 3))
    with sg.Multigrid(dims, per, precision="fp64", max_coarse=4096, bottom="direct") as mg:
        mg.setup_matrices(points=A.reshape(-1, 27, 9))
        mg.setup_fields(r=b.reshape(-1, 3))
        mg.v_cycle()
        x = mg.get_x().reshape(o, n, m, 3)
    res, pad = b.copy(), np.pad(x, ((1, 1),) * 3 + ((0, 0),))
    for d in range(27):
        i, j, k = d % 3, d // 3 % 3, d // 9
        res -= np.einsum("kjirc,kjic->kjir", A[..., d, :, :], pad[k:k + o, j:j + n, i:i + m])
    # |b - A x| <= |A| |x - A^-1 b|, the forward error as above
    assert np.linalg.norm(res) <= 64 * 3 * m * n * o * 2.0 ** -53 * 100 * np.linalg.norm(b)
