"""FP32 sweeps and residuals of levels with per-node rows (csrc/dense.cu) inside
mixed solves, against the clustered tail, which runs dense_row node by node."""
import pytest

from oracle import problem as P
from test_gpu_fp32_levels import solves

pytestmark = pytest.mark.gpu


# level 1: one group of 32 nodes a colour and plane, two, four, and eight or more; odd sizes and every wrap
@pytest.mark.parametrize("dims,per", [((16, 16, 9), (True, True, False)), ((32, 24, 13), (True, True, False)),
                                      ((64, 32, 17), (True, True, False)), ((64, 64, 16), (True, True, True)),
                                      ((25, 21, 13), (False, False, False)), ((67, 69, 11), (False, False, False)),
                                      ((136, 34, 8), (True, False, False)), ((9, 64, 16), (False, True, True))])
@pytest.mark.parametrize("kind", ["lame", "points"])
def test_dense_levels(dims, per, kind, monkeypatch):
    m, n, o = dims
    mu = P.lognormal_mu(5, m, n, o)
    lam = 1.5 * P.lognormal_mu(6, m, n, o)
    h = (1.0 / m,) * 3

    def setup(mg):
        if kind == "lame":
            mg.setup_matrices(mu=mu.reshape(-1), lam=lam.reshape(-1), spacing=h)
        else:
            mg.setup_matrices(points=P.elastic_stencil_points(mu, lam, *h, per))

    solves(monkeypatch, dims, per, setup)
