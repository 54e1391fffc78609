"""The band sweep of FP32 Lame levels against the colour and plane kernels
(STZ_MG_BAND=0) inside mixed solves, at every staged width, bit for bit: one
row arithmetic (lame_row_of) serves both."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,per", [((16, 16, 9), (True, True, False)), ((24, 32, 8), (True, True, True)),
                                      ((32, 24, 17), (True, True, False)), ((40, 16, 10), (True, True, False)),
                                      ((64, 48, 9), (True, True, False)), ((96, 32, 6), (True, True, True)),
                                      ((128, 32, 9), (True, True, False)), ((160, 48, 5), (True, True, False)),
                                      ((256, 32, 7), (True, True, False))])
def test_lame_band(dims, per, monkeypatch):
    import stzpp_gb300 as sg
    m, n, o = dims
    h = (1.0 / m,) * 3
    mu = P.lognormal_mu(5, m, n, o).reshape(-1)
    lam = 1.5 * P.lognormal_mu(6, m, n, o).reshape(-1)
    b = np.random.default_rng(3).standard_normal((m * n * o, 3)) * 1e-3
    b -= b.mean(0)
    out = {}
    for band in ("0", "1"):
        monkeypatch.setenv("STZ_MG_BAND", band)
        with sg.Multigrid(dims, per, precision="mixed", v_down=2, v_up=3, sweep_growth=False, bottom="gs") as mg:
            mg.setup_matrices(mu=mu, lam=lam, spacing=h)
            assert (mg.sweep_kind(0)[0] == "band") == (band == "1")
            mg.setup_fields(r=b)
            out[band] = mg.solve(1e-10, 4, check=False) + (mg.get_x(),)
    assert np.isfinite(out["0"][1])
    assert out["0"][:2] == out["1"][:2]
    assert np.array_equal(out["0"][2], out["1"][2])
