"""The band sweep on rows staged wider than the grid (12 to 96 columns of a
colour, padded to 16, 24, 48, 64, 96 or 128), on full shared stencils, and for
odd counts of sweeps: FP32 cycles inside a mixed solve against the colour and
plane kernels (STZ_MG_BAND=0), bit for bit."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elastic", [True, False])
@pytest.mark.parametrize("dims,cycle", [((24, 32, 18), (2, 3, True)), ((48, 24, 17), (1, 2, False)),
                                        ((40, 48, 9), (2, 2, True)), ((96, 48, 20), (3, 1, False)),
                                        ((112, 64, 9), (2, 2, False)), ((160, 64, 9), (2, 3, False)),
                                        ((192, 96, 11), (1, 1, True)), ((248, 16, 5), (2, 1, False))])
def test_band_widths(dims, cycle, elastic, monkeypatch):
    import stzpp_gb300 as sg
    m, n, o = dims
    per = (True, True, False)
    h = (1.0 / m,) * 3
    st, fix = sg.elastic_stencil(1.0, 2.0, *h)
    if not elastic:   # full blocks: a shear mixes the components
        T = np.eye(3) + 0.1 * np.random.default_rng(2).standard_normal((3, 3))
        st = np.einsum("ab,kbc,dc->kad", T, st.reshape(27, 3, 3), T).reshape(27, 9)
        fix = (T @ fix.reshape(3, 3) @ T.T).reshape(9)
    b = P.rhs_divergence(P.random_strain(4, m, n, o, per), m, n, o, per, *h)
    v_down, v_up, growth = cycle
    out = {}
    for band in ("0", "1"):
        monkeypatch.setenv("STZ_MG_BAND", band)
        with sg.Multigrid(dims, per, precision="mixed", v_down=v_down, v_up=v_up, sweep_growth=growth) as mg:
            mg.setup_matrices(st, fix)
            assert (mg.sweep_kind(0)[0] == "band") == (band == "1")
            mg.setup_fields(r=b)
            out[band] = mg.solve(1e-10, 7, check=False) + (mg.get_x(),)
    assert np.isfinite(out["0"][1]) and out["0"][1] < 0.1
    assert out["0"][:2] == out["1"][:2]
    assert np.array_equal(out["0"][2], out["1"][2])
