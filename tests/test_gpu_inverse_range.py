"""The bottom level's inverse (csrc/inverse.cu) at magnitudes far from one, and
at pivots whose reciprocal lies next to the middle between two doubles."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fourier", ["0", "1"])
@pytest.mark.parametrize("power", [0, 300, 560, -560])
def test_components_of_far_apart_magnitudes(power, fourier, monkeypatch):
    """Three uncoupled components with their equations in units 2^power apart:
    the scaling is exact, so the solution is that of equal units up to the
    rounding of the inverse (64 n eps cond, the shift bounds cond by 100).
    The squares of the outer components' entries are out of range at 560."""
    import stzpp_gb300 as sg
    dims, per = (8, 8, 10), (True, True, False)
    m, n, o = dims
    st, fix = sg.elastic_stencil(1.0, -1.0, *P.grid_spacing(m, n, o, per, h=1.0 / 8))   # lam = -mu: no coupling
    st, fix = np.array(st).reshape(27, 3, 3), np.array(fix).reshape(3, 3)
    st[13] += np.diag(np.diag(st[13]))
    st *= np.eye(3)
    unit = 2.0 ** np.array([-power, 0, power])
    b = np.random.default_rng(2).standard_normal((m * n * o, 3))
    monkeypatch.setenv("STZ_MG_BOTTOM_FOURIER", fourier)
    x = []
    for u in (np.ones(3), unit):
        with sg.Multigrid(dims, per, precision="fp64", max_coarse=m * n * o // 3, bottom="direct") as mg:
            mg.setup_matrices(stencil=(st * u[:, None]).reshape(27, 9), fix=(fix * u[:, None]).reshape(9))
            mg.setup_fields(r=b * u)
            mg.v_cycle()
            assert mg.nlevels == 2
            x.append(mg.get_x())
    assert np.isfinite(x[1]).all() and np.abs(x[0]).max() > 0
    order = 3 * 4 * 4 * 6
    assert np.linalg.norm(x[1] - x[0]) <= 64 * order * 2.0 ** -53 * 100 * np.linalg.norm(x[0])


def test_pivots_are_divided_by():
    """A diagonal matrix: its inverse holds the correctly rounded reciprocals.
    Significands V with V M = 2^106 + d, M odd and |d| small, have theirs
    next to the middle between two doubles."""
    import stzpp_gb300 as sg
    hard = [7857326865746386, 7943203006394820, 8042426583074580, 8413745725510706, 8480179861092514, 8704734016499148,
            8716460134775102, 8974540322080660, 9002296740580796, 9007199254740991, 2 ** 52 + 1, 2 ** 53 - 3]
    dims = (6, 7, 8)
    rng = np.random.default_rng(5)
    v = 2.0 ** rng.uniform(-120, 120, (336, 3)) * rng.choice([-1.0, 1.0], (336, 3))
    v.reshape(-1)[:12 * 40] = (np.ldexp(np.array(hard, float)[None], -52 + rng.integers(-110, 110, 40)[:, None])).reshape(-1)
    A = np.zeros((336, 27, 3, 3))
    A[:, 13] = v[:, :, None] * np.eye(3)
    with sg.Multigrid(dims, (False, False, False), precision="fp64", max_coarse=4096, bottom="direct") as mg:
        mg.setup_matrices(points=A.reshape(336, 27, 9))
        mg.setup_fields(r=np.ones((336, 3)))
        mg.v_cycle()
        x = mg.get_x()
    assert np.array_equal(x, 1.0 / v)
