"""FP64 plane-invariant levels (csrc/plane.cu): the two-launch sweep against
the eight colour launches, bit for bit, and the residual against the level's
own rows applied in numpy, at sizes about the 10 nodes of a warp and the 4 to
128 warps of a plane, sparse (elastic) and full rows."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu

CASES = [((16, 16, 17), True, 1), ((40, 24, 9), True, 1), ((8, 4, 6), False, 1), ((48, 80, 7), True, 1),
         ((64, 16, 10), False, 1), ((160, 96, 8), True, 1), ((96, 96, 9), False, 2), ((200, 136, 5), True, 1)]


def handle(dims, elastic):
    import stzpp_gb300 as sg
    m, n, o = dims
    per = (True, True, False)
    h = P.grid_spacing(m, n, o, per)
    st, fix = sg.elastic_stencil(1.0, 2.0, *h)
    if not elastic:   # full blocks: a shear mixes the components
        T = np.eye(3) + 0.1 * np.random.default_rng(2).standard_normal((3, 3))
        st = np.einsum("ab,kbc,dc->kad", T, st.reshape(27, 3, 3), T).reshape(27, 9)
        fix = (T @ fix.reshape(3, 3) @ T.T).reshape(9)
    mg = sg.Multigrid(dims, per, precision="fp64", max_coarse=16, bottom="gs")
    mg.setup_matrices(st, fix)
    return mg


@pytest.mark.parametrize("dims,elastic,level", CASES)
def test_plane_sweep_is_the_colour_launches(dims, elastic, level):
    mg = handle(dims, elastic)
    rng = np.random.default_rng(7)
    N = mg.level_npts(level)
    x, r = rng.standard_normal((N, 3)), rng.standard_normal((N, 3))
    out = []
    for whole in (True, False):
        mg.level_set_field(level, "x", x)
        mg.level_set_field(level, "r", r)
        for _ in range(2):
            if whole:
                mg.gauss_seidel(level, 1)
            else:
                mg.gauss_seidel_colours(level, 0, 8)
        out.append(mg.level_get_field(level, "x"))
    assert np.array_equal(out[0], out[1])
    assert mg.sweep_kind(level) == ("phase", 2)


@pytest.mark.parametrize("dims,elastic,level", CASES)
def test_plane_residual(dims, elastic, level):
    mg = handle(dims, elastic)
    rng = np.random.default_rng(8)
    N = mg.level_npts(level)
    x, r = rng.standard_normal((N, 3)), rng.standard_normal((N, 3))
    mg.level_set_field(level, "x", x)
    mg.level_set_field(level, "r", r)
    # the restriction forms the level's residual without a norm
    mg.restriction(level + 1)
    got = mg.level_get_field(level, "res")
    m, n, o = mg.level_dims(level)
    A, _ = mg.level_operator(level)
    A, X = A.reshape(o, n, m, 27, 3, 3), x.reshape(o, n, m, 3)
    ref, size = r.reshape(o, n, m, 3).copy(), np.abs(r.reshape(o, n, m, 3))
    for b in range(27):
        nb = np.roll(X, (-(b // 9 - 1), -((b // 3) % 3 - 1), -(b % 3 - 1)), (0, 1, 2))
        ref -= np.einsum("kjirc,kjic->kjir", A[..., b, :, :], nb)
        size += np.einsum("kjirc,kjic->kjir", np.abs(A[..., b, :, :]), np.abs(nb))
    # 81 products and 82 additions, each rounded once on either side
    assert (np.abs(got.reshape(ref.shape) - ref) <= 2 * 84 * 2.0 ** -53 * size).all()


def test_single_periodic_plane():
    """A level of one periodic plane, whose planes above and below are itself,
    sweeps by the colour launches."""
    import stzpp_gb300 as sg
    dims, per = (24, 20, 2), (True, True, True)
    st, fix = sg.elastic_stencil(1.0, 2.0, *P.grid_spacing(*dims, per, h=1.0 / 8))
    st = np.array(st).reshape(27, 3, 3)
    st[13] += np.diag(np.diag(st[13]))
    mg = sg.Multigrid(dims, per, precision="fp64", max_coarse=200, bottom="gs")
    mg.setup_matrices(st.reshape(27, 9), fix)
    assert tuple(mg.level_dims(1)) == (12, 10, 1)
    rng = np.random.default_rng(7)
    x, r = rng.standard_normal((120, 3)), rng.standard_normal((120, 3))
    out = []
    for whole in (True, False):
        mg.level_set_field(1, "x", x)
        mg.level_set_field(1, "r", r)
        if whole:
            mg.gauss_seidel(1, 2)
        else:
            for _ in range(2):
                mg.gauss_seidel_colours(1, 0, 8)
        out.append(mg.level_get_field(1, "x"))
    assert np.array_equal(out[0], out[1])
    assert mg.sweep_kind(1) == ("colour", 8)
