"""Levels with per-node rows (csrc/dense.cu): the two-launch sweep against the
eight colour launches, bit for bit, and the residual against the rows applied
in numpy, at sizes about the kernels' groups of 32 nodes and clusters of 1, 2,
4 and 8 CTAs, odd and even extents, every kind of wrap."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu

CASES = [((8, 8, 5), (True, True, False)), ((16, 16, 9), (True, True, False)),
         ((10, 14, 6), (True, True, True)), ((13, 11, 7), (False, False, False)), ((33, 17, 4), (False, False, False)),
         ((66, 34, 5), (True, False, False)), ((2, 4, 3), (True, True, False)), ((5, 32, 8), (False, True, True)),
         ((36, 30, 3), (True, True, False))]


def handle(dims, per, precision="fp64", seed=3):
    import stzpp_gb300 as sg
    m, n, o = dims
    mu = P.lognormal_mu(seed, m, n, o)
    h = P.grid_spacing(m, n, o, per, h=1.0 / 16)
    A = P.elastic_stencil_points(mu, 2 * mu, *h, per)
    mg = sg.Multigrid(dims, per, precision=precision, max_coarse=1 << 20, bottom="gs")
    mg.setup_matrices(points=A)
    return mg, A


def fields(dims, seed):
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    return rng.standard_normal((n, 3)), rng.standard_normal((n, 3))


@pytest.mark.parametrize("dims,per", CASES)
def test_dense_sweep_is_the_colour_launches(dims, per):
    mg, _ = handle(dims, per)
    x, r = fields(dims, 5)
    out = []
    for whole in (True, False):
        mg.set_x(x)
        mg.set_rhs(r)
        for _ in range(3):
            if whole:
                mg.gauss_seidel(0, 1)
            else:
                mg.gauss_seidel_colours(0, 0, 8)
        out.append(mg.get_x())
    assert np.array_equal(out[0], out[1])
    assert mg.sweep_kind(0) == ("phase", 2)


@pytest.mark.parametrize("dims,per", CASES)
def test_dense_residual(dims, per):
    mg, A = handle(dims, per)
    x, r = fields(dims, 6)
    mg.set_x(x)
    mg.set_rhs(r)
    m, n, o = dims
    A = np.asarray(A).reshape(o, n, m, 27, 3, 3)
    X = x.reshape(o, n, m, 3)
    ref, size = r.reshape(o, n, m, 3).copy(), np.abs(r.reshape(o, n, m, 3))
    for b in range(27):
        nb = np.roll(X, (-(b // 9 - 1), -((b // 3) % 3 - 1), -(b % 3 - 1)), (0, 1, 2))
        ref -= np.einsum("kjirc,kjic->kjir", A[..., b, :, :], nb)
        size += np.einsum("kjirc,kjic->kjir", np.abs(A[..., b, :, :]), np.abs(nb))
    got, sq = mg.residual(0)
    # 81 products and 82 additions, each rounded once on either side
    assert (np.abs(got.reshape(ref.shape) - ref) <= 2 * 84 * 2.0 ** -53 * size).all()
    total = float((got ** 2).sum())
    assert abs(sq - total) <= 1e-13 * total


@pytest.mark.parametrize("dims", [(12, 10, 1), (34, 18, 1)])
def test_single_periodic_plane(dims):
    """The planes above and below a single periodic plane are itself: a colour
    pass reads what the one before wrote there.  Against the same order of
    updates in numpy."""
    per = (True, True, True)
    mg, A = handle(dims, per)
    x, r = fields(dims, 9)
    mg.set_x(x)
    mg.set_rhs(r)
    mg.gauss_seidel(0, 2)
    m, n, o = dims
    A = np.asarray(A).reshape(n, m, 27, 3, 3)
    X, R = x.reshape(n, m, 3).copy(), r.reshape(n, m, 3)
    for q in 2 * [(0, 0), (1, 0), (0, 1), (1, 1)]:
        for j in range(q[1], n, 2):
            for i in range(q[0], m, 2):
                s = R[j, i] - sum(A[j, i, b] @ X[(j + b // 3 % 3 - 1) % n, (i + b % 3 - 1) % m]
                                  for b in range(27) if b != 13)
                X[j, i] = np.linalg.solve(A[j, i, 13], s)
    assert np.abs(mg.get_x().reshape(X.shape) - X).max() <= 1e-12 * np.abs(X).max()
    assert mg.sweep_kind(0) == ("colour", 8)
