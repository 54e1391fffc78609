"""The bottom level's dense inverse (csrc/inverse.cu): x = A^-1 b of a
hierarchy that is its bottom level alone, against numpy's solve, at orders
about the panel width, the tile and the cluster's row split, with and without
wraps, and with a zero block on a diagonal that only pivoting gets past."""
import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu


def matrix(A, dims, per):
    m, n, o = dims
    N = m * n * o
    A = np.asarray(A).reshape(o, n, m, 27, 3, 3)
    M = np.zeros((N, 3, N, 3))
    for k in range(o):
        for j in range(n):
            for i in range(m):
                p = i + m * (j + n * k)
                for b in range(27):
                    q = [i + b % 3 - 1, j + (b // 3) % 3 - 1, k + b // 9 - 1]
                    if any(not w and not 0 <= c < e for c, e, w in zip(q, dims, per)):
                        continue
                    q = [c % e for c, e in zip(q, dims)]
                    M[p, :, q[0] + m * (q[1] + n * q[2])] += A[k, j, i, b]
    return M.reshape(3 * N, 3 * N)


@pytest.mark.parametrize("dims,per", [((2, 2, 3), (True, True, False)), ((4, 4, 2), (True, True, True)),
                                      ((3, 5, 7), (False, False, False)), ((11, 1, 1), (False, True, True)),
                                      ((8, 8, 9), (True, True, False)), ((13, 9, 6), (False, False, False))])
def test_bottom_inverse(dims, per):
    import stzpp_gb300 as sg
    m, n, o = dims
    mu = P.lognormal_mu(4, m, n, o)
    h = P.grid_spacing(m, n, o, per, h=1.0 / 8)
    A = np.array(P.elastic_stencil_points(mu, 2 * mu, *h, per)).reshape(-1, 27, 9)
    # a few strong couplings across components: rows whose largest entry is not on the diagonal
    rng = np.random.default_rng(1)
    for p in rng.choice(len(A), size=max(1, len(A) // 5), replace=False):
        A[p, 13] = A[p, 13].reshape(3, 3)[[1, 2, 0]].reshape(9) + 1e-3 * np.abs(A[p, 13]).max() * rng.random(9)
    M = matrix(A, dims, per)
    b = rng.standard_normal((len(A), 3))
    with sg.Multigrid(dims, per, precision="fp64", max_coarse=4096, bottom="direct") as mg:
        mg.setup_matrices(points=A)
        mg.setup_fields(r=b)
        mg.v_cycle()
        x = mg.get_x().reshape(-1)
    # the forward error of a pivoted elimination of order n: n eps cond(M), with room for its growth
    ref = np.linalg.solve(M, b.reshape(-1))
    assert np.linalg.norm(x - ref) <= 64 * len(M) * 2.0 ** -53 * np.linalg.cond(M) * np.linalg.norm(ref)


@pytest.mark.parametrize("dims,per", [((8, 8, 66), (True, True, False)), ((8, 8, 68), (True, True, False)),
                                      ((8, 8, 200), (True, True, False)), ((92, 92, 2), (True, True, True))])
def test_fourier_inverse_of_tall_columns_and_many(dims, per, monkeypatch):
    """Columns of 34 and 35 planes (systems of order 102, the last in shared
    memory, and 105, the first beyond it), of 101 planes (order 303: more
    rows than a CTA has threads), and 2116 columns of one plane: a V-cycle with
    the Fourier inverse against one with the plain inverse.  The shift bounds the bottom's condition by 100, so
    the two inverses differ by at most 64 n eps 100 of the solution."""
    import stzpp_gb300 as sg
    m, n, o = dims
    st, fix = sg.elastic_stencil(1.0, 2.0, *P.grid_spacing(m, n, o, per, h=1.0 / 8))
    st = np.array(st).reshape(27, 3, 3)
    st[13] += np.diag(np.diag(st[13]))
    b = np.random.default_rng(2).standard_normal((m * n * o, 3))
    x = []
    for fourier in ("0", "1"):
        monkeypatch.setenv("STZ_MG_BOTTOM_FOURIER", fourier)
        with sg.Multigrid(dims, per, precision="fp64", max_coarse=m * n * o // 3, bottom="direct") as mg:
            mg.setup_matrices(stencil=st.reshape(27, 9), fix=fix)
            mg.setup_fields(r=b)
            mg.v_cycle()
            assert mg.nlevels == 2
            x.append(mg.get_x())
    assert np.isfinite(x[0]).all() and np.abs(x[0]).max() > 0
    order = 3 * m * n * o // 4
    assert np.linalg.norm(x[1] - x[0]) <= 64 * order * 2.0 ** -53 * 100 * np.linalg.norm(x[0])


@pytest.mark.parametrize("fourier", ["0", "1"])
def test_box_beyond_one_node_is_refused(fourier, monkeypatch):
    """A level coarsened from a single periodic plane has boxes of more than
    one node: no direct bottom, whichever inverse would run."""
    import stzpp_gb300 as sg
    dims, per = (16, 16, 2), (True, True, True)
    st, fix = sg.elastic_stencil(1.0, 2.0, *P.grid_spacing(*dims, per, h=1.0 / 16))
    st = np.array(st).reshape(27, 3, 3)
    st[13] += np.diag(np.diag(st[13]))
    monkeypatch.setenv("STZ_MG_BOTTOM_FOURIER", fourier)
    with sg.Multigrid(dims, per, precision="fp64", max_coarse=20, bottom="direct") as mg:
        with pytest.raises(sg.StzMgError, match="beyond one node"):
            mg.setup_matrices(stencil=st.reshape(27, 9), fix=fix)
