"""The FP32 sweeps of the small levels inside mixed solves against the
clustered tail (STZ_MG_TAIL=1), which runs the colours' own row functions
(csrc/ops.cuh) node by node: the same cycles and solutions, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solves(monkeypatch, dims, per, setup, component=None):
    import stzpp_gb300 as sg
    m, n, o = dims
    b = np.random.default_rng(3).standard_normal((m * n * o, 3)) * 1e-3
    if component is not None:
        b *= np.eye(3)[component]
    monkeypatch.setenv("STZ_MG_BAND", "0")
    out = []
    for tail in (False, True):
        if tail:
            monkeypatch.setenv("STZ_MG_TAIL", "1")
        else:
            monkeypatch.delenv("STZ_MG_TAIL", raising=False)
        with sg.Multigrid(dims, per, precision="mixed", v_down=2, v_up=3, sweep_growth=False, max_coarse=24,
                          bottom="gs") as mg:
            setup(mg)
            assert mg.nlevels > 2
            if not tail:   # the sweeps under test are those of dense.cu and plane.cu
                assert all(mg.sweep_kind(l) == ("phase", 2) for l in range(1, mg.nlevels - 1))
            mg.setup_fields(r=b)
            out.append(mg.solve(1e-10, 4, check=False) + (mg.get_x(),))
    assert np.isfinite(out[0][1])
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("mu,lam,spacing", [(1.0, 2.0, (1.0, 1.0, 1.0)), (0.7, 1.3, (0.3, 0.3, 0.3)),
                                            (1.1, 0.9, (0.1, 0.13, 0.17)), (0.37, 2.9, (0.013, 0.017, 0.011))])
@pytest.mark.parametrize("dims", [(32, 24, 17), (48, 56, 26), (40, 24, 9)])
def test_plane_levels(dims, mu, lam, spacing, monkeypatch):
    """Moduli and spacings that leave cancellation round-off in the Galerkin
    rows' structural zeros: FP32 kernels skip those, whichever kernel runs."""
    import stzpp_gb300 as sg
    solves(monkeypatch, dims, (True, True, False),
           lambda mg: mg.setup_matrices(*sg.elastic_stencil(mu, lam, *spacing)))


@pytest.mark.parametrize("dims", [(32, 24, 16), (48, 56, 24)])
def test_plane_levels_with_entries_below_the_threshold(dims, monkeypatch):
    """Entries outside the structure of up to 1e-9 of a plane's largest: FP32
    kernels skip them, and on every path (without plates, whose own planes
    have larger ones).  They are all that couples the components here, and one
    component alone is driven: the others show which entries were taken."""
    import stzpp_gb300 as sg
    h = (1.0 / dims[0],) * 3
    st, fix = sg.elastic_stencil(1.0, -1.0, *h)   # lam = -mu: no coupling
    st = np.array(st).reshape(27, 3, 3)
    st[13] += np.diag(np.diag(st[13]))
    for b in (4, 10, 12, 14, 16, 22):   # the face blocks, which are diagonal
        st[b] += 2e-10 * np.abs(st[b]).max() * (1 - np.eye(3))
    outside = np.array([[r != c and not (d[r] and d[c]) for r in range(3) for c in range(3)] for b in range(27)
                        for d in [(b % 3 - 1, b // 3 % 3 - 1, b // 9 - 1)]])

    def setup(mg):
        mg.setup_matrices(st.reshape(27, 9), fix)
        for l in range(1, mg.nlevels):
            m, n, o = mg.level_dims(l)
            A = np.abs(mg.level_operator(l)[0].reshape(o, n * m, 27, 9)[:, 0])
            share = (A * outside).max((1, 2)) / A.max((1, 2))
            assert 0 < share.max() <= 1e-9

    solves(monkeypatch, dims, (True, True, True), setup, component=1)
