"""The advection step at the sizes where its blocks end, against the C
restatement: consecutive cells across rows, 256 to 2048 of them a block, the
cells above the yield stress in a queue per block."""
import numpy as np
import pytest

from oracle import advect as A
from test_gpu_advect import ADV_OUT, TOL, gpu_step, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 8, 8), (33, 9, 17), (31, 7, 5), (1, 300, 1), (257, 1, 2), (160, 144, 31)])
def test_queue_of_plastic_cells(dims):
    prm = A.driver_params(dims[0])
    F = A.random_fields(21, *dims, sigma_scale=0.45)
    P, py = A.port_step(F, *dims, prm, 200.0)
    G, gy = gpu_step(F, dims, prm, 200.0)
    assert gy and py
    for c in ADV_OUT:
        assert rel_err(G[:, c], P[:, c]) <= TOL, f"member {c}: {rel_err(G[:, c], P[:, c]):.3e}"


@pytest.mark.parametrize("c0", [0.4, 1.0 / 3.0, 0.7071067811865476, 1.9999999999999998, 3.3e-7, 1e40])
def test_elastic_step_is_bitwise_for_any_divisor(c0):
    """No cell yields: the quotient of the chi diffusion by c0 is the plain division's."""
    dims = (40, 24, 11)
    prm = dict(A.driver_params(dims[0]), c0=c0)
    F = A.random_fields(22, *dims, sigma_scale=0.05)
    P, py = A.port_step(F, *dims, prm, 300.0)
    G, gy = gpu_step(F, dims, prm, 300.0)
    assert not gy and not py
    assert np.array_equal(G, P)
