"""The advection step on fields of few distinct values, zeros of both signs
among them, so that differences, quotients and sums cancel to zeros of either
sign everywhere: the results are those of the reference's separately rounded
operations down to the sign of a zero."""
import numpy as np
import pytest

from oracle import advect as A
from test_gpu_advect import ADV_OUT, gpu_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("dims", [(16, 12, 9), (33, 8, 5)])
def test_signs_of_zeros(dims, seed):
    rng = np.random.default_rng(seed)
    prm = A.driver_params(dims[0])
    F = A.random_fields(22, *dims, sigma_scale=0.05)
    n = len(F)
    for c in (A.U, A.V, A.W):
        F[:, c] = rng.choice([0.0, -0.0], n) if seed % 2 else rng.choice([0.0, -0.0, 1e-3, -1e-3], n)
    for c in A.STRESS:
        F[:, c] = rng.choice([0.0, -0.0, 0.0, 0.125, -0.125, 0.25, 0.5], n) * 0.25
    F[:, A.CHI] = rng.choice([0.0, -0.0, 0.25, 0.5, 1.0], n)
    for c in A.DSTRESS + [A.CCHI]:
        F[:, c] = rng.choice([0.0, -0.0], n)
    F[:, A.ADPL] = rng.choice([0.0, -0.0, 0.25], n)
    P, py = A.port_step(F, *dims, prm, 300.0)
    G, gy = gpu_step(F, dims, prm, 300.0)
    assert not gy and not py
    assert (P[:, ADV_OUT] == 0).any()
    G, P = (np.ascontiguousarray(a).view(np.int64) for a in (G, P))
    assert not [c for c in ADV_OUT if not np.array_equal(G[:, c], P[:, c])]
