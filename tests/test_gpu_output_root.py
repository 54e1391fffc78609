"""The deviatoric stress of the cube output (csrc/output.cu takes its root in a
Newton step and exactly near the middle between two floats): stresses whose
root is a float, the middle between two floats, a unit of FP64's last place to
either side, tiny, huge, zero, infinite and NaN, against numpy's rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_root_rounds_as_the_exact_one():
    import torch
    from stzpp_gb300 import advect
    nx, ny, nz = 64, 48, 40
    rng = np.random.default_rng(9)
    n = nx * ny * nz
    f = np.exp2(rng.uniform(-20, 20, n)).astype(np.float32)
    mid = (f.astype(np.float64) + np.nextafter(f, np.float32(np.inf)).astype(np.float64)) / 2
    s12 = np.where(np.arange(n) % 3 == 0, f.astype(np.float64), mid)
    step = rng.integers(-40, 41, n)
    s12 = (s12.view(np.int64) + step).view(np.float64)
    s12[:16] = [0.0, -0.0, 1e-300, 1e-160, 5e-324, 1e-40, 1e-35, 1e35, 1e40, 1e150, 1e200, np.inf, -np.inf, np.nan,
                1e-45, 1.0]
    s12 *= np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    g = advect.NGHOST
    shape = (nz + 2 * g, ny + 2 * g, nx + 2 * g)
    F = {k: torch.zeros(shape, dtype=torch.float64) for k in ("s11", "s12", "s13", "s22", "s23", "s33")}
    F["s12"][g:-g, g:-g, g:-g] = torch.from_numpy(s12.reshape(nz, ny, nx))
    F = {k: t.reshape(-1).cuda() for k, t in F.items()}
    got = advect.cube_values(F, (nx, ny, nz), 10).cpu().numpy().reshape(nx, ny, nz)
    with np.errstate(all="ignore"):
        want = np.sqrt(s12 * s12).astype(np.float32).reshape(nz, ny, nx).transpose(2, 1, 0)
    assert np.array_equal(got, want, equal_nan=True)
