"""The HLLD flux in each of its regions (supersonic either way, the outer and inner parts of the
fan, no field, field-aligned flow whose single-star states are degenerate) against the FP64
oracle in the same degeneracy mode. Allowed per field: the reference's parity gate
(test_backends.jl:65-72) plus what the reference's scheme in FP32 (the FP32 oracle) is off."""
import numpy as np
import pytest

import oracle
import pmfmhd
import problems
from mhd_cases import PAR

pytestmark = pytest.mark.gpu

# drift along (1, 1, 1) and mean field; sound speed ~1
REGIONS = {"right": (4.0, (0.4, -0.3, 0.2), 0.1), "left": (-4.0, (0.4, -0.3, 0.2), 0.1),
           "outer": (0.5, (0.05, 0.04, -0.06), 0.02), "inner": (0.02, (1.2, -1.0, 0.9), 0.3),
           "hydro": (0.1, (0.0, 0.0, 0.0), 0.0), "aligned": (0.1, (2.5, 0.0, 0.0), 0.0)}


@pytest.mark.parametrize("dtol", [0.0, 1e-5])
@pytest.mark.parametrize("region", list(REGIONS))
def test_hlld_region_matches_oracle(region, dtol):
    dims = (34, 11, 9)
    drift, b0, db = REGIONS[region]
    i, j, k = problems.cell_coords(dims)
    x, y, z = (2 * np.pi * (a - 0.5) / n for a, n in zip((i, j, k), dims))
    one = np.ones_like(x)
    q = [1 + 0.05 * np.sin(x + y), drift + 0.05 * np.sin(y + z), drift + 0.05 * np.sin(z + x), drift + 0.05 * np.sin(x - y),
         0.6 + 0.05 * np.cos(x + z), b0[0] * one + db * np.sin(y - z), b0[1] * one + db * np.sin(z + x),
         b0[2] * one + db * np.sin(x + y), 0 * x]
    U = problems.prim2cons(np.array(q), 5 / 3).astype(np.float32)
    o32, o64 = (oracle.OracleState(dims, 1.0 / 34, hlld_dtol_rel=dtol, dtype=T) for T in (np.float32, np.float64))
    dev = pmfmhd.set_fields(pmfmhd.allocate_state(dims, 1.0 / 34, hlld_dtol_rel=dtol), U)
    o32.U[:] = U
    o64.U[:] = U
    dt, sp = o32.compute_dt(0.2)
    for _ in range(2):
        o32.step(dt, ch=sp)
        o64.step(dt, ch=sp)
        pmfmhd.step(dev, float(dt), ch=float(sp))
    host = pmfmhd.fields_to_host(dev)
    for v in range(9):
        lim = PAR["atol"] + PAR["rtol"] * np.abs(o64.U[v]).max() + np.abs(o32.U[v] - o64.U[v]).max()
        assert np.abs(host[v] - o64.U[v]).max() <= lim, (region, v)


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_hypersonic_drift_stays_finite(sign):
    """A drift whose fast speed (pressure at its floor) is below the rounding of the velocity: the
    contact speed then equals the far side's signal speed to the last bit."""
    dims = (34, 11, 9)
    i, j, k = problems.cell_coords(dims)
    x, y, z = (2 * np.pi * (a - 0.5) / n for a, n in zip((i, j, k), dims))
    rho = 1 + 1e-3 * np.sin(x + y)
    v = [sign * 2e4 * (1 + 1e-6 * np.sin(z)), sign * 3e4 * (1 + 1e-4 * np.sin(y)), -sign * 1e4 + 0 * x]
    B = [1e-4 * np.sin(y - z), 1e-4 * np.sin(z + x), 1e-4 * np.sin(x + y)]
    E = 0.5 * rho * sum(a * a for a in v) * (1 - 1e-6)
    U = np.array([rho, *(rho * a for a in v), E, *B, 0 * x]).astype(np.float32)
    o = oracle.OracleState(dims, 1.0 / 34, hlld_dtol_rel=1e-5, dtype=np.float32)
    dev = pmfmhd.set_fields(pmfmhd.allocate_state(dims, 1.0 / 34), U)
    o.U[:] = U
    dt, sp = o.compute_dt(0.2)
    for _ in range(2):
        o.step(dt, ch=sp)
        pmfmhd.step(dev, float(dt), ch=float(sp))
    assert np.isfinite(o.U).all() and np.isfinite(pmfmhd.fields_to_host(dev)).all()
