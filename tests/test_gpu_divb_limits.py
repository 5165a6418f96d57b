"""max_divb on fields at the limits of FP32: its screen may not lose a cell whose FP64 value is
finite because the FP32 evaluation overflows, cancels infinities or falls below the normal range.
Cells whose FP64 value is a NaN are passed over, as by the maximum it is compared with."""
import numpy as np
import pytest

import pmfmhd

pytestmark = pytest.mark.gpu
DX = 0.25


def _expected(B):
    with np.errstate(invalid="ignore"):
        d = sum(np.roll(b.astype(np.float64), -1, 2 - a) - np.roll(b.astype(np.float64), 1, 2 - a) for a, b in enumerate(B))
    return np.nanmax(np.abs(d)) / (2 * DX)


def _field(kind, dims):
    rng = np.random.default_rng(7)
    B = rng.standard_normal((3, dims[2], dims[1], dims[0])).astype(np.float32)
    if kind == "huge":  # every FP32 sum overflows in one term or another, with either sign
        return np.clip(B, -3.6, 3.6) * np.float32(0.94e38)
    if kind == "opposite":  # cell (20, 4, 1): inf - inf in FP32, 6.45e38 in FP64, the others at most 3.39e38
        B[0, 1, 4, 21], B[0, 1, 4, 19] = 3.3e38, -3.3e38
        B[1, 1, 5, 20], B[1, 1, 3, 20] = -1.725e38, 1.725e38
        B[2, 2, 4, 20], B[2, 0, 4, 20] = 1.65e38, -1.65e38
        B[0, 0, 4, 9] = 3.39e38  # met first where a chunk has several planes: the bound when the cell is met
    if kind == "inf":
        B[2, 0, 2, 7] = np.inf
    if kind == "nan":
        B[1, 2, 3, 11] = np.nan
        B[0, 0, 0, 0] = -np.inf
        B[2, 3, 1, 30] = 3e38
    if kind == "tiny":  # differences of neighbours below the normal range
        return (np.float32(2e-38) * (1 + 0.05 * B)).astype(np.float32)
    return B


@pytest.mark.parametrize("dims", [(64, 8, 4), (33, 9, 5), (128, 16, 40), (512, 512, 16)])
@pytest.mark.parametrize("kind", ["huge", "opposite", "inf", "nan", "tiny"])
def test_divb_at_the_limits_of_fp32(dims, kind):
    B = _field(kind, dims)
    s = pmfmhd.allocate_state(dims, DX)
    U = np.zeros((9, s.nc), np.float32)
    U[0], U[4] = 1.0, 1.0
    U[5:8] = B.reshape(3, -1)
    pmfmhd.set_fields(s, U)
    # a sum of six doubles in another order: the last bits may differ
    assert pmfmhd.max_divb(s) == pytest.approx(_expected(B), rel=1e-15 * 8)
