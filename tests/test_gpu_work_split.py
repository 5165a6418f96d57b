"""How a step is divided over CTAs (equal column parts, even shares, tile heights) and how the
CT companion kernels are chunked leave no trace in the result; the signal speed reduced by the
step is the standalone reduction's. FP64 diagnostics on sizes and boundaries at the edges of
their tiles and vector loads."""
import numpy as np
import pytest

import pmfmhd
import problems
from test_gpu_back_to_back import _form_bits, _form_state, _form_step

pytestmark = pytest.mark.gpu
DIMS = [(16, 16, 16), (33, 9, 40), (100, 75, 61), (40, 200, 7), (31, 8, 300)]


def _field(dims):
    U = problems.turb_field(dims, 1.0 / max(dims))
    U[0] += np.float32(0.05) * np.sin(np.arange(U.shape[1]) * 0.37).astype(np.float32)
    return U


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("solver", ["glm", "ct"])
def test_division_of_the_work_leaves_the_bits(dims, solver):
    U = _field(dims)
    out = []
    for tile in (None, (8, dims[2]), (9, 1), (13, 3), (5, 16)):
        s = pmfmhd.set_fields(pmfmhd.allocate_state(dims, 1.0 / max(dims), mhd_solver=solver), U)
        if solver == "ct":
            for d in range(3):
                s.ct.slot(d).copy_(s.U[5 + d])
        if tile:
            pmfmhd.set_tile(s, *tile)
        dt, sp = pmfmhd.compute_dt(s, 0.2)
        for _ in range(2):
            pmfmhd.step(s, dt, ch=sp, integrator="ref")
        faces = [] if solver == "glm" else [s.ct.packed[:3 * s.nc].cpu().numpy()]
        out.append([pmfmhd.fields_to_host(s), pmfmhd.last_wavespeed(s), *faces])
        assert out[-1][1] == pytest.approx(pmfmhd.max_wavespeed(s), rel=1e-6)
    for other in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], other))


@pytest.mark.parametrize("dims", [(33, 9, 40), (100, 75, 61), (40, 200, 7), (224, 12, 224)])
@pytest.mark.parametrize("form", ["comp", "ct_comp", "drag", "rad", "rad_ppm", "ct_rad"])
def test_division_of_the_work_leaves_the_bits_of_every_form(dims, form):
    """The forms that keep remainders or corrections; (224, 12, 224) is a box on which the radiation
    step takes 13 rows of its own accord, more than the box has."""
    out = []
    for tile in (None, (8, dims[2]), (9, 1), (13, 3), (5, 16)):
        s, corr = _form_state(form, dims)
        if tile:
            pmfmhd.set_tile(s, *tile)
        dt, sp = pmfmhd.compute_dt(s, 0.2)
        for _ in range(2):
            _form_step(form, s, corr, dt, sp)
        out.append(_form_bits(s, corr))
    for other in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], other))


@pytest.mark.parametrize("dims", DIMS + [(1, 1, 1), (2, 3, 1), (32, 8, 16), (64, 64, 33)])
@pytest.mark.parametrize("bcs", [("periodic",) * 3, ("outflow", "reflecting", "periodic"),
                                 ("reflecting", "periodic", "outflow")])
def test_ledger_and_divb_are_the_fp64_values(dims, bcs):
    nx, ny, nz = dims
    rng = np.random.default_rng(3)
    U = rng.standard_normal((9, nx * ny * nz)).astype(np.float32)
    dx = 1.0 / max(dims)
    s = pmfmhd.set_fields(pmfmhd.allocate_state(dims, dx, bcs=bcs), U)

    def sides(b, axis, n, bc):  # upper and lower neighbour with the wall's sign of the normal field
        i = np.arange(n)
        out = []
        for j in (i + 1, i - 1):
            o = (j < 0) | (j >= n)
            src = j % n if bc == "periodic" else np.clip(j, 0, n - 1)
            sgn = np.where(o & (bc == "reflecting"), -1.0, 1.0).reshape([-1 if a == axis else 1 for a in range(3)])
            out.append(np.take(b, src, axis).astype(np.float64) * sgn)
        return out

    B = [U[5 + d].reshape(nz, ny, nx) for d in range(3)]
    (xp, xm), (yp, ym), (zp, zm) = (sides(B[d], 2 - d, dims[d], bcs[d]) for d in range(3))
    div = np.abs(((((xp - xm) + yp) - ym) + zp) - zm).max() * (1.0 / (2.0 * float(np.float32(dx))))
    assert pmfmhd.max_divb(s) == div
    dV = float(np.float32(np.float32(np.float32(dx) * np.float32(dx)) * np.float32(dx)))
    got = list(pmfmhd.conserved_totals(s).values())
    U64 = U[:8].astype(np.float64)
    # FP64 summation in any order: within n roundings of the sum of the magnitudes
    assert np.all(np.abs(np.array(got) - U64.sum(1) * dV) <= 2.3e-16 * U.shape[1] * np.abs(U64).sum(1) * dV)
