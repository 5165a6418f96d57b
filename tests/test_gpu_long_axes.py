"""The div-B diagnostics on boxes so long in y or z that their tiles exceed what grid dimensions y
and z can count (65535): accepted like any other shape, and the FP64 values."""
import pytest
import torch

import pmfmhd

pytestmark = pytest.mark.gpu
DX = 0.5


def _fill(ts, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    for t in ts:
        t.copy_(torch.randn(t.numel(), device="cuda", generator=g))


# 8 rows a tile: 65535 tiles end at ny = 524280; 16 planes a chunk: at nz = 1048560
@pytest.mark.parametrize("dims", [(1, 524280, 1), (1, 524281, 1), (3, 600000, 2), (64, 524296, 1), (1, 1, 1048561),
                                  (40, 1, 1100003)])
def test_max_divb_of_long_boxes(dims):
    nx, ny, nz = dims
    s = pmfmhd.allocate_state(dims, DX)
    _fill(s.U[5:8], nx + ny)
    B = [b.double().view(nz, ny, nx) for b in s.U[5:8]]
    div = sum(torch.roll(b, -1, 2 - a) - torch.roll(b, 1, 2 - a) for a, b in enumerate(B))
    assert pmfmhd.max_divb(s) == pytest.approx(div.abs().max().item() / (2 * DX), rel=1e-14)


@pytest.mark.parametrize("dims", [(2, 600000, 1), (1, 1, 1048561)])
def test_max_divb_face_of_long_boxes(dims):
    nx, ny, nz = dims
    s = pmfmhd.allocate_state(dims, DX, mhd_solver="ct")
    _fill([s.ct.slot(q) for q in range(3)], 3)
    F = [s.ct.slot(q).double().view(nz, ny, nx) for q in range(3)]
    div = sum(torch.roll(f, -1, 2 - a) - f for a, f in enumerate(F))
    assert pmfmhd.max_divb_face(s) == pytest.approx(div.abs().max().item() / DX, rel=1e-14)
