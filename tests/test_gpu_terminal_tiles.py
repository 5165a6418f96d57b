"""Terminal-regime induction and Maxwell force on cubes around the kernels' 32 x 8 column tiles
and z chunks, and smaller than their stencils, against the NumPy oracle (tolerances of
test_gpu_terminal.py)."""
import numpy as np
import pytest
import torch

import pmfmhd
import problems
import terminal_oracle as to
from test_gpu_terminal import KW, ct_state, f32, glm_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("solver", ["glm", "ct"])
@pytest.mark.parametrize("N", [3, 7, 31, 33, 48])
def test_induction_matches_oracle(N, solver, order):
    rho, B = problems.terminal_abc(N, dtype=np.float32)
    if solver == "ct":
        s = ct_state(N, rho, B)
    else:
        s = glm_state(N, rho, f32(1.5) + f32(0.5) * (B[0] ** 2 + B[1] ** 2 + B[2] ** 2), B)
    h = pmfmhd.fields_to_host(s)
    o = to.TerminalState(N, 1 / N, rho, h[4], [h[5], h[6], h[7]], faces=B if solver == "ct" else None)
    for _ in range(2):
        pmfmhd.terminal_ct_induction(s, 0.05, dissipation_order=order, **KW)
        o.induction(0.05, dissipation_order=order, **KW)
    h = pmfmhd.fields_to_host(s)
    for d in range(3):
        ref = o.B[d].ravel()
        assert np.abs(h[5 + d] - ref).max() <= 2e-7 + 5e-5 * np.abs(ref).max()
    assert np.abs(h[4] - o.E.ravel()).max() <= 2e-6 * np.abs(o.E).max()


@pytest.mark.parametrize("N", [2, 9, 33])
def test_force_matches_oracle(N):
    rng = np.random.default_rng(N)
    B = [rng.standard_normal(N ** 3).astype(f32) for _ in range(3)]
    s = glm_state(N, np.ones(N ** 3, f32), np.ones(N ** 3, f32), B)
    F = [torch.empty(N ** 3, device="cuda") for _ in range(3)]
    pmfmhd.terminal_magnetic_force(s, *F)
    o = to.magnetic_force([b.reshape(N, N, N) for b in B], f32(1) / (f32(2) * f32(1 / N)))
    for d in range(3):
        assert np.abs(F[d].cpu().numpy() - o[d].ravel()).max() <= 1e-6 + 1e-5 * np.abs(o[d]).max()
