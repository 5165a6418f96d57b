"""A terminal induction call that is refused for its subcycle limit writes nothing of the caller's:
state, scratch, faces and CT workspace keep their bits."""
import numpy as np
import pytest
import torch

import pmfmhd
import problems
from test_gpu_terminal import KW, ct_state, f32, glm_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["glm", "ct"])
def test_refused_call_writes_nothing(solver):
    N = 24
    rho, B = problems.terminal_abc(N, dtype=np.float32)
    s = ct_state(N, rho, B) if solver == "ct" else glm_state(N, rho, np.full(N ** 3, 2.0, f32), B)
    for t in s.scratch + ([s.ct.packed[3 * s.nc:]] if solver == "ct" else []):
        t.copy_(torch.randn(t.numel(), device="cuda", generator=torch.Generator("cuda").manual_seed(1)))
    mine = s.U + s.scratch + ([s.ct.packed] if solver == "ct" else [])
    before = [t.clone() for t in mine]
    with pytest.raises(pmfmhd.PMFMHDError, match="subcycles"):
        pmfmhd.terminal_ct_induction(s, 10.0, max_subcycles=1, **KW)
    assert all(torch.equal(a, b) for a, b in zip(before, mine))
