"""pmfmhd_run_glm on boxes whose planes are staged by TMA (x extent a multiple of 4 of at least a
staged plane): recording looks tensor maps up, which takes the context's lock. In a child process with
a time limit, so that a recording that waits for itself fails instead of holding the suite up."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import sys
sys.path[:0] = [{tests!r}, {pkg!r}]
import numpy as np
import pmfmhd, problems
dims, comp = (64, 48, 24), {comp}
U = problems.turb_field(dims, 1 / 64)
a, b = (pmfmhd.set_fields(pmfmhd.allocate_state(dims, 1 / 64, compensated=comp), U) for _ in range(2))
dt, sp = pmfmhd.compute_dt(a, 0.2)
for n in (5, 6, 5):  # odd and even counts, and a recorded graph once more
    for _ in range(n):
        pmfmhd.step_cube(a, dt, sp, 0.97)
    pmfmhd.run_glm(b, n, dt, sp, 0.97)
    assert np.array_equal(pmfmhd.fields_to_host(a), pmfmhd.fields_to_host(b)), n
assert pmfmhd.last_wavespeed(a) == pmfmhd.last_wavespeed(b)
assert pmfmhd.device_status(b) == 0
"""


@pytest.mark.parametrize("comp", [False, True])
def test_recorded_steps_equal_single_steps(comp):
    code = CHILD.format(tests=HERE, pkg=os.path.join(os.path.dirname(HERE), "pmf-glm_b200"), comp=comp)
    subprocess.run([sys.executable, "-c", code], check=True, timeout=180)
