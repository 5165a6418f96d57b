"""Steps launched back to back (each launch may overlap the previous kernel's tail) give the bits of
the same steps with the device waited for in between, with torch operations on the state among
them, on a side stream, and replayed from a caller's CUDA graph."""
import numpy as np
import pytest
import torch

import pmfmhd
import problems

pytestmark = pytest.mark.gpu


def _state(dims, solver):
    s = pmfmhd.set_fields(pmfmhd.allocate_state(dims, 1.0 / max(dims), mhd_solver=solver),
                          problems.turb_field(dims, 1.0 / max(dims)))
    if solver == "ct":
        for d in range(3):
            s.ct.slot(d).copy_(s.U[5 + d])
    return s


def _one(s, dt, sp, torch_op):
    if torch_op:  # an ordinary kernel before and after the step's own
        s.U[1].mul_(1.0009765625)
    pmfmhd.step(s, dt, ch=sp, integrator="ref")
    if torch_op:
        s.U[1].mul_(0.9990234375)


@pytest.mark.parametrize("dims", [(16, 16, 16), (48, 48, 48), (100, 75, 61)])
@pytest.mark.parametrize("solver", ["glm", "ct"])
@pytest.mark.parametrize("torch_op", [False, True])
def test_back_to_back_steps_equal_waited_steps(dims, solver, torch_op):
    a, b, c = (_state(dims, solver) for _ in range(3))
    dt, sp = pmfmhd.compute_dt(a, 0.1)
    for _ in range(12):
        _one(a, dt, sp, torch_op)
    ha, va = pmfmhd.fields_to_host(a), pmfmhd.last_wavespeed(a)
    for _ in range(12):
        _one(b, dt, sp, torch_op)
        torch.cuda.synchronize()
    assert np.array_equal(ha, pmfmhd.fields_to_host(b))
    assert va == pmfmhd.last_wavespeed(b)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(6):
            _one(c, dt, sp, torch_op)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        for _ in range(6):
            _one(c, dt, sp, torch_op)
    graph.replay()
    assert np.array_equal(ha, pmfmhd.fields_to_host(c))
