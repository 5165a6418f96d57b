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


# Every form of the step that overlaps its predecessor and keeps state of its own from step to step:
# remainders, faces and their remainders, tracked corrections.
FORMS = ["comp", "ct_comp", "drag", "ct_drag", "rad", "ct_rad"]


def _form_state(form, dims):
    ct = form.startswith("ct_")
    s = pmfmhd.allocate_state(dims, 1.0 / max(dims), mhd_solver="ct" if ct else "glm", compensated=form.endswith("comp"),
                              recon="ppm" if form.endswith("ppm") else "plm")
    pmfmhd.set_fields(s, problems.turb_field(dims, 1.0 / max(dims)))
    if ct:
        for d in range(3):
            s.ct.slot(d).copy_(s.U[5 + d])
    corr = None
    if "rad" in form:
        corr = pmfmhd.allocate_radiation_correction(s)
        g = torch.Generator("cuda").manual_seed(5)
        corr[s.nc:4 * s.nc] = 2e-3 * torch.randn(3 * s.nc, device="cuda", generator=g)
    return s, corr


def _form_step(form, s, corr, dt, sp):
    if "rad" in form:
        pmfmhd.step_ref_radiation(s, dt, sp, 0.97, 0.05, corr)
        corr[:s.nc].copy_(s.U[8])  # the driver's refresh of slot 0, an ordinary copy between the steps
    elif form.endswith("drag"):
        pmfmhd.step_ref_drag(s, dt, sp, 0.97, 0.05)
    else:
        pmfmhd.step_ref(s, dt, sp, 0.97, compensate_faces=form == "ct_comp")


def _form_bits(s, corr):
    out = [pmfmhd.fields_to_host(s)]
    out += [r.cpu().numpy() for r in s.resid or []]
    if s.ct is not None:
        out += [s.ct.slot(q).cpu().numpy() for q in (0, 1, 2, 18, 19, 20)]
    return out + ([] if corr is None else [corr.cpu().numpy()])


@pytest.mark.parametrize("dims", [(16, 16, 16), (48, 48, 48), (100, 75, 61)])
@pytest.mark.parametrize("form", FORMS)
def test_forms_that_keep_state_equal_waited_steps(dims, form):
    (a, ca), (b, cb), (c, cc) = (_form_state(form, dims) for _ in range(3))
    dt, sp = pmfmhd.compute_dt(a, 0.1)
    for _ in range(10):
        _form_step(form, a, ca, dt, sp)
    bits = _form_bits(a, ca)
    for _ in range(10):
        _form_step(form, b, cb, dt, sp)
        torch.cuda.synchronize()
    assert all(np.array_equal(x, y) for x, y in zip(bits, _form_bits(b, cb)))
    # two steps in a graph, replayed five times back to back
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        for _ in range(2):
            _form_step(form, c, cc, dt, sp)
    for _ in range(5):
        graph.replay()
    assert all(np.array_equal(x, y) for x, y in zip(bits, _form_bits(c, cc)))


@pytest.mark.parametrize("solver", ["glm", "ct"])
def test_evolve_equals_waited_steps(solver):
    dims = (48, 40, 33)
    a, b = (_state(dims, solver) for _ in range(2))
    dt, _ = pmfmhd.compute_dt(a, 0.2)
    t, n = pmfmhd.evolve(a, 9.5 * dt, cfl=0.2)
    wait = lambda *_: torch.cuda.synchronize()  # noqa: E731
    assert (t, n) == pmfmhd.evolve(b, 9.5 * dt, cfl=0.2, callback=wait)
    assert n >= 9 and np.array_equal(pmfmhd.fields_to_host(a), pmfmhd.fields_to_host(b))
