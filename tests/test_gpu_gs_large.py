"""Gauss-Seidel solves whose bands outnumber the CTAs of a launch (GPU required), so that a CTA
takes several bands in turn: three fields with the constant terms in global memory, one field
with both arrays there; and solves of more sweeps than a launch has warps in either form.
Everything must equal the host solver's restatement bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _check(fluid, wl, n, kd, kp):
    d, u, v, ds, us, vs = wl.random_state(n, n, n + kp, vmax=0.2)
    with fluid.FluidSolverGaussSeidel(n, diffuse_iterations=kd, pressure_iterations=kp, device=0) as s:
        s.upload(d, u, v)
        s.upload_sources(ds, us, vs)
        s.step(0.03, 0.01, 0.1)
        got = s.download()
    want = oracle.cpu_solve(d, ds, 0.03, u, v, us, vs, 0.01, 0.1, kd=kd, kp=kp, nsteps=1)
    for g, o in zip(got, want):
        np.testing.assert_array_equal(g, o)


# one CTA to an SM: a band's array alone takes 213 KB of shared memory
@pytest.mark.parametrize("kd,kp", [(3, 2), (26, 1)])
def test_three_fields_of_more_bands_than_ctas(fluid, wl, kd, kp):
    _check(fluid, wl, 2 + 32 * (_sms() // 3) + 17, kd, kp)


def test_both_arrays_in_global_memory_and_a_second_launch(fluid, wl):
    _check(fluid, wl, 1740, 26, 25)


# one CTA to an SM: 24 warps of 80 registers a thread
def test_one_field_of_more_bands_than_ctas(fluid, wl):
    _check(fluid, wl, 2 + 32 * (_sms() + 1) + 5, 1, 24)
