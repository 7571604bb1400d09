"""Which form a demag solve takes (one launch, separate kernels in a loop graph, host polling) and what it may not
change: the potential, the calls that are taken, and what a handle keeps from one call for the next."""

import ctypes as C

import numpy as np
import pytest
import torch

from mumag_matrixfree2_gb300 import _abi, fem_utils
from mumag_matrixfree2_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _problem(workload="cube8_h2_air24", precision="fp64"):
    knt, ijk = syn.box_mesh(syn.WORKLOADS[workload])
    A, K1, Js, k, _ = syn.reduced_materials([syn.Material(), syn.AIR])
    s = fem_utils.prepare(knt, ijk, A, K1, Js, k)
    prob = fem_utils.make_problem(s)
    if precision != "fp64":
        prob.set_precision(precision)
    prob.build_poisson(1e-12, "amgcl")
    return s, prob


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
@pytest.mark.parametrize("offset", [0, 1, 4, 8])
def test_potential_at_any_address(cuda_ok, precision, offset):
    """A potential that no kernel can read as doubles where it lies is copied, as a copy takes any address."""
    s, prob = _problem(precision=precision)
    m = torch.from_numpy(syn.initial_state(s.N, seed=3, amplitude=0.3)).cuda()
    x0 = torch.from_numpy(0.01 * np.random.default_rng(4).standard_normal(s.N) * s.boundary_mask).cuda()
    ref, it0, rr0, _ = prob.solve_u(m, x0.clone(), 1e-10)
    buf = torch.zeros(8 * s.N + 16, dtype=torch.uint8, device="cuda")
    buf[offset:offset + 8 * s.N].copy_(x0.view(torch.uint8))
    torch.cuda.synchronize()
    it, rr = C.c_int(), C.c_double()
    rc = _abi.lib().mm_solve_u_dev(prob.h, C.c_void_p(m.data_ptr()), C.c_void_p(buf.data_ptr() + offset), 1e-10, 2000,
                                   C.byref(it), C.byref(rr))
    assert (rc, it.value, rr.value) == (0, it0, rr0)
    U = np.frombuffer(buf[offset:offset + 8 * s.N].cpu().numpy().tobytes(), np.float64)
    assert np.array_equal(U, ref.cpu().numpy())
    assert not buf[:offset].any() and not buf[offset + 8 * s.N:].any()
