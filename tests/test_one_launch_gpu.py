"""The demag PCG as one launch (mm_pcg.cuh) against the separate kernels: every row and every reduction is
summed in the same order, so solves agree bit for bit, whatever the number of blocks.  The cases cover one
cluster and a cooperative grid, both chunk sizes of the reductions, two to four levels, each kind of coarse
solve and restriction, ragged rows, and solves that stop at once."""

import threading

import numpy as np
import pytest

from mumag_matrixfree2_gb300 import fem_utils
from mumag_matrixfree2_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _setup(mesh):
    if mesh[0] == "ellipsoid":
        mat = syn.Material(Js=1.3, A=8e-12, K1=4.3e6, axis=(0.6, 0.0, 0.8))
        knt, ijk = syn.ellipsoid_mesh(syn.Particle(*mesh[1:], mat))
    else:
        mat = syn.Material()
        knt, ijk = syn.box_mesh(syn.BoxWorkload("case", L=mesh[1], h=mesh[2], r=1.2, n_air=mesh[3], box=mesh[4]))
    A, K1, Js, k, _ = syn.reduced_materials([mat, syn.AIR])
    return fem_utils.prepare(knt, ijk, A, K1, Js, k)


MESHES = {
    "cluster": ("cube", 8.0, 2.0, 3, 24.0),  # 1,331 nodes, two levels
    "odd": ("cube", 15.0, 1.5, 6, 50.0),  # 12,167 nodes
    "ragged": ("ellipsoid", 5.3, 8.1, 12.9),  # uneven rows, three levels
    "four": ("cube", 40.0, 2.0, 9, 200.0),  # 59,319 nodes, four levels
    "large": ("cube", 69.0, 1.5, 6, 130.0),  # 205,379 nodes: partials of eight warps
}


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_one_launch_equals_separate_kernels(cuda_ok, mesh, precision):
    s = _setup(MESHES[mesh])
    prob = fem_utils.make_problem(s)
    if precision != "fp64":
        prob.set_precision(precision)
    prob.build_poisson(1e-12, "amg" if mesh == "odd" else "amgcl")
    m = syn.initial_state(s.N, seed=5, amplitude=0.3)
    x0 = 0.01 * np.random.default_rng(6).standard_normal(s.N) * s.boundary_mask
    U = None
    for coarse, restrict in ((3, 3), (0, 3), (3, 0)):
        prob.set_option("coarse_fuse", coarse)
        prob.set_option("fuse_restrict", restrict)
        for tol, maxiter in ((1e-10, 2000), (1e-3, 2000), (1e-10, 3), (1e-10, 0), (10.0, 5)):
            out = []
            for graph in (1, 0):
                prob.set_option("graph", graph)
                n0 = prob.launch_count()
                out.append((*prob.solve_u(m, x0, tol, maxiter), prob.launch_count() - n0))
            (U1, it1, rr1, rc1, n1), (U0, it0, rr0, rc0, n0) = out
            assert (it1, rr1, rc1) == (it0, rr0, rc0)
            assert np.array_equal(U1, U0)
            assert n1 < n0 or it0 == 0  # the one launch ran
            U = U1 if U is None else U
    assert U is not None and np.abs(U).max() > 0


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond"])
def test_rows_dealt_out_over_every_number_of_lanes(cuda_ok, precision):
    """Its operators are laid out for their lanes; the separate kernels read compressed rows."""
    s = _setup(MESHES["ragged"])
    prob = fem_utils.make_problem(s)
    if precision != "fp64":
        prob.set_precision(precision)
    prob.build_poisson(1e-12, "amgcl")
    m = syn.initial_state(s.N, seed=8, amplitude=0.3)
    for lanes in (2, 4, 8, 16, 32):
        prob.set_option("csr_lanes", lanes)
        out = []
        for graph in (1, 0):
            prob.set_option("graph", graph)
            out.append(prob.solve_u(m, np.zeros(s.N), 1e-10))
        assert out[0][1:] == out[1][1:] and out[0][3] == 0
        assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_folded_levels_are_the_same_preconditioner(cuda_ok, mesh, precision):
    """Prolongation and post-smoothing as one product against the two steps (without the fused restriction no level
    is folded).  Both solves stop at 1e-12, so the potentials agree to that times the operator's condition
    (~(box / h)^2 < 1e5)."""
    s = _setup(MESHES[mesh])
    prob = fem_utils.make_problem(s)
    if precision != "fp64":
        prob.set_precision(precision)
    prob.build_poisson(1e-12, "amgcl")
    m = syn.initial_state(s.N, seed=9, amplitude=0.3)
    out = []
    for restrict in (3, 0):
        prob.set_option("fuse_restrict", restrict)
        out.append(prob.solve_u(m, np.zeros(s.N), 1e-12))
    assert out[0][3] == out[1][3] == 0 and abs(out[0][1] - out[1][1]) <= 1
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-7 * np.abs(out[1][0]).max()


def test_solves_in_flight_share_the_device_and_keep_their_bits(cuda_ok):
    """Several threads' solves: the number in flight changes how each runs, not what it returns."""
    s = _setup(MESHES["ragged"])
    probs = [fem_utils.make_problem(s) for _ in range(6)]
    for p in probs:
        p.build_poisson(1e-12, "amgcl")
    states = [syn.initial_state(s.N, seed=k, amplitude=0.3) for k in range(6)]
    zero = np.zeros(s.N)
    ref = [probs[0].solve_u(m, zero, 1e-10)[0] for m in states]
    bad = []

    def work(k):
        for _ in range(20):
            U = probs[k].solve_u(states[k], zero, 1e-10)[0]
            if not np.array_equal(U, ref[k]):
                bad.append(k)

    for n in (2, 6):
        threads = [threading.Thread(target=work, args=(k,)) for k in range(n)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not bad
