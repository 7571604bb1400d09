"""FP64 energy and gradient by one, two and four lanes a row, at the ends of the ranges of magnetic rows that take them
(9,728 and 19,456 on 152 SMs), with one easy axis and with two, against the matrix-free oracle."""

import numpy as np
import pytest

from mumag_matrixfree2_gb300 import fem_utils
from mumag_matrixfree2_gb300 import synthetic as syn
from oracle import fem as ofem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axes", [1, 2])
@pytest.mark.parametrize("side", [2, 21, 22, 26, 27])
def test_energy_at_the_ends_of_each_number_of_lanes(cuda_ok, side, axes):
    knt, ijk = syn.box_mesh(syn.BoxWorkload("case", L=1.5 * (side - 1), h=1.5, r=1.3, n_air=2, box=1.5 * side + 12.0))
    mats = [syn.Material(axis=(np.sin(0.3), 0.0, np.cos(0.3))), syn.AIR]
    if axes == 2:  # the upper half of the magnet with another easy axis
        mats.insert(1, syn.Material(axis=(0.0, 0.6, 0.8)))
        ijk = ijk.copy()
        top = knt[ijk[:, :4]].mean(1)[:, 2] > 0.0
        ijk[ijk[:, 4] == 2, 4] = 3
        ijk[(ijk[:, 4] == 1) & top, 4] = 2
    A, K1, Js, k, _ = syn.reduced_materials(mats)
    s = fem_utils.prepare(knt, ijk, A, K1, Js, k)
    p = ofem.make_problem(knt, ijk, A, K1, Js, k)
    prob = fem_utils.make_problem(s)
    rng = np.random.default_rng(side)
    m = syn.initial_state(s.N, seed=side, amplitude=0.3)
    U, B = rng.standard_normal(s.N), np.array([0.05, -0.02, -0.3])
    E, g = prob.energy_and_grad(m, U, B)
    E0, g0 = ofem.energy_and_grad_mf(p, m, U, B)
    # the reference's parity bar for energies and gradients
    assert np.abs(g - g0).max() <= 1e-10 * np.abs(g0).max()
    assert abs(E - E0) <= 1e-10 * abs(E0)
