"""Photon numbers on every route the momentum transform takes: row programs of one CTA and of
a cluster, column programs, column chains and tile passes; and the state they leave.

The reference is numpy on the state as the library holds it.  x^2 and p^2 are sums of
2^17 non-negative terms and one transform each: 1e-13 of their size in 64 bits; a complex64
transform rounds its amplitudes to 5e-7 of the norm, its squares' sum to 1e-6.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYOUTS = [([6], 0), ([4, 5], 0), ([8, 3], 0), ([3, 9], 1), ([10, 4], 0), ([13, 3], 0), ([3, 13], 1), ([14, 3], 0),
           ([3, 14], 1), ([15, 2], 0), ([2, 15], 1), ([1, 13, 2], 1), ([3, 1], 0), ([2, 2], 1)]


@pytest.mark.parametrize("precision,tol", [("complex128", 1e-12), ("complex64", 1e-6)])
@pytest.mark.parametrize("qubits,reg", LAYOUTS)
def test_photon_number(qubits, reg, precision, tol):
    from cvdv_b200 import CudaCvdv
    n, N = sum(qubits), 1 << qubits[reg]
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    sim = CudaCvdv(list(qubits), precision=precision, check_errors=True)
    sim.initFromArray(psi)
    held = sim.getState()
    t = np.moveaxis(held.reshape([1 << q for q in qubits]), reg, -1)
    x2 = ((np.arange(N) - (N - 1) / 2) ** 2) * (2 * np.pi / N)
    tw = np.exp(1j * np.pi * (((N - 1) * np.arange(N)) % (2 * N)) / N)
    mom = np.fft.fft(t * tw, axis=-1) / np.sqrt(N)
    qq, pp = ((np.abs(v) ** 2 * x2).sum() for v in (t, mom))
    got = sim.getPhotonNumber(reg)
    assert abs(got - (qq + pp - 1) / 2) < tol * (qq + pp)
    np.testing.assert_array_equal(sim.getState(), held)
