"""Runs of Rx + cd layers in one launch against the separate gate kernels.

Rows of 2^9 .. 2^12 points, one to three qubits above the mode (clusters of two, four and
eight rows), runs of one layer and of several on changing qubits.  The separate kernels
are themselves checked against the oracle; a layer of them and a layer of a run each round a
unit-norm state a few dozen times, so L layers agree to L times the single layer's
tolerance (1e-13 in complex128, 2e-6 in complex64), g values to ten times that.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("complex128", 1e-13), ("complex64", 2e-6)])
@pytest.mark.parametrize("qubits,layers", [([1, 9], 1), ([1, 9], 7), ([1, 1, 10], 5), ([3, 9], 6), ([2, 11], 4),
                                           ([1, 12], 3), ([1, 2, 12], 4)])
def test_run_of_layers_matches_separate_gates(precision, tol, qubits, layers):
    from cvdv_b200 import _lib
    L = _lib.load()
    prec = 0 if precision == "complex128" else 1
    cdt = torch.complex128 if prec == 0 else torch.complex64
    B, n, q = 5, sum(qubits), qubits[-1]
    rng = np.random.default_rng(n * 10 + layers)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def rnd():
        a = rng.standard_normal((B, 1 << n)) + 1j * rng.standard_normal((B, 1 << n))
        return torch.tensor(a / np.linalg.norm(a, axis=1, keepdims=True), dtype=cdt, device="cuda")

    p = np.empty((2 * layers, B))
    p[0::2], p[1::2] = rng.uniform(0, 2 * np.pi, (layers, B)), rng.normal(0, 0.5, (layers, B))
    p = torch.tensor(p, dtype=torch.float64, device="cuda")
    bits = [q + int(rng.integers(n - q)) for _ in range(layers)]
    cbits = (ctypes.c_int * layers)(*bits)
    psi, lam = rnd(), rnd()

    a, b = psi.clone(), psi.clone()
    for l, bit in enumerate(bits):
        assert L.cvdvBatchRx(ptr(a), prec, B, n, bit, ptr(p[2 * l]), 1.0, stream) == 0
        assert L.cvdvBatchCondDisp(ptr(a), prec, B, n, q, bit, ptr(p[2 * l + 1]), 1.0, stream) == 0
    assert L.cvdvBatchLayers(ptr(b), prec, B, n, q, cbits, layers, ptr(p), stream) == 0
    torch.cuda.synchronize()
    assert float((a - b).abs().max()) < layers * tol

    pa, la, pb, lb = psi.clone(), lam.clone(), psi.clone(), lam.clone()
    g = torch.zeros(2 * layers, 2 * B, dtype=torch.float64, device="cuda")
    g2 = torch.full_like(g, np.nan)
    for l in reversed(range(layers)):
        assert L.cvdvBatchCondDispAdjoint(ptr(pa), ptr(la), prec, B, n, q, bits[l], ptr(p[2 * l + 1]),
                                          ptr(g[2 * l + 1]), stream) == 0
        assert L.cvdvBatchRxAdjoint(ptr(pa), ptr(la), prec, B, n, bits[l], ptr(p[2 * l]), ptr(g[2 * l]), stream) == 0
    scratch = torch.empty(4 * layers * B << (n - q), dtype=torch.float64, device="cuda")
    assert L.cvdvBatchLayersAdjoint(ptr(pb), ptr(lb), prec, B, n, q, cbits, layers, ptr(p), ptr(g2), ptr(scratch),
                                    stream) == 0
    torch.cuda.synchronize()
    assert float((pa - pb).abs().max()) < layers * tol and float((la - lb).abs().max()) < layers * tol
    assert float((g - g2).abs().max()) < 10 * layers * tol * (1 + float(g.abs().max()))


def test_run_arguments_are_checked():
    from cvdv_b200 import _lib
    L = _lib.load()
    psi = torch.zeros(1, 1 << 10, dtype=torch.complex64, device="cuda")
    p = torch.zeros(2, 1, dtype=torch.float64, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    one = (ctypes.c_int * 1)
    for n, q, bit, layers in ((10, 8, 9, 1), (10, 9, 8, 1), (10, 9, 10, 1), (10, 9, 9, 0), (10, 9, 9, 65)):
        assert L.cvdvBatchLayers(ptr(psi), 1, 1, n, q, one(bit), layers, ptr(p), None) != 0
