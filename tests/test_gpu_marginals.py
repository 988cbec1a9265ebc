"""Marginals of single registers at the edges of the axis kernel's forms.

Registers with 1 .. 2^4 amplitudes below them (positions) and 2^5 and more (runs), inner
blocks below, at and above 2^8, states smaller than a CTA, registers of two values and of
2^14, several registers above the tile in one readout.  The reference is numpy on the state
as the library holds it (rounded to complex64 there); sums of at most 2^20 non-negative
terms of total one in 64 bits differ by less than 1e-12 in any order.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYOUTS = [[1], [3], [2, 3], [7, 1], [5, 3], [1, 4, 4], [8], [9], [3, 9], [9, 1], [9, 4], [9, 5], [1, 8, 9, 1],
           [13, 2], [2, 13], [6, 14], [14, 6], [1] * 12, [1, 1, 2, 12], [2, 1, 13], [12, 1, 1, 1]]


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
@pytest.mark.parametrize("qubits", LAYOUTS, ids=lambda q: "_".join(map(str, q)))
def test_single_register_marginals(qubits, precision):
    from cvdv_b200 import CudaCvdv
    rng = np.random.default_rng(sum(qubits) * 31 + len(qubits))
    n = sum(qubits)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    if precision == "complex64":
        held = psi.astype(np.complex64).astype(np.complex128)
    else:
        held = psi
    p = (np.abs(held) ** 2).reshape([1 << q for q in qubits])
    ref = [p.sum(axis=tuple(s for s in range(len(qubits)) if s != r)) for r in range(len(qubits))]
    sim = CudaCvdv(qubits, precision=precision, check_errors=True)
    sim.initFromArray(psi)
    for r, m in enumerate(ref):
        np.testing.assert_allclose(sim.m(r), m, rtol=0, atol=1e-12)
    order = list(rng.permutation(len(qubits)))
    for r, m in zip(order, sim.mEach([int(r) for r in order])):
        np.testing.assert_allclose(m, ref[r], rtol=0, atol=1e-12)


def test_separable_arrays_from_any_memory():
    """Register arrays on the host, on the device, and on the device at an odd 8-byte
    offset give the same state (one gather launch, or copies)."""
    import torch
    from cvdv_b200 import CudaCvdv, SeparableState, _lib
    import ctypes
    qubits = [1, 2, 6, 3]
    rng = np.random.default_rng(5)
    arrs = [torch.from_numpy(rng.standard_normal(1 << q) + 1j * rng.standard_normal(1 << q)) for q in qubits]
    ref = arrs[0]
    for a in arrs[1:]:
        ref = torch.outer(ref, a).reshape(-1)
    keep = []

    def shifted(a):  # a device copy that starts 8 bytes after a 16-byte boundary
        buf = torch.empty(2 * a.numel() + 1, dtype=torch.float64, device="cuda")
        buf[1:] = torch.view_as_real(a).reshape(-1).cuda()
        keep.append(buf)
        return buf.data_ptr() + 8

    for where in ("cpu", "cuda", "shifted"):
        sim = CudaCvdv(qubits, check_errors=True)
        if where == "shifted":
            ptrs = (ctypes.c_void_p * 4)(*[ctypes.c_void_p(shifted(a)) for a in arrs])
            torch.cuda.synchronize()
            _lib.load().cvdvInitFromSeparable(sim.ctx, ptrs, 4)
        else:
            sep = SeparableState(qubits, device=where)
            for r, a in enumerate(arrs):
                sep.setCoeffs(r, a)
            sim.initStateVector(sep)
        # one rounding per product of four factors, each at most a few units in size
        np.testing.assert_allclose(sim.getState(), ref.numpy(), rtol=1e-14, atol=1e-14)
