"""Rounding of row and column programs, against 80-bit arithmetic.

Transforms of short registers, of small states and of 2^8-point strided registers run as
programs; the tile passes (column kernels switched off) multiply by twiddles and phases that
are rounded once each.  A program has as many roundings of each kind, so on the same
amplitudes its error may be 1.25 times the passes' (sums in another order), no more.

Linear phases: a displacement by alpha turns the outermost points by hundreds of radians.
Its phases are reduced before they are rounded, so whatever the angle, the error is that of two
transforms (1e-15 at most) and of four phases: a sine and cosine (2^-53 each, twice that for
the first-order step) and a running product of at most ten steps, of which a random
amplitude sees half, 6 2^-53 each.  Together below 1e-15 + 4 x 6 x 1.1e-16 = 3.7e-15; a
phase of a radians formed in one 64-bit word would be off by a 2^-53, 4e-14 at 340 radians.
"""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD, CLD = np.longdouble, np.clongdouble
PI = LD("3.14159265358979323846264338327950288")


def dft(x, sign):
    n = x.shape[-1]
    if n == 1:
        return x
    e, o = dft(x[..., 0::2], sign), dft(x[..., 1::2], sign)
    a = np.arange(n // 2).astype(LD) * (-2 * sign) * PI / n
    o = o * (np.cos(a) + CLD(1j) * np.sin(a))
    return np.concatenate([e + o, e - o], axis=-1)


class Exact:
    """One register's gates on a dense state, in 80-bit arithmetic."""

    def __init__(self, qubits, psi, reg):
        self.shape, self.reg, self.N = [1 << q for q in qubits], reg, 1 << qubits[reg]
        self.t = np.moveaxis(psi.astype(CLD).reshape(self.shape), reg, -1)
        self.n = np.arange(self.N)

    def phase(self, v):
        self.t = self.t * (np.cos(v) + CLD(1j) * np.sin(v))

    def x(self):
        return (self.n.astype(LD) - LD(self.N - 1) / 2) * np.sqrt(2 * PI / self.N)

    def ft(self, sign):
        N = self.N
        half = ((N - 1) * (2 * self.n - N + 1)) % (4 * N)
        self.phase(sign * PI * half.astype(LD) / (2 * N))
        # the centred kernel's phase is split evenly over both sides, up to a constant
        c = -sign * PI * LD(((N - 1) ** 2) % (4 * N)) / (2 * N)
        self.t = dft(self.t, sign) / np.sqrt(LD(N)) * (np.cos(c) - CLD(1j) * np.sin(c))
        self.phase(sign * PI * half.astype(LD) / (2 * N))

    def d(self, alpha):
        s2 = math.sqrt(2.0)
        self.phase(LD(s2 * alpha.imag) * self.x())
        self.ft(1)
        self.phase(LD(-s2 * alpha.real) * self.x())
        self.ft(-1)

    def state(self):
        return np.moveaxis(self.t, -1, self.reg).reshape(-1)


def random_state(rng, n, precision):
    v = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    v /= np.linalg.norm(v)
    return v.astype(np.complex64).astype(np.complex128) if precision == "complex64" else v


def transform_error(qubits, reg, psi, precision, fusion):
    from cvdv_b200 import CudaCvdv
    sim = CudaCvdv(list(qubits), precision=precision, check_errors=True)
    if fusion is not None:
        sim.setFusion(fusion)
    sim.initFromArray(psi)
    ex = Exact(qubits, psi, reg)
    for _ in range(3):
        sim.ftQ2P(reg)
        ex.ft(1)
    d = sim.getState() - ex.state()
    return float(np.sqrt((np.abs(d) ** 2).sum()))


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
@pytest.mark.parametrize("qubits,reg", [([4, 4], 0), ([4, 4], 1), ([5, 3], 0), ([1, 6], 1), ([7, 1], 0), ([8, 1], 0),
                                        ([1, 8], 1), ([9, 1], 0), ([1, 10], 1), ([11], 0), ([8, 6], 0), ([5, 8], 0)])
def test_transforms_round_as_the_tile_passes(qubits, reg, precision):
    n, q = sum(qubits), qubits[reg]
    got = ref = 0.0
    for seed in range(4):
        psi = random_state(np.random.default_rng(100 * n + seed), n, precision)
        got += transform_error(qubits, reg, psi, precision, None)
        # the same amplitudes with the register strided, without column kernels
        strided = np.moveaxis(psi.reshape([1 << k for k in qubits]), reg, 0).reshape(1 << q, -1)
        layout = [q, n - q] if n > q else [q, 1]
        if n == q:
            strided = np.concatenate([strided, np.zeros_like(strided)], axis=1)
        ref += transform_error(layout, 0, np.ascontiguousarray(strided).reshape(-1), precision, 0)
    assert got < 1.25 * ref, (got / 4, ref / 4)


@pytest.mark.parametrize("qubits,reg", [([8], 0), ([1, 10], 1), ([11], 0), ([12], 0), ([9, 1], 0), ([8, 11], 0),
                                        ([9, 11], 0), ([9, 11], 1), ([12, 8], 1), ([6, 13], 1), ([13, 6], 0)])
def test_large_displacements_keep_their_digits(qubits, reg):
    from cvdv_b200 import CudaCvdv
    psi = random_state(np.random.default_rng(sum(qubits)), sum(qubits), "complex128")
    alpha = complex(5.3, -4.7)
    sim = CudaCvdv(list(qubits), check_errors=True)
    sim.initFromArray(psi)
    sim.d(reg, alpha)
    ex = Exact(qubits, psi, reg)
    ex.d(alpha)
    assert float(np.sqrt((np.abs(sim.getState() - ex.state()) ** 2).sum())) < 3.7e-15


def test_large_displacements_of_a_batch_keep_their_digits():
    import torch
    from cvdv_b200.batch import BatchedCircuits
    alpha = complex(5.3, -4.7)
    insts = [dict(qubits=[1, m], gates=[("d", (1, alpha))]) for m in (8, 10, 11, 12, 13)]
    start = [random_state(np.random.default_rng(i), sum(inst["qubits"]), "complex128") for i, inst in enumerate(insts)]
    for row_loge in (None, {m: 4 for m in (8, 10, 11, 12, 13)}):
        B = BatchedCircuits(insts, precision="complex128", row_loge=row_loge)
        B.set_initial([torch.from_numpy(v).cuda() for v in start])
        B.run()
        for i, v in enumerate(start):
            ex = Exact(insts[i]["qubits"], v, 1)
            ex.d(alpha)
            assert float(np.sqrt((np.abs(B.state(i).cpu().numpy() - ex.state()) ** 2).sum())) < 3.7e-15
