"""The launches a variational circuit's sweeps walk: runs of fused layers between
checkpoints.  The plan without a GPU, and gradients through it against autograd."""

import math

import numpy as np
import pytest
import torch

from cvdv_b200.variational import MAX_LAYERS, VariationalCircuit, layered_gates


def mixed_gates(rng, qubits, count):
    """Layers on changing qubits, with lone gates and controls off the rotated qubit between."""
    mode, gates = len(qubits) - 1, []
    while len(gates) < count:
        r = int(rng.integers(mode))
        k = int(rng.integers(qubits[r]))
        kind = int(rng.integers(8))
        if kind == 0:
            gates.append(("rx", r, k))
        elif kind == 1:
            gates.append(("cd", mode, r, k))
        else:
            gates += [("rx", r, k), ("cd", mode, r, k)]
    return gates[:count]


@pytest.mark.parametrize("every", [1, 3, 5, 16, 1000])
@pytest.mark.parametrize("qubits,layered", [([1, 12], True), ([1, 1, 9], True), ([3, 10], True), ([2, 2, 9], False),
                                            ([1, 8], False)])
def test_launches_cover_the_gates_between_checkpoints(qubits, layered, every):
    rng = np.random.default_rng(every)
    for gates in (mixed_gates(rng, qubits, 61), mixed_gates(rng, qubits, 400),
                  [g for _ in range(150) for g in (("rx", 0, 0), ("cd", len(qubits) - 1, 0, 0))]):
        c = VariationalCircuit(qubits, gates, checkpoint_every=every)
        assert [g for g, n in c._launches for g in range(g, g + n)] == list(range(len(gates)))
        starts = {g for g, _ in c._launches}
        assert set(range(0, len(gates), every)) <= starts  # every checkpoint is saved and restored
        singles = {g for g, n in c._steps if n == 1}
        pairs = {g for g, n in c._steps if n == 2}
        for g, n in c._launches:
            if n == 1:
                assert g in singles
            else:
                assert n % 2 == 0 and n <= 2 * MAX_LAYERS and all(k in pairs for k in range(g, g + n, 2))
                assert layered or n == 2


def test_long_runs_are_split():
    c = VariationalCircuit([1, 10], layered_gates(150), checkpoint_every=1000)
    assert c._launches == [(0, 128), (128, 128), (256, 44)]


def loss_by_autograd(gates, qubits, params, psi0, target):
    """The fidelity loss in differentiable 64-bit torch, each gate by its definition."""
    B, nq, N = params.shape[0], sum(qubits[:-1]), 1 << qubits[-1]
    n = torch.arange(N, dtype=torch.float64)
    x = (n - (N - 1) / 2) * math.sqrt(2 * math.pi / N)
    tw = torch.polar(torch.ones_like(x), math.pi * (((N - 1) * torch.arange(N)) % (2 * N)).double() / N)
    psi = psi0.expand(B, -1).reshape(B, 1 << nq, N)
    for g, gate in enumerate(gates):
        reg, k = (gate[1], gate[2]) if gate[0] == "rx" else (gate[2], gate[3])
        bit = sum(qubits[:reg]) + k  # from the front of the qubits
        v = psi.reshape(B, 1 << bit, 2, 1 << (nq - 1 - bit), N)
        if gate[0] == "rx":
            c, s = (f(params[:, g] / 2).reshape(B, 1, 1, 1, 1) for f in (torch.cos, torch.sin))
            v = c * v - 1j * s * v.flip(2)
        else:
            ph = -math.sqrt(2.0) * params[:, g].reshape(B, 1, 1, 1, 1) * x
            ph = torch.cat((ph, -ph), dim=2)
            v = torch.fft.fft(v * tw, norm="ortho") * tw * torch.polar(torch.ones_like(ph), ph)
            v = torch.fft.ifft(v * tw.conj(), norm="ortho") * tw.conj()
        psi = v.reshape(B, 1 << nq, N)
    ov = (target.conj() * psi.reshape(B, -1)).sum(dim=1)
    return 1.0 - (ov.real ** 2 + ov.imag ** 2)


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("qubits,every", [([1, 1, 9], 5), ([3, 10], 7), ([1, 9], 1000)])
def test_gradients_through_runs_match_autograd(qubits, every, graphs):
    """Every gate rounds a unit-norm state a few dozen times: 60 gates stay below 1e-12 of
    the loss and its gradients (of order one) in complex128."""
    rng = np.random.default_rng(sum(qubits))
    gates = mixed_gates(rng, qubits, 60)
    n, B = sum(qubits), 3
    psi = [torch.from_numpy(v / np.linalg.norm(v)) for v in
           (rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n) for _ in range(2))]
    p = torch.from_numpy(rng.uniform(-0.6, 0.6, (B, len(gates))))
    circ = VariationalCircuit(qubits, gates, precision="complex128", checkpoint_every=every, graphs=graphs)
    assert any(k > 2 for _, k in circ._launches)
    # the target is close to the circuit's result, so the gradients are not small
    with torch.no_grad():
        psi[1] = 0.2 * psi[1] + circ.states(p[:1], psi[0].cuda()).cpu()[0]
        psi[1] = psi[1] / psi[1].abs().square().sum().sqrt()
    ref, got = p.clone().requires_grad_(True), p.clone().requires_grad_(True)
    loss = loss_by_autograd(gates, qubits, ref, psi[0], psi[1])
    loss.sum().backward()
    out = circ.fidelity_loss(got, psi[0].cuda(), psi[1].cuda())
    out.sum().backward()
    assert float((out.detach().cpu() - loss.detach()).abs().max()) < 1e-12
    assert float((got.grad.cpu() - ref.grad).abs().max()) < 1e-12 * max(1.0, float(ref.grad.abs().max()))
