"""Row and column programs on short registers and small states against the oracle.

The sizes are the edges of the program kernels' shapes: registers of 2^4 .. 2^12
points, states of fewer rows than a CTA holds, registers with one to four amplitudes
below them, and both sides of the size from which full tiles run.  Tolerances as the
other parity tests: 1e-10 (complex128) and 2e-5 (complex64) of the state's norm.
"""

import numpy as np
import pytest

from oracle.cvdv_oracle import OracleSim

pytestmark = pytest.mark.gpu

TOL = {"complex128": 1e-10, "complex64": 2e-5}


def circuit(rng, qubits, n_gates):
    modes = [r for r, q in enumerate(qubits) if q >= 4]
    seq = []
    for g in range(n_gates):
        m = int(modes[rng.integers(len(modes))])
        c = int(rng.integers(len(qubits)))  # any register, the mode itself included
        k = int(rng.integers(qubits[c]))
        th = float(rng.uniform(-np.pi, np.pi))
        a = complex(rng.normal(0, 0.5), rng.normal(0, 0.5))
        kind = g % 12
        if kind == 0:
            seq.append(("r", (m, th)))
        elif kind == 1:
            seq.append(("d", (m, a)))
        elif kind == 2:
            seq.append(("h", (c, k)))
        elif kind == 3 and c != m:
            seq.append(("cd", (m, c, k, a)))
        elif kind == 4:
            seq.append(("s", (m, float(rng.uniform(0.05, 0.4)))))
        elif kind == 5 and c != m:
            seq.append(("cr", (m, c, k, th)))
        elif kind == 6:
            seq.append(("rx", (c, k, th)))
        elif kind == 7 and len(modes) > 1:
            seq.append(("bs", (modes[0], modes[1], th / 8)))
        elif kind == 8:
            seq.append(("phaseCubic", (m, 0.01)))
        elif kind == 9 and len(modes) > 1 and c not in modes[:2]:
            seq.append(("cbs", (modes[1], modes[0], c, k, th / 8)))
        elif kind == 10:
            seq.append(("ftQ2P", (m,)))
        else:
            seq.append(("rz", (c, k, th)))
    return seq


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
@pytest.mark.parametrize("qubits", [[4], [8], [11], [1, 5], [6, 1], [1, 7], [7, 2], [2, 4, 1], [4, 5], [5, 4, 2],
                                    [1, 10], [10, 1], [9, 2], [2, 12], [12, 1], [6, 6, 6], [1, 8, 9], [9, 10],
                                    [1, 4, 14], [13, 1], [8, 11, 1]])
def test_programs_match_oracle(qubits, precision):
    from cvdv_b200 import CudaCvdv
    rng = np.random.default_rng(sum(qubits) * 7 + len(qubits))
    n = sum(qubits)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    seq = circuit(rng, qubits, 36)
    o = OracleSim(list(qubits))
    o.set_state(psi)
    sim = CudaCvdv(list(qubits), precision=precision, check_errors=True)
    sim.initFromArray(psi)
    for meth, args in seq:
        getattr(o, meth)(*args)
        getattr(sim, meth)(*args)
    marg = sim.mEach(list(range(len(qubits))))
    out, ref = sim.getState(), o.get_state()
    assert np.linalg.norm(out - ref) < TOL[precision]
    for r, m in enumerate(marg):
        assert np.max(np.abs(m - o.m(r))) < TOL[precision]
