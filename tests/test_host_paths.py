"""Host code of the library without a GPU, on a stand-in CUDA runtime (host_runtime.py)."""

import ctypes
import threading

import numpy as np
import pytest

from . import host_runtime


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    return host_runtime.load(tmp_path_factory.mktemp("host"))


def context(L, qubits, precision=0):
    h = L.cvdvCreateEx(len(qubits), (ctypes.c_int * len(qubits))(*qubits), precision)
    L.cvdvClearError(h)
    return h


def error(L, h):
    buf = ctypes.create_string_buffer(512)
    return L.cvdvGetLastError(h, buf, 512), buf.value.decode()


def set_state(L, h):
    n = L.cvdvGetTotalSize(h)
    L.cvdvSetStateFromDevicePtr(h, ctypes.create_string_buffer(16 * n))
    assert error(L, h)[0] == 0


def device_array(L, count):
    p = ctypes.c_void_p()
    assert L.cudaMalloc(ctypes.byref(p), 8 * count) == 0
    return p


def test_stand_in_runs_a_circuit(L):
    h = context(L, [1, 10])
    set_state(L, h)
    before = L.fake_launches()
    L.cvdvRotation(h, 1, 0.3)
    L.cvdvFlush(h)
    assert error(L, h) == (0, "") and L.fake_launches() > before
    L.cvdvDestroy(h)


@pytest.mark.parametrize("count", [3, 12])  # one group of launches, several
def test_a_failed_launch_leaves_the_launched_prefix(L, count):
    """Each parity gate is one launch into the other buffer: after a refused launch the
    state is the buffer that the last accepted one wrote."""
    for k in range(count + 1):
        h = context(L, [2, 2])
        set_state(L, h)
        start = L.cvdvGetStateDevicePtr(h)
        for _ in range(count):
            L.cvdvParity(h, 0)
        L.fake_fail_at(L.fake_launches() + k if k < count else -1)
        L.cvdvFlush(h)
        L.fake_fail_at(-1)
        assert (error(L, h)[0] != 0) == (k < count)
        L.cvdvClearError(h)
        assert (L.cvdvGetStateDevicePtr(h) != start) == bool(k & 1), k
        L.cvdvDestroy(h)


def test_a_failed_launch_before_the_product_leaves_no_state(L):
    """Two launches form the product of the register arrays: without them there is no
    state, after them the gates that were launched count."""
    for k in range(5):
        h = context(L, [2, 2])
        arrays = [ctypes.create_string_buffer(64) for _ in range(2)]
        L.cvdvInitFromSeparable(h, (ctypes.c_void_p * 2)(*[ctypes.addressof(a) for a in arrays]), 2)
        for _ in range(3):
            L.cvdvParity(h, 0)
        L.fake_fail_at(L.fake_launches() + k)
        L.cvdvFlush(h)
        L.fake_fail_at(-1)
        assert error(L, h)[0] != 0
        L.cvdvClearError(h)
        L.cvdvGetNorm(h)
        assert (error(L, h)[0] == 0) == (k >= 2), k
        L.cvdvDestroy(h)


def test_a_failed_launch_inside_a_transform_leaves_no_state(L):
    """A transform of a 2^15-point column is two launches: between them neither buffer
    holds a state."""
    kernels, states = [], []
    for k in range(8):
        h = context(L, [15, 3])
        set_state(L, h)
        L.cvdvFtQ2P(h, 0)
        L.fake_fail_at(L.fake_launches() + k)
        L.cvdvFlush(h)
        L.fake_fail_at(-1)
        if error(L, h)[0] == 0:
            break
        kernels.append("k_colr" in L.fake_last_kernel().decode())
        L.cvdvClearError(h)
        L.cvdvGetNorm(h)
        states.append(error(L, h)[0] == 0)
        L.cvdvDestroy(h)
    assert kernels[-2:] == [True, True] and states == [True] * (len(states) - 1) + [False]


def test_a_second_device_opts_in_to_shared_memory(L):
    """2^8-point columns of a large complex128 state take 70 KB of shared memory: every
    device a process uses has to opt in."""
    for device in (0, 1, 0):
        L.fake_set_device(device)
        h = context(L, [8, 11])
        set_state(L, h)
        L.cvdvRotation(h, 0, 0.3)
        L.cvdvFlush(h)
        assert error(L, h) == (0, ""), device
        L.cvdvDestroy(h)
    L.fake_set_device(0)


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_stages_opt_in_on_every_device(L, precision):
    states, tasks, programs = device_array(L, 64), device_array(L, 64), device_array(L, 1024)
    for device in (0, 1, 0):
        L.fake_set_device(device)
        assert L.cvdvBatchRunStage(states, precision, tasks, 1, programs, 1, None) == 0, device
    L.fake_set_device(0)


def test_state_readbacks_take_no_more_memory(L):
    h = context(L, [22], precision=1)
    set_state(L, h)
    re, im = ((ctypes.c_double * (1 << 22))() for _ in range(2))
    L.cvdvGetState(h, re, im)
    L.cvdvGetState(h, re, im)
    held = L.fake_device_bytes()
    for _ in range(3):
        L.cvdvGetState(h, re, im)
    assert error(L, h)[0] == 0 and L.fake_device_bytes() == held
    L.cvdvDestroy(h)


def test_short_register_arrays_are_refused(L):
    """A device array with fewer amplitudes than its register is an error, not a read
    past its end; with enough of them, at whatever offset, it is taken."""
    h = context(L, [4, 5])
    a, b = device_array(L, 2 << 4), device_array(L, (2 << 5) - 2)
    for short in ((a, b), (ctypes.c_void_p(a.value + 16), device_array(L, 2 << 5))):
        L.cvdvInitFromSeparable(h, (ctypes.c_void_p * 2)(*short), 2)
        assert error(L, h)[0] != 0
        L.cvdvClearError(h)
    c = device_array(L, 2 << 6)
    L.cvdvInitFromSeparable(h, (ctypes.c_void_p * 2)(a, c.value + (16 << 5)), 2)
    assert error(L, h)[0] == 0
    L.cvdvDestroy(h)


def test_readouts_into_device_memory_are_copied(L):
    """The host writes no results to memory that is not its own."""
    h = context(L, [3, 4])
    set_state(L, h)
    out = device_array(L, 8)
    L.cvdvMeasureMultiple(h, (ctypes.c_int * 1)(0), 1, ctypes.cast(out, ctypes.POINTER(ctypes.c_double)))
    assert error(L, h)[0] == 0 and L.fake_copied_to(out) == 64
    L.cvdvDestroy(h)


@pytest.mark.parametrize("readers", [1, 3])  # one takes the staged chunks and their threads, the others plain copies
@pytest.mark.parametrize("shift", [0, 40])
def test_large_readbacks_arrive_whole(L, readers, shift):
    n = 1 << 22
    hs = [context(L, [22], precision=1) for _ in range(readers)]
    outs = [np.full(2 * n + 1024, -1.0) for _ in hs]
    for h in hs:
        set_state(L, h)
        L.cvdvGetNorm(h)

    def first(out):  # on a page, or off it
        return (-out.ctypes.data // 8) % 512 + shift

    def read(h, out):
        L.cvdvGetState(h, *(ctypes.cast(out.ctypes.data + 8 * (first(out) + k * n), ctypes.POINTER(ctypes.c_double))
                            for k in range(2)))

    for h, out in zip(2 * hs, 2 * outs):
        read(h, out)  # (the split arrays have their place from the second on)
    L.fake_count_up()
    for out in outs:
        out[:] = -1.0
    threads = [threading.Thread(target=read, args=a) for a in zip(hs, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for h, out in zip(hs, outs):
        got, at = out[first(out): first(out) + 2 * n], first(out)
        assert error(L, h)[0] == 0 and (np.diff(got) == 1).all()
        assert (out[:at] == -1).all() and (out[at + 2 * n:] == -1).all()
        L.cvdvDestroy(h)
