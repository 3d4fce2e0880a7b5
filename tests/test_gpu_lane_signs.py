"""Zeros' signs through EXACT's unguarded steps: wires whose state comes to
rest with a voltage of exactly zero, and node voltages of -0, in launches of
each kernel's size -- against the divide-routine form, bit for bit."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_exact import EXACT, EXACT_DIVIDE, cnc, device

pytestmark = pytest.mark.gpu

# launches of each kernel: 6 and 300: five lanes per wire,
# 12,000: one thread per wire, 230,001: two wires per thread
WIRES = [6, 300, 12000, 230001]


def wires(oracle, W):
    """W wires with two nodes of their own each."""
    c = oracle.generate(oracle.GenParams(1, 2 * W, W, 100, 5, L_offset=0.001))
    c.in_ptr[:] = 2 * np.arange(W)
    c.out_ptr[:] = c.in_ptr + 1
    c.in_loc[:], c.out_loc[:] = 0, 0
    return c


def at_rest(c, zero):
    """v_k = 16 (k - zero), one step further beyond v_zero: every segment's
    current is 1 but the one after v_zero, 2.  V0 + dt (i_k - i_k+1) / C cancels
    at v_zero (1 - 1) in every step, and all quotients are small integers."""
    v = 16.0 * (np.arange(11) - zero)
    v[zero + 1:] += 16
    i = np.ones(10)
    i[zero] = 2
    c.R[:], c.L[:], c.C[:] = 16, 1e-7, 1e-6
    c.node_voltage[::2], c.node_voltage[1::2] = v[0], v[10]
    c.current[:] = i[:, None]
    c.voltage[:] = (v[1:10] - (i[:-1] - i[1:]))[:, None]


@pytest.mark.parametrize("wires_", WIRES)
@pytest.mark.parametrize("zero", range(1, 10))
def test_voltage_at_rest_at_zero(cuda, oracle, zero, wires_):
    c = wires(oracle, wires_)
    at_rest(c, zero)
    for steps in (32, 64, 256, 1000):
        a = cnc(cuda, device(c), steps, EXACT)
        b = cnc(cuda, device(c), steps, EXACT_DIVIDE)
        assert (b["voltage"][zero - 1].view(np.uint32) == 0).all()  # +0
        for k in ("current", "voltage"):
            assert same_bits(a[k], b[k]), (steps, k)


@pytest.mark.parametrize("wires_", WIRES)
def test_node_voltage_of_negative_zero(cuda, oracle, wires_):
    """Node voltages of -0; without inductance, v_9 swings about zero and is
    exactly zero first after 40 steps, so the last current after 41 is -0.  The
    blocks before the one that meets the zero dividend pass their check."""
    c = wires(oracle, wires_)
    c.L[:], c.R[:], c.C[:] = 0, 2, np.float32(1e-6) * np.float32(2.0625)
    c.node_voltage[::2], c.node_voltage[1::2] = 3.25, -0.0
    c.current[:] = -1e4
    c.voltage[:8] = np.array([1.375, 1.6875, 1.0625, 1.1875, 1.5, 1.375, 1.6875, 1.3125])[:, None]
    c.voltage[8] = np.uint32(0x3EBD86EE).view(np.float32)
    for steps in (40, 41, 42, 100):
        a = cnc(cuda, device(c), steps, EXACT)
        b = cnc(cuda, device(c), steps, EXACT_DIVIDE)
        if steps == 41:
            assert (b["current"][9].view(np.uint32) == 0x80000000).all()  # -0
        for k in ("current", "voltage"):
            assert same_bits(a[k], b[k]), (steps, k)
