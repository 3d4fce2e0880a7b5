"""EXACT mode's first steps from zero currents and voltages (the generated
state, apps/circuit/circuit.cc:1071-1244) against the divide-routine form: the
same bits, zeros' signs among them, for node voltages over the exponent range,
zeros of either sign, and divisors and inductances over theirs."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_exact import EXACT, EXACT_DIVIDE, cnc, device

pytestmark = pytest.mark.gpu


def make(oracle, state, P, npp, wpp):
    c = oracle.generate(oracle.GenParams(P, npp, wpp, 90, 31, L_offset=0.001))
    rng = np.random.default_rng(17)
    W = c.L.size
    c.current[:], c.voltage[:] = 0, 0
    sign = lambda shape: rng.choice(np.array([-1, 1], np.float32), shape)
    if state == "exponents":     # every node voltage of its own magnitude
        c.node_voltage[:] = sign(c.node_voltage.shape) * np.exp2(
            rng.uniform(-140, 127, c.node_voltage.shape)).astype(np.float32)
    elif state == "edges":       # around the magnitudes where the checks turn
        c.node_voltage[:] = np.exp2(rng.choice([-30.0, -20.0, -10.0, 20.0, 40.0],
                                               c.node_voltage.shape)).astype(np.float32)
    elif state == "zeros":       # no voltage at some nodes, -0 in the state
        c.node_voltage[::3] = 0
        c.node_voltage[1::7] = -0.0
        c.current[:] *= sign(c.current.shape)
        c.voltage[:] *= sign(c.voltage.shape)
    elif state == "inductance":  # a1 down to and below the least normal number
        c.L[:] = np.exp2(rng.uniform(-42, -8, W)).astype(np.float32)
    elif state == "divisors":
        c.R[:] = sign(W) * np.exp2(rng.uniform(-7.9, 7.9, W)).astype(np.float32)
        c.C[:] = sign(W) * np.exp2(rng.uniform(-19.9, 29.9, W)).astype(np.float32)
    elif state == "nan_node":
        c.node_voltage[::29] = np.nan
        c.node_voltage[5::31] = np.inf
    return c


@pytest.mark.parametrize("shape", [(3, 100, 701), (61, 300, 1201), (30, 2000, 9001)],
                         ids=["lanes", "solo", "paired"])
@pytest.mark.parametrize("state", ["generated", "exponents", "edges", "zeros", "inductance",
                                   "divisors", "nan_node"])
def test_first_steps_equal_the_divide_routine(cuda, oracle, state, shape):
    c = make(oracle, state, *shape)
    for steps in (32, 33, 60):
        a = cnc(cuda, device(c), steps, EXACT)
        b = cnc(cuda, device(c), steps, EXACT_DIVIDE)
        for k in ("current", "voltage"):
            assert same_bits(a[k], b[k]), (steps, k)
