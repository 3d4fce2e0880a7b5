"""calc_new_currents on both sides of every line between its kernels (five lanes
per wire, one wire per thread, two wires per thread, with and without unguarded
steps), by the device's SM count: EXACT against the divide routine in the
states of test_gpu_free_steps and in starts from zeros with unchecked divisors,
FAST against its scalar form, both initialisations; and the batched kernels of
few steps."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_exact import EXACT, EXACT_DIVIDE, FAST, cnc, device
from test_gpu_free_steps import STATES, make, significand

pytestmark = pytest.mark.gpu

FAST_SCALAR = 2


def sms(cuda):
    return cuda.cuda.get_device_properties(0).multi_processor_count


def exact(cuda, c, steps, init=0):
    for s in steps:
        a = cnc(cuda, device(c), s, EXACT, init)
        b = cnc(cuda, device(c), s, EXACT_DIVIDE, init)
        for k in ("current", "voltage"):
            assert same_bits(a[k], b[k]), (s, k)


@pytest.mark.parametrize("state", STATES)
def test_paired_kernel_in_every_state(cuda, oracle, state):
    W = 1440 * sms(cuda) + 1
    exact(cuda, make(oracle, state, 1, W // 4, W), (33, 200))


@pytest.mark.parametrize("init", [0, 1])
@pytest.mark.parametrize("per_sm,more", [(72, 0), (72, 1), (384, 0), (384, 1), (1440, 0),
                                         (1440, 1)])
def test_lines_between_the_exact_kernels(cuda, oracle, per_sm, more, init):
    W = per_sm * sms(cuda) + more
    for state in ("stable", "zeros", "overflow"):
        exact(cuda, make(oracle, state, 1, W // 4, W), (31, 32, 100), init)


def uncuttable(oracle):
    """Divisors in [1, 2) that only the rounded product is right for."""
    rng, out = np.random.default_rng(3), []
    while len(out) < 4:
        b = np.float32(rng.uniform(1, 2))
        if oracle.split_divisor(float(b))[0] == 1 and oracle.cut_divisor(float(b))[0] == 0:
            out.append(b)
    return np.array(out, np.float32)


@pytest.mark.parametrize("per_sm", [20, 300, 1441], ids=["lanes", "solo", "paired"])
@pytest.mark.parametrize("start", ["generated", "zeros", "stable"])
@pytest.mark.parametrize("divisors", ["cut_R", "cut_C", "cut_both", "corrected"])
def test_unchecked_divisors_through_careful_steps(cuda, oracle, divisors, start, per_sm):
    """Wide and LOW steps with truncated products, and with corrected quotients
    (a warp with both a divisor that needs truncation and one it is wrong for)."""
    W = per_sm * sms(cuda) + 7
    if start == "generated":  # overflows, then all NaN
        c = oracle.generate(oracle.GenParams(1, W // 4, W, 90, 31, L_offset=0.001))
    else:
        c = make(oracle, start, 1, W // 4, W)
        c.current[5, ::3] = 0  # not sound
    rng = np.random.default_rng(2)
    odd = rng.random(W) < 0.2
    if divisors != "cut_C":
        c.R[odd] = rng.choice(significand(oracle, 0), int(odd.sum()))
    if divisors != "cut_R":
        c.C[odd] = rng.choice(significand(oracle, 0), int(odd.sum()))
    if divisors == "corrected":
        c.R[~odd] = rng.choice(uncuttable(oracle), int((~odd).sum()))
    exact(cuda, c, (33, 150))


@pytest.mark.parametrize("init", [0, 1])
@pytest.mark.parametrize("per_sm,more", [(320, 0), (320, 1), (512, 3), (4096, 5)])
def test_lines_between_the_fast_kernels(cuda, oracle, per_sm, more, init):
    W = per_sm * sms(cuda) + more
    for state in ("stable", "overflow"):
        c = make(oracle, state, 1, W // 4, W)
        for steps in (1, 3, 40):
            a = cnc(cuda, device(c), steps, FAST, init)
            b = cnc(cuda, device(c), steps, FAST_SCALAR, init)
            for k in ("current", "voltage"):
                assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), (steps, k)


@pytest.mark.parametrize("block,wpt,schedule", [(128, 1, 0), (256, 1, 1), (128, 2, 2),
                                                (256, 2, 0)])
@pytest.mark.parametrize("steps", [[31, 16, 8, 2, 1], [31, 32, 8, 2, 1]], ids=["few", "mixed"])
def test_batched_rounds_of_few_steps(cuda, oracle, steps, block, wpt, schedule):
    from legionorigins_gb300 import batch as B
    from legionorigins_gb300 import circuit as C
    from legionorigins_gb300.workloads import CircuitSpec

    states = ["stable", "zeros", "wide_divisors", "overflow", "tiny"]
    shapes = [(3, 100, 701), (2, 50, 333), (5, 17, 64), (1, 40, 77), (4, 30, 129)]
    circuits = [make(oracle, st, *sh) for st, sh in zip(states, shapes)]
    fields = ["in_ptr", "out_ptr", "in_loc", "out_loc", "L", "R", "C", "current", "voltage",
              "charge", "node_voltage", "cap", "leak", "locator"]
    b = B.Batch([CircuitSpec(*sh, 90.0, 31, s) for sh, s in zip(shapes, steps)],
                [{k: np.ascontiguousarray(getattr(c, k)) for k in fields} for c in circuits])
    b.set_config(block, wpt, schedule)
    b.run(EXACT)
    assert b.check() == 0
    for i, (c, s) in enumerate(zip(circuits, steps)):
        dc = device(c)
        dc.loop_index_space(C.params(s, EXACT_DIVIDE))
        cuda.cuda.synchronize()
        want, got = dc.to_host(), b.read(i)
        for k in ("current", "voltage", "charge", "node_voltage"):
            assert same_bits(got[k], want[k]), (states[i], k)
    b.close()
