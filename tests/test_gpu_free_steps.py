"""EXACT mode's unguarded steps (blocks checked as a whole, redone with
guarded steps when the check fails) against the divide-routine form
CKT_MODE_EXACT_DIVIDE: the same bits for states that take each of its ways --
sound constants, zeros and tiny values, divisors the split quotient is not
right for, dividends next to a rounding boundary, overflow and NaN on the
way, wires in equilibrium -- at step counts around the block sizes."""
import ctypes

import numpy as np
import pytest

from conftest import same_bits
from test_gpu_exact import EXACT, EXACT_DIVIDE, cnc, device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("divisor", [0, 1], ids=["R", "C"])
def test_split_quotient_of_checked_divisors(cuda, ckt, divisor):
    c = cuda.zeros(4, dtype=cuda.int64, device="cuda")
    n = 1 << 24
    ckt.check(ckt.tools().ckt_check_split_quotient(99 + divisor, n, divisor, c.data_ptr(), None))
    cuda.cuda.synchronize()
    bad, checked, moved, drawn = c.tolist()
    assert bad == 0 and drawn == n
    # C below 2^-20 (10 of the 60 binades drawn) is never accepted
    eligible = n * (1 if divisor == 0 else 50 / 60)
    assert 0.998 * eligible < checked < 1.002 * eligible
    assert 0.010 < moved / eligible < 0.015


def significand(oracle, verdict):
    """Divisors in [1, 2) with the verdict, as many as a wire range needs."""
    rng, out = np.random.default_rng(verdict), []
    while len(out) < 4:
        b = np.float32(rng.uniform(1, 2))
        if oracle.split_divisor(float(b))[0] == verdict:
            out.append(b)
    return np.array(out, np.float32)


def near_tie_dividend(R):
    """A significand a for which a / R lies next to a rounding boundary (odd
    R): the larger of +-2^-25 mod B, B the integer significand of R."""
    B = (R.view(np.uint32).astype(np.int64) & 0x7FFFFF) | 0x800000
    A = np.ones_like(B)
    for _ in range(25):
        A = np.where(A & 1, (A + B) >> 1, A >> 1)
    A = np.maximum(A, B - A)
    return np.where(A >= 1 << 23, A, 1 << 23).astype(np.float32) * np.float32(2.0 ** -23)


def make(oracle, state, P, npp, wpp):
    c = oracle.generate(oracle.GenParams(P, npp, wpp, 90, 31, L_offset=0.001))
    rng = np.random.default_rng(7)
    W = c.L.size
    c.L[:] = rng.uniform(1e-7, 9e-7, W)
    c.C[:] = np.maximum(c.C, 1e-4)
    for a in (c.current, c.voltage, c.node_voltage):
        a[:] = rng.uniform(-1, 1, a.shape)
    some = rng.choice(W, max(1, W // 50), replace=False)
    if state == "zeros":           # not sound: currents and voltages start at 0
        c.current[:], c.voltage[:] = 0, 0
    elif state == "signed_zeros":  # -0 in a few wires' starting values
        c.current[3, some], c.voltage[4, some] = -0.0, -0.0
    elif state == "tiny":          # dividends far below the guarded range
        for a in (c.current, c.voltage, c.node_voltage):
            a *= np.float32(2.0 ** -70)
    elif state == "tiny_voltages":  # just above and below the soundness bounds
        c.voltage[:] *= np.exp2(rng.uniform(-52, -20, c.voltage.shape)).astype(np.float32)
        c.current[:] *= np.exp2(rng.uniform(-52, 0, c.current.shape)).astype(np.float32)
    elif state == "equilibrium":   # equal voltages and currents: zero differences
        c.voltage[:], c.node_voltage[:], c.current[:] = 0.75, 0.75, 0.25
    elif state == "unchecked_R":
        c.R[some] = rng.choice(significand(oracle, 0), some.size)
    elif state == "unchecked_C":
        c.C[some] = rng.choice(significand(oracle, 0), some.size)
    elif state == "moved":
        c.R[:] = rng.choice(significand(oracle, 2), W)
        c.C[:] = rng.choice(significand(oracle, 2), W)
    elif state == "near_ties":     # first step divides 'a' by R; errors grow
        c.R[:] = np.concatenate([rng.uniform(1, 2, W - some.size),
                                 rng.choice(significand(oracle, 2), some.size)])
        c.R[:] = (c.R.view(np.uint32) | 1).view(np.float32)
        a = near_tie_dividend(c.R)
        c.L[:] = 4e-6
        c.node_voltage[:] = 0
        c.voltage[:2] = a, 2 * a
    elif state == "negative":      # divisors of either sign
        for d in (c.R, c.C):
            d[some] = -d[some]
    elif state == "wide_divisors":  # over and past the eligible ranges
        c.R[:] = np.exp2(rng.uniform(-8.2, 8.2, W))
        c.C[:] = np.exp2(rng.uniform(-31, 31, W))
        c.L[:] *= np.exp2(rng.uniform(-25, 5, W)).astype(np.float32)
    elif state == "overflow":      # blows up within the first blocks
        c.L[:] = rng.uniform(1e-5, 1e-3, W)
    elif state == "nan_wires":     # all-NaN wires beside finite ones
        c.current[:, some], c.voltage[:, some] = np.nan, np.nan
    elif state == "nan_node":      # NaN spreads along wires from a few nodes
        c.node_voltage[::17] = np.nan
    return c


STATES = ["stable", "zeros", "signed_zeros", "tiny", "tiny_voltages", "equilibrium",
          "unchecked_R", "unchecked_C", "moved", "near_ties", "negative", "wide_divisors",
          "overflow", "nan_wires", "nan_node"]


@pytest.mark.parametrize("shape", [(1, 3, 1), (3, 100, 701), (61, 300, 1201)],
                         ids=lambda s: f"{s[0] * s[2]}w")
@pytest.mark.parametrize("state", STATES)
def test_exact_equals_divide_routine(cuda, oracle, state, shape):
    c = make(oracle, state, *shape)
    for steps in (8, 15, 16, 17, 25, 73, 400):
        a = cnc(cuda, device(c), steps, EXACT)
        b = cnc(cuda, device(c), steps, EXACT_DIVIDE)
        for k in ("current", "voltage"):
            assert same_bits(a[k], b[k]), (steps, k)


@pytest.mark.parametrize("block,wpt", [(128, 1), (256, 1), (128, 2), (256, 2)])
def test_batched_equals_divide_routine(cuda, oracle, block, wpt):
    """The persistent kernel's tiles of both kinds and sizes: one outer loop
    of circuits in several of the states equals the index-space launches
    with the divide routine."""
    from legionorigins_gb300 import batch as B
    from legionorigins_gb300 import circuit as C
    from legionorigins_gb300.workloads import CircuitSpec

    states = ["stable", "zeros", "unchecked_R", "overflow", "near_ties"]
    shapes = [(3, 100, 701), (2, 50, 333), (5, 17, 64), (1, 40, 77), (4, 30, 129)]
    steps = [60, 33, 16, 15, 40]
    circuits = [make(oracle, st, *sh) for st, sh in zip(states, shapes)]
    fields = ["in_ptr", "out_ptr", "in_loc", "out_loc", "L", "R", "C", "current", "voltage",
              "charge", "node_voltage", "cap", "leak", "locator"]
    b = B.Batch([CircuitSpec(*sh, 90.0, 31, s) for sh, s in zip(shapes, steps)],
                [{k: np.ascontiguousarray(getattr(c, k)) for k in fields} for c in circuits])
    b.set_config(block, wpt, 0)
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
