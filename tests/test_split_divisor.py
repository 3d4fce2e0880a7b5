"""The check that lets EXACT mode divide by a wire's R or C with a split
quotient fma(a, y, a*yl) (apps/circuit/circuit_gpu.cu:119-128 divides), on
the CPU: divisors it accepts, as made or with yl moved by an ulp, round all
2^23 dividend significands as IEEE division does, in the middle of the
exponent range and at the smallest dividends it is used for."""
import concurrent.futures as cf
import math
import os

import numpy as np
import pytest


def divisors(oracle, verdict, count, lo, hi, odd=True):
    """Random divisors of [lo, hi) with the given verdict."""
    rng = np.random.default_rng(verdict * 2 + odd)
    out = []
    while len(out) < count:
        b = np.float32(math.exp2(rng.uniform(math.log2(lo), math.log2(hi))))
        if (int(b.view(np.uint32)) & 1) == odd and oracle.split_divisor(float(b))[0] == verdict:
            out.append(float(b))
    return out


@pytest.mark.parametrize("verdict,odd", [(1, True), (1, False), (2, True)],
                         ids=["odd", "even", "moved"])
def test_accepted_divisors_round_every_significand(oracle, verdict, odd):
    jobs = []
    for lo, hi in ((2.0 ** -8, 2.0 ** 8), (2.0 ** -30, 2.0 ** 30)):
        for b in divisors(oracle, verdict, 6, lo, hi, odd):
            _, y, yl = oracle.split_divisor(b)
            # 2^-77 |b|: the smallest dividends; rounded up to a binade
            jobs += [(b, y, yl, e) for e in (0, math.frexp(b)[1] - 77)]
    with cf.ThreadPoolExecutor(max(1, min(8, os.cpu_count() or 1))) as ex:
        bad = list(ex.map(lambda j: oracle.split_divisor_sweep(*j), jobs))
    assert [j for j, n in zip(jobs, bad) if n] == []


def test_check_rejects_what_rounds_wrongly(oracle):
    """Rejected divisors do have a dividend that rounds wrongly, and the
    moved ones had one before the move: the check is not merely strict."""
    for verdict, count in ((2, 3), (0, 2)):
        for b in divisors(oracle, verdict, count, 1.0, 2.0):
            f = np.float32
            y = f(1) / f(b)
            exact = (1 - float(f(b)) * float(y)) / b
            assert oracle.split_divisor_sweep(b, float(y), float(f(exact)), 0) == 1
    verdicts = [oracle.split_divisor(float(np.float32(b)))[0]
                for b in np.random.default_rng(5).uniform(1, 2, 40000)]
    assert 0.008 < np.mean(np.array(verdicts) != 1) < 0.018
    assert np.mean(np.array(verdicts) == 0) < 0.002
