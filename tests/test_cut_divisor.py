"""The form of EXACT mode's split quotient whose product is truncated,
fma(a, y, RZ(a*yl)), which a warp takes for divisors that the rounded product
is not right for (apps/circuit/circuit_gpu.cu:119-128 divides): accepted
divisors round all 2^23 dividend significands as IEEE division does, on the
CPU; on the GPU the dividends next to a rounding boundary, and whole loops
against the divide-routine form."""
import concurrent.futures as cf
import math
import os

import numpy as np
import pytest

from conftest import same_bits


def divisors(oracle, count, lo, hi, twos=None, unchecked=False):
    """Random divisors of [lo, hi): with so many factors of two in the
    significand, or ones that the rounded product is not right for."""
    rng = np.random.default_rng(7 + (twos or 0))
    out = []
    while len(out) < count:
        u = np.float32(math.exp2(rng.uniform(math.log2(lo), math.log2(hi)))).view(np.uint32)
        if twos is not None:
            u = (u >> np.uint32(twos) | np.uint32(1)) << np.uint32(twos)
        b = float(np.uint32(u).view(np.float32))
        if not unchecked or oracle.split_divisor(b)[0] == 0:
            out.append(b)
    return out


@pytest.mark.parametrize("kind", ["unchecked", 0, 1, 2, 3])
def test_accepted_divisors_round_every_significand(oracle, kind):
    jobs, accepted = [], 0
    for lo, hi in ((2.0 ** -8, 2.0 ** 8), (2.0 ** -20, 2.0 ** 30)):
        for b in divisors(oracle, 8, lo, hi, None if kind == "unchecked" else kind,
                          kind == "unchecked"):
            verdict, y, yl = oracle.cut_divisor(b)
            accepted += verdict != 0
            if verdict:
                jobs += [(b, y, yl, e) for e in (0, math.frexp(b)[1] - 77)]
    assert accepted >= 12
    with cf.ThreadPoolExecutor(max(1, min(8, os.cpu_count() or 1))) as ex:
        bad = list(ex.map(lambda j: oracle.cut_divisor_sweep(*j), jobs))
    assert [j for j, n in zip(jobs, bad) if n] == []


@pytest.mark.gpu
@pytest.mark.parametrize("divisor", [0, 1], ids=["R", "C"])
def test_cut_quotient_on_the_gpu(cuda, ckt, divisor):
    c = cuda.zeros(4, dtype=cuda.int64, device="cuda")
    n = 1 << 23
    ckt.check(ckt.tools().ckt_check_cut_quotient(5 + divisor, n, divisor, c.data_ptr(), None))
    cuda.cuda.synchronize()
    bad, checked, _, drawn = c.tolist()
    assert bad == 0 and drawn == n
    eligible = n * (1 if divisor == 0 else 50 / 60)  # as for the rounded product
    assert 0.99 * eligible < checked < 1.002 * eligible


@pytest.mark.gpu
@pytest.mark.parametrize("mix", ["unchecked", "neither", "signs"])
@pytest.mark.parametrize("shape", [(4, 256, 1024), (61, 300, 1201), (30, 2000, 9001)],
                         ids=["lanes", "solo", "paired"])
def test_loops_equal_the_divide_routine(cuda, oracle, shape, mix):
    from test_gpu_exact import EXACT, EXACT_DIVIDE, cnc, device
    c = oracle.generate(oracle.GenParams(*shape, 90, 31, L_offset=0.001))
    rng = np.random.default_rng(3)
    W = c.L.size
    c.L[:] = rng.uniform(1e-7, 9e-7, W)
    for a in (c.current, c.voltage, c.node_voltage):
        a[:] = rng.uniform(-1, 1, a.shape)
    want = divisors(oracle, 6, 1.0, 2.0, unchecked=True)
    some = rng.choice(W, W // 40, replace=False)
    c.R[some] = rng.choice(np.array(want, np.float32), some.size)
    c.C[:] = rng.uniform(1e-3, 1, W)
    c.C[rng.choice(W, W // 40, replace=False)] = np.float32(want[0] * 2.0 ** -9)
    if mix == "neither":  # beside divisors that the truncated product fails for
        bad = []
        while len(bad) < 2:
            b = np.float32(rng.uniform(1, 2))
            if oracle.cut_divisor(float(b))[0] == 0:
                bad.append(b)
        c.R[rng.choice(W, W // 100, replace=False)] = bad[0]
        c.C[rng.choice(W, W // 100, replace=False)] = bad[1] * np.float32(2.0 ** -5)
    elif mix == "signs":
        for d in (c.R, c.C):
            flip = rng.choice(W, W // 3, replace=False)
            d[flip] = -d[flip]
    for steps in (255, 256, 300):
        a = cnc(cuda, device(c), steps, EXACT)
        b = cnc(cuda, device(c), steps, EXACT_DIVIDE)
        for k in ("current", "voltage"):
            assert same_bits(a[k], b[k]), (steps, k)
