"""redfold over whole blocks of residues (fold_units_kernel): element counts
around its least one and not a multiple of 2^16, bucket counts around the
shared-memory and 16-bit lines, index wrap-around, other seeds -- against the
oracle; and enough elements that every 16-bit counter overflows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    # buckets, batch size, batches, first batch, seeds
    (1, 1 << 23, 1, 0, (12345, 54321)),
    (977, (1 << 22) + 1, 2, (1 << 10) - 1, (12345, 54321)),  # indices wrap at 2^32
    (51200, 2796203, 3, 0, (12345, 54321)),            # 2^23 + 1 elements
    (51201, 8388607, 1, 0, (12345, 54321)),            # one short: the L2 folds
    (51201, 8388608, 1, 1, (12345, 54321)),
    (115711, 4200001, 2, 0, (0xDEADBEEF, 0x12345678)),
    (115712, 4200001, 2, 0, (0, 0xFFFFFFFF)),
    (115713, 1234567, 7, 3, (12345, 54321)),
    (262144, 65536, 130, 0, (7, 7)),
    (1 << 20, 8400000, 1, 0, (12345, 54321)),
    ((1 << 20) + 1, 8400000, 1, 0, (12345, 54321)),    # the L2 folds
]


def run(cuda, p, schedule):
    from legionorigins_gb300 import check, lib
    from legionorigins_gb300 import reductions as R
    import ctypes

    h = cuda.zeros(p.buckets, dtype=cuda.int32, device="cuda")
    need = max(16, R.scratch_bytes(p, schedule)[1])
    buf = cuda.empty(need, dtype=cuda.uint8, device="cuda")
    check(lib().ckt_hist_run(ctypes.byref(p), schedule, h.data_ptr(), buf.data_ptr(), need, None))
    cuda.cuda.synchronize()
    return h.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(str(v) for v in s[:4]))
def test_fold_matches_oracle(cuda, oracle, shape):
    from legionorigins_gb300 import RED_FOLD
    from legionorigins_gb300 import reductions as R

    buckets, bsize, batches, first, seeds = shape
    want = oracle.histogram(buckets, bsize, batches, first_batch=first, seed1=seeds[0],
                            seed2=seeds[1])
    got = run(cuda, R.params(buckets, bsize, batches, first, *seeds), RED_FOLD)
    assert np.array_equal(got, want)


def test_sixteen_bit_counters_overflow(cuda):
    """2^40 elements over 115,712 buckets: about 62,500 adds per counter and
    block, past 2^15 in each.  The indices repeat every 2^32, so the counts
    are 256 times those of 2^32 elements (mod 2^32)."""
    from legionorigins_gb300 import RED_FOLD, RED_SINGLE
    from legionorigins_gb300 import reductions as R

    once = run(cuda, R.params(115712, 1 << 31, 2), RED_SINGLE)
    many = run(cuda, R.params(115712, 1 << 31, 512), RED_FOLD)
    assert once.sum(dtype=np.uint64) == 1 << 32
    assert np.array_equal(many, once * np.uint32(256))
