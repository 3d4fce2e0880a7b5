"""The tiled node pass on small graphs, which take the gather form unless their
waits are given a bound: test_gpu_dctile's comparisons with the bound set on
every graph whose stride is a multiple of 4, so that the tiled form runs (its
kernel is looked for in a profile of the comparison), and a pass after one whose
waits ran out."""
import ctypes

import numpy as np
import pytest

import test_gpu_dctile as D

pytestmark = pytest.mark.gpu


class Bounded(D.Strided):
    def __init__(self, cuda, c, stride):
        from legionorigins_gb300 import check, lib

        super().__init__(cuda, c, stride)
        if stride % 4 == 0:
            check(lib().ckt_graph_set_tile_timeout(self.dc.graph.handle, 1_000_000_000))


@pytest.fixture
def kernels(cuda, monkeypatch):
    """Runs a function with Strided graphs bounded; the names of its kernels."""
    from torch.profiler import ProfilerActivity, profile

    monkeypatch.setattr(D, "Strided", Bounded)
    with profile(activities=[ProfilerActivity.CUDA]):  # the profiler's own start-up
        cuda.zeros(1, device="cuda").add_(1)
        cuda.cuda.synchronize()

    def run(f, *args):
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            f(*args)
            cuda.cuda.synchronize()
        return [e.key for e in p.key_averages()]

    return run


def took(names, *wanted):
    return all(any(w in n for n in names) for w in wanted)


@pytest.mark.parametrize("shape", sorted(D.SHAPES))
@pytest.mark.parametrize("fused", [False, True], ids=["three_launch", "fused"])
def test_tiled_equals_gather_and_oracle(cuda, oracle, kernels, shape, fused):
    names = kernels(D.test_tiled_equals_gather_and_oracle, cuda, oracle, shape, fused)
    assert took(names, "dc_tile_kernel", "dcuv_kernel" if fused else "dc_all_kernel"), names


def test_nan_currents(cuda, oracle, kernels):
    names = kernels(D.test_nan_currents_propagate_identically, cuda, oracle)
    assert took(names, "dc_tile_kernel", "dcuv_kernel"), names


@pytest.mark.parametrize("shape", ["cfg0", "hub", "tiles_straddle_pieces"])
def test_unaligned_node_arrays(cuda, oracle, kernels, shape):
    names = kernels(D.test_unaligned_node_arrays, cuda, oracle, shape)
    assert took(names, "dc_tile_kernel") and not took(names, "dcuv_kernel"), names


@pytest.mark.parametrize("fused", [False, True], ids=["charge", "fused"])
def test_one_graph_shared_by_two_streams(cuda, oracle, kernels, fused):
    names = kernels(D.test_one_graph_shared_by_two_streams, cuda, oracle, fused)
    assert took(names, "dc_tile_kernel", "ghost_pack_kernel"), names
    assert not took(names, "dcuv_kernel") and not took(names, "dc_all_kernel"), names


def test_tiled_pass_after_a_wait_that_ran_out(cuda, oracle, kernels):
    from legionorigins_gb300 import check, lib
    from legionorigins_gb300 import circuit as C

    c = oracle.generate(oracle.GenParams(*D.SHAPES["tiles_straddle_pieces"], L_offset=0.001))
    W = c.params.num_pieces * c.params.wires_per_piece
    tiled, gather = Bounded(cuda, c, W + 4), Bounded(cuda, c, W + 6)
    L, g, prm = lib(), tiled.dc.graph.handle, C.params(2, 0)
    check(L.ckt_graph_set_tile_timeout(g, 1))
    check(L.ckt_distribute_charge_all(g, tiled.wires(), tiled.dc.nodes(), ctypes.byref(prm), None))
    cuda.cuda.synchronize()
    assert D.tile_info(tiled.dc)[3] == 1
    check(L.ckt_graph_set_tile_timeout(g, 1_000_000_000))
    for d in (tiled, gather):
        for k in ("charge", "node_voltage"):
            d.dc.t[k].copy_(cuda.from_numpy(np.ascontiguousarray(getattr(c, k))))
    names = kernels(tiled.loops, prm, 2, True)
    assert took(names, "dc_tile_kernel"), names
    gather.loops(prm, 2, True)
    a, b = tiled.state(cuda), gather.state(cuda)
    for k in D.STATE:
        assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k
    assert D.tile_info(tiled.dc)[3] == 0
