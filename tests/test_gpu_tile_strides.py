"""The tiled node pass on segment strides that are no multiple of 4 (row 9 of
the currents starts off a 16-byte boundary and may end at the last wire), and
on aligned ones, against the gather form: the same bits.  Small graphs take
the gather form by themselves; one whose waits are given a bound takes the
tiled form."""
import ctypes

import numpy as np
import pytest

from test_gpu_dctile import SHAPES, STATE, Strided, tile_info

pytestmark = pytest.mark.gpu

# wires at the edges of chunks (4096) and of 16 bytes
EDGES = {"4097w": (1, 500, 4097, 100, 3), "8191w": (1, 700, 8191, 100, 4),
         "8192w": (2, 400, 4096, 80, 5), "3w": (1, 2, 3, 100, 6), "12290w": (5, 300, 2458, 50, 7)}


@pytest.mark.parametrize("gap", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("fused", [False, True], ids=["dc_uv", "fused"])
@pytest.mark.parametrize("shape", list(SHAPES) + list(EDGES))
def test_tiled_equals_gather(cuda, oracle, shape, fused, gap):
    from legionorigins_gb300 import check, lib
    from legionorigins_gb300 import circuit as C

    c = oracle.generate(oracle.GenParams(*(SHAPES.get(shape) or EDGES[shape]), L_offset=0.001))
    W = c.params.num_pieces * c.params.wires_per_piece
    tiled, gather = Strided(cuda, c, W + gap), Strided(cuda, c, W + gap)
    check(lib().ckt_graph_set_tile_timeout(tiled.dc.graph.handle, 1_000_000_000))
    prm = C.params(2, 0)
    for d in (tiled, gather):
        d.loops(prm, 3, fused)
    a, b = tiled.state(cuda), gather.state(cuda)
    for k in STATE:
        assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k
    assert tile_info(tiled.dc)[3] == 0


@pytest.mark.parametrize("wpp", [32768, 32767])
def test_large_graphs_take_the_tiled_pass(cuda, wpp):
    """Enough nodes for the tiled pass without a bound set, aligned and odd
    strides: the same bits as the per-piece tasks and folds."""
    import torch

    from legionorigins_gb300 import circuit as C

    shape = C.Shape(101, 8000, wpp)
    host = C.generate(101, 8000, wpp, 70.0, 9, 0.001, 0.01)
    host["current"][:] = np.random.default_rng(1).uniform(-1, 1, host["current"].shape)
    prm = C.params(1, 0)
    outs = []
    for per_piece in (False, True):
        dc = C.DeviceCircuit(host, shape)
        if per_piece:
            dc.loop_per_piece(prm)
        else:
            dc.loop_index_space(prm)
        torch.cuda.synchronize()
        outs.append(dc.to_host(("charge", "node_voltage")))
        dc.close()
    for k in outs[0]:
        assert np.array_equal(outs[0][k].view(np.uint32), outs[1][k].view(np.uint32)), k
