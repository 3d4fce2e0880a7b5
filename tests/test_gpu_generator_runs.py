"""The device generator's per-node lists where a warp's 32 nodes have about as
many entries as it stages (384), or more: the counted places and piece flags of
long runs against the host graph, bit for bit."""
import pytest

from test_gpu_generator_edges import test_matches_host as matches_host

pytestmark = pytest.mark.gpu

SHAPES = [
    # pieces, nodes, wires per piece, pct, seed, L_offset, L_scale
    (5, 32, 192, 100.0, 3, 0.1, 0.01),  # 384 entries a warp
    (5, 32, 193, 90.0, 4, 0.1, 0.01),   # and some more, uneven
    (3, 64, 512, 80.0, 5, 0.1, 0.01),   # 16 a node
    (40, 16, 700, 50.0, 6, 0.1, 0.01),  # two pieces a warp, 88 a node, many cross
    (7, 3, 3000, 60.0, 7, 0.1, 0.01),   # eleven pieces a warp, 2000 a node
    (1, 1, 5000, 100.0, 8, 0.1, 0.01),  # all ends at one node
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(str(v) for v in s[:3]))
def test_long_runs_match_host(cuda, shape):
    matches_host(cuda, shape, 1)
