"""The device generator where its pieces meet: one wire per piece, a wire
range of less than a group or exactly around a chunk's wires, every wire or no
wire crossing, more groups than a tile of the top walk, runs longer than the
staged span, inductances its fixed-point form does not take, and arrays off a
16-byte boundary -- against the host generator and graph, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    # pieces, nodes, wires per piece, pct, seed, L_offset, L_scale
    (50, 2, 1, 50.0, 3, 0.1, 0.01),          # one wire per piece
    (1, 1, 1, 0.0, 1, 0.1, 0.01),
    (2, 33, 43, 0.0, 2, 0.1, 0.01),          # every wire crosses; two chunks' worth
    (3, 31, 37, 100.0, 5, 0.1, 0.01),        # none does
    (1, 40, 2752, 95.0, 6, 0.1, 0.01),       # a group's most wires
    (7, 97, 2753, 95.0, 7, 0.0, 1.0),
    (4, 64, 3000, 60.0, 8, -0.001, 0.01),    # no fixed-point form: doubles throughout
    (4, 64, 3000, 60.0, 9, 1e-7, 8e-7),
    (2, 24, 1600, 50.0, 10, 0.1, 0.01),      # 133 entries a node: spans above the stage
    (40, 4096, 250000, 90.0, 11, 0.001, 0.01),  # more groups than a tile of the top walk
]


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(str(v) for v in s[:3]))
def test_matches_host(cuda, shape, skew):
    from legionorigins_gb300 import DeviceCircuitArrays, GenParams, check, lib
    from legionorigins_gb300 import circuit as C

    P, npp, wpp, pct, seed, lo, scale = shape
    if skew and P * wpp > 1 << 20:
        pytest.skip("one size of the large circuit is enough")
    W, N = P * wpp, P * npp
    i32, f32, u8 = cuda.int32, cuda.float32, cuda.uint8
    sizes = {"in_ptr": (W, i32), "out_ptr": (W, i32), "in_loc": (W, u8), "out_loc": (W, u8),
             "inductance": (W, f32), "resistance": (W, f32), "capacitance": (W, f32),
             "current": (10 * W, f32), "voltage": (9 * W, f32), "charge": (N, f32),
             "node_voltage": (N, f32), "node_capacitance": (N, f32), "node_leakage": (N, f32),
             "locator": (N, i32), "off": (N + 1, i32), "ent": (2 * W, i32), "slot_in": (W, i32),
             "slot_out": (W, i32), "gstart": ((2 * W + 31) // 32, i32)}
    d = {}
    for k, (n, t) in sizes.items():
        d[k] = cuda.full((n + 2 * skew,), 7, dtype=t, device="cuda")[skew:skew + n]
    arr = DeviceCircuitArrays(*[d[k].data_ptr() for k, _ in DeviceCircuitArrays._fields_])
    gp = GenParams(P, npp, wpp, 0, pct, seed, lo, scale)
    check(lib().ckt_generate_device(ctypes.byref(gp), ctypes.byref(arr), None))
    cuda.cuda.synchronize()
    dev = {k: v.cpu().numpy() for k, v in d.items()}
    h = C.generate(P, npp, wpp, pct, seed, lo, scale)
    for dk, hk in (("in_ptr", "in_ptr"), ("out_ptr", "out_ptr"), ("in_loc", "in_loc"),
                   ("out_loc", "out_loc"), ("inductance", "L"), ("resistance", "R"),
                   ("capacitance", "C"), ("charge", "charge"), ("node_voltage", "node_voltage"),
                   ("node_capacitance", "cap"), ("node_leakage", "leak"), ("locator", "locator"),
                   ("current", "current"), ("voltage", "voltage")):
        assert np.array_equal(dev[dk].view(np.uint8),
                              np.ascontiguousarray(h[hk]).reshape(-1).view(np.uint8)), dk
    g = C.Graph(C.Shape(P, npp, wpp).pieces(), N, h["in_ptr"], h["out_ptr"], h["in_loc"],
                h["out_loc"])
    ref = {"off": np.empty(N + 1, np.uint32), "ent": np.empty(2 * W, np.uint32),
           "slot_in": np.empty(W, np.uint32), "slot_out": np.empty(W, np.uint32),
           "gstart": np.empty((2 * W + 31) // 32, np.uint32)}
    check(lib().ckt_graph_export(g.handle, *[ref[k].ctypes.data for k in ref]))
    for k, v in ref.items():
        assert np.array_equal(dev[k].view(np.uint32), v), k
    g.close()
