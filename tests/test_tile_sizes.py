"""The choice of the node tiles' size, on the CPU: tiles that divide equal
pieces or hold whole ones, unless that takes another wave of blocks (one per
SM); and the plans of such sizes -- small tiles, tiles that drift across the
pieces' edges -- replayed as the kernel walks them (test_tile_plan's program
with the tile size given)."""
import os
import shutil
import subprocess

import pytest

from test_tile_plan import CSRC, CUDA, INCLUDE, SOURCE

MAIN = r'''
static uint32_t chosen(uint32_t P, uint32_t npp, uint32_t sms) {
  std::vector<ckt_piece> pieces(P);
  for (uint32_t k = 0; k < P; k++) pieces[k] = {0u, 0u, k * npp, npp};
  return choose_tile_nodes(pieces.data(), (int32_t)P, P * npp, sms);
}

int main() {
  const struct { uint32_t P, npp, sms, nodes; } sizes[] = {
      {61, 16001, 152, 8004}, {64, 12000, 152, 6000}, {128, 12000, 152, 6000},
      {300, 3000, 152, 6000}, {64, 16384, 152, 8192}, {101, 8000, 152, 8000},
      {1000, 1001, 152, 8008}, {3, 300001, 152, 8112},
      // another wave: 128 tiles and 190, 118 and 160, 127 and 160, 132 and 180
      {95, 11000, 152, 8192}, {320, 3000, 152, 8192}, {80, 13000, 152, 8192},
      {90, 12000, 152, 8192},
      {95, 11000, 200, 5500}, {95, 11000, 100, 5500},  // by the device's count
      {60, 12000, 152, 8192},  // a small graph
      {300, 5000, 152, 8192},  // tiles of 5,000 are too small
      {300, 3000, 0, 8192}};
  int rc = 0;
  for (const auto &s : sizes)
    if (chosen(s.P, s.npp, s.sms) != s.nodes) {
      printf("%u x %u on %u SMs: %u\n", s.P, s.npp, s.sms, chosen(s.P, s.npp, s.sms));
      rc = 1;
    }
  std::vector<ckt_piece> uneven = {{0, 0, 0, 700000}, {0, 0, 700000, 700004}};
  if (choose_tile_nodes(uneven.data(), 2, 1400004, 152) != kTileNodesMax) rc = 1;
  const struct { int P, npp, wpp, ns; double pct; uint32_t nodes; } plans[] = {
      {5, 6001, 24000, 400, 90, 6004},  {7, 3001, 9000, 300, 80, 6004},
      {3, 16001, 64003, 800, 95, 8004}, {9, 1001, 4000, 100, 50, 8008},
      {2, 5501, 8192, 5501, 30, 5504}};
  for (const auto &c : plans) {
    g_tile_nodes = c.nodes;
    const int r = run(c.P, c.npp, c.wpp, c.ns, c.pct, c.nodes);
    printf("tiles of %u: %s\n", c.nodes, r ? "FAILED" : "ok");
    rc |= r;
  }
  return rc;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_tile_sizes_and_their_plans(tmp_path):
    body = SOURCE[:SOURCE.index("int main()")]
    fixed = "const uint32_t TN = kTileNodesMax,"
    assert fixed in body
    body = body.replace(fixed, "const uint32_t TN = g_tile_nodes,").replace(
        "static int run(", "static uint32_t g_tile_nodes;\nstatic int run(")
    src = tmp_path / "tile_sizes_check.cc"
    src.write_text(body + MAIN)
    exe = tmp_path / "tile_sizes_check"
    lib = os.path.join(CUDA, "lib64")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", INCLUDE, "-I", CSRC,
                    "-I", os.path.join(CUDA, "include"), "-o", str(exe), str(src), "-L", lib,
                    "-lcudart", "-lpthread", f"-Wl,-rpath,{lib}"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
