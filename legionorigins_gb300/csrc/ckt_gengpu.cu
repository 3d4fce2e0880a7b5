// ckt_gengpu.cu -- the circuit generator on the device: the same random
// stream, graph and initial values as ckt_generate (load_circuit,
// apps/circuit/circuit.cc:1071-1288), bit for bit, plus the contribution
// graph of the index-space distribute_charge.
//
// drand48 is a 48-bit linear congruential generator, so the state after d
// draws is A_d*x + C_d (mod 2^48) and any position of the stream can be
// reached in log2(d) steps.  Nodes draw 3 values each; a wire draws 6 values
// (in-piece) or 7 (cross-piece), and which one depends on its own 5th draw,
// so wire start positions are a chain through the stream.  The chain is
// decoded in parallel by speculation: the stream is cut into chunks of
// kChunk draws, each chunk is decoded from all 7 possible entry phases (a
// wire starts at most 6 draws past a chunk boundary), the chunks' phase maps
// are composed, by groups of kGroup chunks and then over the groups, to fix
// every group's true entry phase and first wire index, and a block per group
// then emits its wires.  Locations and the graph follow in data-parallel
// kernels; per-node contribution lists are sorted by (wire, end) so the graph
// is identical to the host-built one.
//
// 4,194,304 wires, 1,048,576 nodes on a GB300: 345 us, of which decode 20,
// gen_wires 123 (26 of it zeros, 35 the degree counts' returned adds), place
// 87 (17 zeros; 8.4 M reads and 8.4 M writes at random in L2), csr_finish 66,
// nodes 12, the map composition 15, the scan 13; 600 us when phases hopped
// wire by wire, three expressions per wire ran on the FP64 pipe, degrees and
// lists took a round of atomics each and zeros their own passes.
#include <algorithm>

#include "ckt_drand.cuh"
#include "ckt_internal.h"

namespace ckt {
namespace {

constexpr uint64_t kA = 0x5DEECE66Dull, kC = 0xBull, kMask = 0xffffffffffffull;
constexpr int kChunk = 256;       // draws per chunk
constexpr int kGroup = 64;        // chunks per group
constexpr int kNear = 1024;       // draws reached by one entry of the near table
constexpr int kMapsBlock = 128;   // chunks per block of the decoding

// States reached by N multiples of some number of draws: a[k]*x + c[k].  Each
// table is written by repeated composition, x -> as (a x + c) + cs.
template <int N>
struct Jumps {
  uint64_t a[N], c[N];
};
template <int N>
constexpr Jumps<N> make_multiples(uint64_t as, uint64_t cs) {  // 0, 1, .., N - 1 times (as, cs)
  Jumps<N> j{};
  uint64_t a = 1, c = 0;
  for (int k = 0; k < N; k++) {
    j.a[k] = a;
    j.c[k] = c;
    c = (as * c + cs) & kMask;
    a = (as * a) & kMask;
  }
  return j;
}
constexpr Jumps<48> make_powers() {  // 2^0, 2^1, .. draws
  Jumps<48> j{};
  uint64_t a = kA, c = kC;
  for (int i = 0; i < 48; i++) {
    j.a[i] = a;
    j.c[i] = c;
    c = (a * c + c) & kMask;
    a = (a * a) & kMask;
  }
  return j;
}

// Part of the module's image, so that they are there for whichever stream
// generates first (copied by the first call, through the legacy stream, they
// were not ordered before the kernels of a non-blocking one).  g_near: k
// draws, k < kNear; g_chunk: k chunks, k < kMapsBlock: jumps from a block's
// first draw (lanes index them independently, so they live in global memory,
// not the constant bank).
constexpr Jumps<48> kPowers = make_powers();
__constant__ const Jumps<48> g_jump = kPowers;
static_assert(kChunk == 256, "g_chunk's stride is 2^8 draws");
__device__ const Jumps<kNear> g_near = make_multiples<kNear>(kA, kC);
__device__ const Jumps<kMapsBlock> g_chunk = make_multiples<kMapsBlock>(kPowers.a[8], kPowers.c[8]);

__device__ __forceinline__ uint64_t skip(uint64_t x, uint64_t d) {
  for (int i = 0; d; i++, d >>= 1)
    if (d & 1) x = (g_jump.a[i] * x + g_jump.c[i]) & kMask;
  return x;
}

// Advances the generator state by one draw and returns it (the draw's value
// is x * 2^-48; the drand helpers evaluate the expressions on x).
__device__ __forceinline__ uint64_t next(uint64_t &x) {
  x = (kA * x + kC) & kMask;
  return x;
}

__device__ __forceinline__ uint64_t near_jump(uint64_t x, uint32_t k) {
  return (__ldg(g_near.a + k) * x + __ldg(g_near.c + k)) & kMask;
}
__device__ __forceinline__ uint64_t chunk_jump(uint64_t x, uint32_t k) {
  return (__ldg(g_chunk.a + k) * x + __ldg(g_chunk.c + k)) & kMask;
}

// random_element of the piece's node set (its reversed order, see
// ckt_gen.cpp): first + npp - 1 - (int)(drand48() * npp).
__device__ __forceinline__ uint32_t pick(uint64_t x, uint32_t piece, uint32_t npp) {
  return piece * npp + npp - 1 - drand::trunc_mul_fast(x, npp);
}

struct GenArgs {
  int32_t P, npp, wpp;
  double L_off, L_scale;
  drand::Affine L, C, leak;  // their fixed-point forms
  uint64_t crossing;  // a wire leaves its piece when its 5th draw is at least this
  uint64_t seed_state;
  uint64_t wpp_magic;  // floor(2^64 / wpp) + 1: w / wpp = high64(w * wpp_magic), w < 2^32
  int64_t W, N;
};

// Node values: draws 3x, 3x+1, 3x+2 (circuit.cc:1121-1125).  A node per
// thread, every store coalesced.
__global__ void __launch_bounds__(256)
    gen_nodes_kernel(GenArgs g, float *charge, float *nvolt, float *cap, float *leak,
                     int32_t *locator) {
  __shared__ uint64_t first;
  if (threadIdx.x == 0) first = skip(g.seed_state, 3 * 256 * (uint64_t)blockIdx.x);
  __syncthreads();
  const int64_t n = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (n >= g.N) return;
  uint64_t x = near_jump(first, 3 * threadIdx.x);
  charge[n] = 0.f;
  nvolt[n] = drand::node_voltage(next(x));
  cap[n] = drand::node_capacitance(next(x));
  next(x);
  float l;
  if (!drand::affine_float(x, g.leak, &l))
    l = __double2float_rn(__dmul_rn((double)0.1f, drand::value(x)));
  leak[n] = l;
  locator[n] = 1;
}

// Arrays set to zero beside a kernel's other work, 16 bytes at a time.  The
// currents' and voltages' zeros are 76 bytes a wire, most of the generator's
// memory traffic (47 us of it at the copy rate, beside whichever kernel).
struct Zeroed {
  uint32_t *p[2];
  uint64_t words[2];
};
__device__ __forceinline__ void zero_slice(const Zeroed &z, uint64_t thread, uint64_t threads) {
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const uint64_t off = (0 - (reinterpret_cast<uintptr_t>(z.p[r]) >> 2)) & 3u;
    const uint64_t head = min(z.words[r], off), quads = (z.words[r] - head) / 4;
    const uint64_t tail = head + 4 * quads;
    uint4 *q = reinterpret_cast<uint4 *>(z.p[r] + head);
    for (uint64_t i = thread; i < quads; i += threads) q[i] = make_uint4(0, 0, 0, 0);
    if (thread < head) z.p[r][thread] = 0;
    if (thread < z.words[r] - tail) z.p[r][tail + thread] = 0;
  }
}

// Per chunk and entry phase q: where the chain leaves the chunk (0..6 past
// its end) and how many wires start inside it, as 9 bits (count << 3 | exit)
// at bit 9q; and the crossing test of every draw, as bits.  The chains are
// followed backwards, all at once: a wire that starts at draw s is followed
// by one at s + 6, or s + 7 if draw s + 4 crosses, so f(s) = f(s + 6 or 7)
// with one wire more; the last 8 values of f stay in registers and no lane
// leaves the others (hopping forward from each phase, lanes did: 9,200
// instructions a warp against 3,700).
constexpr int kChunkWords = (kChunk + 4 + 31) / 32;  // a wire's test lies 4 draws past its start

__global__ void __launch_bounds__(kMapsBlock)
    decode_kernel(GenArgs g, int64_t base, int64_t nchunks, uint32_t *bits, uint64_t *maps,
                  Zeroed zero) {
  __shared__ uint64_t first;
  const uint64_t threads = (uint64_t)gridDim.x * kMapsBlock;
  const int64_t c = (int64_t)blockIdx.x * kMapsBlock + threadIdx.x;
  if (threadIdx.x == 0)
    first = skip(g.seed_state, (uint64_t)base + (uint64_t)blockIdx.x * kMapsBlock * kChunk);
  __syncthreads();
  zero_slice(zero, (uint64_t)c, threads);
  if (c >= nchunks) return;
  // the state in the upper 48 bits of y: no masking, and compared as it is
  uint64_t y = chunk_jump(first, threadIdx.x) << 16;
  const uint64_t crossing = g.crossing << 16;
  const bool any = g.crossing >> 48 == 0;  // 2^48: no draw crosses
  uint32_t test[kChunkWords];
#pragma unroll
  for (int wd = 0; wd < kChunkWords; wd++) {
    uint32_t b = 0;
#pragma unroll
    for (int k = 0; k < (wd < kChunk / 32 ? 32 : 4); k++) {
      y = kA * y + (kC << 16);
      if (y >= crossing) b |= 1u << k;
    }
    test[wd] = any ? b : 0u;
    bits[(int64_t)wd * nchunks + c] = test[wd];
  }
  uint32_t f[8];  // f(s) at s mod 8; past the end: no wire, exit s - kChunk
#pragma unroll
  for (uint32_t j = 0; j < 8; j++) f[j] = j;
#pragma unroll
  for (int wd = kChunk / 32 - 1; wd >= 0; wd--) {
    const uint32_t b = __funnelshift_r(test[wd], test[wd + 1], 4);  // bit k: draw 32 wd + k + 4
#pragma unroll
    for (int k = 31; k >= 0; k--)
      f[k & 7] = ((b >> k) & 1u ? f[(k + 7) & 7] : f[(k + 6) & 7]) + 8u;
  }
  uint64_t map = 0;
#pragma unroll
  for (int q = 0; q < 7; q++) map |= (uint64_t)f[q] << (9 * q);
  maps[c] = map;
}

// One chunk's step of a chain at phase ph: 9 bits of its map.
__device__ __forceinline__ uint32_t map_at(uint64_t map, uint32_t ph) {
  return (uint32_t)(map >> (9 * ph)) & 511u;
}

// A group's chunk maps composed, a warp per group, a lane per entry phase:
// wires << 3 | exit phase.
__global__ void __launch_bounds__(128)
    group_maps_kernel(int64_t nchunks, int64_t ngroups, const uint64_t *__restrict__ maps,
                      uint32_t *gmap) {
  __shared__ uint64_t sm[4][kGroup];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const int64_t g = (int64_t)blockIdx.x * 4 + warp;
  if (g >= ngroups) return;
  const int n = (int)min((int64_t)kGroup, nchunks - g * kGroup);
  for (int k = (int)lane; k < n; k += 32) sm[warp][k] = maps[g * kGroup + k];
  __syncwarp();
  if (lane >= 7) return;
  uint32_t ph = lane, wires = 0;
  for (int k = 0; k < n; k++) {
    const uint32_t e = map_at(sm[warp][k], ph);
    wires += e >> 3;
    ph = e & 7u;
  }
  gmap[g * 7 + lane] = wires << 3 | ph;
}

// The chain through the groups from phase 0 (the first wire starts at the
// first wire draw): every group's entry phase and first wire.  One block; a
// tile of groups at a time in shared memory, cut into kTopSegments whose maps
// are composed side by side, then chained, then walked side by side.
constexpr int kTopTile = 4096, kTopSegments = 128;

__global__ void __launch_bounds__(1024)
    top_kernel(int64_t ngroups, const uint32_t *__restrict__ gmap, uint8_t *gphase,
               uint64_t *gbase) {
  extern __shared__ uint32_t sm[];  // [7 * kTopTile]
  __shared__ uint32_t seg[kTopSegments][7];
  __shared__ uint64_t seg_base[kTopSegments];
  __shared__ uint32_t seg_phase[kTopSegments], phase;
  __shared__ uint64_t wires;
  if (threadIdx.x == 0) {
    phase = 0;
    wires = 0;
  }
  for (int64_t g0 = 0; g0 < ngroups; g0 += kTopTile) {
    const int n = (int)min((int64_t)kTopTile, ngroups - g0);
    const int len = (n + kTopSegments - 1) / kTopSegments;
#pragma unroll 8
    for (int i = threadIdx.x; i < 7 * n; i += 1024) sm[i] = gmap[g0 * 7 + i];
    __syncthreads();
    if (threadIdx.x < 7 * kTopSegments) {
      const int q = threadIdx.x % 7, sg = threadIdx.x / 7;
      uint32_t ph = (uint32_t)q, tot = 0;
      for (int k = sg * len; k < min(n, (sg + 1) * len); k++) {
        const uint32_t e = sm[k * 7 + ph];
        tot += e >> 3;
        ph = e & 7u;
      }
      seg[sg][q] = tot << 3 | ph;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t ph = phase;
      uint64_t tot = wires;
      for (int sg = 0; sg < kTopSegments; sg++) {
        seg_phase[sg] = ph;
        seg_base[sg] = tot;
        const uint32_t e = seg[sg][ph];
        tot += e >> 3;
        ph = e & 7u;
      }
      phase = ph;
      wires = tot;
    }
    __syncthreads();
    if (threadIdx.x < kTopSegments) {
      uint32_t ph = seg_phase[threadIdx.x];
      uint64_t tot = seg_base[threadIdx.x];
      for (int k = threadIdx.x * len; k < min(n, ((int)threadIdx.x + 1) * len); k++) {
        gphase[g0 + k] = (uint8_t)ph;
        gbase[g0 + k] = tot;
        const uint32_t e = sm[k * 7 + ph];
        tot += e >> 3;
        ph = e & 7u;
      }
    }
    __syncthreads();
  }
}

// A group's wires (circuit.cc:1158-1186): the chunks' entry phases and the
// wires' starts in shared memory, then a wire per thread: jump to its first
// draw, draw R, L, C, the in-node, the in-piece test and the out-node, store
// every field coalesced, and count the two nodes' degrees.  What a count
// returns is the entry's place among its node's, so that filling the lists
// needs no second round of atomics.
constexpr int kGroupWires = kGroup * ((kChunk + 5) / 6);

__global__ void __launch_bounds__(256)
    gen_wires_kernel(GenArgs g, int64_t base, int64_t nchunks, const uint32_t *__restrict__ bits,
                     const uint64_t *__restrict__ maps, const uint8_t *__restrict__ gphase,
                     const uint64_t *__restrict__ gbase, uint32_t *in_ptr, uint32_t *out_ptr,
                     float *L, float *R, float *C, int32_t *locator, uint32_t *deg,
                     uint32_t *rank_in, uint32_t *rank_out, Zeroed zero) {
  __shared__ uint64_t smaps[kGroup], state[kGroup], first;
  __shared__ uint32_t sbits[kChunkWords][kGroup], before[kGroup + 1], phase[kGroup];
  __shared__ uint16_t starts[kGroupWires];  // chunk << 8 | draw
  zero_slice(zero, (uint64_t)blockIdx.x * 256 + threadIdx.x, (uint64_t)gridDim.x * 256);
  const int64_t c0 = (int64_t)blockIdx.x * kGroup;
  const uint64_t w0 = gbase[blockIdx.x];
  if (w0 >= (uint64_t)g.W) return;  // the stream is cut for 7 draws a wire
  const uint32_t n = (uint32_t)min((int64_t)kGroup, nchunks - c0);
  if (threadIdx.x < n) smaps[threadIdx.x] = maps[c0 + threadIdx.x];
  if (threadIdx.x == 128) first = skip(g.seed_state, (uint64_t)(base + c0 * kChunk));
  for (uint32_t i = threadIdx.x; i < kChunkWords * kGroup; i += 256) {
    const uint32_t wd = i / kGroup, k = i % kGroup;
    if (k < n) sbits[wd][k] = bits[(int64_t)wd * nchunks + c0 + k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t ph = gphase[blockIdx.x], tot = 0;
    for (uint32_t k = 0; k < n; k++) {
      phase[k] = ph;
      before[k] = tot;
      const uint32_t e = map_at(smaps[k], ph);
      tot += e >> 3;
      ph = e & 7u;
    }
    before[n] = tot;
  }
  if (threadIdx.x >= 64 && threadIdx.x < 64 + n)
    state[threadIdx.x - 64] = chunk_jump(first, threadIdx.x - 64);
  __syncthreads();
  if (threadIdx.x < n) {
    uint32_t s = phase[threadIdx.x];
    for (uint32_t i = before[threadIdx.x]; s < (uint32_t)kChunk; i++) {
      starts[i] = (uint16_t)(threadIdx.x << 8 | s);
      s += 6u + ((sbits[(s + 4) >> 5][threadIdx.x] >> ((s + 4) & 31u)) & 1u);
    }
  }
  __syncthreads();
  const uint32_t total = (uint32_t)min((uint64_t)before[n], (uint64_t)g.W - w0);
  for (uint32_t i = threadIdx.x; i < total; i += 256) {
    const uint32_t w = (uint32_t)w0 + i, st = starts[i];
    uint64_t x = near_jump(state[st >> 8], st & 255u);
    const uint64_t xR = next(x), xL = next(x), xC = next(x), xIn = next(x), xPct = next(x);
    const uint32_t piece =
        g.wpp == 1 ? w : (uint32_t)__umul64hi(g.wpp_magic, (uint64_t)w);
    float l, c;
    if (!drand::affine_float(xL, g.L, &l))
      l = __double2float_rn(__dadd_rn(__dmul_rn(drand::value(xL), g.L_scale), g.L_off));
    if (!drand::affine_float(xC, g.C, &c)) c = __double2float_rn(__dmul_rn(drand::value(xC), 0.1));
    const uint32_t a = pick(xIn, piece, (uint32_t)g.npp);
    uint32_t b;
    if (xPct < g.crossing) {
      b = pick(next(x), piece, (uint32_t)g.npp);
    } else {
      uint32_t to = drand::trunc_mul_fast(next(x), (uint32_t)(g.P - 1));
      if (to >= piece) to++;
      b = pick(next(x), to, (uint32_t)g.npp);
      locator[b] = 0;
    }
    rank_in[w] = atomicAdd(deg + a, 1u);
    rank_out[w] = atomicAdd(deg + b, 1u);
    in_ptr[w] = a;
    out_ptr[w] = b;
    R[w] = drand::resistance(xR);
    L[w] = l;
    C[w] = c;
  }
}

// Exclusive scan of deg[0..n) into off[0..n] (off[n] = total), three passes.
constexpr int kScanBlock = 1024, kScanItems = 4;

__global__ void scan_blocks_kernel(const uint32_t *in, int64_t n, uint32_t *out, uint32_t *sums) {
  __shared__ uint32_t warp_tot[32];
  const int64_t i0 = ((int64_t)blockIdx.x * kScanBlock + threadIdx.x) * kScanItems;
  uint32_t v[kScanItems], t = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    v[k] = (i0 + k < n) ? in[i0 + k] : 0u;
    t += v[k];
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = warp_tot[lane], wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    warp_tot[lane] = wi - w;  // exclusive prefix of warp totals
    if (lane == 31) sums[blockIdx.x] = wi;
  }
  __syncthreads();
  uint32_t run = warp_tot[wid] + incl - t;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (i0 + k < n) out[i0 + k] = run;
    run += v[k];
  }
}

// Exclusive scan of the blocks' sums, one block; *total = their sum.
__global__ void __launch_bounds__(1024)
    scan_sums_kernel(uint32_t *sums, int64_t nblocks, uint32_t *total) {
  __shared__ uint32_t warp_tot[32], carry;
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  for (int64_t b0 = 0; b0 < nblocks; b0 += 1024) {
    const int64_t b = b0 + threadIdx.x;
    const uint32_t v = b < nblocks ? sums[b] : 0u;
    uint32_t incl = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    uint32_t before = carry;
    for (uint32_t k = 0; k < wid; k++) before += warp_tot[k];
    if (b < nblocks) sums[b] = before + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// The blocks' sums added, and private nodes marked.  sums NULL: no wires.
__global__ void scan_add_kernel(uint32_t *out, int64_t n, const uint32_t *sums,
                                const int32_t *locator) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t o = sums ? out[i] + sums[i / ((int64_t)kScanBlock * kScanItems)] : 0u;
  out[i] = o | (locator[i] ? kPrivateBit : 0u);
}

// Locations (circuit.cc:1228-1244), and every wire end into its node's list
// at the place its count gave it.
__global__ void __launch_bounds__(256)
    place_kernel(GenArgs g, const uint32_t *__restrict__ in_ptr,
                 const uint32_t *__restrict__ out_ptr, const uint32_t *__restrict__ off,
                 const uint32_t *__restrict__ rank_in, const uint32_t *__restrict__ rank_out,
                 uint8_t *in_loc, uint8_t *out_loc, uint32_t *tmp, Zeroed zero) {
  zero_slice(zero, (uint64_t)blockIdx.x * 256 + threadIdx.x, (uint64_t)gridDim.x * 256);
  const uint32_t w = blockIdx.x * 256 + threadIdx.x;
  if (w >= (uint32_t)g.W) return;
  const uint32_t a = in_ptr[w], b = out_ptr[w], oa = off[a], ob = off[b];
  const uint32_t first = w / (uint32_t)g.wpp * (uint32_t)g.npp;
  in_loc[w] = oa & kPrivateBit ? CKT_PRIVATE_PTR : CKT_SHARED_PTR;
  out_loc[w] = b - first >= (uint32_t)g.npp
                   ? CKT_GHOST_PTR
                   : (ob & kPrivateBit ? CKT_PRIVATE_PTR : CKT_SHARED_PTR);
  tmp[(oa & kOffsetMask) + rank_in[w]] = w << 1;
  tmp[(ob & kOffsetMask) + rank_out[w]] = w << 1 | 1u;
}

// Per node: its contributions in the order of (wire, end), with their
// piece-group flags, the wire ends' slots and the flag bits.  A warp takes 32
// consecutive nodes, whose runs are one contiguous span, staged in shared
// memory.  A lane takes an entry, not a node: its place is the number of
// smaller entries in its run; lanes of one run read the same words, so banks
// hardly conflict (a node per lane, insertion-sorting its run, reads words 8
// apart).  A span larger than the stage is counted from tmp in the same way,
// the entry before found beside the place.  (Insertion-sorted in place, a node
// per lane, its entries nearly in the order of their wires or not: 1024 nodes
// of 128 entries 2.0 / 2.7 ms for the whole generator, 256 of 512 37 / 38 ms,
// 65,536 of 32 409 / 550 us; counted 0.5 and 6.6 ms, 184 us.)
constexpr uint32_t kFinishSpan = 384;  // entries per warp staged (256 on average)

__global__ void __launch_bounds__(256)
    csr_finish_kernel(GenArgs g, const uint32_t *__restrict__ off,
                      const uint32_t *__restrict__ tmp, uint32_t *ent, uint32_t *slot_in,
                      uint32_t *slot_out, uint32_t *gstart) {
  __shared__ uint32_t sbuf[8][kFinishSpan], sout[8][kFinishSpan], soff[8][33];
  __shared__ uint32_t sfirst[8][kFinishSpan / 32];  // bit j: entry j opens a run
  const uint32_t lane = threadIdx.x & 31u, wp = threadIdx.x >> 5;
  const int64_t x0 = ((int64_t)blockIdx.x * 8 + wp) * 32;
  if (x0 >= g.N) return;
  const int64_t xe = min(g.N, x0 + 32);
  const uint32_t b = off[min(x0 + lane, xe)] & kOffsetMask;
  const uint32_t lo = __shfl_sync(0xffffffffu, b, 0), hi = off[xe] & kOffsetMask;
  const uint32_t span = hi - lo;
  // the first wire of a wire's piece
  auto piece_first = [&g](uint32_t w) {
    return g.wpp == 1 ? w : (uint32_t)__umul64hi(g.wpp_magic, (uint64_t)w) * (uint32_t)g.wpp;
  };
  uint32_t *run = soff[wp];
  run[lane] = b - lo;
  if (lane == 0) run[32] = span;
  __syncwarp();
  auto node_of = [run](uint32_t j) {  // the last node whose run starts at or before j
    uint32_t n = 0;
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1)
      if (run[n + step] <= j) n += step;
    return n;
  };
  if (span <= kFinishSpan) {
    uint32_t *buf = sbuf[wp], *out = sout[wp], *opens = sfirst[wp];
    if (lane < kFinishSpan / 32) opens[lane] = 0;
#pragma unroll 4
    for (uint32_t j = lane; j < span; j += 32) buf[j] = tmp[lo + j];
    __syncwarp();
    if (run[lane] < run[lane + 1]) atomicOr(opens + (run[lane] >> 5), 1u << (run[lane] & 31u));
    for (uint32_t j = lane; j < span; j += 32) {
      const uint32_t n = node_of(j), end = run[n + 1], v = buf[j];
      uint32_t place = run[n];
#pragma unroll 4
      for (uint32_t i = place; i < end; i++) place += buf[i] < v ? 1u : 0u;
      out[place] = v;
    }
    __syncwarp();
    for (uint32_t j0 = 0; j0 < span; j0 += 32) {
      const uint32_t j = j0 + lane;
      bool start = false;
      if (j < span) {
        const uint32_t v = out[j], w = v >> 1;
        start = ((opens[j0 >> 5] >> lane) & 1u) || out[j - 1] >> 1 < piece_first(w);
        ent[lo + j] = (w << 2) | ((v & 1u) << 1) | (start ? 1u : 0u);
        if (v & 1u) slot_out[w] = lo + j;
        else slot_in[w] = lo + j;
      }
      // the group-start bits of these 32 entries, into their one or two words
      const uint32_t m = __ballot_sync(0xffffffffu, start);
      if (lane == 0 && m) {
        const uint32_t i0 = lo + j0, sh = i0 & 31u, wd = i0 >> 5;
        atomicOr(gstart + wd, m << sh);
        if (sh && (m >> (32 - sh))) atomicOr(gstart + wd + 1, m >> (32 - sh));
      }
    }
    return;
  }
  for (uint32_t j = lane; j < span; j += 32) {
    const uint32_t n = node_of(j), end = run[n + 1], v = tmp[lo + j], w = v >> 1;
    uint32_t place = run[n], before = 0;  // 1 + the next smaller entry, or 0
#pragma unroll 8
    for (uint32_t i = place; i < end; i++) {
      const uint32_t u = tmp[lo + i];
      place += u < v ? 1u : 0u;
      before = max(before, u < v ? u + 1u : 0u);
    }
    const uint32_t i = lo + place;
    const bool start = before == 0u || (before - 1u) >> 1 < piece_first(w);
    ent[i] = (w << 2) | ((v & 1u) << 1) | (start ? 1u : 0u);
    if (start) atomicOr(gstart + (i >> 5), 1u << (i & 31u));
    if (v & 1u) slot_out[w] = i;
    else slot_in[w] = i;
  }
}

}  // namespace
}  // namespace ckt

using namespace ckt;

extern "C" int ckt_generate_device(const ckt_gen_params *p, ckt_device_circuit *o, void *stream) {
  NvtxRange range("ckt_generate_device");
  CKT_REQUIRE(p != nullptr && o != nullptr, "NULL argument");
  const int32_t P = p->num_pieces, npp = p->nodes_per_piece, wpp = p->wires_per_piece;
  CKT_REQUIRE(P >= 1 && npp >= 1 && wpp >= 0, "bad shape P=%d npp=%d wpp=%d", P, npp, wpp);
  const int64_t N = (int64_t)P * npp, W = (int64_t)P * wpp;
  CKT_REQUIRE(N < 0x7fffffffLL && W <= kMaxWires, "circuit too large (N=%lld W=%lld)",
              (long long)N, (long long)W);
  CKT_REQUIRE(o->charge && o->node_voltage && o->node_capacitance && o->node_leakage &&
                  o->locator && o->off,
              "node arrays are NULL");
  CKT_REQUIRE(W == 0 || (o->in_ptr && o->out_ptr && o->in_loc && o->out_loc && o->inductance &&
                         o->resistance && o->capacitance && o->current && o->voltage && o->ent &&
                         o->slot_in && o->slot_out && o->gstart),
              "wire arrays are NULL");
  const cudaStream_t s = as_stream(stream);
  GenArgs g;
  g.P = P; g.npp = npp; g.wpp = wpp;
  g.crossing = P > 1 ? drand::first_crossing(drand::pct_threshold(p->pct_wire_in_piece))
                     : 1ull << 48;
  g.L_off = p->L_offset; g.L_scale = p->L_scale;
  g.L = drand::make_affine(g.L_scale, g.L_off);
  g.C = drand::make_affine(0.1, 0.0);
  g.leak = drand::make_affine((double)0.1f, 0.0);
  g.seed_state = (((uint64_t)p->random_seed & 0xffffffffull) << 16) | 0x330Eull;
  g.W = W; g.N = N;
  g.wpp_magic = wpp > 1 ? UINT64_MAX / (uint64_t)wpp + 1 : 0;

  gen_nodes_kernel<<<grid_for(N), 256, 0, s>>>(g, o->charge, o->node_voltage, o->node_capacitance,
                                              o->node_leakage, o->locator);
  CKT_CHECK_LAUNCH();
  if (W == 0) {
    // No contributions: the offsets hold the private-node flags only (every
    // node is private); the entry arrays are never touched.
    scan_add_kernel<<<grid_for(N), 256, 0, s>>>(o->off, N, nullptr, o->locator);
    CKT_CHECK_LAUNCH();
    CKT_CUDA(cudaMemsetAsync(o->off + N, 0, 4, s));
    return CKT_OK;
  }

  // Scratch: draw tests, chunk and group maps, degrees and places, unsorted
  // contributions.
  const int64_t base = 3 * N;
  const int64_t nchunks = (7 * W + 8 + kChunk - 1) / kChunk;
  const int64_t ngroups = (nchunks + kGroup - 1) / kGroup;
  const int64_t scan_blocks = (N + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);
  const size_t sz_bits = nchunks * kChunkWords * 4, sz_maps = nchunks * 8, sz_gmap = ngroups * 7 * 4,
               sz_gph = ngroups, sz_gb = ngroups * 8, sz_deg = N * 4,
               sz_sums = (scan_blocks + 1) * 4, sz_rank = W * 4, sz_tmp = 2 * W * 4;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t total = al(sz_bits) + al(sz_maps) + al(sz_gmap) + al(sz_gph) + al(sz_gb) +
                       al(sz_deg) + al(sz_sums) + 2 * al(sz_rank) + al(sz_tmp);
  char *scratch = nullptr;
  CKT_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&scratch), total, s));
  char *q = scratch;
  auto take = [&q, &al](size_t b) {
    char *r = q;
    q += al(b);
    return r;
  };
  uint32_t *bits = (uint32_t *)take(sz_bits);
  uint64_t *maps = (uint64_t *)take(sz_maps);
  uint32_t *gmap = (uint32_t *)take(sz_gmap);
  uint8_t *gphase = (uint8_t *)take(sz_gph);
  uint64_t *gbase = (uint64_t *)take(sz_gb);
  uint32_t *deg = (uint32_t *)take(sz_deg);
  uint32_t *sums = (uint32_t *)take(sz_sums);
  uint32_t *rank_in = (uint32_t *)take(sz_rank);
  uint32_t *rank_out = (uint32_t *)take(sz_rank);
  uint32_t *tmp = (uint32_t *)take(sz_tmp);
  int rc = CKT_OK;
  auto ok = [&rc](cudaError_t e) {
    if (rc == CKT_OK && e != cudaSuccess)
      rc = set_error(CKT_ECUDA, "device generator: %s", cudaGetErrorString(e));
  };

  const Zeroed counts = {{deg, o->gstart}, {(uint64_t)N, (uint64_t)(2 * W + 31) / 32}};
  const Zeroed with_wires = {{reinterpret_cast<uint32_t *>(o->current), nullptr},
                             {10 * (uint64_t)W, 0}};
  const Zeroed with_places = {{reinterpret_cast<uint32_t *>(o->voltage), nullptr},
                              {9 * (uint64_t)W, 0}};
  decode_kernel<<<grid_for(nchunks, kMapsBlock), kMapsBlock, 0, s>>>(g, base, nchunks, bits, maps,
                                                                    counts);
  ok(cudaGetLastError());
  group_maps_kernel<<<grid_for(ngroups, 4), 128, 0, s>>>(nchunks, ngroups, maps, gmap);
  ok(cudaGetLastError());
  ok(cudaFuncSetAttribute(top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          7 * kTopTile * 4));
  top_kernel<<<1, 1024, 7 * 4 * (size_t)std::min<int64_t>(ngroups, kTopTile), s>>>(ngroups, gmap,
                                                                                  gphase, gbase);
  ok(cudaGetLastError());
  gen_wires_kernel<<<(unsigned)ngroups, 256, 0, s>>>(
      g, base, nchunks, bits, maps, gphase, gbase, o->in_ptr, o->out_ptr, o->inductance,
      o->resistance, o->capacitance, o->locator, deg, rank_in, rank_out, with_wires);
  ok(cudaGetLastError());
  scan_blocks_kernel<<<(unsigned)scan_blocks, kScanBlock, 0, s>>>(deg, N, o->off, sums);
  ok(cudaGetLastError());
  scan_sums_kernel<<<1, 1024, 0, s>>>(sums, scan_blocks, o->off + N);
  ok(cudaGetLastError());
  scan_add_kernel<<<grid_for(N), 256, 0, s>>>(o->off, N, sums, o->locator);
  ok(cudaGetLastError());
  place_kernel<<<grid_for(W), 256, 0, s>>>(g, o->in_ptr, o->out_ptr, o->off, rank_in, rank_out,
                                           o->in_loc, o->out_loc, tmp, with_places);
  ok(cudaGetLastError());
  csr_finish_kernel<<<grid_for(N), 256, 0, s>>>(g, o->off, tmp, o->ent, o->slot_in, o->slot_out,
                                                o->gstart);
  ok(cudaGetLastError());
  cudaFreeAsync(scratch, s);
  return rc;
}
