// k32.cu -- kernels of the FP32 form (see k32.cuh for the data layout).
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "grid_loop.cuh"
#include "launch_next.cuh"
#include "k32.cuh"
#include "philox.h"
#include "swap_dev.cuh"
#include "tc05.cuh"

namespace swapk32 {
namespace {

constexpr int TPB = 256;
constexpr int TPB_PASS = 128;  // particle passes: keeps the shared tiles under 48 KB
// Chunk buffers of the particle passes: chunks k+1 .. k+PASS_STAGES-1 are in
// flight while chunk k is processed (more bytes in flight per SM hides more
// of the HBM latency; each stage costs one chunk of shared memory).
#ifndef SWAP_PASS_STAGES
#define SWAP_PASS_STAGES 2
#endif
constexpr int PASS_STAGES = SWAP_PASS_STAGES;
// Polls of a chunk's mbarrier when a pass that gave up lets its copies in
// flight land before it exits (the wait itself is bounded by
// StepParams::wait_polls).
constexpr uint32_t STAGE_WAIT_POLLS = 1u << 22;
// the device error codes of every kernel (swap_dev.cuh), as ints
constexpr int KERR_DOMAIN = swapk::KERR_DOMAIN, KERR_CAPACITY = swapk::KERR_CAPACITY, KERR_MOVE = swapk::KERR_MOVE,
              KERR_WAIT = swapk::KERR_WAIT, KERR_RANGE = swapk::KERR_RANGE;

inline unsigned nblk(long long n, int tpb = TPB) {
  const long long b = (n + tpb - 1) / tpb;
  return (unsigned)(b < 1 ? 1 : b);
}

#define GSTRIDE(t, n) \
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (n); t += (long long)gridDim.x * blockDim.x)

__device__ __forceinline__ void set_err(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

// dirrank of ions the 27-direction sort does not place: a failed move,
// removed, and moved more than one cell (placed from the far list)
constexpr uint32_t DR_BAD = 0xffffffffu, DR_DEAD = 0xfffffffeu, DR_FAR = 0xfffffffdu;

__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// 0-based linear index of 1-based node (i,j,k) in the (nx,ny,nz) layout
__device__ __forceinline__ long long nid(const G32& g, int i, int j, int k) {
  return (long long)(i - 1) + (long long)g.nx * ((long long)(j - 1) + (long long)g.ny * (long long)(k - 1));
}
// Store v at interior node (i,j,k) and at every ghost node whose image it
// is: the periodic fill of boundary.f:9-52 fused into the producer.
template <class T>
__device__ __forceinline__ void store_img(const G32& g, T* f, int i, int j, int k, T v) {
  const int is[2] = {i, i == 2 ? g.nx : (i == g.nx - 1 ? 1 : -1)};
  const int js[2] = {j, j == 2 ? g.ny : (j == g.ny - 1 ? 1 : -1)};
  const int ks[2] = {k, k == 2 ? g.nz : (k == g.nz - 1 ? 1 : -1)};
  for (int a = 0; a < 2; ++a) {
    if (is[a] < 0) continue;
    for (int b = 0; b < 2; ++b) {
      if (js[b] < 0) continue;
      for (int c = 0; c < 2; ++c) {
        if (ks[c] < 0) continue;
        f[nid(g, is[a], js[b], ks[c])] = v;
      }
    }
  }
}

// 32-bit division: t < ncx*ncy*ncz <= 2^30 (64-bit division is a long
// emulated sequence)
__device__ __forceinline__ void interior_of(const G32& g, long long t, int& i, int& j, int& k) {
  const unsigned u = (unsigned)t, nx = (unsigned)g.ncx, ny = (unsigned)g.ncy;
  const unsigned r = u / nx, r2 = r / ny;
  i = (int)(u - r * nx) + 2;
  j = (int)(r - r2 * ny) + 2;
  k = (int)r2 + 2;
}

__host__ __device__ __forceinline__ long long n_int(const G32& g) { return (long long)g.ncx * g.ncy * g.ncz; }

// Move one axis of a (cell, offset) position by d cells; the whole cells
// carried, as a float.  UPPER: offsets in (0,1] (the '>' cell search of x and
// z, gutsp.f:1396-1412); otherwise [0,1) (the floor of y, gutsp.f:1404).  A
// move that is not finite or spans n - 2 cells or more is not made and clears
// ok (below that one wrap always lands in [0, n), gutsp.f:490-510).  No
// branches, and the caller keeps cells unwrapped and takes its brick and sort
// steps from the carries.
template <bool UPPER>
__device__ __forceinline__ float half_step(float& o, float d, int n, bool& ok) {
  const bool fits = fabsf(d) < (float)(n - 2);
  ok = ok && fits;
  o += fits ? d : 0.0f;
  if (UPPER) {
    // o - k > 0 holds exactly and so in floats: a difference of two floats
    // that differ does not round to zero
    const float k = ceilf(o) - 1.0f;
    o -= k;
    return k;
  }
  const float k = floorf(o);
  o -= k;
  const bool edge = o >= 1.0f;  // a tiny negative o rounds up to the open end
  o = edge ? 0.0f : o;
  return edge ? k + 1.0f : k;
}

// A whole number |x| < 2^22 added to FLOAT_INT is an integer in its low bits.
constexpr float FLOAT_INT = 12582912.0f;  // 1.5 * 2^23
__device__ __forceinline__ int float_int(float x) { return __float_as_int(x) - __float_as_int(FLOAT_INT); }

// Offset of a cell from a brick's first cell along one axis, unwrapped across
// the periodic boundary into the brick tile's window [-1, 4] when one of the
// periodic images lies there (n >= 8, so at most one does).
__device__ __forceinline__ int rel_cell(int c, int c0, int n) {
  int r = c - c0;
  if (r < -1) r += n;
  else if (r > 4) r -= n;
  return r;
}

// Step between two cells along one axis, unwrapped into [-1, 1] when one of
// the periodic images lies there.
__device__ __forceinline__ int step_cell(int c, int c0, int n) {
  int r = c - c0;
  if (r < -1) r += n;
  else if (r > 1) r -= n;
  return r;
}

// ---------------------------------------------------------------------------
// particle passes
// ---------------------------------------------------------------------------

__device__ __forceinline__ int dir_index(int dx, int dy, int dz) { return (dx + 1) + 3 * (dy + 1) + 9 * (dz + 1); }

// The warp's deposit (gutsp.f:1484-1491, 1704-1756): the 32 particles' 8
// corner weights and 4 moments go to shared memory as value-major rows; lane
// v = (moment q, corner c) then sums w_c * m_q down the runs of particles
// that share a cell (sorted particles: usually one or two runs), with the run
// ends known to the whole warp (tested per group of four particles), and adds
// each run's sum to the brick tile with one shared atomic.  t0: the tile index
// of the particle's lower corner node, -1 when it deposits nothing.  ALL_Q:
// every moment (otherwise the density, q = 0, is skipped).  An ion that is not
// live brings moments of zero.
// MOVERS (pass 3, which deposits after a half move): the runs follow trun,
// the particle's cell before the move (sorted, so runs stay long), and the
// few particles that changed cell (mover) take no part in them; each of
// those then adds its 32 values to the tile directly, one per lane.
// Exact moment sums (EXACT): a run sum x goes into the tile in fixed point,
// units of 2^-32, split over two 32-bit words per node (low words first, then
// the high words of all nodes): the high word takes h = floor(x * 2^16), the
// low word the rest, l = (x * 2^16 - h) * 2^16 rounded, in [0, 2^16].  Both
// are plain integer reductions (no returned value), exact and commutative,
// so a node's tile value sum(h) * 2^16 + sum(l) is the exact sum of its
// rounded run sums whatever order the warps add in.  The brick partials are
// written as 64-bit integers, summed the same way and rounded to FP32 once
// per node (k_node_sum).  Bounds: |x| < 2^15 per run sum and per node (the
// high words wrap, so only the total must fit); a larger or non-finite run
// sum is reported (KERR_RANGE).  A low word takes at most 2^16 per add and
// an ion adds at most once per node, so every CARRY_CHUNKS chunks of a brick
// the low words carry into the high words and any number of ions fits.
// Otherwise (plain): FP32 atomics, whose result depends on the order.
constexpr float FIX_INV = 1.0f / 4294967296.0f;  // 2^-32
constexpr float FIX_MAX = 32768.0f;             // 2^15
constexpr int CARRY_CHUNKS = 256;               // 32768 ions: the low words stay below 2^32

// x in units of 2^-32 as the tile holds it: floor(x * 2^16) * 2^16 plus the
// rounded rest (the same two conversions as tile_add).
__device__ __forceinline__ long long to_fixed(float x) {
  const float xs = x * 65536.0f, fh = floorf(xs);
  return (long long)__float2int_rn(fh) * 65536LL + (long long)__float2uint_rn((xs - fh) * 65536.0f);
}

template <bool EXACT, int NT>
__device__ __forceinline__ void tile_add(void* tile, int i, float x, unsigned& bad) {
  if (EXACT) {
    // out of range or not finite: noted here, reported once at the pass's end
    // (a branch to the error word in this loop costs the passes 10%); the
    // conversions saturate, so the adds below stay defined
    bad |= fabsf(x) < FIX_MAX ? 0u : 1u;
    // x * 2^16 and its floor are exact floats; their difference is exact and
    // in [0, 1); only the low part rounds, below 2^-32
    const float xs = x * 65536.0f, fh = floorf(xs);
    unsigned* w = static_cast<unsigned*>(tile);
    atomicAdd(w + i, __float2uint_rn((xs - fh) * 65536.0f));
    atomicAdd(w + NT + i, (unsigned)__float2int_rn(fh));  // two's complement
  } else {
    atomicAdd(static_cast<float*>(tile) + i, x);
  }
}

template <bool ALL_Q, int T, bool MOVERS = false, bool EXACT = true>
__device__ __forceinline__ void warp_deposit(float (*red)[36], bool live, int t0, const float (&w8)[8],
                                             const float (&qdv)[4], void* tile, unsigned& bad, int lane,
                                             int trun = -1, bool mover = false) {
#pragma unroll
  for (int c8 = 0; c8 < 8; ++c8) red[c8][lane] = w8[c8];
#pragma unroll
  for (int q = 0; q < 4; ++q) red[8 + q][lane] = MOVERS && mover ? 0.0f : qdv[q];
  __syncwarp();
  const int key = MOVERS ? trun : t0;
  const int tprev = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != tprev);
  const unsigned ends = heads >> 1;  // the particle before each head (and, below, the last one)
  const int qv = lane >> 3, cv = lane & 7;
  const int off = (cv & 1) + T * (((cv >> 1) & 1) + T * (cv >> 2));
  const bool add_here = ALL_Q || qv != 0;
  const float4* wrow = reinterpret_cast<const float4*>(red[cv]);
  const float4* mrow = reinterpret_cast<const float4*>(red[8 + qv]);
  float acc = 0.0f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // two halves of 16 particles, to bound the registers
    float x[16], m[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 v = wrow[4 * h + q], w = mrow[4 * h + q];
      x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
      m[4 * q] = w.x; m[4 * q + 1] = w.y; m[4 * q + 2] = w.z; m[4 * q + 3] = w.w;
    }
#pragma unroll
    for (int g4 = 0; g4 < 4; ++g4) {
      const unsigned e4 = (ends >> (16 * h + 4 * g4)) & 0xfu;
      if (e4 == 0u) {
#pragma unroll
        for (int r = 4 * g4; r < 4 * g4 + 4; ++r) acc = fmaf(x[r], m[r], acc);
      } else {
#pragma unroll
        for (int r = 4 * g4; r < 4 * g4 + 4; ++r) {
          acc = fmaf(x[r], m[r], acc);
          if ((e4 >> (r - 4 * g4)) & 1u) {
            const int tr = __shfl_sync(0xffffffffu, key, 16 * h + r);
            if (add_here && tr >= 0) tile_add<EXACT, 4 * T * T * T>(tile, qv * T * T * T + tr + off, acc, bad);
            acc = 0.0f;
          }
        }
      }
    }
  }
  const int tr = __shfl_sync(0xffffffffu, key, 31);  // the run that ends at the last particle
  if (add_here && tr >= 0) tile_add<EXACT, 4 * T * T * T>(tile, qv * T * T * T + tr + off, acc, bad);
  if (MOVERS) {
    unsigned mv = __ballot_sync(0xffffffffu, live && mover);
    if (mv) {
      __syncwarp();
      if (live && mover) {
#pragma unroll
        for (int q = 0; q < 4; ++q) red[8 + q][lane] = qdv[q];
      }
      __syncwarp();
      while (mv) {
        const int m = __ffs(mv) - 1;
        mv &= mv - 1;
        const int tm = __shfl_sync(0xffffffffu, t0, m);
        if (add_here)
          tile_add<EXACT, 4 * T * T * T>(tile, qv * T * T * T + tm + off, red[cv][m] * red[8 + qv][m], bad);
      }
    }
  }
  __syncwarp();
}

// extrapol_up's velocity (gutsp.f:144), rounded the same wherever it is formed.
__device__ __forceinline__ float extrapolated(float v, float v1) {
  return __fmaf_rn(1.5f, v, -__fmul_rn(0.5f, v1));
}

__device__ __forceinline__ void corner_weights(float ox, float oy, float oz, float (&w8)[8]) {
  const float wxl = 1.0f - ox, wyl = 1.0f - oy, wzl = 1.0f - oz;
#pragma unroll
  for (int c = 0; c < 8; ++c) w8[c] = ((c & 1) ? ox : wxl) * ((c & 2) ? oy : wyl) * ((c & 4) ? oz : wzl);
}

// A crowded brick: carry the low words into the high words (exact: 2^16 low
// units are one high unit), so that they never wrap.  The whole block calls.
template <int TNOD>
__device__ __forceinline__ void carry_tile(unsigned* s_dep) {
  __syncthreads();
  for (int t = threadIdx.x; t < 4 * TNOD; t += blockDim.x) {
    const unsigned lo = s_dep[t];
    s_dep[t] = lo & 0xFFFFu;
    s_dep[4 * TNOD + t] += lo >> 16;
  }
  __syncthreads();
}

// The brick's partial tile: FP32, or the node's fixed-point value (high words *
// 2^16 + low words).
template <bool EXACT, int TNOD>
__device__ __forceinline__ void write_tile(const unsigned* s_dep, void* partial, long long b) {
  if (EXACT) {
    long long* out = static_cast<long long*>(partial) + b * (4 * TNOD);
    for (int t = threadIdx.x; t < 4 * TNOD; t += blockDim.x)
      out[t] = (long long)(int)s_dep[4 * TNOD + t] * 65536LL + (long long)s_dep[t];
  } else {
    float* out = static_cast<float*>(partial) + b * (4 * TNOD);
    for (int t = threadIdx.x; t < 4 * TNOD; t += blockDim.x) out[t] = __uint_as_float(s_dep[t]);
  }
}

// One CTA per brick; its particles are the contiguous range of the brick's
// keys and lie in their key's cell (every move happens in pass 3, after
// which the sort restores that).
//   P1: deposit np and up at v_n = 1.5 v - 0.5 vp1 (maind.f:385-387, 399).
//   P2: gather, Ep, v-/v+, deposit up at 0.5 (v+ + v-) (maind.f:400-402).
//   P3: gather, Ep, v-/v+, vp1 = v, v = v+ + dt/2 Ep (maind.f:404-406), the
//       half move of maind.f:408 and the deposit of np and up at it
//       (:411-413), then the half move of maind.f:479 (v is unchanged by the
//       field subcycles in between), open-x outflow after each move and
//       res_chex after the second (maind.f:484).  It also prepares the sort:
//       the direction of every particle's new cell from its key's cell and
//       its rank among the particles of that key and direction, in order.
// Bound by issue (77% of the slots in P3, 74% in P2) and by shared memory
// (59%, 75%): about 760 warp instructions per 32 ions in P3, 475 in P2.  An
// ion's tile index, key and direction come from its cell word and the whole
// cells it moves, and wraps, outflow and far moves stand in a branch that
// bricks away from the faces take for far ions only: 33.5M ions, P3 0.97 ->
// 0.865 ms (990 instructions when every ion unpacked, wrapped and checked its
// cells).  The barrier after each warp's turn in the ranks stays: letting the
// warps run apart (a named barrier to the next warp, or no barrier after the
// last turn) took P3 to 0.91 and 0.885 ms.
// PGRAD: the isothermal electron-pressure term in the gathered E (kitg:
// its face gradient centred per node, as get_Ep's gradient extension).
template <int PASS, bool CHEX = false, bool EXACT = true, bool PGRAD = false>
__global__ void __launch_bounds__(TPB_PASS, PASS == 3 ? 7 : 8) k_pass(G32 g, Part p, Species sp, StepParams sprm,
                                              const int64_t* __restrict__ start, const float4* __restrict__ kit,
                                              const float4* __restrict__ kitg, void* __restrict__ partial,
                                              uint32_t* __restrict__ dirrank, uint16_t* __restrict__ dep, int* err,
                                              FarList far) {
  // the chunk's particles, copied in by the bulk-copy engine (double-buffered):
  // offsets and v, plus vp1 in P1; cell words; species bytes
  constexpr int NF = PASS == 1 ? 9 : 6, NS = PASS_STAGES;
  __shared__ __align__(128) float s_f[NS][NF][TPB_PASS];
  __shared__ __align__(128) int32_t s_c[NS][TPB_PASS];
  __shared__ __align__(128) uint8_t s_s[NS][TPB_PASS];
  __shared__ uint64_t s_full[NS];
  // the field-gather tile: (aj-up, B_x) and (B_y, B_z) per node
  // deposit tile: T nodes per axis; a cell rx of the brick (rx in [-1,4] for
  // pass 3's movers, [0,3] otherwise) has its lower corner at offset rx + O.
  // The gather happens before any move: its tile is TN_IN wide, origin 0.
  constexpr int T = pass_tile(PASS), TNOD = T * T * T, O = PASS == 3 ? 1 : 0;
  __shared__ float4 s_kitA[PASS == 1 ? 1 : TNODES_IN];
  __shared__ float2 s_kitB[PASS == 1 ? 1 : TNODES_IN];
  __shared__ float4 s_kitG[PGRAD && PASS != 1 ? TNODES_IN : 1];
  // the deposit tile per node and moment: FP32, or (EXACT) fixed point as
  // low words [4 * TNOD] then high words [4 * TNOD]
  __shared__ __align__(8) unsigned s_dep[(EXACT ? 2 : 1) * 4 * TNOD];
  // per warp: [8 weights, 4 moments][particle]; rows padded to 36 floats so
  // that the 8 rows a reducing lane group reads start on different banks
  __shared__ __align__(16) float s_red[TPB_PASS / 32][12][36];
  __shared__ uint16_t s_rank[PASS == 3 ? BCELLS * NDIR : 2];   // running count per (local key, direction)
  const long long b = blockIdx.x;
  const int bi = (int)(b % g.nbx), bj = (int)((b / g.nbx) % g.nby), bk = (int)(b / ((long long)g.nbx * g.nby));
  const int c0x = 4 * bi, c0y = 4 * bj, c0z = 4 * bk;
  const int32_t brick = pk(c0x, c0y, c0z);
  // a brick at the grid's faces: a step of one cell may wrap or leave there
  const bool rim = bi == 0 || bj == 0 || bk == 0 || bi == g.nbx - 1 || bj == g.nby - 1 || bk == g.nbz - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (PASS != 1) {
    for (int t = threadIdx.x; t < TNODES_IN; t += blockDim.x) {
      const int tx = t % TN_IN, ty = (t / TN_IN) % TN_IN, tz = t / (TN_IN * TN_IN);
      const int P = wrapi(c0x - 1 + tx, g.ncx), Q = wrapi(c0y - 1 + ty, g.ncy), R = wrapi(c0z - 1 + tz, g.ncz);
      const long long src = 2 * ((long long)P + (long long)g.ncx * (Q + (long long)g.ncy * R));
      s_kitA[t] = kit[src];
      const float4 hi = kit[src + 1];
      s_kitB[t] = make_float2(hi.x, hi.y);
      if (PGRAD) s_kitG[t] = kitg[src / 2];
    }
  }
  for (int t = threadIdx.x; t < (EXACT ? 2 : 1) * 4 * TNOD; t += blockDim.x) s_dep[t] = 0u;
  if (PASS == 3)
    for (int t = threadIdx.x; t < BCELLS * NDIR; t += blockDim.x) s_rank[t] = 0;
  if (threadIdx.x == 0) {
    for (int q = 0; q < NS; ++q) tc05::mbar_init(&s_full[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  const float hdt = 0.5f * sprm.dt;
  const long long first = start[b * BCELLS], last = start[b * BCELLS + BCELLS];
  // chunks of 128 particles from a 16-aligned start (every copy then starts
  // on a 16-byte boundary); lanes outside [first, last) are masked
  const long long a0 = first & ~15LL;
  const int nchunk = last > first ? (int)((last - a0 + TPB_PASS - 1) / TPB_PASS) : 0;
  // one thread copies chunk k's particle arrays into buffer k % NS
  int issued = 0;  // chunks whose copies thread 0 has started
  auto issue = [&](int k) {
    const int u = k % NS;
    issued = k + 1;
    const long long i0 = a0 + (long long)TPB_PASS * k;
    constexpr uint32_t FB = TPB_PASS * 4;
    tc05::mbar_expect_tx(&s_full[u], (NF + 1) * FB + (p.sp ? TPB_PASS : 0));
    tc05::bulk_g2s(s_c[u], p.cell + i0, FB, &s_full[u]);
    const float* src[9] = {p.ox, p.oy, p.oz, p.vx, p.vy, p.vz, p.wx, p.wy, p.wz};
#pragma unroll
    for (int f = 0; f < NF; ++f) tc05::bulk_g2s(s_f[u][f], src[f] + i0, FB, &s_full[u]);
    if (p.sp) tc05::bulk_g2s(s_s[u], p.sp + i0, TPB_PASS, &s_full[u]);
  };
  if (threadIdx.x == 0)
    for (int k = 0; k < NS - 1 && k < nchunk; ++k) issue(k);
  unsigned n_chex = 0;
  unsigned bad = 0;  // EXACT: a run sum beyond the fixed-point range
  // warp-uniform trip count: every lane takes part in the deposit reduction
  for (int kc = 0; kc < nchunk; ++kc) {
    const int u = kc % NS;
    bool got = true;
    if (threadIdx.x == 0) got = tc05::mbar_wait(&s_full[u], (kc / NS) & 1, sprm.wait_polls);
    // the barrier publishes the chunk to every thread and frees the buffer of
    // chunk kc-1, which every thread is done with: chunk kc+NS-1 goes there
    if (__syncthreads_or(!got)) {
      set_err(err, KERR_WAIT);
      // let the copies still in flight land before the CTA's shared memory
      // is released (each wait bounded)
      if (threadIdx.x == 0)
        for (int k = kc; k < issued; ++k) tc05::mbar_wait(&s_full[k % NS], (k / NS) & 1, STAGE_WAIT_POLLS);
      // pass 3: the brick's ions not reached are dropped by the next sort, so
      // that it sees a consistent set of ranks and counts
      if (PASS == 3 && dirrank)
        for (long long q = a0 + (long long)TPB_PASS * kc + threadIdx.x; q < last; q += TPB_PASS)
          if (q >= first) dirrank[q] = DR_DEAD;
      break;
    }
    if (threadIdx.x == 0 && kc + NS - 1 < nchunk) issue(kc + NS - 1);
    const long long l = a0 + (long long)TPB_PASS * kc + threadIdx.x;
    const bool mine = l >= first && l < last;
    const int32_t c = mine ? s_c[u][threadIdx.x] : CELL_DEAD;
    bool live = c >= 0;  // outside the range, or removed
    if (PASS == 3 && dirrank && !live && mine) dirrank[l] = DR_DEAD;
    if (live && (c & ~(pk(3, 3, 3) | CELL_FRESH)) != brick) {  // not sorted
      set_err(err, KERR_MOVE);
      if (PASS == 3 && dirrank) dirrank[l] = DR_BAD;
      live = false;
    }
    int t0 = -1;
    int t0o = -1;        // P3: tile index of the cell before the move
    int dir = 0, grp = -1;  // P3: the sort's direction; local key * NDIR + dir, -1 when not sorted
    float ox = 0.f, oy = 0.f, oz = 0.f;
    float qdv[4] = {};
    if (live) {
      const int bx4 = pk_i(c) & 3, by4 = pk_j(c) & 3, bz4 = pk_k(c) & 3;  // the ion's cell within the brick
      ox = s_f[u][0][threadIdx.x]; oy = s_f[u][1][threadIdx.x]; oz = s_f[u][2][threadIdx.x];
      float vx = s_f[u][3][threadIdx.x], vy = s_f[u][4][threadIdx.x], vz = s_f[u][5][threadIdx.x];
      int s = p.sp ? min((int)s_s[u][threadIdx.x], MAX_SPECIES - 1) : 0;
      float mr = sp.mrat[s], qw = sp.qw[s];
      float dvx = 0.f, dvy = 0.f, dvz = 0.f;  // velocity deposited
      t0 = (bx4 + O) + T * ((by4 + O) + T * (bz4 + O));
      t0o = t0;
      if (PASS == 1) {
        if (c & CELL_FRESH) p.cell[l] = c & ~CELL_FRESH;
        // extrapol_up (gutsp.f:144)
        dvx = extrapolated(vx, s_f[u][PASS == 1 ? 6 : 0][threadIdx.x]);
        dvy = extrapolated(vy, s_f[u][PASS == 1 ? 7 : 0][threadIdx.x]);
        dvz = extrapolated(vz, s_f[u][PASS == 1 ? 8 : 0][threadIdx.x]);
      } else {
        // trilinear gather of (ajc-upc, btc) at the 8 corners (gutsp.f:217-251)
        const float wxl = 1.0f - ox, wxu = ox, wyl = 1.0f - oy, wyu = oy, wzl = 1.0f - oz, wzu = oz;
        const int tg = bx4 + TN_IN * (by4 + TN_IN * bz4);
        float ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0, qx = 0, qy = 0, qz = 0;
#pragma unroll
        for (int cz = 0; cz < 2; ++cz)
#pragma unroll
          for (int cy = 0; cy < 2; ++cy)
#pragma unroll
            for (int cx = 0; cx < 2; ++cx) {
              const float w = (cx ? wxu : wxl) * (cy ? wyu : wyl) * (cz ? wzu : wzl);
              const int t = tg + cx + TN_IN * (cy + TN_IN * cz);
              const float4 f0 = s_kitA[t];
              const float2 f1 = s_kitB[t];
              ax = fmaf(w, f0.x, ax); ay = fmaf(w, f0.y, ay); az = fmaf(w, f0.z, az);
              bx = fmaf(w, f0.w, bx); by = fmaf(w, f1.x, by); bz = fmaf(w, f1.y, bz);
              if (PGRAD) {
                const float4 f2 = s_kitG[t];
                qx = fmaf(w, f2.x, qx); qy = fmaf(w, f2.y, qy); qz = fmaf(w, f2.z, qz);
              }
            }
        // Ep = ((aj-up) x B - gradP) * mrat (gutsp.f:260-270; q: gradP, zero without PGRAD)
        const float ex = ((ay * bz - az * by) - qx) * mr, ey = ((az * bx - ax * bz) - qy) * mr,
                    ez = ((ax * by - ay * bx) - qz) * mr;
        // v- and the rotation of get_vplus_vminus (gutsp.f:302-397)
        const float mx = vx + hdt * ex, my = vy + hdt * ey, mz = vz + hdt * ez;
        const float Bx = bx * mr, By = by * mr, Bz = bz * mr;
        const float B2 = Bx * Bx + By * By + Bz * Bz;
        const float dt2 = sprm.dt * sprm.dt;
        const float ad = 1.0f / (1.0f + 0.25f * B2 * dt2);
        const float a1 = (1.0f - 0.25f * B2 * dt2) * ad, a2 = sprm.dt * ad, a3 = 0.5f * dt2 * ad;
        const float mdb = mx * Bx + my * By + mz * Bz;
        const float px = a1 * mx + a2 * (my * Bz - mz * By) + a3 * mdb * Bx;
        const float py = a1 * my + a2 * (mz * Bx - mx * Bz) + a3 * mdb * By;
        const float pz = a1 * mz + a2 * (mx * By - my * Bx) + a3 * mdb * Bz;
        if (PASS == 2) {  // improve_up (gutsp.f:422)
          dvx = 0.5f * (px + mx);
          dvy = 0.5f * (py + my);
          dvz = 0.5f * (pz + mz);
        } else {
          // get_vp_final (gutsp.f:444-445).  vp1 = the old v stays where it
          // is: the new v goes into the vp1 arrays, and the host swaps the
          // two after the pass (12 bytes per ion not written)
          vx = px + hdt * ex;
          vy = py + hdt * ey;
          vz = pz + hdt * ez;
          dvx = vx; dvy = vy; dvz = vz;
          // move_ion_half of maind.f:408 (gutsp.f:473-510): the deposit position
          const float mvx = vx * hdt * g.inv_dx, mvy = vy * hdt * g.inv_dy, mvz = vz * hdt * g.inv_dz;
          bool ok = true;
          const float kx = half_step<true>(ox, mvx, g.ncx, ok), ky = half_step<false>(oy, mvy, g.ncy, ok),
                      kz = half_step<true>(oz, mvz, g.ncz, ok);
          const float dox = ox, doy = oy, doz = oz;
          // move_ion_half of maind.f:479: the stored position
          const float lx = half_step<true>(ox, mvx, g.ncx, ok), ly = half_step<false>(oy, mvy, g.ncy, ok),
                      lz = half_step<true>(oz, mvz, g.ncz, ok);
          if (!ok) set_err(err, KERR_MOVE);
          // steps from the ion's own cell, of at most one cell per axis for a
          // near ion: the tile index, the sort's direction and the new cell
          // word are whole numbers below 2^22 and come straight from floats
          const float sx = kx + lx, sy = ky + ly, sz = kz + lz;
          const bool near = fabsf(kx) <= 1.f && fabsf(ky) <= 1.f && fabsf(kz) <= 1.f && fabsf(sx) <= 1.f &&
                            fabsf(sy) <= 1.f && fabsf(sz) <= 1.f;
          t0 += float_int(fmaf((float)(T * T), kz, fmaf((float)T, ky, kx + FLOAT_INT)));
          dir = float_int(fmaf(9.f, sz, fmaf(3.f, sy, sx + (FLOAT_INT + 13.f))));
          int32_t c2 = (c & ~CELL_FRESH) + float_int(fmaf(1048576.f, sz, fmaf(1024.f, sy, sx + FLOAT_INT)));
          bool out1 = false, out2 = false;
          bool far_ion = false;  // moved more than one cell: placed through the far list
          bool beside = near;    // ends in its own cell or next to it
          if (rim || !near) {
            const int ix = (int)kx, iy = (int)ky, iz = (int)kz;
            int cx1 = pk_i(c) + ix, cy1 = pk_j(c) + iy, cz1 = pk_k(c) + iz;  // not wrapped
            const int cx2 = cx1 + (int)lx;
            // outflow through an open x face
            out1 = sprm.x_open && (cx1 < 0 || cx1 >= g.ncx);
            out2 = out1 || (sprm.x_open && (cx2 < 0 || cx2 >= g.ncx));
            // one wrap brings a near ion's cell home, a far one's takes one
            // per half move
            const int ci2 = wrapi(near ? cx2 : wrapi(cx1, g.ncx) + (int)lx, g.ncx),
                      cj2 = wrapi(near ? cy1 + (int)ly : wrapi(cy1, g.ncy) + (int)ly, g.ncy),
                      ck2 = wrapi(near ? cz1 + (int)lz : wrapi(cz1, g.ncz) + (int)lz, g.ncz);
            c2 = pk(ci2, cj2, ck2);
            if (!near) {
              // the periodic image in the tile's window, and next to the ion's
              // own cell, counts: a move about once around the box (33.6M ions,
              // 64 a cell: P3 0.823 -> 0.827 ms with the images looked at)
              const int rx = rel_cell(wrapi(cx1, g.ncx), c0x, g.ncx), ry = rel_cell(wrapi(cy1, g.ncy), c0y, g.ncy),
                        rz = rel_cell(wrapi(cz1, g.ncz), c0z, g.ncz);
              const bool inside = rx >= -1 && rx <= 4 && ry >= -1 && ry <= 4 && rz >= -1 && rz <= 4;
              t0 = inside ? (rx + O) + T * ((ry + O) + T * (rz + O)) : -1;
              const int wx = step_cell(ci2, pk_i(c), g.ncx), wy = step_cell(cj2, pk_j(c), g.ncy),
                        wz = step_cell(ck2, pk_k(c), g.ncz);
              beside = wx >= -1 && wx <= 1 && wy >= -1 && wy <= 1 && wz >= -1 && wz <= 1;
              dir = dir_index(wx, wy, wz);
              // a deposit position outside the tile's window takes the far path too
              far_ion = (!out2 && !beside) || (!out1 && !inside);
            }
          }
          if (CHEX && !out2 && sprm.heavy_of[s] != s) {
            // res_chex (chem_rates.f:823-840) at the end of the step, FP32
            const float x = (float)g.qx1 + ((float)pk_i(c2) + ox) * g.dx - sprm.cloud_x;
            const float y = (float)g.qy1 + ((float)pk_j(c2) + oy) * g.dy - sprm.cloud_y;
            const float z = (float)g.qz1 + ((float)pk_k(c2) + oz) * g.dz - sprm.cloud_z;
            const float vrel = sqrtf(vx * vx + vy * vy + vz * vz);
            const float sigma = vrel > 0.f ? sprm.cx_a - sprm.cx_b * logf(vrel) : 0.f;
            if (sigma > 0.f) {
              const float dens = sprm.cloud_N0 / (1.0f + (x * x + y * y + z * z) * sprm.inv_r0sq);
              const float prob = sprm.dt * dens * sigma * vrel;
              if (swapk::source_uniform_f32(sprm.seed, swapk::RNG_CHEX, sprm.chex_step, l) < prob) {
                vx = vy = vz = 0.f;
                p.vx[l] = 0.f;  // vp1 too
                p.vy[l] = 0.f;
                p.vz[l] = 0.f;
                p.sp[l] = (uint8_t)sprm.heavy_of[s];
                ++n_chex;
              }
            }
          }
          p.wx[l] = vx; p.wy[l] = vy; p.wz[l] = vz;
          if (out2) {
            p.cell[l] = CELL_DEAD;
            if (dirrank) dirrank[l] = DR_DEAD;
          } else {
            p.cell[l] = c2;
            p.ox[l] = ox; p.oy[l] = oy; p.oz[l] = oz;
            if (beside) grp = (bx4 + 4 * by4 + 16 * bz4) * NDIR + dir;
          }
          ox = dox; oy = doy; oz = doz;  // the deposit uses the maind.f:408 position
          if (out1) live = false;
          if (far_ion) {
            const int cx1 = pk_i(c) + (int)kx, cy1 = pk_j(c) + (int)ky, cz1 = pk_k(c) + (int)kz;
            const int slot = far.n ? atomicAdd(far.n, 1) : FAR_CAP;
            if (slot < FAR_CAP) {
              far.idx[slot] = l;
              far.key[slot] = out2 ? -1LL : key_of(g, pk_i(c2), pk_j(c2), pk_k(c2));
              far.dcell[slot] = live ? pk(wrapi(cx1, g.ncx), wrapi(cy1, g.ncy), wrapi(cz1, g.ncz)) : -1;
              far.o[slot] = ox; far.o[FAR_CAP + slot] = oy; far.o[2 * FAR_CAP + slot] = oz;
              far.q[slot] = qw; far.q[FAR_CAP + slot] = qw * dvx;
              far.q[2 * FAR_CAP + slot] = qw * dvy; far.q[3 * FAR_CAP + slot] = qw * dvz;
              atomicAdd(far.total, 1ULL);
              if (!out2 && dirrank) dirrank[l] = DR_FAR;
            } else {
              set_err(err, KERR_MOVE);
              if (!out2 && dirrank) dirrank[l] = DR_BAD;
            }
            grp = -1;
            live = false;  // neither in the tile nor in the ranks
          }
        }
      }
      if (live) {
        qdv[0] = qw;
        qdv[1] = qw * dvx;
        qdv[2] = qw * dvy;
        qdv[3] = qw * dvz;
      }
    }
    // an ion that deposits nothing: moments zero, no tile index
    if (!live) t0 = -1;
    const bool mover = PASS == 3 && t0 != t0o;  // deposits in another cell than its own
    float w8[8];
    corner_weights(ox, oy, oz, w8);
    if (__any_sync(0xffffffffu, live))  // (a brick's last chunk seldom fills its warps)
      warp_deposit<PASS != 2, T, PASS == 3, EXACT>(s_red[warp], live, t0, w8, qdv, s_dep, bad, lane, t0o, mover);
    if (PASS == 3 && dirrank) {
      // stable ranks per (key, direction): the warps of the CTA take their
      // turn in order, each adding its particles after the earlier ones
      const unsigned peers = __match_any_sync(0xffffffffu, grp >= 0 ? grp : -1 - lane);
      const unsigned lt = peers & ((1u << lane) - 1u);
      for (int w = 0; w < TPB_PASS / 32; ++w) {
        if (warp == w) {
          const unsigned before = grp >= 0 ? s_rank[grp] : 0u;
          __syncwarp();
          if (grp >= 0) {
            dirrank[l] = ((uint32_t)dir << 26) | (before + __popc(lt));
            if (lt == 0) s_rank[grp] = (uint16_t)(before + __popc(peers));
          }
        }
        __syncthreads();
      }
    }
    if (EXACT && (kc + 1) % CARRY_CHUNKS == 0 && kc + 1 < nchunk) carry_tile<TNOD>(s_dep);
  }
  if (EXACT && bad) set_err(err, KERR_RANGE);
  if (CHEX) {
    for (int o = 16; o > 0; o >>= 1) n_chex += __shfl_down_sync(0xffffffffu, n_chex, o);
    if (lane == 0 && n_chex) atomicAdd(sprm.chex_count, (unsigned long long)n_chex);
  }
  __syncthreads();
  write_tile<EXACT, TNOD>(s_dep, partial, b);

  if (PASS == 3 && dep)
    for (int t = threadIdx.x; t < BCELLS * NDIR; t += blockDim.x)  // direction-major: dep[dir][key]
      dep[(long long)(t / BCELLS) * g.nkeys + b * BCELLS + t % BCELLS] =
          (uint16_t)s_rank[(t % BCELLS) * NDIR + t / BCELLS];
}

// Pass 1 on ions that the last sort has ranked but not moved: perm[l] is the
// place in src of the ion that belongs at l (~q: new ion q of stage).  Each
// thread copies its ion's fields into shared memory one chunk ahead (4-byte
// asynchronous copies; places two chunks ahead), writes them to dst, and
// deposits them as k_pass<1> does.  The ions so cross HBM once between two
// steps' pushes (86 B and the 4 B of perm) where the sort's scatter (86 B) and
// pass 1 (41 B) each read them: 134M ions, 2.41 ms and 0.45 for the places
// against 2.78 + 1.61.  No thread reads another's copies, so the chunks need
// no barrier.  (Three buffers instead of two: 3.42 ms.)
template <bool EXACT>
__global__ void __launch_bounds__(TPB_PASS, 8) k_pass1_sort(G32 g, Part s, Part n, Part d, Species sp,
                                                            const int64_t* __restrict__ start,
                                                            const int32_t* __restrict__ perm,
                                                            void* __restrict__ partial, int* err) {
  constexpr int T = TN_IN, TNOD = T * T * T, NF = 10;
  __shared__ __align__(16) float s_f[2][NF][TPB_PASS];
  __shared__ unsigned s_dep[(EXACT ? 2 : 1) * 4 * TNOD];
  __shared__ __align__(16) float s_red[TPB_PASS / 32][12][36];
  const long long b = blockIdx.x;
  const int bi = (int)(b % g.nbx), bj = (int)((b / g.nbx) % g.nby), bk = (int)(b / ((long long)g.nbx * g.nby));
  const int32_t brick = pk(4 * bi, 4 * bj, 4 * bk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int t = tid; t < (EXACT ? 2 : 1) * 4 * TNOD; t += TPB_PASS) s_dep[t] = 0u;
  __syncthreads();
  const long long first = start[b * BCELLS], last = start[b * BCELLS + BCELLS];
  const long long a0 = first & ~15LL;  // k_pass<1>'s warps: the same sums, bit for bit
  const int nchunk = last > first ? (int)((last - a0 + TPB_PASS - 1) / TPB_PASS) : 0;
  constexpr int32_t NONE = 0x7fffffff;
  auto place = [&](int k) {
    const long long l = a0 + (long long)TPB_PASS * k + tid;
    return k < nchunk && l >= first && l < last ? perm[l] : NONE;
  };
  // starts the copies of the ion at place q into buffer u; its species byte
  auto fetch = [&](int32_t q, int u) -> int {
    if (q == NONE) return 0;
    const bool old = q >= 0;
    const long long i = old ? q : ~q;
    const void* src[NF] = {old ? (const void*)s.cell : n.cell, old ? s.ox : n.ox, old ? s.oy : n.oy,
                           old ? s.oz : n.oz, old ? s.vx : n.vx, old ? s.vy : n.vy, old ? s.vz : n.vz,
                           old ? s.wx : n.wx, old ? s.wy : n.wy, old ? s.wz : n.wz};
#pragma unroll
    for (int f = 0; f < NF; ++f) tc05::cp_async4(&s_f[u][f][tid], static_cast<const float*>(src[f]) + i);
    return (old ? s.sp : n.sp)[i];
  };
  unsigned bad = 0;
  int32_t q0 = place(0), q1 = place(1);
  int sp0 = fetch(q0, 0), sp1;
  tc05::cp_async_commit();
  for (int kc = 0; kc < nchunk; ++kc) {
    const int u = kc & 1;
    const int32_t q2 = place(kc + 2);
    sp1 = fetch(q1, u ^ 1);
    tc05::cp_async_commit();
    tc05::cp_async_wait<1>();  // this thread's copies of chunk kc have landed
    const long long l = a0 + (long long)TPB_PASS * kc + tid;
    const int32_t c = q0 != NONE ? __float_as_int(s_f[u][0][tid]) & ~CELL_FRESH : CELL_DEAD;
    bool live = q0 != NONE;
    int t0 = -1;
    float ox = 0.f, oy = 0.f, oz = 0.f;
    float qdv[4] = {};
    if (live) {
      ox = s_f[u][1][tid]; oy = s_f[u][2][tid]; oz = s_f[u][3][tid];
      const float vx = s_f[u][4][tid], vy = s_f[u][5][tid], vz = s_f[u][6][tid];
      const float wx = s_f[u][7][tid], wy = s_f[u][8][tid], wz = s_f[u][9][tid];
      d.cell[l] = c;
      d.ox[l] = ox; d.oy[l] = oy; d.oz[l] = oz;
      d.vx[l] = vx; d.vy[l] = vy; d.vz[l] = vz;
      d.wx[l] = wx; d.wy[l] = wy; d.wz[l] = wz;
      d.sp[l] = (uint8_t)sp0;
      const float qw = sp.qw[min(sp0, MAX_SPECIES - 1)];
      if ((c & ~pk(3, 3, 3)) != brick) {  // not sorted
        set_err(err, KERR_MOVE);
        live = false;
      } else {
        t0 = (pk_i(c) & 3) + T * ((pk_j(c) & 3) + T * (pk_k(c) & 3));
        // extrapol_up (gutsp.f:144)
        qdv[0] = qw;
        qdv[1] = qw * extrapolated(vx, wx);
        qdv[2] = qw * extrapolated(vy, wy);
        qdv[3] = qw * extrapolated(vz, wz);
      }
    }
    float w8[8];
    corner_weights(ox, oy, oz, w8);
    if (__any_sync(0xffffffffu, live))
      warp_deposit<true, T, false, EXACT>(s_red[warp], live, t0, w8, qdv, s_dep, bad, lane);
    if (EXACT && (kc + 1) % CARRY_CHUNKS == 0 && kc + 1 < nchunk) carry_tile<TNOD>(s_dep);
    q0 = q1;
    q1 = q2;
    sp0 = sp1;
  }
  tc05::cp_async_wait_all();
  if (EXACT && bad) set_err(err, KERR_RANGE);
  __syncthreads();
  write_tile<EXACT, TNOD>(s_dep, partial, b);
}

// Sum, at every interior node, the brick tiles (T nodes per axis) that cover
// it: along each axis node p lies in the tile of brick floor((p+1+O)/4) at
// offset (p+1+O)%4 and in the one before at offset +4 when that is < T
// (O = 1 for the 7-node tiles, whose origin is one node lower).  The density
// is stored with its ghost images (boundary.f:167-206 fused in).
// All of a node's tile values (up to 8 tiles times NQ moments) are loaded
// before the first is added: a loop over the tiles that are there left one
// load in flight per node (256x128x128 cells, ms per step: 0.57 -> 0.36).
template <int T, int NQ, bool EXACT>
__global__ void k_node_sum(G32 g, const void* partial, float* np, float* S) {
  swapk::after_previous();
  constexpr int O = T == TN ? 1 : 0, TNOD = T * T * T;
  using V = typename std::conditional<EXACT, long long, float>::type;
  GSTRIDE(t, n_int(g)) {
    int i, j, k;
    interior_of(g, t, i, j, k);
    const int P = i - 2, Q = j - 2, R = k - 2;
    // per axis: the tile that starts below the node, and the one before it
    // when it reaches this far
    const int ox = (P + 1 + O) & 3, oy = (Q + 1 + O) & 3, oz = (R + 1 + O) & 3;
    int bx = (P + 1 + O) >> 2, by = (Q + 1 + O) >> 2, bz = (R + 1 + O) >> 2;
    if (bx >= g.nbx) bx -= g.nbx;
    if (by >= g.nby) by -= g.nby;
    if (bz >= g.nbz) bz -= g.nbz;
    const int bx1 = bx == 0 ? g.nbx - 1 : bx - 1, by1 = by == 0 ? g.nby - 1 : by - 1, bz1 = bz == 0 ? g.nbz - 1 : bz - 1;
    V v[8][NQ];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const bool there = (!(c & 1) || ox + 4 < T) && (!(c & 2) || oy + 4 < T) && (!(c & 4) || oz + 4 < T);
      const long long brick =
          (c & 1 ? bx1 : bx) + (long long)g.nbx * ((c & 2 ? by1 : by) + (long long)g.nby * (c & 4 ? bz1 : bz));
      const V* src = static_cast<const V*>(partial) + brick * (4 * TNOD) + (ox + (c & 1 ? 4 : 0)) +
                     T * ((oy + (c & 2 ? 4 : 0)) + T * (oz + (c & 4 ? 4 : 0)));
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[c][q] = there ? src[(4 - NQ + q) * TNOD] : (V)0;
    }
    float acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      V s = v[0][q];
      // (plain form: the order of the tiles is x outermost)
#pragma unroll
      for (int r = 1; r < 8; ++r) s += v[(r >> 2 & 1) | (r & 2) | (r & 1) << 2][q];
      // exact: the one rounding of the sum, from the 64-bit integer (by way of
      // double the FP64 pipe bound it; 1M nodes, mean of a step's three sums:
      // 37.4 -> 33.5 us)
      acc[q] = EXACT ? __ll2float_rn((long long)s) * FIX_INV : (float)s;
    }
    const long long o = nid(g, i, j, k);
    if (NQ == 4) store_img(g, np, i, j, k, acc[0]);  // np with its ghost images
    S[o] = acc[NQ - 3];
    S[o + g.C] = acc[NQ - 2];
    S[o + 2 * g.C] = acc[NQ - 1];
  }
}

// ---------------------------------------------------------------------------
// fields (interior nodes, ghost images written by the producer)
// ---------------------------------------------------------------------------

// The isothermal electron-pressure gradient at the face of component m
// (node o to o + e_m): grad_pe * (np(o+e_m) - np(o)) / d_m / n_face, n_face
// the face average of np as in curlB.
template <int m, class I = long long>
__device__ __forceinline__ float gpe_face(const G32& g, const float* np, float gp, I o) {
  const I s = m == 0 ? (I)1 : (m == 1 ? (I)g.nx : (I)g.nx * (I)g.ny);
  const float inv = m == 0 ? g.inv_dx : (m == 1 ? g.inv_dy : g.inv_dz);
  return gp * ((np[o + s] - np[o]) * inv) / (0.5f * (np[o] + np[o + s]));
}

// ---- the field subcycle: two fused kernels per half step ----
//
// Launched over the interior nodes as a 3D grid (no index division).  Every
// field keeps its periodic ghost images (written by store_img), so a value at
// a ghost coordinate is computed at the interior image.

constexpr int FBX = 32, FBY = 4;

// Bring `bytes` (a multiple of 16) from the 16-byte boundary at or below p to L2.
__device__ __forceinline__ void prefetch_l2(const float* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((unsigned long long)p & ~15ull), "r"(bytes));
}

#define FIELD_NODE(i, j, k)                                   \
  const int i = blockIdx.x * FBX + threadIdx.x + 2;          \
  const int j = blockIdx.y * FBY + threadIdx.y + 2;          \
  const int k = blockIdx.z + 2;                              \
  if (i > g.ncx + 1 || j > g.ncy + 1) return

// Neighbours by 32-bit offsets, at the periodic image where the
// neighbour is a ghost.  Every load of a node stands before its first store:
// one round trip to memory per node, also on the boundary; and the ghost
// images of all outputs are stored together.  (A separate path for boundary
// nodes that mapped each neighbour's index and stored each output's images on
// its own: 20 steps of 128x64x64 cells 46.9 ms against 42.9, of 256x128x128
// cells 338 against 331; in the field loop below 307 us a step of 64x32x32
// cells against 182.)

// Offsets are in bytes and 32 bits wide (addressable(), k32.cuh), beside
// bases that the whole grid shares: the address of a load is then its base
// and one register (20 steps of 128x64x64 cells with 64-bit element indices
// 16.2 ms against 16.0).
struct Off {
  int xm, xp, ym, yp, zm, zp;
};
struct In {
  const float* p;
  __device__ __forceinline__ float operator[](unsigned at) const {
    return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + at);
  }
};
__device__ __forceinline__ void put(float* p, unsigned at, float v) {
  *reinterpret_cast<float*>(reinterpret_cast<char*>(p) + at) = v;
}
__device__ __forceinline__ unsigned at_node(const G32& g, int i, int j, int k) {
  return 4u * ((unsigned)(i - 1) + (unsigned)g.nx * ((unsigned)(j - 1) + (unsigned)g.ny * (unsigned)(k - 1)));
}
__device__ __forceinline__ Off off_of(const G32& g, int i, int j, int k) {
  const int sy = 4 * g.nx, sz = 4 * g.nx * g.ny;
  Off d;
  d.xm = i == 2 ? 4 * (g.ncx - 1) : -4;
  d.xp = i == g.nx - 1 ? 4 * (1 - g.ncx) : 4;
  d.ym = j == 2 ? (g.ncy - 1) * sy : -sy;
  d.yp = j == g.ny - 1 ? (1 - g.ncy) * sy : sy;
  d.zm = k == 2 ? (g.ncz - 1) * sz : -sz;
  d.zp = k == g.nz - 1 ? (1 - g.ncz) * sz : sz;
  return d;
}

// v[q] at the ghost images of node (i,j,k) in f[q] (at least 8 cells per axis:
// one image per axis at most).
template <int N>
__device__ __forceinline__ void ghost_images(const G32& g, int i, int j, int k, float* const (&f)[N],
                                             const float (&v)[N]) {
  const int di = i == 2 ? g.ncx : (i == g.nx - 1 ? -g.ncx : 0), dj = j == 2 ? g.ncy : (j == g.ny - 1 ? -g.ncy : 0),
            dk = k == 2 ? g.ncz : (k == g.nz - 1 ? -g.ncz : 0);
  if (!(di | dj | dk)) return;
  const long long o = nid(g, i, j, k);
  const int x = di, y = dj * g.nx, z = dk * g.nx * g.ny;
  if ((di != 0) + (dj != 0) + (dk != 0) == 1) {  // a face: one image
    const long long t = o + x + y + z;
#pragma unroll
    for (int q = 0; q < N; ++q) f[q][t] = v[q];
    return;
  }
#pragma unroll 1
  for (int c = 1; c < 8; ++c) {
    if (((c & 1) && !x) || ((c & 2) && !y) || ((c & 4) && !z)) continue;
    const long long t = o + ((c & 1) ? x : 0) + ((c & 2) ? y : 0) + ((c & 4) ? z : 0);
#pragma unroll
    for (int q = 0; q < N; ++q) f[q][t] = v[q];
  }
}

// dB at a node and its lower neighbours: what curl dB there and one step down
// each axis and the centred B need.
struct Stencil {
  float b1, b1y, b1z, b1yz, b2, b2x, b2z, b2xz, b3, b3x, b3y, b3xy;
};
__device__ __forceinline__ Stencil stencil_of(const G32& g, const float* db, unsigned o, const Off& d) {
  const In B1{db}, B2{db + g.C}, B3{db + 2 * g.C};
  return Stencil{B1[o], B1[o + d.ym], B1[o + d.zm], B1[o + d.ym + d.zm], B2[o], B2[o + d.xm], B2[o + d.zm],
                 B2[o + d.xm + d.zm], B3[o], B3[o + d.xm], B3[o + d.ym], B3[o + d.xm + d.ym]};
}
// Component m of curl dB (gutsf.f:202-239) at the node, and (curl_down) one
// step down axis m.
__device__ __forceinline__ float curl_term(float f, float fm, float gm, float h, float i1, float i2) {
  return (f - fm) * i1 + (gm - h) * i2;
}
template <int m>
__device__ __forceinline__ float curl_at(const G32& g, const Stencil& s) {
  if (m == 0) return curl_term(s.b3, s.b3y, s.b2z, s.b2, g.inv_dy, g.inv_dz);
  if (m == 1) return curl_term(s.b1, s.b1z, s.b3x, s.b3, g.inv_dz, g.inv_dx);
  return curl_term(s.b2, s.b2x, s.b1y, s.b1, g.inv_dx, g.inv_dy);
}
template <int m>
__device__ __forceinline__ float curl_down(const G32& g, const Stencil& s) {
  if (m == 0) return curl_term(s.b3x, s.b3xy, s.b2xz, s.b2x, g.inv_dy, g.inv_dz);
  if (m == 1) return curl_term(s.b1y, s.b1yz, s.b3xy, s.b3y, g.inv_dz, g.inv_dx);
  return curl_term(s.b2z, s.b2xz, s.b1yz, s.b1z, g.inv_dx, g.inv_dy);
}
// Cell-centre B from the edge field's values at the node, one step down two
// axes, and both (edge_to_center, grid_interp.f:35-51, with ratios 1/2).
__device__ __forceinline__ float centre(float v, float v1, float v2, float v12) {
  return 0.25f * ((v2 + v12) + (v + v1));  // (the halvings of each average are exact)
}

// ct = S/np (zero where no ion deposits; the fast divide, two ulps: n is a
// density, far from where it loses accuracy).
__device__ __forceinline__ float ct_of(float s, float n) { return n == 0.0f ? 0.0f : __fdividef(s, n); }

// The approximate reciprocal of a normal number: a times it is the fast divide
// without the scaling that __fdividef keeps for denormals.
__device__ __forceinline__ float reciprocal(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// update_up's face average (gutsp.f:1825-1836) of ct, with ghost images, and
// the whistler Courant time of check_time_step (gutsf.f:1782-1792) per node,
// ghosts included, with its smallest value.  look[0]: that value (set large
// before); look[1]: the error word as it stands (see field_loop).
__global__ void __launch_bounds__(TPB) k_up_courant(G32 g, const float* np, const float* S,
                                                    const float* db, const float* b0c,
                                                    float alpha, float dx, float* up,
                                                    float* dtn, unsigned* look, const int* err) {
  swapk::after_previous();
  float mn = 3.0e38f;
  if (blockIdx.x == 0 && threadIdx.x == 0) look[1] = (unsigned)*err;
  GSTRIDE(t, n_int(g)) {
    int i, j, k;
    interior_of(g, t, i, j, k);
    const Off d = off_of(g, i, j, k);
    const long long C = g.C;
    const unsigned o = at_node(g, i, j, k);
    const In s1{S}, s2{S + C}, s3{S + 2 * C}, N{np}, D1{db}, D2{db + C}, D3{db + 2 * C};
    const float n = N[o], nx = N[o + d.xp], ny = N[o + d.yp], nz = N[o + d.zp];
    const float a0 = s1[o], a1 = s1[o + d.xp], c0 = s2[o], c1 = s2[o + d.yp], e0 = s3[o], e1 = s3[o + d.zp];
    const float b1 = D1[o] + b0c[0], b2 = D2[o] + b0c[1], b3 = D3[o] + b0c[2];
    const float btot = sqrtf(b1 * b1 + b2 * b2 + b3 * b3);
    const float ak = 2.0f / dx;
    const float q1 = ak * ak * btot / (alpha * n);
    const float q2 = (ak * btot) * (ak * btot) / (alpha * n);
    const float womega = 0.5f * (q1 + sqrtf(q1 * q1 + 4.0f * q2));
    const float dt = dx / (womega / ak);
    mn = fminf(mn, dt > 0.0f ? dt : 0.0f);
    float* const f[4] = {up, up + C, up + 2 * C, dtn};
    const float v[4] = {0.5f * (ct_of(a0, n) + ct_of(a1, nx)), 0.5f * (ct_of(c0, n) + ct_of(c1, ny)),
                        0.5f * (ct_of(e0, n) + ct_of(e1, nz)), dt};
#pragma unroll
    for (int q = 0; q < 4; ++q) put(f[q], o, v[q]);
    ghost_images(g, i, j, k, f, v);
  }
  // one atomic per block (a grid of a few per SM): atomics from every warp to
  // the one address serialise in L2
  __shared__ float s_mn[TPB / 32];
  for (int off = 16; off > 0; off >>= 1) mn = fminf(mn, __shfl_down_sync(0xffffffffu, mn, off));
  if ((threadIdx.x & 31) == 0) s_mn[threadIdx.x >> 5] = mn;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mn = fminf(mn, s_mn[w]);
    atomicMin(look, __float_as_uint(mn));
  }
}

// The passes' gather kit per physical node, from the moment sums and dB
// alone: (ajc - upc, btc) with aj of curlB (gutsf.f:202-239) and up of
// update_up (gutsp.f:1825-1836) at the node and one step down each axis,
// face_to_center (grid_interp.f:163-170) of their difference, and
// edge_to_center of dB plus the centred b0.  (256x128x128 cells, ms per
// step with k_up_courant: 0.33; as up, curlB, kit and the Courant time in
// kernels of their own with their arrays in between: 0.47.)
// kitg (may be null): the pressure gradient centred like aj, for get_Ep.
// Thread 0 also resets the far list's count and the Courant word, which the
// rest of the step writes.
__global__ void __launch_bounds__(TPB) k_kit(G32 g, const float* S, const float* db,
                                             const float* b0c, const float* np, float alpha,
                                             float gp, float4* kit, float4* kitg, int* far_n,
                                             unsigned* look) {
  swapk::after_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *far_n = 0;
    look[0] = 0x7f7fffffu;  // FLT_MAX
  }
  GSTRIDE(t, n_int(g)) {
    int i, j, k;
    interior_of(g, t, i, j, k);
    const Off d = off_of(g, i, j, k);
    const long long C = g.C;
    const unsigned o = at_node(g, i, j, k);
    const Stencil s = stencil_of(g, db, o, d);
    const In N{np}, s1{S}, s2{S + C}, s3{S + 2 * C};
    const float n0 = N[o], nxm = N[o + d.xm], nxp = N[o + d.xp], nym = N[o + d.ym], nyp = N[o + d.yp],
                nzm = N[o + d.zm], nzp = N[o + d.zp];
    const float x0 = ct_of(s1[o], n0), xm = ct_of(s1[o + d.xm], nxm), xp = ct_of(s1[o + d.xp], nxp);
    const float y0 = ct_of(s2[o], n0), ym = ct_of(s2[o + d.ym], nym), yp = ct_of(s2[o + d.yp], nyp);
    const float z0 = ct_of(s3[o], n0), zm = ct_of(s3[o + d.zm], nzm), zp = ct_of(s3[o + d.zp], nzp);
    const float ux = 0.5f * (x0 + xp), uxm = 0.5f * (xm + x0), uy = 0.5f * (y0 + yp), uym = 0.5f * (ym + y0),
                uz = 0.5f * (z0 + zp), uzm = 0.5f * (zm + z0);
    const float a1 = curl_at<0>(g, s) / (0.5f * (n0 + nxp) * alpha), a1m = curl_down<0>(g, s) / (0.5f * (nxm + n0) * alpha);
    const float a2 = curl_at<1>(g, s) / (0.5f * (n0 + nyp) * alpha), a2m = curl_down<1>(g, s) / (0.5f * (nym + n0) * alpha);
    const float a3 = curl_at<2>(g, s) / (0.5f * (n0 + nzp) * alpha), a3m = curl_down<2>(g, s) / (0.5f * (nzm + n0) * alpha);
    kit[2 * t] = make_float4(0.5f * ((a1 - ux) + (a1m - uxm)), 0.5f * ((a2 - uy) + (a2m - uym)),
                             0.5f * ((a3 - uz) + (a3m - uzm)), centre(s.b1, s.b1y, s.b1z, s.b1yz) + b0c[0]);
    kit[2 * t + 1] = make_float4(centre(s.b2, s.b2x, s.b2z, s.b2xz) + b0c[1],
                                 centre(s.b3, s.b3y, s.b3x, s.b3xy) + b0c[2], 0.0f, 0.0f);
    if (kitg) {
      const unsigned n = o / 4, sy = (unsigned)g.nx, sz = (unsigned)(g.nx * g.ny);
      kitg[t] = make_float4(0.5f * (gpe_face<0>(g, np, gp, n) + gpe_face<0>(g, np, gp, n - 1u)),
                            0.5f * (gpe_face<1>(g, np, gp, n) + gpe_face<1>(g, np, gp, n - sy)),
                            0.5f * (gpe_face<2>(g, np, gp, n) + gpe_face<2>(g, np, gp, n - sz)), 0.0f);
    }
  }
}

// curlB (gutsf.f:202-239; curl b0 = 0 for the uniform b0), face_to_center(aj -
// up) and the cross product of get_E (gutsf.f:1059-1075, crossf2 gutsf.f:
// 65-76): writes aj and ct.  Predictor: B at cell centres from edge_to_center
// of dB (grid_interp.f:35-51).  Corrector: B at m+1/2 through edge_to_face
// then face_to_center (gutsf.f:1268-1269), i.e. component m is the 1-2-1
// average along axis m of edge_to_center.  The divide is the fast one (two
// ulps): the denominator, a density times alpha, is far from the range where
// it loses accuracy.
// Bound by issue (ncu, 4.2M nodes: 86 and 89% of the slots in the predictor and
// the corrector, b_step 79 and 66%), so the halvings are folded, the quotient
// is two instructions and a face node stores its one image without the loop
// over all seven: 20 steps of 4 ions a cell, 64x64x64 9.91 -> 9.28 ms,
// 128x64x64 15.97 -> 15.27, 256x128x128 105.5 -> 103.4; the same bits.
// FaceTerms: what the density and up give there, the same in every subcycle:
// the reciprocals of the face densities times alpha at the node (r) and one
// step down each axis (rm), and up there.
struct FaceTerms {
  float r1, r2, r3, r1m, r2m, r3m, ux, uxm, uy, uym, uz, uzm;
};
__device__ __forceinline__ FaceTerms face_terms(const G32& g, const float* np, const float* up, float alpha, int i,
                                                int j, int k) {
  const Off d = off_of(g, i, j, k);
  const unsigned o = at_node(g, i, j, k);
  const In u1{up}, u2{up + g.C}, u3{up + 2 * g.C}, N{np};
  const float n0 = N[o], nxm = N[o + d.xm], nxp = N[o + d.xp], nym = N[o + d.ym], nyp = N[o + d.yp],
              nzm = N[o + d.zm], nzp = N[o + d.zp];
  FaceTerms f;
  f.ux = u1[o]; f.uxm = u1[o + d.xm]; f.uy = u2[o]; f.uym = u2[o + d.ym]; f.uz = u3[o]; f.uzm = u3[o + d.zm];
  const float ha = 0.5f * alpha;
  f.r1 = reciprocal((n0 + nxp) * ha); f.r2 = reciprocal((n0 + nyp) * ha); f.r3 = reciprocal((n0 + nzp) * ha);
  f.r1m = reciprocal((nxm + n0) * ha); f.r2m = reciprocal((nym + n0) * ha); f.r3m = reciprocal((nzm + n0) * ha);
  return f;
}
template <bool CORR>
__device__ __forceinline__ void aj_ct_node(const G32& g, const float* db, const FaceTerms& ft, const float* b0c,
                                           float* aj, float* ct, int i, int j, int k) {
  const Off d = off_of(g, i, j, k);
  const long long C = g.C;
  const unsigned o = at_node(g, i, j, k);
  const Stencil s = stencil_of(g, db, o, d);
  // the same four values one step down and up the component's own axis
  float m[3][4], p[3][4];
  if (CORR) {
    const int e[3][3] = {{0, d.ym, d.zm}, {0, d.xm, d.zm}, {0, d.ym, d.xm}};
    const int lo[3] = {d.xm, d.ym, d.zm}, hi[3] = {d.xp, d.yp, d.zp};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const In B{db + C * q};
      const unsigned a = o + lo[q], b = o + hi[q];
      m[q][0] = B[a]; m[q][1] = B[a + e[q][1]]; m[q][2] = B[a + e[q][2]]; m[q][3] = B[a + e[q][1] + e[q][2]];
      p[q][0] = B[b]; p[q][1] = B[b + e[q][1]]; p[q][2] = B[b + e[q][2]]; p[q][3] = B[b + e[q][1] + e[q][2]];
    }
  }
  const float c0x = b0c[0], c0y = b0c[1], c0z = b0c[2];
  const float a1 = curl_at<0>(g, s) * ft.r1;
  const float a2 = curl_at<1>(g, s) * ft.r2;
  const float a3 = curl_at<2>(g, s) * ft.r3;
  const float a1m = curl_down<0>(g, s) * ft.r1m;
  const float a2m = curl_down<1>(g, s) * ft.r2m;
  const float a3m = curl_down<2>(g, s) * ft.r3m;
  const float ax = 0.5f * ((a1 - ft.ux) + (a1m - ft.uxm));
  const float ay = 0.5f * ((a2 - ft.uy) + (a2m - ft.uym));
  const float az = 0.5f * ((a3 - ft.uz) + (a3m - ft.uzm));
  float bx = centre(s.b1, s.b1y, s.b1z, s.b1yz), by = centre(s.b2, s.b2x, s.b2z, s.b2xz),
        bz = centre(s.b3, s.b3y, s.b3x, s.b3xy);
  if (CORR) {
    float lo[3], hi[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      lo[q] = centre(m[q][0], m[q][1], m[q][2], m[q][3]);
      hi[q] = centre(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
    bx = 0.25f * (lo[0] + 2.0f * bx + hi[0]);
    by = 0.25f * (lo[1] + 2.0f * by + hi[1]);
    bz = 0.25f * (lo[2] + 2.0f * bz + hi[2]);
  }
  bx += c0x;
  by += c0y;
  bz += c0z;
  float* const f[6] = {aj, aj + C, aj + 2 * C, ct, ct + C, ct + 2 * C};
  const float v[6] = {a1, a2, a3, ay * bz - az * by, az * bx - ax * bz, ax * by - ay * bx};
#pragma unroll
  for (int q = 0; q < 6; ++q) put(f[q], o, v[q]);
  ghost_images(g, i, j, k, f, v);
}

template <bool CORR>
__global__ void __launch_bounds__(FBX * FBY) k_aj_ct(G32 g, const float* db,
                                                     const float* np, const float* up,
                                                     const float* b0c, float alpha,
                                                     float* aj, float* ct, int ahead) {
  swapk::after_previous();
  FIELD_NODE(i, j, k);
  // rows of later planes, as in k_bstep; the predictor's kernel runs further
  // ahead, having the least to do per node.  With the addresses above, us per
  // launch, predictor and corrector: 256x128x128 cells 55.8 -> 51.7 and 73.9 ->
  // 65.8, 512x256x128 195 -> 175 and 274 -> 220
  if (blockIdx.x == 0 && threadIdx.x == 0 && ahead && k + ahead <= g.ncz + 1) {
    const unsigned t = (unsigned)nid(g, i, j, k + ahead), nb = (g.ncx * 4 + 16) & ~15;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      prefetch_l2(db + t + g.C * m, nb);
      prefetch_l2(up + t + g.C * m, nb);
    }
    prefetch_l2(np + t, nb);
  }
  aj_ct_node<CORR>(g, db, face_terms(g, np, up, alpha, i, j, k), b0c, aj, ct, i, j, k);
}

// Component m of E = face average of ct + nu*aj at node (i,j,k) (gutsf.f:
// 94-96, 1082), less the electron-pressure face gradient gpf when given
// (the isothermal extension of the commented "- gradP", gutsf.f:1083,1283).
template <int m>
__device__ __forceinline__ float e_o(const G32& g, const float* ct, const float* nu,
                                     const float* aj, const float* gpf, long long o) {
  const long long C = g.C;
  const long long s = m == 0 ? 1 : (m == 1 ? (long long)g.nx : (long long)g.nx * g.ny);
  const float e = 0.5f * (ct[o + C * m] + ct[o + s + C * m]) + nu[o] * aj[o + C * m];
  return gpf ? e - gpf[o + C * m] : e;
}


// Double-float arithmetic (a pair of floats carrying 48 significant bits):
// the FP32 form accumulates B across subcycles in it, because GB300's FP64
// pipe runs at a small fraction of its FP32 rate.  Dekker/Knuth error-free
// transformations with explicitly rounded operations (never contracted).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// (bh + bl) - (ch + cl) * x
__device__ __forceinline__ void df_sub_mul(float bh, float bl, float ch, float cl, float x, float& rh, float& rl) {
  const float p = __fmul_rn(ch, x);
  const float q = __fmaf_rn(cl, x, __fmaf_rn(ch, x, -p));  // low part of the product
  float s, e;
  two_sum(bh, -p, s, e);
  e = __fadd_rn(e, __fsub_rn(bl, q));
  rh = __fadd_rn(s, e);
  rl = __fsub_rn(e, __fsub_rn(rh, s));
}

// E on the fly, curlE (gutsf.f:288-299) and B_new = base - coef*curlE
// (predict_B gutsf.f:1158-1159 with coef = 2 dtsub on b12; correct_B
// gutsf.f:1349-1350 with coef = dtsub on b1) in double-float; dB of the
// result in FP32.  Predictor: only dB at m+1/2 = (dB_new + dB1)/2
// (gutsf.f:1210-1219), the one use of the predicted B: the corrector rewrites
// B and dB from b1.  WRITE_E: store E (the step's last corrector).  e_acc: the
// sum of the correctors' E over a step, the surrogate's target.
template <bool PRED, bool WRITE_E>
__device__ __forceinline__ void bstep_node(const G32& g, const float* ct, const float* nu, const float* aj,
                                           const float* gpf, const float* bh, const float* bl, float ch, float cl,
                                           const float* b0c, float* oh, float* ol, float* dbo, const float* db1,
                                           float* dbtp1, float* E, float* e_acc, int i, int j, int k) {
  const Off d = off_of(g, i, j, k);
  const long long C = g.C;
  const unsigned o = at_node(g, i, j, k), ox = o + d.xp, oy = o + d.yp, oz = o + d.zp;
  const In c1{ct}, c2{ct + C}, c3{ct + 2 * C}, j1{aj}, j2{aj + C}, j3{aj + 2 * C}, nus{nu};
  const float n0 = nus[o], nx = nus[ox], ny = nus[oy], nz = nus[oz];
  float e1 = 0.5f * (c1[o] + c1[ox]) + n0 * j1[o], e1y = 0.5f * (c1[oy] + c1[oy + d.xp]) + ny * j1[oy],
        e1z = 0.5f * (c1[oz] + c1[oz + d.xp]) + nz * j1[oz];
  float e2 = 0.5f * (c2[o] + c2[oy]) + n0 * j2[o], e2x = 0.5f * (c2[ox] + c2[ox + d.yp]) + nx * j2[ox],
        e2z = 0.5f * (c2[oz] + c2[oz + d.yp]) + nz * j2[oz];
  float e3 = 0.5f * (c3[o] + c3[oz]) + n0 * j3[o], e3x = 0.5f * (c3[ox] + c3[ox + d.zp]) + nx * j3[ox],
        e3y = 0.5f * (c3[oy] + c3[oy + d.zp]) + ny * j3[oy];
  float h[3], l[3], c0[3], old[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    h[m] = In{bh + C * m}[o];
    l[m] = In{bl + C * m}[o];
    c0[m] = b0c[m];
    old[m] = PRED ? In{db1 + C * m}[o] : 0.0f;
  }
  if (gpf) {
    const In g1{gpf}, g2{gpf + C}, g3{gpf + 2 * C};
    e1 -= g1[o]; e1y -= g1[oy]; e1z -= g1[oz];
    e2 -= g2[o]; e2x -= g2[ox]; e2z -= g2[oz];
    e3 -= g3[o]; e3x -= g3[ox]; e3y -= g3[oy];
  }
  const float ce[3] = {(e3y - e3) * g.inv_dy + (e2 - e2z) * g.inv_dz,
                       (e3 - e3x) * g.inv_dx + (e1z - e1) * g.inv_dz,
                       (e1 - e1y) * g.inv_dy + (e2x - e2) * g.inv_dx};
  constexpr int N = (PRED ? 3 : 9) + (WRITE_E ? 3 : 0);
  float* f[N];
  float v[N];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    float rh, rl;
    df_sub_mul(h[m], l[m], ch, cl, ce[m], rh, rl);
    const float b = __fadd_rn(__fsub_rn(rh, c0[m]), rl);
    if (PRED) {
      f[m] = dbtp1 + C * m;
      v[m] = 0.5f * (b + old[m]);
    } else {
      f[m] = oh + C * m;
      v[m] = rh;
      f[3 + m] = ol + C * m;
      v[3 + m] = rl;
      f[6 + m] = dbo + C * m;
      v[6 + m] = b;
    }
  }
  if (WRITE_E) {
    f[N - 3] = E; f[N - 2] = E + C; f[N - 1] = E + 2 * C;
    v[N - 3] = e1; v[N - 2] = e2; v[N - 1] = e3;
  }
#pragma unroll
  for (int q = 0; q < N; ++q) put(f[q], o, v[q]);
  float* const(&cf)[N] = f;
  ghost_images(g, i, j, k, cf, v);
  if (e_acc) {
    put(e_acc, o, In{e_acc}[o] + e1);
    put(e_acc + C, o, In{e_acc + C}[o] + e2);
    put(e_acc + 2 * C, o, In{e_acc + 2 * C}[o] + e3);
  }
}

template <bool PRED, bool WRITE_E>
__global__ void __launch_bounds__(FBX * FBY) k_bstep(G32 g, const float* ct,
                                                     const float* nu, const float* aj,
                                                     const float* gpf,
                                                     const float* bh, const float* bl,
                                                     float ch, float cl, const float* b0c,
                                                     float* oh, float* ol,
                                                     float* dbo, const float* db1,
                                                     float* dbtp1, float* E,
                                                     float* e_acc, int ahead) {
  swapk::after_previous();
  FIELD_NODE(i, j, k);
  // grids that do not fit L2 (ahead > 0): one thread per row asks for the row
  // that the blocks after the resident ones will read, `ahead` planes up
  // (whole rows, from the 16-byte boundary below; within the arrays, whose
  // last plane holds ghosts).  The resident warps' own loads leave HBM idle
  // while they compute and store: 256x128x128 cells, us per launch, predictor
  // 74.0 -> 63.5, corrector 79.8 -> 75.6
  if (blockIdx.x == 0 && threadIdx.x == 0 && ahead && k + ahead <= g.ncz + 1) {
    const unsigned t = (unsigned)nid(g, i, j, k + ahead), nb = (g.ncx * 4 + 16) & ~15;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      prefetch_l2(ct + t + g.C * m, nb);
      prefetch_l2(aj + t + g.C * m, nb);
      prefetch_l2(bh + t + g.C * m, nb);
      prefetch_l2(bl + t + g.C * m, nb);
      if (PRED) prefetch_l2(db1 + t + g.C * m, nb);
    }
    prefetch_l2(nu + t, nb);
  }
  bstep_node<PRED, WRITE_E>(g, ct, nu, aj, gpf, bh, bl, ch, cl, b0c, oh, ol, dbo, db1, dbtp1, E, e_acc, i, j, k);
}

// ---- the whole field step of a small grid in one launch ----
//
// Below FIELD_LOOP_NODES the subcycles' kernels are bound by their launches
// and the latency of a few loads, not by work.  So the 40 half-kernels of ten
// subcycles run as phases of one kernel whose blocks meet at a barrier
// between them (bounded waits).  The same node functions on the same
// operands.  Two forms.  CLUSTER: one cluster of FIELD_CLUSTER blocks, which
// meet at the hardware's cluster barrier (0.24 us) -- up to FIELD_CLUSTER *
// LOOP_TPB nodes.  Otherwise a cooperative launch with a counter in memory
// (0.9 us at 152 blocks; grid_loop.cuh).
// A step of 4 ions per cell, loop against launches, in ms: 33k nodes 0.179
// against 0.21, 65k 0.215 against 0.25, 78k 0.242 against 0.26; with two nodes
// per thread 98k 0.317 against 0.289, 131k 0.362 against 0.336 (the launches
// overlap: launch_next.cuh): hence FIELD_LOOP_NODES, a node per thread.  Its
// place and what the subcycles share are then found once (20 steps of 64x32x32
// cells 5.40 -> 5.19 ms, of 16x8x12 3.32 -> 3.13).
constexpr int LOOP_TPB = 512;

template <bool CLUSTER>
__global__ void __launch_bounds__(LOOP_TPB, 1) k_field_loop(G32 g, FieldLoop f) {
  // uniform over the grid (both words are a snapshot that nothing writes
  // now): a failed pass or a Courant violation leaves the state as it is
  if (*f.failed != 0 || (double)*f.courant <= f.courant_floor) return;
  loop::Barrier bar{f.bar, f.polls, 0u, true};
  // a node per thread (field_loop_fits), and what its subcycles share, found once
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool mine = t < (unsigned)n_int(g);
  int i = 2, j = 2, k = 2;
  if (mine) interior_of(g, t, i, j, k);
  const FaceTerms ft = face_terms(g, f.np, f.up, f.alpha, i, j, k);
  float *b1h = f.b1h, *b1l = f.b1l, *b12h = f.b12h, *b12l = f.b12l, *bph = f.bph, *bpl = f.bpl, *db1 = f.db1,
        *dbp = f.dbp;
  auto each = [&](auto&& node) {
    if (mine) node(i, j, k);
    return bar.template sync<CLUSTER>();
  };
  for (int s = 0; s < f.n; ++s) {
    if (!each([&](int i, int j, int k) {
          aj_ct_node<false>(g, db1, ft, f.b0c, f.aj, f.ct, i, j, k);
        }))
      break;
    if (!each([&](int i, int j, int k) {
          bstep_node<true, false>(g, f.ct, f.nu, f.aj, f.gpf, b12h, b12l, f.ch2, f.cl2, f.b0c, bph, bpl, dbp, db1,
                                  f.dbt, f.E, nullptr, i, j, k);
        }))
      break;
    if (!each([&](int i, int j, int k) {
          aj_ct_node<true>(g, f.dbt, ft, f.b0c, f.aj, f.ct, i, j, k);
        }))
      break;
    const bool last = s + 1 == f.n;
    if (!each([&](int i, int j, int k) {
          if (last)
            bstep_node<false, true>(g, f.ct, f.nu, f.aj, f.gpf, b1h, b1l, f.ch, f.cl, f.b0c, bph, bpl, dbp, nullptr,
                                    nullptr, f.E, f.e_acc, i, j, k);
          else
            bstep_node<false, false>(g, f.ct, f.nu, f.aj, f.gpf, b1h, b1l, f.ch, f.cl, f.b0c, bph, bpl, dbp, nullptr,
                                     nullptr, f.E, f.e_acc, i, j, k);
        }))
      break;
    // f_update_tlev (gutsf.f:10-35): b12 <- b1, b1 <- b1p2
    float* q = b12h; b12h = b1h; b1h = bph; bph = q;
    q = b12l; b12l = b1l; b1l = bpl; bpl = q;
    q = db1; db1 = dbp; dbp = q;
  }
  if (CLUSTER) return;
  if (!bar.ok && threadIdx.x == 0) set_err(f.err, KERR_WAIT);
  bar.done();
}

// B_new = base - coef * curl E for a given E (with ghost images), in
// double-float, with its FP32 dB: the field advance of the surrogate, whose
// discrete curl keeps div B where it was.  th (may be null): also the B one
// subcycle before the end of the step, B_new + f * (base - B_new) on hi parts,
// lo of B_new kept (the predictor's leapfrog base of the next plain subcycle).
__global__ void __launch_bounds__(FBX * FBY) k_bstep_given_e(G32 g, const float* E, const float* bh, const float* bl,
                                                             float ch, float cl, const float* b0c, float* oh,
                                                             float* ol, float* dbo, float f, float* th, float* tl) {
  swapk::after_previous();
  FIELD_NODE(i, j, k);
  const Off d = off_of(g, i, j, k);
  const long long C = g.C;
  const unsigned o = at_node(g, i, j, k);
  const In E1{E}, E2{E + C}, E3{E + 2 * C};
  const float e1 = E1[o], e2 = E2[o], e3 = E3[o], e1y = E1[o + d.yp], e1z = E1[o + d.zp], e2x = E2[o + d.xp],
              e2z = E2[o + d.zp], e3x = E3[o + d.xp], e3y = E3[o + d.yp];
  float h[3], l[3], c0[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    h[m] = In{bh + C * m}[o];
    l[m] = In{bl + C * m}[o];
    c0[m] = b0c[m];
  }
  const float ce[3] = {(e3y - e3) * g.inv_dy + (e2 - e2z) * g.inv_dz, (e3 - e3x) * g.inv_dx + (e1z - e1) * g.inv_dz,
                       (e1 - e1y) * g.inv_dy + (e2x - e2) * g.inv_dx};
  float* out[9];
  float v[9];
  float* lerp[6];
  float w[6];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    float rh, rl;
    df_sub_mul(h[m], l[m], ch, cl, ce[m], rh, rl);
    out[m] = oh + C * m;
    v[m] = rh;
    out[3 + m] = ol + C * m;
    v[3 + m] = rl;
    out[6 + m] = dbo + C * m;
    v[6 + m] = __fadd_rn(__fsub_rn(rh, c0[m]), rl);
    float s, e;
    two_sum(rh, f * (h[m] - rh), s, e);
    e = __fadd_rn(e, rl);
    lerp[m] = th + C * m;
    w[m] = __fadd_rn(s, e);
    lerp[3 + m] = tl + C * m;
    w[3 + m] = __fsub_rn(e, __fsub_rn(w[m], s));
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) put(out[q], o, v[q]);
  ghost_images(g, i, j, k, out, v);
  if (!th) return;
#pragma unroll
  for (int q = 0; q < 6; ++q) put(lerp[q], o, w[q]);
  ghost_images(g, i, j, k, lerp, w);
}

// Block sum (thread 0 holds the result; every thread of the block calls it).
__device__ __forceinline__ double bsum(double v) {
  __shared__ double sh[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    r = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  return r;
}

// The judge's sums over the interior: |B_a - B_b|^2, |B_b|^2, |B_b - b0|^2
// (double-float levels a and b).
__global__ void k_judge(G32 g, const float* __restrict__ ah, const float* __restrict__ al,
                        const float* __restrict__ bh, const float* __restrict__ bl, const float* __restrict__ b0c,
                        double* acc) {
  double s0 = 0, s1 = 0, s2 = 0;
  GSTRIDE(t, n_int(g)) {
    int i, j, k;
    interior_of(g, t, i, j, k);
    const long long o = nid(g, i, j, k);
    for (int m = 0; m < 3; ++m) {
      const double a = (double)ah[o + g.C * m] + (double)al[o + g.C * m];
      const double b = (double)bh[o + g.C * m] + (double)bl[o + g.C * m];
      s0 += (a - b) * (a - b);
      s1 += b * b;
      s2 += (b - (double)b0c[m]) * (b - (double)b0c[m]);
    }
  }
  // one atomic per block and sum (a grid of a few blocks per SM)
  s0 = bsum(s0);
  if (threadIdx.x == 0) atomicAdd(acc, s0);
  s1 = bsum(s1);
  if (threadIdx.x == 0) atomicAdd(acc + 1, s1);
  s2 = bsum(s2);
  if (threadIdx.x == 0) atomicAdd(acc + 2, s2);
}

// The surrogate's inputs at every interior node (voxel v = x + ncx*(y +
// Surrogate inputs per interior node (v = P + ncx*(Q + ncy*R)), FP32
// [V][SUR_NIN]: B = dB + b0, u_p, n_p, p_e = te * n_p, and E0 = ct + nu aj at
// the faces (the plain E of get_E from the predictor's aj and ct; zero when
// ct is null).
// A block's voxels go out through shared memory as whole lines: stores of 14
// floats a thread apart cost 28 us for 262k voxels, these 13.
__global__ void __launch_bounds__(TPB) k_grid_to_voxels(G32 g, const float* db, const float* b0c, const float* up,
                                                        const float* np, float te, const float* ct, const float* aj,
                                                        const float* nu, const float* gpf, const float* b1h,
                                                        const float* b1l, const float* b12h, const float* b12l,
                                                        float* out) {
  __shared__ float s_out[TPB * SUR_NIN];
  swapk::after_previous();
  const long long V = n_int(g);
  for (long long v0 = blockIdx.x * (long long)TPB; v0 < V; v0 += (long long)gridDim.x * TPB) {
    const long long v = v0 + threadIdx.x;
    if (v < V) {
      int i, j, k;
      interior_of(g, v, i, j, k);
      const long long C = g.C, o = nid(g, i, j, k);
      float* r = s_out + threadIdx.x * SUR_NIN;
      r[0] = db[o] + b0c[0];
      r[1] = db[o + C] + b0c[1];
      r[2] = db[o + 2 * C] + b0c[2];
      r[3] = up[o];
      r[4] = up[o + C];
      r[5] = up[o + 2 * C];
      r[6] = np[o];
      r[7] = te * np[o];
      r[8] = ct ? e_o<0>(g, ct, nu, aj, gpf, o) : 0.0f;
      r[9] = ct ? e_o<1>(g, ct, nu, aj, gpf, o) : 0.0f;
      r[10] = ct ? e_o<2>(g, ct, nu, aj, gpf, o) : 0.0f;
#pragma unroll
      for (int m = 0; m < 3; ++m)
        r[11 + m] = b12h ? (b1h[o + C * m] - b12h[o + C * m]) + (b1l[o + C * m] - b12l[o + C * m]) : 0.0f;
    }
    __syncthreads();
    const int n = (int)(V - v0 < TPB ? V - v0 : TPB) * SUR_NIN;
    for (int q = threadIdx.x; q < n; q += TPB) out[v0 * SUR_NIN + q] = s_out[q];
    __syncthreads();
  }
}

// E = E0 + the predicted correction ([V][3]) into the field layout with ghost
// images (E0 from the inputs vin, none when vin is null).
__global__ void k_voxels_to_grid(G32 g, const float* ev, const float* vin,
                                 float* E) {
  swapk::after_previous();
  GSTRIDE(v, n_int(g)) {
    int i, j, k;
    interior_of(g, v, i, j, k);
    for (int m = 0; m < 3; ++m)
      store_img(g, E + g.C * m, i, j, k, ev[v * 3 + m] + (vin ? vin[v * SUR_NIN + 8 + m] : 0.0f));
  }
}

// Grid E (interior) times f into [V][3] per voxel, less E0 from vin (when given).
__global__ void k_grid_e_to_voxels(G32 g, const float* __restrict__ E, float f, const float* __restrict__ vin,
                                   float* __restrict__ ev) {
  GSTRIDE(v, n_int(g)) {
    int i, j, k;
    interior_of(g, v, i, j, k);
    const long long o = nid(g, i, j, k);
    for (int m = 0; m < 3; ++m) ev[v * 3 + m] = f * E[o + g.C * m] - (vin ? vin[v * SUR_NIN + 8 + m] : 0.0f);
  }
}

// FP64 <-> double-float.
__global__ void k_split_df(long long n, const double* __restrict__ a, float* __restrict__ h, float* __restrict__ l) {
  GSTRIDE(t, n) {
    const double v = a[t];
    const float vh = (float)v;
    h[t] = vh;
    l[t] = (float)(v - (double)vh);
  }
}
__global__ void k_join_df(long long n, const float* __restrict__ h, const float* __restrict__ l,
                          double* __restrict__ a) {
  GSTRIDE(t, n) a[t] = (double)h[t] + (double)l[t];
}

// ---------------------------------------------------------------------------
// stable counting sort by cell key for particles that moved at most one cell
// per axis since the last sort
// ---------------------------------------------------------------------------

// One warp per old key K: direction of every particle of K and its rank
// among the particles of K with the same direction, in array order.
__global__ void k_sort_prep(G32 g, const int64_t* __restrict__ start, const int32_t* __restrict__ cell,
                            uint32_t* __restrict__ dirrank, uint16_t* __restrict__ dep, int* err) {
  __shared__ unsigned s_cnt[TPB / 32][NDIR];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long K = blockIdx.x * (long long)(blockDim.x >> 5) + w; K < g.nkeys; K += nwarps) {
    if (lane < NDIR) s_cnt[w][lane] = 0;
    __syncwarp();
    int i0, j0, k0;
    cell_of_key(g, K, i0, j0, k0);
    const long long a = start[K], e = start[K + 1];
    for (long long base = a; base < e; base += 32) {
      const long long l = base + lane;
      const bool live = l < e;
      int d = NDIR;  // sentinel for idle lanes
      if (live && cell[l] < 0) {
        d = NDIR + 2;  // removed (outflow): not counted, skipped by the scatter
      } else if (live) {
        const int32_t c = cell[l];
        const int dx = step_cell(pk_i(c), i0, g.ncx), dy = step_cell(pk_j(c), j0, g.ncy),
                  dz = step_cell(pk_k(c), k0, g.ncz);
        if (dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1) {
          set_err(err, KERR_MOVE);
          d = NDIR + 1;  // not counted; the scatter skips it
        } else {
          d = dir_index(dx, dy, dz);
        }
      }
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      const unsigned lt = peers & ((1u << lane) - 1u);
      const int leader = __ffs(peers) - 1;
      const bool counted = live && d < NDIR;
      unsigned basecnt = 0;
      if (counted) basecnt = s_cnt[w][d];
      __syncwarp();
      if (live && !counted) dirrank[l] = d == NDIR + 2 ? DR_DEAD : DR_BAD;
      if (counted) {
        dirrank[l] = ((uint32_t)d << 26) | (basecnt + __popc(lt));
        if (lane == leader) s_cnt[w][d] = basecnt + __popc(peers);
      }
      __syncwarp();
    }
    if (lane < NDIR) dep[(long long)lane * g.nkeys + K] = (uint16_t)s_cnt[w][lane];
    __syncwarp();
  }
}

// The old key from which direction d arrives at the cell of key X.
__device__ __forceinline__ long long src_key(const G32& g, int i, int j, int k, int d) {
  const int dx = d % 3 - 1, dy = (d / 3) % 3 - 1, dz = d / 9 - 1;
  return key_of(g, wrapi(i - dx, g.ncx), wrapi(j - dy, g.ncy), wrapi(k - dz, g.ncz));
}

// Per new key X: the count of arriving particles and, for every direction d,
// how many of them come from sources earlier in key order than the source of
// d (the stable order), so the scatter needs one lookup per particle.
// The key order of a cell's 27 sources depends only on its place in its brick
// and on which of its neighbours lie beyond a periodic seam: `order` lists,
// per such class (cell_class), the directions by increasing source key.  (A
// separate path for the cells at the seams compared the 27 keys pairwise and
// held the kernel at 128 registers: 4.2M cells 0.38 ms a
// step, 0.31 by class.  Stored rank by rank, a warp's values went to as many
// places as its lanes had classes: 0.21 stored by direction.)
__device__ __forceinline__ int axis_class(int i, int n) { return i == 0 ? 4 : (i == n - 1 ? 5 : i & 3); }
__global__ void __launch_bounds__(TPB) k_sort_count(G32 g, const uint16_t* __restrict__ dep,
                                                    const int32_t* __restrict__ ncount,
                                                    const uint8_t* __restrict__ order, int64_t* __restrict__ count,
                                                    uint16_t* __restrict__ pre, int* err) {
  __shared__ __align__(4) uint8_t s_ord[SORT_CLASSES * NDIR];
  __shared__ uint16_t s_cnt[NDIR][TPB];  // per thread, indexed by direction
  for (int t = threadIdx.x; t < SORT_CLASSES * NDIR / 4; t += blockDim.x)
    reinterpret_cast<uint32_t*>(s_ord)[t] = reinterpret_cast<const uint32_t*>(order)[t];
  __syncthreads();
  GSTRIDE(X, g.nkeys) {
    int i, j, k;
    cell_of_key(g, X, i, j, k);
    unsigned c[NDIR], n = 0;
#pragma unroll
    for (int d = 0; d < NDIR; ++d) c[d] = dep[(long long)d * g.nkeys + src_key(g, i, j, k, d)];
#pragma unroll
    for (int d = 0; d < NDIR; ++d) {
      s_cnt[d][threadIdx.x] = (uint16_t)c[d];
      n += c[d];
    }
    if (n > 65535) set_err(err, KERR_MOVE);
    const uint8_t* ord =
        s_ord + (axis_class(i, g.ncx) + 6 * (axis_class(j, g.ncy) + 6 * axis_class(k, g.ncz))) * NDIR;
    unsigned run = 0;
#pragma unroll 9
    for (int r = 0; r < NDIR; ++r) {
      const int d = ord[r];
      const unsigned here = s_cnt[d][threadIdx.x];
      s_cnt[d][threadIdx.x] = (uint16_t)run;
      run += here;
    }
    // by direction, so that a warp's stores meet (by rank its lanes' directions
    // differ)
#pragma unroll
    for (int d = 0; d < NDIR; ++d) pre[(long long)d * g.nkeys + X] = s_cnt[d][threadIdx.x];
    count[X] = (int64_t)n + (ncount ? ncount[X] : 0);
  }
}

// dest = start_new[X] + (arrivals from sources earlier in key order) + rank.
__global__ void k_sort_scatter(G32 g, long long N, long long cap, const int32_t* __restrict__ cell,
                               const uint32_t* __restrict__ dirrank, const uint16_t* __restrict__ pre,
                               const int64_t* __restrict__ start_new, Part s, Part d, int* err) {
  GSTRIDE(l, N) {
    const int32_t c = cell[l];
    const uint32_t dr = dirrank[l];
    if (dr == DR_DEAD || dr == DR_FAR) continue;
    // every source field is read before the first store: the source and
    // destination buffers are distinct, and loading them together keeps the
    // ion's reads in flight at once instead of one per store
    const float ox = s.ox[l], oy = s.oy[l], oz = s.oz[l];
    const float vx = s.vx[l], vy = s.vy[l], vz = s.vz[l];
    const float wx = s.wx[l], wy = s.wy[l], wz = s.wz[l];
    const uint8_t spc = s.sp ? s.sp[l] : 0;
    const int dd = (int)(dr >> 26);
    if (dd >= NDIR) {
      set_err(err, KERR_MOVE);
      continue;
    }
    const long long X = key_of(g, pk_i(c), pk_j(c), pk_k(c));
    const long long dst = start_new[X] + pre[(long long)dd * g.nkeys + X] + (dr & ((1u << 26) - 1u));
    if (dst < 0 || dst >= cap) {
      set_err(err, KERR_CAPACITY);
      continue;
    }
    d.cell[dst] = c;
    d.ox[dst] = ox; d.oy[dst] = oy; d.oz[dst] = oz;
    d.vx[dst] = vx; d.vy[dst] = vy; d.vz[dst] = vz;
    d.wx[dst] = wx; d.wy[dst] = wy; d.wz[dst] = wz;
    if (s.sp) d.sp[dst] = spc;
  }
}

// Staged new ions: after the arrivals of their key, in staging order.
__global__ void k_new_scatter(G32 g, long long n_host, const int64_t* __restrict__ n_dev, long long n_max, Part s,
                              const int32_t* __restrict__ key, const int32_t* __restrict__ rank,
                              const int32_t* __restrict__ ncount, const int64_t* __restrict__ start_new, Part d,
                              long long cap, int* err) {
  const long long n = n_host + (n_dev ? *n_dev : 0);
  GSTRIDE(q, n < n_max ? n : n_max) {
    const long long X = key[q];
    const int32_t c = s.cell[q];  // all reads before the first store (see k_sort_scatter)
    const float ox = s.ox[q], oy = s.oy[q], oz = s.oz[q];
    const float vx = s.vx[q], vy = s.vy[q], vz = s.vz[q];
    const float wx = s.wx[q], wy = s.wy[q], wz = s.wz[q];
    const uint8_t spc = s.sp[q];
    const long long dst = start_new[X + 1] - ncount[X] + rank[q];
    if (dst < 0 || dst >= cap) {
      set_err(err, KERR_CAPACITY);
      continue;
    }
    d.cell[dst] = c | CELL_FRESH;
    d.ox[dst] = ox; d.oy[dst] = oy; d.oz[dst] = oz;
    d.vx[dst] = vx; d.vy[dst] = vy; d.vz[dst] = vz;
    d.wx[dst] = wx; d.wy[dst] = wy; d.wz[dst] = wz;
    d.sp[dst] = spc;
  }
}

// ---- the sort's moves left to the next step's pass 1 (k_pass1_sort) ----

// perm[dst] = l for the ions the 27-direction sort places (as k_sort_scatter).
// Four ions per thread: the chain from the ion's words to its key's start and
// offset is three trips to memory, and with one ion per thread the card held
// too few of them (134M ions: 0.96 ms, 0.45 this way).
__global__ void __launch_bounds__(TPB) k_sort_perm(G32 g, long long N, long long cap, const int32_t* __restrict__ cell,
                                                   const uint32_t* __restrict__ dirrank,
                                                   const uint16_t* __restrict__ pre,
                                                   const int64_t* __restrict__ start_new, int32_t* __restrict__ perm,
                                                   int* err) {
  const long long l0 = 4 * (blockIdx.x * (long long)TPB + threadIdx.x);
  if (l0 >= N) return;
  const bool whole = l0 + 4 <= N;
  // (the arrays are padded past their last ion)
  const int4 c4 = *reinterpret_cast<const int4*>(cell + l0);
  uint4 d4 = make_uint4(DR_DEAD, DR_DEAD, DR_DEAD, DR_DEAD);
  if (whole) {
    d4 = *reinterpret_cast<const uint4*>(dirrank + l0);
  } else {
    d4.x = dirrank[l0];
    if (l0 + 1 < N) d4.y = dirrank[l0 + 1];
    if (l0 + 2 < N) d4.z = dirrank[l0 + 2];
  }
  const int32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
  const uint32_t dr[4] = {d4.x, d4.y, d4.z, d4.w};
  long long dst[4];
  bool skip[4], bad = false;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    skip[q] = dr[q] == DR_DEAD || dr[q] == DR_FAR;
    const int dd = (int)(dr[q] >> 26);
    if (!skip[q] && dd >= NDIR) {
      bad = true;
      skip[q] = true;
    }
    dst[q] = 0;
    if (!skip[q]) {
      const long long X = key_of(g, pk_i(c[q]), pk_j(c[q]), pk_k(c[q]));
      dst[q] = start_new[X] + pre[(long long)dd * g.nkeys + X] + (dr[q] & ((1u << 26) - 1u));
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (skip[q]) continue;
    if (dst[q] < 0 || dst[q] >= cap) set_err(err, KERR_CAPACITY);
    else perm[dst[q]] = (int32_t)(l0 + q);
  }
  if (bad) set_err(err, KERR_MOVE);
}

// perm[dst] = ~q for staged new ion q (as k_new_scatter).
__global__ void k_new_perm(long long n_host, const int64_t* n_dev, long long n_max, const int32_t* __restrict__ key,
                           const int32_t* __restrict__ rank, const int32_t* __restrict__ ncount,
                           const int64_t* __restrict__ start_new, int32_t* __restrict__ perm, long long cap, int* err) {
  const long long n = n_host + (n_dev ? *n_dev : 0);
  GSTRIDE(q, n < n_max ? n : n_max) {
    const long long X = key[q];
    const long long dst = start_new[X + 1] - ncount[X] + rank[q];
    if (dst < 0 || dst >= cap) set_err(err, KERR_CAPACITY);
    else perm[dst] = ~(int32_t)q;
  }
}

// The moves alone (a run that ends between the sort and the next pass 1).
__global__ void k_move_sorted(long long N, const int32_t* __restrict__ perm, Part s, Part n, Part d) {
  GSTRIDE(l, N) {
    const int32_t q = perm[l];
    const Part& a = q >= 0 ? s : n;
    const long long i = q >= 0 ? q : ~q;
    const int32_t c = a.cell[i];
    const float ox = a.ox[i], oy = a.oy[i], oz = a.oz[i], vx = a.vx[i], vy = a.vy[i], vz = a.vz[i], wx = a.wx[i],
                wy = a.wy[i], wz = a.wz[i];
    const uint8_t spc = a.sp[i];
    d.cell[l] = q >= 0 ? c : (c | CELL_FRESH);
    d.ox[l] = ox; d.oy[l] = oy; d.oz[l] = oz;
    d.vx[l] = vx; d.vy[l] = vy; d.vz[l] = vz;
    d.wx[l] = wx; d.wy[l] = wy; d.wz[l] = wz;
    d.sp[l] = spc;
  }
}

// three-phase exclusive scan of int64 (block sums, scan of sums, add)
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = TPB * SCAN_ITEMS;

__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t* sh, int64_t& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int64_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    int64_t s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < (int)(blockDim.x >> 5)) sh[lane] = s;
  }
  __syncthreads();
  total = sh[(blockDim.x >> 5) - 1];
  const int64_t before = w > 0 ? sh[w - 1] : 0;
  __syncthreads();
  return before + x - v;
}

__global__ void k_scan_reduce(const int64_t* __restrict__ in, long long n, int64_t* __restrict__ sums) {
  __shared__ int64_t sh[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE;
  int64_t v = 0;
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    const long long idx = base + threadIdx.x * SCAN_ITEMS + q;
    if (idx < n) v += in[idx];
  }
  int64_t tot;
  block_excl_scan(v, sh, tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void k_scan_sums(int64_t* sums, long long nb) {
  __shared__ int64_t sh[32];
  int64_t carry = 0;
  for (long long base = 0; base < nb; base += blockDim.x) {
    const long long idx = base + threadIdx.x;
    const int64_t v = idx < nb ? sums[idx] : 0;
    int64_t tot;
    const int64_t ex = block_excl_scan(v, sh, tot);
    if (idx < nb) sums[idx] = carry + ex;
    carry += tot;
  }
}

__global__ void k_scan_apply(const int64_t* __restrict__ in, long long n, const int64_t* __restrict__ sums,
                             int64_t* __restrict__ out) {
  __shared__ int64_t sh[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE;
  int64_t v[SCAN_ITEMS], s = 0;
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    const long long idx = base + threadIdx.x * SCAN_ITEMS + q;
    v[q] = idx < n ? in[idx] : 0;
    s += v[q];
  }
  int64_t tot;
  int64_t run = block_excl_scan(s, sh, tot) + sums[blockIdx.x];
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    const long long idx = base + threadIdx.x * SCAN_ITEMS + q;
    if (idx < n) out[idx] = run;
    run += v[q];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = run;
}

// ---------------------------------------------------------------------------
// conversions and diagnostics
// ---------------------------------------------------------------------------

// The conversion to the FP32 form is bound by the FP64 pipe (a divide holds it
// 135 clocks, any other operation or conversion 16), so what can goes through
// integers.  The bits are those of split_axis and of casts.  f32_begin of 134M
// ions: 20.2 -> 12.9 ms; f32_end 6.2 -> 3.6.

// (float)x rounded to nearest even; what is no normal float by the conversion
// (a call, or it would be made every time and selected).
__device__ __noinline__ float narrow_any(double x) { return (float)x; }
__device__ __forceinline__ float narrow(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x), m = h & 0x7fffffffu;
  if (m - 0x38100000u >= 0x0fd00000u) return narrow_any(x);  // exponents -126 to 126
  const unsigned b = (m - 0x38000000u) << 3 | l >> 29;
  const unsigned rest = (l << 3) | (b & 1u);  // above one half, or one half and odd: up
  return __uint_as_float((h & 0x80000000u) | (b + (rest > 0x80000000u ? 1u : 0u)));
}

// split_axis with the reciprocal r of d (1/d rounded; UNIT: d is one): the
// quotient from one product and its exact remainder (Markstein 1990), the
// nearest whole number by adding 1.5 * 2^52.  What that does not cover
// (differences or quotients of 2^15 and more -- a quotient beyond 2^31 would wrap
// in the low word --, tiny or zero differences, NaN) goes to split_axis.
struct Spacing {
  double d[3], r[3];
};
template <bool UPPER, bool UNIT>
__device__ __forceinline__ bool split_fast(double x, double q1, double d, double r, int n, int& c, float& o) {
  const double a = x - q1;
  const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu;
  if (ha - 0x20000000u >= 0x20e00000u) return split_axis(x, q1, d, n, UPPER, c, o);  // |a| outside [2^-511, 2^15)
  double u = a;
  if (!UNIT) {
    u = a * r;
    u = __fma_rn(__fma_rn(-u, d, a), r, u);
    if (((unsigned)__double2hiint(u) & 0x7fffffffu) >= 0x40e00000u) return split_axis(x, q1, d, n, UPPER, c, o);
  }
  constexpr double M = 6755399441055744.0;
  const double t = u + M;
  int i = __double2loint(t);
  double f = u - (t - M);  // in [-1/2, 1/2], exact
  const int h = __double2hiint(f);
  // (f is no negative zero: u is not zero)
  if (UPPER ? h < 0 || (h | __double2loint(f)) == 0 : h < 0) {
    f += 1.0;
    --i;
  }
  if (i < 0 || i >= n) return false;
  c = i;
  o = narrow(f);
  if (UPPER && o <= 0.0f) o = 1e-7f;
  if (!UPPER && o >= 1.0f) o = 0.99999994f;
  return true;
}
// (double)x; zeros, denormals, infinities and NaN by the conversion itself.
__device__ __noinline__ double widen_any(float x) { return (double)x; }
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x);
  if (((b + 0x00800000u) & 0x7fffffffu) < 0x01000000u) return widen_any(x);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
// q1 + (c + o) * d, c a cell index
__device__ __forceinline__ double position(double q1, int c, float o, double d) {
  return q1 + ((__hiloint2double(0x43300000, c) - 4503599627370496.0) + widen(o)) * d;
}

template <bool UNIT>
__global__ void k_from_f64(G32 g, Spacing sp3, long long N, long long NM, const double* __restrict__ xp,
                           const double* __restrict__ vp, const double* __restrict__ vp1,
                           const double* __restrict__ mrat, const double* __restrict__ beta_p, Species sp, Part p,
                           int* err) {
  GSTRIDE(l, N) {
    int ci = 0, cj = 0, ck = 0;
    float ox = 0.5f, oy = 0.5f, oz = 0.5f;
    const bool ok = split_fast<true, UNIT>(xp[l], g.qx1, sp3.d[0], sp3.r[0], g.ncx, ci, ox) &&
                    split_fast<false, UNIT>(xp[l + NM], g.qy1, sp3.d[1], sp3.r[1], g.ncy, cj, oy) &&
                    split_fast<true, UNIT>(xp[l + 2 * NM], g.qz1, sp3.d[2], sp3.r[2], g.ncz, ck, oz);
    if (!ok) set_err(err, KERR_DOMAIN);
    p.cell[l] = pk(ci, cj, ck);
    p.ox[l] = ox; p.oy[l] = oy; p.oz[l] = oz;
    p.vx[l] = narrow(vp[l]); p.vy[l] = narrow(vp[l + NM]); p.vz[l] = narrow(vp[l + 2 * NM]);
    p.wx[l] = narrow(vp1[l]); p.wy[l] = narrow(vp1[l + NM]); p.wz[l] = narrow(vp1[l + 2 * NM]);
  }
}

__global__ void k_assign_species(long long N, const double* __restrict__ mrat, const double* __restrict__ beta_p,
                                 const double* __restrict__ tab_mrat, const double* __restrict__ tab_bp, int n,
                                 uint8_t* __restrict__ spid, int* miss) {
  GSTRIDE(l, N) {
    int s = -1;
    for (int q = 0; q < n; ++q)
      if (tab_mrat[q] == mrat[l] && tab_bp[q] == beta_p[l]) { s = q; break; }
    if (s < 0) {
      atomicMin(miss, (int)(l & 0x7fffffff));  // the first particle of a pair not in the table
      s = 0;
    }
    spid[l] = (uint8_t)s;
  }
}

__global__ void k_to_f64(G32 g, double3 d3, long long N, long long NM, Part p, double* __restrict__ xp, double* __restrict__ vp,
                         double* __restrict__ vp1) {
  GSTRIDE(l, N) {
    const int32_t c = p.cell[l];
    xp[l] = position(g.qx1, pk_i(c), p.ox[l], d3.x);
    xp[l + NM] = position(g.qy1, pk_j(c), p.oy[l], d3.y);
    xp[l + 2 * NM] = position(g.qz1, pk_k(c), p.oz[l], d3.z);
    vp[l] = widen(p.vx[l]); vp[l + NM] = widen(p.vy[l]); vp[l + 2 * NM] = widen(p.vz[l]);
    vp1[l] = widen(p.wx[l]); vp1[l + NM] = widen(p.wy[l]); vp1[l + 2 * NM] = widen(p.wz[l]);
  }
}

__global__ void k_species_to_f64(long long N, const uint8_t* __restrict__ spid, const double* __restrict__ tm,
                                 const double* __restrict__ tb, double* __restrict__ mrat, double* __restrict__ beta_p) {
  GSTRIDE(l, N) {
    const int q = min((int)spid[l], MAX_SPECIES - 1);
    mrat[l] = tm[q];
    beta_p[l] = tb[q];
  }
}

// The write-back without the ions staged for a step not taken: tiles of
// KEEP_TILE ions, each block's count of kept ions, then (after a scan of the
// counts) the order-preserving conversion of the kept ones.
constexpr int KEEP_TILE = TPB * 8;
__device__ __forceinline__ bool kept(int32_t c) { return c >= 0 && !(c & CELL_FRESH); }

__global__ void k_keep_count(long long N, const int32_t* __restrict__ cell, int64_t* __restrict__ bcount) {
  __shared__ int64_t sh[32];
  const long long base = (long long)blockIdx.x * KEEP_TILE;
  int64_t n = 0;
  for (int q = 0; q < KEEP_TILE / TPB; ++q) {
    const long long l = base + q * TPB + threadIdx.x;
    n += (l < N && kept(cell[l])) ? 1 : 0;
  }
  int64_t tot;
  block_excl_scan(n, sh, tot);
  if (threadIdx.x == 0) bcount[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(TPB) k_to_f64_kept(G32 g, double3 d3, long long N, long long NM, Part p, const int64_t* __restrict__ bstart,
                              const double* __restrict__ tm, const double* __restrict__ tb, double* __restrict__ xp,
                              double* __restrict__ vp, double* __restrict__ vp1, double* __restrict__ mrat,
                              double* __restrict__ beta_p) {
  // the kept ions' places in the tile, all at once: a scan per 256 ions left
  // their loads one behind the other (16.8M ions: 699 us, this way 391)
  constexpr int ROUNDS = KEEP_TILE / TPB, WARPS = TPB / 32;
  __shared__ int at[ROUNDS * WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = (long long)blockIdx.x * KEEP_TILE;
  int32_t c[ROUNDS];
  int d[ROUNDS];
#pragma unroll
  for (int q = 0; q < ROUNDS; ++q) {
    const long long l = base + q * TPB + threadIdx.x;
    c[q] = l < N ? p.cell[l] : CELL_DEAD;
  }
#pragma unroll
  for (int q = 0; q < ROUNDS; ++q) {
    const unsigned m = __ballot_sync(0xffffffffu, kept(c[q]));
    d[q] = __popc(m & ((1u << lane) - 1u));
    if (lane == 0) at[q * WARPS + warp] = __popc(m);
  }
  __syncthreads();
  static_assert(ROUNDS * WARPS == 64, "two counts a lane");
  if (warp == 0) {
    const int n0 = at[2 * lane], n1 = at[2 * lane + 1];
    int sum = n0 + n1;
    for (int o = 1; o < 32; o <<= 1) {
      const int below = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += below;
    }
    at[2 * lane] = sum - n1 - n0;
    at[2 * lane + 1] = sum - n1;
  }
  __syncthreads();
  const long long first = bstart[blockIdx.x];
#pragma unroll
  for (int q = 0; q < ROUNDS; ++q) {
    if (!kept(c[q])) continue;
    const long long l = base + q * TPB + threadIdx.x, t = first + at[q * WARPS + warp] + d[q];
    const float ox = p.ox[l], oy = p.oy[l], oz = p.oz[l], vx = p.vx[l], vy = p.vy[l], vz = p.vz[l], wx = p.wx[l],
                wy = p.wy[l], wz = p.wz[l];
    const int s = p.sp ? min((int)p.sp[l], MAX_SPECIES - 1) : 0;
    xp[t] = position(g.qx1, pk_i(c[q]), ox, d3.x);
    xp[t + NM] = position(g.qy1, pk_j(c[q]), oy, d3.y);
    xp[t + 2 * NM] = position(g.qz1, pk_k(c[q]), oz, d3.z);
    vp[t] = widen(vx); vp[t + NM] = widen(vy); vp[t + 2 * NM] = widen(vz);
    vp1[t] = widen(wx); vp1[t + NM] = widen(wy); vp1[t + 2 * NM] = widen(wz);
    mrat[t] = tm[s];
    beta_p[t] = tb[s];
  }
}

__global__ void k_keys(G32 g, long long N, const int32_t* __restrict__ cell, int32_t* __restrict__ key) {
  GSTRIDE(l, N) {
    const int32_t c = cell[l];
    key[l] = (int32_t)key_of(g, pk_i(c), pk_j(c), pk_k(c));
  }
}

// Keys non-decreasing?  Counts per key (for the cell starts).
__global__ void k_sorted_hist(long long N, const int32_t* __restrict__ key, long long nkeys, int* unsorted,
                              int64_t* __restrict__ count) {
  GSTRIDE(l, N) {
    const int32_t k = key[l];
    if (l + 1 < N && key[l + 1] < k) atomicExch(unsorted, 1);
    const bool ok = k >= 0 && k < nkeys;
    if (!ok) atomicExch(unsorted, 2);
    // one atomic per group of the warp's lanes with the same key (sorted
    // keys: one or two groups), not one per particle on the same address
    const unsigned peers = __match_any_sync(__activemask(), ok ? k : -1);
    if (ok && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
      atomicAdd(reinterpret_cast<unsigned long long*>(count + k), (unsigned long long)__popc(peers));
  }
}

__global__ void k_gather_perm(long long N, const int64_t* __restrict__ perm, Part s, Part d) {
  GSTRIDE(l, N) {
    const long long q = perm[l];
    const int32_t c = s.cell[q];  // all reads before the first store (see k_sort_scatter)
    const float ox = s.ox[q], oy = s.oy[q], oz = s.oz[q];
    const float vx = s.vx[q], vy = s.vy[q], vz = s.vz[q];
    const float wx = s.wx[q], wy = s.wy[q], wz = s.wz[q];
    const uint8_t spc = s.sp ? s.sp[q] : 0;
    d.cell[l] = c;
    d.ox[l] = ox; d.oy[l] = oy; d.oz[l] = oz;
    d.vx[l] = vx; d.vy[l] = vy; d.vz[l] = vz;
    d.wx[l] = wx; d.wy[l] = wy; d.wz[l] = wz;
    if (s.sp) d.sp[l] = spc;
  }
}

__global__ void k_f64_to_f32(long long n, const double* __restrict__ a, const double* __restrict__ b,
                             float* __restrict__ out) {
  GSTRIDE(t, n) out[t] = (float)(b ? a[t] - b[t] : a[t]);
}

__global__ void k_f32_to_f64(long long n, const float* __restrict__ a, double* __restrict__ out) {
  GSTRIDE(t, n) out[t] = (double)a[t];
}

// kf[q] = 0.5 m_q w_q for species q (m = 1/mrat, w = qw*vol the particle's
// weight 1/(beta*beta_p)): kinetic energy kf * v^2, summed in FP32 per thread
// (a thread sees a few hundred particles) and in FP64 across threads.
struct KinFactor {
  float k[MAX_SPECIES];
};
__global__ void k_energy_p(long long N, Part p, KinFactor kf, double* acc) {
  float sf = 0.0f;
  GSTRIDE(l, N) {
    // every load issued before the test, so that an ion's loads are in
    // flight together (the kernel streams 17 B per ion)
    const int32_t c = p.cell[l];
    const int q = p.sp ? min((int)p.sp[l], MAX_SPECIES - 1) : 0;
    const float vx = p.vx[l], vy = p.vy[l], vz = p.vz[l];
    const float e = kf.k[q] * fmaf(vx, vx, fmaf(vy, vy, vz * vz));
    if (c >= 0 && !(c & CELL_FRESH)) sf += e;  // not removed, not created for the coming step
  }
  const double s = bsum((double)sf);
  if (threadIdx.x == 0) atomicAdd(acc, s);
}

__global__ void k_energy_f(G32 g, const double* __restrict__ b0, const float* __restrict__ b1h,
                           const float* __restrict__ b1l, const float* __restrict__ E, double alpha, double vol,
                           double* acc) {
  // sums of squares per thread, scaled once per block: the FP64 pipe of
  // this part is narrow, and a division per node would dominate the kernel
  double s1 = 0, s2 = 0, s3 = 0;
  GSTRIDE(t, n_int(g)) {
    int i, j, k;
    interior_of(g, t, i, j, k);
    const long long o = nid(g, i, j, k);
    for (int m = 0; m < 3; ++m) {
      const double bb = (double)b1h[o + g.C * m] + (double)b1l[o + g.C * m];
      const double d = bb - b0[o + g.C * m];
      const float e = E[o + g.C * m];
      s1 = fma(d, d, s1);
      s2 = fma(bb, bb, s2);
      s3 += (double)(e * e);
    }
  }
  const double kb = 0.5 * vol / alpha;
  s1 = bsum(s1);
  if (threadIdx.x == 0) atomicAdd(acc + 1, s1 * kb);
  s2 = bsum(s2);
  if (threadIdx.x == 0) atomicAdd(acc + 2, s2 * kb);
  s3 = bsum(s3);
  if (threadIdx.x == 0) atomicAdd(acc + 3, s3 * (0.5 * vol));
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
#define RET(...)                 \
  do {                           \
    __VA_ARGS__;                 \
    return cudaGetLastError();   \
  } while (0)

// One pass launch; the first launch of each form asks for the largest
// shared-memory carve-out, so that the occupancy the launch bounds name (7 or
// 8 CTAs per SM) fits the CTAs' shared tiles.
template <int PASS, bool CHEX, bool EXACT, bool PGRAD = false>
cudaError_t launch_pass(unsigned grid, cudaStream_t st, const G32& g, const Part& p, const Species& sp,
                        const StepParams& s, const int64_t* start, const float4* kit, const float4* kitg,
                        void* partial, uint32_t* dirrank, uint16_t* dep, int* err, const FarList& far) {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(k_pass<PASS, CHEX, EXACT, PGRAD>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
  });
  k_pass<PASS, CHEX, EXACT, PGRAD><<<grid, TPB_PASS, 0, st>>>(g, p, sp, s, start, kit, kitg, partial, dirrank, dep,
                                                               err, far);
  return cudaGetLastError();
}

cudaError_t pass(int which, const G32& g, const Part& p, const Species& sp, const StepParams& s, const int64_t* start,
                 const float4* kit, void* partial, uint32_t* dirrank, uint16_t* dep, int* err, bool exact,
                 cudaStream_t st, const FarList* far, const float4* kitg) {
  const unsigned grid = (unsigned)g.nbricks;
  if (which == 3 && !far) return cudaErrorInvalidValue;
  const FarList none{};
  const FarList& fl = far ? *far : none;
#define PASS_ARGS grid, st, g, p, sp, s, start, kit, kitg, partial, dirrank, dep, err, fl
  if (kitg && which != 1) {  // the electron-pressure term: exact moment sums only
    if (!exact) return cudaErrorInvalidValue;
    if (which == 2) return launch_pass<2, false, true, true>(PASS_ARGS);
    if (s.chex) return launch_pass<3, true, true, true>(PASS_ARGS);
    return launch_pass<3, false, true, true>(PASS_ARGS);
  }
  if (exact) {
    if (which == 1) return launch_pass<1, false, true>(PASS_ARGS);
    if (which == 2) return launch_pass<2, false, true>(PASS_ARGS);
    if (s.chex) return launch_pass<3, true, true>(PASS_ARGS);
    return launch_pass<3, false, true>(PASS_ARGS);
  }
  if (which == 1) return launch_pass<1, false, false>(PASS_ARGS);
  if (which == 2) return launch_pass<2, false, false>(PASS_ARGS);
  if (s.chex) return launch_pass<3, true, false>(PASS_ARGS);
  return launch_pass<3, false, false>(PASS_ARGS);
#undef PASS_ARGS
}
cudaError_t node_sum(const G32& g, int pass, const void* partial, bool exact, float* np, float* S, cudaStream_t st) {
  const unsigned nb = nblk(n_int(g));
  // pass 2 deposits no density
  if (pass == 3 && exact) return swapk::launch_next(k_node_sum<TN, 4, true>, nb, TPB, st, g, partial, np, S);
  if (pass == 3) return swapk::launch_next(k_node_sum<TN, 4, false>, nb, TPB, st, g, partial, np, S);
  if (pass == 2 && exact) return swapk::launch_next(k_node_sum<TN_IN, 3, true>, nb, TPB, st, g, partial, np, S);
  if (pass == 2) return swapk::launch_next(k_node_sum<TN_IN, 3, false>, nb, TPB, st, g, partial, np, S);
  if (exact) return swapk::launch_next(k_node_sum<TN_IN, 4, true>, nb, TPB, st, g, partial, np, S);
  return swapk::launch_next(k_node_sum<TN_IN, 4, false>, nb, TPB, st, g, partial, np, S);
}
cudaError_t up_courant(const G32& g, const float* np, const float* S, const float* db, const float* b0c, float alpha,
                       float dx, float* up, float* dtn, float* look, const int* err, cudaStream_t st) {
  const unsigned nb = nblk(n_int(g)) < 152u * 8u ? nblk(n_int(g)) : 152u * 8u;
  return swapk::launch_next(k_up_courant, nb, TPB, st, g, np, S, db, b0c, alpha, dx, up, dtn,
                            reinterpret_cast<unsigned*>(look), err);
}
cudaError_t build_kit(const G32& g, const float* S, const float* db, const float* b0c, const float* np, float alpha,
                      float gp, float4* kit, float4* kitg, int* far_n, float* look, cudaStream_t st) {
  return swapk::launch_next(k_kit, nblk(n_int(g)), TPB, st, g, S, db, b0c, np, alpha, gp, kit, kitg, far_n,
                            reinterpret_cast<unsigned*>(look));
}
__global__ void k_gpe(G32 g, const float* __restrict__ np, float gp, float* __restrict__ gpf) {
  GSTRIDE(t, n_int(g)) {
    int i, j, k;
    interior_of(g, t, i, j, k);
    const long long C = g.C, o = nid(g, i, j, k);
    store_img(g, gpf, i, j, k, gpe_face<0>(g, np, gp, o));
    store_img(g, gpf + C, i, j, k, gpe_face<1>(g, np, gp, o));
    store_img(g, gpf + 2 * C, i, j, k, gpe_face<2>(g, np, gp, o));
  }
}
cudaError_t gpe_faces(const G32& g, const float* np, float gp, float* gpf, cudaStream_t st) {
  RET((k_gpe<<<nblk(n_int(g)), TPB, 0, st>>>(g, np, gp, gpf)));
}
// How far ahead of its blocks a field kernel asks for rows, in planes.
static int planes_ahead(const G32& g, int nodes) {
  const int plane = g.ncx * g.ncy;
  return n_int(g) >= B_AHEAD_NODES ? std::max(1, (nodes + plane / 2) / plane) : 0;
}
cudaError_t aj_ct(const G32& g, bool corr, const float* db, const float* np, const float* up, const float* b0c,
                  float alpha, float* aj, float* ct, cudaStream_t st) {
  const dim3 grid((g.ncx + FBX - 1) / FBX, (g.ncy + FBY - 1) / FBY, g.ncz), blk(FBX, FBY);
  return swapk::launch_next(corr ? k_aj_ct<true> : k_aj_ct<false>, grid, blk, st, g, db, np, up, b0c, alpha, aj, ct,
                            planes_ahead(g, corr ? 200000 : 400000));
}
cudaError_t b_step(const G32& g, bool pred, bool write_e, const float* ct, const float* nu, const float* aj,
                   const float* gpf, const float* bh, const float* bl, double coef, const float* b0c, float* oh,
                   float* ol, float* dbo, const float* db1, float* dbtp1, float* E, float* e_acc, cudaStream_t st) {
  const dim3 grid((g.ncx + FBX - 1) / FBX, (g.ncy + FBY - 1) / FBY, g.ncz), blk(FBX, FBY);
  const float ch = (float)coef, cl = (float)(coef - (double)ch);
  const auto k = pred ? (write_e ? k_bstep<true, true> : k_bstep<true, false>)
                      : (write_e ? k_bstep<false, true> : k_bstep<false, false>);
  return swapk::launch_next(k, grid, blk, st, g, ct, nu, aj, gpf, bh, bl, ch, cl, b0c, oh, ol, dbo, db1, dbtp1, E,
                            e_acc, planes_ahead(g, 200000));
}
static int sm_count() {
  int dev = 0, sms = 0;
  const bool ok = cudaGetDevice(&dev) == cudaSuccess &&
                  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
  return ok ? sms : 0;
}
bool field_loop_fits(const G32& g) {
  return n_int(g) <= FIELD_LOOP_NODES && n_int(g) <= (long long)sm_count() * LOOP_TPB;
}

cudaError_t field_loop(const G32& g, const FieldLoop& f, cudaStream_t st) {
  const long long need = (n_int(g) + LOOP_TPB - 1) / LOOP_TPB;
  if (need <= FIELD_CLUSTER) {  // always the whole cluster: fewer warps share an SM's load path
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(FIELD_CLUSTER);
    cfg.blockDim = dim3((unsigned)(((n_int(g) + FIELD_CLUSTER - 1) / FIELD_CLUSTER + 31) / 32 * 32));
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = FIELD_CLUSTER;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_field_loop<true>, g, f);
  }
  G32 gg = g;
  FieldLoop ff = f;
  void* args[] = {&gg, &ff};
  // the nodes evenly over the SMs, a block on each (whole groups of four
  // warps: fewer blocks meet at the barrier)
  const long long n = n_int(g), sms = sm_count(), t = ((n + sms - 1) / sms + 127) / 128 * 128;
  return loop::launch(reinterpret_cast<const void*>(&k_field_loop<false>), (n + t - 1) / t, (int)t, args, st);
}
cudaError_t b_step_given_e(const G32& g, const float* E, const float* bh, const float* bl, double coef,
                           const float* b0c, float* oh, float* ol, float* dbo, float f, float* th, float* tl,
                           cudaStream_t st) {
  const dim3 grid((g.ncx + FBX - 1) / FBX, (g.ncy + FBY - 1) / FBY, g.ncz), blk(FBX, FBY);
  const float ch = (float)coef, cl = (float)(coef - (double)ch);
  return swapk::launch_next(k_bstep_given_e, grid, blk, st, g, E, bh, bl, ch, cl, b0c, oh, ol, dbo, f, th, tl);
}
cudaError_t grid_to_voxels(const G32& g, const float* db, const float* b0c, const float* up, const float* np,
                           float te, const float* ct, const float* aj, const float* nu, const float* gpf,
                           const float* b1h, const float* b1l, const float* b12h, const float* b12l, float* out,
                           cudaStream_t st) {
  return swapk::launch_next(k_grid_to_voxels, nblk(n_int(g)), TPB, st, g, db, b0c, up, np, te, ct, aj, nu, gpf, b1h, b1l, b12h,
                                                         b12l, out);
}
cudaError_t judge_sums(const G32& g, const float* ah, const float* al, const float* bh, const float* bl,
                       const float* b0c, double* acc3, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(acc3, 0, 3 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  const unsigned nb = nblk(n_int(g)) < 152u * 8u ? nblk(n_int(g)) : 152u * 8u;
  RET((k_judge<<<nb, TPB, 0, st>>>(g, ah, al, bh, bl, b0c, acc3)));
}
cudaError_t voxels_to_grid(const G32& g, const float* ev, const float* vin, float* E, cudaStream_t st) {
  return swapk::launch_next(k_voxels_to_grid, nblk(n_int(g)), TPB, st, g, ev, vin, E);
}
cudaError_t grid_e_to_voxels(const G32& g, const float* E, float f, const float* vin, float* ev, cudaStream_t st) {
  RET((k_grid_e_to_voxels<<<nblk(n_int(g)), TPB, 0, st>>>(g, E, f, vin, ev)));
}
cudaError_t split_df(long long n, const double* a, float* h, float* l, cudaStream_t st) {
  RET((k_split_df<<<nblk(n), TPB, 0, st>>>(n, a, h, l)));
}
cudaError_t join_df(long long n, const float* h, const float* l, double* a, cudaStream_t st) {
  RET((k_join_df<<<nblk(n), TPB, 0, st>>>(n, h, l, a)));
}
// ---------------------------------------------------------------------------
// ions that moved more than one cell in a step (pass 3's far list)
// ---------------------------------------------------------------------------

// Each listed ion's 8 corner weights times (qw, qw v) into the partial tile
// of its deposit cell's brick, as that tile would hold a run of one ion
// (fixed point: 64-bit integer adds, exact and order-independent).
template <bool EXACT>
__global__ void k_far_deposit(G32 g, FarList f, void* partial, int* err) {
  swapk::after_previous();
  const int n = min(*f.n, FAR_CAP);
  unsigned bad = 0;
  GSTRIDE(i, n) {
    const int32_t c = f.dcell[i];
    if (c < 0) continue;
    const int ci = pk_i(c), cj = pk_j(c), ck = pk_k(c);
    const long long b = (long long)(ci >> 2) + (long long)g.nbx * ((cj >> 2) + (long long)g.nby * (ck >> 2));
    const int t0 = ((ci & 3) + 1) + TN * (((cj & 3) + 1) + TN * ((ck & 3) + 1));
    const float ox = f.o[i], oy = f.o[FAR_CAP + i], oz = f.o[2 * FAR_CAP + i];
    const float wxl = 1.0f - ox, wxu = ox, wyl = 1.0f - oy, wyu = oy, wzl = 1.0f - oz, wzu = oz;
    float q[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) q[m] = f.q[m * FAR_CAP + i];
#pragma unroll
    for (int cc = 0; cc < 8; ++cc) {
      const float w = ((cc & 1) ? wxu : wxl) * (((cc >> 1) & 1) ? wyu : wyl) * ((cc >> 2) ? wzu : wzl);
      const int t = t0 + (cc & 1) + TN * (((cc >> 1) & 1) + TN * (cc >> 2));
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float x = w * q[m];
        const long long at = b * (4 * TNODES) + m * TNODES + t;
        if (EXACT) {
          bad |= fabsf(x) < FIX_MAX ? 0u : 1u;
          atomicAdd(static_cast<unsigned long long*>(partial) + at, (unsigned long long)to_fixed(x));
        } else {
          atomicAdd(static_cast<float*>(partial) + at, x);
        }
      }
    }
  }
  if (bad) set_err(err, KERR_RANGE);
}

__global__ void k_far_count(FarList f, int64_t* __restrict__ count) {
  const int n = min(*f.n, FAR_CAP);
  GSTRIDE(i, n) {
    const long long X = f.key[i];
    if (X >= 0) atomicAdd(reinterpret_cast<unsigned long long*>(count + X), 1ULL);
  }
}

// Each survivor's rank among the listed arrivals of its key by array index
// (a scan of the whole list: the list is short, and this keeps the order
// deterministic), then a copy after the near arrivals.
__global__ void k_far_scatter(G32 g, FarList f, const int32_t* __restrict__ ncount,
                              const int64_t* __restrict__ start_new, Part s, Part d, long long cap,
                              int32_t* __restrict__ perm, int* err) {
  const int n = min(*f.n, FAR_CAP);
  GSTRIDE(i, n) {
    const long long X = f.key[i];
    if (X < 0) continue;
    const long long li = f.idx[i];
    int cnt = 0, r = 0;
    for (int j = 0; j < n; ++j)
      if (f.key[j] == X) {
        ++cnt;
        r += f.idx[j] < li ? 1 : 0;
      }
    const long long dst = start_new[X + 1] - (ncount ? ncount[X] : 0) - cnt + r;
    if (dst < 0 || dst >= cap) {
      set_err(err, KERR_CAPACITY);
      continue;
    }
    if (perm) {  // the move is left to the next pass 1
      perm[dst] = (int32_t)li;
      continue;
    }
    d.cell[dst] = s.cell[li];
    d.ox[dst] = s.ox[li]; d.oy[dst] = s.oy[li]; d.oz[dst] = s.oz[li];
    d.vx[dst] = s.vx[li]; d.vy[dst] = s.vy[li]; d.vz[dst] = s.vz[li];
    d.wx[dst] = s.wx[li]; d.wy[dst] = s.wy[li]; d.wz[dst] = s.wz[li];
    if (s.sp) d.sp[dst] = s.sp[li];
  }
}

cudaError_t far_deposit(const G32& g, const FarList& far, void* partial, bool exact, int* err, cudaStream_t st) {
  if (exact) return swapk::launch_next(k_far_deposit<true>, 64, TPB, st, g, far, partial, err);
  return swapk::launch_next(k_far_deposit<false>, 64, TPB, st, g, far, partial, err);
}
cudaError_t far_count(const FarList& far, int64_t* count, cudaStream_t st) {
  RET((k_far_count<<<64, TPB, 0, st>>>(far, count)));
}
cudaError_t far_scatter(const G32& g, const FarList& far, const int32_t* ncount, const int64_t* start_new,
                        const Part& src, const Part& dst, long long cap, int32_t* perm, int* err, cudaStream_t st) {
  RET((k_far_scatter<<<FAR_CAP / TPB, TPB, 0, st>>>(g, far, ncount, start_new, src, dst, cap, perm, err)));
}

cudaError_t sort_prep(const G32& g, const int64_t* start, const int32_t* cell, uint32_t* dirrank, uint16_t* dep,
                      int* err, cudaStream_t st) {
  const long long warps = g.nkeys;
  long long blocks = (warps + (TPB / 32) - 1) / (TPB / 32);
  if (blocks > 65535LL * 16) blocks = 65535LL * 16;
  RET((k_sort_prep<<<(unsigned)blocks, TPB, 0, st>>>(g, start, cell, dirrank, dep, err)));
}
cudaError_t sort_count(const G32& g, const uint16_t* dep, const int32_t* ncount, const uint8_t* order,
                       int64_t* count, uint16_t* pre, int* err, cudaStream_t st) {
  RET((k_sort_count<<<nblk(g.nkeys), TPB, 0, st>>>(g, dep, ncount, order, count, pre, err)));
}
void sort_order_table(uint8_t* out) {
  for (int cls = 0; cls < SORT_CLASSES; ++cls) {
    const int ax[3] = {cls % 6, cls / 6 % 6, cls / 36};  // axis_class
    long long rank[NDIR];
    int dirs[NDIR];
    for (int d = 0; d < NDIR; ++d) {
      const int step[3] = {d % 3 - 1, (d / 3) % 3 - 1, d / 9 - 1};
      int brick[3], local = 0;
      for (int a = 2; a >= 0; --a) {
        const int place = ax[a] == 4 ? 0 : (ax[a] == 5 ? 3 : ax[a]);
        const int src = place - step[a];  // the source cell, relative to this brick
        brick[a] = src < 0 ? -1 : (src > 3 ? 1 : 0);
        local = 4 * local + (src - 4 * brick[a]);
        // beyond a seam: the axis' last brick, or its first
        if (brick[a] < 0 && ax[a] == 4) brick[a] = 2;
        if (brick[a] > 0 && ax[a] == 5) brick[a] = -2;
      }
      rank[d] = (((brick[2] + 2) * 5 + (brick[1] + 2)) * 5 + (brick[0] + 2)) * (long long)BCELLS + local;
      dirs[d] = d;
    }
    std::sort(dirs, dirs + NDIR, [&](int a, int b) { return rank[a] < rank[b]; });
    for (int r = 0; r < NDIR; ++r) out[cls * NDIR + r] = (uint8_t)dirs[r];
  }
}
cudaError_t new_scatter(const G32& g, long long n_host, const int64_t* n_dev, long long n_max, const Part& stage,
                        const int32_t* key, const int32_t* rank, const int32_t* ncount, const int64_t* start_new,
                        const Part& dst, long long cap, int* err, cudaStream_t st) {
  if (n_max <= 0) return cudaSuccess;
  RET((k_new_scatter<<<nblk(n_max), TPB, 0, st>>>(g, n_host, n_dev, n_max, stage, key, rank, ncount, start_new, dst,
                                                  cap, err)));
}

cudaError_t scan_exclusive(const int64_t* in, int64_t* out, long long n, int64_t* sums, cudaStream_t st) {
  const long long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_reduce<<<(unsigned)(nb < 1 ? 1 : nb), TPB, 0, st>>>(in, n, sums);
  k_scan_sums<<<1, 1024, 0, st>>>(sums, nb < 1 ? 1 : nb);
  RET((k_scan_apply<<<(unsigned)(nb < 1 ? 1 : nb), TPB, 0, st>>>(in, n, sums, out)));
}
cudaError_t sort_scatter(const G32& g, long long N, long long cap, const int32_t* cell, const uint32_t* dirrank,
                         const uint16_t* pre, const int64_t* start_new, const Part& src, const Part& dst, int* err,
                         cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_sort_scatter<<<nblk(N), TPB, 0, st>>>(g, N, cap, cell, dirrank, pre, start_new, src, dst, err)));
}
cudaError_t sort_perm(const G32& g, long long N, long long cap, const int32_t* cell, const uint32_t* dirrank,
                      const uint16_t* pre, const int64_t* start_new, int32_t* perm, int* err, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_sort_perm<<<nblk((N + 3) / 4), TPB, 0, st>>>(g, N, cap, cell, dirrank, pre, start_new, perm, err)));
}
cudaError_t new_perm(long long n_host, const int64_t* n_dev, long long n_max, const int32_t* key, const int32_t* rank,
                     const int32_t* ncount, const int64_t* start_new, int32_t* perm, long long cap, int* err,
                     cudaStream_t st) {
  if (n_max <= 0) return cudaSuccess;
  RET((k_new_perm<<<nblk(n_max), TPB, 0, st>>>(n_host, n_dev, n_max, key, rank, ncount, start_new, perm, cap, err)));
}
cudaError_t move_sorted(long long N, const int32_t* perm, const Part& src, const Part& stage, const Part& dst,
                        cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_move_sorted<<<nblk(N), TPB, 0, st>>>(N, perm, src, stage, dst)));
}
cudaError_t pass1_sort(const G32& g, const Part& src, const Part& stage, const Part& dst, const Species& sp,
                       const int64_t* start, const int32_t* perm, void* partial, bool exact, int* err,
                       cudaStream_t st) {
  if (exact)
    RET((k_pass1_sort<true><<<(unsigned)g.nbricks, TPB_PASS, 0, st>>>(g, src, stage, dst, sp, start, perm, partial, err)));
  RET((k_pass1_sort<false><<<(unsigned)g.nbricks, TPB_PASS, 0, st>>>(g, src, stage, dst, sp, start, perm, partial, err)));
}
cudaError_t from_f64(const G32& g, long long N, long long NM, const double* xp, const double* vp, const double* vp1,
                     const double* mrat, const double* beta_p, const Species& sp, Part p, int* err, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  const Spacing sp3{{g.dx, g.dy, g.dz}, {1.0 / (double)g.dx, 1.0 / (double)g.dy, 1.0 / (double)g.dz}};
  if (g.dx == 1.0f && g.dy == 1.0f && g.dz == 1.0f)
    RET((k_from_f64<true><<<nblk(N), TPB, 0, st>>>(g, sp3, N, NM, xp, vp, vp1, mrat, beta_p, sp, p, err)));
  RET((k_from_f64<false><<<nblk(N), TPB, 0, st>>>(g, sp3, N, NM, xp, vp, vp1, mrat, beta_p, sp, p, err)));
}
cudaError_t assign_species(long long N, const double* mrat, const double* beta_p, const double* tab_mrat,
                           const double* tab_bp, int n, uint8_t* spid, int* miss, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_assign_species<<<nblk(N), TPB, 0, st>>>(N, mrat, beta_p, tab_mrat, tab_bp, n, spid, miss)));
}
__global__ void k_not_uniform(long long C, const double* __restrict__ b, int* flag) {
  GSTRIDE(t, 3 * C) {
    if (b[t] != b[(t / C) * C]) atomicExch(flag, 1);
  }
}
cudaError_t not_uniform(long long C, const double* b, int* flag, cudaStream_t st) {
  RET((k_not_uniform<<<nblk(3 * C), TPB, 0, st>>>(C, b, flag)));
}
cudaError_t to_f64(const G32& g, long long N, long long NM, const Part& p, double* xp, double* vp, double* vp1,
                   cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_to_f64<<<nblk(N), TPB, 0, st>>>(g, make_double3(g.dx, g.dy, g.dz), N, NM, p, xp, vp, vp1)));
}
cudaError_t species_to_f64(long long N, const uint8_t* spid, const double* tab_mrat, const double* tab_bp,
                           double* mrat, double* beta_p, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_species_to_f64<<<nblk(N), TPB, 0, st>>>(N, spid, tab_mrat, tab_bp, mrat, beta_p)));
}
cudaError_t to_f64_kept(const G32& g, long long N, long long NM, const Part& p, const double* tab_mrat,
                        const double* tab_bp, double* xp, double* vp, double* vp1, double* mrat, double* beta_p,
                        int64_t* bcount, int64_t* bstart, int64_t* sums, long long* kept_out, cudaStream_t st) {
  *kept_out = 0;
  if (N <= 0) return cudaSuccess;
  const long long nb = (N + KEEP_TILE - 1) / KEEP_TILE;
  cudaError_t e;
  k_keep_count<<<(unsigned)nb, TPB, 0, st>>>(N, p.cell, bcount);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = scan_exclusive(bcount, bstart, nb, sums, st)) != cudaSuccess) return e;
  k_to_f64_kept<<<(unsigned)nb, TPB, 0, st>>>(g, make_double3(g.dx, g.dy, g.dz), N, NM, p, bstart, tab_mrat, tab_bp, xp, vp, vp1, mrat, beta_p);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  int64_t n = 0;
  if ((e = cudaMemcpyAsync(&n, bstart + nb, sizeof(int64_t), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  *kept_out = n;
  return cudaSuccess;
}
cudaError_t keys_of(const G32& g, long long N, const int32_t* cell, int32_t* key, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_keys<<<nblk(N), TPB, 0, st>>>(g, N, cell, key)));
}
cudaError_t sorted_hist(long long N, const int32_t* key, long long nkeys, int* unsorted, int64_t* count,
                        cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(count, 0, (nkeys + 1) * sizeof(int64_t), st);
  if (e != cudaSuccess) return e;
  if (N <= 0) return cudaSuccess;
  RET((k_sorted_hist<<<nblk(N), TPB, 0, st>>>(N, key, nkeys, unsorted, count)));
}
cudaError_t gather_perm(long long N, const int64_t* perm, const Part& src, Part dst, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  RET((k_gather_perm<<<nblk(N), TPB, 0, st>>>(N, perm, src, dst)));
}
cudaError_t grid_f64_to_f32(long long n, const double* a, const double* b, float* out, cudaStream_t st) {
  RET((k_f64_to_f32<<<nblk(n), TPB, 0, st>>>(n, a, b, out)));
}
cudaError_t grid_f32_to_f64(long long n, const float* a, double* out, cudaStream_t st) {
  RET((k_f32_to_f64<<<nblk(n), TPB, 0, st>>>(n, a, out)));
}
cudaError_t energy32(const G32& g, long long N, const Part& p, const Species& sp, double vol, const double* b0,
                     const float* b1h, const float* b1l, const float* E, double alpha, double* acc4,
                     cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(acc4, 0, 4 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  const unsigned cap = 152 * 16;  // many particles per thread, few atomics, the SMs full
  if (N > 0) {
    KinFactor kf{};
    for (int q = 0; q < MAX_SPECIES && q < sp.n; ++q)
      kf.k[q] = (float)(0.5 * (1.0 / (double)sp.mrat[q]) * (double)sp.qw[q] * vol);
    const unsigned nb = nblk(N) < cap ? nblk(N) : cap;
    k_energy_p<<<nb, TPB, 0, st>>>(N, p, kf, acc4);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  const long long nn = (long long)g.ncx * g.ncy * g.ncz;
  RET((k_energy_f<<<nblk(nn) < cap ? nblk(nn) : cap, TPB, 0, st>>>(g, b0, b1h, b1l, E, alpha, vol, acc4)));
}

}  // namespace swapk32
