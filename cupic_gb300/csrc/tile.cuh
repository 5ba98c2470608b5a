// tile.cuh -- the Poisson solve with the whole tile in registers.
//
// CTA (bx, by) of an nbx x nby grid owns a block of the mesh and keeps it,
// with a halo of K nodes on the sides that have neighbours, in registers for
// the whole solve: a strip of R rows is held by one lane group, 4 columns a
// lane, so a sweep (jacobi_iteration, mesh.cu:297-381) takes its west and
// east neighbours from two shuffles a row, the rows inside a strip from
// registers, and only the rows just below and above a strip from shared
// memory (two 16-byte stores and loads a thread, one block barrier).
//   nbx == 1 (rings)  the lanes of a strip hold a full mesh row and the
//                     shuffles go around it (column 0's west neighbour is
//                     column nnx-2); W = nnx-1 <= 128 columns, and several
//                     strips share a warp where W is small.
//   nbx > 1 (halo)    K (a multiple of 4) halo columns on each side, updated
//                     redundantly like the halo rows, so no lane needs more
//                     than its two neighbours, for every W.
// Every K sweeps the blocks trade the K nodes inside each boundary.  Rings of
// up to kTileCluster CTAs are one cluster: a row's columns go from registers
// into the neighbour's shared memory, whose barrier counts their bytes.  Other
// grids trade by way of L2, as 64-bit words {value, epoch} (one round trip, no
// flag and no fence).  Every value is computed with the same operands in the
// same order on every layout, so all layouts give the same bits.
//
// Convergence checks never wait in the sweep loop: the maxima of a block of
// K sweeps are combined over the grid while the next block runs, and when
// a sweep turns out to have passed the stop test the state at the start of
// its block (kept in shared memory) is restored and swept up to it.
//
// What bounds it: the latency of a sweep on a small tile (170 cycles with one
// row a thread on 8 warps, 280 on 15: barrier, shared-memory rows, shuffles)
// and instruction issue on a large one (16 a row and warp), plus the exchange
// every K sweeps (1000 cycles in a cluster, 3000-5000 by way of L2, where the
// instructions of 16 warps weigh as much as the round trip).  Against the
// shared-memory sweep and register strips of jacobi.cu, 200 sweeps in a step:
// 512x2048 0.334 -> 0.154 ms, 256x1024 0.191 -> 0.092, 301x700 (rows of no
// multiple of 4) 0.325 -> 0.093, 32x128 0.127 -> 0.038; with a check after
// each of 2000 sweeps, 64x256 5.0 -> 0.54 ms.
#pragma once

#include <math.h>

#include "cupic_internal.cuh"
#include "draws.cuh"
#include "kernels.h"

namespace cupic {
namespace tile {

enum { kHalo = 0, kRing = 1, kRingRagged = 2 };  // ragged: W % 4 != 0

constexpr unsigned kFull = 0xffffffffu;
constexpr int kSoloBlock = 32;  // sweeps between stop tests of a solve on one CTA
constexpr long long kSpinLimit = 1ll << 22;

__device__ __forceinline__ void st_word(unsigned long long *p, float v, unsigned ep) {
  const unsigned long long w = ((unsigned long long)ep << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void st_word2(unsigned long long *p, float v0, float v1, unsigned ep) {
  const unsigned long long h = (unsigned long long)ep << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(h | __float_as_uint(v0)),
               "l"(h | __float_as_uint(v1))
               : "memory");
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}
__device__ __forceinline__ void ld_word2(const unsigned long long *p, unsigned long long &a,
                                         unsigned long long &b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Rings of a cluster: a row's columns go straight into the neighbour's shared
// memory, whose barrier counts the bytes.
__device__ __forceinline__ unsigned cluster_addr(unsigned addr, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(unsigned to, const float4 &v, unsigned bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
      "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
      : "memory");
}
__device__ __forceinline__ bool cluster_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0u;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_join() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void sts4(float *p, const float4 &v) { *reinterpret_cast<float4 *>(p) = v; }

// Waits: look() until it is true for every lane.  The lanes leave a wait
// together, by a vote, so that the warp is whole when it comes to the block's
// next barrier.  False if the wait gave up or another CTA did.
template <class Look>
__device__ __forceinline__ bool wait_for(const Ctl *ctl, Look &&look) {
  for (long long it = 0;; ++it) {
    if (__all_sync(kFull, look())) return true;
    if ((it & 255) == 255) {
      const bool quit = it >= kSpinLimit || *(const volatile int *)&ctl->abort;
      if (__any_sync(kFull, quit)) return false;
    }
  }
}

// static shared scratch
struct Scratch {
  unsigned cm[4][32];  // per-sweep maxima of a block of sweeps, 4 blocks in turn
  int dec[2];          // a block's stop decision: index of the stopping sweep, or -1
  float decv[2];       // its residual
  int bail;
  uint64_t arrived[2];  // a cluster's exchanges, odd and even ones
  uint64_t voted[2];    // the maxima of its checked blocks, likewise
  unsigned long long w64[16], res64[2];  // a correction's max |r| per warp, and over the grid
};

// one thread's place in its tile
struct Lane {
  int nvalid;        // rows of the strip
  int row0;          // its first mesh row
  int i0;            // extended column of element 0 (-K .. W+K-1)
  int rm;            // ragged ring, last lane: valid elements (1..3), else 0
  int srcw, srce;    // rings: lanes of the west and east neighbours
  int me;            // element whose east neighbour is the mirror column (-1: none)
  unsigned own;      // elements this CTA owns (bits 0..3)
  unsigned ownrows;  // rows this CTA owns (bits 0..R-1)
  bool full;         // no lane of the warp has a partial strip
};

// A node is formed from quarters, with b a quarter of the source term: a product
// by 1/4 is exact, so a fused multiply-add rounds a quarter of what the sum does
// to a quarter of what the sum rounds to, and a node takes four operations
// instead of five.  (Two differences.  Sums below 2^-124 in size are rounded as
// subnormals, where the sum would be exact and its quarter rounded once: by
// 2^-150 at most for each of the four.  Sums of 2^128 and more are finite where
// their quarter is.)
__device__ __forceinline__ float node(float b, float w, float e, float n, float s) {
  return __fmaf_rn(0.25f, s, __fmaf_rn(0.25f, n, __fmaf_rn(0.25f, e, __fmaf_rn(0.25f, w, b))));
}
__device__ __forceinline__ float quarter(float v) { return __fmul_rn(0.25f, v); }

// The source term of fixed-point charge f, (float)((double)f * cb).  Three FP64
// operations a node were 13 us of a 512x2048 solve; the product in
// double-float arithmetic rounds to the same float (draws.cuh) but for a few
// nodes in a million and charges of `most` on, 2^16 units, which take FP64 (all
// do, most = 0, where cb is so small or large that the products leave the
// normal floats).
// (The FP64 fallbacks here and below are calls: inlined, the compiler computes
// them always and selects.)
static __device__ __noinline__ float source_f64(long long f, double cb) { return __double2float_rn((double)f * cb); }
// pow2: cb is a power of two, so the charge's own rounding is the only one.
__device__ __forceinline__ float source(long long f, double cb, const df &cbf, bool pow2, unsigned long long most) {
  const unsigned long long u = f < 0 ? 0ull - (unsigned long long)f : (unsigned long long)f;
  const df n = df_int(u);
  bool ok = u < most;
  float v = __fmul_rn(n.h, cbf.h);
  if (!pow2) v = df_round(df_mul(n, cbf), ok);
  if (!ok) return source_f64(f, cb);
  return f < 0 ? -v : v;
}

// asynchronous copies of 4 and 8 bytes from global to shared memory
__device__ __forceinline__ void copy4(void *to, const void *from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void copy8(void *to, const void *from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(to)), "l"(from) : "memory");
}

// A warp's FP64 operation holds the SM's FP64 pipe for about 24 cycles, so the
// correction's conversions and its product by 4 go through the integer pipe:
// the same bits (round to nearest even), with the hardware's conversion for
// what is not normal on both sides.
static __device__ __noinline__ float to_float_slow(double v) { return __double2float_rn(v); }
static __device__ __noinline__ double to_double_slow(float v) { return (double)v; }
static __device__ __noinline__ double times4_slow(double v) { return 4.0 * v; }
__device__ __forceinline__ float to_float(double v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned e = (unsigned)(u >> 52) & 0x7ffu;
  if (e - 897u >= 254u) return u << 1 ? to_float_slow(v) : __uint_as_float((unsigned)(u >> 32));
  const unsigned t = (unsigned)(((u & 0x7fffffffffffffffull) + 0x0fffffffull + ((u >> 29) & 1ull)) >> 29);
  return __uint_as_float((t - (896u << 23)) | ((unsigned)(u >> 32) & 0x80000000u));
}
__device__ __forceinline__ double to_double(float v) {
  const unsigned b = __float_as_uint(v), e = (b >> 23) & 0xffu;
  if (e - 1u >= 254u) return (b << 1) == 0u ? __hiloint2double((int)b, 0) : to_double_slow(v);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
}
__device__ __forceinline__ double times4(double v) {
  const int hi = __double2hiint(v);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  if (e - 1u >= 0x7fcu) return times4_slow(v);
  return __hiloint2double(hi + 0x200000, __double2loint(v));
}

// One sweep of a strip: v = ((((b + west) + east) + north) + south) / 4.
// FULL: all R rows of the strip are in the tile (the row above the last is
// then x[R]'s place, taken from n4); otherwise the rows past the strip's end
// compute values nothing reads.  FIRST: the solve's first sweep, which reads
// the caller's mirror column (its value may differ from column 0's; every
// later one equals it; used only when some value does differ).  Returns the max |v - old| over owned nodes (CHECK).
template <int R, int MODE, bool FULL, bool CHECK, bool FIRST>
__device__ __forceinline__ float sweep(float4 (&x)[R], const float4 (&b)[R], const float4 s4,
                                       const float4 n4, const Lane &g, const float *mirror) {
  float4 prev = s4;
  float md = 0.0f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 c = x[r];
    float lf, rt;
    float4 e = make_float4(c.y, c.z, c.w, 0.0f);  // east neighbours
    if (MODE == kHalo) {
      lf = __shfl_up_sync(kFull, c.w, 1);
      rt = __shfl_down_sync(kFull, c.x, 1);
    } else {
      float last = c.w;
      if (MODE == kRingRagged) last = g.rm == 0 ? c.w : (g.rm == 1 ? c.x : (g.rm == 2 ? c.y : c.z));
      lf = __shfl_sync(kFull, last, g.srcw);
      rt = __shfl_sync(kFull, c.x, g.srce);
      if (MODE == kRingRagged) {
        e.x = g.rm == 1 ? rt : e.x;
        e.y = g.rm == 2 ? rt : e.y;
        e.z = g.rm == 3 ? rt : e.z;
      }
    }
    e.w = rt;
    float mir = 0.0f;
    if (FIRST && r < g.nvalid) mir = mirror[r];
    if (FIRST && g.me >= 0) {
      e.x = g.me == 0 ? mir : e.x;
      e.y = g.me == 1 ? mir : e.y;
      e.z = g.me == 2 ? mir : e.z;
      e.w = g.me == 3 ? mir : e.w;
    }
    const float4 nx = r + 1 < R ? x[r + 1 < R ? r + 1 : r] : n4;
    const float4 n = (r + 1 < R && !FULL && r + 1 >= g.nvalid) ? n4 : nx;
    float4 v;
    v.x = node(b[r].x, lf, e.x, n.x, prev.x);
    v.y = node(b[r].y, c.x, e.y, n.y, prev.y);
    v.z = node(b[r].z, c.y, e.z, n.z, prev.z);
    v.w = node(b[r].w, c.z, e.w, n.w, prev.w);
    if (CHECK) {
      constexpr bool kAll = MODE == kRing;  // a lane with rows owns all its columns
      float d = kAll || (g.own & 1u) ? fabsf(__fsub_rn(v.x, c.x)) : 0.0f;
      d = kAll || (g.own & 2u) ? fmaxf(d, fabsf(__fsub_rn(v.y, c.y))) : d;
      d = kAll || (g.own & 4u) ? fmaxf(d, fabsf(__fsub_rn(v.z, c.z))) : d;
      d = kAll || (g.own & 8u) ? fmaxf(d, fabsf(__fsub_rn(v.w, c.w))) : d;
      if (FIRST && g.i0 == 0 && (g.own & 1u)) d = fmaxf(d, fabsf(__fsub_rn(v.x, mir)));
      md = (g.ownrows >> r) & 1u ? fmaxf(md, d) : md;
    }
    x[r] = v;
    prev = c;
  }
  return md;
}

// A strip's rows in shared memory: those below and above it (read), its
// first and last (written; the last at +to_last), this sweep's (A) and the
// next one's (B).
struct Rows {
  const float *sA, *nA, *sB, *nB;
  float *wA, *wB;
  int to_last;
};

// Sweeps m .. end-1 of a block.  (Measured slower: the strip's outer rows
// first, an mbarrier arrival and the rows between while the others catch
// up, 100 cycles more a sweep; the same order with __syncthreads, no gain.)
// CHECK: a sweep's maximum goes through the warp's reduction while the next
// sweep waits for its rows, and to the lane of its number in keep after that;
// md holds the last one's (reduced before the stores and the barrier, it
// added 260 cycles to a sweep).
template <int R, int MODE, bool FULL, bool CHECK>
__device__ __forceinline__ void sweeps(float4 (&x)[R], const float4 (&b)[R], const Lane &g, Rows &w, int &m, int end,
                                       float &md, unsigned &keep) {
#pragma unroll 2
  for (; m < end; ++m) {
    const float4 s4 = lds4(w.sA), n4 = lds4(w.nA);
    unsigned v = 0u;
    if (CHECK) v = __reduce_max_sync(kFull, __float_as_uint(md));
    md = sweep<R, MODE, FULL, CHECK, false>(x, b, s4, n4, g, nullptr);
    sts4(w.wB, x[0]);
    if (R > 1) sts4(w.wB + w.to_last, x[R - 1]);
    if (CHECK && (int)(threadIdx.x & 31) == m - 1) keep = v;
    const float *t = w.sA;
    w.sA = w.sB;
    w.sB = t;
    t = w.nA;
    w.nA = w.nB;
    w.nB = t;
    float *u = w.wA;
    w.wA = w.wB;
    w.wB = u;
    __syncthreads();
  }
}

template <int R, int MODE, bool REFINE>
__device__ __forceinline__ void solve(const SimArgs &a, const JacobiArgs &J, const int c, float *sm,
                                      Scratch *js) {
  Ctl *ctl = a.ctl;
  // one round trip for the three words of the control block
  const bool halt = halted(ctl);
  const int cur = *reinterpret_cast<volatile int *>(&ctl->cur);
  const unsigned ebase = *reinterpret_cast<volatile unsigned *>(&ctl->jepoch);
  if (halt) return;
  const bool near = MODE != kHalo && J.near;
  const int G = J.G, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
  const int nnx = a.nnx, nny = a.nny, W = nnx - 1, M = nny - 2;
  const int nbx = MODE == kHalo ? J.nbx : 1, nby = J.nby;
  const int K = J.depth;
  const int bx = MODE == kHalo ? c % nbx : 0, by = MODE == kHalo ? c / nbx : c;
  const int r0 = 1 + by * M / nby, r1 = 1 + (by + 1) * M / nby;  // (tile_plan bounds nby * M)
  int x0 = 0, x1 = W;
  if (MODE == kHalo) {
    const int W4 = (W + 3) >> 2;
    x0 = 4 * ((bx * W4) / nbx);
    x1 = min(W, 4 * (((bx + 1) * W4) / nbx));
  }
  const int KX = MODE == kHalo ? K : 0;  // halo columns on each side
  // updated rows lo..hi; rows lo-1 and hi+1 are the tile's edge rows
  const int lo = nby > 1 ? max(1, r0 - (K - 1)) : 1, hi = nby > 1 ? min(nny - 2, r1 + K - 2) : nny - 2;
  // lane -> strip
  const int nl = J.nl, segs = J.segs;
  const uint32_t near_bytes = ((by > 0 ? 1 : 0) + (by < nby - 1 ? 1 : 0)) * 16u * K * nl;
  if (near) {
    if (tid == 0) {
      for (int k = 0; k < 2; ++k) {
        mbar_init(&js->arrived[k], 1);
        mbar_init(&js->voted[k], 1);
      }
      fence_mbar_init();
      for (int k = 0; k < 2; ++k) {
        mbar_arrive_expect_tx(&js->arrived[k], near_bytes);
        mbar_arrive_expect_tx(&js->voted[k], 128u * G);
      }
    }
    __syncwarp();
    cluster_arrive();
  }
  const int seg = segs == 1 ? 0 : lane / nl, li = segs == 1 ? lane : lane - seg * nl;
  const bool act = segs == 1 ? lane < nl : seg < segs;
  Lane g;
  g.row0 = lo + (warp * segs + seg) * R;
  g.nvalid = act ? min(max(hi + 1 - g.row0, 0), R) : 0;
  g.i0 = x0 - KX + 4 * li;
  g.rm = MODE == kRingRagged && act && li == nl - 1 ? W - 4 * (nl - 1) : 0;
  g.srcw = !act ? lane : (li == 0 ? lane + nl - 1 : lane - 1);
  g.srce = !act ? lane : (li == nl - 1 ? lane - (nl - 1) : lane + 1);
  g.me = -1;
  g.own = 0u;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = g.i0 + q;
    if (act && (i == W - 1 || i == -1)) g.me = q;
    if (act && i >= x0 && i < x1) g.own |= 1u << q;
  }
  g.ownrows = 0u;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r < g.nvalid && g.row0 + r >= r0 && g.row0 + r < r1) g.ownrows |= 1u << r;
  g.full = __all_sync(kFull, !act || g.nvalid == R);
  // shared memory: first and last rows of every strip in two parities, the
  // edge rows of 4 blocks of sweeps in turn, then (below) the received halo
  // nodes, the table of halo words and two snapshots of the strips
  const int par = nthr * 4;
  float *const first = sm, *const last = R > 1 ? sm + 2 * par : sm;  // one row is both
  float *const edge = sm + 4 * par;  // [4][south, north][128]
  const int mine = tid * 4;
  const int soff = seg > 0 ? mine - 4 * nl : (warp - 1) * 128 + 4 * ((segs - 1) * nl + li);
  const int noff = seg < segs - 1 ? mine + 4 * nl : (warp + 1) * 128 + 4 * li;
  const bool south_edge = g.row0 == lo, north_edge = g.nvalid > 0 && g.row0 + g.nvalid - 1 == hi;
  const bool idle = g.nvalid == 0;

  float *const phi = a.phi;
  const long long *acc = reinterpret_cast<const long long *>(a.rho[cur]);
  // An image of the tile in shared memory, rows lo-1 .. hi+1 of tp columns: the
  // mesh is read and written through it a warp to a row, coalesced, and halo
  // nodes pass through it.  The mirror column and the tables of exchange words
  // follow it, then the snapshots, whose place first holds the charges.
  const int tp = 4 * nl, rows = hi - lo + 1, nwarp = nthr >> 5;
  float *const timg0 = edge + 4 * 2 * 128;  // row lo-1
  float *const timg = timg0 + tp;           // row lo
  long long *const wcol = reinterpret_cast<long long *>(timg0 + (size_t)(J.trows + 2) * tp);  // the mirror column's
  float *const mcol = reinterpret_cast<float *>(wcol + (J.trows + 1) / 2 * 2);  // charge, and potential at the start
  uint2 *const table = reinterpret_cast<uint2 *>(mcol + (J.trows + 3) / 4 * 4);
  uint2 *const ptable = table + J.tpairs;
  float4 *const snap = reinterpret_cast<float4 *>(ptable + J.ppairs);
  // the accumulator the step's push deposits into, cleared in equal shares
  // (called with loads in flight)
  auto clear_next = [&]() {
    if (!J.zero_next) return;
    unsigned long long *const nx = a.rho[cur ^ 1];
    const long long nodes = (long long)nnx * nny;
    const long long k0 = nodes * c / G, k1 = nodes * (c + 1) / G;
    const long long e0 = min(k1, (k0 + 1) & ~1ll), e1 = max(e0, k1 & ~1ll);
    if (tid == 0 && e0 > k0) nx[k0] = 0ull;
    if (tid == 0 && e1 < k1) nx[e1] = 0ull;
    for (long long k = e0 + 2 * tid; k < e1; k += 2 * nthr)
      *reinterpret_cast<ulonglong2 *>(nx + k) = make_ulonglong2(0ull, 0ull);
  };
  // real column of tile column tc (-1: none)
  const int nc = x1 - x0 + 2 * KX;
  auto real = [&](int tc) {
    const int i = x0 - KX + tc;
    return tc >= nc ? -1 : (i < 0 ? i + W : (i >= W ? i - W : i));
  };
  // The mesh comes in by asynchronous copies, a warp to a row, each lane down
  // one column at a time (its place in the mesh worked out once), and the
  // source terms are formed by the strips' own threads, four at a time: going
  // through the tile element by element took 150 instructions an element and
  // 10 us of a 512x2048 solve of 163.  These one-time phases are loops and
  // not unrolled: their instructions are fetched anew in every solve, and
  // straight-line code of them took longer to fetch than the data.
  float4 x[R], b[R];
#pragma unroll
  for (int r = 0; r < R; ++r) x[r] = b[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  bool seam = false;  // the mirror column differs from column 0 somewhere
  if (!REFINE) {
    long long *const aimg = reinterpret_cast<long long *>(snap);  // charges of rows lo..hi, then their source terms
#pragma unroll 1
    for (int tc = lane; tc < tp; tc += 32) {  // a lane's column, down the warp's rows
      const int i = real(tc);
      const size_t step = (size_t)nwarp * nnx;
      const float *from = phi + (size_t)(lo - 1 + warp) * nnx + max(i, 0);
      const long long *cfrom = acc + (size_t)(lo - 1 + warp) * nnx + max(i, 0);
#pragma unroll 2
      for (int r = warp; r < rows + 2; r += nwarp) {
        float *const to = timg0 + r * tp + tc;
        const bool inner = r > 0 && r <= rows;
        if (i >= 0) {
          copy4(to, from);
          if (inner) copy8(aimg + (r - 1) * tp + tc, cfrom);
        } else {
          *to = 0.0f;
          if (inner) aimg[(r - 1) * tp + tc] = 0ll;
        }
        from += step;
        cfrom += step;
      }
    }
    for (int r = tid; r < rows; r += nthr) {  // the mirror column
      copy4(mcol + r, phi + (size_t)(lo + r) * nnx + W);
      copy8(wcol + r, acc + (size_t)(lo + r) * nnx + W);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    clear_next();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const bool pow2 = (__double_as_longlong(a.cb) & 0xfffffffffffffll) == 0ll;
    const df cb = df_of(a.cb);
    const unsigned long long most = df_plain(cb, 0x1p-90f, 0x1p75f) ? 1ull << 48 : 0ull;
    for (int k = tid; k < 2 * tp; k += nthr) {
      const int up = k >= tp ? 1 : 0, tc = k - up * tp;
      const float v = timg0[up * (rows + 1) * tp + tc];
#pragma unroll
      for (int q = 0; q < 4; ++q) edge[(2 * q + up) * 128 + tc] = v;
    }
    // the strip's source terms, in the place of its charges; column 0 (or its
    // image past column W-1) is folded with the mirror column
    const int z = !act ? -1 : (g.i0 == 0 ? 0 : (MODE == kHalo && W >= g.i0 && W < g.i0 + 4 ? W - g.i0 : -1));
#pragma unroll 1
    for (int r = 0; r < g.nvalid; ++r) {
      const int j = g.row0 - lo + r;
      long long *const ar = aimg + j * tp + 4 * li;
      longlong2 u = *reinterpret_cast<const longlong2 *>(ar), v = *reinterpret_cast<const longlong2 *>(ar + 2);
      if (z >= 0) {
        const long long m = wcol[j];
        u.x += z == 0 ? m : 0ll;
        u.y += z == 1 ? m : 0ll;
        v.x += z == 2 ? m : 0ll;
        v.y += z == 3 ? m : 0ll;
        seam = seam || !(mcol[j] == timg[j * tp + 4 * li + z]);
      }
      auto b4 = [&](long long f) { return quarter(source(f, a.cb, cb, pow2, most)); };
      sts4(reinterpret_cast<float *>(ar), make_float4(b4(u.x), b4(u.y), b4(v.x), b4(v.y)));
    }
    seam = __syncthreads_or(seam);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < g.nvalid) {
        const int j = g.row0 - lo + r;
        x[r] = lds4(timg + j * tp + 4 * li);
        b[r] = lds4(reinterpret_cast<const float *>(aimg + j * tp + 4 * li));
      }
  } else {
    for (int k = tid; k < 4 * 2 * 128; k += nthr) edge[k] = 0.0f;
    for (int k = tid; k < (rows + 2) * tp; k += nthr) timg0[k] = 0.0f;
    clear_next();
  }
  sts4(first + mine, x[0]);
  if (R > 1) sts4(last + mine, x[R - 1]);
  if (near) cluster_join();

  // exchange words, two parities of: rows [by][bottom, top][K][ip] by
  // extended column, then (halo tiles) columns [row][bx][left, right][K]
  const int ip = J.ip, ipad = MODE == kHalo ? 16 : 0;
  const unsigned vbase = (unsigned)nby * 2u * K * ip, pwords = J.pwords;
  auto hrow = [&](int b_, int side, int k) { return (unsigned)(((b_ * 2 + side) * K + k) * ip + ipad); };
  auto vcol = [&](int j, int b_, int side) { return vbase + (unsigned)(((j * nbx + b_) * 2 + side) * K); };
  // Words go out and come in as pairs by way of an image of the tile in shared
  // memory, shared out evenly over the threads by tables of {word offset,
  // place in the image}.  In: rows of the blocks below and above over all the
  // tile's columns (the outermost one to the edge row), then the columns
  // beside the owned rows.  Out: the owned nodes within K of a boundary, and
  // the periodic images of those within K of column 0 or W.  kEdge marks a
  // place in the edge rows, kOne a single word (odd widths).
  constexpr unsigned kEdge = 1u << 30, kOne = 1u << 31;
  const int nc2 = (nc + 1) >> 1, h = r1 - r0;
  const int nlow = by > 0 ? K * nc2 : 0, nhigh = by < nby - 1 ? K * nc2 : 0;
  const int npair = G > 1 ? nlow + nhigh + (MODE == kHalo ? h * K : 0) : 0;
  const int w = x1 - x0, w2 = (w + 1) >> 1;
  const int plow = by > 0 ? K * w2 : 0, phigh = by < nby - 1 ? K * w2 : 0;
  // the periodic images of a row: as pairs when W is even, else word by word
  const int ni = W & 1 ? K : K >> 1, istep = W & 1 ? 1 : 2;
  const bool im0 = MODE == kHalo && x0 < K, im1 = MODE == kHalo && x1 > W - K;
  const int per = ((im0 ? 1 : 0) + (im1 ? 1 : 0)) * ni;
  const int nside = MODE == kHalo ? h * K : 0;
  const int nout = G > 1 ? plow + phigh + nside + per * ((by > 0 ? K : 0) + (by < nby - 1 ? K : 0)) : 0;
  if (G > 1 && !near) {
#pragma unroll 1
    for (int t = warp; t < 2 * K; t += nwarp) {  // row t of the bottom (t < K) and top boundaries
      const bool low = t < K;
      const int k = low ? t : t - K;
      if (low ? by == 0 : by == nby - 1) continue;
      const int jin = low ? r0 - K + k : r1 + k, jout = low ? r0 + k : r1 - K + k;
      const unsigned qin = hrow(low ? by - 1 : by + 1, low ? 1 : 0, k) + x0 - KX, qout = hrow(by, low ? 0 : 1, k);
      const unsigned to = jin < lo ? kEdge : (jin > hi ? kEdge | 128u : (unsigned)((jin - lo) * tp));
      for (int v = lane; v < nc2; v += 32)
        table[(low ? 0 : nlow) + k * nc2 + v] =
            make_uint2(qin + 2 * v, (to + 2 * v) | (2 * v + 1 >= nc ? kOne : 0u));
      const unsigned from = (unsigned)((jout - lo) * tp + KX);
      for (int v = lane; v < w2; v += 32)
        ptable[(low ? 0 : plow) + k * w2 + v] =
            make_uint2(qout + x0 + 2 * v, (from + 2 * v) | (2 * v + 1 >= w ? kOne : 0u));
      for (int v = lane; v < per; v += 32) {
        const bool at0 = im0 && v < ni;  // columns 0..K-1 again at W..W+K-1, W-K..W-1 at -K..-1
        const int kk = istep * (at0 ? v : v - (im0 ? ni : 0)), i = at0 ? kk : W - K + kk;
        ptable[plow + phigh + nside + ((low || by == 0 ? 0 : K) + k) * per + v] =
            make_uint2(qout + (at0 ? i + W : i - W), (from + i - x0) | (istep == 1 ? kOne : 0u));
      }
    }
    if (MODE == kHalo) {
#pragma unroll 1
      for (int row = warp; row < h; row += nwarp) {  // K/2 pairs on the left, K/2 on the right
        const int j = r0 + row, k = lane;
        if (k < K) {
          const bool left = k < (K >> 1);
          const int kk = 2 * (left ? k : k - (K >> 1));
          const unsigned qin = left ? vcol(j, bx == 0 ? nbx - 1 : bx - 1, 1) : vcol(j, bx + 1 == nbx ? 0 : bx + 1, 0);
          table[nlow + nhigh + row * K + k] =
              make_uint2(qin + kk, (unsigned)((j - lo) * tp + (left ? kk : nc - K + kk)));
          ptable[plow + phigh + row * K + k] =
              make_uint2(vcol(j, bx, left ? 0 : 1) + kk, (unsigned)((j - lo) * tp + KX + (left ? kk : w - K + kk)));
        }
      }
    }
  }
  // this thread's nodes that go out: rows within K of the block's bottom and
  // top, and every owned row of the lanes within K of its sides
  unsigned outrows = 0u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = g.row0 + r;
    if ((g.ownrows >> r) & 1u)
      if ((by > 0 && j < r0 + K) || (by < nby - 1 && j >= r1 - K) ||
          (MODE == kHalo && g.own && (g.i0 < x0 + K || g.i0 + 3 >= x1 - K)))
        outrows |= 1u << r;
  }
  // owned nodes into the image; then, after a barrier, out of it
  auto show = [&]() {
    float *const q = timg + (g.row0 - lo) * tp + 4 * li;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((outrows >> r) & 1u) sts4(q + r * tp, x[r]);
  };
  auto publish = [&](int e) {
    const unsigned ep = ebase + (unsigned)e;
    unsigned long long *const hw = J.halo + ((e & 1) ? pwords : 0u);
#pragma unroll 4
    for (int v0 = tid - lane; v0 < nout; v0 += nthr) {  // the same for a warp's lanes
      if (v0 + lane >= nout) continue;
      const uint2 t = ptable[v0 + lane];
      const float *from = timg + (t.y & ~kOne);
      if (t.y & kOne)
        st_word(hw + t.x, from[0], ep);
      else
        st_word2(hw + t.x, from[0], from[1], ep);
    }
  };
  // waits for the words of exchange e and puts them in shared memory; false
  // if the wait gave up
  auto receive = [&](int e, int to_edge) -> bool {
    const unsigned ep = ebase + (unsigned)e;
    const unsigned long long *const hw = J.halo + ((e & 1) ? pwords : 0u);
    constexpr int NB = 4;  // pairs of a thread in flight
    for (int v0 = tid - lane; v0 < npair; v0 += NB * nthr) {  // the same for a warp's lanes
      const int u0 = min(v0 + lane, npair - 1);
      uint2 t[NB];
      unsigned long long w[NB][2];
#pragma unroll
      for (int q = 0; q < NB; ++q)  // past the end: the first pair again (no branch around a load)
        t[q] = table[u0 + q * nthr < npair ? u0 + q * nthr : u0];
      auto here = [&](int q) {
        return (unsigned)(w[q][0] >> 32) == ep && ((t[q].y & kOne) || (unsigned)(w[q][1] >> 32) == ep);
      };
      // Wait on the first pair alone: the others come from the same blocks, and
      // polling all of them loads L2 while the blocks are still writing
      // (512x2048, depth 8: 0.79 us a sweep against 0.74).
      if (!wait_for(ctl, [&]() {
            ld_word2(hw + t[0].x, w[0][0], w[0][1]);
            return here(0);
          }))
        return false;
      if (!wait_for(ctl, [&]() {
            bool all = true;
#pragma unroll
            for (int q = 1; q < NB; ++q) ld_word2(hw + t[q].x, w[q][0], w[q][1]);
#pragma unroll
            for (int q = 1; q < NB; ++q) all = all && here(q);
            return all;
          }))
        return false;
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        float *to = (t[q].y & kEdge) ? edge + to_edge * 256 : timg;
        to += t[q].y & ~(kEdge | kOne);
        to[0] = __uint_as_float((unsigned)w[q][0]);
        if (!(t[q].y & kOne)) to[1] = __uint_as_float((unsigned)w[q][1]);
      }
    }
    return true;
  };
  // this thread's rows with halo nodes from the image, which holds the owned
  // nodes beside them as well (show)
  unsigned inrows = 0u;
  const bool beside = MODE == kHalo && act && g.own != 15u && g.i0 < x1 + KX;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r < g.nvalid && (beside || !((g.ownrows >> r) & 1u))) inrows |= 1u << r;
  auto take = [&]() {
    const float *const img = timg + (g.row0 - lo) * tp + 4 * li;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((inrows >> r) & 1u) x[r] = lds4(img + r * tp);
  };
  // The same exchange inside a cluster: the rows [2][bottom, top][K][tp] that
  // the neighbours write, in place of the tables.  A neighbour sends exchange
  // e+2 once it has exchange e+1 of this CTA, which takes e before that.
  float *const got = reinterpret_cast<float *>(table);
  // and after them the maxima of checked blocks [2][CTA][sweep], from every CTA
  float *const votes = got + 4 * K * tp;
  const bool dn = by > 0, up = by < nby - 1;
  const unsigned gpar = 8u * K * tp;  // bytes of one exchange's rows
  // where this strip's first row goes and comes from, and its rows (bits 0-7:
  // to the block below, 8-15: above; 16-23: those from above in a strip that
  // also has rows from below)
  const unsigned dto = near ? cluster_addr(smem_addr(got), max(by - 1, 0)) + 16u * li + 4u * (K + g.row0 - r0) * tp : 0u;
  const unsigned uto =
      near ? cluster_addr(smem_addr(got), min(by + 1, nby - 1)) + 16u * li + 4u * (K + g.row0 - r1) * tp : 0u;
  const float *const zin = got + 4 * li + (K + g.row0 - (g.row0 < r0 ? r0 : r1)) * tp;
  unsigned trades = 0u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = g.row0 + r;
    if ((outrows >> r) & 1u) {
      if (dn && j < r0 + K) trades |= 1u << r;
      if (up && j >= r1 - K) trades |= 0x100u << r;
    }
    if (j >= r1 && g.row0 < r0) trades |= 0x10000u << r;
  }
  const bool eslow = !idle && south_edge && dn, eshigh = !idle && north_edge && up;
  auto send = [&](int e) {
    const unsigned o = (e & 1) ? gpar : 0u;
    const unsigned bar = smem_addr(&js->arrived[e & 1]);
    if (trades & 0xffu) {
      const unsigned nb = cluster_addr(bar, by - 1);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((trades >> r) & 1u) st_cluster(dto + o + 4u * r * tp, x[r], nb);
    }
    if (trades & 0xff00u) {
      const unsigned nb = cluster_addr(bar, by + 1);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((trades >> (8 + r)) & 1u) st_cluster(uto + o + 4u * r * tp, x[r], nb);
    }
  };
  auto await = [&](int e) -> bool {
    const unsigned bar = smem_addr(&js->arrived[e & 1]), parity = ((unsigned)(e - 1) >> 1) & 1u;
    if (!wait_for(ctl, [&]() { return cluster_wait(bar, parity); })) return false;
    if (tid == 0) mbar_arrive_expect_tx(&js->arrived[e & 1], near_bytes);  // for exchange e+2
    return true;
  };
  auto take_rows = [&](int e, int to_edge) {
    const int o = (e & 1) ? 2 * K * tp : 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((inrows >> r) & 1u) x[r] = lds4(zin + o + (r - ((trades >> (16 + r)) & 1u ? h : 0)) * tp);
    if (eslow) sts4(edge + to_edge * 256 + 4 * li, lds4(got + o + 4 * li));
    if (eshigh) sts4(edge + to_edge * 256 + 128 + 4 * li, lds4(got + o + (2 * K - 1) * tp + 4 * li));
  };
  auto fail = [&]() {
    js->bail = 1;
    if (!*(volatile int *)&ctl->abort) {
      atomicExch(&ctl->abort, 1);
      atomicOr(&ctl->step_flags, (uint32_t)CUPIC_FLAG_TIMEOUT);
    }
  };

  // an exchange up to the arrival of the neighbours' nodes, and (after a
  // barrier, outside a cluster) their way into the strips; between() reads
  // what the grid has found while the nodes are on their way
  auto trade_out = [&](int &e, int &es, auto &&between) {
    ++e;
    es = (es + 1) & 3;
    if (near) {
      send(e);
      between();
      if (!await(e)) fail();
    } else {
      show();
      __syncthreads();
      publish(e);
      between();
      if (!receive(e, es)) fail();
    }
  };
  auto trade_in = [&](int e, int es) {
    if (near)
      take_rows(e, es);
    else
      take();
  };

  auto rows_at = [&](int es_, int p_) {
    Rows w_;
    w_.sA = south_edge ? edge + es_ * 256 + 4 * li : last + p_ * par + soff;
    w_.nA = north_edge || idle ? edge + es_ * 256 + 128 + 4 * li : first + p_ * par + noff;
    w_.sB = south_edge ? w_.sA : last + (p_ ^ 1) * par + soff;
    w_.nB = north_edge || idle ? w_.nA : first + (p_ ^ 1) * par + noff;
    w_.wA = first + p_ * par + mine;
    w_.wB = first + (p_ ^ 1) * par + mine;
    w_.to_last = 2 * par;
    return w_;
  };
  // the last CTA to finish puts the counters back to zero and advances the
  // epochs past this solve's
  auto finish = [&](int used) {
    unsigned next = ebase + (unsigned)used + 2u;
    const bool wrap = next > kEpochEnd;  // start over, above the tags left in gmax
    if (wrap) next = 0u;
    for (int k = 0; k < (G > 1 ? 4 : 0); ++k) J.tbar[k] = 0u;
    for (int k = 0; k < (wrap ? 128 : REFINE && G > 1 ? 4 : 0); ++k) J.gmax[k] = 0ull;
    ctl->jepoch = next;
  };

  // ---- the precision form (refine.cu) -----------------------------------
  // phi64 of the tile, halo included, stays in shared memory: a correction
  // forms the FP64 residual of every node as its source, runs its sweeps from
  // zero, trades once more so that the halo holds the neighbours' correction
  // too, and adds it.  The residual's maximum goes to the grid while the
  // sweeps run and is looked at before the correction is added; a solve that
  // had already passed its test drops it.  Same operations, same order, same
  // bits as one launch per residual, solve and update.  Bound by the FP64
  // pipe (six operations a node of the tile) and the sweeps with their
  // exchanges: a 512x2048 correction of 32 sweeps takes 52 us; a launch per
  // correction, with a grid barrier and every residual's potential read
  // again, took 96.
  if constexpr (REFINE) {
    double *const p64 = reinterpret_cast<double *>(ptable + J.ppairs);  // rows lo-1 .. hi+1, [tp]
    double *const q64 = p64 + (g.row0 - lo + 1) * tp + 4 * li;          // this strip's first row
    int cc[4];  // real columns of the lane's elements (-1: none)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = g.i0 + q;
      cc[q] = !act || (MODE != kHalo && i >= W) || i >= x1 + KX ? -1 : (i < 0 ? i + W : (i >= W ? i - W : i));
    }
    double *const phi64 = J.r64_phi;
#pragma unroll 1
    for (int r = warp; r < rows + 2; r += nwarp)
#pragma unroll 1
      for (int tc = lane; tc < tp; tc += 32) {
        const int i = real(tc);
        if (i >= 0)
          copy8(p64 + r * tp + tc, phi64 + (size_t)(lo - 1 + r) * nnx + i);
        else
          p64[r * tp + tc] = 0.0;
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the columns west and east of this lane's, relative to them
    const int wc = MODE == kHalo ? (li == 0 ? 0 : -1) : (li == 0 ? W - 1 : -1);
    const int ring0 = -4 * li;  // column 0 of a ring
    const int m_ = J.max_sweeps;  // sweeps of a correction
    const unsigned long long inf64 = 0x7ff0000000000000ull;
    int e = 0, es = 0, p = 0, done = 0, q = 0;
    double res = 0.0;
    __syncthreads();
    // the grid's maximum of correction n (warp 0)
    auto wait_res = [&](int n) {
      const unsigned target = (unsigned)G * ((unsigned)n / 4u + 1u);
      const bool ok = wait_for(ctl, [&]() { return ld_acquire(&J.tbar[n & 3]) >= target; });
      const unsigned long long most = ld_word(&J.gmax[n & 3]);
      if (lane == 0) js->res64[n & 1] = most;
      if (!ok) fail();
    };
    for (;;) {
      unsigned long long mx = 0ull;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        b[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < g.nvalid) {
          const double *const z = q64 + r * tp;
          const double *const src = J.r64_b + (size_t)(g.row0 + r) * nnx;
          // the strip's columns in 16-byte loads
          auto row4 = [](const double *q, double (&d)[4]) {
            const double2 u = *reinterpret_cast<const double2 *>(q), v_ = *reinterpret_cast<const double2 *>(q + 2);
            d[0] = u.x;
            d[1] = u.y;
            d[2] = v_.x;
            d[3] = v_.y;
          };
          double zc[4], zn[4], zs[4];
          row4(z, zc);
          row4(z + tp, zn);
          row4(z - tp, zs);
          const double zw = z[wc], ze = z[MODE != kHalo && g.me == 3 ? ring0 : 4], z0 = MODE == kRingRagged ? z[ring0] : 0.0;
          float v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double wv = k == 0 ? zw : zc[k > 0 ? k - 1 : 0];
            double ev = k == 3 ? ze : zc[k < 3 ? k + 1 : 3];
            if (MODE == kRingRagged && g.me == k) ev = z0;
            const double rr = (cc[k] >= 0 ? src[cc[k]] : 0.0) - (times4(zc[k]) - (((wv + ev) + zn[k]) + zs[k]));
            v[k] = quarter(to_float(rr));
            const unsigned long long bits = (unsigned long long)__double_as_longlong(rr) & 0x7fffffffffffffffull;
            if (((g.own >> k) & 1u) && ((g.ownrows >> r) & 1u) && bits <= inf64 && bits > mx) mx = bits;
          }
          b[r] = make_float4(v[0], v[1], v[2], v[3]);
        }
        x[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
      if (lane == 0) js->w64[warp] = mx;
      __syncthreads();
      if (warp == 0) {
        mx = lane < (nthr >> 5) ? js->w64[lane] : 0ull;
        for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
        if (lane == 0) {
          if (G > 1) {
            // slot q+2 was last read before anyone could add to slot q
            if (c == 0) *(volatile unsigned long long *)&J.gmax[(q + 2) & 3] = 0ull;
            atomicMax(&J.gmax[q & 3], mx);
            __threadfence();
            atomicAdd(&J.tbar[q & 3], 1u);
          } else {
            js->res64[q & 1] = mx;
          }
        }
        if (G > 1 && done >= J.r64_mx) wait_res(q);
      }
      // the correction starts from zero
      sts4(first + p * par + mine, x[0]);
      if (R > 1) sts4(last + p * par + mine, x[R - 1]);
      if (!idle && south_edge) sts4(edge + es * 256 + 4 * li, x[0]);
      if (!idle && north_edge) sts4(edge + es * 256 + 128 + 4 * li, x[0]);
      __syncthreads();
      if (js->bail) break;
      if (G == 1 || done >= J.r64_mx) {
        res = __longlong_as_double((long long)js->res64[q & 1]);
        if (done >= J.r64_mx || (done >= J.r64_mn && res < J.r64_tol && !J.trial)) break;
      }
      const int todo = min(m_, J.r64_mx - done);
      for (int sw = 0; sw < todo;) {
        const int nsw = G > 1 ? min(K, todo - sw) : todo;
        Rows at = rows_at(es, p);
        int m = 0;
        float md = 0.0f;
        unsigned keep = 0u;
        if (g.full)
          sweeps<R, MODE, true, false>(x, b, g, at, m, nsw, md, keep);
        else
          sweeps<R, MODE, false, false>(x, b, g, at, m, nsw, md, keep);
        p ^= nsw & 1;
        sw += nsw;
        if (G > 1) {  // also after the last sweep: the halo's correction is added too
          trade_out(e, es, [&]() {
            if (sw >= todo && warp == 0) wait_res(q);
          });
          if (!near) __syncthreads();
          trade_in(e, es);
          p ^= 1;
          sts4(first + p * par + mine, x[0]);
          if (R > 1) sts4(last + p * par + mine, x[R - 1]);
          __syncthreads();
          if (js->bail) break;
        }
      }
      if (js->bail) break;
      if (G > 1) {
        res = __longlong_as_double((long long)js->res64[q & 1]);
        if (done >= J.r64_mn && res < J.r64_tol && !J.trial) break;
      }
      auto add_row = [&](double *z, const float4 &d) {
        double2 u = *reinterpret_cast<double2 *>(z), v = *reinterpret_cast<double2 *>(z + 2);
        u.x += to_double(d.x);
        u.y += to_double(d.y);
        v.x += to_double(d.z);
        v.y += to_double(d.w);
        *reinterpret_cast<double2 *>(z) = u;
        *reinterpret_cast<double2 *>(z + 2) = v;
      };
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r < g.nvalid) add_row(q64 + r * tp, x[r]);
      if (!idle && south_edge && by > 0) add_row(p64 + 4 * li, lds4(edge + es * 256 + 4 * li));
      if (!idle && north_edge && by < nby - 1)
        add_row(p64 + (rows + 1) * tp + 4 * li, lds4(edge + es * 256 + 128 + 4 * li));
      done += todo;
      ++q;
      __syncthreads();
    }
    // phi64, its FP32 copy and the field (mesh.cu:413-468, rounded once), row
    // by row; a quotient by a power of two is the product by its inverse
    const double d1 = a.ds_d, d2 = 2.0 * a.ds_d;
    const bool pow2 = (__double_as_longlong(d1) & 0xfffffffffffffll) == 0ll;
    const double i1 = 1.0 / d1, i2 = 1.0 / d2;
    auto over = [&](double v, double d, double i) { return pow2 ? v * i : v / d; };
    __syncthreads();
    const int ja = by == 0 ? 0 : r0, jb = by == nby - 1 ? nny : r1;
#pragma unroll 1
    for (int j = ja + warp; j < jb; j += nwarp) {
      const double *const z = p64 + (j - lo + 1) * tp;
#pragma unroll 1
      for (int i = x0 + lane; i < x1; i += 32) {
        const int tc = i - x0 + KX;
        const size_t o = (size_t)j * nnx + i;
        if (j > 0 && j < nny - 1) {
          phi64[o] = z[tc];
          if (i == 0) phi64[o + W] = z[tc];
        }
        const float f = to_float(z[tc]);
        a.phi[o] = f;
        if (i == 0) a.phi[o + W] = f;
        if (J.do_field) {
          double ex = 0.0, ey;
          if (j == 0) {
            ey = over(z[tc] - z[tc + tp], d1, i1);
          } else if (j == nny - 1) {
            ey = over(z[tc - tp] - z[tc], d1, i1);
          } else {
            const double wv = z[MODE != kHalo && tc == 0 ? W - 1 : tc - 1], ev = z[MODE != kHalo && tc == W - 1 ? 0 : tc + 1];
            ex = over(wv - ev, d2, i2);
            ey = over(z[tc - tp] - z[tc + tp], d2, i2);
          }
          const float2 E = make_float2(to_float(ex), to_float(ey));
          a.E[o] = E;
          if (i == 0) a.E[o + W] = E;
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(&ctl->jdone, 1u) == (unsigned)G - 1u) {
        __threadfence();
        ctl->jdone = 0u;
        if (J.r64_stats) {
          ctl->sweeps = done;
          ctl->residual = (float)res;
        }
        finish(e);
      }
    }
    return;
  }

  // ---- sweeps ----------------------------------------------------------
  // A checked sweep is one that the stop rule looks at; when the solve cannot
  // stop early only its last sweep is checked, for the report.  Blocks of at
  // most K sweeps end with an exchange; nq counts the blocks that had
  // checked sweeps, whose maxima use slot nq & 3.
  const bool report = J.write_stats || J.tol > 0.0;
  const bool early = J.tol > 0.0 && J.min_sweeps < J.max_sweeps;
  bool checks = report;  // cleared while a stopped solve sweeps up to its last sweep
  const int KB = G > 1 ? K : kSoloBlock;
  int maxs = J.max_sweeps, p = 0, es = 0, done = 0, e = 0, nq = 0;
  float resv = INFINITY;
  bool pend = false;  // the decision on block nq-1 is outstanding
  int pstart = 0, pes = 0;
  unsigned pmask = 0u;
  // the stop decision on checked block q, taken by warp 0 once every CTA's
  // maxima are in (usually long before it asks).  In a cluster every CTA has
  // sent them here: reading a counter and then the maxima from L2 took two
  // round trips a block (64x256, 2000 checked sweeps: 610 -> 543 us).
  auto decide = [&](int q, unsigned mask) {
    const bool mineck = (mask >> lane) & 1u;
    bool ok;
    float v = 0.0f;
    if (near) {
      const unsigned bar = smem_addr(&js->voted[q & 1]), parity = ((unsigned)q >> 1) & 1u;
      ok = wait_for(ctl, [&]() { return cluster_wait(bar, parity); });
      for (int k = 0; k < G; ++k) v = fmaxf(v, votes[((q & 1) * G + k) * 32 + lane]);
      if (lane == 0) mbar_arrive_expect_tx(&js->voted[q & 1], 128u * G);  // for block q+2, sent after this CTA's q+1
    } else {
      const unsigned target = (unsigned)G * ((unsigned)q / 4u + 1u);
      ok = wait_for(ctl, [&]() { return ld_acquire(&J.tbar[q & 3]) >= target; });
      if (mineck) v = __uint_as_float((unsigned)ld_word(&J.gmax[(q & 3) * 32 + lane]));
    }
    const unsigned pass = __ballot_sync(kFull, mineck && (double)v < J.tol && !J.trial);
    const int k = pass ? __ffs(pass) - 1 : 31 - __clz(mask);
    const float vk = __shfl_sync(kFull, v, k);
    if (lane == 0) {
      js->dec[q & 1] = pass ? k : -1;
      js->decv[q & 1] = vk;
      if (!ok) fail();
    }
  };
  auto stop_at = [&](int start, int k, int slot, int es_) {
    // back to the start of the block, then up to its sweep k
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = snap[(slot * R + r) * nthr + tid];
    es = es_;
    done = start;
    maxs = start + k + 1;
    checks = false;
    sts4(first + p * par + mine, x[0]);
    if (R > 1) sts4(last + p * par + mine, x[R - 1]);
    __syncthreads();
  };
  const bool owns = __any_sync(kFull, g.ownrows != 0u);
  for (int k = tid; k < 128; k += nthr) js->cm[k >> 5][k & 31] = 0u;
  __syncthreads();
  for (;;) {
    if (done >= maxs) {
      if (!pend) break;
      if (warp == 0) decide(nq - 1, pmask);
      __syncthreads();
      pend = false;
      if (js->bail) break;
      resv = js->decv[(nq - 1) & 1];
      const int k = js->dec[(nq - 1) & 1];
      if (k < 0) break;
      stop_at(pstart, k, (nq - 1) & 1, pes);
    }
    // Whole blocks without a checked sweep, and not the last ones: what the
    // general path below decides costs some 600 cycles a block (512x2048, depth
    // 8: 0.72 -> 0.62 us a sweep; 256x1024, depth 4: 0.69 -> 0.56).
    if (G > 1 && !pend && !(seam && done == 0)) {
      int next = maxs;  // the next checked or last sweep
      if (checks && early) {
        const unsigned s = (unsigned)max(done + 1, J.min_sweeps), ev = (unsigned)J.check_every;
        next = (int)min((unsigned)next, ev == 1u ? s : (s + ev - 1u) / ev * ev);
      }
      for (int n = (next - 1 - done) / K; n > 0; --n) {
        Rows at = rows_at(es, p);
        int m = 0;
        float md = 0.0f;
        unsigned keep = 0u;
        if (g.full)
          sweeps<R, MODE, true, false>(x, b, g, at, m, K, md, keep);
        else
          sweeps<R, MODE, false, false>(x, b, g, at, m, K, md, keep);
        p ^= (K & 1) ^ 1;
        done += K;
        trade_out(e, es, []() {});
        if (!near) __syncthreads();
        trade_in(e, es);
        sts4(first + p * par + mine, x[0]);
        if (R > 1) sts4(last + p * par + mine, x[R - 1]);
        __syncthreads();
        if (js->bail) break;
      }
      if (js->bail) break;
    }
    const int nsw = min(KB, maxs - done), start = done, es0 = es;
    unsigned mask = 0u, keep = 0u;
    if (checks) {
      if (early && J.check_every == 1) {
        const int s = max(J.min_sweeps - start - 1, 0);
        if (s < nsw) mask = (kFull >> (32 - nsw)) & (kFull << s);
      } else if (early) {
        for (int s = (start / J.check_every + 1) * J.check_every; s <= start + nsw; s += J.check_every)
          if (s >= J.min_sweeps) mask |= 1u << (s - start - 1);
      }
      if (start + nsw == J.max_sweeps) mask |= 1u << (nsw - 1);
      if (mask && early) {
#pragma unroll
        for (int r = 0; r < R; ++r) snap[((G > 1 ? nq & 1 : 0) * R + r) * nthr + tid] = x[r];
      }
    }
    Rows at = rows_at(es, p);
    int m = 0;
    float md = 0.0f;
    if (seam && start == 0) {  // the first sweep reads the caller's mirror column
      md = sweep<R, MODE, false, true, true>(x, b, lds4(at.sA), lds4(at.nA), g, mcol + (g.row0 - lo));
      const unsigned u = __reduce_max_sync(kFull, __float_as_uint(md));
      if (lane == 0) keep = u;
      sts4(at.wB, x[0]);
      if (R > 1) sts4(at.wB + at.to_last, x[R - 1]);
      __syncthreads();
      at = rows_at(es, p ^ 1);
      m = 1;
    }
    // sweeps before the next checked one; rows of a halo alone are not looked at
    const int plain = mask >> m && owns ? m + __ffs(mask >> m) - 1 : nsw;
    if (g.full) {
      sweeps<R, MODE, true, false>(x, b, g, at, m, plain, md, keep);
      sweeps<R, MODE, true, true>(x, b, g, at, m, nsw, md, keep);
    } else {
      sweeps<R, MODE, false, false>(x, b, g, at, m, plain, md, keep);
      sweeps<R, MODE, false, true>(x, b, g, at, m, nsw, md, keep);
    }
    p ^= nsw & 1;
    done += nsw;
    if (mask && owns) {
      const unsigned u = __reduce_max_sync(kFull, __float_as_uint(md));
      if (lane == nsw - 1) keep = u;
    }
    if ((mask >> lane) & 1u) atomicMax(&js->cm[nq & 3][lane], keep);
    // the last exchange serves the field; a solve of less than K sweeps
    // trades once too, so that no CTA stores its rows before its neighbours
    // have loaded them
    const bool trade = G > 1 && ((nsw == K && (done < maxs || J.do_field)) || (done >= maxs && e == 0));
    auto look = [&]() {
      if (pend && warp == 0) decide(nq - 1, pmask);
    };
    if (trade)
      trade_out(e, es, look);
    else
      look();
    if (!near || !trade) __syncthreads();
    if (trade) {
      trade_in(e, es);
      p ^= 1;
      sts4(first + p * par + mine, x[0]);
      if (R > 1) sts4(last + p * par + mine, x[R - 1]);
      __syncthreads();
    }
    if (js->bail) break;
    if (pend) {
      pend = false;
      const int k = js->dec[(nq - 1) & 1];
      if (k >= 0) {
        resv = js->decv[(nq - 1) & 1];
        stop_at(pstart, k, (nq - 1) & 1, pes);
        continue;
      }
    }
    if (mask) {
      if (G == 1) {
        const float v = __uint_as_float(js->cm[nq & 3][lane]);
        const unsigned pass = __ballot_sync(kFull, early && ((mask >> lane) & 1u) && (double)v < J.tol && !J.trial);
        const int k = pass ? __ffs(pass) - 1 : 31 - __clz(mask);
        resv = __shfl_sync(kFull, v, k);
        if (warp == 0) js->cm[(nq + 2) & 3][lane] = 0u;
        ++nq;
        if (pass) stop_at(start, k, 0, es0);
      } else {
        if (near && early) {
          if (warp == 0) {  // eight lanes to a CTA
            const float4 u = lds4(reinterpret_cast<const float *>(js->cm[nq & 3]) + 4 * (lane & 7));
            const unsigned to = smem_addr(votes + ((nq & 1) * G + c) * 32) + 16u * (lane & 7), bar = smem_addr(&js->voted[nq & 1]);
            for (int k = lane >> 3; k < G; k += 4) st_cluster(cluster_addr(to, k), u, cluster_addr(bar, k));
            __syncwarp();
            js->cm[(nq + 2) & 3][lane] = 0u;
          }
        } else if (warp == 0) {
          if ((mask >> lane) & 1u)
            atomicMax(&J.gmax[(nq & 3) * 32 + lane],
                      ((unsigned long long)(ebase + (unsigned)nq + 1u) << 32) | js->cm[nq & 3][lane]);
          js->cm[(nq + 2) & 3][lane] = 0u;
          __threadfence();
          __syncwarp();
          if (lane == 0) atomicAdd(&J.tbar[nq & 3], 1u);
        }
        pend = early;
        pstart = start;
        pes = es0;
        pmask = mask;
        ++nq;
      }
    }
  }

  // ---- results: the image with its edge rows, then row by row phi and
  // E = -grad phi (mesh.cu:413-468) of the owned nodes ----------------------
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r < g.nvalid) sts4(timg + (g.row0 - lo + r) * tp + 4 * li, x[r]);
  for (int k = tid; k < 2 * tp; k += nthr) {
    const int up = k >= tp ? 1 : 0, tc = k - up * tp;
    timg0[up * (rows + 1) * tp + tc] = edge[es * 256 + up * 128 + tc];
  }
  __syncthreads();
  // a quotient by a power of two is the product by its inverse, exactly
  const bool pow2 = (__float_as_uint(a.ds) & 0x7fffffu) == 0u;
  const float inv1 = __fdiv_rn(1.0f, a.ds), inv2 = __fdiv_rn(1.0f, a.two_ds);
  auto over = [&](float v, float d, float i) { return pow2 ? __fmul_rn(v, i) : __fdiv_rn(v, d); };
#pragma unroll 1
  for (int j = r0 + warp; j < r1; j += nwarp) {
    const float *const z = timg + (j - lo) * tp + KX - x0;
    float *const pr = phi + (size_t)j * nnx;
    float2 *const er = a.E + (size_t)j * nnx;
#pragma unroll 2
    for (int i = x0 + lane; i < x1; i += 32) {
      const float *const q = z + i;
      pr[i] = q[0];
      if (i == 0) pr[W] = q[0];
      if (J.do_field) {
        const float wv = q[MODE != kHalo && i == 0 ? W - 1 : -1], ev = q[MODE != kHalo && i == W - 1 ? 1 - W : 1];
        const float2 E =
            make_float2(over(__fsub_rn(wv, ev), a.two_ds, inv2), over(__fsub_rn(q[-tp], q[tp]), a.two_ds, inv2));
        er[i] = E;
        if (i == 0) {
          // beside a Dirichlet row, whose mirror column keeps its own value
          const float sv = j == 1 ? phi[W] : q[-tp], nv = j == nny - 2 ? phi[(size_t)(nny - 1) * nnx + W] : q[tp];
          er[W] = make_float2(E.x, over(__fsub_rn(sv, nv), a.two_ds, inv2));
        }
      }
    }
  }
  if (J.do_field)
    for (int side = 0; side < 2; ++side) {  // the Dirichlet rows
      if (side == 0 ? by > 0 : by < nby - 1) continue;
      const int j = side == 0 ? 0 : nny - 1;
      const float *const z = side == 0 ? timg : timg + (rows - 1) * tp;  // the row beside it
      for (int i = x0 + tid; i < x1 + (x0 == 0 ? 1 : 0); i += nthr) {
        const int ii = i < x1 ? i : W;  // the mirror column goes with column 0
        const float d = phi[(size_t)j * nnx + ii], v = z[(i < x1 ? i : 0) - x0 + KX];
        a.E[(size_t)j * nnx + ii] =
            make_float2(0.0f, side == 0 ? over(__fsub_rn(d, v), a.ds, inv1) : over(__fsub_rn(v, d), a.ds, inv1));
      }
    }
  // the last CTA to finish also writes the report
  if (G > 1) __syncthreads();
  if (tid == 0) {
    if (G > 1) __threadfence();
    if (G == 1 || atomicAdd(&ctl->jdone, 1u) == (unsigned)G - 1u) {
      if (G > 1) __threadfence();
      ctl->jdone = 0u;
      if (J.write_stats) {
        ctl->sweeps = done;
        ctl->residual = G > 1 && report && !early && nq > 0
                            ? __uint_as_float((unsigned)ld_word(&J.gmax[((nq - 1) & 3) * 32 + ((J.max_sweeps - 1) % KB)]))
                            : resv;
      }
      finish(max(e, nq));
    }
  }
}

template <int R, int MODE, bool REFINE>
__global__ void __launch_bounds__(32 * kTileWarps, 1) k_tile(SimArgs a, JacobiArgs J) {
  extern __shared__ __align__(16) float tsm[];
  __shared__ Scratch js;
  if (threadIdx.x == 0) js.bail = 0;
  __syncthreads();
  solve<R, MODE, REFINE>(a, J, blockIdx.x, tsm, &js);
  if (MODE != kHalo && J.near) {
    // A CTA whose wait gave up stays until its neighbours have stopped sending;
    // without that, all that was sent here has been taken.
    __syncthreads();
    if (js.bail) {
      cluster_arrive();
      cluster_join();
      __nanosleep(100000);
    }
  }
}

using Kernel = void (*)(SimArgs, JacobiArgs);

// the kernel of MODE with strips of r rows (1..kTileRows)
template <int MODE, bool REFINE>
inline Kernel pick(int r) {
  switch (r) {
    case 1: return k_tile<1, MODE, REFINE>;
    case 2: return k_tile<2, MODE, REFINE>;
    case 3: return k_tile<3, MODE, REFINE>;
    case 4: return k_tile<4, MODE, REFINE>;
    case 5: return k_tile<5, MODE, REFINE>;
    case 6: return k_tile<6, MODE, REFINE>;
    case 7: return k_tile<7, MODE, REFINE>;
    default: return k_tile<8, MODE, REFINE>;
  }
}

}  // namespace tile
}  // namespace cupic
