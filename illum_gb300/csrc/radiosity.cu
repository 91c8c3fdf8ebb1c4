// radiosity.cu — solve (I - F) x = E for the form-factor matrix (CSR by
// receiver row), the linear system the reference solves with a forward
// solve plus Gauss-Seidel sweeps (src/cpp/arma_util.cpp:4-17,
// src/cpp/illum_cli.cpp:425-440).
//
// GPU scheme: Jacobi sweeps x <- E + F x over the rows that have entries
// (rows without entries are x = E exactly) inside ONE persistent cooperative
// kernel, one grid barrier per sweep. The solve works on facets renumbered in
// the LBVH's Morton order, and the matrix is cut into row tiles: runs of
// Morton-consecutive rows with about nnz / (co-resident blocks) entries each.
// A tile's rows see a compact set of facets (its halo), so a block first
// gathers the halo's x values into shared memory and then streams the tile's
// entries, each a 16-bit halo index (with the pair's row-end bits) and a value. The
// stream reaches shared memory by bulk copies (cp.async.bulk with mbarrier
// completion) that one producer warp issues ahead of the 31 consumer warps,
// so DRAM keeps working while the consumers gather the next tile's halo or
// finish a tile's rows. The
// tile's entries, row after row, are split into equal runs, one per thread
// (entries of a row that straddles threads are combined in a fixed order),
// so every thread of every block does the same amount of work whatever the
// row lengths. The per-tile residual partials meet in integer accumulators
// (order-independent sums), so all blocks take the same stop decisions and
// results are run-to-run deterministic. The residual of iterate x_k is
// E - (I - F) x_k = x_{k+1} - x_k, so it comes for free with the next sweep;
// iteration stops once its 2-norm is <= tol.
// With albedo-scaled form factors the iteration matrix has spectral radius
// well below 1, so Jacobi converges in a handful of sweeps; a multicolour
// Gauss-Seidel would need one grid barrier per colour, and the cliques of
// mutually visible crater facets force hundreds of colours.
//
// FP64 arithmetic runs at about one fused multiply-add per clock per SM on
// GB300, so the double-precision sweeps evaluate their dot products in
// FP32-pair ("double-float") arithmetic on the FP32 pipes instead: each
// value and each x is split into hi + lo floats (48 significant bits), the
// product hi*hi is taken exactly with an FMA, the cross terms are added,
// and the running sum is kept as an unevaluated float pair by TwoSum
// (Dekker 1971; Knuth TAOCP vol. 2, 4.2.2). The relative error of a row sum
// is ~2^-46 (vs 2^-53 for FP64), orders of magnitude below the solve
// tolerance. The iterate is kept as its scattered part s = x - E, also a
// double-float, with E in FP64: x = E + s is formed in FP64 only when the
// solve ends, so the result carries E exactly and s to ~2^-46 of |s|
// (|s| <= albedo * max x). Per row and sweep the finishing work (s' = F x,
// the change s' - s, the halo copy x' = E + s') is FP32 arithmetic, and the
// squared changes are summed in FP32 (a stop decision needs a few digits).
//
// The double-float values are stored as two arrays, hi = fl(F) and
// lo = fl(F - hi).
//
// Mixed precision: values stored as bf16 with a per-row fp32 scale, fp32
// accumulation for the inner sweeps, and an outer refinement whose residual
// r = fl(F) x - s is accumulated in double-float from the fp32 values hi (x and
// s in double-float, E in FP64, r rounded to fp32 for the inner sweeps): the
// fixed point is that of (I - fl(F)) x = E,
// within ~1e-7 of the scattered flux of the fp64 system's. A mesh whose
// sweep budget runs out in a refinement round stops after the round's update
// without another residual pass. A round runs min(budget, RAD_INNER) inner
// sweeps (the smallest budget of the launch's meshes), so max_sweeps = 1 or
// 2 gives one refinement round per step (the next step's first residual
// includes what is left).
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>
#include <thread>
#include <vector>

#include "internal.cuh"

namespace ilg {

namespace {

constexpr int RAD_THREADS = 992;             // consumer threads (31 warps): one entry run each
// Registers per thread: 1,024 threads leave 8,192 of the SM's in the FP64 and
// 16,384 in the mixed solve, one block of 128 or 256 threads of the direct
// insolation that runs beside it (direct.cu k_direct_beside). The FP64 solves
// are long enough to hide the smaller block and lose 8% at 48 registers. At 48
// the one-pass solve's first pass spills 160 bytes per thread (the others
// none).
#define RAD_REGS64 56
#define RAD_REGSM 48
constexpr int RAD_BLOCK = RAD_THREADS + 32;  // and one producer warp that issues the entry-stream copies
constexpr int RAD_HALO = 8192;           // halo values per tile (double-float: 64 KB of shared memory)
constexpr int RAD_ROWS = 3072;           // rows per tile (their sums: 24 KB of shared memory)
constexpr int RAD_MAX_MESH = 1024;
constexpr int RAD_MESH_BYTES = 13;       // shared memory per mesh of the view (MeshState)
constexpr int RAD_INNER = 2;             // most fp32 sweeps per refinement of the mixed solve: the bf16 error
                                         // (~4e-3 of the correction) already dominates rho^(k+1), rho ~ 0.013
constexpr int64_t RAD_SPLIT_MIN = 131072;  // entries: tiles above twice the split target are halved
// Tile balance, in stored entries: a block's sweep time is about
// c + 1.35e-4 us per stored entry + 8.8e-4 us per row + 1.5e-4 us per halo
// facet (per-block timings of the FP64 sweep on GB300, 152 tiles of an
// 81,920-facet mesh), i.e. a row costs ~7 entries and a halo facet ~1.
constexpr int64_t RAD_ROW_COST = 7;
constexpr int64_t RAD_HALO_COST = 1;
constexpr int64_t RAD_GROUP = 4 * RAD_THREADS;  // stored entries per group (4 per thread): a tile's stream is whole groups
// Smallest tile, in entries: one group. A small mesh's sweep is bound by its
// longest tile (each further group ~1 us) and a barrier whose cost does not
// grow from 3 blocks to 94, so it takes as many blocks as it has groups: FP64
// steps of 5,120 facets (45,577 entries) take 57 us in 12 tiles of one group,
// 60 in 6, 70 in 4, 77 in 3 and 96 in 2; of 20,480 facets (728,586) 83 us in
// 94 tiles, 90 in 38, 106 in 21; in mixed precision 34 / 42 and 37 / 39 us.
constexpr int64_t RAD_MIN_TILE = RAD_GROUP;
// One group in shared memory: its columns (u16), then its values (f32 hi, or
// bf16 for the mixed inner sweeps); the f32 lo of double-floats take a stage
// of their own. Every piece is a multiple of 16 bytes, and a group starts at a
// multiple of RAD_GROUP entries, so each is one bulk copy. (Three stages wide
// enough for double-floats left the change sweeps, six of seven, with three
// groups in flight: 605 us instead of 589 for 16 meshes.)
constexpr int RAD_CF_BYTES = (int)RAD_GROUP * 2;
constexpr int RAD_F32_BYTES = (int)RAD_GROUP * 4;
constexpr int RAD_STAGE = RAD_CF_BYTES + RAD_F32_BYTES;
constexpr int RAD_STAGES = 5;
constexpr size_t RAD_RING = (size_t)RAD_STAGES * RAD_STAGE;
static_assert(RAD_CF_BYTES % 16 == 0 && RAD_F32_BYTES % 16 == 0, "bulk copies move multiples of 16 bytes");
constexpr size_t RAD_SMEM = RAD_RING + (size_t)RAD_HALO * sizeof(float2) + RAD_THREADS * sizeof(float2) +
                            RAD_ROWS * sizeof(float2) + RAD_THREADS + 2 * RAD_STAGES * sizeof(unsigned long long);

// Most polls of one grid-barrier wait (an L2 round trip each, ~0.4 us). A device variable so that a test can shrink it (ilg_debug_barrier_
// timeout) and watch a wait run out without a long stall.
constexpr long long BARRIER_POLLS = 1LL << 23;
__device__ long long g_barrier_polls = BARRIER_POLLS;

// Grid barrier for a cooperative launch (all blocks co-resident) on an
// arrival counter that only grows during the launch (zeroed before it):
// every block counts its barriers in gen, and barrier number gen opens once
// the counter reaches gen * nblocks, so the last block to arrive releases
// the others with its own increment (no reset on the critical path). The
// wait is bounded: after g_barrier_polls polls it records DERR_BARRIER and
// returns false (as does every block that sees the flag while waiting).
// The fence before the arrival and the acquiring load (or fence) after it
// make the iterates written before the barrier visible to the loads after it.
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned x;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
  return x;
}
__device__ bool grid_barrier(unsigned* bar, unsigned nblocks, unsigned& gen, int* derr) {
  __shared__ int ok;
  ++gen;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    const unsigned target = gen * nblocks;
    const long long limit = g_barrier_polls;
    __threadfence();
    if (atomicAdd(bar, 1u) + 1u < target) {
      long long it = 0;
      while (ld_acquire(bar) < target) {
        if (++it > limit || ((it & 63) == 0 && *(volatile int*)&derr[DERR_BARRIER])) {
          atomicExch(&derr[DERR_BARRIER], 1);
          ok = 0;
          break;
        }
      }
    } else {
      __threadfence();
    }
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ int mesh_of_facet(const StepView& v, int g) { return v.mesh_of ? v.mesh_of[g] : 0; }

// Matrix loads: read-only for the whole solve, so the non-coherent path, no
// L1 allocation (each entry is used once per sweep), and an L2 evict-last
// policy on 3/4 of the lines so that repeated sweeps find most of the
// matrix in L2 when it is about as large as L2. A matrix much larger than
// L2 is streamed with evict-first instead (nothing of it survives until the
// next pass, and evict-last lines would only crowd out the iterates).
__device__ __forceinline__ uint64_t l2_keep_policy(int stream) {
  uint64_t pol;
  if (stream)
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  else
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 0.75;" : "=l"(pol));
  return pol;
}
// The entry stream of a block's tiles reaches shared memory by 1-D bulk
// copies (cp.async.bulk) into a ring of stages: the producer warp's lane 0
// waits until a stage is free (its empty barrier), announces the bytes on the
// stage's full barrier and issues the copies; consumers wait on the full
// barrier, read their four entries and arrive on the empty barrier. Both
// sides walk the same sequence of (tile, group) pairs from the start of the
// launch, stage by stage, so each wait is on the parity of the stage's use.
// Every wait is bounded: after RAD_MBAR_POLLS polls
// it records DERR_STREAM, and from then on the block's waits return at once
// and its consumers treat the stream as empty (all-zero entries, which index
// no halo value beyond slot 0 and end no row).
constexpr long long RAD_MBAR_POLLS = 1LL << 22;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// true if the use with this parity has completed (the hardware may wait a
// little for it)
__device__ __forceinline__ bool mbar_try(unsigned long long* bar, unsigned parity) {
  unsigned done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return done != 0;
}
// true once the use with this parity has completed; false after the poll
// limit (flagged) or when the block's stream has already failed
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int* bad, int* derr) {
  if (*(volatile int*)bad) return false;
  for (long long it = 0; it < RAD_MBAR_POLLS; ++it) {
    if (mbar_try(bar, parity)) return true;
    if (*(volatile int*)bad) return false;
  }
  *(volatile int*)bad = 1;
  atomicExch(&derr[DERR_STREAM], 1);
  return false;
}
__device__ __forceinline__ void bulk_copy(unsigned dst, const void* src, unsigned bytes, unsigned long long* bar,
                                          uint64_t pol) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol) : "memory");
}

// Value sources of tile_rows: how a group's values are copied into a stage
// (after its columns) and read back, four consecutive entries per thread.
struct ValsDF { const float* hi; const float* lo; };   // double-float (hi, lo)
struct ValsHi { const float* hi; };                    // fl(F) as a double-float with lo = 0
struct ValsBF { const __nv_bfloat16* v; };             // bf16, scaled per row
struct ValsHiF { const float* hi; };                   // fl(F) as a float
__device__ __forceinline__ unsigned vals_bytes(ValsHi) { return RAD_F32_BYTES; }
__device__ __forceinline__ unsigned vals_bytes(ValsHiF) { return RAD_F32_BYTES; }
__device__ __forceinline__ unsigned vals_bytes(ValsBF) { return RAD_CF_BYTES; }
__device__ __forceinline__ void copy_vals(ValsHi s, unsigned dst, size_t e, unsigned long long* bar, uint64_t pol) {
  bulk_copy(dst, s.hi + e, RAD_F32_BYTES, bar, pol);
}
__device__ __forceinline__ void copy_vals(ValsHiF s, unsigned dst, size_t e, unsigned long long* bar, uint64_t pol) {
  bulk_copy(dst, s.hi + e, RAD_F32_BYTES, bar, pol);
}
__device__ __forceinline__ void copy_vals(ValsBF s, unsigned dst, size_t e, unsigned long long* bar, uint64_t pol) {
  bulk_copy(dst, s.v + e, RAD_CF_BYTES, bar, pol);
}
__device__ __forceinline__ void read_vals(ValsHi, const unsigned char* st, int tid, float2 (&w)[4]) {
  const float4 h = *reinterpret_cast<const float4*>(st + 16 * tid);
  w[0] = make_float2(h.x, 0.f);
  w[1] = make_float2(h.y, 0.f);
  w[2] = make_float2(h.z, 0.f);
  w[3] = make_float2(h.w, 0.f);
}
__device__ __forceinline__ void read_vals(ValsHiF, const unsigned char* st, int tid, float (&w)[4]) {
  const float4 h = *reinterpret_cast<const float4*>(st + 16 * tid);
  w[0] = h.x;
  w[1] = h.y;
  w[2] = h.z;
  w[3] = h.w;
}
__device__ __forceinline__ void read_vals(ValsBF, const unsigned char* st, int tid, float (&w)[4]) {
  const uint2 r = *reinterpret_cast<const uint2*>(st + 8 * tid);
  w[0] = __uint_as_float(r.x << 16);
  w[1] = __uint_as_float(r.x & 0xffff0000u);
  w[2] = __uint_as_float(r.y << 16);
  w[3] = __uint_as_float(r.y & 0xffff0000u);
}
template <class W> __device__ __forceinline__ void zero_vals(W (&w)[4]);
template <> __device__ __forceinline__ void zero_vals(float2 (&w)[4]) {
  for (int j = 0; j < 4; ++j) w[j] = make_float2(0.f, 0.f);
}
template <> __device__ __forceinline__ void zero_vals(float (&w)[4]) {
  for (int j = 0; j < 4; ++j) w[j] = 0.f;
}

// The block's stream ring and its position in it (per thread; every
// consumer and the producer lane advance it identically): the stage, and the
// parity of its current use.
struct Pipe {
  unsigned char* ring;
  unsigned long long* full;
  unsigned long long* empty;
  int* bad;
  int s;
  unsigned parity;
  __device__ __forceinline__ void advance() {
    if (++s == RAD_STAGES) {
      s = 0;
      parity ^= 1u;
    }
  }
};

// Producer (lane 0 of the producer warp): the copies of every group of tile
// T. A stage is free once its previous use has been read; the wait on a
// stage's first use passes at once (the phase before an mbarrier's first
// counts as completed).
template <class V>
__device__ __forceinline__ void produce_tile(Pipe& p, const StepView& v, const RowTile& T, V vals, uint64_t pol) {
  const int ng = T.lam >> 2;
  const unsigned bytes = (unsigned)RAD_CF_BYTES + vals_bytes(vals);
  for (int g = 0; g < ng; ++g, p.advance()) {
    if (!mbar_wait(p.empty + p.s, p.parity ^ 1u, p.bad, v.derr)) continue;
    if (*(volatile int*)p.bad) continue;
    const unsigned dst = smem_u32(p.ring + (size_t)p.s * RAD_STAGE);
    const size_t e = (size_t)T.e0 + (size_t)g * RAD_GROUP;
    mbar_expect(p.full + p.s, bytes);
    bulk_copy(dst, v.t_cf + e, RAD_CF_BYTES, p.full + p.s, pol);
    copy_vals(vals, dst + RAD_CF_BYTES, e, p.full + p.s, pol);
  }
}
// Double-floats take two stages per group, the low parts in the second.
__device__ __forceinline__ void produce_tile(Pipe& p, const StepView& v, const RowTile& T, ValsDF vals, uint64_t pol) {
  const int ng = T.lam >> 2;
  for (int q = 0; q < 2 * ng; ++q, p.advance()) {
    if (!mbar_wait(p.empty + p.s, p.parity ^ 1u, p.bad, v.derr)) continue;
    if (*(volatile int*)p.bad) continue;
    const unsigned dst = smem_u32(p.ring + (size_t)p.s * RAD_STAGE);
    const size_t e = (size_t)T.e0 + (size_t)(q >> 1) * RAD_GROUP;
    if (q & 1) {
      mbar_expect(p.full + p.s, RAD_F32_BYTES);
      bulk_copy(dst, vals.lo + e, RAD_F32_BYTES, p.full + p.s, pol);
    } else {
      mbar_expect(p.full + p.s, RAD_CF_BYTES + RAD_F32_BYTES);
      bulk_copy(dst, v.t_cf + e, RAD_CF_BYTES, p.full + p.s, pol);
      bulk_copy(dst + RAD_CF_BYTES, vals.hi + e, RAD_F32_BYTES, p.full + p.s, pol);
    }
  }
}

// Consumer: the next group's four entries of this thread (columns and
// values), then the stage is released (one arrival per warp).
template <class V, class W>
__device__ __forceinline__ void take_group(Pipe& p, const StepView& v, V vals, uint2& c, W (&w)[4]) {
  const unsigned char* st = p.ring + p.s * RAD_STAGE;
  if (mbar_try(p.full + p.s, p.parity) || mbar_wait(p.full + p.s, p.parity, p.bad, v.derr)) {
    c = *reinterpret_cast<const uint2*>(st + 8 * threadIdx.x);
    read_vals(vals, st + RAD_CF_BYTES, threadIdx.x, w);
  } else {
    c = make_uint2(0u, 0u);
    zero_vals(w);
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(p.empty + p.s);
  p.advance();
}

__device__ __forceinline__ void take_group(Pipe& p, const StepView& v, ValsDF vals, uint2& c, float2 (&w)[4]) {
  float h[4], l[4];
  take_group(p, v, ValsHiF{vals.hi}, c, h);
  const float* st = reinterpret_cast<const float*>(p.ring + p.s * RAD_STAGE);
  if (mbar_try(p.full + p.s, p.parity) || mbar_wait(p.full + p.s, p.parity, p.bad, v.derr)) {
    const float4 q = *reinterpret_cast<const float4*>(st + 4 * threadIdx.x);
    l[0] = q.x;
    l[1] = q.y;
    l[2] = q.z;
    l[3] = q.w;
  } else {
    zero_vals(l);
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(p.empty + p.s);
  p.advance();
  for (int j = 0; j < 4; ++j) w[j] = make_float2(h[j], l[j]);
}

// Barrier of the consumer threads only (the producer warp does not take
// part in the tile work).
__device__ __forceinline__ void cbar() { asm volatile("bar.sync 1, %0;" ::"n"(RAD_THREADS) : "memory"); }

__device__ __forceinline__ double warp_sum(double x) {
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Double-float: v = hi + lo with hi = fl(v), lo = fl(v - hi).
__device__ __forceinline__ float2 split_df(double x) {
  float h = __double2float_rn(x);
  return make_float2(h, __double2float_rn(x - (double)h));
}

// Running sum of double-float products. add(): p + e = w.hi * x.hi exactly
// (FMA), plus the cross terms w.hi * x.lo + w.lo * x.hi in e; (h, l) += p
// by TwoSum, l += e. Intrinsics keep the compiler from contracting or
// reassociating the error-free steps.
struct AccDF {
  static constexpr bool CHEAP = false;
  typedef float2 W;
  typedef float2 X;
  typedef float2 Part;
  typedef float2 Sum;
  float h, l;
  __device__ __forceinline__ void zero() { h = 0.f; l = 0.f; }
  __device__ __forceinline__ void two_sum(float p) {
    float t = __fadd_rn(h, p);
    float bp = __fsub_rn(t, h);
    float err = __fadd_rn(__fsub_rn(h, __fsub_rn(t, bp)), __fsub_rn(p, bp));
    h = t;
    l = __fadd_rn(l, err);
  }
  __device__ __forceinline__ void add(float2 w, float2 x) {
    float p = __fmul_rn(w.x, x.x);
    float e = __fmaf_rn(w.x, x.x, -p);
    e = __fmaf_rn(w.x, x.y, e);
    e = __fmaf_rn(w.y, x.x, e);
    two_sum(p);
    l = __fadd_rn(l, e);
  }
  __device__ __forceinline__ Part part() const { return make_float2(h, l); }
  __device__ __forceinline__ void merge(Part q) {
    two_sum(q.x);
    l = __fadd_rn(l, q.y);
  }
  __device__ __forceinline__ float2 get() const { return make_float2(h, l); }
};

__device__ __forceinline__ double df_value(float2 s) { return (double)s.x + (double)s.y; }

// Double-float sum a + b (TwoSum of the high parts, then renormalised),
// FP32 operations only.
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
  float s = __fadd_rn(a.x, b.x);
  float bb = __fsub_rn(s, a.x);
  float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb));
  e = __fadd_rn(e, __fadd_rn(a.y, b.y));
  float t = __fadd_rn(s, e);
  return make_float2(t, __fsub_rn(e, __fsub_rn(t, s)));
}

__device__ __forceinline__ float2 df_neg(float2 a) { return make_float2(-a.x, -a.y); }

// Plain fp32 sum (mixed inner sweeps: bf16 values, fp32 iterates).
struct AccF32 {
  static constexpr bool CHEAP = true;
  typedef float W;
  typedef float X;
  typedef float Part;
  typedef float Sum;
  float s;
  __device__ __forceinline__ void zero() { s = 0.f; }
  __device__ __forceinline__ void add(float w, float x) { s = fmaf(w, x, s); }
  __device__ __forceinline__ Part part() const { return s; }
  __device__ __forceinline__ void merge(Part q) { s += q; }
  __device__ __forceinline__ float get() const { return s; }
};

// Two fp32 sums over the same entries (the one-pass mixed solve: the
// iterate's change and the next frame's change of the direct flux).
struct AccF2 {
  static constexpr bool CHEAP = true;
  typedef float W;
  typedef float2 X;
  typedef float2 Part;
  typedef float2 Sum;
  float a, b;
  __device__ __forceinline__ void zero() { a = 0.f; b = 0.f; }
  __device__ __forceinline__ void add(float w, float2 x) {
    a = fmaf(w, x.x, a);
    b = fmaf(w, x.y, b);
  }
  __device__ __forceinline__ Part part() const { return make_float2(a, b); }
  __device__ __forceinline__ void merge(Part q) {
    a += q.x;
    b += q.y;
  }
  __device__ __forceinline__ float2 get() const { return make_float2(a, b); }
};

__device__ __forceinline__ float2 to_halo(float2 x, float2*) { return x; }
__device__ __forceinline__ float to_halo(float x, float*) { return x; }

// Iterates written by other blocks during the solve are read at L2 (never
// from a possibly stale L1 line).
__device__ __forceinline__ double ld_it(const double* p) { return __ldcg(p); }
__device__ __forceinline__ float ld_it(const float* p) { return __ldcg(p); }
__device__ __forceinline__ float2 ld_it(const float2* p) { return __ldcg(p); }

// Gather the tile's halo values x[halo[h]] into shared memory.
template <class XS, class XG>
__device__ __forceinline__ void stage_halo(const StepView& v, const RowTile& T, const XG* xg, XS* sx) {
  const uint32_t* hp = v.t_halo + T.h0;
  int h = threadIdx.x;
  for (; h + 3 * RAD_THREADS < T.nhalo; h += 4 * RAD_THREADS) {
    uint32_t a = __ldg(hp + h), b = __ldg(hp + h + RAD_THREADS), c = __ldg(hp + h + 2 * RAD_THREADS),
             d = __ldg(hp + h + 3 * RAD_THREADS);
    XG xa = ld_it(xg + a), xb = ld_it(xg + b), xc = ld_it(xg + c), xd = ld_it(xg + d);
    sx[h] = to_halo(xa, sx);
    sx[h + RAD_THREADS] = to_halo(xb, sx);
    sx[h + 2 * RAD_THREADS] = to_halo(xc, sx);
    sx[h + 3 * RAD_THREADS] = to_halo(xd, sx);
  }
  for (; h < T.nhalo; h += RAD_THREADS) sx[h] = to_halo(ld_it(xg + __ldg(hp + h)), sx);
  cbar();
}

// As stage_halo, x = eh + s formed from its two parts.
__device__ __forceinline__ void stage_halo_sum(const StepView& v, const RowTile& T, const float2* eh, const float2* s,
                                               float2* sx) {
  const uint32_t* hp = v.t_halo + T.h0;
  int h = threadIdx.x;
  for (; h + RAD_THREADS < T.nhalo; h += 2 * RAD_THREADS) {
    const uint32_t a = __ldg(hp + h), b = __ldg(hp + h + RAD_THREADS);
    const float2 ea = ld_it(eh + a), eb = ld_it(eh + b), sa = ld_it(s + a), sb = ld_it(s + b);
    sx[h] = df_add(ea, sa);
    sx[h + RAD_THREADS] = df_add(eb, sb);
  }
  if (h < T.nhalo) {
    const uint32_t a = __ldg(hp + h);
    sx[h] = df_add(ld_it(eh + a), ld_it(s + a));
  }
  cbar();
}

// The thread's first row in tile t (t_start), loaded ahead of its use.
__device__ __forceinline__ uint32_t tile_start(const StepView& v, int t) {
  return __ldg(v.t_start + (size_t)t * RAD_THREADS + threadIdx.x);
}

// Column codes: a pair of entries in 32 bits, the first one's halo index in
// bits 0-12, the second one's in bits 16-28, and the row-end bits of both
// beside the first, so that an index takes one operation.
constexpr unsigned CF_INDEX = 0x1fffu, CF_END0 = 0x8000u, CF_END1 = 0x4000u;

// One tile (s0: tile_start): thread t owns entries [t*lam, (t+1)*lam) of the tile's entry
// stream (rows in order, each row's entries in column order), stored so that
// a group of 4 RAD_THREADS entries is contiguous: entry k of thread t at
// e0 + (k/4)*RAD_GROUP + 4t + k%4. The groups arrive in shared memory by
// bulk copies (the block's Pipe). Each thread accumulates sequentially and
// stores the sum of every row that starts and ends in its run in rs[row]
// (shared memory). A row that began in an earlier thread is completed by the
// thread where it ends: the partial sums of the threads it spans, in thread
// order, then its own part. Ends with a consumer barrier: rs holds every
// row sum of the tile.
template <class Acc, class V>
__device__ __forceinline__ void tile_rows(const StepView& v, const RowTile& T, uint32_t s0, Pipe& p, V vals,
                                          const typename Acc::X* sx, typename Acc::Part* tail, unsigned char* tnew,
                                          typename Acc::Sum* rs) {
  typedef typename Acc::W W;
  const int tid = threadIdx.x;
  const int r = (int)(s0 & 0x7fffffffu);
  const bool cont = (s0 >> 31) != 0;
  // where the open row's sum goes when the row ends: rs, or for a row that
  // began in an earlier thread the thread's own tail slot (read back below)
  typename Acc::Sum* const first = cont ? tail + tid : rs + r;
  typename Acc::Sum *dst = first, *next = rs + r + 1;
  Acc acc;
  acc.zero();
  const int ng = T.lam >> 2;
  auto end = [&]() {   // the row's last entry
    *dst = acc.get();
    dst = next;
    ++next;
    acc.zero();
  };
  for (int g = 0; g < ng; ++g) {
    uint2 c;
    W w[4];
    take_group(p, v, vals, c, w);
    const typename Acc::X x0 = sx[c.x & CF_INDEX], x1 = sx[c.x >> 16], x2 = sx[c.y & CF_INDEX], x3 = sx[c.y >> 16];
    if (Acc::CHEAP && ((c.x | c.y) & (CF_END0 | CF_END1)) == 0) {
      acc.add(w[0], x0);
      acc.add(w[1], x1);
      acc.add(w[2], x2);
      acc.add(w[3], x3);
    } else {
      acc.add(w[0], x0);
      if (c.x & CF_END0) end();
      acc.add(w[1], x1);
      if (c.x & CF_END1) end();
      acc.add(w[2], x2);
      if (c.y & CF_END0) end();
      acc.add(w[3], x3);
      if (c.y & CF_END1) end();
    }
  }
  const bool any = dst != first, has_head = cont && any;
  Acc head;
  head.zero();
  if (has_head) head.merge(tail[tid]);
  tail[tid] = acc.part();
  tnew[tid] = (any || !cont) ? 1 : 0;
  cbar();
  if (has_head) {
    int u = tid - 1;
    while (!tnew[u]) --u;   // thread 0 starts a row, so this stops
    Acc s;
    s.zero();
    for (; u < tid; ++u) s.merge(tail[u]);
    s.merge(head.part());
    rs[r] = s.get();
  }
  cbar();
}

// Sum over the consumer threads in a fixed order (FP32), valid in thread 0.
// Ends with a consumer barrier (the tile's shared arrays are free again).
__device__ __forceinline__ float warp_sumf(float x) {
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ float block_sum(float d, float* red) {
  d = warp_sumf(d);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = d;
  cbar();
  float t = 0.f;
  if (threadIdx.x < 32) t = warp_sumf(threadIdx.x < RAD_THREADS / 32 ? red[threadIdx.x] : 0.f);
  cbar();
  return t;
}

// Per-mesh convergence. Each tile's squared change (FP32 partial) is
// recorded in tile_d2 (double-buffered by sweep parity) and added, as an
// integer, to its mesh's accumulator: the partial in units of tol^2 / 2^20,
// rounded up and capped at 2^40 (a NaN counts as the cap). Integer sums do
// not depend on the order of the atomic adds, so every block reads the same
// total after the grid barrier and takes the same decision with one load,
// and a mesh's decisions are the same alone and in a batch. A mesh stops
// when its total is <= 2^20 units, i.e. sum of partials <= tol^2 (at most
// ntiles units conservative). The accumulators lie in the barrier's buffer,
// three buffers of RES_LEVELS x nmesh by residual number
// mod 3: buffer k + 1 is cleared during residual k (its last reader,
// decision k - 2, finished before the barrier that precedes residual k), and
// the accumulators of residual 0 are cleared before the first barrier. The
// FP64 solve also needs totals far above the cap (it tracks how much the
// change has shrunk): it counts a partial of more than 2^40 units in units
// of 2^40 (level 1) or 2^80 (level 2), the mixed solves use level 0 only.
constexpr unsigned long long RES_UNITS = 1ull << 20;
constexpr unsigned long long RES_CAP = 1ull << 40;
constexpr int RES_LEVELS = 3;

// Words of the barrier buffer before the solo solve's sweep words (grid <=
// RAD_MAX_GRID blocks, 2 x 16 bytes each), and before the accumulators.
constexpr int RAD_MAX_GRID = 1024;
constexpr int RAD_BAR_WORDS0 = 4;
constexpr int RAD_BAR_WORDS1 = RAD_BAR_WORDS0 + RAD_MAX_GRID * 8;
__device__ __forceinline__ unsigned long long* res_acc(const StepView& v, int k, int level = 0) {
  return reinterpret_cast<unsigned long long*>(v.barrier + RAD_BAR_WORDS1) + (size_t)((k % 3) * RES_LEVELS + level) * v.nmesh;
}

// done[m]: 0 running; 1 + (parity of the mesh's last residual) once
// stopped; 1 for meshes that never ran. unit[m]: residual units per unit of
// squared change, 2^20 / tol^2 enlarged by 2^-16 so that the FP32 products
// below never round a partial's units down (+inf when tol is 0).
// The arrays follow the tile buffers in dynamic shared memory, sized for the
// view's meshes (a kernel beside this one needs what they leave).
struct MeshState {
  int* done;
  int* sweeps;
  float* unit;
  unsigned char* now;   // stopped at the latest decision
  __device__ __forceinline__ explicit MeshState(int nmesh);
};

__device__ __forceinline__ unsigned long long res_units(float d2, float unit) {
  if (isnan(d2)) return RES_CAP;
  if (!(d2 > 0.f)) return 0ull;
  const float q = __fmul_ru(d2, unit);
  return q < (float)RES_CAP ? (unsigned long long)ceilf(q) : RES_CAP;
}

// Thread 0, after block_sum: record tile t's partial of residual k.
__device__ __forceinline__ void post_partial(const StepView& v, const MeshState& st, const RowTile& T, int t, int k,
                                             float d2) {
  if (threadIdx.x != 0) return;
  v.tile_d2[(size_t)(k & 1) * v.ntiles + t] = (double)d2;
  atomicAdd(res_acc(v, k) + T.mesh, res_units(d2, st.unit[T.mesh]));
  res_acc(v, k + 1)[T.mesh] = 0ull;
}

__device__ __forceinline__ void init_meshes(const StepView& v, MeshState& st) {
  for (int m = threadIdx.x; m < v.nmesh; m += blockDim.x) {
    const MeshDesc& M = v.md[m];
    st.done[m] = (M.active && M.ntiles > 0) ? 0 : 1;
    st.sweeps[m] = 0;
    st.unit[m] = M.tol2 > 0.0 ? (float)((double)RES_UNITS / M.tol2 * (1.0 + 1.0 / 65536.0)) : INFINITY;
  }
  // accumulators of residual 0 (read only after the first barrier)
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  for (int m = gt; m < v.nmesh; m += gridDim.x * blockDim.x) res_acc(v, 0)[m] = 0ull;
}

// Every block, after the barrier that completes residual k: stop decisions
// and the number of meshes still running. Block 0 records the sweep counts.
__device__ __forceinline__ int decide_meshes(const StepView& v, MeshState& st, int inc, int first, int k) {
  __syncthreads();
  const unsigned long long* acc = res_acc(v, k);
  for (int m = threadIdx.x; m < v.nmesh; m += blockDim.x) {
    st.now[m] = 0;
    if (st.done[m]) continue;
    const unsigned long long q = __ldcg(acc + m);
    const int sw = st.sweeps[m] + (first ? 0 : inc);
    st.sweeps[m] = sw;
    if (q <= RES_UNITS || sw >= v.md[m].max_sweeps) {
      st.done[m] = 1 + (k & 1);
      st.now[m] = 1;
    }
    if (blockIdx.x == 0) v.md[m].sweeps = sw;
  }
  int running = 0;
  for (int m0 = 0; m0 < v.nmesh; m0 += blockDim.x) {
    int m = m0 + threadIdx.x;
    running += __syncthreads_count(m < v.nmesh && !st.done[m]);
  }
  return running;
}

// Block 0, at the end of the launch: each solved mesh's last residual
// (sum of its tiles' partials, lane-strided then a fixed warp tree) into
// the mesh table.
__device__ __forceinline__ void record_residuals(const StepView& v, const MeshState& st) {
  if (blockIdx.x != 0 || threadIdx.x >= RAD_THREADS) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m = warp; m < v.nmesh; m += RAD_THREADS / 32) {
    const MeshDesc& M = v.md[m];
    if (!M.active || M.ntiles == 0) continue;
    const double* d2 = v.tile_d2 + (size_t)(st.done[m] - 1) * v.ntiles;
    double t = 0.0;
    for (int j = lane; j < M.ntiles; j += 32) t += ld_it(d2 + M.tile0 + j);
    t = warp_sum(t);
    if (lane == 0) v.md[m].res2 = t;
  }
}

// ---- the FP64 solve's sweeps ----
//
// A sweep evaluates s' = F x for x = E + s. Written as a change, with
// d = s - (the previous s), the same sweep is d' = F d, s' = s + d': the
// iterates are Jacobi's either way. A full sweep evaluates F x in
// double-float (10 B per entry, ~20 FP32 operations, 8 B halos); a change
// sweep evaluates F d in FP32 with the high parts of the values (6 B, one
// FMA, 4 B halos) and adds it to the double-float s. What FP32 loses stays in
// s: at most c |d| per sweep, c = n 2^-24 || |F| ||_2 with n the longest chain
// of additions to a row's sum (radiosity_prepare bounds both), so at most
// c A in all, A = the sum of |d| over the change sweeps since the last full
// one. So the solve begins with a full sweep, continues with change sweeps,
// and stops when the residual is known to be small enough; a full sweep,
// which recomputes s from x and so removes the errors, comes in between where
// they would be too large for that:
//   a solve stops after a full sweep with |d| <= tol, or after a change sweep
//   with |d| + c A <= tol (which it reports as its residual);
//   a full sweep follows when the errors may have reached the change, |d| <=
//   4 c A; when c A > tol but a full sweep now would leave a sixteenth of tol
//   at the rate of the last two sweeps; when |d| is small enough or expected
//   to be after the next sweep (|d|^2 <= tol |d before|, at first |d| <= 8
//   tol) and c A > tol / 2; and when |d| <= tol did not stop the solve;
//   another change sweep follows otherwise.
// The bound holds for any matrix, also one whose rounding errors all have the
// same sign in every sweep. (Taken as 2^-23 A, whatever the row lengths: rows
// of 8,000 equal entries were left with residuals above tol.)
// The last sweep of a budget is a full one, so that a solve which reaches tol
// within its budget by full sweeps alone still does. |d| comes from the
// integer residual totals, so the choice is the same in every block, on every
// run, and alone or in a batch. A tolerance of zero (or one whose units
// overflow) runs full sweeps only.
struct MeshState64 {
  int* sweeps;
  float* acc;             // A in units of tol, with the last |d|
  float* prev;            // the last |d| in units of tol
  unsigned char* mode;    // bit 0: the next sweep is a change sweep; bit 1: s is in S1; from bit 2: as MeshState::done
  __device__ __forceinline__ explicit MeshState64(int nmesh);
};
constexpr int MODE_DONE = 2;   // shift of the done bits
constexpr float CHG_RANGE = 5.6294995e14f;   // 2^49: above it the totals are at their cap

// A partial in residual units, and the level they are counted at.
__device__ __forceinline__ unsigned long long res_units64(float d2, float unit, int& level) {
  level = 2;
  if (isnan(d2)) return RES_CAP;
  const float q = d2 > 0.f ? __fmul_ru(d2, unit) : 0.f;
  const float cap = (float)RES_CAP;   // 2^40, exact
  if (q < cap) {
    level = 0;
    return (unsigned long long)ceilf(q);
  }
  if (q < cap * cap) {
    level = 1;
    return (unsigned long long)ceilf(q * (1.f / cap));
  }
  const float q2 = q * (1.f / cap) * (1.f / cap);
  return q2 < cap ? (unsigned long long)ceilf(q2) : RES_CAP;
}

// Thread 0, after block_sum: record tile t's partial of residual k.
__device__ __forceinline__ void post_partial64(const StepView& v, const RowTile& T, int t, int k, float unit,
                                               float d2) {
  if (threadIdx.x != 0) return;
  v.tile_d2[(size_t)(k & 1) * v.ntiles + t] = (double)d2;
  int level;
  const unsigned long long u = res_units64(d2, unit, level);
  if (u) atomicAdd(res_acc(v, k, level) + T.mesh, u);
  for (int l = 0; l < RES_LEVELS; ++l) res_acc(v, k + 1, l)[T.mesh] = 0ull;
}

// What follows a sweep (see above), from its totals, the errors' factor c and
// A and |d| before it (zero before the first).
struct Sweep64 {
  bool stop, next_change;
  float dn, acc, err;   // |d|, A, and the errors in the result, in units of tol
};
__device__ __forceinline__ Sweep64 sweep_decision(unsigned long long q0, unsigned long long q1, unsigned long long q2,
                                                  bool change, float c, float acc, float prev) {
  const float cap = (float)RES_CAP;
  Sweep64 r;
  r.dn = sqrtf((float)q0 + cap * ((float)q1 + cap * (float)q2)) * (1.f / 1024.f);
  r.err = change ? c * acc : 0.f;
  r.acc = change ? acc + r.dn : r.dn;
  r.stop = change ? r.dn + r.err <= 1023.f / 1024.f : ((q1 | q2) == 0) & (q0 <= RES_UNITS);
  const float e = c * r.acc;   // the errors after another change sweep
  const bool last = (r.dn <= 1.f) | ((e > 0.5f) & (r.dn * r.dn <= (prev > 0.f ? prev : 8.f * r.dn)));
  const bool renew = (e > 1.f) & (r.dn * (16.f * c * prev) <= prev - r.dn);
  r.next_change = !last & !renew & (r.dn > 4.f * e) & (r.dn < CHG_RANGE);
  return r;
}

__device__ __forceinline__ void init_meshes64(const StepView& v, MeshState64& st) {
  for (int m = threadIdx.x; m < v.nmesh; m += blockDim.x) {
    const MeshDesc& M = v.md[m];
    st.mode[m] = (M.active && M.ntiles > 0) ? 0 : 1 << MODE_DONE;
    st.sweeps[m] = 0;
    st.acc[m] = st.prev[m] = 0.f;
    if (blockIdx.x == 0) v.md[m].full_sweeps = 0;
  }
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  for (int m = gt; m < RES_LEVELS * v.nmesh; m += gridDim.x * blockDim.x) res_acc(v, 0)[m] = 0ull;
}

// Every block, after the barrier that completes sweep k: stop decisions,
// the kind of the next sweep, and the number of meshes still running.
__device__ __forceinline__ int decide_meshes64(const StepView& v, MeshState64& st, int k) {
  int running = 0;
  for (int m0 = 0; m0 < v.nmesh; m0 += blockDim.x) {
    const int m = m0 + threadIdx.x;
    bool run = m < v.nmesh && !(st.mode[m] >> MODE_DONE);
    if (run) {
      // every load before the first store (one trip to L2 instead of three)
      const unsigned long long q0 = __ldcg(res_acc(v, k, 0) + m), q1 = __ldcg(res_acc(v, k, 1) + m),
                               q2 = __ldcg(res_acc(v, k, 2) + m);
      const float c = v.md[m].rad_err;
      const int budget = v.md[m].max_sweeps;
      const bool change = st.mode[m] & 1;
      const Sweep64 dec = sweep_decision(q0, q1, q2, change, c, st.acc[m], st.prev[m]);
      const int sw = ++st.sweeps[m];
      const int in_s1 = change ? st.mode[m] & 2 : (st.mode[m] & 2) ^ 2;
      st.mode[m] = in_s1 | (dec.next_change && sw + 1 < budget ? 1 : 0);
      st.acc[m] = dec.acc;
      st.prev[m] = dec.dn;
      if (dec.stop || sw >= budget) {
        st.mode[m] |= (1 + (k & 1)) << MODE_DONE;
        run = false;
        st.acc[m] = dec.err;   // for record_residuals64
      }
      if (blockIdx.x == 0) {
        v.md[m].sweeps = sw;
        if (!change) atomicAdd(&v.md[m].full_sweeps, 1);   // (nothing waits for it)
      }
    }
    running += __syncthreads_count(run);
  }
  return running;
}

// Squared residual plus the bound on the change sweeps' errors.
__device__ __forceinline__ double with_errors(double r2, float err, double tol2) {
  if (!(err > 0.f)) return r2;
  const double r = sqrt(r2) + (double)err * sqrt(tol2);
  return r * r;
}

// Block 0, at the end of the launch: each solved mesh's last residual into
// the mesh table: the root of the sum of its tiles' partials (lane-strided
// then a fixed warp tree), plus the bound on the change sweeps' errors.
__device__ __forceinline__ void record_residuals64(const StepView& v, const MeshState64& st) {
  if (blockIdx.x != 0 || threadIdx.x >= RAD_THREADS) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m = warp; m < v.nmesh; m += RAD_THREADS / 32) {
    const MeshDesc& M = v.md[m];
    if (!M.active || M.ntiles == 0) continue;
    const double* d2 = v.tile_d2 + (size_t)((st.mode[m] >> MODE_DONE) - 1) * v.ntiles;
    double t = 0.0;
    for (int j = lane; j < M.ntiles; j += 32) t += ld_it(d2 + M.tile0 + j);
    t = warp_sum(t);
    if (lane == 0) v.md[m].res2 = with_errors(t, st.acc[m], M.tol2);
  }
}

// The solve works on radiosity positions (Morton order within each mesh),
// gathered through rperm at entry: EP = E (FP64), S0 / S1 = the iterates'
// scattered parts s = x - E (double-floats), H0 / H1 = the iterates
// x = E + s as double-floats (what the halos gather) and EH = E as a
// double-float. Start values: rows without entries are x = E exactly
// (s = 0); the others start at s = 0 (cold) or at the mesh's previous
// solution, extrapolated linearly once two solutions exist (warm). The warm
// start predicts the scattered part and takes the step's own E:
// s0 = S(n) + (S(n) - S(n-1)). E jumps where a facet enters or leaves
// shadow; S = F x varies smoothly, so the start is off by about F dE there
// instead of dE. sprev holds S(n) and, after it, its last change; for the
// one-pass mixed solve (predicted) the predicted change F (E(n+1) - E(n))
// instead, so that s0 = S(n) + P from the second step on.
// The FP64 solve keeps s in S0 or S1 (a full sweep writes the other one, a
// change sweep adds in place) and its last change d, as floats by sweep
// parity, in D0 / D1 (H0's memory); a full sweep's halos form x = EH + s.
struct RadBufs {
  double* EP;
  float2 *S0, *S1, *H0, *H1, *EH;
  float *D0, *D1;
  __device__ __forceinline__ explicit RadBufs(const StepView& v) {
    EP = v.rbuf;
    S0 = reinterpret_cast<float2*>(v.rbuf + v.nt);
    S1 = reinterpret_cast<float2*>(v.rbuf + 2 * (size_t)v.nt);
    H0 = reinterpret_cast<float2*>(v.rbuf + 3 * (size_t)v.nt);
    H1 = H0 + v.nt;
    EH = H1 + v.nt;
    D0 = reinterpret_cast<float*>(H0);
    D1 = D0 + v.nt;
  }
};

// The solve's own per-row state is kept by radiosity position p (Morton
// order): the warm-start record sprev, row_act, and the mesh of a position
// (a mesh's positions and facets occupy the same range, so mesh_of serves
// both). Only E (read) and x (written) are in facet order: one gather and
// one scatter through rperm per row and solve. Each thread takes
// RAD_ILP positions at once so that their loads are in flight together.
constexpr int RAD_ILP = 4;

// free_rows (the mixed solve): also write the result of the rows without
// entries (x = E, s = 0) and their warm-start record, for a kernel that
// scatters its tile rows itself; that solve reads only EP, S0 and H0 (and
// x32), the FP64 sweeps EP, S0, S1, EH and the rows' changes D0 / D1, which
// stay zero for rows without entries.
// kind (the one-pass mixed solve, per mesh: 0 bf16 step, 1 reference step, 2
// first reference step): the warm start is S(n) + P, and the pass's halo
// vector EH = (x - x_ref, E(n+1) - E(n)) and the reference iterate H1 are
// written here too; x32 then holds only P (zero for rows without entries).
__device__ __forceinline__ void init_x(const StepView& v, double* x, int warm, int gt, int nthreads,
                                       bool free_rows, const unsigned char* kind = nullptr) {
  const RadBufs B(v);
  const bool predicted = kind != nullptr;
  for (int p0 = gt; p0 < v.nt; p0 += RAD_ILP * nthreads) {
    int g[RAD_ILP], mi[RAD_ILP];   // facet and mesh of each position (mesh -1: none)
    double d[RAD_ILP];
    float2 sp0[RAD_ILP], sp1[RAD_ILP];
    float de[RAD_ILP];
    uint8_t act[RAD_ILP];
#pragma unroll
    for (int k = 0; k < RAD_ILP; ++k) {
      const int p = p0 + k * nthreads;
      g[k] = 0;
      mi[k] = -1;
      if (p >= v.nt) continue;
      const int mk = mesh_of_facet(v, p);
      const MeshDesc* m = v.md + mk;
      if (!m->active || m->ntiles == 0) continue;
      mi[k] = mk;
      g[k] = (int)v.rperm[p];
      act[k] = v.row_act[p];
      sp0[k] = warm ? v.sprev[p] : make_float2(0.f, 0.f);
      sp1[k] = warm ? v.sprev[v.nt + p] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < RAD_ILP; ++k) {
      if (mi[k] < 0) continue;
      const MeshDesc& Mk = v.md[mi[k]];
      const double dk = v.E[e_slot(Mk.frame) * v.nt + g[k]];
      const bool ref = Mk.coupling == ILG_COUPLE_REFERENCE;
      const double fs = ref ? v.Fsurf[g[k]] : 0.0;
      // the change of the direct flux to the next frame (none after the
      // table's last sun)
      if (predicted)
        de[k] = (!Mk.host_sun && Mk.sun_idx + 1 < Mk.nsun)
                    ? (float)(v.E[e_slot(Mk.frame + 1) * v.nt + g[k]] - dk)
                    : 0.f;
      // the frame's direct flux, coupled as src/cpp/illum_cli.cpp:415-421
      // when the mesh follows the reference (rad = -Fsurf_prev + direct)
      d[k] = ref ? (-fs + dk) : dk;
    }
#pragma unroll
    for (int k = 0; k < RAD_ILP; ++k) {
      if (mi[k] < 0) continue;
      const int p = p0 + k * nthreads;
      const MeshDesc& Mk = v.md[mi[k]];
      const double e = d[k];
      float2 s0 = make_float2(0.f, 0.f);
      if (warm && act[k] && Mk.frame >= 1) s0 = Mk.frame >= 2 || predicted ? df_add(sp0[k], sp1[k]) : sp0[k];
      if (free_rows && !act[k]) {
        x[g[k]] = e;
        if (warm) {
          v.sprev[v.nt + p] = df_neg(sp0[k]);
          v.sprev[p] = make_float2(0.f, 0.f);
        }
      }
      const float2 eh = split_df(e);
      const float2 x0 = df_add(eh, s0);
      B.EP[p] = e;
      B.S0[p] = s0;
      if (free_rows) B.H0[p] = x0;
      if (predicted) {
        // x - x_ref, high parts first (exact when within a factor of 2)
        const int kd = kind[mi[k]];
        float dx;
        if (kd == 2) {
          dx = __fadd_rn(x0.x, x0.y);
        } else {
          const float2 xr = B.H1[p];
          dx = __fadd_rn(__fsub_rn(x0.x, xr.x), __fsub_rn(x0.y, xr.y));
        }
        if (kd) B.H1[p] = x0;
        B.EH[p] = make_float2(dx, de[k]);
        if (!act[k]) v.x32[v.nt + p] = 0.f;
      } else if (free_rows) {
        v.x32[p] = 0.f;
        v.x32[v.nt + p] = 0.f;
      } else {
        B.EH[p] = eh;
        if (!act[k]) {
          B.S1[p] = make_float2(0.f, 0.f);
          B.D0[p] = 0.f;
          B.D1[p] = 0.f;
        }
      }
    }
  }
}

// Scatter the solved meshes' last iterate x = E + s back to facet order
// (FP64); warm solves also record s and its change for the next step's start.
// Rows without entries keep s = 0 in both buffers. src(p): the buffer of
// position p's s, or nullptr where its mesh was not solved.
template <class Src>
__device__ __forceinline__ void scatter_from(const StepView& v, Src src, double* x, int warm, int gt, int nthreads) {
  const RadBufs B(v);
  for (int p0 = gt; p0 < v.nt; p0 += RAD_ILP * nthreads) {
    int g[RAD_ILP];
    bool ok[RAD_ILP];
    double e[RAD_ILP];
    float2 s[RAD_ILP], sp[RAD_ILP];
#pragma unroll
    for (int k = 0; k < RAD_ILP; ++k) {
      const int p = p0 + k * nthreads;
      ok[k] = false;
      if (p >= v.nt) continue;
      const float2* S = src(p);
      if (!S) continue;
      ok[k] = true;
      g[k] = (int)v.rperm[p];
      s[k] = ld_it(S + p);
      e[k] = B.EP[p];
      sp[k] = warm ? v.sprev[p] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < RAD_ILP; ++k) {
      if (!ok[k]) continue;
      const int p = p0 + k * nthreads;
      x[g[k]] = e[k] + df_value(s[k]);
      if (warm) {
        v.sprev[v.nt + p] = df_add(s[k], df_neg(sp[k]));
        v.sprev[p] = s[k];
      }
    }
  }
}
__device__ __forceinline__ void scatter_x(const StepView& v, const MeshState64& st, double* x, int warm, int gt,
                                          int nthreads) {
  const RadBufs B(v);
  scatter_from(v, [&](int p) -> const float2* {
    const int m = mesh_of_facet(v, p);
    const MeshDesc& M = v.md[m];
    if (!M.active || M.ntiles == 0) return nullptr;
    return (st.mode[m] & 2) ? B.S1 : B.S0;
  }, x, warm, gt, nthreads);
}
__device__ __forceinline__ void scatter_solo(const StepView& v, const float2* S, double* x, int warm, int gt,
                                             int nthreads) {
  scatter_from(v, [&](int) { return S; }, x, warm, gt, nthreads);
}

// The rows of this block's tiles whose mesh stopped at the latest decision
// (st.now): x = E + s into facet order, and the warm-start record, as
// scatter_x. The block's rows are dealt to its consumer threads in one run
// over all its tiles (a thread takes every RAD_THREADS-th row of the
// concatenation), so each thread has a few rows in a row instead of a
// fraction of one per tile.
__device__ __forceinline__ void scatter_block(const StepView& v, const MeshState& st, const float2* S, double* x,
                                              int warm, const float* pred = nullptr) {
  const RadBufs B(v);
  int r = threadIdx.x;
  for (int k = v.blk_start[blockIdx.x]; k < v.blk_start[blockIdx.x + 1]; ++k) {
    const int t = v.blk_tile[k];
    const RowTile T = v.tiles[t];
    if (!st.now[T.mesh]) continue;
    const uint32_t* rows = v.t_row + T.r0;
    for (; r < T.nrows; r += RAD_THREADS) {
      const uint32_t i = __ldg(rows + r);
      const int g = (int)v.rperm[i];
      const float2 sv = ld_it(S + i);
      x[g] = B.EP[i] + df_value(sv);
      if (warm) {
        v.sprev[v.nt + i] = pred ? make_float2(ld_it(pred + i), 0.f) : df_add(sv, df_neg(v.sprev[i]));
        v.sprev[i] = sv;
      }
    }
    r -= T.nrows;
  }
}

struct RadSmem {
  unsigned char* ring;       // entry-stream stages (RAD_RING bytes)
  float2* sx;                // halo values (RAD_HALO double-floats, or floats)
  float2* tail;              // per-thread open-row partials
  float2* rs;                // row sums of the tile (RAD_ROWS double-floats, or floats)
  unsigned char* tnew;       // per thread: its last open row began in its run
  unsigned long long* full;  // per stage: its copies have landed
  unsigned long long* empty; // per stage: every consumer warp has read it
};

__device__ __forceinline__ RadSmem rad_smem() {
  extern __shared__ __align__(128) unsigned char rad_dyn[];
  RadSmem m;
  m.ring = rad_dyn;
  m.sx = reinterpret_cast<float2*>(rad_dyn + RAD_RING);
  m.tail = m.sx + RAD_HALO;
  m.rs = m.tail + RAD_THREADS;
  m.tnew = reinterpret_cast<unsigned char*>(m.rs + RAD_ROWS);
  m.full = reinterpret_cast<unsigned long long*>(m.tnew + RAD_THREADS);
  m.empty = m.full + RAD_STAGES;
  return m;
}
static_assert((RAD_RING + (size_t)(RAD_HALO + RAD_THREADS + RAD_ROWS) * 8 + RAD_THREADS) % 8 == 0,
              "stage barriers are 8-byte aligned");
// Dynamic shared memory of a launch over nmesh meshes.
constexpr size_t rad_smem_bytes(int nmesh) { return RAD_SMEM + (((size_t)nmesh * RAD_MESH_BYTES + 15) & ~(size_t)15); }

__device__ __forceinline__ MeshState::MeshState(int nmesh) {
  extern __shared__ __align__(128) unsigned char rad_dyn[];
  done = reinterpret_cast<int*>(rad_dyn + RAD_SMEM);
  sweeps = done + nmesh;
  unit = reinterpret_cast<float*>(sweeps + nmesh);
  now = reinterpret_cast<unsigned char*>(unit + nmesh);
}
__device__ __forceinline__ MeshState64::MeshState64(int nmesh) {
  extern __shared__ __align__(128) unsigned char rad_dyn[];
  sweeps = reinterpret_cast<int*>(rad_dyn + RAD_SMEM);
  acc = reinterpret_cast<float*>(sweeps + nmesh);
  prev = acc + nmesh;
  mode = reinterpret_cast<unsigned char*>(prev + nmesh);
}

// The ring's barriers, set up by thread 0 before the launch's first block
// barrier (inside init_meshes' caller): full counts the producer's one
// arrival plus the copied bytes, empty one arrival per consumer warp.
__device__ __forceinline__ Pipe make_pipe(const RadSmem& m, int* bad) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < RAD_STAGES; ++s) {
      mbar_init(m.full + s, 1);
      mbar_init(m.empty + s, RAD_THREADS / 32);
    }
    *bad = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  Pipe p;
  p.ring = m.ring;
  p.full = m.full;
  p.empty = m.empty;
  p.bad = bad;
  p.s = 0;
  p.parity = 0;
  return p;
}

// Producer warp: the copies of one pass over the block's tiles (lane 0
// issues; the other lanes only follow the launch's block barriers).
template <class V>
__device__ __forceinline__ void produce_pass(Pipe& p, const StepView& v, const MeshState& st, V vals, uint64_t pol) {
  if ((threadIdx.x & 31) != 0) return;
  for (int k = v.blk_start[blockIdx.x]; k < v.blk_start[blockIdx.x + 1]; ++k) {
    const int t = v.blk_tile[k];
    const RowTile T = v.tiles[t];
    if (st.done[T.mesh]) continue;
    produce_tile(p, v, T, vals, pol);
  }
}

// FP64 Jacobi to each mesh's tolerance, full and change sweeps as above.
// x: solution (and warm start).
__global__ void __maxnreg__(RAD_REGS64) k_radiosity64(StepView v, double* x, int warm) {
  MeshState64 st(v.nmesh);
  __shared__ float red[32];
  __shared__ int bad;
  const RadSmem sm = rad_smem();
  const bool producer = threadIdx.x >= RAD_THREADS;
  const int gt = blockIdx.x * RAD_THREADS + threadIdx.x;
  const int nthreads = gridDim.x * RAD_THREADS;
  unsigned gen = 0;
  Pipe pipe = make_pipe(sm, &bad);
  init_meshes64(v, st);
  if (!producer) init_x(v, x, warm, gt, nthreads, false);
  if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
  const uint64_t pol = l2_keep_policy(v.l2_stream);
  const ValsDF vals{v.t_vhi, v.t_vlo};
  const ValsHiF vhi{v.t_vhi};
  const int b0 = v.blk_start[blockIdx.x], b1 = v.blk_start[blockIdx.x + 1];
  for (int it = 0;; ++it) {
    if (producer) {
      if ((threadIdx.x & 31) == 0)
        for (int k = b0; k < b1; ++k) {
          const RowTile T = v.tiles[v.blk_tile[k]];
          const int mode = st.mode[T.mesh];
          if (mode >> MODE_DONE) continue;
          if (mode & 1) produce_tile(pipe, v, T, vhi, pol);
          else produce_tile(pipe, v, T, vals, pol);
        }
      __syncwarp();
    } else {
      const RadBufs B(v);
      const float* dcur = (it & 1) ? B.D1 : B.D0;   // the change of the sweep before
      float* dnxt = (it & 1) ? B.D0 : B.D1;
      for (int k = b0; k < b1; ++k) {
        const int t = v.blk_tile[k];
        const RowTile T = v.tiles[t];
        const int mode = st.mode[T.mesh];
        if (mode >> MODE_DONE) continue;
        const float unit = v.md[T.mesh].res_unit;
        float2* cur = (mode & 2) ? B.S1 : B.S0;
        const uint32_t* rows = v.t_row + T.r0;
        float d2 = 0.f;
        if (mode & 1) {
          float* sxf = reinterpret_cast<float*>(sm.sx);
          float* rsf = reinterpret_cast<float*>(sm.rs);
          const uint32_t s0 = tile_start(v, t);
          stage_halo(v, T, dcur, sxf);
          tile_rows<AccF32>(v, T, s0, pipe, vhi, sxf, reinterpret_cast<float*>(sm.tail), sm.tnew, rsf);
          for (int r = threadIdx.x; r < T.nrows; r += RAD_THREADS) {
            const uint32_t i = __ldg(rows + r);
            const float d = rsf[r];              // d' = F d
            cur[i] = df_add(ld_it(cur + i), make_float2(d, 0.f));
            dnxt[i] = d;
            d2 = __fmaf_rn(d, d, d2);
          }
        } else {
          float2* nxt = (mode & 2) ? B.S0 : B.S1;
          const uint32_t s0 = tile_start(v, t);
          stage_halo_sum(v, T, B.EH, cur, sm.sx);
          tile_rows<AccDF>(v, T, s0, pipe, vals, sm.sx, sm.tail, sm.tnew, sm.rs);
          for (int r = threadIdx.x; r < T.nrows; r += RAD_THREADS) {
            const uint32_t i = __ldg(rows + r);
            const float2 sn = sm.rs[r];          // s' = F x
            const float2 sc = ld_it(cur + i);
            // s' - s: exact high-part difference when the two are within a
            // factor of two, else rounded relative to the change itself
            const float d = __fadd_rn(__fsub_rn(sn.x, sc.x), __fsub_rn(sn.y, sc.y));
            nxt[i] = sn;
            dnxt[i] = d;
            d2 = __fmaf_rn(d, d, d2);
          }
        }
        post_partial64(v, T, t, it, unit, block_sum(d2, red));
      }
    }
    if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
    if (decide_meshes64(v, st, it) == 0) break;
  }
  if (!producer) scatter_x(v, st, x, warm, gt, nthreads);
  record_residuals64(v, st);
}

// ---- the FP64 solve of one mesh with at most one tile per block ----
//
// The same sweeps on the same tiles, bit for bit, for the usual single-mesh
// solve. A sweep of such a mesh is short (about 1 us of entries per block for
// 5,120 facets, 5 us for 81,920), so what it waits for decides: after a grid
// barrier the L1 is empty and every load is an L2 round trip. Here
// everything that does not change from sweep to sweep (the tile, the halo's
// and rows' positions, each thread's first row) and the block's own s stay in
// registers, and the barrier carries the residual: each block publishes its
// partial with the sweep's number in one 128-bit word, and every block reads
// all of them, instead of an atomic counter to wait for and a total to load
// after it.
// tile_d2 and the totals are those of k_radiosity64, so the decisions are.
// 81,920 facets, 8.1 M entries: a change sweep takes 11.6 us, 7 us of it the
// entries, which come from L2 at 8.5 TB/s (a full sweep's at 9.7, the copies
// alone at 10.9: taking half the shared-memory accesses out, or the row-end
// selections, changed nothing), 1.9 us the barrier even for the last block
// and 1 us the spread between blocks; 16.8 us a full one. In k_radiosity64
// they took 12.5 and 18.3 us.
struct __align__(16) SweepWord {
  unsigned long long units, tag;   // residual units; level << 32 | sweep number (from 1)
};
__device__ __forceinline__ SweepWord* sweep_words(const StepView& v) {
  return reinterpret_cast<SweepWord*>(v.barrier + RAD_BAR_WORDS0);
}
__device__ __forceinline__ void word_store(SweepWord* p, unsigned long long a, unsigned long long b) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ SweepWord word_load(const SweepWord* p) {
  SweepWord w;
  asm volatile("{\n\t.reg .b128 t;\n\tld.acquire.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(w.units), "=l"(w.tag) : "l"(p) : "memory");
  return w;
}

struct SoloShared {
  float red[32];
  int bad, ok, mode, stop;   // mode as MeshState64::mode
  float acc, prev, err;
};

constexpr int SOLO_HALO = 3;   // halo positions kept per thread (81,920 facets: 2,050 per tile on average)

// End of sweep `it` of the block whose partial is d2 (thread 0's): publish,
// wait for every block's (nb of them: the grid's), and decide. All threads;
// false once a wait ran out.
// A word is written after a fence and read by an acquiring load, so what the
// other blocks stored before theirs is visible to the loads after this (a
// fence after the wait instead: 0.2 us a sweep more).
__device__ __forceinline__ bool solo_sweep_end(const StepView& v, SoloShared& S, int it, float d2, float unit,
                                               float c, int budget, unsigned nb) {
  __syncthreads();   // the block's stores of this sweep come before its word
  SweepWord* words = sweep_words(v);
  if (threadIdx.x == 0) {
    int level;
    const unsigned long long u = res_units64(d2, unit, level);
    __threadfence();
    word_store(words + 2 * blockIdx.x + (it & 1), u, ((unsigned long long)level << 32) | (unsigned)(it + 1));
  }
  if (threadIdx.x < 32) {
    unsigned long long q0 = 0, q1 = 0, q2 = 0;
    bool ok = true;
    const long long limit = g_barrier_polls;
    for (unsigned b = threadIdx.x; b < nb && ok; b += 32) {
      SweepWord w;
      for (long long poll = 0;; ++poll) {
        w = word_load(words + 2 * b + (it & 1));
        if ((unsigned)w.tag == (unsigned)(it + 1)) break;
        if (poll > limit || ((poll & 255) == 255 && *(volatile int*)&v.derr[DERR_BARRIER])) {
          atomicExch(&v.derr[DERR_BARRIER], 1);
          ok = false;
          break;
        }
      }
      const int level = (int)(w.tag >> 32);
      q0 += level == 0 ? w.units : 0ull;
      q1 += level == 1 ? w.units : 0ull;
      q2 += level == 2 ? w.units : 0ull;
    }
    ok = __all_sync(0xffffffffu, ok);
    for (int o = 16; o; o >>= 1) {
      q0 += __shfl_xor_sync(0xffffffffu, q0, o);
      q1 += __shfl_xor_sync(0xffffffffu, q1, o);
      q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    }
    if (threadIdx.x == 0) {
      const bool change = S.mode & 1;
      const Sweep64 dec = sweep_decision(q0, q1, q2, change, c, S.acc, S.prev);
      const int cur = change ? S.mode & 2 : (S.mode & 2) ^ 2;
      const int sw = it + 1;
      S.mode = cur | (dec.next_change && sw + 1 < budget ? 1 : 0);
      S.stop = dec.stop || sw >= budget;
      S.acc = dec.acc;
      S.prev = dec.dn;
      S.err = dec.err;
      S.ok = ok;
    }
  }
  __syncthreads();
  return S.ok != 0;
}

__global__ void __maxnreg__(RAD_REGS64) k_radiosity64_solo(StepView v, double* x, int warm) {
  __shared__ SoloShared S;
  const RadSmem sm = rad_smem();
  const bool producer = threadIdx.x >= RAD_THREADS;
  const int gt = blockIdx.x * RAD_THREADS + threadIdx.x;
  const int nthreads = gridDim.x * RAD_THREADS;
  // blocks beyond the tiles (which the schedule gives to the first blocks) help
  // at the ends only: their tile is the empty one after the others
  const int t = blockIdx.x < v.ntiles ? v.blk_tile[v.blk_start[blockIdx.x]] : v.ntiles;
  const RowTile T = v.tiles[t];
  const float unit = v.md[0].res_unit, c = v.md[0].rad_err;
  const int budget = v.md[0].max_sweeps;
  if (!v.md[0].active) return;
  // the ring holds two and a half groups of a full sweep or five of a change sweep
  // (every group of a sweep is taken before the next sweep's first copy)
  Pipe pipe = make_pipe(sm, &S.bad);
  if (threadIdx.x == 0) {
    S.mode = 0;
    S.acc = S.prev = 0.f;
  }
  const RadBufs B(v);
  const ValsDF vals{v.t_vhi, v.t_vlo};
  const ValsHiF vhi{v.t_vhi};
  const uint64_t pol = l2_keep_policy(v.l2_stream);
  // a thread's first row stays in registers (most tiles have fewer rows than
  // threads), further ones are loaded again every sweep
  uint32_t s0 = 0, hpos[SOLO_HALO], rpos = 0;
  const bool has_row = !producer && threadIdx.x < T.nrows;
  if (!producer) {
    init_x(v, x, warm, gt, nthreads, false);
    s0 = t < v.ntiles ? tile_start(v, t) : 0u;
#pragma unroll
    for (int q = 0; q < SOLO_HALO; ++q) {
      const int h = threadIdx.x + q * RAD_THREADS;
      hpos[q] = h < T.nhalo ? __ldg(v.t_halo + T.h0 + h) : 0u;
    }
    if (has_row) rpos = __ldg(v.t_row + T.r0 + threadIdx.x);
  }
  unsigned gen = 0;
  if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
  float2 sown = has_row ? ld_it(B.S0 + rpos) : make_float2(0.f, 0.f);
  int it = 0, full = 0;
  for (;; ++it) {
    const int mode = S.mode;
    full += 1 - (mode & 1);
    float d2 = 0.f;
    if (producer) {
      if ((threadIdx.x & 31) == 0) {
        if (mode & 1) produce_tile(pipe, v, T, vhi, pol);
        else produce_tile(pipe, v, T, vals, pol);
      }
      __syncwarp();
    } else {
      float2* cur = (mode & 2) ? B.S1 : B.S0;
      const float* dcur = (it & 1) ? B.D1 : B.D0;
      float* dnxt = (it & 1) ? B.D0 : B.D1;
      if (mode & 1) {
        float* sxf = reinterpret_cast<float*>(sm.sx);
        float* rsf = reinterpret_cast<float*>(sm.rs);
        float g[SOLO_HALO];
#pragma unroll
        for (int q = 0; q < SOLO_HALO; ++q)
          if (threadIdx.x + q * RAD_THREADS < T.nhalo) g[q] = ld_it(dcur + hpos[q]);
#pragma unroll
        for (int q = 0; q < SOLO_HALO; ++q)
          if (threadIdx.x + q * RAD_THREADS < T.nhalo) sxf[threadIdx.x + q * RAD_THREADS] = g[q];
        for (int h = threadIdx.x + SOLO_HALO * RAD_THREADS; h < T.nhalo; h += RAD_THREADS)
          sxf[h] = ld_it(dcur + __ldg(v.t_halo + T.h0 + h));
        cbar();
        tile_rows<AccF32>(v, T, s0, pipe, vhi, sxf, reinterpret_cast<float*>(sm.tail), sm.tnew, rsf);
        auto finish = [&](uint32_t i, float d, float2& so) {
          so = df_add(so, make_float2(d, 0.f));
          cur[i] = so;
          dnxt[i] = d;
          d2 = __fmaf_rn(d, d, d2);
        };
        if (has_row) finish(rpos, rsf[threadIdx.x], sown);
        for (int r = threadIdx.x + RAD_THREADS; r < T.nrows; r += RAD_THREADS) {
          const uint32_t i = __ldg(v.t_row + T.r0 + r);
          float2 so = ld_it(cur + i);
          finish(i, rsf[r], so);
        }
      } else {
        float2* nxt = (mode & 2) ? B.S0 : B.S1;
        stage_halo_sum(v, T, B.EH, cur, sm.sx);
        tile_rows<AccDF>(v, T, s0, pipe, vals, sm.sx, sm.tail, sm.tnew, sm.rs);
        auto finish = [&](uint32_t i, float2 sn, float2& so) {
          const float d = __fadd_rn(__fsub_rn(sn.x, so.x), __fsub_rn(sn.y, so.y));
          so = sn;
          nxt[i] = sn;
          dnxt[i] = d;
          d2 = __fmaf_rn(d, d, d2);
        };
        if (has_row) finish(rpos, sm.rs[threadIdx.x], sown);
        for (int r = threadIdx.x + RAD_THREADS; r < T.nrows; r += RAD_THREADS) {
          const uint32_t i = __ldg(v.t_row + T.r0 + r);
          float2 so = ld_it(cur + i);
          finish(i, sm.rs[r], so);
        }
      }
      d2 = block_sum(d2, S.red);
      if (threadIdx.x == 0 && t < v.ntiles) v.tile_d2[(size_t)(it & 1) * v.ntiles + t] = (double)d2;
    }
    if (!solo_sweep_end(v, S, it, d2, unit, c, budget, gridDim.x)) return;
    if (S.stop) break;
  }
  if (!producer) {
    scatter_solo(v, (S.mode & 2) ? B.S1 : B.S0, x, warm, gt, nthreads);
    if (blockIdx.x == 0 && threadIdx.x < 32) {
      double r2 = 0.0;
      const double* d2 = v.tile_d2 + (size_t)(it & 1) * v.ntiles;
      for (int j = threadIdx.x; j < v.ntiles; j += 32) r2 += ld_it(d2 + j);
      r2 = warp_sum(r2);
      if (threadIdx.x == 0) {
        v.md[0].sweeps = it + 1;
        v.md[0].full_sweeps = full;
        v.md[0].res2 = with_errors(r2, S.err, v.md[0].tol2);
      }
    }
  }
}

// Mixed precision: outer refinement with the residual r = E - (I - fl(F)) x
// = fl(F) x - s (double-float sums), inner fp32 Jacobi on (I - F~) d = r with
// bf16 F~ (inner sweeps, 1..RAD_INNER), s += d. A mesh stops when
// ||r||_2 <= tol, or after the update of the round that reaches max_sweeps;
// each tile's block writes its rows' results.
__global__ void __maxnreg__(RAD_REGSM) k_radiosity_mixed(StepView v, double* x, int warm, int inner) {
  MeshState st(v.nmesh);
  __shared__ float red[32];
  __shared__ int bad;
  const RadSmem sm = rad_smem();
  const bool producer = threadIdx.x >= RAD_THREADS;
  float* sxf = reinterpret_cast<float*>(sm.sx);
  float* tailf = reinterpret_cast<float*>(sm.tail);
  float* rsf = reinterpret_cast<float*>(sm.rs);
  const int gt = blockIdx.x * RAD_THREADS + threadIdx.x;
  const int nthreads = gridDim.x * RAD_THREADS;
  float* xa = v.x32;
  float* xb = v.x32 + v.nt;
  float* r32 = v.x32 + 2 * (size_t)v.nt;
  unsigned gen = 0;
  Pipe pipe = make_pipe(sm, &bad);
  init_meshes(v, st);
  if (!producer) init_x(v, x, warm, gt, nthreads, true);
  if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
  const uint64_t pol = l2_keep_policy(v.l2_stream);
  const RadBufs B(v);
  const ValsHi vhi{v.t_vhi};
  const ValsBF vbf{v.t_vbf};
  float2* S = B.S0;     // the iterate's scattered part s = x - E (radiosity positions)
  float2* XH = B.H0;    // x = E + s, what the halos gather
  int first = 1;
  for (int round = 0;; ++round) {
    if (producer) {
      produce_pass(pipe, v, st, vhi, pol);
      __syncwarp();
    } else {
      for (int k = v.blk_start[blockIdx.x]; k < v.blk_start[blockIdx.x + 1]; ++k) {
        const int t = v.blk_tile[k];
        const RowTile T = v.tiles[t];
        if (st.done[T.mesh]) continue;
        const uint32_t s0 = tile_start(v, t);
        stage_halo(v, T, XH, sm.sx);
        tile_rows<AccDF>(v, T, s0, pipe, vhi, sm.sx, sm.tail, sm.tnew, sm.rs);
        const uint32_t* rows = v.t_row + T.r0;
        float d2 = 0.f;
        for (int r = threadIdx.x; r < T.nrows; r += RAD_THREADS) {
          uint32_t i = __ldg(rows + r);
          // r = E + fl(F) x - x = fl(F) x - s
          const float2 fx = sm.rs[r], s = ld_it(S + i);
          const float res = __fadd_rn(__fsub_rn(fx.x, s.x), __fsub_rn(fx.y, s.y));
          r32[i] = res;
          xa[i] = res;     // inner start: d0 = r
          d2 = __fmaf_rn(res, res, d2);
        }
        post_partial(v, st, T, t, round, block_sum(d2, red));
      }
    }
    if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
    int running = decide_meshes(v, st, inner, first, round);
    first = 0;
    // meshes that stopped on their residual: each block writes its own
    // tiles' rows (their s was last written by this block)
    if (!producer) scatter_block(v, st, S, x, warm);
    if (running == 0) break;
    float* cur = xa;
    float* nxt = xb;
    for (int it = 0; it < inner; ++it) {
      if (producer) {
        produce_pass(pipe, v, st, vbf, pol);
        __syncwarp();
      } else {
        for (int k = v.blk_start[blockIdx.x]; k < v.blk_start[blockIdx.x + 1]; ++k) {
          const int t = v.blk_tile[k];
          const RowTile T = v.tiles[t];
          if (st.done[T.mesh]) continue;
          const uint32_t s0 = tile_start(v, t);
          stage_halo(v, T, cur, sxf);
          tile_rows<AccF32>(v, T, s0, pipe, vbf, sxf, tailf, sm.tnew, rsf);
          const uint32_t* rows = v.t_row + T.r0;
          const float* scale = v.t_scale + T.r0;
          if (it + 1 < inner) {
            for (int r = threadIdx.x; r < T.nrows; r += RAD_THREADS) {
              uint32_t i = __ldg(rows + r);
              nxt[i] = ld_it(r32 + i) + __ldg(scale + r) * rsf[r];
            }
          } else {   // last sweep: nobody reads d again, s += d directly
            // (x for the halos only if the mesh runs another round)
            const bool more = st.sweeps[T.mesh] + inner < v.md[T.mesh].max_sweeps;
            for (int r = threadIdx.x; r < T.nrows; r += RAD_THREADS) {
              uint32_t i = __ldg(rows + r);
              const float2 d = make_float2(ld_it(r32 + i) + __ldg(scale + r) * rsf[r], 0.f);
              S[i] = df_add(ld_it(S + i), d);
              if (more) XH[i] = df_add(ld_it(XH + i), d);
            }
          }
          cbar();
        }
      }
      if (it + 1 < inner) {
        if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
        float* tmp = cur; cur = nxt; nxt = tmp;
      }
    }
    // meshes whose budget this round used up stop here (same decision in
    // every block: it depends on the counts only) and take their results
    // (each block its own tiles' rows, whose s it wrote)
    int left = 0;
    for (int m0 = 0; m0 < v.nmesh; m0 += blockDim.x) {
      int m = m0 + threadIdx.x;
      bool run = m < v.nmesh && !st.done[m];
      if (m < v.nmesh) st.now[m] = 0;
      if (run && st.sweeps[m] + inner >= v.md[m].max_sweeps) {
        st.done[m] = 1 + (round & 1);
        st.sweeps[m] += inner;
        st.now[m] = 1;
        if (blockIdx.x == 0) v.md[m].sweeps = st.sweeps[m];
        run = false;
      }
      left += __syncthreads_count(run);
    }
    if (!producer) scatter_block(v, st, S, x, warm);
    if (left == 0) break;   // every result is written (by its tile's block)
    if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
  }
  record_residuals(v, st);
}

// Mixed precision, one pass over the matrix per step (refine_every = K >=
// 1). The pass applies F to x - x_ref, where x = E + s0 is the step's
// iterate and x_ref the iterate of the mesh's last reference step:
//   s = s_ref + F (x - x_ref),
// with the f32 values on a reference step (every K-th step of a mesh, and
// a step without an earlier reference, where x_ref = 0 and s_ref = 0: the
// mesh's first, or its first after a new matrix or another solve on its
// buffers), which then keeps (s, x) as the new reference, and the bf16 copy
// F~ on the steps between:
// s = F x - (F - F~)(x - x_ref), the bf16 error confined to the change
// since the reference step. Sums in FP32 (the terms are changes); s and
// s_ref stay double-float. A single sweep from the previous solution would
// leave the multiple scattering of a change of E one order behind (F^2 dE
// for a facet that crosses the terminator), so the warm start predicts it:
// the same pass also forms P = F (E(n+1) - E(n)) with the next frame's
// direct flux (a second right-hand side on the same matrix entries, 8 B
// halos of (x - x_ref, dE)), and the next step starts from s0 = s + P, off by
// F^2 dE instead of F dE. The step's squared change |s - s0|^2 is recorded
// as its residual.
__global__ void __maxnreg__(RAD_REGSM) k_radiosity_lagged(StepView v, double* x, int warm) {
  MeshState st(v.nmesh);
  __shared__ float red[32];
  __shared__ int bad;
  // each mesh's kind of pass (0: bf16 step, 1: reference step, 2: reference
  // step without an earlier reference) lives in st.now, unused until the pass
  // is over
  unsigned char* kind = st.now;
  const RadSmem sm = rad_smem();
  const bool producer = threadIdx.x >= RAD_THREADS;
  const int gt = blockIdx.x * RAD_THREADS + threadIdx.x;
  const int nthreads = gridDim.x * RAD_THREADS;
  const RadBufs B(v);
  float2* XD = B.EH;            // by position: (x - x_ref, E(n+1) - E(n))
  float* pred = v.x32 + v.nt;   // by position: P, the predicted change of s
  unsigned gen = 0;
  Pipe pipe = make_pipe(sm, &bad);
  init_meshes(v, st);
  for (int m = threadIdx.x; m < v.nmesh; m += blockDim.x) {
    const MeshDesc& M = v.md[m];
    kind[m] = M.ref_age < 0 ? 2 : (M.ref_age + 1 >= M.refine_every ? 1 : 0);
  }
  __syncthreads();
  if (!producer) init_x(v, x, warm, gt, nthreads, true, kind);
  if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
  // every block has read the ages: block 0 advances them
  if (blockIdx.x == 0)
    for (int m = threadIdx.x; m < v.nmesh; m += blockDim.x)
      if (!st.done[m]) v.md[m].ref_age = kind[m] ? 0 : v.md[m].ref_age + 1;
  const uint64_t pol = l2_keep_policy(v.l2_stream);
  const ValsHiF vhi{v.t_vhi};
  const ValsBF vbf{v.t_vbf};
  if (producer) {
    if ((threadIdx.x & 31) == 0)
      for (int k = v.blk_start[blockIdx.x]; k < v.blk_start[blockIdx.x + 1]; ++k) {
        const RowTile T = v.tiles[v.blk_tile[k]];
        if (st.done[T.mesh]) continue;
        if (kind[T.mesh]) produce_tile(pipe, v, T, vhi, pol);
        else produce_tile(pipe, v, T, vbf, pol);
      }
    __syncwarp();
  } else {
    for (int k = v.blk_start[blockIdx.x]; k < v.blk_start[blockIdx.x + 1]; ++k) {
      const int t = v.blk_tile[k];
      const RowTile T = v.tiles[t];
      if (st.done[T.mesh]) continue;
      const int kd = kind[T.mesh];
      const uint32_t s0t = tile_start(v, t);
      stage_halo(v, T, XD, sm.sx);
      if (kd) tile_rows<AccF2>(v, T, s0t, pipe, vhi, sm.sx, sm.tail, sm.tnew, sm.rs);
      else tile_rows<AccF2>(v, T, s0t, pipe, vbf, sm.sx, sm.tail, sm.tnew, sm.rs);
      const uint32_t* rows = v.t_row + T.r0;
      const float* scale = v.t_scale + T.r0;
      float d2 = 0.f;
      for (int r = threadIdx.x; r < T.nrows; r += RAD_THREADS) {
        const uint32_t i = __ldg(rows + r);
        const float2 a = sm.rs[r];   // F (x - x_ref), F dE of the row
        const float sc = kd ? 1.f : __ldg(scale + r);
        const float2 sref = kd == 2 ? make_float2(0.f, 0.f) : ld_it(B.S1 + i);
        const float2 sn = df_add(sref, make_float2(sc * a.x, 0.f));
        const float2 s0 = ld_it(B.S0 + i);
        const float df = __fadd_rn(__fsub_rn(sn.x, s0.x), __fsub_rn(sn.y, s0.y));
        if (kd) B.S1[i] = sn;
        B.S0[i] = sn;
        pred[i] = sc * a.y;
        d2 = __fmaf_rn(df, df, d2);
      }
      post_partial(v, st, T, t, 0, block_sum(d2, red));
    }
  }
  // every solved mesh stops after this pass: each block writes its own
  // tiles' rows (whose s and P it wrote); the residual record waits for all
  // tiles
  __syncthreads();
  for (int m = threadIdx.x; m < v.nmesh; m += blockDim.x) {
    st.now[m] = st.done[m] ? 0 : 1;
    if (!st.done[m]) {
      st.done[m] = 1;
      st.sweeps[m] = 1;
      if (blockIdx.x == 0) v.md[m].sweeps = 1;
    }
  }
  __syncthreads();
  if (!producer) scatter_block(v, st, B.S0, x, warm, pred);
  if (!grid_barrier(v.barrier, gridDim.x, gen, v.derr)) return;
  record_residuals(v, st);
}

// Bounds of the change sweeps' errors (the FP64 solve): || |F| ||_2 is at most
// the root of the largest row sum times the largest column sum of |F|. The
// column sums are integers, in units of max |F| / 2^32, so that the result
// does not depend on the order of the additions.
struct FNorms {
  unsigned max_abs, row_sum;    // rounded up, as the bits of floats, whose order is theirs (a NaN counts as largest)
  unsigned long long col_sum;   // in units
};
// An entry's |F| in units.
__device__ __forceinline__ unsigned long long norm_units(double f, const FNorms* norms) {
  return __float2ull_ru(__fmul_ru(__fdiv_ru(__double2float_ru(fabs(f)), __uint_as_float(norms->max_abs)), 4294967296.f));
}
__global__ void k_col_max(const unsigned long long* __restrict__ sums, int nt, FNorms* norms) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long m = j < nt ? sums[j] : 0ull;
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(&norms->col_sum, m);
}

// Per-row fp32 scale = max |F_ij| of the row (the bf16 copy stores F/scale).
// One warp per row, here and in k_row_keys: with one thread per row 22 M
// entries in 130,050 rows took 134 and 463 us.
__global__ void k_row_scale(const int64_t* __restrict__ rowptr, const double* __restrict__ val, int nt,
                            float* rscale, FNorms* norms) {
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= nt) return;
  double m = 0.0;
  float sum = 0.f;
  for (int64_t k = rowptr[i] + lane; k < rowptr[i + 1]; k += 32) {
    const double a = fabs(val[k]);
    m = fmax(m, a);
    sum = __fadd_ru(sum, __double2float_ru(a));
  }
  for (int o = 16; o; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    sum = __fadd_ru(sum, __shfl_xor_sync(0xffffffffu, sum, o));
  }
  if (lane == 0) {
    rscale[i] = m > 0.0 ? (float)m : 1.f;
    if (sum != 0.f) {   // (most rows are not the largest so far)
      const unsigned mb = __float_as_uint(__double2float_ru(m)), sb = __float_as_uint(fabsf(sum));
      if (mb > *(volatile unsigned*)&norms->max_abs) atomicMax(&norms->max_abs, mb);
      if (sb > *(volatile unsigned*)&norms->row_sum) atomicMax(&norms->row_sum, sb);
    }
  }
}

// key = row << rb | Morton position of the column; value = CSR entry.
__global__ void k_row_keys(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                           const uint32_t* __restrict__ rank, int nt, int rb, unsigned long long* key,
                           uint32_t* src) {
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= nt) return;
  const unsigned long long hi = (unsigned long long)i << rb;
  for (int64_t k = rowptr[i] + lane; k < rowptr[i + 1]; k += 32) {
    key[k] = hi | rank[col[k]];
    src[k] = (uint32_t)k;
  }
}

// Tile build on the device.
// key = (tile of the entry's row) << rb | Morton rank of its column; value =
// the entry's index in the row-sorted order.
__global__ void k_tile_keys(const unsigned long long* __restrict__ skey, int64_t n, int rb,
                            const int* __restrict__ tile_of, unsigned long long* key, uint32_t* idx) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned long long cm = (1ull << rb) - 1;
  const int g = (int)(skey[k] >> rb);
  key[k] = ((unsigned long long)tile_of[g] << rb) | (skey[k] & cm);
  idx[k] = (uint32_t)k;
}

// 1 where a (tile, column) run starts in the sorted keys.
__global__ void k_run_flags(const unsigned long long* __restrict__ key, int64_t n, uint32_t* flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  flag[i] = (i == 0 || key[i] != key[i - 1]) ? 1u : 0u;
}

// Runs are the tiles' halo facets, in (tile, Morton rank) order: the run
// index is the facet's slot in t_halo, and a tile's first run is its h0.
__global__ void k_halo_runs(const unsigned long long* __restrict__ key, const uint32_t* __restrict__ flag,
                            const unsigned long long* __restrict__ before, int64_t n, int rb, uint32_t* t_halo,
                            int* tile_first) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !flag[i]) return;
  const unsigned long long cm = (1ull << rb) - 1;
  const int64_t r = (int64_t)before[i];
  t_halo[r] = (uint32_t)(key[i] & cm);
  const int t = (int)(key[i] >> rb);
  if (i == 0 || (int)(key[i - 1] >> rb) != t) tile_first[t] = (int)r;
}

// Each entry to its stored slot: entry j of a tile (rows in Morton order,
// each row's entries in column order) belongs to thread t = j / lam as its
// kk = j % lam-th, stored at e0 + (kk / 4) RAD_GROUP + 4 t + kk % 4; the slot
// holds the entry's halo index (run - h0) with the row-end bit, the CSR
// entry it takes its value from, and its row (for the row scale).
__global__ void k_tile_slots(const unsigned long long* __restrict__ key, const uint32_t* __restrict__ idx,
                             const uint32_t* __restrict__ flag, const unsigned long long* __restrict__ before,
                             int64_t n, int rb, const unsigned long long* __restrict__ skey,
                             const uint32_t* __restrict__ ssrc, const int64_t* __restrict__ rowptr,
                             const int* __restrict__ rowoff, const RowTile* __restrict__ tiles, uint16_t* cf,
                             uint32_t* esrc, uint32_t* efac, const double* __restrict__ val,
                             const uint32_t* __restrict__ order, const FNorms* norms, unsigned long long* col_sums) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool in = i < n;
  {   // the column sums, a run of equal columns at a time (one atomic per entry: 0.65 ms for 22 M)
    unsigned long long u = in ? norm_units(val[ssrc[idx[i]]], norms) : 0ull;
    const unsigned heads = __ballot_sync(0xffffffffu, !in || flag[i] || lane == 0);
    const int start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, u, o);
      if (lane - o >= start) u += y;
    }
    const bool last = lane == 31 || ((heads >> (lane + 1)) & 1);
    if (in && last) atomicAdd(col_sums + order[key[i] & ((1ull << rb) - 1ull)], u);
  }
  if (!in) return;
  const int t = (int)(key[i] >> rb);
  const RowTile T = tiles[t];
  const int64_t run = (int64_t)before[i] + flag[i] - 1;
  const uint32_t loc = (uint32_t)(run - T.h0);
  const int64_t k = idx[i];
  const int g = (int)(skey[k] >> rb);
  const int64_t j = rowoff[g] + (k - rowptr[g]);
  const int64_t th = j / T.lam, kk = j - th * T.lam;
  const int64_t off = T.e0 + (kk >> 2) * 4 * RAD_THREADS + 4 * th + (kk & 3);
  cf[off] = (uint16_t)(loc | (k + 1 == rowptr[g + 1] ? 0x8000u : 0u));
  esrc[off] = ssrc[k];
  efac[off] = (uint32_t)g;
}

// Order of the entries within each piece of a row (the entries of one row in
// one thread's run; their sum may be taken in any order): the 32 lanes of a
// warp read one halo value each per step, from wherever their rows' columns
// lie, and random columns hit the same bank of shared memory 3.5 times (two
// words per value: 6.1). Each step's entries are chosen from the next
// BANK_WINDOW of every lane's piece: lanes propose an entry whose bank is
// still free (for one-word values: 32 banks; for two-word values, which the
// hardware serves half a warp at a time: 16 pairs), the lowest lane of those
// that propose the same one takes it, and the others look again; then the
// same with banks used once; then the first entry. Random columns come to 2.2
// and 4.2 accesses (a window of 32 entries and eight rounds: 2.1 and 3.9). The
// one-pass mixed solve of 36.7 M entries takes 95 us instead of 103; the FP64
// sweeps are bound by the stream from L2 and take what they took.
// One warp per warp of a tile, in place.
constexpr int BANK_WINDOW = 4;
constexpr int BANK_ROUNDS = 2;

__global__ void __launch_bounds__(128) k_tile_banks(const RowTile* __restrict__ tiles, int ntiles, uint16_t* cf,
                                                    uint32_t* esrc) {
  constexpr int WARPS = RAD_THREADS / 32;
  __shared__ uint32_t window[4][BANK_WINDOW][32];   // the candidates' CSR entries
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (w >= (int64_t)ntiles * WARPS) return;
  uint32_t(&src)[BANK_WINDOW][32] = window[threadIdx.x >> 5];
  const RowTile T = tiles[w / WARPS];
  const int64_t base = T.e0 + 4 * (32 * (w % WARPS) + lane);
  auto at = [&](int k) { return base + (int64_t)(k >> 2) * RAD_GROUP + (k & 3); };
  unsigned c[BANK_WINDOW];   // the candidates' halo indices
  unsigned have = 0;         // slots in use
  bool open = true, ends = false;   // the piece has entries after the window; its last one ends its row
  int next = 0;
  unsigned pair = 0;   // the even entry's code
  for (int k = 0; k < T.lam; ++k) {
    if (!have) open = true;
#pragma unroll
    for (int i = 0; i < BANK_WINDOW; ++i)
      if (open && !((have >> i) & 1)) {
        const unsigned v = cf[at(next)];
        c[i] = v & 0x7fffu;
        src[i][lane] = esrc[at(next)];
        have |= 1u << i;
        ++next;
        ends = (v & 0x8000u) != 0;
        open = !ends && next < T.lam;
      }
    int q = -1;
    unsigned loc = 0;
    // banks (32) and, by half warp, bank pairs (2 x 16) in use: once, twice
    unsigned b1 = 0, b2 = 0, h1 = 0, h2 = 0;
    const int half = lane & 16;
    for (int phase = 0; phase < 2; ++phase) {
      for (int r = 0; r < BANK_ROUNDS; ++r) {
        const unsigned bu = phase ? b2 : b1, hu = phase ? h2 : h1;
        int want = -1;
        unsigned wc = 0;
        if (q < 0) {
#pragma unroll
          for (int i = 0; i < BANK_WINDOW; ++i)
            if (want < 0 && ((have >> i) & 1) && !((bu >> (c[i] & 31)) & 1) &&
                !((hu >> (half + (c[i] & 15))) & 1)) {
              want = i;
              wc = c[i];
            }
        }
        const unsigned asking = __ballot_sync(0xffffffffu, want >= 0);
        if (!asking) break;
        unsigned same = asking;
#pragma unroll
        for (int bit = 0; bit < 4; ++bit) {
          const bool one = (wc >> bit) & 1;
          const unsigned m = __ballot_sync(0xffffffffu, one);
          same &= one ? m : ~m;
        }
        // the same pair in this half of the warp, the same bank anywhere
        const unsigned m4 = __ballot_sync(0xffffffffu, (wc >> 4) & 1);
        const unsigned bank = same & (((wc >> 4) & 1) ? m4 : ~m4);
        const unsigned rivals = (same & (half ? 0xffff0000u : 0xffffu)) | bank;
        const bool win = want >= 0 && (rivals & ((1u << lane) - 1u)) == 0;
        const unsigned nb = __reduce_or_sync(0xffffffffu, win ? 1u << (wc & 31) : 0u);
        const unsigned nh = __reduce_or_sync(0xffffffffu, win ? 1u << (half + (wc & 15)) : 0u);
        b2 |= b1 & nb;
        b1 |= nb;
        h2 |= h1 & nh;
        h1 |= nh;
        if (win) {
          q = want;
          loc = wc;
        }
      }
    }
    if (q < 0) {
      q = __ffs(have) - 1;
#pragma unroll
      for (int i = 0; i < BANK_WINDOW; ++i)
        if (i == q) loc = c[i];
    }
    have &= ~(1u << q);
    const bool end = !have && !open && ends;
    if (k & 1) {
      *reinterpret_cast<uint32_t*>(cf + at(k - 1)) = pair | loc << 16 | (end ? CF_END1 : 0u);
    } else {
      pair = loc | (end ? CF_END0 : 0u);
    }
    esrc[at(k)] = src[q][lane];
  }
}

// Each thread's first row (with a continuation bit when its run starts
// inside the row): rowj0 holds each tile row's first entry index within the
// tile, tile rows in order.
__global__ void k_tile_starts(const RowTile* __restrict__ tiles, int ntiles, const int64_t* __restrict__ ne,
                              const int* __restrict__ rowj0, uint32_t* tstart) {
  int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)ntiles * RAD_THREADS) return;
  const int tid = (int)(q / RAD_THREADS), t = (int)(q % RAD_THREADS);
  const RowTile T = tiles[tid];
  const int64_t j0 = (int64_t)t * T.lam;
  if (j0 >= ne[tid]) { tstart[q] = (uint32_t)T.nrows; return; }
  const int* rj = rowj0 + T.r0;
  int lo = 0, hi = T.nrows;   // last row with rj <= j0
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((int64_t)rj[mid] <= j0) lo = mid; else hi = mid;
  }
  tstart[q] = (uint32_t)lo | ((int64_t)rj[lo] != j0 ? 0x80000000u : 0u);
}

// Stored entry e takes CSR entry src[e] (value as a double-float, and its
// bf16 copy scaled by its row's scale), or zero for padding (src = ~0).
__global__ void k_tile_fill(const uint32_t* __restrict__ src, const uint32_t* __restrict__ fac, int64_t n,
                            const double* __restrict__ val, const float* __restrict__ rscale, float* t_vhi,
                            float* t_vlo, __nv_bfloat16* t_vbf) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  uint32_t k = src[e];
  double w = k == 0xffffffffu ? 0.0 : val[k];
  float2 hl = split_df(w);
  t_vhi[e] = hl.x;
  t_vlo[e] = hl.y;
  t_vbf[e] = __float2bfloat16_rn(k == 0xffffffffu ? 0.f : (float)(w / (double)rscale[fac[e]]));
}

__global__ void k_tile_scale(const uint32_t* __restrict__ t_row, const uint32_t* __restrict__ rperm, int n,
                             const float* __restrict__ rscale, float* t_scale) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) t_scale[k] = rscale[rperm[t_row[k]]];
}

int g_rad_nsm = 0, g_rad_per_sm64 = 0, g_rad_per_smm = 0;
std::atomic<bool> g_rad_ready{false};
std::mutex g_rad_mu;

// Once per process, before any capture: the kernels' shared-memory opt-in
// and their co-residency. Safe to call from several host threads.
int radiosity_setup() {
  if (g_rad_ready.load(std::memory_order_acquire)) return ILG_OK;
  std::lock_guard<std::mutex> lock(g_rad_mu);
  if (g_rad_ready.load(std::memory_order_relaxed)) return ILG_OK;
  int dev, nsm;
  ILG_CUDA(cudaGetDevice(&dev));
  ILG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const size_t most = rad_smem_bytes(RAD_MAX_MESH);
  for (const void* k : {(const void*)k_radiosity64, (const void*)k_radiosity64_solo, (const void*)k_radiosity_mixed,
                        (const void*)k_radiosity_lagged}) {
    int per = 0;   // one grid (and tile schedule) serves every kernel
    ILG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    ILG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, RAD_BLOCK, most));
    const bool fp64 = k == (const void*)k_radiosity64 || k == (const void*)k_radiosity64_solo;
    int& least = fp64 ? g_rad_per_sm64 : g_rad_per_smm;
    least = least > 0 ? std::min(least, per) : per;
  }
  if (g_rad_per_sm64 < 1 || g_rad_per_smm < 1) { set_error("radiosity kernel cannot be resident"); return ILG_ERR_CUDA; }
  g_rad_nsm = nsm;
  g_rad_ready.store(true, std::memory_order_release);
  return ILG_OK;
}

}  // namespace

// Row tiles of the form-factor matrix in Morton order (see the top of the
// file). Tile sizes target nnz / (co-resident blocks) entries, at least
// RAD_MIN_TILE, and a tile closes early when its halo would exceed RAD_HALO
// or its rows RAD_ROWS.
int radiosity_prepare(Context& c) {
  ILG_TRY(radiosity_setup());
  c.ref_age = -1;   // a new matrix or layout: no one-pass reference
  cudaStream_t s = c.stream;
  const int nt = c.nt;
  const int64_t nnz = c.nnz;
  ILG_TRY(c.row_scale.alloc(nt));
  dbuf<FNorms> norms;
  dbuf<unsigned long long> col_sums;
  ILG_TRY(norms.alloc(1));
  ILG_TRY(col_sums.alloc(nt));
  ILG_CUDA(cudaMemsetAsync(norms.p, 0, sizeof(FNorms), s));
  ILG_CUDA(cudaMemsetAsync(col_sums.p, 0, (size_t)nt * 8, s));
  k_row_scale<<<div_up((int64_t)nt * 32, 256), 256, 0, s>>>(c.rowptr.p, c.val.p, nt, c.row_scale.p, norms.p);
  ILG_CUDA(cudaGetLastError());
  ILG_TRY(c.rperm.alloc(nt));
  ILG_CUDA(cudaMemcpyAsync(c.rperm.p, c.morton_order.p, (size_t)nt * 4, cudaMemcpyDeviceToDevice, s));

  // Each row's entries in Morton order of their columns, sorted on the
  // device: key = (row, Morton position of the column), value = CSR entry.
  // Only N-sized data (row pointers, the Morton order, per-row halo bounds)
  // comes to the host, which cuts the tiles; everything per entry stays on
  // the device.
  int rb = 1;
  while ((1 << rb) < nt) ++rb;
  std::vector<int64_t> rp((size_t)nt + 1);
  std::vector<uint32_t> order((size_t)nt);
  ILG_CUDA(cudaMemcpyAsync(rp.data(), c.rowptr.p, rp.size() * 8, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaMemcpyAsync(order.data(), c.morton_order.p, (size_t)nt * 4, cudaMemcpyDeviceToHost, s));
  dbuf<unsigned long long> dkey;
  dbuf<uint32_t> dsv;
  if (nnz > 0) {
    ILG_TRY(dkey.alloc(nnz));
    ILG_TRY(dsv.alloc(nnz));
    k_row_keys<<<div_up((int64_t)nt * 32, 256), 256, 0, s>>>(c.rowptr.p, c.col.p, c.leaf_rank.p, nt, rb, dkey.p, dsv.p);
    ILG_CUDA(cudaGetLastError());
    ILG_TRY(radix_sort_u64(dkey.p, dsv.p, nnz, 2 * rb, c.sort, s));
  }
  ILG_CUDA(cudaStreamSynchronize(s));

  // active rows (with entries) in Morton order
  std::vector<uint8_t> act((size_t)nt, 0);
  std::vector<int> arow;   // positions
  for (int p = 0; p < nt; ++p) {
    int g = (int)order[p];
    int64_t len = rp[g + 1] - rp[g];
    if (len > 0) {
      if (len > RAD_HALO) {
        set_error("facet %d sees %lld facets; the radiosity solve supports at most %d per facet", g,
                  (long long)len, RAD_HALO);
        return ILG_ERR_ARG;
      }
      act[p] = 1;
      arow.push_back(p);
    }
  }
  c.n_active = (int)arow.size();

  // Tile cuts. A tile's stream time follows its whole groups (every thread
  // runs ceil(entries / RAD_GROUP) groups of four), so tiles get equal group
  // counts: the smallest ng for which a greedy pass with at most ng * RAD_GROUP
  // entries per tile needs no more tiles than co-resident blocks. A second
  // pass also closes a tile early once its weighed cost (entries + rows)
  // exceeds ng * RAD_GROUP plus the first pass's mean row cost, so row-heavy
  // tiles carry fewer entries; it is kept if it still fits the grid. If the
  // row cap forces more tiles than blocks (very large meshes), the cuts are
  // equal shares of the estimated work (entries + rows), several tiles per
  // block. Halos are then counted exactly on the device and a tile whose
  // halo exceeds the shared-memory capacity is split in two, until none
  // does.
  const int Gdev = g_rad_nsm * std::min(g_rad_per_sm64, g_rad_per_smm);
  const int G = c.tile_blocks > 0 ? std::min(Gdev, c.tile_blocks) : Gdev;
  std::vector<RowTile> tiles;
  std::vector<size_t> tile_a;   // first active row of each tile
  std::vector<int64_t> tile_ne;  // entries of each tile
  const int64_t NOCAP = std::numeric_limits<int64_t>::max() / 4;
  auto rlen = [&](size_t q) { const int g = (int)order[arow[q]]; return rp[g + 1] - rp[g]; };
  auto push_tile = [&](size_t a, size_t b, int64_t ne) {
    RowTile T{};
    T.lam = (int)(((ne + RAD_THREADS - 1) / RAD_THREADS + 3) & ~(int64_t)3);
    T.nrows = (int)(b - a);
    T.mesh = 0;
    tiles.push_back(T);
    tile_a.push_back(a);
    tile_ne.push_back(ne);
  };
  // One greedy pass. cap > 0: at most cap entries and cap + slack weighed
  // cost per tile; returns false once more than max_tiles are needed, and
  // counts the tiles closed by the row cap. cap == 0: cumulative equal
  // shares of total_cost over ntarget tiles.
  auto cut = [&](int64_t cap, int64_t slack, int64_t total_cost, int64_t ntarget, size_t max_tiles,
                 int* capped) -> bool {
    tiles.clear();
    tile_a.clear();
    tile_ne.clear();
    if (capped) *capped = 0;
    int64_t done_cost = 0;
    size_t a = 0;
    while (a < arow.size()) {
      if (tiles.size() >= max_tiles) return false;
      const int tid = (int)tiles.size();
      const int64_t bound = cap > 0 ? 0 : (int64_t)((double)total_cost * (double)(tid + 1) / (double)ntarget);
      size_t b = a;
      int64_t ne = 0;
      while (b < arow.size()) {
        if (b > a && (int64_t)(b - a) >= RAD_ROWS) {
          if (capped) ++*capped;
          break;
        }
        const int64_t len = rlen(b);
        if (cap > 0 && b > a && ne + len > cap) break;
        if (cap > 0 && b > a && ne + len + RAD_ROW_COST * (int64_t)(b - a + 1) > cap + slack) break;
        ne += len;
        ++b;
        if (cap == 0 && done_cost + ne + RAD_ROW_COST * (int64_t)(b - a) >= bound && tid + 1 < ntarget) break;
      }
      push_tile(a, b, ne);
      done_cost += ne + RAD_ROW_COST * (int64_t)(b - a);
      a = b;
    }
    return true;
  };
  {
    int64_t ng = std::max<int64_t>((RAD_MIN_TILE + RAD_GROUP - 1) / RAD_GROUP,
                                   (nnz + (int64_t)G * RAD_GROUP - 1) / ((int64_t)G * RAD_GROUP));
    bool ok = false;
    int capped = 0;
    for (int tries = 0; tries < 4; ++tries, ++ng) {
      ok = cut(ng * RAD_GROUP, NOCAP, 0, 0, (size_t)G, &capped);
      if (ok || capped > 0) break;   // a larger ng cannot lift the row cap
    }
    if (ok && !tiles.empty()) {
      int64_t extra = 0;
      for (const RowTile& T : tiles) extra += RAD_ROW_COST * T.nrows;
      const int64_t slack = extra / (int64_t)tiles.size();
      if (!cut(ng * RAD_GROUP, slack, 0, 0, (size_t)G, nullptr)) cut(ng * RAD_GROUP, NOCAP, 0, 0, (size_t)G, nullptr);
    } else if (!ok) {
      const int64_t ntarget = std::max<int64_t>(1, std::min<int64_t>(G, (nnz + RAD_MIN_TILE - 1) / RAD_MIN_TILE));
      const int64_t total_cost = nnz + RAD_ROW_COST * (int64_t)arow.size();
      cut(0, 0, total_cost, ntarget, (size_t)-1, nullptr);
    }
  }
  // per row: its tile and first entry within the tile; per tile: stored
  // offset and rows; then the exact halos on the device (the entries
  // sorted by (tile, column): runs = halo facets), splitting over-full tiles
  std::vector<int> tile_of((size_t)nt, 0), rowoff((size_t)nt, 0);
  std::vector<uint32_t> trow(arow.size());
  std::vector<int> rowj0(arow.size());
  std::vector<int> tfirst;
  int64_t stored_total = 0;
  int ntile = 0;
  dbuf<uint32_t> t_halo_tmp;
  dbuf<int> dtile_of, drowoff, dtfirst;
  dbuf<unsigned long long> key2, before;
  dbuf<uint32_t> idx2, flag;
  if (!tiles.empty()) {
    ILG_TRY(dtile_of.alloc(nt));
    ILG_TRY(drowoff.alloc(nt));
    ILG_TRY(key2.alloc(nnz));
    ILG_TRY(idx2.alloc(nnz));
    ILG_TRY(flag.alloc(nnz));
    ILG_TRY(before.alloc(nnz));
    ILG_TRY(t_halo_tmp.alloc(nnz));
  }
  // Tiles much larger than nnz / (4 x blocks) entries are halved as well
  // (when that is above RAD_SPLIT_MIN): with a few tiles per block the
  // longest-first schedule keeps the blocks' loads within a tile of each
  // other.
  const int64_t split_target = std::max<int64_t>(RAD_SPLIT_MIN, nnz / (4 * (int64_t)G));
  for (int iter = 0; !tiles.empty(); ++iter) {
    ntile = (int)tiles.size();
    stored_total = 0;
    int64_t rows_total = 0;
    for (int tid = 0; tid < ntile; ++tid) {
      RowTile& T = tiles[tid];
      T.e0 = stored_total;
      T.r0 = (int)rows_total;
      stored_total += (int64_t)T.lam * RAD_THREADS;
      int64_t j = 0;
      for (int q = 0; q < T.nrows; ++q) {
        const int p = arow[tile_a[tid] + q];
        const int g = (int)order[p];
        tile_of[g] = tid;
        rowoff[g] = (int)j;
        trow[(size_t)rows_total + q] = (uint32_t)p;
        rowj0[(size_t)rows_total + q] = (int)j;
        j += rp[g + 1] - rp[g];
      }
      rows_total += T.nrows;
    }
    ILG_TRY(dtfirst.reserve(ntile + 1));
    ILG_CUDA(cudaMemcpyAsync(dtile_of.p, tile_of.data(), (size_t)nt * 4, cudaMemcpyHostToDevice, s));
    ILG_CUDA(cudaMemcpyAsync(drowoff.p, rowoff.data(), (size_t)nt * 4, cudaMemcpyHostToDevice, s));
    k_tile_keys<<<div_up(nnz, 256), 256, 0, s>>>(dkey.p, nnz, rb, dtile_of.p, key2.p, idx2.p);
    ILG_CUDA(cudaGetLastError());
    int tb = 1;
    while ((1 << tb) < ntile) ++tb;
    ILG_TRY(radix_sort_u64(key2.p, idx2.p, nnz, tb + rb, c.sort, s));
    k_run_flags<<<div_up(nnz, 256), 256, 0, s>>>(key2.p, nnz, flag.p);
    ILG_CUDA(cudaGetLastError());
    ILG_TRY(scan_exclusive_u32_to_u64(flag.p, before.p, nnz, c.scan, s));
    k_halo_runs<<<div_up(nnz, 256), 256, 0, s>>>(key2.p, flag.p, before.p, nnz, rb, t_halo_tmp.p, dtfirst.p);
    ILG_CUDA(cudaGetLastError());
    tfirst.assign((size_t)ntile + 1, 0);
    unsigned long long last_before = 0;
    uint32_t last_flag = 0;
    ILG_CUDA(cudaMemcpyAsync(tfirst.data(), dtfirst.p, (size_t)ntile * 4, cudaMemcpyDeviceToHost, s));
    ILG_CUDA(cudaMemcpyAsync(&last_before, before.p + nnz - 1, 8, cudaMemcpyDeviceToHost, s));
    ILG_CUDA(cudaMemcpyAsync(&last_flag, flag.p + nnz - 1, 4, cudaMemcpyDeviceToHost, s));
    ILG_CUDA(cudaStreamSynchronize(s));
    tfirst[ntile] = (int)(last_before + last_flag);
    bool split = false;
    std::vector<RowTile> nt_tiles;
    std::vector<size_t> nt_a;
    std::vector<int64_t> nt_ne;
    for (int tid = 0; tid < ntile; ++tid) {
      RowTile T = tiles[tid];
      T.h0 = tfirst[tid];
      T.nhalo = tfirst[tid + 1] - tfirst[tid];
      if (T.nhalo < 1) { set_error("row tile without a halo"); return ILG_ERR_CUDA; }
      const bool big = tile_ne[tid] > 2 * split_target;
      if ((T.nhalo <= RAD_HALO && !big) || T.nrows < 2) {
        if (T.nhalo > RAD_HALO) { set_error("row tile halo of %d facets", T.nhalo); return ILG_ERR_CUDA; }
        nt_tiles.push_back(T);
        nt_a.push_back(tile_a[tid]);
        nt_ne.push_back(tile_ne[tid]);
        continue;
      }
      // split at the row where the entries reach half
      split = true;
      const size_t a = tile_a[tid], b = a + T.nrows;
      size_t m = a;
      int64_t ne0 = 0;
      while (m + 1 < b && 2 * (ne0 + rlen(m)) <= tile_ne[tid]) ne0 += rlen(m++);
      if (m == a) ne0 += rlen(m++);
      for (int half = 0; half < 2; ++half) {
        const size_t ha = half ? m : a, hb = half ? b : m;
        const int64_t hne = half ? tile_ne[tid] - ne0 : ne0;
        RowTile H{};
        H.lam = (int)(((hne + RAD_THREADS - 1) / RAD_THREADS + 3) & ~(int64_t)3);
        H.nrows = (int)(hb - ha);
        H.mesh = 0;
        nt_tiles.push_back(H);
        nt_a.push_back(ha);
        nt_ne.push_back(hne);
      }
    }
    tiles.swap(nt_tiles);
    tile_a.swap(nt_a);
    tile_ne.swap(nt_ne);
    if (!split) break;
    if (iter > 40) { set_error("row tiles: halos do not fit after %d splits", iter); return ILG_ERR_CUDA; }
  }
  if (ntile > 0) {
    c.ntiles = ntile;
    c.tile_elems = stored_total;
    c.tiles_h = tiles;
    const int64_t ns = stored_total;
    ILG_TRY(c.tiles.alloc((size_t)ntile + 1));   // and an empty one (k_radiosity64_solo)
    ILG_CUDA(cudaMemsetAsync(c.tiles.p + ntile, 0, sizeof(RowTile), s));
    ILG_TRY(c.t_cf.alloc(ns));
    ILG_TRY(c.t_vhi.alloc(ns));
    ILG_TRY(c.t_vlo.alloc(ns));
    ILG_TRY(c.t_vbf.alloc(ns));
    ILG_TRY(c.t_row.alloc(trow.size()));
    ILG_TRY(c.t_scale.alloc(trow.size()));
    ILG_TRY(c.t_halo.alloc(tfirst[ntile]));
    ILG_TRY(c.t_start.alloc((size_t)ntile * RAD_THREADS));
    ILG_TRY(c.tile_d2.alloc(2 * (size_t)ntile));
    dbuf<uint32_t> dsrc, dfac;
    dbuf<int> drowj0;
    dbuf<int64_t> dne;
    ILG_TRY(dsrc.alloc(ns));
    ILG_TRY(dfac.alloc(ns));
    ILG_TRY(drowj0.alloc(rowj0.size()));
    ILG_TRY(dne.alloc(ntile));
    ILG_CUDA(cudaMemcpyAsync(c.tiles.p, tiles.data(), tiles.size() * sizeof(RowTile), cudaMemcpyHostToDevice, s));
    ILG_CUDA(cudaMemcpyAsync(c.t_row.p, trow.data(), trow.size() * 4, cudaMemcpyHostToDevice, s));
    ILG_CUDA(cudaMemcpyAsync(drowj0.p, rowj0.data(), rowj0.size() * 4, cudaMemcpyHostToDevice, s));
    ILG_CUDA(cudaMemcpyAsync(dne.p, tile_ne.data(), (size_t)ntile * 8, cudaMemcpyHostToDevice, s));
    ILG_CUDA(cudaMemcpyAsync(c.t_halo.p, t_halo_tmp.p, (size_t)tfirst[ntile] * 4, cudaMemcpyDeviceToDevice, s));
    // padding slots: no entry (zero halo index, no source)
    ILG_CUDA(cudaMemsetAsync(c.t_cf.p, 0, (size_t)ns * 2, s));
    ILG_CUDA(cudaMemsetAsync(dsrc.p, 0xff, (size_t)ns * 4, s));
    ILG_CUDA(cudaMemsetAsync(dfac.p, 0, (size_t)ns * 4, s));
    k_tile_slots<<<div_up(nnz, 256), 256, 0, s>>>(key2.p, idx2.p, flag.p, before.p, nnz, rb, dkey.p, dsv.p,
                                                  c.rowptr.p, drowoff.p, c.tiles.p, c.t_cf.p, dsrc.p, dfac.p,
                                                  c.val.p, c.morton_order.p, norms.p, col_sums.p);
    ILG_CUDA(cudaGetLastError());
    k_col_max<<<div_up(nt, 256), 256, 0, s>>>(col_sums.p, nt, norms.p);
    ILG_CUDA(cudaGetLastError());
    k_tile_banks<<<div_up((int64_t)ntile * (RAD_THREADS / 32), 4), 128, 0, s>>>(c.tiles.p, ntile, c.t_cf.p, dsrc.p);
    ILG_CUDA(cudaGetLastError());
    k_tile_starts<<<div_up((int64_t)ntile * RAD_THREADS, 256), 256, 0, s>>>(c.tiles.p, ntile, dne.p, drowj0.p,
                                                                            c.t_start.p);
    ILG_CUDA(cudaGetLastError());
    k_tile_fill<<<div_up(ns, 256), 256, 0, s>>>(dsrc.p, dfac.p, ns, c.val.p, c.row_scale.p, c.t_vhi.p, c.t_vlo.p,
                                                c.t_vbf.p);
    ILG_CUDA(cudaGetLastError());
    k_tile_scale<<<div_up((int64_t)trow.size(), 256), 256, 0, s>>>(c.t_row.p, c.rperm.p, (int)trow.size(),
                                                                  c.row_scale.p, c.t_scale.p);
    ILG_CUDA(cudaGetLastError());
    FNorms norms_h;
    ILG_CUDA(cudaMemcpyAsync(&norms_h, norms.p, sizeof(FNorms), cudaMemcpyDeviceToHost, s));
    ILG_CUDA(cudaStreamSynchronize(s));
    // errors of a change sweep's row sums: a row's entries in its threads' runs,
    // then the runs, and the rounding of the values (see FNorms)
    int64_t chain = 0;
    for (int t = 0; t < ntile; ++t) {
      int64_t longest = 0;
      const int* j0 = rowj0.data() + tiles[t].r0;
      for (int q = 1; q < tiles[t].nrows; ++q) longest = std::max<int64_t>(longest, j0[q] - j0[q - 1]);
      longest = std::max(longest, tile_ne[t] - j0[tiles[t].nrows - 1]);
      const int64_t lam = tiles[t].lam;
      chain = std::max(chain, std::min(longest, lam) + (longest + lam - 1) / lam + 3);
    }
    float max_abs, row_sum;
    std::memcpy(&max_abs, &norms_h.max_abs, 4);
    std::memcpy(&row_sum, &norms_h.row_sum, 4);
    const double col_sum = (double)norms_h.col_sum * ((double)max_abs / 4294967296.0);
    c.rad_err = (float)((double)chain * std::ldexp(1.02, -24) * std::sqrt((double)row_sum * col_sum));
    c.sched_grid = radiosity_grid(ntile, nt);
    ILG_TRY(radiosity_schedule(tiles, c.sched_grid, c.sched_start, c.sched_tile, s));
  } else {
    c.sched_grid = radiosity_grid(0, nt);
    ILG_TRY(radiosity_schedule({}, c.sched_grid, c.sched_start, c.sched_tile, s));
    c.ntiles = 0;
    c.rad_err = 0.f;
    c.tile_elems = 0;
    c.tiles_h.clear();
    ILG_TRY(c.tiles.alloc(1));
    ILG_TRY(c.t_cf.alloc(1));
    ILG_TRY(c.t_vhi.alloc(1));
    ILG_TRY(c.t_vlo.alloc(1));
    ILG_TRY(c.t_vbf.alloc(1));
    ILG_TRY(c.t_row.alloc(1));
    ILG_TRY(c.t_scale.alloc(1));
    ILG_TRY(c.t_halo.alloc(1));
    ILG_TRY(c.t_start.alloc(RAD_THREADS));
    ILG_TRY(c.tile_d2.alloc(2));
  }
  ILG_TRY(c.row_act.alloc(nt));
  ILG_CUDA(cudaMemcpyAsync(c.row_act.p, act.data(), (size_t)nt, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  return ILG_OK;
}

int radiosity_max_meshes() { return RAD_MAX_MESH; }
int radiosity_threads() { return RAD_THREADS; }
// 10 bytes per stored entry (u16 column, f32 hi, f32 lo or bf16): streamed
// when it would not stay in the 126 MB L2 between passes.
int radiosity_l2_stream(int64_t stored) { return stored * 10 > (int64_t)96 << 20 ? 1 : 0; }

float radiosity_res_unit(double tol2) {
  return tol2 > 0.0 ? (float)((double)RES_UNITS / tol2 * (1.0 + 1.0 / 65536.0)) : INFINITY;
}

size_t radiosity_barrier_words(int nmesh) { return RAD_BAR_WORDS1 + 2 * 3 * RES_LEVELS * (size_t)(nmesh > 0 ? nmesh : 1); }

// Cooperative grid size for ntiles tiles (at most the co-resident blocks).
// Both solves launch the same block shape and shared memory, so one grid
// (and one tile schedule) serves either precision.
// A view of few tiles and many facets gets further blocks, without a tile: the
// passes over all facets before and after the sweeps take RAD_ILP of them per
// thread and turn. With one block for the one tile of a body with a single
// small crater (81,920 facets, 134 entries) an FP64 solve took 288 us and a
// one-pass one 391 us, 41 and 37 us with 21 blocks.
int radiosity_grid(int ntiles, int64_t nt) {
  if (radiosity_setup() != ILG_OK || ntiles < 1) return 1;
  const int64_t facets = (nt + RAD_ILP * RAD_THREADS - 1) / (RAD_ILP * RAD_THREADS);
  return (int)std::min<int64_t>((int64_t)std::min(g_rad_per_smm, g_rad_per_sm64) * g_rad_nsm,
                                std::max<int64_t>(ntiles, facets));
}

// Tile cost in stored entries (RAD_ROW_COST per row, RAD_HALO_COST per halo
// facet, plus a fixed cost of one group for the tile's set-up).
int radiosity_schedule(const std::vector<RowTile>& tiles, int grid, dbuf<int>& start, dbuf<int>& order,
                       cudaStream_t s) {
  const int n = (int)tiles.size();
  if (grid < 1) grid = 1;
  std::vector<int> idx(n);
  std::vector<int64_t> cost(n);
  for (int t = 0; t < n; ++t) {
    const RowTile& T = tiles[t];
    idx[t] = t;
    cost[t] = (int64_t)T.lam * RAD_THREADS + RAD_ROW_COST * T.nrows + RAD_HALO_COST * T.nhalo + RAD_GROUP;
  }
  std::sort(idx.begin(), idx.end(), [&](int a, int b) { return cost[a] != cost[b] ? cost[a] > cost[b] : a < b; });
  std::vector<int64_t> load((size_t)grid, 0);
  std::vector<std::vector<int>> lists((size_t)grid);
  // least loaded block: a binary heap of (load, block)
  std::vector<std::pair<int64_t, int>> heap;
  for (int b = 0; b < grid; ++b) heap.push_back({0, b});
  auto cmp = [](const std::pair<int64_t, int>& a, const std::pair<int64_t, int>& b) {
    return a.first != b.first ? a.first > b.first : a.second > b.second;
  };
  std::make_heap(heap.begin(), heap.end(), cmp);
  for (int t : idx) {
    std::pop_heap(heap.begin(), heap.end(), cmp);
    auto& top = heap.back();
    lists[(size_t)top.second].push_back(t);
    top.first += cost[t];
    std::push_heap(heap.begin(), heap.end(), cmp);
  }
  std::vector<int> st((size_t)grid + 1, 0), ord;
  ord.reserve(n);
  for (int b = 0; b < grid; ++b) {
    std::sort(lists[(size_t)b].begin(), lists[(size_t)b].end());
    for (int t : lists[(size_t)b]) ord.push_back(t);
    st[(size_t)b + 1] = (int)ord.size();
  }
  ILG_TRY(start.alloc((size_t)grid + 1));
  ILG_TRY(order.alloc(n > 0 ? (size_t)n : 1));
  ILG_CUDA(cudaMemcpyAsync(start.p, st.data(), st.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  if (n > 0) ILG_CUDA(cudaMemcpyAsync(order.p, ord.data(), ord.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  return ILG_OK;
}

// Launches the cooperative solve for every active mesh of the view with
// tiles. x: result (also the warm start when warm). Per-mesh sweep counts
// and residuals land in the mesh table.
int radiosity_inner(int max_sweeps) { return max_sweeps < 1 ? 1 : (max_sweeps < RAD_INNER ? max_sweeps : RAD_INNER); }

namespace {
// Waits at one grid barrier that expects `expected` arrivals: with
// expected > gridDim.x nobody can open it and every block's wait runs out.
__global__ void k_barrier_probe(unsigned* bar, unsigned expected, int* derr) {
  unsigned gen = 0;
  grid_barrier(bar, expected, gen, derr);
}
// The same for the end of a solo solve's sweep.
__global__ void k_sweep_word_probe(StepView v, unsigned expected) {
  __shared__ SoloShared S;
  if (threadIdx.x == 0) {
    S.mode = 0;
    S.acc = S.prev = 0.f;
  }
  solo_sweep_end(v, S, 0, 1.f, 1.f, 0.f, 1, expected);
}
}  // namespace

// One cooperative launch of `blocks` blocks waiting at a barrier (words: for
// one another's sweep words) that `unreachable` keeps shut, with the poll limit set to `polls` for the
// launch (and restored after it). The wait's outcome is in the view's error
// flags, read by the caller.
int radiosity_barrier_probe(unsigned* bar, int* derr, int blocks, long long polls, int unreachable, bool words,
                            cudaStream_t s) {
  if (blocks < 1 || blocks > 8 || polls < 1) { set_error("invalid barrier probe"); return ILG_ERR_ARG; }
  ILG_CUDA(cudaMemcpyToSymbolAsync(g_barrier_polls, &polls, sizeof(polls), 0, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemsetAsync(bar, 0, (RAD_BAR_WORDS0 + 8 * (blocks + 1)) * sizeof(unsigned), s));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(32);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const unsigned expected = (unsigned)blocks + (unreachable ? 1u : 0u);
  StepView v{};
  v.barrier = bar;
  v.derr = derr;
  const cudaError_t e = words ? cudaLaunchKernelEx(&cfg, k_sweep_word_probe, v, expected)
                              : cudaLaunchKernelEx(&cfg, k_barrier_probe, bar, expected, derr);
  const long long standard = BARRIER_POLLS;
  const cudaError_t e2 = cudaMemcpyToSymbolAsync(g_barrier_polls, &standard, sizeof(standard), 0,
                                                 cudaMemcpyHostToDevice, s);
  ILG_CUDA(e);
  ILG_CUDA(e2);
  ILG_CUDA(cudaStreamSynchronize(s));
  return ILG_OK;
}

int radiosity_launch(const StepView& v, double* x, int warm, int precision, int grid, int inner, bool lagged,
                     cudaStream_t s) {
  ILG_TRY(radiosity_setup());
  if (!v.blk_start || grid != v.sched_grid) {
    set_error("radiosity grid %d has no tile schedule (made for %d blocks)", grid, v.sched_grid);
    return ILG_ERR_ARG;
  }
  // one mesh, at most one tile per block (so the schedule deals them out when
  // there are no more tiles than blocks)
  const bool solo = precision != ILG_PREC_MIXED && v.nmesh == 1 && v.ntiles <= grid && grid <= RAD_MAX_GRID;
  ILG_CUDA(cudaMemsetAsync(v.barrier, 0, (RAD_BAR_WORDS0 + (solo ? 8 * (size_t)grid : 0)) * sizeof(unsigned), s));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(RAD_BLOCK);
  cfg.dynamicSmemBytes = rad_smem_bytes(v.nmesh);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // all blocks co-resident: the grid barrier is safe
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (precision == ILG_PREC_MIXED && lagged)
    ILG_CUDA(cudaLaunchKernelEx(&cfg, k_radiosity_lagged, v, x, warm));
  else if (precision == ILG_PREC_MIXED)
    ILG_CUDA(cudaLaunchKernelEx(&cfg, k_radiosity_mixed, v, x, warm, radiosity_inner(inner)));
  else if (solo)
    ILG_CUDA(cudaLaunchKernelEx(&cfg, k_radiosity64_solo, v, x, warm));
  else
    ILG_CUDA(cudaLaunchKernelEx(&cfg, k_radiosity64, v, x, warm));
  return ILG_OK;
}

}  // namespace ilg
