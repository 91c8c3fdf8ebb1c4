// primitives.cu — device prefix scan and stable LSD radix sort used by the
// LBVH build (Morton codes) and the form-factor CSR assembly (row/column
// keys). Reduce-then-scan with 2048-element tiles; the radix sort ranks keys
// inside a tile by warp votes on their bits, which keeps it stable.
#include <algorithm>
#include <utility>

#include "common.cuh"

namespace ilg {

namespace {

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

typedef unsigned long long u64;

template <class T>
__global__ void k_tile_sums(const T* __restrict__ in, u64* __restrict__ sums, int64_t n) {
  __shared__ u64 wsum[SCAN_THREADS / 32];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  u64 s = 0;
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    int64_t idx = base + (int64_t)i * SCAN_THREADS + threadIdx.x;
    if (idx < n) s += (u64)in[idx];
  }
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    u64 v = threadIdx.x < SCAN_THREADS / 32 ? wsum[threadIdx.x] : 0;
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
  }
}

// Exclusive scan of one tile (thread t owns SCAN_ITEMS consecutive elements),
// plus the tile's offset.
template <class T>
__global__ void k_tile_scan(const T* __restrict__ in, u64* __restrict__ out, int64_t n,
                            const u64* __restrict__ offsets) {
  __shared__ u64 wsum[SCAN_THREADS / 32];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
  u64 v[SCAN_ITEMS];
  u64 local = 0;
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    int64_t idx = base + i;
    v[i] = idx < n ? (u64)in[idx] : 0;
    local += v[i];
  }
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u64 inc = local;
  for (int o = 1; o < 32; o <<= 1) {
    u64 y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  if (w == 0) {
    u64 x = lane < SCAN_THREADS / 32 ? wsum[lane] : 0;
    u64 xi = x;
    for (int o = 1; o < 32; o <<= 1) {
      u64 y = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += y;
    }
    if (lane < SCAN_THREADS / 32) wsum[lane] = xi - x;
  }
  __syncthreads();
  u64 run = (offsets ? offsets[blockIdx.x] : 0) + wsum[w] + (inc - local);
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    int64_t idx = base + i;
    if (idx < n) out[idx] = run;
    run += v[i];
  }
}

template <class T>
int scan_impl(const T* in, u64* out, int64_t n, ScanScratch& tmp, cudaStream_t s, int depth) {
  if (n <= 0) return ILG_OK;
  int nb = div_up(n, SCAN_TILE);
  if (nb == 1) {
    k_tile_scan<T><<<1, SCAN_THREADS, 0, s>>>(in, out, n, nullptr);
    ILG_CUDA(cudaGetLastError());
    return ILG_OK;
  }
  // level buffers: a (depth 0), b (depth 1), c (depth 2); three levels cover
  // 2048^3 elements.
  dbuf<u64>& sums = depth == 0 ? tmp.a : (depth == 1 ? tmp.b : tmp.c);
  if (depth > 2) { set_error("scan: input too large"); return ILG_ERR_ARG; }
  ILG_TRY(sums.reserve((size_t)nb));
  u64* sp = sums.p;
  k_tile_sums<T><<<nb, SCAN_THREADS, 0, s>>>(in, sp, n);
  ILG_CUDA(cudaGetLastError());
  ILG_TRY(scan_impl<u64>(sp, sp, nb, tmp, s, depth + 1));
  k_tile_scan<T><<<nb, SCAN_THREADS, 0, s>>>(in, out, n, sp);
  ILG_CUDA(cudaGetLastError());
  return ILG_OK;
}

// ---------------------------------------------------------------- radix sort
// Stable LSD sort, 8 bits or less per pass. One launch counts the digits of
// all passes; a pass then reads and writes every key once: a tile ranks its
// keys, publishes its digit counts, adds up those of the tiles before it
// (their own counts, or a running sum where one has been published: the
// decoupled look-back of Merrill and Garland 2016, in the arrangement of
// Adinets and Merrill's one-sweep radix sort, 2022)
// and writes the tile out in digit order through shared memory, in runs of
// about TILE / 128 keys. Tiles take their number from a counter, so the tiles
// that one waits for are running or done. Bound by the ranking and the
// look-back (33% issue, 27% of the copy rate) for large n and by the launches
// for small n: 22 M keys of 34 bits with 32-bit values 1.28 ms, 20,480 keys of
// 63 bits 80 us (a counting, three scan and a scatter launch per pass: 1.46 ms
// and 210 us, the gaps between the launches aside).
constexpr int RS_BINS = 256;
constexpr int RS_PASSES = 8;
constexpr int RS_LOOK = 4;          // tiles looked back at together: their loads overlap (1: 6% slower, 16: 5%)
constexpr int RS_POLLS = 1 << 20;   // look-back polls before a tile counts for itself

template <int THREADS_, int ITEMS_, int BLOCKS_>
struct RadixTile {
  static constexpr int BLOCKS = BLOCKS_, THREADS = THREADS_, ITEMS = ITEMS_, WARPS = THREADS / 32, TILE = THREADS * ITEMS;
  static constexpr size_t SMEM = (size_t)TILE * 12;   // keys and values in digit order
};
typedef RadixTile<512, 12, 2> RadixLarge;   // spills 44 bytes, 96 with values
typedef RadixTile<256, 8, 2> RadixSmall;   // up to RS_SMALL keys: more tiles than a few
constexpr int64_t RS_SMALL = 1 << 19;

// Digit counts of all passes: hist[pass][digit] += counts.
__global__ void __launch_bounds__(256) k_radix_digits(const u64* __restrict__ keys, int64_t n, int passes, int width,
                                                      u64* __restrict__ hist) {
  __shared__ unsigned h[RS_PASSES * RS_BINS];
  const int lane = threadIdx.x & 31;
  const unsigned bins = 1u << width;
  for (int i = threadIdx.x; i < passes * RS_BINS; i += 256) h[i] = 0;
  __syncthreads();
  for (int64_t base = (int64_t)blockIdx.x * 256; base < n; base += (int64_t)gridDim.x * 256) {
    const int64_t i = base + threadIdx.x;
    const bool in = i < n;
    const u64 k = in ? keys[i] : 0ull;
    for (int p = 0; p < passes; ++p) {
      const unsigned d = in ? (unsigned)(k >> (p * width)) & (bins - 1) : bins;
      if (__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {   // neighbours often share their high digits
        if (lane == 0 && in) atomicAdd(&h[p * RS_BINS + d], 32u);
      } else if (in) {
        atomicAdd(&h[p * RS_BINS + d], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * RS_BINS; i += 256)
    if (h[i]) atomicAdd(&hist[i], (u64)h[i]);
}

// A tile's published digit count: value << 8 | code, the code 2 pass + 1 for
// the tile's own count and 2 pass + 2 for the sum up to and with it.
__device__ __forceinline__ void publish(u64* at, u64 value, int code) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(at), "l"((value << 8) | (u64)code) : "memory");
}
__device__ __forceinline__ u64 published(const u64* at) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(at) : "memory");
  return v;
}

// Exclusive scans over the digits of two values, one digit per thread (the
// first RS_BINS threads; every thread calls).
template <int WARPS>
__device__ __forceinline__ void scan_digits(unsigned a, u64 b, unsigned& ea, u64& eb, unsigned* wa, u64* wb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned ia = a;
  u64 ib = b;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned ya = __shfl_up_sync(0xffffffffu, ia, o);
    const u64 yb = __shfl_up_sync(0xffffffffu, ib, o);
    if (lane >= o) {
      ia += ya;
      ib += yb;
    }
  }
  if (lane == 31 && warp < RS_BINS / 32) {
    wa[warp] = ia;
    wb[warp] = ib;
  }
  __syncthreads();
  ea = ia - a;
  eb = ib - b;
  if (warp < RS_BINS / 32)
    for (int w = 0; w < warp; ++w) {
      ea += wa[w];
      eb += wb[w];
    }
}

template <class R, bool HASV>
__global__ void __launch_bounds__(R::THREADS, R::BLOCKS)
k_radix_pass(const u64* __restrict__ kin, const uint32_t* __restrict__ vin, u64* __restrict__ kout,
             uint32_t* __restrict__ vout, int64_t n, int pass, int width, const u64* __restrict__ hist, u64* state,
             unsigned* taken, int polls) {
  constexpr int WARPS = R::WARPS, ITEMS = R::ITEMS, TILE = R::TILE;
  extern __shared__ u64 rs_keys[];                              // [TILE], then the values
  uint32_t* rs_vals = reinterpret_cast<uint32_t*>(rs_keys + TILE);
  __shared__ unsigned wcnt[WARPS][RS_BINS];
  __shared__ int64_t goff[RS_BINS];                             // digit's place in the output minus in the tile
  __shared__ unsigned wa[RS_BINS / 32], tile_s;
  __shared__ u64 wb[RS_BINS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, shift = pass * width;
  const unsigned mask = (1u << width) - 1u, lt = (1u << lane) - 1u;
  if (threadIdx.x == 0) tile_s = atomicAdd(taken, 1u);
  for (int i = threadIdx.x; i < WARPS * RS_BINS; i += R::THREADS) (&wcnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t tile = tile_s, first = tile * TILE;
  const int count = (int)min((int64_t)TILE, n - first);
  u64 k[ITEMS];
  uint32_t v[ITEMS];
  unsigned rank[ITEMS];
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const int i = warp * (32 * ITEMS) + it * 32 + lane;
    k[it] = i < count ? kin[first + i] : ~0ull;
    if (HASV) v[it] = i < count ? vin[first + i] : 0u;
  }
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const bool in = warp * (32 * ITEMS) + it * 32 + lane < count;
    const unsigned d = in ? (unsigned)(k[it] >> shift) & mask : mask + 1;
    unsigned peers = 0xffffffffu;   // lanes with the same digit (a vote per bit: a third of match_any's time)
    for (int b = 0; b <= width; ++b) {
      const bool one = (d >> b) & 1;
      const unsigned m = __ballot_sync(0xffffffffu, one);
      peers &= one ? m : ~m;
    }
    const unsigned before = peers & lt;
    const unsigned base = in ? wcnt[warp][d] : 0u;
    __syncwarp();
    if (in && before == 0) wcnt[warp][d] = base + __popc(peers);
    __syncwarp();
    rank[it] = base + __popc(before);
  }
  __syncthreads();
  const int d = threadIdx.x;
  unsigned cnt = 0;
  u64* mine = state + tile * RS_BINS + d;
  if (d < RS_BINS) {
    for (int w = 0; w < WARPS; ++w) {
      const unsigned c = wcnt[w][d];
      wcnt[w][d] = cnt;
      cnt += c;
    }
    publish(mine, cnt, 2 * pass + (tile == 0 ? 2 : 1));
  }
  unsigned loc;
  u64 gbase;
  scan_digits<WARPS>(cnt, d < RS_BINS ? hist[d] : 0ull, loc, gbase, wa, wb);
  // look-back
  u64 before = 0;
  bool lost = false;
  if (d < RS_BINS && tile > 0) {
    int64_t p = tile - 1;
    int left = polls;
    for (bool done = false; !done;) {
      u64 w[RS_LOOK];
      bool open = true;
#pragma unroll
      for (int q = 0; q < RS_LOOK; ++q) w[q] = p - q >= 0 ? published(state + (p - q) * RS_BINS + d) : 0ull;
#pragma unroll
      for (int q = 0; q < RS_LOOK; ++q) {
        const int code = (int)(w[q] & 255ull) - 2 * pass;
        open = open && !done && (code == 1 || code == 2);
        if (open) {
          before += w[q] >> 8;
          --p;
          done = code == 2;
        }
      }
      if (!done && --left < 0) {
        lost = true;
        done = true;
      }
    }
  }
  if (__syncthreads_or(lost)) {   // count the keys before the tile directly
    for (int i = threadIdx.x; i < RS_BINS; i += R::THREADS) goff[i] = 0;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < first; i += R::THREADS)
      atomicAdd(reinterpret_cast<u64*>(&goff[(unsigned)(kin[i] >> shift) & mask]), 1ull);
    __syncthreads();
    if (d < RS_BINS) before = (u64)goff[d];
  }
  if (d < RS_BINS) {
    if (tile > 0) publish(mine, before + cnt, 2 * pass + 2);
    goff[d] = (int64_t)(gbase + before) - (int64_t)loc;
    for (int w = 0; w < WARPS; ++w) wcnt[w][d] += loc;
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    if (warp * (32 * ITEMS) + it * 32 + lane < count) {
      const unsigned at = wcnt[warp][(unsigned)(k[it] >> shift) & mask] + rank[it];
      rs_keys[at] = k[it];
      if (HASV) rs_vals[at] = v[it];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < count; i += R::THREADS) {
    const u64 key = rs_keys[i];
    const int64_t at = goff[(unsigned)(key >> shift) & mask] + i;
    kout[at] = key;
    if (HASV) vout[at] = rs_vals[i];
  }
}

template <class R>
int radix_passes(u64* keys, uint32_t* vals, int64_t n, int bits, SortScratch& tmp, cudaStream_t s, int polls) {
  const int64_t tiles = (n + R::TILE - 1) / R::TILE;
  const int passes = (bits + 7) / 8, width = (bits + passes - 1) / passes;
  // digit counts, tile counters and tile states, all zero at first
  const size_t head = (size_t)passes * RS_BINS + RS_PASSES;
  ILG_TRY(tmp.hist.reserve(head + (size_t)tiles * RS_BINS));
  u64* hist = tmp.hist.p;
  unsigned* taken = reinterpret_cast<unsigned*>(hist + (size_t)passes * RS_BINS);
  u64* state = hist + head;
  ILG_CUDA(cudaMemsetAsync(hist, 0, (head + (size_t)tiles * RS_BINS) * 8, s));
  k_radix_digits<<<(int)std::min<int64_t>((n + 2047) / 2048, 152 * 8), 256, 0, s>>>(keys, n, passes, width, hist);
  ILG_CUDA(cudaGetLastError());
  auto kern = vals ? k_radix_pass<R, true> : k_radix_pass<R, false>;
  ILG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::SMEM));
  u64 *ka = keys, *kb = tmp.keys_alt.p;
  uint32_t *va = vals, *vb = vals ? tmp.vals_alt.p : nullptr;
  for (int p = 0; p < passes; ++p) {
    kern<<<(int)tiles, R::THREADS, R::SMEM, s>>>(ka, va, kb, vb, n, p, width, hist + (size_t)p * RS_BINS, state,
                                                 taken + p, polls);
    ILG_CUDA(cudaGetLastError());
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (passes & 1) {
    ILG_CUDA(cudaMemcpyAsync(keys, ka, (size_t)n * 8, cudaMemcpyDeviceToDevice, s));
    if (vals) ILG_CUDA(cudaMemcpyAsync(vals, va, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
  }
  return ILG_OK;
}

}  // namespace

int scan_exclusive_u32_to_u64(const uint32_t* in, u64* out, int64_t n, ScanScratch& tmp, cudaStream_t s) {
  return scan_impl<uint32_t>(in, out, n, tmp, s, 0);
}

int radix_sort_u64(u64* keys, uint32_t* vals, int64_t n, int bits, SortScratch& tmp, cudaStream_t s, int polls) {
  if (polls < 0) polls = RS_POLLS;
  if (n <= 1 || bits <= 0) return ILG_OK;
  ILG_TRY(tmp.keys_alt.reserve((size_t)n));
  if (vals) ILG_TRY(tmp.vals_alt.reserve((size_t)n));
  return n <= RS_SMALL ? radix_passes<RadixSmall>(keys, vals, n, bits, tmp, s, polls)
                       : radix_passes<RadixLarge>(keys, vals, n, bits, tmp, s, polls);
}

}  // namespace ilg
