// gauss_seidel.cu — the reference's fixed-sweep radiosity solve: a forward
// solve of L x = E with L = I - tril(F), then gs_steps Gauss-Seidel sweeps
// x = L^{-1}(E - U x) with U = -triu(F), all in natural row order
// (src/cpp/arma_util.cpp:4-17, src/cpp/illum_cli.cpp:425-433).
//
// Natural-order Gauss-Seidel is a sparse lower-triangular solve per sweep.
// Row i depends on the rows j < i of its lower part. A sweep is one
// cooperative launch: warps take rows in an order in which every row comes
// after the ones it depends on (by dependency level: level(i) = 1 + max
// level of its lower columns, 0 for none), and wait for a row's columns one
// by one. A finished row is published as a 16-byte word of its value and the
// sweep's number, written and read by single 128-bit accesses, so the value
// arrives with its flag and no fence is needed. The lanes of a warp hold 32
// columns' products and add them in order as they become ready: when the
// last column of a row arrives, one addition is left. The first unfinished
// row in the order never waits for a row behind it, so the warps, which are
// all resident, cannot wait for one another in a circle; every wait is
// bounded all the same.
// Each row sums in the reference's order: the upper product accumulated from
// zero over its columns in ascending order (Armadillo's sparse product) of
// the previous sweep's iterate (a launch of its own before the sweep, one
// thread per row), added to E, then the lower terms in ascending column order
// (the forward solve); this file is compiled without fused multiply-adds, so
// the result equals the CPU oracle's restatement of that order bit for bit.
// The levels are found on the device by relaxation (one pass per level, each
// O(nnz)) the first time the mode is used after the form factors change; a
// mesh of 81,920 facets has a few hundred levels.
#include <algorithm>
#include <vector>

#include "internal.cuh"

namespace ilg {

namespace {

// One relaxation pass of the levels: lev[i] = 1 + max lev[j] over the
// row's lower columns (columns are ascending within a row).
__global__ void k_gs_levels(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col, int n, int* lev,
                            int* changed) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int m = 0;
  for (int64_t k = rowptr[i]; k < rowptr[i + 1]; ++k) {
    int j = col[k];
    if (j >= i) break;
    m = max(m, __ldcg(lev + j) + 1);
  }
  if (m != lev[i]) {
    lev[i] = m;
    *changed = 1;
  }
}

// Right-hand side of a step's solve: the frame's direct flux, coupled as
// src/cpp/illum_cli.cpp:415-421 when the mesh follows the reference.
__global__ void k_gs_rhs(StepView v, double* Eg) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= v.nt) return;
  const MeshDesc& M = v.md[0];
  const double d = v.E[e_slot(M.frame) * v.nt + g];
  Eg[g] = M.coupling == ILG_COUPLE_REFERENCE ? (-v.Fsurf[g] + d) : d;
}

// A row's value and the sweep that produced it.
struct __align__(16) GsWord {
  double x;
  unsigned long long sweep;
};
__device__ __forceinline__ GsWord gs_load(const GsWord* p) {
  unsigned long long x, sw;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(x), "=l"(sw) : "l"(p) : "memory");
  GsWord w;
  w.x = __longlong_as_double((long long)x);
  w.sweep = sw;
  return w;
}
__device__ __forceinline__ void gs_store(GsWord* p, double x, unsigned long long sweep) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               ::"l"(p), "l"((unsigned long long)__double_as_longlong(x)), "l"(sweep) : "memory");
}

// Per row: its entries before the first column >= i.
__global__ void k_gs_lower(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col, int n, int* nlow) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t k0 = rowptr[i], k1 = rowptr[i + 1];
  int64_t kd = k0;   // first column >= i
  while (kd < k1 && col[kd] < i) ++kd;
  nlow[i] = (int)(kd - k0);
}

// b = E + U x for the previous sweep's x: U = -triu(F) and L = I - tril(F)
// both hold F's diagonal (zero for computed form factors), so the upper
// product includes it. One thread per row: the sums are serial, and a warp's
// 32 rows share each FP64 instruction.
__global__ void k_gs_upper(const uint32_t* __restrict__ rows, int n, const int64_t* __restrict__ rowptr,
                           const int32_t* __restrict__ col, const double* __restrict__ val,
                           const int* __restrict__ nlow, const double* __restrict__ E,
                           const GsWord* __restrict__ xold, double* __restrict__ b) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int i = (int)rows[t];
  const int64_t k1 = rowptr[i + 1];
  int64_t k = rowptr[i] + nlow[i];
  double u = 0.0;
  for (; k + 8 <= k1; k += 8) {
    double p[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) p[q] = __ldg(val + k + q) * xold[__ldg(col + k + q)].x;
#pragma unroll
    for (int q = 0; q < 8; ++q) u = u + p[q];
  }
  for (; k < k1; ++k) u = u + val[k] * xold[col[k]].x;
  b[i] = E[i] + u;
}

// One sweep's forward solve, x = L^{-1} b, by warps over rows[0, n) (see the
// top of the file). x: published words (sweep number `sweep`), and plain
// values into xout if given. Bound by the longest chain of dependent rows:
// each link is one store's way to L2 and one load's way back; the additions in
// column order keep the FP64 pipe 75% busy meanwhile (359 us per sweep below).
// 81,920 facets, 3.9 M lower entries, 203 levels, a forward solve and one
// sweep: 36.1 ms with a launch per level and one thread per row, 1.0 ms this
// way.
constexpr int GS_THREADS = 256;
constexpr long long GS_POLLS = 1LL << 21;
constexpr int GS_BLOCKS_PER_SM = 2;   // more warps only wait further ahead (1: 7%, 4: 10%, 8: 35% slower)

__global__ void __launch_bounds__(GS_THREADS) k_gs_sweep(const uint32_t* __restrict__ rows, int n,
                                                         const int64_t* __restrict__ rowptr,
                                                         const int32_t* __restrict__ col,
                                                         const double* __restrict__ val, const int* __restrict__ nlow,
                                                         const double* __restrict__ b, GsWord* x,
                                                         unsigned long long sweep, double* xout, int* derr,
                                                         long long polls) {
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (GS_THREADS / 32);
  for (int t = blockIdx.x * (GS_THREADS / 32) + (threadIdx.x >> 5); t < n; t += nw) {
    const int i = (int)__ldg(rows + t);
    const int64_t k0 = __ldg(rowptr + i), k1 = __ldg(rowptr + i + 1);
    const int nl = __ldg(nlow + i);
    double xi = b[i];
    // the forward solve divides by L's diagonal 1 - F_ii (exactly 1 without one)
    const double fii = (k0 + nl < k1 && __ldg(col + k0 + nl) == i) ? __ldg(val + k0 + nl) : 0.0;
    int j = 0;
    double w = 0.0;
    if (lane < nl) {
      j = __ldg(col + k0 + lane);
      w = __ldg(val + k0 + lane);
    }
    for (int c0 = 0; c0 < nl; c0 += 32) {
      const int m = min(32, nl - c0);
      const int jc = j;
      const double wc = w;
      if (c0 + 32 + lane < nl) {   // the next 32 columns, ahead of their use
        j = __ldg(col + k0 + c0 + 32 + lane);
        w = __ldg(val + k0 + c0 + 32 + lane);
      }
      bool ready = lane >= m;
      double p = 0.0;
      int pos = 0;
      for (long long it = 0; pos < m; ++it) {
        if (!ready) {
          const GsWord v = gs_load(x + jc);
          if (v.sweep == sweep) {
            p = wc * v.x;
            ready = true;
          }
        }
        const unsigned waiting = ~__ballot_sync(0xffffffffu, ready);
        const int end = waiting ? min(m, __ffs(waiting) - 1) : m;
        if (pos == 0 && end == 32) {
#pragma unroll
          for (int q = 0; q < 32; ++q) xi = xi + __shfl_sync(0xffffffffu, p, q);
          pos = 32;
        }
        for (; pos < end; ++pos) xi = xi + __shfl_sync(0xffffffffu, p, pos);
        if ((it & 1023) == 1023 || it > polls) {   // give up together with the others, or alone
          int stop = 0;
          if (lane == 0) {
            if (it > polls) atomicExch(&derr[DERR_BARRIER], 1);
            stop = *(volatile int*)&derr[DERR_BARRIER];
          }
          if (__shfl_sync(0xffffffffu, stop, 0)) return;
        }
      }
    }
    if (fii != 0.0) xi = xi / (1.0 - fii);
    if (lane == 0) {
      gs_store(x + i, xi, sweep);
      if (xout) xout[i] = xi;
    }
  }
}

// Squared residual of row i of (I - F) x = E, in the CPU oracle's order.
__global__ void k_gs_residual(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                              const double* __restrict__ val, const double* __restrict__ E,
                              const double* __restrict__ x, int n, double* r2) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double ax = x[i];
  int64_t k = rowptr[i];
  const int64_t k1 = rowptr[i + 1];
  for (; k + 8 <= k1; k += 8) {   // eight products in flight
    double p[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) p[q] = __ldg(val + k + q) * x[__ldg(col + k + q)];
#pragma unroll
    for (int q = 0; q < 8; ++q) ax = ax - p[q];
  }
  for (; k < k1; ++k) ax = ax - val[k] * x[col[k]];
  const double r = ax - E[i];
  r2[i] = r * r;
}

}  // namespace

int gs_residual_launch(const Context& c, const double* E, const double* x, double* r2, cudaStream_t s) {
  k_gs_residual<<<div_up(c.nt, 256), 256, 0, s>>>(c.rowptr.p, c.col.p, c.val.p, E, x, c.nt, r2);
  ILG_CUDA(cudaGetLastError());
  return ILG_OK;
}

int gs_prepare(Context& c) {
  if (c.gs_ready) return ILG_OK;
  if (!c.have_F) { set_error("no form factors"); return ILG_ERR_ARG; }
  const int n = c.nt;
  dbuf<int> lev, flag;
  ILG_TRY(lev.alloc(n));
  ILG_TRY(flag.alloc(1));
  ILG_CUDA(cudaMemsetAsync(lev.p, 0, (size_t)n * sizeof(int), c.stream));
  for (int pass = 0;; ++pass) {
    if (pass > n) { set_error("Gauss-Seidel levels did not settle"); return ILG_ERR_DEVICE; }
    int h = 0;
    ILG_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), c.stream));
    k_gs_levels<<<div_up(n, 256), 256, 0, c.stream>>>(c.rowptr.p, c.col.p, n, lev.p, flag.p);
    ILG_CUDA(cudaGetLastError());
    ILG_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    ILG_CUDA(cudaStreamSynchronize(c.stream));
    if (!h) break;
  }
  // rows in level order (a counting sort of N levels on the host)
  std::vector<int> lh(n);
  ILG_CUDA(cudaMemcpy(lh.data(), lev.p, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost));
  int nlev = n ? *std::max_element(lh.begin(), lh.end()) + 1 : 0;
  std::vector<int> ptr(nlev + 1, 0);
  for (int i = 0; i < n; ++i) ++ptr[lh[i] + 1];
  for (int l = 0; l < nlev; ++l) ptr[l + 1] += ptr[l];
  std::vector<uint32_t> rows(n);
  std::vector<int> fill(ptr.begin(), ptr.end() - 1);
  for (int i = 0; i < n; ++i) rows[fill[lh[i]]++] = (uint32_t)i;
  ILG_TRY(c.gs_rows.alloc(std::max(n, 1)));
  ILG_TRY(c.gs_nlow.alloc(std::max(n, 1)));
  ILG_TRY(c.gs_x.alloc(6 * (size_t)std::max(n, 1)));   // two iterates' words, b, the right-hand side
  k_gs_lower<<<div_up(n, 256), 256, 0, c.stream>>>(c.rowptr.p, c.col.p, n, c.gs_nlow.p);
  ILG_CUDA(cudaGetLastError());
  int dev = 0, nsm = 0, per_sm = 0;
  ILG_CUDA(cudaGetDevice(&dev));
  ILG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  ILG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gs_sweep, GS_THREADS, 0));
  if (per_sm < 1) { set_error("the Gauss-Seidel kernel cannot be resident"); return ILG_ERR_CUDA; }
  c.gs_grid = std::max(1, std::min(nsm * std::min(per_sm, GS_BLOCKS_PER_SM), div_up(n, GS_THREADS / 32)));
  ILG_CUDA(cudaMemcpy(c.gs_rows.p, rows.data(), (size_t)n * sizeof(uint32_t), cudaMemcpyHostToDevice));
  c.gs_lptr = std::move(ptr);
  c.gs_ready = true;
  return ILG_OK;
}

double* gs_rhs(const Context& c) { return c.gs_x.p + 5 * (size_t)c.nt; }

int gs_levels(const Context& c) { return c.gs_ready ? (int)c.gs_lptr.size() - 1 : 0; }

// 1 + gs_steps sweeps from zero of the system with right-hand side E
// (device, facet order); the result into x (device, facet order).
int gs_solve_launch(const Context& c, const double* E, double* x, int gs_steps, cudaStream_t s) {
  const int n = c.nt;
  GsWord* buf[2] = {reinterpret_cast<GsWord*>(c.gs_x.p), reinterpret_cast<GsWord*>(c.gs_x.p) + n};
  double* b = c.gs_x.p + 4 * (size_t)n;
  // no word may carry this solve's sweep numbers (1, 2, ...) from an earlier one
  ILG_CUDA(cudaMemsetAsync(c.gs_x.p, 0, 2 * (size_t)n * sizeof(GsWord), s));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(c.gs_grid);
  cfg.blockDim = dim3(GS_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // all blocks co-resident: warps wait for one another's rows
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  for (int sw = 0; sw <= gs_steps; ++sw) {
    if (sw > 0) {
      k_gs_upper<<<div_up(n, 128), 128, 0, s>>>(c.gs_rows.p, n, c.rowptr.p, c.col.p, c.val.p, c.gs_nlow.p, E,
                                               buf[(sw - 1) & 1], b);
      ILG_CUDA(cudaGetLastError());
    }
    const double* rhs = sw == 0 ? E : b;
    GsWord* out = buf[sw & 1];
    const unsigned long long number = (unsigned long long)sw + 1;
    double* xo = sw == gs_steps ? x : nullptr;
    ILG_CUDA(cudaLaunchKernelEx(&cfg, k_gs_sweep, (const uint32_t*)c.gs_rows.p, n, (const int64_t*)c.rowptr.p,
                                (const int32_t*)c.col.p, (const double*)c.val.p, (const int*)c.gs_nlow.p, rhs, out,
                                number, xo, c.derr.p, c.gs_polls > 0 ? c.gs_polls : GS_POLLS));
  }
  return ILG_OK;
}

// A step's solve (the fused loop's radiosity phase in the fixed-sweep mode).
int gs_step_launch(const Context& c, const StepView& v, int gs_steps, cudaStream_t s) {
  double* Eg = gs_rhs(c);
  k_gs_rhs<<<div_up(c.nt, 256), 256, 0, s>>>(v, Eg);
  ILG_CUDA(cudaGetLastError());
  return gs_solve_launch(c, Eg, v.rad, gs_steps, s);
}

}  // namespace ilg
