// bvh.cu — LBVH build (Morton codes, radix sort, Karras hierarchy, bottom-up
// boxes), closest-hit / any-hit traversal, the horizon bisection kernel
// (src/cpp/illum.cpp:274-363) and the visibility + form-factor assembly
// (src/cpp/illum.cpp:31-237). Compiled with -fmad=false: the ray origins,
// directions and the mt64 predicate must round exactly as geom.h specifies.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

#include "geom.h"
#include "internal.cuh"

namespace ilg {

namespace {

typedef unsigned long long u64;

__device__ __forceinline__ f3 f3of(float4 a) { return mk(a.x, a.y, a.z); }

// ------------------------------------------------------------------ build
__global__ void k_prepare(const float* __restrict__ verts, const int32_t* __restrict__ tris,
                          const float* __restrict__ normals, int nt, float4* tri_o, float4* cen, float4* nrm,
                          double* area, double* frame, float4* frame32) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const float* a = verts + 3 * (int64_t)tris[3 * t];
  const float* b = verts + 3 * (int64_t)tris[3 * t + 1];
  const float* d = verts + 3 * (int64_t)tris[3 * t + 2];
  f3 v0 = mk(a[0], a[1], a[2]), v1 = mk(b[0], b[1], b[2]), v2 = mk(d[0], d[1], d[2]);
  f3 c = tri_centroid(v0, v1, v2);
  f3 n = normals ? mk(normals[3 * t], normals[3 * t + 1], normals[3 * t + 2]) : tri_normal(v0, v1, v2);
  float r = tri_radius(v0, v1, v2, c);
  tri_o[3 * t] = make_float4(v0.x, v0.y, v0.z, 0.f);
  tri_o[3 * t + 1] = make_float4(v1.x, v1.y, v1.z, 0.f);
  tri_o[3 * t + 2] = make_float4(v2.x, v2.y, v2.z, 0.f);
  cen[t] = make_float4(c.x, c.y, c.z, r);
  nrm[t] = make_float4(n.x, n.y, n.z, 0.f);
  area[t] = tri_area(v0, v1, v2);
  frame3 F = tri_frame(v0, v1, n);
  double* fr = frame + 9 * (int64_t)t;
  fr[0] = F.b.x; fr[1] = F.b.y; fr[2] = F.b.z;
  fr[3] = F.t.x; fr[4] = F.t.y; fr[5] = F.t.z;
  fr[6] = F.n.x; fr[7] = F.n.y; fr[8] = F.n.z;
  frame32[3 * t] = make_float4((float)F.b.x, (float)F.b.y, (float)F.b.z, 0.f);
  frame32[3 * t + 1] = make_float4((float)F.t.x, (float)F.t.y, (float)F.t.z, 0.f);
  frame32[3 * t + 2] = make_float4((float)F.n.x, (float)F.n.y, (float)F.n.z, 0.f);
}

__device__ __forceinline__ u64 spread3(u64 x) {   // 21 bits -> every third bit
  x &= 0x1fffffull;
  x = (x | (x << 32)) & 0x1f00000000ffffull;
  x = (x | (x << 16)) & 0x1f0000ff0000ffull;
  x = (x | (x << 8)) & 0x100f00f00f00f00full;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

__global__ void k_morton(const float4* __restrict__ cen, int nt, float3 lo, float3 inv_ext, u64* keys,
                         uint32_t* vals) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  float4 c = cen[t];
  float q = 2097151.0f;
  float x = fminf(fmaxf((c.x - lo.x) * inv_ext.x, 0.f), 1.f) * q;
  float y = fminf(fmaxf((c.y - lo.y) * inv_ext.y, 0.f), 1.f) * q;
  float z = fminf(fmaxf((c.z - lo.z) * inv_ext.z, 0.f), 1.f) * q;
  keys[t] = (spread3((u64)x) << 2) | (spread3((u64)y) << 1) | spread3((u64)z);
  vals[t] = (uint32_t)t;
}

__device__ __forceinline__ int delta(const u64* keys, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  u64 a = keys[i], b = keys[j];
  if (a == b) return 64 + __clz((unsigned)(i ^ j));
  return __clzll((long long)(a ^ b));
}

// Karras (2012) radix-tree construction: internal node i covers a key range
// and splits it at the highest differing bit. Child codes: >= 0 internal,
// ~k leaf k. parent arrays: [0, n-1) internal, [n-1, 2n-1) leaves. range: the
// leaves [lo, hi] below each internal node.
__global__ void k_karras(const u64* __restrict__ keys, int n, int2* child, int* parent, int2* range) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = delta(keys, n, i, j);
  int s = 0;
  int t = l;
  do {
    t = (t + 1) >> 1;
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  int g = i + s * d + (d < 0 ? -1 : 0);
  int lo = i < j ? i : j, hi = i < j ? j : i;
  int left = (lo == g) ? ~g : g;
  int right = (hi == g + 1) ? ~(g + 1) : (g + 1);
  child[i] = make_int2(left, right);
  range[i] = make_int2(lo, hi);
  parent[left >= 0 ? left : (n - 1) + ~left] = i;
  parent[right >= 0 ? right : (n - 1) + ~right] = i;
}

// Leaf boxes (inflated by pad) and bottom-up union: the second child to
// arrive at a node computes its box (atomic arrival counter, no waiting).
__global__ void k_refit(const float4* __restrict__ tri_o, const uint32_t* __restrict__ order, int n,
                        const int2* __restrict__ child, const int* __restrict__ parent, float4* box_lo,
                        float4* box_hi, int* flags, float pad, float4* tri_s, int* depth_out) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int t = (int)order[k];
  float4 a = tri_o[3 * t], b = tri_o[3 * t + 1], c = tri_o[3 * t + 2];
  tri_s[3 * k] = make_float4(a.x, a.y, a.z, __int_as_float(t));
  // the edges' l1 norms, for the error bounds of the ray test
  const f3 v0 = f3of(a);
  tri_s[3 * k + 1] = make_float4(b.x, b.y, b.z, l1(sub(f3of(b), v0)));
  tri_s[3 * k + 2] = make_float4(c.x, c.y, c.z, l1(sub(f3of(c), v0)));
  float4 lo = make_float4(fminf(fminf(a.x, b.x), c.x) - pad, fminf(fminf(a.y, b.y), c.y) - pad,
                          fminf(fminf(a.z, b.z), c.z) - pad, 0.f);
  float4 hi = make_float4(fmaxf(fmaxf(a.x, b.x), c.x) + pad, fmaxf(fmaxf(a.y, b.y), c.y) + pad,
                          fmaxf(fmaxf(a.z, b.z), c.z) + pad, 0.f);
  int slot = (n - 1) + k;
  box_lo[slot] = lo;
  box_hi[slot] = hi;
  if (n == 1) return;
  int depth = 0;
  int p = parent[slot];
  while (p >= 0) {
    __threadfence();
    if (atomicAdd(&flags[p], 1) == 0) return;
    int2 ch = child[p];
    int sl = ch.x >= 0 ? ch.x : (n - 1) + ~ch.x;
    int sr = ch.y >= 0 ? ch.y : (n - 1) + ~ch.y;
    float4 l0 = __ldcg(&box_lo[sl]), h0 = __ldcg(&box_hi[sl]);
    float4 l1 = __ldcg(&box_lo[sr]), h1 = __ldcg(&box_hi[sr]);
    box_lo[p] = make_float4(fminf(l0.x, l1.x), fminf(l0.y, l1.y), fminf(l0.z, l1.z), 0.f);
    box_hi[p] = make_float4(fmaxf(h0.x, h1.x), fmaxf(h0.y, h1.y), fmaxf(h0.z, h1.z), 0.f);
    ++depth;
    p = parent[p];
  }
  atomicMax(depth_out, depth);
}

// Morton position of each facet, and the longest path from a leaf to the
// root (whole warps).
__global__ void k_leaf_rank(const uint32_t* __restrict__ order, const int* __restrict__ parent, int n, uint32_t* rank,
                            int* longest) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  int d = 0;
  if (k < n) {
    rank[order[k]] = (uint32_t)k;
    for (int p = parent[(n - 1) + k]; p >= 0; p = parent[p]) ++d;
  }
  d = __reduce_max_sync(0xffffffffu, d);
  if ((threadIdx.x & 31) == 0) atomicMax(longest, d);
}

// Oriented slabs. A patch of surface that is tilted against the axes fills
// its box's diagonal only, so rays that graze the surface, as horizon and
// visibility rays do, pass through the boxes of patches far below them. Each
// node therefore also has a slab dmin <= m . x <= dmax around its triangles,
// m the direction of their summed area vectors: as thin as the patch is
// rough, and a plane for a leaf. Nodes of more than SLAB_LEAVES leaves keep
// an unbounded one. slab_m: (m, dmin), slab_d: dmax, by slot (internal
// nodes, then leaves); widened by `pad` on both sides. One warp per node.
constexpr int SLAB_LEAVES = 1024;

__global__ void k_slabs(const float4* __restrict__ tri_s, const int2* __restrict__ range, int n, float pad,
                        float4* slab_m, float* slab_d) {
  const int lane = threadIdx.x & 31;
  const int slot = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);   // leaves: one thread each, below
  const int ni = n - 1;
  const int leaf_warps = (n + 31) / 32;
  if (slot < leaf_warps) {
    const int k = slot * 32 + lane;
    if (k >= n) return;
    const f3 v0 = f3of(tri_s[3 * (int64_t)k]), v1 = f3of(tri_s[3 * (int64_t)k + 1]),
             v2 = f3of(tri_s[3 * (int64_t)k + 2]);
    const f3 c = cross(sub(v1, v0), sub(v2, v0));
    const float l = len(c);
    f3 m = mk(0.f, 0.f, 0.f);
    float lo = -3e38f, hi = 3e38f;
    if (l > 0.f && l < 3e38f) {
      m = mk(c.x / l, c.y / l, c.z / l);
      const float a = dot(m, v0), b = dot(m, v1), d = dot(m, v2);
      lo = fminf(a, fminf(b, d)) - pad;
      hi = fmaxf(a, fmaxf(b, d)) + pad;
    }
    slab_m[ni + k] = make_float4(m.x, m.y, m.z, lo);
    slab_d[ni + k] = hi;
    return;
  }
  const int i = slot - leaf_warps;
  if (i >= ni) return;
  const int2 r = range[i];
  f3 m = mk(0.f, 0.f, 0.f);
  float lo = -3e38f, hi = 3e38f;
  if (r.y - r.x < SLAB_LEAVES) {
    f3 sum = mk(0.f, 0.f, 0.f);
    for (int k = r.x + lane; k <= r.y; k += 32) {
      const f3 v0 = f3of(tri_s[3 * (int64_t)k]), v1 = f3of(tri_s[3 * (int64_t)k + 1]),
               v2 = f3of(tri_s[3 * (int64_t)k + 2]);
      sum = add(sum, cross(sub(v1, v0), sub(v2, v0)));
    }
    for (int o = 16; o; o >>= 1)
      sum = add(sum, mk(__shfl_xor_sync(0xffffffffu, sum.x, o), __shfl_xor_sync(0xffffffffu, sum.y, o),
                        __shfl_xor_sync(0xffffffffu, sum.z, o)));
    const float l = len(sum);
    if (l > 0.f && l < 3e38f) {
      m = mk(sum.x / l, sum.y / l, sum.z / l);
      lo = 3e38f;
      hi = -3e38f;
      for (int k = r.x + lane; k <= r.y; k += 32)
        for (int q = 0; q < 3; ++q) {
          const float a = dot(m, f3of(tri_s[3 * (int64_t)k + q]));
          lo = fminf(lo, a);
          hi = fmaxf(hi, a);
        }
      for (int o = 16; o; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      lo -= pad;
      hi += pad;
    }
  }
  if (lane == 0) {
    slab_m[i] = make_float4(m.x, m.y, m.z, lo);
    slab_d[i] = hi;
  }
}

// Node record, NODE_W float4: both children's boxes, their slabs, and
// (left dmax, right dmax, left code, right code).
__global__ void k_pack_nodes(const int2* __restrict__ child, const float4* __restrict__ box_lo,
                             const float4* __restrict__ box_hi, const float4* __restrict__ slab_m,
                             const float* __restrict__ slab_d, int n, float4* nodes) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int2 ch = child[i];
  int sl = ch.x >= 0 ? ch.x : (n - 1) + ~ch.x;
  int sr = ch.y >= 0 ? ch.y : (n - 1) + ~ch.y;
  float4 l0 = box_lo[sl], h0 = box_hi[sl], l1 = box_lo[sr], h1 = box_hi[sr];
  float4* nd = nodes + (int64_t)NODE_W * i;
  nd[0] = make_float4(l0.x, l0.y, l0.z, h0.x);
  nd[1] = make_float4(h0.y, h0.z, l1.x, l1.y);
  nd[2] = make_float4(l1.z, h1.x, h1.y, h1.z);
  nd[3] = slab_m[sl];
  nd[4] = slab_m[sr];
  nd[5] = make_float4(slab_d[sl], slab_d[sr], __int_as_float(ch.x), __int_as_float(ch.y));
}

// ------------------------------------------------------------------ traversal
struct NodeBoxes { f3 llo, lhi, rlo, rhi; int left, right; };

__device__ __forceinline__ NodeBoxes load_node(const float4* __restrict__ nodes, int i) {
  const float4* nd = nodes + (int64_t)NODE_W * i;
  float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2), d = __ldg(nd + 5);
  NodeBoxes nb;
  nb.llo = mk(a.x, a.y, a.z); nb.lhi = mk(a.w, b.x, b.y);
  nb.rlo = mk(b.z, b.w, c.x); nb.rhi = mk(c.y, c.z, c.w);
  nb.left = __float_as_int(d.z); nb.right = __float_as_int(d.w);
  return nb;
}

// Closest hit under geom.h's mt64 (smallest t, ties to the smaller original
// index). Returns the original facet index or -1; sets *err on stack
// overflow; *t_out (if given) receives the hit's mt64 t.
//
// The FP64 test runs only where single precision cannot decide. A leaf that
// mt32_classify calls a certain hit comes with an enclosure [tlo, thi] of its
// mt64 t; the best hit so far is kept as such an enclosure [blo, bhi] and
// compared by intervals: tlo > bhi means certainly farther, thi < blo
// certainly closer (so no tie is possible). Only when the intervals overlap,
// or the leaf is undecided, are the exact t of both hits computed and
// compared with the tie rule. The argmin of (t, index) over all mt64 hits is
// therefore the one an all-FP64 traversal finds; rays aimed at facet
// centroids almost never need the FP64 path.
__device__ int trace_closest(const float4* __restrict__ nodes, const float4* __restrict__ tri_s, int root,
                             f3 o, f3 d, double* t_out, int* err) {
  ray_inv ri = make_ray_inv(o, d);
  int besti = -1, bk = 0;
  float blo = 3.0e38f, bhi = 3.0e38f;   // encloses the best hit's mt64 t
  double bt = 0.0;                      // that t, once computed (bex)
  bool bex = false;
  float tmaxf = 3.0e38f;
  int stack[TRACE_STACK];
  int sp = 0;
  int node = root;
  for (;;) {
    if (node < 0) {
      int k = ~node;
      float4 a = __ldg(&tri_s[3 * k]), b = __ldg(&tri_s[3 * k + 1]), c = __ldg(&tri_s[3 * k + 2]);
      f3 v0 = f3of(a), v1 = f3of(b), v2 = f3of(c);
      int idx = __float_as_int(a.w);
      float tlo, thi;
      int cls = mt32_classify(o, d, v0, v1, v2, &tlo, &thi);
      bool take = false;
      if (cls == 1 && (besti < 0 || thi < blo)) {
        take = true;                    // certainly the closest so far
        bex = false;
        blo = tlo;
        bhi = thi;
      } else if (cls == 2 || (cls == 1 && !(tlo > bhi))) {
        double th;
        if (mt64(o, d, v0, v1, v2, &th)) {
          if (besti >= 0 && !bex) {     // exact t of the current best
            float4 ba = __ldg(&tri_s[3 * bk]), bb = __ldg(&tri_s[3 * bk + 1]), bc = __ldg(&tri_s[3 * bk + 2]);
            bex = mt64(o, d, f3of(ba), f3of(bb), f3of(bc), &bt);
          }
          if (besti < 0 || th < bt || (th == bt && idx < besti)) {
            take = true;
            bex = true;
            bt = th;
            float tf = (float)th;
            blo = tf * (1.0f - 2.4e-7f);
            bhi = tf * (1.0f + 2.4e-7f) + 1e-37f;
          }
        }
      }
      if (take) {
        besti = idx;
        bk = k;
        tmaxf = bhi * 1.000001f + 1e-30f;
      }
      if (sp == 0) break;
      node = stack[--sp];
      continue;
    }
    NodeBoxes nb = load_node(nodes, node);
    float tl = slab(ri, nb.llo, nb.lhi, tmaxf);
    float tr = slab(ri, nb.rlo, nb.rhi, tmaxf);
    bool hl = tl >= 0.f, hr = tr >= 0.f;
    if (hl && hr) {
      if (sp == TRACE_STACK) { atomicExch(err, 1); break; }
      if (tl <= tr) { stack[sp++] = nb.right; node = nb.left; }
      else { stack[sp++] = nb.left; node = nb.right; }
    } else if (hl) {
      node = nb.left;
    } else if (hr) {
      node = nb.right;
    } else {
      if (sp == 0) break;
      node = stack[--sp];
    }
  }
  if (t_out) {
    if (besti >= 0 && !bex) {
      float4 ba = __ldg(&tri_s[3 * bk]), bb = __ldg(&tri_s[3 * bk + 1]), bc = __ldg(&tri_s[3 * bk + 2]);
      mt64(o, d, f3of(ba), f3of(bb), f3of(bc), &bt);
    }
    *t_out = besti >= 0 ? bt : 1e300;
  }
  return besti;
}

// Any hit under mt64.
__device__ bool trace_any(const float4* __restrict__ nodes, const float4* __restrict__ tri_s, int root, f3 o,
                          f3 d, int* err) {
  ray_inv ri = make_ray_inv(o, d);
  int stack[TRACE_STACK];
  int sp = 0;
  int node = root;
  for (;;) {
    if (node < 0) {
      int k = ~node;
      float4 a = __ldg(&tri_s[3 * k]), b = __ldg(&tri_s[3 * k + 1]), c = __ldg(&tri_s[3 * k + 2]);
      f3 v0 = f3of(a), v1 = f3of(b), v2 = f3of(c);
      float tlo, thi;
      int cls = mt32_classify(o, d, v0, v1, v2, &tlo, &thi);
      if (cls == 1) return true;
      if (cls == 2) {
        double th;
        if (mt64(o, d, v0, v1, v2, &th)) return true;
      }
      if (sp == 0) return false;
      node = stack[--sp];
      continue;
    }
    NodeBoxes nb = load_node(nodes, node);
    float tl = slab(ri, nb.llo, nb.lhi, 3.0e38f);
    float tr = slab(ri, nb.rlo, nb.rhi, 3.0e38f);
    bool hl = tl >= 0.f, hr = tr >= 0.f;
    if (hl && hr) {
      if (sp == TRACE_STACK) { atomicExch(err, 1); return false; }
      if (tl <= tr) { stack[sp++] = nb.right; node = nb.left; }
      else { stack[sp++] = nb.left; node = nb.right; }
    } else if (hl) {
      node = nb.left;
    } else if (hr) {
      node = nb.right;
    } else {
      if (sp == 0) return false;
      node = stack[--sp];
    }
  }
}

__global__ void k_trace(const float4* __restrict__ nodes, const float4* __restrict__ tri_s, int root, int nrays,
                        const float* __restrict__ orig, const float* __restrict__ dir, int any_hit, int32_t* hit,
                        double* thit, int* derr) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrays) return;
  f3 o = mk(orig[3 * r], orig[3 * r + 1], orig[3 * r + 2]);
  f3 d = mk(dir[3 * r], dir[3 * r + 1], dir[3 * r + 2]);
  if (any_hit) {
    hit[r] = trace_any(nodes, tri_s, root, o, d, &derr[DERR_STACK]) ? 1 : -1;
    thit[r] = -1.0;
  } else {
    double t;
    int h = trace_closest(nodes, tri_s, root, o, d, &t, &derr[DERR_STACK]);
    hit[r] = h;
    thit[r] = h >= 0 ? t : -1.0;
  }
}

// ------------------------------------------------------------------ renderer
// One closest-hit ray per pixel of src/cpp/illum_renderer_cli.cpp:228-276:
// mode 0 orthographic from direction (az, el) at distance 1.1 r_model,
// mode 1 equal-area cylindrical map (rays from a sphere of radius
// 1.1 r_model towards the model centre). out: facet index or -1.
struct RenderCam {
  int mode, width, height;
  double rad, aspect, az, el;
  float px, py, pz, ex, ey, ez, ux, uy, uz, rx, ry, rz;   // orthographic camera (float, as Vector3)
  float cx, cy, cz;                                     // model centre
};

__global__ void k_render(const float4* __restrict__ nodes, const float4* __restrict__ tri_s, int root, RenderCam cam,
                         int32_t* out, int* derr) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (int64_t)cam.width * cam.height) return;
  const int i = (int)(k / cam.width), j = (int)(k % cam.width);
  f3 o, d;
  if (cam.mode == 0) {
    double y_eye = (2.0 * (1.0 - (double)i / (cam.height - 1)) - 1.0) * cam.rad;
    double x_eye = (2.0 * (double)j / (cam.width - 1) - 1.0) * cam.aspect * cam.rad;
    float ye = (float)y_eye, xe = (float)x_eye;
    o = mk(cam.px + ye * cam.ux + xe * cam.rx, cam.py + ye * cam.uy + xe * cam.ry, cam.pz + ye * cam.uz + xe * cam.rz);
    d = mk(cam.ex, cam.ey, cam.ez);
  } else {
    const double PI_D = 3.141592653589793;
    double theta = asin(2.0 * (double)(i + 1) / (cam.height + 1) - 1.0) - cam.el;
    double phi = 2.0 * PI_D * (double)j / cam.width - cam.az;
    f3 p = mk((float)(cam.rad * cos(phi) * sin(theta)), (float)(cam.rad * sin(phi) * sin(theta)),
              (float)(cam.rad * cos(theta)));
    d = normalize(mk(-p.x, -p.y, -p.z));
    o = mk(p.x + cam.cx, p.y + cam.cy, p.z + cam.cz);
  }
  out[k] = trace_closest(nodes, tri_s, root, o, d, nullptr, &derr[DERR_STACK]);
}

// ------------------------------------------------------------------ rays from a facet
// Horizon and visibility rays start at a facet (its centroid, offset along
// the normal), and a warp's rays all start at the same one. The boxes on the
// path from the root to that facet's leaf contain the origin, so a traversal
// from the root would test and enter each of them for every ray. Instead the
// warp keeps the path's siblings (the other child at every node, deepest
// first; together with the leaf itself they cover the whole tree) in shared
// memory, each ray tests them in one loop that all lanes run together
// (broadcast reads, no stack), and traverses only the subtrees it enters,
// nearest first: the deepest siblings surround the origin.
//
// Where the lanes differ, node visits and triangle tests alternate in phases:
// lanes at internal nodes step until few are left, then the lanes that have
// reached a leaf test it together, so that neither the visits nor the
// (longer) triangle test runs for a few lanes at a time; lanes whose ray has
// ended wait until enough of them can begin their next ray together. What
// this gave stands at k_horizons and k_vis_rays. Tried and slower: path
// entries taken in a phase of their own (2%), three-operand min / max in the
// box test (5%), a branch around the slab test (4%).
constexpr int PATH_MOST = 64;              // bits of a lane's mask of path entries
constexpr int LANE_IDLE = 0x7fffffff;      // no node left (codes of internal nodes are < 2^31 - 1)
// Lanes at internal nodes below which pending leaves are tested, and idle
// lanes from which new rays begin (form factors of 81,920 facets: 8..20 lanes
// with 4..28 idle ones took 268..145 ms; horizon maps are 1% faster with 12
// than with 16).
constexpr int NODE_LANES = 12;
constexpr int REFILL_LANES = 28;

struct PathEntry {
  float4 a, b, c;   // box (lo.xyz, hi.x), (hi.y, hi.z, child code as int bits, dmin - m . o), slab (m, dmax - m . o)
};

// The entry of the whole tree: no bounds.
__device__ __forceinline__ void whole_tree(PathEntry& e, int root) {
  e.a = make_float4(-3e38f, -3e38f, -3e38f, 3e38f);
  e.b = make_float4(3e38f, 3e38f, __int_as_float(root), -3e38f);
  e.c = make_float4(0.f, 0.f, 0.f, 3e38f);
}

// Path of leaf k (position in Morton order) into path[]: its siblings from
// the deepest to the root's other child. Whole warp; returns their number,
// at most `entries`: a longer path (more than PATH_MOST levels) ends with the
// whole tree in place of the rest. o: the rays' origin.
__device__ __forceinline__ int load_path(const float4* __restrict__ nodes, const int* __restrict__ parent, int n, int k,
                                         f3 o, PathEntry* path, int entries, int lane) {
  int came = ~k, p = __ldg(parent + (n - 1) + k), e = 0;
  while (p >= 0) {
    const int up = __ldg(parent + p);
    if (e == entries - 1 && up >= 0) {
      if (lane == 0) whole_tree(path[e], 0);
      ++e;
      break;
    }
    const float4* nd = nodes + (int64_t)NODE_W * p;
    const float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2), l = __ldg(nd + 3), r = __ldg(nd + 4),
                 d = __ldg(nd + 5);
    if (lane == 0) {
      const bool from_left = __float_as_int(d.z) == came;
      const float4 m = from_left ? r : l;
      const float mo = dot(f3of(m), o);
      if (from_left) {
        path[e].a = make_float4(b.z, b.w, c.x, c.y);
        path[e].b = make_float4(c.z, c.w, d.w, m.w - mo);
        path[e].c = make_float4(m.x, m.y, m.z, d.y - mo);
      } else {
        path[e].a = a;
        path[e].b = make_float4(b.x, b.y, d.z, m.w - mo);
        path[e].c = make_float4(m.x, m.y, m.z, d.x - mo);
      }
    }
    came = p;
    p = up;
    ++e;
  }
  __syncwarp();
  return e;
}

// The path of rays that walk the tree from its root.
__device__ __forceinline__ int load_root(int root, PathEntry* path, int lane) {
  if (lane == 0) whole_tree(path[0], root);
  __syncwarp();
  return 1;
}

// Slab test of a ray that starts near the tree (rays_near), with the origin
// folded into a fused multiply-add, lo * inv + oi, oi = -o * inv. Its rounding
// displaces a plane by at most ~2^-24 |o|, far inside the boxes' padding of
// 1e-6 of the scene's magnitude, besides the relative errors that the slack
// covers as in geom.h slab; so it never rejects a box that contains an mt64
// hit either. From further away 2^-24 |o| exceeds the padding (it was 16
// times the scene's magnitude: hits were lost), so those rays (NEAR false)
// take the differences, as geom.h slab does, whose errors stay relative.
// Direction components below 1e-18 of a unit direction count as 1e-18 (a
// displacement of 1e-18 of the ray's length), which keeps o * inv finite for
// coordinates up to 1e20.
struct RayF {
  f3 o, d, inv, oi;
};
__device__ __forceinline__ RayF make_rayf(f3 o, f3 d) {
  RayF r;
  r.o = o;
  r.d = d;
  const float dx = fabsf(d.x) < 1e-18f ? copysignf(1e-18f, d.x) : d.x;
  const float dy = fabsf(d.y) < 1e-18f ? copysignf(1e-18f, d.y) : d.y;
  const float dz = fabsf(d.z) < 1e-18f ? copysignf(1e-18f, d.z) : d.z;
  r.inv = mk(__frcp_rn(dx), __frcp_rn(dy), __frcp_rn(dz));
  r.oi = mk(-(o.x * r.inv.x), -(o.y * r.inv.y), -(o.z * r.inv.z));
  return r;
}
__device__ __forceinline__ float dotf(f3 a, f3 b) { return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, a.x * b.x)); }
// Whether the ray meets the box within tmax; [tn, tf]: where.
template <bool NEAR>
__device__ __forceinline__ bool in_box(const RayF& r, float lx, float ly, float lz, float hx, float hy, float hz,
                                       float tmax, float& tn, float& tf) {
  auto plane = [](float x, float o, float inv, float oi) {
    return NEAR ? __fmaf_rn(x, inv, oi) : __fmul_rn(__fsub_rn(x, o), inv);
  };
  const float tx0 = plane(lx, r.o.x, r.inv.x, r.oi.x), tx1 = plane(hx, r.o.x, r.inv.x, r.oi.x);
  const float ty0 = plane(ly, r.o.y, r.inv.y, r.oi.y), ty1 = plane(hy, r.o.y, r.inv.y, r.oi.y);
  const float tz0 = plane(lz, r.o.z, r.inv.z, r.oi.z), tz1 = plane(hz, r.o.z, r.inv.z, r.oi.z);
  tn = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fmaxf(fminf(tz0, tz1), 0.0f));
  tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fminf(fmaxf(tz0, tz1), tmax)) * 1.0000005f;
  return tn <= tf;
}
// Whether the ray's stretch [tn, tf] (inside the node's box) meets its slab:
// the heights at the two ends, mo + t m . d, bound it. Within the box every
// term is below ~2 sqrt(3) of the scene's magnitude, so the heights' rounding
// stays below ~1.2e-6 of it; the slabs are widened by 2e-6. A direction that
// is not a number enters every slab, as it does every box.
__device__ __forceinline__ bool in_slab(const RayF& r, f3 m, float mo, float dmin, float dmax, float tn, float tf) {
  const float md = dotf(m, r.d);
  const float a = __fmaf_rn(tn, md, mo), b = __fmaf_rn(tf, md, mo);
  return !(fminf(a, b) > dmax) && !(fmaxf(a, b) < dmin);
}
template <bool NEAR>
__device__ __forceinline__ bool in_entry(const RayF& r, const PathEntry& e, float tmax) {
  float tn, tf;
  return in_box<NEAR>(r, e.a.x, e.a.y, e.a.z, e.a.w, e.b.x, e.b.y, tmax, tn, tf) &&
         in_slab(r, f3of(e.c), 0.f, e.b.w, e.c.w, tn, tf);
}

// geom.h mt32_classify with fused multiply-adds in its products: each triple
// product's error is smaller than without them, so the same bounds hold.
__device__ __forceinline__ f3 crossf(f3 a, f3 b) {
  return mk(__fmaf_rn(a.y, b.z, -(a.z * b.y)), __fmaf_rn(a.z, b.x, -(a.x * b.z)), __fmaf_rn(a.x, b.y, -(a.y * b.x)));
}
// n1, n2: the edges' l1 norms (kept with the leaf).
__device__ __forceinline__ int classify_fma(f3 o, f3 d, f3 v0, f3 v1, f3 v2, float n1, float n2, float* tlo,
                                            float* thi) {
  const float K = 64.0f * 5.9604645e-08f;
  const f3 e1 = sub(v1, v0), e2 = sub(v2, v0), s = sub(o, v0);
  const f3 p = crossf(d, e2), q = crossf(s, e1);
  float det = dotf(e1, p), U = dotf(s, p), V = dotf(d, q), T = dotf(e2, q);
  const float ns = l1(s), nd = l1(d);
  const float Bd = K * (n1 * nd) * n2, Bu = K * (ns * nd) * n2, Bv = K * (ns * nd) * n1, Bt = K * (n2 * ns) * n1;
  if (det < 0.0f) { det = -det; U = -U; V = -V; T = -T; }
  if (det <= Bd) return 2;
  if (U + Bu < 0.0f || V + Bv < 0.0f || T + Bt <= 0.0f) return 0;
  if ((U - Bu) + (V - Bv) > det + Bd) return 0;
  if (U - Bu > 0.0f && V - Bv > 0.0f && (U + Bu) + (V + Bv) < det - Bd && T - Bt > 0.0f) {
    if (tlo) {
      *tlo = ((T - Bt) / (det + Bd)) * (1.0f - 4.0f * 5.9604645e-08f);
      *thi = ((T + Bt) / (det - Bd)) * (1.0f + 4.0f * 5.9604645e-08f);
    }
    return 1;
  }
  return 2;
}

// A lane's walk of the subtrees its ray enters: a node stack (an array of
// its own, in local memory), and the path entries still to visit as bits
// (lowest first).
struct Walk {
  int sp, cur;          // cur: internal node (>= 0), leaf (~k < 0), or LANE_IDLE
  u64 mask;
};
template <bool NEAR>
__device__ __forceinline__ u64 enter_mask(const RayF& r, const PathEntry* path, int ne, float tmax) {
  unsigned lo = 0, hi = 0;
  for (int e = 0; e < ne; ++e)
    if (in_entry<NEAR>(r, path[e], tmax)) {
      if (e < 32) lo |= 1u << e;
      else hi |= 1u << (e - 32);
    }
  return (u64)lo | ((u64)hi << 32);
}
// The next node: the stack's top, else the nearest path entry (within tmax
// where that has shrunk since the entries were tested).
template <bool SHRINKS, bool NEAR>
__device__ __forceinline__ void walk_next(Walk& w, const int* stack, const RayF& r, const PathEntry* path, float tmax) {
  if (w.sp) {
    w.cur = stack[--w.sp];
    return;
  }
  while (w.mask) {
    const int e = __ffsll((long long)w.mask) - 1;
    w.mask &= w.mask - 1;
    if (!SHRINKS || in_entry<NEAR>(r, path[e], tmax)) {
      w.cur = __float_as_int(path[e].b.z);
      return;
    }
  }
  w.cur = LANE_IDLE;
}
// One internal node: the nearer child that the ray enters is next, the other
// one is pushed. The slabs are for rays that start near the tree (the error
// bound of in_slab).
template <bool SHRINKS, bool NEAR>
__device__ __forceinline__ void walk_visit(Walk& w, int* stack, const float4* __restrict__ nodes, const RayF& r,
                                           const PathEntry* path, float tmax, int* err) {
  const float4* nd = nodes + (int64_t)NODE_W * w.cur;
  const float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2), d = __ldg(nd + 5);
  float tl, fl, tr, fr;
  bool hl = in_box<NEAR>(r, a.x, a.y, a.z, a.w, b.x, b.y, tmax, tl, fl);
  bool hr = in_box<NEAR>(r, b.z, b.w, c.x, c.y, c.z, c.w, tmax, tr, fr);
  if (NEAR) {
    const float4 ml = __ldg(nd + 3), mr = __ldg(nd + 4);
    hl = hl & in_slab(r, f3of(ml), dotf(f3of(ml), r.o), ml.w, d.x, tl, fl);
    hr = hr & in_slab(r, f3of(mr), dotf(f3of(mr), r.o), mr.w, d.y, tr, fr);
  }
  const int left = __float_as_int(d.z), right = __float_as_int(d.w);
  if (hl && hr) {
    const bool lfirst = tl <= tr;
    if (w.sp == TRACE_STACK) {
      atomicExch(err, 1);
      w.sp = 0;
      w.mask = 0;
      w.cur = LANE_IDLE;
      return;
    }
    stack[w.sp++] = lfirst ? right : left;
    w.cur = lfirst ? left : right;
  } else if (hl) {
    w.cur = left;
  } else if (hr) {
    w.cur = right;
  } else {
    walk_next<SHRINKS, NEAR>(w, stack, r, path, tmax);
  }
}
// Visits by all lanes at internal nodes, until fewer than NODE_LANES are
// left while others wait at a leaf (or none is).
template <bool SHRINKS, bool NEAR>
__device__ __forceinline__ void walk_nodes(Walk& w, int* stack, const float4* __restrict__ nodes, const RayF& r,
                                           const PathEntry* path, float tmax, int* err) {
  for (;;) {
    const bool in = w.cur >= 0 && w.cur != LANE_IDLE;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (m == 0 || (__popc(m) < NODE_LANES && __any_sync(0xffffffffu, w.cur < 0))) break;
    if (in) walk_visit<SHRINKS, NEAR>(w, stack, nodes, r, path, tmax, err);
  }
}

// ------------------------------------------------------------------ horizons
// One lane per (facet, azimuth): walk the precomputed bisection tree of
// src/cpp/illum.cpp:304-316 (hit -> hi = mid, miss -> lo = mid), one any-hit
// ray per level, until a terminal node. A warp has one facet (or HZ_FACETS
// when nphi < 32), and a lane whose azimuth is done takes the next one: the
// azimuths' work differs several times over, and with one per lane a warp
// waited for its longest. A ray first tests the triangle its lane's last ray
// hit: the next angle of the bisection often hits it again.
// Bound by issue and node-load latency (rays of one facet differ most in
// length); 8 blocks per SM hide the loads best, at 28 bytes of spills (7 were
// 6% slower, 9 spill more).
// 81,920 facets x 64 azimuths: 23.6 ms with a root-to-leaf walk over boxes
// alone, 18.9 ms with one azimuth per lane, 16.5 ms this way; 20,480 x 32
// 1.03 -> 0.79 ms; a 256 x 256 terrain x 128 68 -> 60 ms. With two or four
// facets per warp: 16.8 and 17.6, 1.04 and 1.19 (too few warps), 61 and 64 ms.
// Ray directions in FP64 and a facet frame computed per warp kept that pipe
// 54% busy (0.90 ms for 20,480 x 32): the frame is read instead, and a
// direction is rounded from double-floats that know when they are not sure.
constexpr int HZ_THREADS = 128;
constexpr int HZ_FACETS = 4;      // most facets per warp

struct HzFacet {                  // one of a warp's facets
  frame3 F;
  float2 n[3];                    // F.n as double-floats
  f3 o;
  int own, ne;                    // its leaf (-1: not in the tree) and path entries
};
__device__ __forceinline__ float2 split_df(double x) {
  const float hi = (float)x;
  return make_float2(hi, (float)(x - (double)hi));
}

__device__ __forceinline__ bool hit_any(const float4* __restrict__ tri_s, int k, f3 o, f3 d) {
  const float4 a = __ldg(&tri_s[3 * (int64_t)k]), b = __ldg(&tri_s[3 * (int64_t)k + 1]),
               c = __ldg(&tri_s[3 * (int64_t)k + 2]);
  const int cls = classify_fma(o, d, f3of(a), f3of(b), f3of(c), b.w, c.w, nullptr, nullptr);
  if (cls != 2) return cls == 1;
  double th;
  return mt64(o, d, f3of(a), f3of(b), f3of(c), &th);
}

// fl(s g + c n) of one component of a ray's direction, s, c, g, n as
// double-floats: geom.h horizon_dir rounds an FP64 value within 2^-50 of this
// sum to float, so unless the sum (good to 2^-43) is as near as that to a
// rounding boundary the float is the same. false: it may not be.
__device__ __forceinline__ bool dir_component(float2 s, float2 g, float2 c, float2 n, float& out) {
  const float p = __fmul_rn(s.x, g.x), q = __fmul_rn(c.x, n.x);
  float e = __fmaf_rn(s.x, g.x, -p), f = __fmaf_rn(c.x, n.x, -q);
  e = __fmaf_rn(s.x, g.y, e);
  f = __fmaf_rn(c.x, n.y, f);
  e = __fmaf_rn(s.y, g.x, e);
  f = __fmaf_rn(c.y, n.x, f);
  const float a = __fadd_rn(p, q), bb = __fsub_rn(a, p);
  const float err = __fadd_rn(__fsub_rn(p, __fsub_rn(a, bb)), __fsub_rn(q, bb));   // TwoSum
  const float lo = __fadd_rn(err, __fadd_rn(e, f));
  const float h = __fadd_rn(a, lo), l = __fsub_rn(lo, __fsub_rn(h, a));
  const float E = 2.2737368e-13f;   // 2^-42
  out = h;
  return __fadd_rn(h, __fadd_rn(l, E)) == h && __fadd_rn(h, __fsub_rn(l, E)) == h;
}

// NEAR: the facets are leaves of the tree and the rays start near it. Else
// (another mesh's tree, whose coordinates may differ in magnitude, or a large
// offset) the walk begins at the root.
template <bool NEAR>
__global__ void __launch_bounds__(HZ_THREADS, 8)
k_horizons(const float4* __restrict__ nodes, const float4* __restrict__ tri_s, int root,
           const int* __restrict__ parent, const uint32_t* __restrict__ rank, const double* __restrict__ frame,
           const float4* __restrict__ cen, const float4* __restrict__ nrm, int nt, int nphi,
           const double* __restrict__ cph, const double* __restrict__ sph, const HorizonNode* __restrict__ tree,
           int tree_size, float offset, int slots, int entries, double* H, int* derr) {
  extern __shared__ PathEntry hz_paths[];   // [warp][slots][entries]
  __shared__ HzFacet hz_facets[HZ_THREADS / 32][HZ_FACETS];
  __shared__ float2 hz_dir[3][HZ_THREADS];   // the lane's azimuth: cos b + sin t
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PathEntry* paths = hz_paths + (size_t)warp * slots * entries;
  HzFacet* facets = hz_facets[warp];
  const int f0 = (blockIdx.x * (HZ_THREADS / 32) + warp) * slots;
  if (f0 >= nt) return;
  const int nf = min(slots, nt - f0), items = nf * nphi;
  for (int q = 0; q < nf; ++q) {
    const f3 n = f3of(nrm[f0 + q]);
    const f3 o = add(f3of(cen[f0 + q]), scl(n, offset));
    int m, own = -1;
    if (NEAR) {
      own = (int)__ldg(rank + f0 + q);
      m = load_path(nodes, parent, nt, own, o, paths + q * entries, entries, lane);
    } else {
      m = load_root(root, paths + q * entries, lane);
    }
    if (lane == q) {
      const double* fr = frame + 9 * (int64_t)(f0 + q);
      const frame3 F{mkd(fr[0], fr[1], fr[2]), mkd(fr[3], fr[4], fr[5]), mkd(fr[6], fr[7], fr[8])};
      facets[q] = HzFacet{F, {split_df(F.n.x), split_df(F.n.y), split_df(F.n.z)}, o, own, m};
    }
  }
  __syncwarp();
  // the lane's azimuth: item q * nphi + k of the warp's; the next one to take
  int item = lane, next = 32;
  bool on = item < items;
  int q = on ? item / nphi : 0;
  const PathEntry* path = paths + q * entries;
  f3 o = facets[q].o;
  auto aim = [&]() {
    const frame3& F = facets[q].F;
    const double cp = __ldg(cph + (item - q * nphi)), sp = __ldg(sph + (item - q * nphi));
    hz_dir[0][threadIdx.x] = split_df(F.b.x * cp + F.t.x * sp);
    hz_dir[1][threadIdx.x] = split_df(F.b.y * cp + F.t.y * sp);
    hz_dir[2][threadIdx.x] = split_df(F.b.z * cp + F.t.z * sp);
  };
  if (on) aim();
  int node = 1, last = -1;
  RayF r = make_rayf(o, mk(0.f, 0.f, 1.f));
  Walk wk;
  int stack[TRACE_STACK];
  wk.sp = 0;
  wk.mask = 0;
  wk.cur = LANE_IDLE;
  bool fresh = on;      // begins its next ray
  const float TMAX = 3.0e38f;
  for (;;) {
    if (fresh) {
      const HorizonNode* hn = tree + node;
      const bool bad = node >= tree_size;
      if (bad || hn->terminal) {
        if (bad) atomicExch(&derr[DERR_HORIZON], 1);
        H[(int64_t)f0 * nphi + item] = bad ? 0.0 : hn->mid;
        on = fresh = false;
      }
    }
    // lanes without an azimuth take the warp's next ones (the tree's root is
    // never terminal: an azimuth has one ray at least)
    if (next < items) {
      const unsigned idle = __ballot_sync(0xffffffffu, !on);
      const int mine = next + __popc(idle & ((1u << lane) - 1u));
      next += __popc(idle);
      if (!on && mine < items) {
        item = mine;
        q = item / nphi;
        path = paths + q * entries;
        o = facets[q].o;
        aim();
        node = 1;
        last = -1;
        on = fresh = true;
      }
    }
    if (fresh) {
      const int k = item - q * nphi, own = facets[q].own;
      const HorizonNode* hn = tree + node;
      f3 dir;
      const float2 sd = hn->sdf, cd = hn->cdf;
      const HzFacet& fc = facets[q];
      if (!(dir_component(sd, hz_dir[0][threadIdx.x], cd, fc.n[0], dir.x) &
            dir_component(sd, hz_dir[1][threadIdx.x], cd, fc.n[1], dir.y) &
            dir_component(sd, hz_dir[2][threadIdx.x], cd, fc.n[2], dir.z)))
        dir = horizon_dir(fc.F, __ldg(cph + k), __ldg(sph + k), hn->c, hn->s);
      r = make_rayf(o, dir);
      bool hit = last >= 0 && hit_any(tri_s, last, o, r.d);
      if (!hit && own >= 0 && own != last) hit = hit_any(tri_s, own, o, r.d);
      if (hit) {
        node = 2 * node;              // still fresh: the next angle
      } else {
        fresh = false;
        wk.sp = 0;
        wk.mask = enter_mask<NEAR>(r, path, facets[q].ne, TMAX);
        walk_next<false, NEAR>(wk, stack, r, path, TMAX);
        if (wk.cur == LANE_IDLE) {    // enters nothing: a miss
          node = 2 * node + 1;
          fresh = true;
        }
      }
    }
    const unsigned onm = __ballot_sync(0xffffffffu, on);
    if (!onm) return;
    const unsigned fm = __ballot_sync(0xffffffffu, fresh);
    // enough lanes (or all) that can begin a ray: begin them
    if (fm && (__popc(fm) >= REFILL_LANES || fm == onm)) continue;
    for (;;) {
      walk_nodes<false, NEAR>(wk, stack, nodes, r, path, TMAX, &derr[DERR_STACK]);
      if (wk.cur < 0) {
        const int kl = ~wk.cur;
        if (hit_any(tri_s, kl, o, r.d)) {
          last = kl;
          node = 2 * node;
          fresh = true;
          wk.cur = LANE_IDLE;
        } else {
          walk_next<false, NEAR>(wk, stack, r, path, TMAX);
        }
      }
      if (on && !fresh && wk.cur == LANE_IDLE) {
        node = 2 * node + 1;
        fresh = true;
      }
      const unsigned f2 = __ballot_sync(0xffffffffu, fresh);
      if (__popc(f2) >= REFILL_LANES || f2 == onm) break;
    }
  }
}

// fp32 copies of a facet's horizon and of its min / max (the insolation
// filters compare in fp32 with margins).
__global__ void k_horizon_f32(const double* __restrict__ H, int nt, int nphi, float* H32, float2* hmm) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nt) return;
  const double* h = H + (int64_t)f * nphi;
  float* h32 = H32 + (int64_t)f * nphi;
  double lo = h[0], hi = h[0];
  for (int k = 0; k < nphi; ++k) {
    lo = fmin(lo, h[k]);
    hi = fmax(hi, h[k]);
    h32[k] = (float)h[k];
  }
  hmm[f] = make_float2((float)lo, (float)hi);
}

// ------------------------------------------------------------------ visibility
// Candidates of source j: every i != j passing the facing test of
// src/cpp/illum.cpp:65-68 (and the optional distance cutoff). The leaves in
// Morton order are grouped by 32 (level 0), the groups by 32 (level 1) and
// those by 32 (level 2), each with the box of its triangles; a warp
// enumerates one source's candidates by testing 32 boxes of a level at a
// time (a box whose farthest point along n_j is below -r_max, or that is
// farther than the cutoff, holds none) and then the 32 facets of each group
// that remains, one per lane: all loads are coalesced, and a candidate list
// never exists in device memory.
__device__ __forceinline__ float box_dist2(f3 p, f3 lo, f3 hi) {
  float dx = fmaxf(fmaxf(lo.x - p.x, p.x - hi.x), 0.f);
  float dy = fmaxf(fmaxf(lo.y - p.y, p.y - hi.y), 0.f);
  float dz = fmaxf(fmaxf(lo.z - p.z, p.z - hi.z), 0.f);
  return dx * dx + dy * dy + dz * dz;
}

struct LeafGroups {
  const float4* cen_s;          // centroid and bounding radius by Morton position
  const uint32_t* order;        // facet by Morton position
  const float4 *lo[3], *hi[3];  // boxes of the levels
  int n[3];                     // their counts
  int nt;
  float lim;                    // -r_max - slack
  float cut2, box_cut2;         // squared cutoff, < 0: none
};

// Level 0 boxes (padded as the LBVH's) and the Morton-ordered centroids.
__global__ void k_leaf_groups(const float4* __restrict__ tri_s, const float4* __restrict__ cen,
                              const uint32_t* __restrict__ order, int nt, float pad, float4* cen_s, float4* lo,
                              float4* hi) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  float l[3] = {3e38f, 3e38f, 3e38f}, h[3] = {-3e38f, -3e38f, -3e38f};
  if (k < nt) {
    cen_s[k] = cen[order[k]];
    for (int q = 0; q < 3; ++q) {
      const float4 v = tri_s[3 * (int64_t)k + q];
      l[0] = fminf(l[0], v.x); l[1] = fminf(l[1], v.y); l[2] = fminf(l[2], v.z);
      h[0] = fmaxf(h[0], v.x); h[1] = fmaxf(h[1], v.y); h[2] = fmaxf(h[2], v.z);
    }
  }
  for (int o = 16; o; o >>= 1)
    for (int a = 0; a < 3; ++a) {
      l[a] = fminf(l[a], __shfl_xor_sync(0xffffffffu, l[a], o));
      h[a] = fmaxf(h[a], __shfl_xor_sync(0xffffffffu, h[a], o));
    }
  if ((threadIdx.x & 31) == 0 && k < nt) {
    lo[k >> 5] = make_float4(l[0] - pad, l[1] - pad, l[2] - pad, 0.f);
    hi[k >> 5] = make_float4(h[0] + pad, h[1] + pad, h[2] + pad, 0.f);
  }
}
// The next level's boxes from 32 of this level's each.
__global__ void k_group_boxes(const float4* __restrict__ lo, const float4* __restrict__ hi, int n, float4* lo2,
                              float4* hi2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  float4 l = make_float4(3e38f, 3e38f, 3e38f, 0.f), h = make_float4(-3e38f, -3e38f, -3e38f, 0.f);
  if (k < n) { l = lo[k]; h = hi[k]; }
  for (int o = 16; o; o >>= 1) {
    l.x = fminf(l.x, __shfl_xor_sync(0xffffffffu, l.x, o));
    l.y = fminf(l.y, __shfl_xor_sync(0xffffffffu, l.y, o));
    l.z = fminf(l.z, __shfl_xor_sync(0xffffffffu, l.z, o));
    h.x = fmaxf(h.x, __shfl_xor_sync(0xffffffffu, h.x, o));
    h.y = fmaxf(h.y, __shfl_xor_sync(0xffffffffu, h.y, o));
    h.z = fmaxf(h.z, __shfl_xor_sync(0xffffffffu, h.z, o));
  }
  if ((threadIdx.x & 31) == 0 && k < n) { lo2[k >> 5] = l; hi2[k >> 5] = h; }
}

// One source's enumeration (warp-uniform state).
struct Enumerate {
  int j;
  f3 p_j, n_j;
  int base2, cur2, cur1;          // next batch of level 2, current level-2 batch / level-1 box
  int b2;
  unsigned m2, m1, m0;            // boxes still to open
  __device__ __forceinline__ void start(const LeafGroups& G, int source, f3 p, f3 n) {
    j = source;
    p_j = p;
    n_j = n;
    base2 = cur2 = cur1 = b2 = 0;
    m2 = m1 = m0 = 0;
  }
  __device__ __forceinline__ unsigned open(const LeafGroups& G, int level, int first, int lane) const {
    bool ok = false;
    const int q = first + lane;
    if (q < G.n[level]) {
      const float4 l4 = __ldg(G.lo[level] + q), h4 = __ldg(G.hi[level] + q);
      const f3 lo = f3of(l4), hi = f3of(h4);
      const float m = (n_j.x >= 0.f ? (hi.x - p_j.x) * n_j.x : (lo.x - p_j.x) * n_j.x) +
                      (n_j.y >= 0.f ? (hi.y - p_j.y) * n_j.y : (lo.y - p_j.y) * n_j.y) +
                      (n_j.z >= 0.f ? (hi.z - p_j.z) * n_j.z : (lo.z - p_j.z) * n_j.z);
      ok = m > G.lim;
      if (G.cut2 >= 0.f) ok = ok && box_dist2(p_j, lo, hi) <= G.box_cut2;   // centroids lie inside the boxes
    }
    return __ballot_sync(0xffffffffu, ok);
  }
  // The next group with possible candidates, as the mask of its lanes that
  // pass and its first leaf position; false once there is none.
  __device__ __forceinline__ bool next(const LeafGroups& G, int lane, int& k0, unsigned& pass) {
    for (;;) {
      if (m0) {
        const int g = cur1 * 32 + __ffs(m0) - 1;
        m0 &= m0 - 1;
        k0 = 32 * g;
        const int k = k0 + lane;
        bool ok = false;
        if (k < G.nt) {
          const float4 c = __ldg(G.cen_s + k);
          ok = (int)__ldg(G.order + k) != j && facing(f3of(c), c.w, p_j, n_j) && within_cutoff(f3of(c), p_j, G.cut2);
        }
        pass = __ballot_sync(0xffffffffu, ok);
        if (pass) return true;
      } else if (m1) {
        cur1 = cur2 * 32 + __ffs(m1) - 1;
        m1 &= m1 - 1;
        m0 = open(G, 0, cur1 * 32, lane);
      } else if (m2) {
        cur2 = b2 + __ffs(m2) - 1;
        m2 &= m2 - 1;
        m1 = open(G, 1, cur2 * 32, lane);
      } else if (base2 < G.n[2]) {
        b2 = base2;
        base2 += 32;
        m2 = open(G, 2, b2, lane);
      } else {
        return false;
      }
    }
  }
};

// Candidates of each source: source q is the facet src[q], or the facet at
// Morton position q.
__global__ void __launch_bounds__(128) k_count_pairs(LeafGroups G, const float4* __restrict__ nrm,
                                                     const float4* __restrict__ cen, const int* __restrict__ src,
                                                     int nsrc, uint32_t* count) {
  const int lane = threadIdx.x & 31;
  const int64_t q = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (q >= nsrc) return;
  const int j = src ? src[q] : (int)G.order[q];
  Enumerate en;
  en.start(G, j, f3of(cen[j]), f3of(nrm[j]));
  uint32_t c = 0;
  int k0;
  unsigned pass;
  while (en.next(G, lane, k0, pass)) c += __popc(pass);
  if (lane == 0) count[q] = c;
}

// One visibility ray per candidate pair (src/cpp/illum.cpp:72-83): from the
// offset centroid q_j towards p_i, closest hit. A ray that hits a facet h
// other than j yields the key (h << bits) | j, in ukeys in any order and
// possibly more than once (it is sorted and made unique afterwards); hits
// that the warp has seen lately for the same source are dropped.
//
// A warp takes one unit at a time (from a counter): a source, or a part of
// one with many candidates, and keeps its lanes filled from the source's
// enumeration. Every ray begins with the triangle
// it is aimed at, which bounds its length before any box is tested, and with
// its own facet; the order of the tests does not change the closest hit.
// Bound by issue (62%, 17 of 32 lanes active) and L1 bandwidth (54%). Form
// factors of 81,920 facets (766 M rays) 234 -> 145 ms, of a 256 x 256 terrain
// within 30 m (92 M rays) 53 -> 37 ms, of 20,480 facets (7.4 M) 7.1 -> 2.3 ms
// against a candidate list in device memory (a counting and a filling walk per
// source, 0.4 and 0.17 of the ray kernel's time) and one root-to-leaf walk
// over boxes per ray. The enumeration waits in shared memory, which leaves the
// walk with 12 bytes of spills at seven blocks per SM (five: 13% slower, six
// 4%).
constexpr int VIS_THREADS = 128;
constexpr int VIS_QUEUE = 64;      // candidates waiting (at most 31 + 32)
constexpr int VIS_KEYS = 64;       // keys waiting to be written (at most 31 + 32)
constexpr int VIS_SEEN = 128;      // recent hits per warp

// Candidates per unit. A facet deep in a crater has twenty times the
// candidates of one outside, and as one unit its rays would keep one warp
// busy after the others have run out: 20,480 facets (7.4 M rays, at most
// 4,522 of one source, 229 in the middle) took 2.23 ms that way, with SMs at
// work for 72% of it on average, and 1.4 ms in parts. A part first counts through the candidates before it
// and loads the path anew, so sources are only split where the mean warp has
// few units: at VIS_SHARES parts of a warp's share of the rays, at least
// VIS_PART_MIN.
constexpr int VIS_PART_MIN = 256;
constexpr int VIS_SHARES = 8;

// The units of sources [a, b): (source, its part), in any order.
__global__ void k_vis_units(const uint32_t* __restrict__ count, int a, int b, uint32_t part, uint2* units,
                            unsigned* nunits) {
  const int q = a + blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const unsigned n = q < b ? (count[q] + part - 1) / part : 0;
  unsigned at = n;
  for (int o = 1; o < 32; o *= 2) {
    const unsigned t = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += t;
  }
  unsigned base = 0;
  if (lane == 31 && at) base = atomicAdd(nunits, at);
  base = __shfl_sync(0xffffffffu, base, 31);
  at += base - n;
  for (unsigned k = 0; k < n; ++k) units[at + k] = make_uint2((unsigned)q, k);
}

struct VisWarp {
  Enumerate en;              // the unit's enumeration, out of the walk's registers
  unsigned passed;           // candidates it has passed
  int queue[VIS_QUEUE];
  int seen[VIS_SEEN];
  unsigned long long keys[VIS_KEYS];
};

// The closest hit so far: facet, leaf position, and an enclosure of its mt64 t.
struct Best {
  int i, k;
  float lo, hi, tmax;
};
__device__ __forceinline__ void test_closest(const float4* __restrict__ tri_s, int k, f3 o, f3 d, Best& B) {
  const float4 a = __ldg(&tri_s[3 * (int64_t)k]), b = __ldg(&tri_s[3 * (int64_t)k + 1]),
               c = __ldg(&tri_s[3 * (int64_t)k + 2]);
  const f3 v0 = f3of(a), v1 = f3of(b), v2 = f3of(c);
  const int idx = __float_as_int(a.w);
  float tlo = 0.f, thi = 0.f;
  const int cls = classify_fma(o, d, v0, v1, v2, b.w, c.w, &tlo, &thi);
  bool take = false;
  if (cls == 1 && (B.i < 0 || thi < B.lo)) {
    take = true;                    // certainly the closest so far
  } else if (cls == 2 || (cls == 1 && !(tlo > B.hi))) {
    double th;
    if (mt64(o, d, v0, v1, v2, &th)) {
      bool closer = B.i < 0;
      if (!closer) {                // exact t of the current best
        double bt = 0.0;
        const float4 ba = __ldg(&tri_s[3 * (int64_t)B.k]), bb = __ldg(&tri_s[3 * (int64_t)B.k + 1]),
                     bc = __ldg(&tri_s[3 * (int64_t)B.k + 2]);
        mt64(o, d, f3of(ba), f3of(bb), f3of(bc), &bt);
        closer = th < bt || (th == bt && idx < B.i);
      }
      if (closer) {
        take = true;
        const float tf = (float)th;
        tlo = tf * (1.0f - 2.4e-7f);
        thi = tf * (1.0f + 2.4e-7f) + 1e-37f;
      }
    }
  }
  if (take) {
    B.i = idx;
    B.k = k;
    B.lo = tlo;
    B.hi = thi;
    B.tmax = thi * 1.000001f + 1e-30f;
  }
}

// NEAR: the rays start near the tree. Else they walk it from the root.
template <bool NEAR>
__global__ void __launch_bounds__(VIS_THREADS, 7)
k_vis_rays(const float4* __restrict__ nodes, const float4* __restrict__ tri_s, int root, const int* __restrict__ parent,
           const uint32_t* __restrict__ rank, LeafGroups G, const float4* __restrict__ cen,
           const float4* __restrict__ nrm, const int* __restrict__ src, const uint2* __restrict__ units,
           const unsigned* __restrict__ nunits, unsigned part, float offset, int bits, int entries,
           unsigned* next_unit, unsigned long long* ukeys, unsigned long long* ucount, int* derr) {
  __shared__ VisWarp sh[VIS_THREADS / 32];
  extern __shared__ PathEntry vis_paths[];   // [warp][entries]
  PathEntry* path = vis_paths + (size_t)(threadIdx.x >> 5) * entries;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  VisWarp& S = sh[threadIdx.x >> 5];
  int nkeys = 0;
  auto flush = [&]() {   // the waiting keys
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(ucount, (unsigned long long)nkeys);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int t = lane; t < nkeys; t += 32) ukeys[base + t] = S.keys[t];
    __syncwarp();
    nkeys = 0;
  };
  const unsigned nu = __ldg(nunits);
  for (;;) {
    unsigned u = 0;
    if (lane == 0) u = atomicAdd(next_unit, 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= nu) break;
    const uint2 unit = __ldg(units + u);
    const int q = (int)unit.x;
    const int j = src ? src[q] : (int)G.order[q];
    const f3 p_j = f3of(cen[j]), n_j = f3of(nrm[j]);
    const f3 o = add(p_j, scl(n_j, offset));
    __syncwarp();
    if (lane == 0) {
      S.en.start(G, j, p_j, n_j);
      S.passed = 0;
    }
    __syncwarp();
    int qn = 0;                 // candidates in the queue
    // The next candidates into the queue, at least `want`; false: no more.
    // The unit's are those of rank [first, first + part) in the source's
    // enumeration.
    auto fetch = [&](int want) -> bool {
      Enumerate en = S.en;
      unsigned at = S.passed;
      const unsigned first = unit.y * part;
      bool more = true;
      while (qn < want) {
        int k0;
        unsigned pass;
        more = at < first + part && en.next(G, lane, k0, pass);
        if (!more) break;
        const unsigned r = at + __popc(pass & lt);
        const bool in = ((pass >> lane) & 1) && r >= first && r < first + part;
        const unsigned take = __ballot_sync(0xffffffffu, in);
        if (in) S.queue[qn + __popc(take & lt)] = k0 + lane;
        qn += __popc(take);
        at += __popc(pass);
      }
      __syncwarp();
      if (lane == 0) {
        S.en = en;
        S.passed = at;
      }
      __syncwarp();
      return more;
    };
    bool more = true;
    const int own = (int)__ldg(rank + j);
    const int ne = NEAR ? load_path(nodes, parent, G.nt, own, o, path, entries, lane) : load_root(root, path, lane);
    for (int t = lane; t < VIS_SEEN; t += 32) S.seen[t] = -1;
    __syncwarp();
    bool on = false;            // this lane has a ray
    RayF r = make_rayf(o, mk(0.f, 0.f, 1.f));
    Best B{-1, 0, 3.0e38f, 3.0e38f, 3.0e38f};
    Walk wk;
    int stack[TRACE_STACK];
    wk.sp = 0;
    wk.mask = 0;
    wk.cur = LANE_IDLE;
    int target = -1;
    for (;;) {
      // rays that have ended: their hits
      const bool ended = on && wk.cur == LANE_IDLE;
      bool emit = ended && B.i >= 0 && B.i != j;
      if (emit) emit = S.seen[B.i & (VIS_SEEN - 1)] != B.i;
      if (__any_sync(0xffffffffu, emit)) {
        const unsigned same = __match_any_sync(0xffffffffu, emit ? B.i : -1 - lane);
        emit = emit && (same & lt) == 0;
        if (emit) S.seen[B.i & (VIS_SEEN - 1)] = B.i;
        const unsigned em = __ballot_sync(0xffffffffu, emit);
        if (emit)
          S.keys[nkeys + __popc(em & lt)] = ((unsigned long long)B.i << bits) | (unsigned long long)j;
        nkeys += __popc(em);
        if (nkeys >= 32) flush();
        __syncwarp();
      }
      if (ended) on = false;
      // fill the idle lanes
      const unsigned idle = __ballot_sync(0xffffffffu, !on);
      const int want = __popc(idle);
      if (more && qn < want) more = fetch(want);
      const int take = min(want, qn);
      if (!on && __popc(idle & lt) < take) {
        target = S.queue[qn - 1 - __popc(idle & lt)];
        on = true;
        r = make_rayf(o, normalize(sub(f3of(__ldg(G.cen_s + target)), o)));
        B = Best{-1, 0, 3.0e38f, 3.0e38f, 3.0e38f};
        test_closest(tri_s, target, o, r.d, B);
        test_closest(tri_s, own, o, r.d, B);
        wk.sp = 0;
        wk.mask = enter_mask<NEAR>(r, path, ne, B.tmax);
        walk_next<true, NEAR>(wk, stack, r, path, B.tmax);
      }
      qn -= take;
      __syncwarp();
      const unsigned onm = __ballot_sync(0xffffffffu, on);
      if (!onm) break;
      const bool refillable = more || qn > 0;
      for (;;) {
        walk_nodes<true, NEAR>(wk, stack, nodes, r, path, B.tmax, &derr[DERR_STACK]);
        if (wk.cur < 0) {
          if (~wk.cur != target) test_closest(tri_s, ~wk.cur, o, r.d, B);
          walk_next<true, NEAR>(wk, stack, r, path, B.tmax);
        }
        const int run = __popc(__ballot_sync(0xffffffffu, wk.cur != LANE_IDLE));
        if (run == 0 || (refillable && 32 - run >= REFILL_LANES)) break;
      }
    }
  }
  if (nkeys > 0) flush();
}

// After sorting: first occurrence of each (row, col) -> form factor
// (src/cpp/illum.cpp:100-130), albedo row scale (:225-234); zeros dropped.
__global__ void k_ff_values(const unsigned long long* __restrict__ keys, int64_t n, int bits, int nt,
                            const float4* __restrict__ cen, const float4* __restrict__ nrm,
                            const double* __restrict__ area, const double* __restrict__ albedo, double albedo_scalar,
                            uint32_t* keep, double* fval, int* derr) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  unsigned long long key = keys[k];
  unsigned long long mask = (1ull << bits) - 1ull;
  int i = (int)(key >> bits), j = (int)(key & mask);
  uint32_t kp = 0;
  double F = 0.0;
  if (k == 0 || keys[k - 1] != key) {
    F = form_factor(f3of(cen[i]), f3of(nrm[i]), f3of(cen[j]), f3of(nrm[j]), area[j]);
    if (isnan(F)) {
      atomicExch(&derr[DERR_NAN], 1);
    } else if (F != 0.0) {
      double rho = albedo ? albedo[i] : albedo_scalar;
      F = F * rho;
      kp = 1;
    }
  }
  keep[k] = kp;
  fval[k] = F;
}

// Sampled visibility: every distinct (hit i, source j) key with a nonzero
// form factor counts for its source's sample slot, and for every radius its
// centroid distance does not exceed.
__global__ void k_sample_count(const unsigned long long* __restrict__ keys, int64_t n, int bits,
                               const float4* __restrict__ cen, const float4* __restrict__ nrm,
                               const double* __restrict__ area, const int* __restrict__ slot,
                               const double* __restrict__ radii, int nradii, unsigned long long* per_src,
                               unsigned long long* within) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned long long key = keys[k];
  if (k > 0 && keys[k - 1] == key) return;
  const unsigned long long mask = (1ull << bits) - 1ull;
  const int i = (int)(key >> bits), j = (int)(key & mask);
  const double F = form_factor(f3of(cen[i]), f3of(nrm[i]), f3of(cen[j]), f3of(nrm[j]), area[j]);
  if (!(F > 0.0)) return;
  atomicAdd(&per_src[slot[j]], 1ull);
  const float4 a = cen[i], b = cen[j];
  const double dx = (double)a.x - b.x, dy = (double)a.y - b.y, dz = (double)a.z - b.z;
  const double d = sqrt(dx * dx + dy * dy + dz * dz);
  for (int q = 0; q < nradii; ++q)
    if (d <= radii[q]) atomicAdd(&within[q], 1ull);
}

// A chunk's kept entries (first occurrence, nonzero form factor): key and
// value at their scan position.
__global__ void k_ff_pack(const unsigned long long* __restrict__ keys, int64_t n, const uint32_t* __restrict__ keep,
                          const unsigned long long* __restrict__ pos, const double* __restrict__ fval,
                          unsigned long long* okey, double* oval) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || !keep[k]) return;
  const int64_t p = (int64_t)pos[k];
  okey[p] = keys[k];
  oval[p] = fval[k];
}

// The entries in (row, column) order: row and column from the sorted key,
// the value through the sort's permutation (idx == nullptr: no
// permutation).
__global__ void k_ff_unpack(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ idx,
                            const double* __restrict__ vals, int64_t n, int bits, int32_t* rows, int32_t* col,
                            double* val) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned long long key = keys[k];
  rows[k] = (int32_t)(key >> bits);
  col[k] = (int32_t)(key & ((1ull << bits) - 1ull));
  val[k] = vals[idx ? idx[k] : k];
}

__global__ void k_iota_u32(uint32_t* a, int64_t n) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) a[k] = (uint32_t)k;
}

__global__ void k_rowptr(const int32_t* __restrict__ rows, int64_t nnz, int nt, int64_t* rowptr) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > nt) return;
  int64_t lo = 0, hi = nnz;   // first index with rows[idx] >= r
  while (lo < hi) {
    int64_t m = (lo + hi) >> 1;
    if (rows[m] < r) lo = m + 1; else hi = m;
  }
  rowptr[r] = lo;
}

}  // namespace

// ====================================================================== host

// Padding of the boxes (see geom.h slab and RayF for what it has to cover).
static float box_pad(const Context& c) { return 1e-6f * c.scene_mag; }
// Whether rays from the facets' centroids, `offset` along the normals, start
// near the context's own tree: within a quarter of the scene's magnitude of
// it, where the folded plane tests displace a plane by 0.1e-6 of the scene's
// magnitude (padding 1e-6) and the slabs' heights are good to 1.3e-6 of it
// (widened by 2e-6); and coordinates small enough for o * inv.
static bool rays_near(const Context& c, float offset) {
  return std::fabs(offset) * c.nrm_max <= 0.25f * c.scene_mag && c.scene_mag < 1e19f;
}
// Most path entries of a facet: one per level, as many as the mask's bits (a
// test entry may lower it to exercise paths that end with the whole tree).
static std::atomic<int> g_path_most{PATH_MOST};
int path_set_most(int entries) {
  g_path_most.store(entries > 0 ? std::min(entries, PATH_MOST) : PATH_MOST);
  return ILG_OK;
}
static int path_entries(const Context& c) { return std::max(1, std::min(c.bvh_longest, g_path_most.load())); }

int bvh_build(Context& c, const float* verts_h, int nv, const int32_t* tris_h, const float* normals_h) {
  int nt = c.nt;
  cudaStream_t s = c.stream;
  // scene bounds and magnitude (host)
  float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
  float mag = 0.f;
  for (int v = 0; v < nv; ++v)
    for (int a = 0; a < 3; ++a) {
      float x = verts_h[3 * v + a];
      if (!(x == x) || std::isinf(x)) { set_error("vertex %d has a non-finite coordinate", v); return ILG_ERR_ARG; }
      lo[a] = std::min(lo[a], x); hi[a] = std::max(hi[a], x); mag = std::max(mag, std::fabs(x));
    }
  for (int t = 0; t < 3 * nt; ++t)
    if (tris_h[t] < 0 || tris_h[t] >= nv) { set_error("triangle %d has vertex index %d out of range", t / 3, tris_h[t]); return ILG_ERR_ARG; }
  c.scene_mag = mag > 0.f ? mag : 1.f;
  c.nrm_max = 1.f;
  for (int t = 0; normals_h && t < nt; ++t) {
    const float* n = normals_h + 3 * (size_t)t;
    c.nrm_max = std::max(c.nrm_max, std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]));
  }

  dbuf<float> dverts, dnormals;
  dbuf<int32_t> dtris;
  ILG_TRY(dverts.alloc((size_t)nv * 3));
  ILG_TRY(dtris.alloc((size_t)nt * 3));
  ILG_CUDA(cudaMemcpyAsync(dverts.p, verts_h, (size_t)nv * 12, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemcpyAsync(dtris.p, tris_h, (size_t)nt * 12, cudaMemcpyHostToDevice, s));
  if (normals_h) {
    ILG_TRY(dnormals.alloc((size_t)nt * 3));
    ILG_CUDA(cudaMemcpyAsync(dnormals.p, normals_h, (size_t)nt * 12, cudaMemcpyHostToDevice, s));
  }
  ILG_TRY(c.tri_o.alloc((size_t)nt * 3));
  ILG_TRY(c.cen.alloc(nt));
  ILG_TRY(c.nrm.alloc(nt));
  ILG_TRY(c.area.alloc(nt));
  ILG_TRY(c.frame.alloc((size_t)nt * 9));
  ILG_TRY(c.frame32.alloc((size_t)nt * 3));
  k_prepare<<<div_up(nt, 256), 256, 0, s>>>(dverts.p, dtris.p, dnormals.p, nt, c.tri_o.p, c.cen.p, c.nrm.p,
                                            c.area.p, c.frame.p, c.frame32.p);
  ILG_CUDA(cudaGetLastError());

  // r_max on the host copy of the radii
  std::vector<float4> cen_h(nt);
  ILG_CUDA(cudaMemcpyAsync(cen_h.data(), c.cen.p, (size_t)nt * 16, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  float rmax = 0.f;
  for (int t = 0; t < nt; ++t) rmax = std::max(rmax, cen_h[t].w);
  c.r_max = rmax;

  dbuf<unsigned long long> keys;
  dbuf<uint32_t>& order = c.morton_order;   // kept: facets in Morton order
  ILG_TRY(keys.alloc(nt));
  ILG_TRY(order.alloc(nt));
  float3 blo = make_float3(lo[0], lo[1], lo[2]);
  float3 inv = make_float3(hi[0] > lo[0] ? 1.f / (hi[0] - lo[0]) : 0.f, hi[1] > lo[1] ? 1.f / (hi[1] - lo[1]) : 0.f,
                           hi[2] > lo[2] ? 1.f / (hi[2] - lo[2]) : 0.f);
  k_morton<<<div_up(nt, 256), 256, 0, s>>>(c.cen.p, nt, blo, inv, keys.p, order.p);
  ILG_CUDA(cudaGetLastError());
  ILG_TRY(radix_sort_u64(keys.p, order.p, nt, 63, c.sort, s));

  dbuf<int2> child, range;
  dbuf<int>& parent = c.parent;   // kept: the paths of the facets' rays start at their leaves
  dbuf<int> flags, depth;
  dbuf<float4> box_lo, box_hi;
  int ni = nt > 1 ? nt - 1 : 1;
  ILG_TRY(child.alloc(ni));
  ILG_TRY(range.alloc(ni));
  ILG_TRY(parent.alloc((size_t)2 * nt));
  ILG_TRY(flags.alloc(ni));
  ILG_TRY(depth.alloc(2));
  ILG_TRY(box_lo.alloc((size_t)2 * nt));
  ILG_TRY(box_hi.alloc((size_t)2 * nt));
  ILG_TRY(c.tri_s.alloc((size_t)nt * 3));
  ILG_TRY(c.leaf_rank.alloc(nt));
  ILG_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int) * ni, s));
  ILG_CUDA(cudaMemsetAsync(depth.p, 0, 2 * sizeof(int), s));
  ILG_CUDA(cudaMemsetAsync(parent.p, 0xff, sizeof(int) * 2 * nt, s));   // -1: root has no parent
  if (nt > 1) {
    k_karras<<<div_up(nt - 1, 256), 256, 0, s>>>(keys.p, nt, child.p, parent.p, range.p);
    ILG_CUDA(cudaGetLastError());
  }
  k_leaf_rank<<<div_up(nt, 256), 256, 0, s>>>(order.p, parent.p, nt, c.leaf_rank.p, depth.p + 1);
  ILG_CUDA(cudaGetLastError());
  float pad = box_pad(c);
  k_refit<<<div_up(nt, 256), 256, 0, s>>>(c.tri_o.p, order.p, nt, child.p, parent.p, box_lo.p, box_hi.p, flags.p,
                                          pad, c.tri_s.p, depth.p);
  ILG_CUDA(cudaGetLastError());
  if (nt > 1) {
    dbuf<float4> slab_m;
    dbuf<float> slab_d;
    ILG_TRY(slab_m.alloc((size_t)2 * nt));
    ILG_TRY(slab_d.alloc((size_t)2 * nt));
    const int64_t warps = div_up(nt, 32) + (int64_t)(nt - 1);
    k_slabs<<<div_up(warps, 8), 256, 0, s>>>(c.tri_s.p, range.p, nt, 2.f * pad, slab_m.p, slab_d.p);
    ILG_CUDA(cudaGetLastError());
    ILG_TRY(c.nodes.alloc((size_t)(nt - 1) * NODE_W));
    k_pack_nodes<<<div_up(nt - 1, 256), 256, 0, s>>>(child.p, box_lo.p, box_hi.p, slab_m.p, slab_d.p, nt, c.nodes.p);
    ILG_CUDA(cudaGetLastError());
    c.root = 0;
  } else {
    ILG_TRY(c.nodes.alloc(NODE_W));
    c.root = ~0;
  }
  int dh2[2] = {0, 0};
  ILG_CUDA(cudaMemcpyAsync(dh2, depth.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  const int dh = dh2[0];
  c.bvh_depth = dh;
  c.bvh_longest = dh2[1];
  c.bvh_nodes = nt > 1 ? 2LL * nt - 1 : 1;
  if (dh + 2 > TRACE_STACK) {
    set_error("LBVH depth %d exceeds the traversal stack (%d)", dh, TRACE_STACK);
    return ILG_ERR_DEVICE;
  }
  return ILG_OK;
}

int bvh_trace(Context& c, int nrays, const float* orig_h, const float* dir_h, int any_hit, int32_t* hit_h,
              double* t_h) {
  if (nrays <= 0) return ILG_OK;
  cudaStream_t s = c.stream;
  dbuf<float> o, d;
  dbuf<int32_t> h;
  dbuf<double> t;
  ILG_TRY(o.alloc((size_t)nrays * 3));
  ILG_TRY(d.alloc((size_t)nrays * 3));
  ILG_TRY(h.alloc(nrays));
  ILG_TRY(t.alloc(nrays));
  ILG_CUDA(cudaMemcpyAsync(o.p, orig_h, (size_t)nrays * 12, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemcpyAsync(d.p, dir_h, (size_t)nrays * 12, cudaMemcpyHostToDevice, s));
  k_trace<<<div_up(nrays, 128), 128, 0, s>>>(c.nodes.p, c.tri_s.p, c.root, nrays, o.p, d.p, any_hit, h.p, t.p,
                                             c.derr.p);
  ILG_CUDA(cudaGetLastError());
  ILG_CUDA(cudaMemcpyAsync(hit_h, h.p, (size_t)nrays * 4, cudaMemcpyDeviceToHost, s));
  if (t_h) ILG_CUDA(cudaMemcpyAsync(t_h, t.p, (size_t)nrays * 8, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  return read_device_errors(c);
}

int bvh_render(Context& c, int mode, double az_deg, double el_deg, int width, int height, int32_t* out_h) {
  cudaStream_t s = c.stream;
  std::vector<float4> cen((size_t)c.nt);
  ILG_CUDA(cudaMemcpyAsync(cen.data(), c.cen.p, (size_t)c.nt * sizeof(float4), cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  double mx = 0, my = 0, mz = 0;
  for (const float4& q : cen) { mx += q.x; my += q.y; mz += q.z; }
  mx /= c.nt; my /= c.nt; mz /= c.nt;
  double r_model = 0;
  for (const float4& q : cen)
    r_model = std::max(r_model, std::sqrt((q.x - mx) * (q.x - mx) + (q.y - my) * (q.y - my) + (q.z - mz) * (q.z - mz)));
  RenderCam cam{};
  cam.mode = mode; cam.width = width; cam.height = height;
  cam.rad = 1.1 * r_model;
  cam.aspect = (double)width / height;
  const double D2R = 3.141592653589793 / 180.0;
  cam.az = az_deg * D2R;
  cam.el = el_deg * D2R;
  cam.cx = (float)mx; cam.cy = (float)my; cam.cz = (float)mz;
  if (mode == 0) {
    auto sph = [](double phi, double theta, double r, float* v) {
      v[0] = (float)(r * std::cos(phi) * std::sin(theta));
      v[1] = (float)(r * std::sin(phi) * std::sin(theta));
      v[2] = (float)(r * std::cos(theta));
    };
    float p[3], up[3];
    sph(cam.az, cam.el, cam.rad, p);
    sph(cam.az, cam.el - 3.141592653589793 / 2, 1.0, up);
    float pl = std::sqrt(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
    float e[3] = {-p[0] / pl, -p[1] / pl, -p[2] / pl};
    cam.ex = e[0]; cam.ey = e[1]; cam.ez = e[2];
    cam.ux = up[0]; cam.uy = up[1]; cam.uz = up[2];
    cam.rx = e[1] * up[2] - e[2] * up[1];   // n_eye x n_up
    cam.ry = e[2] * up[0] - e[0] * up[2];
    cam.rz = e[0] * up[1] - e[1] * up[0];
    cam.px = p[0] + cam.cx; cam.py = p[1] + cam.cy; cam.pz = p[2] + cam.cz;
  }
  const int64_t npx = (int64_t)width * height;
  dbuf<int32_t> dout;
  ILG_TRY(dout.alloc(npx));
  k_render<<<div_up(npx, 128), 128, 0, s>>>(c.nodes.p, c.tri_s.p, c.root, cam, dout.p, c.derr.p);
  ILG_CUDA(cudaGetLastError());
  ILG_CUDA(cudaMemcpyAsync(out_h, dout.p, (size_t)npx * 4, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  return read_device_errors(c);
}

// Bisection tree of src/cpp/illum.cpp:304-316 for a given theta_eps, in heap
// order (root 1, hit child 2k, miss child 2k+1). Node values are produced by
// exactly the reference's double arithmetic, so the returned mid values are
// the reference's.
static int build_horizon_tree(double theta_eps, std::vector<HorizonNode>& tree) {
  const int MAXD = 20;
  tree.assign(2, HorizonNode{});
  struct St { double lo, hi, mid; };
  std::vector<St> st(2);
  st[1] = St{0.0, PI, PI / 2.0};
  tree[1].mid = PI / 2.0;
  tree[1].terminal = 0;
  sincos_x(tree[1].mid, &tree[1].s, &tree[1].c);
  for (int depth = 0; depth < MAXD; ++depth) {
    size_t b = (size_t)1 << depth, e = (size_t)1 << (depth + 1);
    bool any = false;
    tree.resize(2 * e);
    st.resize(2 * e);
    for (size_t k = b; k < e; ++k) {
      if (tree[k].terminal || (k > 1 && tree[k].pad)) {   // pad marks unreachable
        tree[2 * k] = HorizonNode{0, 0, 0, 1, 1};
        tree[2 * k + 1] = HorizonNode{0, 0, 0, 1, 1};
        continue;
      }
      any = true;
      St cur = st[k];
      for (int h = 0; h < 2; ++h) {
        double lo = cur.lo, hi = cur.hi;
        if (h == 0) hi = cur.mid; else lo = cur.mid;
        double mid = (lo + hi) / 2.0;
        HorizonNode nd;
        nd.mid = mid;
        sincos_x(mid, &nd.s, &nd.c);
        nd.terminal = std::fabs(mid - cur.mid) > theta_eps ? 0 : 1;
        nd.pad = 0;
        tree[2 * k + h] = nd;
        st[2 * k + h] = St{lo, hi, mid};
      }
    }
    if (!any) { tree.resize(e); return ILG_OK; }
  }
  for (size_t k = (size_t)1 << MAXD; k < tree.size(); ++k)
    if (!tree[k].terminal) {
      set_error("theta_eps %g needs more than %d bisection levels", theta_eps, MAXD);
      return ILG_ERR_ARG;
    }
  return ILG_OK;
}

int horizons_build(Context& c, int nphi, double theta_eps, double offset, const Context* hmesh) {
  if (nphi < 2) { set_error("nphi must be >= 2"); return ILG_ERR_ARG; }
  if (!(theta_eps > 0.0)) { set_error("theta_eps must be > 0"); return ILG_ERR_ARG; }
  cudaStream_t s = c.stream;
  std::vector<HorizonNode> tree;
  ILG_TRY(build_horizon_tree(theta_eps, tree));
  for (HorizonNode& nd : tree) {
    nd.sdf = split_df_host(nd.s);
    nd.cdf = split_df_host(nd.c);
  }
  std::vector<double> cph(nphi), sph(nphi);
  double dphi = TWO_PI / (double)(nphi - 1);
  for (int k = 0; k < nphi; ++k) {
    double ph = (k == nphi - 1) ? TWO_PI : (double)k * dphi;   // arma::linspace
    sincos_x(ph, &sph[k], &cph[k]);
  }
  dbuf<HorizonNode> dtree;
  dbuf<double> dc, ds;
  ILG_TRY(dtree.alloc(tree.size()));
  ILG_TRY(dc.alloc(nphi));
  ILG_TRY(ds.alloc(nphi));
  ILG_CUDA(cudaMemcpyAsync(dtree.p, tree.data(), tree.size() * sizeof(HorizonNode), cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemcpyAsync(dc.p, cph.data(), nphi * 8, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemcpyAsync(ds.p, sph.data(), nphi * 8, cudaMemcpyHostToDevice, s));
  ILG_TRY(c.H.alloc((size_t)c.nt * nphi));
  // the rays of a separate horizon mesh's facets-independent BVH, or the
  // context's own (src/cpp/illum.cpp:333-360), where a facet's rays start at
  // its own leaf
  const Context& hb = hmesh ? *hmesh : c;
  const int slots = nphi >= 32 ? 1 : HZ_FACETS;
  const int warps = div_up(c.nt, slots);
  const bool near = !hmesh && rays_near(c, (float)offset);
  const int entries = near ? path_entries(c) : 1;
  const size_t smem = (size_t)(HZ_THREADS / 32) * slots * entries * sizeof(PathEntry);
  auto kern = near ? k_horizons<true> : k_horizons<false>;
  // the most that any launch asks for: the attribute is the kernel's, and other
  // contexts launch it at the same time
  constexpr size_t most = (size_t)(HZ_THREADS / 32) * HZ_FACETS * PATH_MOST * sizeof(PathEntry);
  ILG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  kern<<<div_up(warps, HZ_THREADS / 32), HZ_THREADS, smem, s>>>(
      hb.nodes.p, hb.tri_s.p, hb.root, c.parent.p, c.leaf_rank.p, c.frame.p, c.cen.p, c.nrm.p, c.nt,
      nphi, dc.p, ds.p, dtree.p, (int)tree.size(), (float)offset, slots, entries, c.H.p, c.derr.p);
  ILG_CUDA(cudaGetLastError());
  c.nphi = nphi;
  c.dphi = dphi;
  ILG_TRY(horizons_f32(c));
  return read_device_errors(c);
}

int horizons_f32(Context& c) {
  ILG_TRY(c.H32.alloc((size_t)c.nt * c.nphi));
  ILG_TRY(c.hmm32.alloc(c.nt));
  k_horizon_f32<<<div_up(c.nt, 256), 256, 0, c.stream>>>(c.H.p, c.nt, c.nphi, c.H32.p, c.hmm32.p);
  ILG_CUDA(cudaGetLastError());
  ILG_CUDA(cudaStreamSynchronize(c.stream));
  return ILG_OK;
}

// Keys held on the device at once (8 bytes each).
constexpr int64_t FF_CHUNK = int64_t(1) << 29;
// The chunk size in force (a test entry may lower it to exercise the
// several-chunk path on a small mesh).
std::atomic<int64_t> g_ff_chunk{FF_CHUNK};

int ff_set_chunk(int64_t pairs) {
  g_ff_chunk.store(pairs > 0 ? pairs : FF_CHUNK);
  return ILG_OK;
}

// The leaf groups of a build (LeafGroups over its own buffers).
struct GroupBufs {
  dbuf<float4> cen_s, lo[3], hi[3];
  dbuf<uint32_t> cnt;         // candidates per source (count_pairs)
  dbuf<uint2> units;          // of the chunk being cast
  LeafGroups G{};
  int build(const Context& c, double cutoff, cudaStream_t s) {
    const int nt = c.nt;
    G.nt = nt;
    G.order = c.morton_order.p;
    G.n[0] = div_up(nt, 32);
    G.n[1] = div_up(G.n[0], 32);
    G.n[2] = div_up(G.n[1], 32);
    ILG_TRY(cen_s.alloc(nt));
    for (int l = 0; l < 3; ++l) {
      ILG_TRY(lo[l].alloc(G.n[l]));
      ILG_TRY(hi[l].alloc(G.n[l]));
      G.lo[l] = lo[l].p;
      G.hi[l] = hi[l].p;
    }
    G.cen_s = cen_s.p;
    k_leaf_groups<<<div_up(nt, 256), 256, 0, s>>>(c.tri_s.p, c.cen.p, c.morton_order.p, nt, box_pad(c), cen_s.p,
                                                  lo[0].p, hi[0].p);
    ILG_CUDA(cudaGetLastError());
    for (int l = 1; l < 3; ++l) {
      k_group_boxes<<<div_up(G.n[l - 1], 256), 256, 0, s>>>(lo[l - 1].p, hi[l - 1].p, G.n[l - 1], lo[l].p, hi[l].p);
      ILG_CUDA(cudaGetLastError());
    }
    G.lim = -c.r_max - 1e-5f * c.scene_mag;
    G.cut2 = cutoff > 0.0 ? (float)(cutoff * cutoff) : -1.0f;
    // box test: the squared distance to a box is computed in float with at
    // most a few ulps of error; the margin keeps every centroid within the
    // cutoff reachable
    G.box_cut2 = cutoff > 0.0 ? (float)((cutoff + 1e-5 * c.scene_mag) * (cutoff + 1e-5 * c.scene_mag)) * 1.0001f
                              : -1.0f;
    return ILG_OK;
  }
};

// Candidate pairs per source (of the facets src, or all of them by Morton
// position): their exclusive sums, with the total behind them.
static int count_pairs(Context& c, GroupBufs& g, const int* src, int nsrc, std::vector<unsigned long long>& offs_h,
                       cudaStream_t s) {
  dbuf<unsigned long long> offs;
  ILG_TRY(g.cnt.alloc(nsrc));
  ILG_TRY(offs.alloc(nsrc));
  k_count_pairs<<<div_up(nsrc, 4), 128, 0, s>>>(g.G, c.nrm.p, c.cen.p, src, nsrc, g.cnt.p);
  ILG_CUDA(cudaGetLastError());
  ILG_TRY(scan_exclusive_u32_to_u64(g.cnt.p, offs.p, nsrc, c.scan, s));
  offs_h.resize((size_t)nsrc + 1);
  uint32_t last_cnt = 0;
  ILG_CUDA(cudaMemcpyAsync(offs_h.data(), offs.p, 8 * (size_t)nsrc, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaMemcpyAsync(&last_cnt, g.cnt.p + (nsrc - 1), 4, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  offs_h[nsrc] = offs_h[nsrc - 1] + last_cnt;
  return ILG_OK;
}

// The rays of sources [a, b), npairs in all: keys into ukeys (room for every
// pair), their number in *nk. counters: two words, ucount and (units, units
// taken).
static int cast_visibility(Context& c, GroupBufs& g, const int* src, int a, int b, int64_t npairs, float offset,
                           int bits, unsigned long long* ukeys, unsigned long long* counters, unsigned long long* nk,
                           cudaStream_t s) {
  ILG_CUDA(cudaMemsetAsync(counters, 0, 16, s));
  unsigned* nunits = reinterpret_cast<unsigned*>(counters + 1);
  const int warps = VIS_THREADS / 32, most = 152 * 16;   // blocks; warps take units from a counter
  const uint32_t part = (uint32_t)std::min<int64_t>(
      std::max<int64_t>(VIS_PART_MIN, npairs / ((int64_t)VIS_SHARES * 152 * 7 * warps)), 1 << 30);
  const int64_t cap = (int64_t)(b - a) + npairs / part;   // sum of ceil(count / part)
  ILG_TRY(g.units.reserve(cap));
  k_vis_units<<<div_up(b - a, 256), 256, 0, s>>>(g.cnt.p, a, b, part, g.units.p, nunits);
  ILG_CUDA(cudaGetLastError());
  const int blocks = (int)std::min<int64_t>((cap + warps - 1) / warps, most);
  const bool near = rays_near(c, offset);
  const int entries = near ? path_entries(c) : 1;
  const size_t smem = (size_t)warps * entries * sizeof(PathEntry);
  auto kern = near ? k_vis_rays<true> : k_vis_rays<false>;
  kern<<<blocks, VIS_THREADS, smem, s>>>(c.nodes.p, c.tri_s.p, c.root, c.parent.p, c.leaf_rank.p, g.G, c.cen.p, c.nrm.p,
                                               src, g.units.p, nunits, part, offset, bits, entries, nunits + 1,
                                               ukeys, counters, c.derr.p);
  ILG_CUDA(cudaGetLastError());
  ILG_CUDA(cudaMemcpyAsync(nk, counters, 8, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  return ILG_OK;
}

int form_factors_build(Context& c, const double* albedo_h, double albedo_scalar, double offset, double cutoff,
                       int64_t* rays_out) {
  cudaStream_t s = c.stream;
  int nt = c.nt;
  GroupBufs groups;
  ILG_TRY(groups.build(c, cutoff, s));
  std::vector<unsigned long long> offs_h;
  ILG_TRY(count_pairs(c, groups, nullptr, nt, offs_h, s));
  const int64_t npairs = (int64_t)offs_h[nt];
  if (rays_out) *rays_out = npairs;
  int bits = 1;
  while ((1LL << bits) < nt) ++bits;   // row and column fields

  // Sources (in Morton order) in chunks of at most FF_CHUNK pairs (a source
  // with more pairs is a chunk of its own): a chunk's keys, at most one per
  // pair, exist together.
  const int64_t chunk = g_ff_chunk.load();
  std::vector<int> cut{0};
  int64_t cap = 1;
  while (cut.back() < nt) {
    int a = cut.back(), b = a + 1;
    while (b < nt && (int64_t)(offs_h[b + 1] - offs_h[a]) <= chunk) ++b;
    cap = std::max<int64_t>(cap, (int64_t)(offs_h[b] - offs_h[a]));
    cut.push_back(b);
  }
  c.have_F = false;
  c.gs_ready = false;
  c.ntiles = 0;
  // Per chunk: its rays' distinct hit keys (sorted), their form factors, and
  // the kept entries (first occurrence, nonzero) packed into the chunk's own
  // arrays. Chunks own disjoint sources, so no key repeats across chunks and
  // only the kept entries outlive their chunk.
  std::vector<dbuf<unsigned long long>> ck;
  std::vector<dbuf<double>> cv;
  std::vector<int64_t> cn;
  {
    dbuf<unsigned long long> ukeys, ucount, pos;
    dbuf<uint32_t> keep;
    dbuf<double> fval, alb;
    ILG_TRY(ukeys.alloc(cap));
    ILG_TRY(ucount.alloc(2));
    if (albedo_h) {
      ILG_TRY(alb.alloc(nt));
      ILG_CUDA(cudaMemcpyAsync(alb.p, albedo_h, (size_t)nt * 8, cudaMemcpyHostToDevice, s));
    }
    for (size_t q = 0; q + 1 < cut.size(); ++q) {
      const int a = cut[q], b = cut[q + 1];
      const int64_t np = (int64_t)(offs_h[b] - offs_h[a]);
      if (np == 0) continue;
      unsigned long long nk = 0;
      ILG_TRY(cast_visibility(c, groups, nullptr, a, b, np, (float)offset, bits, ukeys.p, ucount.p, &nk, s));
      if (nk == 0) continue;
      if (nk > 1) ILG_TRY(radix_sort_u64(ukeys.p, nullptr, (int64_t)nk, 2 * bits, c.sort, s));
      ILG_TRY(keep.reserve(nk));
      ILG_TRY(fval.reserve(nk));
      ILG_TRY(pos.reserve(nk));
      k_ff_values<<<div_up((int64_t)nk, 256), 256, 0, s>>>(ukeys.p, (int64_t)nk, bits, nt, c.cen.p, c.nrm.p,
                                                          c.area.p, alb.p, albedo_scalar, keep.p, fval.p, c.derr.p);
      ILG_CUDA(cudaGetLastError());
      ILG_TRY(scan_exclusive_u32_to_u64(keep.p, pos.p, (int64_t)nk, c.scan, s));
      unsigned long long lp = 0;
      uint32_t lk = 0;
      ILG_CUDA(cudaMemcpyAsync(&lp, pos.p + (nk - 1), 8, cudaMemcpyDeviceToHost, s));
      ILG_CUDA(cudaMemcpyAsync(&lk, keep.p + (nk - 1), 4, cudaMemcpyDeviceToHost, s));
      ILG_CUDA(cudaStreamSynchronize(s));
      const int64_t nkeep = (int64_t)lp + lk;
      if (nkeep == 0) continue;
      ck.emplace_back();
      cv.emplace_back();
      ILG_TRY(ck.back().alloc(nkeep));
      ILG_TRY(cv.back().alloc(nkeep));
      cn.push_back(nkeep);
      k_ff_pack<<<div_up((int64_t)nk, 256), 256, 0, s>>>(ukeys.p, (int64_t)nk, keep.p, pos.p, fval.p,
                                                         ck.back().p, cv.back().p);
      ILG_CUDA(cudaGetLastError());
    }
  }
  int64_t nnz = 0;
  for (int64_t x : cn) nnz += x;
  if (nnz > (int64_t)0xffffffffLL) { set_error("%lld form-factor entries exceed the 32-bit entry index", (long long)nnz); return ILG_ERR_ARG; }
  ILG_TRY(read_device_errors(c));
  // all entries in (row, column) order: one chunk is sorted already; several
  // are concatenated and sorted by key, the values following the permutation
  dbuf<int32_t> rows;
  auto alloc_csr = [&]() -> int {
    ILG_TRY(rows.alloc(nnz > 0 ? nnz : 1));
    ILG_TRY(c.col.alloc(nnz > 0 ? nnz : 1));
    ILG_TRY(c.val.alloc(nnz > 0 ? nnz : 1));
    return ILG_OK;
  };
  ILG_TRY(c.rowptr.alloc((size_t)nt + 1));
  if (ck.size() <= 1) ILG_TRY(alloc_csr());
  if (ck.size() == 1) {
    k_ff_unpack<<<div_up(nnz, 256), 256, 0, s>>>(ck[0].p, nullptr, cv[0].p, nnz, bits, rows.p, c.col.p, c.val.p);
    ILG_CUDA(cudaGetLastError());
    ck.clear();
    cv.clear();
  } else if (ck.size() > 1) {
    dbuf<unsigned long long> ekeys;
    dbuf<double> evals;
    dbuf<uint32_t> eidx;
    ILG_TRY(ekeys.alloc(nnz));
    ILG_TRY(evals.alloc(nnz));
    int64_t off = 0;
    for (size_t q = 0; q < ck.size(); ++q) {
      ILG_CUDA(cudaMemcpyAsync(ekeys.p + off, ck[q].p, (size_t)cn[q] * 8, cudaMemcpyDeviceToDevice, s));
      ILG_CUDA(cudaMemcpyAsync(evals.p + off, cv[q].p, (size_t)cn[q] * 8, cudaMemcpyDeviceToDevice, s));
      off += cn[q];
      ck[q].release();
      cv[q].release();
    }
    ck.clear();
    cv.clear();
    ILG_TRY(eidx.alloc(nnz));
    k_iota_u32<<<div_up(nnz, 256), 256, 0, s>>>(eidx.p, nnz);
    ILG_CUDA(cudaGetLastError());
    ILG_TRY(radix_sort_u64(ekeys.p, eidx.p, nnz, 2 * bits, c.sort, s));
    c.sort.release();
    ILG_TRY(alloc_csr());
    k_ff_unpack<<<div_up(nnz, 256), 256, 0, s>>>(ekeys.p, eidx.p, evals.p, nnz, bits, rows.p, c.col.p, c.val.p);
    ILG_CUDA(cudaGetLastError());
  }
  k_rowptr<<<div_up(nt + 1, 256), 256, 0, s>>>(rows.p, nnz, nt, c.rowptr.p);
  ILG_CUDA(cudaGetLastError());
  ILG_CUDA(cudaStreamSynchronize(s));
  c.nnz = nnz;
  c.have_F = true;
  rows.release();
  ILG_TRY(radiosity_prepare(c));
  // the sort and scan scratch grew to the entry count: not kept resident
  c.sort.release();
  c.scan.release();
  if (nnz > (int64_t(1) << 26)) ILG_TRY(pool_trim(s));
  return read_device_errors(c);
}

int visibility_sample(Context& c, double cutoff, double offset, const int* src_h, int nsrc, const double* radii_h,
                      int nradii, int64_t* per_src_h, int64_t* within_h, int64_t* rays_out) {
  if (nsrc < 1 || !src_h || nradii < 0 || (nradii > 0 && !radii_h)) { set_error("invalid sample"); return ILG_ERR_ARG; }
  cudaStream_t s = c.stream;
  const int nt = c.nt;
  std::vector<int> slot_h((size_t)nt, -1);
  for (int q = 0; q < nsrc; ++q) {
    if (src_h[q] < 0 || src_h[q] >= nt) { set_error("source %d out of range", src_h[q]); return ILG_ERR_ARG; }
    if (slot_h[src_h[q]] >= 0) { set_error("source %d listed twice", src_h[q]); return ILG_ERR_ARG; }
    slot_h[src_h[q]] = q;
  }
  dbuf<int> dsrc, dslot;
  dbuf<double> dradii;
  dbuf<unsigned long long> per_src, within, ukeys, ucount;
  ILG_TRY(dsrc.alloc(nsrc));
  ILG_TRY(dslot.alloc(nt));
  ILG_TRY(dradii.alloc(std::max(nradii, 1)));
  ILG_TRY(per_src.alloc(nsrc));
  ILG_TRY(within.alloc(std::max(nradii, 1)));
  ILG_TRY(ucount.alloc(2));
  ILG_CUDA(cudaMemcpyAsync(dsrc.p, src_h, (size_t)nsrc * 4, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemcpyAsync(dslot.p, slot_h.data(), (size_t)nt * 4, cudaMemcpyHostToDevice, s));
  if (nradii > 0) ILG_CUDA(cudaMemcpyAsync(dradii.p, radii_h, (size_t)nradii * 8, cudaMemcpyHostToDevice, s));
  ILG_CUDA(cudaMemsetAsync(per_src.p, 0, (size_t)nsrc * 8, s));
  ILG_CUDA(cudaMemsetAsync(within.p, 0, (size_t)std::max(nradii, 1) * 8, s));
  GroupBufs groups;
  ILG_TRY(groups.build(c, cutoff, s));
  std::vector<unsigned long long> offs_h;
  ILG_TRY(count_pairs(c, groups, dsrc.p, nsrc, offs_h, s));
  if (rays_out) *rays_out = (int64_t)offs_h[nsrc];
  int bits = 1;
  while ((1LL << bits) < nt) ++bits;
  // chunks of at most FF_CHUNK candidate pairs; each chunk's distinct hit
  // keys are sorted, counted and dropped (the sample's keys never coexist)
  std::vector<int> cutq{0};
  int64_t cap = 1;
  while (cutq.back() < nsrc) {
    int a = cutq.back(), b = a + 1;
    while (b < nsrc && (int64_t)(offs_h[b + 1] - offs_h[a]) <= FF_CHUNK) ++b;
    cap = std::max<int64_t>(cap, (int64_t)(offs_h[b] - offs_h[a]));
    cutq.push_back(b);
  }
  ILG_TRY(ukeys.alloc(cap));
  for (size_t q = 0; q + 1 < cutq.size(); ++q) {
    const int a = cutq[q], b = cutq[q + 1];
    const int64_t np = (int64_t)(offs_h[b] - offs_h[a]);
    if (np == 0) continue;
    unsigned long long nk = 0;
    ILG_TRY(cast_visibility(c, groups, dsrc.p, a, b, np, (float)offset, bits, ukeys.p, ucount.p, &nk, s));
    if (nk > 1) ILG_TRY(radix_sort_u64(ukeys.p, nullptr, (int64_t)nk, 2 * bits, c.sort, s));
    if (nk > 0) {
      k_sample_count<<<div_up((int64_t)nk, 256), 256, 0, s>>>(ukeys.p, (int64_t)nk, bits, c.cen.p, c.nrm.p, c.area.p,
                                                             dslot.p, dradii.p, nradii, per_src.p, within.p);
      ILG_CUDA(cudaGetLastError());
    }
  }
  ILG_CUDA(cudaMemcpyAsync(per_src_h, per_src.p, (size_t)nsrc * 8, cudaMemcpyDeviceToHost, s));
  if (nradii > 0 && within_h) ILG_CUDA(cudaMemcpyAsync(within_h, within.p, (size_t)nradii * 8, cudaMemcpyDeviceToHost, s));
  ILG_CUDA(cudaStreamSynchronize(s));
  return read_device_errors(c);
}

}  // namespace ilg
