// gpv_kernels.cu -- sm_103a kernels of the Level1 stage, batched over meshes.
//
// Pipeline (all on one stream; a plain voxelization is a batch of one):
//   k_prep        per triangle: pack vertices as 3 float4, Level1 SAT candidate box (the
//                 reference's own range, src/Object.cpp:2280-2325), conservative x/y box for the
//                 ray tests, 1/det of the ray test, work counts.
//   k_level1      persistent: warps pull tickets of triangles from a device queue; groups of 32 are
//                 staged in shared memory by bulk async copies (TMA) on the warp's mbarriers.
//                 (a) SAT units = (triangle, column) running the z run top-down, cut to the
//                     triangle's plane; passes set the boundary bit (atomicOr) and emit
//                     (column-major voxel key, triangle|topmost).
//                 (b) fill units = (triangle, column) running the column part of the +z
//                     Moller-Trumbore test; a passing unit XORs the parity toggles
//                     d(k) = hit(k) ^ hit(k+1) into a column-major plane, from the triangle's height
//                     over the column.
//   k_fill_finish suffix XOR of the toggles per column -> parity, transposed to the linear (x fastest)
//                 inside plane; the boundary plane transposed to the pair keys' order.
//   scan          per-word boundary counts, boundaryPrefixSum.
//   k_expand      .raw bytes of Level1, boundaryPrefixSum, boundaryIndex.
//   sort / Level2 gpv_sort.cu, gpv_level2.cu.
#include "gpv_internal.h"
#include "gpv_rows.cuh"

namespace gpv {

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ uint32_t pack2(int lo, int hi) {
  return (uint32_t)(lo & 0xffff) | ((uint32_t)(hi & 0xffff) << 16);
}
__device__ __forceinline__ int lo16(uint32_t v) { return (int)(v & 0xffffu); }
__device__ __forceinline__ int hi16(uint32_t v) { return (int)(v >> 16); }

// smallest i in [0,n] with tab[i] >= x (tab nondecreasing of spacing ~1 / inv from c0); approximate
// start then adjust.
__device__ __forceinline__ int first_ge(const float *tab, int n, float x, float c0, float inv) {
  float f = (x - c0) * inv;
  int i;
  if (!(f > 0.f)) i = 0;
  else if (f >= (float)n) i = n;
  else i = (int)ceilf(f);
  while (i > 0 && __ldg(tab + i - 1) >= x) --i;
  while (i < n && __ldg(tab + i) < x) ++i;
  return i;
}
// largest i in [-1,n-1] with tab[i] <= x.
__device__ __forceinline__ int last_le(const float *tab, int n, float x, float c0, float inv) {
  float f = (x - c0) * inv;
  int i;
  if (!(f > 0.f)) i = -1;
  else if (f >= (float)n) i = n - 1;
  else i = (int)floorf(f);
  while (i < n - 1 && __ldg(tab + i + 1) <= x) ++i;
  while (i >= 0 && __ldg(tab + i) > x) --i;
  return i;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const unsigned lane = threadIdx.x & 31u;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t o = __shfl_up_sync(FULL, v, d);
    if (lane >= (unsigned)d) v += o;
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
  return v;
}

// Adds v to *dst once per warp when every lane targets the same counter, else per lane.
__device__ __forceinline__ void warp_add(unsigned long long *dst, unsigned long long v) {
  const unsigned long long a = (unsigned long long)dst;
  if (__all_sync(FULL, __shfl_sync(FULL, a, 0) == a)) {
    v = warp_sum(v);
    if ((threadIdx.x & 31u) == 0 && v) atomicAdd(dst, v);
  } else if (v) {
    atomicAdd(dst, v);
  }
}

// The prep counters of a 256-thread block: one atomic each per block when every thread of
// the block works on the same mesh (the common case), else per warp.  Thousands of per-warp
// atomics on one counter serialise at L2.
__device__ __forceinline__ void block_add_prep(MeshStats *st, unsigned long long a,
                                               unsigned long long b, unsigned long long c,
                                               unsigned long long d) {
  __shared__ unsigned long long s_acc[4][8];
  __shared__ MeshStats *s_first;
  if (threadIdx.x == 0) s_first = st;
  __syncthreads();
  if (__syncthreads_and(st == s_first)) {
    a = warp_sum(a); b = warp_sum(b); c = warp_sum(c); d = warp_sum(d);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) {
      s_acc[0][warp] = a; s_acc[1][warp] = b; s_acc[2][warp] = c; s_acc[3][warp] = d;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
      unsigned long long v = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += s_acc[threadIdx.x][w];
      unsigned long long *dst = threadIdx.x == 0 ? &st->sat1 : threadIdx.x == 1 ? &st->sat_units
                                : threadIdx.x == 2 ? &st->fill_units : &st->ray1;
      if (v) atomicAdd(dst, v);
    }
  } else {
    warp_add(&st->sat1, a);
    warp_add(&st->sat_units, b);
    warp_add(&st->fill_units, c);
    warp_add(&st->ray1, d);
  }
}

// Conservative x/y box of the columns whose +z ray can pass the u/v tests of this triangle.
// Outside the box every column fails them in float arithmetic; ill-conditioned projections get
// the whole plane; triangles failing the |det| test get an empty box.
__device__ __forceinline__ float4 ray_box(const float *V, const GridDev &g) {
  const float e1x = fs(V[3], V[0]), e1y = fs(V[4], V[1]);
  const float e2x = fs(V[6], V[0]), e2y = fs(V[7], V[1]);
  const float det = fa(fm(e1x, -e2y), fm(e1y, e2x));
  const float inf = __int_as_float(0x7f800000);
  if (!(det < -g.thr || det > g.thr)) return make_float4(inf, inf, -inf, -inf);
  const float adet = fabsf(det);
  const float sd = fabsf(e1x * e2y) + fabsf(e1y * e2x);
  const float rel = 4.f * EPS24 * sd / adet;
  if (!(rel <= 0.125f)) return make_float4(-inf, -inf, inf, inf);
  float G = fmaxf(fmaxf(fabsf(g.bmin[0] - V[0]), fabsf(g.bmax[0] - V[0])),
                  fmaxf(fabsf(g.bmin[1] - V[1]), fabsf(g.bmax[1] - V[1])));
  G = G * 1.0001f + 1e-30f;
  const float au = 4.f * EPS24 * G * (fabsf(e2x) + fabsf(e2y)) / adet;
  const float av = 4.f * EPS24 * G * (fabsf(e1x) + fabsf(e1y)) / adet;
  const float mu = 2.f * (rel + au + av) + 1e-6f;
  float lo[2], hi[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    float mn = fminf(V[a], fminf(V[3 + a], V[6 + a]));
    float mx = fmaxf(V[a], fmaxf(V[3 + a], V[6 + a]));
    float w = mx - mn;
    float m = 2.f * mu * w + 8.f * EPS24 * (fabsf(mn) + fabsf(mx) + w) + 1e-30f;
    lo[a] = mn - m;
    hi[a] = mx + m;
  }
  return make_float4(lo[0], lo[1], hi[0], hi[1]);
}

// ---------------------------------------------------------------------------------------------
constexpr int kHeavyUnits = 64;   // a triangle with more (triangle, column) units is split ...
constexpr int kHeavyChunks = 4;   // ... into pieces of this many 32-unit chunks, or
// ... or of one in calls of few triangles where its box has more than kLongRun layers: a wall's columns
// run through all of them (12 triangles of a box on 100x70x88, the no-alloc call: 220 us in pieces of four
// chunks, 121 of one); with many triangles the other pieces hide it, and the list has room for longer ones
constexpr int kLongRun = 32, kFewTriangles = 4096;

// cell_of(v) from its estimate e = (v - mn) * inv, inv = n / (mx - mn).  The float quotient times n is
// within four roundings of e, an absolute 1e-6 covering inv's denormals: where both ends truncate to one
// cell that is it, elsewhere (about one in 10^4, and where inv or e overflow) the quotient itself decides.
__device__ __forceinline__ int cell_near(float v, float mn, float mx, int n, float inv) {
  const float e = (v - mn) * inv, w = ff(fabsf(e), 8.f * EPS24, 1e-6f), nf = (float)n + 1.0f;
  const int a = __float2int_rz(fminf(fmaxf(e - w, -1.0f), nf)), b = __float2int_rz(fminf(fmaxf(e + w, -1.0f), nf));
  if (a != b || !(w < 1e30f)) return cell_of(v, mn, mx, n);  // (NaN too)
  return a == n && v == mx ? a - 1 : a;
}

// Bound by latency (loads, then the table searches), at 45% of the issue slots: 1.3M triangles in 51 us.
// (57 with nine quotients and a divide for each table search; triangles read, or read and written, by
// consecutive lanes through shared memory took 53-71: the barriers cost more than the partial lines.)
__global__ void __launch_bounds__(256) k_prep(BatchDev bd) {
  const int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = gi < bd.total_tris;
  const int m = find_mesh<&MeshDesc::tri_base>(bd.md, bd.nmesh, live ? gi : bd.total_tris - 1);
  const MeshDesc &d = bd.md[m];
  const GridDev &g = d.g;
  unsigned long long sat1 = 0, su = 0, fu = 0, r1 = 0;
  uint32_t pieces = 0, chunks = 0;
  if (live) {
    const int64_t t = gi - d.tri_base;
    float V[9];
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      V[k] = __ldg(d.tris + 9 * t + k);
      finite = finite && isfinite(V[k]);
    }
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // cell_of grows with v but for the step down from n to n - 1 at v == max, so the cells of the
      // smallest and the largest coordinate bound the third's unless that one is at max, where the
      // smallest may lie just under it, in cell n (a hi past the last cell is cut to it)
      const float inv = (float)g.n[a] / (g.bmax[a] - g.bmin[a]);
      const int c0 = cell_near(fminf(V[a], fminf(V[3 + a], V[6 + a])), g.bmin[a], g.bmax[a], g.n[a], inv);
      const int c1 = cell_near(fmaxf(V[a], fmaxf(V[3 + a], V[6 + a])), g.bmin[a], g.bmax[a], g.n[a], inv);
      const bool at_max = V[a] == g.bmax[a] || V[3 + a] == g.bmax[a] || V[6 + a] == g.bmax[a];
      lo[a] = max(min(c0, at_max ? min(c1, g.n[a] - 1) : c1), 0);
      hi[a] = min(max(c0, c1), g.n[a] - 1);
    }
    float4 fb = ray_box(V, g);
    int fx0 = 1, fx1 = 0, fy0 = 1, fy1 = 0;
    if (!finite) {
      atomicOr(&d.stats->status, (unsigned)ST_BAD_INPUT);
      lo[0] = 1; hi[0] = 0;
      fb = make_float4(1.f, 1.f, 0.f, 0.f);
    } else {
      const float ix = 1.f / g.g[0], iy = 1.f / g.g[1];
      fx0 = first_ge(g.c1[0], g.n[0], fb.x, g.c1[0][0], ix);
      fx1 = last_le(g.c1[0], g.n[0], fb.z, g.c1[0][0], ix);
      fy0 = first_ge(g.c1[1], g.n[1], fb.y, g.c1[1][0], iy);
      fy1 = last_le(g.c1[1], g.n[1], fb.w, g.c1[1][0], iy);
      // exact x/y box of the triangle for the ray1 work count
      const float mnx = fminf(V[0], fminf(V[3], V[6])), mxx = fmaxf(V[0], fmaxf(V[3], V[6]));
      const float mny = fminf(V[1], fminf(V[4], V[7])), mxy = fmaxf(V[1], fmaxf(V[4], V[7]));
      const int ax = last_le(g.c1[0], g.n[0], mxx, g.c1[0][0], ix) -
                     first_ge(g.c1[0], g.n[0], mnx, g.c1[0][0], ix) + 1;
      const int ay = last_le(g.c1[1], g.n[1], mxy, g.c1[1][0], iy) -
                     first_ge(g.c1[1], g.n[1], mny, g.c1[1][0], iy) + 1;
      if (ax > 0 && ay > 0) r1 = (unsigned long long)ax * ay * g.n[2];
    }
    const bool sat_ok = lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2];
    if (sat_ok) {
      su = (unsigned long long)(hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1);
      sat1 = su * (hi[2] - lo[2] + 1);
    } else {
      lo[0] = 1; hi[0] = 0;
    }
    if (fx0 <= fx1 && fy0 <= fy1) fu = (unsigned long long)(fx1 - fx0 + 1) * (fy1 - fy0 + 1);
    else { fx0 = 1; fx1 = 0; fy0 = 1; fy1 = 0; }
    if (bd.fill != GPV_FILL_RAY) {  // the stencil kernel fills instead (or nothing fills)
      fx0 = 1; fx1 = 0; fy0 = 1; fy1 = 0;
      fu = 0;
      r1 = 0;
    }
    // 1/det of the +z ray test (src/TriRayIntersection.cpp:99), shared by every column
    const float det = fa(fm(fs(V[3], V[0]), -fs(V[7], V[1])), fm(fs(V[4], V[1]), fs(V[6], V[0])));
    d.ptri[3 * t + 0] = make_float4(V[0], V[1], V[2], __uint_as_float(pack2(fx0, fx1)));
    d.ptri[3 * t + 1] = make_float4(V[3], V[4], V[5], __uint_as_float(pack2(fy0, fy1)));
    d.ptri[3 * t + 2] = make_float4(V[6], V[7], V[8], __fdiv_rn(1.0f, det));
    d.rng[t] = make_int4((int)pack2(lo[0], hi[0]), (int)pack2(lo[1], hi[1]), (int)pack2(lo[2], hi[2]), 0);
    d.fbox[t] = fb;
    if (bd.heavy && su + fu > (unsigned long long)kHeavyUnits) {
      chunks = sat_ok && hi[2] - lo[2] >= kLongRun && bd.total_tris <= kFewTriangles ? 1u : (uint32_t)kHeavyChunks;
      const unsigned long long n = ((su + 31) / 32 + (fu + 31) / 32 + chunks - 1) / chunks;
      if (n <= bd.heavy_cap) pieces = (uint32_t)n;
    }
  }
  // A triangle with many units (large against the cells) goes to the heavy list, in pieces of
  // `chunks` chunks that any warp of the Level1 kernel takes, and is flagged so that its group
  // leaves it out; where the list is full it stays with its group.  One atomic a warp: one a triangle
  // took 120 us where 262k triangles were all heavy.
  if (__any_sync(FULL, pieces != 0u)) {
    const uint32_t inc = warp_incl_scan(pieces);  // (32 lanes of at most kHeavyCap)
    unsigned long long pos = 0;
    if ((threadIdx.x & 31u) == 31u) pos = atomicAdd(bd.heavy_n, (unsigned long long)inc);
    pos = __shfl_sync(FULL, pos, 31) + (inc - pieces);
    if (pieces) {
      const unsigned long long cap = bd.heavy_cap;
      const int64_t t = gi - d.tri_base;
      const bool listed = pos < cap && cap - pos >= pieces;
      if (listed) d.rng[t].w = 1;
      const uint32_t room = pos < cap ? (uint32_t)min(cap - pos, (unsigned long long)pieces) : 0u;
      for (uint32_t k = 0; k < room; ++k)
        bd.heavy[pos + k] = make_uint4((uint32_t)m, (uint32_t)t, k, listed ? chunks : 0u);
    }
  }
  block_add_prep(d.stats, sat1, su, fu, r1);
}

// Per-mesh pair emission segments from the candidate counts prep just produced: exclusive prefix
// of sat1 over the meshes, capped by the buffer capacity (a mesh past the end gets a short or
// empty segment; its Level1 then raises ST_PAIR_OVERFLOW).  One block; meshes in rounds of 1024.
__global__ void __launch_bounds__(1024) k_pair_bases(int nmesh, MeshDesc *md, uint32_t *keys,
                                                     uint32_t *vals, int64_t cap) {
  __shared__ unsigned long long s_w[32];
  __shared__ unsigned long long s_carry;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int m0 = 0; m0 < nmesh; m0 += 1024) {
    const int m = m0 + (int)threadIdx.x;
    const unsigned long long v = m < nmesh ? md[m].stats->sat1 : 0ull;
    unsigned long long x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long o = __shfl_up_sync(FULL, x, d);
      if (lane >= (unsigned)d) x += o;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    if (warp == 0) {
      unsigned long long w = s_w[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long o = __shfl_up_sync(FULL, w, d);
        if (lane >= (unsigned)d) w += o;
      }
      s_w[lane] = w;
    }
    __syncthreads();
    const unsigned long long base = s_carry + (warp ? s_w[warp - 1] : 0ull) + x - v;
    if (m < nmesh) {
      const int64_t b = (int64_t)base;
      md[m].emit_base = b;
      md[m].pair_cap = max((int64_t)0, min((int64_t)v, cap - b));
      md[m].keys = keys + min(b, cap);
      md[m].vals = vals + min(b, cap);
    }
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = base + v;
    __syncthreads();
  }
}

// One-graph calls: the second half's per-mesh bases and sizes from the first half's counts (one
// block; meshes in rounds of 1024, six running sums scanned together).  The sums, per mesh:
// 0 boundary voxels (boundaryIndex slices), 1 the same for meshes with a Level2 grid (sorted
// segments), 2 their Level2 bytes, 3 their pair-sort tiles, 4 their pairs, 5 meshes with a raised
// status.
constexpr int kPlanSums = 6;
__global__ void __launch_bounds__(1024) k_plan(int nmesh, MeshDesc *md, int32_t *bindex,
                                               uint8_t *l2, PlanCaps caps,
                                               DevPlan *plan) {
  __shared__ unsigned long long s_w[32][kPlanSums];
  __shared__ unsigned long long s_carry[kPlanSums];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x < kPlanSums) s_carry[threadIdx.x] = 0;
  __syncthreads();
  for (int m0 = 0; m0 < nmesh; m0 += 1024) {
    const int m = m0 + (int)threadIdx.x;
    unsigned long long v[kPlanSums] = {};
    if (m < nmesh) {
      const MeshStats &st = *md[m].stats;
      const bool has = md[m].has_l2 != 0;
      const unsigned long long b = st.boundary, p = st.pairs;
      const unsigned long long cells =
          (unsigned long long)md[m].g.n2[0] * md[m].g.n2[1] * md[m].g.n2[2];
      v[0] = b;
      v[1] = has ? b : 0ull;
      v[2] = has ? b * cells : 0ull;
      v[3] = has ? (p + kSortTileItems - 1) / kSortTileItems : 0ull;
      v[4] = has ? p : 0ull;
      v[5] = st.status != 0u;
    }
    unsigned long long x[kPlanSums];
#pragma unroll
    for (int k = 0; k < kPlanSums; ++k) {
      x[k] = v[k];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long o = __shfl_up_sync(FULL, x[k], d);
        if (lane >= (unsigned)d) x[k] += o;
      }
      if (lane == 31) s_w[warp][k] = x[k];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int k = 0; k < kPlanSums; ++k) {
        unsigned long long w = s_w[lane][k];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const unsigned long long o = __shfl_up_sync(FULL, w, d);
          if (lane >= (unsigned)d) w += o;
        }
        s_w[lane][k] = w;
      }
    }
    __syncthreads();
    if (m < nmesh) {
      unsigned long long e[kPlanSums];
#pragma unroll
      for (int k = 0; k < kPlanSums; ++k)
        e[k] = s_carry[k] + (warp ? s_w[warp - 1][k] : 0ull) + x[k] - v[k];
      md[m].u_base = (int64_t)e[1];
      md[m].pair_base = (int64_t)e[4];
      md[m].stile_base = (int64_t)e[3];
      md[m].l2_base = (int64_t)e[2];
      md[m].bindex = bindex + min((long long)e[0], (long long)caps.B);
      md[m].l2 = l2 + min((long long)e[2], (long long)caps.l2bytes);
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < kPlanSums; ++k) s_carry[k] += s_w[31][k];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const unsigned long long *t = s_carry;
    DevPlan p;
    p.ok = t[5] == 0 && t[0] <= (unsigned long long)caps.B && t[1] <= (unsigned long long)caps.U &&
           t[2] <= (unsigned long long)caps.l2bytes && t[3] <= (unsigned long long)caps.tiles &&
           t[4] <= (unsigned long long)caps.P;
    p.ub = (uint32_t)min(t[1], 0xffffffffull);
    p.ntiles = (uint32_t)min(t[3], 0xffffffffull);
    p.P2 = t[4];
    p.Btot = t[0];
    p.l2bytes = t[2];
    *plan = p;
  }
}

// ---------------------------------------------------------------------------------------------
constexpr int kPlaneRun = 4;   // z runs past this many voxels are cut to the triangle's plane first
constexpr int kL1Warps = 4;
constexpr int kL1Group = 32;   // triangles of one group (a lane each)
constexpr int kL1Pairs = 128;  // records a warp collects before it takes room for them
constexpr uint32_t kWaitLimit = 1u << 22;

// last index lt in [0, 31] with off[lt] <= u (off nondecreasing, off[0] = 0)
__device__ __forceinline__ int group_search(const uint32_t *off, uint32_t u) {
  int lo = 0;
#pragma unroll
  for (int st = 16; st > 0; st >>= 1)
    if (off[lo + st] <= u) lo += st;
  return lo;
}

struct L1Warp {
  float4 tri[3 * kL1Group];  // the staged group
  int4 rng[kL1Group];
  uint32_t soff[kL1Group], foff[kL1Group];  // exclusive prefixes of the SAT and fill units
  uint32_t key[kL1Pairs], val[kL1Pairs];    // collected records
  uint64_t bar;
  // the current mesh's grid and planes: a shared copy, since every global atomic makes the compiler
  // read the descriptor's fields again
  GridDev g;
  uint32_t *bplane, *toggles;
};

// A group of consecutive triangles of one mesh and this warp's share of its chunks of units: every
// S-th from the part-th, or (a piece of a heavy triangle) `piece` of them from there.
constexpr int kNoItemYet = -2;
struct L1Item {
  int m;           // mesh, -1: none left
  int64_t t0;      // first triangle
  int64_t tend;    // end of the ticket's triangles
  uint32_t part;
  uint32_t piece;  // 0: no piece
};

// z interval outside which the SAT's plane test fails for certain in the column at (cx, cy): on
// return [z0, z1] is cut to it.  With R the largest |V - c| (edges up to 2 R), the float test's value
// is within 264 eps R^2 (R + h) of exact and the one below within 200; E has room for twice both and
// for the distance of the z table from its affine form, so cells past H + E are rejected by the test.
__device__ __forceinline__ void plane_range(const float *V, const GridDev &g, float cx, float cy,
                                            int &z0, int &z1) {
  const float a0 = V[3] - V[0], a1 = V[4] - V[1], a2 = V[5] - V[2];
  const float b0 = V[6] - V[3], b1 = V[7] - V[4], b2 = V[8] - V[5];
  const float nx = a1 * b2 - a2 * b1, ny = a2 * b0 - a0 * b2;
  float nz = a0 * b1 - a1 * b0;
  const float ca = __ldg(g.c1[2] + z0), cb = __ldg(g.c1[2] + z1);
  float R = 0.f;  // the largest |V - c| of the run
#pragma unroll
  for (int i = 0; i < 9; i += 3)
    R = fmaxf(R, fmaxf(fmaxf(fabsf(V[i] - cx), fabsf(V[i + 1] - cy)), fmaxf(fabsf(V[i + 2] - ca), fabsf(V[i + 2] - cb))));
  R = fmaxf(R * 1.0001f, fmaxf(g.e1[0], fmaxf(g.e1[1], g.e1[2])));
  if (!(R > 1e-9f && R < 1e9f)) return;
  const float h = fmaxf(g.e1[0], fmaxf(g.e1[1], g.e1[2]));
  const float E = 1024.f * EPS24 * R * R * (R + h) + 2.4f * EPS24 * fmaxf(fabsf(ca), fabsf(cb)) * fabsf(nz);
  const float H = fabsf(nx) * g.e1[0] + fabsf(ny) * g.e1[1] + fabsf(nz) * g.e1[2] + E;
  const float s = nx * (V[0] - cx) + ny * (V[1] - cy);
  nz = copysignf(fmaxf(fabsf(nz), E * rcp_fast(512.f * R)), nz);  // (moves the value by less than E/512)
  const float rn = rcp_fast(nz), ig = rcp_fast(2.f * g.e1[2]);
  const float zc = V[2] - ca;
  const float x1 = (zc + (s - H) * rn) * ig, x2 = (zc + (s + H) * rn) * ig;  // layers above z0
  const float w = 16.f * EPS24 * (float)(z1 - z0) + 1e-4f;  // index arithmetic
  const int b = z0;
  z0 = b + min(max(__float2int_ru(fminf(x1, x2) - w - 16.f * EPS24 * fmaxf(fabsf(x1), fabsf(x2))), 0), z1 - b + 1);
  z1 = b + min(__float2int_rd(fmaxf(x1, x2) + w + 16.f * EPS24 * fmaxf(fabsf(x1), fabsf(x2))), z1 - b);
}

// Toggles of one (triangle, column) pair that passed u/v: d(k) = hit(k) ^ hit(k + 1).  The exact t*
// falls by the rise of the origin, so the hits are the voxels under the triangle's plane over the
// column; X = the plane's height over the first centre, less 1e-6, in voxels.  As in the Level2 fill
// the float t decides as t* outside 1.35 (8.2 eps M0 / |det| + 1e-6) of the crossing (rel <= 1/8),
// X is off by about as much and by the centre table's distance from its affine form, and only the
// voxels within that of the crossing (all of them for an ill-conditioned projection) run the test.
__device__ __forceinline__ void column_toggles(const RayTri &rt, const RayCol &rc, const GridDev &g,
                                               uint32_t *tog, size_t stride) {
  const int nz = g.n[2];
  const float *oz = g.c1[2];
  const float ad = fabsf(rt.inv_det);
  const float sd = fabsf(rt.e1x * rt.e2y) + fabsf(rt.e1y * rt.e2x);
  int n1 = 0, n2 = nz;  // hits below n1 and misses from n2 for certain
  if (4.f * EPS24 * sd * ad <= 0.125f) {
    const float o0 = __ldg(oz), ig = rcp_fast(2.f * g.e1[2]);
    const float atx = fabsf(rc.Tx), aty = fabsf(rc.Ty);
    const float zt2 = 2.f * fmaxf(fabsf(rt.e1z), fmaxf(fabsf(rt.e2z), fabsf(rt.e2z - rt.e1z)));
    const float M0 = fabsf(rt.e2x) * (aty * fabsf(rt.e1z) + zt2 * fabsf(rt.e1y)) +
                     fabsf(rt.e2y) * (zt2 * fabsf(rt.e1x) + atx * fabsf(rt.e1z)) +
                     fabsf(rt.e2z) * (atx * fabsf(rt.e1y) + aty * fabsf(rt.e1x));
    const float t0 = (rt.e2x * (rc.Ty * rt.e1z) - rt.e2y * (rc.Tx * rt.e1z) +
                      rt.e2z * (rc.Tx * rt.e1y - rc.Ty * rt.e1x)) * rt.inv_det;
    const float X = ((rt.v1z - o0) + t0 - g.thr) * ig;
    const float w = ig * (EPS24 * (40.f * M0 * ad + 8.f * zt2 +
                                   4.2f * fmaxf(fabsf(g.bmin[2]), fabsf(g.bmax[2]))) + 0.35f * g.thr) +
                    16.f * EPS24 * (float)nz + 1e-4f;
    if (w < 1e6f) {  // (false for NaN too)
      n1 = min(max(__float2int_ru(X - w), 0), nz);
      n2 = min(max(__float2int_ru(X + w), 0), nz);
    }
  }
  bool above = false;
  for (int k = n2 - 1; k >= n1; --k) {
    const bool hit = ray_t(rt, rc, __ldg(oz + k), g.thr);
    if (hit != above) atomicXor(tog + (size_t)(k >> 5) * stride, 1u << (k & 31));
    above = hit;
  }
  if (n1 > 0 && !above) atomicXor(tog + (size_t)((n1 - 1) >> 5) * stride, 1u << ((n1 - 1) & 31));
}

// Every warp works by itself: it takes tickets of bd.tile triangles from the queue, stages them 32 at
// a time by bulk async copies (TMA) on its own mbarrier and runs their SAT and fill units 32 at a
// time.  With S > 1 (few triangles), S warps share a group's units.  Bound by instruction issue and
// table loads where the units are many and by latency where they are few.  Against blocks of eight
// warps on tiles of up to 256 triangles, whose closing barriers were the main stall (8 of 18 cycles per
// issue), with every column's hits evaluated over all its voxels by a whole warp and a counter update
// per 32 units: 262k triangles at 128^3 61 -> 36 us, 1.3M at 256^3 226 -> 108, 1M at 512^3 without
// Level2 441 -> 176, 7k large ones at 150x170x130 265 -> 40, 9M in 256 meshes 3.8 -> 1.4 ms.  Without
// the pieces of large triangles the last were 67 us and 4.1 ms: a group of them on one warp was the
// launch's tail.
__global__ void __launch_bounds__(kL1Warps * 32, 8) k_level1(BatchDev bd, uint32_t S) {
  __shared__ __align__(16) L1Warp s_warp[kL1Warps];
  const unsigned lane = threadIdx.x & 31u;
  L1Warp &ws = s_warp[threadIdx.x >> 5];
  if (lane == 0) {
    mbar_init(&ws.bar, 1);
    fence_mbar_init();
  }
  __syncwarp();

  const uint32_t nheavy = bd.heavy ? (uint32_t)min(*bd.heavy_n, (unsigned long long)bd.heavy_cap) : 0u;
  const uint32_t nitems = nheavy + (uint32_t)(bd.total_tiles * S);
  // the group after `it`: the next of its ticket, or the first of a new ticket
  // (a warp's first ticket is its own place in the grid, the heavy pieces spread over the blocks; one from
  // the queue, an atomic a warp on one word, and another to learn that none is left, were 8 us of a small call)
  const uint32_t nwarps = gridDim.x * kL1Warps;
  auto advance = [&](L1Item &it) {
    if (it.m >= 0 && it.t0 + kL1Group < it.tend) {
      it.t0 += kL1Group;
      return;
    }
    uint32_t tk = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (it.m != kNoItemYet) {
      tk = nwarps;
      if (nitems > nwarps) {
        if (lane == 0) tk += atomicAdd(&bd.queue[0], 1u);
        tk = __shfl_sync(FULL, tk, 0);
      }
    }
    if (tk >= nitems) {
      it.m = -1;
      return;
    }
    it.piece = 0u;
    if (tk < nheavy) {  // the heavy pieces first
      const uint4 h = __ldg(bd.heavy + tk);
      it.m = (int)h.x;
      it.t0 = h.y;
      it.tend = it.t0 + (h.w ? 1 : 0);  // (an entry of a triangle that did not fit the list: nothing)
      it.part = h.z * h.w;
      it.piece = max(h.w, 1u);
      return;
    }
    tk -= nheavy;
    const int64_t tile = tk / S;
    it.part = tk % S;
    it.m = find_mesh<&MeshDesc::tile_base>(bd.md, bd.nmesh, tile);
    const MeshDesc &d = bd.md[it.m];
    it.t0 = (tile - d.tile_base) * bd.tile;
    it.tend = min(d.T, it.t0 + bd.tile);
  };
  auto stage = [&](const L1Item &it) {
    if (it.m < 0 || lane != 0) return;
    const MeshDesc &d = bd.md[it.m];
    const uint32_t n = (uint32_t)max(min((int64_t)kL1Group, it.tend - it.t0), (int64_t)1);
    mbar_expect_tx(&ws.bar, n * 64u);
    bulk_g2s(ws.tri, d.ptri + 3 * it.t0, n * 48u, &ws.bar);
    bulk_g2s(ws.rng, d.rng + it.t0, n * 16u, &ws.bar);
  };

  uint32_t nbuf = 0;  // collected records of mesh `bm`
  int bm = -1;
  // Room for n records of a mesh in its segment; positions past its capacity raise the status, once for
  // all of them (once per record, the atomics of 7.5M records on one word took 5 ms of a first call).
  auto take_room = [&](const MeshDesc &d, uint32_t n) {
    unsigned long long pos = 0;
    if (lane == 0) {
      pos = atomicAdd(&d.stats->pairs, (unsigned long long)n);
      if (pos + n > (unsigned long long)d.pair_cap) atomicOr(&d.stats->status, (unsigned)ST_PAIR_OVERFLOW);
    }
    return __shfl_sync(FULL, pos, 0);
  };
  auto flush = [&]() {
    if (!nbuf) return;
    const MeshDesc &d = bd.md[bm];
    __syncwarp();
    const unsigned long long pos = take_room(d, nbuf);
    const uint64_t cap = (uint64_t)d.pair_cap;
    for (uint32_t i = lane; i < nbuf && pos + i < cap; i += 32) {
      d.keys[pos + i] = ws.key[i];
      d.vals[pos + i] = ws.val[i];
    }
    __syncwarp();
    nbuf = 0;
  };

  L1Item it = {kNoItemYet, 0, 0, 0, 0u};
  advance(it);
  stage(it);
  for (uint32_t phase = 0; it.m >= 0; phase ^= 1u) {
    const MeshDesc &d = bd.md[it.m];
    const GridDev &g = ws.g;
    if (bm != it.m) {
      flush();
      bm = it.m;
      __syncwarp();
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&d.g);
      uint32_t *dst = reinterpret_cast<uint32_t *>(&ws.g);
      for (int i = lane; i < (int)(sizeof(GridDev) / 4); i += 32) dst[i] = src[i];
      if (lane == 0) {
        ws.bplane = d.bplane;
        ws.toggles = d.toggles;
      }
      __syncwarp();
    }
    // bounded wait (bd.wait_limit polls, kWaitLimit when 0); bd.fail_wait makes it give up at once
    // (failure-detection tests).  On giving up, the status word is raised and the warp waits, bounded
    // again, for the copies in flight to land before it returns.
    const bool ok = !bd.fail_wait &&
                    mbar_wait_bounded(&ws.bar, phase, bd.wait_limit ? bd.wait_limit : kWaitLimit);
    if (__any_sync(FULL, !ok)) {
      if (lane == 0) atomicOr(&d.stats->status, (unsigned)ST_WAIT_TIMEOUT);
      mbar_wait_bounded(&ws.bar, phase, kWaitLimit);
      return;
    }
    const float4 *tri = ws.tri;
    const int4 *rng = ws.rng;
    const int64_t t0 = it.t0;
    const int nt = (int)min((int64_t)kL1Group, it.tend - t0);

    // ---- per-triangle unit counts and their scan
    uint32_t cs = 0, cf = 0;
    if ((int)lane < nt && (it.piece || !rng[lane].w)) {
      const int4 r = rng[lane];
      const int x0 = lo16(r.x), x1 = hi16(r.x), y0 = lo16(r.y), y1 = hi16(r.y);
      if (x0 <= x1 && y0 <= y1) cs = (uint32_t)((x1 - x0 + 1) * (y1 - y0 + 1));
      const uint32_t fxr = __float_as_uint(tri[3 * lane].w), fyr = __float_as_uint(tri[3 * lane + 1].w);
      if (lo16(fxr) <= hi16(fxr) && lo16(fyr) <= hi16(fyr))
        cf = (uint32_t)((hi16(fxr) - lo16(fxr) + 1) * (hi16(fyr) - lo16(fyr) + 1));
    }
    const uint32_t is = warp_incl_scan(cs), iff = warp_incl_scan(cf);
    ws.soff[lane] = is - cs;
    ws.foff[lane] = iff - cf;
    const uint32_t Us = __shfl_sync(FULL, is, 31), Uf = __shfl_sync(FULL, iff, 31);
    __syncwarp();
    const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
    const bool emit = d.has_l2 || bd.emit_all;  // the records are read later (else only counted)
    const uint32_t nsc = (Us + 31u) >> 5;
    const uint32_t step = it.piece ? 1u : S;
    const uint32_t cend = it.piece ? min(it.part + it.piece, nsc + ((Uf + 31u) >> 5)) : nsc + ((Uf + 31u) >> 5);
    unsigned long long counted = 0;
    uint32_t chunk = it.part;

    // ---- (a) SAT units: (triangle, column), a z run each
    for (; chunk < min(nsc, cend); chunk += step) {
      const uint32_t u = chunk * 32u + lane;
      int lt = 0, p = 0, q = 0, z0 = 0, zc = -1;
      float V[9];
      SatCol sc;
      if (u < Us) {
        lt = group_search(ws.soff, u);
        const int4 r = rng[lt];
        const int x0 = lo16(r.x), x1 = hi16(r.x), y0 = lo16(r.y);
        z0 = lo16(r.z);
        const uint32_t c = u - ws.soff[lt];
        const uint32_t nxr = (uint32_t)(x1 - x0 + 1), row = c / nxr;
        p = x0 + (int)(c - row * nxr);
        q = y0 + (int)row;
        const float4 a0 = tri[3 * lt], a1 = tri[3 * lt + 1], a2 = tri[3 * lt + 2];
        V[0] = a0.x; V[1] = a0.y; V[2] = a0.z; V[3] = a1.x; V[4] = a1.y; V[5] = a1.z;
        V[6] = a2.x; V[7] = a2.y; V[8] = a2.z;
        const float cx = __ldg(g.c1[0] + p), cy = __ldg(g.c1[1] + q);
        if (sat_col(V, cx, cy, g.e1, sc)) {
          zc = hi16(r.z);
          if (zc - z0 >= kPlaneRun) plane_range(V, g, cx, cy, z0, zc);
        }
      }
      bool first = true;
      const uint32_t tglob = (uint32_t)(t0 + lt);
      while (__any_sync(FULL, zc >= z0)) {
        uint32_t mask = 0;
        const int ztop = zc;
        if (zc >= z0) {
          const int nrun = min(32, zc - z0 + 1);
          for (int dd = 0; dd < nrun; ++dd)
            if (sat_z(sc, V, __ldg(g.c1[2] + (ztop - dd)), g.e1)) mask |= 1u << dd;
          zc -= nrun;
        }
        const uint32_t cnt = __popc(mask);
        uint32_t pos = 0;          // in the collected records
        unsigned long long gpos = 0;  // or in the mesh's segment
        bool direct = false;
        if (emit) {
          const uint32_t inc = warp_incl_scan(cnt);
          const uint32_t tot = __shfl_sync(FULL, inc, 31);
          if (tot == 0) continue;
          if (nbuf + tot > (uint32_t)kL1Pairs) flush();
          pos = nbuf + inc - cnt;
          direct = tot > (uint32_t)kL1Pairs;
          if (direct) gpos = take_room(d, tot) + inc - cnt;
          else nbuf += tot;
        } else {
          counted += cnt;
        }
        while (mask) {
          const int dd = __ffs(mask) - 1;
          mask &= mask - 1u;
          const int r = ztop - dd;
          const uint32_t key = (uint32_t)(((uint64_t)q * nx + p) * nz + r);
          const uint32_t val = tglob | (first ? 0x80000000u : 0u);
          if (direct) {
            if (gpos < (uint64_t)d.pair_cap) {
              d.keys[gpos] = key;
              d.vals[gpos] = val;
            }
            ++gpos;
          } else if (emit) {
            ws.key[pos] = key;
            ws.val[pos] = val;
            ++pos;
          }
          first = false;
          atomicOr(&ws.bplane[((size_t)r * ny + q) * g.nxw + (p >> 5)], 1u << (p & 31));
        }
        __syncwarp();
      }
    }
    if (!emit) {
      counted = warp_sum(counted);
      if (lane == 0 && counted) atomicAdd(&d.stats->pairs, counted);
    }

    // ---- (b) fill units: (triangle, column)
    for (; chunk < cend; chunk += step) {
      const uint32_t u = (chunk - nsc) * 32u + lane;
      if (u >= Uf) continue;
      const int lt = group_search(ws.foff, u);
      const float4 a0 = tri[3 * lt], a1 = tri[3 * lt + 1], a2 = tri[3 * lt + 2];
      const uint32_t fxr = __float_as_uint(a0.w), fyr = __float_as_uint(a1.w);
      const uint32_t c = u - ws.foff[lt];
      const uint32_t nxr = (uint32_t)(hi16(fxr) - lo16(fxr) + 1), row = c / nxr;
      const int i = lo16(fxr) + (int)(c - row * nxr), j = lo16(fyr) + (int)row;
      const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
      RayTri rt;
      ray_tri_pre(V, a2.w, rt);  // fill units exist only for triangles passing the det test
      RayCol rc;
      if (ray_col(rt, __ldg(g.c1[0] + i), __ldg(g.c1[1] + j), rc))
        column_toggles(rt, rc, g, ws.toggles + (size_t)j * nx + i, (size_t)nx * ny);
    }
    __syncwarp();  // the buffer may be staged again
    advance(it);
    stage(it);
  }
  flush();
}

// ---------------------------------------------------------------------------------------------
// 32 x 32 bits across a warp: bit c of lane r becomes bit r of lane c.
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x) {
  const unsigned lane = threadIdx.x & 31u;
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1, m ^= m << j) {
    const uint32_t y = __shfl_xor_sync(FULL, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

// A block takes kFinishGroups consecutive groups of 32 columns (a warp each; consecutive words of a
// layer's plane) and walks their layers 32 at a time: the parity of each column's voxels from its
// toggles, transposed to the linear inside plane, and, for meshes with pair lists, the boundary plane
// transposed the other way, to one word per column at the columns' place in key order.  Both planes
// move through shared memory, 32 bytes of a layer together.  Ray fill: the suffix XOR of the toggles, from
// the top layers down.  Stencil fill: the parity of each of the voxel column's four sample columns is
// the prefix XOR of its slice toggles, lowest slice first, and a voxel is inside where at least three
// of the four are odd.  Bound by latency on small grids and by the planes' traffic on large ones (a
// warp per 32 columns and 32 layers, which read all words above its own for the carry and wrote four
// bytes of a sector, took 102 us at 512^3 and 17 at 256^3; this 25 and 10).
__global__ void __launch_bounds__(kFinishGroups * 32) k_fill_finish(BatchDev bd) {
  __shared__ uint32_t s_in[2][32][kFinishGroups + 1], s_bd[2][32][kFinishGroups + 1];
  const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
  const int m = find_mesh<&MeshDesc::fblk_base>(bd.md, bd.nmesh, blockIdx.x);
  const MeshDesc &d = bd.md[m];
  const GridDev &g = d.g;
  const int nx = g.n[0], ny = g.n[1], nz = g.n[2], nzw = g.nzw;
  const int64_t ngrp = (int64_t)ny * g.nxw;  // words of a plane's layer
  const int64_t grp0 = ((int64_t)blockIdx.x - d.fblk_base) * kFinishGroups, grp = grp0 + warp;
  const int j = (int)(grp / g.nxw), ig = (int)(grp - (int64_t)j * g.nxw);
  const int i = ig * 32 + lane;
  const bool valid = grp < ngrp && i < nx;
  const size_t ncol = (size_t)nx * ny, col = (size_t)j * nx + i;
  const bool stencil = bd.fill == GPV_FILL_STENCIL;
  uint32_t *const km = bd.kmask && (d.has_l2 || bd.normals) ? bd.kmask + d.word_base : nullptr;
  // this thread's place in a plane tile: layer tl, group tg
  const int tl = (int)threadIdx.x / kFinishGroups, tg = (int)threadIdx.x % kFinishGroups;
  const bool tok = grp0 + tg < ngrp;
  const uint32_t *sc[4] = {nullptr, nullptr, nullptr, nullptr};
  if (stencil && valid) {
    const size_t SW = 2 * (size_t)nx;
    sc[0] = d.stg + ((size_t)(2 * j) * SW + 2 * (size_t)i) * nzw;
    sc[1] = sc[0] + nzw;
    sc[2] = sc[0] + SW * nzw;
    sc[3] = sc[2] + nzw;
  }
  uint32_t carry = 0;  // ray: the toggles above are odd; stencil, bit a: those below of sample a
  constexpr int kAhead = 4;
  for (int t0 = 0; t0 < nzw; t0 += kAhead) {
    // the next words' loads together
    uint32_t dv[kAhead], bv[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int t = t0 + k, w = stencil ? t : nzw - 1 - t, z = w * 32 + tl;
      dv[k] = t < nzw && valid && !stencil ? __ldg(d.toggles + (size_t)w * ncol + col) : 0u;
      bv[k] = t < nzw && km && tok && z < nz ? __ldg(d.bplane + (size_t)z * ngrp + grp0 + tg) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int t = t0 + k;
      if (t >= nzw) break;
      const int w = stencil ? t : nzw - 1 - t, buf = t & 1;
      uint32_t s;
      if (stencil) {
        uint32_t x[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint32_t D = valid ? sc[a][w] : 0u;
          uint32_t y = D;
          y ^= y << 1; y ^= y << 2; y ^= y << 4; y ^= y << 8; y ^= y << 16;
          if ((carry >> a) & 1u) y = ~y;
          carry ^= (uint32_t)(__popc(D) & 1) << a;
          x[a] = y;
        }
        s = (x[0] & x[1] & (x[2] | x[3])) | (x[2] & x[3] & (x[0] | x[1]));
      } else {
        s = dv[k];
        s ^= s >> 1; s ^= s >> 2; s ^= s >> 4; s ^= s >> 8; s ^= s >> 16;
        if (carry) s = ~s;
        carry ^= (uint32_t)(__popc(dv[k]) & 1);
      }
      s_in[buf][lane][warp] = warp_transpose(s);
      if (km) s_bd[buf][tl][tg] = bv[k];
      __syncthreads();
      const int z = w * 32 + tl;
      if (tok && z < nz) d.iplane[(size_t)z * ngrp + grp0 + tg] = s_in[buf][tl][tg];
      if (km) {
        const uint32_t bw = s_bd[buf][lane][warp];
        if (__any_sync(FULL, bw != 0u)) {
          const uint32_t cw = warp_transpose(bw);
          if (cw) {
            const uint64_t bit = (uint64_t)col * nz + (uint64_t)w * 32;
            const unsigned sh = (unsigned)(bit & 31u);
            atomicOr(km + (bit >> 5), cw << sh);
            if (sh && (cw >> (32 - sh))) atomicOr(km + (bit >> 5) + 1, cw >> (32 - sh));
          }
        }
      }
    }
  }
}

// B_m = boundary voxels of mesh m, from the exclusive scan over the batch's plane words.
__global__ void k_boundary_counts(BatchDev bd, const uint32_t *__restrict__ wpre,
                                  const uint32_t *__restrict__ wtotal) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= bd.nmesh) return;
  const uint32_t s = wpre[bd.md[m].word_base];
  const uint32_t e = m + 1 < bd.nmesh ? wpre[bd.md[m + 1].word_base] : *wtotal;
  bd.md[m].stats->boundary = e - s;
}

// A chunk is 32 words of a mesh's bit planes (up to 1024 voxels, x fastest): state bytes,
// boundaryPrefixSum, boundaryIndex.  A lane loads a word of each plane and its prefix; then every lane
// takes four voxels at a time (one where rows or buffers are not aligned) of the words in order, which it
// gets by shuffles, whatever the row length.  Bound by the writes: 512^3 voxels in 117 us, 5.7 TB/s; a
// lane loading the words of its own four voxels waited for them (215 us).
constexpr int kExpandWarps = 8;
struct ExpandMesh {
  const uint32_t *bplane, *iplane, *wp;
  uint8_t *l1;
  int32_t *prefix, *bindex;
  int64_t first;  // its first chunk
  uint32_t words, nx, nxw, pbase;
  uint32_t pw, mul;  // pieces (of four voxels or one) of a full word, ceil(2^20 / pw)
  bool vec;       // rows of a multiple of four voxels and aligned outputs (the batch's arenas are, a
                  // no-alloc caller's buffers may not be)
};
__device__ __forceinline__ ExpandMesh expand_mesh(const MeshDesc &d, const uint32_t *__restrict__ wpre) {
  ExpandMesh e;
  e.bplane = d.bplane;
  e.iplane = d.iplane;
  e.wp = wpre + d.word_base;
  e.l1 = d.l1;
  e.prefix = d.prefix;
  e.bindex = d.bindex;
  e.first = d.xc_base;
  e.nx = (uint32_t)d.g.n[0];
  e.nxw = (uint32_t)d.g.nxw;
  e.words = e.nxw * (uint32_t)d.g.n[1] * (uint32_t)d.g.n[2];
  e.pbase = wpre[d.word_base];
  e.vec = (e.nx & 3u) == 0 && (reinterpret_cast<uintptr_t>(d.l1) & 3u) == 0 &&
          (reinterpret_cast<uintptr_t>(d.prefix) & 15u) == 0;
  e.pw = min(e.nx, 32u) / (e.vec ? 4u : 1u);
  e.mul = ((1u << 20) + e.pw - 1u) / e.pw;
  return e;
}
// Words [j0, j1) of a chunk by one warp; returns the lane's inside-voxel count.
__device__ __forceinline__ uint32_t expand_chunk(const ExpandMesh &e, int64_t gc, uint32_t j0, uint32_t j1,
                                                 uint32_t lane) {
  const uint32_t w = (uint32_t)(gc - e.first) * 32u + lane;
  uint32_t bw = 0, iw = 0, p = 0, v0 = 0, cnt = 0, nin = 0;
  if (w < e.words) {
    bw = __ldg(e.bplane + w);
    iw = __ldg(e.iplane + w) & ~bw;
    p = __ldg(e.wp + w) - e.pbase;
    const uint32_t row = w / e.nxw, x0 = (w - row * e.nxw) * 32u;
    v0 = row * e.nx + x0;
    cnt = min(32u, e.nx - x0);
    if (lane >= j0 && lane < j1) {
      nin = (uint32_t)__popc(iw & (0xffffffffu >> (32u - cnt)));
      uint32_t q = p;
      for (uint32_t k = bw; k; k &= k - 1u) e.bindex[q++] = (int32_t)(v0 + (uint32_t)__ffs(k) - 1u);
    }
  }
  const uint32_t i1 = j1 * e.pw;
#pragma unroll 2
  for (uint32_t i0 = j0 * e.pw; i0 < i1; i0 += 32u) {
    const uint32_t i = i0 + lane;
    // i < 1024 and the excess of mul over 2^20 / pw below one: the quotient is exact
    const uint32_t j = i * e.mul >> 20, b = i - j * e.pw;
    const uint32_t B = __shfl_sync(FULL, bw, j), I = __shfl_sync(FULL, iw, j), P = __shfl_sync(FULL, p, j),
                   V = __shfl_sync(FULL, v0, j), n = __shfl_sync(FULL, cnt, j);
    if (i >= i1) continue;
    if (e.vec) {
      const uint32_t b0 = 4u * b;
      if (b0 >= n) continue;
      const uint32_t bb = (B >> b0) & 0xfu, ib = (I >> b0) & 0xfu;
      const uint32_t q = P + __popc(B & ((1u << b0) - 1u));
      // (4 bits to 4 bytes: bit j to byte j)
      const uint32_t bytes = ((bb * 0x00204081u) & 0x01010101u) * 254u + ((ib * 0x00204081u) & 0x01010101u) * 127u;
      const uint32_t q1 = q + (bb & 1u), q2 = q1 + ((bb >> 1) & 1u), q3 = q2 + ((bb >> 2) & 1u);
      *reinterpret_cast<uint32_t *>(e.l1 + V + b0) = bytes;
      *reinterpret_cast<int4 *>(e.prefix + V + b0) = make_int4((int)q, (int)q1, (int)q2, (int)q3);
    } else {
      if (b >= n) continue;
      const uint32_t isb = (B >> b) & 1u, isi = (I >> b) & 1u;
      e.l1[V + b] = (uint8_t)(isb * 254u + isi * 127u);
      e.prefix[V + b] = (int32_t)(P + __popc(B & ((1u << b) - 1u)));
    }
  }
  return nin;
}

// A block takes `iters` x kExpandWarps consecutive parts of chunks (`split` to a chunk), warp w the
// parts w + k x kExpandWarps of them.  Thread 0 looks up the mesh of the block's first chunk once (a binary search over
// the descriptors), and each warp walks forward from it as its chunks pass mesh boundaries, so
// the search is not repeated per chunk.  A warp adds its inside count to the statistics when it
// leaves a mesh; the block adds the warps' last runs with one atomic per mesh.
__global__ void __launch_bounds__(kExpandWarps * 32) k_expand(BatchDev bd,
                                                            const uint32_t *__restrict__ wpre,
                                                            int iters, int split) {
  __shared__ int s_mesh;
  __shared__ int s_m[kExpandWarps];
  __shared__ unsigned long long s_nin[kExpandWarps];
  // one-graph calls whose sizes did not fit: the call is re-run
  if (bd.plan && !bd.plan->ok) return;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int64_t c0 = (int64_t)blockIdx.x * kExpandWarps * iters;
  if (threadIdx.x == 0) s_mesh = find_mesh<&MeshDesc::xc_base>(bd.md, bd.nmesh, c0 / split);
  __syncthreads();
  int m = s_mesh;
  ExpandMesh em = expand_mesh(bd.md[m], wpre);
  int64_t next = m + 1 < bd.nmesh ? bd.md[m + 1].xc_base : bd.total_xchunks;
  unsigned long long nin = 0;
#pragma unroll 1
  for (int k = 0; k < iters; ++k) {
    const int64_t gp = c0 + (int64_t)k * kExpandWarps + warp, gc = gp / split;
    const uint32_t part = (uint32_t)(gp - gc * split), pn = 32u / (uint32_t)split;
    if (gc >= bd.total_xchunks) break;  // warp-uniform
    if (gc >= next) {
      const unsigned long long t = warp_sum(nin);
      if (lane == 0 && t) atomicAdd(&bd.md[m].stats->l1_inside, t);
      nin = 0;
      while (m + 1 < bd.nmesh && bd.md[m + 1].xc_base <= gc) ++m;
      em = expand_mesh(bd.md[m], wpre);
      next = m + 1 < bd.nmesh ? bd.md[m + 1].xc_base : bd.total_xchunks;
    }
    nin += expand_chunk(em, gc, part * pn, (part + 1u) * pn, lane);
  }
  // the warps' last mesh runs: one atomic per mesh of the block
  const unsigned long long t = warp_sum(nin);
  if (lane == 0) {
    s_m[warp] = m;
    s_nin[warp] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int cur = s_m[0];
    unsigned long long acc = 0;
    for (int w = 0; w < kExpandWarps; ++w) {
      if (s_m[w] != cur) {
        if (acc) atomicAdd(&bd.md[cur].stats->l1_inside, acc);
        cur = s_m[w];
        acc = 0;
      }
      acc += s_nin[w];
    }
    if (acc) atomicAdd(&bd.md[cur].stats->l1_inside, acc);
  }
}

__global__ void k_heads(const uint32_t *__restrict__ keys, int64_t P, uint32_t *__restrict__ flags) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < P) flags[e] = (e == 0 || keys[e] != keys[e - 1]) ? 1u : 0u;
}

// Every mesh's first pair starts a segment even when its key equals the previous mesh's last.
__global__ void k_mesh_pair_heads(BatchDev bd, int64_t P, uint32_t *__restrict__ flags) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= bd.nmesh) return;
  const int64_t b = bd.md[m].pair_base;
  const int64_t e = m + 1 < bd.nmesh ? bd.md[m + 1].pair_base : P;
  if (e > b) flags[b] = 1u;
}

__global__ void k_useg(const uint32_t *__restrict__ flags, const uint32_t *__restrict__ uidx,
                       int64_t P, uint32_t *__restrict__ useg) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < P && flags[e]) useg[uidx[e]] = (uint32_t)e;
  if (e == P - 1) useg[uidx[e] + flags[e]] = (uint32_t)P;
}

// Copies and clears of StageOps (see StageList): 16-byte accesses where both addresses allow,
// 4-byte ones otherwise.  Sources are read with cache-volatile loads: page-locked host staging is
// rewritten by the host between launches.
__global__ void __launch_bounds__(256) k_stage(StageOps L) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int k = 0; k < L.n; ++k) {
    const uint32_t *src = L.op[k].src;
    uint32_t *dst = L.op[k].dst;
    const int64_t w = L.op[k].words;
    int64_t i0 = 0;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
      const int64_t w4 = w >> 2;
      uint4 *d4 = reinterpret_cast<uint4 *>(dst);
      const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
      if (src)
        for (int64_t i = t; i < w4; i += stride) d4[i] = __ldcv(s4 + i);
      else
        for (int64_t i = t; i < w4; i += stride) d4[i] = make_uint4(0u, 0u, 0u, 0u);
      i0 = w4 << 2;
    }
    if (src)
      for (int64_t i = i0 + t; i < w; i += stride) dst[i] = __ldcv(src + i);
    else
      for (int64_t i = i0 + t; i < w; i += stride) dst[i] = 0u;
  }
}

}  // namespace

// ---- launchers --------------------------------------------------------------------------------
void launch_prep(const BatchDev &bd, cudaStream_t s) {
  if (bd.total_tris <= 0) return;
  k_prep<<<(unsigned)((bd.total_tris + 255) / 256), 256, 0, s>>>(bd);
  count_launch();
}

// Boundary-voxel rank at the start of each z slab of one mesh (slab k = layers [k*zslab,
// (k+1)*zslab)): the exclusive word prefix at the slab's first word, the total past the end.
__global__ void k_slab_offsets(const uint32_t *__restrict__ wpre, const uint32_t *__restrict__ wtot,
                               int64_t words_per_layer, int nz, int zslab, int nslab,
                               uint32_t *__restrict__ out) {
  const int t = (int)threadIdx.x;
  if (t > nslab) return;
  const int z0 = min(t * zslab, nz);
  out[t] = z0 >= nz ? *wtot : wpre[(int64_t)z0 * words_per_layer];
}

void launch_slab_offsets(const uint32_t *wpre, const uint32_t *wtot, int64_t words_per_layer,
                         int nz, int zslab, int nslab, uint32_t *out, cudaStream_t s) {
  k_slab_offsets<<<1, 32, 0, s>>>(wpre, wtot, words_per_layer, nz, zslab, nslab, out);
  count_launch();
}

void StageList::add(void *dst, const void *src, size_t bytes) {
  if (bytes == 0) return;
  if (bytes & 3u) {
    if (src)
      cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, s_);
    else
      cudaMemsetAsync(dst, 0, bytes, s_);
    return;
  }
  if (ops_.n == StageOps::kMax) launch();
  ops_.op[ops_.n++] = {static_cast<const uint32_t *>(src), static_cast<uint32_t *>(dst),
                       (int64_t)(bytes / 4)};
}

void StageList::launch() {
  if (ops_.n == 0) return;
  int64_t w = 0;
  for (int k = 0; k < ops_.n; ++k) w = std::max(w, ops_.op[k].words);
  const int64_t blocks = std::min<int64_t>((w / 4 + 255) / 256 + 1, 2 * (int64_t)sms_);
  k_stage<<<(unsigned)blocks, 256, 0, s_>>>(ops_);
  count_launch();
  ops_.n = 0;
}

void launch_pair_bases(const BatchDev &bd, MeshDesc *d_md, uint32_t *keys, uint32_t *vals,
                       int64_t cap, cudaStream_t s) {
  k_pair_bases<<<1, 1024, 0, s>>>(bd.nmesh, d_md, keys, vals, cap);
  count_launch();
}

void launch_plan(const BatchDev &bd, MeshDesc *d_md, int32_t *bindex, uint8_t *l2,
                 const PlanCaps &caps, DevPlan *plan, cudaStream_t s) {
  k_plan<<<1, 1024, 0, s>>>(bd.nmesh, d_md, bindex, l2, caps, plan);
  count_launch();
}

void launch_level1(const BatchDev &bd, int num_sms, cudaStream_t s) {
  if (bd.total_tiles <= 0) return;
  // Few triangles (a coarse model on a fine grid): several warps share a group's units, so that
  // every SM has its 32 warps.
  const int64_t warps = (int64_t)num_sms * 8 * kL1Warps;
  const int64_t S = std::max<int64_t>(1, std::min<int64_t>(warps / bd.total_tiles, 4096));
  const int64_t items = bd.total_tiles * S;
  const int64_t grid = std::min<int64_t>((items + kL1Warps - 1) / kL1Warps, (int64_t)num_sms * 8);
  k_level1<<<(unsigned)grid, kL1Warps * 32, 0, s>>>(bd, (uint32_t)S);
  count_launch();
}

void launch_fill_finish(const BatchDev &bd, cudaStream_t s) {
  if (bd.total_fblks <= 0) return;
  k_fill_finish<<<(unsigned)bd.total_fblks, kFinishGroups * 32, 0, s>>>(bd);
  count_launch();
}

void launch_boundary_counts(const BatchDev &bd, const uint32_t *wpre, const uint32_t *wtotal,
                            cudaStream_t s) {
  k_boundary_counts<<<(unsigned)((bd.nmesh + 127) / 128), 128, 0, s>>>(bd, wpre, wtotal);
  count_launch();
}

void launch_expand(const BatchDev &bd, const uint32_t *wpre, int num_sms, cudaStream_t s) {
  if (bd.total_xchunks <= 0) return;
  // few chunks: parts of them, so that each SM has 16 warps (128^3 voxels, 2048 chunks: 9.6 us; 32
  // warps 12, whose parts each load the chunk's words); many: up to four per warp
  int split = 1;
  while (split < 8 && bd.total_xchunks * split < (int64_t)num_sms * 16) split *= 2;
  const int64_t parts = bd.total_xchunks * split, spread = parts / ((int64_t)num_sms * 64);
  const int iters = (int)(spread < 1 ? 1 : spread > 4 ? 4 : spread);
  const int64_t per_block = (int64_t)kExpandWarps * iters;
  k_expand<<<(unsigned)((parts + per_block - 1) / per_block), kExpandWarps * 32, 0, s>>>(bd, wpre, iters, split);
  count_launch();
}

void launch_heads(const uint32_t *keys, int64_t P, uint32_t *flags, const BatchDev &bd,
                  cudaStream_t s) {
  if (P <= 0) return;
  k_heads<<<(unsigned)((P + 255) / 256), 256, 0, s>>>(keys, P, flags);
  k_mesh_pair_heads<<<(unsigned)((bd.nmesh + 127) / 128), 128, 0, s>>>(bd, P, flags);
  count_launch(2);
}

void launch_useg(const uint32_t *flags, const uint32_t *uidx, int64_t P, uint32_t *useg,
                 cudaStream_t s) {
  if (P <= 0) return;
  k_useg<<<(unsigned)((P + 255) / 256), 256, 0, s>>>(flags, uidx, P, useg);
  count_launch();
}

}  // namespace gpv
