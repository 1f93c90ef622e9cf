// gpv_level2.cu -- Level2 refinement of the boundary voxels, organised per Level1 column.
//
// Reference semantics (src/Object.cpp:1111-1207 and :2344-2400): for boundary voxel b at
// (i,j,k), a Level2 cell is 2 if the SAT passes for any triangle recorded in b; otherwise 1 if
// the +z ray from the cell's origin crosses an odd number of distinct triangles among those
// recorded in voxels (i,j,z) with z >= k; otherwise 0.
//
// Work unit (one warp): the SAT's is a run of consecutive boundary voxels, the fill's a chunk of up to
// CH consecutive boundary voxels of one Level1 column.
//   SAT   -- each axis test of the SAT that crosses an edge with a box axis depends on two of the
//            three coordinates, so the cells that pass the nine of them are the ones whose x/y, y/z
//            and x/z squares pass three two-dimensional tests.  Those are solved a row at a time
//            (solve_rows): the interval of cells that certainly pass and the one outside which every
//            cell certainly fails, with the float tests' error bounds.  A sub-column's cells are the
//            intersection of two such intervals with the plane test's, written with one atomic.
//            Only sub-columns with a cell between the two intervals (about one in a hundred) run
//            the exact float tests.
//   fill  -- the column's triangle entries flagged as topmost occurrences are the union sets
//            of all voxels of the chunk at once (voxel k sees the triangles whose topmost z is
//            >= k).  The sub-columns whose ray meets the triangle come from the same row solver;
//            the height of the triangle's plane there gives the number of ray origins below it, so
//            one toggle marks the highest voxel that is hit entirely (a suffix XOR over the chunk's
//            voxels expands it) and one run of bits the voxel that holds the crossing.  Rays and
//            crossings within the error bounds run the exact float tests.
#include "gpv_internal.h"
#include "gpv_rows.cuh"

namespace gpv {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kWarps = 4;
constexpr int kDirectCells = 4;  // a triangle whose box meets at most this many cells is tested exactly
// Where the centre tables lie further than this many cells from their affine form (coordinates large
// against the cells), the solved rows leave nearly every cell open: the triangles' sub-columns are
// tested exactly instead.  262k-triangle torus at 128^3 / 8^3, SAT us, rows and exact, by the distance:
// 0.5 cells 326 and 445, 1.4 546 and 470, 2.9 784 and 500, 4.8 890 and 535, 14 1715 and 818.
constexpr float kWide = 1.0f;
constexpr float kFar = 0.125f;  // cells; from there on SAT runs are short (far_grid)
constexpr int kMaskWords = 512;  // words of one mask kind per warp (sets the chunk length)

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

// Bits of one Level2 column (n2z cells along z) start at bit (q*n2x + p)*n2z of a voxel's mask.
__device__ __forceinline__ void or_column(uint32_t *m, int colidx, int n2z, uint32_t bits) {
  const int off = colidx * n2z, sh = off & 31;
  atomicOr(&m[off >> 5], bits << sh);
  if (sh + n2z > 32) atomicOr(&m[(off >> 5) + 1], bits >> (32 - sh));
}
__device__ __forceinline__ void xor_column(uint32_t *m, int colidx, int n2z, uint32_t bits) {
  const int off = colidx * n2z, sh = off & 31;
  atomicXor(&m[off >> 5], bits << sh);
  if (sh + n2z > 32) atomicXor(&m[(off >> 5) + 1], bits >> (32 - sh));
}

// t of the +z test for one origin height (same operations as ray_t).
__device__ __forceinline__ float ray_tval(const RayTri &r, const RayCol &c, float oz) {
  const float Tz = fs(oz, r.v1z);
  const float q0 = fs(fm(c.Ty, r.e1z), fm(Tz, r.e1y));
  const float q1 = fs(fm(Tz, r.e1x), fm(c.Tx, r.e1z));
  const float q2 = fs(fm(c.Tx, r.e1y), fm(c.Ty, r.e1x));
  return fm(fa(fa(fm(r.e2x, q0), fm(r.e2y, q1)), fm(r.e2z, q2)), r.inv_det);
}

// Number of origins r in [0, n) with otop - oz[r] > dthr (float subtraction), for an increasing
// table oz of spacing ~1/inv: the count is a prefix length because otop - oz[r] rounds
// monotonically; an arithmetic estimate is corrected by table comparisons.
__device__ __forceinline__ int count_drop_above(const float *oz, int n, float otop, float dthr,
                                                float inv) {
  const float f = (otop - dthr - __ldg(oz)) * inv;
  int i;
  if (!(f > 0.f)) i = 0;
  else if (f >= (float)n) i = n;
  else i = (int)ceilf(f);
#pragma unroll 1
  while (i > 0 && !(otop - __ldg(oz + i - 1) > dthr)) --i;
#pragma unroll 1
  while (i < n && otop - __ldg(oz + i) > dthr) ++i;
  return i;
}

constexpr int kSol = 512;    // solved rows of one batch (a triangle has at most 96); the output stage
                             // keeps 16 layers of 32 lanes there
constexpr int kCols = 1024;  // its sub-columns (a triangle has at most that many)

struct __align__(16) WarpScratch {
  float4 xa[32], xb[32];  // per-triangle constants
  uint4 me[32];        // triangle id; voxel in the chunk (fill: voxels of the chunk up to its topmost) |
                       // exact tests only << 8 | first sub-column << 16 | first row << 24; its solved
                       // rows of y/z | of x/z << 16; first layer | end << 8 where tests are exact
  uint32_t seg[36];    // SAT: first pair of each voxel of the chunk, and the end
  uint32_t sol[kSol];  // solved rows
  uint32_t rtri[64];   // queued exact work: triangle id and
  uint32_t rpos[64];   // voxel (or voxel count), sub-column and cell range
  uint32_t utri[64];   // fill: queued triangles and the voxels of the chunk that see them
  uint8_t ujm[64];
  uint16_t cols[kCols];  // the batch's sub-columns: triangle slot | row << 5 | column << 10 (both from
                         // the triangle's first) | certain to pass the x/y tests << 15
};
static_assert(sizeof(WarpScratch) % 16 == 0, "layout");

// A triangle of the stencil fill: for each edge the edge function at sample (0, 0) (64 bits), dx and dy;
// first sample column | columns << 6 | first row << 13 | the edges' top-left flags << 19, 1 / area and
// the heights of two vertices; the third's, 1 / columns and its first sample of the batch's.
struct __align__(16) StRec {
  int4 e[3];
  float4 a, b;
};
struct StScratch {    // the triangles of a batch that have samples, in order
  StRec r[32];
};
static_assert(sizeof(StScratch) >= 16 * 32 * 4, "the output stage keeps 16 layers of 32 lanes there");

// The samples of a batch of triangles (one per lane, `has`: it has samples), taken one per lane.  An edge
// function costs two widening multiply-adds from its value at the first sample, the owner of a sample a
// reduction over the lanes whose triangle starts among the 32, its slice an estimate that the table
// corrects, and the scratch is 2.5 KB, so that 24 warps fit an SM: the 262k-triangle torus at 128^3 / 8^3
// took 440 us in the fill and 70 in k_stencil_segment with 64-bit products, searches over the prefix and
// the slices, and 16 warps; 215 and 36 so (the heights' comparison added about 10 us to both since).  Bound by latency (about half of the issue slots).
struct StBatch {
  uint32_t start, cnt, total;  // this lane's triangle's first sample and samples; the batch's
  __device__ __forceinline__ StBatch(StRec *recs, bool has, const StTri &t) {
    const unsigned lane = threadIdx.x & 31u;
    const int nsx = t.sx1 - t.sx0 + 1;
    cnt = has ? (uint32_t)(nsx * (t.sy1 - t.sy0 + 1)) : 0u;
    const uint32_t inc = warp_incl_scan(cnt);
    start = inc - cnt;
    total = __shfl_sync(FULL, inc, 31);
    const uint32_t bal = __ballot_sync(FULL, has);
    if (has) {
      StRec &r = recs[__popc(bal & ((1u << lane) - 1u))];
      uint32_t tl = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int i = (k + 1) % 3, j = (k + 2) % 3;
        const int32_t dx = t.X[j] - t.X[i], dy = t.Y[j] - t.Y[i];
        const long long w = (long long)dx * (128 - t.Y[i]) - (long long)dy * (128 - t.X[i]);
        r.e[k] = make_int4((int)(uint32_t)w, (int)(w >> 32), dx, dy);
        if (dy < 0 || (dy == 0 && dx > 0)) tl |= 1u << k;
      }
      const uint32_t rng = (uint32_t)t.sx0 | ((uint32_t)nsx << 6) | ((uint32_t)t.sy0 << 13) | (tl << 19);
      r.a = make_float4(__uint_as_float(rng), t.rA, t.z[0], t.z[1]);
      r.b = make_float4(t.z[2], rcp_fast((float)nsx), __uint_as_float(start), 0.f);
    }
  }
  // The record of sample w0 + lane (all lanes call; w0 a multiple of 32).
  __device__ __forceinline__ const StRec &owner(const StRec *recs, uint32_t w0) const {
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t here = __reduce_or_sync(FULL, cnt && start - w0 < 32u ? 1u << (start - w0) : 0u);
    const uint32_t before = (uint32_t)__popc(__ballot_sync(FULL, cnt && start < w0));
    return recs[before + (uint32_t)__popc(here & ((2u << lane) - 1u)) - 1u];
  }
};

// Coverage of sample w of the batch (as st_cover), its place and the surface height there.
__device__ __forceinline__ bool st_sample(const StRec &r, uint32_t w, int &sx, int &sy, float &zs) {
  const float4 a = r.a, b = r.b;
  const uint32_t rng = __float_as_uint(a.x), loc = w - __float_as_uint(b.z);
  const uint32_t nsx = (rng >> 6) & 127u;
  // (loc + 1/2) / nsx stays at least 1/128 away from an integer, far above the rounding
  const uint32_t row = (uint32_t)__float2int_rz(((float)loc + 0.5f) * b.y);
  sx = (int)((rng & 63u) + (loc - row * nsx));
  sy = (int)(((rng >> 13) & 63u) + row);
  long long v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int4 e = r.e[k];
    v[k] = (long long)(((unsigned long long)(uint32_t)e.y << 32) | (uint32_t)e.x) + (long long)e.z * (sy * 256) -
           (long long)e.w * (sx * 256);
    if (!(v[k] > 0 || (v[k] == 0 && ((rng >> (19 + k)) & 1u)))) return false;
  }
  zs = fa(fa(fm(fm(__ll2float_rn(v[0]), a.y), a.z), fm(fm(__ll2float_rn(v[1]), a.y), a.w)),
          fm(fm(__ll2float_rn(v[2]), a.y), b.x));
  return true;
}

// ---- item construction -----------------------------------------------------------------------
__device__ __forceinline__ int mesh_of_u(const MeshDesc *md, int nmesh, int64_t u) {
  int lo = 0, hi = nmesh - 1;
#pragma unroll 1
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (md[mid].u_base <= u) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Boundary voxels of the sorted meshes: B, or (one-graph calls, B the capacity) the device
// plan's count, none when the plan did not fit.
__device__ __forceinline__ int64_t sorted_voxels(const BatchDev &bd, int64_t B) {
  if (!bd.plan) return B;
  return bd.plan->ok ? min(B, (int64_t)bd.plan->ub) : 0;
}

// Work item of the Level2 kernels: a run of boundary voxels of one Level1 column.
struct __align__(16) Item {
  uint32_t ua;       // first boundary voxel
  uint32_t m_mesh;   // voxels (1..32) | first of its column << 6 | mesh << 7
                     // (a SAT run has the voxels and the mesh only)
  uint32_t col;      // column (y * nx + x)
  uint32_t col_end;  // first boundary voxel of the next column
};

// Marked voxels of all meshes up to and with `key` of mesh d (kpre: the exclusive prefix of kmask's
// bits by word, kpre[0] the bits before the plane).
__device__ __forceinline__ uint32_t marked_through(const BatchDev &bd, const MeshDesc &d,
                                                   const uint32_t *__restrict__ kpre, uint32_t key) {
  const int64_t w = d.word_base + (key >> 5);
  return __ldg(kpre + w) - __ldg(kpre) + __popc(__ldg(bd.kmask + w) & (0xffffffffu >> (31u - (key & 31u))));
}

// The SAT kernel takes runs of consecutive boundary voxels, whatever their columns: its pairs are
// tested by voxel.  A run ends where its masks fill the warp's share of shared memory and, so that
// batches of 32 pairs are full and warps finish together, after about q pairs: nb batches less an
// average list (a run's pairs vary by about one list around q), nb giving a warp two runs, and a
// quarter of that for the last eighth of the pairs.  Where a full run's masks hold less than two
// batches, pairs only bound the longest lists.  Against the fill's items, whose columns are mostly
// short: a 16k-triangle sphere at 64^3 / 4^3 52 -> 31 us (its longest columns took that long), 7k
// triangles at 150x170x130 / 6^3 73 -> 53, 256 mixed meshes 5.4 -> 4.0 ms, the 1.3M-triangle star at
// 256^3 / 16^3 690 -> 677; a 262k-triangle torus, whose columns are long, 113..119 -> 119.  One run
// a warp instead of two: torus 135 us, batch 4.1 ms; three: batch 3.9 ms, star 684 us.
constexpr int kSatWords = 512;  // (1024, with a block less per SM, took 688 us for the star)
__host__ __device__ __forceinline__ int sat_run_cap(const GridDev &g) {
  const int n = kSatWords / ((g.n2[0] * g.n2[1] * g.n2[2] + 31) >> 5);
  return n < 1 ? 1 : n > 32 ? 32 : n;
}
// Far from the origin (the centre tables an eighth of a cell and more off their affine form) a pair can be
// hundreds of exact tests, so a run has no more pairs than half a warp's share.  Calls of small meshes
// around 10000, us, with runs of full batches and so (and with the exact kernel before the row solver): 900
// triangles at 56x65x54 / 8^3, 2 cells off, 665, 339 (418); 484 at 42x82x77 / 9^3 758, 493 (604); 440 at
// 58x44x53 / 7^3 408, 245 (363); 1.3k at 45x69x41 / 15^3 765, 752 (686); 5.3k at 23x30x31 / 8^3, 0.3 off,
// 235, 225 (414); where pairs are many nothing changes.
__device__ __forceinline__ bool far_grid(const GridDev &g) {
  float w = 0.f;
#pragma unroll
  for (int a = 0; a < 3; ++a) w = fmaxf(w, 2.02f * EPS24 * fmaxf(fabsf(g.bmin[a]), fabsf(g.bmax[a])) * g.inv_g2[a]);
  return w > kFar;
}
struct SatRuns {
  uint32_t q, qt, tail, nq;
  __device__ __forceinline__ SatRuns(uint32_t pairs, uint32_t voxels, int slots, uint32_t cap, bool far) {
    const uint32_t avg = pairs / voxels, nb = max(pairs / (32u * (uint32_t)slots), 1u);
    q = max(32u * nb, avg + 16u) - avg;
    qt = max(32u * max(nb / 4u, 1u), avg + 16u) - avg;
    if (cap * avg < 64u) {
      q = max(q, 256u);
      qt = q;
    }
    if (far) q = qt = min(q, max(pairs / (uint32_t)slots, 1u));
    tail = pairs - pairs / 8u;
    nq = tail / q + 1u;
  }
  __device__ __forceinline__ uint32_t bucket(uint32_t e) const { return e < tail ? e / q : nq + (e - tail) / qt; }
};

// The items: one starts every MeshDesc::ch voxels from its column's first boundary voxel and, with z
// slabs (zslab > 0), also where the column enters a new slab of zslab Level1 layers.  The ends of a
// voxel's column and slab are ranks among the marked voxels, so each voxel knows by itself whether an
// item starts there and how long it is; blocks append theirs in any order.  runs (nullptr with z slabs,
// where the SAT takes the items): the SAT kernel's; counts: the numbers of both.  iflag (stencil fill, else
// nullptr): 1 where an item starts.  Bound by latency; two scans over the voxels and four kernels
// instead (column flags, heads, item flags, starts) made a 16k-triangle call 25 us longer, the 262k-
// triangle torus (98k boundary voxels) 21 us.
constexpr int kItemThreads = 256;
__global__ void __launch_bounds__(kItemThreads) k_items(
    BatchDev bd, const uint32_t *__restrict__ kpre, const uint32_t *__restrict__ keys,
    const uint32_t *__restrict__ useg, int64_t Bcap, int zslab, uint32_t *__restrict__ iflag,
    Item *__restrict__ items, Item *__restrict__ runs, int slots, uint32_t *__restrict__ counts) {
  __shared__ int s_mesh[2];
  __shared__ uint32_t s_cnt[2][kItemThreads / 32];
  const int64_t B = sorted_voxels(bd, Bcap);
  const int64_t u0 = (int64_t)blockIdx.x * kItemThreads, u = u0 + threadIdx.x;
  if (u0 >= B) return;
  if ((threadIdx.x & 31u) == 0 && threadIdx.x < 64)
    s_mesh[threadIdx.x >> 5] = mesh_of_u(bd.md, bd.nmesh, threadIdx.x ? min(u0 + kItemThreads, B) - 1 : u0);
  __syncthreads();
  Item it = {}, run = {};
  bool start = false, rstart = false;
  if (u < B) {
    const int m0 = s_mesh[0], mesh = m0 + mesh_of_u(bd.md + m0, s_mesh[1] - m0 + 1, u);
    const MeshDesc &d = bd.md[mesh];
    if (d.has_l2) {  // meshes sorted for their normals only get no items
      const uint32_t nz = (uint32_t)d.g.n[2], key = __ldg(keys + __ldg(useg + u)), col = key / nz;
      const uint32_t k0 = col * nz, uu = (uint32_t)u;
      const uint32_t head = k0 ? marked_through(bd, d, kpre, k0 - 1u) : (uint32_t)d.u_base;
      it.ua = uu;
      it.col = col;
      it.col_end = marked_through(bd, d, kpre, k0 + nz - 1u);
      const uint32_t ch = (uint32_t)d.ch, r = (uu - head) % ch;
      uint32_t end = min(it.col_end, uu + ch - r);
      start = r == 0;
      if (zslab > 0) {
        const uint32_t z0 = (key - k0) / (uint32_t)zslab * (uint32_t)zslab;
        const uint32_t z1 = min(nz, z0 + (uint32_t)zslab);
        start = start || (z0 && uu == marked_through(bd, d, kpre, k0 + z0 - 1u));
        end = min(end, marked_through(bd, d, kpre, k0 + z1 - 1u));
      }
      it.m_mesh = (end - uu) | (uu == head ? 64u : 0u) | ((uint32_t)mesh << 7);
      if (runs) {
        const uint32_t cap = (uint32_t)sat_run_cap(d.g);
        const SatRuns sr(__ldg(useg + B), (uint32_t)B, slots, cap, far_grid(d.g));
        const uint32_t r0 = (uu - (uint32_t)d.u_base) % cap, b = sr.bucket(__ldg(useg + u));
        rstart = r0 == 0 || sr.bucket(__ldg(useg + u - 1)) != b;
        if (rstart) {
          const uint32_t mend = mesh + 1 < bd.nmesh ? (uint32_t)bd.md[mesh + 1].u_base : (uint32_t)B;
          const uint32_t last = min(mend, uu + cap - r0);
          uint32_t e = uu + 1;
          while (e < last && sr.bucket(__ldg(useg + e)) == b) ++e;
          run.ua = uu;
          run.m_mesh = (e - uu) | ((uint32_t)mesh << 7);
        }
      }
    }
    if (iflag) iflag[u] = start ? 1u : 0u;
  }
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t bal = __ballot_sync(FULL, start), rbal = __ballot_sync(FULL, rstart);
  if (lane == 0) {
    s_cnt[0][warp] = (uint32_t)__popc(bal);
    s_cnt[1][warp] = (uint32_t)__popc(rbal);
  }
  __syncthreads();
  if (warp < 2) {
    const uint32_t c = lane < kItemThreads / 32 ? s_cnt[warp][lane] : 0u, inc = warp_incl_scan(c);
    uint32_t base = 0;
    if (lane == 31 && inc) base = atomicAdd(counts + warp, inc);
    base = __shfl_sync(FULL, base, 31);
    if (lane < kItemThreads / 32) s_cnt[warp][lane] = base + inc - c;
  }
  __syncthreads();
  const uint32_t below = (1u << lane) - 1u;
  if (start) items[s_cnt[0][warp] + (uint32_t)__popc(bal & below)] = it;
  if (rstart) runs[s_cnt[1][warp] + (uint32_t)__popc(rbal & below)] = run;
}

// Items of one mesh ordered by z slab (order within a slab is free): per-slab counts, their
// exclusive prefix (ioff[0..nslab]), then each item placed in its slab's range.
__global__ void k_item_slab_count(const Item *__restrict__ items,
                                  const uint32_t *__restrict__ nitems, const uint32_t *__restrict__ keys,
                                  const uint32_t *__restrict__ useg, int nz, int zslab,
                                  uint32_t *__restrict__ cnt) {
  const int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= (int64_t)*nitems) return;
  atomicAdd(&cnt[(keys[useg[items[it].ua]] % (uint32_t)nz) / (uint32_t)zslab], 1u);
}

__global__ void k_item_slab_offsets(uint32_t *__restrict__ cnt, int nslab, uint32_t *__restrict__ ioff) {
  if (threadIdx.x != 0) return;
  uint32_t a = 0;
  for (int k = 0; k < nslab; ++k) {
    ioff[k] = a;
    a += cnt[k];
    cnt[k] = ioff[k];  // becomes the slab's placement cursor
  }
  ioff[nslab] = a;
}

__global__ void k_item_slab_place(const Item *__restrict__ items,
                                  const uint32_t *__restrict__ nitems, const uint32_t *__restrict__ keys,
                                  const uint32_t *__restrict__ useg, int nz, int zslab,
                                  uint32_t *__restrict__ cur, uint32_t *__restrict__ ilist) {
  const int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= (int64_t)*nitems) return;
  const uint32_t sl = (keys[useg[items[it].ua]] % (uint32_t)nz) / (uint32_t)zslab;
  ilist[atomicAdd(&cur[sl], 1u)] = (uint32_t)it;
}

// 4 bits -> 4 bytes holding 0 or 1 (bit j to byte j; the shifted copies land on distinct bits).
__device__ __forceinline__ uint32_t byte_flags4(uint32_t x) { return (x * 0x00204081u) & 0x01010101u; }

// 16 cells' mask bits -> their output bytes, 254 boundary, 127 inside, 0 outside.
__device__ __forceinline__ uint4 state_bytes(uint32_t sat, uint32_t in) {
  uint32_t o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    o[k] = byte_flags4((sat >> (4 * k)) & 0xfu) * 254u + byte_flags4((in >> (4 * k)) & 0xfu) * 127u;
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// 16 bits to the even bits of a word.
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x = (x | (x << 8)) & 0x00ff00ffu;
  x = (x | (x << 4)) & 0x0f0f0f0fu;
  x = (x | (x << 2)) & 0x33333333u;
  return (x | (x << 1)) & 0x55555555u;
}

// Transposes 16 sub-columns of a mask (NZ layers each, NZ / 2 words) in place: afterwards half r & 1
// of word r >> 1 holds layer r, bit c for sub-column c.  The usual block swaps: halves, quarters, ...
template <int NZ>
__device__ __forceinline__ void transpose16(uint32_t (&w)[NZ / 2]) {
  if constexpr (NZ == 16) {  // 16 x 16 bits, two sub-columns per word
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t t = ((w[i] >> 8) ^ w[i + 4]) & 0x00ff00ffu;
      w[i + 4] ^= t;
      w[i] ^= t << 8;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = (k & 1) + 4 * (k >> 1);
      const uint32_t t = ((w[i] >> 4) ^ w[i + 2]) & 0x0f0f0f0fu;
      w[i + 2] ^= t;
      w[i] ^= t << 4;
    }
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const uint32_t t = ((w[i] >> 2) ^ w[i + 1]) & 0x33333333u;
      w[i + 1] ^= t;
      w[i] ^= t << 2;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t t = ((w[i] >> 1) ^ (w[i] >> 16)) & 0x5555u;
      w[i] ^= (t << 16) | (t << 1);
    }
  } else {  // two 8 x 8 blocks of four sub-columns per word
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t t = (w[i] ^ (w[i] >> 7)) & 0x00aa00aau;
      w[i] ^= t ^ (t << 7);
      t = (w[i] ^ (w[i] >> 14)) & 0x0000ccccu;
      w[i] ^= t ^ (t << 14);
    }
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      const uint32_t t = ((w[i] >> 4) ^ w[i + 1]) & 0x0f0f0f0fu;
      w[i + 1] ^= t;
      w[i] ^= t << 4;
    }
    // bytes: layers 0-3 of sub-columns 0-7 | layers 4-7 | the same of 8-15 -> halves by layer
    const uint32_t a = w[0], b = w[1], c = w[2], d = w[3];
    w[0] = __byte_perm(a, c, 0x5140);
    w[1] = __byte_perm(a, c, 0x7362);
    w[2] = __byte_perm(b, d, 0x5140);
    w[3] = __byte_perm(b, d, 0x7362);
  }
}

// Output of a chunk whose n2z is NZ (8 or 16), with a multiple of 16 sub-columns and 16-byte aligned
// blocks.  A lane takes 16 sub-columns of one voxel: their SAT and parity bits, transposed to layers,
// are kept in `stage` (a word per layer, conflict-free) and written layer by layer, 16 bytes a lane.  HOST
// (outputs in host memory, voxels of a power of two of units): in output order, 512 bytes of a warp at
// once instead of 64 (8^3 cells) or 256, which the link moves faster: 192^3 / 8^3 host to host 1076 ->
// 1001 us, 1.28 GB of 16^3 cells 6.58 -> 6.47 ms; device memory takes the layers 1-4% faster.
// With `codes`, the voxels whose output index is below `pkend` go out as 2-bit codes instead, a word
// per 16 cells (cell k at bits 2k: 0 outside, 1 inside, 2 boundary), for the host to expand.
template <int NZ, bool HOST>
__device__ __forceinline__ void write_chunk(uint8_t *l2, uint32_t *codes, uint32_t pkend, uint32_t vown,
                                            const uint32_t *satm, const uint32_t *par, const uint32_t *ft,
                                            int m, int ncol2, uint32_t *stage, unsigned long long &nbd,
                                            unsigned long long &nin) {
  const int lane = (int)(threadIdx.x & 31u);
  constexpr int S = HOST && NZ == 8 ? 36 : 32;  // (36: eight layers of four units read without conflicts)
  constexpr int LZ = NZ == 8 ? 3 : 4;
  const int upv = ncol2 >> 4, W = (ncol2 * NZ) >> 5, FW = (ncol2 + 31) >> 5;
  const bool linear = HOST && (upv & (upv - 1)) == 0 && upv <= 32;
  const int sh = 31 - __clz(upv);
  auto put = [&](size_t c, bool packed, uint32_t w) {  // 16-cell group c of the output
    const uint32_t sb = w & 0xffffu, ib = w >> 16;
    if (packed) __stcs(codes + c, spread16(sb) * 2u | spread16(ib));
    else __stcs(reinterpret_cast<uint4 *>(l2) + c, state_bytes(sb, ib));
  };
  uint32_t nb = 0, ni = 0;
#pragma unroll 1
  for (int u0 = 0; u0 < m * upv; u0 += 32) {
    const int u = u0 + lane;
    const bool live = u < m * upv;
    const int jv = live ? u / upv : 0, k = u - jv * upv;  // 16 sub-columns from 16 k
    const uint32_t vidx = __shfl_sync(FULL, vown, jv);
    if (live) {
      uint32_t a[NZ / 2], b[NZ / 2];
      const uint32_t *sw = satm + jv * W + k * (NZ / 2), *pw = par + jv * W + k * (NZ / 2);
#pragma unroll
      for (int i = 0; i < NZ / 2; ++i) {
        a[i] = sw[i];
        b[i] = pw[i];
        nb += (uint32_t)__popc(a[i]);
      }
      transpose16<NZ>(a);
      transpose16<NZ>(b);
      uint32_t f = (ft[jv * FW + (k >> 1)] >> ((k & 1) * 16)) & 0xffffu;
      f |= f << 16;
#pragma unroll
      for (int i = 0; i < NZ / 2; ++i) {
        b[i] = (b[i] ^ f) & ~a[i];
        ni += (uint32_t)__popc(b[i]);
        stage[(2 * i) * S + lane] = __byte_perm(a[i], b[i], 0x5410);
        stage[(2 * i + 1) * S + lane] = __byte_perm(a[i], b[i], 0x7632);
      }
    }
    // streaming stores: the output is not read again, so it should not displace the working set
    if (linear) {
      __syncwarp();
      const int total = min(32, m * upv - u0) * NZ;
#pragma unroll 1
      for (int i0 = 0; i0 < total; i0 += 32) {
        const int i = i0 + lane, slot = i >> (sh + LZ), rem = i & ((NZ << sh) - 1);
        const uint32_t v = __shfl_sync(FULL, vown, ((u0 >> sh) + slot) & 31);
        const uint32_t w = stage[(rem >> sh) * S + (slot << sh) + (rem & (upv - 1))];
        if (i < total) put((size_t)v * (size_t)(NZ * upv) + (size_t)rem, v < pkend, w);
      }
      __syncwarp();
    } else if (live) {
      const size_t c0 = (size_t)vidx * (size_t)(NZ * upv) + (size_t)k;  // 16-cell group of layer 0
#pragma unroll 1
      for (int r = 0; r < NZ; ++r) put(c0 + (size_t)(r * upv), vidx < pkend, stage[r * S + lane]);
    }
  }
  nbd += nb;
  nin += ni;
}

// Output of a chunk of any other layout in host memory, for voxels of at least kHostBytes cells: a lane
// takes 16 bytes at a 16-byte boundary of a voxel's block, in output order, and stores the words of a
// block's two ends one by one.  (A byte a lane and layer, as in device memory, left the link waiting:
// 262k-triangle torus at 128^3 host to host, us, by bytes and so: 5^3 722 and 623, 7^3 1215 and 792, 12^3
// 3007 and 1567; 4^3 479 and 398, but 3^3, whose blocks are mostly ends, 487 and 530.)
constexpr int kHostBytes = 64;
__device__ __forceinline__ void write_host_bytes(uint8_t *l2, uint32_t vown, const uint32_t *satm,
                                                 const uint32_t *par, const uint32_t *ft, int m, int ncol2,
                                                 int n2z, unsigned long long &nbd, unsigned long long &nin) {
  const int lane = (int)(threadIdx.x & 31u);
  const int cells = ncol2 * n2z, W = (cells + 31) >> 5, FW = (ncol2 + 31) >> 5;
  const int groups = (cells + 30) >> 4;  // 16-byte blocks that a voxel's bytes can touch
  uint32_t nb = 0, ni = 0;
#pragma unroll 1
  for (int u0 = 0; u0 < m * groups; u0 += 32) {
    const int u = u0 + lane;
    const bool live = u < m * groups;
    const int jv = live ? u / groups : 0;
    uint8_t *const o = l2 + (size_t)__shfl_sync(FULL, vown, jv) * cells;
    const int c0 = 16 * (u - jv * groups) - (int)(reinterpret_cast<uintptr_t>(o) & 15u);  // cell of byte 0
    const int b0 = max(-c0, 0), b1 = min(cells - c0, 16);
    if (!live || b0 >= b1) continue;
    const uint32_t *sv = satm + jv * W, *pv = par + jv * W, *fv = ft + jv * FW;
    int r = (c0 + b0) / ncol2, pq = c0 + b0 - r * ncol2;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int b = 0; b < 16; ++b) {
      if (b < b0 || b >= b1) continue;
      const int off = pq * n2z + r;
      const uint32_t s = (sv[off >> 5] >> (off & 31)) & 1u;
      const uint32_t i = ((pv[off >> 5] >> (off & 31)) ^ (fv[pq >> 5] >> (pq & 31))) & 1u & ~s;
      w[b >> 2] |= (s * 254u + i * 127u) << (8 * (b & 3));
      nb += s;
      ni += i;
      if (++pq == ncol2) {
        pq = 0;
        ++r;
      }
    }
    if (b1 - b0 == 16) {
      __stcs(reinterpret_cast<uint4 *>(o + c0), make_uint4(w[0], w[1], w[2], w[3]));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (b0 <= 4 * k && b1 >= 4 * k + 4) {
          __stcs(reinterpret_cast<uint32_t *>(o + c0) + k, w[k]);
        } else {
#pragma unroll
          for (int b = 4 * k; b < 4 * k + 4; ++b)
            if (b >= b0 && b < b1) __stcs(reinterpret_cast<char *>(o + c0) + b, (char)(w[k] >> (8 * (b & 3))));
        }
      }
    }
  }
  nbd += nb;
  nin += ni;
}

// n2z bits of a Level2 column starting at bit `off` of a mask.
__device__ __forceinline__ uint32_t column_bits(const uint32_t *m, int off, int n2z) {
  const int sh = off & 31;
  uint32_t b = m[off >> 5] >> sh;
  if (sh + n2z > 32) b |= m[(off >> 5) + 1] << (32 - sh);
  return b;
}

// ---- stencil fill, column prefix ------------------------------------------------------------------
// A triangle whose topmost record in a Level1 column lies below voxel v is not recorded in any
// voxel from v up, so within the column's x/y extent it lies below v's bottom face, up to the
// SAT's rounding: every covered sample keeps it in every slice of v and above, unless that rounding
// exceeds the half Level2 cell to v's first clip height (coordinates large against the cells, slivers).
// The heights show where it does; the column's chunks above then draw all of its triangles.
// Elsewhere a Level2 chunk starts from the XOR of
// the sample coverage of the column's triangles whose topmost record lies below its first voxel,
// and draws only the triangles recorded from that voxel up (otherwise every chunk of a tall
// column would draw all the triangles below it again).  Two passes, since the XOR is order-free:
//   k_stencil_segment  one warp per work item: the coverage XOR of the triangles whose topmost
//                      record lies in the item's own voxels (items that end their column skip it),
//                      stored at the item's first voxel, with a last word that says whether one of
//                      the samples is not below the next item's clip heights;
//   k_stencil_scan     one warp per column with more than one item: those masks turned in place
//                      into exclusive XOR prefixes, the mask each item starts from, and the last
//                      words into 0 or, above such a sample, 1 + the column's first voxel.
// (One warp per column walking all of its records was latency-bound on the few long columns:
// 186 us on torus262k at 22% warps active.)
constexpr int kPrefixWarps = 4;
constexpr int kPrefixMaskWords = 128;  // 4 * 32 * 32 samples / 32

__global__ void __launch_bounds__(kPrefixWarps * 32) k_stencil_segment(
    BatchDev bd, const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals,
    const uint32_t *__restrict__ useg, const Item *__restrict__ items, const uint32_t *__restrict__ nitems) {
  __shared__ uint32_t s_mask[kPrefixWarps][kPrefixMaskWords];
  __shared__ StRec s_t[kPrefixWarps][32];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int64_t it = (int64_t)blockIdx.x * kPrefixWarps + warp;
  if (it >= (int64_t)*nitems) return;
  const Item w = items[it];
  const uint32_t ua = w.ua, ue = ua + (w.m_mesh & 63u);  // the item's voxels [ua, ue)
  if (ue >= w.col_end) return;  // the column's last item: no item reads it
  const MeshDesc &d = bd.md[w.m_mesh >> 7];
  const GridDev &g = d.g;
  const int n2x = g.n2[0], n2y = g.n2[1], nx = g.n[0];
  const int SW = 2 * n2x, SH = 2 * n2y;
  const int FWS = (4 * n2x * n2y + 31) >> 5;
  const uint32_t col = w.col;
  const int ci = (int)(col % (uint32_t)nx), cj = (int)(col / (uint32_t)nx);
  const float lx = fa(fm((float)ci, g.g[0]), g.bmin[0]), hx = fa(lx, g.g[0]);
  const float ly = fa(fm((float)cj, g.g[1]), g.bmin[1]), hy = fa(ly, g.g[1]);
  uint32_t *mask = s_mask[warp];
  for (int w = lane; w < FWS; w += 32) mask[w] = 0;
  __syncwarp();
  // the lowest clip height of the column's voxels from ue up (where the heights do not increase, less
  // their distance from their affine form)
  const uint32_t kz = keys[useg[ue]] - col * (uint32_t)g.n[2];
  float clip = __ldg(g.o2[2] + (size_t)kz * g.n2[2]);
  if (!g.oz_monotone) clip -= 10.3f * EPS24 * fmaxf(fabsf(g.bmin[2]), fabsf(g.bmax[2]));
  bool over = false;
  const float4 *__restrict__ ptri = d.ptri;
  const uint32_t e0 = useg[ua], e1 = useg[ue];
  for (uint32_t b0 = e0; b0 < e1; b0 += 32) {
    const uint32_t e = b0 + lane;
    const uint32_t vv = e < e1 ? vals[e] : 0u;
    StTri st = {};
    bool has = false;
    if (vv & 0x80000000u) {  // the triangle's topmost record in the column
      const uint32_t t = vv & 0x7fffffffu;
      const float4 a0 = __ldg(ptri + 3 * (size_t)t), a1 = __ldg(ptri + 3 * (size_t)t + 1),
                   a2 = __ldg(ptri + 3 * (size_t)t + 2);
      const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
      has = st_setup(V, lx, hx, ly, hy, SW, SH, st);
    }
    const StBatch batch(s_t[warp], has, st);
    __syncwarp();
    for (uint32_t w0 = 0; w0 < batch.total; w0 += 32) {
      const StRec &r = batch.owner(s_t[warp], w0);
      int sx, sy;
      float zs;
      if (w0 + lane < batch.total && st_sample(r, w0 + lane, sx, sy, zs)) {
        const int sidx = sy * SW + sx;
        atomicXor(&mask[sidx >> 5], 1u << (sidx & 31));
        over = over || !(zs <= clip);
      }
    }
    __syncwarp();
  }
  uint32_t *out = bd.stp + (size_t)ua * bd.stp_words;
  for (int w = lane; w < FWS; w += 32) out[w] = mask[w];
  over = __any_sync(FULL, over);
  if (lane == 0) out[bd.stp_words - 1] = over ? 1u : 0u;
}

__global__ void __launch_bounds__(kPrefixWarps * 32) k_stencil_scan(
    BatchDev bd, const uint32_t *__restrict__ iflag, const Item *__restrict__ items,
    const uint32_t *__restrict__ nitems) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int64_t it = (int64_t)blockIdx.x * kPrefixWarps + warp;
  if (it >= (int64_t)*nitems) return;
  const Item w0 = items[it];
  const uint32_t u0 = w0.ua, u1 = w0.col_end;
  // the warp of a column's first item takes the column; a one-item column has nothing to scan
  if (!((w0.m_mesh >> 6) & 1u) || u0 + (w0.m_mesh & 63u) >= u1) return;
  const MeshDesc &d = bd.md[w0.m_mesh >> 7];
  const int FWS = (4 * d.g.n2[0] * d.g.n2[1] + 31) >> 5;  // <= kPrefixMaskWords
  uint32_t acc[kPrefixMaskWords / 32] = {}, over = 0;
  // the column's item starts 32 voxels at a time (one flag load per lane), then each in order
  for (uint32_t base = u0; base < u1; base += 32) {
    const uint32_t uu = base + lane;
    uint32_t starts = __ballot_sync(FULL, uu < u1 && (uu == u0 || iflag[uu] != 0u));
    while (starts) {
      const uint32_t u = base + (uint32_t)(__ffs(starts) - 1);
      starts &= starts - 1u;
      uint32_t *m = bd.stp + (size_t)u * bd.stp_words;
#pragma unroll
      for (int k = 0; k < kPrefixMaskWords / 32; ++k) {
        const int w = (int)lane + 32 * k;
        if (w < FWS) {
          const uint32_t seg = m[w];  // (the column's last item wrote none: its value goes unused)
          m[w] = acc[k];
          acc[k] ^= seg;
        }
      }
      if (lane == 0) {
        const uint32_t o = m[bd.stp_words - 1];
        m[bd.stp_words - 1] = over ? u0 + 1u : 0u;
        over |= o;
      }
    }
  }
}

// ---- Level2 ------------------------------------------------------------------------------------
// The exact SAT of queued (triangle, voxel, sub-column, cell range) records, one per lane: cells
// that another triangle has marked already are left out (the state is an OR).
__device__ __noinline__ void sat_exact(const MeshDesc &d, WarpScratch &ws, uint32_t *sat,
                                       const int *kz, const uint32_t *xy, uint32_t nr) {
  const unsigned lane = threadIdx.x & 31u;
  __syncwarp();
  if (lane < nr) {
    const GridDev &g = d.g;
    const int n2x = g.n2[0], n2z = g.n2[2];
    const int W = (n2x * g.n2[1] * n2z + 31) >> 5;
    const uint32_t t = ws.rtri[lane], pos = ws.rpos[lane];
    const int jv = (int)(pos & 31u), p = (int)((pos >> 5) & 31u), q = (int)((pos >> 10) & 31u);
    const int lo = (int)((pos >> 15) & 63u), end = (int)(pos >> 21);
    uint32_t *m = sat + jv * W;
    const int off = (q * n2x + p) * n2z, sh = off & 31;
    uint32_t done = m[off >> 5] >> sh;
    if (sh + n2z > 32) done |= m[(off >> 5) + 1] << (32 - sh);
    uint32_t todo = ((0xffffffffu >> (32 - (end - lo))) << lo) & ~done;
    if (todo) {
      const float4 a0 = __ldg(d.ptri + 3 * (size_t)t), a1 = __ldg(d.ptri + 3 * (size_t)t + 1),
                   a2 = __ldg(d.ptri + 3 * (size_t)t + 2);
      const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
      const float h[3] = {g.e2[0], g.e2[1], g.e2[2]};
      const uint32_t c = xy[jv];
      SatCol sc;
      if (sat_col(V, __ldg(g.c2s[0] + (size_t)(c & 0xffffu) * n2x + p),
                  __ldg(g.c2s[1] + (size_t)(c >> 16) * g.n2[1] + q), h, sc)) {
        const float *sz = g.c2s[2] + (size_t)kz[jv] * n2z;
        uint32_t bits = 0;
#pragma unroll 1
        while (todo) {
          const int r = __ffs(todo) - 1;
          todo &= todo - 1u;
          if (sat_z(sc, V, __ldg(sz + r), h)) bits |= 1u << r;
        }
        if (bits) {
          atomicOr(&m[off >> 5], bits << sh);
          if (sh + n2z > 32) atomicOr(&m[(off >> 5) + 1], bits >> (32 - sh));
        }
      }
    }
  }
  __syncwarp();
}

// The exact x/y tests of a sub-column of the voxel at xy.
__device__ __noinline__ bool column_passes(const MeshDesc &d, uint32_t t, uint32_t xy, int p, int q) {
  const GridDev &g = d.g;
  const float4 a0 = __ldg(d.ptri + 3 * (size_t)t), a1 = __ldg(d.ptri + 3 * (size_t)t + 1),
               a2 = __ldg(d.ptri + 3 * (size_t)t + 2);
  const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
  const float h[3] = {g.e2[0], g.e2[1], g.e2[2]};
  SatCol sc;
  return sat_col(V, __ldg(g.c2s[0] + (size_t)(xy & 0xffffu) * g.n2[0] + p),
                 __ldg(g.c2s[1] + (size_t)(xy >> 16) * g.n2[1] + q), h, sc);
}

// The exact ray tests of queued (triangle, sub-column) records, one per lane: the toggles of the
// chunk's voxels at or below the triangle's topmost voxel, top down.
__device__ __noinline__ void fill_exact(const MeshDesc &d, WarpScratch &ws, uint32_t *par,
                                        uint32_t *ft, const int *kz, int m, int ci, int cj,
                                        uint32_t nr) {
  const unsigned lane = threadIdx.x & 31u;
  __syncwarp();
  if (lane < nr) {
    const GridDev &g = d.g;
    const int n2x = g.n2[0], n2z = g.n2[2], ncol2 = n2x * g.n2[1];
    const int W = (ncol2 * n2z + 31) >> 5, FW = (ncol2 + 31) >> 5;
    const uint32_t t = ws.rtri[lane], pos = ws.rpos[lane];
    const int p = (int)((pos >> 6) & 31u), q = (int)(pos >> 11), pq = q * n2x + p;
    const float4 a0 = __ldg(d.ptri + 3 * (size_t)t), a1 = __ldg(d.ptri + 3 * (size_t)t + 1),
                 a2 = __ldg(d.ptri + 3 * (size_t)t + 2);
    const float4 fb = __ldg(d.fbox + t);
    const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
    RayTri rt;
    ray_tri_pre(V, a2.w, rt);
    RayCol rc;
    if (ray_col(rt, __ldg(g.o2[0] + (size_t)ci * n2x + p), __ldg(g.o2[1] + (size_t)cj * g.n2[1] + q), rc)) {
      const float *ozt = g.o2[2];
      // Certification bound E2, or 0 where there is none: an unbounded box marks an ill-conditioned
      // x/y projection.  |t - t*| <= 8.2 eps M1 |1/det| for every origin of the chunk (t* exact,
      // affine and decreasing in the origin height), with M1 taken at the largest |Tz| over the
      // chunk's origins; 16 eps gives the float evaluation room.
      float E2 = 0.f;
      if (g.oz_monotone && !isinf(fb.x) && !isinf(fb.z)) {
        const float Zm = fmaxf(fabsf(__ldg(ozt + (size_t)kz[0] * n2z) - rt.v1z),
                               fabsf(__ldg(ozt + (size_t)kz[m - 1] * n2z + n2z - 1) - rt.v1z)) * 1.0001f;
        const float atx = fabsf(rc.Tx), aty = fabsf(rc.Ty);
        const float M1 = fabsf(rt.e2x) * (aty * fabsf(rt.e1z) + Zm * fabsf(rt.e1y)) +
                         fabsf(rt.e2y) * (Zm * fabsf(rt.e1x) + atx * fabsf(rt.e1z)) +
                         fabsf(rt.e2z) * (atx * fabsf(rt.e1y) + aty * fabsf(rt.e1x));
        E2 = 2.f * 16.f * EPS24 * M1 * fabsf(rt.inv_det) * 1.0001f;
      }
      const bool well = E2 > 0.f;
#pragma unroll 1
      for (int jv = (int)(pos & 63u) - 1; jv >= 0; --jv) {
        const float *oz = ozt + (size_t)kz[jv] * n2z;
        uint32_t bits = 0;
        if (well) {
          const float otop = __ldg(oz + n2z - 1);
          const float ttop = ray_tval(rt, rc, otop);
          if (ttop > g.thr + E2) {
            // this voxel and every lower voxel of the chunk are hit at every origin
            atomicXor(&ft[jv * FW + (pq >> 5)], 1u << (pq & 31));
            break;
          }
          // Along +z, t* (exact) grows by exactly the drop of the origin below otop:
          // t*(oz) = t*(otop) + (otop - oz), and the float t at every origin and at otop lies
          // within E2/2 of t*.  So with d = otop - oz, the float t exceeds thr when
          // d > thr - ttop + E2 and does not when d <= thr - ttop - E2; the thresholds carry the
          // rounding of d and of themselves (K bounds every magnitude involved).  Origins
          // between the two run the exact test.
          const float dmax = otop - __ldg(oz);
          const float K = fabsf(ttop) + dmax + g.thr;
          const float slack = E2 * 1.0001f + 8.f * EPS24 * K + 1e-30f;
          const float dhit = (g.thr - ttop) + slack, dmiss = (g.thr - ttop) - slack;
          // d = otop - oz rounds monotonically and falls as r grows, so the certain hits are the
          // origins r < rh and the exact tests the band rh <= r < rm
          const int rh = count_drop_above(oz, n2z, otop, dhit, g.inv_g2[2]);
          const int rm = count_drop_above(oz, n2z, otop, dmiss, g.inv_g2[2]);
          bits = rh >= 32 ? 0xffffffffu : ((1u << rh) - 1u);
#pragma unroll 1
          for (int r = rh; r < rm; ++r)
            if (ray_t(rt, rc, __ldg(oz + r), g.thr)) bits |= 1u << r;
        } else {
#pragma unroll 1
          for (int r = 0; r < n2z; ++r)
            if (ray_t(rt, rc, __ldg(oz + r), g.thr)) bits |= 1u << r;
        }
        if (bits) xor_column(par + jv * W, pq, n2z, bits);
      }
    }
  }
  __syncwarp();
}

// The exact u/v test of a sub-column's ray.
__device__ __noinline__ bool ray_passes(const MeshDesc &d, uint32_t t, int ci, int cj, int p, int q) {
  const GridDev &g = d.g;
  const float4 a0 = __ldg(d.ptri + 3 * (size_t)t), a1 = __ldg(d.ptri + 3 * (size_t)t + 1),
               a2 = __ldg(d.ptri + 3 * (size_t)t + 2);
  const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
  RayTri rt;
  ray_tri_pre(V, a2.w, rt);
  RayCol rc;
  return ray_col(rt, __ldg(g.o2[0] + (size_t)ci * g.n2[0] + p), __ldg(g.o2[1] + (size_t)cj * g.n2[1] + q), rc);
}

// Appends the records of the lanes with `push` to the exact-work queue and returns its length.
__device__ __forceinline__ uint32_t queue_push(WarpScratch &ws, uint32_t nrec, bool push, uint32_t tri,
                                               uint32_t pos) {
  const uint32_t bal = __ballot_sync(FULL, push);
  if (!bal) return nrec;
  if (push) {
    const uint32_t k = nrec + __popc(bal & ((1u << (threadIdx.x & 31u)) - 1u));
    ws.rtri[k] = tri;
    ws.rpos[k] = pos;
  }
  return nrec + (uint32_t)__popc(bal);
}
// Moves the records beyond the first 32 to the front (fewer than 32 of them).
__device__ __forceinline__ uint32_t queue_shift(WarpScratch &ws, uint32_t nrec) {
  const unsigned lane = threadIdx.x & 31u;
  const bool more = lane + 32 < nrec;
  const uint32_t a = more ? ws.rtri[lane + 32] : 0u, b = more ? ws.rpos[lane + 32] : 0u;
  __syncwarp();
  if (more) {
    ws.rtri[lane] = a;
    ws.rpos[lane] = b;
  }
  __syncwarp();
  return nrec - 32;
}

// The next work item of a persistent launch (one ticket per warp): all items, or (z slabs) this
// launch's slab of the slab-ordered item list.  False: none left.
// With `parts` > 1 each item comes that many times, its `part` counted up.
__device__ __forceinline__ bool next_item(uint32_t *ticket, const Item *__restrict__ items,
                                          const uint32_t *__restrict__ nitems, int slab,
                                          const uint32_t *__restrict__ ilist,
                                          const uint32_t *__restrict__ ioff, uint32_t parts, Item &it,
                                          uint32_t &part) {
  uint32_t tk = 0;
  if ((threadIdx.x & 31u) == 0) tk = atomicAdd(ticket, 1u);
  tk = __shfl_sync(FULL, tk, 0);
  part = 0;
  if (parts > 1) {
    part = tk % parts;
    tk /= parts;
  }
  if (ilist) {
    const uint32_t i0 = ioff[slab];
    if (tk >= ioff[slab + 1] - i0) return false;
    tk = ilist[i0 + tk];
  } else if (tk >= *nitems) {
    return false;
  }
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(items + tk));
  it = {v.x, v.y, v.z, v.w};
  return true;
}

// Words of a boundary voxel's SAT mask in BatchDev::smask: disjoint for every (mesh, voxel), since
// the l2_base cells and u_base voxels of the meshes before fill fewer.
__device__ __forceinline__ uint32_t *sat_words(const BatchDev &bd, const MeshDesc &d, uint32_t u, int W) {
  return bd.smask + (d.l2_base >> 5) + d.u_base + ((int64_t)u - d.u_base) * W;
}

// The SAT and the fill are two kernels: one with both is 72 KB of code, and its warps, spread over
// all of it, waited for instructions more than for anything else (4.9 of 12.5 cycles per issue on a
// 262k-triangle torus, 128^3 / 8^3; 0.2 with two kernels).  The SAT masks go through device memory
// (one bit per cell).  Both kernels are bound by instruction issue.  Measured against one kernel
// testing every (triangle, sub-column) and listed cell exactly, both kernels together: the torus
// 487 -> 200 us, a 1.3M-triangle star at 256^3 / 16^3 3.51 -> 1.25 ms, 256 mixed meshes in one call
// 19.9 -> 8.5 ms.  A twentieth of the instructions are exact tests (0.4-2.7% of the sub-columns on these
// meshes, whose coordinates are of the grid's own size; far from the origin the share grows: see kWide).
// Rows are solved by a lane per triangle looping over them (a lane per row took 190 us for the torus'
// SAT against 134); the sub-columns they leave are listed and taken a lane each, because lanes that
// walked their own row had 43-52% of them at work in the SAT and 34% in the fill (the star: SAT
// 787 -> 690 us, fill 712 -> 577; the torus 135 -> 113 and 101 -> 84; the batch 5.7 -> 5.4 ms and
// 5.1 -> 4.5).
//
// k_level2c_sat: bd.smask gets every boundary voxel's mask of Level2 boundary cells.
__global__ void __launch_bounds__(kWarps * 32, 6) k_level2c_sat(
    BatchDev bd, const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals,
    const uint32_t *__restrict__ useg, const Item *__restrict__ items,
    const uint32_t *__restrict__ nitems, int per_warp, int slab, const uint32_t *__restrict__ ilist,
    const uint32_t *__restrict__ ioff, int parts) {
  extern __shared__ __align__(16) uint32_t sm[];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  WarpScratch &ws = *reinterpret_cast<WarpScratch *>(sm + (size_t)warp * per_warp);
  int *const kz = reinterpret_cast<int *>(&ws + 1);
  uint32_t *const xy = reinterpret_cast<uint32_t *>(kz + 32), *const sat = xy + 32;
  Item it;
  uint32_t part;
  while (next_item(bd.queue + 1 + kSlabsMax + slab, items, nitems, slab, ilist, ioff, (uint32_t)parts, it, part)) {
  const uint32_t ua = it.ua;
  const MeshDesc &d = bd.md[it.m_mesh >> 7];
  const GridDev &g = d.g;
  const float4 *__restrict__ ptri = d.ptri;
  const int n2x = g.n2[0], n2y = g.n2[1], n2z = g.n2[2];
  const int W = (n2x * n2y * n2z + 31) >> 5;
  const int m = (int)(it.m_mesh & 63u);
#pragma unroll 1
  for (int w = lane; w < m * W; w += 32) sat[w] = 0;
  if ((int)lane < m) {
    const uint32_t e = useg[ua + lane], key = keys[e], col = key / (uint32_t)g.n[2];
    const uint32_t cj = col / (uint32_t)g.n[0];
    ws.seg[lane] = e;
    kz[lane] = (int)(key - col * (uint32_t)g.n[2]);
    xy[lane] = (col - cj * (uint32_t)g.n[0]) | (cj << 16);
  }
  if (lane == 0) ws.seg[m] = useg[ua + m];
  __syncwarp();

  // ---------------- SAT of each voxel's own triangles: the run's (voxel, triangle) pairs are
  // contiguous in the sorted lists and are taken 32 at a time across voxel boundaries.
  const float gx = g.g2[0], gy = g.g2[1], gz = g.g2[2];
  uint32_t nrec = 0;
  {
    const float h0 = g.e2[0], h1 = g.e2[1], h2 = g.e2[2];
    // this part's share of the pairs
    const uint32_t n0 = ws.seg[0], np_ = ws.seg[m] - n0;
    const uint32_t S0 = n0 + (uint32_t)((uint64_t)np_ * part / (uint32_t)parts);
    const uint32_t S1 = n0 + (uint32_t)((uint64_t)np_ * (part + 1) / (uint32_t)parts);
    uint32_t taken;  // pairs of a batch: 32, fewer where their rows or sub-columns would not fit
#pragma unroll 1
    for (uint32_t b0 = S0; b0 < S1; b0 += taken) {
      // ---- one triangle per lane: its cell ranges, its plane and its rows
      const uint32_t e = b0 + lane;
      int p0 = 0, p1 = -1, pi = 0, pe = 0, q0 = 0, q1 = -1, qi = 0, qe = 0, r0 = 0, r1 = -1, ri = 0, re = 0;
      bool direct = false, wide = false, on = false;
      uint32_t nsolve = 0, ncol = 0, t = 0;
      int jv = 0;  // last voxel whose segment starts at or before e
      float4 a0, a1, a2;
      float R = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
      const float *sx = nullptr, *sy = nullptr, *sz = nullptr;
      if (e < S1) {
#pragma unroll
        for (int st = 16; st > 0; st >>= 1)
          if (jv + st <= m - 1 && ws.seg[jv + st] <= e) jv += st;
        const uint32_t c = xy[jv];
        sx = g.c2s[0] + (size_t)(c & 0xffffu) * n2x;
        sy = g.c2s[1] + (size_t)(c >> 16) * n2y;
        sz = g.c2s[2] + (size_t)kz[jv] * n2z;
        const float sx0 = __ldg(sx), sx1 = __ldg(sx + n2x - 1), sy0 = __ldg(sy), sy1 = __ldg(sy + n2y - 1);
        const float sz0 = __ldg(sz), sz1 = __ldg(sz + n2z - 1);
        t = vals[e] & 0x7fffffffu;
        a0 = __ldg(ptri + 3 * (size_t)t), a1 = __ldg(ptri + 3 * (size_t)t + 1),
        a2 = __ldg(ptri + 3 * (size_t)t + 2);
        const float xn = fminf(a0.x, fminf(a1.x, a2.x)), xx = fmaxf(a0.x, fmaxf(a1.x, a2.x));
        const float yn = fminf(a0.y, fminf(a1.y, a2.y)), yx = fmaxf(a0.y, fmaxf(a1.y, a2.y));
        const float zn = fminf(a0.z, fminf(a1.z, a2.z)), zx = fmaxf(a0.z, fmaxf(a1.z, a2.z));
        // Distance of the centre tables from their affine form within a voxel: two roundings (eps
        // times the coordinate) of the formulas' doubles.
        tx = 2.02f * EPS24 * fmaxf(fabsf(sx0), fabsf(sx1));
        ty = 2.02f * EPS24 * fmaxf(fabsf(sy0), fabsf(sy1));
        tz = 2.02f * EPS24 * fmaxf(fabsf(sz0), fabsf(sz1));
        cell_ranges(xn, xx, sx0, g.inv_g2[0], n2x, ff(tx, g.inv_g2[0], kIdx), p0, p1, pi, pe);
        cell_ranges(yn, yx, sy0, g.inv_g2[1], n2y, ff(ty, g.inv_g2[1], kIdx), q0, q1, qi, qe);
        cell_ranges(zn, zx, sz0, g.inv_g2[2], n2z, ff(tz, g.inv_g2[2], kIdx), r0, r1, ri, re);
        // R bounds every vertex coordinate relative to a cell of the range, |V - c|, and with it
        // every edge.  In units of eps R^2 (eps = 2^-24) the float sides of an edge test are off
        // by less than 12 + 4 (position, radius), solve_rows' by less than 13 + 4 + 15 + 6 + 8
        // (position, radius, S, sums, slope): 62, and 66 with the slope's 1/16.  In units of
        // eps R^2 (R + h) the plane test's value is off by less than 78 and the one below by less
        // than 90: 168, 179 with the slope's.
        R = 1.0001f * fmaxf(xx - xn + 1.25f * gx + 2.f * tx,
                            fmaxf(yx - yn + 1.25f * gy + 2.f * ty, zx - zn + 1.25f * gz + 2.f * tz));
        if (p0 <= p1 && q0 <= q1 && r0 <= r1) {
          const int np = p1 - p0 + 1, nq = q1 - q0 + 1;
          // A few cells are tested as fast as they are solved; outside these magnitudes the
          // bounds' own arithmetic could leave the normal range.
          wide = fmaxf(tx * g.inv_g2[0], fmaxf(ty * g.inv_g2[1], tz * g.inv_g2[2])) > kWide;
          direct = np * nq * (r1 - r0 + 1) <= kDirectCells || !(R > 1e-9f && R < 1e9f) || wide;
          on = true;
          nsolve = direct ? 0u : (uint32_t)(2 * nq + np);
        }
      }
      const uint32_t is = warp_incl_scan(nsolve);
      taken = (uint32_t)__popc(__ballot_sync(FULL, is <= (uint32_t)kSol));
      on = on && lane < taken;
      const uint32_t so0 = is - nsolve;
      if (on) {
        const int np_ = p1 - p0 + 1, nq_ = q1 - q0 + 1;
        ws.me[lane] = make_uint4(t, (uint32_t)(jv | (direct ? 256 : 0) | (wide ? 512 : 0) | (p0 << 16) | (q0 << 24)),
                                 (so0 + (uint32_t)nq_) | ((so0 + 2u * (uint32_t)nq_) << 16),
                                 (uint32_t)(r0 | ((r1 + 1) << 8)));
        ncol = (uint32_t)(np_ * nq_);
        if (!direct) {
          const int np = p1 - p0 + 1, nq = q1 - q0 + 1;
          const float c0x = __ldg(sx + p0), c0y = __ldg(sy + q0), c0z = __ldg(sz + r0);
          const float ux = a0.x - c0x, uy = a0.y - c0y, uz = a0.z - c0z;
          const float vx = a1.x - c0x, vy = a1.y - c0y, vz = a1.z - c0z;
          const float wx = a2.x - c0x, wy = a2.y - c0y, wz = a2.z - c0z;
          // plane: a cell passes when |n . (V0 - c)| <= Hs; along z that is one interval
          float nx = (vy - uy) * (wz - vz) - (vz - uz) * (wy - vy);
          float ny = (vz - uz) * (wx - vx) - (vx - ux) * (wz - vz);
          float nz_ = (vx - ux) * (wy - vy) - (vy - uy) * (wx - vx);
          if (nz_ < 0.f) { nx = -nx; ny = -ny; nz_ = -nz_; }
          const float E = 192.f * EPS24 * R * R * (R + fmaxf(h0, fmaxf(h1, h2))) +
                          1.1f * (fabsf(nx) * tx + fabsf(ny) * ty + nz_ * tz);
          const float inv = rcp_fast(fmaxf(nz_ * gz, E * (1.f / 512.f)));
          const float w = ff(E, inv, kIdx);
          ws.xa[lane] = make_float4(nx * ux + ny * uy + nz_ * uz, nx * gx, ny * gy,
                                    fabsf(nx) * h0 + fabsf(ny) * h1 + nz_ * h2);
          ws.xb[lane] = make_float4(inv, (float)r0 - w, (float)r0 + w, 0.f);
          const float dl = 72.f * EPS24 * R * R, bx = 1.1f * tx, by = 1.1f * ty, bz = 1.1f * tz;
          uint32_t *so = ws.sol + so0;
          const uint32_t xl = (uint32_t)(p0 | (pi << 16)), xe = (uint32_t)(pe | ((p1 + 1) << 16));
          const uint32_t zl = (uint32_t)(r0 | (ri << 16)), ze = (uint32_t)(re | ((r1 + 1) << 16));
          ncol = solve_rows(so, nq, ux, vx, wx, uy, vy, wy, h0, h1, gx, gy, dl, bx, by, p0, xl, xe, qi - q0, qe - q0);
          solve_rows(so + nq, nq, uz, vz, wz, uy, vy, wy, h2, h1, gz, gy, dl, bz, by, r0, zl, ze, qi - q0, qe - q0);
          solve_rows(so + 2 * nq, np, uz, vz, wz, ux, vx, wx, h2, h0, gz, gx, dl, bz, bx, r0, zl, ze, pi - p0, pe - p0);
        }
      }
      // ---- the sub-columns that can pass x/y, listed so that every lane takes one
      if (!on) ncol = 0;
      const uint32_t ic = warp_incl_scan(ncol);
      taken = (uint32_t)__popc(__ballot_sync(FULL, lane < taken && ic <= (uint32_t)kCols));
      if (on && lane < taken)
        list_columns(ws.cols + (ic - ncol), direct ? nullptr : ws.sol + so0, (int)lane, p0, p1 - p0 + 1, 0, q1 - q0 + 1);
      const uint32_t C = __shfl_sync(FULL, ic, (int)taken - 1);
      __syncwarp();
#pragma unroll 1
      for (uint32_t c0 = 0; c0 < C; c0 += 32) {
        const uint32_t c = c0 + lane;
        bool amb = false;
        uint32_t tri = 0, pos = 0;
        if (c < C) {
          const uint32_t en = ws.cols[c];
          const int tl = (int)(en & 31u), dq = (int)((en >> 5) & 31u), dp = (int)((en >> 10) & 31u);
          const uint4 me = ws.me[tl];
          const int p = (int)((me.y >> 16) & 255u) + dp, q = (int)(me.y >> 24) + dq;
          const int j = (int)(me.y & 255u);
          int lo, end;
          if (me.y & 256u) {
            lo = (int)(me.w & 255u);
            end = (int)(me.w >> 8);
            amb = !(me.y & 512u) || column_passes(d, me.x, xy[j], p, q);
          } else {
            const float4 xa = ws.xa[tl], xb = ws.xb[tl];
            const uint32_t syz = ws.sol[(me.z & 0xffffu) + (uint32_t)dq], sxz = ws.sol[(me.z >> 16) + (uint32_t)dp];
            const float nv = ff(-(float)dp, xa.y, ff(-(float)dq, xa.z, xa.x));
            const float va = nv - xa.w, vb = nv + xa.w;
            const uint32_t L = __vimax3_s16x2(cvt_pair_ceil(ff(va, xb.x, xb.y), ff(va, xb.x, xb.z)),
                                              __byte_perm(syz, 0, 0x4140), __byte_perm(sxz, 0, 0x4140));
            const uint32_t E = __vimin3_s16x2(
                cvt_pair_floor(ff(vb, xb.x, xb.y + 1.f), ff(vb, xb.x, xb.z + 1.f)),
                __byte_perm(syz, 0, 0x4342), __byte_perm(sxz, 0, 0x4342));
            const int lo_i = (int)L >> 16, end_i = (int)(short)(E & 0xffffu);
            lo = (int)(short)(L & 0xffffu);
            end = (int)E >> 16;
            const bool sure = (en & 0x8000u) != 0;
            if (sure && lo_i < end_i)
              or_column(sat + j * W, q * n2x + p, n2z, (0xffffffffu >> (32 - (end_i - lo_i))) << lo_i);
            amb = lo < end && !(sure && lo == lo_i && end == end_i);
          }
          tri = me.x;
          pos = (uint32_t)(j | (p << 5) | (q << 10) | (lo << 15) | (end << 21));
        }
        nrec = queue_push(ws, nrec, amb, tri, pos);
        if (nrec >= 32) {
          sat_exact(d, ws, sat, kz, xy, 32);
          nrec = queue_shift(ws, nrec);
        }
      }
      __syncwarp();
    }
    if (nrec) sat_exact(d, ws, sat, kz, xy, nrec);
    nrec = 0;
  }
  // the masks out
  uint32_t *out = sat_words(bd, d, ua, W);
#pragma unroll 1
  for (int w = lane; w < m * W; w += 32) {
    if (parts == 1) out[w] = sat[w];
    else if (sat[w]) atomicOr(out + w, sat[w]);
  }
  __syncwarp();
  }  // next item
}

// k_level2c_fill: the inside fill, and the Level2 states from it and the SAT masks.
// ST: the stencil fill (ClassifyInOut2xLevel2) instead of the ray fill.
// HOST: the states go to host memory (write_chunk, write_host_bytes).
template <bool ST, bool HOST>
__global__ void __launch_bounds__(kWarps * 32, 6) k_level2c_fill(
    BatchDev bd, const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals,
    const uint32_t *__restrict__ useg, const Item *__restrict__ items,
    const uint32_t *__restrict__ nitems, int per_warp, int slab, const uint32_t *__restrict__ ilist,
    const uint32_t *__restrict__ ioff) {
  extern __shared__ __align__(16) uint32_t sm[];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t *const scratch = sm + (size_t)warp * per_warp;
  WarpScratch &ws = *reinterpret_cast<WarpScratch *>(scratch);  // (ray fill)
  StScratch &ss = *reinterpret_cast<StScratch *>(scratch);      // (stencil fill)
  uint32_t *const stage = ST ? scratch : ws.sol;
  int *const kz = ST ? reinterpret_cast<int *>(&ss + 1) : reinterpret_cast<int *>(&ws + 1);
  uint32_t *const par = reinterpret_cast<uint32_t *>(kz + 32);
  Item it;
  uint32_t part;
  while (next_item(bd.queue + 1 + slab, items, nitems, slab, ilist, ioff, 1u, it, part)) {
  const uint32_t ua = it.ua;
  const MeshDesc &d = bd.md[it.m_mesh >> 7];
  const GridDev &g = d.g;
  const float4 *__restrict__ ptri = d.ptri;
  const float4 *__restrict__ fbox = d.fbox;
  const int CH = d.ch;
  const int n2x = g.n2[0], n2y = g.n2[1], n2z = g.n2[2];
  const int cells = n2x * n2y * n2z;
  const int W = (cells + 31) >> 5;
  const int ncol2 = n2x * n2y;
  const int FW = (ncol2 + 31) >> 5;
  uint32_t *ft = par + CH * W;
  // stencil fill: per voxel, (2 n2x * 2 n2y) sample columns of n2z slice toggle bits; per voxel
  // one bit per sample toggling every slice of that voxel and of the voxels above it
  uint32_t *stg = ft + CH * FW;
  const int SWd = 4 * W;
  const int FWS = (4 * ncol2 + 31) >> 5;
  uint32_t *sft = stg + CH * SWd, *sftacc = sft + CH * FWS;

  const uint32_t ucol_end = it.col_end;
  const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const uint32_t col = it.col;
  const int m = (int)(it.m_mesh & 63u);
  const int ci = (int)(col % (uint32_t)nx), cj = (int)(col / (uint32_t)nx);
  // clear the masks of the chunk's m voxels only (the arrays are sized for CH voxels)
#pragma unroll 1
  for (int w = lane; w < m * W; w += 32) par[w] = 0;
#pragma unroll 1
  for (int w = lane; w < m * FW; w += 32) ft[w] = 0;
  uint32_t udraw = ua;  // stencil fill: the first voxel whose triangles are drawn
  if (ST) {
#pragma unroll 1
    for (int w = lane; w < m * SWd; w += 32) stg[w] = 0;
#pragma unroll 1
    for (int w = lane; w < m * FWS; w += 32) sft[w] = 0;
    // the coverage parity of the column's triangles recorded only below the chunk (none below a
    // column's first voxel; the prefix pass writes the masks of the later chunk starts), or none, and
    // those triangles drawn too
    const uint32_t *const pre = bd.stp + (size_t)ua * bd.stp_words;
    const uint32_t head = (it.m_mesh >> 6) & 1u ? ua + 1u : pre[bd.stp_words - 1];
    if (head) udraw = head - 1u;
#pragma unroll 1
    for (int w = lane; w < FWS; w += 32) sftacc[w] = head ? 0u : pre[w];
  }
  if ((int)lane < m) kz[lane] = (int)(keys[useg[ua + lane]] - col * (uint32_t)nz);
  __syncwarp();
  const float *ox = g.o2[0] + (size_t)ci * n2x, *oy = g.o2[1] + (size_t)cj * n2y;
  uint32_t *const satm = sat_words(bd, d, ua, W);

  uint64_t nun = 0;
  if (ST) {
    // ---------------- stencil fill: the triangles recorded anywhere in the Level1 column (the
    // voxel strip of CreateVoxelStripDisplayLists, src/Object.cpp:605-633: each once, at its
    // topmost record) are drawn into 2 n2x x 2 n2y samples over the Level1 voxel's x/y extent
    // (glOrtho over [i*gridSizeX + bBoxMin, + gridSizeX], :1241-1266).  Slice s of voxel k clips
    // at the Level2 ray-origin height o2z[k][s] (minZ + (s + 0.5)*gridSizeZ2, :1297), so a
    // covered sample at height zs counts in every slice from the first with o2z >= zs: one
    // toggle bit there, expanded by a prefix XOR below.
    // triangles recorded from the chunk's first voxel up (those below are in the prefix, where there is one)
    const uint32_t g0 = useg[udraw], g1 = useg[ucol_end];
    const int SW = 2 * n2x, SH = 2 * n2y;
    const float lx = fa(fm((float)ci, g.g[0]), g.bmin[0]), hx = fa(lx, g.g[0]);
    const float ly = fa(fm((float)cj, g.g[1]), g.bmin[1]), hy = fa(ly, g.g[1]);
    const float *ozt = g.o2[2];
    // with increasing clip heights, the chunk's highest one is its top voxel's last slice
    const float top_clip = __ldg(ozt + (size_t)kz[m - 1] * n2z + n2z - 1);
    const int kz0 = kz[0], span = (kz[m - 1] - kz0 + 1) * n2z;  // clip heights from the chunk's first voxel up
    const float *clip = ozt + (size_t)kz0 * n2z;
    const float clip0 = __ldg(clip), inv_n2z = rcp_fast((float)n2z);
    // bit i: layer kz0 + i belongs to the chunk
    const uint32_t layers = __reduce_or_sync(FULL, ((int)lane < m && kz[lane] - kz0 < 32) ? 1u << (kz[lane] - kz0) : 0u);
#pragma unroll 1
    for (uint32_t b0 = g0; b0 < g1; b0 += 32) {
      const uint32_t e = b0 + lane;
      const uint32_t vv = e < g1 ? vals[e] : 0u;
      StTri st = {};
      bool has = false;
      if (vv & 0x80000000u) {
        const uint32_t t = vv & 0x7fffffffu;
        const float4 a0 = __ldg(ptri + 3 * (size_t)t), a1 = __ldg(ptri + 3 * (size_t)t + 1),
                     a2 = __ldg(ptri + 3 * (size_t)t + 2);
        const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
        // The interpolated height of a covered sample is a convex combination of the vertex
        // heights up to 7 eps max|z| of rounding, so a triangle whose lowest vertex lies more
        // than 16 eps max|z| above the chunk's highest clip height counts in none of its slices.
        const float zmn = fminf(V[2], fminf(V[5], V[8]));
        const float zmag = fmaxf(fabsf(V[2]), fmaxf(fabsf(V[5]), fabsf(V[8])));
        const bool above = g.oz_monotone && zmn - 16.f * EPS24 * zmag > top_clip;
        has = !above && st_setup(V, lx, hx, ly, hy, SW, SH, st);
      }
      const StBatch batch(ss.r, has, st);
      __syncwarp();
#pragma unroll 1
      for (uint32_t w0 = 0; w0 < batch.total; w0 += 32) {
        const StRec &r = batch.owner(ss.r, w0);
        int sx, sy;
        float zs;
        if (!(w0 + lane < batch.total && st_sample(r, w0 + lane, sx, sy, zs))) continue;
        const int sidx = sy * SW + sx, sbit = sidx * n2z;
        if (g.oz_monotone) {
          // clip heights increase through the chunk: the lowest voxel whose top clip keeps zs
          // gets its toggle at the first such slice, and every voxel above it keeps zs in all
          // slices (one bit in its sample-toggle row, accumulated upwards).  The first height from
          // the chunk's lowest that keeps zs, estimated and corrected by the table:
          const float f = (zs - clip0) * g.inv_g2[2];
          int i = !(f > 0.f) ? 0 : f >= (float)span ? span : __float2int_ru(f);
#pragma unroll 1
          while (i > 0 && __ldg(clip + i - 1) >= zs) --i;
#pragma unroll 1
          while (i < span && !(__ldg(clip + i) >= zs)) ++i;
          if (i < span) {
            const int kq = __float2int_rz(((float)i + 0.5f) * inv_n2z);
            int jv;  // the lowest voxel in or above that layer
            if (kq < 32) {
              jv = __popc(layers & ((1u << kq) - 1u));
            } else {
              jv = 0;
#pragma unroll 1
              while (kz[jv] - kz0 < kq) ++jv;
            }
            const int b = sbit + (kz[jv] - kz0 == kq ? i - kq * n2z : 0);
            atomicXor(&stg[jv * SWd + (b >> 5)], 1u << (b & 31));
            if (jv + 1 < m) atomicXor(&sft[(jv + 1) * FWS + (sidx >> 5)], 1u << (sidx & 31));
          }
        } else {
#pragma unroll 1
          for (int jv = m - 1; jv >= 0; --jv) {
            const int s0 = st_first_slice(ozt + (size_t)kz[jv] * n2z, n2z, zs);
            if (s0 < n2z) {
              const int b = sbit + s0;
              atomicXor(&stg[jv * SWd + (b >> 5)], 1u << (b & 31));
            }
          }
        }
      }
      __syncwarp();
    }
    // a cell is inside when at least 3 of its 4 samples are odd (ClassifyInOut2xLevel2,
    // :1383-1401): parity per slice = prefix XOR of the sample column's toggles
    const uint32_t zmask = n2z >= 32 ? 0xffffffffu : ((1u << n2z) - 1u);
#pragma unroll 1
    for (int jv = 0; jv < m; ++jv) {
      // samples toggled in every slice of this voxel: the XOR of the rows of it and below
#pragma unroll 1
      for (int w = lane; w < FWS; w += 32) sftacc[w] ^= sft[jv * FWS + w];
      __syncwarp();
      const uint32_t *sj = stg + jv * SWd;
#pragma unroll 1
      for (int pq = lane; pq < ncol2; pq += 32) {
        const int q = pq / n2x, p = pq - q * n2x;
        uint32_t x[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const int sidx = (2 * q + (a >> 1)) * SW + 2 * p + (a & 1);
          uint32_t y = column_bits(sj, sidx * n2z, n2z);
          y ^= y << 1; y ^= y << 2; y ^= y << 4; y ^= y << 8; y ^= y << 16;
          if ((sftacc[sidx >> 5] >> (sidx & 31)) & 1u) y = ~y;
          x[a] = y;
        }
        const uint32_t in = ((x[0] & x[1] & (x[2] | x[3])) | (x[2] & x[3] & (x[0] | x[1]))) & zmask;
        if (in) or_column(par + jv * W, pq, n2z, in);
      }
    }
    __syncwarp();
  } else {
  // ---------------- fill: the sub-columns whose rays meet each triangle, for the whole chunk
  const float gx = g.g2[0], gy = g.g2[1];
  uint32_t nrec = 0;
  const uint32_t f0 = useg[ua], f1 = useg[ucol_end];
  const float *ozt = g.o2[2];
  const int kz0 = kz[0];
  const float ozb = __ldg(ozt + (size_t)kz0 * n2z), ozl = __ldg(ozt + (size_t)kz[m - 1] * n2z + n2z - 1);
  const float ox0 = __ldg(ox), oy0 = __ldg(oy), ox1 = __ldg(ox + n2x - 1), oy1 = __ldg(oy + n2y - 1);
  // distance of the origin tables from their affine form: within a voxel two roundings; over the
  // chunk's heights the voxels' own corners (a float product and sum) too
  const float tox = 2.02f * EPS24 * fmaxf(fabsf(ox0), fabsf(ox1));
  const float toy = 2.02f * EPS24 * fmaxf(fabsf(oy0), fabsf(oy1));
  const float toz = EPS24 * (6.1f * fmaxf(fabsf(ozb), fabsf(ozl)) + 4.1f * fabsf(g.bmin[2]));
  const float mx = ff(tox, g.inv_g2[0], kIdx), my = ff(toy, g.inv_g2[1], kIdx);
  const int span = (kz[m - 1] - kz0 + 1) * n2z;  // ray origins from the chunk's first voxel to its last
  const float inv_n2z = rcp_fast((float)n2z);
  // bit i: layer kz0 + i belongs to the chunk
  const uint32_t layers = __reduce_or_sync(FULL, ((int)lane < m && kz[lane] - kz0 < 32) ? 1u << (kz[lane] - kz0) : 0u);
  const bool near = kz[m - 1] - kz0 < 32;
  uint32_t nuni = 0;  // queued triangles (utri, ujm)
#pragma unroll 1
  for (uint32_t b0 = f0; b0 < f1; b0 += 32) {
    // ---- the next entries' triangles whose rays may meet the chunk: about a third of the entries, so
    // they are queued and taken 32 at a time
    {
      const uint32_t e = b0 + lane;
      const uint32_t vv = e < f1 ? vals[e] : 0u;
      bool keep = false;
      int jm = 0;
      if (vv & 0x80000000u) {
        const int dz = (int)(keys[e] - col * (uint32_t)nz) - kz0;  // layers above the chunk's first
        if (dz >= 0) {
          if (dz < 31) jm = __popc(layers & ((2u << dz) - 1u));
          else if (near) jm = m;
          else
#pragma unroll 1
            while (jm < m && kz[jm] - kz0 <= dz) ++jm;
        }
        nun += (uint64_t)jm;
        if (jm > 0) {
          const float4 fb = __ldg(fbox + (vv & 0x7fffffffu));
          keep = fb.x <= ox1 && fb.z >= ox0 - tox && fb.y <= oy1 && fb.w >= oy0 - toy && fb.x <= fb.z;
        }
      }
      const uint32_t bal = __ballot_sync(FULL, keep);
      if (keep) {
        const uint32_t k = nuni + __popc(bal & ((1u << lane) - 1u));
        ws.utri[k] = vv & 0x7fffffffu;
        ws.ujm[k] = (uint8_t)jm;
      }
      nuni += (uint32_t)__popc(bal);
      __syncwarp();
    }
#pragma unroll 1
    while (nuni >= 32 || (nuni > 0 && b0 + 32 >= f1)) {
    uint32_t nsolve = 0, ncol = 0;
    int p0 = 0, p1 = 0, nq = 0;
    float ux = 0.f, uy = 0.f, vx = 0.f, vy = 0.f, wx = 0.f, wy = 0.f, dl = 0.f;
    bool direct = false;
    if (lane < nuni) {
      const uint32_t t = ws.utri[lane];
      const int jm = ws.ujm[lane];
      const float4 fb = __ldg(fbox + t);
      {
        // sub-columns whose origins can lie in the box (all of them where the spacing's inverse overflows)
        p0 = max(__float2int_ru((fb.x - ox0) * g.inv_g2[0] - mx), 0);
        p1 = __float2int_rd(fminf((fb.z - ox0) * g.inv_g2[0] + mx, (float)(n2x - 1)));
        const int q0 = max(__float2int_ru((fb.y - oy0) * g.inv_g2[1] - my), 0);
        const int q1 = __float2int_rd(fminf((fb.w - oy0) * g.inv_g2[1] + my, (float)(n2y - 1)));
        if (p0 <= p1 && q0 <= q1) {
          const int np = p1 - p0 + 1;
          nq = q1 - q0 + 1;
          const float4 a0 = __ldg(ptri + 3 * (size_t)t), a1 = __ldg(ptri + 3 * (size_t)t + 1),
                       a2 = __ldg(ptri + 3 * (size_t)t + 2);
          const float o0 = __ldg(ox + p0), o1 = __ldg(oy + q0);
          ux = a0.x - o0, uy = a0.y - o1, vx = a1.x - o0, vy = a1.y - o1, wx = a2.x - o0, wy = a2.y - o1;
          // Tx = ox - v1x and so on, over the triangle's sub-columns: at most atx, aty
          const float atx = fmaxf(fabsf(ux), fmaxf(fabsf(vx), fabsf(wx))) + (float)(np - 1) * gx;
          const float aty = fmaxf(fabsf(uy), fmaxf(fabsf(vy), fabsf(wy))) + (float)(nq - 1) * gy;
          const float R = 1.0001f * fmaxf(fmaxf(atx, fmaxf(ux, fmaxf(vx, wx)) - fminf(ux, fminf(vx, wx))),
                                          fmaxf(aty, fmaxf(uy, fmaxf(vy, wy)) - fminf(uy, fminf(vy, wy))));
          // In units of eps R^2 the float u, v and u + v (times det) are off by less than 48 and
          // solve_rows' sides by less than 42: 90, 96 with the slope's.  An unbounded box marks an
          // ill-conditioned x/y projection, which has no bound on t: exact tests only.
          direct = !g.oz_monotone || isinf(fb.x) || isinf(fb.z) || !(R > 1e-9f && R < 1e9f) || isinf(g.inv_g2[2]);
          ncol = (uint32_t)(np * nq);
          if (!direct) {
            nsolve = (uint32_t)nq;
            // The plane's height over an origin is affine in (p, q): X = its height above the
            // chunk's first origin, less 1e-6, in Level2 cells; the origins r < X are hit.  The
            // float t of an origin differs from the exact t* by at most 8.2 eps M1 / |det| with
            // M1 growing by at most 0.26 of |t*| away from the crossing (the box is bounded:
            // rel <= 1/8), so it decides as t* does outside 1.35 (8.2 eps M0 / |det| + 1e-6)
            // of the crossing, M0 being M1 at the triangle's own heights; X itself is off by
            // less than 20 eps M0 / |det| and the roundings of the index arithmetic.
            const float e1x = vx - ux, e1y = vy - uy, e1z = a1.z - a0.z, e2x = wx - ux, e2y = wy - uy, e2z = a2.z - a0.z;
            const float Nx = e1y * e2z - e1z * e2y, Ny = e1z * e2x - e1x * e2z, Nz = e1x * e2y - e1y * e2x;
            const float rn = rcp_fast(Nz), igz = g.inv_g2[2];
            const float zt2 = 2.f * fmaxf(fabsf(e1z), fmaxf(fabsf(e2z), fabsf(e2z - e1z)));
            const float M0 = fabsf(e2x) * (aty * fabsf(e1z) + zt2 * fabsf(e1y)) +
                             fabsf(e2y) * (zt2 * fabsf(e1x) + atx * fabsf(e1z)) +
                             fabsf(e2z) * (atx * fabsf(e1y) + aty * fabsf(e1x));
            const float Kx = -(Nx * rn) * igz, Ky = -(Ny * rn) * igz;  // per unit of x, y
            const float w = igz * (EPS24 * (40.f * M0 * fabsf(rn) + 8.f * zt2) + toz + 0.35f * g.thr) +
                            fabsf(Kx) * tox + fabsf(Ky) * toy + 8.f * EPS24 * (float)span + kIdx;
            dl = 104.f * EPS24 * R * R;
            ws.xa[lane] = make_float4(((a0.z - ozb) - g.thr) * igz - Kx * ux - Ky * uy, Kx * gx, Ky * gy, w);
          }
          ws.me[lane] = make_uint4(t, (uint32_t)(jm | (direct ? 256 : 0) | (p0 << 16) | (q0 << 24)), 0u, 0u);
        }
      }
    }
    const uint32_t is = warp_incl_scan(nsolve);
    // triangles of this batch: 32 (or the queue's last), fewer where their rows or sub-columns would
    // not fit
    uint32_t taken = (uint32_t)__popc(__ballot_sync(FULL, lane < nuni && is <= (uint32_t)kSol));
    if (lane >= taken) ncol = 0;
    if (ncol && nsolve)
      ncol = solve_rows(ws.sol + (is - nsolve), nq, ux, vx, wx, uy, vy, wy, 0.f, 0.f, gx, gy, dl, 1.1f * tox,
                        1.1f * toy, p0, (uint32_t)p0, (uint32_t)(n2x | ((p1 + 1) << 16)), 0, 64);
    const uint32_t ic = warp_incl_scan(ncol);
    taken = (uint32_t)__popc(__ballot_sync(FULL, lane < taken && ic <= (uint32_t)kCols));
    if (ncol && lane < taken)
      list_columns(ws.cols + (ic - ncol), nsolve ? ws.sol + (is - nsolve) : nullptr, (int)lane, p0, p1 - p0 + 1, 0, nq);
    const uint32_t C = __shfl_sync(FULL, ic, (int)taken - 1);
    __syncwarp();
    {
#pragma unroll 1
      for (uint32_t c0 = 0; c0 < C; c0 += 32) {
        const uint32_t c = c0 + lane;
        bool amb = false;
        uint32_t tri = 0, pos = 0;
        if (c < C) {
          const uint32_t en = ws.cols[c];
          const int tl = (int)(en & 31u), dq = (int)((en >> 5) & 31u), dp = (int)((en >> 10) & 31u);
          const uint4 me = ws.me[tl];
          const int p = (int)((me.y >> 16) & 255u) + dp, q = (int)(me.y >> 24) + dq;
          const int jm = (int)(me.y & 255u);
          amb = !(en & 0x8000u);
          // Triangles that no row is solved for list every sub-column of their box, most of which the ray
          // misses: those stay off the queue, whose lanes then work on heights together (262k-triangle
          // torus at 128^3 / 8^3, coordinates around 10000, where neighbouring origins can round to one
          // height: fill 2059 -> 480 us).
          if (me.y & 256u) {
            amb = ray_passes(d, me.x, ci, cj, p, q);
          } else if (!amb) {
            const float4 xa = ws.xa[tl];
            const float x = ff((float)dp, xa.y, ff((float)dq, xa.z, xa.x));
            const int N = min(max(__float2int_ru(x - xa.w), 0), span);
            amb = N != min(max(__float2int_ru(x + xa.w), 0), span);
            if (!amb && N > 0) {
              const int pq = q * n2x + p;
              const int kq = __float2int_rz(((float)N + 0.5f) * inv_n2z), rem = N - kq * n2z;
              int below;  // voxels of the chunk under layer kz0 + kq
              bool here;  // ... and whether that layer belongs to it
              if (kq < 32) {
                below = __popc(layers & ((1u << kq) - 1u));
                here = (layers >> kq) & 1u;
              } else if (near) {
                below = m;
                here = false;
              } else {
                below = 0;
#pragma unroll 1
                while (below < m && kz[below] < kz0 + kq) ++below;
                here = below < m && kz[below] == kz0 + kq;
              }
              const int nf = min(below, jm);
              if (nf > 0) atomicXor(&ft[(nf - 1) * FW + (pq >> 5)], 1u << (pq & 31));
              if (here && rem > 0 && below < jm) xor_column(par + below * W, pq, n2z, (1u << rem) - 1u);
            }
          }
          tri = me.x;
          pos = (uint32_t)(jm | (p << 6) | (q << 11));
        }
        nrec = queue_push(ws, nrec, amb, tri, pos);
        if (nrec >= 32) {
          fill_exact(d, ws, par, ft, kz, m, ci, cj, 32);
          nrec = queue_shift(ws, nrec);
        }
      }
      __syncwarp();
    }
    // the queue's rest to its front
    {
      const uint32_t k = lane + taken, k2 = k + 32;
      const uint32_t t0 = k < nuni ? ws.utri[k] : 0u, t1 = k2 < nuni ? ws.utri[k2] : 0u;
      const uint8_t j0 = k < nuni ? ws.ujm[k] : 0, j1 = k2 < nuni ? ws.ujm[k2] : 0;
      __syncwarp();
      if (k < nuni) { ws.utri[lane] = t0; ws.ujm[lane] = j0; }
      if (k2 < nuni) { ws.utri[lane + 32] = t1; ws.ujm[lane + 32] = j1; }
      nuni -= taken;
      __syncwarp();
    }
    }
  }
  if (nrec) fill_exact(d, ws, par, ft, kz, m, ci, cj, nrec);
  __syncwarp();

  }

  // ---------------- output.  The full-hit toggles accumulate downwards first.
#pragma unroll 1
  for (int w = lane; w < FW; w += 32)
#pragma unroll 1
    for (int jv = m - 2; jv >= 0; --jv) ft[jv * FW + w] ^= ft[(jv + 1) * FW + w];
  __syncwarp();
  unsigned long long nin = 0, nbd = 0;
  const uint32_t zmask_all = n2z >= 32 ? 0xffffffffu : ((1u << n2z) - 1u);
  // packed codes for the host: the voxels of this launch's slab below BatchDev::pk_end (the host
  // enables it only where the 16-byte layout below applies)
  const uint32_t pkend = d.l2codes ? bd.pk_end[slab] : 0u;
  const uint32_t vown = (int)lane < m ? (uint32_t)d.prefix[((int64_t)kz[lane] * ny + cj) * nx + ci] : 0u;
  if ((n2z == 8 || n2z == 16) && (ncol2 & 15) == 0 && (reinterpret_cast<uintptr_t>(d.l2) & 15) == 0) {
    if (n2z == 8) write_chunk<8, HOST>(d.l2, d.l2codes, pkend, vown, satm, par, ft, m, ncol2, stage, nbd, nin);
    else write_chunk<16, HOST>(d.l2, d.l2codes, pkend, vown, satm, par, ft, m, ncol2, stage, nbd, nin);
    __syncwarp();
  } else if (HOST && cells >= kHostBytes) {
    write_host_bytes(d.l2, vown, satm, par, ft, m, ncol2, n2z, nbd, nin);
    __syncwarp();
  } else {
    // One lane per sub-column of the chunk: its n2z SAT and parity bits are read once and written
    // as n2z bytes at stride n2x*n2y (consecutive lanes write consecutive bytes of each z layer).
    uint32_t nb = 0, ni = 0;
#pragma unroll 1
    for (int i0 = 0; i0 < m * ncol2; i0 += 32) {
      const int i = i0 + (int)lane;
      const bool live = i < m * ncol2;
      const int jv = live ? i / ncol2 : 0, pq = i - jv * ncol2;
      const uint32_t vidx = __shfl_sync(FULL, vown, jv);
      if (live) {
        const uint32_t sb = column_bits(satm + jv * W, pq * n2z, n2z) & zmask_all;
        uint32_t pb = column_bits(par + jv * W, pq * n2z, n2z);
        if ((ft[jv * FW + (pq >> 5)] >> (pq & 31)) & 1u) pb = ~pb;
        const uint32_t ib = pb & ~sb & zmask_all;
        nb += (unsigned)__popc(sb);
        ni += (unsigned)__popc(ib);
        uint8_t *o = d.l2 + (size_t)vidx * cells + pq;
#pragma unroll 1
        for (int r = 0; r < n2z; ++r)
          __stcs(reinterpret_cast<char *>(o + (size_t)r * ncol2), (char)(((sb >> r) & 1u) * 254u + ((ib >> r) & 1u) * 127u));
      }
    }
    nbd += nb;
    nin += ni;
  }
  nin = warp_sum(nin);
  nbd = warp_sum(nbd);
  nun = warp_sum(nun);
  if (lane == 0) {
    if (nin) atomicAdd(&d.stats->l2_inside, nin);
    if (nbd) atomicAdd(&d.stats->l2_boundary, nbd);
    if (nun) atomicAdd(&d.stats->ray2, (unsigned long long)nun * (unsigned long long)cells);
  }
  __syncwarp();
  }  // next item
}

}  // namespace

int level2_chunk(const GridDev &g, int cap) {
  const int cells = g.n2[0] * g.n2[1] * g.n2[2];
  const int W = (cells + 31) >> 5;
  return std::max(1, std::min(std::min(32, std::max(cap, 1)), kMaskWords / W));
}

// Shared-memory words one warp of the two Level2 kernels needs for a mesh with this grid.
Level2Words level2_warp_words(const GridDev &g, int cap, bool stencil) {
  const int cells = g.n2[0] * g.n2[1] * g.n2[2];
  const int W = (cells + 31) >> 5;
  const int FW = (g.n2[0] * g.n2[1] + 31) >> 5;
  const int CH = level2_chunk(g, cap);
  const int FWS = (4 * g.n2[0] * g.n2[1] + 31) >> 5;
  const int base = (int)(sizeof(WarpScratch) / 4) + 32;
  const int base_fill = (int)((stencil ? sizeof(StScratch) : sizeof(WarpScratch)) / 4) + 32;
  auto al = [](int words) { return (words + 3) & ~3; };  // a warp's region starts 16-byte aligned
  return {al(base + 32 + std::max(CH, sat_run_cap(g)) * W), al(base_fill + CH * W + CH * FW + (stencil ? 4 * CH * W + CH * FWS + FWS : 0))};
}

int level2_parts(int64_t B, int num_sms) {
  const int64_t warps = (int64_t)num_sms * 24;
  return (int)std::max<int64_t>(1, std::min<int64_t>(64, warps / std::max<int64_t>(4 * B, 1)));
}
int level2_few_chunk(int ch, int64_t B, int num_sms) {
  const int64_t warps = (int64_t)num_sms * 24;
  return (int)std::max<int64_t>(1, std::min<int64_t>(ch, ch * B / (4 * warps)));
}

size_t level2_smem_bytes(int warp_words) { return (size_t)warp_words * 4 * kWarps; }

int64_t level2_temp_words(int64_t B) { return 10 * B + 16 + 2 * (kSlabsMax + 4); }

// Builds the chunk items from the sorted pair lists and runs the persistent Level2 kernel.
void launch_level2(const BatchDev &bd, const uint32_t *keys, const uint32_t *vals,
                   const uint32_t *useg, const uint32_t *kpre, int64_t B, uint32_t *tmp, int64_t smask_words, Level2Words words, int num_sms,
                   cudaStream_t s, const std::function<void()> &before_kernel, int zslab,
                   int nslab, const std::function<void(int, cudaStream_t)> &after_slab, int slab_nz,
                   const SlabStreams *aux) {
  if (B <= 0) return;
  // (tmp is 256-byte aligned: the items come first)
  Item *items = reinterpret_cast<Item *>(tmp);
  Item *runs = items + B;
  uint32_t *iflag = tmp + 8 * B, *slabcnt = iflag + B, *ioff = slabcnt + (kSlabsMax + 4),
           *ilist = ioff + (kSlabsMax + 4), *nitems = bd.queue + kQueueItems;
  if (nslab <= 1) zslab = 0;
  if (zslab > 0) runs = nullptr;
  const unsigned nb = (unsigned)((B + 255) / 256);
  const bool stp = bd.fill == GPV_FILL_STENCIL && bd.stp;
  // (one-graph calls: B is the capacity, the kernels read the device count)
  k_items<<<(unsigned)((B + kItemThreads - 1) / kItemThreads), kItemThreads, 0, s>>>(
      bd, kpre, keys, useg, B, zslab, stp ? iflag : nullptr, items, runs, 2 * 24 * num_sms, nitems);
  count_launch(1);
  if (stp) {
    const unsigned nbp = (unsigned)((B + kPrefixWarps - 1) / kPrefixWarps);  // items <= B
    k_stencil_segment<<<nbp, kPrefixWarps * 32, 0, s>>>(bd, keys, vals, useg, items, nitems);
    k_stencil_scan<<<nbp, kPrefixWarps * 32, 0, s>>>(bd, iflag, items, nitems);
    count_launch(2);
  }
  const bool st = bd.fill == GPV_FILL_STENCIL;
  static OncePerDevice once[5];
  // a kernel's persistent grid (one-graph calls: B is a capacity, the queue ends the work)
  auto grid_of = [&](auto *k, int kv, size_t smem, int64_t jobs) {
    allow_shared_memory(once[kv], k, 200 * 1024);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kWarps * 32, smem);
    const int64_t full = (int64_t)num_sms * std::max(per_sm, 1);
    return (unsigned)(bd.plan ? full : std::min<int64_t>((jobs + kWarps - 1) / kWarps, full));
  };
  // Few voxels (a coarse grid): several warps share an item's pairs, their masks OR-ed into cleared
  // words.  42 voxels of 7k triangles: the SAT kernel 424 -> 17 us.
  const int parts = level2_parts(B, num_sms);
  if (parts > 1) cudaMemsetAsync(bd.smask, 0, (size_t)smask_words * sizeof(uint32_t), s);
  const bool host = bd.l2_host;
  auto *const fill = st ? (host ? k_level2c_fill<true, true> : k_level2c_fill<true, false>)
                        : (host ? k_level2c_fill<false, true> : k_level2c_fill<false, false>);
  const size_t smem_sat = level2_smem_bytes(words.sat), smem_fill = level2_smem_bytes(words.fill);
  const unsigned grid_sat = grid_of(k_level2c_sat, 0, smem_sat, B * parts);
  const unsigned grid_fill = grid_of(fill, 1 + 2 * st + host, smem_fill, B);
  const int nz = slab_nz;
  if (zslab > 0) {
    // single mesh: order the items by slab so that each launch takes only its own
    cudaMemsetAsync(slabcnt, 0, (kSlabsMax + 4) * sizeof(uint32_t), s);
    k_item_slab_count<<<nb, 256, 0, s>>>(items, nitems, keys, useg, nz, zslab, slabcnt);
    k_item_slab_offsets<<<1, 32, 0, s>>>(slabcnt, nslab, ioff);
    k_item_slab_place<<<nb, 256, 0, s>>>(items, nitems, keys, useg, nz, zslab, slabcnt, ilist);
    count_launch(3);
  }
  if (before_kernel) before_kernel();
  // one launch of each kernel, or one per z slab over that slab's items; the slabs' SAT kernels run on
  // one stream and their fills, each after its SAT, on another (when given), so that a slab's SAT
  // overlaps the writes of the one before, and the slabs finish in order (fills of two slabs side by
  // side finished together and left their copies or expansion to the end: 192^3 / 8^3 host to host
  // 1098 against 1076 us)
  const int launches = zslab > 0 ? nslab : 1;
  const bool two = zslab > 0 && launches > 1 && aux;
  if (two) {
    cudaEventRecord(aux->fork, s);
    cudaStreamWaitEvent(aux->st[0], aux->fork, 0);
    cudaStreamWaitEvent(aux->st[1], aux->fork, 0);
  }
  for (int sl = 0; sl < launches; ++sl) {
    const uint32_t *list = zslab > 0 ? ilist : nullptr;
    cudaStream_t ss = two ? aux->st[0] : s, ls = two ? aux->st[1] : s;
    k_level2c_sat<<<grid_sat, kWarps * 32, smem_sat, ss>>>(bd, keys, vals, useg, runs ? runs : items,
                                                          nitems + (runs ? 1 : 0), words.sat, sl, list, ioff,
                                                          parts);
    if (two) {
      cudaEventRecord(aux->join[0], ss);
      cudaStreamWaitEvent(ls, aux->join[0], 0);
    }
    fill<<<grid_fill, kWarps * 32, smem_fill, ls>>>(bd, keys, vals, useg, items, nitems, words.fill, sl,
                                                    list, ioff);
    count_launch(2);
    if (after_slab) after_slab(sl, ls);
  }
  if (two) {
    cudaEventRecord(aux->join[0], aux->st[0]);
    cudaEventRecord(aux->join[1], aux->st[1]);
    cudaStreamWaitEvent(s, aux->join[0], 0);
    cudaStreamWaitEvent(s, aux->join[1], 0);
  }
}

}  // namespace gpv
