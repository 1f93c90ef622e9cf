// gpv_normals.cu -- Level1 and Level2 voxel normals (optional; gpv_set_normals).
//
// Reference semantics (the CPU path):
//   face normal   VectorCrossProduct(v1 - v0, v2 - v0), VectorNormalize (src/Object.cpp:522-526,
//                 includes/FloatVector.h:293-296,333-342), float arithmetic, IEEE sqrt/divide.
//   Level1        for every voxel with recorded triangles: the float sum of their face normals in
//                 list order, divided by the count, normalised (src/Object.cpp:3219-3253);
//                 other voxels 0 (:3151-3152).
//   Level2        every SAT pass of (triangle, sub-cell) adds the face normal and 1 to the cell
//                 (AddPointToVoxel, :2715-2719), triangles in list order; sum / count,
//                 normalised (:2402-2424); cells without a pass 0 (:3309-3310).
// The list order of the CPU path is ascending triangle id (ClassifyTessellation records the
// triangles in file order, :2267-2340); with normals on, each voxel's triangles are put in id order too
// (by k_seg_sort and k_seg_sort_long, or, with long lists on average, by a radix sort of all pairs by id
// and voxel), so every float sum runs in the reference's order.
//
// Outputs per mode: GPV_NORMALS_BYTES writes the .raw encoding uint8(n * float(256/3) + 127)
// (src/Object.cpp:2940-2941, :3033-3035), three bytes per voxel / cell; GPV_NORMALS_FLOAT writes
// the three floats.
#include <algorithm>

#include "gpv_internal.h"
#include "gpv_rows.cuh"

namespace gpv {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kNWarps = 4;
constexpr int kNTileCells = 512;  // Level2 cells accumulated at once per warp

__device__ __forceinline__ void normalize3(float &x, float &y, float &z) {
  const float mag = __fsqrt_rn(fa(fa(fm(x, x), fm(y, y)), fm(z, z)));
  if (mag != 0.f) {
    x = __fdiv_rn(x, mag);
    y = __fdiv_rn(y, mag);
    z = __fdiv_rn(z, mag);
  }
}

__device__ __forceinline__ void store_normal(void *base, int mode, int64_t idx, float x, float y,
                                             float z) {
  if (mode == GPV_NORMALS_FLOAT) {
    float *o = static_cast<float *>(base) + 3 * idx;
    o[0] = x; o[1] = y; o[2] = z;
  } else {
    const float sc = (float)(256.0 / 3.0);
    uint8_t *o = static_cast<uint8_t *>(base) + 3 * idx;
    o[0] = (uint8_t)__float2int_rz(fa(fm(x, sc), 127.f));
    o[1] = (uint8_t)__float2int_rz(fa(fm(y, sc), 127.f));
    o[2] = (uint8_t)__float2int_rz(fa(fm(z, sc), 127.f));
  }
}

template <int64_t MeshDesc::*F>
__device__ __forceinline__ int mesh_by(const MeshDesc *md, int nmesh, int64_t idx) {
  int lo = 0, hi = nmesh - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (md[mid].*F <= idx) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(256) k_face_normals(BatchDev bd) {
  const int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= bd.total_tris) return;
  const MeshDesc &d = bd.md[mesh_by<&MeshDesc::tri_base>(bd.md, bd.nmesh, gi)];
  const int64_t t = gi - d.tri_base;
  const float *v = d.tris + 9 * t;
  const float a0 = fs(v[3], v[0]), a1 = fs(v[4], v[1]), a2 = fs(v[5], v[2]);
  const float b0 = fs(v[6], v[0]), b1 = fs(v[7], v[1]), b2 = fs(v[8], v[2]);
  float x = fs(fm(a1, b2), fm(b1, a2));
  float y = fs(fm(a2, b0), fm(b2, a0));
  float z = fs(fm(a0, b1), fm(b0, a1));
  normalize3(x, y, z);
  d.fnorm[t] = make_float4(x, y, z, 0.f);
}

// One thread per boundary voxel of the sorted meshes: sum in list order, average, normalise.  The
// loads of a list of up to kThreadList triangles run kAhead at a time; longer lists are summed by the
// whole warp, one after the other: a load per lane, the next ones under way, and the additions in
// list order from the lanes.  A warp takes per_warp voxels, 32 or (few voxels) one.  (A dependent load per triangle was the whole cost where a voxel holds
// hundreds: 217 us for 42 voxels of 7k triangles, now 56.)
constexpr int kAhead = 8;
constexpr uint32_t kThreadList = 64;
__global__ void __launch_bounds__(256) k_level1_normals(BatchDev bd, const uint32_t *__restrict__ keys,
                                                        const uint32_t *__restrict__ vals,
                                                        const uint32_t *__restrict__ useg, int64_t U,
                                                        int per_warp) {
  const unsigned lane = threadIdx.x & 31u;
  const int64_t u = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per_warp + lane;
  const bool live = (int)lane < per_warp && u < U;
  const MeshDesc &d = bd.md[mesh_by<&MeshDesc::u_base>(bd.md, bd.nmesh, live ? u : U - 1)];
  const float4 *__restrict__ fnorm = d.fnorm;
  const uint32_t e0 = live ? useg[u] : 0u, e1 = live ? useg[u + 1] : 0u;
  const bool is_long = e1 - e0 > kThreadList;
  float sx = 0.f, sy = 0.f, sz = 0.f;
  if (!is_long)
    for (uint32_t e = e0; e < e1; e += kAhead) {
      float4 f[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) f[k] = __ldg(fnorm + (vals[min(e + k, e1 - 1)] & 0x7fffffffu));
#pragma unroll
      for (int k = 0; k < kAhead; ++k)
        if (e + k < e1) {
          sx = fa(sx, f[k].x);
          sy = fa(sy, f[k].y);
          sz = fa(sz, f[k].z);
        }
    }
  for (uint32_t todo = __ballot_sync(FULL, is_long); todo; todo &= todo - 1u) {
    const int own = __ffs(todo) - 1;
    const uint32_t a = __shfl_sync(FULL, e0, own), b = __shfl_sync(FULL, e1, own);
    const float4 *fn = reinterpret_cast<const float4 *>(__shfl_sync(FULL, (unsigned long long)fnorm, own));
    float x = 0.f, y = 0.f, z = 0.f;
    float4 f = __ldg(fn + (vals[min(a + lane, b - 1)] & 0x7fffffffu));
    for (uint32_t e = a; e < b; e += 32) {
      const float4 cur = f;
      if (e + 32 < b) f = __ldg(fn + (vals[min(e + 32 + lane, b - 1)] & 0x7fffffffu));
      const int n = (int)min(b - e, 32u);
#pragma unroll 4
      for (int k = 0; k < n; ++k) {
        x = fa(x, __shfl_sync(FULL, cur.x, k));
        y = fa(y, __shfl_sync(FULL, cur.y, k));
        z = fa(z, __shfl_sync(FULL, cur.z, k));
      }
    }
    if ((int)lane == own) {
      sx = x;
      sy = y;
      sz = z;
    }
  }
  if (!live) return;
  const float cnt = (float)(e1 - e0);
  float x = __fdiv_rn(sx, cnt), y = __fdiv_rn(sy, cnt), z = __fdiv_rn(sz, cnt);
  normalize3(x, y, z);
  const int nx = d.g.n[0], ny = d.g.n[1], nz = d.g.n[2];
  const uint32_t key = keys[e0];  // column-major: (j*nx + i)*nz + k
  const uint32_t col = key / (uint32_t)nz;
  const int64_t vlin = ((int64_t)(key - col * (uint32_t)nz) * ny + col / (uint32_t)nx) * nx +
                       col % (uint32_t)nx;
  store_normal(d.l1n, bd.normals, vlin, x, y, z);
}

// ---- a voxel's triangles by id ------------------------------------------------------------------
// The counting sort leaves each voxel's triangles in any order; their normals are summed in ascending
// id.  One warp per voxel: up to 32 in registers, up to kSegWarp in its shared memory; longer lists
// are noted for k_seg_sort_long.  (With a few triangles a voxel this replaces the radix sort of all
// pairs by id and voxel: 430k pairs of 53k voxels, sort and lists 202 -> 62 us with the counting sort.)
constexpr int kSegWarp = 512;
constexpr int kSegBlock = 8192;
constexpr uint32_t kIdMask = 0x7fffffffu;

// Bitonic sort by id of n <= N values in shared memory (N a power of two; padded with kIdMask).
template <typename Sync>
__device__ __forceinline__ void bitonic_ids(uint32_t *v, int N, int t, int nt, Sync sync) {
  for (int k = 2; k <= N; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = t; i < N / 2; i += nt) {
        const int lo = 2 * i - (i & (j - 1)), hi = lo + j;
        const uint32_t a = v[lo], b = v[hi];
        if (((a & kIdMask) > (b & kIdMask)) == ((lo & k) == 0)) {
          v[lo] = b;
          v[hi] = a;
        }
      }
      sync();
    }
}

__global__ void __launch_bounds__(kNWarps * 32) k_seg_sort(uint32_t *__restrict__ vals,
                                                           const uint32_t *__restrict__ useg, int64_t U,
                                                           uint32_t *__restrict__ longs) {
  __shared__ uint32_t s_v[kNWarps][kSegWarp];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int64_t u = (int64_t)blockIdx.x * kNWarps + warp;
  if (u >= U) return;
  const uint32_t e0 = useg[u], n = useg[u + 1] - e0;
  if (n <= 1) return;
  if (n <= 32) {
    uint32_t v = lane < n ? vals[e0 + lane] : kIdMask;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const uint32_t o = __shfl_xor_sync(FULL, v, j);
        const bool up = (lane & k) == 0, low = (lane & j) == 0;
        if (((v & kIdMask) > (o & kIdMask)) == (up == low) && (v & kIdMask) != (o & kIdMask)) v = o;
      }
    if (lane < n) vals[e0 + lane] = v;
    return;
  }
  if (n > (uint32_t)kSegWarp) {
    if (lane == 0) longs[1 + atomicAdd(longs, 1u)] = (uint32_t)u;
    return;
  }
  int N = 64;
  while ((uint32_t)N < n) N <<= 1;
  uint32_t *v = s_v[warp];
  for (int i = lane; i < N; i += 32) v[i] = (uint32_t)i < n ? vals[e0 + i] : kIdMask;
  __syncwarp();
  bitonic_ids(v, N, (int)lane, 32, [] { __syncwarp(); });
  for (uint32_t i = lane; i < n; i += 32) vals[e0 + i] = v[i];
}

// The noted lists, a block each.  Up to kSegBlock triangles: the network in shared memory.  Longer ones:
// a voxel's ids are distinct, so they are marked in a bit map of the mesh's triangles, kMapIds at a time,
// and read back in order, through `spare` (as long as the lists).  Sort and lists of 27k short lists and one
// of 9k triangles 83 us, of 30k 123, of 300k 820 (mostly the counting sort's atomics on one voxel); with
// the network in global memory 213, 452 and 11400; the radix sort of all pairs, whose passes do not
// depend on the lists' lengths, 181, 180 and 195.
constexpr int kMapIds = 12 * 1024 * 32;  // ids of a pass: 48 KB of marks and 48 KB of their top flags

__global__ void __launch_bounds__(1024) k_seg_sort_long(const BatchDev bd, uint32_t *__restrict__ vals,
                                                        const uint32_t *__restrict__ useg,
                                                        const uint32_t *__restrict__ longs,
                                                        uint32_t *__restrict__ spare) {
  extern __shared__ uint32_t s_long[];
  __shared__ uint32_t s_warp[33];
  const uint32_t nl = longs[0];
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint32_t l = blockIdx.x; l < nl; l += gridDim.x) {
    const uint32_t u = longs[1 + l], e0 = useg[u], n = useg[u + 1] - e0;
    if (n <= (uint32_t)kSegBlock) {
      int N = 1024;
      while ((uint32_t)N < n) N <<= 1;
      for (int i = tid; i < N; i += 1024) s_long[i] = (uint32_t)i < n ? vals[e0 + i] : kIdMask;
      __syncthreads();
      bitonic_ids(s_long, N, tid, 1024, [] { __syncthreads(); });
      for (uint32_t i = tid; i < n; i += 1024) vals[e0 + i] = s_long[i];
      __syncthreads();
      continue;
    }
    const int64_t T = bd.md[mesh_by<&MeshDesc::u_base>(bd.md, bd.nmesh, (int64_t)u)].T;
    uint32_t done = 0;  // ids placed
    for (int64_t id0 = 0; id0 < T && done < n; id0 += kMapIds) {
      const int ids = (int)min(T - id0, (int64_t)kMapIds), words = (ids + 31) >> 5;
      uint32_t *const mark = s_long, *const top = s_long + kMapIds / 32;
      for (int i = tid; i < words; i += 1024) mark[i] = top[i] = 0u;
      __syncthreads();
      for (uint32_t i = tid; i < n; i += 1024) {
        const uint32_t v = vals[e0 + i];
        const int64_t id = (int64_t)(v & kIdMask) - id0;
        if (id < 0 || id >= ids) continue;
        atomicOr(&mark[id >> 5], 1u << (id & 31));
        if (v >> 31) atomicOr(&top[id >> 5], 1u << (id & 31));
      }
      __syncthreads();
      // each warp takes a run of words, a word a lane: the places of their ids from the counts before them
      const int per = ((words + 31) / 32 + 31) & ~31, w0 = warp * per, w1 = min(w0 + per, words);
      uint32_t cnt = 0;
      for (int i = w0 + lane; i < w1; i += 32) cnt += (uint32_t)__popc(mark[i]);
      cnt = __reduce_add_sync(FULL, cnt);
      if (lane == 0) s_warp[warp] = cnt;
      __syncthreads();
      if (warp == 0) {
        uint32_t inc = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t x = __shfl_up_sync(FULL, inc, o);
          if (lane >= o) inc += x;
        }
        const uint32_t own = s_warp[lane];
        s_warp[lane] = inc - own;
        if (lane == 31) s_warp[32] = inc;
      }
      __syncthreads();
      uint32_t at = e0 + done + s_warp[warp];
      for (int i0 = w0; i0 < w1; i0 += 32) {
        const int i = i0 + lane;
        const uint32_t m = i < w1 ? mark[i] : 0u, f = i < w1 ? top[i] : 0u;
        uint32_t inc = (uint32_t)__popc(m);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t x = __shfl_up_sync(FULL, inc, o);
          if (lane >= o) inc += x;
        }
        uint32_t q = at + inc - (uint32_t)__popc(m);
        for (uint32_t x = m; x; x &= x - 1u, ++q) {
          const int b = __ffs(x) - 1;
          spare[q] = (uint32_t)(id0 + 32 * (int64_t)i + b) | (((f >> b) & 1u) << 31);
        }
        at += __shfl_sync(FULL, inc, 31);
      }
      done += s_warp[32];
      __syncthreads();
    }
    for (uint32_t i = tid; i < done; i += 1024) vals[e0 + i] = spare[e0 + i];
    __syncthreads();
  }
}

// One warp per run of boundary voxels, or (few voxels, large sub-grids) per voxel and tile of at most
// `tile` consecutive cells in output order.  The voxels' triangles come in list order, 32 at a time: a
// lane each solves its rows of cells (gpv_rows.cuh) and lists the sub-columns that can pass the x/y tests;
// then the lanes take a sub-column each, whose cells are the run between the rows' and the plane's
// bounds, with the exact SAT where those leave a cell open.  Each cell's sum is kept in shared memory and
// takes its triangles in list order: lanes that hold the same sub-column add one after the other.
// On 430k pairs of 53k voxels at 8^3 and 7k triangles in 42 voxels at 4^3 this took 263 and 202 us; a
// voxel's triangles solved by as many lanes and then added one triangle at a time 374 and 320; every
// candidate cell of every triangle tested exactly 561 and 1271.  Bound by latency (16 warps per SM, by
// registers and the 14 KB of sums and lists of each) at 60% of the issue slots on the former, by the
// longest list's batches, one after the other, on the latter.
constexpr int kFewCells = 4;  // a triangle whose box meets at most this many cells is tested exactly
constexpr int kNSol = 448;    // solved rows of one batch (a triangle has at most 96)
constexpr int kNCols = 1024;  // its sub-columns (a triangle has at most that many)
constexpr int kNRun = 8;      // voxels of a run, at most

struct __align__(16) NWarp {
  float sum[3 * kNTileCells];  // x, y, z of each cell (the output's layout) and the triangles added,
  float cnt[kNTileCells];      // zero before each voxel
  float4 xa[32], xb[32];       // per-triangle constants
  uint4 me[32];  // triangle id; voxel of the run | kind << 8 | first sub-column << 16 | first row << 24;
                 // its solved rows of y/z | of x/z << 16 (few cells: bit i the exact result of cell i of
                 // its box, x fastest); first layer | end << 8 | columns of its box << 16 | rows << 24
  uint32_t sol[kNSol];
  uint32_t que[64];  // tiles: queued triangles that meet the tile, in list order
  uint32_t seg[kNRun + 4], kz[kNRun], xy[kNRun];
  uint16_t cols[kNCols];
};
static_assert(sizeof(NWarp) % 16 == 0, "layout");

// Sums to normals, and a voxel's (or tile's) tc values out; the sums are cleared.
__device__ __noinline__ void finish_voxel(NWarp &ws, int tc, int mode, void *l2n, int64_t obase) {
  const int lane = (int)(threadIdx.x & 31u);
  // averages of the cells with a triangle (about one in seven), 32 at a time
  uint32_t nhit = 0;  // queued cells, in `que`: its triangles are done
  for (int cb = 0; cb < tc; cb += 32) {
    const int c = cb + lane;
    const bool hit = c < tc && ws.cnt[c] > 0.f;
    const uint32_t bal = __ballot_sync(FULL, hit);
    if (hit) ws.que[nhit + __popc(bal & ((1u << lane) - 1u))] = (uint32_t)c;
    nhit += (uint32_t)__popc(bal);
    __syncwarp();
    const bool last = cb + 32 >= tc;
    while (nhit >= 32 || (last && nhit)) {
      const uint32_t n = min(nhit, 32u);
      if (lane < (int)n) {
        const uint32_t h = ws.que[lane];
        float *v = ws.sum + 3 * h;
        const float w = ws.cnt[h];
        float x = __fdiv_rn(v[0], w), y = __fdiv_rn(v[1], w), z = __fdiv_rn(v[2], w);
        normalize3(x, y, z);
        v[0] = x;
        v[1] = y;
        v[2] = z;
        ws.cnt[h] = 0.f;
      }
      const uint32_t rest = (uint32_t)lane + n < nhit ? ws.que[lane + n] : 0u;
      __syncwarp();
      if ((uint32_t)lane + n < nhit) ws.que[lane] = rest;
      nhit -= n;
      __syncwarp();
    }
  }
  // out, consecutive values by consecutive lanes, four at a time where their places are aligned
  float4 *s4 = reinterpret_cast<float4 *>(ws.sum);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int n = 3 * tc;
  if (mode == GPV_NORMALS_FLOAT) {
    float *o = static_cast<float *>(l2n) + 3 * obase;
    if ((n & 3) == 0 && ((uintptr_t)o & 15u) == 0) {
      for (int i = lane; i < n / 4; i += 32) {
        __stcs(reinterpret_cast<float4 *>(o) + i, s4[i]);
        s4[i] = zero;
      }
    } else {
      for (int i = lane; i < n; i += 32) {
        __stcs(o + i, ws.sum[i]);
        ws.sum[i] = 0.f;
      }
    }
  } else {
    const float sc = (float)(256.0 / 3.0);
    uint8_t *o = static_cast<uint8_t *>(l2n) + 3 * obase;
    auto enc = [&](float v) { return (uint32_t)(uint8_t)__float2int_rz(fa(fm(v, sc), 127.f)); };
    if ((n & 3) == 0 && ((uintptr_t)o & 3u) == 0) {
      for (int i = lane; i < n / 4; i += 32) {
        const float4 v = s4[i];
        reinterpret_cast<uint32_t *>(o)[i] = enc(v.x) | enc(v.y) << 8 | enc(v.z) << 16 | enc(v.w) << 24;
        s4[i] = zero;
      }
    } else {
      for (int i = lane; i < n; i += 32) {
        o[i] = (uint8_t)enc(ws.sum[i]);
        ws.sum[i] = 0.f;
      }
    }
  }
  __syncwarp();
}

// The exact SAT of the cells [lo, end) of a sub-column at (cx, cy).
__device__ __noinline__ uint32_t exact_cells(const float4 *__restrict__ pt, float cx, float cy,
                                             const float *__restrict__ sz, float h0, float h1, float h2, int lo,
                                             int end) {
  const float4 v0 = __ldg(pt), v1 = __ldg(pt + 1), v2 = __ldg(pt + 2);
  const float V[9] = {v0.x, v0.y, v0.z, v1.x, v1.y, v1.z, v2.x, v2.y, v2.z};
  const float h[3] = {h0, h1, h2};
  SatCol sc;
  uint32_t bits = 0;
  if (sat_col(V, cx, cy, h, sc))
    for (int r = lo; r < end; ++r)
      if (sat_z(sc, V, __ldg(sz + r), h)) bits |= 1u << r;
  return bits;
}

__global__ void __launch_bounds__(kNWarps * 32, 4) k_level2_normals(BatchDev bd,
                                                                    const uint32_t *__restrict__ keys,
                                                                    const uint32_t *__restrict__ vals,
                                                                    const uint32_t *__restrict__ useg,
                                                                    int64_t U, int tile, int max_tiles, int run) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int lane = (int)(threadIdx.x & 31u);
  NWarp &ws = reinterpret_cast<NWarp *>(s_raw)[threadIdx.x >> 5];
  for (int i = lane; i < 3 * kNTileCells; i += 32) ws.sum[i] = 0.f;
  for (int i = lane; i < kNTileCells; i += 32) ws.cnt[i] = 0.f;
  __syncwarp();
  // jobs: runs of `run` voxels (one tile), or (voxel, tile) with run = 1
  const int64_t njobs = max_tiles > 1 ? U * max_tiles : (U + run - 1) / run;
  int64_t ua = 0, ub = 0;  // voxels left of the job: a run is cut where the mesh changes
  int tno = 0;
#pragma unroll 1
  for (;;) {
    if (ua >= ub) {
      uint32_t tk = 0;
      if (lane == 0) tk = atomicAdd(bd.queue + kQueueNormals, 1u);
      const int64_t job = __shfl_sync(FULL, tk, 0);
      if (job >= njobs) break;
      ua = max_tiles > 1 ? job / max_tiles : job * run;
      ub = min(ua + run, U);
      tno = max_tiles > 1 ? (int)(job - ua * max_tiles) : 0;
    }
    const int mesh = mesh_by<&MeshDesc::u_base>(bd.md, bd.nmesh, ua);
    const MeshDesc &d = bd.md[mesh];
    const int nv = (int)(mesh + 1 < bd.nmesh ? min(ub, bd.md[mesh + 1].u_base) - ua : ub - ua);
    const int64_t u0 = ua;
    ua += nv;
    if (!d.has_l2) continue;  // warp-uniform
    const GridDev &g = d.g;
    const int n2x = g.n2[0], n2y = g.n2[1], n2z = g.n2[2];
    const int ncol2 = n2x * n2y, cells = ncol2 * n2z;
    const int c0 = tno * tile;
    if (c0 >= cells) continue;
    const int c1 = min(cells, c0 + tile), tc = c1 - c0;
    const bool all = tc == cells;
    const int rz0 = c0 / ncol2, rz1 = (c1 - 1) / ncol2;
    // rows of the tile (all of them unless it lies in one layer)
    const int ty0 = rz0 == rz1 ? (c0 - rz0 * ncol2) / n2x : 0;
    const int ty1 = rz0 == rz1 ? (c1 - 1 - rz0 * ncol2) / n2x : n2y - 1;
    const uint32_t layers = (0xffffffffu >> (31 - rz1)) & (0xffffffffu << rz0);
    if (lane <= nv) {
      const uint32_t e = useg[u0 + lane];
      ws.seg[lane] = e;
      if (lane < nv) {
        const uint32_t key = keys[e], col = key / (uint32_t)g.n[2], cj = col / (uint32_t)g.n[0];
        ws.kz[lane] = key - col * (uint32_t)g.n[2];
        ws.xy[lane] = (col - cj * (uint32_t)g.n[0]) | (cj << 16);
      }
    }
    __syncwarp();
    const float h0 = g.e2[0], h1 = g.e2[1], h2 = g.e2[2], gx = g.g2[0], gy = g.g2[1], gz = g.g2[2];
    // Where the tile is the voxel every triangle is taken; otherwise those that meet its layers and
    // rows are queued first, so that the lanes are full.
    const uint32_t e1 = ws.seg[nv];
    uint32_t scan = ws.seg[0], nq_ = 0, taken;  // the next list entry to look at; queued triangles
    int vcur = 0;
#pragma unroll 1
    while (vcur < nv) {
      if (all) nq_ = min(e1 - scan, 32u);
#pragma unroll 1
      while (!all && nq_ < 32 && scan < e1) {
        const uint32_t e = scan + (uint32_t)lane;
        bool keep = e < e1;
        uint32_t id = 0;
        if (keep) {
          id = vals[e] & 0x7fffffffu;
          const float4 v0 = __ldg(d.ptri + 3 * (size_t)id), v1 = __ldg(d.ptri + 3 * (size_t)id + 1),
                       v2 = __ldg(d.ptri + 3 * (size_t)id + 2);
          const float *sy = g.c2s[1] + (size_t)(ws.xy[0] >> 16) * n2y, *sz = g.c2s[2] + (size_t)ws.kz[0] * n2z;
          const float sy0 = __ldg(sy), sz0 = __ldg(sz);
          const float ty = 2.02f * EPS24 * fmaxf(fabsf(sy0), fabsf(__ldg(sy + n2y - 1)));
          const float tz = 2.02f * EPS24 * fmaxf(fabsf(sz0), fabsf(__ldg(sz + n2z - 1)));
          int a, b, x, y;
          cell_ranges(fminf(v0.z, fminf(v1.z, v2.z)), fmaxf(v0.z, fmaxf(v1.z, v2.z)), sz0, g.inv_g2[2], n2z,
                      ff(tz, g.inv_g2[2], kIdx), a, b, x, y);
          keep = max(a, rz0) <= min(b, rz1);
          cell_ranges(fminf(v0.y, fminf(v1.y, v2.y)), fmaxf(v0.y, fmaxf(v1.y, v2.y)), sy0, g.inv_g2[1], n2y,
                      ff(ty, g.inv_g2[1], kIdx), a, b, x, y);
          keep = keep && max(a, ty0) <= min(b, ty1);
        }
        const uint32_t bal = __ballot_sync(FULL, keep);
        if (keep) ws.que[nq_ + __popc(bal & ((1u << lane) - 1u))] = id;
        nq_ += (uint32_t)__popc(bal);
        scan += 32;
        __syncwarp();
      }
      // ---- a triangle per lane: its cell ranges, its plane and its rows
      const uint32_t n = min(nq_, 32u);
      int p0 = 0, p1 = -1, pi = 0, pe = 0, q0 = 0, q1 = -1, qi = 0, qe = 0, r0 = 0, r1 = -1, ri = 0, re = 0;
      int jv = 0;
      uint32_t t = 0, nsolve = 0;
      float4 a0, a1, a2;
      const float *sx = nullptr, *sy = nullptr, *sz = nullptr;
      float R = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
      bool on = false, direct = false, few = false;
      if (lane < (int)n) {
        if (all) {
          const uint32_t e = scan + (uint32_t)lane;
          while (jv + 1 < nv && ws.seg[jv + 1] <= e) ++jv;
          t = vals[e] & 0x7fffffffu;
        } else {
          t = ws.que[lane];
        }
        a0 = __ldg(d.ptri + 3 * (size_t)t), a1 = __ldg(d.ptri + 3 * (size_t)t + 1),
        a2 = __ldg(d.ptri + 3 * (size_t)t + 2);
        const uint32_t c = ws.xy[jv];
        sx = g.c2s[0] + (size_t)(c & 0xffffu) * n2x;
        sy = g.c2s[1] + (size_t)(c >> 16) * n2y;
        sz = g.c2s[2] + (size_t)ws.kz[jv] * n2z;
        const float sx0 = __ldg(sx), sy0 = __ldg(sy), sz0 = __ldg(sz);
        // (the bounds' constants as in the Level2 SAT, gpv_level2.cu)
        tx = 2.02f * EPS24 * fmaxf(fabsf(sx0), fabsf(__ldg(sx + n2x - 1)));
        ty = 2.02f * EPS24 * fmaxf(fabsf(sy0), fabsf(__ldg(sy + n2y - 1)));
        tz = 2.02f * EPS24 * fmaxf(fabsf(sz0), fabsf(__ldg(sz + n2z - 1)));
        const float xn = fminf(a0.x, fminf(a1.x, a2.x)), xx = fmaxf(a0.x, fmaxf(a1.x, a2.x));
        const float yn = fminf(a0.y, fminf(a1.y, a2.y)), yx = fmaxf(a0.y, fmaxf(a1.y, a2.y));
        const float zn = fminf(a0.z, fminf(a1.z, a2.z)), zx = fmaxf(a0.z, fmaxf(a1.z, a2.z));
        cell_ranges(xn, xx, sx0, g.inv_g2[0], n2x, ff(tx, g.inv_g2[0], kIdx), p0, p1, pi, pe);
        cell_ranges(yn, yx, sy0, g.inv_g2[1], n2y, ff(ty, g.inv_g2[1], kIdx), q0, q1, qi, qe);
        cell_ranges(zn, zx, sz0, g.inv_g2[2], n2z, ff(tz, g.inv_g2[2], kIdx), r0, r1, ri, re);
        on = p0 <= p1 && max(q0, ty0) <= min(q1, ty1) && max(r0, rz0) <= min(r1, rz1);
        if (on) {
          const int np = p1 - p0 + 1, nq = q1 - q0 + 1;
          R = 1.0001f * fmaxf(xx - xn + 1.25f * gx + 2.f * tx,
                              fmaxf(yx - yn + 1.25f * gy + 2.f * ty, zx - zn + 1.25f * gz + 2.f * tz));
          few = np * nq * (r1 - r0 + 1) <= kFewCells;
          direct = few || !(R > 1e-9f && R < 1e9f);
          nsolve = direct ? 0u : (uint32_t)(2 * nq + np);
        }
      }
      uint32_t is = nsolve;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, is, o);
        if (lane >= o) is += v;
      }
      taken = (uint32_t)__popc(__ballot_sync(FULL, lane < (int)n && is <= (uint32_t)kNSol));
      on = on && lane < (int)taken;
      const uint32_t so0 = is - nsolve;
      const int d0 = max(q0, ty0) - q0, d1 = min(q1, ty1) - q0 + 1;  // its rows in the tile
      uint32_t ncol = 0;
      if (on) {
        const int np = p1 - p0 + 1, nq = q1 - q0 + 1;
        ncol = (uint32_t)(np * (d1 - d0));
        uint32_t mz = (so0 + (uint32_t)nq) | ((so0 + 2u * (uint32_t)nq) << 16);
        if (few) {
          const float V[9] = {a0.x, a0.y, a0.z, a1.x, a1.y, a1.z, a2.x, a2.y, a2.z};
          const float h[3] = {h0, h1, h2};
          uint32_t bits = 0;
          int i = 0;
#pragma unroll 1
          for (int r = r0; r <= r1; ++r)
#pragma unroll 1
            for (int q = q0; q <= q1; ++q)
#pragma unroll 1
              for (int p = p0; p <= p1; ++p, ++i) {
                const float c3[3] = {__ldg(sx + p), __ldg(sy + q), __ldg(sz + r)};
                if (tri_box(V, c3, h)) bits |= 1u << i;
              }
          mz = bits;
          if (!bits) ncol = 0;
        }
        ws.me[lane] = make_uint4(t, (uint32_t)(jv | (few ? 512 : direct ? 256 : 0) | (p0 << 16) | (q0 << 24)), mz,
                                 (uint32_t)(r0 | ((r1 + 1) << 8) | (np << 16) | (nq << 24)));
        if (!direct) {
          const float c0x = __ldg(sx + p0), c0y = __ldg(sy + q0), c0z = __ldg(sz + r0);
          const float ux = a0.x - c0x, uy = a0.y - c0y, uz = a0.z - c0z;
          const float vx = a1.x - c0x, vy = a1.y - c0y, vz = a1.z - c0z;
          const float wx = a2.x - c0x, wy = a2.y - c0y, wz = a2.z - c0z;
          float nnx = (vy - uy) * (wz - vz) - (vz - uz) * (wy - vy);
          float nny = (vz - uz) * (wx - vx) - (vx - ux) * (wz - vz);
          float nnz = (vx - ux) * (wy - vy) - (vy - uy) * (wx - vx);
          if (nnz < 0.f) { nnx = -nnx; nny = -nny; nnz = -nnz; }
          const float E = 192.f * EPS24 * R * R * (R + fmaxf(h0, fmaxf(h1, h2))) +
                          1.1f * (fabsf(nnx) * tx + fabsf(nny) * ty + nnz * tz);
          const float inv = rcp_fast(fmaxf(nnz * gz, E * (1.f / 512.f)));
          const float w = ff(E, inv, kIdx);
          ws.xa[lane] = make_float4(nnx * ux + nny * uy + nnz * uz, nnx * gx, nny * gy,
                                    fabsf(nnx) * h0 + fabsf(nny) * h1 + nnz * h2);
          ws.xb[lane] = make_float4(inv, (float)r0 - w, (float)r0 + w, 0.f);
          const float dl = 72.f * EPS24 * R * R, bx = 1.1f * tx, by = 1.1f * ty, bz = 1.1f * tz;
          uint32_t *so = ws.sol + so0;
          const uint32_t xl = (uint32_t)(p0 | (pi << 16)), xe = (uint32_t)(pe | ((p1 + 1) << 16));
          const uint32_t zl = (uint32_t)(r0 | (ri << 16)), ze = (uint32_t)(re | ((r1 + 1) << 16));
          ncol = solve_rows(so, nq, ux, vx, wx, uy, vy, wy, h0, h1, gx, gy, dl, bx, by, p0, xl, xe, qi - q0, qe - q0);
          solve_rows(so + nq, nq, uz, vz, wz, uy, vy, wy, h2, h1, gz, gy, dl, bz, by, r0, zl, ze, qi - q0, qe - q0);
          solve_rows(so + 2 * nq, np, uz, vz, wz, ux, vx, wx, h2, h0, gz, gx, dl, bz, bx, r0, zl, ze, pi - p0, pe - p0);
          if (!all) {
            ncol = 0;
#pragma unroll 1
            for (int dq = d0; dq < d1; ++dq) ncol += max(so[dq] >> 24, so[dq] & 255u) - (so[dq] & 255u);
          }
        }
      }
      uint32_t ic = ncol;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, ic, o);
        if (lane >= o) ic += v;
      }
      taken = (uint32_t)__popc(__ballot_sync(FULL, lane < (int)taken && ic <= (uint32_t)kNCols));
      if (lane >= (int)taken) jv = -1;
      if (ncol && lane < (int)taken)
        list_columns(ws.cols + (ic - ncol), direct ? nullptr : ws.sol + so0, lane, p0, p1 - p0 + 1, d0, d1);
      // the rest of the list, or of the queue to its front
      bool rest;  // the voxel has more triangles
      if (all) {
        scan += taken;
        rest = true;  // (by voxel, below)
      } else {
        const uint32_t i0 = (uint32_t)lane + taken, i1 = i0 + 32;
        const uint32_t k0 = i0 < nq_ ? ws.que[i0] : 0u, k1 = i1 < nq_ ? ws.que[i1] : 0u;
        __syncwarp();
        if (i0 < nq_) ws.que[lane] = k0;
        if (i1 < nq_) ws.que[lane + 32] = k1;
        nq_ -= taken;
        rest = nq_ > 0 || scan < e1;
      }
      __syncwarp();
      // ---- the sub-columns, voxel by voxel, in list order
      uint32_t pos = 0;
#pragma unroll 1
      while (vcur < nv) {
        const uint32_t bal = __ballot_sync(FULL, jv == vcur);
        const uint32_t end_ = bal ? __shfl_sync(FULL, ic, 31 - __clz(bal)) : pos;
        const uint32_t cv = ws.xy[vcur];
        const float *vx_ = g.c2s[0] + (size_t)(cv & 0xffffu) * n2x, *vy_ = g.c2s[1] + (size_t)(cv >> 16) * n2y,
                    *vz_ = g.c2s[2] + (size_t)ws.kz[vcur] * n2z;
#pragma unroll 1
        for (; pos < end_; pos += 32) {
          const uint32_t c = pos + (uint32_t)lane;
          uint32_t m = 0, pq = 0x8000u | (uint32_t)lane;
          float4 fnv = make_float4(0.f, 0.f, 0.f, 0.f);
          if (c < end_) {
            const uint32_t en = ws.cols[c];
            const int tl = (int)(en & 31u), dq = (int)((en >> 5) & 31u), dp = (int)((en >> 10) & 31u);
            const uint4 me = ws.me[tl];
            fnv = __ldg(d.fnorm + me.x);
            const int p = (int)((me.y >> 16) & 255u) + dp, q = (int)(me.y >> 24) + dq;
            if (me.y & 512u) {  // few cells: exact results
              const int np = (int)((me.w >> 16) & 255u), box = np * (int)(me.w >> 24);
              uint32_t b = me.z >> (dq * np + dp);
#pragma unroll 1
              for (int r = (int)(me.w & 255u); b; ++r, b >>= box) m |= (b & 1u) << r;
            } else {
              int lo = (int)(me.w & 255u), end = (int)((me.w >> 8) & 255u);
              bool exact = true;
              if (!(me.y & 256u)) {
                const float4 xa = ws.xa[tl], xb = ws.xb[tl];
                const uint32_t syz = ws.sol[(me.z & 0xffffu) + (uint32_t)dq];
                const uint32_t sxz = ws.sol[(me.z >> 16) + (uint32_t)dp];
                const float nv_ = ff(-(float)dp, xa.y, ff(-(float)dq, xa.z, xa.x));
                const float va = nv_ - xa.w, vb = nv_ + xa.w;
                const uint32_t L = __vimax3_s16x2(cvt_pair_ceil(ff(va, xb.x, xb.y), ff(va, xb.x, xb.z)),
                                                  __byte_perm(syz, 0, 0x4140), __byte_perm(sxz, 0, 0x4140));
                const uint32_t E = __vimin3_s16x2(
                    cvt_pair_floor(ff(vb, xb.x, xb.y + 1.f), ff(vb, xb.x, xb.z + 1.f)),
                    __byte_perm(syz, 0, 0x4342), __byte_perm(sxz, 0, 0x4342));
                lo = (int)(short)(L & 0xffffu);
                end = (int)E >> 16;
                exact = !((en & 0x8000u) && lo == (int)L >> 16 && end == (int)(short)(E & 0xffffu));
              }
              lo = max(lo, rz0);
              end = min(end, rz1 + 1);
              if (lo < end)
                m = exact ? exact_cells(d.ptri + 3 * (size_t)me.x, __ldg(vx_ + p), __ldg(vy_ + q), vz_, h0, h1, h2,
                                        lo, end)
                          : (0xffffffffu >> (32 - (end - lo))) << lo;
            }
            m &= layers;
            if (m) pq = (uint32_t)(q * n2x + p);
          }
          const uint32_t peers = __match_any_sync(FULL, pq);
          const int rank = __popc(peers & ((1u << lane) - 1u));
          const int rounds = __reduce_max_sync(FULL, rank);
#pragma unroll 1
          for (int k = 0; k <= rounds; ++k) {
            if (k == rank) {
#pragma unroll 1
              while (m) {
                const int r = __ffs(m) - 1;
                m &= m - 1u;
                const int ct = r * ncol2 + (int)pq - c0;
                if (ct < 0 || ct >= tc) continue;
                float *v = ws.sum + 3 * ct;
                v[0] = fa(v[0], fnv.x);
                v[1] = fa(v[1], fnv.y);
                v[2] = fa(v[2], fnv.z);
                ws.cnt[ct] = fa(ws.cnt[ct], 1.f);
              }
            }
            __syncwarp();
          }
        }
        pos = end_;
        if (all ? ws.seg[vcur + 1] > scan : rest) break;  // more of this voxel in the next batch
        const int64_t vlin = ((int64_t)ws.kz[vcur] * g.n[1] + (cv >> 16)) * g.n[0] + (cv & 0xffffu);
        finish_voxel(ws, tc, bd.normals, d.l2n, (int64_t)d.prefix[vlin] * cells + c0);
        ++vcur;
      }
      __syncwarp();
    }
  }
}

}  // namespace

void launch_face_normals(const BatchDev &bd, cudaStream_t s) {
  if (bd.total_tris <= 0) return;
  k_face_normals<<<(unsigned)((bd.total_tris + 255) / 256), 256, 0, s>>>(bd);
  count_launch();
}

int64_t seg_sort_words(int64_t U) { return U + 1; }

void launch_seg_sort(const BatchDev &bd, uint32_t *vals, const uint32_t *useg, int64_t U, uint32_t *longs,
                     uint32_t *spare, int num_sms, cudaStream_t s) {
  if (U <= 0) return;
  cudaMemsetAsync(longs, 0, sizeof(uint32_t), s);
  k_seg_sort<<<(unsigned)((U + kNWarps - 1) / kNWarps), kNWarps * 32, 0, s>>>(vals, useg, U, longs);
  const size_t smem = kMapIds / 4;  // two bits an id
  static OncePerDevice once;
  allow_shared_memory(once, k_seg_sort_long, smem);
  k_seg_sort_long<<<(unsigned)std::min<int64_t>(U, num_sms), 1024, smem, s>>>(bd, vals, useg, longs, spare);
  count_launch(2);
}

void launch_normals(const BatchDev &bd, const uint32_t *keys, const uint32_t *vals,
                    const uint32_t *useg, int64_t U, int64_t P, int max_cells, int num_sms,
                    cudaStream_t s) {
  if (U <= 0) return;
  const int per_warp = U < (int64_t)num_sms * 32 ? 1 : 32;
  k_level1_normals<<<(unsigned)((U + 4 * per_warp - 1) / (4 * per_warp)), 128, 0, s>>>(bd, keys, vals, useg, U,
                                                                                     per_warp);
  count_launch();
  if (max_cells <= 0) return;
  const size_t smem = kNWarps * sizeof(NWarp);
  static OncePerDevice once;
  allow_shared_memory(once, k_level2_normals, smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_level2_normals, kNWarps * 32, smem);
  const int64_t warps = (int64_t)num_sms * std::max(per_sm, 1) * kNWarps;
  // Few voxels (a coarse grid with long lists): smaller tiles, so that every SM has warps.  A warp
  // walks its voxel's whole list, but only the triangles that meet its tile's layers and rows cost more
  // than their ranges.
  int tile = std::min(kNTileCells, std::max(max_cells, 1));
  while (tile > 4 && U * ((max_cells + tile - 1) / tile) < warps) tile = (tile + 1) / 2;
  const int tiles = (max_cells + tile - 1) / tile;
  // voxels of a run: about one batch of triangles (53k voxels of 8 triangles: runs of 2, 3, 4, 5 and 8
  // voxels 277, 263, 264, 266 and 282 us), while every warp still gets a few runs
  const int64_t batch = 32 * U / std::max<int64_t>(P, 1);
  const int run = tiles > 1 ? 1 : (int)std::max<int64_t>(1, std::min({(int64_t)kNRun, batch, U / (4 * warps)}));
  const int64_t grid = std::min<int64_t>((U * tiles / run + kNWarps) / kNWarps, (int64_t)num_sms * std::max(per_sm, 1));
  k_level2_normals<<<(unsigned)grid, kNWarps * 32, smem, s>>>(bd, keys, vals, useg, U, tile, tiles, run);
  count_launch();
}

}  // namespace gpv
