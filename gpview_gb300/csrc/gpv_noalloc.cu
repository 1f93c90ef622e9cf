// gpv_noalloc.cu -- Level1 voxelization that allocates nothing.
//
// Some callers cannot call cudaMalloc: code that runs inside another allocator's or memory
// pool's hooks (a call back into the allocator would recurse or deadlock), host paths that must
// not take the implicit device synchronisation that cudaMalloc/cudaFree can cause, and plugin
// hosts that hand a library its buffers and forbid it to acquire device memory of its own.
// gpv_voxelize_level1_noalloc serves them: the caller passes the triangles and the three Level1
// outputs, and every intermediate lives in g_noalloc_scratch, a file-scope __device__ array of
// fixed size (kScratchBytes, 32 MiB) that every GPU loading this library holds until the
// process exits.
//
// Rules of use:
//   * Host code cannot use the array's name as a device address.  Every call looks the address
//     up with cudaGetSymbolAddress while the caller's device is current and checks the result
//     (a lookup costs far less than the call's own stream synchronisation, and it stays right
//     after a device reset, which loads the module -- and the array -- again).
//   * A call copies its tables from host memory and waits for its stream, so it cannot be
//     recorded into a graph: a call on a stream that is capturing is refused.
//   * All calls share the one array, which keeps the previous call's contents.  Each call clears
//     the regions that must start at zero.  Calls whose GPU work overlaps -- on different
//     streams or host threads -- race on the array; serialise them.
//   * Sizes whose intermediates do not fit the array are rejected with GPV_ERR_INVALID and a
//     message from gpv_noalloc_last_error() (kept per host thread); nothing is launched then.
//   * No cudaMalloc, cudaFree, host heap or library allocation is made.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "gpv_internal.h"

namespace gpv {
namespace {

constexpr size_t kScratchBytes = size_t(32) << 20;
constexpr int kMaxTableFloats = 12288;  // nx + ny + nz
// Scratch bytes per triangle (packed vertices 48, SAT box 16, ray box 16).  Triangle counts are
// checked against the array with this before any size is formed, so no size can wrap.
constexpr size_t kBytesPerTriangle = 80;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

thread_local char g_err[256] = "";
// failure-detection hooks of this host thread's calls (gpv_noalloc_set_debug)
thread_local uint32_t g_wait_limit = 0;
thread_local int g_fail_wait = 0;

void set_err(const char *msg) {
  std::snprintf(g_err, sizeof(g_err), "%s", msg);
}

size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

}  // namespace
}  // namespace gpv

using namespace gpv;

extern "C" const char *gpv_noalloc_last_error(void) { return g_err; }

extern "C" int gpv_noalloc_set_debug(int what, int64_t value) {
  if (value < 0 || value > 0xffffffffll) return GPV_ERR_INVALID;
  switch (what) {
    case GPV_DEBUG_WAIT_LIMIT: g_wait_limit = (uint32_t)value; return GPV_OK;
    case GPV_DEBUG_FAIL_WAIT: g_fail_wait = value != 0; return GPV_OK;
    default: return GPV_ERR_INVALID;
  }
}

extern "C" int gpv_voxelize_level1_noalloc(const float *d_tris, int64_t num_triangles,
                                           const gpv_grid_spec *spec, uint8_t *d_level1_inout,
                                           int32_t *d_level1_prefix, int32_t *d_boundary_index,
                                           int64_t *num_boundary, cudaStream_t stream) {
  if (!spec || !d_level1_inout || !d_level1_prefix || !d_boundary_index || !num_boundary ||
      num_triangles < 0 || (num_triangles > 0 && !d_tris)) {
    set_err("null argument or negative triangle count");
    return GPV_ERR_INVALID;
  }
  if (num_triangles > 0 && (reinterpret_cast<uintptr_t>(d_tris) & 15u)) {
    set_err("triangle buffer must be 16-byte aligned");
    return GPV_ERR_INVALID;
  }
  {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      set_err("stream is capturing (the call copies from host memory and waits for the stream)");
      return GPV_ERR_INVALID;
    }
  }
  if (num_triangles > (int64_t)(kScratchBytes / kBytesPerTriangle)) {
    char msg[160];
    std::snprintf(msg, sizeof(msg),
                  "%lld triangles exceed the fixed no-alloc scratch (%zu bytes, %zu per triangle)",
                  (long long)num_triangles, kScratchBytes, kBytesPerTriangle);
    set_err(msg);
    return GPV_ERR_INVALID;
  }
  // Level2 divisions are not used here, but a specification gpv_voxelize would reject is
  // rejected here too: each in 0..32, all zero or all positive.
  {
    const int32_t *n2 = spec->ndiv2;
    const bool any2 = n2[0] || n2[1] || n2[2], all2 = n2[0] && n2[1] && n2[2];
    if (n2[0] < 0 || n2[1] < 0 || n2[2] < 0 || n2[0] > 32 || n2[1] > 32 || n2[2] > 32 ||
        (any2 && !all2)) {
      set_err("invalid grid specification (Level2 divisions)");
      return GPV_ERR_INVALID;
    }
  }
  // ---- grid, derived exactly as the plain path does (no host heap: tables on the stack)
  GridDev g;
  std::memset(&g, 0, sizeof(g));
  int64_t N1 = 1;
  int ntab = 0;
  for (int a = 0; a < 3; ++a) {
    const int n = spec->ndiv[a];
    if (n < 1 || n > 65535 || !std::isfinite(spec->bbox_min[a]) ||
        !std::isfinite(spec->bbox_max[a]) || !(spec->bbox_max[a] > spec->bbox_min[a])) {
      set_err("invalid grid specification");
      return GPV_ERR_INVALID;
    }
    N1 *= n;
    ntab += n;
  }
  if (ntab > kMaxTableFloats || N1 >= ((int64_t)1 << 31)) {
    set_err("grid exceeds the no-alloc limits (nx+ny+nz <= 12288)");
    return GPV_ERR_INVALID;
  }
  float tab[kMaxTableFloats];
  int off = 0;
  for (int a = 0; a < 3; ++a) {
    const int n = spec->ndiv[a];
    const float span = spec->bbox_max[a] - spec->bbox_min[a];
    g.bmin[a] = spec->bbox_min[a];
    g.bmax[a] = spec->bbox_max[a];
    g.n[a] = n;
    g.n2[a] = 0;
    g.g[a] = (float)(span / (n * 1.0));
    g.e1[a] = (float)(g.g[a] / 2.0);
    for (int i = 0; i < n; ++i) tab[off + i] = (float)((i + 0.5) * g.e1[a] * 2 + (double)spec->bbox_min[a]);
    off += n;
  }
  g.nxw = (g.n[0] + 31) / 32;
  g.nzw = (g.n[2] + 31) / 32;
  g.thr = eps_threshold();
  const int64_t T = num_triangles;
  const int64_t N1w = (int64_t)g.n[2] * g.n[1] * g.nxw;
  const int64_t ncol = (int64_t)g.n[0] * g.n[1];

  // ---- scratch layout and limit
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align256(o + bytes); return at; };
  const size_t o_tab = take(sizeof(float) * ntab);
  const size_t o_ptri = take(48 * (size_t)T);
  const size_t o_rng = take(16 * (size_t)T);
  const size_t o_fbox = take(16 * (size_t)T);
  const size_t o_bp = take(4 * (size_t)N1w);
  const size_t o_ip = take(4 * (size_t)N1w);
  const size_t o_tg = take(4 * (size_t)(ncol * g.nzw));
  const size_t o_hv = take(4 * (size_t)N1w);  // pieces of large triangles
  const size_t o_wp = take(4 * (size_t)N1w);
  const size_t o_sc = take(4 * (size_t)scan_temp_words(N1w));
  const size_t o_st = take(sizeof(MeshStats));
  const size_t o_tot = take(16);
  const size_t o_md = take(sizeof(MeshDesc));
  if (o > kScratchBytes) {
    char msg[160];
    std::snprintf(msg, sizeof(msg),
                  "inputs need %zu bytes of scratch; the fixed no-alloc scratch holds %zu", o,
                  kScratchBytes);
    set_err(msg);
    return GPV_ERR_INVALID;
  }

  // ---- the array's device address on the current device (looked up on every call)
  unsigned char *base = nullptr;
  int num_sms = 1;
  {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      set_err("cudaGetSymbolAddress failed for the no-alloc scratch array (no usable device?)");
      return GPV_ERR_CUDA;
    }
    base = static_cast<unsigned char *>(p);
  }

  float *d_tab = reinterpret_cast<float *>(base + o_tab);
  for (int a = 0, oo = 0; a < 3; ++a) { g.c1[a] = d_tab + oo; oo += g.n[a]; }
  MeshDesc md;
  std::memset(&md, 0, sizeof(md));
  md.g = g;
  md.tris = d_tris;
  md.T = T;
  md.ptri = reinterpret_cast<float4 *>(base + o_ptri);
  md.rng = reinterpret_cast<int4 *>(base + o_rng);
  md.fbox = reinterpret_cast<float4 *>(base + o_fbox);
  md.bplane = reinterpret_cast<uint32_t *>(base + o_bp);
  md.iplane = reinterpret_cast<uint32_t *>(base + o_ip);
  md.toggles = reinterpret_cast<uint32_t *>(base + o_tg);
  md.stats = reinterpret_cast<MeshStats *>(base + o_st);
  md.l1 = d_level1_inout;
  md.prefix = d_level1_prefix;
  md.bindex = d_boundary_index;
  MeshDesc *d_md = reinterpret_cast<MeshDesc *>(base + o_md);
  uint32_t *wpre = reinterpret_cast<uint32_t *>(base + o_wp);
  uint32_t *stmp = reinterpret_cast<uint32_t *>(base + o_sc);
  uint32_t *d_tot = reinterpret_cast<uint32_t *>(base + o_tot);
  BatchDev bd;
  std::memset(&bd, 0, sizeof(bd));
  bd.md = d_md;
  bd.nmesh = 1;
  bd.tile = 32;
  bd.total_tiles = (T + 31) / 32;
  bd.queue = d_tot + 1;  // (the total takes the first word)
  // the pieces of large triangles: their own region, or what the array has left where that is more
  const size_t own_cap = (size_t)N1w / 4, rest_cap = (kScratchBytes - o) / sizeof(uint4);
  bd.heavy_cap = (uint32_t)std::min<size_t>(std::max(own_cap, rest_cap), kHeavyCap);
  bd.heavy = bd.heavy_cap ? reinterpret_cast<uint4 *>(base + (rest_cap > own_cap ? o : o_hv)) : nullptr;
  bd.heavy_n = reinterpret_cast<unsigned long long *>(d_tot + 2);
  bd.wait_limit = g_wait_limit;
  bd.fail_wait = g_fail_wait;
  bd.total_tris = T;
  bd.total_fblks = finish_blocks((int64_t)g.n[1] * g.nxw);
  bd.total_xchunks = (N1w + 31) / 32;
  bd.total_words = N1w;

  // The array keeps the last call's data: clear everything that must start at zero.  The
  // descriptor and the tables are copied from this function's stack (pageable memory: the copy
  // has been staged by the time cudaMemcpyAsync returns).
  cudaError_t e = cudaMemcpyAsync(d_tab, tab, sizeof(float) * ntab, cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_md, &md, sizeof(md), cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(md.stats, 0, sizeof(MeshStats), stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_tot, 0, 16, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(md.bplane, 0, 4 * (size_t)N1w, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(md.toggles, 0, 4 * (size_t)(ncol * g.nzw), stream);
  if (e != cudaSuccess) {
    set_err(cudaGetErrorString(e));
    return GPV_ERR_CUDA;
  }
  launch_prep(bd, stream);
  launch_level1(bd, num_sms, stream);  // (no Level2 grid: the records are counted, not written)
  launch_fill_finish(bd, stream);
  scan_u32(md.bplane, wpre, N1w, d_tot, stmp, stream, true);
  launch_expand(bd, wpre, num_sms, stream);
  uint32_t nb = 0;
  MeshStats hs;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&nb, d_tot, sizeof(nb), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hs, md.stats, sizeof(hs), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) {
    set_err(cudaGetErrorString(e));
    return GPV_ERR_CUDA;
  }
  if (hs.status & ST_BAD_INPUT) {
    set_err("non-finite vertex");
    return GPV_ERR_INVALID;
  }
  if (hs.status) {
    set_err("device status raised in Level1 (a bounded wait gave up)");
    return GPV_ERR_DEVICE;
  }
  *num_boundary = (int64_t)nb;
  set_err("");
  return GPV_OK;
}
