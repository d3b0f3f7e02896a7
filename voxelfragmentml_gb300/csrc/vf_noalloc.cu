// vf_noalloc.cu -- flood fracture without any device allocation.
//
// Some callers cannot allocate device memory while they run this step: a
// renderer or simulation that owns every allocation through its own pool,
// code that must not grow its footprint after start-up, or an embedding
// whose allocator is not the CUDA runtime's.  vf_flood_noalloc serves them:
// the caller passes its own device buffers for the input grid, the seeds and
// the output labels, and every intermediate (the flood's row states,
// candidate masks, gang tables and job state) lives in one file-scope device
// array, g_scratch, of VF_NOALLOC_SCRATCH_BYTES.
//
// Properties of the scratch array:
//   - it is part of the library image: every GPU that loads the library
//     holds it until the process exits;
//   - every call on a device shares it and it keeps the contents of the last
//     call; each call clears what must start at zero before using it;
//   - calls whose work overlaps on the GPU (two host threads, or two streams
//     without ordering between them) race on it and give wrong results;
//   - its flood is a cooperative launch whose CTAs wait for one another: a
//     call must not overlap a vf_ctx's batched flood (vf_batch_run,
//     vf_pipeline_*, a vf_server) on another stream either, or a wait may
//     run out (VF_ERR_TIMEOUT).
// When the call returns an error the contents of d_labels are unspecified.
//
// Host code cannot use the name g_scratch as a device address (on the host
// it is only a stand-in symbol).  The first call on each device, with that
// device current, resolves the address with cudaGetSymbolAddress and caches
// it; make that first call before any stream capture begins.
#include <cstddef>
#include <utility>
#include <mutex>
#include <string>

#include "vf_runtime.h"

#define VF_NOALLOC_SCRATCH_BYTES (32u << 20)

static __device__ __align__(256) unsigned char g_scratch[VF_NOALLOC_SCRATCH_BYTES];

namespace {

std::mutex g_mu;
void* g_addr[64] = {};  // resolved scratch address per device
int g_sms[64] = {};     // multiprocessor count per device

size_t up(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace

extern "C" vf_status vf_flood_noalloc(const uint16_t* d_grid, uint16_t* d_labels, uint32_t X,
                                      uint32_t Y, uint32_t Z, const uint32_t* d_seeds_xyzw,
                                      uint32_t nseeds, int distance, void* stream) {
  using vfr::fail;
  if (!d_grid || !d_labels || (nseeds && !d_seeds_xyzw))
    return fail(VF_ERR_INVALID, "vf_flood_noalloc: NULL buffer");
  if (X < 1 || Y < 1 || Z < 1 || X > VF_MAX_DIM || Y > VF_MAX_DIM || Z > VF_MAX_DIM)
    return fail(VF_ERR_INVALID, "vf_flood_noalloc: dims must be in [1, 4096]");
  if (distance < VF_EUCLIDEAN || distance > VF_CHEBYSHEV)
    return fail(VF_ERR_INVALID, "vf_flood_noalloc: distance out of range");
  if (nseeds > VF_MAX_SEEDS) return fail(VF_ERR_RANGE, "vf_flood_noalloc: at most 4095 seeds");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return fail(VF_ERR_NOT_BUILT, "vf_flood_noalloc: no current CUDA device");
  void* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_addr[dev]) {
      cudaError_t e = cudaGetSymbolAddress(&g_addr[dev], g_scratch);
      if (e != cudaSuccess) {
        g_addr[dev] = nullptr;
        return fail(VF_ERR_CUDA, std::string("vf_flood_noalloc: cudaGetSymbolAddress: ") +
                                     cudaGetErrorString(e));
      }
    }
    base = g_addr[dev];
    if (!g_sms[dev] &&
        cudaDeviceGetAttribute(&g_sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      g_sms[dev] = 0;
      return fail(VF_ERR_CUDA, "vf_flood_noalloc: device query failed");
    }
  }
  const int num_sms = g_sms[dev];
  // Size limit: the scratch rule of a padded copy of the grid, 4 bytes of
  // state per voxel and 93 bytes per brick, which callers were promised; the
  // rows need at most 0.83 of it (over all shapes at the rule's edge).
  const size_t nb = (size_t)((X + VF_BX - 1) / VF_BX) * ((Y + VF_BY - 1) / VF_BY) * ((Z + VF_BZ - 1) / VF_BZ);
  const size_t rule = up(sizeof(JobDesc)) + up(sizeof(JobState)) + up(4096) + 256 + 6 * up(nb * 4) + up(nb) +
                      up(nb * 68) + up((size_t)X * Y * vf_roundup(Z, 8) * 2) + up((size_t)X * Y * vf_roundup(Z, 4) * 4);
  if (rule > VF_NOALLOC_SCRATCH_BYTES)
    return fail(VF_ERR_RANGE, "vf_flood_noalloc: the grid needs " + std::to_string(rule) +
                                  " bytes of scratch; the no-allocation flood holds " +
                                  std::to_string(VF_NOALLOC_SCRATCH_BYTES) +
                                  " bytes (about 5 million voxels)");
  // Words along z; along the longest axis where z is shorter than a word, so
  // that a thin grid does not pay for empty bits.  Lanes along the longer of
  // the other two.
  const uint32_t D[3] = {X, Y, Z};
  uint32_t w = 2;
  if (Z < 32) {
    if (X > D[w]) w = 0;
    if (Y > D[w]) w = 1;
  }
  uint32_t o = w == 0 ? 1 : 0, l = w == 2 ? 1 : 2;
  if (D[o] > D[l]) std::swap(o, l);
  const size_t stride[3] = {(size_t)Y * Z, Z, 1};
  const uint32_t sw = vfk::wave_state_words(nseeds);
  // a scratch layout too large with these axes takes the order that needs least
  auto bytes = [&](uint32_t a, uint32_t b, uint32_t c) {
    return vfk::wave_rows(D[a], D[b], (D[c] + 31) / 32) * (sw * 4ull + 16 + 1);
  };
  if (bytes(o, l, w) > VF_NOALLOC_SCRATCH_BYTES / 2) {
    const uint32_t perm[6][3] = {{0, 1, 2}, {1, 0, 2}, {0, 2, 1}, {2, 0, 1}, {1, 2, 0}, {2, 1, 0}};
    for (const auto& q : perm)
      if (bytes(q[0], q[1], q[2]) < bytes(o, l, w)) { o = q[0]; l = q[1]; w = q[2]; }
  }
  const vfk::FlatAxes A = {{stride[o], stride[l], stride[w]}, D[o], D[l], D[w], {X, Y, Z}, o | (l << 4) | (w << 8)};
  vfk::WaveJob W = {};
  vfk::wave_layout(W, 0, D[o], D[l], (D[w] + 31) / 32);
  W.conn6 = distance == VF_MANHATTAN ? 1u : 0u;
  W.order = A.order;
  const vfk::WaveShape shape = vfk::flood_shape(sw, 1, num_sms, 0);
  const size_t blocks = (size_t)shape.blocks, rows = ((size_t)W.nrows + 255) / 256 * 256;
  // layout of the scratch array: job state, flood words, barrier and masks
  // (cleared per call), gang tables, row states
  size_t off = 0;
  const size_t o_state = off; off += up(sizeof(JobState));
  const size_t o_scal = off; off += up(4096);
  const size_t o_bar = off; off += up(vfk::WAVE_BAR_WORDS * 4);
  const size_t o_last = off; off += up(4);
  const size_t o_cand = off; off += up(2 * (rows / 32) * 4);
  const size_t cleared = off;
  const size_t o_job = off; off += up(sizeof(vfk::WaveJob));
  const size_t o_gang = off; off += up(sizeof(vfk::WaveGang));
  const size_t o_cta = off; off += up(sizeof(vfk::WaveCta) * blocks);
  const size_t o_ent = off; off += up(sizeof(vfk::WaveEntry) * blocks);
  const size_t o_in = off; off += up(rows * 16);
  const size_t o_rows = off; off += up(rows * sw * 4);
  if (off > VF_NOALLOC_SCRATCH_BYTES)
    return fail(VF_ERR_RANGE, "vf_flood_noalloc: the grid needs " + std::to_string(off) + " bytes of scratch");
  unsigned char* S = static_cast<unsigned char*>(base);
  JobState* dstate = reinterpret_cast<JobState*>(S + o_state);
  vfk::FloodScratch fs;
  fs.arr = {reinterpret_cast<uint32_t*>(S + o_rows), reinterpret_cast<uint2*>(S + o_in),
            reinterpret_cast<uint32_t*>(S + o_cand), (uint32_t)(rows / 32)};
  fs.jobs = reinterpret_cast<vfk::WaveJob*>(S + o_job);
  fs.njobs = 1;
  fs.gangs = reinterpret_cast<vfk::WaveGang*>(S + o_gang);
  fs.cta = reinterpret_cast<vfk::WaveCta*>(S + o_cta);
  fs.entries = reinterpret_cast<vfk::WaveEntry*>(S + o_ent);
  fs.shape = shape;
  fs.sw = sw;
  fs.bar = reinterpret_cast<uint32_t*>(S + o_bar);
  fs.last = reinterpret_cast<uint32_t*>(S + o_last);
  fs.stats = reinterpret_cast<uint32_t*>(S + o_scal);
  fs.err = &dstate->disjoint;  // next to err and has_prefix: one copy reads all three
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define NA_CK(call)                                                                         \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      return fail(VF_ERR_CUDA, std::string("vf_flood_noalloc: ") + cudaGetErrorString(e_)); \
  } while (0)
  NA_CK(cudaMemsetAsync(S, 0, cleared, st));
  vfk::flat_init(st, d_grid, fs.arr, W, A, sw, dstate, num_sms);
  // Without seeds nothing is claimed: occupied voxels come out FREE (1), as
  // FloodFracturer::build leaves them after homogenize.
  if (nseeds) {
    vfk::flat_seed(st, W, A, fs, d_seeds_xyzw, nseeds, dstate);
    NA_CK(vfk::flood_waves(st, dstate, fs));
  }
  vfk::flat_labels(st, fs.arr, W, A, sw, d_seeds_xyzw, nullptr, d_labels, num_sms);
  NA_CK(cudaGetLastError());
  static_assert(offsetof(JobState, disjoint) == offsetof(JobState, err) + 8, "err, has_prefix, disjoint in a row");
  uint32_t status[3] = {0, 0, 0};
  NA_CK(cudaMemcpyAsync(status, &dstate->err, sizeof(status), cudaMemcpyDeviceToHost, st));
  NA_CK(cudaStreamSynchronize(st));
#undef NA_CK
  const uint32_t err = status[0], has_prefix = status[1], ferr = status[2];
  if (err & VF_JERR_INVALID) return fail(VF_ERR_INVALID, "vf_flood_noalloc: seed outside the grid or label not a valid fragment label (<= 0x7FFF, low byte >= 2)");
  if (has_prefix)
    return fail(VF_ERR_INVALID, "vf_flood_noalloc: seed labels with sub-seed prefixes (> 255) need vf_fracture");
  if (ferr) return fail(VF_ERR_TIMEOUT, "vf_flood_noalloc: flood did not converge (bounded wait expired)");
  if (err & VF_JERR_DIST_OVERFLOW) return fail(VF_ERR_RANGE, "vf_flood_noalloc: geodesic distance overflow");
  return VF_OK;
}
