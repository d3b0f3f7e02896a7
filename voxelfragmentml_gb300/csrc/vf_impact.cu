// vf_impact.cu -- the impact path on sm_103a: the voxel a ray enters first
// (RegularGrid::getClosestEntryVoxel -> rayTraversalAmanatidesWoo,
// RegularGrid.cpp:265-270, 853-1004) for a batch of rays, and the seeds
// placed around impacts (Seeder::nearSeeds, Seeder.cpp:49-113), as
// CADScene::hit and CADScene::fractureModel use them (CADScene.cpp:508-520,
// 629-645).
//
//   k_occ_bits    (batches of rays) the grid's occupancy packed 1 bit per
//                 voxel in an L2-resident bitmap, and 1 bit per cell of 8^3
//                 voxels or more, which the walks hold in shared memory
//   k_ray_entry   a lane per ray, refilled (few rays, on the labels:
//                 k_ray_labels): the reference's slab test and Amanatides-Woo walk in its operation order (every float
//                 step rounded as written); the walk is bounded by
//                 X + Y + Z + 3 steps, more than a ray can take
//   k_near_seeds  one CTA running vfnear::place (vf_near.cuh): impacts in
//                 order, rounds of 256 candidates tested in parallel, the
//                 first valid ones in candidate order kept, then sorted in
//                 (x, y, z) order (the reference's std::set) and labelled
#include <cfloat>

#include "vf.h"
#include "vf_kernels.h"
#include "vf_near.cuh"

namespace {

constexpr uint32_t EMPTY = 0u;

__device__ __forceinline__ uint16_t gat(const vfk::ImpactGrid& G, uint32_t x, uint32_t y, uint32_t z) {
  return G.g[((uint64_t)x * G.Y + y) * G.Zp + z];
}

__device__ bool ray_box(const float o[3], const float d[3], const float mn[3], const float mx[3],
                        float& tmin, float& tmax) {
  float tMin, tMax, tYMin, tYMax, tZMin, tZMax;
  const float xi = __fdiv_rn(1.0f, d[0]);
  if (xi >= 0) {
    tMin = __fmul_rn(__fsub_rn(mn[0], o[0]), xi);
    tMax = __fmul_rn(__fsub_rn(mx[0], o[0]), xi);
  } else {
    tMin = __fmul_rn(__fsub_rn(mx[0], o[0]), xi);
    tMax = __fmul_rn(__fsub_rn(mn[0], o[0]), xi);
  }
  const float yi = __fdiv_rn(1.0f, d[1]);
  if (yi >= 0) {
    tYMin = __fmul_rn(__fsub_rn(mn[1], o[1]), yi);
    tYMax = __fmul_rn(__fsub_rn(mx[1], o[1]), yi);
  } else {
    tYMin = __fmul_rn(__fsub_rn(mx[1], o[1]), yi);
    tYMax = __fmul_rn(__fsub_rn(mn[1], o[1]), yi);
  }
  if (tMin > tYMax || tYMin > tMax) return false;
  if (tYMin > tMin) tMin = tYMin;
  if (tYMax < tMax) tMax = tYMax;
  const float zi = __fdiv_rn(1.0f, d[2]);
  if (zi >= 0) {
    tZMin = __fmul_rn(__fsub_rn(mn[2], o[2]), zi);
    tZMax = __fmul_rn(__fsub_rn(mx[2], o[2]), zi);
  } else {
    tZMin = __fmul_rn(__fsub_rn(mx[2], o[2]), zi);
    tZMax = __fmul_rn(__fsub_rn(mn[2], o[2]), zi);
  }
  if (tMin > tZMax || tZMin > tMax) return false;
  if (tZMin > tMin) tMin = tZMin;
  if (tZMax < tMax) tMax = tZMax;
  tmin = tMin;
  tmax = tMax;
  return tMin < FLT_MAX && tMax > 0.0f;
}

// occupancy bits (label != EMPTY) of grid row r: word r * Zw + z / 32, and one
// bit per cell of 2^shift voxels a side that holds an occupied one (x slowest).
// A warp takes a row, a lane 8 labels of it at a time (the row padding is EMPTY).
__global__ void __launch_bounds__(256) k_occ_bits(vfk::ImpactGrid G, uint32_t Zw, uint32_t* bits,
                                                  vfk::RayCells C, uint32_t* cells, uint32_t* state) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    state[0] = 0;            // rays taken
    state[1] = 0xFFFFFFFFu;  // lowest ray without a direction
  }
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t span = C.shift < 8 ? 1u << (C.shift - 3) : 32u;  // lanes to a cell
  const uint64_t rows = (uint64_t)G.X * G.Y;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
    const uint16_t* row = G.g + r * G.Zp;
    const uint32_t x = (uint32_t)r / G.Y, y = (uint32_t)r - x * G.Y;
    const uint32_t cell0 = ((x >> C.shift) * C.ny + (y >> C.shift)) * C.nz;
    for (uint32_t z0 = 0; z0 < G.Z; z0 += 256) {
      const uint32_t z = z0 + 8 * lane;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (z < G.Zp) v = *reinterpret_cast<const uint4*>(row + z);
      auto two = [](uint32_t w) { return ((w & 0xFFFFu) ? 1u : 0u) | ((w >> 16) ? 2u : 0u); };
      const uint32_t b = two(v.x) | two(v.y) << 2 | two(v.z) << 4 | two(v.w) << 6;
      uint32_t word = b << (8 * (lane & 3));
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
      if ((lane & 3) == 0 && z < G.Z) bits[r * Zw + (z >> 5)] = word;
      const unsigned any = __ballot_sync(0xFFFFFFFFu, b != 0);
      if ((lane & (span - 1)) == 0 && ((any >> lane) & (0xFFFFFFFFu >> (32 - span)))) {
        const uint32_t cell = cell0 + (z >> C.shift), bit = 1u << (cell & 31);
        // 64 rows and more share a cell: most find it set
        if (!(__ldcg(cells + (cell >> 5)) & bit)) atomicOr(cells + (cell >> 5), bit);
      }
    }
  }
}

// the walk of a ray through the voxels, in the reference's float steps
struct RayWalk {
  uint32_t cur[3], step[3];  // cur: 0-based; past the grid either way is >= the dims
  float tNext[3], tDelta[3];
  // false: no direction, or the ray misses the grid's box
  __device__ bool begin(const vfk::ImpactGrid& G, const float o[3], const float d[3], bool none) {
    float tMin = 0.0f, tMax = 0.0f;
    if (none || !ray_box(o, d, G.amin, G.amax, tMin, tMax)) return false;
    if (tMin < 0.0f) tMin = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float start = __fadd_rn(o[a], __fmul_rn(d[a], tMin));
      const float c = ceilf(__fdiv_rn(__fsub_rn(start, G.amin[a]), G.cell[a]));
      cur[a] = (uint32_t)(c > 1.0f ? c : 1.0f) - 1u;
      // the plane ahead
      const float plane =
          __fadd_rn(G.amin[a], __fmul_rn((float)(d[a] > 0.0f ? cur[a] + 1u : cur[a]), G.cell[a]));
      if (d[a] > 0.0f || d[a] < 0.0f) {
        step[a] = d[a] > 0.0f ? 1u : 0xFFFFFFFFu;
        tDelta[a] = __fdiv_rn(G.cell[a], d[a] > 0.0f ? d[a] : -d[a]);
        tNext[a] = __fadd_rn(tMin, __fdiv_rn(__fsub_rn(plane, start), d[a]));
      } else {
        step[a] = 0u;
        tDelta[a] = FLT_MAX;
        tNext[a] = FLT_MAX;
      }
    }
    return true;
  }
  __device__ bool inside(const vfk::ImpactGrid& G) const { return cur[0] < G.X && cur[1] < G.Y && cur[2] < G.Z; }
  __device__ void advance() {
    const bool ax = tNext[0] < tNext[1] && tNext[0] < tNext[2], ay = !ax && tNext[1] < tNext[2];
    const bool go[3] = {ax, ay, !ax && !ay};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      cur[a] += go[a] ? step[a] : 0u;
      tNext[a] = go[a] ? __fadd_rn(tNext[a], tDelta[a]) : tNext[a];
    }
  }
};
__device__ __forceinline__ uint32_t walk_limit(const vfk::ImpactGrid& G) { return G.X + G.Y + G.Z + 3; }
__device__ __forceinline__ bool ray_load(const float* rays, uint32_t r, float o[3], float d[3]) {
  const float2* ray = reinterpret_cast<const float2*>(rays + 6 * (size_t)r);
  const float2 r0 = ray[0], r1 = ray[1], r2 = ray[2];
  o[0] = r0.x; o[1] = r0.y; o[2] = r1.x;
  d[0] = r1.y; d[1] = r2.x; d[2] = r2.y;
  return d[0] == 0.0f && d[1] == 0.0f && d[2] == 0.0f;
}

// few rays: one per lane, on the labels
__global__ void __launch_bounds__(256) k_ray_labels(vfk::ImpactGrid G, const float* rays, uint32_t n, uint32_t* out) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  float o[3], d[3];
  const bool none = ray_load(rays, r, o, d);
  uint32_t res[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
  RayWalk W;
  if (W.begin(G, o, d, none))
    for (uint32_t it = 0; it < walk_limit(G) && W.inside(G); ++it) {
      if (gat(G, W.cur[0], W.cur[1], W.cur[2]) != EMPTY) {
#pragma unroll
        for (int a = 0; a < 3; ++a) res[a] = W.cur[a] + 1u;
        break;
      }
      W.advance();
    }
#pragma unroll
  for (int a = 0; a < 3; ++a) out[3 * (size_t)r + a] = res[a];
}

// A ray's voxels are visited one after another, about 25 instructions each; rays
// take few or hundreds.  Bound by instruction issue, so lanes that are done get new
// rays as soon as RAY_IDLE of the warp are (state[0] deals them out), and a step
// looks up the cells in shared memory and, in an occupied cell, the bits in L2:
// 2^20 rays through 240 x 239 x 256 voxels 470 us, against 1166 us with a ray per
// thread at a time and a step on the bits in L2 (742 us with the cells alone).
// state[1]: the lowest ray of direction 0, which the caller refuses.
constexpr int RAY_IDLE = 12, RAY_STEPS = 4;
__global__ void __launch_bounds__(256) k_ray_entry(vfk::ImpactGrid G, uint32_t Zw, const uint32_t* bits, vfk::RayCells C,
                                                   const uint32_t* cells, const float* rays, uint32_t n,
                                                   uint32_t* out, uint32_t* state) {
  extern __shared__ uint32_t occupied[];
  for (uint32_t i = threadIdx.x; i < C.words; i += blockDim.x) occupied[i] = cells[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint32_t r = 0, left = 0;  // the lane's ray, and its steps left (0: none)
  RayWalk W;
  bool more = true;  // uniform: rays may be left
  auto store = [&](uint32_t a, uint32_t b, uint32_t c) {
    out[3 * (size_t)r + 0] = a;
    out[3 * (size_t)r + 1] = b;
    out[3 * (size_t)r + 2] = c;
  };
  for (;;) {
    const unsigned done = __ballot_sync(0xFFFFFFFFu, left == 0);
    if (more && (__popc(done) >= RAY_IDLE)) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&state[0], (uint32_t)__popc(done));
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      more = base < n && n - base > (uint32_t)__popc(done);
      base += __popc(done & ((1u << lane) - 1u));
      if (left == 0 && base < n) {
        r = base;
        float o[3], d[3];
        const bool none = ray_load(rays, r, o, d);
        if (none) atomicMin(&state[1], r);
        if (W.begin(G, o, d, none)) left = walk_limit(G) + 1;
        else store(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
      }
      continue;
    }
    if (done == 0xFFFFFFFFu) break;
#pragma unroll 1
    for (int k = 0; k < RAY_STEPS; ++k) {
      if (left == 0) continue;
      if (--left == 0 || !W.inside(G)) {
        left = 0;
        store(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        continue;
      }
      const uint32_t x = W.cur[0], y = W.cur[1], z = W.cur[2];
      const uint32_t cell = ((x >> C.shift) * C.ny + (y >> C.shift)) * C.nz + (z >> C.shift);
      if (((occupied[cell >> 5] >> (cell & 31u)) & 1u) &&
          ((__ldg(bits + ((uint64_t)x * G.Y + y) * Zw + (z >> 5)) >> (z & 31u)) & 1u)) {
        left = 0;
        store(x + 1u, y + 1u, z + 1u);
        continue;
      }
      W.advance();
    }
  }
}

struct ImpactView {
  const vfk::ImpactGrid& G;
  __device__ bool occupied(uint32_t x, uint32_t y, uint32_t z) const { return gat(G, x, y, z) != EMPTY; }
  // RegularGrid::isBoundary(x, y, z, 1) (RegularGrid.cpp:543-559)
  __device__ bool boundary(uint32_t x, uint32_t y, uint32_t z) const {
    const int lo0 = max((int)x - 1, 0), lo1 = max((int)y - 1, 0), lo2 = max((int)z - 1, 0);
    const int hi0 = min((int)x + 1, (int)G.X - 1), hi1 = min((int)y + 1, (int)G.Y - 1),
              hi2 = min((int)z + 1, (int)G.Z - 1);
    for (int i = lo0; i <= hi0; ++i)
      for (int j = lo1; j <= hi1; ++j)
        for (int k = lo2; k <= hi2; ++k)
          if (gat(G, (uint32_t)i, (uint32_t)j, (uint32_t)k) == EMPTY) return true;
    return false;
  }
};

// status[0] = count placed, status[1] = 0 or VF_ERR_SEED_SEARCH
__global__ void __launch_bounds__(256) k_near_seeds(vfk::ImpactGrid G, const uint32_t* frags,
                                                    uint32_t nfrags, uint32_t num_impacts,
                                                    uint32_t num_seeds, uint32_t spreading,
                                                    uint64_t seed, uint32_t label0, uint32_t* out,
                                                    uint32_t* status) {
  __shared__ unsigned long long cand[256];
  __shared__ unsigned long long acc[4096];
  __shared__ uint32_t cnt;
  const int n = vfnear::place(ImpactView{G}, G.X, G.Y, G.Z, frags, nfrags, num_impacts, num_seeds,
                              spreading, seed, label0, cand, acc, &cnt, out);
  if (threadIdx.x == 0) {
    status[0] = n < 0 ? 0u : (uint32_t)n;
    status[1] = n < 0 ? (uint32_t)VF_ERR_SEED_SEARCH : 0u;
  }
}

}  // namespace

namespace vfk {

RayCells ray_cells(uint32_t X, uint32_t Y, uint32_t Z) {
  // the smallest cells whose bits fit 32 KiB of shared memory, of 8 voxels or more
  RayCells C;
  for (C.shift = 3;; ++C.shift) {
    const uint32_t m = (1u << C.shift) - 1u;
    const uint64_t nx = (X + m) >> C.shift;
    C.ny = (Y + m) >> C.shift;
    C.nz = (Z + m) >> C.shift;
    const uint64_t words = (nx * C.ny * C.nz + 31) / 32;
    if (words <= 8192) {
      C.words = (uint32_t)words;
      return C;
    }
  }
}

cudaError_t ray_entry(cudaStream_t st, const ImpactGrid& G, const float* rays, uint32_t n, uint32_t* out,
                      uint32_t* bits, const RayCells& C, uint32_t* state, int num_sms) {
  if (!n) return cudaSuccess;
  if (bits) {
    const uint32_t Zw = (G.Z + 31) / 32;
    const uint64_t rows = (uint64_t)G.X * G.Y;
    const int bb = (int)std::max<uint64_t>(1, std::min<uint64_t>((rows * 32 + 255) / 256, (uint64_t)num_sms * 8));
    uint32_t* const cells = bits + rows * Zw;
    const cudaError_t e = cudaMemsetAsync(cells, 0, (size_t)C.words * 4, st);
    if (e != cudaSuccess) return e;
    k_occ_bits<<<bb, 256, 0, st>>>(G, Zw, bits, C, cells, state);
    // enough warps to issue every cycle; fewer give each more rays
    k_ray_entry<<<std::min<uint32_t>((n + 255) / 256, (uint32_t)num_sms * 6), 256, C.words * 4, st>>>(
        G, Zw, bits, C, cells, rays, n, out, state);
  } else {
    k_ray_labels<<<(n + 255) / 256, 256, 0, st>>>(G, rays, n, out);
  }
  return cudaGetLastError();
}

void near_seeds(cudaStream_t st, const ImpactGrid& G, const uint32_t* frags, uint32_t nfrags,
                uint32_t num_impacts, uint32_t num_seeds, uint32_t spreading, uint64_t seed,
                uint32_t label0, uint32_t* out, uint32_t* status) {
  k_near_seeds<<<1, 256, 0, st>>>(G, frags, nfrags, num_impacts, num_seeds, spreading, seed, label0,
                                  out, status);
}

}  // namespace vfk
