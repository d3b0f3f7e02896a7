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
//   k_ray_entry   a lane per ray, refilled: the reference's slab test and
//                 Amanatides-Woo walk in its operation order (every float
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
// bit per cell of 2^shift voxels a side that holds an occupied one (x slowest)
__global__ void __launch_bounds__(256) k_occ_bits(vfk::ImpactGrid G, uint32_t Zw, uint32_t* bits,
                                                  vfk::RayCells C, uint32_t* cells, uint32_t* state) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    state[0] = 0;            // rays taken
    state[1] = 0xFFFFFFFFu;  // lowest ray without a direction
  }
  const int lane = threadIdx.x & 31;
  const uint64_t rows = (uint64_t)G.X * G.Y;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
    const uint16_t* row = G.g + r * G.Zp;
    const uint32_t cell0 = ((uint32_t)(r / G.Y) >> C.shift) * C.ny * C.nz + ((uint32_t)(r % G.Y) >> C.shift) * C.nz;
    for (uint32_t z0 = 0; z0 < G.Z; z0 += 32) {
      const uint32_t z = z0 + lane;
      const unsigned m = __ballot_sync(0xFFFFFFFFu, z < G.Z && row[z] != EMPTY);
      if (lane == 0) bits[r * Zw + (z0 >> 5)] = m;
      // the first lane of each cell
      const uint32_t span = C.shift < 5 ? 1u << C.shift : 32u;
      if ((lane & (span - 1)) == 0 && (m >> lane) & (0xFFFFFFFFu >> (32 - span))) {
        const uint32_t cell = cell0 + (z >> C.shift);
        atomicOr(cells + (cell >> 5), 1u << (cell & 31));
      }
    }
  }
}

// Occupancy of a voxel: from the label grid, or (many rays) from the cells in
// shared memory and, in an occupied cell, the packed bits, which stay in L2.
struct LabelOcc {
  const vfk::ImpactGrid& G;
  __device__ void stage(uint32_t*) {}
  __device__ bool operator()(uint32_t x, uint32_t y, uint32_t z) const { return gat(G, x, y, z) != EMPTY; }
};
struct BitOcc {
  const uint32_t* bits;
  uint32_t Y, Zw;
  vfk::RayCells C;
  const uint32_t* cells;
  const uint32_t* staged;
  __device__ void stage(uint32_t* smem) {
    for (uint32_t i = threadIdx.x; i < C.words; i += blockDim.x) smem[i] = cells[i];
    __syncthreads();
    staged = smem;
  }
  __device__ bool operator()(uint32_t x, uint32_t y, uint32_t z) const {
    const uint32_t cell = ((x >> C.shift) * C.ny + (y >> C.shift)) * C.nz + (z >> C.shift);
    if (!((staged[cell >> 5] >> (cell & 31u)) & 1u)) return false;
    return (__ldg(bits + ((uint64_t)x * Y + y) * Zw + (z >> 5)) >> (z & 31u)) & 1u;
  }
};

// A ray's voxels are visited one after another in the reference's float steps,
// about 25 instructions each; rays take few or hundreds.  Bound by instruction
// issue, so lanes that are done get new rays as soon as RAY_IDLE of the warp
// are (state[0] deals them out), and a step's look-up is a shared memory load:
// 2^20 rays through 240 x 239 x 256 voxels 480 us, against 1166 us with a ray per
// thread at a time and a step on the bits in L2 (742 us with the cells alone).
// Without state (few rays) every lane takes its own rays.  state[1]: the lowest
// ray of direction 0, which the caller refuses.
constexpr int RAY_IDLE = 12, RAY_STEPS = 4;
template <typename Occ>
__global__ void __launch_bounds__(256) k_ray_entry(vfk::ImpactGrid G, Occ occ, const float* rays, uint32_t n,
                                                   uint32_t* out, uint32_t* state) {
  extern __shared__ uint32_t smem_cells[];
  occ.stage(smem_cells);
  const int lane = threadIdx.x & 31;
  const uint32_t dims[3] = {G.X, G.Y, G.Z};
  uint32_t own = blockIdx.x * blockDim.x + threadIdx.x;  // the next ray of the lane, without state
  uint32_t r = 0, left = 0;                              // the lane's ray, and its steps left (0: none)
  uint32_t cur[3] = {0, 0, 0}, step[3] = {0, 0, 0};      // cur: 0-based; past the grid either way is >= dims
  float tNext[3] = {0.0f, 0.0f, 0.0f}, tDelta[3] = {0.0f, 0.0f, 0.0f};
  bool more = true;  // with state: rays may be left
  auto store = [&](uint32_t a, uint32_t b, uint32_t c) {
    out[3 * (size_t)r + 0] = a;
    out[3 * (size_t)r + 1] = b;
    out[3 * (size_t)r + 2] = c;
  };
  for (;;) {
    // done lanes, and those a ray may be left for
    const unsigned done = __ballot_sync(0xFFFFFFFFu, left == 0);
    const unsigned idle = state ? (more ? done : 0u) : __ballot_sync(0xFFFFFFFFu, left == 0 && own < n);
    if (__popc(idle) >= RAY_IDLE || (idle && done == 0xFFFFFFFFu)) {
      uint32_t base = own;
      if (state) {
        if (lane == 0) base = atomicAdd(&state[0], (uint32_t)__popc(idle));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        more = base < n && n - base > (uint32_t)__popc(idle);
        base += __popc(idle & ((1u << lane) - 1u));
      } else {
        if (left == 0 && own < n) own = n - own > gridDim.x * blockDim.x ? own + gridDim.x * blockDim.x : n;
      }
      if (left == 0 && base < n) {
        r = base;
        const float2* ray = reinterpret_cast<const float2*>(rays + 6 * (size_t)r);
        const float2 r0 = ray[0], r1 = ray[1], r2 = ray[2];
        const float o[3] = {r0.x, r0.y, r1.x};
        const float d[3] = {r1.y, r2.x, r2.y};
        float tMin = 0.0f, tMax = 0.0f;
        const bool none = d[0] == 0.0f && d[1] == 0.0f && d[2] == 0.0f;
        if (none && state) atomicMin(&state[1], r);
        if (!none && ray_box(o, d, G.amin, G.amax, tMin, tMax)) {
          if (tMin < 0.0f) tMin = 0.0f;
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const float start = __fadd_rn(o[a], __fmul_rn(d[a], tMin));
            const float c = ceilf(__fdiv_rn(__fsub_rn(start, G.amin[a]), G.cell[a]));
            cur[a] = (uint32_t)(c > 1.0f ? c : 1.0f) - 1u;
            // the plane ahead: of cell cur + 1 (1-based cur) or cur - 1
            const float plane = __fadd_rn(
                G.amin[a], __fmul_rn((float)(d[a] > 0.0f ? cur[a] + 1u : cur[a]), G.cell[a]));
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
          left = dims[0] + dims[1] + dims[2] + 4;
        } else {
          store(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        }
      }
      continue;
    }
    if (done == 0xFFFFFFFFu) break;
#pragma unroll 1
    for (int k = 0; k < RAY_STEPS; ++k) {
      if (left == 0) continue;
      if (--left == 0 || cur[0] >= dims[0] || cur[1] >= dims[1] || cur[2] >= dims[2]) {
        left = 0;
        store(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
      } else if (occ(cur[0], cur[1], cur[2])) {
        left = 0;
        store(cur[0] + 1u, cur[1] + 1u, cur[2] + 1u);
      } else {
        const bool ax = tNext[0] < tNext[1] && tNext[0] < tNext[2], ay = !ax && tNext[1] < tNext[2];
        const bool go[3] = {ax, ay, !ax && !ay};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          cur[a] += go[a] ? step[a] : 0u;
          tNext[a] = go[a] ? __fadd_rn(tNext[a], tDelta[a]) : tNext[a];
        }
      }
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
  const int blocks = (int)std::min<uint32_t>((n + 255) / 256, (uint32_t)num_sms * 8);
  if (bits) {
    const uint32_t Zw = (G.Z + 31) / 32;
    const uint64_t rows = (uint64_t)G.X * G.Y;
    const int bb = (int)std::max<uint64_t>(1, std::min<uint64_t>((rows * 32 + 255) / 256, (uint64_t)num_sms * 8));
    uint32_t* const cells = bits + rows * Zw;
    cudaError_t e = cudaMemsetAsync(cells, 0, (size_t)C.words * 4, st);
    if (e != cudaSuccess) return e;
    k_occ_bits<<<bb, 256, 0, st>>>(G, Zw, bits, C, cells, state);
    // enough warps to issue every cycle; fewer give each more rays
    k_ray_entry<<<std::min(blocks, num_sms * 6), 256, C.words * 4, st>>>(G, BitOcc{bits, G.Y, Zw, C, cells, nullptr},
                                                                         rays, n, out, state);
  } else {
    k_ray_entry<<<blocks, 256, 0, st>>>(G, LabelOcc{G}, rays, n, out, nullptr);
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
