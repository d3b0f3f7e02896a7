// vf_gridops.cu -- seeding, naive Voronoi, perturbation, boundary detection,
// erosion, isolated-voxel removal and per-fragment counts on sm_103a.
//
// Brick kernels: one CTA (256 threads) per live brick of 16 x 16 rows of VF_BZ = 32
// voxels.  A stencil stages the brick with an xy halo of H voxels and a z window
// [z0-8, z0+40) in shared memory with 16-byte loads (rows are 16-byte aligned
// because Zp % 8 == 0); boundaries of size 1 keep their units of 8 voxels in
// registers, the others stage the rows alone.  The voxels that have work are dealt
// to the threads from a queue (units of 8 for boundaries of size 1).  Results go
// back as 16-byte stores of whole units (padding z >= Z written as 0).  Halo voxels
// outside the grid read as EMPTY; voxels of bricks that are not live are EMPTY in
// memory (both grid buffers start as the voxelizer output).
//
// The CTAs of a launch loop over the live-brick list (its length is read on
// the device, so launches need no host synchronisation).
#include <algorithm>

#include "vf_kernels.h"
#include "vf_near.cuh"

#include <cfloat>

namespace {

constexpr int ZW = VF_BZ + 16;  // z window of a staged tile (u16)

template <int H>
struct Tile {
  static constexpr int NX = VF_BX + 2 * H, NY = VF_BY + 2 * H;
  static constexpr int ROWS = NX * NY;
  static constexpr int BYTES = ROWS * ZW * 2;
};

__device__ __forceinline__ void brick_coords(const JobDesc& J, uint32_t b, uint32_t& x0,
                                             uint32_t& y0, uint32_t& z0) {
  const uint32_t lb = b - J.brick_base;
  const uint32_t bz = lb % J.nbz, by = (lb / J.nbz) % J.nby, bx = lb / (J.nbz * J.nby);
  x0 = bx * VF_BX;
  y0 = by * VF_BY;
  z0 = bz * VF_BZ;
}

// stage src rows [x0-H, x0+16+H) x [y0-H, y0+16+H) x [z0-8, z0+40) into tile
template <int H>
__device__ __forceinline__ void load_tile(const JobDesc& J, const uint16_t* src, uint32_t x0,
                                          uint32_t y0, uint32_t z0, uint16_t* tile) {
  using T = Tile<H>;
  uint4* t4 = reinterpret_cast<uint4*>(tile);
  constexpr int PER_ROW = ZW / 8;
  for (int q = threadIdx.x; q < T::ROWS * PER_ROW; q += blockDim.x) {
    const int row = q / PER_ROW, part = q % PER_ROW;
    const int x = (int)x0 - H + row / T::NY, y = (int)y0 - H + row % T::NY;
    const int z = (int)z0 - 8 + part * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (x >= 0 && y >= 0 && z >= 0 && x < (int)J.X && y < (int)J.Y && z < (int)J.Zp)
      v = __ldg(reinterpret_cast<const uint4*>(src + vf_gidx(J, x, y, z)));
    t4[q] = v;
  }
}
template <int H>
__device__ __forceinline__ uint16_t tval(const uint16_t* tile, int lx, int ly, int lz) {
  // lx, ly in [-H, 16+H), lz in [-8, 40) relative to the brick origin
  return tile[((lx + H) * Tile<H>::NY + (ly + H)) * ZW + (lz + 8)];
}


// ===========================================================================
// Seeding: Seeder::uniform (Seeder.cpp:154-208) + mergeSeeds (:115-152).
// One 1024-thread block per job.  Attempts are evaluated 1024 at a time in
// parallel; warp 0 then accepts them in attempt order (duplicates skipped),
// which is exactly the sequential rejection loop of the reference.
__device__ __forceinline__ bool occupied_at(const JobDesc& J, int x, int y, int z) {
  return J.grid[vf_gidx(J, x, y, z)] != VOXEL_EMPTY;
}
__device__ bool is_boundary(const JobDesc& J, int x, int y, int z) {
  // RegularGrid::isBoundary(x,y,z,1) (RegularGrid.cpp:543-559)
  const int x0 = vf_clampi(x - 1, 0, J.X - 1), x1 = vf_clampi(x + 1, 0, J.X - 1);
  const int y0 = vf_clampi(y - 1, 0, J.Y - 1), y1 = vf_clampi(y + 1, 0, J.Y - 1);
  const int z0 = vf_clampi(z - 1, 0, J.Z - 1), z1 = vf_clampi(z + 1, 0, J.Z - 1);
  for (int a = x0; a <= x1; ++a)
    for (int b = y0; b <= y1; ++b)
      for (int c = z0; c <= z1; ++c)
        if (J.grid[vf_gidx(J, a, b, c)] == VOXEL_EMPTY) return true;
  return false;
}

struct SeedSmem {
  unsigned long long acc[4096];
  unsigned long long cand[1024];
  uint16_t near_[4096];
  uint32_t idf[256];
  uint32_t cnt;
  uint32_t fail;
};

// returns false on SeederSearchError; out receives n xyzw entries
__device__ bool uniform_block(const JobDesc& J, SeedSmem& S, uint32_t n, uint64_t seed,
                              int location, uint32_t* out) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) { S.cnt = 0; S.fail = 0; }
  __syncthreads();
  const float fx = (float)(J.X - 1), fy = (float)(J.Y - 1), fz = (float)(J.Z - 1);
  for (uint32_t base = 0;; base += 1024) {
    if (S.cnt >= n || S.fail) break;
    if (base >= VF_MAX_TRIES) { if (t == 0) S.fail = 1; __syncthreads(); break; }
    const uint32_t a = base + t;
    unsigned long long key = ~0ull;
    if (a < VF_MAX_TRIES) {
      const int x = (int)__fmul_rn(fx, vf_u01(vf_hash(seed, VF_STREAM_SEEDS, 3ull * a + 0)));
      const int y = (int)__fmul_rn(fy, vf_u01(vf_hash(seed, VF_STREAM_SEEDS, 3ull * a + 1)));
      const int z = (int)__fmul_rn(fz, vf_u01(vf_hash(seed, VF_STREAM_SEEDS, 3ull * a + 2)));
      bool ok = occupied_at(J, x, y, z);
      if (ok && location != 2) ok = ((location == 1) == is_boundary(J, x, y, z));
      if (ok) key = ((unsigned long long)x << 24) | ((unsigned long long)y << 12) | (unsigned long long)z;
    }
    S.cand[t] = key;
    __syncthreads();
    if (warp == 0) {
      // 32 attempts at a time, only the valid ones compared: 64 seeds in a hollow
      // 192 voxel model 23 us (62 us one attempt at a time)
      uint32_t cnt = S.cnt;
      for (int i0 = 0; i0 < 1024 && cnt < n; i0 += 32) {
        const unsigned long long mine = S.cand[i0 + lane];
        unsigned m = __ballot_sync(0xFFFFFFFFu, mine != ~0ull);
        for (; m && cnt < n; m &= m - 1) {
          const unsigned long long k = __shfl_sync(0xFFFFFFFFu, mine, __ffs(m) - 1);
          bool dup = false;
          for (uint32_t q = lane; q < cnt; q += 32) dup |= (S.acc[q] == k);
          dup = __any_sync(0xFFFFFFFFu, dup);
          if (!dup) {
            if (lane == 0) S.acc[cnt] = k;
            ++cnt;
          }
          __syncwarp();
        }
      }
      if (lane == 0) S.cnt = cnt;
    }
    __syncthreads();
  }
  __syncthreads();
  if (S.fail || S.cnt < n) return false;
  // sort lexicographically (std::set<uvec3>), bitonic over the next power of 2
  uint32_t P = 1;
  while (P < n) P <<= 1;
  for (uint32_t i = n + t; i < P; i += blockDim.x) S.acc[i] = ~0ull;
  __syncthreads();
  for (uint32_t k = 2; k <= P; k <<= 1)
    for (uint32_t jx = k >> 1; jx > 0; jx >>= 1) {
      for (uint32_t i = t; i < P; i += blockDim.x) {
        const uint32_t l = i ^ jx;
        if (l > i) {
          const unsigned long long a = S.acc[i], b = S.acc[l];
          const bool up = (i & k) == 0;
          if ((a > b) == up) { S.acc[i] = b; S.acc[l] = a; }
        }
      }
      __syncthreads();
    }
  for (uint32_t i = t; i < n; i += blockDim.x) {
    const unsigned long long k = S.acc[i];
    out[4 * i] = (uint32_t)(k >> 24);
    out[4 * i + 1] = (uint32_t)((k >> 12) & 0xFFF);
    out[4 * i + 2] = (uint32_t)(k & 0xFFF);
    out[4 * i + 3] = VOXEL_FREE + 1 + i;
  }
  __syncthreads();
  return true;
}

// Seeder::nearSeeds (vfnear::place) on the job's occupancy grid, after its nf
// main seeds in `seeds`: appends the placed seeds, labelled on from the last
// main seed; returns their count, or -1 when an impact runs out of candidates
struct JobGrid {
  const JobDesc& J;
  __device__ bool occupied(uint32_t x, uint32_t y, uint32_t z) const {
    return occupied_at(J, (int)x, (int)y, (int)z);
  }
  __device__ bool boundary(uint32_t x, uint32_t y, uint32_t z) const {
    return is_boundary(J, (int)x, (int)y, (int)z);
  }
};

__device__ int near_block(const JobDesc& J, SeedSmem& S, uint32_t* seeds, uint32_t nf) {
  return vfnear::place(JobGrid{J}, J.X, J.Y, J.Z, seeds, nf, (uint32_t)J.num_impacts,
                       (uint32_t)J.bias_seeds, (uint32_t)J.bias_focus, J.seed, seeds[4 * (nf - 1) + 3],
                       S.cand, S.acc, &S.cnt, seeds + 4 * (uint64_t)nf);
}

__device__ __forceinline__ float seed_dist(int dfunc, const uint32_t* s, const uint32_t* f) {
  const float dx = __fsub_rn((float)s[0], (float)f[0]), dy = __fsub_rn((float)s[1], (float)f[1]),
              dz = __fsub_rn((float)s[2], (float)f[2]);
  if (dfunc == 0)
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
  if (dfunc == 1) return __fadd_rn(__fadd_rn(fabsf(dx), fabsf(dy)), fabsf(dz));
  return fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz)));
}

__global__ void __launch_bounds__(1024) k_seeds(const JobDesc* jobs, JobState* st) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SeedSmem& S = *reinterpret_cast<SeedSmem*>(smem_raw);
  const JobDesc& J = jobs[blockIdx.x];
  JobState& js = st[blockIdx.x];
  const int t = threadIdx.x;
  if (!J.active) return;
  if (J.seeds_given) {
    if (t == 0) {
      js.nseeds = J.seeds_given;
      uint32_t hp = 0;
      for (uint32_t i = 0; i < J.seeds_given; ++i) hp |= J.seeds[4 * i + 3] > 0xFFu;
      js.has_prefix = hp;
    }
    return;
  }
  uint32_t nm = (uint32_t)J.num_seeds;
  const uint32_t ne = (uint32_t)J.num_extra;
  if (J.X < 2 || J.Y < 2 || J.Z < 2 || nm > 254 || 2 * nm + ne > J.seeds_cap) {
    if (t == 0) { js.err |= VF_JERR_INVALID; js.nseeds = 0; }
    return;
  }
  if (!uniform_block(J, S, nm, J.seed, J.seed_location, J.seeds)) {
    if (t == 0) { js.err |= VF_JERR_SEED_SEARCH; js.nseeds = 0; }
    return;
  }
  if (J.num_impacts > 0 && nm > 0 && J.bias_seeds > 0) {
    // CADScene.cpp:636-638: nearSeeds(seeds, numImpacts, biasSeeds, biasFocus)
    if (J.bias_focus < 1 || (uint32_t)J.bias_focus > min(J.X, min(J.Y, J.Z))) {
      if (t == 0) { js.err |= VF_JERR_INVALID; js.nseeds = 0; }
      return;
    }
    const int placed = near_block(J, S, J.seeds, nm);
    if (placed < 0) {
      if (t == 0) { js.err |= VF_JERR_SEED_SEARCH; js.nseeds = 0; }
      return;
    }
    nm += (uint32_t)placed;
    if (nm > 254) {  // 8-bit fragment ids 2..255
      if (t == 0) { js.err |= VF_JERR_RANGE; js.nseeds = 0; }
      return;
    }
  }
  uint32_t total = nm;
  if (ne > 0 && nm > 0) {
    // extraSeeds = uniform(BOTH) after a copy of the main seeds, merged
    // (CADScene.cpp:647-655); seed value seed + golden ratio
    uint32_t* list = J.seeds + 4 * (size_t)nm;
    for (uint32_t i = t; i < 4 * nm; i += blockDim.x) list[i] = J.seeds[i];
    __syncthreads();
    if (!uniform_block(J, S, ne, J.seed + 0x9E3779B97F4A7C15ull, 2, list + 4 * (size_t)nm)) {
      if (t == 0) { js.err |= VF_JERR_SEED_SEARCH; js.nseeds = 0; }
      return;
    }
    const uint32_t nl = nm + ne;
    for (uint32_t k = t; k < nl; k += blockDim.x) {
      float best = FLT_MAX;
      int nearest = 0;
      for (uint32_t i = 0; i < nm; ++i) {
        const float d = seed_dist(J.merge_distance, list + 4 * k, J.seeds + 4 * i);
        if (d < best) { best = d; nearest = (int)i; }
      }
      S.near_[k] = (uint16_t)nearest;
    }
    for (uint32_t i = t; i < 256; i += blockDim.x) S.idf[i] = 0;
    __syncthreads();
    if (t == 0) {
      for (uint32_t k = 0; k < nl; ++k) {
        const uint32_t w = J.seeds[4 * S.near_[k] + 3];
        const uint32_t pre = ++S.idf[w & 0xFFu];
        if (pre > 127) js.err |= VF_JERR_RANGE;
        list[4 * k + 3] = w | (pre << 8);
      }
    }
    total = 2 * nm + ne;
  }
  __syncthreads();
  if (t == 0) {
    js.nseeds = total;
    uint32_t hp = 0;
    for (uint32_t i = 0; i < total; ++i) hp |= J.seeds[4 * i + 3] > 0xFFu;
    js.has_prefix = hp;
  }
}

// ===========================================================================
// A brick's 256 label rows between global memory and shared memory (34-u16 row
// pitch: the u16 of one z from 32 threads falls on 32 distinct banks), 4 lanes
// per row along z; units at or past Zp are zero / not written.
constexpr int ROW_PITCH = VF_BZ + 2;
__device__ __forceinline__ void rows_in(const JobDesc& J, const uint16_t* src, uint32_t x0, uint32_t y0, uint32_t z0,
                                        uint16_t* rows) {
  const uint32_t nz = min((uint32_t)VF_BZ, J.Zp - z0);
  uint4 w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t u = i * 256 + threadIdx.x, row = u >> 2, q = u & 3;
    const uint32_t x = x0 + row / VF_BY, y = y0 + row % VF_BY;
    w[i] = (x < J.X && y < J.Y && 8 * q < nz) ? *reinterpret_cast<const uint4*>(src + vf_gidx(J, x, y, z0 + 8 * q))
                                              : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t u = i * 256 + threadIdx.x, row = u >> 2, q = u & 3;
    // 4-byte aligned: 68-byte row pitch, 16-byte units
    uint32_t* d = reinterpret_cast<uint32_t*>(rows + row * ROW_PITCH + 8 * q);
    d[0] = w[i].x; d[1] = w[i].y; d[2] = w[i].z; d[3] = w[i].w;
  }
}
__device__ __forceinline__ void rows_out(const JobDesc& J, uint16_t* dst, uint32_t x0, uint32_t y0, uint32_t z0,
                                         const uint16_t* rows) {
  const uint32_t nz = min((uint32_t)VF_BZ, J.Zp - z0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t u = i * 256 + threadIdx.x, row = u >> 2, q = u & 3;
    const uint32_t x = x0 + row / VF_BY, y = y0 + row % VF_BY;
    if (x < J.X && y < J.Y && 8 * q < nz) {
      const uint32_t* r = reinterpret_cast<const uint32_t*>(rows + row * ROW_PITCH + 8 * q);
      *reinterpret_cast<uint4*>(dst + vf_gidx(J, x, y, z0 + 8 * q)) = make_uint4(r[0], r[1], r[2], r[3]);
    }
  }
}
// bit z: voxel z of 32 (16 u16 pairs) is above `floor`
__device__ __forceinline__ uint32_t pair_bits(uint32_t w, uint32_t floor, int k) {
  const uint32_t g = __vsetgtu2(w, floor * 0x00010001u);
  return ((g | (g >> 15)) & 3u) << (2 * k);
}
__device__ __forceinline__ uint32_t voxels_above(const uint16_t* row /* 4-byte aligned */, uint32_t floor) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < VF_BZ / 2; ++k) m |= pair_bits(reinterpret_cast<const uint32_t*>(row)[k], floor, k);
  return m;
}
__device__ __forceinline__ uint32_t tile_voxels_above(const uint16_t* row /* 16-byte aligned */, uint32_t floor) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < VF_BZ / 8; ++k) {
    const uint4 w = reinterpret_cast<const uint4*>(row)[k];
    m |= pair_bits(w.x, floor, 4 * k) | pair_bits(w.y, floor, 4 * k + 1) | pair_bits(w.z, floor, 4 * k + 2) |
         pair_bits(w.w, floor, 4 * k + 3);
  }
  return m;
}
// The voxels of a brick chosen by m (bit z of the thread's row, row = thread), as
// row << 5 | z in row order, into vq (all 256 threads call it; wq: 8 words).
// The voxels of a thin wall are few and uneven per row: dealt from the queue
// they keep every lane busy.
__device__ __forceinline__ uint32_t queue_voxels(uint32_t m, uint16_t* vq, uint32_t* wq) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t c = (uint32_t)__popc(m);
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) wq[warp] = incl;
  __syncthreads();
  uint32_t base = incl - c, total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    base += w < warp ? wq[w] : 0u;
    total += wq[w];
  }
  while (m) {
    const uint32_t z = (uint32_t)__ffs(m) - 1;
    m &= m - 1;
    vq[base++] = (uint16_t)((t << 5) | z);
  }
  __syncthreads();
  return total;
}

// NaiveFracturer::buildCPU (NaiveFracturer.cpp:26-68): every occupied voxel
// takes the label of the nearest seed; strict '<' keeps the lowest index.
//
// Per brick, only the seeds that can be nearest to one of its voxels are
// compared: a seed is dropped when its distance to the brick's box exceeds the
// largest distance some other seed has to it.  The bounds are whole numbers
// (squares for VF_EUCLIDEAN); a 2^-18 margin on squares is far above the
// rounding of the float distances (2^-23), so a dropped seed never ties.  Seeds
// far outside every grid (no rule refuses them) are always compared.
// Bound by the distance arithmetic of the voxels left: 64 seeds on 180 x 179 x
// 192 voxels 25 us (531 us with every seed against all voxels of the rows).
constexpr uint32_t NAIVE_SEEDS = 256;  // compared per round, plus at most as many
constexpr uint32_t SEED_NEAR = 8192;  // twice the largest grid side; squares of coordinates below it add up in u32
__global__ void __launch_bounds__(256) k_naive(const JobDesc* jobs, const JobState* st,
                                               const uint32_t* list, const uint32_t* count,
                                               const uint32_t* brick_job) {
  __shared__ uint4 sd[2 * NAIVE_SEEDS];  // position, index
  __shared__ __align__(16) uint16_t rows[256 * ROW_PITCH];
  __shared__ uint16_t vq[256 * VF_BZ];
  __shared__ uint32_t wq[8], s_bound;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const uint32_t j = brick_job[b];
    const JobDesc& J = jobs[j];
    const uint32_t ns = st[j].nseeds;
    if (!J.active || ns == 0) continue;  // uniform across the CTA
    const uint4* const seeds = reinterpret_cast<const uint4*>(J.seeds);
    const int dist = J.distance;
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    __syncthreads();  // the previous brick is done with the shared arrays
    rows_in(J, J.grid, x0, y0, z0, rows);
    if (t == 0) s_bound = 0xFFFFFFFFu;
    __syncthreads();
    const uint32_t total = queue_voxels(voxels_above(rows + t * ROW_PITCH, VOXEL_EMPTY), vq, wq);
    // smallest (near) and largest (far) distance of a seed to the brick's voxels
    auto reach = [&](const uint4& sp, uint32_t& near, uint32_t& far) {
      const uint32_t p[3] = {sp.x, sp.y, sp.z}, lo[3] = {x0, y0, z0};
      const uint32_t hi[3] = {min(x0 + VF_BX, J.X) - 1, min(y0 + VF_BY, J.Y) - 1, min(z0 + VF_BZ, J.Z) - 1};
      near = 0;
      far = 0xFFFFFFFFu;
      if (max(max(sp.x, sp.y), sp.z) >= SEED_NEAR) return;
      far = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const uint32_t l = p[a] < lo[a] ? lo[a] - p[a] : (p[a] > hi[a] ? p[a] - hi[a] : 0u);
        const uint32_t f = max(p[a] > lo[a] ? p[a] - lo[a] : lo[a] - p[a], p[a] > hi[a] ? p[a] - hi[a] : hi[a] - p[a]);
        if (dist == 0) { near += l * l; far += f * f; }
        else if (dist == 1) { near += l; far += f; }
        else { near = max(near, l); far = max(far, f); }
      }
    };
    uint32_t bound = 0xFFFFFFFFu;
    for (uint32_t i = t; i < ns; i += 256) {
      uint32_t near, far;
      reach(seeds[i], near, far);
      bound = min(bound, far);
    }
    bound = __reduce_min_sync(0xFFFFFFFFu, bound);
    if (lane == 0) atomicMin(&s_bound, bound);
    __syncthreads();
    bound = s_bound;
    if (dist == 0 && bound != 0xFFFFFFFFu) bound += (bound >> 18) + 1;
    // From here a voxel's entry holds the index of its nearest seed so far.
    uint32_t kept = 0;
    bool first = true;
    for (uint32_t c0 = 0; c0 < ns; c0 += 256) {
      uint4 sp = make_uint4(0, 0, 0, 0);
      bool keep = false;
      if (c0 + t < ns) {
        sp = seeds[c0 + t];
        uint32_t near, far;
        reach(sp, near, far);
        keep = near <= bound;
      }
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, keep);
      if (lane == 0) wq[warp] = (uint32_t)__popc(m);
      __syncthreads();
      uint32_t at = kept + (uint32_t)__popc(m & ((1u << lane) - 1u));
#pragma unroll
      for (uint32_t w = 0; w < 8; ++w) {
        at += w < warp ? wq[w] : 0u;
        kept += wq[w];
      }
      if (keep) sd[at] = make_uint4(sp.x, sp.y, sp.z, c0 + t);
      __syncthreads();
      if (kept < NAIVE_SEEDS && c0 + 256 < ns) continue;  // room for another 256
      for (uint32_t i = t; i < total; i += 256) {
        const uint32_t e = vq[i], row = e >> 5, z = e & 31u;
        const int x = (int)(x0 + row / VF_BY), y = (int)(y0 + row % VF_BY), gz = (int)(z0 + z);
        uint16_t* const v = rows + row * ROW_PITCH + z;
        uint32_t lead = first ? 0u : *v;
        if (dist == 0) {
          // the square root keeps the order, so only a smaller square can be a
          // smaller distance; equal roots of unequal squares go to the lower index
          float best = FLT_MAX, best2 = FLT_MAX;
          auto square = [&](const uint4& q) {
            const float fx = (float)(x - (int)q.x), fy = (float)(y - (int)q.y), fz = (float)(gz - (int)q.z);
            return __fadd_rn(__fadd_rn(__fmul_rn(fx, fx), __fmul_rn(fy, fy)), __fmul_rn(fz, fz));
          };
          if (!first) {
            best2 = square(seeds[lead]);
            best = __fsqrt_rn(best2);
          }
          for (uint32_t k = 0; k < kept; ++k) {
            const uint4 q = sd[k];
            const float d2 = square(q);
            if (d2 < best2) {
              const float d = __fsqrt_rn(d2);
              if (d < best) { best = d; best2 = d2; lead = q.w; }
            }
          }
        } else {
          auto steps = [&](const uint4& q) {
            const int dx = abs(x - (int)q.x), dy = abs(y - (int)q.y), dz = abs(gz - (int)q.z);
            return (float)(dist == 1 ? dx + dy + dz : max(dx, max(dy, dz)));
          };
          float best = first ? FLT_MAX : steps(seeds[lead]);
          for (uint32_t k = 0; k < kept; ++k) {
            const uint4 q = sd[k];
            const float d = steps(q);
            if (d < best) { best = d; lead = q.w; }
          }
        }
        *v = (uint16_t)lead;
      }
      kept = 0;
      first = false;
      __syncthreads();
    }
    for (uint32_t i = t; i < total; i += 256) {
      const uint32_t e = vq[i];
      uint16_t* const v = rows + (e >> 5) * ROW_PITCH + (e & 31u);
      *v = (uint16_t)seeds[*v].w;
    }
    __syncthreads();
    rows_out(J, J.grid, x0, y0, z0, rows);
  }
}

// ===========================================================================
// Boundary perturbation (no reference counterpart).  Lattice values are
// precomputed per job; per voxel the 3-channel trilinear noise gives the
// offset of the voxel whose label is taken.  Reads src, writes dst.
__global__ void k_lattice(const JobDesc* jobs) {
  const JobDesc& J = jobs[blockIdx.y];
  if (!J.active) return;
  const uint32_t n = J.lat_nx * J.lat_ny * J.lat_nz * 3;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t c = i % 3, p = i / 3;
    const uint32_t iz = p % J.lat_nz, iy = (p / J.lat_nz) % J.lat_ny, ix = p / (J.lat_nz * J.lat_ny);
    const uint64_t ctr = (((uint64_t)ix << 40) | ((uint64_t)iy << 20) | iz) * 4u + c;
    J.lattice[i] = __fsub_rn(__fmul_rn(vf_u01(vf_hash(J.seed, VF_STREAM_NOISE, ctr)), 2.0f), 1.0f);
  }
}

__device__ __forceinline__ float lerp_(float a, float b, float t) {
  return __fadd_rn(a, __fmul_rn(t, __fsub_rn(b, a)));
}

// The noise of a brick's voxels: where at most PERT_COLS lattice columns reach the
// brick (periods of 6 and more), their values at the brick's 32 z, taken along z
// first as the oracle does, are tabled once, and a voxel is left with two lerps
// per channel in y and one in x; else a voxel reads its 8 lattice points.
// Bound by the voxels' arithmetic and their gathers: 476 x 476 x 512 voxels, period
// 16, 118 us (156 us with 24 lattice loads a voxel).
constexpr uint32_t PERT_COLS = 25;
__global__ void __launch_bounds__(256) k_perturb(const JobDesc* jobs, const uint32_t* list,
                                                 const uint32_t* count, const uint32_t* brick_job) {
  // per brick: the lattice index and in-cell coordinate of its 16 x, 16 y
  // and 32 z values, t = (c mod P) / P rounded as the oracle divides
  __shared__ float t0s[VF_BX], t1s[VF_BY], t2s[VF_BZ];
  __shared__ uint32_t i0s[VF_BX], i1s[VF_BY], i2s[VF_BZ];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* const table = reinterpret_cast<float4*>(smem_raw);  // [column][z]
  uint16_t* const vrows = reinterpret_cast<uint16_t*>(table + PERT_COLS * VF_BZ);
  uint16_t* const vq = vrows + 256 * ROW_PITCH;
  __shared__ uint32_t wq[8];
  const int t = threadIdx.x;
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const JobDesc& J = jobs[brick_job[b]];
    if (!J.active) continue;  // uniform across the CTA
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    const uint32_t P = J.noise_period;
    const float fp = (float)P;
    __syncthreads();  // the previous brick is done with the tables, rows and queue
    if (t < VF_BZ) {
      const uint32_t gz = z0 + t;
      t2s[t] = __fdiv_rn((float)(gz % P), fp);
      i2s[t] = gz / P;
    } else if (t < VF_BZ + VF_BX) {
      const uint32_t gx = x0 + (t - VF_BZ);
      t0s[t - VF_BZ] = __fdiv_rn((float)(gx % P), fp);
      i0s[t - VF_BZ] = gx / P;
    } else if (t < VF_BZ + VF_BX + VF_BY) {
      const uint32_t gy = y0 + (t - VF_BZ - VF_BX);
      t1s[t - VF_BZ - VF_BX] = __fdiv_rn((float)(gy % P), fp);
      i1s[t - VF_BZ - VF_BX] = gy / P;
    }
    const uint16_t* src = J.grid;
    rows_in(J, src, x0, y0, z0, vrows);
    __syncthreads();
    const uint32_t sy = J.lat_nz * 3, sx = J.lat_ny * sy;
    // the lattice columns from (x0 / P, y0 / P) to past the brick's last voxel
    // inside the grid
    const uint32_t cx = i0s[0], cy = i1s[0];
    const uint32_t nx = (min(x0 + VF_BX, J.X) - 1) / P + 2 - cx, ny = (min(y0 + VF_BY, J.Y) - 1) / P + 2 - cy;
    const bool tabled = nx * ny <= PERT_COLS;
    if (tabled)
      for (uint32_t i = t; i < nx * ny * VF_BZ; i += 256) {
        const uint32_t col = i / VF_BZ, z = i % VF_BZ;
        if (z0 + z >= J.Z) continue;
        const float* L = J.lattice + (size_t)(cx + col / ny) * sx + (size_t)(cy + col % ny) * sy + (size_t)i2s[z] * 3;
        const float t2 = t2s[z];
        table[i] = make_float4(lerp_(L[0], L[3], t2), lerp_(L[1], L[4], t2), lerp_(L[2], L[5], t2), 0.0f);
      }
    // (the queue's barriers separate the table from its readers)
    const uint32_t total = queue_voxels(voxels_above(vrows + t * ROW_PITCH, VOXEL_FREE), vq, wq);
    // Per labelled voxel: a 3-channel trilinear value noise n(v / P) from the
    // lattice (lerp along z, then y, then x, as the oracle), offset
    // floor(A * n + 0.5) per axis, and the label found there if it is labelled.
    const float amp = J.noise_amplitude;
    for (uint32_t i = t; i < total; i += blockDim.x) {
      const uint32_t e = vq[i], row = e >> 5, z = e & 31u;
      const uint32_t lx = row / VF_BY, ly = row % VF_BY;
      const uint32_t xr = x0 + lx, yr = y0 + ly, gz = z0 + z;
      const float t0 = t0s[lx], t1 = t1s[ly];
      float4 c00, c01, c10, c11;
      if (tabled) {
        const float4* T = table + ((i0s[lx] - cx) * ny + (i1s[ly] - cy)) * VF_BZ + z;
        c00 = T[0];
        c01 = T[VF_BZ];
        c10 = T[ny * VF_BZ];
        c11 = T[(ny + 1) * VF_BZ];
      } else {
        const float* L = J.lattice + (size_t)i0s[lx] * sx + (size_t)i1s[ly] * sy + (size_t)i2s[z] * 3;
        const float t2 = t2s[z];
        auto along = [&](const float* l) {
          return make_float4(lerp_(l[0], l[3], t2), lerp_(l[1], l[4], t2), lerp_(l[2], l[5], t2), 0.0f);
        };
        c00 = along(L);
        c01 = along(L + sy);
        c10 = along(L + sx);
        c11 = along(L + sx + sy);
      }
      auto offset = [&](float a00, float a01, float a10, float a11) {
        const float nzv = lerp_(lerp_(a00, a01, t1), lerp_(a10, a11, t1), t0);
        return (int)floorf(__fadd_rn(__fmul_rn(amp, nzv), 0.5f));
      };
      // amplitudes are at most 64: the sums stay in range, and a negative one is
      // past every grid
      const uint32_t ux = xr + (uint32_t)offset(c00.x, c01.x, c10.x, c11.x),
                     uy = yr + (uint32_t)offset(c00.y, c01.y, c10.y, c11.y),
                     uz = gz + (uint32_t)offset(c00.z, c01.z, c10.z, c11.z);
      if (ux >= J.X || uy >= J.Y || uz >= J.Z) continue;
      const uint16_t u = src[vf_gidx(J, ux, uy, uz)];
      if (u > VOXEL_FREE) vrows[row * ROW_PITCH + z] = u;
    }
    __syncthreads();
    rows_out(J, J.grid2, x0, y0, z0, vrows);
  }
}
constexpr int PERT_BYTES = PERT_COLS * VF_BZ * 16 + 256 * ROW_PITCH * 2 + 256 * VF_BZ * 2;

// ===========================================================================
// detectBoundaries-comp.glsl:18-43 (in place; neighbour reads clear bit 15,
// so concurrent updates of neighbours cannot change the outcome).
//
// load_tile that also tells whether a voxel of the brick can be a boundary: the
// labelled voxels staged (a z halo of 2 or 4 voxels of the 8) must have two
// different values, or one of the brick's own bit 15 set.  A fragment is wider
// than a brick, so most bricks end here.  wr: 8 words; ends in a barrier.
template <int H>
__device__ __forceinline__ bool load_tile_mixed(const JobDesc& J, uint32_t x0, uint32_t y0, uint32_t z0,
                                                uint16_t* tile, uint32_t* wr) {
  using T = Tile<H>;
  uint4* t4 = reinterpret_cast<uint4*>(tile);
  constexpr int PER_ROW = ZW / 8;
  uint32_t mn = 0xFFFFFFFFu, mx = 0, own = 0;
  auto take = [&](uint32_t w) {
    const uint32_t u = w & 0x7FFF7FFFu, g = __vcmpgtu2(u, 0x00010001u);
    mn = __vminu2(mn, u | ~g);
    mx = __vmaxu2(mx, u & g);
  };
  for (int q = threadIdx.x; q < T::ROWS * PER_ROW; q += blockDim.x) {
    const int row = q / PER_ROW, part = q % PER_ROW;
    const int rx = row / T::NY - H, ry = row % T::NY - H;
    const int x = (int)x0 + rx, y = (int)y0 + ry;
    const int z = (int)z0 - 8 + part * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (x >= 0 && y >= 0 && z >= 0 && x < (int)J.X && y < (int)J.Y && z < (int)J.Zp)
      v = __ldg(reinterpret_cast<const uint4*>(J.grid + vf_gidx(J, x, y, z)));
    t4[q] = v;
    if (part != 0) { take(v.x); if (H > 1) take(v.y); }
    if (part != PER_ROW - 1) { take(v.w); if (H > 1) take(v.z); }
    if (part != 0 && part != PER_ROW - 1) {
      if (H == 1) { take(v.y); take(v.z); }
      if (rx >= 0 && ry >= 0 && rx < VF_BX && ry < VF_BY) own |= v.x | v.y | v.z | v.w;
    }
  }
  const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, min(mn & 0xFFFFu, mn >> 16));
  const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, max(mx & 0xFFFFu, mx >> 16));
  own = __reduce_or_sync(0xFFFFFFFFu, own & 0x80008000u);
  if ((threadIdx.x & 31) == 0) wr[threadIdx.x >> 5] = lo | hi << 16 | (own ? 0x80000000u : 0u);
  __syncthreads();
  uint32_t a = 0xFFFFu, c = 0, f = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    a = min(a, wr[w] & 0xFFFFu);
    c = max(c, (wr[w] >> 16) & 0x7FFFu);
    f |= wr[w] & 0x80000000u;
  }
  return f != 0 || (c != 0 && a != c);
}

// Any boundary size up to H.  The labelled voxels of the bricks left look
// through their whole window (7^3 voxels at size 3) unless it ends early; bound
// by those shared memory reads: 180 x 179 x 192 voxels in 64 cells 79 us (220 us
// with a row per thread and no early end).
template <int H>
__global__ void __launch_bounds__(256) k_detect(const JobDesc* jobs, const uint32_t* list,
                                                const uint32_t* count, const uint32_t* brick_job) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint16_t* tile = reinterpret_cast<uint16_t*>(smem_raw);
  uint16_t* vq = reinterpret_cast<uint16_t*>(smem_raw + Tile<H>::BYTES);
  __shared__ uint32_t wq[8], wr[8];
  const int t = threadIdx.x;
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const JobDesc& J = jobs[brick_job[b]];
    if (!J.active) continue;  // uniform across the CTA
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    __syncthreads();
    if (!load_tile_mixed<H>(J, x0, y0, z0, tile, wr)) continue;
    const int bs = J.boundary_size;
    // rows past the grid and the z padding are staged as 0
    const uint16_t* own = tile + ((t / VF_BY + H) * Tile<H>::NY + t % VF_BY + H) * ZW + 8;
    const uint32_t total = queue_voxels(tile_voxels_above(own, VOXEL_FREE), vq, wq);
    for (uint32_t i = t; i < total; i += 256) {
      const uint32_t e = vq[i], row = e >> 5;
      const int lx = row / VF_BY, ly = row % VF_BY, z = e & 31;
      const uint16_t g = tval<H>(tile, lx, ly, z);
      bool bd = false;
      for (int a = lx - bs; a <= lx + bs && !bd; ++a)
        for (int c = ly - bs; c <= ly + bs && !bd; ++c)
          for (int d = z - bs; d <= z + bs; ++d) {
            const uint32_t u = tval<H>(tile, a, c, d) & 0x7FFFu;
            bd |= u > VOXEL_FREE && u != g;
          }
      if (bd) J.grid[vf_gidx(J, x0 + lx, y0 + ly, z0 + z)] = g | 0x8000u;
    }
  }
}

// detectBoundaries with boundary size <= 1, by window extrema.  Over the
// labelled voxels of the clamped 3x3x3 window (masked value u = w & 0x7FFF,
// labelled when u > 1; voxels outside the grid or the live bricks are 0),
// let mn / mx be the smallest / largest u.  A voxel g > 1 is a boundary in
// the reference's test (some labelled u != g) exactly when a labelled voxel
// exists and not all of them equal g: mn != none and (mn != g or mx != g).
// The window extrema are separable: phase 1 takes the z-window of every
// row (brick + 1-voxel halo) into two u16x2 planes, a thread per unit of 8
// voxels, the neighbour voxels from the lanes beside it; phase 2 takes the 3x3
// rows around each unit of the brick that holds a labelled voxel (a wall fills
// few), dealt to the threads.  Both with paired 16-bit min/max.  Bricks whose
// voxels and halo have one label end before that.
// Bound by latency (loads, barriers) and shared memory: 476 x 476 x 512 voxels 78 us,
// 128 mixed jobs 886 us (114 and 1430 us with the tile staged first, three CTAs to an
// SM, and phase 2 over every row; 1000 and 1230 us at 3 and 5 CTAs).
constexpr int D1_ROWS = (VF_BX + 2) * (VF_BY + 2);
constexpr int D1_UNITS = (D1_ROWS * 4 + 255) / 256;  // per thread
constexpr int D1_W = VF_BZ / 2;                      // u16 pairs per row
constexpr int D1_BYTES = 2 * D1_ROWS * D1_W * 4;
// 16-byte chunk c of window row r is stored at chunk c ^ ((r >> 1) & 3): the
// chunk-q loads of any 8 consecutive rows then fall on 8 distinct bank groups
__device__ __forceinline__ int d1_swz(int r, int c) { return c ^ ((r >> 1) & 3); }

__global__ void __launch_bounds__(256, 4) k_detect1(const JobDesc* jobs, const uint32_t* list,
                                                 const uint32_t* count, const uint32_t* brick_job) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t* zmin = reinterpret_cast<uint32_t*>(smem_raw);
  uint32_t* zmax = zmin + D1_ROWS * D1_W;
  __shared__ uint32_t wr[8], s_units;
  __shared__ uint16_t uq[256 * 4];
  const int t = threadIdx.x, c = t & 3;  // the thread's units are all unit c of their rows
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const JobDesc& J = jobs[brick_job[b]];
    if (!J.active) continue;  // uniform across the CTA
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    if (J.boundary_size <= 0) continue;  // the window is the voxel itself: a mark it may have stays
    // the thread's units, and for the first and last of a row the two voxels beyond
    uint4 a[D1_UNITS];
    uint32_t e[D1_UNITS];
#pragma unroll
    for (int k = 0; k < D1_UNITS; ++k) {
      const int r = 64 * k + (t >> 2);
      const int x = (int)x0 - 1 + r / (VF_BY + 2), y = (int)y0 - 1 + r % (VF_BY + 2);
      const uint32_t z = z0 + 8 * c;
      const bool ok = r < D1_ROWS && x >= 0 && y >= 0 && x < (int)J.X && y < (int)J.Y;
      const uint16_t* row = J.grid + (ok ? vf_gidx(J, x, y, 0) : 0);
      a[k] = ok && z < J.Zp ? *reinterpret_cast<const uint4*>(row + z) : make_uint4(0, 0, 0, 0);
      e[k] = 0;
      if (ok && c == 0 && z0) e[k] = *reinterpret_cast<const uint32_t*>(row + z0 - 2);
      if (ok && c == 3 && z0 + VF_BZ < J.Zp) e[k] = *reinterpret_cast<const uint32_t*>(row + z0 + VF_BZ);
    }
    // can a voxel of the brick be a boundary?  The labelled voxels must have two
    // different values, or one of the brick's own bit 15 set
    uint32_t mn = 0xFFFFFFFFu, mx = 0, own = 0;
    auto lo = [](uint32_t w) {
      const uint32_t u = w & 0x7FFF7FFFu;
      return u | ~__vcmpgtu2(u, 0x00010001u);
    };
    auto hi = [](uint32_t w) {
      const uint32_t u = w & 0x7FFF7FFFu;
      return u & __vcmpgtu2(u, 0x00010001u);
    };
#pragma unroll
    for (int k = 0; k < D1_UNITS; ++k) {
      const int r = 64 * k + (t >> 2), rx = r / (VF_BY + 2), ry = r % (VF_BY + 2);
      const uint32_t w[5] = {a[k].x, a[k].y, a[k].z, a[k].w, e[k]};
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        mn = __vminu2(mn, lo(w[i]));
        mx = __vmaxu2(mx, hi(w[i]));
      }
      if (rx >= 1 && ry >= 1 && rx <= VF_BX && ry <= VF_BY) own |= a[k].x | a[k].y | a[k].z | a[k].w;
    }
    const uint32_t wlo = __reduce_min_sync(0xFFFFFFFFu, min(mn & 0xFFFFu, mn >> 16));
    const uint32_t whi = __reduce_max_sync(0xFFFFFFFFu, max(mx & 0xFFFFu, mx >> 16));
    own = __reduce_or_sync(0xFFFFFFFFu, own & 0x80008000u);
    __syncthreads();  // the previous brick is done with the shared arrays
    if ((t & 31) == 0) wr[t >> 5] = wlo | whi << 16 | (own ? 0x80000000u : 0u);
    if (t == 0) s_units = 0;
    __syncthreads();
    uint32_t least = 0xFFFFu, most = 0, marks = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      least = min(least, wr[w] & 0xFFFFu);
      most = max(most, (wr[w] >> 16) & 0x7FFFu);
      marks |= wr[w] & 0x80000000u;
    }
    if (!marks && (most == 0 || least == most)) continue;
    // phase 1: z-window extrema.  The window of pair p is (2p-1, 2p), (2p, 2p+1)
    // and (2p+1, 2p+2); labelled halves keep u = w & 0x7FFF, the others
    // become 0xFFFF (min) / 0 (max).  The masks act on each 16-bit half
    // alone, so they are taken once per word and the shifted windows are
    // byte permutes of the masked words.
#pragma unroll
    for (int k = 0; k < D1_UNITS; ++k) {
      const int r = 64 * k + (t >> 2), rx = r / (VF_BY + 2), ry = r % (VF_BY + 2);
      const uint32_t below = __shfl_up_sync(0xFFFFFFFFu, a[k].w, 1), above = __shfl_down_sync(0xFFFFFFFFu, a[k].x, 1);
      if (r >= D1_ROWS) continue;
      const uint32_t w[6] = {c ? below : e[k], a[k].x, a[k].y, a[k].z, a[k].w, c < 3 ? above : e[k]};
      uint32_t L[6], H[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) { L[i] = lo(w[i]); H[i] = hi(w[i]); }
      uint32_t zl[4], zh[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        zl[i] = __vminu2(__vminu2(__byte_perm(L[i], L[i + 1], 0x5432), L[i + 1]),
                         __byte_perm(L[i + 1], L[i + 2], 0x5432));
        zh[i] = __vmaxu2(__vmaxu2(__byte_perm(H[i], H[i + 1], 0x5432), H[i + 1]),
                         __byte_perm(H[i + 1], H[i + 2], 0x5432));
      }
      const int o = r * D1_W + (d1_swz(r, c) << 2);
      *reinterpret_cast<uint4*>(zmin + o) = make_uint4(zl[0], zl[1], zl[2], zl[3]);
      *reinterpret_cast<uint4*>(zmax + o) = make_uint4(zh[0], zh[1], zh[2], zh[3]);
      // the brick's units with a label above 1 (rows past the grid and the z
      // padding were read as 0)
      if (rx >= 1 && ry >= 1 && rx <= VF_BX && ry <= VF_BY &&
          ((a[k].x | a[k].y | a[k].z | a[k].w) & 0xFFFEFFFEu) != 0)
        uq[atomicAdd(&s_units, 1u)] = (uint16_t)(r << 2 | c);
    }
    __syncthreads();
    const uint32_t units = s_units;
#pragma unroll 1
    for (uint32_t i = t; i < units; i += 256) {
      const int r0 = uq[i] >> 2, q = uq[i] & 3;
      const uint32_t x = x0 - 1 + r0 / (VF_BY + 2), y = y0 - 1 + r0 % (VF_BY + 2);
      uint4* const at = reinterpret_cast<uint4*>(J.grid + vf_gidx(J, x, y, z0)) + q;
      const uint4 gq = *at;  // only this thread writes it
      const uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w};
      uint32_t out[4], marked = 0;
      // phase 2: the 3x3 rows around this row
      uint4 zl = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
      uint4 zh = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const int row = r0 + (k / 3 - 1) * (VF_BY + 2) + k % 3 - 1;
        const uint4 p = reinterpret_cast<const uint4*>(zmin + row * D1_W)[d1_swz(row, q)];
        const uint4 h = reinterpret_cast<const uint4*>(zmax + row * D1_W)[d1_swz(row, q)];
        zl.x = __vminu2(zl.x, p.x); zl.y = __vminu2(zl.y, p.y);
        zl.z = __vminu2(zl.z, p.z); zl.w = __vminu2(zl.w, p.w);
        zh.x = __vmaxu2(zh.x, h.x); zh.y = __vmaxu2(zh.y, h.y);
        zh.z = __vmaxu2(zh.z, h.z); zh.w = __vmaxu2(zh.w, h.w);
      }
      // per 16-bit half: marked when g > FREE, some labelled voxel is in
      // the window (min != 0xFFFF) and the window is not uniformly g
      const uint32_t mns[4] = {zl.x, zl.y, zl.z, zl.w}, mxs[4] = {zh.x, zh.y, zh.z, zh.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t bd = __vcmpgtu2(gw[k], 0x00010001u) & __vcmpne2(mns[k], 0xFFFFFFFFu) &
                            (__vcmpne2(mns[k], gw[k]) | __vcmpne2(mxs[k], gw[k]));
        out[k] = gw[k] | (bd & 0x80008000u);
        marked |= bd;
      }
      // a unit is written only where a voxel was marked
      if (marked) *at = make_uint4(out[0], out[1], out[2], out[3]);
    }
  }
}

// A brick's rows from the tile to dst without the voxels of drop (bit z per row).
template <int H>
__device__ __forceinline__ void rows_kept(const JobDesc& J, uint16_t* dst, uint32_t x0, uint32_t y0, uint32_t z0,
                                          const uint16_t* tile, const uint32_t* drop) {
  const uint32_t nz = min((uint32_t)VF_BZ, J.Zp - z0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t u = i * 256 + threadIdx.x, row = u >> 2, q = u & 3;
    const uint32_t lx = row / VF_BY, ly = row % VF_BY;
    if (x0 + lx >= J.X || y0 + ly >= J.Y || 8 * q >= nz) continue;
    uint4 w = *reinterpret_cast<const uint4*>(tile + ((lx + H) * Tile<H>::NY + ly + H) * ZW + 8 + 8 * q);
    const uint32_t m = drop[row] >> (8 * q);
    auto keep = [&](int k) { return ((m >> k) & 1u ? 0u : 0xFFFFu) | ((m >> k) & 2u ? 0u : 0xFFFF0000u); };
    if (m & 0xFFu) { w.x &= keep(0); w.y &= keep(2); w.z &= keep(4); w.w &= keep(6); }
    *reinterpret_cast<uint4*>(dst + vf_gidx(J, x0 + lx, y0 + ly, z0 + 8 * q)) = w;
  }
}

// erodeGrid-comp.glsl:26-59: src -> dst.  Gate bool(unmaskedBit(v,15)) holds
// for every labelled voxel; full 16-bit equality; globalCount = clamped
// window size; noise[idx % 1e6] from the counter RNG.  The mask holds zeros and
// ones; voxels outside the grid are staged as 0 and equal no gated voxel, so
// the equal voxels are counted over the mask's ones alone, wherever they lie.
constexpr int ERODE_MASK = 343;
template <int H>
__device__ __forceinline__ void erode_brick(const JobDesc& J, uint32_t x0, uint32_t y0, uint32_t z0,
                                            uint16_t* tile, uint16_t* vq, uint32_t* drop, uint32_t* wq,
                                            int16_t* ones, uint32_t& nones) {
  const int t = threadIdx.x, k = J.ek;
  load_tile<H>(J, J.grid, x0, y0, z0, tile);
  drop[t] = 0;
  for (int i = t; i < k * k * k; i += 256)
    if (J.emask[i] >= 1.0f)
      ones[atomicAdd(&nones, 1u)] =
          (int16_t)(((i / (k * k) - H) * Tile<H>::NY + (i / k) % k - H) * ZW + i % k - H);
  __syncthreads();
  const uint16_t* own = tile + ((t / VF_BY + H) * Tile<H>::NY + t % VF_BY + H) * ZW + 8;
  uint32_t m = tile_voxels_above(own, VOXEL_FREE);
  const uint32_t total = queue_voxels(m, vq, wq);
  const int nm = (int)nones;
  for (uint32_t i = t; i < total; i += 256) {
    const uint32_t e = vq[i], row = e >> 5;
    const int lx = row / VF_BY, ly = row % VF_BY, z = e & 31;
    const uint16_t* at = tile + ((lx + H) * Tile<H>::NY + ly + H) * ZW + 8 + z;
    const uint32_t g = *at;
    if ((g & 0x7FFFu) == 0) continue;
    const int x = (int)x0 + lx, y = (int)y0 + ly, gz = (int)z0 + z;
    const uint32_t nidx = (uint32_t)((((unsigned long long)x * J.Y + y) * J.Z + gz) % VF_NOISE_BUFFER);
    if (!(vf_u01(vf_hash(J.seed, VF_STREAM_ERODE, nidx)) < J.erosion_probability)) continue;
    const int global = (min(x + H, (int)J.X - 1) - max(x - H, 0) + 1) * (min(y + H, (int)J.Y - 1) - max(y - H, 0) + 1) *
                       (min(gz + H, (int)J.Z - 1) - max(gz - H, 0) + 1);
    uint32_t cnt = 0;
#pragma unroll 9
    for (int o = 0; o < nm; ++o) cnt += at[ones[o]] == g;
    if (__fdiv_rn((float)cnt, (float)global) < J.elimit) atomicOr(&drop[row], 1u << z);
  }
  __syncthreads();
  rows_kept<H>(J, J.grid2, x0, y0, z0, tile, drop);
}
constexpr int ERODE_BYTES = Tile<3>::BYTES + 256 * VF_BZ * 2;
// Bound by the window counts of the gated voxels: 200 x 197 x 208 voxels, windows
// of 3, 38 us (119 us with a row per thread and a halo of 3).
__global__ void __launch_bounds__(256) k_erode(const JobDesc* jobs, const uint32_t* list,
                                               const uint32_t* count, const uint32_t* brick_job) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint16_t* tile = reinterpret_cast<uint16_t*>(smem_raw);
  uint16_t* vq = reinterpret_cast<uint16_t*>(smem_raw + Tile<3>::BYTES);
  __shared__ uint32_t drop[256], wq[8], nones;
  __shared__ int16_t ones[ERODE_MASK];
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const JobDesc& J = jobs[brick_job[b]];
    if (!J.active) continue;
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    __syncthreads();  // the previous brick is done with the shared arrays
    if (threadIdx.x == 0) nones = 0;
    __syncthreads();
    // a tile with the window's own halo: windows of 3 are the common ones
    if (J.ek <= 1) erode_brick<0>(J, x0, y0, z0, tile, vq, drop, wq, ones, nones);
    else if (J.ek == 3) erode_brick<1>(J, x0, y0, z0, tile, vq, drop, wq, ones, nones);
    else if (J.ek == 5) erode_brick<2>(J, x0, y0, z0, tile, vq, drop, wq, ones, nones);
    else erode_brick<3>(J, x0, y0, z0, tile, vq, drop, wq, ones, nones);
  }
}

// removeIsolatedRegionsGrid-comp.glsl:16-39, src -> dst (Jacobi).  Voxels
// outside the grid are staged as 0 and equal no occupied one.
// Bound by the window counts: 200 x 197 x 208 voxels 24 us (92 us with a row per thread).
__global__ void __launch_bounds__(256) k_isolated(const JobDesc* jobs, const uint32_t* list,
                                                  const uint32_t* count, const uint32_t* brick_job) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint16_t* tile = reinterpret_cast<uint16_t*>(smem_raw);
  __shared__ uint16_t vq[256 * VF_BZ];
  __shared__ uint32_t drop[256], wq[8];
  const int t = threadIdx.x;
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const JobDesc& J = jobs[brick_job[b]];
    if (!J.active) continue;
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    __syncthreads();
    load_tile<1>(J, J.grid, x0, y0, z0, tile);
    drop[t] = 0;
    __syncthreads();
    const uint16_t* own = tile + ((t / VF_BY + 1) * Tile<1>::NY + t % VF_BY + 1) * ZW + 8;
    const uint32_t total = queue_voxels(tile_voxels_above(own, VOXEL_EMPTY), vq, wq);
    for (uint32_t i = t; i < total; i += 256) {
      const uint32_t e = vq[i], row = e >> 5, z = e & 31u;
      const uint16_t* at = tile + ((row / VF_BY + 1) * Tile<1>::NY + row % VF_BY + 1) * ZW + 8 + z;
      const uint32_t g = *at;
      int c = -1;
#pragma unroll
      for (int r = 0; r < 9; ++r)
#pragma unroll
        for (int d = -1; d <= 1; ++d) c += at[((r / 3 - 1) * Tile<1>::NY + r % 3 - 1) * ZW + d] == g;
      if (c < 6) atomicOr(&drop[row], 1u << z);
    }
    __syncthreads();
    rows_kept<1>(J, J.grid2, x0, y0, z0, tile, drop);
  }
}

// RegularGrid::countValues (RegularGrid.cpp:601-625).  Bound by latency, a brick
// per CTA at a time: 476 x 476 x 512 voxels 27 us (61 us with an add per voxel).
__global__ void __launch_bounds__(256) k_counts(const JobDesc* jobs, JobState* st,
                                                const uint32_t* list, const uint32_t* count,
                                                const uint32_t* brick_job) {
  __shared__ uint32_t hist[256];
  __shared__ unsigned long long occ;
  const uint32_t n = *count;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const uint32_t b = list[it];
    const uint32_t j = brick_job[b];
    const JobDesc& J = jobs[j];
    if (!J.active) continue;
    uint32_t x0, y0, z0;
    brick_coords(J, b, x0, y0, z0);
    __syncthreads();
    hist[threadIdx.x] = 0;
    if (threadIdx.x == 0) occ = 0;
    __syncthreads();
    // four lanes per row, each 16 bytes (8 voxels) of the row's 64: a warp
    // reads 8 rows as contiguous segments; 4 passes cover the brick's 256 rows
    uint32_t mine = 0, err = 0;
    // a thread's voxels come in runs of one label: one add per run
    uint32_t val = 0, run = 0;
    auto flush = [&]() {
      if (!run) return;
      if (val < 256) atomicAdd(&hist[val], run);
      else if (val < J.ncounts) atomicAdd(&J.counts[val], run);
      else err = 1;
      mine += run;
      run = 0;
    };
    const uint32_t nz = min((uint32_t)VF_BZ, J.Zp - z0);
    const uint32_t part = threadIdx.x & 3u;
    uint4 wv[4];
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
      const uint32_t row = (threadIdx.x >> 2) + 64u * pass;
      const uint32_t x = x0 + row / VF_BY, y = y0 + row % VF_BY;
      wv[pass] = make_uint4(0, 0, 0, 0);
      if (x < J.X && y < J.Y && 8u * part < nz)
        wv[pass] = *reinterpret_cast<const uint4*>(J.grid + vf_gidx(J, x, y, z0 + 8u * part));
    }
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
      const uint32_t ww[4] = {wv[pass].x, wv[pass].y, wv[pass].z, wv[pass].w};
      // 8 voxels of one label, or of none
      const uint32_t w0 = ww[0];
      if (w0 == ww[1] && w0 == ww[2] && w0 == ww[3] && (w0 >> 16) == (w0 & 0xFFFFu)) {
        if ((w0 & 0xFFFFu) > VOXEL_FREE) {
          if ((w0 & 0x7FFFu) != val) {
            flush();
            val = w0 & 0x7FFFu;
          }
          run += 8;
        }
        continue;
      }
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        const uint32_t g = (ww[h >> 1] >> (16 * (h & 1))) & 0xFFFFu;
        if (g > VOXEL_FREE) {
          if ((g & 0x7FFFu) != val) {
            flush();
            val = g & 0x7FFFu;
          }
          ++run;
        }
      }
    }
    flush();
    mine = __reduce_add_sync(0xFFFFFFFFu, mine);
    if ((threadIdx.x & 31) != 0) mine = 0;
    if (mine) atomicAdd(&occ, (unsigned long long)mine);
    if (err) atomicOr(&st[j].err, VF_JERR_RANGE);
    __syncthreads();
    const uint32_t h = hist[threadIdx.x];
    if (h) {
      if (threadIdx.x < J.ncounts) atomicAdd(&J.counts[threadIdx.x], h);
      else atomicOr(&st[j].err, VF_JERR_RANGE);
    }
    if (threadIdx.x == 0 && occ) atomicAdd(&st[j].occupied, occ);
  }
}


// ---------------------------------------------------------------------------
// Label download, 16-byte path: a caller's buffer the GPU writes directly (mapped
// pinned host memory, 16-byte aligned), Z a multiple of 4.  The job's output is a
// flat array of X*Y*Z labels written in 16-byte units (8 labels); each unit is two
// 8-byte halves, and a half never crosses a row, so it is one 8-byte load from row
// (e / Z) at z = e % Z.  Units go to consecutive lanes, so every warp store is 512
// contiguous bytes.
__global__ void __launch_bounds__(256) k_pack16(const JobDesc* jobs, int njobs) {
  for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
    const JobDesc& J = jobs[j];
    if (!J.out || J.out_dma || (J.Z & 3u) || (reinterpret_cast<uintptr_t>(J.out) & 15u)) continue;
    const unsigned long long total = (unsigned long long)J.X * J.Y * J.Z;
    const unsigned long long units = total / 8;
    uint4* d = reinterpret_cast<uint4*>(J.out);
    const uint32_t Z = J.Z;
    if (total < (1ull << 32)) {
      // one 32-bit division per unit; the second half's row follows from the first
      for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < (uint32_t)units;
           u += gridDim.x * blockDim.x) {
        const uint32_t e0 = 8 * u;
        const uint32_t r0 = e0 / Z, o0 = e0 - r0 * Z;
        const uint32_t r1 = o0 + 4 < Z ? r0 : r0 + 1, o1 = o0 + 4 < Z ? o0 + 4 : o0 + 4 - Z;
        const uint2 a = *reinterpret_cast<const uint2*>(J.grid + (size_t)r0 * J.Zp + o0);
        const uint2 b = *reinterpret_cast<const uint2*>(J.grid + (size_t)r1 * J.Zp + o1);
        d[u] = make_uint4(a.x, a.y, b.x, b.y);
      }
    } else {
      for (unsigned long long u = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; u < units;
           u += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long e0 = 8 * u, e1 = e0 + 4;
        const unsigned long long r0 = e0 / Z, r1 = e1 / Z;
        const uint2 a = *reinterpret_cast<const uint2*>(J.grid + r0 * J.Zp + (e0 - r0 * Z));
        const uint2 b = *reinterpret_cast<const uint2*>(J.grid + r1 * J.Zp + (e1 - r1 * Z));
        d[u] = make_uint4(a.x, a.y, b.x, b.y);
      }
    }
    // the last total % 8 labels (a multiple of 4)
    if (blockIdx.x == 0 && threadIdx.x == 0 && (total & 7u)) {
      const unsigned long long e = total - 4, r = e / J.Z;
      *reinterpret_cast<uint2*>(J.out + e) = *reinterpret_cast<const uint2*>(J.grid + r * J.Zp + (e - r * J.Z));
    }
  }
}

// Labels without the z padding into J.out (a device staging buffer, or a caller's
// buffer k_pack16 does not take).  The rows of all jobs are numbered consecutively
// (row_base per job); a warp takes 4 consecutive ones, 8 lanes per row (rows are
// 64..384 labels: 8..48 16-byte units), so it has four rows' loads in flight, and
// copies each with the widest access its alignment allows.  A warp's rows only
// increase, so its job is found by walking forward from the previous one.
__global__ void __launch_bounds__(256) k_pack(const JobDesc* jobs, int njobs, unsigned long long row0,
                                              unsigned long long total_rows) {
  const int lane = threadIdx.x & 31, sub = lane & 7;
  const unsigned long long nw = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  int j = 0;
  for (unsigned long long r0 = (((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4;
       r0 < total_rows; r0 += nw * 4) {
    unsigned long long r = r0 + (lane >> 3);
    if (r >= total_rows) continue;
    r += row0;
    while (j + 1 < njobs && jobs[j + 1].row_base <= r) ++j;
    const JobDesc& J = jobs[j];
    if (!J.out) continue;
    if (!J.out_dma && (J.Z & 3u) == 0u && (reinterpret_cast<uintptr_t>(J.out) & 15u) == 0u) continue;  // k_pack16
    const unsigned long long lr = r - J.row_base;
    const uint16_t* src = J.grid + lr * J.Zp;  // 16-byte aligned (Zp is a multiple of 8)
    uint16_t* dst = J.out + lr * J.Z;
    const uintptr_t da = reinterpret_cast<uintptr_t>(dst);
    const uint32_t Z = J.Z;
    if ((Z & 7u) == 0u && (da & 15u) == 0u) {
      const uint4* s4 = reinterpret_cast<const uint4*>(src);
      uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll 2
      for (uint32_t q = sub; q < Z / 8; q += 8) d4[q] = __ldcs(s4 + q);
    } else if ((Z & 3u) == 0u && (da & 7u) == 0u) {
      const uint2* s2 = reinterpret_cast<const uint2*>(src);
      uint2* d2 = reinterpret_cast<uint2*>(dst);
      for (uint32_t q = sub; q < Z / 4; q += 8) d2[q] = __ldcs(s2 + q);
    } else if ((Z & 1u) == 0u && (da & 3u) == 0u) {
      const uint32_t* s1 = reinterpret_cast<const uint32_t*>(src);
      uint32_t* d1 = reinterpret_cast<uint32_t*>(dst);
      for (uint32_t q = sub; q < Z / 2; q += 8) d1[q] = __ldcs(s1 + q);
    } else {
      for (uint32_t q = sub; q < Z; q += 8) dst[q] = src[q];
    }
  }
}
}  // namespace

namespace vfk {

static inline int brick_grid(uint32_t max_count) {
  uint32_t g = max_count ? max_count : 1;
  return (int)(g > (1u << 20) ? (1u << 20) : g);
}

void sample_seeds(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs) {
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_seeds, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SeedSmem));
    attr[dv] = true;
  }
  if (njobs > 0) k_seeds<<<njobs, 1024, sizeof(SeedSmem), st>>>(dj, ds);
}

void naive(cudaStream_t st, const JobDesc* dj, const JobState* ds, const uint32_t* list,
           const uint32_t* count, uint32_t max_count, const uint32_t* brick_job) {
  if (max_count) k_naive<<<brick_grid(max_count), 256, 0, st>>>(dj, ds, list, count, brick_job);
}

void lattice(cudaStream_t st, const JobDesc* dj, int njobs) {
  if (njobs > 0) k_lattice<<<dim3(64, njobs), 256, 0, st>>>(dj);
}
void perturb(cudaStream_t st, const JobDesc* dj, const uint32_t* list, const uint32_t* count,
             uint32_t max_count, const uint32_t* brick_job) {
  if (!max_count) return;
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_perturb, cudaFuncAttributeMaxDynamicSharedMemorySize, PERT_BYTES);
    attr[dv] = true;
  }
  k_perturb<<<brick_grid(max_count), 256, PERT_BYTES, st>>>(dj, list, count, brick_job);
}

void detect_boundaries(cudaStream_t st, const JobDesc* dj, const uint32_t* list,
                       const uint32_t* count, uint32_t max_count, const uint32_t* brick_job) {
  // boundary sizes 0..1 (the default): window extrema; 2..3: detect_boundaries_wide
  if (!max_count) return;
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_detect1, cudaFuncAttributeMaxDynamicSharedMemorySize, D1_BYTES);
    attr[dv] = true;
  }
  k_detect1<<<brick_grid(max_count), 256, D1_BYTES, st>>>(dj, list, count, brick_job);
}
void detect_boundaries_wide(cudaStream_t st, const JobDesc* dj, const uint32_t* list,
                            const uint32_t* count, uint32_t max_count, const uint32_t* brick_job) {
  if (!max_count) return;
  constexpr int bytes = Tile<3>::BYTES + 256 * VF_BZ * 2;
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_detect<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    attr[dv] = true;
  }
  k_detect<3><<<brick_grid(max_count), 256, bytes, st>>>(dj, list, count, brick_job);
}

void erode(cudaStream_t st, const JobDesc* dj, const uint32_t* list, const uint32_t* count,
           uint32_t max_count, const uint32_t* brick_job) {
  if (!max_count) return;
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_erode, cudaFuncAttributeMaxDynamicSharedMemorySize, ERODE_BYTES);
    attr[dv] = true;
  }
  k_erode<<<brick_grid(max_count), 256, ERODE_BYTES, st>>>(dj, list, count, brick_job);
}
void remove_isolated(cudaStream_t st, const JobDesc* dj, const uint32_t* list,
                     const uint32_t* count, uint32_t max_count, const uint32_t* brick_job) {
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_isolated, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<1>::BYTES);
    attr[dv] = true;
  }
  if (max_count)
    k_isolated<<<brick_grid(max_count), 256, Tile<1>::BYTES, st>>>(dj, list, count, brick_job);
}
void count_values(cudaStream_t st, const JobDesc* dj, JobState* ds, const uint32_t* list,
                  const uint32_t* count, uint32_t max_count, const uint32_t* brick_job) {
  if (max_count) k_counts<<<brick_grid(max_count), 256, 0, st>>>(dj, ds, list, count, brick_job);
}

void pack_labels(cudaStream_t st, const JobDesc* dj, int njobs, uint64_t row0, uint64_t rows, int num_sms,
                 int ctas_per_sm) {
  if (njobs <= 0 || !rows) return;
  const int per_job = std::max(1, num_sms * ctas_per_sm / njobs);
  k_pack16<<<dim3(per_job, std::min(njobs, 65535)), 256, 0, st>>>(dj, njobs);
  k_pack<<<num_sms * ctas_per_sm, 256, 0, st>>>(dj, njobs, row0, (unsigned long long)rows);
}

}  // namespace vfk
