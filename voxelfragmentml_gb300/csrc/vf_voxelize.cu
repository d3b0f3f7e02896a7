// vf_voxelize.cu -- solid voxelization of triangle meshes on sm_103a.
//
// Occupancy of a voxel = (some triangle overlaps the voxel box: FP32 SAT in
// the operation order of Intersections3D.h:204-258) OR (the voxel sample
// point is inside the mesh by tetra parity: Tetravoxelizer.cpp:42-92, 198-315).
//
// Stages, all batched over every job of a batch:
//   centroid_and_slices : a cluster of 8 CTAs per job; fixed-order lane sums
//                         of the vertices + the slice planes
//   tetra_prep          : one thread per face -> its vertices in NDC sorted
//                         by y, the slice planes crossing it, one use of each
//                         edge in the job's edge parity table
//   parity_raster       : the tetra-parity fill computed from edge crossings
//                         (derivation above k_tetra): (face, slice) segments
//                         flattened by a prefix sum over the faces and run in
//                         warp-interleaved runs, the internal faces of edges
//                         used an odd number of times, then a prefix XOR
//                         along x turns the per-row crossing markers into the
//                         parity plane
//   shell_sat           : columns of each triangle's footprint in even units
//                         (prefix sum over groups of 32 faces); interval forms
//                         with margins decide nearly all cells, the exact SAT
//                         the rest
//   combine             : one CTA per brick; bit planes -> uint16 0/1 rows,
//                         brick liveness
// All float arithmetic uses the _rn intrinsics (and the file is compiled
// with -fmad=false): every result is bit-identical to the CPU oracle.
#include <cooperative_groups.h>
#include <cuda_pipeline_primitives.h>

#include "vf_kernels.h"
#include "vf_slices.h"

namespace {

__device__ __forceinline__ int job_of_face(const JobDesc* J, int njobs, uint32_t f) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (J[mid].face_base <= f) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// The oracle's 1024 interleaved sums of the vertices, then its tree over them.  A
// cluster of 8 CTAs per job takes 128 sums each, 32 vertices of each sum on their
// way to shared memory: 393 k vertices 40 us (98 us in one CTA).
constexpr int CEN_CTAS = 8, CEN_LANES = 1024 / CEN_CTAS, CEN_FLIGHT = 32;
constexpr int CEN_BYTES = CEN_FLIGHT * 3 * CEN_LANES * 4;
__global__ void __cluster_dims__(CEN_CTAS, 1, 1) __launch_bounds__(CEN_LANES) k_centroid(const JobDesc* jobs, JobState* st) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const JobDesc& J = jobs[blockIdx.x / CEN_CTAS];
  JobState& S = st[blockIdx.x / CEN_CTAS];
  __shared__ float sum[3][1024];  // of the first CTA
  const int t = threadIdx.x, rank = (int)cluster.block_rank(), lane = rank * CEN_LANES + t;
  // rows of the CTA's 128 vertices (1536 contiguous bytes of every 1024 vertices),
  // CEN_FLIGHT of them in GROUPS copies of 16-byte units
  constexpr uint32_t GROUPS = 4, PER = CEN_FLIGHT / GROUPS, UNITS = 3 * CEN_LANES / 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float(*const ring)[3 * CEN_LANES] = reinterpret_cast<float(*)[3 * CEN_LANES]>(smem_raw);
  const uint32_t n = J.nverts, row0 = (uint32_t)rank * CEN_LANES;
  const uint32_t rows = row0 < n ? (n - row0 - 1u) / 1024u + 1u : 0u;
  const size_t floats = 3 * (size_t)n;
  auto fetch = [&](uint32_t g) {
    for (uint32_t u = t; u < PER * UNITS; u += CEN_LANES) {
      const uint32_t m = g * PER + u / UNITS, e = 4 * (u % UNITS);
      const size_t at = 3 * (row0 + 1024u * (size_t)m) + e;
      float* const to = &ring[m % CEN_FLIGHT][e];
      if (at + 4 <= floats) __pipeline_memcpy_async(to, J.verts + at, 16);
      else
        for (uint32_t k = 0; at + k < floats; ++k) to[k] = J.verts[at + k];
    }
    __pipeline_commit();
  };
  for (uint32_t g = 0; g < GROUPS; ++g) fetch(g);
  float a[3] = {0.0f, 0.0f, 0.0f};
  for (uint32_t g = 0; g * PER < rows; ++g) {
    __pipeline_wait_prior(GROUPS - 1);
    __syncthreads();
    const float* const at = ring[(g * PER) % CEN_FLIGHT] + 3 * t;
    float v[PER][3];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[k][c] = at[k * 3 * CEN_LANES + c];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
      const bool in = (size_t)lane + 1024u * (size_t)(g * PER + k) < n;
#pragma unroll
      for (int c = 0; c < 3; ++c) a[c] = in ? __fadd_rn(a[c], v[k][c]) : a[c];
    }
    __syncthreads();
    fetch(g + GROUPS);
  }
  __pipeline_wait_prior(0);
  cluster.sync();  // every CTA of the cluster runs: its shared memory may be written
  float(*const to)[1024] = cluster.map_shared_rank(sum, 0);
#pragma unroll
  for (int c = 0; c < 3; ++c) to[c][lane] = a[c];
  cluster.sync();
  if (rank == 1 && t == 0) {
    // ySlice = -1; ySlice += 2/res.y (Tetravoxelizer.cpp:280-293)
    float* const ys = J.ys;
    const uint32_t Y = J.Y;
    const float step = __fdiv_rn(2.0f, (float)Y);
    float acc = -1.0f;
    for (uint32_t s = 0; s < Y; ++s) {
      ys[s] = acc;
      acc = __fadd_rn(acc, step);
    }
  }
  if (rank) return;
  for (int s = 512; s >= 1; s >>= 1) {
    for (int k = t; k < s; k += CEN_LANES)
#pragma unroll
      for (int c = 0; c < 3; ++c) sum[c][k] = __fadd_rn(sum[c][k], sum[c][k + s]);
    __syncthreads();
  }
  if (t < 3) S.centroid[t] = __fdiv_rn(sum[t][0], (float)n);
  if (t == 0) S.odd_edges = 0;
}

struct tv { float x, y, z; };

__device__ __forceinline__ tv to_ndc(const float* v, const float* ctr, const float* dim) {
  // scaleToNDC: 2*(v - c)/dim (Tetravoxelizer.h:70-72)
  tv r;
  r.x = __fdiv_rn(__fmul_rn(2.0f, __fsub_rn(v[0], ctr[0])), dim[0]);
  r.y = __fdiv_rn(__fmul_rn(2.0f, __fsub_rn(v[1], ctr[1])), dim[1]);
  r.z = __fdiv_rn(__fmul_rn(2.0f, __fsub_rn(v[2], ctr[2])), dim[2]);
  return r;
}

// ---- parity by edge crossings ---------------------------------------------
// The reference rasterises, for every slice plane, the cross-section of every
// tetrahedron (face + centroid) with XOR at pixel centres (GL rules: 8
// sub-pixel bits, top-left ownership of samples on edges).  With that rule a
// sample p is inside a cross-section triangle exactly when the point
// p + (e, e^2) (e -> 0) is inside the open triangle, and that point lies on
// no edge and no vertex line.  A ray from it towards -x therefore crosses the
// triangle's boundary an odd number of times exactly when p is inside; for a
// zero-area triangle (never rasterised) the crossings are even.  Hence the
// XOR of all rasterised triangles at p is the parity of the number of
// cross-section EDGES that the ray crosses, and an edge's crossing depends
// only on its two snapped end points:
//   edge (u, v), u.z < v.z (fixed point), crosses at pixel centre
//   p = (256 i + 128, 256 k + 128)  iff  u.z <= p.z < v.z  and
//   (v.x - u.x)(p.z - u.z) - (v.z - u.z)(p.x - u.x) <= 0.
// Each cross-section edge lies on one face of its tetrahedron and its end
// points are INTERP on two tetrahedron edges (lower-y vertex first).  An
// internal face (mesh edge + centroid) is shared by every tetrahedron whose
// mesh face holds that edge, and each computes the same end points, so the
// copies cancel in pairs: only the mesh faces' own segments and the internal
// faces of mesh edges used an odd number of times (open or non-manifold
// meshes) contribute.  Per segment and pixel row the first crossed pixel
// gets a marker bit; a prefix XOR along x then yields the parity plane.
// The quad split's diagonal belongs to both of its triangles and cancels.

// slot value of an edge parity table: lo << 32 | hi (lo < hi < 2^31), bit 63
// toggled once per use of the edge; an empty slot is all ones
#define VF_EDGE_EMPTY 0xFFFFFFFFFFFFFFFFull
#define VF_EDGE_ODD 0x8000000000000000ull

// returns the change of the number of edges used an odd number of times; a first
// use is one atomic
__device__ __forceinline__ int edge_use(const JobDesc& J, uint32_t a, uint32_t b) {
  if (a == b) return 0;  // a degenerate edge bounds a zero-area face: no crossing
  const unsigned long long key =
      a < b ? ((unsigned long long)a << 32 | b) : ((unsigned long long)b << 32 | a);
  const uint32_t mask = J.ecap - 1;
  uint32_t h = (uint32_t)vf_mix64(key) & mask;
  for (uint32_t probe = 0; probe < J.ecap; ++probe) {
    const unsigned long long old = atomicCAS(J.etab + h, VF_EDGE_EMPTY, key | VF_EDGE_ODD);
    if (old == VF_EDGE_EMPTY) return 1;
    if ((old & ~VF_EDGE_ODD) == key) return (atomicXor(J.etab + h, VF_EDGE_ODD) & VF_EDGE_ODD) ? -1 : 1;
    h = (h + 1) & mask;
  }
  return 0;
}

__device__ __forceinline__ void sort3_y(tv* v) {
  tv t;
#define SW(a, b) if (v[a].y > v[b].y) { t = v[a]; v[a] = v[b]; v[b] = t; }
  SW(0, 1) SW(1, 2) SW(0, 1)
#undef SW
}

// per face: NDC vertices sorted by y, the slice planes crossing the face
// (P0.y < ys[s] <= P2.y), and one use of each of its edges; returns the change of
// the job's odd edges
__device__ __forceinline__ int tetra_face(const JobDesc& J, JobState& st, uint32_t f, uint32_t* pcnt) {
  const uint32_t i0 = J.faces[3 * (size_t)f], i1 = J.faces[3 * (size_t)f + 1],
                 i2 = J.faces[3 * (size_t)f + 2];
  if (i0 >= J.nverts || i1 >= J.nverts || i2 >= J.nverts) {
    atomicOr(&st.err, VF_JERR_INVALID);  // bad face: never dereferenced
    J.tet_range[f] = 0xFFFFu;
    *pcnt = 0;
    return 0;
  }
  float ctr[3], dim[3];
  for (int a = 0; a < 3; ++a) {
    ctr[a] = __fmul_rn(0.5f, __fadd_rn(J.amin[a], J.amax[a]));
    dim[a] = __fsub_rn(J.amax[a], J.amin[a]);
  }
  tv v[3];
  v[0] = to_ndc(J.verts + 3 * (size_t)i0, ctr, dim);
  v[1] = to_ndc(J.verts + 3 * (size_t)i1, ctr, dim);
  v[2] = to_ndc(J.verts + 3 * (size_t)i2, ctr, dim);
  sort3_y(v);
  float4* o = J.tets + 3 * (size_t)f;
  o[0] = make_float4(v[0].x, v[0].y, v[0].z, v[1].x);
  o[1] = make_float4(v[1].y, v[1].z, v[2].x, v[2].y);
  o[2] = make_float4(v[2].z, 0.0f, 0.0f, 0.0f);
  const uint32_t s0 = slice_above(J.ys, J.Y, v[0].y);
  const uint32_t s1e = slice_above(J.ys, J.Y, v[2].y);
  J.tet_range[f] = (s1e > s0) ? (s0 | ((s1e - 1) << 16)) : 0xFFFFu;
  *pcnt = s1e > s0 ? s1e - s0 : 0u;  // (face, slice) items
  return edge_use(J, i0, i1) + edge_use(J, i1, i2) + edge_use(J, i2, i0);
}
__global__ void __launch_bounds__(256) k_tetra(const JobDesc* jobs, JobState* st, int njobs, uint32_t total,
                        uint32_t* pcnt) {
  __shared__ int s_odd;
  __shared__ int s_job;
  for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < total; g0 += gridDim.x * blockDim.x) {
    // the odd edges of the CTA's first face's job add up in shared memory
    __syncthreads();
    if (threadIdx.x == 0) {
      s_odd = 0;
      s_job = job_of_face(jobs, njobs, g0);
    }
    __syncthreads();
    int j = s_job;
    const uint32_t g = g0 + threadIdx.x;
    int odd = 0;
    if (g < total) {
      while (j + 1 < njobs && jobs[j + 1].face_base <= g) ++j;
      odd = tetra_face(jobs[j], st[j], g - jobs[j].face_base, pcnt + g);
    }
    const int mine = j == s_job ? odd : 0;
    if (odd && !mine) atomicAdd(&st[j].odd_edges, (uint32_t)odd);
    const int sum = __reduce_add_sync(0xFFFFFFFFu, mine);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&s_odd, sum);
    __syncthreads();
    if (threadIdx.x == 0 && s_odd) atomicAdd(&st[s_job].odd_edges, (uint32_t)s_odd);
  }
}

// ---- exact segment arithmetic (INTERP and the raster rule of the oracle) ---
__device__ __forceinline__ float interp_c(float a, float b, float t) {
  return __fadd_rn(__fmul_rn(a, __fsub_rn(1.0f, t)), __fmul_rn(b, t));
}
__device__ __forceinline__ void interp(const tv& A, const tv& B, float s, float& ox, float& oz) {
  float t = __fdiv_rn(__fsub_rn(s, A.y), __fsub_rn(B.y, A.y));
  ox = interp_c(A.x, B.x, t);
  oz = interp_c(A.z, B.z, t);
}
__device__ __forceinline__ int32_t to_fixed(float ndc, float half) {
  float w = __fadd_rn(__fmul_rn(ndc, half), half);
  return __float2int_rn(__fmul_rn(w, 256.0f));
}
__device__ __forceinline__ int ceil_div_i(int a, int b) {  // b > 0
  return a >= 0 ? (a + b - 1) / b : -((-a) / b);
}
__device__ __forceinline__ long long ceil_div_ll(long long a, long long b) {  // b > 0
  return a >= 0 ? (a + b - 1) / b : -((-a) / b);
}

// markers of one snapped segment in the parity plane of `slice`: per pixel
// row k it crosses, the first pixel column i whose centre the -x ray from
// (centre + (e, e^2)) sees the segment from
__device__ void segment_markers(const JobDesc& J, uint32_t slice, int ax, int az, int bx, int bz) {
  if (az == bz) return;  // horizontal: the ray at z + e^2 never meets it
  int ux = ax, uz = az, vx = bx, vz = bz;
  if (uz > vz) { ux = bx; uz = bz; vx = ax; vz = az; }
  const int klo = max(ceil_div_i(uz - 128, 256), 0);
  const int khi = min(ceil_div_i(vz - 128, 256) - 1, (int)J.Z - 1);
  if (klo > khi) return;
  const long long dz = vz - uz, dx = vx - ux;
  const long long den = 256 * dz;
  uint32_t* const col = J.par + (size_t)slice * J.Zw;
  const size_t istride = (size_t)J.Y * J.Zw;
  for (int k = klo; k <= khi; ++k) {
    // pixel centre x >= u.x + dx (pz - u.z) / dz
    const long long num = dz * ux + dx * ((long long)k * 256 + 128 - uz) - 128 * dz;
    long long i = ceil_div_ll(num, den);
    if (i < 0) i = 0;
    if (i >= (long long)J.X) continue;
    atomicXor(col + (size_t)i * istride + (k >> 5), 1u << (k & 31));
  }
}

// the segment of triangle P (sorted by y, P0.y < sl <= P2.y) in plane sl:
// INTERP on P0-P2 and on P0-P1 or P1-P2 (Tetravoxelizer.cpp:45-89)
__device__ __forceinline__ void face_segment(const JobDesc& J, const tv& P0, const tv& P1,
                                             const tv& P2, uint32_t s) {
  const float sl = J.ys[s];
  float ax, az, bx, bz;
  interp(P0, P2, sl, ax, az);
  const bool lo = sl <= P1.y;
  interp(lo ? P0 : P1, lo ? P1 : P2, sl, bx, bz);
  const float hw = __fmul_rn(0.5f, (float)J.X), hh = __fmul_rn(0.5f, (float)J.Z);
  segment_markers(J, s, to_fixed(ax, hw), to_fixed(az, hh), to_fixed(bx, hw), to_fixed(bz, hh));
}

// ---- exclusive scan of the per-face pair counts (1024 faces per block) -----
__device__ __forceinline__ unsigned long long warp_incl_scan(unsigned long long v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}
// block-wide exclusive scan of one value per thread (blockDim 1024)
__device__ unsigned long long block_excl_scan(unsigned long long v, unsigned long long* total) {
  __shared__ unsigned long long ws[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned long long inc = warp_incl_scan(v);
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    const unsigned long long x = ws[lane];
    ws[lane] = warp_incl_scan(x) - x;
  }
  __syncthreads();
  const unsigned long long r = ws[w] + inc - v;
  if (total && threadIdx.x == blockDim.x - 1) *total = r + v;
  __syncthreads();
  return r;
}
__global__ void __launch_bounds__(1024) k_scan_local(const uint32_t* in, unsigned long long* out,
                                                     unsigned long long* sums, uint32_t n,
                                                     unsigned long long* grand) {
  const uint32_t i = blockIdx.x * 1024u + threadIdx.x;
  const unsigned long long v = i < n ? in[i] : 0ull;
  __shared__ unsigned long long tot;
  const unsigned long long r = block_excl_scan(v, &tot);
  if (i < n) out[i] = r;
  if (threadIdx.x == 0) {
    sums[blockIdx.x] = tot;
    if (gridDim.x == 1) *grand = tot;  // nothing to add
  }
}
// up to 1024 blocks: each adds up the sums before it, and adds them to its own
// values; the last one knows the total
__global__ void __launch_bounds__(1024) k_scan_base(unsigned long long* out, const unsigned long long* sums, uint32_t n,
                                                    unsigned long long* grand) {
  const uint32_t b = blockIdx.x, t = threadIdx.x;
  __shared__ unsigned long long ws[32];
  unsigned long long v = t < b ? sums[t] : 0ull;
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  if ((t & 31) == 0) ws[t >> 5] = v;
  __syncthreads();
  v = ws[t & 31];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  const uint32_t i = b * 1024u + t;
  if (i < n) out[i] += v;
  if (b == gridDim.x - 1 && t == 0) *grand = v + sums[b];
}
__global__ void __launch_bounds__(1024) k_scan_sums(unsigned long long* sums, uint32_t nb,
                                                    unsigned long long* grand) {
  // one block: each thread owns a contiguous chunk of block sums
  const uint32_t per = (nb + 1023) / 1024;
  const uint32_t b0 = threadIdx.x * per, b1 = min(b0 + per, nb);
  unsigned long long acc = 0;
  for (uint32_t b = b0; b < b1; ++b) acc += sums[b];
  __shared__ unsigned long long tot;
  unsigned long long base = block_excl_scan(acc, &tot);
  for (uint32_t b = b0; b < b1; ++b) {
    const unsigned long long t = sums[b];
    sums[b] = base;
    base += t;
  }
  if (threadIdx.x == 0) *grand = tot;
}
__global__ void k_scan_add(unsigned long long* out, const unsigned long long* sums, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += sums[i / 1024u];
}

// Warp-interleaved runs over a flattened work list (faces in batch order,
// items of a face contiguous): a warp owns a run of consecutive items and
// lane l takes items base + l, base + l + 32, ...  Neighbouring lanes work on
// neighbouring items of the same face, so control flow stays coherent and no
// lane idles when a face has few items.  One binary search per warp run; each
// lane then steps its face cursor forward.  A run is an even share of the items
// per warp, 32 to 512: with 512 always, a 12 k face mesh kept one warp per SM
// busy for 16 items in a row (parity 73 us against 14, shell 63 against 14).
__device__ __forceinline__ uint32_t warp_run(unsigned long long total, unsigned long long nwarps) {
  const unsigned long long share = (total + nwarps - 1) / nwarps;
  return 32u * (uint32_t)min(16ull, max(1ull, (share + 31) / 32));
}

__device__ __forceinline__ uint32_t face_of_item(const unsigned long long* base, uint32_t nfaces,
                                                 unsigned long long p) {
  uint32_t lo = 0, hi = nfaces - 1;  // last face whose first item is <= p
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (base[mid] <= p) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(256) k_parity_flat(const JobDesc* jobs, int njobs,
                                                  const uint32_t* pcnt,
                                                  const unsigned long long* pbase,
                                                  const unsigned long long* ptotal,
                                                  uint32_t total_faces) {
  const unsigned long long total = *ptotal;
  const int lane = threadIdx.x & 31;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  const uint32_t run = warp_run(total, nwarps);
  const unsigned long long nwruns = (total + run - 1) / run;
  for (unsigned long long wr = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
       wr < nwruns; wr += nwarps) {
    const unsigned long long base = wr * run;
    const unsigned long long end = min(base + run, total);
    uint32_t g = 0;
    if (lane == 0) g = face_of_item(pbase, total_faces, base);
    g = __shfl_sync(0xFFFFFFFFu, g, 0);
    uint32_t cached = 0xFFFFFFFFu;
    tv P0, P1, P2;
    const JobDesc* J = nullptr;
    uint32_t s0 = 0;
    unsigned long long fb = 0;
    for (unsigned long long p = base + lane; p < end; p += 32) {
      // advance the face cursor (faces with no item have pbase equal to the next)
      while (p >= pbase[g] + pcnt[g]) ++g;
      if (g != cached) {
        cached = g;
        J = &jobs[job_of_face(jobs, njobs, g)];
        const uint32_t f = g - J->face_base;
        const float4* o = J->tets + 3 * (size_t)f;
        const float4 q0 = o[0], q1 = o[1], q2 = o[2];
        P0 = {q0.x, q0.y, q0.z};
        P1 = {q0.w, q1.x, q1.y};
        P2 = {q1.z, q1.w, q2.x};
        s0 = J->tet_range[f] & 0xFFFFu;
        fb = pbase[g];
      }
      face_segment(*J, P0, P1, P2, s0 + (uint32_t)(p - fb));
    }
  }
}

// internal faces (mesh edge + centroid) of the edges used an odd number of
// times: one warp per table word of 32 slots, lanes over the slice planes
__global__ void __launch_bounds__(256) k_odd_edges(const JobDesc* jobs, const JobState* st,
                                                   int njobs) {
  const int lane = threadIdx.x & 31;
  for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
    const JobDesc& J = jobs[j];
    if (!J.nfaces || !J.ecap || !st[j].odd_edges) continue;  // closed meshes have none
    float ctr[3], dim[3];
    for (int a = 0; a < 3; ++a) {
      ctr[a] = __fmul_rn(0.5f, __fadd_rn(J.amin[a], J.amax[a]));
      dim[a] = __fsub_rn(J.amax[a], J.amin[a]);
    }
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < J.ecap / 32;
         w += (gridDim.x * blockDim.x) >> 5) {
      const unsigned long long v = J.etab[w * 32 + lane];
      unsigned m = __ballot_sync(0xFFFFFFFFu, v != VF_EDGE_EMPTY && (v & VF_EDGE_ODD));
      while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const unsigned long long key = __shfl_sync(0xFFFFFFFFu, v, src) & ~VF_EDGE_ODD;
        tv p[3];
        p[0] = to_ndc(J.verts + 3 * (size_t)(uint32_t)(key >> 32), ctr, dim);
        p[1] = to_ndc(J.verts + 3 * (size_t)(uint32_t)key, ctr, dim);
        p[2] = to_ndc(st[j].centroid, ctr, dim);
        sort3_y(p);
        const uint32_t s0 = slice_above(J.ys, J.Y, p[0].y);
        const uint32_t s1e = slice_above(J.ys, J.Y, p[2].y);
        for (uint32_t s = s0 + lane; s < s1e; s += 32) face_segment(J, p[0], p[1], p[2], s);
      }
    }
  }
}

// markers -> parity: prefix XOR along x of every (y, z-word) column.  A CTA takes
// 32 columns, a warp 16 consecutive x of them in registers, 128 x at a time; the
// warps' totals meet in shared memory.  Bound by latency: 476 x 476 x 512 cells 11 us, 128
// mixed jobs 50 us (57 and 76 us with a thread per column; 12 and 91 us with 512 x a CTA).
__global__ void __launch_bounds__(256) k_prefix_x(const JobDesc* jobs, int njobs) {
  __shared__ uint32_t tot[2][8][32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr uint32_t R = 16;
  uint32_t odd = 0;  // the totals of one step are read while the next are written
  for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
    const JobDesc& J = jobs[j];
    if (!J.nfaces) continue;
    const uint32_t cols = J.Y * J.Zw;
    for (uint32_t c0 = 32 * blockIdx.x; c0 < cols; c0 += 32 * gridDim.x) {
      uint32_t* const p = J.par + c0 + lane;
      const bool ok = c0 + lane < cols;
      uint32_t carry = 0;
      for (uint32_t x0 = 0; x0 < J.X; x0 += 8 * R, odd ^= 1) {
        const uint32_t x = x0 + warp * R;
        uint32_t w[R], run = 0;
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) w[k] = ok && x + k < J.X ? p[(size_t)(x + k) * cols] : 0u;
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
          run ^= w[k];
          w[k] = run;
        }
        tot[odd][warp][lane] = run;
        __syncthreads();
        uint32_t before = carry;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          const uint32_t v = tot[odd][k][lane];
          before ^= k < warp ? v : 0u;
          carry ^= v;
        }
#pragma unroll
        for (uint32_t k = 0; k < R; ++k)
          if (ok && x + k < J.X) p[(size_t)(x + k) * cols] = before ^ w[k];
      }
    }
  }
}

// ---- SAT (Intersections3D.h:204-420), FP32 without contraction -----------
struct satd { tv v0, v1, v2, r; };

__device__ __forceinline__ bool ax_test(float pa, float pb, float rad) {
  float mn = pa < pb ? pa : pb, mx = pa < pb ? pb : pa;
  return !(mn > rad || mx < -rad);
}
#define MUL __fmul_rn
#define ADD __fadd_rn
#define SUB __fsub_rn
__device__ __forceinline__ bool x01(const satd& d, float a, float b, float fa, float fb) {
  float p0 = SUB(MUL(a, d.v0.y), MUL(b, d.v0.z)), p2 = SUB(MUL(a, d.v2.y), MUL(b, d.v2.z));
  return ax_test(p0, p2, ADD(MUL(fa, d.r.y), MUL(fb, d.r.z)));
}
__device__ __forceinline__ bool x2(const satd& d, float a, float b, float fa, float fb) {
  float p0 = SUB(MUL(a, d.v0.y), MUL(b, d.v0.z)), p1 = SUB(MUL(a, d.v1.y), MUL(b, d.v1.z));
  return ax_test(p0, p1, ADD(MUL(fa, d.r.y), MUL(fb, d.r.z)));
}
__device__ __forceinline__ bool y02(const satd& d, float a, float b, float fa, float fb) {
  float p0 = ADD(MUL(-a, d.v0.x), MUL(b, d.v0.z)), p2 = ADD(MUL(-a, d.v2.x), MUL(b, d.v2.z));
  return ax_test(p0, p2, ADD(MUL(fa, d.r.x), MUL(fb, d.r.z)));
}
__device__ __forceinline__ bool y1(const satd& d, float a, float b, float fa, float fb) {
  float p0 = ADD(MUL(-a, d.v0.x), MUL(b, d.v0.z)), p1 = ADD(MUL(-a, d.v1.x), MUL(b, d.v1.z));
  return ax_test(p0, p1, ADD(MUL(fa, d.r.x), MUL(fb, d.r.z)));
}
__device__ __forceinline__ bool z12(const satd& d, float a, float b, float fa, float fb) {
  float p1 = SUB(MUL(a, d.v1.x), MUL(b, d.v1.y)), p2 = SUB(MUL(a, d.v2.x), MUL(b, d.v2.y));
  // zAxisTest_12 orders (p2, p1): same min/max
  return ax_test(p1, p2, ADD(MUL(fa, d.r.x), MUL(fb, d.r.y)));
}
__device__ __forceinline__ bool z0(const satd& d, float a, float b, float fa, float fb) {
  float p0 = SUB(MUL(a, d.v0.x), MUL(b, d.v0.y)), p1 = SUB(MUL(a, d.v1.x), MUL(b, d.v1.y));
  return ax_test(p0, p1, ADD(MUL(fa, d.r.x), MUL(fb, d.r.y)));
}
__device__ __forceinline__ void mm3(float a, float b, float c, float& mn, float& mx) {
  mn = mx = a;
  if (b < mn) mn = b;
  if (b > mx) mx = b;
  if (c < mn) mn = c;
  if (c > mx) mx = c;
}
// The SAT, every test evaluated as Intersections3D.h:204-258 does.
__device__ __forceinline__ bool tri_box(const tv& p0, const tv& p1, const tv& p2, const tv& c, const tv& r) {
  satd d;
  d.r = r;
  d.v0 = {SUB(p0.x, c.x), SUB(p0.y, c.y), SUB(p0.z, c.z)};
  d.v1 = {SUB(p1.x, c.x), SUB(p1.y, c.y), SUB(p1.z, c.z)};
  d.v2 = {SUB(p2.x, c.x), SUB(p2.y, c.y), SUB(p2.z, c.z)};
  tv e0 = {SUB(d.v1.x, d.v0.x), SUB(d.v1.y, d.v0.y), SUB(d.v1.z, d.v0.z)};
  tv e1 = {SUB(d.v2.x, d.v1.x), SUB(d.v2.y, d.v1.y), SUB(d.v2.z, d.v1.z)};
  tv e2 = {SUB(d.v0.x, d.v2.x), SUB(d.v0.y, d.v2.y), SUB(d.v0.z, d.v2.z)};
  float fx = fabsf(e0.x), fy = fabsf(e0.y), fz = fabsf(e0.z);
  if (!x01(d, e0.z, e0.y, fz, fy)) return false;
  if (!y02(d, e0.z, e0.x, fz, fx)) return false;
  if (!z12(d, e0.y, e0.x, fy, fx)) return false;
  fx = fabsf(e1.x); fy = fabsf(e1.y); fz = fabsf(e1.z);
  if (!x01(d, e1.z, e1.y, fz, fy)) return false;
  if (!y02(d, e1.z, e1.x, fz, fx)) return false;
  if (!z0(d, e1.y, e1.x, fy, fx)) return false;
  fx = fabsf(e2.x); fy = fabsf(e2.y); fz = fabsf(e2.z);
  if (!x2(d, e2.z, e2.y, fz, fy)) return false;
  if (!y1(d, e2.z, e2.x, fz, fx)) return false;
  if (!z12(d, e2.y, e2.x, fy, fx)) return false;
  float mn, mx;
  mm3(d.v0.x, d.v1.x, d.v2.x, mn, mx);
  if (mn > d.r.x || mx < -d.r.x) return false;
  mm3(d.v0.y, d.v1.y, d.v2.y, mn, mx);
  if (mn > d.r.y || mx < -d.r.y) return false;
  mm3(d.v0.z, d.v1.z, d.v2.z, mn, mx);
  if (mn > d.r.z || mx < -d.r.z) return false;
  tv n = {SUB(MUL(e0.y, e1.z), MUL(e1.y, e0.z)), SUB(MUL(e0.z, e1.x), MUL(e1.z, e0.x)),
          SUB(MUL(e0.x, e1.y), MUL(e1.x, e0.y))};
  // planeBoxOverlap
  float nv[3] = {n.x, n.y, n.z}, vv[3] = {d.v0.x, d.v0.y, d.v0.z}, m[3] = {r.x, r.y, r.z};
  float vmin[3], vmax[3];
  for (int q = 0; q < 3; ++q) {
    if (nv[q] > 0.0f) { vmin[q] = SUB(-m[q], vv[q]); vmax[q] = SUB(m[q], vv[q]); }
    else { vmin[q] = SUB(m[q], vv[q]); vmax[q] = SUB(-m[q], vv[q]); }
  }
  if (ADD(ADD(MUL(nv[0], vmin[0]), MUL(nv[1], vmin[1])), MUL(nv[2], vmin[2])) > 0.0f) return false;
  if (ADD(ADD(MUL(nv[0], vmax[0]), MUL(nv[1], vmax[1])), MUL(nv[2], vmax[2])) >= 0.0f) return true;
  return false;
}

// the voxel box of cell (i, j, k) as RegularGrid::getAABBs builds it
__device__ __forceinline__ void cell_box(const JobDesc& J, const float* cs, int i, int jj, int k,
                                         tv& ce, tv& r) {
  tv bmin = {ADD(J.amin[0], MUL(cs[0], (float)i)), ADD(J.amin[1], MUL(cs[1], (float)jj)),
             ADD(J.amin[2], MUL(cs[2], (float)k))};
  tv bmax = {ADD(bmin.x, cs[0]), ADD(bmin.y, cs[1]), ADD(bmin.z, cs[2])};
  // (max + min) / 2: x * 0.5 and x / 2 are the same correctly rounded value
  ce = {MUL(ADD(bmax.x, bmin.x), 0.5f), MUL(ADD(bmax.y, bmin.y), 0.5f),
        MUL(ADD(bmax.z, bmin.z), 0.5f)};
  r = {SUB(bmax.x, ce.x), SUB(bmax.y, ce.y), SUB(bmax.z, ce.z)};
}

__device__ __forceinline__ int float_cell(float f, int n) {
  if (!(f > -1.0e9f)) f = -1.0e9f;
  if (f > 1.0e9f) f = 1.0e9f;
  return vf_clampi((int)floorf(f), -2, n + 1);
}

// The shell marks every cell whose box the float SAT above accepts.  The SAT
// itself runs for few cells: with the face's column axis c (the axis of its
// largest normal component) and a column of cells (a, b), each of its 13 tests
// is, in exact arithmetic, either the same for the whole column or an interval
// of positions along c.  Per face the tests are written as linear forms in cell
// units relative to the face's first vertex; per column their intervals are
// intersected twice, once widened and once narrowed by a margin m above the
// rounding of the float SAT and of the forms:
//   outside the wide one    no float test can accept: no hit
//   inside the narrow one   no float test can reject: a hit, marked at once
//   in between              the SAT decides
// With M the largest coordinate in play and eps = 2^-24 M, the SAT's box centres,
// half sizes and vertex offsets carry at most 10 eps, its edges 6 eps, so a test
// on an edge (e, f) with offsets up to D carries at most
// (24 (|e| + |f|) + 12 D + 6 cells) eps, and its form here (13 (|e| + |f|) + 6 D)
// eps; the margin is 48 (|e| + |f| + D) eps, and likewise for the plane.
// Coordinates far from the origin only widen it: then the SAT decides more cells.
// Work items are columns; faces whose normal has no clear axis (slivers) leave
// every cell of their box, in columns along z, to the SAT.
struct ShellBox {
  int lo[3], n[3];  // cells touching the triangle's box along x, y, z
  float M;          // largest coordinate in play
  int c;            // column axis
  bool prune;       // by columns
  uint32_t items;
};

template <class T>
__device__ __forceinline__ T sel3(const T* v, int i) {  // a register select
  return i == 0 ? v[0] : (i == 1 ? v[1] : v[2]);
}

__device__ bool shell_box(const JobDesc& J, uint32_t f, float q0[3], float q1[3], float q2[3], ShellBox& S) {
  const int dims[3] = {(int)J.X, (int)J.Y, (int)J.Z};
  const uint32_t* fi = J.faces + 3 * (size_t)f;
  const uint32_t i0 = fi[0], i1 = fi[1], i2 = fi[2];
  if (i0 >= J.nverts || i1 >= J.nverts || i2 >= J.nverts) return false;
  S.M = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    q0[a] = J.verts[3 * (size_t)i0 + a];
    q1[a] = J.verts[3 * (size_t)i1 + a];
    q2[a] = J.verts[3 * (size_t)i2 + a];
    S.M = fmaxf(S.M, fmaxf(fabsf(J.amin[a]), fabsf(J.amax[a])));
    S.M = fmaxf(S.M, fmaxf(fabsf(q0[a]), fmaxf(fabsf(q1[a]), fabsf(q2[a]))));
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float mn, mx;
    mm3(q0[a], q1[a], q2[a], mn, mx);
    // Cells that touch the triangle's extent along a, widened by 0.01 cell +
    // 256 ulp of M: a cell further out fails the exact SAT's box-axis test,
    // whose roundings are a few ulp of M; the 0.01 cell covers the rounding
    // of these index computations (below 2^-11 cell for 4096 cells).
    const float mc = 0.01f + 4.0f * (S.M * 7.62939453125e-6f) * J.ics[a];
    S.lo[a] = vf_clampi(float_cell(SUB(mn, J.amin[a]) * J.ics[a] - mc, dims[a]), 0, dims[a] - 1);
    const int hi = vf_clampi(float_cell(SUB(mx, J.amin[a]) * J.ics[a] + mc, dims[a]), 0, dims[a] - 1);
    S.n[a] = hi - S.lo[a] + 1;
  }
  const float e1[3] = {q1[0] - q0[0], q1[1] - q0[1], q1[2] - q0[2]};
  const float e2[3] = {q2[0] - q0[0], q2[1] - q0[1], q2[2] - q0[2]};
  const float nr[3] = {fabsf(e1[1] * e2[2] - e1[2] * e2[1]), fabsf(e1[2] * e2[0] - e1[0] * e2[2]),
                       fabsf(e1[0] * e2[1] - e1[1] * e2[0])};
  int c = nr[1] > nr[0] ? 1 : 0;
  if (nr[2] > (c ? nr[1] : nr[0])) c = 2;
  const float e1n = fabsf(e1[0]) + fabsf(e1[1]) + fabsf(e1[2]);
  const float e2n = fabsf(e2[0]) + fabsf(e2[1]) + fabsf(e2[2]);
  const float nrc = sel3(nr, c);
  S.prune = nrc > 1e-3f * e1n * e2n && nrc > 0.0f;
  S.c = S.prune ? c : 2;
  const int ax = c == 2 ? 0 : c + 1, bx = c == 0 ? 2 : c - 1;
  S.items = S.prune ? (uint32_t)(sel3(S.n, ax) * sel3(S.n, bx)) : (uint32_t)(S.n[0] * S.n[1]);
  return true;
}

// The faces are taken in groups of 32, a lane each; a group's items in even units
// of at most `run`.  A unit builds the forms of its faces again, so units are
// long, but no longer than what gives every warp of the GPU a few.
__host__ __device__ inline uint32_t shell_run(uint32_t groups) {
  const uint32_t r = groups / 32 & ~31u;
  return r < 64 ? 64 : (r > 1024 ? 1024 : r);
}
__device__ __forceinline__ int group_job(const JobDesc* jobs, int njobs, uint32_t g0, uint32_t g) {
  int j = job_of_face(jobs, njobs, g0);
  while (j + 1 < njobs && jobs[j + 1].face_base <= g) ++j;
  return j;
}
__global__ void __launch_bounds__(256) k_shell_count(const JobDesc* jobs, int njobs, uint32_t total, uint32_t* units) {
  const uint32_t groups = (total + 31) / 32, run = shell_run(groups), lane = threadIdx.x & 31;
  for (uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < groups; p += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t g = 32 * p + lane;
    unsigned long long items = 0;
    if (g < total) {
      const JobDesc& J = jobs[group_job(jobs, njobs, 32 * p, g)];
      ShellBox S;
      float q0[3], q1[3], q2[3];
      if (shell_box(J, g - J.face_base, q0, q1, q2, S)) items = S.items;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) items += __shfl_xor_sync(0xFFFFFFFFu, items, o);
    if (lane == 0) units[p] = (uint32_t)((items + run - 1) / run);
  }
}

// A face's forms in shared memory, 13 uint4 (an odd number: 8 faces' loads of
// one uint4 fall on distinct bank groups):
//   0 first item of the face in the unit, 2^32 / n_b, n_b | n_c << 16, job
//   1 lo_a | lo_b << 16, lo_c | c << 16, sure cells a, b (lo | end << 16)
//   2 centre of cell (lo_a, lo_b, lo_c) fa fb fc, sure cells c
//   3-5 column tests: |x a + y b - z| <= 1, sure below w
//   6-11 tests along c: centre x v + y, half widths z (wide), w (narrow), v = b
//        (6-8) or a (9-11)
//   12 plane: centre x a + y b, half widths z, w
constexpr int SHELL_REC = 13;
__device__ __forceinline__ void shell_forms(const JobDesc& J, const ShellBox& S, const float q0[3], const float q1[3],
                                            const float q2[3], uint32_t first, uint32_t job, uint4* rec) {
  const int c = S.c, ax = c == 2 ? 0 : c + 1, bx = c == 0 ? 2 : c - 1;
  const int lo_a = sel3(S.lo, ax), lo_b = sel3(S.lo, bx), lo_c = sel3(S.lo, c);
  const int n_a = sel3(S.n, ax), n_b = sel3(S.n, bx), n_c = sel3(S.n, c);
  rec[0] = make_uint4(first, 0xFFFFFFFFu / (uint32_t)n_b, (uint32_t)(n_b | n_c << 16), job);
  const uint32_t w10 = (uint32_t)(lo_a | lo_b << 16), w11 = (uint32_t)(lo_c | c << 16);
  rec[1] = make_uint4(w10, w11, 0u, 0u);
  // cell units: vertices relative to the first
  float V1[3], V2[3], F[3], mn[3], mx[3], ext = 0.0f, mics = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    V1[a] = (q1[a] - q0[a]) * J.ics[a];
    V2[a] = (q2[a] - q0[a]) * J.ics[a];
    F[a] = ((J.amin[a] - q0[a]) + J.cs[a] * ((float)S.lo[a] + 0.5f)) * J.ics[a];
    mn[a] = fminf(0.0f, fminf(V1[a], V2[a]));
    mx[a] = fmaxf(0.0f, fmaxf(V1[a], V2[a]));
    ext = fmaxf(ext, mx[a] - mn[a]);
    mics = fmaxf(mics, J.ics[a]);
  }
  const float V1a = sel3(V1, ax), V1b = sel3(V1, bx), V1c = sel3(V1, c);
  const float V2a = sel3(V2, ax), V2b = sel3(V2, bx), V2c = sel3(V2, c);
  const float fa = sel3(F, ax), fb = sel3(F, bx), fc = sel3(F, c);
  const float u = S.M * mics * 2.86102294921875e-6f;  // 48 * 2^-24
  const float D = ext + 0.6f + 12.0f * u;             // largest offset of a vertex from a cell of the box
  const float Na = V1b * V2c - V1c * V2b, Nb = V1c * V2a - V1a * V2c, Nc = V1a * V2b - V1b * V2a;
  float4* const r4 = reinterpret_cast<float4*>(rec);
  if (!S.prune || !(u < 1.0f) || !(fabsf(Nc) > 1e-20f)) {
    // no clear axis, or a margin above a cell: every cell of the box through the SAT
    r4[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int i = 3; i < 6; ++i) r4[i] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    for (int i = 6; i < 13; ++i) r4[i] = make_float4(0.0f, 0.0f, 1e30f, -1.0f);
    return;
  }
  // sure cells of the box axes, relative to lo: lo | end << 16
  auto sure = [&](float lo, float hi, float f, int n) {
    const float m = 0.001f + u;
    const int k0 = max(0, min(n, __float2int_ru(lo - 0.5f - f + m)));
    const int k1 = max(k0, min(n - 1, __float2int_rd(hi + 0.5f - f - m)) + 1);
    return (uint32_t)(k0 | k1 << 16);
  };
  rec[1] = make_uint4(w10, w11, sure(sel3(mn, ax), sel3(mx, ax), fa, n_a), sure(sel3(mn, bx), sel3(mx, bx), fb, n_b));
  rec[2] = make_uint4(__float_as_uint(fa), __float_as_uint(fb), __float_as_uint(fc),
                      sure(sel3(mn, c), sel3(mx, c), fc, n_c));
  // edges 0 (V0 -> V1), 1 (V1 -> V2), 2 (V2 -> V0); (on) a vertex of the edge, (off) the third
  const float Ea[3] = {V1a, V2a - V1a, -V2a}, Eb[3] = {V1b, V2b - V1b, -V2b}, Ec[3] = {V1c, V2c - V1c, -V2c};
  const float on_a[3] = {0.0f, V2a, 0.0f}, on_b[3] = {0.0f, V2b, 0.0f}, on_c[3] = {0.0f, V2c, 0.0f};
  const float off_a[3] = {V2a, 0.0f, V1a}, off_b[3] = {V2b, 0.0f, V1b}, off_c[3] = {V2c, 0.0f, V1c};
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    {  // axis e x c: e_a x_b - e_b x_a, the same along the column
      const float s0 = Ea[e] * on_b[e] - Eb[e] * on_a[e], s1 = Ea[e] * off_b[e] - Eb[e] * off_a[e];
      const float E = fabsf(Ea[e]) + fabsf(Eb[e]), half = 0.5f * (fabsf(s1 - s0) + E), m = u * (E + D);
      const float r = __fdividef(1.0f, half + m);
      r4[3 + e] = make_float4(-Eb[e] * r, Ea[e] * r, 0.5f * (s0 + s1) * r, (half - m) * r);
    }
    {  // axis e x a: e_c x_b - e_b x_c; a slope divisor below u is taken as u (the second D covers it)
      const float s0 = Ec[e] * on_b[e] - Eb[e] * on_c[e], s1 = Ec[e] * off_b[e] - Eb[e] * off_c[e];
      const float E = fabsf(Ec[e]) + fabsf(Eb[e]), half = 0.5f * (fabsf(s1 - s0) + E), m = u * (E + 2.0f * D);
      const float ir = __fdividef(1.0f, fmaxf(fabsf(Eb[e]), u)), r = copysignf(ir, Eb[e]);
      r4[6 + e] = make_float4(Ec[e] * r, -0.5f * (s0 + s1) * r, (half + m) * ir, (half - m) * ir);
    }
    {  // axis e x b: e_c x_a - e_a x_c
      const float s0 = Ec[e] * on_a[e] - Ea[e] * on_c[e], s1 = Ec[e] * off_a[e] - Ea[e] * off_c[e];
      const float E = fabsf(Ec[e]) + fabsf(Ea[e]), half = 0.5f * (fabsf(s1 - s0) + E), m = u * (E + 2.0f * D);
      const float ir = __fdividef(1.0f, fmaxf(fabsf(Ea[e]), u)), r = copysignf(ir, Ea[e]);
      r4[9 + e] = make_float4(Ec[e] * r, -0.5f * (s0 + s1) * r, (half + m) * ir, (half - m) * ir);
    }
  }
  const float En = fabsf(V1a) + fabsf(V1b) + fabsf(V1c) + fabsf(V2a) + fabsf(V2b) + fabsf(V2c);
  const float Nn = fabsf(Na) + fabsf(Nb) + fabsf(Nc), in = 1.0f / Nc;
  const float m = u * (2.0f * En * D + Nn);
  r4[12] = make_float4(-Na * in, -Nb * in, (0.5f * Nn + m) * fabsf(in), (0.5f * Nn - m) * fabsf(in));
}

__device__ __forceinline__ void red_or(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// the SAT of one queued cell (face, job, x | y << 16, z) and the mark
__device__ __forceinline__ void shell_cell(const JobDesc* jobs, const uint4& e) {
  const JobDesc& J = jobs[e.y];
  const uint32_t* fi = J.faces + 3 * (size_t)(e.x - J.face_base);
  const float* p0 = J.verts + 3 * (size_t)fi[0];
  const float* p1 = J.verts + 3 * (size_t)fi[1];
  const float* p2 = J.verts + 3 * (size_t)fi[2];
  const int x = e.z & 0xFFFF, y = e.z >> 16, z = e.w;
  tv ce, r;
  cell_box(J, J.cs, x, y, z, ce, r);
  if (tri_box({p0[0], p0[1], p0[2]}, {p1[0], p1[1], p1[2]}, {p2[0], p2[1], p2[2]}, ce, r))
    red_or(J.shell + ((size_t)x * J.Y + y) * J.Zw + (z >> 5), 1u << (z & 31));
}

// A warp per unit: a lane builds a face's forms in shared memory, then the lanes
// take the columns of the unit's faces.  Cells the forms leave open go to the
// warp's queue, and through the SAT 32 at a time.
// Bound by instruction issue (69% of cycles; 0.5 cells a face go to the SAT): 128
// meshes, 6.4 M faces of 8 to 19 columns, 1575 us, and 48 of them 494 us, against
// 3396 and 1104 us with the SAT's column tests and then the SAT for every cell.
constexpr int SHELL_WARPS = 8;
struct ShellWarp {
  uint4 rec[32 * SHELL_REC];
  uint4 queue[64];     // cells for the SAT
  uint32_t cols[64];   // columns kept: face of the group | da << 5 | db << 18 | sure << 31
  uint32_t start[36];  // first item of each face in the unit, and the end
};
__global__ void __launch_bounds__(SHELL_WARPS * 32, 3)
    k_shell_flat(const JobDesc* jobs, int njobs, const unsigned long long* ubase, const unsigned long long* utotal,
                 uint32_t total_faces) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ShellWarp& W = reinterpret_cast<ShellWarp*>(smem_raw)[threadIdx.x >> 5];
  const unsigned long long total = *utotal;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  const uint32_t groups = (total_faces + 31) / 32, run = shell_run(groups);
  uint32_t queued = 0;  // the same in all lanes, below 32 between rounds
  for (unsigned long long unit = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5; unit < total;
       unit += nwarps) {
    uint32_t p = 0;
    if (lane == 0) p = face_of_item(ubase, groups, unit);
    p = __shfl_sync(0xFFFFFFFFu, p, 0);
    const unsigned long long ub = ubase[p], units = (p + 1 < groups ? ubase[p + 1] : total) - ub;
    const uint32_t g0 = 32 * p, g = g0 + lane;
    {
      const int j = g < total_faces ? group_job(jobs, njobs, g0, g) : 0;
      ShellBox S;
      float q0[3], q1[3], q2[3];
      const bool ok = g < total_faces && shell_box(jobs[j], g - jobs[j].face_base, q0, q1, q2, S);
      const unsigned long long items = ok ? S.items : 0u;
      unsigned long long upto = items;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, upto, o);
        if (lane >= o) upto += t;
      }
      const unsigned long long first = upto - items;
      // the unit's share of the group's items
      const unsigned long long all = __shfl_sync(0xFFFFFFFFu, upto, 31);
      const uint32_t share = units == 1 ? run : (uint32_t)((all + units - 1) / units);
      const unsigned long long from = (unit - ub) * share;
      auto clip = [&](unsigned long long i) { return (uint32_t)min((unsigned long long)share, i > from ? i - from : 0ull); };
      const uint32_t s0 = clip(first), s1 = clip(upto);
      __syncwarp();  // the previous unit's forms are read
      W.start[lane] = s0;
      if (lane == 31) W.start[32] = s1;
      if (s0 < s1) shell_forms(jobs[j], S, q0, q1, q2, (uint32_t)(first - from), (uint32_t)j, W.rec + lane * SHELL_REC);
      __syncwarp();
    }
    // Columns (slot, da, db) the tests across the face keep are collected, then
    // taken 32 at a time.
    const uint32_t stop = W.start[32];
    uint32_t slot = 0, ncols = 0;
    for (uint32_t i0 = 0; i0 < stop || ncols; i0 += 32) {
      const uint32_t i = i0 + lane;
      bool keep = false;
      uint32_t col = 0;
      if (i < stop) {
        while (i >= W.start[slot + 1]) ++slot;
        const uint4* rec = W.rec + slot * SHELL_REC;
        const float4* r4 = reinterpret_cast<const float4*>(rec);
        const uint4 h0 = rec[0], h1 = rec[1];
        const uint32_t q = i - h0.x, n_b = h0.z & 0xFFFFu;
        uint32_t da = __umulhi(q, h0.y), db = q - da * n_b;
        if (db >= n_b) { ++da; db -= n_b; }  // the rounded-down reciprocal is at most 1 short
        const float4 h2 = r4[2];
        const float xa = (float)da + h2.x, xb = (float)db + h2.y;
        uint32_t sure = da >= (h1.z & 0xFFFFu) && da < (h1.z >> 16) && db >= (h1.w & 0xFFFFu) && db < (h1.w >> 16);
        keep = true;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const float4 t = r4[3 + e];
          const float d = fabsf(fmaf(t.x, xa, fmaf(t.y, xb, -t.z)));
          keep &= !(d > 1.0f);
          sure &= d < t.w;
        }
        col = slot | da << 5 | db << 18 | sure << 31;
      }
      const unsigned mk = __ballot_sync(0xFFFFFFFFu, keep);
      if (keep) W.cols[ncols + __popc(mk & lt)] = col;
      ncols += __popc(mk);
      if (ncols < 32 && i0 + 32 < stop) continue;
      __syncwarp();
      uint32_t face = 0, job = 0;
      int c = 2, ia = 0, ib = 0;  // the column, and cells open to the SAT:
      int k0 = 0, n0 = 0, k1 = 0, n1 = 0;
      if (lane < (int)ncols) {
        const uint32_t e = W.cols[lane], da = (e >> 5) & 0x1FFFu, db = (e >> 18) & 0x1FFFu;
        const uint4* rec = W.rec + (e & 31u) * SHELL_REC;
        const float4* r4 = reinterpret_cast<const float4*>(rec);
        const uint4 h0 = rec[0], h1 = rec[1];
        const float4 h2 = r4[2];
        face = g0 + (e & 31u);
        job = h0.w;
        const int lo_c = h1.y & 0xFFFF, n_c = (int)(h0.z >> 16);
        c = (h1.y >> 16) & 3;
        ia = (int)((h1.x & 0xFFFFu) + da);
        ib = (int)((h1.x >> 16) + db);
        const float xa = (float)da + h2.x, xb = (float)db + h2.y;
        float wlo = -1e30f, whi = 1e30f, nlo = -1e30f, nhi = 1e30f;
        auto along = [&](float at, float w, float n) {
          wlo = fmaxf(wlo, at - w); whi = fminf(whi, at + w);
          nlo = fmaxf(nlo, at - n); nhi = fminf(nhi, at + n);
        };
#pragma unroll
        for (int t3 = 0; t3 < 3; ++t3) {
          const float4 t = r4[6 + t3];
          along(fmaf(t.x, xb, t.y), t.z, t.w);
        }
#pragma unroll
        for (int t3 = 0; t3 < 3; ++t3) {
          const float4 t = r4[9 + t3];
          along(fmaf(t.x, xa, t.y), t.z, t.w);
        }
        const float4 t = r4[12];
        along(fmaf(t.x, xa, t.y * xb), t.z, t.w);
        // cells relative to lo_c; 0.001 covers the rounding of these sums
        const uint32_t kc = __float_as_uint(h2.w);
        const int a0 = max(0, __float2int_ru(wlo - h2.z - 0.001f));
        const int a1 = min(n_c - 1, __float2int_rd(whi - h2.z + 0.001f)) + 1;
        int b0 = max(max((int)(kc & 0xFFFFu), a0), __float2int_ru(nlo - h2.z + 0.001f));
        int b1 = min(min((int)(kc >> 16), a1) - 1, __float2int_rd(nhi - h2.z - 0.001f)) + 1;
        if (!(e >> 31) || b1 <= b0) b0 = b1 = max(a0, a1);
        // [a0, b0) open, [b0, b1) hits, [b1, a1) open
        k0 = lo_c + a0; n0 = max(b0 - a0, 0);
        k1 = lo_c + b1; n1 = max(a1 - b1, 0);
        if (b1 > b0) {
          const JobDesc& J = jobs[job];
          int k = lo_c + b0;
          const int ke = lo_c + b1;
          if (c == 2) {
            uint32_t* row = J.shell + ((size_t)ia * J.Y + ib) * J.Zw;
            while (k < ke) {
              const int w = k >> 5, stop_k = min(ke, (w + 1) << 5);
              red_or(row + w, (0xFFFFFFFFu << (k & 31)) & (0xFFFFFFFFu >> (31 - ((stop_k - 1) & 31))));
              k = stop_k;
            }
          } else {
            // c = 0: (x, y, z) = (k, a, b); c = 1: (b, k, a)
            const int z = c == 0 ? ib : ia;
            const size_t row = c == 0 ? (size_t)k * J.Y + ia : (size_t)ib * J.Y + k;
            const size_t step = c == 0 ? (size_t)J.Y * J.Zw : J.Zw;
            uint32_t* w = J.shell + row * J.Zw + (z >> 5);
            for (; k < ke; ++k, w += step) red_or(w, 1u << (z & 31));
          }
        }
      }
      const uint32_t done = min(ncols, 32u);
      ncols -= done;
      const uint32_t left = W.cols[32 + lane];
      __syncwarp();
      if (lane < (int)ncols) W.cols[lane] = left;
      for (unsigned m; (m = __ballot_sync(0xFFFFFFFFu, n0 + n1 > 0)) != 0;) {
        if (n0 + n1 > 0) {
          const int k = n0 > 0 ? k0 : k1;
          if (n0 > 0) { ++k0; --n0; } else { ++k1; --n1; }
          const int x = c == 0 ? k : (c == 1 ? ib : ia), y = c == 0 ? ia : (c == 1 ? k : ib),
                    z = c == 0 ? ib : (c == 1 ? ia : k);
          W.queue[queued + __popc(m & lt)] = make_uint4(face, job, (uint32_t)(x | y << 16), (uint32_t)z);
        }
        queued += __popc(m);
        if (queued >= 32) {
          __syncwarp();
          shell_cell(jobs, W.queue[lane]);
          queued -= 32;
          const uint4 rest = W.queue[32 + lane];
          __syncwarp();
          if (lane < (int)queued) W.queue[lane] = rest;
        }
      }
    }
  }
  __syncwarp();
  if (lane < (int)queued) shell_cell(jobs, W.queue[lane]);
}
#undef MUL
#undef ADD
#undef SUB

// One CTA per brick, four lanes per (x, y) row: a row of the brick is one word of
// the bit planes (bits at z >= Z are never set, so the row padding is written as
// 0) and four 16-byte label units.
// grid2 (the second label buffer) needs zeros in bricks that are not live:
// stencil tiles read their halo from them.  Live bricks of grid2 are written
// in full by the first stage that targets it, so only non-live bricks are
// cleared there (dual != 0).  Bound by the stores: 240 x 240 x 256 voxels 13 us, 128
// mixed jobs (0.8 G voxels) 637 us; a warp per row of a column of bricks, most lanes
// past the row's end, took 55 and 846 us.
__global__ void __launch_bounds__(256) k_combine(const JobDesc* jobs, const uint32_t* brick_job,
                                                 uint32_t total, uint8_t* live, int dual) {
  for (uint32_t b = blockIdx.x; b < total; b += gridDim.x) {
    const JobDesc& J = jobs[brick_job[b]];
    const uint32_t lb = b - J.brick_base;
    const uint32_t bz = lb % J.nbz, by = (lb / J.nbz) % J.nby, bx = lb / (J.nbz * J.nby);
    const uint32_t q = threadIdx.x & 3, z = bz * VF_BZ + 8 * q;
    uint32_t word[4];
    size_t at[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t row = 64 * k + (threadIdx.x >> 2);
      const uint32_t x = bx * VF_BX + row / VF_BY, y = by * VF_BY + row % VF_BY;
      const bool ok = x < J.X && y < J.Y;
      at[k] = ok ? (size_t)x * J.Y + y : ~(size_t)0;
      word[k] = ok ? J.par[at[k] * J.Zw + bz] | J.shell[at[k] * J.Zw + bz] : 0u;
    }
    const bool occ = __syncthreads_or((word[0] | word[1] | word[2] | word[3]) != 0u);
    if (threadIdx.x == 0) live[b] = occ;
    if (z >= J.Zp) continue;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (at[k] == ~(size_t)0) continue;
      const uint32_t bits = word[k] >> (8 * q);
      auto pair = [](uint32_t v) { return ((v & 3u) * 0x8001u) & 0x00010001u; };
      *reinterpret_cast<uint4*>(J.grid + at[k] * J.Zp + z) =
          make_uint4(pair(bits), pair(bits >> 2), pair(bits >> 4), pair(bits >> 6));
      if (dual && !occ) *reinterpret_cast<uint4*>(J.grid2 + at[k] * J.Zp + z) = make_uint4(0, 0, 0, 0);
    }
  }
}

__global__ void __launch_bounds__(256) k_mark_live(const JobDesc* jobs, const uint32_t* brick_job,
                                                   uint32_t total, uint8_t* live) {
  for (uint32_t b = blockIdx.x; b < total; b += gridDim.x) {
    const JobDesc& J = jobs[brick_job[b]];
    const uint32_t lb = b - J.brick_base;
    const uint32_t bz = lb % J.nbz, by = (lb / J.nbz) % J.nby, bx = lb / (J.nbz * J.nby);
    const uint32_t x = bx * VF_BX + threadIdx.x / VF_BY, y = by * VF_BY + threadIdx.x % VF_BY;
    const uint32_t z0 = bz * VF_BZ;
    int any = 0;
    if (x < J.X && y < J.Y) {
      const uint32_t nz = min((uint32_t)VF_BZ, J.Zp - z0);
      const uint4* src = reinterpret_cast<const uint4*>(J.grid + vf_gidx(J, x, y, z0));
      for (uint32_t q = 0; q < nz / 8; ++q) {
        uint4 v = src[q];
        any |= (v.x | v.y | v.z | v.w) != 0;
      }
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) live[b] = any ? 1 : 0;
  }
}

// the live ones of bricks [first, first + total)
__global__ void k_compact(const uint8_t* live, uint32_t first, uint32_t total, uint32_t* list, uint32_t* count) {
  const int lane = threadIdx.x & 31;
  // grid-stride over bricks, warp-aggregated append (ballot + popc)
  for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < total;
       i0 += gridDim.x * blockDim.x) {
    const uint32_t i = i0 + lane;
    const bool keep = i < total && live[first + i];
    const unsigned m = __ballot_sync(0xFFFFFFFFu, keep);
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (keep) list[base + __popc(m & ((1u << lane) - 1u))] = first + i;
  }
}

}  // namespace

namespace vfk {

static inline int grid_for(uint32_t n, int per, int cap) {
  uint64_t g = (n + (uint64_t)per - 1) / per;
  if (g < 1) g = 1;
  if (g > (uint64_t)cap) g = cap;
  return (int)g;
}

void centroid_and_slices(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs) {
  if (njobs <= 0) return;
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_centroid, cudaFuncAttributeMaxDynamicSharedMemorySize, CEN_BYTES);
    attr[dv] = true;
  }
  k_centroid<<<njobs * CEN_CTAS, CEN_LANES, CEN_BYTES, st>>>(dj, ds);
}
void tetra_prep(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs,
                uint32_t total_faces, const FaceScratch& fs) {
  if (total_faces)
    k_tetra<<<grid_for(total_faces, 256, 65535), 256, 0, st>>>(dj, ds, njobs, total_faces, fs.pcnt);
}
void parity_raster(cudaStream_t st, const JobDesc* dj, const JobState* ds, int njobs,
                   uint32_t total_faces, const FaceScratch& fs, int num_sms, int grid_mult) {
  if (!total_faces) return;
  exclusive_scan(st, fs.pcnt, fs.pbase, fs.psums, total_faces, fs.ptotal);
  k_parity_flat<<<num_sms * grid_mult, 256, 0, st>>>(dj, njobs, fs.pcnt, fs.pbase, fs.ptotal, total_faces);
  const unsigned gy = (unsigned)(njobs < 65535 ? njobs : 65535);
  k_odd_edges<<<dim3(std::max(1, num_sms * 8 / njobs), gy), 256, 0, st>>>(dj, ds, njobs);
  const int px = std::max(1, num_sms * 16 / njobs);
  k_prefix_x<<<dim3(px, gy), 256, 0, st>>>(dj, njobs);
}
void exclusive_scan(cudaStream_t st, const uint32_t* in, unsigned long long* out,
                    unsigned long long* sums, uint32_t n, unsigned long long* total) {
  if (!n) {
    cudaMemsetAsync(total, 0, sizeof(unsigned long long), st);
    return;
  }
  const uint32_t nb = (n + 1023) / 1024;
  k_scan_local<<<nb, 1024, 0, st>>>(in, out, sums, n, total);
  if (nb == 1) return;
  if (nb <= 1024) {  // a launch less (3 us); the blocks read nb * nb / 2 sums in all
    k_scan_base<<<nb, 1024, 0, st>>>(out, sums, n, total);
    return;
  }
  k_scan_sums<<<1, 1024, 0, st>>>(sums, nb, total);
  k_scan_add<<<(n + 255) / 256, 256, 0, st>>>(out, sums, n);
}

void shell_sat(cudaStream_t st, const JobDesc* dj, int njobs, uint32_t total_faces,
               const FaceScratch& fs, int num_sms, int grid_mult) {
  if (!total_faces) return;
  k_shell_count<<<grid_for(total_faces, 256, 65535), 256, 0, st>>>(dj, njobs, total_faces, fs.pcnt);
  exclusive_scan(st, fs.pcnt, fs.pbase, fs.psums, (total_faces + 31) / 32, fs.ptotal);
  constexpr int bytes = SHELL_WARPS * sizeof(ShellWarp);
  static bool attr[64] = {};  // per device
  const int dv = cur_dev();
  if (!attr[dv]) {
    cudaFuncSetAttribute(k_shell_flat, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    attr[dv] = true;
  }
  k_shell_flat<<<num_sms * grid_mult, SHELL_WARPS * 32, bytes, st>>>(dj, njobs, fs.pbase, fs.ptotal, total_faces);
}
void combine(cudaStream_t st, const JobDesc* dj, const uint32_t* brick_job,
             uint32_t total_bricks, uint8_t* live, int dual) {
  if (total_bricks)
    k_combine<<<grid_for(total_bricks, 1, 1 << 20), 256, 0, st>>>(dj, brick_job, total_bricks, live, dual);
}
void mark_live(cudaStream_t st, const JobDesc* dj, const uint32_t* brick_job,
               uint32_t total_bricks, uint8_t* live) {
  if (total_bricks)
    k_mark_live<<<grid_for(total_bricks, 1, 1 << 20), 256, 0, st>>>(dj, brick_job, total_bricks, live);
}
void compact_live(cudaStream_t st, const uint8_t* live, uint32_t first, uint32_t total_bricks, uint32_t* list,
                  uint32_t* count) {
  cudaMemsetAsync(count, 0, sizeof(uint32_t), st);
  if (total_bricks)
    k_compact<<<grid_for(total_bricks, 256, 4096), 256, 0, st>>>(live, first, total_bricks, list, count);
}

}  // namespace vfk
