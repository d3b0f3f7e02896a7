// vf_flood.cu -- FloodFracturer (FloodFracturer.cpp:98-191) on sm_103a.
//
// The reference runs a breadth-first flood, one compute dispatch and one
// host read-back per wave, and lets the last writer win a tie.  With the
// rule "a voxel claimed in wave t takes the claim of the lowest seed index
// among its wave-(t-1) neighbours", the label of every voxel is the label of
// the seed nearest to it in grid-graph distance through occupied voxels
// (6-neighbourhood for Manhattan, 26 for Euclidean and Chebyshev), ties to
// the lowest seed index.
//
// The GPU runs those waves bit-parallel.  32 voxels along z (in a large flat
// grid along its longest axis: wave_order) are one word of bit planes:
//
//   A, B         EMPTY, occupied and not claimed yet (U), or claimed in a wave of
//                either parity (E0, E1): vf_wave_state.h
//   L0 .. L(n-1) the claiming seed's slot, bit by bit
//
// and, apart from them, the smallest slot that reaches the word's two end
// voxels from the words below and above (in), kept by the claims there.
//
// A wave t dilates the bits claimed in wave t (E(t & 1)) over the
// neighbourhood, carries the smallest slot along with bit-sliced minima, and
// claims the unclaimed occupied bits it reaches into E((t + 1) & 1).  Every
// voxel is claimed once.  E(t & 1) also holds the bits of waves t-2, t-4,
// ..., but no unclaimed voxel is next to one of those (it would have been
// claimed by the following wave), so they change nothing; and a row's owner
// claims with one bit of one plane, which the same wave's readers mask out
// whether they see it or not, and its slot with it.  So there is no frontier to
// clear, and no order is needed between the rows' loads and stores of a wave.
//
// A lane takes one row (x, y, word) of 32 voxels with its 8 neighbour rows.
// Rows are numbered linearly with EMPTY rows around each axis (WaveJob), so
// a neighbour is an index difference and no bounds are tested.  Which rows a
// wave looks at is a candidate bit per row, set by the claims of the previous
// wave: a row is a candidate when a claimed bit reaches one of its unclaimed
// bits.  A wave scans the candidate words of its jobs (4 bytes per 32 rows, so
// there are no queues), lists the rows in shared memory and deals them to the
// lanes: the rows of a front are few and scattered, and a warp per run of
// neighbouring rows left 27 of 32 lanes idle.
//
// All waves of all jobs of a batch run in ONE cooperative launch, on gangs of
// CTAs that flood a set of jobs in step (vfk::WaveGang): wave t of all of them,
// then the gang's barrier.  A batch has two gangs of one CTA per SM, so that
// one gang's scan and barrier run under the other's visits; jobs of a batch of
// small ones, and a small job alone, have a gang each, of one CTA where they hold
// few voxels, which synchronises with __syncthreads and keeps the candidate words
// in shared memory.  The barrier of a larger gang is a counter in global memory
// whose spin is bounded (it sets an error word and the kernel returns instead of
// hanging).
//
// What bounds it: the latency of a wave's four steps (scan, row list, visits,
// barrier), each 1300 to 4000 cycles, while the front is small, and the L1's
// tag lookups of the 9 row loads while it is large (about 20 lines per warp
// load).  Flood launch of a batch of 128 uneven jobs: 3.96 ms, where relaxing
// bricks of keys in shared memory to local convergence, a queue of bricks per
// pass, took 10.56 ms (7 key updates per voxel claimed, bound by the chain
// along each row); 48 jobs 1.64 against 4.01 ms; one job of 476 x 476 x 512
// 0.79 against 2.15 ms, of 240 x 240 x 256 0.51 against 1.36 ms; of 60 x 57 x
// 64 0.27 against 0.26 ms.  Solids by Manhattan, whose fronts cross a row's 32 voxels
// in 32 waves, and large thin plates take longer than by bricks (full cubes of 128^3
// 0.78 against 0.63 ms, of 400^3 4.1 against 2.6).  A gang per job in proportion to its size instead of
// two gangs in step took 6.1 ms for the 128 jobs (the longest job's gang
// finished last), a word of 30 neighbouring rows per warp 15.3 ms.
//
// Sub-seed prefixes (extra seeds merged into fragments, Seeder.cpp:115-152)
// then go through the reference's competition and disjoint cleanup
// (floodFracturer-comp.glsl:49-62, disjointSet*-comp.glsl): within a
// connected component of one fragment the lowest prefix wins; per fragment
// only voxels with the fragment's minimum prefix survive; the rest is
// re-flooded from all survivors (ties to the lowest label value).  The voxels a
// seed claims are connected (each was claimed by a neighbour with its slot),
// so a component of a fragment is a set of slots: k_slot_unions joins the slots
// of one fragment that touch, k_slot_resolve gives each set its lowest prefix.
// One pass over the rows; relaxing prefixes voxel by voxel, a whole-grid launch
// and a host read per round, took 11.1 of 11.7 ms of the fracture of 200 x 197 x
// 208 voxels with 8 + 16 seeds.
#include <algorithm>
#include <vector>

#include "vf_kernels.h"
#include "vf_wave_state.h"

namespace {

typedef unsigned long long u64;
using vfk::WaveArrays;
using vfk::WaveCta;
using vfk::WaveEntry;
using vfk::WaveGang;
using vfk::WaveJob;

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr uint32_t MAX_LEVEL = 0xFFFFEu;  // largest geodesic distance a flood takes
constexpr int SCAN = 4;                   // times 32 candidate words a warp reads per round
constexpr uint32_t WORDS = 1024;          // words with candidates listed per round
constexpr uint32_t LIST = 2048;           // rows of each kind listed per round
constexpr uint32_t UNITS = 2048;          // units of 256 rows a CTA keeps a list of
// Floods of at most SMALL_ROWS rows (64^3 voxels: 12.9 k) have a gang each in a batch,
// and the candidate words of one CTA hold them.  One with at most LONE_VOXELS occupied
// voxels, counted with its row states, runs on the first CTA of its gang alone,
// without a global barrier: its waves are a pass or two of one CTA.  Flood of 64 x 64
// x 64 voxels, Manhattan, on one CTA and on 13: a wall of 40 k voxels 287 and 293 us,
// a vessel of 38 k in 60 x 57 x 64 268 and 291; a ball of 58 k in 48^3 225 and 184, of
// 137 k 410 and 229, a full cube 918 and 334 (328 us by relaxing bricks; the rows
// alone do not tell these apart).
constexpr uint32_t SMALL_ROWS = 16384;
constexpr uint32_t LONE_VOXELS = 48 << 10;
constexpr uint32_t PRUNE = 16;            // waves between dropping the finished jobs' units

struct WaveArgs {
  WaveArrays arr;
  const WaveJob* jobs;
  const WaveGang* gangs;
  const WaveCta* cta;        // [gridDim.x] its entries
  const WaveEntry* entries;  // gang, rank, gang size
  JobState* st;
  uint32_t* bar;             // [gangs][WAVE_BAR_WORDS] arrivals, last wave with candidates (zeroed)
  uint32_t* last;            // [wave jobs] a wave with claims, + 1 (zeroed)
  uint32_t* err;
  uint32_t* stats;           // [0] rows visited, [1] waves, [3] timeouts, [7] voxels claimed
  uint32_t* wave_sizes;      // rows visited in each of the first 256 waves (or null)
  uint32_t wait_spins;       // polls of a gang barrier before it gives up
  uint32_t smem_words;       // candidate words that fit the shared memory of a one-CTA gang
  uint32_t lone_voxels;      // small floods of at most so many voxels run on one CTA
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// words per row state with n slot planes: A, B and the planes, in units of 16
// bytes
__host__ __device__ constexpr int state_words(int n) { return (n + 2 + 3) / 4 * 4; }

// the row state at p (rows of 32 bytes in one access)
template <int NB>
__device__ __forceinline__ void load_row(const uint32_t* p, uint32_t (&w)[state_words(NB)]) {
  constexpr int SW = state_words(NB);
  if (SW % 8 == 0) {
#pragma unroll
    for (int i = 0; i + 7 < SW; i += 8)
      asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]), "=r"(w[i + 4]), "=r"(w[i + 5]),
                     "=r"(w[i + 6]), "=r"(w[i + 7])
                   : "l"(p + i)
                   : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < SW; i += 4) {
      const uint4 v = *reinterpret_cast<const uint4*>(p + i);
      w[i] = v.x; w[i + 1] = v.y; w[i + 2] = v.z; w[i + 3] = v.w;
    }
  }
}

// Per bit, the smallest slot among K sources (bit-sliced: F[i] says which
// bits source i has, P[i] its planes) by elimination from the top plane: where
// some source left has a 0, the sources with a 1 drop out.
template <int NB, int K>
__device__ __forceinline__ uint32_t min_slots(uint32_t (&F)[K], const uint32_t (&P)[K][NB], uint32_t (&L)[NB]) {
  uint32_t f = 0;
#pragma unroll
  for (int i = 0; i < K; ++i) f |= F[i];
#pragma unroll
  for (int b = NB - 1; b >= 0; --b) {
    uint32_t z3[3] = {0, 0, 0};  // three short chains
#pragma unroll
    for (int i = 0; i < K; ++i) z3[i % 3] |= F[i] & ~P[i][b];
    const uint32_t z = z3[0] | z3[1] | z3[2];
    L[b] = ~z;
#pragma unroll
    for (int i = 0; i < K; ++i) F[i] &= ~(z & P[i][b]);
  }
  return f;
}

template <int V>
struct Int {
  static constexpr int value = V;
};

// a job of the gang in shared memory: rows between x, between words (bit 31:
// 6-neighbourhood), the rows that are visited
struct JobRow {
  uint32_t sx, sy, lo, hi;
};

// key of a claim of level `level` by `slot` in WaveJob::in; a later level is smaller
__device__ __forceinline__ uint32_t in_key(uint32_t level, uint32_t slot) { return ((0xFFFFFu - level) << 12) | slot; }

// reductions without a result (the atomics of CUDA C++ return one on generic
// pointers, used or not)
template <bool SMEM>
__device__ __forceinline__ void red_or(uint32_t* p, uint32_t v) {
  if (SMEM)
    asm volatile("red.relaxed.cta.shared::cta.or.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v)
                 : "memory");
  else
    asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_min(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.min.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// candidate bits of the rows i - 1, i, i + 1 (bits 0 .. 2 of m)
template <bool SMEM>
__device__ __forceinline__ void set_candidates(uint32_t* cand, uint32_t i, uint32_t m) {
  const uint32_t k = i - 1, sh = k & 31u;
  uint32_t* c = cand + (k >> 5);
  if (m) red_or<SMEM>(c, m << sh);
  const uint32_t hi = (m >> 1) >> (31u - sh);
  if (hi) red_or<SMEM>(c + 1, hi);
}

// One row in wave t: claims and the next wave's candidates.  Returns whether
// a candidate was set (bit 0) and whether a voxel was claimed (bit 1).
template <int NB, int CONN, bool SMEM>
__device__ __forceinline__ uint32_t visit_row(const WaveArrays& arr, const JobRow& J, uint32_t i, uint32_t t,
                                              uint32_t* next, uint32_t* err, uint32_t& claims) {
  constexpr int SW = state_words(NB);
  const uint32_t sy = J.sy & 0x7FFFFFFFu, sx = J.sx;
  // a claim at a word end names rows beyond it unseen: of the EMPTY ones around the
  // grid, some have neighbours of their own that would lie outside the job
  if (i < J.lo || i >= J.hi) return 0;
  uint32_t* const p0 = arr.state + (size_t)i * SW;
  const size_t xs = (size_t)sx * SW;
  uint32_t A4, B4, O[NB], U[9], F[9], P[9][NB];
  // the 3 x 3 rows around the row (6: the cross)
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int dx = r / 3 - 1, dy = r % 3 - 1;
    if (CONN == 6 && dx && dy) {
      U[r] = F[r] = 0;
      continue;
    }
    uint32_t w[SW];
    load_row<NB>((dx < 0 ? p0 - xs : (dx > 0 ? p0 + xs : p0)) + dy * SW, w);
    U[r] = wave_unclaimed(w[0], w[1]);
    F[r] = wave_front(w[0], w[1], t);
#pragma unroll
    for (int b = 0; b < NB; ++b) P[r][b] = w[2 + b];
    if (r == 4) {
      A4 = w[0];
      B4 = w[1];
#pragma unroll
      for (int b = 0; b < NB; ++b) O[b] = w[2 + b];
    }
  }
  // slots that claims of this wave's level bring in from the words below / above
  const uint2 in = arr.in[2 * (size_t)i + (t & 1u)];
  const uint32_t base = in_key(t, 0), dlo = in.x - base, dhi = in.y - base;
  const uint32_t lo_f = dlo < 4095u ? 1u : 0u, hi_f = dhi < 4095u ? 1u << 31 : 0u;  // slots are below 4095
  uint32_t L[NB], f;
  if (CONN == 26) {
    uint32_t W[NB];  // over the 3 x 3 rows, then z - 1, z, z + 1
    const uint32_t g = min_slots<NB, 9>(F, P, W);
    uint32_t G[3] = {g, (g << 1) | lo_f, (g >> 1) | hi_f}, Q[3][NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      Q[0][b] = W[b];
      Q[1][b] = __funnelshift_l(dlo << (31 - b), W[b], 1);
      Q[2][b] = __funnelshift_r(W[b], dhi >> b, 1);
    }
    f = min_slots<NB, 3>(G, Q, L);
  } else {
    const uint32_t g = F[4];
    uint32_t G[6] = {F[1], F[3], F[5], F[7], (g << 1) | lo_f, (g >> 1) | hi_f}, Q[6][NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      Q[0][b] = P[1][b];
      Q[1][b] = P[3][b];
      Q[2][b] = P[5][b];
      Q[3][b] = P[7][b];
      Q[4][b] = __funnelshift_l(dlo << (31 - b), P[4][b], 1);
      Q[5][b] = __funnelshift_r(P[4][b], dhi >> b, 1);
    }
    f = min_slots<NB, 6>(G, Q, L);
  }
  const uint32_t N = f & U[4];
  if (!N) return 0;
  if (t >= MAX_LEVEL) {  // the claims would lie beyond the largest distance
    atomicOr(err, VF_JERR_DIST_OVERFLOW);
    return 0;
  }
  claims += (uint32_t)__popc(N);
  U[4] &= ~N;
  {
    uint32_t w[SW];
    w[0] = A4;
    w[1] = B4;
    wave_claim(w[0], w[1], N, t);
#pragma unroll
    for (int b = 0; b < SW - 2; ++b) w[2 + b] = b < NB ? (O[b < NB ? b : 0] & ~N) | (L[b < NB ? b : 0] & N) : 0u;
#pragma unroll
    for (int k = 0; k < SW; k += 4)
      *reinterpret_cast<uint4*>(p0 + k) = make_uint4(w[k], w[k + 1], w[k + 2], w[k + 3]);
  }
  // rows the claims reach: exactly in this word (their unclaimed bits as read:
  // a row claimed meanwhile is looked at in vain), row by row in the words
  // below and above
  const uint32_t nz = N | (N << 1) | (N >> 1);
  uint32_t any = 0;
#pragma unroll
  for (int dx = -1; dx <= 1; ++dx) {
    uint32_t m = 0;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      const int r = (dx + 1) * 3 + dy + 1;
      const uint32_t reach = CONN == 26 ? nz : (r == 4 ? (N << 1) | (N >> 1) : N);
      m |= (reach & U[r]) ? 1u << (dy + 1) : 0u;
    }
    set_candidates<SMEM>(next, i + (uint32_t)dx * sx, m);
    any |= m;
  }
  if ((N & 0x80000001u) != 0) {
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      if (k == 0 ? !(N & 1u) : !(N >> 31)) continue;
      uint32_t slot = 0;
#pragma unroll
      for (int b = 0; b < NB; ++b) slot |= (k ? L[b] >> 31 : L[b] & 1u) << b;
      const uint32_t key = in_key(t + 1u, slot);
      // row i is below (k = 1) or above the rows j it reaches: their .x / .y
      const uint32_t j = k ? i + sy : i - sy;
      uint32_t* const to = reinterpret_cast<uint32_t*>(arr.in + 2 * (size_t)j + ((t + 1) & 1u)) + (1 - k);
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        if (CONN == 6 && dx) continue;
        uint32_t* const q = to + 4 * (dx < 0 ? -(ptrdiff_t)sx : (dx > 0 ? (ptrdiff_t)sx : 0));
        red_min(q, key);
        if (CONN == 26) {
          red_min(q - 4, key);
          red_min(q + 4, key);
        }
        set_candidates<SMEM>(next, j + (uint32_t)dx * sx, CONN == 26 ? 7u : 2u);
      }
    }
    any = 1;
  }
  return any ? 3u : 2u;
}

// the dynamic shared memory of k_wave; the candidate words of a one-CTA gang follow
struct WaveShared {
  JobRow job[vfk::WAVE_GANG_JOBS];
  uint32_t last[vfk::WAVE_GANG_JOBS];  // this CTA's last wave with claims, + 1
  uint8_t live[vfk::WAVE_GANG_JOBS];
  uint32_t bits[WORDS], word[WORDS];   // the round's words with candidates
  uint8_t wjob[WORDS];                 // their jobs
  uint32_t row[2][LIST];               // the round's rows: 26- / 6-neighbourhood
  uint8_t rjob[2][LIST];               // their jobs
  uint32_t unit[UNITS];                // this CTA's units | job << 24
};

template <int NB, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1) k_wave(WaveArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WaveShared& S = *reinterpret_cast<WaveShared*>(smem_raw);
  uint32_t* const s_cand = reinterpret_cast<uint32_t*>(smem_raw + sizeof(WaveShared));
  __shared__ WaveGang G;
  __shared__ uint32_t s_n[2][2], s_w[2], s_any[2], s_again[2], s_go, s_ok, s_units, s_rank, s_size;
  __shared__ uint32_t s_stat[2];
  constexpr uint32_t warps = THREADS / 32;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const WaveCta mine = a.cta[blockIdx.x];
  if (tid < 2) s_stat[tid] = 0;
  uint32_t claims = 0;  // this thread's
  for (uint32_t e = 0; e < mine.count; ++e) {
    __syncthreads();
    if (tid == 0) {
      const WaveEntry en = a.entries[mine.first + e];
      G = a.gangs[en.gang];
      s_rank = en.rank;
      s_size = en.size;
      if (en.size > 1 && G.count == 1 && G.units * 256 <= SMALL_ROWS &&
          a.st[a.jobs[G.first].job].wave_voxels <= a.lone_voxels)
        s_size = 1;  // the first CTA's alone
      s_n[0][0] = s_n[0][1] = s_n[1][0] = s_n[1][1] = s_w[0] = s_w[1] = s_any[0] = s_any[1] = s_again[0] = s_again[1] = 0;
    }
    __syncthreads();
    if (s_rank >= s_size) continue;
    const uint32_t rank = s_rank, size = s_size, first = G.first, njobs = G.count;
    const uint32_t word_lo = G.unit_lo * 8, words = G.units * 8;
    for (uint32_t j = tid; j < njobs; j += THREADS) {
      const WaveJob& W = a.jobs[first + j];
      S.job[j] = {W.sx, W.sy | (W.conn6 << 31), W.row0, W.base + W.nrows - (W.sx + W.sy + 1)};
      S.last[j] = 0;
    }
    const bool in_smem = size == 1 && 2 * words <= a.smem_words;
    if (in_smem)
      for (uint32_t i = tid; i < words; i += THREADS) {
        s_cand[i] = a.arr.cand[word_lo + i];
        s_cand[words + i] = 0;
      }
    __syncthreads();
    // Candidate words in units of 8 (256 rows, one job); the gang's units are
    // dealt to its CTAs in turn, so that the rows of a front spread evenly.
    // The job of a unit: the last whose rows start at or before it.
    auto unit_of = [&](uint32_t k) {
      const uint32_t u = G.unit_lo + k * size + rank;
      uint32_t lo = 0, hi = njobs - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (a.jobs[first + mid].base <= u * 256u) lo = mid; else hi = mid - 1;
      }
      return u | (lo << 24);
    };
    uint32_t nunits = G.units > rank ? (G.units - rank + size - 1) / size : 0;
    const bool listed = nunits <= UNITS;
    if (listed)
      for (uint32_t k = tid; k < nunits; k += THREADS) S.unit[k] = unit_of(k);
    if (tid == 0) s_units = nunits;
    __syncthreads();
    uint32_t* const bar = a.bar + (size_t)(size > 1 ? a.entries[mine.first + e].gang : 0) * vfk::WAVE_BAR_WORDS;
    uint32_t rr = 0;  // rounds done: parity of the list counters
    uint32_t t = 0;
    for (;; ++t) {
      uint32_t* const gcur = a.arr.cand + (t & 1u) * (size_t)a.arr.nwords;
      uint32_t* const gnext = a.arr.cand + ((t + 1) & 1u) * (size_t)a.arr.nwords;
      uint32_t* const scur = s_cand + (t & 1u) * words - word_lo;
      uint32_t* const snext = s_cand + ((t + 1) & 1u) * words - word_lo;
      bool any = false, stop = false;
      uint32_t active = t;  // the last wave with candidates (thread 0; a gang's word of it)
      if (tid == 0 && size > 1 && t) active = ld_relaxed(bar + 16);
      nunits = s_units;
      const uint32_t rounds = (nunits + 4 * warps * SCAN - 1) / (4 * warps * SCAN);
      for (bool again = true, once = true; again; ++rr, once = false) {
        // 1. the words with candidates: SCAN loads of the next round in flight
        // while a round's words are listed
        uint32_t b[SCAN], g[SCAN];
        auto read = [&](uint32_t r) {
#pragma unroll
          for (int k = 0; k < SCAN; ++k) {
            const uint32_t q = 4 * ((r * SCAN + k) * warps + warp) + lane / 8;
            b[k] = g[k] = 0;
            if (q < nunits) {
              g[k] = listed ? S.unit[q] : unit_of(q);  // unit | job << 24
              const uint32_t w = (g[k] & 0xFFFFFFu) * 8 + lane % 8;
              b[k] = in_smem ? scur[w] : gcur[w];
            }
          }
        };
        read(0);
#pragma unroll 1
        for (uint32_t r = 0; r < rounds; ++r) {
          uint32_t c[SCAN], h[SCAN], full = 0;
          unsigned m[SCAN];
#pragma unroll
          for (int k = 0; k < SCAN; ++k) {
            c[k] = b[k];
            h[k] = g[k];
          }
          if (r + 1 < rounds) read(r + 1);
#pragma unroll
          for (int k = 0; k < SCAN; ++k) {
            m[k] = __ballot_sync(FULL, c[k] != 0);
            full += (uint32_t)__popc(m[k]);
          }
          if (!full) continue;
          uint32_t pos = 0;
          if (lane == 0) pos = atomicAdd(&s_w[rr & 1u], full);
          pos = __shfl_sync(FULL, pos, 0);
          if (pos + full > WORDS) {  // no room: these words stay for another round
            for (uint32_t i = pos + lane; i < min(WORDS, pos + full); i += 32) S.bits[i] = 0;
            if (lane == 0) s_again[rr & 1u] = 1u;
            continue;
          }
#pragma unroll
          for (int k = 0; k < SCAN; ++k) {
            if (c[k]) {
              const uint32_t i = pos + __popc(m[k] & ((1u << lane) - 1u)), w = (h[k] & 0xFFFFFFu) * 8 + lane % 8;
              S.bits[i] = c[k];
              S.word[i] = w;
              S.wjob[i] = (uint8_t)(h[k] >> 24);
              if (in_smem) scur[w] = 0; else gcur[w] = 0;  // wave t + 2 starts with empty words
            }
            pos += (uint32_t)__popc(m[k]);
          }
        }
        if (tid == 0 && once) s_go = (int32_t)(active - t) >= 0 ? 1u : 0u;
        __syncthreads();
        if (once && !s_go) {
          stop = true;
          break;
        }
        // 2. their rows, a lane per half word
        const uint32_t nwords = min(s_w[rr & 1u], WORDS);
        for (uint32_t k0 = warp * 16; k0 < nwords; k0 += warps * 16) {
          const uint32_t k = k0 + lane / 2;
          uint32_t bits = 0, w = 0, jid = 0;
          if (k < nwords) {
            bits = S.bits[k];
            w = S.word[k];
            jid = S.wjob[k];
          }
          bits &= lane & 1 ? 0xFFFF0000u : 0xFFFFu;
          if (!__any_sync(FULL, bits != 0)) continue;
          // both kinds in one scan: rows of the 6-neighbourhood in the high half
          const uint32_t six = S.job[jid].sy >> 31, n = (uint32_t)__popc(bits) << (16 * six);
          uint32_t incl = n;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) incl += v;
          }
          const uint32_t total = __shfl_sync(FULL, incl, 31);
          uint32_t pos = 0;
          if (lane < 2) pos = atomicAdd(&s_n[rr & 1u][lane], (total >> (16 * lane)) & 0xFFFFu);
          const uint32_t pos0 = __shfl_sync(FULL, pos, 0), pos1 = __shfl_sync(FULL, pos, 1);
          const uint32_t end = six ? pos1 + (total >> 16) : pos0 + (total & 0xFFFFu);
          pos = (six ? pos1 : pos0) + (((incl - n) >> (16 * six)) & 0xFFFFu);
          if (end > LIST) {  // no room: back into the word
            if (bits) {
              if (in_smem) atomicOr(scur + w, bits); else atomicOr(gcur + w, bits);
              s_again[rr & 1u] = 1u;
            }
            const uint32_t stop = min(LIST, pos + (uint32_t)__popc(bits));
            for (; pos < stop; ++pos) S.row[six][pos] = 0xFFFFFFFFu;
            bits = 0;
          }
          while (bits) {
            const uint32_t bit = (uint32_t)__ffs(bits) - 1;
            bits &= bits - 1;
            S.row[six][pos] = (w << 5) | bit;
            S.rjob[six][pos++] = (uint8_t)jid;
          }
        }
        __syncthreads();
        const uint32_t n26 = min(s_n[rr & 1u][0], LIST), n6 = min(s_n[rr & 1u][1], LIST);
        again = s_again[rr & 1u] != 0;
        if (tid == 0) {
          s_n[(rr + 1) & 1u][0] = s_n[(rr + 1) & 1u][1] = 0;
          s_w[(rr + 1) & 1u] = s_again[(rr + 1) & 1u] = 0;
          if (once) s_any[(t + 1) & 1u] = 0;
          s_stat[0] += n26 + n6;
          if (a.wave_sizes && n26 + n6 && t < 256) atomicAdd(a.wave_sizes + t, n26 + n6);
        }
        auto visit = [&](auto conn, uint32_t i) {
          constexpr int CONN = decltype(conn)::value;
          const uint32_t row = S.row[CONN == 6][i], j = S.rjob[CONN == 6][i];
          if (row == 0xFFFFFFFFu) return;
          const JobRow J = S.job[j];
          uint32_t* const err = &a.st[a.jobs[first + j].job].err;
          const uint32_t f = in_smem ? visit_row<NB, CONN, true>(a.arr, J, row, t, snext, err, claims)
                                     : visit_row<NB, CONN, false>(a.arr, J, row, t, gnext, err, claims);
          any |= (f & 1u) != 0;
          if (f) S.last[j] = t + 1;
        };
        for (uint32_t i = tid; i < n26; i += THREADS) visit(Int<26>{}, i);
        // the 6-neighbourhood rows start at the warp after the others' last one
        const uint32_t off = ((n26 + 31) / 32 % warps) * 32;
        for (uint32_t i = (tid + THREADS - off) % THREADS; i < n6; i += THREADS) visit(Int<6>{}, i);
        if (any) s_any[t & 1u] = 1u;
        __syncthreads();
      }
      if (stop) break;
      if (size == 1) {
        if (!s_any[t & 1u]) {
          ++t;
          break;
        }
        continue;
      }
      const bool prune = listed && njobs > 1 && t % PRUNE == PRUNE - 1;
      if (prune) {
        for (uint32_t j = tid; j < njobs; j += THREADS)
          if (S.last[j] == t + 1) atomicMax(a.last + first + j, t + 1);
        __syncthreads();
      }
      // Gang barrier: one arrival counter that only grows, which every CTA
      // polls.  Whether a wave follows is in a word of its own, the last wave
      // with candidates; it is read while the next wave scans.
      if (tid == 0) {
        if (s_any[t & 1u]) atomicMax(bar + 16, t + 1u);
        red_release(bar, 1u);
        const uint32_t target = (t + 1u) * size;
        uint32_t spins = 0, ok = 1;
        while ((int32_t)(ld_acquire(bar) - target) < 0) {
          if (++spins > a.wait_spins || ((spins & 63u) == 0 && ld_acquire(a.err) != 0)) {
            atomicOr(a.err, 2u);
            atomicAdd(a.stats + 3, 1u);
            ok = 0;
            break;
          }
        }
        s_ok = ok;
      }
      __syncthreads();
      if (!s_ok) return;  // timed out: the error word is set
      if (prune) {
        // a job without claims in this wave has no candidates any more: its
        // units leave the list (warp 0, in place)
        for (uint32_t j = tid; j < njobs; j += THREADS) S.live[j] = ld_relaxed(a.last + first + j) == t + 1;
        __syncthreads();
        if (warp == 0) {
          uint32_t out = 0;
          for (uint32_t k0 = 0; k0 < nunits; k0 += 32) {
            const uint32_t k = k0 + lane, u = k < nunits ? S.unit[k] : 0u;
            const bool live = k < nunits && S.live[u >> 24];
            const unsigned m = __ballot_sync(FULL, live);
            if (live) S.unit[out + __popc(m & ((1u << lane) - 1u))] = u;
            __syncwarp();
            out += __popc(m);
          }
          if (lane == 0) s_units = out;
        }
        __syncthreads();
      }
    }
    for (uint32_t j = tid; j < njobs; j += THREADS)
      if (S.last[j]) atomicMax(&a.st[a.jobs[first + j].job].passes, S.last[j]);
    if (tid == 0 && rank == 0) atomicMax(a.stats + 1, t);
  }
  claims = __reduce_add_sync(FULL, claims);
  if (lane == 0 && claims) atomicAdd(&s_stat[1], claims);
  __syncthreads();
  if (tid == 0) {
    if (s_stat[0]) atomicAdd(a.stats + 0, s_stat[0]);
    if (s_stat[1]) atomicAdd(a.stats + 7, s_stat[1]);
  }
}

// ---------------------------------------------------------------------------
__device__ __forceinline__ void add_voxels(uint32_t* to, uint32_t n) {
  n = __reduce_add_sync(FULL, n);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(to, n);
}

// Row states from the label grid: occupied voxels unclaimed, all else EMPTY,
// the rows around the grid included (bricks without occupied voxels are not
// read).  A CTA takes 256 consecutive rows of one job, eight lanes per row, 4
// voxels per lane (a warp instruction reads 4 whole 64-byte rows); the lanes
// then write the row's state together.
//
// Small floods have their occupied voxels counted (LONE_VOXELS).
__global__ void __launch_bounds__(256) k_wave_init(const JobDesc* jobs, JobState* st, WaveArrays arr, const WaveJob* wj,
                                                   uint32_t njobs, const uint8_t* live) {
  uint32_t lo = 0, hi = njobs - 1;  // the job of these rows: the last that starts at or before them
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (wj[mid].base <= blockIdx.x * 256u) lo = mid; else hi = mid - 1;
  }
  const WaveJob& W = wj[lo];
  if (W.order != vfk::WAVE_XYZ) return;  // k_flat_init's
  const JobDesc& J = jobs[W.job];
  const uint32_t q = threadIdx.x & 7, r0 = threadIdx.x >> 3;
  const uint32_t first = blockIdx.x * 256u;
  uint2 a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    a[i] = make_uint2(0, 0);
    const uint32_t row = first + r0 + 32u * i;
    if (row < W.row0) continue;
    const uint32_t r = row - W.row0, x = r / W.sx, yz = r - x * W.sx, zw = yz / W.sy, y = yz - zw * W.sy;
    if (x >= J.X || y >= J.Y || zw >= J.nbz) continue;
    const uint32_t z = zw * VF_BZ + 4 * q;
    // Zp >= Zk: the lane's 4 labels are inside the row
    if (z < J.Zk && live[J.brick_base + ((x / VF_BX) * J.nby + y / VF_BY) * J.nbz + zw])
      a[i] = *reinterpret_cast<const uint2*>(J.grid + vf_gidx(J, x, y, z));
  }
  uint32_t voxels = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t row = first + r0 + 32u * i;
    uint32_t w = ((a[i].x & 0xFFFFu) ? 1u : 0u) | ((a[i].x >> 16) ? 2u : 0u) | ((a[i].y & 0xFFFFu) ? 4u : 0u) |
                 ((a[i].y >> 16) ? 8u : 0u);
    w <<= 4 * q;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) w |= __shfl_xor_sync(FULL, w, o);
    if (q == 0) voxels += (uint32_t)__popc(w);
    uint32_t* d = arr.state + (size_t)row * J.wsw;  // up to the next job's base

    for (uint32_t k = q; k < J.wsw; k += 8) d[k] = k == 0 ? wave_empty_a(w) : (k == 1 ? wave_empty_b(w) : 0u);
    if (q < 4) reinterpret_cast<uint32_t*>(arr.in + 2 * (size_t)row)[q] = 0xFFFFFFFFu;
  }
  if (W.nrows <= SMALL_ROWS) add_voxels(&st[W.job].wave_voxels, voxels);
}

// The same from the voxelizer's bit planes, which hold the rows' words already: a
// thread per row writes its state.  Bound by the stores: 128 mixed jobs 377 us, from
// the labels 1018 us.
__global__ void __launch_bounds__(256) k_wave_planes(const JobDesc* jobs, JobState* st, WaveArrays arr, const WaveJob* wj,
                                                     uint32_t njobs, uint32_t units) {
  for (uint32_t unit = blockIdx.x; unit < units; unit += gridDim.x) {
    uint32_t lo = 0, hi = njobs - 1;  // the job of these rows: the last that starts at or before them
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (wj[mid].base <= unit * 256u) lo = mid; else hi = mid - 1;
    }
    const WaveJob& W = wj[lo];
    if (W.order != vfk::WAVE_XYZ) continue;  // k_flat_init's
    const JobDesc& J = jobs[W.job];
    const uint32_t row = unit * 256u + threadIdx.x;
    uint32_t w = 0;
    if (row >= W.row0) {
      const uint32_t r = row - W.row0, x = r / W.sx, yz = r - x * W.sx, zw = yz / W.sy, y = yz - zw * W.sy;
      if (x < J.X && y < J.Y && zw < J.Zw) {
        const size_t at = ((size_t)x * J.Y + y) * J.Zw + zw;
        w = J.par[at] | J.shell[at];
      }
    }
    if (W.nrows <= SMALL_ROWS) add_voxels(&st[W.job].wave_voxels, (uint32_t)__popc(w));
    uint4* const d = reinterpret_cast<uint4*>(arr.state + (size_t)row * J.wsw);  // up to the next job's base
    d[0] = make_uint4(wave_empty_a(w), wave_empty_b(w), 0u, 0u);
    for (uint32_t k = 1; k < J.wsw / 4; ++k) d[k] = make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4*>(arr.in)[row] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
  }
}

// seed bricks must be live (a caller may seed an EMPTY voxel); seeds are
// checked, the fragments' prefix minima reset.  One CTA per job.
__global__ void __launch_bounds__(128) k_seed_bricks(const JobDesc* jobs, JobState* st, uint8_t* live,
                                                     uint32_t* list, uint32_t* count) {
  __shared__ int dead;
  const JobDesc& J = jobs[blockIdx.x];
  if (!J.active) return;
  JobState& s = st[blockIdx.x];
  for (int f = threadIdx.x; f < 256; f += blockDim.x) s.minprefix[f] = 0xFFFFFFFFu;
  if (threadIdx.x == 0) {
    s.passes = 0;
    s.disjoint = 0;
    dead = 0;
  }
  __syncthreads();
  const uint32_t ns = s.nseeds;
  auto brick = [&](uint32_t i) {
    return J.brick_base + ((J.seeds[4 * i] / VF_BX) * J.nby + J.seeds[4 * i + 1] / VF_BY) * J.nbz +
           J.seeds[4 * i + 2] / VF_BZ;
  };
  auto valid = [&](uint32_t i) {
    // label = frag | prefix << 8 (Seeder.cpp:150), fragment id >= 2
    const uint32_t w = J.seeds[4 * i + 3];
    return J.seeds[4 * i] < J.X && J.seeds[4 * i + 1] < J.Y && J.seeds[4 * i + 2] < J.Z && w <= 0x7FFFu &&
           (w & 0xFFu) > VOXEL_FREE;
  };
  for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x) {
    if (!valid(i)) atomicOr(&s.err, VF_JERR_INVALID);
    else if (!live[brick(i)]) dead = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0 && dead)
    for (uint32_t i = 0; i < ns; ++i) {
      if (!valid(i)) continue;
      const uint32_t b = brick(i);
      if (!live[b]) {
        live[b] = 1;
        list[atomicAdd(count, 1u)] = b;
      }
    }
}

// Seeds into the row states (later seeds win a shared voxel, as grid.set in
// list order does, FloodFracturer.cpp:101-103), the rows around them into
// wave 0's candidate masks.  One CTA per job; works on any axis order (the
// seed's axis a is coordinate ax[a] of the state).
// uf[i] (or null): i when the seed holds its voxel, else NO_SLOT.
constexpr uint32_t NO_SLOT = 0xFFFFFFFFu;
__device__ void seed_waves(const WaveArrays& arr, const WaveJob& W, uint32_t* uf, const uint32_t* seeds, uint32_t ns, uint32_t sw, int nb,
                           uint32_t order, u64* pos) {
  const int t = threadIdx.x;
  auto coord = [&](uint32_t i, int a) { return seeds[4 * i + ((order >> (4 * a)) & 15u)]; };
  for (uint32_t i = t; i < ns; i += blockDim.x)
    pos[i] = ((u64)coord(i, 0) << 40) | ((u64)coord(i, 1) << 20) | coord(i, 2);
  __syncthreads();
  for (uint32_t i = t; i < ns; i += blockDim.x) {
    bool won = true;
    for (uint32_t k = i + 1; k < ns && won; ++k) won = pos[k] != pos[i];
    if (!won) continue;
    if (uf) uf[i] = i;
    const uint32_t x = (uint32_t)(pos[i] >> 40), y = (uint32_t)(pos[i] >> 20) & 0xFFFFFu,
                   z = (uint32_t)pos[i] & 0xFFFFFu;
    const uint32_t zw = z >> 5, bit = 1u << (z & 31u);
    const uint32_t row = W.row0 + x * W.sx + zw * W.sy + y;
    uint32_t* d = arr.state + (size_t)row * sw;
    atomicAnd(d, ~bit);  // E0
    atomicAnd(d + 1, ~bit);
    for (int b = 0; b < nb; ++b)
      if ((i >> b) & 1u) atomicOr(d + 2 + b, bit);
    const bool lo = (z & 31u) == 0, hi = (z & 31u) == 31;
    for (int dx = -1; dx <= 1; ++dx) {
      const uint32_t r = row + (uint32_t)dx * W.sx;
      set_candidates<false>(arr.cand, r, 7u);
      if (lo) set_candidates<false>(arr.cand, r - W.sy, 7u);
      if (hi) set_candidates<false>(arr.cand, r + W.sy, 7u);
      for (int dy = -1; dy <= 1; ++dy) {
        if (W.conn6 && (dx || dy)) continue;  // level 0 reaches wave 0
        if (lo) atomicMin(&arr.in[2 * (size_t)(r - W.sy + dy)].y, in_key(0, i));
        if (hi) atomicMin(&arr.in[2 * (size_t)(r + W.sy + dy)].x, in_key(0, i));
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_wave_seed(const JobDesc* jobs, const JobState* st, WaveArrays arr,
                                                   const WaveJob* wj) {
  __shared__ u64 pos[4096];
  const WaveJob& W = wj[blockIdx.x];
  const JobDesc& J = jobs[W.job];
  const JobState& s = st[W.job];
  if (!J.active) return;
  if (J.uf) {
    for (uint32_t i = threadIdx.x; i < s.nseeds; i += blockDim.x) J.uf[i] = NO_SLOT;
    __syncthreads();
  }
  if (s.err) return;
  seed_waves(arr, W, J.uf, J.seeds, min(s.nseeds, 4096u), J.wsw, (int)J.wsw - 2, W.order, pos);
}

// ---- a flood on a grid of any strides, any axis order ----------------------
// (vf_flood_noalloc on a caller's device grid; flat grids of the batched path).
// Voxel (a, b, c) of the state, c along the words, is the grid's element
// a * s[0] + b * s[1] + c * s[2].
// One warp per row, a lane per voxel; consecutive warps take consecutive words
// of a grid row, whose voxels are contiguous.
__device__ __forceinline__ bool flat_row(const WaveJob& W, const vfk::FlatAxes& A, uint32_t k, uint32_t lane,
                                         uint32_t& row, size_t& at) {
  // k numbers the rows of the padded box [nx + 2][ny + 1][nw + 1], words fastest
  const uint32_t nw1 = W.sx / W.sy, zw = k % nw1, y = (k / nw1) % W.sy, x = k / W.sx;
  row = W.row0 - W.sx + x * W.sx + zw * W.sy + y;
  const uint32_t z = 32 * zw + lane;
  at = (x - 1) * A.s[0] + y * A.s[1] + z * A.s[2];
  return x >= 1 && x <= A.nx && y < A.ny && z < A.nz;
}

__global__ void __launch_bounds__(256) k_flat_init(const uint16_t* grid, WaveArrays arr, WaveJob W,
                                                   vfk::FlatAxes A, uint32_t sw, JobState* st) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t box = (A.nx + 2) * W.sx, nwarps = (gridDim.x * blockDim.x) >> 5;
  auto put = [&](uint32_t row, uint32_t m) {
    if (lane < sw)
      arr.state[(size_t)row * sw + lane] = lane == 0 ? wave_empty_a(m) : (lane == 1 ? wave_empty_b(m) : 0u);
    if (lane < 4) reinterpret_cast<uint32_t*>(arr.in + 2 * (size_t)row)[lane] = 0xFFFFFFFFu;
  };
  for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < box; k += nwarps) {
    uint32_t row;
    size_t at;
    const bool in = flat_row(W, A, k, lane, row, at);
    const uint32_t m = __ballot_sync(FULL, in && grid[at] != VOXEL_EMPTY);
    put(row, m);
    if (W.nrows <= SMALL_ROWS && lane == 0 && m) atomicAdd(&st->wave_voxels, (uint32_t)__popc(m));
  }
  // the rows before and after the box
  const uint32_t before = W.row0 - W.sx - W.base, after = W.nrows - before - box;
  for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < before + after; k += nwarps)
    put(W.base + (k < before ? k : box + k), 0u);
}

// wave job and gang table, then the seeds (labels 2..255 without prefix)
__global__ void __launch_bounds__(256) k_flat_seed(WaveArrays arr, WaveJob W, vfk::FlatAxes A, uint32_t sw,
                                                   const uint32_t* seeds, uint32_t ns, uint32_t size,
                                                   uint32_t blocks, JobState* st, WaveJob* jobs, WaveGang* gang,
                                                   WaveCta* cta, WaveEntry* entries) {
  __shared__ u64 pos[4096];
  __shared__ uint32_t bad, prefix;
  if (threadIdx.x == 0) {
    *jobs = W;
    *gang = {0, 1, 0, (W.nrows + 255) / 256};
    bad = prefix = 0;
  }
  for (uint32_t c = threadIdx.x; c < blocks; c += blockDim.x) {
    cta[c] = {c, c < size ? 1u : 0u};
    entries[c] = {0, c, size, 0};
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x) {
    const uint32_t w = seeds[4 * i + 3];
    if (seeds[4 * i] >= A.dims[0] || seeds[4 * i + 1] >= A.dims[1] || seeds[4 * i + 2] >= A.dims[2] ||
        w > 0x7FFFu || (w & 0xFFu) <= VOXEL_FREE)
      bad = 1;
    if (w > 0xFFu) prefix = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    st->nseeds = ns;
    st->err = bad ? VF_JERR_INVALID : 0u;
    st->has_prefix = prefix;
  }
  if (!bad && !prefix) seed_waves(arr, W, nullptr, seeds, ns, sw, (int)sw - 2, A.order, pos);
}

// st: the job of a batch (null: no sub-seed prefixes)
__global__ void __launch_bounds__(256) k_flat_labels(WaveArrays arr, WaveJob W, vfk::FlatAxes A, uint32_t sw,
                                                     const uint32_t* seeds, const JobState* st, uint16_t* labels) {
  const uint32_t lane = threadIdx.x & 31;
  const bool second = st && st->has_prefix && st->disjoint;  // slots are ranks
  const uint32_t box = (A.nx + 2) * W.sx, nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < box; k += nwarps) {
    uint32_t row;
    size_t at;
    const bool in = flat_row(W, A, k, lane, row, at);
    if (!__any_sync(FULL, in)) continue;
    const uint32_t word = lane < sw ? arr.state[(size_t)row * sw + lane] : 0u;
    const uint32_t a = __shfl_sync(FULL, word, 0), b = __shfl_sync(FULL, word, 1);
    const uint32_t v = wave_claimed(a, b), u = wave_unclaimed(a, b);
    uint32_t l = (u >> lane) & 1u;
    if (v) {  // uniform
      uint32_t slot = 0;
      for (uint32_t k = 0; k + 2 < sw; ++k) slot |= ((__shfl_sync(FULL, word, 2 + k) >> lane) & 1u) << k;
      if ((v >> lane) & 1u) l = (second ? st->rank_value[slot] : seeds[4 * slot + 3]) & 0xFFu;
    }
    if (in) labels[at] = (uint16_t)l;
  }
}

// row states -> labels (undoMask fused: & 0xFF).
// Live bricks, dealt to resident CTAs; four lanes per row, each 8 voxels (16 bytes
// of labels).  EMPTY 0, unclaimed FREE, claimed: the slot's label.  Bound by the
// chain brick -> job -> rows -> labels, so a CTA keeps its job's label table from
// brick to brick and reads the next brick's number beside this one's rows (a CTA per
// brick, each with its own table: 42 us in a 476x476x512 job, 535 us in 128 mixed
// ones; four CTAs per SM: 30 and 420).  A lane takes the slots of its voxels one
// after another (most have one, at a border two): a slot's voxels are an and of the
// planes.
__global__ void __launch_bounds__(256, 4) k_wave_labels(const JobDesc* jobs, const JobState* st,
                                                        const uint32_t* list, const uint32_t* count,
                                                        const uint32_t* brick_job) {
  // fragment of each slot for the job of the current brick (reloaded when the
  // job changes): the seed's, or after a second flood the rank's
  __shared__ uint16_t lab[4096];
  int cached = -1;
  const uint32_t n = *count, part = threadIdx.x & 3u, sh = 8 * part, row = threadIdx.x >> 2;
  uint32_t b = blockIdx.x < n ? list[blockIdx.x] : 0u;
  uint32_t j = blockIdx.x < n ? brick_job[b] : 0u;
  for (uint32_t it = blockIdx.x; it < n;) {
    const JobDesc& J = jobs[j];
    const JobState& s = st[j];
    const bool active = J.active != 0 && !J.wflat;  // uniform across the CTA
    const uint32_t lb = b - J.brick_base;
    const uint32_t bz = lb % J.nbz, by = (lb / J.nbz) % J.nby, bx = lb / (J.nbz * J.nby);
    const uint32_t x = bx * VF_BX + row / VF_BY, y = by * VF_BY + row % VF_BY, z = bz * VF_BZ + sh;
    const uint32_t nq = J.wsw / 4;
    static_assert(64 % VF_BY == 0, "a pass is whole columns of rows");
    constexpr uint32_t DX = 64 / VF_BY;  // rows of a pass: DX columns
    const uint4* src = reinterpret_cast<const uint4*>(J.wstate + (size_t)(J.wrow0 + x * J.wsx + bz * J.wsy + y) * J.wsw);
    const size_t step = (size_t)DX * J.wsx * nq;  // from pass to pass
    const bool in = active && y < J.Y && z < J.Zp;
    const uint32_t X = J.X;
    uint16_t* const grid = J.grid + vf_gidx(J, x, y, z);
    const size_t gstep = (size_t)DX * J.Y * J.Zp;
    if (active && (int)j != cached) {  // uniform
      __syncthreads();
      const bool second = s.has_prefix && s.disjoint;
      const uint32_t nl = second ? 256u : min(s.nseeds, 4096u);
      for (uint32_t k = threadIdx.x; k < nl; k += blockDim.x)
        lab[k] = (uint16_t)((second ? s.rank_value[k] : J.seeds[4 * k + 3]) & 0xFFu);
      cached = (int)j;
      __syncthreads();
    }
    it += gridDim.x;
    if (it < n) {  // the next brick, on its way beside this one's rows
      b = list[it];
      j = brick_job[b];
    }
#pragma unroll
    for (int pass = 0; pass < 4; pass += 2) {
      uint4 a[2], c[2];  // planes A, B and slot bits 0 .. 5
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        a[h] = c[h] = make_uint4(0, 0, 0, 0);
        if (in && x + (pass + h) * DX < X) {
          a[h] = __ldcs(src + (pass + h) * step);
          c[h] = __ldcs(src + (pass + h) * step + 1);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!in || x + (pass + h) * DX >= X) continue;
        const uint32_t v = (wave_claimed(a[h].x, a[h].y) >> sh) & 0xFFu,
                       u = (wave_unclaimed(a[h].x, a[h].y) >> sh) & 0xFFu;
        auto pair = [](uint32_t m) { return ((m & 3u) * 0x8001u) & 0x00010001u; };
        uint4 out = make_uint4(pair(u), pair(u >> 2), pair(u >> 4), pair(u >> 6));
        const uint32_t p[6] = {a[h].z >> sh, a[h].w >> sh, c[h].x >> sh, c[h].y >> sh, c[h].z >> sh, c[h].w >> sh};
        for (uint32_t rem = v; rem;) {
          const uint32_t k = (uint32_t)__ffs(rem) - 1;
          uint32_t slot = 0, m = rem;  // the first voxel's slot, and its voxels
          auto plane = [&](uint32_t w, uint32_t bit) {
            const uint32_t one = (w >> k) & 1u;
            slot |= one << bit;
            m &= w ^ (one - 1u);
          };
#pragma unroll
          for (uint32_t bit = 0; bit < 6; ++bit) plane(p[bit], bit);
          for (uint32_t q = 2; q < nq; ++q) {  // more than 64 seeds
            const uint4 e = src[(pass + h) * step + q];
            plane(e.x >> sh, 4 * q - 2);
            plane(e.y >> sh, 4 * q - 1);
            plane(e.z >> sh, 4 * q);
            plane(e.w >> sh, 4 * q + 1);
          }
          const uint32_t L = lab[slot & 4095u];
          out.x += pair(m) * L;
          out.y += pair(m >> 2) * L;
          out.z += pair(m >> 4) * L;
          out.w += pair(m >> 6) * L;
          rem &= ~m;
        }
        *reinterpret_cast<uint4*>(grid + (pass + h) * gstep) = out;
      }
    }
  }
}
// ---- sub-seed prefixes ------------------------------------------------------
__device__ uint32_t slot_find(volatile uint32_t* uf, uint32_t a) {
  for (;;) {
    const uint32_t p = uf[a];
    if (p == a) return a;
    const uint32_t g = uf[p];
    if (g != p) uf[a] = g;  // halve the path; a is no root, so nobody else hooks it
    a = g;
  }
}
__device__ void slot_join(uint32_t* uf, uint32_t a, uint32_t b) {
  a = slot_find(uf, a);
  b = slot_find(uf, b);
  while (a != b) {
    if (a < b) {
      const uint32_t t = a;
      a = b;
      b = t;
    }
    const uint32_t old = atomicCAS(uf + a, a, b);  // hook the larger root
    if (old == a) return;
    a = slot_find(uf, old);
    b = slot_find(uf, b);
  }
}

// Joins the slots of one fragment whose voxels touch.  One thread per row: its
// own z neighbours, the four rows ahead of it in (x, y) at z - 1, z, z + 1, and
// from its top voxel the 3 x 3 rows of the word above; a difference of the
// planes finds the pairs, and only those are looked at voxel by voxel.  The same
// pair turns up all along a border, and a join waits for several reads of uf: a
// CTA remembers the pairs it has taken (a lost entry repeats a join).  200 x 197 x
// 208 voxels, 32 slots: 92 us (269 us with every pair joined).
__global__ void __launch_bounds__(256) k_slot_unions(const JobDesc* jobs, const JobState* st, WaveArrays arr,
                                                     const WaveJob* wj, uint32_t njobs) {
  uint32_t lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (wj[mid].base <= blockIdx.x * 256u) lo = mid; else hi = mid - 1;
  }
  const WaveJob& W = wj[lo];
  if (!st[W.job].has_prefix) return;
  const JobDesc& J = jobs[W.job];
  __shared__ uint32_t seen[1024];
  for (uint32_t k = threadIdx.x; k < 1024; k += 256) seen[k] = 0xFFFFFFFFu;
  __syncthreads();
  const uint32_t i = blockIdx.x * 256u + threadIdx.x, sw = J.wsw, nb = sw - 2;
  if (i < W.row0 || i + W.sx + W.sy + 1 >= W.base + W.nrows) return;
  const uint32_t* p = arr.state + (size_t)i * sw;
  const uint32_t V = wave_claimed(p[0], p[1]);
  if (!V) return;
  uint32_t L[14];
#pragma unroll
  for (uint32_t b = 0; b < 14; ++b) L[b] = b < nb ? p[2 + b] : 0u;
  // pairs of own bit k with bit k + s of row r (s = 31: bit 31 with bit 0)
  auto join = [&](uint32_t r, int s) {
    const uint32_t* q = arr.state + (size_t)r * sw;
    auto shift = [s](uint32_t v) { return s == 0 ? v : (s == 1 ? v >> 1 : (s == -1 ? v << 1 : v << 31)); };
    const uint32_t both = V & shift(wave_claimed(q[0], q[1]));
    if (!both) return;
    uint32_t d = 0;
#pragma unroll
    for (uint32_t b = 0; b < 14; ++b)
      if (b < nb) d |= L[b] ^ shift(q[2 + b]);
    uint32_t last = NO_SLOT;
    for (d &= both; d; d &= d - 1) {
      const uint32_t k = (uint32_t)__ffs(d) - 1;
      uint32_t a = 0, c = 0;
#pragma unroll
      for (uint32_t b = 0; b < 14; ++b)
        if (b < nb) {
          a |= ((L[b] >> k) & 1u) << b;
          c |= ((shift(q[2 + b]) >> k) & 1u) << b;
        }
      const uint32_t pair = min(a, c) << 12 | max(a, c);
      if (pair == last) continue;
      last = pair;
      volatile uint32_t* const at = seen + ((a * 31u + c * 31u + (a ^ c)) & 1023u);
      if (*at == pair) continue;
      *at = pair;
      if (((J.seeds[4 * a + 3] ^ J.seeds[4 * c + 3]) & 0xFFu) == 0) slot_join(J.uf, a, c);
    }
  };
  const uint32_t sx = W.sx, sy = W.sy;
  join(i, 1);
  if (W.conn6) {
    join(i + 1, 0);
    join(i + sx, 0);
    join(i + sy, 31);
    return;
  }
  const uint32_t ahead[4] = {i + 1, i + sx - 1, i + sx, i + sx + 1};
#pragma unroll 1
  for (int n = 0; n < 4; ++n)
    for (int s = -1; s <= 1; ++s) join(ahead[n], s);
#pragma unroll 1
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy) join(i + sy + (uint32_t)dx * sx + dy, 31);
}

// Per job: the lowest prefix of each set of slots, per fragment the minimum;
// uf becomes the second flood's slot of a slot's voxels, or NO_SLOT where they
// are reset.  One CTA per job.
__global__ void __launch_bounds__(256) k_slot_resolve(const JobDesc* jobs, JobState* st) {
  __shared__ uint32_t low[4096];
  __shared__ uint32_t reset;
  const JobDesc& J = jobs[blockIdx.x];
  JobState& s = st[blockIdx.x];
  if (!J.active || !s.has_prefix) return;
  const uint32_t ns = min(s.nseeds, 4096u);
  for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x) low[i] = 0xFFFFFFFFu;
  if (threadIdx.x == 0) reset = 0;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x)
    if (J.uf[i] != NO_SLOT) atomicMin(&low[slot_find(J.uf, i)], J.seeds[4 * i + 3] >> 8);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x)
    if (J.uf[i] != NO_SLOT) atomicMin(&s.minprefix[J.seeds[4 * i + 3] & 0xFFu], low[slot_find(J.uf, i)]);
  __syncthreads();
  if (threadIdx.x == 0) {
    // surviving values sorted -> re-flood slots (ties to the lowest value)
    uint32_t nr = 0;
    for (uint32_t f = 0; f < 256; ++f)
      if (s.minprefix[f] != 0xFFFFFFFFu) s.rank_value[nr++] = f | (s.minprefix[f] << 8);
    for (uint32_t a = 1; a < nr; ++a) {  // insertion sort, <= 254 entries
      const uint32_t v = s.rank_value[a];
      uint32_t b = a;
      while (b > 0 && s.rank_value[b - 1] > v) { s.rank_value[b] = s.rank_value[b - 1]; --b; }
      s.rank_value[b] = v;
    }
    for (uint32_t r = 0; r < nr; ++r) s.value_rank[s.rank_value[r] & 0xFFu] = r;
    s.nranks = nr;
  }
  // the roots are read before uf is rewritten
  uint32_t to[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const uint32_t i = threadIdx.x + 256u * k;
    to[k] = NO_SLOT;
    if (i < ns && J.uf[i] != NO_SLOT) {
      const uint32_t f = J.seeds[4 * i + 3] & 0xFFu;
      if (low[slot_find(J.uf, i)] == s.minprefix[f]) to[k] = f;
      else reset = 1;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const uint32_t i = threadIdx.x + 256u * k;
    if (i < ns) J.uf[i] = to[k] == NO_SLOT ? NO_SLOT : s.value_rank[to[k]];
  }
  if (threadIdx.x == 0) s.disjoint = reset;
}

// `in` of the jobs that flood again
__global__ void __launch_bounds__(256) k_slot_clear(const JobState* st, WaveArrays arr, const WaveJob* wj,
                                                    uint32_t njobs) {
  uint32_t lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (wj[mid].base <= blockIdx.x * 256u) lo = mid; else hi = mid - 1;
  }
  const JobState& s = st[wj[lo].job];
  if (!s.has_prefix || !s.disjoint) return;
  const size_t i = blockIdx.x * 256u + threadIdx.x;
  *reinterpret_cast<uint4*>(arr.in + 2 * i) = make_uint4(~0u, ~0u, ~0u, ~0u);
}

// disjointSetStack: voxels of non-minimal prefixes -> unclaimed; the survivors
// are the second flood's wave 0, keyed by their rank.  One thread per row;
// every row with unclaimed voxels becomes a candidate of wave 0.
__global__ void __launch_bounds__(256) k_slot_reset(const JobDesc* jobs, const JobState* st, WaveArrays arr,
                                                    const WaveJob* wj, uint32_t njobs) {
  uint32_t lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (wj[mid].base <= blockIdx.x * 256u) lo = mid; else hi = mid - 1;
  }
  const WaveJob& W = wj[lo];
  const JobState& s = st[W.job];
  if (!s.has_prefix || !s.disjoint) return;
  const JobDesc& J = jobs[W.job];
  const uint32_t i = blockIdx.x * 256u + threadIdx.x, sw = J.wsw;
  if (i < W.row0 || i + W.sx + W.sy + 1 >= W.base + W.nrows) return;
  uint32_t* p = arr.state + (size_t)i * sw;
  uint32_t v = wave_claimed(p[0], p[1]), u = wave_unclaimed(p[0], p[1]);
  if (!(u | v)) return;
  uint32_t L[14], w[14];
#pragma unroll
  for (uint32_t b = 0; b < 14; ++b) {
    L[b] = b < sw - 2 ? p[2 + b] : 0u;
    w[b] = 0;
  }
  uint32_t keep = 0;
  for (uint32_t m = v; m; m &= m - 1) {
    const uint32_t k = (uint32_t)__ffs(m) - 1, bit = m & (0u - m);
    uint32_t slot = 0;
#pragma unroll
    for (uint32_t b = 0; b < 14; ++b) slot |= ((L[b] >> k) & 1u) << b;
    const uint32_t r = J.uf[slot];
    if (r == NO_SLOT) continue;
    keep |= bit;
#pragma unroll
    for (uint32_t b = 0; b < 8; ++b) w[b] |= (r >> b) & 1u ? bit : 0u;  // ranks are below 256
    // wave 0's claims at the word's ends reach the rows below and above
    for (int e = 0; e < 2; ++e) {
      if (k != (e ? 31u : 0u)) continue;
      const uint32_t j = e ? i + W.sy : i - W.sy;
      for (int dx = -1; dx <= 1; ++dx)
        for (int dy = -1; dy <= 1; ++dy) {
          if (W.conn6 && (dx || dy)) continue;
          uint2* to = arr.in + 2 * (size_t)(j + (uint32_t)dx * W.sx + dy);
          atomicMin(e ? &to->x : &to->y, in_key(0, r));
        }
    }
  }
  u |= v & ~keep;
  p[0] = wave_empty_a(u | keep);  // the survivors as E0
  p[1] = wave_empty_b(u);
#pragma unroll
  for (uint32_t b = 0; b < 14; ++b)
    if (b < sw - 2) p[2 + b] = w[b];
  if (u) atomicOr(arr.cand + (i >> 5), 1u << (i & 31u));
}

}  // namespace

namespace vfk {

static inline int brick_grid(uint32_t max_count) {
  uint32_t g = max_count ? max_count : 1;
  return (int)(g > (1u << 20) ? (1u << 20) : g);
}

uint32_t wave_state_words(uint32_t nseeds) {
  // 6 planes (64 slots) fill 32 bytes with A and B, one 256-bit load per row; 10
  // planes fill 48; 12 hold every slot (4095 seeds) in 64
  return (uint32_t)(nseeds <= 64 ? state_words(6) : (nseeds <= 1024 ? state_words(10) : state_words(12)));
}
uint64_t wave_rows(uint32_t nx, uint32_t ny, uint32_t nw) {
  const uint64_t sy = ny + 1ull, sx = (nw + 1ull) * sy;
  return (nx + 2ull) * sx + sy + 3;
}
void wave_layout(WaveJob& W, uint32_t base, uint32_t nx, uint32_t ny, uint32_t nw) {
  W.base = base;
  W.sy = ny + 1;
  W.sx = (nw + 1) * W.sy;
  W.row0 = base + W.sx + W.sy + 1;
  W.nrows = (uint32_t)wave_rows(nx, ny, nw);
}
uint32_t wave_order(uint32_t X, uint32_t Y, uint32_t Z) {
  // Words along z, also in a flat grid, whose words are mostly empty bits: a front
  // that runs along the plane claims such a row in one wave (1024 x 1024 x 8 voxels,
  // full, Manhattan: 2.29 ms, 2.55 with words along x).  Where a large grid has at
  // least 8 times fewer rows with words along its longest axis (z up to 5 voxels), the
  // scans and the memory of the others count: 4096 x 4096 x 2 8.4 against 13.3 ms and
  // 0.1 against 1.6 GB, 2048 x 2048 x 4 4.9 against 5.0 ms.
  constexpr uint64_t FLAT_ROWS = 4 << 20, FLAT_GAIN = 8;
  const uint32_t D[3] = {X, Y, Z}, w = X > Y ? 0u : 1u, l = 1u - w;
  const uint64_t rows = wave_rows(X, Y, (Z + 31) / 32);
  if (rows < FLAT_ROWS || wave_rows(Z, D[l], (D[w] + 31) / 32) * FLAT_GAIN > rows) return WAVE_XYZ;
  return 2u | l << 4 | w << 8;
}
uint64_t wave_job_rows(uint32_t X, uint32_t Y, uint32_t Z) {
  const FlatAxes A = wave_axes(X, Y, Z, Z);
  return wave_rows(A.nx, A.ny, (A.nz + 31) / 32);
}
FlatAxes wave_axes(uint32_t X, uint32_t Y, uint32_t Z, uint32_t pitch) {
  const uint32_t D[3] = {X, Y, Z}, order = wave_order(X, Y, Z);
  const size_t stride[3] = {(size_t)Y * pitch, pitch, 1};
  const uint32_t a = order & 15u, b = (order >> 4) & 15u, c = order >> 8;
  return {{stride[a], stride[b], stride[c]}, D[a], D[b], D[c], {X, Y, Z}, order};
}

void flood_seed_bricks(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs, uint8_t* live,
                       uint32_t* list, uint32_t* count) {
  if (njobs > 0) k_seed_bricks<<<njobs, 128, 0, st>>>(dj, ds, live, list, count);
}

void flood_init(cudaStream_t st, const JobDesc* dj, JobState* ds, const FloodScratch& fs, const uint8_t* live, bool planes) {
  if (!fs.units) return;
  if (planes)
    k_wave_planes<<<std::min<uint32_t>(fs.units, (uint32_t)fs.shape.sms * 32), 256, 0, st>>>(dj, ds, fs.arr, fs.jobs,
                                                                                           fs.njobs, fs.units);
  else
    k_wave_init<<<fs.units, 256, 0, st>>>(dj, ds, fs.arr, fs.jobs, fs.njobs, live);
}

// launch shape of k_wave: threads per CTA and dynamic shared memory
namespace {
constexpr size_t WAVE_SMEM = sizeof(WaveShared) + 2 * 4 * (SMALL_ROWS / 32 + 8);

template <int NB, int THREADS>
int wave_per_sm() {
  static int per_sm[64] = {};  // per device: the attribute is set on each device
  const int dv = cur_dev();
  if (per_sm[dv] < 1) {
    int n = 0;
    const auto k = k_wave<NB, THREADS>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WAVE_SMEM);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, THREADS, WAVE_SMEM) != cudaSuccess) n = 1;
    per_sm[dv] = n < 1 ? 1 : n;
  }
  return per_sm[dv];
}
template <int THREADS>
int wave_per_sm(uint32_t sw) {
  return sw <= 8 ? wave_per_sm<6, THREADS>() : (sw <= 12 ? wave_per_sm<10, THREADS>() : wave_per_sm<12, THREADS>());
}
template <int THREADS>
const void* wave_kernel(uint32_t sw) {
  return sw <= 8 ? (const void*)k_wave<6, THREADS>
                 : (sw <= 12 ? (const void*)k_wave<10, THREADS> : (const void*)k_wave<12, THREADS>);
}
}  // namespace

WaveShape flood_shape(uint32_t sw, uint32_t njobs, int num_sms, int ctas_per_sm) {
  WaveShape s;
  s.sms = num_sms;
  // one flood: the rows of a wave fit one CTA per SM, whose 16 warps hide each
  // other's latency; a batch: two CTAs, one of each gang
  s.threads = njobs < 2 ? 512 : 256;
  int per = s.threads == 512 ? wave_per_sm<512>(sw) : wave_per_sm<256>(sw);
  if (ctas_per_sm > 0) per = std::min(per, ctas_per_sm);
  s.blocks = per * num_sms;
  return s;
}

uint32_t flood_gang(uint64_t rows, uint32_t blocks, uint32_t min_size) {
  // A CTA per 1024 rows up to 128 of them, then per 4096.  Full cubes, Manhattan, with
  // 4096 and 1024 rows a CTA throughout: 128^3 965 and 760 us, 160^3 1200 and 987, 200^3
  // 1405 and 1306; a vessel of 240 x 240 x 256 (525 k rows) 510 on 129 CTAs, 520 on 152.
  const uint64_t size = std::max<uint64_t>(std::min<uint64_t>((rows + 1023) / 1024, 128), (rows + 4095) / 4096);
  return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(size, min_size), blocks);
}

uint32_t flood_gangs(const uint64_t* rows, uint32_t n, uint32_t* gang_of) {
  bool small = true;
  for (uint32_t i = 0; i < n; ++i) small &= rows[i] <= SMALL_ROWS;
  if (small) {
    for (uint32_t i = 0; i < n; ++i) gang_of[i] = i;
    return n;
  }
  if (n < 2) {
    gang_of[0] = 0;
    return 1;
  }
  // two sets of equal size, the largest job first, each to the smaller set
  // (more sets where a set would have too many jobs)
  const uint32_t k = std::max(2u, (n + WAVE_GANG_JOBS / 2 - 1) / (WAVE_GANG_JOBS / 2));
  std::vector<uint32_t> order(n);
  for (uint32_t i = 0; i < n; ++i) order[i] = i;
  std::sort(order.begin(), order.end(),
            [&](uint32_t a, uint32_t b) { return rows[a] != rows[b] ? rows[a] > rows[b] : a < b; });
  std::vector<uint64_t> load(k, 0);
  std::vector<uint32_t> count(k, 0);
  for (uint32_t i : order) {
    uint32_t best = k;
    for (uint32_t g = 0; g < k; ++g)
      if (count[g] < WAVE_GANG_JOBS && (best == k || load[g] < load[best])) best = g;
    gang_of[i] = best;
    load[best] += rows[i];
    ++count[best];
  }
  return k;
}

// One-CTA gangs are dealt to all CTAs, the largest first, each to the least
// loaded one.  Larger gangs of small floods lie side by side, as wide as all of them
// fit; those of large floods alternate between as many sets of CTAs as fit an SM.
// Every CTA runs its gangs of several CTAs in their order, so that none waits for one
// that waits for it.
uint32_t flood_schedule(const WaveGang* gangs, uint32_t n, const WaveShape& shape, uint32_t min_size, WaveCta* cta,
                        WaveEntry* entries) {
  const uint32_t C = (uint32_t)shape.blocks, sms = (uint32_t)std::max(shape.sms, 1);
  std::vector<std::vector<WaveEntry>> lists(C);
  bool small_floods = true;
  for (uint32_t g = 0; g < n; ++g) small_floods &= gangs[g].units * 256 <= SMALL_ROWS;
  const uint32_t sets = n > 1 ? std::max(1u, std::min(n, C / sms)) : 1u;
  const uint32_t width = std::max(1u, std::min(small_floods && n ? std::max(C / n, min_size) : C / sets, sms));
  std::vector<uint32_t> small;
  uint32_t next = 0;  // of small floods: the first CTA past the last gang's
  for (uint32_t g = 0; g < n; ++g) {
    const uint32_t size = flood_gang((uint64_t)gangs[g].units * 256, std::min(width, C), min_size);
    if (size < 2) {
      small.push_back(g);
      continue;
    }
    if (next + size > C) next = 0;
    const uint32_t at = small_floods ? next : (g % sets) * width;
    next += size;
    for (uint32_t r = 0; r < size; ++r) lists[at + r].push_back({g, r, size, 0});
  }
  std::sort(small.begin(), small.end(), [&](uint32_t a, uint32_t b) {
    return gangs[a].units != gangs[b].units ? gangs[a].units > gangs[b].units : a < b;
  });
  std::vector<uint64_t> load(C, 0);
  for (uint32_t c = 0; c < C; ++c)
    for (const WaveEntry& e : lists[c]) load[c] += gangs[e.gang].units / e.size + 1;
  auto later = [&](uint32_t a, uint32_t b) { return load[a] != load[b] ? load[a] > load[b] : a > b; };
  std::vector<uint32_t> heap(C);
  for (uint32_t c = 0; c < C; ++c) heap[c] = c;
  std::make_heap(heap.begin(), heap.end(), later);
  for (uint32_t g : small) {
    std::pop_heap(heap.begin(), heap.end(), later);
    const uint32_t c = heap.back();
    lists[c].push_back({g, 0, 1, 0});
    load[c] += gangs[g].units;
    std::push_heap(heap.begin(), heap.end(), later);
  }
  uint32_t at = 0;
  for (uint32_t c = 0; c < C; ++c) {
    cta[c] = {at, (uint32_t)lists[c].size()};
    for (const WaveEntry& e : lists[c]) entries[at++] = e;
  }
  return at;
}

cudaError_t flood_seed(cudaStream_t st, const JobDesc* dj, const JobState* ds, const FloodScratch& fs) {
  cudaError_t e = cudaMemsetAsync(fs.zero, 0, fs.zero_bytes, st);
  if (e == cudaSuccess && fs.njobs) k_wave_seed<<<fs.njobs, 256, 0, st>>>(dj, ds, fs.arr, fs.jobs);
  return e;
}

cudaError_t flood_waves(cudaStream_t st, JobState* ds, const FloodScratch& fs) {
  WaveArgs a;
  a.arr = fs.arr;
  a.jobs = fs.jobs;
  a.gangs = fs.gangs;
  a.last = fs.last;
  a.cta = fs.cta;
  a.entries = fs.entries;
  a.st = ds;
  a.bar = fs.bar;
  a.err = fs.err;
  a.stats = fs.stats;
  a.wave_sizes = fs.wave_sizes;
  a.wait_spins = fs.wait_spins ? fs.wait_spins : (1u << 23);
  a.smem_words = (uint32_t)((WAVE_SMEM - sizeof(WaveShared)) / 4);
  a.lone_voxels = fs.wait_spins ? 0u : LONE_VOXELS;  // a wait limit is for gangs that wait
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(fs.shape.threads == 512 ? wave_kernel<512>(fs.sw) : wave_kernel<256>(fs.sw),
                                     dim3(fs.shape.blocks), dim3(fs.shape.threads), args, WAVE_SMEM, st);
}

static int flat_grid(const WaveJob& W, int num_sms) {  // a warp per row, 16 CTAs per SM at most
  return (int)std::max<uint32_t>(1, std::min<uint32_t>((W.nrows + 7) / 8, 16u * (uint32_t)num_sms));
}
void flat_init(cudaStream_t st, const uint16_t* grid, const WaveArrays& arr, const WaveJob& W, const FlatAxes& A,
               uint32_t sw, JobState* ds, int num_sms) {
  k_flat_init<<<flat_grid(W, num_sms), 256, 0, st>>>(grid, arr, W, A, sw, ds);
}
void flat_seed(cudaStream_t st, const WaveJob& W, const FlatAxes& A, const FloodScratch& fs, const uint32_t* seeds,
               uint32_t ns, JobState* ds) {
  const uint32_t size = flood_gang(W.nrows, (uint32_t)std::min(fs.shape.blocks, fs.shape.sms), 1);
  k_flat_seed<<<1, 256, 0, st>>>(fs.arr, W, A, fs.sw, seeds, ns, size, (uint32_t)fs.shape.blocks, ds,
                                 const_cast<WaveJob*>(fs.jobs), const_cast<WaveGang*>(fs.gangs),
                                 const_cast<WaveCta*>(fs.cta), const_cast<WaveEntry*>(fs.entries));
}
void flat_labels(cudaStream_t st, const WaveArrays& arr, const WaveJob& W, const FlatAxes& A, uint32_t sw,
                 const uint32_t* seeds, const JobState* ds, uint16_t* labels, int num_sms) {
  k_flat_labels<<<flat_grid(W, num_sms), 256, 0, st>>>(arr, W, A, sw, seeds, ds, labels);
}

void flood_labels(cudaStream_t st, const JobDesc* dj, const JobState* ds, const uint32_t* list,
                  const uint32_t* count, uint32_t max_count, const uint32_t* brick_job, int num_sms) {
  // resident CTAs: four of 256 threads fit an SM beside their 64 registers
  if (max_count)
    k_wave_labels<<<std::min(brick_grid(max_count), std::max(num_sms, 1) * 4), 256, 0, st>>>(dj, ds, list, count, brick_job);
}

cudaError_t flood_prefixes(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs, const FloodScratch& fs) {
  if (!fs.units) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(fs.zero, 0, fs.zero_bytes, st);
  if (e != cudaSuccess) return e;
  k_slot_unions<<<fs.units, 256, 0, st>>>(dj, ds, fs.arr, fs.jobs, fs.njobs);
  k_slot_resolve<<<njobs, 256, 0, st>>>(dj, ds);
  k_slot_clear<<<fs.units, 256, 0, st>>>(ds, fs.arr, fs.jobs, fs.njobs);
  k_slot_reset<<<fs.units, 256, 0, st>>>(dj, ds, fs.arr, fs.jobs, fs.njobs);
  return cudaGetLastError();
}

}  // namespace vfk
