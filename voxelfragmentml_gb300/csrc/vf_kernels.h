// vf_kernels.h -- host launchers of the device stages (internal).
//
// Every launcher takes a device array of JobDesc (one table per stage, see
// vf_runtime.cu) plus the per-job JobState array, and enqueues on `st`.
// Brick-parallel stages take the list of live bricks and brick_job map.
#pragma once
#include <string>
#include "vf_common.cuh"

namespace vfk {

// ---- voxelizer (Tetravoxelizer + tri-box SAT) ----
// flattened per-face work list (parity: slice planes crossing the face;
// shell: candidate columns): per-face counts and their exclusive prefix sums
// over the faces of all jobs
struct FaceScratch {
  uint32_t* pcnt;                // [total_faces]
  unsigned long long* pbase;     // [total_faces]
  unsigned long long* psums;     // [ceil(total_faces / 1024)]
  unsigned long long* ptotal;    // [1]
};
void centroid_and_slices(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs);
void tetra_prep(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs,
                uint32_t total_faces, const FaceScratch& fs);
void parity_raster(cudaStream_t st, const JobDesc* dj, const JobState* ds, int njobs,
                   uint32_t total_faces, const FaceScratch& fs, int num_sms, int grid_mult = 16);
// reuses the face scratch after the parity raster (counts, scan, runs)
void shell_sat(cudaStream_t st, const JobDesc* dj, int njobs, uint32_t total_faces,
               const FaceScratch& fs, int num_sms, int grid_mult = 12);
// writes 0/1 labels (grid, and grid2 when dual) for every brick of every
// job and sets live[b]
void combine(cudaStream_t st, const JobDesc* dj, const uint32_t* brick_job,
             uint32_t total_bricks, uint8_t* live, int dual);
void mark_live(cudaStream_t st, const JobDesc* dj, const uint32_t* brick_job,
               uint32_t total_bricks, uint8_t* live);
void compact_live(cudaStream_t st, const uint8_t* live, uint32_t first, uint32_t total_bricks,
                  uint32_t* list, uint32_t* count);

// labels of every job with a device-accessible `out` (T_CNT table: the
// final buffer) into `out`, rows of Z without the z padding
// rows [row0, row0 + rows) of the batch are those of the njobs jobs at dj
void pack_labels(cudaStream_t st, const JobDesc* dj, int njobs, uint64_t row0, uint64_t rows, int num_sms,
                 int ctas_per_sm);

// exclusive prefix sum of n u32 into u64 (sums: ceil(n / 1024) + 1 scratch
// words); *total = the sum
void exclusive_scan(cudaStream_t st, const uint32_t* in, unsigned long long* out,
                    unsigned long long* sums, uint32_t n, unsigned long long* total);

// ---- RLE export (vf_rle.cu) ----
// run starts counted per (x, y) row of a grid [X][Y][Zp]
void rle_count(cudaStream_t st, const uint16_t* g, uint32_t X, uint32_t Y, uint32_t Z, uint32_t Zp,
               uint32_t* row_cnt, int num_sms);
// records {u16 value, u32 repetitions} as 3 u16 per run, from the scanned
// row counts; starts: scratch of one u64 per run
void rle_write(cudaStream_t st, const uint16_t* g, uint32_t X, uint32_t Y, uint32_t Z, uint32_t Zp,
               const unsigned long long* row_base, const unsigned long long* nruns,
               unsigned long long* starts, uint16_t* records, int num_sms);

// ---- marching cubes per fragment (vf_mesh.cu) ----
struct MeshGrid {
  const uint16_t* g;  // [X][Y][Zp] labels
  uint32_t X, Y, Z, Zp;
};
// the case table packed for the kernels: 4 bits per edge, triangle count
void mc_pack_table(unsigned long long tri[256], uint8_t ntri[256]);
// exposed-face masks (X*Y*Z bytes), vertices per grid row, present[value]
void mc_vertex_count(cudaStream_t st, const MeshGrid& G, uint8_t* mask, uint32_t* rcnt,
                     uint8_t* present, int num_sms);
// vertex id base per voxel, fragment key and (voxel * 8 + direction) per vertex
void mc_vertex_emit(cudaStream_t st, const MeshGrid& G, const uint8_t* mask,
                    const unsigned long long* rbase, const uint16_t* dense, uint32_t* vbase,
                    uint16_t* vkey, unsigned long long* vown, int num_sms);
// triangles per cell row ((X+1)*(Y+1) rows of Z+1 cells)
void mc_tri_count(cudaStream_t st, const MeshGrid& G, const unsigned long long* tri,
                  const uint8_t* ntri, uint32_t* rcnt, int num_sms);
void mc_tri_emit(cudaStream_t st, const MeshGrid& G, const unsigned long long* tri,
                 const uint8_t* ntri, const unsigned long long* rbase, const uint8_t* mask,
                 const uint32_t* vbase, const uint16_t* dense, uint16_t* tkey, uint4* tv,
                 uint32_t* vflag, uint32_t* err, int num_sms);
// stable order of items 0..n-1 by key[item] (< nkeys <= 65536) into out;
// tmp: n words (two passes), hist: split_hist_words(n) words, hbase the
// same count of u64, sums/tot: exclusive_scan scratch for that many words;
// off[f] = first sorted position with key >= f, f = 0..nkeys
size_t split_hist_words(uint64_t n);
void stable_split16(cudaStream_t st, const uint16_t* key, uint64_t n, uint32_t nkeys, uint32_t* tmp,
                    uint32_t* out, uint32_t* hist, unsigned long long* hbase,
                    unsigned long long* sums, unsigned long long* tot, unsigned long long* off);
// bnd (or NULL): inc_chunks(V) zeroed counts, of the boundary vertices of each
// inc_chunk(V) vertices
uint32_t inc_chunk(uint64_t V);
uint32_t inc_chunks(uint64_t V);
void mc_outputs(cudaStream_t st, const MeshGrid& G, const uint32_t* vperm,
                const unsigned long long* vown, const uint32_t* vflag, uint64_t V, const float s[3],
                const float c[3], uint32_t* vinv, float4* vert, const uint32_t* tperm,
                const uint4* tv, uint64_t T, uint4* gface, uint32_t* bnd, int num_sms);
// smoothSurface (MarchingCubes.cpp:489-510), in two steps.  mc_smooth_lists:
// per vertex, the distinct neighbours (with multiplicity) of the faces its
// pass sums; scratch deg V u32, start V + 1 u64, sums exclusive_scan scratch for
// V, ent one uint2 per counted face incidence (at most 3 T), nbr
// inc_entries(V, T) u32, item /
// meta V u32 / uint2, bnd / bbase mc_outputs' counts and as many u64, stats 4 u64
// (boundary vertices, their neighbour entries, all entries, scratch); err bit 2 if a vertex has more incidences
// than its meta holds; needs V < 2^28.  mc_smooth_iterate: nb_iters over the
// non-boundary vertices, then b_iters over the boundary ones (tmp: V float4).
uint64_t inc_entries(uint64_t V, uint64_t T);
cudaError_t mc_smooth_lists(cudaStream_t st, const uint4* gface, uint64_t T, const float4* vert,
                            uint64_t V, const uint32_t* bnd, unsigned long long* bbase, uint32_t* deg,
                            unsigned long long* start, unsigned long long* sums, uint2* ent, uint32_t* nbr,
                            uint32_t* item, uint2* meta, uint32_t* err, unsigned long long* stats, int num_sms);
cudaError_t mc_smooth_iterate(cudaStream_t st, float4* vert, float4* tmp, uint64_t V,
                              const uint32_t* item, const uint2* meta, const uint32_t* nbr,
                              const unsigned long long* stats, uint32_t nb_iters, float nb_weight,
                              uint32_t b_iters, float b_weight, int num_sms);
void mc_local_faces(cudaStream_t st, const uint4* gface, const uint32_t* tperm, const uint16_t* tkey,
                    const unsigned long long* voff, uint64_t T, uint4* out, int num_sms);

// ---- impact path (vf_impact.cu) ----
struct ImpactGrid {
  const uint16_t* g;  // [X][Y][Zp] labels
  uint32_t X, Y, Z, Zp;
  float amin[3], amax[3], cell[3];  // the grid's box and (amax - amin) / dims
};
// cells of 2^shift voxels a side with an occupied voxel, one bit each
struct RayCells {
  uint32_t shift, ny, nz, words;
};
RayCells ray_cells(uint32_t X, uint32_t Y, uint32_t Z);
// per ray (origin xyz, direction xyz): the 1-based index of the first occupied
// voxel, 0xFFFFFFFF x3 when none.  bits (X * Y * ceil(Z / 32) + cells.words words,
// or NULL): scratch for the packed occupancy the walks read instead of the labels;
// state (with bits; 2 words): scratch, and the lowest ray without a direction or
// 0xFFFFFFFF (without bits the caller looks for them)
cudaError_t ray_entry(cudaStream_t st, const ImpactGrid& G, const float* rays, uint32_t n, uint32_t* out,
                      uint32_t* bits, const RayCells& cells, uint32_t* state, int num_sms);
// Seeder::nearSeeds: the new seeds (4 uint32 each, labels label0 + 1, ...)
// in (x, y, z) order into out; status[0] = count, status[1] = 0 or
// VF_ERR_SEED_SEARCH.  Needs nfrags >= 1, num_seeds <= 4095 and
// 1 <= spreading <= min(dims) when num_impacts > 0.
void near_seeds(cudaStream_t st, const ImpactGrid& G, const uint32_t* frags, uint32_t nfrags,
                uint32_t num_impacts, uint32_t num_seeds, uint32_t spreading, uint64_t seed,
                uint32_t label0, uint32_t* out, uint32_t* status);

// ---- point sampling of meshes (vf_sample.cu) ----
struct SampleMeshes {
  const float4* verts;  // x, y, z, (w)
  const uint4* faces;   // three vertex indices within the mesh, (w)
  const unsigned long long* vert_off;  // F + 1
  const unsigned long long* face_off;  // F + 1
  const uint32_t* keys;                // F: the noise and draw key of each mesh
  uint32_t F;
  uint64_t nfaces;
};
// areas, per-chunk sums (chunks of at most 1024 faces that start at each
// mesh's first face: cstart/cend, mchunk[m] = first chunk of mesh m, F + 1),
// per mesh sumArea (msum) and noise length (nb)
void pc_areas(cudaStream_t st, const SampleMeshes& M, float* area, const unsigned long long* cstart,
              const unsigned long long* cend, uint32_t nchunks, double* csum, float* cmax,
              const unsigned long long* mchunk, uint32_t S, float* msum, uint64_t* nb, int num_sms);
// for the meshes listed in sel (S <= T): S distinct faces into the bitmap
// chosen (one bit per global face, zeroed); err bit 0 if the draws run out
void pc_select(cudaStream_t st, const SampleMeshes& M, const uint32_t* sel, uint32_t nsel, uint32_t S,
               uint64_t seed, uint32_t* chosen, uint32_t* err);
// samples per face (cnt), their exclusive scan (soff, nfaces + 1), P per mesh
void pc_count(cudaStream_t st, const SampleMeshes& M, const float* area, const float* msum,
              const uint8_t* big, uint32_t S, const uint32_t* chosen, uint32_t* cnt,
              unsigned long long* P, unsigned long long* soff, unsigned long long* sums, int num_sms);
// the points (x, y, z, 1) of mesh m at out[out_off[m] ..]
void pc_points(cudaStream_t st, const SampleMeshes& M, const uint32_t* cnt, const unsigned long long* soff,
               const uint64_t* nb, const uint8_t* big, const unsigned long long* out_off, uint32_t S,
               uint64_t seed, float4* out, int num_sms);

// ---- seeds ----
void sample_seeds(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs);

// ---- fracturers ----
void naive(cudaStream_t st, const JobDesc* dj, const JobState* ds, const uint32_t* list,
           const uint32_t* count, uint32_t max_count, const uint32_t* brick_job);

// ---- grid passes (brick kernels, live bricks only) ----
void lattice(cudaStream_t st, const JobDesc* dj, int njobs);
void perturb(cudaStream_t st, const JobDesc* dj, const uint32_t* list, const uint32_t* count,
             uint32_t max_count, const uint32_t* brick_job);
void detect_boundaries(cudaStream_t st, const JobDesc* dj, const uint32_t* list,
                       const uint32_t* count, uint32_t max_count, const uint32_t* brick_job);
// boundary sizes 2..3
void detect_boundaries_wide(cudaStream_t st, const JobDesc* dj, const uint32_t* list,
                            const uint32_t* count, uint32_t max_count, const uint32_t* brick_job);
void erode(cudaStream_t st, const JobDesc* dj, const uint32_t* list, const uint32_t* count,
           uint32_t max_count, const uint32_t* brick_job);
void remove_isolated(cudaStream_t st, const JobDesc* dj, const uint32_t* list,
                     const uint32_t* count, uint32_t max_count, const uint32_t* brick_job);
void count_values(cudaStream_t st, const JobDesc* dj, JobState* ds, const uint32_t* list,
                  const uint32_t* count, uint32_t max_count, const uint32_t* brick_job);

// the current device, as an index into per-device caches of launch
// attributes (a kernel's shared-memory limit is set once per device)
inline int cur_dev() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) d = 0;
  return d & 63;
}

// ---- flood (vf_flood.cu) ----
// The floods of a batch share arrays of rows, 32 voxels along a word axis
// each.
struct WaveArrays {
  uint32_t* state;  // [rows] state words (wave_state_words)
  uint2* in;        // [rows][2] what reaches the word ends from below (.x) / above (.y), by wave parity
  uint32_t* cand;   // [2][nwords] a candidate bit per row, by wave parity
  uint32_t nwords;  // rows / 32
};
// One flood: rows base .. base + nrows of the arrays (base a multiple of 256, up
// to the next job's base).  Row (outer x, word, y) is row0 + x * sx + word * sy
// + y, with at least one EMPTY row on each side of every axis, so the
// neighbours of a row are rows +- sx, +- sy, +- 1.  A job's axes are (x, y, z) with
// words along z, or any permutation.
struct WaveJob {
  uint32_t base, nrows, row0, sx, sy;
  uint32_t conn6;  // 6-neighbourhood (Manhattan), else 26
  uint32_t job;    // its JobState
  uint32_t order;  // nibble a: the grid axis of state axis a (outer, rows, words)
};
constexpr uint32_t WAVE_XYZ = 0x210u;  // words along z
struct FlatAxes {
  size_t s[3];       // element strides of the state's axes (outer, rows, words)
  uint32_t nx, ny, nz;  // voxels along them
  uint32_t dims[3];  // X, Y, Z
  uint32_t order;    // nibble a: the grid axis of state axis a
};
uint64_t wave_rows(uint32_t nx, uint32_t ny, uint32_t nw);
// the axes of a job's state, the rows it needs with them; pitch: elements of a z row
uint32_t wave_order(uint32_t X, uint32_t Y, uint32_t Z);
FlatAxes wave_axes(uint32_t X, uint32_t Y, uint32_t Z, uint32_t pitch);
uint64_t wave_job_rows(uint32_t X, uint32_t Y, uint32_t Z);
void wave_layout(WaveJob& W, uint32_t base, uint32_t nx, uint32_t ny, uint32_t nw);
// Jobs flooded in step: wave jobs first .. first + count, whose rows are units
// unit_lo .. unit_lo + units of 256 rows
struct WaveGang {
  uint32_t first, count, unit_lo, units;
};
constexpr uint32_t WAVE_GANG_JOBS = 256;  // most jobs of a gang
struct WaveEntry {
  uint32_t gang, rank, size, pad;  // this CTA's rank in the gang, CTAs of the gang
};
struct WaveCta {
  uint32_t first, count;  // entries of one CTA, run in order
};
// u32 words of a row state for floods of up to nseeds seeds (8, 12 or 16)
uint32_t wave_state_words(uint32_t nseeds);
constexpr uint32_t WAVE_BAR_WORDS = 32;  // barrier words per gang

struct WaveShape {
  int blocks = 0, threads = 256, sms = 0;
};
struct FloodScratch {
  WaveArrays arr = {};
  uint32_t units = 0;                  // 256-row units of all jobs
  const WaveJob* jobs = nullptr;       // device, njobs
  uint32_t njobs = 0;
  const WaveGang* gangs = nullptr;     // device
  const WaveCta* cta = nullptr;        // device, shape.blocks
  const WaveEntry* entries = nullptr;  // device
  WaveShape shape;                     // of the launch (flood_shape)
  uint32_t sw = 8;                     // state words of every job of the batch
  uint32_t* bar = nullptr;             // [gangs][WAVE_BAR_WORDS]
  uint32_t* last = nullptr;            // [njobs]
  void* zero = nullptr;                // candidate words, bar, last: cleared before a flood
  size_t zero_bytes = 0;
  uint32_t* err = nullptr;             // [1] global error word
  uint32_t* stats = nullptr;           // [VF_FLOOD_NCOUNTERS]
  uint32_t* wave_sizes = nullptr;      // statistics: rows visited per wave (256)
  uint32_t wait_spins = 0;             // polls of a gang barrier before it gives up (0: 2^23, ~4 s)
};
// launch shape of the waves of njobs floods (ctas_per_sm > 0: at most that many
// CTAs per SM); also sets the kernel's attributes (once per device, outside a
// stream capture)
WaveShape flood_shape(uint32_t sw, uint32_t njobs, int num_sms, int ctas_per_sm);
// the gangs of n floods of rows[i] rows: their number, the gang of each
uint32_t flood_gangs(const uint64_t* rows, uint32_t n, uint32_t* gang_of);
// CTAs of a gang, min_size to blocks
uint32_t flood_gang(uint64_t rows, uint32_t blocks, uint32_t min_size);
// the CTAs of n gangs: cta[shape.blocks], entries (at most n * shape.sms + n);
// returns the entries
uint32_t flood_schedule(const WaveGang* gangs, uint32_t n, const WaveShape& shape, uint32_t min_size, WaveCta* cta,
                    WaveEntry* entries);
void flood_seed_bricks(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs, uint8_t* live,
                       uint32_t* list, uint32_t* count);
// row states from the labels
// planes: the labels are the voxelizer's occupancy, still in its bit planes
void flood_init(cudaStream_t st, const JobDesc* dj, JobState* ds, const FloodScratch& fs, const uint8_t* live,
                bool planes);
cudaError_t flood_seed(cudaStream_t st, const JobDesc* dj, const JobState* ds, const FloodScratch& fs);
cudaError_t flood_waves(cudaStream_t st, JobState* ds, const FloodScratch& fs);
void flood_labels(cudaStream_t st, const JobDesc* dj, const JobState* ds, const uint32_t* list,
                  const uint32_t* count, uint32_t max_count, const uint32_t* brick_job, int num_sms);
// sub-seed prefix competition and the disjoint cleanup after a flood: the jobs
// whose voxels were reset are ready for the second flood
cudaError_t flood_prefixes(cudaStream_t st, const JobDesc* dj, JobState* ds, int njobs, const FloodScratch& fs);

// ---- a flood on an unpadded device grid (vf_flood_noalloc) ----
void flat_init(cudaStream_t st, const uint16_t* grid, const WaveArrays& arr, const WaveJob& W, const FlatAxes& A,
               uint32_t sw, JobState* ds, int num_sms);
// checks and places the seeds; writes the wave job and its gang's tables
void flat_seed(cudaStream_t st, const WaveJob& W, const FlatAxes& A, const FloodScratch& fs, const uint32_t* seeds,
               uint32_t ns, JobState* ds);
void flat_labels(cudaStream_t st, const WaveArrays& arr, const WaveJob& W, const FlatAxes& A, uint32_t sw,
                 const uint32_t* seeds, const JobState* ds, uint16_t* labels, int num_sms);

// ---- plain (reference-shaped) per-voxel kernels for one job ----
void plain_init_keys(cudaStream_t st, const JobDesc* dj, const JobDesc& hj);
void plain_seed(cudaStream_t st, const JobDesc* dj, JobState* ds, uint32_t* frontier,
                uint32_t* fcount);
void plain_wave(cudaStream_t st, const JobDesc* dj, JobState* ds, const JobDesc& hj,
                const uint32_t* cur, uint32_t ncur, uint32_t* next, uint32_t* ncount);
void plain_finalize(cudaStream_t st, const JobDesc* dj, const JobState* ds, const JobDesc& hj,
                    int pass2);
void plain_undo_mask(cudaStream_t st, const JobDesc* dj, const JobDesc& hj);
void plain_detect(cudaStream_t st, const JobDesc* dj, const JobDesc& hj);
void plain_erode(cudaStream_t st, const JobDesc* dj, const JobDesc& hj);
void plain_remove_isolated(cudaStream_t st, const JobDesc* dj, const JobDesc& hj);
void plain_perturb(cudaStream_t st, const JobDesc* dj, const JobDesc& hj);
void plain_naive(cudaStream_t st, const JobDesc* dj, const JobState* ds, const JobDesc& hj);
void plain_counts(cudaStream_t st, const JobDesc* dj, JobState* ds, const JobDesc& hj);
void plain_competition(cudaStream_t st, const JobDesc* dj, JobState* ds, const JobDesc& hj);
void plain_disjoint(cudaStream_t st, const JobDesc* dj, JobState* ds, const JobDesc& hj,
                    uint32_t* frontier, uint32_t* fcount);

}  // namespace vfk
