// pbf_kernels.h — host-visible declarations of the device kernels and launch
// helpers.  The float passes exist twice (exact / fast) and are reached
// through a PassTable of kernel pointers.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "pbf_params.h"

namespace pbf {

// Launches a kernel that begins with chain_begin(); early: it may be set up
// while the stream's previous kernel ends (programmatic dependent launch), so
// a chain of short kernels does not pay a full launch gap per link.
template <class... P, class... A>
cudaError_t launch_chain(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                         A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
// Slots up to which the step's kernels are launched early.  A frame of one
// graph-replayed substep of 4 iterations, with and without: 2,197 slots 58.5 and
// 62.7 us (exact mode 82 and 86), 27,000 exact 205 and 209, 68,921 148 and 153
// (exact 429 and 433), 220,000 667 and 674; at 2^20 slots it is within the noise
// (2215, 2208), and 16 batched scenes got 1 % slower.
constexpr uint32_t kEarlyMax = 1u << 18;

// The neighbour passes with several lanes a slot, for small scenes.
struct LaneSet {
  uint32_t lanes = 0, max_n = 0;  // up to max_n slots
  void (*lambda)(SimParams, int, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*, float4*,
                 SolverAux) = nullptr;
  void (*deltap)(SimParams, SolverAux, int, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*,
                 float4*, float4*) = nullptr;
  void (*density_velocity)(SimParams, SolverAux, const float4*, uint32_t, const uint32_t*, const uint32_t*, float4*,
                           float4*) = nullptr;
  void (*vorticity)(SimParams, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*, float4*,
                    float4*) = nullptr;
  void (*xsph)(SimParams, const float4*, const float4*, const float4*, const float4*, uint32_t, const uint32_t*,
               const uint32_t*, float4*, ExportArgs) = nullptr;
  void (*vorticity_split)(SimParams, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*,
                          float4*, float4*, float4*, float4*) = nullptr;
  void (*xsph_split)(SimParams, const float4*, const float4*, const float4*, const float4*, const float4*, uint32_t,
                     const uint32_t*, const uint32_t*, float4*, ExportArgs) = nullptr;
};

// The step's passes of one variant: single scene or batch (scene table),
// one tile per CTA or persistent (grid-stride).
struct PassSet {
  void (*predict)(SimParams, GridParams, SceneTab, const float4*, const float4*, const float4*, float4*, uint32_t*,
                  uint32_t*, uint32_t*, ClearArgs);
  void (*nbr_build)(SimParams, GridParams, SceneTab, const float4*, const uint32_t*, uint32_t, uint32_t*, uint32_t*,
                    uint32_t*, uint32_t*);
  void (*nbr_build2)(SimParams, GridParams, SceneTab, const float4*, const uint32_t*, uint32_t, uint32_t*,
                     uint32_t*, uint32_t*, uint32_t*);  // two slots per thread
  void (*nbr_build_warp)(SimParams, GridParams, SceneTab, const float4*, const uint32_t*, uint32_t, uint32_t*,
                         uint32_t*, uint32_t*, uint32_t*);  // warp-cooperative per cell
  void (*band)(SimParams, SceneTab, const float4*, BandArgs);
  void (*boundary_band)(SimParams, FieldParams, const float*, const float*, FieldBlocks, SceneTab, const float4*,
                        float4*, float*, const uint32_t*, const uint32_t*, uint32_t*, const int*);
  void (*lambda)(SimParams, int, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*, float4*,
                 SolverAux);
  void (*lambda_feat)(SimParams, int, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*,
                      float4*, SolverAux);
  void (*lambda_stats)(SimParams, int, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*,
                      float4*, SolverAux);     // null in batch sets
  void (*nbr_build_feat)(SimParams, GridParams, const float4*, const uint32_t*, uint32_t, uint32_t*, uint32_t*,
                         uint32_t*, uint32_t*, int, const float4*, SolverAux);  // null in batch sets
  void (*deltap)(SimParams, SolverAux, int, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*,
                 float4*, float4*);
  void (*density_velocity)(SimParams, SolverAux, const float4*, uint32_t, const uint32_t*, const uint32_t*, float4*,
                           float4*);
  void (*vorticity)(SimParams, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*, float4*,
                    float4*);
  void (*xsph)(SimParams, const float4*, const float4*, const float4*, const float4*, uint32_t, const uint32_t*,
               const uint32_t*, float4*, ExportArgs);
  LaneSet lanes[2];  // more lanes first; max_n = 0 where not built
  // fast mode: XSPH's neighbour sum split over the vorticity and XSPH passes (null in exact mode)
  void (*vorticity_split)(SimParams, const float4*, const float4*, uint32_t, const uint32_t*, const uint32_t*,
                          float4*, float4*, float4*, float4*);
  void (*xsph_split)(SimParams, const float4*, const float4*, const float4*, const float4*, const float4*, uint32_t,
                     const uint32_t*, const uint32_t*, float4*, ExportArgs);
};

// The cell-block passes of one membership variant (pbf_cellblock.cuh).
struct CbSet {
  void (*lambda)(SimParams, CbArgs, int, const float4*, const float4*, float4*, SolverAux);
  void (*lambda_feat)(SimParams, CbArgs, int, const float4*, const float4*, float4*, SolverAux);
  void (*lambda_stats)(SimParams, CbArgs, int, const float4*, const float4*, float4*, SolverAux);
  void (*deltap)(SimParams, CbArgs, SolverAux, int, const float4*, const float4*, float4*, float4*);
  void (*density_velocity)(SimParams, CbArgs, SolverAux, const float4*, float4*, float4*, uint32_t*);
  void (*vorticity)(SimParams, CbArgs, const float4*, const float4*, float4*, float4*);
  void (*xsph)(SimParams, CbArgs, const float4*, const float4*, const float4*, const float4*, float4*);
  void (*vorticity_split)(SimParams, CbArgs, const float4*, const float4*, float4*, float4*, float4*, float4*);
  void (*xsph_split)(SimParams, CbArgs, const float4*, const float4*, const float4*, const float4*, const float4*,
                     float4*);
  void (*fallback)(FallbackArgs, CbArgs);  // cooperative launch only
};

struct PassTable {
  PassSet set[2][2];  // [batch][persistent]
  void (*fallback)(FallbackArgs);  // cooperative launch only
  // cell-block passes: the search (masks; with the learned start's features)
  // and the passes per membership variant [mask, test]
  void (*cb_build)(SimParams, CbArgs, uint32_t*, uint16_t*, uint32_t*, int, const float4*, SolverAux);
  void (*cb_build_feat)(SimParams, CbArgs, uint32_t*, uint16_t*, uint32_t*, int, const float4*, SolverAux);
  CbSet cb[2];
};

namespace exact {
void fill_pass_table(PassTable* tbl);
}
namespace fast {
void fill_pass_table(PassTable* tbl);
}

// ---- integer pipeline (pbf_sort.cu) ---------------------------------------------
// Elements per tile of the single-pass scan.
constexpr size_t kScanTileElements = 2048;
// Scratch of the single-pass scan for up to `n` elements, in bytes:
// 256 bytes (tile counter) + one 8-byte status word per tile.
size_t scan_scratch_bytes(size_t n);
// Exclusive scan of n u32 (out may alias nothing in in).  `scratch` holds
// scan_scratch_bytes(n) bytes; err receives PBF_DEVERR_SCAN_TIMEOUT when a
// bounded look-back wait gives up.
cudaError_t launch_exclusive_scan(const uint32_t* in, uint32_t* out, size_t n, void* scratch, uint32_t* err,
                                  cudaStream_t st);
// The same with the scratch already cleared by the caller's own kernel.
cudaError_t launch_exclusive_scan_cleared(const uint32_t* in, uint32_t* out, size_t n, void* scratch, uint32_t* err,
                                          cudaStream_t st, const ScanExtra& X, bool early);
// Self-test of the scan's bounded look-back wait (a predecessor status that
// nothing writes): *err receives PBF_DEVERR_SCAN_TIMEOUT.
cudaError_t launch_scan_timeout_selftest(uint32_t* err, cudaStream_t st);

// The step's counting sort.  The caller has cleared cell_count, the scan's
// scratch and big_count (k_predict clears the last two).
struct SortBuffers {
  uint32_t* key;        // [n] cell key per input slot
  uint32_t* rank;       // [n] warp-aggregated (unordered) rank per input slot
  uint32_t* cell_count; // [cells + 1]
  uint32_t* count_next; // [cells + 1] cleared by the scan: the next substep's counts
  uint32_t* cell_start; // [cells + 1] exclusive scan of cell_count
  uint32_t* perm_raw;   // [n] scattered slots (unordered within a cell)
  uint32_t* id_raw;     // [n] particle id of perm_raw entries
  uint32_t* perm;       // [n] output: sorted slot -> input slot, stable by id
  uint32_t* tmp_a;      // [n] radix scratch for very full cells
  uint32_t* tmp_b;      // [n]
  uint32_t* big_list;   // [cells] cells sorted by the block radix path
  uint32_t* big_count;  // [1]
  void* scan_scratch;
  uint32_t* err;
};
// The particle state moved into the new order with the sort: positions,
// predicted positions and ids, f (optional): one scalar per particle (the
// learned start's previous multiplier sum); skey_out / xs0_out (optional, for
// the cell-block passes): the cell key of each sorted slot and a second copy
// of x*_0 that the solve leaves untouched.
struct GatherArgs {
  const float4* pos_in;
  const float4* xs_in;
  const uint32_t* key;
  const float* f_in;
  float4* pos_out;
  float4* xs_out;
  uint32_t* id_out;
  float* f_out;
  uint32_t* skey_out;
  float4* xs0_out;
};

// Stable LSD radix sort of points in particle-id order by cell key (the
// stand-alone search), n > 0: keys[n] (by id) receive the cell keys, skeys[n]
// the sorted keys and order[n] (and order2, optional) the ids in sorted order,
// stable by id.  tmp_k / tmp_v: two pairs of n-entry scratch arrays; scratch:
// radix_scratch_bytes(n) bytes.  after_keys (optional) is recorded after the
// keys.  cell_count (cells + 1 entries) receives the cell counts from the last
// pass and scan_scratch (for a scan of cells + 1) is cleared.
struct RadixPlan {
  int passes, width;
  size_t tiles;
};
RadixPlan radix_plan(uint32_t cells, size_t n);
size_t radix_scratch_bytes(size_t n);
cudaError_t launch_radix_sort_idorder(GridParams g, const float4* pos, uint32_t n, uint32_t* keys, uint32_t* skeys,
                                      uint32_t* order, uint32_t* order2, uint32_t* const tmp_k[2],
                                      uint32_t* const tmp_v[2], void* scratch, uint32_t* err, cudaStream_t st,
                                      cudaEvent_t after_keys, uint32_t* cell_count, void* scan_scratch);
// rank_out[order[q]] = q - cell_start[skeys[q]].
cudaError_t launch_rank_sorted(uint32_t n, const uint32_t* skeys, const uint32_t* order, const uint32_t* cell_start,
                               uint32_t* rank_out, cudaStream_t st);
// Scan of the counts, scatter, stable within-cell order with the state moved along.
cudaError_t launch_sort_by_cell(GridParams g, uint32_t n, const uint32_t* ids, SortBuffers& b, uint32_t id_bits,
                                const GatherArgs& G, cudaStream_t st);
cudaError_t launch_scatter_by_id(uint32_t n, const uint32_t* id, const float4* src, float4* dst, cudaStream_t st);
// dst[id[t]] = src[t].w (a scalar kept in the w lane of a packed float4 array)
cudaError_t launch_scatter_w_by_id(uint32_t n, const uint32_t* id, const float4* src, float* dst, cudaStream_t st);
cudaError_t launch_scatter_by_id_u32(uint32_t n, const uint32_t* id, const uint32_t* src, uint32_t* dst,
                                     cudaStream_t st);
// Neighbour lists of the stand-alone search (27 cells, |d|^2 <= h2): sorted[t]
// = (position, id) of order[t], the neighbour count by particle id (n + 1
// entries, the last 0), its exclusive scan offset and the 64-bit sum *total;
// then the lists of neighbour ids at offset[id], written only if *total <=
// capacity.  scan: scan_scratch_bytes(n + 1) bytes.
cudaError_t launch_ns_count(uint32_t n, const GridParams& g, float h2, const uint32_t* order, const float4* pos,
                            const uint32_t* cell_start, float4* sorted, uint32_t* count, uint32_t* offset,
                            unsigned long long* total, void* scan, uint32_t* err, cudaStream_t st);
cudaError_t launch_ns_list(uint32_t n, const GridParams& g, float h2, const float4* sorted, const uint32_t* cell_start,
                           const uint32_t* count, const uint32_t* offset, const unsigned long long* total,
                           uint32_t* list, uint32_t capacity, cudaStream_t st);

// Metrics (max / mean density error, kinetic energy, non-finite and penetration counts).
struct MetricsAccum {
  float max_compression;
  float max_abs_err;
  double sum_abs_err;
  double kinetic;
  uint32_t nonfinite;
  uint32_t penetrations;
};
cudaError_t launch_metrics(SimParams p, FieldParams f, const float* sdf, const float4* pos, const float4* vel,
                           const uint32_t* nbr_count, uint32_t n, float* accum_f, double* accum_d, uint32_t* accum_u,
                           cudaStream_t st);

// Learned start (pbf_learned.cu).
}  // namespace pbf
#include "../../include/pbf_gb300.h"
namespace pbf {
// lambda_hat per feature row into d_lambda, or, with d_xl, packed as
// d_xl[r] = (d_xs[r].xyz, lambda_hat); d_lam_sum (optional) starts the sum.
cudaError_t launch_mlp_infer(const float* d_params, const pbf_mlp& model, const float* d_feat, uint32_t rows,
                             float* d_lambda, float* d_lam_sum, cudaStream_t st, const float4* d_xs = nullptr,
                             float4* d_xl = nullptr);
// The same on the 5th-generation tensor cores (tcgen05.mma, TMEM
// accumulators; pbf_mlp_tc.cu); d_err receives PBF_DEVERR_MMA_TIMEOUT when a
// bounded completion wait gives up.
cudaError_t launch_mlp_infer_tc(const float* d_params, const pbf_mlp& model, const float* d_feat, uint32_t rows,
                                float* d_lambda, float* d_lam_sum, cudaStream_t st, const float4* d_xs,
                                float4* d_xl, uint32_t* d_err, LateBoundary lb = LateBoundary{});
// Forward + backward on tcgen05.mma (pbf_mlp_tc.cu): the gradient accumulates
// into d_grad (atomically), the summed squared error into d_loss; d_err
// receives PBF_DEVERR_MMA_TIMEOUT when a bounded completion wait gives up.
cudaError_t launch_mlp_grad_tc(const float* d_params, const pbf_mlp& model, const float* d_feat,
                               const float* d_target, uint32_t rows, float* d_grad, float* d_loss, uint32_t* d_err,
                               cudaStream_t st);
cudaError_t launch_mlp_grad(const float* d_params, const pbf_mlp& model, const float* d_feat, const float* d_target,
                            uint32_t rows, float* d_grad, float* d_loss, cudaStream_t st);
cudaError_t launch_fallback_decide(SolveStats* stats, float bound, int* flag, uint32_t* fallbacks, float* last_mean,
                                   cudaStream_t st);
// Lagged iteration control (counts[0] decisions, counts[1] substeps that iterated).
cudaError_t launch_lagged_decide(const float* last_mean, float threshold, int* flag, uint32_t* counts,
                                 cudaStream_t st);
// The adaptive iteration's test (counts[0] tests, counts[1] position updates run).
cudaError_t launch_iterate_decide(SolveStats* stats, float bound, int* flag, uint32_t* counts, float* last_mean,
                                  cudaStream_t st);
cudaError_t launch_stats_record(SolveStats* stats, float* rec, cudaStream_t st);
cudaError_t launch_trace_append(uint32_t n, const uint32_t* ids, const float4* feat, const float* lam_sum,
                                uint32_t stride, uint32_t salt, float* tf, float* tt, uint32_t* count, uint32_t cap,
                                cudaStream_t st);
// ---- scene seeding (pbf_seed.cu) -------------------------------------------------
// Writes the points of `items` (cube / sphere / mesh lattices, in order) to
// out[0 .. *total) as (x, y, z, 0), applies the host jitter's splitmix64
// draws when jitter > 0 and sets ids[i] = i.  *total gets the number of
// points the items make even on PBF_ECAPACITY (nothing beyond capacity is
// written).  Synchronises `st` before returning.
int seed_device(const pbf_seed_item* items, uint32_t count, double radius, float jitter, uint64_t seed, float4* out,
                uint32_t* ids, uint32_t capacity, uint32_t* total, cudaStream_t st);
// SPH.voxelizeMesh on the device with the kept points copied to *pts (when
// emit) and their number in *kept.
int voxelize_mesh_host(const float* vertices, uint32_t vertex_count, const uint32_t* indices, uint32_t triangle_count,
                       const double* world, double particle_radius, bool emit, std::vector<float>* pts,
                       uint32_t* kept);

}  // namespace pbf
