// Batched work plan shared by the host planner and the persistent kernels.
//
// One contiguous buffer, identical on host and device:
//   PlanHeader | MatDesc[n_mat] | View[total views] | int cta_off[n_ctas+1]
//   | int order[n_tiles] | int2 tiles[n_tiles] (material, first texel)
//   | int mat_tile_off[n_mat+1] | float coord tables (per material: x[W], then y[H])
//   | int4 seq[n_tiles] (order[k]'s tile, material and first texel, in CTA order; a tile
//     of variants 2 and 3 ends where its material's next one starts, the others have tile_texels texels)
//   | variants 2 and 3: int run_tile[n_runs] | int cta_run[n_ctas+1] | int mat_run[n_mat+1]
// Tiles of one material are contiguous in tile-index order (mat_tile_off), so each material's loss is a
// fixed-order sum over a tile range, or in variants 2 and 3 over its runs: a run is a CTA's
// consecutive tiles of one material, named by its first tile. cta_off[c]..cta_off[c+1] indexes
// `order`, the tile ids of CTA c; `order` is the identity.
#pragma once

#include "svbrdf_math.cuh"

namespace svb {

struct PlanHeader {
  int magic;
  int n_mat;
  int n_tiles;
  int n_ctas;
  int threads;      // consumer threads per CTA
  int tile_texels;
  int off_mats;     // byte offsets from the plan base
  int off_views;
  int off_cta;
  int off_order;
  int off_tiles;
  int off_mat_tiles;
  int off_coords;
  int variant;      // 0: direct loads, 1: bulk-copy (TMA) pipeline, 2: the pipeline on texel pairs
  int ring_slots;   // variants 1 and 2: shared-memory ring depth
  int general;      // 1 when some material has a view whose light is not at the camera
  int off_seq;      // int4 (tile, material, first texel, 0) per entry of `order`
  int light;        // 1 when some material's light power is learnable (MatDesc::lstate)
  int off_runs;     // variants 2 and 3: first tile of each run (a CTA's tiles of one material) ...
  int off_cta_run;  // ... the first run of each CTA [n_ctas + 1] ...
  int off_mat_run;  // ... and of each material [n_mat + 1]
  long long total_bytes;
  double total_cost;
};

struct __align__(16) MatDesc {
  float* tex;
  float* m1;
  float* m2;
  const float* tgt;
  float* lpow;
  float* lstate;      // light power Adam state [6] (exp_avg, exp_avg_sq), or null: light fixed
  int H, W, V, view_off;
  float size, scale;  // scale = 2 / (3 V H W), the loss-gradient normaliser
  float inv_w;        // 1 / W for the row/column split of a texel index
  int coord_off;      // float index of this material's x table (y follows at +W)
  int all_coloc;      // 1 when every view has the light at the camera
  int pad;
  double inv_n;       // 1 / (3 V H W)
};

// Another value with every change of the layout: a plan that another build made is refused, where its
// offsets would be read as other ones.
constexpr int kPlanMagic = 0x53564233;  // "SVB3"

// Adam hyper-parameters of a batched launch; the step itself lives on the device so
// one captured graph can be replayed indefinitely.
struct AdamHyper {
  float lr, beta1, beta2, eps;
};

// Workspace of a batched launch: [0] completion counter, [1] error word, [2] number of the last
// iteration that a cooperative launch has finished (it only ever counts up), then from byte
// 256 the per-(tile, warp) partial losses, then (plans with a learnable light) the
// per-(tile, warp) partial light-power gradients, 3 floats each, then one total per tile and quantity.
// Variants 2 and 3 use the slots of a run's first tile for the whole run.
constexpr int kWsCounter = 0;
constexpr int kWsError = 1;
constexpr int kWsIteration = 2;
constexpr size_t kWsLossOffset = 256;

// Error codes written to the workspace error word by a kernel that gave up waiting.
enum DeviceError : int {
  kDevOk = 0,
  kDevTimeoutFull = 1,   // a consumer waited too long for a bulk copy
  kDevTimeoutEmpty = 2,  // the producer waited too long for consumers to free a slot
  kDevTimeoutDrain = 3,  // in-flight copies did not land while shutting down
  kDevTimeoutGrid = 4,   // a CTA waited too long for the others to finish an iteration
};

}  // namespace svb
