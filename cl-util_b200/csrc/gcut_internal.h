// Internal interfaces between the translation units of libgcut.so.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/gcut.h"
#include "gcut_common.cuh"

static_assert(gcut::K_COUNT == GC_NKERN, "kernel kinds");

namespace gcut {

enum ScanMode {
  GC_SCAN_MODE_SCAN = 0,     // exclusive scan of values
  GC_SCAN_MODE_COMPACT = 1,  // indices of non-zero values
  GC_SCAN_MODE_FLAG = 2,     // indices where op1(in, a1)
  GC_SCAN_MODE_LOGICAL = 3,  // indices where op1(in, a1) AND/OR op2(in2, a2)
};

int scan_chunks(int n);
// Records the message returned by gc_last_error() for the calling thread; returns code.
int set_last_error(int code, const char* msg);
int launch_scan(int mode, const int32_t* in, const int32_t* in2, int32_t* scan_out,
                int32_t* list_out, int32_t* total_out, int n, int op1,
                int32_t a1, int op2, int32_t a2, int logical, const ScanState& st,
                cudaStream_t s);
// One warp waits on a look-back predecessor that never publishes, until st.spin_limit
// polls run out (sets *st.err); needs st.max_chunks >= 2.
int launch_lookback_selftest(const ScanState& st, cudaStream_t s);
int launch_increment_logical(int32_t* tiles, const int32_t* tiles2, int n, int op1, int op2,
                             int32_t a1, int32_t a2, int logical, int32_t iteration,
                             cudaStream_t s);
int launch_fill(int32_t* p, int n, int32_t v, cudaStream_t s);
int launch_tiles_view(const int32_t* tiles, int tiles_w, int tiles_h, int tile_w, int tile_h,
                      int32_t iteration, int width, int height, uint32_t* out, cudaStream_t s);

// One image inside a tile pool.
struct ImageDesc {
  int W, H;      // pixel size
  int tw, th;    // tile grid
  int tile0;     // first tile id; tiles are row-major from there
};

// Per-image accumulators on the device.
struct ImageAcc {
  unsigned long long sumpos_t;   // sum max(t-link, 0)  (two's complement int64)
  unsigned long long sumpos_e;   // sum max(excess, 0) at the end of a solve
  int32_t bad_caps;              // negative capacities seen at upload
  int32_t pad;
};

// Solver kernels (gcut_solver.cu).
int launch_upload(const PoolView& P, const ImageDesc& im, int img, const int32_t* up,
                  const int32_t* down, const int32_t* left, const int32_t* right,
                  const int32_t* excess, int32_t* tl, ImageAcc* acc, cudaStream_t s);
// rebuilds the row masks of the selected tiles whose planes changed since they were written
int launch_masks(const PoolView& P, int grid, cudaStream_t s);

// n-link table of gc_upload_rgba: weight(d) = floor(50 * exp(-beta * d) + 0.5) for d = |dI|^2
// equals the number of entries t[k] >= d (t[k] = largest d with weight >= k + 1).
constexpr int GC_NLINK_LEVELS = 50;
// tab: the device table of launch_nlinks (exp weighting), or null for the reference's weighting
// floor(lambda / (0.1 sqrt(d) + 0.05) + 0.5) (gc_upload_rgba_lambda)
int launch_upload_rgba(const PoolView& P, const ImageDesc& im, int img, const uint32_t* rgba,
                       const int32_t* excess, const int32_t* tab, int lambda, int32_t* tl,
                       ImageAcc* acc, cudaStream_t s);
// The mean |dI|^2 of an image and the n-link table from it (tab: 50 thresholds and a float),
// one launch; state: two zeroed words, zero again afterwards.  Clears *acc for the upload.
int launch_nlinks(const uint32_t* rgba, int W, int H, unsigned long long* state, int32_t* tab,
                  ImageAcc* acc, int sms, cudaStream_t s);
// reads the worklist queue[ctl[CTL_PULSE] & 1], builds the other one; hlim: pixels below this
// height are active
int launch_discharge(const PoolView& P, int iters, int hlim, int grid, cudaStream_t s);
int launch_edge_relabel_build(const PoolView& P, int32_t* list, int32_t* count,
                              const ScanState& st, cudaStream_t s);
// first: 0 frontier round, 1 first round over the selected tiles, 2 over those of the images
// live at stamp `live`; distances beyond `cap` stay GC_HINF.
int launch_bfs_round(const PoolView& P, int first, int cap, int live, int grid, cudaStream_t s);
// mode: 0 frontier round; first rounds over the selected tiles: 1 all, 2 those of the images
// live at `stamp`, 3 those of the images that continue from a previous flow; abort_hit:
// frontier rounds skip images that reached a sink (they carry `stamp` in img_hit)
int launch_flood_round(const PoolView& P, int mode, int abort_hit, int stamp, ImageAcc* acc,
                       int grid, cudaStream_t s);
// retires the images whose flood reached no sink; all: every image that continues from a flow
int launch_flood_check(const PoolView& P, int all, int stamp, ImageAcc* acc, cudaStream_t s);
int launch_ctl_begin(const PoolView& P, int max_rounds, ImageAcc* acc, cudaStream_t s);
// active tiles of the selected images live at stamp `live`; fresh: freshly uploaded images
// take part by fresh_tile_active; grid: most CTAs, which loop over the selection's chunks
int launch_active_list(const PoolView& P, const ScanState& st, int32_t* list, int32_t* count,
                       int live, int fresh, int grid, cudaStream_t s);
// The whole solve as one cooperative launch of `grid` CTAs (at most occupancy_solve()).
struct SolveArgs : SolvePlan {
  ImageAcc* acc;
  int ranges, tiles;        // the selection's size (its ranges are in P.sel)
  int4 sel0;                // its first range
  int mode0;                // and its mode
  int clean;                // leave the counters and sums at zero (the results reach the host)
  int lmode;                // 0 no labels; image im's labels: 1 a byte per pixel, 2 packed
  uint8_t* labels;
  ImageDesc im;
};
int launch_solve(const PoolView& P, const SolveArgs& a, int grid, cudaStream_t s);
int launch_acc_reset(ImageAcc* acc, int n, cudaStream_t s);
int launch_ctl_cycle(const PoolView& P, cudaStream_t s);
// neighbour ids and image index of the tiles of image img (a session-pool slot)
int launch_image_tiles(const PoolView& P, const ImageDesc& im, int img, cudaStream_t s);
int launch_labels_out(const PoolView& P, const ImageDesc& im, uint8_t* out, cudaStream_t s);
int launch_labels_packed(const PoolView& P, const ImageDesc& im, uint8_t* out, cudaStream_t s);
int launch_state_out(const PoolView& P, const ImageDesc& im, const int32_t* plane,
                     int32_t* out, cudaStream_t s);
int launch_edit(const PoolView& P, const ImageDesc& im, int img, const int32_t* idx,
                const int32_t* val, int n, int32_t* tl, ImageAcc* acc, cudaStream_t s);
// Whether an edit of npts points carries them in its launch (pts_dev is then not read).
bool edit_points_inline(int npts);
// pts_dev / pts_host: the same (x, y) pairs on the device and on the host (for the bounds).
int launch_stroke(const PoolView& P, const ImageDesc& im, int img, const int32_t* pts_dev,
                  const int32_t* pts_host, int npts, int radius, int32_t value, int32_t* tl,
                  ImageAcc* acc, cudaStream_t s);
// The reference brush's pixel set (gc_edit_brush); radius <= 0 counts as 1; GC_ERR_INVALID
// above 1024.
int launch_brush(const PoolView& P, const ImageDesc& im, int img, const int32_t* pts_dev,
                 const int32_t* pts_host, int npts, int radius, int32_t value, int32_t* tl,
                 ImageAcc* acc, cudaStream_t s);
// Loads every kernel of the library on the current device (once per device; called by the
// first handle creation and the first stand-alone primitive on a device).
void preload_kernels();
void preload_scan_kernels();
// gc_view_colorize; ramp9: range lo, hi, hue lo, hi, saturation lo, hi, value lo, hi, opacity
int launch_view_colorize(const int32_t* values, int values_w, int values_h, int cell_w,
                         int cell_h, int width, int height, const float* ramp9,
                         const uint32_t* base, uint32_t* out, cudaStream_t s);
int occupancy_discharge(int device);
int occupancy_warps(int device);
int occupancy_solve(int device);

}  // namespace gcut
