// Tiled push-relabel kernels for sm_100a.
//
// Reference path: GraphCut.cut (GraphCut.pyx:348-418) driving graphcut.cl.  The reference
// runs one OpenCL kernel per push direction (push_down/up/right/left, graphcut.cl:158-536)
// with an 8-pixel wave per work-item, merges tile overspill with add_border (:114-156),
// relabels the whole image with a Jacobi pass (:538-577) and computes the global relabel
// with init_bfs/bfs_intratile/bfs_intertile (:582-1016) over compacted tile lists.  Here:
//
//  * k_solve       a whole solve in one cooperative launch: the steps below with grid barriers
//                  between them, the loops decided on the device.  The kernels named here run
//                  the same steps as launches of their own, for the manual stepping calls and
//                  the host-driven loop.
//  * k_discharge   one CTA of 256 threads per listed tile (persistent over the device-side
//                  list): the tile's excess, height and four residual planes arrive in shared
//                  memory by bulk copy (the next tile's copy overlaps this tile's work), with
//                  the halo heights, and the CTA runs `iters` rounds of {push along every
//                  admissible edge (all 4 directions), Jacobi relabel}.  Flow leaving the tile
//                  is added to the neighbour's excess and reverse residual with atomics (no
//                  border buffer, no add_border launch); tile-edge pixels rise at most 2 per
//                  launch, so the labelling stays valid whether a neighbouring CTA saw a
//                  pixel's start or final height.  Each finished
//                  tile's bookkeeping (next list, dirty flags) is settled in batches.
//  * k_edge_relabel_build   relabels the active tile-edge pixels (Jacobi) and rebuilds the
//                  active-tile list with the single-pass decoupled look-back compaction in
//                  the same launch (IncrementalTileList.build + StreamCompact + PrefixSum);
//                  the manual relabel step (GraphCut.relabel) only.
//  * k_bfs_round   global relabel, exact up to a distance cap: per tile, one warp runs a
//                  bit-parallel multi-source BFS (32-bit row masks of residual edges, lane =
//                  row) seeded by sink pixels and by the halo distances, and queues neighbours
//                  whose edge distances could drop for the next round.
//  * k_flood_round canonical cut: the same tile rounds flood the set reachable from excess
//                  pixels over residual edges (the minimal source set).
#include <cstdio>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "gcut_common.cuh"
#include "gcut_internal.h"

namespace gcut {

constexpr int DIS_THREADS = 256;
constexpr int DIS_LOG = 32;       // tiles per bookkeeping flush in k_discharge (<= DIS_THREADS / 5)
constexpr int WARPS_PER_CTA = 4;   // warp-per-tile kernels (BFS, flood, mask rebuild)

__device__ __forceinline__ int imin(int a, int b) { return a < b ? a : b; }

// ------------------------------------------------------------------------------------
// Upload: row-major planes -> tile planes; boundary capacities zeroed; padding pixels are
// isolated (all zero).  Heights start at 0 for sink pixels and 1 otherwise (a valid
// labelling).  Replaces init_gc + load_tiles (graphcut.cl:63-112, 1033-1132).
// ------------------------------------------------------------------------------------
// Row masks of four rows from a warp whose thread (g, q) holds pixels 4q..4q+3 of row g: thread
// (g, k) returns mask k of row g (0-3: residual edge up / down / left / right, 4: sink, 5:
// positive excess; 6, 7: nothing).  Each thread packs its four pixels of every mask as nibble k
// of a word, and the eight threads of a row transpose their 8 x 8 nibbles: three shuffles.  (A
// ballot per mask and pixel, its bits then spread, took 300 instructions a thread for 70, and
// kept the ALU pipe of the uploads 68 % busy: 2048x2048 planes 35.5 us, now 32.2.)
__device__ __forceinline__ uint32_t row_masks(const int (&e)[4], const int (&cu)[4], const int (&cd)[4],
                                              const int (&cl)[4], const int (&cr)[4], int lane) {
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w |= cu[j] > 0 ? 1u << j : 0u;
    w |= cd[j] > 0 ? 0x10u << j : 0u;
    w |= cl[j] > 0 ? 0x100u << j : 0u;
    w |= cr[j] > 0 ? 0x1000u << j : 0u;
    w |= e[j] < 0 ? 0x10000u << j : 0u;
    w |= e[j] > 0 ? 0x100000u << j : 0u;
  }
  const unsigned F = 0xffffffffu;
  // halves, bytes, nibbles with the thread 4, 2, 1 further
  w = __byte_perm(w, __shfl_xor_sync(F, w, 4), lane & 4 ? 0x3276 : 0x5410);
  w = __byte_perm(w, __shfl_xor_sync(F, w, 2), lane & 2 ? 0x3715 : 0x6240);
  const uint32_t o = __shfl_xor_sync(F, w, 1);
  const uint32_t keep = lane & 1 ? 0xf0f0f0f0u : 0x0f0f0f0fu;
  return (w & keep) | (__funnelshift_l(o, o, lane & 1 ? 28 : 4) & ~keep);
}

// Row masks of tile t (residual edge up / down / left / right, sink, positive excess) from
// the values the block's 256 threads hold: thread (r, q) holds pixels (r, 4q .. 4q+3).  The
// BFS and the flood read these instead of the planes.  Every thread of the block calls it.
__device__ __forceinline__ void write_tile_masks(const PoolView& P, int t, const int (&e)[4],
                                                 const int (&cu)[4], const int (&cd)[4],
                                                 const int (&cl)[4], const int (&cr)[4]) {
  const int lane = threadIdx.x & 31, k = lane & 7;
  const uint32_t m = row_masks(e, cu, cd, cl, cr, lane);
  uint32_t* const dst = k < 4 ? P.mcan + (long long)t * 128 + 32 * k : (k == 4 ? P.msink : P.mexc) + (long long)t * 32;
  if (k < 6) dst[threadIdx.x >> 3] = m;
}

// Tile t's planes changed after its masks were written: the first flood round that covers
// it (or k_masks) rebuilds them.  A plain store: nothing reads the flag until a later kernel.
__device__ __forceinline__ void mark_dirty(const PoolView& P, int t) { P.mdirty[t] = 1; }

// Row masks of one tile row, as write_tile_masks writes them.
struct RowMasks { uint32_t up, down, left, right, sink, exc; };

// Rebuilds tile t's row masks and its sum of max(excess, 0) from its planes with one warp:
// lane c reads column c of REB_ROWS rows at a time (one 128-byte line per row and plane), and a
// ballot over the lanes is the row's mask.  Writes the masks and the sum, clears the dirty
// flag, and returns row `lane`'s masks to each lane and the tile's sum to every lane.
constexpr int REB_ROWS = 8;
__device__ __forceinline__ RowMasks warp_rebuild_masks(const PoolView& P, int t, int lane,
                                                       long long* tile_pos) {
  const unsigned F = 0xffffffffu;
  const long long base = (long long)t * GC_TILE_PX + lane;
  RowMasks out{0u, 0u, 0u, 0u, 0u, 0u};
  long long pos = 0;
#pragma unroll 1
  for (int r0 = 0; r0 < GC_TILE; r0 += REB_ROWS) {
    int v[REB_ROWS][5];
#pragma unroll
    for (int k = 0; k < REB_ROWS; ++k) {
      const long long o = base + (r0 + k) * GC_TILE;
      v[k][0] = P.exc[o];
      v[k][1] = P.cap[DUP][o];
      v[k][2] = P.cap[DDOWN][o];
      v[k][3] = P.cap[DLEFT][o];
      v[k][4] = P.cap[DRIGHT][o];
    }
#pragma unroll
    for (int k = 0; k < REB_ROWS; ++k) {
      const uint32_t mu = __ballot_sync(F, v[k][1] > 0), md = __ballot_sync(F, v[k][2] > 0);
      const uint32_t ml = __ballot_sync(F, v[k][3] > 0), mr = __ballot_sync(F, v[k][4] > 0);
      const uint32_t ms = __ballot_sync(F, v[k][0] < 0), me = __ballot_sync(F, v[k][0] > 0);
      if (lane == r0 + k) {
        out.up = mu; out.down = md; out.left = ml; out.right = mr;
        out.sink = ms; out.exc = me;
      }
      pos += v[k][0] > 0 ? v[k][0] : 0;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) pos += __shfl_xor_sync(F, pos, o);
  uint32_t* mc = P.mcan + (long long)t * 128;
  mc[lane] = out.up;
  mc[32 + lane] = out.down;
  mc[64 + lane] = out.left;
  mc[96 + lane] = out.right;
  P.msink[(long long)t * 32 + lane] = out.sink;
  P.mexc[(long long)t * 32 + lane] = out.exc;
  if (lane == 0) {
    P.tpos[t] = pos;
    P.mdirty[t] = 0;
  }
  *tile_pos = pos;
  return out;
}

// The state of one uploaded tile, from the values the block's threads hold (thread (r, q) holds
// pixels (r, 4q .. 4q+3)): planes, trivial labelling, t-links, row masks, flags, and the
// image's sums.  Every thread of the block calls it.
__device__ __forceinline__ void store_uploaded_tile(const PoolView& P, int t, int img, int r, int c0,
                                                    const int (&e)[4], const int (&cu)[4],
                                                    const int (&cd)[4], const int (&cl)[4],
                                                    const int (&cr)[4], int32_t* __restrict__ tl,
                                                    ImageAcc* acc) {
  int h[4], bad = 0;
  unsigned lo = 0, hi = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    bad |= (cu[j] | cd[j] | cl[j] | cr[j]) < 0;
    h[j] = e[j] < 0 ? 0 : 1;
    const unsigned p = e[j] > 0 ? e[j] : 0;
    lo += p & 0xffffu;   // halves that fit 32 bits over a warp's 128 pixels
    hi += p >> 16;
  }
  const bool p4 = e[0] > 0 || e[1] > 0 || e[2] > 0 || e[3] > 0;
  const bool s4 = e[0] < 0 || e[1] < 0 || e[2] < 0 || e[3] < 0;
  unsigned tf = (p4 ? TF_POS | (r == 0 ? TF_POS_UP : 0) | (r == 31 ? TF_POS_DOWN : 0) : 0) |
                (s4 ? TF_SINK | (r == 0 ? TF_SINK_UP : 0) | (r == 31 ? TF_SINK_DOWN : 0) : 0) |
                (c0 == 0 ? (e[0] > 0 ? TF_POS_LEFT : 0) | (e[0] < 0 ? TF_SINK_LEFT : 0) : 0) |
                (c0 == 28 ? (e[3] > 0 ? TF_POS_RIGHT : 0) | (e[3] < 0 ? TF_SINK_RIGHT : 0) : 0) |
                (bad ? TF_BAD : 0);
  const long long off = (long long)t * GC_TILE_PX + r * GC_TILE + c0;
  *(int4*)(P.exc + off) = make_int4(e[0], e[1], e[2], e[3]);
  *(int4*)(tl + off) = make_int4(e[0], e[1], e[2], e[3]);
  *(int4*)(P.hgt + off) = make_int4(h[0], h[1], h[2], h[3]);
  *(int4*)(P.cap[DUP] + off) = make_int4(cu[0], cu[1], cu[2], cu[3]);
  *(int4*)(P.cap[DDOWN] + off) = make_int4(cd[0], cd[1], cd[2], cd[3]);
  *(int4*)(P.cap[DLEFT] + off) = make_int4(cl[0], cl[1], cl[2], cl[3]);
  *(int4*)(P.cap[DRIGHT] + off) = make_int4(cr[0], cr[1], cr[2], cr[3]);
  write_tile_masks(P, t, e, cu, cd, cl, cr);
  if (threadIdx.x < 32) P.mreach[(long long)t * 32 + threadIdx.x] = 0u;   // no flood yet
  __shared__ long long wpos[DIS_THREADS / 32];
  __shared__ unsigned wflag[DIS_THREADS / 32];
  lo = __reduce_add_sync(0xffffffffu, lo);
  hi = __reduce_add_sync(0xffffffffu, hi);
  const long long pos = (long long)hi * 65536 + lo;
  tf = __reduce_or_sync(0xffffffffu, tf);
  if ((threadIdx.x & 31) == 0) {
    wpos[threadIdx.x >> 5] = pos;
    wflag[threadIdx.x >> 5] = tf;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long tp = 0;
    tf = 0;
    for (int k = 0; k < DIS_THREADS / 32; ++k) {
      tp += wpos[k];
      tf |= wflag[k];
    }
    P.tpos[t] = tp;
    // one add per tile: the adds of all of an image's tiles go to one address
    if (tp) atomicAdd(&acc[img].sumpos_t, (unsigned long long)tp);
    if (tf & TF_BAD) atomicAdd(&acc[img].bad_caps, 1);
    P.tflag[t] = (int32_t)tf;
    P.hstate[t] = 0;
    P.tact[t] = (tf & TF_POS) != 0;
    P.touched[t] = 0;
    P.act_int[t] = 0;
    P.mark[0][t] = 0;
    P.mark[1][t] = 0;
    P.inq[0][t] = 0;
    P.inq[1][t] = 0;
    P.img_of[t] = img;
    P.mdirty[t] = 0;     // the masks above are current
  }
}

// gc_upload: row-major capacity planes.
struct PlaneSource {
  const int32_t *up, *down, *left, *right, *excess;
  bool vec;   // all planes 16-byte aligned and the width a multiple of 4: int4 row loads
};

__global__ void __launch_bounds__(DIS_THREADS)
k_upload(PoolView P, ImageDesc im, int img, PlaneSource src, int32_t* __restrict__ tl, ImageAcc* acc) {
  trace_mark(P, TR_UPLOAD);
  const int bt = blockIdx.x;
  const int tx = bt % im.tw, ty = bt / im.tw;
  const int r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;
  const int y = ty * GC_TILE + r, x0 = tx * GC_TILE + c0;
  int e[4], cu[4], cd[4], cl[4], cr[4];
  const bool top = y == 0, bottom = y == im.H - 1;
  if (src.vec && y < im.H && x0 + 3 < im.W) {
    const long long i = (long long)y * im.W + x0;
    const int4 a = *reinterpret_cast<const int4*>(src.excess + i);
    const int4 b = *reinterpret_cast<const int4*>(src.up + i);
    const int4 c = *reinterpret_cast<const int4*>(src.down + i);
    const int4 d = *reinterpret_cast<const int4*>(src.left + i);
    const int4 f = *reinterpret_cast<const int4*>(src.right + i);
    e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w;
    cu[0] = top ? 0 : b.x; cu[1] = top ? 0 : b.y; cu[2] = top ? 0 : b.z; cu[3] = top ? 0 : b.w;
    cd[0] = bottom ? 0 : c.x; cd[1] = bottom ? 0 : c.y; cd[2] = bottom ? 0 : c.z; cd[3] = bottom ? 0 : c.w;
    cl[0] = x0 == 0 ? 0 : d.x; cl[1] = d.y; cl[2] = d.z; cl[3] = d.w;
    cr[0] = f.x; cr[1] = f.y; cr[2] = f.z; cr[3] = x0 + 3 == im.W - 1 ? 0 : f.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int x = x0 + j;
      e[j] = cu[j] = cd[j] = cl[j] = cr[j] = 0;
      if (x < im.W && y < im.H) {
        const long long i = (long long)y * im.W + x;
        e[j] = src.excess[i];
        cu[j] = top ? 0 : src.up[i];
        cd[j] = bottom ? 0 : src.down[i];
        cl[j] = x > 0 ? src.left[i] : 0;
        cr[j] = x < im.W - 1 ? src.right[i] : 0;
      }
    }
  }
  store_uploaded_tile(P, im.tile0 + bt, img, r, c0, e, cu, cd, cl, cr, tl, acc);
}

// |a - b|^2 of two colours whose alpha byte is 0: byte differences and their dot product, two
// instructions.
constexpr uint32_t RGB_MASK = 0x00ffffffu;
__device__ __forceinline__ int rgb_dist2(uint32_t a, uint32_t b) {
  const unsigned d = __vabsdiffu4(a, b);
  return (int)__dp4a(d, d, 0u);
}

// Weight of the reference's n-link rule, rounded to an integer: floor(x + 0.5) for
// x = lambda / (0.1 sqrt(d) + 0.05) = 20 lambda / (2 sqrt(d) + 1) (graphcut.cl:1018-1031,
// LAMBDA and EPSILON from GraphCut.pyx:25-26,92-93), exactly.  For k >= 1,
// floor(x + 0.5) >= k  <=>  b = 40 lambda - 2k + 1 >= 0  and  4 (2k - 1)^2 d <= b^2,
// so the weight is the largest k satisfying that integer test (monotone in k).  A float32
// estimate of k (its error is below 0.01 of a level at lambda <= 1000) is settled by the test
// itself; with lambda <= 1000 and d <= 3 * 255^2 every product fits in 64 bits.
__device__ __forceinline__ bool ref_weight_at_least(int k, int d, int a40) {
  if (k < 1) return true;
  const int b = a40 - 2 * k + 1, a = 2 * k - 1;
  return b >= 0 && 4LL * ((long long)a * a) * d <= (long long)b * b;
}
__device__ __forceinline__ int ref_weight(int d, int lambda) {
  const int a40 = 40 * lambda;
  const float sd = sqrtf((float)d);
  int k = (int)(((float)a40 + 1.0f + 2.0f * sd) / (4.0f * sd + 2.0f));
  while (k > 0 && !ref_weight_at_least(k, d, a40)) --k;
  while (ref_weight_at_least(k + 1, d, a40)) ++k;
  return k;
}

// n-link weights from |dI|^2.  Exp weighting: the number of table entries >= d (the entries
// t[0..50) do not increase).  The formula itself in float32 gives the level to within one: its
// error is below 1e-4 of a level, so the level is off only next to a boundary, and the entries
// on both sides of it, one 64-bit read, settle it.  (A binary search chains six reads.)
struct ExpWeight {
  float scale;   // -beta * log2(e)
  __device__ __forceinline__ int operator()(const int2* s_tab, int d) const {
    const int k = (int)(50.0f * exp2f(scale * (float)d) + 0.5f);   // 0 .. 50
    const int2 t = s_tab[k];                                       // t[k - 1], t[k]
    return k + (t.y >= d ? 1 : 0) - (t.x < d ? 1 : 0);
  }
};
struct RefWeight {
  int lambda;
  __device__ __forceinline__ int operator()(const int2*, int d) const { return ref_weight(d, lambda); }
};

// The upload from an RGBA image: the weights of an n-link are the same both ways, so a thread
// computes those to the right of and below its four pixels and takes the other two directions
// from its neighbours (a lane of the same warp, shared memory for the row above); the tile's
// first row and column compute theirs from the pixels across the side.  5 weights a thread
// (9 in the tile's first warp) where one per pixel and direction takes 16.  A distance is a byte
// difference and a byte dot product (two instructions, not eleven).
//
// Bound by the planes it writes, 28 of 36 bytes a pixel (92 us at 4096x4096 and the copy rate):
// 119 us there (166 with the distances a channel at a time, two dependent table reads a weight
// and a ballot per mask and pixel), 1920x1080 16.5 us (23.6).  Eight CTAs an SM in place of five change nothing.
struct RgbaSource {
  const uint32_t* rgba;
  const int32_t* excess;
  const int32_t* tab;   // exp weighting: 50 thresholds, then the float scale; null: reference rule
  int lambda;           // reference weighting
  bool vec;             // both 16-byte aligned and the width a multiple of 4: int4 row loads
};

template <class Weight>
__global__ void __launch_bounds__(DIS_THREADS)
k_upload_rgba(PoolView P, ImageDesc im, int img, RgbaSource src, Weight weight,
              int32_t* __restrict__ tl, ImageAcc* acc) {
  trace_mark(P, TR_UPLOAD);
  __shared__ int2 s_tab[GC_NLINK_LEVELS + 1];   // the thresholds on both sides of a level
  __shared__ int4 s_down[GC_TILE][8];
  const int tid = threadIdx.x, q = tid & 7;
  if constexpr (std::is_same_v<Weight, ExpWeight>) {
    if (tid <= GC_NLINK_LEVELS)
      s_tab[tid] = make_int2(tid > 0 ? src.tab[tid - 1] : 0x7fffffff, tid < GC_NLINK_LEVELS ? src.tab[tid] : -1);
    weight.scale = __int_as_float(src.tab[GC_NLINK_LEVELS]);
    __syncthreads();
  }
  const int bt = blockIdx.x;
  const int tx = bt % im.tw, ty = bt / im.tw;
  const int r = tid >> 3, c0 = q * 4;
  const int y = ty * GC_TILE + r, x0 = tx * GC_TILE + c0;
  const bool row_in = y < im.H, below_in = y + 1 < im.H;
  const long long i = (long long)y * im.W + x0;
  uint32_t px[4] = {0u, 0u, 0u, 0u}, below[4] = {0u, 0u, 0u, 0u};
  int e[4] = {0, 0, 0, 0};
  if (src.vec && x0 + 3 < im.W) {
    if (row_in) {
      const uint4 a = *reinterpret_cast<const uint4*>(src.rgba + i);
      const int4 b = *reinterpret_cast<const int4*>(src.excess + i);
      px[0] = a.x; px[1] = a.y; px[2] = a.z; px[3] = a.w;
      e[0] = b.x; e[1] = b.y; e[2] = b.z; e[3] = b.w;
    }
    if (below_in) {
      const uint4 a = *reinterpret_cast<const uint4*>(src.rgba + i + im.W);
      below[0] = a.x; below[1] = a.y; below[2] = a.z; below[3] = a.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (x0 + j >= im.W) continue;
      if (row_in) {
        px[j] = src.rgba[i + j];
        e[j] = src.excess[i + j];
      }
      if (below_in) below[j] = src.rgba[i + im.W + j];
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    px[j] &= RGB_MASK;
    below[j] &= RGB_MASK;
  }
  // the pixel to the right of the four, and (first column) the one to the left
  const unsigned F = 0xffffffffu;
  uint32_t next = __shfl_down_sync(F, px[0], 1);
  if (q == 7 && row_in && x0 + 4 < im.W) next = src.rgba[i + 4] & RGB_MASK;
  uint32_t side = 0;   // first column: the pixel to the left
  const bool has_left = q == 0 && row_in && x0 > 0 && x0 < im.W;
  if (has_left) side = src.rgba[i - 1] & RGB_MASK;
  int cu[4], cd[4], cl[4], cr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t nx = j < 3 ? px[j < 3 ? j + 1 : 3] : next;
    cr[j] = row_in && x0 + j + 1 < im.W ? weight(s_tab, rgb_dist2(px[j], nx)) : 0;
    cd[j] = below_in && x0 + j < im.W ? weight(s_tab, rgb_dist2(px[j], below[j])) : 0;
  }
  cl[0] = __shfl_up_sync(F, cr[3], 1);
  if (q == 0) cl[0] = has_left ? weight(s_tab, rgb_dist2(px[0], side)) : 0;
  cl[1] = cr[0]; cl[2] = cr[1]; cl[3] = cr[2];
  s_down[r][q] = make_int4(cd[0], cd[1], cd[2], cd[3]);
  __syncthreads();
  if (r > 0) {
    const int4 a = s_down[r - 1][q];
    cu[0] = a.x; cu[1] = a.y; cu[2] = a.z; cu[3] = a.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      cu[j] = y > 0 && row_in && x0 + j < im.W
                  ? weight(s_tab, rgb_dist2(px[j], src.rgba[i - im.W + j] & RGB_MASK)) : 0;
  }
  store_uploaded_tile(P, im.tile0 + bt, img, r, c0, e, cu, cd, cl, cr, tl, acc);
}

// The mean |dI|^2 over all 4-neighbour pairs and the exp weighting's table, in one launch.
//
// A thread walks down 8 rows of a strip of 4 pixels, or 4 rows of one column where the rows are
// not 16-byte aligned (more rows take registers that loads in flight need), with the row above in registers and the pixel to the left from the
// lane beside it, so every pixel is read once (and a strip's upper row twice), all rows' loads
// in flight.  The CTAs are one wave that loops over the strips: at 4096x4096 the tails of eight
// waves (64-bit reduction, ticket) were a third of the time.  Sums are exact: 32 bits a thread
// and strip (at most 2 * PX * ROWS * 3 * 255^2), 64 above.  The last CTA turns the total into
// the table and clears the total and the ticket for the next call.
// Bound by memory at 4096x4096 (64 MiB: 10.6 us at the copy rate, 25 us here, 37 us with one
// column of 16 rows a thread and a CTA a strip); at 1920x1080 6.6 us (8.5), launch and tail.
//
// The table: weight(d) = floor(50 exp(-beta d) + 0.5) with beta = 1 / (2 mean |dI|^2) (0 when
// the mean is 0) does not increase with d, so it is stored as t[k - 1] = the largest d in
// [0, 3 * 255^2] with weight >= k.  Thread k - 1 locates t[k - 1] from the real root of
// 50 exp(-beta d) + 0.5 = k and settles it by evaluating the formula itself at the integers
// around it, in double, so the table reproduces a float64 evaluation of the formula pixel by
// pixel.  t[50] holds -beta * log2(e) as a float (ExpWeight's estimate).
constexpr int DSUM_THREADS = 256;
template <int PX> constexpr int DSUM_ROWS = PX == 4 ? 8 : 4;

__device__ __forceinline__ void nlink_table(unsigned long long sum, long long npairs, int k,
                                            int32_t* tab) {
  const long kMax = 3L * 255 * 255;
  const double mean = (double)sum / (double)(npairs > 1 ? npairs : 1);
  const double beta = mean > 0 ? 1.0 / (2.0 * mean) : 0.0;
  if (k == 1) tab[GC_NLINK_LEVELS] = __float_as_int((float)(-beta * 1.4426950408889634));
  if (beta <= 0) { tab[k - 1] = (int32_t)kMax; return; }
  auto w = [&](long d) { return (int)floor(50.0 * exp(-beta * (double)d) + 0.5); };
  const double root = log(50.0 / (k - 0.5)) / beta;   // weight(d) >= k  <=>  d <= root
  long d = root >= (double)kMax ? kMax : (root < 0 ? 0 : (long)floor(root));
  while (d < kMax && w(d + 1) >= k) ++d;
  while (d >= 0 && w(d) < k) --d;
  tab[k - 1] = (int32_t)d;
}

// state: [0] the running sum, [1] the ticket (both zero between calls)
template <int PX>
__global__ void __launch_bounds__(DSUM_THREADS)
k_nlinks(const uint32_t* __restrict__ rgba, int W, int H, long long npairs,
         unsigned long long* state, int32_t* __restrict__ tab, ImageAcc* acc) {
  constexpr int ROWS = DSUM_ROWS<PX>;
  __shared__ unsigned long long part[DSUM_THREADS / 32];
  __shared__ unsigned long long s_total;
  __shared__ int s_last;
  const int lane = threadIdx.x & 31;
  const int cols = (W / PX + DSUM_THREADS - 1) / DSUM_THREADS, rows = (H + ROWS - 1) / ROWS;
  unsigned long long acc64 = 0;
  for (long long b = blockIdx.x; b < (long long)cols * rows; b += gridDim.x) {
    const long long x = ((b % cols) * DSUM_THREADS + threadIdx.x) * PX;
    const int y0 = (int)(b / cols) * ROWS;
    const bool in = x < W;          // with PX == 4 the width is a multiple of 4
    unsigned sum = 0;
    uint32_t c[ROWS + 1][PX], l[ROWS];
#pragma unroll
    for (int k = 0; k <= ROWS; ++k) {   // c[0]: the row above the strip
      const int y = y0 + k - 1;
      const bool on = in && y >= 0 && y < H;
      const uint32_t* const p = rgba + (long long)y * W + x;
      if constexpr (PX == 4) {
        const uint4 v = on ? *reinterpret_cast<const uint4*>(p) : make_uint4(0u, 0u, 0u, 0u);
        c[k][0] = v.x & RGB_MASK; c[k][1] = v.y & RGB_MASK; c[k][2] = v.z & RGB_MASK; c[k][3] = v.w & RGB_MASK;
      } else {
        c[k][0] = on ? *p & RGB_MASK : 0u;
      }
      if (k > 0)                             // lane 0: the pixel left of the warp's columns
        l[k - 1] = lane == 0 && on && x > 0 ? p[-1] & RGB_MASK : 0u;
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const uint32_t beside = __shfl_up_sync(0xffffffffu, c[k + 1][PX - 1], 1);
      if (!in || y0 + k >= H) continue;
      const uint32_t left = lane == 0 ? l[k] : beside;
      if (x > 0) sum += (unsigned)rgb_dist2(c[k + 1][0], left);
#pragma unroll
      for (int j = 0; j < PX; ++j) {
        if (y0 + k > 0) sum += (unsigned)rgb_dist2(c[k + 1][j], c[k][j]);
        if (j > 0) sum += (unsigned)rgb_dist2(c[k + 1][j], c[k + 1][j - 1]);
      }
    }
    acc64 += sum;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) acc64 += __shfl_xor_sync(0xffffffffu, acc64, o);
  if (lane == 0) part[threadIdx.x >> 5] = acc64;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tsum = 0;
    for (int k = 0; k < DSUM_THREADS / 32; ++k) tsum += part[k];
    if (tsum) atomicAdd(state, tsum);
    __threadfence();
    s_last = atomicAdd(state + 1, 1ull) == gridDim.x - 1;
    if (s_last) {
      __threadfence();
      s_total = *((volatile unsigned long long*)state);
      state[0] = 0;
      state[1] = 0;
      *acc = ImageAcc{};   // the image's sums start afresh with the upload that follows
    }
  }
  __syncthreads();
  if (s_last && threadIdx.x < GC_NLINK_LEVELS) nlink_table(s_total, npairs, threadIdx.x + 1, tab);
}

// Whether a freshly uploaded tile belongs in the first list of a solve: it holds excess, and a
// sink lies in the tile or just across one of its sides.  Under the trivial labelling (0 at
// sinks, 1 elsewhere) the first sweep of any other tile pushes nothing, and its excess is too
// far from a sink to deliver any within the first cycle; if it can reach one, the relabel
// after the cycle's flood lists its tile with exact distances.  On six 1024^2 synthetic grids
// the rule lists 146 to 661 tiles of the 654 to 927 that hold excess (median 270 of 792).
__device__ __forceinline__ bool fresh_tile_active(const PoolView& P, int t) {
  const int f = P.tflag[t];
  if (!(f & TF_POS)) return false;
  if (f & TF_SINK) return true;
  const int4 nb = P.nbr[t];
  return ((f & TF_POS_UP) && nb.x >= 0 && (P.tflag[nb.x] & TF_SINK_DOWN)) ||
         ((f & TF_POS_DOWN) && nb.y >= 0 && (P.tflag[nb.y] & TF_SINK_UP)) ||
         ((f & TF_POS_LEFT) && nb.z >= 0 && (P.tflag[nb.z] & TF_SINK_RIGHT)) ||
         ((f & TF_POS_RIGHT) && nb.w >= 0 && (P.tflag[nb.w] & TF_SINK_LEFT));
}

// Mask rebuild of the selected tiles whose planes changed since their masks were written
// (dirty flag set), one warp per tile.  The solve loops do not need it: their first flood
// round rebuilds the dirty tiles it covers.  It precedes a global relabel that no flood
// precedes (gc_start_bfs).
__global__ void __launch_bounds__(WARPS_PER_CTA * 32)
k_masks(PoolView P) {
  trace_mark(P, TR_MASKS);
  __shared__ int s_n, s_nr;
  if (threadIdx.x == 0) {
    int n = *((volatile int32_t*)&P.nsel[1]), nr = *((volatile int32_t*)&P.nsel[0]);
    if (n < 0 || n > P.nt || nr < 0 || nr > P.nimg) {   // self-check
      record_bad(P, 9, n);
      n = nr = 0;
    }
    s_n = n;
    s_nr = nr;
  }
  __syncthreads();
  const int n = s_n;
  const int lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * WARPS_PER_CTA + (threadIdx.x >> 5);
  const int stride = gridDim.x * WARPS_PER_CTA;
  SelCursor cursor(P, s_nr, i0 < n ? i0 : 0);
  for (int i = i0; i < n; i += stride) {
    const int t = cursor.tile(i);
    if (P.mdirty[t] == 0) continue;   // the same word for every lane: warp-uniform
    long long pos;
    warp_rebuild_masks(P, t, lane, &pos);
    if (lane == 0 && P.ktiles) atomicAdd(&P.ktiles[K_MASKS], 1ull);
  }
}

// ------------------------------------------------------------------------------------
// Discharge.  Thread (r, q) owns pixels (r, 4q .. 4q+3) of the tile.
//
// Every pixel pushes along all admissible edges and relabels, tile-edge pixels included,
// but a tile-edge pixel rises by at most 2 above its height at the start of the launch.
// A neighbouring CTA that pushes into an edge pixel v saw either v's start height or its
// final height; with h_final(v) <= h_start(v) + 2 every such push leaves a valid labelling
// (h(v) <= h(u) + 1 on the new residual edge v -> u), and pushes out of the tile read the
// neighbour's height under the same bound.  Flow leaving the tile is added to the
// neighbour's excess and reverse residual with atomics at the end of the tile.
//
// Active tiles form a worklist: a pulse reads queue[c] (c = pulse parity) and appends,
// deduplicated by inq[c ^ 1], every tile that is still active or received flow to
// queue[c ^ 1].  No compaction between pulses; the last pulse before a relabel appends
// nothing in k_solve, since the relabel rebuilds the list.
// ------------------------------------------------------------------------------------
struct DisSmem {
  int32_t hs[GC_TILE_PX + 2 * GC_TILE];   // heights, with a halo row above and below
  int32_t fu[GC_TILE_PX + GC_TILE];       // flow pushed up by each pixel this sweep, and a zero row
  int32_t fd[GC_TILE_PX + GC_TILE];       // a zero row, and flow pushed down
  int32_t eo_top[GC_TILE], eo_bot[GC_TILE], eo_left[GC_TILE], eo_right[GC_TILE];
  int32_t xv_top[GC_TILE], xv_bot[GC_TILE];   // flow out of the tile across its first / last row
};

// A worklist of tiles: list, length, and the per-tile flag that keeps a tile in it once.
// local: a shared-memory counter of the tiles this CTA appends (k_solve; null elsewhere).
struct Worklist {
  int32_t *list, *count, *in;
  int* local = nullptr;
};

__device__ __forceinline__ void worklist_append(const PoolView& P, const Worklist& w, int t) {
  const int pos = atomicAdd(w.count, 1);
  if (pos < P.nt) w.list[pos] = t;   // each tile at most once, so pos < nt always holds
  else record_bad(P, 1, pos);
}

__device__ __forceinline__ int4 lds4(const int32_t* p) { return *reinterpret_cast<const int4*>(p); }
__device__ __forceinline__ void sts4(int32_t* p, int a, int b, int c, int d) {
  *reinterpret_cast<int4*>(p) = make_int4(a, b, c, d);
}

// Bulk copies global -> shared memory (cp.async.bulk, completion on an mbarrier).  The
// copies are plain (no cluster multicast); every wait on the mbarrier is bounded.
__device__ __forceinline__ void mbar_init(uint64_t* mbar, unsigned count) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mbar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, unsigned bytes) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mbar);
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* mbar) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const unsigned m = (unsigned)__cvta_generic_to_shared(mbar);
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(d), "l"(src), "r"(bytes), "r"(m) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* mbar, unsigned parity) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mbar);
  unsigned ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok != 0;
}
// Asynchronous copies of a few bytes global -> shared memory by one thread (cp.async).
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A tile copy normally lands in microseconds; a wait gives up after this long.  The bound
// is on time, not on polls: try_wait may return at once, and a poll count then would allow
// only milliseconds under load (a CTA that gave up early would leave while its copy is
// still landing in shared memory).
constexpr unsigned long long GC_COPY_WAIT_NS = 2000000000ull;
// Bounded wait: false when the copy did not complete within limit_ns.  The iteration cap
// only guards against a timer that does not advance.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, unsigned parity,
                                          unsigned long long limit_ns = GC_COPY_WAIT_NS) {
  if (mbar_try_wait(mbar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (unsigned i = 1; i < (1u << 31); ++i) {
    if (mbar_try_wait(mbar, parity)) return true;
    if ((i & 255u) == 0 && global_ns() - t0 > limit_ns) return false;
  }
  return false;
}

constexpr int DIS_PLANES = 6;                                  // excess, height, 4 residuals
constexpr unsigned DIS_TILE_BYTES = DIS_PLANES * GC_TILE_PX * 4;  // 24 KiB
// dynamic shared memory: the tile staging buffer + the per-round exchange arrays
constexpr size_t DIS_DYN_SMEM = (size_t)DIS_TILE_BYTES + sizeof(DisSmem);

__device__ __forceinline__ const int32_t* dis_plane(const PoolView& P, int k) {
  return k == 0 ? P.exc : k == 1 ? P.hgt : P.cap[k - 2];
}

// Thread 0: start the bulk copy of tile t's six planes into buffer `buf`.
__device__ __forceinline__ void dis_prefetch(const PoolView& P, int t, int32_t* buf, uint64_t* mbar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // buffer was last read by threads
  mbar_expect_tx(mbar, DIS_TILE_BYTES);
#pragma unroll
  for (int k = 0; k < DIS_PLANES; ++k)
    bulk_g2s(buf + k * GC_TILE_PX, dis_plane(P, k) + (long long)t * GC_TILE_PX, GC_TILE_PX * 4, mbar);
}

// Discharges the n tiles of list `in` with the CTAs 0 .. nb-1 (this is CTA `bid`); the tiles
// active afterwards or sent flow go to list `out` (none: out.list null).  hlim: pixels with a
// smaller height are active (GC_HINF: all that can reach a sink; smaller after a relabel capped
// at distance hlim - 1, whose heights from hlim on only mean "at least hlim").  A pixel that
// rises to hlim stays there, inactive until the next relabel.  buf, S and mbar are the CTA's
// staging buffer, exchange arrays and (initialised) mbarrier; `phase` its parity, kept from
// call to call.  Every thread of the CTA calls it.
//
// What bounds it: with a few hundred tiles in a list each CTA has one, and the pulse is one
// tile's latency; with more, instruction issue.  So the sweep has no divergent branch (a
// pixel's four pushes and its relabel are selects and minima), the horizontal neighbours come
// by shuffle, only vertical exchange goes through shared memory, and a tile's bookkeeping is
// one pass at the end.  Cycles of one tile alone on its SM, against branches per direction and
// exchange through shared memory only: about 1200 a sweep (1000 to 2650), 1700 for the
// write-back (3000).  3 CTAs per SM (80 registers) beat 4 (64, with spills) by 5 to 10 %.
__device__ __forceinline__ void discharge_phase(const PoolView& P, int iters, int hlim, int bid,
                                                int nb_ctas, const Worklist& in, int n,
                                                const Worklist& out, int32_t* buf, DisSmem& S,
                                                uint64_t* mbar, unsigned& phase) {
  const unsigned F = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  const int r = tid >> 3, q = tid & 7, c0 = q * 4;
  // Bookkeeping log: each tile leaves (tile, neighbours, flags) here, and the CTA's threads
  // settle up to DIS_LOG tiles at once (its list entry, and the list entries and dirty flags
  // of the neighbours it sent flow to), so the dependent L2 round trips of that bookkeeping
  // are paid once per flush, not once per tile.  Nothing in this pulse reads what it writes:
  // the next list, the dirty flags and act_int are read by later steps.  A flush comes before
  // the write-back of its last tile: the warps it occupies wait for the list's atomics while
  // the others store.
  __shared__ int s_logt[DIS_LOG];
  __shared__ unsigned s_logf[DIS_LOG];
  __shared__ int4 s_lognb[DIS_LOG];
  int nlog = 0;   // the same in every thread
  auto flush_log = [&](int cnt) {
    for (int b = 0; b < cnt * 5; b += DIS_THREADS) {
      const int w = b + tid;
      bool won = false;
      int target = 0;
      if (w < cnt * 5) {
        const int i = w / 5, k = w - i * 5;       // k = 0: the tile; 1..4: up, down, left, right
        const int tt = s_logt[i];
        const unsigned f = s_logf[i];
        const int4 nbb = s_lognb[i];
        target = k == 0 ? tt : k == 1 ? nbb.x : k == 2 ? nbb.y : k == 3 ? nbb.z : nbb.w;
        if (k == 0 || ((f >> (k - 1)) & 1)) {
          P.touched[target] = 1;
          mark_dirty(P, target);   // its masks are rebuilt by the next flood's first round
          if (k == 0) {
            P.act_int[tt] = (f >> 5) & 1;
            P.hstate[tt] = 0;
          }
          if (out.list && (k != 0 || ((f >> 4) & 1))) won = atomicExch(&out.in[target], 1) == 0;
          if (k == 0 && P.ktiles) atomicAdd(&P.ktiles[K_DISCHARGE], 1ull);
        }
      }
      // one add of the list's length per warp
      const unsigned m = __ballot_sync(F, won);
      if (m) {
        int pos = 0;
        if (lane == 0) {
          pos = atomicAdd(out.count, __popc(m));
          if (out.local) atomicAdd(out.local, __popc(m));
        }
        pos = __shfl_sync(F, pos, 0) + __popc(m & ((1u << lane) - 1u));
        if (won) {
          if (pos < P.nt) out.list[pos] = target;   // `in` deduplicates, so pos < nt always holds
          else record_bad(P, 1, pos);
        }
      }
    }
  };
  if (n < 0 || n > P.nt) {   // self-check: a list never holds more than every tile once
    if (tid == 0 && bid == 0) record_bad(P, 2, n);
    n = 0;
  }
  // list entry li: every position below the checked count was written with a tile id of
  // the pool (by a pulse, a relabel or a compaction) before this pulse
  auto entry = [&](int li) { return in.list[li]; };
  const bool erow = r == 0 || r == 31, ecol = q == 0 || q == 7;
  const int pix = r * GC_TILE + c0;
  const bool left = q == 0;
  int32_t* const hs = S.hs + GC_TILE + pix;        // this thread's heights (rows -1 and 32: halo)
  if (tid < GC_TILE) {   // no flow enters from beyond the first and last row
    S.fu[GC_TILE_PX + tid] = 0;
    S.fd[tid] = 0;
  }
  // Tile ids and neighbour ids run ahead of the tiles (thread 0, asynchronous copies into
  // shared memory), so no warp waits for a list entry before its tile's sweeps: while tile k
  // is worked on, the entry of tile k + 2 and the neighbours of tile k + 1 arrive.
  __shared__ int s_id[2];            // entries of the tiles after this one, by parity
  __shared__ __align__(16) int4 s_nb[2];   // neighbour ids by parity
  bool failed = false;
  int par = 0;
  if (bid < n) {
    if (tid == 0) {
      const int t0 = entry(bid);
      dis_prefetch(P, t0, buf, mbar);
      s_id[0] = t0;
      s_nb[0] = P.nbr[t0];
      if (bid + nb_ctas < n) s_id[1] = entry(bid + nb_ctas);
    }
    __syncthreads();
  }
  for (int li = bid; li < n; li += nb_ctas, par ^= 1) {
    const int t = s_id[par];
    const int4 nb = s_nb[par];
    // halo heights, loaded while the tile's copy lands
    int4 hv = make_int4(GC_HINF, GC_HINF, GC_HINF, GC_HINF);   // first / last row: across the side
    int hside = GC_HINF;                                       // first / last strip: across the side
    const int nv = r == 0 ? nb.x : nb.y, nh_ = left ? nb.z : nb.w;
    if (erow && nv >= 0)
      hv = *reinterpret_cast<const int4*>(P.hgt + (long long)nv * GC_TILE_PX + (r == 0 ? 31 * GC_TILE : 0) + c0);
    if (ecol && nh_ >= 0) hside = P.hgt[(long long)nh_ * GC_TILE_PX + r * GC_TILE + (left ? 31 : 0)];
    if (tid == 0) {
      in.in[t] = 0;
      s_logt[nlog] = t;
      s_lognb[nlog] = nb;
      s_logf[nlog] = 0;
    }
    const bool ok = mbar_wait(mbar, phase);
    if (__syncthreads_or(!ok)) { failed = true; break; }  // block-uniform
    phase ^= 1u;
    int e[4], h[4], cu[4], cd[4], cl[4], cr[4], hcap[4];
    {
      int4 v = lds4(buf + 0 * GC_TILE_PX + pix); e[0] = v.x; e[1] = v.y; e[2] = v.z; e[3] = v.w;
      // launch-start excess of the pixels that also receive atomics from neighbouring tiles
      // (written back as deltas against it)
      if (erow) {
        sts4((r == 0 ? S.eo_top : S.eo_bot) + c0, v.x, v.y, v.z, v.w);
        sts4((r == 0 ? S.xv_top : S.xv_bot) + c0, 0, 0, 0, 0);
      }
      if (ecol) (left ? S.eo_left : S.eo_right)[r] = left ? v.x : v.w;
      v = lds4(buf + 1 * GC_TILE_PX + pix); h[0] = v.x; h[1] = v.y; h[2] = v.z; h[3] = v.w;
      sts4(hs, v.x, v.y, v.z, v.w);
      v = lds4(buf + 2 * GC_TILE_PX + pix); cu[0] = v.x; cu[1] = v.y; cu[2] = v.z; cu[3] = v.w;
      v = lds4(buf + 3 * GC_TILE_PX + pix); cd[0] = v.x; cd[1] = v.y; cd[2] = v.z; cd[3] = v.w;
      v = lds4(buf + 4 * GC_TILE_PX + pix); cl[0] = v.x; cl[1] = v.y; cl[2] = v.z; cl[3] = v.w;
      v = lds4(buf + 5 * GC_TILE_PX + pix); cr[0] = v.x; cr[1] = v.y; cr[2] = v.z; cr[3] = v.w;
    }
    if (r == 0) sts4(hs - GC_TILE, hv.x, hv.y, hv.z, hv.w);
    if (r == 31) sts4(hs + GC_TILE, hv.x, hv.y, hv.z, hv.w);
    // heights a pixel may reach in this pulse: tile-edge pixels 2 above their start
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool edge = erow || (j == 0 && q == 0) || (j == 3 && q == 7);
      hcap[j] = edge ? imin(h[j] + 2, hlim) : hlim;
    }
    int xh = 0;   // flow out of the tile across the first / last column (rows: S.xv_*)
    __syncthreads();   // every thread has its values in registers: the buffer is free
    // prefetch this CTA's next tile into the buffer while this one is worked on
    if (tid == 0 && li + nb_ctas < n) {
      const int tn = s_id[par ^ 1];
      dis_prefetch(P, tn, buf, mbar);
      copy_async<16>(&s_nb[par ^ 1], P.nbr + tn);
      if (li + 2 * nb_ctas < n) copy_async<4>(&s_id[par], in.list + li + 2 * nb_ctas);
    }

    for (int it = 0; it < iters; ++it) {
      // neighbour heights (fixed during the sweep)
      const int4 hup = lds4(hs - GC_TILE), hdn = lds4(hs + GC_TILE);
      const int hnu[4] = {hup.x, hup.y, hup.z, hup.w}, hnd[4] = {hdn.x, hdn.y, hdn.z, hdn.w};
      int hl = __shfl_up_sync(F, h[3], 1), hr = __shfl_down_sync(F, h[0], 1);
      if (q == 0) hl = hside;
      if (q == 7) hr = hside;
      const int hnl[4] = {hl, h[0], h[1], h[2]}, hnr[4] = {h[1], h[2], h[3], hr};
      // push along every admissible edge: down, up, right, left
      int ou[4] = {0, 0, 0, 0}, od[4] = {0, 0, 0, 0}, ol[4] = {0, 0, 0, 0}, orr[4] = {0, 0, 0, 0};
      int changed = 0;
      if (__any_sync(F, (e[0] > 0 && h[0] < hlim) || (e[1] > 0 && h[1] < hlim) ||
                            (e[2] > 0 && h[2] < hlim) || (e[3] > 0 && h[3] < hlim))) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // the height to push to (none for an inactive pixel: no height is negative)
          const int hm1 = e[j] > 0 && h[j] < hlim ? h[j] - 1 : -1;
          od[j] = hnd[j] == hm1 ? imin(e[j], cd[j]) : 0;
          e[j] -= od[j]; cd[j] -= od[j];
          ou[j] = hnu[j] == hm1 ? imin(e[j], cu[j]) : 0;
          e[j] -= ou[j]; cu[j] -= ou[j];
          orr[j] = hnr[j] == hm1 ? imin(e[j], cr[j]) : 0;
          e[j] -= orr[j]; cr[j] -= orr[j];
          ol[j] = hnl[j] == hm1 ? imin(e[j], cl[j]) : 0;
          e[j] -= ol[j]; cl[j] -= ol[j];
          changed |= od[j] | ou[j] | orr[j] | ol[j];
        }
      }
      // flow leaving the tile is delivered at the end of the tile
      if (r == 0) {
        const int4 x = lds4(S.xv_top + c0);
        sts4(S.xv_top + c0, x.x + ou[0], x.y + ou[1], x.z + ou[2], x.w + ou[3]);
      }
      if (r == 31) {
        const int4 x = lds4(S.xv_bot + c0);
        sts4(S.xv_bot + c0, x.x + od[0], x.y + od[1], x.z + od[2], x.w + od[3]);
      }
      xh += q == 0 ? ol[0] : q == 7 ? orr[3] : 0;
      sts4(S.fu + pix, ou[0], ou[1], ou[2], ou[3]);
      sts4(S.fd + GC_TILE + pix, od[0], od[1], od[2], od[3]);
      int fl = __shfl_up_sync(F, orr[3], 1), fr = __shfl_down_sync(F, ol[0], 1);
      if (q == 0) fl = 0;
      if (q == 7) fr = 0;
      __syncthreads();
      // gather inflow; a pixel receiving flow gains the reverse residual
      {
        const int4 a = lds4(S.fu + pix + GC_TILE), b = lds4(S.fd + pix);
        const int below[4] = {a.x, a.y, a.z, a.w}, above[4] = {b.x, b.y, b.z, b.w};
        const int fromleft[4] = {fl, orr[0], orr[1], orr[2]};
        const int fromright[4] = {ol[1], ol[2], ol[3], fr};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          e[j] += below[j] + above[j] + fromleft[j] + fromright[j];
          cd[j] += below[j];
          cu[j] += above[j];
          cl[j] += fromleft[j];
          cr[j] += fromright[j];
        }
      }
      // relabel (Jacobi) to one above the lowest residual neighbour m.  The labelling is valid,
      // so h <= m + 1, with equality exactly when an admissible edge is left: the pixel then
      // keeps its height.  So does one at its limit, and an inactive one (h >= hlim >= hcap);
      // a warp of only such pixels skips the step.
      if (__any_sync(F, (e[0] > 0 && h[0] < hcap[0]) || (e[1] > 0 && h[1] < hcap[1]) || (e[2] > 0 && h[2] < hcap[2]) || (e[3] > 0 && h[3] < hcap[3]))) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          int m = GC_HINF;
          m = cd[j] > 0 ? imin(m, hnd[j]) : m;
          m = cu[j] > 0 ? imin(m, hnu[j]) : m;
          m = cr[j] > 0 ? imin(m, hnr[j]) : m;
          m = cl[j] > 0 ? imin(m, hnl[j]) : m;
          const int up = imin(m + 1, hcap[j]);
          const int to = e[j] > 0 && up > h[j] ? up : h[j];
          changed |= to ^ h[j];
          ou[j] = to;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) ou[j] = h[j];
      }
      // every read of S.hs in this sweep happened before the flow barrier above, so the new
      // heights can be written now; the next reads follow the barrier below
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = ou[j];
      sts4(hs, h[0], h[1], h[2], h[3]);
      if (!__syncthreads_or(changed)) break;
    }

    // bits 0-3: sent up, down, left, right; 4: active; 5: interior active
    unsigned flags = 0;
    int4 xo = make_int4(0, 0, 0, 0);
    if (erow) xo = lds4((r == 0 ? S.xv_top : S.xv_bot) + c0);
    if (xo.x | xo.y | xo.z | xo.w) flags |= r == 0 ? 1u : 2u;
    if (xh) flags |= left ? 4u : 8u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool edge = erow || (j == 0 && q == 0) || (j == 3 && q == 7);
      if (e[j] > 0 && h[j] < hlim) flags |= edge ? 16u : 48u;
    }
    flags = __reduce_or_sync(F, flags);
    if (lane == 0 && flags) atomicOr(&s_logf[nlog], flags);
    if (tid == 0) copy_async_wait();   // the next tile's ids
    __syncthreads();   // the log entry is complete; orders the exchange arrays' reuse, too
    // (an entry is rewritten after a flush behind at least one more barrier, but for entry 0,
    // which only lanes of thread 0's warp read)
    if (++nlog == DIS_LOG || li + nb_ctas >= n) {
      flush_log(nlog);
      nlog = 0;
      __syncwarp();
    }

    // write back: interior values are owned by this CTA; tile-edge excess and the outward
    // residual of edge pixels also receive atomics from neighbouring tiles, so they are
    // written as deltas.  Flow across a side goes to the neighbour pixel's excess and its
    // reverse residual.
    const long long off = (long long)t * GC_TILE_PX + pix;
    *(int4*)(P.hgt + off) = make_int4(h[0], h[1], h[2], h[3]);
    if (r != 0) *(int4*)(P.cap[DUP] + off) = make_int4(cu[0], cu[1], cu[2], cu[3]);
    if (r != 31) *(int4*)(P.cap[DDOWN] + off) = make_int4(cd[0], cd[1], cd[2], cd[3]);
    if (q != 0) *(int4*)(P.cap[DLEFT] + off) = make_int4(cl[0], cl[1], cl[2], cl[3]);
    if (q != 7) *(int4*)(P.cap[DRIGHT] + off) = make_int4(cr[0], cr[1], cr[2], cr[3]);
    if (!erow && !ecol) *(int4*)(P.exc + off) = make_int4(e[0], e[1], e[2], e[3]);
    if (erow) {
      const int4 v = lds4((r == 0 ? S.eo_top : S.eo_bot) + c0);
      const int e0[4] = {v.x, v.y, v.z, v.w}, xv[4] = {xo.x, xo.y, xo.z, xo.w};
      int32_t* const own = (r == 0 ? P.cap[DUP] : P.cap[DDOWN]) + off;
      const long long o = (long long)nv * GC_TILE_PX + (r == 0 ? 31 * GC_TILE : 0) + c0;
      int32_t* const rev = (r == 0 ? P.cap[DDOWN] : P.cap[DUP]) + o;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (e[j] != e0[j]) atomicAdd(P.exc + off + j, e[j] - e0[j]);
        if (xv[j]) {   // only where the neighbour exists: capacities out of the image are 0
          atomicAdd(own + j, -xv[j]);
          atomicAdd(P.exc + o + j, xv[j]);
          atomicAdd(rev + j, xv[j]);
        }
      }
    }
    if (ecol) {
      int32_t* const own = (left ? P.cap[DLEFT] : P.cap[DRIGHT]) + off;   // the strip's plane
      const int s0 = left ? 1 : 0;   // its three pixels that are not on the side
      own[s0] = left ? cl[1] : cr[0];
      own[s0 + 1] = left ? cl[2] : cr[1];
      own[s0 + 2] = left ? cl[3] : cr[2];
      const int js = left ? 0 : 3;
      if (!erow) {
        P.exc[off + s0] = left ? e[1] : e[0];
        P.exc[off + s0 + 1] = left ? e[2] : e[1];
        P.exc[off + s0 + 2] = left ? e[3] : e[2];
        const int d = left ? e[0] - S.eo_left[r] : e[3] - S.eo_right[r];
        if (d) atomicAdd(P.exc + off + js, d);
      }
      if (xh) {
        const long long o = (long long)nh_ * GC_TILE_PX + r * GC_TILE + (left ? 31 : 0);
        atomicAdd(own + js, -xh);
        atomicAdd(P.exc + o, xh);
        atomicAdd((left ? P.cap[DRIGHT] : P.cap[DLEFT]) + o, xh);
      }
    }
  }
  if (failed) {
    flush_log(nlog);   // the tiles done before
    // a bulk copy did not complete in time: record it, let our copy drain, stop
    if (tid == 0) {
      atomicExch(&P.ctl[CTL_ERR], 3);
      abort_solve(P);
      mbar_wait(mbar, phase, 5 * GC_COPY_WAIT_NS);
    }
    __syncthreads();
  }
}

// One pulse of the host-driven loop or of a manual push: the worklist of the pulse parity.
__global__ void __launch_bounds__(DIS_THREADS, 3)
k_discharge(PoolView P, int iters, int hlim) {
  trace_mark(P, TR_DISCHARGE);
  extern __shared__ __align__(128) int32_t dsm[];
  DisSmem& S = *reinterpret_cast<DisSmem*>(dsm + DIS_PLANES * GC_TILE_PX);
  __shared__ uint64_t mbar;
  __shared__ int s_cur, s_n;
  if (threadIdx.x == 0) {
    s_cur = *((volatile int32_t*)&P.ctl[CTL_PULSE]) & 1;
    s_n = *((volatile int32_t*)&P.qcount[s_cur]);
    mbar_init(&mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int cur = s_cur, nxt = cur ^ 1;
  const Worklist in{P.queue[cur], P.qcount + cur, P.inq[cur]};
  const Worklist out{P.queue[nxt], P.qcount + nxt, P.inq[nxt]};
  unsigned phase = 0;
  discharge_phase(P, iters, hlim, blockIdx.x, gridDim.x, in, s_n, out, dsm, S, &mbar, phase);
  // last CTA: the queue just read is consumed; the next launch reads the other one
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const int d = atomicAdd(&P.ctl[CTL_DDONE], 1);
    if (d == (int)gridDim.x - 1) {
      P.qcount[cur] = 0;
      P.ctl[CTL_PULSE] = P.ctl[CTL_PULSE] + 1;
      P.ctl[CTL_DDONE] = 0;
      __threadfence();
    }
  }
}

// ------------------------------------------------------------------------------------
// Edge relabel + active-tile list.
// ------------------------------------------------------------------------------------
constexpr int EB_THREADS = 512;
constexpr int EB_WARPS = EB_THREADS / 32;
constexpr int EB_TILES = 64;                 // tiles per CTA (4 per warp)

// Relabels up to four tile-edge pixels of one lane (Jacobi: neighbour heights are read
// as they are, a concurrent update only makes them larger, which keeps the labelling
// valid).  Returns whether one of them is active afterwards.
__device__ __forceinline__ int edge_relabel_lane(const PoolView& P, int t, int4 nb, int lane) {
  int rr[4] = {0, 31, lane, lane}, cc[4] = {lane, lane, 0, 31};
  const bool use[4] = {true, true, lane > 0 && lane < 31, lane > 0 && lane < 31};
  const long long base = (long long)t * GC_TILE_PX;
  int e[4], h[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long long o = base + rr[k] * GC_TILE + cc[k];
    e[k] = use[k] ? P.exc[o] : 0;
    h[k] = use[k] ? P.hgt[o] : GC_HINF;
  }
  int act = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!(e[k] > 0 && h[k] < GC_HINF)) continue;
    const int r = rr[k], c = cc[k];
    const long long o = base + r * GC_TILE + c;
    const int cu = P.cap[DUP][o], cd = P.cap[DDOWN][o], cl = P.cap[DLEFT][o], cr = P.cap[DRIGHT][o];
    int hu = GC_HINF, hd = GC_HINF, hl = GC_HINF, hr = GC_HINF;
    if (r > 0) hu = P.hgt[o - GC_TILE]; else if (nb.x >= 0) hu = P.hgt[(long long)nb.x * GC_TILE_PX + 31 * GC_TILE + c];
    if (r < 31) hd = P.hgt[o + GC_TILE]; else if (nb.y >= 0) hd = P.hgt[(long long)nb.y * GC_TILE_PX + c];
    if (c > 0) hl = P.hgt[o - 1]; else if (nb.z >= 0) hl = P.hgt[(long long)nb.z * GC_TILE_PX + r * GC_TILE + 31];
    if (c < 31) hr = P.hgt[o + 1]; else if (nb.w >= 0) hr = P.hgt[(long long)nb.w * GC_TILE_PX + r * GC_TILE];
    const int hh = h[k];
    const bool adm = (cu > 0 && hh == hu + 1) || (cd > 0 && hh == hd + 1) || (cl > 0 && hh == hl + 1) ||
                     (cr > 0 && hh == hr + 1);
    if (adm) { act = 1; continue; }
    int m = GC_HINF;
    if (cu > 0) m = imin(m, hu + 1);
    if (cd > 0) m = imin(m, hd + 1);
    if (cl > 0) m = imin(m, hl + 1);
    if (cr > 0) m = imin(m, hr + 1);
    m = imin(m, GC_HINF);
    if (m != hh) P.hgt[o] = m;
    act |= m < GC_HINF;
  }
  return act;
}

// Edge relabel + active-tile list (one launch).  A CTA owns EB_TILES consecutive tiles by
// arrival ticket; each warp takes 4 of them and relabels only the touched ones (one warp
// per tile, 4 edge pixels per lane).  A tile is active when an interior pixel was active
// after its discharge or a tile-edge pixel is active after this relabel.  The active tiles
// are compacted in tile order with a warp-parallel decoupled look-back.
__global__ void __launch_bounds__(EB_THREADS)
k_edge_relabel_build(PoolView P, int32_t* list, int32_t* count, ScanState st) {
  __shared__ int32_t flag[EB_TILES];
  __shared__ int32_t s_chunk;
  __shared__ uint32_t s_tag;
  if (threadIdx.x == 0) {
    s_chunk = atomicAdd(st.ticket, 1);
    s_tag = *((volatile uint32_t*)st.seq);
  }
  __syncthreads();
  const int chunk = s_chunk;
  const int nchunks = (P.nt + EB_TILES - 1) / EB_TILES;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int PER_WARP = EB_TILES / EB_WARPS;
  const int t0 = chunk * EB_TILES + warp * PER_WARP;
  int touched = 0;
  if (lane < PER_WARP && t0 + lane < P.nt) {
    touched = P.touched[t0 + lane];
    P.inq[0][t0 + lane] = 0;  // the worklists are replaced by the rebuilt list
    P.inq[1][t0 + lane] = 0;
  }
  unsigned todo = __ballot_sync(0xffffffffu, touched != 0);
  if (lane < PER_WARP) flag[warp * PER_WARP + lane] = 0;
  __syncwarp();
  while (todo) {
    const int k = __ffs(todo) - 1;
    todo &= todo - 1;
    const int t = t0 + k;
    const int4 nb = P.nbr[t];
    const int a = edge_relabel_lane(P, t, nb, lane);
    const int active = __any_sync(0xffffffffu, a) | P.act_int[t];
    if (lane == 0) {
      flag[warp * PER_WARP + k] = active;
      P.touched[t] = 0;
      P.hstate[t] = 0;   // its heights may have changed
      if (P.ktiles) atomicAdd(&P.ktiles[K_EDGE_BUILD], 1ull);
    }
  }
  __syncthreads();
  if (warp == 0) {
    const int v0 = flag[2 * lane], v1 = flag[2 * lane + 1];   // two flags per lane
    const int v = v0 + v1;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int agg = __shfl_sync(0xffffffffu, x, 31);
    const int excl = lookback_exclusive_warp(st, s_tag, chunk, agg);
    int pos = excl + x - v;
    const int tb = chunk * EB_TILES + 2 * lane;
    if ((unsigned)pos + (unsigned)(v0 + v1) <= (unsigned)P.nt) {
      if (v0) list[pos++] = tb;
      if (v1) list[pos] = tb + 1;
    } else if (v) {
      scan_error(st, 2);   // only after a look-back that gave up
    }
    if (chunk == nchunks - 1 && lane == 0) *count = excl + agg;
    if (lane == 0) scan_finish(st, nchunks);
  }
}

// ------------------------------------------------------------------------------------
// Global relabel: bit-parallel BFS per tile, one warp per tile, lane = row.
// ------------------------------------------------------------------------------------

__device__ __forceinline__ int warp_min(int v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = imin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Multi-source BFS inside a tile on the row masks, level by level (a bucketed BFS with unit
// steps): level 0 holds the sink pixels; a tile-edge pixel with a residual edge into the
// neighbour tile is also seeded at (neighbour height + 1).  Lane c holds the seeds of column c
// in the top row (`top`) and the bottom row (`bot`); lane r holds the seeds of row r at column
// 0 (`sl`) and 31 (`sr`); GC_HINF where there is none.  Level L visits the unvisited pixels
// that are seeds of value L or neighbours, over residual edges, of level L - 1; an empty level
// jumps to the smallest unvisited seed.  Levels above `cap` stay unreached.  Lane r writes the
// distances of row r into `row` (GC_HINF where unreached) and gets the mask of reached pixels.
__device__ __forceinline__ uint32_t tile_bfs_seeded(int* row, uint32_t sink, uint32_t canU,
                                                    uint32_t canD, uint32_t canL, uint32_t canR,
                                                    int lane, int top, int bot, int sl, int sr,
                                                    int cap) {
  const unsigned FULL = 0xffffffffu;
#pragma unroll
  for (int c = 0; c < 32; ++c) row[c] = GC_HINF;
  uint32_t vis = 0, F = 0;
  const int last = imin(cap, GC_HINF - 1);
  int L = __any_sync(FULL, sink != 0) ? 0 : warp_min(imin(imin(top, bot), imin(sl, sr)));
  // every step visits a pixel or jumps to an unvisited seed: at most 1024 + 128 steps
  for (int step = 0; step < 2 * GC_TILE_PX && L <= last; ++step) {
    uint32_t Fu = __shfl_up_sync(FULL, F, 1);
    uint32_t Fd = __shfl_down_sync(FULL, F, 1);
    if (lane == 0) Fu = 0;
    if (lane == 31) Fd = 0;
    const uint32_t bt = __ballot_sync(FULL, top == L);
    const uint32_t bb = __ballot_sync(FULL, bot == L);
    uint32_t S = (L == 0 ? sink : 0u) | (sl == L ? 1u : 0u) | (sr == L ? 0x80000000u : 0u);
    if (lane == 0) S |= bt;
    if (lane == 31) S |= bb;
    const uint32_t N = (((F >> 1) & canR) | ((F << 1) & canL) | (Fu & canU) | (Fd & canD) | S) & ~vis;
    vis |= N;
    F = N;
    for (uint32_t b = N; b; b &= b - 1) row[__ffs(b) - 1] = L;
    if (__any_sync(FULL, F != 0)) {
      ++L;
      continue;
    }
    // the frontier is empty: the next level that still has an unvisited seed
    const uint32_t v0 = __shfl_sync(FULL, vis, 0), v31 = __shfl_sync(FULL, vis, 31);
    int cand = GC_HINF;
    if (top > L && !((v0 >> lane) & 1u)) cand = imin(cand, top);
    if (bot > L && !((v31 >> lane) & 1u)) cand = imin(cand, bot);
    if (sl > L && !(vis & 1u)) cand = imin(cand, sl);
    if (sr > L && !(vis >> 31)) cand = imin(cand, sr);
    L = warp_min(cand);
  }
  return vis;
}

// Frontier rounds.  The first round of a relabel or flood processes the solve's selected
// tiles (grid-stride over the selection); round r > 0 processes the list fq[r & 1] built by
// round r - 1.  A tile whose boundary
// values changed queues its neighbours in fq[(r + 1) & 1], deduplicated by mark[(r + 1) & 1];
// the round that processes a tile clears its mark.  In the host-driven loops only the CTAs
// the list needs take part (at least one, so every launched round is finalised), and the last
// of them consumes the list and advances the round number (device memory, ctl[CTL_RND]).
__device__ __forceinline__ int frontier_round_number(const PoolView& P, int first) {
  return first ? 0 : *((volatile int32_t*)&P.ctl[CTL_RND]);
}

// Work of this round: *count tiles (the selected tiles for a first round, the frontier list
// otherwise), *nranges the selection's ranges, and the number of CTAs that take part; CTAs
// beyond it return at once.  Called by every thread of the CTA.
__device__ __forceinline__ void frontier_work(const PoolView& P, int first, int in, int per_cta,
                                              int* count, int* participants, int* nranges) {
  __shared__ int s_n, s_nr;
  if (threadIdx.x == 0) {
    int n = first ? *((volatile int32_t*)&P.nsel[1]) : *((volatile int32_t*)&P.fcount[in]);
    int nr = *((volatile int32_t*)&P.nsel[0]);
    if (n < 0 || n > P.nt) {   // self-check: a list holds each tile at most once
      record_bad(P, 6, n);
      n = 0;
    }
    if (nr < 0 || nr > P.nimg) {   // self-check: one range per image at most
      record_bad(P, 9, nr);
      n = nr = 0;
    }
    s_n = n;
    s_nr = nr;
  }
  __syncthreads();
  const int n = s_n;
  *count = n;
  *nranges = s_nr;
  const int need = (n + per_cta - 1) / per_cta;
  *participants = need < 1 ? 1 : (need < (int)gridDim.x ? need : (int)gridDim.x);
}

// Queue tile t for the next round (once).  No look at the mark first: a round is a chain of L2
// trips, and the exchange answers as soon as a load would.
__device__ __forceinline__ void frontier_push(const PoolView& P, const Worklist& out, int t) {
  if (atomicExch(&out.in[t], 1) == 0) {
    const int pos = atomicAdd(out.count, 1);
    if (pos < P.nt) out.list[pos] = t;   // the mark deduplicates, so pos < nt always holds
    else record_bad(P, 5, pos);
    if (out.local) atomicAdd(out.local, 1);
  }
}

__device__ __forceinline__ void frontier_round_end(const PoolView& P, int first, int in,
                                                   int total_slot, int participants) {
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  const int d = atomicAdd(&P.ctl[CTL_DONE], 1);
  if (d != participants - 1) return;
  __threadfence();
  volatile int32_t* ctl = P.ctl;
  const int out = in ^ 1;
  const int next = *((volatile int32_t*)&P.fcount[out]);
  P.fcount[in] = 0;   // this round's list is consumed
  ctl[CTL_LASTCNT] = next;
  ctl[CTL_RND] = first ? 1 : ctl[CTL_RND] + 1;
  const int rounds = first ? 1 : ctl[CTL_ROUNDS] + 1;
  ctl[CTL_ROUNDS] = rounds;
  ctl[total_slot] = ctl[total_slot] + 1;
  ctl[CTL_DONE] = 0;
  const bool more = next > 0 && ctl[CTL_ERR] < 3;   // a copy or self-check error ends the loop
  if (more && rounds >= ctl[CTL_MAXROUNDS]) ctl[CTL_ERR] = 1;
  __threadfence();
}

// Solve prologue: reset the control words and the image stamps; the images of the
// selection take their mode for this solve and restart their flow sums (the others keep
// their results).  One CTA.
// Stamps of the host-driven loop: the floods are numbered, 1 the flood before the first
// pulses (only warm images), 2 + c the flood of cycle c; an image is live at the stamp of the
// next flood it takes part in.
__global__ void k_ctl_begin(PoolView P, int max_rounds, ImageAcc* acc) {
  trace_mark(P, TR_BEGIN);
  for (int i = threadIdx.x; i < CTL_N; i += blockDim.x) P.ctl[i] = 0;
  for (int i = threadIdx.x; i < P.nimg; i += blockDim.x) {
    P.img_live[i] = 0;
    P.img_hit[i] = 0;
    P.img_mode[i] = 0;
  }
  __syncthreads();
  const int nr = *((volatile int32_t*)&P.nsel[0]);
  for (int k = threadIdx.x; k < nr && k < P.nimg; k += blockDim.x) {
    const int img = P.sel[k].w;
    if ((unsigned)img >= (unsigned)P.nimg) continue;
    P.img_mode[img] = P.sel_mode[k];
    if (P.sel_mode[k] == 1) P.img_live[img] = 2;
    acc[img].sumpos_e = 0;   // the floods of this solve accumulate it
  }
  if (threadIdx.x == 0) {
    P.ctl[CTL_MAXROUNDS] = max_rounds;
    P.fcount[0] = 0;
    P.fcount[1] = 0;
  }
}

// The solve's results written straight into pinned host memory by k_solve, so no copy follows
// it: the control words, then the sums of the solve's images at their places in the host
// mirror (the other images' sums have not changed since their own solves).  One CTA calls it.
// The host reads the block only after synchronising with the solve's stream, which makes
// every write of the finished kernel visible to it, so no system-scope fence is needed.
__device__ __forceinline__ void publish_results(const PoolView& P, const ImageAcc* acc) {
  if (!P.host_out) return;
  constexpr int AW = (int)(sizeof(ImageAcc) / sizeof(int32_t));
  int nr = *((volatile int32_t*)&P.nsel[0]);
  nr = nr < 0 ? 0 : nr > P.nimg ? P.nimg : nr;
  const volatile int32_t* c = P.ctl;
  const volatile int32_t* a = reinterpret_cast<const volatile int32_t*>(acc);
  for (int i = threadIdx.x; i < CTL_N + AW * nr; i += blockDim.x) {
    if (i < CTL_N) {
      P.host_out[i] = c[i];
    } else {
      const int img = P.sel[(i - CTL_N) / AW].w, w = (i - CTL_N) % AW;
      if ((unsigned)img < (unsigned)P.nimg) P.host_out[CTL_N + AW * img + w] = a[AW * img + w];
    }
  }
}

// The active-tile list of the host-driven loop, in one launch: a single-pass scan (chunks by
// arrival ticket, decoupled look-back) of the activity flags of the selected tiles whose
// image is live at stamp `live` writes the ids of the active tiles in order.  fresh: the
// first list of a solve, in which freshly uploaded images follow fresh_tile_active.
//
// The grid is a fixed number of CTAs (a few per SM) that take chunk tickets in a loop until
// the selection's chunks run out, so a pool of millions of tiles costs no more launch work
// than one image.  Every ticket holder is already running, so a look-back only ever waits for
// a running CTA.
constexpr int ACT_THREADS = 256;
constexpr int ACT_ITEMS = 4;
constexpr int ACT_CHUNK = ACT_THREADS * ACT_ITEMS;

__global__ void __launch_bounds__(ACT_THREADS)
k_active_list(PoolView P, ScanState st, int32_t* list, int32_t* count, int live, int fresh) {
  trace_mark(P, TR_ACTIVE_LIST);
  __shared__ int32_t sm[32];
  __shared__ int32_t s_chunk, s_excl, s_n, s_nr;
  __shared__ uint32_t s_tag;
  if (threadIdx.x == 0) {
    s_chunk = atomicAdd(st.ticket, 1);
    s_tag = *((volatile uint32_t*)st.seq);
    int n = *((volatile int32_t*)&P.nsel[1]), nr = *((volatile int32_t*)&P.nsel[0]);
    if (n < 0 || n > P.nt || nr < 0 || nr > P.nimg) {   // self-check
      record_bad(P, 9, n);
      n = nr = 0;
    }
    s_n = n;
    s_nr = nr;
  }
  __syncthreads();
  const int n = s_n;
  const int nchunks = (n + ACT_CHUNK - 1) / ACT_CHUNK;
  for (int chunk = s_chunk; chunk < nchunks;) {
    const int base = chunk * ACT_CHUNK + threadIdx.x * ACT_ITEMS;
    SelCursor cursor(P, s_nr, base < n ? base : 0);
    int32_t v[ACT_ITEMS], tl[ACT_ITEMS];
    int32_t tsum = 0;
#pragma unroll
    for (int k = 0; k < ACT_ITEMS; ++k) {
      tl[k] = -1;
      v[k] = 0;
      if (base + k >= n) continue;
      tl[k] = cursor.tile(base + k);
      const int im = cursor.image();
      if ((unsigned)tl[k] >= (unsigned)P.nt || (unsigned)im >= (unsigned)P.nimg) {
        record_bad(P, 4, (unsigned)im < (unsigned)P.nimg ? tl[k] : im);
        continue;
      }
      if (P.img_live[im] != live) continue;
      v[k] = fresh && P.img_mode[im] == 1 ? fresh_tile_active(P, tl[k]) : P.tact[tl[k]] != 0;
      tsum += v[k];
    }
    int32_t agg;
    const int32_t tex = block_exclusive_scan(tsum, sm, &agg);
    if (threadIdx.x < 32) {
      const int32_t ex = lookback_exclusive_warp(st, s_tag, chunk, agg);
      if (threadIdx.x == 0) s_excl = ex;
    }
    __syncthreads();
    int32_t run = s_excl + tex;
#pragma unroll
    for (int k = 0; k < ACT_ITEMS; ++k) {
      if (!v[k]) continue;
      if ((unsigned)run < (unsigned)P.nt) list[run] = tl[k];
      else scan_error(st, 2);   // only after a look-back that gave up
      ++run;
    }
    if (chunk == nchunks - 1 && threadIdx.x == 0) *count = s_excl + agg;
    // the first tickets are 0 .. gridDim.x - 1: when they cover every chunk, none is left
    if ((int)gridDim.x >= nchunks) break;
    __syncthreads();   // every thread has read s_chunk and s_excl
    if (threadIdx.x == 0) s_chunk = atomicAdd(st.ticket, 1);
    __syncthreads();
    chunk = s_chunk;
  }
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(st.done, 1) != (int)gridDim.x - 1) return;
  // last CTA: close the scan (tickets, tag)
  __threadfence();
  *st.ticket = 0;
  *st.done = 0;
  uint32_t sq = *st.seq + 1;
  if ((sq & 0x3fffffffu) == 0) sq = 1;
  *st.seq = sq;
  volatile int32_t* ctl = P.ctl;
  if (nchunks == 0) *count = 0;
  ctl[CTL_PULSE] = 0;   // the list sits in queue[0]
  ctl[CTL_DDONE] = 0;
  P.qcount[1] = 0;
  ctl[CTL_NACT] = ctl[CTL_NACT] + 1;
  // a look-back that gave up (here or in an earlier list of this solve) reaches the host
  // with the control words
  ctl[CTL_SCANERR] = ctl[CTL_SCANERR] | *((volatile int32_t*)st.err);
  __threadfence();
}

// After the active-tile compaction of a manual step: the list becomes the first worklist.
__global__ void k_ctl_cycle(PoolView P) {
  if (threadIdx.x != 0) return;
  volatile int32_t* ctl = P.ctl;
  ctl[CTL_PULSE] = 0;   // the compacted list sits in queue[0]
  ctl[CTL_DDONE] = 0;
  P.qcount[1] = 0;
  __threadfence();
}

// ---- distances as bit planes --------------------------------------------------------
// The distances of a tile above its lowest seed (`base`) mostly fit in BFS_PLANES bits.  Lane r
// keeps bit b of those of row r in plane[b], so a level costs a few logic operations instead of
// a store per pixel, and the rows are turned into int4 stores once at the end.  Tiles with a
// seed further out than BFS_RANGE above their lowest fall back on tile_bfs_seeded.
constexpr int BFS_PLANES = 8;
constexpr int BFS_RANGE = (1 << BFS_PLANES) - 1;
constexpr int BFS_GROUP = 2;   // levels a vote

struct PlaneBfs {
  int base;                      // lowest level
  uint32_t vis;                  // reached pixels of row `lane`
  uint32_t plane[BFS_PLANES];    // their distances above base (0 where not reached)
  bool whole;                    // false: levels beyond base + BFS_RANGE are missing
  // distances of row `lane`'s pixel at column c (0 or 31)
  __device__ __forceinline__ int side(int c) const {
    int d = base;
#pragma unroll
    for (int b = 0; b < BFS_PLANES; ++b) d += (int)((plane[b] >> c) & 1u) << b;
    return (vis >> c) & 1u ? d : GC_HINF;
  }
  // distance of column `lane`'s pixel in row `row` (uniform)
  __device__ __forceinline__ int across(int row, int lane) const {
    int d = base;
#pragma unroll
    for (int b = 0; b < BFS_PLANES; ++b)
      d += (int)((__shfl_sync(0xffffffffu, plane[b], row) >> lane) & 1u) << b;
    return (__shfl_sync(0xffffffffu, vis, row) >> lane) & 1u ? d : GC_HINF;
  }
};

// tile_bfs_seeded on bit planes.  A level is a chain of a shuffle and three logic operations
// (40 cycles); the vote on an empty frontier would double it, so BFS_GROUP levels share one (a
// level without a frontier or a seed visits nothing).  A frontier round of a few tiles takes 11 us
// at a cap of 64 and 15 us without one (13 with a vote a level, 22 with a store per pixel); of
// that 7 us are its chain of L2 trips and the barrier.  (4 levels a vote: the same, more spills;
// 7 planes: the same up to 127, slower beyond.)
__device__ __forceinline__ PlaneBfs tile_bfs_planes(uint32_t sink, uint32_t canU, uint32_t canD,
                                                    uint32_t canL, uint32_t canR, int lane,
                                                    bool seeded, int top, int bot, int sl, int sr,
                                                    int cap) {
  const unsigned FULL = 0xffffffffu;
  PlaneBfs B;
  B.vis = 0;
  B.whole = true;
#pragma unroll
  for (int b = 0; b < BFS_PLANES; ++b) B.plane[b] = 0;
  uint32_t Fr = 0, over = 0;
  if (lane == 0) canU = 0;     // the row above / below lies in another tile (seeds stand for it)
  if (lane == 31) canD = 0;
  int L = 0;
  if (!__any_sync(FULL, sink != 0)) L = seeded ? warp_min(imin(imin(top, bot), imin(sl, sr))) : GC_HINF;
  B.base = L;
  const int lim = imin(cap, GC_HINF - 1);
  const int last = L <= lim - BFS_RANGE ? L + BFS_RANGE : lim;
  // L rises by BFS_GROUP or jumps to a later seed
  while (L <= last) {
#pragma unroll
    for (int k = 0; k < BFS_GROUP; ++k, ++L) {
      uint32_t N = ((Fr >> 1) & canR) | ((Fr << 1) & canL) | (__shfl_up_sync(FULL, Fr, 1) & canU) |
                   (__shfl_down_sync(FULL, Fr, 1) & canD);
      if (k == 0 && L == 0) N |= sink;
      if (seeded) {
        const uint32_t bt = __ballot_sync(FULL, top == L), bb = __ballot_sync(FULL, bot == L);
        N |= (sl == L ? 1u : 0u) | (sr == L ? 0x80000000u : 0u);
        if (lane == 0) N |= bt;
        if (lane == 31) N |= bb;
      }
      N &= ~B.vis;
      if (L > last) {   // too far out to hold
        over |= N;
        N = 0;
      }
      B.vis |= N;
      const int d = L - B.base;
#pragma unroll
      for (int b = 0; b < BFS_PLANES; ++b) B.plane[b] |= (d >> b) & 1 ? N : 0u;
      Fr = N;
    }
    if (__any_sync(FULL, Fr != 0)) continue;
    if (L > last + 1 && __any_sync(FULL, over != 0)) break;
    if (!seeded) return B;
    // the frontier is empty: the next level that still has an unvisited seed
    const uint32_t v0 = __shfl_sync(FULL, B.vis, 0), v31 = __shfl_sync(FULL, B.vis, 31);
    int cand = GC_HINF;
    if (!((v0 >> lane) & 1u)) cand = imin(cand, top);
    if (!((v31 >> lane) & 1u)) cand = imin(cand, bot);
    if (!(B.vis & 1u)) cand = imin(cand, sl);
    if (!(B.vis >> 31)) cand = imin(cand, sr);
    L = warp_min(cand);
    if (L > lim) return B;
  }
  // something lies beyond `last`: beyond the cap, or only beyond the planes' range
  B.whole = last == lim;
  return B;
}

// The four low bits of x in the low bits of four bytes.
__device__ __forceinline__ uint32_t spread4(uint32_t x) { return ((x & 15u) * 0x00204081u) & 0x01010101u; }

// One tile of a global relabel, by one warp: the in-tile BFS seeded by the tile's sink pixels
// and (frontier rounds) the halo distances, the heights written back, and the neighbours queued
// that a changed edge distance could lower.  T: the warp's 32 x 33 words of shared memory (used
// where distances span more than BFS_RANGE only).  Returns whether the tile holds an active pixel (-1: nothing
// changed since the tile's last round).
//
// Bound by latency and by the 4 KiB of heights a tile stores.  So: a tile whose heights are all
// 0 or all unreached, and were so before, stores nothing (hstate; most tiles of a large image);
// a frontier tile none of whose seeds is below its edge's distance stops after 8 loads; and a
// neighbour is queued only if one of its edge pixels has a residual edge into a changed pixel
// and is no sink itself (in the first round nearly every tile used to queue all four).
__device__ __forceinline__ int bfs_tile(const PoolView& P, int t, int lane, int first, int cap,
                                        int32_t* T, const Worklist& out) {
  const unsigned FULL = 0xffffffffu;
  const int4 nb = P.nbr[t];
  const long long base = (long long)t * GC_TILE_PX;
  // the masks are current: the flood that precedes every global relabel of a solve (or
  // k_masks, before gc_start_bfs) rebuilt every tile that changed since they were written
  const uint32_t* mc = P.mcan + (long long)t * 128;
  const uint32_t canU = mc[lane], canD = mc[32 + lane], canL = mc[64 + lane], canR = mc[96 + lane];
  const uint32_t sink = P.msink[(long long)t * 32 + lane];
  const uint32_t pos = P.mexc[(long long)t * 32 + lane];
  // edge pixels of the neighbours that a distance of this tile could lower (a word over the
  // columns for up and down; a flag of this lane's row for left and right)
  uint32_t wantU = 0, wantD = 0, wantL = 0, wantR = 0;
  if (nb.x >= 0) wantU = P.mcan[(long long)nb.x * 128 + 32 + 31] & ~P.msink[(long long)nb.x * 32 + 31];
  if (nb.y >= 0) wantD = P.mcan[(long long)nb.y * 128] & ~P.msink[(long long)nb.y * 32];
  if (nb.z >= 0) wantL = (P.mcan[(long long)nb.z * 128 + 96 + lane] & ~P.msink[(long long)nb.z * 32 + lane]) >> 31;
  if (nb.w >= 0) wantR = P.mcan[(long long)nb.w * 128 + 64 + lane] & ~P.msink[(long long)nb.w * 32 + lane] & 1u;
  // seeds from the neighbour tiles' heights (frontier rounds only): an edge pixel with a
  // residual edge into the neighbour starts at the neighbour's height + 1
  int top = GC_HINF, bot = GC_HINF, sl = GC_HINF, sr = GC_HINF;
  int oT = GC_HINF, oB = GC_HINF, oL = GC_HINF, oR = GC_HINF;   // this tile's edges before
  if (!first) {
    const uint32_t cu0 = __shfl_sync(FULL, canU, 0);
    const uint32_t cd31 = __shfl_sync(FULL, canD, 31);
    const int vu = nb.x >= 0 ? P.hgt[(long long)nb.x * GC_TILE_PX + 31 * GC_TILE + lane] : GC_HINF;
    const int vd = nb.y >= 0 ? P.hgt[(long long)nb.y * GC_TILE_PX + lane] : GC_HINF;
    const int vl = nb.z >= 0 ? P.hgt[(long long)nb.z * GC_TILE_PX + lane * GC_TILE + 31] : GC_HINF;
    const int vr = nb.w >= 0 ? P.hgt[(long long)nb.w * GC_TILE_PX + lane * GC_TILE] : GC_HINF;
    oT = P.hgt[base + lane];
    oB = P.hgt[base + 31 * GC_TILE + lane];
    oL = P.hgt[base + lane * GC_TILE];
    oR = P.hgt[base + lane * GC_TILE + 31];
    if (((cu0 >> lane) & 1u) && vu < GC_HINF) top = vu + 1;
    if (((cd31 >> lane) & 1u) && vd < GC_HINF) bot = vd + 1;
    if ((canL & 1u) && vl < GC_HINF) sl = vl + 1;
    if ((canR >> 31) && vr < GC_HINF) sr = vr + 1;
    const int lim = imin(cap, GC_HINF - 1);
    if (!__any_sync(FULL, (top < oT && top <= lim) || (bot < oB && bot <= lim) ||
                              (sl < oL && sl <= lim) || (sr < oR && sr <= lim)))
      return -1;
  }
  int nT, nB, nL, nR;   // the edges now
  int state = 0;        // hstate: 1 all 0, 2 all unreached, 0 neither
  const PlaneBfs B = tile_bfs_planes(sink, canU, canD, canL, canR, lane, !first, top, bot, sl, sr, cap);
  uint32_t fin = B.vis;
  if (B.whole) {
    uint32_t any = 0;
#pragma unroll
    for (int b = 0; b < BFS_PLANES; ++b) any |= B.plane[b];
    if (B.base == 0 && __all_sync(FULL, fin == FULL && any == 0)) state = 1;
    else if (__all_sync(FULL, fin == 0)) state = 2;
    nT = B.across(0, lane);
    nB = B.across(31, lane);
    nL = B.side(0);
    nR = B.side(31);
    if (state == 0 || P.hstate[t] != state) {
      const int q = lane & 7;
#pragma unroll 2
      for (int k = 0; k < 8; ++k) {   // rows 4k .. 4k+3; this lane: four pixels of row 4k + lane / 8
        const int src = 4 * k + (lane >> 3);
        uint32_t d4 = 0;
#pragma unroll
        for (int b = 0; b < BFS_PLANES; ++b)
          d4 |= spread4(__shfl_sync(FULL, B.plane[b], src) >> (4 * q)) << b;
        const uint32_t f4 = __shfl_sync(FULL, B.vis, src) >> (4 * q);
        const int4 v = make_int4(f4 & 1u ? B.base + (int)(d4 & 255u) : GC_HINF,
                                 f4 & 2u ? B.base + (int)((d4 >> 8) & 255u) : GC_HINF,
                                 f4 & 4u ? B.base + (int)((d4 >> 16) & 255u) : GC_HINF,
                                 f4 & 8u ? B.base + (int)(d4 >> 24) : GC_HINF);
        *(int4*)(P.hgt + base + src * GC_TILE + 4 * q) = v;
      }
    }
  } else {
    fin = tile_bfs_seeded(T + lane * 33, sink, canU, canD, canL, canR, lane, top, bot, sl, sr, cap);
    __syncwarp();
    for (int rr = 0; rr < 32; ++rr) P.hgt[base + rr * GC_TILE + lane] = T[rr * 33 + lane];
    nT = T[lane];
    nB = T[31 * 33 + lane];
    nL = T[lane * 33];
    nR = T[lane * 33 + 31];
    __syncwarp();
  }
  if (lane == 0) P.hstate[t] = state;
  const int chU = __any_sync(FULL, nT < oT && ((wantU >> lane) & 1u));
  const int chD = __any_sync(FULL, nB < oB && ((wantD >> lane) & 1u));
  const int chL = __any_sync(FULL, nL < oL && wantL);
  const int chR = __any_sync(FULL, nR < oR && wantR);
  const int act = __any_sync(FULL, (pos & fin) != 0);
  // the neighbours to queue, one lane each (their atomics run in parallel)
  if (lane < 4) {
    const int go = lane == 0 ? chU : lane == 1 ? chD : lane == 2 ? chL : chR;
    const int nt = lane == 0 ? nb.x : lane == 1 ? nb.y : lane == 2 ? nb.z : nb.w;
    if (go && nt >= 0) frontier_push(P, out, nt);
  }
  return act;
}

__global__ void __launch_bounds__(WARPS_PER_CTA * 32)
k_bfs_round(PoolView P, int first, int cap, int live) {
  trace_mark(P, first ? TR_BFS_FIRST : TR_BFS);
  __shared__ int32_t tr[WARPS_PER_CTA][32 * 33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int in = frontier_round_number(P, first) & 1;
  const Worklist out{P.fq[in ^ 1], P.fcount + (in ^ 1), P.mark[in ^ 1]};
  int32_t* const markin = P.mark[in];
  int done = 0;
  // first == 2: a global relabel inside the solve loop covers the images live at stamp `live`
  int n, parts, nr;
  frontier_work(P, first, in, WARPS_PER_CTA, &n, &parts, &nr);
  if ((int)blockIdx.x >= parts) return;
  const int i0 = blockIdx.x * WARPS_PER_CTA + warp;
  SelCursor cursor(P, first ? nr : 0, i0);
  for (int i = i0; i < n; i += parts * WARPS_PER_CTA) {
    const int t = first ? cursor.tile(i) : P.fq[in][i];
    if (!first) {
      if (lane == 0) markin[t] = 0;
    } else {
      if (first == 2) {
        const int img = P.img_of[t];
        if ((unsigned)img >= (unsigned)P.nimg) {   // self-check
          if (lane == 0) record_bad(P, 4, img);
          continue;
        }
        if (P.img_live[img] != live) continue;
      }
      if (lane == 0) {
        P.inq[0][t] = 0;  // the worklists are rebuilt from the relabelled state
        P.inq[1][t] = 0;
      }
    }
    ++done;
    const int act = bfs_tile(P, t, lane, first, cap, tr[warp], out);
    if (lane == 0 && act >= 0) P.tact[t] = act;
  }
  if (lane == 0 && done && P.ktiles)
    atomicAdd(&P.ktiles[first ? K_BFS_FIRST : K_BFS], (unsigned long long)done);
  frontier_round_end(P, first, in, CTL_BFS_TOTAL, parts);
}

// After a flood of the host-driven loop: an image whose flood reached no sink pixel is solved
// (its flood is the canonical cut, its sums are final) and leaves the live set; the others go
// on to a global relabel, live at stamp + 1, with their sums and sink-reached stamps cleared.
// all != 0: the images that continue from a previous flow (img_mode == 2; the first check of
// a solve); else the images live at `stamp`.  One CTA.
__global__ void k_flood_check(PoolView P, int all, int stamp, ImageAcc* acc) {
  __shared__ int s_left;
  if (threadIdx.x == 0) {
    s_left = 0;
    trace_record(P, TR_CHECK);
  }
  __syncthreads();
  volatile int32_t* ctl = P.ctl;
  int left = 0;
  for (int i = threadIdx.x; i < P.nimg; i += blockDim.x) {
    const bool part = all ? *((volatile int32_t*)&P.img_mode[i]) == 2
                          : *((volatile int32_t*)&P.img_live[i]) == stamp;
    if (!part) continue;
    if (*((volatile int32_t*)&P.img_hit[i]) == stamp) {
      P.img_live[i] = stamp + 1;
      P.img_hit[i] = 0;
      acc[i].sumpos_e = 0;
      ++left;
    } else {
      P.img_live[i] = 0;   // solved: no later stamp equals 0
    }
  }
  if (left) atomicAdd(&s_left, left);
  __syncthreads();
  if (threadIdx.x != 0) return;
  int n = s_left;
  if (ctl[CTL_ERR] != 0) n = 0;   // a cap or a self-check ends the loops
  ctl[CTL_LEFT] = n;
  ctl[CTL_NCHECK] = ctl[CTL_NCHECK] + 1;
  if (n == 0) trace_record(P, TR_END);
}

// ------------------------------------------------------------------------------------
// Canonical cut: flood from excess pixels over residual edges (forward direction).
// The first flood round also sums max(excess, 0) per image for the flow value.
//
// The flood also decides termination: an excess pixel can reach a sink pixel exactly when
// the flood from the excess pixels reaches one, so an image whose flood reaches no sink
// pixel is solved (its flood is the canonical cut) and one whose flood does needs another
// global relabel and push cycle.  Every round stamps img_hit[img] with the flood's stamp
// when a tile's reached set meets its sink pixels.
// ------------------------------------------------------------------------------------
// Sum of max(excess, 0) of the tiles a warp has flooded, added to an image's word when the
// image changes (flood_sum_flush adds the rest, once per image and CTA).
struct FloodSum {
  int img = -1;
  unsigned long long sum = 0;
  __device__ __forceinline__ void add(ImageAcc* acc, int i, long long v) {
    if (i != img) {
      if (sum) atomicAdd(&acc[img].sumpos_e, sum);
      img = i;
      sum = 0;
    }
    sum += (unsigned long long)v;
  }
};

// The masks a warp floods a tile with: lane = row.
struct TileMasks { uint32_t canU, canD, canL, canR, sink, exc; };

__device__ __forceinline__ TileMasks load_masks(const PoolView& P, int t, int lane) {
  const uint32_t* mc = P.mcan + (long long)t * 128;
  return TileMasks{mc[lane], mc[32 + lane], mc[64 + lane], mc[96 + lane],
                   P.msink[(long long)t * 32 + lane], P.mexc[(long long)t * 32 + lane]};
}

// Everything in a row that the pixels of R reach to the right over the edges M (bit x: x to
// x + 1): the carry of (R & M) + M runs through each run of edges from its lowest seed to the
// pixel after its end.  (A seed inside the run flips back, but is in R.)
__device__ __forceinline__ uint32_t fill_up_bits(uint32_t R, uint32_t M) { return R | (((R & M) + M) ^ M); }

// Floods tile t from R (which it extends) inside the tile, by one warp; writes the reached set,
// stamps the image when it meets a sink, and queues the neighbours it reaches into.  R0: the
// reached set before (0 in a first round).  hits: counts the images whose stamp this flood
// sets (null: not counted).
__device__ __forceinline__ void flood_fill(const PoolView& P, int t, int4 nb, int lane, int img,
                                           int stamp, const TileMasks& m, uint32_t R, uint32_t R0,
                                           int32_t* hits, const Worklist& out) {
  const unsigned FULL = 0xffffffffu;
  const uint32_t toDown = lane == 31 ? 0u : m.canD, toUp = lane == 0 ? 0u : m.canU;
  const uint32_t leftRev = __brev(m.canL);
  // every step reaches at least one pixel more; rows fill at once
  for (int guard = 0; guard < GC_TILE_PX + 1; ++guard) {
    uint32_t dn = __shfl_up_sync(FULL, R & toDown, 1);   // row r-1 flows down into r
    uint32_t up = __shfl_down_sync(FULL, R & toUp, 1);   // row r+1 flows up into r
    if (lane == 0) dn = 0;
    if (lane == 31) up = 0;
    uint32_t N = R | dn | up;
    N = fill_up_bits(N, m.canR);
    N = __brev(fill_up_bits(__brev(N), leftRev));
    if (!__any_sync(FULL, N != R)) break;
    R = N;
  }
  P.mreach[(long long)t * 32 + lane] = R;
  if (__any_sync(FULL, (R & m.sink) != 0) && lane == 0 &&
      *((volatile int32_t*)&P.img_hit[img]) != stamp) {
    if (!hits) P.img_hit[img] = stamp;
    else if (atomicExch(&P.img_hit[img], stamp) != stamp) atomicAdd(hits, 1);
  }
  const uint32_t nw = R & ~R0;
  const int sU = __any_sync(FULL, lane == 0 && (nw & m.canU));
  const int sD = __any_sync(FULL, lane == 31 && (nw & m.canD));
  const int sL = __any_sync(FULL, (nw & m.canL & 1u) != 0);
  const int sR = __any_sync(FULL, ((nw & m.canR) >> 31) != 0);
  if (lane < 4) {   // the neighbours to queue, one lane each
    const int go = lane == 0 ? sU : lane == 1 ? sD : lane == 2 ? sL : sR;
    const int nt = lane == 0 ? nb.x : lane == 1 ? nb.y : lane == 2 ? nb.z : nb.w;
    if (go && nt >= 0) frontier_push(P, out, nt);
  }
}

// One tile of a frontier round: what it had reached, and what the neighbours' reached sets
// reach across its sides.
__device__ __forceinline__ void flood_frontier_tile(const PoolView& P, int t, int lane, int img,
                                                    int stamp, int32_t* hits, const Worklist& out) {
  const int4 nb = P.nbr[t];
  const TileMasks m = load_masks(P, t, lane);
  const uint32_t R0 = P.mreach[(long long)t * 32 + lane];
  uint32_t R = R0;
  if (lane == 0 && nb.x >= 0)
    R |= P.mreach[(long long)nb.x * 32 + 31] & P.mcan[(long long)nb.x * 128 + 32 + 31];
  if (lane == 31 && nb.y >= 0)
    R |= P.mreach[(long long)nb.y * 32] & P.mcan[(long long)nb.y * 128 + 0];
  if (nb.z >= 0 && ((P.mreach[(long long)nb.z * 32 + lane] & P.mcan[(long long)nb.z * 128 + 96 + lane]) >> 31))
    R |= 1u;
  if (nb.w >= 0 && ((P.mreach[(long long)nb.w * 32 + lane] & P.mcan[(long long)nb.w * 128 + 64 + lane]) & 1u))
    R |= 0x80000000u;
  if (!__any_sync(0xffffffffu, R != R0)) return;   // nothing new comes in
  flood_fill(P, t, nb, lane, img, stamp, m, R, R0, hits, out);
}

// One tile of a first round, by one warp; a tile that changed since its masks were written (a
// discharge or an edit) gets them rebuilt first, before anything reads them (every tile of an
// image a first round covers is done in it, so the frontier rounds and the global relabel
// after it see them).
__device__ __forceinline__ void flood_first_tile(const PoolView& P, int t, int lane, int img,
                                                 int stamp, const Worklist& out, ImageAcc* acc,
                                                 FloodSum& fs) {
  const int4 nb = P.nbr[t];
  TileMasks m;
  long long ps = 0;
  if (P.mdirty[t] != 0) {
    const RowMasks rm = warp_rebuild_masks(P, t, lane, &ps);
    m = TileMasks{rm.up, rm.down, rm.left, rm.right, rm.sink, rm.exc};
  } else {
    m = load_masks(P, t, lane);
    ps = P.tpos[t];
  }
  if (lane == 0 && ps) fs.add(acc, img, ps);   // taken with the tile's masks
  flood_fill(P, t, nb, lane, img, stamp, m, m.exc, 0, nullptr, out);
}

// The CTA's warps add their sums, once per image.  Every thread of the CTA calls it.
template <int WARPS>
__device__ __forceinline__ void flood_sum_flush(ImageAcc* acc, const FloodSum& fs) {
  __shared__ int s_img[WARPS];
  __shared__ unsigned long long s_sum[WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s_img[warp] = fs.sum ? fs.img : -1;
    s_sum[warp] = fs.sum;
  }
  __syncthreads();
  if (warp == 0) {   // lane a: the sum of the warps that hold warp a's image, added by the first
    const int mine = lane < WARPS ? s_img[lane] : -1;
    const unsigned long long v = lane < WARPS ? s_sum[lane] : 0ull;
    unsigned long long total = 0;
    bool first = true;
#pragma unroll
    for (int b = 0; b < WARPS; ++b) {
      const bool same = __shfl_sync(0xffffffffu, mine, b) == mine;
      const unsigned long long x = __shfl_sync(0xffffffffu, v, b);
      if (same) total += x;
      if (same && b < lane) first = false;
    }
    if (lane < WARPS && mine >= 0 && first) atomicAdd(&acc[mine].sumpos_e, total);
  }
}

// A flood round of the host-driven loop.  mode: 0 frontier round; first rounds over the
// selected tiles: 1 all of them, 2 those of the images live in this cycle (img_live ==
// the flood's stamp), 3 those of the images that continue from a previous flow (img_mode == 2).
// abort_hit: frontier rounds skip the tiles of images already stamped (their flood is redone
// in a later cycle).
__global__ void __launch_bounds__(WARPS_PER_CTA * 32)
k_flood_round(PoolView P, int mode, int abort_hit, int stamp, ImageAcc* acc) {
  trace_mark(P, mode ? TR_FLOOD_FIRST : TR_FLOOD);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = mode != 0;
  const int in = frontier_round_number(P, first) & 1;
  const Worklist out{P.fq[in ^ 1], P.fcount + (in ^ 1), P.mark[in ^ 1]};
  int32_t* const markin = P.mark[in];
  int done = 0;
  int n, parts, nr;
  frontier_work(P, first, in, WARPS_PER_CTA, &n, &parts, &nr);
  if ((int)blockIdx.x >= parts) return;
  const int i0 = blockIdx.x * WARPS_PER_CTA + warp;
  SelCursor cursor(P, first ? nr : 0, i0);
  FloodSum fs;
  for (int i = i0; i < n; i += parts * WARPS_PER_CTA) {
    const int t = first ? cursor.tile(i) : P.fq[in][i];
    if (!first && lane == 0) markin[t] = 0;
    const int img = P.img_of[t];
    if ((unsigned)img >= (unsigned)P.nimg) {   // self-check
      if (lane == 0) record_bad(P, 4, img);
      continue;
    }
    if (mode == 2 && P.img_live[img] != stamp) continue;
    if (mode == 3 && P.img_mode[img] != 2) continue;
    if (mode == 0 && abort_hit && *((volatile int32_t*)&P.img_hit[img]) == stamp) continue;
    ++done;
    if (first) flood_first_tile(P, t, lane, img, stamp, out, acc, fs);
    else flood_frontier_tile(P, t, lane, img, stamp, nullptr, out);
  }
  if (lane == 0 && done && P.ktiles)
    atomicAdd(&P.ktiles[first ? K_FLOOD_FIRST : K_FLOOD], (unsigned long long)done);
  if (first) flood_sum_flush<WARPS_PER_CTA>(acc, fs);
  frontier_round_end(P, first, in, CTL_FLOOD_TOTAL, parts);
}

// Neighbour tile ids and image index of one image's tiles (row-major from im.tile0), for an
// image placed in a session pool.
__global__ void k_image_tiles(PoolView P, ImageDesc im, int img) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= im.tw * im.th) return;
  const int tx = k % im.tw, ty = k / im.tw, t = im.tile0 + k;
  P.nbr[t] = make_int4(ty > 0 ? t - im.tw : -1, ty < im.th - 1 ? t + im.tw : -1,
                       tx > 0 ? t - 1 : -1, tx < im.tw - 1 ? t + 1 : -1);
  P.img_of[t] = img;
}

// Labels of one image, row-major, padding excluded: threads i0, i0 + stride, ... each write the
// 32 pixels of a tile row (one mask word); consecutive threads take consecutive tiles of an
// image row.
__device__ __forceinline__ void write_labels(const PoolView& P, const ImageDesc& im, uint8_t* out,
                                             long long i0, long long stride) {
  const long long n = (long long)im.H * im.tw;
  for (long long i = i0; i < n; i += stride) {
    const int y = (int)(i / im.tw), tx = (int)(i % im.tw);
    const int t = im.tile0 + (y >> 5) * im.tw + tx;
    const uint32_t m = P.mreach[(long long)t * 32 + (y & 31)];
    const int x0 = tx * GC_TILE;
    uint8_t* row = out + (long long)y * im.W + x0;
    if (x0 + GC_TILE <= im.W && (((uintptr_t)row) & 3) == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t b = (m >> (4 * k)) & 0xfu;
        const uint32_t w = (b & 1u) | ((b & 2u) << 7) | ((b & 4u) << 14) | ((b & 8u) << 21);
        reinterpret_cast<uint32_t*>(row)[k] = w;
      }
    } else {
      for (int c = 0; c < GC_TILE && x0 + c < im.W; ++c) row[c] = (uint8_t)((m >> c) & 1u);
    }
  }
}

// Bit-packed labels: thread (y, tx) writes the up to four bytes of tile column tx in row y
// (row stride (W + 7) / 8 bytes, little bit order).  Pixels of a ragged tile beyond the
// image have no capacities and no excess, so their reach bits are 0.
__device__ __forceinline__ void write_labels_packed(const PoolView& P, const ImageDesc& im,
                                                    uint8_t* out, long long i0, long long step) {
  const long long n = (long long)im.H * im.tw;
  const int stride = (im.W + 7) >> 3;
  for (long long i = i0; i < n; i += step) {
    const int y = (int)(i / im.tw), tx = (int)(i % im.tw);
    const int t = im.tile0 + (y >> 5) * im.tw + tx;
    const uint32_t m = P.mreach[(long long)t * 32 + (y & 31)];
    uint8_t* row = out + (long long)y * stride + 4 * tx;
    const int nb = stride - 4 * tx < 4 ? stride - 4 * tx : 4;
    if (nb == 4 && (((uintptr_t)row) & 3) == 0) {
      *reinterpret_cast<uint32_t*>(row) = m;
    } else {
      for (int k = 0; k < nb; ++k) row[k] = (uint8_t)(m >> (8 * k));
    }
  }
}

__global__ void k_labels_out(PoolView P, ImageDesc im, uint8_t* out) {
  trace_mark(P, TR_LABELS);
  write_labels(P, im, out, (long long)blockIdx.x * blockDim.x + threadIdx.x,
               (long long)gridDim.x * blockDim.x);
}
__global__ void k_labels_packed(PoolView P, ImageDesc im, uint8_t* out) {
  trace_mark(P, TR_LABELS);
  write_labels_packed(P, im, out, (long long)blockIdx.x * blockDim.x + threadIdx.x,
                      (long long)gridDim.x * blockDim.x);
}

// ------------------------------------------------------------------------------------
// The whole solve as one cooperative launch: every CTA runs the same steps (pulses, flood
// rounds, relabel rounds), with a grid barrier after each.
//
// Bound by latency: a step of a few tiles is its barrier (1.5 us), a chain of L2 trips and one
// tile's work, and a solve is 5 to 30 such steps (hundreds on the hardest grids); the pulses of
// large grids are bound by the ALU pipe (integer minima and selects run at half rate).  As a
// CUDA graph (the same steps as kernel nodes under WHILE and IF nodes) each step paid a launch
// and a drain, and 5-11 us per conditional node: 256x192 98-169 us from upload to labels against
// 35-71 now, 2048x2048 300-690 against 145-230, strokes at 4096x4096 210-650 against 112-123.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier and step change: every CTA's writes before it are visible to every CTA after
// it, its bulk copies included, and `s` holds the next step.  The CTAs' counts of queued tiles
// travel in the arrival word, so the loop decision needs no second trip to L2 (0.35 us).  What
// the CTAs read of a full word is the same.  A wait gives up after bar_wait_ns: it raises the
// abort flag, and every CTA leaves at its next barrier.  A solve that was aborted ends.
__device__ __forceinline__ void solve_barrier(const PoolView& P, const SolveArgs& A, SolveState& s) {
  // this thread's writes to the planes, before later bulk copies (a flood writes none)
  if (s.step != ST_FLOOD_FIRST && s.step != ST_FLOOD) asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long* const word = P.bar + BAR_ARRIVE + (int)(s.bar & 1) * BAR_STRIDE;
    __threadfence();
    atomicAdd(word, bar_add(s, blockIdx.x == 0));
    bool ok = false;
    unsigned long long t0 = 0, v = 0;
    for (unsigned i = 1; i < (1u << 31); ++i) {
      v = ld_acquire(word);
      if (v & GC_BAR_ABORT) break;
      if (bar_full(s, gridDim.x, v)) { ok = true; break; }
      if ((i & 1023u) == 0) {
        const unsigned long long now = global_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > bar_wait_ns(s, gridDim.x)) {
          atomicCAS(&P.ctl[CTL_ERR], 0, 5);
          __threadfence();
          abort_solve(P);
          break;
        }
      }
    }
    __threadfence();
    asm volatile("fence.proxy.async;" ::: "memory");
    if (!ok) {
      s.err = 5;
      s.step = ST_END;
    } else {
      const int total = (int)bar_pass(s, gridDim.x, v), was = s.step;
      next_step(P.ctl, P.nt, A, s, total);
      if (blockIdx.x == 0 && total == 0 && (was == ST_FLOOD_FIRST || was == ST_FLOOD)) trace_record(P, TR_CHECK);
      if (s.err == 4) record_bad(P, 6, total);
    }
  }
  __syncthreads();
}

constexpr int SOLVE_WARPS = DIS_THREADS / 32;

// The first round of a flood in k_solve: SOLVE_WARPS tiles of the selection at a time, a warp
// per tile.  The tiles among them that changed since their masks were written are rebuilt
// first: up to REB_SPLIT by the whole CTA, one after another with the next one's loads in
// flight (5 vector loads a thread and tile, one trip to L2), more by a warp each (a chain of
// trips, but all tiles at once).  Over 48 tiles, one per CTA, the round takes 6.7 us against
// 9.2 with a warp per tile; over 4096 tiles with three to five changed ones per CTA the whole
// CTA took 26 us where the warps take 18.
// sm: SOLVE_WARPS x REB_WORDS (6 x 32 words of masks, 2 x 8 half sums).
constexpr int REB_WORDS = 6 * 32 + 2 * SOLVE_WARPS;
constexpr int REB_SPLIT = 2;

__device__ __forceinline__ void flood_first_phase(const PoolView& P, const SolveArgs& A,
                                                  SolveState& st, uint32_t* sm) {
  __shared__ int s_dt[2][SOLVE_WARPS];
  const unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bid = blockIdx.x, nb_ctas = gridDim.x, n = A.tiles;
  const int stamp = st.stamp, prev = st.prev, cyc = st.cyc;
  int32_t* const hits = &P.ctl[CTL_H0 + stamp % 3];
  const Worklist out{(st.fk & 1) ? P.fq[0] : P.fq[1], &P.ctl[CTL_F0 + (st.fk + 1) % 3],
                     (st.fk & 1) ? P.mark[0] : P.mark[1], &st.push};
  const int i0 = warp * nb_ctas + bid;
  SelCursor cursor(P, A.ranges, i0 < n ? i0 : 0, A.sel0);
  FloodSum fs;
  int par = 0;
  for (int b = 0; b < n; b += SOLVE_WARPS * nb_ctas, par ^= 1) {   // the same for every warp
    const int i = b + i0;
    int t = -1, img = 0, dirty = 0;
    int4 nb = make_int4(-1, -1, -1, -1);
    TileMasks m{0u, 0u, 0u, 0u, 0u, 0u};
    long long ps = 0;
    if (i < n) {
      t = cursor.tile(i);
      img = cursor.image();
      if ((unsigned)img >= (unsigned)P.nimg || (unsigned)t >= (unsigned)P.nt) {   // self-check
        if (lane == 0) record_bad(P, 4, img);
        t = -1;
      } else {
        // all loads before the first decision
        const int hit = *((volatile int32_t*)&P.img_hit[img]);
        const int mode = A.ranges == 1 ? A.mode0 : P.sel_mode[cursor.range()];
        dirty = P.mdirty[t];
        nb = P.nbr[t];
        m = load_masks(P, t, lane);
        ps = P.tpos[t];
        const bool part = cyc == 0 ? mode == 2
                                   : (hit == stamp || (prev > 0 && hit == prev) || (cyc == 1 && mode == 1));
        if (!part) t = -1;
      }
    }
    if (t < 0) dirty = 0;
    if (lane == 0) s_dt[par][warp] = dirty ? t : -1;
    const int ndirty = __syncthreads_count(dirty && lane == 0);
    if (ndirty > REB_SPLIT) {
      if (dirty) {
        const RowMasks rm = warp_rebuild_masks(P, t, lane, &ps);
        m = TileMasks{rm.up, rm.down, rm.left, rm.right, rm.sink, rm.exc};
      }
    } else if (ndirty > 0) {
      // rebuild: thread (r, q) reads pixels (r, 4q .. 4q+3); this warp makes rows 4 warp .. + 3
      const int dt = s_dt[par][lane & (SOLVE_WARPS - 1)];
      unsigned todo = __ballot_sync(FULL, dt >= 0) & ((1u << SOLVE_WARPS) - 1u);
      int4 v[5];
      auto load = [&](int td) {
        const long long o = (long long)td * GC_TILE_PX + tid * 4;
        v[0] = *(const int4*)(P.cap[DUP] + o);
        v[1] = *(const int4*)(P.cap[DDOWN] + o);
        v[2] = *(const int4*)(P.cap[DLEFT] + o);
        v[3] = *(const int4*)(P.cap[DRIGHT] + o);
        v[4] = *(const int4*)(P.exc + o);
      };
      load(__shfl_sync(FULL, dt, __ffs(todo) - 1));
      while (todo) {
        const int w = __ffs(todo) - 1;
        const int td = __shfl_sync(FULL, dt, w);
        todo &= todo - 1;
        const uint32_t mk = row_masks({v[4].x, v[4].y, v[4].z, v[4].w}, {v[0].x, v[0].y, v[0].z, v[0].w},
                                      {v[1].x, v[1].y, v[1].z, v[1].w}, {v[2].x, v[2].y, v[2].z, v[2].w},
                                      {v[3].x, v[3].y, v[3].z, v[3].w}, lane);
        // sum of the positive excess, in halves that fit 32 bits over a warp's 128 pixels
        const unsigned e0 = v[4].x > 0 ? v[4].x : 0, e1 = v[4].y > 0 ? v[4].y : 0;
        const unsigned e2 = v[4].z > 0 ? v[4].z : 0, e3 = v[4].w > 0 ? v[4].w : 0;
        const unsigned lo = (e0 & 0xffffu) + (e1 & 0xffffu) + (e2 & 0xffffu) + (e3 & 0xffffu);
        const unsigned hi = (e0 >> 16) + (e1 >> 16) + (e2 >> 16) + (e3 >> 16);
        if (todo) load(__shfl_sync(FULL, dt, __ffs(todo) - 1));   // the next tile's, in flight
        const unsigned slo = __reduce_add_sync(FULL, lo), shi = __reduce_add_sync(FULL, hi);
        uint32_t* const sw = sm + w * REB_WORDS;
        const int k = lane & 7, row = tid >> 3;
        if (k < 6) {
          (k < 4 ? P.mcan + (long long)td * 128 + 32 * k : (k == 4 ? P.msink : P.mexc) + (long long)td * 32)[row] = mk;
          sw[32 * k + row] = mk;
        }
        if (lane == 0) {
          sw[192 + 2 * warp] = slo;
          sw[193 + 2 * warp] = shi;
        }
      }
      __syncthreads();
      if (dirty) {
        const uint32_t* const sw = sm + warp * REB_WORDS;
        m = TileMasks{sw[lane], sw[32 + lane], sw[64 + lane], sw[96 + lane], sw[128 + lane], sw[160 + lane]};
        ps = 0;
#pragma unroll
        for (int w = 0; w < SOLVE_WARPS; ++w)
          ps += (long long)sw[192 + 2 * w] + ((long long)sw[193 + 2 * w] << 16);
        if (lane == 0) {
          P.tpos[t] = ps;
          P.mdirty[t] = 0;
        }
      }
    }
    if (t < 0) continue;
    if (lane == 0 && ps) fs.add(A.acc, img, ps);   // taken with the tile's masks
    flood_fill(P, t, nb, lane, img, stamp, m, m.exc, 0, hits, out);
  }
  flood_sum_flush<SOLVE_WARPS>(A.acc, fs);
}

// The solve over the selection (see Pool::solve_images): images that continue from a previous
// flow (mode 2) are flooded first, and those whose flood reaches a sink pixel get a global
// relabel; freshly uploaded ones (mode 1) start from the trivial labelling.  Then cycles of
// {pulses of discharge, flood, relabel of the images whose flood reached a sink}, until no
// flood does: each image's last flood is its canonical cut.  A flood's stamp is its number
// in the solve; an image whose flood reached a sink carries that stamp in img_hit, which
// selects it for the relabel and for the next flood.
//
// Cap of the relabel's distances.  Excess moves at most pulses x iters pixels a cycle, so
// only excess near a sink matters to a cycle; distances beyond the cap are not computed, and
// pixels there stay inactive.  Exact distances would be the chain of tile rounds across every
// region that has excess and one unsaturated edge left (up to 34 rounds of 14-25 us at
// 4096^2), with all its tiles discharged.  The labels stay valid: below the cap they are
// exact, and at or above it "not below".  The cap doubles with every cycle, and at once when no
// excess lies within it, so the schedule ends in exact relabels and terminates as they do.
//
// 3 CTAs of 256 threads per SM (see discharge_phase); the relabel's and the flood's staging
// share the discharge's shared memory.
constexpr size_t SOLVE_BFS_SMEM = (size_t)SOLVE_WARPS * 32 * 33 * sizeof(int32_t);
constexpr size_t SOLVE_DYN_SMEM = DIS_DYN_SMEM > SOLVE_BFS_SMEM ? DIS_DYN_SMEM : SOLVE_BFS_SMEM;
static_assert(SOLVE_WARPS * REB_WORDS * sizeof(uint32_t) <= SOLVE_DYN_SMEM, "rebuild staging");

__global__ void __launch_bounds__(DIS_THREADS, 3)
k_solve(PoolView P, SolveArgs A) {
  extern __shared__ __align__(128) int32_t dsm[];
  __shared__ uint64_t mbar;
  __shared__ SolveState st;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bid = blockIdx.x, nb = gridDim.x;
  unsigned phase = 0;     // of mbar
  // ---- prologue: no reset and no barrier (the solve before left counters and sums at zero, and
  // stamps of another solve equal none of this one's)
  trace_mark(P, TR_BEGIN);
  if (tid == 0) {
    st = SolveState{};
    st.cap = A.cap;
    st.hlim = kFirstLimit;    // no relabel yet: trivial labels
    st.stamp = A.stamp0;
    st.step = ST_LIST;
    if (A.warm) {
      st.step = ST_FLOOD_FIRST;
      ++st.stamp;
    } else if (nb >= A.tiles) {
      // a tile per CTA: the first list needs no step of its own.  It has one entry per CTA, and
      // to a CTA whose tile is not active it is empty.
      if (bid == 0) trace_record(P, TR_ACTIVE_LIST);
      begin_cycle(A, st, 0);
      if (bid < A.tiles) {
        SelCursor cursor(P, A.ranges, bid, A.sel0);
        const int t = cursor.tile(bid);
        if (fresh_tile_active(P, t)) {
          P.queue[0][bid] = t;
          st.n = bid + 1;
        }
      }
    }
    mbar_init(&mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  for (int step = st.step; step != ST_END; step = st.step) {
    if (bid == 0 && tid == 0 && list_slot_cleared(st) >= 0) P.ctl[list_slot_cleared(st)] = 0;
    if (step == ST_PULSE) {
      trace_mark(P, TR_DISCHARGE);
      const int qk = st.qk;
      const Worklist in{(qk & 1) ? P.queue[1] : P.queue[0], nullptr, (qk & 1) ? P.inq[1] : P.inq[0]};
      Worklist out{(qk & 1) ? P.queue[0] : P.queue[1], &P.ctl[list_slot(st)],
                   (qk & 1) ? P.inq[0] : P.inq[1], &st.push};
      if (st.pulse == st.pulses - 1) out.list = nullptr;   // the relabel makes the next list
      discharge_phase(P, st.iters, st.hlim, bid, nb, in, st.n, out, dsm,
                      *reinterpret_cast<DisSmem*>(dsm + DIS_PLANES * GC_TILE_PX), &mbar, phase);
    } else if (step == ST_FLOOD_FIRST) {
      trace_mark(P, TR_FLOOD_FIRST);
      if (bid == 0 && tid == 0) {
        P.ctl[CTL_H0 + (st.stamp + 1) % 3] = 0;
        P.ctl[CTL_F0 + (st.fk + 2) % 3] = 0;
      }
      flood_first_phase(P, A, st, reinterpret_cast<uint32_t*>(dsm));
    } else if (step == ST_FLOOD) {
      trace_mark(P, TR_FLOOD);
      const int fk = st.fk, stamp = st.stamp, n = st.n;
      const Worklist out{(fk & 1) ? P.fq[0] : P.fq[1], &P.ctl[CTL_F0 + (fk + 1) % 3],
                         (fk & 1) ? P.mark[0] : P.mark[1], &st.push};
      const int32_t* const list = (fk & 1) ? P.fq[1] : P.fq[0];
      int32_t* const mark = (fk & 1) ? P.mark[1] : P.mark[0];
      if (bid == 0 && tid == 0) P.ctl[CTL_F0 + (fk + 2) % 3] = 0;
      for (int i = warp * nb + bid; i < n; i += SOLVE_WARPS * nb) {
        const int t = list[i];
        const int img = P.img_of[t];
        if (lane == 0) mark[t] = 0;
        if ((unsigned)img >= (unsigned)P.nimg) {   // self-check
          if (lane == 0) record_bad(P, 4, img);
          continue;
        }
        // an image whose flood reached a sink is not solved: it is flooded again later
        if (*((volatile int32_t*)&P.img_hit[img]) == stamp) continue;
        flood_frontier_tile(P, t, lane, img, stamp, &P.ctl[CTL_H0 + stamp % 3], out);
      }
    } else if (step == ST_BFS_FIRST || step == ST_BFS) {
      // global relabel of the images not solved; it lists their active tiles
      const int first = step == ST_BFS_FIRST;
      trace_mark(P, first ? TR_BFS_FIRST : TR_BFS);
      const int fk = st.fk, stamp = st.stamp, cap = st.cap, qk = st.qk;
      const int n = first ? A.tiles : st.n;
      if (first && bid == 0)   // their sums start afresh with their next flood
        for (int i = tid; i < P.nimg; i += DIS_THREADS)
          if (P.img_hit[i] == stamp) A.acc[i].sumpos_e = 0;
      const Worklist act_out{(qk & 1) ? P.queue[1] : P.queue[0], &P.ctl[list_slot(st)], nullptr};
      const Worklist out{(fk & 1) ? P.fq[0] : P.fq[1], &P.ctl[CTL_F0 + (fk + 1) % 3],
                         (fk & 1) ? P.mark[0] : P.mark[1], &st.push};
      const int32_t* const list = (fk & 1) ? P.fq[1] : P.fq[0];
      int32_t* const mark = (fk & 1) ? P.mark[1] : P.mark[0];
      if (bid == 0 && tid == 0) P.ctl[CTL_F0 + (fk + 2) % 3] = 0;
      const int i0 = warp * nb + bid;
      SelCursor cursor(P, first ? A.ranges : 0, i0 < n ? i0 : 0, A.sel0);
      for (int i = i0; i < n; i += SOLVE_WARPS * nb) {
        const int t = first ? cursor.tile(i) : list[i];
        if (first && P.img_hit[cursor.image()] != stamp) continue;
        if (!first && lane == 0) mark[t] = 0;
        const int act = bfs_tile(P, t, lane, first, cap, dsm + warp * (32 * 33), out);
        if (lane == 0) {
          // a tile becomes active once (its reached set only grows): list it then
          if (act > 0 && (first || P.tact[t] == 0)) worklist_append(P, act_out, t);
          if (first || act > 0) P.tact[t] = act;
        }
      }
    } else if (step == ST_LIST) {
      // the fresh images' first list
      trace_mark(P, TR_ACTIVE_LIST);
      const int qk = st.qk;
      const Worklist act_out{(qk & 1) ? P.queue[1] : P.queue[0], &P.ctl[list_slot(st)], nullptr};
      const int i0 = bid * DIS_THREADS + tid;
      SelCursor cursor(P, A.ranges, i0 < A.tiles ? i0 : 0, A.sel0);
      for (int b = bid * DIS_THREADS; b < A.tiles; b += nb * DIS_THREADS) {   // CTA-uniform
        int t = -1;
        if (b + tid < A.tiles) {
          t = cursor.tile(b + tid);
          const int mode = A.ranges == 1 ? A.mode0 : P.sel_mode[cursor.range()];
          if (mode != 1 || !fresh_tile_active(P, t)) t = -1;
        }
        const unsigned m = __ballot_sync(0xffffffffu, t >= 0);
        if (m == 0) continue;
        int pos = 0;
        if (lane == 0) pos = atomicAdd(act_out.count, __popc(m));
        pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(m & ((1u << lane) - 1u));
        if (t >= 0) {
          if (pos < P.nt) act_out.list[pos] = t;
          else record_bad(P, 1, pos);
        }
      }
    }
    solve_barrier(P, A, st);
  }

  // ---- results: control words and sums to the host, labels of a one-image handle
  if (bid == 0) {
    if (tid == 0) {
      volatile int32_t* ctl = P.ctl;
      if (st.err) atomicCAS(&P.ctl[CTL_ERR], 0, st.err);
      ctl[CTL_BFS_TOTAL] = st.nb;
      ctl[CTL_FLOOD_TOTAL] = st.nf;
      ctl[CTL_CYCLES] = st.cycles;
      ctl[CTL_NACT] = A.fresh ? 1 : 0;
      ctl[CTL_PULSE] = st.np;
      trace_record(P, TR_END);
    }
    __syncthreads();
    publish_results(P, A.acc);
    if (A.clean) {   // the images' sums start the next solve at zero
      __syncthreads();
      for (int k = tid; k < A.ranges; k += DIS_THREADS) {
        const int img = P.sel[k].w;
        if ((unsigned)img < (unsigned)P.nimg) A.acc[img].sumpos_e = 0;
      }
    }
  }
  if (A.lmode && !st.err) {
    trace_mark(P, TR_LABELS);
    const long long i0 = (long long)bid * DIS_THREADS + tid, step = (long long)nb * DIS_THREADS;
    if (A.lmode == 2) write_labels_packed(P, A.im, A.labels, i0, step);
    else write_labels(P, A.im, A.labels, i0, step);
  }
  // the last CTA to leave clears the counters and the barrier for the next launch
  __syncthreads();
  if (tid == 0) __threadfence();
  if (tid == 0 && atomicAdd(P.bar + BAR_EXIT, 1ull) == (unsigned long long)nb - 1) {
    if (A.clean)
      for (int k = CTL_Q0; k < CTL_H0 + 3; ++k) P.ctl[k] = 0;
    P.bar[BAR_EXIT] = 0;
    P.bar[BAR_ARRIVE] = 0;
    P.bar[BAR_ARRIVE + BAR_STRIDE] = 0;
  }
}

// One plane of one image back to row-major.
__global__ void k_state_out(ImageDesc im, const int32_t* __restrict__ plane, int32_t* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)im.W * im.H) return;
  const int y = (int)(i / im.W), x = (int)(i % im.W);
  const int t = im.tile0 + (y >> 5) * im.tw + (x >> 5);
  out[i] = plane[(long long)t * GC_TILE_PX + (y & 31) * GC_TILE + (x & 31)];
}

// T-link edits: excess moves by (new - old) t-link; returns the change of the pixel's term in
// the running sum of max(t, 0).
__device__ __forceinline__ long long apply_tlink(const PoolView& P, const ImageDesc& im, int x, int y,
                                                 int32_t v, int32_t* tl) {
  const int t = im.tile0 + (y >> 5) * im.tw + (x >> 5);
  const long long o = (long long)t * GC_TILE_PX + (y & 31) * GC_TILE + (x & 31);
  const int32_t old = tl[o];
  if (old == v) return 0;
  tl[o] = v;
  atomicAdd(P.exc + o, v - old);
  mark_dirty(P, t);
  return (long long)(v > 0 ? v : 0) - (long long)(old > 0 ? old : 0);
}

// Adds the CTA's changes to the image's sum: one add a warp that has any (an add per pixel, all
// to one address, was most of a stroke's 27 us).  Every thread of the warp calls it.
__device__ __forceinline__ void add_tlink_sum(ImageAcc* acc, int img, long long dpos) {
  if (!__any_sync(0xffffffffu, dpos != 0)) return;
#pragma unroll
  for (int o = 16; o; o >>= 1) dpos += __shfl_xor_sync(0xffffffffu, dpos, o);
  if ((threadIdx.x & 31) == 0 && dpos) atomicAdd(&acc[img].sumpos_t, (unsigned long long)dpos);
}

__global__ void k_edit(PoolView P, ImageDesc im, int img, const int32_t* __restrict__ idx,
                       const int32_t* __restrict__ val, int n, int32_t* tl, ImageAcc* acc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  long long dpos = 0;
  if (i < n) {
    const int p = idx[i];
    if (p >= 0 && p < im.W * im.H) dpos = apply_tlink(P, im, p % im.W, p / im.W, val[i], tl);
  }
  add_tlink_sum(acc, img, dpos);
}

// A polyline of an edit.  Up to EDIT_INLINE points travel in the launch itself, so an edit is
// one launch and no wait; more are read from device memory.
constexpr int EDIT_INLINE = 64;
struct InlinePts {
  int32_t v[2 * EDIT_INLINE];
  __device__ __forceinline__ int32_t operator[](int i) const { return v[i]; }
};
struct DevicePts {
  const int32_t* v;
  __device__ __forceinline__ int32_t operator[](int i) const { return v[i]; }
};

// Stroke: pixels within `radius` of the polyline get t-link `value`.  Exact integer test:
// with a = p - A, b = B - A, L = b.b, s = a.b: inside iff |p - A|^2 <= r^2 (s <= 0),
// |p - B|^2 <= r^2 (s >= L), else |a|^2 L - s^2 <= r^2 L.
__device__ __forceinline__ bool in_segment(int px, int py, long long ax, long long ay, long long bx,
                                           long long by, long long r2) {
  const long long dx = px - ax, dy = py - ay, ux = bx - ax, uy = by - ay;
  const long long L = ux * ux + uy * uy, s = dx * ux + dy * uy;
  if (L == 0 || s <= 0) return dx * dx + dy * dy <= r2;
  if (s >= L) {
    const long long ex = px - bx, ey = py - by;
    return ex * ex + ey * ey <= r2;
  }
  return (dx * dx + dy * dy) * L - s * s <= r2 * L;
}

// A CTA covers 32 x 8 pixels of the polyline's bounding box.  Its warps first mark the
// segments whose own box, widened by the radius, meets the CTA's pixels; most CTAs of a long
// stroke's box meet none and leave.
constexpr int STROKE_W = 32, STROKE_H = 8;

template <class Pts>
__global__ void __launch_bounds__(STROKE_W * STROKE_H)
k_stroke(PoolView P, ImageDesc im, int img, const Pts pts, int npts, int radius, int32_t value,
         int x0, int y0, int x1, int y1, int32_t* tl, ImageAcc* acc) {
  __shared__ unsigned s_near[32];   // segments to test, a bit each
  const int tid = threadIdx.x;
  const int bx0 = x0 + (int)blockIdx.x * STROKE_W, by0 = y0 + (int)blockIdx.y * STROKE_H;
  const int nseg = npts > 1 ? npts - 1 : 1;
  if (tid < 32) s_near[tid] = 0;
  __syncthreads();
  bool any = false;
  for (int k = tid; k < nseg; k += STROKE_W * STROKE_H) {
    const long long ax = pts[2 * k], ay = pts[2 * k + 1];
    const long long bx = npts > 1 ? pts[2 * k + 2] : ax, by = npts > 1 ? pts[2 * k + 3] : ay;
    if ((ax < bx ? ax : bx) - radius < bx0 + STROKE_W && (ax > bx ? ax : bx) + radius >= bx0 &&
        (ay < by ? ay : by) - radius < by0 + STROKE_H && (ay > by ? ay : by) + radius >= by0) {
      atomicOr(&s_near[k >> 5], 1u << (k & 31));
      any = true;
    }
  }
  if (!__syncthreads_or(any)) return;
  const int x = bx0 + (tid & (STROKE_W - 1)), y = by0 + tid / STROKE_W;
  bool hit = false;
  const long long r2 = (long long)radius * radius;
  if (x <= x1 && y <= y1)
    for (int w = 0; w <= (nseg - 1) >> 5 && !hit; ++w)
      for (unsigned m = s_near[w]; m && !hit; m &= m - 1) {
        const int k = 32 * w + __ffs(m) - 1;
        const int32_t ax = pts[2 * k], ay = pts[2 * k + 1];
        hit = in_segment(x, y, ax, ay, npts > 1 ? pts[2 * k + 2] : ax, npts > 1 ? pts[2 * k + 3] : ay, r2);
      }
  add_tlink_sum(acc, img, hit ? apply_tlink(P, im, x, y, value, tl) : 0);
}

// Reference brush (gc_edit_brush): the pixel set of Brush.points (brush.pyx:138-161), the
// line pixels of each segment (skimage.draw.line: Bresenham, the minor axis stepping while
// the error term d = 2 dr - dc + ... is >= 0) widened by the disc of skimage.draw.circle, whose
// points satisfy (dy / R)^2 + (dx / R)^2 < 1 in float64.  The disc is centred on every line
// pixel (the reference adds circle(R, R, R), a disc shifted by +R) and pixels outside the
// image are skipped (the reference's y * W + x wraps them).
//
// Along the major axis (n steps, minor-axis travel m) Bresenham's i-th pixel has minor
// offset floor((2 m i + n) / (2 n)): the loop steps the minor axis once for every time the
// error term 2 m (i + 1) - n - 2 n k reaches 0, which is rounding m i / n to the nearest
// integer with halves up.  Each thread tests one pixel of the bounding box against the
// line pixels within R - 1 of it along the major axis, so every pixel is written once.
constexpr int GC_BRUSH_MAX_RADIUS = 1024;

// skimage's disc test for the offset (dy, dx): two quotients, two squares and a sum, each
// rounded on its own as numpy evaluates ((y - cy) / ry) ** 2 + ((x - cx) / rx) ** 2 < 1.
__device__ __forceinline__ bool brush_disk(int dy, int dx, int R) {
  const double a = __ddiv_rn((double)dy, (double)R), b = __ddiv_rn((double)dx, (double)R);
  return __dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)) < 1.0;
}

template <class Pts>
__device__ __forceinline__ bool in_brush(int px, int py, const Pts& pts, int npts, int R,
                                         const int32_t* half) {
  const int nseg = npts > 1 ? npts - 1 : 1;
  for (int k = 0; k < nseg; ++k) {
    const int x0 = pts[2 * k], y0 = pts[2 * k + 1];
    const int x1 = npts > 1 ? pts[2 * k + 2] : x0, y1 = npts > 1 ? pts[2 * k + 3] : y0;
    const int dr = abs(y1 - y0), dc = abs(x1 - x0);
    const int sr = (y1 - y0) > 0 ? 1 : -1, sc = (x1 - x0) > 0 ? 1 : -1;
    const bool steep = dr > dc;
    const int n = steep ? dr : dc, m = steep ? dc : dr;       // major steps, minor travel
    const int a0 = steep ? y0 : x0, b0 = steep ? x0 : y0;     // major / minor start
    const int sa = steep ? sr : sc, sb = steep ? sc : sr;
    const int pa = steep ? py : px;
    const int t = sa * (pa - a0);                             // pixel's major-axis step
    const int ilo = max(t - (R - 1), 0), ihi = min(t + (R - 1), n);
    for (int i = ilo; i <= ihi; ++i) {
      const int bi = n > 0 ? b0 + sb * (int)((2LL * m * i + n) / (2LL * n)) : b0;
      const int ai = a0 + sa * i;
      const int dy = py - (steep ? ai : bi), dx = px - (steep ? bi : ai);
      if (dy < 1 - R || dy > R - 1) continue;
      const int w = half[dy + R - 1];
      if (dx >= -w && dx <= w) return true;
    }
  }
  return false;
}

template <class Pts>
__global__ void k_brush(PoolView P, ImageDesc im, int img, const Pts pts, int npts, int R, 
                        int32_t value, int x0, int y0, int bw, int bh,
                        int32_t* tl, ImageAcc* acc) {
  // half[dy + R - 1] = the largest dx >= 0 with the offset (dy, dx) inside the disc (the
  // test is monotone in |dx|; dx = 0 is inside for |dy| <= R - 1)
  __shared__ int32_t half[2 * GC_BRUSH_MAX_RADIUS - 1];
  for (int j = threadIdx.x; j < 2 * R - 1; j += blockDim.x) {
    const int dy = j - (R - 1);
    int lo = 0, hi = R - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (brush_disk(dy, mid, R)) lo = mid; else hi = mid - 1;
    }
    half[j] = lo;
  }
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long dpos = 0;
  if (i < (long long)bw * bh) {
    const int x = x0 + (int)(i % bw), y = y0 + (int)(i / bw);
    if (x >= 0 && y >= 0 && x < im.W && y < im.H && in_brush(x, y, pts, npts, R, half))
      dpos = apply_tlink(P, im, x, y, value, tl);
  }
  add_tlink_sum(acc, img, dpos);
}

// ------------------------------------------------------------------------------------
// Launchers
// ------------------------------------------------------------------------------------
static inline int ok() { return cudaGetLastError() == cudaSuccess ? GC_OK : GC_ERR_CUDA; }

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int launch_upload(const PoolView& P, const ImageDesc& im, int img, const int32_t* up,
                  const int32_t* down, const int32_t* left, const int32_t* right,
                  const int32_t* excess, int32_t* tl, ImageAcc* acc, cudaStream_t s) {
  const bool vec = im.W % 4 == 0 && aligned16(up) && aligned16(down) && aligned16(left) &&
                   aligned16(right) && aligned16(excess);
  const PlaneSource src{up, down, left, right, excess, vec};
  k_upload<<<im.tw * im.th, DIS_THREADS, 0, s>>>(P, im, img, src, tl, acc);
  return ok();
}

int launch_upload_rgba(const PoolView& P, const ImageDesc& im, int img, const uint32_t* rgba,
                       const int32_t* excess, const int32_t* tab, int lambda, int32_t* tl,
                       ImageAcc* acc, cudaStream_t s) {
  const RgbaSource src{rgba, excess, tab, lambda, im.W % 4 == 0 && aligned16(rgba) && aligned16(excess)};
  if (tab)
    k_upload_rgba<<<im.tw * im.th, DIS_THREADS, 0, s>>>(P, im, img, src, ExpWeight{0.0f}, tl, acc);
  else
    k_upload_rgba<<<im.tw * im.th, DIS_THREADS, 0, s>>>(P, im, img, src, RefWeight{lambda}, tl, acc);
  return ok();
}

int launch_nlinks(const uint32_t* rgba, int W, int H, unsigned long long* state, int32_t* tab,
                  ImageAcc* acc, int sms, cudaStream_t s) {
  const long long npairs = (long long)(H - 1) * W + (long long)H * (W - 1);
  const int px = W % 4 == 0 && aligned16(rgba) ? 4 : 1;   // ragged rows have no aligned strips
  const int rows = px == 4 ? DSUM_ROWS<4> : DSUM_ROWS<1>;
  const long long blocks = (long long)((W / px + DSUM_THREADS - 1) / DSUM_THREADS) * ((H + rows - 1) / rows);
  const long long wave = (px == 4 ? 4LL : 8LL) * sms;   // resident CTAs: strips of 4 take the registers
  const int grid = (int)(blocks < wave ? blocks : wave);
  if (px == 4) k_nlinks<4><<<grid, DSUM_THREADS, 0, s>>>(rgba, W, H, npairs, state, tab, acc);
  else k_nlinks<1><<<grid, DSUM_THREADS, 0, s>>>(rgba, W, H, npairs, state, tab, acc);
  return ok();
}

int launch_masks(const PoolView& P, int grid, cudaStream_t s) {
  k_masks<<<grid, WARPS_PER_CTA * 32, 0, s>>>(P);
  return ok();
}

int launch_discharge(const PoolView& P, int iters, int hlim, int grid, cudaStream_t s) {
  k_discharge<<<grid, DIS_THREADS, DIS_DYN_SMEM, s>>>(P, iters, hlim);
  return ok();
}

int launch_edge_relabel_build(const PoolView& P, int32_t* list, int32_t* count,
                              const ScanState& st, cudaStream_t s) {
  const int nch = (P.nt + EB_TILES - 1) / EB_TILES;
  if (nch > st.max_chunks) return GC_ERR_INVALID;
  k_edge_relabel_build<<<nch, EB_THREADS, 0, s>>>(P, list, count, st);
  return ok();
}

int launch_bfs_round(const PoolView& P, int first, int cap, int live, int grid, cudaStream_t s) {
  k_bfs_round<<<grid, WARPS_PER_CTA * 32, 0, s>>>(P, first, cap, live);
  return ok();
}

int launch_flood_round(const PoolView& P, int mode, int abort_hit, int stamp, ImageAcc* acc,
                       int grid, cudaStream_t s) {
  k_flood_round<<<grid, WARPS_PER_CTA * 32, 0, s>>>(P, mode, abort_hit, stamp, acc);
  return ok();
}

int launch_flood_check(const PoolView& P, int all, int stamp, ImageAcc* acc, cudaStream_t s) {
  k_flood_check<<<1, 256, 0, s>>>(P, all, stamp, acc);
  return ok();
}

int launch_solve(const PoolView& P, const SolveArgs& a, int grid, cudaStream_t s) {
  PoolView p = P;
  SolveArgs args = a;
  void* params[] = {&p, &args};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_solve, dim3(grid), dim3(DIS_THREADS),
                                                    params, SOLVE_DYN_SMEM, s);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess ? GC_OK : GC_ERR_CUDA;
}

__global__ void k_acc_reset(ImageAcc* acc, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) acc[i].sumpos_e = 0;
}

int launch_acc_reset(ImageAcc* acc, int n, cudaStream_t s) {
  k_acc_reset<<<(n + 255) / 256, 256, 0, s>>>(acc, n);
  return ok();
}

int launch_ctl_begin(const PoolView& P, int max_rounds, ImageAcc* acc, cudaStream_t s) {
  k_ctl_begin<<<1, 256, 0, s>>>(P, max_rounds, acc);
  return ok();
}

int launch_active_list(const PoolView& P, const ScanState& st, int32_t* list, int32_t* count,
                       int live, int fresh, int grid, cudaStream_t s) {
  const int nch = (P.nt + ACT_CHUNK - 1) / ACT_CHUNK;   // enough for any selection
  if (nch > st.max_chunks) return GC_ERR_INVALID;
  grid = grid < nch ? grid : nch;
  k_active_list<<<grid > 0 ? grid : 1, ACT_THREADS, 0, s>>>(P, st, list, count, live, fresh);
  return ok();
}

int launch_ctl_cycle(const PoolView& P, cudaStream_t s) {
  k_ctl_cycle<<<1, 32, 0, s>>>(P);
  return ok();
}

int launch_image_tiles(const PoolView& P, const ImageDesc& im, int img, cudaStream_t s) {
  const int n = im.tw * im.th;
  if (n <= 0) return GC_OK;
  k_image_tiles<<<(n + 255) / 256, 256, 0, s>>>(P, im, img);
  return ok();
}

// one thread per tile row of the image
static unsigned labels_grid(const ImageDesc& im) {
  const long long g = ((long long)im.H * im.tw + 255) / 256;
  return (unsigned)(g < 1 ? 1 : g);
}

int launch_labels_out(const PoolView& P, const ImageDesc& im, uint8_t* out, cudaStream_t s) {
  k_labels_out<<<labels_grid(im), 256, 0, s>>>(P, im, out);
  return ok();
}

int launch_labels_packed(const PoolView& P, const ImageDesc& im, uint8_t* out, cudaStream_t s) {
  k_labels_packed<<<labels_grid(im), 256, 0, s>>>(P, im, out);
  return ok();
}

int launch_state_out(const PoolView& P, const ImageDesc& im, const int32_t* plane,
                     int32_t* out, cudaStream_t s) {
  (void)P;
  const long long n = (long long)im.W * im.H;
  k_state_out<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(im, plane, out);
  return ok();
}

int launch_edit(const PoolView& P, const ImageDesc& im, int img, const int32_t* idx,
                const int32_t* val, int n, int32_t* tl, ImageAcc* acc, cudaStream_t s) {
  if (n <= 0) return GC_OK;
  k_edit<<<(n + 255) / 256, 256, 0, s>>>(P, im, img, idx, val, n, tl, acc);
  return ok();
}

bool edit_points_inline(int npts) { return npts <= EDIT_INLINE; }

static InlinePts inline_pts(const int32_t* pts_host, int npts) {
  InlinePts p{};
  for (int k = 0; k < 2 * npts; ++k) p.v[k] = pts_host[k];
  return p;
}

int launch_stroke(const PoolView& P, const ImageDesc& im, int img, const int32_t* pts_dev,
                  const int32_t* pts_host, int npts, int radius, int32_t value, int32_t* tl,
                  ImageAcc* acc, cudaStream_t s) {
  int xmin = pts_host[0], xmax = pts_host[0], ymin = pts_host[1], ymax = pts_host[1];
  for (int k = 1; k < npts; ++k) {
    xmin = xmin < pts_host[2 * k] ? xmin : pts_host[2 * k];
    xmax = xmax > pts_host[2 * k] ? xmax : pts_host[2 * k];
    ymin = ymin < pts_host[2 * k + 1] ? ymin : pts_host[2 * k + 1];
    ymax = ymax > pts_host[2 * k + 1] ? ymax : pts_host[2 * k + 1];
  }
  int x0 = xmin - radius, y0 = ymin - radius, x1 = xmax + radius, y1 = ymax + radius;
  x0 = x0 < 0 ? 0 : x0; y0 = y0 < 0 ? 0 : y0;
  x1 = x1 > im.W - 1 ? im.W - 1 : x1; y1 = y1 > im.H - 1 ? im.H - 1 : y1;
  if (x1 < x0 || y1 < y0) return GC_OK;   // (so the grid below covers pixels of the image only)
  const dim3 grid((x1 - x0) / STROKE_W + 1, (y1 - y0) / STROKE_H + 1);
  if (npts <= EDIT_INLINE)
    k_stroke<<<grid, STROKE_W * STROKE_H, 0, s>>>(P, im, img, inline_pts(pts_host, npts), npts, radius,
                                                  value, x0, y0, x1, y1, tl, acc);
  else
    k_stroke<<<grid, STROKE_W * STROKE_H, 0, s>>>(P, im, img, DevicePts{pts_dev}, npts, radius, value,
                                                  x0, y0, x1, y1, tl, acc);
  return ok();
}

int launch_brush(const PoolView& P, const ImageDesc& im, int img, const int32_t* pts_dev,
                 const int32_t* pts_host, int npts, int radius, int32_t value, int32_t* tl,
                 ImageAcc* acc, cudaStream_t s) {
  const int R = radius < 1 ? 1 : radius;
  if (R > GC_BRUSH_MAX_RADIUS) return GC_ERR_INVALID;
  int xmin = pts_host[0], xmax = pts_host[0], ymin = pts_host[1], ymax = pts_host[1];
  for (int k = 1; k < npts; ++k) {
    xmin = xmin < pts_host[2 * k] ? xmin : pts_host[2 * k];
    xmax = xmax > pts_host[2 * k] ? xmax : pts_host[2 * k];
    ymin = ymin < pts_host[2 * k + 1] ? ymin : pts_host[2 * k + 1];
    ymax = ymax > pts_host[2 * k + 1] ? ymax : pts_host[2 * k + 1];
  }
  long long x0 = (long long)xmin - (R - 1), y0 = (long long)ymin - (R - 1);
  long long x1 = (long long)xmax + (R - 1), y1 = (long long)ymax + (R - 1);
  x0 = x0 < 0 ? 0 : x0; y0 = y0 < 0 ? 0 : y0;
  x1 = x1 > im.W - 1 ? im.W - 1 : x1; y1 = y1 > im.H - 1 ? im.H - 1 : y1;
  if (x1 < x0 || y1 < y0) return GC_OK;
  const int bw = (int)(x1 - x0 + 1), bh = (int)(y1 - y0 + 1);
  const long long n = (long long)bw * bh;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (npts <= EDIT_INLINE)
    k_brush<<<grid, 256, 0, s>>>(P, im, img, inline_pts(pts_host, npts), npts, R, value, (int)x0,
                                 (int)y0, bw, bh, tl, acc);
  else
    k_brush<<<grid, 256, 0, s>>>(P, im, img, DevicePts{pts_dev}, npts, R, value, (int)x0, (int)y0,
                                 bw, bh, tl, acc);
  return ok();
}

// Loads every kernel of the library on the current device.  With lazy module loading (the
// CUDA default) a kernel is loaded at its first launch; doing it
// here, once per device under a lock, keeps that loading away from threads that solve on
// several streams at once.
void preload_kernels() {
  static std::mutex mu;
  static std::unordered_map<int, bool> done;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return;
  cudaFuncAttributes a;
  const void* kernels[] = {
      (const void*)k_upload, (const void*)k_upload_rgba<ExpWeight>,
      (const void*)k_upload_rgba<RefWeight>, (const void*)k_nlinks<1>, (const void*)k_nlinks<4>,
      (const void*)k_masks, (const void*)k_discharge, (const void*)k_edge_relabel_build,
      (const void*)k_bfs_round, (const void*)k_flood_round, (const void*)k_ctl_begin,
      (const void*)k_active_list, (const void*)k_ctl_cycle, (const void*)k_flood_check,
      (const void*)k_solve,
      (const void*)k_image_tiles,
      (const void*)k_acc_reset, (const void*)k_labels_out, (const void*)k_labels_packed,
      (const void*)k_state_out, (const void*)k_edit,
      (const void*)k_stroke<InlinePts>, (const void*)k_stroke<DevicePts>,
      (const void*)k_brush<InlinePts>, (const void*)k_brush<DevicePts>};
  for (const void* k : kernels) cudaFuncGetAttributes(&a, k);
  preload_scan_kernels();
  cudaGetLastError();
  done[dev] = true;
}

namespace {
// Launch geometry per device, set up once: the dynamic shared memory opt-in of k_discharge
// changes the function's state, so it is not repeated while other threads launch or
// launch it.
struct Geometry { int dis = 0, warps = 0, solve = 0; };
std::mutex g_geom_mu;
std::unordered_map<int, Geometry> g_geom;

Geometry device_geometry(int device) {
  std::lock_guard<std::mutex> lock(g_geom_mu);
  auto it = g_geom.find(device);
  if (it != g_geom.end()) return it->second;
  preload_kernels();
  int per_dis = 0, per_bfs = 0, per_solve = 0, sms = 0;
  cudaFuncSetAttribute(k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLVE_DYN_SMEM);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_solve, k_solve, DIS_THREADS, SOLVE_DYN_SMEM);
  cudaFuncSetAttribute(k_discharge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DIS_DYN_SMEM);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_dis, k_discharge, DIS_THREADS, DIS_DYN_SMEM);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_bfs, k_bfs_round, WARPS_PER_CTA * 32, 0);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  sms = sms > 0 ? sms : 1;
  Geometry g{(per_dis > 0 ? per_dis : 1) * sms, (per_bfs > 0 ? per_bfs : 1) * sms,
             (per_solve > 0 ? per_solve : 1) * sms};
  g_geom.emplace(device, g);
  return g;
}
}  // namespace

int occupancy_discharge(int device) { return device_geometry(device).dis; }
int occupancy_warps(int device) { return device_geometry(device).warps; }
int occupancy_solve(int device) { return device_geometry(device).solve; }

}  // namespace gcut
