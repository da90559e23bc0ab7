// Halo-tiled implicit-GEMM convolution (conv_halo.cu): interface between the plans and the kernel.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "elb_common.cuh"

namespace elb {

enum : int { HALO_I8 = 0, HALO_F32 = 1 };
constexpr int HALO_HEIGHTS = 5;
constexpr int HALO_MAX_OC = 2048;      // per-channel constants kept in shared memory

// n / d for 0 <= n < 2^31 as a multiply and a shift (the role loops divide once per tile)
struct FastDiv {
  uint32_t mul = 0, shift = 0, d = 1;
  void set(uint32_t div) {
    d = div;
    if (div <= 1) { mul = 0; shift = 0; return; }
    uint32_t s = 0;
    while ((1ull << s) < div) ++s;
    mul = static_cast<uint32_t>(((1ull << (31 + s)) + div - 1) / div);
    shift = s - 1;
  }
#ifdef __CUDACC__
  __device__ __forceinline__ uint32_t div(uint32_t n) const { return d == 1 ? n : __umulhi(n, mul) >> shift; }
#endif
};

// What a launch needs besides its tensor maps and constants (HaloArgs)
struct HaloParams {
  const uint8_t *b_img;              // packed weights [n tile][group][K step][...]
  const float *scale, *shift;        // int8: [OCP] requantisation constants; f32: shift = bias (null: none)
  const float *shift_tbl;            // int8, zero point with padding: shift vectors by (row class, column class)
  const int *hclass, *wclass;
  void *out;
  int32_t *acc_dump;
  int *status;
  Requant rq;
  int zp_nw, zp_full;
  int N, OH, OW, OCB;
  int period;                        // output rows per image in the stacked row space (OH + shared padding rows)
  int row_tiles, col_tiles, n_tiles, total_tiles;
  FastDiv div_n, div_col, div_period, div_px;
  int BN;                            // output channels of a tile (multiple of 16)
  // The K loop walks channel groups and, within one, the parity planes that have taps (stride 1: one plane).
  int groups, kch, planes;           // channel groups; 16-byte chunks of one pixel per group; planes
  int pitch;                         // bytes of one input row of one group in shared memory: kch * pxw * 16
  int pxw;                           // pixels of such a row
  int a_bytes, raw_bytes, a_stages;  // one ring stage of operand rows (f32: of its hi or lo half), of raw f32 rows; ring depth
  int ksteps;                        // K steps of a channel group, all planes
  int b_per_tile;                    // weight stages of a tile
  int wide;                          // fp32: `out` is 32-byte aligned (the library promises 16)
  int fast;                          // int8: u8 result, ReLU at 0, no residual, one shift vector (1: constants in cst)
  int row_units;                     // a weight stage holds a filter row's taps (1) or one tap (0) of a plane
  int kstep_bytes, b_stages, b_stage_bytes;
  int pair;                          // clusters of two CTAs multiply two row tiles by weights of which each holds half
  int split;                         // CTAs that share a tile's K loop (1: none; else one tile per cluster)
  int bufs;                          // accumulators in tensor memory: 4 of up to 128 columns or 2 of up to 256
  int spread;                        // int8: all epilogue warps share each tile (halo_launch() says when)
  int resident;                      // every weight stage of the (single) n tile stays in shared memory
  int stack;                         // f32: hi and lo weight rows of a chunk stacked (BN <= 128)
  int sep;                           // f32: the lo products have accumulators of their own, BN columns behind the hi ones
  int fine, chunk_groups;            // f32: the K loop runs in parts of so many channel groups (conv_halo.cu, FINE)
  int strided;                       // stride > 1: five-dimensional maps of the parity planes
  int cb_step;                       // channel blocks per group
  int row0[4], rows[4], col0[4];     // rows a tile reads of each plane: first (relative to the tile's), count; first column
  int tap_rows[4], tap_cols[4];      // the plane's taps: a rectangle, rows from row0, columns from col0
};

// Parameters of a kernel that reads up to PLANES planes and keeps the constants of up to OC channels here: 1216, 2176, 3136 or 4096
// bytes; with room for four planes and 256 channels every launch carried 5120.  An empty kernel that is waited for takes 9.3 us
// with 64 bytes and 9.8 with 5120 (medians of 40 x 200 calls), enqueued back to back 2.7 and 2.8; on another host it was 11.0 and
// 13.9, enqueued 4.8 and 7.0.
template <int PLANES, int OC>
struct HaloArgs : HaloParams {
  // [row / column parity plane of the input (stride 1: one)][rows a copy brings: 1, 2, 4, 8, all of a tile's]
  alignas(64) CUtensorMap tmap[PLANES][HALO_HEIGHTS];
  CUtensorMap tmap_b;                // pairs of CTAs: the packed weights as rows of 512 bytes
  // int8, up to OC channels: {scale, shift} in the parameter space.  The epilogue reads its constants with
  // every 16 outputs of a pixel, and from the constant bank those reads stay off the shared-memory port, which
  // the MMAs of narrow tiles fill (64 -> 128 channels at 112 x 112, 64 images: 63 -> 47 us without the loads).
  alignas(16) float cst[2][OC > 0 ? OC : 1];
};

// Geometry, packing order and launch parameters of one plan, filled by halo_plan().
struct HaloPlan {
  int kind = HALO_I8;
  HaloParams p{};
  size_t smem_bytes = 0, b_bytes = 0;
  double est_us = 0;                 // modelled time of the whole batch
  bool steps_ready = false;          // int8: halo_init() was called for launches with a step
  double gather_ratio = 0;           // int8: time of a tile's rows pixel by pixel (16 bytes per clock) over that of its MMAs
  double loop_ratio = 0;             // int8: modelled time of a tile's K loop over its epilogue's
  int max_clusters = 0;              // pairs the device holds at once
  int stride = 1, IH = 0, IW = 0, CB = 0;
  int parity[4] = {0, 0, 0, 0};      // of each plane: row parity * stride + column parity
  struct Chunk { int tap, cb; };     // tap -1: zero weights
  std::vector<Chunk> order;          // two (i8) chunks per K step of a group; f32: cb = quarter of the block
  CUtensorMap tmap_b{};
  std::vector<float> scale, shift;   // int8: host copies of the requantisation constants, [OCP]
  void *d_b = nullptr;               // packed weights (owned by the plan that owns this)
  // Tensor maps of the image counts (and input steps) seen so far, whatever the address: a launch copies them and sets its
  // input's address in those that its tiles use (`heights`: bit i = the maps of HaloArgs::tmap[plane][i]).
  struct Maps { int cnt, step, src_h, src_w; uint8_t heights[4]; CUtensorMap m[4][HALO_HEIGHTS]; };
  std::vector<Maps> maps;            // at most 16, the oldest replaced
  size_t next_map = 0;
};
// false: the shape does not suit the kernel (err says why).  max_acc (f32; 0: any): how many MMAs may add into one
// accumulator before it is added up in the epilogue's registers.
bool halo_plan(HaloPlan &hp, int kind, int n, int ic, int oc, int ih, int iw, int oh, int ow, int kh, int kw, int stride,
               int pad_t, int pad_l, int num_sms, std::string &err, int max_acc = 0);
// Weights in the order the kernel reads them: i8 from q[OCP][taps][ICP], f32 from u[OCP][taps][ICP].
std::vector<uint8_t> halo_pack_i8(const HaloPlan &hp, const int8_t *q, int OCP, int taps, int ICP);
std::vector<uint8_t> halo_pack_f32(const HaloPlan &hp, const float *u, int OCP, int taps, int ICP);
bool halo_set_weights(HaloPlan &hp, void *d_b, std::string &err);      // the packed weights on the device
cudaError_t halo_init(HaloPlan &hp, bool stepped = false);      // once per plan and device; stepped: before launches with a step, too
// Run `images` images: in / p.out address the first; p: a copy of hp.p with the per-call pointers set.
// step > 1 (stride 1 only): the tensor holds src_h x src_w pixels per plane, of which every step-th row and column is read.
bool halo_launch(HaloPlan &hp, HaloParams &p, const void *in, int images, int num_sms, cudaStream_t s, std::string &err,
                 int step = 1, int src_h = 0, int src_w = 0);

}  // namespace elb
