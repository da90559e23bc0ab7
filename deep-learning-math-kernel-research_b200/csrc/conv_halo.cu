// Convolution (INT8 u8 x s8 -> s32, and fp32 as 3xTF32) as an implicit GEMM whose activation operand
// is fetched ONCE per channel group and reused by every filter tap.
//
// Replaces, for filters larger than one pixel, strides above one and 1x1 layers of few tiles, the reference's
// elx_int8_conv_direct_t (src/elx_int8_conv_direct.cpp:502-571, kernels
// src/kernel/elk_u8s8_conv.hxx:254-677) and elx_conv_direct_t (src/elx_conv_direct.cpp,
// src/kernel/elk_conv.hxx).
//
// Tile: 16 output rows x 8 output columns = the 128 rows of one tcgen05.mma, times BN output channels.
// The input pixels the tile's taps touch (for a 3x3 stride-1 filter 18 x 10 pixels) are fetched row by row
// with tiled TMA copies into shared memory as [row][16-byte channel chunk][pixel][16 B].  Eight
// horizontally adjacent pixels of one chunk are 128 contiguous bytes, i.e. one core matrix of the
// no-swizzle K-major operand layout, the next eight rows of the operand are the next image row (stride
// `pitch`), and shifting the tile by a tap moves only the operand's START ADDRESS (16-byte granular in
// this layout).  So all taps multiply the same bytes: 1.4 x the tile's own pixels cross from L2 instead of
// the 9 x an implicit GEMM with one copy per tap moves, which is what bounded that form (94 B/clk per
// SM wanted at BN = 256 for int8, where an SM takes in about 60).  Stride 2 does the same on the four
// (row, column) parity planes of the input, one tensor map each.
//
// Small images: the output rows of all images of the batch are stacked into one tall row space with
// `period` = OH + the padding rows two neighbours can share, so 16-row tiles run across image borders and
// a 7x7 layer fills 7/8 of its tile rows; the copies are per row, so each finds its own image, and rows
// outside an image arrive as zeros.
//
// Warp roles: 0 activation rows (TMA) | 1, 3 MMA issuers (even / odd tiles of the CTA, 1 owns tensor memory)
// | 2 weights (bulk copies) | 4.. epilogue | (fp32) four warps that split the landed rows into tf32 hi / lo
// planes in shared memory.
// Two accumulators in tensor memory (int8 up to 128 channels per tile: four), filled by two issuers in turn.  An issuer
// spends 8 cycles on an MMA while its warp stays converged (umma_i8_el), and some hundreds per tile and stage on
// waits; two of them keep the pipe busy on tiles of 18 MMAs that last 864 cycles in all.
#include "conv_halo.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "host_prep.hpp"
#include "umma.cuh"

namespace elb {

namespace {

constexpr int BM = 128, TILE_H = 16, TILE_W = 8;
constexpr int MAX_A = 8, MAX_B = 16, RAW_STAGES = 4, MAX_BUFS = 4;
// int8: an epilogue group of four warps per (accumulator, half of the column blocks); fp32: per half
constexpr int EPI_WARP0 = 4, SPLIT_WARPS = 4;
constexpr int EPI_WARPS_I8 = 16, EPI_WARPS_F32 = 8;
constexpr int SPLIT_WARP0 = EPI_WARP0 + EPI_WARPS_F32;
constexpr int THREADS_I8 = (EPI_WARP0 + EPI_WARPS_I8) * 32, THREADS_F32 = (SPLIT_WARP0 + SPLIT_WARPS) * 32;
constexpr int SMEM_LIMIT = 232448 - 1024;      // dynamic shared memory the plan may fill

struct Bars {
  uint64_t afull[MAX_A], aempty[MAX_A], rfull[RAW_STAGES], rempty[RAW_STAGES], bfull[MAX_B], bempty[MAX_B], tfull[MAX_BUFS], tempty[MAX_BUFS], turn[2], parts;
  uint32_t tmem_slot;
  int abort_flag;
};

// All lanes wait (one instruction for the converged warp); the verdict is warp-uniform.
__device__ __forceinline__ bool wait_all(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  const bool ok = mbar_wait(bar, parity, abort_flag);
  return __all_sync(0xFFFFFFFFu, ok ? 1 : 0) != 0;
}

// Lane 0's value: the compiler then knows that the value is the same in the whole warp.  The MMA operands live in
// uniform registers; from values it cannot prove uniform (anything behind a branch on threadIdx) it builds them
// with a loop around every MMA.
__device__ __forceinline__ int uni(int v) { return __shfl_sync(0xFFFFFFFFu, v, 0); }

// requant_store16 for the common case: u8 result, ReLU at zero without an upper bound, no residual.  The
// saturating conversion is the ReLU; scale and shift on channel pairs (each lane rounds as the scalar fma).
__device__ __forceinline__ void requant_relu_u8(const int (&acc)[16], const float *sc, const float *sh, uint8_t *out) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const ulonglong2 c = reinterpret_cast<const ulonglong2 *>(sc)[i], h = reinterpret_cast<const ulonglong2 *>(sh)[i];
    int r[4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      unsigned long long f;
      asm("mov.b64 %0, {%1, %2};" : "=l"(f) : "f"(__int2float_rn(acc[4 * i + 2 * j])), "f"(__int2float_rn(acc[4 * i + 2 * j + 1])));
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(f) : "l"(f), "l"(j ? c.y : c.x), "l"(j ? h.y : h.x));
      float lo, hi;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(f));
      r[2 * j] = __float2int_rn(lo);
      r[2 * j + 1] = __float2int_rn(hi);
    }
    uint32_t t;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(t) : "r"(r[3]), "r"(r[2]));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(w[i]) : "r"(r[1]), "r"(r[0]), "r"(t));
  }
  *reinterpret_cast<uint4 *>(out) = make_uint4(w[0], w[1], w[2], w[3]);
}

// 32 bytes in one store: a lane's two 16-byte stores into one 32-byte sector would be two partial writes.  The address
// must be 32-byte aligned (HaloParams::wide).
__device__ __forceinline__ void store_v8(float *p, const float (&f)[16], int at) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + at), "f"(f[at]), "f"(f[at + 1]),
               "f"(f[at + 2]), "f"(f[at + 3]), "f"(f[at + 4]), "f"(f[at + 5]), "f"(f[at + 6]), "f"(f[at + 7])
               : "memory");
}

// PAIRS: K steps of one tap, each two 16-byte channel chunks (fp32: 2).  0: a group is ONE chunk wide (at most
// 16 int8 channels) and a K step takes the chunk of two neighbouring taps of a filter row.
// FORM: how the issuer walks the taps.  FORM_3X3_* are 3x3 stride 1 (a weight stage per filter row, per tap, or
// all weights resident) with a channel group's MMAs as straight-line code; FORM_ANY loops over rows and taps.
// STACK: fp32 with at most 128 output channels per tile, see HaloParams::stack.
// All are compile-time because the issuer is one warp: a loop iteration costs it 55 to 65 cycles whatever it
// does, an address from a table in the parameter space 70, and a wait on a completed barrier 100 to 160.  With
// loops, tables and a wait per filter row issuing took 2900 cycles per tile of 18 MMAs that last 864 (64 -> 64
// channels at 224 x 224).
// FORM_3X3S2: 3x3 stride 2 with one padding column (planes of 1, 2, 2 and 4 taps), FORM_1X1: one tap; a weight stage
// per tap.  (As loops a unit of four MMAs that last 512 cycles took 500 to 650 to issue.)
enum : int { FORM_ANY = 0, FORM_3X3_ROWS = 1, FORM_3X3_TAPS = 2, FORM_3X3_RESIDENT = 3, FORM_3X3S2 = 4, FORM_1X1 = 5 };
// pixels of a shared-memory row (what halo_plan() computes)
__host__ __device__ constexpr int pxw_of(int form, int kind, int pairs) {
  return form == FORM_1X1 ? (pairs ? 8 : 16)
       : form == FORM_3X3S2 ? (kind == HALO_F32 || pairs == 2 ? 10 : pairs == 4 ? 9 : pairs == 0 ? 16 : 12)
                            : (kind == HALO_F32 || pairs == 2 || pairs == 4 ? 10 : pairs == 0 ? 16 : 12);
}

// Planes and channels of a kernel's HaloArgs
__host__ __device__ constexpr int planes_of(int form) { return form == FORM_ANY || form == FORM_3X3S2 ? 4 : 1; }
// (constants of 256 channels cost every call another kilobyte and gain nothing: 16 x 80 -> 208 at 33x33 8.0 us, 7.6 without)
constexpr int PARAM_OC = 128;
__host__ __device__ constexpr int oc_of(int kind, bool split) { return kind == HALO_F32 || split ? 0 : PARAM_OC; }

// PAIR: clusters of two CTAs.  One tcgen05.mma.cta_group::2 multiplies two row tiles (128 rows per CTA) by the BN
// weight rows of which each CTA stages HALF: what an SM takes in per MMA from L2 and what the MMA reads from its
// shared memory both fall by the weights' half, and these two (about 50 B/clk, 128 B/clk) bound the tiles of
// 256 output channels on single CTAs.
// SPLIT: one tile per cluster of p.split CTAs, each of which multiplies a share of the channel groups; the partial
// sums meet in the CTAs' own shared memory (always added in the same order).  For problems of a few tiles: a
// 3x3 layer of one 14x14 image is two pixel tiles, whose K loop alone would keep a few SMs busy for longer than the
// whole call should take.
// FINE: fp32, 3x3 stride 1, BN <= 128.  The tensor core cuts the sum off when it adds to an accumulator in tensor memory, so
// the error of a sum grows with the number of MMAs that add into it (against 64 bits 1.9e-8 of the result each, always
// toward zero): 144 of them for 128 channels, where the transform kernels' GEMM has 32.  So the K loop runs in parts of
// p.chunk_groups channel groups, each afresh in the other accumulator buffer, and up to 64 output channels the two K steps of a tap
// have accumulators of their own; the epilogue adds all that up in registers, rounding to nearest.
// STEPPED: an int8 3x3 form, stride 1, on every step-th pixel of a larger input.  Compiled apart: a second row loop beside the plain one
// cost every call of these forms 0.1 us (7 x 64 -> 80 at 11x11 3.12 -> 3.25, 10 x 112 -> 64 at 13x9 3.57 -> 3.67), a test at every copy narrow
// tiles 2 to 3 %.
template <int KIND, int PAIRS, int FORM, bool STACK, bool PAIR, bool SPLIT, bool FINE, bool STEPPED>
__global__ void __launch_bounds__(KIND == HALO_I8 ? THREADS_I8 : THREADS_F32, 1)
conv_halo_kernel(const __grid_constant__ HaloArgs<planes_of(FORM), oc_of(KIND, SPLIT)> p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_aligned(smem_raw);
  constexpr int PLANES = KIND == HALO_I8 ? 1 : 2, EPI_WARPS = KIND == HALO_I8 ? EPI_WARPS_I8 : EPI_WARPS_F32;
  const int a_stage = p.a_bytes * PLANES;
  uint8_t *raw = smem + p.a_stages * a_stage;
  uint8_t *b_ring = raw + (KIND == HALO_F32 ? RAW_STAGES * p.raw_bytes : 0);
  float *s_scale = reinterpret_cast<float *>(b_ring + p.b_stages * p.b_stage_bytes);
  const int n_const = p.n_tiles * p.BN;
  float *s_shift = KIND == HALO_I8 ? s_scale + n_const : s_scale;
  Bars &bar = *reinterpret_cast<Bars *>(s_shift + n_const);
  volatile int *abort_flag = &bar.abort_flag;

  const int warp = uni(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  // this CTA's (pair's, cluster's) tiles
  const int share = SPLIT ? p.split : 1, first = PAIR ? blockIdx.x >> 1 : SPLIT ? blockIdx.x / share : blockIdx.x,
            step = PAIR ? gridDim.x >> 1 : SPLIT ? gridDim.x / share : gridDim.x;
  const int srank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  const int g0 = SPLIT ? p.groups * srank / share : 0, g1 = SPLIT ? p.groups * (srank + 1) / share : p.groups;
  // Set-up in two groups: the copying warps need the barriers only, and are on their way while the others allocate
  // tensor memory and load constants (pairs: everybody waits for the peer's barriers).
  const bool copies = warp == 0 || warp == 2;
  if (warp == 1) {
    for (int i = lane; i < MAX_B; i += 32) { mbar_init(&bar.bfull[i], 1); mbar_init(&bar.bempty[i], 1); }
    if (lane < MAX_A) {
      mbar_init(&bar.afull[lane], KIND == HALO_I8 ? 1 : SPLIT_WARPS * (PAIR ? 2 : 1));
      mbar_init(&bar.aempty[lane], 1);
    }
    if (lane < RAW_STAGES) { mbar_init(&bar.rfull[lane], 1); mbar_init(&bar.rempty[lane], SPLIT_WARPS); }
    if (lane < 2) mbar_init(&bar.turn[lane], 1);
    if (lane < MAX_BUFS) { mbar_init(&bar.tfull[lane], 1); mbar_init(&bar.tempty[lane], (KIND == HALO_I8 && p.spread ? EPI_WARPS : p.bufs == 4 ? 4 : 8) * (PAIR ? 2 : 1)); }
    if (lane == 31) { mbar_init(&bar.parts, 1); *abort_flag = 0; }
    fence_barrier_init();
    fence_proxy_async_smem();
    __syncwarp();
  } else if (warp == 0) {
    if (lane < p.planes) { tma_prefetch_desc(&p.tmap[lane][HALO_HEIGHTS - 1]); tma_prefetch_desc(&p.tmap[lane][3]); }
  } else if (warp >= EPI_WARP0 && warp < EPI_WARP0 + EPI_WARPS && p.fast != 1) {
    const int OCP = p.OCB * 16;
    for (int i = threadIdx.x - EPI_WARP0 * 32; i < n_const; i += EPI_WARPS * 32) {
      if (KIND == HALO_I8) s_scale[i] = i < OCP ? p.scale[i] : 0.0f;
      s_shift[i] = (i < OCP && p.shift) ? p.shift[i] : 0.0f;
    }
  }
  if (copies || warp == 1) named_bar_sync(1, 96);
  if (PAIR || !copies) {
    if (warp == 1) {
      if (PAIR) tmem_alloc2(&bar.tmem_slot, 512);
      else tmem_alloc(&bar.tmem_slot, 512);
    }
    tc_fence_before_sync();
    if (PAIR) {
      __syncthreads();
      cluster_sync_all();          // the peer's barriers exist before anyone signals them
    } else {
      named_bar_sync(2, blockDim.x - 64);
    }
    tc_fence_after_sync();
  }
  const uint32_t tmem_base = copies ? 0u : bar.tmem_slot;
  // (the kernel behind this one may set itself up now; see griddep_wait)
  if (threadIdx.x == 0) griddep_launch_dependents();
  int fail_code = 0;

  // ---- what the epilogue does with 16 output channels of a pixel
  struct Pixel { bool valid; size_t pix; const float *shift_row; };
  auto locate = [&](int mt, int row) {
    const int rt = p.div_col.div(mt), ct = mt - rt * p.col_tiles;
    const int v = rt * TILE_H + (row >> 3);
    const int n = p.div_period.div(v), oh = v - n * p.period, ow = ct * TILE_W + (row & 7);
    Pixel x;
    x.valid = n < p.N && oh < p.OH && ow < p.OW;
    x.pix = (static_cast<size_t>(n) * p.OCB * p.OH + oh) * p.OW + ow;
    x.shift_row = s_shift;
    if (KIND == HALO_I8 && p.shift_tbl && x.valid) {
      const int cls = __ldg(p.hclass + oh) * p.zp_nw + __ldg(p.wclass + ow);
      if (cls != p.zp_full) x.shift_row = p.shift_tbl + static_cast<size_t>(cls) * (p.OCB * 16);
    }
    return x;
  };
  auto emit = [&](const Pixel &px, int ocb, uint32_t (&r)[16], const uint4 *prev) {
    if (!px.valid || ocb >= p.OCB) return;
    const size_t off = (px.pix + ocb * (static_cast<size_t>(p.OH) * p.OW)) * 16;
    if (KIND == HALO_I8) {
      int a[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) a[i] = static_cast<int>(r[i]);
      if (p.acc_dump) {
        int4 *d = reinterpret_cast<int4 *>(p.acc_dump + off);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = make_int4(a[4 * i], a[4 * i + 1], a[4 * i + 2], a[4 * i + 3]);
      }
      if (p.fast == 2) requant_relu_u8(a, s_scale + ocb * 16, s_shift + ocb * 16, static_cast<uint8_t *>(p.out) + off);
      else if (oc_of(KIND, SPLIT) > 0 && p.fast) requant_relu_u8(a, p.cst[0] + ocb * 16, p.cst[1] + ocb * 16, static_cast<uint8_t *>(p.out) + off);
      else requant_store16(a, s_scale + ocb * 16, px.shift_row + ocb * 16, static_cast<uint8_t *>(p.out) + off * (p.rq.out_type == OUT_F32 ? 4 : 1), p.rq, prev);
    } else {
      float f[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(r[i]);
      float *o = static_cast<float *>(p.out) + off;
      if (p.shift) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 b = reinterpret_cast<const float4 *>(s_shift + ocb * 16)[i];
          f[4 * i] = __fadd_rn(f[4 * i], b.x); f[4 * i + 1] = __fadd_rn(f[4 * i + 1], b.y);
          f[4 * i + 2] = __fadd_rn(f[4 * i + 2], b.z); f[4 * i + 3] = __fadd_rn(f[4 * i + 3], b.w);
        }
      }
      if (p.rq.with_sum) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 b = reinterpret_cast<const float4 *>(o)[i];
          f[4 * i] = __fadd_rn(f[4 * i], b.x); f[4 * i + 1] = __fadd_rn(f[4 * i + 1], b.y);
          f[4 * i + 2] = __fadd_rn(f[4 * i + 2], b.z); f[4 * i + 3] = __fadd_rn(f[4 * i + 3], b.w);
        }
      }
      if (p.rq.relu) {
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = fminf(fmaxf(f[i], p.rq.relu_lo), p.rq.relu_hi);
      }
      if (p.wide) {
        store_v8(o, f, 0);
        store_v8(o, f, 8);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<float4 *>(o)[i] = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
      }
    }
  };
  const int part_pitch = p.BN / 4 + 1;      // SPLIT: 16-byte words per row of partial sums (odd: no bank conflicts)

  if (warp == 0) {
    // ---------------------------------------------------------------- activation rows
    griddep_wait();
    constexpr bool PAIR_A = PAIR && KIND == HALO_I8;      // (fp32 rows are split first: they count on their own CTA's barrier)
    uint64_t *full = KIND == HALO_I8 ? bar.afull : bar.rfull, *empty = KIND == HALO_I8 ? bar.aempty : bar.rempty;
    const int stages = KIND == HALO_I8 ? p.a_stages : RAW_STAGES;
    uint8_t *ring = KIND == HALO_I8 ? smem : raw;
    const int stage_bytes = KIND == HALO_I8 ? p.a_bytes : p.raw_bytes;
    const int planes = uni(p.planes), period = uni(p.period), pitch = uni(p.pitch), cb_step = uni(p.cb_step);
    constexpr bool PLAIN = KIND == HALO_I8 && (FORM == FORM_3X3_ROWS || FORM == FORM_3X3_TAPS || FORM == FORM_3X3_RESIDENT);
    const bool strided = FORM == FORM_3X3S2 || (PLAIN ? STEPPED : uni(p.strided) != 0);
    // stride 1: 8-byte elements, so that the copy engine moves whole rows
    const int x_unit = strided ? 1 : KIND == HALO_I8 ? 2 : 8;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = first; tile < p.total_tiles && ok; tile += step) {
      const int mt = PAIR ? 2 * p.div_n.div(tile) + rank : p.div_n.div(tile);
      const int rt = p.div_col.div(mt), ct = mt - rt * p.col_tiles;
      // Which copies bring this tile's rows, the same for every channel group; lane r stands for row r.  Rows of one
      // image go in one copy (lane 0 issues it).  A tile across images takes each image's share in pieces of 8, 4, 2
      // and 1 rows, issued by the lane of a piece's first row (a copy costs its issuer about 100 cycles).
      constexpr int Q = FORM == FORM_ANY || FORM == FORM_3X3S2 ? 4 : 1;      // planes the code is written out for
      int idx[Q], img[Q], row[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (Q > 1 && q >= planes) continue;
        const int rows = p.rows[q], v0 = rt * TILE_H + p.row0[q];
        int n = 0, h = v0;                        // (rows in front of the first image: zeros, like its padding)
        if (v0 > 0) { n = p.div_period.div(v0); h = v0 - n * period; }
        idx[q] = -1;
        if (h + rows <= period) {
          if (lane == 0) idx[q] = HALO_HEIGHTS - 1;
        } else {
          const int v = v0 + lane;
          n = v > 0 ? p.div_period.div(v) : 0;
          h = v - n * period;
          const int n_prev = __shfl_up_sync(0xFFFFFFFFu, n, 1);
          const uint32_t starts = __ballot_sync(0xFFFFFFFFu, lane == 0 || n != n_prev || lane == rows);
          if (lane < rows) {
            const int seg = 31 - __clz(starts & (0xFFFFFFFFu >> (31 - lane)));      // first row of this lane's image
            const uint32_t above = lane == 31 ? 0u : starts & (0xFFFFFFFEu << lane);
            const int len = (above ? __ffs(above) - 1 : rows) - seg, at = lane - seg;
            if (at < (len & ~7)) {
              if ((at & 7) == 0) idx[q] = 3;
            } else {
              const int sub = at & 7, rest = len - at;
              if (sub == 0 || (rest < (sub & -sub) && ((len & 7) & sub) == sub)) idx[q] = 31 - __clz(rest);
            }
          }
        }
        img[q] = n; row[q] = h;
      }
      for (int g = g0; g < g1 && ok; ++g) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (Q > 1 && (q >= planes || !ok)) continue;
          if (!wait_all(&empty[s], ph ^ 1u, abort_flag)) { ok = false; fail_code = ST_WAIT_TIMEOUT_PRODUCER; continue; }
          if (lane == 0 && (rank == 0 || !PAIR_A))
            mbar_arrive_expect_tx(&full[s], static_cast<uint32_t>(p.rows[q] * pitch) * (PAIR_A ? 2u : 1u));
          if (idx[q] >= 0) {
            uint8_t *d = ring + s * stage_bytes + lane * pitch;
            const int x = (ct * TILE_W + p.col0[q]) * x_unit, c = g * cb_step;
            if (PAIR_A) {
              const uint32_t pair_bar = mapa_u32(&full[s], 0);
              if (!strided) tma_tile_4d_pair(d, &p.tmap[0][idx[q]], x, c, row[q], img[q], pair_bar);
              else tma_tile_5d_pair(d, &p.tmap[q][idx[q]], 0, x, c, row[q], img[q], pair_bar);
            } else {
              if (!strided) tma_tile_4d(d, &p.tmap[0][idx[q]], x, c, row[q], img[q], &full[s]);
              else tma_tile_5d(d, &p.tmap[q][idx[q]], 0, x, c, row[q], img[q], &full[s]);
            }
          }
          __syncwarp();
          if (++s == stages) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------------- weights
    // (written before this launch's stream could reach it and never again: no griddep_wait)
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    const size_t group_bytes = static_cast<size_t>(p.ksteps) * p.kstep_bytes * (PAIR ? 2 : 1);
    for (int tile = first; tile < p.total_tiles && ok; tile += step) {
      const int nt = tile - p.div_n.div(tile) * p.n_tiles;
      const uint8_t *src = p.b_img + (static_cast<size_t>(nt) * p.groups + g0) * group_bytes;
      for (int g = g0; g < g1 && ok; ++g)
      for (int q = 0; q < p.planes && ok; ++q) {
        const int cols = p.tap_cols[q], row_steps = PAIRS == 0 ? (cols + 1) >> 1 : cols * PAIRS;
        const int units = p.row_units ? p.tap_rows[q] : p.tap_rows[q] * cols;
        const uint32_t bytes = static_cast<uint32_t>(p.row_units ? row_steps : PAIRS) * p.kstep_bytes;
        for (int u = 0; u < units; ++u) {
          if (!wait_all(&bar.bempty[s], ph ^ 1u, abort_flag)) { ok = false; fail_code = ST_WAIT_TIMEOUT_PRODUCER; break; }
          if (elect_one()) {
            if (PAIR) {      // (a stage in memory: the leader's half, the peer's half)
              if (rank == 0) mbar_arrive_expect_tx(&bar.bfull[s], 2 * bytes);
              tma_tile_2d_pair(b_ring + s * p.b_stage_bytes, &p.tmap_b, 0, static_cast<int>((src - p.b_img + rank * bytes) >> 9),
                               mapa_u32(&bar.bfull[s], 0));
            } else {
              mbar_arrive_expect_tx(&bar.bfull[s], bytes);
              tma_bulk_g2s(b_ring + s * p.b_stage_bytes, src, bytes, &bar.bfull[s]);
            }
          }
          __syncwarp();
          src += PAIR ? 2 * bytes : bytes;
          if (++s == p.b_stages) { s = 0; ph ^= 1u; }
        }
      }
      if (p.resident) break;
    }
  } else if (warp == 1 || warp == 3) {
    // ---------------------------------------------------------------- MMA issuers (pairs: the leader's)
    if (rank == 0) {
    constexpr bool STRAIGHT = FORM != FORM_ANY;
    constexpr int M = PAIR ? 2 * BM : BM, PXW = pxw_of(FORM, KIND, PAIRS), CHUNKS = PAIRS ? 2 * PAIRS : 1;
    const int BN = uni(p.BN), total = uni(p.total_tiles), groups = uni(p.groups), planes = FORM == FORM_3X3S2 ? 4 : STRAIGHT ? 1 : uni(p.planes),
              b_stages = uni(p.b_stages), a_stages = uni(p.a_stages), bufs = uni(p.bufs);
    const bool row_units = uni(p.row_units) != 0, resident = FORM == FORM_ANY ? uni(p.resident) != 0 : FORM == FORM_3X3_RESIDENT;
    const uint32_t idesc = KIND == HALO_I8 ? umma_idesc(2, 0, 1, M, BN) : umma_idesc(1, 2, 2, M, BN);
    const uint32_t idesc2 = umma_idesc(1, 2, 2, M, 2 * BN);
    // (in a cluster an address carries the CTA's rank in its upper bits; a descriptor takes the offset alone)
    const uint32_t a_base = (smem_u32(smem) >> 4) & 0x3FFFu, b_base = (smem_u32(b_ring) >> 4) & 0x3FFFu;
    // descriptors: low word = address | chunk distance << 16, high word = 8-row group distance | version
    const uint32_t pitch16 = STRAIGHT ? CHUNKS * PXW : uni(p.pitch) >> 4, pair16 = STRAIGHT ? 2 * PXW : 2u * uni(p.pxw);
    const uint32_t a_hi = pitch16 | (1u << 14), b_hi = (128u >> 4) | (1u << 14);
    const uint32_t b_lbo = static_cast<uint32_t>(STACK ? 2 * BN : PAIR ? BN / 2 : BN) << 16;
    const uint32_t ks16 = uni(p.kstep_bytes) >> 4, lo16 = uni(p.a_bytes) >> 4, a16 = lo16 * PLANES, b16 = uni(p.b_stage_bytes) >> 4;
    const uint32_t a_lbo = static_cast<uint32_t>(PAIRS == 0 ? 1 : pair16 >> 1) << 16;      // (one pixel / one chunk further)
    const uint32_t d_lo = KIND == HALO_F32 && uni(p.sep) != 0 ? BN : 0;      // columns of the lo products behind the others'
    const uint32_t d_alt = FINE && BN <= 64 ? 2 * BN : 0;                      // and of a tap's second K step
    auto desc = [](uint32_t lo, uint32_t hi) { return static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32); };
    const uint32_t el = elect_one() ? 1u : 0u;
    auto commit = [](uint64_t *b, uint32_t e) {
      if (PAIR) umma_commit_2cta_el(b, e);
      else umma_commit_el(b, e);
    };
    const int me = warp >> 1;      // this issuer takes tiles me, me + 2, ... of the CTA's
    // ring positions; the stages of the other issuer's tiles are skipped
    // (FINE: units of work are parts of tiles; part c has the groups from g0 + c * chunk_groups)
    const int own = SPLIT ? g1 - g0 : groups, chunk_groups = FINE ? uni(p.chunk_groups) : own, chunks = FINE ? (own + chunk_groups - 1) / chunk_groups : 1;
    const int b_tile = resident ? 0 : uni(p.b_per_tile), b_group = FINE ? b_tile / groups : 0;
    int as = 0, bs = 0, chunk = 0;
    uint32_t aph = 0, bph = 0;
    auto skip = [&]() {      // the unit behind this one
      const int next = FINE && chunk + 1 < chunks ? chunk + 1 : 0, n = FINE ? min(chunk_groups, own - next * chunk_groups) : groups;
      as += n * planes;
      while (as >= a_stages) { as -= a_stages; aph ^= 1u; }
      bs += FINE ? n * b_group : b_tile;
      while (bs >= b_stages) { bs -= b_stages; bph ^= 1u; }
    };
    auto next_b = [&]() {
      if (++bs == b_stages) { bs = 0; bph ^= 1u; }
    };
    int tile = first;
    auto advance = [&](int units) {
      if (FINE) {
        for (chunk += units; chunk >= chunks; chunk -= chunks) tile += step;
      } else {
        tile += units * step;
      }
    };
    if (me) {
      chunk = chunks - 1;      // (behind which comes the first unit)
      skip();
      chunk = 0;
      advance(1);
    }
    bool ok = true, b_ready = false;
    int t = me;
    for (; tile < total && ok; t += 2, skip(), advance(2)) {
      const uint32_t buf = t & (bufs - 1), tph = (bufs == 4 ? t >> 2 : t >> 1) & 1u, my_ph = (t >> 1) & 1u;
      const uint32_t d_tmem = tmem_base + buf * (bufs == 4 ? 128u : 256u);
      // An issuer looks at the rings only once the other has seen every stage of the tile before: a barrier tells
      // the last completed phase from the one before it, not from older ones.
      if ((t > 0 && !wait_all(&bar.turn[me], my_ph ^ (me ^ 1u), abort_flag)) ||
          !wait_all(&bar.tempty[buf], tph ^ 1u, abort_flag)) { ok = false; fail_code = ST_WAIT_TIMEOUT_MMA; break; }
      uint32_t acc = 0;
      const int gb = (SPLIT ? g0 : 0) + (FINE ? chunk * chunk_groups : 0), ge = FINE ? min(SPLIT ? g1 : groups, gb + chunk_groups) : SPLIT ? g1 : groups;
      for (int g = gb; g < ge && ok; ++g)
      for (int q = 0; q < planes && ok; ++q) {
        if (!wait_all(&bar.afull[as], aph, abort_flag)) { ok = false; fail_code = ST_WAIT_TIMEOUT_MMA; break; }
        if (resident && g == ge - 1 && q == planes - 1 && el) mbar_arrive(&bar.turn[me ^ 1u]);
        tc_fence_after_sync();
        uint32_t a_row = (a_base + as * a16) | a_lbo, b_lo = 0;
        auto mma = [&](uint32_t d, uint32_t al, uint32_t bl, uint32_t accumulate) {
          if (KIND == HALO_I8) {
            if (PAIR) umma_i8_2cta_el(d, desc(al, a_hi), desc(bl, b_hi), idesc, accumulate, el);
            else umma_i8_el(d, desc(al, a_hi), desc(bl, b_hi), idesc, accumulate, el);
          } else if (STACK) {
            // hi * [hi; lo] in one MMA of 2 * BN columns, lo * hi in one of BN (the first BN rows are hi), added to the
            // other lo products: the hi sum takes one addition per K step, and what is cut off the lo sum is 2^-11 of that
            umma_tf32_el(d, desc(al, a_hi), desc(bl, b_hi), idesc2, accumulate, el);
            umma_tf32_el(d + BN, desc(al + lo16, a_hi), desc(bl, b_hi), idesc, 1u, el);
          } else {
            // planes: the two hi chunks, then the two lo chunks
            const uint64_t bh = desc(bl, b_hi), blo = desc(bl + (ks16 >> 1), b_hi);
            auto one = [&](uint32_t dd, uint64_t ad, uint64_t bd, uint32_t ac) {
              if (PAIR) umma_tf32_2cta_el(dd, ad, bd, idesc, ac, el);
              else umma_tf32_el(dd, ad, bd, idesc, ac, el);
            };
            one(d + d_lo, desc(al + lo16, a_hi), bh, accumulate);
            one(d + d_lo, desc(al, a_hi), blo, 1u);
            one(d, desc(al, a_hi), bh, d_lo ? accumulate : 1u);
          }
        };
        // `n` taps from column c of the row at a_row (PAIRS = 0: n pairs of taps), unrolled
        auto taps = [&](auto n, int c) {
          constexpr int N = decltype(n)::value, P = PAIRS ? PAIRS : 1;
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < P; ++j)
              mma(FINE && j ? d_tmem + d_alt : d_tmem, a_row + c + i * (PAIRS ? 1 : 2) + j * pair16, b_lo + (i * P + j) * ks16,
                  (i | j) == 0 || (FINE && i == 0 && d_alt) ? acc : 1u);
          acc = 1u;
          b_lo += N * P * ks16;
        };
        constexpr int ROW_STEPS = PAIRS ? 3 : 2;      // of a 3x3 filter row, for taps()
        if constexpr (FORM == FORM_3X3_RESIDENT) {
          if (!b_ready)      // the first tile waits for the weights, stage by stage; after that they stay
            for (int i = 0; i < b_stages && ok; ++i) ok = wait_all(&bar.bfull[i], 0u, abort_flag);
          b_ready = true;
          b_lo = (b_base + (groups == 1 ? 0u : g * 3 * b16)) | b_lbo;
#pragma unroll
          for (int r = 0; r < 3; ++r, a_row += pitch16) taps(std::integral_constant<int, ROW_STEPS>{}, 0);
        } else if constexpr (STRAIGHT) {
          // R x C taps of the plane; a weight stage holds one tap or, FORM_3X3_ROWS, a row of them
          auto units = [&](auto r_const, auto c_const) {
            constexpr int C = decltype(c_const)::value, UNITS = decltype(r_const)::value * (FORM == FORM_3X3_ROWS ? 1 : C);
            bool seen = mbar_test_wait(&bar.bfull[bs], bph);
#pragma unroll
            for (int u = 0; u < UNITS; ++u) {
              if (!__all_sync(0xFFFFFFFFu, seen)) {
                ok = wait_all(&bar.bfull[bs], bph, abort_flag);
                if (!ok) break;
              }
              tc_fence_after_sync();
              b_lo = (b_base + bs * b16) | b_lbo;
              uint64_t *done = &bar.bempty[bs];
              next_b();
              // the next stage is tested in front of this one's MMAs, so the answer is there when they are issued
              if (u + 1 < UNITS) seen = mbar_test_wait(&bar.bfull[bs], bph);
              if (FORM == FORM_3X3_ROWS) taps(std::integral_constant<int, ROW_STEPS>{}, 0);
              else taps(std::integral_constant<int, 1>{}, u % C);
              commit(done, el);
              if (FORM == FORM_3X3_ROWS || u % C == C - 1) a_row += pitch16;
            }
          };
          using One = std::integral_constant<int, 1>;
          using Two = std::integral_constant<int, 2>;
          using Three = std::integral_constant<int, 3>;
          if constexpr (FORM == FORM_3X3S2) {
            if (q == 0) units(One{}, One{});
            else if (q == 1) units(One{}, Two{});
            else if (q == 2) units(Two{}, One{});
            else units(Two{}, Two{});
          } else if constexpr (FORM == FORM_1X1) {
            units(One{}, One{});
          } else {
            units(Three{}, Three{});
          }
        } else {
          const int rows = uni(p.tap_rows[q]), cols = uni(p.tap_cols[q]);
          auto begin_unit = [&]() {
            ok = wait_all(&bar.bfull[bs], resident ? 0u : bph, abort_flag);
            tc_fence_after_sync();
            b_lo = (b_base + bs * b16) | b_lbo;
          };
          auto end_unit = [&]() {
            if (!resident) commit(&bar.bempty[bs], el);
            next_b();
          };
          if (row_units) {
            const int steps = PAIRS ? cols : (cols + 1) >> 1;
#pragma unroll 1
            for (int r = 0; r < rows; ++r, a_row += pitch16) {
              begin_unit();
              if (!ok) break;
#pragma unroll 1
              for (int c = 0; c < steps; c += 4) {
                const int at = PAIRS ? c : 2 * c;
                switch (min(steps - c, 4)) {
                  case 1: taps(std::integral_constant<int, 1>{}, at); break;
                  case 2: taps(std::integral_constant<int, 2>{}, at); break;
                  case 3: taps(std::integral_constant<int, 3>{}, at); break;
                  default: taps(std::integral_constant<int, 4>{}, at);
                }
              }
              end_unit();
            }
          } else {
#pragma unroll 1
            for (int r = 0; r < rows && ok; ++r, a_row += pitch16)
#pragma unroll 1
              for (int c = 0; c < cols; ++c) {
                begin_unit();
                if (!ok) break;
                taps(std::integral_constant<int, 1>{}, c);
                end_unit();
              }
          }
        }
        if (!ok) { fail_code = ST_WAIT_TIMEOUT_MMA; break; }
        commit(&bar.aempty[as], el);
        if (++as == a_stages) { as = 0; aph ^= 1u; }
      }
      if (resident) bs = 0;
      if (ok) commit(&bar.tfull[buf], el);
      if (!resident && el) mbar_arrive(&bar.turn[me ^ 1u]);
      __syncwarp();
    }
    }
  } else if (KIND == HALO_F32 && warp >= SPLIT_WARP0) {
    // ---------------------------------------------------------------- fp32 rows -> tf32 hi / lo planes
    // hi = round-to-nearest tf32(x), lo = x - hi (exact); done once per pixel, used by every tap
    const int tid = threadIdx.x - SPLIT_WARP0 * 32;
    int rs = 0, as = 0;
    uint32_t rph = 0, aph = 0;
    bool ok = true;
    for (int tile = first; tile < p.total_tiles && ok; tile += step) {
      for (int g = g0; g < g1 && ok; ++g)
      for (int q = 0; q < p.planes; ++q) {
        const int items = p.rows[q] * p.pxw * 4;       // 16-byte pieces: [row][pixel][4 chunks]
        if (!wait_all(&bar.rfull[rs], rph, abort_flag) || !wait_all(&bar.aempty[as], aph ^ 1u, abort_flag)) {
          ok = false; fail_code = ST_WAIT_TIMEOUT_MMA; break;
        }
        const float4 *src = reinterpret_cast<const float4 *>(raw + rs * p.raw_bytes);
        uint8_t *hi = smem + as * a_stage;
        // (four pieces per thread in flight: one at a time a round trip through shared memory and the
        // conversions was about 110 cycles)
#pragma unroll 4
        for (int i = tid; i < items; i += SPLIT_WARPS * 32) {
          const float4 v = src[i];
          const int px_all = i >> 2, c = i & 3;
          const int row = p.div_px.div(px_all), px = px_all - row * p.pxw;
          const float x[4] = {v.x, v.y, v.z, v.w};
          float h[4], l[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t hb;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(x[j]));
            h[j] = __uint_as_float(hb);
            l[j] = __fsub_rn(x[j], h[j]);
          }
          uint8_t *d = hi + row * p.pitch + (c * p.pxw + px) * 16;
          *reinterpret_cast<float4 *>(d) = make_float4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<float4 *>(d + p.a_bytes) = make_float4(l[0], l[1], l[2], l[3]);
        }
        fence_proxy_async_smem();      // these stores -> visible to the tensor core's reads
        __syncwarp();
        if (lane == 0) {
          if (PAIR && rank) mbar_arrive_cluster(mapa_u32(&bar.afull[as], 0));
          else mbar_arrive(&bar.afull[as]);
          mbar_arrive(&bar.rempty[rs]);
        }
        if (++rs == RAW_STAGES) { rs = 0; rph ^= 1u; }
        if (++as == p.a_stages) { as = 0; aph ^= 1u; }
      }
    }
  } else if (warp >= EPI_WARP0 && warp < EPI_WARP0 + EPI_WARPS) {
    // ---------------------------------------------------------------- epilogue: one output pixel per thread
    // int8: group g of four warps serves accumulator g of four, or column half g & 1 of accumulator g >> 1 of two, or
    // (HaloParams::spread) a quarter of the columns of every tile.  (A third value of the step, or this loop compiled twice,
    // costs 2 to 4 % on other layers.)
    const int quarter = warp & 3, group = (warp - EPI_WARP0) >> 2;
    const bool four = p.bufs == 4, spread = KIND == HALO_I8 && p.spread != 0, whole = four || spread, sep = STACK || (KIND == HALO_F32 && PAIR && p.sep);
    const int row = quarter * 32 + lane;
    const int nb16 = p.BN >> 4, share = (nb16 + 3) >> 2;
    const int half = spread ? group * share : whole ? 0 : group & 1, blk_step = whole ? 1 : 2;      // first block of columns, step
    const int cnt = spread ? min(share, nb16 - half) : whole ? nb16 : (nb16 - half + 1) >> 1;
    const int t_step = KIND == HALO_F32 || spread ? 1 : p.bufs, t_shift = four ? 2 : 1;
    int t = KIND == HALO_F32 || spread ? 0 : four ? group : group >> 1;
    bool ok = true;
    // the residual this tile adds: on its way to L2 while the MMAs run
    auto prefetch_residual = [&](const Pixel &px, int nt) {
      if (!p.rq.with_sum || !px.valid) return;
      const int elt = KIND == HALO_F32 || p.rq.out_type == OUT_F32 ? 4 : 1;
      for (int k = 0; k < cnt; ++k) {
        const int ocb = nt * nb16 + half + blk_step * k;
        if (ocb < p.OCB)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint8_t *>(p.out) +
                                                        (px.pix + ocb * (static_cast<size_t>(p.OH) * p.OW)) * 16 * elt));
      }
    };
    auto release = [&](uint32_t buf) {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && rank) mbar_arrive_cluster(mapa_u32(&bar.tempty[buf], 0));
        else mbar_arrive(&bar.tempty[buf]);
      }
    };
    auto finish = [&](const Pixel &px, int nt, int blk, uint32_t (&r)[16], const uint4 *pv) {
      if (SPLIT) {      // (every copy into the rings has landed and every MMA has read them: the space is free)
        uint4 *d = reinterpret_cast<uint4 *>(smem) + row * part_pitch + blk * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
      } else {
        emit(px, nt * nb16 + blk, r, pv);
      }
    };
    if constexpr (FINE) {
      for (int tile = first; tile < p.total_tiles && ok; tile += step) {
        const int mu = p.div_n.div(tile), nt = tile - mu * p.n_tiles, mt = PAIR ? 2 * mu + rank : mu;
        const Pixel px = SPLIT ? Pixel{} : locate(mt, row);
        if (!SPLIT) prefetch_residual(px, nt);
        float sum[4][16];      // (BN <= 128: at most four blocks per warp)
        const int ways = p.BN <= 64 ? 2 : 1;
        for (int g = g0, c = 0; g < g1; g += p.chunk_groups, ++c, ++t) {
          const uint32_t buf = t & 1;
          if (!wait_all(&bar.tfull[buf], (t >> 1) & 1u, abort_flag)) { ok = false; fail_code = ST_WAIT_TIMEOUT_EPILOGUE; break; }
          tc_fence_after_sync();
          const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * 256u + half * 16;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (k >= cnt) continue;
#pragma unroll 1
            for (int w = 0; w < ways; ++w) {
              uint32_t r[16], q[16];
              tmem_ld16(t_addr + 2 * w * p.BN + k * 32, r);
              tmem_ld16(t_addr + (2 * w + 1) * p.BN + k * 32, q);
              tmem_ld_wait16(r);
              tmem_ld_wait16(q);
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const float v = __fadd_rn(__uint_as_float(r[i]), __uint_as_float(q[i]));
                sum[k][i] = (c | w) == 0 ? v : __fadd_rn(sum[k][i], v);
              }
            }
          }
          release(buf);
        }
        if (!ok) break;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k >= cnt) continue;
          uint32_t r[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(sum[k][i]);
          finish(px, nt, half + 2 * k, r, nullptr);
        }
      }
    } else
    for (int tile = first + t * step; tile < p.total_tiles && ok; tile += t_step * step, t += t_step) {
      const int mu = p.div_n.div(tile), nt = tile - mu * p.n_tiles, mt = PAIR ? 2 * mu + rank : mu;
      const Pixel px = SPLIT ? Pixel{} : locate(mt, row);
      const uint32_t buf = t & (p.bufs - 1), tph = (t >> t_shift) & 1u;
      if (!SPLIT) prefetch_residual(px, nt);
      if (!wait_all(&bar.tfull[buf], tph, abort_flag)) { ok = false; fail_code = ST_WAIT_TIMEOUT_EPILOGUE; break; }
      tc_fence_after_sync();
      const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * (four ? 128u : 256u) + half * 16;
      auto take = [&](int blk, uint32_t (&r)[16], uint32_t (&r2)[16], const uint4 &pv) {
        if (sep) {
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__fadd_rn(__uint_as_float(r[i]), __uint_as_float(r2[i])));
        }
        finish(px, nt, blk, r, KIND == HALO_I8 ? &pv : nullptr);
      };
      // int8: the stored output that block k adds, fetched a block ahead
      const bool add = KIND == HALO_I8 && !SPLIT && p.rq.with_sum && px.valid;
      auto residual = [&](int k, uint4 &pv) {
        const int ocb = nt * nb16 + half + blk_step * k;
        if (add && ocb < p.OCB)
          pv = *reinterpret_cast<const uint4 *>(static_cast<const uint8_t *>(p.out) + (px.pix + ocb * (static_cast<size_t>(p.OH) * p.OW)) * 16);
      };
      // blocks half, half + blk_step, ... of this warp, two in flight: while one is converted and stored the next is
      // on its way out of tensor memory
      uint32_t r0[16], r1[16], q0[16], q1[16];
      uint4 pv0 = make_uint4(0, 0, 0, 0), pv1 = pv0;
      auto load = [&](int k, uint32_t (&r)[16], uint32_t (&q)[16]) {
        tmem_ld16(t_addr + k * (16 * blk_step), r);
        if (sep) tmem_ld16(t_addr + p.BN + k * (16 * blk_step), q);
      };
      if (cnt > 0) { load(0, r0, q0); residual(0, pv0); }
#pragma unroll 1
      for (int k = 0; k < cnt; k += 2) {
        tmem_ld_wait16(r0);
        if (sep) tmem_ld_wait16(q0);
        if (k + 1 < cnt) { load(k + 1, r1, q1); residual(k + 1, pv1); }
        take(half + blk_step * k, r0, q0, pv0);
        if (k + 1 < cnt) {
          tmem_ld_wait16(r1);
          if (sep) tmem_ld_wait16(q1);
          if (k + 2 < cnt) { load(k + 2, r0, q0); residual(k + 2, pv0); }
          take(half + blk_step * (k + 1), r1, q1, pv1);
        }
      }
      release(buf);
    }
  }

  if (fail_code != 0) report_status(p.status, fail_code);
  if (SPLIT) {
    // Every CTA finishes a share of the tile's rows.  The rows' partial sums travel as one bulk copy from each CTA
    // into a second area behind the first (loads of remote shared memory took 12 us here: 16 bytes of another row per
    // lane), once every CTA is done with its rings; they are added in rank order.
    const int nb16 = p.BN >> 4, rows = BM / share;
    const uint32_t part_bytes = static_cast<uint32_t>(rows * part_pitch) * 16;
    uint8_t *inbox = smem + BM * part_pitch * 16;
    fence_proxy_async_smem();
    __syncthreads();
    cluster_sync_all();
    if (warp == 0) {
      if (lane == 0) mbar_arrive_expect_tx(&bar.parts, part_bytes * share);
      __syncwarp();
      if (lane < share)
        bulk_s2cluster(mapa_u32(inbox + srank * part_bytes, lane), smem + lane * part_bytes, part_bytes, mapa_u32(&bar.parts, lane));
    }
    if (warp >= EPI_WARP0 && warp < EPI_WARP0 + EPI_WARPS) {
      const int mt = p.div_n.div(first), nt = first - mt * p.n_tiles;
      if (wait_all(&bar.parts, 0u, abort_flag)) {
        for (int i = threadIdx.x - EPI_WARP0 * 32; i < rows * nb16; i += EPI_WARPS * 32) {
          const int row = i & (rows - 1), blk = i / rows;
          const uint4 *src = reinterpret_cast<const uint4 *>(inbox) + row * part_pitch + blk * 4;
          uint32_t sum[16];
          for (int c = 0; c < share; ++c, src += rows * part_pitch) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 v = src[j];
              const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int k = 0; k < 4; ++k)
                sum[4 * j + k] = c == 0 ? x[k] : KIND == HALO_I8 ? sum[4 * j + k] + x[k]
                                               : __float_as_uint(__fadd_rn(__uint_as_float(sum[4 * j + k]), __uint_as_float(x[k])));
            }
          }
          emit(locate(mt, srank * rows + row), nt * nb16 + blk, sum, nullptr);
        }
      } else {
        report_status(p.status, ST_WAIT_TIMEOUT_EPILOGUE);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR || SPLIT) cluster_sync_all();      // nobody leaves (or frees tensor memory) while the other CTA may still use it
  tc_fence_after_sync();
  if (warp == 1) {
    if (PAIR) tmem_dealloc2(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

int alignup(int v, int a) { return (v + a - 1) / a * a; }

// Modelled cycles of one K step: the tensor pipe (N / 2 per MMA of 128 or 256 x N x 32 bytes), the shared-memory
// port at 128 B/clk (operand reads of the MMAs, incoming copies, fp32: the split), the SM's intake from L2 at
// about 48 B/clk.  b: bytes of weights an SM takes in per K step (0: resident), a: of input.
double kstep_cycles(int kind, int BN, bool pair, double b, double a, bool strided = false) {
  const double read_n = BN / (pair ? 8.0 : 4.0);
  double tensor, port;
  if (kind == HALO_I8) { tensor = BN / 2.0; port = 32 + read_n; }
  else if (!pair && BN <= 128) { tensor = 1.5 * BN; port = 64 + 3 * read_n; }      // (stacked hi / lo rows)
  else { tensor = 1.5 * BN; port = 3 * (32 + read_n); }
  port += (b + a * (kind == HALO_F32 ? 4 : 1)) / 128;
  // (a parity plane of int8 arrives 16 bytes at a time)
  return std::max(std::max(tensor, port), b / 48 + a / (strided && kind == HALO_I8 ? 16 : 48));
}

int tap_form(const HaloPlan &hp);

}  // namespace

bool halo_plan(HaloPlan &hp, int kind, int n, int ic, int oc, int ih, int iw, int oh, int ow, int kh, int kw, int stride,
               int pad_t, int pad_l, int num_sms, std::string &err, int max_acc) {
  HaloParams &p = hp.p;
  hp.kind = kind; hp.stride = stride; hp.IH = ih; hp.IW = iw;
  hp.CB = (ic + 15) / 16;
  p.OCB = (oc + 15) / 16;
  if (stride < 1 || stride > 2 || ih < stride || iw < stride) { err = "stride"; return false; }
  p.N = n; p.OH = oh; p.OW = ow; p.strided = stride > 1;
  auto fdiv = [](int e, int s) { return e >= 0 ? e / s : -((-e + s - 1) / s); };
  // which parity plane each tap reads, and by how many rows / columns it shifts there
  const int taps = kh * kw;
  std::vector<int> plane(taps), dr(taps), dc(taps);
  int rmin[4], rmax[4], cmin[4], cmax[4];
  for (int i = 0; i < 4; ++i) { rmin[i] = cmin[i] = 1 << 20; rmax[i] = cmax[i] = -(1 << 20); }
  for (int t = 0; t < taps; ++t) {
    const int eh = t / kw - pad_t, ew = t % kw - pad_l;
    dr[t] = fdiv(eh, stride); dc[t] = fdiv(ew, stride);
    plane[t] = (eh - dr[t] * stride) * stride + (ew - dc[t] * stride);
    const int q = plane[t];
    rmin[q] = std::min(rmin[q], dr[t]); rmax[q] = std::max(rmax[q], dr[t]);
    cmin[q] = std::min(cmin[q], dc[t]); cmax[q] = std::max(cmax[q], dc[t]);
  }
  int span_c = 0, rows = 0, period = oh;
  p.planes = 0;
  for (int q = 0; q < stride * stride; ++q) {
    if (rmin[q] > rmax[q]) continue;
    if (rmin[q] < -24 || rmax[q] > 24) { err = "padding"; return false; }
    const int i = p.planes++;
    hp.parity[i] = q;
    p.row0[i] = rmin[q]; p.rows[i] = TILE_H + rmax[q] - rmin[q]; p.col0[i] = cmin[q];
    span_c = std::max(span_c, cmax[q] - cmin[q]);
    if (p.rows[i] > 32) { err = "filter height"; return false; }
    rows = std::max(rows, p.rows[i]);
    // Stacked images: the rows above image i are read as rows period + d of image i - 1 and must lie outside
    // it (zeros); the rows below its last output row must not reach image i + 1.
    const int hp_rows = (ih - q / stride + stride - 1) / stride;
    if (rmax[q] > 0) period = std::max(period, oh + rmax[q]);
    if (rmin[q] < 0) period = std::max(period, hp_rows - rmin[q]);
  }
  p.period = period;
  p.div_period.set(period);
  // (the kernel's row numbers, up to a tile and its halo past the last image, are 32-bit)
  if (static_cast<long long>(n) * period + 64 > 0x7FFFFFFFll) { err = "size"; return false; }
  // Channel groups.  fp32: one 16-channel block (four chunks).  int8: an even number of blocks, at most eight,
  // that wastes the fewest chunks past the last block (narrow groups cost more hand-overs per MMA), or one.
  int kch = 4;
  if (kind == HALO_I8) {
    double best_k = 0;
    kch = 0;
    for (int k = 8; k >= 2; k -= 2) {
      if (k > 2 && k - 2 >= hp.CB) continue;
      if (rows * alignup((TILE_W + span_c) * k, 8) * 16 > 48 * 1024) continue;
      const double c = static_cast<double>((hp.CB + k - 1) / k) * (k + 0.5);
      if (kch == 0 || c < best_k) { best_k = c; kch = k; }
    }
    if (hp.CB == 1 || kch == 0) kch = 1;
  }
  int pxw = TILE_W + span_c + (kch == 1 && !(span_c & 1));      // (the last tap of an odd row pairs up with a zero weight)
  while ((kind == HALO_F32 ? pxw * 64 : kch * pxw * 16) % 128) ++pxw;      // (a TMA destination is 128-byte aligned)
  if (pxw > 32) { err = "filter width"; return false; }
  p.kch = kch; p.pxw = pxw;
  p.div_px.set(pxw);
  p.pitch = kch * pxw * 16;
  p.a_bytes = rows * p.pitch;
  if (p.a_bytes > 48 * 1024) { err = "filter size"; return false; }
  p.cb_step = kind == HALO_F32 ? 1 : kch;
  p.groups = kind == HALO_F32 ? hp.CB : (hp.CB + kch - 1) / kch;
  p.raw_bytes = kind == HALO_F32 ? p.a_bytes : 0;
  // K steps in the order the issuer takes them: two chunks each
  hp.order.clear();
  p.ksteps = 0;
  for (int i = 0; i < p.planes; ++i) {
    const int q = hp.parity[i], ph = q / stride, pw = q % stride;
    p.tap_rows[i] = rmax[q] - rmin[q] + 1; p.tap_cols[i] = cmax[q] - cmin[q] + 1;
    for (int r = 0; r < p.tap_rows[i]; ++r)
      for (int c = 0; c < p.tap_cols[i]; c += kch == 1 ? 2 : 1) {
        const int t = ((rmin[q] + r) * stride + ph + pad_t) * kw + (cmin[q] + c) * stride + pw + pad_l;
        if (kch == 1) {
          hp.order.push_back({t, 0});
          if (c + 1 < p.tap_cols[i]) hp.order.push_back({t + stride, 0});
          else hp.order.push_back({-1, 0});
        } else {
          for (int b = 0; b < kch; ++b) hp.order.push_back({t, b});
        }
      }
  }
  p.ksteps = static_cast<int>(hp.order.size()) / 2;
  // tile width: the smallest modelled time over the whole chip
  const int OCP = p.OCB * 16;
  p.row_tiles = (static_cast<int>((static_cast<long long>(n - 1) * period) + oh) + TILE_H - 1) / TILE_H;
  p.col_tiles = (ow + TILE_W - 1) / TILE_W;
  const double m_tiles = static_cast<double>(p.row_tiles) * p.col_tiles;
  if (m_tiles * p.OCB > 1e9 || OCP > HALO_MAX_OC) { err = "size"; return false; }
  const int planes_bytes = p.a_bytes * (kind == HALO_F32 ? 2 : 1);
  const int pairs = kch / 2;
  const double group_min = kind == HALO_F32 ? 1900 : 0;      // the way of a stage through the split, where a filter has few taps to hide it
  double best = 0;
  p.BN = 0;
  for (int nt = (OCP + 255) / 256; nt <= p.OCB; ++nt) {
    const int BN = alignup((OCP + nt - 1) / nt, 16);
    if ((OCP + BN - 1) / BN != nt) continue;
    const double kb = BN * (kind == HALO_F32 ? 64.0 : 32.0), ab = static_cast<double>(p.a_bytes) * p.planes / p.ksteps;
    const double all = kb * p.ksteps * p.groups;
    const bool stays = nt == 1 && all + 2.0 * planes_bytes + 8192 + BN * 8 <= SMEM_LIMIT - RAW_STAGES * p.raw_bytes;
    // (int8: the epilogue, about 9 outputs per clock)
    const double epilogue = kind == HALO_I8 ? 400 + 128.0 * BN / 9 : 0;
    // fp32: does max_acc allow `groups` channel groups per CTA, and if only in parts (FINE), how many groups in each?
    struct Parts { bool ok; int fine, groups, count; };
    auto parts_of = [&](int groups) -> Parts {
      if (!max_acc || p.ksteps * (BN <= 128 ? 1 : 3) * groups <= max_acc) return {true, 0, groups, 1};
      const int each = std::min(groups, max_acc / (BN <= 64 ? p.ksteps / 2 : p.ksteps));
      if (BN > 128 || stride != 1 || kh != 3 || kw != 3 || each == 0) return {false, 0, 0, 0};
      return {true, 1, each, (groups + each - 1) / each};
    };
    for (int pair = 0; pair < 2; ++pair) {
      // pairs take the weights tap by tap, in rows of 512 bytes per half
      // (with a stride the CTAs wait for one another at every parity plane: 128 -> 256, 56x56: fp32 150 -> 180 us, int8
      // with a residual 27.8 -> 29.9; 512 -> 512, 14x14: 13.3 -> 17.5)
      if (pair && (stride > 1 || pairs < 2 || BN % 32 || stays || m_tiles < 2 || kb * pairs > 48 * 1024 || kb * pairs * 3 <= 24 * 1024)) continue;
      const Parts parts = parts_of(p.groups);
      if (!parts.ok) continue;
      const double b = stays ? 0.0 : pair ? kb / 2 : kb;
      const double loop = std::max(kstep_cycles(kind, BN, pair != 0, b, ab, stride > 1) * p.ksteps, group_min) * p.groups + 600 + 300 * (parts.count - 1);
      const double tile = std::max(loop, epilogue);
      const double waves = pair ? std::ceil(std::ceil(m_tiles / 2) * nt / (num_sms / 2)) : std::ceil(m_tiles * nt / num_sms);
      const double t = waves * tile + 4000;
      if (p.BN == 0 || t < best * 0.98) { best = t; hp.loop_ratio = loop / std::max(epilogue, 1.0); hp.gather_ratio = ab / 16 / kstep_cycles(kind, BN, pair != 0, 0, 0); p.BN = BN; p.n_tiles = nt; p.pair = pair; p.split = 1; p.fine = parts.fine; p.chunk_groups = parts.groups; }
    }
    // few tiles: several CTAs share the K loop of each.  Partial sums cross shared memories at about 9 B/clk.  An SM
    // holds one CTA, and the device no more clusters than its GPCs have room for (15 of 8, 33 of 4).
    for (int split = 2; split <= 8 && split <= p.groups && m_tiles * nt * split <= num_sms * (split == 8 ? 0.8 : 0.88); split *= 2) {
      const double sums = 128.0 * (BN + 4) * 4;
      const Parts parts = parts_of((p.groups + split - 1) / split);
      if (kch == 1 || 2 * sums > 150 * 1024 || !parts.ok) continue;
      const double t = std::max(kstep_cycles(kind, BN, false, kb, ab, stride > 1) * p.ksteps, group_min) * ((p.groups + split - 1) / split) + 600 +
                       4000 + 2000 + sums / 9 + 300 * (parts.count - 1);
      if (t < best * 0.95) { best = t; hp.gather_ratio = ab / 16 / kstep_cycles(kind, BN, false, 0, 0); p.BN = BN; p.n_tiles = nt; p.pair = 0; p.split = split; p.fine = parts.fine; p.chunk_groups = parts.groups; }
    }
  }
  if (p.BN == 0) { err = "precision"; return false; }
  hp.est_us = best / 1750;
  p.stack = kind == HALO_F32 && p.BN <= 128 && !p.pair;
  p.sep = kind == HALO_F32 && p.BN <= 128;
  p.bufs = kind == HALO_I8 && p.BN <= 128 ? 4 : 2;      // accumulators in the 512 columns of tensor memory
  p.div_n.set(p.n_tiles);
  p.div_col.set(p.col_tiles);
  // shared memory: operand rows first, the rest is the weight ring
  p.kstep_bytes = p.BN * (kind == HALO_F32 ? 64 : 32) / (p.pair ? 2 : 1);      // (of one CTA)
  const int fixed = p.n_tiles * p.BN * (kind == HALO_F32 ? 4 : 8) + static_cast<int>(sizeof(Bars)) + 256;
  const int room = SMEM_LIMIT - fixed - RAW_STAGES * p.raw_bytes;
  int b_per_group = 0, most_c = 0;      // weight stages of a channel group; longest filter row
  for (int i = 0; i < p.planes; ++i) most_c = std::max(most_c, p.tap_cols[i]);
  const int row_steps = kch == 1 ? (most_c + 1) / 2 : most_c * pairs;
  // a stage costs its hand-over whatever it holds: whole filter rows while they are small
  auto set_units = [&](bool rows_of_taps) {
    p.row_units = rows_of_taps;
    b_per_group = 0;
    for (int i = 0; i < p.planes; ++i) b_per_group += p.row_units ? p.tap_rows[i] : p.tap_rows[i] * p.tap_cols[i];
    p.b_per_tile = b_per_group * p.groups;
    p.b_stage_bytes = (p.row_units ? row_steps : pairs) * p.kstep_bytes;
  };
  auto fit_b = [&](int a_stages) -> bool {
    p.a_stages = a_stages;
    p.b_stages = std::min(MAX_B, (room - a_stages * planes_bytes) / p.b_stage_bytes);
    return p.b_stages >= 1;
  };
  const long long b_all = static_cast<long long>(p.groups) * p.ksteps * p.kstep_bytes;
  p.resident = 0;
  if (p.n_tiles == 1 && !p.pair && p.split == 1 && b_all <= room - 2ll * planes_bytes) {
    // the whole filter fits: it is fetched once per CTA
    set_units(true);
    for (int a = MAX_A; a >= 2 && !p.resident; --a)
      if (a * static_cast<long long>(planes_bytes) + b_all <= room) {
        fit_b(a);
        if (p.groups * b_per_group <= MAX_B && p.groups * b_per_group <= p.b_stages) {
          p.resident = 1;
          p.b_stages = p.groups * b_per_group;
        }
      }
  }
  if (kind == HALO_I8 && p.resident && taps == 1 && stride == 1 && p.groups > 1) {
    // The issuer's general loop serves these, and a channel group takes it 650 to 1000 cycles whatever the tile: 49 x 149 -> 16 at 41x66
    // (five groups) modelled as 7.0 us takes 20.9, 9 x 144 -> 32 at 72x114 5.2 / 12.2.
    const double epilogue = 400 + 128.0 * p.BN / 9, loop = hp.loop_ratio * epilogue, slow = std::max(loop, 600.0 * p.groups);
    hp.est_us += std::ceil(m_tiles / num_sms) * (std::max(slow, epilogue) - std::max(loop, epilogue)) / 1750;
    hp.loop_ratio = slow / epilogue;
  }
  if (!p.resident) {
    const int form = tap_form(hp);
    set_units(!p.pair && form != FORM_3X3S2 && form != FORM_1X1 && (kch == 1 || row_steps * p.kstep_bytes <= 24 * 1024));
    // Ring depths.  A stage comes back about 4500 cycles after the MMAs that read it were issued (their end, the
    // hand-overs, the copy); weights, which wait for nothing else, 3000.  An operand stage may last only a few
    // hundred cycles (a parity plane, a 1x1 filter).  fp32 rows have the raw ring in front.
    const double k_cyc = kstep_cycles(kind, p.BN, p.pair != 0, 0, 0);
    const double a_cyc = k_cyc * p.ksteps / p.planes, b_cyc = k_cyc * p.ksteps / b_per_group;
    const int a_min = planes_bytes <= 24 * 1024 ? 3 : 2;
    const int a_want = kind == HALO_F32 ? a_min : std::max(a_min, std::min(MAX_A, 1 + static_cast<int>(std::ceil(4500 / a_cyc))));
    const int b_want = std::max(3, std::min(8, static_cast<int>(std::ceil(3000 / b_cyc))));
    bool ok = false;
    for (int a = a_want; a > a_min && !ok; --a) ok = fit_b(a) && p.b_stages >= b_want;
    for (int a = a_min; a >= 1 && !ok; --a) ok = fit_b(a) && p.b_stages >= 3;
    if (!ok) { err = "shared memory"; return false; }
  }
  if (p.split > 1 && 2 * 128 * (p.BN + 4) * 4 > p.a_stages * planes_bytes + RAW_STAGES * p.raw_bytes + p.b_stages * p.b_stage_bytes) {
    err = "shared memory";      // (the partial sums take the rings' place)
    return false;
  }
  hp.smem_bytes = static_cast<size_t>(p.a_stages) * planes_bytes + RAW_STAGES * static_cast<size_t>(p.raw_bytes) +
                  static_cast<size_t>(p.b_stages) * p.b_stage_bytes + fixed;
  hp.b_bytes = static_cast<size_t>(p.n_tiles) * b_all * (p.pair ? 2 : 1);
  return true;
}

// [n tile][group][K step]: single CTAs: the BN rows of both chunks (fp32: hi and lo rows); pairs: the K steps of
// one tap for the leader's BN / 2 rows, then for the peer's.
template <typename PutChunk>
static void pack_walk(const HaloPlan &hp, uint8_t *dst, PutChunk put) {
  const HaloParams &p = hp.p;
  const int halves = p.pair ? 2 : 1, rows = p.BN / halves, unit = p.pair ? (hp.kind == HALO_F32 ? 2 : p.kch / 2) : 1;
  const size_t group_bytes = static_cast<size_t>(p.ksteps) * p.kstep_bytes * halves;
  host::parallel_for(p.n_tiles * p.groups, group_bytes * p.n_tiles * p.groups, [&](int i) {
    const int nt = i / p.groups, g = i - nt * p.groups;
    uint8_t *at = dst + i * group_bytes;
    for (int k0 = 0; k0 < p.ksteps; k0 += unit)
      for (int h = 0; h < halves; ++h)
        for (int k = k0; k < k0 + unit; ++k, at += p.kstep_bytes)
          for (int j = 0; j < 2; ++j) put(at, j, hp.order[2 * k + j], g, nt * p.BN + h * rows, rows);
  });
}

std::vector<uint8_t> halo_pack_i8(const HaloPlan &hp, const int8_t *q, int OCP, int taps, int ICP) {
  std::vector<uint8_t> img(hp.b_bytes, 0);
  pack_walk(hp, img.data(), [&](uint8_t *dst, int j, HaloPlan::Chunk c, int g, int o0, int rows) {
    const int cb = g * hp.p.kch + c.cb;
    if (c.tap < 0 || cb >= hp.CB) return;
    for (int r = 0; r < rows && o0 + r < OCP; ++r)
      std::memcpy(dst + (j * rows + r) * 16, q + (static_cast<size_t>(o0 + r) * taps + c.tap) * ICP + cb * 16, 16);
  });
  return img;
}

std::vector<uint8_t> halo_pack_f32(const HaloPlan &hp, const float *u, int OCP, int taps, int ICP) {
  std::vector<uint8_t> img(hp.b_bytes, 0);
  pack_walk(hp, img.data(), [&](uint8_t *dst, int j, HaloPlan::Chunk c, int g, int o0, int rows) {
    // c.cb: which four channels of the block
    float *hi = reinterpret_cast<float *>(dst) + static_cast<size_t>(j) * (hp.p.stack ? 2 * rows : rows) * 4;
    float *lo = hi + static_cast<size_t>(hp.p.stack ? rows : 2 * rows) * 4;
    for (int r = 0; r < rows && o0 + r < OCP; ++r) {
      const float *src = u + (static_cast<size_t>(o0 + r) * taps + c.tap) * ICP + g * 16 + c.cb * 4;
      for (int e = 0; e < 4; ++e) {
        const float h = host::tf32_rna(src[e]);
        hi[r * 4 + e] = h;
        lo[r * 4 + e] = src[e] - h;      // (exact)
      }
    }
  });
  return img;
}

namespace {

// First byte of parity plane q of the tensor at `in` (one plane: the tensor itself)
void *plane_base(const HaloPlan &hp, const void *in, int q) {
  const int s = hp.stride, ph = hp.parity[q] / s, pw = hp.parity[q] % s;
  return const_cast<uint8_t *>(static_cast<const uint8_t *>(in)) + (static_cast<size_t>(ph) * hp.IW + pw) * (hp.kind == HALO_F32 ? 64 : 16);
}

// Which copies the tiles of `images` images take of plane q (bit i: of HaloArgs::tmap[q][i]'s height): the walk of the
// kernel's row warp.  The tiles' offsets in an image repeat after at most `period` tiles.
int copy_heights(const HaloParams &p, int images, int q) {
  const long long row_tiles = (static_cast<long long>(images - 1) * p.period + p.OH + TILE_H - 1) / TILE_H;
  int seen = 0;
  for (int rt = 0; rt < row_tiles && rt <= p.period; ++rt) {
    const int v0 = rt * TILE_H + p.row0[q], rows = p.rows[q];
    if ((v0 > 0 ? v0 % p.period : v0) + rows <= p.period) {
      seen |= 1 << (HALO_HEIGHTS - 1);
      continue;
    }
    for (int r = 0; r < rows;) {
      const int v = v0 + r, left = v > 0 ? p.period - v % p.period : p.period - v;      // rows of this image from here
      const int len = std::min(left, rows - r);
      if (len >= 8) seen |= 8;
      seen |= len & 7;
      r += len;
    }
  }
  return seen;
}

// Tensor maps of `cnt` images at `in`.
bool encode_maps(const HaloPlan &hp, const void *in, int cnt, int step, int src_h, int src_w, CUtensorMap (*out)[HALO_HEIGHTS],
                 std::string &err) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) { err = "cuTensorMapEncodeTiled is not available from the driver"; return false; }
  const HaloParams &p = hp.p;
  const cuuint64_t px = hp.kind == HALO_F32 ? 64 : 16, IW = hp.IW, IH = hp.IH, CB = hp.CB;
  const cuuint32_t blocks = p.cb_step, estr[5] = {1, 1, 1, 1, 1};
  CUresult r = CUDA_SUCCESS;
  // (dimensions in the order the operand rows lie in shared memory: pixels, channel blocks, rows)
  for (int q = 0; q < p.planes; ++q)
    for (int i = 0; i < HALO_HEIGHTS && r == CUDA_SUCCESS; ++i) {
      const cuuint32_t height = i == HALO_HEIGHTS - 1 ? p.rows[q] : 1u << i;
      if (step > 1) {
        // one plane of every step-th pixel of a larger one (pixel by pixel, like the parity planes)
        const cuuint64_t SH = src_h, SW = src_w, st = step;
        cuuint64_t dims[5] = {16, IW, CB, IH, static_cast<cuuint64_t>(cnt)};
        cuuint64_t strides[4] = {st * px, SH * SW * px, st * SW * px, CB * SH * SW * px};
        cuuint32_t box[5] = {16, static_cast<cuuint32_t>(p.pxw), blocks, height, 1};
        r = enc(&out[q][i], hp.kind == HALO_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 5,
                const_cast<void *>(in), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      } else if (!p.strided) {
        cuuint64_t dims[4] = {IW * px / 8, CB, IH, static_cast<cuuint64_t>(cnt)};
        cuuint64_t strides[3] = {IH * IW * px, IW * px, CB * IH * IW * px};
        cuuint32_t box[4] = {static_cast<cuuint32_t>(p.pxw * px / 8), blocks, height, 1};
        r = enc(&out[q][i], CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, const_cast<void *>(in), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      } else {
        const int s = hp.stride, ph = hp.parity[q] / s, pw = hp.parity[q] % s;
        void *base = plane_base(hp, in, q);
        cuuint64_t dims[5] = {16, static_cast<cuuint64_t>((hp.IW - pw + s - 1) / s), CB,
                              static_cast<cuuint64_t>((hp.IH - ph + s - 1) / s), static_cast<cuuint64_t>(cnt)};
        cuuint64_t strides[4] = {s * px, IH * IW * px, s * IW * px, CB * IH * IW * px};
        cuuint32_t box[5] = {16, static_cast<cuuint32_t>(p.pxw), blocks, height, 1};
        r = enc(&out[q][i], hp.kind == HALO_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, base, dims,
                strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      }
    }
  if (r != CUDA_SUCCESS) { err = "cuTensorMapEncodeTiled failed (" + std::to_string(static_cast<int>(r)) + ")"; return false; }
  return true;
}

}  // namespace

namespace {

// A kernel and what its parameters hold
struct HaloKernel {
  const void *fn = nullptr;
  int planes = 0, oc = 0;
};
template <int KIND, int PAIRS, int FORM, bool STACK, bool PAIR, bool SPLIT, bool FINE>
HaloKernel kernel_of(bool stepped = false) {
  if constexpr (KIND == HALO_I8 && (FORM == FORM_3X3_ROWS || FORM == FORM_3X3_TAPS || FORM == FORM_3X3_RESIDENT))
    if (stepped)
      return {reinterpret_cast<const void *>(conv_halo_kernel<KIND, PAIRS, FORM, STACK, PAIR, SPLIT, FINE, true>), planes_of(FORM), oc_of(KIND, SPLIT)};
  return {reinterpret_cast<const void *>(conv_halo_kernel<KIND, PAIRS, FORM, STACK, PAIR, SPLIT, FINE, false>), planes_of(FORM), oc_of(KIND, SPLIT)};
}
template <int FORM, bool PAIR = false, bool SPLIT = false>
HaloKernel pick_kernel(const HaloPlan &hp, bool stepped) {
  if (hp.kind == HALO_F32) {
    if constexpr (FORM == FORM_3X3_TAPS || (!PAIR && (FORM == FORM_3X3_ROWS || (!SPLIT && FORM == FORM_3X3_RESIDENT))))
      if (hp.p.fine) return kernel_of<HALO_F32, 2, FORM, !PAIR, PAIR, SPLIT, true>();
    if (hp.p.fine) return {};      // (halo_plan() makes no such plan)
    if constexpr (!PAIR)
      if (hp.p.stack) return kernel_of<HALO_F32, 2, FORM, true, false, SPLIT, false>();
    return kernel_of<HALO_F32, 2, FORM, false, PAIR, SPLIT, false>();
  }
  switch (hp.p.kch) {
    case 8: return kernel_of<HALO_I8, 4, FORM, false, PAIR, SPLIT, false>(stepped);
    case 6: return kernel_of<HALO_I8, 3, FORM, false, PAIR, SPLIT, false>(stepped);
    case 4: return kernel_of<HALO_I8, 2, FORM, false, PAIR, SPLIT, false>(stepped);
  }
  if constexpr (!PAIR) {
    if (hp.p.kch == 2) return kernel_of<HALO_I8, 1, FORM, false, false, SPLIT, false>(stepped);
    if constexpr (!SPLIT) return kernel_of<HALO_I8, 0, FORM, false, false, false, false>(stepped);
  }
  return {};
}
// The issue loop's form for a geometry (before the weight stages are laid out); FORM_3X3_TAPS stands for all 3x3 ones.
int tap_form(const HaloPlan &hp) {
  const HaloParams &p = hp.p;
  const int pairs = p.kch / 2, *r = p.tap_rows, *c = p.tap_cols;
  int form = FORM_ANY;
  if (hp.stride == 1 && r[0] == 3 && c[0] == 3) form = FORM_3X3_TAPS;
  else if (p.planes == 4 && pairs && r[0] == 1 && c[0] == 1 && r[1] == 1 && c[1] == 2 && r[2] == 2 && c[2] == 1 && r[3] == 2 && c[3] == 2) form = FORM_3X3S2;
  else if (p.planes == 1 && pairs && r[0] == 1 && c[0] == 1) form = FORM_1X1;
  return p.pxw == pxw_of(form, hp.kind, pairs) ? form : FORM_ANY;
}
template <bool PAIR, bool SPLIT>
HaloKernel pick_form(const HaloPlan &hp, int form, bool stepped) {
  switch (form) {
    case FORM_3X3_ROWS:
      if constexpr (!PAIR) return pick_kernel<FORM_3X3_ROWS, false, SPLIT>(hp, stepped);
      return {};
    case FORM_3X3_TAPS: return pick_kernel<FORM_3X3_TAPS, PAIR, SPLIT>(hp, stepped);
    case FORM_3X3S2: return pick_kernel<FORM_3X3S2, PAIR, SPLIT>(hp, stepped);
    case FORM_1X1: return pick_kernel<FORM_1X1, PAIR, SPLIT>(hp, stepped);
  }
  return pick_kernel<FORM_ANY, PAIR, SPLIT>(hp, stepped);
}
HaloKernel pick_kernel(const HaloPlan &hp, bool stepped) {
  const HaloParams &p = hp.p;
  int form = tap_form(hp);
  if (p.resident) return form == FORM_3X3_TAPS && p.b_stages == 3 * p.groups ? pick_kernel<FORM_3X3_RESIDENT>(hp, stepped) : pick_kernel<FORM_ANY>(hp, stepped);
  if (p.row_units) form = form == FORM_3X3_TAPS ? FORM_3X3_ROWS : FORM_ANY;
  return p.split > 1 ? pick_form<false, true>(hp, form, stepped) : p.pair ? pick_form<true, false>(hp, form, stepped) : pick_form<false, false>(hp, form, stepped);
}

// Launch configuration: may overlap its set-up with the kernel before it (launch_overlapped), pairs as clusters of two.
struct LaunchConfig {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  LaunchConfig(const HaloPlan &hp, int ctas, cudaStream_t s) {
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(hp.kind == HALO_F32 ? THREADS_F32 : THREADS_I8);
    cfg.dynamicSmemBytes = hp.smem_bytes;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = hp.p.pair ? 2 : hp.p.split; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = hp.p.pair || hp.p.split > 1 ? 2 : 1;
  }
  LaunchConfig(const LaunchConfig &) = delete;
};

}  // namespace

cudaError_t halo_init(HaloPlan &hp, bool stepped) {
  const HaloKernel k = pick_kernel(hp, stepped);
  cudaError_t e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT + 1024);
  if (e == cudaSuccess && hp.p.pair && !stepped) {
    LaunchConfig lc(hp, 2, nullptr);
    e = cudaOccupancyMaxActiveClusters(&hp.max_clusters, k.fn, &lc.cfg);
    if (e == cudaSuccess && hp.max_clusters < 1) e = cudaErrorInvalidConfiguration;
  }
  return e;
}

// The packed weights as rows of 512 bytes (pairs fetch them with tiled copies, whose bytes may count on the leader's barrier)
bool halo_set_weights(HaloPlan &hp, void *d_b, std::string &err) {
  hp.d_b = d_b;
  if (!hp.p.pair) return true;
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) { err = "cuTensorMapEncodeTiled is not available from the driver"; return false; }
  cuuint64_t dims[2] = {64, hp.b_bytes / 512}, strides[1] = {512};
  cuuint32_t box[2] = {64, static_cast<cuuint32_t>(hp.p.b_stage_bytes / 512)}, estr[2] = {1, 1};
  const CUresult r = enc(&hp.tmap_b, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, d_b, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { err = "cuTensorMapEncodeTiled failed (" + std::to_string(static_cast<int>(r)) + ")"; return false; }
  return true;
}

namespace {
// Launches `k` with the plan's maps (their addresses set to `base[plane]`) and constants behind p
template <int PLANES, int OC>
bool launch_args(const HaloPlan &hp, const HaloParams &p, const HaloPlan::Maps &maps, void *const *base, const HaloKernel &k,
                 const cudaLaunchConfig_t &cfg, std::string &err) {
  HaloArgs<PLANES, OC> a;
  static_cast<HaloParams &>(a) = p;
  const PFN_replaceAddress set_address = get_replace_address();
  if (!set_address) { err = "cuTensorMapReplaceAddress is not available from the driver"; return false; }
  // (with five maps per plane encoded for every new address a call took 7.2 us of host time, strided 8.3, against 4.4)
  for (int q = 0; q < p.planes; ++q)
    for (int i = 0; i < HALO_HEIGHTS; ++i) {
      a.tmap[q][i] = maps.m[q][i];
      if (((maps.heights[q] >> i) & 1) && set_address(&a.tmap[q][i], base[q]) != CUDA_SUCCESS) {
        err = "cuTensorMapReplaceAddress failed";
        return false;
      }
    }
  if (p.pair) a.tmap_b = hp.tmap_b;
  if (OC > 0 && p.fast == 1) {
    std::copy_n(hp.scale.data(), p.OCB * 16, a.cst[0]);
    std::copy_n(hp.shift.data(), p.OCB * 16, a.cst[1]);
  }
  void *args[] = {&a};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, k.fn, args);
  if (e != cudaSuccess) err = std::string("kernel launch failed: ") + cudaGetErrorString(e);
  return e == cudaSuccess;
}
}  // namespace

bool halo_launch(HaloPlan &hp, HaloParams &p, const void *in, int images, int num_sms, cudaStream_t s, std::string &err,
                 int step, int src_h, int src_w) {
  const HaloPlan::Maps *hit = nullptr;
  for (const auto &m : hp.maps)
    if (m.cnt == images && m.step == step && (step == 1 || (m.src_h == src_h && m.src_w == src_w))) { hit = &m; break; }
  if (!hit) {
    HaloPlan::Maps m{};
    m.cnt = images; m.step = step; m.src_h = src_h; m.src_w = src_w;
    for (int q = 0; q < p.planes; ++q) m.heights[q] = static_cast<uint8_t>(copy_heights(p, images, q));
    if (!encode_maps(hp, in, images, step, src_h, src_w, m.m, err)) return false;
    if (hp.maps.size() < 16) hp.maps.push_back(m);
    else hp.maps[hp.next_map] = m;
    hit = &hp.maps[hp.next_map];
    hp.next_map = (hp.next_map + 1) % 16;
  }
  void *base[4];
  for (int q = 0; q < p.planes; ++q) base[q] = step > 1 ? const_cast<void *>(in) : plane_base(hp, in, q);
  const HaloKernel kernel = pick_kernel(hp, step > 1);
  if (p.planes > kernel.planes) { err = "internal: planes"; return false; }
  p.b_img = static_cast<const uint8_t *>(hp.d_b);
  p.wide = reinterpret_cast<uintptr_t>(p.out) % 32 == 0;
  const bool fast = p.rq.out_type == OUT_U8 && p.rq.relu && p.rq.relu_lo == 0.0f && p.rq.relu_hi >= 3.0e38f && !p.rq.with_sum &&
                    !p.shift_tbl;
  p.fast = !fast ? 0 : p.OCB * 16 <= kernel.oc ? 1 : 2;
  p.N = images;
  if (step > 1) p.strided = 1;
  p.row_tiles = ((images - 1) * p.period + p.OH + TILE_H - 1) / TILE_H;
  const int m_tiles = p.row_tiles * p.col_tiles;
  p.total_tiles = (p.pair ? (m_tiles + 1) / 2 : m_tiles) * p.n_tiles;
  const int units = p.split > 1 ? p.total_tiles : std::min(p.total_tiles, p.pair ? hp.max_clusters : num_sms);
  // int8: sixteen epilogue warps on each tile finish it in a quarter (BN <= 128) or half of the time that a group's share of the
  // warps takes, but every warp then pays a tile's fixed cost (locating its pixel, waits, releases).  Graph replays, us without / with:
  //  * one tile per CTA (a split K loop too): the launch ends with it: 1 x 128 -> 544 1x1 at 27x27 with f32 results 3.64 / 3.44;
  //  * two tiles, results of bytes: 42 x 298 -> 128 1x1 at 24x24 with a residual 10.8 / 8.7, 26 x 80 -> 128 3x3 at 27x31 10.2 / 8.7; with
  //    more than 128 columns (half of the warps work on a tile as it is) only where the K loop is not much shorter than the epilogue:
  //    7 x 25 -> 160 at 70x70 8.4 / 9.0 and 39 x 119 -> 528 at 14x14 5.7 / 6.1 (ratios 0.3, 0.5), 3 x 528 -> 192 at 101x107 9.0 / 8.8 (0.8);
  //  * a K loop that outlasts the epilogue anyway: 128 -> 256 3x3 stride 2 with a residual 28.4 / 26.0, 4 x 608 -> 144 1x1 at 104x97 11.7 / 11.2;
  //    of pairs by half as much again, because a tile waits for 32 warps of two CTAs to hand an accumulator back: 5 x 176 -> 1439
  //    3x3 at 41x41 28.1 / 26.0 (ratio 1.85), 4 x 128 -> 640 3x3 at 41x41 11.6 / 12.1 (1.30);
  //  * of pairs on a 1x1 filter, in launches of up to five tiles per CTA: 21 x 656 -> 848 at 15x14 with a residual 13.5 / 11.8, 6 x 656 -> 1264
  //    at 40x40 17.8 / 16.7 (1.03); 44 x 560 -> 1035 at 57x57 (60 tiles) 122 / 142, 18 x 592 -> 305 at 46x49 (160 columns, 1.26) 21.8 / 23.2.
  // Elsewhere it loses: 64 -> 64 at 224x224 29.6 / 36.2, 63 x 336 -> 848 1x1 at 37x37 72.2 / 77.4 (ratio 0.95); so do f32 results, which are
  // bound by their stores, behind the first tile (6 x 640 -> 297 1x1 at 74x62 18.2 / 19.7), one block of columns, which feeds a single group
  // (16 columns: 42 x 357 -> 16 at 24x26 5.5 / 5.8), and tiles of few blocks in a row (20 x 48 -> 48 at 100x100 9.4 / 11.6).
  const bool pair_1x1 = p.pair && 2 * p.ksteps == p.kch;
  const double need = pair_1x1 ? (p.BN >= 224 ? 1.0 : 1.4) : p.pair ? 1.5 : p.bufs == 4 ? 1.2 : 1.0;
  const bool two = p.total_tiles <= 2 * units && (p.pair ? hp.loop_ratio > need : p.BN <= 128 || hp.loop_ratio > 0.65);
  const bool loop = p.BN >= 112 && hp.loop_ratio > need && !(pair_1x1 && p.total_tiles > 5 * units);
  p.spread = hp.kind == HALO_I8 && p.BN >= 32 && (p.total_tiles <= units || (p.rq.out_type != OUT_F32 && (two || loop)));
  LaunchConfig lc(hp, units * (p.split > 1 ? p.split : p.pair ? 2 : 1), s);
  if (kernel.planes == 1)
    return kernel.oc ? launch_args<1, PARAM_OC>(hp, p, *hit, base, kernel, lc.cfg, err) : launch_args<1, 0>(hp, p, *hit, base, kernel, lc.cfg, err);
  return kernel.oc ? launch_args<4, PARAM_OC>(hp, p, *hit, base, kernel, lc.cfg, err) : launch_args<4, 0>(hp, p, *hit, base, kernel, lc.cfg, err);
}

}  // namespace elb
