// Direct-tap forward convolution on the tensor cores (sm_100a): every kernel tap is one K-major slice of the reduction,
//
//     y[n, o, k] = sum over taps t and channels c of x[n, s * o + t - p, c] * U[t][k][c]
//
// with the x operand of *all* taps read from one shared-memory slab.  A 128-row tile is 16 groups of 8 pixels along W (the
// groups run over output rows, or over rows and images where the image is small); its slab holds those pixels and the halo
// of the kernel, [rows][images][8 + kW - 1 pixels][64 channels] as TMA writes it with the 128-byte swizzle.  The swizzle is a
// function of the absolute address, so a tcgen05 operand may start at any pixel of the slab: tap (kh, kw) is the same slab
// read from kh rows and kw pixels further on, with a group stride of one slab row.  No im2col copy, no transform, nothing
// but the filter is reloaded per tap.
//
// What bounds it: the tensor pipe needs N / 2 clocks per (M = 128, N, K = 16) instruction, shared memory delivers 128 B per
// clock.  Per tap and 64 channels of a 256-column tile of a CTA pair an SM reads 4 x (4 KB of A + 4 KB of B) and TMA writes
// 16 KB of filter and about 2.6 KB of slab: 50 KB in the 512 clocks the MMAs take, where a kernel that loads its A operand
// tap by tap moves 64 KB.  F(2,3) row pieces do two thirds of the multiplies but move 74 KB per 256 columns' worth of work
// and spend an epilogue and a producer pass on the transforms.
//
// Roles of a CTA: warp 0 TMA slabs, warp 1 TMA filter tiles, warps 2-3 MMA issue (one per 128-row block; warp 2 owns the
// tensor memory), warps 4-11 epilogue (lane quarter x alternate 128-byte column chunks: bias, ReLU, 2x2 pool, TMA stores; items of few
// MMAs come with a second such set, warps 12-19, and the sets take items in turn),
// for fp32 also warps 12-15, which split every landed slab into a tf32 part and its remainder (three products per multiply,
// the filter comes split from its transform).
// Few channels (an RGB stem) would leave most of a 16-channel step empty and cannot be loaded by TMA (16-byte pixels).  There
// the taps along W are folded into the channels: a slab row is an input row, its entries the 8 output pixels, an entry the
// kW * C values those pixels' taps see; only the taps along H remain.  7x7 at stride 2 over RGB is 7 x 2 K steps instead of 49.
// Warps 12-15 gather the entries from a patch of raw rows of x as it lies (either layout) that warp 0 loads by TMA, or, where
// rows are not 16-byte multiples, with plain loads (the latency of those is what it costs: 130 us against 45 for the stem).
// Small problems run with one item per cluster of 2, 4 or 8 CTAs that share its reduction and add their accumulators through
// distributed shared memory.  Every mbarrier wait is bounded and reports through the error word.
//
// Stands in for the chain of src/base_conv_launchers.cu:338-381 where no output tile larger than 1 is worth its transforms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

#include "wino_launch.h"
#include "wino_sm100.cuh"

namespace wino {

__device__ unsigned int g_direct_error = 0;

namespace dconv {

using namespace sm100;

constexpr int BM = 128;
constexpr int EPI_WARP0 = 4, EPI_WARPS = 8, SPLIT_WARP0 = 12, SPLIT_WARPS = 4;
constexpr int STAGE_BYTES = 4096;      // epilogue staging per warp: 32 rows of 128 bytes
constexpr int MAX_TAPS = 100;
constexpr int BAR_BYTES = 512;
constexpr unsigned RAW_BUFS = 4;       // raw patches in flight (few channels): small, and thousands of clocks away
constexpr int FIXED_BYTES = 1024 /*alignment*/ + EPI_WARPS * STAGE_BYTES + BAR_BYTES;
constexpr int SET_BYTES = EPI_WARPS * STAGE_BYTES;     // staging of a second set of epilogue warps (warps 12-19)
__host__ __device__ constexpr int threads_of(bool splits, int sets) { return 32 * (SPLIT_WARP0 + (splits ? SPLIT_WARPS : 0) + (sets - 1) * EPI_WARPS); }

enum ErrCode : unsigned { ERR_A_EMPTY = 0x401, ERR_B_EMPTY = 0x402, ERR_ACC = 0x403, ERR_A = 0x404, ERR_B = 0x405, ERR_EPI = 0x406, ERR_SPLIT = 0x407 };

struct DGeom {
  int N, K, oD, oH;
  int sD, sH, sW, pD, kD;
  int yH[4], yW[4];                  // stored extents (of each variant)
  long long y_off[4], ys_n, ys_d, ys_h, ys_w;   // first element of each variant, element strides
  // A block's 128 rows are 16 groups of 8, numbered (output row, image group) with TH * TN == 16; the 8 rows of a group are
  // 8 / TI pixels along W of TI images, image innermost (TI > 1 where 8 pixels would not divide a small image).
  int TN, tn_shift, TH, TI, ti_shift, PW;   // PW: pixels of a slab row
  int map_mode;                      // order of the tensor maps' dimensions: see tile_load
  int n_wb, n_hb, n_tiles, n_kb, n_items, var_items;   // n_items = var_items x variants
  int n_ph, n_var, org_h[4], org_w[4], taps[4], tap0[4], T_hw;   // parts of the taps: all of them per item, or one (variants)
  int n_chunks, ch_el, k_full, k_tail;   // channel chunks, channels per chunk, MMA K steps of a full and of the last chunk
  int units;                         // kD * T_hw * n_chunks: (tap, chunk) pairs of the whole reduction
  int G, split;                      // taps per filter stage, CTAs (pairs) per item
  unsigned epilogue;
  int y_tma, bias_vec, bias_f32;
  uint32_t a_hi, b_hi;               // high descriptor words
  int mb_off16;                      // slab offset of the second row block (16-byte units)
  // fold: x's strides and extents, channels and taps of an entry, slab rows and how far apart the rows of neighbouring outputs are
  long long fx_n, fx_d, fx_h;
  int fx_w, fx_c, fD, fH, fW, fC, fkW, fold_rows;
  // ... and the raw patch: by TMA or not, element strides of its rows, pixels and channels, elements before the first pixel
  int raw_tma, raw_row, raw_w, raw_c, raw_rem;
  uint16_t tap_off[MAX_TAPS + 1];    // offset of each tap's first pixel in the slab (16-byte units), phase by phase
};
struct DSmem {
  int slab_bytes, a_bytes, lo_off;   // bytes TMA delivers, bytes of a stage, offset of the remainder copy (fp32)
  int b_tile, b_lo, b_bytes, n_a, n_b;   // bytes of one tap's filter tile (hi part, and lo part for fp32), of a stage
  int off_b, off_stage, off_raw, raw_bytes, off_bars;   // raw_bytes: of a raw patch, a multiple of 128
};

template <typename T> struct OutWord {   // one 32-bit word of output: a 16-bit pair
  static constexpr int COLS = 64;
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) { return Pair16<T>::max2(a, b); }
};
template <> struct OutWord<float> {
  static constexpr int COLS = 32;
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) { return __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b))); }
};

// V bias values from k on, stored as T or as floats
template <typename TB, int V> __device__ __forceinline__ void load_bias(const TB *bias, int k, int K, int vec, float *b) {
  if (vec && k + V <= K) {
#pragma unroll
    for (int i = 0; i < V * (int)sizeof(TB) / 16; ++i) {
      const uint4 q = *reinterpret_cast<const uint4 *>(bias + k + i * (16 / (int)sizeof(TB)));
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (sizeof(TB) == 4) b[4 * i + j] = __uint_as_float(w[j]);
        else { const float2 f = Pair16<TB>::unpack(w[j]); b[8 * i + 2 * j] = f.x; b[8 * i + 2 * j + 1] = f.y; }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) b[i] = k + i < K ? Elem<TB>::load(bias + k + i) : 0.f;
  }
}

struct MapSet { CUtensorMap m[4]; };      // the output of each variant

struct Tile { int var, kb, n0, od, oh0, ow0; bool valid; };
// item -> variant, channel block and the tile (of this CTA: a pair's CTAs take neighbouring tiles)
template <int MB, bool PAIR> __device__ __forceinline__ Tile decode(const DGeom &g, int item, uint32_t rank) {
  Tile t;
  t.var = g.n_var > 1 ? item / g.var_items : 0;
  const unsigned it = (unsigned)(item - t.var * g.var_items), tb = it / (unsigned)g.n_kb;
  t.kb = (int)(it - tb * (unsigned)g.n_kb);
  const unsigned tile = PAIR ? 2u * tb + rank : tb;
  t.valid = tile < (unsigned)g.n_tiles;
  unsigned q = tile / (unsigned)g.n_wb;
  t.ow0 = (int)(tile - q * (unsigned)g.n_wb) * (8 >> g.ti_shift);
  unsigned r = q / (unsigned)g.n_hb;
  t.oh0 = (int)(q - r * (unsigned)g.n_hb) * (MB * g.TH);
  q = r / (unsigned)g.oD;
  t.od = (int)(r - q * (unsigned)g.oD);
  t.n0 = (int)q * (g.TN * g.TI);     // a tile past the end starts at an image past the end: TMA fills zeros
  return t;
}

// The maps order a tensor's dimensions so that a box lands in the block's row order: mode 0 [channel, W, image, H, depth];
// mode 1 (TI > 1, TN == 1) [channel, image, W, H, depth]; mode 2 (TI > 1 and TN > 1, 2-D, the batch a multiple of TI)
// [channel, image within a group, W, image group, H].
template <bool PAIR>
__device__ __forceinline__ void tile_load(const DGeom &g, uint32_t dst, const CUtensorMap *map, uint32_t bar, int c, int w, int n, int h, int d) {
  const int c1 = g.map_mode == 0 ? w : g.map_mode == 1 ? n : 0, c2 = g.map_mode == 0 ? n : w;
  const int c3 = g.map_mode == 2 ? n >> g.ti_shift : h, c4 = g.map_mode == 2 ? h : d;
  if (PAIR) tma_load_5d_pair(dst, map, bar, c, c1, c2, c3, c4);
  else tma_load_5d(dst, map, bar, c, c1, c2, c3, c4);
}
__device__ __forceinline__ void tile_store(const DGeom &g, const CUtensorMap *map, uint32_t src, int k, int w, int n, int h, int d) {
  const int c1 = g.map_mode == 0 ? w : g.map_mode == 1 ? n : 0, c2 = g.map_mode == 0 ? n : w;
  const int c3 = g.map_mode == 2 ? n >> g.ti_shift : h, c4 = g.map_mode == 2 ? h : d;
  tma_store_5d(map, src, k, c1, c2, c3, c4);
}

// Calls body(kd, p, ch, t0, t1) for the steps (depth tap, polyphase part, channel chunk) whose taps [t0, t1) fall into this
// CTA's share [u0, u1) of the reduction, until it returns false; returns whether all of them ran.
template <typename F> __device__ __forceinline__ bool for_steps(const DGeom &g, int var, int u0, int u1, F &&body) {
  int s0 = 0;
  const int p0 = g.n_var > 1 ? var : 0, p1 = g.n_var > 1 ? var + 1 : g.n_ph;
  for (int kd = 0; kd < g.kD; ++kd)
    for (int p = p0; p < p1; ++p) {
      const int tp = g.taps[p];
      for (int ch = 0; ch < g.n_chunks; ++ch, s0 += tp) {
        const int t0 = max(0, u0 - s0), t1 = min(tp, u1 - s0);
        if (t0 < t1 && !body(kd, p, ch, t0, t1)) return false;
      }
    }
  return true;
}

// fp32: two threads take alternate K steps of a block into accumulators of their own (one thread issues an MMA every 60 to
// 85 clocks, three products a step), and the products with a remainder go to another pair: the accumulator is cut off after
// every MMA, so its error grows with the number of MMAs that went into it times its size -- small products in a small
// accumulator cost nothing.  After ACC_STEPS K steps the accumulators are handed to the epilogue, which keeps the sum in
// registers, rounded to nearest, while the next ones fill: no chain is longer than ACC_STEPS / 2 and a filter stage.  2-norm
// errors against 64 bits over 8 layers of 8 to 512 channels, 1x1 to 9x9: 1.6e-7 to 2.2e-7 and 3.0e-7 (17836 products) with 16
// steps, 1.6e-7 to 2.4e-7 with 8, 2.5e-7 to 7.9e-6 without handing over; one step of 16 costs 5 % (64 -> 64 5x5 at 56x56, N = 8:
// 57 us; with 8 steps 63), which one MMA for both parts of the filter (N = 128 instead of two of 64) gives back.
__host__ __device__ constexpr int accumulators_of_a_block(bool f32) { return f32 ? 4 : 1; }
constexpr int ACC_STEPS = 16;

template <typename T, int BN, int MB, bool PAIR, bool FOLD, int SETS>
__global__ void __launch_bounds__(threads_of(std::is_same<T, float>::value || FOLD, SETS), 1)
    direct_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_u,
                  const __grid_constant__ MapSet maps_y, const T *__restrict__ x, T *__restrict__ y, const T *__restrict__ bias,
                  const __grid_constant__ DGeom g, const __grid_constant__ DSmem sl, uint32_t idesc) {
  constexpr bool F32 = std::is_same<T, float>::value;
  constexpr int COLS = OutWord<T>::COLS;            // output columns of one 128-byte staging row
  constexpr int KS = F32 ? 2 : 1;                   // threads that share a block's K steps
  constexpr int N_ACC = accumulators_of_a_block(F32);
  constexpr int ACC = MB * BN * N_ACC;              // accumulator columns of a buffer
  constexpr int N_ISSUE = MB >= 2 || KS == 2 ? 2 : 1;
  constexpr int BNH = PAIR ? BN / 2 : BN;           // filter rows this CTA loads
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw);
  const uint32_t bars = base + sl.off_bars;         // a_full[8] a_empty[8] b_full[8] b_empty[8] a_split[8] acc_full[2] acc_empty[2]
  auto a_full = [&](int i) { return bars + 8u * i; };
  auto a_empty = [&](int i) { return bars + 64u + 8u * i; };
  auto b_full = [&](int i) { return bars + 128u + 8u * i; };
  auto b_empty = [&](int i) { return bars + 192u + 8u * i; };
  auto a_split = [&](int i) { return bars + 256u + 8u * i; };
  auto raw_empty = [&](int i) { return bars + 352u + 8u * i; };     // (raw_full: a_split)
  auto acc_full = [&](int i) { return bars + 320u + 8u * i; };
  auto acc_empty = [&](int i) { return bars + 336u + 8u * i; };
  volatile unsigned *abort_word = reinterpret_cast<volatile unsigned *>(base_ptr + sl.off_bars + 384);
  const uint32_t tmem_slot = bars + 388u;
  unsigned *err = &g_direct_error;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // the warp index in a uniform register
  // Set-up, spread over warps and lanes (it is a fifth of a one-wave launch): descriptors fetched, barriers initialised,
  // tensor memory allocated.
  if (warp == 1 && lane == 0) { prefetch_map(&map_x); prefetch_map(&map_u); prefetch_map(&maps_y.m[0]); }
  if (warp == 0) {
    if (lane < 8) {
      mbar_init(a_full(lane), FOLD ? SPLIT_WARPS : 1); mbar_init(a_empty(lane), N_ISSUE); mbar_init(a_split(lane), FOLD ? 1 : SPLIT_WARPS);
    } else if (lane < 16) {
      mbar_init(b_full(lane - 8), 1); mbar_init(b_empty(lane - 8), N_ISSUE);
    } else if (lane < 18) {
      mbar_init(acc_full(lane - 16), N_ISSUE); mbar_init(acc_empty(lane - 16), PAIR ? 2 * EPI_WARPS : EPI_WARPS);
    } else if (lane < 22) {
      mbar_init(raw_empty(lane - 18), SPLIT_WARPS);
    } else if (lane == 22) {
      *abort_word = 0u;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint32_t crank = PAIR ? cluster_ctarank() : 0u, rank = crank & 1u;   // rank within the pair
  const bool leader = rank == 0;                   // issues the MMAs of the pair
  const uint32_t tmem_cols = g.split > 1 && !F32 ? ACC : 2 * ACC;      // a shared item needs one accumulator
  if (warp == 2) tmem_alloc<PAIR>(tmem_slot, tmem_cols);
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the barriers of both CTAs exist before either arrives at the other's
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
  tmem = __shfl_sync(0xffffffffu, tmem, 0);
  grid_launch_dependents();
  grid_dependency_wait();

  // work of this CTA: items item0, item0 + step, ... and the share [u0, u1) of each one's reduction
  int item0, item_step, u0 = 0, u1 = g.units;
  uint32_t part = 0;
  const int unit_cta = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;     // a CTA, or a pair
  if (g.split > 1) {
    item0 = unit_cta / g.split;
    item_step = g.n_items;
    part = (uint32_t)(unit_cta - item0 * g.split);
    u0 = (int)((long long)g.units * part / g.split);
    u1 = (int)((long long)g.units * (part + 1) / g.split);
  } else { item0 = unit_cta; item_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x; }
  // one channel block whose whole filter fits the ring: loaded once, its stages are never handed back
  const bool resident = g.n_kb == 1 && g.split == 1 && g.n_var == 1 && g.kD * g.n_ph * g.n_chunks * ((g.taps[0] + g.G - 1) / g.G) <= sl.n_b;
  bool alive = true;

  // fp32: how many times an item's accumulators change hands, the K steps of the last time, and an epilogue warp's sum of 32 columns
  int n_hand = 1, last_steps = 0;
  float sum[32];
  uint32_t n_acc = 0;
  auto sum_accumulators = [&]() -> bool {
    if constexpr (F32) {
#pragma unroll
      for (int i = 0; i < 32; ++i) sum[i] = 0.f;
      const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(((warp - EPI_WARP0) >> 2) * 32);
      for (int f = 0; f < n_hand; ++f, ++n_acc) {
        const int buf = (int)(n_acc & 1u);
        if (!mbar_wait_warp(acc_full(buf), (n_acc >> 1) & 1u, abort_word, err, ERR_EPI) || *abort_word != 0u) return false;
        tc_fence_after();
        const bool both = f + 1 < n_hand || last_steps >= 2;      // a single step is the first thread's
#pragma unroll 1
        for (int a = 0; a < (both ? N_ACC : N_ACC / 2); ++a) {
          uint32_t r[32];
          tmem_ld_x32(ta + (uint32_t)(buf * ACC + a * BN), r);
          tmem_wait_ld_x32(r);
#pragma unroll
          for (int i = 0; i < 32; ++i) sum[i] += __uint_as_float(r[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(buf));
      }
    }
    return true;
  };
  if (F32 && warp >= EPI_WARP0 && warp < EPI_WARP0 + EPI_WARPS)
    for_steps(g, 0, u0, u1, [&](int, int, int ch, int t0, int t1) -> bool {
      const int nk = ch == g.n_chunks - 1 ? g.k_tail : g.k_full;
      for (int t = t0; t < t1; t += g.G) {
        if (last_steps >= ACC_STEPS) { ++n_hand; last_steps = 0; }
        last_steps += min(g.G, t1 - t) * nk;
      }
      return true;
    });

  if (warp == 0 && FOLD) {
    // ---------------------------------------------------------------- raw patches, from which warps 12-15 gather the slabs
    uint32_t it = 0;
    for (int item = item0; item < g.n_items && alive && g.raw_tma; item += item_step) {
      const Tile t = decode<MB, PAIR>(g, item, rank);
      alive = for_steps(g, t.var, u0, u1, [&](int kd, int, int, int, int) -> bool {
        const int s = (int)(it & (RAW_BUFS - 1u));
        if (!mbar_wait_warp(raw_empty(s), ((it / RAW_BUFS) & 1u) ^ 1u, abort_word, err, ERR_A_EMPTY)) return false;
        if (lane == 0) {
          const uint32_t dst = base + (uint32_t)(sl.off_raw + s * sl.raw_bytes);
          const int w = (g.sW * t.ow0 + g.org_w[0]) * g.raw_w - g.raw_rem, h = g.sH * t.oh0 + g.org_h[0], d = g.sD * t.od + kd - g.pD;
          mbar_expect_tx(a_split(s), (uint32_t)sl.slab_bytes);
          if (g.raw_c == 1) tma_load_5d(dst, &map_x, a_split(s), w, h, d, t.n0, 0);     // [W * C][H][D][N]
          else tma_load_5d(dst, &map_x, a_split(s), w, h, d, 0, t.n0);                  // [W][H][D][C][N]
        }
        ++it;
        return true;
      });
    }
    if (*abort_word != 0u) {
      const long long start = clock64();
      while (clock64() - start < 2000000LL) { }
    }
  } else if (warp == 0) {
    // ---------------------------------------------------------------- slabs
    int s = 0;
    uint32_t ph = 1;
    for (int item = item0; item < g.n_items && alive; item += item_step) {
      const Tile t = decode<MB, PAIR>(g, item, rank);
      alive = for_steps(g, t.var, u0, u1, [&](int kd, int p, int ch, int t0, int t1) -> bool {
        (void)t0; (void)t1;
        if (!mbar_wait_warp(a_empty(s), ph, abort_word, err, ERR_A_EMPTY)) return false;
        if (lane == 0) {
          const uint32_t dst = base + (uint32_t)(s * sl.a_bytes);
          const int cw = g.sW * t.ow0 + g.org_w[p], chh = g.sH * t.oh0 + g.org_h[p], cd = g.sD * t.od + kd - g.pD;
          if (!PAIR || leader) mbar_expect_tx(a_full(s), (PAIR ? 2u : 1u) * (uint32_t)sl.slab_bytes);
          tile_load<PAIR>(g, dst, &map_x, a_full(s), ch * g.ch_el, cw, t.n0, chh, cd);
        }
        if (++s == sl.n_a) { s = 0; ph ^= 1u; }
        return true;
      });
    }
    if (*abort_word != 0u) {   // loads in flight must land before the shared memory goes away
      const long long start = clock64();
      while (clock64() - start < 2000000LL) { }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- filter tiles
    int s = 0;
    uint32_t ph = 1;
    for (int item = item0; item < g.n_items && alive; item += item_step) {
      if (resident && item != item0) break;
      const Tile tl = decode<MB, PAIR>(g, item, rank);
      const int row = tl.kb * BN + (PAIR ? (int)rank * BNH : 0);
      alive = for_steps(g, tl.var, u0, u1, [&](int kd, int p, int ch, int t0, int t1) -> bool {
        const int tap = kd * g.T_hw + g.tap0[p];
        for (int t = t0; t < t1; t += g.G) {
          if (!mbar_wait_warp(b_empty(s), ph, abort_word, err, ERR_B_EMPTY)) return false;
          const int n = min(g.G, t1 - t);
          if (lane == 0) {
            const uint32_t bytes = (uint32_t)(n * sl.b_tile);
            if (!PAIR || leader) mbar_expect_tx(b_full(s), PAIR ? 2u * bytes : bytes);
            uint32_t dst = base + (uint32_t)(sl.off_b + s * sl.b_bytes);
            for (int j = 0; j < n; ++j, dst += (uint32_t)sl.b_tile) {
              if (F32) {     // [tap][hi / lo][K][C]
                tma_load_3d(dst, &map_u, b_full(s), ch * g.ch_el, row, 2 * (tap + t + j));
                tma_load_3d(dst + (uint32_t)sl.b_lo, &map_u, b_full(s), ch * g.ch_el, row, 2 * (tap + t + j) + 1);
              } else if (PAIR) {
                tma_load_3d_pair(dst, &map_u, b_full(s), ch * g.ch_el, row, tap + t + j);
              } else {
                tma_load_3d(dst, &map_u, b_full(s), ch * g.ch_el, row, tap + t + j);
              }
            }
          }
          if (++s == sl.n_b) { s = 0; ph ^= 1u; }
        }
        return true;
      });
    }
    if (*abort_word != 0u) {
      const long long start = clock64();
      while (clock64() - start < 2000000LL) { }
    }
  } else if (warp < 2 + N_ISSUE) {
    // ---------------------------------------------------------------- MMA issue (rank 0 of a pair issues for both CTAs)
    if (leader) {
      const int me = warp - 2;
      const uint16_t pair_mask = (uint16_t)(3u << (crank & ~1u));
      int as = 0, bs = 0;
      uint32_t a_ph = 0, b_ph = 0, n_done = 0;
      for (int item = item0; item < g.n_items && alive; item += item_step, ++n_done) {
        int buf = 0;
        uint32_t d0 = 0, acc = 0, cnt = 0;        // whether this thread's accumulators hold something; K steps that went into them
        auto take = [&]() -> bool {
          buf = (int)(n_acc & 1u);
          if (!mbar_wait_warp(acc_empty(buf), ((n_acc >> 1) & 1u) ^ 1u, abort_word, err, ERR_ACC)) return false;
          tc_fence_after();
          d0 = tmem + (uint32_t)(buf * ACC + me * BN * (F32 ? 2 : 1));
          acc = cnt = 0;
          ++n_acc;
          return true;
        };
        if (!take()) { alive = false; break; }
        const bool loaded = resident && n_done > 0;
        if (resident) { bs = 0; }
        alive = for_steps(g, g.n_var > 1 ? item / g.var_items : 0, u0, u1, [&](int kd, int p, int ch, int t0, int t1) -> bool {
          if (!mbar_wait_warp(F32 ? a_split(as) : a_full(as), a_ph, abort_word, err, ERR_A)) return false;
          tc_fence_after();
          const uint32_t a_lo = desc_lo(base + (uint32_t)(as * sl.a_bytes)) + (uint32_t)(KS == 2 ? 0 : me * g.mb_off16);
          const int nk = ch == g.n_chunks - 1 ? g.k_tail : g.k_full;
          const uint16_t *rows = g.tap_off + g.tap0[p];
          for (int t = t0; t < t1; t += g.G) {
            if (!loaded) {
              if (!mbar_wait_warp(b_full(bs), b_ph, abort_word, err, ERR_B)) return false;
              tc_fence_after();
            }
            if (F32 && cnt >= (uint32_t)ACC_STEPS) {
              if (elect_one()) umma_commit<PAIR>(acc_full(buf), pair_mask);
              if (!take()) return false;
            }
            const int n = min(g.G, t1 - t);
            uint32_t b_lo = desc_lo(base + (uint32_t)(sl.off_b + bs * sl.b_bytes));
            auto k_step = [&](uint32_t a_t, int k, uint32_t keep) {
#pragma unroll
              for (int mb = 0; mb < MB; mb += N_ISSUE) {   // blocks me, me + 2, ...
                const uint32_t a_k = a_t + (uint32_t)(mb * g.mb_off16) + 2u * k, b_k = b_lo + 2u * k, d = d0 + (uint32_t)(mb * BN);
                if (F32) {     // the filter's remainders lie behind its tf32 parts: both against the slab's tf32 part in one MMA
                  umma<PAIR, F32>(d, a_k, g.a_hi, b_k, g.b_hi, idesc + ((uint32_t)(BN >> 3) << 17), keep);
                  umma<PAIR, F32>(d + BN, a_k + (uint32_t)(sl.lo_off >> 4), g.a_hi, b_k, g.b_hi, idesc, 1u);
                } else {
                  umma<PAIR, F32>(d, a_k, g.a_hi, b_k, g.b_hi, idesc, keep);
                }
              }
            };
            const bool whole = nk == 4;
            if (elect_one()) {
              // straight-line code per tap for the usual numbers of K steps, the offset of the next tap read ahead: a loop over
              // the steps costs this lone thread 180 clocks an MMA
              auto taps_of = [&](auto steps) {
                constexpr int NK = decltype(steps)::value;
                uint32_t off = rows[t];
                for (int j = 0; j < n; ++j, b_lo += (uint32_t)(sl.b_tile >> 4)) {
                  const uint32_t a_t = a_lo + off;
                  off = rows[t + j + 1];
                  if (KS == 2) { k_step(a_t, me, acc); k_step(a_t, me + 2, 1u); }
                  else {
                    k_step(a_t, 0, acc);
#pragma unroll
                    for (int k = 1; k < NK; ++k) k_step(a_t, k, 1u);
                  }
                  acc = 1u;
                }
              };
              if (whole) taps_of(std::integral_constant<int, 4>());
              else if (KS == 1 && nk == 2) taps_of(std::integral_constant<int, 2>());
              else if (KS == 1 && nk == 1) taps_of(std::integral_constant<int, 1>());
              else {
                uint32_t c = cnt;
                for (int j = 0; j < n; ++j, b_lo += (uint32_t)(sl.b_tile >> 4)) {
                  const uint32_t a_t = a_lo + rows[t + j];
                  for (int k = 0; k < nk; ++k, ++c)
                    if (KS == 1 || (c & 1u) == (uint32_t)me) { k_step(a_t, k, acc); acc = 1u; }
                }
              }
            }
            // what the elected lane did, for the others (and the next election)
            const uint32_t m = (uint32_t)(n * nk);
            if (KS == 1 || whole || m + (((cnt ^ (uint32_t)me) & 1u) ^ 1u) >= 2u) acc = 1u;
            cnt += m;
            if (!resident && elect_one()) umma_commit<PAIR>(b_empty(bs), pair_mask);
            if (++bs == sl.n_b) { bs = 0; b_ph ^= 1u; }
          }
          if (elect_one()) umma_commit<PAIR>(a_empty(as), pair_mask);
          if (++as == sl.n_a) { as = 0; a_ph ^= 1u; }
          return true;
      });
        if (resident) b_ph = 0;
        if (elect_one()) umma_commit<PAIR>(acc_full(buf), pair_mask);
      }
    }
  } else if (FOLD && warp >= SPLIT_WARP0) {
    // ---------------------------------------------------------------- gathered slabs: a thread keeps one 16-byte vector of the entries
    const int st = threadIdx.x - SPLIT_WARP0 * 32;
    const int v_shift = g.k_full == 1 ? 1 : g.k_full == 2 ? 2 : 3, v = st & ((1 << v_shift) - 1);
    const int rb_shift = v_shift + 4, swz_shift = 7 - rb_shift, swz_mask = (1 << v_shift) - 1;
    int off[8], raw_off[8];        // element offsets of the vector's values in x and in a raw patch, -1 beyond the last
    uint32_t taps_w[2] = {0, 0};   // their taps along W, four bits each
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = v * 8 + j, kw = e / g.fC, c = e - kw * g.fC;
      off[j] = kw < g.fkW ? kw * g.fx_w + c * g.fx_c : -1;
      raw_off[j] = kw < g.fkW ? kw * g.raw_w + c * g.raw_c + g.raw_rem : -1;
      taps_w[j >> 2] |= (uint32_t)(kw & 15) << (8 * (j & 3));
    }
    int s = 0;
    uint32_t ph = 1, it = 0;
    for (int item = item0; item < g.n_items && alive; item += item_step) {
      const Tile t = decode<MB, PAIR>(g, item, rank);
      alive = for_steps(g, t.var, u0, u1, [&](int kd, int, int, int, int) -> bool {
        if (!mbar_wait_warp(a_empty(s), ph, abort_word, err, ERR_A_EMPTY)) return false;
        if (g.raw_tma) {
          const int rs = (int)(it & (RAW_BUFS - 1u));
          if (!mbar_wait_warp(a_split(rs), (it / RAW_BUFS) & 1u, abort_word, err, ERR_A)) return false;
          const uint8_t *patch = base_ptr + sl.off_raw + rs * sl.raw_bytes;
          const uint32_t slab_a = base + (uint32_t)(s * sl.a_bytes);
          if (v < 2 * g.k_full) {
            const int step_px = g.sW * g.raw_w;
#pragma unroll 2
            for (int i = st >> v_shift; i < g.fold_rows * 8; i += (SPLIT_WARPS * 32) >> v_shift) {
              const unsigned short *src = reinterpret_cast<const unsigned short *>(patch) + (i >> 3) * g.raw_row + (i & 7) * step_px;
              uint32_t e[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) e[j] = raw_off[j] >= 0 ? src[raw_off[j]] : 0u;
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(slab_a + (uint32_t)((i << rb_shift) + ((v ^ ((i >> swz_shift) & swz_mask)) << 4))),
                           "r"(e[0] | (e[1] << 16)), "r"(e[2] | (e[3] << 16)), "r"(e[4] | (e[5] << 16)), "r"(e[6] | (e[7] << 16)) : "memory");
            }
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) { mbar_arrive(a_full(s)); mbar_arrive(raw_empty(rs)); }
          ++it;
          if (++s == sl.n_a) { s = 0; ph ^= 1u; }
          return true;
        }
        uint8_t *slab = base_ptr + s * sl.a_bytes;
        const int id = g.sD * t.od + kd - g.pD, ih0 = g.sH * t.oh0 + g.org_h[0], iw00 = g.sW * t.ow0 + g.org_w[0];
        const bool plane = (unsigned)id < (unsigned)g.fD && t.n0 < g.N;
        const unsigned short *xp = reinterpret_cast<const unsigned short *>(x) + t.n0 * g.fx_n + id * g.fx_d;
        if (v < 2 * g.k_full) {
#pragma unroll 2
          for (int i = st >> v_shift; i < g.fold_rows * 8; i += (SPLIT_WARPS * 32) >> v_shift) {
            const int ih = ih0 + (i >> 3), iw = iw00 + g.sW * (i & 7);
            uint32_t e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = 0;
            if (plane && (unsigned)ih < (unsigned)g.fH) {
              const unsigned short *src = xp + ih * g.fx_h + (long long)iw * g.fx_w;
              if (iw >= 0 && iw + g.fkW <= g.fW) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (off[j] >= 0) e[j] = __ldg(src + off[j]);
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (off[j] >= 0 && (unsigned)(iw + (int)((taps_w[j >> 2] >> (8 * (j & 3))) & 15u)) < (unsigned)g.fW) e[j] = __ldg(src + off[j]);
              }
            }
            *reinterpret_cast<uint4 *>(slab + (i << rb_shift) + ((v ^ ((i >> swz_shift) & swz_mask)) << 4)) =
                make_uint4(e[0] | (e[1] << 16), e[2] | (e[3] << 16), e[4] | (e[5] << 16), e[6] | (e[7] << 16));
          }
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full(s));
        if (++s == sl.n_a) { s = 0; ph ^= 1u; }
        return true;
      });
    }
  } else if (F32 && warp >= SPLIT_WARP0) {
    // ---------------------------------------------------------------- fp32: slab -> tf32 part in place, remainder beside it
    int s = 0;
    uint32_t ph = 0;
    const int st = threadIdx.x - SPLIT_WARP0 * 32;
    for (int item = item0; item < g.n_items && alive; item += item_step) {
      alive = for_steps(g, g.n_var > 1 ? item / g.var_items : 0, u0, u1, [&](int kd, int p, int ch, int t0, int t1) -> bool {
        (void)kd; (void)p; (void)ch; (void)t0; (void)t1;
        if (!mbar_wait_warp(a_full(s), ph, abort_word, err, ERR_SPLIT)) return false;
        float4 *hi = reinterpret_cast<float4 *>(base_ptr + s * sl.a_bytes);
        float4 *lo = reinterpret_cast<float4 *>(base_ptr + s * sl.a_bytes + sl.lo_off);
#pragma unroll 4
        for (int i = st; i < sl.slab_bytes / 16; i += SPLIT_WARPS * 32) {
          const float4 v = hi[i];
          float4 h;
          h.x = tf32_round(v.x); h.y = tf32_round(v.y); h.z = tf32_round(v.z); h.w = tf32_round(v.w);
          hi[i] = h;
          lo[i] = make_float4(tf32_round(v.x - h.x), tf32_round(v.y - h.y), tf32_round(v.z - h.z), tf32_round(v.w - h.w));
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_split(s));
        if (++s == sl.n_a) { s = 0; ph ^= 1u; }
        return true;
      });
    }
  } else if (warp >= EPI_WARP0 && g.split == 1) {
    // ---------------------------------------------------------------- epilogue
    // a set of eight warps per accumulator buffer, or one for both
    const int set = SETS == 2 && warp >= EPI_WARP0 + EPI_WARPS ? 1 : 0;
    const int ew = warp - EPI_WARP0 - set * EPI_WARPS;
    const int q = warp & 3, half = ew >> 2;
    const uint32_t stage = base + (uint32_t)(sl.off_stage + (set * EPI_WARPS + ew) * STAGE_BYTES);
    const uint8_t *stage_ptr = base_ptr + sl.off_stage + (set * EPI_WARPS + ew) * STAGE_BYTES;
    const bool relu = (g.epilogue & WINOCONV_EPI_RELU) != 0, has_bias = (g.epilogue & WINOCONV_EPI_BIAS) != 0;
    const bool pool = (g.epilogue & WINOCONV_EPI_POOL2) != 0;
    constexpr int CH_PER_MB = BN / COLS, N_CH = MB * CH_PER_MB;
    const int tnm = g.TN - 1;
    // this lane's pixel within the block, and the staging row its output goes to (-1: none)
    const int grp = q * 4 + (lane >> 3), h_l = grp >> g.tn_shift, w_l = (lane & 7) >> g.ti_shift, i_l = lane & (g.TI - 1);
    int srow = lane;
    if (pool) srow = ((h_l | w_l) & 1) ? -1 : ((g.TN == 1 ? lane >> 4 : grp & tnm) << 2) + ((w_l >> 1) << g.ti_shift) + i_l;
    uint32_t n_done = (uint32_t)set;
    for (int item = item0 + set * item_step; item < g.n_items; item += SETS * item_step, n_done += (uint32_t)SETS) {
      const Tile t = decode<MB, PAIR>(g, item, rank);
      const int kb = t.kb, yH = g.yH[t.var], yW = g.yW[t.var];
      const int buf = (int)(n_done & 1u);
      if constexpr (F32) {
        if (!sum_accumulators()) { alive = false; break; }
      } else {
        if (!mbar_wait_warp(acc_full(buf), (n_done >> 1) & 1u, abort_word, err, ERR_EPI)) { alive = false; break; }
        if (*abort_word != 0u) { alive = false; break; }
        tc_fence_after();
      }
      bool handed = F32;
#pragma unroll 1
      for (int ci = half; ci < N_CH; ci += 2) {
        const int mb = ci / CH_PER_MB, c0 = (ci - mb * CH_PER_MB) * COLS;
        const int k0 = kb * BN + c0;
        const int oh_b = t.oh0 + mb * g.TH;
        const bool wanted = k0 < g.K && t.valid && oh_b < g.oH;
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * ACC + mb * BN + c0);
        // 32 columns at a time, in a loop: twice the code for 64 in one piece ran slower (an epilogue warp executes it once per
        // item, mostly out of cold instruction caches)
#pragma unroll 1
        for (int hc = 0; hc < COLS; hc += 32) {
          uint32_t r[32];
          if constexpr (F32) {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(sum[i]);
          } else if (wanted) {
            tmem_ld_x32(ta + (uint32_t)hc, r);
            tmem_wait_ld_x32(r);
          }
          if (!F32 && ci + 2 >= N_CH && hc + 32 >= COLS) {      // this warp's last columns are in registers: its share of the hand-back
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { if (PAIR) mbar_arrive_rank0(acc_empty(buf)); else mbar_arrive(acc_empty(buf)); }
            handed = true;
          }
          if (!wanted) continue;
          if (has_bias) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float b[8];
              if (!F32 && g.bias_f32) load_bias<float, 8>(reinterpret_cast<const float *>(bias), k0 + hc + 8 * v, g.K, g.bias_vec, b);
              else load_bias<T, 8>(bias, k0 + hc + 8 * v, g.K, g.bias_vec, b);
#pragma unroll
              for (int i = 0; i < 8; ++i) r[8 * v + i] = __float_as_uint(__uint_as_float(r[8 * v + i]) + b[i]);
            }
          }
          constexpr int OW = 32 * (int)sizeof(T) / 4;      // words of output: 16 pairs, or 32 floats
          uint32_t o[OW];
#pragma unroll
          for (int i = 0; i < OW; ++i) {
            if constexpr (F32) o[i] = r[i];
            else o[i] = Pair16<T>::round(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          }
          if (pool) {
#pragma unroll
            for (int i = 0; i < OW; ++i) {
              o[i] = OutWord<T>::max2(o[i], __shfl_xor_sync(0xffffffffu, o[i], g.TI));
              o[i] = OutWord<T>::max2(o[i], __shfl_xor_sync(0xffffffffu, o[i], 8 << g.tn_shift));
            }
          }
          if (relu) {
#pragma unroll
            for (int i = 0; i < OW; ++i) o[i] = OutWord<T>::max2(o[i], 0u);
          }
          if (hc == 0) {
            if (lane == 0) bulk_wait_read();       // the previous store has read the staging rows
            __syncwarp();
          }
          if (srow >= 0) {
            const uint32_t dst = stage + (uint32_t)srow * 128u;
            const int v0 = hc * (int)sizeof(T) / 16;
#pragma unroll
            for (int v = 0; v < OW / 4; ++v)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)(((v0 + v) ^ (srow & 7)) << 4)), "r"(o[4 * v]),
                           "r"(o[4 * v + 1]), "r"(o[4 * v + 2]), "r"(o[4 * v + 3]) : "memory");
          }
        }
        if (!wanted) continue;
        // first pixel of this warp's rows
        const int g0 = q * 4, h0 = g0 >> g.tn_shift, n0 = (g0 & tnm) << g.ti_shift;
        if (g.y_tma) {
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && (pool ? (oh_b + h0) >> 1 : oh_b + h0) < yH && t.n0 + n0 < g.N && (pool ? t.ow0 >> 1 : t.ow0) < yW) {
            if (pool) tile_store(g, &maps_y.m[t.var], stage, k0, t.ow0 >> 1, t.n0 + n0, (oh_b + h0) >> 1, t.od);
            else tile_store(g, &maps_y.m[t.var], stage, k0, t.ow0, t.n0 + n0, oh_b + h0, t.od);
            bulk_commit();
          }
        } else {            // rows of y are not 16-byte aligned: a row of the staging tile per step, consecutive lanes, consecutive channels
          __syncwarp();
          constexpr int E = 4 / (int)sizeof(T);
          const int rows_out = pool ? 8 : 32;
          for (int rr = 0; rr < rows_out; ++rr) {
            int oh, ow, n;
            if (pool) {
              const int a = rr >> 2;
              ow = (t.ow0 >> 1) + ((rr & 3) >> g.ti_shift);
              oh = ((oh_b + h0) >> 1) + (g.TN == 1 ? a : 0);
              n = t.n0 + ((g.TN == 1 ? 0 : a) << g.ti_shift) + (rr & (g.TI - 1));
            } else {
              const int gg = g0 + (rr >> 3);
              oh = oh_b + (gg >> g.tn_shift); n = t.n0 + ((gg & tnm) << g.ti_shift) + (rr & (g.TI - 1)); ow = t.ow0 + ((rr & 7) >> g.ti_shift);
            }
            if (oh >= yH || ow >= yW || n >= g.N) continue;
            const T *src = reinterpret_cast<const T *>(stage_ptr + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) + (lane & 3) * 4);
            T *dst = y + g.y_off[t.var] + n * g.ys_n + t.od * g.ys_d + oh * g.ys_h + ow * g.ys_w + k0 + lane * E;
#pragma unroll
            for (int e = 0; e < E; ++e)
              if (k0 + lane * E + e < g.K) dst[e] = src[e];
          }
          __syncwarp();
        }
      }
      if (!handed && lane == 0) { if (PAIR) mbar_arrive_rank0(acc_empty(buf)); else mbar_arrive(acc_empty(buf)); }
    }
    if (lane == 0) bulk_wait_read();     // the staging rows are read before the CTA's shared memory goes
  }
  if (F32 && g.split > 1 && warp >= EPI_WARP0 && warp < EPI_WARP0 + EPI_WARPS && item0 < g.n_items) alive = sum_accumulators();
  if (g.split > 1) {
    // ---------------------------------------------------------------- the cluster's shares of one item added up
    // Every CTA puts its accumulator into its own shared memory (the operand rings are idle by then) and finishes 1 / split
    // of the rows from all of them.
    constexpr int ROW_F = BN + 4;                  // floats per row: 16-byte accesses of neighbouring rows hit other banks
    const bool epi = warp >= EPI_WARP0 && warp < EPI_WARP0 + EPI_WARPS;
    __syncthreads();
    if (epi && item0 < g.n_items) {
      const int q = warp & 3, half = (warp - EPI_WARP0) >> 2;
      if (F32 || mbar_wait_warp(acc_full(0), 0u, abort_word, err, ERR_EPI)) {
        tc_fence_after();
        for (int c0 = half * 32; c0 < MB * BN; c0 += 64) {
          uint32_t r[32];
          if constexpr (F32) {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(sum[i]);
          } else {
            tmem_ld_x32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, r);
            tmem_wait_ld_x32(r);
          }
          const int mb = c0 / BN;
          float4 *dst = reinterpret_cast<float4 *>(base_ptr) + ((mb * BM + q * 32 + lane) * ROW_F + (c0 - mb * BN)) / 4;
#pragma unroll
          for (int v = 0; v < 8; ++v)
            dst[v] = make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]), __uint_as_float(r[4 * v + 2]), __uint_as_float(r[4 * v + 3]));
        }
        tc_fence_before();
      }
    }
    cluster_sync_all();
    if (epi && *abort_word == 0u) {
      const Tile t = decode<MB, PAIR>(g, item0, rank);
      const int kb = t.kb;
      const bool relu = (g.epilogue & WINOCONV_EPI_RELU) != 0, has_bias = (g.epilogue & WINOCONV_EPI_BIAS) != 0;
      const bool pool = (g.epilogue & WINOCONV_EPI_POOL2) != 0;
      constexpr int V = 4;                         // a warp reads 512 consecutive bytes of a row of each peer
      const int rows = MB * BM / g.split, tid = threadIdx.x - EPI_WARP0 * 32;
      const int work = (pool ? rows / 4 : rows) * (BN / V);
      for (int i = tid; i < work; i += EPI_WARPS * 32) {
        const int rr = i / (BN / V), c = (i - rr * (BN / V)) * V;
        const int k = kb * BN + c;
        if (k >= g.K) continue;
        float best[V];
        int oh = 0, ow = 0, n = 0;
        const int n_src = pool ? 4 : 1;
        for (int a = 0; a < n_src; ++a) {
          int row = (int)part * rows;
          if (pool) {    // pooled pixel rr: row pair, image group, column pair and image within this CTA's rows
            const int wp = (rr & 3) >> g.ti_shift, np = (rr >> 2) & (g.TN - 1), hp = rr >> (2 + g.tn_shift);
            row += (((2 * hp + (a >> 1)) << g.tn_shift) + np) * 8 + ((2 * wp + (a & 1)) << g.ti_shift) + (rr & (g.TI - 1));
          } else row += rr;
          float f[V];
#pragma unroll
          for (int v = 0; v < V; ++v) f[v] = 0.f;
          const uint32_t src = base + (uint32_t)((row * ROW_F + c) * 4);
          // all peers' values in flight at once: one remote read takes as long as eight
          auto add_peers = [&](auto n_peers) {
            constexpr int S = decltype(n_peers)::value;
            float4 u[S];
#pragma unroll
            for (int i2 = 0; i2 < S; ++i2) {
              const uint32_t pr = ((uint32_t)i2 + part) & (uint32_t)(S - 1);     // every CTA starts at another peer
              u[i2] = ld_cluster_f4(map_to_rank(src, PAIR ? 2u * pr + rank : pr));   // (of a pair's, those with the same pixels)
            }
#pragma unroll
            for (int i2 = 0; i2 < S; ++i2) { f[0] += u[i2].x; f[1] += u[i2].y; f[2] += u[i2].z; f[3] += u[i2].w; }
          };
          if (g.split == 2) add_peers(std::integral_constant<int, 2>());
          else if (g.split == 4) add_peers(std::integral_constant<int, 4>());
          else add_peers(std::integral_constant<int, 8>());
          if (a == 0) {
            const int mb = row >> 7, grp = (row & 127) >> 3;
            oh = t.oh0 + mb * g.TH + (grp >> g.tn_shift); n = t.n0 + ((grp & (g.TN - 1)) << g.ti_shift) + (row & (g.TI - 1));
            ow = t.ow0 + ((row & 7) >> g.ti_shift);
          }
#pragma unroll
          for (int v = 0; v < V; ++v) best[v] = a == 0 ? f[v] : fmaxf(best[v], f[v]);
        }
        if (pool) { oh >>= 1; ow >>= 1; }
        if (oh >= g.yH[t.var] || ow >= g.yW[t.var] || n >= g.N || !t.valid) continue;
        if (has_bias) {
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (k + v < g.K) best[v] += g.bias_f32 ? reinterpret_cast<const float *>(bias)[k + v] : Elem<T>::load(bias + k + v);
        }
        if (relu) {
#pragma unroll
          for (int v = 0; v < V; ++v) best[v] = fmaxf(best[v], 0.f);
        }
        T *dst = y + g.y_off[t.var] + n * g.ys_n + t.od * g.ys_d + oh * g.ys_h + ow * g.ys_w + k;
        if (g.y_tma) VecIO<T, 4>::store(dst, best);       // K a multiple of 8 (4): whole, aligned vectors
        else {
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (k + v < g.K) Elem<T>::store(dst + v, best[v]);
        }
      }
    }
    cluster_sync_all();      // no CTA leaves while another reads its shared memory
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  if (warp == 2) {
    tc_fence_after();
    tmem_free<PAIR>(tmem, tmem_cols);
  }
}

// U[tap][o][i] = w[o, i, tap] in the order the kernel walks the taps, rounded once to T; fp32 as [tap][tf32 part, remainder][o][i].
// The weights are read through strides, so a data gradient's filter (channels exchanged, taps mirrored) is the same kernel.
struct FGeomD {
  int O, I, Ip, kD, n_hw, fold;      // fold > 0: input i is tap i / fold along W of channel i % fold
  long long s_o, s_i, s_d, off_d, s_w;
  int off_hw[MAX_TAPS];       // element offset of each (h, w) tap in walking order
};
template <typename TW, typename T>
__global__ void __launch_bounds__(256) direct_filter_kernel(const TW *__restrict__ w, T *__restrict__ u, const __grid_constant__ FGeomD f) {
  const unsigned idx = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned total = (unsigned)f.O * (unsigned)f.Ip;
  if (idx >= total) return;
  const int o = (int)(idx / (unsigned)f.Ip), i = (int)(idx - (unsigned)o * (unsigned)f.Ip);
  const int kw = f.fold ? i / f.fold : 0;
  const TW *src = w + o * f.s_o + (i - kw * f.fold) * f.s_i + kw * f.s_w;
  const bool real = i < f.I;
  const int kd = blockIdx.y;
  for (int t = blockIdx.z; t < f.n_hw; t += gridDim.z) {
    const float v = real ? Elem<TW>::load(src + f.off_d + kd * f.s_d + f.off_hw[t]) : 0.f;
    const long long tap = (long long)kd * f.n_hw + t;
    if constexpr (std::is_same<T, float>::value) {
      const float h = tf32_round(v);
      u[2 * tap * total + idx] = h;
      u[(2 * tap + 1) * total + idx] = tf32_round(v - h);      // the tensor core would cut it off
    } else {
      Elem<T>::store(u + tap * total + idx, v);
    }
  }
}

static int sm_count_of_current_device() {
  static std::mutex mu;
  static std::map<int, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  auto f = cache.find(dev);
  if (f != cache.end()) return f->second;
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
  return cache[dev] = n;
}

}  // namespace dconv

using namespace dconv;

// Clusters of this many CTAs that 148 SMs hold at once, one CTA per SM (cudaOccupancyMaxActiveClusters on B200: clusters of 4
// and 8 do not fill every GPC).
static int clusters_at_once(int width) { return width == 1 ? 148 : width == 2 ? 74 : width == 4 ? 33 : 15; }

// Estimated clocks of a launch with this configuration on 148 SMs.  An item takes as long as its MMAs (66 / 130 clocks an
// instruction of 128 / 256 columns; of 64 columns 60 from one issuing thread, 48 from two), its shared-memory traffic at 128 B
// per clock, or its loads: about 28 B per clock and SM from L2 when all SMs load, at most 60 for one.  Set-up, first loads
// and drain of a launch were measured at about 8000 clocks, 800 more for a pair, 4600 for a cluster's exchange of partial sums.
static double item_clocks(const DirectPlan &p, double k_steps, int n_steps, int n_var, bool f32) {
  const double t_mma = p.BN == 256 ? 130 : p.BN == 128 ? 66 : p.MB >= 2 || f32 ? 48 : 60;
  const int bn_own = p.pair ? p.BN / 2 : p.BN;
  const double mma = k_steps * p.MB * t_mma * (f32 ? 3 : 1);
  const double loads = n_steps * (double)p.slab_bytes + k_steps * bn_own * 32.0 * (f32 ? 2 : 1);
  const double smem = k_steps * p.MB * (f32 ? 3 : 1) * (4096.0 + bn_own * 32.0) + loads + (f32 ? 3.0 * n_steps * p.slab_bytes : 0.0);
  const double active = std::min(148.0, (double)p.n_items * n_var * (p.pair ? 2 : 1) * p.split);
  const double l2 = loads / std::min(60.0, 28.0 * 148 / active);
  return std::max(mma, std::max(smem / 128.0, l2));
}
static double waves_of(const DirectPlan &p, int n_var) {
  const int slots = clusters_at_once((p.pair ? 2 : 1) * p.split);
  return (p.n_items * n_var + slots - 1) / slots;
}
static double estimate(const DirectPlan &p, double k_steps, int n_steps, int n_var, bool f32) {
  const double item = item_clocks(p, k_steps, n_steps, n_var, f32), waves = waves_of(p, n_var);
  const double epi = 400.0 + 350.0 * p.MB * p.BN / 64;
  const double tail = 1500.0 * ((p.MB * p.BN / (f32 ? 32 : 64) + 1) / 2 - 1);     // the last epilogue
  if (p.split > 1) return 8000.0 + (p.pair ? 800.0 : 0.0) + item / p.split + 4000.0 + 10.0 * p.BN * p.MB;
  return 8000.0 + (p.pair ? 800.0 : 0.0) + waves * std::max(item + 200.0, epi) + tail;
}

// Stages of the slab and filter rings within `budget` bytes, the ring that looks less far ahead growing first; taps per filter
// stage (G) so that a stage is worth its barrier round trip.
static bool ring_depths(DirectPlan &q, int taps, int budget) {
  for (int G = std::max(1, std::min(taps, 24 * 1024 / q.b_tile)); G >= 1; --G) {
    q.G = G;
    q.b_bytes = (G * q.b_tile + 1023) / 1024 * 1024;
    int na = 2, nb = 2;
    if (2 * q.a_bytes + 2 * q.b_bytes > budget) {
      na = 1;
      if (q.a_bytes + 2 * q.b_bytes > budget) continue;
    }
    const double groups = (taps + G - 1) / G;
    for (bool grew = true; grew;) {
      grew = false;
      const bool want_b = nb / groups <= na;
      for (int turn = 0; turn < 2 && !grew; ++turn) {
        const bool b = turn == 0 ? want_b : !want_b;
        if (b && nb < 8 && na * q.a_bytes + (nb + 1) * q.b_bytes <= budget) { ++nb; grew = true; }
        if (!b && na < 8 && (na + 1) * q.a_bytes + nb * q.b_bytes <= budget) { ++na; grew = true; }
      }
    }
    q.n_a = na; q.n_b = nb;
    return true;
  }
  return false;
}

void direct_forward_desc(DirectDesc *q, int dtype, int N, int C, int K, const int in[3], const int ker[3], const int stride[3],
                         const int pad[3], const int out[3], int yH, int yW, unsigned epilogue, int weight_layout) {
  std::memset(q, 0, sizeof *q);
  q->dtype = dtype; q->N = N; q->C = q->Cw = C; q->K = K; q->D = in[0]; q->H = in[1]; q->W = in[2];
  q->oD = out[0]; q->oH = out[1]; q->oW = out[2]; q->yH = yH; q->yW = yW;
  q->sD = stride[0]; q->sH = stride[1]; q->sW = stride[2]; q->pD = pad[0];
  q->kD = q->kD_w = ker[0]; q->kH_w = ker[1]; q->kW_w = ker[2];
  q->d0 = 0; q->ds = 1;
  q->ys_w = K; q->ys_h = q->ys_w * yW; q->ys_d = q->ys_h * yH; q->ys_n = q->ys_d * out[0];
  q->epilogue = epilogue; q->weight_layout = weight_layout;
  for (int a = 0; a < stride[1]; ++a)
    for (int b = 0; b < stride[2]; ++b) {
      DirectPart p;
      std::memset(&p, 0, sizeof p);
      p.th = (ker[1] - a + stride[1] - 1) / stride[1]; p.tw = (ker[2] - b + stride[2] - 1) / stride[2];
      if (p.th <= 0 || p.tw <= 0) continue;
      p.org_h = a - pad[1]; p.org_w = b - pad[2];
      p.t0_h = a; p.ts_h = stride[1]; p.t0_w = b; p.ts_w = stride[2];
      q->parts[q->n_parts++] = p;
    }
}

// grad_x[i] = sum over taps t with (i + p - t) divisible by s of grad_y[(i + p - t) / s] w[t].  For inputs i = s j + r these are
// the taps t = t0 + s m, t0 = (r + p) mod s, and the gradient is a stride-1 convolution of grad_y over j with the taps m
// mirrored: a part per residue (r_h, r_w), writing every s-th pixel.
bool direct_grad_desc(DirectDesc *q, int dtype, int N, int C, int K, int Km, const int in[3], const int ker[3], const int stride[3],
                      const int pad[3], const int out[3], int weight_layout, int e, bool *zero_fill) {
  std::memset(q, 0, sizeof *q);
  struct Axis { int r, m, org, t0, n; };       // residue, taps, first input of output 0, last tap (mirrored order starts there), outputs
  auto axis = [&](int i, int r) {
    Axis a;
    const int s = stride[i], t0 = (r + pad[i]) % s;
    a.r = r;
    a.m = ker[i] > t0 ? (ker[i] - t0 + s - 1) / s : 0;
    a.org = (r + pad[i] - t0) / s - (a.m - 1);
    a.t0 = t0 + s * (a.m - 1);
    a.n = (in[i] - r + s - 1) / s;
    return a;
  };
  const Axis dz = axis(0, e);
  q->dtype = dtype; q->N = N; q->C = Km; q->Cw = K; q->K = C; q->D = out[0]; q->H = out[1]; q->W = out[2];
  q->oD = dz.n; q->sD = q->sH = q->sW = 1; q->pD = -dz.org; q->kD = dz.m; q->d0 = dz.t0; q->ds = -stride[0];
  q->kD_w = ker[0]; q->kH_w = ker[1]; q->kW_w = ker[2];
  const long long w_ = C, h_ = w_ * in[2], d_ = h_ * in[1], n_ = d_ * in[0];
  q->ys_w = w_ * stride[2]; q->ys_h = h_ * stride[1]; q->ys_d = d_ * stride[0]; q->ys_n = n_;
  q->weight_layout = weight_layout; q->transposed = 1; q->variants = 1;
  if (dz.n <= 0) return true;                  // no input of this parity
  for (int a = 0; a < stride[1]; ++a)
    for (int b = 0; b < stride[2]; ++b) {
      const Axis h = axis(1, a), w = axis(2, b);
      if (h.n <= 0 || w.n <= 0) continue;
      if (h.m == 0 || w.m == 0 || dz.m == 0) { *zero_fill = true; continue; }      // inputs that no output reads
      DirectPart p;
      p.org_h = h.org; p.org_w = w.org; p.th = h.m; p.tw = w.m;
      p.t0_h = h.t0; p.ts_h = -stride[1]; p.t0_w = w.t0; p.ts_w = -stride[2];
      p.oH = h.n; p.oW = w.n;
      p.y_off = e * d_ + a * h_ + b * w_;
      q->oH = std::max(q->oH, h.n); q->oW = std::max(q->oW, w.n);
      q->parts[q->n_parts++] = p;
    }
  q->yH = q->oH; q->yW = q->oW;
  return true;
}

bool direct_fold_desc(DirectDesc *q, const int pad[3], int x_first) {
  if (q->dtype == WINOCONV_F32 || q->variants || q->transposed || q->Cw * q->kW_w > 64 || q->kW_w > 10) return false;
  if ((long long)q->D * q->H * q->W * q->Cw > 0x7fffffffLL) return false;      // offsets within an image are 32-bit
  q->fold = 1;
  q->x_first = x_first;
  q->n_parts = 1;
  DirectPart &p = q->parts[0];
  std::memset(&p, 0, sizeof p);
  p.th = q->kH_w; p.tw = 1; p.ts_h = 1; p.ts_w = 1;
  p.org_h = -pad[1]; p.org_w = -pad[2];
  return true;
}

// The folded kernel: 64 columns, one or two row blocks (two keep both halves of the epilogue warps busy), the filter resident
// where one channel block covers K.
static bool fold_plan(const DirectDesc &d, DirectPlan *out) {
  DirectPlan p;
  std::memset(&p, 0, sizeof p);
  const int fold = d.Cw * d.kW_w, rows = d.parts[0].th;
  p.k_full = p.k_tail = (fold + 15) / 16;
  p.ch_el = p.k_full == 1 ? 16 : p.k_full == 2 ? 32 : 64;
  p.rb = 2 * p.ch_el;
  p.n_chunks = 1;
  p.taps[0] = p.max_taps = p.n_taps = rows;
  p.units = d.kD * rows;
  p.filter_elems = (long long)d.kD * rows * d.K * p.ch_el;
  p.BN = 64; p.split = 1; p.TN = 1; p.TH = 16; p.TI = 1; p.PW = 8;
  p.n_kb = (d.K + 63) / 64;
  p.n_wb = (d.oW + 7) / 8;
  for (int mb = 2; mb >= 1; --mb) {
    DirectPlan q = p;
    q.MB = mb;
    q.n_hb = (d.oH + 16 * mb - 1) / (16 * mb);
    const long long tiles = (long long)q.n_wb * q.n_hb * d.oD * d.N;
    if (tiles * p.n_kb > 0x3fffffffLL) continue;
    if (mb == 2 && tiles * p.n_kb < 148) continue;       // not even one item per SM
    q.n_tiles = (int)tiles; q.n_items = (int)(tiles * p.n_kb);
    q.slab_rows_h = d.sH * (16 * mb - 1) + rows;
    q.slab_bytes = q.slab_rows_h * 8 * q.rb;
    q.a_bytes = q.lo_off = (q.slab_bytes + 1023) / 1024 * 1024;
    q.b_lo = q.b_tile = 64 * q.rb;
    // the raw patch (see launch): rows of (8 - 1) * stride + kW pixels of C channels from a multiple of eight elements on
    const int px = d.sW * 7 + d.kW_w;
    const bool first = d.x_first != 0;
    const long long row = first ? d.W : (long long)d.W * d.Cw;
    q.raw_rem = first ? ((d.parts[0].org_w % 8) + 8) % 8 : ((d.parts[0].org_w * d.Cw) % 8 + 8) % 8;
    q.raw_el = ((first ? px : px * d.Cw) + q.raw_rem + 7) / 8 * 8;
    q.raw_tma = row % 8 == 0 && q.raw_el <= 256 && q.slab_rows_h <= 256 && (!first || d.Cw <= 256);
    q.raw_box = q.raw_tma ? q.slab_rows_h * q.raw_el * 2 * (first ? d.Cw : 1) : 0;
    const int raws = (int)RAW_BUFS * ((q.raw_box + 127) / 128 * 128);
    q.epi_sets = 1;
    if (!ring_depths(q, rows, 227 * 1024 - FIXED_BYTES - raws)) continue;
    q.smem = FIXED_BYTES + raws + q.n_a * q.a_bytes + q.n_b * q.b_bytes;
    *out = q;
    return true;
  }
  return false;
}

bool direct_plan(const DirectDesc &d, DirectPlan *out) {
  if (d.n_parts == 0) return false;
  if (d.fold) return fold_plan(d, out);
  const bool f32 = d.dtype == WINOCONV_F32;
  const int esz = f32 ? 4 : 2, vec = 16 / esz;
  if (d.C % vec != 0 || (f32 && d.variants)) return false;
  const bool pool = (d.epilogue & WINOCONV_EPI_POOL2) != 0;
  DirectPlan p;
  std::memset(&p, 0, sizeof p);
  // channels per slab row: 128-byte rows, or 64 / 32-byte rows where the channels fit them
  const int cap = 128 / esz;
  p.ch_el = d.C > cap / 2 ? cap : d.C > cap / 4 ? cap / 2 : cap / 4;
  p.rb = p.ch_el * esz;
  p.n_chunks = (d.C + p.ch_el - 1) / p.ch_el;
  const int k_el = 32 / esz;                 // channels of one MMA K step
  p.k_full = p.ch_el / k_el;
  p.k_tail = (d.C - (p.n_chunks - 1) * p.ch_el + k_el - 1) / k_el;
  int Th = 0, Tw = 0, n_taps = 0;            // largest part
  for (int q = 0; q < d.n_parts; ++q) {
    Th = std::max(Th, d.parts[q].th); Tw = std::max(Tw, d.parts[q].tw);
    p.taps[q] = d.parts[q].th * d.parts[q].tw;
    p.tap0[q] = n_taps;
    n_taps += p.taps[q];
    p.max_taps = std::max(p.max_taps, p.taps[q]);
  }
  if (n_taps == 0 || n_taps > MAX_TAPS) return false;
  p.n_taps = n_taps;
  p.filter_elems = (long long)d.kD * n_taps * d.K * d.C * (f32 ? 2 : 1);
  const int n_var = d.variants ? d.n_parts : 1, item_taps = d.variants ? p.max_taps : n_taps;
  p.units = d.kD * item_taps * p.n_chunks;
  const double k_steps = (double)d.kD * n_taps / n_var * ((p.n_chunks - 1) * p.k_full + p.k_tail);
  const int n_steps = d.kD * (d.variants ? 1 : d.n_parts) * p.n_chunks;

  struct Cfg { int BN, MB, pair; };
  static const Cfg cfgs16[] = {{256, 1, 1}, {128, 2, 1}, {128, 1, 1}, {64, 2, 1}, {128, 1, 0}, {64, 1, 0}, {64, 2, 0}};
  static const Cfg cfgs32[] = {{64, 1, 0}};
  const Cfg *cfgs = f32 ? cfgs32 : cfgs16;
  const int n_cfgs = f32 ? 1 : 7;
  double best = 1e30;
  bool found = false;
  for (int ci = 0; ci < n_cfgs; ++ci) {
    const Cfg &c = cfgs[ci];
    if (c.BN > 64 && d.K <= c.BN / 2) continue;
    const int n_kb = (d.K + c.BN - 1) / c.BN;
    for (int ti = 1; ti <= 8; ti *= 2)
    for (int tn = 1; tn <= 16; tn *= 2) {
      if (pool && (tn > 2 || ti > 4)) continue;
      if (ti * tn > 1 && ti * tn / 2 >= d.N) continue;
      if (ti > 1 && tn > 1 && (d.D != 1 || d.oD != 1 || d.kD != 1 || d.pD != 0 || d.N % ti != 0)) continue;
      DirectPlan q = p;
      q.BN = c.BN; q.MB = c.MB; q.pair = c.pair; q.TN = tn; q.TH = 16 / tn; q.TI = ti;
      q.PW = 8 / ti + Tw - 1;
      const int rows_h = c.MB * q.TH + Th - 1;
      if (q.PW * d.sW > 256 || rows_h * d.sH > 256) continue;
      q.slab_rows_h = rows_h;
      q.slab_bytes = rows_h * tn * q.PW * ti * q.rb;
      const int a1 = (q.slab_bytes + 1023) / 1024 * 1024;
      q.a_bytes = f32 ? 2 * a1 : a1;
      q.lo_off = a1;
      q.b_lo = (c.pair ? c.BN / 2 : c.BN) * q.rb;
      q.b_tile = q.b_lo * (f32 ? 2 : 1);
      q.n_wb = (d.oW + 8 / ti - 1) / (8 / ti); q.n_hb = (d.oH + c.MB * q.TH - 1) / (c.MB * q.TH);
      const long long tiles = (long long)q.n_wb * q.n_hb * d.oD * ((d.N + tn * ti - 1) / (tn * ti));
      if (tiles * n_kb * n_var > 0x3fffffffLL) continue;
      q.n_tiles = (int)tiles; q.n_kb = n_kb;
      q.n_items = (int)((c.pair ? (tiles + 1) / 2 : tiles) * n_kb);
      for (int split = 1; split <= 8; split *= 2) {
        const int width = split * (c.pair ? 2 : 1);
        if (split > 1 && (width > 8 || d.variants || q.n_items > clusters_at_once(width) || split > q.units)) break;
        if (split > 1 && pool && c.MB * BM / split < 16 * tn) break;
        q.split = split;
        if (!ring_depths(q, p.max_taps, 227 * 1024 - FIXED_BYTES)) continue;
        if (split > 1 && c.MB * BM * (c.BN + 4) * 4 > q.n_a * q.a_bytes + q.n_b * q.b_bytes) continue;
        const double e = estimate(q, k_steps, n_steps, n_var, f32);
        if (e < best) { best = e; *out = q; found = true; }
      }
    }
  }
  if (!found) return false;
  out->estimate = best;
  out->epi_sets = 1;
  // A second set of epilogue warps, where a CTA has several items and their epilogues (about 4000 clocks for two 64-column pieces,
  // one each for the two halves of a set) take more than twice as long as their loads and MMAs.  us on B200, one set / two, N = 32:
  // 1x1 64 -> 64 at 112x112 26.5 / 22.1, 64 -> 256 at 56x56 24.5 / 20.7; 3x3 16 -> 64 at 112x112 24.5 / 21.1, 8 -> 64 26.2 / 22.7.
  // With more MMAs an item it loses ring depth and registers (640 threads: 80 each): 1x1 256 -> 64 at 56x56 13.0 / 13.9, 3x3
  // 64 -> 64 at 112x112 30.5 / 31.3; the gathered stem (7x7 at stride 2, 768 threads, spills) 37.4 / 50.0.
  if (!f32 && out->split == 1 && waves_of(*out, n_var) > 1 &&
      2.0 * (item_clocks(*out, k_steps, n_steps, n_var, f32) + 200.0) < 4000.0 * ((out->MB * out->BN / 64 + 1) / 2)) {
    DirectPlan q = *out;
    if (ring_depths(q, p.max_taps, 227 * 1024 - FIXED_BYTES - SET_BYTES)) { *out = q; out->epi_sets = 2; }
  }
  out->smem = FIXED_BYTES + (out->epi_sets - 1) * SET_BYTES + out->n_a * out->a_bytes + out->n_b * out->b_bytes;
  return true;
}

// Microseconds of a folded layer: what an item takes -- the gather (an iteration moves 128 vectors, from a TMA patch or by plain
// loads), the MMAs or the epilogue -- times the rounds of items on 148 SMs.  Fitted to 1300 folded layers of 1 to 64 channels,
// 1x1 to 9x9, K = 16 to 512, 2-D and 3-D, strides 1 and 2 on B200: rms 10 %, at most 45 % off.
static double fold_us(const DirectDesc &d, const DirectPlan &p) {
  const int lanes = p.k_full == 1 ? 2 : p.k_full == 2 ? 4 : 8;
  const double gather = d.kD * (std::ceil(p.slab_rows_h * 8 * lanes / 128.0) * (p.raw_tma ? 230.0 : 725.0) + 950.0);
  const double mma = 48.0 * d.kD * d.parts[0].th * p.k_full * p.MB;
  return 7.0 + std::ceil(p.n_items / 148.0) * std::max(std::max(gather, 550.0 + 1580.0 * p.MB), mma) / 1900.0;
}
// ... and of the same layer on padded channels, its copy included (rms 13 %; `estimate` is half of what layers of so few
// channels take).
static double padded_us(const DirectDesc &d, const DirectPlan &p) {
  const double copied = d.C == d.Cw ? 0.0 : 2.0 * d.N * d.D * d.H * d.W * (d.C + d.Cw);
  return 1.2 + 1.98 * p.estimate / 1900.0 + copied / 5.25e6;
}

// Folding saves the copy and most K steps, but every 64 output channels gather x again: it loses where those are many, entries
// long or rows not 16-byte multiples.  us folded / padded on B200: 3 -> 64 7x7 s2, N = 32, at 225x225 (plain loads) 101 / 58; 6 -> 328
// 3x3x3 s2 at 24x34x41, N = 16: 369 / 69; 16 -> 96 1x1 at 99x99, N = 61, from torch's order 134 / 51 with the copy; 3 -> 64 3x3 at
// 56x56, N = 16: 12 / 15.  Over 2849 layers of 1 to 64 channels the rule takes 0.79 of always folding; it folds where the two are
// close, and is slower than folding by more than 5 % on 25 of them (at most 15 %).
bool direct_fold_pays(const DirectDesc &fold, const DirectPlan &fp, const DirectDesc &plain, const int pad[3]) {
  DirectPlan p;
  if (!direct_plan(plain, &p)) return true;
  double other = padded_us(plain, p);
  if (!fold.x_first) return fold_us(fold, fp) < 1.25 * other;
  if (plain.C != plain.Cw) {
    DirectDesc last = plain;
    last.C = last.Cw;
    if (direct_fold_desc(&last, pad, 0) && direct_plan(last, &p)) other = std::min(other, fold_us(last, p));
  }
  const double turn = 2.3 + 4.0 * fold.N * fold.D * fold.H * fold.W * fold.Cw / 9.9e6;
  return fold_us(fold, fp) < 1.15 * (turn + other);
}

cudaError_t launch_direct_filter_transform(const DirectDesc &d, const DirectPlan &p, int w_dtype, const void *w, void *u, cudaStream_t s) {
  FGeomD f;
  std::memset(&f, 0, sizeof f);
  f.O = d.K; f.I = d.fold ? d.Cw * d.kW_w : d.Cw; f.Ip = d.fold ? p.ch_el : d.C; f.kD = d.kD; f.n_hw = p.n_taps; f.fold = d.fold ? d.Cw : 0;
  // the weights' own channel counts: [Kw][Cw][taps] or [taps][Cw][Kw]
  const long long Kw = d.transposed ? d.Cw : d.K, Cw = d.transposed ? d.K : d.Cw;
  const bool kcrs = d.weight_layout == WINOCONV_W_KCRS;
  const long long hw = (long long)d.kH_w * d.kW_w, tap_stride = kcrs ? 1 : Cw * Kw;
  const long long s_k = kcrs ? Cw * d.kD_w * hw : 1, s_c = kcrs ? d.kD_w * hw : Kw;
  f.s_o = d.transposed ? s_c : s_k;
  f.s_i = d.transposed ? s_k : s_c;
  f.s_w = tap_stride;
  f.off_d = d.d0 * hw * tap_stride;
  f.s_d = d.ds * hw * tap_stride;
  for (int q = 0; q < d.n_parts; ++q) {
    const DirectPart &a = d.parts[q];
    for (int t = 0; t < p.taps[q]; ++t) {
      const int th = t / a.tw, tw = t - th * a.tw;
      f.off_hw[p.tap0[q] + t] = (int)(((a.t0_h + a.ts_h * th) * d.kW_w + a.t0_w + a.ts_w * tw) * tap_stride);
    }
  }
  const unsigned blocks = (unsigned)(((long long)f.O * f.Ip + 255) / 256);
  const dim3 grid(blocks, (unsigned)d.kD, blocks >= 296 ? 1 : std::min(p.n_taps, (int)(592 / blocks) + 1));
#define WINO_FILT(TW, T) direct_filter_kernel<TW, T><<<grid, 256, 0, s>>>((const TW *)w, (T *)u, f)
  if (d.dtype == WINOCONV_F32) WINO_FILT(float, float);
  else if (d.dtype == WINOCONV_F16) { if (w_dtype == WINOCONV_F32) WINO_FILT(float, __half); else WINO_FILT(__half, __half); }
  else { if (w_dtype == WINOCONV_F32) WINO_FILT(float, __nv_bfloat16); else WINO_FILT(__nv_bfloat16, __nv_bfloat16); }
#undef WINO_FILT
  return cudaGetLastError();
}

template <typename T, int BN, int MB, bool PAIR, bool FOLD = false, int SETS = 1>
static cudaError_t launch_one(const DirectPlan &p, const CUtensorMap &mx, const CUtensorMap &mu, const MapSet &my, const void *x, void *y,
                              const void *bias, const DGeom &g, const DSmem &sl, uint32_t idesc, int sms, cudaStream_t s) {
  auto kern = direct_kernel<T, BN, MB, PAIR, FOLD, SETS>;
  static std::mutex mu_;
  static std::map<int, int> pairs_of;     // device -> resident CTA pairs (0: attribute set, not asked)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(threads_of(std::is_same<T, float>::value || FOLD, SETS), 1, 1);
  cfg.dynamicSmemBytes = (size_t)p.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (PAIR ? 2u : 1u) * (unsigned)p.split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (PAIR || p.split > 1) ? 2 : 1;
  int pairs = 0;
  {
    std::lock_guard<std::mutex> lock(mu_);
    auto f = pairs_of.find(dev);
    if (f == pairs_of.end()) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      f = pairs_of.emplace(dev, 0).first;
      if (PAIR) {
        cfg.gridDim = dim3(2, 1, 1);
        cfg.dynamicSmemBytes = 227 * 1024;
        attr[1].val.clusterDim.x = 2;
        if (cudaOccupancyMaxActiveClusters(&f->second, kern, &cfg) != cudaSuccess || f->second <= 0) f->second = sms / 2;
        cfg.dynamicSmemBytes = (size_t)p.smem;
        attr[1].val.clusterDim.x = 2u * (unsigned)p.split;
      }
    }
    pairs = f->second;
  }
  if (p.split > 1) cfg.gridDim = dim3((unsigned)(g.n_items * p.split) * (PAIR ? 2u : 1u), 1, 1);
  else if (PAIR) cfg.gridDim = dim3((unsigned)(2 * std::min(g.n_items, std::min(pairs, sms / 2))), 1, 1);
  else cfg.gridDim = dim3((unsigned)std::min(g.n_items, sms), 1, 1);
  return cudaLaunchKernelEx(&cfg, kern, mx, mu, my, (const T *)x, (T *)y, (const T *)bias, g, sl, idesc);
}

cudaError_t launch_direct_forward(const DirectDesc &d, const DirectPlan &p, const void *x, const void *u, const void *bias, void *y,
                                  cudaStream_t s, const char **detail) {
  *detail = "";
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) { *detail = "cuTensorMapEncodeTiled unavailable"; return cudaErrorNotSupported; }
  const bool f32 = d.dtype == WINOCONV_F32, pool = (d.epilogue & WINOCONV_EPI_POOL2) != 0;
  const cuuint64_t esz = f32 ? 4 : 2;
  const CUtensorMapDataType dt = map_dtype(d.dtype);
  const CUtensorMapSwizzle swz = p.rb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : p.rb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
  const uint32_t swz_code = p.rb == 128 ? 2u : p.rb == 64 ? 4u : 6u;
  CUtensorMap mx, mu;
  MapSet my;
  std::memset(&mx, 0, sizeof mx);
  // order of the dimensions (see tile_load): dims / strides / box / element strides of channel, W, image, H, depth
  const int mode = p.TI == 1 ? 0 : p.TN == 1 ? 1 : 2;
  auto tile_map = [&](CUtensorMap *m, const void *ptr, cuuint64_t C_, cuuint64_t W_, cuuint64_t H_, cuuint64_t D_, cuuint64_t sw_, cuuint64_t sh_,
                      cuuint64_t sd_, cuuint64_t sn_, cuuint32_t bc, cuuint32_t bw, cuuint32_t bn, cuuint32_t bh, cuuint32_t ew, cuuint32_t eh,
                      CUtensorMapSwizzle sw) -> bool {     // byte strides of W, H, depth and image
    const cuuint64_t N_ = (cuuint64_t)d.N, TI_ = (cuuint64_t)p.TI;
    cuuint64_t dims[5], st[4];
    cuuint32_t box[5], es[5] = {1u, 1u, 1u, 1u, 1u};
    dims[0] = C_; box[0] = bc;
    if (mode == 0) {
      dims[1] = W_; dims[2] = N_; dims[3] = H_; dims[4] = D_;
      st[0] = sw_; st[1] = sn_; st[2] = sh_; st[3] = sd_;
      box[1] = bw; box[2] = bn; box[3] = bh; box[4] = 1u; es[1] = ew; es[3] = eh;
    } else if (mode == 1) {
      dims[1] = N_; dims[2] = W_; dims[3] = H_; dims[4] = D_;
      st[0] = sn_; st[1] = sw_; st[2] = sh_; st[3] = sd_;
      box[1] = (cuuint32_t)p.TI; box[2] = bw; box[3] = bh; box[4] = 1u; es[2] = ew; es[3] = eh;
    } else {
      dims[1] = TI_; dims[2] = W_; dims[3] = N_ / TI_; dims[4] = H_;
      st[0] = sn_; st[1] = sw_; st[2] = sn_ * TI_; st[3] = sh_;
      box[1] = (cuuint32_t)p.TI; box[2] = bw; box[3] = bn; box[4] = bh; es[2] = ew; es[4] = eh;
    }
    return enc(m, dt, 5, const_cast<void *>(ptr), dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  const cuuint64_t xw = (cuuint64_t)d.C * esz, xh = xw * d.W, xd = xh * d.H, xn = xd * d.D;
  if (!d.fold && !tile_map(&mx, x, d.C, d.W, d.H, d.D, xw, xh, xd, xn, p.ch_el, p.PW * d.sW, p.TN, p.slab_rows_h * d.sH, d.sW, d.sH, swz)) {
    *detail = "cuTensorMapEncodeTiled failed for the input";
    return cudaErrorInvalidValue;
  }
  {   // filter tiles [tap][K][C] (fp32: two per tap)
    const cuuint64_t row = d.fold ? (cuuint64_t)p.ch_el : (cuuint64_t)d.C;
    const cuuint64_t dims[3] = {row, (cuuint64_t)d.K, (cuuint64_t)d.kD * p.n_taps * (f32 ? 2 : 1)};
    const cuuint64_t st[2] = {row * esz, row * esz * d.K};
    const cuuint32_t box[3] = {(cuuint32_t)p.ch_el, (cuuint32_t)(p.pair ? p.BN / 2 : p.BN), 1u};
    const cuuint32_t es[3] = {1u, 1u, 1u};
    if (enc(&mu, dt, 3, const_cast<void *>(u), dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) { *detail = "cuTensorMapEncodeTiled failed for the filter"; return cudaErrorInvalidValue; }
  }
  const int n_var = d.variants ? d.n_parts : 1;
  const bool y_tma = ((cuuint64_t)d.K * esz) % 16 == 0;
  if (y_tma) {   // one epilogue warp's 32 pixels (8 when pooled) x 128 bytes of channels
    const cuuint32_t sn = (cuuint32_t)std::min(p.TN, 4), sh = 4u / sn, w_px = (cuuint32_t)(8 / p.TI);
    for (int v = 0; v < n_var; ++v) {
      const DirectPart &a = d.parts[v];
      const int yw = d.variants ? a.oW : d.yW, yh = d.variants ? a.oH : d.yH;
      if (!tile_map(&my.m[v], (uint8_t *)y + (d.variants ? a.y_off : 0) * (long long)esz, d.K, yw, yh, d.oD, d.ys_w * esz, d.ys_h * esz, d.ys_d * esz, d.ys_n * esz,
                    (cuuint32_t)(128 / esz), pool ? w_px / 2 : w_px, sn, pool ? sh / 2 : sh, 1u, 1u, CU_TENSOR_MAP_SWIZZLE_128B)) {
        *detail = "cuTensorMapEncodeTiled failed for the output";
        return cudaErrorInvalidValue;
      }
    }
  } else my.m[0] = mx;
  DGeom g;
  std::memset(&g, 0, sizeof g);
  g.N = d.N; g.K = d.K; g.oD = d.oD; g.oH = d.oH;
  g.sD = d.sD; g.sH = d.sH; g.sW = d.sW; g.pD = d.pD; g.kD = d.kD;
  g.ys_n = d.ys_n; g.ys_d = d.ys_d; g.ys_h = d.ys_h; g.ys_w = d.ys_w;
  for (int v = 0; v < n_var; ++v) {
    g.yH[v] = d.variants ? d.parts[v].oH : d.yH; g.yW[v] = d.variants ? d.parts[v].oW : d.yW;
    g.y_off[v] = d.variants ? d.parts[v].y_off : 0;
  }
  g.TN = p.TN; g.TH = p.TH; g.TI = p.TI; g.PW = p.PW; g.map_mode = mode;
  while ((1 << g.tn_shift) < p.TN) ++g.tn_shift;
  while ((1 << g.ti_shift) < p.TI) ++g.ti_shift;
  g.n_wb = p.n_wb; g.n_hb = p.n_hb; g.n_tiles = p.n_tiles; g.n_kb = p.n_kb; g.var_items = p.n_items; g.n_items = p.n_items * n_var;
  g.n_ph = d.n_parts; g.n_var = n_var; g.T_hw = p.n_taps;
  for (int q = 0; q < d.n_parts; ++q) {
    g.org_h[q] = d.parts[q].org_h; g.org_w[q] = d.parts[q].org_w; g.taps[q] = p.taps[q]; g.tap0[q] = p.tap0[q];
    for (int t = 0; t < p.taps[q]; ++t) {
      const int th = t / d.parts[q].tw, tw = t - th * d.parts[q].tw;
      g.tap_off[p.tap0[q] + t] = (uint16_t)((th * p.TN * p.PW + tw) * p.TI * (p.rb / 16));
    }
  }
  if (d.fold) {
    const long long C = d.Cw, plane = (long long)d.H * d.W;
    g.raw_tma = p.raw_tma; g.raw_rem = p.raw_rem; g.raw_row = p.raw_el;
    g.raw_w = d.x_first ? 1 : d.Cw; g.raw_c = d.x_first ? p.slab_rows_h * p.raw_el : 1;
    if (p.raw_tma) {
      cuuint64_t dims[5], st[4];
      cuuint32_t box[5] = {(cuuint32_t)p.raw_el, (cuuint32_t)p.slab_rows_h, 1u, 1u, 1u};
      const cuuint32_t es[5] = {1u, 1u, 1u, 1u, 1u};
      const cuuint64_t row = d.x_first ? (cuuint64_t)d.W : (cuuint64_t)d.W * d.Cw;
      dims[0] = row; dims[1] = (cuuint64_t)d.H; dims[2] = (cuuint64_t)d.D;
      st[0] = row * 2; st[1] = st[0] * d.H; st[2] = st[1] * d.D;
      if (d.x_first) {
        dims[3] = (cuuint64_t)d.Cw; dims[4] = (cuuint64_t)d.N; st[3] = st[2] * d.Cw;
        box[3] = (cuuint32_t)d.Cw;
      } else {
        dims[3] = (cuuint64_t)d.N; dims[4] = 1; st[3] = st[2] * d.N;
      }
      if (enc(&mx, dt, 5, const_cast<void *>(x), dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        *detail = "cuTensorMapEncodeTiled failed for the few-channel input";
        return cudaErrorInvalidValue;
      }
    }
    if (d.x_first) { g.fx_c = (int)(plane * d.D); g.fx_w = 1; g.fx_h = d.W; g.fx_d = plane; g.fx_n = C * plane * d.D; }
    else { g.fx_c = 1; g.fx_w = (int)C; g.fx_h = C * d.W; g.fx_d = C * plane; g.fx_n = C * plane * d.D; }
    g.fD = d.D; g.fH = d.H; g.fW = d.W; g.fC = d.Cw; g.fkW = d.kW_w; g.fold_rows = p.slab_rows_h;
  }
  g.n_chunks = p.n_chunks; g.ch_el = p.ch_el; g.k_full = p.k_full; g.k_tail = p.k_tail; g.units = p.units;
  g.G = p.G; g.split = p.split; g.epilogue = d.epilogue;
  g.y_tma = y_tma; g.bias_f32 = d.bias_f32; g.bias_vec = y_tma && (reinterpret_cast<uintptr_t>(bias) & 15u) == 0;
  const int row_step = d.fold ? d.sH : 1;      // slab rows between neighbouring output rows
  g.a_hi = desc_hi((uint32_t)(row_step * p.PW * p.TI * p.rb), swz_code);
  g.b_hi = desc_hi((uint32_t)(8 * p.rb), swz_code);
  g.mb_off16 = row_step * p.TH * p.TN * p.PW * p.TI * p.rb / 16;
  DSmem sl;
  sl.slab_bytes = p.slab_bytes; sl.a_bytes = p.a_bytes; sl.lo_off = p.lo_off;
  sl.b_tile = p.b_tile; sl.b_lo = p.b_lo; sl.b_bytes = p.b_bytes; sl.n_a = p.n_a; sl.n_b = p.n_b;
  sl.off_b = p.n_a * p.a_bytes; sl.off_stage = sl.off_b + p.n_b * p.b_bytes;
  sl.off_raw = sl.off_stage + p.epi_sets * EPI_WARPS * STAGE_BYTES;
  sl.raw_bytes = (p.raw_box + 127) / 128 * 128;
  if (d.fold) sl.slab_bytes = p.raw_box;       // what TMA delivers
  sl.off_bars = sl.off_raw + (int)RAW_BUFS * sl.raw_bytes;
  const int sms = sm_count_of_current_device();
  if (sms <= 0) { *detail = "no device"; return cudaErrorNoDevice; }
  const uint32_t fmt = f32 ? 2u : d.dtype == WINOCONV_F16 ? 0u : 1u;
  const uint32_t m_rows = p.pair ? 2u * BM : (uint32_t)BM;
  const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.BN >> 3) << 17) | ((m_rows >> 4) << 24);
#define WINO_GO(T, BN_, MB_, P_)                                                                                              \
  return p.epi_sets == 2 ? launch_one<T, BN_, MB_, P_, false, 2>(p, mx, mu, my, x, y, bias, g, sl, idesc, sms, s)              \
                         : launch_one<T, BN_, MB_, P_>(p, mx, mu, my, x, y, bias, g, sl, idesc, sms, s)
#define WINO_FOLD(T, MB_) return launch_one<T, 64, MB_, false, true>(p, mx, mu, my, x, y, bias, g, sl, idesc, sms, s)
#define WINO_PICK(T)                                                             \
  do {                                                                           \
    if (d.fold) { if (p.MB == 2) WINO_FOLD(T, 2); WINO_FOLD(T, 1); }             \
    if (p.pair) {                                                                \
      if (p.BN == 256) WINO_GO(T, 256, 1, true);                                 \
      if (p.BN == 128) { if (p.MB == 2) WINO_GO(T, 128, 2, true); WINO_GO(T, 128, 1, true); } \
      WINO_GO(T, 64, 2, true);                                                   \
    }                                                                            \
    if (p.BN == 128) WINO_GO(T, 128, 1, false);                                  \
    if (p.MB == 2) WINO_GO(T, 64, 2, false);                                     \
    WINO_GO(T, 64, 1, false);                                                    \
  } while (0)
  if (d.dtype == WINOCONV_F16) WINO_PICK(__half);
  if (d.dtype == WINOCONV_BF16) WINO_PICK(__nv_bfloat16);
  return launch_one<float, 64, 1, false>(p, mx, mu, my, x, y, bias, g, sl, idesc, sms, s);
#undef WINO_PICK
#undef WINO_FOLD
#undef WINO_GO
}

cudaError_t read_and_clear_direct_error(cudaStream_t s, unsigned int *code) {
  unsigned int host = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbolAsync(&host, g_direct_error, sizeof(host), 0, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(g_direct_error, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  *code = host;
  return e;
}

}  // namespace wino
