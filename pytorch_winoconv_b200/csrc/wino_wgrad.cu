// Weight gradient of a convolution on the tensor cores (sm_100a), 16-bit activations, fp32 accumulate:
//
//     dW[k][t][c] = sum over images and output pixels of gy[n, o, k] * x[n, s * o + t - p, c]
//
// The reduction runs over pixels, which both operands have as their slow dimension: a block of 128 output pixels (16 groups
// of 8, as in the direct-tap forward) of gy [pixels][64 channels] and the slab of x that its taps touch are exactly what an
// MN-major operand with the 128-byte swizzle looks like, so neither tensor is transposed or copied.  The operand of a tap is
// the slab read from that tap's first pixel on; its M = 128 rows are 2 x 64, 4 x 32 or 8 x 16 (tap, channel) pairs, because
// the blocks of an MN-major operand may lie any distance apart -- one tap's distance here.  One slab thus serves all taps and
// a 64-channel layer still fills the instruction.
//
// A CTA keeps one accumulator of 128 (tap, channel) rows x N output channels per bundle of taps in tensor memory (at most 512
// columns) and walks its share of the pixel blocks; shares are added up by a second kernel that also puts the result into
// the weight's own order.  What bounds it: the shares.  Their number times dW is written and read once, 148 CTAs x up to
// 256 KB, so small layers use fewer, longer shares (see wgrad_plan).
//
// The bias gradient rides along: warps 4-7 add up the gy tiles as they lie in shared memory, in fp32 and in short chains (as
// one more accumulator, against an operand of ones, the tensor core's cut-off sums had twice the error of an fp32 sum).
//
// Roles: warp 0 TMA (x slabs), warp 1 TMA (gy tiles), warps 2-3 MMA issue (alternate bundles), warps 4-7 bias sums; then all eight warps move the
// accumulators to global memory, laid out so that a warp's store is 128 consecutive bytes: [share][channel block][bundle][k][row].
// Every mbarrier wait is bounded and reports through the error word.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>

#include "wino_launch.h"
#include "wino_sm100.cuh"

namespace wino {

__device__ unsigned int g_wgrad_error = 0;

namespace wgrad {

using namespace sm100;

constexpr int N_THREADS = 256;
constexpr int MAX_BUNDLES = 80, MAX_STEPS = 40, MAX_GROUPS = 24;
constexpr int SUMS_BYTES = 4 * 128 * 4;       // bias sums of four warps
constexpr int BAR_BYTES = 256;

enum ErrCode : unsigned { ERR_X_EMPTY = 0x501, ERR_G_EMPTY = 0x502, ERR_X = 0x503, ERR_G = 0x504, ERR_EPI = 0x505 };

// A slab of x (depth tap, polyphase part) and the bundles of taps that read it.
struct Step { int8_t kd, ph_h, ph_w, pad; int16_t b0, b1; };
struct Bundle { uint16_t off, lead, tap, n_taps; };   // first pixel and distance of its taps (16-byte units), first tap and how many

struct WGeom {
  int oD, oH, oW, sD, sH, sW, pD, pH, pW;
  int TN, TI, ti_shift, TH, PW, map_mode;
  int n_wb, n_hb, n_blocks, split;       // pixel blocks, shares
  int n_groups, n_kb, n_cb;
  int g_step0[MAX_GROUPS + 1], g_b0[MAX_GROUPS + 1];   // bundle groups: first step and first bundle of each (one past the last at the end)
  int N_mma, n_k;                        // columns of an MMA, output channels of a CTA
  int ch_el;
  int K, C, taps, all_bundles;           // real extents of dW
  uint32_t a_hi, b_hi, b_lead, b_tile;   // descriptor words; distance of gy's 64-channel blocks (16-byte units), bytes of one
  int n_gblk;                            // 64-channel blocks of a gy tile
  int bias_on;
  int slab_bytes, x_bytes, g_bytes, n_x, n_g, off_g, off_sums, off_bars;
  long long part_stride, bias_off;       // floats of one share, offset of the bias sums in it
  Step steps[MAX_STEPS];
  Bundle bundles[MAX_BUNDLES];
};

struct Block { int n0, od, oh0, ow0; };
__device__ __forceinline__ Block decode(const WGeom &g, unsigned b) {
  Block t;
  unsigned q = b / (unsigned)g.n_wb;
  t.ow0 = (int)(b - q * (unsigned)g.n_wb) * (8 >> g.ti_shift);
  unsigned r = q / (unsigned)g.n_hb;
  t.oh0 = (int)(q - r * (unsigned)g.n_hb) * g.TH;
  q = r / (unsigned)g.oD;
  t.od = (int)(r - q * (unsigned)g.oD);
  t.n0 = (int)q * (g.TN * g.TI);
  return t;
}
__device__ __forceinline__ void tile_load(const WGeom &g, uint32_t dst, const CUtensorMap *map, uint32_t bar, int c, int w, int n, int h, int d) {
  const int c1 = g.map_mode == 0 ? w : g.map_mode == 1 ? n : 0, c2 = g.map_mode == 0 ? n : w;
  const int c3 = g.map_mode == 2 ? n >> g.ti_shift : h, c4 = g.map_mode == 2 ? h : d;
  tma_load_5d(dst, map, bar, c, c1, c2, c3, c4);
}

__global__ void __launch_bounds__(N_THREADS, 1)
    wgrad_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_g, float *__restrict__ part,
                 int bf16, const __grid_constant__ WGeom g, uint32_t idesc) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw);
  const uint32_t bars = base + g.off_bars;      // x_full[4] x_empty[4] g_full[4] g_empty[4] done
  auto x_full = [&](int i) { return bars + 8u * i; };
  auto x_empty = [&](int i) { return bars + 32u + 8u * i; };
  auto g_full = [&](int i) { return bars + 64u + 8u * i; };
  auto g_empty = [&](int i) { return bars + 96u + 8u * i; };
  const uint32_t done = bars + 128u, tmem_slot = bars + 196u;
  volatile unsigned *abort_word = reinterpret_cast<volatile unsigned *>(base_ptr + g.off_bars + 192);
  unsigned *err = &g_wgrad_error;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  // this CTA: share, bundle group, channel blocks
  unsigned q = blockIdx.x / (unsigned)g.n_kb;
  const int kb = (int)(blockIdx.x - q * (unsigned)g.n_kb);
  unsigned r = q / (unsigned)g.n_cb;
  const int cb = (int)(q - r * (unsigned)g.n_cb);
  q = r / (unsigned)g.n_groups;
  const int grp = (int)(r - q * (unsigned)g.n_groups);
  const int share = (int)q;
  const int blk0 = (int)((long long)g.n_blocks * share / g.split), blk1 = (int)((long long)g.n_blocks * (share + 1) / g.split);
  const int gb0 = g.g_b0[grp], gb1 = g.g_b0[grp + 1];            // bundles of the group
  const bool bias = g.bias_on && cb == 0 && grp == 0;

  if (warp == 1 && lane == 0) { prefetch_map(&map_x); prefetch_map(&map_g); }
  if (warp == 0) {
    if (lane < 4) { mbar_init(x_full(lane), 1); mbar_init(x_empty(lane), 2); }
    else if (lane < 8) { mbar_init(g_full(lane - 4), 1); mbar_init(g_empty(lane - 4), bias ? 6 : 2); }
    else if (lane == 8) mbar_init(done, 2);
    else if (lane == 9) *abort_word = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) tmem_alloc<false>(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
  tmem = __shfl_sync(0xffffffffu, tmem, 0);
  grid_launch_dependents();
  grid_dependency_wait();

  const int st0 = g.g_step0[grp];
  bool alive = true;

  // steps of the group: from st0 while their bundles overlap [gb0, gb1)
  auto for_steps = [&](auto &&body) -> bool {
    for (int s = st0; s < MAX_STEPS; ++s) {
      const int b0 = max((int)g.steps[s].b0, gb0), b1 = min((int)g.steps[s].b1, gb1);
      if (b0 >= b1) break;
      if (!body(s, b0, b1)) return false;
    }
    return true;
  };

  if (warp == 0) {
    int s = 0;
    uint32_t ph = 1;
    for (int b = blk0; b < blk1 && alive; ++b) {
      const Block t = decode(g, (unsigned)b);
      alive = for_steps([&](int st, int, int) -> bool {
        if (!mbar_wait_warp(x_empty(s), ph, abort_word, err, ERR_X_EMPTY)) return false;
        if (lane == 0) {
          mbar_expect_tx(x_full(s), (uint32_t)g.slab_bytes);
          tile_load(g, base + (uint32_t)(s * g.x_bytes), &map_x, x_full(s), cb * g.ch_el, g.sW * t.ow0 + g.steps[st].ph_w - g.pW, t.n0,
                    g.sH * t.oh0 + g.steps[st].ph_h - g.pH, g.sD * t.od + g.steps[st].kd - g.pD);
        }
        if (++s == g.n_x) { s = 0; ph ^= 1u; }
        return true;
      });
    }
    if (*abort_word != 0u) {   // loads in flight must land before the shared memory goes away
      const long long start = clock64();
      while (clock64() - start < 2000000LL) { }
    }
  } else if (warp == 1) {
    int s = 0;
    uint32_t ph = 1;
    for (int b = blk0; b < blk1; ++b) {
      const Block t = decode(g, (unsigned)b);
      if (!mbar_wait_warp(g_empty(s), ph, abort_word, err, ERR_G_EMPTY)) break;
      if (lane == 0) {
        mbar_expect_tx(g_full(s), (uint32_t)(g.n_gblk * (int)g.b_tile));
        for (int j = 0; j < g.n_gblk; ++j)
          tile_load(g, base + (uint32_t)(g.off_g + s * g.g_bytes) + (uint32_t)j * g.b_tile, &map_g, g_full(s), kb * g.n_k + j * 64, t.ow0, t.n0, t.oh0, t.od);
      }
      if (++s == g.n_g) { s = 0; ph ^= 1u; }
    }
    if (*abort_word != 0u) {
      const long long start = clock64();
      while (clock64() - start < 2000000LL) { }
    }
  } else if (warp < 4) {
    const int me = warp - 2;
    int xs = 0, gs = 0;
    uint32_t x_ph = 0, g_ph = 0, acc = 0;
    const uint32_t x_pair = 2u * (g.a_hi & 0x3FFFu), g_pair = 128u;      // two groups of 8 pixels further on (16-byte units)
    for (int b = blk0; b < blk1 && alive; ++b) {
      if (!mbar_wait_warp(g_full(gs), g_ph, abort_word, err, ERR_G)) { alive = false; break; }
      tc_fence_after();
      const uint32_t b_lo = (((base + (uint32_t)(g.off_g + gs * g.g_bytes)) & 0x3FFFFu) >> 4) | (g.b_lead << 16);
      alive = for_steps([&](int st, int b0, int b1) -> bool {
        (void)st;
        if (!mbar_wait_warp(x_full(xs), x_ph, abort_word, err, ERR_X)) return false;
        tc_fence_after();
        const uint32_t x_lo = ((base + (uint32_t)(xs * g.x_bytes)) & 0x3FFFFu) >> 4;
        if (elect_one()) {
          for (int i = b0 + ((b0 ^ me) & 1); i < b1; i += 2) {
            const uint32_t a = (x_lo + g.bundles[i].off) | ((uint32_t)g.bundles[i].lead << 16), d = tmem + (uint32_t)((i - gb0) * g.N_mma);
#pragma unroll
            for (int k = 0; k < 8; ++k) umma<false, false>(d, a + (uint32_t)k * x_pair, g.a_hi, b_lo + (uint32_t)k * g_pair, g.b_hi, idesc, k == 0 ? acc : 1u);
          }
          umma_commit<false>(x_empty(xs), 0);
        }
        __syncwarp();
        if (++xs == g.n_x) { xs = 0; x_ph ^= 1u; }
        return true;
      });
      if (elect_one()) umma_commit<false>(g_empty(gs), 0);
      if (++gs == g.n_g) { gs = 0; g_ph ^= 1u; }
      acc = 1u;
    }
    if (elect_one()) umma_commit<false>(done, 0);
  } else if (bias) {
    // a warp takes 32 pixels of every tile, a lane two neighbouring channels of each 64-channel block
    int gs = 0;
    uint32_t g_ph = 0;
    float total[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    for (int b = blk0; b < blk1; ++b) {
      if (!mbar_wait_warp(g_full(gs), g_ph, abort_word, err, ERR_G)) break;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (j >= g.n_gblk) break;
        const uint8_t *tile = base_ptr + g.off_g + gs * g.g_bytes + j * (int)g.b_tile + (warp - 4) * 4096 + (lane & 3) * 4;
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t v = *reinterpret_cast<const uint32_t *>(tile + i * 128 + (((lane >> 2) ^ (i & 7)) << 4));
          const float2 f = bf16 ? Pair16<__nv_bfloat16>::unpack(v) : Pair16<__half>::unpack(v);
          a[2 * (i & 3)] += f.x;
          a[2 * (i & 3) + 1] += f.y;
        }
        total[j][0] += (a[0] + a[2]) + (a[4] + a[6]);
        total[j][1] += (a[1] + a[3]) + (a[5] + a[7]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(g_empty(gs));
      if (++gs == g.n_g) { gs = 0; g_ph ^= 1u; }
    }
    float *sums = reinterpret_cast<float *>(base_ptr + g.off_sums);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      sums[(warp - 4) * 128 + j * 64 + 2 * lane] = total[j][0];
      sums[(warp - 4) * 128 + j * 64 + 2 * lane + 1] = total[j][1];
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const int c = threadIdx.x - 128, k = kb * g.n_k + c;
    if (c < g.n_k && k < g.K) part[(long long)share * g.part_stride + g.bias_off + k] = (sums[c] + sums[128 + c]) + (sums[256 + c] + sums[384 + c]);
  }
  __syncwarp();
  if (mbar_wait_warp(done, 0, abort_word, err, ERR_EPI) && *abort_word == 0u) {
    tc_fence_after();
    const int qd = warp & 3, half = warp >> 2;
    const uint32_t t_row = tmem + ((uint32_t)(qd * 32) << 16);
    const int n_b = gb1 - gb0, n_ch = (g.N_mma + 31) / 32;
    for (int i = half; i < n_b * n_ch; i += 2) {
      const int bu = i / n_ch, k0 = (i - bu * n_ch) * 32;
      uint32_t v[32];
      tmem_ld_x32(t_row + (uint32_t)(bu * g.N_mma + k0), v);
      tmem_wait_ld_x32(v);
      const int k = kb * g.n_k + k0;
      float *dst = part + (long long)share * g.part_stride + (((long long)cb * g.all_bundles + gb0 + bu) * g.K + k) * 128 + qd * 32 + lane;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (k + j < g.K) dst[j * 128] = __uint_as_float(v[j]);
    }
    tc_fence_before();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_free<false>(tmem, 512);
  }
}

// dW[(k * C + c) * taps + t] = sum over shares of part[share][channel block][bundle][k][row]; the last threads add up the bias
// sums.  One thread per value: reads are 512-byte runs with eight shares in flight per thread, and as many threads as values
// keep the L2 busy (a block per run of outputs, turned in shared memory, took 10 us where this takes 3 for 18 MB of shares); the
// writes, a value every taps x 4 bytes, are a few per cent of the traffic.
struct RGeom {
  int K, C, taps, split, n_bundles, ch_el;
  long long part_stride, bias_off;
  Bundle bundles[MAX_BUNDLES];
  uint16_t tap_of[400];         // position in the weight of each walked tap
  // what pixel_sum reads
  int bf16, N, D, H, W, oD, oH, oW, sD, sH, sW, pD, pH, pW, kH, kW, Cm, Km;
};

// A block that reaches beyond the output multiplies zeros of gy by pixels of x which another tap has a use for.  Where such a pixel
// is infinite or not a number, so is the sum: a sum that is not a number is done again over the output's own pixels.  It ends
// where it has become one by rights.  Layers without such blocks run the kernel without this code; in it, it costs the others about 5 %
// of their time (128 -> 128 3x3 at 57x57, N = 32: 41.1 -> 43.1 us with the first kernel's; 32 registers as before).  One infinite pixel
// at the edge costs 64 -> 64 at 114x114, N = 64, 0.37 s.
__device__ __forceinline__ float pixel_sum(const unsigned short *__restrict__ x, const unsigned short *__restrict__ gy, const RGeom &g, int k, int c, int tap) {
  const int tw = tap % g.kW, th = tap / g.kW % g.kH, td = tap / (g.kW * g.kH);
  auto value = [&](unsigned short v) { return g.bf16 ? __uint_as_float((uint32_t)v << 16) : Pair16<__half>::unpack(v).x; };
  float total = 0.f;
  for (int n = 0; n < g.N; ++n)
    for (int od = 0; od < g.oD; ++od)
      for (int oh = 0; oh < g.oH; ++oh) {
        const int id = g.sD * od + td - g.pD, ih = g.sH * oh + th - g.pH;
        const bool row_in = (unsigned)id < (unsigned)g.D && (unsigned)ih < (unsigned)g.H;
        const unsigned short *gr = gy + (((long long)n * g.oD + od) * g.oH + oh) * g.oW * g.Km + k;
        const unsigned short *xr = x + (((long long)n * g.D + id) * g.H + ih) * g.W * g.Cm + c;
        float row = 0.f;
        for (int o0 = 0; o0 < g.oW; o0 += 8) {      // eight pixels' loads in flight: a thread has nothing else to wait with
          unsigned short a[8], b[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int ow = o0 + i, iw = g.sW * ow + tw - g.pW;
            a[i] = ow < g.oW ? gr[(long long)ow * g.Km] : 0;
            b[i] = ow < g.oW && row_in && (unsigned)iw < (unsigned)g.W ? xr[(long long)iw * g.Cm] : 0;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) row = fmaf(value(a[i]), value(b[i]), row);
        }
        total += row;
        if (total != total) return total;
      }
  return total;
}
template <typename T, bool REDO>
__global__ void __launch_bounds__(256, 8) wgrad_reduce_kernel(const float *__restrict__ part, T *__restrict__ dw, float *__restrict__ dbias,
                                                           const unsigned short *__restrict__ x, const unsigned short *__restrict__ gy,
                                                           const __grid_constant__ RGeom g, int n_values) {
  grid_dependency_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n_values) return;
  const bool is_bias = i >= (int)g.bias_off;
  const int row = i & 127, k = (i >> 7) % g.K, cbb = (i >> 7) / g.K, cb = cbb / g.n_bundles, bu = cbb - cb * g.n_bundles;
  const int tl = row / g.ch_el, c = cb * g.ch_el + row - tl * g.ch_el;      // tap within the bundle, channel
  if (!is_bias && (c >= g.C || tl >= g.bundles[bu].n_taps)) return;
  float s = 0.f;
  const float *src = part + i;
  int j = 0;
  for (; j + 8 <= g.split; j += 8) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = src[(j + e) * g.part_stride];
    s += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  for (; j < g.split; ++j) s += src[j * g.part_stride];
  if (is_bias) { dbias[i - (int)g.bias_off] = s; return; }
  const int tap = g.tap_of[g.bundles[bu].tap + tl];
  if constexpr (REDO) { if (s != s) s = pixel_sum(x, gy, g, k, c, tap); }
  Elem<T>::store(dw + ((long long)k * g.C + c) * g.taps + tap, s);
}

}  // namespace wgrad

using namespace wgrad;

bool wgrad_plan(const WgradDesc &d, WgradPlan *out) {
  static_assert(sizeof(WGeom) <= sizeof(out->geom), "plan blob too small");
  if (d.dtype == WINOCONV_F32 || d.Cm % 8 != 0 || d.Km % 8 != 0) return false;
  if (d.sH > 2 || d.sW > 2 || d.sD > 2 || d.pH > 64 || d.pW > 64) return false;
  const int n_taps = d.kD * d.kH * d.kW;
  if (n_taps > 400) return false;      // the reducing kernel's table
  WGeom g0;
  std::memset(&g0, 0, sizeof g0);
  g0.oD = d.oD; g0.oH = d.oH; g0.oW = d.oW; g0.sD = d.sD; g0.sH = d.sH; g0.sW = d.sW; g0.pD = d.pD; g0.pH = d.pH; g0.pW = d.pW;
  g0.K = d.K; g0.C = d.C; g0.taps = n_taps; g0.bias_on = d.bias;
  // channels of a slab row: 64, or 32 / 16 where they hold all channels (then 4 / 8 taps fill the 128 rows of an MMA)
  g0.ch_el = d.Cm > 32 ? 64 : d.Cm > 16 ? 32 : 16;
  const int rb = g0.ch_el * 2, per_bundle = 128 / g0.ch_el;
  g0.n_cb = (d.Cm + g0.ch_el - 1) / g0.ch_el;
  const int Th = (d.kH + d.sH - 1) / d.sH, Tw = (d.kW + d.sW - 1) / d.sW;
  double best = 1e30;
  bool found = false;
  for (int ti = 1; ti <= 8; ti *= 2)
    for (int tn = 1; tn <= 16; tn *= 2) {
      if (ti * tn > 1 && ti * tn / 2 >= d.N) continue;
      if (ti > 1 && tn > 1 && (d.D != 1 || d.kD != 1 || d.pD != 0 || d.N % ti != 0)) continue;
      WGeom g = g0;
      g.TI = ti; g.TN = tn; g.TH = 16 / tn; g.PW = 8 / ti + Tw - 1;
      while ((1 << g.ti_shift) < ti) ++g.ti_shift;
      g.map_mode = ti == 1 ? 0 : tn == 1 ? 1 : 2;
      const int rows_h = g.TH + Th - 1;
      if (g.PW * d.sW > 256 || rows_h * d.sH > 256) continue;
      g.slab_bytes = rows_h * tn * g.PW * ti * rb;
      g.x_bytes = (g.slab_bytes + 1023) / 1024 * 1024;
      g.n_wb = (d.oW + 8 / ti - 1) / (8 / ti); g.n_hb = (d.oH + g.TH - 1) / g.TH;
      const long long blocks = (long long)g.n_wb * g.n_hb * d.oD * ((d.N + tn * ti - 1) / (tn * ti));
      if (blocks > 0x3fffffffLL) continue;
      g.n_blocks = (int)blocks;
      // steps and their bundles of taps
      int n_steps = 0, n_b = 0;
      bool fits = true;
      for (int kd = 0; kd < d.kD && fits; ++kd)
        for (int a = 0; a < d.sH && fits; ++a)
          for (int b = 0; b < d.sW && fits; ++b) {
            const int th = (d.kH - a + d.sH - 1) / d.sH, tw = (d.kW - b + d.sW - 1) / d.sW;
            if (th <= 0 || tw <= 0) continue;
            if (n_steps == MAX_STEPS) { fits = false; break; }
            Step &st = g.steps[n_steps++];
            st.kd = (int8_t)kd; st.ph_h = (int8_t)a; st.ph_w = (int8_t)b; st.b0 = (int16_t)n_b;
            auto off = [&](int t) { return ((t / tw) * tn * g.PW + t % tw) * ti * (rb / 16); };
            int tap0 = 0;      // taps walked before this step
            if (n_steps > 1) tap0 = g.bundles[n_b - 1].tap + g.bundles[n_b - 1].n_taps;
            for (int t = 0; t < th * tw;) {
              if (n_b == MAX_BUNDLES) { fits = false; break; }
              Bundle &bu = g.bundles[n_b++];
              bu.off = (uint16_t)off(t);
              bu.tap = (uint16_t)(tap0 + t);
              // two taps may lie any distance apart; more must be neighbours along W
              int n = per_bundle == 2 ? std::min(2, th * tw - t) : std::min(per_bundle, tw - t % tw);
              bu.n_taps = (uint16_t)n;
              bu.lead = (uint16_t)(per_bundle == 2 ? (n == 2 ? off(t + 1) - off(t) : 0) : ti * (rb / 16));
              t += n;
            }
            st.b1 = (int16_t)n_b;
          }
      if (!fits) continue;
      g.all_bundles = n_b;
      if ((long long)g.n_cb * n_b * d.K * 128 > 0x7fffffffLL - d.K) continue;
      for (int n_k = 128; n_k >= 64; n_k -= 64) {
        if (n_k == 128 && d.Km <= 64) continue;
        WGeom q = g;
        q.n_k = n_k;
        q.n_kb = (d.Km + n_k - 1) / n_k;
        q.N_mma = q.n_kb > 1 ? n_k : (d.Km + 15) / 16 * 16;
        q.n_gblk = (std::min(n_k, d.Km) + 63) / 64;
        q.b_tile = 16384; q.b_lead = 16384 >> 4;
        q.g_bytes = q.n_gblk * 16384;
        const int cap = (q.N_mma % 32 == 0 ? 512 : 496) / q.N_mma;
        if (cap < 2) continue;
        q.n_groups = (n_b + cap - 1) / cap;
        if (q.n_groups > MAX_GROUPS) continue;
        int widest = 0, most_steps = 0;
        for (int i = 0; i <= q.n_groups; ++i) q.g_b0[i] = (int)((long long)n_b * i / q.n_groups);
        for (int i = 0; i < q.n_groups; ++i) {
          widest = std::max(widest, q.g_b0[i + 1] - q.g_b0[i]);
          int s0 = 0, n = 0;
          while (g.steps[s0].b1 <= q.g_b0[i]) ++s0;
          q.g_step0[i] = s0;
          for (int s = s0; s < n_steps && g.steps[s].b0 < q.g_b0[i + 1]; ++s) ++n;
          most_steps = std::max(most_steps, n);
        }
        // rings: two gy tiles, then slabs, then more of both
        const int budget = 227 * 1024 - 1024 - SUMS_BYTES - BAR_BYTES - 1024;
        q.n_g = 2; q.n_x = 1;
        if (q.n_g * q.g_bytes + q.n_x * q.x_bytes > budget) continue;
        while (q.n_x < 4 && q.n_g * q.g_bytes + (q.n_x + 1) * q.x_bytes <= budget) ++q.n_x;
        while (q.n_g < 4 && (q.n_g + 1) * q.g_bytes + q.n_x * q.x_bytes <= budget) ++q.n_g;
        if (q.n_x < 2 && most_steps > 1) continue;
        const int combos = q.n_groups * q.n_kb * q.n_cb;
        const double t_mma = q.N_mma > 64 ? 66 : 50;
        const double bytes = (double)most_steps * q.slab_bytes + q.n_gblk * 16384.0;
        for (int split = 1; split <= q.n_blocks && split * combos <= 2 * 148; ++split) {
          const long long ctas = (long long)combos * split;
          const int waves = (int)((ctas + 147) / 148);
          if (waves > 1 && split > 1) break;
          const double active = std::min<double>(148.0, (double)ctas);
          const double block = std::max(widest * 8 * t_mma, std::max(bytes / std::min(60.0, 28.0 * 148 / active),
                                        (widest * 8 * (4096.0 + q.N_mma * 32.0) + bytes) / 128.0));
          const double reduce = (double)split * q.n_cb * n_b * d.K * 128 * 8.0 / 2400.0;
          const double e = 8000.0 + waves * (((q.n_blocks + split - 1) / split) * block + widest * q.N_mma * 8.0) + 6000.0 + reduce;
          if (e < best) {
            best = e; found = true;
            q.split = split;
            std::memcpy(out->geom, &q, sizeof q);
          }
        }
        if (combos > 296 && best == 1e30) {      // more CTAs than two waves even without shares
          q.split = 1; found = true; best = 1e29;
          std::memcpy(out->geom, &q, sizeof q);
        }
      }
    }
  if (!found) return false;
  WGeom &g = *reinterpret_cast<WGeom *>(out->geom);
  g.a_hi = desc_hi((uint32_t)(g.PW * g.TI * rb), rb == 128 ? 2u : rb == 64 ? 4u : 6u);
  g.b_hi = desc_hi(1024, 2);
  g.off_g = g.n_x * g.x_bytes;
  g.off_sums = g.off_g + g.n_g * g.g_bytes;
  g.off_bars = g.off_sums + SUMS_BYTES;
  g.bias_off = (long long)g.n_cb * g.all_bundles * d.K * 128;
  g.part_stride = (g.bias_off + d.K + 31) / 32 * 32;
  out->smem = 1024 + g.off_bars + BAR_BYTES;
  out->ws_bytes = (unsigned long long)g.split * g.part_stride * 4;
  out->slab_rows_h = g.TH + Th - 1;
  return true;
}

template <typename T>
static cudaError_t launch_reduce(const RGeom &r, bool redo, const float *part, void *dw, float *db, const void *x, const void *gy, int n, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((n + 255) / 256)); cfg.blockDim = dim3(256); cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  const auto *xs = (const unsigned short *)x, *gs = (const unsigned short *)gy;
  return redo ? cudaLaunchKernelEx(&cfg, wgrad_reduce_kernel<T, true>, part, (T *)dw, db, xs, gs, r, n)
              : cudaLaunchKernelEx(&cfg, wgrad_reduce_kernel<T, false>, part, (T *)dw, db, xs, gs, r, n);
}

cudaError_t launch_wgrad(const WgradDesc &d, const WgradPlan &p, const void *x, const void *gy, void *dw, int dw_dtype, float *dbias,
                         void *ws, cudaStream_t s, const char **detail) {
  *detail = "";
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) { *detail = "cuTensorMapEncodeTiled unavailable"; return cudaErrorNotSupported; }
  const WGeom &g = *reinterpret_cast<const WGeom *>(p.geom);
  const int rb = g.ch_el * 2;
  const CUtensorMapDataType dt = map_dtype(d.dtype);
  auto tile_map = [&](CUtensorMap *m, const void *ptr, cuuint64_t C_, cuuint64_t W_, cuuint64_t H_, cuuint64_t D_, cuuint32_t bc, cuuint32_t bw,
                      cuuint32_t bh, cuuint32_t ew, cuuint32_t eh, CUtensorMapSwizzle sw) -> bool {
    const cuuint64_t sw_ = C_ * 2, sh_ = sw_ * W_, sd_ = sh_ * H_, sn_ = sd_ * D_, N_ = (cuuint64_t)d.N, TI_ = (cuuint64_t)g.TI;
    cuuint64_t dims[5] = {C_, W_, N_, H_, D_}, st[4] = {sw_, sn_, sh_, sd_};
    cuuint32_t box[5] = {bc, bw, (cuuint32_t)g.TN, bh, 1u}, es[5] = {1u, ew, 1u, eh, 1u};
    if (g.map_mode == 1) {
      dims[1] = N_; dims[2] = W_; st[0] = sn_; st[1] = sw_;
      box[1] = (cuuint32_t)g.TI; box[2] = bw; es[1] = 1u; es[2] = ew;
    } else if (g.map_mode == 2) {
      dims[1] = TI_; dims[2] = W_; dims[3] = N_ / TI_; dims[4] = H_;
      st[0] = sn_; st[1] = sw_; st[2] = sn_ * TI_; st[3] = sh_;
      box[1] = (cuuint32_t)g.TI; box[2] = bw; box[3] = (cuuint32_t)g.TN; box[4] = bh; es[1] = 1u; es[2] = ew; es[3] = 1u; es[4] = eh;
    }
    return enc(m, dt, 5, const_cast<void *>(ptr), dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  CUtensorMap mx, mg;
  if (!tile_map(&mx, x, d.Cm, d.W, d.H, d.D, g.ch_el, g.PW * d.sW, p.slab_rows_h * d.sH, d.sW, d.sH,
                rb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : rb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B) ||
      !tile_map(&mg, gy, d.Km, d.oW, d.oH, d.oD, 64u, (cuuint32_t)(8 / g.TI), (cuuint32_t)g.TH, 1u, 1u, CU_TENSOR_MAP_SWIZZLE_128B)) {
    *detail = "cuTensorMapEncodeTiled failed";
    return cudaErrorInvalidValue;
  }
  {
    static std::mutex mu;
    static std::map<int, bool> set;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    if (!set[dev]) {
      e = cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      set[dev] = true;
    }
  }
  // A = B = f16 / bf16, both MN-major, D = f32, M = 128
  const uint32_t fmt = d.dtype == WINOCONV_F16 ? 0u : 1u;
  const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(g.N_mma >> 3) << 17) | ((128u >> 4) << 24);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(g.split * g.n_groups * g.n_cb * g.n_kb)); cfg.blockDim = dim3(N_THREADS);
  cfg.dynamicSmemBytes = (size_t)p.smem; cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, wgrad_kernel, mx, mg, (float *)ws, d.dtype == WINOCONV_BF16 ? 1 : 0, g, idesc);
  if (e != cudaSuccess) return e;
  RGeom r;
  std::memset(&r, 0, sizeof r);
  r.K = d.K; r.C = d.C; r.taps = g.taps; r.split = g.split; r.part_stride = g.part_stride; r.bias_off = g.bias_off;
  r.n_bundles = g.all_bundles; r.ch_el = g.ch_el;
  r.bf16 = d.dtype == WINOCONV_BF16;
  r.N = d.N; r.D = d.D; r.H = d.H; r.W = d.W; r.oD = d.oD; r.oH = d.oH; r.oW = d.oW; r.Cm = d.Cm; r.Km = d.Km;
  r.sD = d.sD; r.sH = d.sH; r.sW = d.sW; r.pD = d.pD; r.pH = d.pH; r.pW = d.pW; r.kH = d.kH; r.kW = d.kW;
  std::memcpy(r.bundles, g.bundles, sizeof r.bundles);
  int nt = 0;     // the order the kernel walks the taps in: depth tap, polyphase part, row, column
  for (int kd = 0; kd < d.kD; ++kd)
    for (int a = 0; a < d.sH; ++a)
      for (int b = 0; b < d.sW; ++b)
        for (int th = a; th < d.kH; th += d.sH)
          for (int tw = b; tw < d.kW; tw += d.sW) r.tap_of[nt++] = (uint16_t)((kd * d.kH + th) * d.kW + tw);
  const int n = (int)g.bias_off + (g.bias_on ? d.K : 0);
  const bool redo = g.n_wb * (8 / g.TI) != d.oW || g.n_hb * g.TH != d.oH;      // blocks that reach beyond the output
  if (dw_dtype == WINOCONV_F32) return launch_reduce<float>(r, redo, (const float *)ws, dw, dbias, x, gy, n, s);
  if (dw_dtype == WINOCONV_F16) return launch_reduce<__half>(r, redo, (const float *)ws, dw, dbias, x, gy, n, s);
  return launch_reduce<__nv_bfloat16>(r, redo, (const float *)ws, dw, dbias, x, gy, n, s);
}

cudaError_t read_and_clear_wgrad_error(cudaStream_t s, unsigned int *code) {
  unsigned int host = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbolAsync(&host, g_wgrad_error, sizeof(host), 0, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(g_wgrad_error, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  *code = host;
  return e;
}

}  // namespace wino
