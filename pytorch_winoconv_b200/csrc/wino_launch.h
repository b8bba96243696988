// Host-side launch functions shared between the translation units of libwinoconv_b200.
#pragma once

#include <cuda_runtime.h>

#include "wino_common.cuh"

namespace wino {

cudaError_t launch_filter_transform(const Geom &g, int dtype, const void *w, void *u, cudaStream_t s);
cudaError_t launch_input_transform(const Geom &g, int dtype, const void *x, void *v, long long t0, int n_tiles,
                                   cudaStream_t s);
cudaError_t launch_output_transform(const Geom &g, int dtype, int product_dtype, const void *m, void *y,
                                    const void *bias, long long t0, int n_tiles, cudaStream_t s);
cudaError_t launch_split(const float *x, float *out, int N, int D, int H, int W, int C, int bD, int bH, int bW,
                         int oD, int oH, int oW, int nD, int nH, int nW, cudaStream_t s);
cudaError_t launch_concat(const float *tiles, float *y, int N, int oD, int oH, int oW, int K, int mD, int mH, int mW,
                          cudaStream_t s);
// [N, C, P] -> [N, P, Cs] (zeros from channel C on) and [N, P, C] -> [N, C, P] (+ bias), converting the element type
cudaError_t launch_to_channels_last(int in_dtype, int out_dtype, const void *x, void *y, int N, int C, int P, int Cs, cudaStream_t s);
cudaError_t launch_to_channels_first(int in_dtype, int out_dtype, const void *x, void *y, const float *bias, int N, int C, int P, cudaStream_t s);
cudaError_t launch_add(const float *a, const float *b, float *c, long long n, cudaStream_t s);

// m[p][t][k] = sum_c v[p][t][c] u[p][k][c]; fp32 accumulate.
cudaError_t launch_gemm_simt(int dtype, int product_dtype, int positions, long long tiles, int c_pad, int k_out,
                             const void *v, const void *u, void *m, cudaStream_t s);
// tcgen05 / TMEM / TMA version (f16 / bf16).  `detail` receives a message on failure.
cudaError_t launch_gemm_tcgen05(int dtype, int product_dtype, int positions, long long tiles, int c_pad, int k_out,
                                const void *v, const void *u, void *m, cudaStream_t s, const char **detail);

// fp32 operands on the tensor cores (kind::tf32): split = 0 plain tf32 products, split = 1 three products of a
// hi / lo split made in shared memory (fp32-class accuracy).  m in fp32.
cudaError_t launch_gemm_tf32(int split, int positions, long long tiles, int c_pad, int k_out, const void *v,
                             const void *u, void *m, cudaStream_t s, const char **detail);

// F(4x4,3x3) input transform of a whole 16-bit layer with the raw patches staged through shared memory by TMA
// (channels a multiple of eight, one pass over all tiles); `applies` says whether a call qualifies.
bool input_f43_tma_applies(const Geom &g, int dtype, const void *x, long long t0, long long n_tiles);
cudaError_t launch_input_f43_tma(const Geom &g, int dtype, const void *x, void *v, cudaStream_t s, const char **detail);

// The matching output transform (output channels a multiple of eight, bias / ReLU epilogue, one pass over all tiles).
bool output_f43_tma_applies(const Geom &g, int dtype, int product_dtype, const void *m, long long t0, long long n_tiles);
cudaError_t launch_output_f43_tma(const Geom &g, int dtype, int product_dtype, const void *m, void *y, const void *bias,
                                  cudaStream_t s, const char **detail);

// Fused F(2x2,3x3) path (f16 / bf16): transformed filter u [16][K][R], then one kernel for the whole layer.
cudaError_t launch_fused_filter_transform(const FGeom &g, int dtype, const void *w, void *u, cudaStream_t s);
cudaError_t launch_fused_forward(const FGeom &g, int dtype, const void *x, const void *u, const void *bias, void *y,
                                 cudaStream_t s, const char **detail);
cudaError_t read_and_clear_fused_error(cudaStream_t s, unsigned int *code);

// x [pixels][C] -> xp [pixels][Cp], zeros from C on
cudaError_t launch_pad_channels(int dtype, const void *x, void *xp, long long pixels, int C, int Cp, cudaStream_t s);

// Row-piece DWM kernel (f16 / bf16, stride 1): 1 x 3 pieces, F(2,3) along W, taps along H / depth summed in TMEM.
struct RowDesc {
  int N, C, K, D, H, W, oD, oH, oW, yH, yW;
  int sD, sH, sW, pD, pH, pW, kD, kH, kW;
  unsigned epilogue;
  int weight_layout;
  // Stride 2 as a stride-1 problem (polyphase parts folded into the channels): when `phases` > 1 the fields above
  // describe the stride-1 convolution the kernel runs -- C = phases x C0 channels, kernel ceil(k0 / 2) per strided
  // dimension, no padding, input extent out + k - 1 -- and the fields below the tensor the caller passes in.
  int phases;                 // 1: plain stride-1 problem
  int fD, fH, fW;             // phase count per dimension (1 or 2)
  int C0, D0, H0, W0;         // caller's input [N, D0, H0, W0, C0]
  int pD0, pH0, pW0;          // caller's padding
  int kD0, kH0, kW0;          // caller's kernel
};
struct RowPlan {
  int Cp, PW, BN, MB, CBW, RB, n_rb, n_cb, slab_rows, patch_h, patch_w, n_chunks, n_nblocks, slabs;
  long long filter_elems, n_items;
  int raw_bytes, a_bytes, b_stage_bytes, n_b_stages, n_a_bufs, smem_total;
  int b_group;   // filter stages per barrier group (1, or 3 = all rows of a 3-row kernel)
  int s2_chunks;   // > 0: a stride-2 layer read from the caller's tensor through an element-strided tensor map (ceil(C0 / 32) chunks per phase)
  int raw_c, raw_off, raw_row_el;   // raw_c > 0: few-channel x is read as it lies (rows of W * C elements)
  int raw_seg, raw_fh, raw_pd, raw_ph, raw_pw;   // elements per pixel and raw row, raw rows per patch row, padding in x's own coordinates
  int pair;   // 1: CTA pairs (two images per work item, one M = 256 MMA over both SMs, filter slabs split between them)
};
bool rowfused_plan(const RowDesc &d, RowPlan *out);
cudaError_t launch_rowfused_filter_transform(const RowDesc &d, const RowPlan &p, int dtype, const void *w, void *u, cudaStream_t s);
cudaError_t launch_rowfused_forward(const RowDesc &d, const RowPlan &p, int dtype, const void *x, const void *u,
                                    const void *bias, void *y, void *pad_ws, cudaStream_t s, const char **detail);
cudaError_t read_and_clear_row_error(cudaStream_t s, unsigned int *code);

// Direct-tap kernel (wino_direct.cu): 16-bit layers, and fp32 layers with three tf32 products per multiply.
// A polyphase part of the taps along H and W: tap (th, tw) of the part reads the input (stride * output + org + tap) and is
// tap (t0 + ts * th, ...) of the weights.  A strided forward sums its parts; a strided data gradient writes each part's sums to
// output pixels of its own ("variants").
struct DirectPart {
  int org_h, org_w, th, tw, t0_h, ts_h, t0_w, ts_w;
  int oH, oW;                        // variants: output extents (before pooling)
  long long y_off;                   // variants: first output element
};
struct DirectDesc {
  int dtype, N, C, Cw, K, D, H, W;   // C: channels of the input tensor; Cw: of the weights (the rest are zeros)
  int oD, oH, oW, yH, yW;            // output extents (the largest part's), stored extents after pooling
  int sD, sH, sW, pD, kD, d0, ds;    // input step per output; depth taps kD, tap kd is depth d0 + ds * kd of the weights
  int kD_w, kH_w, kW_w;              // kernel extents of the weights
  int n_parts, variants;
  DirectPart parts[4];
  long long ys_n, ys_d, ys_h, ys_w;  // element strides of the output
  unsigned epilogue;
  int bias_f32;                      // the bias is fp32 whatever dtype is
  int fold;                          // few channels: the taps along W are folded into the channels and x is gathered by the kernel
  int x_first;                       // (fold only) x is [N, C, D, H, W]
  int weight_layout, transposed;     // transposed: K and C exchanged in the weights (data gradient)
};
// A forward layer; and the part of a layer's data gradient with input depths of parity e (e < stride along depth).
void direct_forward_desc(DirectDesc *q, int dtype, int N, int C, int K, const int in[3], const int ker[3], const int stride[3],
                         const int pad[3], const int out[3], int yH, int yW, unsigned epilogue, int weight_layout);
bool direct_grad_desc(DirectDesc *q, int dtype, int N, int C, int K, int Km, const int in[3], const int ker[3], const int stride[3],
                      const int pad[3], const int out[3], int weight_layout, int e, bool *zero_fill);
struct DirectPlan {
  int BN, MB, pair, split;           // columns and row blocks of an item, CTA pairs, CTAs that share an item's reduction
  int epi_sets;                      // sets of eight epilogue warps
  int TN, TH, TI, PW, slab_rows_h;   // a block's image groups and output rows, images within a group of 8 rows, pixels of a slab row, slab rows
  int ch_el, rb, n_chunks, k_full, k_tail;
  int taps[4], tap0[4], max_taps, n_taps, units;
  int n_wb, n_hb, n_tiles, n_kb, n_items;   // n_items: of one variant
  int slab_bytes, a_bytes, lo_off, b_tile, b_lo, b_bytes, G, n_a, n_b, smem;
  int raw_tma, raw_rem, raw_el, raw_box;   // fold: the raw patch loaded by TMA, elements before its first pixel, of a row, bytes
  long long filter_elems;
  double estimate;                   // clocks
};
bool direct_plan(const DirectDesc &d, DirectPlan *out);
bool direct_fold_desc(DirectDesc *q, const int pad[3], int x_first);   // turns a forward description into a folded one where it applies
// Whether the folded form is the faster one; `plain` is the layer on (padded) channels-last channels.
bool direct_fold_pays(const DirectDesc &fold, const DirectPlan &fp, const DirectDesc &plain, const int pad[3]);
cudaError_t launch_direct_filter_transform(const DirectDesc &d, const DirectPlan &p, int w_dtype, const void *w, void *u, cudaStream_t s);
cudaError_t launch_direct_forward(const DirectDesc &d, const DirectPlan &p, const void *x, const void *u, const void *bias, void *y,
                                  cudaStream_t s, const char **detail);
// Weight gradient (wino_wgrad.cu): 16-bit x and gy whose channel strides Cm, Km are multiples of 8; dW [K][C][taps] and the bias
// sums from fp32 accumulators.
struct WgradDesc {
  int dtype, N, C, K, Cm, Km, D, H, W, oD, oH, oW;
  int sD, sH, sW, pD, pH, pW, kD, kH, kW;
  int bias;
};
struct WgradPlan {
  alignas(8) unsigned char geom[2048];
  int smem, slab_rows_h;
  unsigned long long ws_bytes;
};
bool wgrad_plan(const WgradDesc &d, WgradPlan *out);
cudaError_t launch_wgrad(const WgradDesc &d, const WgradPlan &p, const void *x, const void *gy, void *dw, int dw_dtype, float *dbias,
                         void *ws, cudaStream_t s, const char **detail);
cudaError_t read_and_clear_wgrad_error(cudaStream_t s, unsigned int *code);
cudaError_t read_and_clear_direct_error(cudaStream_t s, unsigned int *code);

// Reads the error word of the bounded device waits, clears it and synchronises the stream.
cudaError_t read_and_clear_device_error(cudaStream_t s, unsigned int *code);

}  // namespace wino
