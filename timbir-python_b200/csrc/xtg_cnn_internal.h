// xtg_cnn_internal.h -- shared declarations of the warm-start network's kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace xtc {

// channels-last volume [nb][Y][X][Z][cin] convolved to n output channels
struct ConvShape {
  int nb, Y, X, Z;
  int cin;   // input channels as stored (multiple of 8)
  int n;     // output channels (multiple of 16, <= 256)
  int kpad;  // K-major weight row length: 27 * cin rounded up to 64
};

cudaError_t conv_forward(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias,
                         void *out, int epi, int sign, int *err, cudaStream_t st);
// the first layer (2 FP32 input channels, the input packing fused in): w64 [n][64], k = 2 tap + channel
cudaError_t conv_first(int nb, int Y, int X, int Z, const float *a, const float *b, float scale,
                       const __nv_bfloat16 *w64, const float *bias, int n, __nv_bfloat16 *out, int *err,
                       cudaStream_t st);
// its weight gradient (32 output channels), added to dw [2 tap + channel][32]
cudaError_t wgrad_first(int nb, int Y, int X, int Z, const float *a, const float *b, float scale,
                        const __nv_bfloat16 *dout, float *dw, int *err, cudaStream_t st);
// the staged tile kernel (cnn_conv_tile.cu): X a multiple of 128, Z even,
// n <= 64; weights pre-packed (PACK_TILE) into conv_tile_wp_elems values
bool conv_tile_supported(const ConvShape &s);
size_t conv_tile_wp_elems(int cin, int n);
// (epi 3: the output head on relu(acc + bias) in BF16, out = base + (h . w + b) / scale in FP32)
struct TileHead {
  const float *w = nullptr, *b = nullptr, *base = nullptr;
  float scale = 1.f;
};
// with `up`, channels [0, ca) are the 2x nearest upsampling of that coarse
// volume (ca channels) and `in` holds the other cin - ca (epi 0)
cudaError_t conv_forward_tile(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *wp, const float *bias,
                              void *out, int epi, int sign, int *err, cudaStream_t st, const __nv_bfloat16 *up = nullptr,
                              int ca = 0, const TileHead &hd = TileHead{});
// TMA boxes of 128 voxels per tap (cnn_conv_box.cu): any volume, cin and n
// multiples of 16; weights pre-packed (PACK_BOX) into
// conv_box_wp_elems values (the sign stays an argument)
bool conv_box_supported(const ConvShape &s);
size_t conv_box_wp_elems(int cin, int n);
cudaError_t conv_forward_box(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *wp, const float *bias,
                             void *out, int epi, int sign, int *err, cudaStream_t st);
bool wgrad_box_supported(const ConvShape &s);
cudaError_t conv_wgrad_box(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *dout, float *dw, int *err,
                           cudaStream_t st);
// weight gradient: the TMA tile kernel where wgrad_tile_supported (cout 32,
// cin a multiple of 16, X a multiple of 128, Z even), else the gather kernel;
// path 1 forces the gather kernel, 2 the tile kernel (cudaErrorNotSupported
// where it does not apply)
cudaError_t conv_wgrad(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *dout, float *dw, int *err,
                       cudaStream_t st, int path = 0);
bool wgrad_tile_supported(const ConvShape &s);
cudaError_t conv_wgrad_tile(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *dout, float *dw,
                            int *err, cudaStream_t st);

void pack_input(long long nv, const float *a, const float *b, float scale, __nv_bfloat16 *out, cudaStream_t st);
void avgpool(int nb, int Y, int X, int Z, int C, const __nv_bfloat16 *in, __nv_bfloat16 *out, cudaStream_t st);
void up_concat(int nb, int Y, int X, int Z, int Ca, int Cb, const __nv_bfloat16 *a, const __nv_bfloat16 *skip,
               __nv_bfloat16 *out, cudaStream_t st);
// gradient of up_concat w.r.t. its coarse input; the skip's is dout's channels from Ca on
void up_back(int nb, int Y, int X, int Z, int Ca, int Cb, const float *dout, float *da, cudaStream_t st);
// dpost: rows of ld floats, the C channels from off on; pooled (or null): gradient of the 2x pooling of the same layer
void relu_back(int nb, int Y, int X, int Z, int C, const float *dpost, int ld, int off, const float *pooled,
               const __nv_bfloat16 *post, __nv_bfloat16 *dpre, float *dbias, cudaStream_t st);
void head(long long nv, int C, const __nv_bfloat16 *h, const float *w, const float *bias, const float *base, float scale,
          float *y, cudaStream_t st);
void head_train(long long nv, const __nv_bfloat16 *h, const float *w, const float *bias, const float *base, float scale,
                const float *target, double *loss, float *dh, float *dw, float *db, cudaStream_t st);
// master weights of a layer -> its K-major BF16 rows, and the transposed ones (wt may be null)
struct PackLayer {
  int cin_real, cin, cout, kpad, kpad_t;
  const float *p;
  __nv_bfloat16 *w, *wt;
};
void pack_weights(const PackLayer *layers, int count, cudaStream_t st);  // 16 layers at most
// K-major rows w[n][kpad] -> the order a kernel reads: the tile kernel's (with
// the taps' sign), the box and halo kernels', or the first layer's [n][64]
enum PackKind { PACK_TILE, PACK_BOX, PACK_FIRST };
struct PackJob {
  int kind, cin, n, kpad, sign;
  const __nv_bfloat16 *w;
  __nv_bfloat16 *wp;
};
cudaError_t pack_kernel_weights(const PackJob *jobs, int count, cudaStream_t st);  // 64 jobs at most
// channels per TMA row of the box kernels, and where 16-byte unit u of such a row r lies in its swizzle
__host__ __device__ constexpr int box_ch(int cin) { return (cin + 63) / 64 * 64 <= (cin + 31) / 32 * 32 ? 64 : 32; }
__host__ __device__ constexpr int box_swizzle(int ch, int r, int u) { return ch == 64 ? u ^ (r & 7) : u ^ ((r >> 1) & 3); }
void adam(long long n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps, int t,
          cudaStream_t st);
void crop(int np, const float *const *src, const int4 *org, int Y, int X, int Z, int py, int px, int pz, float *dst,
          cudaStream_t st);

cudaError_t wait_selftest(int arrive, long long limit, int *err, cudaStream_t st);
}  // namespace xtc
