// cnn_ops.cu -- the warm-start network's non-convolution kernels: input
// packing, 2x average pooling, nearest 2x upsampling with skip concatenation,
// ReLU and bias gradients, the 1x1 output head with the loss, weight packing
// and the Adam update.  Channels-last BF16 volumes [nb][Y][X][Z][C].
#include <cuda_bf16.h>

#include <algorithm>

#include "xtg_cnn_internal.h"

namespace xtc {

static unsigned blocks(long long n, int t = 256) {
  long long b = (n + t - 1) / t;
  return (unsigned)(b < 1 ? 1 : (b > 148 * 32 ? 148 * 32 : b));
}
#define GRID_STRIDE(i, n) for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (n); i += (long long)gridDim.x * blockDim.x)

// two FP32 volumes [nb][Y][X][Z] -> BF16 [..][8] (channels 0, 1; rest 0), times scale
__global__ void k_pack_input(long long nv, const float *a, const float *b, float scale, __nv_bfloat16 *out) {
  GRID_STRIDE(v, nv) {
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int c = 0; c < 8; c++) h[c] = __float2bfloat16_rn(0.f);
    h[0] = __float2bfloat16_rn(a[v] * scale);
    h[1] = __float2bfloat16_rn(b[v] * scale);
    *reinterpret_cast<int4 *>(out + v * 8) = *reinterpret_cast<const int4 *>(h);
  }
}

// 2x2x2 average pooling (dims even)
__global__ void k_avgpool(int nb, int Y, int X, int Z, int C, const __nv_bfloat16 *in, __nv_bfloat16 *out) {
  const int Yo = Y / 2, Xo = X / 2, Zo = Z / 2;
  const long long n = (long long)nb * Yo * Xo * Zo * C;
  GRID_STRIDE(i, n) {
    long long r = i;
    const int c = (int)(r % C);
    r /= C;
    const int z = (int)(r % Zo);
    r /= Zo;
    const int x = (int)(r % Xo);
    r /= Xo;
    const int y = (int)(r % Yo);
    const int b = (int)(r / Yo);
    float s = 0.f;
    for (int d = 0; d < 8; d++) {
      const int yy = 2 * y + (d >> 2), xx = 2 * x + ((d >> 1) & 1), zz = 2 * z + (d & 1);
      s += __bfloat162float(in[((((size_t)b * Y + yy) * X + xx) * Z + zz) * C + c]);
    }
    out[i] = __float2bfloat16_rn(s * 0.125f);
  }
}

// the same pooling on 8-channel groups (C a multiple of 8): 16-byte loads and
// stores, each channel summed in the same order as above
__global__ void k_avgpool8(int nb, int Y, int X, int Z, int G, const int4 *in, int4 *out) {
  const int Yo = Y / 2, Xo = X / 2, Zo = Z / 2;
  const long long n = (long long)nb * Yo * Xo * Zo * G;
  GRID_STRIDE(i, n) {
    long long r = i;
    const int g = (int)(r % G);
    r /= G;
    const int z = (int)(r % Zo);
    r /= Zo;
    const int x = (int)(r % Xo);
    r /= Xo;
    const int y = (int)(r % Yo);
    const int b = (int)(r / Yo);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int d = 0; d < 8; d++) {
      const int yy = 2 * y + (d >> 2), xx = 2 * x + ((d >> 1) & 1), zz = 2 * z + (d & 1);
      const int4 q = __ldg(in + ((((size_t)b * Y + yy) * X + xx) * Z + zz) * G + g);
      const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&q);
#pragma unroll
      for (int c = 0; c < 8; c++) s[c] += __bfloat162float(h[c]);
    }
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int c = 0; c < 8; c++) o[c] = __float2bfloat16_rn(s[c] * 0.125f);
    out[i] = *reinterpret_cast<const int4 *>(o);
  }
}

// out[v] = [up2(a)[v] (Ca channels), skip[v] (Cb channels)] at the fine grid
__global__ void k_up_concat(int nb, int Y, int X, int Z, int Ca, int Cb, const __nv_bfloat16 *a,
                            const __nv_bfloat16 *skip, __nv_bfloat16 *out) {
  const int C = Ca + Cb;
  const long long n = (long long)nb * Y * X * Z * C;
  GRID_STRIDE(i, n) {
    long long r = i;
    const int c = (int)(r % C);
    r /= C;
    const int z = (int)(r % Z);
    r /= Z;
    const int x = (int)(r % X);
    r /= X;
    const int y = (int)(r % Y);
    const int b = (int)(r / Y);
    out[i] = c < Ca ? a[((((size_t)b * (Y / 2) + y / 2) * (X / 2) + x / 2) * (Z / 2) + z / 2) * Ca + c]
                    : skip[((((size_t)b * Y + y) * X + x) * Z + z) * Cb + (c - Ca)];
  }
}

// the same on 8-channel groups (Ca, Cb multiples of 8): one 16-byte copy per
// group, consecutive threads on consecutive output groups; GA, GB fixed at
// compile time (0: taken from the arguments) and 32-bit indices (n < 2^31)
template <int GA, int GB>
__global__ void k_up_concat8(int nb, int Y, int X, int Z, int ga, int gb, const int4 *__restrict__ a,
                             const int4 *__restrict__ skip, int4 *__restrict__ out) {
  const unsigned Ga = GA ? GA : ga, Gb = GB ? GB : gb, G = Ga + Gb;
  const unsigned n = (unsigned)nb * Y * X * Z * G;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned v = i / G, g = i - v * G;
    if (g < Ga) {
      const unsigned z = v % Z, r1 = v / Z, x = r1 % X, r2 = r1 / X;  // r2 = b * Y + y
      const unsigned cv = ((r2 >> 1) * (X >> 1) + (x >> 1)) * (Z >> 1) + (z >> 1);  // Y even: b*Y/2 + y/2
      out[i] = __ldg(a + (size_t)cv * Ga + g);
    } else {
      out[i] = __ldg(skip + (size_t)v * Gb + (g - Ga));
    }
  }
}

// gradient of k_up_concat with respect to a: da (coarse, FP32) sums the eight
// fine voxels' first Ca channels of dout (four channels a thread; the skip's
// channels are read in place by k_relu_back)
__global__ void k_up_back(int nb, int Yo, int Xo, int Zo, int Ca4, int C4, const float4 *__restrict__ dout,
                          float4 *__restrict__ da) {
  const int X = 2 * Xo, Z = 2 * Zo;
  const long long n = (long long)nb * Yo * Xo * Zo * Ca4;
  GRID_STRIDE(i, n) {
    const int c = (int)(i % Ca4);
    const unsigned v = (unsigned)(i / Ca4);
    const unsigned z = v % Zo, r1 = v / Zo, x = r1 % Xo, r2 = r1 / Xo;  // r2 = b * Yo + y
    const float4 *p = dout + (((size_t)r2 * 2 * X + 2 * x) * Z + 2 * z) * C4 + c;
    float4 q[8];
#pragma unroll
    for (int d = 0; d < 8; d++) q[d] = __ldg(p + ((size_t)((d >> 2) * X + ((d >> 1) & 1)) * Z + (d & 1)) * C4);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int d = 0; d < 8; d++) {
      s.x += q[d].x;
      s.y += q[d].y;
      s.z += q[d].z;
      s.w += q[d].w;
    }
    da[i] = s;
  }
}

// dpre = dpost * (post > 0), FP32 in -> BF16 out, and the bias gradient summed
// per channel.  dpost has rows of ld floats, the layer's C channels first
// at off; with `pooled` the gradient of the 2x pooling that also read the layer
// (coarse, rows of C floats) is added, an eighth of it per voxel.  Eight
// channels a thread; the block and the grid stride are multiples of C / 8, so
// a thread keeps its channels and their bias sums in registers.  Bound by
// memory: level 0 of a 8 x 32 x 128 x 32 step (8 bytes an element) 190 -> 48 us,
// and the pooling's and the skip's own passes over FP32 gradients (0.6 ms) go.
__global__ void __launch_bounds__(192) k_relu_back(unsigned nv, int C8, const float *__restrict__ dpost, int ld, int off,
                                                   const int4 *__restrict__ post, int4 *__restrict__ dpre, float *dbias,
                                                   const float *__restrict__ pooled, int Y, int X, int Z) {
  extern __shared__ float sb[];
  for (int c = threadIdx.x; c < 8 * C8; c += blockDim.x) sb[c] = 0.f;
  __syncthreads();
  const int g = threadIdx.x % C8;
  float bs[8];
#pragma unroll
  for (int c = 0; c < 8; c++) bs[c] = 0.f;
  const unsigned vpb = blockDim.x / C8;  // voxels a block takes at once
  for (unsigned v = blockIdx.x * vpb + threadIdx.x / C8; v < nv; v += gridDim.x * vpb) {
    const float4 *p = reinterpret_cast<const float4 *>(dpost + (size_t)v * ld + off) + 2 * g;
    const float4 a = __ldcs(p), b = __ldcs(p + 1);
    float d[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const int4 q = __ldg(post + (size_t)v * C8 + g);
    if (pooled) {
      const unsigned z = v % Z, r1 = v / Z, x = r1 % X, r2 = r1 / X;  // r2 = batch * Y + y, Y even
      const size_t cv = ((size_t)(r2 >> 1) * (X >> 1) + (x >> 1)) * (Z >> 1) + (z >> 1);
      const float4 *pp = reinterpret_cast<const float4 *>(pooled) + (cv * C8 + g) * 2;
      const float4 e = __ldg(pp), f = __ldg(pp + 1);
      const float pv[8] = {e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
#pragma unroll
      for (int c = 0; c < 8; c++) d[c] += 0.125f * pv[c];
    }
    const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&q);
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float t = __bfloat162float(h[c]) > 0.f ? d[c] : 0.f;
      o[c] = __float2bfloat16_rn(t);
      bs[c] += t;
    }
    dpre[(size_t)v * C8 + g] = *reinterpret_cast<const int4 *>(o);
  }
#pragma unroll
  for (int c = 0; c < 8; c++) atomicAdd(&sb[8 * g + c], bs[c]);
  __syncthreads();
  for (int c = threadIdx.x; c < 8 * C8; c += blockDim.x) atomicAdd(&dbias[c], sb[c]);
}

// 1x1 head: y[v] = base[v] + (sum_c h[v][c] w[c] + bias) / scale
__global__ void k_head(long long nv, int C, const __nv_bfloat16 *h, const float *w, const float *bias,
                       const float *base, float scale, float *y) {
  GRID_STRIDE(v, nv) {
    float acc = bias[0];
    for (int c0 = 0; c0 < C; c0 += 8) {
      const int4 q = __ldg(reinterpret_cast<const int4 *>(h + v * C + c0));
      const __nv_bfloat16 *hq = reinterpret_cast<const __nv_bfloat16 *>(&q);
#pragma unroll
      for (int c = 0; c < 8; c++) acc += __bfloat162float(hq[c]) * w[c0 + c];
    }
    y[v] = base[v] + acc / scale;
  }
}

// The head in training, 32 channels: loss = mean((y - target)^2 scale^2),
// accumulated in FP64, and its gradients with respect to h (FP32), w and bias.
// A warp takes 32 voxels: a lane each for the output (channels added in order,
// as in k_head), then four lanes a voxel, eight channels each, for the
// gradients, so that the stores are contiguous over the warp and a lane's
// weight-gradient sums stay in registers until the end (a shared atomic per
// voxel and channel before: 662 -> 42 us for 8 x 32 x 128 x 32 voxels;
// memory-bound).
__global__ void __launch_bounds__(256) k_head_train(long long nv, const __nv_bfloat16 *__restrict__ h,
                                                    const float *__restrict__ w, const float *__restrict__ bias,
                                                    const float *__restrict__ base, float scale,
                                                    const float *__restrict__ target, double *loss,
                                                    float *__restrict__ dh, float *dw, float *db, float inv_n) {
  __shared__ float sh[33];
  if (threadIdx.x < 33) sh[threadIdx.x] = 0.f;
  __syncthreads();
  const int sub = threadIdx.x & 3, lane = threadIdx.x & 31;
  float wv[8], dwv[8], dbv = 0.f;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    wv[c] = w[8 * sub + c];
    dwv[c] = 0.f;
  }
  const float b0 = bias[0];
  double lsum = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; v0 < nv; v0 += stride) {
    const long long v = v0 + lane;
    float g = 0.f;  // d loss / d acc
    if (v < nv) {
      float acc = b0;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int4 q = __ldg(reinterpret_cast<const int4 *>(h + v * 32) + u);
        const __nv_bfloat16 *hq = reinterpret_cast<const __nv_bfloat16 *>(&q);
#pragma unroll
        for (int c = 0; c < 8; c++) acc += __bfloat162float(hq[c]) * w[8 * u + c];
      }
      const float out = base[v] + acc / scale;
      const float diff = (out - target[v]) * scale;
      lsum += (double)diff * diff;
      g = 2.f * diff * inv_n;
      dbv += g;
    }
#pragma unroll
    for (int it = 0; it < 4; it++) {
      const long long vv = v0 + 8 * it + (lane >> 2);
      const float gg = __shfl_sync(0xffffffffu, g, 8 * it + (lane >> 2));
      if (vv < nv) {
        const int4 q = __ldg(reinterpret_cast<const int4 *>(h + vv * 32) + sub);
        const __nv_bfloat16 *hq = reinterpret_cast<const __nv_bfloat16 *>(&q);
        float4 *d = reinterpret_cast<float4 *>(dh + vv * 32) + 2 * sub;
        d[0] = make_float4(gg * wv[0], gg * wv[1], gg * wv[2], gg * wv[3]);
        d[1] = make_float4(gg * wv[4], gg * wv[5], gg * wv[6], gg * wv[7]);
#pragma unroll
        for (int c = 0; c < 8; c++) dwv[c] += gg * __bfloat162float(hq[c]);
      }
    }
  }
  __syncwarp();
  for (int off = 4; off < 32; off <<= 1) {
#pragma unroll
    for (int c = 0; c < 8; c++) dwv[c] += __shfl_xor_sync(0xffffffffu, dwv[c], off);
  }
  for (int off = 1; off < 32; off <<= 1) {
    dbv += __shfl_xor_sync(0xffffffffu, dbv, off);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
  }
  if (lane < 4) {
#pragma unroll
    for (int c = 0; c < 8; c++) atomicAdd(&sh[8 * sub + c], dwv[c]);
    if (sub == 0) {
      atomicAdd(&sh[32], dbv);
      atomicAdd(loss, lsum * inv_n);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) atomicAdd(&dw[threadIdx.x], sh[threadIdx.x]);
  if (threadIdx.x == 32) atomicAdd(db, sh[32]);
}

// master weights P[(tap*cin + ci)][cout] (FP32) -> W[cout][kpad] and Wt[ci][kpad_t]
// (BF16), a layer per grid row
struct PackLayers {
  PackLayer l[16];
};
__global__ void k_pack_weights(const __grid_constant__ PackLayers L) {
  const PackLayer &l = L.l[blockIdx.y];
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int i = i0; i < l.cout * l.kpad; i += step) {
    const int co = i / l.kpad, k = i % l.kpad;
    float v = 0.f;
    if (k < 27 * l.cin) {
      const int tap = k / l.cin, ci = k % l.cin;
      if (ci < l.cin_real) v = l.p[((size_t)tap * l.cin_real + ci) * l.cout + co];
    }
    l.w[i] = __float2bfloat16_rn(v);
  }
  if (!l.wt) return;
  for (int i = i0; i < l.cin * l.kpad_t; i += step) {
    const int ci = i / l.kpad_t, k = i % l.kpad_t;
    float v = 0.f;
    if (k < 27 * l.cout && ci < l.cin_real) {
      const int tap = k / l.cout, co = k % l.cout;
      v = l.p[((size_t)tap * l.cin_real + ci) * l.cout + co];
    }
    l.wt[i] = __float2bfloat16_rn(v);
  }
}

// element i of a packed layout: where it comes from in w[n][kpad] (k = tap * cin +
// ci, tap = (dy+1)*9 + (dx+1)*3 + (dz+1)), or -1 for a zero.
// Tile kernel: Wp[chunk][(ey+1)*3 + (ex+1)][half][dzi][n][8], ci = 16 chunk + 8
// half + e, effective offsets (ey, ex, ez = 1 - dzi) = sign x (dy, dx, dz)
__device__ __forceinline__ int tile_source(const PackJob &j, int i) {
  const int e = i % 8, r = i / 8, nn = r % j.n, q = r / j.n, dzi = q % 3, h = q / 3 % 2, g = q / 6 % 9, c = q / 54;
  const int ci = 16 * c + 8 * h + e;
  const int dy = j.sign * (g / 3 - 1), dx = j.sign * (g % 3 - 1), dz = j.sign * (1 - dzi);
  const int t = (dy + 1) * 9 + (dx + 1) * 3 + (dz + 1);
  return ci < j.cin ? nn * j.kpad + t * j.cin + ci : -1;
}
// box and halo kernels: rows of CH channels per (tap, chunk, n), 16-byte units swizzled
template <int CH>
__device__ __forceinline__ int box_source(const PackJob &j, int i) {
  const int e = i % 8, u = i / 8 % (CH / 8), row = i / CH, nn = row % j.n, tc = row / j.n;
  const int nchunk = (j.cin + CH - 1) / CH, c = tc % nchunk, t = tc / nchunk;
  const int ci = c * CH + box_swizzle(CH, nn, u) * 8 + e;
  return ci < j.cin ? nn * j.kpad + t * j.cin + ci : -1;
}
// first layer (two real channels): [n][64], k = 2 tap + ci
__device__ __forceinline__ int first_source(const PackJob &j, int i) {
  const int nn = i / 64, k = i % 64;
  return k < 54 ? nn * j.kpad + k / 2 * j.cin + k % 2 : -1;
}
__host__ __device__ inline int pack_elems(const PackJob &j) {
  if (j.kind == PACK_TILE) return (j.cin + 15) / 16 * 27 * 16 * j.n;
  if (j.kind == PACK_FIRST) return j.n * 64;
  const int ch = box_ch(j.cin);
  return 27 * ((j.cin + ch - 1) / ch) * j.n * ch;
}

// every layout of every layer in one launch, a job per grid row: a launch each
// (47 of them) took 120 us of a training step beside 50 for k_pack_weights, now
// 25 beside 12.
struct PackJobs {
  PackJob j[64];
};
__global__ void k_pack_jobs(const __grid_constant__ PackJobs J) {
  const PackJob &j = J.j[blockIdx.y];
  const int total = pack_elems(j), ch = box_ch(j.cin);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int src = j.kind == PACK_TILE    ? tile_source(j, i)
                    : j.kind == PACK_FIRST ? first_source(j, i)
                    : ch == 64             ? box_source<64>(j, i)
                                           : box_source<32>(j, i);
    j.wp[i] = src >= 0 ? j.w[src] : __float2bfloat16_rn(0.f);
  }
}

// Adam (Kingma & Ba 2015) with bias correction
__global__ void k_adam(long long n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  GRID_STRIDE(i, n) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// patch batch: dst[p] = src_vol[p][y0:y0+py][x0:x0+px][z0:z0+pz]
__global__ void k_crop(int np, const float *const *src, const int4 *org, int Y, int X, int Z, int py, int px, int pz,
                       float *dst) {
  const long long n = (long long)np * py * px * pz;
  GRID_STRIDE(i, n) {
    long long r = i;
    const int z = (int)(r % pz);
    r /= pz;
    const int x = (int)(r % px);
    r /= px;
    const int y = (int)(r % py);
    const int p = (int)(r / py);
    const int4 o = org[p];
    dst[i] = src[o.w][(((size_t)(o.x + y)) * X + (o.y + x)) * Z + (o.z + z)];
  }
}

// ---------------------------------------------------------------- launchers
void crop(int np, const float *const *src, const int4 *org, int Y, int X, int Z, int py, int px, int pz, float *dst,
          cudaStream_t st) {
  k_crop<<<blocks((long long)np * py * px * pz), 256, 0, st>>>(np, src, org, Y, X, Z, py, px, pz, dst);
}
void pack_input(long long nv, const float *a, const float *b, float scale, __nv_bfloat16 *out, cudaStream_t st) {
  k_pack_input<<<blocks(nv), 256, 0, st>>>(nv, a, b, scale, out);
}
void avgpool(int nb, int Y, int X, int Z, int C, const __nv_bfloat16 *in, __nv_bfloat16 *out, cudaStream_t st) {
  if (C % 8 == 0)
    k_avgpool8<<<blocks((long long)nb * Y * X * Z * C / 64), 256, 0, st>>>(
        nb, Y, X, Z, C / 8, reinterpret_cast<const int4 *>(in), reinterpret_cast<int4 *>(out));
  else
    k_avgpool<<<blocks((long long)nb * Y * X * Z * C / 8), 256, 0, st>>>(nb, Y, X, Z, C, in, out);
}
void up_concat(int nb, int Y, int X, int Z, int Ca, int Cb, const __nv_bfloat16 *a, const __nv_bfloat16 *skip,
               __nv_bfloat16 *out, cudaStream_t st) {
  const long long n8 = (long long)nb * Y * X * Z * (Ca + Cb) / 8;
  if (Ca % 8 == 0 && Cb % 8 == 0 && Y % 2 == 0 && n8 < (1ll << 31)) {
    const int ga = Ca / 8, gb = Cb / 8;
    auto k = (ga == 6 && gb == 4)   ? k_up_concat8<6, 4>
             : (ga == 8 && gb == 6)  ? k_up_concat8<8, 6>
             : (ga == 12 && gb == 8) ? k_up_concat8<12, 8>
                                     : k_up_concat8<0, 0>;
    k<<<blocks(n8), 256, 0, st>>>(nb, Y, X, Z, ga, gb, reinterpret_cast<const int4 *>(a),
                                  reinterpret_cast<const int4 *>(skip), reinterpret_cast<int4 *>(out));
  } else
    k_up_concat<<<blocks((long long)nb * Y * X * Z * (Ca + Cb)), 256, 0, st>>>(nb, Y, X, Z, Ca, Cb, a, skip, out);
}
void up_back(int nb, int Y, int X, int Z, int Ca, int Cb, const float *dout, float *da, cudaStream_t st) {
  k_up_back<<<blocks((long long)nb * Y * X * Z / 8 * Ca / 4), 256, 0, st>>>(
      nb, Y / 2, X / 2, Z / 2, Ca / 4, (Ca + Cb) / 4, reinterpret_cast<const float4 *>(dout), reinterpret_cast<float4 *>(da));
}
void relu_back(int nb, int Y, int X, int Z, int C, const float *dpost, int ld, int off, const float *pooled,
               const __nv_bfloat16 *post, __nv_bfloat16 *dpre, float *dbias, cudaStream_t st) {
  const unsigned nv = (unsigned)nb * Y * X * Z;
  const int c8 = C / 8, vpb = 192 / c8;  // C / 8 is 4, 6, 8 or 12
  const unsigned grid = (unsigned)std::min<long long>(((long long)nv + vpb - 1) / vpb, 148 * 10);
  k_relu_back<<<grid, (unsigned)(vpb * c8), C * sizeof(float), st>>>(nv, c8, dpost, ld, off,
                                                                     reinterpret_cast<const int4 *>(post),
                                                                     reinterpret_cast<int4 *>(dpre), dbias, pooled, Y, X, Z);
}
void head(long long nv, int C, const __nv_bfloat16 *h, const float *w, const float *bias, const float *base, float scale,
          float *y, cudaStream_t st) {
  k_head<<<blocks(nv), 256, 0, st>>>(nv, C, h, w, bias, base, scale, y);
}
void head_train(long long nv, const __nv_bfloat16 *h, const float *w, const float *bias, const float *base, float scale,
                const float *target, double *loss, float *dh, float *dw, float *db, cudaStream_t st) {
  const unsigned grid = (unsigned)std::min<long long>((nv + 255) / 256, 148 * 8);
  k_head_train<<<grid, 256, 0, st>>>(nv, h, w, bias, base, scale, target, loss, dh, dw, db, 1.f / (float)nv);
}
void pack_weights(const PackLayer *layers, int count, cudaStream_t st) {
  PackLayers L{};
  int most = 1;
  for (int i = 0; i < count; i++) {
    L.l[i] = layers[i];
    most = std::max(most, std::max(layers[i].cout * layers[i].kpad, layers[i].cin * layers[i].kpad_t));
  }
  k_pack_weights<<<dim3((unsigned)std::min((most + 255) / 256, 256), (unsigned)count), 256, 0, st>>>(L);
}
cudaError_t pack_kernel_weights(const PackJob *jobs, int count, cudaStream_t st) {
  PackJobs J{};
  int most = 1;
  for (int i = 0; i < count; i++) {
    J.j[i] = jobs[i];
    most = std::max(most, pack_elems(jobs[i]));
  }
  k_pack_jobs<<<dim3((unsigned)std::min((most + 255) / 256, 256), (unsigned)count), 256, 0, st>>>(J);
  return cudaGetLastError();
}
void adam(long long n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps, int t,
          cudaStream_t st) {
  const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
  k_adam<<<blocks(n), 256, 0, st>>>(n, p, g, m, v, lr, b1, b2, eps, c1, c2);
}

}  // namespace xtc
