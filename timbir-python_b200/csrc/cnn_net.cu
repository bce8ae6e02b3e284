// cnn_net.cu -- the warm-start network: a 3D encoder-decoder (four levels,
// 32/48/64/96 channels, two 3x3x3 convolutions + ReLU per level and side,
// 2x average pooling down, nearest 2x upsampling + skip concatenation up, a
// 1x1 head) mapping (FBP image, image after a few ICD equits) to a residual
// correction of the latter: out = icd + head / scale.  About 1.44 M parameters,
// FP32 master weights, BF16 weights and activations on the tcgen05 tensor
// cores, FP32 gradients, Adam.  All compute runs in this library's kernels;
// the host only sequences launches.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/xtg.h"
#include "../../include/xtg_cnn.h"
#include "xtg_cnn_internal.h"

void xtg_set_error_text(const char *msg);

namespace {

using bf16 = __nv_bfloat16;
constexpr float kScale = 100.f;  // inputs and correction in units of 1/100 per voxel length
constexpr int kLayers = 14;
// (cin as used by the data, cin as stored (multiple of 8), cout)
constexpr int kSpec[kLayers][2] = {{2, 32},  {32, 32}, {32, 48}, {48, 48},  {48, 64}, {64, 64},  {64, 96},
                                   {96, 96}, {160, 64}, {64, 64}, {112, 48}, {48, 48}, {80, 32}, {32, 32}};
constexpr int kHeadC = 32;

int kpad_of(int cin) { return (27 * cin + 63) / 64 * 64; }
int cin_store(int cin_real) { return (cin_real + 7) / 8 * 8; }

struct Layer {
  int cin_real, cin, cout, kpad, kpad_t;
  size_t off_w, off_b;  // offsets in the parameter vector
  bf16 *W = nullptr, *Wt = nullptr;
  bf16 *Wp = nullptr;   // W packed for the tile kernel
  bf16 *Wtp = nullptr;  // Wt packed for the tile kernel (input gradient, layers with cin <= 64)
  bf16 *Wb = nullptr;   // W and Wt packed for the box kernel
  bf16 *Wtb = nullptr;
  bf16 *W64 = nullptr;  // the first layer's W as [cout][64], k = 2 tap + channel
};

struct Buf {
  void *p = nullptr;
  size_t bytes = 0;
  cudaError_t ensure(size_t n) {
    if (n <= bytes) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMalloc(&p, n);
    if (e == cudaSuccess) bytes = n;
    return e;
  }
  ~Buf() {
    if (p) cudaFree(p);
  }
  template <class T>
  T *as() const {
    return reinterpret_cast<T *>(p);
  }
};

}  // namespace

struct xtc_net {
  Layer L[kLayers];
  size_t n_params = 0, off_hw = 0, off_hb = 0;
  float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;  // parameters, gradients, Adam moments
  double *d_loss = nullptr;
  int *d_err = nullptr;
  int step = 0;
  bool packed = false;
  cudaStream_t st = 0;
  // activations (BF16) and gradients (FP32) for the current batch shape
  int nb = 0, Y = 0, X = 0, Z = 0;
  bool grads = false;  // the gradient buffers fit that shape too
  Buf in0, a[kLayers], u0, u1, u2, p0, p1, p2, g32, gtmp, gcat[3], gpre;  // gcat: gradients of u0, u1, u2
  Buf start;  // the learned start's three images (xtg_warm.cu), kept between calls
};

namespace {

int set_fail(const char *what, cudaError_t e) {
  char b[256];
  snprintf(b, sizeof b, "%s: %s", what, cudaGetErrorString(e));
  xtg_set_error_text(b);
  return XTG_E_CUDA;
}
#define NCK(x)                                   \
  do {                                           \
    cudaError_t e_ = (x);                        \
    if (e_ != cudaSuccess) return set_fail(#x, e_); \
  } while (0)

uint64_t mix(uint64_t &s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
double gauss(uint64_t &s) {  // Box-Muller
  const double u1 = ((mix(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0);
  const double u2 = ((mix(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0);
  return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
}

int pack_all(xtc_net *n) {
  xtc::PackLayer layers[kLayers];
  xtc::PackJob jobs[4 * kLayers + 1];
  int nj = 0;
  for (int i = 0; i < kLayers; i++) {
    Layer &l = n->L[i];
    layers[i] = {l.cin_real, l.cin, l.cout, l.kpad, l.kpad_t, n->P + l.off_w, l.W, i ? l.Wt : nullptr};
    if (l.Wp) jobs[nj++] = {xtc::PACK_TILE, l.cin, l.cout, l.kpad, 1, l.W, l.Wp};
    if (l.Wtp) jobs[nj++] = {xtc::PACK_TILE, l.cout, l.cin, l.kpad_t, -1, l.Wt, l.Wtp};
    if (l.Wb) jobs[nj++] = {xtc::PACK_BOX, l.cin, l.cout, l.kpad, 1, l.W, l.Wb};
    if (l.Wtb) jobs[nj++] = {xtc::PACK_BOX, l.cout, l.cin, l.kpad_t, 1, l.Wt, l.Wtb};
    if (l.W64) jobs[nj++] = {xtc::PACK_FIRST, l.cin, l.cout, l.kpad, 1, l.W, l.W64};
  }
  xtc::pack_weights(layers, kLayers, n->st);
  NCK(xtc::pack_kernel_weights(jobs, nj, n->st));
  n->packed = true;
  return 0;
}

int check_err(xtc_net *n) {
  int h = 0;
  NCK(cudaMemcpyAsync(&h, n->d_err, sizeof(int), cudaMemcpyDeviceToHost, n->st));
  NCK(cudaStreamSynchronize(n->st));
  if (h) {
    cudaMemsetAsync(n->d_err, 0, sizeof(int), n->st);
    xtg_set_error_text("xtc_net: tensor-core pipeline wait timed out");
    return XTG_E_TIMEOUT;
  }
  return 0;
}

// activation buffers for a batch shape, and gradient buffers for training
int ensure_buffers(xtc_net *n, int nb, int Y, int X, int Z, bool training) {
  if (n->nb == nb && n->Y == Y && n->X == X && n->Z == Z && (n->grads || !training)) return 0;
  n->nb = 0;  // no shape's buffers, until all of them are there
  const size_t v0 = (size_t)nb * Y * X * Z, v1 = v0 / 8, v2 = v1 / 8, v3 = v2 / 8;
  const size_t lv[kLayers] = {v0, v0, v1, v1, v2, v2, v3, v3, v2, v2, v1, v1, v0, v0};
  if (training) NCK(n->in0.ensure(v0 * 8 * sizeof(bf16)));
  size_t gmax = 0;
  for (int i = 0; i < kLayers; i++) {
    if (i < 13 || training) NCK(n->a[i].ensure(lv[i] * n->L[i].cout * sizeof(bf16)));  // (forward: where it is stored)
    if (i != 8 && i != 10 && i != 12) gmax = std::max(gmax, lv[i] * (size_t)n->L[i].cin);  // (those go to gcat)
    gmax = std::max(gmax, lv[i] * (size_t)n->L[i].cout);
  }
  NCK(n->p0.ensure(v1 * 32 * sizeof(bf16)));
  NCK(n->p1.ensure(v2 * 48 * sizeof(bf16)));
  NCK(n->p2.ensure(v3 * 64 * sizeof(bf16)));
  if (training) {
    NCK(n->g32.ensure(gmax * sizeof(float)));
    NCK(n->gtmp.ensure(gmax * sizeof(float)));
    NCK(n->gpre.ensure(gmax * sizeof(bf16)));
    NCK(n->gcat[0].ensure(v0 * 80 * sizeof(float)));
    NCK(n->gcat[1].ensure(v1 * 112 * sizeof(float)));
    NCK(n->gcat[2].ensure(v2 * 160 * sizeof(float)));
  }
  n->nb = nb;
  n->Y = Y;
  n->X = X;
  n->Z = Z;
  n->grads = training;
  return 0;
}

int conv(xtc_net *n, int li, const bf16 *in, int lvl, bf16 *out) {
  const Layer &l = n->L[li];
  xtc::ConvShape s{n->nb, n->Y >> lvl, n->X >> lvl, n->Z >> lvl, l.cin, l.cout, l.kpad};
  if (l.Wp && xtc::conv_tile_supported(s)) {
    const cudaError_t e = xtc::conv_forward_tile(s, in, l.Wp, n->P + l.off_b, out, 0, 1, n->d_err, n->st);
    if (e != cudaErrorNotSupported) {
      NCK(e);
      return 0;
    }
    cudaGetLastError();
  }
  if (l.Wb && xtc::conv_box_supported(s)) {
    const cudaError_t e = xtc::conv_forward_box(s, in, l.Wb, n->P + l.off_b, out, 0, 1, n->d_err, n->st);
    if (e != cudaErrorNotSupported) {
      NCK(e);
      return 0;
    }
    cudaGetLastError();
  }
  NCK(xtc::conv_forward(s, in, l.W, n->P + l.off_b, out, 0, 1, n->d_err, n->st));
  return 0;
}

// conv li of the concatenation of a's 2x upsampling (ca channels) and skip: read
// in place where the tile kernel takes the shape, else (or where training needs
// it later) formed in cat
int conv_cat(xtc_net *n, int li, const bf16 *a, int ca, const bf16 *skip, int cb, int lvl, Buf &cat, bf16 *out, bool keep) {
  const Layer &l = n->L[li];
  xtc::ConvShape s{n->nb, n->Y >> lvl, n->X >> lvl, n->Z >> lvl, l.cin, l.cout, l.kpad};
  if (!keep && l.Wp && xtc::conv_tile_supported(s)) {
    const cudaError_t e = xtc::conv_forward_tile(s, skip, l.Wp, n->P + l.off_b, out, 0, 1, n->d_err, n->st, a, ca);
    if (e != cudaErrorNotSupported) {
      NCK(e);
      return 0;
    }
    cudaGetLastError();
  }
  NCK(cat.ensure((size_t)s.nb * s.Y * s.X * s.Z * l.cin * sizeof(bf16)));
  xtc::up_concat(n->nb, s.Y, s.X, s.Z, ca, cb, a, skip, cat.as<bf16>(), n->st);
  return conv(n, li, cat.as<bf16>(), lvl, out);
}

int forward(xtc_net *n, const float *fbp, const float *icd, float *out, const float *target) {
  const int nb = n->nb, Y = n->Y, X = n->X, Z = n->Z;
  const long long v0 = (long long)nb * Y * X * Z;
  cudaStream_t st = n->st;
  bf16 *A[kLayers];
  for (int i = 0; i < kLayers; i++) A[i] = n->a[i].as<bf16>();
  int rc;
  if (target) {  // training's first layer sums over the packed input, in the general kernels' order
    xtc::pack_input(v0, fbp, icd, kScale, n->in0.as<bf16>(), st);
    if ((rc = conv(n, 0, n->in0.as<bf16>(), 0, A[0]))) return rc;
  } else {
    NCK(xtc::conv_first(nb, Y, X, Z, fbp, icd, kScale, n->L[0].W64, n->P + n->L[0].off_b, n->L[0].cout, A[0],
                        n->d_err, st));
  }
  if ((rc = conv(n, 1, A[0], 0, A[1]))) return rc;
  xtc::avgpool(nb, Y, X, Z, 32, A[1], n->p0.as<bf16>(), st);
  if ((rc = conv(n, 2, n->p0.as<bf16>(), 1, A[2]))) return rc;
  if ((rc = conv(n, 3, A[2], 1, A[3]))) return rc;
  xtc::avgpool(nb, Y / 2, X / 2, Z / 2, 48, A[3], n->p1.as<bf16>(), st);
  if ((rc = conv(n, 4, n->p1.as<bf16>(), 2, A[4]))) return rc;
  if ((rc = conv(n, 5, A[4], 2, A[5]))) return rc;
  xtc::avgpool(nb, Y / 4, X / 4, Z / 4, 64, A[5], n->p2.as<bf16>(), st);
  if ((rc = conv(n, 6, n->p2.as<bf16>(), 3, A[6]))) return rc;
  if ((rc = conv(n, 7, A[6], 3, A[7]))) return rc;
  const bool keep = target != nullptr;
  if ((rc = conv_cat(n, 8, A[7], 96, A[5], 64, 2, n->u2, A[8], keep))) return rc;
  if ((rc = conv(n, 9, A[8], 2, A[9]))) return rc;
  if ((rc = conv_cat(n, 10, A[9], 64, A[3], 48, 1, n->u1, A[10], keep))) return rc;
  if ((rc = conv(n, 11, A[10], 1, A[11]))) return rc;
  if ((rc = conv_cat(n, 12, A[11], 48, A[1], 32, 0, n->u0, A[12], keep))) return rc;
  if (!target) {
    // the last layer and the head in one kernel where the tile kernel takes the shape
    const Layer &l = n->L[13];
    const xtc::ConvShape s{nb, Y, X, Z, l.cin, l.cout, l.kpad};
    if (l.Wp && xtc::conv_tile_supported(s)) {
      const cudaError_t e = xtc::conv_forward_tile(s, A[12], l.Wp, n->P + l.off_b, out, 3, 1, n->d_err, st, nullptr, 0,
                                                   {n->P + n->off_hw, n->P + n->off_hb, icd, kScale});
      if (e != cudaErrorNotSupported) {
        NCK(e);
        return 0;
      }
      cudaGetLastError();
    }
    NCK(n->a[13].ensure((size_t)v0 * l.cout * sizeof(bf16)));
    A[13] = n->a[13].as<bf16>();
  }
  if ((rc = conv(n, 13, A[12], 0, A[13]))) return rc;
  if (target) {
    NCK(cudaMemsetAsync(n->d_loss, 0, sizeof(double), st));
    xtc::head_train(v0, A[13], n->P + n->off_hw, n->P + n->off_hb, icd, kScale, target, n->d_loss, n->g32.as<float>(),
                    n->G + n->off_hw, n->G + n->off_hb, st);
  } else {
    xtc::head(v0, kHeadC, A[13], n->P + n->off_hw, n->P + n->off_hb, icd, kScale, out, st);
  }
  NCK(cudaGetLastError());
  return 0;
}

// backward of conv li with post-ReLU gradient dpost (FP32, rows of ld floats,
// the layer's channels from off on; plus the pooling's, `pooled`, where the
// layer was pooled too) and post-activation `post`; writes the input gradient
// (FP32) to din when din != nullptr.  The first layer has no `in` but the two
// input volumes.
int conv_back(xtc_net *n, int li, const float *dpost, const bf16 *post, const bf16 *in, int lvl, float *din, int ld = 0,
              int off = 0, const float *pooled = nullptr, const float *fbp = nullptr, const float *icd = nullptr) {
  const Layer &l = n->L[li];
  bf16 *dpre = n->gpre.as<bf16>();
  xtc::relu_back(n->nb, n->Y >> lvl, n->X >> lvl, n->Z >> lvl, l.cout, dpost, ld ? ld : l.cout, off, pooled, post, dpre,
                 n->G + l.off_b, n->st);
  xtc::ConvShape s{n->nb, n->Y >> lvl, n->X >> lvl, n->Z >> lvl, l.cin, l.cout, l.kpad};
  if (!in)
    NCK(xtc::wgrad_first(n->nb, n->Y, n->X, n->Z, fbp, icd, kScale, dpre, n->G + l.off_w, n->d_err, n->st));
  else
    NCK(xtc::conv_wgrad(s, in, dpre, n->G + l.off_w, n->d_err, n->st));
  if (din) {
    // the input gradient: the same convolution with transposed weights and
    // negated offsets, on the tile kernel where the shape allows
    xtc::ConvShape t{n->nb, n->Y >> lvl, n->X >> lvl, n->Z >> lvl, l.cout, l.cin, l.kpad_t};
    if (l.Wtp && xtc::conv_tile_supported(t)) {
      const cudaError_t e = xtc::conv_forward_tile(t, dpre, l.Wtp, nullptr, din, 2, -1, n->d_err, n->st);
      if (e != cudaErrorNotSupported) {
        NCK(e);
        return 0;
      }
      cudaGetLastError();
    }
    if (l.Wtb && xtc::conv_box_supported(t)) {
      const cudaError_t e = xtc::conv_forward_box(t, dpre, l.Wtb, nullptr, din, 2, -1, n->d_err, n->st);
      if (e != cudaErrorNotSupported) {
        NCK(e);
        return 0;
      }
      cudaGetLastError();
    }
    NCK(xtc::conv_forward(t, dpre, l.Wt, nullptr, din, 2, -1, n->d_err, n->st));
  }
  return 0;
}

int backward(xtc_net *n, const float *fbp, const float *icd) {
  const int nb = n->nb, Y = n->Y, X = n->X, Z = n->Z;
  cudaStream_t st = n->st;
  bf16 *A[kLayers];
  for (int i = 0; i < kLayers; i++) A[i] = n->a[i].as<bf16>();
  float *g = n->g32.as<float>(), *t = n->gtmp.as<float>();
  float *u0 = n->gcat[0].as<float>(), *u1 = n->gcat[1].as<float>(), *u2 = n->gcat[2].as<float>();
  int rc;
  // decoder, level 0: g = d A13 (from the head)
  if ((rc = conv_back(n, 13, g, A[13], A[12], 0, t))) return rc;                   // t = d A12
  if ((rc = conv_back(n, 12, t, A[12], n->u0.as<bf16>(), 0, u0))) return rc;       // u0 = d (up A11, A1)
  xtc::up_back(nb, Y, X, Z, 48, 32, u0, t, st);                                    // t = d A11
  if ((rc = conv_back(n, 11, t, A[11], A[10], 1, g))) return rc;                   // g = d A10
  if ((rc = conv_back(n, 10, g, A[10], n->u1.as<bf16>(), 1, u1))) return rc;       // u1 = d (up A9, A3)
  xtc::up_back(nb, Y / 2, X / 2, Z / 2, 64, 48, u1, g, st);                        // g = d A9
  if ((rc = conv_back(n, 9, g, A[9], A[8], 2, t))) return rc;                      // t = d A8
  if ((rc = conv_back(n, 8, t, A[8], n->u2.as<bf16>(), 2, u2))) return rc;         // u2 = d (up A7, A5)
  xtc::up_back(nb, Y / 4, X / 4, Z / 4, 96, 64, u2, t, st);                        // t = d A7
  // bottom
  if ((rc = conv_back(n, 7, t, A[7], A[6], 3, g))) return rc;                      // g = d A6
  if ((rc = conv_back(n, 6, g, A[6], n->p2.as<bf16>(), 3, t))) return rc;          // t = d p2
  // encoder, level 2..0: an encoder output's gradient is its skip's and its pooling's
  if ((rc = conv_back(n, 5, u2, A[5], A[4], 2, g, 160, 96, t))) return rc;         // g = d A4
  if ((rc = conv_back(n, 4, g, A[4], n->p1.as<bf16>(), 2, t))) return rc;          // t = d p1
  if ((rc = conv_back(n, 3, u1, A[3], A[2], 1, g, 112, 64, t))) return rc;         // g = d A2
  if ((rc = conv_back(n, 2, g, A[2], n->p0.as<bf16>(), 1, t))) return rc;          // t = d p0
  if ((rc = conv_back(n, 1, u0, A[1], A[0], 0, g, 80, 48, t))) return rc;          // g = d A0
  if ((rc = conv_back(n, 0, g, A[0], nullptr, 0, nullptr, 0, 0, nullptr, fbp, icd))) return rc;
  NCK(cudaGetLastError());
  return 0;
}

int check_dims(int nb, int Y, int X, int Z) {
  if (nb < 1 || Y < 8 || X < 8 || Z < 8 || Y % 8 || X % 8 || Z % 8) {
    xtg_set_error_text("xtc_net: volume dimensions must be positive multiples of 8");
    return XTG_E_ARG;
  }
  return 0;
}

}  // namespace

extern "C" {

int xtc_net_create(uint64_t seed, xtc_net **out) {
  if (!out) return XTG_E_ARG;
  xtc_net *n = new xtc_net();
  size_t off = 0;
  for (int i = 0; i < kLayers; i++) {
    Layer &l = n->L[i];
    l.cin_real = kSpec[i][0];
    l.cin = cin_store(l.cin_real);
    l.cout = kSpec[i][1];
    l.kpad = kpad_of(l.cin);
    l.kpad_t = kpad_of(l.cout);
    l.off_w = off;
    off += (size_t)27 * l.cin_real * l.cout;
    l.off_b = off;
    off += l.cout;
  }
  n->off_hw = off;
  off += kHeadC;
  n->off_hb = off;
  off += 1;
  n->n_params = off;
  std::vector<float> h(off, 0.f);
  uint64_t s = seed;
  for (int i = 0; i < kLayers; i++) {
    const Layer &l = n->L[i];
    const double sd = std::sqrt(2.0 / (27.0 * l.cin_real));  // He initialisation
    for (size_t k = 0; k < (size_t)27 * l.cin_real * l.cout; k++) h[l.off_w + k] = (float)(sd * gauss(s));
  }
  // the head starts at zero: the untrained network returns its ICD input
  cudaError_t e = cudaSuccess;
  auto A = [&](void **p, size_t b) {
    if (e == cudaSuccess) e = cudaMalloc(p, b);
  };
  A((void **)&n->P, off * 4);
  A((void **)&n->G, off * 4);
  A((void **)&n->M, off * 4);
  A((void **)&n->V, off * 4);
  A((void **)&n->d_loss, 8);
  A((void **)&n->d_err, 4);
  for (int i = 0; i < kLayers; i++) {
    Layer &l = n->L[i];
    A((void **)&l.W, (size_t)l.cout * l.kpad * 2);
    if (i) A((void **)&l.Wt, (size_t)l.cin * l.kpad_t * 2);
    if (l.cout <= 64) A((void **)&l.Wp, xtc::conv_tile_wp_elems(l.cin, l.cout) * 2);
    if (i && l.cin <= 64 && l.cin % 16 == 0) A((void **)&l.Wtp, xtc::conv_tile_wp_elems(l.cout, l.cin) * 2);
    if (i) A((void **)&l.Wb, xtc::conv_box_wp_elems(l.cin, l.cout) * 2);
    if (i) A((void **)&l.Wtb, xtc::conv_box_wp_elems(l.cout, l.cin) * 2);
    if (i == 0) A((void **)&l.W64, (size_t)l.cout * 64 * 2);
  }
  if (e == cudaSuccess) e = cudaMemcpy(n->P, h.data(), off * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(n->M, 0, off * 4);
  if (e == cudaSuccess) e = cudaMemset(n->V, 0, off * 4);
  if (e == cudaSuccess) e = cudaMemset(n->G, 0, off * 4);
  if (e == cudaSuccess) e = cudaMemset(n->d_err, 0, 4);
  if (e != cudaSuccess) {
    xtc_net_destroy(n);
    return set_fail("xtc_net_create", e);
  }
  *out = n;
  return 0;
}

void xtc_net_destroy(xtc_net *n) {
  if (!n) return;
  for (float *p : {n->P, n->G, n->M, n->V})
    if (p) cudaFree(p);
  if (n->d_loss) cudaFree(n->d_loss);
  if (n->d_err) cudaFree(n->d_err);
  for (int i = 0; i < kLayers; i++) {
    if (n->L[i].W) cudaFree(n->L[i].W);
    if (n->L[i].Wt) cudaFree(n->L[i].Wt);
    if (n->L[i].Wp) cudaFree(n->L[i].Wp);
    if (n->L[i].Wtp) cudaFree(n->L[i].Wtp);
    if (n->L[i].Wb) cudaFree(n->L[i].Wb);
    if (n->L[i].Wtb) cudaFree(n->L[i].Wtb);
    if (n->L[i].W64) cudaFree(n->L[i].W64);
  }
  delete n;
}

int64_t xtc_net_param_count(const xtc_net *n) { return n ? (int64_t)n->n_params : 0; }

int xtc_net_get_params(const xtc_net *n, float *host, int32_t which) {
  if (!n || !host || which < 0 || which > 1) return XTG_E_ARG;
  NCK(cudaStreamSynchronize(n->st));
  NCK(cudaMemcpy(host, which ? n->G : n->P, n->n_params * 4, cudaMemcpyDeviceToHost));
  return 0;
}

int xtc_net_set_params(xtc_net *n, const float *host) {
  if (!n || !host) return XTG_E_ARG;
  NCK(cudaMemcpy(n->P, host, n->n_params * 4, cudaMemcpyHostToDevice));
  n->packed = false;
  return 0;
}

int xtc_net_save(const xtc_net *n, const char *path) {
  if (!n || !path) return XTG_E_ARG;
  std::vector<float> h(n->n_params);
  int rc = xtc_net_get_params(n, h.data(), 0);
  if (rc) return rc;
  FILE *f = fopen(path, "wb");
  if (!f) {
    xtg_set_error_text("xtc_net_save: cannot open the file");
    return XTG_E_ARG;
  }
  const uint32_t hdr[3] = {0x4E435458u /* "XTCN" */, 1u, (uint32_t)n->n_params};
  const bool ok = fwrite(hdr, 4, 3, f) == 3 && fwrite(h.data(), 4, h.size(), f) == h.size();
  fclose(f);
  if (!ok) {
    xtg_set_error_text("xtc_net_save: short write");
    return XTG_E_ARG;
  }
  return 0;
}

int xtc_net_load(xtc_net *n, const char *path) {
  if (!n || !path) return XTG_E_ARG;
  FILE *f = fopen(path, "rb");
  if (!f) {
    xtg_set_error_text("xtc_net_load: cannot open the file");
    return XTG_E_ARG;
  }
  uint32_t hdr[3];
  std::vector<float> h(n->n_params);
  const bool ok = fread(hdr, 4, 3, f) == 3 && hdr[0] == 0x4E435458u && hdr[1] == 1u && hdr[2] == n->n_params &&
                  fread(h.data(), 4, h.size(), f) == h.size();
  fclose(f);
  if (!ok) {
    xtg_set_error_text("xtc_net_load: not a weight file of this network");
    return XTG_E_ARG;
  }
  return xtc_net_set_params(n, h.data());
}

}  // extern "C"

// a device buffer of at least `floats` FP32 values owned by the network and
// kept until it is destroyed (grown when a larger volume asks for more)
float *xtc_net_start_buffer(xtc_net *n, size_t floats) {
  if (!n || n->start.ensure(floats * sizeof(float)) != cudaSuccess) return nullptr;
  return n->start.as<float>();
}

extern "C" {

int xtc_net_forward(xtc_net *n, const float *fbp, const float *icd, float *out, int32_t nb, int32_t Y, int32_t X,
                    int32_t Z) {
  if (!n || !fbp || !icd || !out) return XTG_E_ARG;
  int rc = check_dims(nb, Y, X, Z);
  if (rc) return rc;
  if ((rc = ensure_buffers(n, nb, Y, X, Z, false))) return rc;
  if (!n->packed && (rc = pack_all(n))) return rc;
  if ((rc = forward(n, fbp, icd, out, nullptr))) return rc;
  return check_err(n);
}

int xtc_net_backward(xtc_net *n, const float *fbp, const float *icd, const float *target, int32_t nb, int32_t Y,
                     int32_t X, int32_t Z, double *loss) {
  if (!n || !fbp || !icd || !target) return XTG_E_ARG;
  int rc = check_dims(nb, Y, X, Z);
  if (rc) return rc;
  if ((rc = ensure_buffers(n, nb, Y, X, Z, true))) return rc;
  if (!n->packed && (rc = pack_all(n))) return rc;
  NCK(cudaMemsetAsync(n->G, 0, n->n_params * 4, n->st));
  if ((rc = forward(n, fbp, icd, nullptr, target))) return rc;
  if ((rc = backward(n, fbp, icd))) return rc;
  if (loss) NCK(cudaMemcpyAsync(loss, n->d_loss, sizeof(double), cudaMemcpyDeviceToHost, n->st));
  return check_err(n);
}

int xtc_net_adam_step(xtc_net *n, float lr) {
  if (!n || !(lr > 0.f)) return XTG_E_ARG;
  n->step++;
  xtc::adam((long long)n->n_params, n->P, n->G, n->M, n->V, lr, 0.9f, 0.999f, 1e-8f, n->step, n->st);
  NCK(cudaGetLastError());
  return pack_all(n);
}

int xtc_net_train(xtc_net *n, const float *const *fbp, const float *const *icd, const float *const *target,
                  int32_t nvol, int32_t Y, int32_t X, int32_t Z, int32_t py, int32_t px, int32_t pz, int32_t batch,
                  int32_t steps, float lr, uint64_t seed, float *losses) {
  if (!n || !fbp || !icd || !target || nvol < 1 || steps < 1 || batch < 1 || py > Y || px > X || pz > Z)
    return XTG_E_ARG;
  int rc = check_dims(batch, py, px, pz);
  if (rc) return rc;
  const size_t pv = (size_t)batch * py * px * pz;
  Buf bf, bi, bt, src, org;
  NCK(bf.ensure(pv * 4));
  NCK(bi.ensure(pv * 4));
  NCK(bt.ensure(pv * 4));
  NCK(src.ensure(3 * (size_t)nvol * sizeof(float *)));
  NCK(org.ensure((size_t)batch * sizeof(int4)));
  std::vector<const float *> hp(3 * (size_t)nvol);
  for (int v = 0; v < nvol; v++) {
    hp[v] = fbp[v];
    hp[nvol + v] = icd[v];
    hp[2 * nvol + v] = target[v];
  }
  NCK(cudaMemcpy(src.p, hp.data(), hp.size() * sizeof(float *), cudaMemcpyHostToDevice));
  const float *const *dsrc = src.as<const float *>();
  uint64_t s = seed;
  std::vector<int4> ho(batch);
  for (int it = 0; it < steps; it++) {
    for (int b = 0; b < batch; b++) {
      ho[b].w = (int)(mix(s) % (uint64_t)nvol);
      ho[b].x = (int)(mix(s) % (uint64_t)(Y - py + 1));
      ho[b].y = (int)(mix(s) % (uint64_t)(X - px + 1));
      ho[b].z = (int)(mix(s) % (uint64_t)(Z - pz + 1));
    }
    NCK(cudaMemcpyAsync(org.p, ho.data(), batch * sizeof(int4), cudaMemcpyHostToDevice, n->st));
    xtc::crop(batch, dsrc, org.as<int4>(), Y, X, Z, py, px, pz, bf.as<float>(), n->st);
    xtc::crop(batch, dsrc + nvol, org.as<int4>(), Y, X, Z, py, px, pz, bi.as<float>(), n->st);
    xtc::crop(batch, dsrc + 2 * nvol, org.as<int4>(), Y, X, Z, py, px, pz, bt.as<float>(), n->st);
    double loss = 0;
    if ((rc = xtc_net_backward(n, bf.as<float>(), bi.as<float>(), bt.as<float>(), batch, py, px, pz, &loss))) return rc;
    if ((rc = xtc_net_adam_step(n, lr))) return rc;
    if (losses) losses[it] = (float)loss;
  }
  NCK(cudaStreamSynchronize(n->st));
  return 0;
}

}  // extern "C"
