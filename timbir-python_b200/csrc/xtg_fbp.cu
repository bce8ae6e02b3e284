// xtg_fbp.cu -- filtered backprojection start for ICD.
//
// The reference starts ICD from a zero object (initObject, XT_ICD_update.c:
// 454-458) or from a coarser stage; its launchers compute FBP images with
// scikit-image outside the engine (4D_Recon_Launcher_for_Real_Data/
// XT_FBP_Reconstruction.py).  This is the parallel-beam FBP of Kak & Slaney
// (Principles of Computerized Tomographic Imaging, ch. 3, eqs. 61-63) on the
// engine's own geometry, used as a warm start:
//   q_p(r_k, t) = dr * sum_n h(k - n) (y[p][n][t] - d[n][t]),
//     h(0) = 1 / (4 dr^2), h(m odd) = -1 / (m^2 pi^2 dr^2), h(m even) = 0;
//   x(j, k, z) = (pi / V_f) sum_{views p of the frame} q_p(x cos th - y sin th, t)
// with linear interpolation between bin centres R0 + (i + 0.5) dr and the
// zovl detector rows of slice z averaged.  Columns outside the reconstruction
// disk get 0; with positivity the image is clamped at 0.
#include <algorithm>

#include "xtg_internal.h"

namespace xtg {

// The zovl detector rows of a slice are summed as the filter reads them (both
// steps are linear), so the filtered sinogram holds one value per slice,
// [N_p][N_r][N_z].

// Ramp filter: one CTA per (view, TT slices), the view's rows in shared memory.
// h is zero at even distances, so an output of one parity reads the inputs of
// the other and itself.  A thread forms RQ outputs two bins apart for two
// slices: per input one 8-byte load, one tap (the taps of its RQ outputs are a
// window that moves by one per input) and RQ packed multiply-adds.  Bound by
// FP32 issue; with one output and two loads per tap pair (shared memory) the
// filter of 512 bins x 64 rows x 1024 views took 3.3 ms, now 0.55.
constexpr int RQ = 8;

template <int TT>
__global__ void __launch_bounds__(256) k_ramp(DevGeo G, const float *__restrict__ y, const float *__restrict__ d,
                                              float *__restrict__ q) {
  extern __shared__ __align__(16) float fbp_sm[];
  constexpr int LZ = TT / 2;                   // lanes over slice pairs
  float *s = fbp_sm;                           // [N_r][TT]
  float *h = fbp_sm + (size_t)G.N_r * TT;      // h[|m|], odd |m| < N_r, index |m| / 2
  const int p = blockIdx.x, z0 = blockIdx.y * TT, nz = min(TT, G.N_z - z0);
  const double dr = (double)G.delta_r;
  for (int i = threadIdx.x; i < G.N_r * TT; i += blockDim.x) {
    const int r = i / TT, zz = i - r * TT;
    float v = 0.f;
    if (zz < nz)
      for (int o = 0; o < G.zovl; o++) {
        const int t = (z0 + zz) * G.zovl + o;
        v += y[((size_t)p * G.N_r + r) * G.N_t + t] - (d ? d[(size_t)r * G.N_t + t] : 0.f);
      }
    s[i] = v;
  }
  for (int m = 2 * threadIdx.x + 1; m < G.N_r; m += 2 * blockDim.x)
    h[m / 2] = (float)(-1.0 / ((double)m * m * M_PI * M_PI * dr * dr));
  __syncthreads();
  const int zl = threadIdx.x % LZ, grp = threadIdx.x / LZ;
  constexpr int NG = 256 / LZ;
  const float h0 = (float)(1.0 / (4.0 * dr * dr)), drf = (float)dr;
  const int nblk = (G.N_r + 2 * RQ - 1) / (2 * RQ);  // blocks of 2 RQ bins, both parities
  for (int b = grp; b < 2 * nblk; b += NG) {
    const int par = b & 1, r0 = (b >> 1) * 2 * RQ + par;  // outputs r0, r0 + 2, ..., r0 + 2 (RQ - 1)
    float2 acc[RQ], hw[RQ];
    const int n0 = par ^ 1;                               // the other parity's first bin
    auto tap = [&](int m) {                               // h at distance m (odd); 0 past the table
      const int am = m < 0 ? -m : m;
      const float v = am < G.N_r ? h[am >> 1] : 0.f;
      return make_float2(v, v);
    };
#pragma unroll
    for (int u = 0; u < RQ; u++) {
      const int r = r0 + 2 * u;
      const float2 sv = r < G.N_r ? *reinterpret_cast<const float2 *>(s + r * TT + 2 * zl) : make_float2(0.f, 0.f);
      acc[u] = make_float2(h0 * sv.x, h0 * sv.y);
    }
    // hw[(u + k) % RQ] holds the tap of output u at the loop's k-th input
#pragma unroll
    for (int u = 1; u < RQ; u++) hw[u] = tap(n0 - 2 - (r0 + 2 * (u - 1)));
    int n = n0;
    for (; n + 2 * (RQ - 1) < G.N_r; n += 2 * RQ) {
#pragma unroll
      for (int k = 0; k < RQ; k++) {
        // the window moves: output u takes output u - 1's previous tap
        hw[(RQ - k) % RQ] = tap(n + 2 * k - r0);
        const float2 sv = *reinterpret_cast<const float2 *>(s + (n + 2 * k) * TT + 2 * zl);
#pragma unroll
        for (int u = 0; u < RQ; u++) acc[u] = __ffma2_rn(hw[(u + RQ - k) % RQ], sv, acc[u]);
      }
    }
    for (; n < G.N_r; n += 2) {
      const float2 sv = *reinterpret_cast<const float2 *>(s + n * TT + 2 * zl);
#pragma unroll
      for (int u = 0; u < RQ; u++) acc[u] = __ffma2_rn(tap(n - r0 - 2 * u), sv, acc[u]);
    }
#pragma unroll
    for (int u = 0; u < RQ; u++) {
      const int r = r0 + 2 * u;
      if (r >= G.N_r) continue;
      float *o = q + ((size_t)p * G.N_r + r) * G.N_z + z0 + 2 * zl;
      if (2 * zl < nz) o[0] = drf * acc[u].x;
      if (2 * zl + 1 < nz) o[1] = drf * acc[u].y;
    }
  }
}

// Backprojection.  A CTA owns 16 columns along x by 8 * 32 / LT rows along y and
// 4 LT slices; LT lanes (four slices each) walk the 16 columns of one row with
// their sums in registers.  Per view the filtered bins the tile can reach are
// staged in shared memory (asynchronous copies, BP_STAGES views ahead, zero
// outside the detector).  Along a row the bin moves by |cos| voxel widths, so
// consecutive columns share bins: the two rows interpolated stay in registers
// and a column that moved on loads one.  Lanes compute the bin and weight of
// one (row, column) each and hand them round through shared memory.  Bound by
// shared-memory reads and issue; with both bins of every (column, view) read
// from L1 by a warp per column 512^2 x 64, 1024 views took 33 ms, now 6.4.
constexpr int BP_C = 16;       // columns of a strip
constexpr int BP_STAGES = 4;
// CTAs wanted, in fills of the GPU (6: 7.4 ms at 512^2 x 64, its tiles of 8 rows
// stage more bins per column; 1 and 3 keep 16 rows there, 6.4)
constexpr int BP_WAVES = 3;

__device__ __forceinline__ void fbp_cp16(uint32_t s, const void *g, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fbp_cp4(uint32_t s, const void *g, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}

template <int LT>
__global__ void __launch_bounds__(256, 2) k_backproject(DevGeo G, const float *__restrict__ q,
                                                        const float *__restrict__ cosv, const float *__restrict__ sinv,
                                                        const int *__restrict__ view_idx,
                                                        const int *__restrict__ view_start,
                                                        const int *__restrict__ view_num,
                                                        const int *__restrict__ col_rank, float *__restrict__ x, int rb,
                                                        int vsplit) {
  constexpr int SPW = 32 / LT;                 // strips (image rows) per warp
  const int NS = 8 * SPW / vsplit;             // per CTA
  constexpr int TZ = 4 * LT;                   // slices
  constexpr int EPL = SPW * BP_C / 32;         // (strip, column) entries a lane computes
  extern __shared__ __align__(16) float bp_sm[];
  float *sq = bp_sm;                           // [BP_STAGES][vsplit][rb][TZ]
  __shared__ __align__(16) float4 sw[8][SPW][BP_C + 1];  // near weight twice, far weight twice
  __shared__ int si[8][SPW][BP_C];                       // first bin, relative to the staged ones
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k0 = blockIdx.x * BP_C, j0 = blockIdx.y * NS;
  const int nch = (G.N_z + TZ - 1) / TZ;
  const int fr = blockIdx.z / nch, z0 = (blockIdx.z - fr * nch) * TZ;
  const int V = view_num[fr], vs = view_start[fr];
  // vsplit warps share the rows of warp group wg, each every vsplit-th view
  const int wg = warp / vsplit, wv = warp - wg * vsplit;
  // a tile outside the object-support disk is 0 (512^2 x 64, 1024 views, a whole
  // start: disk of half the width 12.2 ms, of a quarter 8.7; 13.3 when every tile was
  // summed)
  bool used = false;
  for (int i = tid; i < NS * BP_C; i += 256) {
    const int j = j0 + i / BP_C, k = k0 + i % BP_C;
    used = used || (j < G.N_y && k < G.N_x && col_rank[(size_t)j * G.N_x + k] >= 0);
  }
  if (!__syncthreads_or(used)) {  // uniform over the CTA
    const int nz = min(TZ, G.N_z - z0);
    for (int i = tid; i < NS * BP_C * TZ; i += 256) {
      const int zz = i % TZ, j = j0 + i / (TZ * BP_C), k = k0 + i / TZ % BP_C;
      if (zz < nz && j < G.N_y && k < G.N_x) x[(((size_t)fr * G.N_y + j) * G.N_x + k) * G.N_z + z0 + zz] = 0.f;
    }
    return;
  }
  // the lane's own strip and slices
  const int sl = lane / LT, tl = lane % LT;
  // the entries it computes: column lane % 16 of strips 2 m + lane / 16
  const float xc = xt_coord(G.x0, k0 + (lane & 15), G.delta_xy);
  float yc[EPL];
#pragma unroll
  for (int m = 0; m < EPL; m++) yc[m] = xt_coord(G.y0, j0 + wg * SPW + 2 * m + (lane >> 4), G.delta_xy);
  // the tile's centre and half extents, for the bins it can reach
  const float xm = G.x0 + ((float)k0 + 0.5f * BP_C) * G.delta_xy, ym = G.y0 + ((float)j0 + 0.5f * NS) * G.delta_xy;
  const float hx = 0.5f * (BP_C - 1) * G.delta_xy, hy = 0.5f * (NS - 1) * G.delta_xy;
  auto first_bin = [&](float cp, float sp) {
    const float r = xm * cp - ym * sp - (hx * fabsf(cp) + hy * fabsf(sp));
    return (int)floorf((r - G.R0) / G.delta_r - 0.5f) - 1;
  };
  const bool al = (G.N_z & 3) == 0;
  auto stage = [&](int st) {
    for (int w = 0; w < vsplit; w++) {
      const int v = st * vsplit + w;
      if (v >= V) break;
      const int p = view_idx[vs + v];
      const int lo = first_bin(cosv[p], sinv[p]);
      float *d = sq + (size_t)((st % BP_STAGES) * vsplit + w) * rb * TZ;
      for (int i = tid; i < rb * LT; i += 256) {
        const int r = i / LT, zz = (i - r * LT) * 4, bin = lo + r;
        const bool in = bin >= 0 && bin < G.N_r;
        const int nz = in ? min(4, G.N_z - z0 - zz) : 0;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(d + r * TZ + zz);
        const float *src = nz > 0 ? q + ((size_t)p * G.N_r + bin) * G.N_z + z0 + zz : q;
        if (al) {
          fbp_cp16(dst, src, nz > 0 ? 16 : 0);
        } else {
#pragma unroll
          for (int c = 0; c < 4; c++) fbp_cp4(dst + 4 * c, c < nz ? src + c : q, c < nz ? 4 : 0);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 acc[BP_C][2];
#pragma unroll
  for (int c = 0; c < BP_C; c++) acc[c][0] = acc[c][1] = make_float2(0.f, 0.f);
  const int steps = (V + vsplit - 1) / vsplit;
  for (int st = 0; st < BP_STAGES - 1; st++) stage(st);
  for (int st = 0; st < steps; st++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(BP_STAGES - 2) : "memory");
    __syncthreads();  // step st has landed for every thread; step st - 1's stage is free
    stage(st + BP_STAGES - 1);
    const int v = st * vsplit + wv;
    if (v >= V) continue;  // uniform over the warp; the next step's barrier is met by all
    const int p = view_idx[vs + v];
    const float cp = cosv[p], sp = sinv[p];
    const int lo = first_bin(cp, sp), dir = cp >= 0.f ? 1 : -1;
    unsigned moved = 0, jumped = 0;
#pragma unroll
    for (int m = 0; m < EPL; m++) {
      const float r = xc * cp - yc[m] * sp;
      const float u = (r - G.R0) / G.delta_r - 0.5f;
      const float fl = floorf(u);
      const float f = u - fl;
      const int il = min(max((int)fl - lo, 0), rb - 2);
      const int prev = __shfl_up_sync(0xffffffffu, il, 1, 16);
      const int step = (lane & 15) ? (il - prev) * dir : 0;
      const unsigned mv = __ballot_sync(0xffffffffu, step == 1), jp = __ballot_sync(0xffffffffu, step != 0 && step != 1);
      jumped |= jp;
      if (sl >> 1 == m) moved = (mv >> ((sl & 1) * 16)) & 0xffffu;
      const float wn = dir > 0 ? 1.f - f : f, wf = dir > 0 ? f : 1.f - f;
      sw[warp][2 * m + (lane >> 4)][lane & 15] = make_float4(wn, wn, wf, wf);
      si[warp][2 * m + (lane >> 4)][lane & 15] = il;
    }
    __syncwarp();
    const float *base = sq + (size_t)((st % BP_STAGES) * vsplit + wv) * rb * TZ + 4 * tl;
    const float4 *wp = &sw[warp][sl][0];
    float4 nr = make_float4(0.f, 0.f, 0.f, 0.f), fa = nr;
    auto add = [&](int c) {
      const float4 w = wp[c];
      const float2 wn = make_float2(w.x, w.y), wf = make_float2(w.z, w.w);
      acc[c][0] = __ffma2_rn(wn, make_float2(nr.x, nr.y), acc[c][0]);
      acc[c][1] = __ffma2_rn(wn, make_float2(nr.z, nr.w), acc[c][1]);
      acc[c][0] = __ffma2_rn(wf, make_float2(fa.x, fa.y), acc[c][0]);
      acc[c][1] = __ffma2_rn(wf, make_float2(fa.z, fa.w), acc[c][1]);
    };
    if (!jumped) {  // uniform over the warp
      const float *pt = base + (si[warp][sl][0] + (dir > 0 ? 0 : 1)) * TZ;
      nr = *reinterpret_cast<const float4 *>(pt);
      pt += dir * TZ;
      fa = *reinterpret_cast<const float4 *>(pt);
#pragma unroll
      for (int c = 0; c < BP_C; c++) {
        if (c && ((moved >> c) & 1u)) {
          nr = fa;
          pt += dir * TZ;
          fa = *reinterpret_cast<const float4 *>(pt);
        }
        add(c);
      }
    } else {  // voxels wider than a bin
#pragma unroll
      for (int c = 0; c < BP_C; c++) {
        const float *pt = base + (si[warp][sl][c] + (dir > 0 ? 0 : 1)) * TZ;
        nr = *reinterpret_cast<const float4 *>(pt);
        fa = *reinterpret_cast<const float4 *>(pt + dir * TZ);
        add(c);
      }
    }
    __syncwarp();  // the weights are rewritten for the next view
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // the sums of the warps that shared rows, halves onto halves
  float2 *sr = reinterpret_cast<float2 *>(bp_sm);  // [4 warps][2 BP_C][32]
  for (int h = vsplit >> 1; h > 0; h >>= 1) {
    float2 *slot = sr + (size_t)(wg * h + wv % h) * 2 * BP_C * 32 + lane;
    if (wv >= h && wv < 2 * h) {
#pragma unroll
      for (int c = 0; c < BP_C; c++) {
        slot[(2 * c) * 32] = acc[c][0];
        slot[(2 * c + 1) * 32] = acc[c][1];
      }
    }
    __syncthreads();
    if (wv < h) {
#pragma unroll
      for (int c = 0; c < BP_C; c++) {
        acc[c][0] = __fadd2_rn(acc[c][0], slot[(2 * c) * 32]);
        acc[c][1] = __fadd2_rn(acc[c][1], slot[(2 * c + 1) * 32]);
      }
    }
    __syncthreads();
  }
  const int j = j0 + wg * SPW + sl, z = z0 + 4 * tl;
  if (wv != 0 || j >= G.N_y || z >= G.N_z) return;
  const float scale = (float)(M_PI / (double)V) / (float)G.zovl;
#pragma unroll
  for (int c = 0; c < BP_C; c++) {
    const int k = k0 + c;
    if (k >= G.N_x) break;
    const bool in = col_rank[(size_t)j * G.N_x + k] >= 0;
    float o[4] = {acc[c][0].x, acc[c][0].y, acc[c][1].x, acc[c][1].y};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      o[i] = in ? o[i] * scale : 0.f;
      if (G.positivity && o[i] < 0.f) o[i] = 0.f;
    }
    float *xz = x + (((size_t)fr * G.N_y + j) * G.N_x + k) * G.N_z + z;
    if (al) {
      *reinterpret_cast<float4 *>(xz) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (z + i < G.N_z) xz[i] = o[i];
    }
  }
}

template <int TT>
static cudaError_t launch_ramp(const DevGeo &G, const float *y, const float *d, float *q, cudaStream_t st) {
  const size_t smem = ((size_t)G.N_r * TT + (size_t)(G.N_r / 2 + 1)) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute((const void *)k_ramp<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_ramp<TT><<<dim3((unsigned)G.N_p, (unsigned)((G.N_z + TT - 1) / TT)), 256, smem, st>>>(G, y, d, q);
  return cudaGetLastError();
}

template <int LT>
static cudaError_t launch_bp(const DevGeo &G, const float *q, const float *cosv, const float *sinv, const int *view_idx,
                             const int *view_start, const int *view_num, const int *col_rank, float *x, cudaStream_t st) {
  constexpr int TZ = 4 * LT;
  struct Tile {
    dim3 grid;
    int rb;
    size_t smem;
  };
  auto tile = [&](int vsplit) {
    const int ns = 8 * 32 / LT / vsplit;
    Tile t;
    t.grid = dim3((unsigned)((G.N_x + BP_C - 1) / BP_C), (unsigned)((G.N_y + ns - 1) / ns),
                  (unsigned)(G.N_time * ((G.N_z + TZ - 1) / TZ)));
    // bins across the tile at the worst angle, one more on each side for
    // rounding and the second bin of an interpolation
    const double diag = sqrt((double)(BP_C - 1) * (BP_C - 1) + (double)(ns - 1) * (ns - 1));
    t.rb = (int)ceil(diag * G.delta_xy / G.delta_r) + 5;
    const size_t red = vsplit > 1 ? (size_t)4 * 2 * BP_C * 32 * sizeof(float2) : 0;
    t.smem = std::max(red, (size_t)BP_STAGES * vsplit * t.rb * TZ * sizeof(float));
    return t;
  };
  // warps per group of rows: more of them (smaller tiles, more CTAs) until the
  // GPU is filled BP_WAVES times over, two CTAs per SM
  int vsplit = 1;
  Tile t = tile(1);
  while (vsplit < 8 && (long long)t.grid.x * t.grid.y * t.grid.z < BP_WAVES * 2 * 148 && tile(2 * vsplit).smem <= 100 * 1024) {
    vsplit *= 2;
    t = tile(vsplit);
  }
  cudaError_t e = cudaFuncSetAttribute((const void *)k_backproject<LT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)t.smem);
  if (e != cudaSuccess) return e;
  k_backproject<LT><<<t.grid, 256, t.smem, st>>>(G, q, cosv, sinv, view_idx, view_start, view_num, col_rank, x, t.rb, vsplit);
  return cudaGetLastError();
}

cudaError_t launch_fbp(const DevGeo &G, const float *y, const float *d, float *q, const float *cosv,
                       const float *sinv, const int *view_idx, const int *view_start, const int *view_num,
                       const int *col_rank, float *x, cudaStream_t st) {
  cudaError_t e = G.N_z <= 8 ? launch_ramp<8>(G, y, d, q, st) : launch_ramp<32>(G, y, d, q, st);
  if (e != cudaSuccess) return e;
  // lanes per image row: as many as the slices fill
  if (G.N_z <= 16) return launch_bp<4>(G, q, cosv, sinv, view_idx, view_start, view_num, col_rank, x, st);
  if (G.N_z <= 32) return launch_bp<8>(G, q, cosv, sinv, view_idx, view_start, view_num, col_rank, x, st);
  return launch_bp<16>(G, q, cosv, sinv, view_idx, view_start, view_num, col_rank, x, st);
}

}  // namespace xtg
