// xtg_proj.cu -- forward projection and the A-matrix column table.
//
// Forward projection (initErrorSinogam + forward_project_voxel_AMat1D,
// Source_Code_4D_Fast/XT_ICD_update.c:551-569, XT_ForwardProject.c:8-25) as a
// gather: one warp per (view, 32 detector bins, 64 detector rows), partial
// sums in shared memory owned by that warp.  The warp walks image rows in
// increasing order and, within a row, the columns that can reach its bins in
// increasing order, so every sinogram entry is summed in the reference's
// (row, column) order: the FP32 result is bit-identical to the reference's,
// and FP64 accumulation gives the resync / MAP-cost data term.
//
// A-matrix column table (calcAMatrixColumnforAngle, XT_AMatrix.c:50-110,
// for every masked column and every view of its frame, stored once): CSC
// form, per (frame, column) a run of entries {offset (p*N_r + bin)*N_t,
// A*delta_t} in view order, FP32 or FP16 with one FP32 scale per column.
// The ICD kernel streams these runs instead of recomputing A per visit.
#include <cuda_fp16.h>

#include "xtg_internal.h"

namespace xtg {

// candidate columns of row yv for bin window [lo, hi] of r_col (conservative)
__device__ __forceinline__ bool fp_col_range(const DevGeo &G, float cp, float sp, float yv, double lo, double hi,
                                             int *klo, int *khi) {
  const double ys = (double)yv * (double)sp;
  if (fabs((double)cp) < 1e-12) {
    if (-ys >= lo && -ys <= hi) {
      *klo = 0;
      *khi = G.N_x - 1;
      return true;
    }
    return false;
  }
  double xa = (lo + ys) / (double)cp, xb = (hi + ys) / (double)cp;
  if (xa > xb) {
    const double t = xa;
    xa = xb;
    xb = t;
  }
  const double ka = (xa - (double)G.x0) / (double)G.delta_xy - 0.5;
  const double kb = (xb - (double)G.x0) / (double)G.delta_xy - 0.5;
  if (kb < -4.0 || ka > (double)G.N_x + 4.0) return false;
  *klo = max(0, (int)floor(ka) - 2);
  *khi = min(G.N_x - 1, (int)ceil(kb) + 2);
  return *klo <= *khi;
}

// MODE 0: out = A x; 1: out = e = y - A x - d (FP32, the reference's order
// and its projector, which leaves out delta_t, XT_ForwardProject.c:17);
// 2: FP64 sums, out = (float)(y - delta_t A x - d), data cost into cost slots;
// 3: FP64 data cost only.  Modes 2 and 3 use A * delta_t, the matrix the
// voxel update subtracts from e (XT_VoxUpdate.c:27, 67): the error sinogram
// the reference carries from its zero start; with delta_t = 1 all modes agree.
// Warp w of the CTA owns 32 consecutive detector bins of view p and keeps
// their partial sums for 64 detector rows in shared memory (lane owns rows
// lane and lane + 32, so the shared accesses are free of bank conflicts).  For each image row (in increasing order) the warp
// evaluates, one column per lane, the exact A entries of the columns that can
// reach its bins, then walks those columns in increasing order: one
// coalesced z-line load per column, and each of the column's entries that
// falls on the warp's bins is added with a plain shared-memory read-add-write
// (the warp owns those sums, so no atomics).  Control flow is uniform within
// the warp.
template <int MODE, typename ACC, int NS>
__global__ void __launch_bounds__(FP_WARPS * 32) k_fp_bins(DevGeo G, FpArgs F) {
  extern __shared__ __align__(16) unsigned char fp_sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ACC *acc = reinterpret_cast<ACC *>(fp_sm) + (size_t)warp * 32 * 64;  // [32 bins][64 rows]
  // the A entries of the warp's 32 candidate columns, [lane][NS]
  float *vsm = reinterpret_cast<float *>(fp_sm + (size_t)FP_WARPS * 32 * 64 * sizeof(ACC)) + (size_t)warp * 32 * NS;
  const int p = F.order ? F.order[blockIdx.x] : (int)blockIdx.x;
  const int rb = (blockIdx.y * FP_WARPS + warp) * 32;
  const int t0 = blockIdx.z * 64, nt = min(64, G.N_t - t0);
  if (rb >= G.N_r) return;  // whole warp; no block-wide barrier follows
#pragma unroll 4
  for (int b = 0; b < 32; b++) {
    acc[b * 64 + lane] = (ACC)0;
    acc[b * 64 + lane + 32] = (ACC)0;
  }
  __syncwarp();
  const int fr = F.fov[p];
  const float cp = F.cosv[p], sp = F.sinv[p];
  const float *H = F.hr + (size_t)p * XT_HR_STRIDE;
  const double lo = (double)G.R0 + (double)rb * G.delta_r - G.delta_xy - F.win_margin;
  const double hi = (double)G.R0 + (double)(rb + 32) * G.delta_r + G.delta_xy + F.win_margin;
  const int ta = lane, tb = lane + 32;  // this lane's rows (relative to t0)
  // slices of those rows (detector row t belongs to slice t / zovl)
  const bool va = ta < nt, vb = tb < nt;
  const int za = (t0 + ta) / G.zovl, zb2 = (t0 + tb) / G.zovl;
  for (int j = 0; j < G.N_y; j++) {
    int klo, khi;
    if (!fp_col_range(G, cp, sp, xt_coord(G.y0, j, G.delta_xy), lo, hi, &klo, &khi)) continue;
    const float *xrow = F.x + ((size_t)fr * G.N_y + j) * G.N_x * G.N_z;
    for (int kb = klo; kb <= khi; kb += 32) {
      const int k = kb + lane;
      float v[NS];
#pragma unroll
      for (int s = 0; s < NS; s++) v[s] = 0.f;
      int first = 0, n = 0;
      if (k <= khi) n = xt_amatrix_regs<NS>(G, H, cp, sp, j, k, v, &first);
      // entries of this lane's column that land on the warp's bins
      const int slo = max(0, rb - first), shi = min(n, rb + 32 - first);
      const unsigned hit = __ballot_sync(0xffffffffu, slo < shi);
      if (!hit) continue;
      // each column's entries go to shared memory, its (first - rb, slo, shi)
      // into one word, so a hit column costs one shuffle and its entries that
      // land on the warp's bins are read by a loop over exactly those
#pragma unroll
      for (int s = 0; s < NS; s++) vsm[lane * NS + s] = v[s];
      // for a hit column first - rb lies in (-NS, 32), so the +64 keeps it positive
      const int pk = (int)(((unsigned)(first - rb + 64) << 16) | ((unsigned)slo << 8) | (unsigned)shi);
      __syncwarp();
      unsigned mk = hit;
      // the z-line of the next hit column is loaded while the current one is added
      float xa = 0.f, xb = 0.f;
      {
        const float *xp = xrow + (size_t)(kb + __ffs(mk) - 1) * G.N_z;
        xa = va ? __ldg(xp + za) : 0.f;
        xb = vb ? __ldg(xp + zb2) : 0.f;
      }
      while (mk) {
        const int l = __ffs(mk) - 1;
        mk &= mk - 1;
        const int q = __shfl_sync(0xffffffffu, pk, l);
        const int sl = (q >> 8) & 0xFF, sh = q & 0xFF;
        const float ca = xa, cb = xb;
        if (mk) {
          const float *xp = xrow + (size_t)(kb + __ffs(mk) - 1) * G.N_z;
          xa = va ? __ldg(xp + za) : 0.f;
          xb = vb ? __ldg(xp + zb2) : 0.f;
        }
        ACC *qa = acc + ((q >> 16) - 64 + sl) * 64;
        const float *vl = vsm + l * NS;
        for (int s = sl; s < sh; s++, qa += 64) {
          const float a = vl[s];
          if (a != 0.f) {
            if (MODE <= 1) {
              qa[ta] = __fadd_rn(qa[ta], __fmul_rn(ca, a));
              qa[tb] = __fadd_rn(qa[tb], __fmul_rn(cb, a));
            } else {
              qa[ta] += (ACC)ca * (ACC)a;
              qa[tb] += (ACC)cb * (ACC)a;
            }
          }
        }
      }
      __syncwarp();  // the staged entries are rewritten by the next round
    }
  }
  __syncwarp();
  double cacc = 0.0;
  for (int b = 0; b < 32; b++) {
    const int r = rb + b;
    if (r >= G.N_r) break;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int t = lane + 32 * h;
      if (t >= nt) continue;
      const ACC sacc = acc[b * 64 + t];
      const size_t o = ((size_t)p * G.N_r + r) * G.N_t + t0 + t;
      const size_t od = (size_t)r * G.N_t + t0 + t;
      if (MODE == 0) {
        F.out[o] = (float)sacc;
      } else if (MODE == 1) {
        F.out[o] = __fsub_rn(__fsub_rn(F.y[o], (float)sacc), F.d[od]);
      } else {
        // A * delta_t: the system matrix of the voxel update (XT_VoxUpdate.c:27, 67)
        const double e64 = (double)F.y[o] - (double)G.delta_t * (double)sacc - (double)F.d[od];
        if (MODE == 2) F.out[o] = (float)e64;
        const double sw = e64 * sqrt((double)F.w[o]);
        if (fabs(sw) < (double)F.T)
          cacc += sw * sw;
        else
          cacc += 2.0 * (double)F.delta * (double)F.T * fabs(sw) + (double)F.T * (double)F.T * (1.0 - 2.0 * (double)F.delta);
      }
    }
  }
  if (MODE >= 2) {
    for (int off = 16; off > 0; off >>= 1) cacc += __shfl_xor_sync(0xffffffffu, cacc, off);
    if (lane == 0) atomicAdd(&F.cost_slots[(blockIdx.x * 5 + blockIdx.y * 3 + blockIdx.z + warp) % 64], cacc);
  }
}

template <int MODE, typename ACC>
static cudaError_t launch_fp_t(const DevGeo &G, const FpArgs &F, int ns, cudaStream_t st) {
  const int nsv = ns <= 3 ? 3 : ns <= 4 ? 4 : 12;
  const size_t smem = (size_t)FP_WARPS * 32 * 64 * sizeof(ACC) + (size_t)FP_WARPS * 32 * nsv * sizeof(float);
  dim3 grid((unsigned)(F.order ? F.nviews : G.N_p), (unsigned)((G.N_r + FP_WARPS * 32 - 1) / (FP_WARPS * 32)),
            (unsigned)((G.N_t + 63) / 64));
  typedef void (*K)(DevGeo, FpArgs);
  K k = ns <= 3 ? k_fp_bins<MODE, ACC, 3> : ns <= 4 ? k_fp_bins<MODE, ACC, 4> : k_fp_bins<MODE, ACC, 12>;
  cudaError_t e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<grid, FP_WARPS * 32, smem, st>>>(G, F);
  return cudaGetLastError();
}

cudaError_t launch_fp(const DevGeo &G, const FpArgs &F, int mode, int ns, cudaStream_t st) {
  switch (mode) {
    case 0: return launch_fp_t<0, float>(G, F, ns, st);
    case 1: return launch_fp_t<1, float>(G, F, ns, st);
    case 2: return launch_fp_t<2, double>(G, F, ns, st);
    default: return launch_fp_t<3, double>(G, F, ns, st);
  }
}

// ------------------------------------------------ bin-major A table ------
// The A entries regrouped by sinogram row pair (view p, detector bins 2 i and
// 2 i + 1): a row lists {column j N_x + k, its A at each of the two bins} for
// every column of p's frame that reaches either, in increasing (j, k) -- the
// order in which the reference adds a column's contribution to those entries
// (initErrorSinogam, XT_ICD_update.c:551-569).  A column reaches 2.14 bins on
// average at voxels one bin wide, so 1.57 records stand for 2.14 entries, and
// the z-line a record names is loaded once for both bins.  Built once per
// context by the enumeration of k_fp_bins, so every value is the exact A of
// calcAMatrixColumnforAngle (XT_AMatrix.c:50-110).  Lane b of a warp owns bin
// rb + b of the warp's 32 bins: for each hit column the lanes test their own
// bin in parallel, so the appends of a pair (its even lane's) stay in column
// order without atomics.
template <int FILL, int NS>
__global__ void __launch_bounds__(FP_WARPS * 32) k_csr_build(DevGeo G, CsrBuildArgs B) {
  extern __shared__ __align__(16) unsigned char cb_sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float *vsm = reinterpret_cast<float *>(cb_sm) + (size_t)warp * 32 * NS;
  const int p = B.order[blockIdx.x];
  const int rb = (blockIdx.y * FP_WARPS + warp) * 32;
  if (rb >= G.N_r) return;  // whole warp; no block-wide barrier follows
  const float cp = B.cosv[p], sp = B.sinv[p];
  const float *H = B.hr + (size_t)p * XT_HR_STRIDE;
  const double lo = (double)G.R0 + (double)rb * G.delta_r - G.delta_xy - B.win_margin;
  const double hi = (double)G.R0 + (double)(rb + 32) * G.delta_r + G.delta_xy + B.win_margin;
  const int r = rb + lane, np2 = (G.N_r + 1) / 2;
  const bool own = r < G.N_r, head = own && !(lane & 1);
  const size_t row = (size_t)p * np2 + r / 2;
  long long cur = 0;
  int cnt = 0, ent = 0;
  if (FILL && head) cur = B.ptr[row];
  for (int j = 0; j < G.N_y; j++) {
    int klo, khi;
    if (!fp_col_range(G, cp, sp, xt_coord(G.y0, j, G.delta_xy), lo, hi, &klo, &khi)) continue;
    for (int kb = klo; kb <= khi; kb += 32) {
      const int k = kb + lane;
      float v[NS];
#pragma unroll
      for (int q = 0; q < NS; q++) v[q] = 0.f;
      int first = 0, n = 0;
      if (k <= khi) n = xt_amatrix_regs<NS>(G, H, cp, sp, j, k, v, &first);
      const int slo = max(0, rb - first), shi = min(n, rb + 32 - first);
      const unsigned hit = __ballot_sync(0xffffffffu, slo < shi);
      if (!hit) continue;
#pragma unroll
      for (int q = 0; q < NS; q++) vsm[lane * NS + q] = v[q];
      const int pk = (int)(((unsigned)(first - rb + 64) << 16) | ((unsigned)slo << 8) | (unsigned)shi);
      __syncwarp();
      unsigned mk = hit;
      while (mk) {
        const int l = __ffs(mk) - 1;
        mk &= mk - 1;
        const int q = __shfl_sync(0xffffffffu, pk, l);
        const int sl = (q >> 8) & 0xFF, sh = q & 0xFF;
        const int sidx = lane - ((q >> 16) - 64);  // this lane's bin within the column's run
        float a = 0.f;
        if (own && sidx >= sl && sidx < sh) a = vsm[l * NS + sidx];
        const float a1 = __shfl_down_sync(0xffffffffu, a, 1);
        ent += a != 0.f;
        if (head && (a != 0.f || a1 != 0.f)) {
          if (FILL) {
            B.off[cur] = (j * G.N_x + kb + l) * G.N_z;
            B.val[cur++] = make_float2(a, a1);
          } else {
            cnt++;
          }
        }
      }
      __syncwarp();  // the staged entries are rewritten by the next round
    }
  }
  if (FILL && head)
    for (; cur < B.ptr[row + 1]; cur++) {  // up to a multiple of 4 records: A = 0 at column 0
      B.off[cur] = 0;
      B.val[cur] = make_float2(0.f, 0.f);
    }
  if (!FILL) {
    if (head) B.count[row] = cnt;
    for (int off = 16; off > 0; off >>= 1) ent += __shfl_xor_sync(0xffffffffu, ent, off);
    if (lane == 0) atomicAdd(&B.entries[p], (unsigned long long)ent);
  }
}

template <int FILL>
static cudaError_t launch_csr_build_t(const DevGeo &G, const CsrBuildArgs &B, int ns, cudaStream_t st) {
  const int nsv = ns <= 3 ? 3 : ns <= 4 ? 4 : 12;
  const size_t smem = (size_t)FP_WARPS * 32 * nsv * sizeof(float);
  dim3 grid((unsigned)B.nviews, (unsigned)((G.N_r + FP_WARPS * 32 - 1) / (FP_WARPS * 32)));
  if (ns <= 3)
    k_csr_build<FILL, 3><<<grid, FP_WARPS * 32, smem, st>>>(G, B);
  else if (ns <= 4)
    k_csr_build<FILL, 4><<<grid, FP_WARPS * 32, smem, st>>>(G, B);
  else
    k_csr_build<FILL, 12><<<grid, FP_WARPS * 32, smem, st>>>(G, B);
  return cudaGetLastError();
}

cudaError_t launch_csr_build(const DevGeo &G, const CsrBuildArgs &B, int fill, int ns, cudaStream_t st) {
  return fill ? launch_csr_build_t<1>(G, B, ns, st) : launch_csr_build_t<0>(G, B, ns, st);
}

// Forward projection from the bin-major table.  LT lanes, four detector rows
// each, take one (view, bin pair) and 4 LT rows, and accumulate both bins in
// registers, records in table order: in FP32 (__fadd_rn(__fmul_rn)) that is
// the reference's summation order, so MODE 0 / 1 are bit-identical to
// k_fp_bins and to initErrorSinogam; MODE 2 / 3 accumulate in FP64 in the same
// order (a product of two FP32 values is exact in FP64, so the sums equal
// k_fp_bins' bit for bit).  A bin that a record's column does not reach (A = 0)
// is passed over, so no value of that column touches it.  VEC: a z-line's four
// rows are one 16-byte load (one detector row per slice, N_z a multiple of 4).
//
// What bounds it: L1, which returns 64-128 bytes of z-line a cycle, and in
// FP64 the conversions to it (16 lanes a cycle; A is converted by integer
// operations instead, being positive and normal).  Per bin, a warp over the 64
// rows loaded 2.14 z-lines a (column, view), here 1.57; a CTA takes the same
// bins of CSR_WARPS views that follow each other in angle (T.order), whose
// rays cross the same columns at the same time, so most z-lines are L1 hits
// (eight bins of one view before).  Latency: with records read as they are
// needed the pairs alone were no faster (9.3 ms).  512^2 x 64, 1024 views: e = y -
// A x - d 9.6 -> 6.3 ms, FP64 cost 12.8 -> 8.0 ms; 256^2 x 32, 512 views 1.46 ->
// 0.53 ms.
// (s0, s1) += (x0, x1) a, product and sum each rounded, two rows per
// instruction.  The product is a multiply-add of -0, which leaves it as it is
// (neg0 is an argument so that nothing knows its value): with a packed multiply
// and a packed add the sums had one rounding a term and not the reference's bits,
// as k_fp_bins shows them.
__device__ __forceinline__ void mul_add2(float &s0, float &s1, float x0, float x1, float a, float neg0) {
  asm("{\n\t.reg .b64 x, a, s, z;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 a, {%4, %4};\n\tmov.b64 s, {%0, %1};\n\tmov.b64 z, {%5, %5};\n\t"
      "fma.rn.f32x2 x, x, a, z;\n\tadd.rn.f32x2 s, s, x;\n\tmov.b64 {%0, %1}, s;\n\t}"
      : "+f"(s0), "+f"(s1)
      : "f"(x0), "f"(x1), "f"(a), "f"(neg0));
}

#define CSR_WARPS 8  // consecutive views of a CTA, one per warp
// resident CTAs the FP32 registers are cut for (3 and 5: 6.8 and 6.7 ms)
#define CSR_CTAS 4
template <int MODE, typename ACC, int LT, int R, bool VEC>
__global__ void __launch_bounds__(CSR_WARPS * 32, MODE < 2 ? CSR_CTAS : 3) k_fp_csr(DevGeo G, FpArgs F, CsrView T) {
  constexpr int PW = 32 / LT;  // pairs per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LT;
  const int ov = blockIdx.x * CSR_WARPS + warp, np2 = (G.N_r + 1) / 2, pair = blockIdx.y * PW + lane / LT;
  if (ov >= T.nviews) return;  // whole warp; no block-wide barrier follows
  const int p = T.order[ov];
  const int t0 = blockIdx.z * (R * LT) + R * sub;  // this lane's first row
  const int nt = min(R, G.N_t - t0);               // rows it has (may be none)
  const float *xf = F.x + (size_t)F.fov[p] * G.N_y * G.N_x * G.N_z;
  const float *xl = xf + (VEC ? (nt > 0 ? t0 : 0) : 0);
  int zr[R];
#pragma unroll
  for (int c = 0; c < R; c++) zr[c] = c < nt ? (t0 + c) / G.zovl : 0;
  long long i = 0, e1 = 0;
  if (pair < np2) {  // (lanes without rows load records too)
    i = T.ptr[(size_t)p * np2 + pair];
    e1 = T.ptr[(size_t)p * np2 + pair + 1];
  }
  ACC acc0[R], acc1[R];
#pragma unroll
  for (int c = 0; c < R; c++) acc0[c] = acc1[c] = (ACC)0;
  struct Rows {
    float x[R];
  };
  auto load = [&](int off) {
    Rows v;
    if constexpr (VEC) {
      const float4 q = __ldg(reinterpret_cast<const float4 *>(xl + off));
      v.x[0] = q.x;
      v.x[R / 4] = q.y;
      v.x[R / 2] = q.z;
      v.x[R - 1] = q.w;
    } else {
#pragma unroll
      for (int c = 0; c < R; c++) v.x[c] = __ldg(xl + off + zr[c]);
    }
    return v;
  };
  auto add1 = [&](ACC (&acc)[R], const ACC (&x)[R], float a) {
    if constexpr (MODE <= 1 && R == 1) {
      acc[0] = __fadd_rn(acc[0], __fmul_rn(x[0], a));
    } else if constexpr (MODE <= 1) {
#pragma unroll
      for (int c = 0; c + 1 < R; c += 2) mul_add2(acc[c], acc[c + 1], x[c], x[c + 1], a, F.neg0);
    } else {
      const uint32_t u = __float_as_uint(a);  // FP64 form of a positive normal: a shift and a bias
      const double ad = __hiloint2double((int)((u >> 3) + 0x38000000u), (int)(u << 29));
#pragma unroll
      for (int c = 0; c < R; c++) acc[c] += x[c] * ad;
    }
  };
  auto add = [&](const Rows &v, float a0, float a1) {
    ACC x[R];
#pragma unroll
    for (int c = 0; c < R; c++) x[c] = (ACC)v.x[c];
    if (a0 != 0.f) add1(acc0, x, a0);
    if (a1 != 0.f) add1(acc1, x, a1);
  };
  // Sixteen records of each pair at a time: its lanes load them in one coalesced
  // run while the sixteen before are added, and read them back from shared
  // memory; z-lines are loaded four records ahead.  (Records past the row's
  // end: A = 0 at column 0.)  Offsets and values lie in arrays of their own, 12
  // bytes a record, a row at a multiple of four records: with four a lane they are
  // one 16-byte and one 32-byte load (16-byte records {offset, two values, 0} against
  // that: 256^2 x 16 x 8 frames 0.44 -> 0.41 ms, 512^2 x 8 2.71 -> 2.51, 512^2 x 64 6.33 ->
  // 6.30; 200^2 x 5 0.227 -> 0.243).
  constexpr int RC = 16, RL = (RC + LT - 1) / LT;  // records a lane loads
  __shared__ __align__(16) int4 recs[CSR_WARPS][2][PW][RC + 1];
  const int len = (int)(e1 - i), most = __reduce_max_sync(0xffffffffu, len);
  int nxo[RL];
  float2 nxv[RL];
  auto fetch = [&](int r0) {
    if constexpr (RL == 4) {  // four in a row
      const int r = r0 + sub * RL;
      int4 q = make_int4(0, 0, 0, 0);
      float2 a = make_float2(0.f, 0.f), b = a, c = a, d = a;
      if (r < len) {
        q = __ldcs(reinterpret_cast<const int4 *>(T.off + i + r));
        asm volatile("ld.global.cs.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(a.x), "=f"(a.y), "=f"(b.x), "=f"(b.y), "=f"(c.x), "=f"(c.y), "=f"(d.x), "=f"(d.y)
                     : "l"(T.val + i + r));
      }
      nxo[0] = q.x; nxo[RL / 4] = q.y; nxo[RL / 2] = q.z; nxo[RL - 1] = q.w;
      nxv[0] = a; nxv[RL / 4] = b; nxv[RL / 2] = c; nxv[RL - 1] = d;
    } else {
#pragma unroll
      for (int m = 0; m < RL; m++) {
        const int r = r0 + sub + m * LT;
        const bool in = r < len && (LT <= RC || sub < RC);
        nxo[m] = in ? __ldcs(T.off + i + r) : 0;
        nxv[m] = in ? __ldcs(T.val + i + r) : make_float2(0.f, 0.f);
      }
    }
  };
  fetch(0);
  for (int r0 = 0, buf = 0; r0 < most; r0 += RC, buf ^= 1) {
    int4 *rec = recs[warp][buf][lane / LT];
#pragma unroll
    for (int m = 0; m < RL; m++)
      if (LT <= RC || sub < RC) rec[RL == 4 ? sub * RL + m : sub + m * LT] = make_int4(nxo[m], __float_as_int(nxv[m].x), __float_as_int(nxv[m].y), 0);
    __syncwarp();  // (the other buffer was read before the last one's barrier)
    fetch(r0 + RC);
    Rows v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = load(rec[u].x);
#pragma unroll
    for (int g = 0; g < RC; g += 4) {
      Rows vn[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (g + 4 < RC) vn[u] = load(rec[g + 4 + u].x);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        add(v[u], __int_as_float(rec[g + u].y), __int_as_float(rec[g + u].z));
      }
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = vn[u];
    }
  }
  double cacc = 0.0;
  if (pair < np2) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = 2 * pair + h;
      if (r >= G.N_r) continue;
#pragma unroll
      for (int c = 0; c < R; c++) {
        if (c >= nt) continue;
        const ACC sacc = h ? acc1[c] : acc0[c];
        const size_t o = ((size_t)p * G.N_r + r) * G.N_t + t0 + c;
        const size_t od = (size_t)r * G.N_t + t0 + c;
        if (MODE == 0) {
          F.out[o] = (float)sacc;
        } else if (MODE == 1) {
          F.out[o] = __fsub_rn(__fsub_rn(F.y[o], (float)sacc), F.d[od]);
        } else {
          // A * delta_t: the system matrix of the voxel update (XT_VoxUpdate.c:27, 67)
          const double e64 = (double)F.y[o] - (double)G.delta_t * (double)sacc - (double)F.d[od];
          if (MODE == 2) F.out[o] = (float)e64;
          const double sw = e64 * sqrt((double)F.w[o]);
          if (fabs(sw) < (double)F.T)
            cacc += sw * sw;
          else
            cacc += 2.0 * (double)F.delta * (double)F.T * fabs(sw) + (double)F.T * (double)F.T * (1.0 - 2.0 * (double)F.delta);
        }
      }
    }
  }
  if (MODE >= 2) {
    __syncwarp();
    for (int off = 16; off > 0; off >>= 1) cacc += __shfl_xor_sync(0xffffffffu, cacc, off);
    if (lane == 0) atomicAdd(&F.cost_slots[(blockIdx.x * 7 + blockIdx.y + warp + blockIdx.z) % 64], cacc);
  }
}

template <int LT, int R, bool VEC>
static void launch_fp_csr_t(const DevGeo &G, const FpArgs &F, const CsrView &T, int mode, cudaStream_t st) {
  const int np2 = (G.N_r + 1) / 2, pw = 32 / LT;
  const dim3 grid((unsigned)((T.nviews + CSR_WARPS - 1) / CSR_WARPS), (unsigned)((np2 + pw - 1) / pw),
                  (unsigned)((G.N_t + R * LT - 1) / (R * LT)));
  switch (mode) {
    case 0: k_fp_csr<0, float, LT, R, VEC><<<grid, CSR_WARPS * 32, 0, st>>>(G, F, T); break;
    case 1: k_fp_csr<1, float, LT, R, VEC><<<grid, CSR_WARPS * 32, 0, st>>>(G, F, T); break;
    case 2: k_fp_csr<2, double, LT, R, VEC><<<grid, CSR_WARPS * 32, 0, st>>>(G, F, T); break;
    default: k_fp_csr<3, double, LT, R, VEC><<<grid, CSR_WARPS * 32, 0, st>>>(G, F, T); break;
  }
}

cudaError_t launch_fp_csr(const DevGeo &G, const FpArgs &F, const CsrView &T, int mode, cudaStream_t st) {
  // one 16-byte load for four rows where rows and slices are the same and
  // z-lines keep 16-byte alignment; lanes per pair: as many as the rows fill
  const bool vec = G.zovl == 1 && G.N_z % 4 == 0;
  // Else fewer rows a lane and more lanes a pair, where loads and conversions
  // row by row are what a warp waits for.  One row up to 16 (FP64 cost, four rows
  // a lane against one: 100^2 x 5, 128 views 214 -> 118 us; 400^2 x 13, 600 views 3.64
  // -> 2.09 ms; FP32 FBP start there 3.56 -> 3.18), two in FP64 above that, in
  // tiles of 64 rows where they leave no more empty than tiles of 32 (256^2 x 31,
  // 512 views: four rows 1.73 ms, one 1.36, two 1.13; 300^2 x 62, 300 views 2.67, 2.35,
  // 1.90).  In FP32 four rows stay the faster there (300^2 x 62: 2.84 against 3.12).
  if (!vec && (mode >= 2 || G.N_t <= 16)) {
    if (G.N_t <= 4)
      launch_fp_csr_t<4, 1, false>(G, F, T, mode, st);
    else if (G.N_t <= 8)
      launch_fp_csr_t<8, 1, false>(G, F, T, mode, st);
    else if (G.N_t <= 16)
      launch_fp_csr_t<16, 1, false>(G, F, T, mode, st);
    else if ((G.N_t + 63) / 64 * 2 == (G.N_t + 31) / 32)
      launch_fp_csr_t<32, 2, false>(G, F, T, mode, st);
    else
      launch_fp_csr_t<16, 2, false>(G, F, T, mode, st);
  } else if (G.N_t <= 16) {
    vec ? launch_fp_csr_t<4, 4, true>(G, F, T, mode, st) : launch_fp_csr_t<4, 4, false>(G, F, T, mode, st);
  } else if (G.N_t <= 32) {
    vec ? launch_fp_csr_t<8, 4, true>(G, F, T, mode, st) : launch_fp_csr_t<8, 4, false>(G, F, T, mode, st);
  } else {
    vec ? launch_fp_csr_t<16, 4, true>(G, F, T, mode, st) : launch_fp_csr_t<16, 4, false>(G, F, T, mode, st);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------- A column table --
// entries of (frame f, masked column ci): one warp, lanes over views
template <int NS>
__global__ void k_table_count(DevGeo G, TableArgs T, long long *count) {
  const int lane = threadIdx.x & 31;
  const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (gw >= (long long)G.N_time * T.n_masked) return;
  const int f = (int)(gw / T.n_masked), c = T.mcols[gw % T.n_masked];
  const int row = c / G.N_x, col = c % G.N_x, V = T.view_num[f], vs = T.view_start[f];
  int n = 0;
  for (int v = lane; v < V; v += 32) {
    const int p = T.view_idx[vs + v];
    float vals[NS];
    int first;
    n += xt_amatrix_regs<NS>(G, T.hr + (size_t)p * XT_HR_STRIDE, T.cosv[p], T.sinv[p], row, col, vals, &first);
  }
  for (int off = 16; off > 0; off >>= 1) n += __shfl_xor_sync(0xffffffffu, n, off);
  if (lane == 0) count[gw] = n;
}

template <int NS>
__global__ void k_table_fill(DevGeo G, TableArgs T) {
  const int lane = threadIdx.x & 31;
  const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (gw >= (long long)G.N_time * T.n_masked) return;
  const int f = (int)(gw / T.n_masked), c = T.mcols[gw % T.n_masked];
  const int row = c / G.N_x, col = c % G.N_x, V = T.view_num[f], vs = T.view_start[f];
  float mx = 0.f;
  if (T.val16) {
    for (int v = lane; v < V; v += 32) {
      const int p = T.view_idx[vs + v];
      float vals[NS];
      int first;
      const int n = xt_amatrix_regs<NS>(G, T.hr + (size_t)p * XT_HR_STRIDE, T.cosv[p], T.sinv[p], row, col, vals, &first);
#pragma unroll
      for (int s = 0; s < NS; s++)
        if (s < n) mx = fmaxf(mx, __fmul_rn(vals[s], G.delta_t));
    }
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  const float sc = mx > 0.f ? mx : 1.f;
  if (T.val16 && lane == 0) T.scale[gw] = sc;
  long long pos = T.start[gw];
  for (int v0 = 0; v0 < V; v0 += 32) {
    const int v = v0 + lane;
    float vals[NS];
    int first = 0, n = 0;
    if (v < V) {
      const int p = T.view_idx[vs + v];
      n = xt_amatrix_regs<NS>(G, T.hr + (size_t)p * XT_HR_STRIDE, T.cosv[p], T.sinv[p], row, col, vals, &first);
      first = (int)(((long long)p * G.N_r + first) * G.N_t);  // offset of the first entry's rows
    }
    int incl = n;  // inclusive prefix of n over the warp keeps the view order
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += y;
    }
    const long long my = pos + incl - n;
#pragma unroll
    for (int s = 0; s < NS; s++) {
      if (s < n) {
        T.off[my + s] = first + s * G.N_t;
        const float a = __fmul_rn(vals[s], G.delta_t);
        if (T.val16)
          T.val16[my + s] = __float2half_rn(a / sc);
        else
          T.val32[my + s] = a;
      }
    }
    pos += __shfl_sync(0xffffffffu, incl, 31);
  }
}

cudaError_t launch_table_count(const DevGeo &G, const TableArgs &T, int ns, long long *count, cudaStream_t st) {
  const long long warps = (long long)G.N_time * T.n_masked;
  const unsigned grid = (unsigned)((warps + 7) / 8);
  if (ns <= 3)
    k_table_count<3><<<grid, 256, 0, st>>>(G, T, count);
  else if (ns <= 4)
    k_table_count<4><<<grid, 256, 0, st>>>(G, T, count);
  else
    k_table_count<12><<<grid, 256, 0, st>>>(G, T, count);
  return cudaGetLastError();
}

cudaError_t launch_table_fill(const DevGeo &G, const TableArgs &T, int ns, cudaStream_t st) {
  const long long warps = (long long)G.N_time * T.n_masked;
  const unsigned grid = (unsigned)((warps + 7) / 8);
  if (ns <= 3)
    k_table_fill<3><<<grid, 256, 0, st>>>(G, T);
  else if (ns <= 4)
    k_table_fill<4><<<grid, 256, 0, st>>>(G, T);
  else
    k_table_fill<12><<<grid, 256, 0, st>>>(G, T);
  return cudaGetLastError();
}

}  // namespace xtg
