// xtg_icd.cu -- the ICD column kernel: one CTA updates one x-y column's
// z-line (or one z-block of it) of one time frame.
//
// Parallel-beam A is z-invariant: every slice of a column sees the same
// (view, bin) entries, and the rows of slice z are t = z*zovl .. z*zovl+zovl-1.
// So the CTA puts the column's A into shared memory once (computed in
// registers, or read from the FP16 table), then streams the column's
// footprint e[p][bin][t0..t0+T) and w[...] (contiguous in t) with 16-byte
// loads, thread (view group, t lane) accumulating theta1/theta2 for its rows;
// shuffles reduce them over view groups inside a warp.  The qGGMRF surrogate
// sums over the neighbours that the visit does not change are formed by all
// threads before the footprint is read; then one warp adds the theta partials
// and takes the slices' steps in red/black z order, a lane per voxel (or
// strictly in increasing z on one thread, the reference's order, in
// sequential mode), while another fetches the next item's record, and the e
// update goes back with vector red.global.add, so columns in flight that
// share sinogram entries never lose an update.
//
// What bounds it.  Short items: the fixed chain of an item.  With the whole
// surrogate step between two barriers, per-phase barriers and block-wide
// statistics a 16-row item of 137 entries took 35,000 cycles, 11,000 of them
// in that step; with four barriers and the split above 19,000 (4D 256^2 x 16 x
// 16: 24.8 -> 19.4 ms an iteration, 128^2 x 4: 2.67 -> 2.40 ms).  Long ones:
// the L2, which serves 9 TB/s of e and w plus the reductions in the footprint
// loop of plain 3D (117.5 -> 115.6 ms).
//
// Reference: updateVoxels_Aditya + compute_voxel_update_Aditya
// (Source_Code_4D_Fast/XT_VoxUpdate.c:11-254), CE_FunctionalSubstitution
// (XT_ICD_update.c:130-179); the z-line batching follows updateVoxels_AttTomo
// (XT_VoxUpdate.c:266-586).
#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "xtg_internal.h"

namespace xtg {

// Threads per CTA.  An item's row groups (16 bytes of e and of w of one
// footprint entry) are dealt to the CTA's threads, so small items want small
// CTAs (the fixed work of an item -- neighbourhood, A staging, barriers, the
// surrogate step -- then overlaps over more items at once) and long items, or
// few columns in flight, want large ones.  icd_threads takes the largest size
// that keeps the columns in flight resident, down to
// XTG_GROUPS_PER_THREAD row groups a thread, below which a larger CTA no
// longer helps to fill the SMs.
#define XTG_GROUPS_PER_THREAD 8
#define XTG_NT_MIN 64
#define XTG_NT_MAX 1024

// Footprint loads with L2 cache hints: e (re-read and updated through L2 by
// other columns' reductions) is kept (evict_last), w (read once per visit) is
// evicted first; neither is allocated in L1.
__device__ __forceinline__ float4 ld_e(const float *p) {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  float4 v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float4 ld_w(const float *p, bool keep) {
  uint64_t pol;
  if (keep)  // e and w fit in L2 together: keep w as well
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  else
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  float4 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p), "l"(pol));
  return v;
}

// Asynchronous global -> shared copies (no registers held while in flight);
// cp_wait_all completes the calling thread's copies and makes them visible to it.
__device__ __forceinline__ uint32_t icd_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async4(void *s, const void *g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(icd_smem(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A work item and where its column run lies in the A column table, fetched
// for the next item while the current one is processed.
struct ItemMeta {
  int4 item;           // frame, row, column, z-block
  long long s0, s1;    // tstart[ti], tstart[ti + 1]
  float sc;            // tscale[ti] (FP16 table)
  int it;              // launch-wide item index (>= the launch's total: none)
};

// Packed FP32 (two lanes per instruction, sm_100) for the footprint
// arithmetic of 16-byte rows
#ifndef XTG_F32X2
#define XTG_F32X2 1
#endif

// Footprint entries a thread loads before it uses any of them (table modes,
// 16-byte rows): more loads in flight per warp to cover L2/HBM latency.
// Three measured equal in the 256-thread CTAs (a few bytes spilled) and 1 %
// slower in the 64-thread ones, which keep two whatever this is set to.
#ifndef XTG_UNROLL
#define XTG_UNROLL 2
#endif

// sigma_q times the surrogate coefficient rho'(d) / d of the qGGMRF prior with
// q = 2 (CE_QGGMRF, XT_ICD_update.c:79-125): with t = |d|^(2-p) / sigma_qp it is
// (2 - (2-p) t / (c+t)) / (c+t) = (2c + p t) / (c+t)^2, one reciprocal; t comes
// from the special-function unit's log2 and 2^x (lq = log2 sigma_qp).  The log2 of a
// subnormal d, flushed to -inf, is taken as that of the smallest one: with p = 2
// (e2p = 0) its product would be NaN.  The step size only needs a few digits, the
// fixed point of the iteration is unchanged.
__device__ __forceinline__ float qcoef(float d, float c, float lq, float e2p, float p) {
  const float ad = fabsf(d);
  float l, t;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(ad));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(e2p, fmaxf(l, -149.f), -lq)));
  t = ad == 0.f ? 0.f : t;
  const float r = __fdividef(1.0f, c + t);
  return fmaf(p, t, 2.0f * c) * r * r;
}

// Every CTA size keeps 1024 threads resident per SM (64 registers a thread;
// 1280, 48 registers with spills, measured 8 % slower on plain 3D).
template <int VEC, int AMODE, int SEQ, int AS, int NT = XTG_THREADS>
__global__ void __launch_bounds__(NT, 1024 / NT) k_icd_columns(DevGeo G, IcdArgs A, int vmax, int zmax) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NW = NT / 32;
  unsigned char *smem = smem_raw;
  // AMODE 0 (A computed here): per view {first | n << 24, view index, AS values}
  int *sPack = reinterpret_cast<int *>(smem);            // [vmax]
  int *sView = sPack + vmax;                              // [vmax]
  float *sVal = reinterpret_cast<float *>(sView + vmax);  // [AS][vmax] A * delta_t
  // AMODE 1/2 (column table): the column's entry run, vmax = longest run,
  // {(p*N_r + bin)*N_t, bits of A * delta_t} per entry (one 8-byte load)
  int2 *sEnt = reinterpret_cast<int2 *>(smem);           // [vmax]
  const int rowsmax = zmax * G.zovl, rp = (rowsmax + 3) & ~3;
  float *sRed = (AMODE == 0) ? sVal + (size_t)vmax * AS : reinterpret_cast<float *>(sEnt + vmax);  // [2][NW][rp]
  float *sNb = sRed + 2 * NW * rp;                        // [9][zmax+2]
  float *sTn = sNb + 9 * (zmax + 2);                      // [2][zmax]
  float *sDelta = sTn + 2 * zmax;                         // [zmax]
  float *sNum = sDelta + zmax;                            // [zmax] sum of b * neighbour, then
  float *sDen = sNum + zmax;                              // [zmax] sum of b, over the slots outside the column
  int *sPos = reinterpret_cast<int *>(sDen + zmax);       // [zmax] one of those neighbours is positive

  __shared__ float sW[28];                  // filter weight / sigma_q: 27 spatial slots, temporal
  __shared__ double sAbs[32];               // statistics of warp 0's lanes over the CTA's items
  __shared__ unsigned sUpd[32], sZero[32];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nitems = A.n_items_dev ? min(*A.n_items_dev, A.n_items) : A.n_items;
  const bool hlo = A.halo_lo != nullptr, hhi = A.halo_hi != nullptr;
  const int total = nitems * A.nsub;
  // The first lane of the last warp fetches the next item's record and table
  // run (a chain of four dependent reads) while warp 0 does the current
  // item's surrogate step.  Items are taken A.grab at a time and the CTA's
  // statistics are flushed once at the end: with tens of thousands of items
  // per launch, per-item atomics on the same few addresses would queue at L2.
  constexpr int META = NT - 32;
  __shared__ __align__(16) ItemMeta sMeta[2];
  int mb = 0;  // sMeta[mb]: the current item; sMeta[mb ^ 1]: the next
  __shared__ int sGrab[2];  // the batch taken last: next item, items left
  auto item_index = [&](int i) -> int {
    const int ii = A.nsub == 1 ? i : i % nitems;
    return A.item_lo + (A.use_perm ? (int)xt_perm((uint32_t)ii, (uint32_t)nitems, A.perm_key) : ii);
  };
  auto fetch_meta = [&](ItemMeta &N) {  // thread META only
    if (sGrab[1] == 0) {
      sGrab[0] = atomicAdd(A.counter, A.grab);
      sGrab[1] = A.grab;
    }
    N.it = sGrab[0]++;
    sGrab[1]--;
    if (N.it >= total) return;
    const int4 q = A.items[item_index(N.it)];
    N.item = q;
    if (AMODE != 0) {
      const long long ti = (long long)q.x * A.n_masked + A.col_rank[q.y * G.N_x + q.z];
      N.s0 = A.tstart[ti];
      N.s1 = A.tstart[ti + 1];
      N.sc = (AMODE == 1) ? A.tscale[ti] : 1.f;
    }
  };
  if (tid == META) {
    sGrab[1] = 0;
    fetch_meta(sMeta[0]);
  }
  if (warp == 0) {
    sAbs[lane] = 0.0;
    sUpd[lane] = 0u;
    sZero[lane] = 0u;
    if (lane < 27) sW[lane] = G.SF[lane] * A.inv_sq;
    if (lane == 27) sW[27] = G.TF * A.inv_tq;
  }
  unsigned ncol = 0;  // items whose first piece this CTA took

  for (;; mb ^= 1) {
    __syncthreads();  // the item's record is in place, the previous item is done with shared memory
    const int it = sMeta[mb].it;
    if (it >= total) break;
    const int piece = A.nsub == 1 ? 0 : it / nitems;
    const int4 item = sMeta[mb].item;
    const int fr = item.x, row = item.y, col = item.z, blk = item.w;
    int zb = 0, ze = G.N_z - 1;
    if (blk >= 0) {
      zb = blk * G.zstep;
      ze = (blk >= G.nzb - 1) ? G.N_z - 1 : (blk + 1) * G.zstep - 1;
    }
    zb += piece * A.zslab;
    if (zb > ze) {  // this item has fewer pieces (uniform over the CTA)
      if (tid == META) fetch_meta(sMeta[mb ^ 1]);
      continue;
    }
    if (piece == 0) ncol++;
    ze = min(ze, zb + A.zslab - 1);
    const int Z = ze - zb + 1, T = Z * G.zovl, t0 = zb * G.zovl;

    // 1. the column's table run (times delta_t, XT_VoxUpdate.c:27) goes to
    //    shared memory asynchronously, so that its round trip overlaps the
    //    neighbourhood's; a quiet line (below) has fetched it for nothing
    const long long s0 = AMODE != 0 ? sMeta[mb].s0 : 0;
    const int ne = AMODE != 0 ? (int)(sMeta[mb].s1 - s0) : 0;
    if (AMODE != 0) {
      for (int e = tid; e < ne; e += NT) {
        cp_async4(&sEnt[e].x, A.toff + s0 + e);
        if (AMODE == 2) cp_async4(&sEnt[e].y, A.tval32 + s0 + e);
      }
    }
    // the neighbourhood: the 3x3 columns' z-lines over [zb-1, ze+1], and the
    // same column in frames fr-1 and fr+1 (0 outside the volume; slices -1
    // and N_z from the neighbouring slabs' halo planes when present, as the
    // reference's ranks read Object[i][0] / [N_z+1], XT_VoxUpdate.c:94-99)
    const size_t plane = (size_t)G.N_y * G.N_x;
    // Zero skipping (XT_VoxUpdate.c:208-232) decided for the whole z-line
    // before any footprint work: from the second iteration a voxel equal to 0
    // with no positive spatial or temporal neighbour is not updated.  When
    // that holds for every voxel of the item, theta is never used, so the
    // footprint is not read.  Each thread tests
    // the values it stages.
    bool quiet = A.iter > 1;
    // k / (Z + 2) as (k * mz2) >> 20: exact while k (Z + 2) < 2^20, and here
    // k < 9 (Z + 2) with Z + 2 <= 130
    const uint32_t z2 = (uint32_t)Z + 2u, mz2 = ((1u << 20) + z2 - 1u) / z2;
    for (int k = tid; k < 9 * (Z + 2); k += NT) {
      const int c = (int)(((uint32_t)k * mz2) >> 20), zz = k - c * (Z + 2);
      const int jj = row + c / 3 - 1, kk = col + c % 3 - 1, za = zb - 1 + zz;
      float v = 0.f;
      if (jj >= 0 && jj < G.N_y && kk >= 0 && kk < G.N_x) {
        const size_t q = (size_t)fr * plane + (size_t)jj * G.N_x + kk;
        if (za >= 0 && za < G.N_z)
          v = A.x[q * G.N_z + za];
        else if (za < 0 && hlo)
          v = A.halo_lo[q];
        else if (za >= G.N_z && hhi)
          v = A.halo_hi[q];
      }
      sNb[c * (zmax + 2) + zz] = v;
      const bool self = (c == 4) && zz >= 1 && zz <= Z;
      if (self ? (v != 0.f) : (v > 0.f)) quiet = false;
    }
    for (int k = tid; k < 2 * Z; k += NT) {
      const int s = k >= Z ? 1 : 0, z = k - s * Z, f2 = fr + (s ? 1 : -1);
      float v = 0.f;
      if (f2 >= 0 && f2 < G.N_time) v = A.x[(((size_t)f2 * plane) + (size_t)row * G.N_x + col) * G.N_z + zb + z];
      sTn[s * zmax + z] = v;
      if (v > 0.f) quiet = false;
    }
    if (AMODE == 1) {
      const float sc = sMeta[mb].sc;
      for (int e = tid; e < ne; e += NT) sEnt[e].y = __float_as_int(__half2float(A.tval16[s0 + e]) * sc);
    }
    if (AMODE != 0) cp_wait_all();
    const bool skip_all = __syncthreads_and(quiet) != 0;
    // MagUpdateMap[frame][block][row][col] = sum |delta| over the block's
    // slices of this visit (XT_VoxUpdate.c:128, 236), lanes of one warp over blocks
    auto write_magmap = [&]() {
      for (int b = lane; b < G.nzb; b += 32) {
        const int bz0 = b * G.zstep, bz1 = (b >= G.nzb - 1) ? G.N_z - 1 : (b + 1) * G.zstep - 1;
        const int lo = max(bz0, zb), hi = min(bz1, ze);
        if (lo > hi) continue;
        float m = 0.f;
        if (!skip_all)
          for (int z = lo; z <= hi; z++) m += fabsf(sDelta[z - zb]);
        float *mp = A.magmap + (((size_t)fr * G.nzb + b) * G.N_y + row) * G.N_x + col;
        if (A.nsub > 1)
          atomicAdd(mp, m);  // pieces of one block add into the entry zeroed before the launch
        else if (bz0 >= zb && bz1 <= ze)
          *mp = m;
      }
    };
    if (skip_all) {  // uniform over the CTA
      if (tid == 0) sZero[0] += (unsigned)Z;
      if (tid == META) fetch_meta(sMeta[mb ^ 1]);
      if (warp == NW - 1) write_magmap();
      continue;
    }
    int V = 0;
    if (AMODE == 0) {
      const int vs = A.view_start[fr];
      V = A.view_num[fr];
      for (int v = tid; v < V; v += NT) {
        const int p = A.view_idx[vs + v];
        float vals[AS];
        int first;
        const int n = xt_amatrix_regs<AS>(G, A.hr + (size_t)p * XT_HR_STRIDE, A.cosv[p], A.sinv[p], row, col, vals,
                                          &first);
        sPack[v] = first | (n << 24);
        sView[v] = p;
#pragma unroll
        for (int s = 0; s < AS; s++) sVal[s * vmax + v] = __fmul_rn(vals[s], G.delta_t);
      }
      __syncthreads();
    }

    // 2. the surrogate sums over the slots that this visit does not change:
    //    8 neighbouring columns x 3 slices and the two frames, 1 << lv lanes
    //    per voxel (as many as the CTA's threads give).  Out of the update
    //    step below, whose two passes every other warp waits for, they took it
    //    from a third of a short item's time to a tenth.
    const uint32_t cm = (col > 0 ? 0111u : 0u) | 0222u | (col + 1 < G.N_x ? 0444u : 0u);
    const uint32_t colmask = ((row > 0 ? 0007u : 0u) | 0070u | (row + 1 < G.N_y ? 0700u : 0u)) & cm;
    if (!SEQ) {
      int lv = 0;
      while (lv < 5 && (Z << (lv + 1)) <= NT) lv++;
      const int sub = tid & ((1 << lv) - 1);
      for (int z0 = 0; z0 < Z; z0 += NT >> lv) {
        const int z = z0 + (tid >> lv);
        float num = 0.f, den = 0.f;
        int pos = 0;
        if (z < Z) {
          const float Vv = sNb[4 * (zmax + 2) + z + 1];
          const int za = zb + z;
          const uint32_t zm = (za > 0 || hlo ? 1u : 0u) | 2u | (za + 1 < G.N_z || hhi ? 4u : 0u);
          for (int n = sub; n < 26; n += 1 << lv) {
            float v, w, c, lq;
            bool in;
            if (n < 24) {
              const int dz = n >> 3, cc = (n & 7) + ((n & 4) >> 2);
              v = sNb[cc * (zmax + 2) + z + dz];
              w = sW[dz * 9 + cc];
              in = ((colmask >> cc) & (zm >> dz) & 1u) != 0u;
              c = G.C_S;
              lq = A.l_sqp;
            } else {
              v = sTn[(n - 24) * zmax + z];
              w = sW[27];
              in = n == 24 ? fr > 0 : fr + 1 < G.N_time;
              c = G.C_T;
              lq = A.l_tqp;
            }
            const float b = in ? w * qcoef(Vv - v, c, lq, A.e2p, G.MRF_P) : 0.f;
            num = fmaf(b, v, num);
            den += b;
            pos |= v > 0.f;  // absent slots read 0
          }
        }
        for (int off = 1; off < (1 << lv); off <<= 1) {
          num += __shfl_xor_sync(0xffffffffu, num, off);
          den += __shfl_xor_sync(0xffffffffu, den, off);
          pos |= __shfl_xor_sync(0xffffffffu, pos, off);
        }
        if (sub == 0 && z < Z) {
          sNum[z] = num;
          sDen[z] = den;
          sPos[z] = pos;
        }
      }
    }

    // 3. theta1 / theta2 over the column's footprint (XT_VoxUpdate.c:20-51)
    const int tln = (T + VEC - 1) / VEC;
    // threads per entry tlp = 2^lg >= tln; the small CTAs group by shifts
    // (+3 % on 16-row items), the 256-thread ones keep the division (0.5 %
    // faster there as measured)
    int lg = 0;
    while ((1 << lg) < tln) lg++;
    const int tlp = 1 << lg;
    const int vgs = NT < XTG_THREADS ? NT >> lg : NT / tlp, tl = tid & (tlp - 1),
              vg = NT < XTG_THREADS ? tid >> lg : tid / tlp;
    float th1[VEC], th2[VEC];
#pragma unroll
    for (int c = 0; c < VEC; c++) th1[c] = th2[c] = 0.f;
    // one footprint entry: rows [off, off + VEC) past this thread's first row
    // of one (view, bin), weight a.  Generalized-Huber (zinger) weight
    // (XT_VoxUpdate.c:34-48): w where |e sqrt(w)| < T, else
    // we = T delta sqrt(w) / |e| = T delta w rsqrt(e^2 w), so that
    //   theta2 += a^2 we = a^2 T delta sqrt(w) / |e|,
    //   theta1 -= a e we = a T delta sign(e) sqrt(w);
    // rsqrt comes from the special-function unit, and the weighted branch
    // runs only when some lane of the warp meets a zinger.
    const int trow0 = t0 + tl * VEC;
    const float *eb = A.e + trow0;
    const float *wb = A.w + trow0;
    auto accumulate_arr = [&](const float (&ev)[VEC], const float (&wv)[VEC], float a) {
      const float a2 = a * a, na = -a;
      if constexpr (VEC == 4 && XTG_F32X2) {
        // two rows per instruction on the packed FP32 path; every product and
        // fused multiply-add is rounded as the scalar one would be
        const float2 e0 = make_float2(ev[0], ev[1]), e1 = make_float2(ev[2], ev[3]);
        const float2 w0 = make_float2(wv[0], wv[1]), w1 = make_float2(wv[2], wv[3]);
        const float2 ew0 = __fmul2_rn(e0, w0), ew1 = __fmul2_rn(e1, w1);
        const float2 q0 = __fmul2_rn(e0, ew0), q1 = __fmul2_rn(e1, ew1);  // e^2 w
        const float qm = fmaxf(fmaxf(q0.x, q0.y), fmaxf(q1.x, q1.y));
        const float2 aa = make_float2(a2, a2), nn = make_float2(na, na);
        float2 t20 = make_float2(th2[0], th2[1]), t21 = make_float2(th2[2], th2[3]);
        float2 t10 = make_float2(th1[0], th1[1]), t11 = make_float2(th1[2], th1[3]);
        if (__any_sync(__activemask(), qm >= A.T2)) {
          // the weight is w, or T delta w / sqrt(e^2 w) (= T delta sqrt(w) / |e|)
          // where |e sqrt(w)| >= T
          auto wgt = [&](float q, float w) { return q >= A.T2 ? A.Tdelta * w * rsqrtf(q) : w; };
          const float2 we0 = make_float2(wgt(q0.x, w0.x), wgt(q0.y, w0.y));
          const float2 we1 = make_float2(wgt(q1.x, w1.x), wgt(q1.y, w1.y));
          t20 = __ffma2_rn(aa, we0, t20);
          t21 = __ffma2_rn(aa, we1, t21);
          t10 = __ffma2_rn(nn, __fmul2_rn(e0, we0), t10);
          t11 = __ffma2_rn(nn, __fmul2_rn(e1, we1), t11);
        } else {
          t20 = __ffma2_rn(aa, w0, t20);
          t21 = __ffma2_rn(aa, w1, t21);
          t10 = __ffma2_rn(nn, ew0, t10);
          t11 = __ffma2_rn(nn, ew1, t11);
        }
        th2[0] = t20.x; th2[1] = t20.y; th2[2] = t21.x; th2[3] = t21.y;
        th1[0] = t10.x; th1[1] = t10.y; th1[2] = t11.x; th1[3] = t11.y;
        return;
      }
      float ew[VEC], q[VEC];
      float qm = 0.f;
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        ew[c] = ev[c] * wv[c];
        q[c] = ev[c] * ew[c];  // e^2 w
        qm = fmaxf(qm, q[c]);
      }
      if (__any_sync(__activemask(), qm >= A.T2)) {
        // branch-free per row: the weight is w, or T delta w / sqrt(e^2 w)
        // (= T delta sqrt(w) / |e|) where |e sqrt(w)| >= T
#pragma unroll
        for (int c = 0; c < VEC; c++) {
          const float we = q[c] >= A.T2 ? A.Tdelta * wv[c] * rsqrtf(q[c]) : wv[c];
          th2[c] = fmaf(a2, we, th2[c]);
          th1[c] = fmaf(na, ev[c] * we, th1[c]);
        }
      } else {
#pragma unroll
        for (int c = 0; c < VEC; c++) {
          th2[c] = fmaf(a2, wv[c], th2[c]);
          th1[c] = fmaf(na, ew[c], th1[c]);
        }
      }
    };
    auto accumulate_vals = [&](const float4 e4, const float4 w4, float a) {
      float ev[VEC], wv[VEC];
      const float ea[4] = {e4.x, e4.y, e4.z, e4.w}, wa[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        ev[c] = ea[c < 4 ? c : 0];
        wv[c] = wa[c < 4 ? c : 0];
      }
      accumulate_arr(ev, wv, a);
    };
    auto accumulate = [&](int off, float a) {
      float ev[VEC], wv[VEC];
      if (VEC == 4) {
        const float4 e4 = ld_e(eb + off);
        const float4 w4 = ld_w(wb + off, A.w_keep);
        ev[0] = e4.x; ev[1] = e4.y; ev[2] = e4.z; ev[3] = e4.w;
        wv[0] = w4.x; wv[1] = w4.y; wv[2] = w4.z; wv[3] = w4.w;
      } else {
#pragma unroll
        for (int c = 0; c < VEC; c++) {
          ev[c] = __ldcg(eb + off + c);
          wv[c] = __ldg(wb + off + c);
        }
      }
      accumulate_arr(ev, wv, a);
    };
    if (tl < tln) {
      if (AMODE == 0) {
        for (int v = vg; v < V; v += vgs) {
          const int pk = sPack[v], first = pk & 0xffffff, n = pk >> 24;
          const int off = (sView[v] * G.N_r + first) * G.N_t;
#pragma unroll
          for (int s = 0; s < AS; s++)
            if (s < n) accumulate(off + s * G.N_t, sVal[s * vmax + v]);
        }
      } else if (VEC == 4) {
        int e = vg;
        constexpr int UNR = NT < XTG_THREADS ? 2 : XTG_UNROLL;
        for (; e + (UNR - 1) * vgs < ne; e += UNR * vgs) {
          int2 en[UNR];
          float4 e4[UNR], w4[UNR];
#pragma unroll
          for (int u = 0; u < UNR; u++) en[u] = sEnt[e + u * vgs];
#pragma unroll
          for (int u = 0; u < UNR; u++) {
            e4[u] = ld_e(eb + en[u].x);
            w4[u] = ld_w(wb + en[u].x, A.w_keep);
          }
#pragma unroll
          for (int u = 0; u < UNR; u++) accumulate_vals(e4[u], w4[u], __int_as_float(en[u].y));
        }
        for (; e < ne; e += vgs) {
          const int2 en = sEnt[e];
          accumulate(en.x, __int_as_float(en.y));
        }
      } else {
        // single rows: four entries' loads in flight (one at a time left the
        // loop waiting on each round trip)
        int e = vg;
        constexpr int UNR = 4;
        for (; e + (UNR - 1) * vgs < ne; e += UNR * vgs) {
          int2 en[UNR];
          float ev[UNR], wv[UNR];
#pragma unroll
          for (int u = 0; u < UNR; u++) en[u] = sEnt[e + u * vgs];
#pragma unroll
          for (int u = 0; u < UNR; u++) {
            ev[u] = __ldcg(eb + en[u].x);
            wv[u] = __ldg(wb + en[u].x);
          }
#pragma unroll
          for (int u = 0; u < UNR; u++) {
            const float e1[VEC] = {ev[u]}, w1[VEC] = {wv[u]};
            accumulate_arr(e1, w1, __int_as_float(en[u].y));
          }
        }
        for (; e < ne; e += vgs) {
          const int2 en = sEnt[e];
          accumulate(en.x, __int_as_float(en.y));
        }
      }
    }
    // reduce over view groups: lanes with equal tl inside a warp, then warps
#pragma unroll
    for (int c = 0; c < VEC; c++) {
      for (int off = tlp; off < 32; off <<= 1) {
        th1[c] += __shfl_xor_sync(0xffffffffu, th1[c], off);
        th2[c] += __shfl_xor_sync(0xffffffffu, th2[c], off);
      }
    }
    if (lane < tlp && tl < tln) {
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        sRed[warp * rp + tl * VEC + c] = th1[c];
        sRed[(NW + warp) * rp + tl * VEC + c] = th2[c];
      }
    }
    __syncthreads();

    // 4. qGGMRF surrogate step per slice (CE_FunctionalSubstitution,
    //    XT_ICD_update.c:130-179) with zero skipping (XT_VoxUpdate.c:208-232).
    //    theta of a slice: its rows' partials over warps (every warp wrote its
    //    own, zeros if idle)
    auto theta = [&](int z, float &t1, float &t2) {
      t1 = t2 = 0.f;
      for (int r = z * G.zovl; r < (z + 1) * G.zovl; r++) {
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int wq = 0; wq < NW; wq++) {
          s1 += sRed[wq * rp + r];
          s2 += sRed[(NW + wq) * rp + r];
        }
        t1 += s1;
        t2 += s2;
      }
    };
    // the new value of slice z; returns false where the voxel is skipped
    auto update = [&](int z, float Vv, float num, float den) {
      float t1, t2;
      theta(z, t1, t2);
      const float u = (num + t2 * Vv - t1) / (den + t2);
      float nvx = Vv + G.alpha * (u - Vv);
      if (G.positivity && nvx <= 0.f) nvx = 0.f;
      if (!isfinite(nvx)) {
        atomicExch(A.err, 1);
        nvx = Vv;
      }
      sNb[4 * (zmax + 2) + z + 1] = nvx;
      A.x[(((size_t)fr * plane) + (size_t)row * G.N_x + col) * G.N_z + zb + z] = nvx;
      sDelta[z] = nvx - Vv;
      sAbs[lane] += (double)fabsf(nvx);
      sUpd[lane]++;
    };
    // the slots of the column itself, slices z - 1 and z + 1
    auto own_terms = [&](int z, float Vv, float &num, float &den, bool &pos) {
      const float vl = sNb[4 * (zmax + 2) + z], vh = sNb[4 * (zmax + 2) + z + 2];
      const float bl = zb + z > 0 || hlo ? sW[4] * qcoef(Vv - vl, G.C_S, A.l_sqp, A.e2p, G.MRF_P) : 0.f;
      const float bh = zb + z + 1 < G.N_z || hhi ? sW[22] * qcoef(Vv - vh, G.C_S, A.l_sqp, A.e2p, G.MRF_P) : 0.f;
      num = fmaf(bl, vl, fmaf(bh, vh, num));
      den += bl + bh;
      pos = pos || vl > 0.f || vh > 0.f;
    };
    if (SEQ) {
      // slices in increasing z on one thread, the reference's order
      if (tid == 0) {
        for (int z = 0; z < Z; z++) {
          const float Vv = sNb[4 * (zmax + 2) + z + 1];
          const uint32_t zm = (zb + z > 0 || hlo ? 1u : 0u) | 2u | (zb + z + 1 < G.N_z || hhi ? 4u : 0u);
          float num = 0.f, den = 0.f;
          bool pos = false;
          for (int n = 0; n < 29; n++) {
            if (n == 13) continue;
            const int dz = n / 9, cc = n % 9;
            const float v = n < 27 ? sNb[cc * (zmax + 2) + z + dz] : sTn[(n - 27) * zmax + z];
            const bool in = n < 27 ? ((colmask >> cc) & (zm >> dz) & 1u) != 0u : n == 27 ? fr > 0 : fr + 1 < G.N_time;
            const float b = !in      ? 0.f
                            : n < 27 ? sW[n] * qcoef(Vv - v, G.C_S, A.l_sqp, A.e2p, G.MRF_P)
                                     : sW[27] * qcoef(Vv - v, G.C_T, A.l_tqp, A.e2p, G.MRF_P);
            num += b * v;
            den += b;
            pos = pos || v > 0.f;
          }
          if (Vv == 0.f && A.iter > 1 && !pos) {
            sDelta[z] = 0.f;
            sZero[0]++;
          } else {
            update(z, Vv, num, den);
          }
        }
      }
    } else if (warp == 0) {
      // red/black in z: the even slices from the old values, the odd ones from
      // the new; one lane per voxel, so one warp does both passes
      for (int par = 0; par < 2; par++) {
        const int zfirst = ((zb & 1) == par) ? 0 : 1;  // first z (relative) with absolute parity par
        for (int z = zfirst + 2 * lane; z < Z; z += 64) {
          const float Vv = sNb[4 * (zmax + 2) + z + 1];
          float num = sNum[z], den = sDen[z];
          bool pos = sPos[z] != 0;
          own_terms(z, Vv, num, den, pos);
          if (Vv == 0.f && A.iter > 1 && !pos) {
            sDelta[z] = 0.f;
            sZero[lane]++;
          } else {
            update(z, Vv, num, den);
          }
        }
        __syncwarp();
      }
    }
    if (tid == META) fetch_meta(sMeta[mb ^ 1]);
    __syncthreads();
    if (warp == NW - 1) write_magmap();

    // 5. e -= (A delta_t) * delta_x on the footprint (XT_VoxUpdate.c:62-82)
    if (tl < tln) {
      float dv[VEC];
      bool any = false;
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        const int rr = tl * VEC + c;
        dv[c] = (rr < T) ? sDelta[G.zovl == 1 ? rr : rr / G.zovl] : 0.f;
        any |= (dv[c] != 0.f);
      }
      if (any) {
        float *ebw = A.e + trow0;
        auto scatter = [&](int off, float a) {
          if constexpr (VEC == 4 && XTG_F32X2) {
            const float2 na2 = make_float2(-a, -a);
            const float2 m0 = __fmul2_rn(na2, make_float2(dv[0], dv[1]));
            const float2 m1 = __fmul2_rn(na2, make_float2(dv[2], dv[3]));
            xt_red_add4(ebw + off, m0.x, m0.y, m1.x, m1.y);
          } else if (VEC == 4) {
            xt_red_add4(ebw + off, -(a * dv[0]), -(a * dv[1]), -(a * dv[2]), -(a * dv[3]));
          } else {
#pragma unroll
            for (int c = 0; c < VEC; c++)
              if (dv[c] != 0.f) atomicAdd(ebw + off + c, -(a * dv[c]));
          }
        };
        if (AMODE == 0) {
          for (int v = vg; v < V; v += vgs) {
            const int pk = sPack[v], first = pk & 0xffffff, n = pk >> 24;
            const int off = (sView[v] * G.N_r + first) * G.N_t;
#pragma unroll
            for (int s = 0; s < AS; s++)
              if (s < n) scatter(off + s * G.N_t, sVal[s * vmax + v]);
          }
        } else {
          for (int e = vg; e < ne; e += vgs) {
            const int2 en = sEnt[e];
            scatter(en.x, __int_as_float(en.y));
          }
        }
      }
    }
  }
  if (warp == 0) {
    double ab = sAbs[lane];
    unsigned long long up = sUpd[lane], zr = sZero[lane];
    for (int off = 16; off > 0; off >>= 1) {
      ab += __shfl_xor_sync(0xffffffffu, ab, off);
      up += __shfl_xor_sync(0xffffffffu, up, off);
      zr += __shfl_xor_sync(0xffffffffu, zr, off);
    }
    if (lane == 0 && (up || zr || ncol)) {
      atomicAdd(&A.st_absx[blockIdx.x & 63], ab);
      atomicAdd(&A.st_cnt[0], up);
      atomicAdd(&A.st_cnt[1], zr);
      atomicAdd(&A.st_cnt[2], (unsigned long long)ncol);
    }
  }
}

size_t icd_smem_bytes(int vmax, int zmax, int zovl, int as, int amode, int vec, int nt) {
  size_t b = 0;
  if (amode == 0)
    b += (size_t)vmax * (4 * 2 + 4 * (size_t)as);  // sPack, sView, sVal
  else
    b += (size_t)vmax * 8;                         // sEnt
  b += 2 * (size_t)(nt / 32) * (((size_t)zmax * zovl + 3) / 4 * 4) * 4;  // sRed
  b += 9 * (size_t)(zmax + 2) * 4;                 // sNb
  b += 2 * (size_t)zmax * 4;                       // sTn
  b += 4 * (size_t)zmax * 4;                       // sDelta, sNum, sDen, sPos
  return b;
}


typedef void (*IcdKernel)(DevGeo, IcdArgs, int, int);

// A computed in the kernel (amode 0): slot count 3 covers delta_xy <= delta_r,
// 4 covers delta_xy <= 1.5 delta_r, 12 covers delta_xy <= 5.5 delta_r.  The
// table modes (1 = FP16, 2 = FP32) have no per-view slots.
static IcdKernel icd_kernel(int vec, int amode, int seq, int as, int nt) {
#define XTG_K(V, S) (as == 3 ? k_icd_columns<V, 0, S, 3> : as == 4 ? k_icd_columns<V, 0, S, 4> : k_icd_columns<V, 0, S, 12>)
#define XTG_T(V, M, S) k_icd_columns<V, M, S, 3>
  if (amode != 0 && !seq) {
#define XTG_N(V, M)                                                                                                 \
  switch (nt) {                                                                                                     \
    case 64: return k_icd_columns<V, M, 0, 3, 64>;                                                                  \
    case 128: return k_icd_columns<V, M, 0, 3, 128>;                                                                \
    case 256: return k_icd_columns<V, M, 0, 3, 256>;                                                                \
    case 512: return k_icd_columns<V, M, 0, 3, 512>;                                                                \
    default: return k_icd_columns<V, M, 0, 3, 1024>;                                                                \
  }
    if (vec == 4 && amode == 1) XTG_N(4, 1)
    if (vec == 4) XTG_N(4, 2)
    if (amode == 1) XTG_N(1, 1)
    XTG_N(1, 2)
#undef XTG_N
  }
  if (vec == 4) {
    if (amode == 0) return seq ? XTG_K(4, 1) : XTG_K(4, 0);
    return amode == 1 ? XTG_T(4, 1, 1) : XTG_T(4, 2, 1);
  }
  if (amode == 0) return seq ? XTG_K(1, 1) : XTG_K(1, 0);
  return amode == 1 ? XTG_T(1, 1, 1) : XTG_T(1, 2, 1);
#undef XTG_K
#undef XTG_T
}

// Zeroes MagUpdateMap[frame][block][row][col] for every (item, block the
// item covers) of an ICD launch whose items are split into z pieces, which
// then add their partial sums into it.
__global__ void k_magmap_zero(DevGeo G, IcdArgs A) {
  const int nitems = A.n_items_dev ? min(*A.n_items_dev, A.n_items) : A.n_items;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nitems; i += gridDim.x * blockDim.x) {
    const int q = A.use_perm ? (int)xt_perm((uint32_t)i, (uint32_t)nitems, A.perm_key) : i;
    const int4 item = A.items[A.item_lo + q];
    const int b0 = item.w >= 0 ? item.w : 0, b1 = item.w >= 0 ? item.w : G.nzb - 1;
    for (int b = b0; b <= b1; b++)
      A.magmap[(((size_t)item.x * G.nzb + b) * G.N_y + item.y) * G.N_x + item.z] = 0.f;
  }
}

cudaError_t launch_magmap_zero(const DevGeo &G, const IcdArgs &A, int grid, cudaStream_t st) {
  k_magmap_zero<<<grid, 256, 0, st>>>(G, A);
  return cudaGetLastError();
}

// Columns in flight: CTAs of a launch, and the items each takes at a time.
//
// Columns updated at the same time read each other's stale error sinogram, so
// how many there are, and in which groups, is part of an iteration's result.
// Near neighbours share most of their footprint: too many of them at once
// overshoot (Jacobi-like) and the cost stops falling -- on a 32^2-column grid 64
// and more at once left the cost oscillating 20-50 % above the converged value,
// 32 did not.  The schedule that sets the iterations' course is one column in
// 32, no more than are resident in CTAs of 64 threads for items of at most 16
// rows, 128 for runs of at most 1024 entries, 256 otherwise, the first two eight
// items at a time (so an eighth of a launch's items are in flight).  Items that
// spend less of their time outside [first read of e, last write of e] are staler
// at the same number: with it this kernel moves an iteration's update percentage
// by up to 3.3 times what runs differ by, with twice as many by 5 to 9 times
// (64^2 x 8, 4 frames of 48 views, iteration 8: 0.168 -> 0.173 %).  Hence, where
// the fixed work weighs (shift in units of the run-to-run spread, which is 0.05 to
// 0.3 % of the percentage, without -> with):
//   one column in 33 for single-row and long items read from a table (128^2 x 9
//     +1.0 -> +0.3), one in 36 for short ones
//   an eighth fewer than are resident for short items with runs of at most 512
//     entries (256^2 x 16 x 16 frames +1.7 -> +0.7) and for long ones where that is more
//     than one column in 256; three sixteenths fewer for single rows above one in 320
//     (180^2 x 27 +2.1 -> -0.1, 148^2 x 12 +1.8 -> +0.1)
//   for such runs ten items at a time in the 128-thread class and nine in the
//     64-thread one above 1536 rows x entries (140^2 x 32, 4 frames +2.6 -> +0.4;
//     96^2 x 32, 8 frames +3.3 -> +0.4; 96^2 x 16, 4 frames +1.4 -> 0.0)
// 114 volumes of 64^2 to 512^2, 3 to 80 rows, 1 to 16 frames lie between -2.2 and
// +1.8 with it (one of 8 frames with A computed here +2.7), half of them within
// 0.4.  It costs time: 80^2 x 8, 500 views 1.4 ms an iteration with twice the
// columns, 2.5 so; 256^2 x 32, 512 views 7.7 and 10.0; 128^2 x 4 1.1 and 1.5.
IcdFlight icd_flight(int vec, int amode, int as, int vmax, int zmax, int zovl, long long columns, int sms) {
  const int rows = zmax * zovl;
  const int unit = vec != 4 || amode == 0 ? XTG_THREADS : rows <= 16 ? 64 : vmax <= 1024 ? 128 : XTG_THREADS;
  // shared memory of such a CTA: run, 128 partial sums twice a warp, neighbourhood
  const size_t smem = (size_t)vmax * (amode == 0 ? 8 + 4 * as : 8) + (size_t)unit * 32 + (size_t)rows * 8 + (size_t)zmax * 48 + 1280;
  long long resident = (long long)sms * std::max(1, std::min(1024 / unit, (int)(228 * 1024 / smem)));
  if (amode && vec == 4 && (unit < XTG_THREADS ? vmax <= 512 : resident * 256 > columns)) resident -= resident / 8;
  if (amode && vec != 4 && resident * 320 > columns) resident -= resident * 3 / 16;
  IcdFlight f;
  f.cols = (int)std::min(resident, std::max(8ll, columns / (amode == 0 ? 32 : unit == XTG_THREADS ? 33 : 36)));
  f.batch = unit == XTG_THREADS ? 1 : vmax > 512 ? 8 : unit == 128 ? 10 : rows * vmax > 1536 ? 9 : 8;
  return f;
}

// Threads per CTA for items of zmax slices, `cols` of them in flight on `sms`
// SMs.  Table modes, parallel schedule; otherwise XTG_THREADS.  A larger CTA
// keeps more partial sums beside the column run (2 rows a warp), so sizes past
// what an SM's shared memory holds are not taken either.
int icd_threads(int vec, int amode, int as, int zmax, int zovl, int vmax, int cols, int sms) {
  if (amode == 0) return XTG_THREADS;
  int tlp = 1;
  while (tlp * vec < zmax * zovl) tlp *= 2;
  const long long groups = (long long)tlp * vmax;
  int nt = XTG_NT_MIN;
  while (nt < XTG_NT_MAX && groups > (long long)nt * XTG_GROUPS_PER_THREAD &&
         (long long)sms * icd_occupancy(vec, amode, 0, as, vmax, zmax, zovl, 2 * nt) >= std::max(cols, 1))
    nt *= 2;
  return nt;
}

cudaError_t launch_icd(const DevGeo &G, const IcdArgs &A, int vec, int amode, int seq, int as, int vmax, int zmax,
                       int grid, int nt, cudaStream_t st) {
  const size_t smem = icd_smem_bytes(vmax, zmax, G.zovl, as, amode, vec, nt);
  IcdKernel k = icd_kernel(vec, amode, seq, as, nt);
  // e and w stream through L2 (e must, it is updated by other CTAs' atomics),
  // so the unified L1/shared space goes to shared memory: more CTAs per SM
  cudaError_t e = full_smem((const void *)k);
  if (e != cudaSuccess) return e;
  k<<<grid, nt, smem, st>>>(G, A, vmax, zmax);
  return cudaGetLastError();
}

// CTAs of nt threads on an SM; 0 where one alone does not fit
int icd_occupancy(int vec, int amode, int seq, int as, int vmax, int zmax, int zovl, int nt) {
  const size_t smem = icd_smem_bytes(vmax, zmax, zovl, as, amode, vec, nt);
  IcdKernel k = icd_kernel(vec, amode, seq, as, nt);
  // asked once per kernel, size and device (2 us of host time a launch)
  struct Entry {
    const void *fn;
    size_t smem;
    int dev, nb;
  };
  static std::mutex mu;
  static std::vector<Entry> seen;
  int dev = 0, nb = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lk(mu);
  for (const Entry &q : seen)
    if (q.fn == (const void *)k && q.smem == smem && q.dev == dev) return q.nb;
  if (full_smem((const void *)k) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, (const void *)k, nt, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (seen.size() >= 1024) seen.clear();
  seen.push_back(Entry{(const void *)k, smem, dev, nb});
  return nb;
}

// Once per kernel and device: as much dynamic shared memory as the device
// gives a CTA, and the L1/shared split in favour of shared memory.
cudaError_t full_smem(const void *fn) {
  static std::mutex mu;
  static std::vector<std::pair<const void *, int>> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  for (const auto &q : done)
    if (q.first == fn && q.second == dev) return cudaSuccess;
  int most = 0;
  cudaFuncAttributes at;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess ||
      (e = cudaFuncGetAttributes(&at, fn)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)at.sharedSizeBytes)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared)) !=
          cudaSuccess)
    return e;
  done.emplace_back(fn, dev);
  return cudaSuccess;
}

}  // namespace xtg
