// cnn_conv_box.cu -- 3x3x3 convolutions and weight gradients of the warm-start
// network for any volume size, operands staged by TMA (BF16 in, FP32
// accumulation in TMEM).
//
// The gather kernels (cnn_conv.cu) build every operand row with per-thread
// loads; the tile kernels (cnn_conv_tile.cu) need rows of 128 x-voxels.  Here a
// tile is a box of 128 voxels, z x x x y x batch with power-of-two sides chosen
// to cover the volume with the fewest boxes, and the operand of a tap is the
// same box read at the tap's offset: one TMA load of 128 voxels x CH channels,
// zero filled outside the volume (the padding) and past the last channel.
// Each input voxel is fetched 27 times, from L2: the rate at which an SM's TMA
// unit takes rows (about four cycles each, 64- or 128-byte ones alike) bounds
// these kernels, not the MMAs.  Where the planes are not too small for it a tile is
// 8 z x 16 x of one y-row, its halo read once for nine taps (k_conv_halo,
// k_wgrad_halo below).
//
// CH is 64 (128-byte rows, the 128-byte swizzle) or 32 (64-byte rows, 64-byte
// swizzle), whichever pads the channels less.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "cnn_tc.cuh"
#include "xtg_cnn_internal.h"

namespace xtc {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

namespace {

constexpr long long kLim = 1ll << 24;  // polls of a bounded wait

// the 128-voxel box: sides (powers of two) and the boxes along each dimension
struct Box {
  int z, x, y, b;
  int nz, nx, ny, nbx;
  __host__ __device__ int count() const { return nz * nx * ny * nbx; }
};

// fewest boxes; among equals the longest runs in memory (z, then x)
bool choose_box(const ConvShape &s, Box *out) {
  long long best = -1;
  for (int z = 1; z <= 128; z *= 2)
    for (int x = 1; z * x <= 128; x *= 2)
      for (int y = 1; z * x * y <= 128; y *= 2) {
        const int b = 128 / (z * x * y);
        auto up = [](int n, int d) { return (n + d - 1) / d; };
        const long long n = (long long)up(s.Z, z) * up(s.X, x) * up(s.Y, y) * up(s.nb, b);
        if (best < 0 || n < best || (n == best && (z > out->z || (z == out->z && x > out->x)))) {
          best = n;
          *out = Box{z, x, y, b, up(s.Z, z), up(s.X, x), up(s.Y, y), up(s.nb, b)};
        }
      }
  return best > 0 && best < (1ll << 30);
}

__device__ __forceinline__ void box_origin(const Box &B, int t, int &z0, int &x0, int &y0, int &b0) {
  z0 = (t % B.nz) * B.z;
  t /= B.nz;
  x0 = (t % B.nx) * B.x;
  t /= B.nx;
  y0 = (t % B.ny) * B.y;
  b0 = (t / B.ny) * B.b;
}

// Halo tiles: `mv` (1 or 2) M tiles of 8 z x 16 x of one y-row, read by one box
// of 10 x (16 mv + 2) voxels: in its rows (z fastest) every (dx, dz) shift of an
// M tile is 16 groups of 8 rows, 10 rows apart, so one box serves nine taps.
struct Halo {
  int mv, nz, nx, Y, nb;
  __host__ __device__ int count() const { return nz * nx * Y * nb; }
};
constexpr int HZ = 8, HX = 16, HZS = HZ + 2;
__host__ __device__ constexpr int halo_rows(int mv) { return HZS * (HX * mv + 2); }
// bytes of a box in shared memory (an unused upper half of an M tile reads one row past it)
__host__ __device__ constexpr uint32_t halo_bytes(int mv, int ch) {
  return (uint32_t)(((halo_rows(mv) + 1) * ch * 2 + 1023) / 1024 * 1024);
}

__device__ __forceinline__ void halo_origin(const Halo &H, int t, int &z0, int &x0, int &y, int &b) {
  z0 = (t % H.nz) * HZ;
  t /= H.nz;
  x0 = (t % H.nx) * (HX * H.mv);
  t /= H.nx;
  y = t % H.Y;
  b = t / H.Y;
}

// K-major operand: rows of CH channels, 8-row groups CH * 16 bytes apart
template <int CH>
__device__ __forceinline__ uint64_t desc_k(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)CH << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)(CH == 64 ? 2 : 4) << 61);
}
// MN-major operand: a row per K index, 8-row groups CH * 16 bytes apart (SBO),
// atoms of CH channels `lbo` bytes apart
template <int CH>
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)CH << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)(CH == 64 ? 2 : 4) << 61);
}

// halo operand: 8-row groups HZS rows of CH channels apart; MN-major atoms `lbo` bytes apart
template <int CH>
__device__ __forceinline__ uint64_t desc_halo(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)(HZS * CH * 2 / 16) << 32) | ((uint64_t)1 << 46) | ((uint64_t)(CH == 64 ? 2 : 4) << 61);
}

__host__ __device__ constexpr uint32_t pow2_cols(int n) {
  uint32_t c = 32;
  while (c < (uint32_t)n) c *= 2;
  return c;
}

__device__ __forceinline__ void tap_of(int t, int &dy, int &dx, int &dz) {
  dy = t / 9 - 1;
  dx = t / 3 % 3 - 1;
  dz = t % 3 - 1;
}

// this lane's accumulator row (N columns from `acc` on) to voxel vox of out, where `in`
template <int EPI>
__device__ __forceinline__ void drain(bool in, size_t vox, int N, uint32_t acc, const float *__restrict__ bias, void *out) {
  for (int n0 = 0; n0 < N; n0 += 16) {
    __align__(16) float v[16];
    tmem_ld16(acc + (uint32_t)n0, v);
    if (in) {
      if (EPI == 2) {
        float *o = reinterpret_cast<float *>(out) + vox * N + n0;
        store32(o, *reinterpret_cast<const int4 *>(v), *reinterpret_cast<const int4 *>(v + 4));
        store32(o + 8, *reinterpret_cast<const int4 *>(v + 8), *reinterpret_cast<const int4 *>(v + 12));
      } else {
        __align__(16) __nv_bfloat16 h[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
          float f = v[i];
          if (EPI == 0) f = fmaxf(f + bias[n0 + i], 0.f);
          h[i] = __float2bfloat16_rn(f);
        }
        __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(out) + vox * N + n0;
        store32(o, *reinterpret_cast<const int4 *>(h), *reinterpret_cast<const int4 *>(h + 8));
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Forward and input gradient.  Persistent CTAs of 192 threads: warp 4 (one
// thread) issues a stage's copies -- the tap's box and the matching weight
// rows, packed and swizzled beforehand, in one bulk copy -- warp 5 (one
// thread) the MMAs, M = the box's voxels, N = cout, K = CH; warps 0-3 drain
// the finished accumulator while the other TMEM buffer fills.  The K order
// (tap, then channel) is the gather kernel's, so the results are its bits.
//
// Kernel times in a training step of 8 patches of 32 x 128 x 32, gather -> box (all
// of these shapes run on halo tiles now): 48 -> 48 (131072 voxels) 195 -> 57 us,
// 160 -> 64 (16384 voxels) 215 -> 56, 96 -> 96 (2048 voxels) 147 -> 38.
template <int CH, int EPI>
__global__ void __launch_bounds__(192) k_conv_box(const __grid_constant__ CUtensorMap tin, ConvShape s, Box B, int sign,
                                                  const __nv_bfloat16 *__restrict__ wp, const float *__restrict__ bias,
                                                  void *out, int nstage, int *err) {
  extern __shared__ __align__(1024) uint8_t sm_raw[];
  // stages start on the 1024 bytes the swizzle repeats over
  uint8_t *sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
  constexpr uint32_t ABYTES = 128 * CH * 2;
  constexpr int MAXST = 8;
  const int N = s.n;
  const uint32_t BBYTES = (uint32_t)N * CH * 2, STAGE = ABYTES + BBYTES;
  __shared__ uint64_t full[MAXST], empty[MAXST], acc_full[2], acc_empty[2], done;
  __shared__ uint32_t tbase;
  __shared__ volatile int bad;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int nchunk = (s.cin + CH - 1) / CH, nk = 27 * nchunk;
  const int ntiles = B.count();
  const int mine = ntiles > (int)blockIdx.x ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const uint32_t cols = pow2_cols(2 * N);
  if (tid == 0) {
    for (int i = 0; i < nstage; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 4);
    }
    mbar_init(&done, 1);
    mbar_init_fence();
    bad = 0;
  }
  if (warp == 0) tmem_alloc(&tbase, cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  if (warp == 4) {
    if (lane == 0) {
      int q = 0;
      bool ok = true;
      for (int tl = 0; tl < mine && ok; tl++) {
        int z0, x0, y0, b0;
        box_origin(B, (int)blockIdx.x + tl * (int)gridDim.x, z0, x0, y0, b0);
        for (int t = 0; t < 27 && ok; t++) {
          int dy, dx, dz;
          tap_of(t, dy, dx, dz);
          for (int c = 0; c < nchunk; c++, q++) {
            const int st = q % nstage;
            if (q >= nstage && (!mbar_wait(&empty[st], (uint32_t)(q / nstage - 1) & 1u, kLim) || bad)) {
              ok = false;
              break;
            }
            uint8_t *a = sm + (size_t)st * STAGE;
            mbar_expect_tx(&full[st], STAGE);
            tma_load_5d(a, &tin, c * CH, z0 + sign * dz, x0 + sign * dx, y0 + sign * dy, b0, &full[st]);
            bulk_load(a + ABYTES, wp + (size_t)(t * nchunk + c) * N * CH, BBYTES, &full[st]);
          }
        }
      }
      if (!ok) {
        atomicExch(err, 1);
        bad = 1;
      }
      // the copies issued last land before the shared memory is released
      for (int i = q > nstage ? q - nstage : 0; i < q; i++) mbar_wait(&full[i % nstage], (uint32_t)(i / nstage) & 1u, kLim);
    }
    __syncwarp();
  } else if (warp == 5) {
    const uint32_t idesc = idesc_bf16(N, 0, 0);
    const bool lead = elect_one();
    bool ok = true;
    int st = 0;
    uint32_t ph = 0;
    for (int tl = 0; tl < mine && ok; tl++) {
      const int ab = tl & 1;
      if (tl >= 2 && !mbar_wait_warp(&acc_empty[ab], (uint32_t)((tl >> 1) - 1) & 1u, kLim)) {
        ok = false;
        break;
      }
      const uint32_t acc = tmem + (uint32_t)(ab * N);
      for (int k = 0; k < nk; k++) {
        if (!mbar_wait_warp(&full[st], ph, kLim)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a0 = smem_u32(sm) + (uint32_t)st * STAGE;
        const uint64_t da = desc_k<CH>(a0), db = desc_k<CH>(a0 + ABYTES);
        if (lead) {
#pragma unroll
          for (int ks = 0; ks < CH / 16; ks++)
            mma_bf16(acc, da + (uint64_t)(2 * ks), db + (uint64_t)(2 * ks), idesc, (k > 0 || ks > 0) ? 1u : 0u);
          mma_commit(&empty[st]);
        }
        __syncwarp();
        if (++st == nstage) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (ok && lead) mma_commit(&acc_full[ab]);
      ok = __all_sync(0xffffffffu, ok && !bad);
    }
    if (!ok && lead) {
      atomicExch(err, 1);
      bad = 1;
    }
    if (lead) mma_commit(&done);
    __syncwarp();
    mbar_wait(&done, 0, kLim);  // every MMA issued above has completed
  } else {
    // row r of a box: z fastest, then x, y, batch
    const int r = warp * 32 + lane;
    const int rz = r % B.z, rx = r / B.z % B.x, ry = r / (B.z * B.x) % B.y, rb = r / (B.z * B.x * B.y);
    for (int tl = 0; tl < mine; tl++) {
      const int ab = tl & 1;
      const bool gone = !mbar_wait(&acc_full[ab], (uint32_t)(tl >> 1) & 1u, kLim) || bad;
      if (__any_sync(0xffffffffu, gone)) {
        if (lane == 0) atomicExch(err, 1);
        bad = 1;
        break;
      }
      tc_fence_after();
      int z, x, y, b;
      box_origin(B, (int)blockIdx.x + tl * (int)gridDim.x, z, x, y, b);
      z += rz;
      x += rx;
      y += ry;
      b += rb;
      const bool in = z < s.Z && x < s.X && y < s.Y && b < s.nb;
      const size_t vox = (((size_t)b * s.Y + y) * s.X + x) * s.Z + z;
      drain<EPI>(in, vox, N, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(ab * N), bias, out);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[ab]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, cols);
  }
}

// ---------------------------------------------------------------------------
// Forward and input gradient from halo tiles: a step of one dy is read once (all
// its channel chunks) and serves nine taps x mv M tiles; the weights come tap by
// tap through their own ring.  K order as in k_conv_box, so the bits are the
// same.  Warps 0-3 drain the accumulators, 4 loads halos, 5 issues the MMAs, 6
// loads weights.  k_conv_box spends 27 x 128 TMA rows on 128 voxels, at about 4
// cycles a row its bound; here it is 3 x 180, or 3 x 340 for 256 voxels.  What
// bounds it now is the MMA warp's issue and waits, tap by tap.
//
// Whole calls (weights packed), box -> halo: 48 -> 48, 131072 voxels 112 -> 79 us;
// 112 -> 48 150 -> 114; 160 -> 64, 16384 voxels 107 -> 69; 32 -> 80, 1048576 voxels
// 479 -> 314.
constexpr int CH_BST = 6;  // weight stages at most
template <int CH, int EPI>
__global__ void __launch_bounds__(224) k_conv_halo(const __grid_constant__ CUtensorMap tin, ConvShape s, Halo H, int sign,
                                                      const __nv_bfloat16 *__restrict__ wp, const float *__restrict__ bias,
                                                      void *out, int nbst, int *err) {
  extern __shared__ __align__(1024) uint8_t sm_raw[];
  uint8_t *sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
  constexpr uint32_t ROW = CH * 2;
  const int N = s.n, mv = H.mv;
  const int nchunk = (s.cin + CH - 1) / CH;
  const uint32_t ACH = halo_bytes(mv, CH), ASTAGE = (uint32_t)nchunk * ACH, BCH = (uint32_t)N * CH * 2,
                 BSTAGE = (uint32_t)nchunk * BCH, BSLOT = (BSTAGE + 1023u) / 1024u * 1024u;
  uint8_t *sA = sm, *sB = sm + 2 * ASTAGE;
  __shared__ uint64_t fullA[2], emptyA[2], fullB[CH_BST], emptyB[CH_BST], acc_full[2], acc_empty[2], done;
  __shared__ uint32_t tbase;
  __shared__ volatile int bad;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int ntiles = H.count();
  const int mine = ntiles > (int)blockIdx.x ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const uint32_t cols = pow2_cols(2 * mv * N);
  if (tid == 0) {
    for (int i = 0; i < nbst; i++) {
      mbar_init(&fullB[i], 1);
      mbar_init(&emptyB[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&fullA[i], 1);
      mbar_init(&emptyA[i], 1);
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 4);
    }
    mbar_init(&done, 1);
    mbar_init_fence();
    bad = 0;
  }
  if (warp == 0) tmem_alloc(&tbase, cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  if (warp == 4) {
    if (lane == 0) {
      const int n = 3 * mine;
      bool ok = true;
      int q = 0, dyi = 0, z0, x0, y, b;
      for (; q < n; q++) {
        const int st = q & 1;
        if (q >= 2 && (!mbar_wait(&emptyA[st], (uint32_t)((q >> 1) - 1) & 1u, kLim) || bad)) {
          ok = false;
          break;
        }
        if (dyi == 0) halo_origin(H, (int)blockIdx.x + q / 3 * (int)gridDim.x, z0, x0, y, b);
        mbar_expect_tx(&fullA[st], (uint32_t)(nchunk * halo_rows(mv)) * ROW);
        for (int c = 0; c < nchunk; c++)
          tma_load_5d(sA + st * ASTAGE + c * ACH, &tin, c * CH, z0 - 1, x0 - 1, y + sign * (dyi - 1), b, &fullA[st]);
        dyi = dyi == 2 ? 0 : dyi + 1;
      }
      if (!ok) {
        atomicExch(err, 1);
        bad = 1;
      }
      // the copies issued last land before the shared memory is released
      for (int i = q > 2 ? q - 2 : 0; i < q; i++) mbar_wait(&fullA[i & 1], (uint32_t)(i >> 1) & 1u, kLim);
    }
    __syncwarp();
  } else if (warp == 6) {
    if (lane == 0) {
      const int n = 27 * mine;
      bool ok = true;
      int q = 0, st = 0, tap = 0;
      uint32_t ph = 1;  // (the first round's waits pass at once)
      const size_t tstep = (size_t)nchunk * N * CH;
      for (; q < n; q++) {
        if (!mbar_wait(&emptyB[st], ph, kLim) || bad) {
          ok = false;
          break;
        }
        mbar_expect_tx(&fullB[st], BSTAGE);
        bulk_load(sB + (size_t)st * BSLOT, wp + tap * tstep, BSTAGE, &fullB[st]);
        tap = tap == 26 ? 0 : tap + 1;
        if (++st == nbst) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (!ok) {
        atomicExch(err, 1);
        bad = 1;
      }
      for (int i = q > nbst ? q - nbst : 0; i < q; i++) mbar_wait(&fullB[i % nbst], (uint32_t)(i / nbst) & 1u, kLim);
    }
    __syncwarp();
  } else if (warp == 5) {
    const uint32_t idesc = idesc_bf16(N, 0, 0);
    const bool lead = elect_one();
    const uint32_t vstep = HX * HZS * ROW >> 4, cstep = ACH >> 4, bstep = BCH >> 4;
    bool ok = true;
    int st = 0;
    uint32_t ph = 0, pa = 0;
    for (int tl = 0; tl < mine && ok; tl++) {
      const int ab = tl & 1;
      if (tl >= 2 && !mbar_wait_warp(&acc_empty[ab], (uint32_t)((tl >> 1) - 1) & 1u, kLim)) {
        ok = false;
        break;
      }
      const uint32_t acc = tmem + (uint32_t)(ab * mv * N);
      for (int dyi = 0; dyi < 3 && ok; dyi++, pa++) {
        if (!mbar_wait_warp(&fullA[pa & 1], (pa >> 1) & 1u, kLim)) {
          ok = false;
          break;
        }
        // the taps' first row: (dx, dz) = (-1, -1) times sign
        uint64_t da = desc_halo<CH>(smem_u32(sA) + (pa & 1) * ASTAGE + (uint32_t)((1 - sign) * (HZS + 1)) * ROW, 16);
        for (int dxi = 0; dxi < 3 && ok; dxi++, da += (int64_t)(sign * (HZS - 3)) * (int64_t)(ROW >> 4))
          for (int dzi = 0; dzi < 3; dzi++, da += (int64_t)sign * (int64_t)(ROW >> 4)) {
            if (!mbar_wait_warp(&fullB[st], ph, kLim)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t db = desc_k<CH>(smem_u32(sB) + (uint32_t)st * BSLOT);
            const uint32_t first = (dyi | dxi | dzi) ? 1u : 0u;
            if (lead) {
              for (int c = 0; c < nchunk; c++) {
                const uint64_t dac = da + c * cstep, dbc = db + c * bstep;
#pragma unroll
                for (int ks = 0; ks < CH / 16; ks++) {
                  const uint32_t on = ks > 0 ? 1u : (first | (c > 0 ? 1u : 0u));
                  mma_bf16(acc, dac + (uint64_t)(2 * ks), dbc + (uint64_t)(2 * ks), idesc, on);
                  if (mv == 2)
                    mma_bf16(acc + (uint32_t)N, dac + vstep + (uint64_t)(2 * ks), dbc + (uint64_t)(2 * ks), idesc, on);
                }
              }
              mma_commit(&emptyB[st]);
            }
            __syncwarp();
            if (++st == nbst) {
              st = 0;
              ph ^= 1u;
            }
          }
        if (ok && lead) mma_commit(&emptyA[pa & 1]);
      }
      if (ok && lead) mma_commit(&acc_full[ab]);
      if (bad) ok = false;
      ok = __all_sync(0xffffffffu, ok);
    }
    if (!ok && lead) {
      atomicExch(err, 1);
      bad = 1;
    }
    if (lead) mma_commit(&done);
    __syncwarp();
    mbar_wait(&done, 0, kLim);  // every MMA issued above has completed
  } else if (warp < 4) {
    const int r = warp * 32 + lane, rz = r % HZ, rx = r / HZ;
    for (int tl = 0; tl < mine; tl++) {
      const int ab = tl & 1;
      const bool gone = !mbar_wait(&acc_full[ab], (uint32_t)(tl >> 1) & 1u, kLim) || bad;
      if (__any_sync(0xffffffffu, gone)) {
        if (lane == 0) atomicExch(err, 1);
        bad = 1;
        break;
      }
      tc_fence_after();
      int z0, x0, y, b;
      halo_origin(H, (int)blockIdx.x + tl * (int)gridDim.x, z0, x0, y, b);
      for (int v = 0; v < mv; v++) {
        const int z = z0 + rz, x = x0 + v * HX + rx;
        drain<EPI>(z < s.Z && x < s.X, (((size_t)b * s.Y + y) * s.X + x) * s.Z + z, N,
                   tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((ab * mv + v) * N), bias, out);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[ab]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, cols);
  }
}

// ---------------------------------------------------------------------------
// Weight gradient: dW[tap][ci][co] += sum_v in[v + d(tap)][ci] dout[v][co].  A CTA owns
// the nine taps of one dy and one chunk of CH input channels over a slice of
// the boxes.  K is the box's 128 voxels, so both operands are MN-major as they
// lie in memory: A stacks 128 / CH taps along M (one TMA box each), B is the
// box of dout, kept for the nine taps.  The accumulators of the ceil(9 CH / 128)
// M tiles stay in TMEM over the slice and are added into dw at the end.
//
// Training step, 8 patches of 32 x 128 x 32, gather -> box (on halo tiles now):
// level 1 48 x 48 320 -> 63 us, 112 x 48 813 -> 117 us, level 2 160 x 64 165 -> 31 us.
constexpr int WB_SLOTS = 4;                    // A slots (one M tile each)
constexpr uint32_t WB_A = 128 * 128 * 2;       // bytes of a slot
template <int CH>
__host__ __device__ constexpr int wb_mtiles() {
  return (9 * CH + 127) / 128;
}

template <int CH>
__host__ __device__ constexpr int wh_mtiles() {
  return CH == 64 ? 5 : 3;
}

// the accumulators of MT M tiles of TPM taps x CH channels, added into dw
template <int CH, int TPM, int MT>
__device__ __forceinline__ void add_wgrad(const ConvShape &s, int dyi, int ck, int warp, int lane, uint32_t tmem, float *dw) {
  const int N = s.n;
  const int r = warp * 32 + lane;  // accumulator row: tap u of the M tile, channel
  const int u = r / CH, ci = ck * CH + r % CH;
  const bool al = (reinterpret_cast<uintptr_t>(dw) & 15) == 0;
  for (int m = 0; m < MT; m++) {
    const int t9 = m * TPM + u;
    const bool in = u < TPM && t9 < 9 && ci < s.cin;
    // tap (dy, dx, dz): t9 = 3 (dx + 1) + (dz + 1)
    float *o = dw + ((size_t)(dyi * 9 + t9) * s.cin + ci) * N;
    for (int n0 = 0; n0 < N; n0 += 16) {
      float v[16];
      tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(m * N + n0), v);
      if (in && al) {
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o + n0 + i), "f"(v[i]), "f"(v[i + 1]),
                       "f"(v[i + 2]), "f"(v[i + 3])
                       : "memory");
      } else if (in) {
#pragma unroll
        for (int i = 0; i < 16; i++) atomicAdd(o + n0 + i, v[i]);
      }
      __syncwarp();
    }
  }
}

template <int CH, int CHB>
__global__ void __launch_bounds__(192, 1) k_wgrad_box(const __grid_constant__ CUtensorMap tin,
                                                      const __grid_constant__ CUtensorMap tdy, ConvShape s, Box B,
                                                      float *dw, int slices, int *err) {
  extern __shared__ __align__(1024) uint8_t sm_raw[];
  // stages start on the 1024 bytes the swizzle repeats over
  uint8_t *sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
  constexpr int MT = wb_mtiles<CH>(), TPM = 128 / CH;  // M tiles, taps per M tile
  constexpr uint32_t ABOX = 128 * CH * 2, BBOX = 128 * CHB * 2;
  const int N = s.n, nbc = (N + CHB - 1) / CHB;
  const uint32_t BSLOT = (uint32_t)nbc * BBOX;
  uint8_t *sA = sm, *sB = sm + WB_SLOTS * WB_A;
  __shared__ uint64_t fullA[WB_SLOTS], emptyA[WB_SLOTS], fullB[2], emptyB[2], acc_full;
  __shared__ uint32_t tbase;
  __shared__ volatile int bad;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int nchunk = (s.cin + CH - 1) / CH;
  const int grp = (int)blockIdx.x / slices, slice = (int)blockIdx.x % slices;
  const int dyi = grp / nchunk, ck = grp % nchunk;
  const int ntiles = B.count();
  const int mine = ntiles > slice ? (ntiles - 1 - slice) / slices + 1 : 0;
  const uint32_t cols = pow2_cols(MT * N);
  if (tid == 0) {
    for (int i = 0; i < WB_SLOTS; i++) {
      mbar_init(&fullA[i], 1);
      mbar_init(&emptyA[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&fullB[i], 1);
      mbar_init(&emptyB[i], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init_fence();
    bad = 0;
  }
  if (warp == 0) tmem_alloc(&tbase, cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  if (warp == 4) {
    if (lane == 0) {
      bool ok = true;
      int q = 0, nb = 0;  // A slots, B slots filled so far
      for (int tl = 0; tl < mine && ok; tl++) {
        int z0, x0, y0, b0;
        box_origin(B, slice + tl * slices, z0, x0, y0, b0);
        if (tl >= 2 && (!mbar_wait(&emptyB[tl & 1], (uint32_t)((tl >> 1) - 1) & 1u, kLim) || bad)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&fullB[tl & 1], BSLOT);
        for (int c = 0; c < nbc; c++)
          tma_load_5d(sB + (tl & 1) * BSLOT + c * BBOX, &tdy, c * CHB, z0, x0, y0, b0, &fullB[tl & 1]);
        nb++;
        for (int m = 0; m < MT; m++, q++) {
          const int st = q % WB_SLOTS;
          if (q >= WB_SLOTS && (!mbar_wait(&emptyA[st], (uint32_t)(q / WB_SLOTS - 1) & 1u, kLim) || bad)) {
            ok = false;
            break;
          }
          const int nt = m * TPM + TPM <= 9 ? TPM : 9 - m * TPM;  // taps of this M tile
          mbar_expect_tx(&fullA[st], (uint32_t)nt * ABOX);
          for (int u = 0; u < nt; u++) {
            const int t9 = m * TPM + u;
            tma_load_5d(sA + st * WB_A + u * ABOX, &tin, ck * CH, z0 + t9 % 3 - 1, x0 + t9 / 3 - 1, y0 + dyi - 1, b0,
                        &fullA[st]);
          }
        }
      }
      if (!ok) {
        atomicExch(err, 1);
        bad = 1;
      }
      // the copies issued last land before the shared memory is released
      for (int i = q > WB_SLOTS ? q - WB_SLOTS : 0; i < q; i++)
        mbar_wait(&fullA[i % WB_SLOTS], (uint32_t)(i / WB_SLOTS) & 1u, kLim);
      for (int i = nb > 2 ? nb - 2 : 0; i < nb; i++) mbar_wait(&fullB[i & 1], (uint32_t)(i >> 1) & 1u, kLim);
    }
    __syncwarp();
  } else if (warp == 5) {
    const uint32_t idesc = idesc_bf16(N, 1, 1);
    const bool lead = elect_one();
    bool ok = true;
    int q = 0;
    for (int tl = 0; tl < mine && ok; tl++) {
      if (!mbar_wait_warp(&fullB[tl & 1], (uint32_t)(tl >> 1) & 1u, kLim)) {
        ok = false;
        break;
      }
      const uint32_t b0 = smem_u32(sB) + (uint32_t)(tl & 1) * BSLOT;
      for (int m = 0; m < MT; m++, q++) {
        const int st = q % WB_SLOTS;
        if (!mbar_wait_warp(&fullA[st], (uint32_t)(q / WB_SLOTS) & 1u, kLim)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t da = desc_mn<CH>(smem_u32(sA) + (uint32_t)st * WB_A, ABOX), db = desc_mn<CHB>(b0, BBOX);
        if (lead) {
#pragma unroll
          for (int ks = 0; ks < 8; ks++)  // 16 voxels each
            mma_bf16(tmem + (uint32_t)(m * N), da + (uint64_t)(ks * 2 * CH), db + (uint64_t)(ks * 2 * CHB), idesc,
                     (tl > 0 || ks > 0) ? 1u : 0u);
          mma_commit(&emptyA[st]);
        }
        __syncwarp();
      }
      if (ok && lead) mma_commit(&emptyB[tl & 1]);
      ok = __all_sync(0xffffffffu, ok && !bad);
    }
    if (!ok && lead) {
      atomicExch(err, 1);
      bad = 1;
    }
    if (lead) mma_commit(&acc_full);  // arrives once every MMA issued above has completed
    __syncwarp();
    mbar_wait(&acc_full, 0, kLim);
  } else {
    bool ready = mbar_wait(&acc_full, 0, kLim);
    if (!ready) {
      if (lane == 0) atomicExch(err, 1);
      bad = 1;
    }
    ready = !__any_sync(0xffffffffu, !ready || bad);
    tc_fence_after();
    if (ready && mine > 0) add_wgrad<CH, TPM, MT>(s, dyi, ck, warp, lane, tmem, dw);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, cols);
  }
}

// ---------------------------------------------------------------------------
// The weight gradient from halo tiles: as k_wgrad_box, but the nine taps of a
// step read one box, shifted by their rows: an M tile stacks 2 (CH 64) or 3
// (CH 32: dz = -1, 0, 1) taps, its atoms the distance of the taps' rows apart.
// 180 + 128 rows a step in place of 1152 + 128: TMA takes about 4 cycles a row
// whatever its width, which bounded k_wgrad_box.
// Now the MMA warp's issue does.
//
// Whole calls, box -> halo: 48 x 48, 131072 voxels 98 -> 69 us (64 -> 35 in the
// kernel); 112 x 48 157 -> 97; 32 x 80, 1048576 voxels 320 -> 193.
template <int CH, int CHB>
__global__ void __launch_bounds__(192, 1) k_wgrad_halo(const __grid_constant__ CUtensorMap tin,
                                                       const __grid_constant__ CUtensorMap tdy, ConvShape s, Halo H,
                                                       float *dw, int slices, int nstage, int *err) {
  extern __shared__ __align__(1024) uint8_t sm_raw[];
  uint8_t *sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
  constexpr int MAXST = 4;
  constexpr int MT = wh_mtiles<CH>(), TPM = CH == 64 ? 2 : 3;  // M tiles, taps per M tile
  constexpr uint32_t ROW = CH * 2, ABOX = halo_rows(1) * ROW, ASLOT = halo_bytes(1, CH), BBOX = 128 * CHB * 2;
  const int N = s.n, nbc = (N + CHB - 1) / CHB;
  const uint32_t STAGE = ASLOT + (uint32_t)nbc * BBOX;
  __shared__ uint64_t full[MAXST], empty[MAXST], acc_full;
  __shared__ uint32_t tbase;
  __shared__ volatile int bad;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int nchunk = (s.cin + CH - 1) / CH;
  const int grp = (int)blockIdx.x / slices, slice = (int)blockIdx.x % slices;
  const int dyi = grp / nchunk, ck = grp % nchunk;
  const int ntiles = H.count();
  const int mine = ntiles > slice ? (ntiles - 1 - slice) / slices + 1 : 0;
  const uint32_t cols = pow2_cols(MT * N);
  if (tid == 0) {
    for (int i = 0; i < nstage; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init_fence();
    bad = 0;
  }
  if (warp == 0) tmem_alloc(&tbase, cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  if (warp == 4) {
    if (lane == 0) {
      bool ok = true;
      int q = 0;
      for (; q < mine; q++) {
        const int st = q % nstage;
        if (q >= nstage && (!mbar_wait(&empty[st], (uint32_t)(q / nstage - 1) & 1u, kLim) || bad)) {
          ok = false;
          break;
        }
        int z0, x0, y, b;
        halo_origin(H, slice + q * slices, z0, x0, y, b);
        uint8_t *a = sm + (size_t)st * STAGE;
        mbar_expect_tx(&full[st], ABOX + (uint32_t)nbc * BBOX);
        tma_load_5d(a, &tin, ck * CH, z0 - 1, x0 - 1, y + dyi - 1, b, &full[st]);
        for (int c = 0; c < nbc; c++) tma_load_5d(a + ASLOT + c * BBOX, &tdy, c * CHB, z0, x0, y, b, &full[st]);
      }
      if (!ok) {
        atomicExch(err, 1);
        bad = 1;
      }
      // the copies issued last land before the shared memory is released
      for (int i = q > nstage ? q - nstage : 0; i < q; i++) mbar_wait(&full[i % nstage], (uint32_t)(i / nstage) & 1u, kLim);
    }
    __syncwarp();
  } else if (warp == 5) {
    const uint32_t idesc = idesc_bf16(N, 1, 1);
    const bool lead = elect_one();
    bool ok = true;
    int st = 0;
    uint32_t ph = 0;
    for (int q = 0; q < mine && ok; q++) {
      if (!mbar_wait_warp(&full[st], ph, kLim)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t a0 = smem_u32(sm) + (uint32_t)st * STAGE;
      const uint64_t db = desc_mn<CHB>(a0 + ASLOT, BBOX);
      const uint32_t first = q > 0 ? 1u : 0u;
      if (lead) {
#pragma unroll
        for (int m = 0; m < MT; m++) {
          // rows of the M tile's first tap, and how far on its second one lies
          const int t9 = m * TPM, r0 = t9 / 3 * HZS + t9 % 3, t1 = t9 + 1 < 9 ? t9 + 1 : t9;
          const uint64_t da = desc_halo<CH>(a0, (uint32_t)(t1 > t9 ? t1 / 3 * HZS + t1 % 3 - r0 : 1) * ROW);
#pragma unroll
          for (int ks = 0; ks < 8; ks++)  // 16 voxels each
            mma_bf16(tmem + (uint32_t)(m * N), da + (uint64_t)((r0 + ks * 2 * HZS) * (ROW >> 4)),
                     db + (uint64_t)(ks * 2 * CHB), idesc, ks > 0 ? 1u : first);
        }
        mma_commit(&empty[st]);
      }
      __syncwarp();
      if (++st == nstage) {
        st = 0;
        ph ^= 1u;
      }
      ok = __all_sync(0xffffffffu, ok && !bad);
    }
    if (!ok && lead) {
      atomicExch(err, 1);
      bad = 1;
    }
    if (lead) mma_commit(&acc_full);  // arrives once every MMA issued above has completed
    __syncwarp();
    mbar_wait(&acc_full, 0, kLim);
  } else {
    bool ready = mbar_wait(&acc_full, 0, kLim);
    if (!ready) {
      if (lane == 0) atomicExch(err, 1);
      bad = 1;
    }
    ready = !__any_sync(0xffffffffu, !ready || bad);
    tc_fence_after();
    if (ready && mine > 0) add_wgrad<CH, TPM, MT>(s, dyi, ck, warp, lane, tmem, dw);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, cols);
  }
}

// activations [nb][Y][X][Z][c] seen as (c, z, x, y, b), boxes of ch channels x 128 voxels
bool encode_box(CUtensorMap *m, const __nv_bfloat16 *p, const ConvShape &s, int c, int ch, const Box &B) {
  const cuuint64_t C2 = (cuuint64_t)c * 2;
  const cuuint64_t dims[5] = {(cuuint64_t)c, (cuuint64_t)s.Z, (cuuint64_t)s.X, (cuuint64_t)s.Y, (cuuint64_t)s.nb};
  const cuuint64_t strides[4] = {C2, (cuuint64_t)s.Z * C2, (cuuint64_t)s.X * s.Z * C2, (cuuint64_t)s.Y * s.X * s.Z * C2};
  const cuuint32_t box[5] = {(cuuint32_t)ch, (cuuint32_t)B.z, (cuuint32_t)B.x, (cuuint32_t)B.y, (cuuint32_t)B.b};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return tensor_map_encode()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<__nv_bfloat16 *>(p), dims, strides, box,
                             estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             ch == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t sm_count(int *n) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  return e == cudaSuccess ? cudaDeviceGetAttribute(n, cudaDevAttrMultiProcessorCount, dev) : e;
}

Halo make_halo(const ConvShape &s, int mv) {
  return Halo{mv, (s.Z + HZ - 1) / HZ, (s.X + HX * mv - 1) / (HX * mv), s.Y, s.nb};
}
long long halo_count(const ConvShape &s) {
  return (long long)((s.Z + HZ - 1) / HZ) * ((s.X + HX - 1) / HX) * s.Y * s.nb;
}
// Halo tiles are of one shape, so they cover small or odd planes with more tiles
// than the boxes.  Forward: worth it up to twice as many (48 -> 48: ratio 1, 131072
// voxels, 104 -> 79 us; ratio 1.6 68 -> 59; 2 77 -> 73 and 88 -> 99; 4 74 -> 101), and
// always where they fill one wave at most (ratio 4 with 128 tiles, 96 -> 96: 91 ->
// 71).  Weight gradient: up to 1.5 (1 93 -> 72; 1.43 86 -> 82; 1.6 55 -> 58; 2 58 -> 62).
bool use_halo_fwd(const ConvShape &s, const Box &B, int sms) {
  return halo_count(s) < 2ll * B.count() || halo_count(s) <= sms;
}
bool use_halo_wgrad(const ConvShape &s, const Box &B) { return 2 * halo_count(s) <= 3ll * B.count(); }
size_t halo_smem(const ConvShape &s, int ch, int mv, int nbst) {
  const size_t nchunk = (s.cin + ch - 1) / ch;
  return 2 * nchunk * halo_bytes(mv, ch) + nbst * ((nchunk * s.n * ch * 2 + 1023) / 1024 * 1024);
}
// M tiles a CTA takes at once, weight stages and CTAs per SM; false where they
// do not fit.  Two M tiles halve the weights' way from L2 (48 -> 48, 1024 M tiles:
// 99 -> 89 us; 256 of them 78 -> 73), two CTAs fill each other's waits (99 -> 89).
bool plan_halo(const ConvShape &s, int ch, Halo *H, int *nbst, int *per_sm) {
  for (int mv = s.X > HX ? 2 : 1; mv >= 1; mv--) {
    *H = make_halo(s, mv);
    if (2 * mv * s.n > 512) continue;
    for (*per_sm = 2; *per_sm >= 1; --*per_sm) {
      if (*per_sm == 2 && pow2_cols(2 * mv * s.n) > 256) continue;
      for (*nbst = CH_BST; *nbst >= 3; --*nbst)
        if (halo_smem(s, ch, mv, *nbst) <= (size_t)(*per_sm == 2 ? 110 : 222) * 1024) return true;
    }
  }
  return false;
}
// the box of a halo tile
Box halo_box(int mv) { return Box{HZS, HX * mv + 2, 1, 1, 0, 0, 0, 0}; }

bool shape_ok(const ConvShape &s) {
  return s.nb >= 1 && s.Y >= 1 && s.X >= 1 && s.Z >= 1 && s.cin >= 16 && s.cin % 16 == 0 && s.n >= 16 && s.n % 16 == 0 &&
         tensor_map_encode() != nullptr;
}

}  // namespace

bool conv_box_supported(const ConvShape &s) {
  Box B;
  return shape_ok(s) && s.n <= 256 && choose_box(s, &B);
}

size_t conv_box_wp_elems(int cin, int n) {
  const int ch = box_ch(cin);
  return (size_t)27 * ((cin + ch - 1) / ch) * n * ch;
}

cudaError_t conv_forward_box(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *wp, const float *bias,
                             void *out, int epi, int sign, int *err, cudaStream_t st) {
  Box B;
  if (!conv_box_supported(s) || !choose_box(s, &B) || (epi == 0 && !bias) || epi < 0 || epi > 2 || (sign != 1 && sign != -1))
    return cudaErrorNotSupported;
  const int ch = box_ch(s.cin);
  CUtensorMap m;
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  Halo H;
  int nbst, hper;
  if (use_halo_fwd(s, B, sms) && plan_halo(s, ch, &H, &nbst, &hper)) {
    if (!encode_box(&m, in, s, s.cin, ch, halo_box(H.mv))) return cudaErrorNotSupported;
    typedef void (*K)(const CUtensorMap, ConvShape, Halo, int, const __nv_bfloat16 *, const float *, void *, int, int *);
    K k = ch == 64 ? (epi == 0 ? k_conv_halo<64, 0> : epi == 1 ? k_conv_halo<64, 1> : k_conv_halo<64, 2>)
                   : (epi == 0 ? k_conv_halo<32, 0> : epi == 1 ? k_conv_halo<32, 1> : k_conv_halo<32, 2>);
    // (no more CTAs on an SM than its TMEM columns hold)
    const size_t smem = 1024 + std::max(halo_smem(s, ch, H.mv, nbst), (size_t)(hper == 2 ? 78 : 116) * 1024);
    e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)std::min(H.count(), sms * hper), 224, smem, st>>>(m, s, H, sign, wp, bias, out, nbst, err);
    return cudaGetLastError();
  }
  if (!encode_box(&m, in, s, s.cin, ch, B)) return cudaErrorNotSupported;
  typedef void (*K)(const CUtensorMap, ConvShape, Box, int, const __nv_bfloat16 *, const float *, void *, int, int *);
  K k = ch == 64 ? (epi == 0 ? k_conv_box<64, 0> : epi == 1 ? k_conv_box<64, 1> : k_conv_box<64, 2>)
                 : (epi == 0 ? k_conv_box<32, 0> : epi == 1 ? k_conv_box<32, 1> : k_conv_box<32, 2>);
  // two CTAs per SM where their accumulators fit the SM's 512 TMEM columns
  const int per_sm = pow2_cols(2 * s.n) <= 256 ? 2 : 1;
  const size_t stage = (size_t)(128 + s.n) * ch * 2, room = per_sm == 2 ? 110 * 1024 : 200 * 1024;
  const int nstage = (int)std::min<size_t>(8, room / stage);
  // (one per SM: more shared memory than two would leave)
  const size_t smem = 1024 + std::max(nstage * stage, per_sm == 2 ? (size_t)78 * 1024 : (size_t)116 * 1024);
  e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int grid = std::min(B.count(), sms * per_sm);
  k<<<(unsigned)grid, 192, smem, st>>>(m, s, B, sign, wp, bias, out, nstage, err);
  return cudaGetLastError();
}

bool wgrad_box_supported(const ConvShape &s) {
  Box B;
  if (!shape_ok(s) || !choose_box(s, &B)) return false;
  return (box_ch(s.cin) == 64 ? wb_mtiles<64>() : wb_mtiles<32>()) * s.n <= 512 && s.n <= 128;
}

cudaError_t conv_wgrad_box(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *dout, float *dw, int *err,
                           cudaStream_t st) {
  Box B;
  if (!wgrad_box_supported(s) || !choose_box(s, &B)) return cudaErrorNotSupported;
  const int ch = box_ch(s.cin), chb = box_ch(s.n);
  CUtensorMap mi, md;
  if (use_halo_wgrad(s, B)) {
    const Halo H = make_halo(s, 1);
    if (!encode_box(&mi, in, s, s.cin, ch, halo_box(1)) || !encode_box(&md, dout, s, s.n, chb, Box{HZ, HX, 1, 1, 0, 0, 0, 0}))
      return cudaErrorNotSupported;
    typedef void (*K)(const CUtensorMap, const CUtensorMap, ConvShape, Halo, float *, int, int, int *);
    K k = ch == 64 ? (chb == 64 ? k_wgrad_halo<64, 64> : k_wgrad_halo<64, 32>)
                   : (chb == 64 ? k_wgrad_halo<32, 64> : k_wgrad_halo<32, 32>);
    int sms = 0;
    cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    const int groups = 3 * ((s.cin + ch - 1) / ch), slices = std::max(1, std::min(H.count(), sms / groups));
    const size_t stage = halo_bytes(1, ch) + (size_t)((s.n + chb - 1) / chb) * 128 * chb * 2;
    const int nstage = (int)std::min<size_t>(4, 220 * 1024 / stage);
    // (one CTA per SM: more shared memory than two would leave)
    const size_t smem = 1024 + std::max(nstage * stage, (size_t)116 * 1024);
    e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)(groups * slices), 192, smem, st>>>(mi, md, s, H, dw, slices, nstage, err);
    return cudaGetLastError();
  }
  if (!encode_box(&mi, in, s, s.cin, ch, B) || !encode_box(&md, dout, s, s.n, chb, B)) return cudaErrorNotSupported;
  typedef void (*K)(const CUtensorMap, const CUtensorMap, ConvShape, Box, float *, int, int *);
  K k = ch == 64 ? (chb == 64 ? k_wgrad_box<64, 64> : k_wgrad_box<64, 32>)
                 : (chb == 64 ? k_wgrad_box<32, 64> : k_wgrad_box<32, 32>);
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  const int groups = 3 * ((s.cin + ch - 1) / ch);
  const int slices = std::max(1, std::min(B.count(), sms / groups));
  const size_t smem = 1024 + (size_t)WB_SLOTS * WB_A + 2 * (size_t)((s.n + chb - 1) / chb) * 128 * chb * 2;
  e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<(unsigned)(groups * slices), 192, smem, st>>>(mi, md, s, B, dw, slices, err);
  return cudaGetLastError();
}

}  // namespace xtc
