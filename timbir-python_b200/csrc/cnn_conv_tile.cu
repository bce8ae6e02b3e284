// cnn_conv_tile.cu -- 3x3x3 convolutions of the warm-start network on staged
// tiles (BF16 in, FP32 accumulation in TMEM).
//
// The gather kernel in cnn_conv.cu builds every A row (voxel x 64 K values)
// with per-thread loads: each input voxel is fetched 27 times.  Here a CTA
// owns an output tile of 128 x-voxels x TZ z-lines of one y-row, and a stage
// holds, for one 16-channel chunk, one of the three y-rows of the tile's input
// halo (130 x (TZ + 2) voxels, zero filled outside the volume) in shared
// memory, one 32-byte row per voxel (16 channels, the 32-byte swizzle), x
// fastest: row r = z' * TXS + x'.  In that layout the A operand of tap (dx, dz)
// for output line z is the run of 128 rows starting at (z + 1 + dz) * TXS + 1 +
// dx -- one shared-memory descriptor with a shifted start address.  No im2col
// gather is ever materialised.
//
// One MMA serves up to three output lines: staged z-line L feeds output lines
// L - 1, L and L + 1 through the taps dz = +1, 0, -1, so with the weights of
// those three taps stacked along N (the accumulators of consecutive output
// lines are consecutive TMEM columns) each (L, dy, dx) is one MMA of N = up to
// 3 cout -- half the MMAs, and half the A reads from shared memory, of one
// MMA per (output line, tap).  The accumulators are zeroed by the epilogue
// warps (tcgen05.st) and every MMA accumulates.
//
// Weights come pre-packed per 16-channel chunk as
// Wp[chunk][dy, dx][half][dz = +1, 0, -1][n][8] (offsets as the kernel applies
// them, i.e. mirrored for sign -1) and are copied with one bulk copy per stage.
// Up to six stages run ahead of the MMAs, across tile boundaries too
// (persistent CTAs), and the accumulators are double-buffered in TMEM so the
// epilogue of one tile overlaps the next.  Every wait is bounded and reports
// through *err.
//
// Shapes: X a multiple of 128, Z even, cin a multiple of 8, cout a multiple of
// 16 up to 64.  Tiles are 4 z-lines high for cout <= 32 (stages of 25,600 +
// 288 cout bytes), else 2 (17,408 + 288 cout).  Other shapes use the box or the
// gather kernel.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "cnn_tc.cuh"
#include "xtg_cnn_internal.h"

namespace xtc {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encode();  // cnn_conv_box.cu

namespace {

constexpr int TX = 128, TXS = TX + 2;  // output x-voxels per tile, staged with one halo each side
constexpr int TN_MAX = 64;

// per tile height TZ (output z-lines): 4 for cout <= 32, else 2 (shared memory)
template <int TZ>
struct TileDims {
  static constexpr int TZS = TZ + 2;                   // staged z-lines
  static constexpr int ROWS = TZS * TXS;               // staged voxels of a y-row, one 32-byte row (16 channels) each
  static constexpr uint32_t A_STAGE = (ROWS * 32 + 1023) / 1024 * 1024;  // stages stay aligned to the swizzle atom
};

// K-major operand with 32-byte rows in the 32-byte swizzle (16-byte chunk
// index XOR address bit 7, as TMA's SWIZZLE_32B writes it): the two 8-element
// K halves of a row are one 16-byte unit apart, 8-row groups 256 bytes apart.
// The swizzle is a function of the absolute shared-memory address, so a
// descriptor may start at any row.
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)6 << 61);
}

// a stage's weights: nine taps of 16 channels
__host__ __device__ constexpr uint32_t b_stage_bytes(int n) { return 9u * (uint32_t)n * 32u; }

constexpr int TILE_LOADERS = 128;  // threads of warps 5-8 (eight warps: no faster over a whole pass)
constexpr int TILE_THREADS = 160 + TILE_LOADERS;
constexpr int TILE_STAGES = 6;     // at most; as many as shared memory holds
constexpr int TILE_AHEAD = 2;      // stages a loader has in flight before it waits for the oldest

// Persistent: each CTA walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// A stage is one (16-channel chunk, dy): the staged y-row y + dy and its nine
// taps' weights.  Warps 5-8 copy it in with 16-byte asynchronous copies (a row
// is two of them; zero filled outside the volume), several stages ahead, and
// publish it to the tensor core's proxy once it has landed; warp 4 issues the
// MMAs; the accumulators alternate between two TMEM
// buffers, so warps 0-3 (TMEM lanes 32w .. 32w + 31) drain tile i while tile
// i + 1 is computed.
//
// What bounds it: the copies and the MMAs about equally (with either left out
// 1.25 and 1.17 ms of 1.27 at 512^2 x 64 voxels, 32 -> 32 channels).  As one TMA
// box a chunk (2340 rows of 32 bytes for TZ 4) the copies took 3.4 cycles a
// row and set the time, 1.86 ms; 80 -> 32 4.21 -> 2.85 ms, 48 -> 48 at half the
// resolution 496 -> 414 us.
//
// CAT: the input is the concatenation of a 2x nearest upsampling (the first ca
// channels, read from the coarse volume `up`) and `in` (the others); it is
// never formed.  At 512^2 x 64 forming it took 0.85 ms for the 80-channel
// level and 1.02 ms in all; read in place the 80 -> 32 convolution takes the
// same time.
//
// EPI 3 (inference's last layer): the 1x1 head on the rounded outputs, added in
// the order of k_head, in place of storing them (k_head took 0.21 ms at 512^2 x 64,
// the stores it read about as much).
//
// With the MMAs issued from a warp-uniform loop and whole sectors stored 32 -> 32
// takes 1.23 ms (1.27 before), 80 -> 32 2.55 (2.86), 48 -> 48 at half the
// resolution 0.36 (0.41).  Alone the copies, the MMAs (about 65 cycles each, near
// what reading A's 4 KB from shared memory takes) and the epilogue need 0.9, 0.85
// and 0.6 ms of the 1.23.
template <int EPI, int TZ, bool CAT>
__global__ void __launch_bounds__(TILE_THREADS, 1)
    k_conv_tile(const __nv_bfloat16 *__restrict__ in, const __nv_bfloat16 *__restrict__ up, int ca, ConvShape s,
                const __nv_bfloat16 *__restrict__ wp,
                const float *__restrict__ bias, void *out, TileHead hd, int nstage, int *err) {
  using D = TileDims<TZ>;
  constexpr int TZS = D::TZS;
  extern __shared__ __align__(1024) uint8_t sm[];
  const int N = s.n;
  const uint32_t BB = b_stage_bytes(N), STAGE = D::A_STAGE + (BB + 1023u) / 1024u * 1024u;
  __shared__ uint64_t full[TILE_STAGES], empty[TILE_STAGES], acc_full[2], acc_empty[2], done;
  __shared__ uint32_t tbase;
  __shared__ volatile int bad;
  __shared__ __align__(16) float sbias[64], shead[64];
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int nchunk = (s.cin + 15) >> 4;
  const int XT = s.X / TX, ZT = s.Z / TZ;
  const int ntiles = XT * ZT * s.nb * s.Y;
  const int mine = ntiles > (int)blockIdx.x ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const uint32_t acc_cols = tmem_cols(2 * TZ * N);
  const long long lim = 1ll << 24;
  if (tid == 0) {
    for (int i = 0; i < nstage; i++) {
      mbar_init(&full[i], TILE_LOADERS + 1);  // each loader, and the weights' transaction
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
  if ((EPI == 0 || EPI == 3) && tid < N) sbias[tid] = bias[tid];
  if (EPI == 3 && tid < N) shead[tid] = hd.w[tid];
  if (warp == 0) tmem_alloc(&tbase, acc_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  if (warp < 4) {  // both accumulator buffers start at zero
    for (int col = 0; col < 2 * TZ * N; col += 16) tmem_st16_zero(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)col);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  auto tile_of = [&](int tl, int &x0, int &z0, int &y, int &b) {
    int t = (int)blockIdx.x + tl * (int)gridDim.x;
    x0 = (t % XT) * TX;
    t /= XT;
    z0 = (t % ZT) * TZ;
    t /= ZT;
    y = t % s.Y;
    b = t / s.Y;
  };
  const int nq = 3 * nchunk;  // stages of a tile
  if (warp >= 5) {
    const int lt = tid - 160;
    bool ok = true;
    int q = 0, st = 0, landed = 0;  // stages issued and published
    uint32_t ph = 1;                // parity of the stage's last release (none yet: passes)
    // This thread's copies, the same in every stage: (x, z, half) of the staged
    // y-row, the halves and z of one x next to each other in memory.  Source
    // and destination offsets are worked out once (done per stage they were
    // the kernel's bound), and which copies lie on the tile's edges.
    constexpr int NE = (TXS * TZS * 2 + TILE_LOADERS - 1) / TILE_LOADERS;
    const int cs = CAT ? s.cin - ca : s.cin;  // channels of `in`
    int off[NE], upo[CAT ? NE : 1];
    uint32_t dst[NE], have = 0, on_x0 = 0, on_x1 = 0, on_z0 = 0, on_z1 = 0, on_h1 = 0;
#pragma unroll
    for (int e = 0; e < NE; e++) {
      const int i = lt + e * TILE_LOADERS;
      const int xx = i / (TZS * 2), rem = i - xx * (TZS * 2), zz = rem >> 1, h = rem & 1, r = zz * TXS + xx;
      off[e] = (xx * s.Z + zz) * cs + 8 * h;
      // (x0 and z0 are even: voxel x0 - 1 + xx lies in coarse voxel x0 / 2 + floor((xx - 1) / 2))
      if (CAT) upo[e] = (((xx - 1) >> 1) * (s.Z >> 1) + ((zz - 1) >> 1)) * ca + 8 * h;
      dst[e] = (uint32_t)r * 32u + (uint32_t)((h ^ ((r >> 2) & 1)) << 4);
      if (xx < TXS) have |= 1u << e;
      if (xx == 0) on_x0 |= 1u << e;
      if (xx == TXS - 1) on_x1 |= 1u << e;
      if (zz == 0) on_z0 |= 1u << e;
      if (zz == TZS - 1) on_z1 |= 1u << e;
      if (h) on_h1 |= 1u << e;
    }
    // stages up to `upto` have landed for this thread: make them visible to the
    // async proxy and arrive
    auto publish = [&](int upto) {
      fence_async_smem();
      for (; landed < upto; landed++) mbar_arrive(&full[landed % nstage]);
    };
    for (int tl = 0; tl < mine && ok; tl++) {
      int x0, z0, y, b;
      tile_of(tl, x0, z0, y, b);
      // the copies inside the volume in x and z
      uint32_t inside = have;
      if (x0 == 0) inside &= ~on_x0;
      if (x0 + TX == s.X) inside &= ~on_x1;
      if (z0 == 0) inside &= ~on_z0;
      if (z0 + TZ == s.Z) inside &= ~on_z1;
      const __nv_bfloat16 *row = in + (((long long)b * s.Y + y - 1) * s.X + x0 - 1) * s.Z * cs + (z0 - 1) * cs - (CAT ? ca : 0);
      const long long ystep = (long long)s.X * s.Z * cs;
      int c = 0, dyi = 0;
      for (int k = 0; k < nq; k++) {
        if (!mbar_wait(&empty[st], ph, lim) || bad) {
          ok = false;
          break;
        }
        uint8_t *a = sm + (size_t)st * STAGE;
        if (lt == 0) {
          mbar_expect_tx(&full[st], BB);
          bulk_load(a + D::A_STAGE, wp + (size_t)k * (BB / 2), BB, &full[st]);
        }
        const int y2 = y + dyi - 1;
        uint32_t m = y2 >= 0 && y2 < s.Y ? inside : 0u;
        if (16 * c + 8 >= s.cin) m &= ~on_h1;  // a half chunk
        const bool coarse = CAT && 16 * c < ca;
        const __nv_bfloat16 *src =
            coarse ? up + (((long long)b * (s.Y >> 1) + (y2 >> 1)) * (s.X >> 1) + (x0 >> 1)) * (s.Z >> 1) * ca + (z0 >> 1) * ca + 16 * c
                   : row + dyi * ystep + 16 * c;
        const uint32_t sa = smem_u32(a);
#pragma unroll
        for (int e = 0; e < NE; e++) {
          const bool v = (m >> e) & 1u;
          const __nv_bfloat16 *g = v ? src + (CAT && coarse ? upo[CAT ? e : 0] : off[e]) : in;
          if (e + 1 < NE || ((have >> e) & 1u))
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa + dst[e]), "l"(g), "r"(v ? 16 : 0)
                         : "memory");
        }
        if (++dyi == 3) {
          dyi = 0;
          c++;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        q++;
        if (++st == nstage) {
          st = 0;
          ph ^= 1u;
        }
        if (q > TILE_AHEAD) {
          asm volatile("cp.async.wait_group %0;" ::"n"(TILE_AHEAD) : "memory");
          publish(q - TILE_AHEAD);
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    publish(q);
    if (!ok && lane == 0) {
      atomicExch(err, 1);
      bad = 1;
    }
    // the weights issued last land before the shared memory is released
    for (int i = q > nstage ? q - nstage : 0; i < q; i++) mbar_wait(&full[i % nstage], (uint32_t)(i / nstage) & 1u, lim);
  } else if (warp == 4) {
    const uint32_t idesc[3] = {idesc_bf16(N, 0, 0), idesc_bf16(2 * N, 0, 0), idesc_bf16(3 * N, 0, 0)};
    const bool lead = elect_one();
    bool ok = true;
    int st = 0;
    uint32_t ph = 0;
    for (int tl = 0; tl < mine && ok; tl++) {
      const int ab = tl & 1;
      if (!mbar_wait_warp(&acc_empty[ab], (uint32_t)(((tl >> 1) & 1) ^ 1), lim)) {
        ok = false;
        break;
      }
      const uint32_t acc = tmem + (uint32_t)(ab * TZ * N);
      for (int k = 0; k < nq; k++) {
        if (!mbar_wait_warp(&full[st], ph, lim)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // descriptors advance in 16-byte units: an A row by 2; a (dy, dx)
        // B block (2 halves x 3 dz x N rows x 16 bytes) by 6N, one dz block by N
        const uint32_t a0 = smem_u32(sm) + (uint32_t)st * STAGE;
        const uint64_t da0 = sdesc_sw32(a0);
        uint64_t db = sdesc(a0 + D::A_STAGE, (uint32_t)N * 48, 128);
        if (lead) {
#pragma unroll
          for (int dxi = 0; dxi < 3; dxi++) {
#pragma unroll
            for (int zl = 0; zl < TZS; zl++) {
              // staged line zl (z = z0 - 1 + zl) feeds output lines zl - 2 .. zl
              // (relative to z0) through dz = +1, 0, -1; keep those inside the tile
              const int zf = zl - 2 < 0 ? 0 : zl - 2, zt = zl > TZ - 1 ? TZ - 1 : zl;
              const int cnt = zt - zf + 1, blk = zf - (zl - 2);
              mma_bf16(acc + (uint32_t)(zf * N), da0 + (uint64_t)(2 * (zl * TXS + dxi)), db + (uint64_t)(blk * N),
                       idesc[cnt - 1], 1u);
            }
            db += (uint64_t)(6 * N);
          }
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
    mbar_wait(&done, 0, lim);  // every MMA issued above has completed
  } else {
    // epilogue: warp w drains accumulator rows (x) 32w .. 32w + 31
    for (int tl = 0; tl < mine; tl++) {
      const int ab = tl & 1;
      const bool gone = !mbar_wait(&acc_full[ab], (uint32_t)(tl >> 1) & 1u, lim) || bad;
      if (__any_sync(0xffffffffu, gone)) {
        if (lane == 0) atomicExch(err, 1);
        bad = 1;
        break;
      }
      tc_fence_after();
      int x0, z0, y, b;
      tile_of(tl, x0, z0, y, b);
      const size_t vox0 = (((size_t)b * s.Y + y) * s.X + x0 + warp * 32 + lane) * s.Z + z0;
      __align__(16) float yv[TZ];  // EPI 3: the head's outputs
#pragma unroll
      for (int zo = 0; zo < TZ; zo++) {
        const size_t vox = vox0 + zo;
        float acc = EPI == 3 ? hd.b[0] : 0.f;
        for (int n0 = 0; n0 < N; n0 += 16) {
          __align__(16) float v[16];
          tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((ab * TZ + zo) * N + n0), v);
          if (EPI == 2) {
            float *o = reinterpret_cast<float *>(out) + vox * N + n0;
            store32(o, *reinterpret_cast<const int4 *>(v), *reinterpret_cast<const int4 *>(v + 4));
            store32(o + 8, *reinterpret_cast<const int4 *>(v + 8), *reinterpret_cast<const int4 *>(v + 12));
          } else {
            __align__(16) __nv_bfloat16 h[16];
#pragma unroll
            for (int q = 0; q < 16; q++) {
              float t = v[q];
              if (EPI != 1) t = fmaxf(t + sbias[n0 + q], 0.f);
              h[q] = __float2bfloat16_rn(t);
            }
            if (EPI == 3) {
#pragma unroll
              for (int q = 0; q < 16; q++) acc += __bfloat162float(h[q]) * shead[n0 + q];
            } else {
              __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(out) + vox * N + n0;
              store32(o, *reinterpret_cast<const int4 *>(h), *reinterpret_cast<const int4 *>(h + 8));
            }
          }
        }
        if (EPI == 3) yv[zo] = acc / hd.scale;
      }
      if (EPI == 3) {  // (TZ 4)
        float *o = reinterpret_cast<float *>(out) + vox0;
        const float4 p = *reinterpret_cast<const float4 *>(hd.base + vox0);
        *reinterpret_cast<float4 *>(o) = make_float4(p.x + yv[0], p.y + yv[1], p.z + yv[TZ - 2], p.w + yv[TZ - 1]);
      }
      // the buffer starts the CTA's next tile at zero
      for (int col = 0; col < TZ * N; col += 16)
        tmem_st16_zero(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(ab * TZ * N + col));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[ab]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, acc_cols);
  }
}

// ---------------------------------------------------------------------------
// Weight gradient on staged tiles (cout = 32, cin a multiple of 16, X a
// multiple of 128, Z even):
//   dW[dy, dx, dz][ci][co] = sum_v dY[v][co] X[v + (dy, dx, dz)][ci]
//                          = sum_u dY[u - (dy, 0, 0)][co] X[u + (0, dx, dz)][ci]
// (dY and X are zero outside the volume, so the substitution v = u - dy
// drops nothing).  In the second form one MMA covers the three dy taps along
// M and the three dz taps along N.  A CTA walks tiles u = 128 x-voxels x 2
// z-lines of one y-row y0 and keeps D[(dy, co)][(dx, dz, ci)] for up to three
// 16-channel input chunks in TMEM over all its tiles.  Per tile it stages, by
// TMA, one 32-byte row (16 channels) per voxel:
//   A (M x K, MN-major): dY rows y0 + 1, y0, y0 - 1 (dy = -1, 0, +1) x 2
//     channel halves = 6 boxes of 2 x 128 rows, stacked along M at a uniform
//     atom stride (M = 96; the MMA's rows 96..127 read the next box and are
//     discarded);
//   B (N x K, MN-major): per input chunk, the X halo of row y0
//     (130 x-voxels x 4 z-lines, zero fill outside); for (dx, output line z)
//     the three z-lines z - 1, z, z + 1 (dz = -1, 0, +1) are atoms one z-line
//     (130 rows) apart, and dx shifts the start row.
// K is the x-voxel: 16 rows per MMA.  Warp 4 (one thread) issues the copies
// and MMAs through two stages; warps 0-2 (TMEM lanes = (dy, co)) add the
// accumulators into dw once at the end.  Every wait is bounded.
constexpr int WG_TZ = 2;                                 // output z-lines per tile
constexpr uint32_t WG_XB = (WG_TZ + 2) * TXS * 32;       // one X box: 16,640 bytes
constexpr uint32_t WG_XS = (WG_XB + 1023) / 1024 * 1024; // its stride in a stage
constexpr uint32_t WG_DB = WG_TZ * TX * 32;              // one dY box: 8,192 bytes
constexpr uint32_t WG_A = 6 * WG_DB;                     // 3 y-rows x 2 channel halves
constexpr int WG_CPG = 3;                                // input chunks per CTA: 3 x 144 TMEM columns
constexpr uint32_t WG_SLACK = 16384;                     // past the second stage
constexpr int WG_N = 48;                                 // 3 dz x 16 channels

__host__ __device__ constexpr uint32_t wg_stage(int cpg) { return WG_A + (uint32_t)cpg * WG_XS; }

// MN-major operand, 32-byte swizzle: 16-element (32-byte) rows, one per K
// index, 8-row groups 256 bytes apart (SBO); MN atoms of 16 elements `lbo`
// bytes apart (LBO).
__device__ __forceinline__ uint64_t sdesc_mn_sw32(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)6 << 61);
}

__global__ void __launch_bounds__(160, 1)
    k_wgrad_tile(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tdy, ConvShape s,
                 float *dw, int slices, int *err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t full[2], empty[2], acc_full;
  __shared__ uint32_t tbase;
  __shared__ volatile int bad;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int nchunk = s.cin >> 4;
  const int cpg = nchunk < WG_CPG ? nchunk : WG_CPG;
  const uint32_t STAGE = wg_stage(cpg);
  const int grp = (int)blockIdx.x / slices, slice = (int)blockIdx.x % slices;
  const int c0 = grp * cpg, nck = nchunk - c0 < cpg ? nchunk - c0 : cpg;
  const int XT = s.X / TX, ZT = s.Z / WG_TZ;
  const int ntiles = XT * ZT * s.nb * s.Y;
  const int mine = ntiles > slice ? (ntiles - 1 - slice) / slices + 1 : 0;
  const long long lim = 1ll << 24;
  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init_fence();
    bad = 0;
  }
  if (warp == 0) tmem_alloc(&tbase, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  const int ncols = nck * 3 * WG_N;
  if (warp < 4) {
    for (int col = 0; col < ncols; col += 16) tmem_st16_zero(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)col);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  auto tile_of = [&](int tl, int &x0, int &z0, int &y, int &b) {
    int t = slice + tl * slices;
    x0 = (t % XT) * TX;
    t /= XT;
    z0 = (t % ZT) * WG_TZ;
    t /= ZT;
    y = t % s.Y;
    b = t / s.Y;
  };
  if (warp == 4) {
    const bool lead = elect_one();
    bool ok = true;
    if (mine > 0) {
      const uint32_t idesc = idesc_bf16(WG_N, 1, 1);
      int issued = 0, landed = 0;  // tiles whose copies were issued, have landed
      auto load = [&](int q) {
        const int st = q & 1;
        int x0, z0, y, b;
        tile_of(q, x0, z0, y, b);
        uint8_t *g = sm + (size_t)st * STAGE;
        if (lead) {
          mbar_expect_tx(&full[st], 6 * WG_DB + (uint32_t)nck * WG_XB);
          // box j = dy + 1 holds dY row y0 - dy (zero fill outside)
          for (int j = 0; j < 3; j++)
            for (int h = 0; h < 2; h++) tma_load_5d(g + (j * 2 + h) * WG_DB, &tdy, 16 * h, x0, z0, y + 1 - j, b, &full[st]);
          for (int c = 0; c < nck; c++)
            tma_load_5d(g + WG_A + c * WG_XS, &tin, 16 * (c0 + c), x0 - 1, z0 - 1, y, b, &full[st]);
        }
        __syncwarp();
        issued++;
      };
      load(0);
      if (mine > 1) load(1);
      for (int q = 0; q < mine && ok; q++) {
        const int st = q & 1;
        if (!mbar_wait_warp(&full[st], (uint32_t)(q >> 1) & 1u, lim)) {
          ok = false;
          break;
        }
        landed++;
        tc_fence_after();
        const uint32_t g = smem_u32(sm) + (uint32_t)st * STAGE;
        const uint64_t da = sdesc_mn_sw32(g, WG_DB);
        if (lead) {
          for (int c = 0; c < nck; c++) {
            const uint64_t db = sdesc_mn_sw32(g + WG_A + (uint32_t)c * WG_XS, TXS * 32);
            const uint32_t acc = tmem + (uint32_t)(c * 3 * WG_N);
#pragma unroll
            for (int q3 = 0; q3 < 3; q3++)  // dx = q3 - 1
#pragma unroll
              for (int zo = 0; zo < WG_TZ; zo++)
#pragma unroll
                for (int ks = 0; ks < TX / 16; ks++)
                  mma_bf16(acc + (uint32_t)(q3 * WG_N), da + (uint64_t)(2 * (zo * TX + ks * 16)),
                           db + (uint64_t)(2 * (zo * TXS + ks * 16 + q3)), idesc, 1u);
          }
          mma_commit(&empty[st]);
        }
        __syncwarp();
        if (q >= 1 && q + 1 < mine) {
          // tile q + 1 reuses the stage of tile q - 1 once its MMAs are done
          if (!mbar_wait_warp(&empty[(q - 1) & 1], (uint32_t)((q - 1) >> 1) & 1u, lim)) {
            ok = false;
            break;
          }
          load(q + 1);
        }
      }
      // after a wait that gave up, let the copies already issued land before the
      // shared memory is released
      if (!ok)
        for (; landed < issued; landed++) mbar_wait(&full[landed & 1], (uint32_t)(landed >> 1) & 1u, lim);
    }
    if (!ok && lead) {
      atomicExch(err, 1);
      bad = 1;
    }
    if (lead) mma_commit(&acc_full);  // arrives once every MMA issued above has completed
    __syncwarp();
  } else {
    const bool ready = mbar_wait(&acc_full, 0, lim);
    if (!ready) {
      if (lane == 0) atomicExch(err, 1);
      bad = 1;
    }
    tc_fence_after();
    if (warp < 3 && ready && !bad && mine > 0) {
      // TMEM lane 32 w + co holds dy = w - 1, output channel co
      for (int c = 0; c < nck; c++)
        for (int q3 = 0; q3 < 3; q3++)
          for (int n0 = 0; n0 < WG_N; n0 += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((c * 3 + q3) * WG_N + n0), v);
            const int tap = warp * 9 + q3 * 3 + n0 / 16;
            float *o = dw + ((size_t)tap * s.cin + (size_t)(c0 + c) * 16) * 32 + lane;
#pragma unroll
            for (int i = 0; i < 16; i++) atomicAdd(o + (size_t)i * 32, v[i]);
          }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, 512);
  }
}

}  // namespace

// tile height for a shape: 4 z-lines when cout <= 32 and Z allows, else 2
static int tile_tz(const ConvShape &s) { return (s.n <= 32 && s.Z % 4 == 0) ? 4 : 2; }

bool wgrad_tile_supported(const ConvShape &s) {
  return s.nb >= 1 && s.Y >= 1 && s.X >= TX && s.X % TX == 0 && s.Z >= WG_TZ && s.Z % WG_TZ == 0 && s.cin >= 16 &&
         s.cin % 16 == 0 && s.n == 32 && (long long)(s.X / TX) * (s.Z / WG_TZ) * s.nb * s.Y < (1ll << 31) &&
         tensor_map_encode() != nullptr;
}

// activations [nb][Y][X][Z][c] seen as (c, x, z, y, b), boxes of 16 channels
static bool encode_act(CUtensorMap *m, const __nv_bfloat16 *p, const ConvShape &s, int c, int bx, int bz) {
  const cuuint64_t C2 = (cuuint64_t)c * 2;
  const cuuint64_t dims[5] = {(cuuint64_t)c, (cuuint64_t)s.X, (cuuint64_t)s.Z, (cuuint64_t)s.Y, (cuuint64_t)s.nb};
  const cuuint64_t strides[4] = {(cuuint64_t)s.Z * C2, C2, (cuuint64_t)s.X * s.Z * C2, (cuuint64_t)s.Y * s.X * s.Z * C2};
  const cuuint32_t box[5] = {16, (cuuint32_t)bx, (cuuint32_t)bz, 1, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return tensor_map_encode()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<__nv_bfloat16 *>(p), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t conv_wgrad_tile(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *dout, float *dw,
                            int *err, cudaStream_t st) {
  if (!wgrad_tile_supported(s)) return cudaErrorNotSupported;
  CUtensorMap mi, md;
  if (!encode_act(&mi, in, s, s.cin, TXS, WG_TZ + 2) || !encode_act(&md, dout, s, s.n, TX, WG_TZ))
    return cudaErrorNotSupported;
  const int nchunk = s.cin / 16, cpg = std::min(nchunk, WG_CPG);
  const int groups = (nchunk + cpg - 1) / cpg;
  static int sms = 0;
  cudaError_t e;
  if (!sms) {
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  }
  const long long ntiles = (long long)(s.X / TX) * (s.Z / WG_TZ) * s.nb * s.Y;
  const int slices = (int)std::max(1ll, std::min(ntiles, (long long)std::max(1, sms / groups)));
  const size_t smem = 2 * (size_t)wg_stage(cpg) + WG_SLACK;
  e = cudaFuncSetAttribute((const void *)k_wgrad_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_wgrad_tile<<<(unsigned)(groups * slices), 160, smem, st>>>(mi, md, s, dw, slices, err);
  return cudaGetLastError();
}

bool conv_tile_supported(const ConvShape &s) {
  return s.nb >= 1 && s.Y >= 1 && s.X >= TX && s.X % TX == 0 && s.Z >= 2 && s.Z % 2 == 0 && s.cin >= 8 &&
         s.cin % 8 == 0 && s.n >= 16 && s.n % 16 == 0 && s.n <= TN_MAX &&
         (long long)(s.X / TX) * (s.Z / 2) * s.nb * s.Y < (1ll << 31) && tensor_map_encode() != nullptr;
}

size_t conv_tile_wp_elems(int cin, int n) { return (size_t)((cin + 15) / 16) * 27 * 2 * n * 8; }

cudaError_t conv_forward_tile(const ConvShape &s, const __nv_bfloat16 *in, const __nv_bfloat16 *wp, const float *bias,
                              void *out, int epi, int sign, int *err, cudaStream_t st, const __nv_bfloat16 *up, int ca,
                              const TileHead &hd) {
  if (!conv_tile_supported(s) || (epi % 3 == 0 && !bias) || epi < 0 || epi > 3 || (sign != 1 && sign != -1) ||
      (reinterpret_cast<uintptr_t>(in) & 15))
    return cudaErrorNotSupported;
  if (up && (epi != 0 || ca < 16 || ca % 16 || s.cin <= ca || s.cin % 16 || s.Y % 2 || s.X % 2 || s.Z % 2 ||
             (reinterpret_cast<uintptr_t>(up) & 15)))
    return cudaErrorNotSupported;
  if (epi == 3 && (up || !hd.w || tile_tz(s) != 4 || ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(hd.base)) & 15)))
    return cudaErrorNotSupported;
  const int tz = tile_tz(s);
  typedef void (*K)(const __nv_bfloat16 *, const __nv_bfloat16 *, int, ConvShape, const __nv_bfloat16 *, const float *,
                    void *, TileHead, int, int *);
  K k;
  // the sign lives in the packed weights
  if (up)
    k = tz == 4 ? k_conv_tile<0, 4, true> : k_conv_tile<0, 2, true>;
  else if (epi == 3)
    k = k_conv_tile<3, 4, false>;
  else if (tz == 4)
    k = epi == 0 ? k_conv_tile<0, 4, false> : epi == 1 ? k_conv_tile<1, 4, false> : k_conv_tile<2, 4, false>;
  else
    k = epi == 0 ? k_conv_tile<0, 2, false> : epi == 1 ? k_conv_tile<1, 2, false> : k_conv_tile<2, 2, false>;
  const size_t stage =
      (size_t)(tz == 4 ? TileDims<4>::A_STAGE : TileDims<2>::A_STAGE) + (b_stage_bytes(s.n) + 1023) / 1024 * 1024;
  const int nstage = (int)std::min<size_t>(TILE_STAGES, (size_t)220 * 1024 / stage);
  const size_t smem = nstage * stage;
  cudaError_t e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  }
  const long long ntiles = (long long)(s.X / TX) * (s.Z / tz) * s.nb * s.Y;
  const unsigned grid = (unsigned)std::min<long long>(ntiles, sms);  // one CTA per SM (shared memory)
  k<<<grid, TILE_THREADS, smem, st>>>(in, up, ca, s, wp, bias, out, hd, nstage, err);
  return cudaGetLastError();
}

}  // namespace xtc
