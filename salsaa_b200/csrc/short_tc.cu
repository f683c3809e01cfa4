// short_tc.cu — fold over short witness rows on the tensor cores.
#include <cuda_runtime.h>

#include "short_tc.cuh"
#include "umma.cuh"

namespace salsaa {

namespace {

// s8 x s8 -> s32, K-major operands.
constexpr u32 IDESC_S8 = (2u << 4) | (1u << 7) | (1u << 10);
__host__ __device__ constexpr u32 idesc_s8(u32 M, u32 N) { return IDESC_S8 | ((N >> 3) << 17) | ((M >> 4) << 24); }

// ---------------------------------------------------------------------------
// Fold (src/subroutines/fold.rs:22-27) in coefficient form: with ternary
// challenges c_k and byte rows w_k, out = sum_k c_k w_k mod X^d + 1 is an
// exact integer product of negacyclic Toeplitz matrices (entries -1, 0, 1)
// with the rows, |out| <= 8 x 256 x 128 < 2^19: no transforms at all.  Per
// (row, 64 elements): M = 128 output positions, N = 64 elements, K = d
// positions, accumulated over the rows in TMEM.
//
// A Toeplitz tile's 8 x 16-byte core matrices depend on (position - K
// position) only, so a row's matrix is d / 4 blocks of 128 bytes in order of
// falling difference: with the 8-position groups of M reversed, the next
// group is the next block (stride 128) and the next K slice the block after
// it (256).  The rows arrive as byte tiles, operands as they lie.  Persistent
// CTAs: a warp copies tiles into a ring, a warp issues the MMAs, eight warps
// write the finished 64 elements as words, 256 contiguous bytes a warp.
// Bound by HBM: 8 bytes out and one per row in a coefficient, against 16 per
// row and 32 more for the slot-form fold and its inverse transform.
// ---------------------------------------------------------------------------
constexpr u32 FT_EPI = 256, FT_THREADS = FT_EPI + 64, FT_EL = 64;

template <u32 D>
struct FtGeom {
  static constexpr u32 MT = D / 128;                    // M tiles
  static constexpr u32 TZ = 32 * D;                     // Toeplitz blocks of a row
  static constexpr u32 TILE = FT_EL * D;                // one row's 64 elements
  static constexpr u32 STAGES = D == 128 ? 8 : 6;
  static constexpr u32 COLS = MT * FT_EL;               // TMEM columns of a unit
};

template <u32 D>
__global__ void __launch_bounds__(FT_THREADS, 1)
    fold_tc_kernel(C8Rows w, const int8_t* __restrict__ tz, u64 q, u64* __restrict__ out, u64* mag_or,
                   const u32* flag, u32* err) {
  using Geo = FtGeom<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[Geo::STAGES], empty_bar[Geo::STAGES], acc_full[2], acc_empty[2], tz_bar;
  __shared__ uint32_t tslot;
  if (*flag) return;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const u32 units = (u32)(w.width / FT_EL), rows = w.rows;
  uint8_t* const ring = smem + rows * Geo::TZ;
  if (tid == 0) {
    for (u32 i = 0; i < Geo::STAGES; i++) {
      umma::mbar_init(&full_bar[i], 1);
      umma::mbar_init(&empty_bar[i], 1);
    }
    for (u32 i = 0; i < 2; i++) {
      umma::mbar_init(&acc_full[i], 1);
      umma::mbar_init(&acc_empty[i], FT_EPI);
    }
    umma::mbar_init(&tz_bar, 1);
    umma::mbar_fence_init();
    umma::mbar_expect_tx(&tz_bar, rows * Geo::TZ);
    for (u32 k = 0; k < rows; k++) umma::bulk_g2s(smem + k * Geo::TZ, tz + k * Geo::TZ, Geo::TZ, &tz_bar);
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;

  if (warp == FT_EPI / 32) {
    bool ok = true;
    u32 it = 0, st = 0, par = 1;
    for (u32 unit = blockIdx.x; ok && unit < units; unit += gridDim.x)
      for (u32 k = 0; k < rows; k++, it++) {
        if (it >= Geo::STAGES && !(ok = umma::mbar_wait(&empty_bar[st], par, err, 41))) break;
        if (umma::elect_one()) {
          umma::mbar_expect_tx(&full_bar[st], Geo::TILE);
          umma::bulk_g2s(ring + st * Geo::TILE,
                         w.p + w.row[k] * w.stride + (w.off[k] + (u64)unit * FT_EL) * D, Geo::TILE, &full_bar[st]);
        }
        __syncwarp();
        if (++st == Geo::STAGES) {
          st = 0;
          par ^= 1;
        }
      }
    for (u32 c = it >= Geo::STAGES ? it - Geo::STAGES : 0; c < it; c++)
      umma::mbar_wait(&full_bar[c % Geo::STAGES], (c / Geo::STAGES) & 1, err, 42);
  } else if (warp == FT_EPI / 32 + 1) {
    const u32 idesc = idesc_s8(128, FT_EL);
    const uint64_t bd0 = umma::desc_kmajor(umma::smem_u32(ring), 1024, 128);
    bool ok = umma::mbar_wait(&tz_bar, 0, err, 43);
    u32 it = 0, ui = 0, st = 0, par = 0;
    for (u32 unit = blockIdx.x; ok && unit < units; unit += gridDim.x, ui++) {
      const u32 nb = ui & 1;
      if (ui >= 2 && !(ok = umma::mbar_wait(&acc_empty[nb], ((ui >> 1) - 1) & 1, err, 44))) break;
      umma::fence_after_sync();
      for (u32 k = 0; k < rows; k++, it++) {
        if (!(ok = umma::mbar_wait(&full_bar[st], par, err, 45))) break;
        umma::fence_after_sync();
        const uint64_t bd = bd0 + st * (Geo::TILE >> 4);
        const uint64_t ad = umma::desc_kmajor(umma::smem_u32(smem) + k * Geo::TZ, 256, 128);
        if (umma::elect_one()) {
#pragma unroll
          for (u32 mt = 0; mt < Geo::MT; mt++)
#pragma unroll
            for (u32 ks = 0; ks < D / 32; ks++)
              umma::mma_i8_u(tmem + nb * Geo::COLS + mt * FT_EL, ad + ((D - 128 - 128 * mt) + 32 * ks), bd + ks * 128,
                             idesc, (k > 0 || ks > 0) ? 1u : 0u);
          umma::commit(&empty_bar[st]);
          if (k + 1 == rows) umma::commit(&acc_full[nb]);
        }
        __syncwarp();
        if (++st == Geo::STAGES) {
          st = 0;
          par ^= 1;
        }
      }
    }
    for (u32 c = it >= Geo::STAGES ? it - Geo::STAGES : 0; c < it; c++)
      umma::mbar_wait(&empty_bar[c % Geo::STAGES], (c / Geo::STAGES) & 1, err, 46);
  } else {
    // TMEM lane r holds position 8 (15 - r / 8) + r % 8 of the M tile; the two
    // warps of a lane take 32 elements each
    const u32 r = (warp & 3) * 32 + lane, p0 = 8 * (15 - r / 8) + r % 8, half = warp >> 2;
    u32 ui = 0, mag = 0;
    for (u32 unit = blockIdx.x; unit < units; unit += gridDim.x, ui++) {
      const u32 nb = ui & 1;
      const bool ok = umma::mbar_wait(&acc_full[nb], (ui >> 1) & 1, err, 47);
      if (!__all_sync(0xffffffffu, ok)) break;
      umma::fence_after_sync();
#pragma unroll
      for (u32 mt = 0; mt < Geo::MT; mt++) {
        const u32 tb = tmem + (((warp & 3) * 32) << 16) + nb * Geo::COLS + mt * FT_EL + half * 32;
        uint32_t v[32];
        {
          uint32_t a[16], b[16];
          umma::tmem_ld16(tb, a);
          umma::tmem_ld16(tb + 16, b);
          umma::tmem_wait_ld();
#pragma unroll
          for (u32 i = 0; i < 16; i++) {
            v[i] = a[i];
            v[16 + i] = b[i];
          }
        }
        if (mt + 1 == Geo::MT) {
          umma::fence_before_sync();
          umma::mbar_arrive(&acc_empty[nb]);
        }
        u64* dst = out + ((u64)unit * FT_EL + half * 32) * D + mt * 128 + p0;
#pragma unroll
        for (u32 i = 0; i < 32; i++) {
          const int c = (int)v[i];
          mag |= (u32)(c < 0 ? -c : c);
          dst[(u64)i * D] = (u64)(long long)c + (c < 0 ? q : 0);
        }
      }
    }
    if (mag_or) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mag |= __shfl_xor_sync(0xffffffffu, mag, o);
      if (lane == 0 && mag) atomicOr((unsigned long long*)mag_or, (unsigned long long)mag);
    }
  }
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
  if (tid == 0) umma::mbar_wait(&tz_bar, 0, err, 48);
}

// Byte (r8, kk) of block b of row k: coefficient delta = d - 8 - 8 b + r8 - kk
// of the challenge, negated and moved by d when delta < 0.
__global__ void fold_chal_tz_kernel(const DevState* ds, u32 round, u32 rows, u32 d, u64 q, u64* c, int8_t* tz) {
  const u64 key = prf_key(ds->seed, domain_id(DOM_FOLD, round, 0));
  const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < rows * d) {
    const u64 v = __umul64hi(prf_at(key, t), 3);
    c[t] = v == 0 ? q - 1 : (v == 1 ? 0 : 1);
  }
  if (t >= rows * 32 * d) return;
  const u32 k = t / (32 * d), b = t / 128 % (d / 4), r8 = t / 16 % 8, kk = t % 16;
  const int delta = (int)(d - 8 - 8 * b + r8) - (int)kk;
  int v = 0;
  if (delta > -(int)d && delta < (int)d) {
    const u32 j = (u32)(delta < 0 ? delta + (int)d : delta);
    v = (int)__umul64hi(prf_at(key, (u64)k * d + j), 3) - 1;
    if (delta < 0) v = -v;
  }
  tz[t] = (int8_t)v;
}

}  // namespace

int launch_fold_challenge_tz(const DevState* ds, u32 round, u32 rows, u32 d, u64 q, u64* c_coef, int8_t* tz,
                             cudaStream_t st) {
  const u32 tot = rows * 32 * d;
  fold_chal_tz_kernel<<<(tot + 255) / 256, 256, 0, st>>>(ds, round, rows, d, q, c_coef, tz);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "fold_challenge_tz");
}

bool fold_tc_ok(const C8Rows& w, u32 d) {
  return (d == 128 || d == 256) && w.rows >= 1 && w.rows <= 8 && w.width >= FT_EL && w.width % FT_EL == 0;
}

int launch_fold_tc(const C8Rows& w, u32 d, u64 q, const int8_t* tz, u64* out, u64* mag_or, const u32* flag,
                   cudaStream_t st) {
  if (!fold_tc_ok(w, d) || !flag) return salsaa_set_error(-2, "fold_tc: rows outside the byte-tile path");
  const size_t smem = (size_t)w.rows * 32 * d + (d == 128 ? (size_t)FtGeom<128>::STAGES * FtGeom<128>::TILE
                                                          : (size_t)FtGeom<256>::STAGES * FtGeom<256>::TILE);
  const u64 units = w.width / FT_EL;
  const unsigned grid = (unsigned)(units < 148 ? units : 148);
  auto kern = d == 128 ? fold_tc_kernel<128> : fold_tc_kernel<256>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "fold_tc smem attribute");
  kern<<<grid, FT_THREADS, smem, st>>>(w, tz, q, out, mag_or, flag, tc_error_word());
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "fold_tc launch");
}

}  // namespace salsaa
