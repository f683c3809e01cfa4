// short_tc.cu — fold, projection and statement rows over short witness rows on the tensor cores.
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
// exact integer product of negacyclic Toeplitz matrices with the rows, no
// transforms at all: |out| <= 8 x 256 x 128 <= 2^18 for the proof's ternary
// challenges and, since launch_fold_words_tz takes coefficients up to 127,
// <= 8 x 256 x 127 x 128 < 2^25 for given ones, either way within the s32 sums.  Per
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
constexpr u32 FT_EPI = 256, FT_THREADS = FT_EPI + 64, FT_EL = 64, FT_MAX_ROWS = 8;

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
    fold_tc_kernel(C8Rows w, const int8_t* __restrict__ tz, u64 q, u64 nout, u64* __restrict__ out, u64* mag_or,
                   const u32* flag, u32* err) {
  pdl_wait();
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
        const u64 e0 = (u64)unit * FT_EL + half * 32;
        const u32 left = e0 + 32 <= nout ? 32 : (e0 < nout ? (u32)(nout - e0) : 0);
        u64* dst = out + e0 * D + mt * 128 + p0;
#pragma unroll
        for (u32 i = 0; i < 32; i++) {
          const int c = (int)v[i];
          mag |= (u32)(c < 0 ? -c : c);
          if (i < left) dst[(u64)i * D] = (u64)(long long)c + (c < 0 ? q : 0);
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
  pdl_wait();
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

// ---------------------------------------------------------------------------
// Statement rows (the scalar rows of parallel_dot_series_matrix,
// src/arithmetic.rs:459-505) over byte rows.  Per (byte row, 128 positions,
// element block of one s_hi factor or a part of it): D[position][8 j + x] =
// sum_i w(i, position) byte_x(s_lo_j(i)), M = 128 positions (the byte tile
// MN-major), N = 8 columns a row, K = elements; the row's sum is
// s_hi sum_x 2^(8 x) D_x.  A CTA takes a run of items in element order and
// keeps the residues in registers (lane = position, 8 rows a warp) until the
// (byte row, positions) changes, then adds them to the accumulators.  Where
// sc_umma_kernel turns every value into three byte limbs, here both operands
// are bulk copies.  Bound by the copies' latency and L2 traffic: 16 KB per 64
// elements with 16 rows; a launch takes two groups of 16 rows.  Together with
// the products that the proof no longer recomputes (<projected_lhs, folded> is
// a combination of <projected_lhs, w_k>): 1222 -> 374 us of an 8-round proof
// over 2^19 elements, d = 128.
// ---------------------------------------------------------------------------
constexpr u32 ST_EPI = 256, ST_THREADS = ST_EPI + 64, ST_STAGES = 8;
constexpr u32 ST_A = 64 * 128, ST_STAGE = ST_A + 64 * 128;

__global__ void __launch_bounds__(ST_THREADS, 1)
    sc_tc_kernel(Sc8Rows w, u32 rows, u32 d, u32 Bw, u32 nhi, u32 split, ScRange rg, const u64* s_hi, ModQ M,
                 u64* acc, const uint8_t* __restrict__ img, u32* err) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[ST_STAGES], empty_bar[ST_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tslot;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const u32 npb = d / 128, per = nhi * split, items = w.w.rows * npb * per * rg.groups();
  const u32 i0 = (u32)((u64)blockIdx.x * items / gridDim.x), i1 = (u32)((u64)(blockIdx.x + 1) * items / gridDim.x);
  const u32 steps = Bw / 64 / split;
  // item: (group of scalar rows, byte row, positions, elements)
  auto brow = [&](u32 rp) { return rp / npb % w.w.rows; };
  auto group = [&](u32 rp) { return rp / npb / w.w.rows; };
  auto open = [&](u32 item) { return *w.wide[w.dst[brow(item / per)]] == 0; };
  auto ncol = [&](u32 g) { return (rg.rows(g) * 8 + 15) / 16 * 16; };  // N, whole 16-column groups
  if (tid == 0) {
    for (u32 i = 0; i < ST_STAGES; i++) {
      umma::mbar_init(&full_bar[i], 1);
      umma::mbar_init(&empty_bar[i], 1);
    }
    for (u32 i = 0; i < 2; i++) {
      umma::mbar_init(&acc_full[i], 1);
      umma::mbar_init(&acc_empty[i], ST_EPI);
    }
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;

  if (warp == ST_EPI / 32) {
    bool ok = true;
    u32 it = 0, st = 0, par = 1;
    for (u32 item = i0; ok && item < i1; item++) {
      if (!open(item)) continue;
      const u32 hs = item % per, rp = item / per, pb = rp % npb, r = brow(rp), g = group(rp), np = ncol(g);
      const u32 e0 = hs / split * Bw + hs % split * steps * 64, l0 = hs % split * steps * 64;
      const int8_t* src = w.w.p + w.w.row[r] * w.w.stride + (w.w.off[r] + e0) * d + pb * ST_A;
      for (u32 c = 0; c < steps; c++, it++) {
        if (it >= ST_STAGES && !(ok = umma::mbar_wait(&empty_bar[st], par, err, 51))) break;
        if (umma::elect_one()) {
          uint8_t* stage = smem + st * ST_STAGE;
          umma::mbar_expect_tx(&full_bar[st], ST_A + 4 * np * 16);
          umma::bulk_g2s(stage, src + (u64)c * 64 * d, ST_A, &full_bar[st]);
          const uint8_t* im = img + (u64)g * Bw * 128 + (u64)(l0 / 16 + 4 * c) * 2048;
          for (u32 j = 0; j < 4; j++)
            umma::bulk_g2s(stage + ST_A + j * 2048, im + j * 2048, np * 16, &full_bar[st]);
        }
        __syncwarp();
        if (++st == ST_STAGES) {
          st = 0;
          par ^= 1;
        }
      }
    }
    for (u32 c = it >= ST_STAGES ? it - ST_STAGES : 0; c < it; c++)
      umma::mbar_wait(&full_bar[c % ST_STAGES], (c / ST_STAGES) & 1, err, 52);
  } else if (warp == ST_EPI / 32 + 1) {
    // A: s8, MN-major (position slices 1024 apart, 8-element blocks 128);
    // B: u8, K-major
    const uint64_t ad0 = umma::desc_kmajor(umma::smem_u32(smem), 128, 1024);
    const uint64_t bd0 = umma::desc_kmajor(umma::smem_u32(smem + ST_A), 2048, 128);
    bool ok = true;
    u32 it = 0, ui = 0, st = 0, par = 0;
    for (u32 item = i0; ok && item < i1; item++) {
      if (!open(item)) continue;
      const u32 nb = ui & 1;
      const u32 np = ncol(group(item / per));
      const u32 idesc = (2u << 4) | (1u << 7) | (1u << 15) | ((np >> 3) << 17) | ((128u >> 4) << 24);
      if (ui >= 2 && !(ok = umma::mbar_wait(&acc_empty[nb], ((ui >> 1) - 1) & 1, err, 53))) break;
      umma::fence_after_sync();
      for (u32 c = 0; c < steps; c++, it++) {
        if (!(ok = umma::mbar_wait(&full_bar[st], par, err, 54))) break;
        umma::fence_after_sync();
        const uint64_t so = (uint64_t)st * (ST_STAGE >> 4);
        if (umma::elect_one()) {
#pragma unroll
          for (u32 ks = 0; ks < 2; ks++)
            umma::mma_i8_u(tmem + nb * 128, ad0 + so + ks * 32, bd0 + so + ks * 256, idesc,
                           (c > 0 || ks > 0) ? 1u : 0u);
          umma::commit(&empty_bar[st]);
          if (c + 1 == steps) umma::commit(&acc_full[nb]);
        }
        __syncwarp();
        if (++st == ST_STAGES) {
          st = 0;
          par ^= 1;
        }
      }
      ui++;
    }
    for (u32 c = it >= ST_STAGES ? it - ST_STAGES : 0; c < it; c++)
      umma::mbar_wait(&empty_bar[c % ST_STAGES], (c / ST_STAGES) & 1, err, 55);
  } else {
    const u32 m = (warp & 3) * 32 + lane, ch = warp >> 2;  // position; rows 8 ch .. + 7
    const u64 q = M.q, p32 = ((u64)1 << 32) % q;
    u64 sum[8];
#pragma unroll
    for (u32 j = 0; j < 8; j++) sum[j] = 0;
    u32 ui = 0;
    for (u32 item = i0; item < i1; item++) {
      const u32 hs = item % per, rp = item / per, grp = group(rp), nrow = rg.rows(grp), j0 = rg.first(grp) + 8 * ch;
      if (open(item)) {
        const u32 nb = ui & 1;
        const bool ok = umma::mbar_wait(&acc_full[nb], (ui >> 1) & 1, err, 56);
        if (!__all_sync(0xffffffffu, ok)) break;
        umma::fence_after_sync();
        const u32 tb = tmem + (((warp & 3) * 32) << 16) + nb * 128 + ch * 64;
        uint32_t v[4][16];
#pragma unroll
        for (u32 g = 0; g < 4; g++)
          if (8 * ch + 2 * g < nrow) umma::tmem_ld16(tb + g * 16, v[g]);
        umma::tmem_wait_ld();
        umma::fence_before_sync();
        umma::mbar_arrive(&acc_empty[nb]);
        ui++;
#pragma unroll
        for (u32 j = 0; j < 8; j++) {
          if (8 * ch + j < nrow) {
            const uint32_t* D = &v[j / 2][8 * (j & 1)];
            // |D_x| <= 2048 x 255 x 128 < 2^26
            const long long lo = (long long)(int)D[0] + ((long long)(int)D[1] << 8) + ((long long)(int)D[2] << 16) +
                                 ((long long)(int)D[3] << 24);
            const long long hi = (long long)(int)D[4] + ((long long)(int)D[5] << 8) + ((long long)(int)D[6] << 16);
            // |hi| < 2^43 < q; |lo| < 2^51 <= 16 q
            u64 x = mul_mod(M, hi < 0 ? (u64)(hi + (long long)q) : (u64)hi, p32);
            x = reduce64(M, x + (u64)(lo + (long long)(16 * q)));
            x = mul_mod(M, x, __ldg(s_hi + (u64)(j0 + j) * nhi + hs / split));
            sum[j] = add_mod(sum[j], x, q);
          }
        }
      }
      if (item + 1 == i1 || rp != (item + 1) / per) {  // the run of this byte row and these positions ends
        const u32 pb = rp % npb, r = brow(rp), k = w.dst[r];
        const u64 sc = ((u64)1 << w.shift[r]) % q;
#pragma unroll
        for (u32 j = 0; j < 8; j++) {
          if (8 * ch + j < nrow && sum[j])
            atomic_add_mod(acc + ((u64)(j0 + j) * rows + k) * d + pb * 128 + m, mul_mod(M, sum[j], sc), q, true);
          sum[j] = 0;
        }
      }
    }
  }
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

// fold_chal_tz_kernel's Toeplitz blocks of given challenges c (rows x d words).
__global__ void fold_words_tz_kernel(const u64* c, u32 rows, u32 d, u64 q, int8_t* tz, u32* wide) {
  pdl_wait();
  const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= rows * 32 * d) return;
  const u32 k = t / (32 * d), b = t / 128 % (d / 4), r8 = t / 16 % 8, kk = t % 16;
  const int delta = (int)(d - 8 - 8 * b + r8) - (int)kk;
  long long v = 0;
  if (delta > -(int)d && delta < (int)d) {
    const u64 x = c[(u64)k * d + (u32)(delta < 0 ? delta + (int)d : delta)];
    v = (long long)(x - (x > (q >> 1) ? q : 0));
    if (v > 127 || v < -127) *wide = 1;
    if (delta < 0) v = -v;
  }
  tz[t] = (int8_t)v;
}

// ---------------------------------------------------------------------------
// Words to byte tiles.  A warp takes 16 elements x 16 positions: eight lanes
// read the 128 bytes of an element's 16 words, and after each lane has put
// its bytes together (two a word pair, then eight lanes' by shuffles) every
// 16-byte unit is one store and the warp's 256 bytes are one run.  Nine
// bytes a value at 4.8 .. 5.1 TB/s of DRAM and 58% of the issue slots.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) words_to_c8_kernel(RowSet src, u64 width, u64 wpad, u32 d, u64 q, int8_t* c8,
                                                          u32* wide) {
  pdl_wait();
  const u32 lane = threadIdx.x & 31, k = blockIdx.y, npg = d / 16;
  const u64 tasks = wpad / 16 * npg, half_q = q >> 1;
  const u64* x = src.p[k];
  int8_t* out = c8 + (u64)k * wpad * d;
  for (u64 t = (u64)blockIdx.x * 8 + (threadIdx.x >> 5); t < tasks; t += (u64)gridDim.x * 8) {
    // a warp that meets a wide value stops, and so do those that see the flag
    if (__any_sync(0xffffffffu, *(volatile u32*)wide != 0)) break;
    bool bad = false;
    const u64 eg = t / npg;
    const u32 pg = (u32)(t % npg);
    ulonglong2 v[4];
#pragma unroll
    for (u32 i = 0; i < 4; i++) {
      const u64 e = eg * 16 + 4 * i + (lane >> 3);
      v[i] = e < width ? __ldg((const ulonglong2*)(x + e * d + pg * 16 + 2 * (lane & 7))) : make_ulonglong2(0, 0);
    }
#pragma unroll
    for (u32 i = 0; i < 4; i++) {
      const u64 a = v[i].x + 128 - (v[i].x > half_q ? q : 0), b = v[i].y + 128 - (v[i].y > half_q ? q : 0);
      bad |= (a | b) > 255;
      u32 p = ((u32)a & 255) | ((u32)b & 255) << 8;  // two bytes, then four, eight, sixteen
      p ^= 0x8080u;
      p |= __shfl_down_sync(0xffffffffu, p, 1) << 16;
      const u32 p1 = __shfl_down_sync(0xffffffffu, p, 2);
      const u32 p2 = __shfl_down_sync(0xffffffffu, p, 4);
      const u32 p3 = __shfl_down_sync(0xffffffffu, p, 6);
      if ((lane & 7) == 0) {
        const u64 e = eg * 16 + 4 * i + (lane >> 3);
        *(uint4*)(out + c8_offset(e, pg * 16, d)) = make_uint4(p, p1, p2, p3);
      }
    }
    if (__any_sync(0xffffffffu, bad)) {
      // an atomic: stores and the other warps' polls of one address made the
      // attempt on 8 rows x 20001 x 128 wide values take 214 us, this 35
      if (lane == 0) atomicOr(wide, 1u);
      break;
    }
  }
}

// ---------------------------------------------------------------------------
// Projection (project, src/subroutines/project.rs:50-103) over byte rows: per
// (chunk of cw elements, 128 positions) D[position][J row] = sum_l w(l,
// position) J[row][l], M = 128 positions (the byte tile MN-major), N = 256 J
// rows (their image K-major) or a part of them, K = elements, one item per
// unit of a persistent grid, two accumulators.  A lane holds one position, so
// each column is stored as whole sectors.  Bound by the words it writes (8
// bytes for 256 / rows input bytes) and, with long chunks, by its copies from
// L2: 24 KB per 64 elements.  Where project_umma_kernel converts the witness
// words itself, here both operands are bulk copies: 789 -> 203 us of an
// 8-round proof over 2^19 elements, d = 128.
// ---------------------------------------------------------------------------
constexpr u32 PT_EPI = 256, PT_THREADS = PT_EPI + 64, PT_STAGES = 8, PT_ROWS = 256;
constexpr u32 PT_A = 64 * 128, PT_STAGE = PT_A + 64 * PT_ROWS;

__global__ void __launch_bounds__(PT_THREADS, 1)
    project_tc_kernel(C8Rows w, u32 d, u64 q, u32 cw, u32 nch, u32 nsplit, const int8_t* __restrict__ Jc,
                      u64* __restrict__ out, const u32* wide, u32* err) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[PT_STAGES], empty_bar[PT_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tslot;
  if (*(volatile const u32*)wide) return;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const u32 npb = d / 128, items = w.rows * nch * npb * nsplit, nr = PT_ROWS / nsplit, steps = cw / 64;
  if (tid == 0) {
    for (u32 i = 0; i < PT_STAGES; i++) {
      umma::mbar_init(&full_bar[i], 1);
      umma::mbar_init(&empty_bar[i], 1);
    }
    for (u32 i = 0; i < 2; i++) {
      umma::mbar_init(&acc_full[i], 1);
      umma::mbar_init(&acc_empty[i], PT_EPI);
    }
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;

  if (warp == PT_EPI / 32) {
    bool ok = true;
    u32 it = 0, st = 0, par = 1;
    for (u32 item = blockIdx.x; ok && item < items; item += gridDim.x) {
      const u32 ns = item % nsplit, pb = item / nsplit % npb, idx = item / (nsplit * npb), r = idx / nch, j = idx % nch;
      const int8_t* src = w.p + w.row[r] * w.stride + (w.off[r] + (u64)j * cw) * d + pb * PT_A;
      for (u32 c = 0; c < steps; c++, it++) {
        if (it >= PT_STAGES && !(ok = umma::mbar_wait(&empty_bar[st], par, err, 61))) break;
        if (umma::elect_one()) {
          uint8_t* stage = smem + st * PT_STAGE;
          umma::mbar_expect_tx(&full_bar[st], PT_A + 64 * nr);
          umma::bulk_g2s(stage, src + (u64)c * 64 * d, PT_A, &full_bar[st]);
          const int8_t* im = Jc + (u64)c * 64 * PT_ROWS + ns * nr * 16;
          if (nsplit == 1) umma::bulk_g2s(stage + PT_A, im, 64 * PT_ROWS, &full_bar[st]);
          else
            for (u32 x = 0; x < 4; x++)
              umma::bulk_g2s(stage + PT_A + x * nr * 16, im + x * PT_ROWS * 16, nr * 16, &full_bar[st]);
        }
        __syncwarp();
        if (++st == PT_STAGES) {
          st = 0;
          par ^= 1;
        }
      }
    }
    for (u32 c = it >= PT_STAGES ? it - PT_STAGES : 0; c < it; c++)
      umma::mbar_wait(&full_bar[c % PT_STAGES], (c / PT_STAGES) & 1, err, 62);
  } else if (warp == PT_EPI / 32 + 1) {
    // A: s8, MN-major (position slices 1024 apart, 8-element blocks 128); B: s8, K-major
    const u32 idesc = (2u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((nr >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t ad0 = umma::desc_kmajor(umma::smem_u32(smem), 128, 1024);
    const uint64_t bd0 = umma::desc_kmajor(umma::smem_u32(smem + PT_A), nr * 16, 128);
    bool ok = true;
    u32 it = 0, ui = 0, st = 0, par = 0;
    for (u32 item = blockIdx.x; ok && item < items; item += gridDim.x, ui++) {
      const u32 nb = ui & 1;
      if (ui >= 2 && !(ok = umma::mbar_wait(&acc_empty[nb], ((ui >> 1) - 1) & 1, err, 63))) break;
      umma::fence_after_sync();
      for (u32 c = 0; c < steps; c++, it++) {
        if (!(ok = umma::mbar_wait(&full_bar[st], par, err, 64))) break;
        umma::fence_after_sync();
        const uint64_t so = (uint64_t)st * (PT_STAGE >> 4);
        if (umma::elect_one()) {
#pragma unroll
          for (u32 ks = 0; ks < 2; ks++)
            umma::mma_i8_u(tmem + nb * 256, ad0 + so + ks * 32, bd0 + so + ks * 2 * nr, idesc,
                           (c > 0 || ks > 0) ? 1u : 0u);
          umma::commit(&empty_bar[st]);
          if (c + 1 == steps) umma::commit(&acc_full[nb]);
        }
        __syncwarp();
        if (++st == PT_STAGES) {
          st = 0;
          par ^= 1;
        }
      }
    }
    for (u32 c = it >= PT_STAGES ? it - PT_STAGES : 0; c < it; c++)
      umma::mbar_wait(&empty_bar[c % PT_STAGES], (c / PT_STAGES) & 1, err, 65);
  } else {
    const u32 m = (warp & 3) * 32 + lane, cols = nr / 2, c0 = (warp >> 2) * cols;
    u32 ui = 0;
    for (u32 item = blockIdx.x; item < items; item += gridDim.x, ui++) {
      const u32 ns = item % nsplit, pb = item / nsplit % npb, idx = item / (nsplit * npb), nb = ui & 1;
      const bool ok = umma::mbar_wait(&acc_full[nb], (ui >> 1) & 1, err, 66);
      if (!__all_sync(0xffffffffu, ok)) break;
      umma::fence_after_sync();
      const u32 tb = tmem + (((warp & 3) * 32) << 16) + nb * 256 + c0;
      u64* dst = out + ((u64)idx * PT_ROWS + ns * nr + c0) * d + pb * 128 + m;
      for (u32 g = 0; g < cols; g += 32) {
        uint32_t v[2][16];
        umma::tmem_ld16(tb + g, v[0]);
        umma::tmem_ld16(tb + g + 16, v[1]);
        umma::tmem_wait_ld();
        if (g + 32 == cols) {
          umma::fence_before_sync();
          umma::mbar_arrive(&acc_empty[nb]);
        }
#pragma unroll
        for (u32 e = 0; e < 32; e++) {
          const int x = (int)v[e / 16][e % 16];
          dst[(u64)(g + e) * d] = x >= 0 ? (u64)x : q - (u64)(-(long long)x);
        }
      }
    }
  }
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

}  // namespace

int launch_fold_challenge_tz(const DevState* ds, u32 round, u32 rows, u32 d, u64 q, u64* c_coef, int8_t* tz,
                             cudaStream_t st) {
  const u32 tot = rows * 32 * d;
  pdl(fold_chal_tz_kernel, (tot + 255) / 256, 256, 0, st)(ds, round, rows, d, q, c_coef, tz);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "fold_challenge_tz");
}

bool fold_tc_ok(const C8Rows& w, u32 d) {
  return (d == 128 || d == 256) && w.rows >= 1 && w.rows <= FT_MAX_ROWS && w.width >= FT_EL && w.width % FT_EL == 0;
}

int launch_fold_words_tz(const u64* c, u32 rows, u32 d, u64 q, int8_t* tz, u32* wide, cudaStream_t st) {
  pdl(fold_words_tz_kernel, (rows * 32 * d + 255) / 256, 256, 0, st)(c, rows, d, q, tz, wide);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "fold_words_tz launch");
}

int launch_fold_tc(const C8Rows& w, u32 d, u64 q, const int8_t* tz, u64 nout, u64* out, u64* mag_or, const u32* flag,
                   cudaStream_t st) {
  if (!fold_tc_ok(w, d) || !flag || nout > w.width)
    return salsaa_set_error(-2, "fold_tc: rows outside the byte-tile path");
  const size_t ring = d == 128 ? (size_t)FtGeom<128>::STAGES * FtGeom<128>::TILE
                               : (size_t)FtGeom<256>::STAGES * FtGeom<256>::TILE;
  const size_t smem = (size_t)w.rows * 32 * d + ring;
  const u64 units = w.width / FT_EL;
  const unsigned grid = (unsigned)(units < 148 ? units : 148);
  auto kern = d == 128 ? fold_tc_kernel<128> : fold_tc_kernel<256>;
  cudaError_t e = smem_limit(kern, (size_t)FT_MAX_ROWS * 32 * d + ring);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "fold_tc smem attribute");
  pdl(kern, grid, FT_THREADS, smem, st)(w, tz, q, nout, out, mag_or, flag, tc_error_word());
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "fold_tc launch");
}

int launch_words_to_c8(const RowSet& src, u32 rows, u64 width, u32 d, u64 q, int8_t* c8, u32* wide, cudaStream_t st) {
  if (src.narrow || rows == 0 || rows > (u32)MAX_WROWS || width == 0 || d % 16 || !rowset_aligned(src, rows, 16, 16))
    return salsaa_set_error(-2, "words_to_c8: bad rows");
  const u64 wpad = c8_width(width), tasks = wpad / 16 * (d / 16);
  const u64 want = (tasks + 7) / 8, most = 148 * 8;
  pdl(words_to_c8_kernel, dim3((unsigned)(want < most ? want : most), rows), 256, 0, st)(src, width, wpad, d, q, c8,
                                                                                         wide);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "words_to_c8 launch");
}

bool project_tc_ok(const C8Rows& w, u32 d, u32 cw) {
  // 2^31 bounds the sums: cw x 128
  return d % 128 == 0 && d <= 1024 && cw >= 64 && cw % 64 == 0 && cw <= (1u << 23) && w.rows > 0 &&
         w.rows <= (u32)MAX_WROWS && w.width >= cw && w.width % cw == 0 && w.width / cw * w.rows <= 65535;
}

int launch_project_tc(const C8Rows& w, u32 d, u64 q, u32 cw, const int8_t* Jc, u64* out, const u32* wide,
                      cudaStream_t st) {
  if (!project_tc_ok(w, d, cw)) return salsaa_set_error(-2, "project_tc: rows outside the byte-tile path");
  const u32 nch = (u32)(w.width / cw), base = w.rows * nch * (d / 128);
  // few chunks: part of the J rows per CTA
  u32 nsplit = 1;
  while (nsplit < 4 && base * nsplit * 2 <= 148) nsplit *= 2;
  const u32 items = base * nsplit;
  const size_t smem = (size_t)PT_STAGES * PT_STAGE;
  cudaError_t e = cudaFuncSetAttribute(project_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "project_tc smem attribute");
  pdl(project_tc_kernel, items < 148 ? items : 148, PT_THREADS, smem, st)(w, d, q, cw, nch, nsplit, Jc, out, wide,
                                                                         tc_error_word());
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "project_tc launch");
}

int launch_sc_tc(const Sc8Rows& w, u32 rows, u32 d, u32 Bw, u32 nhi, const ScRange& rg, const u64* s_hi,
                 const ModQ& M, u64* acc, const uint8_t* img, cudaStream_t st) {
  // q above 2^47 for the bounds, below 2^50 so that plain adds of at most one
  // residue per CTA and byte row cannot overflow
  if ((d != 128 && d != 256) || Bw % 64 || rg.n == 0 || rg.groups() > 2 || M.q >= (1ULL << 50) ||
      M.q < (1ULL << 47) || w.w.rows == 0 || w.w.rows > (u32)MAX_WROWS || (u64)Bw * nhi > w.w.width)
    return salsaa_set_error(-2, "sc_tc: rows outside the byte-tile path");
  // few items: split each element block over several CTAs
  const u64 base = (u64)w.w.rows * (d / 128) * nhi;
  u32 split = 1;
  while (split * 4 <= Bw / 64 && base * split < 148) split *= 2;
  const u64 items = base * split * rg.groups();
  const size_t smem = (size_t)ST_STAGES * ST_STAGE;
  cudaError_t e = cudaFuncSetAttribute(sc_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "sc_tc smem attribute");
  pdl(sc_tc_kernel, (unsigned)(items < 148 ? items : 148), ST_THREADS, smem, st)(w, rows, d, Bw, nhi, split, rg, s_hi, M,
                                                                                acc, img, tc_error_word());
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "sc_tc launch");
}

}  // namespace salsaa
