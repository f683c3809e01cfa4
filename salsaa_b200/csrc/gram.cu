// gram.cu — four sumcheck rounds per pass through 16 x 16 Gram matrices (see gram.cuh).
#include <cuda_runtime.h>

#include "gram.cuh"
#include "umma.cuh"

namespace salsaa {

namespace {

constexpr u32 GR_T = 4, GR_WORK = 256, GR_THREADS = GR_WORK + 32;

__device__ __forceinline__ void work_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// lambda[m] of the four challenges ch.
__device__ __forceinline__ u64 gr_lambda(const ModQ& M, const u64* ch, u32 m) {
  u64 lam = 1 % M.q;
#pragma unroll
  for (u32 t = 0; t < GR_T; t++)
    lam = mul_mod(M, lam, ((m >> (GR_T - 1 - t)) & 1) ? ch[t] : salsaa::sub_mod(1 % M.q, ch[t], M.q));
  return lam;
}

// ---------------------------------------------------------------------------
// Words.  A tile of 256 groups is stored as it lies in memory, two words of a
// group (m, m + 1) in one 16-byte unit, unit (8-group block, m / 2, group % 8):
// the eight bytes of a word are its base-256 digits, and the one image is
//   * the K-major A operand (M = 128 groups, K = the 128 bytes (m, x)) of the
//     fold against the bytes of mu[m, x] = 2^(8x) lambda[m] mod q
//     (N = (rep, byte y)), and
//   * the MN-major A and B operands (M = N = (m, x), K = groups) of the Gram
//     product, accumulated in TMEM over the tiles of a segment.
// x'[g] = sum_y 2^(8y) D[g][rep, y]; C[m1][m2] = sum 2^(8 (x1 + x2))
// D[(m1, x1)][(m2, x2)] mod q.  Any 64-bit word is exact: no range check and
// no second pass.  Eight warps load (one group a thread), store the image and
// write the folded words, a ninth issues the MMAs; two CTAs a SM, so that one
// loads while the other multiplies.  Bound by HBM: 8.5 bytes a word (9 with
// two repetitions), against 112 clocks of MMAs per 8 KB.  It takes the place
// of 60 products and 15 folds a group on the CUDA cores: 64 vectors of 2^16 to
// 2^22 words 433 -> 141 us, the first pass over 2^24 words (then four signed
// limbs and a flag for larger values) 50 -> 39, the second pass 20 -> 16.
// ---------------------------------------------------------------------------
constexpr u32 GW_IMG = GRAM_TILE * 128, GW_SMEM = GW_IMG + 2048 + 1024;
constexpr u32 GW_SEG = 128;  // tiles a segment: 255^2 x 256 x 128 < 2^31

struct GwArgs {
  RowSet w;  // FIRST
  const u64* in;
  u64 sin;
  u64* out;
  u64 sout, L;
  u32 rows, round, j;
  const SbInst* inst;  // BATCH
  u32 ninst;
  u64 seed;
  const DevState* ds;
  u64* gram;
  const u32* gate;
  u64 w32p;  // Shoup companion of 2^32 mod q (a 128-bit division)
  u32 ntiles;
  bool plain;
};

enum GwMode { GW_FIRST, GW_ROUND, GW_BATCH };

template <int MODE>
__global__ void __launch_bounds__(GR_THREADS, 2) gram_words_kernel(const __grid_constant__ GwArgs a, ModQ M, u32* err) {
  pdl_wait();
  constexpr u32 REPS = MODE == GW_FIRST ? 2 : 1;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t full_bar, done_bar;
  __shared__ uint32_t tslot;
  __shared__ u64 ch[REPS][GR_T];
  __shared__ u32 t0s[MODE == GW_BATCH ? SB_MAX_INST + 1 : 1];
  if (a.gate && *(volatile const u32*)a.gate == 0) return;
  uint8_t* smem = smem_raw;
  uint8_t* btab = smem + GW_IMG;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const u64 q = M.q;
  const u32 t0 = (u32)((u64)blockIdx.x * a.ntiles / gridDim.x);
  const u32 t1 = (u32)((u64)(blockIdx.x + 1) * a.ntiles / gridDim.x);
  if (MODE == GW_BATCH)
    for (u32 i = tid; i <= a.ninst; i += GR_THREADS) t0s[i] = i < a.ninst ? (u32)a.inst[i].tile0 * SB_GPT : a.ntiles;
  if (tid == 0) {
    umma::mbar_init(&full_bar, GR_WORK);
    umma::mbar_init(&done_bar, 1);
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;  // columns 0..127 Gram, 128 + 16 h fold of half h
  const u32 tpi = MODE == GW_BATCH ? 1 : (u32)(a.L / 16 / GRAM_TILE);

  // instance of a tile: its index and first and last + 1 tile
  auto find = [&](u32 t, u32& id, u32& first, u32& end) {
    if (MODE == GW_BATCH) {
      u32 lo = 0, hi = a.ninst;  // t0s[lo] <= t < t0s[hi]
      while (hi - lo > 1) {
        const u32 mid = (lo + hi) / 2;
        if (t0s[mid] <= t) lo = mid;
        else hi = mid;
      }
      id = lo;
      first = t0s[lo];
      end = t0s[lo + 1];
    } else {
      id = t / tpi;
      first = id * tpi;
      end = first + tpi;
    }
  };
  auto seg_end = [&](u32 t, u32 end) {
    u32 e = t + GW_SEG;
    e = e < t1 ? e : t1;
    return e < end ? e : end;
  };

  if (warp == GR_WORK / 32) {
    // u8 x u8: Gram (both MN-major, M = N = 128), fold (both K-major, M = 128, N = 16)
    const u32 id_gram = (2u << 4) | (1u << 15) | (1u << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const u32 id_fold = (2u << 4) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
    // MN-major: LBO = stride of 8-group K blocks, SBO = stride of 16-byte MN slices
    const uint64_t dg0 = umma::desc_kmajor(umma::smem_u32(smem), 1024, 128);
    const uint64_t da0 = umma::desc_kmajor(umma::smem_u32(smem), 128, 1024);
    const uint64_t db0 = umma::desc_kmajor(umma::smem_u32(btab), 256, 128);
    u32 it = 0, issued = 0;
    bool ok = true;
    for (u32 t = t0; ok && t < t1;) {
      u32 id, first, end;
      find(t, id, first, end);
      const u32 se = seg_end(t, end);
      for (u32 i = t; i < se; i++, it++) {
        if (!(ok = umma::mbar_wait(&full_bar, it & 1, err, 71))) break;
        umma::fence_after_sync();
        if (umma::elect_one()) {
#pragma unroll
          for (u32 h = 0; h < 2; h++)
#pragma unroll
            for (u32 j = 0; j < 4; j++)
              umma::mma_i8_u(tmem + 128 + h * 16, da0 + h * 1024 + j * 16, db0 + j * 32, id_fold, j ? 1u : 0u);
#pragma unroll
          for (u32 kb = 0; kb < GRAM_TILE / 32; kb++)
            umma::mma_i8_u(tmem, dg0 + kb * 256, dg0 + kb * 256, id_gram, (i > t || kb > 0) ? 1u : 0u);
          umma::commit(&done_bar);
        }
        __syncwarp();
        issued = it + 1;
      }
      t = se;
    }
    if (!ok && issued) umma::mbar_wait(&done_bar, (issued - 1) & 1, err, 75);
  } else {
    u64 wv[16];
    u32 lid = 0, lfirst = 0, lend = 0;  // instance of the loaded tile
    const u64* lsrc = nullptr;
    u64 lng = 0;
    bool lnar = false;
    auto locate = [&](u32 t) {
      find(t, lid, lfirst, lend);
      if (MODE == GW_FIRST) {
        lsrc = a.w.p[lid];
        lnar = (a.w.narrow >> lid) & 1;
        lng = a.L / 16;
      } else if (MODE == GW_ROUND) {
        lsrc = a.in + (u64)lid * a.sin;
        lng = a.L / 16;
      } else {
        lsrc = a.inst[lid].in;
        lng = a.inst[lid].L / 16;
      }
    };
    auto load = [&](u32 t) {
      if (t >= lend) locate(t);
      const u64 g = (u64)(t - lfirst) * GRAM_TILE + tid;
      if (MODE == GW_FIRST && lnar) {
#pragma unroll
        for (u32 m = 0; m < 16; m++) {
          const int v = __ldg((const int*)lsrc + g + m * lng);
          wv[m] = v < 0 ? (u64)((long long)q + v) : (u64)v;
        }
      } else {
#pragma unroll
        for (u32 m = 0; m < 16; m++) wv[m] = __ldg(lsrc + g + m * lng);
      }
    };
    const u64 w32 = ((u64)1 << 32) % q;
    const u32 col0 = (warp >> 2) * 64;
    u64 pw = 1 % q;  // 2^(8 x1) mod q of this thread's Gram lane (m1, x1)
    for (u32 x = 0; x < (lane & 7); x++) pw = mul_mod(M, pw, 256);
    u32 it = 0;
    bool ok = true;
    if (t0 < t1) load(t0);
    for (u32 t = t0; t < t1;) {
      const u32 id = lid, first = lfirst, se = seg_end(t, lend);
      u64* out;
      u32 rep0, j0;
      u64* gram;
      if (MODE == GW_BATCH) {
        out = a.inst[id].out;
        rep0 = a.inst[id].id;
        j0 = a.inst[id].j;
        gram = a.gram + (u64)rep0 * 256;
      } else {
        out = a.out + (u64)id * a.sout;
        rep0 = MODE == GW_ROUND ? id / a.rows : 0;
        j0 = a.j;
        gram = a.gram + (u64)id * 256;
      }
      // fold B table (K-major, 16 rows (rep, y), K = 128 bytes (m, x)); the
      // segment before has been multiplied
      if (tid < REPS * GR_T) {
        const u64 key = prf_key(MODE == GW_BATCH ? a.seed : a.ds->seed, domain_id(DOM_NC, a.round, rep0 + tid / GR_T));
        ch[tid / GR_T][tid % GR_T] = uni_mod(prf_at(key, j0 + tid % GR_T), q);
      }
      work_sync();
      {
        const u32 rep = tid >> 7, m = (tid >> 3) & 15, x = tid & 7, kk = m * 8 + x;
        u64 mv = 0;
        if (rep < REPS) {
          mv = gr_lambda(M, ch[rep < REPS ? rep : 0], m);
          mv = mul_mod(M, mv, pw);  // x = lane & 7
        }
#pragma unroll
        for (u32 y = 0; y < 8; y++)
          btab[(kk / 16) * 256 + rep * 128 + y * 16 + kk % 16] = (uint8_t)(mv >> (8 * y));
      }
      for (u32 i = t; i < se; i++, it++) {
#pragma unroll
        for (u32 m2 = 0; m2 < 8; m2++)
          *(ulonglong2*)(smem + (tid >> 3) * 1024 + m2 * 128 + (tid & 7) * 16) =
              make_ulonglong2(wv[2 * m2], wv[2 * m2 + 1]);
        umma::fence_proxy_async();
        umma::fence_before_sync();
        umma::mbar_arrive(&full_bar);
        if (i + 1 < t1) load(i + 1);
        // after a wait that gave up, run on without waiting: the barriers between
        // segments are for every warp
        if (ok) ok = __all_sync(0xffffffffu, umma::mbar_wait(&done_bar, it & 1, err, 72));
        umma::fence_after_sync();
        uint32_t r[16];
        umma::tmem_ld16(tmem + (((warp & 3) * 32) << 16) + 128 + (warp >> 2) * 16, r);
        umma::tmem_wait_ld();
        const u64 g = (u64)(i - first) * GRAM_TILE + tid;  // TMEM lane of half warp >> 2
#pragma unroll
        for (u32 rep = 0; rep < REPS; rep++) {
          const uint32_t* D = r + rep * 8;  // below 128 x 255^2 < 2^23
          u64 lo = (u64)D[0] + ((u64)D[1] << 8) + ((u64)D[2] << 16) + ((u64)D[3] << 24);
          const u64 hi = (u64)D[4] + ((u64)D[5] << 8) + ((u64)D[6] << 16) + ((u64)D[7] << 24);
          if (lo >= q) lo -= q;  // lo < 2^48 < 2 q
          out[(MODE == GW_FIRST ? (u64)rep * a.rows * a.sout : 0) + g] =
              salsaa::add_mod(mul_shoup(hi, w32, a.w32p, q), lo, q);
        }
      }
      // Gram of the segment: lane (m1, x1), eight m2 a warp
#pragma unroll 1
      for (u32 cb = 0; cb < 4; cb++) {
        uint32_t r[16];
        umma::tmem_ld16(tmem + (((warp & 3) * 32) << 16) + col0 + cb * 16, r);
        umma::tmem_wait_ld();
#pragma unroll
        for (u32 e = 0; e < 2; e++) {
          const uint32_t* D = r + e * 8;  // below 2^31
          const u64 lo = (u64)D[0] + ((u64)D[1] << 8) + ((u64)D[2] << 16) + ((u64)D[3] << 24);
          const u64 hi = (u64)D[4] + ((u64)D[5] << 8) + ((u64)D[6] << 16) + ((u64)D[7] << 24);
          u64 v = mul_mod(M, salsaa::add_mod(mul_shoup(hi, w32, a.w32p, q), reduce64(M, lo), q), pw);
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) v = salsaa::add_mod(v, __shfl_xor_sync(0xffffffffu, v, o), q);
          const u32 m1 = ((warp & 3) * 32 + lane) >> 3, m2 = (warp >> 2) * 8 + cb * 2 + e;
          if ((lane & 7) == (m2 & 7)) atomic_add_mod(gram + m1 * 16 + m2, v, q, a.plain);
        }
      }
      umma::fence_before_sync();
      t = se;
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

template <int MODE>
int gw_launch(GwArgs& a, const ModQ& M, cudaStream_t st) {
  a.w32p = (u64)(((unsigned __int128)(((u64)1 << 32) % M.q) << 64) / M.q);
  const u32 grid = a.ntiles < 296 ? a.ntiles : 296;
  // adds to one Gram entry: one per segment
  a.plain = M.q < (1ULL << 50) && a.ntiles / GW_SEG + grid + SB_MAX_INST < (1u << 13);
  cudaError_t e = smem_limit(gram_words_kernel<MODE>, GW_SMEM);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "gram_words smem attribute");
  pdl(gram_words_kernel<MODE>, grid, GR_THREADS, GW_SMEM, st)(a, M, tc_error_word());
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "gram_words launch");
}

// ---------------------------------------------------------------------------
// Byte rows (byte tiles, see ntt_img.cuh): a value is one signed byte, so an
// element-block of 16 m x 64 elements x 16 positions is 16 KB.  It is stored
// as 16-byte units (16 positions of one m and element i = 8 b + s) at
// s GC_SL + b 256 + m 16, which is
//   * the K-major A and B operands (M = N = (b, m), K = (s, position)) of the
//     Gram product, whose eight diagonal 16 x 16 blocks add up to C, and
//   * the MN-major A operand (M = (s, position), K = (b parity, m)) of the
//     fold, two b at a time against lambda's bytes (N = (b parity, rep, y)).
// Both repetitions in one pass.  Bound by the words it writes (8 for 8 input
// bytes) and their reductions; where the words' kernel reads 4 or 8 bytes a
// value this one reads one: the first passes of an 8-round proof over 2^19
// elements, d = 128, 638 -> 301 us.
// ---------------------------------------------------------------------------
constexpr u32 GC_SL = 2048 + 16;  // slice stride: eight lanes' units in distinct banks
constexpr u32 GC_IMG = 8 * GC_SL, GC_SMEM = GC_IMG + 1024;
constexpr u32 GC_MAX = 1000;  // steps a CTA: 128^2 x 128 x 1000 < 2^31

__global__ void __launch_bounds__(GR_THREADS, 2)
    gram_c8_kernel(C8Rows w, u32 d, ModQ M, const DevState* ds, u32 round, u64* out, u64 sout, u64* gram,
                   const u32* wide, u64 w32p, bool plain, u32* err) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar, done_bar;
  __shared__ uint32_t tslot;
  __shared__ u64 ch[2][GR_T];
  __shared__ long long C[256];
  if (*(volatile const u32*)wide) return;
  uint8_t* btab = smem + GC_IMG;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, k = blockIdx.y;
  const u64 q = M.q;
  const u32 npb = d / 16, steps = (u32)(w.width / 1024) * npb;
  const u32 t0 = (u32)((u64)blockIdx.x * steps / gridDim.x), t1 = (u32)((u64)(blockIdx.x + 1) * steps / gridDim.x);
  if (tid < 2 * GR_T) {
    const u64 key = prf_key(ds->seed, domain_id(DOM_NC, round, tid / GR_T));
    ch[tid / GR_T][tid % GR_T] = uni_mod(prf_at(key, tid % GR_T), q);
  }
  if (tid == 0) {
    umma::mbar_init(&full_bar, GR_WORK);
    umma::mbar_init(&done_bar, 1);
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;  // columns 0..127 Gram, 128 + 32 bp fold of b pair bp

  if (warp == GR_WORK / 32) {
    // Gram: s8 x s8, K-major, M = N = 128; fold: s8 (MN-major) x u8, M = 128, N = 32
    const u32 id_gram = (2u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const u32 id_fold = (2u << 4) | (1u << 7) | (1u << 15) | ((32u >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t dg0 = umma::desc_kmajor(umma::smem_u32(smem), GC_SL, 128);
    const uint64_t da0 = umma::desc_kmajor(umma::smem_u32(smem), 128, GC_SL);
    const uint64_t db0 = umma::desc_kmajor(umma::smem_u32(btab), 512, 128);
    bool ok = true;
    for (u32 t = t0; ok && t < t1; t++) {
      if (!(ok = umma::mbar_wait(&full_bar, (t - t0) & 1, err, 73))) break;
      umma::fence_after_sync();
      if (umma::elect_one()) {
#pragma unroll
        for (u32 bp = 0; bp < 4; bp++) umma::mma_i8_u(tmem + 128 + bp * 32, da0 + bp * 32, db0, id_fold, 0u);
#pragma unroll
        for (u32 s = 0; s < 4; s++)
          umma::mma_i8_u(tmem, dg0 + s * (2 * GC_SL / 16), dg0 + s * (2 * GC_SL / 16), id_gram,
                         (t > t0 || s > 0) ? 1u : 0u);
        umma::commit(&done_bar);
      }
      __syncwarp();
    }
  } else {
    {  // lambda's bytes: rows (parity, rep, y), K = (parity, m), zero off the parity
      const u32 n8 = (tid >> 5) & 3, kk = tid & 31;  // rows 8 n8 .. + 7
      if (tid < 128) {
        const u32 par = n8 >> 1, rep = n8 & 1;
        const u64 lam = (kk >> 4) == par ? gr_lambda(M, ch[rep], kk & 15) : 0;
#pragma unroll
        for (u32 y = 0; y < 8; y++) btab[(kk / 16) * 512 + n8 * 128 + y * 16 + kk % 16] = (uint8_t)(lam >> (8 * y));
      }
      C[tid] = 0;
    }
    const u64 w32 = ((u64)1 << 32) % q;
    const u64 mrun = w.width / 16 * d;  // bytes between a group's m
    const int8_t* src = w.p + w.row[k] * w.stride + w.off[k] * d + (u64)(tid >> 6) * mrun + (tid & 63) * 16;
    uint4 v[4];
    auto load = [&](u32 t) {
      const int8_t* s = src + (u64)t * 1024;  // 64-element tiles and their position blocks are one run
#pragma unroll
      for (u32 j = 0; j < 4; j++) v[j] = __ldg((const uint4*)(s + (u64)(4 * j) * mrun));
    };
    const u32 i0 = tid & 63;
    uint8_t* dst = smem + (i0 & 7) * GC_SL + (i0 >> 3) * 256 + (tid >> 6) * 16;
    const u32 row = (warp & 3) * 32 + lane;
    bool ok = true;
    if (t0 < t1) load(t0);
    for (u32 t = t0; t < t1; t++) {
#pragma unroll
      for (u32 j = 0; j < 4; j++) *(uint4*)(dst + j * 64) = v[j];
      umma::fence_proxy_async();
      umma::fence_before_sync();
      umma::mbar_arrive(&full_bar);
      if (t + 1 < t1) load(t + 1);
      ok = umma::mbar_wait(&done_bar, (t - t0) & 1, err, 74);
      if (!(ok = __all_sync(0xffffffffu, ok))) break;
      umma::fence_after_sync();
      const u32 tile = t / npb, pb = t % npb;
      // element 64 tile + 8 b + s at this lane's slice s = row / 16 and position
      u64* o = out + (u64)k * sout + ((u64)tile * 64 + (row >> 4)) * d + pb * 16 + (row & 15);
#pragma unroll
      for (u32 h = 0; h < 2; h++) {
        const u32 bp = (warp >> 2) * 2 + h;
        uint32_t r[2][16];
        umma::tmem_ld16(tmem + (((warp & 3) * 32) << 16) + 128 + bp * 32, r[0]);
        umma::tmem_ld16(tmem + (((warp & 3) * 32) << 16) + 128 + bp * 32 + 16, r[1]);
        umma::tmem_wait_ld();
#pragma unroll
        for (u32 p = 0; p < 2; p++)
#pragma unroll
          for (u32 rep = 0; rep < 2; rep++) {
            const int* D = (const int*)r[p] + rep * 8;  // |D| <= 16 x 128 x 255 < 2^20
            const long long lo = (long long)D[0] + ((long long)D[1] << 8) + ((long long)D[2] << 16) +
                                 ((long long)D[3] << 24);
            const long long hi = (long long)D[4] + ((long long)D[5] << 8) + ((long long)D[6] << 16);
            const u64 loc = lo < 0 ? (u64)(lo + (long long)q) : (u64)lo;  // |lo| < 2^45 < q
            const u64 hic = hi < 0 ? (u64)(hi + (long long)q) : (u64)hi;
            o[(u64)rep * w.rows * sout + (u64)(8 * (2 * bp + p)) * d] =
                salsaa::add_mod(mul_shoup(hic, w32, w32p, q), loc, q);
          }
      }
      umma::fence_before_sync();
    }
    work_sync();  // C is zero
    if (ok && t0 < t1 && warp < 4) {
      // this lane's diagonal block b = row / 16: the warp's two blocks, one of them its own
      uint32_t r[2][16];
      umma::tmem_ld16(tmem + ((warp * 32) << 16) + warp * 32, r[0]);
      umma::tmem_ld16(tmem + ((warp * 32) << 16) + warp * 32 + 16, r[1]);
      umma::tmem_wait_ld();
#pragma unroll
      for (u32 e = 0; e < 16; e++) {
        const long long x = (int)(lane < 16 ? r[0][e] : r[1][e]);
        atomicAdd((unsigned long long*)&C[(lane & 15) * 16 + e], (unsigned long long)x);
      }
    }
    work_sync();
    if (ok && t0 < t1) {
      const long long x = C[tid];  // |x| < 2^34 < q
      atomic_add_mod(gram + (u64)k * 256 + tid, x < 0 ? (u64)(x + (long long)q) : (u64)x, q, plain);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

}  // namespace

int launch_gram_first(const RowSet& w, u32 rows, u64 n, const ModQ& M, const DevState* ds, u32 round, u64* out,
                      u64 sout, u64* gram, const u32* gate, cudaStream_t st) {
  if (!gram_words_ok(n, M.q) || rows == 0 || rows > (u32)MAX_WROWS || n / 16 / GRAM_TILE * rows >= (1ULL << 31))
    return salsaa_set_error(-2, "gram: bad shape");
  GwArgs a{};
  a.w = w;
  a.out = out;
  a.sout = sout;
  a.L = n;
  a.rows = rows;
  a.round = round;
  a.ds = ds;
  a.gram = gram;
  a.gate = gate;
  a.ntiles = (u32)(n / 16 / GRAM_TILE * rows);
  return gw_launch<GW_FIRST>(a, M, st);
}

int launch_gram_round(const u64* in, u64 sin, u64* out, u64 sout, u64 L, u32 rows, const ModQ& M, const DevState* ds,
                      u32 round, u32 j, u64* gram, cudaStream_t st) {
  if (!gram_words_ok(L, M.q) || L / 16 / GRAM_TILE * 2 * rows >= (1ULL << 31))
    return salsaa_set_error(-2, "gram: bad shape");
  GwArgs a{};
  a.in = in;
  a.sin = sin;
  a.out = out;
  a.sout = sout;
  a.L = L;
  a.rows = rows;
  a.round = round;
  a.j = j;
  a.ds = ds;
  a.gram = gram;
  a.ntiles = (u32)(L / 16 / GRAM_TILE * 2 * rows);
  return gw_launch<GW_ROUND>(a, M, st);
}

int launch_gram_batch(const SbInst* inst, u32 ninst, u64 ntiles, const ModQ& M, u64 seed, u32 round, u64* gram,
                      cudaStream_t st) {
  if (!inst || ninst == 0 || ninst > SB_MAX_INST || ntiles == 0 || ntiles * SB_GPT >= (1ULL << 31))
    return salsaa_set_error(-2, "gram: bad batch");
  GwArgs a{};
  a.inst = inst;
  a.ninst = ninst;
  a.seed = seed;
  a.round = round;
  a.gram = gram;
  a.ntiles = (u32)(ntiles * SB_GPT);
  return gw_launch<GW_BATCH>(a, M, st);
}

bool gram_c8_ok(const C8Rows& w, u32 d, u64 q) {
  return q > (1ULL << 47) && q < (1ULL << 56) && d % 16 == 0 && w.width % 1024 == 0 && w.width >= 1024 &&
         w.rows > 0 && w.rows <= (u32)MAX_WROWS && w.width / 1024 * (d / 16) < (1ULL << 31);
}

int launch_gram_c8(const C8Rows& w, u32 d, const ModQ& M, const DevState* ds, u32 round, u64* out, u64 sout,
                   u64* gram, const u32* wide, cudaStream_t st) {
  if (!gram_c8_ok(w, d, M.q)) return salsaa_set_error(-2, "gram_c8: bad shape");
  const u32 steps = (u32)(w.width / 1024) * (d / 16);
  u32 nb = (296 + w.rows - 1) / w.rows;
  const u32 need = (steps + GC_MAX - 1) / GC_MAX;
  if (nb < need) nb = need;
  if (nb > steps) nb = steps;
  const u64 w32p = (u64)(((unsigned __int128)(((u64)1 << 32) % M.q) << 64) / M.q);
  const bool plain = M.q < (1ULL << 50) && nb < (1u << 13);
  pdl(gram_c8_kernel, dim3(nb, w.rows), GR_THREADS, GC_SMEM, st)(w, d, M, ds, round, out, sout, gram, wide, w32p, plain,
                                                                tc_error_word());
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "gram_c8 launch");
}

}  // namespace salsaa
