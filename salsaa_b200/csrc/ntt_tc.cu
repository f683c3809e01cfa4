// ntt_tc.cu — forward incomplete transforms of short values on the tensor
// cores, writing the byte image of the slot form (ntt_img.cuh).
#include <cuda_runtime.h>

#include "ntt_img.cuh"
#include "ntt_tile.cuh"
#include "umma.cuh"

namespace salsaa {

namespace {

// The protocol transforms short values: a ternary witness, digits below 2^7,
// projected rows below 2^15.  For those the transform is an exact integer
// product with the bytes of its matrix: D_y[s][i] = sum_k byte_y(W[s][k]) v_k
// (u8 x s8 -> s32, |D_y| < 2^22), and value = sum_y 2^(8 y) D_y mod q, so a
// coefficient costs 7 multiply-accumulate rows on the tensor cores and about
// 15 integer instructions instead of 39 FP64 ones, which bound the FP64
// transforms.  The byte matrix is 7 tiles of 128 x 128 (112 KiB), resident in
// shared memory of one persistent CTA per SM.  For n = 64 a row serves one
// half of an interleaved element and its other columns are zero, so elements
// go in as they lie; for n = 128 the halves are separate columns.
//
// An item is 4096 source words, a unit 32 columns of it: all 32 elements (n =
// 64) or 16 elements x 2 halves (n = 128), per digit; or (limb, element)
// pairs.  Warps 0 .. 15, in two groups that take alternate units, turn an
// accumulator (7 x 32 TMEM columns, one per group) into words, transpose 16
// elements of a (slot, half) into 7 byte rows of a shared tile and copy that
// to the image in full sectors; eight warps turn a source ring, which one
// thread keeps filled with bulk copies, into bytes of the operand ring; one
// warp issues 28 MMAs per unit.  (Loads into registers left the converters
// waiting: a thread's proxy fence waits for its earlier loads, so they could
// not run ahead.)
//
// Values that do not fit raise *flag; the FP64 kernel, launched after this
// one and gated on the flag, then rewrites everything.  A CTA whose first
// unit does not fit stops at once, so witnesses of full-size residues cost a
// few microseconds here.
//
// It takes 52 .. 57% of the issue slots and 4.6 .. 5.2 TB/s of DRAM (one limb
// and digits), the tensor pipe 12 .. 17% busy.  2^26 ternary words to their image 196 us (5.1 TB/s of 15 bytes per
// coefficient), against 294 us for the FP64 kernel (which its FP64 pipe and its
// four barriers per tile bound).
//
// Every wait is bounded; a role that gives up stops, and the others then
// give up on the arrivals it no longer makes.
constexpr u32 TC_EPI = 512, TC_CONV = 256, TC_THREADS = TC_EPI + TC_CONV + 64;
constexpr u32 TC_COLS = 32, TC_STAGES = 4;
constexpr u32 TC_PREFETCH = 4;  // items between a bulk prefetch to L2 and the copy to shared memory
constexpr u32 TC_RAW = 4, TC_RAW_BYTES = 4096 * 8 / TC_RAW;  // source ring: quarters of an item
constexpr u32 TC_SLICE = TC_COLS * 16;  // one 16-byte K slice
constexpr u32 TC_BTILE = 8 * TC_SLICE;
enum TcMode { TC_BYTES = 0, TC_DIGITS = 1, TC_LIMBS = 2 };

template <int LOGN, int MODE>
struct TcGeom {
  static constexpr u32 N = 1u << LOGN, D = 2 * N;
  static constexpr u32 SEL = 4096 / D, SELLOG = 11 - LOGN;  // source elements per item
  static constexpr u32 SUB = MODE == TC_BYTES ? 1 : 2;    // units per item
  static constexpr u32 WPT = SEL * D / TC_CONV;           // words per converter thread
  // image tile of a unit: TR rows per (slot, 16-element group), IU 16-byte
  // units per slot, odd, so neighbouring slots start on different bank groups
  static constexpr u32 JG = LOGN == 6 && MODE != TC_LIMBS ? 2 : 1;  // 16-element groups
  static constexpr u32 TR = LOGN == 7 && MODE == TC_LIMBS ? 7 : 14;
  static constexpr u32 IU = TR * JG | 1;
  static constexpr u32 TILES = MODE == TC_LIMBS ? 4 : 2;
  static constexpr u32 IMG = N * IU * 16;
  static constexpr u32 SMEM = (u32)TCW_BYTES + TC_STAGES * TC_BTILE + TC_RAW * TC_RAW_BYTES + TILES * IMG;
};

// Constants of tc_word's reductions.  C is a multiple of q that makes the sum
// positive, added as cl = C mod 2^32 and hb = C >> 32; nq = -q mod 2^64;
// k = floor(2^81 / q), below 2^32 for q > 2^49.
struct TcRed {
  u64 nq;
  long long hb;
  u32 cl, k;
};

// A residue of sum_y 2^(8 y) d_y mod q in [0, 1.02 q), below 2^51: the image's
// bytes need no canonical residue, so the last subtraction is left out.
//
// SHORT (n = 64, one limb): for y > 0 column k = 0 of the matrix is zero (its
// entry is 1), so |d_y| <= 63 x 255 x 128, and byte 6 is at most 3: pairs
// combine in 32 bits and |hi + (lo >> 32)| < 2^31 - 2^24.  With hb = 2^31 - (less than
// 2^18), x lies in [0, 2^32), and c = floor(x k / 2^49) is at most x 2^32 / q and less than 1 + 2^-17 below it.
// Else |hi + (lo >> 32)| < 2^41, hb about 2^41, x < 2^42, and
// c = floor(floor(x / 2^10) k / 2^39) is less than 1 + 2^-7 + 2^-7 below.
template <bool SHORT>
__device__ __forceinline__ u64 tc_word(int d0, int d1, int d2, int d3, int d4, int d5, int d6, const TcRed& red) {
  if (SHORT) {
    const int t01 = d1 * 256 + d0, t23 = d3 * 256 + d2, hi = d6 * 65536 + (d5 * 256 + d4);
    long long lo;
    asm("mad.wide.s32 %0, %1, 65536, %2;" : "=l"(lo) : "r"(t23), "l"((long long)red.cl));
    asm("mad.wide.s32 %0, %1, 1, %0;" : "+l"(lo) : "r"(t01));
    const u32 x = (u32)hi + (u32)(lo >> 32) + (u32)red.hb;
    const u32 c = __umulhi(x, red.k) >> 17;
    u64 r = (((u64)x << 32) | (u32)lo) + (u64)c * (u32)red.nq;
    r += (u64)(c * (u32)(red.nq >> 32)) << 32;
    return r;
  }
  long long lo = (long long)d1 * 256 + (long long)red.cl;
  lo += (long long)d2 * 65536;
  lo += (long long)d3 * 16777216;
  lo += d0;
  long long hi = (long long)d5 * 256 + d4;
  hi += (long long)d6 * 65536;
  const u64 x = (u64)(hi + (lo >> 32) + red.hb);
  const u32 c = __umulhi((u32)(x >> 10), red.k) >> 7;
  u64 r = ((x << 32) | (u32)lo) + (u64)c * (u32)red.nq;
  r += (u64)(c * (u32)(red.nq >> 32)) << 32;
  return r;
}

__device__ __forceinline__ void tc_transpose4(const u64 (&w)[4], u32 (&p)[7]) {
  const u32 t0 = __byte_perm((u32)w[0], (u32)w[1], 0x5140), t1 = __byte_perm((u32)w[0], (u32)w[1], 0x7362);
  const u32 t2 = __byte_perm((u32)w[2], (u32)w[3], 0x5140), t3 = __byte_perm((u32)w[2], (u32)w[3], 0x7362);
  p[0] = __byte_perm(t0, t2, 0x5410);
  p[1] = __byte_perm(t0, t2, 0x7632);
  p[2] = __byte_perm(t1, t3, 0x5410);
  p[3] = __byte_perm(t1, t3, 0x7632);
  const u32 h0 = (u32)(w[0] >> 32), h1 = (u32)(w[1] >> 32), h2 = (u32)(w[2] >> 32), h3 = (u32)(w[3] >> 32);
  const u32 s0 = __byte_perm(h0, h1, 0x5140), s1 = __byte_perm(h0, h1, 0x7362);
  const u32 s2 = __byte_perm(h2, h3, 0x5140), s3 = __byte_perm(h2, h3, 0x7362);
  p[4] = __byte_perm(s0, s2, 0x5410);
  p[5] = __byte_perm(s0, s2, 0x7632);
  p[6] = __byte_perm(s1, s3, 0x5410);
}

__device__ __forceinline__ void tmem_ld4(u32 taddr, int (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

// The and of p over `bar`'s THREADS threads, and a barrier among them.
template <u32 THREADS>
__device__ __forceinline__ bool bar_tc_and(bool p, u32 bar) {
  uint32_t r;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}\n"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(bar), "n"(THREADS)
      : "memory");
  return r != 0;
}

template <int LOGN, int MODE>
__global__ void __launch_bounds__(TC_THREADS, 1) ntt_tc_kernel(TcArgs a, CkImage im, const uint8_t* __restrict__ tcw,
                                                               u64 q, TcRed red, u32* err) {
  pdl_wait();
  using Geo = TcGeom<LOGN, MODE>;
  constexpr u32 N = Geo::N, D = Geo::D, SEL = Geo::SEL, SELLOG = Geo::SELLOG, SUB = Geo::SUB, WPT = Geo::WPT;
  constexpr u32 JG = Geo::JG, US = Geo::IU;
  constexpr u32 EPI = MODE == TC_LIMBS ? 128 : 256;  // threads per unit
  // a barrier pair per set of threads that shares units, so each set sees
  // every phase of its own (a parity wait cannot skip one)
  constexpr u32 NBAR = TC_EPI / EPI;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], acc_full[NBAR], acc_empty[NBAR], w_bar;
  __shared__ uint64_t raw_full[TC_RAW], raw_empty[TC_RAW];
  __shared__ uint32_t tslot;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const ImgRows& R = a.rows;
  uint8_t* const btile = smem + TCW_BYTES;
  uint8_t* const raw = btile + TC_STAGES * TC_BTILE;
  uint8_t* const itile = raw + TC_RAW * TC_RAW_BYTES;
  const u32 items = (u32)(R.rows * (R.width / SEL));
  u32 rlog = 0, dmask = 0;
  if (MODE == TC_DIGITS) {
    const u64 orv = *a.bw_or;
    const u32 bw = orv ? 64u - (u32)__clzll((long long)orv) : 0u;
    rlog = (bw + 1) / 2;
    if (blockIdx.x == 0 && tid == 0) {
      *a.rlog_out = rlog;
      if (a.radix_out) *a.radix_out = 1ULL << rlog;
      *a.flag = rlog > 7;
    }
    if (rlog > 7) return;  // the FP64 kernel takes the launch
    dmask = (1u << rlog) - 1;
  }

  // ---- loads and conversion of one item by 128 threads ----
  const u32 ct = tid - TC_EPI;
  const u32 qlo = (u32)q, qhi = (u32)(q >> 32);
  // quad i of thread t: 4 consecutive coefficients; a warp takes 32
  // coefficients of 4 neighbouring elements, so its 4-byte operand stores hit
  // a bank twice at most
  auto quad = [&](u32 i, u32 t, u32& el, u32& p) {
    const u32 j = i * (TC_CONV / 32) + (t >> 5), l = t & 31;
    el = j / (D / 32) * 4 + (l >> 3);
    p = j % (D / 32) * 32 + (l & 7) * 4;
  };
  auto source = [&](u32 item) -> const u64* {
    u32 k;
    u64 e0;
    img_item(R, im, SELLOG, item, k, e0);
    return R.src[k] + e0 * D;
  };
  // Centred value, plus 2^15 + 2^7 with two limbs (its bytes are then the signed
  // limbs + 128).  A short residue has a zero high word or, as q minus at most
  // 2^16 <= q mod 2^32, that of q, and the difference of the low words to 0 or
  // q is negative in the second case only: a low word near 2^32 above a zero
  // high word, or a small one above q's, is a value far from zero.  fit and
  // fith collect what contradicts.
  constexpr u32 BIAS = MODE == TC_LIMBS ? 0x8080u : 0u;
  auto centred = [&](u64 v, u32& fit, u32& fith) -> u32 {
    const u32 hi = (u32)(v >> 32);
    if (hi) fith |= hi ^ qhi;
    if (MODE == TC_LIMBS) {
      const u32 s = (u32)v - (hi ? qlo : 0u);
      fit |= s + BIAS;
      fith |= (hi ? ~s : s) & 0x80000000u;
      return s + BIAS;
    }
    const u32 w = (u32)v - (hi ? qlo - 128u : 0u);  // 0 .. 127 from 0 or from -128
    fit |= w;
    return hi ? w ^ 128u : w;  // its low byte
  };
  auto unfit = [&](u32 fit, u32 fith) { return (fit >> (MODE == TC_LIMBS ? 16 : 7)) != 0 || fith != 0; };

  // a CTA whose first item does not fit leaves before it starts
  if (MODE != TC_DIGITS) {
    u32 fit = 0, fith = 0;
    const ulonglong2* src = (const ulonglong2*)source(blockIdx.x);
    for (u32 i = tid; i < 2048; i += TC_THREADS) {
      const ulonglong2 v = __ldg(src + i);
      centred(v.x, fit, fith);
      centred(v.y, fit, fith);
    }
    if (__syncthreads_or(unfit(fit, fith))) {
      if (tid == 0) *a.flag = 1;
      return;
    }
  }

  if (tid == 0) {
    for (u32 i = 0; i < TC_STAGES; i++) {
      umma::mbar_init(&full_bar[i], TC_CONV);
      umma::mbar_init(&empty_bar[i], 1);
    }
    for (u32 i = 0; i < NBAR; i++) {
      umma::mbar_init(&acc_full[i], 1);
      umma::mbar_init(&acc_empty[i], EPI);
    }
    for (u32 i = 0; i < TC_RAW; i++) {
      umma::mbar_init(&raw_full[i], 1);
      umma::mbar_init(&raw_empty[i], TC_CONV);
    }
    umma::mbar_init(&w_bar, 1);
    umma::mbar_fence_init();
    umma::mbar_expect_tx(&w_bar, (u32)TCW_BYTES);
    for (u32 y = 0; y < 7; y++) umma::bulk_g2s(smem + y * 16384, tcw + y * 16384, 16384, &w_bar);
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;

  if (warp >= TC_EPI / 32 && warp < (TC_EPI + TC_CONV) / 32) {
    u32 fit = 0, fith = 0, mag = 0;
    bool ok = true;
    u32 it = 0;
    u32 ri = 0;  // items so far: the parity of their source ring uses
    for (u32 item = blockIdx.x; ok && item < items; item += gridDim.x) {
      u32 k;
      u64 e0;
      img_item(R, im, SELLOG, item, k, e0);
      // the operand stages of the item's units
      uint8_t* B[SUB];
#pragma unroll
      for (u32 sub = 0; sub < SUB; sub++) {
        const u32 st = (it + sub) % TC_STAGES, use = (it + sub) / TC_STAGES;
        if (use > 0 && !(ok = umma::mbar_wait(&empty_bar[st], (use - 1) & 1, err, 21))) break;
        B[sub] = btile + st * TC_BTILE;
      }
      if (!ok) break;
      // limb bytes of the quads: pk[.][0] the first limb or digit, [1] the second
      u32 pk[WPT / 4][MODE == TC_BYTES ? 1 : 2];
#pragma unroll
      for (u32 i = 0; i < WPT / 4; i++) {
        if (!(ok = umma::mbar_wait(&raw_full[i], ri & 1, err, 30))) break;
        u32 el, p;
        quad(i, ct, el, p);
        const ulonglong2* rw = (const ulonglong2*)(raw + (el * D + p) * 8);
        const ulonglong2 wa = rw[0], wb = rw[1];
        const u64 v[4] = {wa.x, wa.y, wb.x, wb.y};
        if (MODE == TC_DIGITS) {
          u32 d0[4], d1[4];
#pragma unroll
          for (u32 e = 0; e < 4; e++) {
            const bool neg = (u32)(v[e] >> 32) != 0;          // q minus less than 2^14
            const u32 m = neg ? qlo - (u32)v[e] : (u32)v[e];  // below 2^14
            const u32 x0 = m & dmask, x1 = (m >> rlog) & dmask;
            d0[e] = neg ? 0u - x0 : x0;
            d1[e] = neg ? 0u - x1 : x1;
          }
          pk[i][0] = __byte_perm(__byte_perm(d0[0], d0[1], 0x0040), __byte_perm(d0[2], d0[3], 0x0040), 0x5410);
          pk[i][MODE == TC_BYTES ? 0 : 1] =
              __byte_perm(__byte_perm(d1[0], d1[1], 0x0040), __byte_perm(d1[2], d1[3], 0x0040), 0x5410);
        } else {
          u32 x[4];
#pragma unroll
          for (u32 e = 0; e < 4; e++) {
            x[e] = centred(v[e], fit, fith);
            if (MODE == TC_LIMBS) {
              const int c = (int)(x[e] - BIAS);
              mag |= (u32)(c < 0 ? -c : c);
            }
          }
          const u32 x01 = __byte_perm(x[0], x[1], 0x5140), x23 = __byte_perm(x[2], x[3], 0x5140);
          pk[i][0] = __byte_perm(x01, x23, 0x5410) ^ (MODE == TC_LIMBS ? 0x80808080u : 0u);
          if (MODE == TC_LIMBS) pk[i][MODE == TC_BYTES ? 0 : 1] = __byte_perm(x01, x23, 0x7632) ^ 0x80808080u;
        }
#pragma unroll
        for (u32 sub = 0; sub < SUB; sub++) {
          if (LOGN == 6) {
            // K = position; columns: the elements (unit = digit sub), or
            // (limb, element) of the element group sub
            const u32 o = (p / 16) * TC_SLICE + p % 16;
            if (MODE == TC_LIMBS) {
              if (i / (WPT / 8) == sub) {
                *(u32*)(B[sub] + o + (el % 16) * 16) = pk[i][0];
                *(u32*)(B[sub] + o + (16 + el % 16) * 16) = pk[i][MODE == TC_BYTES ? 0 : 1];
              }
            } else {
              *(u32*)(B[sub] + o + el * 16) = pk[i][MODE == TC_BYTES ? 0 : sub];
            }
          } else {
            // K = index within a half; bytes 0, 2 belong to half 0, 1, 3 to half 1
            const u32 kk = p / 2, o = (kk / 16) * TC_SLICE + kk % 16;
            if (MODE == TC_LIMBS) {  // unit = half sub, columns (limb, element)
#pragma unroll
              for (u32 l = 0; l < 2; l++) {
                const u32 x = pk[i][MODE == TC_BYTES ? 0 : l];
                *(uint16_t*)(B[sub] + o + (l * 16 + el) * 16) = (uint16_t)__byte_perm(x, 0, sub ? 0x4431 : 0x4420);
              }
            } else {  // unit = digit sub, columns (half, element)
              const u32 x = pk[i][MODE == TC_BYTES ? 0 : sub];
              *(uint16_t*)(B[sub] + o + el * 16) = (uint16_t)__byte_perm(x, 0, 0x4420);
              *(uint16_t*)(B[sub] + o + (16 + el) * 16) = (uint16_t)__byte_perm(x, 0, 0x4431);
            }
          }
        }
        // The arrival hands this quarter to the next bulk copy, so the loads
        // from it must have returned: the stores above need their values.  (An
        // arrival directly after the loads let the copy overtake them.)
        umma::mbar_arrive(&raw_empty[i]);
      }
      if (!ok) break;
      ri++;
      umma::fence_proxy_async();
#pragma unroll
      for (u32 sub = 0; sub < SUB; sub++, it++) umma::mbar_arrive(&full_bar[it % TC_STAGES]);
      // the short values themselves, four per lane (after the fence, which
      // would wait for these stores)
      if (a.c8) {
#pragma unroll
        for (u32 i = 0; i < WPT / 4; i++) {
          u32 el, p;
          quad(i, ct, el, p);
          const u64 o = c8_offset(e0 + el, p, D);
#pragma unroll
          for (u32 c = 0; c < (MODE == TC_BYTES ? 1u : 2u); c++)
            *(u32*)(a.c8 + (u64)(MODE == TC_BYTES ? k : 2 * k + c) * R.width * D + o) = pk[i][c];
        }
      }
      if (MODE == TC_DIGITS && a.coef) {
#pragma unroll
        for (u32 i = 0; i < WPT / 4; i++) {
          u32 el, p;
          quad(i, ct, el, p);
#pragma unroll
          for (u32 c = 0; c < 2; c++) {
            const u32 x = pk[i][MODE == TC_BYTES ? 0 : c];
            *(int4*)(a.coef + ((u64)(2 * k + c) * R.width + e0 + el) * D + p) =
                make_int4((int)(int8_t)x, (int)(int8_t)(x >> 8), (int)(int8_t)(x >> 16), (int)(int8_t)(x >> 24));
          }
        }
      }
    }
    if (MODE != TC_DIGITS && R.mag_or) {
      // magnitudes of a thread whose values all fit (else the FP64 kernel
      // collects them)
      if (unfit(fit, fith)) mag = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mag |= __shfl_xor_sync(0xffffffffu, mag, o);
      if (lane == 0 && mag) atomicOr((unsigned long long*)R.mag_or, (unsigned long long)mag);
    }
    if (MODE != TC_DIGITS && unfit(fit, fith)) *a.flag = 1;
  } else if (warp == (TC_EPI + TC_CONV) / 32 + 1) {
    bool ok = true;
    u32 ri = 0;
    for (u32 item = blockIdx.x; ok && item < items; item += gridDim.x, ri++) {
      const uint8_t* src = (const uint8_t*)source(item);
      const u32 pre = item + TC_PREFETCH * gridDim.x;
      if (pre < items && umma::elect_one())
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(source(pre)), "r"(4096 * 8) : "memory");
      __syncwarp();
      for (u32 i = 0; i < TC_RAW; i++) {
        if (ri > 0 && !(ok = umma::mbar_wait(&raw_empty[i], (ri - 1) & 1, err, 31))) break;
        if (umma::elect_one()) {
          umma::mbar_expect_tx(&raw_full[i], TC_RAW_BYTES);
          umma::bulk_g2s(raw + i * TC_RAW_BYTES, src + i * TC_RAW_BYTES, TC_RAW_BYTES, &raw_full[i]);
        }
        __syncwarp();
      }
    }
    // the last copies land before the CTA ends
    for (u32 i = 0; i < TC_RAW && ri > 0; i++) umma::mbar_wait(&raw_full[i], (ri - 1) & 1, err, 32);
  } else if (warp == (TC_EPI + TC_CONV) / 32) {
    // u8 (matrix) x s8 (values), M = 128, N = 32
    const u32 idesc = umma::idesc_u8(128, TC_COLS) | (1u << 10);
    const uint64_t ad0 = umma::desc_kmajor(umma::smem_u32(smem), 2048, 128);
    const uint64_t bd0 = umma::desc_kmajor(umma::smem_u32(btile), TC_SLICE, 128);
    bool ok = umma::mbar_wait(&w_bar, 0, err, 22);
    u32 it = 0, st = 0, par = 0;
    for (u32 item = blockIdx.x; ok && item < items; item += gridDim.x) {
#pragma unroll
      for (u32 sub = 0; sub < SUB; sub++, it++) {
        const u32 nb = it & 1;
        // TMEM buffer nb was last used by unit it - 2
        if (it >= 2 && !(ok = umma::mbar_wait(&acc_empty[(it - 2) % NBAR], ((it - 2) / NBAR) & 1, err, 23))) break;
        if (!(ok = umma::mbar_wait(&full_bar[st], par, err, 24))) break;
        umma::fence_after_sync();
        const uint64_t bd = bd0 + st * (TC_BTILE >> 4);
        if (umma::elect_one()) {
#pragma unroll
          for (u32 y = 0; y < 7; y++)
#pragma unroll
            for (u32 ks = 0; ks < 4; ks++)
              umma::mma_i8_u(tmem + nb * (7 * TC_COLS) + y * TC_COLS, ad0 + y * 1024 + ks * 256,
                             bd + ks * (2 * TC_SLICE >> 4), idesc, ks > 0 ? 1u : 0u);
          umma::commit(&empty_bar[st]);
          umma::commit(&acc_full[it % NBAR]);
        }
        __syncwarp();
        if (++st == TC_STAGES) {
          st = 0;
          par ^= 1;
        }
      }
    }
    // MMAs still in flight complete before TMEM is freed
    for (u32 c = it >= 2 ? it - 2 : 0; c < it; c++) umma::mbar_wait(&acc_full[c % NBAR], (c / NBAR) & 1, err, 25);
  } else {
    // group eg takes the units it = eg mod 2; TMEM lane m; ch: half of the
    // columns, or (two limbs) of the group's units
    const u32 eg = warp >> 3, m = (warp & 3) * 32 + lane, ch = (warp >> 2) & 1;
    const u32 bar = MODE == TC_LIMBS ? 1 + 2 * eg + ch : 1 + eg;
    uint4* const tile = (uint4*)(itile + (MODE == TC_LIMBS ? 2 * eg + ch : eg) * Geo::IMG);
    const u32 out_rows = MODE == TC_DIGITS ? 2 * R.rows : R.rows;
    const u64 w2 = R.split ? R.width / 2 : R.width;
    const u32 s = LOGN == 6 ? m & 63 : m;
    uint4* const out = (uint4*)im.p;
    // neighbouring threads copy neighbouring units of a (slot, 16-element
    // group)'s 224 bytes (slots 4 VP units apart, groups VP); two limbs with
    // n = 128: the 7 rows of one half
    constexpr u32 RW = Geo::TR * JG, NCP = N * RW / EPI;
    static_assert(N * RW % EPI == 0 && NCP % 7 == 0, "whole batches of 7 copies per thread");
    const u32 et = MODE == TC_LIMBS ? m : tid & 255;  // thread of those that share the unit
    u32 it = 0;
    bool ok = true;
    for (u32 item = blockIdx.x; ok && item < items; item += gridDim.x) {
#pragma unroll 1
      for (u32 sub = 0; sub < SUB; sub++, it++) {
        const u32 nb = it & 1;
        if (nb != eg || (MODE == TC_LIMBS && ((it >> 1) & 1) != ch)) continue;
        // all threads of the unit stop together, also when only some of them
        // gave up; the barrier also orders the copies out of this tile before
        // its new rows
        ok = umma::mbar_wait(&acc_full[it % NBAR], (it / NBAR) & 1, err, 26);
        if (!(ok = bar_tc_and<EPI>(ok, bar))) break;
        umma::fence_after_sync();
        const u32 tb = tmem + (((warp & 3) * 32) << 16) + nb * (7 * TC_COLS) + (MODE == TC_LIMBS ? 0 : ch * 16);
        u32 pl[7][4];
#pragma unroll
        for (u32 q4 = 0; q4 < 4; q4++) {
          int dd[7][4];
#pragma unroll
          for (u32 y = 0; y < 7; y++) tmem_ld4(tb + y * TC_COLS + q4 * 4, dd[y]);
          if (MODE == TC_LIMBS) {
            int d1[7][4];
#pragma unroll
            for (u32 y = 0; y < 7; y++) tmem_ld4(tb + y * TC_COLS + 16 + q4 * 4, d1[y]);
            umma::tmem_wait_ld();
#pragma unroll
            for (u32 y = 0; y < 7; y++)
#pragma unroll
              for (u32 j = 0; j < 4; j++) dd[y][j] += d1[y][j] * 256;
          } else {
            umma::tmem_wait_ld();
          }
          if (q4 == 3) {
            umma::fence_before_sync();
            umma::mbar_arrive(&acc_empty[it % NBAR]);
          }
          u64 wv[4];
#pragma unroll
          for (u32 e = 0; e < 4; e++)
            wv[e] = tc_word<LOGN == 6 && MODE != TC_LIMBS>(dd[0][e], dd[1][e], dd[2][e], dd[3][e], dd[4][e], dd[5][e],
                                                           dd[6][e], red);
          u32 p[7];
          tc_transpose4(wv, p);
#pragma unroll
          for (u32 y = 0; y < 7; y++) pl[y][q4] = p[y];
        }
        // the 7 rows of (slot s, half h) and this thread's 16-element group
        const u32 h = LOGN == 6 ? m >> 6 : (MODE == TC_LIMBS ? 0 : ch), jg = JG == 2 ? ch : 0;
#pragma unroll
        for (u32 y = 0; y < 7; y++)
          tile[s * US + jg * 14 + h * 7 + y] = make_uint4(pl[y][0], pl[y][1], pl[y][2], pl[y][3]);
        u32 k;
        u64 e0;
        img_item(R, im, SELLOG, item, k, e0);
        const u64 i0 = e0 + (LOGN == 6 && MODE == TC_LIMBS ? 16 * sub : 0);
        const bool second = i0 >= w2;
        const u32 row = MODE == TC_DIGITS ? 2 * k + sub : k;
        uint4* const dst = out + cki_unit(im, R.k0 + row + (second ? out_rows : 0), second ? i0 - w2 : i0) +
                           (LOGN == 7 && MODE == TC_LIMBS ? 7 * sub : 0);
        bar_tc_and<EPI>(true, bar);
        u32 ss = et / RW, rem = et % RW;
#pragma unroll
        for (u32 b = 0; b < NCP; b += 7) {
          uint4 v[7];
          u32 o[7];
#pragma unroll
          for (u32 i = 0; i < 7; i++) {
            v[i] = tile[ss * US + rem];
            const u32 g = JG == 2 && rem >= 14 ? 1 : 0;
            o[i] = (ss * 4 + g) * im.VP + rem - 14 * g;
            ss += EPI / RW;
            rem += EPI % RW;
            if (rem >= RW) {
              rem -= RW;
              ss++;
            }
          }
#pragma unroll
          for (u32 i = 0; i < 7; i++) dst[o[i]] = v[i];
        }
      }
    }
  }
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
  // a CTA without items still has the matrix copy in flight
  if (tid == 0) umma::mbar_wait(&w_bar, 0, err, 27);
}

TcRed tc_red(u64 q, bool sh) {
  TcRed r{};
  const unsigned __int128 one = 1;
  const unsigned __int128 C = sh ? (one << 63) / q * q : ((one << 73) / q + 1) * q;
  r.nq = 0 - q;
  r.hb = (long long)(C >> 32);
  r.cl = (u32)C;
  r.k = (u32)((((unsigned __int128)1) << 81) / q);
  return r;
}

template <int LOGN, int MODE>
int tc_go(const TcArgs& a, const CkImage& im, const NttDev& T, cudaStream_t st) {
  using Geo = TcGeom<LOGN, MODE>;
  auto kern = ntt_tc_kernel<LOGN, MODE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Geo::SMEM);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "ntt_tc smem attribute");
  const u64 items = a.rows.rows * (a.rows.width / Geo::SEL);
  if (items > 0x3fffffffULL || cki_bytes(im) / 16 > 0xffffffffULL)
    return salsaa_set_error(-2, "ntt_tc: batch too large");
  const double coeffs = (double)a.rows.rows * a.rows.width * Geo::D;
  const int tr = salsaa_trace_begin(MODE == TC_DIGITS ? "ntt_digits_kernel" : "ntt_kernel", st,
                                    coeffs * (8 + (MODE == TC_DIGITS ? 2 : 1) * (a.c8 ? 8 : 7)));
  pdl(kern, (unsigned)(items < 148 ? items : 148), TC_THREADS, Geo::SMEM, st)(a, im, T.tcw, T.q,
                                                                             tc_red(T.q, LOGN == 6 && MODE != TC_LIMBS),
                                                                             tc_error_word());
  salsaa_trace_end(tr, st);
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ntt_tc launch");
}

}  // namespace

// q in (2^49, 2^50), and short negative residues keep q's high word
bool ntt_tc_ok(const NttDev& T) { return T.tcw != nullptr && T.q > (1ULL << 49) && (u32)T.q >= (1u << 16); }

int ntt_tc_launch(const TcArgs& a, int limbs, const CkImage& im, const NttDev& T, cudaStream_t st) {
  const ImgRows& R = a.rows;
  const bool digits = a.bw_or != nullptr;
  const u64 w2 = R.split ? R.width / 2 : R.width;
  const u32 out_rows = (digits ? 2 : 1) * R.rows;
  // magnitudes are collected for two limbs only
  if (!ntt_tc_ok(T) || !a.flag || (R.mag_or && (digits || limbs != 2)) || !im.p || im.n != T.n || im.width != w2 ||
      R.k0 + out_rows * (R.split ? 2 : 1) > im.R || R.rows == 0 || R.rows > MAX_WROWS || w2 < CKI_CHUNK ||
      (R.width & (R.width - 1)) || limbs < 1 || limbs > 2 || (digits && !a.rlog_out))
    return salsaa_set_error(-2, "ntt_tc: rows outside the image");
  for (u32 k = 0; k < R.rows; k++)
    if (!R.src[k] || (uintptr_t)R.src[k] % 16) return salsaa_set_error(-2, "ntt_tc: rows must be 16-byte aligned");
  const int mode = digits ? TC_DIGITS : limbs == 2 ? TC_LIMBS : TC_BYTES;
  if (T.logn == 6)
    return mode == TC_DIGITS ? tc_go<6, TC_DIGITS>(a, im, T, st)
                             : mode == TC_LIMBS ? tc_go<6, TC_LIMBS>(a, im, T, st) : tc_go<6, TC_BYTES>(a, im, T, st);
  return mode == TC_DIGITS ? tc_go<7, TC_DIGITS>(a, im, T, st)
                           : mode == TC_LIMBS ? tc_go<7, TC_LIMBS>(a, im, T, st) : tc_go<7, TC_BYTES>(a, im, T, st);
}

int ntt_short_img_launch(const ImgRows& a, u32* flag, const CkImage& im, const NttDev& T, cudaStream_t st) {
  if (!ntt_tc_ok(T)) return ntt_img_launch(a, im, T, st);
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(u32), st);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "ntt_tc flag");
  TcArgs t{};
  t.rows = a;
  t.flag = flag;
  int rc = ntt_tc_launch(t, 1, im, T, st);
  if (rc) return rc;
  ImgRows g = a;
  g.gate = flag;
  return ntt_img_launch(g, im, T, st);
}

}  // namespace salsaa
