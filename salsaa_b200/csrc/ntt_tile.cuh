// ntt_tile.cuh — thread mappings, butterflies and exchanges of the register
// NTT, shared by the transform kernels (ntt.cu) and the transforms that write
// byte images of the slot form (ntt_img.cu).
#pragma once
#include "ntt.cuh"

namespace salsaa {

// ---------------------------------------------------------------------------
// Register-resident NTT for 16 <= n <= 4096 (q < 2^62, which the tables
// guarantee).  Each thread holds 16 coefficients of one transform unit (a
// full polynomial, or one half of a ring element in incomplete mode) and runs
// up to 4 butterfly stages on them in registers between exchanges through
// shared memory, so a 1024-point transform takes 3 exchanges instead of 10.
// Butterflies are Harvey's lazy variants of the Cooley-Tukey (forward) and
// Gentleman-Sande (inverse) butterflies with Shoup multiplication: forward
// values stay in [0, 4q) and inverse values in [0, 2q), which needs 4q < 2^64;
// one correction at the end makes the outputs canonical, so they equal the
// fully reduced transform exactly.
//
// For q < 2^50 (the protocol's primes) the RELAX variants drop the per-
// butterfly corrections: forward values grow by at most 2q per stage, so stay
// below (2 log n + 1) q, and inverse sums at most double per stage, so stay
// below 2^(log n) q, with the difference offset by C = 2^(log n) q instead of
// 2q; both bounds are far below 2^63 for log n <= 12.  One Shoup reduction by
// 1 (x - floor(x floor(2^64/q) / 2^64) q, in [0, 2q)) and a subtraction make
// the outputs canonical.
//
// Stage numbering follows the generic kernel above: forward stage g pairs
// elements t = n >> (g+1) apart with twiddle fwd[2^g + j / 2t]; inverse stage
// g pairs elements t = 2^g apart with twiddle inv[(n >> (g+1)) + j / 2t].  A
// phase covering stages g0 .. g0+S-1 gives each thread "mini-blocks" of 2^S
// elements e = blk * (stride << S) + r + k * stride, k < 2^S, whose pairs in
// all S stages stay inside the mini-block (stride = n >> (g0+S) forward,
// 2^g0 inverse).
//
// The first phase reads global memory and the last writes it directly: the
// strided side (forward input, inverse output) is coalesced across lanes,
// including the even/odd interleave of incomplete mode (lanes alternate
// halves); the contiguous side (forward output, inverse input: 2^S
// consecutive coefficients per thread) uses 16-byte vector accesses, so it
// needs 16-byte aligned buffers.  Shared memory holds 4096 coefficients with
// one padding word every 16 to spread the strided phases over the banks.
// ---------------------------------------------------------------------------
namespace {

__host__ __device__ constexpr int ph_count(int L) { return (L + 3) / 4; }
__host__ __device__ constexpr int ph_size(int L, int p) { return L / ph_count(L) + (p < L % ph_count(L) ? 1 : 0); }
__host__ __device__ constexpr int ph_start(int L, int p) { return p == 0 ? 0 : ph_start(L, p - 1) + ph_size(L, p - 1); }

constexpr u32 NR_TILE = 4096;  // coefficients per CTA
constexpr u64 NR_RELAX_Q = 1ULL << 50;  // below this, butterflies skip their corrections
__device__ __forceinline__ u32 npad(u32 p) { return p + (p >> 4); }

// x * w mod q in [0, 2q) for any 64-bit x (Shoup, without the final correction)
__device__ __forceinline__ u64 shoup_lazy(u64 x, u64 w, u64 wp, u64 q) { return x * w - __umul64hi(x, wp) * q; }

struct NrCtx {
  const NttDev* T;
  u64 q, q2;
};

// Butterflies of phase P on one mini-block v[0 .. 2^S) with block index blk.
template <int LOGN, int P, bool INV, bool RELAX>
__device__ __forceinline__ void nr_block(u64* v, u32 blk, const NttDev& T, u64 q, u64 q2) {
  // inverse difference offset: 2q, or 2^LOGN q when sums are left unreduced
  const u64 cdiff = RELAX ? (q << LOGN) : q2;
  constexpr int S = ph_size(LOGN, P), G0 = ph_start(LOGN, P);
  constexpr u32 N = 1u << LOGN, K = 1u << S;
  // pairs p < 2^(S-1) of level l: k = (sb << (l'+1)) + kk, one twiddle per sb
#pragma unroll
  for (int l = 0; l < S; l++) {
    const u32 lt = INV ? l : S - 1 - l;  // log2 of the pair distance in k
    const u32 t = 1u << lt;
    u64 w = 0, wp = 0;
#pragma unroll
    for (u32 p = 0; p < K / 2; p++) {
      const u32 sb = p >> lt, kk = p & (t - 1), k = (sb << (lt + 1)) + kk;
      if (kk == 0) {
        const u32 idx = INV ? (N >> (G0 + l + 1)) + (blk << (S - l - 1)) + sb : (1u << (G0 + l)) + (blk << l) + sb;
        w = __ldg((INV ? T.inv : T.fwd) + idx);
        wp = __ldg((INV ? T.invp : T.fwdp) + idx);
      }
      if (!INV) {
        u64 a = v[k];
        if (!RELAX) a = a >= q2 ? a - q2 : a;
        const u64 b = shoup_lazy(v[k + t], w, wp, q);
        v[k] = a + b;
        v[k + t] = a - b + q2;
      } else {
        const u64 a = v[k], b = v[k + t];
        u64 s2 = a + b;
        if (!RELAX) s2 = s2 >= q2 ? s2 - q2 : s2;
        v[k] = s2;
        v[k + t] = shoup_lazy(a - b + cdiff, w, wp, q);
      }
    }
  }
}

template <int LOGN, int P, bool INV, bool RELAX>
__device__ __forceinline__ void nr_compute(u64 (&x)[16], u32 tu, const NttDev& T, u64 q, u64 q2) {
  constexpr int S = ph_size(LOGN, P), G0 = ph_start(LOGN, P);
  constexpr u32 N = 1u << LOGN, TPU = N / 16, MB = 16 >> S;
  constexpr u32 LSTR = INV ? G0 : LOGN - G0 - S;  // log2(stride)
#pragma unroll
  for (u32 j = 0; j < MB; j++) nr_block<LOGN, P, INV, RELAX>(x + j * (1u << S), (tu + j * TPU) >> LSTR, T, q, q2);
}

// element index (within its unit) of register (j, k) in phase P
template <int LOGN, int P, bool INV>
__device__ __forceinline__ u32 nr_elem(u32 tu, u32 j, u32 k) {
  constexpr int S = ph_size(LOGN, P), G0 = ph_start(LOGN, P);
  constexpr u32 N = 1u << LOGN, TPU = N / 16;
  constexpr u32 LSTR = INV ? G0 : LOGN - G0 - S;
  const u32 mb = tu + j * TPU, blk = mb >> LSTR, r = mb & ((1u << LSTR) - 1);
  return (blk << (LSTR + S)) + r + (k << LSTR);
}

// Shared-memory exchange: a thread reads and writes the same positions within
// a phase, so a phase can update the tile in place.
template <int LOGN, int P, bool INV, typename W>
__device__ __forceinline__ void nr_load_smem(W (&x)[16], const W* sm, u32 unit, u32 tu) {
  constexpr int S = ph_size(LOGN, P);
  constexpr u32 N = 1u << LOGN, MB = 16 >> S, K = 1u << S;
#pragma unroll
  for (u32 j = 0; j < MB; j++)
#pragma unroll
    for (u32 k = 0; k < K; k++) x[j * K + k] = sm[npad(unit * N + nr_elem<LOGN, P, INV>(tu, j, k))];
}
template <int LOGN, int P, bool INV, typename W>
__device__ __forceinline__ void nr_store_smem(const W (&x)[16], W* sm, u32 unit, u32 tu) {
  constexpr int S = ph_size(LOGN, P);
  constexpr u32 N = 1u << LOGN, MB = 16 >> S, K = 1u << S;
#pragma unroll
  for (u32 j = 0; j < MB; j++)
#pragma unroll
    for (u32 k = 0; k < K; k++) sm[npad(unit * N + nr_elem<LOGN, P, INV>(tu, j, k))] = x[j * K + k];
}

// Global side of the first phase (P = 0).
template <int LOGN, bool INC, bool INV>
__device__ __forceinline__ void nr_load_global(u64 (&x)[16], const u64* __restrict__ in, u64 ug, u32 tu) {
  constexpr int S = ph_size(LOGN, 0);
  constexpr u32 N = 1u << LOGN, MB = 16 >> S, K = 1u << S;
  if (!INV) {  // strided: e = r + k * stride (blk = 0), coalesced across lanes
#pragma unroll
    for (u32 j = 0; j < MB; j++)
#pragma unroll
      for (u32 k = 0; k < K; k++) {
        const u32 e = nr_elem<LOGN, 0, INV>(tu, j, k);
        const u64 g = INC ? (ug >> 1) * (2 * N) + 2 * e + (ug & 1) : ug * N + e;
        x[j * K + k] = __ldg(in + g);
      }
  } else {  // contiguous 2^S coefficients per mini-block
#pragma unroll
    for (u32 j = 0; j < MB; j++) {
      const ulonglong2* src = (const ulonglong2*)(in + ug * N + nr_elem<LOGN, 0, INV>(tu, j, 0));
#pragma unroll
      for (u32 k = 0; k < K / 2; k++) {
        const ulonglong2 v = __ldg(src + k);
        x[j * K + 2 * k] = v.x;
        x[j * K + 2 * k + 1] = v.y;
      }
    }
  }
}

__device__ __forceinline__ u64 nr_canon4(u64 a, u64 q, u64 q2) {  // [0, 4q) -> [0, q)
  a = a >= q2 ? a - q2 : a;
  return a >= q ? a - q : a;
}
// forward output -> [0, q): [0, 4q) normally, any value below 2^64 when relaxed
template <bool RELAX>
__device__ __forceinline__ u64 nr_canon(u64 a, u64 q, u64 q2, u64 onep) {
  if (!RELAX) return nr_canon4(a, q, q2);
  a = shoup_lazy(a, 1, onep, q);
  return a >= q ? a - q : a;
}

// Global side of the last phase: canonical forward output (contiguous), or
// the inverse output scaled by 1/n (strided).
__device__ __forceinline__ u64 nr_mag(u64 v, u64 q) { return 2 * v > q ? q - v : v; }

template <int LOGN, bool INC, bool INV, bool RELAX>
__device__ __forceinline__ void nr_store_global(const u64 (&x)[16], u64* __restrict__ out, u64 ug, u32 tu,
                                                const NttDev& T, u64 q, u64 q2, u64* mag = nullptr) {
  constexpr int P = ph_count(LOGN) - 1, S = ph_size(LOGN, P);
  constexpr u32 N = 1u << LOGN, MB = 16 >> S, K = 1u << S;
  if (!INV) {
#pragma unroll
    for (u32 j = 0; j < MB; j++) {
      ulonglong2* dst = (ulonglong2*)(out + ug * N + nr_elem<LOGN, P, INV>(tu, j, 0));
#pragma unroll
      for (u32 k = 0; k < K / 2; k++)
        dst[k] = make_ulonglong2(nr_canon<RELAX>(x[j * K + 2 * k], q, q2, T.onep),
                                 nr_canon<RELAX>(x[j * K + 2 * k + 1], q, q2, T.onep));
    }
  } else {
#pragma unroll
    for (u32 j = 0; j < MB; j++)
#pragma unroll
      for (u32 k = 0; k < K; k++) {
        const u32 e = nr_elem<LOGN, P, INV>(tu, j, k);
        u64 v = shoup_lazy(x[j * K + k], T.ninv, T.ninvp, q);
        v = v >= q ? v - q : v;
        const u64 g = INC ? (ug >> 1) * (2 * N) + 2 * e + (ug & 1) : ug * N + e;
        out[g] = v;
        if (mag) *mag |= nr_mag(v, q);
      }
  }
}

// Phases P .. PEND-1 entirely through shared memory.
template <int LOGN, int P, int PEND, bool INV, bool RELAX>
__device__ __forceinline__ void nr_mid(u64 (&x)[16], u64* sm, u32 unit, u32 tu, bool active, const NttDev& T,
                                       u64 q, u64 q2) {
  if constexpr (P < PEND) {
    if (active) {
      nr_load_smem<LOGN, P, INV>(x, sm, unit, tu);
      nr_compute<LOGN, P, INV, RELAX>(x, tu, T, q, q2);
      nr_store_smem<LOGN, P, INV>(x, sm, unit, tu);
    }
    __syncthreads();
    nr_mid<LOGN, P + 1, PEND, INV, RELAX>(x, sm, unit, tu, active, T, q, q2);
  }
}

// Thread -> (unit in tile, thread within unit); in incomplete mode lanes
// alternate the two halves of an element so the interleaved side coalesces.
template <int LOGN, bool INC>
__device__ __forceinline__ void nr_map(u32 tid, u32& unit, u32& tu) {
  constexpr u32 TPU = (1u << LOGN) / 16;
  if (INC) {
    unit = 2 * (tid / (2 * TPU)) + (tid & 1);
    tu = (tid % (2 * TPU)) >> 1;
  } else {
    unit = tid / TPU;
    tu = tid % TPU;
  }
}

// ---------------------------------------------------------------------------
// FP64 butterflies for q < 2^50 (the protocol's primes).  On B200 the FP64
// pipe multiplies and adds 53-bit integers exactly at a far higher rate than
// the 32-bit integer multipliers assemble 64-bit Shoup products, so these
// kernels keep the coefficients as integer-valued doubles and reduce with
// error-free transformations (Dekker's exact product via FMA, as used for
// modular arithmetic in floating point by van der Hoeven, Lecerf and Quintin,
// "Modular SIMD arithmetic in Mathemagix", ACM TOMS 2016):
//
//   x * w mod q, |x| < 2^52, 0 <= w < q:  h = fl(x w), l = x w - h (one FMA,
//   exact), c = nearest integer to x fl(w / 2q) (one FMA against the
//   rounding constant 1.5 * 2^52 and one subtraction), r = (h - 2q c) + l.
//   Since |x w / 2q - c| <= 0.625 the integer x w - 2q c has magnitude at most
//   1.25 q < 2^51, so the FMA h - 2q c and the addition of l are exact: r is
//   x w mod q as an integer in [-1.25 q, 1.25 q].
//
//   v mod q, |v| < 2^52: c = nearest integer to v fl(1/q), r = v - c q
//   (exact, in [-q/2 - 1, q/2 + 1]).
//
// Forward (Cooley-Tukey): inputs in [0, q); each stage adds at most 1.25 q
// to a magnitude; all values are reduced after every odd-numbered stage, so
// magnitudes stay below 4 q < 2^52 and multiplicands below 2.5 q.  Inverse
// (Gentleman-Sande): the sum a + b is reduced in every stage (magnitudes of
// sums below 3 q, of differences below 3 q, of products below 1.25 q).  The
// outputs are reduced once more and shifted into [0, q), so they are the
// canonical residues, the same words as the integer kernels produce.
// Conversions between canonical words and doubles go through the exponent
// bits of 2^52 (v + 2^52 has v in its low 52 mantissa bits), one integer
// and one FP64 instruction each.
// ---------------------------------------------------------------------------
// Butterflies of phase P on one mini-block v[0 .. 2^S) with block index blk.
template <int LOGN, int P, bool INV>
__device__ __forceinline__ void nf_block(double* v, u32 blk, const NttDev& T) {
  constexpr int S = ph_size(LOGN, P), G0 = ph_start(LOGN, P);
  constexpr u32 N = 1u << LOGN, K = 1u << S;
  const double q2d = T.q2d, qd = T.qd, qinv = T.qinv;
#pragma unroll
  for (int l = 0; l < S; l++) {
    const u32 lt = INV ? l : S - 1 - l;
    const u32 t = 1u << lt;
    double w = 0, wh = 0;
#pragma unroll
    for (u32 p = 0; p < K / 2; p++) {
      const u32 sb = p >> lt, kk = p & (t - 1), k = (sb << (lt + 1)) + kk;
      if (kk == 0) {
        const u32 idx = INV ? (N >> (G0 + l + 1)) + (blk << (S - l - 1)) + sb : (1u << (G0 + l)) + (blk << l) + sb;
        w = __ldg((INV ? T.inv_d : T.fwd_d) + idx);
        wh = __ldg((INV ? T.inv_h : T.fwd_h) + idx);
      }
      const double a = v[k], b = v[k + t];
      if (!INV) {
        const double m = fp_mulmod(b, w, wh, q2d);
        v[k] = __dadd_rn(a, m);
        v[k + t] = __dsub_rn(a, m);
      } else {
        v[k] = fp_reduce(__dadd_rn(a, b), qinv, qd);
        v[k + t] = fp_mulmod(__dsub_rn(a, b), w, wh, q2d);
      }
    }
    if (!INV && ((G0 + l) & 1)) {
#pragma unroll
      for (u32 i = 0; i < K; i++) v[i] = fp_reduce(v[i], qinv, qd);
    }
  }
}

template <int LOGN, int P, bool INV>
__device__ __forceinline__ void nf_compute(double (&x)[16], u32 tu, const NttDev& T) {
  constexpr int S = ph_size(LOGN, P), G0 = ph_start(LOGN, P);
  constexpr u32 N = 1u << LOGN, TPU = N / 16, MB = 16 >> S;
  constexpr u32 LSTR = INV ? G0 : LOGN - G0 - S;
#pragma unroll
  for (u32 j = 0; j < MB; j++) nf_block<LOGN, P, INV>(x + j * (1u << S), (tu + j * TPU) >> LSTR, T);
}

// First-phase loads (as nr_load_global) converted to doubles; the OR of the
// centred magnitudes of the loaded words goes to *mag when mag is not null.
template <int LOGN, bool INC, bool INV>
__device__ __forceinline__ void nf_load_global(double (&x)[16], const u64* __restrict__ in, u64 ug, u32 tu,
                                               u64 q, u64* mag) {
  u64 w[16];
  nr_load_global<LOGN, INC, INV>(w, in, ug, tu);
#pragma unroll
  for (u32 i = 0; i < 16; i++) {
    if (mag) *mag |= nr_mag(w[i], q);
    x[i] = fp_from_word(w[i]);
  }
}

// Last-phase stores (as nr_store_global): canonical words, the inverse scaled by 1/n.
template <int LOGN, bool INC, bool INV>
__device__ __forceinline__ void nf_store_global(const double (&x)[16], u64* __restrict__ out, u64 ug, u32 tu,
                                                const NttDev& T, u64* mag) {
  constexpr int P = ph_count(LOGN) - 1, S = ph_size(LOGN, P);
  constexpr u32 N = 1u << LOGN, MB = 16 >> S, K = 1u << S;
  const double qd = T.qd, qinv = T.qinv;
  if (!INV) {
#pragma unroll
    for (u32 j = 0; j < MB; j++) {
      ulonglong2* dst = (ulonglong2*)(out + ug * N + nr_elem<LOGN, P, INV>(tu, j, 0));
#pragma unroll
      for (u32 k = 0; k < K / 2; k++)
        dst[k] = make_ulonglong2(fp_to_word(x[j * K + 2 * k], qinv, qd), fp_to_word(x[j * K + 2 * k + 1], qinv, qd));
    }
  } else {
#pragma unroll
    for (u32 j = 0; j < MB; j++)
#pragma unroll
      for (u32 k = 0; k < K; k++) {
        const u32 e = nr_elem<LOGN, P, INV>(tu, j, k);
        const u64 v = fp_to_word(fp_mulmod(x[j * K + k], T.ninv_d, T.ninv_h, T.q2d), qinv, qd);
        const u64 g = INC ? (ug >> 1) * (2 * N) + 2 * e + (ug & 1) : ug * N + e;
        out[g] = v;
        if (mag) *mag |= nr_mag(v, T.q);
      }
  }
}

template <int LOGN, int P, int PEND, bool INV>
__device__ __forceinline__ void nf_mid(double (&x)[16], double* sm, u32 unit, u32 tu, bool active, const NttDev& T) {
  if constexpr (P < PEND) {
    if (active) {
      nr_load_smem<LOGN, P, INV>(x, sm, unit, tu);
      nf_compute<LOGN, P, INV>(x, tu, T);
      nr_store_smem<LOGN, P, INV>(x, sm, unit, tu);
    }
    __syncthreads();
    nf_mid<LOGN, P + 1, PEND, INV>(x, sm, unit, tu, active, T);
  }
}

// Incomplete transforms of degree-128 ring elements (two 64-point halves)
// with FP64 butterflies, one thread per (element, column r < 8) holding
// both halves: 8 coefficients of each, e = r + 8k in the strided phase and
// e = 8r + k in the contiguous one.  The same butterflies and exchange as
// ntt_fp_kernel<6, true, INV> (identical words), with fewer L1 wavefronts
// per coefficient, the limit of that kernel: the interleaved side moves one
// 16-byte (half 0, half 1) pair per load or store, 8 lanes covering 128
// contiguous bytes of an element; the slot-form side moves 32 bytes per
// lane (256-bit loads and stores, rows 32-byte aligned); the exchange tile
// holds (half 0, half 1) pairs with 16 bytes of padding per 8 pairs, so
// both exchange patterns are free of bank conflicts.
// ---------------------------------------------------------------------------
constexpr u32 NP6_EL = 32;   // ring elements per CTA (4096 coefficients)
constexpr u32 NP6_ROW = 72;  // pairs per element in the exchange tile (64 + 8 padding)
__device__ __forceinline__ u32 np6_pos(u32 el, u32 e) { return el * NP6_ROW + e + (e >> 3); }

__device__ __forceinline__ void st_v4_u64(u64* p, u64 a, u64 b, u64 c, u64 d) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}
__device__ __forceinline__ void ld_v4_u64(const u64* p, u64& a, u64& b, u64& c, u64& d) {
  asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

// Strided phase of the forward transform, exchange and contiguous phase;
// x0 / x1 hold half 0 / 1 at e = r + 8k on entry and at e = 8r + k on exit.
__device__ __forceinline__ void np6_forward(double (&x0)[8], double (&x1)[8], double2* sm, u32 el, u32 r,
                                            bool active, const NttDev& T) {
  if (active) {
    nf_block<6, 0, false>(x0, 0, T);
    nf_block<6, 0, false>(x1, 0, T);
#pragma unroll
    for (u32 k = 0; k < 8; k++) sm[np6_pos(el, r + 8 * k)] = make_double2(x0[k], x1[k]);
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (u32 k = 0; k < 8; k++) {
      const double2 v = sm[np6_pos(el, 8 * r + k)];
      x0[k] = v.x;
      x1[k] = v.y;
    }
    nf_block<6, 1, false>(x0, r, T);
    nf_block<6, 1, false>(x1, r, T);
  }
}

// Canonical words of the slot-form rows (2 e + h) of element e: 32 bytes per store.
__device__ __forceinline__ void np6_store_slots(const double (&x0)[8], const double (&x1)[8], u64* out, u64 eg,
                                                u32 r, const NttDev& T) {
  const double qd = T.qd, qinv = T.qinv;
  u64* d0 = out + 2 * eg * 64 + 8 * r;
#pragma unroll
  for (u32 h = 0; h < 2; h++) {
    const double* x = h ? x1 : x0;
#pragma unroll
    for (u32 c = 0; c < 2; c++)
      st_v4_u64(d0 + h * 64 + 4 * c, fp_to_word(x[4 * c], qinv, qd), fp_to_word(x[4 * c + 1], qinv, qd),
                fp_to_word(x[4 * c + 2], qinv, qd), fp_to_word(x[4 * c + 3], qinv, qd));
  }
}

}  // namespace
}  // namespace salsaa
