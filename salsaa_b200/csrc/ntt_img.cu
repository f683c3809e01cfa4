// ntt_img.cu — forward incomplete transforms that write the byte image of
// the slot form (ntt_img.cuh) for the tensor-core key-row product.
#include "ntt_img.cuh"
#include "ntt_tile.cuh"

namespace salsaa {

namespace {

// A CTA transforms EL ring elements (16 values per thread) and writes their
// image rows: EL / 16 units of 16 elements per (slot, byte row).  The
// transform is ntt_fp6_kernel's (d = 128) or ntt_fp_kernel's (d = 256, 512);
// its canonical words go back to the exchange tile, each thread gathers 16
// elements of one (slot, half), transposes them into 7 byte rows of 16
// bytes, and the rows of a slot (224 bytes) leave as full sectors through a
// second shared tile.  Tiles: IU units per slot, odd, so neighbouring slots
// start on different bank groups.
template <int LOGN>
struct ImgGeom {
  static constexpr u32 N = 1u << LOGN, D = 2 * N;
  static constexpr u32 THREADS = LOGN == 8 ? 512 : 256;
  static constexpr u32 EL = THREADS * 16 / D, JG = EL / 16;
  static constexpr u32 IU = 14 * JG + 1;
  static constexpr u32 WORDS = LOGN == 6 ? NP6_EL * NP6_ROW * 2 : THREADS * 17;  // exchange tile, words
  static constexpr u32 IMG = N * IU * 16;                                        // image tile, bytes
  static constexpr u32 SMEM = WORDS * 8 > IMG ? WORDS * 8 : IMG;
};

__device__ __forceinline__ void img_transpose4(u32 a, u32 b, u32 c, u32 d, u32& o0, u32& o1, u32& o2, u32& o3) {
  const u32 t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
  const u32 t2 = __byte_perm(c, d, 0x5140), t3 = __byte_perm(c, d, 0x7362);
  o0 = __byte_perm(t0, t2, 0x5410);
  o1 = __byte_perm(t0, t2, 0x7632);
  o2 = __byte_perm(t1, t3, 0x5410);
  o3 = __byte_perm(t1, t3, 0x7632);
}

// Digit c (shift sh, mask) of a canonical word: centred and canonical.
__device__ __forceinline__ u64 img_digit(u64 v, u64 q, u32 sh, u64 mask, long long& centred) {
  const bool neg = 2 * v > q;
  const u64 m = neg ? q - v : v;
  const u64 dg = sh >= 64 ? 0 : ((m >> sh) & mask);
  centred = neg ? -(long long)dg : (long long)dg;
  return neg && dg ? q - dg : dg;
}

template <int LOGN, bool DIG>
__global__ void __launch_bounds__(ImgGeom<LOGN>::THREADS) ntt_img_kernel(ImgDigits a, CkImage im, NttDev T) {
  pdl_wait();
  using Geo = ImgGeom<LOGN>;
  constexpr u32 N = Geo::N, D = Geo::D, JG = Geo::JG, EL = Geo::EL;
  extern __shared__ __align__(16) unsigned char ni_smem[];
  const u32 tid = threadIdx.x;
  const ImgRows& R = a.rows;
  const u64 q = T.q;
  // source element group of this CTA: elements e0 .. of source row k; the
  // digit transform takes 16 source elements and both digits (d = 128: one
  // CTA, digit = local element & 1), or one digit per CTA
  constexpr u32 SEL = DIG ? 16 : EL;  // source elements per CTA
  if (R.gate && !*R.gate) return;
  const u64 nblk = R.rows * (R.width / SEL) * (DIG && JG == 1 ? 2 : 1);
  u32 rlog = 0;
  u64 mask = 0, mag = 0;
  if (DIG) {
    const u64 orv = *a.bw_or;
    const u32 bw = orv ? 64u - (u32)__clzll((long long)orv) : 0u;
    rlog = (bw + 1) / 2;
    mask = rlog >= 64 ? ~0ULL : ((1ULL << rlog) - 1);
    if (blockIdx.x == 0 && tid == 0) {
      *a.rlog_out = rlog;
      if (a.radix_out) *a.radix_out = 1ULL << rlog;
    }
  }
  for (u64 b0 = blockIdx.x; b0 < nblk; b0 += gridDim.x) {
    u64 blk = b0;
    u32 dig = 0;
    if (DIG && JG == 1) {
      dig = (u32)(blk & 1);
      blk >>= 1;
    }
    u32 k;
    u64 e0;
    img_item(R, im, SEL == 32 ? 5 : 4, (u32)blk, k, e0);
    const u64* src = R.src[k] + e0 * D;
    // output row of the (split) digit or source space for group jg
    auto out_row = [&](u32 jg) -> u32 { return DIG ? 2 * k + (JG == 2 ? jg : dig) : k; };
    const u32 out_rows = DIG ? 2 * R.rows : R.rows;

    // ---- transform; the words end in the exchange tile ----
    u64* words = (u64*)ni_smem;
    if constexpr (LOGN == 6) {
      double2* sm = (double2*)ni_smem;
      const u32 el = tid >> 3, r = tid & 7;
      const u32 sel = DIG ? el >> 1 : el, c = DIG ? el & 1 : 0;
      double x0[8], x1[8];
#pragma unroll
      for (u32 kk = 0; kk < 8; kk++) {
        const u32 e = r + 8 * kk;
        ulonglong2 v = __ldg((const ulonglong2*)(src + sel * D + 2 * e));
        if (DIG) {
          long long d0, d1;
          v.x = img_digit(v.x, q, c * rlog, mask, d0);
          v.y = img_digit(v.y, q, c * rlog, mask, d1);
          if (a.coef)
            *(int2*)(a.coef + ((u64)(2 * k + c) * R.width + e0 + sel) * D + 2 * e) = make_int2((int)d0, (int)d1);
        } else if (R.mag_or) {
          mag |= nr_mag(v.x, q) | nr_mag(v.y, q);
        }
        x0[kk] = fp_from_word(v.x);
        x1[kk] = fp_from_word(v.y);
      }
      np6_forward(x0, x1, sm, el, r, true, T);
      const double qd = T.qd, qinv = T.qinv;
      u64 w0[8], w1[8];
#pragma unroll
      for (u32 kk = 0; kk < 8; kk++) {
        w0[kk] = fp_to_word(x0[kk], qinv, qd);
        w1[kk] = fp_to_word(x1[kk], qinv, qd);
      }
      if (R.slots) {
        u64* d0 = R.slots + ((u64)out_row(c) * R.width + e0 + sel) * D + 8 * r;
#pragma unroll
        for (u32 h = 0; h < 2; h++) {
          const u64* w = h ? w1 : w0;
          st_v4_u64(d0 + h * N, w[0], w[1], w[2], w[3]);
          st_v4_u64(d0 + h * N + 4, w[4], w[5], w[6], w[7]);
        }
      }
      // a thread rewrites the exchange positions it read itself
      ulonglong2* smw = (ulonglong2*)ni_smem;
#pragma unroll
      for (u32 kk = 0; kk < 8; kk++) smw[np6_pos(el, 8 * r + kk)] = make_ulonglong2(w0[kk], w1[kk]);
    } else {
      constexpr int PL = ph_count(LOGN) - 1;
      double* sm = (double*)ni_smem;
      u32 unit, tu;
      nr_map<LOGN, true>(tid, unit, tu);
      u64 w[16];
      double x[16];
      nr_load_global<LOGN, true, false>(w, src, unit, tu);
#pragma unroll
      for (u32 i = 0; i < 16; i++) {
        if (DIG) {
          long long d0;
          w[i] = img_digit(w[i], q, dig * rlog, mask, d0);
          if (a.coef) {
            constexpr u32 K0 = 1u << ph_size(LOGN, 0);
            const u32 e = nr_elem<LOGN, 0, false>(tu, i / K0, i % K0);
            a.coef[((u64)(2 * k + dig) * R.width + e0 + (unit >> 1)) * D + 2 * e + (unit & 1)] = (int)d0;
          }
        } else if (R.mag_or) {
          mag |= nr_mag(w[i], q);
        }
        x[i] = fp_from_word(w[i]);
      }
      nf_compute<LOGN, 0, false>(x, tu, T);
      nr_store_smem<LOGN, 0, false>(x, sm, unit, tu);
      __syncthreads();
      nf_mid<LOGN, 1, PL, false>(x, sm, unit, tu, true, T);
      nr_load_smem<LOGN, PL, false>(x, sm, unit, tu);
      nf_compute<LOGN, PL, false>(x, tu, T);
#pragma unroll
      for (u32 i = 0; i < 16; i++) w[i] = fp_to_word(x[i], T.qinv, T.qd);
      if (R.slots) {
        constexpr u32 KL = 1u << ph_size(LOGN, PL);
        u64* d0 = R.slots + ((u64)out_row(0) * R.width + e0) * D + (u64)unit * N;
#pragma unroll
        for (u32 i = 0; i < 16; i += 2)
          *(ulonglong2*)(d0 + nr_elem<LOGN, PL, false>(tu, i / KL, i % KL)) = make_ulonglong2(w[i], w[i + 1]);
      }
      nr_store_smem<LOGN, PL, false>(w, words, unit, tu);
    }
    __syncthreads();

    // ---- byte rows of (slot s, half h, group jg) ----
    constexpr u32 US = Geo::IU;
    u32 s, h, jg;
    if constexpr (LOGN == 6) {
      h = tid & 1;
      s = (tid >> 1) & (N - 1);
      jg = tid >> 7;
    } else {
      s = tid & (N - 1);
      h = tid >> LOGN;
      jg = 0;
    }
    uint4 pl[7];
#pragma unroll
    for (u32 q4 = 0; q4 < 4; q4++) {
      u32 lo[4], hi[4], p[8];
#pragma unroll
      for (u32 e = 0; e < 4; e++) {
        const u32 t = 4 * q4 + e;
        u64 w;
        if constexpr (LOGN == 6) {
          const u32 el = DIG ? 2 * t + jg : 16 * jg + t;
          w = words[2 * np6_pos(el, s) + h];
        } else {
          w = words[npad((2 * t + h) * N + s)];
        }
        lo[e] = (u32)w;
        hi[e] = (u32)(w >> 32);
      }
      img_transpose4(lo[0], lo[1], lo[2], lo[3], p[0], p[1], p[2], p[3]);
      img_transpose4(hi[0], hi[1], hi[2], hi[3], p[4], p[5], p[6], p[7]);
#pragma unroll
      for (u32 y = 0; y < 7; y++) {
        if (q4 == 0) pl[y].x = p[y];
        if (q4 == 1) pl[y].y = p[y];
        if (q4 == 2) pl[y].z = p[y];
        if (q4 == 3) pl[y].w = p[y];
      }
    }
    __syncthreads();
    uint4* tile = (uint4*)ni_smem;
#pragma unroll
    for (u32 y = 0; y < 7; y++) tile[s * US + jg * 14 + h * 7 + y] = pl[y];
    __syncthreads();
    // image units of the JG groups: 14 units per (slot, group)
    const u64 w2 = R.split ? R.width / 2 : R.width;
    u64 base[JG];
#pragma unroll
    for (u32 g = 0; g < JG; g++) {
      const u64 i = DIG ? e0 : e0 + 16 * g;
      const u32 row = out_row(g);
      const bool second = i >= w2;
      base[g] = cki_unit(im, R.k0 + row + (second ? out_rows : 0), second ? i - w2 : i);
    }
    uint4* out = (uint4*)im.p;
    const u32 sstride = 4 * im.VP;
    for (u32 u = tid; u < N * 14 * JG; u += Geo::THREADS) {
      const u32 ss = u / (14 * JG), rem = u % (14 * JG);
      const u32 g = JG == 2 && rem >= 14 ? 1 : 0;
      out[(g ? base[JG - 1] : base[0]) + (u64)ss * sstride + (rem - 14 * g)] = tile[ss * US + rem];
    }
    __syncthreads();
  }
  if (!DIG && R.mag_or) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mag |= __shfl_xor_sync(0xffffffffu, mag, o);
    if ((tid & 31) == 0 && mag) atomicOr((unsigned long long*)R.mag_or, (unsigned long long)mag);
  }
}

template <int LOGN, bool DIG>
int img_go(const ImgDigits& a, const CkImage& im, const NttDev& T, cudaStream_t st) {
  using Geo = ImgGeom<LOGN>;
  const u32 sel = DIG ? 16 : Geo::EL;
  const u64 blocks = a.rows.rows * (a.rows.width / sel) * (DIG && Geo::JG == 1 ? 2 : 1);
  if (blocks > 0x7fffffffULL) return salsaa_set_error(-2, "ntt_img: batch too large");
  auto kern = ntt_img_kernel<LOGN, DIG>;
  if (Geo::SMEM > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Geo::SMEM);
    if (e != cudaSuccess) return salsaa_set_cuda_error(e, "ntt_img smem attribute");
  }
  // words in, words out or 7 image bytes; nothing behind a gate, which is nearly always closed
  const double coeffs = a.rows.gate ? 0.0 : (double)a.rows.rows * a.rows.width * Geo::D;
  const int tr = salsaa_trace_begin(DIG ? "ntt_digits_kernel" : "ntt_kernel", st,
                                    coeffs * (DIG ? 8 + 2 * (7 + 4 + (a.rows.slots ? 8 : 0))
                                                  : 15 + (a.rows.slots ? 8 : 0)));
  // gated: a grid that leaves quickly when the gate is closed
  const u64 grid = a.rows.gate && blocks > 444 ? 444 : blocks;
  pdl(kern, (unsigned)grid, Geo::THREADS, Geo::SMEM, st)(a, im, T);
  salsaa_trace_end(tr, st);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ntt_img launch");
}

template <bool DIG>
int img_launch(const ImgDigits& a, const CkImage& im, const NttDev& T, cudaStream_t st) {
  const ImgRows& R = a.rows;
  const u64 w2 = R.split ? R.width / 2 : R.width;
  const u32 out_rows = (DIG ? 2 : 1) * R.rows;
  if (!im.p || im.n != T.n || im.width != w2 || R.k0 + out_rows * (R.split ? 2 : 1) > im.R || R.rows == 0 ||
      R.rows > MAX_WROWS || w2 < CKI_CHUNK || (R.width & (R.width - 1)))
    return salsaa_set_error(-2, "ntt_img: rows outside the image");
  for (u32 k = 0; k < R.rows; k++)
    if (!R.src[k] || (uintptr_t)R.src[k] % 16) return salsaa_set_error(-2, "ntt_img: rows must be 16-byte aligned");
  if ((uintptr_t)R.slots % 32) return salsaa_set_error(-2, "ntt_img: slot rows must be 32-byte aligned");
  switch (T.logn) {
    case 6: return img_go<6, DIG>(a, im, T, st);
    case 7: return img_go<7, DIG>(a, im, T, st);
    case 8: return img_go<8, DIG>(a, im, T, st);
    default: return salsaa_set_error(-2, "ntt_img: needs 64, 128 or 256 slots");
  }
}

// Gated inverse incomplete transform (ntt_fp_kernel's, one 4096-coefficient
// tile per step of a grid that leaves quickly when the gate is closed).
template <int LOGN>
__global__ void __launch_bounds__(256) ntt_inv_gated_kernel(const u64* in, u64* out, u64 units, NttDev T,
                                                            const u32* gate, u64* mag_or) {
  pdl_wait();
  constexpr int PL = ph_count(LOGN) - 1;
  constexpr u32 UPT = NR_TILE >> LOGN;
  __shared__ double sm[NR_TILE + NR_TILE / 16];
  if (!*gate) return;
  u32 unit, tu;
  nr_map<LOGN, true>(threadIdx.x, unit, tu);
  u64 mag = 0;
  for (u64 b = blockIdx.x; b * UPT < units; b += gridDim.x) {
    const u64 ug = b * UPT + unit;
    const bool active = ug < units;
    double x[16];
    if (active) {
      nf_load_global<LOGN, true, true>(x, in, ug, tu, T.q, nullptr);
      nf_compute<LOGN, 0, true>(x, tu, T);
      nr_store_smem<LOGN, 0, true>(x, sm, unit, tu);
    }
    __syncthreads();
    if (active) {
      nr_load_smem<LOGN, PL, true>(x, sm, unit, tu);
      nf_compute<LOGN, PL, true>(x, tu, T);
      nf_store_global<LOGN, true, true>(x, out, ug, tu, T, mag_or ? &mag : nullptr);
    }
    __syncthreads();
  }
  if (mag_or) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mag |= __shfl_xor_sync(0xffffffffu, mag, o);
    if ((threadIdx.x & 31) == 0 && mag) atomicOr((unsigned long long*)mag_or, (unsigned long long)mag);
  }
}

}  // namespace

int ntt_inv_gated_launch(const u64* in, u64* out, u64 count, const NttDev& T, const u32* gate, u64* mag_or,
                         cudaStream_t st) {
  if ((T.logn != 6 && T.logn != 7) || T.q >= NR_RELAX_Q || (uintptr_t)in % 16 || (uintptr_t)out % 16 || !gate)
    return salsaa_set_error(-2, "ntt_inv_gated: shape or alignment not supported");
  const u64 units = 2 * count, tiles = (units * T.n + NR_TILE - 1) / NR_TILE;
  const unsigned grid = (unsigned)(tiles < 592 ? tiles : 592);
  if (T.logn == 6) pdl(ntt_inv_gated_kernel<6>, grid, 256, 0, st)(in, out, units, T, gate, mag_or);
  else pdl(ntt_inv_gated_kernel<7>, grid, 256, 0, st)(in, out, units, T, gate, mag_or);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ntt_inv_gated launch");
}

int ntt_img_launch(const ImgRows& a, const CkImage& im, const NttDev& T, cudaStream_t st) {
  ImgDigits d{};
  d.rows = a;
  return img_launch<false>(d, im, T, st);
}
int ntt_img_digits_launch(const ImgDigits& a, const CkImage& im, const NttDev& T, cudaStream_t st) {
  if (!a.bw_or || !a.rlog_out) return salsaa_set_error(-2, "ntt_img: digits need their magnitude word");
  return img_launch<true>(a, im, T, st);
}

}  // namespace salsaa
