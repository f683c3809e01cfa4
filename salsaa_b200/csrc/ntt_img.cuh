// ntt_img.cuh — byte images of slot-form witnesses: the operand layout the
// tensor-core key-row product (ck_img.cu) copies straight into shared memory,
// and the forward transforms (ntt_img.cu) that write it.
#pragma once
#include "kernels.cuh"

namespace salsaa {

// Byte image of R witness rows of `width` ring elements in slot form.  With
// bt = min(width, key-table block), element i = hi bt + lo.  G key blocks
// (hi = hg G + g) are stacked as virtual rows v = g R + k, so one tile shares
// its key bytes among them.  Row (v, half h, byte y) of a tile is
// 14 v + 7 h + y; rows are padded to VP (a multiple of 8).  The 16 bytes of
// elements 16 j .. 16 j + 15 of one row are one unit:
//   unit(hg, chunk c = lo / 64, slot s, j = (lo / 16) % 4, row)
//     = (((hg nlc + c) n + s) 4 + j) VP + row,
// i.e. a (chunk, slot) tile is 64 VP contiguous bytes in the K-major operand
// layout (16-byte K slices of VP rows each), one bulk copy.
struct CkImage {
  uint8_t* p;
  u32 R, G, VP, n, btlog, nlc, nhg, glog;  // glog: log2 G
  u64 width;
};
constexpr u32 CKI_CHUNK = 64;
// Most virtual rows of a tile: 9 x 14 = 126 of the MMA's 128 rows.
constexpr u32 CKI_MAX_V = 9;

inline u32 cki_vp(u32 V) { return (V * 14 + 7) / 8 * 8; }
// Shape of the image of R rows x width under a key table of ck_bt elements per block.
CkImage cki_shape(u32 R, u64 width, u32 n, u32 ck_bt);
u64 cki_bytes(const CkImage& im);
// n, q and the key table fit the image path: FP64 transforms (q < 2^50) of
// n = 64, 128 or 256 slots, a power-of-two width of at least 64 elements.
bool cki_ok(u32 R, u64 width, u32 n, u32 ck_bt, u64 q);

// 16-byte unit index of (image row k, element i, slot 0, byte row 0); i a multiple of 16.
__device__ __forceinline__ u64 cki_unit(const CkImage& im, u32 k, u64 i) {
  const u32 hi = (u32)(i >> im.btlog), lo = (u32)i & ((1u << im.btlog) - 1);
  const u32 g = hi & (im.G - 1), hg = hi >> im.glog;
  return (u64)((hg * im.nlc + (lo >> 6)) * im.n * 4 + ((lo >> 4) & 3)) * im.VP + (g * im.R + k) * 14;
}

// Forward incomplete transform of coefficient-form rows (canonical words)
// into the image.  Row r of the source (rows x width) becomes image row
// k0 + r; with split != 0 its two halves become the image rows k0 + r and
// k0 + rows + r of width / 2.
struct ImgRows {
  const u64* src[MAX_WROWS];
  u32 rows, k0, split;
  u64 width;
  u64* slots;        // slot-form words too (rows x width), or null
  u64* mag_or;       // OR of the centred magnitudes of the source, or null
  const u32* gate;   // run only if *gate != 0 (the tensor-core transform gave up), or null
};
int ntt_img_launch(const ImgRows& a, const CkImage& im, const NttDev& T, cudaStream_t st);

// Source row k and first element e0 of item `item` (2^sellog elements, at most
// 64).  All rows of one tile (source rows, halves, stacked key blocks) come
// from consecutive items, so the 224-byte runs that they write side by side
// meet in L2.  32-bit arithmetic: a 64-bit division costs hundreds of clocks.
__device__ __forceinline__ void img_item(const ImgRows& R, const CkImage& im, u32 sellog, u32 item, u32& k, u64& e0) {
  const u32 slog = R.split ? 1 : 0, t = item / (R.rows << (slog + im.glog));
  u32 f = item - t * (R.rows << (slog + im.glog));
  const u32 f2 = f / R.rows, hs = f2 & slog, g = f2 >> slog;
  k = f - f2 * R.rows;
  const u32 pl = im.btlog - sellog, lg = t & ((1u << pl) - 1), hg = t >> pl;
  e0 = (hs ? R.width / 2 : 0) + ((u64)((hg << im.glog) + g) << im.btlog) + ((u64)lg << sellog);
}

// The same for the two decomposition digits of each source row: digit c of
// row r is row 2 r + c of the digit space (2 rows x width), whose halves
// become image rows as above.  bw_or, rlog_out, radix_out as in
// ntt_digits_launch; coef: the digits as centred int32.
struct ImgDigits {
  ImgRows rows;
  const u64* bw_or;
  u64* rlog_out;
  u64* radix_out;
  int* coef;
};
int ntt_img_digits_launch(const ImgDigits& a, const CkImage& im, const NttDev& T, cudaStream_t st);

// The same transforms on the tensor cores, for short values (ntt_tc.cu; d =
// 128 or 256): source values of 8 bits (limbs = 1) or 16 (limbs = 2) or, with
// bw_or, the two digits when they are at most 7 bits.  Values that do not fit
// set *flag (zeroed by the caller; digits write it), and the image is then
// incomplete: launch ntt_img_launch / ntt_img_digits_launch gated on it.
// c8: the short values themselves as byte tiles (see below), rows as the
// source's (digits: row 2 r + c; two limbs: rows 2 r and 2 r + 1, low and high
// byte, both signed), or null.
struct TcArgs {
  ImgRows rows;  // slots are not used
  u32* flag;
  int8_t* c8;
  int* coef;         // the digits as centred int32 in source order, or null
  const u64* bw_or;  // digits only
  u64* rlog_out;
  u64* radix_out;
};
// Byte tiles of a row of width x d values: 64 elements each, 16-position
// slices of 64 x 16 bytes,
//   offset(i, p) = (i / 64) 64 d + (p / 16) 1024 + (i % 64) 16 + p % 16.
// One tile is contiguous and an operand as it lies: K-major with elements as
// rows and positions as K, or MN-major with positions as rows and elements as K.
__host__ __device__ inline u64 c8_offset(u64 i, u32 p, u32 d) {
  return (i >> 6) * 64 * d + (u64)(p >> 4) * 1024 + (i & 63) * 16 + (p & 15);
}
bool ntt_tc_ok(const NttDev& T);
int ntt_tc_launch(const TcArgs& a, int limbs, const CkImage& im, const NttDev& T, cudaStream_t st);

// Transform of rows that are usually short: on the tensor cores when the
// shapes allow, else (or, gated on *flag, when a value does not fit) FP64.
int ntt_short_img_launch(const ImgRows& a, u32* flag, const CkImage& im, const NttDev& T, cudaStream_t st);

// Inverse incomplete transform of `count` elements (n = 64 or 128, q < 2^50),
// run only if *gate != 0; mag_or as in ntt_launch.
int ntt_inv_gated_launch(const u64* in, u64* out, u64 count, const NttDev& T, const u32* gate, u64* mag_or,
                         cudaStream_t st);

// Key rows x image (q < 2^50): the sums of key row r and witness row k are
// added to acc row r * R + k (slot form, zeroed by the caller).
struct CkImgArgs {
  const uint8_t* tk8;
  const u64* thi;
  u32 nck, ck_bt, ck_nhi;
  u64* acc;
};
int launch_ck_img(const CkImgArgs& a, const CkImage& im, const ModQ& M, const u64* zeta, cudaStream_t st);

}  // namespace salsaa
