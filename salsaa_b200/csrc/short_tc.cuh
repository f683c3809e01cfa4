// short_tc.cuh — prover steps over short witness rows (byte tiles, see
// ntt_img.cuh) on the tensor cores.  Each takes a flag word: the rows were
// short, and the step runs, only while it is zero.
#pragma once
#include "ntt_img.cuh"

namespace salsaa {

// Rows of byte tiles: row k at p + k stride (stride bytes a row), of which
// elements off[k] .. off[k] + width - 1 are used (off a multiple of 64).
struct C8Rows {
  const int8_t* p;
  u64 stride;
  u32 row[MAX_WROWS];
  u64 off[MAX_WROWS];
  u32 rows;
  u64 width;
};

// Fold challenges of (seed, round) as coefficients c (rows x d words) and as
// the negacyclic Toeplitz blocks the fold multiplies by (fold_tz_bytes).
inline u64 fold_tz_bytes(u32 rows, u32 d) { return (u64)rows * 32 * d; }
int launch_fold_challenge_tz(const DevState* ds, u32 round, u32 rows, u32 d, u64 q, u64* c_coef, int8_t* tz,
                             cudaStream_t st);
// The blocks of given challenges c (rows x d canonical words); raises *wide
// when a coefficient is not in [-127, 127].
int launch_fold_words_tz(const u64* c, u32 rows, u32 d, u64 q, int8_t* tz, u32* wide, cudaStream_t st);
// out (nout x d canonical words, the first nout <= width elements) = sum_k c_k w_k in R_q, coefficient form;
// d = 128 or 256, at most 8 rows.  mag_or: OR of the outputs' centred magnitudes.
bool fold_tc_ok(const C8Rows& w, u32 d);
int launch_fold_tc(const C8Rows& w, u32 d, u64 q, const int8_t* tz, u64 nout, u64* out, u64* mag_or, const u32* flag,
                   cudaStream_t st);

// Projection of launch_project (kernels.cuh): rows w.rows, chunks of cw
// elements, out word rows [(row, chunk)][256][d]; runs only while *wide == 0.
bool project_tc_ok(const C8Rows& w, u32 d, u32 cw);
int launch_project_tc(const C8Rows& w, u32 d, u64 q, u32 cw, const int8_t* Jc, u64* out, const u32* wide,
                      cudaStream_t st);

// Byte tiles (rows one after the other) of the word rows src; raises *wide
// when a value does not fit a byte (the tiles are then incomplete).  Rows of
// c8_width(width) elements, zero past the width; d a multiple of 16.
inline u64 c8_width(u64 width) { return (width + 63) / 64 * 64; }
int launch_words_to_c8(const RowSet& src, u32 rows, u64 width, u32 d, u64 q, int8_t* c8, u32* wide, cudaStream_t st);

// Statement rows of launch_commit (kernels.cuh) over byte rows: byte row r
// adds 2^shift[r] times its sums to witness row dst[r], unless *wide[dst[r]]
// is nonzero (then launch_sc_umma takes that row).
struct Sc8Rows {
  C8Rows w;
  u32 dst[MAX_WROWS], shift[MAX_WROWS];
  const u32* wide[MAX_WROWS];  // per witness row
};
int launch_sc_tc(const Sc8Rows& w, u32 rows, u32 d, u32 Bw, u32 nhi, const ScRange& rg, const u64* s_hi,
                 const ModQ& M, u64* acc, const uint8_t* img, cudaStream_t st);

}  // namespace salsaa
