// gram.cuh — streaming passes of the norm-check sumchecks on the tensor cores
// (norm_check_1 and sum_check, src/subroutines/fast_norm_check.rs:135-320).
//
// A pass takes four rounds.  It reads groups v_g = (x[g + m ng])_{m < 16} of a
// vector; the fold challenges are known up front, so
//   * the folded vector is x'[g] = sum_m lambda[m] v_g[m] with
//     lambda[m] = prod_t (bit_{3-t}(m) ? c_t : 1 - c_t), and
//   * every value of the four rounds is a fixed linear combination of v_g, so
//     all the rounds' sums follow from the 16 x 16 Gram matrix
//     C = sum_g v_g v_g^T mod q (gram_sums in kernels.cu).
#pragma once
#include "kernels.cuh"
#include "short_tc.cuh"

namespace salsaa {

// One vector of a batched pass (launch_sumcheck_batch).
struct SbInst {
  const u64* in;
  u64* out;
  u64 L;     // current length
  u64 tile0; // first tile of this instance in the level's tile space
  u32 j;     // index of the next round
  u32 id;    // instance index: its challenge stream and its rows of sums
};
constexpr u32 SB_MAX_INST = 64, SB_GPT = 4, SB_TILE_GROUPS = 256 * SB_GPT;

constexpr u32 GRAM_TILE = 256;  // groups of one tile of words

// Words below 2^64 as eight bytes each; vectors of 4096 values and more.
inline bool gram_words_ok(u64 len, u64 q) {
  return q > (1ULL << 47) && q < (1ULL << 62) && len % (16ULL * GRAM_TILE) == 0 && len >= 16ULL * GRAM_TILE;
}

// Rounds 0..3 of both repetitions over `rows` witness rows (words or int32) of
// n values: out[(rep rows + k) sout + g] and gram[k][256] (added to; zero at
// first).  gate: run only while *gate is nonzero (null: always).
int launch_gram_first(const RowSet& w, u32 rows, u64 n, const ModQ& M, const DevState* ds, u32 round, u64* out,
                      u64 sout, u64* gram, const u32* gate, cudaStream_t st);
// Rounds j .. j + 3 of 2 rows vectors of L words, vector (rep, k) at
// in + (rep rows + k) sin; gram[rep rows + k][256].
int launch_gram_round(const u64* in, u64 sin, u64* out, u64 sout, u64 L, u32 rows, const ModQ& M, const DevState* ds,
                      u32 round, u32 j, u64* gram, cudaStream_t st);
// One level of a batch: ninst vectors over ntiles tiles of SB_TILE_GROUPS
// groups (inst in device memory); gram[id][256].
int launch_gram_batch(const SbInst* inst, u32 ninst, u64 ntiles, const ModQ& M, u64 seed, u32 round, u64* gram,
                      cudaStream_t st);
// launch_gram_first over byte rows; runs only while *wide is zero.
bool gram_c8_ok(const C8Rows& w, u32 d, u64 q);
int launch_gram_c8(const C8Rows& w, u32 d, const ModQ& M, const DevState* ds, u32 round, u64* out, u64 sout,
                   u64* gram, const u32* wide, cudaStream_t st);

}  // namespace salsaa
