// ck_umma.cu — tensor-core (tcgen05 / TMEM) paths for the commitment
// products, and a self-test of the int8 tensor-core building block.
#include <cuda_runtime.h>

#include "../../include/salsaa_gpu.h"
#include "kernels.cuh"
#include "ntt.cuh"
#include "umma.cuh"

using namespace salsaa;

namespace {

// D (128 x N, s32) = A (128 x K, u8) * B (N x K, u8)^T on one CTA: the
// operands are packed into the canonical K-major layout by the threads, the
// MMAs are issued by one thread, and the accumulator is read back from TMEM.
__global__ void __launch_bounds__(128) umma_selftest_kernel(const uint8_t* A, const uint8_t* B, u32 N, u32 K,
                                                            int32_t* out, u32* err) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t mbar;
  __shared__ uint32_t tslot;
  uint8_t* sa = sm;
  uint8_t* sb = sm + 128 * K;
  const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (u32 t = tid; t < 128 * K; t += 128) {
    const u32 r = t / K, k = t % K;
    sa[(k / 16) * (128 * 16) + r * 16 + k % 16] = A[t];
  }
  for (u32 t = tid; t < N * K; t += 128) {
    const u32 r = t / K, k = t % K;
    sb[(k / 16) * (N * 16) + r * 16 + k % 16] = B[t];
  }
  if (tid == 0) {
    umma::mbar_init(&mbar, 1);
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 256);
  umma::fence_proxy_async();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;
  if (tid == 0) {
    const u32 idesc = umma::idesc_u8(128, N);
    for (u32 ks = 0; ks < K / 32; ks++) {
      const uint64_t ad = umma::desc_kmajor(umma::smem_u32(sa + ks * 2 * 128 * 16), 128 * 16, 128);
      const uint64_t bd = umma::desc_kmajor(umma::smem_u32(sb + ks * 2 * N * 16), N * 16, 128);
      umma::mma_i8(tmem, ad, bd, idesc, ks > 0);
    }
    umma::commit(&mbar);
  }
  __syncwarp();
  bool ok = umma::mbar_wait(&mbar, 0, err, 1);
  ok = __all_sync(0xffffffffu, ok);
  umma::fence_after_sync();
  if (ok) {
    for (u32 c = 0; c < N; c += 16) {
      uint32_t r[16];
      umma::tmem_ld16(tmem + ((warp * 32) << 16) + c, r);
      umma::tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; j++) out[(warp * 32 + lane) * N + c + j] = (int32_t)r[j];
    }
  } else {
    umma::mbar_wait(&mbar, 0, err, 2);  // give an MMA in flight more time before freeing TMEM
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------
// Commitment-key rows on tcgen05 (q < 2^56).  Per NTT slot s the key rows'
// contribution to the commitment is a matrix product over F_q[X]/(X^2 - zeta):
// with the key power T = (c, d) and the witness value W = (a, b),
//   re = sum c a + zeta sum d b,    im = sum c b + sum d a.
// Every value is split into 7 bytes, so one u8 x u8 -> s32 tensor-core
// product per slot gives all four sums exactly (2048 byte products per block
// stay below 2^27):
//   A (M = 128): witness rows (k, part a|b, byte y), y-th byte of W,
//   B (N = nkp): key rows (r, comp c|d, byte x), x-th byte of T,
//   D[(k,p,y)][(r,c,x)] = sum_i byte_y(W_k,p(i)) byte_x(T_r,c(i)),
// and value = sum_{x,y} 2^(8(x+y)) D mod q.  The key bytes are laid out once
// per context in the operand's shared-memory image (ck_tk8), so each
// 64-element chunk of both slots' key tiles is one bulk copy.
//
// CTA = (slot pair s0, s0 + 1; block of Bw elements), warp-specialised per
// 64-element chunk, with no CTA-wide barrier inside the loop: warps 0..13
// load the witness pairs (one 16-byte load covers both slots) and split them
// into byte planes in shared memory, then arrive on the stage's a_full
// mbarrier; one thread of warp 14 bulk-copies the two key tiles as soon as
// the MMAs that read the stage's previous keys complete (key_full); one
// thread of warp 15 issues 2 x 2 MMAs (K = 32) into two TMEM accumulators
// once both are full, and commits them to the stage's done mbarrier, which
// frees the stage for the next witness and key copies.  Two stages.  Every
// wait is bounded; a role that gives up stops its loop, and the others then
// give up on the arrivals it no longer makes.  Epilogue: each thread reads its TMEM lane (one
// witness byte row), folds the key bytes x, the block's 7 y-rows are folded
// through shared memory, and the result is multiplied by the block's high
// key factor and added into the accumulator as in the CUDA-core path.
// ---------------------------------------------------------------------------
constexpr u32 CKU_CHUNK = 64;  // elements per pipeline step (K of 2 MMAs per slot)
constexpr u32 CKU_THREADS = 512;
constexpr u32 CKU_CONV = 448;  // witness-converting threads (warps 0..13); warps 14, 15 copy keys and issue MMAs
constexpr u32 CKU_ATILE = 128 * CKU_CHUNK;  // witness byte tile of one slot

__global__ void ck_tk8_kernel(const u64* tlo, u32 nck, u32 n, u32 bt, u32 nkp, bool packed, uint8_t* tk8) {
  pdl_wait();
  const u64 tot = (u64)bt * n * nkp;
  for (u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (u64)gridDim.x * blockDim.x) {
    const u32 b = (u32)(t % 16);
    u64 rest = t / 16;
    const u32 row = (u32)(rest % nkp);
    rest /= nkp;
    const u32 j = (u32)(rest % (CKU_CHUNK / 16));
    rest /= CKU_CHUNK / 16;
    const u32 s = (u32)(rest % n), cc = (u32)(rest / n);
    uint8_t v = 0;
    if (row < nck * 14) {
      const u32 r = row / 14, comp = (row / 7) % 2, x = row % 7;
      const u32 lo = cc * CKU_CHUNK + j * 16 + b;
      u64 val = tlo[((u64)r * bt + lo) * 3 * n + (u64)comp * n + s];
      if (packed) val = ((val >> 32) << 25) | (val & 0x1FFFFFFull);
      v = (uint8_t)(val >> (8 * x));
    }
    tk8[t] = v;
  }
}

__device__ u32 g_tc_error;  // set when a tensor-core wait gave up

// o_i = byte i of a, b, c, d (in that order, a in the low byte)
__device__ __forceinline__ void transpose4x4(u32 a, u32 b, u32 c, u32 d, u32& o0, u32& o1, u32& o2, u32& o3) {
  const u32 t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
  const u32 t2 = __byte_perm(c, d, 0x5140), t3 = __byte_perm(c, d, 0x7362);
  o0 = __byte_perm(t0, t2, 0x5410);
  o1 = __byte_perm(t0, t2, 0x7632);
  o2 = __byte_perm(t1, t3, 0x5410);
  o3 = __byte_perm(t1, t3, 0x7632);
}

// One CTA of the key-row product: element-block group `by` of the witness w
// (rows x width, slot form); its sums go to acc rows (r * acc_rows + koff + k).
__device__ __forceinline__ void ck_umma_body(const uint8_t* __restrict__ tk8, const RowSet& w, u32 rows, u32 G,
                                             u32 nck, u32 nkp, u32 n, u32 bt, u32 Bw, const u64* thi, u32 nhi_t,
                                             const ModQ& M, const u64* zeta, u64* acc, u32 acc_rows, u32 koff,
                                             bool plain, u32 by) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t key_full[2], a_full[2], done_bar[2];
  __shared__ uint32_t tslot, last_commit;
  const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const u32 s0 = 2 * blockIdx.x, d = 2 * n;
  // element blocks g < G of this CTA start at i0 + g bt: the same offsets in
  // the key block, so they share every key tile; their witness rows stack as
  // the virtual rows g * rows + k of the MMA's M dimension
  const u32 lob = bt / Bw, lo_b = by % lob, hg = by / lob;
  const u64 i0 = (u64)hg * G * bt + (u64)lo_b * Bw;
  const u32 vrows = rows * G;
  const u32 btile = nkp * CKU_CHUNK;                  // one slot's key tile
  const u32 stage_bytes = 2 * CKU_ATILE + 2 * btile;  // A0 A1 B0 B1
  const u32 nchunks = Bw / CKU_CHUNK;
  const u32 cc0 = (u32)((i0 % bt) / CKU_CHUNK);
  u32* err = &g_tc_error;

  // zero both stages' witness tiles once: rows >= 14 * rows stay zero
  for (u32 v = tid; v < 2 * 2 * CKU_ATILE / 16; v += CKU_THREADS) {
    const u32 st = v / (2 * CKU_ATILE / 16), o = v % (2 * CKU_ATILE / 16);
    *(uint4*)(smem + st * stage_bytes + o * 16) = make_uint4(0, 0, 0, 0);
  }
  // converter tasks: TS task slots per chunk (kp in groups of 4, elements in
  // quads).  When two groups of TS threads fit, group g takes the chunks
  // c = g mod 2, so few witness rows still keep many loads in flight.  At
  // most two groups: then each stage (c & 1) and its two barriers belong to
  // one group, whose chunks pass them in order; with more groups a group
  // could wait on a stage barrier more than one phase ahead, where a parity
  // wait cannot tell the phases apart.
  const u32 nkpw = 2 * vrows, kpb = (nkpw + 3) / 4, TS = 32 * kpb * (CKU_CHUNK / 32);
  const u32 NG = CKU_CONV / TS >= 2 ? 2 : 1;
  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      umma::mbar_init(&key_full[i], 1);
      umma::mbar_init(&a_full[i], TS);
      umma::mbar_init(&done_bar[i], 1);
    }
    last_commit = 0xffffffffu;
    umma::mbar_fence_init();
  }
  // two accumulators of nkp columns: 2 x 128 columns when they fit, so two
  // CTAs with small key tables can share an SM's 512 TMEM columns
  const u32 cs = nkp <= 128 ? 128 : 256;
  if (warp == 0) umma::tmem_alloc(&tslot, 2 * cs);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;
  bool ok = true;

  if (tid < NG * TS) {
    // witness task t of group gi: (i4lo, kp within a group of 4, i4mid, kp
    // group, i4hi); kp = (virtual row, part).  The same task in every chunk
    // of the group: its source (chunk 0) and shared-memory offset are
    // computed once.  Four register buffers hold the loads of the group's
    // next four chunks.
    const u32 gi = tid / TS, t = tid % TS;
    const u32 i4lo = t & 3, kpi = (t >> 2) & 3, i4mid = (t >> 4) & 1, rest = t >> 5;
    const u32 kp = kpi + 4 * (rest % kpb), i4hi = rest / kpb;
    const bool tval = kp < nkpw;
    const u32 v = kp >> 1, part = kp & 1, k = tval ? v % rows : 0, g = tval ? v / rows : 0;
    const u32 i4 = (i4hi * 2 + i4mid) * 4 + i4lo;  // elements 4 * i4 .. + 3 of the chunk
    const u64* tsrc = w.p[k] + (i0 + (u64)g * bt + i4 * 4) * d + part * n + s0;
    const u32 toff = (i4 >> 2) * (128 * 16) + (kp * 7) * 16 + (i4 & 3) * 4;
    uint4 wb[4][4];
    auto fetch = [&](u32 c, uint4 (&wv)[4]) {
      if (tval) {
        const u64* src = tsrc + (u64)c * CKU_CHUNK * d;
#pragma unroll
        for (u32 e = 0; e < 4; e++) wv[e] = __ldg((const uint4*)(src + (u64)e * d));
      }
    };
    auto stash = [&](u32 st, const uint4 (&wv)[4]) {
      if (!tval) return;
      uint8_t* A = smem + st * stage_bytes;
      // byte plane b of the four elements: a 4 x 4 byte transpose of their
      // low words (planes 0..3) and high words (planes 4..6)
#pragma unroll
      for (u32 sg = 0; sg < 2; sg++) {
        u32 lo[4], hi[4], p[8];
#pragma unroll
        for (u32 e = 0; e < 4; e++) {
          lo[e] = sg ? wv[e].z : wv[e].x;
          hi[e] = sg ? wv[e].w : wv[e].y;
        }
        transpose4x4(lo[0], lo[1], lo[2], lo[3], p[0], p[1], p[2], p[3]);
        transpose4x4(hi[0], hi[1], hi[2], hi[3], p[4], p[5], p[6], p[7]);
#pragma unroll
        for (u32 b = 0; b < 7; b++) *(u32*)(A + sg * CKU_ATILE + toff + b * 16) = p[b];
      }
    };
    // chunk c = gi + NG m: stage c & 1 (last read by the MMAs of chunk c - 2),
    // loads in buffer m & 3, refilled with chunk c + 4 NG once stashed
    auto step = [&](u32 c, uint4 (&wv)[4]) -> bool {
      const u32 st = c & 1;
      if (c >= 2 && !umma::mbar_wait(&done_bar[st], ((c - 2) >> 1) & 1, err, 1)) return false;
      stash(st, wv);
      if (c + 4 * NG < nchunks) fetch(c + 4 * NG, wv);
      umma::fence_proxy_async();
      umma::mbar_arrive(&a_full[st]);
      return true;
    };
#pragma unroll
    for (u32 b = 0; b < 4; b++)
      if (gi + b * NG < nchunks) fetch(gi + b * NG, wb[b]);
    for (u32 c = gi; c < nchunks; c += 4 * NG) {
      if (!(ok = step(c, wb[0]))) break;
      if (c + NG < nchunks && !(ok = step(c + NG, wb[1]))) break;
      if (c + 2 * NG < nchunks && !(ok = step(c + 2 * NG, wb[2]))) break;
      if (c + 3 * NG < nchunks && !(ok = step(c + 3 * NG, wb[3]))) break;
    }
  } else if (warp == CKU_CONV / 32 && lane == 0) {
    // key tiles of both slots, one bulk copy per chunk, into the stage freed
    // by the MMAs of chunk c - 2
    u32 issued = 0;
    for (u32 c = 0; c < nchunks; c++) {
      const u32 st = c & 1;
      if (c >= 2 && !(ok = umma::mbar_wait(&done_bar[st], ((c - 2) >> 1) & 1, err, 4))) break;
      umma::mbar_expect_tx(&key_full[st], 2 * btile);
      umma::bulk_g2s(smem + st * stage_bytes + 2 * CKU_ATILE, tk8 + ((u64)(cc0 + c) * n + s0) * btile, 2 * btile,
                     &key_full[st]);
      issued = c + 1;
    }
    // the copies still in flight (the last one of each stage) land before the CTA moves on
    for (u32 c = issued >= 2 ? issued - 2 : 0; c < issued; c++)
      umma::mbar_wait(&key_full[c & 1], (c >> 1) & 1, err, 5);
  } else if (warp == CKU_CONV / 32 + 1 && lane == 0) {
    const u32 idesc = umma::idesc_u8(128, nkp);
    for (u32 c = 0; c < nchunks; c++) {
      const u32 st = c & 1;
      uint8_t* stage = smem + st * stage_bytes;
      if (!(ok = umma::mbar_wait(&a_full[st], (c >> 1) & 1, err, 2))) break;
      if (!(ok = umma::mbar_wait(&key_full[st], (c >> 1) & 1, err, 2))) break;
      umma::fence_after_sync();
#pragma unroll
      for (u32 sg = 0; sg < 2; sg++)
#pragma unroll
        for (u32 ks = 0; ks < CKU_CHUNK / 32; ks++) {
          const uint64_t ad =
              umma::desc_kmajor(umma::smem_u32(stage + sg * CKU_ATILE + ks * 2 * 128 * 16), 128 * 16, 128);
          const uint64_t bd =
              umma::desc_kmajor(umma::smem_u32(stage + 2 * CKU_ATILE + sg * btile + ks * 2 * nkp * 16), nkp * 16, 128);
          umma::mma_i8(tmem + sg * cs, ad, bd, idesc, (c > 0 || ks > 0) ? 1u : 0u);
        }
      umma::commit(&done_bar[st]);
      last_commit = c;
    }
  }
  // all MMAs done (the last commit covers every earlier MMA of its thread)
  __syncthreads();
  const u32 lc = last_commit;
  if (lc != 0xffffffffu) ok &= umma::mbar_wait(&done_bar[lc & 1], (lc >> 1) & 1, err, 3);
  ok &= lc == nchunks - 1;
  ok = __syncthreads_and(ok);
  umma::fence_after_sync();

  // ---- epilogue ----
  u64* Pm = (u64*)smem;  // [slot][128 lanes][2 nck] partial sums over x
  const u32 ng = 2 * nck;
  // warp w: slot (w >> 2) & 1, TMEM lanes 32 (w & 3) .., and one half of the
  // 2 nck column groups (w >> 3), split at a group boundary
  const u32 sg = (warp >> 2) & 1, row = (warp & 3) * 32 + lane, ch = warp >> 3;
  if (ok) {
    const bool valid = row < vrows * 14;
    const u32 y = row % 7;
    const u64 pw = ((u64)1 << (8 * y)) % M.q;
    const u32 jb = 7 * (ch ? nck : 0), je = 7 * (ch ? 2 * nck : nck);
    u64 hi = 0, lo = 0;
    for (u32 cb = jb / 16; cb * 16 < je; cb++) {
      uint32_t r[16];
      umma::tmem_ld16(tmem + (((warp & 3) * 32) << 16) + sg * cs + cb * 16, r);
      umma::tmem_wait_ld();
#pragma unroll
      for (u32 i = 0; i < 16; i++) {
        const u32 j = cb * 16 + i;
        if (j >= jb && j < je) {
          const u32 x = j % 7;
          const u64 v = (u64)r[i];
          const u64 sl = v << (8 * x), sh = x ? (v >> (64 - 8 * x)) : 0;
          lo += sl;
          hi += sh + (lo < sl);
          if (x == 6) {
            u64 p = (M.s >= 39) ? barrett128(M, hi, lo) : reduce128_any(M, hi, lo);
            if (valid) Pm[((u64)sg * 128 + row) * ng + j / 7] = mul_mod(M, p, pw);
            hi = lo = 0;
          }
        }
      }
    }
  }
  __syncthreads();
  if (ok) {
    for (u32 t = tid; t < 2 * vrows * nck; t += CKU_THREADS) {
      const u32 r = t % nck, v = (t / nck) % vrows, g2 = t / (nck * vrows);
      const u32 k = v % rows, hi_t = (u32)(i0 / bt) + v / rows;
      const u32 s = s0 + g2;
      const u64* P = Pm + (u64)g2 * 128 * ng;
      u64 ca = 0, db = 0, cb = 0, da = 0;
#pragma unroll
      for (u32 y = 0; y < 7; y++) {
        const u64* pa = P + (u64)((2 * v) * 7 + y) * ng;      // part a rows
        const u64* pb = P + (u64)((2 * v + 1) * 7 + y) * ng;  // part b rows
        ca = salsaa::add_mod(ca, pa[2 * r], M.q);
        da = salsaa::add_mod(da, pa[2 * r + 1], M.q);
        cb = salsaa::add_mod(cb, pb[2 * r], M.q);
        db = salsaa::add_mod(db, pb[2 * r + 1], M.q);
      }
      u64 re = salsaa::add_mod(ca, mul_mod(M, zeta[s], db), M.q);
      u64 im = salsaa::add_mod(cb, da, M.q);
      const u64* th = thi + ((u64)r * nhi_t + hi_t) * d;
      slot_mul(M, re, im, th[s], th[n + s], zeta[s], re, im);
      u64* dst = acc + ((u64)r * acc_rows + koff + k) * d;
      atomic_add_mod(dst + s, re, M.q, plain);
      atomic_add_mod(dst + n + s, im, M.q, plain);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 2 * cs);
}

__global__ void __launch_bounds__(CKU_THREADS, 1)
    ck_umma_kernel(const uint8_t* __restrict__ tk8, RowSet w, u32 rows, u32 G, u32 nck, u32 nkp, u32 n, u32 bt,
                   u32 Bw, const u64* thi, u32 nhi_t, ModQ M, const u64* zeta, u64* acc, bool plain) {
  pdl_wait();
  ck_umma_body(tk8, w, rows, G, nck, nkp, n, bt, Bw, thi, nhi_t, M, zeta, acc, rows, 0, plain, blockIdx.y);
}

// Several witnesses (uneven widths and row counts) against the same key rows
// in one launch: witness i owns the grid rows [ystart[i], ystart[i+1]) and
// its own accumulator acc[i] (nck x rows[i] ring elements).
struct CkMulti {
  RowSet w[CKU_MULTI_MAX];
  u64* acc[CKU_MULTI_MAX];
  u32 rows[CKU_MULTI_MAX], G[CKU_MULTI_MAX], Bw[CKU_MULTI_MAX];
  u32 ystart[CKU_MULTI_MAX + 1];
  uint8_t plain[CKU_MULTI_MAX];
  u32 count;
};

__global__ void __launch_bounds__(CKU_THREADS, 1)
    ck_umma_multi_kernel(const uint8_t* __restrict__ tk8, CkMulti m, u32 nck, u32 nkp, u32 n, u32 bt,
                         const u64* thi, u32 nhi_t, ModQ M, const u64* zeta) {
  pdl_wait();
  u32 i = 0;
  while (i + 1 < m.count && m.ystart[i + 1] <= blockIdx.y) i++;
  ck_umma_body(tk8, m.w[i], m.rows[i], m.G[i], nck, nkp, n, bt, m.Bw[i], thi, nhi_t, M, zeta, m.acc[i], m.rows[i],
               0, m.plain[i] != 0, blockIdx.y - m.ystart[i]);
}

}  // namespace

namespace salsaa {

int launch_ck_tk8(const u64* tlo, u32 nck, u32 n, u32 bt, bool packed, uint8_t* tk8, cudaStream_t st) {
  const u32 nkp = ck_tk8_nkp(nck);
  const u64 tot = (u64)bt * n * nkp;
  u64 g = (tot + 255) / 256;
  if (g > 65535 * 16) g = 65535 * 16;
  pdl(ck_tk8_kernel, (unsigned)g, 256, 0, st)(tlo, nck, n, bt, nkp, packed, tk8);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ck_tk8");
}

// The smallest shared-memory carveout (percent of the SM's 228 KiB) that
// holds one CTA's stages plus its static barriers: the rest stays L1, which
// holds the witness loads in flight (one 16-byte load per 32-byte sector).
static int ck_carveout(size_t smem) {
  const size_t need = smem + 2048;
  const size_t pct = (need * 100 + 228 * 1024 - 1) / (228 * 1024);
  return pct > 100 ? 100 : (int)pct;
}

// Dynamic shared memory for nck key rows: two stages, or the epilogue's sums over them.
static size_t cku_smem(u32 nck) {
  const size_t stage = 2 * (size_t)CKU_ATILE + 2 * (size_t)ck_tk8_nkp(nck) * CKU_CHUNK;
  const size_t epi = 2 * 128 * (size_t)(2 * nck) * sizeof(u64);
  return 2 * stage > epi ? 2 * stage : epi;
}
static const size_t CKU_MAX_SMEM = cku_smem(CKU_MAX_KEYS);

bool ck_umma_ok(const CommitArgs& a, u32 n) {
  if (!a.tk8 || a.rows == 0 || a.rows > CKU_MAX_WROWS || a.nck == 0 || a.nck > CKU_MAX_KEYS || (n & 1)) return false;
  if (a.width < CKU_CHUNK || a.ck_bt < CKU_CHUNK) return false;
  for (u32 k = 0; k < a.rows; k++)
    if ((uintptr_t)a.w.p[k] % 16) return false;
  return true;
}

void ck_umma_shape(u64 width, u32 rows, u32 n, u32 ck_bt, u32* Bk_out, u32* G_out) {
  // element block per CTA: a whole key-table block (one epilogue per block),
  // halved while the grid would not fill the GPU
  u32 Bk = (u32)(width < ck_bt ? width : ck_bt);
  while (Bk > CK_BLOCK && (u64)(n / 2) * (width / Bk) < 296) Bk /= 2;
  // few witness rows: G blocks one key block apart per CTA share the key
  // tiles (virtual rows g * rows + k), while the grid keeps a full wave
  u32 G = 1;
  while (width >= ck_bt && rows * G * 2 <= CKU_MAX_WROWS && (width / ck_bt) % (G * 2) == 0 &&
         (u64)(n / 2) * (width / Bk) / (G * 2) >= 148)
    G *= 2;
  *Bk_out = Bk;
  *G_out = G;
}

int launch_ck_umma_multi(const CommitArgs* a, u32 ninst, u32 n, const ModQ& M, const u64* zeta, cudaStream_t st) {
  if (ninst == 0 || ninst > CKU_MULTI_MAX) return salsaa_set_error(-2, "ck_umma_multi: 1..8 witnesses per launch");
  CkMulti m{};
  u32 y = 0;
  double wit_bytes = 0, out_bytes = 0, ops = 0, macs = 0;
  for (u32 i = 0; i < ninst; i++) {
    const CommitArgs& c = a[i];
    if (!ck_umma_ok(c, n) || c.nck != a[0].nck || c.tk8 != a[0].tk8)
      return salsaa_set_error(-2, "ck_umma_multi: a witness does not fit the tensor-core key-row product");
    u32 Bk, G;
    ck_umma_shape(c.width, c.rows, n, c.ck_bt, &Bk, &G);
    if (c.rows * G > CKU_MAX_WROWS || c.ck_bt % Bk || c.width % ((u64)Bk * G))
      return salsaa_set_error(-2, "ck_umma_multi: bad block grouping");
    u64 CH = c.width / 512;
    if (CH < 128) CH = 128;
    if (CH > Bk) CH = Bk;
    m.w[i] = c.w;
    m.rows[i] = c.rows;
    m.G[i] = G;
    m.Bw[i] = Bk;
    m.acc[i] = c.acc;
    m.plain[i] = (M.q < (1ULL << 50) && (c.width / CH) < (1ULL << 13)) ? 1 : 0;
    m.ystart[i] = y;
    y += (u32)(c.width / Bk / G);
    wit_bytes += 8.0 * c.rows * (double)c.width * 2 * n;
    out_bytes += 8.0 * c.nck * c.rows * 2 * n;
    ops += 2.0 * 196.0 * c.nck * c.rows * (double)c.width * n;
    macs += (double)c.nck * c.rows * (double)c.width * 2 * n;
  }
  m.ystart[ninst] = y;
  m.count = ninst;
  const u32 nck = a[0].nck, nkp = ck_tk8_nkp(nck);
  const size_t smem = cku_smem(nck);
  cudaError_t e = smem_limit(ck_umma_multi_kernel, CKU_MAX_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ck_umma_multi_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, ck_carveout(smem));
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "ck_umma_multi smem attribute");
  const int tr = salsaa_trace_begin("ck_umma_kernel", st, wit_bytes + out_bytes);
  salsaa_trace_alias(tr, "ck_umma_kernel:int8", ops);
  salsaa_trace_alias(tr, "ck_umma_kernel:mac", macs);
  pdl(ck_umma_multi_kernel, dim3(n / 2, y), CKU_THREADS, smem, st)(a[0].tk8, m, nck, nkp, n, a[0].ck_bt, a[0].thi,
                                                                   a[0].ck_nhi, M, zeta);
  salsaa_trace_end(tr, st);
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ck_umma_multi launch");
}

int launch_ck_umma(const CommitArgs& a, u32 n, u32 Bw, u32 G, const ModQ& M, const u64* zeta, bool plain,
                   cudaStream_t st) {
  if (G == 0 || a.rows * G > CKU_MAX_WROWS || (G > 1 && (a.width < a.ck_bt || (a.width / a.ck_bt) % G)) ||
      a.ck_bt % Bw || a.width % ((u64)Bw * G))
    return salsaa_set_error(-2, "ck_umma: bad block grouping");
  const u32 nkp = ck_tk8_nkp(a.nck);
  const size_t smem = cku_smem(a.nck);
  cudaError_t e = smem_limit(ck_umma_kernel, CKU_MAX_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ck_umma_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, ck_carveout(smem));
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "ck_umma smem attribute");
  dim3 g(n / 2, (unsigned)(a.width / Bw / G));
  // Traced measures of one launch: algorithmic HBM bytes (the slot-form
  // witness read once, the accumulators written once), the int8 operations
  // the tensor cores execute (2 x 14 x 14 byte products per key row, witness
  // row, element and slot pair half), and the exact mod-q multiply-accumulates
  // of the ring products (2d per key row, witness row and element).
  const double wit_bytes = 8.0 * a.rows * (double)a.width * 2 * n;
  const double out_bytes = 8.0 * a.nck * a.rows * 2 * n;
  const int tr = salsaa_trace_begin("ck_umma_kernel", st, wit_bytes + out_bytes);
  salsaa_trace_alias(tr, "ck_umma_kernel:int8", 2.0 * 196.0 * a.nck * a.rows * (double)a.width * n);
  salsaa_trace_alias(tr, "ck_umma_kernel:mac", (double)a.nck * a.rows * (double)a.width * 2 * n);
  pdl(ck_umma_kernel, g, CKU_THREADS, smem, st)(a.tk8, a.w, a.rows, G, a.nck, nkp, n, a.ck_bt, Bw, a.thi, a.ck_nhi,
                                               M, zeta, a.acc, plain);
  salsaa_trace_end(tr, st);
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ck_umma launch");
}

// ---------------------------------------------------------------------------
// Projection on tcgen05 (project, src/subroutines/project.rs:50-103): per
// chunk of cw witness elements, out[256 x d] = J (256 x cw, entries -1/0/1) x
// W (cw x d, centre-lifted, int8).  CTA = (chunk, block of 128 coefficient
// positions); per 64-element step thread 0 bulk-copies the 256 rows of
// J from their canonical image (Jc, see launch_proj_tables) and issues
// 2 x 4 MMAs (kind::i8, signed x signed, M = 128 J rows, N = 128 positions,
// K = 32) into two TMEM accumulators; the threads convert the witness step to
// int8 in the canonical layout.  A value outside [-128, 127] sets the flag and
// the exact CUDA-core kernel recomputes every output (same as the mma.sync
// path).  Two stages: the witness of step c + 1 is staged while the MMAs of
// step c run.
// ---------------------------------------------------------------------------
constexpr u32 PU_POS = 128, PU_KS = 64;
constexpr u32 PU_A = 2 * 128 * PU_KS;  // both J halves of one step (16 KiB)
constexpr u32 PU_B = PU_POS * PU_KS;   // witness int8 tile (8 KiB)
constexpr u32 PU_STAGE = PU_A + PU_B;

__global__ void __launch_bounds__(256, 2)
    project_umma_kernel(RowSet in, u32 d, u64 q, u32 cw, u64 nch, const int8_t* __restrict__ Jc,
                        u64* __restrict__ out, u64* flag, const u32* gate) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[2], done_bar[2];
  __shared__ uint32_t tslot;
  if (gate && *(volatile const u32*)gate == 0) return;  // the byte rows were projected
  const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const u32 nblk = blockIdx.x;
  const u64 idx = blockIdx.y;
  const u32 i = (u32)(idx / nch);
  const u64 j = idx % nch;
  const bool nar = (in.narrow >> i) & 1;
  const u64* chunk = row_advance(in.p[i], nar, (j * cw) * d + (u64)nblk * PU_POS);
  const u64 half_q = q >> 1;
  const u32 nsteps = cw / PU_KS;
  u32* err = &g_tc_error;
  if (tid == 0) {
    for (int b = 0; b < 2; b++) {
      umma::mbar_init(&full_bar[b], 1);
      umma::mbar_init(&done_bar[b], 1);
    }
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;
  // signed int8 x signed int8 -> s32, M = N = 128
  const u32 idesc = umma::idesc_u8(128, PU_POS) | (1u << 7) | (1u << 10);
  bool bad = false, ok = true;
  // task of this thread: 16 consecutive elements x 2 neighbouring positions,
  // one 16-byte load per element for word rows (two u64 values) and one
  // 8-byte load for narrow rows (two int32 values, kept in wv[e].x); a
  // step's values stay in registers from their loads (issued before the
  // previous step's barrier) to their conversion
  ulonglong2 wv[16];
  const u32 nkq = tid >> 6, np2 = tid & 63;
  auto load = [&](u32 c) {
    if (nar) {
      const int* src = (const int*)chunk + (u64)c * PU_KS * d;
#pragma unroll
      for (u32 e = 0; e < 16; e++)
        wv[e].x = (u64)__ldg((const long long*)(src + (u64)(16 * nkq + e) * d + 2 * np2));
    } else {
      const u64* src = chunk + (u64)c * PU_KS * d;
#pragma unroll
      for (u32 e = 0; e < 16; e++) wv[e] = __ldg((const ulonglong2*)(src + (u64)(16 * nkq + e) * d + 2 * np2));
    }
  };
  load(0);
  for (u32 c = 0; c < nsteps; c++) {
    const u32 st = c & 1;
    uint8_t* stage = smem + st * PU_STAGE;
    if (c >= 2) ok &= umma::mbar_wait(&done_bar[st], ((c - 2) >> 1) & 1, err, 1);
    if (tid == 0) {  // K slices of this step from the image
      umma::mbar_expect_tx(&full_bar[st], PU_A);
      umma::bulk_g2s(stage, Jc + (u64)c * PU_A, PU_A, &full_bar[st]);
    }
    // witness step: 128 positions x 64 elements as int8, (k / 16, pos, k % 16):
    // the 16 bytes of one position are one 16-byte store
    uint8_t* B = stage + PU_A;
#pragma unroll
    for (u32 p = 0; p < 2; p++) {
      u32 w4[4];
#pragma unroll
      for (u32 g = 0; g < 4; g++) {
        u32 tq[4];  // centred value + 128: below 256 iff it fits int8
#pragma unroll
        for (u32 e = 0; e < 4; e++) {
          const ulonglong2 v2 = wv[4 * g + e];
          if (nar) {
            const int cv = (int)(u32)(p ? (v2.x >> 32) : v2.x);
            bad |= (cv > 127) | (cv < -128);
            tq[e] = (u32)cv + 128u;
          } else {
            const u64 v = p ? v2.y : v2.x;
            const long long cv = v > half_q ? (long long)v - (long long)q : (long long)v;
            const unsigned long long tb = (unsigned long long)(cv + 128);
            bad |= tb > 255ULL;
            tq[e] = (u32)tb;
          }
        }
        // low bytes of the four values, e in byte e
        const u32 packed =
            __byte_perm(__byte_perm(tq[0], tq[1], 0x0040), __byte_perm(tq[2], tq[3], 0x0040), 0x5410);
        w4[g] = packed ^ 0x80808080u;
      }
      *(uint4*)(B + nkq * (PU_POS * 16) + (2 * np2 + p) * 16) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
    }
    if (c + 1 < nsteps) load(c + 1);
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
      umma::fence_after_sync();
      ok &= umma::mbar_wait(&full_bar[st], (c >> 1) & 1, err, 2);
#pragma unroll
      for (u32 h = 0; h < 2; h++)
#pragma unroll
        for (u32 ks = 0; ks < PU_KS / 32; ks++) {
          const uint64_t ad =
              umma::desc_kmajor(umma::smem_u32(stage + h * 128 * 16 + ks * 2 * 256 * 16), 256 * 16, 128);
          const uint64_t bd = umma::desc_kmajor(umma::smem_u32(B + ks * 2 * PU_POS * 16), PU_POS * 16, 128);
          umma::mma_i8(tmem + h * 128, ad, bd, idesc, (c > 0 || ks > 0) ? 1u : 0u);
        }
      umma::commit(&done_bar[st]);
    }
  }
  ok &= umma::mbar_wait(&done_bar[(nsteps - 1) & 1], ((nsteps - 1) >> 1) & 1, err, 3);
  ok = __syncthreads_and(ok);
  if (bad) atomicOr((unsigned long long*)flag, 1ULL);
  umma::fence_after_sync();
  if (ok) {
    const u32 h = warp >> 2, row = (warp & 3) * 32 + lane;
    u64* dst = out + ((idx * 256) + h * 128 + row) * d + (u64)nblk * PU_POS;
    for (u32 cb = 0; cb < PU_POS; cb += 16) {
      uint32_t r[16];
      umma::tmem_ld16(tmem + (((warp & 3) * 32) << 16) + h * 128 + cb, r);
      umma::tmem_wait_ld();
#pragma unroll
      for (u32 e = 0; e < 16; e += 2) {
        const int v0 = (int)r[e], v1 = (int)r[e + 1];
        const u64 a = v0 >= 0 ? (u64)v0 : q - (u64)(-(long long)v0);
        const u64 b = v1 >= 0 ? (u64)v1 : q - (u64)(-(long long)v1);
        *(ulonglong2*)(dst + cb + e) = make_ulonglong2(a, b);
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

int launch_project_umma(RowSet in, u32 rows, u64 nch, u32 d, u64 q, u32 cw, const int8_t* Jc, u64* out, u64* flag,
                        const u32* gate, cudaStream_t st) {
  const size_t smem = 2 * (size_t)PU_STAGE;
  cudaError_t e = cudaFuncSetAttribute(project_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "project_umma smem attribute");
  dim3 g(d / PU_POS, (unsigned)(rows * nch));
  pdl(project_umma_kernel, g, 256, smem, st)(in, d, q, cw, nch, Jc, out, flag, gate);
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "project_umma launch");
}

// ---------------------------------------------------------------------------
// TENSOR statement rows on tcgen05 (the scalar rows of
// parallel_dot_series_matrix, src/arithmetic.rs:459-505, whose weights are
// s(i) = s_hi[i / Bw] s_lo[i % Bw]), over the coefficient-form witness.
// For one witness row k, one block of Bw elements (one s_hi factor) and 128
// coefficient positions, sum_i s_lo(i) w(i) is an integer matrix product:
//   A (M = 128): rows (tensor row r, byte x) of s_lo, unsigned bytes,
//   B (N = 128): coefficient positions, the centred witness split into three
//     signed byte limbs (exact for |w| < 2^23), one MMA chain per limb,
//   D_l[(r,x)][pos] = sum_i byte_x(s_lo(i)) limb_l(w(i, pos)),
// and the row sum is sum_{x,l} 2^(8(x+l)) D_l mod q.  A work item that meets a
// larger value is redone exactly on CUDA cores.  The sums land in the coefficient-
// form accumulators that launch_commit moves to slot form.
// ---------------------------------------------------------------------------
constexpr u32 SU_POS = 128, SU_KS = 128, SU_LIMBS = 3;
constexpr u32 SU_A = 128 * SU_KS;                   // scalar byte tile (16 KiB)
constexpr u32 SU_B = SU_POS * SU_KS;                // one limb tile (16 KiB)
constexpr u32 SU_STAGE = SU_A + SU_LIMBS * SU_B;    // 64 KiB

__global__ void sc_img_kernel(const u64* s_lo, u32 Bw, ScRange rg, uint8_t* img) {
  pdl_wait();
  const u32 tot = Bw * 128 * rg.groups();  // (group, chunk, slice, row, byte) = groups x Bw / 128 x 8 x 128 x 16
  for (u32 t = blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += gridDim.x * blockDim.x) {
    const u32 b = t % 16, row = t / 16 % 128, sl = t / 2048 % 8, cc = t / 16384 % (Bw / 128), g = t / (Bw * 128);
    uint8_t v = 0;
    if (row < rg.rows(g) * 8 && row % 8 < 7) {
      const u32 r = row / 8, x = row % 8;
      v = (uint8_t)(s_lo[(u64)(rg.first(g) + r) * Bw + cc * 128 + sl * 16 + b] >> (8 * x));
    }
    img[t] = v;
  }
}

__global__ void __launch_bounds__(512, 1)
    sc_umma_kernel(RowSet wc, u32 rows, u32 d, u32 Bw, u32 nhi, u32 split, ScRange rg,
                   const uint8_t* __restrict__ img0, const u64* s_lo, const u64* s_hi, ModQ M, u64* acc, bool plain,
                   ScGates gates) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[2], done_bar[2];
  __shared__ uint32_t tslot;
  const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (gates.all_closed()) return;
  const u64 q = M.q, half_q = q >> 1;
  const u32 nsteps = Bw / SU_KS / split;
  u32* err = &g_tc_error;
  if (tid == 0) {
    for (int b = 0; b < 2; b++) {
      umma::mbar_init(&full_bar[b], 1);
      umma::mbar_init(&done_bar[b], 1);
    }
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;
  // unsigned bytes (A) x signed bytes (B) -> s32, M = N = 128
  const u32 idesc = umma::idesc_u8(128, SU_POS) | (1u << 10);
  bool ok = true;
  // work items: positions pb, element block hb (one s_hi factor), its part sub
  // of split, witness row k and group grp of scalar rows; g0 counts the steps
  // of earlier items
  const u32 npb = d / SU_POS, per = npb * nhi * split * rows, items = per * rg.groups();
  u32 g0 = 0;
  for (u32 item = blockIdx.x; item < items; item += gridDim.x) {
    const u32 pb = item % npb, hs = item / npb % (nhi * split), k = item / (npb * nhi * split) % rows;
    const u32 grp = item / per, nrow = rg.rows(grp), j0 = rg.first(grp);
    const u32 hb = hs / split, sub = hs % split;
    if (!gates.open(k)) continue;
    const u32 c0 = sub * nsteps;
    const bool nar = (wc.narrow >> k) & 1;
    const u64* src0 = row_advance(wc.p[k], nar, ((u64)hb * Bw + (u64)c0 * SU_KS) * d + (u64)pb * SU_POS);
    const uint8_t* img = img0 + (u64)grp * Bw * 128 + (u64)c0 * SU_A;
    bool bad = false;
    // task of this thread: 16 consecutive elements x 2 neighbouring positions,
    // one 16-byte load per element for word rows (two u64 values) and one
    // 8-byte load for narrow rows (two int32 values, kept in wv[e].x); one
    // 16-byte store per limb plane and position
    ulonglong2 wv[16];
    const u32 nkq = tid >> 6, np2 = tid & 63;
    auto load = [&](u32 c) {
      if (nar) {
        const int* src = (const int*)src0 + (u64)c * SU_KS * d;
#pragma unroll
        for (u32 e = 0; e < 16; e++)
          wv[e].x = (u64)__ldg((const long long*)(src + (u64)(16 * nkq + e) * d + 2 * np2));
      } else {
        const u64* src = src0 + (u64)c * SU_KS * d;
#pragma unroll
        for (u32 e = 0; e < 16; e++) wv[e] = __ldg((const ulonglong2*)(src + (u64)(16 * nkq + e) * d + 2 * np2));
      }
    };
    load(0);
    for (u32 c = 0; c < nsteps; c++) {
      const u32 g = g0 + c, st = g & 1;
      uint8_t* stage = smem + st * SU_STAGE;
      if (g >= 2) ok &= umma::mbar_wait(&done_bar[st], ((g - 2) >> 1) & 1, err, 1);
      if (tid == 0) {
        umma::mbar_expect_tx(&full_bar[st], SU_A);
        umma::bulk_g2s(stage, img + (u64)c * SU_A, SU_A, &full_bar[st]);
      }
#pragma unroll
      for (u32 p = 0; p < 2; p++) {
        u32 l0[4], l1[4], l2[4];
#pragma unroll
        for (u32 g = 0; g < 4; g++) {
          u32 wq[4];
#pragma unroll
          for (u32 e = 0; e < 4; e++) {
            const ulonglong2 v2 = wv[4 * g + e];
            // centred value + 0x808080: its bytes are the signed limbs + 128 when
            // the value lies in [-0x808080, 0x7f7f7f] (three balanced base-256 digits)
            if (nar) {
              const int v = (int)(u32)(p ? (v2.x >> 32) : v2.x);
              bad |= (v > 0x7f7f7f) | (v < -0x808080);  // the value needs a fourth limb
              wq[e] = ((u32)v + 0x808080u) ^ 0x808080u;
            } else {
              const u64 v = p ? v2.y : v2.x;
              const u64 tb = v + 0x808080ULL - (v > half_q ? q : 0);
              bad |= (tb >> 24) != 0;
              wq[e] = (u32)tb ^ 0x808080u;
            }
          }
          // limb planes of the four values: byte l of wq[0..3]
          const u32 lo01 = __byte_perm(wq[0], wq[1], 0x5140), lo23 = __byte_perm(wq[2], wq[3], 0x5140);
          const u32 hi01 = __byte_perm(wq[0], wq[1], 0x0062), hi23 = __byte_perm(wq[2], wq[3], 0x0062);
          l0[g] = __byte_perm(lo01, lo23, 0x5410);
          l1[g] = __byte_perm(lo01, lo23, 0x7632);
          l2[g] = __byte_perm(hi01, hi23, 0x5410);
        }
        const u32 off = SU_A + nkq * (SU_POS * 16) + (2 * np2 + p) * 16;
        *(uint4*)(stage + off) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
        *(uint4*)(stage + off + SU_B) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
        *(uint4*)(stage + off + 2 * SU_B) = make_uint4(l2[0], l2[1], l2[2], l2[3]);
      }
      if (c + 1 < nsteps) load(c + 1);
      umma::fence_proxy_async();
      umma::fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        umma::fence_after_sync();
        ok &= umma::mbar_wait(&full_bar[st], (g >> 1) & 1, err, 2);
#pragma unroll
        for (u32 l = 0; l < SU_LIMBS; l++)
#pragma unroll
          for (u32 ks = 0; ks < SU_KS / 32; ks++) {
            const uint64_t ad = umma::desc_kmajor(umma::smem_u32(stage + ks * 2 * 128 * 16), 128 * 16, 128);
            const uint64_t bd =
                umma::desc_kmajor(umma::smem_u32(stage + SU_A + l * SU_B + ks * 2 * SU_POS * 16), SU_POS * 16, 128);
            umma::mma_i8(tmem + l * 128, ad, bd, idesc, (c > 0 || ks > 0) ? 1u : 0u);
          }
        umma::commit(&done_bar[st]);
      }
    }
    const u32 gl = g0 + nsteps - 1;
    ok &= umma::mbar_wait(&done_bar[gl & 1], (gl >> 1) & 1, err, 3);
    ok = __syncthreads_and(ok);
    bad = __syncthreads_or(bad);
    umma::fence_after_sync();
    g0 += nsteps;
    if (ok && !bad) {
      // per TMEM lane (row (r, x)), per position: sum_l 2^(8l) D_l, reduced, times 2^(8x)
      u64* Pm = (u64*)smem;  // 128 rows x 128 positions
      const u32 row = (warp & 3) * 32 + lane, quarter = warp >> 2;  // four groups of 32 positions
      const u32 x = row % 8;  // column 7 of a row's eight is zero
      const u64 pw = ((u64)1 << (8 * x)) % q;
      const u64 cpos = ((((u64)1 << 62) / q) + 1) * q;
      for (u32 cb = quarter * 32; cb < quarter * 32 + 32; cb += 16) {
        uint32_t r0[16], r1[16], r2[16];
        const u32 base = tmem + (((warp & 3) * 32) << 16) + cb;
        umma::tmem_ld16(base, r0);
        umma::tmem_ld16(base + 128, r1);
        umma::tmem_ld16(base + 256, r2);
        umma::tmem_wait_ld();
#pragma unroll
        for (u32 e = 0; e < 16; e++) {
          const long long v = (long long)(int)r0[e] + ((long long)(int)r1[e] << 8) + ((long long)(int)r2[e] << 16);
          const u64 red = reduce64(M, v < 0 ? (u64)(v + (long long)cpos) : (u64)v);
          Pm[(u64)row * 128 + cb + e] = mul_mod(M, red, pw);
        }
      }
    }
    __syncthreads();
    if (ok && !bad) {
      const u64* Pm = (const u64*)smem;
      for (u32 t = tid; t < nrow * SU_POS; t += 512) {
        const u32 r = t / SU_POS, pos = t % SU_POS;
        u64 v = 0;
#pragma unroll
        for (u32 x = 0; x < 7; x++) v = salsaa::add_mod(v, Pm[(u64)(r * 8 + x) * 128 + pos], q);
        const u32 j = j0 + r;
        v = mul_mod(M, v, s_hi[(u64)j * nhi + hb]);
        atomic_add_mod(acc + ((u64)j * rows + k) * d + (u64)pb * SU_POS + pos, v, q, plain);
      }
    }
    if (ok && bad) {  // exact CUDA-core sums of this item
      for (u32 t = tid; t < nrow * SU_POS; t += 512) {
        const u32 r = t / SU_POS, pos = t % SU_POS, j = j0 + r;
        u64 v = 0;
        for (u32 i = 0; i < nsteps * SU_KS; i++)
          v = salsaa::add_mod(v, mul_mod(M, s_lo[(u64)j * Bw + c0 * SU_KS + i], wres(src0, nar, (u64)i * d + pos, q)), q);
        v = mul_mod(M, v, s_hi[(u64)j * nhi + hb]);
        atomic_add_mod(acc + ((u64)j * rows + k) * d + (u64)pb * SU_POS + pos, v, q, plain);
      }
    }
    // the next item's copies and MMAs reuse the stages and TMEM read above
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (!ok) break;
  }
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

int launch_sc_img(const u64* s_lo, u32 Bw, const ScRange& rg, uint8_t* img, cudaStream_t st) {
  const u64 g = ((u64)Bw * 128 * rg.groups() + 255) / 256;
  pdl(sc_img_kernel, (unsigned)(g < 4096 ? g : 4096), 256, 0, st)(s_lo, Bw, rg, img);
  salsaa_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "sc_img launch");
}

int launch_sc_umma(const RowSet& wc, u32 rows, u32 d, u32 Bw, u32 nhi, const ScRange& rg, const u64* s_lo,
                   const u64* s_hi, const ModQ& M, u64* acc, bool plain, const uint8_t* img, const ScGates& gates,
                   cudaStream_t st) {
  // short witnesses: split each element block over several CTAs (linear sums)
  // while the items stay within one wave (one CTA per SM)
  const u64 base = (u64)(d / SU_POS) * nhi * rows;
  u32 split = 1;
  while (split * 2 <= Bw / SU_KS && base * split * 2 <= 148) split *= 2;
  const u64 items = base * split * rg.groups();
  const size_t smem = 2 * (size_t)SU_STAGE;
  cudaError_t e = cudaFuncSetAttribute(sc_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "sc_umma smem attribute");
  pdl(sc_umma_kernel, (unsigned)(items < 148 ? items : 148), 512, smem, st)(wc, rows, d, Bw, nhi, split, rg, img, s_lo,
                                                                           s_hi, M, acc, plain, gates);
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "sc_umma launch");
}

// Looked up on each call: the address belongs to the current context, and a
// device reset or another context of the device has another.
u32* tc_error_word() {
  void* v = nullptr;
  return cudaGetSymbolAddress(&v, g_tc_error) == cudaSuccess ? (u32*)v : nullptr;
}

int tc_error_check() {
  u32 h = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&h, g_tc_error, sizeof(u32));
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "tensor-core status");
  if (h) return salsaa_set_error(-4, "a tensor-core wait timed out; results of that launch are invalid");
  return ntt_error_check();
}

}  // namespace salsaa

extern "C" int salsaa_selftest_umma_i8(const uint8_t* d_a, const uint8_t* d_b, uint32_t n, uint32_t k,
                                       int32_t* d_out, void* stream) {
  if (!d_a || !d_b || !d_out) return salsaa_set_error(-1, "selftest_umma_i8: null argument");
  if (n < 16 || n > 256 || n % 16 || k == 0 || k > 256 || k % 32)
    return salsaa_set_error(-1, "selftest_umma_i8: needs 16 <= n <= 256 (multiple of 16), k multiple of 32 <= 256");
  cudaStream_t st = (cudaStream_t)stream;
  u32* err = nullptr;
  cudaError_t e = cudaMallocAsync(&err, sizeof(u32), st);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "selftest_umma_i8: alloc");
  cudaMemsetAsync(err, 0, sizeof(u32), st);
  const size_t smem = (size_t)(128 + n) * k;
  e = cudaFuncSetAttribute(umma_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) {
    pdl(umma_selftest_kernel, 1, 128, smem, st)(d_a, d_b, n, k, d_out, err);
    salsaa_count_launch();
    e = cudaGetLastError();
  }
  u32 h = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, err, sizeof(u32), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFreeAsync(err, st);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "selftest_umma_i8");
  if (h) return salsaa_set_error(-4, "selftest_umma_i8: tensor-core wait timed out");
  return 0;
}
