// ck_img.cu — commitment-key rows on tcgen05 over byte images of the
// slot-form witness (ntt_img.cuh), q < 2^50.
#include <cuda_runtime.h>

#include "ntt_img.cuh"
#include "umma.cuh"

namespace salsaa {

namespace {

// The product is ck_umma_kernel's: per NTT slot, D[(v, half, y)][(r, comp, x)]
// = sum_lo byte_y(w) byte_x(T) accumulates exactly in TMEM, and
// value = sum_{x, y} 2^(8 (x + y)) D mod q.  Here both operands arrive in
// their shared-memory layout, so the kernel is bulk copies and MMAs.
//
// A tile is (slot s, Bw elements of a key block, E groups of G key blocks);
// its E accumulators (nkp TMEM columns each) share every key tile.
// Persistent CTAs, one per SM (they own its TMEM): warp 8 copies 64-element
// chunks into a ring of stages, warp 9 issues the MMAs, warps 0 .. 7 turn
// finished accumulators into residues.  What bounds it is the L2 -> shared
// memory traffic of the chunks (19 KB per chunk and accumulator at 9 witness
// and 12 key rows: 12.6 TB/s, and 6.2 from DRAM, at 9 rows x 2^16; 7.5 and 4.7
// at 3 rows x 2^17, whose accumulators share key tiles) and, for short
// witnesses, reading the key table once (92 MB at 12 key rows); the tensor
// pipe is busy 41 .. 42% of the time.  With 2 E nkp <= 512 columns the accumulators are
// double-buffered, so the epilogue runs beside the next tile's MMAs.
//
// Epilogue: a thread folds the 7 key bytes x of its TMEM lane's sums into a
// 54-bit and a 46-bit part, by shifts and without reduction, and gives TMEM
// back; a second pass sums the 7 byte rows y as one 128-bit integer (below
// 2^126) per (virtual row, half, key row, component) and reduces once, four
// lanes per (key row, row).  Its table constants are loaded before it waits
// for the MMAs: a dependent global load takes microseconds under the copies.
//
// One A0 proof's eight launches (B200, summed): 1932 us in ck_umma_kernel,
// which split words into bytes itself, 590 here.  Round 0 (3 rows x 2^18): 439
// -> 167 us, round 1 (9 x 2^17): 593 -> 197 us.
//
// Every wait is bounded; a role that gives up stops, and the others then
// give up on the arrivals it no longer makes.
constexpr u32 CKI_EPI = 256, CKI_THREADS = CKI_EPI + 64;
constexpr u32 CKI_MAX_STAGES = 8;

struct CkImgTiles {
  u32 E, NB;          // accumulators per tile (the kernel's E), TMEM buffers of E accumulators
  u32 Bw, lob, nE;    // elements per tile, tiles per key block, groups of E hg values
  u32 ntiles, nst;
  u32 a_bytes, b_bytes, stage_bytes;  // per accumulator, key tile, whole stage
};

__device__ __forceinline__ void bar_epi() { asm volatile("bar.sync 1, %0;" ::"r"(CKI_EPI) : "memory"); }

__device__ __forceinline__ bool bar_epi_and(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}\n"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(CKI_EPI)
      : "memory");
  return r != 0;
}

// 128-bit accumulation of v << sh (sh < 128 - 64 + 1, the sums stay below 2^128)
__device__ __forceinline__ void add_shifted(u64& hi, u64& lo, u64 v, u32 sh) {
  u64 l, h;
  if (sh == 0) {
    l = v;
    h = 0;
  } else if (sh < 64) {
    l = v << sh;
    h = v >> (64 - sh);
  } else {
    l = 0;
    h = v << (sh - 64);
  }
  lo += l;
  hi += h + (lo < l);
}

// Key-row pairs m (28 TMEM columns from 28 m): the four (key row, component)
// groups of 7 key bytes, folded to (x = 0 .. 3, x = 4 .. 6) parts.  M4 = m % 4
// fixes the columns' offset in their 16-column chunks.
template <u32 M4>
__device__ __forceinline__ void fold_pair(u32 tb, u32 m, u32 nkp, ulonglong2 (&f)[4]) {
  constexpr u32 OFF = 28 * M4 % 16, NCH = (OFF + 28 + 15) / 16;
  const u32 cb = (28 * m - OFF) / 16;
  uint32_t r[NCH][16];
#pragma unroll
  for (u32 c = 0; c < NCH; c++) {
    if ((cb + c) * 16 < nkp) {
      umma::tmem_ld16(tb + (cb + c) * 16, r[c]);
    } else {
#pragma unroll
      for (u32 i = 0; i < 16; i++) r[c][i] = 0;
    }
  }
  umma::tmem_wait_ld();
#pragma unroll
  for (u32 g = 0; g < 4; g++) {
    u64 lo = 0, hi = 0;
#pragma unroll
    for (u32 x = 0; x < 7; x++) {
      const u32 col = OFF + 7 * g + x;
      const u64 v = r[col / 16][col % 16];
      if (x < 4) lo += v << (8 * x);
      else hi += v << (8 * (x - 4));
    }
    f[g] = make_ulonglong2(lo, hi);
  }
}
// PAIRS pairs per epilogue warp, the two warps of a TMEM lane taking alternate ones.
template <u32 PAIRS>
__device__ __forceinline__ void fold_pairs(u32 tb, u32 ch, u32 npair, u32 nkp, ulonglong2 (&f)[PAIRS][4]) {
#pragma unroll
  for (u32 i = 0; i < PAIRS; i++) {
    const u32 m = 2 * i + ch;
    if (m < npair) {
      if (ch == 0) {
        if (i % 2 == 0) fold_pair<0>(tb, m, nkp, f[i]);
        else fold_pair<2>(tb, m, nkp, f[i]);
      } else {
        if (i % 2 == 0) fold_pair<1>(tb, m, nkp, f[i]);
        else fold_pair<3>(tb, m, nkp, f[i]);
      }
    }
  }
}

// E accumulators per tile; PAIRS >= a quarter of the key rows.
template <u32 E, u32 PAIRS>
__global__ void __launch_bounds__(CKI_THREADS, 1)
    ck_img_kernel(const uint8_t* __restrict__ tk8, CkImage im, CkImgTiles t, u32 nck, u32 nkp, u32 nkc,
                  const u64* thi, u32 nhi_t, ModQ M, const u64* zeta, u64* acc, bool plain, u32* err) {
  pdl_wait();
  // finishing tasks per thread: 4 lanes per (virtual row, key row)
  constexpr u32 NIT = (CKI_MAX_V * 4 * PAIRS * 4 + CKI_EPI - 1) / CKI_EPI;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[CKI_MAX_STAGES], empty_bar[CKI_MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tslot;
  const u32 tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const u32 n = im.n, d = 2 * n, V = im.R * im.G;
  const u32 nchunks = t.Bw / CKI_CHUNK;
  // stages, then the epilogue's partial sums
  ulonglong2* Pm = (ulonglong2*)(smem + (size_t)t.nst * t.stage_bytes);
  if (tid == 0) {
    for (u32 i = 0; i < t.nst; i++) {
      umma::mbar_init(&full_bar[i], 1);
      umma::mbar_init(&empty_bar[i], 1);
    }
    for (u32 i = 0; i < 2; i++) {
      umma::mbar_init(&acc_full[i], 1);
      umma::mbar_init(&acc_empty[i], CKI_EPI);
    }
    umma::mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc(&tslot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const u32 tmem = tslot;

  if (warp == CKI_EPI / 32) {
    bool ok = true;
    u32 it = 0, st = 0, par = 1;  // chunk counter over all tiles, its stage, parity of the stage's previous use
    const u64 astep = (u64)n * t.a_bytes, bstep = (u64)n * t.b_bytes;
    for (u32 tile = blockIdx.x; ok && tile < t.ntiles; tile += gridDim.x) {
      const u32 he = tile % t.nE, rest = tile / t.nE, lb = rest % t.lob, s = rest / t.lob;
      const u32 c0 = lb * nchunks;
      const uint8_t* pa = im.p + (((u64)he * E * im.nlc + c0) * n + s) * t.a_bytes;
      const uint8_t* pb = tk8 + ((u64)c0 * n + s) * t.b_bytes;
      const u64 estep = (u64)im.nlc * astep;
      for (u32 c = 0; c < nchunks; c++, it++, pa += astep, pb += bstep) {
        if (it >= t.nst && !(ok = umma::mbar_wait(&empty_bar[st], par, err, 11))) break;
        if (umma::elect_one()) {
          uint8_t* stage = smem + st * t.stage_bytes;
          umma::mbar_expect_tx(&full_bar[st], E * t.a_bytes + t.b_bytes);
          umma::bulk_g2s(stage, pa, t.a_bytes, &full_bar[st]);
          if (E == 2) umma::bulk_g2s(stage + t.a_bytes, pa + estep, t.a_bytes, &full_bar[st]);
          umma::bulk_g2s(stage + E * t.a_bytes, pb, t.b_bytes, &full_bar[st]);
        }
        __syncwarp();
        if (++st == t.nst) {
          st = 0;
          par ^= 1;
        }
      }
    }
    // copies still in flight land before the CTA ends
    for (u32 c = it >= t.nst ? it - t.nst : 0; c < it; c++)
      umma::mbar_wait(&full_bar[c % t.nst], (c / t.nst) & 1, err, 12);
  } else if (warp == CKI_EPI / 32 + 1) {
    const u32 idesc = umma::idesc_u8(128, nkp), lbo = im.VP * 16;
    // descriptors of stage 0; a stage, an accumulator and a K step are constant address steps
    const uint64_t ad0 = umma::desc_kmajor(umma::smem_u32(smem), lbo, 128);
    const uint64_t bd0 = umma::desc_kmajor(umma::smem_u32(smem + E * t.a_bytes), nkp * 16, 128);
    const u32 sstep = t.stage_bytes >> 4, estep = t.a_bytes >> 4, ka = lbo >> 3, kb = nkp * 2;
    bool ok = true;
    u32 it = 0, ti = 0, st = 0, par = 0;
    for (u32 tile = blockIdx.x; ok && tile < t.ntiles; tile += gridDim.x, ti++) {
      const u32 nb = ti % t.NB, use = ti / t.NB;
      if (use > 0 && !(ok = umma::mbar_wait(&acc_empty[nb], (use - 1) & 1, err, 13))) break;
      umma::fence_after_sync();
      const u32 tm = tmem + nb * E * nkc;
      for (u32 c = 0; c < nchunks; c++, it++) {
        if (!(ok = umma::mbar_wait(&full_bar[st], par, err, 14))) break;
        umma::fence_after_sync();
        const uint64_t ad = ad0 + st * sstep, bd = bd0 + st * sstep;
        if (umma::elect_one()) {
#pragma unroll
          for (u32 ks = 0; ks < CKI_CHUNK / 32; ks++)
            umma::mma_i8_u(tm, ad + ks * ka, bd + ks * kb, idesc, (c > 0 || ks > 0) ? 1u : 0u);
          if (E == 2)
#pragma unroll
            for (u32 ks = 0; ks < CKI_CHUNK / 32; ks++)
              umma::mma_i8_u(tm + nkc, ad + estep + ks * ka, bd + ks * kb, idesc, (c > 0 || ks > 0) ? 1u : 0u);
          umma::commit(&empty_bar[st]);
          if (c + 1 == nchunks) umma::commit(&acc_full[nb]);
        }
        __syncwarp();
        if (++st == t.nst) {
          st = 0;
          par ^= 1;
        }
      }
    }
    // MMAs still in flight complete before TMEM is freed
    for (u32 c = it >= t.nst ? it - t.nst : 0; c < it; c++)
      umma::mbar_wait(&empty_bar[c % t.nst], (c / t.nst) & 1, err, 15);
  } else if (warp < CKI_EPI / 32) {
    const u32 ng = 2 * nck, pst = ng + 1;  // an odd row stride keeps 8 lanes on 8 bank groups
    const u32 row = (warp & 3) * 32 + lane, ch = warp >> 2;  // TMEM lane; parity of the key-row pairs
    const bool valid = row < V * 14;
    const u32 npair = (nck + 1) / 2;
    u32 ti = 0;
    for (u32 tile = blockIdx.x; tile < t.ntiles; tile += gridDim.x, ti++) {
      const u32 nb = ti % t.NB, use = ti / t.NB;
      const u32 he = tile % t.nE, rest = tile / t.nE, s = rest / t.lob;
      // the finishing tasks' constants, loaded while the MMAs run: under the
      // copies' traffic a dependent global load takes microseconds
      const u64 z = __ldg(zeta + s);
      u64 te[E][NIT], to[E][NIT];
#pragma unroll
      for (u32 e = 0; e < E; e++)
#pragma unroll
        for (u32 i = 0; i < NIT; i++) {
          const u32 vr = (i * CKI_EPI + tid) >> 2, r = vr % nck, v = vr / nck;
          te[e][i] = to[e][i] = 0;
          if (v < V) {
            const u64* th = thi + ((u64)r * nhi_t + (he * E + e) * im.G + v / im.R) * d + s;
            te[e][i] = __ldg(th);
            to[e][i] = __ldg(th + n);
          }
        }
      // all epilogue threads stop together, also when only some of them gave
      // up; the barrier also orders the last tile's reads before new sums
      if (!bar_epi_and(umma::mbar_wait(&acc_full[nb], use & 1, err, 16))) break;
      umma::fence_after_sync();
      const u32 tb = tmem + (((warp & 3) * 32) << 16) + nb * E * nkc;
      ulonglong2 f[E][PAIRS][4];
#pragma unroll
      for (u32 e = 0; e < E; e++) fold_pairs<PAIRS>(tb + e * nkc, ch, npair, nkp, f[e]);
      umma::fence_before_sync();
      umma::mbar_arrive(&acc_empty[nb]);
#pragma unroll
      for (u32 e = 0; e < E; e++) {
        if (e > 0) bar_epi();  // accumulator 0's sums have been read
        if (valid)
#pragma unroll
          for (u32 i = 0; i < PAIRS; i++)
#pragma unroll
            for (u32 g = 0; g < 4; g++) {
              const u32 grp = 4 * (2 * i + ch) + g;
              if (grp < ng) Pm[row * pst + grp] = f[e][i][g];
            }
        bar_epi();
        // combos of (virtual row v, key row r): lane 0 c a, 1 d b, 2 c b, 3 d a
#pragma unroll
        for (u32 i = 0; i < NIT; i++) {
          const u32 w = i * CKI_EPI + tid;
          if (i * CKI_EPI >= V * nck * 4) break;
          const bool act = w < V * nck * 4;
          const u32 combo = w & 3, vr = act ? w >> 2 : 0, r = vr % nck, v = vr / nck;
          const u32 half = (combo == 1 || combo == 2) ? 1 : 0, comp = combo & 1;
          const ulonglong2* p = Pm + (14 * v + 7 * half) * pst + 2 * r + comp;
          u64 h128 = 0, l128 = 0;
#pragma unroll
          for (u32 y = 0; y < 7; y++) {
            const ulonglong2 pv = p[y * pst];
            add_shifted(h128, l128, pv.x, 8 * y);
            add_shifted(h128, l128, pv.y, 8 * y + 32);
          }
          u64 val = reduce128_any(M, h128, l128);
          if (combo == 1) val = mul_mod(M, z, val);
          // lanes 0, 1: re = c a + zeta d b; lanes 2, 3: im = c b + d a
          val = add_mod(val, __shfl_xor_sync(0xffffffffu, val, 1), M.q);
          const u64 other = __shfl_xor_sync(0xffffffffu, val, 2);
          const u64 re = combo < 2 ? val : other, imv = combo < 2 ? other : val;
          // (re + X im) (te + X to): lane 0 re te, 1 zeta im to, 2 im te, 3 re to
          u64 pr = mul_mod(M, (combo == 0 || combo == 3) ? re : imv, (combo & 1) ? to[e][i] : te[e][i]);
          if (combo == 1) pr = mul_mod(M, z, pr);
          pr = add_mod(pr, __shfl_xor_sync(0xffffffffu, pr, 1), M.q);
          if (act && !(combo & 1))
            atomic_add_mod(acc + ((u64)r * im.R + v % im.R) * d + (combo ? n : 0) + s, pr, M.q, plain);
        }
      }
    }
  }
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

}  // namespace

CkImage cki_shape(u32 R, u64 width, u32 n, u32 ck_bt) {
  CkImage im{};
  im.R = R;
  im.n = n;
  im.width = width;
  const u64 bt = width < ck_bt ? width : ck_bt;
  im.btlog = 63u - (u32)__builtin_clzll(bt);
  im.nlc = (u32)(bt / CKI_CHUNK);
  const u64 nhi = width / bt;
  // few rows: stack key blocks while they fit the MMA's 128 rows
  im.G = 1;
  while (2 * im.G * R <= CKI_MAX_V && nhi % (2 * im.G) == 0) {
    im.G *= 2;
    im.glog++;
  }
  im.nhg = (u32)(nhi / im.G);
  im.VP = cki_vp(R * im.G);
  return im;
}
u64 cki_bytes(const CkImage& im) { return (u64)im.nhg * im.nlc * im.n * 64 * im.VP; }
bool cki_ok(u32 R, u64 width, u32 n, u32 ck_bt, u64 q) {
  return q < (1ULL << 50) && (n == 64 || n == 128 || n == 256) && R >= 1 && R <= CKI_MAX_V && width >= CKI_CHUNK &&
         (width & (width - 1)) == 0 && ck_bt >= CKI_CHUNK;
}

// Tile shape: the block width that minimises waves x (chunks + the exposed
// part of an epilogue, about 4 chunk times), plus the last epilogue.
static CkImgTiles cki_tiles(const CkImage& im, u32 nck, u32 nkp, u32 nkc) {
  CkImgTiles t{};
  const u32 bt = 1u << im.btlog;
  // Two accumulators share a key tile when it outweighs a witness tile by
  // half: 3 rows x 2^18 under 12 keys 167 us against 182 us, but 9 x 2^17 203
  // against 197 us (one accumulator is double-buffered) and 9 x 2^14 58
  // against 49 us.  Above 12 key rows the epilogue could not hold both in registers.
  t.E = im.nhg % 2 == 0 && nck <= 12 && 2 * nkp >= 3 * im.VP ? 2 : 1;
  t.NB = 2 * t.E * nkc <= 512 ? 2 : 1;
  t.nE = im.nhg / t.E;
  t.a_bytes = 64 * im.VP;
  t.b_bytes = CKI_CHUNK * nkp;
  t.stage_bytes = (t.E * t.a_bytes + t.b_bytes + 127) / 128 * 128;
  double best = 0;
  // 2^14 byte products of at most 255^2 keep a sum below 2^31
  const u32 top = bt < 16384 ? bt : 16384;
  for (u32 Bw = top; Bw >= 512 || Bw == top; Bw /= 2) {
    const u64 tiles = (u64)im.n * (bt / Bw) * t.nE;
    const u64 waves = (tiles + 147) / 148;
    const double cost = (double)waves * (Bw / CKI_CHUNK + 4.0) + 8.0 * t.E;
    if (best == 0 || cost < best) {
      best = cost;
      t.Bw = Bw;
    }
  }
  t.lob = bt / t.Bw;
  t.ntiles = im.n * t.lob * t.nE;
  return t;
}

int launch_ck_img(const CkImgArgs& a, const CkImage& im, const ModQ& M, const u64* zeta, cudaStream_t st) {
  const u32 nkp = ck_tk8_nkp(a.nck), V = im.R * im.G;
  u32 nkc = 32;  // TMEM columns between accumulators
  while (nkc < nkp) nkc *= 2;
  if (!im.p || !a.tk8 || V == 0 || V > CKI_MAX_V || a.nck == 0 || a.nck > CKU_MAX_KEYS ||
      im.width > (u64)a.ck_bt * a.ck_nhi)
    return salsaa_set_error(-2, "ck_img: shape outside the image path");
  CkImgTiles t = cki_tiles(im, a.nck, nkp, nkc);
  const size_t epi = (size_t)V * 14 * (2 * a.nck + 1) * 16;
  // the MMA reads 128 rows of the last 16-byte slice: up to 2 KiB past the
  // stage's own bytes, inside the next stage or the partial sums
  constexpr size_t most = 225 * 1024;
  const size_t room = most - (epi > 2048 ? epi : 2048);
  t.nst = (u32)(room / t.stage_bytes);
  if (t.nst > CKI_MAX_STAGES) t.nst = CKI_MAX_STAGES;
  if (t.nst < 2) return salsaa_set_error(-2, "ck_img: stages do not fit shared memory");
  const size_t smem = (size_t)t.nst * t.stage_bytes + (epi > 2048 ? epi : 2048);
  auto kern = t.E == 2 ? ck_img_kernel<2, 3> : a.nck <= 12 ? ck_img_kernel<1, 3> : ck_img_kernel<1, 5>;
  cudaError_t e = smem_limit(kern, most);
  if (e != cudaSuccess) return salsaa_set_cuda_error(e, "ck_img smem attribute");
  const bool plain = M.q < (1ULL << 50) && im.width / t.Bw < (1ULL << 13);
  // the image and the key table's tiles once, the sums once
  const double bytes = (double)cki_bytes(im) + (double)((u64)im.n * nkp << im.btlog) + 8.0 * a.nck * im.R * 2 * im.n;
  const int tr = salsaa_trace_begin("ck_img_kernel", st, bytes);
  salsaa_trace_alias(tr, "ck_img_kernel:int8", 2.0 * 196.0 * a.nck * im.R * (double)im.width * im.n);
  salsaa_trace_alias(tr, "ck_img_kernel:mac", (double)a.nck * im.R * (double)im.width * 2 * im.n);
  const u32 grid = t.ntiles < 148 ? t.ntiles : 148;
  pdl(kern, grid, CKI_THREADS, smem, st)(a.tk8, im, t, a.nck, nkp, nkc, a.thi, a.ck_nhi, M, zeta, a.acc,
                                                 plain, tc_error_word());
  salsaa_trace_end(tr, st);
  salsaa_count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : salsaa_set_cuda_error(e, "ck_img launch");
}

}  // namespace salsaa
