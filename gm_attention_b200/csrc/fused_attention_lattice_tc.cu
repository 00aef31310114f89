// Tensor-core version of the lattice fast path for bf16 node fields.
//
// Same layer, same compact tables as fused_attention_lattice.cu.  The identity
// that makes the contraction a matrix product: the transport phase commutes
// with the sum over copies,
//
//   <q_i, tau k_j> = G0 + sum_n Re( tau_n(i, j) * G_n ),   G_n = sum_c conj(q_{i,c}) k_{j,c},
//   sum_j alpha_ij tau_n v_j = ((alpha o tau_n) V)_i,
//
// so for 8 consecutive owners (targets; sources in the backward's source-major
// pass) of one lattice row and 16 neighbour positions the
// Gram blocks G0, Re G_n, Im G_n are plain bf16 x bf16 -> fp32 products, the
// phases / bias / window enter elementwise on the tile in registers, and the value
// sums are products with the weights as an operand.  The
// positions are the M dimension of the MMAs (16 per step) and a warp's owners the
// N dimension (8 per warp):
//
//   S^T   (16 positions x 8 owners)  = tile (positions x columns) * owners^T      A: shared memory, B: loop-invariant registers
//   out^T (16 columns   x 8 owners) += tile^T (columns x positions) * (P o tau)^T  A: shared memory (ldmatrix.trans), B: P^T
//
// * Only the longitude band of a row pair is visited: 8 owners see 7 + cnt positions of a neighbour row.  The positions of
//   all neighbour rows are PACKED into steps of 16 (ldmatrix takes each of its 16 rows from anywhere), so the narrow
//   equatorial windows (cnt <= 7, 9 to 14 positions a row) leave no step half empty; pairs outside an owner's window and the
//   list's padding meet a table entry with bias -inf, without a bounds test.
// * Im G_n uses a pre-swapped copy of the OWNERS' fragments, (re, im) -> (-im, re) or (im, -re), made once per (sample, head).
// * The imaginary part of the phase accumulates into a second accumulator set; the multiplication by +-i (the pair
//   swap) is applied once in the epilogue, so the staged value tile is never swapped.
// * The weights P (accumulator layout: position rows, owner columns) become a B operand with movmatrix (8 x 8 b16
//   transpose in registers); the same instruction turns the result tiles into 4-byte stores per owner.
// * The softmax reference maximum of an owner moves only when it is exceeded by 2^8 (lazy rescaling).
//
// One CTA: a tile of four lattice rows x 8 (or 16) longitudes, a warp per row and 8 longitudes, which share the staged
// neighbourhood (the rows' windows overlap: 120 staged rows serve 32 owners at radius 3, against 250 for 32 owners of one
// row); it walks over (sample, head) pairs with one list of positions and one set of table entries.  The next pair's rows are
// under way (cp.async, both fields of a position in one shared-memory row whose pitch is an odd multiple of 16 bytes: no
// bank conflicts) while this pair's results are written.  Neighbourhoods that outgrow shared memory -- the polar rows' -- come
// in chunks.  The lists depend on the windows alone: gm_lattice_plan_build works them out once per table, gm_lattice_plan_refresh
// adds the entries in front of every pass, and a CTA copies both; a row tile whose windows are no longer the plan's, and every CTA
// without a plan, works them out itself (128 x 256, batch 4, 8 x (m <= 3): 1 953 against 1 670 us for the three passes).
// Tensor-core instruction: mma.sync m16n8k16 (bf16 inputs, fp32 accumulate).
//
// What it measured against the kernel before it (one row of 32 longitudes and one (sample, head) per CTA, a step per
// neighbour row, TMA staging), us forward / pass T / pass S: 128 x 256, batch 4, 4 heads of 8 x (m <= 3): 603 / 904 / 995 ->
// 433 / 560 / 677; 256 x 512, batch 8, 4 heads of 16 x (m <= 2): 3 670 / 4 896 / 6 643 -> 3 358 / 4 648 / 6 163; heads that
// are not 16 copies wide, batch 1 to 8: 1.2 to 4 times faster.  What bounds it: of the last forward 2.1 ms are the steps
// (shared-memory bandwidth: ten ldmatrix.x4 and the entries, about 100 of 114 cycles a step), 1.4 ms the staging and the
// per-pair prologue and epilogue, which overlap only across the SM's two CTAs.  16 longitudes per CTA pay in the forward
// (3 998 -> 3 422 us at first); passes T and S want 168 registers a thread, so three CTAs of 4 warps.
//
// Backward, two deterministic passes (no atomics):
//   pass T: owners = targets.  Delta = <dO, O> per (target, head) from the owners' own rows (written out for pass S);
//           Gram blocks of (q, k) and of (dO, v) give the logits and d alpha; ds = scale p (d alpha - Delta)
//           weights (ds o tau) K -> dq.
//   pass S: owners = SOURCES, neighbours = the targets that see them (transposed tables, their lse / Delta
//           staged with them).  Same Gram blocks with the roles swapped, then (ds o conj tau) Q -> dk and
//           (p o conj tau) dO -> dv.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace gmb {
namespace {

constexpr float TC_LOG2E = 1.4426950408889634f, TC_LN2 = 0.6931471805599453f;
constexpr int TC_MAX_CF = 3;
constexpr int TC_MAX_WIN = 33;  // 2 W + 1 neighbour rows at most

struct TcPlan {
  int a0, ac, n_cf;
  int real_off;
  int cf_off[TC_MAX_CF];
  int cf_order[TC_MAX_CF];
};

struct PkCaps {  // what a chunk of a tile's neighbourhood may hold: staged rows, entry pairs
  int rows, entries;
};

struct TcArgs {
  const __nv_bfloat16 *own1, *own2;   // owners' fields:     q, -  |  q, dO  |  k, v
  const __nv_bfloat16 *nb1, *nb2;     // neighbours' fields: k, v  |  k, v   |  q, dO
  const float *lse, *delta;           // (nodes, H), backward
  const __nv_bfloat16* out_fwd;       // pass T with delta_out: the forward's output, Delta = <dO, O> is formed here
  float* delta_out;                   // pass T: where Delta is written for the source-major pass (null: read `delta`)
  __nv_bfloat16 *res1, *res2;         // out | dq | dk, dv
  float* lse_out;                     // forward
  const int *win_cnt, *win_lo, *win_off;
  const float* entries;               // (n_entries, 8): (cos, sin) of orders 1..NORD, bias at 2 NORD
  const int* row_order;
  int rows, nlon, D, H, W, NORD;
  int even;     // and every block starts on an even column and has an even width: 4-byte accesses throughout
  int padded;   // blocks narrower than 16 (scalar) / 16 KSC (complex) columns
  int unit, units;  // staging: bytes of one copy (16, 8, 4; 2: element by element), copies per head row and field
  int n_order;      // rows in row_order (all of them: the list is not read)
  PkCaps caps;                                     // what shared memory holds (a chunk)
  const int* plan_first;                           // with a plan: (row tiles + 1) first record of a row tile, and the records
  const unsigned char* records;
  int64_t record_bytes;
  int n_bh, heavy_bh, light_bh;                    // (sample, head) pairs: all, and per CTA of a polar / any other row tile
  int heavy_tiles, heavy_ctas;                     // row tiles next to the poles, and the CTAs (the first of the grid) that take them
  float scale;
  TcPlan plan;
  int slots;  // row tiles the grid is made for: all of them, or as many as a short row list can touch
  int words;    // rows and owners' / result fields are whole 4-byte words: 4-byte accesses to (even column, next column)
};

enum { TC_FWD = 0, TC_BWD_T = 1, TC_BWD_S = 2 };

__device__ __forceinline__ int tc_wrap(int x, int n) {
  x %= n;
  return x < 0 ? x + n : x;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16-byte asynchronous copy global -> shared; src_bytes = 0 writes zeros
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(addr), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int BYTES>
__device__ __forceinline__ void cp_async_ca(void* dst, const void* src) {  // 4 or 8 bytes
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(addr), "l"(src), "n"(BYTES));
}
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// (re, im) -> (im, -re) / (-im, re): the B operand of the imaginary Gram part for owners carrying q / carrying k
__device__ __forceinline__ unsigned swap_neg(unsigned w) { return __byte_perm(w, 0, 0x1032) ^ 0x80000000u; }
__device__ __forceinline__ unsigned swap_neg_lo(unsigned w) { return __byte_perm(w, 0, 0x1032) ^ 0x00008000u; }

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&v);
}

__device__ __forceinline__ unsigned movmatrix_trans(unsigned x) {
  unsigned y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void mma_bf16_b2(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) { mma_bf16(d, a, b[0], b[1]); }
// d = a * b (no accumulator to zero first)
__device__ __forceinline__ void mma_bf16_b2_init(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ float fast_exp2(float x) {  // ex2.approx: exp2(-inf) = 0, relative error ~2^-22
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// S^T blocks of 16 packed positions x 8 owners: g0 (scalar block), gr / gi per complex frequency.
// fb: the owners' fragments, fs: their pre-swapped copies for the imaginary part (complex k-steps only).
// addr: shared-memory address of this lane's position (lane & 15) and half (lane >> 4) of the field's first 16 columns.
template <int KS0, int NCF, int KSC>
__device__ __forceinline__ void gram_step(const unsigned (&fb)[KS0 + NCF * KSC][2], const unsigned (&fs)[NCF * KSC][2], unsigned addr, float (&g0)[4],
                                          float (&gr)[NCF][4], float (&gi)[NCF][4]) {
  if constexpr (KS0 > 0) {
    unsigned af[4];
    ldsm_x4(af, addr);
    mma_bf16_b2_init(g0, af, fb[0]);
  } else {
    g0[0] = g0[1] = g0[2] = g0[3] = 0.f;
  }
#pragma unroll
  for (int f = 0; f < NCF; ++f)
#pragma unroll
    for (int sub = 0; sub < KSC; ++sub) {
      unsigned af[4];
      ldsm_x4(af, addr + 32 * (KS0 + f * KSC + sub));
      if (sub == 0) {
        mma_bf16_b2_init(gr[f], af, fb[KS0 + f * KSC + sub]);
        mma_bf16_b2_init(gi[f], af, fs[f * KSC + sub]);
      } else {
        mma_bf16_b2(gr[f], af, fb[KS0 + f * KSC + sub]);
        mma_bf16_b2(gi[f], af, fs[f * KSC + sub]);
      }
    }
}

// acc^T (padded head columns x 8 owners) += tile^T (columns x 16 packed positions) * B, B = x0 for the scalar block,
// xr[f] into the real-phase accumulators and xi[f] into the imaginary-phase accumulators of frequency f.
// addr: shared-memory address of position 8 (lane >> 4) + (lane & 7) and half (lane >> 3 & 1) of the field's first 16 columns.
template <int KS0, int NCF, int KSC>
__device__ __forceinline__ void accumulate_step(float (&acc0)[4], float (&accr)[NCF * KSC][4], float (&acci)[NCF * KSC][4], const unsigned (&x0)[2],
                                                const unsigned (&xr)[NCF][2], const unsigned (&xi)[NCF][2], unsigned addr) {
  if constexpr (KS0 > 0) {
    unsigned af[4];
    ldsm_x4_trans(af, addr);
    mma_bf16_b2(acc0, af, x0);
  }
#pragma unroll
  for (int f = 0; f < NCF; ++f)
#pragma unroll
    for (int sub = 0; sub < KSC; ++sub) {
      unsigned af[4];
      ldsm_x4_trans(af, addr + 32 * (KS0 + f * KSC + sub));
      mma_bf16_b2(accr[f * KSC + sub], af, xr[f]);
      mma_bf16_b2(acci[f * KSC + sub], af, xi[f]);
    }
}

// Flat column of the pair of padded head-local columns (col, col + 1) of k-step / m-tile `kt` (compile-time), col even in
// 0 .. 14: first = flat column or -1 (padding), second likewise.  No division: the block is known at compile time.
template <int KS0, int NCF, int KSC, int KT>
__device__ __forceinline__ void flat_pair(const TcPlan& P, int h, int col, int& g0, int& g1) {
  if constexpr (KT < KS0) {
    const int cc = 16 * KT + col;
    g0 = cc < P.a0 ? P.real_off + h * P.a0 + cc : -1;
    g1 = cc + 1 < P.a0 ? P.real_off + h * P.a0 + cc + 1 : -1;
  } else {
    constexpr int F = (KT - KS0) / KSC, SUB = (KT - KS0) % KSC;
    const int cc = 16 * SUB + col;
    g0 = cc < 2 * P.ac ? P.cf_off[F] + 2 * h * P.ac + cc : -1;
    g1 = g0 >= 0 ? g0 + 1 : -1;  // 2 ac is even: a (re, im) pair is never split
  }
}

// First flat column of k-step / m-tile KT of head h
template <int KS0, int NCF, int KSC, int KT>
__device__ __forceinline__ int block_column(const TcPlan& P, int h) {
  if constexpr (KT < KS0) return P.real_off + P.a0 * h + 16 * KT;
  else return P.cf_off[(KT - KS0) / KSC] + 2 * P.ac * h + 16 * ((KT - KS0) % KSC);
}
// Whether word r of this lane (columns 8 r + 2 c, 8 r + 2 c + 1 of k-step / m-tile KT) holds columns of the head rather than
// padding, every block being of an even width
template <int KS0, int NCF, int KSC, int KT>
__device__ __forceinline__ bool in_block(const TcPlan& P, int c, int r) {
  return 2 * c + 8 * r + (KT < KS0 ? 16 * KT : 16 * ((KT - KS0) % KSC)) < (KT < KS0 ? P.a0 : 2 * P.ac);
}

// B-operand fragments of one owner (column n = g of the warp's 8) for every k-step of the padded head layout
template <int KS0, int NCF, int KSC, int KT = 0>
__device__ __forceinline__ void load_owner_columns(const TcPlan& P, const __nv_bfloat16* src, bool even, bool words, int h, int c,
                                                   unsigned (&fb)[KS0 + NCF * KSC][2]) {
  if constexpr (KT < KS0 + NCF * KSC) {
    if (even) {
      const unsigned* w = reinterpret_cast<const unsigned*>(src + block_column<KS0, NCF, KSC, KT>(P, h)) + c;
      fb[KT][0] = in_block<KS0, NCF, KSC, KT>(P, c, 0) ? w[0] : 0u;
      fb[KT][1] = in_block<KS0, NCF, KSC, KT>(P, c, 1) ? w[4] : 0u;
    } else {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        int g0, g1;
        flat_pair<KS0, NCF, KSC, KT>(P, h, 2 * c + 8 * r, g0, g1);
        unsigned w = 0u;
        if (words && g0 >= 0 && g1 == g0 + 1 && (g0 & 1) == 0) {
          w = *reinterpret_cast<const unsigned*>(src + g0);
        } else {
          if (g0 >= 0) w = __bfloat16_as_ushort(src[g0]);
          if (g1 >= 0) w |= (unsigned)__bfloat16_as_ushort(src[g1]) << 16;
        }
        fb[KT][r] = w;
      }
    }
    load_owner_columns<KS0, NCF, KSC, KT + 1>(P, src, even, words, h, c, fb);
  }
}

// One m-tile (16 head columns x 8 owners, accumulator layout) of a result -> global memory: transposed in registers
// (movmatrix) so that a thread holds two adjacent columns of ONE owner (own_b): 4-byte stores.
template <int KS0, int NCF, int KSC, int KT>
__device__ __forceinline__ void store_tile(const TcPlan& P, __nv_bfloat16* dst, bool present, bool even, bool words, int h, int c, const float (&v)[4]) {
  const unsigned w0 = movmatrix_trans(pack_bf16(v[0], v[1]));  // (owner own_b; columns 2c, 2c + 1)
  const unsigned w1 = movmatrix_trans(pack_bf16(v[2], v[3]));  // (owner own_b; columns 2c + 8, 2c + 9)
  if (even) {
    unsigned* w = reinterpret_cast<unsigned*>(dst + block_column<KS0, NCF, KSC, KT>(P, h)) + c;
    if (present && in_block<KS0, NCF, KSC, KT>(P, c, 0)) w[0] = w0;
    if (present && in_block<KS0, NCF, KSC, KT>(P, c, 1)) w[4] = w1;
    return;
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const unsigned w = r ? w1 : w0;
    int g0, g1;
    flat_pair<KS0, NCF, KSC, KT>(P, h, 2 * c + 8 * r, g0, g1);
    if (!present) continue;
    if (words && g0 >= 0 && g1 == g0 + 1 && (g0 & 1) == 0) {
      *reinterpret_cast<unsigned*>(dst + g0) = w;
    } else {
      if (g0 >= 0) dst[g0] = __ushort_as_bfloat16((unsigned short)(w & 0xffffu));
      if (g1 >= 0) dst[g1] = __ushort_as_bfloat16((unsigned short)(w >> 16));
    }
  }
}

// combine the phase accumulators of every complex m-tile and store all m-tiles of one result
template <int KS0, int NCF, int KSC, bool CONJ, int M = 0>
__device__ __forceinline__ void store_result(const TcPlan& P, __nv_bfloat16* dst, bool present, bool even, bool words, int h, int g, int c,
                                             const float (&inv)[2],
                                             const float (&acc0)[4], const float (&accr)[NCF * KSC > 0 ? NCF * KSC : 1][4],
                                             const float (&acci)[NCF * KSC > 0 ? NCF * KSC : 1][4]) {
  if constexpr (M == 0 && KS0 > 0) {
    const float v[4] = {acc0[0] * inv[0], acc0[1] * inv[1], acc0[2] * inv[0], acc0[3] * inv[1]};
    store_tile<KS0, NCF, KSC, 0>(P, dst, present, even, words, h, c, v);
  }
  if constexpr (M < NCF * KSC) {
    // rows of an accumulator m-tile are head columns g, g + 8: even = real part, odd = imaginary part.
    // With i the sums under the table's -sin:
    //   tau:      re = r_re + i_im,  im = r_im - i_re;      conj tau:  re = r_re - i_im,  im = r_im + i_re
    const float sgn = ((g & 1) != 0) == CONJ ? 1.f : -1.f;
    float v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) v[x] = (accr[M][x] + sgn * __shfl_xor_sync(0xffffffffu, acci[M][x], 4)) * inv[x & 1];
    store_tile<KS0, NCF, KSC, KS0 + M>(P, dst, present, even, words, h, c, v);
    store_result<KS0, NCF, KSC, CONJ, M + 1>(P, dst, present, even, words, h, g, c, inv, acc0, accr, acci);
  }
}

// ---- packed pairs of floats (one 64-bit register pair, one instruction for two elements)
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned pack_bf16(f32x2 v) {
  float lo, hi;
  unpack2(v, lo, hi);
  return pack_bf16(lo, hi);
}

// ---- tile shape and shared memory
constexpr int pk_warps(int mode) { return mode == TC_FWD ? 8 : 4; }  // four owner rows x 8 longitudes per four warps
constexpr int pk_ctas(int warps) { return warps == 4 ? 3 : 2; }      // per SM: 12 warps of 168 registers, 16 of 128
constexpr int PK_ROWS = 4;                  // lattice rows of a CTA's owner tile
constexpr int PK_MAX_SEG = TC_MAX_WIN + PK_ROWS - 1;  // neighbour rows of the tile
constexpr int PK_DUMMY = 8;                 // entries with bias -inf at the start of the table (a packed list's padding points at the last but one)

template <int KS0, int NCF, int KSC>
struct PkLayout {
  static constexpr int KQ = KS0 + NCF * KSC;
  static constexpr int FIELD = 32 * KQ;         // bytes of one field of a staged row: the scalar block, then every frequency, 32 bytes per k-step
  static constexpr int PITCH = 2 * FIELD + 16;  // both fields and (lse, Delta): an odd multiple of 16 bytes, so ldmatrix meets no bank conflict
  static constexpr int ENTRY = 16 * NCF + 8;    // bytes of a table entry pair
};

struct PkSegment {  // one neighbour row of the tile: its row, first longitude offset from the tile's first column, staged positions
  int j, lo, len;
};
struct PkCursor {
  int seg, at;  // next segment, positions of it already taken
};
struct PkWindows {  // the tables a tile's neighbourhood is read from
  const int *win_cnt, *win_lo, *win_off;
  int rows, nlon, W;
};
struct PkTile {  // a tile's neighbour rows, in shared memory
  int4 win[PK_ROWS][PK_MAX_SEG];  // of (owner row, neighbour row): count, first offset, first entry
  PkSegment seg[PK_MAX_SEG];      // the non-empty neighbour rows
  int n_seg;
};
struct PkPair {
  int h;
  int64_t row0, node0;  // first node of the warp's owner row, of the sample
};
struct PkChunk {
  int rows, entries, steps;  // staged rows, entry pairs (with the dummies), this warp's steps of 16 positions
};

// The windows of the rows r0 .. r0 + 3, and the neighbour rows some of them see.  Ends with a barrier.
template <int WARPS>
__device__ __forceinline__ void pk_open_tile(const PkWindows& t, int r0, PkTile& tile) {
  constexpr int TLON = 8 * (WARPS / PK_ROWS);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, spans = 2 * t.W + PK_ROWS;
  for (int x = threadIdx.x; x < spans * PK_ROWS; x += 32 * WARPS) {
    const int i = x & (PK_ROWS - 1), s = x / PK_ROWS, j = r0 - t.W + s, w = s - i;  // w: place of row j in owner row i's windows
    int4 v = make_int4(0, 0, 0, 0);
    if (r0 + i < t.rows && j >= 0 && j < t.rows && w >= 0 && w <= 2 * t.W) {
      const int at = (r0 + i) * (2 * t.W + 1) + w;
      v = make_int4(t.win_cnt[at], t.win_lo[at], t.win_off[at], 0);
    }
    tile.win[i][s] = v;
  }
  __syncthreads();
  if (warp == 0) {  // compact the non-empty neighbour rows
    int filled = 0;
    for (int s0 = 0; s0 < spans; s0 += 32) {
      const int s = s0 + lane;
      int lo = 0x7fffffff, hi = -0x7fffffff;
      int4 w[PK_ROWS];
#pragma unroll
      for (int i = 0; i < PK_ROWS; ++i) {
        w[i] = s < spans ? tile.win[i][s] : make_int4(0, 0, 0, 0);
        if (w[i].x > 0) {
          lo = min(lo, w[i].y);
          hi = max(hi, w[i].y + w[i].x);
        }
      }
      const unsigned have = __ballot_sync(0xffffffffu, hi > lo);
      const int k = filled + __popc(have & ((1u << lane) - 1u));
      __syncwarp();
      if (hi > lo) {
        tile.seg[k] = PkSegment{r0 - t.W + s, lo, hi - lo + TLON - 1};
#pragma unroll
        for (int i = 0; i < PK_ROWS; ++i) tile.win[i][k] = w[i];  // k <= s: only places that have been read
      }
      __syncwarp();
      filled += __popc(have);
    }
    if (lane == 0) tile.n_seg = filled;
  }
  __syncthreads();
}

// One chunk: as many neighbour positions as `caps` allows, from the cursor on (which advances).  Every warp works the chunk
// out for itself, lane p looking after the p-th segment; chunk boundaries depend on the tables alone, not on which rows are
// asked for.  Written: the staged rows' nodes through put_node(row, neighbour row, offset from the tile's first column), the
// entry pairs (x, x - 1) through put_pair(place, index of entry x, index of entry x - 1), -1 outside the window, and this warp's
// list of packed positions if it wants one.  `write` false: nothing, the chunk is only measured.
template <int WARPS, typename PutNode, typename PutPair>
__device__ __forceinline__ PkChunk pk_build(const PkTile& tile, PkCursor& cur, PkCaps caps, int pitch16, bool write, bool wants, unsigned* list,
                                            const PutNode& put_node, const PutPair& put_pair) {
  constexpr int TLON = 8 * (WARPS / PK_ROWS);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, my_row = warp & (PK_ROWS - 1), l0 = 8 * (warp / PK_ROWS);
  const int R = caps.rows, E = caps.entries, n_seg = tile.n_seg;
  const int s = cur.seg + lane;
  const bool have = s < n_seg;
  const PkSegment sg = have ? tile.seg[s] : PkSegment{0, 0, 0};
  const int skip = lane == 0 ? cur.at : 0, len = have ? sg.len - skip : 0;
  int before = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += y;
  }
  before -= len;
  int take = min(min(len, max(R - before, 0)), (E - PK_DUMMY) / PK_ROWS - TLON);
  const unsigned cut = __ballot_sync(0xffffffffu, take < len || !have);
  if (cut != 0 && lane > __ffs(cut) - 1) take = 0;
  const int ua = sg.lo + skip;  // the piece's first offset from the tile's first column
  int xa = 0, xn = 0, eb = 0, entries = 0;  // my row's entries of the piece: first offset, count, place
  int4 win = make_int4(0, 0, 0, 0);
#pragma unroll
  for (int i = 0; i < PK_ROWS; ++i) {
    const int4 w = have ? tile.win[i][s] : make_int4(0, 0, 0, 0);
    const int from = max(w.y - 6, ua - TLON + 2), to = min(w.y + w.x + 7, ua + take);
    const int n = take > 0 && w.x > 0 ? max(to - from, 0) : 0;
    if (i == my_row) {
      xa = from;
      xn = n;
      eb = entries;
      win = w;
    }
    entries += n;
  }
  int e_before = entries;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, e_before, o);
    if (lane >= o) e_before += y;
  }
  if (e_before > E - PK_DUMMY) take = 0;  // a suffix of the pieces: the counts are never negative
  eb += e_before - entries + PK_DUMMY;
  const unsigned taken = __ballot_sync(0xffffffffu, take > 0);
  const int pieces = __popc(taken), last = pieces - 1;
  PkChunk chunk;
  chunk.rows = pieces ? __shfl_sync(0xffffffffu, before + take, last) : 0;
  chunk.entries = PK_DUMMY + (pieces ? __shfl_sync(0xffffffffu, e_before, last) : 0);
  const int last_take = __shfl_sync(0xffffffffu, take, last), last_len = __shfl_sync(0xffffffffu, len, last), last_skip = __shfl_sync(0xffffffffu, skip, last);
  // my positions of the piece
  const int pa = max(ua, win.y + l0), pn = wants && take > 0 && win.x > 0 ? max(min(ua + take, win.y + win.x + l0 + 7) - pa, 0) : 0;
  int placed = 0;
  for (int p = 0; p < pieces; ++p) {
    const int ln = __shfl_sync(0xffffffffu, pn, p);
    if (write) {
      const int base = __shfl_sync(0xffffffffu, before, p), u = __shfl_sync(0xffffffffu, ua, p), n = __shfl_sync(0xffffffffu, take, p);
      const int px = __shfl_sync(0xffffffffu, xa, p), pxn = __shfl_sync(0xffffffffu, xn, p), pe = __shfl_sync(0xffffffffu, eb, p);
      const int wlo = __shfl_sync(0xffffffffu, win.y, p), wcnt = __shfl_sync(0xffffffffu, win.x, p), woff = __shfl_sync(0xffffffffu, win.z, p);
      const int lu = __shfl_sync(0xffffffffu, pa, p), j = __shfl_sync(0xffffffffu, sg.j, p);
      if ((p & (WARPS - 1)) == warp)
        for (int x = lane; x < n; x += 32) put_node(base + x, j, u + x);
      if (WARPS == PK_ROWS || (p & 1) == warp / PK_ROWS)
        for (int x = lane; x < pxn; x += 32) {
          const int at = px + x - wlo;
          put_pair(pe + x, at >= 0 && at < wcnt ? woff + at : -1, at >= 1 && at <= wcnt ? woff + at - 1 : -1);
        }
      for (int x = lane; x < ln; x += 32)
        list[placed + x] = (unsigned)((base + lu + x - u) * pitch16) | (unsigned)(pe + lu + x - l0 - px) << 16;
    }
    placed += ln;
  }
  chunk.steps = (placed + 15) / 16;
  if (write)
    for (int x = placed + lane; x < 16 * chunk.steps; x += 32) list[x] = (unsigned)(R * pitch16) | (PK_DUMMY - 2u) << 16;
  if (last_take < last_len) {
    cur.seg += last;
    cur.at = last_skip + last_take;
  } else {
    cur.seg += pieces;
    cur.at = 0;
  }
  return chunk;
}

// The entry pair at place x: phase (stride E) x (cos x, cos x - 1, -sin x, -sin x - 1), bias x (bias x, bias x - 1) times log2 e,
// from entries i0 and i1 of the table; -1: outside the window, no weight.
template <int NCF>
__device__ __forceinline__ void pk_put_entries(const float* entries, int i0, int i1, float4* phase, float2* bias, int E, int x) {
  float e0[8], e1[8];
#pragma unroll
  for (int z = 0; z < 2; ++z) {
    float* e = z ? e1 : e0;
    const int i = z ? i1 : i0;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4* src = reinterpret_cast<const float4*>(entries + (size_t)(i < 0 ? 0 : i) * 8);
    const float4 v0 = i < 0 ? none : __ldg(src);
    e[0] = v0.x; e[1] = v0.y; e[2] = v0.z; e[3] = v0.w;
    if constexpr (NCF >= 2) {
      const float4 v1 = i < 0 ? none : __ldg(src + 1);
      e[4] = v1.x; e[5] = v1.y; e[6] = v1.z; e[7] = v1.w;
    }
    e[2 * NCF] = i < 0 ? -INFINITY : TC_LOG2E * e[2 * NCF];
  }
#pragma unroll
  for (int f = 0; f < NCF; ++f) phase[f * E + x] = make_float4(e0[2 * f], e1[2 * f], -e0[2 * f + 1], -e1[2 * f + 1]);
  bias[x] = make_float2(e0[2 * NCF], e1[2 * NCF]);
}

// ---- plans: what every longitude tile of a row tile has in common.  The packed lists follow from the windows and are worked out
// once per table; the entries are read in every launch (lattice_plan_refresh_kernel).
constexpr int PK_HEADER = 16;  // ints at the start of a chunk's record
enum { PK_HAS_ROWS = 0, PK_HAS_PAIRS = 1, PK_HAS_STEPS = 2, PK_ROW_TILE = 14, PK_READY = 15 };  // staged rows, entry pairs, every warp's steps; its row tile; refreshed
constexpr int pk_window_words(int W) { return 3 * PK_ROWS * (2 * W + 1); }  // count, first offset and first entry of a row tile's windows
// A record: header, staged rows (rows x 2 ints: first node of the neighbour row, longitude offset), entry pairs as in shared
// memory (before it is refreshed the pairs' indices are in the biases' place), lists (warp x rows), the windows it was made from
inline int pk_record_bytes(PkCaps caps, int warps, int W, int ncf) {
  return 4 * PK_HEADER + 8 * caps.rows + caps.entries * (16 * ncf + 8) + 4 * warps * caps.rows + 4 * pk_window_words(W);
}
struct PkRecord {
  int* header;
  int2* nodes;
  float4* phase;
  float2* bias;
  unsigned* list;
  __device__ __forceinline__ int2* pairs() const { return reinterpret_cast<int2*>(bias); }
  __device__ __forceinline__ int* windows(PkCaps caps, int warps) const { return reinterpret_cast<int*>(list + warps * caps.rows); }
};
// bytes: of a record
template <int NCF>
__device__ __forceinline__ PkRecord pk_record(const unsigned char* plan, int64_t index, int64_t bytes, PkCaps caps) {
  unsigned char* p = const_cast<unsigned char*>(plan) + index * bytes;
  unsigned char* phase = p + 4 * PK_HEADER + 8 * caps.rows;
  unsigned char* bias = phase + (size_t)16 * NCF * caps.entries;
  return PkRecord{reinterpret_cast<int*>(p), reinterpret_cast<int2*>(p + 4 * PK_HEADER), reinterpret_cast<float4*>(phase), reinterpret_cast<float2*>(bias),
                  reinterpret_cast<unsigned*>(bias + (size_t)8 * caps.entries)};
}
// Word x of the windows of a row tile (rows beyond the lattice's last: 0)
__device__ __forceinline__ int pk_window_word(const PkWindows& t, int row_tile, int x) {
  const int span = 2 * t.W + 1, kind = x / (PK_ROWS * span), at = row_tile * PK_ROWS * span + x - kind * PK_ROWS * span;
  if (at >= t.rows * span) return 0;
  return (kind == 0 ? t.win_cnt : kind == 1 ? t.win_lo : t.win_off)[at];
}

// A CTA per row tile.  records null: counts[tile] = its chunks; else its chunks' records from first[tile] on, not refreshed.
template <int NCF, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) lattice_plan_kernel(PkWindows t, PkCaps caps, int pitch16, int bytes, int* counts, const int* first,
                                                                  unsigned char* records) {
  __shared__ PkTile tile;
  const int r0 = blockIdx.x * PK_ROWS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = r0 + (warp & (PK_ROWS - 1));
  pk_open_tile<WARPS>(t, r0, tile);
  PkCursor cur{0, 0};
  int n = 0;
  do {
    PkRecord rec{};
    if (records) rec = pk_record<NCF>(records, first[blockIdx.x] + n, bytes, caps);
    const PkChunk chunk = pk_build<WARPS>(tile, cur, caps, pitch16, records != nullptr, row < t.rows, rec.list + (records ? warp * caps.rows : 0),
                                          [&](int r, int j, int u) { rec.nodes[r] = make_int2(j * t.nlon, tc_wrap(u, t.nlon)); },
                                          [&](int x, int i0, int i1) { rec.pairs()[x] = make_int2(i0, i1); });
    if (records) {
      if (threadIdx.x == 0) {
        rec.header[PK_HAS_ROWS] = chunk.rows;
        rec.header[PK_HAS_PAIRS] = chunk.entries;
        rec.header[PK_ROW_TILE] = blockIdx.x;
        rec.header[PK_READY] = 0;
      }
      if (lane == 0) rec.header[PK_HAS_STEPS + warp] = chunk.steps;
      if (threadIdx.x < PK_DUMMY) rec.pairs()[threadIdx.x] = make_int2(-1, -1);
      for (int x = threadIdx.x; x < pk_window_words(t.W); x += 32 * WARPS) rec.windows(caps, WARPS)[x] = pk_window_word(t, blockIdx.x, x);
    }
    ++n;
  } while (cur.seg < tile.n_seg);
  if (!records && threadIdx.x == 0) counts[blockIdx.x] = n;
}

// A CTA per record: the plan's record with the entries the table holds now; an empty one that is not ready where the row tile's
// windows are no longer those it was made from.  Runs in front of every pass that has a plan: a pass that kept a copy of the
// entries from call to call would not see a write into the table.
// Latency bound, so all that can is loaded at once: the entries do not wait for the windows (their indices are only kept below
// the table's end).
constexpr int PK_REFRESH_THREADS = 512;
template <int NCF>
__global__ void __launch_bounds__(PK_REFRESH_THREADS) lattice_plan_refresh_kernel(PkWindows t, const float* entries, int64_t n_entries, PkCaps caps, int warps,
                                                                                  int bytes, const unsigned char* plan, unsigned char* records) {
  const PkRecord from = pk_record<NCF>(plan, blockIdx.x, bytes, caps), to = pk_record<NCF>(records, blockIdx.x, bytes, caps);
  const int x0 = threadIdx.x, row_tile = __ldg(from.header + PK_ROW_TILE), n_pairs = __ldg(from.header + PK_HAS_PAIRS);
  const int2 first_pair = x0 < caps.entries ? __ldg(from.pairs() + x0) : make_int2(-1, -1);  // beyond n_pairs: whatever was there, not used
  uint4* const lists_to = reinterpret_cast<uint4*>(to.list);
  const uint4* const lists_from = reinterpret_cast<const uint4*>(from.list);
  for (int x = x0; x < caps.rows; x += PK_REFRESH_THREADS) to.nodes[x] = __ldg(from.nodes + x);
  for (int x = x0; x < warps * caps.rows / 4; x += PK_REFRESH_THREADS) lists_to[x] = __ldg(lists_from + x);
  int same = 1;
  for (int x = x0; x < pk_window_words(t.W); x += PK_REFRESH_THREADS) same &= __ldg(from.windows(caps, warps) + x) == pk_window_word(t, row_tile, x);
  for (int x = x0; x < n_pairs; x += PK_REFRESH_THREADS) {
    const int2 at = x == x0 ? first_pair : __ldg(from.pairs() + x);
    pk_put_entries<NCF>(entries, at.x < n_entries ? at.x : -1, at.y < n_entries ? at.y : -1, to.phase, to.bias, caps.entries, x);
  }
  same = __syncthreads_and(same);
  if (x0 < PK_HEADER) to.header[x0] = x0 == PK_READY ? same : same ? __ldg(from.header + x0) : 0;
}

template <int NCF>
__device__ __forceinline__ bool pk_ready(const TcArgs& a, int row_tile) {
  return pk_record<NCF>(a.records, a.plan_first[row_tile], a.record_bytes, a.caps).header[PK_READY] != 0;
}

// One tile of owners: PK_ROWS rows x TLON longitudes, (sample, head) pairs [bh, bh_end)
template <int KS0, int NCF, int KSC, int MODE, int WARPS, bool PLANNED>
__device__ __forceinline__ void pk_cta(const TcArgs& a, int row_tile, int lon_tile, int bh, int bh_end) {
  using L = PkLayout<KS0, NCF, KSC>;
  constexpr int THREADS = 32 * WARPS, TLON = 8 * (WARPS / PK_ROWS);
  constexpr int KQ = L::KQ, NCK = NCF * KSC, PITCH = L::PITCH, FIELD = L::FIELD;
  constexpr bool FWD = MODE == TC_FWD, PASS_S = MODE == TC_BWD_S;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ typename std::conditional<PLANNED, char, PkTile>::type tile_desc;
  __shared__ int member_s;
  const TcPlan& P = a.plan;
  const int R = a.caps.rows, E = a.caps.entries, LIST = R;
  unsigned char* const tile_s = smem;                                                   // (R + 1) rows, the last all zeros
  unsigned char* const phase_s = tile_s + (size_t)(R + 1) * PITCH;                      // NCF arrays of E x (cos x, cos x - 1, -sin x, -sin x - 1)
  float2* const bias_s = reinterpret_cast<float2*>(phase_s + (size_t)NCF * 16 * E);     // E x (bias x, bias x - 1), times log2 e
  unsigned* const list_s = reinterpret_cast<unsigned*>(bias_s + E);                     // per warp LIST x (row offset / 16 | entry << 16)
  int* const node_s = reinterpret_cast<int*>(list_s + WARPS * LIST);                    // R staged rows: node within the sample

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  int chunk = 0, n_chunks = 1;
  if constexpr (PLANNED) {
    chunk = a.plan_first[row_tile];
    n_chunks = a.plan_first[row_tile + 1] - chunk;
  }
  const int r0 = row_tile * PK_ROWS, c0 = lon_tile * TLON;
  const int my_row = warp & (PK_ROWS - 1), row = r0 + my_row, l0 = 8 * (warp / PK_ROWS);
  const float cscale = a.scale * TC_LOG2E;
  const bool words = a.words != 0;
  const bool even = a.even != 0;

  // ---- setup, once per CTA: which rows are asked for
  if (threadIdx.x == 0) member_s = a.n_order == a.rows ? (1 << PK_ROWS) - 1 : 0;
  for (int x = threadIdx.x; x < PITCH / 16; x += THREADS) reinterpret_cast<uint4*>(tile_s + (size_t)R * PITCH)[x] = make_uint4(0, 0, 0, 0);
  if (a.padded)  // padding columns are never copied: they must be zero
    for (int x = threadIdx.x; x < R * (PITCH / 16); x += THREADS) reinterpret_cast<uint4*>(tile_s)[x] = make_uint4(0, 0, 0, 0);
  if constexpr (!PLANNED)
    for (int x = threadIdx.x; x < PK_DUMMY; x += THREADS) {
      bias_s[x] = make_float2(-INFINITY, -INFINITY);
      for (int f = 0; f < NCF; ++f) reinterpret_cast<float4*>(phase_s)[f * E + x] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  __syncthreads();
  if (a.n_order != a.rows) {
    int mine = 0;
    for (int x = threadIdx.x; x < a.n_order; x += THREADS) {
      const int d = a.row_order[x] - r0;
      if (d >= 0 && d < PK_ROWS) mine |= 1 << d;
    }
    if (mine) atomicOr(&member_s, mine);
    __syncthreads();
  }
  if (member_s == 0) return;
  const bool active = (member_s >> my_row & 1) && row < a.rows && c0 + l0 < a.nlon;  // this warp has owners to write

  // ---- the chunks of the tile's neighbourhood: from the plan, or worked out here
  PkCursor cur{0, 0};
  if constexpr (!PLANNED) pk_open_tile<WARPS>(PkWindows{a.win_cnt, a.win_lo, a.win_off, a.rows, a.nlon, a.W}, r0, tile_desc);
  const int first_chunk = chunk;
  int n_rows = 0, n_steps = 0;
  // the next chunk (the first one again after the last): staged rows' nodes, entry pairs, lists; its copies join the fields'
  auto load_chunk = [&](bool restart) {
    if constexpr (PLANNED) {
      if (restart) chunk = first_chunk;
      const PkRecord rec = pk_record<NCF>(a.records, chunk, a.record_bytes, a.caps);
      n_rows = rec.header[PK_HAS_ROWS];
      const int n_entries = rec.header[PK_HAS_PAIRS];
      n_steps = active ? rec.header[PK_HAS_STEPS + warp] : 0;
      ++chunk;
      for (int r = threadIdx.x; r < n_rows; r += THREADS) {
        const int2 at = rec.nodes[r];
        const int lon = c0 + at.y;  // both below nlon
        node_s[r] = at.x + (lon >= a.nlon ? lon - a.nlon : lon);
      }
      float4* const phase = reinterpret_cast<float4*>(phase_s);
#pragma unroll
      for (int f = 0; f < NCF; ++f)
        for (int x = threadIdx.x; x < n_entries; x += THREADS) cp_async16(phase + f * E + x, rec.phase + f * E + x, 16);
      for (int x = threadIdx.x; 2 * x < n_entries; x += THREADS) cp_async16(bias_s + 2 * x, rec.bias + 2 * x, 16);
      for (int x = lane; x < 4 * n_steps; x += 32) cp_async16(list_s + warp * LIST + 4 * x, rec.list + warp * LIST + 4 * x, 16);
    } else {
      if (restart) cur = PkCursor{0, 0};
      const PkChunk built = pk_build<WARPS>(tile_desc, cur, a.caps, PITCH / 16, true, active, list_s + warp * LIST,
                                            [&](int r, int j, int u) { node_s[r] = j * a.nlon + tc_wrap(c0 + u, a.nlon); },
                                            [&](int x, int i0, int i1) { pk_put_entries<NCF>(a.entries, i0, i1, reinterpret_cast<float4*>(phase_s), bias_s, E, x); });
      n_rows = built.rows;
      n_steps = built.steps;
    }
  };
  auto more_chunks = [&]() {
    if constexpr (PLANNED) return chunk < first_chunk + n_chunks;
    else return cur.seg < tile_desc.n_seg;
  };

  // ---- staging: a thread keeps one unit (2 .. 16 bytes) of the head's columns and strides the staged rows
  const int units = a.units, per_pass = THREADS / units, st_row = threadIdx.x / units;
  int st_block, st_stride, st_dst;  // flat column of the unit for head 0, columns from head to head, byte in the staged field
  {
    const int u = (threadIdx.x - st_row * units) * a.unit;  // byte within the head's columns, unpadded
    if (u < 2 * P.a0) {
      st_block = P.real_off + u / 2;
      st_stride = P.a0;
      st_dst = u;
    } else {
      const int v = u - 2 * P.a0, f = v / (4 * P.ac), w = v - f * 4 * P.ac;
      st_block = P.cf_off[f < NCF ? f : 0] + w / 2;
      st_stride = 2 * P.ac;
      st_dst = 32 * KS0 + f * 32 * KSC + w;
    }
  }
  auto issue = [&](const PkPair& at_pair) {  // asynchronous copies of the chunk's rows of a (sample, head) pair
    const int h = at_pair.h;
    const int64_t node0 = at_pair.node0;
    if (st_row < per_pass) {
      const int64_t col = node0 * a.D + st_block + (int64_t)h * st_stride;
      const __nv_bfloat16 *s1 = a.nb1 + col, *s2 = a.nb2 + col;
      unsigned char* d = tile_s + st_dst + st_row * PITCH;
      if (a.unit == 16) {
        for (int r = st_row; r < n_rows; r += per_pass, d += per_pass * PITCH) {
          const int64_t at = (int64_t)node_s[r] * a.D;
          cp_async16(d, s1 + at, 16);
          cp_async16(d + FIELD, s2 + at, 16);
        }
      } else if (a.unit == 8) {
        for (int r = st_row; r < n_rows; r += per_pass, d += per_pass * PITCH) {
          const int64_t at = (int64_t)node_s[r] * a.D;
          cp_async_ca<8>(d, s1 + at);
          cp_async_ca<8>(d + FIELD, s2 + at);
        }
      } else if (a.unit == 4) {
        for (int r = st_row; r < n_rows; r += per_pass, d += per_pass * PITCH) {
          const int64_t at = (int64_t)node_s[r] * a.D;
          cp_async_ca<4>(d, s1 + at);
          cp_async_ca<4>(d + FIELD, s2 + at);
        }
      } else {  // odd columns: element by element
        for (int r = st_row; r < n_rows; r += per_pass, d += per_pass * PITCH) {
          const int64_t at = (int64_t)node_s[r] * a.D;
          *reinterpret_cast<__nv_bfloat16*>(d) = s1[at];
          *reinterpret_cast<__nv_bfloat16*>(d + FIELD) = s2[at];
        }
      }
    }
    if constexpr (PASS_S) {
      for (int r = threadIdx.x; r < n_rows; r += THREADS) {
        const int64_t at = (node0 + node_s[r]) * a.H + h;
        cp_async_ca<4>(tile_s + r * PITCH + 2 * FIELD, a.lse + at);
        cp_async_ca<4>(tile_s + r * PITCH + 2 * FIELD + 4, a.delta + at);
      }
    }
    cp_async_commit();
  };

  const int own_b = l0 + g;      // the owner whose column this thread holds in B fragments (and stores in the epilogue)
  const int own_c = l0 + 2 * c;  // the owners (own_c, own_c + 1) of this thread's accumulator columns
  const bool own_b_present = active && c0 + own_b < a.nlon;
  const unsigned tile_addr = (unsigned)__cvta_generic_to_shared(tile_s);
  const unsigned gram_lane = tile_addr + 16 * (lane >> 4), sum_lane = tile_addr + 16 * (lane >> 3 & 1);
  const int sum_pos = 8 * (lane >> 4) + (lane & 7);
  const unsigned char* const phase_lane = phase_s - 32 * c;
  const float2* const bias_lane = bias_s - 2 * c;
  const unsigned* const my_list = list_s + warp * LIST;
  const f32x2 cscale2 = pack2(cscale, cscale);

  load_chunk(true);
  const bool single = !more_chunks();  // the whole neighbourhood is one chunk: lists and entries serve every (sample, head)
  __syncthreads();
  // owners' fragments (B operands) and their pre-swapped copies:
  //   owners carry q: Im = sum_cols tile[col] * q'[col], q' = (-q_im, q_re);   owners carry k: k' = (k_im, -k_re)
  unsigned f1[KQ][2], s1[NCK][2], f2[FWD ? 1 : KQ][2], s2[FWD ? 1 : NCK][2], of[MODE == TC_BWD_T ? KQ : 1][2];
  float lse_o[2] = {0.f, 0.f}, dl_o[2] = {0.f, 0.f};  // pass T: the two accumulator-column owners' lse (base 2) and Delta
  const int lon_b = min(c0 + own_b, a.nlon - 1);      // an owner beyond the last longitude reads that one's; nothing of it is written
  auto fetch_owners = [&](const PkPair& at) {  // loads only; used by finish_owners
    if (!active) return;
    const int64_t base = (at.row0 + lon_b) * a.D;
    load_owner_columns<KS0, NCF, KSC>(P, a.own1 + base, even, words, at.h, c, f1);
    if constexpr (!FWD) load_owner_columns<KS0, NCF, KSC>(P, a.own2 + base, even, words, at.h, c, f2);
    if constexpr (MODE == TC_BWD_T) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t x = (at.row0 + min(c0 + own_c + e, a.nlon - 1)) * a.H + at.h;
        lse_o[e] = a.lse[x] * TC_LOG2E;
        if (a.delta_out == nullptr) dl_o[e] = a.delta[x];
      }
      if (a.delta_out != nullptr) load_owner_columns<KS0, NCF, KSC>(P, a.out_fwd + base, even, words, at.h, c, of);
    }
  };
  auto finish_owners = [&](const PkPair& at) {
    if (!active) return;
#pragma unroll
    for (int kc = 0; kc < NCK; ++kc)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        s1[kc][r] = PASS_S ? swap_neg(f1[KS0 + kc][r]) : swap_neg_lo(f1[KS0 + kc][r]);
        if constexpr (!FWD) s2[kc][r] = PASS_S ? swap_neg(f2[KS0 + kc][r]) : swap_neg_lo(f2[KS0 + kc][r]);
      }
    if constexpr (MODE == TC_BWD_T)
      if (a.delta_out != nullptr) {
        // Delta = <dO, O> over the head's columns of owner own_b: this thread holds 2 of every 8 columns of dO (f2) and O,
        // then the four lanes of the owner add up.  Written for the source-major pass, and handed to the lanes that hold
        // the owner as an accumulator column.
        float d = 0.f;
#pragma unroll
        for (int ks = 0; ks < KQ; ++ks)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            d = fmaf(__uint_as_float(f2[ks][r] << 16), __uint_as_float(of[ks][r] << 16), d);
            d = fmaf(__uint_as_float(f2[ks][r] & 0xffff0000u), __uint_as_float(of[ks][r] & 0xffff0000u), d);
          }
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        if (c == 0 && own_b_present) a.delta_out[(at.row0 + c0 + own_b) * a.H + at.h] = d;
#pragma unroll
        for (int e = 0; e < 2; ++e) dl_o[e] = __shfl_sync(0xffffffffu, d, (2 * c + e) << 2);
      }
  };
  // the (sample, head) pairs in turn, heads fastest
  PkPair pair{bh % a.H, ((int64_t)(bh / a.H) * a.rows + row) * a.nlon, (int64_t)(bh / a.H) * a.rows * a.nlon};
  auto following = [&](const PkPair& at) {
    const bool wrap = at.h + 1 == a.H;
    const int64_t sample = wrap ? (int64_t)a.rows * a.nlon : 0;
    return PkPair{wrap ? 0 : at.h + 1, at.row0 + sample, at.node0 + sample};
  };
  issue(pair);
  if constexpr (!PASS_S) fetch_owners(pair);
  for (;; ++bh) {
    if constexpr (PASS_S) fetch_owners(pair);
    finish_owners(pair);
    float a1_0[4] = {0.f, 0.f, 0.f, 0.f}, a1_r[NCK][4], a1_i[NCK][4];
    float a2_0[4] = {0.f, 0.f, 0.f, 0.f}, a2_r[PASS_S ? NCK : 1][4], a2_i[PASS_S ? NCK : 1][4];
#pragma unroll
    for (int m = 0; m < NCK; ++m)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        a1_r[m][x] = a1_i[m][x] = 0.f;
        if constexpr (PASS_S) a2_r[m][x] = a2_i[m][x] = 0.f;
      }
    float m_o[2] = {-1e30f, -1e30f}, l_o[2] = {0.f, 0.f};  // forward: reference maximum (base-2 logits), partial sums of the two owners

    for (;;) {
      cp_async_wait<0>();
      __syncthreads();
      // ---- this warp's steps: 16 packed positions each
      const unsigned* at = my_list;
      unsigned at_gram = at[lane & 15], at_sum = at[sum_pos], at_e0 = at[g], at_e1 = at[g + 8];
      for (int step = 0; step < n_steps; ++step) {
        const unsigned gram_addr = gram_lane + (at_gram & 0xffffu) * 16u, sum_addr = sum_lane + (at_sum & 0xffffu) * 16u;
        const unsigned w0 = at_e0, w1 = at_e1;
        at += 16;  // the next step's (behind the last one's: not used)
        at_gram = at[lane & 15];
        at_sum = at[sum_pos];
        at_e0 = at[g];
        at_e1 = at[g + 8];
        // element x of a fragment: packed position g + 8 (x >> 1), owner own_c + (x & 1)
        f32x2 tr[2][NCF], nti[2][NCF];  // cos, -sin of the elements (0, 1) and (2, 3)
        float2 bias[2];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const unsigned e = (y ? w1 : w0) >> 16;
#pragma unroll
          for (int f = 0; f < NCF; ++f) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(phase_lane + 16 * (f * E + e));
            tr[y][f] = t.x;
            nti[y][f] = t.y;
          }
          bias[y] = bias_lane[e];
        }
        float w[4], p[4];  // the weights the two accumulations use: forward p | pass T ds | pass S ds, p
        {
          float s0[4], sr[NCF][4], si[NCF][4];
          gram_step<KS0, NCF, KSC>(f1, s1, gram_addr, s0, sr, si);
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            f32x2 sum = pack2(s0[2 * y], s0[2 * y + 1]);
#pragma unroll
            for (int f = 0; f < NCF; ++f) {
              sum = fma2(tr[y][f], pack2(sr[f][2 * y], sr[f][2 * y + 1]), sum);
              sum = fma2(nti[y][f], pack2(si[f][2 * y], si[f][2 * y + 1]), sum);
            }
            sum = fma2(cscale2, sum, pack2(bias[y].x, bias[y].y));
            unpack2(sum, p[2 * y], p[2 * y + 1]);
          }
        }
        const bool ok[4] = {bias[0].x > -INFINITY, bias[0].y > -INFINITY, bias[1].x > -INFINITY, bias[1].y > -INFINITY};
        if constexpr (FWD) {
          // online softmax over the 16 positions.  The reference maximum of an owner only moves when the new maximum exceeds
          // it by more than 2^8 (weights stay below 256: exact in the normalised result); whether some owner's has to move
          // can be told from each thread's own four logits: most steps skip the column maxima as well as the rescaling
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (!ok[x]) p[x] = -INFINITY;  // outside the window, whatever the neighbour holds
          const bool grow = fmaxf(p[0], p[2]) > m_o[0] + 8.f || fmaxf(p[1], p[3]) > m_o[1] + 8.f;
          if (__any_sync(0xffffffffu, grow)) {
            float mx[2] = {fmaxf(p[0], p[2]), fmaxf(p[1], p[3])};
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) {
              mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], d));
              mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], d));
            }
            const float nm[2] = {mx[0] > m_o[0] + 8.f ? mx[0] : m_o[0], mx[1] > m_o[1] + 8.f ? mx[1] : m_o[1]};
            const float corr[2] = {fast_exp2(m_o[0] - nm[0]), fast_exp2(m_o[1] - nm[1])};
            m_o[0] = nm[0]; m_o[1] = nm[1];
            l_o[0] *= corr[0]; l_o[1] *= corr[1];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              a1_0[x] *= corr[x & 1];
#pragma unroll
              for (int m = 0; m < NCK; ++m) { a1_r[m][x] *= corr[x & 1]; a1_i[m][x] *= corr[x & 1]; }
            }
          }
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            w[x] = fast_exp2(p[x] - m_o[x & 1]);
            l_o[x & 1] += w[x];
          }
        } else {
          // p from the logits first (the (q, k) Gram blocks die here), then d alpha from the (dO, v) Gram blocks
          float delta[4];
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            float lse[2] = {lse_o[0], lse_o[1]};
            delta[2 * y] = dl_o[0];
            delta[2 * y + 1] = dl_o[1];
            if constexpr (PASS_S) {
              const float2 st = *reinterpret_cast<const float2*>(tile_s + ((y ? w1 : w0) & 0xffffu) * 16u + 2 * FIELD);
              lse[0] = lse[1] = st.x * TC_LOG2E;
              delta[2 * y] = delta[2 * y + 1] = st.y;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) p[2 * y + x] = ok[2 * y + x] ? fast_exp2(p[2 * y + x] - lse[x]) : 0.f;
          }
          float h0[4], hr[NCF][4], hi[NCF][4];
          gram_step<KS0, NCF, KSC>(f2, s2, gram_addr + FIELD, h0, hr, hi);
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            f32x2 dal = pack2(h0[2 * y], h0[2 * y + 1]);
#pragma unroll
            for (int f = 0; f < NCF; ++f) {
              dal = fma2(tr[y][f], pack2(hr[f][2 * y], hr[f][2 * y + 1]), dal);
              dal = fma2(nti[y][f], pack2(hi[f][2 * y], hi[f][2 * y + 1]), dal);
            }
            float d0, d1;
            unpack2(dal, d0, d1);
            w[2 * y] = a.scale * p[2 * y] * (d0 - delta[2 * y]);
            w[2 * y + 1] = a.scale * p[2 * y + 1] * (d1 - delta[2 * y + 1]);
          }
        }
        // B operands: the weights (x phase parts), transposed to (owner column, position rows)
        auto operands = [&](const float (&v)[4], unsigned (&x0)[2], unsigned (&xr)[NCF][2], unsigned (&xi)[NCF][2]) {
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const f32x2 v2 = pack2(v[2 * y], v[2 * y + 1]);
            x0[y] = movmatrix_trans(pack_bf16(v2));
#pragma unroll
            for (int f = 0; f < NCF; ++f) {
              xr[f][y] = movmatrix_trans(pack_bf16(mul2(v2, tr[y][f])));
              xi[f][y] = movmatrix_trans(pack_bf16(mul2(v2, nti[y][f])));
            }
          }
        };
        unsigned x0[2], xr[NCF][2], xi[NCF][2];
        operands(w, x0, xr, xi);
        if constexpr (FWD) {
          accumulate_step<KS0, NCF, KSC>(a1_0, a1_r, a1_i, x0, xr, xi, sum_addr + FIELD);  // out += (p tau) v
        } else {
          accumulate_step<KS0, NCF, KSC>(a1_0, a1_r, a1_i, x0, xr, xi, sum_addr);  // dq += (ds tau) k  |  dk += (ds conj tau) q
          if constexpr (PASS_S) {
            operands(p, x0, xr, xi);
            accumulate_step<KS0, NCF, KSC>(a2_0, a2_r, a2_i, x0, xr, xi, sum_addr + FIELD);  // dv += (p conj tau) dO
          }
        }
      }
      // ---- the next chunk, or the next pair's copies: under way while this pair's results are written
      const bool more = more_chunks();
      if (!more && bh + 1 >= bh_end) break;
      __syncthreads();  // everyone is done with the tile, the lists and the entries
      if (!single) {
        load_chunk(!more);
        __syncthreads();
      }
      if (more) {
        issue(pair);
      } else {
        issue(following(pair));
        break;
      }
    }
    const PkPair done = pair;
    if (bh + 1 < bh_end) {
      pair = following(pair);
      if constexpr (!PASS_S) fetch_owners(pair);  // (the source-major pass has no registers for them beside its results)
    }

    // ---- epilogue: normalise, combine the two phase accumulators (multiplication by +-i = pair swap across rows g, g ^ 1),
    // transpose in registers, store
    if (active) {
      float inv[2] = {1.f, 1.f};
      if constexpr (FWD) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int d = 4; d < 32; d <<= 1) l_o[e] += __shfl_xor_sync(0xffffffffu, l_o[e], d);
          inv[e] = l_o[e] > 0.f ? 1.f / l_o[e] : 0.f;
          if (g == 0 && c0 + own_c + e < a.nlon)
            a.lse_out[(done.row0 + c0 + own_c + e) * a.H + done.h] = l_o[e] > 0.f ? (m_o[e] + log2f(l_o[e])) * TC_LN2 : -INFINITY;
        }
      }
      const int64_t base = (done.row0 + c0 + own_b) * a.D;
      store_result<KS0, NCF, KSC, PASS_S>(P, a.res1 + base, own_b_present, even, words, done.h, g, c, inv, a1_0, a1_r, a1_i);
      if constexpr (PASS_S) store_result<KS0, NCF, KSC, true>(P, a.res2 + base, own_b_present, even, words, done.h, g, c, inv, a2_0, a2_r, a2_i);
    }
    if (bh + 1 >= bh_end) break;
  }
}

// The x-th row tile, from both ends on, that some row of a short list lies in; -1: there are not that many
constexpr int PK_LISTED_TILES = 8192;  // lattices with more row tiles have a grid for all of them
template <int THREADS>
__device__ __forceinline__ int pk_listed_tile(const int* row_order, int n_order, int row_tiles, int x, unsigned* bits) {
  const int words = (row_tiles + 31) / 32;
  for (int w = threadIdx.x; w < words; w += THREADS) bits[w] = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < n_order; k += THREADS) {
    const int row = row_order[k], tile = row / PK_ROWS;
    if (row < 0 || tile >= row_tiles) continue;
    const int place = 2 * tile < row_tiles ? 2 * tile : 2 * (row_tiles - 1 - tile) + 1;  // from_both_ends, the other way
    atomicOr(bits + place / 32, 1u << place % 32);
  }
  __syncthreads();
  int found = -1;
  for (int w = 0; w < words && found < 0; ++w) {
    const unsigned have = bits[w];
    const int n = __popc(have);
    if (x < n) found = 32 * w + (int)__fns(have, 0, x + 1);
    x -= n;
  }
  __syncthreads();  // the bits' place is used again
  return found < 0 ? -1 : (int)from_both_ends(found, row_tiles);
}

template <int KS0, int NCF, int KSC, int MODE, int WARPS, bool PLANNED>
__global__ void __launch_bounds__(32 * WARPS, pk_ctas(WARPS)) lattice_packed_kernel(const __grid_constant__ TcArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int TLON = 8 * (WARPS / PK_ROWS);
  // which tile, which (sample, head) pairs: the first heavy_ctas CTAs take the row tiles next to the poles
  const int lon_tiles = (a.nlon + TLON - 1) / TLON, row_tiles = (a.rows + PK_ROWS - 1) / PK_ROWS;
  int row_tile, lon_tile, bh, bh_end, x = blockIdx.x;
  if (x < a.heavy_ctas) {
    lon_tile = x % lon_tiles;
    x /= lon_tiles;
    const int chunks = (a.n_bh + a.heavy_bh - 1) / a.heavy_bh;
    bh = (x % chunks) * a.heavy_bh;
    bh_end = min(bh + a.heavy_bh, a.n_bh);
    row_tile = x / chunks;
  } else {
    x -= a.heavy_ctas;
    lon_tile = x % lon_tiles;
    x /= lon_tiles;
    const int light = a.slots - a.heavy_tiles;
    row_tile = a.heavy_tiles + x % light;
    bh = (x / light) * a.light_bh;
    bh_end = min(bh + a.light_bh, a.n_bh);
  }
  if (a.slots == row_tiles) {
    row_tile = (int)from_both_ends(row_tile, row_tiles);
  } else {
    row_tile = pk_listed_tile<32 * WARPS>(a.row_order, a.n_order, row_tiles, row_tile, reinterpret_cast<unsigned*>(smem));
    if (row_tile < 0) return;
  }
  pk_cta<KS0, NCF, KSC, MODE, WARPS, PLANNED>(a, row_tile, lon_tile, bh, bh_end);
}

// The row tiles whose windows are not the ones the plan was made from, behind the planned launch (to which their records were
// empty: it wrote zeros); none as a rule, which each of a few CTAs finds out for itself.
template <int KS0, int NCF, int KSC, int MODE, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, pk_ctas(WARPS)) lattice_packed_stale_kernel(const __grid_constant__ TcArgs a) {
  constexpr int TLON = 8 * (WARPS / PK_ROWS);
  const int lon_tiles = (a.nlon + TLON - 1) / TLON, row_tiles = (a.rows + PK_ROWS - 1) / PK_ROWS;
  int stale = 0;
  for (int x = threadIdx.x; x < row_tiles; x += 32 * WARPS) stale |= !pk_ready<NCF>(a, x);
  if (!__syncthreads_or(stale)) return;
  for (int row_tile = 0; row_tile < row_tiles; ++row_tile) {
    if (pk_ready<NCF>(a, row_tile)) continue;
    for (int64_t x = blockIdx.x; x < (int64_t)lon_tiles * a.n_bh; x += gridDim.x) {
      const int bh = (int)(x / lon_tiles);
      pk_cta<KS0, NCF, KSC, MODE, WARPS, false>(a, row_tile, (int)(x % lon_tiles), bh, bh + 1);
      __syncthreads();
    }
  }
}

// Delta[node, h] = <dO, O> over the head's columns
__global__ void tc_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out, float* __restrict__ delta,
                                int64_t n_nodes, int D, int H, TcPlan P) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= n_nodes * H) return;
  const int64_t node = w / H;
  const int h = (int)(w % H);
  float acc = 0.f;
  for (int x = lane; x < P.a0; x += 32) {
    const int64_t gidx = node * D + P.real_off + h * P.a0 + x;
    acc += __bfloat162float(dout[gidx]) * __bfloat162float(out[gidx]);
  }
  for (int f = 0; f < P.n_cf; ++f)
    for (int x = lane; x < 2 * P.ac; x += 32) {
      const int64_t gidx = node * D + P.cf_off[f] + 2 * h * P.ac + x;
      acc += __bfloat162float(dout[gidx]) * __bfloat162float(out[gidx]);
    }
  acc = warp_sum(acc);
  if (lane == 0) delta[node * H + h] = acc;
}

// Same, one warp per node with 16-byte loads: every 8-column chunk of the row belongs to one head (host-checked).
__global__ void tc_delta_vec_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out, float* __restrict__ delta,
                                    int64_t n_nodes, int D, int H, TcPlan P) {
  const int lane = threadIdx.x & 31;
  const int64_t node = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (node >= n_nodes) return;
  float part[2] = {0.f, 0.f};
  int head[2] = {-1, -1};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int col = 8 * (lane + 32 * r);
    if (col >= D) continue;
    if (P.a0 > 0 && col >= P.real_off && col < P.real_off + H * P.a0) head[r] = (col - P.real_off) / P.a0;
    for (int f = 0; f < P.n_cf; ++f)
      if (col >= P.cf_off[f] && col < P.cf_off[f] + 2 * H * P.ac) head[r] = (col - P.cf_off[f]) / (2 * P.ac);
    if (head[r] < 0) continue;
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(dout + node * D + col));
    const uint4 b = __ldg(reinterpret_cast<const uint4*>(out + node * D + col));
    const unsigned wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int x = 0; x < 4; ++x)
      part[r] += __uint_as_float(wa[x] << 16) * __uint_as_float(wb[x] << 16) + __uint_as_float(wa[x] & 0xffff0000u) * __uint_as_float(wb[x] & 0xffff0000u);
  }
  for (int h = 0; h < H; ++h) {
    const float v = warp_sum((head[0] == h ? part[0] : 0.f) + (head[1] == h ? part[1] : 0.f));
    if (lane == 0) delta[node * H + h] = v;
  }
}

int make_tc_plan(const int64_t* desc_host, int F, int H, int D, TcPlan& P) {
  P = TcPlan{};
  GM_REQUIRE(F >= 1 && F <= TC_MAX_CF + 1, GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): at most %d frequencies", TC_MAX_CF + 1);
  for (int f = 0; f < F; ++f) {
    const int n = (int)desc_host[5 * f], a_n = (int)desc_host[5 * f + 1], off = (int)desc_host[5 * f + 2];
    const int dim = n == 0 ? 1 : 2;
    GM_REQUIRE(n >= 0 && a_n >= 1 && off >= 0 && off + H * a_n * dim <= D, GM_ERR_ARGUMENT,
               "gm_lattice_attention: descriptor row %d leaves the width D=%d", f, D);
    if (n == 0) {
      GM_REQUIRE(P.a0 == 0 && a_n <= 16, GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): one scalar block of at most 16 copies");
      P.a0 = a_n;
      P.real_off = off;
    } else {
      GM_REQUIRE(P.n_cf < TC_MAX_CF && a_n <= 16 && (P.ac == 0 || P.ac == a_n), GM_ERR_UNSUPPORTED,
                 "gm_lattice_attention (tensor cores): at most %d complex frequencies of one multiplicity <= 16", TC_MAX_CF);
      P.ac = a_n;
      P.cf_off[P.n_cf] = off;
      P.cf_order[P.n_cf] = n;
      ++P.n_cf;
    }
  }
  return GM_OK;
}

// Staged rows and entry pairs of a tile whose windows are as narrow as this lattice's get (its equator), from the halo W
// alone: a neighbourhood of W + 1/2 rows' radius, longitudes scaled by the lattice's aspect.
void narrow_tile(int rows_of, int nlon, int W, int tile_lons, int& rows, int& entries) {
  const double aspect = nlon / (2.0 * rows_of);
  rows = entries = 0;
  for (int s = -W; s < W + PK_ROWS; ++s) {
    int widest = 0;
    for (int i = 0; i < PK_ROWS; ++i) {
      const int d = s > i ? s - i : i - s;
      if (d > W) continue;
      const double chord = sqrt((W + 0.5) * (W + 0.5) - (double)d * d) * aspect;
      const int cnt = (int)fmin(2.0 * floor(chord) + 1.0, (double)nlon);
      widest = cnt > widest ? cnt : widest;
      entries += cnt + 13;
    }
    rows += widest + tile_lons - 1;
  }
}

// Shared memory of a chunk: room for the narrow tiles' whole neighbourhood (lists and entries then serve every (sample,
// head) pair of a CTA) with a margin for wider ones, for as many CTAs per SM as that allows.
template <int KS0, int NCF, int KSC, int WARPS>
size_t chunk_caps(int rows_of, int nlon, int W, PkCaps& caps) {
  using L = PkLayout<KS0, NCF, KSC>;
  constexpr int TLON = 8 * (WARPS / PK_ROWS);
  int want_rows, want_entries;
  narrow_tile(rows_of, nlon, W, TLON, want_rows, want_entries);
  const size_t per_row = L::PITCH + 4 * WARPS + 4, per_entry = L::ENTRY;
  const double ratio = (double)want_entries / want_rows;
  for (int ctas = pk_ctas(WARPS);; --ctas) {
    const size_t budget = 227 * 1024 / ctas - 4096;  // the system's 1 KB and the static arrays
    const size_t fixed = 2 * L::PITCH + 64 * WARPS + 16 * PK_DUMMY * NCF + 1024 + 4 * (TLON + 8) * per_entry;
    int rows = (int)((budget - fixed) / (per_row + ratio * per_entry));
    if (rows < want_rows && ctas > 2) continue;
    rows = rows < want_rows * 2 ? rows : want_rows * 2;
    rows = rows < 32 ? 32 : rows;
    caps.rows = rows / 16 * 16;
    caps.entries = (int)(ratio * caps.rows) / 8 * 8 + 4 * (TLON + 8) + PK_DUMMY;
    return (size_t)(caps.rows + 1) * L::PITCH + (size_t)caps.entries * L::ENTRY + (size_t)(WARPS + 1) * caps.rows * 4;
  }
}

template <int KS0, int NCF, int KSC, int MODE>
int launch_tn(TcArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream) {
  constexpr int WARPS = pk_warps(MODE), TLON = 8 * (WARPS / PK_ROWS);
  const void* ptrs[6] = {a.own1, a.own2, a.nb1, a.nb2, a.res1, a.res2};
  uint64_t all = (uint64_t)a.D * 2;  // in bytes
  for (const void* q : ptrs) all |= reinterpret_cast<uintptr_t>(q);
  if (MODE == TC_BWD_T && a.delta_out) all |= reinterpret_cast<uintptr_t>(a.out_fwd);
  a.words = all % 4 == 0;
  all |= (uint64_t)a.plan.a0 * 2 | (KS0 ? (uint64_t)a.plan.real_off * 2 : 0);
  for (int f = 0; f < a.plan.n_cf; ++f) all |= (uint64_t)a.plan.cf_off[f] * 2;
  a.even = all % 4 == 0;
  a.padded = (KS0 && a.plan.a0 != 16) || 2 * a.plan.ac != 16 * KSC;
  // the widest copy that every block of every head is made of: all that is added to the fields' addresses, in bytes
  uint64_t bits = reinterpret_cast<uintptr_t>(a.nb1) | reinterpret_cast<uintptr_t>(a.nb2) | (uint64_t)a.D * 2 | (uint64_t)a.plan.a0 * 2 |
                  (uint64_t)a.plan.ac * 4 | (KS0 ? (uint64_t)a.plan.real_off * 2 : 0);
  for (int f = 0; f < a.plan.n_cf; ++f) bits |= (uint64_t)a.plan.cf_off[f] * 2;
  a.unit = 16;
  while (a.unit > 2 && bits % a.unit) a.unit /= 2;
  a.units = (2 * a.plan.a0 + NCF * 4 * a.plan.ac) / a.unit;
  a.n_order = n_order_rows;
  const size_t smem = chunk_caps<KS0, NCF, KSC, WARPS>(a.rows, a.nlon, a.W, a.caps);
  a.record_bytes = pk_record_bytes(a.caps, WARPS, a.W, NCF);
  // Polar rows see whole rings: their tiles start first and hold few (sample, head) pairs each.  Elsewhere a CTA takes as
  // many pairs as leave a few waves of CTAs, up to 16: lists and entries are made once for all of them.  Pass T, us, with
  // 6 waves (24 and at most 2 pairs next to the poles) / 4 (12, 4) / 4 (8, 4) / 2 (12, 2): 128 x 256, batch 4, 8 x (m <= 3) 587 / 560 / 552 / 605;
  // 91 x 180, batch 3, 16 x (m <= 2) 218 / 206 / 206 / 208; 100 x 200, batch 5, 8 heads 681 / 666 / 667 / 700; 200 x 100, batch 4 237 / 239 / 239 / 239;
  // 256 x 512, batch 8 4 645 / 4 648 / 4 660 / 4 647; its upper half alone, batch 1, where the polar CTAs' four pairs in turn are the
  // launch, 351 / 349 / 405; forward at 180 x 360, batch 2 491 / 499 / 493 / 509.
  const int64_t lon_tiles = (a.nlon + TLON - 1) / TLON, row_tiles = (a.rows + PK_ROWS - 1) / PK_ROWS;
  const int64_t n_bh = (int64_t)a.H * batch, slots = (int64_t)sm_count() * pk_ctas(WARPS);
  GM_REQUIRE(n_bh < (1ll << 31), GM_ERR_LIMIT, "gm_lattice_attention (tensor cores): too many (sample, head) pairs");
  // a list of a few rows (a band's next to its halo): CTAs for the tiles it can touch.  256 x 512, batch 2, 4 heads of 16 x (m <= 2),
  // three rows, forward / pass T / pass S: 25 / 45 / 45 us (CTAs for all tiles, most of them idle:
  // 59 / 99 / 125)
  const int64_t listed = n_order_rows < row_tiles && row_tiles <= PK_LISTED_TILES ? n_order_rows : row_tiles;
  a.slots = (int)listed;
  int64_t heavy_tiles = 2 * ((2 * a.W + 2 + PK_ROWS - 1) / PK_ROWS);
  if (heavy_tiles > listed) heavy_tiles = listed;
  const int64_t light_tiles = (listed - heavy_tiles) * lon_tiles;
  const int64_t busy_tiles = std::min<int64_t>(listed, (n_order_rows + PK_ROWS - 1) / PK_ROWS) * lon_tiles;  // of a longer list: about as many have work
  auto pairs_per_cta = [&](int64_t tiles, int64_t waves, int64_t most) {
    int64_t n = tiles * n_bh / (slots * waves);
    n = n < 1 ? 1 : n > most ? most : n;
    const int64_t chunks = (n_bh + n - 1) / n;
    return (int)((n_bh + chunks - 1) / chunks);
  };
  a.n_bh = (int)n_bh;
  a.light_bh = pairs_per_cta(std::min(light_tiles, busy_tiles), 4, 16);
  a.heavy_bh = pairs_per_cta(busy_tiles, 12, 4);
  a.heavy_tiles = (int)heavy_tiles;
  const int64_t heavy = heavy_tiles * lon_tiles * ((n_bh + a.heavy_bh - 1) / a.heavy_bh);
  const int64_t light = light_tiles * ((n_bh + a.light_bh - 1) / a.light_bh);
  GM_REQUIRE(heavy + light < (1ll << 31), GM_ERR_LIMIT, "gm_lattice_attention (tensor cores): %lld tiles exceed a grid", (long long)(heavy + light));
  a.heavy_ctas = (int)heavy;
  auto go = [&](auto kernel, int64_t ctas) {
    const int st = allow_smem(kernel, smem, "gm_lattice_attention (tensor cores)");
    if (st != GM_OK) return st;
    kernel<<<(unsigned)ctas, 32 * WARPS, smem, stream>>>(a);
    return launch_status("gm_lattice_attention (tensor cores)");
  };
  if (!a.records) return go(lattice_packed_kernel<KS0, NCF, KSC, MODE, WARPS, false>, heavy + light);
  const int st = go(lattice_packed_kernel<KS0, NCF, KSC, MODE, WARPS, true>, heavy + light);
  return st != GM_OK ? st : go(lattice_packed_stale_kernel<KS0, NCF, KSC, MODE, WARPS>, std::min<int64_t>(slots, heavy + light));
}

// f(KS0, NCF, KSC) as integral constants for the layouts that have kernels
template <typename F>
int for_layout(const TcPlan& plan, int NORD, const F& f) {
  const int ks0 = plan.a0 > 0 ? 1 : 0, ksc = plan.ac > 8 ? 2 : 1, ncf = plan.n_cf;
  for (int x = 0; x < ncf; ++x)
    GM_REQUIRE(plan.cf_order[x] == x + 1, GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): complex frequencies must be the orders 1 .. %d", ncf);
  GM_REQUIRE(NORD == ncf, GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): the tables must hold exactly the orders 1 .. %d (they hold %d)", ncf, NORD);
  using std::integral_constant;
  auto with = [&](auto a, auto b, auto c) { return f(a, b, c); };
#define GM_LAYOUT(A, B, C) \
  if (ks0 == A && ncf == B && ksc == C) return with(integral_constant<int, A>(), integral_constant<int, B>(), integral_constant<int, C>());
  GM_LAYOUT(1, 2, 2)
  GM_LAYOUT(1, 2, 1)
  GM_LAYOUT(1, 3, 1)
  GM_LAYOUT(1, 1, 2)
  GM_LAYOUT(1, 1, 1)
  GM_LAYOUT(0, 2, 1)
#undef GM_LAYOUT
  return fail(GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): no kernel for this head layout (a0=%d, %d x %d complex)", plan.a0, ncf, plan.ac);
}

template <int MODE>
int dispatch_tc(TcArgs& a, int n_order_rows, int64_t batch, cudaStream_t cs) {
  return for_layout(a.plan, a.NORD, [&](auto ks0, auto ncf, auto ksc) { return launch_tn<ks0.value, ncf.value, ksc.value, MODE>(a, n_order_rows, batch, cs); });
}

int fill_tc_args(TcArgs& a, const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H, int W, int ES, int NORD,
                 double scale) {
  GM_REQUIRE(rows >= 1 && nlon >= 1 && batch >= 1 && D >= 1 && H >= 1 && H <= 65535 && batch <= 65535, GM_ERR_ARGUMENT,
             "gm_lattice_attention (tensor cores): bad sizes");
  GM_REQUIRE(W >= 0 && NORD >= 0, GM_ERR_ARGUMENT, "gm_lattice_attention (tensor cores): bad table sizes");
  GM_REQUIRE(2 * W + 1 <= TC_MAX_WIN, GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): neighbourhoods span more than %d lattice rows", TC_MAX_WIN);
  GM_REQUIRE(ES == 8 && 2 * NORD + 1 <= 8, GM_ERR_UNSUPPORTED, "gm_lattice_attention (tensor cores): entries must be 8 floats wide (orders <= 3)");
  GM_REQUIRE(desc_host, GM_ERR_ARGUMENT, "gm_lattice_attention (tensor cores): null descriptor");
  int status = make_tc_plan(desc_host, F, H, D, a.plan);
  if (status != GM_OK) return status;
  for (int f = 0; f < a.plan.n_cf; ++f)
    GM_REQUIRE(a.plan.cf_order[f] <= NORD, GM_ERR_ARGUMENT, "gm_lattice_attention (tensor cores): tables hold %d orders", NORD);
  a.rows = rows; a.nlon = nlon; a.D = D; a.H = H; a.W = W; a.NORD = NORD; a.scale = (float)scale;
  return GM_OK;
}

}  // namespace
}  // namespace gmb

using namespace gmb;

// ---- plans.  gm_lattice_plan_size: bytes of one record and the number of row tiles; _count: chunks per row tile; _fill: the
// records, row tile x's from first[x] on (first: the running sum of the counts, row tiles + 1 numbers).
extern "C" int gm_lattice_plan_size(const int64_t* desc_host, int F, int rows, int nlon, int D, int H, int W, int NORD, int mode,
                                    int64_t* record_bytes, int64_t* row_tiles) {
  GM_REQUIRE(record_bytes && row_tiles, GM_ERR_ARGUMENT, "gm_lattice_plan_size: null pointer");
  TcArgs a{};
  int status = fill_tc_args(a, desc_host, F, rows, nlon, 1, D, H, W, 8, NORD, 1.0);
  if (status != GM_OK) return status;
  *row_tiles = (rows + PK_ROWS - 1) / PK_ROWS;
  return for_layout(a.plan, NORD, [&](auto ks0, auto ncf, auto ksc) {
    auto size = [&](auto warps) {
      PkCaps caps;
      chunk_caps<ks0.value, ncf.value, ksc.value, warps.value>(rows, nlon, W, caps);
      *record_bytes = pk_record_bytes(caps, warps.value, W, ncf.value);
      return (int)GM_OK;
    };
    return mode == TC_FWD ? size(std::integral_constant<int, pk_warps(TC_FWD)>()) : size(std::integral_constant<int, pk_warps(TC_BWD_S)>());
  });
}

extern "C" int gm_lattice_plan_build(const int* win_cnt, const int* win_lo, const int* win_off, const float* entries, const int64_t* desc_host, int F,
                                     int rows, int nlon, int D, int H, int W, int NORD, int mode, int* counts, const int* first, void* records, void* stream) {
  GM_REQUIRE(win_cnt && win_lo && win_off && entries && (records ? first != nullptr : counts != nullptr), GM_ERR_ARGUMENT, "gm_lattice_plan_build: null pointer");
  TcArgs a{};
  int status = fill_tc_args(a, desc_host, F, rows, nlon, 1, D, H, W, 8, NORD, 1.0);
  if (status != GM_OK) return status;
  return for_layout(a.plan, NORD, [&](auto ks0, auto ncf, auto ksc) {
    auto build = [&](auto warps) {
      PkCaps caps;
      chunk_caps<ks0.value, ncf.value, ksc.value, warps.value>(rows, nlon, W, caps);
      const PkWindows t{win_cnt, win_lo, win_off, rows, nlon, W};
      lattice_plan_kernel<ncf.value, warps.value><<<(unsigned)((rows + PK_ROWS - 1) / PK_ROWS), 32 * warps.value, 0, (cudaStream_t)stream>>>(
          t, caps, PkLayout<ks0.value, ncf.value, ksc.value>::PITCH / 16, pk_record_bytes(caps, warps.value, W, ncf.value), counts, first, (unsigned char*)records);
      return launch_status("gm_lattice_plan_build");
    };
    return mode == TC_FWD ? build(std::integral_constant<int, pk_warps(TC_FWD)>()) : build(std::integral_constant<int, pk_warps(TC_BWD_S)>());
  });
}

extern "C" int gm_lattice_plan_refresh(const int* win_cnt, const int* win_lo, const int* win_off, const float* entries, const int64_t* desc_host, int F,
                                       int rows, int nlon, int D, int H, int W, int NORD, int mode, int64_t n_entries, const void* plan,
                                       int64_t n_records, void* records, void* stream) {
  GM_REQUIRE(win_cnt && win_lo && win_off && entries && plan && records, GM_ERR_ARGUMENT, "gm_lattice_plan_refresh: null pointer");
  GM_REQUIRE(n_entries >= 1, GM_ERR_ARGUMENT, "gm_lattice_plan_refresh: empty table");
  GM_REQUIRE(n_records >= 1 && n_records < (1ll << 31) && (reinterpret_cast<uintptr_t>(plan) | reinterpret_cast<uintptr_t>(records)) % 16 == 0, GM_ERR_ARGUMENT,
             "gm_lattice_plan_refresh: bad records");
  TcArgs a{};
  int status = fill_tc_args(a, desc_host, F, rows, nlon, 1, D, H, W, 8, NORD, 1.0);
  if (status != GM_OK) return status;
  return for_layout(a.plan, NORD, [&](auto ks0, auto ncf, auto ksc) {
    auto refresh = [&](auto warps) {
      PkCaps caps;
      chunk_caps<ks0.value, ncf.value, ksc.value, warps.value>(rows, nlon, W, caps);
      lattice_plan_refresh_kernel<ncf.value><<<(unsigned)n_records, PK_REFRESH_THREADS, 0, (cudaStream_t)stream>>>(
          PkWindows{win_cnt, win_lo, win_off, rows, nlon, W}, entries, n_entries, caps, warps.value, pk_record_bytes(caps, warps.value, W, ncf.value), (const unsigned char*)plan, (unsigned char*)records);
      return launch_status("gm_lattice_plan_refresh");
    };
    return mode == TC_FWD ? refresh(std::integral_constant<int, pk_warps(TC_FWD)>()) : refresh(std::integral_constant<int, pk_warps(TC_BWD_S)>());
  });
}

extern "C" int gm_lattice_attention_forward_planned(const void* q, const void* k, const void* v, const int* win_cnt, const int* win_lo,
                                               const int* win_off, const float* entries, const int* row_order, int n_order_rows,
                                               const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H, int W,
                                               int ES, int NORD, double scale, const int* plan_first, const void* plan_records, void* out, float* lse,
                                               void* stream) {
  using B = __nv_bfloat16;
  TcArgs a{};
  GM_REQUIRE(!plan_records || (plan_first && reinterpret_cast<uintptr_t>(plan_records) % 16 == 0), GM_ERR_ARGUMENT, "gm_lattice_attention_forward_planned: bad plan");
  a.plan_first = plan_first; a.records = (const unsigned char*)plan_records;
  int status = fill_tc_args(a, desc_host, F, rows, nlon, batch, D, H, W, ES, NORD, scale);
  if (status != GM_OK) return status;
  GM_REQUIRE(q && k && v && win_cnt && win_lo && win_off && entries && row_order && out && lse, GM_ERR_ARGUMENT,
             "gm_lattice_attention_forward_tc: null pointer");
  if (n_order_rows == 0) return GM_OK;
  a.own1 = (const B*)q; a.nb1 = (const B*)k; a.nb2 = (const B*)v; a.res1 = (B*)out; a.lse_out = lse;
  a.win_cnt = win_cnt; a.win_lo = win_lo; a.win_off = win_off; a.entries = entries; a.row_order = row_order;
  return dispatch_tc<TC_FWD>(a, n_order_rows, batch, (cudaStream_t)stream);
}

extern "C" int gm_lattice_attention_forward_tc(const void* q, const void* k, const void* v, const int* win_cnt, const int* win_lo,
                                               const int* win_off, const float* entries, const int* row_order, int n_order_rows,
                                               const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H, int W,
                                               int ES, int NORD, double scale, void* out, float* lse, void* stream) {
  return gm_lattice_attention_forward_planned(q, k, v, win_cnt, win_lo, win_off, entries, row_order, n_order_rows, desc_host, F, rows, nlon, batch, D, H,
                                              W, ES, NORD, scale, nullptr, nullptr, out, lse, stream);
}

extern "C" int gm_lattice_attention_backward_tc_passes(const void* dout, const void* q, const void* k, const void* v, const void* out,
                                                       const float* lse, const int* win_cnt, const int* win_lo, const int* win_off,
                                                       const float* entries, const int* row_order, int n_order_rows,
                                                       const int* t_win_cnt, const int* t_win_lo, const int* t_win_off,
                                                       const float* t_entries, const int* t_row_order, int t_n_order_rows,
                                                       const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H,
                                                       int W, int ES, int NORD, double scale, void* dq, void* dk, void* dv, float* delta,
                                                       int passes, void* stream);

extern "C" int gm_lattice_attention_backward_tc(const void* dout, const void* q, const void* k, const void* v, const void* out,
                                                const float* lse, const int* win_cnt, const int* win_lo, const int* win_off,
                                                const float* entries, const int* row_order, int n_order_rows, const int* t_win_cnt,
                                                const int* t_win_lo, const int* t_win_off, const float* t_entries,
                                                const int* t_row_order, int t_n_order_rows, const int64_t* desc_host, int F, int rows,
                                                int nlon, int64_t batch, int D, int H, int W, int ES, int NORD, double scale, void* dq,
                                                void* dk, void* dv, float* delta, void* stream) {
  return gm_lattice_attention_backward_tc_passes(dout, q, k, v, out, lse, win_cnt, win_lo, win_off, entries, row_order, n_order_rows,
                                                 t_win_cnt, t_win_lo, t_win_off, t_entries, t_row_order, t_n_order_rows, desc_host, F, rows,
                                                 nlon, batch, D, H, W, ES, NORD, scale, dq, dk, dv, delta, 7, stream);
}

// passes: bit 0 = Delta, bit 1 = the target-major pass (dq), bit 2 = the source-major pass (dk, dv).  Running a
// subset is for timing the passes separately.  Bits 0 and 1 together: pass T forms Delta itself; without bit 0 the
// passes read the Delta an earlier call left in `delta`.
extern "C" int gm_lattice_attention_backward_planned(const void* dout, const void* q, const void* k, const void* v, const void* out,
                                                       const float* lse, const int* win_cnt, const int* win_lo, const int* win_off,
                                                       const float* entries, const int* row_order, int n_order_rows,
                                                       const int* t_win_cnt, const int* t_win_lo, const int* t_win_off,
                                                       const float* t_entries, const int* t_row_order, int t_n_order_rows,
                                                       const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H,
                                                       int W, int ES, int NORD, double scale, void* dq, void* dk, void* dv, float* delta,
                                                       int passes, const int* plan_first, const void* plan_records,
                                                       const int* t_plan_first, const void* t_plan_records, void* stream) {
  using B = __nv_bfloat16;
  cudaStream_t cs = (cudaStream_t)stream;
  TcArgs a{};
  int status = fill_tc_args(a, desc_host, F, rows, nlon, batch, D, H, W, ES, NORD, scale);
  if (status != GM_OK) return status;
  GM_REQUIRE(dout && q && k && v && out && lse && win_cnt && win_lo && win_off && entries && row_order && t_win_cnt && t_win_lo &&
                 t_win_off && t_entries && t_row_order && dq && dk && dv && delta,
             GM_ERR_ARGUMENT, "gm_lattice_attention_backward_tc: null pointer");
  GM_REQUIRE((!plan_records || (plan_first && reinterpret_cast<uintptr_t>(plan_records) % 16 == 0)) &&
                 (!t_plan_records || (t_plan_first && reinterpret_cast<uintptr_t>(t_plan_records) % 16 == 0)),
             GM_ERR_ARGUMENT, "gm_lattice_attention_backward_planned: bad plan");
  const int64_t n_nodes = batch * rows * (int64_t)nlon;
  bool chunked = D % 8 == 0 && D <= 512 && a.plan.a0 % 8 == 0 && (2 * a.plan.ac) % 8 == 0 && a.plan.real_off % 8 == 0 &&
                 reinterpret_cast<uintptr_t>(dout) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
  for (int f = 0; f < a.plan.n_cf; ++f) chunked = chunked && a.plan.cf_off[f] % 8 == 0;
  // Delta = <dO, O>: formed inside the target-major pass when that pass runs in this call; by its own kernel otherwise
  const bool fused_delta = (passes & 2) != 0 && n_order_rows > 0;
  if (!(passes & 1) || fused_delta) {
  } else if (chunked)
    tc_delta_vec_kernel<<<(unsigned)((n_nodes + 7) / 8), 256, 0, cs>>>((const B*)dout, (const B*)out, delta, n_nodes, D, H, a.plan);
  else
    tc_delta_kernel<<<(unsigned)((n_nodes * H + 7) / 8), 256, 0, cs>>>((const B*)dout, (const B*)out, delta, n_nodes, D, H, a.plan);
  status = launch_status("gm_lattice_attention_backward_tc (delta)");
  if (status != GM_OK) return status;
  a.lse = lse; a.delta = delta;
  if (n_order_rows > 0 && (passes & 2)) {
    a.own1 = (const B*)q; a.own2 = (const B*)dout; a.nb1 = (const B*)k; a.nb2 = (const B*)v; a.res1 = (B*)dq; a.res2 = nullptr;
    a.out_fwd = (const B*)out; a.delta_out = (passes & 1) ? delta : nullptr;
    a.win_cnt = win_cnt; a.win_lo = win_lo; a.win_off = win_off; a.entries = entries; a.row_order = row_order;
    a.plan_first = plan_first; a.records = (const unsigned char*)plan_records;
    status = dispatch_tc<TC_BWD_T>(a, n_order_rows, batch, cs);
    if (status != GM_OK) return status;
  }
  if (t_n_order_rows > 0 && (passes & 4)) {
    a.own1 = (const B*)k; a.own2 = (const B*)v; a.nb1 = (const B*)q; a.nb2 = (const B*)dout; a.res1 = (B*)dk; a.res2 = (B*)dv;
    a.out_fwd = nullptr; a.delta_out = nullptr;
    a.win_cnt = t_win_cnt; a.win_lo = t_win_lo; a.win_off = t_win_off; a.entries = t_entries; a.row_order = t_row_order;
    a.plan_first = t_plan_first; a.records = (const unsigned char*)t_plan_records;
    status = dispatch_tc<TC_BWD_S>(a, t_n_order_rows, batch, cs);
  }
  return status;
}

extern "C" int gm_lattice_attention_backward_tc_passes(const void* dout, const void* q, const void* k, const void* v, const void* out,
                                                       const float* lse, const int* win_cnt, const int* win_lo, const int* win_off,
                                                       const float* entries, const int* row_order, int n_order_rows,
                                                       const int* t_win_cnt, const int* t_win_lo, const int* t_win_off,
                                                       const float* t_entries, const int* t_row_order, int t_n_order_rows,
                                                       const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H,
                                                       int W, int ES, int NORD, double scale, void* dq, void* dk, void* dv, float* delta,
                                                       int passes, void* stream) {
  return gm_lattice_attention_backward_planned(dout, q, k, v, out, lse, win_cnt, win_lo, win_off, entries, row_order, n_order_rows, t_win_cnt, t_win_lo,
                                               t_win_off, t_entries, t_row_order, t_n_order_rows, desc_host, F, rows, nlon, batch, D, H, W, ES, NORD,
                                               scale, dq, dk, dv, delta, passes, nullptr, nullptr, nullptr, nullptr, stream);
}

extern "C" int gm_lattice_attention_tc_wait_expired(int* expired) {
  GM_REQUIRE(expired, GM_ERR_ARGUMENT, "gm_lattice_attention_tc_wait_expired: null pointer");
  *expired = 0;
  return GM_OK;
}
