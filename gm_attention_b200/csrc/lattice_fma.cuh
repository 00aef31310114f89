// Fused gauge attention on an equiangular lattice with longitude-equivariant
// frames: the fast path of gm_attention_forward / backward, fp32 arithmetic.
//
// On such a lattice every per-edge quantity depends on (target row, source
// row, longitude offset) only, so the per-edge tables of the general kernel
// (8 + 8 * orders + 5 bytes per edge, per-edge index) collapse to one entry per
// (row pair, offset) -- ~26 k entries for the 256 x 512 lattice instead of
// 13.5 M edges -- and the neighbours of a target in one source row are a
// contiguous (cyclic) run of longitudes.  Same arithmetic as the general kernel
// (reference semantics: src/gm_attention/nn/fused/attention.h:145-165, 295-316
// for the scores and softmax, src/gm_attention/nn/kernels.py:156-189 for the
// transported values).
//
// What bounds it: multiply-adds (two contractions per pair forward, three in pass T, four in pass S) and the
// shared-memory reads that feed them.  Work split: a lane owns C copies of the scalar block and of every frequency of
// one owner (target in the forward and pass T, source in pass S), so L = 1, 2 or 4 lanes cover a head of up to 4, 8 or
// 16 copies; few lanes per owner keep the per-pair work that every lane repeats (logit, exponential, phases, shuffles)
// small beside the copies' multiply-adds.  The forward holds TT = 2 adjacent owners per lane (every neighbour value read
// from shared memory serves both); the backward passes hold more state per owner and take one, which also visits no
// pair outside an owner's window.
//
// The neighbour rows of one lattice row are copied by cp.async, all of a stage in flight together, into 16-byte chunks
// laid out [chunk][position]: lanes of consecutive owners then read consecutive 16-byte words, without bank conflicts.
// Ragged heads (copies not a multiple of C) are padded with zeros there, so every layout runs the same inner loop.
// The forward has one buffer (its 128 owners x 2 fields fill it; the SM's other CTAs compute while one copies), the
// backward passes two.  On 128 x 256, batch 4, 4 heads of 8 x (m <= 3), float32, the layer's training pass measured
// 13.06 ms with staging by a loop of dependent loads and 4 / 8 lanes per owner, and 6.2 ms in this form (1.7 + 2.1 + 2.4).
// Issue slots are 42 % busy: two or three CTAs of 4 warps are what registers and shared memory allow, and 7 to 9 steps per
// stage on the equatorial rows leave the barriers and the copies' latency visible (64-thread CTAs, twice the lanes with
// half the copies, and equal stages of a wide window measured the same or slower).
//
// Small problems: PARTS lanes share an owner's neighbours (r = part, part + PARTS, ...) and merge their softmax states /
// sums at the end, so that a polar row's few hundred neighbours are not one lane's serial chain.
//
// The backward is deterministic and atomic-free: pass T (owners = targets)
// recomputes the logits from the saved log-sum-exp and accumulates dq; pass S
// (owners = SOURCES, neighbours = targets, transposed tables) recomputes them
// again and accumulates dk and dv, each element written exactly once.
#pragma once
#include "common.cuh"

namespace gmb {
namespace lat {

constexpr int LAT_MAX_CF = 4;   // complex frequencies per head
constexpr int LAT_THREADS = 128;
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
enum { MODE_FWD = 0, MODE_BWD_T = 1, MODE_BWD_S = 2 };

// A head's layout: optionally a_0 scalar copies, then n_cf complex frequencies of a_c copies each.
struct LatPlan {
  int a0, ac, n_cf;
  int real_off;               // flat offset of the scalar block (all heads)
  int cf_off[LAT_MAX_CF];     // flat offset of each complex frequency's block (all heads)
  int cf_order[LAT_MAX_CF];   // its frequency n >= 1
};

struct LatArgs {
  const void *f1, *f2;   // neighbour-side fields staged in shared memory (k, v | k, v | q, dO)
  const void *o1, *o2;   // owner-side fields held in registers          (q, - | q, dO | k, v)
  const float *lse, *delta;  // (batch * rows * nlon, H)
  const void* out_fwd;    // pass T: when set, Delta = <dO, O> is formed here ...
  float* delta_out;       // ... and written for pass S
  void *r1, *r2;          // results: out | dq | dk, dv
  float* lse_out;
  const int *win_cnt, *win_lo, *win_off;  // (rows, 2W + 1)
  const float* entries;                   // (n_entries, ES): (cos, sin) of orders 1..NORD, then bias
  const int* row_order;                   // owner rows, heaviest first
  int rows, nlon, D, H, W, ES, NORD, parts;
  float scale;
  LatPlan plan;
};

// Tile sizes of one instantiation.  Position p of a stage sits in 16-byte column idx(p) of every chunk; with two owners per
// lane (positions 2 apart between neighbouring lanes) the even positions come first.  The pitch NP makes the L lanes of
// one owner fall on other banks than their neighbours' (L = 2: NP = 2 mod 4, L = 4: NP odd).
template <int C, int L, int NCF, int MODE>
struct Tile {
  static constexpr int TT = MODE == MODE_FWD ? 2 : 1;
  static constexpr int CH = (C + 1) / 2;               // 16-byte chunks of a lane's run of C complex copies
  static constexpr int CHUNKS = L * (1 + NCF * CH);    // chunks of a padded head row
  static constexpr int TL = LAT_THREADS / L * TT;      // owners per CTA (PARTS = 1)
  static constexpr int SC = TL + 8;                    // positions per stage
  static constexpr int NP = SC + (L == 4 ? 1 : 2);
  static constexpr int HALF = TT == 2 ? (NP + 1) / 2 : 0;
  static constexpr int NBUF = MODE == MODE_FWD ? 1 : 2;
  static constexpr int EW = (2 * NCF + 1 + 3) / 4 * 4;  // floats per staged table entry: phases, bias
  static constexpr int EN = SC + TL;
  static constexpr int FIELD = CHUNKS * NP * 16;
  static constexpr int STAGE = 2 * FIELD + EN * EW * 4 + (MODE == MODE_BWD_S ? SC * 8 : 0);
  static_assert(STAGE % 16 == 0, "stages start on 16-byte boundaries");
  // registers of state per lane decide how many CTAs share an SM (65536 / 128 threads: 4 at 128, 3 at 168, 2 at 255)
  static constexpr int SLICE = C * (1 + 2 * NCF);
  static constexpr int STATE = (MODE == MODE_FWD ? 4 : MODE == MODE_BWD_T ? 3 : 4) * SLICE + (MODE == MODE_FWD ? 1 : 2) * SLICE;
  // (pass T at 8 x (m <= 3): 202 registers, two CTAs 2.20 ms; held to 168, three CTAs 2.10 ms; the forward held to 168 loses:
  // 1.72 against 2.09 ms, pass S too: 2.38 against 3.57 ms)
  static constexpr int BY_STATE = STATE <= 72 ? 4 : STATE <= (MODE == MODE_BWD_T ? 140 : 124) ? 3 : 2;
  // ... and no more than shared memory admits (228 KB per SM; 1.5 KB of a CTA's are the system's and the row pairs'):
  // registers held down for a CTA that cannot come only cost (pass T of 16 x 3 copies x frequencies held to 165 registers for
  // nothing: the backward 2.13 ms, 2.04 without; 6 x 4: 1.59, 1.55; 4 x 3, 12 x 3 and 12 x 4 the same within 1 %)
  static constexpr int BY_SMEM = 228 * 1024 / (NBUF * STAGE + 1536);
  static constexpr int CTAS = BY_STATE < BY_SMEM ? BY_STATE : BY_SMEM;
  static __device__ __forceinline__ int idx(int p) { return TT == 2 ? (p >> 1) + (p & 1) * HALF : p; }
};

__device__ __forceinline__ int wrap(int x, int n) {
  x %= n;
  return x < 0 ? x + n : x;
}
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src, int src_bytes) {  // the rest of BYTES is filled with zeros
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(addr), "l"(src), "r"(src_bytes));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(addr), "l"(src), "n"(BYTES), "r"(src_bytes));
}

// One row's slice owned by a lane: C scalars and NCF * C complex numbers.
template <int C, int NCF>
struct Slice {
  float re[C];
  float cr[NCF * C], ci[NCF * C];
};

struct RowPair {
  int cnt, lo, j, off;
};

template <typename S, int C, int L, int NCF, int MODE>
__global__ void __launch_bounds__(LAT_THREADS, (Tile<C, L, NCF, MODE>::CTAS)) lattice_kernel(const __grid_constant__ LatArgs a) {
  using T = Tile<C, L, NCF, MODE>;
  constexpr int TT = T::TT, CH = T::CH, NP = T::NP, SC = T::SC, EW = T::EW;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int n_pairs_s;
  RowPair* pairs_s = reinterpret_cast<RowPair*>(smem + T::NBUF * T::STAGE);
  const LatPlan& P = a.plan;
  const S* f1 = static_cast<const S*>(a.f1);
  const S* f2 = static_cast<const S*>(a.f2);
  const int parts = a.parts;
  const int lanes = L * parts, groups_per_warp = 32 / lanes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ls = lane % L, part = (lane / L) & (parts - 1);
  const int group = warp * groups_per_warp + lane / lanes;  // the owners TT * group, ... of the CTA's tile
  const int TL = T::TL / parts;                             // owners per CTA
  const int tiles = (a.nlon + TL - 1) / TL;
  const int row = a.row_order[blockIdx.x / tiles];
  const int c0 = (blockIdx.x % tiles) * TL;
  const int h = blockIdx.y;
  const int64_t b = blockIdx.z;
  const int64_t node0 = (b * a.rows + row) * (int64_t)a.nlon;
  const float cscale = a.scale * LOG2E;

  // ---- the non-empty neighbour rows, once per CTA
  if (warp == 0) {
    int filled = 0;
    for (int x0 = 0; x0 < 2 * a.W + 1; x0 += 32) {
      const int x = x0 + lane, j = row + x - a.W, widx = row * (2 * a.W + 1) + x;
      const int cnt = x < 2 * a.W + 1 && j >= 0 && j < a.rows ? a.win_cnt[widx] : 0;
      const unsigned have = __ballot_sync(0xffffffffu, cnt > 0);
      if (cnt > 0) pairs_s[filled + __popc(have & ((1u << lane) - 1u))] = RowPair{cnt, a.win_lo[widx], j, a.win_off[widx]};
      filled += __popc(have);
    }
    if (lane == 0) n_pairs_s = filled;
  }

  // ---- owners: a lane's run is scalars / copies u = C ls .. C ls + C - 1; slots beyond the head's copies stay zero
  const int u0 = C * ls;
  Slice<C, NCF> o1[TT], o2[MODE == MODE_FWD ? 1 : TT], acc1[TT], acc2[MODE == MODE_BWD_S ? TT : 1];
  float own_lse[TT], own_delta[TT], m[TT], l[TT];
  bool own_ok[TT];
  auto column = [&](int f) { return P.cf_off[f] + 2 * (h * P.ac + u0); };
  auto load_owner = [&](const void* field, bool present, int64_t base, Slice<C, NCF>& s) {
    const S* p = static_cast<const S*>(field) + base;
#pragma unroll
    for (int x = 0; x < C; ++x) s.re[x] = present && u0 + x < P.a0 ? ld<float>(p + P.real_off + h * P.a0 + u0 + x) : 0.f;
#pragma unroll
    for (int f = 0; f < NCF; ++f)
#pragma unroll
      for (int x = 0; x < C; ++x) {
        const bool ok = present && f < P.n_cf && u0 + x < P.ac;
        s.cr[f * C + x] = ok ? ld<float>(p + column(f) + 2 * x) : 0.f;
        s.ci[f * C + x] = ok ? ld<float>(p + column(f) + 2 * x + 1) : 0.f;
      }
  };
#pragma unroll
  for (int tt = 0; tt < TT; ++tt) {
    const int t = c0 + group * TT + tt;
    own_ok[tt] = t < a.nlon;
    m[tt] = -1e30f;
    l[tt] = 0.f;
    own_lse[tt] = own_delta[tt] = 0.f;
    const int64_t node = node0 + (own_ok[tt] ? t : 0), base = node * a.D;
    load_owner(a.o1, own_ok[tt], base, o1[tt]);
#pragma unroll
    for (int x = 0; x < C; ++x) {
      acc1[tt].re[x] = 0.f;
      if constexpr (MODE == MODE_BWD_S) acc2[tt].re[x] = 0.f;
    }
#pragma unroll
    for (int x = 0; x < NCF * C; ++x) {
      acc1[tt].cr[x] = acc1[tt].ci[x] = 0.f;
      if constexpr (MODE == MODE_BWD_S) acc2[tt].cr[x] = acc2[tt].ci[x] = 0.f;
    }
    if constexpr (MODE != MODE_FWD) load_owner(a.o2, own_ok[tt], base, o2[tt]);
    if constexpr (MODE == MODE_BWD_T) {
      if (own_ok[tt]) own_lse[tt] = LOG2E * a.lse[node * a.H + h];
      if (a.out_fwd != nullptr) {
        Slice<C, NCF> of;
        load_owner(a.out_fwd, own_ok[tt], base, of);
        float d = 0.f;
#pragma unroll
        for (int x = 0; x < C; ++x) d += o2[tt].re[x] * of.re[x];
#pragma unroll
        for (int x = 0; x < NCF * C; ++x) d += o2[tt].cr[x] * of.cr[x] + o2[tt].ci[x] * of.ci[x];
#pragma unroll
        for (int o = L >> 1; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        own_delta[tt] = d;
        if (own_ok[tt] && ls == 0 && part == 0) a.delta_out[node * a.H + h] = d;
      } else if (own_ok[tt]) {
        own_delta[tt] = a.delta[node * a.H + h];
      }
    }
  }

  // ---- staging: a thread keeps one 16-byte chunk of the padded head row and strides the positions
  constexpr int PER_PASS = LAT_THREADS / T::CHUNKS;
  static_assert(PER_PASS >= 1, "a pass covers at least one position");
  const int st_p = threadIdx.x / T::CHUNKS, st_ch = threadIdx.x - st_p * T::CHUNKS;
  int st_col = 0, st_n = 0;  // first flat column of the chunk, elements of it that exist (0 .. 4)
  if (st_ch < L) {
    st_col = P.real_off + h * P.a0 + C * st_ch;
    st_n = min(max(P.a0 - C * st_ch, 0), C);
  } else {
    const int cc = st_ch - L, f = cc / (L * CH), run = (cc / CH) % L, k = cc % CH, u = C * run + 2 * k;
    st_col = P.cf_off[f] + 2 * (h * P.ac + u);
    st_n = f < P.n_cf ? 2 * min(max(min(C * run + C, P.ac) - u, 0), 2) : 0;
  }
  if (st_n == 0) st_col = 0;
  const bool st_16 = a.D % 4 == 0 && ((reinterpret_cast<uintptr_t>(f1 + st_col) | reinterpret_cast<uintptr_t>(f2 + st_col)) & (4 * sizeof(S) - 1)) == 0;
  const bool st_8 = a.D % 2 == 0 && ((reinterpret_cast<uintptr_t>(f1 + st_col) | reinterpret_cast<uintptr_t>(f2 + st_col)) & (2 * sizeof(S) - 1)) == 0;
  auto issue = [&](int buf, const RowPair& rp, int p0) {
    unsigned char* stage = smem + buf * T::STAGE;
    const int np = min(SC, TL + rp.cnt - 1 - p0);
    const int64_t nrow0 = (b * a.rows + rp.j) * (int64_t)a.nlon;
    const int lon0 = wrap(c0 + rp.lo + p0, a.nlon);
    if (st_p < PER_PASS) {
      int lon = lon0 + st_p;
      while (lon >= a.nlon) lon -= a.nlon;
      const S* s1 = f1 + nrow0 * a.D + st_col;
      const S* s2 = f2 + nrow0 * a.D + st_col;
      unsigned char* d1 = stage + st_ch * NP * 16;
      const int step = PER_PASS % a.nlon;
      for (int p = st_p; p < np; p += PER_PASS) {
        unsigned char* d = d1 + T::idx(p) * 16;
        const int64_t at = (int64_t)lon * a.D;
        if constexpr (sizeof(S) == 4) {
          if (st_16) {
            cp_async<16>(d, s1 + at, 4 * st_n);
            cp_async<16>(d + T::FIELD, s2 + at, 4 * st_n);
          } else if (st_8) {
#pragma unroll
            for (int x = 0; x < 4; x += 2) {
              const int bytes = 4 * min(max(st_n - x, 0), 2), skip = bytes ? x : 0;
              cp_async<8>(d + 4 * x, s1 + at + skip, bytes);
              cp_async<8>(d + 4 * x + T::FIELD, s2 + at + skip, bytes);
            }
          } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int bytes = x < st_n ? 4 : 0, skip = bytes ? x : 0;
              cp_async<4>(d + 4 * x, s1 + at + skip, bytes);
              cp_async<4>(d + 4 * x + T::FIELD, s2 + at + skip, bytes);
            }
          }
        } else {
          float v1[4], v2[4];
          if (st_16 && st_n == 4) {  // four bf16 in one word pair: a bf16 is the upper half of the fp32 with the same value
            const uint2 w1 = __ldg(reinterpret_cast<const uint2*>(s1 + at)), w2 = __ldg(reinterpret_cast<const uint2*>(s2 + at));
            v1[0] = __uint_as_float(w1.x << 16); v1[1] = __uint_as_float(w1.x & 0xffff0000u);
            v1[2] = __uint_as_float(w1.y << 16); v1[3] = __uint_as_float(w1.y & 0xffff0000u);
            v2[0] = __uint_as_float(w2.x << 16); v2[1] = __uint_as_float(w2.x & 0xffff0000u);
            v2[2] = __uint_as_float(w2.y << 16); v2[3] = __uint_as_float(w2.y & 0xffff0000u);
          } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              v1[x] = x < st_n ? ld<float>(s1 + at + x) : 0.f;
              v2[x] = x < st_n ? ld<float>(s2 + at + x) : 0.f;
            }
          }
          *reinterpret_cast<float4*>(d) = make_float4(v1[0], v1[1], v1[2], v1[3]);
          *reinterpret_cast<float4*>(d + T::FIELD) = make_float4(v2[0], v2[1], v2[2], v2[3]);
        }
        lon += step;
        if (lon >= a.nlon) lon -= a.nlon;
      }
    }
    // table entries of the offsets the stage can meet: x from max(0, p0 - (TL - 1)) on
    float* ent_s = reinterpret_cast<float*>(stage + 2 * T::FIELD);
    const int x0 = max(0, p0 - (TL - 1)), nx = min(rp.cnt, p0 + np) - x0;
    for (int i = threadIdx.x; i < nx * EW; i += LAT_THREADS) {
      const int x = i / EW, w = i - x * EW;
      if (w > 2 * NCF) continue;
      const int f = w >> 1;
      const int from = w == 2 * NCF ? 2 * a.NORD : (f < P.n_cf ? 2 * (P.cf_order[f] - 1) + (w & 1) : -1);
      cp_async<4>(ent_s + i, a.entries + (size_t)(rp.off + x0 + x) * a.ES + max(from, 0), from >= 0 ? 4 : 0);
    }
    if constexpr (MODE == MODE_BWD_S) {
      float* stat = ent_s + T::EN * EW;
      for (int i = threadIdx.x; i < 2 * np; i += LAT_THREADS) {
        int lon = lon0 + (i >> 1);
        while (lon >= a.nlon) lon -= a.nlon;
        const int64_t nn = (nrow0 + lon) * a.H + h;
        cp_async<4>(stat + i, (i & 1 ? a.delta : a.lse) + nn, 4);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  auto load_slice = [&](const unsigned char* lane_base, int pl, Slice<C, NCF>& s) {  // lane_base: the lane's first chunk of the field
    const float4* p = reinterpret_cast<const float4*>(lane_base) + T::idx(pl);
    const float4 t = p[ls * NP];
    const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int x = 0; x < C; ++x) s.re[x] = tv[x];
    const float4* pc = p + (L + ls * CH) * NP;
#pragma unroll
    for (int f = 0; f < NCF; ++f)
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const float4 z = pc[(f * L * CH + k) * NP];
        s.cr[f * C + 2 * k] = z.x; s.ci[f * C + 2 * k] = z.y;
        if (2 * k + 1 < C) { s.cr[f * C + (2 * k + 1 < C ? 2 * k + 1 : 0)] = z.z; s.ci[f * C + (2 * k + 1 < C ? 2 * k + 1 : 0)] = z.w; }
      }
  };

  __syncthreads();
  const int n_pairs = n_pairs_s;
  int pair = 0, p0 = 0;            // the stage being consumed
  int next_pair = 0, next_p0 = 0;  // the stage to copy next
  auto advance = [&](int& pr, int& q) {
    if (q + SC < TL + pairs_s[pr].cnt - 1) q += SC;
    else { ++pr; q = 0; }
  };
  int buf = 0;
  if (T::NBUF == 2 && n_pairs > 0) {
    issue(0, pairs_s[0], 0);
    advance(next_pair, next_p0);
  }
  const int q0 = group * TT;
  const int qw_lo = warp * groups_per_warp * TT, qw_hi = qw_lo + (groups_per_warp - 1) * TT;
  while (pair < n_pairs) {
    const RowPair rp = pairs_s[pair];
    if constexpr (T::NBUF == 2) {
      if (next_pair < n_pairs) {
        issue(buf ^ 1, pairs_s[next_pair], next_p0);
        advance(next_pair, next_p0);
        asm volatile("cp.async.wait_group 1;\n" ::);
      } else {
        asm volatile("cp.async.wait_group 0;\n" ::);
      }
    } else {
      issue(0, rp, p0);
      asm volatile("cp.async.wait_group 0;\n" ::);
    }
    __syncthreads();
    const unsigned char* stage = smem + buf * T::STAGE;
    const float* ent_s = reinterpret_cast<const float*>(stage + 2 * T::FIELD);
    const float* stat = ent_s + T::EN * EW;
    const int cnt = rp.cnt, np = min(SC, TL + cnt - 1 - p0), x0 = max(0, p0 - (TL - 1));
    // An owner at tile offset q reads the positions p = q + x, x in [0, cnt).  The walk is over r = p - q0, the SAME range
    // for every lane of the warp (the shuffles need all lanes in step); lanes whose p is not staged idle through the step.
    const int r_begin = max(0, p0 - qw_hi), r_end = min(TT - 1 + cnt, p0 + np - qw_lo);
    for (int r = r_begin + part; r - part < r_end; r += parts) {
      const int p = q0 + r;
      const bool staged = p >= p0 && p < p0 + np;
      const int pl = staged ? p - p0 : 0;
      Slice<C, NCF> n1;
      load_slice(stage, pl, n1);
      float tr[TT][NCF], ti[TT][NCF], logit[TT], dal[TT];
      bool valid[TT];
#pragma unroll
      for (int tt = 0; tt < TT; ++tt) {
        const int x = r - tt;
        valid[tt] = staged && own_ok[tt] && x >= 0 && x < cnt;
        const float* e = ent_s + (valid[tt] ? x - x0 : 0) * EW;
        float t[2 * NCF + 2];
        if constexpr (NCF >= 2) {
          const float4 q = *reinterpret_cast<const float4*>(e);
          t[0] = q.x; t[1] = q.y; t[2] = q.z; t[3] = q.w;
          if constexpr (NCF == 3) { const float2 q2 = *reinterpret_cast<const float2*>(e + 4); t[4] = q2.x; t[5] = q2.y; }
          if constexpr (NCF == 4) { const float4 q2 = *reinterpret_cast<const float4*>(e + 4); t[4] = q2.x; t[5] = q2.y; t[6] = q2.z; t[7] = q2.w; }
        } else {
          const float2 q = *reinterpret_cast<const float2*>(e);
          t[0] = q.x; t[1] = q.y;
        }
        float sum = 0.f;
#pragma unroll
        for (int x = 0; x < C; ++x) sum += o1[tt].re[x] * n1.re[x];
#pragma unroll
        for (int f = 0; f < NCF; ++f) {
          tr[tt][f] = t[2 * f];
          ti[tt][f] = t[2 * f + 1];
          // G = sum over copies of conj(q) k  (q on the owner side in passes FWD / T, on the neighbour side in pass S)
          float gr = 0.f, gi = 0.f;
#pragma unroll
          for (int u = 0; u < C; ++u) {
            const int s = f * C + u;
            gr += o1[tt].cr[s] * n1.cr[s];
            gr += o1[tt].ci[s] * n1.ci[s];
            if (MODE == MODE_BWD_S) {
              gi += n1.cr[s] * o1[tt].ci[s];
              gi -= n1.ci[s] * o1[tt].cr[s];
            } else {
              gi += o1[tt].cr[s] * n1.ci[s];
              gi -= o1[tt].ci[s] * n1.cr[s];
            }
          }
          sum += tr[tt][f] * gr;  // Re(tau G)
          sum -= ti[tt][f] * gi;
        }
#pragma unroll
        for (int o = L >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        // logits are kept in base 2 (scale and bias carry log2 e), so the exponentials are single ex2 instructions
        logit[tt] = valid[tt] ? cscale * sum + LOG2E * e[2 * NCF] : -INFINITY;
      }
      Slice<C, NCF> n2;
      load_slice(stage + T::FIELD, pl, n2);
      if constexpr (MODE == MODE_FWD) {
#pragma unroll
        for (int tt = 0; tt < TT; ++tt) {
          // the reference maximum moves only when it is exceeded by 2^8 (the weights then stay below 256, and the
          // normalised result does not depend on it)
          if (logit[tt] > m[tt] + 8.f) {
            const float corr = exp2f(m[tt] - logit[tt]);
            l[tt] *= corr;
#pragma unroll
            for (int s = 0; s < C; ++s) acc1[tt].re[s] *= corr;
#pragma unroll
            for (int s = 0; s < NCF * C; ++s) { acc1[tt].cr[s] *= corr; acc1[tt].ci[s] *= corr; }
            m[tt] = logit[tt];
          }
          const float pr = exp2f(logit[tt] - m[tt]);  // 2^(-inf) = 0 for masked or out-of-window pairs
          l[tt] += pr;
#pragma unroll
          for (int s = 0; s < C; ++s) acc1[tt].re[s] += pr * n2.re[s];
#pragma unroll
          for (int f = 0; f < NCF; ++f) {
            const float ar = pr * tr[tt][f], ai = pr * ti[tt][f];  // alpha * tau
#pragma unroll
            for (int u = 0; u < C; ++u) {
              const int s = f * C + u;
              acc1[tt].cr[s] += ar * n2.cr[s];
              acc1[tt].cr[s] -= ai * n2.ci[s];
              acc1[tt].ci[s] += ar * n2.ci[s];
              acc1[tt].ci[s] += ai * n2.cr[s];
            }
          }
        }
      } else {
        float lse = own_lse[0], delta = own_delta[0];
        if (MODE == MODE_BWD_S) {
          const float2 st = *reinterpret_cast<const float2*>(stat + 2 * pl);
          lse = LOG2E * st.x;
          delta = st.y;
        }
        float sum = 0.f;
#pragma unroll
        for (int x = 0; x < C; ++x) sum += o2[0].re[x] * n2.re[x];
#pragma unroll
        for (int f = 0; f < NCF; ++f) {
          float hr = 0.f, hi = 0.f;
#pragma unroll
          for (int u = 0; u < C; ++u) {
            const int s = f * C + u;
            hr += o2[0].cr[s] * n2.cr[s];
            hr += o2[0].ci[s] * n2.ci[s];
            if (MODE == MODE_BWD_S) {
              hi += n2.cr[s] * o2[0].ci[s];
              hi -= n2.ci[s] * o2[0].cr[s];
            } else {
              hi += o2[0].cr[s] * n2.ci[s];
              hi -= o2[0].ci[s] * n2.cr[s];
            }
          }
          sum += tr[0][f] * hr;
          sum -= ti[0][f] * hi;
        }
#pragma unroll
        for (int o = L >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        dal[0] = sum;
        const float pr = valid[0] ? exp2f(logit[0] - lse) : 0.f;
        const float ds = a.scale * pr * (dal[0] - delta);
#pragma unroll
        for (int s = 0; s < C; ++s) {
          acc1[0].re[s] += ds * n1.re[s];                                                     // dq += ds k   | dk += ds q
          if constexpr (MODE == MODE_BWD_S) acc2[0].re[s] += pr * n2.re[s];                   //               dv += p dO
        }
#pragma unroll
        for (int f = 0; f < NCF; ++f) {
          const float ar = ds * tr[0][f], ai = ds * ti[0][f];
#pragma unroll
          for (int u = 0; u < C; ++u) {
            const int s = f * C + u;
            if constexpr (MODE == MODE_BWD_T) {  // dq += ds tau k
              acc1[0].cr[s] += ar * n1.cr[s];
              acc1[0].cr[s] -= ai * n1.ci[s];
              acc1[0].ci[s] += ar * n1.ci[s];
              acc1[0].ci[s] += ai * n1.cr[s];
            } else {                             // dk += ds conj(tau) q ; dv += p conj(tau) dO
              acc1[0].cr[s] += ar * n1.cr[s];
              acc1[0].cr[s] += ai * n1.ci[s];
              acc1[0].ci[s] += ar * n1.ci[s];
              acc1[0].ci[s] -= ai * n1.cr[s];
            }
          }
          if constexpr (MODE == MODE_BWD_S) {
            const float cr = pr * tr[0][f], ci = pr * ti[0][f];
#pragma unroll
            for (int u = 0; u < C; ++u) {
              const int s = f * C + u;
              acc2[0].cr[s] += cr * n2.cr[s];
              acc2[0].cr[s] += ci * n2.ci[s];
              acc2[0].ci[s] += cr * n2.ci[s];
              acc2[0].ci[s] -= ci * n2.cr[s];
            }
          }
        }
      }
    }
    __syncthreads();  // everyone is done with the buffer before it is copied into again
    advance(pair, p0);
    if (T::NBUF == 2) buf ^= 1;
  }

  // ---- merge the parts' states (every lane ends with the owner's totals), then write the owners' results
  for (int o = L; o < lanes; o <<= 1) {
#pragma unroll
    for (int tt = 0; tt < TT; ++tt) {
      float mine = 1.f, other = 1.f;
      if constexpr (MODE == MODE_FWD) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m[tt], o), mm = fmaxf(m[tt], m2);
        mine = exp2f(m[tt] - mm);
        other = exp2f(m2 - mm);
        m[tt] = mm;
        l[tt] = mine * l[tt] + other * __shfl_xor_sync(0xffffffffu, l[tt], o);
      }
      auto merge = [&](float& v) { v = mine * v + other * __shfl_xor_sync(0xffffffffu, v, o); };
#pragma unroll
      for (int s = 0; s < C; ++s) {
        merge(acc1[tt].re[s]);
        if constexpr (MODE == MODE_BWD_S) merge(acc2[tt].re[s]);
      }
#pragma unroll
      for (int s = 0; s < NCF * C; ++s) {
        merge(acc1[tt].cr[s]);
        merge(acc1[tt].ci[s]);
        if constexpr (MODE == MODE_BWD_S) { merge(acc2[tt].cr[s]); merge(acc2[tt].ci[s]); }
      }
    }
  }
  if (part != 0) return;
  auto store_owner = [&](void* field, int64_t base, float inv, const Slice<C, NCF>& s) {
    S* p = static_cast<S*>(field) + base;
    const bool vec = sizeof(S) == 4 && C == 4 && a.D % 4 == 0 && (reinterpret_cast<uintptr_t>(field) & 15) == 0;
    S* q = p + P.real_off + h * P.a0 + u0;
    if (vec && u0 + C <= P.a0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0) {
      *reinterpret_cast<float4*>(q) = make_float4(s.re[0] * inv, s.re[1] * inv, s.re[2 % C] * inv, s.re[3 % C] * inv);
    } else {
#pragma unroll
      for (int x = 0; x < C; ++x)
        if (u0 + x < P.a0) st<S>(q + x, s.re[x] * inv);
    }
#pragma unroll
    for (int f = 0; f < NCF; ++f) {
      if (f >= P.n_cf) continue;
      q = p + column(f);
      if (vec && u0 + C <= P.ac && (reinterpret_cast<uintptr_t>(q) & 15) == 0) {
#pragma unroll
        for (int k = 0; k < C / 2; ++k)
          *reinterpret_cast<float4*>(q + 4 * k) = make_float4(s.cr[f * C + 2 * k] * inv, s.ci[f * C + 2 * k] * inv,
                                                              s.cr[f * C + 2 * k + 1] * inv, s.ci[f * C + 2 * k + 1] * inv);
      } else {
#pragma unroll
        for (int x = 0; x < C; ++x) {
          if (u0 + x >= P.ac) continue;
          st<S>(q + 2 * x, s.cr[f * C + x] * inv);
          st<S>(q + 2 * x + 1, s.ci[f * C + x] * inv);
        }
      }
    }
  };
#pragma unroll
  for (int tt = 0; tt < TT; ++tt) {
    if (!own_ok[tt]) continue;
    const int64_t node = node0 + c0 + group * TT + tt;
    const float inv = MODE == MODE_FWD ? (l[tt] > 0.f ? 1.f / l[tt] : 0.f) : 1.f;
    store_owner(a.r1, node * a.D, inv, acc1[tt]);
    if constexpr (MODE == MODE_BWD_S) store_owner(a.r2, node * a.D, 1.f, acc2[tt]);
    if (MODE == MODE_FWD && ls == 0) a.lse_out[node * a.H + h] = l[tt] > 0.f ? (m[tt] + log2f(l[tt])) * LN2 : -INFINITY;
  }
}

// How many lanes share an owner's neighbours: 1 where the owners alone fill the chip, otherwise the power of two (up to 8)
// that brings the launch to about two CTAs of 128 threads per SM.  A polar owner's chain of a few hundred neighbours is
// what a small lattice waits for; a large one is bound by throughput and would only pay for the merge.
inline int choose_parts(int64_t owners, int lanes_per_owner, int owners_per_lane, int max_parts) {
  const int64_t want = (int64_t)sm_count() * 2 * LAT_THREADS;
  int parts = 1;
  while (parts < max_parts && owners * lanes_per_owner * parts / owners_per_lane < want) parts *= 2;
  return parts;
}

template <typename S, int C, int L, int NCF, int MODE>
int launch_tile(LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream) {
  using T = Tile<C, L, NCF, MODE>;
  a.parts = choose_parts((int64_t)n_order_rows * a.nlon * a.H * batch, L, T::TT, 8);
  const int TL = T::TL / a.parts, tiles = (a.nlon + TL - 1) / TL;
  const size_t smem = (size_t)T::NBUF * T::STAGE + (size_t)(2 * a.W + 1) * sizeof(RowPair);
  auto kernel = lattice_kernel<S, C, L, NCF, MODE>;
  const int status = allow_smem(kernel, smem, "gm_lattice_attention");
  if (status != GM_OK) return status;
  dim3 grid((unsigned)(n_order_rows * tiles), (unsigned)a.H, (unsigned)batch);
  kernel<<<grid, LAT_THREADS, smem, stream>>>(a);
  return launch_status("gm_lattice_attention");
}

// Copies per lane and lanes per owner: the fewest lanes that hold the head's larger multiplicity with at most 4 copies each.
template <typename S, int NCF, int MODE>
int launch_copies(LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream) {
  const int most = a.plan.a0 > a.plan.ac ? a.plan.a0 : a.plan.ac;
  if (most <= 4) return launch_tile<S, 4, 1, NCF, MODE>(a, n_order_rows, batch, stream);
  if (most <= 6) return launch_tile<S, 3, 2, NCF, MODE>(a, n_order_rows, batch, stream);
  if (most <= 8) return launch_tile<S, 4, 2, NCF, MODE>(a, n_order_rows, batch, stream);
  if (most <= 12) return launch_tile<S, 3, 4, NCF, MODE>(a, n_order_rows, batch, stream);
  if (most <= 16) return launch_tile<S, 4, 4, NCF, MODE>(a, n_order_rows, batch, stream);
  return fail(GM_ERR_UNSUPPORTED, "gm_lattice_attention: no kernel for %d scalar / %d x %d complex copies", a.plan.a0, a.plan.n_cf, a.plan.ac);
}

template <typename S, int MODE>
int launch_mode(LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream) {
  switch (a.plan.n_cf) {
    case 0:
    case 1: return launch_copies<S, 1, MODE>(a, n_order_rows, batch, stream);
    case 2: return launch_copies<S, 2, MODE>(a, n_order_rows, batch, stream);
    case 3: return launch_copies<S, 3, MODE>(a, n_order_rows, batch, stream);
    default: return launch_copies<S, 4, MODE>(a, n_order_rows, batch, stream);
  }
}

// One pass over the owners in row_order (mode = MODE_*); a: everything but the tile choice filled in.
int lattice_pass_f32(int mode, LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream);
int lattice_pass_bf16(int mode, LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream);

template <typename S>
int lattice_pass(int mode, LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream) {
  if (mode == MODE_FWD) return launch_mode<S, MODE_FWD>(a, n_order_rows, batch, stream);
  if (mode == MODE_BWD_T) return launch_mode<S, MODE_BWD_T>(a, n_order_rows, batch, stream);
  return launch_mode<S, MODE_BWD_S>(a, n_order_rows, batch, stream);
}

}  // namespace lat
}  // namespace gmb
