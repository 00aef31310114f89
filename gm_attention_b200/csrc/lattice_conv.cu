// Depthwise steerable convolution on a longitude-symmetric lattice with the per-edge coefficients replaced by a
// per-(row pair, longitude offset) table.
//
// The reference's depthwise op (nn/fused/attention.h:174-206, 265-287) streams E * (a_0 + W) coefficients: per edge a
// real factor R per scalar channel and complex A, B per complex copy, applied as  m = A z + w B conj(z),  z = tau_n v_j,
// w = (r/c)^{2n} e^{2 i n phi}, and summed with the edge's aggregation weight.  On a lattice whose frames turn with the
// longitude every one of those quantities depends on (target row, source row, longitude offset) only, and
// z -> A z + w B conj(z) is a real-linear map of the plane, so the whole edge collapses into ONE real 2 x 2 matrix per
// (table entry, complex copy) and one real factor per (entry, scalar channel).  The kernels here are
//
//   fold        the entries' coefficients, phases and weights -> that table, and its gradient -> the coefficients'
//               (gm_attention_b200/nn/lattice_depthwise.py: FoldTable; fold there is the same in tensor algebra)
//   apply       y[i, l] = sum over entries (j, d) of row i   M[entry] x[j, l + lo + d]      (forward; with the transposed
//               windows and M^T it is the gradient with respect to the node field)
//   table_grad  dM[entry] = sum over longitudes l and samples  dy[i, l] (x) x[j, l + lo + d]
//
// apply and table_grad are bound by arithmetic, not HBM (4 multiply-adds per complex copy, edge and sample against 0.01 bytes of
// compulsory traffic).  bfloat16 fields whose rows are whole 16-byte words have tensor-core kernels (lattice_conv_tc.cu), taken where
// they are the faster ones; the kernels here, on the FMA pipe, serve everything else.  A thread owns
// one item -- a complex copy, or a pair of scalar channels -- so a warp reads 32 neighbouring items of a node as one
// 128-byte line; it keeps 8 longitudes x 2 samples of accumulators in registers and slides a register window of 8
// source longitudes (apply) or 8 target longitudes (table_grad) past them, so every loaded value is used for 8 x 4
// multiply-adds without shared memory.  apply has a second form that stages both operands and packs the arithmetic, taken
// wherever a stage fits.  Results do not depend on the launch geometry: no atomics.
#include "lattice_conv.cuh"

namespace gmb {
namespace {

using lconv::ConvArgs;

constexpr int LON = 8;  // longitudes (apply) / longitude offsets (table_grad) per thread
constexpr int THREADS = 160;  // at most; three CTAs per SM (128 registers per thread); more items than threads are looped over

// Two neighbouring elements of a node's row: loaded as one word (bf16) or two (float), unpacked when used, so that a
// value in flight between its load and its use costs one register per bf16 pair.
template <typename S> struct Pair;
template <> struct Pair<float> {
  using Raw = float2;
  static __device__ __forceinline__ Raw load(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
  static __device__ __forceinline__ Raw zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ float2 unpack(Raw r) { return r; }
  static __device__ __forceinline__ void store(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
};
template <> struct Pair<__nv_bfloat16> {
  using Raw = unsigned;
  static __device__ __forceinline__ Raw load(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const unsigned*>(p)); }
  static __device__ __forceinline__ Raw zero() { return 0u; }
  static __device__ __forceinline__ float2 unpack(Raw r) { return make_float2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u)); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float2 v) {
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(v.x, v.y);
  }
};

// ---------------------------------------------------------------------------------------------------------------- apply
// TL targets (consecutive longitudes) x NB samples per thread.
template <typename S, int NB, int TL>
__global__ void __launch_bounds__(THREADS, 3) conv_apply_kernel(const ConvArgs a) {
  constexpr int PF = 4;  // steps in flight (a power of two <= 8)
  const int row = a.order[blockIdx.y];
  const int l0 = blockIdx.x * TL;
  const int b0 = blockIdx.z * NB;
  const int span = 2 * a.halo + 1;
  const size_t sample = (size_t)a.rows * a.nlon * a.width;
  const S* x = static_cast<const S*>(a.x) + (size_t)b0 * sample;
  S* y = static_cast<S*>(a.y) + (size_t)b0 * sample;
  const int nb = min(NB, a.batch - b0);

  for (int item = threadIdx.x; item < a.n_items; item += blockDim.x) {
    const int kind = a.items[3 * item], col = a.items[3 * item + 1], fcol = a.items[3 * item + 2];
    float2 acc[TL][NB];
#pragma unroll
    for (int l = 0; l < TL; ++l)
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[l][b] = make_float2(0.f, 0.f);

    for (int c = 0; c < span; ++c) {
      const int j = row + c - a.halo;
      if (j < 0 || j >= a.rows) continue;
      const int cnt = a.win_cnt[row * span + c];
      if (cnt == 0) continue;
      const int lo = a.win_lo[row * span + c];
      const float* table = a.table + (size_t)a.win_off[row * span + c] * a.table_width + fcol;
      const S* xrow = x + (size_t)j * a.nlon * a.width + col;
      int p = (l0 + lo) % a.nlon;
      if (p < 0) p += a.nlon;
      // Position t of the source row is longitude l0 + lo + t; under offset d the block's target l sees position d + l.
      // A register window holds the 8 most recent positions and slides by one per offset, so every offset is 8 targets x
      // NB samples of multiply-adds on true neighbours only: no ramp, no validity tests.
      auto matrix = [&](int d) {
        const float* f = table + (size_t)d * a.table_width;
        if (kind == 0) {
          const float4 m = __ldg(reinterpret_cast<const float4*>(f));
          return a.transpose ? make_float4(m.x, m.z, m.y, m.w) : m;
        }
        const float2 m = __ldg(reinterpret_cast<const float2*>(f));
        return make_float4(m.x, 0.f, 0.f, m.y);
      };
      int ahead = p;  // longitude of the next position to load
      auto source = [&](int b) { return b < nb ? Pair<S>::load(xrow + b * sample + (size_t)ahead * a.width) : Pair<S>::zero(); };
      auto advance = [&]() { ahead = ahead + 1 == a.nlon ? 0 : ahead + 1; };
      float2 xs[TL][NB];  // xs[t % 8] = position t
#pragma unroll
      for (int t = 0; t < TL - 1; ++t) {
#pragma unroll
        for (int b = 0; b < NB; ++b) xs[t][b] = Pair<S>::unpack(source(b));
        advance();
      }
      // ring of PF offsets in flight: matrix d + PF and position d + 7 + PF are loaded when offset d is consumed
      typename Pair<S>::Raw ring_v[PF][NB];
      float4 ring_m[PF];
#pragma unroll
      for (int t = 0; t < PF; ++t) {
        if (t < cnt) {
          ring_m[t] = matrix(t);
#pragma unroll
          for (int b = 0; b < NB; ++b) ring_v[t][b] = source(b);
          advance();
        }
      }
      for (int d0 = 0; d0 < cnt; d0 += TL) {
#pragma unroll
        for (int u = 0; u < TL; ++u) {
          const int d = d0 + u;
          if (d >= cnt) break;
          const float4 m = ring_m[u % PF];
#pragma unroll
          for (int b = 0; b < NB; ++b) xs[(u + TL - 1) & (TL - 1)][b] = Pair<S>::unpack(ring_v[u % PF][b]);
          if (d + PF < cnt) {
            ring_m[u % PF] = matrix(d + PF);
#pragma unroll
            for (int b = 0; b < NB; ++b) ring_v[u % PF][b] = source(b);
            advance();
          }
          if (kind == 0) {
#pragma unroll
            for (int l = 0; l < TL; ++l)
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                const float2 v = xs[(u + l) & (TL - 1)][b];
                acc[l][b].x = fmaf(m.x, v.x, fmaf(m.y, v.y, acc[l][b].x));
                acc[l][b].y = fmaf(m.z, v.x, fmaf(m.w, v.y, acc[l][b].y));
              }
          } else {  // two independent scalar channels: no cross terms, so a non-finite value stays in its channel
#pragma unroll
            for (int l = 0; l < TL; ++l)
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                const float2 v = xs[(u + l) & (TL - 1)][b];
                acc[l][b].x = fmaf(m.x, v.x, acc[l][b].x);
                acc[l][b].y = fmaf(m.w, v.y, acc[l][b].y);
              }
          }
        }
      }
    }
#pragma unroll
    for (int l = 0; l < TL; ++l) {
      if (l0 + l >= a.nlon) break;
#pragma unroll
      for (int b = 0; b < NB; ++b)
        if (b < nb) Pair<S>::store(y + b * sample + ((size_t)row * a.nlon + l0 + l) * a.width + col, acc[l][b]);
    }
  }
}

// ------------------------------------------------------------------------------------------------------- apply, staged
// The same sums with the window's sources and table entries brought to shared memory first.  A CTA covers G tiles of 8
// longitudes (thread = tile x item); a stage holds up to SO offsets of one window: their table entries, read once per CTA
// instead of once per tile, and the 8 G + SO - 1 source positions of NB samples they meet.  The copies of the next stage
// (cp.async, 16 bytes where the field's rows allow) run while the current one is consumed, so a window's first sources are
// not waited for, and the inner loop has no addresses to form.
//
// The arithmetic is packed: fma.rn.f32x2 on the targets (l, l + 4), whose sources (t, t + 4) form a register pair; moving
// one offset on renames three of the four pairs and rebuilds the fourth from its own upper half and the new source, so the
// window costs one move per value.  Per offset, copy and NB samples 16 NB packed multiply-adds stand against about 8 moves
// (the matrix, duplicated into pairs) and 6 NB of loads, conversions and window moves.  Same order of operations per
// output as conv_apply_kernel: bit-identical results.  256 x 512, radius 4 pi / 256, batch 4, 64 x (m <= 2), bf16: 7.92 ms
// with conv_apply_kernel, 4.51 in this form (FMA pipe about 40 % busy, 10 warps' barriers and the per-stage set-up beside
// it; a field of that size takes the tensor cores now); 45 x 88, batch 3, 32 x (m <= 2), float32: 220 us before, 128 now.
struct StagedShape {
  int tiles, so, threads, stage_bytes, pos_bytes;  // G, SO, G * n_items, bytes of a stage, bytes of one node's row
  int vec16;                                       // rows and bases are multiples of 16 bytes
};

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(addr), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(addr), "l"(src), "n"(BYTES) : "memory");
}
template <typename S> __device__ __forceinline__ float2 shared_pair(const unsigned char* p) {
  if constexpr (sizeof(S) == 4) return *reinterpret_cast<const float2*>(p);
  else return Pair<__nv_bfloat16>::unpack(*reinterpret_cast<const unsigned*>(p));
}
// `bytes` consecutive bytes of a cyclic row of row_bytes, from byte `at` on, into shared memory
template <int BYTES>
__device__ __forceinline__ void copy_cyclic(unsigned char* dst, const unsigned char* row, int at, int bytes, int row_bytes, int threads) {
  for (int u = threadIdx.x * BYTES; u < bytes; u += threads * BYTES) {
    int o = at + u;
    while (o >= row_bytes) o -= row_bytes;
    copy_async<BYTES>(dst + u, row + o);
  }
}

// KIND 0: complex copies (2 x 2 matrices), 1: pairs of scalar channels.  One stage's offsets for one thread.
template <typename S, int NB, int KIND>
__device__ __forceinline__ void consume_stage(const unsigned char* table, int entry_bytes, const unsigned char* pos, int pos_bytes, int sample_bytes,
                                              int n, bool transpose, unsigned long long (&ax)[4][NB], unsigned long long (&ay)[4][NB]) {
  unsigned long long px[4][NB], py[4][NB];  // slot (d + j) & 3: sources (d + j, d + j + 4)
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    float2 v[7];
#pragma unroll
    for (int t = 0; t < 7; ++t) v[t] = shared_pair<S>(pos + b * sample_bytes + t * pos_bytes);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      px[j][b] = pack2(v[j].x, v[j + 4].x);
      py[j][b] = pack2(v[j].y, v[j + 4].y);
    }
    // the first step turns slot 3 into (source 3, source 7): as after every step, the lower half comes from the upper one
    px[3][b] = pack2(0.f, v[3].x);
    py[3][b] = pack2(0.f, v[3].y);
  }
  pos += 7 * pos_bytes;
  for (int d0 = 0; d0 < n; d0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (d0 + u >= n) break;
      // source d + 7 completes the pair (d + 3, d + 7): its lower half is the upper half of the pair that left the window
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const float2 v = shared_pair<S>(pos + b * sample_bytes);
        px[(u + 3) & 3][b] = pack2(unpack2(px[(u + 3) & 3][b]).y, v.x);
        py[(u + 3) & 3][b] = pack2(unpack2(py[(u + 3) & 3][b]).y, v.y);
      }
      pos += pos_bytes;
      if constexpr (KIND == 0) {
        const float4 m = *reinterpret_cast<const float4*>(table);
        const float my = transpose ? m.z : m.y, mz = transpose ? m.y : m.z;
        const unsigned long long m00 = pack2(m.x, m.x), m01 = pack2(my, my), m10 = pack2(mz, mz), m11 = pack2(m.w, m.w);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            const unsigned long long x = px[(u + j) & 3][b], y = py[(u + j) & 3][b];
            ax[j][b] = fma2(m00, x, fma2(m01, y, ax[j][b]));
            ay[j][b] = fma2(m10, x, fma2(m11, y, ay[j][b]));
          }
      } else {  // two independent scalar channels: no cross terms, so a non-finite value stays in its channel
        const float2 m = *reinterpret_cast<const float2*>(table);
        const unsigned long long m0 = pack2(m.x, m.x), m1 = pack2(m.y, m.y);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            ax[j][b] = fma2(m0, px[(u + j) & 3][b], ax[j][b]);
            ay[j][b] = fma2(m1, py[(u + j) & 3][b], ay[j][b]);
          }
      }
      table += entry_bytes;
    }
  }
}

constexpr int STAGED_THREADS = 320;

template <typename S, int NB>
__global__ void __launch_bounds__(STAGED_THREADS, 2) conv_apply_staged_kernel(const ConvArgs a, const StagedShape sh) {
  extern __shared__ __align__(16) unsigned char stage_smem[];
  const int row = a.order[blockIdx.y];
  const int l0 = blockIdx.x * 8 * sh.tiles;
  const int b0 = blockIdx.z * NB;
  const int nb = min(NB, a.batch - b0);
  const int span = 2 * a.halo + 1;
  const int row_bytes = a.nlon * sh.pos_bytes, entry_bytes = 4 * a.table_width;
  const size_t sample = (size_t)a.rows * row_bytes;
  const unsigned char* x = static_cast<const unsigned char*>(a.x) + b0 * sample;
  const int tile = threadIdx.x / a.n_items, item = threadIdx.x - tile * a.n_items;
  const int kind = a.items[3 * item], col = a.items[3 * item + 1], fcol = a.items[3 * item + 2];
  const int most_pos = 8 * sh.tiles + sh.so - 1, sample_bytes = most_pos * sh.pos_bytes;
  const int table_at = (NB * sample_bytes + 15) / 16 * 16;

  // stages: offsets [d, d + n) of window c of this row
  struct Stage { int c, d, n, cnt; };
  auto first_of = [&](int c) {
    for (; c < span; ++c) {
      const int j = row + c - a.halo;
      if (j < 0 || j >= a.rows) continue;
      const int cnt = a.win_cnt[row * span + c];
      if (cnt > 0) return Stage{c, 0, min(sh.so, cnt), cnt};
    }
    return Stage{span, 0, 0, 0};
  };
  auto next_of = [&](const Stage& s) {
    const int d = s.d + s.n;
    return d < s.cnt ? Stage{s.c, d, min(sh.so, s.cnt - d), s.cnt} : first_of(s.c + 1);
  };
  auto issue = [&](int buf, const Stage& s) {
    unsigned char* dst = stage_smem + (size_t)buf * sh.stage_bytes;
    const int j = row + s.c - a.halo, w = row * span + s.c;
    int p = l0 + a.win_lo[w] + s.d;
    while (p < 0) p += a.nlon;
    while (p >= a.nlon) p -= a.nlon;
    const int at = p * sh.pos_bytes, bytes = (8 * sh.tiles + s.n - 1) * sh.pos_bytes;
    for (int b = 0; b < nb; ++b) {
      const unsigned char* src = x + b * sample + (size_t)j * row_bytes;
      if (sh.vec16) copy_cyclic<16>(dst + b * sample_bytes, src, at, bytes, row_bytes, sh.threads);
      else copy_cyclic<4>(dst + b * sample_bytes, src, at, bytes, row_bytes, sh.threads);
    }
    const unsigned char* entries = reinterpret_cast<const unsigned char*>(a.table) + (size_t)(a.win_off[w] + s.d) * entry_bytes;
    for (int u = threadIdx.x * 16; u < s.n * entry_bytes; u += sh.threads * 16) copy_async<16>(dst + table_at + u, entries + u);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  unsigned long long ax[4][NB], ay[4][NB];  // targets (j, j + 4)
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int b = 0; b < NB; ++b) ax[j][b] = ay[j][b] = 0ull;

  Stage cur = first_of(0);
  if (cur.c < span) issue(0, cur);
  int buf = 0;
  while (cur.c < span) {
    const Stage nxt = next_of(cur);
    if (nxt.c < span) {
      issue(buf ^ 1, nxt);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const unsigned char* st = stage_smem + (size_t)buf * sh.stage_bytes;
    const unsigned char* pos = st + 8 * tile * sh.pos_bytes + col * (int)sizeof(S);
    const unsigned char* table = st + table_at + 4 * fcol;
    if (kind == 0) consume_stage<S, NB, 0>(table, entry_bytes, pos, sh.pos_bytes, sample_bytes, cur.n, a.transpose != 0, ax, ay);
    else consume_stage<S, NB, 1>(table, entry_bytes, pos, sh.pos_bytes, sample_bytes, cur.n, false, ax, ay);
    __syncthreads();
    cur = nxt;
    buf ^= 1;
  }
  S* y = static_cast<S*>(a.y) + ((size_t)b0 * a.rows + row) * a.nlon * a.width + col;
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const float2 vx = unpack2(ax[j][b]), vy = unpack2(ay[j][b]);
      const int l = l0 + 8 * tile + j;
      if (b >= nb || l >= a.nlon) continue;  // nlon is a multiple of 8: a tile is whole or absent
      S* at = y + b * (size_t)a.rows * a.nlon * a.width + (size_t)l * a.width;
      Pair<S>::store(at, make_float2(vx.x, vy.x));
      Pair<S>::store(at + (size_t)4 * a.width, make_float2(vx.y, vy.y));
    }
}

// ----------------------------------------------------------------------------------------------------------- table_grad
// One CTA: one window (target row, source row) and 8 consecutive offsets d0 .. d0 + 7 of it; it walks once around the
// source row.  Step u brings the source at longitude u + lo + d0; offset d0 + k pairs it with the target u - k (cyclic),
// whose gradient row sits in a register window of the 8 most recent targets.
template <typename S, int NB>
__global__ void __launch_bounds__(THREADS, 3) conv_table_grad_kernel(const ConvArgs a) {
  constexpr int PF = 4;  // steps in flight (a power of two <= 8; nlon >= 8)
  const int w = a.order[2 * blockIdx.x], d0 = a.order[2 * blockIdx.x + 1];
  const int span = 2 * a.halo + 1;
  const int row = w / span, j = row + w % span - a.halo;
  const int cnt = a.win_cnt[w], lo = a.win_lo[w];
  const size_t sample = (size_t)a.rows * a.nlon * a.width;
  const int valid = min(LON, cnt - d0);

  for (int item = threadIdx.x; item < a.n_items; item += blockDim.x) {
    const int kind = a.items[3 * item], col = a.items[3 * item + 1], fcol = a.items[3 * item + 2];
    float4 acc[LON];
#pragma unroll
    for (int k = 0; k < LON; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b0 = 0; b0 < a.batch; b0 += NB) {
      const int nb = min(NB, a.batch - b0);
      const S* xrow = static_cast<const S*>(a.x) + (size_t)b0 * sample + (size_t)j * a.nlon * a.width + col;
      const S* grow = static_cast<const S*>(a.g) + (size_t)b0 * sample + (size_t)row * a.nlon * a.width + col;
      float2 window[LON][NB];  // window[t % 8] = gradient of target t
#pragma unroll
      for (int t = 1; t < LON; ++t)  // targets -7 .. -1 (cyclic) are seen by the first steps
#pragma unroll
        for (int b = 0; b < NB; ++b)
          window[(LON - t) & (LON - 1)][b] = b < nb ? Pair<S>::unpack(Pair<S>::load(grow + b * sample + (size_t)(a.nlon - t) * a.width)) : make_float2(0.f, 0.f);
      int p = (lo + d0) % a.nlon;
      if (p < 0) p += a.nlon;
      // ring of PF steps in flight: the source and the target of step u + PF are loaded when step u is consumed
      typename Pair<S>::Raw ring_v[PF][NB], ring_g[PF][NB];
      int ahead = p;
#pragma unroll
      for (int t = 0; t < PF; ++t) {
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          ring_v[t][b] = b < nb ? Pair<S>::load(xrow + b * sample + (size_t)ahead * a.width) : Pair<S>::zero();
          ring_g[t][b] = b < nb ? Pair<S>::load(grow + b * sample + (size_t)t * a.width) : Pair<S>::zero();
        }
        ahead = ahead + 1 == a.nlon ? 0 : ahead + 1;
      }
      for (int u0 = 0; u0 < a.nlon; u0 += LON) {  // nlon is a multiple of 8 (checked by the host)
#pragma unroll
        for (int u = 0; u < LON; ++u) {
          float2 v[NB];
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            v[b] = Pair<S>::unpack(ring_v[u % PF][b]);
            window[u][b] = Pair<S>::unpack(ring_g[u % PF][b]);
          }
          if (u0 + u + PF < a.nlon) {
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              ring_v[u % PF][b] = b < nb ? Pair<S>::load(xrow + b * sample + (size_t)ahead * a.width) : Pair<S>::zero();
              ring_g[u % PF][b] = b < nb ? Pair<S>::load(grow + b * sample + (size_t)(u0 + u + PF) * a.width) : Pair<S>::zero();
            }
            ahead = ahead + 1 == a.nlon ? 0 : ahead + 1;
          }
#pragma unroll
          for (int k = 0; k < LON; ++k) {
            if (k >= valid) break;  // offsets beyond the window: their pairs are not edges
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              const float2 g = window[(u - k) & (LON - 1)][b];
              acc[k].x = fmaf(g.x, v[b].x, acc[k].x);
              acc[k].y = fmaf(g.x, v[b].y, acc[k].y);
              acc[k].z = fmaf(g.y, v[b].x, acc[k].z);
              acc[k].w = fmaf(g.y, v[b].y, acc[k].w);
            }
          }
        }
      }
    }
    float* out = a.dtable + (size_t)(a.win_off[w] + d0) * a.table_width + fcol;
#pragma unroll
    for (int k = 0; k < LON; ++k) {
      if (k >= valid) break;
      if (kind == 0) *reinterpret_cast<float4*>(out + (size_t)k * a.table_width) = acc[k];
      else *reinterpret_cast<float2*>(out + (size_t)k * a.table_width) = make_float2(acc[k].x, acc[k].w);
    }
  }
}

// ----------------------------------------------------------------------------------------------------------------- fold
// An entry's coefficients -> its row of the table, and back (gm_attention_b200/nn/lattice_depthwise.py: fold writes the same in
// tensor algebra, about 35 launches forward and 50 backward over the entries' complex temporaries): scalar factors times
// the weight w; per complex copy a = w tau A, b = w omega conj(tau) B and the real 2 x 2 matrix of z -> a z + b conj(z).
// One CTA per entry, a thread per column: bound by reading the coefficients and writing the table once each (45 x 88, batch
// 3, 32 x (m <= 2): 4.7 us each way; the pass 1.87 -> 0.72 ms, 134 -> 35 launches, of which the host was the bound).
struct FoldArgs {
  const float *rc, *cc, *weights;
  const float2 *tau, *omega;  // (entries, nf)
  const int* items;           // (n_complex, 3): coefficient column of A, of B, frequency index
  const float* dtable;
  float *table, *drc, *dcc;
  int a0, padded, width, n_complex, nf, table_width;
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

template <bool BACKWARD>
__global__ void __launch_bounds__(128) conv_fold_kernel(const FoldArgs a) {
  const size_t e = blockIdx.x;
  const float w = a.weights[e];
  for (int x = threadIdx.x; x < a.padded + a.n_complex; x += 128) {
    if (x < a.padded) {
      if constexpr (BACKWARD) {
        if (x < a.a0 && a.drc) a.drc[e * a.a0 + x] = w * a.dtable[e * a.table_width + x];
      } else {
        a.table[e * a.table_width + x] = x < a.a0 ? w * a.rc[e * a.a0 + x] : 0.f;
      }
      continue;
    }
    const int c = x - a.padded, at_a = a.items[3 * c], at_b = a.items[3 * c + 1], f = a.items[3 * c + 2];
    const float2 tau = a.tau[e * a.nf + f], omega = a.omega[e * a.nf + f];
    const float2 fa = make_float2(w * tau.x, w * tau.y);
    const float2 ot = cmul(omega, make_float2(tau.x, -tau.y)), fb = make_float2(w * ot.x, w * ot.y);
    const size_t ca = e * a.width + at_a, cb = e * a.width + at_b, out = e * a.table_width + a.padded + 4 * c;
    if constexpr (BACKWARD) {
      const float4 d = *reinterpret_cast<const float4*>(a.dtable + out);
      const float2 da = cmul(make_float2(fa.x, -fa.y), make_float2(d.x + d.w, d.z - d.y));
      const float2 db = cmul(make_float2(fb.x, -fb.y), make_float2(d.x - d.w, d.y + d.z));
      a.dcc[ca] = da.x; a.dcc[ca + 1] = da.y;
      a.dcc[cb] = db.x; a.dcc[cb + 1] = db.y;
    } else {
      const float2 va = cmul(fa, make_float2(a.cc[ca], a.cc[ca + 1])), vb = cmul(fb, make_float2(a.cc[cb], a.cc[cb + 1]));
      *reinterpret_cast<float4*>(a.table + out) = make_float4(va.x + vb.x, vb.y - va.y, va.y + vb.y, va.x - vb.x);
    }
  }
}

// Tiles, offsets per stage and samples per thread of the staged apply kernel; returns the samples, 0 where it cannot run.
// Two samples and two CTAs of 320 threads per SM (88 to 95 registers) measured 4.5 ms against 4.7 for four samples and one CTA,
// 5.8 to 6.0 for CTAs of one tile (256 x 512, batch 4, 64 x (m <= 2), bf16, which takes the tensor cores now).  A stage should hold the equator's windows
// whole: where half of the shared memory holds fewer than 8 offsets (float32 rows of 320 columns: 3) a CTA takes all of it.
// Tiles: as many as 320 threads take, fewer while the launch has less than two CTAs per SM (a small lattice waits for
// its polar rows' chains of offsets).
int staged_shape(const ConvArgs& a, int elem, int n_order, StagedShape& sh) {
  if (a.n_items > STAGED_THREADS) return 0;
  sh.pos_bytes = a.width * elem;
  if ((int64_t)a.nlon * sh.pos_bytes > (1ll << 28)) return 0;  // offsets within a row are 32-bit
  const uintptr_t base = reinterpret_cast<uintptr_t>(a.x);
  sh.vec16 = sh.pos_bytes % 16 == 0 && base % 16 == 0;
  const int nb = a.batch >= 2 ? 2 : 1;
  sh.tiles = max(1, min(STAGED_THREADS / a.n_items, a.nlon / 8));
  const int64_t want = 2 * (int64_t)sm_count();
  auto ctas = [&]() { return (int64_t)n_order * ((a.nlon / 8 + sh.tiles - 1) / sh.tiles) * ((a.batch + nb - 1) / nb); };
  while (ctas() < want && sh.tiles > 1) sh.tiles = (sh.tiles + 1) / 2;
  sh.threads = sh.tiles * a.n_items;
  for (const int budget : {55 * 1024, 110 * 1024})  // of the two buffers' one
    for (sh.so = 16; sh.so >= (budget < 64 * 1024 ? 8 : 1); --sh.so) {
      const int64_t pos = ((int64_t)nb * (8 * sh.tiles + sh.so - 1) * sh.pos_bytes + 15) / 16 * 16;
      const int64_t bytes = pos + (int64_t)sh.so * a.table_width * 4;
      if (bytes <= budget) {
        sh.stage_bytes = (int)bytes;
        return nb;
      }
    }
  return 0;
}

int check_common(const char* what, const void* x, const float* table, const int* items, int n_items, const int* win_cnt, const int* win_lo,
                 const int* win_off, int rows, int nlon, int batch, int width, int halo, int table_width, int dtype) {
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_BF16, GM_ERR_UNSUPPORTED, "%s: node fields are float32 or bfloat16", what);
  GM_REQUIRE(x && table && items && win_cnt && win_lo && win_off, GM_ERR_ARGUMENT, "%s: null pointer", what);
  GM_REQUIRE(rows > 0 && nlon > 0 && batch > 0 && width > 0 && halo >= 0 && n_items > 0, GM_ERR_ARGUMENT, "%s: empty or negative sizes", what);
  GM_REQUIRE(nlon % LON == 0, GM_ERR_UNSUPPORTED, "%s: the number of longitudes must be a multiple of %d", what, LON);
  GM_REQUIRE(width % 2 == 0 && table_width % 4 == 0, GM_ERR_UNSUPPORTED,
             "%s: the field width must be even and the table width a multiple of 4 (8- and 16-byte accesses)", what);
  GM_REQUIRE(reinterpret_cast<uintptr_t>(x) % 8 == 0 && reinterpret_cast<uintptr_t>(table) % 16 == 0, GM_ERR_ARGUMENT,
             "%s: the field must sit on an 8-byte and the table on a 16-byte boundary", what);
  return GM_OK;
}

}  // namespace
}  // namespace gmb

using namespace gmb;

// y = table applied along the windows.  order: n_order target rows (any subset, any order).  transpose != 0 applies the
// transposed matrices (the windows and the table are then the transposed ones: gradient with respect to the field).
static int conv_apply(bool tensor_cores, const void* x, const float* table, const int32_t* items, int n_items, const int32_t* win_cnt, const int32_t* win_lo,
                      const int32_t* win_off, const int32_t* order, int n_order, int rows, int nlon, int batch, int width, int halo, int table_width,
                      int transpose, int dtype, void* y, void* stream) {
  if (n_order == 0) return GM_OK;
  if (int status = check_common("gm_lattice_conv_apply", x, table, items, n_items, win_cnt, win_lo, win_off, rows, nlon, batch, width, halo,
                                table_width, dtype))
    return status;
  GM_REQUIRE(order && y && n_order > 0 && n_order <= 65535, GM_ERR_ARGUMENT, "gm_lattice_conv_apply: bad row list");
  ConvArgs a{};
  a.x = x; a.table = table; a.items = items; a.win_cnt = win_cnt; a.win_lo = win_lo; a.win_off = win_off; a.order = order; a.y = y;
  a.n_items = n_items; a.rows = rows; a.nlon = nlon; a.batch = batch; a.width = width; a.halo = halo; a.table_width = table_width;
  a.transpose = transpose;
  cudaStream_t cs = (cudaStream_t)stream;
  GM_REQUIRE(!tensor_cores || (dtype == GM_BF16 && lconv::tensor_cores_can(a)), GM_ERR_UNSUPPORTED,
             "gm_lattice_conv_apply_tc: bfloat16 fields whose rows are whole 16-byte words on 16-byte boundaries");
  if (tensor_cores ? lconv::tensor_cores_hold(a) : dtype == GM_BF16 && lconv::tensor_cores_apply(a)) return lconv::apply_tc(a, n_order, cs);
  const int elem = dtype == GM_F32 ? 4 : 2;
  StagedShape sh{};
  const int nb = staged_shape(a, elem, n_order, sh);
  if (nb > 0) {
    const size_t smem = 2 * (size_t)sh.stage_bytes;
    const dim3 grid((nlon / 8 + sh.tiles - 1) / sh.tiles, n_order, (batch + nb - 1) / nb);
    GM_REQUIRE(grid.z <= 65535, GM_ERR_LIMIT, "gm_lattice_conv_apply: batch too large");
    auto go = [&](auto kernel) {
      const int st = allow_smem(kernel, smem, "gm_lattice_conv_apply");
      if (st != GM_OK) return st;
      kernel<<<grid, sh.threads, smem, cs>>>(a, sh);
      return launch_status("gm_lattice_conv_apply");
    };
    auto pick = [&](auto tag) {
      using S = decltype(tag);
      return nb == 2 ? go(conv_apply_staged_kernel<S, 2>) : go(conv_apply_staged_kernel<S, 1>);
    };
    return dtype == GM_F32 ? pick(float()) : pick(__nv_bfloat16());
  }
  // what a stage cannot hold: more items than a CTA has threads, or rows so wide that 8 + 1 positions outgrow shared memory
  const int threads = min(THREADS, (n_items + 31) / 32 * 32);
  const int pair = batch >= 2 ? 2 : 1;
  GM_REQUIRE((batch + pair - 1) / pair <= 65535, GM_ERR_LIMIT, "gm_lattice_conv_apply: batch too large");
  dim3 grid(nlon / LON, n_order, (batch + pair - 1) / pair);
#define GM_APPLY(S, NB) conv_apply_kernel<S, NB, LON><<<grid, threads, 0, cs>>>(a)
  if (dtype == GM_F32) {
    if (pair == 2) GM_APPLY(float, 2); else GM_APPLY(float, 1);
  } else {
    if (pair == 2) GM_APPLY(__nv_bfloat16, 2); else GM_APPLY(__nv_bfloat16, 1);
  }
#undef GM_APPLY
  return launch_status("gm_lattice_conv_apply");
}

extern "C" int gm_lattice_conv_apply(const void* x, const float* table, const int32_t* items, int n_items, const int32_t* win_cnt, const int32_t* win_lo,
                                     const int32_t* win_off, const int32_t* order, int n_order, int rows, int nlon, int batch, int width, int halo,
                                     int table_width, int transpose, int dtype, void* y, void* stream) {
  return conv_apply(false, x, table, items, n_items, win_cnt, win_lo, win_off, order, n_order, rows, nlon, batch, width, halo, table_width, transpose,
                    dtype, y, stream);
}

extern "C" int gm_lattice_conv_apply_tc(const void* x, const float* table, const int32_t* items, int n_items, const int32_t* win_cnt, const int32_t* win_lo,
                                        const int32_t* win_off, const int32_t* order, int n_order, int rows, int nlon, int batch, int width, int halo,
                                        int table_width, int transpose, int dtype, void* y, void* stream) {
  return conv_apply(true, x, table, items, n_items, win_cnt, win_lo, win_off, order, n_order, rows, nlon, batch, width, halo, table_width, transpose,
                    dtype, y, stream);
}

// dtable[entry] = sum over longitudes and samples of g (target) (x) x (source).  blocks: (n_blocks, 2) int32 = (window
// index = target row * (2 * halo + 1) + source row - target row + halo, first offset), 8 offsets each; entries no block
// covers are left untouched.
static int conv_table_grad(bool tensor_cores, const void* g, const void* x, const int32_t* items, int n_items, const int32_t* win_cnt, const int32_t* win_lo,
                           const int32_t* win_off, const int32_t* blocks, int64_t n_blocks, int rows, int nlon, int batch, int width, int halo,
                           int table_width, int dtype, float* dtable, void* stream) {
  if (n_blocks == 0) return GM_OK;
  if (int status = check_common("gm_lattice_conv_table_grad", x, dtable, items, n_items, win_cnt, win_lo, win_off, rows, nlon, batch, width,
                                halo, table_width, dtype))
    return status;
  GM_REQUIRE(g && blocks && n_blocks > 0 && n_blocks < (int64_t)1 << 31, GM_ERR_ARGUMENT, "gm_lattice_conv_table_grad: bad block list");
  ConvArgs a{};
  a.x = x; a.g = g; a.items = items; a.win_cnt = win_cnt; a.win_lo = win_lo; a.win_off = win_off; a.order = blocks; a.dtable = dtable;
  a.n_items = n_items; a.rows = rows; a.nlon = nlon; a.batch = batch; a.width = width; a.halo = halo; a.table_width = table_width;
  const int threads = min(THREADS, (n_items + 31) / 32 * 32);
  const int nb = batch >= 2 ? 2 : 1;  // four samples' windows would take every register a thread can have
  cudaStream_t cs = (cudaStream_t)stream;
  GM_REQUIRE(!tensor_cores || (dtype == GM_BF16 && lconv::tensor_cores_can(a)), GM_ERR_UNSUPPORTED,
             "gm_lattice_conv_table_grad_tc: bfloat16 fields whose rows are whole 16-byte words on 16-byte boundaries");
  if (tensor_cores || (dtype == GM_BF16 && lconv::tensor_cores_table_grad(a))) return lconv::table_grad_tc(a, n_blocks, cs);
#define GM_GRAD(S, NB) conv_table_grad_kernel<S, NB><<<(unsigned)n_blocks, threads, 0, cs>>>(a)
  if (dtype == GM_F32) {
    if (nb == 2) GM_GRAD(float, 2); else GM_GRAD(float, 1);
  } else {
    if (nb == 2) GM_GRAD(__nv_bfloat16, 2); else GM_GRAD(__nv_bfloat16, 1);
  }
#undef GM_GRAD
  return launch_status("gm_lattice_conv_table_grad");
}

extern "C" int gm_lattice_conv_table_grad(const void* g, const void* x, const int32_t* items, int n_items, const int32_t* win_cnt,
                                          const int32_t* win_lo, const int32_t* win_off, const int32_t* blocks, int64_t n_blocks, int rows, int nlon,
                                          int batch, int width, int halo, int table_width, int dtype, float* dtable, void* stream) {
  return conv_table_grad(false, g, x, items, n_items, win_cnt, win_lo, win_off, blocks, n_blocks, rows, nlon, batch, width, halo, table_width, dtype,
                         dtable, stream);
}

extern "C" int gm_lattice_conv_table_grad_tc(const void* g, const void* x, const int32_t* items, int n_items, const int32_t* win_cnt,
                                             const int32_t* win_lo, const int32_t* win_off, const int32_t* blocks, int64_t n_blocks, int rows, int nlon,
                                             int batch, int width, int halo, int table_width, int dtype, float* dtable, void* stream) {
  return conv_table_grad(true, g, x, items, n_items, win_cnt, win_lo, win_off, blocks, n_blocks, rows, nlon, batch, width, halo, table_width, dtype,
                         dtable, stream);
}

// The table of per-entry coefficients (dtable null: forward, writes table) or the coefficients' gradients from the table's
// (writes drc, dcc).  rc (entries, a0), cc (entries, width), weights (entries), tau / omega (entries, nf, 2), items
// (n_complex, 3) as conv_fold_kernel reads them; table_width = a0 rounded up to 4, plus 4 per complex copy.
extern "C" int gm_lattice_conv_fold(const float* rc, const float* cc, const float* weights, const float* tau, const float* omega,
                                    const int32_t* items, const float* dtable, int64_t entries, int a0, int width, int n_complex, int nf,
                                    float* table, float* drc, float* dcc, void* stream) {
  if (entries == 0) return GM_OK;
  const int padded = (a0 + 3) / 4 * 4;
  GM_REQUIRE(entries > 0 && entries < (int64_t)1 << 31 && a0 >= 0 && width >= 0 && n_complex >= 0 && nf >= 0, GM_ERR_ARGUMENT, "gm_lattice_conv_fold: bad sizes");
  GM_REQUIRE(weights && (n_complex == 0 || (tau && omega && items)), GM_ERR_ARGUMENT, "gm_lattice_conv_fold: null pointer");
  GM_REQUIRE(dtable ? (a0 == 0 || drc) && (n_complex == 0 || dcc) : table && (a0 == 0 || rc) && (n_complex == 0 || cc), GM_ERR_ARGUMENT,
             "gm_lattice_conv_fold: null pointer");
  GM_REQUIRE(reinterpret_cast<uintptr_t>(table) % 16 == 0 && reinterpret_cast<uintptr_t>(dtable) % 16 == 0 && reinterpret_cast<uintptr_t>(tau) % 8 == 0 &&
                 reinterpret_cast<uintptr_t>(omega) % 8 == 0, GM_ERR_ARGUMENT, "gm_lattice_conv_fold: misaligned table or phases");
  FoldArgs a{rc, cc, weights, reinterpret_cast<const float2*>(tau), reinterpret_cast<const float2*>(omega), items, dtable, table, drc, dcc,
             a0, padded, width, n_complex, nf, padded + 4 * n_complex};
  if (dtable) conv_fold_kernel<true><<<(unsigned)entries, 128, 0, (cudaStream_t)stream>>>(a);
  else conv_fold_kernel<false><<<(unsigned)entries, 128, 0, (cudaStream_t)stream>>>(a);
  return launch_status("gm_lattice_conv_fold");
}
