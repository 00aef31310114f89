// Lattice convolution of bfloat16 fields on the tensor cores (the operation and its table: lattice_conv.cu).
//
// A window's correlation along the longitudes has no contraction over channels, but it becomes a matrix product per
// channel pair (a complex copy, or two scalar channels) when the longitudes are cut into tiles of 8, l = 8 t + s:
//
//   apply       y[8 t + s] = sum over r  T[s, r] x[8 t + r],   T[s, r] = M[r - s]  (0 outside the window)
//               rows m = (s, component), columns t, contraction over (r, component): m16n8k16, 8 positions r per k-step
//   table_grad  P[s, r] = sum over t  g[8 t + s] x[8 t + r],   dM[d] = sum over s  P[s, s + d]
//               rows m = (s, component of g), columns (r, component of x), contraction over t, 16 tiles per k-step
//
// Of the (s, r) pairs of a window of cnt offsets 8 cnt in 8 (7 + cnt), rounded up to 8, are wanted: half at cnt = 8.
// Precision: field values are bfloat16 as they are.  The table is float32, so apply writes each of its numbers as a sum of three
// bfloat16 (8 + 8 + 8 bits: exact) and takes three products, smallest first.  An mma cuts its sum off instead of rounding it, so
// no chain is longer than one k-step (8 positions): its sum is added in float32, rounded to nearest.  Root mean square error
// against float64 of sums of N(0, 1) terms that cancel, one chain through all windows / this way / the FMA kernel's single
// additions: rings of 512, terms in order of size 9.5e-4 / 4.9e-5 / 1.3e-4, in random order 1.3e-4 / 6.0e-6 / 1.7e-5; 24 x 48, radius
// 2.5 pi / 24, 6.4e-6 / 1.1e-6 / 3.2e-6 and 2.1e-6 / 4.3e-7 / 1.1e-6.  It costs a fifth of apply's time (256 x 512, radius
// 2 pi / 256, 64 x (m <= 2): 322 -> 406 us; by the FMA kernel 469).
//
// In shared memory a node's 32 columns (64 bytes) sit at [position % 8][position / 8], rows of 80 bytes: a lane reads four
// channel pairs of one position with one 16-byte load, the lanes of a load on different banks.  The (re, im) words are B
// fragments of apply as they are; table_grad contracts over positions and pairs the words of t and t + 1 with two byte
// permutations.
#include "lattice_conv.cuh"

namespace gmb {
namespace lconv {
namespace {

constexpr int TC_THREADS = 256;         // 8 warps: 4 groups of 4 channel pairs x 2
constexpr int TC_COLS = 32;             // columns of the field per CTA
constexpr int TC_PAIRS = TC_COLS / 2;   // channel pairs
constexpr int TC_PITCH = 5;             // 16-byte words per staged position (4 and one of padding)

__device__ __forceinline__ void mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_first(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {  // d = a * b
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// d += a * b with the addition to d rounded to nearest
__device__ __forceinline__ void mma_add(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  float p[4];
  mma_first(p, a[0], a[1], a[2], a[3], b0, b1);
#pragma unroll
  for (int x = 0; x < 4; ++x) d[x] += p[x];
}
// 16 bytes global -> shared, asynchronously; bytes = 0 writes zeros
__device__ __forceinline__ void copy16(uint4* dst, const void* src, int bytes) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(addr), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Staged copies of `count` positions from longitude `lon` of a row (cyclic) on: position q to [q % 8][q / 8], SP 16-byte words
// between the eight.  Columns beyond the field's are zeros.
template <int SP>
__device__ __forceinline__ void stage_positions(uint4* dst, const unsigned char* row, int lon, int count, int nlon, int row_bytes, int col_byte) {
  const int k = threadIdx.x & 3, byte = col_byte + 16 * k;
  const bool in = byte < row_bytes;
  const unsigned char* src = row + (in ? byte : 0);
  int at = lon + ((int)threadIdx.x >> 2);
  while (at >= nlon) at -= nlon;
  const int step = (TC_THREADS / 4) % nlon;
  for (int q = threadIdx.x >> 2; q < count; q += TC_THREADS / 4) {
    copy16(dst + (q & 7) * SP + (q >> 3) * TC_PITCH + k, src + (size_t)at * row_bytes, in ? 16 : 0);
    at += step;
    if (at >= nlon) at -= nlon;
  }
}

struct PairItem {
  int kind, fcol;  // -1: no item on these columns
};
__device__ __forceinline__ void find_items(const ConvArgs& a, int col0, PairItem* pairs_s) {
  if (threadIdx.x < TC_PAIRS) pairs_s[threadIdx.x] = PairItem{-1, 0};
  __syncthreads();
  for (int x = threadIdx.x; x < a.n_items; x += TC_THREADS) {
    const int col = a.items[3 * x + 1] - col0;
    if (col >= 0 && col < TC_COLS) pairs_s[col >> 1] = PairItem{a.items[3 * x], a.items[3 * x + 2]};
  }
  __syncthreads();
}

// ----------------------------------------------------------------------------------------------------------- table_grad
constexpr int TG_TILES = 32;                      // tiles t per stage: two k-steps
constexpr int TG_SPG = TG_TILES * TC_PITCH + 1;   // odd: the lanes' eight s fall on different banks beside their four t
constexpr int TG_SPX = (TG_TILES + 4) * TC_PITCH + 1;
constexpr int TG_STAGE = 8 * (TG_SPG + TG_SPX);   // 16-byte words
constexpr int TG_PS = 18;                         // floats between the s of a P block
constexpr int TG_BLOCK = 8 * TG_PS;               // floats of a P block: 8 s x 16 r
constexpr int TG_PAIR = 4 * TG_BLOCK + 2;         // floats of a channel pair's four: the pairs start on different banks
constexpr int TG_MERGE = 3;                       // blocks of 8 offsets one CTA takes: 24 + 7 positions are four groups of 8
static_assert(2 * TC_PAIRS * TG_PAIR * 4 <= 2 * TG_STAGE * 16, "the P blocks reuse the stages");

// One CTA: up to three consecutive blocks (of 8 offsets) of one window, 32 columns.  A window with up to 9 offsets has one or
// two groups of 8 positions: the two warps of a channel group then split the contraction; with more they split the groups.
__global__ void __launch_bounds__(TC_THREADS, 2) conv_table_grad_tc_kernel(const ConvArgs a, int n_blocks) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PairItem pairs_s[TC_PAIRS];
  const int block = blockIdx.x, w = a.order[2 * block], d0 = a.order[2 * block + 1], b8 = d0 / 8;
  auto is = [&](int x, int d) { return a.order[2 * x] == w && a.order[2 * x + 1] == d; };
  if (b8 % TG_MERGE != 0 && block > 0 && is(block - 1, d0 - 8)) return;  // an earlier block's CTA takes this one too
  int merged = 1;
  while ((b8 + merged) % TG_MERGE != 0 && block + merged < n_blocks && is(block + merged, d0 + 8 * merged)) ++merged;
  const int span = 2 * a.halo + 1, row = w / span, j = row + w % span - a.halo;
  const int valid = min(8 * merged, a.win_cnt[w] - d0), groups = (7 + valid + 7) / 8;
  const int col0 = blockIdx.y * TC_COLS, row_bytes = 2 * a.width;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, cg = warp & 3, half = warp >> 2;
  const bool split_k = groups <= 2;
  const int first_group = split_k ? 0 : 2 * half, mine = min(groups - first_group, 2);
  const int T = a.nlon / 8, chunks = (T + TG_TILES - 1) / TG_TILES, stages = chunks * a.batch;
  find_items(a, col0, pairs_s);
  int shift = (a.win_lo[w] + d0) % a.nlon;
  if (shift < 0) shift += a.nlon;
  const size_t sample = (size_t)a.rows * a.nlon * row_bytes;
  const unsigned char* grow = static_cast<const unsigned char*>(a.g) + (size_t)row * a.nlon * row_bytes;
  const unsigned char* xrow = static_cast<const unsigned char*>(a.x) + (size_t)j * a.nlon * row_bytes;
  uint4* const stage_s = reinterpret_cast<uint4*>(smem);
  auto issue = [&](int s) {
    const int b = s / chunks, t0 = (s - b * chunks) * TG_TILES, tl = min(TG_TILES, T - t0);
    uint4* dst = stage_s + (s & 1) * TG_STAGE;
    stage_positions<TG_SPG>(dst, grow + b * sample, 8 * t0, 8 * tl, a.nlon, row_bytes, 2 * col0);
    stage_positions<TG_SPX>(dst + 8 * TG_SPG, xrow + b * sample, shift + 8 * t0, 8 * (tl + groups - 1), a.nlon, row_bytes, 2 * col0);
    commit();
  };
  float acc[4][2][2][4];  // channel pair, group, component of x: rows (s = g: component 0 of g, g + 8: 1), columns r = 2 c, 2 c + 1
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[p][n][q][x] = 0.f;

  issue(0);
  int k_index = 0;
  for (int s = 0; s < stages; ++s) {
    if (s + 1 < stages) {
      issue(s + 1);
      wait_copies<1>();
    } else {
      wait_copies<0>();
    }
    __syncthreads();
    const int t0 = (s % chunks) * TG_TILES, tl = min(TG_TILES, T - t0);
    const uint4* gs = stage_s + (s & 1) * TG_STAGE + g * TG_SPG + cg;
    const uint4* xs = stage_s + (s & 1) * TG_STAGE + 8 * TG_SPG + g * TG_SPX + first_group * TC_PITCH + cg;
    // the words of tile t = k0 + 2 c (+ 1, + 8, + 9); both operands are zero beyond the last tile
    auto step = [&](int k0, auto is_ragged) {
      auto word = [&](const uint4* base, int t, int n) {
        uint4 v = base[(t + n) * TC_PITCH];
        if (decltype(is_ragged)::value && t >= tl) v = make_uint4(0, 0, 0, 0);
        return v;
      };
      const int t = k0 + 2 * c;
      unsigned fa[4][4];
      {
        const uint4 v0 = word(gs, t, 0), v1 = word(gs, t + 1, 0), v8 = word(gs, t + 8, 0), v9 = word(gs, t + 9, 0);
        const unsigned w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
        const unsigned w8[4] = {v8.x, v8.y, v8.z, v8.w}, w9[4] = {v9.x, v9.y, v9.z, v9.w};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          fa[p][0] = __byte_perm(w0[p], w1[p], 0x5410);
          fa[p][1] = __byte_perm(w0[p], w1[p], 0x7632);
          fa[p][2] = __byte_perm(w8[p], w9[p], 0x5410);
          fa[p][3] = __byte_perm(w8[p], w9[p], 0x7632);
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        if (n < mine) {
          const uint4 v0 = word(xs, t, n), v1 = word(xs, t + 1, n), v8 = word(xs, t + 8, n), v9 = word(xs, t + 9, n);
          const unsigned w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
          const unsigned w8[4] = {v8.x, v8.y, v8.z, v8.w}, w9[4] = {v9.x, v9.y, v9.z, v9.w};
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            mma_add(acc[p][n][0], fa[p], __byte_perm(w0[p], w1[p], 0x5410), __byte_perm(w8[p], w9[p], 0x5410));
            mma_add(acc[p][n][1], fa[p], __byte_perm(w0[p], w1[p], 0x7632), __byte_perm(w8[p], w9[p], 0x7632));
          }
        }
      }
    };
    for (int k0 = 0; k0 < tl; k0 += 16, ++k_index) {
      if (split_k && (k_index & 1) != half) continue;
      if (k0 + 16 <= tl) step(k0, std::false_type{});
      else step(k0, std::true_type{});
    }
    __syncthreads();
  }

  // ---- P blocks (half, channel pair, components) to shared memory, then the sums along their diagonals, always in one order
  float* const p_s = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float* at = p_s + (half * TC_PAIRS + 4 * cg + p) * TG_PAIR + q * TG_BLOCK + g * TG_PS + 8 * n + 2 * c;
        *reinterpret_cast<float2*>(at) = make_float2(acc[p][n][q][0], acc[p][n][q][1]);                 // component 0 of g
        *reinterpret_cast<float2*>(at + 2 * TG_BLOCK) = make_float2(acc[p][n][q][2], acc[p][n][q][3]);  // component 1
      }
  __syncthreads();
  for (int x = threadIdx.x; x < TC_PAIRS * valid; x += TC_THREADS) {
    const int p = x % TC_PAIRS, d = x / TC_PAIRS;
    const PairItem it = pairs_s[p];
    if (it.kind < 0) continue;
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float sum = 0.f;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int r = s + d;
        const float* at = p_s + p * TG_PAIR + q * TG_BLOCK + s * TG_PS;
        constexpr int OTHER = TC_PAIRS * TG_PAIR;
        if (split_k) sum += at[r] + at[r + OTHER];
        else sum += r < 16 ? at[r] : at[r - 16 + OTHER];
      }
      v[q] = sum;
    }
    float* out = a.dtable + (size_t)(a.win_off[w] + d0 + d) * a.table_width + it.fcol;
    if (it.kind == 0) *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<float2*>(out) = make_float2(v[0], v[3]);
  }
}

// ---------------------------------------------------------------------------------------------------------------- apply
constexpr int AP_TILES = 64;                              // tiles of 8 longitudes per CTA
constexpr int AP_OFFSETS = 17;                            // offsets per stage: 17 + 7 positions are three k-steps
constexpr int AP_SP = (AP_TILES + 2) * TC_PITCH;          // = 2 mod 8: the lanes' four r fall on different banks beside their two t
static_assert(AP_SP % 8 == 2, "conflict-free 16-byte loads");
constexpr int AP_SLOTS = 32;                              // offsets -7 .. 24 of a split table row, 8 bytes each
constexpr int AP_PAIR = 3 * AP_SLOTS + 1;                 // 8-byte words per channel pair
constexpr int AP_STAGE = 8 * AP_SP + (TC_PAIRS * AP_PAIR * 8 + 15) / 16;  // 16-byte words

// What a CTA works on: 32 columns of a target row's longitudes 8 t0 .. 8 (t0 + tl) - 1, one sample (`field`)
struct ApplyTile {
  const unsigned char* field;
  int row, t0, tl, col0;
};
// Stages: offsets [d, d + n) of a window of the row
struct ApplyStage {
  int w, d, n, cnt;  // w = 2 halo + 1: past the last
};
__device__ __forceinline__ ApplyStage first_stage(const ConvArgs& a, int row, int w) {  // of the windows from w on
  const int span = 2 * a.halo + 1;
  for (; w < span; ++w) {
    const int j = row + w - a.halo;
    if (j < 0 || j >= a.rows) continue;
    const int cnt = a.win_cnt[row * span + w];
    if (cnt > 0) return ApplyStage{w, 0, min(AP_OFFSETS, cnt), cnt};
  }
  return ApplyStage{span, 0, 0, 0};
}
__device__ __forceinline__ ApplyStage next_stage(const ConvArgs& a, int row, const ApplyStage& s) {
  const int d = s.d + s.n;
  return d < s.cnt ? ApplyStage{s.w, d, min(AP_OFFSETS, s.cnt - d), s.cnt} : first_stage(a, row, s.w + 1);
}
__device__ __forceinline__ void issue_stage(const ConvArgs& a, const ApplyTile& t, const ApplyStage& s, uint4* dst) {
  int lon = (8 * t.t0 + a.win_lo[t.row * (2 * a.halo + 1) + s.w] + s.d) % a.nlon;
  if (lon < 0) lon += a.nlon;
  const int steps = (7 + s.n + 7) / 8, row_bytes = 2 * a.width;
  stage_positions<AP_SP>(dst, t.field + (size_t)(t.row + s.w - a.halo) * a.nlon * row_bytes, lon, 8 * (t.tl + steps - 1), a.nlon, row_bytes, 2 * t.col0);
  commit();
}
// The matrix of channel pair `it` at offset d of the stage
__device__ __forceinline__ float4 table_matrix(const ConvArgs& a, int row, const ApplyStage& s, int d, PairItem it) {
  const float* f = a.table + (size_t)(a.win_off[row * (2 * a.halo + 1) + s.w] + s.d + d) * a.table_width + it.fcol;
  if (it.kind == 0) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(f));
    return a.transpose ? make_float4(v.x, v.z, v.y, v.w) : v;
  }
  const float2 v = __ldg(reinterpret_cast<const float2*>(f));
  return make_float4(v.x, 0.f, 0.f, v.y);
}
// Column col of the tile's row in the result
__device__ __forceinline__ __nv_bfloat16* apply_output(const ConvArgs& a, const ApplyTile& t, int b, int col) {
  return static_cast<__nv_bfloat16*>(a.y) + ((size_t)b * a.rows + t.row) * a.nlon * a.width + col;
}

// The CTA's outputs whose sums were not finite, by themselves: such a sum may owe it to a value outside its window (0 x Inf) or
// to another component, so it is formed again from its own neighbours alone, on the FMA pipe from the staged positions.  A warp
// leaves out the channel pairs that have no such output, or none that is not NaN already (and stays so).  `bad`: bit
// 8 p + 2 i + e = channel pair p at longitude 8 (8 (half + 2 i) + 2 c + e) + g.  128 x 256, radius 4 pi / 128, batch 2, 32 x (m <= 2): a
// field of NaN 324 us, one Inf in a polar row (whose rings all see it) 567, nothing 264; the FMA kernel 344 whatever it meets, each
// output by its own thread from global memory 9 058 and 1 196.
__device__ __noinline__ void apply_again(const ConvArgs& a, const ApplyTile& tile, int b, uint4* stage_s, const PairItem* pairs_s, unsigned bad) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, cg = warp & 3, half = warp >> 2;
  float2 y[4][4][2];
  bool open[4];  // pairs the warp still works on
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    open[p] = __any_sync(0xffffffffu, bad >> 8 * p & 0xff);
#pragma unroll
    for (int i = 0; i < 4; ++i) y[p][i][0] = y[p][i][1] = make_float2(0.f, 0.f);
  }
  ApplyStage s = first_stage(a, tile.row, 0);
  if (s.w <= 2 * a.halo) issue_stage(a, tile, s, stage_s);
  int buf = 0;
  while (s.w <= 2 * a.halo) {
    const ApplyStage nxt = next_stage(a, tile.row, s);
    if (nxt.w <= 2 * a.halo) {
      issue_stage(a, tile, nxt, stage_s + (buf ^ 1) * AP_STAGE);
      wait_copies<1>();
    } else {
      wait_copies<0>();
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if (!open[p]) continue;
      const PairItem it = pairs_s[4 * cg + p];
      const unsigned* words = reinterpret_cast<const unsigned*>(stage_s + buf * AP_STAGE + cg) + p;
      float4 next = table_matrix(a, tile.row, s, 0, it);
      for (int d = 0; d < s.n; ++d) {
        const float4 m = next;
        next = table_matrix(a, tile.row, s, min(d + 1, s.n - 1), it);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int q = 8 * (8 * (half + 2 * i) + 2 * c + e) + g + d;
            const unsigned w = words[4 * ((q & 7) * AP_SP + (q >> 3) * TC_PITCH)];
            const float vx = __uint_as_float(w << 16), vy = __uint_as_float(w & 0xffff0000u);
            float2& out = y[p][i][e];
            if (it.kind == 0) {
              out.x = fmaf(m.x, vx, fmaf(m.y, vy, out.x));
              out.y = fmaf(m.z, vx, fmaf(m.w, vy, out.y));
            } else {
              out.x = fmaf(m.x, vx, out.x);
              out.y = fmaf(m.w, vy, out.y);
            }
          }
      }
      bool undecided = false;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) undecided = undecided || ((bad >> (8 * p + 2 * i + e) & 1) && !(isnan(y[p][i][e].x) && isnan(y[p][i][e].y)));
      open[p] = __any_sync(0xffffffffu, undecided);
    }
    if (!__syncthreads_or(open[0] || open[1] || open[2] || open[3])) break;
    s = nxt;
    buf ^= 1;
  }
  wait_copies<0>();
  __nv_bfloat16* at = apply_output(a, tile, b, tile.col0 + 8 * cg);
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (bad >> (8 * p + 2 * i + e) & 1) {
          const int l = 8 * (tile.t0 + 8 * (half + 2 * i) + 2 * c + e) + g;
          *reinterpret_cast<__nv_bfloat162*>(at + (size_t)l * a.width + 2 * p) = __floats2bfloat162_rn(y[p][i][e].x, y[p][i][e].y);
        }
}

// (x, y) = sum of three bfloat16 pairs, largest first
__device__ __forceinline__ void split3(float x, float y, unsigned (&w)[3]) {
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    w[s] = *reinterpret_cast<const unsigned*>(&h);
    x -= __uint_as_float(w[s] << 16);
    y -= __uint_as_float(w[s] & 0xffff0000u);
  }
}

__global__ void __launch_bounds__(TC_THREADS, 2) conv_apply_tc_kernel(const __grid_constant__ ConvArgs a, int col_blocks, int lon_blocks) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PairItem pairs_s[TC_PAIRS];
  int x = blockIdx.x;
  const int cb = x % col_blocks;
  x /= col_blocks;
  const int lb = x % lon_blocks;
  x /= lon_blocks;
  const int b = x % a.batch, row = a.order[x / a.batch];  // heaviest rows first
  const int col0 = cb * TC_COLS, row_bytes = 2 * a.width, span = 2 * a.halo + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, cg = warp & 3, half = warp >> 2;
  const int T = a.nlon / 8, t0 = lb * AP_TILES, tl = min(AP_TILES, T - t0), tiles = (tl + 7) / 8;
  find_items(a, col0, pairs_s);
  const unsigned char* field = static_cast<const unsigned char*>(a.x) + (size_t)b * a.rows * a.nlon * row_bytes;
  uint4* const stage_s = reinterpret_cast<uint4*>(smem);

  const ApplyTile tile{field, row, t0, tl, col0};
  // this thread's two slots of the split table: a channel pair and the offsets slot - 7
  const int tp = threadIdx.x & (TC_PAIRS - 1), ts = threadIdx.x / TC_PAIRS;
  const PairItem item = pairs_s[tp];
  auto fetch = [&](const ApplyStage& s, float4 (&m)[2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int d = ts + 16 * i - 7;
      m[i] = d >= 0 && d < s.n && item.kind >= 0 ? table_matrix(a, row, s, d, item) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto place = [&](int buf, const float4 (&m)[2]) {
    uint2* dst = reinterpret_cast<uint2*>(stage_s + buf * AP_STAGE + 8 * AP_SP) + tp * AP_PAIR + ts;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      unsigned w0[3], w1[3];
      split3(m[i].x, m[i].y, w0);
      split3(m[i].z, m[i].w, w1);
#pragma unroll
      for (int s = 0; s < 3; ++s) dst[s * AP_SLOTS + 16 * i] = make_uint2(w0[s], w1[s]);
    }
  };

  float acc[4][4][4];  // channel pair, tile of 8 t: rows (s = g: component 0, g + 8: component 1), columns t = 2 c, 2 c + 1
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[p][i][v] = 0.f;

  ApplyStage cur = first_stage(a, row, 0);
  float4 m[2];
  if (cur.w < span) {
    issue_stage(a, tile, cur, stage_s);
    fetch(cur, m);
    place(0, m);
  }
  int buf = 0;
  while (cur.w < span) {
    const ApplyStage nxt = next_stage(a, row, cur);
    const bool more = nxt.w < span;
    if (more) {
      issue_stage(a, tile, nxt, stage_s + (buf ^ 1) * AP_STAGE);
      fetch(nxt, m);
      wait_copies<1>();
    } else {
      wait_copies<0>();
    }
    __syncthreads();
    const uint4* xs = stage_s + buf * AP_STAGE + c * AP_SP + cg;
    const uint2* ms = reinterpret_cast<const uint2*>(stage_s + buf * AP_STAGE + 8 * AP_SP) + 4 * cg * AP_PAIR + 7 + c - g;
    const int steps = (7 + cur.n + 7) / 8;
    auto walk = [&](auto mine) {  // tiles half, half + 2, ... of the CTA's (a tile too many reads what a stage left behind: its own columns)
      constexpr int MINE = decltype(mine)::value;
      for (int k = 0; k < steps; ++k) {
        unsigned fb[MINE][2][4];
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
          const uint4* at = xs + (8 * (half + 2 * i) + g + k) * TC_PITCH;
          const uint4 v0 = at[0], v4 = at[4 * AP_SP];
          fb[i][0][0] = v0.x; fb[i][0][1] = v0.y; fb[i][0][2] = v0.z; fb[i][0][3] = v0.w;
          fb[i][1][0] = v4.x; fb[i][1][1] = v4.y; fb[i][1][2] = v4.z; fb[i][1][3] = v4.w;
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const uint2* f = ms + p * AP_PAIR + 8 * k;
          const uint2 l01 = f[2 * AP_SLOTS], l23 = f[2 * AP_SLOTS + 4], m01 = f[AP_SLOTS], m23 = f[AP_SLOTS + 4], h01 = f[0], h23 = f[4];
          float sum[MINE][4];
#pragma unroll
          for (int i = 0; i < MINE; ++i) mma_first(sum[i], l01.x, l01.y, l23.x, l23.y, fb[i][0][p], fb[i][1][p]);
#pragma unroll
          for (int i = 0; i < MINE; ++i) mma(sum[i], m01.x, m01.y, m23.x, m23.y, fb[i][0][p], fb[i][1][p]);
#pragma unroll
          for (int i = 0; i < MINE; ++i) mma(sum[i], h01.x, h01.y, h23.x, h23.y, fb[i][0][p], fb[i][1][p]);
#pragma unroll
          for (int i = 0; i < MINE; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[p][i][v] += sum[i][v];
        }
      }
    };
    if (tiles > 4) walk(std::integral_constant<int, 4>());
    else if (tiles > 2) walk(std::integral_constant<int, 2>());
    else walk(std::integral_constant<int, 1>());
    if (more) place(buf ^ 1, m);
    __syncthreads();
    cur = nxt;
    buf ^= 1;
  }

  // ---- four channel pairs of a position are 16 bytes of its row
  const int col = col0 + 8 * cg;
  unsigned bad = 0;  // outputs whose sums are not finite
  if (col < a.width) {
    __nv_bfloat16* y = apply_output(a, tile, b, col);
    bool whole = true;
#pragma unroll
    for (int p = 0; p < 4; ++p) whole = whole && pairs_s[4 * cg + p].kind >= 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 8 * (half + 2 * i) + 2 * c + e;
        if (t >= tl) continue;
        unsigned word[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const float2 v = make_float2(acc[p][i][e], acc[p][i][2 + e]);
          if (!(fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY) && pairs_s[4 * cg + p].kind >= 0) bad |= 1u << (8 * p + 2 * i + e);
          const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
          word[p] = *reinterpret_cast<const unsigned*>(&h);
        }
        __nv_bfloat16* at = y + (size_t)(8 * (t0 + t) + g) * a.width;
        if (whole) {
          *reinterpret_cast<uint4*>(at) = make_uint4(word[0], word[1], word[2], word[3]);
        } else {
#pragma unroll
          for (int p = 0; p < 4; ++p)
            if (pairs_s[4 * cg + p].kind >= 0) *reinterpret_cast<unsigned*>(at + 2 * p) = word[p];
        }
      }
  }
  if (__syncthreads_or(bad != 0)) apply_again(a, tile, b, stage_s, pairs_s, bad);
}

}  // namespace

bool tensor_cores_can(const ConvArgs& a) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.g) | reinterpret_cast<uintptr_t>(a.y);
  return a.nlon % 8 == 0 && a.width % 8 == 0 && bits % 16 == 0;
}

// The FMA kernels stay the faster ones where a launch is short or its tiles are mostly padding.  96 shapes from 24 x 24 to
// 256 x 512, batch 1 to 4, widths 24 to 320, us FMA / tensor cores:
//   apply        up to 8 tiles of 8 longitudes leave half of a CTA's warps without one (64 x 64, batch 4, width 320: 53 / 143; 32 x 64,
//                batch 1, width 40: 39 / 47); with one sample and a narrow field the launch is the polar rows' chain of stages, which is
//                longer here (256 x 512, width 40: 367 / 526; 128 x 512, width 96: 371 / 489), from two samples on it is not (91 x 184,
//                width 96: 259 / 170; 45 x 88, width 40: 72 / 66).  Wide fields fill the chip with one sample, and then it is padding
//                that decides (256 x 512, width 320: 848 / 604; 64 x 128, batch 2, width 320: 174 / 199).
//   table_grad   contracts over the tiles, 16 a step: 23 tiles and more are always faster (91 x 184, batch 1, width 80: 75 / 58; 128 x
//                256, width 24: 99 / 50), 16 with four samples in sequence (64 x 128, width 320: 270 / 239; batch 2: 143 / 175), 9 to 15 then
//                where the field is not wide (45 x 88, width 80: 60 / 57, width 320: 132 / 159; 100 x 104: 105 / 103 and 224 / 307).  One
//                block of 32 columns, for which the FMA kernel has less than a warp of items, from 8 tiles on (64 x 64: 22 / 20; 45 x 88:
//                26 / 19); fewer tiles go either way (100 x 48, batch 4: 28 / 32; 24 x 48: 26 / 17).
bool tensor_cores_apply(const ConvArgs& a) {
  const int tiles = a.nlon / 8;
  return tensor_cores_can(a) && tiles > 8 && (a.width < 256 ? a.batch >= 2 : tiles >= 32);
}
bool tensor_cores_table_grad(const ConvArgs& a) {
  const int tiles = a.nlon / 8;
  const bool pays = tiles >= 20 || (tiles >= 8 && a.width <= TC_COLS) || (a.batch >= 4 && (tiles >= 16 || (tiles > 8 && a.width <= 96)));
  return tensor_cores_can(a) && pays;
}

int apply_tc(const ConvArgs& a, int n_order, cudaStream_t stream) {
  const int col_blocks = (a.width + TC_COLS - 1) / TC_COLS, lon_blocks = (a.nlon / 8 + AP_TILES - 1) / AP_TILES;
  const int64_t ctas = (int64_t)col_blocks * lon_blocks * a.batch * n_order;
  GM_REQUIRE(ctas < (1ll << 31), GM_ERR_LIMIT, "gm_lattice_conv_apply: too many tiles");
  const size_t smem = 2 * (size_t)AP_STAGE * 16;
  const int st = allow_smem(conv_apply_tc_kernel, smem, "gm_lattice_conv_apply");
  if (st != GM_OK) return st;
  conv_apply_tc_kernel<<<(unsigned)ctas, TC_THREADS, smem, stream>>>(a, col_blocks, lon_blocks);
  return launch_status("gm_lattice_conv_apply");
}

int table_grad_tc(const ConvArgs& a, int64_t n_blocks, cudaStream_t stream) {
  const int col_blocks = (a.width + TC_COLS - 1) / TC_COLS;
  const size_t smem = 2 * (size_t)TG_STAGE * 16;
  const int st = allow_smem(conv_table_grad_tc_kernel, smem, "gm_lattice_conv_table_grad");
  if (st != GM_OK) return st;
  conv_table_grad_tc_kernel<<<dim3((unsigned)n_blocks, col_blocks), TC_THREADS, smem, stream>>>(a, (int)n_blocks);
  return launch_status("gm_lattice_conv_table_grad");
}

}  // namespace lconv
}  // namespace gmb
