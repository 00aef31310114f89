// The factored steerable kernel (the operation: factored_ops.cu) on the tensor cores, float32.
//
// Both directions are small matrix products over a source's edges: U(e, c) = sum_t h_t(e) Z_t(c) forward, dh(e, t) = sum_c
// W_c(e) Z_t(c) and dZ_t(c) = sum_e h_t(e) W_c(e) backward, t over the trunk's (up to 16) outputs, c over the packed columns.
// Each is m16n8k16 with 16 edges as rows (forward, dh) or as the contraction (dZ).  The constant trunk output h~_0 = 1 has no
// product: Z_0 is added, and the sums of W are dZ_0.
//
// Columns: a block's copies in tiles of four, (re, im) side by side, so a lane's two columns of a tile are one complex number:
// the block factors, and the sum over the blocks of one output, are applied to the accumulators in registers.  A real block is a
// complex one whose imaginary columns are zero.
//
// Precision: every float32 operand is the sum of three bfloat16 (8 + 8 + 8 bits: exactly, mma.cuh), and of the nine products the six that
// reach 2^-24 of the result are taken, in two chains of three, smallest first; everything that is summed over more than one
// k-step (the 16 edges of dZ, the two tiles of dh) is added in float32, rounded to nearest.
// What it measured, 128 x 256, radius 3 pi / 128 (3.0 M edges), 13 blocks to {4, 4, 4}, trunk 16, us on CUDA cores -> here: forward 1 036 -> 731,
// backward 2 463 -> 1 830.  Bound by latency and issue (issue 44 / 46 %, tensor pipe 17 / 14 %): a step of 16 edges is 78 / 168 products
// among 1 600 / 4 400 instructions, most of them the splits, the factors and the records' copies.  With the records read where
// they are (1 245 / 3 225 us) every step waited for its chain of gathers; they are copied a step ahead.  Four tiles a backward warp:
// eight 2 095 us (the loop over tiles, unrolled for its accumulators, outgrew the instruction cache), two 1 946.  168 registers
// and twelve warps an SM instead of sixteen: 2 077.  Errors against float64: 0.85 to 0.98 of the CUDA-core kernels' for rows
// (shorter trunks go to those: FWD_LEAST_K), 0.2 to 0.8 for the gradients; weights' gradients are the same.
// Infinities and numbers of 2^60 and more do not go through the splits: what they are operands of is formed by single
// multiply-adds (a step of the forward, a source of the backward), so that infinite and finite results are those of the
// CUDA-core kernel; NaN spreads as it would there.  128 x 256, 13 blocks to {4, 4, 4}: the test for them takes 1 % of the backward; an
// infinity in one polar node's Z makes the forward 731 -> 1 042, in one row of the gradient the backward 1 838 -> 3 572, and
// nothing but infinities 3 400 and 10 807 (CUDA-core kernels 1 040 and 2 470).
#include <algorithm>
#include <cmath>

#include "factored.cuh"
#include "mma.cuh"

namespace gmb {
namespace factored {
namespace {

constexpr int TRUNK = 16;      // trunk outputs beside the constant one, at most: a k-step
constexpr int ROWS = 16;       // edges per step
constexpr int FWD_WARPS = 2;   // a source's steps are dealt to two warps
constexpr int BWD_TILES = 4;   // tiles of a backward warp: every warp sees all of a source's edges and its own columns
constexpr int MAX_WARPS = 8;
constexpr int DH_PITCH = TRUNK + 2;
constexpr int FWD_CTAS = 64, BWD_CTAS = 64;  // CTAs of the grid per SM

// sum = a b (rows g and g + 8, two columns each) of operands in three parts (largest first), in float32
__device__ __forceinline__ void product(f32x2 (&sum)[2], const unsigned (&a)[3][4], const uint2 (&b)[3], const float (&zero)[4]) {
  float low[4], d[4];
  auto first = [&](float (&to)[4], int p, int q) { mma_first(to, a[p][0], a[p][1], a[p][2], a[p][3], b[q].x, b[q].y, zero); };
  auto next = [&](float (&to)[4], int p, int q) { mma(to, a[p][0], a[p][1], a[p][2], a[p][3], b[q].x, b[q].y); };
  first(low, 2, 0);
  first(d, 1, 0);
  next(low, 0, 2);
  next(d, 0, 1);
  next(low, 1, 1);
  next(d, 0, 0);
  sum[0] = pack2(low[0], low[1]);
  sum[1] = pack2(low[2], low[3]);
  add2(sum[0], d[0], d[1]);
  add2(sum[1], d[2], d[3]);
}
// Operands of 2^60 and more, infinities among them, go to single multiply-adds: of smaller ones no product and no sum here
// overflows, where parts of opposite signs could make a NaN of an infinity.  (NaN goes where it would go there.)
// The larger magnitudes of two pairs of bfloat16, under whatever sign, NaN left out
__device__ __forceinline__ unsigned larger(unsigned x, unsigned y) {
  unsigned m;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(m) : "r"(x), "r"(y));
  return m;
}
__device__ __forceinline__ bool too_large(unsigned m) { return fmaxf(fabsf(__uint_as_float(m << 16)), fabsf(__uint_as_float(m & 0xffff0000u))) >= 0x1p60f; }
__device__ __forceinline__ unsigned transposed(unsigned x) {  // of an 8 x 8 matrix of bfloat16, a row's pairs over four lanes
  unsigned y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
  return y;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(addr), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Four copies of a block, in the order of (output, four copies of it, block)
struct Tile {
  int column;  // of zc (complex) or zr
  int block;
  int output;  // flat output column of the first copy
  int flags;   // copies that exist (of four), those of its output columns << 8, and:
};
// a real block; real part only; the first and the last one of its output columns
constexpr int TILE_REAL = 8, TILE_REAL_OUT = 16, TILE_FIRST = 32, TILE_LAST = 64;

// Tiles of blocks of equally many copies; where they are not, there may be more, and the kernels take several rounds of tiles
inline int likely_tiles(int wc, int wr, int n_blocks) { return n_blocks * (((wc + wr + n_blocks - 1) / n_blocks + 3) / 4); }

// The tiles [base, base + capacity) of all blocks, a thread per block.  Returned: how many there are in all.  Blocks are sorted by
// output offset; those of one offset add into the same columns.
__device__ __forceinline__ int list_tiles(const int32_t* desc, int n_blocks, int base, int capacity, Tile* tiles) {
  int total = 0;
  for (int x = 0; x < n_blocks; ++x) total += (desc[x * FDESC + 2] + 3) / 4;
  for (int b = threadIdx.x; b < n_blocks; b += blockDim.x) {
    const int32_t* d = desc + b * FDESC;
    int first = b, last = b + 1, before = 0;
    while (first > 0 && desc[(first - 1) * FDESC + 6] == d[6]) --first;
    while (last < n_blocks && desc[last * FDESC + 6] == d[6]) ++last;
    for (int x = 0; x < first; ++x) before += (desc[x * FDESC + 2] + 3) / 4;
    const bool real_out = desc[first * FDESC] == 0 || desc[first * FDESC + 7] != 0;
    for (int sub = 0; 4 * sub < d[2]; ++sub) {
      int at = before - base, ahead = 0, behind = 0, columns = 0;
      for (int x = first; x < last; ++x) {
        const int copies = desc[x * FDESC + 2], n = (copies + 3) / 4;
        at += min(n, sub);
        ahead += x < b && n > sub;
        behind += x > b && n > sub;
        columns = max(columns, min(4, copies - 4 * sub));
      }
      at += ahead;
      if (at >= 0 && at < capacity)
        tiles[at] = Tile{d[1] + 4 * sub, b, d[6] + (real_out ? 4 : 8) * sub,
                         min(4, d[2] - 4 * sub) | columns << 8 | (d[0] == 0 ? TILE_REAL : 0) | (real_out ? TILE_REAL_OUT : 0) |
                             (ahead == 0 ? TILE_FIRST : 0) | (behind == 0 ? TILE_LAST : 0)};
    }
  }
  return total;
}

// A step's records in shared memory, a row per edge: trunk outputs, angular and transport phases, the phase one, the powers of rho
// (or the scales), and in the backward the gradient row and the forward's row.  Rows are copied asynchronously in words of 4 or 8
// bytes, a thread keeping its part of the row.
struct Record {
  int angular, transport, one, rho, grad, row, pitch;  // floats
  __host__ __device__ Record(int k, int n_f, int n_rho, int d_out, bool backward) {
    angular = (k - 1 + 1) / 2 * 2;
    transport = angular + 2 * n_f;
    one = transport + 2 * n_f;
    grad = one + 2;
    const int d2 = (d_out + 1) / 2 * 2;
    row = grad + (backward ? d2 : 0);
    rho = row + (backward ? d2 : 0);
    pitch = 2 * ((rho + n_rho + 1) / 2 | 1);  // an odd number of 8-byte words: the rows of a half-warp on different banks
  }
};
struct CopyUnit {  // one word of a row: bytes from src + index * stride on to `to`; by the edge's or (grad) its gradient row's index
  const char* src;
  unsigned stride;
  int to, kind;  // kind: 0 none, 1 a word, 2 a word of the gradient row, 3 one float
};
__device__ __forceinline__ int copy_units(const FArgs<float>& a, int n_rho, int words, bool backward) {
  return (a.k - 1) / words + 4 * a.n_f / words + (backward ? a.d_out / words * (a.rows ? 2 : 1) : 0) + n_rho;
}
__device__ __forceinline__ CopyUnit copy_unit(const FArgs<float>& a, const Record& rec, int n_rho, int words, bool backward, int u) {
  const int h = (a.k - 1) / words, phases = 2 * a.n_f / words, d = backward ? a.d_out / words : 0;
  auto unit = [&](const float* from, int width, int to, int kind) { return CopyUnit{reinterpret_cast<const char*>(from), 4u * width, to, kind}; };
  if (u < h) return unit(a.h + words * u, a.k - 1, words * u, 1);
  u -= h;
  if (u < phases) return unit(a.angular + words * u, 2 * a.n_f, rec.angular + words * u, 1);
  u -= phases;
  if (u < phases) return unit(a.transport + words * u, 2 * a.n_f, rec.transport + words * u, 1);
  u -= phases;
  if (u < d) return unit(a.g + words * u, a.d_out, rec.grad + words * u, 2);
  u -= d;
  if (backward && a.rows) {
    if (u < d) return unit(a.rows + words * u, a.d_out, rec.row + words * u, 1);
    u -= d;
  }
  if (u < n_rho) return unit(a.rho + u, n_rho, rec.rho + u, 3);
  return CopyUnit{nullptr, 0, 0, 0};
}
// Whether every row and table is made of 8-byte words
__device__ __forceinline__ int word_floats(const FArgs<float>& a, bool backward) {
  uintptr_t all = reinterpret_cast<uintptr_t>(a.h) | reinterpret_cast<uintptr_t>(a.angular) | reinterpret_cast<uintptr_t>(a.transport) | (uintptr_t)(a.k - 1) * 4;
  if (backward) all |= reinterpret_cast<uintptr_t>(a.g) | reinterpret_cast<uintptr_t>(a.rows) | (uintptr_t)a.d_out * 4;
  return all % 8 == 0 ? 2 : 1;
}
// The unit of all 16 rows; index(r): the r-th row's, asked for by every thread
template <typename Index>
__device__ __forceinline__ void copy_rows(const CopyUnit& u, int words, float* dst, int pitch, const Index& index) {
  const bool wide = words == 2 && (u.kind == 1 || u.kind == 2), narrow = !wide && u.kind != 0;
  dst += u.to;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float* from = reinterpret_cast<const float*>(u.src + (size_t)index(r) * u.stride);
    if (wide) copy_async<8>(dst + r * pitch, from);
    if (narrow) copy_async<4>(dst + r * pitch, from);
  }
}
// A block's factor e^{i ang phi} e^{i trn gamma} (r / c)^p, from places of the record: no branches
struct Factor {
  int angular, transport, power;  // places of the phases; the power of rho, or the place of the scale
  unsigned conjugate;             // bit 31 / 30: of the angular / transport phase
};
template <bool SCALED>
__device__ __forceinline__ Factor block_place(const int32_t* d, const Record& rec) {
  const bool real = d[0] == 0;  // the factor one
  return Factor{d[3] && !real ? rec.angular + 2 * abs(d[3]) : rec.one, d[4] && !real ? rec.transport + 2 * abs(d[4]) : rec.one,
                real ? (SCALED ? rec.one : 0) : (SCALED ? rec.rho + d[5] : d[5]), (d[3] < 0 ? 0x80000000u : 0u) | (d[4] < 0 ? 0x40000000u : 0u)};
}
template <bool SCALED>
__device__ __forceinline__ float2 record_factor(const float* rec, const Factor& f, float rho) {
  const float2 p = *reinterpret_cast<const float2*>(rec + f.angular), t = *reinterpret_cast<const float2*>(rec + f.transport);
  const float pi = __uint_as_float(__float_as_uint(p.y) ^ (f.conjugate & 0x80000000u)), ti = __uint_as_float(__float_as_uint(t.y) ^ (f.conjugate << 1 & 0x80000000u));
  float s = 1.f;
  if constexpr (SCALED) s = rec[f.power];
  else
    for (int x = 0; x < f.power; ++x) s *= rho;
  return make_float2(s * (p.x * t.x - pi * ti), s * (p.x * ti + pi * t.x));
}
// The trunk's outputs of two edges (their records) as the A operand of 16 edges x 16 outputs; returned: their largest magnitudes
__device__ __forceinline__ unsigned load_trunk(const float* r0, const float* r1, int n, int c, unsigned (&h)[3][4]) {
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int t = 2 * c + 8 * (x >> 1);
    float2 v = make_float2(0.f, 0.f);
    if (t < n) v = *reinterpret_cast<const float2*>((x & 1 ? r1 : r0) + t);
    if (t + 1 >= n) v.y = 0.f;
    unsigned w[3];
    split3(v.x, v.y, w);
#pragma unroll
    for (int p = 0; p < 3; ++p) h[p][x] = w[p];
  }
  return larger(larger(h[0][0], h[0][1]), larger(h[0][2], h[0][3]));
}

// Shared memory of the forward
struct ForwardPlan {
  int tiles;                                                 // of a round
  size_t z0, factor, record, tile, places, desc, total;  // bytes; Z's fragments (tile, part, lane) come first
  __host__ __device__ ForwardPlan(int tiles_, int n_blocks, const Record& rec) {
    tiles = tiles_;
    z0 = (size_t)tiles * 3 * 32 * sizeof(uint2);
    tile = z0 + (size_t)tiles * 4 * sizeof(float2);
    places = tile + (size_t)tiles * sizeof(Tile);
    factor = places + (size_t)n_blocks * sizeof(Factor);
    record = factor + (size_t)FWD_WARPS * n_blocks * ROWS * sizeof(float2);
    desc = record + (size_t)FWD_WARPS * 2 * ROWS * rec.pitch * sizeof(float);
    total = desc + (size_t)n_blocks * FDESC * sizeof(int32_t);
  }
};

// The columns of two edges that a lane's copy c of a tile belongs to: written, or (add) added to
__device__ __forceinline__ void write_columns(const Tile& tile, int c, float* out0, float* out1, bool in0, bool in1, bool add, float2 y0, float2 y1) {
  if (c >= tile.flags >> 8) return;
  const bool real = tile.flags & TILE_REAL_OUT;
  const int col = tile.output + (real ? c : 2 * c);
  if (add) {
    if (in0) y0.x += out0[col];
    if (in1) y1.x += out1[col];
    if (!real && in0) y0.y += out0[col + 1];
    if (!real && in1) y1.y += out1[col + 1];
  }
  if (in0) out0[col] = y0.x;
  if (in1) out1[col] = y1.x;
  if (!real) {
    if (in0) out0[col + 1] = y0.y;
    if (in1) out1[col + 1] = y1.y;
  }
}

// A step of the forward where an operand is too large: by single multiply-adds, from the records and the node's own
// numbers.  (Not inlined: few steps come here.)
__device__ __noinline__ void forward_step_by_products(const FArgs<float>* args, int64_t j, const Tile* tile_s, int n_tiles, bool later_round, const float* row0,
                                                    const float* row1, const float2* f_at, int c, float* out0, float* out1, bool in0, bool in1) {
  const FArgs<float>& a = *args;
  const float *zc = a.zc + j * a.k * 2 * a.wc, *zr = a.zr + j * a.k * a.wr;
  float2 y0 = make_float2(0.f, 0.f), y1 = y0;
  bool continued = later_round && !(tile_s[0].flags & TILE_FIRST);
#pragma unroll 1
  for (int x = 0; x < n_tiles; ++x) {
    const Tile tile = tile_s[x];
    if (c < (tile.flags & 7)) {
      const bool real = tile.flags & TILE_REAL;
      float2 u0 = make_float2(0.f, 0.f), u1 = u0;
#pragma unroll 2
      for (int t = 0; t < a.k; ++t) {
        const float h0 = t ? row0[t - 1] : 1.f, h1 = t ? row1[t - 1] : 1.f;
        const float* z = real ? zr + t * a.wr + tile.column + c : zc + 2 * (t * a.wc + tile.column + c);
        u0.x = fmaf(h0, z[0], u0.x);
        u1.x = fmaf(h1, z[0], u1.x);
        if (real) continue;
        u0.y = fmaf(h0, z[1], u0.y);
        u1.y = fmaf(h1, z[1], u1.y);
      }
      if (real) {
        y0.x += u0.x;
        y1.x += u1.x;
      } else {
        const float2 f0 = f_at[tile.block * ROWS], f1 = f_at[tile.block * ROWS + 8];
        y0.x = fmaf(-f0.y, u0.y, fmaf(f0.x, u0.x, y0.x));
        y0.y = fmaf(f0.y, u0.x, fmaf(f0.x, u0.y, y0.y));
        y1.x = fmaf(-f1.y, u1.y, fmaf(f1.x, u1.x, y1.x));
        y1.y = fmaf(f1.y, u1.x, fmaf(f1.x, u1.y, y1.y));
      }
    }
    if ((tile.flags & TILE_LAST) || x + 1 == n_tiles) {
      write_columns(tile, c, out0, out1, in0, in1, continued, y0, y1);
      continued = false;
      y0 = y1 = make_float2(0.f, 0.f);
    }
  }
}

template <bool SCALED>
__global__ void __launch_bounds__(32 * FWD_WARPS, 10) factored_forward_tc_kernel(const __grid_constant__ FArgs<float> a, int tiles) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int n_rho = SCALED ? a.n_scales : 1;
  const Record rec(a.k, a.n_f, n_rho, a.d_out, false);
  const ForwardPlan plan(tiles, a.n_blocks, rec);
  uint2* const z_s = reinterpret_cast<uint2*>(raw);               // (tile, part, lane): B fragments
  float2* const z0_s = reinterpret_cast<float2*>(raw + plan.z0);  // (tile, copy)
  Tile* const tile_s = reinterpret_cast<Tile*>(raw + plan.tile);
  Factor* const place_s = reinterpret_cast<Factor*>(raw + plan.places);
  int32_t* const desc_s = reinterpret_cast<int32_t*>(raw + plan.desc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  float2* const f_s = reinterpret_cast<float2*>(raw + plan.factor) + warp * a.n_blocks * ROWS;                // (block, edge)
  float* const rec_s = reinterpret_cast<float*>(raw + plan.record) + (size_t)warp * 2 * ROWS * rec.pitch;  // two steps
  for (int x = threadIdx.x; x < a.n_blocks * FDESC; x += 32 * FWD_WARPS) desc_s[x] = a.desc[x];
  *reinterpret_cast<float2*>(rec_s + lane * rec.pitch + rec.one) = make_float2(1.f, 0.f);
  __syncthreads();
  for (int b = threadIdx.x; b < a.n_blocks; b += 32 * FWD_WARPS) place_s[b] = block_place<SCALED>(desc_s + b * FDESC, rec);
  int all_tiles = list_tiles(desc_s, a.n_blocks, 0, plan.tiles, tile_s);
  float zero[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) zero[v] = __int_as_float(a.k >> 31 & (v + 1));
  const int words = word_floats(a, false), units = copy_units(a, n_rho, words, false);
  const CopyUnit unit = copy_unit(a, rec, n_rho, words, false, lane);
  // the rows of 16 edges (lane x < 16 holds the x-th)
  auto stage = [&](float* dst, unsigned e) {
    auto index = [&](int r) { return __shfl_sync(0xffffffffu, e, r); };
    copy_rows(unit, words, dst, rec.pitch, index);
    for (int u0 = 32; u0 < units; u0 += 32) copy_rows(copy_unit(a, rec, n_rho, words, false, u0 + lane), words, dst, rec.pitch, index);  // long phase tables
  };
  for (int base = 0; base < all_tiles; base += plan.tiles) {
    if (base > 0) {
      __syncthreads();
      list_tiles(desc_s, a.n_blocks, base, plan.tiles, tile_s);
    }
    const int n_tiles = min(all_tiles - base, plan.tiles);
    for (int64_t g0 = blockIdx.x; g0 < a.n_groups; g0 += gridDim.x) {
      const int64_t grp = from_both_ends(g0, a.n_groups);
      const int64_t j = a.group_source[grp], first = a.group_ptr[grp], last = a.group_ptr[grp + 1];
      if (first == last) continue;
      int64_t x0 = first + ROWS * warp;  // this warp's steps: every FWD_WARPS-th
      auto edge = [&](int64_t x) { return (unsigned)a.order[min(x + (lane & 15), last - 1)]; };
      unsigned e = x0 < last ? edge(x0) : 0, e_next = x0 + ROWS * FWD_WARPS < last ? edge(x0 + ROWS * FWD_WARPS) : 0;
      __syncthreads();
      unsigned largest = 0;
      {  // lane (column n, outputs 2 c, 2 c + 1 (+ 8 for the second warp)) of every tile
        const int n = lane >> 2, t = 1 + 2 * (lane & 3) + 8 * warp;
        const bool in0 = t < a.k, in1 = t + 1 < a.k;
        const float *zc = a.zc + (j * a.k + t) * 2 * a.wc + n, *zr = a.zr + (j * a.k + t) * a.wr + n / 2;
#pragma unroll 4
        for (int x = 0; x < n_tiles; ++x) {
          const Tile tile = tile_s[x];
          float v0 = 0.f, v1 = 0.f;
          const bool real = tile.flags & TILE_REAL, in = n / 2 < (tile.flags & 7) && !(real && (n & 1));
          const float* z = real ? zr + tile.column : zc + 2 * tile.column;
          if (in && in0) v0 = __ldg(z);
          if (in && in1) v1 = __ldg(z + (real ? a.wr : 2 * a.wc));
          unsigned w[3];
          split3(v0, v1, w);
          largest = larger(largest, w[0]);
#pragma unroll
          for (int p = 0; p < 3; ++p) reinterpret_cast<unsigned*>(z_s)[2 * ((x * 3 + p) * 32 + lane) + warp] = w[p];
        }
      }
      for (int x = threadIdx.x; x < n_tiles * 8; x += 32 * FWD_WARPS) {
        const Tile tile = tile_s[x >> 3];
        const int copy = x >> 1 & 3, im = x & 1;
        float v = 0.f;
        if (copy < (tile.flags & 7)) {
          if (!(tile.flags & TILE_REAL)) v = __ldg(a.zc + (j * a.k * a.wc + tile.column + copy) * 2 + im);
          else if (!im) v = __ldg(a.zr + j * a.k * a.wr + tile.column + copy);
        }
        reinterpret_cast<float*>(z0_s)[x] = v;
      }
      if (x0 < last) stage(rec_s, e);
      const bool large_node = __syncthreads_or(too_large(largest));
      for (int buf = 0; x0 < last; x0 += ROWS * FWD_WARPS, buf ^= 1) {
        const int n_rows = (int)min((int64_t)ROWS, last - x0);
        copy_wait();
        __syncwarp();  // the records are there, and everyone is done with the other buffer and the factors
        const unsigned e0 = __shfl_sync(0xffffffffu, e, g), e1 = __shfl_sync(0xffffffffu, e, g + 8);
        e = e_next;
        if (x0 + ROWS * FWD_WARPS < last) stage(rec_s + (buf ^ 1) * ROWS * rec.pitch, e);
        if (x0 + 2 * ROWS * FWD_WARPS < last) e_next = edge(x0 + 2 * ROWS * FWD_WARPS);
        const float* rows = rec_s + buf * ROWS * rec.pitch;
        {
          const float* row = rows + (lane & 15) * rec.pitch;
          const float rho = row[rec.rho];
#pragma unroll 2
          for (int b = lane >> 4; b < a.n_blocks; b += 2) f_s[b * ROWS + (lane & 15)] = record_factor<SCALED>(row, place_s[b], rho);
        }
        unsigned h[3][4];
        const bool large = __any_sync(0xffffffffu, too_large(load_trunk(rows + g * rec.pitch, rows + (g + 8) * rec.pitch, a.k - 1, c, h)) || large_node);
        __syncwarp();  // the factors are there (a vote orders no memory)
        const bool in0 = g < n_rows, in1 = g + 8 < n_rows;
        float *out0 = a.out + (size_t)e0 * a.d_out, *out1 = a.out + (size_t)e1 * a.d_out;
        if (large) {
          forward_step_by_products(&a, j, tile_s, n_tiles, base > 0, rows + g * rec.pitch, rows + (g + 8) * rec.pitch, f_s + g, c, out0, out1, in0, in1);
          continue;
        }
        float2 y0 = make_float2(0.f, 0.f), y1 = y0;
        bool continued = base > 0 && !(tile_s[0].flags & TILE_FIRST);  // a later round's first columns: the sum goes on
        const uint2* z_at = z_s + lane;
        const float2 *z0_at = z0_s + c, *f_at = f_s + g;
#pragma unroll 2
        for (int x = 0; x < n_tiles; ++x, z_at += 96, z0_at += 4) {
          const Tile tile = tile_s[x];
          const uint2 z[3] = {z_at[0], z_at[32], z_at[64]};
          const float2 z0 = *z0_at, f0 = f_at[tile.block * ROWS], f1 = f_at[tile.block * ROWS + 8];
          f32x2 sum[2];
          product(sum, h, z, zero);
          add2(sum[0], z0.x, z0.y);
          add2(sum[1], z0.x, z0.y);
          const float2 u0 = unpack2(sum[0]), u1 = unpack2(sum[1]);
          y0.x = fmaf(f0.x, u0.x, fmaf(-f0.y, u0.y, y0.x));
          y0.y = fmaf(f0.x, u0.y, fmaf(f0.y, u0.x, y0.y));
          y1.x = fmaf(f1.x, u1.x, fmaf(-f1.y, u1.y, y1.x));
          y1.y = fmaf(f1.x, u1.y, fmaf(f1.y, u1.x, y1.y));
          if ((tile.flags & TILE_LAST) || x + 1 == n_tiles) {
            write_columns(tile, c, out0, out1, in0, in1, continued, y0, y1);
            continued = false;
            y0 = y1 = make_float2(0.f, 0.f);
          }
        }
      }
    }
  }
}

// Shared memory of the backward
struct BackwardPlan {
  int tiles;                                                       // of a round: BWD_TILES a warp
  size_t edge, tile, places, factor, dh, record, desc, total;  // bytes; Z's fragments (pair of tiles, eight outputs, part, lane) come first
  __host__ __device__ BackwardPlan(int n_blocks, const Record& rec, int warps) {
    tiles = warps * BWD_TILES;
    edge = (size_t)tiles * 3 * 32 * sizeof(uint2);
    tile = edge + (size_t)4 * ROWS * 4 * sizeof(unsigned);
    places = tile + (size_t)tiles * sizeof(Tile);
    factor = places + (size_t)n_blocks * sizeof(Factor);
    dh = factor + (size_t)tiles * ROWS * sizeof(float2);
    record = dh + (size_t)2 * warps * ROWS * DH_PITCH * sizeof(float);
    desc = record + (size_t)2 * ROWS * rec.pitch * sizeof(float);
    total = desc + (size_t)n_blocks * FDESC * sizeof(int32_t);
  }
};

// A source of the backward where an operand is too large: dZ of this round's tiles and dh as it is after this round, again by single
// multiply-adds.  W of 16 edges and of a round's columns takes the place of Z's fragments.  (Not inlined.)
constexpr int W_PITCH = ROWS + 1;
static_assert(4 * W_PITCH * sizeof(float2) <= 3 * 32 * sizeof(uint2), "a tile's W fits where its fragments were");
template <bool SCALED>
__device__ __noinline__ void backward_source_by_products(const FArgs<float>* args, int64_t j, int64_t first, int64_t last, int base, int capacity, const int32_t* desc_s,
                                                       Tile* tile_s, float2* w_s, float* h_s, unsigned* edge_s) {
  const FArgs<float>& a = *args;
  const int threads = blockDim.x, n_trunk = a.k - 1;
  for (int b0 = 0; b0 <= base; b0 += capacity) {
    __syncthreads();
    const int n_tiles = min(list_tiles(desc_s, a.n_blocks, b0, capacity, tile_s) - b0, capacity), columns = 4 * n_tiles;
    for (int64_t x0 = first; x0 < last; x0 += ROWS) {
      const int n = (int)min((int64_t)ROWS, last - x0);
      __syncthreads();
      if (threadIdx.x < ROWS) edge_s[threadIdx.x] = (unsigned)a.order[min(x0 + threadIdx.x, last - 1)];
      __syncthreads();
      for (int i = threadIdx.x; i < ROWS * n_trunk; i += threads) h_s[i / n_trunk * DH_PITCH + i % n_trunk] = a.h[(size_t)edge_s[i / n_trunk] * n_trunk + i % n_trunk];
      for (int i = threadIdx.x; i < columns * ROWS; i += threads) {
        const Tile tile = tile_s[i / (4 * ROWS)];
        const int c = i / ROWS & 3, r = i % ROWS;
        float2 w = make_float2(0.f, 0.f);
        if (c < (tile.flags & 7) && r < n) {
          const int64_t e = edge_s[r];
          const float weight = a.weights ? a.weights[e] : 1.f, *g = a.g + (a.target ? a.target[e] : e) * a.d_out + tile.output;
          if (tile.flags & TILE_REAL) {
            w.x = weight * g[c];
          } else {
            float fr, fi;
            table_factor<SCALED>(a, e, desc_s + tile.block * FDESC, fr, fi);
            const bool real = tile.flags & TILE_REAL_OUT;
            const float gr = weight * g[real ? c : 2 * c], gi = real ? 0.f : weight * g[2 * c + 1];
            w = make_float2(gr * fr + gi * fi, gi * fr - gr * fi);
          }
        }
        w_s[i / ROWS * W_PITCH + r] = w;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < ROWS * n_trunk; i += threads) {  // dh
        const int r = i % ROWS, t = 1 + i / ROWS;
        if (r >= n) continue;
        float* to = a.dh + (size_t)edge_s[r] * n_trunk + t - 1;
        float s = b0 ? *to : 0.f;
        for (int x = 0; x < n_tiles; ++x) {
          const Tile tile = tile_s[x];
          const bool real = tile.flags & TILE_REAL;
          const float* z = real ? a.zr + (j * a.k + t) * a.wr + tile.column : a.zc + ((j * a.k + t) * a.wc + tile.column) * 2;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c >= (tile.flags & 7)) continue;
            const float2 w = w_s[(4 * x + c) * W_PITCH + r];
            s = fmaf(w.x, z[real ? c : 2 * c], s);
            if (!real) s = fmaf(w.y, z[2 * c + 1], s);
          }
        }
        *to = s;
      }
      for (int i = threadIdx.x; i < a.k * columns; i += threads) {  // dZ; a thread keeps its entries
        const int t = i / columns, x = i % columns, c = x & 3;
        const Tile tile = tile_s[x / 4];
        if (c >= (tile.flags & 7)) continue;
        const bool real = tile.flags & TILE_REAL;
        float* to = real ? a.dzr + (j * a.k + t) * a.wr + tile.column + c : a.dzc + ((j * a.k + t) * a.wc + tile.column + c) * 2;
        float2 s = x0 == first ? make_float2(0.f, 0.f) : make_float2(to[0], real ? 0.f : to[1]);
#pragma unroll 4
        for (int r = 0; r < n; ++r) {
          const float h = t ? h_s[r * DH_PITCH + t - 1] : 1.f;
          const float2 w = w_s[x * W_PITCH + r];
          s.x = fmaf(h, w.x, s.x);
          s.y = fmaf(h, w.y, s.y);
        }
        to[0] = s.x;
        if (!real) to[1] = s.y;
      }
    }
  }
}

template <bool SCALED>
__global__ void __launch_bounds__(32 * MAX_WARPS, 2) factored_backward_tc_kernel(const __grid_constant__ FArgs<float> a) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int threads = blockDim.x, warps = threads >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int n_rho = SCALED ? a.n_scales : 1;
  const Record rec(a.k, a.n_f, n_rho, a.d_out, true);
  const BackwardPlan plan(a.n_blocks, rec, warps);
  uint2* const z_s = reinterpret_cast<uint2*>(raw);                       // (pair of tiles, eight outputs, part, lane): B fragments
  unsigned* const edge_s = reinterpret_cast<unsigned*>(raw + plan.edge);  // four steps of 16: edges
  unsigned* const target_s = edge_s + 4 * ROWS;                           // the rows of g that reach them
  float* const weight_s = reinterpret_cast<float*>(target_s + 4 * ROWS);
  Tile* const tile_s = reinterpret_cast<Tile*>(raw + plan.tile);
  Factor* const place_s = reinterpret_cast<Factor*>(raw + plan.places);
  int32_t* const desc_s = reinterpret_cast<int32_t*>(raw + plan.desc);
  float2* const f_s = reinterpret_cast<float2*>(raw + plan.factor) + warp * BWD_TILES * ROWS;  // (tile, edge): weight x factor
  float* const dh_s = reinterpret_cast<float*>(raw + plan.dh);                                 // two buffers of (warp, edge, output)
  float* const rec_s = reinterpret_cast<float*>(raw + plan.record);                            // two steps
  for (int x = threadIdx.x; x < a.n_blocks * FDESC; x += threads) desc_s[x] = a.desc[x];
  if (threadIdx.x < 2 * ROWS) *reinterpret_cast<float2*>(rec_s + threadIdx.x * rec.pitch + rec.one) = make_float2(1.f, 0.f);
  __syncthreads();
  for (int b = threadIdx.x; b < a.n_blocks; b += threads) place_s[b] = block_place<SCALED>(desc_s + b * FDESC, rec);
  const int all_tiles = list_tiles(desc_s, a.n_blocks, 0, plan.tiles, tile_s);
  int complex_copies = 0, real_copies = 0;
  for (int b = 0; b < a.n_blocks; ++b) (desc_s[b * FDESC] ? complex_copies : real_copies) += desc_s[b * FDESC + 2];
  const bool covered = complex_copies == a.wc && real_copies == a.wr;
  float zero[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) zero[v] = __int_as_float(a.k >> 31 & (v + 1));
  const int words = word_floats(a, true), units = copy_units(a, n_rho, words, true);
  const CopyUnit unit = copy_unit(a, rec, n_rho, words, true, threadIdx.x);
  auto stage = [&](int step) {  // the records of a step: a thread keeps its part of the rows
    float* dst = rec_s + (step & 1) * ROWS * rec.pitch;
    auto copy = [&](const CopyUnit& u) {
      const unsigned* row = (u.kind == 2 ? target_s : edge_s) + (step & 3) * ROWS;
      copy_rows(u, words, dst, rec.pitch, [&](int r) { return row[r]; });
    };
    if (unit.kind) copy(unit);
    for (int u = threadIdx.x + threads; u < units; u += threads) copy(copy_unit(a, rec, n_rho, words, true, u));
  };
  // (one round unless the blocks' copies are uneven; the rounds add up dh)
  for (int base = 0; base < max(all_tiles, 1); base += plan.tiles) {
    if (base > 0) {
      __syncthreads();
      list_tiles(desc_s, a.n_blocks, base, plan.tiles, tile_s);
    }
    const int n_tiles = min(all_tiles - base, plan.tiles), t0 = warp * BWD_TILES, mine = min(n_tiles - t0, BWD_TILES);  // mine: this warp's tiles
    for (int64_t g0 = blockIdx.x; g0 < a.n_groups; g0 += gridDim.x) {
      const int64_t grp = from_both_ends(g0, a.n_groups);
      const int64_t j = a.group_source[grp], first = a.group_ptr[grp], last = a.group_ptr[grp + 1];
      const int steps = (int)((last - first + ROWS - 1) / ROWS);
      // the edges of a step, two steps ahead of its copies; the first warp's first half looks after them
      auto edge = [&](int step) { return (unsigned)a.order[min(first + (int64_t)step * ROWS + lane, last - 1)]; };
      auto put_edges = [&](int step, unsigned e) {
        edge_s[(step & 3) * ROWS + lane] = e;
        target_s[(step & 3) * ROWS + lane] = a.target ? (unsigned)a.target[e] : e;
        weight_s[(step & 3) * ROWS + lane] = a.weights ? a.weights[e] : 1.f;
      };
      unsigned e_ahead = 0;
      __syncthreads();
      if (threadIdx.x < ROWS) {
        if (steps > 0) put_edges(0, edge(0));
        if (steps > 1) put_edges(1, edge(1));
        if (steps > 2) e_ahead = edge(2);
      }
      unsigned largest = 0;
      {  // lane (output 8 half + g, columns of copy c of tile 2 pair + r)
        const int n_items = (n_tiles + 1) / 2 * 4;  // (pair, half, r)
#pragma unroll 4
        for (int x = warp; x < n_items; x += warps) {
          const int r = x & 1, half = x >> 1 & 1, pair = x >> 2, at = 2 * pair + r, t = 1 + 8 * half + g;
          const Tile tile = at < n_tiles ? tile_s[at] : Tile{0, 0, 0, 0};
          const bool real = tile.flags & TILE_REAL, in = t < a.k && c < (tile.flags & 7);
          const float* z = real ? a.zr + (j * a.k + t) * a.wr + tile.column + c : a.zc + ((j * a.k + t) * a.wc + tile.column + c) * 2;
          const float re = in ? __ldg(z) : 0.f, im = in && !real ? __ldg(z + 1) : 0.f;
          unsigned w[3];
          split3(re, im, w);
          largest = larger(largest, w[0]);
#pragma unroll
          for (int p = 0; p < 3; ++p) reinterpret_cast<unsigned*>(z_s)[2 * (((pair * 2 + half) * 3 + p) * 32 + lane) + r] = w[p];
        }
      }
      if (!covered && base == 0) {  // columns that no block has
        for (int64_t x = threadIdx.x; x < (int64_t)a.k * 2 * a.wc; x += threads) a.dzc[j * a.k * 2 * a.wc + x] = 0.f;
        for (int64_t x = threadIdx.x; x < (int64_t)a.k * a.wr; x += threads) a.dzr[j * a.k * a.wr + x] = 0.f;
      }
      __syncthreads();
      f32x2 acc[BWD_TILES][2];  // rows t = 1 + g, 9 + g; columns (re, im) of copy c
      f32x2 sum[BWD_TILES];     // of W over this lane's edges
#pragma unroll
      for (int x = 0; x < BWD_TILES; ++x) {
        acc[x][0] = acc[x][1] = 0;
        sum[x] = 0;
      }
      if (steps > 0) stage(0);
      // the warps' parts of a step's dh, added in one order
      auto write_dh = [&](int step) {
        const int n_rows = (int)min((int64_t)ROWS, last - first - (int64_t)step * ROWS);
        for (int x = threadIdx.x; x < n_rows * TRUNK; x += threads) {
          const int row = x / TRUNK, t = x % TRUNK;
          if (t >= a.k - 1) continue;
          float* to = a.dh + (size_t)edge_s[(step & 3) * ROWS + row] * (a.k - 1) + t;
          float s = base ? *to : 0.f;
          for (int v = 0; v < warps; ++v) s += dh_s[(((step & 1) * warps + v) * ROWS + row) * DH_PITCH + t];
          *to = s;
        }
      };
      for (int step = 0; step < steps; ++step) {
        const int n_rows = (int)min((int64_t)ROWS, last - first - (int64_t)step * ROWS);
        copy_wait();
        __syncthreads();  // the step's records and the next one's edges are there; everyone is done with the step before
        if (step + 1 < steps) stage(step + 1);
        if (threadIdx.x < ROWS && step + 2 < steps) {
          put_edges(step + 2, e_ahead);
          if (step + 3 < steps) e_ahead = edge(step + 3);
        }
        if (step > 0) write_dh(step - 1);
        const float* rows = rec_s + (step & 1) * ROWS * rec.pitch;
        const bool in0 = g < n_rows, in1 = g + 8 < n_rows;
        {
          const float *row = rows + (lane & 15) * rec.pitch, rho = row[rec.rho], weight = weight_s[(step & 3) * ROWS + (lane & 15)];
#pragma unroll 2
          for (int x = lane >> 4; x < mine; x += 2) {
            const float2 f = record_factor<SCALED>(row, place_s[tile_s[t0 + x].block], rho);
            f_s[x * ROWS + (lane & 15)] = make_float2(weight * f.x, weight * f.y);
          }
        }
        unsigned ht[3][4];  // the trunk's outputs as 16 outputs x 16 edges
        {
          unsigned h[3][4];
          const unsigned most = load_trunk(rows + g * rec.pitch, rows + (g + 8) * rec.pitch, a.k - 1, c, h);
          largest = larger(largest, most);
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            ht[p][0] = transposed(in0 ? h[p][0] : 0u);
            ht[p][1] = transposed(in0 ? h[p][2] : 0u);
            ht[p][2] = transposed(in1 ? h[p][1] : 0u);
            ht[p][3] = transposed(in1 ? h[p][3] : 0u);
          }
        }
        __syncwarp();
        f32x2 dh[2][2] = {{0, 0}, {0, 0}};  // outputs 1 + 8 half + 2 c, + 1 of the edges g, g + 8
        const float* grad0 = rows + g * rec.pitch + rec.grad;
        const float* grad1 = grad0 + 8 * rec.pitch;
#pragma unroll
        for (int q = 0; q < BWD_TILES / 2; ++q) {
          if (2 * q >= mine) break;
          unsigned w[3][4];  // W of two tiles: 16 edges x 16 columns
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int x = 2 * q + r;
            float2 w0 = make_float2(0.f, 0.f), w1 = w0;
            if (x < mine) {
              const Tile tile = tile_s[t0 + x];
              const bool has = c < (tile.flags & 7), im = !(tile.flags & TILE_REAL_OUT);
              const int at = has ? tile.output + (im ? 2 * c : c) : 0;
              const float2 f0 = f_s[x * ROWS + g], f1 = f_s[x * ROWS + g + 8];
              const float x0 = grad0[at], y0 = im ? grad0[at + 1] : 0.f, x1 = grad1[at], y1 = im ? grad1[at + 1] : 0.f;
              const bool complex_block = !(tile.flags & TILE_REAL);
              if (has && in0) w0 = make_float2(fmaf(x0, f0.x, y0 * f0.y), complex_block ? fmaf(y0, f0.x, -x0 * f0.y) : 0.f);  // W = G conj(F)
              if (has && in1) w1 = make_float2(fmaf(x1, f1.x, y1 * f1.y), complex_block ? fmaf(y1, f1.x, -x1 * f1.y) : 0.f);
            }
            add2(sum[x], w0.x, w0.y);
            add2(sum[x], w1.x, w1.y);
            unsigned s0[3], s1[3];
            split3(w0.x, w0.y, s0);
            split3(w1.x, w1.y, s1);
            largest = larger(largest, larger(s0[0], s1[0]));
            uint2 wt[3];  // 16 edges x 8 columns as a B operand
#pragma unroll
            for (int p = 0; p < 3; ++p) {
              w[p][2 * r] = s0[p];
              w[p][2 * r + 1] = s1[p];
              wt[p] = make_uint2(transposed(s0[p]), transposed(s1[p]));
            }
            f32x2 u[2];
            product(u, ht, wt, zero);
            add2(acc[x][0], u[0]);
            add2(acc[x][1], u[1]);
          }
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const uint2* z_at = z_s + ((t0 / 2 + q) * 2 + half) * 96 + lane;
            const uint2 z[3] = {z_at[0], z_at[32], z_at[64]};
            f32x2 u[2];
            product(u, w, z, zero);
            add2(dh[half][0], u[0]);
            add2(dh[half][1], u[1]);
          }
        }
        if (warp == warps - 1 && base == 0 && a.dweights) {  // dweights_e = <g_i, row_e>, two lanes per edge
          const float* row = rows + (lane >> 1) * rec.pitch;
          float part[4] = {0.f, 0.f, 0.f, 0.f};  // every eighth column: the sums, and their order, of the CUDA-core kernel's eight lanes
#pragma unroll 1
          for (int x = lane & 1; x < a.d_out; x += 8) {
#pragma unroll
            for (int v = 0; v < 4; ++v)
              if (x + 2 * v < a.d_out) part[v] = fmaf(row[rec.grad + x + 2 * v], row[rec.row + x + 2 * v], part[v]);
          }
          float s = (part[0] + part[2]) + (part[1] + part[3]);
          s += __shfl_xor_sync(0xffffffffu, s, 1);
          if ((lane & 1) == 0 && lane / 2 < n_rows) a.dweights[edge_s[(step & 3) * ROWS + lane / 2]] = s;
        }
        float* mine_s = dh_s + ((step & 1) * warps + warp) * ROWS * DH_PITCH;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          *reinterpret_cast<float2*>(mine_s + g * DH_PITCH + 8 * half + 2 * c) = unpack2(dh[half][0]);
          *reinterpret_cast<float2*>(mine_s + (g + 8) * DH_PITCH + 8 * half + 2 * c) = unpack2(dh[half][1]);
        }
      }
      const bool again = __syncthreads_or(too_large(largest));
      if (steps > 0) write_dh(steps - 1);
      // ---- dZ: rows t from the accumulators, row 0 from the lanes' sums
#pragma unroll
      for (int x = 0; x < BWD_TILES; ++x) {
        if (x >= mine) break;
        const Tile tile = tile_s[t0 + x];
        float2 s = unpack2(sum[x]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
          s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if (c >= (tile.flags & 7)) continue;
#pragma unroll
        for (int part = 0; part < 3; ++part) {
          const int t = part == 0 ? 0 : 1 + g + 8 * (part - 1);
          if (t >= a.k || (part == 0 && g != 0)) continue;
          const float2 v = part == 0 ? s : unpack2(acc[x][part - 1]);
          if (tile.flags & TILE_REAL) {
            a.dzr[(j * a.k + t) * a.wr + tile.column + c] = v.x;
          } else {
            float* z = a.dzc + ((j * a.k + t) * a.wc + tile.column + c) * 2;
            z[0] = v.x;
            z[1] = v.y;
          }
        }
      }
      if (again) backward_source_by_products<SCALED>(&a, j, first, last, base, plan.tiles, desc_s, tile_s, reinterpret_cast<float2*>(z_s), dh_s, edge_s);
    }
  }
}

constexpr size_t SMEM_MOST = 200 * 1024;

int n_rho(const FArgs<float>& a) { return a.n_scales ? a.n_scales : 1; }
ForwardPlan forward_plan(const FArgs<float>& a) {
  return ForwardPlan(std::max(likely_tiles(a.wc, a.wr, a.n_blocks), 1), a.n_blocks, Record(a.k, a.n_f, n_rho(a), a.d_out, false));
}
int backward_warps(const FArgs<float>& a) { return std::min((std::max(likely_tiles(a.wc, a.wr, a.n_blocks), 1) + BWD_TILES - 1) / BWD_TILES, MAX_WARPS); }
BackwardPlan backward_plan(const FArgs<float>& a) {
  return BackwardPlan(a.n_blocks, Record(a.k, a.n_f, n_rho(a), a.d_out, true), backward_warps(a));
}
// Where the tensor-core kernels are the faster ones: 949 timings, lattices from 24 x 48 to 128 x 256, radius 1 to 4 rows (7 to 144 edges per
// source), k 2 to 17, 5, 13 or 25 blocks of 2 to 8 copies.  A source's columns are split once for all of its edges (few edges: no),
// tiles of four copies may be part empty, and a step takes as long whatever k is, where the CUDA-core kernels' products grow with
// it, four trunk outputs (a quad) at a time.  us, CUDA cores / tensor cores:
//   forward   from 24 edges on (92 edges, 13 blocks of 4 copies, k 17: 1 034 / 734, k 11 873 / 691; 38, 13 of 8: 337 / 259), with part-empty tiles from 4.5 edges a tile on (69 edges, 13 blocks of 3: 55 / 48; 133, 13 of 2: 262 / 246;
//             but 43 edges, 13 of 3, 1.06 to 1.09 of the time, 92, 13 of 5, 1.07 to 1.16).
//   backward  k 17: 92 edges, 13 blocks of 4, 2 475 / 1 838; 80, 13 of 3, 495 / 439; 80, 13 of 8, 867 / 838; 133, 13 of 8, 1 319 / 1 196; but 80, 13 of 2,
//             400 / 432; 38, 13 of 8, 532 / 570.  k 11: 80, 13 of 4, 518 / 437, but 80, 13 of 8, 771 / 825.  k 9: 80, 13 of 8, 602 / 803; 43, 5 of 4, 818 / 594.
//             Small launches last as long as their longest source's steps, which are longer here.  The lines are fitted to that: at worst
//             10 % (k 10 on 26 tiles, 45 x 90 with k 2), at k 16 and 17 5 %.  Where the other kernel would pass a source's edges twice (25 blocks of 8:
//             0.71 to 0.76 of its time) always.
// (Edge indices are 32-bit here.)
struct Split {
  int tiles;
  double fill, edges;  // share of the tiles' copies that exist, edges per source
  explicit Split(const FArgs<float>& a)
      : tiles(std::max(likely_tiles(a.wc, a.wr, a.n_blocks), 1)), fill((double)(a.wc + a.wr) / (4 * tiles)), edges((double)a.n_edges / a.n_groups) {}
};
bool serves(const FArgs<float>& a) {
  if (a.k < 2 || a.k > TRUNK + 1 || a.n_blocks < 1 || a.n_edges >= (1ll << 31)) return false;
  const Split s(a);
  return s.fill * s.fill * s.edges >= 24;
}

// Rows: with few trunk outputs the roundings of a column's two chains and of Z_0 weigh more than those of the CUDA-core kernel's single
// chain.  Error against float64, here over there, by k: 2 1.10 to 1.16, 3 1.12 to 1.19, 5 1.09 to 1.13, 7 1.05 to 1.07, 8 1.03, 9 1.01, 10 0.98,
// 11 0.96, 13 0.92 to 0.94, 17 0.85 to 0.88 (three field types, powers and scales).  The backward's are 0.2 to 0.8 for any k.
constexpr int FWD_LEAST_K = 10;

}  // namespace

bool tensor_cores_forward(const FArgs<float>& a) {
  if (a.k < FWD_LEAST_K || !serves(a)) return false;
  const Split s(a);
  return (s.fill > 0.999 || s.edges >= 4.5 * s.tiles) && forward_plan(a).total <= SMEM_MOST;
}
bool tensor_cores_backward(const FArgs<float>& a) {
  if (!serves(a)) return false;
  const Split s(a);
  const int quads = (a.k + 2) / 4, patches = (a.k + 4) / 5 * ((2 * a.wc + a.wr + 3) / 4);
  const bool pays = patches > 256 || (quads == 4 && std::pow(s.fill, 3) * s.edges >= 2 * s.tiles) ||
                    ((quads > 2 || s.tiles <= 5) && quads * std::pow(s.fill, 1.5) * std::pow((double)a.n_edges, 0.25) >= 3.7 * s.tiles);
  return pays && backward_plan(a).total <= SMEM_MOST;
}

int forward_tc(const FArgs<float>& a, cudaStream_t stream) {
  const ForwardPlan plan = forward_plan(a);
  auto kernel = a.n_scales ? factored_forward_tc_kernel<true> : factored_forward_tc_kernel<false>;
  const int st = allow_smem(kernel, plan.total, "gm_factored_forward");
  if (st != GM_OK) return st;
  const int64_t cap = (int64_t)sm_count() * FWD_CTAS;
  kernel<<<(unsigned)std::min(a.n_groups, cap), 32 * FWD_WARPS, plan.total, stream>>>(a, plan.tiles);
  return launch_status("gm_factored_forward");
}

int backward_tc(const FArgs<float>& a, cudaStream_t stream) {
  const BackwardPlan plan = backward_plan(a);
  auto kernel = a.n_scales ? factored_backward_tc_kernel<true> : factored_backward_tc_kernel<false>;
  const int st = allow_smem(kernel, plan.total, "gm_factored_backward");
  if (st != GM_OK) return st;
  const int64_t cap = (int64_t)sm_count() * BWD_CTAS;
  kernel<<<(unsigned)std::min(a.n_groups, cap), 32 * backward_warps(a), plan.total, stream>>>(a);
  return launch_status("gm_factored_backward");
}

}  // namespace factored
}  // namespace gmb
