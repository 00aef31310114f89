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
// 2.5 pi / 24, 6.4e-6 / 1.1e-6 / 3.2e-6 and 2.1e-6 / 4.3e-7 / 1.1e-6.  It cost a fifth of the time of apply as
// it was first.
//
// A CTA is four producer warps and four consumer warps (named barriers, registers 56 / 200 a thread).  The producers copy the
// positions and, for apply, fetch, split and place the table; the consumers multiply.  With every warp doing both (8 or 12 warps an
// SM), a CTA's copies, table entries and products followed each other and the tensor pipe stood at 34 %: 256 x 512, radius
// 4 pi / 256, batch 4, 64 x (m <= 2): apply 3 230 us, 2 475 with stages handed over by one barrier and cut by positions instead of
// offsets, 2 010 with producers; table_grad 2 440, 2 000 with producers.  128 x 256, batch 2: 502 -> 269 and 439 -> 345; 45 x 88, batch 3, 32 x (m <= 2): 104
// -> 46 and 75 -> 60.  What bounds them now: the producers alone take 1 490 / 1 420 us, the consumers alone 1 590 / 1 400 (their
// products 880 / 300, their shared-memory reads 740 / 400), and they share the load / store unit.
//
// In shared memory the positions 8 t + e of a plane e follow each other, so that a lane reads four channel pairs of one position
// with one 16-byte load, the eight lanes of a phase on different banks.  The (re, im) words are B fragments of apply as they are;
// table_grad contracts over positions and pairs the words of t and t + 1 with two byte permutations.
#include <algorithm>

#include "lattice_conv.cuh"
#include "mma.cuh"

namespace gmb {
namespace lconv {
namespace {

// 16 bytes global -> shared, asynchronously; bytes = 0 writes zeros
__device__ __forceinline__ void copy16(uint4* dst, const void* src, int bytes) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(addr), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Where the positions e, 8 + e, 16 + e, ... start, in 16-byte words
template <int SP, bool SKEW> __device__ __forceinline__ int plane(int e) { return e * SP + (SKEW ? (e & 1) + 2 * (e & 2) : 0); }

// Staged copies of `count` positions from longitude `lon` of a row (cyclic) on, WORDS 16-byte words each: position q to
// [q % 8][q / 8], SP words between the eight, PITCH between positions.  Columns beyond the field's are zeros.
template <int THREADS, int WORDS, int SP, int PITCH, bool SKEW>
__device__ __forceinline__ void stage_positions(uint4* dst, const unsigned char* row, int lon, int count, int nlon, int row_bytes, int col_byte) {
  constexpr int PASS = THREADS / WORDS;
  const int first = threadIdx.x % THREADS / WORDS, k = threadIdx.x % WORDS, byte = col_byte + 16 * k;
  const bool in = byte < row_bytes;
  const unsigned char* src = row + (in ? byte : 0);
  int at = lon + first;
  while (at >= nlon) at -= nlon;
  int step = PASS;
  while (step >= nlon) step -= nlon;
  static_assert(PASS % 8 == 0, "a thread's positions lie in one plane");
  dst += plane<SP, SKEW>(first & 7) + k;
  for (int q = first; q < count; q += PASS) {
    copy16(dst + (q >> 3) * PITCH, src + (size_t)at * row_bytes, in ? 16 : 0);
    at += step;
    if (at >= nlon) at -= nlon;
  }
}

// ---- producers and consumers: a CTA is two groups of 128 threads.  The producers fill stages in shared memory, the consumers
// multiply; a stage's named barriers say that it is there (the producers arrive, the consumers wait) and that its buffer is free
// (the other way round).  Both walk the same list of stages, so every arrival is met.
constexpr int GROUP = 128;
constexpr int BAR_CONSUMERS = 1, BAR_STAGES = 2;  // ids: the consumers among themselves; then (full, empty) of every buffer
__device__ __forceinline__ void barrier_sync(int id) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(2 * GROUP) : "memory"); }
__device__ __forceinline__ void barrier_arrive(int id) { asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(2 * GROUP) : "memory"); }
__device__ __forceinline__ int full_barrier(int buf) { return BAR_STAGES + 2 * buf; }
__device__ __forceinline__ int empty_barrier(int buf) { return BAR_STAGES + 2 * buf + 1; }
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync %0, %1;\n" ::"n"(BAR_CONSUMERS), "n"(GROUP) : "memory"); }
__device__ __forceinline__ bool consumer_or(bool x) {
  unsigned any;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}\n"
               : "=r"(any) : "r"((unsigned)x), "n"(BAR_CONSUMERS), "n"(GROUP) : "memory");
  return any != 0;
}
// The launch's 128 registers a thread (256 threads, two CTAs an SM) split over the groups: 56 + 200
__device__ __forceinline__ void producer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 56;\n"); }
__device__ __forceinline__ void consumer_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 200;\n"); }
// The producers' way through `BUFFERS` stages in turn, up to FLIGHT of them being copied at a time
template <int BUFFERS, int FLIGHT>
struct Ring {
  int n = 0, buf = 0;
  template <int PENDING>
  __device__ __forceinline__ void finish() const {  // the stage issued before the PENDING last is complete
    if (n <= PENDING) return;
    wait_copies<PENDING>();
    barrier_arrive(full_barrier(buf > PENDING ? buf - PENDING - 1 : buf + BUFFERS - PENDING - 1));
  }
  __device__ __forceinline__ void begin() const {  // hand over the oldest stage, wait for a free buffer
    finish<FLIGHT - 1>();
    if (n >= BUFFERS) barrier_sync(empty_barrier(buf));
  }
  __device__ __forceinline__ void advance() {
    ++n;
    buf = buf == BUFFERS - 1 ? 0 : buf + 1;
  }
  __device__ __forceinline__ void drain() const {  // hand over the rest, meet the consumers' last arrivals
    if constexpr (FLIGHT > 1) finish<1>();
    finish<0>();
    const int open = min(n, BUFFERS);
    for (int x = 0; x < open; ++x) barrier_sync(empty_barrier((n - open + x) % BUFFERS));
  }
  static_assert(FLIGHT <= 2 && FLIGHT < BUFFERS + 1, "");
};

struct PairItem {
  int kind, fcol;  // -1: no item on these columns
};
template <int COLS, int THREADS>
__device__ __forceinline__ void find_items(const ConvArgs& a, int col0, PairItem* pairs_s) {
  if (threadIdx.x < COLS / 2) pairs_s[threadIdx.x] = PairItem{-1, 0};
  __syncthreads();
  for (int x = threadIdx.x; x < a.n_items; x += THREADS) {
    const int col = a.items[3 * x + 1] - col0;
    if (col >= 0 && col < COLS) pairs_s[col >> 1] = PairItem{a.items[3 * x], a.items[3 * x + 2]};
  }
  __syncthreads();
}

// ----------------------------------------------------------------------------------------------------------- table_grad
constexpr int TG_COLS = 32;                       // columns of the field at a time: a consumer warp has four channel pairs
constexpr int TG_PAIRS = TG_COLS / 2;
constexpr int TG_GROUP = 5;                       // blocks of 32 columns that a CTA works on one after the other, at most
constexpr int TG_BUFFERS = 4, TG_FLIGHT = 2;
constexpr int TG_PITCH = 5;                       // 16-byte words per staged position (4 and one of padding)
constexpr int TG_TILES = 16;                      // tiles t per stage: a k-step
constexpr int TG_SPG = TG_TILES * TG_PITCH + 1;   // odd: the lanes' eight s fall on different banks beside their four t
constexpr int TG_SPX = (TG_TILES + 4) * TG_PITCH + 1;
constexpr int TG_STAGE = 8 * (TG_SPG + TG_SPX);   // 16-byte words
constexpr int TG_MERGE = 3;                       // blocks of 8 offsets one CTA takes: 24 + 7 positions are four groups of 8
constexpr int TG_PS = 34;                         // floats between the s of a P block: 32 r, and 2 so that rows start on other banks
constexpr int TG_BLOCK = 8 * TG_PS + 8;           // floats of a P block: 8 s x 32 r

// One CTA: up to three consecutive blocks (of 8 offsets) of one window, 32 columns at a time.
__global__ void __launch_bounds__(2 * GROUP, 2) conv_table_grad_tc_kernel(const __grid_constant__ ConvArgs a, int n_blocks, int col_blocks, int group) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PairItem pairs_s[TG_GROUP * TG_PAIRS];
  const int block = blockIdx.x, w = a.order[2 * block], d0 = a.order[2 * block + 1], b8 = d0 / 8;
  auto is = [&](int x, int d) { return a.order[2 * x] == w && a.order[2 * x + 1] == d; };
  if (b8 % TG_MERGE != 0 && block > 0 && is(block - 1, d0 - 8)) return;  // an earlier block's CTA takes this one too
  int merged = 1;
  while ((b8 + merged) % TG_MERGE != 0 && block + merged < n_blocks && is(block + merged, d0 + 8 * merged)) ++merged;
  const int span = 2 * a.halo + 1, row = w / span, j = row + w % span - a.halo;
  const int valid = min(8 * merged, a.win_cnt[w] - d0), groups = (7 + valid + 7) / 8;
  const int cb0 = blockIdx.y * group, n_cb = min(group, col_blocks - cb0), row_bytes = 2 * a.width;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, cg = warp & 3;
  const int T = a.nlon / 8, chunks = (T + TG_TILES - 1) / TG_TILES;
  uint4* const stage_s = reinterpret_cast<uint4*>(smem);
  find_items<TG_GROUP * TG_COLS, 2 * GROUP>(a, cb0 * TG_COLS, pairs_s);

  if (warp >= GROUP / 32) {
    // ---- producers: the stages are the samples' chunks of tiles, columns by columns
    producer_registers();
    int shift = (a.win_lo[w] + d0) % a.nlon;
    if (shift < 0) shift += a.nlon;
    const size_t sample = (size_t)a.rows * a.nlon * row_bytes;
    const unsigned char* grow = static_cast<const unsigned char*>(a.g) + (size_t)row * a.nlon * row_bytes;
    const unsigned char* xrow = static_cast<const unsigned char*>(a.x) + (size_t)j * a.nlon * row_bytes;
    Ring<TG_BUFFERS, TG_FLIGHT> ring;
    for (int cb = 0; cb < n_cb; ++cb)
      for (int b = 0; b < a.batch; ++b)
        for (int t0 = 0; t0 < T; t0 += TG_TILES) {
          const int tl = min(TG_TILES, T - t0), col_byte = 2 * (cb0 + cb) * TG_COLS;
          ring.begin();
          uint4* dst = stage_s + ring.buf * TG_STAGE;
          stage_positions<GROUP, TG_COLS / 8, TG_SPG, TG_PITCH, false>(dst, grow + b * sample, 8 * t0, 8 * tl, a.nlon, row_bytes, col_byte);
          stage_positions<GROUP, TG_COLS / 8, TG_SPX, TG_PITCH, false>(dst + 8 * TG_SPG, xrow + b * sample, shift + 8 * t0, 8 * (tl + groups - 1),
                                                                       a.nlon, row_bytes, col_byte);
          commit();
          ring.advance();
        }
    ring.drain();
    return;
  }
  // ---- consumers
  consumer_registers();
  float* const p_s = reinterpret_cast<float*>(stage_s + TG_BUFFERS * TG_STAGE) + warp * 4 * TG_BLOCK;
  float zero[4];  // zeros that the compiler does not see through: it would clear four registers for every product
#pragma unroll
  for (int v = 0; v < 4; ++v) zero[v] = __int_as_float(a.nlon >> 31 & (v + 1));
  int buf = 0;
  auto columns = [&](auto count, int cb) {
    constexpr int GROUPS = decltype(count)::value;
    f32x2 acc[4][GROUPS][2][2];  // channel pair, group, component of x: rows (s = g: component 0 of g, g + 8: 1), columns r = 2 c, 2 c + 1
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int n = 0; n < GROUPS; ++n)
#pragma unroll
        for (int q = 0; q < 2; ++q) acc[p][n][q][0] = acc[p][n][q][1] = 0;
    for (int s = 0; s < chunks * a.batch; ++s) {
      const int tl = min(TG_TILES, T - s % chunks * TG_TILES);
      barrier_sync(full_barrier(buf));
      const uint4* gs = stage_s + buf * TG_STAGE + g * TG_SPG + cg;
      const uint4* xs = stage_s + buf * TG_STAGE + 8 * TG_SPG + g * TG_SPX + cg;
      // the words of tile t = k0 + 2 c (+ 1, + 8, + 9); both operands are zero beyond the last tile
      auto step = [&](int k0, auto is_ragged) {
        const int t = k0 + 2 * c;
        auto words = [&](const uint4* base, int n, unsigned (&lo)[4], unsigned (&hi)[4], int from) {  // tiles t + from, t + from + 1: component 0, 1
          uint4 v0 = base[(t + from + n) * TG_PITCH], v1 = base[(t + from + 1 + n) * TG_PITCH];
          if (decltype(is_ragged)::value) {
            if (t + from >= tl) v0 = make_uint4(0, 0, 0, 0);
            if (t + from + 1 >= tl) v1 = make_uint4(0, 0, 0, 0);
          }
          const unsigned w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            lo[p] = __byte_perm(w0[p], w1[p], 0x5410);
            hi[p] = __byte_perm(w0[p], w1[p], 0x7632);
          }
        };
        unsigned a0[4], a1[4], a2[4], a3[4];
        words(gs, 0, a0, a1, 0);
        words(gs, 0, a2, a3, 8);
#pragma unroll
        for (int n = 0; n < GROUPS; ++n) {
          unsigned b00[4], b10[4], b01[4], b11[4];
          words(xs, n, b00, b10, 0);
          words(xs, n, b01, b11, 8);
          float sum[4][2][4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            mma_first(sum[p][0], a0[p], a1[p], a2[p], a3[p], b00[p], b01[p], zero);
            mma_first(sum[p][1], a0[p], a1[p], a2[p], a3[p], b10[p], b11[p], zero);
          }
#pragma unroll
          for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              add2(acc[p][n][q][0], sum[p][q][0], sum[p][q][1]);
              add2(acc[p][n][q][1], sum[p][q][2], sum[p][q][3]);
            }
        }
      };
      for (int k0 = 0; k0 < tl; k0 += 16) {
        if (k0 + 16 <= tl) step(k0, std::false_type{});
        else step(k0, std::true_type{});
      }
      barrier_arrive(empty_barrier(buf));
      buf = buf == TG_BUFFERS - 1 ? 0 : buf + 1;
    }
    // ---- a channel pair's four P blocks to shared memory, then the sums along their diagonals, a lane per offset
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const PairItem it = pairs_s[cb * TG_PAIRS + 4 * cg + p];
      __syncwarp();
#pragma unroll
      for (int n = 0; n < GROUPS; ++n)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float* at = p_s + q * TG_BLOCK + g * TG_PS + 8 * n + 2 * c;
          *reinterpret_cast<float2*>(at) = unpack2(acc[p][n][q][0]);                 // component 0 of g
          *reinterpret_cast<float2*>(at + 2 * TG_BLOCK) = unpack2(acc[p][n][q][1]);  // component 1
        }
      __syncwarp();
      if (lane >= valid || it.kind < 0) continue;
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s < 8; ++s) sum += p_s[q * TG_BLOCK + s * TG_PS + s + lane];
        v[q] = sum;
      }
      float* out = a.dtable + (size_t)(a.win_off[w] + d0 + lane) * a.table_width + it.fcol;
      if (it.kind == 0) *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
      else *reinterpret_cast<float2*>(out) = make_float2(v[0], v[3]);
    }
  };
  for (int cb = 0; cb < n_cb; ++cb) {
    if (groups <= 2) columns(std::integral_constant<int, 2>(), cb);
    else if (groups == 3) columns(std::integral_constant<int, 3>(), cb);
    else columns(std::integral_constant<int, 4>(), cb);
  }
}

// ---------------------------------------------------------------------------------------------------------------- apply
constexpr int AP_GROUP = 5;                              // blocks of 16 columns that a CTA works on one after the other, at most
constexpr int AP_BUFFERS = 3;                             // stages in shared memory
constexpr int AP_COLS = 16;                               // columns of the field at a time: 2 groups of 4 channel pairs x 2 sets of tiles
constexpr int AP_PAIRS = AP_COLS / 2;
constexpr int AP_TILES = 64;                              // tiles of 8 longitudes per CTA, of one sample or of several
constexpr int AP_STEPS = 3;                               // k-steps of 8 positions per stage
constexpr int AP_HALO = AP_STEPS - 1;                     // tiles staged beyond a sample's last
constexpr int AP_STAGED = 72;                             // staged tiles: the CTA's and the samples' halos
constexpr int AP_PITCH = 2;                               // 16-byte words per staged position
// A lane reads position c of tile t, eight lanes (c = 0 .. 3, two t) at a time: the planes of c start 0, 1, 4, 5 words off a
// multiple of eight, so that their sixteen-byte words 2 t + 0, 1, 4, 5 and 2 (t + 1) + 0, 1, 4, 5 fall on different banks
constexpr int AP_SP = AP_STAGED * AP_PITCH + 8;
static_assert(AP_SP % 8 == 0, "conflict-free 16-byte loads");
constexpr int AP_SLOTS = 32;                              // offsets -7 .. 24 of a stage's first position, 8 bytes each
constexpr int AP_PAIR = 3 * AP_SLOTS + 1;                 // 8-byte words per channel pair
constexpr int AP_STAGE = 8 * AP_SP + (AP_PAIRS * AP_PAIR * 8 + 15) / 16;  // 16-byte words
constexpr int AP_MAX_SPAN = 4096;                         // neighbour rows whose windows a CTA lists in shared memory

// What a CTA works on: 16 columns of a target row's longitudes 8 t0 .. 8 (t0 + tl) - 1, the samples b0 .. b0 + nb - 1; their
// tiles, sample by sample, are the columns of its products.
struct ApplyTile {
  int row, col0, t0, tl, b0, nb;
};
struct Window {
  int cnt, lo, off, row;
};
// Stages: positions [r, r + 8 steps) of the cnt + 7 that the eight longitudes of a tile see through a window
struct ApplyStage {
  int w, r, steps;
};
__device__ __forceinline__ ApplyStage stage_at(const Window* windows, int n_windows, int w, int r) {
  return ApplyStage{w, r, w < n_windows ? min(AP_STEPS, (windows[w].cnt + 7 - r + 7) / 8) : 0};
}
__device__ __forceinline__ ApplyStage next_stage(const Window* windows, int n_windows, const ApplyStage& s) {
  const int r = s.r + 8 * s.steps;
  return r < windows[s.w].cnt + 7 ? stage_at(windows, n_windows, s.w, r) : stage_at(windows, n_windows, s.w + 1, 0);
}
// Tile n of the CTA's in the staged tiles
__device__ __forceinline__ int staged_tile(const ApplyTile& t, int n) { return n + AP_HALO * (n / t.tl); }

__device__ __forceinline__ void issue_stage(const ConvArgs& a, const ApplyTile& t, const Window& w, const ApplyStage& s, uint4* dst) {
  const int row_bytes = 2 * a.width, tiles = t.tl + s.steps - 1;
  int lon = 8 * t.t0 + w.lo + s.r;
  while (lon < 0) lon += a.nlon;
  const size_t sample = (size_t)a.rows * a.nlon * row_bytes;
  const unsigned char* row = static_cast<const unsigned char*>(a.x) + t.b0 * sample + (size_t)w.row * a.nlon * row_bytes;
  for (int b = 0; b < t.nb; ++b, row += sample, dst += (t.tl + AP_HALO) * AP_PITCH)
    stage_positions<GROUP, AP_COLS / 8, AP_SP, AP_PITCH, true>(dst, row, lon, 8 * tiles, a.nlon, row_bytes, 2 * t.col0);
  commit();
}
// The matrix of channel pair `it` at offset d of the window
__device__ __forceinline__ float4 table_matrix(const ConvArgs& a, const Window& w, int d, PairItem it) {
  const float* f = a.table + (size_t)(w.off + d) * a.table_width + it.fcol;
  if (it.kind == 0) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(f));
    return a.transpose ? make_float4(v.x, v.z, v.y, v.w) : v;
  }
  const float2 v = __ldg(reinterpret_cast<const float2*>(f));
  return make_float4(v.x, 0.f, 0.f, v.y);
}
// Longitude s of tile n of the CTA's in the result, column col
__device__ __forceinline__ __nv_bfloat16* apply_output(const ConvArgs& a, const ApplyTile& t, int n, int s, int col) {
  const int b = t.b0 + n / t.tl, l = 8 * (t.t0 + n % t.tl) + s;
  return static_cast<__nv_bfloat16*>(a.y) + (((size_t)b * a.rows + t.row) * a.nlon + l) * a.width + col;
}

// The CTA's outputs whose sums were not finite, by themselves: such a sum may owe it to a value outside its window (0 x Inf) or
// to another component, so it is formed again from its own neighbours alone, on the FMA pipe from the staged positions.  A warp
// leaves out the channel pairs that have no such output, or none that is not NaN already (and stays so).  `bad`: bit
// 8 p + 2 i + e = channel pair p at longitude g of tile 8 (half + 2 i) + 2 c + e.
__device__ __forceinline__ void apply_again(const ConvArgs& a, const ApplyTile& tile, const Window* windows, int n_windows, uint4* stage_s,
                                         const PairItem* pairs_s, unsigned bad) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, cg = warp & 1, half = warp >> 1;
  float2 y[4][4][2];
  int at[4][2];  // word of position 0 of the tiles' eight
  bool open[4];  // pairs the warp still works on
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    open[p] = __any_sync(0xffffffffu, bad >> 8 * p & 0xff);
#pragma unroll
    for (int i = 0; i < 4; ++i) y[p][i][0] = y[p][i][1] = make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) at[i][e] = 4 * (staged_tile(tile, min(8 * (half + 2 * i) + 2 * c + e, tile.nb * tile.tl - 1)) * AP_PITCH + cg);
  ApplyStage s = stage_at(windows, n_windows, 0, 0);
  if (s.w < n_windows) issue_stage(a, tile, windows[s.w], s, stage_s);
  int buf = 0;
  while (s.w < n_windows) {
    const Window win = windows[s.w];
    const ApplyStage nxt = next_stage(windows, n_windows, s);
    wait_copies<0>();
    consumer_sync();
    if (nxt.w < n_windows) issue_stage(a, tile, windows[nxt.w], nxt, stage_s + (buf ^ 1) * AP_STAGE);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if (!open[p]) continue;
      const PairItem it = pairs_s[4 * cg + p];
      const unsigned* words = reinterpret_cast<const unsigned*>(stage_s + buf * AP_STAGE) + p;
      // position r of the window is offset r - g of the lane's longitudes
      auto matrix = [&](int r) { return table_matrix(a, win, min(max(s.r + r - g, 0), win.cnt - 1), it); };
      float4 next = matrix(0);
      for (int r = 0; r < 8 * s.steps; ++r) {
        const float4 m = next;
        next = matrix(min(r + 1, 8 * s.steps - 1));
        if (s.r + r < g || s.r + r - g >= win.cnt) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const unsigned w = words[at[i][e] + 4 * (plane<AP_SP, true>(r & 7) + (r >> 3) * AP_PITCH)];
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
    if (!consumer_or(open[0] || open[1] || open[2] || open[3])) break;
    s = nxt;
    buf ^= 1;
  }
  wait_copies<0>();
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (bad >> (8 * p + 2 * i + e) & 1)
          *reinterpret_cast<__nv_bfloat162*>(apply_output(a, tile, 8 * (half + 2 * i) + 2 * c + e, g, tile.col0 + 8 * cg + 2 * p)) =
              __floats2bfloat162_rn(y[p][i][e].x, y[p][i][e].y);
}

__global__ void __launch_bounds__(2 * GROUP, 2) conv_apply_tc_kernel(const __grid_constant__ ConvArgs a, int col_blocks, int single_rows, int single_ctas, int group,
                                                                     int lon_blocks, int samples) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PairItem pairs_s[AP_GROUP * AP_PAIRS];
  __shared__ unsigned bad_s[AP_GROUP][GROUP];
  __shared__ int n_windows_s;
  int x = blockIdx.x, first_row = 0;
  if (x < single_ctas) {
    group = 1;
  } else {
    x -= single_ctas;
    first_row = single_rows;
  }
  const int groups = (col_blocks + group - 1) / group, cb0 = x % groups * group, n_cb = min(group, col_blocks - cb0);
  x /= groups;
  const int lb = x % lon_blocks;
  x /= lon_blocks;
  const int chunks = (a.batch + samples - 1) / samples, b0 = (x % chunks) * samples, row = a.order[first_row + x / chunks];  // heaviest rows first
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, cg = warp & 1, half = warp >> 1 & 1;
  const int T = a.nlon / 8, per = (T + lon_blocks - 1) / lon_blocks, t0 = lb * per;
  ApplyTile tile{row, cb0 * AP_COLS, t0, min(per, T - t0), b0, min(samples, a.batch - b0)};
  const int n_tiles = tile.nb * tile.tl, mine = ((n_tiles + 7) / 8 - half + 1) / 2;  // this warp's eights of tiles: half, half + 2, ...
  uint4* const stage_s = reinterpret_cast<uint4*>(smem);
  Window* const windows = reinterpret_cast<Window*>(stage_s + AP_BUFFERS * AP_STAGE);
  if (warp == 0) {
    const int span = 2 * a.halo + 1;
    int filled = 0;
    for (int w0 = 0; w0 < span; w0 += 32) {
      const int w = w0 + lane, j = row + w - a.halo, cnt = w < span && j >= 0 && j < a.rows ? a.win_cnt[row * span + w] : 0;
      const unsigned have = __ballot_sync(0xffffffffu, cnt > 0);
      if (cnt > 0) windows[filled + __popc(have & ((1u << lane) - 1u))] = Window{cnt, a.win_lo[row * span + w] % a.nlon, a.win_off[row * span + w], j};
      filled += __popc(have);
    }
    if (lane == 0) n_windows_s = filled;
  }
  find_items<AP_GROUP * AP_COLS, 2 * GROUP>(a, tile.col0, pairs_s);
  const int n_windows = n_windows_s;

  if (warp >= GROUP / 32) {
    // ---- producers
    producer_registers();
    // this thread's two slots of the split table: a channel pair and the offsets slot - 7 from the stage's first position
    const int tp = threadIdx.x % AP_PAIRS, ts = threadIdx.x % GROUP / AP_PAIRS;
    PairItem item = pairs_s[tp];
    // (the loaded words are looked at by place alone, so that a stage's products run while they are under way)
    auto fetch = [&](const ApplyStage& s, float2 (&m)[2][2]) {
      const Window w = windows[s.w];
      const float* f = a.table + (size_t)w.off * a.table_width + item.fcol;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int d = s.r + ts + 16 * i - 7;
        const bool in = (i == 0 || s.steps > 1) && d >= 0 && d < w.cnt && item.kind >= 0;
        const float2* from = reinterpret_cast<const float2*>(f + (size_t)d * a.table_width);
        m[i][0] = m[i][1] = make_float2(0.f, 0.f);
        if (in) m[i][0] = __ldg(from);
        if (in && item.kind == 0) m[i][1] = __ldg(from + 1);
      }
    };
    auto place = [&](int buf, const ApplyStage& s, const PairItem& item, const float2 (&m)[2][2]) {
      uint2* dst = reinterpret_cast<uint2*>(stage_s + buf * AP_STAGE + 8 * AP_SP) + tp * AP_PAIR + ts;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (i == 1 && s.steps == 1) break;  // one k-step reads 15 slots
        float4 v = make_float4(m[i][0].x, m[i][0].y, m[i][1].x, m[i][1].y);
        if (item.kind == 1) v = make_float4(v.x, 0.f, 0.f, v.y);
        else if (a.transpose) v = make_float4(v.x, v.z, v.y, v.w);
        unsigned w0[3], w1[3];
        split3(v.x, v.y, w0);
        split3(v.z, v.w, w1);
#pragma unroll
        for (int q = 0; q < 3; ++q) dst[q * AP_SLOTS + 16 * i] = make_uint2(w0[q], w1[q]);
      }
    };

    ApplyStage cur = stage_at(windows, n_windows, 0, 0);
    float2 m[2][2];
    if (cur.w < n_windows) fetch(cur, m);
    Ring<AP_BUFFERS, 1> ring;
    for (int cb = 0; n_windows > 0 && cb < n_cb;) {
      ring.begin();
      issue_stage(a, tile, windows[cur.w], cur, stage_s + ring.buf * AP_STAGE);
      const PairItem placed = item;
      ApplyStage nxt = next_stage(windows, n_windows, cur);
      if (nxt.w == n_windows) {  // on to the next columns
        nxt = stage_at(windows, n_windows, 0, 0);
        ++cb;
        tile.col0 += AP_COLS;
        if (cb < n_cb) item = pairs_s[cb * AP_PAIRS + tp];
      }
      float2 ahead[2][2];
      if (cb < n_cb) fetch(nxt, ahead);
      place(ring.buf, cur, placed, m);
#pragma unroll
      for (int i = 0; i < 2; ++i) { m[i][0] = ahead[i][0]; m[i][1] = ahead[i][1]; }
      cur = nxt;
      ring.advance();
    }
    ring.drain();
    return;
  }
  // ---- consumers
  consumer_registers();
  // (zeros and the identity of a byte permutation that the compiler does not see through: it would clear four registers for every
  // product that starts a chain, and pair the words of a B operand again for each of its three products)
  float zero[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) zero[v] = __int_as_float(a.nlon >> 31 & (v + 1));
  const unsigned same = a.nlon > 0 ? 0x3210u : 0u;
  int at[4];  // 16-byte word of position c of this lane's tiles
#pragma unroll
  for (int i = 0; i < 4; ++i) at[i] = plane<AP_SP, true>(c) + staged_tile(tile, min(8 * (half + 2 * i) + g, n_tiles - 1)) * AP_PITCH + cg;

  int buf = 0;
  for (int cb = 0; cb < n_cb; ++cb, tile.col0 += AP_COLS) {
    f32x2 acc[4][4][2];  // channel pair, eight of tiles: rows (s = g: component 0, g + 8: component 1), columns t = 2 c, 2 c + 1
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[p][i][0] = acc[p][i][1] = 0;
    ApplyStage cur = stage_at(windows, n_windows, 0, 0);
    while (cur.w < n_windows) {
      barrier_sync(full_barrier(buf));
      const uint4* xs = stage_s + buf * AP_STAGE;
      const uint2* ms = reinterpret_cast<const uint2*>(stage_s + buf * AP_STAGE + 8 * AP_SP) + 4 * cg * AP_PAIR + 7 + c - g;
      auto walk = [&](auto count) {
        constexpr int MINE = decltype(count)::value;
        for (int k = 0; k < cur.steps; ++k) {
          unsigned fb[MINE][2][4];
#pragma unroll
          for (int i = 0; i < MINE; ++i) {
            const uint4* from = xs + at[i] + k * AP_PITCH;
            const uint4 v0 = from[0], v4 = from[4 * AP_SP];
            fb[i][0][0] = v0.x; fb[i][0][1] = v0.y; fb[i][0][2] = v0.z; fb[i][0][3] = v0.w;
            fb[i][1][0] = v4.x; fb[i][1][1] = v4.y; fb[i][1][2] = v4.z; fb[i][1][3] = v4.w;
          }
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const uint2* f = ms + p * AP_PAIR + 8 * k;
            const uint2 l01 = f[2 * AP_SLOTS], l23 = f[2 * AP_SLOTS + 4], m01 = f[AP_SLOTS], m23 = f[AP_SLOTS + 4], h01 = f[0], h23 = f[4];
            float sum[MINE][4];
            unsigned b0[MINE], b1[MINE];
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
              b0[i] = __byte_perm(fb[i][0][p], 0, same);
              b1[i] = __byte_perm(fb[i][1][p], 0, same);
            }
#pragma unroll
            for (int i = 0; i < MINE; ++i) mma_first(sum[i], l01.x, l01.y, l23.x, l23.y, b0[i], b1[i], zero);
#pragma unroll
            for (int i = 0; i < MINE; ++i) mma(sum[i], m01.x, m01.y, m23.x, m23.y, b0[i], b1[i]);
#pragma unroll
            for (int i = 0; i < MINE; ++i) mma(sum[i], h01.x, h01.y, h23.x, h23.y, b0[i], b1[i]);
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
              add2(acc[p][i][0], sum[i][0], sum[i][1]);
              add2(acc[p][i][1], sum[i][2], sum[i][3]);
            }
          }
        }
      };
      if (mine == 4) walk(std::integral_constant<int, 4>());
      else if (mine == 3) walk(std::integral_constant<int, 3>());
      else if (mine == 2) walk(std::integral_constant<int, 2>());
      else if (mine == 1) walk(std::integral_constant<int, 1>());
      barrier_arrive(empty_barrier(buf));
      cur = next_stage(windows, n_windows, cur);
      buf = buf == AP_BUFFERS - 1 ? 0 : buf + 1;
    }

    // ---- four channel pairs of a position are 16 bytes of its row
    const int col = tile.col0 + 8 * cg;
    unsigned bad = 0;  // outputs whose sums are not finite
    if (col < a.width) {
      bool whole = true;
#pragma unroll
      for (int p = 0; p < 4; ++p) whole = whole && pairs_s[cb * AP_PAIRS + 4 * cg + p].kind >= 0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int n = 8 * (half + 2 * i) + 2 * c + e;
          if (n >= n_tiles) continue;
          unsigned word[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const float2 re = unpack2(acc[p][i][0]), im = unpack2(acc[p][i][1]);
            const float2 v = e ? make_float2(re.y, im.y) : make_float2(re.x, im.x);
            if (!(fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY) && pairs_s[cb * AP_PAIRS + 4 * cg + p].kind >= 0) bad |= 1u << (8 * p + 2 * i + e);
            const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
            word[p] = *reinterpret_cast<const unsigned*>(&h);
          }
          __nv_bfloat16* out = apply_output(a, tile, n, g, col);
          if (whole) {
            *reinterpret_cast<uint4*>(out) = make_uint4(word[0], word[1], word[2], word[3]);
          } else {
#pragma unroll
            for (int p = 0; p < 4; ++p)
              if (pairs_s[cb * AP_PAIRS + 4 * cg + p].kind >= 0) *reinterpret_cast<unsigned*>(out + 2 * p) = word[p];
          }
        }
    }
    bad_s[cb][threadIdx.x] = bad;
  }
  tile.col0 = cb0 * AP_COLS;
  for (int cb = 0; cb < n_cb; ++cb, tile.col0 += AP_COLS) {
    const unsigned bad = bad_s[cb][threadIdx.x];
    if (consumer_or(bad != 0)) apply_again(a, tile, windows, n_windows, stage_s, pairs_s + cb * AP_PAIRS, bad);
  }
}

}  // namespace

bool tensor_cores_can(const ConvArgs& a) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.g) | reinterpret_cast<uintptr_t>(a.y);
  return a.nlon % 8 == 0 && a.width % 8 == 0 && bits % 16 == 0;
}
bool tensor_cores_hold(const ConvArgs& a) { return 2 * (int64_t)a.halo + 1 <= AP_MAX_SPAN; }

// How apply cuts a field: blocks of columns, of tiles along a row, and samples that share a CTA: of a short row as many as its
// tiles hold with their halos
struct ApplyGrid {
  int col_blocks, lon_blocks, samples;
  int64_t per_block;  // CTAs of a row and a block of columns
};
static ApplyGrid apply_grid(const ConvArgs& a) {
  const int T = a.nlon / 8, lon_blocks = (T + AP_TILES - 1) / AP_TILES, per = (T + lon_blocks - 1) / lon_blocks;
  const int samples = lon_blocks > 1 ? 1 : std::max(1, std::min({a.batch, AP_TILES / per, AP_STAGED / (per + AP_HALO)}));
  return {(a.width + AP_COLS - 1) / AP_COLS, lon_blocks, samples, (int64_t)lon_blocks * ((a.batch + samples - 1) / samples)};
}

// The FMA kernels stay the faster ones where the tiles are mostly padding and there are enough of them to fill the chip.  333
// shapes from 24 x 24 to 256 x 512, batch 1 to 4, widths 24 to 320, us FMA / tensor cores:
//   apply        a CTA takes up to 64 tiles of 8 longitudes.  From 32 on it is the faster one (128 x 128, width 320, batch 2: 179 / 179, batch
//                4: 333 / 237; 256 x 512, width 320: 1 336 / 540), with fewer while the launch has few CTAs and lasts as long as the polar
//                rows' chains of stages, which are shorter here (64 x 128, batch 1, width 160: 81 / 42, width 320: 78 / 70; 128 x 128, batch
//                1, width 160: 116 / 81, but width 320: 112 / 154).  With up to 8 tiles a row the FMA kernel's chains are short too (32 x 64:
//                50 / 25, width 320: 48 / 47; 200 x 48, width 24: 24 / 22, width 40: 24 / 28, width 320: 28 / 116).
//   table_grad   contracts over the tiles of all samples, 16 a step; the FMA kernel takes samples by two.  The least tiles by samples and
//                width are where radius 2, 2.5, 3 and 4 rows come out even (736 timings, 9 to 32 tiles; the share of the FMA time for each radius): one
//                sample, width 320, 22 tiles 1.18, 0.99, 1.08, 0.98, 24 1.11, 0.89, 0.95, 0.90; width 160, 18 tiles 1.29, 1.22, 0.92, 0.95, 20 1.14, 0.86, 0.91,
//                0.87; two, width 320, 20 tiles 1.14, 1.00, 1.06, 0.96, 22 1.09, 0.95, 0.96, 0.87; width 160, 13 tiles 0.97, 1.01, 1.02, 0.88, 16 0.99, 0.82,
//                0.81, 0.79; width 96, 11 tiles 1.12, 1.01, 1.27, 1.02, 13 0.89, 0.94, 0.89, 0.81; three, width 96, 9 tiles 0.77, width 320, 11 tiles 0.82 and (radius 4)
//                0.74.  One block of 32 columns always (9 tiles 0.50), 8 tiles with three samples or four (35 x 64: 23 / 15 us, 32 x 64: 32 / 22).  256 x 512: 1 701 / 738 us.
bool tensor_cores_apply(const ConvArgs& a) {
  if (!tensor_cores_can(a) || !tensor_cores_hold(a)) return false;
  const int T = a.nlon / 8;
  const ApplyGrid grid = apply_grid(a);
  const int64_t ctas = grid.per_block * grid.col_blocks * a.rows, fill = (int64_t)grid.samples * std::min(T, AP_TILES);
  return T > 8 ? fill >= 32 || ctas <= 80 * fill : T >= 3 && ctas <= 80 * T;
}
bool tensor_cores_table_grad(const ConvArgs& a) {
  const bool narrow = a.width <= TG_COLS;
  const int by_width = a.width <= 96 ? 0 : a.width <= 160 ? 1 : 2;
  constexpr int LEAST[4][3] = {{20, 20, 24}, {13, 16, 22}, {9, 11, 11}, {9, 9, 9}};  // samples, width
  const int least = narrow ? (a.batch >= 3 ? 8 : 9) : LEAST[std::min(a.batch, 4) - 1][by_width];
  return tensor_cores_can(a) && a.nlon / 8 >= least;
}

int apply_tc(const ConvArgs& a, int n_order, cudaStream_t stream) {
  const ApplyGrid grid = apply_grid(a);
  // Light rows take several blocks of columns one after the other while that leaves six waves of CTAs (256 x 512, radius 4 pi / 256,
  // batch 4, width 320: 2 134 us one, 2 053 two, 2 011 five at a time); the heaviest rows, whose chains of stages a launch could
  // end in, always one (128 x 256, batch 2: every row five at a time 424 us, one 277).
  const int single_rows = (n_order + 7) / 8;
  const int64_t light = grid.per_block * grid.col_blocks * (n_order - single_rows);
  const int group = (int)std::max<int64_t>(1, std::min<int64_t>({AP_GROUP, grid.col_blocks, light / (12 * sm_count())}));
  const int64_t singles = grid.per_block * grid.col_blocks * single_rows;
  const int64_t ctas = singles + grid.per_block * ((grid.col_blocks + group - 1) / group) * (n_order - single_rows);
  GM_REQUIRE(ctas < (1ll << 31), GM_ERR_LIMIT, "gm_lattice_conv_apply: too many tiles");
  const size_t smem = AP_BUFFERS * (size_t)AP_STAGE * 16 + (2 * (size_t)a.halo + 1) * sizeof(Window);
  const int st = allow_smem(conv_apply_tc_kernel, smem, "gm_lattice_conv_apply");
  if (st != GM_OK) return st;
  conv_apply_tc_kernel<<<(unsigned)ctas, 2 * GROUP, smem, stream>>>(a, grid.col_blocks, single_rows, (int)singles, group, grid.lon_blocks, grid.samples);
  return launch_status("gm_lattice_conv_apply");
}

int table_grad_tc(const ConvArgs& a, int64_t n_blocks, cudaStream_t stream) {
  const int col_blocks = (a.width + TG_COLS - 1) / TG_COLS;
  const int group = std::min(TG_GROUP, col_blocks);
  const size_t smem = TG_BUFFERS * (size_t)TG_STAGE * 16 + (GROUP / 32) * 4 * TG_BLOCK * sizeof(float);
  const int st = allow_smem(conv_table_grad_tc_kernel, smem, "gm_lattice_conv_table_grad");
  if (st != GM_OK) return st;
  conv_table_grad_tc_kernel<<<dim3((unsigned)n_blocks, (col_blocks + group - 1) / group), 2 * GROUP, smem, stream>>>(a, (int)n_blocks, col_blocks, group);
  return launch_status("gm_lattice_conv_table_grad");
}

}  // namespace lconv
}  // namespace gmb
