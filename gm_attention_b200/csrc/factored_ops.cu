// The factored steerable kernel behind the reference extension's entry points
// forward / aggregate / backward / backward_aggregated
// (src/gm_attention/nn/fused/factored_cpu.cpp:77-219; arithmetic
// src/gm_attention/nn/fused/factored.h:118-347).
//
// Per edge e with source j:  row_e = sum over blocks of F_b(e) * sum_t h~_t(e) Z_{t,b}(j),
// h~ = (1, h), F_b = e^{i ang phi} e^{i trn gamma} (r / c)^p (negative orders conjugate,
// the power by repeated multiplication), blocks that share an output offset summed
// before the write, rows n -> 0 keep the real part.
//
// Forward: one CTA per source node (the caller's grouping order / group_ptr /
// group_source), Z(j) staged once in shared memory, the source's edges in tiles of
// 64.  The packed width 2 wc + wr is bounded only by shared memory (the reference
// stops at 320); what the tiles cannot hold has a form of its own.
//
// The edges of a source are scattered over the target-major edge list, so their records (h, both phase rows, rho; the
// gradient row in the backward) are copied into shared memory element by element, consecutive threads taking consecutive
// elements of one edge: read by the edge's own thread straight from global memory, each of the ~60 loads of the forward
// touched 32 lines.  With the register tiles below, on 128 x 256, radius 3 pi / 128 (3.0 M edges), 13 blocks to {4, 4, 4},
// trunk 16, float32: forward 1.40 -> 1.36 ms, backward 4.64 -> 2.56; sources taken from both ends of the list: 1.30, 2.48.
//
// Backward: one CTA per source again, so dZ(j) needs no atomics.  Edges are taken
// in tiles; the CTA builds its edges' packed rows W(e) = scale * G conj(F) in shared
// memory, then forms dh(e, t) = <W(e), Z_t(j)> and dZ(t, c) += h~_t(e) W_c(e).  Both are small matrix products whose
// bound is shared-memory bandwidth, so both run on register tiles: 2 edges x 4 t over 4 columns per step for dh (6
// 16-byte reads for 32 multiply-adds), 5 t x 4 columns over 4 edges per step for dZ (9 reads for 80), the latter owned by
// fixed threads for the whole source.
#include "factored.cuh"

namespace gmb {
namespace {

using namespace factored;

constexpr int FMAX_K = 20;
constexpr int FTHREADS = 128;
constexpr int MAX_TILE = 64;       // edges per tile, at most (a power of two; less where shared memory is short)
constexpr int MAX_OWNED = 64;      // K * C <= 64 * 128 in the backward
// A tile of 64 edges while six CTAs of it share an SM, 32 beyond: a wide packed row (13 blocks to {4, 4, 4}: 100 columns, 53 KB at
// 64 edges) leaves four CTAs' warps to hide the barriers, a narrow one (18 columns) pays them twice as often for nothing.
// 128 x 256, radius 3 pi / 128, 100 columns: forward 1 309 us with 64 edges, 1 034 with 32, 1 122 with 16; backward 2 494, 2 460, 3 076.
// Narrow rows lose with 32: 118 x 236, radius 4 pi / 118, 18 columns, the pass 4.08 -> 4.50 ms.  Between: the pass at 64 x 128, radius
// 3 pi / 64, 13 blocks to {2, 2, 2} (50 columns) 984 -> 988 us, to {8, 8, 8} (200) 2 546 -> 1 874.  float64, whose rows are twice as
// wide: 18 columns 994 -> 992, 36 3 160 -> 2 497 (radius 4), 50 1 660 -> 1 458, 100 2 637 -> 2 187, 200 5 948 -> 4 220.
constexpr size_t FSMEM_SIXTH = 227 * 1024 / 6 - 1024;
constexpr size_t FSMEM_MOST = 224 * 1024;  // dynamic shared memory a CTA may ask for, beside the static arrays
constexpr int TP = 5;              // rows t of a dZ patch (4 columns wide)

// An edge's record in shared memory: angular phases (n_f, 2), transport phases (n_f, 2), rho or the scales; odd pitch.
__host__ __device__ inline int record_pitch(int n_f, int n_scales) { return n_scales ? (4 * n_f + n_scales) | 1 : 4 * n_f + 1; }

// One element global -> shared, asynchronously.
template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(addr), "l"(src), "n"((int)sizeof(T)) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// f(le, w) for every edge le < n of a tile and every element w < width of its row: consecutive threads on consecutive
// elements, one division per thread and call (a division per element cost as much as the rows' arithmetic)
template <typename F>
__device__ __forceinline__ void for_rows(int n, int width, const F& f) {
  if (width <= 0) return;
  const int per = max(FTHREADS / width, 1), le0 = (int)threadIdx.x / width;
  if (width <= FTHREADS) {
    const int w = (int)threadIdx.x - le0 * width;
    if (le0 < per)
      for (int le = le0; le < n; le += per) f(le, w);
  } else {
    for (int le = 0; le < n; ++le)
      for (int w = threadIdx.x; w < width; w += FTHREADS) f(le, w);
  }
}

// dst[le][w] = src[row_s[le] * width + w]
template <typename T>
__device__ __forceinline__ void stage_rows(T* dst, int pitch, const T* src, int width, int n, const int64_t* row_s) {
  for_rows(n, width, [&](int le, int w) { copy_async(dst + le * pitch + w, src + row_s[le] * width + w); });
}

// The records of n edges (edges_s: their indices)
template <bool SCALED, typename T>
__device__ __forceinline__ void stage_records(const FArgs<T>& a, const int64_t* edges_s, int n, T* rec) {
  const int w = 2 * a.n_f, pitch = record_pitch(a.n_f, SCALED ? a.n_scales : 0);
  stage_rows(rec, pitch, a.angular, w, n, edges_s);
  stage_rows(rec + w, pitch, a.transport, w, n, edges_s);
  stage_rows(rec + 2 * w, pitch, a.rho, SCALED ? a.n_scales : 1, n, edges_s);
}

// The block's per-edge factor (factored.h:118-144), from the edge's record; SCALED: "power" names a scale.
template <bool SCALED, typename T>
__device__ __forceinline__ void block_factor(const T* rec, int n_f, const int32_t* d, T& fr, T& fi) {
  fr = T(1);
  fi = T(0);
  const int ang = d[3], trn = d[4], power = d[5];
  if (ang != 0) {
    const int o = ang < 0 ? -ang : ang;
    const T pr = rec[2 * o], pi = ang < 0 ? -rec[2 * o + 1] : rec[2 * o + 1];
    const T nr = fr * pr - fi * pi, ni = fr * pi + fi * pr;
    fr = nr;
    fi = ni;
  }
  if (trn != 0) {
    const int o = trn < 0 ? -trn : trn;
    const T* t = rec + 2 * n_f;
    const T pr = t[2 * o], pi = trn < 0 ? -t[2 * o + 1] : t[2 * o + 1];
    const T nr = fr * pr - fi * pi, ni = fr * pi + fi * pr;
    fr = nr;
    fi = ni;
  }
  T s = T(1);
  if constexpr (SCALED) {
    s = rec[4 * n_f + power];
  } else {
    const T r = rec[4 * n_f];
    for (int x = 0; x < power; ++x) s *= r;
  }
  fr *= s;
  fi *= s;
}
// Z(j) of one node into shared memory: row t = [zc (wc, 2) | zr (wr)], `pitch` elements apart; asynchronous.
template <typename T>
__device__ __forceinline__ void stage_node(const FArgs<T>& a, int64_t j, T* z_s, int pitch) {
  const int wc2 = 2 * a.wc;
  const T* zc = a.zc + j * a.k * wc2;
  const T* zr = a.zr + j * a.k * a.wr;
  for_rows(a.k, wc2, [&](int t, int c) { copy_async(z_s + t * pitch + c, zc + t * wc2 + c); });
  for_rows(a.k, a.wr, [&](int t, int c) { copy_async(z_s + t * pitch + wc2 + c, zr + t * a.wr + c); });
}

template <typename T> struct Vec4 { T v[4]; };
template <typename T>
__device__ __forceinline__ Vec4<T> load4(const T* p) {  // 16-byte aligned
  Vec4<T> r;
  if constexpr (sizeof(T) == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    r.v[0] = q.x; r.v[1] = q.y; r.v[2] = q.z; r.v[3] = q.w;
  } else {
    const double2 q0 = *reinterpret_cast<const double2*>(p), q1 = *reinterpret_cast<const double2*>(p + 2);
    r.v[0] = q0.x; r.v[1] = q0.y; r.v[2] = q1.x; r.v[3] = q1.y;
  }
  return r;
}

template <typename T>
__device__ __forceinline__ void store4(T* p, const T (&v)[4]) {  // 16-byte aligned
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
  }
}

// Forward, per tile of a source's edges: U(c, e) = sum_t h~_t(e) Z_t(c) as a matrix product in register tiles of 4 edges x
// 4 packed columns (two 16-byte reads for 16 multiply-adds), the blocks' factors F(b, e), then a thread per (edge, output
// column) adds up its blocks.  Everything indexed by edge has the edge fastest, so a warp's 32 edges read one line.
// (A thread per edge that walked the blocks with all of Z broadcast measured 1.40 ms, 1.62 with staged records alone; this
// form 1.36.)
template <typename T>
struct ForwardLayout {  // shared memory, in elements of T
  int tile, pitch, cols, e_pitch, rec_pitch, row_pitch;
  int z, h, u, f, rec, total;
  __host__ __device__ ForwardLayout(int k, int C, int n_f, int n_scales, int n_blocks, int d_out, int tile_) {
    tile = tile_;
    cols = (C + 3) / 4 * 4;
    pitch = cols;
    e_pitch = tile + 4;
    rec_pitch = record_pitch(n_f, n_scales);
    row_pitch = d_out | 1;
    z = 0;
    h = z + k * pitch;
    u = h + k * e_pitch;
    f = u + cols * e_pitch;
    rec = f + 2 * n_blocks * tile;  // the records; the finished rows afterwards
    total = (rec + tile * (rec_pitch > row_pitch ? rec_pitch : row_pitch) + 3) / 4 * 4;
  }
};

template <typename T, bool SCALED>
__global__ void __launch_bounds__(FTHREADS) factored_forward_kernel(FArgs<T> a, int tile) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int64_t edges_s[MAX_TILE];
  __shared__ int n_out_s;
  const int wc2 = 2 * a.wc, C = wc2 + a.wr;
  const ForwardLayout<T> L(a.k, C, a.n_f, SCALED ? a.n_scales : 0, a.n_blocks, a.d_out, tile);
  T* base_s = reinterpret_cast<T*>(raw);
  T* z_s = base_s + L.z;      // (k, pitch)
  T* h_s = base_s + L.h;      // (k, e_pitch): h~ transposed
  T* u_s = base_s + L.u;      // (cols, e_pitch)
  T* f_s = base_s + L.f;      // (n_blocks, 2, tile)
  T* rec_s = base_s + L.rec;  // (tile, rec_pitch), then rows (tile, row_pitch)
  int4* block_s = reinterpret_cast<int4*>(base_s + L.total);            // (n_blocks): U row 0, F row (-1: none), columns
  int4* out_s = block_s + a.n_blocks;                                   // (<= d_out): first block, blocks, column, output column (~: real)
  int32_t* desc_s = reinterpret_cast<int32_t*>(out_s + a.d_out);        // (n_blocks, FDESC)
  for (int x = threadIdx.x; x < L.rec; x += FTHREADS) base_s[x] = T(0);  // padding columns and edges beyond a tile stay finite
  for (int x = threadIdx.x; x < a.n_blocks * FDESC; x += FTHREADS) desc_s[x] = a.desc[x];
  __syncthreads();
  if (threadIdx.x == 0) {
    // blocks are sorted by output offset; blocks of one offset add into the same columns
    int n = 0;
    for (int b = 0; b < a.n_blocks;) {
      int last = b + 1;
      while (last < a.n_blocks && desc_s[last * FDESC + 6] == desc_s[b * FDESC + 6]) ++last;
      const int32_t* d = desc_s + b * FDESC;
      const bool real_column = d[0] == 0 || d[7] != 0;
      for (int c = 0; c < d[2] && n < a.d_out; ++c, ++n) out_s[n] = make_int4(b, last, c, real_column ? ~(d[6] + c) : d[6] + 2 * c);
      b = last;
    }
    n_out_s = n;
  }
  if ((int)threadIdx.x < a.n_blocks) {
    for (int b = threadIdx.x; b < a.n_blocks; b += FTHREADS) {
      const int32_t* d = desc_s + b * FDESC;
      block_s[b] = d[0] == 0 ? make_int4((wc2 + d[1]) * L.e_pitch, -1, d[2], 0) : make_int4(2 * d[1] * L.e_pitch, 2 * b * tile, d[2], 0);
    }
  }
  const int le = threadIdx.x & (tile - 1), sub = threadIdx.x / tile, subs = FTHREADS / tile;
  for (int64_t g0 = blockIdx.x; g0 < a.n_groups; g0 += gridDim.x) {
    const int64_t grp = from_both_ends(g0, a.n_groups);
    const int64_t j = a.group_source[grp], first = a.group_ptr[grp], last = a.group_ptr[grp + 1];
    copy_wait();  // where the source before had no edges, no tile waited for its copies, and these go to the same place
    __syncthreads();
    stage_node(a, j, z_s, L.pitch);
    for (int64_t x0 = first; x0 < last; x0 += tile) {
      const int n_tile = (int)min((int64_t)tile, last - x0);
      __syncthreads();
      if ((int)threadIdx.x < n_tile) edges_s[threadIdx.x] = a.order[x0 + threadIdx.x];
      __syncthreads();
      for_rows(n_tile, a.k - 1, [&](int e, int t) { copy_async(h_s + (t + 1) * L.e_pitch + e, a.h + edges_s[e] * (a.k - 1) + t); });
      stage_records<SCALED>(a, edges_s, n_tile, rec_s);
      if ((int)threadIdx.x < tile) h_s[threadIdx.x] = T(1);
      copy_wait();
      __syncthreads();
      const int eqs = (n_tile + 3) / 4;
      for (int x = threadIdx.x; x < eqs * (L.cols / 4); x += FTHREADS) {
        const int cq = x / eqs, e0 = 4 * (x - cq * eqs);
        const T* zp = z_s + 4 * cq;
        const T* hp = h_s + e0;
        T acc[4][4];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[c][e] = T(0);
#pragma unroll 4
        for (int t = 0; t < a.k; ++t) {
          const Vec4<T> zv = load4(zp + t * L.pitch), hv = load4(hp + t * L.e_pitch);
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[c][e] += hv.v[e] * zv.v[c];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) store4(u_s + (4 * cq + c) * L.e_pitch + e0, acc[c]);
      }
      if (le < n_tile)
        for (int b = sub; b < a.n_blocks; b += subs) {
          if (desc_s[b * FDESC] == 0) continue;
          T fr, fi;
          block_factor<SCALED>(rec_s + le * L.rec_pitch, a.n_f, desc_s + b * FDESC, fr, fi);
          f_s[2 * b * tile + le] = fr;
          f_s[(2 * b + 1) * tile + le] = fi;
        }
      __syncthreads();
      T* row = rec_s + le * L.row_pitch;
      if (le < n_tile)
        for (int n = sub; n < n_out_s; n += subs) {
          const int4 o = out_s[n];
          const int c = o.z;
          T vr = T(0), vi = T(0);
          for (int b = o.x; b < o.y; ++b) {
            const int4 at = block_s[b];
            if (c >= at.z) continue;
            if (at.y < 0) {
              vr += u_s[at.x + c * L.e_pitch + le];
              continue;
            }
            const T* u = u_s + at.x + 2 * c * L.e_pitch + le;
            const T* f = f_s + at.y + le;
            const T ur = u[0], ui = u[L.e_pitch], fr = f[0], fi = f[tile];
            vr += fr * ur;
            vr -= fi * ui;
            vi += fr * ui;
            vi += fi * ur;
          }
          if (o.w < 0) {
            row[~o.w] = vr;
          } else {
            row[o.w] = vr;
            row[o.w + 1] = vi;
          }
        }
      __syncthreads();
      for_rows(n_tile, a.d_out, [&](int e, int c) { a.out[edges_s[e] * a.d_out + c] = rec_s[e * L.row_pitch + c]; });
    }
  }
}

// The forward where the tiled form does not fit: packed rows of thousands of columns over a short trunk (k = 1: 4 460 in
// float32; U takes more room than Z there), phase tables of hundreds of orders.  A thread per edge walks the blocks, all
// threads reading the same address of Z(j); phases come straight from the tables.  571 us against 312 for the tiled form on
// 64 x 128, radius 3 pi / 64, 13 blocks to {4, 4, 4}, trunk 16, float32, so only what that form cannot hold comes here.
template <typename T, bool SCALED>
__global__ void __launch_bounds__(FTHREADS) factored_forward_wide_kernel(FArgs<T> a, int pitch) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int wc2 = 2 * a.wc, nc = a.k * wc2, nr = a.k * a.wr;
  T* zc_s = reinterpret_cast<T*>(raw);  // (k, wc, 2)
  T* zr_s = zc_s + nc;                  // (k, wr)
  T* rows_s = zr_s + (nr + 3) / 4 * 4;  // (FTHREADS, pitch)
  T* row = rows_s + (size_t)threadIdx.x * pitch;
  for (int64_t g0 = blockIdx.x; g0 < a.n_groups; g0 += gridDim.x) {
    const int64_t grp = from_both_ends(g0, a.n_groups);
    const int64_t j = a.group_source[grp], first = a.group_ptr[grp], last = a.group_ptr[grp + 1];
    if (first == last) continue;
    __syncthreads();
    for (int x = threadIdx.x; x < nc; x += FTHREADS) zc_s[x] = a.zc[j * nc + x];
    for (int x = threadIdx.x; x < nr; x += FTHREADS) zr_s[x] = a.zr[j * nr + x];
    __syncthreads();
    for (int64_t x0 = first; x0 < last; x0 += FTHREADS) {
      const int n = (int)min((int64_t)FTHREADS, last - x0);
      if ((int)threadIdx.x < n) {
        const int64_t e = a.order[x0 + threadIdx.x];
        T hh[FMAX_K];
        hh[0] = T(1);
#pragma unroll
        for (int t = 1; t < FMAX_K; ++t) hh[t] = t < a.k ? a.h[e * (a.k - 1) + t - 1] : T(0);
        for (int c = 0; c < a.d_out; ++c) row[c] = T(0);
        for (int b = 0; b < a.n_blocks; ++b) {
          const int32_t* d = a.desc + b * FDESC;
          const int zoff = d[1], bm = d[2];
          T* out = row + d[6];
          if (d[0] == 0) {
            for (int c = 0; c < bm; ++c) {
              T s = T(0);
#pragma unroll
              for (int t = 0; t < FMAX_K; ++t)
                if (t < a.k) s += hh[t] * zr_s[t * a.wr + zoff + c];
              out[c] += s;
            }
            continue;
          }
          T fr, fi;
          table_factor<SCALED>(a, e, d, fr, fi);
          for (int c = 0; c < bm; ++c) {
            T ur = T(0), ui = T(0);
#pragma unroll
            for (int t = 0; t < FMAX_K; ++t)
              if (t < a.k) {
                ur += hh[t] * zc_s[t * wc2 + 2 * (zoff + c)];
                ui += hh[t] * zc_s[t * wc2 + 2 * (zoff + c) + 1];
              }
            const T vr = fr * ur - fi * ui, vi = fr * ui + fi * ur;
            if (d[7] != 0) {
              out[c] += vr;
            } else {
              out[2 * c] += vr;
              out[2 * c + 1] += vi;
            }
          }
        }
      }
      __syncthreads();
      for_rows(n, a.d_out, [&](int r, int c) { a.out[a.order[x0 + r] * a.d_out + c] = rows_s[r * pitch + c]; });
      __syncthreads();
    }
  }
}

// out_i = sum over the target's edges of w_e * row_e  (factored.h:337-347): a warp per target.  What bounds it: the rows' stream, and
// the polar targets' chains of edges.  Lanes are vectors of V columns, and as many edges at a time as the vectors leave room for, whose
// sums meet at the end: one after the other, or (TREE) half of them added to the others at a time.  128 x 256, radius 3 pi / 128, 20
// columns, float32: 45 us (a lane per column, an edge at a time: 120).  The tree is for rows of one or two vectors (40 000 targets of
// 37 edges, 4 columns 30 -> 15 us), and for columns one by one (33: 73 -> 56); with it the compiler has fewer rows under way,
// which longer rows notice (128 columns: 118 -> 129; four rows a step written out: 128 to 141).
template <typename T, int V, bool TREE>
__global__ void aggregate_kernel(const T* __restrict__ rows, const T* __restrict__ weights, const int64_t* __restrict__ row_ptr,
                                 int64_t n_targets, int d_out, T* __restrict__ out) {
  struct alignas(V * sizeof(T)) Vec { T x[V]; };
  const int lane = threadIdx.x & 31, vectors = d_out / V;
  const int64_t x = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (x >= n_targets) return;
  const int64_t i = from_both_ends(x, n_targets);
  const int64_t e0 = row_ptr[i], e1 = row_ptr[i + 1];
  for (int q0 = 0; q0 < vectors; q0 += 32) {
    const int width = min(32, vectors - q0), slots = 32 / width, slot = lane / width, c = V * (q0 + lane % width);
    T acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = T(0);
    if (slot < slots) {
#pragma unroll 4
      for (int64_t e = e0 + slot; e < e1; e += slots) {
        const T w = weights[e];
        const Vec row = *reinterpret_cast<const Vec*>(rows + e * d_out + c);
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += w * row.x[v];
      }
    }
    if constexpr (TREE) {
      for (int n = slots; n > 1;) {
        const int half = (n + 1) / 2;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const T other = __shfl_sync(0xffffffffu, acc[v], (lane + half * width) & 31);
          if (slot + half < n) acc[v] += other;
        }
        n = half;
      }
    } else {
      for (int s = 1; s < slots; ++s) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const T other = __shfl_sync(0xffffffffu, acc[v], (lane + s * width) & 31);
          if (slot == 0) acc[v] += other;
        }
      }
    }
    if (slot == 0) {
      Vec sum;
#pragma unroll
      for (int v = 0; v < V; ++v) sum.x[v] = acc[v];
      *reinterpret_cast<Vec*>(out + i * d_out + c) = sum;
    }
  }
}
// The same with a lane per column, an edge at a time: for many targets of few edges, whose rows are soon read, so that the division
// of the lanes and the meeting of their sums would cost more than they save.
template <typename T>
__global__ void aggregate_columns_kernel(const T* __restrict__ rows, const T* __restrict__ weights, const int64_t* __restrict__ row_ptr,
                                         int64_t n_targets, int d_out, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t x = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (x >= n_targets) return;
  const int64_t i = from_both_ends(x, n_targets);
  const int64_t e0 = row_ptr[i], e1 = row_ptr[i + 1];
  for (int c = lane; c < d_out; c += 32) {
    T acc = T(0);
    for (int64_t e = e0; e < e1; ++e) acc += weights[e] * rows[e * d_out + c];
    out[i * d_out + c] = acc;
  }
}

// Backward.  C = 2 wc + wr packed columns; the rows of Z, W lie at `pitch` >= C elements: a multiple of 4 (16-byte vectors)
// that is an odd number of them (rows of neighbouring edges on different banks); padding columns stay zero.
template <typename T>
struct BackwardLayout {  // shared memory, in elements of T
  int pitch, quads, tgroups, h_pitch, rec_pitch, g_pitch, tile;
  int z, w, h, rec, g, scale, total;
  __host__ __device__ BackwardLayout(int k, int C, int n_f, int n_scales, int d_out, int tile_, bool staged) {
    const int vecs = (C + 3) / 4;
    tile = tile_;
    pitch = 4 * (vecs | 1);
    quads = (k - 1 + 3) / 4;           // groups of 4 trunk rows t = 1 ..
    tgroups = (k + TP - 1) / TP;
    h_pitch = tile + 4;                // h~ transposed: (t, edge)
    rec_pitch = staged ? record_pitch(n_f, n_scales) : 0;
    g_pitch = d_out | 1;
    z = 0;
    const int z_rows = 1 + 4 * quads;
    w = z + z_rows * pitch;
    h = w + tile * pitch;
    rec = h + tgroups * TP * h_pitch;
    g = rec + tile * rec_pitch;
    scale = g + tile * g_pitch;
    total = scale + tile;
  }
};

// NP: dZ patches per thread and pass over the source's edges (wider kernels take several passes).  STAGED: the edges'
// records go through shared memory; phase tables of hundreds of orders leave no room for them and are read where they are.
// (float64 with one patch: four CTAs' registers suffice without spills; left to itself the compiler took 168 for the SCALED form
// and 64 x 128, {2, 2} -> {2, 2}, trunk 8 went from 233 to 291 us)
template <typename T, int NP, bool STAGED, bool SCALED>
__global__ void __launch_bounds__(FTHREADS, (SCALED && sizeof(T) == 8 && NP == 1 ? 4 : 0)) factored_backward_kernel(FArgs<T> a, int C, int tile) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int64_t edges_s[MAX_TILE], g_rows_s[MAX_TILE];  // the tile's edges, and the rows of g that reach them
  const BackwardLayout<T> L(a.k, C, a.n_f, SCALED ? a.n_scales : 0, a.d_out, tile, STAGED);
  const int K = a.k, wc2 = 2 * a.wc, pitch = L.pitch;
  T* base_s = reinterpret_cast<T*>(raw);
  T* z_s = base_s + L.z;      // (1 + 4 quads, pitch): packed per t as [zc (wc, 2) | zr (wr) | 0]
  T* w_s = base_s + L.w;      // (tile, pitch)
  T* h_s = base_s + L.h;      // (TP tgroups, h_pitch)
  T* rec_s = base_s + L.rec;  // (tile, rec_pitch)
  T* g_s = base_s + L.g;      // (tile, g_pitch): the edge's output-gradient row
  T* scale_s = base_s + L.scale;
  for (int x = threadIdx.x; x < L.rec; x += FTHREADS) base_s[x] = T(0);  // padding rows and columns are never written again
  // (C = 0: one quad of padding, so that dh and dweights are written)
  const int col_quads = (max(C, 1) + 3) / 4, patches = L.tgroups * col_quads;
  const int passes = (patches + NP * FTHREADS - 1) / (NP * FTHREADS);
  for (int64_t g0 = blockIdx.x; g0 < a.n_groups; g0 += gridDim.x) {
    const int64_t grp = from_both_ends(g0, a.n_groups);
    const int64_t j = a.group_source[grp], first = a.group_ptr[grp], last = a.group_ptr[grp + 1];
    copy_wait();  // as in the forward
    __syncthreads();
    stage_node(a, j, z_s, pitch);
    for (int pass = 0; pass < passes; ++pass) {
      T acc[NP][TP][4];
#pragma unroll
      for (int o = 0; o < NP; ++o)
#pragma unroll
        for (int t = 0; t < TP; ++t)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[o][t][v] = T(0);
      for (int64_t base = first; base < last; base += tile) {
        const int n_tile = (int)min((int64_t)tile, last - base);
        __syncthreads();
        if ((int)threadIdx.x < n_tile) {
          const int64_t e = a.order[base + threadIdx.x];
          edges_s[threadIdx.x] = e;
          g_rows_s[threadIdx.x] = a.target ? a.target[e] : e;
        }
        __syncthreads();
        if constexpr (STAGED) stage_records<SCALED>(a, edges_s, n_tile, rec_s);
        stage_rows(g_s, L.g_pitch, a.g, a.d_out, n_tile, g_rows_s);
        for_rows(n_tile, K - 1, [&](int le, int t) { copy_async(h_s + (t + 1) * L.h_pitch + le, a.h + edges_s[le] * (K - 1) + t); });
        // edges beyond the tile's end (their h~ multiplies whatever W rows an earlier tile left): zero
        for (int x = threadIdx.x; x < (tile - n_tile) * K; x += FTHREADS) h_s[(x % K) * L.h_pitch + n_tile + x / K] = T(0);
        if ((int)threadIdx.x < n_tile) {
          h_s[threadIdx.x] = T(1);
          scale_s[threadIdx.x] = a.weights ? a.weights[edges_s[threadIdx.x]] : T(1);
        }
        // rows of W beyond the tile's end: zero as well, a non-finite leftover must not meet that zero
        for (int x = threadIdx.x; x < (tile - n_tile) * pitch; x += FTHREADS) w_s[n_tile * pitch + x] = T(0);
        copy_wait();
        __syncthreads();
        // W(e): a warp takes 32 edges of one block
        const int le = threadIdx.x & (tile - 1);
        for (int b = threadIdx.x / tile; b < a.n_blocks && le < n_tile; b += FTHREADS / tile) {
          const int32_t* d = a.desc + b * FDESC;
          const int kind = d[0], zoff = d[1], bm = d[2], ooff = d[6];
          const bool take_real = d[7] != 0;
          const T scale = scale_s[le];
          const T* g = g_s + le * L.g_pitch + ooff;
          T* w = w_s + le * pitch;
          if (kind == 0) {
            for (int c = 0; c < bm; ++c) w[wc2 + zoff + c] = scale * g[c];
          } else {
            T fr, fi;
            if constexpr (STAGED) block_factor<SCALED>(rec_s + le * L.rec_pitch, a.n_f, d, fr, fi);
            else table_factor<SCALED>(a, edges_s[le], d, fr, fi);
            for (int c = 0; c < bm; ++c) {
              const T gr = scale * (take_real ? g[c] : g[2 * c]);
              const T gi = take_real ? T(0) : scale * g[2 * c + 1];
              w[(zoff + c) * 2] = gr * fr + gi * fi;  // W = G conj(F)
              w[(zoff + c) * 2 + 1] = gi * fr - gr * fi;
            }
          }
        }
        if (a.dweights && pass == 0) {  // dweights_e = <g_i, row_e>: eight lanes per edge
          const int sub = threadIdx.x & 7;
          for (int l0 = 0; l0 < n_tile; l0 += FTHREADS / 8) {
            const int le = l0 + (threadIdx.x >> 3);
            T s = T(0);
            if (le < n_tile)
              for (int c = sub; c < a.d_out; c += 8) s += g_s[le * L.g_pitch + c] * a.rows[edges_s[le] * a.d_out + c];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (le < n_tile && sub == 0) a.dweights[edges_s[le]] = s;
          }
        }
        __syncthreads();
        if (pass == 0) {  // dh(e, t) = <W(e), Z_t>, t >= 1: edges le, le + tile / 2 and four t per thread
          const int half = tile / 2;
          for (int x = threadIdx.x; x < half * L.quads; x += FTHREADS) {
            const int le = x / L.quads, t0 = 1 + 4 * (x - le * L.quads);
            const T* w0 = w_s + le * pitch;
            const T* w1 = w0 + half * pitch;
            const T* z = z_s + t0 * pitch;
            T s0[4] = {T(0), T(0), T(0), T(0)}, s1[4] = {T(0), T(0), T(0), T(0)};
            for (int c = 0; c < 4 * col_quads; c += 4) {
              const Vec4<T> v0 = load4(w0 + c), v1 = load4(w1 + c);
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const Vec4<T> zv = load4(z + t * pitch + c);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                  s0[t] += v0.v[v] * zv.v[v];
                  s1[t] += v1.v[v] * zv.v[v];
                }
              }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              if (t0 + t >= K) break;
              if (le < n_tile) a.dh[edges_s[le] * (K - 1) + t0 + t - 1] = s0[t];
              if (le + half < n_tile) a.dh[edges_s[le + half] * (K - 1) + t0 + t - 1] = s1[t];
            }
          }
        }
        // dZ(t, c) += h~_t(e) W_c(e): patch x stays with this thread through the pass
#pragma unroll
        for (int o = 0; o < NP; ++o) {
          const int x = threadIdx.x + (pass * NP + o) * FTHREADS;
          if (x < patches) {
            const int tg = x / col_quads, c = 4 * (x - tg * col_quads);
            const T* hr = h_s + tg * TP * L.h_pitch;
            for (int le = 0; le < n_tile; le += 4) {
              Vec4<T> wv[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) wv[u] = load4(w_s + (le + u) * pitch + c);
#pragma unroll
              for (int t = 0; t < TP; ++t) {
                const Vec4<T> hv = load4(hr + t * L.h_pitch + le);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                  for (int v = 0; v < 4; ++v) acc[o][t][v] += hv.v[u] * wv[u].v[v];
              }
            }
          }
        }
      }
#pragma unroll
      for (int o = 0; o < NP; ++o) {
        const int x = threadIdx.x + (pass * NP + o) * FTHREADS;
        if (x >= patches) continue;
        const int tg = x / col_quads, c0 = 4 * (x - tg * col_quads);
#pragma unroll
        for (int t = 0; t < TP; ++t)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int64_t tt = tg * TP + t;
            const int c = c0 + v;
            if (tt >= K) continue;
            if (c < wc2) a.dzc[(j * K + tt) * wc2 + c] = acc[o][t][v];
            else if (c < C) a.dzr[(j * K + tt) * a.wr + (c - wc2)] = acc[o][t][v];
          }
      }
    }
  }
}

int check_factored(const void* h, const void* zc, const void* zr, const void* angular, const void* transport, const void* rho,
                   const int32_t* desc, const int64_t* source, int64_t n_edges, int k, int wc, int wr, int n_f, int n_blocks, int d_out,
                   int n_scales, int dtype) {
  GM_REQUIRE(n_scales >= 0, GM_ERR_ARGUMENT, "gm_factored: negative n_scales");
  GM_REQUIRE(n_edges >= 0 && wc >= 0 && wr >= 0 && n_f >= 1 && n_blocks >= 0, GM_ERR_ARGUMENT, "gm_factored: bad sizes");
  GM_REQUIRE(k >= 1 && k <= FMAX_K, GM_ERR_ARGUMENT, "gm_factored: k exceeds MAX_K");
  GM_REQUIRE(d_out >= 1 && d_out <= 128, GM_ERR_ARGUMENT, "gm_factored: d_out must be in [1, MAX_OUT]");
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_F64, GM_ERR_UNSUPPORTED, "gm_factored: dtype must be float32 or float64");
  if (n_edges == 0) return GM_OK;
  GM_REQUIRE(h || k == 1, GM_ERR_ARGUMENT, "gm_factored: null h");
  GM_REQUIRE((zc || wc == 0) && (zr || wr == 0) && angular && transport && rho && desc && source, GM_ERR_ARGUMENT, "gm_factored: null pointer");
  return GM_OK;
}

}  // namespace
}  // namespace gmb

using namespace gmb;

extern "C" int gm_factored_forward(const void* h, const void* zc, const void* zr, const void* angular, const void* transport,
                                   const void* rho, const int32_t* desc, const int64_t* source, const int64_t* order,
                                   const int64_t* group_ptr, const int64_t* group_source, int64_t n_edges, int64_t n_groups, int k,
                                   int wc, int wr, int n_f, int n_blocks, int d_out, int dtype, void* out, void* stream) {
  return gm_factored_forward_scaled(h, zc, zr, angular, transport, rho, 0, desc, source, order, group_ptr, group_source, n_edges, n_groups, k,
                                    wc, wr, n_f, n_blocks, d_out, dtype, out, stream);
}

extern "C" int gm_factored_forward_scaled(const void* h, const void* zc, const void* zr, const void* angular, const void* transport,
                                          const void* rho, int n_scales, const int32_t* desc, const int64_t* source, const int64_t* order,
                                          const int64_t* group_ptr, const int64_t* group_source, int64_t n_edges, int64_t n_groups, int k,
                                          int wc, int wr, int n_f, int n_blocks, int d_out, int dtype, void* out, void* stream) {
  int status = check_factored(h, zc, zr, angular, transport, rho, desc, source, n_edges, k, wc, wr, n_f, n_blocks, d_out, n_scales, dtype);
  if (status != GM_OK || n_edges == 0) return status;
  GM_REQUIRE(order && group_ptr && group_source && out && n_groups >= 1, GM_ERR_ARGUMENT, "gm_factored_forward: null grouping / output");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    FArgs<T> a{};
    a.n_edges = n_edges; a.n_groups = n_groups; a.k = k; a.wc = wc; a.wr = wr; a.n_f = n_f; a.n_blocks = n_blocks; a.d_out = d_out; a.n_scales = n_scales;
    a.h = (const T*)h; a.zc = (const T*)zc; a.zr = (const T*)zr; a.angular = (const T*)angular; a.transport = (const T*)transport;
    a.rho = (const T*)rho; a.desc = desc; a.source = source; a.order = order; a.group_ptr = group_ptr; a.group_source = group_source;
    a.out = (T*)out;
    if constexpr (sizeof(T) == 4)
      if (tensor_cores_forward(a)) return forward_tc(a, (cudaStream_t)stream);
    const int C = 2 * wc + wr;
    const size_t extra = (size_t)(n_blocks * FDESC) * sizeof(int32_t) + (size_t)(n_blocks + d_out) * sizeof(int4);
    // 64 or 32 edges per tile; fewer where the packed width or the phase tables leave no room for them
    int tile = MAX_TILE;
    if (ForwardLayout<T>(k, C, n_f, n_scales, n_blocks, d_out, tile).total * sizeof(T) + extra > FSMEM_SIXTH) tile /= 2;
    while (tile > 8 && ForwardLayout<T>(k, C, n_f, n_scales, n_blocks, d_out, tile).total * sizeof(T) + extra > 200 * 1024) tile /= 2;
    size_t smem = ForwardLayout<T>(k, C, n_f, n_scales, n_blocks, d_out, tile).total * sizeof(T) + extra;
    // the CTAs stride the sources, so that the column list is built once for several; with the smaller tiles more of them pay
    // (16 per SM 1 149 us, 64 1 034; with 64 edges 1 309 and 1 330)
    const int64_t cap = (int64_t)sm_count() * (tile < MAX_TILE ? 64 : 16);
    const unsigned blocks = (unsigned)(n_groups < cap ? n_groups : cap);
    auto go = [&](auto kernel, int x) {
      const int st = allow_smem(kernel, smem, "gm_factored_forward");
      if (st == GM_OK) kernel<<<blocks, FTHREADS, smem, (cudaStream_t)stream>>>(a, x);
      return st == GM_OK ? launch_status("gm_factored_forward") : st;
    };
    if (smem > FSMEM_MOST) {
      const int pitch = d_out | 1;  // odd: no bank conflicts between the threads' rows
      smem = ((size_t)k * 2 * wc + ((size_t)k * wr + 3) / 4 * 4 + (size_t)FTHREADS * pitch) * sizeof(T);
      return n_scales ? go(factored_forward_wide_kernel<T, true>, pitch) : go(factored_forward_wide_kernel<T, false>, pitch);
    }
    return n_scales ? go(factored_forward_kernel<T, true>, tile) : go(factored_forward_kernel<T, false>, tile);
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}

extern "C" int gm_factored_aggregate(const void* rows, const void* weights, const int64_t* row_ptr, int64_t n_targets, int64_t n_edges,
                                     int d_out, int dtype, void* out, void* stream) {
  GM_REQUIRE(n_targets >= 0 && n_edges >= 0 && d_out >= 1 && d_out <= 128, GM_ERR_ARGUMENT, "gm_factored_aggregate: bad sizes");
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_F64, GM_ERR_UNSUPPORTED, "gm_factored_aggregate: dtype must be float32 or float64");
  if (n_targets == 0) return GM_OK;
  GM_REQUIRE(row_ptr && out && (n_edges == 0 || (rows && weights)), GM_ERR_ARGUMENT, "gm_factored_aggregate: null pointer");
  const unsigned blocks = (unsigned)((n_targets + 7) / 8);
  auto run = [&](auto tag) {
    using T = decltype(tag);
    constexpr int V = 16 / sizeof(T);
    auto go = [&](auto kernel) { kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>((const T*)rows, (const T*)weights, row_ptr, n_targets, d_out, (T*)out); };
    const bool vectors = d_out % V == 0 && ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    // us by columns / by vectors, 40 000 targets: of 8 edges, 20 columns 9 / 14 (float64 12 / 14), 64 columns 20 / 16; of 16 edges, 20 columns 13 / 16
    // (float64 35 / 30), 33 columns 22 / 30, 40 columns 29 / 26; of 24, 20 columns 19 / 17, 33 columns 37 / 40.  4 000 targets are too few to
    // tell (3 us), and of those of 8 x 16 edges the longest take 7 / 4.
    const bool few = n_targets > 12288 && n_edges < 24 * n_targets &&
                     ((int64_t)sizeof(T) * n_edges * d_out < 1600 * n_targets || (!vectors && d_out > 32));
    if (few) go(aggregate_columns_kernel<T>);
    else if (!vectors) go(aggregate_kernel<T, 1, true>);
    else if (d_out <= 2 * V) go(aggregate_kernel<T, V, true>);
    else go(aggregate_kernel<T, V, false>);
  };
  if (dtype == GM_F32) run(float());
  else run(double());
  return launch_status("gm_factored_aggregate");
}

extern "C" int gm_factored_backward(const void* g, const int64_t* target, const void* weights, const void* rows, const void* h,
                                    const void* zc, const void* zr, const void* angular, const void* transport, const void* rho,
                                    const int32_t* desc, const int64_t* source, const int64_t* order, const int64_t* group_ptr,
                                    const int64_t* group_source, int64_t n_edges, int64_t n_groups, int k, int wc, int wr, int n_f,
                                    int n_blocks, int d_out, int dtype, void* dh, void* dzc, void* dzr, void* dweights, void* stream) {
  return gm_factored_backward_scaled(g, target, weights, rows, h, zc, zr, angular, transport, rho, 0, desc, source, order, group_ptr, group_source,
                                     n_edges, n_groups, k, wc, wr, n_f, n_blocks, d_out, dtype, dh, dzc, dzr, dweights, stream);
}

extern "C" int gm_factored_backward_scaled(const void* g, const int64_t* target, const void* weights, const void* rows, const void* h,
                                           const void* zc, const void* zr, const void* angular, const void* transport, const void* rho, int n_scales,
                                           const int32_t* desc, const int64_t* source, const int64_t* order, const int64_t* group_ptr,
                                           const int64_t* group_source, int64_t n_edges, int64_t n_groups, int k, int wc, int wr, int n_f,
                                           int n_blocks, int d_out, int dtype, void* dh, void* dzc, void* dzr, void* dweights, void* stream) {
  int status = check_factored(h, zc, zr, angular, transport, rho, desc, source, n_edges, k, wc, wr, n_f, n_blocks, d_out, n_scales, dtype);
  if (status != GM_OK || n_edges == 0) return status;
  GM_REQUIRE(g && order && group_ptr && group_source && n_groups >= 1, GM_ERR_ARGUMENT, "gm_factored_backward: null pointer");
  GM_REQUIRE((dh || k == 1) && (dzc || wc == 0) && (dzr || wr == 0), GM_ERR_ARGUMENT, "gm_factored_backward: null output");
  const bool aggregated = target != nullptr;
  GM_REQUIRE(!aggregated || (weights && rows && dweights), GM_ERR_ARGUMENT, "gm_factored_backward: the aggregated form needs weights, rows and dweights");
  const int C = 2 * wc + wr;
  GM_REQUIRE(k * ((C + 3) / 4 * 4) <= MAX_OWNED * FTHREADS, GM_ERR_LIMIT, "gm_factored_backward: k * (2 wc + wr) = %d exceeds %d", k * C, MAX_OWNED * FTHREADS);
  auto run = [&](auto tag) {
    using T = decltype(tag);
    FArgs<T> a{};
    a.n_edges = n_edges; a.n_groups = n_groups; a.k = k; a.wc = wc; a.wr = wr; a.n_f = n_f; a.n_blocks = n_blocks; a.d_out = d_out; a.n_scales = n_scales;
    a.h = (const T*)h; a.zc = (const T*)zc; a.zr = (const T*)zr; a.angular = (const T*)angular; a.transport = (const T*)transport;
    a.rho = (const T*)rho; a.desc = desc; a.source = source; a.order = order; a.group_ptr = group_ptr; a.group_source = group_source;
    a.g = (const T*)g; a.target = target; a.weights = aggregated ? (const T*)weights : nullptr; a.rows = aggregated ? (const T*)rows : nullptr;
    a.dh = (T*)dh; a.dzc = (T*)dzc; a.dzr = (T*)dzr; a.dweights = aggregated ? (T*)dweights : nullptr;
    if constexpr (sizeof(T) == 4)
      if (tensor_cores_backward(a)) return backward_tc(a, (cudaStream_t)stream);
    // 64 or 32 edges per tile; fewer where the packed width is so large that they do not fit shared memory
    int tile = MAX_TILE;
    auto layout = [&](bool staged) { return BackwardLayout<T>(k, C, n_f, n_scales, d_out, tile, staged); };
    if (layout(true).total * sizeof(T) > FSMEM_SIXTH) tile /= 2;
    while (tile > 8 && layout(true).total * sizeof(T) > 200 * 1024) tile /= 2;
    const bool staged = layout(true).total * sizeof(T) <= FSMEM_MOST;
    const BackwardLayout<T> L = layout(staged);
    const size_t smem = (size_t)L.total * sizeof(T);
    const unsigned blocks = (unsigned)(n_groups < (1 << 20) ? n_groups : (1 << 20));
    auto go = [&](auto kernel) {
      int st = allow_smem(kernel, smem, "gm_factored_backward");
      if (st != GM_OK) return st;
      kernel<<<blocks, FTHREADS, smem, (cudaStream_t)stream>>>(a, C, tile);
      return launch_status("gm_factored_backward");
    };
    const bool one = L.tgroups * ((C + 3) / 4) <= FTHREADS;
    auto form = [&](auto scaled) {
      constexpr bool SC = decltype(scaled)::value;
      if (staged) return one ? go(factored_backward_kernel<T, 1, true, SC>) : go(factored_backward_kernel<T, 2, true, SC>);
      return one ? go(factored_backward_kernel<T, 1, false, SC>) : go(factored_backward_kernel<T, 2, false, SC>);
    };
    return n_scales ? form(std::true_type{}) : form(std::false_type{});
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}
