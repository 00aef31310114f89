// Node-side products of a steerable kernel's readout with a node field, Z(j): per block (n -> m, role) and trunk column t
//
//   Z_{t,b}(j) = sum_a M_t[b, a] x~_n(j)[a],     M_0 = the readout's bias, M_t = its weight column t - 1,
//
// x~ = x (real for n = 0), or conj(x) for antilinear blocks and for n -> 0.  Phases are per edge and commute with the sum
// over a, so M(e) (pre(e) u~(e)) of the pair terms (pairs_ops.cu; reference src/gm_attention/nn/fused/pairs.h:201-365) is
// phase * sum_t h~_t(e) Z_t(source(e)), the form factored_ops.cu evaluates: an edge then costs trunk * b multiply-adds per
// block instead of trunk * a * b, and the readout's gradient is a sum over nodes instead of edges.
//
// What bounds it: instruction issue (eight multiply-adds, a pair of shared-memory words and some addressing per block entry and
// node; the fields pass once).  In the forward and in the readout's gradient a thread owns an entry (t, b) of all blocks' columns,
// holds its A_HELD copies' coefficients (or sums) in registers and walks the nodes: Z and dZ then move in whole rows, and x~ is
// the same for a block's threads.  In the gradient of x lanes are nodes, warps share a block's entries, and coefficients are
// broadcast.  The readout's gradient, a sum over all nodes, is cut into chunks of nodes whose partial sums the caller adds: no
// atomics.
//
// Against an entry's thread that read every coefficient and word of Z for 8 nodes at a time, float32, trunk 16, us forward, dx,
// readout's gradient:                        8 192 nodes                           30 000 nodes
//   {8, 8, 8} -> {4, 4, 4}     92, 201, 213 -> 55, 61, 65        298, 682, 920 -> 165, 191, 153
//   {16, 16} -> {8, 8}         81, 188, 352 -> 71, 82, 83
//   {2, 2} -> {8, 8}           36,  72,  72 -> 28, 41, 41        160, 241, 227 ->  91, 123,  92
// 1 000 nodes of the first: 47, 126, 69 -> 17, 46, 47.  Of this the loads under way made dx 96 -> 60 (all of a chunk before its
// first store) and the readout's gradient 92 -> 65 (four nodes'; eight the same), one wave of CTAs the forward 68 -> 55; three CTAs
// of dx to an SM instead of two matter on 30 000 nodes (232 -> 191).  64 threads to a CTA: 57, 60, 72.
#include <algorithm>

#include "common.cuh"

namespace gmb {
namespace {

constexpr int NDESC = 8;
enum { X_REAL = 0, X_COMPLEX = 1, X_CONJ = 2 };

template <typename T>
struct NArgs {
  int64_t n_nodes;
  int n_blocks, din, k, wc, wr, crows, rrows, chunk, staged;  // nodes a CTA walks, and of these at a time in shared memory
  const T *x, *cw, *cb, *rw, *rb;
  const int32_t* desc;  // (n_blocks, 8): complex block, Z column, b, a, x offset, x mode, first readout row, -
  T *zc, *zr;
  bool pairs;           // zc, dzc start on a boundary of two elements
  const T *dzc, *dzr;
  T *dx, *dcw, *drw;    // dcw (chunks, crows, k), drw (chunks, rrows, k): bias gradient in column 0
};

template <typename T> struct alignas(2 * sizeof(T)) Pair { T r, i; };
// Complex element at of a field; pairs: the field starts on a boundary of two elements
template <typename T>
__device__ __forceinline__ Pair<T> load_pair(const T* p, int64_t at, bool pairs) {
  return pairs ? reinterpret_cast<const Pair<T>*>(p)[at] : Pair<T>{p[2 * at], p[2 * at + 1]};
}
template <typename T>
__device__ __forceinline__ void store_pair(T* p, int64_t at, bool pairs, T r, T i) {
  if (pairs) reinterpret_cast<Pair<T>*>(p)[at] = Pair<T>{r, i};
  else p[2 * at] = r, p[2 * at + 1] = i;
}

// readout entry of row r, column t (0: bias)
template <typename T>
__device__ __forceinline__ T coefficient(const T* w, const T* bias, int r, int t, int k) {
  return t == 0 ? (bias ? bias[r] : T(0)) : w[(int64_t)r * (k - 1) + t - 1];
}

constexpr int ENTRY_THREADS = 128, A_HELD = 16, A_SUMMED = 8, FLIGHT = 4;  // copies a thread holds coefficients, sums of; nodes whose dZ is under way

// A thread's entry: column c of trunk column t, complex entries first, then the real ones from a CTA of their own on.
struct Entry {
  bool is_complex, present;
  int t, c, b, am, xoff, mode, row0;
  __device__ Entry(const int32_t* desc, int n_blocks, int k, int wc, int wr) {
    const int tiles_c = (k * wc + ENTRY_THREADS - 1) / ENTRY_THREADS;
    is_complex = (int)blockIdx.y < tiles_c;
    const int width = is_complex ? wc : wr, i = ((int)blockIdx.y - (is_complex ? 0 : tiles_c)) * ENTRY_THREADS + (int)threadIdx.x;
    t = i / width;
    c = i - t * width;
    present = false;
    b = am = xoff = mode = row0 = 0;
    for (int x = 0; x < n_blocks && t < k; ++x) {  // (a column may belong to no block)
      const int32_t* d = desc + x * NDESC;
      if ((d[0] != 0) == is_complex && c >= d[1] && c < d[1] + d[2]) {
        present = true;
        b = c - d[1]; am = d[3]; xoff = d[4]; mode = d[5]; row0 = d[6];
      }
    }
  }
  __device__ int row(int a) const { return row0 + (is_complex ? 2 : 1) * (b * am + a); }
};
inline unsigned entry_tiles(int k, int wc, int wr) {
  return (unsigned)((k * wc + ENTRY_THREADS - 1) / ENTRY_THREADS + (k * wr + ENTRY_THREADS - 1) / ENTRY_THREADS);
}

// f(a, x[a]) of the held copies a < n of one node's row of pairs
template <int HELD, typename T, typename F>
__device__ __forceinline__ void for_copies(const Pair<T>* x, const Entry& en, int n, F f) {
  const bool real = en.mode == X_REAL;
  const int stride = real ? 1 : 2;
#pragma unroll
  for (int g = 0; g < HELD; g += 4) {
    if (g + 4 <= n) {
#pragma unroll
      for (int a = g; a < g + 4; ++a) {
        const Pair<T> v = x[0];
        f(a, v.r, real ? T(0) : v.i);
        x += stride;
      }
    } else if (g < n) {
#pragma unroll
      for (int a = g; a < g + 3; ++a)
        if (a < n) {
          const Pair<T> v = x[0];
          f(a, v.r, real ? T(0) : v.i);
          x += stride;
        }
    }
  }
}

// The CTA's nodes j0 .. j1, p.staged at a time in shared memory as pairs of neighbouring columns, so that every complex number is
// one word wherever it starts: f(first node, their rows, how many)
template <typename T, typename F>
__device__ __forceinline__ void for_nodes(const NArgs<T>& p, Pair<T>* x_s, F f) {
  const int64_t j0 = (int64_t)blockIdx.x * p.chunk, j1 = min(j0 + p.chunk, p.n_nodes);
  for (int64_t s0 = j0; s0 < j1; s0 += p.staged) {
    const int n = (int)min((int64_t)p.staged, j1 - s0), count = n * p.din;
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += ENTRY_THREADS) {
      const T* x = p.x + s0 * p.din + i;
      x_s[i] = Pair<T>{x[0], i + 1 < count ? x[1] : T(0)};
    }
    __syncthreads();
    f(s0, x_s, n);
  }
}

template <typename T>
__global__ void __launch_bounds__(ENTRY_THREADS) node_products_forward_kernel(const __grid_constant__ NArgs<T> p) {
  extern __shared__ __align__(16) unsigned char raw[];
  Pair<T>* x_s = reinterpret_cast<Pair<T>*>(raw);  // (staged, din)
  const Entry en(p.desc, p.n_blocks, p.k, p.wc, p.wr);
  const T sign = en.mode == X_CONJ ? T(-1) : T(1);  // M conj(x) = conj(conj(M) x)
  for (int a0 = 0; __syncthreads_or(en.present && (a0 == 0 || a0 < en.am)); a0 += A_HELD) {
    const int n = en.present ? min(en.am - a0, A_HELD) : 0;
    T mr[A_HELD], mi[A_HELD];
#pragma unroll
    for (int a = 0; a < A_HELD; ++a) {
      mr[a] = mi[a] = T(0);
      if (a < n) {
        const int row = en.row(a0 + a);
        mr[a] = en.is_complex ? coefficient(p.cw, p.cb, row, en.t, p.k) : coefficient(p.rw, p.rb, row, en.t, p.k);
        if (en.is_complex) mi[a] = sign * coefficient(p.cw, p.cb, row + 1, en.t, p.k);
      }
    }
    const bool first = a0 == 0, writes = en.present && (first || n > 0);
    const int64_t step = (int64_t)p.k * (en.is_complex ? p.wc : p.wr);
    for_nodes(p, x_s, [&](int64_t j, const Pair<T>* x, int nodes) {
      int64_t at = j * step + (int64_t)en.t * (en.is_complex ? p.wc : p.wr) + en.c;
      x += en.xoff + a0 * (en.mode == X_REAL ? 1 : 2);
      for (int v = 0; v < nodes; ++v, at += step, x += p.din) {
        T zr = T(0), zi = T(0);
        if (writes && !first) {  // more copies than a thread holds
          const Pair<T> z = en.is_complex ? load_pair(p.zc, at, p.pairs) : Pair<T>{p.zr[at], T(0)};
          zr = z.r;
          zi = sign * z.i;
        }
        for_copies<A_HELD>(x, en, n, [&](int a, T xr, T xi) {
          zr += mr[a] * xr;
          zr -= mi[a] * xi;
          zi += mr[a] * xi;
          zi += mi[a] * xr;
        });
        if (!writes) continue;
        if (en.is_complex) store_pair(p.zc, at, p.pairs, zr, sign * zi);
        else p.zr[at] = zr;
      }
    });
  }
}

// dM_t[b, a] over one chunk of nodes: dZ conj(x~), the nodes in order
template <typename T>
__global__ void __launch_bounds__(ENTRY_THREADS) node_products_dw_kernel(const __grid_constant__ NArgs<T> p) {
  extern __shared__ __align__(16) unsigned char raw[];
  Pair<T>* x_s = reinterpret_cast<Pair<T>*>(raw);  // (staged, din)
  const Entry en(p.desc, p.n_blocks, p.k, p.wc, p.wr);
  const T sign = en.mode == X_CONJ ? T(-1) : T(1);  // M conj(x) = conj(conj(M) x)
  for (int a0 = (int)blockIdx.z * A_SUMMED; __syncthreads_or(en.present && a0 < en.am); a0 += (int)gridDim.z * A_SUMMED) {
    const int n = en.present ? max(min(en.am - a0, A_SUMMED), 0) : 0;
    T gr[A_SUMMED], gi[A_SUMMED];
#pragma unroll
    for (int a = 0; a < A_SUMMED; ++a) gr[a] = gi[a] = T(0);
    const int64_t step = (int64_t)p.k * (en.is_complex ? p.wc : p.wr);
    for_nodes(p, x_s, [&](int64_t j, const Pair<T>* x, int nodes) {
      int64_t at = j * step + (int64_t)en.t * (en.is_complex ? p.wc : p.wr) + en.c;
      x += en.xoff + a0 * (en.mode == X_REAL ? 1 : 2);
      for (int v = 0; v < nodes; v += FLIGHT) {
        Pair<T> z[FLIGHT];
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u, at += step) {
          z[u] = Pair<T>{T(0), T(0)};
          if (n > 0 && v + u < nodes) {
            if (en.is_complex) z[u] = load_pair(p.dzc, at, p.pairs);
            else z[u].r = p.dzr[at];
          }
        }
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u, x += p.din) {
          if (v + u >= nodes) continue;
          const T zr = z[u].r, zi = sign * z[u].i;
          for_copies<A_SUMMED>(x, en, n, [&](int a, T xr, T xi) {
            gr[a] += zr * xr;
            gr[a] += zi * xi;
            gi[a] += zi * xr;
            gi[a] -= zr * xi;
          });
        }
      }
    });
#pragma unroll
    for (int a = 0; a < A_SUMMED; ++a) {
      if (a >= n) continue;
      const int row = en.row(a0 + a);
      if (en.is_complex) {
        T* out = p.dcw + ((int64_t)blockIdx.x * p.crows + row) * p.k + en.t;
        out[0] = gr[a];
        out[p.k] = sign * gi[a];
      } else {
        p.drw[((int64_t)blockIdx.x * p.rrows + row) * p.k + en.t] = gr[a];
      }
    }
  }
}

// dx(j)[a] = sum over blocks, b, t of conj(M) dZ (conjugated back for conj operands).  A CTA's lanes are DX_NODES nodes.  Blocks
// that read the same copies and follow one another in Z's columns are taken together, up to DX_ENTRIES columns: their entries
// (t, column) are staged with DX_COPIES copies' coefficients, as many t at a time as fit, the warps share them, and the warps' sums
// meet in shared memory.
constexpr int DX_THREADS = 256, DX_WARPS = DX_THREADS / 32, DX_NODES = 32, DX_COPIES = 8, DX_ENTRIES = 128, DX_PITCH = DX_NODES + 1;
template <typename T> constexpr size_t dx_smem() { return sizeof(Pair<T>) * DX_ENTRIES * (DX_PITCH + DX_COPIES); }

template <typename T>
__global__ void __launch_bounds__(DX_THREADS, sizeof(T) == 4 ? 3 : 1) node_products_dx_kernel(const __grid_constant__ NArgs<T> p) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int row_s[DX_ENTRIES];                    // first readout row of a column's copies
  __shared__ T sign_s[DX_ENTRIES];                     // -1: conj operand
  Pair<T>* m_s = reinterpret_cast<Pair<T>*>(raw);      // (entry, copy)
  Pair<T>* z_s = m_s + DX_ENTRIES * DX_COPIES;         // (entry, node)
  T* sum_s = reinterpret_cast<T*>(z_s);                // (warp, copy and part, node), when the entries are done with
  static_assert(2 * DX_ENTRIES >= DX_WARPS * 2 * DX_COPIES, "the warps' sums fit where the entries were");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t j0 = (int64_t)blockIdx.x * DX_NODES;
  const int nodes = (int)min((int64_t)DX_NODES, p.n_nodes - j0);
  for (int i = threadIdx.x; i < nodes * p.din; i += DX_THREADS) p.dx[j0 * p.din + i] = T(0);
  for (int blk = 0, b0 = 0; blk < p.n_blocks;) {
    const int32_t* first = p.desc + blk * NDESC;
    const bool is_complex = first[0] != 0, real = first[5] == X_REAL;
    const int c0 = first[1] + b0, am = first[3], xoff = first[4], step = is_complex ? 2 : 1;
    int width = 0;
    __syncthreads();
    while (blk < p.n_blocks && width < DX_ENTRIES) {
      const int32_t* d = p.desc + blk * NDESC;
      if ((d[0] != 0) != is_complex || (d[5] == X_REAL) != real || d[3] != am || d[4] != xoff || d[1] + b0 != c0 + width) break;
      const int take = min(d[2] - b0, DX_ENTRIES - width);
      for (int i = threadIdx.x; i < take; i += DX_THREADS) {
        row_s[width + i] = d[6] + step * (b0 + i) * am;
        sign_s[width + i] = d[5] == X_CONJ ? T(-1) : T(1);
      }
      width += take;
      b0 += take;
      if (b0 == d[2]) ++blk, b0 = 0;
    }
    if (width == 0) continue;  // (a block of no columns)
    const int rounds = (p.k + DX_ENTRIES / width - 1) / (DX_ENTRIES / width), trunk = (p.k + rounds - 1) / rounds;  // equal chunks of t
    for (int a0 = 0; a0 < am; a0 += DX_COPIES) {
      T gr[DX_COPIES], gi[DX_COPIES];
#pragma unroll
      for (int a = 0; a < DX_COPIES; ++a) gr[a] = gi[a] = T(0);
      for (int t0 = 0; t0 < p.k; t0 += trunk) {
        const int nt = min(trunk, p.k - t0), n = nt * width;
        __syncthreads();
        // every load of the chunk is under way before the first word is stored
        constexpr int M_EACH = DX_ENTRIES * DX_COPIES / DX_THREADS, Z_EACH = DX_ENTRIES / 32, V_EACH = DX_NODES / DX_WARPS;
        Pair<T> m[M_EACH], z[Z_EACH][V_EACH];
        int m_at[M_EACH];
#pragma unroll
        for (int q = 0; q < M_EACH; ++q) {  // (t fastest: the readout's rows are contiguous in it)
          const int i = (int)threadIdx.x + q * DX_THREADS, a = i / n, e = i - a * n, c = e / nt, t = e - c * nt;
          m[q] = Pair<T>{T(0), T(0)};
          m_at[q] = a < DX_COPIES ? (t * width + c) * DX_COPIES + a : -1;
          if (a < DX_COPIES && a0 + a < am) {
            const int row = row_s[c] + step * (a0 + a);
            m[q].r = is_complex ? coefficient(p.cw, p.cb, row, t0 + t, p.k) : coefficient(p.rw, p.rb, row, t0 + t, p.k);
            if (is_complex) m[q].i = sign_s[c] * coefficient(p.cw, p.cb, row + 1, t0 + t, p.k);
          }
        }
#pragma unroll
        for (int q = 0; q < Z_EACH; ++q) {
          const int i = lane + 32 * q, t = i / width, c = i - t * width;
          int64_t at = ((j0 + warp) * p.k + t0 + t) * (is_complex ? p.wc : p.wr) + c0 + c;
#pragma unroll
          for (int u = 0; u < V_EACH; ++u, at += (int64_t)DX_WARPS * p.k * (is_complex ? p.wc : p.wr)) {
            z[q][u] = Pair<T>{T(0), T(0)};
            if (i < n && warp + u * DX_WARPS < nodes) {
              if (is_complex) z[q][u] = load_pair(p.dzc, at, p.pairs);
              else z[q][u].r = p.dzr[at];
            }
          }
        }
#pragma unroll
        for (int q = 0; q < M_EACH; ++q)
          if (m_at[q] >= 0) m_s[m_at[q]] = m[q];
#pragma unroll
        for (int q = 0; q < Z_EACH; ++q) {
          const int i = lane + 32 * q;
          if (i >= n) continue;
          const T sign = sign_s[i % width];  // conj(M) dZ conjugated back: M and dZ conjugated
#pragma unroll
          for (int u = 0; u < V_EACH; ++u) z_s[i * DX_PITCH + warp + u * DX_WARPS] = Pair<T>{z[q][u].r, sign * z[q][u].i};
        }
        __syncthreads();
#pragma unroll 2
        for (int i = warp; i < n; i += DX_WARPS) {
          const Pair<T> z = z_s[i * DX_PITCH + lane];
#pragma unroll
          for (int a = 0; a < DX_COPIES; ++a) {
            const Pair<T> m = m_s[i * DX_COPIES + a];
            gr[a] += m.r * z.r;
            gr[a] += m.i * z.i;
            gi[a] += m.r * z.i;
            gi[a] -= m.i * z.r;
          }
        }
      }
      __syncthreads();
#pragma unroll
      for (int a = 0; a < DX_COPIES; ++a) {
        sum_s[((warp * DX_COPIES + a) * 2) * DX_PITCH + lane] = gr[a];
        sum_s[((warp * DX_COPIES + a) * 2 + 1) * DX_PITCH + lane] = gi[a];
      }
      __syncthreads();
      const int parts = real ? 1 : 2;
      for (int i = threadIdx.x; i < DX_NODES * 2 * DX_COPIES; i += DX_THREADS) {
        const int q = i % (2 * DX_COPIES), v = i / (2 * DX_COPIES), a = q >> 1, part = q & 1;
        if (v >= nodes || a0 + a >= am || part >= parts) continue;
        T sum = T(0);
#pragma unroll
        for (int w = 0; w < DX_WARPS; ++w) sum += sum_s[((w * DX_COPIES + a) * 2 + part) * DX_PITCH + v];
        p.dx[(j0 + v) * p.din + xoff + parts * (a0 + a) + part] += sum;
      }
    }
  }
}

template <typename T>
NArgs<T> node_args(const void* x, const void* cw, const void* cb, const void* rw, const void* rb, const int32_t* desc, int64_t n_nodes, int n_blocks,
                   int din, int k, int wc, int wr) {
  NArgs<T> p{};
  p.x = (const T*)x; p.cw = (const T*)cw; p.cb = (const T*)cb; p.rw = (const T*)rw; p.rb = (const T*)rb; p.desc = desc;
  p.n_nodes = n_nodes; p.n_blocks = n_blocks; p.din = din; p.k = k; p.wc = wc; p.wr = wr;
  return p;
}

// p.staged: the chunk's nodes whose rows fit in 20 KB (eight CTAs to an SM), one at least.  Their bytes.
template <typename T>
size_t stage_nodes(NArgs<T>& p) {
  const size_t row = (size_t)p.din * sizeof(Pair<T>);
  p.staged = (int)std::max<size_t>(std::min<size_t>(20 * 1024 / row, (size_t)p.chunk), 1);
  return p.staged * row;
}

int check_nodes(const char* what, const void* x, const void* cw, const void* rw, const int32_t* desc, int64_t n_nodes, int n_blocks, int din, int k,
                int wc, int wr, int dtype) {
  GM_REQUIRE(n_nodes >= 0 && n_blocks >= 0 && n_blocks <= 65535 && din >= 1 && din <= 2048 && k >= 2 && wc >= 0 && wr >= 0, GM_ERR_ARGUMENT,
             "%s: bad sizes", what);
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_F64, GM_ERR_UNSUPPORTED, "%s: dtype must be float32 or float64", what);
  GM_REQUIRE(n_nodes == 0 || n_blocks == 0 || (x && desc && (cw || wc == 0) && (rw || wr == 0)), GM_ERR_ARGUMENT, "%s: null pointer", what);
  GM_REQUIRE(n_nodes / 8 < ((int64_t)1 << 31) - 1, GM_ERR_LIMIT, "%s: too many nodes", what);
  return GM_OK;
}

}  // namespace
}  // namespace gmb

using namespace gmb;

extern "C" int gm_node_products_forward(const void* x, const void* cw, const void* cb, const void* rw, const void* rb, const int32_t* desc,
                                        int64_t n_nodes, int n_blocks, int din, int k, int wc, int wr, int dtype, void* zc, void* zr, void* stream) {
  const int status = check_nodes("gm_node_products_forward", x, cw, rw, desc, n_nodes, n_blocks, din, k, wc, wr, dtype);
  if (status != GM_OK || n_nodes == 0 || n_blocks == 0) return status;
  GM_REQUIRE((zc || wc == 0) && (zr || wr == 0), GM_ERR_ARGUMENT, "gm_node_products_forward: null output");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    NArgs<T> p = node_args<T>(x, cw, cb, rw, rb, desc, n_nodes, n_blocks, din, k, wc, wr);
    p.zc = (T*)zc; p.zr = (T*)zr;
    p.pairs = reinterpret_cast<uintptr_t>(zc) % (2 * sizeof(T)) == 0;
    // as many nodes to a CTA as make one wave of six CTAs per SM, 16 at least: the coefficients are read once per CTA
    const unsigned tiles = entry_tiles(k, wc, wr);
    if (tiles == 0) return (int)GM_OK;
    const int64_t resident = 6 * sm_count();
    p.chunk = (int)std::clamp<int64_t>((n_nodes * tiles + resident - 1) / resident, 16, 1 << 20);
    const size_t smem = stage_nodes(p);
    const int st = allow_smem(node_products_forward_kernel<T>, smem, "gm_node_products_forward");
    if (st != GM_OK) return st;
    const dim3 grid((unsigned)((n_nodes + p.chunk - 1) / p.chunk), tiles);
    node_products_forward_kernel<T><<<grid, ENTRY_THREADS, smem, (cudaStream_t)stream>>>(p);
    return launch_status("gm_node_products_forward");
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}

extern "C" int gm_node_products_backward(const void* x, const void* cw, const void* cb, const void* rw, const void* rb, const int32_t* desc,
                                         const void* dzc, const void* dzr, int64_t n_nodes, int n_blocks, int din, int k, int wc, int wr, int crows,
                                         int rrows, int chunk, int dtype, void* dx, void* dcw, void* drw, void* stream) {
  const int status = check_nodes("gm_node_products_backward", x, cw, rw, desc, n_nodes, n_blocks, din, k, wc, wr, dtype);
  if (status != GM_OK || n_nodes == 0 || n_blocks == 0) return status;
  GM_REQUIRE((dzc || wc == 0) && (dzr || wr == 0) && dx && (dcw || wc == 0) && (drw || wr == 0) && chunk >= 1, GM_ERR_ARGUMENT,
             "gm_node_products_backward: null pointer");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    NArgs<T> p = node_args<T>(x, cw, cb, rw, rb, desc, n_nodes, n_blocks, din, k, wc, wr);
    p.dzc = (const T*)dzc; p.dzr = (const T*)dzr; p.dx = (T*)dx; p.dcw = (T*)dcw; p.drw = (T*)drw;
    p.pairs = reinterpret_cast<uintptr_t>(dzc) % (2 * sizeof(T)) == 0;
    p.crows = crows; p.rrows = rrows; p.chunk = chunk;
    int st = allow_smem(node_products_dx_kernel<T>, dx_smem<T>(), "gm_node_products_backward");
    if (st != GM_OK) return st;
    node_products_dx_kernel<T><<<(unsigned)((n_nodes + DX_NODES - 1) / DX_NODES), DX_THREADS, dx_smem<T>(), (cudaStream_t)stream>>>(p);
    st = launch_status("gm_node_products_backward");
    if (st != GM_OK) return st;
    if (entry_tiles(k, wc, wr) == 0) return (int)GM_OK;
    const size_t smem = stage_nodes(p);
    st = allow_smem(node_products_dw_kernel<T>, smem, "gm_node_products_backward");
    if (st != GM_OK) return st;
    // CTAs in z share an entry's copies, of which a row's width tells the most there can be
    const dim3 grid((unsigned)((n_nodes + chunk - 1) / chunk), entry_tiles(k, wc, wr), (unsigned)std::clamp((din + A_SUMMED - 1) / A_SUMMED, 1, 4));
    node_products_dw_kernel<T><<<grid, ENTRY_THREADS, smem, (cudaStream_t)stream>>>(p);
    return launch_status("gm_node_products_backward");
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}
