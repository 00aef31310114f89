// Node-side products of a steerable kernel's readout with a node field, Z(j): per block (n -> m, role) and trunk column t
//
//   Z_{t,b}(j) = sum_a M_t[b, a] x~_n(j)[a],     M_0 = the readout's bias, M_t = its weight column t - 1,
//
// x~ = x (real for n = 0), or conj(x) for antilinear blocks and for n -> 0.  Phases are per edge and commute with the sum
// over a, so M(e) (pre(e) u~(e)) of the pair terms (pairs_ops.cu; reference src/gm_attention/nn/fused/pairs.h:201-365) is
// phase * sum_t h~_t(e) Z_t(source(e)), the form factored_ops.cu evaluates: an edge then costs trunk * b multiply-adds per
// block instead of trunk * a * b, and the readout's gradient is a sum over nodes instead of edges.
//
// The work is small (nodes * trunk * a * b per block); what matters is that weights are read once per NODES nodes and that
// the readout's gradient, a sum over all nodes, is cut into chunks of nodes whose partial sums the caller adds: no atomics.
//
// NODES = 4 / 8 / 16, us forward, then backward (dx, the readout's gradient and the sum of its parts), float32:
//   {8, 8, 8} -> {4, 4, 4}, trunk 16    8 192 nodes 127 / 87 / 137, 428 / 396 / 498    30 000 nodes 300 / 288 / 434, 1 680 / 1 659 / 1 762
//   {16, 16} -> {8, 8}, trunk 16        8 192 nodes 134 / 85 / 154, 491 / 470 / 577    30 000 nodes 301 / 255 / 466, 2 025 / 1 997 / 2 181
//   {2, 2} -> {8, 8}, trunk 16          8 192 nodes  52 / 40 /  53, 145 / 141 / 176    30 000 nodes 135 / 162 / 199,   478 /   490 /   572
// On 1 000 nodes 4 wins (46 / 51, 166 / 219 for the first), where a pass of some 700 us waits for its launches; float64 leans
// to 4 on 30 000 nodes (409 / 459 / 698, 1 974 / 2 145 / 2 806 for the first) and to 8 on 8 192 (153 / 125 / 173, 584 / 581 / 764).
#include "common.cuh"

namespace gmb {
namespace {

constexpr int NODES = 8, NTHREADS = 128, NDESC = 8;
enum { X_REAL = 0, X_COMPLEX = 1, X_CONJ = 2 };

template <typename T>
struct NArgs {
  int64_t n_nodes;
  int n_blocks, din, k, wc, wr, crows, rrows, chunk;
  const T *x, *cw, *cb, *rw, *rb;
  const int32_t* desc;  // (n_blocks, 8): complex block, Z column, b, a, x offset, x mode, first readout row, -
  T *zc, *zr;
  const T *dzc, *dzr;
  T *dx, *dcw, *drw;    // dcw (chunks, crows, k), drw (chunks, rrows, k): bias gradient in column 0
};

// x~[a] of one node's row
template <typename T>
__device__ __forceinline__ void operand(const T* x, int xoff, int mode, int a, T& xr, T& xi) {
  if (mode == X_REAL) {
    xr = x[xoff + a];
    xi = T(0);
  } else {
    xr = x[xoff + 2 * a];
    xi = mode == X_CONJ ? -x[xoff + 2 * a + 1] : x[xoff + 2 * a + 1];
  }
}
// readout entry of row r, column t (0: bias)
template <typename T>
__device__ __forceinline__ T coefficient(const T* w, const T* bias, int r, int t, int k) {
  return t == 0 ? (bias ? bias[r] : T(0)) : w[(int64_t)r * (k - 1) + t - 1];
}

template <typename T>
__global__ void __launch_bounds__(NTHREADS) node_products_forward_kernel(NArgs<T> p) {
  extern __shared__ __align__(16) unsigned char raw[];
  T* x_s = reinterpret_cast<T*>(raw);  // (NODES, din)
  const int64_t j0 = (int64_t)blockIdx.x * NODES;
  const int n = (int)min((int64_t)NODES, p.n_nodes - j0);
  for (int i = threadIdx.x; i < NODES * p.din; i += NTHREADS) x_s[i] = i < n * p.din ? p.x[j0 * p.din + i] : T(0);
  __syncthreads();
  for (int blk = 0; blk < p.n_blocks; ++blk) {
    const int32_t* d = p.desc + blk * NDESC;
    const int zoff = d[1], bm = d[2], am = d[3], xoff = d[4], mode = d[5], row0 = d[6];
    for (int i = threadIdx.x; i < bm * p.k; i += NTHREADS) {
      const int b = i / p.k, t = i - b * p.k;
      T zr[NODES], zi[NODES];
#pragma unroll
      for (int v = 0; v < NODES; ++v) zr[v] = zi[v] = T(0);
      for (int a = 0; a < am; ++a) {
        const int idx = b * am + a;
        const T mr = d[0] ? coefficient(p.cw, p.cb, row0 + 2 * idx, t, p.k) : coefficient(p.rw, p.rb, row0 + idx, t, p.k);
        const T mi = d[0] ? coefficient(p.cw, p.cb, row0 + 2 * idx + 1, t, p.k) : T(0);
#pragma unroll
        for (int v = 0; v < NODES; ++v) {
          T xr, xi;
          operand(x_s + v * p.din, xoff, mode, a, xr, xi);
          zr[v] += mr * xr;
          zr[v] -= mi * xi;
          zi[v] += mr * xi;
          zi[v] += mi * xr;
        }
      }
#pragma unroll
      for (int v = 0; v < NODES; ++v) {
        if (v >= n) break;
        const int64_t at = (j0 + v) * p.k + t;
        if (d[0]) {
          p.zc[(at * p.wc + zoff + b) * 2] = zr[v];
          p.zc[(at * p.wc + zoff + b) * 2 + 1] = zi[v];
        } else {
          p.zr[at * p.wr + zoff + b] = zr[v];
        }
      }
    }
  }
}

// dx(j)[a] = sum over blocks, b, t of conj(M) dZ (conjugated back for conj operands): a warp owns the copies a = warp,
// warp + 4, ... of every block, its lanes the (b, t) pairs.
template <typename T>
__global__ void __launch_bounds__(NTHREADS) node_products_dx_kernel(NArgs<T> p) {
  extern __shared__ __align__(16) unsigned char raw[];
  T* dx_s = reinterpret_cast<T*>(raw);  // (NODES, din)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t j0 = (int64_t)blockIdx.x * NODES;
  const int n = (int)min((int64_t)NODES, p.n_nodes - j0);
  for (int i = threadIdx.x; i < NODES * p.din; i += NTHREADS) dx_s[i] = T(0);
  __syncthreads();
  for (int blk = 0; blk < p.n_blocks; ++blk) {
    const int32_t* d = p.desc + blk * NDESC;
    const int zoff = d[1], bm = d[2], am = d[3], xoff = d[4], mode = d[5], row0 = d[6];
    for (int a = warp; a < am; a += NTHREADS / 32) {
      T gr[NODES], gi[NODES];
#pragma unroll
      for (int v = 0; v < NODES; ++v) gr[v] = gi[v] = T(0);
      for (int i = lane; i < bm * p.k; i += 32) {
        const int t = i / bm, b = i - t * bm, idx = b * am + a;
        const T mr = d[0] ? coefficient(p.cw, p.cb, row0 + 2 * idx, t, p.k) : coefficient(p.rw, p.rb, row0 + idx, t, p.k);
        const T mi = d[0] ? coefficient(p.cw, p.cb, row0 + 2 * idx + 1, t, p.k) : T(0);
#pragma unroll
        for (int v = 0; v < NODES; ++v) {
          if (v >= n) break;
          const int64_t at = (j0 + v) * p.k + t;
          const T zr = d[0] ? p.dzc[(at * p.wc + zoff + b) * 2] : p.dzr[at * p.wr + zoff + b];
          const T zi = d[0] ? p.dzc[(at * p.wc + zoff + b) * 2 + 1] : T(0);
          gr[v] += mr * zr;  // conj(M) dZ
          gr[v] += mi * zi;
          gi[v] += mr * zi;
          gi[v] -= mi * zr;
        }
      }
#pragma unroll
      for (int v = 0; v < NODES; ++v) {
        const T sr = warp_sum(gr[v]), si = warp_sum(gi[v]);
        if (lane == 0) {
          if (mode == X_REAL) {
            dx_s[v * p.din + xoff + a] += sr;
          } else {
            dx_s[v * p.din + xoff + 2 * a] += sr;
            dx_s[v * p.din + xoff + 2 * a + 1] += mode == X_CONJ ? -si : si;
          }
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n * p.din; i += NTHREADS) p.dx[j0 * p.din + i] = dx_s[i];
}

// dM_t[b, a] over one chunk of nodes: dZ conj(x~), a thread per entry (b fastest: neighbouring threads read neighbouring
// columns of dZ), the nodes in order.
template <typename T>
__global__ void __launch_bounds__(NTHREADS) node_products_dw_kernel(NArgs<T> p) {
  const int32_t* d = p.desc + blockIdx.y * NDESC;
  const int zoff = d[1], bm = d[2], am = d[3], xoff = d[4], mode = d[5], row0 = d[6];
  const int64_t j0 = (int64_t)blockIdx.x * p.chunk, j1 = min(j0 + p.chunk, p.n_nodes);
  for (int i = threadIdx.x + blockIdx.z * NTHREADS; i < bm * am * p.k; i += NTHREADS * gridDim.z) {
    const int b = i % bm, a = (i / bm) % am, t = i / (bm * am), idx = b * am + a;
    T gr = T(0), gi = T(0);
#pragma unroll 4
    for (int64_t j = j0; j < j1; ++j) {
      T xr, xi;
      operand(p.x + j * p.din, xoff, mode, a, xr, xi);
      const int64_t at = j * p.k + t;
      if (d[0]) {
        const T zr = p.dzc[(at * p.wc + zoff + b) * 2], zi = p.dzc[(at * p.wc + zoff + b) * 2 + 1];
        gr += zr * xr;
        gr += zi * xi;
        gi += zi * xr;
        gi -= zr * xi;
      } else {
        gr += p.dzr[at * p.wr + zoff + b] * xr;
      }
    }
    if (d[0]) {
      T* out = p.dcw + ((int64_t)blockIdx.x * p.crows + row0 + 2 * idx) * p.k + t;
      out[0] = gr;
      out[p.k] = gi;
    } else {
      p.drw[((int64_t)blockIdx.x * p.rrows + row0 + idx) * p.k + t] = gr;
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

int check_nodes(const char* what, const void* x, const void* cw, const void* rw, const int32_t* desc, int64_t n_nodes, int n_blocks, int din, int k,
                int wc, int wr, int dtype) {
  GM_REQUIRE(n_nodes >= 0 && n_blocks >= 0 && n_blocks <= 65535 && din >= 1 && din <= 2048 && k >= 2 && wc >= 0 && wr >= 0, GM_ERR_ARGUMENT,
             "%s: bad sizes", what);
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_F64, GM_ERR_UNSUPPORTED, "%s: dtype must be float32 or float64", what);
  GM_REQUIRE(n_nodes == 0 || n_blocks == 0 || (x && desc && (cw || wc == 0) && (rw || wr == 0)), GM_ERR_ARGUMENT, "%s: null pointer", what);
  GM_REQUIRE(n_nodes / NODES < ((int64_t)1 << 31) - 1, GM_ERR_LIMIT, "%s: too many nodes", what);
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
    const size_t smem = (size_t)NODES * din * sizeof(T);
    const int st = allow_smem(node_products_forward_kernel<T>, smem, "gm_node_products_forward");
    if (st != GM_OK) return st;
    node_products_forward_kernel<T><<<(unsigned)((n_nodes + NODES - 1) / NODES), NTHREADS, smem, (cudaStream_t)stream>>>(p);
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
    p.crows = crows; p.rrows = rrows; p.chunk = chunk;
    const size_t smem = (size_t)NODES * din * sizeof(T);
    int st = allow_smem(node_products_dx_kernel<T>, smem, "gm_node_products_backward");
    if (st != GM_OK) return st;
    node_products_dx_kernel<T><<<(unsigned)((n_nodes + NODES - 1) / NODES), NTHREADS, smem, (cudaStream_t)stream>>>(p);
    st = launch_status("gm_node_products_backward");
    if (st != GM_OK) return st;
    const dim3 grid((unsigned)((n_nodes + chunk - 1) / chunk), (unsigned)n_blocks, 4);
    node_products_dw_kernel<T><<<grid, NTHREADS, 0, (cudaStream_t)stream>>>(p);
    return launch_status("gm_node_products_backward");
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}
