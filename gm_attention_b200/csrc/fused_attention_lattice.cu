// Entry points of the lattice fast path with fp32 arithmetic (float32 or bfloat16 node fields); the kernels and their
// description are in lattice_fma.cuh, instantiated per storage type in lattice_fma_f32.cu and lattice_fma_bf16.cu.
#include "lattice_fma.cuh"

namespace gmb {
namespace {

using lat::LatArgs;
using lat::LatPlan;
using lat::LAT_MAX_CF;

// delta[node, h] = sum over the head's columns of dO * O
template <typename S>
__global__ void lattice_delta_kernel(const S* __restrict__ dout, const S* __restrict__ out, float* __restrict__ delta, int64_t n_rows,
                                     int D, int H, LatPlan P) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= n_rows * H) return;
  const int64_t node = w / H;
  const int h = (int)(w % H);
  float acc = 0.f;
  for (int c = lane; c < P.a0; c += 32) {
    const int64_t g = node * D + P.real_off + h * P.a0 + c;
    acc += ld<float>(dout + g) * ld<float>(out + g);
  }
  for (int f = 0; f < P.n_cf; ++f)
    for (int c = lane; c < 2 * P.ac; c += 32) {
      const int64_t g = node * D + P.cf_off[f] + 2 * h * P.ac + c;
      acc += ld<float>(dout + g) * ld<float>(out + g);
    }
  acc = warp_sum(acc);
  if (lane == 0) delta[node * H + h] = acc;
}

// The layouts the lattice kernels serve: an optional scalar block and complex frequencies that share one
// multiplicity.  Anything else is GM_ERR_UNSUPPORTED (callers then use the general CSR kernels).
int make_lat_plan(const int64_t* desc_host, int F, int H, int D, LatPlan& P) {
  GM_REQUIRE(F >= 1 && F <= LAT_MAX_CF + 1, GM_ERR_UNSUPPORTED, "gm_lattice_attention: at most %d frequencies per head", LAT_MAX_CF + 1);
  P = LatPlan{};
  for (int f = 0; f < F; ++f) {
    const int n = (int)desc_host[5 * f], a_n = (int)desc_host[5 * f + 1], off = (int)desc_host[5 * f + 2];
    const int dim = n == 0 ? 1 : 2;
    GM_REQUIRE(n >= 0 && a_n >= 1 && off >= 0 && off + H * a_n * dim <= D, GM_ERR_ARGUMENT,
               "gm_lattice_attention: descriptor row %d leaves the width D=%d", f, D);
    if (n == 0) {
      GM_REQUIRE(P.a0 == 0, GM_ERR_ARGUMENT, "gm_lattice_attention: two scalar rows");
      P.a0 = a_n;
      P.real_off = off;
    } else {
      GM_REQUIRE(P.n_cf < LAT_MAX_CF, GM_ERR_UNSUPPORTED, "gm_lattice_attention: more than %d complex frequencies", LAT_MAX_CF);
      GM_REQUIRE(P.ac == 0 || P.ac == a_n, GM_ERR_UNSUPPORTED, "gm_lattice_attention: complex frequencies must share one multiplicity");
      P.ac = a_n;
      P.cf_off[P.n_cf] = off;
      P.cf_order[P.n_cf] = n;
      ++P.n_cf;
    }
  }
  return GM_OK;
}

int run_pass(int mode, LatArgs& a, int n_order_rows, int64_t batch, int dtype, cudaStream_t stream) {
  for (int f = 0; f < a.plan.n_cf; ++f)
    GM_REQUIRE(a.plan.cf_order[f] <= a.NORD, GM_ERR_ARGUMENT, "gm_lattice_attention: tables hold %d orders, frequency %d needs more", a.NORD, a.plan.cf_order[f]);
  return dtype == GM_F32 ? lat::lattice_pass_f32(mode, a, n_order_rows, batch, stream) : lat::lattice_pass_bf16(mode, a, n_order_rows, batch, stream);
}

int check_lattice(int rows, int nlon, int64_t batch, int D, int H, int W, int ES, int NORD, int dtype) {
  GM_REQUIRE(rows >= 1 && nlon >= 1 && batch >= 1 && D >= 1, GM_ERR_ARGUMENT, "gm_lattice_attention: bad sizes");
  GM_REQUIRE(H >= 1 && H <= 65535 && batch <= 65535, GM_ERR_LIMIT, "gm_lattice_attention: heads and batch must fit a grid dimension");
  GM_REQUIRE(W >= 0 && NORD >= 0 && ES >= 2 * NORD + 1, GM_ERR_ARGUMENT, "gm_lattice_attention: entry stride %d too small for %d orders", ES, NORD);
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_BF16, GM_ERR_UNSUPPORTED, "gm_lattice_attention: float32 or bfloat16 node fields (fp32 arithmetic)");
  return GM_OK;
}

}  // namespace
}  // namespace gmb

using namespace gmb;

extern "C" int gm_lattice_attention_forward(const void* q, const void* k, const void* v, const int* win_cnt, const int* win_lo,
                                            const int* win_off, const float* entries, const int* row_order, int n_order_rows,
                                            const int64_t* desc_host, int F, int rows, int nlon, int64_t batch, int D, int H, int W,
                                            int ES, int NORD, double scale, int dtype, void* out, float* lse, void* stream) {
  int status = check_lattice(rows, nlon, batch, D, H, W, ES, NORD, dtype);
  if (status != GM_OK) return status;
  GM_REQUIRE(q && k && v && win_cnt && win_lo && win_off && entries && row_order && desc_host && out && lse, GM_ERR_ARGUMENT,
             "gm_lattice_attention_forward: null pointer");
  if (n_order_rows == 0) return GM_OK;
  LatArgs a{};
  status = make_lat_plan(desc_host, F, H, D, a.plan);
  if (status != GM_OK) return status;
  a.f1 = k; a.f2 = v; a.o1 = q; a.r1 = out; a.lse_out = lse;
  a.win_cnt = win_cnt; a.win_lo = win_lo; a.win_off = win_off; a.entries = entries; a.row_order = row_order;
  a.rows = rows; a.nlon = nlon; a.D = D; a.H = H; a.W = W; a.ES = ES; a.NORD = NORD; a.scale = (float)scale;
  return run_pass(lat::MODE_FWD, a, n_order_rows, batch, dtype, (cudaStream_t)stream);
}

extern "C" int gm_lattice_attention_backward(const void* dout, const void* q, const void* k, const void* v, const void* out,
                                             const float* lse, const int* win_cnt, const int* win_lo, const int* win_off,
                                             const float* entries, const int* row_order, int n_order_rows, const int* t_win_cnt,
                                             const int* t_win_lo, const int* t_win_off, const float* t_entries,
                                             const int* t_row_order, int t_n_order_rows, const int64_t* desc_host, int F, int rows,
                                             int nlon, int64_t batch, int D, int H, int W, int ES, int NORD, double scale, int dtype,
                                             void* dq, void* dk, void* dv, float* delta, void* stream) {
  int status = check_lattice(rows, nlon, batch, D, H, W, ES, NORD, dtype);
  if (status != GM_OK) return status;
  GM_REQUIRE(dout && q && k && v && out && lse && win_cnt && win_lo && win_off && entries && row_order && t_win_cnt && t_win_lo &&
                 t_win_off && t_entries && t_row_order && desc_host && dq && dk && dv && delta,
             GM_ERR_ARGUMENT, "gm_lattice_attention_backward: null pointer");
  cudaStream_t cs = (cudaStream_t)stream;
  LatArgs a{};
  status = make_lat_plan(desc_host, F, H, D, a.plan);
  if (status != GM_OK) return status;
  a.rows = rows; a.nlon = nlon; a.D = D; a.H = H; a.W = W; a.ES = ES; a.NORD = NORD; a.scale = (float)scale;
  a.lse = lse; a.delta = delta;
  // Delta = <dO, O>: formed inside pass T when that pass owns every target row (one sweep over dO and O less: 0.22 ms of
  // 13.1 at 128 x 256, batch 4, 4 heads of 8 x (m <= 3)); a row list that leaves targets out gets the kernel
  const bool fused_delta = n_order_rows == rows;
  if (!fused_delta) {
    const int64_t n_rows = batch * rows * (int64_t)nlon, warps = n_rows * H;
    if (dtype == GM_F32)
      lattice_delta_kernel<float><<<(unsigned)((warps + 7) / 8), 256, 0, cs>>>((const float*)dout, (const float*)out, delta, n_rows, D, H, a.plan);
    else
      lattice_delta_kernel<__nv_bfloat16><<<(unsigned)((warps + 7) / 8), 256, 0, cs>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)out, delta,
                                                                                       n_rows, D, H, a.plan);
    status = launch_status("gm_lattice_attention_backward (delta)");
    if (status != GM_OK) return status;
  }
  if (n_order_rows > 0) {
    LatArgs t = a;
    t.f1 = k; t.f2 = v; t.o1 = q; t.o2 = dout; t.r1 = dq;
    if (fused_delta) { t.out_fwd = out; t.delta_out = delta; }
    t.win_cnt = win_cnt; t.win_lo = win_lo; t.win_off = win_off; t.entries = entries; t.row_order = row_order;
    status = run_pass(lat::MODE_BWD_T, t, n_order_rows, batch, dtype, cs);
    if (status != GM_OK) return status;
  }
  if (t_n_order_rows > 0) {
    a.f1 = q; a.f2 = dout; a.o1 = k; a.o2 = v; a.r1 = dk; a.r2 = dv;
    a.win_cnt = t_win_cnt; a.win_lo = t_win_lo; a.win_off = t_win_off; a.entries = t_entries; a.row_order = t_row_order;
    status = run_pass(lat::MODE_BWD_S, a, t_n_order_rows, batch, dtype, cs);
  }
  return status;
}
