// What the kernels of the factored steerable kernel share (factored_ops.cu: CUDA cores, factored_tc.cu: tensor cores).
#pragma once
#include "common.cuh"

namespace gmb {
namespace factored {

constexpr int FDESC = 8;  // numbers of a block's descriptor: kind (0 real), first column, copies, angular and transport order, power, output offset, real part only

template <typename T>
struct FArgs {
  int64_t n_edges, n_groups;
  int k, wc, wr, n_f, n_blocks, d_out;
  int n_scales;  // 0: rho (n_edges), a block's scale is a power of it; else (SCALED) rho (n_edges, n_scales), its scale a column of it
  const T *h, *zc, *zr, *angular, *transport, *rho;
  const int32_t* desc;
  const int64_t *source, *order, *group_ptr, *group_source;
  T* out;
  // backward
  const T* g;
  const int64_t* target;
  const T *weights, *rows;
  T *dh, *dzc, *dzr, *dweights;
};

// A block's per-edge factor (factored.h:118-144) from the phase tables; SCALED: "power" names a scale.  (Its own body: one over pointers to the three parts, or over accessors, cost the staged
// kernels registers and 1 to 6 %.)
template <bool SCALED, typename T>
__device__ __forceinline__ void table_factor(const FArgs<T>& a, int64_t e, const int32_t* d, T& fr, T& fi) {
  const T *angular = a.angular + e * a.n_f * 2, *t = a.transport + e * a.n_f * 2, *scale = a.rho + e * (SCALED ? a.n_scales : 1);
  fr = T(1);
  fi = T(0);
  const int ang = d[3], trn = d[4], power = d[5];
  if (ang != 0) {
    const int o = ang < 0 ? -ang : ang;
    const T pr = angular[2 * o], pi = ang < 0 ? -angular[2 * o + 1] : angular[2 * o + 1];
    const T nr = fr * pr - fi * pi, ni = fr * pi + fi * pr;
    fr = nr;
    fi = ni;
  }
  if (trn != 0) {
    const int o = trn < 0 ? -trn : trn;
    const T pr = t[2 * o], pi = trn < 0 ? -t[2 * o + 1] : t[2 * o + 1];
    const T nr = fr * pr - fi * pi, ni = fr * pi + fi * pr;
    fr = nr;
    fi = ni;
  }
  T s = T(1);
  if constexpr (SCALED) {
    s = scale[power];
  } else {
    const T r = scale[0];
    for (int x = 0; x < power; ++x) s *= r;
  }
  fr *= s;
  fi *= s;
}

// Tensor-core forms for float32: whether the sizes allow them and they are the faster ones, and the launches.
bool tensor_cores_forward(const FArgs<float>& a);
bool tensor_cores_backward(const FArgs<float>& a);
int forward_tc(const FArgs<float>& a, cudaStream_t stream);
int backward_tc(const FArgs<float>& a, cudaStream_t stream);

}  // namespace factored
}  // namespace gmb
