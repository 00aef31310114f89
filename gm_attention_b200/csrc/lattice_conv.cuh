// What the kernels of the lattice convolution share (lattice_conv.cu: CUDA cores, lattice_conv_tc.cu: tensor cores).
#pragma once
#include "common.cuh"

namespace gmb {
namespace lconv {

struct ConvArgs {
  const void* x;        // (batch, rows * nlon, width) node field
  const void* g;        // table_grad: the output gradient, same layout
  const float* table;   // (entries, table_width)
  const int* items;     // (n_items, 3): kind (0 complex copy, 1 pair of scalar channels), field column, table column
  const int* win_cnt;   // (rows, 2 * halo + 1)
  const int* win_lo;
  const int* win_off;
  const int* order;     // apply: target rows, heaviest first; table_grad: (blocks, 2) = window index, first offset
  void* y;              // apply: (batch, rows * nlon, width)
  float* dtable;        // table_grad: (entries, table_width)
  int n_items, rows, nlon, batch, width, halo, table_width, transpose;
};

// Tensor-core forms for bfloat16 fields: whether the sizes and addresses allow them, whether they are the faster ones, and the
// launches.
bool tensor_cores_can(const ConvArgs& a);   // the fields are such as the kernels read
bool tensor_cores_hold(const ConvArgs& a);  // apply's list of neighbour rows
bool tensor_cores_apply(const ConvArgs& a);
bool tensor_cores_table_grad(const ConvArgs& a);
int apply_tc(const ConvArgs& a, int n_order, cudaStream_t stream);
int table_grad_tc(const ConvArgs& a, int64_t n_blocks, cudaStream_t stream);

}  // namespace lconv
}  // namespace gmb
