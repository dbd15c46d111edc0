// dim2d_nodebc.cu -- launch of the node boundary pass of one field; the
// per-cell work is node_bc_cell() in dim2d_nodebc.cuh.
#include "dim2d_nodebc.cuh"

namespace dim2d {

namespace {
__global__ void __launch_bounds__(128) k_node_bc(NodeBcArgs a) {
  wait_for_launch_before();
  node_bc_cell(a, blockIdx.x * blockDim.x + threadIdx.x);
}

}  // namespace

cudaError_t launch_node_bc(const NodeBcArgs& a, cudaStream_t s) {
  const int n = node_bc_count(a);
  NodeBcArgs aa = a;
  void* args[] = {&aa};
  return launch_dependent((const void*)k_node_bc, (unsigned)((n + 127) / 128), 128, 0, s, args);
}

}  // namespace dim2d
