// fp32 sparse 1x1 convolution with the activations in tensor memory (sparse_tmem.cu).
#pragma once
#include <cstring>
#include <vector>

#include "common.cuh"

namespace plb {

// The non-zeros of one layer as this kernel walks them, laid out once when the layer is prepared:
//   pixels                  pixels per lane: 512 / pixels input channels are held at a time (a chunk)
//   rows[chunk * cout + oc] = {first 16-byte word of its batches, entries, bias bits, 0}
//   batches                 rows of whole batches of 8 (4 at eight pixels) entries: the columns, pixels * (input channel
//                           within the chunk), then every weight twice; one empty batch behind the last row
struct SparseTmemLists {
  int pixels;
  std::vector<int4> rows;
  std::vector<int> batches;
};
// false: a row does not name its input channels in ascending order (chunks would change the order of its sum), or an image
// is too large for 32-bit offsets
bool sparse_tmem_build(int cin, int cout, long hw, const std::vector<int>& row_ptr, const std::vector<int>& col,
                       const std::vector<float>& val, const float* bias, SparseTmemLists* out);

struct SparseTmemProblem {
  int batch, cin, cout, hw, pixels;
  long nnz;
  const float* x;     // [batch, cin, hw]
  const void* rows;   // SparseTmemLists on the device
  const void* batches;
  int act;
  float alpha;
  float* y;           // [batch, cout, hw]
};
// Whether it is the faster kernel for these sizes and addresses.
bool sparse_tmem_better(const SparseTmemProblem& p, int sm_count);
int sparse_tmem_launch(plb_ctx* ctx, const SparseTmemProblem& p);

}  // namespace plb
