// Host-side interface of the tile-sparse linear with the activations resident in tensor memory (in_feat up to 1024).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstddef>

namespace et {

struct ResidentWeight;

// Modelled clocks of a launch; 1e30 where the form does not exist (in_feat above 1024).
double resident_cost(int tokens, int N, int K, double density);
// Packs a validated weight (tile-BSR arrays as in tile_weight_pack; no tile twice in a block-row).
int resident_pack(ResidentWeight** out, int K, int N, const half* data, const int* row_ptr, const int* row_offset);
void resident_free(ResidentWeight* w);
size_t resident_bytes(const ResidentWeight* w);
// Block-rows per group of features, and groups.
int resident_block_rows();
int resident_groups(const ResidentWeight* w);
// bias_given: the bias is the caller's and may be the result of the kernel before.
int resident_run(const ResidentWeight* w, half* Y, const half* X, const half* bias, bool bias_given, int T, int gelu, int* err, cudaStream_t st);

}  // namespace et
