// Host-side interface of the tile-sparse linear with the activations resident in tensor memory (in_feat up to 1024).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstddef>

namespace et {

struct ResidentWeight;

// How far a launch's activations and results exceed what L2 holds of them beside the next launch's: 0 up to 60 MB, 1 from 140 MB. In between
// the tile and resident forms go from 0.93 to 1.2 times what their models say (the power limit comes to long launches as well), the dense form from 1.01 to 1.03. (Of short K
// ranges the dense form's model knows as little: 47112 x 512 -> 1024 52 us, 38 by the model.)
inline double beyond_l2(double tokens, int K, int N) {
    if (K < 640) return 0.0;
    const double mb = 2e-6 * tokens * (K + N);
    return mb <= 60.0 ? 0.0 : mb >= 140.0 ? 1.0 : (mb - 60.0) / 80.0;
}
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
