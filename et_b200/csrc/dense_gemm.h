// Host-side interface of the dense linear (weights whose zero tiles are cheaper to multiply with than to skip).
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace et {

// Tile width and number of CTAs that share a tile's K range (1: pairs of CTAs, each with the whole range), and the modelled
// clocks of a launch.
struct DensePlan {
    int bn = 0, split = 1;
    double cost = 0;
};
DensePlan dense_plan(int tokens, int N, int K);
// W: dense [N x K] on the device; the map holds its address.
int dense_map_weight(CUtensorMap* map, const half* W, int N, int K, const DensePlan& plan);
// kept: device bitmap of the kept tiles ([N / 16] rows of whole 32-bit words, a bit per 16 inputs), null when none was pruned.
int dense_run(const CUtensorMap& tmW, const half* W, const uint32_t* kept, const DensePlan& plan, half* Y, const half* X, const half* bias,
              int T, int N, int K, int gelu, int* err, cudaStream_t st);

}  // namespace et
