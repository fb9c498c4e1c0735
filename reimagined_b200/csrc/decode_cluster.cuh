// decode_cluster.cu -- the blocks of a decode step as one launch: a thread-block cluster carries a few sequences through all of them.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/ternary_b200.h"

namespace tbl {

// Where a block's device state lies (the caller's layout).
struct ClusterBlockState {
    float* ring;
    float* ssm;
    float* k_cache;
    float* v_cache;
};

// True where launch_decode_cluster takes the model at this batch and cache capacity; fills the launch's shape.
struct ClusterShape {
    int ctas;           // of a cluster
    int rows;           // sequences of a cluster
    int clusters;
    size_t smem;
};
bool decode_cluster_shape(const tbl_decode_model& m, int batch, int capacity, ClusterShape* shape);

// All blocks of one step: the embedding rows of token_ids go through them, the residual stream in front of the final norm is left in
// hidden_out [batch, d_model], positions are advanced.  trace (optional): [n_blocks, batch, d_model], the stream entering each block.
cudaError_t launch_decode_cluster(const tbl_decode_model& m, const ClusterShape& shape, int batch, int capacity, const ClusterBlockState* state,
                                  int32_t* positions, const int32_t* token_ids, float* hidden_out, float* trace, int* status, cudaStream_t st);

}  // namespace tbl
