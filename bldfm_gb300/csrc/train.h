// One training step of the surrogate MLP (train.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#define MLP_KC 32  // K columns of a streamed weight chunk

// bf16 index of element (n, k) of a 256 x 256 hidden weight operand stored as
// eight K chunks of 256 x MLP_KC core-matrix blocks
__host__ __device__ __forceinline__ uint32_t mlp_chunk_index(int n, int k)
{
    const int kk = k & (MLP_KC - 1);
    return (uint32_t)((k / MLP_KC) * 256 * MLP_KC + (n >> 3) * (MLP_KC / 8) * 64 + (kk >> 3) * 64 + (n & 7) * 8 +
                      (kk & 7));
}

// device buffers of one training step (owned by the network's handle)
struct MlpTrainBuf {
    uint16_t *H[3];        // hidden activations 1..3, 128-row core-matrix tiles of 64 KB
    uint16_t *D[4];        // dZ of hidden layers 1..4, same tiles
    uint16_t *G[3];        // gelu' of hidden layers 1..3, per tile [8-column group][row]
    uint16_t *Xp;          // inputs as three bf16 pieces and a column of ones, 128 x 32 tiles
    float *part_w, *part_o;  // partial sums of the gradients
};

// floats of part_w and part_o for a batch capacity of `batch` samples
size_t mlp_train_part_w(int batch, int nsm);
size_t mlp_train_part_o(int batch, int nsm);

// bf16 operand blocks of the hidden weights: Wf (rows out, K in) and Wb (rows
// in, K out) in K chunks for the training step, Wt (rows out, K in) for the
// layer-by-layer forward pass, Wq = Wt / 2 as four 128 x 128 quarters for serving
struct MlpBlocks {
    uint16_t *Wf[3], *Wb[3], *Wt[3], *Wq[3];
};

struct MlpAdam {
    float *P, *G, *m, *v, *loss;
    float lr, b1, b2, eps, c1, c2;  // lr = 0: gradients only
};

// forward, backward, weight gradients and (lr != 0) the Adam update of n
// samples (a multiple of 256)
cudaError_t launch_mlp_train(const float *X, const float *T, const float *w, int n, const MlpTrainBuf &buf,
                             const MlpBlocks &blk, const MlpAdam &adam, int *err, int nsm, cudaStream_t st);
// every block layout from the FP32 parameters
cudaError_t launch_mlp_blocks(const float *P, const MlpBlocks &blk, cudaStream_t st);
