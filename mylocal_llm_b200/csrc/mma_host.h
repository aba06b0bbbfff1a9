// Request descriptor shared by the C ABI dispatcher and the tensor-core GEMV launcher.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200q {

struct MmaRequest {
    int mode;  // 0 linear, 1 SwiGLU, 2 grouped gate/up, 3 grouped down
    const uint8_t *wa;
    const uint8_t *wb;
    int fmt_a, fmt_b;
    long long stride_a, stride_b;
    const unsigned long long *table_a, *table_b;   // optional per-expert pointer tables
    int tables_aligned16;                          // caller vouches: every table entry is 16-byte aligned
    int tiled;                                     // Q4_K / Q5_K weights in their tile layout (direct kernel only)
    int n, k, m;
    const void *x;
    int x_dtype;
    void *y;
    int y_dtype;
    int topk;
    const int32_t *order;
    const int32_t *seg_expert;
    const int32_t *seg_begin;
    const int32_t *seg_count;
    const int32_t *num_segments;
    int max_segments;
    const float *route;
    int flat_rows;
    const uint64_t *y_table;
    int rows_per_rank;
    int *status;
    // optional: mode 2: per-token activation images (direct_token_images) of the rows of x; mode 3: images of the hidden
    // activations (hidden_images), one per sorted assignment
    const void *images;
};

// Launches the tensor-core kernel when the request fits it (alignment, K multiple of 256, shared
// memory); otherwise leaves *launched false and the caller runs the FP32-lane kernel.
int mma_try_launch(const MmaRequest &q, cudaStream_t stream, bool *launched);
// Tokens per mma_try_launch() request for this format / mode / K: 8, or 16 where the direct kernel
// is in use and serves two token tiles per pass.
int mma_tokens_per_pass(int fmt, int mode, int k, int x_dtype, bool tiled);

// Same contract for the direct-load kernel (Q4_K / Q5_K only); tried first.
int direct_try_launch(const MmaRequest &q, cudaStream_t stream, bool *launched);
// Tokens per launch the direct kernel takes for this format / mode / K (8, or 16 in the dense modes
// when two token tiles fit in shared memory).
int direct_tokens_per_pass(int fmt, int mode, int k, int x_dtype);

// Activation images for the grouped gate/up launch of the direct kernel: what that kernel would prepare for
// a token (scaled FP16 fragments, sub-block sums, the scale), written once per token so that an expert
// segment only gathers its tokens' images. Bytes per token (0 = this K / dtype has no images), and the
// launch that fills `images` [rows x bytes] from x [rows x k].
int direct_token_image_bytes(int k, int x_dtype);
int direct_token_images(const void *x, int x_dtype, int rows, int k, void *images, cudaStream_t stream);

// Grouped launches over images (grouped_stream.cu). grouped_*_kp: the warps per row group with which a plan of that bound
// streams (fmt: B200Q_Q4_K / Q5_K tiles for gate/up, B200Q_Q6_K_TILED / Q8_0_TILED for down), 0 where the block-structured
// kernels are the better ones or two segment buffers do not fit; a function of types, sizes and the bound alone, so that
// the block-structured kernels take the same kp when such a plan comes without images (or with peers' rows) and add in the
// same order. *launched stays false where the request does not stream.
int grouped_gate_up_kp(int fmt, int n, int k, int x_dtype, int max_segments);
int grouped_down_kp(int fmt, int n, int k, int max_segments);
int grouped_gate_up_launch(const MmaRequest &q, cudaStream_t stream, bool *launched);
int grouped_down_launch(const MmaRequest &q, cudaStream_t stream, bool *launched);
// A block-structured grouped kernel holds its outstanding loads in L1. Behind a streaming one an SM would keep the split
// that leaves it 28 KB (the hint is what makes the driver set it anew): gate/up streaming, then down of 64 experts of
// 2048 x 2048 at 128 tokens, 277 us without the hint for kernels that take 134 and 115 alone, 251 with it.
inline void roomy_l1(const void *kernel) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1) != cudaSuccess) cudaGetLastError();
}
int hidden_image_bytes(int k);
int hidden_images(const float *h, int rows, int k, void *images, cudaStream_t stream);

// Weights in the Q6_K / Q8_0 tile layouts (mode 0 or 3, at most tiled_tokens_per_pass() tokens):
// there is no other kernel for these layouts, so a request that does not fit returns an error
// instead of declining.
int q6k_tiled_launch(const MmaRequest &q, cudaStream_t stream);

// The kernel arguments and dynamic shared memory the two grouped launches above would use for a request,
// without launching (the persistent one-token MoE step runs the same bodies with the same split of the work).
struct DirectArgs;
struct Q6TiledArgs;
bool direct_plan_args(const MmaRequest &q, DirectArgs *out, long long *smem_out);
int tiled_plan_args(const MmaRequest &q, Q6TiledArgs *out, long long *smem_out);
int tiled_tokens_per_pass(int mode, int k, int x_dtype);

}  // namespace b200q
