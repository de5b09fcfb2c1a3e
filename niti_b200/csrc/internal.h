// Launchers shared between the translation units of the library (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace niti {

// error plumbing: both return NITI_ERR_CUDA (or 0 for cudaSuccess) and remember the text
int set_cuda_error(cudaError_t e);
int set_cuda_error_text(const char* text);
int launched(cudaError_t e);  // the result of one kernel launch: as set_cuda_error, and counts those that went through (niti_launch_count)

// What a launcher returns (never the library) where the driver has fewer SMs or clusters for a launch than its thread blocks, which
// wait for one another, need at a time: on a stream or in a context that is held to part of the device.  Nothing has been enqueued.
constexpr int LAUNCH_REFUSED = -1000;

// Requantisation fused into a contraction's epilogue: the kernel narrows with the shift it finds in
// state[0] and its last CTA verifies that shift; `only_if_redo` launches are no-ops unless state[2] is set.
struct FusedArgs {
    int32_t* state;        // {shift, max|acc|, redo flag, redo count, exit ticket, barrier arrivals, -, -}
    int only_if_redo;
    int one;               // 1: the streaming kernel narrows again in the same launch where its guess was wrong (forward layers)
    int parked;            // 1: accumulator-parking kernel (exact in one launch; needs umma_conv_fits_parked)
    int mode, relu;
    const unsigned long long* seed;
    unsigned rng_stream;
    unsigned long long rng_offset;
    int kind, target_bits;
    const int32_t* exp_a; const int32_t* exp_b; int32_t* exp_out; int32_t* shift_out;
    const int8_t* relu_mask;  // optional, same shape as the output: zero the output where this tensor is <= 0
    int8_t* pool_out;         // optional (forward, parked kernel): 2x2 / stride-2 max-pooled copy of the output
    void* side;               // optional (streaming kernel, round-to-nearest, no ReLU): outputs / 4 bytes of side codes
    int whole;                // 1: one thread block to a tile, however few there are
};

extern int g_two_cta;    // CTA pairs (cta_group::2) where the shape allows: bit 0 for GEMMs, bit 1 for convolutions
extern int g_cooperative;  // 1: cooperative launches for the kernels with a grid barrier (see umma_kernels.cu)
extern int g_opt_wgrad_reduce;  // NITI_OPT_WGRAD_TMA_REDUCE
extern int g_stage_cap;  // experiments: cap on the shared-memory stages the GEMM / conv kernels use (0 = all)

// tensor-core (tcgen05) paths, umma_kernels.cu; `out` is int32 (fused == null) or int8
int umma_gemm_splits(int M, int N, int K);
int umma_gemm(const int8_t* A, const int8_t* B, void* out, unsigned* maxabs, int M, int N, int K, int trans_a,
              int trans_b, int splits, const FusedArgs* fused, int32_t* status, cudaStream_t st, int rows32 = 0,
              int lda = 0, int ldc = 0);  // row pitches of A and of an int32 result in elements (0: dense)
int umma_conv(const int8_t* x, const int8_t* w, void* out, unsigned* maxabs, int Nimg, int H, int W, int C, int K,
              int R, int S, int pad, int flip, const FusedArgs* fused, int32_t* status, cudaStream_t st);
// red / outc: reduction channels per tap, output channels; k3: 3x3 filters, padding 1
bool umma_conv_fits_parked(int Nimg, int H, int W, int red, int outc, bool k3, int flip);
bool umma_conv_pool_fusable(int Nimg, int H, int W, int outc);  // the fused forward kernel can also emit the 2x2-pooled output
size_t umma_wgrad_scratch_bytes(int Nimg, int H, int W, int C, int K, int R, int S);
// max_splits > 0 caps the number of pixel-range splits (and with it the size of `partial`)
// direct == 1: `partial` is the zeroed gradient and the CTAs add into it (TMA reduction) instead of storing partials
int umma_conv_wgrad_partials(const int8_t* x, const int8_t* err, int32_t* partial, int* splits_out, int max_splits,
                             int Nimg, int H, int W, int C, int K, int R, int S, int pad, int32_t* status, cudaStream_t st,
                             int direct = 0);
// gradient, cleared by the launch, and for small layers (*updated) the update, in one (cooperative) launch of one wave of thread
// blocks; state: int32[4], zero between calls; words: cleared, the first is max |g| of an update; may return LAUNCH_REFUSED
bool umma_conv_wgrad_update_fits(int Nimg, int H, int W, int C, int K, int R);
int umma_conv_wgrad_update(const int8_t* x, const int8_t* err, int32_t* out, int8_t* w, uint32_t* words, int num_words, int32_t* state,
                           int Nimg, int H, int W, int C, int K, int R, int S, int pad, int mu, int mode, const unsigned long long* seed,
                           unsigned rng_stream, bool* updated, int32_t* status, cudaStream_t st);
// operands with the batch innermost ([channels][H][W][N]) -> out [C][R][S][K] (zeroed by the caller)
int umma_conv_wgrad_batch_inner(const int8_t* x_t, const int8_t* err_t, int32_t* out, int Nimg, int H, int W, int C, int K, int R,
                                int S, int pad, int32_t* status, cudaStream_t st);
// several layers' weight gradients, each ADDED into its g32, in one launch (umma_kernels.cu)
struct WgradJob { const int8_t* x; const int8_t* err; int32_t* g32; int N, H, W, C, K, R, S, pad; };
int umma_wgrad_multi_max();
int umma_conv_wgrad_multi(const WgradJob* jobs, int count, int32_t* status, cudaStream_t st);
int absmax_i32(const int32_t* acc, long long n, unsigned* maxabs, cudaStream_t st);  // reduces into *maxabs (not cleared)

// CUDA-core paths, simt_kernels.cu
int simt_conv_fprop(const int8_t* x, const int8_t* w, int32_t* y32, unsigned* maxabs, int Nimg, int H, int W, int C,
                    int K, int R, int S, int pad, cudaStream_t st);
int simt_conv_dgrad(const int8_t* err, const int8_t* w, int32_t* e32, unsigned* maxabs, int Nimg, int H, int W, int C,
                    int K, int R, int S, int pad, cudaStream_t st);
int simt_conv_wgrad(const int8_t* x, const int8_t* err, int32_t* g32, unsigned* maxabs, int Nimg, int H, int W, int C,
                    int K, int R, int S, int pad, cudaStream_t st);
int simt_gemm(const int8_t* A, const int8_t* B, int32_t* C32, unsigned* maxabs, int M, int N, int K, int trans_a,
              int trans_b, cudaStream_t st);
int clear_words(void* p, int n, cudaStream_t st);  // n (few) 32-bit words to zero
int reduce_partials(const int32_t* partial, int splits, long long n, int32_t* out, unsigned* maxabs, cudaStream_t st);
int reduce_rows32(const int32_t* partial, int splits, int rows, int cols_out, int32_t* out, unsigned* maxabs, cudaStream_t st);
// xcol[pixels][32] and wp[K][32] in the order the MMA reads 32-byte rows in (rows32 of umma_gemm).
// w / wp / K: optionally the layer's filters w[K][R*S*C] are padded to wp[K][32] by the same launch
int im2col32(const int8_t* x, int8_t* xcol, int Nimg, int H, int W, int C, int R, int S, int pad, cudaStream_t st,
             const int8_t* w = nullptr, int8_t* wp = nullptr, int K = 0);
// rows of `bytes` bytes from one pitch (in bytes) to another; everything a multiple of `unit` (1 or 4)
int copy_rows(const void* src, long long src_pitch, void* dst, long long dst_pitch, long long bytes, long long rows, int unit, cudaStream_t st);
int unpack_i4(const uint8_t* in, int8_t* out, long long nbytes, cudaStream_t st);  // two int4 per byte (low nibble first) -> int8

}  // namespace niti
