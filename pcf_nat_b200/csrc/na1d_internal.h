// Internal C++ interface between the C ABI (na1d_api.cu) and the kernel families.
#pragma once
#include "na1d_common.cuh"

namespace na1d {

// ---- CUDA-core family (na1d_simt.cu)
bool simt_supports_channels(int C);
cudaError_t simt_qk(float* attn, const void* a, const void* b, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t simt_band_x(void* out, const float* band, const void* x, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t simt_bandT_x(void* out, const float* band, const void* x, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t simt_fused_fwd(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                           const int* valid_len, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t simt_delta(float* delta, const void* d_o, const void* o, int rows, int C, int dtype, cudaStream_t st);
cudaError_t simt_fused_bwd(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                           const void* v, const float* lse, const float* delta, const float* rpb, const int* valid_len,
                           const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t window_index(int* j_out, unsigned char* inr, int T, int win, int left, int dil, cudaStream_t st);

// ---- fused pair on warp-level matrix instructions (na1d_mma.cu): what the tcgen05 kernels do not take, up to 128 channels
bool mma_supports(const Geometry& gm);
cudaError_t mma_fused_fwd(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb, const int* valid_len,
                          const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t mma_fused_bwd(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k, const void* v,
                          const void* o, const float* lse, const float* rpb, const int* valid_len, const Geometry& gm, int dtype,
                          cudaStream_t st);
// ---- narrow rows with everything in registers (na1d_march.cu), any strides
bool march_supports(const Geometry& gm, bool backward);
cudaError_t march_fused_fwd(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb, const int* valid_len,
                            const Strides& sq, const Strides& sk, const Strides& sv, const Strides& so, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t march_fused_bwd(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k, const void* v, const float* lse,
                            const float* rpb, const int* valid_len, const Strides& sdq, const Strides& sdk, const Strides& sdv, const Strides& sdo,
                            const Strides& sq, const Strides& sk, const Strides& sv, const Geometry& gm, int dtype, cudaStream_t st);
bool march_band_supports(const Geometry& gm);   // 16, 32 or 64 channels, one head (sequences), dilation 1
cudaError_t march_band_out(float* band, const void* a, const void* b, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t march_band_rows(void* out, const float* band, const void* x, bool transposed, const Geometry& gm, int dtype, cudaStream_t st);

bool mma_band_supports(const Geometry& gm);
cudaError_t mma_band_out(float* band, const void* a, const void* b, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t mma_band_rows(void* out, const float* band, const void* x, bool transposed, const Geometry& gm, int dtype, cudaStream_t st);

// ---- tcgen05 / TMA family (na1d_tc_fwd.cu)
bool tc_fwd_supports(const Geometry& gm);  // shape limits of the tcgen05 forward
cudaError_t tc_fused_fwd(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                         const int* valid_len, const Geometry& gm, int dtype, cudaStream_t st);
// status words of the tcgen05 translation units (read and cleared; the call synchronises the device): 0 = no bounded
// wait expired, > 0 = a code naming the wait, < 0 = the read failed
int tc_read_status();
int tc_bwd_read_status();
int tc_seg_read_status();
int tc_bwd_seg_read_status();

// ---- tcgen05 / TMA family, segmented tiling (na1d_tc_fwd_seg.cu, na1d_tc_bwd_seg.cu): any dilation, strided tensors
SegGeom seg_geometry(const Geometry& gm, int step);
bool tc_seg_supports(const Geometry& gm);
bool tc_bwd_seg_supports(const Geometry& gm, bool has_bias = false, bool wants_bias_grad = false);
cudaError_t tc_fused_fwd_seg(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                             const int* valid_len, const Strides& sq, const Strides& sk, const Strides& sv, const Strides& so,
                             const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t tc_fused_bwd_seg(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                             const void* v, const float* lse, const float* rpb, const int* valid_len, float* scratch,
                             size_t scratch_floats, const Strides& sdq, const Strides& sdk, const Strides& sdv, const Strides& sdo,
                             const Strides& sq, const Strides& sk, const Strides& sv, const Geometry& gm, int dtype, cudaStream_t st);
bool bias_grad_partial_rows();   // NA1D_BIAS_GRAD_ROWS=1: per-CTA rows of the bias gradient in the scratch, added up in a fixed order
void tensor_map_cache_stats(long long* hits, long long* misses);

// ---- the unfused pair on the tcgen05 kernels (na1d_tc_unfused.cu): flat tiling, same shape limits as the fused forward
bool tc_unfused_supports(const Geometry& gm);
cudaError_t tc_qk(float* attn, const void* a, const void* b, const Geometry& gm, int dtype, cudaStream_t st);
cudaError_t tc_band_x(void* out, const float* band, const void* x, const Geometry& gm, int dtype, cudaStream_t st);
int tc_unfused_read_status();
bool tc_unfused_t_supports(const Geometry& gm);
cudaError_t tc_bandT_x(void* out, const float* band, const void* x, const Geometry& gm, int dtype, cudaStream_t st);
int tc_unfused_t_read_status();

// ---- fused pair with attention dropout (na1d_tc_fwd_drop.cu, na1d_tc_bwd_drop.cu): flat tiling of the tcgen05 kernels
cudaError_t tc_fused_fwd_dropout(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                                 const int* valid_len, const Geometry& gm, int dtype, const DropoutCfg& drop, cudaStream_t st);
cudaError_t tc_fused_bwd_dropout(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                                 const void* v, const float* lse, const float* rpb, const int* valid_len, float* scratch,
                                 size_t scratch_floats, const Geometry& gm, int dtype, const DropoutCfg& drop, cudaStream_t st);
int tc_drop_read_status();
int tc_bwd_drop_read_status();
// shape limits of the tcgen05 backward, including whether its shared memory fits with a bias table (has_bias) and the
// bias-gradient accumulators (wants_bias_grad)
bool tc_bwd_supports(const Geometry& gm, bool has_bias = false, bool wants_bias_grad = false);
cudaError_t tc_fused_bwd(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                         const void* v, const float* lse, const float* rpb, const int* valid_len, float* scratch,
                         size_t scratch_floats, const Geometry& gm, int dtype, cudaStream_t st);

// ---- parameter gradients of projections (na1d_wgrad.cu): d_w[i] (M, N) = dy[i]^T x[i] with dy (rows, M), x (rows, N), d_b[i] (M) = column
// sums of dy[i]; either may be null, count <= 2
size_t wgrad_scratch_floats(const int64_t* M, const int64_t* N, int count, int64_t rows);
cudaError_t wgrad(void* const* d_w, void* const* d_b, const void* const* dy, const void* const* x, const int64_t* M, const int64_t* N, int count,
                  int64_t rows, float* scratch, bool out32, int dtype, cudaStream_t st);
int wgrad_read_status();

// ---- a block's MLP, out = s + GELU(h w1^T + b1) w2^T + b2 (na1d_mlp.cu)
bool mlp_supports(int64_t D, int64_t F);
size_t mlp_scratch_floats(int64_t rows, int64_t F);
cudaError_t mlp_forward(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const void* b1, const void* w2, const void* b2, bool rounded,
                        float* scratch, int64_t rows, int64_t F, int dtype, cudaStream_t st);
int mlp_read_status();
// its backward (na1d_mlp_bwd.cu): df = (d w2) GELU'(f), dh = df w1, gelu = GELU(f); dh, df, gelu, f (and the forward's f) 32-byte aligned
cudaError_t mlp_backward(void* dh, void* df, void* gelu, const void* d, const void* f, const void* w1, const void* w2, float* scratch, int64_t rows, int64_t F,
                         int dtype, cudaStream_t st);
int mlp_bwd_read_status();

// ---- row and column kernels of a transformer block and of the statistics pooling (na1d_block.cu)
int block_partial_rows(long long rows);
cudaError_t block_valid_tokens(int* out, const void* padding, bool is64, int n_padding, int N, int T, cudaStream_t st);
cudaError_t block_ln_fwd(void* y, void* sum, float* mean, float* rstd, const void* x, const void* dx, const float* w, const float* b,
                         int rows, int D, float eps, int dtype, cudaStream_t st);
cudaError_t block_ln_bwd(void* dx, float* sums, float* part, const void* dy, const void* x, const float* mean, const float* rstd,
                         const float* w, const void* res, int rows, int D, int dtype, cudaStream_t st);
// (sums null: the partial sums stay in `part`, for block_ln_sums, which adds those of two)
cudaError_t block_ln_sums(float* const* sums, const float* const* part, int rows, int D, cudaStream_t st);
cudaError_t block_gelu_fwd(void* y, const void* x, long long n, int dtype, cudaStream_t st);
cudaError_t block_gelu_bwd(void* dx, float* sums, float* part, const void* dy, const void* x, int rows, int F, int dtype, cudaStream_t st);
cudaError_t block_column_sums(float* sums, float* part, const void* x, int rows, int F, int dtype, cudaStream_t st);
cudaError_t block_cast(void* out, const float* const* src, const int64_t* dst, const int64_t* n, int count, int dtype, cudaStream_t st);
cudaError_t block_permute_heads(void* out, const void* in, int batch, int T, int parts, int heads, int C, bool to_dense, cudaStream_t st);
cudaError_t block_transpose(void* out, const void* in, int N, int C, int T, bool to_tokens, int dtype, cudaStream_t st);
cudaError_t block_pack_grouped(void* out_w, void* out_b, const void* w, const void* b, bool src32, int C, int groups, int parts, int dtype,
                               cudaStream_t st);
cudaError_t block_unpack_grouped(void* d_w, void* d_b, const float* dense, const float* sums, bool dst32, int C, int groups, int parts, int dtype,
                                 cudaStream_t st);
cudaError_t block_add_to_rows(void* out, long long ld, const void* x, const void* dx, int rows, int D, int dtype, cudaStream_t st);
cudaError_t block_pool_fwd(float* out, float* stats, const void* logits, const void* x, long long ldx, int N, int T, int C, float floor_var,
                           int dtype, cudaStream_t st);
cudaError_t block_pool_bwd(void* d_logits, void* dx, const float* d_out, const float* out, const float* stats,
                           const void* logits, const void* x, int N, int T, int C, float floor_var, int dtype, cudaStream_t st);

}  // namespace na1d
