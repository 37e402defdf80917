/*
 * na1d_b200.h -- C ABI of the B200 (sm_100a) 1-D neighbourhood-attention library.
 *
 * All pointers are DEVICE pointers unless a comment says otherwise; all tensors are dense and
 * row-major.  Every function is asynchronous on `stream` (a cudaStream_t passed as void*, NULL =
 * legacy default stream), allocates nothing unless stated, and returns 0 (NA1D_OK) or a negative
 * NA1D_ERR_* code after validating its arguments on the host; no argument error ever reaches
 * the device.  The library is re-entrant; the caller owns every buffer.
 *
 * Geometry shared by all entry points (reference: models/PCF_NATransformer.py:47-56, 153-171):
 *   N sequences (= batch*heads, head index fastest: n = b*heads + h), T tokens, C channels per
 *   head (multiple of 8), window `win` with `left` neighbours before the query, dilation `dil`.
 *   Neighbour kk of query t is key j = t + (kk-left)*dil; keys outside [0,T) read as zero rows.
 *
 * Each declaration cites the interface of the reference project (ChenNan1996/PCF-NAT) that it
 * replaces, as file:line inside that project.
 */
#ifndef NA1D_B200_H
#define NA1D_B200_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* element type of the 16-bit tensors */
#define NA1D_BF16 0 /* replaces the bf16_ana1d module, na1d_tensorcore/nattn.py:12-20 */
#define NA1D_FP16 1 /* replaces the fp16_ana1d module, na1d_tensorcore/nattn.py:21-29 */

/* status codes */
#define NA1D_OK 0
#define NA1D_ERR_NULL_POINTER (-1)   /* a required pointer is NULL */
#define NA1D_ERR_BAD_SHAPE (-2)      /* N,T,C <= 0, C % 8 != 0, C > 256, or a product overflows int32 */
#define NA1D_ERR_BAD_WINDOW (-3)     /* win <= 0, win > NA1D_MAX_WINDOW, left outside [0,win), dil <= 0 */
#define NA1D_ERR_BAD_DTYPE (-4)      /* dtype is neither NA1D_BF16 nor NA1D_FP16 */
#define NA1D_ERR_BAD_HEADS (-5)      /* heads <= 0 or N % heads != 0 */
#define NA1D_ERR_MISALIGNED (-6)     /* a 16-bit tensor pointer is not 16-byte aligned */
#define NA1D_ERR_CUDA (-7)           /* a CUDA runtime/driver call failed; see na1d_last_cuda_error() */
#define NA1D_ERR_DEVICE_TIMEOUT (-8) /* a bounded wait inside a kernel expired (reported by na1d_device_status) */
#define NA1D_ERR_TOO_LARGE (-9)      /* problem exceeds a fixed capacity of the entry point */
#define NA1D_ERR_UNSUPPORTED (-10)   /* the requested kernel family / tiling cannot run this shape */
#define NA1D_ERR_BAD_DROPOUT (-12)   /* dropout probability outside [0,1) */
#define NA1D_ERR_BAD_STRIDE (-11)    /* a stride is not a positive multiple of 8 elements, or the token stride is below C */

#define NA1D_MAX_WINDOW 128 /* the reference asserts win <= 80, models/PCF_NATransformer.py:53 */

/* Human-readable text for a status code (host pointer, static storage). */
const char* na1d_status_string(int status);
/* cudaError_t value of the most recent failing CUDA call on this host thread (0 if none). */
int na1d_last_cuda_error(void);
/* Library version, major*100+minor. */
int na1d_version(void);

/* ------------------------------------------------------------------------------------------
 * Unfused pair: the six entry points of the reference extension, same argument meaning.
 * `dil` extends them (the reference kernels support dil == 1 only, na1d_tensorcore/nattn.py:130).
 * ---------------------------------------------------------------------------------------- */

/* attn[n,t,kk] = sum_c q[n,t,c] * k[n,j,c]            attn: (N,T,win) fp32; q,k: (N,T,C) 16-bit.
 * Replaces torch_ana_qk_forward, na1d_tensorcore/bf16_ana1d.cpp:8-27 (kernels
 * bf16_ana1d_kernel.cu:42-282; fp16 twin fp16_ana1d.cpp:8-27). */
int na1d_qk_forward(float* attn, const void* q, const void* k, int64_t N, int64_t T, int64_t C,
                    int64_t win, int64_t left, int64_t dil, int dtype, void* stream);

/* q_gd[n,t,c] = sum_kk attn_gd[n,t,kk] * k[n,j,c]      q_gd: (N,T,C) 16-bit.
 * Replaces torch_ana_q_backward, na1d_tensorcore/bf16_ana1d.cpp:29-41 (kernel :285-391). */
int na1d_q_backward(void* q_gd, const float* attn_gd, const void* k, int64_t N, int64_t T, int64_t C,
                    int64_t win, int64_t left, int64_t dil, int dtype, void* stream);

/* k_gd[n,j,c] = sum_kk attn_gd[n,t,kk] * q[n,t,c] over all (t,kk) whose neighbour is j.
 * Replaces torch_ana_k_backward, na1d_tensorcore/bf16_ana1d.cpp:43-55 (kernel :394-492). */
int na1d_k_backward(void* k_gd, const float* attn_gd, const void* q, int64_t N, int64_t T, int64_t C,
                    int64_t win, int64_t left, int64_t dil, int dtype, void* stream);

/* result[n,t,c] = sum_kk attn[n,t,kk] * v[n,j,c].
 * Replaces torch_ana_av_forward, na1d_tensorcore/bf16_ana1d.cpp:57-69. */
int na1d_av_forward(void* result, const float* attn, const void* v, int64_t N, int64_t T, int64_t C,
                    int64_t win, int64_t left, int64_t dil, int dtype, void* stream);

/* attn_gd[n,t,kk] = sum_c result_gd[n,t,c] * v[n,j,c].
 * Replaces torch_ana_a_backward, na1d_tensorcore/bf16_ana1d.cpp:71-90. */
int na1d_a_backward(float* attn_gd, const void* result_gd, const void* v, int64_t N, int64_t T, int64_t C,
                    int64_t win, int64_t left, int64_t dil, int dtype, void* stream);

/* v_gd[n,j,c] = sum_kk attn[n,t,kk] * result_gd[n,t,c] over all (t,kk) whose neighbour is j.
 * Replaces torch_ana_v_backward, na1d_tensorcore/bf16_ana1d.cpp:92-104. */
int na1d_v_backward(void* v_gd, const float* attn, const void* result_gd, int64_t N, int64_t T, int64_t C,
                    int64_t win, int64_t left, int64_t dil, int dtype, void* stream);

/* ------------------------------------------------------------------------------------------
 * Fused layer core: everything NAttention.forward does between the head split and the head
 * merge (models/PCF_NATransformer.py:141-150; MFA twin models/MFA_NATransformer.py:141-150):
 *   s[kk] = scale * q[t].k[j] + rpb[h,kk] + (masked ? -100 : 0);  p = softmax(s);  o = sum p[kk] v[j]
 *   masked = j outside [0,T)  or  j >= valid_len[b]  or  t >= valid_len[b]      (:87-116)
 * The fp32 (N,T,win) tensor of the unfused pair never exists in memory.
 * ---------------------------------------------------------------------------------------- */

/* o: (N,T,C) 16-bit; lse: (N,T) fp32 = log sum_kk exp(s[kk]) (kept for the backward pass; may be NULL);
 * rpb: (heads,win) fp32 or NULL; valid_len: (N/heads) int32 or NULL (= no padding). */
int na1d_fused_forward(void* o, float* lse, const void* q, const void* k, const void* v,
                       const float* rpb, const int32_t* valid_len, int64_t N, int64_t heads, int64_t T,
                       int64_t C, int64_t win, int64_t left, int64_t dil, float scale, int dtype,
                       void* stream);

/* Gradients of na1d_fused_forward. dq,dk,dv: (N,T,C) 16-bit. d_rpb: (heads,win) fp32, ACCUMULATED
 * into (caller zeroes it), or NULL. delta_ws: caller-provided scratch of N*T fp32. The CUDA-core
 * kernels keep the row sums of d_o*o there (written by a pre-pass, read by the main kernel); the
 * others need no such pre-pass: every CTA adds its partial d_rpb to the result with atomics at
 * its end. With NA1D_BIAS_GRAD_ROWS=1 in the environment the shapes that the tcgen05 kernels take stay with
 * them when d_rpb is wanted, and these write one partial row per CTA to delta_ws, summed in a fixed order by a
 * second small kernel.
 * Replaces the autograd chain AV.backward -> softmax backward -> QK.backward,
 * na1d_tensorcore/nattn.py:46-54 and :69-78. */
int na1d_fused_backward(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q,
                        const void* k, const void* v, const void* o, const float* lse, const float* rpb,
                        const int32_t* valid_len, float* delta_ws, int64_t N, int64_t heads, int64_t T,
                        int64_t C, int64_t win, int64_t left, int64_t dil, float scale, int dtype,
                        void* stream);

/* Floats that na1d_fused_backward needs behind delta_ws for a shape: N * T, or 0 where it does not touch them (delta_ws may then be any
 * pointer but NULL). Host-only. The answer is that of the kernels the call would run now: it holds while the family override
 * (na1d_set_kernel_family) is the same and follows NA1D_BIAS_GRAD_ROWS, which a process reads once. */
int64_t na1d_fused_backward_workspace_floats(int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                                             int dtype, int has_bias, int wants_bias_grad);
/* Zeros `bytes` of device memory (a bias gradient before the call that adds to it). */
int na1d_zero(void* p, int64_t bytes, void* stream);

/* Backward pass for callers that must not allocate device memory and have no spare buffer to lend.
 * (No counterpart in the reference project: its Python layer allocates every tensor with torch.)
 *
 * Who needs it: a host that drives this library from a place where device allocation is forbidden or
 * simply unavailable -- a serving or training loop whose memory pool is frozen after start-up, a thread
 * that is between cudaStreamBeginCapture and cudaStreamEndCapture, or a plain C/C++ runtime that hands
 * a plug-in fixed input/output buffers and no allocator handle. na1d_fused_backward asks such a caller
 * for an N*T-float workspace (delta_ws) it cannot produce. This variant takes the same inputs and
 * outputs but keeps that workspace inside the library, in a fixed device array.
 *
 * Same results as na1d_fused_backward with the CUDA-core kernels (it always runs those: they are the
 * backward kernels that use the workspace). Limits and rules:
 *   - N*T <= NA1D_STATIC_SCRATCH_ROWS, otherwise NA1D_ERR_TOO_LARGE is returned and nothing is launched.
 *     The array (NA1D_STATIC_SCRATCH_ROWS floats = 4 MiB) exists once per GPU that loads the library and
 *     stays resident until the process exits.
 *   - It calls no cudaMalloc/cudaFree and no allocating library routine, on any call.
 *   - The first call on each device looks up the array's device address (cudaGetSymbolAddress, with that
 *     device current). Make that first call outside any stream capture.
 *   - All calls on one device share the array. Every call overwrites the part it uses before reading
 *     it, so nothing has to be cleared between calls -- but two calls whose kernels can overlap on the
 *     GPU (different streams, no dependency) would race on it; order them on one stream or with events.
 *   - d_rpb, when given, is accumulated into exactly as in na1d_fused_backward (the caller zeroes it).
 */
#define NA1D_STATIC_SCRATCH_ROWS (1 << 20)
int na1d_fused_backward_static(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q,
                               const void* k, const void* v, const void* o, const float* lse,
                               const float* rpb, const int32_t* valid_len, int64_t N, int64_t heads,
                               int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, float scale,
                               int dtype, void* stream);

/* ------------------------------------------------------------------------------------------
 * Strided forms of the fused pair: q, k, v, o (and the gradients) may be views with arbitrary batch / head / token
 * strides, so that the head split and merge around the operator need no copies. Each `*_strides` argument is a HOST
 * pointer to three int64 element strides {batch, head, token} of a tensor addressed as [batch][head][token][channel]
 * (channel stride 1): a dense (N,T,C) tensor has {heads*T*C, T*C, C}; the q slice of a packed projection output
 * (batch, T, 3, heads, C) has {T*3*heads*C, C, 3*heads*C} and starts at the packed tensor's base (k: + heads*C
 * elements, v: + 2*heads*C); an output laid out (batch, T, heads, C) has {T*heads*C, C, heads*C}. Strides must be
 * positive multiples of 8 elements and pointers 16-byte aligned (NA1D_ERR_BAD_STRIDE / NA1D_ERR_MISALIGNED otherwise);
 * output views must not overlap themselves or each other. lse stays dense (N,T). These calls run the tcgen05 kernels on
 * the segmented tiling only (C in {16,32,64}, win <= 33, heads <= 32, T >= 2*dil; NA1D_ERR_UNSUPPORTED otherwise --
 * make dense copies and use the dense entry points then).
 * Replaces the head split of models/MFA_NATransformer.py:127-137 (and models/PCF_NATransformer.py:126-138), the head
 * merge of :151-152, and their autograd copies, together with the fused layer core above.
 * ---------------------------------------------------------------------------------------- */
/* 1 when the strided forward AND backward accept this shape (with a bias / with its gradient wanted), 0 when not,
 * negative for an invalid geometry. Host-only; lets a layer choose between the strided and the dense route up front. */
int na1d_fused_strided_supported(int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                                 int dtype, int has_bias, int wants_bias_grad);

int na1d_fused_forward_strided(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                               const int32_t* valid_len, const int64_t* o_strides, const int64_t* q_strides,
                               const int64_t* k_strides, const int64_t* v_strides, int64_t N, int64_t heads,
                               int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, float scale, int dtype,
                               void* stream);

/* scratch: `scratch_floats` fp32 of device memory for the per-CTA partial rows of d_rpb, which are written with
 * NA1D_BIAS_GRAD_ROWS=1 in the environment (148 * heads * win is always enough; with less, or NULL, and by default, the kernels
 * add to d_rpb with atomics). o is not needed. */
int na1d_fused_backward_strided(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q,
                                const void* k, const void* v, const float* lse, const float* rpb,
                                const int32_t* valid_len, float* scratch, int64_t scratch_floats,
                                const int64_t* dq_strides, const int64_t* dk_strides, const int64_t* dv_strides,
                                const int64_t* d_o_strides, const int64_t* q_strides, const int64_t* k_strides,
                                const int64_t* v_strides, int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win,
                                int64_t left, int64_t dil, float scale, int dtype, void* stream);

/* ------------------------------------------------------------------------------------------
 * Fused pair with attention dropout: p' = keep ? p / (1 - drop_p) : 0 on the normalised probabilities before the product
 * with v, as `self.attn_drop(attn)` between softmax and AV (models/PCF_NATransformer.py:149; the reference's configs set
 * the probability to 0). The keep decision of probability (row, kk) is a hash of (seed, dense row index n*T+t, kk) -- see
 * drop_hash in pcf_nat_b200/csrc/na1d_common.cuh; the backward re-derives the same mask from the same seed, nothing is
 * stored. lse is the log-sum-exp of the undropped logits. drop_p in [0,1); drop_p == 0 is the plain forward. Runs on the
 * tcgen05 kernels (flat tiling) only: NA1D_ERR_UNSUPPORTED for other shapes. `scratch` as in the strided backward.
 * ---------------------------------------------------------------------------------------- */
/* The keep decisions the dropout kernels derive, computed on the HOST into a HOST buffer of rows*win bytes
 * (keep_host[row*win + kk] = 1 if probability kk of dense row `row` = n*T+t is kept), for bit-exact checking of a
 * restatement of the hash. No device work. No counterpart in the reference (torch's dropout draws from the Philox stream). */
int na1d_dropout_keep_mask(uint8_t* keep_host, int64_t rows, int64_t win, float drop_p, uint64_t seed);

int na1d_fused_forward_dropout(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                               const int32_t* valid_len, int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win,
                               int64_t left, int64_t dil, float scale, float drop_p, uint64_t seed, int dtype,
                               void* stream);
int na1d_fused_backward_dropout(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q,
                                const void* k, const void* v, const float* lse, const float* rpb,
                                const int32_t* valid_len, float* scratch, int64_t scratch_floats, int64_t N,
                                int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                                float scale, float drop_p, uint64_t seed, int dtype, void* stream);

/* ------------------------------------------------------------------------------------------
 * The passes of a transformer block and of attentive statistics pooling that are not contractions (LayerNorm and residual,
 * GELU, column sums, rounding of parameters, pooling; models/PCF_NATransformer.py:228-303). 16-bit activations of `dtype`,
 * fp32 parameters and statistics. Rows are dense; D, F, C are multiples of 8, D <= 1024; every pointer 16-byte aligned.
 * `scratch` holds at least na1d_block_scratch_floats(rows, D, F) floats (column sums leave the CTAs as partial rows and
 * are added in a fixed order: the same bits from run to run).
 * ---------------------------------------------------------------------------------------- */
/* out (N): clamp(T - padding, 0, T); padding is int32 or (is64) int64, n_padding = N or 1 (one value for all). Any alignment. */
int na1d_valid_tokens(int32_t* out, const void* padding, int is64, int64_t n_padding, int64_t N, int64_t T, void* stream);
int64_t na1d_block_scratch_floats(int64_t rows, int64_t D, int64_t F);
/* y = LN(s) * w + b over rows of D; s = x, or with dx: s = x + dx, rounded and written to `sum`. mean, rstd: (rows) or NULL. */
int na1d_layer_norm_forward(void* y, void* sum, float* mean, float* rstd, const void* x, const void* dx, const float* w,
                            const float* b, int64_t rows, int64_t D, float eps, int dtype, void* stream);
/* dx = gradient of the normalised rows x + res (res may be NULL); sums (3, D): gradients of w and b, column sums of dx. */
int na1d_layer_norm_backward(void* dx, float* sums, float* scratch, const void* dy, const void* x, const float* mean,
                             const float* rstd, const float* w, const void* res, int64_t rows, int64_t D, int dtype, void* stream);
/* The same without the sums, whose partial results stay in `scratch`, and the sums of two such passes over as many rows of D. */
int na1d_layer_norm_backward_rows(void* dx, float* scratch, const void* dy, const void* x, const float* mean, const float* rstd, const float* w,
                                  const void* res, int64_t rows, int64_t D, int dtype, void* stream);
int na1d_layer_norm_sums(float* sums0, float* sums1, const float* scratch0, const float* scratch1, int64_t rows, int64_t D, void* stream);
/* y = x Phi(x) (the exact form), n elements (n a multiple of 8). */
int na1d_gelu_forward(void* y, const void* x, int64_t n, int dtype, void* stream);
/* dx = dy * d gelu(x), (rows, F); sums (F): column sums of dx. */
int na1d_gelu_backward(void* dx, float* sums, float* scratch, const void* dy, const void* x, int64_t rows, int64_t F, int dtype,
                       void* stream);
/* sums (F) = column sums of x (rows, F). */
int na1d_column_sums(float* sums, float* scratch, const void* x, int64_t rows, int64_t F, int dtype, void* stream);
/* A transformer block's MLP in one kernel: out = s + GELU(h w1^T + b1) w2^T + b2 (models/PCF_NATransformer.py:228-303). s, h, out
 * (rows, D), w1 (F, D), w2 (D, F) 16-bit, biases fp32; out has rows of ld >= D elements (a multiple of 8); D = 256, F a multiple of
 * 128 up to 1280. f (rows, F), 16-bit, or NULL: takes the hidden layer before GELU, for a backward pass. s and f are 32-byte
 * aligned.
 * `scratch`: na1d_mlp_scratch_floats floats (0: may be NULL; -1: not a size that this takes). */
int64_t na1d_mlp_scratch_floats(int64_t rows, int64_t D, int64_t F);
int na1d_mlp_forward(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const float* b1, const void* w2, const float* b2,
                     float* scratch, int64_t rows, int64_t D, int64_t F, int dtype, void* stream);
/* The same with the rounding points of its passes one by one: biases of `dtype`, GELU of the hidden layer's 16-bit values (which f takes).
 * Without f every sum over the hidden layer is one chain, as in a product that is not split, and scratch is not read (may be NULL). */
int na1d_mlp_forward_rounded(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const void* b1, const void* w2, const void* b2,
                             float* scratch, int64_t rows, int64_t D, int64_t F, int dtype, void* stream);
/* Its backward for the gradient d (rows, D) of out: df (rows, F) = (d w2) * gelu'(f), dh (rows, D) = df w1, g (rows, F) = gelu(f), all
 * 16-bit and, like f, 32-byte aligned; sizes and `scratch` as above. What the parameters need is left to na1d_projection_gradients. */
int na1d_mlp_backward(void* dh, void* df, void* g, const void* d, const void* f, const void* w1, const void* w2, float* scratch, int64_t rows, int64_t D,
                      int64_t F, int dtype, void* stream);
/* Parameter gradients of `count` (at most 2) projections in one launch: d_w[i] (M[i], N[i]) = dy[i]^T x[i], d_b[i] (M[i]) = column
 * sums of dy[i]; dy[i] (rows, M[i]) and x[i] (rows, N[i]) 16-bit, results fp32 (out32) or of `dtype`, either may be NULL. Host arrays
 * of device pointers. Partial sums go through `scratch` and are added in a fixed order. */
int64_t na1d_projection_gradients_scratch(const int64_t* M, const int64_t* N, int count, int64_t rows);
int na1d_projection_gradients(void* const* d_w, void* const* d_b, const void* const* dy, const void* const* x, const int64_t* M,
                              const int64_t* N, int count, int64_t rows, float* scratch, int out32, int dtype, void* stream);
/* Rounds `count` fp32 tensors (DEVICE pointers in the HOST array src, n[i] elements) to 16 bits at out + dst[i] (elements,
 * multiples of 8; each slot is padded with zeros to a multiple of 8) in one launch; count <= NA1D_CAST_MAX. */
#define NA1D_CAST_MAX 16
int na1d_cast_parameters(void* out, const float* const* src, const int64_t* dst, const int64_t* n, int count, int dtype,
                         void* stream);
/* out[r * ld + c] = x[r, c] + dx[r, c] (dx may be NULL: a copy), 16-bit, rows of D inside wider rows of ld elements (multiples of
 * 8): a stage's output written straight into its slice of the concatenated features (models/PCF_NATransformer.py:440-455). */
int na1d_add_to_rows(void* out, int64_t ld, const void* x, const void* dx, int64_t rows, int64_t D, int dtype, void* stream);
/* (N, C, T) -> (N, T, C) (to_tokens) or (N, T, C) -> (N, C, T), 16-bit; C a multiple of 8, the (N, T, C) side 16-byte aligned.
 * Replaces the transposing copies around the channels-first layer, models/PCF_NATransformer.py:126-151. */
int na1d_transpose(void* out, const void* in, int64_t N, int64_t C, int64_t T, int to_tokens, int dtype, void* stream);
/* (batch, T, parts, heads, C) -> (parts, batch, heads, T, C) (to_dense) or back, 16-bit, C a multiple of 8: the head split and merge
 * around the dense entry points (models/PCF_NATransformer.py:126-138, 151) for shapes the strided ones do not take. */
int na1d_permute_heads(void* out, const void* in, int64_t batch, int64_t T, int64_t parts, int64_t heads, int64_t C, int to_dense,
                       void* stream);
/* A grouped 1x1 convolution (models/PCF_NATransformer.py:66-68) as one dense matrix: w (parts*C, C/groups) and b (parts*C or
 * NULL), fp32 (src32) or 16-bit, to out_w (parts*C, C) and out_b, 16-bit, zeros outside the group's columns. parts = 3 orders
 * the rows as (q|k|v, head, channel): row which*C + f is output channel ((f % (C/groups))*groups + f / (C/groups))*3 + which, the
 * channel shuffle and head split of :127-129. parts = 1 keeps the order. */
int na1d_pack_grouped(void* out_w, void* out_b, const void* w, const void* b, int src32, int64_t C, int64_t groups, int parts,
                      int dtype, void* stream);
/* The transposed step for gradients: dense (parts*C, C) and sums (parts*C or NULL), fp32, to d_w (parts*C, C/groups) and d_b (or
 * NULL), fp32 (dst32) or 16-bit. */
int na1d_unpack_grouped(void* d_w, void* d_b, const float* dense, const float* sums, int dst32, int64_t C, int64_t groups, int parts,
                        int dtype, void* stream);
/* out (N, 2C) fp32 = [mu, std] with a = softmax over T of logits (N, T, C), mu = sum a x, std = sqrt(max(sum a x^2 - mu^2,
 * floor)). x has rows of ldx >= C elements (a multiple of 8). stats (3, N, C), for the backward (may be NULL): the logits' maximum, 1 / sum exp, sum a x^2. N <= 65535. */
int na1d_stats_pool_forward(float* out, float* stats, const void* logits, const void* x, int64_t ldx, int64_t N, int64_t T,
                            int64_t C, float floor, int dtype, void* stream);
int na1d_stats_pool_backward(void* d_logits, void* dx, const float* d_out, const float* out, const float* stats,
                             const void* logits, const void* x, int64_t N, int64_t T, int64_t C,
                             float floor, int dtype, void* stream);

/* ------------------------------------------------------------------------------------------
 * Window index arithmetic as the kernels compute it, for bit-exact checking:
 * j_out[t,kk] = t + (kk-left)*dil (int32, (T,win)); in_range[t,kk] = 1 if 0 <= j < T else 0.
 * Restates the implicit pad+unfold indexing of models/PCF_NATransformer.py:158-165.
 * ---------------------------------------------------------------------------------------- */
int na1d_window_index(int32_t* j_out, uint8_t* in_range, int64_t T, int64_t win, int64_t left,
                      int64_t dil, void* stream);

/* Which kernel family the fused entry points would pick for a shape (16-channel rows, and 32-channel rows in some
 * forwards, run on the marching kernels, na1d_march.cu, and report the family that otherwise takes the shape): 0 = the general kernels (warp-level matrix
 * instructions up to 128 channels, CUDA-core kernels above),
 * 1 = tcgen05/TMA kernels. Host-only query, no device work. The answer assumes one head, no bias and
 * no bias gradient: more than 32 heads, or 64-channel rows with an effective window above 17 together
 * with a bias of several heads or its gradient (no shared memory left for them), still move a call
 * to the CUDA-core kernels. */
int na1d_fused_kernel_family(int64_t N, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                             int dtype, int backward);

/* As na1d_fused_kernel_family, but tells the two tilings of the tcgen05 kernels apart: 0 = CUDA-core kernels,
 * 1 = tcgen05 on the flat tiling (tiles over the dense (N*T, C) matrix; dilation 1, or a power of two with
 * (win-1)*dil+1 <= 33), 2 = tcgen05 on the segmented tiling (tiles inside one residue class t = r mod dil of one
 * sequence: every dilation; also what the strided entry points run). Mirrors the tile heuristics of the reference's
 * launchers, na1d_tensorcore/bf16_ana1d_kernel.cu:495-580. */
int na1d_fused_kernel_tiling(int64_t N, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                             int dtype, int backward);

/* Which kernels a dense fused call runs: 0 = CUDA cores, 1 = tcgen05 on the flat tiling, 2 = on the segmented tiling, 3 = the warp-level
 * matrix kernels, 4 = the marching kernels (as the numbers of na1d_set_kernel_family); negative = status code. Host-only. The two
 * queries above tell the tcgen05 and general kernels apart alone: which of them takes the shape where the marching ones do not. */
int na1d_fused_kernel_route(int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                            int dtype, int backward, int has_bias, int wants_bias_grad);

/* Force a kernel family for the fused entry points: -1 = automatic (default), 0 = CUDA-core,
 * 1 = tcgen05/TMA (the flat tiling wherever it can run, else the segmented one; for the unfused entry points: also
 * where the automatic choice would take a CUDA-core kernel), 2 = what the strided entry points run: the segmented tiling, or the
 * marching kernels where those stand for it, 5 = tcgen05/TMA on the segmented tiling and nothing else, 3 = the warp-level matrix
 * kernels wherever they can run (up to 128 channels), else CUDA-core, 4 = the marching kernels where they can run (windows up
 * to 33; fused entry points at 16 channels, forward at 32 too, unfused ones at 16, 32 and 64), else as 3. Process-wide;
 * meant for tests and benchmarks. Returns the previous setting. */
int na1d_set_kernel_family(int family);

/* Hits and misses of the library's cache of encoded TMA tensor maps since the process started (the cache is keyed by
 * pointer, extents, strides, box and element type; its only global state, behind a lock). Host-only.
 * No counterpart in the reference (its kernels take raw pointers). */
int na1d_tensor_map_cache_stats(int64_t* hits, int64_t* misses);

/* Synchronises the device, then returns and clears the device-side status word: 0 = every bounded
 * wait inside the tcgen05 kernels completed, otherwise NA1D_ERR_DEVICE_TIMEOUT. */
int na1d_device_status(void);

#ifdef __cplusplus
}
#endif
#endif /* NA1D_B200_H */
