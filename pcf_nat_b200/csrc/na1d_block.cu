// Row and column kernels around the projections of a transformer block and of the statistics pooling: residual add +
// LayerNorm, GELU, their backward passes with the parameter and bias gradients (column sums) taken in the same pass, the
// rounding of a block's fp32 parameters to 16 bits in one launch, and attentive statistics pooling.
//
// All of them are bound by HBM: every 16-bit activation is read once and every result written once, all arithmetic is fp32.
// A lane owns 8 adjacent columns (one 16-byte access), a warp 256 columns of one row. Column sums stay in the lane's
// registers over all rows of its CTA, meet in shared memory once, and leave as one fp32 row per CTA that a second small
// kernel adds up in a fixed order: no atomics, the same bits from run to run.
#include "../../include/na1d_b200.h"
#include "na1d_internal.h"
#include "na1d_gelu.cuh"

namespace na1d {
namespace {

constexpr int kWarps = 8, kRowThreads = kWarps * 32;

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
using tc::fast_exp2;
using tc::fast_rcp;
template <typename E> __device__ __forceinline__ void load8(const E* p, float* f) {
    Cvt<E>::unpack(*reinterpret_cast<const uint4*>(p), f);
}
template <typename E> __device__ __forceinline__ void store8(E* p, const float* f) { *reinterpret_cast<uint4*>(p) = Cvt<E>::pack(f); }
// through 16 bits and back: what a reader of the stored tensor sees
template <typename E> __device__ __forceinline__ void round8(float* f) {
    const uint4 u = Cvt<E>::pack(f);
    Cvt<E>::unpack(u, f);
}
__device__ __forceinline__ void load8f(const float* p, float* f) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// ---------------------------------------------------------------- LayerNorm
// R values per lane, each summed over the warp: the first steps halve the values a lane carries on with, the totals come back to all
// lanes (R = 4: 6 + 4 exchanges in place of 20, in five steps that do not wait for one another)
template <int R> __device__ __forceinline__ void warp_sums(float (&v)[R], int lane) {
    static_assert(R == 1 || R == 2 || R == 4, "rows at a time");
#pragma unroll
    for (int w = R / 2; w > 0; w >>= 1) {
        const bool up = lane & (w * (32 / R));
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const float keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w * (32 / R));
        }
    }
    float t = v[0];
#pragma unroll
    for (int o = 16 / R; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = R == 1 ? t : __shfl_sync(0xffffffffu, t, i * (32 / R));
}

// y = LN(s) w + b with s = x, or s = round(x + dx) written to `sum` (the residual stream): R rows of a warp at a time, which stay in
// registers (mean first, then the centred squares) while the next R are on their way.
// 153600 rows of 256, with / without the addition: 55 / 39 us a row at a time (its loads, a sum over the warp and again: too few bytes in
// flight without the second input), 54 / 28 us with four (49 / 24 of HBM time). 231 + 37 us by the framework's kernels.
template <typename E, int CH, int R, bool ADD>
__global__ void __launch_bounds__(kRowThreads) ln_fwd_kernel(E* __restrict__ y, E* __restrict__ sum, float* __restrict__ mean,
                                                             float* __restrict__ rstd, const E* __restrict__ x,
                                                             const E* __restrict__ dx, const float* __restrict__ w,
                                                             const float* __restrict__ b, int rows, int D, float eps) {
    const int lane = threadIdx.x & 31;
    const float inv_d = 1.f / (float)D;
    uint4 nx[R][CH], nd[R][ADD ? CH : 1];
    auto fetch = [&](int row) {
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int col = c * 256 + lane * 8;
                nx[u][c] = make_uint4(0u, 0u, 0u, 0u);
                if (ADD) nd[u][ADD ? c : 0] = make_uint4(0u, 0u, 0u, 0u);
                if (row + u < rows && col < D) {
                    nx[u][c] = *reinterpret_cast<const uint4*>(x + (size_t)(row + u) * D + col);
                    if (ADD) nd[u][ADD ? c : 0] = *reinterpret_cast<const uint4*>(dx + (size_t)(row + u) * D + col);
                }
            }
    };
    const int step = gridDim.x * kWarps * R;
    int row = (blockIdx.x * kWarps + (threadIdx.x >> 5)) * R;
    fetch(row);
    for (; row < rows; row += step) {
        float v[R][CH][8], mu[R], rs[R];
#pragma unroll
        for (int u = 0; u < R; ++u) {
            mu[u] = 0.f;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int col = c * 256 + lane * 8;
                Cvt<E>::unpack(nx[u][c], v[u][c]);
                if (ADD) {
                    float r[8];
                    Cvt<E>::unpack(nd[u][ADD ? c : 0], r);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[u][c][i] += r[i];
                    round8<E>(v[u][c]);
                    if (row + u < rows && col < D) store8(sum + (size_t)(row + u) * D + col, v[u][c]);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) mu[u] += v[u][c][i];
            }
        }
        fetch(row + step);
        warp_sums<R>(mu, lane);
#pragma unroll
        for (int u = 0; u < R; ++u) {
            mu[u] *= inv_d;
            rs[u] = 0.f;
#pragma unroll
            for (int c = 0; c < CH; ++c)
                if (c * 256 + lane * 8 < D) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) rs[u] = fmaf(v[u][c][i] - mu[u], v[u][c][i] - mu[u], rs[u]);
                }
        }
        warp_sums<R>(rs, lane);
#pragma unroll
        for (int u = 0; u < R; ++u) rs[u] = rsqrtf(fmaf(rs[u], inv_d, eps));
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int col = c * 256 + lane * 8;
            if (col < D) {
                float wf[8], bf[8];
                load8f(w + col, wf);
                load8f(b + col, bf);
#pragma unroll
                for (int u = 0; u < R; ++u) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[u][c][i] = fmaf((v[u][c][i] - mu[u]) * rs[u], wf[i], bf[i]);
                    if (row + u < rows) store8(y + (size_t)(row + u) * D + col, v[u][c]);
                }
            }
        }
        if (mean && lane == 0) {
#pragma unroll
            for (int u = 0; u < R; ++u)
                if (row + u < rows) { mean[row + u] = mu[u]; rstd[row + u] = rs[u]; }
        }
    }
}

// Adds up the warps' column sums (K sums of 8 columns per lane and chunk) through shared memory and writes the CTA's row of
// partial sums: part[((cta * K) + k) * D + column].
template <int K, int CH>
__device__ __forceinline__ void cta_column_sums(float (&acc)[K][CH][8], float* part, int cta, int D, int col0) {
    __shared__ float sm[kWarps][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 8; ++i) sm[warp][i * 32 + lane] = acc[k][c][i];   // conflict-free: column 8 lane + i at i*32 + lane
            __syncthreads();
            const int col = col0 + c * 256 + threadIdx.x, at = (threadIdx.x & 7) * 32 + (threadIdx.x >> 3);
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < kWarps; ++q) s += sm[q][at];
            if (col < D) part[((size_t)cta * K + k) * D + col] = s;
        }
}

// out[i] = sum over g of part[g * n + i], in a fixed order: 32 warps share the rows of a group of 32 columns (at most 444 rows:
// 14 independent loads a thread). One launch adds up to two arrays (a block's two LayerNorms: 4 us each, and the gap between launches).
struct PartialSums {
    float* out[2];
    const float* part[2];
};
__global__ void __launch_bounds__(1024) partial_sum_kernel(const PartialSums a, int n, int groups) {
    float* __restrict__ out = a.out[blockIdx.y];
    const float* __restrict__ part = a.part[blockIdx.y];
    __shared__ float sm[32][33];
    const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < n) {
#pragma unroll 8
        for (int g = sub; g < groups; g += 32) s += __ldg(part + (size_t)g * n + i);
    }
    sm[sub][lane] = s;
    __syncthreads();
    const float t = warp_sum(sm[lane][sub]);   // warp q adds up column q
    if (lane == 0 && blockIdx.x * 32 + sub < n) out[blockIdx.x * 32 + sub] = t;
}

// dx = rstd (g - mean(g) - xhat mean(g xhat)) + res with g = dy w, and the column sums of dy xhat (weight gradient), dy (bias
// gradient) and dx as stored (the bias gradient of the projection whose output was added to the residual stream).
// 38400 rows of 256: 35 us (input gradient) + 173 us (parameter gradients) + 47 us (bias gradient) before, 22 us here (12 us of
// HBM time; loading the next row ahead, as the forward does, measured 23 us).
template <typename E, int CH>
__global__ void __launch_bounds__(kRowThreads) ln_bwd_kernel(E* __restrict__ dx, float* __restrict__ part, const E* __restrict__ dy,
                                                             const E* __restrict__ x, const float* __restrict__ mean,
                                                             const float* __restrict__ rstd, const float* __restrict__ w,
                                                             const E* __restrict__ res, int rows, int D) {
    const int lane = threadIdx.x & 31;
    const float inv_d = 1.f / (float)D;
    float acc[3][CH][8], wf[CH][8];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int col = c * 256 + lane * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) { acc[0][c][i] = acc[1][c][i] = acc[2][c][i] = 0.f; wf[c][i] = 0.f; }
        if (col < D) load8f(w + col, wf[c]);
    }
    for (int row = blockIdx.x * kWarps + (threadIdx.x >> 5); row < rows; row += gridDim.x * kWarps) {
        const size_t base = (size_t)row * D;
        const float mu = __ldg(mean + row), rs = __ldg(rstd + row);
        float g[CH][8], h[CH][8], r[CH][8], a = 0.f, b = 0.f;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int col = c * 256 + lane * 8;
#pragma unroll
            for (int i = 0; i < 8; ++i) { g[c][i] = 0.f; h[c][i] = mu; r[c][i] = 0.f; }
            if (col < D) {
                load8(dy + base + col, g[c]);
                load8(x + base + col, h[c]);
                if (res) load8(res + base + col, r[c]);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                h[c][i] = (h[c][i] - mu) * rs;
                acc[0][c][i] = fmaf(g[c][i], h[c][i], acc[0][c][i]);
                acc[1][c][i] += g[c][i];
                g[c][i] *= wf[c][i];
                a += g[c][i];
                b = fmaf(g[c][i], h[c][i], b);
            }
        }
        a = warp_sum(a) * inv_d;
        b = warp_sum(b) * inv_d;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int col = c * 256 + lane * 8;
            if (col < D) {
                float o[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = fmaf(rs, g[c][i] - a - h[c][i] * b, r[c][i]);
                const uint4 u = Cvt<E>::pack(o);
                *reinterpret_cast<uint4*>(dx + base + col) = u;
                Cvt<E>::unpack(u, o);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[2][c][i] += o[i];
            }
        }
    }
    cta_column_sums<3, CH>(acc, part, blockIdx.x, D, 0);
}

// ---------------------------------------------------------------- GELU (exact form x Phi(x), na1d_gelu.cuh) and column sums
__device__ __forceinline__ float gelu(float x) {
    float c, e;
    phi(x, c, e);
    return x * c;
}

template <typename E>
__global__ void __launch_bounds__(256) gelu_fwd_kernel(E* __restrict__ y, const E* __restrict__ x, long long chunks) {
    // four independent 16-byte loads in flight per thread
    const long long stride = (long long)gridDim.x * 256;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < chunks; i += 4 * stride) {
        uint4 u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + k * stride < chunks) u[k] = reinterpret_cast<const uint4*>(x)[i + k * stride];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + k * stride < chunks) {
                float f[8];
                Cvt<E>::unpack(u[k], f);
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = gelu(f[j]);
                reinterpret_cast<uint4*>(y)[i + k * stride] = Cvt<E>::pack(f);
            }
    }
}

// Column sums of a (rows, F) matrix with leading dimension F; GELU: the matrix is dx = dy gelu'(x), which is written too
// (38400 x 1024: 63 us backward + 47 us bias gradient before, 52 us here, 37 us of HBM time).
// CTA (bx, by): columns 256 bx .. +255, rows by * 8 + warp, stepping by 8 gridDim.y.
template <typename E, bool GELU>
__global__ void __launch_bounds__(kRowThreads) column_kernel(E* __restrict__ dx, float* __restrict__ part, const E* __restrict__ dy,
                                                             const E* __restrict__ x, int rows, int F) {
    const int lane = threadIdx.x & 31, col = blockIdx.x * 256 + lane * 8;
    float acc[1][1][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[0][0][i] = 0.f;
    constexpr int U = 4;
    const int step = gridDim.y * kWarps;
    if (col < F)
        for (int row = blockIdx.y * kWarps + (threadIdx.x >> 5); row < rows; row += U * step) {
            uint4 a[U], b[U];
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (row + k * step < rows) {
                    const size_t at = (size_t)(row + k * step) * F + col;
                    a[k] = *reinterpret_cast<const uint4*>(dy + at);
                    if constexpr (GELU) b[k] = *reinterpret_cast<const uint4*>(x + at);
                }
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (row + k * step < rows) {
                    float g[8];
                    Cvt<E>::unpack(a[k], g);
                    if constexpr (GELU) {
                        float v[8];
                        Cvt<E>::unpack(b[k], v);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float c, e;
                            phi(v[i], c, e);
                            g[i] *= fmaf(v[i] * 0.3989422804014327f, e, c);   // Phi(x) + x phi(x)
                        }
                        const uint4 u = Cvt<E>::pack(g);
                        *reinterpret_cast<uint4*>(dx + (size_t)(row + k * step) * F + col) = u;
                        Cvt<E>::unpack(u, g);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[0][0][i] += g[i];
                }
        }
    cta_column_sums<1, 1>(acc, part, blockIdx.y, F, blockIdx.x * 256);
}

// ---------------------------------------------------------------- parameters to 16 bits, several tensors in one launch
struct CastList {
    const float* src[NA1D_CAST_MAX];
    long long dst[NA1D_CAST_MAX];   // element offset in the packed output, a multiple of 8
    int n[NA1D_CAST_MAX];
    int first[NA1D_CAST_MAX + 1];   // first CTA of each tensor
    int count;
};
constexpr int kCastPerCta = 256 * 8;
template <typename E> __global__ void __launch_bounds__(256) cast_kernel(E* __restrict__ out, const __grid_constant__ CastList L) {
    int k = 0;
    while (k + 1 < L.count && (int)blockIdx.x >= L.first[k + 1]) ++k;
    const int i0 = ((int)blockIdx.x - L.first[k]) * kCastPerCta + threadIdx.x * 8, n = L.n[k];
    if (i0 >= n) return;
    const float* s = L.src[k] + i0;
    float f[8];
    if (i0 + 8 <= n && (reinterpret_cast<uintptr_t>(s) & 15u) == 0) {
        load8f(s, f);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = i0 + i < n ? s[i] : 0.f;
    }
    *reinterpret_cast<uint4*>(out + L.dst[k] + i0) = Cvt<E>::pack(f);   // the slot of each tensor is padded to 8 elements
}

// out row r (ld elements apart) = x + dx: one 16-byte unit per thread and step
template <typename E>
__global__ void __launch_bounds__(256) add_to_rows_kernel(E* __restrict__ out, long long ld, const E* __restrict__ x, const E* __restrict__ dx, int D,
                                                          long long chunks) {
    const int per_row = D / 8;
    const long long stride = (long long)gridDim.x * 256;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < chunks; i += stride) {
        float a[8], b[8];
        uint4 u = reinterpret_cast<const uint4*>(x)[i];
        if (dx) {
            Cvt<E>::unpack(u, a);
            load8(dx + i * 8, b);
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] += b[k];
            u = Cvt<E>::pack(a);
        }
        const long long row = i / per_row;
        *reinterpret_cast<uint4*>(out + row * ld + (i - row * per_row) * 8) = u;
    }
}

// valid tokens of each utterance from its padding: one launch for what four elementwise ones did
__global__ void __launch_bounds__(256) valid_tokens_kernel(int* __restrict__ out, const void* __restrict__ padding, bool is64, int n_padding, int N, int T) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= N) return;
    const int at = n_padding == 1 ? 0 : i;
    const long long v = T - (is64 ? static_cast<const long long*>(padding)[at] : (long long)static_cast<const int*>(padding)[at]);
    out[i] = (int)(v < 0 ? 0 : v > T ? T : v);
}

// ---------------------------------------------------------------- channels-first layers: transposes and grouped weights
// A 64-channel x 64-token tile through shared memory, as words of two tokens of one channel: the token side is read or written in such
// pairs (4 bytes) where the rows allow it (an even token count, an even base), the channel side in 16-byte units of two tokens
// at a time, so that a value is never moved alone (tokens as single 16-bit values of a [token][channel] tile: 23 us to tokens, 17 back).
// The token side has no bank conflicts with rows of 33 words, the channel side two-way ones.
// 512 x 256 x 150: 14 and 15 us in a series, 12 us of HBM time; 64 x 256 x 997: 24 and 14 (27, 18); 72 us per copy of the framework.
constexpr int kTile = 64, kTilePitch = 33;
template <bool TO_TOKENS, bool PAIRS>
__global__ void __launch_bounds__(256) transpose_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ in, int C, int T) {
    __shared__ uint32_t sm[kTile * kTilePitch];   // [channel][pair of tokens]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = blockIdx.x * kTile, t0 = blockIdx.y * kTile;
    const size_t base = (size_t)blockIdx.z * C * T;
    // channel-major side: lane -> two tokens, warp -> channels warp, warp + 8, ...; token-major side: eight channels of two tokens
    const int t = t0 + 2 * lane, cu = (threadIdx.x & 7) * 8, pair = threadIdx.x >> 3, tok = t0 + 2 * pair;
    if constexpr (TO_TOKENS) {
        uint32_t v[kTile / 8];
#pragma unroll
        for (int i = 0; i < kTile / 8; ++i) {
            const int c = warp + 8 * i;
            v[i] = 0u;
            if (c0 + c < C && t < T) {
                const size_t at = base + (size_t)(c0 + c) * T + t;
                v[i] = PAIRS ? __ldg(reinterpret_cast<const uint32_t*>(in + at)) : (uint32_t)in[at] | (t + 1 < T ? (uint32_t)in[at + 1] << 16 : 0u);
            }
        }
#pragma unroll
        for (int i = 0; i < kTile / 8; ++i) sm[(warp + 8 * i) * kTilePitch + lane] = v[i];
        __syncthreads();
        if (tok < T && c0 + cu < C) {
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = sm[(cu + e) * kTilePitch + pair];
            uint4 first, second;
            first.x = __byte_perm(w[0], w[1], 0x5410); first.y = __byte_perm(w[2], w[3], 0x5410);
            first.z = __byte_perm(w[4], w[5], 0x5410); first.w = __byte_perm(w[6], w[7], 0x5410);
            second.x = __byte_perm(w[0], w[1], 0x7632); second.y = __byte_perm(w[2], w[3], 0x7632);
            second.z = __byte_perm(w[4], w[5], 0x7632); second.w = __byte_perm(w[6], w[7], 0x7632);
            *reinterpret_cast<uint4*>(out + base + (size_t)tok * C + c0 + cu) = first;
            if (tok + 1 < T) *reinterpret_cast<uint4*>(out + base + (size_t)(tok + 1) * C + c0 + cu) = second;
        }
    } else {
        if (tok < T && c0 + cu < C) {
            const size_t unit_at = base + (size_t)tok * C + c0 + cu;
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(in + unit_at));
            const uint4 b = tok + 1 < T ? __ldg(reinterpret_cast<const uint4*>(in + unit_at + C)) : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t f[4] = {a.x, a.y, a.z, a.w}, s[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sm[(cu + 2 * e) * kTilePitch + pair] = __byte_perm(f[e], s[e], 0x5410);
                sm[(cu + 2 * e + 1) * kTilePitch + pair] = __byte_perm(f[e], s[e], 0x7632);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kTile / 8; ++i) {
            const int c = warp + 8 * i;
            if (c0 + c >= C || t >= T) continue;
            const uint32_t v = sm[c * kTilePitch + lane];
            uint16_t* at = out + base + (size_t)(c0 + c) * T + t;
            if constexpr (PAIRS) {
                *reinterpret_cast<uint32_t*>(at) = v;
            } else {
                at[0] = (uint16_t)v;
                if (t + 1 < T) at[1] = (uint16_t)(v >> 16);
            }
        }
    }
}

// Head split or merge: CTA (x, h, z) moves 256 of the T * C / 8 16-byte units of head h of part-and-batch z; the dense side is
// contiguous, the packed side comes in pieces of C channels.
__global__ void __launch_bounds__(256) permute_heads_kernel(uint4* __restrict__ out, const uint4* __restrict__ in, int batch, int T, int parts, int heads,
                                                           int units, bool to_dense) {
    const int i = blockIdx.x * 256 + threadIdx.x, h = blockIdx.y;
    if (i >= T * units) return;
    const int t = i / units, c = i - t * units;
    for (int z = blockIdx.z; z < batch * parts; z += gridDim.z) {
        const int p = z / batch, b = z - p * batch;
        const long long dense = ((long long)z * heads + h) * T * units + i;
        const long long packed = ((((long long)b * T + t) * parts + p) * heads + h) * units + c;
        if (to_dense) out[dense] = __ldg(in + packed);
        else out[packed] = __ldg(in + dense);
    }
}

// convolution output channel of row r of the dense matrix
__device__ __forceinline__ int grouped_channel(int r, int C, int groups, int parts) {
    if (parts == 1) return r;
    const int which = r / C, f = r - which * C, P = C / groups;
    return ((f % P) * groups + f / P) * 3 + which;
}
// one CTA per row of the dense matrix
template <typename E, typename S>
__global__ void __launch_bounds__(128) pack_grouped_kernel(E* __restrict__ out_w, E* __restrict__ out_b, const S* __restrict__ w,
                                                           const S* __restrict__ b, int C, int groups, int parts) {
    const int r = blockIdx.x, P = C / groups, ch = grouped_channel(r, C, groups, parts), first = ch / (parts * P) * P;
    for (int c = threadIdx.x; c < C; c += 128)
        out_w[(size_t)r * C + c] = c >= first && c < first + P ? (E)(float)w[(size_t)ch * P + c - first] : (E)0.f;
    if (b && threadIdx.x == 0) out_b[r] = (E)(float)b[ch];
}
template <typename D>
__global__ void __launch_bounds__(128) unpack_grouped_kernel(D* __restrict__ d_w, D* __restrict__ d_b, const float* __restrict__ dense,
                                                             const float* __restrict__ sums, int C, int groups, int parts) {
    const int r = blockIdx.x, P = C / groups, ch = grouped_channel(r, C, groups, parts), first = ch / (parts * P) * P;
    if (d_w)
        for (int c = threadIdx.x; c < P; c += 128) d_w[(size_t)ch * P + c] = (D)dense[(size_t)r * C + first + c];
    if (d_b && threadIdx.x == 0) d_b[ch] = (D)sums[r];
}

// ---------------------------------------------------------------- attentive statistics pooling
// a = softmax over time of the logits; mu = sum a x, std = sqrt(max(sum a x^2 - mu^2, floor)), per channel. One pass: a lane
// keeps the running maximum and the three sums of its 8 channels; the CTA's warps share the time axis and meet in shared
// memory. Reads logits and x once (512 x 300 x 1536: 0.94 GB; the framework's chain of fp32 copies, strided softmax, products
// and sums took 6.2 ms there; 0.24 ms here, 0.15 ms of HBM time).
constexpr int kPoolWarps = 8;
template <typename E>
__global__ void __launch_bounds__(kPoolWarps * 32) pool_fwd_kernel(float* __restrict__ out, float* __restrict__ stats,
                                                                  const E* __restrict__ logits, const E* __restrict__ x, long long ldx,
                                                                  int T, int C, float floor_var) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = blockIdx.x * 256 + lane * 8;
    const size_t base = (size_t)blockIdx.y * T * C;
    float m[8], s[8], sx[8], sxx[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { m[i] = -INFINITY; s[i] = sx[i] = sxx[i] = 0.f; }
    if (col < C)
#pragma unroll 2
        for (int t = warp; t < T; t += kPoolWarps) {
            float l[8], v[8];
            load8(logits + base + (size_t)t * C + col, l);
            load8(x + ((size_t)blockIdx.y * T + t) * ldx + col, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float z = l[i];
                if (z > m[i]) {   // a new maximum: rescale (rare after the first steps)
                    const float r = fast_exp2((m[i] - z) * kLog2e);
                    s[i] *= r; sx[i] *= r; sxx[i] *= r;
                    m[i] = z;
                }
                // (an infinite logit gives NaN, as the softmax of it does; a logit of -inf next to finite ones gives 0)
                const float p = m[i] == -INFINITY && z == -INFINITY ? 0.f : fast_exp2((z - m[i]) * kLog2e);
                s[i] += p;
                const float px = p * v[i];
                sx[i] += px;
                sxx[i] = fmaf(px, v[i], sxx[i]);
            }
        }
    __shared__ float sm[4][kPoolWarps][256];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        sm[0][warp][i * 32 + lane] = m[i];
        sm[1][warp][i * 32 + lane] = s[i];
        sm[2][warp][i * 32 + lane] = sx[i];
        sm[3][warp][i * 32 + lane] = sxx[i];
    }
    __syncthreads();
    const int c = blockIdx.x * 256 + threadIdx.x, at = (threadIdx.x & 7) * 32 + (threadIdx.x >> 3);
    if (c >= C) return;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kPoolWarps; ++w) M = fmaxf(M, sm[0][w][at]);
    float S = 0.f, X = 0.f, XX = 0.f;
#pragma unroll
    for (int w = 0; w < kPoolWarps; ++w) {
        const float r = sm[0][w][at] == -INFINITY ? 0.f : fast_exp2((sm[0][w][at] - M) * kLog2e);
        S = fmaf(sm[1][w][at], r, S);
        X = fmaf(sm[2][w][at], r, X);
        XX = fmaf(sm[3][w][at], r, XX);
    }
    const float inv = 1.f / S, mu = X * inv, e2 = XX * inv;
    const float var = fmaf(-mu, mu, e2);
    float* o = out + (size_t)blockIdx.y * 2 * C;
    o[c] = mu;
    o[C + c] = sqrtf(var < floor_var ? floor_var : var);
    if (stats) {   // (3, N, C); the maximum and the sum apart: their logarithm's sum loses the sum next to a large maximum
        const size_t at3 = (size_t)blockIdx.y * C + c, plane = (size_t)gridDim.y * C;
        stats[at3] = M;
        stats[at3 + plane] = inv;
        stats[at3 + 2 * plane] = e2;
    }
}

// d_logits = a (q - sum a q) and dx = a (dm + 2 x dv) with q = x dm + x^2 dv, dv = d_std / (2 std) where the variance is not at
// its floor, dm = d_mu - 2 mu dv. The inner sum is mu dm + E[x^2] dv: known per channel, so this is one pass.
template <typename E>
__global__ void __launch_bounds__(kPoolWarps * 32) pool_bwd_kernel(E* __restrict__ d_logits, E* __restrict__ dx,
                                                                  const float* __restrict__ d_out, const float* __restrict__ out,
                                                                  const float* __restrict__ stats, const E* __restrict__ logits,
                                                                  const E* __restrict__ x, int T, int C, float floor_var) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = blockIdx.x * 256 + lane * 8;
    if (col >= C) return;
    const size_t base = (size_t)blockIdx.y * T * C, row = (size_t)blockIdx.y * C + col, row2 = (size_t)blockIdx.y * 2 * C + col;
    float top[8], inv[8], dm[8], dv[8], inner[8];
    {
        float mu[8], sd[8], gm[8], gs[8], e2[8];
        const size_t plane = (size_t)gridDim.y * C;
        load8f(stats + row, top);
        load8f(stats + row + plane, inv);
        load8f(stats + row + 2 * plane, e2);
        load8f(out + row2, mu);
        load8f(out + row2 + C, sd);
        load8f(d_out + row2, gm);
        load8f(d_out + row2 + C, gs);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float var = fmaf(-mu[i], mu[i], e2[i]);   // as the forward pass computed it
            dv[i] = var < floor_var ? 0.f : gs[i] * 0.5f / sd[i];
            dm[i] = gm[i] - 2.f * mu[i] * dv[i];
            inner[i] = mu[i] * dm[i] + e2[i] * dv[i];
        }
    }
#pragma unroll 2
    for (int t = blockIdx.z * kPoolWarps + warp; t < T; t += kPoolWarps * gridDim.z) {
        const size_t at = base + (size_t)t * C + col;
        float l[8], v[8];
        load8(logits + at, l);
        load8(x + at, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float a = fast_exp2((l[i] - top[i]) * kLog2e) * inv[i];
            const float xv = v[i];
            const float q = xv * fmaf(xv, dv[i], dm[i]);
            l[i] = a * (q - inner[i]);
            v[i] = a * fmaf(2.f * xv, dv[i], dm[i]);
        }
        store8(d_logits + at, l);
        store8(dx + at, v);
    }
}

// rows are shared out over the warps of at most per_sm CTAs per SM
int row_grid(long long rows, int per_sm) {
    const long long need = (rows + kWarps - 1) / kWarps, most = (long long)device_sm_count() * per_sm;
    return (int)(need < most ? need : most);
}

template <typename E>
cudaError_t ln_fwd(void* y, void* sum, float* mean, float* rstd, const void* x, const void* dx, const float* w, const float* b,
                   int rows, int D, float eps, cudaStream_t st) {
    // Four rows of a warp (0) where the rows fill the grid with that. A few rows are sooner done one to a warp: 2400 x 256 2.8 us with the
    // addition, 2.5 without (four: 3.2 and 2.6), 38400 x 128 12.1 with it (13.0); 153600 x 256 without it 28 (39). Grids, for 153600 rows:
    // 4 CTAs per SM at most for groups of four; one row at a time 512 channels 103 us with the addition and 60 without at 12 (108, 60
    // at 8; 115, 58 at 4), 768 channels 153 and 88 (153, 95; 167, 124), 1024 channels 198 and 112 (203, 123; 215, 136).
    const int ch = D <= 256 && rows >= (dx ? 1 << 16 : 1 << 15) ? 0 : (D + 255) / 256;
#define NA1D_LN(CH, R, ADD) ln_fwd_kernel<E, CH, R, ADD><<<row_grid((rows + R - 1) / R, R == 4 ? 4 : 12), kRowThreads, 0, st>>>((E*)y, (E*)sum, mean, rstd, (const E*)x, (const E*)dx, w, b, rows, D, eps)
#define NA1D_LN_C(ADD) switch (ch) { case 0: NA1D_LN(1, 4, ADD); break; case 1: NA1D_LN(1, 1, ADD); break; case 2: NA1D_LN(2, 1, ADD); break; case 3: NA1D_LN(3, 1, ADD); break; default: NA1D_LN(4, 1, ADD); }
    if (dx) { NA1D_LN_C(true) } else { NA1D_LN_C(false) }
#undef NA1D_LN_C
#undef NA1D_LN
    return cudaGetLastError();
}
cudaError_t add_partials(float* out, const float* part, int n, int groups, cudaStream_t st) {
    partial_sum_kernel<<<(n + 31) / 32, 1024, 0, st>>>(PartialSums{{out, nullptr}, {part, nullptr}}, n, groups);
    return cudaGetLastError();
}
template <typename E>
cudaError_t ln_bwd(void* dx, float* sums, float* part, const void* dy, const void* x, const float* mean, const float* rstd,
                   const float* w, const void* res, int rows, int D, cudaStream_t st) {
    const int grid = block_partial_rows(rows), ch = (D + 255) / 256;
#define NA1D_LN(CH) ln_bwd_kernel<E, CH><<<grid, kRowThreads, 0, st>>>((E*)dx, part, (const E*)dy, (const E*)x, mean, rstd, w, (const E*)res, rows, D)
    switch (ch) { case 1: NA1D_LN(1); break; case 2: NA1D_LN(2); break; case 3: NA1D_LN(3); break; default: NA1D_LN(4); }
#undef NA1D_LN
    if (cudaError_t e = cudaGetLastError()) return e;
    return sums ? add_partials(sums, part, 3 * D, grid, st) : cudaSuccess;
}
template <typename E, bool GELU>
cudaError_t columns(void* dx, float* sums, float* part, const void* dy, const void* x, int rows, int F, cudaStream_t st) {
    const int bx = (F + 255) / 256;
    int by = block_partial_rows(rows) / bx;
    if (by < 1) by = 1;
    column_kernel<E, GELU><<<dim3(bx, by), kRowThreads, 0, st>>>((E*)dx, part, (const E*)dy, (const E*)x, rows, F);
    if (cudaError_t e = cudaGetLastError()) return e;
    return add_partials(sums, part, F, by, st);
}

}  // namespace

// CTAs of a column-sum pass over `rows` rows, and so the rows of partial sums it needs room for
int block_partial_rows(long long rows) { return row_grid(rows, 3); }

cudaError_t block_valid_tokens(int* out, const void* padding, bool is64, int n_padding, int N, int T, cudaStream_t st) {
    valid_tokens_kernel<<<(N + 255) / 256, 256, 0, st>>>(out, padding, is64, n_padding, N, T);
    return cudaGetLastError();
}
cudaError_t block_ln_fwd(void* y, void* sum, float* mean, float* rstd, const void* x, const void* dx, const float* w, const float* b,
                         int rows, int D, float eps, int dtype, cudaStream_t st) {
    return dtype == 0 ? ln_fwd<__nv_bfloat16>(y, sum, mean, rstd, x, dx, w, b, rows, D, eps, st)
                      : ln_fwd<__half>(y, sum, mean, rstd, x, dx, w, b, rows, D, eps, st);
}
cudaError_t block_ln_bwd(void* dx, float* sums, float* part, const void* dy, const void* x, const float* mean, const float* rstd,
                         const float* w, const void* res, int rows, int D, int dtype, cudaStream_t st) {
    return dtype == 0 ? ln_bwd<__nv_bfloat16>(dx, sums, part, dy, x, mean, rstd, w, res, rows, D, st)
                      : ln_bwd<__half>(dx, sums, part, dy, x, mean, rstd, w, res, rows, D, st);
}
cudaError_t block_ln_sums(float* const* sums, const float* const* part, int rows, int D, cudaStream_t st) {
    partial_sum_kernel<<<dim3((3 * D + 31) / 32, 2), 1024, 0, st>>>(PartialSums{{sums[0], sums[1]}, {part[0], part[1]}}, 3 * D, block_partial_rows(rows));
    return cudaGetLastError();
}
cudaError_t block_gelu_fwd(void* y, const void* x, long long n, int dtype, cudaStream_t st) {
    const long long chunks = n / 8, need = (chunks + 1023) / 1024, most = (long long)device_sm_count() * 8;
    const int grid = (int)(need < most ? need : most);
    if (dtype == 0) gelu_fwd_kernel<<<grid, 256, 0, st>>>((__nv_bfloat16*)y, (const __nv_bfloat16*)x, chunks);
    else gelu_fwd_kernel<<<grid, 256, 0, st>>>((__half*)y, (const __half*)x, chunks);
    return cudaGetLastError();
}
cudaError_t block_gelu_bwd(void* dx, float* sums, float* part, const void* dy, const void* x, int rows, int F, int dtype, cudaStream_t st) {
    return dtype == 0 ? columns<__nv_bfloat16, true>(dx, sums, part, dy, x, rows, F, st) : columns<__half, true>(dx, sums, part, dy, x, rows, F, st);
}
cudaError_t block_column_sums(float* sums, float* part, const void* x, int rows, int F, int dtype, cudaStream_t st) {
    return dtype == 0 ? columns<__nv_bfloat16, false>(nullptr, sums, part, x, nullptr, rows, F, st)
                      : columns<__half, false>(nullptr, sums, part, x, nullptr, rows, F, st);
}
cudaError_t block_cast(void* out, const float* const* src, const int64_t* dst, const int64_t* n, int count, int dtype, cudaStream_t st) {
    CastList L;
    L.count = count;
    L.first[0] = 0;
    for (int i = 0; i < count; ++i) {
        L.src[i] = src[i];
        L.dst[i] = dst[i];
        L.n[i] = (int)n[i];
        L.first[i + 1] = L.first[i] + (int)((n[i] + kCastPerCta - 1) / kCastPerCta);
    }
    if (dtype == 0) cast_kernel<<<L.first[count], 256, 0, st>>>((__nv_bfloat16*)out, L);
    else cast_kernel<<<L.first[count], 256, 0, st>>>((__half*)out, L);
    return cudaGetLastError();
}
cudaError_t block_add_to_rows(void* out, long long ld, const void* x, const void* dx, int rows, int D, int dtype, cudaStream_t st) {
    const long long chunks = (long long)rows * (D / 8), need = (chunks + 255) / 256, most = (long long)device_sm_count() * 16;
    const int grid = (int)(need < most ? need : most);
    if (dtype == 0) add_to_rows_kernel<<<grid, 256, 0, st>>>((__nv_bfloat16*)out, ld, (const __nv_bfloat16*)x, (const __nv_bfloat16*)dx, D, chunks);
    else add_to_rows_kernel<<<grid, 256, 0, st>>>((__half*)out, ld, (const __half*)x, (const __half*)dx, D, chunks);
    return cudaGetLastError();
}
cudaError_t block_permute_heads(void* out, const void* in, int batch, int T, int parts, int heads, int C, bool to_dense, cudaStream_t st) {
    const int units = C / 8, z = batch * parts;
    const dim3 grid((T * units + 255) / 256, heads, z < 32768 ? z : 32768);
    permute_heads_kernel<<<grid, 256, 0, st>>>((uint4*)out, (const uint4*)in, batch, T, parts, heads, units, to_dense);
    return cudaGetLastError();
}
cudaError_t block_transpose(void* out, const void* in, int N, int C, int T, bool to_tokens, int dtype, cudaStream_t st) {
    const dim3 grid((C + kTile - 1) / kTile, (T + kTile - 1) / kTile, N);
    const bool pairs = T % 2 == 0 && (reinterpret_cast<uintptr_t>(to_tokens ? in : out) & 3u) == 0;
    uint16_t* o = (uint16_t*)out;
    const uint16_t* i = (const uint16_t*)in;
    if (to_tokens) { if (pairs) transpose_kernel<true, true><<<grid, 256, 0, st>>>(o, i, C, T); else transpose_kernel<true, false><<<grid, 256, 0, st>>>(o, i, C, T); }
    else { if (pairs) transpose_kernel<false, true><<<grid, 256, 0, st>>>(o, i, C, T); else transpose_kernel<false, false><<<grid, 256, 0, st>>>(o, i, C, T); }
    return cudaGetLastError();
}
cudaError_t block_pack_grouped(void* out_w, void* out_b, const void* w, const void* b, bool src32, int C, int groups, int parts, int dtype,
                               cudaStream_t st) {
    const int rows = parts * C;
    using B = __nv_bfloat16;
    if (dtype == 0) {
        if (src32) pack_grouped_kernel<<<rows, 128, 0, st>>>((B*)out_w, (B*)out_b, (const float*)w, (const float*)b, C, groups, parts);
        else pack_grouped_kernel<<<rows, 128, 0, st>>>((B*)out_w, (B*)out_b, (const B*)w, (const B*)b, C, groups, parts);
    } else {
        if (src32) pack_grouped_kernel<<<rows, 128, 0, st>>>((__half*)out_w, (__half*)out_b, (const float*)w, (const float*)b, C, groups, parts);
        else pack_grouped_kernel<<<rows, 128, 0, st>>>((__half*)out_w, (__half*)out_b, (const __half*)w, (const __half*)b, C, groups, parts);
    }
    return cudaGetLastError();
}
cudaError_t block_unpack_grouped(void* d_w, void* d_b, const float* dense, const float* sums, bool dst32, int C, int groups, int parts, int dtype,
                                 cudaStream_t st) {
    const int rows = parts * C;
    if (dst32) unpack_grouped_kernel<<<rows, 128, 0, st>>>((float*)d_w, (float*)d_b, dense, sums, C, groups, parts);
    else if (dtype == 0) unpack_grouped_kernel<<<rows, 128, 0, st>>>((__nv_bfloat16*)d_w, (__nv_bfloat16*)d_b, dense, sums, C, groups, parts);
    else unpack_grouped_kernel<<<rows, 128, 0, st>>>((__half*)d_w, (__half*)d_b, dense, sums, C, groups, parts);
    return cudaGetLastError();
}
cudaError_t block_pool_fwd(float* out, float* stats, const void* logits, const void* x, long long ldx, int N, int T, int C, float floor_var,
                           int dtype, cudaStream_t st) {
    const dim3 grid((C + 255) / 256, N);
    if (dtype == 0) pool_fwd_kernel<<<grid, kPoolWarps * 32, 0, st>>>(out, stats, (const __nv_bfloat16*)logits, (const __nv_bfloat16*)x, ldx, T, C, floor_var);
    else pool_fwd_kernel<<<grid, kPoolWarps * 32, 0, st>>>(out, stats, (const __half*)logits, (const __half*)x, ldx, T, C, floor_var);
    return cudaGetLastError();
}
cudaError_t block_pool_bwd(void* d_logits, void* dx, const float* d_out, const float* out, const float* stats,
                           const void* logits, const void* x, int N, int T, int C, float floor_var, int dtype, cudaStream_t st) {
    // few utterances: share the time axis among CTAs
    const int cols = (C + 255) / 256, steps = (T + kPoolWarps - 1) / kPoolWarps;
    int split = (int)((4ll * device_sm_count() + (long long)cols * N - 1) / ((long long)cols * N));
    split = split < 1 ? 1 : split > steps ? steps : split;
    const dim3 grid(cols, N, split);
    if (dtype == 0)
        pool_bwd_kernel<<<grid, kPoolWarps * 32, 0, st>>>((__nv_bfloat16*)d_logits, (__nv_bfloat16*)dx, d_out, out, stats, (const __nv_bfloat16*)logits,
                                                          (const __nv_bfloat16*)x, T, C, floor_var);
    else
        pool_bwd_kernel<<<grid, kPoolWarps * 32, 0, st>>>((__half*)d_logits, (__half*)dx, d_out, out, stats, (const __half*)logits, (const __half*)x,
                                                          T, C, floor_var);
    return cudaGetLastError();
}

}  // namespace na1d
