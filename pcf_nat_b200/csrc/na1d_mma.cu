// Fused NA1D on warp-level matrix instructions: the shapes the tcgen05 kernels do not take (channel counts other than 16, 32
// and 64, effective windows above 33, more than 32 heads) up to 128 channels.
//
// What bounds these shapes is arithmetic on the band, not memory: a row needs `win` dot products and `win` row updates of C
// channels in each of its contractions. On the CUDA cores (na1d_simt.cu) that is 2 C win fp32 operations each, plus the loads
// of every neighbour row by every query: 64 x 4 x 203 rows, 48 channels, window 41 took 44 us forward and 231 us backward
// against 9 us of HBM time. Here a warp owns 16 consecutive rows of one residue class (tokens t = r mod dil of a sequence,
// on which a dilated window is a plain one) and walks the 16-row chunks of the other side that meet its band, with
// m16n8k16 products whose operands come from one shared-memory tile by ldmatrix. The tiles are too small for the 128-row
// tcgen05 shape to pay: at these windows most of a 128 x 256 tile would be outside the band.
//
// Precision is that of the fp32 kernel: the logits are products of 16-bit inputs summed in fp32 either way; the probabilities
// and their gradients enter the second contractions whole, as three bf16 pieces (8 + 8 + 8 bits) or, for fp16 inputs, which are exact
// in tf32, as two tf32 pieces (11 + 13 bits with a sign: the first one rounded to nearest), so nothing is rounded but the result.
// Two bf16 pieces (2^-17 of the value) cost 4 % less time and raised the error of the 16-bit results by 1e-6 of itself.
//
// A chunk that meets the band only partly multiplies the rows outside it by an exact zero, which an infinite or NaN row would
// turn into NaN: a CTA whose staged rows hold such a value computes its rows with plain fp32 arithmetic instead.
#include "na1d_internal.h"
#include "na1d_tc_common.cuh"
#include <type_traits>

namespace na1d {
namespace {

constexpr int kWarps = 4, kThreads = kWarps * 32, kRows = kWarps * 16;

// ---------------------------------------------------------------- matrix instructions
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <typename E> __device__ __forceinline__ void mma16(float (&d)[4], const uint32_t* a, uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma16<__nv_bfloat16>(float (&d)[4], const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma16<__half>(float (&d)[4], const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma8_tf32(float (&d)[4], const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A 16 x 16 block of fp32 weights (two accumulator fragments: columns 0-7 and 8-15) as the left operand of weights . rows, in two
// pieces; rows come from shared memory by ldmatrix.trans.
template <typename E> struct Weights;
template <> struct Weights<__nv_bfloat16> {
    uint32_t p[3][4];   // a fragment of m16n8k16: (row, k), (row + 8, k), (row, k + 8), (row + 8, k + 8)
    __device__ __forceinline__ void set(const float (&w)[2][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float a = w[i >> 1][2 * (i & 1)], b = w[i >> 1][2 * (i & 1) + 1];
#pragma unroll
            for (int k = 0; k < 3; ++k) {   // (the remainders are exact)
                p[k][i] = Cvt<__nv_bfloat16>::pack2(a, b);
                a -= __uint_as_float(p[k][i] << 16);
                b -= __uint_as_float(p[k][i] & 0xffff0000u);
            }
        }
    }
    // d[0], d[1] += weights . (16 rows x channels 0-7, 8-15); x: the four matrices of ldsm4_t over those rows and channels
    __device__ __forceinline__ void apply(float (&d0)[4], float (&d1)[4], const uint32_t (&x)[4]) const {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mma16<__nv_bfloat16>(d0, p[k], x[0], x[1]);
            mma16<__nv_bfloat16>(d1, p[k], x[2], x[3]);
        }
    }
};
template <> struct Weights<__half> {
    // m16n8k8 fragments of the two column halves: first piece and remainder. The contraction index may be permuted freely: k = l % 4 and l % 4 + 4 stand for
    // columns 2 (l % 4) and 2 (l % 4) + 1, which is what a thread holds of the accumulator and what ldmatrix.trans gives it.
    uint32_t hi[2][4], lo[2][4];
    __device__ __forceinline__ void set(const float (&w)[2][4]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float v[4] = {w[h][0], w[h][2], w[h][1], w[h][3]};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                hi[h][i] = (__float_as_uint(v[i]) + 0x1000u) & 0xffffe000u;
                lo[h][i] = __float_as_uint(v[i] - __uint_as_float(hi[h][i]));   // at most half a step of 2^-11: 11 bits, exact in tf32
            }
        }
    }
    __device__ __forceinline__ void apply(float (&d0)[4], float (&d1)[4], const uint32_t (&x)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // matrix i: rows 8 (i & 1).., channels 8 (i >> 1)..
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&x[i]));
            const uint32_t b0 = __float_as_uint(v.x), b1 = __float_as_uint(v.y);
            if (i < 2) { mma8_tf32(d0, hi[i & 1], b0, b1); mma8_tf32(d0, lo[i & 1], b0, b1); }
            else { mma8_tf32(d1, hi[i & 1], b0, b1); mma8_tf32(d1, lo[i & 1], b0, b1); }
        }
    }
};

// ---------------------------------------------------------------- tile geometry
struct Tile {
    int n, r, u0, Tr, vl, h;   // sequence, residue, first row (token u = row of the residue), tokens of the residue, valid ones, head
    __device__ __forceinline__ bool init(const Geometry& gm, const int* valid_len, int tps) {
        const int s = (int)blockIdx.x / tps;
        u0 = ((int)blockIdx.x - s * tps) * kRows;
        n = s / gm.dil;
        r = s - n * gm.dil;
        Tr = gm.T > r ? (gm.T - r + gm.dil - 1) / gm.dil : 0;
        h = n % gm.H;
        const int v = valid_len ? min(gm.T, __ldg(valid_len + n / gm.H)) : gm.T;
        vl = v > r ? (v - r + gm.dil - 1) / gm.dil : 0;
        return u0 < Tr;
    }
    __device__ __forceinline__ size_t row(const Geometry& gm, int u) const { return (size_t)n * gm.T + (size_t)u * gm.dil + r; }
};
// shared memory: X rows, Y rows (pitch bytes each: an odd number of 16-byte units, so that eight consecutive rows meet eight
// different bank groups), then floats: bias table, per-row statistics or the warps' band copies
__host__ __device__ constexpr int pitch_bytes(int CP) { return CP * 2 + 16; }
__host__ __device__ inline int chunks_of(int win) { return (win + 30) / 16; }            // 16-row chunks that meet the band of 16 rows
__host__ __device__ inline int staged_rows(int win) { return 16 * (kWarps - 1 + chunks_of(win)); }
__host__ __device__ inline int table_floats(int win) { return 16 * (chunks_of(win) + 1); }
__host__ __device__ inline int band_pitch(int win) { return win | 1; }
// rows that the warps with rows of the residue meet: a short last tile stages no more than it needs (`most` = the full tile's)
__device__ __forceinline__ int needed_rows(const Tile& t, int nch, int most) { return min(most, 16 * ((t.Tr - t.u0 + 15) / 16 - 1 + nch)); }
size_t smem_bytes(int CP, int win, bool backward, bool d_rpb) {
    const int rows = staged_rows(win);
    size_t b = (size_t)2 * rows * pitch_bytes(CP) + (size_t)table_floats(win) * 4;
    if (backward) {
        const size_t stats = (size_t)2 * rows * 4, bands = d_rpb ? (size_t)kWarps * 16 * band_pitch(win) * 4 : 0;
        b += stats > bands ? stats : bands;
    }
    return b;
}

// Stages rows [first, first + rows) of the residue (zeros outside it: the reference's zero padding of keys and values) and
// returns, for the whole CTA, whether any value is infinite or NaN.
template <typename E, int CP>
__device__ __forceinline__ bool stage_rows(uint8_t* x, uint8_t* y, const E* __restrict__ gx, const E* __restrict__ gy, const Tile& t,
                                           const Geometry& gm, int first, int rows) {
    constexpr int CH = CP / 8, U = 4;   // U independent pairs of loads in flight per thread
    bool bad = false;
    for (int i0 = threadIdx.x; i0 < rows * CH; i0 += U * kThreads) {
        uint4 a[U], b[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + k * kThreads, row = i / CH, c = i - row * CH, u = first + row;
            a[k] = b[k] = make_uint4(0, 0, 0, 0);
            if (row < rows && u >= 0 && u < t.Tr && c * 8 < gm.C) {
                const size_t at = t.row(gm, u) * gm.C + c * 8;
                a[k] = __ldg(reinterpret_cast<const uint4*>(gx + at));
                b[k] = __ldg(reinterpret_cast<const uint4*>(gy + at));
            }
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + k * kThreads, row = i / CH, c = i - row * CH;
            if (row >= rows) break;
            *reinterpret_cast<uint4*>(x + row * pitch_bytes(CP) + c * 16) = a[k];
            *reinterpret_cast<uint4*>(y + row * pitch_bytes(CP) + c * 16) = b[k];
            // an exponent of all ones in either half of a word
            constexpr uint32_t m = std::is_same<E, __half>::value ? 0x7c00u : 0x7f80u;
            const uint32_t w[8] = {a[k].x, a[k].y, a[k].z, a[k].w, b[k].x, b[k].y, b[k].z, b[k].w};
#pragma unroll
            for (int e = 0; e < 8; ++e) bad |= (w[e] & m) == m || (w[e] & (m << 16)) == m << 16;
        }
    }
    return __syncthreads_or(bad) != 0;
}
// left-operand fragments of 16 own rows, straight from global memory (zeros outside the residue)
template <typename E, int CP>
__device__ __forceinline__ void own_rows(uint32_t (&f)[CP / 16][4], const E* __restrict__ g, const Tile& t, const Geometry& gm, int u, int lane) {
    const int fr = lane >> 2, fc = 2 * (lane & 3);
#pragma unroll
    for (int ks = 0; ks < CP / 16; ++ks)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = u + fr + 8 * (i & 1), c = ks * 16 + fc + 8 * (i >> 1);
            f[ks][i] = row < t.Tr && c < gm.C ? __ldg(reinterpret_cast<const uint32_t*>(g + t.row(gm, row) * gm.C + c)) : 0u;
        }
}
template <typename E, int CP>
__device__ __forceinline__ void store_rows(E* __restrict__ g, const float (&acc)[CP / 8][4], const Tile& t, const Geometry& gm, int u, int lane,
                                           float f0, float f1) {
    const int fr = lane >> 2, fc = 2 * (lane & 3);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = u + fr + 8 * h;
        if (row >= t.Tr) continue;
        E* dst = g + t.row(gm, row) * gm.C + fc;
        const float f = h ? f1 : f0;
#pragma unroll
        for (int nt = 0; nt < CP / 8; ++nt)
            if (nt * 8 < gm.C) *reinterpret_cast<uint32_t*>(dst + nt * 8) = Cvt<E>::pack2(acc[nt][2 * h] * f, acc[nt][2 * h + 1] * f);
    }
}
// s = own . rows^T for one chunk of 16 staged rows; base: shared address of the chunk's first row plus this lane's ldsm4 offset
template <typename E, int CP>
__device__ __forceinline__ void products(float (&s)[2][4], const uint32_t (&own)[CP / 16][4], uint32_t base) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s[0][i] = s[1][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < CP / 16; ++ks) {
        uint32_t b[4];
        ldsm4(b, base + ks * 32);
        mma16<E>(s[0], own[ks], b[0], b[1]);
        mma16<E>(s[1], own[ks], b[2], b[3]);
    }
}
template <typename E, int CP>
__device__ __forceinline__ void accumulate(float (&acc)[CP / 8][4], const Weights<E>& w, uint32_t base) {
#pragma unroll
    for (int ks = 0; ks < CP / 16; ++ks) {
        uint32_t b[4];
        ldsm4_t(b, base + ks * 32);
        w.apply(acc[2 * ks], acc[2 * ks + 1], b);
    }
}

// ---------------------------------------------------------------- plain fp32 rows (staged values that are not finite)
// One warp per row, four channels per lane; the arithmetic of the CUDA-core kernels.
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
template <typename E> __device__ __forceinline__ void lane4(float (&f)[4], const E* __restrict__ g, size_t row, int C, int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = lane * 4 + i < C ? (float)g[row * C + lane * 4 + i] : 0.f;
}
__device__ __forceinline__ float dot4(const float (&a)[4], const float (&b)[4], int C, int lane) {
    float s = 0.f;
    if (lane * 4 < C) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s = fmaf(a[i], b[i], s);
    }
    return warp_sum(s);
}
__device__ __forceinline__ float mask_of(int u, int j, const Tile& t) { return j < 0 || j >= t.vl || u >= t.vl ? kMaskValue : 0.f; }

template <typename E>
__device__ __noinline__ void plain_fwd_rows(E* o, float* lse, const E* q, const E* k, const E* v, const float* rpb, Tile t, Geometry gm) {
    const int lane = threadIdx.x & 31;
    for (int u = t.u0 + (threadIdx.x >> 5); u < min(t.u0 + kRows, t.Tr); u += kWarps) {
        float qa[4], x[4], acc[4] = {0.f, 0.f, 0.f, 0.f}, m = -INFINITY, l = 0.f;
        const size_t row = t.row(gm, u);
        lane4(qa, q, row, gm.C, lane);
        for (int kk = 0; kk < gm.win; ++kk) {
            const int j = u + kk - gm.left;
            const bool in = j >= 0 && j < t.Tr;
            float s = 0.f;
            if (in) { lane4(x, k, t.row(gm, j), gm.C, lane); s = dot4(qa, x, gm.C, lane); }
            s = fmaf(s, gm.scale * kLog2e, ((rpb ? __ldg(rpb + t.h * gm.win + kk) : 0.f) + mask_of(u, j, t)) * kLog2e);
            const float mn = fmaxf(m, s), ref = mn == -INFINITY ? 0.f : mn;
            const float alpha = exp2f(m - ref), p = exp2f(s - ref);
            l = fmaf(l, alpha, p);
            m = mn;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] *= alpha;
            if (in) {
                lane4(x, v, t.row(gm, j), gm.C, lane);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] = fmaf(p, x[i], acc[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (lane * 4 + i < gm.C) o[row * gm.C + lane * 4 + i] = (E)(acc[i] / l);
        if (lse && lane == 0) lse[row] = (m + log2f(l)) * kLn2;
    }
}

// own rows against the rows of the other side. KEY false: own = query (a1 = q, a2 = d_o; x = k, y = v), out1 = dq and the bias
// gradient; KEY true: own = key (a1 = k, a2 = v; x = q, y = d_o), out1 = dk, out2 = dv.
template <typename E, bool KEY>
__device__ __noinline__ void plain_bwd_rows(E* out1, E* out2, float* d_rpb, const E* a1, const E* a2, const E* x, const E* y, const E* o,
                                            const float* lse, const float* rpb, Tile t, Geometry gm) {
    const int lane = threadIdx.x & 31;
    for (int u = t.u0 + (threadIdx.x >> 5); u < min(t.u0 + kRows, t.Tr); u += kWarps) {
        const size_t row = t.row(gm, u);
        float f1[4], f2[4], xr[4], yr[4], ob[4], c1[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
        lane4(f1, a1, row, gm.C, lane);
        lane4(f2, a2, row, gm.C, lane);
        float delta = 0.f;
        if (!KEY) { lane4(ob, o, row, gm.C, lane); delta = dot4(f2, ob, gm.C, lane); }
        for (int kk = 0; kk < gm.win; ++kk) {
            const int w = KEY ? u - (kk - gm.left) : u + kk - gm.left;   // row of the other side
            const bool in = w >= 0 && w < t.Tr;
            if (KEY && !in) continue;
            float s = 0.f, dp = 0.f;
            const size_t wr = t.row(gm, in ? w : 0);
            if (in) {
                lane4(xr, x, wr, gm.C, lane);
                lane4(yr, y, wr, gm.C, lane);
                s = dot4(f1, xr, gm.C, lane);
                dp = dot4(f2, yr, gm.C, lane);
            }
            const size_t qrow = KEY ? wr : row;
            if (KEY) { lane4(ob, o, wr, gm.C, lane); delta = dot4(yr, ob, gm.C, lane); }
            const float b = (rpb ? __ldg(rpb + t.h * gm.win + kk) : 0.f) + (KEY ? mask_of(w, u, t) : mask_of(u, w, t));
            const float p = exp2f(fmaf(s, gm.scale * kLog2e, b * kLog2e) - __ldg(lse + qrow) * kLog2e);
            const float ds = p * (dp - delta);
            if (in) {
#pragma unroll
                for (int i = 0; i < 4; ++i) { c1[i] = fmaf(ds, xr[i], c1[i]); if (KEY) c2[i] = fmaf(p, yr[i], c2[i]); }
            }
            if (!KEY && d_rpb && lane == 0) atomicAdd(d_rpb + t.h * gm.win + kk, ds);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (lane * 4 + i < gm.C) {
                out1[row * gm.C + lane * 4 + i] = (E)(c1[i] * gm.scale);
                if (KEY) out2[row * gm.C + lane * 4 + i] = (E)c2[i];
            }
    }
}

// ---------------------------------------------------------------- forward
template <typename E, int CP>
__global__ void __launch_bounds__(kThreads) mma_fwd_kernel(E* __restrict__ o, float* __restrict__ lse, const E* __restrict__ q,
                                                          const E* __restrict__ k, const E* __restrict__ v, const float* __restrict__ rpb,
                                                          const int* __restrict__ valid_len, Geometry gm, int tps) {
    extern __shared__ __align__(16) uint8_t smem[];
    Tile t;
    if (!t.init(gm, valid_len, tps)) return;
    const int rows = staged_rows(gm.win), nch = chunks_of(gm.win), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* sx = smem;
    uint8_t* sy = smem + rows * pitch_bytes(CP);
    float* tab = reinterpret_cast<float*>(sy + rows * pitch_bytes(CP));   // log2e * bias at offset + 16, -inf outside the window
    for (int i = threadIdx.x; i < table_floats(gm.win); i += kThreads) {
        const int kk = i - 16;
        tab[i] = kk < 0 || kk >= gm.win ? -INFINITY : rpb ? __ldg(rpb + t.h * gm.win + kk) * kLog2e : 0.f;
    }
    const int u = t.u0 + warp * 16;
    uint32_t qa[CP / 16][4];
    own_rows<E, CP>(qa, q, t, gm, u, lane);   // (in flight together with the staged rows)
    if (stage_rows<E, CP>(sx, sy, k, v, t, gm, t.u0 - gm.left, needed_rows(t, nch, rows))) {
        plain_fwd_rows<E>(o, lse, q, k, v, rpb, t, gm);
        return;
    }
    if (u >= t.Tr) return;
    const int fr = lane >> 2, fc = 2 * (lane & 3);
    const uint32_t kaddr = ptx::smem_u32(sx) + (warp * 16 + (lane & 7) + ((lane >> 4) << 3)) * pitch_bytes(CP) + ((lane >> 3) & 1) * 16;
    const uint32_t vaddr = ptx::smem_u32(sy) + (warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * pitch_bytes(CP) + (lane >> 4) * 16;
    const bool need_mask = u < gm.left || u + 15 + (gm.win - 1 - gm.left) >= t.vl;
    const float sc = gm.scale * kLog2e, mask2 = kMaskValue * kLog2e;
    float acc[CP / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < CP / 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    for (int ch = 0; ch < nch; ++ch) {
        float s[2][4];
        products<E, CP>(s, qa, kaddr + ch * 16 * pitch_bytes(CP));
        float mx[2] = {m[0], m[1]};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int h = i >> 1, c = ch * 16 + nt * 8 + fc + (i & 1), row = fr + 8 * h;   // staged row relative to the warp's first
                const float b = tab[c - row + 16];
                float x = fmaf(s[nt][i], sc, b);
                if (need_mask) {
                    const int j = u - gm.left + c;
                    if (j < 0 || j >= t.vl || u + row >= t.vl) x += mask2;
                }
                x = b == -INFINITY ? b : x;
                s[nt][i] = x;
                mx[h] = fmaxf(mx[h], x);
            }
        mx[0] = tc::quad_max(mx[0]);
        mx[1] = tc::quad_max(mx[1]);
        const float r0 = mx[0] == -INFINITY ? 0.f : mx[0], r1 = mx[1] == -INFINITY ? 0.f : mx[1];
        if (__any_sync(0xffffffffu, mx[0] != m[0] || mx[1] != m[1])) {
            const float a0 = tc::fast_exp2(m[0] - r0), a1 = tc::fast_exp2(m[1] - r1);
            l[0] *= a0;
            l[1] *= a1;
#pragma unroll
            for (int i = 0; i < CP / 8; ++i) { acc[i][0] *= a0; acc[i][1] *= a0; acc[i][2] *= a1; acc[i][3] *= a1; }
            m[0] = mx[0];
            m[1] = mx[1];
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[nt][i] = tc::fast_exp2(s[nt][i] - (i >> 1 ? r1 : r0));
                l[i >> 1] += s[nt][i];
            }
        Weights<E> w;
        w.set(s);
        accumulate<E, CP>(acc, w, vaddr + ch * 16 * pitch_bytes(CP));
    }
    l[0] = tc::quad_sum(l[0]);
    l[1] = tc::quad_sum(l[1]);
    store_rows<E, CP>(o, acc, t, gm, u, lane, 1.f / l[0], 1.f / l[1]);
    if (lse && (lane & 3) == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (u + fr + 8 * h < t.Tr) lse[t.row(gm, u + fr + 8 * h)] = (m[h] + log2f(l[h])) * kLn2;
    }
}

// ---------------------------------------------------------------- backward
// Two views of the band, one CTA each (blockIdx.y): query rows (dq and the bias gradient) against staged keys and values, key rows
// (dk, dv) against staged queries and output gradients. The band is computed in both, so every result has one owner: no
// atomics on dq, dk, dv and no transposition of a fragment. delta = d_o . o per query row is computed where it is used.
template <typename E, int CP, bool KEY>
__device__ __forceinline__ void bwd_view(uint8_t* smem, E* __restrict__ out1, E* __restrict__ out2, float* __restrict__ d_rpb,
                                         const E* __restrict__ ga1, const E* __restrict__ ga2, const E* __restrict__ gx,
                                         const E* __restrict__ gy, const E* __restrict__ o, const float* __restrict__ lse,
                                         const float* __restrict__ rpb, const Tile& t, const Geometry& gm) {
    const int rows = staged_rows(gm.win), nch = chunks_of(gm.win), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int right = gm.win - 1 - gm.left, before = KEY ? right : gm.left;
    uint8_t* sx = smem;
    uint8_t* sy = smem + rows * pitch_bytes(CP);
    float* tab = reinterpret_cast<float*>(sy + rows * pitch_bytes(CP));
    float* extra = tab + table_floats(gm.win);
    for (int i = threadIdx.x; i < table_floats(gm.win); i += kThreads) {
        // other row minus own row, from the first staged one: kk in the query view, win - 1 - kk in the key view
        const int x = i - 16, kk = KEY ? gm.win - 1 - x : x;
        tab[i] = x < 0 || x >= gm.win ? -INFINITY : rpb ? __ldg(rpb + t.h * gm.win + kk) * kLog2e : 0.f;
    }
    float* s_lse = extra;
    float* s_delta = extra + rows;
    if (KEY) {
        // log-sum-exp and delta of the staged query rows; a row outside the sequence has probability 0
        constexpr int CH = CP / 8, G = CH <= 2 ? 2 : CH <= 4 ? 4 : CH <= 8 ? 8 : 16;   // lanes per row
        for (int i = threadIdx.x / G; i < (rows + 31) / 32 * 32; i += kThreads / G) {
            const int w = t.u0 - before + i, c = threadIdx.x % G;
            const bool in = i < rows && w >= 0 && w < t.Tr;
            float d = 0.f;
            if (in && c * 8 < gm.C) {
                const size_t at = t.row(gm, w) * gm.C + c * 8;
                float a[8], b[8];
                Cvt<E>::unpack(__ldg(reinterpret_cast<const uint4*>(gy + at)), a);
                Cvt<E>::unpack(__ldg(reinterpret_cast<const uint4*>(o + at)), b);
#pragma unroll
                for (int e = 0; e < 8; ++e) d = fmaf(a[e], b[e], d);
            }
#pragma unroll
            for (int x = G / 2; x > 0; x >>= 1) d += __shfl_xor_sync(0xffffffffu, d, x);
            if (i < rows && c == 0) { s_delta[i] = d; s_lse[i] = in ? __ldg(lse + t.row(gm, w)) * kLog2e : INFINITY; }
        }
    }
    if (stage_rows<E, CP>(sx, sy, gx, gy, t, gm, t.u0 - before, needed_rows(t, nch, rows))) {
        plain_bwd_rows<E, KEY>(out1, out2, d_rpb, ga1, ga2, gx, gy, o, lse, rpb, t, gm);
        return;
    }
    const int u = t.u0 + warp * 16, fr = lane >> 2, fc = 2 * (lane & 3);
    const bool alive = u < t.Tr;
    float* band = extra + warp * 16 * band_pitch(gm.win);   // query view with a bias gradient: dS of the warp's rows
    if (alive) {
        uint32_t a1[CP / 16][4], a2[CP / 16][4];
        own_rows<E, CP>(a1, ga1, t, gm, u, lane);
        own_rows<E, CP>(a2, ga2, t, gm, u, lane);
        float own_lse[2] = {0.f, 0.f}, own_delta[2] = {0.f, 0.f};
        if (!KEY) {
            uint32_t ob[CP / 16][4];
            own_rows<E, CP>(ob, o, t, gm, u, lane);
#pragma unroll
            for (int ks = 0; ks < CP / 16; ++ks)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float a_lo = Cvt<E>::from_bits((unsigned short)(a2[ks][i] & 0xffffu)), a_hi = Cvt<E>::from_bits((unsigned short)(a2[ks][i] >> 16));
                    const float b_lo = Cvt<E>::from_bits((unsigned short)(ob[ks][i] & 0xffffu)), b_hi = Cvt<E>::from_bits((unsigned short)(ob[ks][i] >> 16));
                    own_delta[i & 1] = fmaf(a_lo, b_lo, fmaf(a_hi, b_hi, own_delta[i & 1]));
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                own_delta[h] = tc::quad_sum(own_delta[h]);
                own_lse[h] = u + fr + 8 * h < t.Tr ? __ldg(lse + t.row(gm, u + fr + 8 * h)) * kLog2e : INFINITY;
            }
        }
        const int first = warp * 16;
        const uint32_t off_n = ((lane & 7) + ((lane >> 4) << 3)) * pitch_bytes(CP) + ((lane >> 3) & 1) * 16;
        const uint32_t off_t = ((lane & 7) + (((lane >> 3) & 1) << 3)) * pitch_bytes(CP) + (lane >> 4) * 16;
        const uint32_t xa = ptx::smem_u32(sx) + first * pitch_bytes(CP), ya = ptx::smem_u32(sy) + first * pitch_bytes(CP);
        const bool need_mask = KEY ? u + 15 + gm.left >= t.vl : u < gm.left || u + 15 + right >= t.vl;
        const float sc = gm.scale * kLog2e, mask2 = kMaskValue * kLog2e;
        float c1[CP / 8][4], c2[KEY ? CP / 8 : 1][4];
#pragma unroll
        for (int i = 0; i < CP / 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) { c1[i][e] = 0.f; if (KEY) c2[i][e] = 0.f; }
#pragma unroll 1
        for (int ch = 0; ch < nch; ++ch) {
            const uint32_t at = ch * 16 * pitch_bytes(CP);
            float s[2][4], dp[2][4];
            products<E, CP>(s, a1, xa + at + off_n);
            products<E, CP>(dp, a2, ya + at + off_n);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int c0 = ch * 16 + nt * 8 + fc;
                float2 cl, cd;
                if (KEY) {
                    cl = *reinterpret_cast<const float2*>(s_lse + first + c0);
                    cd = *reinterpret_cast<const float2*>(s_delta + first + c0);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int h = i >> 1, c = c0 + (i & 1), row = fr + 8 * h;
                    const float b = tab[c - row + 16];
                    float x = fmaf(s[nt][i], sc, b);
                    if (need_mask) {
                        const int w = u - before + c;   // the other side's row: a key (query view) or a query (key view)
                        if (w >= t.vl || u + row >= t.vl || (!KEY && w < 0)) x += mask2;
                    }
                    const bool on = b != -INFINITY;
                    const float p = on ? tc::fast_exp2(x - (KEY ? (i & 1 ? cl.y : cl.x) : own_lse[h])) : 0.f;
                    const float ds = on ? p * (dp[nt][i] - (KEY ? (i & 1 ? cd.y : cd.x) : own_delta[h])) : 0.f;
                    s[nt][i] = p;
                    dp[nt][i] = ds;
                    if (!KEY && d_rpb && (unsigned)(c - row) < (unsigned)gm.win) band[row * band_pitch(gm.win) + c - row] = ds;
                }
            }
            Weights<E> w;
            w.set(dp);
            accumulate<E, CP>(c1, w, xa + at + off_t);
            if constexpr (KEY) {
                w.set(s);
                accumulate<E, CP>(c2, w, ya + at + off_t);
            }
        }
        store_rows<E, CP>(out1, c1, t, gm, u, lane, gm.scale, gm.scale);
        if constexpr (KEY) store_rows<E, CP>(out2, c2, t, gm, u, lane, 1.f, 1.f);
    }
    if (!KEY && d_rpb) {
        // column sums of the warps' bands (pitch odd: conflict-free), one global addition per CTA and offset
        __syncthreads();
        const int live = min(kRows, (t.Tr - t.u0 + 15) / 16 * 16);   // rows of warps that ran; rows past the sequence hold zeros
        for (int kk = threadIdx.x; kk < gm.win; kk += kThreads) {
            float a = 0.f;
            for (int i = 0; i < live; ++i) a += extra[i * band_pitch(gm.win) + kk];
            atomicAdd(d_rpb + t.h * gm.win + kk, a);
        }
    }
}

template <typename E, int CP>
__global__ void __launch_bounds__(kThreads) mma_bwd_kernel(E* __restrict__ dq, E* __restrict__ dk, E* __restrict__ dv, float* __restrict__ d_rpb,
                                                          const E* __restrict__ d_o, const E* __restrict__ q, const E* __restrict__ k,
                                                          const E* __restrict__ v, const E* __restrict__ o, const float* __restrict__ lse,
                                                          const float* __restrict__ rpb, const int* __restrict__ valid_len, Geometry gm, int tps) {
    extern __shared__ __align__(16) uint8_t smem[];
    Tile t;
    if (!t.init(gm, valid_len, tps)) return;
    if (blockIdx.y == 0) bwd_view<E, CP, true>(smem, dk, dv, nullptr, k, v, q, d_o, o, lse, rpb, t, gm);
    else bwd_view<E, CP, false>(smem, dq, nullptr, d_rpb, q, d_o, k, v, o, lse, rpb, t, gm);
}

// ---------------------------------------------------------------- the unfused pair
// The same products with the fp32 band in memory: 128 rows per CTA (the band's halo is staged too: 8 warps keep it at
// (win - 1) / 128). The band goes through shared memory both ways, so that global memory sees whole contiguous rows.
//   band_out: band[t, kk] = a[t] . b[j]          (QK forward, dA)
//   band_rows<false>: out[t] = sum band[t, kk] x[j]     (AV forward, dQ)
//   band_rows<true> : out[j] = sum band[t, kk] x[t]     (dV, dK)
constexpr int kBandWarps = 8, kBandThreads = kBandWarps * 32, kBandRows = kBandWarps * 16;
__host__ __device__ inline int band_staged(int win) { return 16 * (kBandWarps - 1 + chunks_of(win)); }

__device__ __forceinline__ bool band_tile(Tile& t, const Geometry& gm, int tps) {
    const int s = (int)blockIdx.x / tps;
    t.u0 = ((int)blockIdx.x - s * tps) * kBandRows;
    t.n = s / gm.dil;
    t.r = s - t.n * gm.dil;
    t.Tr = gm.T > t.r ? (gm.T - t.r + gm.dil - 1) / gm.dil : 0;
    t.vl = t.Tr;
    t.h = 0;
    return t.u0 < t.Tr;
}
// rows [first, first + rows) of one tensor; whether a value is infinite or NaN
template <typename E, int CP>
__device__ __forceinline__ bool band_stage_rows(uint8_t* x, const E* __restrict__ g, const Tile& t, const Geometry& gm, int first, int rows) {
    constexpr int CH = CP / 8, U = CP <= 32 ? 2 : 4;
    bool bad = false;
    for (int i0 = threadIdx.x; i0 < rows * CH; i0 += U * kBandThreads) {
        uint4 a[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + k * kBandThreads, row = i / CH, c = i - row * CH, u = first + row;
            a[k] = make_uint4(0, 0, 0, 0);
            if (row < rows && u >= 0 && u < t.Tr && c * 8 < gm.C) a[k] = __ldg(reinterpret_cast<const uint4*>(g + t.row(gm, u) * gm.C + c * 8));
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + k * kBandThreads, row = i / CH, c = i - row * CH;
            if (row >= rows) break;
            *reinterpret_cast<uint4*>(x + row * pitch_bytes(CP) + c * 16) = a[k];
            constexpr uint32_t m = std::is_same<E, __half>::value ? 0x7c00u : 0x7f80u;
            const uint32_t w[4] = {a[k].x, a[k].y, a[k].z, a[k].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) bad |= (w[e] & m) == m || (w[e] & (m << 16)) == m << 16;
        }
    }
    return bad;
}
// band rows [first, first + rows) into s (win floats each, zeros outside the residue); thread `id` of `n` takes part
__device__ __forceinline__ bool band_load(float* s, const float* __restrict__ band, const Tile& t, const Geometry& gm, int first, int rows, int id, int n) {
    const int lo = max(0, -first), hi = min(rows, t.Tr - first), total = rows * gm.win;
    bool bad = false;
    auto put = [&](int i, float v) {
        s[i] = v;
        bad |= (__float_as_uint(v) & 0x7f000000u) == 0x7f000000u;   // not finite, or so large that its first piece might not be
    };
    if (gm.dil == 1) {   // the rows are one contiguous piece
        const float* src = band + ((long long)t.n * gm.T + first) * gm.win;
        const int a = lo * gm.win, b = hi * gm.win;
        constexpr int U = 8;
        for (int i0 = id; i0 < total; i0 += U * n) {
            float v[U];
#pragma unroll
            for (int k = 0; k < U; ++k) { const int i = i0 + k * n; v[k] = i >= a && i < b ? __ldg(src + i) : 0.f; }
#pragma unroll
            for (int k = 0; k < U; ++k) if (i0 + k * n < total) put(i0 + k * n, v[k]);
        }
    } else {
        for (int i = id; i < total; i += n) {
            const int row = i / gm.win;
            put(i, row >= lo && row < hi ? __ldg(band + t.row(gm, first + row) * gm.win + (i - row * gm.win)) : 0.f);
        }
    }
    return bad;
}

template <typename E, int CP>
__global__ void __launch_bounds__(kBandThreads) mma_band_out_kernel(float* __restrict__ band, const E* __restrict__ a, const E* __restrict__ b, Geometry gm, int tps) {
    extern __shared__ __align__(16) uint8_t smem[];
    Tile t;
    if (!band_tile(t, gm, tps)) return;
    const int rows = band_staged(gm.win), nch = chunks_of(gm.win), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u = t.u0 + warp * 16, fr = lane >> 2, fc = 2 * (lane & 3);
    float* out = reinterpret_cast<float*>(smem + rows * pitch_bytes(CP)) + warp * 16 * gm.win;
    uint32_t own[CP / 16][4];
    own_rows<E, CP>(own, a, t, gm, u, lane);
    band_stage_rows<E, CP>(smem, b, t, gm, t.u0 - gm.left, needed_rows(t, nch, rows));
    __syncthreads();
    if (u >= t.Tr) return;
    const uint32_t base = ptx::smem_u32(smem) + (warp * 16 + (lane & 7) + ((lane >> 4) << 3)) * pitch_bytes(CP) + ((lane >> 3) & 1) * 16;
    for (int ch = 0; ch < nch; ++ch) {
        float s[2][4];
        products<E, CP>(s, own, base + ch * 16 * pitch_bytes(CP));
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = fr + 8 * (i >> 1), kk = ch * 16 + nt * 8 + fc + (i & 1) - row, j = u - gm.left + row + kk;
                // (a neighbour outside the sequence is a zero row: 0 also where the query is infinite)
                if ((unsigned)kk < (unsigned)gm.win) out[row * gm.win + kk] = (unsigned)j < (unsigned)t.Tr ? s[nt][i] : 0.f;
            }
    }
    __syncwarp();
    const int live = min(16, t.Tr - u) * gm.win;
    if (gm.dil == 1) {
        float* dst = band + t.row(gm, u) * gm.win;
        for (int i = lane; i < live; i += 32) dst[i] = out[i];
    } else {
        for (int i = lane; i < live; i += 32) {
            const int row = i / gm.win;
            band[t.row(gm, u + row) * gm.win + (i - row * gm.win)] = out[i];
        }
    }
}

template <typename E, int CP, bool TRANSPOSED>
__global__ void __launch_bounds__(kBandThreads) mma_band_rows_kernel(E* __restrict__ out, const float* __restrict__ band, const E* __restrict__ x, Geometry gm, int tps) {
    extern __shared__ __align__(16) uint8_t smem[];
    Tile t;
    if (!band_tile(t, gm, tps)) return;
    const int rows = band_staged(gm.win), nch = chunks_of(gm.win), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u = t.u0 + warp * 16, fr = lane >> 2, fc = 2 * (lane & 3), before = TRANSPOSED ? gm.win - 1 - gm.left : gm.left;
    float* sb = reinterpret_cast<float*>(smem + rows * pitch_bytes(CP));
    bool bad;
    const int need = needed_rows(t, nch, rows);
    if (TRANSPOSED) bad = band_load(sb, band, t, gm, t.u0 - before, need, threadIdx.x, kBandThreads);
    else bad = band_load(sb, band, t, gm, t.u0, min(kBandRows, (t.Tr - t.u0 + 15) / 16 * 16), threadIdx.x, kBandThreads);
    bad |= band_stage_rows<E, CP>(smem, x, t, gm, t.u0 - before, need);
    if (__syncthreads_or(bad)) {
        // plain fp32 rows: an exact zero times an infinite or NaN row would not stay zero
        for (int v = t.u0 + warp; v < min(t.u0 + kBandRows, t.Tr); v += kBandWarps) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f}, f[4];
            for (int kk = 0; kk < gm.win; ++kk) {
                const int w = TRANSPOSED ? v - (kk - gm.left) : v + kk - gm.left;
                if (w < 0 || w >= t.Tr) continue;
                const float b = __ldg(band + t.row(gm, TRANSPOSED ? w : v) * gm.win + kk);
                lane4(f, x, t.row(gm, w), gm.C, lane);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] = fmaf(b, f[i], acc[i]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (lane * 4 + i < gm.C) out[t.row(gm, v) * gm.C + lane * 4 + i] = (E)acc[i];
        }
        return;
    }
    if (u >= t.Tr) return;
    const uint32_t base = ptx::smem_u32(smem) + (warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * pitch_bytes(CP) + (lane >> 4) * 16;
    const float* wb = sb + warp * 16 * gm.win;
    float acc[CP / 8][4];
#pragma unroll
    for (int i = 0; i < CP / 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    for (int ch = 0; ch < nch; ++ch) {
        float s[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = fr + 8 * (i >> 1), c = ch * 16 + nt * 8 + fc + (i & 1), d = c - row;
                const int at = TRANSPOSED ? c * gm.win + gm.win - 1 - d : row * gm.win + d;
                s[nt][i] = (unsigned)d < (unsigned)gm.win ? wb[at] : 0.f;
            }
        Weights<E> w;
        w.set(s);
        accumulate<E, CP>(acc, w, base + ch * 16 * pitch_bytes(CP));
    }
    store_rows<E, CP>(out, acc, t, gm, u, lane, 1.f, 1.f);
}

int padded_channels(int C) { return C <= 64 ? (C + 15) / 16 * 16 : C <= 96 ? 96 : 128; }

#define NA1D_MMA_DISPATCH(dtype, C, ...)                                                     \
    switch (padded_channels(C)) {                                                             \
        case 16: { constexpr int CP = 16; if ((dtype) == 0) { using E = __nv_bfloat16; __VA_ARGS__ } else { using E = __half; __VA_ARGS__ } } break; \
        case 32: { constexpr int CP = 32; if ((dtype) == 0) { using E = __nv_bfloat16; __VA_ARGS__ } else { using E = __half; __VA_ARGS__ } } break; \
        case 48: { constexpr int CP = 48; if ((dtype) == 0) { using E = __nv_bfloat16; __VA_ARGS__ } else { using E = __half; __VA_ARGS__ } } break; \
        case 64: { constexpr int CP = 64; if ((dtype) == 0) { using E = __nv_bfloat16; __VA_ARGS__ } else { using E = __half; __VA_ARGS__ } } break; \
        case 96: { constexpr int CP = 96; if ((dtype) == 0) { using E = __nv_bfloat16; __VA_ARGS__ } else { using E = __half; __VA_ARGS__ } } break; \
        default: { constexpr int CP = 128; if ((dtype) == 0) { using E = __nv_bfloat16; __VA_ARGS__ } else { using E = __half; __VA_ARGS__ } }       \
    }

}  // namespace

// 64 rows per CTA and per residue class of a sequence: the grid has N dil ceil(ceil(T / dil) / 64) CTAs
bool mma_supports(const Geometry& gm) {
    const long long tps = (((long long)gm.T + gm.dil - 1) / gm.dil + kRows - 1) / kRows;
    return gm.C <= 128 && gm.win <= 128 && (long long)gm.N * gm.dil * tps < (1ll << 31);
}

cudaError_t mma_fused_fwd(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb, const int* valid_len,
                          const Geometry& gm, int dtype, cudaStream_t st) {
    const int tps = ((gm.T + gm.dil - 1) / gm.dil + kRows - 1) / kRows;
    const dim3 grid((unsigned)((long long)gm.N * gm.dil * tps));
    NA1D_MMA_DISPATCH(dtype, gm.C, {
        auto kern = mma_fwd_kernel<E, CP>;
        const size_t smem = smem_bytes(CP, gm.win, false, false);
        if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
        kern<<<grid, kThreads, smem, st>>>((E*)o, lse, (const E*)q, (const E*)k, (const E*)v, rpb, valid_len, gm, tps);
    })
    return cudaGetLastError();
}

cudaError_t mma_fused_bwd(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k, const void* v,
                          const void* o, const float* lse, const float* rpb, const int* valid_len, const Geometry& gm, int dtype,
                          cudaStream_t st) {
    const int tps = ((gm.T + gm.dil - 1) / gm.dil + kRows - 1) / kRows;
    const dim3 grid((unsigned)((long long)gm.N * gm.dil * tps), 2);
    NA1D_MMA_DISPATCH(dtype, gm.C, {
        auto kern = mma_bwd_kernel<E, CP>;
        const size_t smem = smem_bytes(CP, gm.win, true, d_rpb != nullptr);
        if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
        kern<<<grid, kThreads, smem, st>>>((E*)dq, (E*)dk, (E*)dv, d_rpb, (const E*)d_o, (const E*)q, (const E*)k, (const E*)v, (const E*)o, lse,
                                           rpb, valid_len, gm, tps);
    })
    return cudaGetLastError();
}

// 128 rows per CTA and per residue class of a sequence
bool mma_band_supports(const Geometry& gm) {
    const long long tps = (((long long)gm.T + gm.dil - 1) / gm.dil + kBandRows - 1) / kBandRows;
    return gm.C <= 128 && gm.win <= 128 && (long long)gm.N * gm.dil * tps < (1ll << 31);
}
cudaError_t mma_band_out(float* band, const void* a, const void* b, const Geometry& gm, int dtype, cudaStream_t st) {
    const int tps = ((gm.T + gm.dil - 1) / gm.dil + kBandRows - 1) / kBandRows;
    const unsigned grid = (unsigned)((long long)gm.N * gm.dil * tps);
    NA1D_MMA_DISPATCH(dtype, gm.C, {
        auto kern = mma_band_out_kernel<E, CP>;
        const size_t smem = (size_t)band_staged(gm.win) * pitch_bytes(CP) + (size_t)kBandRows * gm.win * 4;
        if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
        kern<<<grid, kBandThreads, smem, st>>>(band, (const E*)a, (const E*)b, gm, tps);
    })
    return cudaGetLastError();
}
cudaError_t mma_band_rows(void* out, const float* band, const void* x, bool transposed, const Geometry& gm, int dtype, cudaStream_t st) {
    const int tps = ((gm.T + gm.dil - 1) / gm.dil + kBandRows - 1) / kBandRows;
    const unsigned grid = (unsigned)((long long)gm.N * gm.dil * tps);
    NA1D_MMA_DISPATCH(dtype, gm.C, {
        auto kern = transposed ? mma_band_rows_kernel<E, CP, true> : mma_band_rows_kernel<E, CP, false>;
        const size_t smem = (size_t)band_staged(gm.win) * pitch_bytes(CP) + (size_t)(transposed ? band_staged(gm.win) : kBandRows) * gm.win * 4;
        if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
        kern<<<grid, kBandThreads, smem, st>>>((E*)out, band, (const E*)x, gm, tps);
    })
    return cudaGetLastError();
}

}  // namespace na1d
