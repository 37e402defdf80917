// NA1D for narrow rows and the unfused pair: warps that march along a sequence with everything in registers.
//
// At 16 channels a row is one 32-byte sector and the operator should be bound by HBM (512 x 16 x 150 rows: 24 us forward, 43 us
// backward), but a 128-row tcgen05 tile spends most of its time in the chain TMA -> S -> softmax -> P.V -> epilogue with few
// MMAs in it, and its compute warps execute 577 instructions per 16 rows in table lookups, tensor-memory transfers, barriers
// and row bookkeeping, at 0.56 instructions a cycle (76 us forward, 141 us backward; segmented tiling 135 and 193).
//
// Here a warp owns a strip of 16-row blocks of one residue class of a sequence (tokens t = r mod dil, on which a dilated window
// is a plain one) and walks it. The window of block b is the NT = ceil((win + 15) / 16) key tiles b .. b + NT - 1, tile i being
// keys 16 i - left .. + 15, so each step brings one new tile and drops one. Keys, values (and in the backward their
// gradients) stay in registers as operands of m16n8k16 products while the window covers them; nothing passes through shared
// memory and there is no barrier:
//   * a row's channels are loaded and stored as 8 bytes per lane, in an order of the contraction index that makes lane l % 4 hold
//     channels 4 (l % 4) .. + 3 of row l / 4, both as left and as right operand;
//   * operands that contract over rows are the transposes of the same registers (movmatrix);
//   * the window offset of an accumulator element is a constant of the thread: the bias (-inf outside the window) and the bias
//     gradient are 2 (2 NT + 1) registers;
//   * keys and values outside the sequence are zero registers: only the additive mask needs a test, and only in the blocks at a
//     sequence's ends or at its padding.
// Backward: key tile i collects from blocks i - NT + 1 .. i and is stored when block i is done. A strip owns the key tiles of its
// own blocks and recomputes the NT - 1 blocks before it (nothing to recompute when the strip is a whole sequence).
// Measured at 512 x 16 x 150 rows (tcgen05 flat / segmented tiling / here, us): window 27 forward 76 / 135 / 50, backward
// 141 / 193 / 109; window 9 forward 62 / 104 / 40, backward 101 / 154 / 83; 64 x 16 x 997 rows, window 27: 66 / 66 / 37 and
// 115 / 119 / 91. Both are bound by the chain of a block at the number of warps that the registers leave (forward 16, backward 12
// an SM; more of them spill and lose). The scores' arithmetic goes in pairs (fma.rn.f32x2): backward 119 -> 111 us in a series of
// calls; the forward's window changes places by name, not by moves: 57 -> 55 us, at 32 channels 55 -> 49 (the backward's accumulators by
// name spill: 119 us). Sums over a row stay one chain a thread (in pairs, another order, they took the same time).
// Forward at 32 channels: 512 x 300 rows, window 27: 16 / 20 / 13; 4096 x 150: 49 / 85 / 45; the backward there needs more registers
// than a thread has and stays on tcgen05 (82 / 107 against 118).
// Rounding is that of the tcgen05 kernels: probabilities and dS enter the second products in 16 bits, sums are fp32.
#include "na1d_internal.h"
#include "na1d_tc_common.cuh"
#include <type_traits>

namespace na1d {
namespace {

constexpr int kWarps = 4;

__device__ __forceinline__ uint32_t transpose8(uint32_t x) {   // 8x8 16-bit matrix: row l / 4, columns 2 (l % 4), + 1
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
// d = a . b + (FRESH ? 0 : d): the first product of a sum takes a zero operand instead of cleared registers
template <typename E, bool FRESH>
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    const float c0 = FRESH ? 0.f : d[0], c1 = FRESH ? 0.f : d[1], c2 = FRESH ? 0.f : d[2], c3 = FRESH ? 0.f : d[3];
    if constexpr (std::is_same<E, __half>::value)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// pairs of fp32 values in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t&>(d))
        : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)), "l"(reinterpret_cast<const uint64_t&>(c)));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
    return d;
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// A lane's place in a tensor: row l / 4 of the current block or tile (the block's second half is 8 rows on), channels
// 4 (l % 4) .. + 3; one wide multiply-add per step
template <typename E> struct Place {
    E* p;
    int step;   // elements between rows of the residue
    __device__ __forceinline__ Place(E* base, const Strides& s, int b, int h, int r, int dil, int row, int lane)
        : p(base + b * s.batch + h * s.head + r * s.token + (long long)(row + (lane >> 2)) * (s.token * dil) + 4 * (lane & 3)), step((int)s.token * dil) {}
    __device__ __forceinline__ void next() { p += (long long)step * 16; }
    __device__ __forceinline__ E* half(int h) const { return h ? p + (long long)step * 8 : p; }
};

// 16 rows of 16 KC channels: r[h][kc] = channels 16 kc + 4 (l % 4) .. + 3 of row l / 4 + 8 h
template <int KC> struct Rows {
    uint2 r[2][KC];
    // the 16 rows at `at`, whose first is row u - l / 4 of the residue; zeros outside [0, Tr)
    template <typename E> __device__ __forceinline__ void load(const Place<E>& at, int u, int Tr) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool in = (unsigned)(u + 8 * h) < (unsigned)Tr;
#pragma unroll
            for (int kc = 0; kc < KC; ++kc)
                r[h][kc] = in ? __ldg(reinterpret_cast<const uint2*>(at.half(h) + kc * 16)) : make_uint2(0u, 0u);
        }
    }
};
// the transposes of the same registers: right operands of products that contract over the 16 rows; t[kc][j][h]: channel half j
// (channels 4 (p / 2) + 2 j + p % 2 for position p), rows 8 h .. + 7
template <int KC> struct RowsT {
    uint32_t t[KC][2][2];
    __device__ __forceinline__ void set(const Rows<KC>& x) {
#pragma unroll
        for (int kc = 0; kc < KC; ++kc)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                t[kc][0][h] = transpose8(x.r[h][kc].x);
                t[kc][1][h] = transpose8(x.r[h][kc].y);
            }
    }
};
// s0, s1 = a . b^T for b's rows 0-7 and 8-15
template <typename E, int KC> __device__ __forceinline__ void products(float (&s0)[4], float (&s1)[4], const Rows<KC>& a, const Rows<KC>& b) {
    mma<E, true>(s0, a.r[0][0].x, a.r[1][0].x, a.r[0][0].y, a.r[1][0].y, b.r[0][0].x, b.r[0][0].y);
    mma<E, true>(s1, a.r[0][0].x, a.r[1][0].x, a.r[0][0].y, a.r[1][0].y, b.r[1][0].x, b.r[1][0].y);
#pragma unroll
    for (int kc = 1; kc < KC; ++kc) {
        mma<E, false>(s0, a.r[0][kc].x, a.r[1][kc].x, a.r[0][kc].y, a.r[1][kc].y, b.r[0][kc].x, b.r[0][kc].y);
        mma<E, false>(s1, a.r[0][kc].x, a.r[1][kc].x, a.r[0][kc].y, a.r[1][kc].y, b.r[1][kc].x, b.r[1][kc].y);
    }
}
// acc (16 rows x 16 KC channels, channel order of RowsT) = (FRESH ? 0 : acc) + w . x, w a left operand over x's rows
template <typename E, int KC, bool FRESH>
__device__ __forceinline__ void accumulate(float (&acc)[KC][2][4], const uint32_t (&w)[4], const RowsT<KC>& x) {
#pragma unroll
    for (int kc = 0; kc < KC; ++kc)
#pragma unroll
        for (int j = 0; j < 2; ++j) mma<E, FRESH>(acc[kc][j], w[0], w[1], w[2], w[3], x.t[kc][j][0], x.t[kc][j][1]);
}
template <typename E, int KC>
__device__ __forceinline__ void store(const Place<E>& at, int u, int Tr, const float (&acc)[KC][2][4], float f0, float f1) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float f = h ? f1 : f0;
        if ((unsigned)(u + 8 * h) < (unsigned)Tr) {
#pragma unroll
            for (int kc = 0; kc < KC; ++kc) {
                uint2 v;
                v.x = Cvt<E>::pack2(acc[kc][0][2 * h] * f, acc[kc][0][2 * h + 1] * f);
                v.y = Cvt<E>::pack2(acc[kc][1][2 * h] * f, acc[kc][1][2 * h + 1] * f);
                *reinterpret_cast<uint2*>(at.half(h) + kc * 16) = v;
            }
        }
    }
}

// A strip: blocks [b0, b1) of 16 rows of residue r of sequence (b, h). Heads are the slowest digit, so that the warps of a CTA
// share one (their bias gradients are added up before they leave the CTA).
struct MarchGeom {
    int strips;   // strips per residue
    int len;      // blocks per strip
    int per_head; // strips of one head: batch * dil * strips
    long long total;
};
struct Strip {
    int b, h, r, b0, b1, nb, Tr, vl;
    __device__ __forceinline__ bool init(const Geometry& gm, const MarchGeom& m, const int* __restrict__ valid_len, long long id) {
        h = (int)(id / m.per_head);
        int x = (int)(id - (long long)h * m.per_head);
        const int s = x % m.strips;
        x /= m.strips;
        r = x % gm.dil;
        b = x / gm.dil;
        Tr = gm.T > r ? (gm.T - r + gm.dil - 1) / gm.dil : 0;
        nb = (Tr + 15) / 16;
        b0 = s * m.len;
        b1 = min(nb, b0 + m.len);
        const int v = valid_len ? min(gm.T, __ldg(valid_len + b)) : gm.T;
        vl = v > r ? (v - r + gm.dil - 1) / gm.dil : 0;
        return b0 < b1;
    }
};
// bias of the thread's window offsets: pair c = g - h + 1 holds offsets 8 (g - h) + fa and the next (column group g, row half h)
template <int NT> __device__ __forceinline__ void load_bias(float2 (&bias)[2 * NT + 1], const float* __restrict__ rpb, int h, int win, int fa) {
    auto at = [&](int kk) { return (unsigned)kk >= (unsigned)win ? -INFINITY : rpb ? __ldg(rpb + h * win + kk) * kLog2e : 0.f; };
#pragma unroll
    for (int c = 0; c < 2 * NT + 1; ++c) bias[c] = make_float2(at(8 * (c - 1) + fa), at(8 * (c - 1) + fa + 1));
}

template <typename E, int KC, int NT>
__global__ void __launch_bounds__(kWarps * 32) march_fwd_kernel(E* __restrict__ o, float* __restrict__ lse, const E* __restrict__ q, const E* __restrict__ k,
                                                               const E* __restrict__ v, const float* __restrict__ rpb, const int* __restrict__ valid_len,
                                                               Strides sq, Strides sk, Strides sv, Strides so, Geometry gm, MarchGeom mg) {
    const int lane = threadIdx.x & 31, fr = lane >> 2, fa = 2 * (lane & 3) - fr;
    const long long id = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    Strip st;
    if (id >= mg.total || !st.init(gm, mg, valid_len, id)) return;
    float2 bias2[2 * NT + 1];
    load_bias<NT>(bias2, rpb, st.h, gm.win, fa);
    const int right = gm.win - 1 - gm.left;
    const float sc = gm.scale * kLog2e, mask2 = kMaskValue * kLog2e;
    Place<const E> pq(q, sq, st.b, st.h, st.r, gm.dil, 16 * st.b0, lane), pk(k, sk, st.b, st.h, st.r, gm.dil, 16 * st.b0 - gm.left, lane),
        pv(v, sv, st.b, st.h, st.r, gm.dil, 16 * st.b0 - gm.left, lane);
    Place<E> po(o, so, st.b, st.h, st.r, gm.dil, 16 * st.b0, lane);
    float* lp = lse ? lse + ((long long)st.b * gm.H + st.h) * gm.T + (long long)(16 * st.b0 + fr) * gm.dil + st.r : nullptr;
    int u = 16 * st.b0 + fr, uk = u - gm.left;   // this lane's first query row; its first row of the next key tile
    // The window's tiles change places by name, not by moves: step PH (of NT, unrolled) finds tile t of its window in slot (PH + t) % NT,
    // and the tile after the window takes slot PH.
    Rows<KC> kf[NT], q_, vn;
    RowsT<KC> vt[NT];
    auto next_tile = [&](Rows<KC>& kr) {
        kr.load(pk, uk, st.Tr);
        vn.load(pv, uk, st.Tr);
        pk.next(); pv.next(); uk += 16;
    };
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        next_tile(kf[t]);
        if (t + 1 < NT) vt[t].set(vn);
    }
    q_.load(pq, u, st.Tr);
    auto step = [&](int b, auto phase) {
        constexpr int PH = decltype(phase)::value;
        vt[(PH + NT - 1) % NT].set(vn);
        float s[2 * NT][4], mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
        for (int t = 0; t < NT; ++t) products<E, KC>(s[2 * t], s[2 * t + 1], q_, kf[(PH + t) % NT]);
        // the next block's rows are on their way while this one is worked on
        pq.next();
        q_.load(pq, u + 16, st.Tr);
        next_tile(kf[PH]);
        const bool need_mask = 16 * b < gm.left || 16 * b + 15 + right >= st.vl;
#pragma unroll
        for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 x = fma2(make_float2(s[g][2 * h], s[g][2 * h + 1]), both(sc), bias2[g - h + 1]);
                s[g][2 * h] = x.x; s[g][2 * h + 1] = x.y;
            }
        if (need_mask) {
#pragma unroll
            for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int row = u + 8 * (i >> 1), j = row - gm.left + 8 * (g - (i >> 1)) + (i & 1) + fa;
                    if (j < 0 || j >= st.vl || row >= st.vl) s[g][i] += mask2;
                }
        }
#pragma unroll
        for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
            for (int h = 0; h < 2; ++h) mx[h] = max3(mx[h], s[g][2 * h], s[g][2 * h + 1]);
        mx[0] = tc::quad_max(mx[0]);
        mx[1] = tc::quad_max(mx[1]);
        float acc[KC][2][4];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int g = 2 * t; g < 2 * t + 2; ++g)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = add2(make_float2(s[g][2 * h], s[g][2 * h + 1]), both(-mx[h]));
                    s[g][2 * h] = tc::fast_exp2(x.x);
                    s[g][2 * h + 1] = tc::fast_exp2(x.y);
                    l[h] += s[g][2 * h];
                    l[h] += s[g][2 * h + 1];
                }
            const uint32_t w[4] = {Cvt<E>::pack2(s[2 * t][0], s[2 * t][1]), Cvt<E>::pack2(s[2 * t][2], s[2 * t][3]),
                                   Cvt<E>::pack2(s[2 * t + 1][0], s[2 * t + 1][1]), Cvt<E>::pack2(s[2 * t + 1][2], s[2 * t + 1][3])};
            if (t == 0) accumulate<E, KC, true>(acc, w, vt[PH]); else accumulate<E, KC, false>(acc, w, vt[(PH + t) % NT]);
        }
        l[0] = tc::quad_sum(l[0]);
        l[1] = tc::quad_sum(l[1]);
        store<E, KC>(po, u, st.Tr, acc, tc::fast_rcp(l[0]), tc::fast_rcp(l[1]));
        po.next();
        if (lse) {
            if ((lane & 3) == 0) {
                if (u < st.Tr) lp[0] = (mx[0] + tc::fast_log2(l[0])) * kLn2;
                if (u + 8 < st.Tr) lp[8 * gm.dil] = (mx[1] + tc::fast_log2(l[1])) * kLn2;
            }
            lp += 16 * gm.dil;
        }
        u += 16;
    };
#pragma unroll 1
    for (int b = st.b0; b < st.b1; b += NT) {
        step(b, std::integral_constant<int, 0>());
        if (b + 1 < st.b1) step(b + 1, std::integral_constant<int, 1>());
        if (NT == 3 && b + 2 < st.b1) step(b + 2, std::integral_constant<int, NT - 1>());
    }
}

// ---------------------------------------------------------------- backward, 16 channels
// The forward's march with four tensors and two sets of key gradients in flight would take 225 registers and leave eight warps on an SM
// (136 us at 512 x 16 x 150 rows, window 27, bound by latency). So the operands wait in shared memory instead: per warp a
// ring of four key tiles each of k and v and two blocks each of q and d_o, copied asynchronously one step ahead (16 rows x 32
// bytes: one 16-byte copy per lane), and read by ldmatrix, plain or transposed, where they are used.
constexpr int kTileBytes = 16 * 32;
struct WarpTiles {
    uint32_t k, v, q, o;   // shared addresses: rings of 4, 4, 2, 2 tiles
    uint32_t copy, plain, rows;   // this lane's offsets in a tile: its copy, its ldmatrix row as a right operand over channels, and as
                                  // a left operand or a right operand over rows
    __device__ __forceinline__ static uint32_t at(int row, int chunk) { return row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4); }   // conflict-free
    __device__ __forceinline__ WarpTiles(uint32_t base, int lane)
        : k(base), v(base + 4 * kTileBytes), q(base + 8 * kTileBytes), o(base + 10 * kTileBytes), copy(at(lane >> 1, lane & 1)),
          plain(at((lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1)), rows(at((lane & 7) + (((lane >> 3) & 1) << 3), lane >> 4)) {}
};
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool in) {   // zeros where `in` is false
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// acc (16 rows x channels 0-7, 8-15) = (FRESH ? 0 : acc) + w . x
template <typename E, bool FRESH> __device__ __forceinline__ void add_rows(float (&acc)[2][4], const uint32_t (&w)[4], const uint32_t (&x)[4]) {
    mma<E, FRESH>(acc[0], w[0], w[1], w[2], w[3], x[0], x[1]);
    mma<E, FRESH>(acc[1], w[0], w[1], w[2], w[3], x[2], x[3]);
}
// a lane's place in an output: row l / 4 of the block, channels 2 (l % 4), + 1 of each half
template <typename E> struct OutPlace {
    E* p;
    int step;
    __device__ __forceinline__ OutPlace(E* base, const Strides& s, const Strip& st, int dil, int row, int lane)
        : p(base + st.b * s.batch + st.h * s.head + st.r * s.token + (long long)(row + (lane >> 2)) * (s.token * dil) + 2 * (lane & 3)), step((int)s.token * dil) {}
    __device__ __forceinline__ void next() { p += (long long)step * 16; }
    __device__ __forceinline__ void store(int u, int Tr, const float (&acc)[2][4]) const {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if ((unsigned)(u + 8 * h) < (unsigned)Tr) {
                E* d = h ? p + (long long)step * 8 : p;
                *reinterpret_cast<uint32_t*>(d) = Cvt<E>::pack2(acc[0][2 * h], acc[0][2 * h + 1]);
                *reinterpret_cast<uint32_t*>(d + 8) = Cvt<E>::pack2(acc[1][2 * h], acc[1][2 * h + 1]);
            }
    }
};
// and in an input: row l / 2 of the block, channels 8 (l % 2) .. + 7
template <typename E> struct InPlace {
    const E* p;
    int step;
    __device__ __forceinline__ InPlace(const E* base, const Strides& s, const Strip& st, int dil, int row, int lane)
        : p(base + st.b * s.batch + st.h * s.head + st.r * s.token + (long long)(row + (lane >> 1)) * (s.token * dil) + 8 * (lane & 1)), step((int)s.token * dil) {}
    // copies the 16 rows, of which this lane's is row u of the residue, and moves on
    __device__ __forceinline__ void copy(uint32_t dst, int u, int Tr, const E* safe) {
        const bool in = (unsigned)u < (unsigned)Tr;
        copy16(dst, in ? p : safe, in);
        p += (long long)step * 16;
    }
};

template <typename E, int NT>
__global__ void __launch_bounds__(kWarps * 32, NT == 3 ? 3 : 4) march_bwd_kernel(E* __restrict__ dq, E* __restrict__ dk, E* __restrict__ dv, float* __restrict__ d_rpb,
                                                               const E* __restrict__ d_o, const E* __restrict__ q, const E* __restrict__ k,
                                                               const E* __restrict__ v, const float* __restrict__ lse, const float* __restrict__ rpb,
                                                               const int* __restrict__ valid_len, Strides sdq, Strides sdk, Strides sdv, Strides sdo,
                                                               Strides sq, Strides sk, Strides sv, Geometry gm, MarchGeom mg) {
    __shared__ __align__(128) uint8_t tiles[kWarps][12 * kTileBytes];
    __shared__ float s_rpb[kWarps][16 * NT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fa = 2 * (lane & 3) - fr;
    const long long id = (long long)blockIdx.x * kWarps + warp;
    Strip st;
    const bool alive = id < mg.total && st.init(gm, mg, valid_len, id);
    float2 grad[2 * NT + 1];
#pragma unroll
    for (int c = 0; c < 2 * NT + 1; ++c) grad[c] = both(0.f);
    if (alive) {
        float2 bias[2 * NT + 1];
        load_bias<NT>(bias, rpb, st.h, gm.win, fa);
        const int right = gm.win - 1 - gm.left, first = max(0, st.b0 - (NT - 1));
        const float sc = gm.scale * kLog2e, mask2 = kMaskValue * kLog2e;
        const WarpTiles tl(ptx::smem_u32(tiles[warp]), lane);
        InPlace<E> pq(q, sq, st, gm.dil, 16 * first, lane), po(d_o, sdo, st, gm.dil, 16 * first, lane), pk(k, sk, st, gm.dil, 16 * first - gm.left, lane),
            pv(v, sv, st, gm.dil, 16 * first - gm.left, lane);
        OutPlace<E> pdq(dq, sdq, st, gm.dil, 16 * first, lane), pdk(dk, sdk, st, gm.dil, 16 * first - gm.left, lane),
            pdv(dv, sdv, st, gm.dil, 16 * first - gm.left, lane);
        const float* lp = lse + ((long long)st.b * gm.H + st.h) * gm.T + (long long)(16 * first + fr) * gm.dil + st.r;
        int u = 16 * first + fr;                        // this lane's first query row as an accumulator holds it
        auto copy_queries = [&](int b) {
            const int row = 16 * b + (lane >> 1);
            pq.copy(tl.q + (b & 1) * kTileBytes + tl.copy, row, st.Tr, q);
            po.copy(tl.o + (b & 1) * kTileBytes + tl.copy, row, st.Tr, d_o);
        };
        auto copy_keys = [&](int t) {
            const int row = 16 * t - gm.left + (lane >> 1);
            pk.copy(tl.k + (t & 3) * kTileBytes + tl.copy, row, st.Tr, k);
            pv.copy(tl.v + (t & 3) * kTileBytes + tl.copy, row, st.Tr, v);
        };
        float ln[2];
        auto load_lse = [&](int row) {   // +inf for rows outside the sequence: probability 0
            ln[0] = row < st.Tr ? __ldg(lp) * kLog2e : INFINITY;
            ln[1] = row + 8 < st.Tr ? __ldg(lp + 8 * gm.dil) * kLog2e : INFINITY;
            lp += 16 * gm.dil;
        };
        float ak[NT][2][4], av[NT][2][4];
#pragma unroll
        for (int t = 0; t + 1 < NT; ++t)
#pragma unroll
            for (int i = 0; i < 8; ++i) ak[t][i >> 2][i & 3] = av[t][i >> 2][i & 3] = 0.f;
        for (int t = 0; t < NT; ++t) copy_keys(first + t);
        copy_queries(first);
        asm volatile("cp.async.commit_group;" ::: "memory");
        load_lse(u);
#pragma unroll 1
        for (int b = first; b < st.b1; ++b, u += 16) {
            const bool own = b >= st.b0;
            const float l2[2] = {ln[0], ln[1]};
            // the next block's rows (tile b + NT takes the slot of tile b + NT - 4, which the block before read last)
            copy_queries(b + 1);
            copy_keys(b + NT);
            asm volatile("cp.async.commit_group;" ::: "memory");
            load_lse(u + 16);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const uint32_t tq = tl.q + (b & 1) * kTileBytes, to = tl.o + (b & 1) * kTileBytes;
            float s[2 * NT][4], d[2 * NT][4], delta[2];
            float2 part[2][2] = {{both(0.f), both(0.f)}, {both(0.f), both(0.f)}};   // (two chains per row keep the sums short)
            {
                uint32_t qa[4], oa[4];
                ldsm(qa, tq + tl.rows);
                ldsm(oa, to + tl.rows);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const uint32_t slot = ((b + t) & 3) * kTileBytes;
                    uint32_t x[4];
                    ldsm(x, tl.k + slot + tl.plain);
                    mma<E, true>(s[2 * t], qa[0], qa[1], qa[2], qa[3], x[0], x[1]);
                    mma<E, true>(s[2 * t + 1], qa[0], qa[1], qa[2], qa[3], x[2], x[3]);
                    ldsm(x, tl.v + slot + tl.plain);
                    mma<E, true>(d[2 * t], oa[0], oa[1], oa[2], oa[3], x[0], x[1]);
                    mma<E, true>(d[2 * t + 1], oa[0], oa[1], oa[2], oa[3], x[2], x[3]);
                }
            }
            const bool need_mask = 16 * b < gm.left || 16 * b + 15 + right >= st.vl;
#pragma unroll
            for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = fma2(make_float2(s[g][2 * h], s[g][2 * h + 1]), both(sc), bias[g - h + 1]);
                    s[g][2 * h] = x.x; s[g][2 * h + 1] = x.y;
                }
            if (need_mask) {
#pragma unroll
                for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = u + 8 * (i >> 1), j = row - gm.left + 8 * (g - (i >> 1)) + (i & 1) + fa;
                        if (j < 0 || j >= st.vl || row >= st.vl) s[g][i] += mask2;
                    }
            }
#pragma unroll
            for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = add2(make_float2(s[g][2 * h], s[g][2 * h + 1]), both(-l2[h]));
                    s[g][2 * h] = tc::fast_exp2(x.x);
                    s[g][2 * h + 1] = tc::fast_exp2(x.y);
                    part[g & 1][h] = fma2(make_float2(s[g][2 * h], s[g][2 * h + 1]), make_float2(d[g][2 * h], d[g][2 * h + 1]), part[g & 1][h]);
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) delta[h] = tc::quad_sum((part[0][h].x + part[0][h].y) + (part[1][h].x + part[1][h].y));
#pragma unroll
            for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = mul2(make_float2(s[g][2 * h], s[g][2 * h + 1]), add2(make_float2(d[g][2 * h], d[g][2 * h + 1]), both(-delta[h])));
                    d[g][2 * h] = x.x; d[g][2 * h + 1] = x.y;
                }
            if (own && d_rpb) {
#pragma unroll
                for (int g = 0; g < 2 * NT; ++g)
#pragma unroll
                    for (int h = 0; h < 2; ++h) grad[g - h + 1] = add2(grad[g - h + 1], make_float2(d[g][2 * h], d[g][2 * h + 1]));
            }
            uint32_t qt[4], ot[4];
            ldsm_t(qt, tq + tl.rows);
            ldsm_t(ot, to + tl.rows);
            float acc[2][4];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                // left operands over the keys: (rows 0-7, keys 0-7), (rows 8-15, keys 0-7), (rows 0-7, keys 8-15), (rows 8-15, keys 8-15)
                uint32_t w[4], x[4], kt[4];
                ldsm_t(kt, tl.k + ((b + t) & 3) * kTileBytes + tl.rows);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int g = 2 * t + (i >> 1), h = 2 * (i & 1);
                    const float2 y = mul2(make_float2(d[g][h], d[g][h + 1]), both(gm.scale));
                    w[i] = Cvt<E>::pack2(y.x, y.y);
                    x[i] = Cvt<E>::pack2(s[g][h], s[g][h + 1]);
                }
                if (t == 0) add_rows<E, true>(acc, w, kt); else add_rows<E, false>(acc, w, kt);
                // and transposed, over the queries: the off-diagonal matrices change places
                const uint32_t wt[4] = {transpose8(w[0]), transpose8(w[2]), transpose8(w[1]), transpose8(w[3])};
                const uint32_t xt[4] = {transpose8(x[0]), transpose8(x[2]), transpose8(x[1]), transpose8(x[3])};
                if (t + 1 == NT) { add_rows<E, true>(ak[t], wt, qt); add_rows<E, true>(av[t], xt, ot); }   // (the newest tile)
                else { add_rows<E, false>(ak[t], wt, qt); add_rows<E, false>(av[t], xt, ot); }
            }
            __syncwarp();   // the slots are read: the next step's copies may overwrite them
            if (own) {
                pdq.store(u, st.Tr, acc);
                pdk.store(u - gm.left, st.Tr, ak[0]);
                pdv.store(u - gm.left, st.Tr, av[0]);
            }
            pdq.next(); pdk.next(); pdv.next();
#pragma unroll
            for (int t = 0; t + 1 < NT; ++t)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    ak[t][i >> 2][i & 3] = ak[t + 1][i >> 2][i & 3];
                    av[t][i >> 2][i & 3] = av[t + 1][i >> 2][i & 3];
                }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (st.b1 == st.nb) {   // the sequence's last strip owns the tiles behind its last block too
#pragma unroll
            for (int t = 0; t + 1 < NT; ++t) {
                pdk.store(u - gm.left, st.Tr, ak[t]);
                pdv.store(u - gm.left, st.Tr, av[t]);
                pdk.next(); pdv.next(); u += 16;
            }
        }
    }
    if (d_rpb) {
        // A window offset is spread over the lanes with the same offset modulo 8: eight of the warp's registers, added up through
        // shared memory (the drained rings) in a fixed order. Shared-memory atomics took 2.5 us here, a third of a small call:
        // 1 x 1 x 1400 rows, window 27, 9.6 us.
        static_assert((4 * NT + 2) * 32 * 4 <= sizeof(tiles[0]), "a warp's rings hold its gradients");
        float* sums = reinterpret_cast<float*>(tiles[warp]);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 2 * NT + 1; ++c) { sums[2 * c * 32 + lane] = grad[c].x; sums[(2 * c + 1) * 32 + lane] = grad[c].y; }
        __syncwarp();
        for (int kk = lane; kk < gm.win; kk += 32) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {   // lane 4 b + a holds offset 8 (c / 2 - 1) + c % 2 + 2 a - b in register c
                const int a = i >> 1, b = (2 * a - kk + (i & 1)) & 7, c = (kk + 8 - 2 * a + b) >> 3;
                sum += sums[(2 * c + (i & 1)) * 32 + 4 * b + a];
            }
            s_rpb[warp][kk] = sum;
        }
        __syncthreads();
        // warps of one head are neighbours: a run of them is added up and handed over once
        const long long id0 = (long long)blockIdx.x * kWarps;
        for (int kk = threadIdx.x; kk < gm.win; kk += kWarps * 32) {
            float sum = 0.f;
            for (int w = 0; w < kWarps && id0 + w < mg.total; ++w) {
                const int h = (int)((id0 + w) / mg.per_head);
                sum += s_rpb[w][kk];
                if (w + 1 == kWarps || id0 + w + 1 >= mg.total || (int)((id0 + w + 1) / mg.per_head) != h) {
                    atomicAdd(d_rpb + h * gm.win + kk, sum);
                    sum = 0.f;
                }
            }
        }
    }
}

// ---------------------------------------------------------------- the unfused pair (dilation 1)
// The same march with the fp32 band in memory: a block's 16 band rows are one contiguous piece, moved in whole lines through a
// 16 x (16 NT + 8) patch of shared memory per warp in which entry (row, kk) stands at column row + kk, the accumulator's own
// order (pitch 8 mod 32 words: 8-byte accesses without bank conflicts). Positions outside the band are never written and
// stay zero. The patch offsets of a lane's elements are the same in every block and are kept in registers.
// Measured (tcgen05 / warp-level products on 128-row tiles / here, us; HBM time is 33, 38 and 26):
// 8192 x 150 x 16, window 27: q.k 58 / 67 / 42, a.v 81 / 102 / 49, transposed 182 (CUDA core 120) / 116 / 59 (three pieces);
// 6912 x 150 x 32, window 27: 54 / 72 / 47, 78 / 106 / 53, 159 / 122 / 56; 3456 x 150 x 64, window 17: 33 / 52 / 33, 42 / 73 / 38,
// 76 / 75 / 38.
//   march_qk  : band[t, kk] = a[t] . b[j]             (QK forward, dA)
//   march_rows: out[t] = sum band[t, kk] x[j]         (AV forward, dQ), or TRANSPOSED out[j] = sum band[t, kk] x[t] (dV, dK)
// The band enters the products as two 16-bit pieces where the tcgen05 kernels round it to one; the transposed product at 16 and 64 channels
// and windows above 17, which those leave to the CUDA cores, takes three bf16 pieces, all its bits (10 % of that kernel's time). A result that is not finite is computed again, row by row in fp32: the
// zeros outside the band must not meet an infinite row.
template <int NT> constexpr int kPatchPitch = 16 * NT + 8;
template <int NT> constexpr int kPatchIters = (16 * (16 * NT - 15) + 31) / 32;   // 32-element steps of 16 band rows
template <int NT> __device__ __forceinline__ void patch_offsets(int (&off)[kPatchIters<NT>], int win, int lane) {
#pragma unroll
    for (int it = 0; it < kPatchIters<NT>; ++it) {
        const int i = it * 32 + lane, row = i / win;
        off[it] = i < 16 * win ? row * kPatchPitch<NT> + row + (i - row * win) : -1;
    }
}

template <typename E, int KC, int NT>
__global__ void __launch_bounds__(kWarps * 32) march_qk_kernel(float* __restrict__ band, const E* __restrict__ a, const E* __restrict__ b_, Strides sd,
                                                              Geometry gm, MarchGeom mg) {
    __shared__ float patch_all[kWarps][16 * kPatchPitch<NT>];
    const int lane = threadIdx.x & 31, fr = lane >> 2;
    const long long id = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    Strip st;
    if (id >= mg.total || !st.init(gm, mg, nullptr, id)) return;
    float* patch = patch_all[threadIdx.x >> 5];
    int off[kPatchIters<NT>];
    patch_offsets<NT>(off, gm.win, lane);
    Place<const E> pa(a, sd, st.b, 0, 0, 1, 16 * st.b0, lane), pb(b_, sd, st.b, 0, 0, 1, 16 * st.b0 - gm.left, lane);
    float* dst = band + ((long long)st.b * gm.T + 16 * st.b0) * gm.win;
    int u = 16 * st.b0 + fr, uk = u - gm.left;
    Rows<KC> kf[NT], qn, kn;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        kn.load(pb, uk, st.Tr);
        pb.next(); uk += 16;
        if (t + 1 < NT) kf[t + 1] = kn;
    }
    qn.load(pa, u, st.Tr);
#pragma unroll 1
    for (int b = st.b0; b < st.b1; ++b, u += 16) {
#pragma unroll
        for (int t = 0; t + 1 < NT; ++t) kf[t] = kf[t + 1];
        kf[NT - 1] = kn;
        const Rows<KC> qf = qn;
        pa.next();
        qn.load(pa, u + 16, st.Tr);
        kn.load(pb, uk, st.Tr);
        pb.next(); uk += 16;
        const bool edge = 16 * b < gm.left || 16 * b + 15 + gm.win - 1 - gm.left >= st.Tr;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            float s[2][4];
            products<E, KC>(s[0], s[1], qf, kf[t]);
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = 16 * t + 8 * g + 2 * (lane & 3);
                    float2 v = make_float2(s[g][2 * h], s[g][2 * h + 1]);
                    if (edge) {   // a key outside the sequence gives 0 whatever the query holds
                        const int j = 16 * b - gm.left + c;
                        if ((unsigned)j >= (unsigned)st.Tr) v.x = 0.f;
                        if ((unsigned)(j + 1) >= (unsigned)st.Tr) v.y = 0.f;
                    }
                    *reinterpret_cast<float2*>(patch + (fr + 8 * h) * kPatchPitch<NT> + c) = v;
                }
        }
        __syncwarp();
        const int live = min(16, st.Tr - 16 * b) * gm.win;
#pragma unroll
        for (int it = 0; it < kPatchIters<NT>; ++it)
            if (it * 32 + lane < live) dst[it * 32 + lane] = patch[off[it]];
        dst += 16 * gm.win;
        __syncwarp();
    }
}

// 16 result rows from `first` on, by plain fp32 sums: two lanes per row
template <typename E, int KC, bool TRANSPOSED>
__device__ __noinline__ void plain_rows16(E* out, const float* band, const E* x, int seq, int first, Geometry gm) {
    const int lane = threadIdx.x & 31, row = first + (lane >> 1);
    if (row < 0 || row >= gm.T) return;
    for (int c0 = 8 * (lane & 1); c0 < 16 * KC; c0 += 16) {
        float acc[8] = {};
        for (int kk = 0; kk < gm.win; ++kk) {
            const int w = TRANSPOSED ? row - (kk - gm.left) : row + kk - gm.left;
            if (w < 0 || w >= gm.T) continue;
            const float f = __ldg(band + ((long long)seq * gm.T + (TRANSPOSED ? w : row)) * gm.win + kk);
            float v[8];
            Cvt<E>::unpack(__ldg(reinterpret_cast<const uint4*>(x + ((long long)seq * gm.T + w) * (16 * KC) + c0)), v);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = fmaf(f, v[i], acc[i]);
        }
        *reinterpret_cast<uint4*>(out + ((long long)seq * gm.T + row) * (16 * KC) + c0) = Cvt<E>::pack(acc);
    }
}

template <typename E, int KC, int NT, bool TRANSPOSED>
__global__ void __launch_bounds__(kWarps * 32) march_rows_kernel(E* __restrict__ out, const float* __restrict__ band, const E* __restrict__ x, Strides sd,
                                                                Geometry gm, MarchGeom mg) {
    __shared__ float patch_all[kWarps][16 * kPatchPitch<NT>];
    const int lane = threadIdx.x & 31, fr = lane >> 2;
    const long long id = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    Strip st;
    if (id >= mg.total || !st.init(gm, mg, nullptr, id)) return;
    float* patch = patch_all[threadIdx.x >> 5];
    for (int i = lane; i < 16 * kPatchPitch<NT>; i += 32) patch[i] = 0.f;
    int off[kPatchIters<NT>];
    patch_offsets<NT>(off, gm.win, lane);
    const int first = TRANSPOSED ? max(0, st.b0 - (NT - 1)) : st.b0, lead = TRANSPOSED ? 0 : gm.left;
    // x: key tiles (AV), or the block's own rows (transposed)
    Place<const E> px(x, sd, st.b, 0, 0, 1, 16 * first - lead, lane);
    Place<E> po(out, sd, st.b, 0, 0, 1, 16 * first - (TRANSPOSED ? gm.left : 0), lane);
    const float* src = band + ((long long)st.b * gm.T + 16 * first) * gm.win;
    int u = 16 * first + fr, ux = u - lead;
    float bn[kPatchIters<NT>];
    auto load_band = [&](int b) {
        const int live = min(16, st.Tr - 16 * b) * gm.win;
#pragma unroll
        for (int it = 0; it < kPatchIters<NT>; ++it) bn[it] = it * 32 + lane < live ? __ldg(src + it * 32 + lane) : 0.f;
        src += 16 * gm.win;
    };
    Rows<KC> xn;
    RowsT<KC> xt[TRANSPOSED ? 1 : NT];
    float acc[TRANSPOSED ? NT : 1][KC][2][4];
    constexpr int TILES = TRANSPOSED ? 1 : NT, PIECES = TRANSPOSED && NT == 3 && KC != 2 ? 3 : 2;
#pragma unroll
    for (int t = 0; t < TILES; ++t) {
        xn.load(px, ux, st.Tr);
        px.next(); ux += 16;
        if (t + 1 < TILES) xt[t + 1].set(xn);
    }
    if constexpr (TRANSPOSED) {
#pragma unroll
        for (int t = 0; t + 1 < NT; ++t)
#pragma unroll
            for (int i = 0; i < 8 * KC; ++i) acc[t][i >> 3][(i >> 2) & 1][i & 3] = 0.f;
    }
    load_band(first);
    auto finish = [&](int row0, const float (&r)[KC][2][4]) {   // row0: first row of the 16
        float z = 0.f;
#pragma unroll
        for (int i = 0; i < 8 * KC; ++i) z = fmaf(r[i >> 3][(i >> 2) & 1][i & 3], 0.f, z);
        if (__any_sync(0xffffffffu, z != 0.f)) plain_rows16<E, KC, TRANSPOSED>(out, band, x, st.b, row0, gm);
        else store<E, KC>(po, row0 + fr, st.Tr, r, 1.f, 1.f);
    };
    __syncwarp();
#pragma unroll 1
    for (int b = first; b < st.b1; ++b, u += 16) {
#pragma unroll
        for (int t = 0; t + 1 < TILES; ++t) xt[t] = xt[t + 1];
        xt[TILES - 1].set(xn);
#pragma unroll
        for (int it = 0; it < kPatchIters<NT>; ++it)
            if (off[it] >= 0) patch[off[it]] = bn[it];
        __syncwarp();
        if (b + 1 < st.b1) {
            load_band(b + 1);
            xn.load(px, ux, st.Tr);
            px.next(); ux += 16;
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            uint32_t piece[PIECES][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float2 p = *reinterpret_cast<const float2*>(patch + (fr + 8 * (i & 1)) * kPatchPitch<NT> + 16 * t + 8 * (i >> 1) + 2 * (lane & 3));
#pragma unroll
                for (int k = 0; k < PIECES; ++k) {
                    piece[k][i] = Cvt<E>::pack2(p.x, p.y);
                    p.x -= Cvt<E>::from_bits((unsigned short)(piece[k][i] & 0xffffu));
                    p.y -= Cvt<E>::from_bits((unsigned short)(piece[k][i] >> 16));
                }
            }
#pragma unroll
            for (int k = 0; k < PIECES; ++k) {
                if constexpr (TRANSPOSED) {
                    const uint32_t w[4] = {transpose8(piece[k][0]), transpose8(piece[k][2]), transpose8(piece[k][1]), transpose8(piece[k][3])};
                    if (k == 0 && t + 1 == NT) accumulate<E, KC, true>(acc[t], w, xt[0]); else accumulate<E, KC, false>(acc[t], w, xt[0]);
                } else {
                    if (k == 0 && t == 0) accumulate<E, KC, true>(acc[0], piece[k], xt[t]); else accumulate<E, KC, false>(acc[0], piece[k], xt[t]);
                }
            }
        }
        __syncwarp();
        if (!TRANSPOSED || b >= st.b0) finish(16 * b - (TRANSPOSED ? gm.left : 0), acc[0]);
        po.next();
        if constexpr (TRANSPOSED) {
#pragma unroll
            for (int t = 0; t + 1 < NT; ++t)
#pragma unroll
                for (int i = 0; i < 8 * KC; ++i) acc[t][i >> 3][(i >> 2) & 1][i & 3] = acc[t + 1][i >> 3][(i >> 2) & 1][i & 3];
        }
    }
    if constexpr (TRANSPOSED)
        if (st.b1 == st.nb) {
#pragma unroll
            for (int t = 0; t + 1 < NT; ++t) {
                finish(16 * (st.b1 + t) - gm.left, acc[t]);
                po.next();
            }
        }
}

// Blocks per strip. The GPU runs `resident` warps of the kernel per SM at a time, a strip costs its blocks and `extra` blocks' worth
// of start-up (first loads; in the backward the recomputed blocks): the number of strips per residue whose rounds of warps
// take the fewest block steps. Measured (backward, 1024 sequences of 63 blocks, 1776 warps at a time): 1 strip 111 us, 2 (one and
// a bit rounds) 121, 3 (1.7 rounds) 98, 4 (2.3 rounds) 109.
MarchGeom march_geom(const Geometry& gm, int resident, int extra) {
    MarchGeom m;
    const int nb = ((gm.T + gm.dil - 1) / gm.dil + 15) / 16, batch = gm.N / gm.H;
    const long long residues = (long long)gm.N * gm.dil, room = (long long)resident * device_sm_count();
    long long best = 0;
    m.strips = 1;
    for (int s = 1; s <= nb; s += s < 16 ? 1 : s / 8) {
        const long long cost = ((residues * s + room - 1) / room) * ((nb + s - 1) / s + extra);
        if (s == 1 || cost < best) { best = cost; m.strips = s; }
    }
    m.len = (nb + m.strips - 1) / m.strips;
    m.per_head = batch * gm.dil * m.strips;
    m.total = (long long)m.per_head * gm.H;
    return m;
}

// warps of a kernel that an SM holds (asked once per kernel)
int resident_warps(const void* kern) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, kWarps * 32, 0) != cudaSuccess || n < 1) n = 1;
    return n * kWarps;
}
// launches kern<<<...>>>(arguments..., gm, m) with its own strips
#define NA1D_MARCH_LAUNCH(EXTRA, KERN, ...)                                                          \
    do {                                                                                             \
        static const int warps = resident_warps(reinterpret_cast<const void*>(KERN));                \
        const MarchGeom m = march_geom(gm, warps, EXTRA);                                            \
        KERN<<<(unsigned)((m.total + kWarps - 1) / kWarps), kWarps * 32, 0, st>>>(__VA_ARGS__, gm, m); \
    } while (0)

}  // namespace

// 16-channel rows (forward: 32 too; the backward's registers hold 16), windows up to 33 (three key tiles), any dilation, token
// count and number of heads
bool march_supports(const Geometry& gm, bool backward) {
    const long long nb = ((long long)gm.T + 15) / 16 + gm.dil;
    return (gm.C == 16 || (gm.C == 32 && !backward)) && gm.win <= 33 && (long long)gm.N * nb * 2 < (1ll << 31);
}

cudaError_t march_fused_fwd(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb, const int* valid_len,
                            const Strides& sq, const Strides& sk, const Strides& sv, const Strides& so, const Geometry& gm, int dtype, cudaStream_t st) {
#define NA1D_MARCH(E, KC, NT)                                                                                                                        \
    NA1D_MARCH_LAUNCH(2, (march_fwd_kernel<E, KC, NT>), (E*)o, lse, (const E*)q, (const E*)k, (const E*)v, rpb, valid_len, sq, sk, sv, so)
#define NA1D_MARCH_E(E)                                                                 \
    if (gm.C == 16) { if (gm.win <= 17) NA1D_MARCH(E, 1, 2); else NA1D_MARCH(E, 1, 3); } \
    else { if (gm.win <= 17) NA1D_MARCH(E, 2, 2); else NA1D_MARCH(E, 2, 3); }
    if (dtype == 0) { NA1D_MARCH_E(__nv_bfloat16) } else { NA1D_MARCH_E(__half) }
#undef NA1D_MARCH
#undef NA1D_MARCH_E
    return cudaGetLastError();
}
cudaError_t march_fused_bwd(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k, const void* v, const float* lse,
                            const float* rpb, const int* valid_len, const Strides& sdq, const Strides& sdk, const Strides& sdv, const Strides& sdo,
                            const Strides& sq, const Strides& sk, const Strides& sv, const Geometry& gm, int dtype, cudaStream_t st) {
#define NA1D_MARCH(E, NT)                                                                                                                     \
    NA1D_MARCH_LAUNCH(NT, (march_bwd_kernel<E, NT>), (E*)dq, (E*)dk, (E*)dv, d_rpb, (const E*)d_o, (const E*)q, (const E*)k, (const E*)v, lse, \
                      rpb, valid_len, sdq, sdk, sdv, sdo, sq, sk, sv)
    if (dtype == 0) { if (gm.win <= 17) NA1D_MARCH(__nv_bfloat16, 2); else NA1D_MARCH(__nv_bfloat16, 3); }
    else { if (gm.win <= 17) NA1D_MARCH(__half, 2); else NA1D_MARCH(__half, 3); }
#undef NA1D_MARCH
    return cudaGetLastError();
}

// the pair: 16, 32 or 64 channels, one head (sequences), dilation 1
bool march_band_supports(const Geometry& gm) {
    const long long nb = ((long long)gm.T + 15) / 16 + 1;
    return (gm.C == 16 || gm.C == 32 || gm.C == 64) && gm.win <= 33 && gm.dil == 1 && gm.H == 1 && (long long)gm.N * nb * 2 < (1ll << 31) &&
           (long long)gm.T * gm.win < (1ll << 31);
}
#define NA1D_MARCH_E(E)                                                                        \
    if (gm.C == 16) { if (gm.win <= 17) NA1D_MARCH(E, 1, 2); else NA1D_MARCH(E, 1, 3); }        \
    else if (gm.C == 32) { if (gm.win <= 17) NA1D_MARCH(E, 2, 2); else NA1D_MARCH(E, 2, 3); }   \
    else { if (gm.win <= 17) NA1D_MARCH(E, 4, 2); else NA1D_MARCH(E, 4, 3); }
cudaError_t march_band_out(float* band, const void* a, const void* b, const Geometry& gm, int dtype, cudaStream_t st) {
    const Strides d = dense_strides(1, gm.T, gm.C);
#define NA1D_MARCH(E, KC, NT) NA1D_MARCH_LAUNCH(2, (march_qk_kernel<E, KC, NT>), band, (const E*)a, (const E*)b, d)
    if (dtype == 0) { NA1D_MARCH_E(__nv_bfloat16) } else { NA1D_MARCH_E(__half) }
#undef NA1D_MARCH
    return cudaGetLastError();
}
cudaError_t march_band_rows(void* out, const float* band, const void* x, bool transposed, const Geometry& gm, int dtype, cudaStream_t st) {
    const Strides d = dense_strides(1, gm.T, gm.C);
#define NA1D_MARCH(E, KC, NT)                                                                                          \
    do {                                                                                                               \
        if (transposed) NA1D_MARCH_LAUNCH(NT, (march_rows_kernel<E, KC, NT, true>), (E*)out, band, (const E*)x, d);     \
        else NA1D_MARCH_LAUNCH(2, (march_rows_kernel<E, KC, NT, false>), (E*)out, band, (const E*)x, d);                \
    } while (0)
    if (dtype == 0) { NA1D_MARCH_E(__nv_bfloat16) } else { NA1D_MARCH_E(__half) }
#undef NA1D_MARCH
    return cudaGetLastError();
}

}  // namespace na1d
