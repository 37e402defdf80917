// Pieces that the kernels of a block's MLP share: how rows and hidden layer are shared out, rows by sectors.
#pragma once
#include "na1d_gelu.cuh"
#include "na1d_pair.cuh"

namespace na1d {
namespace {

constexpr int kD = 256, kChunk = 128, kMostF = 1280;
constexpr int kRowsBytes = 128 * kD * 2;          // a CTA's rows as an operand: four blocks of 64 channels, [block][row][128 bytes]
constexpr int kSlotBytes = 16 * 1024;             // a CTA's half of half a weight piece
// Tensor-memory columns: the result (256), a piece of the hidden layer as the first product leaves it (128, fp32), and two pieces as the second
// product reads them (64 each, 16 bits). What a product writes is never what an earlier one may still read without a barrier in
// between: products of different shapes are not known to run in the order of their issue. The first product of a piece waits
// until the 16 warps of both CTAs have read the one before out of its columns (s_free; they do so at once, while the second
// product of the piece before runs), and a piece that GELU writes lies where the one two back was, whose second product is among those
// that the signal for this piece's first (s_full) waits for.
constexpr uint32_t kAcc = 0, kHidden = 256, kOperand = 384, kOperandCols = 64;

// Items: whole tiles of 256 rows in full rounds of the CTA pairs, then the tiles of the last, partly filled round split over the hidden
// layer into `parts`, so that those take 1 / parts of the time (150 tiles on 74 pairs: 2.1 instead of 3).
struct Plan {
    int rows, pieces, whole, parts, items;
};
struct Item {
    int tile, part, parts, c0, c1;
};
__device__ __forceinline__ Item item_at(const Plan& p, int i) {
    Item t;
    if (i < p.whole) {
        t.tile = i; t.part = 0; t.parts = 1; t.c0 = 0; t.c1 = p.pieces;
    } else {
        i -= p.whole;
        t.tile = i / p.parts;
        t.part = i - t.tile * p.parts;
        t.tile += p.whole;
        t.parts = p.parts;
        t.c0 = p.pieces * t.part / p.parts;
        t.c1 = p.pieces * (t.part + 1) / p.parts;
    }
    return t;
}

// 32 bytes, a sector, of a row: of each of a warp's 32 rows at a time
__device__ __forceinline__ void load_sector(const void* p, uint32_t* v) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(p));
}
__device__ __forceinline__ void store_sector(void* p, const uint32_t* v) {
    asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
template <typename E> __device__ __forceinline__ void unpack2(const uint4& u, float2* f) {
    float t[8];
    Cvt<E>::unpack(u, t);
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = make_float2(t[2 * i], t[2 * i + 1]);
}
template <typename E> __device__ __forceinline__ float2 unpack2(uint32_t w) {
    if constexpr (sizeof(E) == 2 && tc::Fmt<E>::v == 1) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    else return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <typename E> __device__ __forceinline__ uint4 pack2(const float2* f) {
    return make_uint4(Cvt<E>::pack2(f[0].x, f[0].y), Cvt<E>::pack2(f[1].x, f[1].y), Cvt<E>::pack2(f[2].x, f[2].y), Cvt<E>::pack2(f[3].x, f[3].y));
}
// x + y of eight 16-bit values each, rounded: the residual stream
template <typename E> __device__ __forceinline__ uint4 add_rows(const uint4& x, const uint4& y) {
    float2 a[4], b[4];
    unpack2<E>(x, a);
    unpack2<E>(y, b);
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = add2(a[i], b[i]);
    return pack2<E>(a);
}

// split: the last, partly filled round over the hidden layer
inline Plan make_plan(int64_t rows, int64_t F, bool split = true) {
    Plan p;
    const int pairs = device_sm_count() / 2, tiles = (int)((rows + 255) / 256);
    p.rows = (int)rows;
    p.pieces = (int)(F / kChunk);
    p.whole = tiles / pairs * pairs;
    const int rest = tiles - p.whole;
    p.parts = rest && split ? pairs / rest : 1;
    if (p.parts > p.pieces) p.parts = p.pieces;
    if (p.parts < 2) { p.parts = 1; p.whole = tiles; }
    p.items = p.whole + (tiles - p.whole) * p.parts;
    return p;
}
inline size_t part_floats(const Plan& p) { return p.parts > 1 ? (size_t)(p.items - p.whole) * 256 * kD : 0; }

}  // namespace
}  // namespace na1d
