// The MLP of a transformer block as one kernel: out = s + GELU(h W1^T + b1) W2^T + b2, rows of 256 channels, hidden sizes that are a
// multiple of 128.
//
// As separate passes (product, GELU, product, residual in the next LayerNorm) the hidden layer, four times as wide as the rows, crosses
// HBM four times: 153600 rows take 314 us where the products themselves need 95; 175 us here (38400: 81 and 64, 9600: 28 and 27, 2400: 15
// and 26, which is left to the passes). For a backward pass the layer before GELU is stored, a sector of each row at a time straight
// from the lanes that hold it, and the last round of tiles is split over the hidden layer: 38400 rows 59 us.
// A pair of CTAs keeps 256 rows on chip: the rows as an operand in shared memory, the hidden layer in pieces of 128 columns in tensor
// memory, which GELU turns into the second product's left operand there.
//   warps 0-15   GELU: 32 tensor-memory lanes and a quarter of a piece's columns each
//   warps 16-23  the result: out of tensor memory at once (the next tile's second product waits for that) into registers and shared memory,
//                as much as fits without local memory (L1 has next to no room here: what the compiler moved there made the whole kernel wait,
//                148 us for 153600 rows), then residual and store at leisure, a row per lane
//   warp 24      loads: the rows of the next tile, the residual's into L2, weight pieces (16 KB a CTA: half of the output columns and
//                of the contraction; a ring of four)
//   warp 25      issues the products (leader): piece j + 1 of the hidden layer before the second product of piece j
// Bound: tensor pipe (1024 + 1024 cycles a piece) and GELU at the same length (special functions 2048, FMA pipe 1800; a polynomial for
// log2 Phi, one special function a value, saves a tenth of the kernel and differs from the passes in its last bits); 64 KB of weights a piece from L2.
// Every role's code is a short loop. (With the LayerNorm in it too -- eight warps, rows through registers -- the kernel took 245 us for
// 153600 rows: its arithmetic, and the instructions it needs, come on top of GELU's.)
#include "na1d_internal.h"
#include "na1d_mlp.cuh"

namespace na1d {
namespace {

__device__ int g_mlp_status = 0;

constexpr int kGeluWarps = 16, kResultWarps = 8;
constexpr int kThreads = (kGeluWarps + kResultWarps + 4) * 32;
// registers per thread after the warp groups have traded: 512 x 64 + 256 x 104 + 128 x 32 <= 896 x 72
constexpr int kLaunchRegs = 72, kGeluRegs = 64, kResultRegs = 104, kOtherRegs = 32;
constexpr int kSlots = 4;
constexpr int kStage = 6 * 32 * 16;               // per result warp: 48 columns of its 32 rows
constexpr int kBiases = (kMostF + kD) * 4;
constexpr int kSmem = 2 * kRowsBytes + kSlots * kSlotBytes + kResultWarps * kStage + kBiases + 1024;

struct Barriers {
    uint64_t full[kSlots], empty[kSlots], s_full, s_free, g_ready[2], a_full[2], a_free[2], o_full, o_free;
    uint32_t tmem;
    int abort;
};

struct Maps { CUtensorMap h, s, w1, w2; };
template <typename E> struct Args {
    const E* s;                        // residual stream
    const void *b1, *b2;               // ROUND: 16-bit, else fp32
    E* out;                            // rows ld elements apart
    long long ld;
    E* f;                              // (rows, F): the hidden layer before GELU, for a backward pass
    bool sectors;                      // rows of out start on 32 bytes
    float* part;                       // partial results of the split tiles
};

template <typename E, bool ROUND> __device__ __forceinline__ float bias_at(const void* b, int i) {
    if constexpr (ROUND) return (float)reinterpret_cast<const E*>(b)[i];
    else return reinterpret_cast<const float*>(b)[i];
}

// TRAIN: the hidden layer before GELU is stored. ROUND: GELU is taken of its 16-bit values, also where they are not stored, as a pass over the
// stored layer would.
template <typename E, bool TRAIN, bool ROUND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    mlp_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Plan plan, const __grid_constant__ Args<E> g) {
    extern __shared__ uint8_t raw[];
    uint8_t* rows_smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = rows_smem + 2 * kRowsBytes;
    uint4* stages = reinterpret_cast<uint4*>(ring + kSlots * kSlotBytes);
    float* biases = reinterpret_cast<float*>(stages + kResultWarps * (kStage / 16));   // b2, b1
    __shared__ Barriers bar;
    const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = pair::cta_rank();
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1, F = plan.pieces * kChunk;
    volatile int* abort_flag = &bar.abort;
#define NA1D_MLP_FAIL(code) { atomicExch(&g_mlp_status, code); *abort_flag = 1; ok = false; break; }

    if (warp == kGeluWarps + kResultWarps) {
        if (lane < kSlots) { ptx::mbar_init(&bar.full[lane], 1); ptx::mbar_init(&bar.empty[lane], 1); }
        else if (lane >= 16 && lane < 18) ptx::mbar_init(&bar.g_ready[lane - 16], 2 * kGeluWarps);
        else if (lane == 15) { ptx::mbar_init(&bar.s_full, 1); ptx::mbar_init(&bar.s_free, 2 * kGeluWarps); }
        else if (lane >= 18 && lane < 20) { ptx::mbar_init(&bar.a_full[lane - 18], 1); ptx::mbar_init(&bar.a_free[lane - 18], 1); }
        else if (lane == 9) { ptx::mbar_init(&bar.o_full, 1); ptx::mbar_init(&bar.o_free, 2 * kResultWarps); }
        else if (lane == 10) bar.abort = 0;
        else if (lane == 11) ptx::prefetch_tensormap(&maps.w1);
        else if (lane == 12) ptx::prefetch_tensormap(&maps.w2);
        else if (lane == 13) ptx::prefetch_tensormap(&maps.h);
        ptx::fence_mbar_init();
    }
    if (warp == kGeluWarps + kResultWarps + 2) { pair::tmem_alloc(&bar.tmem, 512); pair::tmem_relinquish(); }
    for (int i = threadIdx.x; i < kD + F; i += kThreads) biases[i] = i < kD ? bias_at<E, ROUND>(g.b2, i) : bias_at<E, ROUND>(g.b1, i - kD);
    ptx::tc_fence_before_sync();
    __syncthreads();
    pair::cluster_sync();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = bar.tmem;
    bool ok = true;

    if (warp < kGeluWarps) {
        ptx::warpgroup_regs_shrink<kGeluRegs>();
        const int q = warp & 3, part = warp >> 2;   // tensor-memory lanes 32 q .. + 31, columns of this quarter
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const uint32_t g_ready0 = pair::in_leader(&bar.g_ready[0]), g_ready1 = pair::in_leader(&bar.g_ready[1]), s_free = pair::in_leader(&bar.s_free);
        auto leave = [&]() {   // the next piece's first product may have these columns
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) pair::arrive_cluster(s_free);
        };
        auto activated = [](const float2& u, uint32_t rounded) {
            const float2 y = gelu2(ROUND ? unpack2<E>(rounded) : u);
            return Cvt<E>::pack2(y.x, y.y);
        };
        int j = 0;
        for (int i = first; ok && i < plan.items; i += step) {
            const Item t = item_at(plan, i);
            const int row = t.tile * 256 + (int)rank * 128 + q * 32 + lane;
            for (int c = t.c0; c < t.c1; ++c, ++j) {
                const int buf = j & 1, col = c * kChunk + part * 32;
                const uint32_t s = tmem + lanes + kHidden + part * 32, to = tmem + lanes + kOperand + buf * kOperandCols + part * 16;
                const float4* b1 = reinterpret_cast<const float4*>(biases + kD + col);
                if (!ptx::mbar_wait(&bar.s_full, j & 1) || *abort_flag) NA1D_MLP_FAIL(1)
                ptx::tc_fence_after_sync();
                if constexpr (TRAIN) {   // sixteen columns at a time: a short loop, and one sector of each row
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        float d[16];
                        pair::tmem_ld16(s + h * 16, d);
                        ptx::tmem_ld_wait();
                        if (h == 1) leave();
                        uint32_t packed[8], hidden[8];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float4 bias = b1[h * 4 + k];
                            const float2 u = add2(make_float2(d[4 * k], d[4 * k + 1]), make_float2(bias.x, bias.y));
                            const float2 v = add2(make_float2(d[4 * k + 2], d[4 * k + 3]), make_float2(bias.z, bias.w));
                            hidden[2 * k] = Cvt<E>::pack2(u.x, u.y);
                            hidden[2 * k + 1] = Cvt<E>::pack2(v.x, v.y);
                            packed[2 * k] = activated(u, hidden[2 * k]);
                            packed[2 * k + 1] = activated(v, hidden[2 * k + 1]);
                        }
                        pair::tmem_st8(to + h * 8, packed);
                        if (row < plan.rows) store_sector(g.f + (size_t)row * F + col + h * 16, hidden);
                    }
                } else {
                    float d[32];
                    pair::tmem_ld32(s, d);
                    ptx::tmem_ld_wait();
                    leave();
                    uint32_t packed[16];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float4 bias = b1[k];
                        const float2 u = add2(make_float2(d[4 * k], d[4 * k + 1]), make_float2(bias.x, bias.y));
                        const float2 v = add2(make_float2(d[4 * k + 2], d[4 * k + 3]), make_float2(bias.z, bias.w));
                        packed[2 * k] = activated(u, ROUND ? Cvt<E>::pack2(u.x, u.y) : 0u);
                        packed[2 * k + 1] = activated(v, ROUND ? Cvt<E>::pack2(v.x, v.y) : 0u);
                    }
                    pair::tmem_st16(to, packed);
                }
                ptx::tmem_st_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) pair::arrive_cluster(buf ? g_ready1 : g_ready0);
            }
        }
    } else if (warp < kGeluWarps + kResultWarps) {
        ptx::warpgroup_regs_grow<kResultRegs>();
        const int w = warp - kGeluWarps, q = warp & 3, half = w >> 2;
        uint4* stage = stages + w * (kStage / 16) + lane;
        const uint32_t o_free = pair::in_leader(&bar.o_free), o = tmem + ((uint32_t)(q * 32) << 16) + kAcc + half * 128;
        int it = 0;
        for (int i = first; i < plan.items; i += step, ++it) {
            const Item t = item_at(plan, i);
            const int row0 = t.tile * 256 + (int)rank * 128 + q * 32;
            if (!ptx::mbar_wait_relaxed(&bar.o_full, it & 1) || *abort_flag) NA1D_MLP_FAIL(2)
            ptx::tc_fence_after_sync();
            // 128 columns of this lane's row: the first 48 into this lane's own place in shared memory, the others into registers (all of them
            // would not fit there: what the compiler then kept in local memory made this drain take 2800 cycles)
            uint4 z[10];
            if (t.parts == 1) {
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    float d[16];
                    pair::tmem_ld16(o + n * 16, d);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float4* b2 = reinterpret_cast<const float4*>(biases + half * 128 + n * 16 + k * 8);
                        const float4 ba = b2[0], bb = b2[1];
                        float* v = d + 8 * k;
                        v[0] += ba.x; v[1] += ba.y; v[2] += ba.z; v[3] += ba.w; v[4] += bb.x; v[5] += bb.y; v[6] += bb.z; v[7] += bb.w;
                        if (n < 3) stage[(2 * n + k) * 32] = Cvt<E>::pack(v);
                        else z[2 * (n - 3) + k] = Cvt<E>::pack(v);
                    }
                }
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) pair::arrive_cluster(o_free);
            } else {   // a partial result, added up by mlp_finish_kernel
                float4* dst = reinterpret_cast<float4*>(g.part) + ((((size_t)(t.tile - plan.whole) * 2 + rank) * kResultWarps + w) * t.parts + t.part) * 32 * 32 + lane;
#pragma unroll 1
                for (int n = 0; n < 4; ++n) {
                    float d[32];
                    pair::tmem_ld32(o + n * 32, d);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int k = 0; k < 8; ++k) dst[(n * 8 + k) * 32] = make_float4(d[4 * k], d[4 * k + 1], d[4 * k + 2], d[4 * k + 3]);
                }
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) pair::arrive_cluster(o_free);
                continue;
            }
            const int row = row0 + lane;
            const bool live = row < plan.rows;
            const E* res = g.s + (size_t)row * kD + half * 128;
            E* dst = g.out + (size_t)row * g.ld + half * 128;
            auto leave = [&](int n, const uint4& x, const uint4& y) {
                uint32_t v[8] = {};
                if (live) load_sector(res + n * 16, v);
                const uint4 a = add_rows<E>(make_uint4(v[0], v[1], v[2], v[3]), x), b = add_rows<E>(make_uint4(v[4], v[5], v[6], v[7]), y);
                const uint32_t sum[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                if (live && g.sectors) store_sector(dst + n * 16, sum);
                else if (live) {
                    *reinterpret_cast<uint4*>(dst + n * 16) = a;
                    *reinterpret_cast<uint4*>(dst + n * 16 + 8) = b;
                }
            };
#pragma unroll
            for (int n = 3; n < 8; ++n) leave(n, z[2 * (n - 3)], z[2 * (n - 3) + 1]);
#pragma unroll 1
            for (int n = 0; n < 3; ++n) leave(n, stage[2 * n * 32], stage[(2 * n + 1) * 32]);
        }
    } else {
        ptx::warpgroup_regs_shrink<kOtherRegs>();
        if (warp == kGeluWarps + kResultWarps && ptx::elect_one()) {
            int slot = 0, n = 0;
            uint32_t phase = 1;
            // pieces in the order in which they are used: W1 of piece j, then W2 of the piece before
            auto load = [&](bool second, int c) {
#pragma unroll 1
                for (int k = 0; k < 2; ++k) {
                    if (!ptx::mbar_wait_relaxed(&bar.empty[slot], phase) || *abort_flag) { atomicExch(&g_mlp_status, 4); *abort_flag = 1; ok = false; return; }
                    const uint32_t full = pair::in_leader(&bar.full[slot]);
                    if (rank == 0) ptx::mbar_expect_tx(&bar.full[slot], 2 * kSlotBytes);
                    if (second) pair::load_3d(ring + slot * kSlotBytes, &maps.w2, full, 0, (int)rank * 128, 2 * c + k);
                    else pair::load_3d(ring + slot * kSlotBytes, &maps.w1, full, 0, c * kChunk + (int)rank * 64, 2 * k);
                    ++n;
                    if (++slot == kSlots) { slot = 0; phase ^= 1; }
                }
            };
            auto rows = [&](int i, int it) {
                if (i >= plan.items) return;
                if (!ptx::mbar_wait_relaxed(&bar.a_free[it & 1], ((it >> 1) & 1) ^ 1) || *abort_flag) { atomicExch(&g_mlp_status, 3); *abort_flag = 1; ok = false; return; }
                if (rank == 0) ptx::mbar_expect_tx(&bar.a_full[it & 1], 2 * kRowsBytes);
                pair::load_3d(rows_smem + (it & 1) * kRowsBytes, &maps.h, pair::in_leader(&bar.a_full[it & 1]), 0, item_at(plan, i).tile * 256 + (int)rank * 128, 0);
            };
            int before = -1, it = 0;
            rows(first, 0);
            for (int i = first; ok && i < plan.items; i += step, ++it) {
                const Item t = item_at(plan, i);
                for (int c = t.c0; ok && c < t.c1; ++c) {
                    load(false, c);
                    if (ok && before >= 0) load(true, before);
                    before = c;
                    if (ok && c == min(t.c0 + 1, t.c1 - 1)) rows(i + step, it + 1);
                    if (t.parts == 1 && c == max(t.c1 - 4, t.c0)) pair::prefetch_3d(&maps.s, 0, t.tile * 256 + (int)rank * 128, 0);
                }
            }
            if (ok && before >= 0) load(true, before);
            if (!ok && rank == 0)   // loads that are on their way arrive before the CTAs leave
                for (int k = n - 1; k >= 0 && k >= n - kSlots; --k) ptx::mbar_wait(&bar.full[k % kSlots], (k / kSlots) & 1, 1u << 14);
            if (!ok && rank == 0)
                for (int k = it + 1; k >= 0 && k >= it; --k) ptx::mbar_wait(&bar.a_full[k & 1], (k >> 1) & 1, 1u << 12);
        }
        if (warp == kGeluWarps + kResultWarps + 1 && rank == 0 && ptx::elect_one()) {
            constexpr uint32_t fmt = tc::Fmt<E>::v;
            constexpr uint32_t idesc1 = ptx::instr_desc(fmt, 0, 0, 256, kChunk), idesc2 = ptx::instr_desc(fmt, 0, 0, 256, kD);
            int slot = 0, j = 0, it = 0;
            uint32_t phase = 0;
            auto next_slot = [&]() {
                if (++slot == kSlots) { slot = 0; phase ^= 1; }
            };
            // second product of piece jj (its item: the it-th), the last one of its item or not
            auto second = [&](int jj, int item, bool opens, bool closes) {
                if (opens && (!ptx::mbar_wait(&bar.o_free, (item & 1) ^ 1) || *abort_flag)) { atomicExch(&g_mlp_status, 5); *abort_flag = 1; ok = false; return; }
                if (!ptx::mbar_wait(&bar.g_ready[jj & 1], (jj >> 1) & 1) || *abort_flag) { atomicExch(&g_mlp_status, 6); *abort_flag = 1; ok = false; return; }
                ptx::tc_fence_after_sync();
                const uint32_t s = tmem + kOperand + (jj & 1) * kOperandCols;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    if (!ptx::mbar_wait(&bar.full[slot], phase) || *abort_flag) { atomicExch(&g_mlp_status, 7); *abort_flag = 1; ok = false; return; }
                    ptx::tc_fence_after_sync();
                    const uint64_t b = pair::k_major(ptx::smem_u32(ring + slot * kSlotBytes));
#pragma unroll
                    for (int k = 0; k < 4; ++k) pair::mma_ts(tmem + kAcc, s + (h * 4 + k) * 8, tc::desc_advance(b, k * 32), idesc2, !opens || h > 0 || k > 0);
                    pair::commit(&bar.empty[slot]);
                    next_slot();
                }
                if (closes) pair::commit(&bar.o_full);
            };
            bool opened = false;   // the piece before opened its item
            for (int i = first; ok && i < plan.items; i += step, ++it) {
                const Item t = item_at(plan, i);
                if (!ptx::mbar_wait(&bar.a_full[it & 1], (it >> 1) & 1) || *abort_flag) NA1D_MLP_FAIL(8)
                const uint64_t a = pair::k_major(ptx::smem_u32(rows_smem + (it & 1) * kRowsBytes));
                for (int c = t.c0; ok && c < t.c1; ++c, ++j) {
                    if (!ptx::mbar_wait(&bar.s_free, (j & 1) ^ 1) || *abort_flag) NA1D_MLP_FAIL(10)
                    ptx::tc_fence_after_sync();
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        if (!ptx::mbar_wait(&bar.full[slot], phase) || *abort_flag) NA1D_MLP_FAIL(9)
                        ptx::tc_fence_after_sync();
                        const uint64_t b = pair::k_major(ptx::smem_u32(ring + slot * kSlotBytes)), ah = tc::desc_advance(a, h * 32768);
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            pair::mma_ss(tmem + kHidden, tc::desc_advance(ah, (k >> 2) * 16384 + (k & 3) * 32), tc::desc_advance(b, (k >> 2) * 8192 + (k & 3) * 32), idesc1, h > 0 || k > 0);
                        pair::commit(&bar.empty[slot]);
                        next_slot();
                    }
                    if (!ok) break;
                    pair::commit(&bar.s_full);   // (and all that was issued before, the second product of the piece two back among it)
                    if (c == t.c1 - 1) pair::commit(&bar.a_free[it & 1]);
                    if (j > 0) second(j - 1, c == t.c0 ? it - 1 : it, opened, c == t.c0);
                    opened = c == t.c0;
                }
            }
            if (ok && j > 0) second(j - 1, it - 1, opened, true);
        }
    }
#undef NA1D_MLP_FAIL
    __syncwarp();
    ptx::tc_fence_before_sync();
    __syncthreads();
    pair::cluster_sync();   // neither CTA leaves while the other may still signal it or read its operands
    if (warp == kGeluWarps + kResultWarps + 2) pair::tmem_dealloc(tmem, 512);
}

// The split tiles' partial results, residual and bias, in the order of the parts: a thread per four columns of a row, a CTA per 32 rows x 32
// columns.
template <typename E, bool ROUND>
__global__ void __launch_bounds__(256) mlp_finish_kernel(const __grid_constant__ Plan plan, const __grid_constant__ Args<E> g) {
    const int n = blockIdx.x & 3, band = blockIdx.x >> 2, w = band & 7, rank = (band >> 3) & 1, tile = plan.whole + (band >> 4);
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    const int row = tile * 256 + rank * 128 + (w & 3) * 32 + lane, col = (w >> 2) * 128 + n * 32 + k * 4;
    if (row >= plan.rows) return;
    const uint2 res = __ldg(reinterpret_cast<const uint2*>(g.s + (size_t)row * kD + col));
    const float4 b = make_float4(bias_at<E, ROUND>(g.b2, col), bias_at<E, ROUND>(g.b2, col + 1), bias_at<E, ROUND>(g.b2, col + 2), bias_at<E, ROUND>(g.b2, col + 3));
    const float4* src = reinterpret_cast<const float4*>(g.part) + (size_t)band * plan.parts * 32 * 32 + (n * 8 + k) * 32 + lane;
    float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int p = 0; p < plan.parts; ++p) {
        const float4 v = __ldg(src + (size_t)p * 32 * 32);
        z.x += v.x; z.y += v.y; z.z += v.z; z.w += v.w;
    }
    const uint2 m = make_uint2(Cvt<E>::pack2(z.x + b.x, z.y + b.y), Cvt<E>::pack2(z.z + b.z, z.w + b.w));
    const uint4 sum = add_rows<E>(make_uint4(res.x, res.y, 0u, 0u), make_uint4(m.x, m.y, 0u, 0u));
    *reinterpret_cast<uint2*>(g.out + (size_t)row * g.ld + col) = make_uint2(sum.x, sum.y);
}

template <typename E, bool TRAIN, bool ROUND>
cudaError_t run(const Maps& maps, const Plan& plan, const Args<E>& a, cudaStream_t st) {
    auto* kern = mlp_kernel<E, TRAIN, ROUND>;
    // a kernel compiled to fewer registers would leave the growing warp groups waiting for ones that never come
    static const int regs = [kern] {
        cudaFuncAttributes fa;
        return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? fa.numRegs : 0;
    }();
    if (regs < kLaunchRegs) return cudaErrorLaunchOutOfResources;
    if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)) return e;
    const int pairs = device_sm_count() / 2, n = plan.items < pairs ? plan.items : pairs;
    kern<<<2 * n, kThreads, kSmem, st>>>(maps, plan, a);
    if (plan.parts == 1) return cudaGetLastError();
    if (cudaError_t e = cudaGetLastError()) return e;
    mlp_finish_kernel<E, ROUND><<<(plan.items - plan.whole) / plan.parts * 2 * kResultWarps * 4, 256, 0, st>>>(plan, a);
    return cudaGetLastError();
}
template <typename E, bool ROUND>
cudaError_t forward(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const void* b1, const void* w2, const void* b2, float* scratch,
                    int64_t rows, int64_t F, int dtype, cudaStream_t st) {
    const Plan plan = make_plan(rows, F, !ROUND || f);
    Maps maps;
    const int64_t dh[3] = {64, rows, kD / 64}, d1[3] = {64, F, kD / 64}, s1[2] = {kD, 64}, d2[3] = {64, kD, F / 64}, s2[2] = {F, 64};
    const int xh[3] = {64, 128, kD / 64}, x1[3] = {64, 64, 2}, x2[3] = {64, 128, 1};
    if (!make_matrix_map(&maps.h, h, dtype, 3, dh, s1, xh) || !make_matrix_map(&maps.s, s, dtype, 3, dh, s1, xh) || !make_matrix_map(&maps.w1, w1, dtype, 3, d1, s1, x1) ||
        !make_matrix_map(&maps.w2, w2, dtype, 3, d2, s2, x2))
        return cudaErrorInvalidValue;
    const Args<E> a = {(const E*)s, b1, b2, (E*)out, ld, (E*)f, ld % 16 == 0 && ((uintptr_t)out & 31) == 0, scratch};
    return f ? run<E, true, ROUND>(maps, plan, a, st) : run<E, false, ROUND>(maps, plan, a, st);
}

}  // namespace

bool mlp_supports(int64_t D, int64_t F) { return D == kD && F > 0 && F % kChunk == 0 && F <= kMostF; }
size_t mlp_scratch_floats(int64_t rows, int64_t F) {
    return part_floats(make_plan(rows, F));
}
cudaError_t mlp_forward(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const void* b1, const void* w2, const void* b2, bool rounded,
                        float* scratch, int64_t rows, int64_t F, int dtype, cudaStream_t st) {
    bind_primary_context();
    using B = __nv_bfloat16;
    using H = __half;
    if (rounded)
        return dtype == 0 ? forward<B, true>(out, ld, f, s, h, w1, b1, w2, b2, scratch, rows, F, dtype, st)
                          : forward<H, true>(out, ld, f, s, h, w1, b1, w2, b2, scratch, rows, F, dtype, st);
    return dtype == 0 ? forward<B, false>(out, ld, f, s, h, w1, b1, w2, b2, scratch, rows, F, dtype, st)
                      : forward<H, false>(out, ld, f, s, h, w1, b1, w2, b2, scratch, rows, F, dtype, st);
}
int mlp_read_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_mlp_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_mlp_status, &zero, sizeof(int));
    return v;
}

}  // namespace na1d
