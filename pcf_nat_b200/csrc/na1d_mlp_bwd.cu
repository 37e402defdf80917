// Backward of a block's MLP (na1d_mlp.cu) as one kernel: df = (d W2) GELU'(f), dh = df W1, and the hidden layer g = GELU(f) again, which
// the gradient of W2 needs and the forward does not keep.
//
// As separate passes (product, GELU' with the bias gradient, product) the gradient of the hidden layer crossed HBM four times: 38400 rows
// took 15 + 52 + 18 us, here 78 (153600: 273). It goes from the first product through GELU' to the second one in tensor memory, as
// in the forward; only df and g leave, for the parameter gradients (the bias gradient is a column sum there). The same shape of kernel:
//   warps 0-15   GELU': 32 tensor-memory lanes and a quarter of a piece's columns each, a row per lane, sixteen columns (one sector) at a
//                time; f of the next sixteen is on its way meanwhile
//   warps 16-23  the result: 32 lanes, half of the columns
//   warp 24      loads: the rows of the next tile, weight pieces (both products contract across their rows), a ring of six; f from HBM into
//                L2 two pieces ahead (without: 271 us for 153600 rows)
//   warp 25      issues the products (leader)
// Bound by HBM: f in, df and g out, three rows of 1024 for every row of 256 in and out (43 us at 38400 rows). GELU and its slope are those of the
// passes (na1d_gelu.cuh), so g is bit for bit what the forward multiplied. In a form of this kernel whose products did not wait for
// GELU's reads (243 us for 153600 rows) the products and GELU' alone took 121, with the reads of f 171, with the stores 216. Sectors of a row straight from registers, without a line in
// L1 (with one: 281), against 315 through a stage in shared memory, whose room the ring needs: weights wait behind the stores on
// their way from L2.
#include "na1d_internal.h"
#include "na1d_mlp.cuh"

namespace na1d {
namespace {

__device__ int g_mlp_bwd_status = 0;

constexpr int kGeluWarps = 16, kResultWarps = 8;
constexpr int kThreads = (kGeluWarps + kResultWarps + 4) * 32;
// registers per thread after the warp groups have traded: 512 x 88 + 256 x 48 + 128 x 40 <= 896 x 72
constexpr int kLaunchRegs = 72, kGeluRegs = 88, kResultRegs = 48, kOtherRegs = 40;
constexpr int kSlots = 6;
constexpr int kSmem = 2 * kRowsBytes + kSlots * kSlotBytes + 1024;

struct Barriers {
    uint64_t full[kSlots], empty[kSlots], s_full, s_free, g_ready[2], a_full[2], a_free[2], o_full, o_free;
    uint32_t tmem;
    int abort;
};
struct Maps { CUtensorMap d, w1, w2, f; };
template <typename E> struct Args {
    const E* f;       // (rows, F)
    E *df, *g;        // (rows, F)
    E* dh;            // (rows, 256)
    float* part;      // partial results of the split tiles
};

template <typename E>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    mlp_bwd_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Plan plan, const __grid_constant__ Args<E> g) {
    extern __shared__ uint8_t raw[];
    uint8_t* rows_smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = rows_smem + 2 * kRowsBytes;
    __shared__ Barriers bar;
    const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = pair::cta_rank();
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1, F = plan.pieces * kChunk;
    volatile int* abort_flag = &bar.abort;
#define NA1D_MLP_FAIL(code) { atomicExch(&g_mlp_bwd_status, code); *abort_flag = 1; ok = false; break; }

    if (warp == kGeluWarps + kResultWarps) {
        if (lane < kSlots) { ptx::mbar_init(&bar.full[lane], 1); ptx::mbar_init(&bar.empty[lane], 1); }
        else if (lane >= 16 && lane < 18) ptx::mbar_init(&bar.g_ready[lane - 16], 2 * kGeluWarps);
        else if (lane == 15) { ptx::mbar_init(&bar.s_full, 1); ptx::mbar_init(&bar.s_free, 2 * kGeluWarps); }
        else if (lane >= 24 && lane < 26) { ptx::mbar_init(&bar.a_full[lane - 24], 1); ptx::mbar_init(&bar.a_free[lane - 24], 1); }
        else if (lane == 19) { ptx::mbar_init(&bar.o_full, 1); ptx::mbar_init(&bar.o_free, 2 * kResultWarps); }
        else if (lane == 20) bar.abort = 0;
        else if (lane == 21) ptx::prefetch_tensormap(&maps.w1);
        else if (lane == 22) ptx::prefetch_tensormap(&maps.w2);
        else if (lane == 23) ptx::prefetch_tensormap(&maps.d);
        else if (lane == 26) ptx::prefetch_tensormap(&maps.f);
        ptx::fence_mbar_init();
    }
    if (warp == kGeluWarps + kResultWarps + 2) { pair::tmem_alloc(&bar.tmem, 512); pair::tmem_relinquish(); }
    ptx::tc_fence_before_sync();
    __syncthreads();
    pair::cluster_sync();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = bar.tmem;
    bool ok = true;

    if (warp < kGeluWarps) {
        ptx::warpgroup_regs_grow<kGeluRegs>();
        const int q = warp & 3, part = warp >> 2;   // tensor-memory lanes 32 q .. + 31, columns of this quarter
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const uint32_t g_ready0 = pair::in_leader(&bar.g_ready[0]), g_ready1 = pair::in_leader(&bar.g_ready[1]), s_free = pair::in_leader(&bar.s_free);
        uint32_t next[8];   // f of the next sixteen columns
        auto fetch = [&](const Item& t, int c, int h) {
            const int row = t.tile * 256 + (int)rank * 128 + q * 32 + lane;
#pragma unroll
            for (int k = 0; k < 8; ++k) next[k] = 0;
            if (row < plan.rows) load_sector(g.f + (size_t)row * F + c * kChunk + part * 32 + h * 16, next);
        };
        int j = 0;
        if (first < plan.items) { const Item t = item_at(plan, first); fetch(t, t.c0, 0); }
        for (int i = first; ok && i < plan.items; i += step) {
            const Item t = item_at(plan, i);
            const int row = t.tile * 256 + (int)rank * 128 + q * 32 + lane;
            for (int c = t.c0; c < t.c1; ++c, ++j) {
                const int buf = j & 1;
                const uint32_t s = tmem + lanes + kHidden + part * 32, to = tmem + lanes + kOperand + buf * kOperandCols + part * 16;
                const size_t at = (size_t)row * F + c * kChunk + part * 32;
                if (!ptx::mbar_wait(&bar.s_full, j & 1) || *abort_flag) NA1D_MLP_FAIL(1)
                ptx::tc_fence_after_sync();
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    float d[16];
                    pair::tmem_ld16(s + h * 16, d);
                    float2 x[8];
                    unpack2<E>(make_uint4(next[0], next[1], next[2], next[3]), x);
                    unpack2<E>(make_uint4(next[4], next[5], next[6], next[7]), x + 4);
                    if (h == 0) fetch(t, c, 1);
                    else if (c + 1 < t.c1) fetch(t, c + 1, 0);
                    else if (i + step < plan.items) { const Item n = item_at(plan, i + step); fetch(n, n.c0, 0); }
                    ptx::tmem_ld_wait();
                    if (h == 1) {   // the next piece's first product may have these columns
                        ptx::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) pair::arrive_cluster(s_free);
                    }
                    uint32_t df[8], val[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        float2 value, slope;
                        gelu_and_slope(x[k], value, slope);
                        slope = mul2(slope, make_float2(d[2 * k], d[2 * k + 1]));
                        val[k] = Cvt<E>::pack2(value.x, value.y);
                        df[k] = Cvt<E>::pack2(slope.x, slope.y);
                    }
                    pair::tmem_st8(to + h * 8, df);
                    if (row < plan.rows) {
                        store_sector(g.g + at + h * 16, val);
                        store_sector(g.df + at + h * 16, df);
                    }
                }
                ptx::tmem_st_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) pair::arrive_cluster(buf ? g_ready1 : g_ready0);
            }
        }
    } else if (warp < kGeluWarps + kResultWarps) {
        ptx::warpgroup_regs_shrink<kResultRegs>();
        const int w = warp - kGeluWarps, q = warp & 3, half = w >> 2;
        const uint32_t o_free = pair::in_leader(&bar.o_free), o = tmem + ((uint32_t)(q * 32) << 16) + kAcc + half * 128;
        int it = 0;
        for (int i = first; i < plan.items; i += step, ++it) {
            const Item t = item_at(plan, i);
            const int row = t.tile * 256 + (int)rank * 128 + q * 32 + lane;
            if (!ptx::mbar_wait_relaxed(&bar.o_full, it & 1) || *abort_flag) NA1D_MLP_FAIL(2)
            ptx::tc_fence_after_sync();
            float4* dst = reinterpret_cast<float4*>(g.part) + ((((size_t)(t.tile - plan.whole) * 2 + rank) * kResultWarps + w) * t.parts + t.part) * 32 * 32 + lane;
#pragma unroll 1
            for (int n = 0; n < 8; ++n) {
                float d[16];
                pair::tmem_ld16(o + n * 16, d);
                ptx::tmem_ld_wait();
                if (t.parts > 1) {   // a partial result, added up by mlp_bwd_finish_kernel
#pragma unroll
                    for (int k = 0; k < 4; ++k) dst[(n * 4 + k) * 32] = make_float4(d[4 * k], d[4 * k + 1], d[4 * k + 2], d[4 * k + 3]);
                } else if (row < plan.rows) {
                    uint32_t v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = Cvt<E>::pack2(d[2 * k], d[2 * k + 1]);
                    store_sector(g.dh + (size_t)row * kD + half * 128 + n * 16, v);
                }
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) pair::arrive_cluster(o_free);
        }
    } else {
        ptx::warpgroup_regs_shrink<kOtherRegs>();
        if (warp == kGeluWarps + kResultWarps && ptx::elect_one()) {
            int slot = 0, n = 0;
            uint32_t phase = 1;
            // pieces in the order in which they are used: W2 of piece j, then W1 of the piece before
            auto load = [&](bool second, int c) {
#pragma unroll 1
                for (int k = 0; k < 2; ++k) {
                    if (!ptx::mbar_wait_relaxed(&bar.empty[slot], phase) || *abort_flag) { atomicExch(&g_mlp_bwd_status, 4); *abort_flag = 1; ok = false; return; }
                    const uint32_t full = pair::in_leader(&bar.full[slot]);
                    if (rank == 0) ptx::mbar_expect_tx(&bar.full[slot], 2 * kSlotBytes);
                    if (second) pair::load_3d(ring + slot * kSlotBytes, &maps.w1, full, 0, c * kChunk + 64 * k, (int)rank * 2);
                    else pair::load_2d(ring + slot * kSlotBytes, &maps.w2, full, c * kChunk + (int)rank * 64, 128 * k);
                    ++n;
                    if (++slot == kSlots) { slot = 0; phase ^= 1; }
                }
            };
            auto rows = [&](int i, int it) {
                if (i >= plan.items) return;
                if (!ptx::mbar_wait_relaxed(&bar.a_free[it & 1], ((it >> 1) & 1) ^ 1) || *abort_flag) { atomicExch(&g_mlp_bwd_status, 3); *abort_flag = 1; ok = false; return; }
                if (rank == 0) ptx::mbar_expect_tx(&bar.a_full[it & 1], 2 * kRowsBytes);
                pair::load_3d(rows_smem + (it & 1) * kRowsBytes, &maps.d, pair::in_leader(&bar.a_full[it & 1]), 0, item_at(plan, i).tile * 256 + (int)rank * 128, 0);
            };
            // f, which GELU' reads from L2, from HBM: two pieces ahead of the product
            int ahead = first, ahead_c = first < plan.items ? item_at(plan, first).c0 : 0;
            auto prefetch = [&]() {
                if (ahead >= plan.items) return;
                const Item t = item_at(plan, ahead);
                const int row = t.tile * 256 + (int)rank * 128;
                if (row < plan.rows) {
                    pair::prefetch_2d(&maps.f, ahead_c * kChunk, row);
                    pair::prefetch_2d(&maps.f, ahead_c * kChunk + 64, row);
                }
                if (++ahead_c == t.c1) {
                    ahead += step;
                    if (ahead < plan.items) ahead_c = item_at(plan, ahead).c0;
                }
            };
            int before = -1, it = 0;
            rows(first, 0);
            prefetch();
            prefetch();
            for (int i = first; ok && i < plan.items; i += step, ++it) {
                const Item t = item_at(plan, i);
                for (int c = t.c0; ok && c < t.c1; ++c) {
                    prefetch();
                    load(false, c);
                    if (ok && before >= 0) load(true, before);
                    before = c;
                    if (ok && c == min(t.c0 + 1, t.c1 - 1)) rows(i + step, it + 1);
                }
            }
            if (ok && before >= 0) load(true, before);
            if (!ok && rank == 0) {   // loads that are on their way arrive before the CTAs leave
                for (int k = n - 1; k >= 0 && k >= n - kSlots; --k) ptx::mbar_wait(&bar.full[k % kSlots], (k / kSlots) & 1, 1u << 14);
                for (int k = it + 1; k >= it; --k) ptx::mbar_wait(&bar.a_full[k & 1], (k >> 1) & 1, 1u << 12);
            }
        }
        if (warp == kGeluWarps + kResultWarps + 1 && rank == 0 && ptx::elect_one()) {
            constexpr uint32_t fmt = tc::Fmt<E>::v;
            constexpr uint32_t idesc1 = ptx::instr_desc(fmt, 0, 1, 256, kChunk), idesc2 = ptx::instr_desc(fmt, 0, 1, 256, kD);
            int slot = 0, j = 0, it = 0;
            uint32_t phase = 0;
            auto next_slot = [&]() {
                if (++slot == kSlots) { slot = 0; phase ^= 1; }
            };
            // second product of piece jj (its item: the item-th), the last one of its item or not
            auto second = [&](int jj, int item, bool opens, bool closes) {
                if (opens && (!ptx::mbar_wait(&bar.o_free, (item & 1) ^ 1) || *abort_flag)) { atomicExch(&g_mlp_bwd_status, 5); *abort_flag = 1; ok = false; return; }
                if (!ptx::mbar_wait(&bar.g_ready[jj & 1], (jj >> 1) & 1) || *abort_flag) { atomicExch(&g_mlp_bwd_status, 6); *abort_flag = 1; ok = false; return; }
                ptx::tc_fence_after_sync();
                const uint32_t s = tmem + kOperand + (jj & 1) * kOperandCols;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    if (!ptx::mbar_wait(&bar.full[slot], phase) || *abort_flag) { atomicExch(&g_mlp_bwd_status, 7); *abort_flag = 1; ok = false; return; }
                    ptx::tc_fence_after_sync();
                    const uint64_t b = pair::mn_major(ptx::smem_u32(ring + slot * kSlotBytes), 8192);
#pragma unroll
                    for (int k = 0; k < 4; ++k) pair::mma_ts(tmem + kAcc, s + (h * 4 + k) * 8, tc::desc_advance(b, k * 2048), idesc2, !opens || h > 0 || k > 0);
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
                        const uint64_t b = pair::mn_major(ptx::smem_u32(ring + slot * kSlotBytes), 8192), ah = tc::desc_advance(a, h * 32768);
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            pair::mma_ss(tmem + kHidden, tc::desc_advance(ah, (k >> 2) * 16384 + (k & 3) * 32), tc::desc_advance(b, k * 2048), idesc1, h > 0 || k > 0);
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

// The split tiles' partial results in the order of the parts: a thread per four columns of a row, a CTA per 32 rows x 32 columns.
template <typename E>
__global__ void __launch_bounds__(256) mlp_bwd_finish_kernel(const __grid_constant__ Plan plan, const __grid_constant__ Args<E> g) {
    const int n = blockIdx.x & 3, band = blockIdx.x >> 2, w = band & 7, rank = (band >> 3) & 1, tile = plan.whole + (band >> 4);
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    const int row = tile * 256 + rank * 128 + (w & 3) * 32 + lane, col = (w >> 2) * 128 + n * 32 + k * 4;
    if (row >= plan.rows) return;
    const float4* src = reinterpret_cast<const float4*>(g.part) + (size_t)band * plan.parts * 32 * 32 + (n * 8 + k) * 32 + lane;
    float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int p = 0; p < plan.parts; ++p) {
        const float4 v = __ldg(src + (size_t)p * 32 * 32);
        z.x += v.x; z.y += v.y; z.z += v.z; z.w += v.w;
    }
    *reinterpret_cast<uint2*>(g.dh + (size_t)row * kD + col) = make_uint2(Cvt<E>::pack2(z.x, z.y), Cvt<E>::pack2(z.z, z.w));
}

template <typename E>
cudaError_t backward(void* dh, void* df, void* gelu, const void* d, const void* f, const void* w1, const void* w2, float* scratch, int64_t rows, int64_t F, int dtype,
                     cudaStream_t st) {
    const Plan plan = make_plan(rows, F);
    Maps maps;
    const int64_t dd[3] = {64, rows, kD / 64}, d1[3] = {64, F, kD / 64}, s1[2] = {kD, 64}, d2[2] = {F, kD}, s2[1] = {F}, d3[2] = {F, rows};
    const int xd[3] = {64, 128, kD / 64}, x1[3] = {64, 64, 2}, x2[2] = {64, 128};   // (of f too: 128 rows of 64)
    if (!make_matrix_map(&maps.d, d, dtype, 3, dd, s1, xd) || !make_matrix_map(&maps.w1, w1, dtype, 3, d1, s1, x1) ||
        !make_matrix_map(&maps.w2, w2, dtype, 2, d2, s2, x2) || !make_matrix_map(&maps.f, f, dtype, 2, d3, s2, x2))
        return cudaErrorInvalidValue;
    const Args<E> a = {(const E*)f, (E*)df, (E*)gelu, (E*)dh, scratch};
    auto* kern = mlp_bwd_kernel<E>;
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
    mlp_bwd_finish_kernel<E><<<(plan.items - plan.whole) / plan.parts * 2 * kResultWarps * 4, 256, 0, st>>>(plan, a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t mlp_backward(void* dh, void* df, void* gelu, const void* d, const void* f, const void* w1, const void* w2, float* scratch, int64_t rows, int64_t F,
                         int dtype, cudaStream_t st) {
    bind_primary_context();
    return dtype == 0 ? backward<__nv_bfloat16>(dh, df, gelu, d, f, w1, w2, scratch, rows, F, dtype, st)
                      : backward<__half>(dh, df, gelu, d, f, w1, w2, scratch, rows, F, dtype, st);
}
int mlp_bwd_read_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_mlp_bwd_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_mlp_bwd_status, &zero, sizeof(int));
    return v;
}

}  // namespace na1d
