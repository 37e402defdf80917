// Parameter gradients of projections, dw = dy^T x and db = column sums of dy, in fp32 and for up to two projections in one launch:
// products of CTA pairs on tcgen05 with the rows split over the SMs.
//
// A gradient has few tiles (256 x 256: 1 to 8) and a contraction over all rows (38400 at 128 x 300 frames). The library's
// products spend 28 to 36 us on each of a block's larger ones (64-column tiles: every input is read from L2 many times over) and a
// reduction after each; a pass over dy for the bias gradient came on top. Here a pair of SMs takes a 256 x 256 tile (the left
// operand's columns split over the two, the right one's too), so a row of inputs crosses from L2 once per 256 columns of the other
// operand, and the warps that later store the results add up the staged columns of dy for the bias gradient. They do so in fp32: as a product
// of the staged dy with ones, which took the same time, the sums were up to 24 times further off than those of a pass over dy, since the
// tensor cores do not round to nearest; they are as exact as that pass now. Bound by the L2's bandwidth
// (8.7 TB/s with nothing but the loads): 38400 rows, 1024 x 256 and 256 x 1024: 48 us with the sum over splits, 314 MB from L2
// (30 us of HBM time), against 88 us for the library's products and two passes of column sums; 768 x 256 and 256 x 256: 38 against 63 us.
#include "na1d_internal.h"
#include "na1d_pair.cuh"

namespace na1d {
namespace {

__device__ int g_wgrad_status = 0;

constexpr int kThreads = 384;                    // warp 0: loads, 1: MMA issue, 2: tensor memory, 4-11: column sums and results
constexpr int kStep = 64;                        // rows per shared-memory stage
constexpr int kTile = 256;
constexpr int kHalf = kTile / 2;                 // columns of either operand in one CTA
constexpr int kBox = 64 * kStep * 2;             // 64 columns of a stage: one row of the 128-byte swizzle per contraction row
constexpr int kStageBytes = 4 * kBox;            // two boxes of each operand
constexpr int kStages = 7;
constexpr int kSmem = kStages * kStageBytes + 1024;
constexpr int kMost = 2;                         // projections per launch
constexpr uint32_t kCols = 256;

struct Barriers {
    uint64_t full[kStages], empty[kStages], used[kStages], acc_full, acc_empty;   // of a stage: loaded, multiplied, added up
    uint32_t tmem;
    int abort;
};
struct Product {
    int M, N;                       // rows and columns of the gradient
    int tiles_n, splits;
    int first;                      // number of this projection's first work item (tile, split)
};
struct Work {
    Product p[kMost];
    int count, items, steps;
};
struct Maps { CUtensorMap a[kMost], b[kMost]; };

struct Item {
    int p, m0, n0, k0, k1;
};
__device__ __forceinline__ Item item_at(const Work& w, int i) {
    Item t;
    t.p = w.count > 1 && i >= w.p[1].first ? 1 : 0;
    const Product& q = w.p[t.p];
    i -= q.first;
    const int tile = i / q.splits, s = i - tile * q.splits, tm = tile / q.tiles_n;
    t.m0 = tm * kTile;
    t.n0 = (tile - tm * q.tiles_n) * kTile;
    t.k0 = (int)((long long)w.steps * s / q.splits);
    t.k1 = (int)((long long)w.steps * (s + 1) / q.splits);
    return t;
}

// Both operands contract across their staged rows. One thread of each CTA loads its half of the columns, one thread of the
// leader issues; partial sums leave in the order tensor memory has them (a row per lane), 512 bytes to an instruction.
template <typename E>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    wgrad_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Work work, float* __restrict__ part, float* __restrict__ part_bias) {
    extern __shared__ uint8_t raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    __shared__ Barriers bar;
    const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = pair::cta_rank();
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
    volatile int* abort_flag = &bar.abort;

    if (warp == 0) {
        if (lane < kStages) { ptx::mbar_init(&bar.full[lane], 1); ptx::mbar_init(&bar.empty[lane], 1); ptx::mbar_init(&bar.used[lane], 8); }
        else if (lane == kStages) { ptx::mbar_init(&bar.acc_full, 1); ptx::mbar_init(&bar.acc_empty, 16); bar.abort = 0; }
        ptx::fence_mbar_init();
    } else if (warp == 1 && lane < work.count) {
        ptx::prefetch_tensormap(&maps.a[lane]);
        ptx::prefetch_tensormap(&maps.b[lane]);
    }
    if (warp == 2) { pair::tmem_alloc(&bar.tmem, kCols); pair::tmem_relinquish(); }
    ptx::tc_fence_before_sync();
    __syncthreads();
    pair::cluster_sync();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = bar.tmem;

    if (warp == 0) {
        if (ptx::elect_one()) {
            int slot = 0, n = 0;
            uint32_t phase = 1;   // the first round finds the slots empty
            bool ok = true;
            for (int i = first; ok && i < work.items; i += step) {
                const Item t = item_at(work, i);
                const CUtensorMap *ma = &maps.a[t.p], *mb = &maps.b[t.p];
                const int m = t.m0 + rank * kHalf, nn = t.n0 + rank * kHalf;
                for (int k = t.k0; k < t.k1; ++k) {
                    if (!ptx::mbar_wait_relaxed(&bar.used[slot], phase) || *abort_flag) { atomicExch(&g_wgrad_status, 1); *abort_flag = 1; ok = false; break; }
                    const uint32_t full = pair::in_leader(&bar.full[slot]);
                    uint8_t* s = smem + slot * kStageBytes;
                    if (rank == 0) ptx::mbar_expect_tx(&bar.full[slot], 2 * kStageBytes);
                    pair::load_2d(s, ma, full, m, k * kStep);
                    pair::load_2d(s + kBox, ma, full, m + 64, k * kStep);
                    pair::load_2d(s + 2 * kBox, mb, full, nn, k * kStep);
                    pair::load_2d(s + 3 * kBox, mb, full, nn + 64, k * kStep);
                    ++n;
                    if (++slot == kStages) { slot = 0; phase ^= 1; }
                }
            }
            if (!ok && rank == 0)   // loads that are on their way arrive before the CTAs leave
                for (int j = n - 1; j >= 0 && j >= n - kStages; --j) ptx::mbar_wait(&bar.full[j % kStages], (j / kStages) & 1, 1u << 14);
        }
    } else if (warp == 1) {
        if (rank == 0 && ptx::elect_one()) {
            constexpr uint32_t fmt = tc::Fmt<E>::v;
            constexpr uint32_t idesc = ptx::instr_desc(fmt, 1, 1, 256, kTile);
            int slot = 0, it = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int i = first; ok && i < work.items; i += step, ++it) {
                const Item t = item_at(work, i);
                if (!ptx::mbar_wait(&bar.acc_empty, (it & 1) ^ 1) || *abort_flag) { atomicExch(&g_wgrad_status, 2); *abort_flag = 1; break; }
                ptx::tc_fence_after_sync();
                for (int k = t.k0; k < t.k1; ++k) {
                    if (!ptx::mbar_wait(&bar.full[slot], phase) || *abort_flag) { atomicExch(&g_wgrad_status, 3); *abort_flag = 1; ok = false; break; }
                    ptx::tc_fence_after_sync();
                    const uint32_t s = ptx::smem_u32(smem + slot * kStageBytes);
                    const uint64_t a = pair::mn_major(s, kBox), b = pair::mn_major(s + 2 * kBox, kBox);
#pragma unroll
                    for (int j = 0; j < kStep / 16; ++j)
                        pair::mma_ss(tmem, tc::desc_advance(a, j * 2048), tc::desc_advance(b, j * 2048), idesc, k > t.k0 || j > 0);
                    pair::commit(&bar.empty[slot]);
                    if (++slot == kStages) { slot = 0; phase ^= 1; }
                }
                pair::commit(&bar.acc_full);
            }
        }
    } else if (warp >= 4) {
        // Column sums, of a stage that the products have read (`empty`: both CTAs learn of it; the loads count on the leader's barriers alone). The
        // stage is loaded again when these warps are through with it too. A lane takes rows r, r + 16, .. of a stage and eight adjacent columns (lanes of one phase of an access: eight rows, whose
        // swizzle puts them on all banks)
        const int r = lane & 15, chunk = 2 * (warp - 4) + (lane >> 4);
        const uint8_t* column = smem + (chunk >> 3) * kBox + r * 128 + (((chunk & 7) ^ (r & 7)) << 4);
        int slot = 0;
        uint32_t phase = 0;
        const int q = warp & 3, h = (warp - 4) >> 2;   // tensor-memory lanes 32 q .. + 31 (those a warp reaches), half h of the columns
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        int it = 0;
        for (int i = first; i < work.items; i += step, ++it) {
            const Item t = item_at(work, i);
            float sum[8] = {};
            bool ok = true;
            for (int k = t.k0; k < t.k1; ++k) {
                if (!pair::wait_cluster(&bar.empty[slot], phase) || *abort_flag) { atomicExch(&g_wgrad_status, 5); *abort_flag = 1; ok = false; break; }
                if (t.n0 == 0) {
                    float v[4][8];
#pragma unroll
                    for (int j = 0; j < 4; ++j) Cvt<E>::unpack(*reinterpret_cast<const uint4*>(column + slot * kStageBytes + j * 16 * 128), v[j]);
#pragma unroll
                    for (int c = 0; c < 8; ++c) sum[c] += (v[0][c] + v[1][c]) + (v[2][c] + v[3][c]);
                }
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&bar.used[slot]);
                if (++slot == kStages) { slot = 0; phase ^= 1; }
            }
            if (!ok) break;
            if (t.n0 == 0) {
#pragma unroll
                for (int c = 0; c < 8; ++c)
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) sum[c] += __shfl_xor_sync(0xffffffffu, sum[c], o);
                if (r == 0) {
                    float4* dst = reinterpret_cast<float4*>(part_bias + ((size_t)i * 8 + rank * 4) * 32 + chunk * 8);
                    dst[0] = make_float4(sum[0], sum[1], sum[2], sum[3]);
                    dst[1] = make_float4(sum[4], sum[5], sum[6], sum[7]);
                }
            }
            if (!ptx::mbar_wait_relaxed(&bar.acc_full, it & 1) || *abort_flag) { atomicExch(&g_wgrad_status, 4); *abort_flag = 1; break; }
            ptx::tc_fence_after_sync();
            const size_t band = (size_t)i * 8 + rank * 4 + q;
            float4* dst = reinterpret_cast<float4*>(part) + band * (kTile / 4) * 32 + lane;
#pragma unroll 1
            for (int c = h * kHalf; c < (h + 1) * kHalf; c += 32) {
                float d[32];
                pair::tmem_ld32(tmem + lanes + c, d);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) dst[(c / 4 + j) * 32] = make_float4(d[4 * j], d[4 * j + 1], d[4 * j + 2], d[4 * j + 3]);
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) pair::arrive_cluster(pair::in_leader(&bar.acc_empty));
        }
    }
    __syncwarp();
    ptx::tc_fence_before_sync();
    __syncthreads();
    pair::cluster_sync();   // neither CTA leaves while the other may still signal it or read its operands
    if (warp == 2) pair::tmem_dealloc(tmem, kCols);
}

// Adds up the splits' partial sums in a fixed order and writes the gradients: a CTA per 32 rows x 32 columns of a tile (the
// splits shared out over its four groups of 64 threads), turned around in shared memory (a partial has a row per lane, the result is
// written along its rows).
struct Sums {
    void *w[kMost], *b[kMost];
    int block0[kMost];
};
template <typename O>
__global__ void __launch_bounds__(1024) wgrad_sum_kernel(const __grid_constant__ Work work, const __grid_constant__ Sums out, const float4* __restrict__ part,
                                                         const float* __restrict__ part_bias) {
    __shared__ float sm[4][32][33];
    const int p = work.count > 1 && (int)blockIdx.x >= out.block0[1] ? 1 : 0;
    const Product& q = work.p[p];
    int x = blockIdx.x - out.block0[p];
    const int piece = x & 7;
    x >>= 3;
    const int band = x & 7, tile = x >> 3, tm = tile / q.tiles_n, n0 = (tile - tm * q.tiles_n) * kTile + piece * 32, m0 = tm * kTile + band * 32;
    if (m0 >= q.M || n0 >= q.N) return;
    const int lane = threadIdx.x & 31, cg = (threadIdx.x >> 5) & 7, quarter = threadIdx.x >> 8;
    const size_t item0 = (size_t)q.first + (size_t)tile * q.splits;
    const float4* src = part + ((item0 * 8 + band) * (kTile / 4) + piece * 8 + cg) * 32 + lane;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 5
    for (int k = quarter; k < q.splits; k += 4) {
        const float4 v = __ldg(src + (size_t)k * 8 * (kTile / 4) * 32);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    float* d = &sm[quarter][lane][cg * 4];
    d[0] = s.x; d[1] = s.y; d[2] = s.z; d[3] = s.w;
    __syncthreads();
    const int row = threadIdx.x >> 5;
    if (out.w[p] && n0 + lane < q.N && m0 + row < q.M)
        reinterpret_cast<O*>(out.w[p])[(size_t)(m0 + row) * q.N + n0 + lane] = O((sm[0][row][lane] + sm[1][row][lane]) + (sm[2][row][lane] + sm[3][row][lane]));
    if (out.b[p] && n0 == 0 && m0 + row < q.M) {   // a warp to a column, a lane to every 32nd split
        float b = 0.f;
        for (int k = lane; k < q.splits; k += 32) b += __ldg(part_bias + ((item0 + k) * 8 + band) * 32 + row);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
        if (lane == 0) reinterpret_cast<O*>(out.b[p])[m0 + row] = O(b);
    }
}

int pairs_on_device() { return device_sm_count() / 2; }
int tiles_of(int64_t x) { return (int)((x + kTile - 1) / kTile); }

Work plan(const int64_t* M, const int64_t* N, int count, int64_t rows) {
    Work w = {};
    w.count = count;
    w.steps = (int)((rows + kStep - 1) / kStep);
    int tiles = 0;
    for (int i = 0; i < count; ++i) tiles += tiles_of(M[i]) * tiles_of(N[i]);
    // one round of pairs; fewer splits where a split would have less than four steps of its own
    int splits = pairs_on_device() / tiles;
    if (splits > w.steps / 4) splits = w.steps / 4;
    if (splits < 1) splits = 1;
    for (int i = 0; i < count; ++i) {
        w.p[i] = Product{(int)M[i], (int)N[i], tiles_of(N[i]), splits, w.items};
        w.items += tiles_of(M[i]) * tiles_of(N[i]) * splits;
    }
    return w;
}
template <typename E, typename O>
cudaError_t run(void* const* d_w, void* const* d_b, const void* const* dy, const void* const* x, const int64_t* M, const int64_t* N, int count,
                int64_t rows, float* scratch, int dtype, cudaStream_t st) {
    const Work w = plan(M, N, count, rows);
    Maps maps;
    Sums out = {};
    int blocks = 0;
    for (int i = 0; i < count; ++i) {
        const int64_t da[2] = {M[i], rows}, sa[1] = {M[i]}, db[2] = {N[i], rows}, sb[1] = {N[i]};
        const int box[2] = {64, kStep};
        if (!make_matrix_map(&maps.a[i], dy[i], dtype, 2, da, sa, box) || !make_matrix_map(&maps.b[i], x[i], dtype, 2, db, sb, box)) return cudaErrorInvalidValue;
        out.w[i] = d_w[i];
        out.b[i] = d_b[i];
        out.block0[i] = blocks;
        blocks += w.p[i].tiles_n * tiles_of(M[i]) * 64;
    }
    auto* kern = wgrad_kernel<E>;
    if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)) return e;
    const int pairs = w.items < pairs_on_device() ? w.items : pairs_on_device();
    float* part_bias = scratch + (size_t)w.items * kTile * kTile;
    kern<<<2 * pairs, kThreads, kSmem, st>>>(maps, w, scratch, part_bias);
    if (cudaError_t e = cudaGetLastError()) return e;
    wgrad_sum_kernel<O><<<blocks, 1024, 0, st>>>(w, out, reinterpret_cast<const float4*>(scratch), part_bias);
    return cudaGetLastError();
}

}  // namespace

size_t wgrad_scratch_floats(const int64_t* M, const int64_t* N, int count, int64_t rows) {
    return (size_t)plan(M, N, count, rows).items * (kTile * kTile + kTile);
}
cudaError_t wgrad(void* const* d_w, void* const* d_b, const void* const* dy, const void* const* x, const int64_t* M, const int64_t* N, int count,
                  int64_t rows, float* scratch, bool out32, int dtype, cudaStream_t st) {
    bind_primary_context();
    using B = __nv_bfloat16;
    if (dtype == 0)
        return out32 ? run<B, float>(d_w, d_b, dy, x, M, N, count, rows, scratch, dtype, st) : run<B, B>(d_w, d_b, dy, x, M, N, count, rows, scratch, dtype, st);
    return out32 ? run<__half, float>(d_w, d_b, dy, x, M, N, count, rows, scratch, dtype, st)
                 : run<__half, __half>(d_w, d_b, dy, x, M, N, count, rows, scratch, dtype, st);
}
int wgrad_read_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_wgrad_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_wgrad_status, &zero, sizeof(int));
    return v;
}

}  // namespace na1d
