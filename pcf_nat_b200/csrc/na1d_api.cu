// C ABI of the library: argument validation, kernel-family choice, launches. No torch types.
#include "../../include/na1d_b200.h"
#include "na1d_internal.h"

#include <atomic>
#include <climits>
#include <cmath>
#include <mutex>

namespace {

thread_local int g_last_cuda_error = 0;
std::atomic<int> g_family_override{-1};

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return NA1D_OK;
    g_last_cuda_error = (int)e;
    return NA1D_ERR_CUDA;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_geometry(int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, int dtype,
                   float scale, na1d::Geometry& g) {
    if (dtype != NA1D_BF16 && dtype != NA1D_FP16) return NA1D_ERR_BAD_DTYPE;
    if (N <= 0 || T <= 0 || C <= 0 || C % 8 != 0 || C > 256) return NA1D_ERR_BAD_SHAPE;
    if (!na1d::simt_supports_channels((int)C)) return NA1D_ERR_BAD_SHAPE;
    if (win <= 0 || win > NA1D_MAX_WINDOW || left < 0 || left >= win || dil <= 0) return NA1D_ERR_BAD_WINDOW;
    if (heads <= 0 || N % heads != 0) return NA1D_ERR_BAD_HEADS;
    // every flat index used by the kernels must fit int32: rows, rows*win, window reach
    if (N * T > INT_MAX || N * T * win > INT_MAX || T * win > INT_MAX || win * dil > INT_MAX / 2 ||
        T + win * dil > INT_MAX / 2)
        return NA1D_ERR_BAD_SHAPE;
    g.N = (int)N; g.H = (int)heads; g.T = (int)T; g.C = (int)C; g.win = (int)win; g.left = (int)left; g.dil = (int)dil;
    g.scale = scale;
    return NA1D_OK;
}

// What a call asks of the kernels, for the cost models below: microseconds, fitted to graph replays of 700 calls of the unfused
// operators and 400 of the fused pair on general shapes (8 to 128 channels, windows 2 to 80, dilations 1 to 4, residues of 2 to 2000
// rows, 100 to a million rows, both types); the median error of a model is 7 to 12 %.
struct Work {
    double rows, C, CP, win, met, meet;   // met: neighbours inside the sequence, on average; meet: at most
    double chunks, ctas, staged, blocks, per_cta;   // 16-row chunks of a block's window; CTAs, staged and own 16-row blocks of the warp-level kernels
    Work(const na1d::Geometry& g, int rows_cta) : rows((double)g.N * g.T), C(g.C), win(g.win) {
        const double tp = (g.T + g.dil - 1) / g.dil, residues = (double)g.N * (g.dil < g.T ? g.dil : g.T);
        auto side = [tp](double n) { n = n < tp - 1 ? n : tp - 1; return n - n * (n + 1) / (2 * tp); };
        met = 1 + side(g.left) + side(g.win - 1 - g.left);
        meet = win < tp ? win : tp;
        CP = g.C <= 64 ? (g.C + 15) / 16 * 16 : g.C <= 96 ? 96 : 128;
        chunks = (g.win + 30) / 16;
        const double tiles = std::ceil(tp / rows_cta), own = std::ceil(tp / 16);
        ctas = residues * tiles;
        blocks = residues * own;
        staged = residues * (own + tiles * (chunks - 1));
        per_cta = own < rows_cta / 16 ? own : rows_cta / 16;
    }
};
// CUDA-core kernels: a thread group walks the window of its row (latency), C operations a neighbour (throughput); neighbours outside
// the sequence are skipped
struct CoreCost {
    double start, met, skipped, row, product, skip;
    double operator()(const Work& w) const {
        return start + met * w.meet + skipped * (w.win - w.meet) + 1e-3 * w.rows * (w.C * (row + product * w.met) + skip * (w.win - w.met));
    }
};
// warp-level kernels: a CTA per 64 or 128 rows of a residue, whatever the window and however few of the rows there are
struct WarpCost {
    double start, chunk, stage, cta, staged, block, product;
    double operator()(const Work& w) const {
        return start + chunk * w.chunks + stage * (w.per_cta + w.chunks - 1) * w.CP +
               1e-3 * (w.ctas * cta + w.staged * w.CP * staged + w.blocks * w.chunks * (block + product * w.CP));
    }
};
// tcgen05 kernels on the flat tiling: rows, in three window buckets
struct TileCost {
    double start, row, channel, bucket[3], neighbour;
    double operator()(const Work& w, int weff) const {
        return start + 1e-3 * w.rows * (row + channel * w.C + bucket[weff <= 9 ? 0 : weff <= 17 ? 1 : 2] + neighbour * w.win);
    }
};
// Which kernels run an unfused operator. Kernels that would lose bits are no candidates:
//   q.k        fp32 results: matrix instructions (fp32 sums rounded towards zero, 2 to 3 times the CUDA-core kernels' error) only where
//              the tcgen05 kernels take the shape;
//   band . x   the marching form splits the fp32 band into two 16-bit pieces, against one in the tcgen05 kernels: only where those take the
//              shape;
//   transposed as band . x, and with three bf16 pieces where the CUDA cores stood; not for fp16, whose pieces lack the band's exponents.
// Dilation 1, windows up to 33, 32 tokens and more (570 drawn calls; us are CUDA core / tcgen05 / warp-level / marching): the marching
// kernels at 16, 32 and 64 channels, but
//   for few products a row the CUDA cores (8192 x 150 rows of 16 channels, window 3: 22 / 40 / 52 / 24; window 5, a.v: 29 / 57 / 76 / 37);
//   at 64 channels the tcgen05 kernels in q.k up to window 30 (1089 x 126 rows, window 30: 65 / 10 / 14 / 12; 3456 x 150, window 33: 253 /
//   55 / 70 / 41), and in a.v of large calls with narrow windows or blocks of 16 with many empty rows (13886 x 33 rows, window 8: 52 / 34 /
//   114 / 42; 3456 x 150, window 27: 167 / 49 / 85 / 41);
//   transposed, large calls of 64 channels with windows of 4 and 5 on tcgen05 (448 x 547 rows, window 4: 18 us, marching 23);
//   transposed fp16 bands go to the CUDA cores, for large calls to tcgen05 at 64 channels and windows up to 17 and at 32 channels and windows
//   up to 20 or short sequences (19636 x 34 rows of 64 channels, window 10: 99 / 86 / 160; 3773 x 40 of 32, window 18: 22 / 18 / 23), else
//   to the warp-level kernels (6912 x 150 rows of 32 channels, window 27: 191 / 159 / 122).
// They take 0.81 (q.k), 0.64 (a.v), 0.59 and 0.66 (transposed, bf16 and fp16) of the time that tcgen05 and, where it does not run, the CUDA
// cores take; 5 of 1140 calls are more than 3 % slower than those, at most 1.12 times.
// Everything else by the cost models, where the kernels that are natural for the shape (tcgen05 where they take it, else CUDA-core) are left
// for a predicted gain of 10 %, the models' error: 0.82 (a.v) and 0.82 (transposed) of the CUDA cores' time over 340 calls, 2 % of them more
// than 3 % slower, at most 1.16 times.
enum class Unfused { core, tcgen05, warp, march };
enum class Op { products, rows, transposed };
Unfused pick_unfused(const na1d::Geometry& g, Op op, int dtype, bool aligned_band) {
    const int forced = g_family_override.load(), weff = (g.win - 1) * g.dil + 1;
    const bool warp_ok = na1d::mma_band_supports(g), march_ok = na1d::march_band_supports(g);
    const bool tiles = na1d::tc_unfused_supports(g) && aligned_band, tc = op == Op::transposed ? na1d::tc_unfused_t_supports(g) : tiles;
    if (forced == 0) return Unfused::core;
    if (forced == 4 && march_ok) return Unfused::march;
    if (forced == 3 || forced == 4) return warp_ok ? Unfused::warp : Unfused::core;
    if (forced == 1 && tc) return Unfused::tcgen05;
    // the tcgen05 form of the transposed product gathers the band along its diagonals: at 16 channels not for windows above 17
    const bool tc_first = tc && !(op == Op::transposed && g.C == 16 && weff > 17);
    if (g.dil == 1 && tiles && march_ok && warp_ok) {
        const int products = g.C * g.win, blocks = (g.T + 15) / 16;
        const bool large = (long long)g.N * g.T > 100000, wide = g.C == 64;
        switch (op) {
            case Op::products: return products <= 64 ? Unfused::core : wide && g.win <= 30 ? Unfused::tcgen05 : Unfused::march;
            case Op::rows:
                if (products <= 112 || (wide && large && g.win <= 3)) return Unfused::core;
                return wide && large && (g.win <= 8 || g.T < 0.87 * 16 * blocks) ? Unfused::tcgen05 : Unfused::march;
            default:
                if (dtype == NA1D_BF16) return products <= (wide ? 192 : 112) ? Unfused::core : wide && large && g.win <= 5 && tc ? Unfused::tcgen05 : Unfused::march;
                if (products <= (g.C == 16 && large ? 340 : 288)) return Unfused::core;
                if (tc_first && wide && (large || g.win <= 9)) return Unfused::tcgen05;
                if (tc_first && g.C == 32 && large && (g.win <= 20 || g.T < 0.8 * 16 * blocks)) return Unfused::tcgen05;
                return Unfused::warp;
        }
    }
    constexpr CoreCost core[3] = {{1.43, 0.244, 0.0796, 0.000374, 0.000189, 0.00513}, {1.41, 0.21, 0.0513, 0.000358, 0.000125, 0.00132},
                                  {1.4, 0.227, 0.0541, 0.000319, 0.000147, 0.00113}};
    constexpr TileCost tile[3] = {{3.04, 0.00879, 0.000315, {0.0115, 0.0131, 0.0128}, 0.000645}, {4.24, 0.0226, 0.000466, {0.00737, 0.0148, 0.0317}, 6.87e-05},
                                  {4.56, 0.0293, 0.000547, {0.00252, 0.022, 0.0421}, 0.000407}};
    constexpr WarpCost warp[3] = {{}, {1.37, 0.406, 0.00316, 1.6, 0.0183, 0.115, 0.}, {0.808, 0.685, 0.00327, 1.63, 0.0211, 0.139, 0.}};
    const Work w(g, 128);
    const int i = (int)op;
    const double natural = 0.9;
    double best = core[i](w) * (tc_first ? 1. : natural);
    Unfused pick = Unfused::core;
    auto consider = [&](Unfused u, double cost) { if (cost < best) { best = cost; pick = u; } };
    if (tc_first) consider(Unfused::tcgen05, natural * tile[i](w, weff));
    if (warp_ok && op != Op::products) consider(Unfused::warp, warp[i](w));
    return pick;
}

// arguments of the row and column kernels of a transformer block
int check_block(int64_t rows, int64_t cols, int64_t most_cols, int dtype) {
    if (dtype != NA1D_BF16 && dtype != NA1D_FP16) return NA1D_ERR_BAD_DTYPE;
    if (rows <= 0 || cols <= 0 || cols % 8 != 0 || cols > most_cols || rows > INT_MAX / 2 || rows > (1ll << 40) / cols) return NA1D_ERR_BAD_SHAPE;
    return NA1D_OK;
}
template <typename... P> int check_pointers(const P*... p) {
    if (((p == nullptr) || ...)) return NA1D_ERR_NULL_POINTER;
    return (aligned16(p) && ...) ? NA1D_OK : NA1D_ERR_MISALIGNED;
}

#define NA1D_REQUIRE_PTR(p) do { if ((p) == nullptr) return NA1D_ERR_NULL_POINTER; } while (0)
#define NA1D_REQUIRE_ALIGNED(p) do { if (!aligned16(p)) return NA1D_ERR_MISALIGNED; } while (0)

// Of the general kernels (na1d_mma.cu, na1d_simt.cu) the cheaper one by the models above, the warp-level one for a gain of 10 %: over 400
// drawn calls 0.46 of the CUDA-core kernels' time in the forward and 0.42 in the backward, geometric mean; eleven of the 800 are more than 3 %
// slower, at most 1.5 times (a window of 76 on sequences of 15 rows). Few neighbours of short residues stay on the CUDA cores: 2048 x 20 rows
// of 48 channels with dilation 4, window 15, take 11 us there and 30 here forward, 66 and 112 backward.
bool use_mma(const na1d::Geometry& g, bool fp16, bool has_bias, bool backward) {
    const int forced = g_family_override.load();
    if (forced == 0 || !na1d::mma_supports(g)) return false;
    if (forced == 3 || forced == 4) return true;
    if ((g.T + g.dil - 1) / g.dil < 8 && g.win < 8) return false;
    const Work w(g, 64);
    // fp16 weights go through products of half the depth
    const double mma = (backward ? WarpCost{3.19, 0.208, 0.00994, 1.84, 0.1, 0., 0.} : WarpCost{2.52, 0.177, 0.00392, 1.39, 0.0177, 0.146, fp16 ? 0.00344 : 0.00103})(w);
    double core = (backward ? CoreCost{3.93, 0.505, 0.267, 0.00224, 0.000938, 0.00919} : CoreCost{1.86, 0.455, 0.179, 0.00035, 0.000339, 0.00659})(w);
    if (has_bias && !backward) core += 1e-3 * w.rows * w.win * 0.000319;
    if (has_bias && backward) {   // its gradient: the rows that share a warp add to the same entry, one after the other
        int lanes = 1, units = g.C / 8;
        while (lanes < 8 && units % 2 == 0) { lanes *= 2; units /= 2; }
        core += w.win * (0.0779 * (32 / lanes) + 1e-3 * w.rows * (units == 3 ? 0.039 : 0.013));
    }
    return mma < 0.9 * core;
}

// The marching kernels: 16-channel rows in everything; 32-channel rows in the forward, where they stand for the segmented tiling
// (any strides, no empty tile rows: 85 -> 51 us for 4096 x 150 rows, window 27) and, on dense tensors, for all but large calls of short
// sequences (below). A forced family 2 takes them too where it takes the shape (a dense call then gives the bits of a strided one); 4 is
// the same without that tiling's own limits, 5 the segmented tiling alone.
// The backward at 16 channels on dense tensors leaves large calls of 33 to 39 rows a residue to the flat tiling, which has no empty rows
// there (three blocks of 16): 26857 x 33 rows, window 25, 92 us against 119; 12592 x 36, window 27, 52 / 60; 18712 x 39, window 26, 92 / 104; 10768 x 43,
// window 33, 55 / 55.
enum class Pass { forward, strided_forward, backward, strided_backward };
template <typename... S> bool use_march(const na1d::Geometry& g, Pass pass, bool wants_bias_grad, const S&... strides) {
    const int forced = g_family_override.load();
    if (forced != -1 && forced != 4 && !(forced == 2 && na1d::tc_seg_supports(g))) return false;
    // (where the CUDA cores stood before -- more than 32 heads, residues of one token -- infinities and NaN stay in their windows: the
    // general kernels see to that, these, like the tcgen05 ones, do not)
    if (forced == -1 && !na1d::tc_seg_supports(g) && !na1d::tc_fwd_supports(g)) return false;
    // (a bias gradient in a fixed order, where the environment asks for it, is the tcgen05 kernels')
    const bool backward = pass == Pass::backward || pass == Pass::strided_backward;
    if (forced == -1 && backward && wants_bias_grad && na1d::bias_grad_partial_rows()) return false;
    const int residue = (g.T + g.dil - 1) / g.dil;
    if (forced == -1 && pass == Pass::backward && residue > 32 && residue < 40 && (long long)g.N * g.T > (1 << 17) &&
        na1d::tc_bwd_supports(g, true, wants_bias_grad))
        return false;
    // Dense forward at 32 channels: large calls with short sequences stay on the flat tiling (2800 x 97 rows, window 9, 21.2 us against 23.1,
    // window 27 24.0 / 24.9: a badly filled second round of warps; at most a tenth is lost by it: 4096 x 150 40.5 / 37.2 and 47.2 / 46.8). Longer
    // ones: 2048 x 300 rows 41.0 / 35.0 (window 9), 46.1 / 45.7 (27), 1600 x 1000 92.5 / 81.1 and 108 / 93. Dilated ones, whose other
    // tiling would be the segmented one or a wide band: 1.0 (2800 x 97, dilation 2) to 3.1 times (8000 x 64, dilation 3: 151 / 49).
    if (forced == -1 && pass == Pass::forward && g.C == 32 && g.dil == 1 && g.T < 256 && (long long)g.N * g.T > (1 << 18)) return false;
    return na1d::march_supports(g, backward) && ((strides.token * g.dil < (1ll << 30)) && ...);
}
}  // namespace

extern "C" {

const char* na1d_status_string(int status) {
    switch (status) {
        case NA1D_OK: return "ok";
        case NA1D_ERR_NULL_POINTER: return "a required pointer is NULL";
        case NA1D_ERR_BAD_SHAPE: return "bad shape: need N,T,C > 0, C a supported multiple of 8 (<= 256), sizes within int32";
        case NA1D_ERR_BAD_WINDOW: return "bad window: need 0 < win <= 128, 0 <= left < win, dil >= 1";
        case NA1D_ERR_BAD_DTYPE: return "bad dtype: expected NA1D_BF16 or NA1D_FP16";
        case NA1D_ERR_BAD_HEADS: return "bad heads: need heads > 0 and N divisible by heads";
        case NA1D_ERR_MISALIGNED: return "a 16-bit tensor pointer is not 16-byte aligned";
        case NA1D_ERR_CUDA: return "a CUDA call failed (see na1d_last_cuda_error)";
        case NA1D_ERR_DEVICE_TIMEOUT: return "a bounded wait inside a kernel expired";
        case NA1D_ERR_TOO_LARGE: return "problem exceeds a fixed capacity of this entry point (e.g. N*T above NA1D_STATIC_SCRATCH_ROWS)";
        case NA1D_ERR_UNSUPPORTED: return "the requested kernel family or tiling does not support this shape";
        case NA1D_ERR_BAD_DROPOUT: return "bad dropout probability: need 0 <= p < 1";
        case NA1D_ERR_BAD_STRIDE: return "bad stride: element strides must be positive multiples of 8, the token stride >= C";
        default: return "unknown status";
    }
}
int na1d_last_cuda_error(void) { return g_last_cuda_error; }
int na1d_version(void) { return 100; }

int na1d_qk_forward(float* attn, const void* q, const void* k, int64_t N, int64_t T, int64_t C, int64_t win,
                    int64_t left, int64_t dil, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(attn); NA1D_REQUIRE_PTR(q); NA1D_REQUIRE_PTR(k);
    NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k);
    na1d::Geometry g;
    if (int s = check_geometry(N, 1, T, C, win, left, dil, dtype, 1.f, g)) return s;
    switch (pick_unfused(g, Op::products, dtype, aligned16(attn))) {   // (the tcgen05 band goes out in 16-byte stores)
        case Unfused::tcgen05: return cuda_status(na1d::tc_qk(attn, q, k, g, dtype, (cudaStream_t)stream));
        case Unfused::march: return cuda_status(na1d::march_band_out(attn, q, k, g, dtype, (cudaStream_t)stream));
        case Unfused::warp: return cuda_status(na1d::mma_band_out(attn, q, k, g, dtype, (cudaStream_t)stream));
        default: return cuda_status(na1d::simt_qk(attn, q, k, g, dtype, (cudaStream_t)stream));
    }
}
int na1d_a_backward(float* attn_gd, const void* result_gd, const void* v, int64_t N, int64_t T, int64_t C, int64_t win,
                    int64_t left, int64_t dil, int dtype, void* stream) {
    return na1d_qk_forward(attn_gd, result_gd, v, N, T, C, win, left, dil, dtype, stream);
}
int na1d_q_backward(void* q_gd, const float* attn_gd, const void* k, int64_t N, int64_t T, int64_t C, int64_t win,
                    int64_t left, int64_t dil, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(q_gd); NA1D_REQUIRE_PTR(attn_gd); NA1D_REQUIRE_PTR(k);
    NA1D_REQUIRE_ALIGNED(q_gd); NA1D_REQUIRE_ALIGNED(k);
    na1d::Geometry g;
    if (int s = check_geometry(N, 1, T, C, win, left, dil, dtype, 1.f, g)) return s;
    switch (pick_unfused(g, Op::rows, dtype, true)) {
        case Unfused::tcgen05: return cuda_status(na1d::tc_band_x(q_gd, attn_gd, k, g, dtype, (cudaStream_t)stream));
        case Unfused::march: return cuda_status(na1d::march_band_rows(q_gd, attn_gd, k, false, g, dtype, (cudaStream_t)stream));
        case Unfused::warp: return cuda_status(na1d::mma_band_rows(q_gd, attn_gd, k, false, g, dtype, (cudaStream_t)stream));
        default: return cuda_status(na1d::simt_band_x(q_gd, attn_gd, k, g, dtype, (cudaStream_t)stream));
    }
}
int na1d_av_forward(void* result, const float* attn, const void* v, int64_t N, int64_t T, int64_t C, int64_t win,
                    int64_t left, int64_t dil, int dtype, void* stream) {
    return na1d_q_backward(result, attn, v, N, T, C, win, left, dil, dtype, stream);
}
int na1d_k_backward(void* k_gd, const float* attn_gd, const void* q, int64_t N, int64_t T, int64_t C, int64_t win,
                    int64_t left, int64_t dil, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(k_gd); NA1D_REQUIRE_PTR(attn_gd); NA1D_REQUIRE_PTR(q);
    NA1D_REQUIRE_ALIGNED(k_gd); NA1D_REQUIRE_ALIGNED(q);
    na1d::Geometry g;
    if (int s = check_geometry(N, 1, T, C, win, left, dil, dtype, 1.f, g)) return s;
    switch (pick_unfused(g, Op::transposed, dtype, true)) {
        case Unfused::tcgen05: return cuda_status(na1d::tc_bandT_x(k_gd, attn_gd, q, g, dtype, (cudaStream_t)stream));
        case Unfused::march: return cuda_status(na1d::march_band_rows(k_gd, attn_gd, q, true, g, dtype, (cudaStream_t)stream));
        case Unfused::warp: return cuda_status(na1d::mma_band_rows(k_gd, attn_gd, q, true, g, dtype, (cudaStream_t)stream));
        default: return cuda_status(na1d::simt_bandT_x(k_gd, attn_gd, q, g, dtype, (cudaStream_t)stream));
    }
}
int na1d_v_backward(void* v_gd, const float* attn, const void* result_gd, int64_t N, int64_t T, int64_t C, int64_t win,
                    int64_t left, int64_t dil, int dtype, void* stream) {
    return na1d_k_backward(v_gd, attn, result_gd, N, T, C, win, left, dil, dtype, stream);
}

// 0 = the general kernels (warp-level matrix instructions up to 128 channels, CUDA-core kernels above), 1 = tcgen05 kernels on the flat tiling, 2 = tcgen05 kernels on the segmented tiling.
// The flat tiling takes dilation 1 and those power-of-two dilations whose dilated window still fits the widest band bucket;
// the segmented tiling takes every dilation (each residue class of a sequence is a dilation-1 problem) at the price of
// partly empty last tiles. With a dilation both can run, the one with the cheaper band bucket per useful row wins.
static int pick_family(const na1d::Geometry& g, int backward, bool has_bias = false, bool wants_bias_grad = false) {
    const int forced = g_family_override.load();
    const bool flat_ok = backward ? na1d::tc_bwd_supports(g, has_bias, wants_bias_grad) : na1d::tc_fwd_supports(g);
    const bool seg_ok = backward ? na1d::tc_bwd_seg_supports(g, has_bias, wants_bias_grad) : na1d::tc_seg_supports(g);
    if (forced == 0 || forced == 3 || forced == 4) return 0;
    if (forced == 2 || forced == 5) return seg_ok ? 2 : NA1D_ERR_UNSUPPORTED;
    if (forced == 1 && flat_ok) return 1;   // forced: the flat tiling wherever it can run (the choice below is for the automatic mode)
    int pick = 0;
    if (flat_ok && seg_ok && g.dil > 1) {
        // relative cost of a tile row in the window buckets 9 / 17 / 33 (measured at 64 utterances x 4 heads, 200 to 1000
        // tokens: the two narrow buckets cost about the same, the widest is bound by its compute warps, more so in the backward
        // with its two fragment sets per block), times the rows the
        // tiling processes per useful row, plus 10 % for the segmented tiling's shorter runs of tiles
        auto bucket_cost = [backward](int w) { return w <= 9 ? 1.0 : w <= 17 ? 1.05 : backward ? 2.0 : 1.5; };
        const int tp = (g.T + g.dil - 1) / g.dil;
        const int step = backward ? 128 - (g.win - 1) : 128;
        const double seg_rows = (double)((tp + step - 1) / step) * step / tp;
        const double flat = bucket_cost((g.win - 1) * g.dil + 1), seg = 1.1 * bucket_cost(g.win) * seg_rows;
        pick = seg < flat ? 2 : 1;
    } else if (flat_ok) {
        pick = 1;
    } else if (seg_ok) {
        pick = 2;
    }
    // Short residues leave a segmented tile of 128 rows mostly empty, and the general kernels (whose tiles hold 64, or a row at a time) take
    // less: forward at 64 channels 2000 x 64 rows, dilation 3 (22 rows a residue) 56 us against 40, 1200 x 150, dilation 4 (38) 56 / 47,
    // dilation 3 (50) 36 / 37; backward 4000 x 31 rows, window 15, dilation 3 (11 rows) 301 / 182 (64 channels), 125 / 115 (32), window 5,
    // dilation 2 (16 rows) 161 / 87 and 80 / 55, but window 15 208 / 184 and 86 / 107. At 32 channels the widest window bucket stays longer: 200000 rows,
    // window 27, residues of 12, 10 and 8 rows 205 / 254, 245 / 241 and 303 / 230 (window 33: 212 / 288, 253 / 273, 313 / 264; 18: 205 / 194 at 12).
    // (With NA1D_BIAS_GRAD_ROWS=1 a bias gradient is summed in a fixed order, which the general kernels' atomics do not give.)
    if (forced == -1 && pick == 2 && g.dil > 1 && !(backward && wants_bias_grad && na1d::bias_grad_partial_rows())) {
        const int tp = (g.T + g.dil - 1) / g.dil;
        if (backward ? tp <= (g.C == 32 && g.win > 22 ? 9 : 12) || (tp <= 16 && g.win <= 9) : tp <= 40) pick = 0;
    }
    if (forced == 1 && pick == 0) return NA1D_ERR_UNSUPPORTED;
    return pick;
}

int na1d_fused_kernel_family(int64_t N, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, int dtype,
                             int backward) {
    na1d::Geometry g;
    if (int s = check_geometry(N, 1, T, C, win, left, dil, dtype, 1.f, g)) return s;
    const int fam = pick_family(g, backward);
    return fam == 2 ? 1 : fam;
}

int na1d_fused_kernel_tiling(int64_t N, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, int dtype,
                             int backward) {
    na1d::Geometry g;
    if (int s = check_geometry(N, 1, T, C, win, left, dil, dtype, 1.f, g)) return s;
    return pick_family(g, backward);
}

int na1d_fused_kernel_route(int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, int dtype, int backward,
                            int has_bias, int wants_bias_grad) {
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, 1.f, g)) return s;
    if (use_march(g, backward ? Pass::backward : Pass::forward, wants_bias_grad != 0, na1d::dense_strides(g.H, g.T, g.C))) return 4;
    if (const int fam = pick_family(g, backward, has_bias != 0, wants_bias_grad != 0)) return fam;
    return use_mma(g, dtype == NA1D_FP16, backward ? wants_bias_grad != 0 : has_bias != 0, backward != 0) ? 3 : 0;
}

int na1d_set_kernel_family(int family) {
    if (family < -1 || family > 5) family = -1;
    return g_family_override.exchange(family);
}

int na1d_tensor_map_cache_stats(int64_t* hits, int64_t* misses) {
    NA1D_REQUIRE_PTR(hits); NA1D_REQUIRE_PTR(misses);
    long long h = 0, m = 0;
    na1d::tensor_map_cache_stats(&h, &m);
    *hits = h; *misses = m;
    return NA1D_OK;
}

int na1d_device_status(void) {
    // every word is read (and cleared) before anything is reported; an expired wait in any kernel wins over a failed read
    const int words[11] = {na1d::mlp_read_status(), na1d::mlp_bwd_read_status(), na1d::wgrad_read_status(), na1d::tc_read_status(), na1d::tc_bwd_read_status(), na1d::tc_seg_read_status(),
                          na1d::tc_bwd_seg_read_status(), na1d::tc_unfused_read_status(), na1d::tc_unfused_t_read_status(),
                          na1d::tc_drop_read_status(), na1d::tc_bwd_drop_read_status()};
    int v = 0, w = 0;
    for (int x : words) { if (x > 0) v = x; if (x < 0) w = x; }
    if (v > 0) return NA1D_ERR_DEVICE_TIMEOUT;
    if (w < 0) {
        const cudaError_t e = cudaGetLastError();
        return cuda_status(e == cudaSuccess ? cudaErrorUnknown : e);
    }
    return NA1D_OK;
}

int na1d_fused_forward(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                       const int32_t* valid_len, int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win,
                       int64_t left, int64_t dil, float scale, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(o); NA1D_REQUIRE_PTR(q); NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v);
    NA1D_REQUIRE_ALIGNED(o); NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    if (use_march(g, Pass::forward, false, na1d::dense_strides(g.H, g.T, g.C))) {
        const na1d::Strides d = na1d::dense_strides(g.H, g.T, g.C);
        return cuda_status(na1d::march_fused_fwd(o, lse, q, k, v, rpb, valid_len, d, d, d, d, g, dtype, (cudaStream_t)stream));
    }
    const int fam = pick_family(g, 0);
    if (fam < 0) return fam;
    if (fam == 1) return cuda_status(na1d::tc_fused_fwd(o, lse, q, k, v, rpb, valid_len, g, dtype, (cudaStream_t)stream));
    if (fam == 2) {
        const na1d::Strides d = na1d::dense_strides(g.H, g.T, g.C);
        return cuda_status(na1d::tc_fused_fwd_seg(o, lse, q, k, v, rpb, valid_len, d, d, d, d, g, dtype, (cudaStream_t)stream));
    }
    if (use_mma(g, dtype == NA1D_FP16, rpb != nullptr, false))
        return cuda_status(na1d::mma_fused_fwd(o, lse, q, k, v, rpb, valid_len, g, dtype, (cudaStream_t)stream));
    return cuda_status(na1d::simt_fused_fwd(o, lse, q, k, v, rpb, valid_len, g, dtype, (cudaStream_t)stream));
}

namespace {
// element strides (batch, head, token) given by the caller as three int64 on the host
int read_strides(const int64_t* p, int64_t batch, int64_t heads, int64_t T, int64_t C, na1d::Strides& out) {
    if (p == nullptr) return NA1D_ERR_NULL_POINTER;
    for (int i = 0; i < 3; ++i)
        if (p[i] <= 0 || p[i] % 8 != 0) return NA1D_ERR_BAD_STRIDE;
    if (p[2] < C) return NA1D_ERR_BAD_STRIDE;
    // the largest element offset must stay far inside int64 and inside what a tensor map can address (2^40 bytes per stride)
    const long double span = (long double)p[0] * (batch - 1) + (long double)p[1] * (heads - 1) + (long double)p[2] * (T - 1) + C;
    if (span > 4.0e12L || p[0] >= (1ll << 38) || p[1] >= (1ll << 38) || p[2] >= (1ll << 38)) return NA1D_ERR_BAD_STRIDE;
    out = na1d::Strides{(long long)p[0], (long long)p[1], (long long)p[2]};
    return NA1D_OK;
}
}  // namespace

int na1d_fused_strided_supported(int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, int dtype,
                                 int has_bias, int wants_bias_grad) {
    na1d::Geometry g;
    if (int s = check_geometry(heads, heads, T, C, win, left, dil, dtype, 1.f, g)) return s;
    return (na1d::tc_seg_supports(g) && na1d::tc_bwd_seg_supports(g, has_bias != 0, wants_bias_grad != 0)) ? 1 : 0;
}

int na1d_fused_forward_strided(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                               const int32_t* valid_len, const int64_t* o_strides, const int64_t* q_strides,
                               const int64_t* k_strides, const int64_t* v_strides, int64_t N, int64_t heads, int64_t T,
                               int64_t C, int64_t win, int64_t left, int64_t dil, float scale, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(o); NA1D_REQUIRE_PTR(q); NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v);
    NA1D_REQUIRE_ALIGNED(o); NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    na1d::Strides so, sq, sk, sv;
    const int64_t batch = N / heads;
    if (int s = read_strides(o_strides, batch, heads, T, C, so)) return s;
    if (int s = read_strides(q_strides, batch, heads, T, C, sq)) return s;
    if (int s = read_strides(k_strides, batch, heads, T, C, sk)) return s;
    if (int s = read_strides(v_strides, batch, heads, T, C, sv)) return s;
    if (!na1d::tc_seg_supports(g)) return NA1D_ERR_UNSUPPORTED;
    if (use_march(g, Pass::strided_forward, false, sq, sk, sv, so)) return cuda_status(na1d::march_fused_fwd(o, lse, q, k, v, rpb, valid_len, sq, sk, sv, so, g, dtype, (cudaStream_t)stream));
    return cuda_status(na1d::tc_fused_fwd_seg(o, lse, q, k, v, rpb, valid_len, sq, sk, sv, so, g, dtype, (cudaStream_t)stream));
}

int na1d_fused_backward_strided(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                                const void* v, const float* lse, const float* rpb, const int32_t* valid_len, float* scratch,
                                int64_t scratch_floats, const int64_t* dq_strides, const int64_t* dk_strides,
                                const int64_t* dv_strides, const int64_t* d_o_strides, const int64_t* q_strides,
                                const int64_t* k_strides, const int64_t* v_strides, int64_t N, int64_t heads, int64_t T,
                                int64_t C, int64_t win, int64_t left, int64_t dil, float scale, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(dq); NA1D_REQUIRE_PTR(dk); NA1D_REQUIRE_PTR(dv); NA1D_REQUIRE_PTR(d_o); NA1D_REQUIRE_PTR(q);
    NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v); NA1D_REQUIRE_PTR(lse);
    NA1D_REQUIRE_ALIGNED(dq); NA1D_REQUIRE_ALIGNED(dk); NA1D_REQUIRE_ALIGNED(dv); NA1D_REQUIRE_ALIGNED(d_o);
    NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    if (d_rpb && heads * win * 4 > 48 * 1024) return NA1D_ERR_TOO_LARGE;
    if (scratch_floats < 0 || (scratch == nullptr && scratch_floats != 0)) return NA1D_ERR_NULL_POINTER;
    na1d::Strides s7[7];
    const int64_t* in[7] = {dq_strides, dk_strides, dv_strides, d_o_strides, q_strides, k_strides, v_strides};
    const int64_t batch = N / heads;
    for (int i = 0; i < 7; ++i)
        if (int s = read_strides(in[i], batch, heads, T, C, s7[i])) return s;
    if (!na1d::tc_bwd_seg_supports(g, rpb != nullptr, d_rpb != nullptr)) return NA1D_ERR_UNSUPPORTED;
    if (use_march(g, Pass::strided_backward, d_rpb != nullptr, s7[0], s7[1], s7[2], s7[3], s7[4], s7[5], s7[6]))
        return cuda_status(na1d::march_fused_bwd(dq, dk, dv, d_rpb, d_o, q, k, v, lse, rpb, valid_len, s7[0], s7[1], s7[2], s7[3], s7[4], s7[5],
                                                 s7[6], g, dtype, (cudaStream_t)stream));
    return cuda_status(na1d::tc_fused_bwd_seg(dq, dk, dv, d_rpb, d_o, q, k, v, lse, rpb, valid_len, scratch, (size_t)scratch_floats,
                                              s7[0], s7[1], s7[2], s7[3], s7[4], s7[5], s7[6], g, dtype, (cudaStream_t)stream));
}

int na1d_fused_backward(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                        const void* v, const void* o, const float* lse, const float* rpb, const int32_t* valid_len,
                        float* delta_ws, int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left,
                        int64_t dil, float scale, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(dq); NA1D_REQUIRE_PTR(dk); NA1D_REQUIRE_PTR(dv); NA1D_REQUIRE_PTR(d_o); NA1D_REQUIRE_PTR(q);
    NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v); NA1D_REQUIRE_PTR(o); NA1D_REQUIRE_PTR(lse); NA1D_REQUIRE_PTR(delta_ws);
    NA1D_REQUIRE_ALIGNED(dq); NA1D_REQUIRE_ALIGNED(dk); NA1D_REQUIRE_ALIGNED(dv); NA1D_REQUIRE_ALIGNED(d_o);
    NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v); NA1D_REQUIRE_ALIGNED(o);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    if (d_rpb && heads * win * 4 > 48 * 1024) return NA1D_ERR_TOO_LARGE;
    cudaStream_t st = (cudaStream_t)stream;
    if (use_march(g, Pass::backward, d_rpb != nullptr, na1d::dense_strides(g.H, g.T, g.C))) {
        const na1d::Strides d = na1d::dense_strides(g.H, g.T, g.C);
        return cuda_status(na1d::march_fused_bwd(dq, dk, dv, d_rpb, d_o, q, k, v, lse, rpb, valid_len, d, d, d, d, d, d, d, g, dtype, st));
    }
    const int fam = pick_family(g, 1, rpb != nullptr, d_rpb != nullptr);
    if (fam < 0) return fam;
    if (fam == 1)  // delta is recomputed inside the kernel from P and dP: o is not read; delta_ws (N*T floats) only holds the
                   // per-CTA partial sums of the bias gradient
        return cuda_status(na1d::tc_fused_bwd(dq, dk, dv, d_rpb, d_o, q, k, v, lse, rpb, valid_len, delta_ws,
                                              (size_t)g.N * (size_t)g.T, g, dtype, st));
    if (fam == 2) {
        const na1d::Strides d = na1d::dense_strides(g.H, g.T, g.C);
        return cuda_status(na1d::tc_fused_bwd_seg(dq, dk, dv, d_rpb, d_o, q, k, v, lse, rpb, valid_len, delta_ws,
                                                  (size_t)g.N * (size_t)g.T, d, d, d, d, d, d, d, g, dtype, st));
    }
    if (use_mma(g, dtype == NA1D_FP16, d_rpb != nullptr, true))
        return cuda_status(na1d::mma_fused_bwd(dq, dk, dv, d_rpb, d_o, q, k, v, o, lse, rpb, valid_len, g, dtype, st));
    if (int s = cuda_status(na1d::simt_delta(delta_ws, d_o, o, g.N * g.T, g.C, dtype, st))) return s;
    return cuda_status(na1d::simt_fused_bwd(dq, dk, dv, d_rpb, d_o, q, k, v, lse, delta_ws, rpb, valid_len, g, dtype, st));
}

int64_t na1d_fused_backward_workspace_floats(int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil, int dtype,
                                             int has_bias, int wants_bias_grad) {
    const int route = na1d_fused_kernel_route(N, heads, T, C, win, left, dil, dtype, 1, has_bias, wants_bias_grad);
    const bool rows = (route == 1 || route == 2) && wants_bias_grad && na1d::bias_grad_partial_rows();
    return route == 0 || route < 0 || rows ? N * T : 0;
}
int na1d_zero(void* p, int64_t bytes, void* stream) {
    NA1D_REQUIRE_PTR(p);
    if (bytes < 0) return NA1D_ERR_BAD_SHAPE;
    return cuda_status(cudaMemsetAsync(p, 0, (size_t)bytes, (cudaStream_t)stream));
}

namespace {
int dropout_cfg(float drop_p, uint64_t seed, na1d::DropoutCfg& cfg) {
    if (!(drop_p >= 0.f) || drop_p >= 1.f) return NA1D_ERR_BAD_DROPOUT;
    const double th = (double)drop_p * 4294967296.0;
    cfg.threshold = th >= 4294967295.0 ? 4294967295u : (uint32_t)th;
    cfg.seed = (uint32_t)(seed ^ (seed >> 32));
    cfg.scale = 1.f / (1.f - drop_p);
    return NA1D_OK;
}
}  // namespace

int na1d_dropout_keep_mask(uint8_t* keep_host, int64_t rows, int64_t win, float drop_p, uint64_t seed) {
    NA1D_REQUIRE_PTR(keep_host);
    if (rows <= 0 || win <= 0 || rows > (int64_t)INT_MAX) return NA1D_ERR_BAD_SHAPE;
    na1d::DropoutCfg cfg;
    if (int s = dropout_cfg(drop_p, seed, cfg)) return s;
    for (int64_t r = 0; r < rows; ++r)
        for (int64_t kk = 0; kk < win; ++kk)
            keep_host[r * win + kk] = na1d::drop_hash((uint32_t)r, (uint32_t)kk, cfg.seed) >= cfg.threshold ? 1 : 0;
    return NA1D_OK;
}

int na1d_fused_forward_dropout(void* o, float* lse, const void* q, const void* k, const void* v, const float* rpb,
                               const int32_t* valid_len, int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win,
                               int64_t left, int64_t dil, float scale, float drop_p, uint64_t seed, int dtype, void* stream) {
    if (drop_p == 0.f) return na1d_fused_forward(o, lse, q, k, v, rpb, valid_len, N, heads, T, C, win, left, dil, scale, dtype, stream);
    NA1D_REQUIRE_PTR(o); NA1D_REQUIRE_PTR(q); NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v);
    NA1D_REQUIRE_ALIGNED(o); NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    na1d::DropoutCfg cfg;
    if (int s = dropout_cfg(drop_p, seed, cfg)) return s;
    if (!na1d::tc_fwd_supports(g)) return NA1D_ERR_UNSUPPORTED;
    return cuda_status(na1d::tc_fused_fwd_dropout(o, lse, q, k, v, rpb, valid_len, g, dtype, cfg, (cudaStream_t)stream));
}

int na1d_fused_backward_dropout(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                                const void* v, const float* lse, const float* rpb, const int32_t* valid_len, float* scratch,
                                int64_t scratch_floats, int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left,
                                int64_t dil, float scale, float drop_p, uint64_t seed, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(dq); NA1D_REQUIRE_PTR(dk); NA1D_REQUIRE_PTR(dv); NA1D_REQUIRE_PTR(d_o); NA1D_REQUIRE_PTR(q);
    NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v); NA1D_REQUIRE_PTR(lse);
    NA1D_REQUIRE_ALIGNED(dq); NA1D_REQUIRE_ALIGNED(dk); NA1D_REQUIRE_ALIGNED(dv); NA1D_REQUIRE_ALIGNED(d_o);
    NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    if (d_rpb && heads * win * 4 > 48 * 1024) return NA1D_ERR_TOO_LARGE;
    if (scratch_floats < 0 || (scratch == nullptr && scratch_floats != 0)) return NA1D_ERR_NULL_POINTER;
    na1d::DropoutCfg cfg;
    if (int s = dropout_cfg(drop_p, seed, cfg)) return s;
    if (!na1d::tc_bwd_supports(g, rpb != nullptr, d_rpb != nullptr)) return NA1D_ERR_UNSUPPORTED;
    return cuda_status(na1d::tc_fused_bwd_dropout(dq, dk, dv, d_rpb, d_o, q, k, v, lse, rpb, valid_len, scratch, (size_t)scratch_floats,
                                                  g, dtype, cfg, (cudaStream_t)stream));
}

// ---- row and column kernels of a transformer block (na1d_block.cu)
int na1d_valid_tokens(int32_t* out, const void* padding, int is64, int64_t n_padding, int64_t N, int64_t T, void* stream) {
    NA1D_REQUIRE_PTR(out); NA1D_REQUIRE_PTR(padding);
    if (N <= 0 || N > INT_MAX / 2 || T <= 0 || T > INT_MAX || (n_padding != 1 && n_padding != N)) return NA1D_ERR_BAD_SHAPE;
    return cuda_status(na1d::block_valid_tokens(out, padding, is64 != 0, (int)n_padding, (int)N, (int)T, (cudaStream_t)stream));
}
int64_t na1d_block_scratch_floats(int64_t rows, int64_t D, int64_t F) {
    if (rows <= 0 || D < 0 || F < 0 || rows > INT_MAX / 2 || D > (1 << 20) || F > (1 << 20)) return 0;
    const int64_t cols = 3 * D > 256 ? 3 * D : 256, n = na1d::block_partial_rows(rows) * cols;
    return n > F ? n : F;
}
int na1d_layer_norm_forward(void* y, void* sum, float* mean, float* rstd, const void* x, const void* dx, const float* w,
                            const float* b, int64_t rows, int64_t D, float eps, int dtype, void* stream) {
    if (int s = check_pointers(y, x, w, b)) return s;
    if ((dx == nullptr) != (sum == nullptr) || (mean == nullptr) != (rstd == nullptr)) return NA1D_ERR_NULL_POINTER;
    if (!aligned16(sum) || !aligned16(dx)) return NA1D_ERR_MISALIGNED;
    if (int s = check_block(rows, D, 1024, dtype)) return s;
    return cuda_status(na1d::block_ln_fwd(y, sum, mean, rstd, x, dx, w, b, (int)rows, (int)D, eps, dtype, (cudaStream_t)stream));
}
int na1d_layer_norm_backward(void* dx, float* sums, float* scratch, const void* dy, const void* x, const float* mean,
                             const float* rstd, const float* w, const void* res, int64_t rows, int64_t D, int dtype, void* stream) {
    if (int s = check_pointers(dx, sums, scratch, dy, x, mean, rstd, w)) return s;
    if (!aligned16(res)) return NA1D_ERR_MISALIGNED;
    if (int s = check_block(rows, D, 1024, dtype)) return s;
    return cuda_status(na1d::block_ln_bwd(dx, sums, scratch, dy, x, mean, rstd, w, res, (int)rows, (int)D, dtype, (cudaStream_t)stream));
}
int na1d_layer_norm_backward_rows(void* dx, float* scratch, const void* dy, const void* x, const float* mean, const float* rstd, const float* w,
                                  const void* res, int64_t rows, int64_t D, int dtype, void* stream) {
    if (int s = check_pointers(dx, scratch, dy, x, mean, rstd, w)) return s;
    if (!aligned16(res)) return NA1D_ERR_MISALIGNED;
    if (int s = check_block(rows, D, 1024, dtype)) return s;
    return cuda_status(na1d::block_ln_bwd(dx, nullptr, scratch, dy, x, mean, rstd, w, res, (int)rows, (int)D, dtype, (cudaStream_t)stream));
}
int na1d_layer_norm_sums(float* sums0, float* sums1, const float* scratch0, const float* scratch1, int64_t rows, int64_t D, void* stream) {
    if (int s = check_pointers(sums0, sums1, scratch0, scratch1)) return s;
    if (int s = check_block(rows, D, 1024, NA1D_BF16)) return s;
    float* const sums[2] = {sums0, sums1};
    const float* const part[2] = {scratch0, scratch1};
    return cuda_status(na1d::block_ln_sums(sums, part, (int)rows, (int)D, (cudaStream_t)stream));
}
int na1d_gelu_forward(void* y, const void* x, int64_t n, int dtype, void* stream) {
    if (int s = check_pointers(y, x)) return s;
    if (dtype != NA1D_BF16 && dtype != NA1D_FP16) return NA1D_ERR_BAD_DTYPE;
    if (n <= 0 || n % 8 != 0 || n > (1ll << 40)) return NA1D_ERR_BAD_SHAPE;
    return cuda_status(na1d::block_gelu_fwd(y, x, n, dtype, (cudaStream_t)stream));
}
int na1d_gelu_backward(void* dx, float* sums, float* scratch, const void* dy, const void* x, int64_t rows, int64_t F, int dtype,
                       void* stream) {
    if (int s = check_pointers(dx, sums, scratch, dy, x)) return s;
    if (int s = check_block(rows, F, 1 << 20, dtype)) return s;
    return cuda_status(na1d::block_gelu_bwd(dx, sums, scratch, dy, x, (int)rows, (int)F, dtype, (cudaStream_t)stream));
}
int na1d_column_sums(float* sums, float* scratch, const void* x, int64_t rows, int64_t F, int dtype, void* stream) {
    if (int s = check_pointers(sums, scratch, x)) return s;
    if (int s = check_block(rows, F, 1 << 20, dtype)) return s;
    return cuda_status(na1d::block_column_sums(sums, scratch, x, (int)rows, (int)F, dtype, (cudaStream_t)stream));
}
static int check_gradients(const int64_t* M, const int64_t* N, int count, int64_t rows) {
    NA1D_REQUIRE_PTR(M); NA1D_REQUIRE_PTR(N);
    if (count <= 0 || count > 2) return NA1D_ERR_TOO_LARGE;
    for (int i = 0; i < count; ++i) {
        if (int s = check_block(rows, M[i], 1 << 20, NA1D_BF16)) return s;
        if (int s = check_block(rows, N[i], 1 << 20, NA1D_BF16)) return s;
        if (M[i] * N[i] > (1ll << 37)) return NA1D_ERR_TOO_LARGE;
    }
    return NA1D_OK;
}
int64_t na1d_projection_gradients_scratch(const int64_t* M, const int64_t* N, int count, int64_t rows) {
    return check_gradients(M, N, count, rows) == NA1D_OK ? (int64_t)na1d::wgrad_scratch_floats(M, N, count, rows) : 0;
}
int na1d_projection_gradients(void* const* d_w, void* const* d_b, const void* const* dy, const void* const* x, const int64_t* M, const int64_t* N, int count,
                              int64_t rows, float* scratch, int out32, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(d_w); NA1D_REQUIRE_PTR(d_b); NA1D_REQUIRE_PTR(dy); NA1D_REQUIRE_PTR(x);
    if (dtype != NA1D_BF16 && dtype != NA1D_FP16) return NA1D_ERR_BAD_DTYPE;
    if (int s = check_gradients(M, N, count, rows)) return s;
    if (int s = check_pointers(scratch)) return s;
    for (int i = 0; i < count; ++i)
        if (int s = check_pointers(dy[i], x[i])) return s;
    return cuda_status(na1d::wgrad(d_w, d_b, dy, x, M, N, count, rows, scratch, out32 != 0, dtype, (cudaStream_t)stream));
}
int64_t na1d_mlp_scratch_floats(int64_t rows, int64_t D, int64_t F) {
    if (!na1d::mlp_supports(D, F) || check_block(rows, F, 1 << 20, NA1D_BF16) != NA1D_OK) return -1;
    return (int64_t)na1d::mlp_scratch_floats(rows, F);
}
static int mlp_forward(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const void* b1, const void* w2, const void* b2, bool rounded,
                       float* scratch, int64_t rows, int64_t D, int64_t F, int dtype, void* stream) {
    if (int e = check_pointers(out, s, h, w1, b1, w2, b2)) return e;
    if ((((uintptr_t)f | (uintptr_t)s) & 31) || !aligned16(scratch)) return NA1D_ERR_MISALIGNED;
    if (int e = check_block(rows, F, 1 << 20, dtype)) return e;
    if (!na1d::mlp_supports(D, F) || ld < D || ld % 8 != 0 || ld > (1ll << 40) / rows) return NA1D_ERR_BAD_SHAPE;
    if (!scratch && na1d::mlp_scratch_floats(rows, F) && (f || !rounded)) return NA1D_ERR_NULL_POINTER;
    return cuda_status(na1d::mlp_forward(out, ld, f, s, h, w1, b1, w2, b2, rounded, scratch, rows, F, dtype, (cudaStream_t)stream));
}
int na1d_mlp_forward(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const float* b1, const void* w2, const float* b2, float* scratch,
                     int64_t rows, int64_t D, int64_t F, int dtype, void* stream) {
    return mlp_forward(out, ld, f, s, h, w1, b1, w2, b2, false, scratch, rows, D, F, dtype, stream);
}
int na1d_mlp_forward_rounded(void* out, int64_t ld, void* f, const void* s, const void* h, const void* w1, const void* b1, const void* w2, const void* b2,
                             float* scratch, int64_t rows, int64_t D, int64_t F, int dtype, void* stream) {
    return mlp_forward(out, ld, f, s, h, w1, b1, w2, b2, true, scratch, rows, D, F, dtype, stream);
}
int na1d_mlp_backward(void* dh, void* df, void* g, const void* d, const void* f, const void* w1, const void* w2, float* scratch, int64_t rows, int64_t D, int64_t F,
                      int dtype, void* stream) {
    if (int e = check_pointers(dh, df, g, d, f, w1, w2)) return e;
    if (!aligned16(scratch) || (((uintptr_t)dh | (uintptr_t)df | (uintptr_t)g | (uintptr_t)f) & 31)) return NA1D_ERR_MISALIGNED;
    if (int e = check_block(rows, F, 1 << 20, dtype)) return e;
    if (!na1d::mlp_supports(D, F)) return NA1D_ERR_BAD_SHAPE;
    if (!scratch && na1d::mlp_scratch_floats(rows, F)) return NA1D_ERR_NULL_POINTER;
    return cuda_status(na1d::mlp_backward(dh, df, g, d, f, w1, w2, scratch, rows, F, dtype, (cudaStream_t)stream));
}
int na1d_cast_parameters(void* out, const float* const* src, const int64_t* dst, const int64_t* n, int count, int dtype,
                         void* stream) {
    if (int s = check_pointers(out)) return s;
    NA1D_REQUIRE_PTR(src); NA1D_REQUIRE_PTR(dst); NA1D_REQUIRE_PTR(n);
    if (dtype != NA1D_BF16 && dtype != NA1D_FP16) return NA1D_ERR_BAD_DTYPE;
    if (count <= 0 || count > NA1D_CAST_MAX) return NA1D_ERR_TOO_LARGE;
    for (int i = 0; i < count; ++i) {
        NA1D_REQUIRE_PTR(src[i]);
        if (dst[i] < 0 || dst[i] % 8 != 0 || n[i] <= 0 || n[i] > INT_MAX / 16) return NA1D_ERR_BAD_SHAPE;
    }
    return cuda_status(na1d::block_cast(out, src, dst, n, count, dtype, (cudaStream_t)stream));
}
int na1d_transpose(void* out, const void* in, int64_t N, int64_t C, int64_t T, int to_tokens, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(out); NA1D_REQUIRE_PTR(in);
    NA1D_REQUIRE_ALIGNED(to_tokens ? out : in);
    if (reinterpret_cast<uintptr_t>(to_tokens ? in : out) & 1u) return NA1D_ERR_MISALIGNED;
    if (int s = check_block(T, C, 1 << 20, dtype)) return s;
    if (N <= 0 || N > 65535 || T > (1 << 20)) return NA1D_ERR_BAD_SHAPE;
    return cuda_status(na1d::block_transpose(out, in, (int)N, (int)C, (int)T, to_tokens != 0, dtype, (cudaStream_t)stream));
}
int na1d_permute_heads(void* out, const void* in, int64_t batch, int64_t T, int64_t parts, int64_t heads, int64_t C, int to_dense,
                       void* stream) {
    if (int s = check_pointers(out, in)) return s;
    if (batch <= 0 || T <= 0 || parts <= 0 || heads <= 0 || heads > 65535 || C <= 0 || C % 8 != 0 || C > 4096 || parts > 16 || batch > (1 << 26) ||
        T * C / 8 > INT_MAX / 2 || T > INT_MAX / 8 || batch * parts > INT_MAX)
        return NA1D_ERR_BAD_SHAPE;
    return cuda_status(na1d::block_permute_heads(out, in, (int)batch, (int)T, (int)parts, (int)heads, (int)C, to_dense != 0, (cudaStream_t)stream));
}
static int check_grouped(int64_t C, int64_t groups, int parts, int dtype) {
    if (dtype != NA1D_BF16 && dtype != NA1D_FP16) return NA1D_ERR_BAD_DTYPE;
    if (C <= 0 || C % 8 != 0 || C > 8192 || groups <= 0 || C % groups != 0 || (parts != 1 && parts != 3)) return NA1D_ERR_BAD_SHAPE;
    return NA1D_OK;
}
int na1d_pack_grouped(void* out_w, void* out_b, const void* w, const void* b, int src32, int64_t C, int64_t groups, int parts,
                      int dtype, void* stream) {
    NA1D_REQUIRE_PTR(out_w); NA1D_REQUIRE_PTR(w);
    if ((out_b == nullptr) != (b == nullptr)) return NA1D_ERR_NULL_POINTER;
    if (int s = check_grouped(C, groups, parts, dtype)) return s;
    return cuda_status(na1d::block_pack_grouped(out_w, out_b, w, b, src32 != 0, (int)C, (int)groups, parts, dtype, (cudaStream_t)stream));
}
int na1d_unpack_grouped(void* d_w, void* d_b, const float* dense, const float* sums, int dst32, int64_t C, int64_t groups, int parts,
                        int dtype, void* stream) {
    if (d_w == nullptr && d_b == nullptr) return NA1D_ERR_NULL_POINTER;
    if ((d_w == nullptr) != (dense == nullptr) || (d_b == nullptr) != (sums == nullptr)) return NA1D_ERR_NULL_POINTER;
    if (int s = check_grouped(C, groups, parts, dtype)) return s;
    return cuda_status(na1d::block_unpack_grouped(d_w, d_b, dense, sums, dst32 != 0, (int)C, (int)groups, parts, dtype, (cudaStream_t)stream));
}
int na1d_add_to_rows(void* out, int64_t ld, const void* x, const void* dx, int64_t rows, int64_t D, int dtype, void* stream) {
    if (int s = check_pointers(out, x)) return s;
    if (!aligned16(dx)) return NA1D_ERR_MISALIGNED;
    if (int s = check_block(rows, D, 1 << 20, dtype)) return s;
    if (ld < D || ld % 8 != 0 || rows > (1ll << 40) / ld) return NA1D_ERR_BAD_STRIDE;
    return cuda_status(na1d::block_add_to_rows(out, ld, x, dx, (int)rows, (int)D, dtype, (cudaStream_t)stream));
}
int na1d_stats_pool_forward(float* out, float* stats, const void* logits, const void* x, int64_t ldx, int64_t N, int64_t T,
                            int64_t C, float floor, int dtype, void* stream) {
    if (int s = check_pointers(out, logits, x)) return s;
    if (!aligned16(stats)) return NA1D_ERR_MISALIGNED;
    if (int s = check_block(T, C, 1 << 20, dtype)) return s;
    if (N <= 0 || N > 65535 || T > (1 << 20)) return NA1D_ERR_BAD_SHAPE;
    if (ldx < C || ldx % 8 != 0 || ldx > (1 << 20)) return NA1D_ERR_BAD_STRIDE;
    return cuda_status(na1d::block_pool_fwd(out, stats, logits, x, ldx, (int)N, (int)T, (int)C, floor, dtype, (cudaStream_t)stream));
}
int na1d_stats_pool_backward(void* d_logits, void* dx, const float* d_out, const float* out, const float* stats,
                             const void* logits, const void* x, int64_t N, int64_t T, int64_t C,
                             float floor, int dtype, void* stream) {
    if (int s = check_pointers(d_logits, dx, d_out, out, stats, logits, x)) return s;
    if (int s = check_block(T, C, 1 << 20, dtype)) return s;
    if (N <= 0 || N > 65535 || T > (1 << 20)) return NA1D_ERR_BAD_SHAPE;
    return cuda_status(na1d::block_pool_bwd(d_logits, dx, d_out, out, stats, logits, x, (int)N, (int)T, (int)C, floor, dtype,
                                            (cudaStream_t)stream));
}

int na1d_window_index(int32_t* j_out, uint8_t* in_range, int64_t T, int64_t win, int64_t left, int64_t dil,
                      void* stream) {
    NA1D_REQUIRE_PTR(j_out); NA1D_REQUIRE_PTR(in_range);
    na1d::Geometry g;
    if (int s = check_geometry(1, 1, T, 8, win, left, dil, NA1D_BF16, 1.f, g)) return s;
    return cuda_status(na1d::window_index(j_out, in_range, g.T, g.win, g.left, g.dil, (cudaStream_t)stream));
}

// ---------------------------------------------------------------------------------------------
// Backward pass without a caller-provided workspace (see the header for who needs this and why).
// The delta workspace of the CUDA-core backward lives in this file-scope device array. In host code
// the name below is only a handle for the runtime; the address a kernel can use is obtained once per
// device with cudaGetSymbolAddress and cached.
static __device__ __align__(256) float g_static_delta[NA1D_STATIC_SCRATCH_ROWS];

namespace {
std::mutex g_static_mutex;
float* g_static_delta_addr[64] = {nullptr};

// Device address of g_static_delta on the current device; looked up on the first call per device.
int static_delta_address(float** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e);
    if (dev < 0 || dev >= 64) return NA1D_ERR_TOO_LARGE;
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (g_static_delta_addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_delta);  // needs `dev` current, which it is
        if (e != cudaSuccess) return cuda_status(e);
        if (p == nullptr) return NA1D_ERR_CUDA;
        g_static_delta_addr[dev] = static_cast<float*>(p);
    }
    *out = g_static_delta_addr[dev];
    return NA1D_OK;
}
}  // namespace

int na1d_fused_backward_static(void* dq, void* dk, void* dv, float* d_rpb, const void* d_o, const void* q, const void* k,
                               const void* v, const void* o, const float* lse, const float* rpb, const int32_t* valid_len,
                               int64_t N, int64_t heads, int64_t T, int64_t C, int64_t win, int64_t left, int64_t dil,
                               float scale, int dtype, void* stream) {
    NA1D_REQUIRE_PTR(dq); NA1D_REQUIRE_PTR(dk); NA1D_REQUIRE_PTR(dv); NA1D_REQUIRE_PTR(d_o); NA1D_REQUIRE_PTR(q);
    NA1D_REQUIRE_PTR(k); NA1D_REQUIRE_PTR(v); NA1D_REQUIRE_PTR(o); NA1D_REQUIRE_PTR(lse);
    NA1D_REQUIRE_ALIGNED(dq); NA1D_REQUIRE_ALIGNED(dk); NA1D_REQUIRE_ALIGNED(dv); NA1D_REQUIRE_ALIGNED(d_o);
    NA1D_REQUIRE_ALIGNED(q); NA1D_REQUIRE_ALIGNED(k); NA1D_REQUIRE_ALIGNED(v); NA1D_REQUIRE_ALIGNED(o);
    na1d::Geometry g;
    if (int s = check_geometry(N, heads, T, C, win, left, dil, dtype, scale, g)) return s;
    if (N * T > (int64_t)NA1D_STATIC_SCRATCH_ROWS) return NA1D_ERR_TOO_LARGE;  // the fixed workspace holds N*T floats
    if (d_rpb && heads * win * 4 > 48 * 1024) return NA1D_ERR_TOO_LARGE;
    float* delta = nullptr;
    if (int s = static_delta_address(&delta)) return s;
    cudaStream_t st = (cudaStream_t)stream;
    // The pre-pass writes delta[0 .. N*T) completely before the main kernel reads it, on the same stream:
    // leftovers of earlier calls are never observed.
    if (int s = cuda_status(na1d::simt_delta(delta, d_o, o, g.N * g.T, g.C, dtype, st))) return s;
    return cuda_status(na1d::simt_fused_bwd(dq, dk, dv, d_rpb, d_o, q, k, v, lse, delta, rpb, valid_len, g, dtype, st));
}

}  // extern "C"
