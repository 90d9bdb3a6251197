// What the two many-token products share (qgemm_split.cu: weights as two f16, qgemm_whole.cu: weights as integers): the CTA's shape, the kernel's arguments,
// raw units, and the way of finished sums into the output.
#pragma once
#include <algorithm>
#include "lc_umma.cuh"

namespace lc {

constexpr int kGemmRows = 128;   // weight rows per CTA = MMA M
constexpr int kGemmTok = 128;    // most tokens per CTA
constexpr int kGemmRaw = 8;      // most raw units in flight
constexpr int kGemmGroups = 4;   // unpack groups of four warps
constexpr int kGemmControl = 4;  // warps ahead of them: activation producer, issuer, raw producer (Q6_K: two)
constexpr int kGemmThreads = 32 * (kGemmControl + 4 * kGemmGroups);

template <uint32_t TYPE> struct RawUnit;  // bytes of a row's unit in shared memory
template <> struct RawUnit<LC_TYPE_Q4_K> { static constexpr int pitch = 144; };
template <> struct RawUnit<LC_TYPE_Q5_K> { static constexpr int pitch = 176; };
template <> struct RawUnit<LC_TYPE_Q4_0> { static constexpr int pitch = 144; };
template <> struct RawUnit<LC_TYPE_Q8_0> { static constexpr int pitch = 272; };
template <> struct RawUnit<LC_TYPE_Q6_K> { static constexpr int pitch = 212; };  // 210 from a word boundary on; an odd number of words: no bank conflicts

struct GemmParams {
    float* out;             // [T, n]
    const float* residual;  // or null
    const __half* xh;       // the activations' high halves, [row][k]
    const float* tok_scale; // [T] power of two that the preparation divided token t by
    const float* row_down0; // [n] power of two that brings row r's weights back (and of the second matrix)
    const float* row_down1;
    const unsigned char *w0, *w1;  // raw blocks
    size_t row_bytes;
    int n, k, T;
    int N;                  // tokens per CTA, a multiple of 16: the box height of the activation tensor maps
    int epi;                // GemvEpilogue; EPI_SILU_MUL: 64 rows of each matrix per CTA
    int raw_stages, b_stages;
    int ksplit;             // CTAs along k per tile (gridDim.z)
    int row_dynamic;        // row_down comes from a kernel ahead of this one in the stream
    float* partial;         // [ksplit][matrices][T][n] f32 for the summing kernel, or null: the CTA holds the whole sum and writes `out`
    // the experts of a mixture layer (see GemmGroup): activation rows in expert order, expert e's from offsets[e] on; null for a plain product
    const CUtensorMap *maps0, *maps1;
    const ExpertRef *refs0, *refs1;
    const int32_t* offsets;
    const int32_t* row_map; // row of `out` that activation row r's result goes to (null: r)
    int n_experts;
    int* error_flag;
};

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// A thread's finished sums: row `grow` of matrix `mat` (row `row` of the tile) for `mine` tokens from t_first on, tokens from tbase on of the CTA's tile.
// stage: the activation stages, which nothing uses any more.  All warps of group g call it.
template <int OWN>
__device__ __forceinline__ void store_sums(const GemmParams& p, float (&y)[OWN], unsigned char* stage, bool pair, int mat, int g, int row, int grow, bool live, int t_first, int tbase,
                                           int mine) {
    const int lane = threadIdx.x & 31;
    if (p.partial) {
        float* dst = p.partial + ((size_t)(blockIdx.z * (pair ? 2 : 1) + mat) * p.T + t_first) * p.n + grow;
#pragma unroll
        for (int t = 0; t < OWN; t++)
            if (live && t < mine) dst[(size_t)t * p.n] = y[t];
    } else if (pair) {
        // rows 0 .. 63 of the tile are gate, 64 .. 127 up: the halves meet in the activation stages, which nothing uses any more
        float* const ex = reinterpret_cast<float*>(stage) + (size_t)tbase * 64 + (row & 63);
        float* const dst = p.out + (size_t)t_first * p.n + grow;
        if (mat == 0) {
#pragma unroll
            for (int t = 0; t < OWN; t++)
                if (t < mine) ex[t * 64] = silu_f(y[t]);
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");  // all of the group's warps come here, whatever their waits gave
        if (mat == 1) {
#pragma unroll
            for (int t = 0; t < OWN; t++)
                if (live && t < mine) dst[(size_t)t * p.n] = __fmul_rn(ex[t * 64], y[t]);
        }
    } else if (p.row_map) {
        const int to = lane < mine ? __ldg(p.row_map + t_first + lane) : 0;
#pragma unroll
        for (int t = 0; t < OWN; t++) {
            const int r = __shfl_sync(0xffffffffu, to, t);
            if (live && t < mine) p.out[(size_t)r * p.n + grow] = y[t];
        }
    } else {
        const size_t o = (size_t)t_first * p.n + grow;
        if (p.epi == EPI_ADD_RESIDUAL) {
            // the loads of sixteen tokens together (`residual` may be `out`): one beside each store takes a trip to L2 for each,
            // 244 us against 197 without a residual for 2,048 tokens x [4096 -> 4096]
#pragma unroll
            for (int t0 = 0; t0 < OWN; t0 += 16) {
                float r[16];
#pragma unroll
                for (int t = 0; t < 16; t++) r[t] = live && t0 + t < mine ? p.residual[o + (size_t)(t0 + t) * p.n] : 0.f;
#pragma unroll
                for (int t = 0; t < 16; t++) y[t0 + t] = __fadd_rn(r[t], y[t0 + t]);
            }
        }
#pragma unroll
        for (int t = 0; t < OWN; t++)
            if (live && t < mine) p.out[o + (size_t)t * p.n] = y[t];
    }
}

// ---- host: how a product is cut ----
struct GemmCut { int N, ks; };  // tokens per CTA, shares of k
// The fewest token tiles, filled evenly.  (More and smaller ones where SMs would be idle: 567 tokens x [2048 -> 2048] in nine tiles 46.7 us, in five 38.8 - 42.)
// step: what N is a multiple of beyond 64 tokens, 16 or, where two CTAs share the tokens, 32.  (Halves of weights with 32, 400 tokens in tiles of 128 instead of 112: Q8_0 x [4096 -> 4096]
// 71.5 us for 69.1, Q6_K 112.2 for 110.4.)
inline int gemm_tokens(int T, int step) {
    const int tt = (T + kGemmTok - 1) / kGemmTok, N = (T + tt - 1) / tt;
    return N <= 64 ? (N + 15) & ~15 : (N + step - 1) / step * step;
}
// Few tiles (a batched decode step, a short prompt): k is cut over several CTAs so that all SMs work, and a second kernel adds the shares in a fixed order.  Cost in cycles: waves
// of (units of a share, measured, + a fixed part: launch, first unit, epilogue), the shares' trip through L2 (at 3,000 bytes per cycle) and the second kernel (4,000); the last two are
// estimates (5.7 TB/s, 2 us).
inline GemmCut gemm_cut(const GemvArgs& a, const GemmWorkspace& ws, int T, int N, int row_tiles, int units, int nmat, double unit_cycles, double fixed_cycles) {
    GemmCut best{N, 1};
    const long tiles = (long)row_tiles * ((T + best.N - 1) / best.N);
    double least = 0;
    for (int c = 1; c <= std::min(8, units); c++) {
        const size_t bytes = (size_t)c * nmat * T * a.w->n * sizeof(float);
        if (c > 1 && (bytes > ws.partial_bytes || !qgemm_sum_ok(a))) break;
        const double cost = (double)((tiles * c + sm_count() - 1) / sm_count()) * ((units + c - 1) / c * unit_cycles + fixed_cycles) + (c > 1 ? 4000 + 2.0 * bytes / 3000 : 0);
        if (c == 1 || cost < least) { least = cost; best.ks = c; }
    }
    return best;
}
// qgemm_whole.cu: Q4_K and Q5_K.  p: filled but for what the cut decides
int32_t launch_qgemm_whole(const GemvArgs& a, const GemmWorkspace& ws, GemmParams& p, const GemmGroup* group, int* summed_slices, cudaStream_t s);

}  // namespace lc
