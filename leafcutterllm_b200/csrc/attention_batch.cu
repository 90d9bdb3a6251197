// Decode attention of a batch: one new token for each of several sequences, over the paged f16 KV cache
// (rust/src/inference/attention.rs:69-113, rust/src/cache/mod.rs:33-77; head_dim 128, 16-token pages).
//
// The unit of work is a (token, kv head, page) item: one 4 KB slab of keys and one of values.  The items of all tokens, in
// (token, kv head, page) order, are cut into one contiguous run per WARP -- worker w of G takes items [w W / G, (w + 1) W / G) -- so the
// warps of the chip stream the same number of bytes each, whatever the contexts' lengths, in a single wave, and no warp waits for another:
//
//   copies   a warp has a ring of its own (three stages of 8 KB) that it fills by TMA three pages ahead, starting BEFORE the kernel looks at
//            its input (cached pages belong to earlier steps); page-table entries are read 32 at a time, one per lane;
//   scores   ldmatrix + mma.sync m16n8k16 against the query heads of the kv group, which are columns of f16 high and low halves
//            (times a power of two per head, so that 22 bits are kept whatever their size);
//   sums     online softmax in log2 units, weights times 2^14 as high and low halves against the transposed values.  The matrix unit truncates when it adds, so it adds up
//            a page and no more (a score: 16 dims); the pages are added in f32, and what those roundings lose is kept beside the low halves' sums;
//   merge    a (token, kv head) that lies within one run is finished by its warp.  Else each of its warps leaves maximum, sum and weighted values in
//            one of its two places (a run has a first and a last shared segment, no more) and takes a ticket; the last one adds all in worker order.
//            At most kMostShares warps share a segment.
//
// Bound: HBM.  The kernel that had a CTA per (token, head, 1,024 keys), f32 FMAs and the rotation's powers, sines and cosines in each CTA took 594 us for
// 2.19 GB (64 sequences of 128 - 4,096 tokens, 32 heads) and 88 us for 67 MB (16 of 1,024, 8 kv heads for 32 heads).
// Now 393 - 404 us (5.4 - 5.6 TB/s of measured 6.4) and 32 us.  Where a step rotates by nothing and there are no kv groups it would gain nothing (attention_batch_applies).
// Runs of whole pieces per CTA would leave the longest sequence's CTA alone at the end.
// The rotation's sines and cosines come from a table that the step's first kernel leaves (`rot`).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include "lc_kernels.h"
#include "lc_attn.cuh"
#include "lc_tma.cuh"

namespace lc {

namespace {

constexpr int kHD = 128;
constexpr int kPage = 16;
constexpr int kKHalf = kPage * 128;          // a TMA box: 16 rows x 64 dims, 128-byte swizzle (chunk j of row r at j ^ (r & 7))
constexpr int kStageBytes = 4 * kKHalf;      // two boxes of keys, two of values
constexpr int kWarps = 8, kStages = 3;        // one CTA per SM (two of four warps, four of two: the same times)
constexpr int kMaxBatch = 1024;              // tokens whose page counts a CTA adds up
constexpr int kStateWords = 4 + kHD;         // maximum, sum, two pad words, weighted values
constexpr int kMostShares = 32;              // a lane for each when they are added
constexpr int kLeastPages = 8;               // of a run: a page costs a warp less than a share costs the warp that adds them (16 sequences of 1,000 and less; 4 and 10: 0 - 2 % slower)
constexpr int kChains = 8;                   // of products in a page's scores
constexpr float kCutOff = 2.7e-8f;           // what a page's weighted values lose on average
constexpr float kWeightScale = 16384.f;      // weights are times 2^14, so that their low halves keep their bits

struct BatchParams {
    AttnParams a;
    int n_tok;
    uint32_t wait_limit;  // of the waits for pages
};

__device__ __forceinline__ uint32_t half_pair(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// the pair's low halves where `low`, else its high ones
__device__ __forceinline__ uint32_t split_pair(float a, float b, bool low) {
    const __half2 h = __floats2half2_rn(a, b);
    return low ? half_pair(a - __low2float(h), b - __high2float(h)) : *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float4 widened(uint2 w) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void rotate_pair(float2& x, float2& y, float4 cs) {  // attention.rs:22-33; cs: cosine and sine of two neighbouring pairs
    const float2 u = x, v = y;
    x.x = __fsub_rn(__fmul_rn(u.x, cs.x), __fmul_rn(v.x, cs.y));
    x.y = __fsub_rn(__fmul_rn(u.y, cs.z), __fmul_rn(v.y, cs.w));
    y.x = __fadd_rn(__fmul_rn(u.x, cs.y), __fmul_rn(v.x, cs.x));
    y.y = __fadd_rn(__fmul_rn(u.y, cs.w), __fmul_rn(v.y, cs.z));
}

// Dims 4 lane ... of a head's vector, turned by its token's row of the table
__device__ __forceinline__ float4 rotated(const float* vec, const float2* row, bool turns, int lane) {
    const int d = 4 * (lane & 15);  // of the pairs' first half; lanes 16 - 31 have the second
    float4 a = __ldcg(reinterpret_cast<const float4*>(vec + d)), b = __ldcg(reinterpret_cast<const float4*>(vec + d + kHD / 2));
    if (turns) {
        const float4* const cs = reinterpret_cast<const float4*>(row + d);
        float2 a0 = make_float2(a.x, a.y), a1 = make_float2(a.z, a.w), b0 = make_float2(b.x, b.y), b1 = make_float2(b.z, b.w);
        rotate_pair(a0, b0, __ldcg(cs));
        rotate_pair(a1, b1, __ldcg(cs + 1));
        a = make_float4(a0.x, a0.y, a1.x, a1.y);
        b = make_float4(b0.x, b0.y, b1.x, b1.y);
    }
    return lane < 16 ? a : b;
}

// A segment of query head `h` once more, keys [first, end), in f32: where a key or a value of the cache is infinite (beyond f16's range), its product with one half of the query or
// of the weight is NaN or of the other sign, and the score's or the sum's is not.  A lane has dims 4 lane ...
struct SegmentState { float most, sum; float4 v; };
__device__ __noinline__ SegmentState plain_segment(const AttnParams& p, int tok, int h, int first, int end, int lane) {
    const KvLayout& kv = p.kv;
    const int kvh = h / (p.n_heads / kv.n_kv);
    const float4 q = rotated(p.q + (size_t)tok * p.q_stride + (size_t)h * kHD, p.rot + (size_t)tok * (kHD / 2), p.tok_rope[tok] != 0, lane);
    const int32_t* const pages = p.page_table + (size_t)p.tok_seq[tok] * p.pages_per_seq;
    const float sc_log2e = 1.4426950408889634f / sqrtf((float)kHD);
    SegmentState s{-INFINITY, 0.f, make_float4(0.f, 0.f, 0.f, 0.f)};
    for (int t = first; t < end; t++) {
        const size_t at = (((size_t)pages[t / kPage] * kv.n_kv + kvh) * kPage + t % kPage) * kHD + 4 * lane;
        const float4 k = widened(*reinterpret_cast<const uint2*>((const __half*)kv.k_pool + at)), v = widened(*reinterpret_cast<const uint2*>((const __half*)kv.v_pool + at));
        const float score = warp_sum(fmaf(q.w, k.w, fmaf(q.z, k.z, fmaf(q.y, k.y, q.x * k.x)))) * sc_log2e;
        if (score > s.most) {
            const float corr = exp2f(s.most - score);
            s.most = score;
            s.sum *= corr;
            s.v = make_float4(s.v.x * corr, s.v.y * corr, s.v.z * corr, s.v.w * corr);
        }
        const float w = score == -INFINITY ? 0.f : exp2f(score - s.most) * kWeightScale;
        s.sum += w;
        s.v = make_float4(fmaf(w, v.x, s.v.x), fmaf(w, v.y, s.v.y), fmaf(w, v.z, s.v.z), fmaf(w, v.w, s.v.w));
    }
    return s;
}

// sum += x; what the addition's rounding lost goes to `low` (of a smaller sum than x: a part of it)
__device__ __forceinline__ void add_keeping(float& sum, float& low, float x) {
    const float s = sum + x;
    low += x - (s - sum);
    sum = s;
}

template <int GSZ>
__global__ void __launch_bounds__(kWarps * 32, 1)
attention_batch_kernel(const __grid_constant__ CUtensorMap ktm, const __grid_constant__ CUtensorMap vtm, const __grid_constant__ BatchParams P) {
    constexpr int NT = (2 * GSZ + 7) / 8;  // n tiles of 8 columns: four heads as (high, low)
    extern __shared__ unsigned char smem_raw[];
    unsigned char* const smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const AttnParams& p = P.a;
    const KvLayout& kv = p.kv;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    unsigned char* const ring = smem + warp * kStages * kStageBytes;
    int* const pre = reinterpret_cast<int*>(smem + kWarps * kStages * kStageBytes);  // [n_tok + 1] pages of the tokens before
    __shared__ __align__(8) uint64_t full_s[kWarps][kStages];
    __shared__ int longest_s;
    uint64_t* const full = full_s[warp];
    if (lane == 0) {
        for (int i = 0; i < kStages; i++) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    pdl_launch_dependents();
    if (!p.positions_settled) pdl_wait();  // the positions themselves may still be in flight
    if (warp == 0) {
        int sum = 0, most = 0;
        if (lane == 0) pre[0] = 0;
        for (int t0 = 0; t0 < P.n_tok; t0 += 32) {
            const int own = t0 + lane < P.n_tok ? p.tok_pos[t0 + lane] / kPage + 1 : 0;
            int v = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            if (t0 + lane < P.n_tok) pre[t0 + lane + 1] = sum + v;
            sum += __shfl_sync(0xffffffffu, v, 31);
            most = max(most, own);
        }
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) longest_s = most;
    }
    __syncthreads();
    const int n_kv = kv.n_kv;
    const long long W = (long long)n_kv * pre[P.n_tok];
    // every run has at least this many pages, so a segment's pages lie in at most kMostShares runs
    const int least = max(kLeastPages, (longest_s + kMostShares - 3) / (kMostShares - 2));
    const long long G = min((long long)gridDim.x * kWarps, max(1ll, W / least));
    const int worker = warp * (int)gridDim.x + (int)blockIdx.x;  // few runs: one per SM
    if (worker >= G) return;
    const long long i_begin = worker * W / G, i_end = (worker + 1) * W / G;
    const int n_items = (int)(i_end - i_begin);

    int tok = 0;  // the token of the first item: the last one with n_kv * pre[tok] <= i_begin
    for (int hi = P.n_tok; hi - tok > 1;) {
        const int mid = (tok + hi) / 2;
        if ((long long)n_kv * pre[mid] <= i_begin) tok = mid; else hi = mid;
    }
    int np = pre[tok + 1] - pre[tok];
    int kvh = (int)(i_begin - (long long)n_kv * pre[tok]) / np;
    int page = (int)(i_begin - (long long)n_kv * pre[tok]) - kvh * np;

    // ---- copies: a place of its own in the run, kStages ahead; ids: page-table entries [id0, id0 + 32) of its sequence, one per lane
    int ptok = tok, pkvh = kvh, ppage = page, pnp = np, id0 = -32, ids = 0;
    auto copy_next = [&](int st) {
        if (ppage - id0 >= 32) {
            id0 = ppage;
            ids = ppage + lane < pnp ? p.page_table[(size_t)p.tok_seq[ptok] * p.pages_per_seq + ppage + lane] : 0;
        }
        const int pg = __shfl_sync(0xffffffffu, ids, ppage - id0);
        if (lane == 0) {
            unsigned char* const dst = ring + st * kStageBytes;
            const int y = (pg * n_kv + pkvh) * kPage;  // first row of the slab in the pool seen as [rows][128]
            mbar_expect_tx(&full[st], kStageBytes);
            tma_load_2d(dst, &ktm, 0, y, &full[st]);
            tma_load_2d(dst + kKHalf, &ktm, 64, y, &full[st]);
            tma_load_2d(dst + 2 * kKHalf, &vtm, 0, y, &full[st]);
            tma_load_2d(dst + 3 * kKHalf, &vtm, 64, y, &full[st]);
        }
        if (++ppage == pnp) {
            ppage = 0;
            if (id0 != 0) id0 = -32;  // the next kv head has the same pages
            if (++pkvh == n_kv) {
                pkvh = 0;
                id0 = -32;
                if (++ptok < P.n_tok) pnp = pre[ptok + 1] - pre[ptok];
            }
        }
    };
    for (int i = 0; i < kStages && i < n_items; i++) copy_next(i);
    if (p.positions_settled) pdl_wait();  // q and this step's k, v come from the projection kernel

    // attention.rs:93-102: softmax(dot / sqrt(head_dim)), in units of log2
    const float sc_log2e = 1.4426950408889634f / sqrtf((float)kHD);
    const int col = lane >> 2, t4 = lane & 3;
    float acc[NT][8][4];         // D[16 dims x 8 columns] per m tile: this lane has dims lane / 4 (+ 8), high and low column of head 4 nt + t4
    float m_own[NT], l_own[NT], l_low[NT], fac[NT];  // of head 4 nt + t4: running maximum, this lane's part of the sum and what its roundings lost, factor from products to scores
    uint32_t qf[NT][8][2];
    bool ok = true, begun = false;
    int first_page = 0, st = 0;
    uint32_t parity = 0;

    auto next_item = [&] {
        if (++page == np) {
            page = 0;
            if (++kvh == n_kv) {
                kvh = 0;
                if (++tok < P.n_tok) np = pre[tok + 1] - pre[tok];
            }
        }
    };
    auto segment_ends = [&](int il) { return page == np - 1 || il + 1 == n_items; };  // the segment, or the run
    auto segment_whole = [&] { return first_page == 0 && page == np - 1; };
    // A ticket of a segment that several warps have a share of; the last one finds the segment's first warp and its number of shares in w_first and shares
    int w_first = 0, shares = 0;
    auto last_of_segment = [&] {
        const long long s_begin = (long long)n_kv * pre[tok] + (long long)kvh * np;
        w_first = (int)(((s_begin + 1) * G - 1) / W);
        shares = (int)(((s_begin + np) * G - 1) / W) - w_first + 1;
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) {
            last = atomicAdd(&p.counters[tok * n_kv + kvh], 1) == shares - 1;
            if (last) p.counters[tok * n_kv + kvh] = 0;  // ready for the next launch
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) __threadfence();
        return last != 0;
    };

    for (int il = 0; il < n_items; il++, next_item()) {
        if (!begun) {
            begun = true;
            first_page = page;
            const int rp = p.tok_rope[tok];
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                // B operand of mma.m16n8k16 (16 dims x 8 columns): column 2h = f16(q of head 4 nt + h), column 2h + 1 = f16 of what that rounding lost
                const int hq = 4 * nt + (col >> 1);
                float2 x[8][2];
                const float* const src = p.q + (size_t)tok * p.q_stride + (size_t)(kvh * GSZ + hq) * kHD + 2 * t4;
#pragma unroll
                for (int kt = 0; kt < 8; kt++)
#pragma unroll
                    for (int r = 0; r < 2; r++)
                        x[kt][r] = hq < GSZ ? __ldcg(reinterpret_cast<const float2*>(src + kt * 16 + 8 * r)) : make_float2(0.f, 0.f);
                if (rp != 0) {
#pragma unroll
                    for (int kt = 0; kt < 4; kt++)
#pragma unroll
                        for (int r = 0; r < 2; r++)
                            rotate_pair(x[kt][r], x[kt + 4][r], __ldcg(reinterpret_cast<const float4*>(p.rot + (size_t)tok * (kHD / 2) + kt * 16 + 2 * t4 + 8 * r)));
                }
                float big = 0.f;
#pragma unroll
                for (int kt = 0; kt < 8; kt++)
#pragma unroll
                    for (int r = 0; r < 2; r++) big = fmaxf(big, fmaxf(fabsf(x[kt][r].x), fabsf(x[kt][r].y)));
                big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
                big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
                // times 2^(14 - its exponent): the head's largest comes to 2^14 ... 2^15 (infinities stay what they are)
                const int ex = max(15, (int)((__float_as_uint(big) >> 23) & 0xFFu));
                const float up = ex == 255 ? 1.f : __uint_as_float((uint32_t)(268 - ex) << 23), down = ex == 255 ? 1.f : __uint_as_float((uint32_t)(ex - 14) << 23);
#pragma unroll
                for (int kt = 0; kt < 8; kt++)
#pragma unroll
                    for (int r = 0; r < 2; r++) qf[nt][kt][r] = split_pair(x[kt][r].x * up, x[kt][r].y * up, col & 1);
                fac[nt] = __shfl_sync(0xffffffffu, down * sc_log2e, 8 * t4);
                m_own[nt] = -INFINITY;
                l_own[nt] = l_low[nt] = 0.f;
#pragma unroll
                for (int mt = 0; mt < 8; mt++) acc[nt][mt][0] = acc[nt][mt][1] = acc[nt][mt][2] = acc[nt][mt][3] = 0.f;
            }
        }
        if (ok && !__all_sync(0xffffffffu, mbar_wait(&full[st], parity, P.wait_limit))) {
            // The copies under way get their time once more to land in this CTA's memory, and no more are requested: a barrier may not be armed again while its phase is open
            ok = false;
            for (int i = 0; i < kStages && il + i < n_items; i++) {
                mbar_wait(&full[st], parity);
                if (++st == kStages) { st = 0; parity ^= 1; }
            }
        }
        __syncwarp();
        if (!ok) {  // the rest of the run is only counted: tickets come out as for the other warps, and the counters are left at zero
            if (segment_ends(il)) {
                if (!segment_whole()) last_of_segment();
                begun = false;
            }
            continue;
        }
        unsigned char* const K_b = ring + st * kStageBytes;
        unsigned char* const V_b = K_b + 2 * kKHalf;
        int nvalid = kPage;
        if (page == np - 1) {
            // this step's token replaces the stale staged row: rotate, round through f16 (cache/mod.rs:35-36), keep in the cache
            const int pos = p.tok_pos[tok], r = pos % kPage, rp = p.tok_rope[tok];
            nvalid = r + 1;
            const float* const kn = p.k_new + (size_t)tok * p.kv_stride + (size_t)kvh * kHD;
            const float4 kr = rotated(kn, p.rot + (size_t)tok * (kHD / 2), rp != 0, lane);
            const float4 vr = __ldcg(reinterpret_cast<const float4*>(p.v_new + (size_t)tok * p.kv_stride + (size_t)kvh * kHD + 4 * lane));
            const uint2 kw = make_uint2(half_pair(kr.x, kr.y), half_pair(kr.z, kr.w)), vw = make_uint2(half_pair(vr.x, vr.y), half_pair(vr.z, vr.w));
            // dims 4 lane ..: box lane / 16, chunk (lane % 16) / 2 (swizzled by the row), 8 bytes into it for odd lanes
            const int off = (lane >> 4) * kKHalf + r * 128 + ((((lane & 15) >> 1) ^ (r & 7)) << 4) + (lane & 1) * 8;
            *reinterpret_cast<uint2*>(K_b + off) = kw;
            *reinterpret_cast<uint2*>(V_b + off) = vw;
            const int pg = p.page_table[(size_t)p.tok_seq[tok] * p.pages_per_seq + page];
            const size_t dst = (((size_t)pg * n_kv + kvh) * kPage + r) * kHD + 4 * lane;
            *reinterpret_cast<uint2*>((__half*)kv.k_pool + dst) = kw;
            *reinterpret_cast<uint2*>((__half*)kv.v_pool + dst) = vw;
            // value rows past this step's position hold whatever the pool held before (Inf, NaN): zero times them is not zero
            for (int ch = lane; ch < (kPage - nvalid) * 16; ch += 32) {
                const int rr = nvalid + (ch >> 4), cj = ch & 15;
                *reinterpret_cast<uint4*>(V_b + (cj >> 3) * kKHalf + rr * 128 + ((cj & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // ahead of the copy that fills the stage next
            __syncwarp();
        }
        {
            float c[NT][kChains][4];
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int i = 0; i < kChains; i++) c[nt][i][0] = c[nt][i][1] = c[nt][i][2] = c[nt][i][3] = 0.f;
            const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8;  // the row this lane addresses for ldmatrix
            const uint32_t lm_row = smem_u32(K_b) + (uint32_t)(lrow * 128);
#pragma unroll
            for (int kt = 0; kt < 8; kt++) {
                const int j = (kt & 3) * 2 + (lane >> 4);  // 16-byte chunk of the 128-byte row, box kt / 4
                uint32_t a[4];
                ldm4(lm_row + (kt >> 2) * kKHalf + ((j ^ (lrow & 7)) << 4), a);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) mma_f16(c[nt][kt & (kChains - 1)], a, qf[nt][kt][0], qf[nt][kt][1]);
            }
            // this lane: keys lane / 4 and lane / 4 + 8 of head 4 nt + t4 (high + low columns)
            float pe[NT][2];
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
#pragma unroll
                for (int o = kChains / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < o; i++)
#pragma unroll
                        for (int r = 0; r < 4; r++) c[nt][i][r] += c[nt][i + o][r];
                const float s0 = col < nvalid ? (c[nt][0][0] + c[nt][0][1]) * fac[nt] : -INFINITY;
                const float s1 = col + 8 < nvalid ? (c[nt][0][2] + c[nt][0][3]) * fac[nt] : -INFINITY;
                float mx = fmaxf(s0, s1);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m_own[nt], mx);
                const float m_sub = m_new == -INFINITY ? 0.f : m_new;  // nothing but scores of minus infinity so far: no weight, not NaN
                const float corr = exp2f(m_own[nt] - m_sub);
                pe[nt][0] = exp2f(s0 - m_sub) * kWeightScale;
                pe[nt][1] = exp2f(s1 - m_sub) * kWeightScale;
                m_own[nt] = m_new;
                if (__any_sync(0xffffffffu, corr != 1.f)) {
                    l_own[nt] *= corr;
                    l_low[nt] *= corr;
#pragma unroll
                    for (int mt = 0; mt < 8; mt++)
#pragma unroll
                        for (int i = 0; i < 4; i++) acc[nt][mt][i] *= corr;
                }
                add_keeping(l_own[nt], l_low[nt], pe[nt][0] + pe[nt][1]);
            }
            // D[16 dims x 8 columns] += V^T[16 dims x 16 keys] . P[16 keys x 8 columns]
            uint32_t pf[NT][2];
            const int hl = col >> 1, src0 = ((2 * t4) << 2) | hl, src1 = ((2 * t4 + 1) << 2) | hl;  // lanes with keys 2 t4, 2 t4 + 1 (and + 8) of head hl
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                float x00 = __shfl_sync(0xffffffffu, pe[nt][0], src0), x01 = __shfl_sync(0xffffffffu, pe[nt][0], src1);
                float x10 = __shfl_sync(0xffffffffu, pe[nt][1], src0), x11 = __shfl_sync(0xffffffffu, pe[nt][1], src1);
                if (4 * nt + hl >= GSZ) x00 = x01 = x10 = x11 = 0.f;
                pf[nt][0] = split_pair(x00, x01, col & 1);
                pf[nt][1] = split_pair(x10, x11, col & 1);
            }
            const int vkey = (lane & 7) + ((lane >> 4) & 1) * 8;  // the key row this lane addresses for the transposing ldmatrix
            const uint32_t lv_row = smem_u32(V_b) + (uint32_t)(vkey * 128);
#pragma unroll
            for (int mt = 0; mt < 8; mt++) {
                const int j = (mt & 3) * 2 + ((lane >> 3) & 1);
                uint32_t a[4];
                ldm4t(lv_row + (mt >> 2) * kKHalf + ((j ^ (vkey & 7)) << 4), a);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    float d[4] = {};
                    mma_f16(d, a, pf[nt][0], pf[nt][1]);
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {
                        acc[nt][mt][i + 1] += d[i + 1];
                        add_keeping(acc[nt][mt][i], acc[nt][mt][i + 1], d[i]);
                    }
                }
            }
        }
        __syncwarp();
        if (il + kStages < n_items) copy_next(st);
        if (++st == kStages) { st = 0; parity ^= 1; }

        if (segment_ends(il)) {
            const bool whole = segment_whole();
            const int slot = first_page > 0 ? 0 : 1;
            float* const mine = p.partial + ((size_t)worker * 2 + slot) * GSZ * kStateWords;
            float* const out = p.out + ((size_t)tok * p.n_heads + (size_t)kvh * GSZ) * kHD;
            uint32_t wild = 0u;  // a bit for each of the group's heads whose sums are infinite or NaN
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                float zero = 0.f * (l_own[nt] + l_low[nt]);
#pragma unroll
                for (int mt = 0; mt < 8; mt++)
#pragma unroll
                    for (int i = 0; i < 4; i++) zero = fmaf(0.f, acc[nt][mt][i], zero);
                const uint32_t lanes = __ballot_sync(0xffffffffu, zero != 0.f);
#pragma unroll
                for (int t = 0; t < 4; t++) wild |= (lanes & (0x11111111u << t)) ? 1u << (4 * nt + t) : 0u;
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                l_own[nt] += l_low[nt];
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) l_own[nt] += __shfl_xor_sync(0xffffffffu, l_own[nt], o);
                const int h = 4 * nt + t4;
                if (h >= GSZ) continue;
                if (!whole && lane < 4) {
                    mine[h * kStateWords] = m_own[nt];
                    mine[h * kStateWords + 1] = l_own[nt];
                }
                float* const dst = whole ? out + h * kHD + col : mine + h * kStateWords + 4 + col;
#pragma unroll
                for (int mt = 0; mt < 8; mt++) {
                    const float v0 = acc[nt][mt][0] + fmaf(acc[nt][mt][0], kCutOff, acc[nt][mt][1]), v1 = acc[nt][mt][2] + fmaf(acc[nt][mt][2], kCutOff, acc[nt][mt][3]);
                    dst[mt * 16] = whole ? v0 / l_own[nt] : v0;
                    dst[mt * 16 + 8] = whole ? v1 / l_own[nt] : v1;
                }
            }
            for (wild &= (1u << GSZ) - 1u; wild; wild &= wild - 1) {
                const int h = __ffs(wild) - 1;
                const SegmentState s = plain_segment(p, tok, kvh * GSZ + h, first_page * kPage, min((page + 1) * kPage, p.tok_pos[tok] + 1), lane);
                __syncwarp();
                if (whole) {
                    reinterpret_cast<float4*>(out + h * kHD)[lane] = make_float4(s.v.x / s.sum, s.v.y / s.sum, s.v.z / s.sum, s.v.w / s.sum);
                } else {
                    if (lane == 0) { mine[h * kStateWords] = s.most; mine[h * kStateWords + 1] = s.sum; }
                    reinterpret_cast<float4*>(mine + h * kStateWords + 4)[lane] = s.v;
                }
            }
            if (!whole && last_of_segment()) {
                const int w = w_first + min(lane, shares - 1);
                const float* const theirs = p.partial + ((size_t)w * 2 + ((long long)n_kv * pre[tok] + (long long)kvh * np < w * W / G ? 0 : 1)) * GSZ * kStateWords;
                const size_t place = (size_t)(theirs - p.partial);
                float e[GSZ], sum[GSZ];  // every load of a round is in flight before the first is used
#pragma unroll
                for (int h = 0; h < GSZ; h++) {
                    e[h] = lane < shares ? __ldcg(theirs + h * kStateWords) : -INFINITY;
                    sum[h] = lane < shares ? __ldcg(theirs + h * kStateWords + 1) : 0.f;
                }
#pragma unroll
                for (int h = 0; h < GSZ; h++) {
                    const float most = warp_max(e[h]);
                    e[h] = e[h] == -INFINITY ? 0.f : exp2f(e[h] - most);
                    sum[h] = warp_sum(sum[h] * e[h]);
                }
                constexpr int kRound = GSZ >= 4 ? 16 / GSZ : 8;
                float4 v[GSZ];
#pragma unroll
                for (int h = 0; h < GSZ; h++) v[h] = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int s0 = 0; s0 < shares; s0 += kRound) {  // in worker order; past the last share: that one again, not added
                    float4 u[kRound][GSZ];
#pragma unroll
                    for (int i = 0; i < kRound; i++) {
                        const size_t at = __shfl_sync(0xffffffffu, (unsigned long long)place, min(s0 + i, shares - 1));
#pragma unroll
                        for (int h = 0; h < GSZ; h++) u[i][h] = __ldcg(reinterpret_cast<const float4*>(p.partial + at + (size_t)h * kStateWords + 4) + lane);
                    }
#pragma unroll
                    for (int i = 0; i < kRound; i++) {
                        if (s0 + i >= shares) break;
#pragma unroll
                        for (int h = 0; h < GSZ; h++) {
                            const float es = __shfl_sync(0xffffffffu, e[h], s0 + i);
                            v[h].x = fmaf(u[i][h].x, es, v[h].x); v[h].y = fmaf(u[i][h].y, es, v[h].y);
                            v[h].z = fmaf(u[i][h].z, es, v[h].z); v[h].w = fmaf(u[i][h].w, es, v[h].w);
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < GSZ; h++)
                    reinterpret_cast<float4*>(out + h * kHD)[lane] = make_float4(v[h].x / sum[h], v[h].y / sum[h], v[h].z / sum[h], v[h].w / sum[h]);
            }
            begun = false;
        }
    }
    if (!ok && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, 1);
}

template <int GSZ>
int32_t launch_batch(const BatchParams& P, cudaStream_t s) {
    constexpr size_t smem = 1024 + (size_t)kWarps * kStages * kStageBytes + (kMaxBatch + 1) * sizeof(int);
    auto kern = attention_batch_kernel<GSZ>;
    LC_CUDA(ensure_smem_limit((const void*)kern, smem));
    CUtensorMap ktm, vtm;
    memcpy(&ktm, P.a.kv.k_tmap, sizeof(ktm));
    memcpy(&vtm, P.a.kv.v_tmap, sizeof(vtm));
    LC_CUDA(launch_pdl(kern, dim3((unsigned)sm_count()), dim3(kWarps * 32), smem, s, ktm, vtm, P));
    return LC_OK;
}

}  // namespace

size_t attention_batch_scratch_bytes(int n_heads, int n_kv, int hd) {
    if (hd != kHD || n_kv <= 0 || n_heads % n_kv != 0) return 0;
    return (size_t)sm_count() * kWarps * 2 * (n_heads / n_kv) * kStateWords * sizeof(float);
}

bool attention_batch_applies(const AttnParams& a, int n_tok, bool turns) {
    const int gsz = a.kv.n_kv > 0 ? a.n_heads / a.kv.n_kv : 0;
    // Where a step turns queries and keys, the kernels of attention.cu were slower for all sizes while they computed the powers, sines and cosines themselves.  Up to four tokens of
    // models without kv groups go to the staged kernel, which has a CTA per 128 keys and less to do ahead of them: 7B shape, 8 layers, us per step staged / here: 3 sequences
    // of 200 768 / 815, of 1,000 870 / 890, of 4,000 1,280 / 1,100.  With kv groups it serves one query head after the other (Mixtral shape, 4 layers, 3 sequences: 1,018 / 965,
    // 1,041 / 990, 1,236 / 1,030).
    // Where nothing turns, the line lies where this kernel is not slower for any context, since a captured step does not know them.  us per layer of a small model, contexts of 60
    // and 1,000, attention.cu / here: up to four sequences, 32 heads on 8, 3 sequences 58.3 / 51.5 and 66.9 / 55.7, but 32 on 16 48.9 / 52.4 and 57.3 / 56.0; more, 32 heads on
    // 8, 6 sequences 68.6 / 75.2 and 80.0 / 79.6, 24 86.3 / 83.1 and 140 / 103, 8 heads on 1, 48 sequences 76.0 / 87.1 and 110 / 94, 128 74.9 / 75.4 and 138 / 88; without
    // groups, 8 heads, 24 sequences 71.2 / 75.5 and 95.8 / 99.6, 128 83.3 / 84.7 and 162 / 162.
    const bool faster = turns ? n_tok > 4 || gsz > 1 : n_tok > 4 ? gsz > 1 && n_tok * a.n_heads >= 1024 : gsz >= 4;
    return n_tok >= 2 && faster && n_tok <= kMaxBatch && a.k_new && a.rot && a.kv.k_tmap && a.kv.v_tmap && a.kv.hd == kHD && !a.kv.kv_f32 && a.kv.page_tokens == kPage &&
           a.n_heads % a.kv.n_kv == 0 && (gsz == 1 || gsz == 2 || gsz == 4 || gsz == 8) && a.q_stride % 4 == 0 && a.kv_stride % 4 == 0;
}

int32_t launch_attention_batch(const AttnParams& a, int n_tok, cudaStream_t s) {
    BatchParams P;
    P.a = a; P.n_tok = n_tok;
    const char* const limit = getenv("LC_ATTN_WAITS");  // read per launch so that a test can make the waits run out: 0, before they look
    P.wait_limit = limit ? (uint32_t)std::clamp(atoi(limit), 0, 1 << 22) : 1u << 22;
    switch (a.n_heads / a.kv.n_kv) {
        case 1: return launch_batch<1>(P, s);
        case 2: return launch_batch<2>(P, s);
        case 4: return launch_batch<4>(P, s);
        default: return launch_batch<8>(P, s);
    }
}

}  // namespace lc
