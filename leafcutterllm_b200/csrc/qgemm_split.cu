// Quantised weights (Q6_K, Q4_0, Q8_0; Q4_K and Q5_K: qgemm_whole.cu) times MANY tokens (prompts, batched decode steps) on the 5th-generation tensor
// cores: the dense contraction of the path (Tensor::matmul with m > 1, rust/src/tensor.rs:107-135,
// over weights that the reference dequantises per call, rust/src/model/loader.rs:213-224).
//
//   y[t, r] = sum_k x[t, k] * w[r, k]
//
// Weights stay as raw GGUF blocks in HBM; nothing dequantised is ever written back.  Both factors enter the tensor cores as sums
// of two f16: a weight, times a power of two of its row, is hi + lo with 22 bits and nothing below 2^-24 (every type but Q6_K has at most 21 bits, so
// it is exact unless it is smaller than 2^-17 of its row's largest, and off by 2^-38 of that at most), an activation, times a power of two
// of its token, is hi + lo with 22 bits.  Three of the four products count
// (lo * lo is 2^-22 of the result): per 16 elements of k
//
//   main  += W_hi * X_hi                       one tcgen05.mma with N = 2 * tokens over [X_hi | X_lo] forms the first two,
//   small += W_hi * X_lo,  small += W_lo * X_hi    a second with N = tokens the third.
//
// The tensor cores truncate when they add to an f32 accumulator: the error grows with the number of additions (measured on
// N(0,1) products: 3.5e-7 of the result after 256 elements of k, 1.2e-6 after 1024, 9.6e-6 after 8192; 3 terms into one accumulator
// 1.0e-6 after 256).  So `main`, 2^11 times larger than `small`, is emptied into registers every 128 or 256 elements and those sums are
// rounded to nearest; `small` runs to the end.  What is cut off points toward zero, 2.8e-7 of a sum after 256 elements on average and 1.6e-7 after
// 128, much the same for normal, one-signed and very unequal data, so results are scaled up by about as much: the error's range, one-sided before,
// then lies around zero.  (Sums that need no cutting, of weights with very few bits, are moved by that much instead.)  Error for normal activations, k = 2048: 3.5e-7
// uncorrected, 2.0e-7 over 256, 1.4e-7 over 128 elements (additions in f32 in the matrix-vector kernels: 1.0e-7; their fixed-point form 3.0e-7).
// Emptying every 128 costs 8 % of a 7B prompt, where the tensor pipe is the bound, and 0.7 % of the short prompts of a small Q4_0 / Q8_0 model,
// whose matrix-vector kernels add in f32: those have it.  Up to 32 tokens tensor memory has room for two sums of 128 elements each, at no cost.
//
// One CTA owns 128 weight rows (the M of tcgen05.mma; for gate/up 64 rows of each, so that SiLU(gate) * up happens here) and up to 128
// tokens, and walks k in chunks of 32 elements:
//
//   producers  one thread requests the activation tiles (64 elements x N tokens, hi and lo, 128-byte swizzle), one the raw blocks of a
//              256-element unit (TMA boxes of 32 rows; Q6_K's 210-byte blocks have no 16-byte alignment: two warps copy them by words);
//   unpack     sixteen warps in four groups that take the chunks in turn (two at a time up to 64 tokens): thread r owns row r, turns the chunk's 32
//              elements into f16 integers by byte permutes, hi = d' q and lo = d' q - hi by two f16x2 instructions (exact), and stores both with
//              tcgen05.st as the A operand in TENSOR MEMORY (lane = row, column = two consecutive k).  A group has a tensor-memory
//              stage of its own, so every barrier has one waiter that sees all of its phases;
//   multiply   one warp, whose elected lane issues;
//   drain      the unpack warps again: when a run is through, group g adds tokens 32 g ... 32 g + 31 of `main` to its registers, one
//              run behind its unpacking, so it never waits for the products it feeds.  `main` has two places that runs take in turn.
//
// What bounds it: the tensor pipe, 192 cycles per 128 rows x 128 tokens x 16 elements (128 + 64 for the two instructions; measured
// 128 / 64 / 32 / 13 cycles at N = 256 / 128 / 64 / 16), i.e. a third of the f16 rate, 68 - 71 % active, and with few tokens the groups' way around
// (3,200 cycles a unit).  In qgemm_whole.cu's order (a run's operand behind one barrier) these types are 4 - 7 % slower: their
// sums are read twice as often.
#include <algorithm>
#include <cstdlib>
#include <cuda_fp16.h>
#include "lc_kernels.h"
#include "lc_quant.cuh"
#include "lc_tma.cuh"
#include "lc_qgemm.cuh"

namespace lc {

namespace {

constexpr int kMaxB = 8;         // activation chunks (64 elements) in flight
// Tensor-memory columns: main of even runs [128 - N, 128), small [128, 128 + N), main of odd runs [128 + N, 128 + 2 N): small borders on
// both, so that one instruction covers main and small of either (odd runs have their activations as [lo | hi]).  Behind them
// the A stages, 32 columns each: 16 of W_hi, 16 of W_lo for 32 elements of k; four, or eight where 64 tokens and fewer leave the room.
constexpr uint32_t kColSmall = 128;
__host__ __device__ constexpr uint32_t col_a(int N) { return N <= 64 ? 256u : 384u; }

// `main` over half a unit at a time (see the header): as runs of their own ...
template <uint32_t TYPE, bool WIDE> constexpr bool kHalves = WIDE && (TYPE == LC_TYPE_Q4_0 || TYPE == LC_TYPE_Q8_0);
// ... or, where tensor memory has room, as two sums of one run: then sets of [main of the first half | small | main of the second], for even units
// from column 0 on and for odd units behind it
constexpr int kTwoSums = 32;  // most tokens

// ---- unpacking ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t h2_neg(uint32_t a) { return a ^ 0x80008000u; }
__device__ __forceinline__ uint32_t f16_at(const unsigned char* p) { return *reinterpret_cast<const uint16_t*>(p); }
// words [0, OUT) of the bytes that begin `shift` (even, below 16) bytes into w; `shift` is the same for the whole warp
template <int IN, int OUT>
__device__ __forceinline__ void shift_words(uint32_t (&w)[IN], int shift, uint32_t (&o)[OUT]) {
    if (shift & 8) {
#pragma unroll
        for (int i = 0; i + 2 < IN; i++) w[i] = w[i + 2];
    }
    if (shift & 4) {
#pragma unroll
        for (int i = 0; i + 1 < IN; i++) w[i] = w[i + 1];
    }
    const uint32_t bits = (uint32_t)(shift & 2) * 8u;
#pragma unroll
    for (int i = 0; i < OUT; i++) o[i] = __funnelshift_r(w[i], w[i + 1 < IN ? i + 1 : i], bits);
}
// hi = s q rounded to f16, lo = what that lost: exact where s q has 22 bits and less
__device__ __forceinline__ void split_product(uint32_t s, uint32_t q, uint32_t& hi, uint32_t& lo) {
    hi = h2_mul(s, q);
    lo = h2_fma(s, q, h2_neg(hi));
}
// Elements 32 j ... 32 j + 31 of a row's unit times `up`, as f16 pairs: column c holds elements 2 c and 2 c + 1.  The integer's factor is a power of two
// that brings it to about 1 and the scale's the inverse: the scale, rounded to f16 before the product, then keeps its bits down to 2^-28 of the row's
// largest (with whole integers to 2^-18 in Q4_K, and an error there that counted 945 times).
// Q6_K: d times `up` and the integer's factor
template <uint32_t TYPE>
__device__ __forceinline__ float load_head(const unsigned char* rp, float up) {
    return TYPE == LC_TYPE_Q6_K ? h2f((uint16_t)f16_at(rp + 208)) * up * 32.f : 0.f;
}
template <uint32_t TYPE>
__device__ __forceinline__ void unpack_chunk(const unsigned char* rp, float head, int j, float up, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
    if constexpr (TYPE == LC_TYPE_Q4_0) {  // mod.rs:16-34: 18 bytes: scale, low nibbles = elements 0..15, high = 16..31
        const int at = 18 * j;
        const uint4* p = reinterpret_cast<const uint4*>(rp + (at & ~15));
        const uint4 a = p[0], b = p[1];  // j <= 7: the block ends within two pieces (at most byte 14 + 18 of them)
        uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}, o[5];
        shift_words(w, at & 15, o);
        const uint32_t d = h2_pair(h2f((uint16_t)(o[0] & 0xFFFFu)) * up * 8.f), f = 0x30003000u, m = 0xD808D808u;  // 2^-3; -129 = -1032 / 8
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t v = __funnelshift_r(o[i], o[i + 1], 16);
            const uint32_t bl = v & 0x0F0F0F0Fu, bh = (v >> 4) & 0x0F0F0F0Fu;
            split_product(d, h2_fma(bias_pair(bl, 0), f, m), hi[2 * i], lo[2 * i]);
            split_product(d, h2_fma(bias_pair(bl, 1), f, m), hi[2 * i + 1], lo[2 * i + 1]);
            split_product(d, h2_fma(bias_pair(bh, 0), f, m), hi[8 + 2 * i], lo[8 + 2 * i]);
            split_product(d, h2_fma(bias_pair(bh, 1), f, m), hi[9 + 2 * i], lo[9 + 2 * i]);
        }
    } else if constexpr (TYPE == LC_TYPE_Q8_0) {  // mod.rs:37-51: 34 bytes: scale, 32 signed bytes
        const int at = 34 * j;
        const uint4* p = reinterpret_cast<const uint4*>(rp + (at & ~15));
        const uint4 a = p[0], b = p[1], e = p[2];  // ends at most at byte 14 + 34 of the three pieces
        uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, e.x, e.y, e.z, e.w}, o[9];
        shift_words(w, at & 15, o);
        const uint32_t d = h2_pair(h2f((uint16_t)(o[0] & 0xFFFFu)) * up * 128.f), f = 0x20002000u, m = 0xC880C880u;  // 2^-7; -9 = -(1024 + 128) / 128
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t v = __funnelshift_r(o[i], o[i + 1], 16) ^ 0x80808080u;  // byte + 128
            split_product(d, h2_fma(bias_pair(v, 0), f, m), hi[2 * i], lo[2 * i]);
            split_product(d, h2_fma(bias_pair(v, 1), f, m), hi[2 * i + 1], lo[2 * i + 1]);
        }
    } else {  // Q6_K, mod.rs:145-180; rp: the block's first byte, on an even address
        const int n = j >> 2, quad = j & 3;
        const uint32_t off = (uint32_t)(uintptr_t)rp & 2u, bits = off * 8u;
        const uint32_t* wl = reinterpret_cast<const uint32_t*>(rp - off) + 16 * n + 8 * (quad & 1);
        const uint32_t* wh = reinterpret_cast<const uint32_t*>(rp - off) + 32 + 8 * n;
        uint32_t l[9], h[9];
#pragma unroll
        for (int i = 0; i < 9; i++) { l[i] = wl[i]; h[i] = wh[i]; }
        uint32_t sh[2], sl[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {  // d sc has 18 bits: two f16
            const float s = head * (float)*reinterpret_cast<const int8_t*>(rp + 192 + 8 * n + 2 * quad + i);
            const float top = __half2float(__float2half_rn(s));
            sh[i] = h2_pair(s);
            sl[i] = h2_pair(s - top);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t vl = __funnelshift_r(l[i], l[i + 1], bits), vh = __funnelshift_r(h[i], h[i + 1], bits);
            const uint32_t b = ((vl >> (4 * (quad >> 1))) & 0x0F0F0F0Fu) | (((vh >> (2 * quad)) & 0x03030303u) << 4);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const uint32_t q = h2_fma(bias_pair(b, k), 0x28002800u, 0xD020D020u);  // 2^-5; -33 = -(1024 + 32) / 32
                const int c = 2 * i + k;
                split_product(sh[i >> 2], q, hi[c], lo[c]);
                lo[c] = h2_fma(sl[i >> 2], q, lo[c]);
            }
        }
    }
}
// ---- row scales ----------------------------------------------------------------------------------------------------------
// A power of two per row that brings its weights up to 2^13 ... 2^14 (Q4_K and Q5_K rows whose largest scales belong to blocks of small sc: less): the low
// half of a weight then keeps its bits above 2^-24, f16's smallest step, unless it is 2^-17 of the row's largest.  One warp per row; down[r] = 2^-s.
__global__ void __launch_bounds__(256) row_scale_kernel(uint32_t typ, const unsigned char* __restrict__ w, size_t row_bytes, int n, int k, float* __restrict__ down) {
    pdl_wait();
    pdl_launch_dependents();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= n) return;
    const unsigned char* rp = w + (size_t)row * row_bytes;
    float bound = 0.f;
    const int blocks = typ == LC_TYPE_Q4_0 || typ == LC_TYPE_Q8_0 ? k / 32 : k / 256;
    for (int b = lane; b < blocks; b += 32) {
        float v = 0.f;
        if (typ == LC_TYPE_Q4_K || typ == LC_TYPE_Q5_K) {
            const unsigned char* p = rp + (size_t)b * (typ == LC_TYPE_Q4_K ? 144 : 176);
            const uint4 h = *reinterpret_cast<const uint4*>(p);
            uint32_t sl, sh, ml, mh;
            unpack_scales_k4(h.y, h.z, h.w, &sl, &sh, &ml, &mh);
            const uint32_t s = __vmaxu4(sl, sh), m = __vmaxu4(ml, mh);
            const float sm = (float)max(max(s & 0xFFu, (s >> 8) & 0xFFu), max((s >> 16) & 0xFFu, s >> 24));
            const float mm = (float)max(max(m & 0xFFu, (m >> 8) & 0xFFu), max((m >> 16) & 0xFFu, m >> 24));
            const float d = fabsf(h2f((uint16_t)(h.x & 0xFFFFu))), dm = fabsf(h2f((uint16_t)(h.x >> 16)));
            v = d * fmaxf(sm, 1.f) * (typ == LC_TYPE_Q4_K ? 8.f : 16.f) + dm * fmaxf(mm, 1.f);  // not below either part of a weight,
            v = fmaxf(v, 512.f * d);                                                            // and 2^10 d comes below 2^15
        } else if (typ == LC_TYPE_Q4_0) {
            v = 8.f * fabsf(h2f((uint16_t)f16_at(rp + (size_t)b * 18)));
        } else if (typ == LC_TYPE_Q8_0) {
            v = 128.f * fabsf(h2f((uint16_t)f16_at(rp + (size_t)b * 34)));
        } else {
            const unsigned char* p = rp + (size_t)b * 210;
            int s = 1;
            for (int i = 0; i < 16; i++) s = max(s, abs((int)*reinterpret_cast<const int8_t*>(p + 192 + i)));
            v = 32.f * (float)s * fabsf(h2f((uint16_t)f16_at(p + 208)));
        }
        if (v < INFINITY) bound = fmaxf(bound, v);  // a broken block gives NaN in its row whatever the scale
    }
    bound = warp_max(bound);
    if (lane == 0) {
        int e = 0;
        if (bound > 0.f) (void)frexpf(bound, &e);  // bound = f 2^e, f in [0.5, 1)
        down[row] = ldexpf(1.0f, e - 14);          // e within f16's range times 63 * 31 or 127 * 32
    }
}

// grid = (row tiles, token tiles, shares of k).  tm0 / tm1: raw blocks of the
// matrix (and of `up` for EPI_SILU_MUL), box = one unit x 32 rows.  tmx: the prepared activations [2 halves][t_cap rows][k] f16, box = 64
// elements x N rows of one half.
// WIDE: more than 64 tokens.  Sub-chunk j (32 elements) of a unit then belongs to group j & 3, stage by stage; else group g has the 64 elements
// from 64 g on as one stage, so that the issuer waits half as often for products that are soon over.
template <uint32_t TYPE, bool WIDE>
__global__ void __launch_bounds__(kGemmThreads, 1)
qgemm_split_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tmx,
                   GemmParams p) {
    constexpr int kPitch = RawUnit<TYPE>::pitch;
    constexpr bool kWords = TYPE == LC_TYPE_Q6_K;  // raw units copied by words
    constexpr uint32_t raw_bytes = kPitch * kGemmRows;
    constexpr int kOwn = WIDE ? 32 : 16;           // tokens whose sums a thread keeps
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const bool pair = p.epi == EPI_SILU_MUL;
    const int N = p.N;
    const int RS = p.raw_stages, BS = p.b_stages;
    const uint32_t b_half = (uint32_t)N * 128u;
    const int row0 = blockIdx.x * (pair ? kGemmRows / 2 : kGemmRows), nunits = p.k / kUnitElems;
    int tok0 = blockIdx.y * N, tok_end = p.T;
    const CUtensorMap *map0 = &tm0, *map1 = &tm1;
    ExpertRef ref0{p.w0, p.row_down0}, ref1{p.w1, p.row_down1};
    if (p.offsets) {  // this CTA's expert and its tile of that expert's rows; the grid has room for the last, short tile of each
        pdl_wait();
        int left = blockIdx.y, e = 0, first = __ldg(p.offsets);
        for (; e < p.n_experts; e++) {
            const int end = __ldg(p.offsets + e + 1), tiles = (end - first + N - 1) / N;
            if (left < tiles) { tok0 = first + left * N; tok_end = end; break; }
            left -= tiles;
            first = end;
        }
        if (e == p.n_experts) return;
        map0 = p.maps0 + e; ref0 = p.refs0[e];
        if (pair) { map1 = p.maps1 + e; ref1 = p.refs1[e]; }
    }

    unsigned char* bt = smem;                          // [BS][two tiles of N x 128 B]
    unsigned char* raw = bt + (size_t)BS * 2 * b_half;  // [RS][raw_bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(raw + (size_t)RS * raw_bytes);
    uint64_t* raw_full = bars;                 // [kGemmRaw] producer -> unpack
    uint64_t* raw_empty = raw_full + kGemmRaw;  // [kGemmRaw] unpack (a warp each) -> producer
    uint64_t* b_full = raw_empty + kGemmRaw;    // [kMaxB]   producer -> issuer
    uint64_t* b_empty = b_full + kMaxB;        // [kMaxB]   commit -> producer
    uint64_t* a_full = b_empty + kMaxB;        // [4]       a group's four warps -> issuer
    uint64_t* a_empty = a_full + 4;            // [4]       commit -> that group
    uint64_t* d_full = a_empty + 4;            // [2]       commit -> drain
    uint64_t* d_empty = d_full + 2;            // [2]       drain (a warp each) -> issuer
    uint64_t* wound = d_empty + 2;             // [1]       products in flight when a wait of the issuer ran out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wound + 1);

    const int drains = WIDE ? 4 * ((N + 31) / 32) : 4 * kGemmGroups;  // warps that keep sums
    if (warp == 0 && lane == 0) {
        for (int i = 0; i < kGemmRaw; i++) { mbar_init(&raw_full[i], kWords ? 64 : 1); mbar_init(&raw_empty[i], 4 * kGemmGroups); }
        for (int i = 0; i < kMaxB; i++) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < kGemmGroups; i++) { mbar_init(&a_full[i], 4); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], drains); }
        mbar_init(wound, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    // this CTA's share of k in units; unit v below is u_begin + v
    const int u_begin = (int)((long long)blockIdx.z * nunits / p.ksplit), nu = (int)((long long)(blockIdx.z + 1) * nunits / p.ksplit) - u_begin;
    constexpr bool halves = kHalves<TYPE, WIDE>;
    const bool two = !WIDE && N <= kTwoSums;
    auto run_of = [&](int v, int c) { return halves ? 2 * v + (c >> 1) : v; };  // of `main`, which has two places that the runs take in turn
    auto swapped = [&](int v, int c) { return (halves || two) ? c >> 1 : v & 1; };  // activations lie as [lo | hi]: small lies ahead of main

    // Stages are counted along, never by division: one takes a single thread 100 cycles (a tile of 17 units took 163k with them, 112k without).
    if (warp == 0) {
        // ---------------------------------------------------------------- producer of the activations
        if (lane == 0) {
            pdl_wait();
            int sb = 0, in_flight = 0;
            uint32_t phase = 1;
            for (int v = 0; v < nu && ok; v++) {
                for (int c = 0; c < 4; c++) {
                    if (!mbar_wait(&b_empty[sb], phase)) { ok = false; break; }
                    const int x = (u_begin + v) * kUnitElems + c * 64;
                    unsigned char* const tile = bt + (size_t)sb * 2 * b_half;
                    const int odd = swapped(v, c);
                    mbar_expect_tx(&b_full[sb], 2 * b_half);
                    tma_load_3d(tile + odd * b_half, &tmx, x, tok0, 0, &b_full[sb]);
                    tma_load_3d(tile + (1 - odd) * b_half, &tmx, x, tok0, 1, &b_full[sb]);
                    in_flight = min(in_flight + 1, BS);
                    if (++sb == BS) { sb = 0; phase ^= 1; }
                }
            }
            if (!ok)  // copies in flight land first: the newest of each stage (phase: that of `empty` for stage sb)
                for (int i = 0; i < in_flight; i++) {
                    if (sb == 0) { sb = BS; phase ^= 1; }
                    mbar_wait(&b_full[--sb], phase ^ 1);
                }
        }
    } else if (!kWords && warp == 2) {
        // ---------------------------------------------------------------- producer of the raw units
        // the weights do not depend on the kernel ahead of this one, so this stream starts before the wait for it
        if (lane == 0) {
            if (p.offsets) {
                tmap_acquire(map0);
                if (pair) tmap_acquire(map1);
            }
            int sr = 0, in_flight = 0;
            uint32_t phase = 1;
            for (int v = 0; v < nu; v++) {
                if (!mbar_wait(&raw_empty[sr], phase)) { ok = false; break; }
                mbar_expect_tx(&raw_full[sr], raw_bytes);
#pragma unroll
                for (int b = 0; b < 4; b++)
                    tma_load_2d(raw + (size_t)sr * raw_bytes + b * 32 * kPitch, pair && b >= 2 ? map1 : map0, (u_begin + v) * (kPitch / 4),
                                row0 + (pair ? b & 1 : b) * 32, &raw_full[sr]);
                in_flight = min(in_flight + 1, RS);
                if (++sr == RS) { sr = 0; phase ^= 1; }
            }
            if (!ok)
                for (int i = 0; i < in_flight; i++) {
                    if (sr == 0) { sr = RS; phase ^= 1; }
                    mbar_wait(&raw_full[--sr], phase ^ 1);
                }
        }
    } else if (kWords && (warp == 2 || warp == 3)) {
        // ---------------------------------------------------------------- the same by words: a warp per row, every other row
        int sr = 0;
        uint32_t phase = 1;
        for (int v = 0; v < nu; v++) {
            ok = __all_sync(0xffffffffu, mbar_wait(&raw_empty[sr], phase));
            if (!ok) break;
            uint32_t dst = smem_u32(raw + (size_t)sr * raw_bytes + (warp - 2) * kPitch) + lane * 4;
#pragma unroll 1
            for (int half = 0; half < 2; half++) {  // rows 0 .. 63, 64 .. 127 (pair: of the second matrix)
                const int first = row0 + (pair ? 0 : half * 64) + warp - 2;
                const unsigned char* src = (pair && half ? ref1.w : ref0.w) + (size_t)(u_begin + v) * 210;
                const size_t step = 2 * p.row_bytes;
                const int live = min(32, (p.n - first + 1) / 2);  // rows past the end: any data, dropped at the end
                const unsigned char* row = src + (size_t)first * p.row_bytes;
#pragma unroll 4
                for (int r = 0; r < live; r++, row += step, dst += 2 * kPitch) {
                    const unsigned char* base = reinterpret_cast<const unsigned char*>((uintptr_t)row & ~(uintptr_t)2) + lane * 4;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(base) : "memory");
                    // words 32 ... 52; of the last one only two bytes where the block began on a word
                    const uint32_t take = lane < 20 ? 4u : 2u + ((uint32_t)(uintptr_t)row & 2u);
                    if (lane < 21) asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 128), "l"(base + 128), "r"(take) : "memory");
                }
                dst += (32 - max(live, 0)) * 2 * kPitch;
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&raw_full[sr])) : "memory");
            if (++sr == RS) { sr = 0; phase ^= 1; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 1) {
        // ---------------------------------------------------------------- multiply
        // the whole warp walks the loop and waits (uniform control flow, so that operands live in uniform registers: one lane walking it alone
        // issues a product every 57 cycles at best, and every 200 here: a tile of 17 units took 112k cycles, now 68k), one lane issues
        const bool one = elect_one();
        const uint32_t id1 = idesc_f16(N), id2 = idesc_f16(2 * N), a0 = tmem + col_a(N);
        auto small_of = [&](int v) { return tmem + (two ? (uint32_t)((v & 1) * 3 + 1) * (uint32_t)N : kColSmall); };
        int sb = 0;
        uint32_t b_phase = 0;
        const uint64_t b_first = umma_desc_sw128(smem_u32(bt)), b_step = (2 * b_half) >> 4, b_tile = b_half >> 4;
        uint64_t b_both = b_first;
        for (int v = 0; v < nu && ok; v++) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int run = run_of(v, c);
                const bool begin = halves ? !(c & 1) : c == 0, end = halves ? (c & 1) : c == 3;  // of the run
                const bool anew = begin || (two && c == 2);
                const uint32_t d_small = small_of(v), odd = (uint32_t)swapped(v, c);
                const uint32_t d_both = odd ? d_small : d_small - (uint32_t)N, d_main = odd ? d_small + (uint32_t)N : d_both;
                const uint64_t to_hi = odd ? b_tile : 0, to_lo = odd ? 0 : b_tile;
                if (begin && run >= 2) ok = ok && mbar_wait(&d_empty[run & 1], (run / 2 - 1) & 1);
                ok = ok && mbar_wait(&b_full[sb], b_phase);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t st = WIDE ? (2 * c + h) & 3 : c, a = a0 + (WIDE ? st * 32 : st * 64 + h * 32);
                    if (WIDE || h == 0) ok = ok && mbar_wait(&a_full[st], (uint32_t)(WIDE ? c >> 1 : v & 1));  // the stage's uses: WIDE 2 v and 2 v + 1, else v
                    tc_fence_after();
                    if (one && ok) {
                        const uint64_t bb = b_both + 4 * h;
                        if (anew && h == 0) {  // main
                            umma_f16_ts(d_main, a, bb + to_hi, id1, 0u);
                            umma_f16_ts(d_small, a, bb + to_lo, id1, (uint32_t)(v > (two ? 1 : 0) || c > 0));
                        } else {
                            umma_f16_ts(d_both, a, bb, id2, 1u);
                        }
                        umma_f16_ts(d_small, a + 16, bb + to_hi, id1, 1u);
                        umma_f16_ts(d_both, a + 8, bb + 2, id2, 1u);
                        umma_f16_ts(d_small, a + 24, bb + 2 + to_hi, id1, 1u);
                        if (WIDE || h == 1) umma_commit(&a_empty[st]);
                        if (h == 1) umma_commit(&b_empty[sb]);
                        if (h == 1 && end) umma_commit(&d_full[run & 1]);
                    }
                    __syncwarp();
                }
                b_both += b_step;
                if (++sb == BS) { sb = 0; b_phase ^= 1; b_both = b_first; }
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
            if (one) umma_commit(wound);
            mbar_wait(wound, 0);
        }
    } else if (warp >= kGemmControl) {
        // ---------------------------------------------------------------- unpack and drain, then the epilogue
        const int g = (warp - kGemmControl) >> 2, quarter = warp & 3;
        const int row = quarter * 32 + lane;  // of the tile; also the tensor-memory lane
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16), a_stage = lane_base + col_a(N) + (uint32_t)g * (WIDE ? 32 : 64);
        const int mat = pair ? quarter >> 1 : 0;
        const unsigned char* const weights = mat ? ref1.w : ref0.w;
        const int own = WIDE ? max(0, min(32, N - 32 * g)) : N / 4, tbase = g * (WIDE ? 32 : N / 4);  // this thread's tokens of the tile
        auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); };
        float y[kOwn];
        constexpr uint32_t kNone = ~0u;
        // skip: a bit for each token that keeps what it has; also: a second column, whose sums are added to the first's (up to 32 tokens, eight a thread)
        auto add_columns = [&](uint32_t col, uint32_t also, uint32_t skip) {
            const uint32_t base = lane_base + tbase;
            if constexpr (WIDE) {
#pragma unroll
                for (int t0 = 0; t0 < 32; t0 += 16)
                    if (t0 < own) {
                        uint32_t a[16];
                        tmem_ld16(base + col + t0, a);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int t = 0; t < 16; t++) y[t0 + t] += (skip >> (t0 + t)) & 1u ? 0.f : __uint_as_float(a[t]);
                    }
            } else {
                uint32_t a[16];
#pragma unroll
                for (int t0 = 0; t0 < 16; t0 += 4)
                    if (t0 < own) tmem_ld4(base + col + t0, a + t0);
                if (also != kNone) {
#pragma unroll
                    for (int t0 = 0; t0 < 8; t0 += 4)
                        if (t0 < own) tmem_ld4(base + also + t0, a + 8 + t0);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (also != kNone) {
#pragma unroll
                    for (int t = 0; t < 8; t++) a[t] = __float_as_uint(__uint_as_float(a[t]) + __uint_as_float(a[8 + t]));
                }
#pragma unroll
                for (int t0 = 0; t0 < 16; t0 += 4)
                    if (t0 < own) {
#pragma unroll
                        for (int t = t0; t < t0 + 4; t++) y[t] += (skip >> t) & 1u ? 0.f : __uint_as_float(a[t]);
                    }
            }
        };
        auto drain = [&](int q) {  // run q
            if (own <= 0) return;
            const int place = q & 1;
            ok = wait_all(&d_full[place], (q >> 1) & 1);
            if (!ok) return;
            tc_fence_after();
            // one call: with one in each branch the kernels of up to 64 tokens spilled (seven tokens x [4096 -> 12288] of Q6_K 63.2 us, 59.6 before and 61.4 so)
            add_columns(two ? (uint32_t)(3 * place * N) : place ? kColSmall + (uint32_t)N : kColSmall - (uint32_t)N, two ? (uint32_t)((3 * place + 2) * N) : kNone, 0u);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&d_empty[place]);
        };
        int sr = 0;
        uint32_t raw_phase = 0, a_phase = 1;
        if (p.row_dynamic) pdl_wait();
        const int grow = row0 + (pair ? row & 63 : row);
        const bool live = grow < p.n;
        const unsigned char* const wrow = weights + (size_t)min(grow, p.n - 1) * p.row_bytes;
        const float down = live ? (mat ? ref1.down : ref0.down)[grow] : 1.0f, up = live ? 1.0f / down : 0.0f;
#pragma unroll
        for (int t = 0; t < kOwn; t++) y[t] = 0.f;
        for (int v = 0; v < nu && ok; v++) {
            ok = wait_all(&raw_full[sr], raw_phase);
            if (!ok) break;
            const unsigned char* rp = raw + (size_t)sr * raw_bytes + (size_t)row * kPitch;
            if constexpr (kWords) rp += (uint32_t)(uintptr_t)(wrow + (size_t)(u_begin + v) * 210) & 2u;
            const float head = load_head<TYPE>(rp, up);
#pragma unroll 1
            for (int jj = 0; jj < 2; jj++) {
                if (!WIDE && jj == 0) {  // the products of the stage's use before are complete
                    ok = wait_all(&a_empty[g], a_phase);
                    if (!ok) break;
                    a_phase ^= 1;
                    tc_fence_after();
                }
                uint32_t hi[16], lo[16];
                unpack_chunk<TYPE>(rp, head, WIDE ? g + 4 * jj : 2 * g + jj, up, hi, lo);
                if (jj == 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&raw_empty[sr]);
                }
                if (WIDE) {
                    ok = wait_all(&a_empty[g], a_phase);
                    if (!ok) break;
                    a_phase ^= 1;
                    tc_fence_after();
                }
                tmem_st16(a_stage + (WIDE ? 0 : jj * 32), hi);
                tmem_st16(a_stage + (WIDE ? 0 : jj * 32) + 16, lo);
                if (WIDE || jj == 1) {
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&a_full[g]);
                }
                if (halves && (jj || v > 0)) {  // the run before
                    drain(2 * v + jj - 1);
                    if (!ok) break;
                }
            }
            if (!halves && ok && v > 0) drain(v - 1);
            if (++sr == RS) { sr = 0; raw_phase ^= 1; }
        }
        if (ok) drain(run_of(nu - 1, 3));
        pdl_wait();
        const int t_first = tok0 + tbase, mine = ok ? min(own, tok_end - t_first) : 0;
        // a lane has one token's scale: a load beside each result's store would wait for it
        const float scale = lane < mine ? __ldg(p.tok_scale + t_first + lane) : 0.f;
        // A negative scale: the token holds an infinity or a NaN (xprep_row).  `main` has its results' signs, W_lo * inf in `small` would be NaN
        // wherever W_lo is zero.
        const uint32_t wild = __ballot_sync(0xffffffffu, scale < 0.f);
        if (ok && own > 0) {  // complete: the last unit's d_full followed every product
            const uint32_t col = two ? (uint32_t)N : kColSmall, also = two && nu > 1 ? (uint32_t)(4 * N) : kNone;
            if (wild) add_columns(col, also, wild);
            else add_columns(col, also, 0u);
        }
        // what `main` lost on average (see the header)
        const float back = down * (1.0f + (halves || two ? 0x1p-23f : 0x1p-22f));
        // two multiplications: the product of the powers may leave f32's range where the result does not
#pragma unroll
        for (int t = 0; t < kOwn; t++) y[t] = (y[t] * back) * fabsf(__shfl_sync(0xffffffffu, scale, t));
        store_sums<kOwn>(p, y, bt, pair, mat, g, row, grow, live, t_first, tbase, mine);
    }
    if (!ok && p.error_flag) atomicCAS(p.error_flag, 0, 3);
    tc_fence_before();
    __syncthreads();
    pdl_launch_dependents();  // at the very end: CTAs of the next kernel that move in earlier take SMs from this one's
    if (warp == 1) {
        tc_fence_after();
        tmem_free(tmem, 512);
    }
}

}  // namespace

// ---- host side --------------------------------------------------------------------------------------------------------
bool qgemm_split_weight_ok(const QWeight& w) {
    switch (w.typ) {
        case LC_TYPE_Q4_K: case LC_TYPE_Q5_K: case LC_TYPE_Q4_0: case LC_TYPE_Q8_0: return w.has_tmap && w.k % kUnitElems == 0;
        case LC_TYPE_Q6_K: return w.k % kUnitElems == 0 && (uintptr_t)w.data % 4 == 0;
        default: return false;
    }
}
int32_t launch_row_scales(const QWeight& w, float* down, cudaStream_t s) {
    LC_CUDA(launch_pdl(row_scale_kernel, dim3((unsigned)((w.n + 7) / 8)), dim3(256), 0, s, w.typ, (const unsigned char*)w.data, w.row_bytes, w.n, w.k, down));
    return LC_OK;
}

namespace {
// Cycles of a unit (k = 4096, one wave): 3,200 for five tokens, 3,500 for 64, 4,000 for 96, 4,400 for 128, of which products are 16 * 3 N / 2.
double unit_cycles(int N) { return 2950 + 11.4 * N; }
constexpr double kFixedCycles = 8000;

template <uint32_t TYPE>
int32_t launch_type(const GemvArgs& a, const GemmWorkspace& ws, GemmParams& p, const GemmGroup* group, int* summed_slices, cudaStream_t s) {
    const int nmat = a.epi == EPI_SILU_MUL ? 2 : 1, tiles = (p.n * nmat + kGemmRows - 1) / kGemmRows;
    const int N = gemm_tokens(group ? group->typical : p.T, 16);
    const GemmCut cut = group ? GemmCut{N, 1} : gemm_cut(a, ws, p.T, N, tiles, p.k / kUnitElems, nmat, unit_cycles(N), kFixedCycles);
    // five activation chunks (with few tokens eight) and the raw units that fit
    const size_t raw = (size_t)RawUnit<TYPE>::pitch * kGemmRows, fixed = 1024 + 512, b = (size_t)2 * cut.N * 128;
    p.N = cut.N;
    p.b_stages = cut.N <= 64 ? kMaxB : 5;
    while (p.b_stages > 3 && fixed + p.b_stages * b + 3 * raw > kMaxSmem) p.b_stages--;
    p.raw_stages = std::min<int>(kGemmRaw, (int)((kMaxSmem - fixed - p.b_stages * b) / raw));
    p.ksplit = cut.ks;
    p.partial = cut.ks > 1 ? ws.partial : nullptr;
    *summed_slices = cut.ks > 1 ? cut.ks * nmat : 0;
    const size_t smem = fixed + p.b_stages * b + p.raw_stages * raw;
    auto kern = cut.N <= 64 ? qgemm_split_kernel<TYPE, false> : qgemm_split_kernel<TYPE, true>;
    LC_CUDA(ensure_smem_limit((const void*)kern, smem));
    alignas(64) CUtensorMap tmx;
    const size_t rows = (size_t)ws.t_cap;
    LC_CHECK(make_bf16_tmap_3d(&tmx, ws.xh, (uint64_t)p.k, rows, 2, (uint64_t)p.k, rows * p.k, 64, (uint32_t)cut.N, 1), LC_ERR_CUDA, "qgemm: activation tensor map");
    const CUtensorMap* t0 = (const CUtensorMap*)a.w->tmap;
    const CUtensorMap* t1 = a.w2 ? (const CUtensorMap*)a.w2->tmap : t0;
    const unsigned ttiles = (unsigned)(group ? p.T / cut.N + group->n_experts : (p.T + cut.N - 1) / cut.N);
    LC_CUDA(launch_pdl(kern, dim3((unsigned)tiles, ttiles, (unsigned)cut.ks), dim3(kGemmThreads), smem, s, *t0, *t1, tmx, p));
    return LC_OK;
}
}  // namespace

// The product of prepared activations (ws.xh, ws.sx, ws.tok_scale).  *slices > 0: the shares are in ws.partial, still to be summed.
int32_t launch_qgemm_split(const GemvArgs& a, GemmWorkspace& ws, const GemmGroup* group, int* slices, int* launches, cudaStream_t s) {
    const int n = a.w->n;
    const bool pair = a.epi == EPI_SILU_MUL;
    GemmParams p{};
    p.row_down0 = a.w->row_down;
    p.row_down1 = pair ? a.w2->row_down : p.row_down0;
    if (group) {
        p.maps0 = (const CUtensorMap*)group->maps0; p.maps1 = (const CUtensorMap*)group->maps1;
        p.refs0 = group->refs0; p.refs1 = group->refs1;
        p.offsets = group->offsets; p.row_map = group->row_map; p.n_experts = group->n_experts;
    } else if (!p.row_down0 || !p.row_down1) {  // a matrix that was not laid out for this product when it was bound
        const size_t need = (size_t)n * 2;
        if (ws.row_cap < need) {
            if (ws.row_tmp) cudaFree(ws.row_tmp);
            ws.row_tmp = nullptr; ws.row_cap = 0;
            LC_CUDA(cudaMalloc((void**)&ws.row_tmp, need * sizeof(float)));
            ws.row_cap = need;
        }
        LC_TRY(launch_row_scales(*a.w, ws.row_tmp, s));
        if (pair) LC_TRY(launch_row_scales(*a.w2, ws.row_tmp + n, s));
        p.row_down0 = ws.row_tmp; p.row_down1 = ws.row_tmp + n;
        p.row_dynamic = 1;
        *launches += pair ? 2 : 1;
    }
    p.out = a.out; p.residual = a.residual; p.xh = (const __half*)ws.xh; p.tok_scale = ws.tok_scale;
    p.w0 = (const unsigned char*)a.w->data; p.w1 = pair ? (const unsigned char*)a.w2->data : p.w0;
    p.row_bytes = a.w->row_bytes;
    p.n = n; p.k = a.w->k; p.T = a.m; p.epi = (int)a.epi;
    p.error_flag = gemv_error_flag_dev();
    *launches += 1;
    switch (a.w->typ) {
        case LC_TYPE_Q4_K: case LC_TYPE_Q5_K: return launch_qgemm_whole(a, ws, p, group, slices, s);
        case LC_TYPE_Q4_0: return launch_type<LC_TYPE_Q4_0>(a, ws, p, group, slices, s);
        case LC_TYPE_Q8_0: return launch_type<LC_TYPE_Q8_0>(a, ws, p, group, slices, s);
        default: return launch_type<LC_TYPE_Q6_K>(a, ws, p, group, slices, s);
    }
}

}  // namespace lc
