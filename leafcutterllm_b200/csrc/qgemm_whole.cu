// Q4_K and Q5_K weights times MANY tokens (prompts, experts' rows) on the 5th-generation tensor cores: the dense contraction of the path
// (Tensor::matmul with m > 1, rust/src/tensor.rs:107-135, over weights that the reference dequantises per call, rust/src/model/loader.rs:213-224).
//
//   y[t, r] = sum_k x[t, k] * w[r, k]
//
// Weights stay as raw GGUF blocks in HBM.  An activation, times a power of two of its token, is hi + lo, two f16 with 22 bits together (xprep_kernel).  A weight is
// d * sc * q - dmin * m = d * (sc * (q - c)) + (c * d * sc - dmin * m), c the middle of q's range (8 or 16): within a 256-element unit the first part is d times an
// integer of at most ten bits, which one f16 holds.  So TWO products give the sum over a unit to f32, and the thread that reads it multiplies by d:
//
//   y += d * (I * X_lo + I * X_hi).
//
// The second part joins as more k: two f16 of a sub-block against the sum of the activations over it, 16 values per unit.  (About the middle, because with q
// itself both parts are large and of opposite signs, and the cut-off sums' error with them: 7.0e-7 of the result for normal activations and 7.3e-5 for positive ones at k = 2048.)
//
// The tensor cores truncate when they add to an f32 accumulator.  A unit's low halves are multiplied first, into an empty accumulator, so that they add little to what is cut
// off; the rest, 2.1e-7 of a sum on average, is put back by a factor (error of a result,
// k = 4,096: 1.3e-7 - 2.2e-7; with three products of halves 2.0e-7 - 2.4e-7).
//
// Two CTAs are a pair (cta_group::2): 128 weight rows each (for gate/up 64 rows of each matrix, so that SiLU(gate) * up happens here), up to 128 tokens, whose
// activations lie half in one's and half in the other's shared memory.  That is why there are pairs: alone, a CTA's activations take 64 bytes a cycle of
// shared memory to write and 64 to read, all that it has (2,048 tokens x [11008 -> 4096]: 411 us alone, 381 in pairs).  k goes by in RUNS, one unit each (or the offsets of 16 units):
//
//   producers  in each CTA one thread requests its half of the activation tiles, one the raw blocks of its rows (TMA boxes of 32 rows);
//   groups     sixteen warps of each CTA in four groups.  Thread r of a group owns row r.  When run q - 2 is through, the group adds its part of the tokens' sums to
//              registers and writes its 64 elements of run q as integers into TENSOR MEMORY (lane = row, column = two consecutive k), where q - 2's were;
//   multiply   one warp of the first CTA, whose elected lane issues for both; a commit tells both CTAs' groups that a run is through.
//
// Tensor memory: sums and operand of an even and of an odd run, 4 x 128 columns.
//
// What bounds it: nearly equally the products (2,048 cycles a unit of 128 tokens) and the groups' way around (clock64: wait 140, sums 500, unpacking 1,100, raw unit 200 of 2,500).
// With stages of 32 elements, a barrier for each and a third of each stage's way spent waiting, a unit took 3,600 cycles.  2,048 tokens x [4096 -> 12288]
// 473 -> 442 us, x [11008 -> 4096] 421 -> 381, 512 tokens 123 -> 113 and 107 -> 96, 128 tokens 48 -> 43.
// Tried: the sums read while a unit is unpacked (spills: 25 % slower), registers moved from the control warps (spills), one lane of a warp waiting for all
// (15 % slower), offsets first or last (see below).
#include <algorithm>
#include <cstdlib>
#include <cuda_fp16.h>
#include "lc_kernels.h"
#include "lc_quant.cuh"
#include "lc_tma.cuh"
#include "lc_qgemm.cuh"

namespace lc {

namespace {

constexpr int kMaxB = 8;         // activation stages (two chunks of 64 elements) in flight
// Tensor-memory columns, for even and for odd runs each: 128 of sums (N; up to 64 tokens 2 N, those with low halves of activations first), 128 of the A operand.
constexpr uint32_t kColPlace = 128, kColA = 256;
// What sums lost on average: put back where a run is multiplied anyway, and the rest (8.9e-8, the mean over k = 4,096 ... 14,336 whole and in eight shares) at the end
constexpr float kCutOff = 1.0f + 0x1p-23f, kCutOffAll = 0x1.8p-24f;
// Offsets times positive activations are of one sign, and a run of them loses the more the more units it adds up: 0.6e-7, 1.1e-7, 2.6e-7 and 4.5e-7 for 5, 7, 11 and 16 units;
// with activations of both signs 0.1e-7, 0.5e-7, 1.0e-7 and 1.9e-7.  This much goes into the operand (a factor of the sums moves in steps of 1.2e-7).  Errors of results with
// positive activations, three products of halves / one factor for runs of eight units and more / this: shares of 7 units 5.8e-8 / 1.18e-7 / 3.7e-8, of 11 1.27e-7 / 1.54e-7 / 1.24e-7,
// of 16 3.5e-7 / 3.7e-7 / 2.8e-7; with normal ones 2.0e-7 / 1.6e-7 / 1.6e-7, 2.0e-7 / 1.7e-7 / 1.9e-7, 2.3e-7 / 2.2e-7 / 2.15e-7.
__device__ __forceinline__ float offsets_loss(int units) { return fminf(1.75e-8f * (float)units, 8.8e-8f + 6.5e-9f * (float)min(units, 16)); }

// ---- tcgen05 wrappers -------------------------------------------------------------------------------------------------
// the registers go through it: nothing that uses what was loaded may be moved ahead of the wait
__device__ __forceinline__ void tmem_wait_ld16(uint32_t (&a)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])::"memory");
}
// A wait that lets the warp sleep until the phase is over (or 20 us) instead of asking again and again: the warps that wait here share the schedulers with
// the one that issues the products.  False after about a second.
constexpr uint32_t kNap = 20000, kNaps = 1u << 16;
__device__ __forceinline__ bool nap_wait(uint64_t* bar, uint32_t parity, uint32_t limit = kNaps) {
    const uint32_t addr = smem_u32(bar);
    uint32_t done = 0;
    for (uint32_t it = 0; it < limit && !done; ++it)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done) : "r"(addr), "r"(parity), "r"(kNap) : "memory");
    return done != 0;
}
__device__ __forceinline__ bool phase_over(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return __all_sync(0xffffffffu, done != 0);
}
// ---- pairs: the two CTAs of a cluster multiply as one (cta_group::2): 128 rows of weights each, the activations' rows half in one's and half in the other's shared memory
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// f32 accumulate, f16 x f16, both K-major, M = 256
__host__ __device__ constexpr uint32_t idesc_pair(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (256u >> 4 << 24); }
__device__ __forceinline__ void commit_pair(uint64_t* bar) {  // arrives at this place in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ uint32_t in_first_cta(const void* p) {  // the same place in the CTA that issues
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
    return a;
}
// (released to the cluster it takes 1,000 cycles; what it announces lies in tensor memory and is ordered by the fence ahead of it)
__device__ __forceinline__ void arrive_first(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(in_first_cta(bar)) : "memory"); }
// into this CTA's shared memory, counted by the first CTA's barrier
__device__ __forceinline__ void load_3d_pair(void* dst, const void* tmap, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)), "l"(tmap),
        "r"(x), "r"(y), "r"(z), "r"(in_first_cta(bar))
        : "memory");
}
__device__ __forceinline__ void sync_pair() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---- unpacking ---------------------------------------------------------------------------------------------------------
// Q4_K (mod.rs:66-98): sub-block j has the low (even j) or high nibbles of bytes 32 (j / 2) ... under scale sc[j]; the nibbles are brought up to
// 16 q, and (1024 + 16 q) (sc / 2^14) - 1152 (sc / 2^14) is one fused multiply-add with the exact result sc (q - 8) / 2^10: 1152 = 9 * 2^7 and a scale of
// six bits make a constant that f16 holds, 1032 would not.  Q5_K (mod.rs:101-142): a fifth bit; 8 q and sc / 2^13 likewise.
struct UnitHead { float d; uint32_t sc_lo, sc_hi; };  // d times `up` and 2^10, the eight scales
__device__ __forceinline__ UnitHead load_head(const unsigned char* rp, float up) {
    UnitHead h;
    const uint4 w = *reinterpret_cast<const uint4*>(rp);  // d, dmin, 12 scale bytes
    uint32_t mn_lo, mn_hi;
    unpack_scales_k4(w.y, w.z, w.w, &h.sc_lo, &h.sc_hi, &mn_lo, &mn_hi);
    h.d = h2f((uint16_t)(w.x & 0xFFFFu)) * up * 1024.f;
    return h;
}
// Sub-block 2 g + jj of a row's unit as integers over 2^10, f16 pairs: column c holds elements 2 c and 2 c + 1
template <uint32_t TYPE>
__device__ __forceinline__ void unpack_integers(const unsigned char* rp, const UnitHead& head, int g, int jj, uint32_t (&col)[16]) {
    constexpr bool fifth = TYPE == LC_TYPE_Q5_K;
    const int j = 2 * g + jj;
    const float fs = (float)(((g < 2 ? head.sc_lo : head.sc_hi) >> (8 * (j & 3))) & 0xFFu) * (fifth ? 0x1p-13f : 0x1p-14f);
    const uint32_t sc = h2_pair(fs), bias = h2_pair(-1152.0f * fs);
    const uint4* q = reinterpret_cast<const uint4*>(rp + (fifth ? 48 : 16) + 32 * g);
    // the nibbles to bits 4 - 7 of their bytes, with a fifth bit to 3 - 6 (what the shift brings from other bytes is masked out)
    const uint32_t rot = fifth ? (jj ? 31 : 3) : (jj ? 0 : 4);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint4 v = q[h];
        const uint32_t vv[4] = {v.x, v.y, v.z, v.w};
        uint32_t hb[4] = {0u, 0u, 0u, 0u};
        if constexpr (fifth) {
            const uint4 hq = *reinterpret_cast<const uint4*>(rp + 16 + 16 * h);
            hb[0] = hq.x; hb[1] = hq.y; hb[2] = hq.z; hb[3] = hq.w;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t b = __funnelshift_l(vv[i], vv[i], rot) & (fifth ? 0x78787878u : 0xF0F0F0F0u);
            if constexpr (fifth) b |= (hb[i] << (7 - j)) & 0x80808080u;
            const int c = h * 8 + i * 2;
            col[c] = h2_fma(bias_pair(b, 0), sc, bias);
            col[c + 1] = h2_fma(bias_pair(b, 1), sc, bias);
        }
    }
}
// The offset operand of a unit: p[i] = c * d * sc[i] - dmin * m[i], hi = f16(p) and lo = f16(p - hi).  Columns 0-3: the eight hi
// as pairs (k' = 0..7), columns 4-7: the eight lo (k' = 8..15); the sums tile holds each sub-block sum at k' and k' + 8.  loss: what their sums will lose (offsets_loss).
template <uint32_t TYPE>
__device__ __forceinline__ void unpack_mins(uint4 w, float up, float loss, uint32_t* col) {
    uint32_t sc_lo, sc_hi, mn_lo, mn_hi;
    unpack_scales_k4(w.y, w.z, w.w, &sc_lo, &sc_hi, &mn_lo, &mn_hi);
    float dmin = h2f((uint16_t)(w.x >> 16)) * up, mid = h2f((uint16_t)(w.x & 0xFFFFu)) * up * (TYPE == LC_TYPE_Q5_K ? 16.f : 8.f);
    dmin = fmaf(dmin, loss, dmin);
    mid = fmaf(mid, loss, mid);
#pragma unroll
    for (int j2 = 0; j2 < 4; j2++) {
        __half hi[2], lo[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = 2 * j2 + e;
            const uint32_t sh = 8 * (i & 3), sc = ((i < 4 ? sc_lo : sc_hi) >> sh) & 0xFFu, mn = ((i < 4 ? mn_lo : mn_hi) >> sh) & 0xFFu;
            const float pr = fmaf(mid, (float)sc, -dmin * (float)mn);  // both products are exact, so this rounds once
            hi[e] = __float2half_rn(pr);
            lo[e] = __float2half_rn(pr - __half2float(hi[e]));
        }
        const __half2 a = __halves2half2(hi[0], hi[1]), b = __halves2half2(lo[0], lo[1]);
        col[j2] = *reinterpret_cast<const uint32_t*>(&a);
        col[4 + j2] = *reinterpret_cast<const uint32_t*>(&b);
    }
}

// What a token's elements [first, first + count) that are infinite or NaN give with a row
__device__ __noinline__ float wild_sum(uint32_t typ, const unsigned char* row, const __half* x, int first, int count) {
    float s = 0.f;
    for (int i = first; i < first + count; i += 8) {
        const uint4 x8 = __ldg(reinterpret_cast<const uint4*>(x + i));
        const uint32_t w[4] = {x8.x, x8.y, x8.z, x8.w};
        for (int e = 0; e < 8; e++) {
            const uint32_t h = (w[e >> 1] >> (16 * (e & 1))) & 0xFFFFu;
            if ((h & 0x7C00u) == 0x7C00u) s += dequant_elem(typ, row, (size_t)i + e) * h2f((uint16_t)h);
        }
    }
    return s;
}

// grid = (row tiles, token tiles, shares of k).  tm0 / tm1: raw blocks of the
// matrix (and of `up` for EPI_SILU_MUL), box = one unit x 32 rows.  tmx: the prepared activations [2 halves][t_cap rows][k] f16, box = 64
// elements x N rows of one half; tms: the sub-block sums [2][t_cap rows][k / 16], the same box.
// WIDE: more than 64 tokens.
template <uint32_t TYPE, bool WIDE>
__global__ void __launch_bounds__(kGemmThreads, 1)
qgemm_whole_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tmx,
                  const __grid_constant__ CUtensorMap tms, GemmParams p) {
    constexpr int kPitch = RawUnit<TYPE>::pitch;
    constexpr uint32_t raw_bytes = kPitch * kGemmRows;
    constexpr int kOwn = WIDE ? 32 : 16;           // tokens whose sums a thread keeps
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const bool pair = p.epi == EPI_SILU_MUL;
    const int N = p.N;
    const int RS = p.raw_stages, BS = p.b_stages;
    // a CTA's stage has two chunks of 64 elements: WIDE, one half (high or low) of its half of the N tokens; else its half, low in the first CTA, of all N tokens
    const uint32_t b_stage = (uint32_t)N * (WIDE ? 128u : 256u);
    const int rank = (int)(blockIdx.x & 1);  // in the pair
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

    unsigned char* bt = smem;                        // [BS][b_stage]
    unsigned char* raw = bt + (size_t)BS * b_stage;  // [RS][raw_bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(raw + (size_t)RS * raw_bytes);
    uint64_t* raw_full = bars;                 // [kGemmRaw] producer -> unpack
    uint64_t* raw_empty = raw_full + kGemmRaw;  // [kGemmRaw] unpack (a warp each) -> producer
    uint64_t* b_full = raw_empty + kGemmRaw;    // [kMaxB]   producer -> issuer
    uint64_t* b_empty = b_full + kMaxB;        // [kMaxB]   commit -> producer
    uint64_t* a_full = b_empty + kMaxB;        // [2]       groups (a warp each) -> issuer, of even and odd runs: the operand is there, the sums of two runs before are read
    uint64_t* d_full = a_full + 2;             // [2]       commit -> groups: a run's products are through
    uint64_t* wound = d_full + 2;              // [1]       products in flight when a wait of the issuer ran out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wound + 1);

    if (warp == 0 && lane == 0) {
        for (int i = 0; i < kGemmRaw; i++) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4 * kGemmGroups); }
        for (int i = 0; i < kMaxB; i++) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&a_full[i], 2 * 4 * kGemmGroups); mbar_init(&d_full[i], 1); }
        mbar_init(wound, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    sync_pair();
    tc_fence_after();
    constexpr uint32_t tmem = 0;  // of all 512 columns, the first: a constant, so that addresses need no registers
    bool ok = *tmem_slot == tmem;

    // this CTA's share of k in units; unit v below is u_begin + v
    const int u_begin = (int)((long long)blockIdx.z * nunits / p.ksplit);
    const int nu = (int)((long long)(blockIdx.z + 1) * nunits / p.ksplit) - u_begin;
    // chunks of sub-block sums, four units each, in n_off runs of up to four chunks ahead of the last unit: the rows' headers have come meanwhile (at the start the products wait
    // for them, 7,000 cycles of a tile of 17 units; at the end the tile does, 4,000), and hardly any additions are made at the offsets' size, which may be well above the result's
    const int sum_chunks = (nu + 3) / 4, n_off = (sum_chunks + 3) / 4, off_at = nu - 1;
    const int nq = n_off + nu;
    auto is_unit = [&](int q) { return q < off_at || q >= off_at + n_off; };
    auto chunks_of = [&](int q) { return is_unit(q) ? 4 : min(4, sum_chunks - 4 * (q - off_at)); };

    // Stages are counted along, never by division: one takes a single thread 100 cycles (a tile of 17 units took 163k with them, 112k without).
    if (warp == 0) {
        // ---------------------------------------------------------------- producer of the activations
        if (lane == 0) {
            pdl_wait();
            int sb = 0, in_flight = 0;
            uint32_t phase = 1;
            for (int q = 0; q < nq && ok; q++) {
                const int nc = chunks_of(q);
                const CUtensorMap* const m = is_unit(q) ? &tmx : &tms;
                const int x0 = is_unit(q) ? (u_begin + (q < off_at ? q : q - n_off)) * kUnitElems : (u_begin + 16 * (q - off_at)) * 16;
                const int half_nc = (nc + 1) / 2;
                for (int i = 0; i < (WIDE ? 2 * half_nc : half_nc); i++) {  // WIDE: the low halves of the run's chunks, then the high ones; else both of a chunk
                    if (!nap_wait(&b_empty[sb], phase)) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(&b_full[sb], 2 * b_stage);
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        unsigned char* const tile = bt + (size_t)sb * b_stage + e * (b_stage / 2);
                        const int c = 2 * (WIDE && i >= half_nc ? i - half_nc : i) + e;
                        if constexpr (WIDE) load_3d_pair(tile, m, x0 + c * 64, tok0 + rank * (N / 2), i >= half_nc ? 0 : 1, &b_full[sb]);
                        else load_3d_pair(tile, m, x0 + c * 64, tok0, 1 - rank, &b_full[sb]);
                    }
                    in_flight = min(in_flight + 1, BS);
                    if (++sb == BS) { sb = 0; phase ^= 1; }
                }
            }
            if (!ok && rank == 0)  // copies in flight land first: the newest of each stage (phase: that of `empty` for stage sb)
                for (int i = 0; i < in_flight; i++) {
                    if (sb == 0) { sb = BS; phase ^= 1; }
                    nap_wait(&b_full[--sb], phase ^ 1);
                }
        }
    } else if (warp == 2) {
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
                if (!nap_wait(&raw_empty[sr], phase)) { ok = false; break; }
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
                    nap_wait(&raw_full[--sr], phase ^ 1);
                }
        }
    } else if (warp == 1 && rank == 0) {
        // ---------------------------------------------------------------- multiply
        // The whole warp walks the loop and waits, one lane issues.  Nothing here may depend on what a wait gave but the last check: the operands' addresses then are
        // the same for all lanes in the compiler's eyes too and live in uniform registers.  When a wait runs out the loop goes on over whatever
        // lies there, with waits that no longer wait.
        // A wait costs 140 cycles here though its phase is long over (clock64; shared memory is busy with both sides of the activations' way), as much as two products
        // of 128 tokens take.  So a stage is two chunks, a run's A operand one barrier, and what the next run needs is asked for ahead of this run's
        // last stage: with a barrier per chunk and group a unit took 3,200 cycles for 2,048 of products.
        const bool one = elect_one();
        const uint32_t id1 = idesc_pair(N), id2 = idesc_pair(2 * N);
        uint32_t limit = kNaps;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (!nap_wait(bar, parity, limit)) { limit = 1; ok = false; }
        };
        const uint64_t b_first = umma_desc_sw128(smem_u32(bt));
        const uint32_t b_step = b_stage >> 4, b_chunk = b_step / 2;
        int sb = 0;
        uint32_t b_phase = 0;
        uint64_t b_at = b_first;
        auto next_b = [&] {
            b_at += b_step;
            if (++sb == BS) { sb = 0; b_phase ^= 1; b_at = b_first; }
        };
        auto may_begin = [&](int q) { return phase_over(&a_full[q & 1], ((uint32_t)q >> 1) & 1u); };
        bool begun = false;
#pragma unroll 1
        for (int q = 0; q < nq; q++) {
            const uint32_t place = (uint32_t)q & 1u, par = ((uint32_t)q >> 1) & 1u, d = place * kColPlace, a0 = kColA + place * kColPlace;
            const int nc = chunks_of(q);
            if (!begun) wait(&a_full[place], par);
            if constexpr (WIDE) {
                // the products with the low halves of all chunks, then those with the high halves
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int c0 = 2 * (i & 1);
                    if (c0 < nc) {
                        if (i == 3 || (i == 2 && nc <= 2)) begun = q + 1 < nq && may_begin(q + 1);
                        wait(&b_full[sb], b_phase);
                        tc_fence_after();
                        if (one) {
#pragma unroll
                            for (int j = 0; j < 8; j++)
                                if (j < 4 || c0 + 1 < nc)
                                    mma_pair(d, a0 + (c0 + (j >> 2)) * 32 + (j & 3) * 8, b_at + (j >> 2) * b_chunk + 2 * (j & 3), id1, (uint32_t)(i + j > 0));
                            commit_pair(&b_empty[sb]);
                        }
                        __syncwarp();
                        next_b();
                    }
                }
            } else {
                // columns [low halves | high halves]: one product of twice the tokens
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int c0 = 2 * i;
                    if (c0 < nc) {
                        if (c0 + 2 >= nc) begun = q + 1 < nq && may_begin(q + 1);
                        wait(&b_full[sb], b_phase);
                        tc_fence_after();
                        if (one) {
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                if (j >= 4 && c0 + 1 >= nc) continue;
                                mma_pair(d, a0 + (c0 + (j >> 2)) * 32 + (j & 3) * 8, b_at + (j >> 2) * b_chunk + 2 * (j & 3), id2, (uint32_t)(i + j > 0));
                            }
                            commit_pair(&b_empty[sb]);
                        }
                        __syncwarp();
                        next_b();
                    }
                }
            }
            if (one) commit_pair(&d_full[place]);
            __syncwarp();
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
            if (one) commit_pair(wound);
            nap_wait(wound, 0);
        }
    } else if (warp >= kGemmControl) {
        // ---------------------------------------------------------------- unpack and drain, then the epilogue
        const int g = (warp - kGemmControl) >> 2, quarter = warp & 3;
        const int row = quarter * 32 + lane;  // of the tile; also the tensor-memory lane
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16), a_own = lane_base + kColA + (uint32_t)g * 32u;
        const int mat = pair ? quarter >> 1 : 0;
        const unsigned char* const weights = mat ? ref1.w : ref0.w;
        const int own = WIDE ? max(0, min(32, N - 32 * g)) : N / 4, tbase = g * (WIDE ? 32 : N / 4);  // this thread's tokens of the tile
        auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, nap_wait(bar, parity)); };  // one lane alone asking: 15 % slower
        float y[kOwn];
        // run q's products are through: its sums may be read and its operand's place be filled
        auto wait_products = [&](int q) {
            ok = wait_all(&d_full[q & 1], ((uint32_t)q >> 1) & 1u);
            tc_fence_after();
        };
        auto drain = [&](int q, float times) {  // its sums times `times` are added to y
            wait_products(q);
            if (!ok) return;
            const uint32_t base = lane_base + ((uint32_t)q & 1u) * kColPlace + tbase;
#pragma unroll
            for (int part = 0; part < 2; part++) {  // WIDE: sixteen tokens each, else the sums with high and with low halves
                uint32_t a[16];
                if constexpr (WIDE) {
                    if (16 * part >= own) break;
                    tmem_ld16(base + 16 * part, a);
                    tmem_wait_ld16(a);
#pragma unroll
                    for (int t = 0; t < 16; t++) y[16 * part + t] = fmaf(times, __uint_as_float(a[t]), y[16 * part + t]);
                } else {
#pragma unroll
                    for (int t0 = 0; t0 < 16; t0 += 4)
                        if (t0 < own) tmem_ld4(base + (1 - part) * N + t0, a + t0);
                    tmem_wait_ld16(a);
#pragma unroll
                    for (int t0 = 0; t0 < 16; t0 += 4)
                        if (t0 < own) {
#pragma unroll
                            for (int t = t0; t < t0 + 4; t++) y[t] = fmaf(times, __uint_as_float(a[t]), y[t]);
                        }
                }
            }
        };
        auto operand_ready = [&](int q) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_first(&a_full[q & 1]);
        };
        int sr = 0;
        uint32_t raw_phase = 0;
        if (p.row_dynamic) pdl_wait();
        const int grow = row0 + (pair ? row & 63 : row);
        const bool live = grow < p.n;
        const unsigned char* const wrow = weights + (size_t)min(grow, p.n - 1) * p.row_bytes;
        const float down = live ? (mat ? ref1.down : ref0.down)[grow] : 1.0f, up = live ? 1.0f / down : 0.0f;
#pragma unroll
        for (int t = 0; t < kOwn; t++) y[t] = 0.f;
        float d1 = 1.0f, d2 = 1.0f;  // what the sums of the last run and the one before are still to be multiplied by
        if (live)
            for (int u = g * 4; u < nu; u += 16)
                for (int e = u; e < min(u + 4, nu); e++) asm volatile("prefetch.global.L2 [%0];" ::"l"(wrow + (size_t)(u_begin + e) * kPitch));
        // the offset operand of run q: sixteen values of each of four units per chunk, from their headers in global memory
        auto offsets = [&](int q) {
            if (q >= 2) drain(q - 2, d2);
            if (!ok) return;
            d2 = d1;
            d1 = 1.0f;
            const float loss = offsets_loss(nu - 16 * (q - off_at));
            // two units' headers at a time: all four take registers that the sums then spill for (777 tokens x [4096 -> 4096] 128 us, so 123)
            const int u = u_begin + ((q - off_at) * 4 + g) * 4;
#pragma unroll
            for (int jj = 0; jj < 2; jj++) {
                uint4 hd[2];
#pragma unroll
                for (int e = 0; e < 2; e++) hd[e] = live && u + 2 * jj + e < u_begin + nu ? __ldg(reinterpret_cast<const uint4*>(wrow + (size_t)(u + 2 * jj + e) * kPitch)) : make_uint4(0u, 0u, 0u, 0u);
                uint32_t col[16];
                unpack_mins<TYPE>(hd[0], up, loss, col);
                unpack_mins<TYPE>(hd[1], up, loss, col + 8);
                tmem_st16(a_own + (q & 1) * kColPlace + jj * 16, col);
            }
            operand_ready(q);
        };
        for (int v = 0; v < nu && ok; v++) {
            ok = wait_all(&raw_full[sr], raw_phase);
            if (!ok) break;
            const unsigned char* rp = raw + (size_t)sr * raw_bytes + (size_t)row * kPitch;
            const UnitHead head = load_head(rp, up);
            if (v == off_at) for (int q = off_at; q < off_at + n_off && ok; q++) offsets(q);
            if (!ok) break;
            const int q = v < off_at ? v : n_off + v;
            if (q >= 2) drain(q - 2, d2);
            if (!ok) break;
            uint32_t col[16];
#pragma unroll
            for (int jj = 0; jj < 2; jj++) {
                unpack_integers<TYPE>(rp, head, g, jj, col);
                tmem_st16(a_own + (q & 1) * kColPlace + jj * 16, col);
            }
            d2 = d1;
            d1 = head.d * kCutOff;
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[sr]);
            operand_ready(q);
            if (++sr == RS) { sr = 0; raw_phase ^= 1; }
        }
        for (int q = max(0, nq - 2); q < nq && ok; q++) drain(q, q == nq - 1 ? d1 : d2);
        pdl_wait();
        const int t_first = tok0 + tbase, mine = ok ? min(own, tok_end - t_first) : 0;
        // a lane has one token's scale: a load beside each result's store would wait for it
        const float scale = lane < mine ? __ldg(p.tok_scale + t_first + lane) : 0.f;
        // A negative scale: the token holds an infinity or a NaN (xprep_row), and what the products give is NaN wherever an integer or a low half is
        // zero.  Its result is what those elements alone give.
        for (uint32_t wild = __ballot_sync(0xffffffffu, scale < 0.f); wild; wild &= wild - 1) {
            const int t = __ffs(wild) - 1;
            const float s = wild_sum(TYPE, wrow, p.xh + (size_t)(t_first + t) * p.k, u_begin * kUnitElems, nu * kUnitElems);
#pragma unroll
            for (int j = 0; j < kOwn; j++)
                if (j == t) y[j] = s;
        }
        // two multiplications: the product of the powers may leave f32's range where the result does not
#pragma unroll
        for (int t = 0; t < kOwn; t++) y[t] = (fmaf(y[t], kCutOffAll, y[t]) * down) * fabsf(__shfl_sync(0xffffffffu, scale, t));
        store_sums<kOwn>(p, y, bt, pair, mat, g, row, grow, live, t_first, tbase, mine);
    }
    if (!ok && p.error_flag) atomicCAS(p.error_flag, 0, 3);
    tc_fence_before();
    sync_pair();  // a pair ends together: products and arrivals reach into the other CTA
    pdl_launch_dependents();  // at the very end: CTAs of the next kernel that move in earlier take SMs from this one's
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- host side --------------------------------------------------------------------------------------------------------
// Cycles of a unit: the groups' way from a run's last product over its sums and the next unit to the next operand, about the same for all N (2,450 for 128 tokens, of
// which 2,048 are products, 2,500 for 16).
constexpr double kUnitCycles = 2500, kFixedCycles = 10000;

template <uint32_t TYPE>
int32_t launch_type(const GemvArgs& a, const GemmWorkspace& ws, GemmParams& p, const GemmGroup* group, int* summed_slices, cudaStream_t s) {
    const int nmat = a.epi == EPI_SILU_MUL ? 2 : 1, units = p.k / kUnitElems;
    const int tiles = ((p.n * nmat + kGemmRows - 1) / kGemmRows + 1) / 2 * 2;  // whole pairs
    const int N = gemm_tokens(group ? group->typical : p.T, 32);
    const GemmCut cut = group ? GemmCut{N, 1} : gemm_cut(a, ws, p.T, N, tiles, units, nmat, kUnitCycles, kFixedCycles);
    const bool wide = cut.N > 64;
    const int box = wide ? cut.N / 2 : cut.N;
    // three raw units, as many activation stages as fit, more raw units
    const size_t raw = (size_t)RawUnit<TYPE>::pitch * kGemmRows, fixed = 1024 + 1024, b = (size_t)cut.N * (wide ? 128 : 256);
    p.N = cut.N;
    p.b_stages = std::min<int>(kMaxB, (int)((kMaxSmem - fixed - 3 * raw) / b));
    p.raw_stages = std::min<int>(kGemmRaw, (int)((kMaxSmem - fixed - p.b_stages * b) / raw));
    p.ksplit = cut.ks;
    p.partial = cut.ks > 1 ? ws.partial : nullptr;
    *summed_slices = cut.ks > 1 ? cut.ks * nmat : 0;
    auto kern = wide ? qgemm_whole_kernel<TYPE, true> : qgemm_whole_kernel<TYPE, false>;
    const size_t smem = fixed + p.b_stages * b + p.raw_stages * raw;
    LC_CUDA(ensure_smem_limit((const void*)kern, smem));
    alignas(64) CUtensorMap tmx, tms;
    const size_t rows = (size_t)ws.t_cap;
    LC_CHECK(make_bf16_tmap_3d(&tmx, ws.xh, (uint64_t)p.k, rows, 2, (uint64_t)p.k, rows * p.k, 64, (uint32_t)box, 1) &&
                 make_bf16_tmap_3d(&tms, ws.sx, (uint64_t)p.k / 16, rows, 2, (uint64_t)p.k / 16, rows * (p.k / 16), 64, (uint32_t)box, 1),
             LC_ERR_CUDA, "qgemm: activation tensor maps");
    const CUtensorMap* t0 = (const CUtensorMap*)a.w->tmap;
    const CUtensorMap* t1 = a.w2 ? (const CUtensorMap*)a.w2->tmap : t0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles, (unsigned)(group ? p.T / cut.N + group->n_experts : (p.T + cut.N - 1) / cut.N), (unsigned)cut.ks);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    LC_CUDA(cudaLaunchKernelEx(&cfg, kern, *t0, *t1, tmx, tms, p));
    return LC_OK;
}

}  // namespace

int32_t launch_qgemm_whole(const GemvArgs& a, const GemmWorkspace& ws, GemmParams& p, const GemmGroup* group, int* summed_slices, cudaStream_t s) {
    return a.w->typ == LC_TYPE_Q5_K ? launch_type<LC_TYPE_Q5_K>(a, ws, p, group, summed_slices, s) : launch_type<LC_TYPE_Q4_K>(a, ws, p, group, summed_slices, s);
}

}  // namespace lc
