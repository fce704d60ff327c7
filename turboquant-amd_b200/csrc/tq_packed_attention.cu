// Contiguous packed decode attention (one query row per BH, no GQA, no paging) and the
// row-wise fast Walsh-Hadamard rotation, for sm_100a.
//
// packed_attention keeps the data layout of the reference's Triton path
// (turboquant/kernels/packed_attention.py:76-227): token-major index bytes,
// sign bytes in the stride-4 order of permute_signs_for_chunked
// (turboquant/kernels/packed_compress.py:180-216) and separate fp16 norm arrays.
// With one query per K/V stream there is no group to share tensor-core tiles, so
// this kernel is CUDA-core code built around conflict-free shared-memory tables:
//  * a warp takes 16 tokens per step, lane = 4 * slot + quarter: the lane reads the quarter's index words of its two
//    tokens and keeps the quarter's 32 query values in registers;
//  * pair table: (c[i0], c[i1]) for every pair of indices, one copy per lane, as two floats for V and as half2 for K (the
//    operands of the score MMAs), so a load per two adjacent dims never collides on a bank;
//  * sign table of the query: for each of a quarter's 8 sign nibbles the 16 sums of +-q' over its 4 dims, one copy
//    per lane; the QJL term is 8 look-ups per lane instead of 32 selects;
//  * every slot runs its own online softmax over the tokens it sees (no shuffles across tokens in the loop, the
//    maximum is only raised when a score exceeds it by 2^8); slots, warps and CTAs are merged at the end.
#include "tq_common.cuh"

namespace tq {
namespace {

// Warps of a CTA: 16, one CTA per SM (up to 128 registers per thread), or 8, up to two CTAs per SM, whose sign tables and merges
// then overlap with one another's steps (2- and 3-bit; the 4-bit tables leave room for one CTA only).
constexpr int kPaWarps = 16, kPaHalfWarps = 8;
__host__ __device__ constexpr int step_tokens(int warps) { return warps * 16; }   // tokens of one step of the CTA, 16 per warp
constexpr int kSignTabBytes = 8 * 16 * 128;     // [nibble position][nibble value][lane]
constexpr float kLog2e = 1.4426950408889634f;

struct PAParams {
    const __half* Q;
    const __half* Qp;
    const uint8_t* k_idx;
    const uint8_t* k_signs;
    const __half* k_rnorm;
    const __half* k_norm;
    const uint8_t* v_idx;
    const __half* v_norm;
    const float* centroids;
    float* ws_acc;   // [slots, 128]
    float2* ws_lse;  // [slots] (max in the log2 domain, sum)
    __half* out;
    float corr_scale;
    int BH, Sk;
    int num_splits;  // > 0: rows are cut into that many parts (slot row * num_splits + part); 0: the CTAs share all steps evenly
};

typedef unsigned long long pa_f2;   // two fp32 in a 64-bit register (sm_100 f32x2 arithmetic)
__device__ __forceinline__ pa_f2 pa_pack(float lo, float hi) {
    pa_f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void pa_unpack(pa_f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ pa_f2 pa_fma(pa_f2 a, pa_f2 b, pa_f2 c) {
    pa_f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ pa_f2 pa_mul(pa_f2 a, pa_f2 b) {
    pa_f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pa_f2 pa_lds64(uint32_t addr) {
    pa_f2 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float pa_lds32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float pa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Byte offset, inside a lane-replicated pair table, of this lane's copy of the entry of dims (2 j, 2 j + 1) of a
// quarter: the 2 * BITS index bits at bit 2 * BITS * j of the quarter's little-endian stream, shifted to the entry
// stride 2^SHIFT, or-ed with the lane's offset inside an entry.  One shift and one logic op.
template <int BITS, int SHIFT>
__device__ __forceinline__ uint32_t pair_offset(const uint32_t (&w)[BITS], int j, uint32_t lane_off) {
    constexpr int PB = 2 * BITS;
    constexpr uint32_t kMask = ((1u << PB) - 1u) << SHIFT;
    const int o = PB * j, lo = o >> 5, sh = o & 31;
    uint32_t x;
    if (sh + PB > 32) x = __funnelshift_r(w[lo], w[lo + 1 < BITS ? lo + 1 : lo], sh - SHIFT);
    else if (sh >= SHIFT) x = w[lo] >> (sh - SHIFT);
    else x = w[lo] << (SHIFT - sh);
    return (x & kMask) | lane_off;
}

template <int BITS>
__device__ __forceinline__ void lds_words(uint32_t addr, uint32_t (&w)[BITS]) {
    if constexpr (BITS == 4) {
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
    } else if constexpr (BITS == 2) {
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr));
    } else {
#pragma unroll
        for (int i = 0; i < BITS; ++i) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[i]) : "r"(addr + 4 * i));
    }
}

constexpr int kPaStages = 2;   // ring of 16-token steps per warp: the one being worked on, the other in flight

template <int BITS, int WARPS>
struct PALayout {
    static constexpr int kThreads = WARPS * 32;
    static constexpr int kStepTokens = step_tokens(WARPS);
    static constexpr int kRow = 16 * BITS;                              // index bytes per token
    static constexpr int kPairs = 1 << (2 * BITS);
    static constexpr int kPairTabBytes = kPairs * 256;                  // (c[i0], c[i1]) as two floats per lane: V
    static constexpr int kHalfTabBytes = kPairs * 128;                  // the same as half2 per lane: K operand of the MMAs
    static constexpr int kSignTabOff = kPairTabBytes + kHalfTabBytes;
    static constexpr int kStageOff = kSignTabOff + kSignTabBytes;
    static constexpr int kStageBytes = 32 * kRow + 256;                 // 16 K rows, 16 V rows, 16 sign rows
    static constexpr int kSmem = kStageOff + WARPS * kPaStages * kStageBytes;
};

// A warp takes 16 tokens per step.  Lane (slot, quarter) = (lane >> 2, lane & 3) owns quarter `quarter` (32 dims) of
// tokens slot and slot + 8 of the step:
//  * K score: the lane's 16 pairs of adjacent dims of both tokens are looked up as half2 and are, as they come, the A
//    operands of 8 m16n8k16 MMAs (row = token, the 16 k-slots of MMA ks are dims 4 ks .. 4 ks + 3 of the four
//    quarters); the B operand carries the query in column 0 only, so the fp32 dot products land in the quarter-0 lanes;
//  * QJL term: per quarter, 8 look-ups in the query's sign table;
//  * V: per token 16 look-ups of (c[i0], c[i1]) as floats, f32x2 multiply-adds into the lane's 32 accumulators.
// Every slot runs its own online softmax (no exchange between tokens inside the loop).
//
// Work: with num_splits = 0 the steps of all rows, laid end to end, are shared evenly by the CTAs of one wave; a CTA writes
// the result of a row that lies inside its share, and leaves at most two partials (slot 2 c + 1: the row starts in the
// share, 2 c: it does not).  A row costs a sign table and a merge wherever it is cut, so cutting rows into equal parts
// until they fill whole waves cost 15 % of the largest shapes.  (Staging by bulk copies was slower than the cp.async pieces
// below: 122 us with three copies per warp and step, 107 with three per CTA and step, against 98 on 64 x 32768, 3-bit.)
struct Segment {   // part of a row
    int row, tok, end;   // tokens [tok, end)
    int slot;            // of its partial; -1: the whole row
};

template <int BITS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, kPaWarps / WARPS) packed_attn_partial(const PAParams p, int n_items) {
    using LO = PALayout<BITS, WARPS>;
    constexpr int ROW = LO::kRow, kStepTokens = LO::kStepTokens;
    extern __shared__ __align__(128) unsigned char pa_smem[];
    unsigned char* pair_tab = pa_smem;
    unsigned char* half_tab = pa_smem + LO::kPairTabBytes;
    unsigned char* sign_tab = pa_smem + LO::kSignTabOff;        // [nibble position][value][lane] float
    __shared__ __align__(16) float sqp[kHeadDim];
    __shared__ __align__(16) float sacc[WARPS][kHeadDim];
    __shared__ float sml[WARPS][2];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slot = lane >> 2, quarter = lane & 3;

    // ---- the CTA's segments ----
    const int steps = (p.Sk + kStepTokens - 1) / kStepTokens;   // per row
    const int64_t total = static_cast<int64_t>(p.BH) * steps;
    const int64_t u0 = total * blockIdx.x / gridDim.x, u1 = total * (blockIdx.x + 1) / gridDim.x;
    const int per = p.num_splits > 0 ? (p.Sk + p.num_splits - 1) / p.num_splits : 0;   // tokens per split (packed_attention.py:98-100)
    auto segment = [&](int64_t at) -> Segment {                 // the segment that starts at step `at`, or item `at`
        Segment g;
        if (p.num_splits > 0) {
            g.row = static_cast<int>(at / p.num_splits);
            const int part = static_cast<int>(at - static_cast<int64_t>(g.row) * p.num_splits);
            g.tok = min(part * per, p.Sk);
            g.end = min(g.tok + per, p.Sk);
            g.slot = p.num_splits == 1 ? -1 : static_cast<int>(at);
        } else {
            g.row = static_cast<int>(at / steps);
            const int k = static_cast<int>(at - static_cast<int64_t>(g.row) * steps);
            const int64_t left = u1 - at;
            g.tok = k * kStepTokens;
            g.end = left < steps - k ? g.tok + static_cast<int>(left) * kStepTokens : p.Sk;
            g.slot = k == 0 && g.end == p.Sk ? -1 : 2 * static_cast<int>(blockIdx.x) + (k == 0 ? 1 : 0);
        }
        return g;
    };
    auto after = [&](int64_t at, const Segment& g) -> int64_t { // where the next segment starts; past `stop`: there is none
        return p.num_splits > 0 ? at + gridDim.x : at + (g.end - g.tok + kStepTokens - 1) / kStepTokens;
    };
    int64_t at = p.num_splits > 0 ? static_cast<int64_t>(blockIdx.x) : u0;
    const int64_t stop = p.num_splits > 0 ? static_cast<int64_t>(n_items) : u1;
    pdl_wait();
    pdl_release();
    if (at >= stop) return;

    // ---- item state: which segment the CTA works on, and the warp's asynchronous staging of it: per step a warp
    // copies its 16 K rows, 16 V rows and 16 sign rows in 16-byte pieces (every row is a multiple of 16 bytes, so any
    // token starts on a 16-byte boundary) ----
    const uint32_t stage0 = smem_u32(pa_smem + LO::kStageOff + warp * kPaStages * LO::kStageBytes);
    Segment seg;
    int t1 = 0, tok16 = 0;                                      // end of the segment, first token of this warp's current step
    const uint8_t *kptr = nullptr, *vptr = nullptr, *sptr = nullptr;
    const uint16_t *knp = nullptr, *krnp = nullptr, *vnp = nullptr;
    int tok_issue = 0, stage_issue = 0;
    uint16_t nrm[6] = {0, 0, 0, 0, 0, 0};                       // kn, krn, vn of token A (slot); of token B (slot + 8)
    uint16_t qp_dim = 0;                                        // dim tid of the segment's sign query
    // token row of this lane's pieces (piece c + lane of the 16 rows); 99 = the lane has no such piece
    int piece_row[(ROW + 31) / 32];
#pragma unroll
    for (int c = 0; c < ROW; c += 32) piece_row[c / 32] = c + lane < ROW ? ((c + lane) * 16) / ROW : 99;
    auto issue = [&]() {
        const uint32_t dst = stage0 + stage_issue * LO::kStageBytes + lane * 16;
#pragma unroll
        for (int c = 0; c < ROW; c += 32) {
            if (tok_issue + piece_row[c / 32] < t1 && piece_row[c / 32] < 16) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + c * 16), "l"(kptr + c * 16) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * ROW + c * 16), "l"(vptr + c * 16) : "memory");
            }
        }
        if (lane < 16 && tok_issue + lane < t1)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 32 * ROW), "l"(sptr) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        kptr += kStepTokens * ROW;
        vptr += kStepTokens * ROW;
        sptr += kStepTokens * 16;
        tok_issue += kStepTokens;
        stage_issue = stage_issue + 1 == kPaStages ? 0 : stage_issue + 1;
    };
    auto load_norms = [&](int tk, uint16_t (&n)[6]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = tk + slot + 8 * h;
            if (t < t1) {
                n[3 * h] = __ldg(knp + t);
                n[3 * h + 1] = __ldg(krnp + t);
                n[3 * h + 2] = __ldg(vnp + t);
            } else {
                n[3 * h] = n[3 * h + 1] = n[3 * h + 2] = 0;
            }
        }
    };
    // Starts a segment: its first copies and norms are requested here, i.e. (from the second one on) before the merge of
    // the one just finished, so their latency is hidden behind it.
    auto begin = [&](int64_t from) {
        seg = segment(from);
        t1 = seg.end;
        const int64_t base = static_cast<int64_t>(seg.row) * p.Sk;
        tok16 = seg.tok + warp * 16;
        kptr = p.k_idx + (base + tok16) * ROW + lane * 16;
        vptr = p.v_idx + (base + tok16) * ROW + lane * 16;
        sptr = p.k_signs + (base + tok16) * 16 + lane * 16;
        knp = reinterpret_cast<const uint16_t*>(p.k_norm) + base;
        krnp = reinterpret_cast<const uint16_t*>(p.k_rnorm) + base;
        vnp = reinterpret_cast<const uint16_t*>(p.v_norm) + base;
        tok_issue = tok16;
        stage_issue = 0;
        // ahead of the tables and merges that come before its use (3-bit 64 x 32768: 90.3 us, loaded where it is used, now 88.7)
        if (tid < kHeadDim) qp_dim = __ldg(reinterpret_cast<const uint16_t*>(p.Qp) + static_cast<int64_t>(seg.row) * kHeadDim + tid);
#pragma unroll
        for (int i = 0; i < kPaStages - 1; ++i) issue();
        load_norms(tok16, nrm);
    };
    // The pair tables are filled behind the first copies.  Every lane holds one centroid; an entry's two come by shuffle.
    {
        const float cv = __ldg(p.centroids + (lane & ((1 << BITS) - 1)));
        begin(at);
        auto pair = [&](int pr) { return make_float2(__shfl_sync(0xffffffffu, cv, pr & ((1 << BITS) - 1)), __shfl_sync(0xffffffffu, cv, pr >> BITS)); };
#pragma unroll
        for (int i = 0; i < (LO::kPairs + 2 * WARPS - 1) / (2 * WARPS); ++i) {       // 16 bytes a lane
            const int p0 = 2 * (i * WARPS + warp);
            if (p0 >= LO::kPairs) break;
            const float2 c = pair(p0 + (lane >> 4));
            *reinterpret_cast<float4*>(pair_tab + p0 * 256 + lane * 16) = make_float4(c.x, c.y, c.x, c.y);
        }
#pragma unroll
        for (int i = 0; i < (LO::kPairs + 4 * WARPS - 1) / (4 * WARPS); ++i) {
            const int p0 = 4 * (i * WARPS + warp);
            if (p0 >= LO::kPairs) break;
            const float2 c = pair(p0 + (lane >> 3));
            const uint32_t h = pack_half2(c.x, c.y);
            *reinterpret_cast<uint4*>(half_tab + p0 * 128 + lane * 16) = make_uint4(h, h, h, h);
        }
    }
    const uint32_t lane8 = lane * 8, lane4 = lane * 4;
    // selector that gathers byte `quarter` of two sign words
    const uint32_t sel_lo = static_cast<uint32_t>(quarter) | (static_cast<uint32_t>(4 + quarter) << 4);
    const uint32_t my_words = stage0 + lane * (4 * BITS);       // this lane's K words of token A inside a stage
    const uint32_t my_signs = stage0 + 32 * ROW + slot * 16;

    while (at < stop) {
        // B operands: the query's quarter `quarter` as loaded (pairs of adjacent dims), in column 0 (slot 0) only
        uint32_t qf[16];
        {
            const uint4* qsrc = reinterpret_cast<const uint4*>(p.Q + static_cast<int64_t>(seg.row) * kHeadDim + 32 * quarter);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 v = slot == 0 ? __ldg(qsrc + i) : make_uint4(0u, 0u, 0u, 0u);
                qf[4 * i] = v.x; qf[4 * i + 1] = v.y; qf[4 * i + 2] = v.z; qf[4 * i + 3] = v.w;
            }
        }
        // ---- the query's sign table ----
        if (tid < kHeadDim) sqp[tid] = __half2float(__ushort_as_half(qp_dim)) * p.corr_scale;
        __syncthreads();
        // Sign nibble g = 2 c + h of a lane's sign word (byte c = byte `quarter` of sign word c) holds, in bit kk, the
        // sign of local dim 4 (4 h + kk) + c (stride-4 order: dim 4 i + c is bit i of word c).  A lane makes the sum of one of
        // eight values of a nibble in one quarter, and the warp spreads the 32 sums over the copies.  (Every lane the sum of every
        // entry it writes was eight times the shared-memory reads, four to a bank: us per launch in a graph, so / now, 4-bit 32 rows x
        // 1000 tokens 8.6 / 7.85, 8 x 300 7.0 / 6.3, 3-bit 32 x 1000 8.2 / 7.4.)
        for (int part = warp; part < 16; part += WARPS) {
            const int g = part >> 1, v0 = 8 * (part & 1), v = v0 + slot, c = g >> 1, h = g & 1;
            float sum = 0.f;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float x = sqp[32 * quarter + 4 * (4 * h + kk) + c];
                sum += ((v >> kk) & 1) ? x : -x;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float*>(sign_tab + ((g * 16 + v0 + i) * 32 + lane) * 4) = __shfl_sync(0xffffffffu, sum, 4 * i + quarter);
        }
        __syncthreads();

        float m_run = -INFINITY, l_run = 0.f;     // this slot's online softmax (log2 domain)
        pa_f2 acc[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] = pa_pack(0.f, 0.f);

        int stage = 0;
        for (; tok16 < t1; tok16 += kStepTokens) {
            const bool valid_a = tok16 + slot < t1, valid_b = tok16 + slot + 8 < t1;
            issue();
            uint16_t nrm_n[6];
            load_norms(tok16 + kStepTokens, nrm_n);
            asm volatile("cp.async.wait_group %0;" ::"n"(kPaStages - 1) : "memory");
            __syncwarp();
            const uint32_t so = stage * LO::kStageBytes;
            uint32_t kwa[BITS], kwb[BITS];
            lds_words<BITS>(my_words + so, kwa);
            lds_words<BITS>(my_words + so + 8 * ROW, kwb);
            uint4 sga, sgb;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(sga.x), "=r"(sga.y), "=r"(sga.z), "=r"(sga.w) : "r"(my_signs + so));
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(sgb.x), "=r"(sgb.y), "=r"(sgb.z), "=r"(sgb.w) : "r"(my_signs + so + 128));
            // ---- K scores: rows = the 16 tokens, column 0 = the query ----
            float mse[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const uint32_t a0 = *reinterpret_cast<const uint32_t*>(half_tab + pair_offset<BITS, 7>(kwa, 2 * ks, lane4));
                const uint32_t a1 = *reinterpret_cast<const uint32_t*>(half_tab + pair_offset<BITS, 7>(kwb, 2 * ks, lane4));
                const uint32_t a2 = *reinterpret_cast<const uint32_t*>(half_tab + pair_offset<BITS, 7>(kwa, 2 * ks + 1, lane4));
                const uint32_t a3 = *reinterpret_cast<const uint32_t*>(half_tab + pair_offset<BITS, 7>(kwb, 2 * ks + 1, lane4));
                mma_f16_16816(mse, a0, a1, a2, a3, qf[2 * ks], qf[2 * ks + 1]);
            }
            // ---- QJL term of this lane's quarter, both tokens ----
            const uint32_t swa = prmt(prmt(sga.x, sga.y, sel_lo), prmt(sga.z, sga.w, sel_lo), 0x5410);
            const uint32_t swb = prmt(prmt(sgb.x, sgb.y, sel_lo), prmt(sgb.z, sgb.w, sel_lo), 0x5410);
            float qja = 0.f, qjb = 0.f;
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                const uint32_t xa = 4 * g >= 7 ? (swa >> (4 * g - 7)) : (swa << (7 - 4 * g));
                const uint32_t xb = 4 * g >= 7 ? (swb >> (4 * g - 7)) : (swb << (7 - 4 * g));
                qja += *reinterpret_cast<const float*>(sign_tab + g * 2048 + ((xa & (15u << 7)) | lane4));
                qjb += *reinterpret_cast<const float*>(sign_tab + g * 2048 + ((xb & (15u << 7)) | lane4));
            }
            // the quarter-0 lane of a slot holds the whole MSE dot product (column 0 of rows slot and slot + 8)
            float pa = __half2float(__ushort_as_half(nrm[1])) * qja, pb = __half2float(__ushort_as_half(nrm[4])) * qjb;
            if (quarter == 0) {
                pa = fmaf(__half2float(__ushort_as_half(nrm[0])), mse[0], pa);
                pb = fmaf(__half2float(__ushort_as_half(nrm[3])), mse[2], pb);
            }
            pa += __shfl_xor_sync(0xffffffffu, pa, 1);
            pb += __shfl_xor_sync(0xffffffffu, pb, 1);
            pa += __shfl_xor_sync(0xffffffffu, pa, 2);
            pb += __shfl_xor_sync(0xffffffffu, pb, 2);
            const float sa = valid_a ? pa * kLog2e : -INFINITY, sb = valid_b ? pb * kLog2e : -INFINITY;
            // ---- online softmax of this slot: the maximum is raised only when a score exceeds it by 2^8 ----
            const float smax = fmaxf(sa, sb);
            if (smax > m_run + 8.f) {
                const float alpha = pa_ex2(m_run - smax);     // 0 on the first token
                const pa_f2 al2 = pa_pack(alpha, alpha);
                l_run *= alpha;
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[j] = pa_mul(acc[j], al2);
                m_run = smax;
            }
            const float pra = valid_a ? pa_ex2(sa - m_run) : 0.f, prb = valid_b ? pa_ex2(sb - m_run) : 0.f;
            l_run += pra + prb;
            // ---- V ----
            {
                uint32_t vw[BITS];
                lds_words<BITS>(my_words + so + 16 * ROW, vw);
                const float wv = pra * __half2float(__ushort_as_half(nrm[2]));
                const pa_f2 wv2 = pa_pack(wv, wv);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    acc[j] = pa_fma(wv2, *reinterpret_cast<const pa_f2*>(pair_tab + pair_offset<BITS, 8>(vw, j, lane8)), acc[j]);
            }
            {
                uint32_t vw[BITS];
                lds_words<BITS>(my_words + so + 24 * ROW, vw);
                const float wv = prb * __half2float(__ushort_as_half(nrm[5]));
                const pa_f2 wv2 = pa_pack(wv, wv);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    acc[j] = pa_fma(wv2, *reinterpret_cast<const pa_f2*>(pair_tab + pair_offset<BITS, 8>(vw, j, lane8)), acc[j]);
            }
#pragma unroll
            for (int i = 0; i < 6; ++i) nrm[i] = nrm_n[i];
            stage = stage + 1 == kPaStages ? 0 : stage + 1;
            __syncwarp();   // every lane has read this stage before the next step's copy may land in it
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        const Segment finished = seg;
        at = after(at, seg);
        if (at < stop) begin(at);

        // ---- merge the 8 slots of the warp, then the warps ----
        float M = m_run;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        const float f = (m_run == -INFINITY) ? 0.f : pa_ex2(m_run - M);
        float L = l_run * f;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        // The eight slots' sums: at each of three steps a lane gives away the half of its values that the other lane keeps, so it
        // ends with four dims: 28 shuffles, where summing every value over all slots took 96 and 1 us a row (us per launch in a
        // graph, so / now: 4-bit 32 rows x 1000 tokens 7.85 / 6.9, 3-bit 1000 x 256 27.6 / 23.4, 64 x 32768 89.0 / 87.0).
        float t[32];
#pragma unroll
        for (int j = 0; j < 16; ++j) pa_unpack(pa_mul(acc[j], pa_pack(f, f)), t[2 * j], t[2 * j + 1]);
        int dim = 0;
#pragma unroll
        for (int o = 16, n = 16; o >= 4; o >>= 1, n >>= 1) {
            const bool upper = lane & o;
            dim += upper ? n : 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float keep = upper ? t[n + i] : t[i], give = upper ? t[i] : t[n + i];
                t[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        *reinterpret_cast<float4*>(&sacc[warp][32 * quarter + dim]) = make_float4(t[0], t[1], t[2], t[3]);
        if (lane == 0) {
            sml[warp][0] = M;
            sml[warp][1] = L;
        }
        __syncthreads();
        if (tid < kHeadDim) {
            float Mc = sml[0][0];
#pragma unroll
            for (int w = 1; w < WARPS; ++w) Mc = fmaxf(Mc, sml[w][0]);
            float o = 0.f, l = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const float fw = (sml[w][0] == -INFINITY) ? 0.f : pa_ex2(sml[w][0] - Mc);
                o = fmaf(fw, sacc[w][tid], o);
                l = fmaf(fw, sml[w][1], l);
            }
            if (finished.slot < 0) {
                p.out[static_cast<int64_t>(finished.row) * kHeadDim + tid] = __float2half_rn(o / l);
            } else {
                p.ws_acc[static_cast<int64_t>(finished.slot) * kHeadDim + tid] = o;
                if (tid == 0) p.ws_lse[finished.slot] = make_float2(Mc, l);
            }
        }
        // The next segment's first __syncthreads stands between these reads and its writes of sacc and the sign table.
    }
}

// One block per row: four warps share the parts, a lane holds four dims.
constexpr int kMergeWarps = 4;
__global__ void __launch_bounds__(kMergeWarps * 32) packed_attn_merge(const PAParams p, int n_ctas, int steps) {
    __shared__ float4 so[kMergeWarps][32];
    __shared__ float sl[kMergeWarps];
    __shared__ float sm[kMergeWarps];
    pdl_release();
    const int bh = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t slot0, parts, step = 1;
    if (p.num_splits > 0) {
        slot0 = static_cast<int64_t>(bh) * p.num_splits;
        parts = p.num_splits;
    } else {
        const int64_t total = static_cast<int64_t>(p.BH) * steps, first = static_cast<int64_t>(bh) * steps;
        // the CTA whose share holds step u is the largest c with floor(c total / n) <= u
        const int64_t c0 = ((first + 1) * n_ctas - 1) / total, c1 = ((first + steps) * n_ctas - 1) / total;
        if (c0 == c1) {                          // written by that CTA
            pdl_wait();
            return;
        }
        slot0 = 2 * c0;                          // slot 2 c0 + 1, then 2 c for the others
        parts = c1 - c0 + 1;
        step = 2;
    }
    auto slot_of = [&](int64_t i) { return slot0 + step * i + (step == 2 && i == 0 ? 1 : 0); };
    const float2* lse = p.ws_lse;
    const float4* part = reinterpret_cast<const float4*>(p.ws_acc);
    pdl_wait();
    // eight parts at a time, fetched independently of the maxima and a turn ahead: what a merge costs is its chain of loads
    float M = -INFINITY, l = 0.f;
    float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int kAtOnce = 8;
    float2 ml[kAtOnce], ml_next[kAtOnce];
    float4 v[kAtOnce], v_next[kAtOnce];
    auto fetch = [&](int64_t i0, float2 (&a)[kAtOnce], float4 (&b)[kAtOnce]) {
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) {
            const int64_t i = i0 + k * kMergeWarps;
            a[k] = make_float2(-INFINITY, 0.f);
            b[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < parts) {
                a[k] = lse[slot_of(i)];
                b[k] = part[slot_of(i) * (kHeadDim / 4) + lane];
            }
        }
    };
    fetch(warp, ml, v);
    for (int64_t i0 = warp; i0 < parts; i0 += kAtOnce * kMergeWarps) {
        fetch(i0 + kAtOnce * kMergeWarps, ml_next, v_next);
        float m = M;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) m = fmaxf(m, ml[k].x);
        const float old = M == -INFINITY ? 0.f : pa_ex2(M - m);   // empty parts carry no weight; a part of NaN sums stays one
        o4.x *= old; o4.y *= old; o4.z *= old; o4.w *= old;
        l *= old;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) {
            const float w = ml[k].x == -INFINITY ? 0.f : pa_ex2(ml[k].x - m);
            o4.x = fmaf(w, v[k].x, o4.x);
            o4.y = fmaf(w, v[k].y, o4.y);
            o4.z = fmaf(w, v[k].z, o4.z);
            o4.w = fmaf(w, v[k].w, o4.w);
            l = fmaf(w, ml[k].y, l);
            ml[k] = ml_next[k];
            v[k] = v_next[k];
        }
        M = m;
    }
    so[warp][lane] = o4;
    if (lane == 0) {
        sl[warp] = l;
        sm[warp] = M;
    }
    __syncthreads();
    if (warp == 0) {
        float Ma = sm[0];
#pragma unroll
        for (int w = 1; w < kMergeWarps; ++w) Ma = fmaxf(Ma, sm[w]);
        o4 = make_float4(0.f, 0.f, 0.f, 0.f);
        l = 0.f;
#pragma unroll
        for (int w = 0; w < kMergeWarps; ++w) {
            const float4 v = so[w][lane];
            const float f = sm[w] == -INFINITY ? 0.f : pa_ex2(sm[w] - Ma);
            o4.x = fmaf(f, v.x, o4.x);
            o4.y = fmaf(f, v.y, o4.y);
            o4.z = fmaf(f, v.z, o4.z);
            o4.w = fmaf(f, v.w, o4.w);
            l = fmaf(f, sl[w], l);
        }
        __half* dst = p.out + static_cast<int64_t>(bh) * kHeadDim + 4 * lane;
        if ((reinterpret_cast<uintptr_t>(p.out) & 7) == 0) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(pack_half2(o4.x / l, o4.y / l), pack_half2(o4.z / l, o4.w / l));
        } else {   // an output that starts anywhere
            dst[0] = __float2half_rn(o4.x / l);
            dst[1] = __float2half_rn(o4.y / l);
            dst[2] = __float2half_rn(o4.z / l);
            dst[3] = __float2half_rn(o4.w / l);
        }
    }
}

// ---- row-wise WHT ----------------------------------------------------------------------
__global__ void __launch_bounds__(128) wht_rows_kernel(const void* in, void* out, int dtype, int64_t n, float scale) {
    pdl_wait();
    pdl_release_if_small();
    const int lane = threadIdx.x & 31;
    const int64_t row = static_cast<int64_t>(blockIdx.x) * 4 + (threadIdx.x >> 5);
    if (row >= n) return;
    float x[4];
    load4(in, row * kHeadDim + 4 * lane, dtype, x);
    float a = x[0] + x[1], b = x[0] - x[1], c = x[2] + x[3], d = x[2] - x[3];
    x[0] = a + c; x[1] = b + d; x[2] = a - c; x[3] = b - d;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const float sgn = (lane & m) ? -1.f : 1.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = fmaf(sgn, x[e], __shfl_xor_sync(0xffffffffu, x[e], m));
    }
    const float k = kWhtScale * scale;
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] *= k;
    const int64_t o = row * kHeadDim + 4 * lane;
    if (dtype == TQ_DTYPE_F32) {
        *reinterpret_cast<float4*>(static_cast<float*>(out) + o) = make_float4(x[0], x[1], x[2], x[3]);
    } else if (dtype == TQ_DTYPE_F16) {
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(out) + o) = make_uint2(pack_half2(x[0], x[1]), pack_half2(x[2], x[3]));
    } else {
        __nv_bfloat162 lo = __floats2bfloat162_rn(x[0], x[1]), hi = __floats2bfloat162_rn(x[2], x[3]);
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(out) + o) =
            make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    }
}

}  // namespace
}  // namespace tq

using namespace tq;

constexpr int64_t kMaxCtas = 512;   // CTAs that share the steps of all rows: at most two per SM

// How a call without an explicit split runs: so many CTAs of so many warps share the steps of all rows.
struct Sharing {
    int warps;
    int64_t ctas;
    double us;    // estimated
    bool whole;   // rows are dealt out whole (no merge kernel); else the steps of all rows are shared
};

// What a call is estimated to take, in us: a launch costs `start`, a step of the CTA `step`, a row (or part of one) of its share `row`
// for the sign table and the merge, the merge kernel kMergeUs and for every further 32 parts of a row kMorePartsUs.  CTAs of 8 warps
// depend on whether another one runs on the SM.  Times of every arrangement of 1339 calls, 1 to 2000 rows of 64 to 65536 tokens, at most 2.7 M
// in all, 2, 3 and 4 bits, in a graph: least squares give 1.0 / 1.5 / 1.6, 2.1 / 1.4 / 1.5 and 2.1 / 0.8 / 0.4, merge 1.25; the
// values below choose best among them (0.2 % over the fastest arrangement in the mean, 13 % at most; steps of 1.4 or 1.5 and rows of 2.2 or
// 2.5 whatever else runs on the SM: 4 % and 35 %).  On 520 other calls 0.2 % and 15 %; against those values 3.6 % faster in the mean, 7 %
// slower at most (35 x 434), 2 % next to that.
struct ShareCosts { double start, step, row; };
constexpr ShareCosts kCostsOneCta = {1.1, 1.5, 1.7}, kCostsTwoCtas = {1.75, 1.45, 1.35}, kCostsHalfCta = {1.75, 0.85, 0.45};
constexpr double kMergeUs = 2.1, kMorePartsUs = 0.65;

// All SMs balance best, but a share that crosses into another row pays for another sign table and merge; with few steps per
// CTA that is dearer than idle SMs.  Candidates: all CTAs; every row cut into the same number of parts; whole rows.
static Sharing share_among(int64_t BH, int64_t Sk, int64_t sms, int warps) {
    const int64_t ctas = warps == kPaWarps ? sms : 2 * sms;
    const int64_t S = (Sk + step_tokens(warps) - 1) / step_tokens(warps), total = BH * S;
    auto costs = [&](int64_t running) { return warps == kPaWarps ? kCostsOneCta : running > sms ? kCostsTwoCtas : kCostsHalfCta; };
    auto share = [&](int64_t running, int64_t steps, int64_t rows) {
        const ShareCosts c = costs(running);
        return c.start + c.step * static_cast<double>(steps) + c.row * static_cast<double>(rows);
    };
    auto merge = [&](int64_t parts) { return kMergeUs + kMorePartsUs * static_cast<double>((parts - 1) / 32); };
    Sharing best = {warps, total < ctas ? total : ctas, 0.0, false};
    const int64_t each = (total + best.ctas - 1) / best.ctas;
    best.us = share(best.ctas, each, 1 + (each - 1 + S - 1) / S) + merge((best.ctas + BH - 1) / BH);
    auto consider = [&](const Sharing& other) {
        if (other.us < best.us) best = other;
    };
    if (BH <= ctas) {
        const int64_t parts = ctas / BH < S ? ctas / BH : S;
        consider({warps, BH * parts, share(BH * parts, (S + parts - 1) / parts, 1) + merge(parts), false});
        consider({warps, BH, share(BH, S, 1), true});
    } else {   // the rows of the last round have an SM to themselves the more the fewer they are
        const int64_t rounds = BH / ctas, left = BH % ctas;
        double us = share(ctas, rounds * S, rounds);
        if (left) {
            const ShareCosts busy = costs(ctas), lone = costs(left);
            const double crowd = left < sms ? static_cast<double>(left) / static_cast<double>(sms) : 1.0;
            const double alone = lone.step * static_cast<double>(S) + lone.row, among = busy.step * static_cast<double>(S) + busy.row;
            us += alone + crowd * (among - alone);
        }
        consider({warps, ctas, us, true});
    }
    return best;
}

// Many rows of few steps are mostly sign tables and merges, which overlap where two CTAs share an SM.  Measured in a graph, us, the best
// arrangement with CTAs of 16 warps / of 8, 3-bit: 150 x 700 tokens 13.5 / 12.2, 256 x 500 12.6 / 10.4, 256 x 2048 30.6 / 28.0, 1000 x 256
// 26.7 / 22.5, 2000 x 64 37.3 / 22.0, 64 x 32768 87.4 / 85.7.  Few steps start sooner with 8: 1 x 1000 6.4 / 4.9, 16 x 500 6.5 / 5.2.  A row of many
// steps takes fewer parts with 16: 1 x 32768 9.1 / 12.7, 2 x 16000 7.5 / 9.4.
static Sharing share_out(int64_t BH, int64_t Sk, int bits, int64_t sms) {
    const Sharing one = share_among(BH, Sk, sms, kPaWarps);
    if (bits == 4) return one;
    const Sharing two = share_among(BH, Sk, sms, kPaHalfWarps);
    return two.us < one.us ? two : one;
}

extern "C" int tq_packed_attention_auto_splits(int BH, int Sk) {
    if (BH <= 0 || Sk <= 0) return TQ_ERR_ARG;
    const int64_t parts = share_among(BH, Sk, 148, kPaWarps).ctas / BH;   // CTAs per row on the 148 SMs of a B200
    return static_cast<int>(parts < 1 ? 1 : parts);
}

extern "C" int64_t tq_packed_attention_workspace_bytes(int BH, int num_splits) {
    if (BH <= 0 || num_splits < 0) return TQ_ERR_ARG;
    const int64_t slots = num_splits > 0 ? static_cast<int64_t>(BH) * num_splits : 2 * kMaxCtas;
    return slots * (kHeadDim + 2) * static_cast<int64_t>(sizeof(float));
}

extern "C" int tq_packed_attention(const void* Q, const void* Q_proj, const uint8_t* k_idx, const uint8_t* k_signs_perm,
                                   const void* k_rnorm, const void* k_norm, const uint8_t* v_idx, const void* v_norm,
                                   const float* centroids, float corr_scale, int BH, int Sk, int bits, int num_splits,
                                   void* workspace, int64_t workspace_bytes, void* out, tq_stream_t stream) {
    if (BH == 0) return TQ_OK;
    if (!Q || !Q_proj || !k_idx || !k_signs_perm || !k_rnorm || !k_norm || !v_idx || !v_norm || !centroids || !out)
        return TQ_ERR_ARG;
    if (BH < 0 || Sk <= 0) return TQ_ERR_ARG;
    if (bits < 2 || bits > 4) return TQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(k_idx) | reinterpret_cast<uintptr_t>(k_signs_perm) |
         reinterpret_cast<uintptr_t>(v_idx)) & 15)
        return TQ_ERR_ARG;
    if (num_splits < 0) num_splits = 0;
    // A workspace that holds the parts of tq_packed_attention_auto_splits, but not those of shared steps: equal parts.
    if (num_splits == 0 && workspace_bytes < tq_packed_attention_workspace_bytes(BH, 0)) num_splits = tq_packed_attention_auto_splits(BH, Sk);
    if (num_splits > Sk) num_splits = Sk;
    if (num_splits > 65535) return TQ_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < tq_packed_attention_workspace_bytes(BH, num_splits) ||
        (reinterpret_cast<uintptr_t>(workspace) & 15))
        return TQ_ERR_WORKSPACE;
    const int64_t slots = num_splits > 0 ? static_cast<int64_t>(BH) * num_splits : 2 * kMaxCtas;
    if (slots > 2147483647) return TQ_ERR_UNSUPPORTED;
    PAParams p;
    p.Q = static_cast<const __half*>(Q);
    p.Qp = static_cast<const __half*>(Q_proj);
    p.k_idx = k_idx;
    p.k_signs = k_signs_perm;
    p.k_rnorm = static_cast<const __half*>(k_rnorm);
    p.k_norm = static_cast<const __half*>(k_norm);
    p.v_idx = v_idx;
    p.v_norm = static_cast<const __half*>(v_norm);
    p.centroids = centroids;
    p.ws_acc = static_cast<float*>(workspace);
    p.ws_lse = reinterpret_cast<float2*>(p.ws_acc + slots * kHeadDim);
    p.BH = BH;
    p.out = static_cast<__half*>(out);
    p.corr_scale = corr_scale;
    p.Sk = Sk;
    p.num_splits = num_splits;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    static bool configured[64] = {false};
    static int sm_count[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TQ_ERR_LAUNCH;
    if (dev < 0 || dev >= 64) return TQ_ERR_UNSUPPORTED;
    if (!configured[dev]) {
        if (cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return TQ_ERR_LAUNCH;
        auto opt_in = [](auto kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess; };
        if (!opt_in(packed_attn_partial<4, kPaWarps>, PALayout<4, kPaWarps>::kSmem) || !opt_in(packed_attn_partial<3, kPaWarps>, PALayout<3, kPaWarps>::kSmem) ||
            !opt_in(packed_attn_partial<2, kPaWarps>, PALayout<2, kPaWarps>::kSmem) || !opt_in(packed_attn_partial<3, kPaHalfWarps>, PALayout<3, kPaHalfWarps>::kSmem) ||
            !opt_in(packed_attn_partial<2, kPaHalfWarps>, PALayout<2, kPaHalfWarps>::kSmem))
            return TQ_ERR_LAUNCH;
        configured[dev] = true;
    }
    const int64_t sms = sm_count[dev] < kMaxCtas / 2 ? sm_count[dev] : kMaxCtas / 2;
    Sharing run = {};
    if (num_splits > 0) {   // items of their own: two CTAs per SM where there are enough of them
        run.warps = bits < 4 && slots > sms ? kPaHalfWarps : kPaWarps;
        const int64_t most = run.warps == kPaWarps ? sms : 2 * sms;
        run.ctas = slots < most ? slots : most;
    } else {
        run = share_out(BH, Sk, bits, sms);
        if (run.whole) p.num_splits = num_splits = 1;
    }
    const int n_items = num_splits > 0 ? BH * num_splits : 0;
    auto partial = [&](auto kernel, int threads, int smem) {
        return launch_chained(kernel, dim3(static_cast<unsigned>(run.ctas)), dim3(threads), smem, st, p, n_items) == cudaSuccess;
    };
    bool launched = false;
    if (run.warps == kPaWarps) {
        switch (bits) {
            case 2: launched = partial(packed_attn_partial<2, kPaWarps>, kPaWarps * 32, PALayout<2, kPaWarps>::kSmem); break;
            case 3: launched = partial(packed_attn_partial<3, kPaWarps>, kPaWarps * 32, PALayout<3, kPaWarps>::kSmem); break;
            case 4: launched = partial(packed_attn_partial<4, kPaWarps>, kPaWarps * 32, PALayout<4, kPaWarps>::kSmem); break;
        }
    } else if (bits == 2) {
        launched = partial(packed_attn_partial<2, kPaHalfWarps>, kPaHalfWarps * 32, PALayout<2, kPaHalfWarps>::kSmem);
    } else {
        launched = partial(packed_attn_partial<3, kPaHalfWarps>, kPaHalfWarps * 32, PALayout<3, kPaHalfWarps>::kSmem);
    }
    if (!launched) return TQ_ERR_LAUNCH;
    if (num_splits == 1 || (num_splits == 0 && run.ctas == 1)) return TQ_OK;   // every row was written whole
    const int steps = (Sk + step_tokens(run.warps) - 1) / step_tokens(run.warps);   // per row
    return launch_chained(packed_attn_merge, dim3(static_cast<unsigned>(BH)), dim3(kMergeWarps * 32), 0, st, p, static_cast<int>(run.ctas), steps) == cudaSuccess
               ? TQ_OK
               : TQ_ERR_LAUNCH;
}

extern "C" int tq_wht_rows(const void* in, void* out, int dtype, int64_t n_rows, float scale, tq_stream_t stream) {
    if (n_rows == 0) return TQ_OK;
    if (!in || !out || n_rows < 0) return TQ_ERR_ARG;
    if (dtype != TQ_DTYPE_F16 && dtype != TQ_DTYPE_BF16 && dtype != TQ_DTYPE_F32) return TQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) return TQ_ERR_ARG;
    const unsigned grid = static_cast<unsigned>((n_rows + 3) / 4);
    return launch_chained(wht_rows_kernel, dim3(grid), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream), in, out, dtype, n_rows, scale) == cudaSuccess
               ? TQ_OK
               : TQ_ERR_LAUNCH;
}
