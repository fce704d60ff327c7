// Asymmetric packed paged decode attention (GQA, split-K, optional Sparse-V) for sm_100a.
//
// One CTA = 4 warps works on a chunk of 16-token pages of one (sequence, kv head,
// group of <= 8 query heads).  Every warp owns every 4th page of the chunk and is
// its own producer and consumer: lane 0 streams the next packed pages from HBM
// into the warp's private shared-memory ring with bulk async copies that
// complete on mbarriers, the whole warp then
//   * turns packed indices into fp16 tensor-core fragments: a masked byte of the packed word is
//     the pair index of two neighbouring dims and addresses a lane-replicated half2 table in
//     shared memory (one byte-extract, one multiply-add, one conflict-free shared load per pair),
//   * scores 16 tokens x 8 query heads with mma.m16n8k16 (tokens on M, the GQA
//     group on N), a second MMA chain for the +-1 QJL sign term,
//   * runs the online softmax on the accumulator fragment,
//   * accumulates P V with mma (the transposed P fragment comes from one
//     movmatrix per 8 tokens; the two dims a lane owns per column are told
//     apart by the row half of the accumulator, so V is fed exactly as stored).
// Warps merge in shared memory; chunks merge in a second small kernel.
//
// Arithmetic restated from the reference: score and softmax of
// turboquant/kernels/packed_attention.py:150-196,273-284, paging and GQA head
// mapping of turboquant/kernels/sparse_v.py:39-48,70-71, skip rule of
// sparse_v.py:108-123,149.
#include <type_traits>

#include "tq_common.cuh"

namespace tq {
namespace {

#ifndef TQ_DEC_WARPS
#define TQ_DEC_WARPS 4
#endif
#ifndef TQ_DEC_STAGES
#define TQ_DEC_STAGES 4
#endif
#ifndef TQ_DEC_MINBLOCKS
#define TQ_DEC_MINBLOCKS 4
#endif
constexpr int kWarps = TQ_DEC_WARPS;
constexpr int kThreads = kWarps * 32;
constexpr int kOPad = 132;  // row stride of the merge buffer (floats)
constexpr int kStages = TQ_DEC_STAGES;  // pages in flight per warp
constexpr int kBarBytes = kWarps * 2 * kStages * 8;  // mbarriers at the start of dynamic shared memory

struct DecodeParams {
    void* out;
    const void* q;
    const void* qp;
    const uint8_t* cache;
    const int32_t* block_tables;
    const int32_t* seq_lens;
    const float* kc;
    const float* vc;
    float* ws_o;
    float* ws_ml;
    int32_t* status;
    uint32_t* skip_stats;
    int64_t bt_stride;
    int64_t num_blocks;
    float qscale;    // sm_scale * log2(e)
    float qpscale;   // sm_scale * corr_scale * log2(e) / kSignUnit
    float log2_thresh;
    int Hq, Hkv, G, ngroups;
    int sub_shift;           // log2(block_size / 16)
    int64_t block_stride;    // bytes between consecutive blocks of the cache
    int chunk_pages, max_chunks;
    int max_pages;           // pages per sequence the block table and the workspace were sized for
    int io_dtype;
    int share_tables;        // K and V use the same codebook: one pair table serves both
    int rotate_q;            // the query is in original space: rotate it (fast WHT) while loading
    int derotate_out;        // write the output in original space
    int use_tcgen05;         // TQ_IO_TCGEN05 was given
};

// ---------------------------------------------------------------------------------
// Pair lookup table in shared memory.  After masking, every byte of an index word holds the
// indices of two neighbouring dims of one token in its two nibbles; that byte addresses a table
// of half2(c[i0], c[i1]) which is replicated per lane (entry stride 128 bytes, lane l reads
// word l of an entry) so that a warp's 32 lookups never collide on a bank.  One byte-extract
// (ALU), one multiply-add for the address (FMA pipe) and one shared load replace the two table
// permutes and the interleave permute of the register-only path: the logic pipe is the
// bottleneck of this kernel, the load/store pipe is not.
// ---------------------------------------------------------------------------------
// 2-bit indices: a whole byte of a packed word (four indices = two pairs: bits 1:0 with 5:4, bits 3:2 with 7:6)
// addresses a table of two half2, so one look-up serves four elements; an entry holds 16 copies of its 8 bytes (a 64-bit
// load is served half a warp at a time, lanes l and l + 16 never meet).
template <int BITS>
__host__ __device__ constexpr int lut_entries() { return BITS == 2 ? 256 : (BITS == 3 ? 128 : 256); }
template <int BITS>
__host__ __device__ constexpr int lut_bytes() { return lut_entries<BITS>() * 128; }

// Every lane fetches one centroid (lane_centroid, rounded to fp16 by the fill) and the entries are assembled from warp
// shuffles, so the fill does not wait on a global load per entry.  Eight lanes write an entry, 16 bytes each: with 4 bytes a
// lane the fill of a 256-entry table took 1.3 us of a launch.
template <int BITS>
__device__ __forceinline__ float lane_centroid(const float* __restrict__ c, int lane) { return __ldg(c + (lane & ((1 << BITS) - 1))); }
// 16 bytes of entry b: the half2 of its two nibbles four times, or, 2-bit, its two half2 (pair A: bits 1:0 with 5:4, pair B:
// bits 3:2 with 7:6) twice.  Nibbles past the codebook are never looked up.
template <int BITS>
__device__ __forceinline__ uint4 pair_entry(float cv, int b) {
    constexpr int kMask = (1 << BITS) - 1;
    const uint32_t a = pack_half2(__shfl_sync(0xffffffffu, cv, b & kMask), __shfl_sync(0xffffffffu, cv, (b >> 4) & kMask));
    if constexpr (BITS > 2) return make_uint4(a, a, a, a);
    const uint32_t o = pack_half2(__shfl_sync(0xffffffffu, cv, (b >> 2) & kMask), __shfl_sync(0xffffffffu, cv, (b >> 6) & kMask));
    return make_uint4(a, o, a, o);
}
template <int BITS>
__device__ __forceinline__ void fill_pair_lut(uint32_t* tab, float centroid, int warp, int lane) {
    const float cv = __half2float(__float2half_rn(centroid));
#pragma unroll 8
    for (int i = 0; i < lut_entries<BITS>() / (4 * kWarps); ++i) {   // unrolled: the shuffles of several entries overlap
        const int b = 4 * (i * kWarps + warp) + (lane >> 3);
        *reinterpret_cast<uint4*>(tab + b * 32 + 4 * (lane & 7)) = pair_entry<BITS>(cv, b);
    }
}

// Words whose bytes are pair indices; word order matches the 8 groups of 4 elements (2 bytes each).
template <int BITS>
__device__ __forceinline__ void masked_words(const uint32_t (&w)[BITS], uint32_t (&mw)[4]) {
    if constexpr (BITS == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mw[j] = w[j];
    } else if constexpr (BITS == 3) {
#pragma unroll
        for (int j = 0; j < 3; ++j) mw[j] = w[j] & 0x77777777u;
        mw[3] = ((w[0] >> 3) & 0x11111111u) | ((w[1] >> 2) & 0x22222222u) | ((w[2] >> 1) & 0x44444444u);
    } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            mw[2 * j] = w[j] & 0x33333333u;
            mw[2 * j + 1] = (w[j] >> 2) & 0x33333333u;
        }
    }
}

// half2(c[i0], c[i1]) for byte k of a masked word; lane_base = shared address of the table + 4 * lane.
__device__ __forceinline__ uint32_t lut_pair(uint32_t lane_base, uint32_t mw, int k) {
    const uint32_t x = prmt(mw, 0u, 0x4440u | static_cast<uint32_t>(k));
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(lane_base + x * 128u));
    return v;
}

// 2-bit tables: (half2 of the pair in bits 1:0 / 5:4, half2 of the pair in bits 3:2 / 7:6) for byte k of a packed
// word; lane_base = shared address of the table + 8 * (lane & 15).
__device__ __forceinline__ uint2 lut_quad(uint32_t lane_base, uint32_t w, int k) {
    const uint32_t x = prmt(w, 0u, 0x4440u | static_cast<uint32_t>(k));
    uint2 v;
    asm("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(lane_base + x * 128u));
    return v;
}

// QJL sign term on fp16 tensor cores with one logic op per pair of signs.
//
// The sign word holds bit l = 1 when the residual of local dim l is >= 0.  A register of the A fragment is a pair of dims
// (j, j + 16), bits j and j + 16, masked where they are: a lone bit 4 .. 11 of an fp16 number is the value 2^-20 .. 2^-13 (the
// subnormal ones too: tensor cores take them as they are).  The other eight pairs come to these bits when the word is rotated by
// a byte, each with its dims swapped or not (qp_frag_signed_from).  This gives value * [sign >= 0] instead of +-1; since
// 2 * [s >= 0] = sigma + 1, a query operand is scaled by 2^7 .. 1, so that every product counts in 2^-13, and the query sum, in
// halves of that, is subtracted once (accumulator start value).  (Bits 12 .. 15 by shifts of four, with operands scaled by up to
// 2^12 that overflowed from 255 on, took 40 instructions a page instead of 34.)
constexpr float kSignUnit = 1.f / 16384.f;   // of sigma * q in the sign sums
__device__ __forceinline__ uint32_t rotate_signs(uint32_t w) { return prmt(w, w, 0x0321u); }
// Pair slot I = 0 .. 15: bits 4 + I of the word w, or for I >= 8 bits I - 4 of w rotated.
template <int I>
__device__ __forceinline__ uint32_t sign_pair(uint32_t w, uint32_t rotated) {
    uint32_t r;
    asm("and.b32 %0, %1, %2;" : "=r"(r) : "r"(I < 8 ? w : rotated), "n"(0x00100010u << (I & 7)));
    return r;
}
// This lane's 32 query values (dims 32 * tig .. 32 * tig + 31 of query row gid) as they are stored, two to a word; zeros when !valid.
__device__ __forceinline__ void load_q_words(const void* q, int64_t row_off, int tig, bool valid, uint32_t (&w)[16]) {
    const uint4* base = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(q) + row_off + tig * 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint4 v = valid ? __ldg(base + i) : make_uint4(0u, 0u, 0u, 0u);
        w[4 * i] = v.x;
        w[4 * i + 1] = v.y;
        w[4 * i + 2] = v.z;
        w[4 * i + 3] = v.w;
    }
}
__device__ __forceinline__ float2 unpack_bf162(uint32_t x) { return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }
// The words' values as fp32.
__device__ __forceinline__ void unpack_q(const uint32_t (&w)[16], int io_dtype, float (&x)[32]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 t = io_dtype == TQ_DTYPE_F16 ? unpack_half2(w[i]) : unpack_bf162(w[i]);
        x[2 * i] = t.x;
        x[2 * i + 1] = t.y;
    }
}

template <bool BF16>
__device__ __forceinline__ void mma_hadamard(float (&d)[4], uint32_t a, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%4,%4,%5}, {%6,%7}, {%8,%8,%8,%8};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%4,%4,%5}, {%6,%7}, {%8,%8,%8,%8};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// (a, b) -> (a + b, a - b) on two pairs of fp32 at a time.
__device__ __forceinline__ void butterfly2(float& a0, float& a1, float& b0, float& b1) {
    asm("{\n\t.reg .b64 a, b, n, s;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tmov.b64 n, {%4, %4};\n\t"
        "add.rn.f32x2 s, a, b;\n\tfma.rn.f32x2 a, b, n, a;\n\tmov.b64 {%0, %1}, s;\n\tmov.b64 {%2, %3}, a;\n\t}"
        : "+f"(a0), "+f"(a1), "+f"(b0), "+f"(b1) : "f"(-1.f));
}
// q' = q H for the eight query rows of a warp, from and to the words of load_q_words, rounded to the io dtype as a separate
// rotation pass writing fp16 / bf16 would.  Four of the seven index bits (dims bits 0, 1, 5 and 6) are one product with a 16 x 16
// matrix of +-1 per four dims a lane: exact products, fp32 sums.  The other three lie in the eight accumulators of a lane.  What
// comes out has the queries across a row of four lanes, where the score products want them across the eight: movmatrix.
// About 110 instructions and no shuffle, against some 400 with 64 shuffles for a butterfly over the lanes, which every warp of a launch
// of few pages ran cold: us per launch in a graph, butterfly / now, 32 query and 8 KV heads: turbo4 1 x 4096 tokens 7.3 / 6.8,
// 4 x 1000 7.85 / 6.95, 8 x 2000 15.2 / 14.0; turbo3 1 x 4096 8.3 / 7.65, 16 x 2000 22.3 / 21.3.
template <bool BF16>
__device__ __forceinline__ void rotate_q_words_as(uint32_t (&w)[16], int lane) {
    const int gid = lane >> 2, tig = lane & 3;
    const uint32_t one = BF16 ? 0x3F803F80u : 0x3C003C00u;
    const uint32_t a = one ^ ((__popc(gid & (2 * tig)) & 1) << 15) ^ (static_cast<uint32_t>(__popc(gid & (2 * tig + 1))) << 31);
    float d[8][4];
#pragma unroll
    for (int s = 0; s < 8; ++s) mma_hadamard<BF16>(d[s], a, a ^ 0x80008000u, w[2 * s], w[2 * s + 1]);
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (!(s & h)) {
                butterfly2(d[s][0], d[s][1], d[s + h][0], d[s + h][1]);
                butterfly2(d[s][2], d[s][3], d[s + h][2], d[s + h][3]);
            }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float x = d[i >> 1][2 * (i & 1)] * kWhtScale, y = d[i >> 1][2 * (i & 1) + 1] * kWhtScale;
        uint32_t pair;
        if constexpr (BF16) {
            const __nv_bfloat162 r = __floats2bfloat162_rn(x, y);
            pair = *reinterpret_cast<const uint32_t*>(&r);
        } else {
            pair = pack_half2(x, y);
        }
        w[i] = movmatrix_trans(pair);
    }
}
__device__ __forceinline__ void rotate_q_words(uint32_t (&w)[16], int lane, int io_dtype) {
    if (io_dtype == TQ_DTYPE_F16) rotate_q_words_as<false>(w, lane);
    else rotate_q_words_as<true>(w, lane);
}
// The words as fp16, the operands of the score products.
__device__ __forceinline__ void q_words_to_half(uint32_t (&w)[16], int io_dtype) {
    if (io_dtype == TQ_DTYPE_F16) return;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 t = unpack_bf162(w[i]);
        w[i] = pack_half2(t.x, t.y);
    }
}

// Query operands of the sign term: half2 of the two dims of slot i times 2^(7 - i % 8); `correction` returns this lane's share of the
// query sum.
__device__ __forceinline__ void qp_frag_signed_from(const float (&x)[32], uint32_t (&f)[16], float& correction) {
    correction = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int lo = (i < 8 ? 4 : 12) + (i & 7), hi = (lo + 16) & 31;
        const float coef = static_cast<float>(1 << (7 - (i & 7)));
        f[i] = pack_half2(coef * x[lo], coef * x[hi]);
        correction += (x[lo] + x[hi]) * kSignUnit;
    }
}

// The coefficients, up to 128, take values of 512 and more out of fp16's range, and infinity times an absent sign is NaN.  A row that
// has such a value (511: it may round up) goes in divided by 256: with the smallest coefficient this rounds coordinates below 1/64 to
// multiples of 2^-16, 2^-25 of the largest one or less.  Returns the lanes of divided rows.  (The maximum as a tree: as a chain it
// costs a launch of few pages 0.1 us.)
__device__ __forceinline__ uint32_t fit_sign_rows(float (&x)[32], int lane) {
    float most[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) most[i] = fmaxf(fabsf(x[2 * i]), fabsf(x[2 * i + 1]));
#pragma unroll
    for (int h = 8; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) most[i] = fmaxf(most[i], most[i + h]);
    const uint32_t over = __ballot_sync(0xffffffffu, most[0] >= 511.f);
    if (!over) return 0;
    const bool row_over = (over >> (lane & 28)) & 15;
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] *= row_over ? 1.f / 256.f : 1.f;
    return __ballot_sync(0xffffffffu, row_over);
}
// What the sign sums of queries 2 tig, 2 tig + 1 are multiplied by then.
__device__ __forceinline__ float2 divided_by(uint32_t rows, int tig) {
    return make_float2((rows >> (8 * tig)) & 1 ? 256.f : 1.f, (rows >> (8 * tig + 4)) & 1 ? 256.f : 1.f);
}

// Shared-memory loads by 32-bit shared address + compile-time offset (one add per page and access pattern instead
// of 64-bit generic pointer arithmetic per load).
template <int OFF>
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}

template <int NW, int OFF>
__device__ __forceinline__ void lds_words(uint32_t addr, uint32_t (&w)[NW]) {
    if constexpr (NW == 4) {
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr), "n"(OFF));
    } else if constexpr (NW == 2) {
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr), "n"(OFF));
    } else {
        w[0] = lds_u32<OFF>(addr);
        if constexpr (NW > 1) w[1] = lds_u32<OFF + 4>(addr);
        if constexpr (NW > 2) w[2] = lds_u32<OFF + 8>(addr);
        if constexpr (NW > 3) w[3] = lds_u32<OFF + 12>(addr);
        if constexpr (NW > 4) w[4] = lds_u32<OFF + 16>(addr);
        static_assert(NW <= 5, "record has at most 4 index words and a sign word");
    }
}

// Output row of a query head from its weighted sum (lane: dims 4 lane .. 4 lane + 3) and denominator.
__device__ __forceinline__ void write_row(const DecodeParams& p, int64_t row, int lane, float (&x)[4], float l) {
    const float inv = 1.f / l;
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] *= inv;
    if (p.derotate_out) {   // two stages in the lane, five across lanes
        const float b0 = x[0] + x[1], b1 = x[0] - x[1], b2 = x[2] + x[3], b3 = x[2] - x[3];
        x[0] = b0 + b2; x[1] = b1 + b3; x[2] = b0 - b2; x[3] = b1 - b3;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const float sgn = (lane & m) ? -1.f : 1.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = fmaf(sgn, x[i], __shfl_xor_sync(0xffffffffu, x[i], m));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] *= kWhtScale;
    }
    uint2 w;
    if (p.io_dtype == TQ_DTYPE_F16) {
        w = make_uint2(pack_half2(x[0], x[1]), pack_half2(x[2], x[3]));
    } else {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(x[0], x[1]), hi = __floats2bfloat162_rn(x[2], x[3]);
        w = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.out) + row * kHeadDim + 4 * lane) = w;
}

template <int KB, int VB, bool QJL, bool SPARSE, int NSTAGE>
__global__ void __launch_bounds__(kThreads, TQ_DEC_MINBLOCKS) decode_partial_kernel(const DecodeParams p) {
    constexpr int NWK = KB + (QJL ? 1 : 0);
    constexpr int RK = 16 * NWK;
    constexpr int KN_OFF = 16 * RK;
    constexpr int KRN_OFF = KN_OFF + 32;
    constexpr int KPART = KN_OFF + 32 + (QJL ? 32 : 0);
    constexpr int VN_OFF = KPART + 256 * VB;
    constexpr int PAGE = KPART + 256 * VB + 32;

    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);                 // [kWarps][2 * NSTAGE]
    uint32_t* tabk = reinterpret_cast<uint32_t*>(smem + kBarBytes);     // pair table of the K codebook
    uint32_t* tabv = p.share_tables ? tabk : tabk + lut_bytes<KB>() / 4;
    uint8_t* ring = smem + kBarBytes + lut_bytes<KB>() + (p.share_tables ? 0 : lut_bytes<VB>());  // [kWarps][NSTAGE][PAGE]
    float* sm_o = reinterpret_cast<float*>(ring);                       // reused after the page loop
    __shared__ float sm_m[kWarps][8];
    __shared__ float sm_l[kWarps][8];

    // A launch of few pages is one chain of latencies, so nothing in it waits that need not: the length, the block-table
    // entries, the query and the codebooks are requested together, and the tables are filled behind the first pages' copies.
    // Entries past the length are fetched too (the table row is max_pages wide), and not looked at.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;
    const int chunk = blockIdx.x;
    const int kvh = blockIdx.y / p.ngroups, qg = blockIdx.y % p.ngroups;
    const int seq = blockIdx.z;
    uint64_t* mybar = bars + warp * 2 * NSTAGE;        // [0..NSTAGE) K (or whole page), [NSTAGE..) V
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < 2 * NSTAGE; ++s) mbar_init(mybar + s, 1);
        fence_barrier_init();
    }
    pdl_wait();
    pdl_release();
    const int L = p.seq_lens[seq];
    const int p0 = chunk * p.chunk_pages;
    const int32_t* bt = p.block_tables + static_cast<int64_t>(seq) * p.bt_stride;
    int32_t bt_first = 0;                               // entry of this warp's page `lane`
    {
        const int pg = p0 + warp + kWarps * lane;
        if (pg < min(p0 + p.chunk_pages, p.max_pages)) bt_first = __ldg(bt + (pg >> p.sub_shift));
    }
    // A length beyond what the block table and the workspace were sized for is cut to that size and flagged:
    // the walk never leaves the table row and a chunk index never leaves the workspace.
    const bool too_long = pages_of_length(L) > p.max_pages;
    const int npages = min(pages_of_length(L), p.max_pages);
    const int g_in_group = qg * 8 + gid;                // query index inside the GQA group
    const int nq = min(8, p.G - qg * 8);                // live query heads in this CTA
    const int head0 = kvh * p.G + qg * 8;
    const float ck = lane_centroid<KB>(p.kc, lane), cv = lane_centroid<VB>(p.vc, lane);
    uint32_t qf[16];
    load_q_words(p.q, (static_cast<int64_t>(seq) * p.Hq + head0 + gid) * kHeadDim, tig, g_in_group < p.G, qf);

    if (L <= 0) {
        if (chunk == 0) {  // zeros for empty sequences
            for (int i = threadIdx.x; i < nq * kHeadDim; i += kThreads) {
                const int64_t o = (static_cast<int64_t>(seq) * p.Hq + head0 + i / kHeadDim) * kHeadDim + i % kHeadDim;
                static_cast<uint16_t*>(p.out)[o] = 0;
            }
        }
        return;
    }
    if (p0 >= npages) return;
    const int p1 = min(p0 + p.chunk_pages, npages);
    const int n_my = (p0 + warp < p1) ? (p1 - p0 - warp + kWarps - 1) / kWarps : 0;

    uint8_t* myring = ring + warp * NSTAGE * PAGE;
    __syncwarp();

    // ---- block-table window: lane l holds the entry of this warp's page jbase + l ---
    int jbase = 0;
    int32_t btreg = 0;
    bool bad_block = false;
    auto take_bt = [&](int jb, int32_t b) {
        jbase = jb;
        if (jb + lane >= n_my) {
            b = 0;
        } else if (b < 0 || b >= p.num_blocks) {
            bad_block = true;
            b = 0;
        }
        btreg = b;
    };
    auto load_bt = [&](int jb) {
        const int j = jb + lane;
        take_bt(jb, j < n_my ? __ldg(bt + ((p0 + warp + kWarps * j) >> p.sub_shift)) : 0);
    };
    const uint8_t* head_base = p.cache + (static_cast<int64_t>(kvh) << p.sub_shift) * PAGE;
    auto page_src = [&](int j) -> const uint8_t* {
        const int32_t blk = __shfl_sync(0xffffffffu, btreg, j - jbase);
        const int pg = p0 + warp + kWarps * j;
        const int sub = pg & ((1 << p.sub_shift) - 1);
        return head_base + static_cast<int64_t>(blk) * p.block_stride + sub * PAGE;
    };
    // Dense mode: one copy of the whole page.  Sparse mode: K part now, V part on demand.
    // whole = K and V parts in one copy (always in dense mode; in sparse mode when the V part is expected to be needed)
    auto issue_k = [&](int j, bool whole = true) {
        const uint8_t* src = page_src(j);
        const int s = j % NSTAGE;
        if (lane == 0) {
            const uint32_t bytes = (SPARSE && !whole) ? KPART : PAGE;
            mbar_expect_tx(mybar + s, bytes);
            bulk_g2s(myring + s * PAGE, src, bytes, mybar + s);
        }
    };
    auto issue_v = [&](int j) {
        const uint8_t* src = page_src(j);
        const int s = j % NSTAGE;
        if (lane == 0) {
            mbar_expect_tx(mybar + NSTAGE + s, PAGE - KPART);
            bulk_g2s(myring + s * PAGE + KPART, src + KPART, PAGE - KPART, mybar + NSTAGE + s);
        }
    };

    // The first pages are requested before the tables and the query fragments are made, which hide part of their latency.
    if (n_my > 0) take_bt(0, bt_first);
#pragma unroll
    for (int j = 0; j < NSTAGE; ++j)
        if (j < n_my) issue_k(j);
    fill_pair_lut<KB>(tabk, ck, warp, lane);
    if (!p.share_tables) fill_pair_lut<VB>(tabv, cv, warp, lane);

    __syncthreads();   // the pair tables are there; the query's operands are made while the first pages are under way
    // ---- query fragments -------------------------------------------------------------------------------
    uint32_t qpf[QJL ? 16 : 1];
    float sq_init0 = 0.f, sq_init1 = 0.f;   // minus the query sums of the one-sided sign forms
    float qpscale0 = 0.f, qpscale1 = 0.f;   // of queries 2 tig, 2 tig + 1
    {
        if (p.rotate_q) rotate_q_words(qf, lane, p.io_dtype);
        if constexpr (QJL) {
            float xq[32], corr;
            if (p.qp) {   // S q' given separately
                load_q_words(p.qp, (static_cast<int64_t>(seq) * p.Hq + head0 + gid) * kHeadDim, tig, g_in_group < p.G, qpf);
                unpack_q(qpf, p.io_dtype, xq);
            } else {
                unpack_q(qf, p.io_dtype, xq);
            }
            const float2 by = divided_by(fit_sign_rows(xq, lane), tig);
            qpscale0 = by.x * p.qpscale;
            qpscale1 = by.y * p.qpscale;
            qp_frag_signed_from(xq, qpf, corr);
            corr += __shfl_xor_sync(0xffffffffu, corr, 1);
            corr += __shfl_xor_sync(0xffffffffu, corr, 2);      // total over the 128 dims of query gid
            sq_init0 = -__shfl_sync(0xffffffffu, corr, 8 * tig);       // query 2 * tig lives on lanes 8 * tig ..
            sq_init1 = -__shfl_sync(0xffffffffu, corr, 8 * tig + 4);   // query 2 * tig + 1
        }
        q_words_to_half(qf, p.io_dtype);
    }

    const uint32_t klut = smem_u32(tabk) + (KB == 2 ? 8 * (lane & 15) : 4 * lane);
    const uint32_t vlut = smem_u32(tabv) + (VB == 2 ? 8 * (lane & 15) : 4 * lane);
    // this lane's three access patterns inside a ring stage: its two K records, the norm slots, the V words
    const uint32_t ring_k = smem_u32(myring) + lane * (NWK * 4);
    const uint32_t ring_n = smem_u32(myring) + gid * 4;
    const uint32_t ring_v = smem_u32(myring) + (tig * 8 + gid) * 4;
    // ---- online-softmax state ---------------------------------------------------------
    float m0 = -INFINITY, m1 = -INFINITY;   // running max for queries 2*tig, 2*tig+1 (log2 domain)
    float l0 = 0.f, l1 = 0.f;               // this lane's share of the denominators
    float oacc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int r = 0; r < 4; ++r) oacc[i][r] = 0.f;
    bool timed_out = false;
    // Sparse-V: a group of fewer than eight heads leaves columns of zero queries, whose scores are all alike; they decide nothing.
    const float thresh0 = 2 * tig < nq ? p.log2_thresh : INFINITY, thresh1 = 2 * tig + 1 < nq ? p.log2_thresh : INFINITY;
    uint32_t v_skipped = 0;
    uint32_t v_parity = 0;                  // bit s: phase of the V barrier of stage s (sparse mode)
    int j_stop = n_my;
    uint32_t v_with_k = (1u << NSTAGE) - 1u;  // sparse mode, bit s: the page in stage s brought its V part along (the first pages do)

    auto wait_v = [&](int j) -> bool {
        const int s = j % NSTAGE;
        const bool ok = mbar_wait_bounded(mybar + NSTAGE + s, (v_parity >> s) & 1u);
        v_parity ^= 1u << s;
        return ok;
    };
    // O += P V for page j (already resident in its ring stage); weights are relative to the running maximum.
    auto accumulate_v = [&](int j, float w0, float w1, float w2, float w3, int valid_tokens) {
        const uint32_t stage = (j % NSTAGE) * PAGE;
        const bool va = gid < valid_tokens, vb = gid + 8 < valid_tokens;
        const float2 vn = unpack_half2(lds_u32<VN_OFF>(ring_n + stage));
        const uint32_t vaddr = ring_v + stage;
        const uint32_t pr0 = pack_half2(va ? w0 * vn.x : 0.f, va ? w1 * vn.x : 0.f);
        const uint32_t pr1 = pack_half2(vb ? w2 * vn.y : 0.f, vb ? w3 * vn.y : 0.f);
        const uint32_t t[2] = {movmatrix_trans(pr0), movmatrix_trans(pr1)};
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const uint32_t vo = vaddr + o * 128;
            const uint32_t pa0 = t[o] & 0xffffu, pa1 = t[o] << 16, pa2 = t[o] >> 16, pa3 = t[o] & 0xffff0000u;
            uint32_t pw[VB];
#pragma unroll
            for (int i = 0; i < VB; ++i)
                pw[i] = i == 0 ? lds_u32<KPART>(vo) : (i == 1 ? lds_u32<KPART + 256>(vo) : (i == 2 ? lds_u32<KPART + 512>(vo) : lds_u32<KPART + 768>(vo)));
            if constexpr (VB == 2) {
                // byte k of packed word jw: the pairs of group u = 2 jw (first half2) and u = 2 jw + 1 (second)
#pragma unroll
                for (int jw = 0; jw < 2; ++jw) {
                    const uint2 a0 = lut_quad(vlut, pw[jw], 0), a1 = lut_quad(vlut, pw[jw], 1);
                    const uint2 b0 = lut_quad(vlut, pw[jw], 2), b1 = lut_quad(vlut, pw[jw], 3);
                    mma_f16_16816(oacc[4 * jw], pa0, pa1, pa2, pa3, a0.x, b0.x);
                    mma_f16_16816(oacc[4 * jw + 1], pa0, pa1, pa2, pa3, a1.x, b1.x);
                    mma_f16_16816(oacc[4 * jw + 2], pa0, pa1, pa2, pa3, a0.y, b0.y);
                    mma_f16_16816(oacc[4 * jw + 3], pa0, pa1, pa2, pa3, a1.y, b1.y);
                }
            } else {
                uint32_t mv[4];
                masked_words<VB>(pw, mv);   // bytes 0,1: token a (dims 4u..4u+3), bytes 2,3: token b
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t a0 = lut_pair(vlut, mv[u], 0), a1 = lut_pair(vlut, mv[u], 1);
                    const uint32_t b0 = lut_pair(vlut, mv[u], 2), b1 = lut_pair(vlut, mv[u], 3);
                    mma_f16_16816(oacc[2 * u], pa0, pa1, pa2, pa3, a0, b0);
                    mma_f16_16816(oacc[2 * u + 1], pa0, pa1, pa2, pa3, a1, b1);
                }
            }
        }
    };

    for (int j = 0; j < n_my; ++j) {
        if constexpr (SPARSE) {
            if ((v_with_k >> (j % NSTAGE)) & 1u) {
#define TQ_PAGE_HAVE_V 1
#include "tq_decode_page.inc"
#undef TQ_PAGE_HAVE_V
            } else {
#define TQ_PAGE_HAVE_V 0
#include "tq_decode_page.inc"
#undef TQ_PAGE_HAVE_V
            }
        } else {
#define TQ_PAGE_HAVE_V 1
#include "tq_decode_page.inc"
#undef TQ_PAGE_HAVE_V
        }
    }
    if (timed_out) {
        // Give copies that were already issued a bounded chance to land before the ring is reused.
        for (int j = j_stop + 1; j < min(n_my, j_stop + NSTAGE); ++j)
            (void)mbar_wait_bounded(mybar + j % NSTAGE, (j / NSTAGE) & 1);
    }

    if (p.status) {
        int bits = 0;
        if (__any_sync(0xffffffffu, bad_block) || too_long) bits |= TQ_STATUS_BAD_BLOCK;
        if (__any_sync(0xffffffffu, timed_out)) bits |= TQ_STATUS_TIMEOUT;
        if (bits && lane == 0) atomicOr(p.status, bits);
    }
    if constexpr (SPARSE) {
        if (p.skip_stats && lane == 0) {
            atomicAdd(p.skip_stats, static_cast<uint32_t>(j_stop));   // pages this warp visited
            atomicAdd(p.skip_stats + 1, v_skipped);
        }
    }

    // ---- merge the 4 warps --------------------------------------------------------------
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, o);
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    __syncthreads();  // every warp is done with its ring; it becomes the merge buffer
    if (gid == 0) {
        sm_m[warp][2 * tig] = m0;
        sm_m[warp][2 * tig + 1] = m1;
        sm_l[warp][2 * tig] = l0;
        sm_l[warp][2 * tig + 1] = l1;
    }
    {
        float* row = sm_o + (warp * 8 + gid) * kOPad;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int dim = 16 * (2 * tig + (r & 1)) + 2 * nt + (r >> 1);
                row[dim + (dim >> 5)] = oacc[nt][r];
            }
    }
    __syncthreads();
    // a warp combines the four partials of query rows warp, warp + 4; a lane holds four dims
    const int nchunks = (npages + p.chunk_pages - 1) / p.chunk_pages;
    for (int g = warp; g < nq; g += kWarps) {
        float M = sm_m[0][g];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) M = fmaxf(M, sm_m[w][g]);
        float l = 0.f, x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float sc = ex2(sm_m[w][g] - M);
            const float* o = sm_o + (w * 8 + g) * kOPad + 4 * lane + (lane >> 3);   // dims d sit at d + d / 32
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = fmaf(sc, o[i], x[i]);
            l = fmaf(sc, sm_l[w][g], l);
        }
        if (nchunks == 1) {
            write_row(p, static_cast<int64_t>(seq) * p.Hq + head0 + g, lane, x, l);
        } else {
            const int64_t slot = ((static_cast<int64_t>(seq) * p.Hkv * p.ngroups + blockIdx.y) * p.max_chunks + chunk) * 8 + g;
            *reinterpret_cast<float4*>(p.ws_o + slot * kHeadDim + 4 * lane) = make_float4(x[0], x[1], x[2], x[3]);
            if (lane == 0) reinterpret_cast<float2*>(p.ws_ml)[slot] = make_float2(M, l);
        }
    }
}

// Weighted combination of partial rows by one warp: part(i) is the 128 sums of part i (fp32), ml(i) its (maximum,
// denominator).  Eight parts are fetched at a time, independently of one another and of the maxima: what a merge costs is the
// latency of its chain of loads.  The first eight are fetched up to part `room`, before `parts` has to be known.
template <typename Part, typename Ml>
__device__ __forceinline__ void merge_parts(int first, int step, int parts, int room, int lane, Part part, Ml ml, float& M, float (&x)[4], float& l) {
    M = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = 0.f;
    constexpr int kAtOnce = 8;
    float4 v[kAtOnce];
    float2 w[kAtOnce];
    auto fetch = [&](int i0, int end) {
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) {
            const int i = i0 + k * step;
            if (i < end) {
                w[k] = ml(i);
                v[k] = *reinterpret_cast<const float4*>(part(i) + 4 * lane);
            }
        }
    };
    fetch(first, room);
    for (int i0 = first; i0 < parts;) {
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k)
            if (i0 + k * step >= parts) {
                w[k] = make_float2(-INFINITY, 0.f);
                v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        float m = M;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) m = fmaxf(m, w[k].x);
        const float old = ex2(M - m);
        l *= old;
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] *= old;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) {
            const float sc = ex2(w[k].x - m);
            l = fmaf(sc, w[k].y, l);
            x[0] = fmaf(sc, v[k].x, x[0]);
            x[1] = fmaf(sc, v[k].y, x[1]);
            x[2] = fmaf(sc, v[k].z, x[2]);
            x[3] = fmaf(sc, v[k].w, x[3]);
        }
        M = m;
        i0 += kAtOnce * step;
        if (i0 < parts) fetch(i0, parts);
    }
}

// One block per query head; its four warps share the chunks.
constexpr int kChunkMergeWarps = 4;
__global__ void __launch_bounds__(kChunkMergeWarps * 32) decode_merge_kernel(const DecodeParams p) {
    __shared__ float4 so[kChunkMergeWarps][32];
    __shared__ float2 sml[kChunkMergeWarps];
    pdl_release();
    pdl_wait();
    const int head = blockIdx.x, seq = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int npages = min(pages_of_length(p.seq_lens[seq]), p.max_pages);   // same cut as the partial kernel
    const int nchunks = (npages + p.chunk_pages - 1) / p.chunk_pages;
    const int kvh = head / p.G, gi = head % p.G;
    const int by = kvh * p.ngroups + gi / 8, g = gi % 8;
    const int64_t base = (static_cast<int64_t>(seq) * p.Hkv * p.ngroups + by) * p.max_chunks;
    float M, l, x[4];
    merge_parts(warp, kChunkMergeWarps, nchunks, p.max_chunks, lane, [&](int c) { return p.ws_o + ((base + c) * 8 + g) * kHeadDim; },
                [&](int c) { return reinterpret_cast<const float2*>(p.ws_ml)[(base + c) * 8 + g]; }, M, x, l);
    if (nchunks <= 1) return;  // written by the partial kernel
    so[warp][lane] = make_float4(x[0], x[1], x[2], x[3]);
    if (lane == 0) sml[warp] = make_float2(M, l);
    __syncthreads();
    if (warp != 0) return;
    float Ma = sml[0].x;
#pragma unroll
    for (int w = 1; w < kChunkMergeWarps; ++w) Ma = fmaxf(Ma, sml[w].x);
    l = 0.f;
    x[0] = x[1] = x[2] = x[3] = 0.f;
#pragma unroll
    for (int w = 0; w < kChunkMergeWarps; ++w) {
        const float sc = ex2(sml[w].x - Ma);
        const float4 v = so[w][lane];
        l = fmaf(sc, sml[w].y, l);
        x[0] = fmaf(sc, v.x, x[0]);
        x[1] = fmaf(sc, v.y, x[1]);
        x[2] = fmaf(sc, v.z, x[2]);
        x[3] = fmaf(sc, v.w, x[3]);
    }
    write_row(p, static_cast<int64_t>(seq) * p.Hq + head, lane, x, l);
}

template <int KB, int VB, bool QJL, bool SPARSE>
int launch_partial(const DecodeParams& p, dim3 grid, cudaStream_t stream) {
    constexpr int PAGE = page_bytes(KB, VB, QJL ? 1 : 0);
    constexpr size_t smem_max = kBarBytes + lut_bytes<KB>() + lut_bytes<VB>() + static_cast<size_t>(kWarps) * kStages * PAGE;
    const size_t smem = smem_max - (p.share_tables ? lut_bytes<VB>() : 0);
    static_assert(static_cast<size_t>(kWarps) * kStages * PAGE >= sizeof(float) * kWarps * 8 * kOPad,
                  "ring must hold the merge buffer");
    auto kern = decode_partial_kernel<KB, VB, QJL, SPARSE, kStages>;
    // The opt-in shared-memory size is a per-device function attribute; set once per device.
    static bool configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TQ_ERR_LAUNCH;
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_max)) != cudaSuccess)
            return TQ_ERR_LAUNCH;
        configured[dev] = true;
    }
    return launch_chained(kern, grid, dim3(kThreads), smem, stream, p) == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
}

}  // namespace
}  // namespace tq

#include "tq_decode_stream.cuh"
#include "tq_decode_umma.cuh"

namespace tq {
namespace {

// What a call runs: the chunked kernel on `grid`, or, with `stream` set, the persistent kernel.
struct Plan {
    dim3 grid;
    const StreamParams* stream;
    bool qjl, sparse;
};

template <int KB, int VB, bool QJL, bool SPARSE>
int launch_planned(const DecodeParams& p, const Plan& plan, cudaStream_t stream) {
    return plan.stream ? launch_stream<KB, VB, QJL, SPARSE>(*plan.stream, stream) : launch_partial<KB, VB, QJL, SPARSE>(p, plan.grid, stream);
}

template <int KB, int VB>
int dispatch_flags(const DecodeParams& p, const Plan& plan, cudaStream_t stream) {
    if constexpr (KB <= 3 && VB <= 3) {
        // on request (TQ_IO_TCGEN05): the tensor-memory kernel, for 2- and 3-bit codebooks without the Sparse-V skip
        if (!plan.sparse && p.use_tcgen05)
            return plan.qjl ? launch_umma<KB, VB, true>(p, plan.grid, stream) : launch_umma<KB, VB, false>(p, plan.grid, stream);
    }
    if (plan.qjl) return plan.sparse ? launch_planned<KB, VB, true, true>(p, plan, stream) : launch_planned<KB, VB, true, false>(p, plan, stream);
    return plan.sparse ? launch_planned<KB, VB, false, true>(p, plan, stream) : launch_planned<KB, VB, false, false>(p, plan, stream);
}

template <int KB>
int dispatch_v(const DecodeParams& p, int vb, const Plan& plan, cudaStream_t stream) {
    switch (vb) {
#ifndef TQ_DEC_QUICK
        case 2: return dispatch_flags<KB, 2>(p, plan, stream);
        case 4: return dispatch_flags<KB, 4>(p, plan, stream);
#endif
        case 3: return dispatch_flags<KB, 3>(p, plan, stream);
    }
    return TQ_ERR_UNSUPPORTED;
}

// Which kernel is the better one, by the pages that the batch can have at most: the table's width (or the longest length, where the
// caller names it), for the lengths are on the device.  The persistent kernel pays 8 to 9 us however few pages there are (all its tables,
// one more level of merging), the chunked one 5 to 7, but it takes 0.4 (4-bit) to 0.5 us (with sign term) per 1000 pages where the chunked
// one takes 0.7 to 0.8; sequences of few pages cost it more, a warp then changes item every few pages.  us per launch in a graph over
// caches that L2 does not hold, rotated queries, 32 query and 8 KV heads, tables as wide as the sequences are long, chunked / persistent,
// turbo4 and turbo3: 1 x 16384 tokens (8192 pages) 14.5 / 15.6 and 13.7 / 16.5, 32 x 512 14.5 / 14.6 and 13.8 / 15.6; 64 x 512 (16384)
// 18.8 / 18.8 and 18.4 / 20.6, 32 x 1024 20.9 / 19.0 and 20.6 / 20.7; 64 x 640 (20480) 21.9 / 21.1 and 21.9 / 23.0.
// The lines do not look at the format, nor at how long the sequences in the table are.  What that costs, for 28 x 1024 tokens (14336 pages) and
// for 28 sequences of 512 and of 100 tokens in tables for 1024:
//   turbo4            20.4 / 18.6   14.6 / 14.6   7.8 / 11.0
//   turbo4 Sparse-V   21.6 / 18.4   15.2 / 14.5   8.1 / 11.0
//   turbo3            20.6 / 20.4   20.1 / 15.5   9.0 / 11.6
//   turbo2            19.6 / 19.2   18.3 / 15.2   9.3 / 11.6
//   K 4, V 3 bits     21.8 / 18.2   13.2 / 14.3   7.7 / 10.9
// (turbo4 27 x 1024, whose 432 chunks run three to an SM in one wave: 14.8 / 17.8.)  A rule that sent more than 444 chunks of 12288 pages or
// more to the persistent kernel took 2 to 4 us from nearly empty tables, such as a captured step of few requests has, and was taken back; from
// 16384 pages on they lose as much (1 sequence of 100 tokens in a table for 32768: 5.8 / 10.1 and 6.1 / 10.6).
constexpr int64_t kStreamMinPages = 16384;
constexpr int64_t kStreamSlots = static_cast<int64_t>(kStreamCtas) * (kStreamWarps + 2);   // partials of warps and of CTAs
int64_t pages_at_most(int64_t ns, int64_t hq, int64_t hkv, int64_t max_pages) { return ns * max_pages * hkv * ((hq / hkv + 7) / 8); }
bool stream_is_better(int64_t pages, int64_t cache_pages, int max_pages) {
    if (pages < kStreamMinPages || pages > INT32_MAX || cache_pages > UINT32_MAX) return false;
    return pages >= 32768 || max_pages >= 64;
}
// Workspace of the persistent kernel, or 0 where no call takes it.
int64_t stream_bytes(int64_t pages, int64_t cache_pages, int max_pages) {
    if (!stream_is_better(pages, cache_pages, max_pages)) return 0;
    return kStreamSlots * (kStreamSlotFloats + 16) * static_cast<int64_t>(sizeof(float)) + kStreamCtas * static_cast<int64_t>(sizeof(int4));
}

}  // namespace
}  // namespace tq

using namespace tq;

extern "C" int tq_decode_auto_chunk_pages(int num_seqs, int num_kv_heads, int num_q_heads, int max_pages_per_seq) {
    if (num_seqs <= 0 || num_kv_heads <= 0 || num_q_heads <= 0 || max_pages_per_seq <= 0) return TQ_ERR_ARG;
    if (num_q_heads % num_kv_heads) return TQ_ERR_ARG;   // also num_q_heads < num_kv_heads: no query group
    // Sizes come from the longest sequence; chunks beyond a shorter sequence's end exit at once.
    // Measured on batch 64 x 8192 tokens with 1, 2, 4 and 8 KV heads per GPU (chunk sizes 32..512 pages):
    //  * about 1024 CTAs (1.7 waves of 148 SMs x 4 CTAs) is the flat optimum, with a power-of-two number
    //    of chunks so that all chunks of a sequence are alike (64-page chunks for 1-2 heads, 128 for 4,
    //    128..256 for 8); uneven splits such as 57 or 74 pages lose 5-10 %;
    //  * a CTA keeps >= 64 pages (16 per warp) so that its prologue (lookup-table fill, query fragments,
    //    first copies) stays amortised, unless that leaves the GPU less than half full (small batches):
    //    then chunks shrink down to 16 pages (see below);
    //  * at most 256 pages per CTA bound the longest CTA when sequence lengths are skewed.
    const int G = num_q_heads / num_kv_heads;
    const int ngroups = (G + 7) / 8;
    const long long pairs = 1LL * num_seqs * num_kv_heads * ngroups;
    const long long slots = 148LL * 4;
    auto ceil_div = [](long long a, long long b) { return (a + b - 1) / b; };
    long long chunks = 1;
    while (pairs * chunks * 2 <= 1024 + pairs * chunks / 2) chunks *= 2;   // power of two nearest to 1024 / pairs
    long long max_big = max_pages_per_seq / 64;
    if (max_big < 1) max_big = 1;
    while (chunks > max_big) chunks /= 2;
    if (chunks < 1) chunks = 1;
    if (pairs * chunks < slots / 2) {
        // Small batches: the smallest power-of-two chunk (>= 16 pages) that keeps the grid within the resident slots.
        // Measured on 1, 2 and 4 sequences of 32768, 16384 and 8192 tokens (8 KV heads): 32-page chunks (512 CTAs)
        // 32.8 / 27.8 / 25.3 us against 35.2 / 32.0 / 30.0 us for the 27-28 pages that fill every slot: the warps of a
        // CTA share a chunk evenly only when it is a multiple of 4 pages, and every extra CTA pays its set-up.
        long long most = slots / pairs;
        if (most < 1) most = 1;
        long long cp = 16;
        while (cp < ceil_div(max_pages_per_seq, most)) cp *= 2;
        if (cp > max_pages_per_seq) cp = max_pages_per_seq;
        return static_cast<int>(cp > 256 ? 256 : cp);
    }
    // Fewer CTAs than resident slots (a GPU that holds one or two KV heads of a sharded batch): an uneven chunk count
    // that fills the slots beats the power of two (64 sequence-heads: 9 chunks of 57 pages = 576 CTAs measured 37.7 us
    // against 39.5 us for 8 x 64), as long as chunks stay >= 32 pages.
    if (pairs * chunks <= slots) {
        const long long fill = slots / pairs;
        if (fill > chunks && max_pages_per_seq / fill >= 32) chunks = fill;
    }
    long long cp = ceil_div(max_pages_per_seq, chunks);
    if (cp > 256) cp = 256;
    return static_cast<int>(cp);
}

extern "C" int64_t tq_decode_workspace_bytes(int num_seqs, int num_q_heads, int num_kv_heads, int max_pages_per_seq,
                                             int chunk_pages) {
    if (num_seqs <= 0 || num_kv_heads <= 0 || num_q_heads <= 0 || max_pages_per_seq <= 0) return TQ_ERR_ARG;
    if (num_q_heads % num_kv_heads) return TQ_ERR_ARG;
    if (chunk_pages <= 0) chunk_pages = tq_decode_auto_chunk_pages(num_seqs, num_kv_heads, num_q_heads, max_pages_per_seq);
    const int G = num_q_heads / num_kv_heads;
    const int ngroups = (G + 7) / 8;
    const int64_t max_chunks = (max_pages_per_seq + chunk_pages - 1) / chunk_pages;
    const int64_t slots = static_cast<int64_t>(num_seqs) * num_kv_heads * ngroups * max_chunks * 8;
    return slots * (kHeadDim + 2) * static_cast<int64_t>(sizeof(float));
}

extern "C" int64_t tq_decode_auto_workspace_bytes(int num_seqs, int num_q_heads, int num_kv_heads, int max_pages_per_seq) {
    const int64_t chunked = tq_decode_workspace_bytes(num_seqs, num_q_heads, num_kv_heads, max_pages_per_seq, 0);
    if (chunked < 0) return chunked;
    const int64_t pages = pages_at_most(num_seqs, num_q_heads, num_kv_heads, max_pages_per_seq);
    // (a cache of too many pages for the persistent kernel is not known here: such a call has the larger workspace and does without)
    const int64_t stream = stream_bytes(pages, 0, max_pages_per_seq);
    return stream > chunked ? stream : chunked;
}

extern "C" int tq_decode_paged(void* out, const void* q_rot, const void* q_proj, int io_dtype, const void* cache,
                               int64_t num_blocks, int block_size, const int32_t* block_tables, int64_t bt_stride,
                               const int32_t* seq_lens, const float* k_centroids, const float* v_centroids,
                               float sm_scale, float corr_scale, float sparse_thresh, void* workspace,
                               int64_t workspace_bytes, int32_t* status, uint32_t* skip_stats, int num_seqs,
                               int num_q_heads, int num_kv_heads, int max_pages_per_seq, int k_bits, int v_bits,
                               int use_qjl, int chunk_pages, tq_stream_t stream) {
    if (num_seqs == 0) return TQ_OK;
    if (!out || !q_rot || !cache || !block_tables || !seq_lens || !k_centroids || !v_centroids) return TQ_ERR_ARG;
    if (num_seqs < 0 || num_q_heads <= 0 || num_kv_heads <= 0 || max_pages_per_seq <= 0 || num_blocks <= 0) return TQ_ERR_ARG;
    if (num_q_heads % num_kv_heads) return TQ_ERR_ARG;
    const int rotate_q = (io_dtype & TQ_IO_ROTATE_Q) ? 1 : 0, derotate_out = (io_dtype & TQ_IO_DEROTATE_OUT) ? 1 : 0;
    const int use_tcgen05 = (io_dtype & TQ_IO_TCGEN05) ? 1 : 0;
    io_dtype &= 0xff;
    if (io_dtype != TQ_DTYPE_F16 && io_dtype != TQ_DTYPE_BF16) return TQ_ERR_UNSUPPORTED;
    if (rotate_q && q_proj) return TQ_ERR_ARG;   // S q' cannot be derived from an unrotated query
    if (block_size < kPageTokens || (block_size & (block_size - 1))) return TQ_ERR_UNSUPPORTED;  // 16, 32, 64, ...
    if (k_bits < 2 || k_bits > 4 || v_bits < 2 || v_bits > 4) return TQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(q_rot) | reinterpret_cast<uintptr_t>(out) |
         reinterpret_cast<uintptr_t>(q_proj)) & 15)
        return TQ_ERR_ARG;
    // The persistent kernel takes the calls that leave the split to the library and bring the workspace for it.
    const bool tensor_memory = use_tcgen05 && k_bits <= 3 && v_bits <= 3 && !(sparse_thresh > 0.f);
    const int64_t pages = pages_at_most(num_seqs, num_q_heads, num_kv_heads, max_pages_per_seq);
    const int64_t cache_pages = num_blocks * num_kv_heads * (block_size / kPageTokens);
    const int64_t stream_need = chunk_pages <= 0 && !tensor_memory ? stream_bytes(pages, cache_pages, max_pages_per_seq) : 0;
    const bool persistent = stream_need > 0 && workspace && workspace_bytes >= stream_need && !(reinterpret_cast<uintptr_t>(workspace) & 15);
    if (chunk_pages <= 0) chunk_pages = tq_decode_auto_chunk_pages(num_seqs, num_kv_heads, num_q_heads, max_pages_per_seq);
    const int64_t need = tq_decode_workspace_bytes(num_seqs, num_q_heads, num_kv_heads, max_pages_per_seq, chunk_pages);
    const int max_chunks = (max_pages_per_seq + chunk_pages - 1) / chunk_pages;
    if (!persistent && max_chunks > 1 && (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 15)))
        return TQ_ERR_WORKSPACE;
    if (num_seqs > 65535 || max_chunks > 65535) return TQ_ERR_UNSUPPORTED;

    DecodeParams p;
    p.out = out;
    p.q = q_rot;
    p.qp = q_proj;
    p.cache = static_cast<const uint8_t*>(cache);
    p.block_tables = block_tables;
    p.seq_lens = seq_lens;
    p.kc = k_centroids;
    p.vc = v_centroids;
    p.G = num_q_heads / num_kv_heads;
    p.ngroups = (p.G + 7) / 8;
    const int64_t slots = static_cast<int64_t>(num_seqs) * num_kv_heads * p.ngroups * max_chunks * 8;
    p.ws_o = static_cast<float*>(workspace);
    p.ws_ml = p.ws_o ? p.ws_o + slots * kHeadDim : nullptr;
    p.status = status;
    p.skip_stats = skip_stats;
    p.bt_stride = bt_stride;
    p.num_blocks = num_blocks;
    p.qscale = sm_scale * kLog2e;
    p.qpscale = sm_scale * corr_scale * kLog2e / kSignUnit;   // what the sign sums count in
    p.log2_thresh = sparse_thresh > 0.f ? log2f(sparse_thresh) : -INFINITY;
    p.Hq = num_q_heads;
    p.Hkv = num_kv_heads;
    p.sub_shift = 0;
    while ((kPageTokens << p.sub_shift) < block_size) ++p.sub_shift;
    p.block_stride = static_cast<int64_t>(num_kv_heads) * (block_size / kPageTokens) *
                     page_bytes(k_bits, v_bits, use_qjl ? 1 : 0);
    p.chunk_pages = chunk_pages;
    p.max_chunks = max_chunks;
    p.max_pages = max_pages_per_seq;
    p.io_dtype = io_dtype;
    p.rotate_q = rotate_q;
    p.derotate_out = derotate_out;
    p.use_tcgen05 = use_tcgen05;
    p.share_tables = (k_bits == v_bits && k_centroids == v_centroids) ? 1 : 0;

    StreamParams sp;
    if (persistent) {
        sp.d = p;
        sp.ns = num_seqs;
        sp.HG = num_kv_heads * p.ngroups;
        sp.weight_thresh = sparse_thresh > 0.f ? 0.5f * sparse_thresh : 0.f;
        sp.two12 = 1u << 12;
        sp.two20 = 1u << 20;
        sp.n_warps = kStreamCtas * kStreamWarps;
        sp.part_o = static_cast<float*>(workspace);
        sp.part_ml = reinterpret_cast<float2*>(sp.part_o + kStreamSlots * kStreamSlotFloats);
        sp.split = reinterpret_cast<int4*>(sp.part_ml + kStreamSlots * 8);
    }
    const Plan plan = {dim3(max_chunks, num_kv_heads * p.ngroups, num_seqs), persistent ? &sp : nullptr, use_qjl != 0, sparse_thresh > 0.f};
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int rc;
    switch (k_bits) {
#ifndef TQ_DEC_QUICK
        case 2: rc = dispatch_v<2>(p, v_bits, plan, st); break;
        case 4: rc = dispatch_v<4>(p, v_bits, plan, st); break;
#endif
        case 3: rc = dispatch_v<3>(p, v_bits, plan, st); break;
        default: return TQ_ERR_UNSUPPORTED;
    }
    if (rc != TQ_OK) return rc;
    if (persistent) {
        if (launch_chained(decode_stream_merge_kernel, dim3(kStreamCtas), dim3(kStreamMergeWarps * 32), 0, st, sp) != cudaSuccess)
            return TQ_ERR_LAUNCH;
    } else if (max_chunks > 1) {
        if (launch_chained(decode_merge_kernel, dim3(num_q_heads, num_seqs), dim3(kChunkMergeWarps * 32), 0, st, p) != cudaSuccess)
            return TQ_ERR_LAUNCH;
    }
    return TQ_OK;
}

// ---------------------------------------------------------------------------------------------
// Decode without a caller-provided workspace.
//
// Some hosts of this library have no way to obtain device memory of their own: an inference
// server that hands every free byte of HBM to its KV-cache pool at start-up (a later cudaMalloc
// simply fails), or a binding in a runtime that only forwards pointers it was given and owns no
// device allocator.  For them the split-K scratch lives in a fixed array inside the library image,
// reserved on every GPU that loads the library for as long as the process runs.
// ---------------------------------------------------------------------------------------------
namespace tq {
namespace {

constexpr size_t kStaticScratchBytes = TQ_DECODE_STATIC_SCRATCH_BYTES;   // 16 MiB, the stated limit
static __device__ __align__(256) unsigned char g_decode_scratch[kStaticScratchBytes];

// In host code `g_decode_scratch` is only a handle for the runtime, not a device address: the
// address a kernel may use comes from cudaGetSymbolAddress, asked once per device.
void* static_scratch_address(int* status) {
    static void* cached[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        *status = TQ_ERR_LAUNCH;
        return nullptr;
    }
    if (!cached[dev]) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_decode_scratch) != cudaSuccess || !ptr) {
            *status = TQ_ERR_LAUNCH;
            return nullptr;
        }
        cached[dev] = ptr;
    }
    *status = TQ_OK;
    return cached[dev];
}

}  // namespace
}  // namespace tq

extern "C" int tq_decode_paged_static(void* out, const void* q_rot, const void* q_proj, int io_dtype, const void* cache,
                                      int64_t num_blocks, int block_size, const int32_t* block_tables,
                                      int64_t bt_stride, const int32_t* seq_lens, const float* k_centroids,
                                      const float* v_centroids, float sm_scale, float corr_scale, float sparse_thresh,
                                      int32_t* status, uint32_t* skip_stats, int num_seqs, int num_q_heads,
                                      int num_kv_heads, int max_pages_per_seq, int k_bits, int v_bits, int use_qjl,
                                      int chunk_pages, tq_stream_t stream) {
    if (num_seqs == 0) return TQ_OK;
    if (num_seqs < 0 || num_q_heads <= 0 || num_kv_heads <= 0 || max_pages_per_seq <= 0) return TQ_ERR_ARG;
    if (num_q_heads % num_kv_heads) return TQ_ERR_ARG;
    if (chunk_pages <= 0) chunk_pages = tq_decode_auto_chunk_pages(num_seqs, num_kv_heads, num_q_heads, max_pages_per_seq);
    // Refuse, before touching the GPU, any problem whose split-K partials do not fit the fixed array.
    const int64_t need = tq_decode_workspace_bytes(num_seqs, num_q_heads, num_kv_heads, max_pages_per_seq, chunk_pages);
    if (need < 0) return static_cast<int>(need);
    if (need > static_cast<int64_t>(tq::kStaticScratchBytes)) return TQ_ERR_WORKSPACE;
    int rc = TQ_OK;
    void* scratch = tq::static_scratch_address(&rc);
    if (rc != TQ_OK) return rc;
    // Nothing in the scratch has to start at zero: every partial a merge reads was written by the
    // partial kernel of the same call, so contents left by an earlier call are never observed.
    return tq_decode_paged(out, q_rot, q_proj, io_dtype, cache, num_blocks, block_size, block_tables, bt_stride,
                           seq_lens, k_centroids, v_centroids, sm_scale, corr_scale, sparse_thresh, scratch,
                           static_cast<int64_t>(tq::kStaticScratchBytes), status, skip_stats, num_seqs, num_q_heads,
                           num_kv_heads, max_pages_per_seq, k_bits, v_bits, use_qjl, chunk_pages, stream);
}
