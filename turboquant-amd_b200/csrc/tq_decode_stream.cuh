// Decode attention for launches that fill the GPU: one persistent CTA of 16 warps per SM, every warp streams its own
// contiguous share of all pages.
//
// All (sequence, KV head, query group) items of the batch are laid end to end, page after page, and cut into one share per
// warp, of equal length to within a page.  The warps never wait for one another while they stream: a warp keeps its running maximum,
// denominators and accumulators while it stays inside an item and writes the output itself when it saw the whole item.
// Otherwise it leaves a partial result; the CTA combines the partials of its 16 (neighbouring) warps and leaves at most
// two of its own, the item it started in the middle of and the item it could not finish, for decode_stream_merge_kernel.
// Against the chunked kernel (4-warp CTAs, one chunk of one item each) this takes away the last wave that is three
// quarters full, the table fill, pipeline start and merge per chunk, and the empty CTAs of a ragged batch.
//
// What bounds it: instruction issue with four warps a scheduler (a tensor instruction costs about three slots) next to the
// shared-memory data path (turbo3: 93 wavefronts a page), and under constant load the GPU's power: at 1000 W the clock falls from 1965
// to 1765 MHz.  Sign operands by logic, 34 instructions and no shared memory, instead of looked up (20 instructions, 32 wavefronts,
// 32 KB of table), us per launch in a graph, looked up / by logic: turbo3 64 x 8192 tokens 145.5 / 142.4, turbo2 64 x 4096 75.1 / 70.5.
// A Sparse-V call does the same arithmetic on the pages that come with their V part: one that skips nothing gives the dense result bit for bit.
// A page without V part is the other way round: there is little else to do, so the instructions count.  Signs looked up there (3 and 4
// bits, K and V of one codebook: the second table is free), rows not divided, and the count of skipped V parts where it needs no
// register, us per launch in a graph, everything by logic / this, V parts skipped in brackets: turbo3 64 x 8192 150.5 / 143.5 (0 %),
// 149 / 142 (45 %), with groups of 4 136 / 130.5 (68 %), 64 x 32768 467 / 446 (82 %), 16 x 32768 with one head a group 121 / 117.5 (88 %); looked up on
// all pages, with 16 registers less of query operands, 427 and 113 of the last two, 153, 147 and 133 of the others.  2 bits: looked up 427, by
// logic 415 (64 x 32768, 82 %).
// 20 warps of 96 registers (151.6 for 145.6) or 24 of 80 (157.6) lose: the look-ups in flight need registers.
// Pages are staged with cp.async, 16 bytes a lane, into a private ring: a page then costs four copy instructions and a counted
// wait, where a bulk copy by one elected lane with its barrier cost about 35 instructions.  Together with a page body that has no
// partly filled pages to look after, table addresses from the multiply-add pipe and loop state in uniform registers, us per
// launch in a graph of 8 or more over different caches, before / now, 8 KV heads: turbo3 64 x 8192 tokens 151.8 / 145.6, turbo4
// 128.5 / 122.3 and 1 x 131072 43.5 / 41.5, turbo3 128 x 512 34.8 / 34.1, turbo3 with a query of the sign term's own 32 x 4096 53.3 / 49.0;
// 4 KV heads, 32 x 4096: 3-bit K and 4-bit V 28.1 / 26.6, turbo4 28.2 / 27.1.  Only large turbo2 batches lost: 64 x 8192 134.1 / 134.9
// (4 KV heads, 32 x 4096: 28.5 / 28.1); norms loaded behind the products or one body for all pages did not bring it back.
// Two pages per iteration came out the same (the loop's own instructions are few now), and so did V operands without the pairing
// of tokens (twice the products with half of the weights zero: 19 instructions fewer, 8 products more).
// 3-bit keys as integer products (m16n8k32: 16-bit queries and centroids as two signed digits, made by byte permutes from the
// packed indices) were slower (147.8) and lost precision where one coordinate of a query is much larger than the others: the digits
// share one step per row, while a looked-up product keeps the fp16 query as it is.  With one coordinate x 100 the error against 64
// bits was 4 times that of the chunked kernel, with x 1000 35 times.
namespace tq {
namespace {

constexpr int kStreamWarps = 16;
constexpr int kStreamThreads = kStreamWarps * 32;
constexpr int kStreamStages = 4;
constexpr int kStreamFirst = 1;              // pages of a ring that are requested at once
constexpr int kStreamTable = 32768;          // 256 entries of 128 bytes
constexpr int kStreamCtas = 148;             // one per SM
constexpr int kStreamSlotFloats = 8 * kHeadDim;

constexpr int kStreamPartBytes = kStreamSlotFloats * 4 + 64;   // a partial in shared memory: 8 rows, then their (maximum, denominator)
constexpr int kStreamStaticMost = 6144;      // the kernel's static arrays are smaller

// Dynamic shared memory: two tables, then one ring per warp, then as many partials as there is room for, at most one per warp.
__host__ __device__ constexpr int stream_pool(int ring) {
    const int room = (227 * 1024 - 1024 - kStreamStaticMost - 2 * kStreamTable - kStreamWarps * ring) / kStreamPartBytes;
    return room < kStreamWarps ? room : kStreamWarps;
}
__host__ __device__ constexpr int stream_smem(int ring) { return 2 * kStreamTable + kStreamWarps * ring + stream_pool(ring) * kStreamPartBytes; }

struct StreamParams {
    DecodeParams d;
    int ns, HG;          // sequences; items per sequence (KV heads x query groups)
    int n_warps;
    float* part_o;       // [n_warps + 2 n_ctas][8][128]: one slot per warp, then two per CTA (1: starts at its item's first page)
    float2* part_ml;     // [n_warps + 2 n_ctas][8] (maximum, denominator)
    int4* split;         // [n_ctas] item that starts in the CTA and ends in a later one: (sequence, item of it, last CTA or -1)
    uint32_t two12, two20;
    float weight_thresh; // Sparse-V: weights are relative to a reference at most one (log2) above the running maximum
};

// Shares of U pages for W warps: the first U % W have one page more.  (W is a constant: a division by a parameter cost a launch 0.2 us.)
struct Shares {
    uint32_t each, more;
    __device__ __forceinline__ explicit Shares(uint32_t pages) : each(pages / (kStreamCtas * kStreamWarps)), more(pages % (kStreamCtas * kStreamWarps)) {}
    __device__ __forceinline__ uint32_t start(uint32_t w) const { return each * w + min(w, more); }
    __device__ __forceinline__ uint32_t owner(uint32_t page) const {
        const uint32_t longer = more * (each + 1);
        return page < longer ? page / (each + 1) : more + (page - longer) / each;
    }
};

// A value that all lanes of the warp have, as one that the compiler knows to be: it then keeps it in a uniform register and
// branches on it without preparing for lanes that part.
__device__ __forceinline__ int uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }

__device__ __forceinline__ int pages_of(const DecodeParams& p, int len) {
    return min(pages_of_length(len), p.max_pages);
}

// Address of the table entry that byte k of w names: a dot product with one weight of 128, the size of an entry.  It runs on the
// multiply-add pipe; the logic pipe, which a byte permute or a shift and a mask would take, is the busier one.
template <int K>
__device__ __forceinline__ uint32_t entry_of(uint32_t w, uint32_t base) {
    uint32_t a;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(0x80u << (8 * K)), "r"(base));
    return a;
}
template <int K>
__device__ __forceinline__ uint32_t table_pair(uint32_t w, uint32_t base) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(entry_of<K>(w, base)));
    return v;
}
template <int K>
__device__ __forceinline__ uint2 table_quad(uint32_t w, uint32_t base) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(entry_of<K>(w, base)));
    return v;
}

// mask ? b : a, bit by bit.  As PTX, so that the shift that makes an operand is not moved behind a mask of
// its own (the compiler then spends two logic instructions on each of these).
__device__ __forceinline__ uint32_t bit_select(uint32_t a, uint32_t b, uint32_t mask) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xd8;" : "=r"(r) : "r"(a), "r"(b), "r"(mask));
    return r;
}
// Words whose bytes address the table.  The table does not look at the spare top bit of a 3-bit nibble.
template <int BITS>
__device__ __forceinline__ void table_words(const uint32_t* w, uint32_t (&mw)[4]) {
    if constexpr (BITS == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mw[j] = w[j];
    } else {
        mw[0] = w[0];
        mw[1] = w[1];
        mw[2] = w[2];
        mw[3] = bit_select(bit_select(w[0] >> 3, w[1] >> 2, 0x22222222u), w[2] >> 1, 0x44444444u);
    }
}

// A V word holds the nibbles e = 0 .. 3 of token a in its low and of token b in its high half.  Bytes 2 and 3 become
// (b_0, a_0), (b_2, a_2) or (a_1, b_1), (a_3, b_3), low nibble first: a table entry is then one dim of two tokens, which
// is what the tensor core wants of V^T as its A operand (dims on M, tokens on K), with all 16 rows in use.
// The shifts are multiplications by kernel parameters: they run on the multiply-add pipe, the logic pipe is the busy one.
__device__ __forceinline__ uint32_t even_pairs(uint32_t w, uint32_t two20) { return bit_select(w * two20, w, 0x0f0f0000u); }
__device__ __forceinline__ uint32_t odd_pairs(uint32_t w, uint32_t two12) { return bit_select(w * two12, w, 0xf0f00000u); }

// 2-bit V words: nibble e of either half holds the indices of dims 4 u + e for u = 2 j (low two bits) and 2 j + 1.  Two swaps
// of fields make byte s' + 2 s of it (a, b) of dim e = s and (a, b) of dim e = s + 2 of u = 2 j + s': the two half2 of an
// entry are then neighbouring registers of one product's A operand, as with the scores.
__device__ __forceinline__ uint32_t paired_dims(uint32_t w, uint32_t two12) {
    w = bit_select(bit_select(w, w * two12, 0x0f0f0000u), w >> 12, 0x0000f0f0u);
    return bit_select(bit_select(w, w << 6, 0x33003300u), w >> 6, 0x00cc00ccu);
}

__device__ __forceinline__ void store_entry(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

template <int BITS>
__device__ __forceinline__ void fill_stream_table(uint32_t smem_addr, float centroid, int warp, int lane) {
    const float cv = __half2float(__float2half_rn(centroid));
#pragma unroll
    for (int i = 0; i < 256 / (4 * kStreamWarps); ++i) {   // eight lanes an entry
        const int b = 4 * (i * kStreamWarps + warp) + (lane >> 3);
        store_entry(smem_addr + b * 128 + 16 * (lane & 7), pair_entry<BITS>(cv, b));
    }
}

// Bytes [FROM, TO) of a page to shared memory, 16 bytes a lane and instruction; all lanes of the warp call it with the same page.
template <int FROM, int TO>
__device__ __forceinline__ void copy_in(uint32_t dst, const uint8_t* page, int lane) {
    static_assert(FROM % 16 == 0 && TO % 16 == 0);
#pragma unroll
    for (int at = FROM; at < TO; at += 512)
        if (at + 512 <= TO || at + 16 * lane < TO)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + at + 16 * lane), "l"(page + at + 16 * lane) : "memory");
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// 16 consecutive values of a row to fp16 / bf16.
__device__ __forceinline__ void store_row16(void* out, int64_t off, int io_dtype, const float (&x)[16]) {
    uint4* dst = reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + off);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = x[8 * i + 2 * j], b = x[8 * i + 2 * j + 1];
            if (io_dtype == TQ_DTYPE_F16) {
                w[j] = pack_half2(a, b);
            } else {
                const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
                w[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
        dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// x H for a row of which this lane holds dims 16 gid .. 16 gid + 15 (gid = lane >> 2): four stages in the lane, three across.
__device__ __forceinline__ void wht_16x8(float (&x)[16], int lane) {
#pragma unroll
    for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (!(i & h)) {
                const float a = x[i], b = x[i + h];
                x[i] = a + b;
                x[i + h] = a - b;
            }
        }
    }
#pragma unroll
    for (int m = 4; m < 32; m <<= 1) {
        const float sgn = (lane & m) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = fmaf(sgn, x[i], __shfl_xor_sync(0xffffffffu, x[i], m));
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] *= kWhtScale;
}

// Sign table, indexed by one nibble of signs (four dims) of token A and one of token B: the four half2 of +-kSignUnit that are the A
// operand of one score product, in its register order (A dims 0 1, B dims 0 1, A dims 2 3, B dims 2 3), 8 copies.  The sums then count
// in what the one-sided operands count in.
__device__ __forceinline__ void fill_sign_table(uint32_t smem_addr, int warp, int lane) {
    auto signs = [](int pair) { return 0x84008400u ^ ((pair & 1) ? 0x8000u : 0u) ^ ((pair & 2) ? 0x80000000u : 0u); };
    for (int b0 = 4 * warp; b0 < 256; b0 += 4 * kStreamWarps) {
        const int b = b0 + (lane >> 3);
        store_entry(smem_addr + b * 128 + 16 * (lane & 7), make_uint4(signs(b), signs(b >> 4), signs(b >> 2), signs(b >> 6)));
    }
}
template <int K>
__device__ __forceinline__ uint4 table_signs(uint32_t w, uint32_t base) {
    uint4 v;
    asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(entry_of<K>(w, base)));
    return v;
}
// Output row g of an item.
__device__ __forceinline__ void finish_row(const DecodeParams& p, int seq, int hg, int g, int lane, float (&x)[4], float l) {
    const int kvh = p.ngroups == 1 ? hg : hg / p.ngroups, qg = hg - kvh * p.ngroups;
    if (g < p.G - qg * 8) write_row(p, static_cast<int64_t>(seq) * p.Hq + kvh * p.G + qg * 8 + g, lane, x, l);
}

// Combines the partials of the CTA's warps: entry 2 w (item that ended inside warp w's share) and 2 w + 1 (the one its share ended in),
// in page order.  A run is the entries of one item.  First warp g finds what the entries of all runs weigh in query row g, lane e for
// entry e, then the rows of all runs are dealt out to the warps.  Entries of even number lie in shared
// memory too while there is room for them.  (One run after the other, each with its own reductions and the even entries in the
// workspace, took 4 us of turbo3 64 x 8192, 5.4 of a mixed turbo2 batch of 256 sequences.  us per launch in a graph, before / now: turbo2
// 64 x 4096 tokens 69.1 / 67.0, turbo3 128 x 512 32.5 / 31.2; the mixed batch 366 / 354.)  sm_scan and sm_len have served their purpose.
template <int RING>
__device__ __forceinline__ void combine_partials(const StreamParams& sp, const int4* sm_part, uint32_t rings, int* sm_scan, int* sm_len) {
    const DecodeParams& p = sp.d;
    float* weight = reinterpret_cast<float*>(sm_scan);     // [8][32]
    float2* sum = reinterpret_cast<float2*>(sm_len);       // [8][32], at a run's first entry: (maximum, denominator)
    static_assert(2 * kStreamWarps == 32 && kStreamThreads * sizeof(int) >= 8 * 32 * sizeof(float2), "one lane an entry; the scan's arrays hold weights and sums");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rows = min(8, p.G);
    const int4 part = sm_part[lane];
    const uint32_t live = __ballot_sync(0xffffffffu, part.x >= 0);
    const int prev = 31 - __clz(live & ((1u << lane) - 1u));   // the live entry before this one, or -1
    const int prev_x = __shfl_sync(0xffffffffu, part.x, max(prev, 0)), prev_y = __shfl_sync(0xffffffffu, part.y, max(prev, 0));
    const uint32_t heads = __ballot_sync(0xffffffffu, part.x >= 0 && (prev < 0 || prev_x != part.x || prev_y != part.y));
    // where entry `lane` lies: an address in shared memory, or 0 for the warp's slot in the workspace
    const int place = part.w >> 1;
    const uint32_t at = (lane & 1) ? rings + (lane >> 1) * RING : place ? rings + kStreamWarps * RING + (place - 1) * kStreamPartBytes : 0;
    if (warp < rows) {
        const uint32_t upto = 0xffffffffu >> (31 - lane);
        const int head = max(31 - __clz(heads & upto), 0), last = (heads & ~upto) ? __ffs(heads & ~upto) - 2 : 31;
        float2 ml = make_float2(-INFINITY, 0.f);
        if (part.x >= 0) {
            if (at) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(ml.x), "=f"(ml.y) : "r"(at + (kStreamSlotFloats + 2 * warp) * 4));
            else ml = __ldcg(sp.part_ml + (blockIdx.x * kStreamWarps + (lane >> 1)) * 8 + warp);
        }
        float M = ml.x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_up_sync(0xffffffffu, M, o);
            if (lane - o >= head) M = fmaxf(M, v);
        }
        M = __shfl_sync(0xffffffffu, M, last);
        const float w = part.x >= 0 ? ex2(ml.x - M) : 0.f;
        float l = w * ml.y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_up_sync(0xffffffffu, l, o);
            if (lane - o >= head) l += v;
        }
        l = __shfl_sync(0xffffffffu, l, last);
        weight[warp * 32 + lane] = w;
        if (lane == head) sum[warp * 32 + lane] = make_float2(M, l);
    } else if (warp == kStreamWarps - 1 && lane == 0) {
        // the item that starts in this CTA and ends in a later one, if there is one, is the last run
        const int4 first = sm_part[heads ? 31 - __clz(heads) : 0], end = sm_part[live ? 31 - __clz(live) : 0];
        int last_cta = -1;
        if (live && (first.w & 1) && end.z > 0) {
            const Shares shares(static_cast<uint32_t>(sm_scan[kStreamThreads]) * sp.HG);
            last_cta = static_cast<int>(shares.owner(shares.start((blockIdx.x + 1) * kStreamWarps) + end.z - 1)) / kStreamWarps;
        }
        sp.split[blockIdx.x] = make_int4(first.y, first.x, last_cta, 0);
    }
    __syncthreads();
    uint32_t after_heads = heads;
    for (int run = 0; after_heads; ++run) {
        const int head = __ffs(after_heads) - 1;
        after_heads &= after_heads - 1;
        const int g = (warp - run * rows) & (kStreamWarps - 1);
        if (g >= rows) continue;
        uint32_t rest = live & ~((1u << head) - 1u) & (after_heads ? (1u << (__ffs(after_heads) - 1)) - 1u : 0xffffffffu);
        const int4 item = sm_part[head];
        const int after = sm_part[31 - __clz(rest)].z;
        const float2 ml = sum[g * 32 + head];
        const bool starts = item.w & 1;
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        while (rest) {   // four entries at a time
            float4 v[4];
            float w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int e = rest ? __ffs(rest) - 1 : -1;
                rest &= rest - 1;
                const uint32_t from = __shfl_sync(0xffffffffu, at, e & 31);
                v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                w[k] = 0.f;
                if (e >= 0) {
                    w[k] = weight[g * 32 + e];
                    if (from)
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[k].x), "=f"(v[k].y), "=f"(v[k].z), "=f"(v[k].w) : "r"(from + (g * kHeadDim + 4 * lane) * 4));
                    else
                        v[k] = __ldcg(reinterpret_cast<const float4*>(sp.part_o + static_cast<int64_t>(blockIdx.x * kStreamWarps + (e >> 1)) * kStreamSlotFloats + g * kHeadDim + 4 * lane));
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                x[0] = fmaf(w[k], v[k].x, x[0]);
                x[1] = fmaf(w[k], v[k].y, x[1]);
                x[2] = fmaf(w[k], v[k].z, x[2]);
                x[3] = fmaf(w[k], v[k].w, x[3]);
            }
        }
        if (starts && after == 0) {
            finish_row(p, item.y, item.x, g, lane, x, ml.y);
        } else {
            const int slot = sp.n_warps + 2 * blockIdx.x + (starts ? 1 : 0);
            *reinterpret_cast<float4*>(sp.part_o + static_cast<int64_t>(slot) * kStreamSlotFloats + g * kHeadDim + 4 * lane) = make_float4(x[0], x[1], x[2], x[3]);
            if (lane == 0) sp.part_ml[slot * 8 + g] = ml;
        }
    }
}

// SIGN_TABLE: Sparse-V with K and V of one codebook and S = I looks up the signs of pages that come without their V part, in the second
// table; the query operands of the index term serve them as well.
template <int KB, int VB, bool QJL, bool SPARSE, bool SIGN_TABLE>
__global__ void __launch_bounds__(kStreamThreads, 1) decode_stream_kernel(const __grid_constant__ StreamParams sp) {
    constexpr int NWK = KB + (QJL ? 1 : 0);
    constexpr int RK = 16 * NWK;
    constexpr int KN_OFF = 16 * RK;
    constexpr int KRN_OFF = KN_OFF + 32;
    constexpr int KPART = KN_OFF + 32 + (QJL ? 32 : 0);
    constexpr int VN_OFF = KPART + 256 * VB;
    constexpr int PAGE = KPART + 256 * VB + 32;
    constexpr int NSTAGE = kStreamStages;
    constexpr int RING = NSTAGE * PAGE;
    static_assert(stream_smem(RING) + kStreamStaticMost + 1024 <= 227 * 1024, "what an SM gives one CTA");
    const DecodeParams& p = sp.d;

    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int sm_scan[kStreamThreads + 1];
    __shared__ __align__(16) int sm_len[kStreamThreads];   // length of the first sequence of each thread's run
    __shared__ int sm_wsum[kStreamWarps];
    __shared__ int4 sm_window[kStreamWarps];     // where the next window of a warp starts: (sequence, item of it, page, pages of the sequence)
    // partials: (item or -1, sequence, pages of the item after this share, bit 0: starts at the item's first page; above it, where an
    // entry of even number lies: partial of the pool from 1, or 0 for the warp's slot in the workspace)
    __shared__ int4 sm_part[2 * kStreamWarps];
    __shared__ int sm_pool;
    __shared__ uint32_t sm_skipped[SIGN_TABLE ? kStreamWarps : 1];
    static_assert(RING >= kStreamPartBytes, "a warp's last partial lies in its ring");
    static_assert(sizeof(sm_scan) + sizeof(sm_len) + sizeof(sm_wsum) + sizeof(sm_window) + sizeof(sm_part) + sizeof(sm_pool) + sizeof(sm_skipped) + 7 * 16 <= kStreamStaticMost,
                  "what stream_pool leaves for static arrays");

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;

    const uint32_t ktab = smem_u32(smem), vtab = ktab + (SIGN_TABLE ? 0 : kStreamTable), stab = ktab + kStreamTable;
    const uint32_t rings = ktab + 2 * kStreamTable, ring = rings + warp * RING;

    if constexpr (SIGN_TABLE) fill_sign_table(stab, warp, lane);   // constants
    if (lane < 2) sm_part[2 * warp + lane] = make_int4(-1, 0, 0, 0);
    if (threadIdx.x == 0) sm_pool = 0;
    pdl_wait();
    pdl_release();
    const float ck = lane_centroid<KB>(p.kc, lane), cv = SIGN_TABLE ? 0.f : lane_centroid<VB>(p.vc, lane);

    // ---- pages before each thread's run of sequences (every CTA does the same scan over all lengths)
    // (With its sums by one reduction, shares by a constant and the K table filled while the block table's entries come, all at once and with a
    // prefetch of the lengths that alone gave nothing and is gone: turbo4 1 x 131072 tokens 40.5 / 39.7 us in a graph, a bf16 decode step of
    // 32 sequences with its append 37.9 / 36.8.)
    const int per = (sp.ns + kStreamThreads - 1) / kStreamThreads;
    int own = 0, len0 = 0;
    for (int s = threadIdx.x * per; s < min(sp.ns, (static_cast<int>(threadIdx.x) + 1) * per); ++s) {
        const int len = p.seq_lens[s];
        if (s == static_cast<int>(threadIdx.x) * per) len0 = len;
        own += pages_of(p, len);
    }
    sm_len[threadIdx.x] = len0;
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) sm_wsum[warp] = incl;
    __syncthreads();
    const int wsum = lane < kStreamWarps ? sm_wsum[lane] : 0;
    const int total = __reduce_add_sync(0xffffffffu, wsum);
    sm_scan[threadIdx.x] = incl - own + __reduce_add_sync(0xffffffffu, lane < warp ? wsum : 0);
    if (threadIdx.x == 0) sm_scan[kStreamThreads] = total;

    const uint32_t gw = blockIdx.x * kStreamWarps + warp;
    uint32_t first;                                     // this warp's first page
    int n;                                              // and how many it has
    {
        const Shares shares(static_cast<uint32_t>(total) * sp.HG);   // at most 2^31 pages
        first = shares.start(gw);
        first = uniform(first);
        n = uniform(static_cast<int>(shares.start(gw + 1) - first));
    }
    __syncthreads();

    // ---- the item and page this warp starts in
    int seq = 0, hg = 0, page = 0, np = 0, len = 0;
    if (n > 0) {
        // the last run that starts at or before page `first`: one probe of every 16th, one of the 16 after it
        auto before = [&](int i) { return static_cast<uint32_t>(sm_scan[i]) * sp.HG <= first; };
        int lo = 16 * (__popc(__ballot_sync(0xffffffffu, before(16 * lane))) - 1);
        lo += __popc(__ballot_sync(0xffffffffu, lane < 16 && before(lo + (lane & 15)))) - 1;
        seq = lo * per;
        len = sm_len[lo];
        uint32_t at = static_cast<uint32_t>(sm_scan[lo]) * sp.HG;
        for (;;) {
            np = pages_of(p, len);
            if (first < at + static_cast<uint32_t>(np) * sp.HG) break;
            at += static_cast<uint32_t>(np) * sp.HG;
            len = __ldg(p.seq_lens + ++seq);
        }
        const int r = static_cast<int>(first - at);
        hg = r / np;
        page = r - hg * np;
        seq = uniform(seq);
        len = uniform(len);
        np = uniform(np);
        hg = uniform(hg);
        page = uniform(page);
    }
    auto kv_head = [&](int h) { return p.ngroups == 1 ? h : h / p.ngroups; };

    // ---- copies in: lane l holds the place in the cache (in pages) of page 32 k + l of the warp's share, one window of 32 ahead
    bool bad_block = false;
    auto block_of = [&](int s, int pg) { return __ldg(p.block_tables + static_cast<int64_t>(s) * p.bt_stride + (pg >> p.sub_shift)); };
    auto place = [&](int32_t blk, int h, int pg) -> uint32_t {
        if (blk < 0 || blk >= p.num_blocks) {
            bad_block = true;
            blk = 0;
        }
        return (static_cast<uint32_t>(blk * p.Hkv + kv_head(h)) << p.sub_shift) + (pg & ((1 << p.sub_shift) - 1));
    };
    auto page_at = [&](uint32_t at) { return p.cache + static_cast<uint64_t>(at) * PAGE; };
    if (lane == 0) sm_window[warp] = make_int4(seq, hg, page, np);
    struct Entry { int32_t blk; int h, pg; bool live; };
    auto window_entry = [&](int base) -> Entry {   // of page base + lane of the share
        __syncwarp();
        const int4 from = sm_window[warp];
        int s = from.x, h = from.y, pg = from.z + lane, m = from.w;
        Entry e = {0, 0, 0, base + lane < n};
        if (e.live) {
            while (pg >= m) {
                pg -= m;
                if (++h == sp.HG) {
                    h = 0;
                    do m = pages_of(p, __ldg(p.seq_lens + ++s)); while (m == 0);
                }
            }
            e.blk = block_of(s, pg);
            e.h = h;
            e.pg = pg;
        }
        __syncwarp();
        if (lane == 31) sm_window[warp] = make_int4(s, h, pg + 1, m);
        return e;
    };
    auto next_window = [&](int base) -> uint32_t {
        const Entry e = window_entry(base);
        return e.live ? place(e.blk, e.h, e.pg) : 0;
    };
    // The words of an item's queries, for the operands made of them when the item begins: requested ahead of the first pages, and from
    // the second item on before the result of the one before is written.
    uint32_t qf[16];
    auto request_queries = [&](int s, int h) {
        const int kvh = kv_head(h), head = kvh * p.G + (h - kvh * p.ngroups) * 8;
        load_q_words(p.q, (static_cast<int64_t>(s) * p.Hq + head + gid) * kHeadDim, tig, kvh * p.G + p.G - head > gid, qf);
    };
    const Entry entry = window_entry(0);
    if (n > 0) request_queries(seq, hg);
    fill_stream_table<KB>(ktab, ck, warp, lane);   // while the block table's entries come
    uint32_t src = entry.live ? place(entry.blk, entry.h, entry.pg) : 0, src_next = src;
    // Full rings of all warps are 13 to 20 MB, 2 to 3 us of the memory's time, in which nothing else comes through: the queries and the
    // first page are requested at once, the rest of the ring when the tables are filled.  us per launch in a graph, rings first and
    // queries last / this: turbo3 128 x 512 tokens 34.1 / 32.4, 32 x 4096 48.0 / 46.9, Sparse-V 32 x 8192 84.6 / 82.7 (two pages at
    // once: 32.9, 46.9, 83.4).
    auto first_copies = [&](int from, int to) {
#pragma unroll
        for (int i = from; i < to; ++i) {
            const uint32_t at = __shfl_sync(0xffffffffu, src, i);
            if (i < n) copy_in<0, PAGE>(ring + i * PAGE, page_at(at), lane);
            copies_end();
        }
    };
    first_copies(0, kStreamFirst);
    if (n > 32) src_next = next_window(32);
    // Flags of lengths that are cut and zeros of empty sequences, behind the first pages' copies: sequence s belongs to warp
    // s / gridDim of CTA s % gridDim (one thread a sequence in CTA 0 took 1.8 ms for 1008 empty sequences of 128 heads).
    for (int s = warp * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x); s < sp.ns; s += sp.n_warps) {
        const int l = p.seq_lens[s];
        if (lane == 0 && p.status && pages_of_length(l) > p.max_pages) atomicOr(p.status, TQ_STATUS_BAD_BLOCK);
        if (l <= 0) {
            uint4* o = reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + static_cast<int64_t>(s) * p.Hq * kHeadDim);
            for (int i = lane; i < p.Hq * kHeadDim / 8; i += 32) o[i] = make_uint4(0, 0, 0, 0);
        }
    }
    if constexpr (!SIGN_TABLE) fill_stream_table<VB>(vtab, cv, warp, lane);   // behind the first pages' copies
    first_copies(kStreamFirst, NSTAGE);
    __syncthreads();

    const uint32_t klut = ktab + (KB == 2 ? 8 * (lane & 15) : 4 * lane);
    const uint32_t vlut = vtab + (VB == 2 ? 8 * (lane & 15) : 4 * lane);
    const uint32_t slut = stab + 16 * (lane & 7);
    const uint32_t ring_k = ring + lane * (NWK * 4);
    const uint32_t ring_n = ring + gid * 4;
    const uint32_t ring_v = ring + (tig * 8 + gid) * 4;

    uint32_t stage = 0;                       // ring stage of the current page
    // Sparse-V: bit s = the page in stage s came without its V part; above the stages' bits how many V parts were never fetched, or in
    // shared memory (us per launch in a graph, here / in shared memory, turbo3 64 x 8192: with the sign table 146.3 / 143.7, without 150.7 / 156)
    uint32_t k_only = 0;
    if constexpr (SIGN_TABLE) {
        if (lane == 0) sm_skipped[warp] = 0;
    }
    int idx = 0;                              // pages of the share that are done

    while (idx < n) {
        const int seg = min(np - page, n - idx);           // pages of this item in the share
        const int kvh = kv_head(hg), qg = hg - kvh * p.ngroups;
        const int head0 = kvh * p.G + qg * 8, nq = min(8, p.G - qg * 8);

        uint32_t qpf[QJL ? 16 : 1];
        float sq_init0 = 0.f, sq_init1 = 0.f;   // minus the query sums of the one-sided sign forms
        uint32_t divided = 0;                   // queries whose one-sided sign operands are divided by 256
        {
            if (p.rotate_q) rotate_q_words(qf, lane, p.io_dtype);
            if constexpr (QJL) {
                float xq[32], corr;
                if (p.qp) {
                    load_q_words(p.qp, (static_cast<int64_t>(seq) * p.Hq + head0 + gid) * kHeadDim, tig, gid < nq, qpf);
                    unpack_q(qpf, p.io_dtype, xq);
                } else {
                    unpack_q(qf, p.io_dtype, xq);
                }
                divided = fit_sign_rows(xq, lane);
                qp_frag_signed_from(xq, qpf, corr);
                corr += __shfl_xor_sync(0xffffffffu, corr, 1);
                corr += __shfl_xor_sync(0xffffffffu, corr, 2);
                sq_init0 = -__shfl_sync(0xffffffffu, corr, 8 * tig);
                sq_init1 = -__shfl_sync(0xffffffffu, corr, 8 * tig + 4);
            }
            q_words_to_half(qf, p.io_dtype);
        }
        // minus the softmax reference of queries 2 tig, 2 tig + 1 (log2 domain).  Sparse-V: columns past the group's heads hold zero
        // queries, whose scores are all alike; with a reference that no score reaches they weigh nothing and decide nothing.
        float r0 = SPARSE && 2 * tig >= nq ? -INFINITY : INFINITY, r1 = SPARSE && 2 * tig + 1 >= nq ? -INFINITY : INFINITY;
        float l0 = 0.f, l1 = 0.f;
        float oacc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int r = 0; r < 4; ++r) oacc[i][r] = 0.f;

        auto one_page = [&](auto have_v, auto partly, auto large, int j) {
            constexpr bool HAVE_V = decltype(have_v)::value, PARTLY = decltype(partly)::value, LARGE = decltype(large)::value;
            constexpr bool LOOK_UP = SIGN_TABLE && !HAVE_V;
            const uint32_t so = stage * PAGE;
            wait_copies<NSTAGE - 1>();
            __syncwarp();
            // ---- scores of 16 tokens x 8 queries
            uint32_t wa[NWK], wb[NWK];
            lds_words<NWK, 0>(ring_k + so, wa);
            lds_words<NWK, 32 * NWK * 4>(ring_k + so, wb);
            uint32_t ra = 0, rb = 0;   // the sign words, rotated; to look up: the nibbles 2 k (ra), 2 k + 1 (rb) of token A, then of token B
            if constexpr (LOOK_UP) {
                ra = bit_select(wb[KB] << 4, wa[KB], 0x0f0f0f0fu);
                rb = bit_select(wb[KB], wa[KB] >> 4, 0x0f0f0f0fu);
            } else if constexpr (QJL) {
                ra = rotate_signs(wa[KB]);
                rb = rotate_signs(wb[KB]);
            }
            float2 kn = unpack_half2(lds_u32<KN_OFF>(ring_n + so)), krn = make_float2(0.f, 0.f);
            if constexpr (QJL) krn = unpack_half2(lds_u32<KRN_OFF>(ring_n + so));
            float sm[4] = {0.f, 0.f, 0.f, 0.f};
            float sq[4] = {sq_init0, sq_init1, sq_init0, sq_init1}, sq2[4] = {0.f, 0.f, 0.f, 0.f};
            if constexpr (LOOK_UP) sq[0] = sq[1] = sq[2] = sq[3] = 0.f;
            auto sign_term = [&](auto quarter) {   // eight dims of two tokens, two products
                constexpr int C = decltype(quarter)::value;
                if constexpr (LOOK_UP) {
                    const uint4 g0 = table_signs<C>(ra, slut), g1 = table_signs<C>(rb, slut);
                    mma_f16_16816(sq, g0.x, g0.y, g0.z, g0.w, qf[4 * C], qf[4 * C + 1]);
                    mma_f16_16816(sq2, g1.x, g1.y, g1.z, g1.w, qf[4 * C + 2], qf[4 * C + 3]);
                } else if constexpr (QJL) {
                    constexpr int I = 4 * C;
                    const uint32_t xa = wa[KB], xb = wb[KB];
                    mma_f16_16816(sq, sign_pair<I>(xa, ra), sign_pair<I>(xb, rb), sign_pair<I + 1>(xa, ra), sign_pair<I + 1>(xb, rb), qpf[I], qpf[I + 1]);
                    mma_f16_16816(sq2, sign_pair<I + 2>(xa, ra), sign_pair<I + 2>(xb, rb), sign_pair<I + 3>(xa, ra), sign_pair<I + 3>(xb, rb),
                                  qpf[I + 2], qpf[I + 3]);
                }
            };
            if constexpr (KB == 2) {
                // An entry holds two half2.  Its byte is made of the pair of indices of token A and that of token B, so that
                // the two are neighbouring registers of the A operand.
                auto quads = [&](auto word) {
                    constexpr int J = decltype(word)::value;
                    const uint32_t y0 = bit_select(wb[J] << 2, wa[J], 0x33333333u), y1 = bit_select(wb[J], wa[J] >> 2, 0x33333333u);
                    auto product = [&](auto first, uint32_t y, int c) {
                        constexpr int B = decltype(first)::value;
                        const uint2 a = table_quad<B>(y, klut), b = table_quad<B + 1>(y, klut);
                        mma_f16_16816(sm, a.x, a.y, b.x, b.y, qf[8 * J + c], qf[8 * J + c + 1]);
                    };
                    product(std::integral_constant<int, 0>{}, y0, 0);
                    product(std::integral_constant<int, 0>{}, y1, 4);
                    sign_term(std::integral_constant<int, 2 * J>{});
                    product(std::integral_constant<int, 2>{}, y0, 2);
                    product(std::integral_constant<int, 2>{}, y1, 6);
                    sign_term(std::integral_constant<int, 2 * J + 1>{});
                };
                quads(std::integral_constant<int, 0>{});
                quads(std::integral_constant<int, 1>{});
            } else {
                uint32_t mwa[4], mwb[4];
                table_words<KB>(wa, mwa);
                table_words<KB>(wb, mwb);
                auto eight_dims = [&](auto word) {
                    constexpr int C = decltype(word)::value;
                    const uint32_t a0 = table_pair<0>(mwa[C], klut), a1 = table_pair<1>(mwa[C], klut);
                    const uint32_t b0 = table_pair<0>(mwb[C], klut), b1 = table_pair<1>(mwb[C], klut);
                    mma_f16_16816(sm, a0, b0, a1, b1, qf[4 * C], qf[4 * C + 1]);
                    const uint32_t a2 = table_pair<2>(mwa[C], klut), a3 = table_pair<3>(mwa[C], klut);
                    const uint32_t b2 = table_pair<2>(mwb[C], klut), b3 = table_pair<3>(mwb[C], klut);
                    mma_f16_16816(sm, a2, b2, a3, b3, qf[4 * C + 2], qf[4 * C + 3]);
                };
                // the signs of a quarter ahead of its look-ups: they need no table and fill the look-ups' latency
                sign_term(std::integral_constant<int, 0>{});
                eight_dims(std::integral_constant<int, 0>{});
                sign_term(std::integral_constant<int, 1>{});
                eight_dims(std::integral_constant<int, 1>{});
                sign_term(std::integral_constant<int, 2>{});
                eight_dims(std::integral_constant<int, 2>{});
                sign_term(std::integral_constant<int, 3>{});
                eight_dims(std::integral_constant<int, 3>{});
            }
            kn.x *= p.qscale;
            kn.y *= p.qscale;
            // tokens gid (s0, s1), gid + 8, queries 2 tig (s0, s2), 2 tig + 1
            float s0 = sm[0] * kn.x, s1 = sm[1] * kn.x, s2 = sm[2] * kn.y, s3 = sm[3] * kn.y;
            if constexpr (QJL) {
                krn.x *= p.qpscale;
                krn.y *= p.qpscale;
                float t0 = sq[0] + sq2[0], t1 = sq[1] + sq2[1], t2 = sq[2] + sq2[2], t3 = sq[3] + sq2[3];
                if constexpr (LARGE && !LOOK_UP) {
                    const float2 by = divided_by(divided, tig);
                    t0 *= by.x;
                    t1 *= by.y;
                    t2 *= by.x;
                    t3 *= by.y;
                }
                s0 = fmaf(t0, krn.x, s0);
                s1 = fmaf(t1, krn.x, s1);
                s2 = fmaf(t2, krn.y, s2);
                s3 = fmaf(t3, krn.y, s3);
            }
            const int valid_tokens = len - (page + j) * kPageTokens;
            if constexpr (PARTLY) {
                if (gid >= valid_tokens) { s0 = -INFINITY; s1 = -INFINITY; }
                if (gid + 8 >= valid_tokens) { s2 = -INFINITY; s3 = -INFINITY; }
            }
            // ---- online softmax.  The reference is raised only when a score exceeds it, and then to one above the
            // largest score, so weights stay <= 1 and most pages need no shuffle and no rescaling.
            const bool over = fmaxf(s0, s2) > -r0 || fmaxf(s1, s3) > -r1;
            if (__any_sync(0xffffffffu, over)) {
                float mx0 = fmaxf(s0, s2), mx1 = fmaxf(s1, s3);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
                    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
                }
                const float rn0 = mx0 > -r0 ? -mx0 - 1.f : r0, rn1 = mx1 > -r1 ? -mx1 - 1.f : r1;
                const float al0 = ex2(rn0 - r0), al1 = ex2(rn1 - r1);
                l0 *= al0;
                l1 *= al1;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    oacc[i][0] *= al0;
                    oacc[i][1] *= al1;
                    oacc[i][2] *= al0;
                    oacc[i][3] *= al1;
                }
                r0 = rn0;
                r1 = rn1;
            }
            const float p0v = ex2(s0 + r0), p1v = ex2(s1 + r1), p2v = ex2(s2 + r0), p3v = ex2(s3 + r1);
            l0 += p0v + p2v;
            l1 += p1v + p3v;

            // ---- Sparse-V: the V part is not needed when no weight of the group exceeds the threshold.  The reference is
            // at most one above the running maximum.
            bool do_v = true;
            if constexpr (SPARSE) do_v = __any_sync(0xffffffffu, fmaxf(fmaxf(p0v, p2v), fmaxf(p1v, p3v)) > sp.weight_thresh);
            bool have = true;
            if constexpr (SPARSE && !HAVE_V) {
                if (do_v) {   // first needed page after a run of skipped ones: fetch its V part now
                    copy_in<KPART, PAGE>(ring + so, page_at(place(block_of(seq, page + j), hg, page + j)), lane);
                    copies_end();
                    wait_copies<0>();
                    __syncwarp();
                } else {
                    if constexpr (!SIGN_TABLE) k_only += 1u << NSTAGE;
                    else if (lane == 0) ++sm_skipped[warp];
                    have = false;
                }
            }
            if (have) {
                float2 vn = unpack_half2(lds_u32<VN_OFF>(ring_n + so));
                if constexpr (PARTLY) {
                    if (gid >= valid_tokens) vn.x = 0.f;
                    if (gid + 8 >= valid_tokens) vn.y = 0.f;
                }
                // B operand: weights of query gid, tokens 2 tig, 2 tig + 1 (then + 8); `back` has the two swapped
                const uint32_t t0 = movmatrix_trans(pack_half2(p0v * vn.x, p1v * vn.x)), t1 = movmatrix_trans(pack_half2(p2v * vn.y, p3v * vn.y));
                const uint32_t back0 = prmt(t0, 0u, 0x1032u), back1 = prmt(t1, 0u, 0x1032u);
                uint32_t va[VB], vb[VB];   // token pairs tig and tig + 4, dim group gid
                va[0] = lds_u32<KPART>(ring_v + so);
                vb[0] = lds_u32<KPART + 128>(ring_v + so);
                va[1] = lds_u32<KPART + 256>(ring_v + so);
                vb[1] = lds_u32<KPART + 384>(ring_v + so);
                if constexpr (VB > 2) {
                    va[2] = lds_u32<KPART + 512>(ring_v + so);
                    vb[2] = lds_u32<KPART + 640>(ring_v + so);
                }
                if constexpr (VB > 3) {
                    va[3] = lds_u32<KPART + 768>(ring_v + so);
                    vb[3] = lds_u32<KPART + 896>(ring_v + so);
                }
                if constexpr (VB == 2) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t ya = paired_dims(va[j], sp.two12), yb = paired_dims(vb[j], sp.two12);
                        auto product = [&](auto byte, float (&acc)[4]) {
                            constexpr int B = decltype(byte)::value;
                            const uint2 a = table_quad<B>(ya, vlut), b = table_quad<B>(yb, vlut);
                            mma_f16_16816(acc, a.x, a.y, b.x, b.y, t0, t1);
                        };
                        product(std::integral_constant<int, 0>{}, oacc[4 * j]);
                        product(std::integral_constant<int, 1>{}, oacc[4 * j + 2]);
                        product(std::integral_constant<int, 2>{}, oacc[4 * j + 1]);
                        product(std::integral_constant<int, 3>{}, oacc[4 * j + 3]);
                    }
                } else {
                    uint32_t ma[4], mb[4];
                    table_words<VB>(va, ma);
                    table_words<VB>(vb, mb);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        {
                            const uint32_t ya = even_pairs(ma[u], sp.two20), yb = even_pairs(mb[u], sp.two20);
                            mma_f16_16816(oacc[2 * u], table_pair<2>(ya, vlut), table_pair<3>(ya, vlut), table_pair<2>(yb, vlut),
                                          table_pair<3>(yb, vlut), back0, back1);
                        }
                        {
                            const uint32_t ya = odd_pairs(ma[u], sp.two12), yb = odd_pairs(mb[u], sp.two12);
                            mma_f16_16816(oacc[2 * u + 1], table_pair<2>(ya, vlut), table_pair<3>(ya, vlut), table_pair<2>(yb, vlut),
                                          table_pair<3>(yb, vlut), t0, t1);
                        }
                    }
                }
            }
            // ---- refill this stage
            __syncwarp();
            const int i = idx + j + NSTAGE;
            if (i < n) {
                if ((i & 31) == 0) {
                    src = src_next;
                    if (i + 32 < n) src_next = next_window(i + 32);
                }
                const uint8_t* next = page_at(__shfl_sync(0xffffffffu, src, i & 31));
                if constexpr (SPARSE) {
                    if (do_v) copy_in<0, PAGE>(ring + so, next, lane);
                    else copy_in<0, KPART>(ring + so, next, lane);
                    if (do_v != HAVE_V) k_only ^= 1u << stage;
                } else {
                    copy_in<0, PAGE>(ring + so, next, lane);
                }
            }
            copies_end();
            if (++stage == NSTAGE) stage = 0;
        };
        auto next_page = [&](auto partly, auto large, int j) {
            if constexpr (SPARSE) {
                if ((SIGN_TABLE && k_only == 0) || !((k_only >> stage) & 1u)) one_page(std::true_type{}, partly, large, j);
                else one_page(std::false_type{}, partly, std::bool_constant<QJL>{}, j);   // (a row that is not divided is multiplied by one)
            } else {
                one_page(std::true_type{}, partly, large, j);
            }
        };
        const int full = min(seg, (len >> 4) - page);   // at most the last page of a sequence is partly filled
        auto pages = [&](auto large) {
            for (int j = 0; j < full; ++j) next_page(std::false_type{}, large, j);
            if (full < seg) next_page(std::true_type{}, large, full);
        };
        if (QJL && divided) pages(std::bool_constant<QJL>{});
        else pages(std::false_type{});

        // ---- the next item
        int next_seq = seq, next_hg = hg, next_len = len, next_np = np;
        if (idx + seg < n) {
            if (++next_hg == sp.HG) {
                next_hg = 0;
                do {
                    next_len = uniform(__ldg(p.seq_lens + ++next_seq));
                    next_np = pages_of(p, next_len);
                } while (next_np == 0);
            }
            request_queries(next_seq, next_hg);
        }
        // ---- the item's result, or this warp's part of it
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, o);
            l1 += __shfl_xor_sync(0xffffffffu, l1, o);
        }
        // accumulator 2 u + s, register r: dim 16 gid + 4 u + s + 2 (r >> 1) of query 2 tig + (r & 1)
        const bool whole_item = page == 0 && seg == np, at_end = idx + seg == n;
        uint32_t keep = 0;      // where in shared memory a partial is kept; the ring has served its purpose at the end of the share
        int place = 0;
        if (!whole_item) {
            if (at_end) {
                keep = ring;
            } else {
                if (lane == 0) place = atomicAdd(&sm_pool, 1) + 1;
                place = __shfl_sync(0xffffffffu, place, 0);
                if (place > stream_pool(RING)) place = 0;
                else keep = rings + kStreamWarps * RING + (place - 1) * kStreamPartBytes;
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int g = 2 * tig + k;
            const float l = k ? l1 : l0;
            float x[16];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) x[4 * u + e] = oacc[2 * u + (e & 1)][(e & 2) + k];
            if (whole_item) {
                const float inv = 1.f / l;
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] *= inv;
                if (p.derotate_out) wht_16x8(x, lane);
                if (g < nq) store_row16(p.out, (static_cast<int64_t>(seq) * p.Hq + head0 + g) * kHeadDim + 16 * gid, p.io_dtype, x);
            } else if (keep) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(keep + (g * kHeadDim + 16 * gid + 4 * i) * 4), "f"(x[4 * i]),
                                 "f"(x[4 * i + 1]), "f"(x[4 * i + 2]), "f"(x[4 * i + 3])
                                 : "memory");
                if (gid == 0) asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(keep + (kStreamSlotFloats + 2 * g) * 4), "f"(k ? -r1 : -r0), "f"(l) : "memory");
            } else {
                float4* dst = reinterpret_cast<float4*>(sp.part_o + static_cast<int64_t>(gw) * kStreamSlotFloats + g * kHeadDim + 16 * gid);
#pragma unroll
                for (int i = 0; i < 4; ++i) dst[i] = make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
                if (gid == 0) sp.part_ml[gw * 8 + g] = make_float2(k ? -r1 : -r0, l);
            }
        }
        if (!whole_item && lane == 0)
            sm_part[2 * warp + (at_end ? 1 : 0)] = make_int4(hg, seq, np - page - seg, (page == 0 ? 1 : 0) | place << 1);
        idx += seg;
        page = 0;
        seq = next_seq;
        hg = next_hg;
        len = next_len;
        np = next_np;
    }
    if (p.status) {
        const bool bad = __any_sync(0xffffffffu, bad_block);
        if (bad && lane == 0) atomicOr(p.status, TQ_STATUS_BAD_BLOCK);
    }
    if constexpr (SPARSE) {
        if (p.skip_stats && lane == 0) {
            atomicAdd(p.skip_stats, static_cast<uint32_t>(idx));
            atomicAdd(p.skip_stats + 1, SIGN_TABLE ? sm_skipped[SIGN_TABLE ? warp : 0] : k_only >> NSTAGE);
        }
    }
    __syncthreads();
    combine_partials<RING>(sp, sm_part, rings, sm_scan, sm_len);
}

template <int KB, int VB, bool QJL, bool SPARSE, bool SIGN_TABLE>
int launch_stream_as(const StreamParams& sp, cudaStream_t stream) {
    auto kern = decode_stream_kernel<KB, VB, QJL, SPARSE, SIGN_TABLE>;
    static bool configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TQ_ERR_LAUNCH;
    constexpr int smem = stream_smem(kStreamStages * page_bytes(KB, VB, QJL ? 1 : 0));
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return TQ_ERR_LAUNCH;
        configured[dev] = true;
    }
    return launch_chained(kern, dim3(sp.n_warps / kStreamWarps), dim3(kStreamThreads), smem, stream, sp) == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
}

template <int KB, int VB, bool QJL, bool SPARSE>
int launch_stream(const StreamParams& sp, cudaStream_t stream) {
    if constexpr (QJL && SPARSE && KB == VB && KB >= 3) {
        if (sp.d.share_tables && !sp.d.qp) return launch_stream_as<KB, VB, QJL, SPARSE, true>(sp, stream);
    }
    return launch_stream_as<KB, VB, QJL, SPARSE, false>(sp, stream);
}

// One block per CTA of the stream kernel: combines the parts of the item that starts there and ends in a later CTA, two
// warps per query row.
constexpr int kStreamMergeWarps = 16;
__global__ void __launch_bounds__(kStreamMergeWarps * 32) decode_stream_merge_kernel(const StreamParams sp) {
    __shared__ float4 so[8][32];
    __shared__ float2 sml[8];
    pdl_release();
    pdl_wait();
    const int cta = blockIdx.x, warp = threadIdx.x >> 5, g = warp & 7, half = warp >> 3, lane = threadIdx.x & 31;
    const int4 item = sp.split[cta];
    if (item.z < 0) return;
    auto slot_of = [&](int i) { return sp.n_warps + 2 * (cta + i) + (i == 0 ? 1 : 0); };   // slot 1 of this CTA, slot 0 of the others
    float M, l, x[4];
    merge_parts(half, 2, item.z - cta + 1, item.z - cta + 1, lane, [&](int i) { return sp.part_o + static_cast<int64_t>(slot_of(i)) * kStreamSlotFloats + g * kHeadDim; },
                [&](int i) { return sp.part_ml[slot_of(i) * 8 + g]; }, M, x, l);
    if (half == 1) {
        so[g][lane] = make_float4(x[0], x[1], x[2], x[3]);
        if (lane == 0) sml[g] = make_float2(M, l);
    }
    __syncthreads();
    if (half == 1) return;
    const float2 other = sml[g];   // at least two parts, so both halves have one
    const float Ma = fmaxf(M, other.x), sa = ex2(M - Ma), sb = ex2(other.x - Ma);
    const float4 v = so[g][lane];
    x[0] = fmaf(sb, v.x, sa * x[0]);
    x[1] = fmaf(sb, v.y, sa * x[1]);
    x[2] = fmaf(sb, v.z, sa * x[2]);
    x[3] = fmaf(sb, v.w, sa * x[3]);
    finish_row(sp.d, item.x, item.y, g, lane, x, fmaf(sb, other.y, sa * l));
}

}  // namespace
}  // namespace tq
