// KV compression for sm_100a: fast WHT, norm, Lloyd-Max bucketize, QJL signs, bit-packing.
//
// Four lanes compress one 128-value vector: lane j of a group holds the 32 dims 32 j .. 32 j + 31
// in registers, a warp works on 8 vectors at a time (first the keys of 8 (token, head) items, then
// their values).  The 128-point Walsh-Hadamard transform is five butterfly stages inside the lane
// and two warp-shuffle stages across the four lanes, so only 2 of 7 stages pay for a shuffle, and
// every per-vector scalar (norm, square root, reciprocal) is amortised over 32 elements per lane.
// A lane's 32 dims are exactly one quarter of a K record of the paged cache, so the packed words
// are assembled in registers and written with one 16-byte store; no cross-lane reduction is needed.
//
// Everything after the rotation follows polarquant_compress of the reference
// (turboquant/core/quantizer.py:141-173) operation by operation in fp32:
//   n = sqrt(sum r^2);  u = r / (n + 1e-8);  idx = #{j : b_j < u};
//   e = (u - c[idx]) * n;  rn = sqrt(sum e^2);  sign = (e >= 0).
// The division is done as a correctly rounded reciprocal followed by one Newton-style correction
// of each quotient (q0 = r * inv; q = q0 + (r - q0 * den) * inv), which returns the IEEE quotient.
// Outputs go either into the paged cache (layout of turboquant/kernels/paged_layout.py) or into
// the contiguous arrays of compress_k / compress_v (turboquant/kernels/packed_compress.py:157-240).
#include <type_traits>

#include "tq_common.cuh"

namespace tq {
namespace {

constexpr int kWarpsPerCta = 4;
constexpr int kItemsPerWarp = 8;
constexpr int kItemsPerCta = kWarpsPerCta * kItemsPerWarp;

// ---- loads: 32 consecutive elements of one row as fp32 ---------------------------------------
__device__ __forceinline__ void load32(const void* base, int64_t elem_off, int dtype, float (&x)[32]) {
    if (dtype == TQ_DTYPE_F32) {
        const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(base) + elem_off);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 v = __ldg(p + i);
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
    } else {
        const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + elem_off);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 v = __ldg(p + i);
            const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (dtype == TQ_DTYPE_F16) {
                    const float2 t = unpack_half2(r[k]);
                    x[8 * i + 2 * k] = t.x;
                    x[8 * i + 2 * k + 1] = t.y;
                } else {
                    x[8 * i + 2 * k] = __uint_as_float(r[k] << 16);
                    x[8 * i + 2 * k + 1] = __uint_as_float(r[k] & 0xffff0000u);
                }
            }
        }
    }
}

__device__ __forceinline__ float group_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}

// ---- bucketize: idx = number of boundaries strictly below u (searchsorted, right=False) -----------
// Branch-free binary search over boundaries held in registers; every index is a compile-time constant.
template <int BITS>
struct Boundaries {
    float b[(1 << BITS) - 1];
    __device__ __forceinline__ void load(const float* __restrict__ g) {
#pragma unroll
        for (int i = 0; i < (1 << BITS) - 1; ++i) b[i] = __ldg(g + i);
    }
    __device__ __forceinline__ int bucket(float u) const {
        if constexpr (BITS == 2) {
            const bool p1 = u > b[1];
            const bool p0 = u > (p1 ? b[2] : b[0]);
            return (p1 ? 2 : 0) + (p0 ? 1 : 0);
        } else if constexpr (BITS == 3) {
            const bool p2 = u > b[3];
            const bool p1 = u > (p2 ? b[5] : b[1]);
            const float hi = p2 ? b[6] : b[2], lo = p2 ? b[4] : b[0];
            const bool p0 = u > (p1 ? hi : lo);
            return (p2 ? 4 : 0) + (p1 ? 2 : 0) + (p0 ? 1 : 0);
        } else {
            const bool p3 = u > b[7];
            const bool p2 = u > (p3 ? b[11] : b[3]);
            const float h1 = p3 ? b[13] : b[5], l1 = p3 ? b[9] : b[1];
            const bool p1 = u > (p2 ? h1 : l1);
            const float c3 = p3 ? b[14] : b[6], c2 = p3 ? b[12] : b[4], c1 = p3 ? b[10] : b[2], c0 = p3 ? b[8] : b[0];
            const float hh = p2 ? c3 : c1, ll = p2 ? c2 : c0;
            const bool p0 = u > (p1 ? hh : ll);
            return (p3 ? 8 : 0) + (p2 ? 4 : 0) + (p1 ? 2 : 0) + (p0 ? 1 : 0);
        }
    }
};

// Result of compressing one quarter (32 dims) of a vector; norm and rnorm are whole-vector values.
struct Quarter {
    uint32_t idx[32];
    uint32_t signs;   // bit l = 1 when the residual of local dim l is >= 0
    float norm, rnorm;
};

// x: this lane's 32 values.  csm: centroids in shared memory (read only when QJL).
template <int BITS, bool QJL>
__device__ __forceinline__ void quantize_quarter(float (&x)[32], bool rotate, int lane, const Boundaries<BITS>& bd,
                                                 const float* csm, Quarter& q) {
    if (rotate) {
        fwht128(x, lane);
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] *= kWhtScale;
    }
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        s0 = fmaf(x[i], x[i], s0);
        s1 = fmaf(x[i + 1], x[i + 1], s1);
        s2 = fmaf(x[i + 2], x[i + 2], s2);
        s3 = fmaf(x[i + 3], x[i + 3], s3);
    }
    const float n = sqrtf(group_sum((s0 + s1) + (s2 + s3)));
    const float den = n + 1e-8f;
    const float inv = __frcp_rn(den);
    float r0 = 0.f, r1 = 0.f;
    uint32_t sb = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const float q0 = x[i] * inv;
        const float u = fmaf(fmaf(-q0, den, x[i]), inv, q0);   // = x / den, correctly rounded
        const int k = bd.bucket(u);
        q.idx[i] = static_cast<uint32_t>(k);
        if constexpr (QJL) {
            const float r = (u - csm[k]) * n;
            if (i & 1) r1 = fmaf(r, r, r1);
            else r0 = fmaf(r, r, r0);
            sb |= (r >= 0.f ? 1u : 0u) << i;   // -0.0 and +0.0 both count as +
        }
    }
    q.signs = sb;
    q.norm = n;
    q.rnorm = QJL ? sqrtf(group_sum(r0 + r1)) : 0.f;
}

// ---- paged stores (bit positions: turboquant/kernels/paged_layout.py) ------------------------------
// K: a lane's 32 dims are one quarter sub-record: BITS index words (+ the sign word).
template <int BITS>
__device__ __forceinline__ void pack_k_quarter(const uint32_t (&idx)[32], uint32_t (&w)[BITS]) {
#pragma unroll
    for (int j = 0; j < BITS; ++j) w[j] = 0;
#pragma unroll
    for (int l = 0; l < 32; ++l) {
        const int c = l >> 2, e = l & 3;
        if constexpr (BITS == 4) {
            w[c >> 1] |= idx[l] << ((c & 1) * 16 + 4 * e);
        } else if constexpr (BITS == 3) {
            if (c < 6) {
                w[c >> 1] |= idx[l] << ((c & 1) * 16 + 4 * e);
            } else {
#pragma unroll
                for (int b = 0; b < 3; ++b) w[b] |= ((idx[l] >> b) & 1u) << ((c - 6) * 16 + 4 * e + 3);
            }
        } else {
            w[c >> 2] |= idx[l] << ((c & 1) * 16 + 4 * e + ((c >> 1) & 1) * 2);
        }
    }
}

template <int BITS, bool QJL>
__device__ __forceinline__ void store_k_paged(uint8_t* page, int t, int quarter, const Quarter& q) {
    constexpr int NW = BITS + (QJL ? 1 : 0);
    constexpr int RK = 16 * NW;
    uint32_t w[BITS];
    pack_k_quarter<BITS>(q.idx, w);
    uint8_t* dst = page + t * RK + quarter * (RK / 4);
    if constexpr (NW == 4) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], QJL ? q.signs : w[BITS - 1]);
    } else if constexpr (NW == 2) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int j = 0; j < BITS; ++j) reinterpret_cast<uint32_t*>(dst)[j] = w[j];
        if constexpr (QJL) reinterpret_cast<uint32_t*>(dst)[BITS] = q.signs;
    }
    if (quarter == 0) {
        reinterpret_cast<__half*>(page + 16 * RK)[norm_slot(t)] = __float2half_rn(q.norm);
        if constexpr (QJL) reinterpret_cast<__half*>(page + 16 * RK + 32)[norm_slot(t)] = __float2half_rn(q.rnorm);
    }
}

// V: a lane's 32 dims are two dim groups g = 2 * quarter + {0, 1}; each gets BITS 16-bit fields.
template <int BITS>
__device__ __forceinline__ void store_v_paged(uint8_t* vpart, int t, int quarter, const Quarter& q) {
    const int pair = t >> 1, half = t & 1;
#pragma unroll
    for (int gg = 0; gg < 2; ++gg) {
        uint32_t f[BITS];
#pragma unroll
        for (int j = 0; j < BITS; ++j) f[j] = 0;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const uint32_t i = q.idx[16 * gg + m];
            const int u = m >> 2, e = m & 3;
            if constexpr (BITS == 4) {
                f[u] |= i << (4 * e);
            } else if constexpr (BITS == 3) {
                if (u < 3) {
                    f[u] |= i << (4 * e);
                } else {
#pragma unroll
                    for (int b = 0; b < 3; ++b) f[b] |= ((i >> b) & 1u) << (4 * e + 3);
                }
            } else {
                f[u >> 1] |= i << (4 * e + (u & 1) * 2);
            }
        }
        const int g = 2 * quarter + gg;
#pragma unroll
        for (int j = 0; j < BITS; ++j)
            *reinterpret_cast<uint16_t*>(vpart + ((j * 8 + pair) * 8 + g) * 4 + half * 2) = static_cast<uint16_t>(f[j]);
    }
    if (quarter == 0) reinterpret_cast<__half*>(vpart + 256 * BITS)[norm_slot(t)] = __float2half_rn(q.norm);
}

// Division by a number that is usually a power of two: a shift then.
struct Divisor {
    uint32_t d;
    int shift;   // -1: not a power of two
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const { return shift >= 0 ? n >> shift : n / d; }
};
Divisor divisor(int d) {
    Divisor r = {static_cast<uint32_t>(d), -1};
    if ((d & (d - 1)) == 0)
        for (r.shift = 0; (1 << r.shift) < d;) ++r.shift;
    return r;
}

struct PagedParams {
    const void* key;
    const void* value;
    uint8_t* cache;
    const int64_t* slot_mapping;
    const float* kc;
    const float* kb;
    const float* vb;
    int32_t* status;
    int64_t ks_t, ks_h, vs_t, vs_h;
    int64_t num_slots;
    int64_t n_items;   // n_tokens * n_kv_heads
    int64_t n_tokens;
    int Hkv, block_size, in_dtype, rotate;
    Divisor div_heads, div_block;
    int use_tcgen05;       // TQ_COMPRESS_TCGEN05 was given
};

// Where one (token, head) item goes in the paged cache; live = false when the item is past the end or its
// slot is out of range (then nothing is stored; a bad slot also raises the status bit).
struct ItemPlace {
    int64_t tok;
    int head, t;
    uint8_t* page;
    bool live;
};

// Which token and KV head an item is; live = false past the end.
struct ItemId {
    int64_t tok;
    int head;
    bool live;
};

__device__ __forceinline__ ItemId identify_item(const PagedParams& p, int64_t item) {
    ItemId id;
    id.tok = 0; id.head = 0;
    id.live = item < p.n_items;
    if (id.live) {
        const uint32_t tk = p.div_heads(static_cast<uint32_t>(item));   // launches have at most 2^30 items
        id.tok = tk;
        id.head = static_cast<int>(static_cast<uint32_t>(item) - tk * static_cast<uint32_t>(p.Hkv));
    }
    return id;
}

// slot: the token's entry of slot_mapping (not looked at unless id.live).
template <int PAGE>
__device__ __forceinline__ ItemPlace place_item(const PagedParams& p, const ItemId& id, int64_t slot, int quarter) {
    ItemPlace w;
    w.tok = id.tok; w.head = id.head; w.t = 0; w.page = nullptr;
    w.live = id.live;
    if (w.live) {
        if (slot < 0) slot = 0;   // the reference clamps padding slots to 0
        if (slot >= p.num_slots) {
            if (quarter == 0 && p.status) atomicOr(p.status, TQ_STATUS_BAD_SLOT);
            w.live = false;
        } else {
            int64_t blk;
            if (p.num_slots <= 0x7fffffff) blk = p.div_block(static_cast<uint32_t>(slot));
            else blk = slot / p.block_size;
            const int off = static_cast<int>(slot - blk * p.block_size);
            const int spb = p.block_size / kPageTokens;
            w.page = p.cache + ((blk * p.Hkv + w.head) * spb + off / kPageTokens) * PAGE;
            w.t = off % kPageTokens;
        }
    }
    return w;
}

template <int PAGE>
__device__ __forceinline__ ItemPlace place_item(const PagedParams& p, const ItemId& id, int quarter) {
    return place_item<PAGE>(p, id, id.live ? p.slot_mapping[id.tok] : 0, quarter);
}

template <int PAGE>
__device__ __forceinline__ ItemPlace place_item(const PagedParams& p, int64_t item, int quarter) {
    return place_item<PAGE>(p, identify_item(p, item), quarter);
}

// Generic path for one group of 8 items per warp: binary-search bucketize over arbitrary sorted boundaries.
// Lanes of items past the end still take part in the shuffles (on zeros) and store nothing.
template <int KB, int VB, bool QJL>
__device__ __noinline__ void compress_items_generic(const PagedParams& p, int64_t item, int lane, const float* csm) {
    constexpr int PAGE = page_bytes(KB, VB, QJL ? 1 : 0);
    constexpr int KPART = k_part_bytes(KB, QJL ? 1 : 0);
    const int quarter = lane & 3;
    const ItemPlace w = place_item<PAGE>(p, item, quarter);
    float x[32];
    Quarter q;
    {
        Boundaries<KB> kbd;
        kbd.load(p.kb);
        if (w.live) load32(p.key, w.tok * p.ks_t + w.head * p.ks_h + 32 * quarter, p.in_dtype, x);
        else {
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = 0.f;
        }
        quantize_quarter<KB, QJL>(x, p.rotate != 0, lane, kbd, csm, q);
        if (w.live) store_k_paged<KB, QJL>(w.page, w.t, quarter, q);
    }
    {
        Boundaries<VB> vbd;
        vbd.load(p.vb);
        if (w.live) load32(p.value, w.tok * p.vs_t + w.head * p.vs_h + 32 * quarter, p.in_dtype, x);
        else {
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = 0.f;
        }
        quantize_quarter<VB, false>(x, p.rotate != 0, lane, vbd, nullptr, q);
        if (w.live) store_v_paged<VB>(w.page + KPART, w.t, quarter, q);
    }
}

}  // namespace
}  // namespace tq

#include "tq_compress_fast.cuh"
#include "tq_compress_tc.cuh"

namespace tq {
namespace {

// ---- contiguous outputs ---------------------------------------------------------------------------
enum class OutMode { kPackedK, kPackedV };

struct ContigParams {
    const void* x;
    const float* c;
    const float* b;
    uint8_t* idx_out;
    uint8_t* sign_out;
    __half* rnorm_h;
    __half* norm_h;
    int64_t* indices;
    float* norms;
    float* mse;
    float* signs;
    float* rnorm;
    int64_t n;
    int in_dtype, rotate, permute;
};

// Reference byte layouts: 2-bit 4 per byte LSB first, 4-bit low nibble first, 3-bit little-endian stream.
// A lane's 32 dims are 8 / 12 / 16 consecutive bytes of the row.
template <int BITS>
__device__ __forceinline__ void store_idx_contig(uint8_t* row, int quarter, const uint32_t (&idx)[32]) {
    uint32_t w[BITS];
#pragma unroll
    for (int j = 0; j < BITS; ++j) w[j] = 0;
#pragma unroll
    for (int l = 0; l < 32; ++l) {
        const int bit = l * BITS;
        w[bit >> 5] |= idx[l] << (bit & 31);
        if ((bit & 31) + BITS > 32) w[(bit >> 5) + 1] |= idx[l] >> (32 - (bit & 31));
    }
    uint32_t* dst = reinterpret_cast<uint32_t*>(row + quarter * (4 * BITS));
    if constexpr (BITS == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    else if constexpr (BITS == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    else {
#pragma unroll
        for (int j = 0; j < BITS; ++j) dst[j] = w[j];
    }
}

// Sign bits and norms of one packed row (this lane's quarter); lanes of rows past the end take part in the shuffles.  signs: bit l = 1 when the residual of local dim l is >= 0.
template <bool QJL>
__device__ __forceinline__ void store_contig_tail(const ContigParams& p, int64_t row, int quarter, uint32_t signs, float norm,
                                                  float rnorm, bool live) {
    if constexpr (QJL) {
        uint8_t* srow = p.sign_out + row * 16;
        if (p.permute) {
            // stride-4 order: output bit 32 c + i <- dim c + 4 i.  This lane's dim 32 q + l has c = l & 3 and
            // i = 8 q + (l >> 2): it fills byte q of each of the four 32-bit words.  Two unshuffles (even bits down, odd bits
            // up) turn bit l into bit 8 (l & 3) + (l >> 2), then the four lanes of the row transpose their bytes, so that
            // lane c holds word c.
            uint32_t v = signs;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t x;
                x = (v ^ (v >> 1)) & 0x22222222u; v ^= x ^ (x << 1);
                x = (v ^ (v >> 2)) & 0x0c0c0c0cu; v ^= x ^ (x << 2);
                x = (v ^ (v >> 4)) & 0x00f000f0u; v ^= x ^ (x << 4);
                x = (v ^ (v >> 8)) & 0x0000ff00u; v ^= x ^ (x << 8);
            }
            const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 2);
            v = (quarter & 2) ? prmt(o, v, 0x7632u) : prmt(v, o, 0x5410u);
            const uint32_t n = __shfl_xor_sync(0xffffffffu, v, 1);
            v = (quarter & 1) ? prmt(n, v, 0x7351u) : prmt(v, n, 0x6240u);
            if (live) reinterpret_cast<uint32_t*>(srow)[quarter] = v;
        } else {
            if (live) reinterpret_cast<uint32_t*>(srow)[quarter] = signs;   // byte j bit b <- dim 8 j + b
        }
        if (live && quarter == 0) p.rnorm_h[row] = __float2half_rn(rnorm);
    }
    if (live && quarter == 0) p.norm_h[row] = __float2half_rn(norm);
}

// One group of 8 rows per warp on the generic quantizer (binary-search bucketize over arbitrary sorted boundaries).
// Lanes of rows past the end still take part in the shuffles (on zeros) and store nothing.  ready() is called when the row has
// been requested: csm has to hold the centroids after it.
template <int BITS, OutMode MODE, class Ready>
__device__ __forceinline__ void compress_contig_rows(const ContigParams& p, int64_t row, int lane, const float* csm, Ready ready) {
    constexpr bool QJL = MODE != OutMode::kPackedV;
    const int quarter = lane & 3;
    const bool live = row < p.n;
    Boundaries<BITS> bd;
    bd.load(p.b);
    float x[32];
    Quarter q;
    if (live) load32(p.x, row * kHeadDim + 32 * quarter, p.in_dtype, x);
    else {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = 0.f;
    }
    ready();
    quantize_quarter<BITS, QJL>(x, p.rotate != 0, lane, bd, csm, q);
    if (live) store_idx_contig<BITS>(p.idx_out + row * (16 * BITS), quarter, q.idx);
    store_contig_tail<QJL>(p, row, quarter, q.signs, q.norm, q.rnorm, live);
}

template <int BITS, OutMode MODE>
__global__ void __launch_bounds__(kWarpsPerCta * 32) compress_contig_kernel(const __grid_constant__ ContigParams p) {
    __shared__ float csm[kWarpsPerCta][1 << BITS];   // a copy per warp: no barrier between the codebook's latency and the row's
    pdl_wait();
    pdl_release_if_small();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr bool QJL = MODE != OutMode::kPackedV;  // V needs no centroids
    const float c = QJL ? p.c[lane & ((1 << BITS) - 1)] : 0.f;
    compress_contig_rows<BITS, MODE>(p, (static_cast<int64_t>(blockIdx.x) * kWarpsPerCta + warp) * kItemsPerWarp + (lane >> 2), lane, csm[warp], [&] {
        if (QJL && lane < (1 << BITS)) csm[warp][lane] = c;
        __syncwarp();
    });
}

// ---- unpacked outputs (polarquant_compress) -------------------------------------------------------------------
// Four fifths of the traffic are stores (int64 indices, fp32 reconstruction and signs), so what counts is that every store
// fills whole 32-byte sectors.  Four lanes share a row as elsewhere, but lane j holds dims 32 i + 8 j .. + 7 for i = 0 .. 3:
// the four lanes write 128 contiguous bytes of fp32 per chunk, each lane one 32-byte access (two accesses of 16 bytes when
// a pointer is not that aligned).  With 32 consecutive dims per lane every 16-byte store met half a sector of its own:
// 65537 fp32 rows with signs took 73 us.
template <bool WIDE>
__device__ __forceinline__ void store8(void* dst, const uint32_t (&w)[8]) {
    if constexpr (WIDE) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
                     "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

template <bool WIDE>
__device__ __forceinline__ void load8(const void* base, int64_t elem_off, int dtype, float* x) {
    if (dtype == TQ_DTYPE_F32) {
        const float* src = static_cast<const float*>(base) + elem_off;
        if constexpr (WIDE) {
            asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7])
                         : "l"(src));
        } else {
            const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
            x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        }
    } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + elem_off));
        const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (dtype == TQ_DTYPE_F16) {
                const float2 t = unpack_half2(r[k]);
                x[2 * k] = t.x;
                x[2 * k + 1] = t.y;
            } else {
                x[2 * k] = __uint_as_float(r[k] << 16);
                x[2 * k + 1] = __uint_as_float(r[k] & 0xffff0000u);
            }
        }
    }
}

// x[8 i + e] is dim 32 i + 8 j + e.  The stages run from dim bit 0 to dim bit 6, as in fwht128: same sums, same rounding.
__device__ __forceinline__ void fwht128_chunks(float (&x)[32], int lane) {
    auto in_lane = [&](int h) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if (!(i & h)) {
                const float a = x[i], b = x[i + h];
                x[i] = a + b;
                x[i + h] = a - b;
            }
        }
    };
    in_lane(1);
    in_lane(2);
    in_lane(4);
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
        const float sgn = (lane & m) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = fmaf(sgn, x[i], __shfl_xor_sync(0xffffffffu, x[i], m));
    }
    in_lane(8);
    in_lane(16);
}

template <int BITS, bool SIGNS, bool WIDE>
__global__ void __launch_bounds__(kWarpsPerCta * 32) compress_unpacked_kernel(const ContigParams p) {
    __shared__ float csm_of[kWarpsPerCta][1 << BITS];   // a copy per warp: no barrier between the codebook's latency and the row's
    pdl_wait();
    pdl_release_if_small();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane & 3;
    float* csm = csm_of[warp];
    const float centroid = p.c[lane & ((1 << BITS) - 1)];
    const int64_t row = (static_cast<int64_t>(blockIdx.x) * kWarpsPerCta + warp) * kItemsPerWarp + (lane >> 2);
    const bool live = row < p.n;   // lanes of rows past the end take part in the shuffles, on zeros
    const int64_t at = row * kHeadDim + 8 * j;
    Boundaries<BITS> bd;
    bd.load(p.b);
    float x[32];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (live) load8<WIDE>(p.x, at + 32 * i, p.in_dtype, x + 8 * i);
        else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[8 * i + e] = 0.f;
        }
    }
    if (lane < (1 << BITS)) csm[lane] = centroid;
    __syncwarp();
    if (p.rotate) {
        fwht128_chunks(x, lane);
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] *= kWhtScale;
    }
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        s0 = fmaf(x[i], x[i], s0);
        s1 = fmaf(x[i + 1], x[i + 1], s1);
        s2 = fmaf(x[i + 2], x[i + 2], s2);
        s3 = fmaf(x[i + 3], x[i + 3], s3);
    }
    const float n = sqrtf(group_sum((s0 + s1) + (s2 + s3)));
    const float den = n + 1e-8f;
    const float inv = __frcp_rn(den);
    float r0 = 0.f, r1 = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t idx[8], mse[8], sign[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = x[8 * i + e];
            const float q0 = v * inv;
            const float u = fmaf(fmaf(-q0, den, v), inv, q0);   // = v / den, correctly rounded
            idx[e] = static_cast<uint32_t>(bd.bucket(u));
            const float c = csm[idx[e]];
            mse[e] = __float_as_uint(c * n);
            if constexpr (SIGNS) {
                const float r = (u - c) * n;
                if (e & 1) r1 = fmaf(r, r, r1);
                else r0 = fmaf(r, r, r0);
                sign[e] = r >= 0.f ? 0x3f800000u : 0xbf800000u;   // -0.0 and +0.0 both count as +
            }
        }
        if (live) {
            const int64_t o = at + 32 * i;
            const uint32_t lo[8] = {idx[0], 0u, idx[1], 0u, idx[2], 0u, idx[3], 0u}, hi[8] = {idx[4], 0u, idx[5], 0u, idx[6], 0u, idx[7], 0u};
            store8<WIDE>(p.indices + o, lo);
            store8<WIDE>(p.indices + o + 4, hi);
            store8<WIDE>(p.mse + o, mse);
            if constexpr (SIGNS) store8<WIDE>(p.signs + o, sign);
        }
    }
    const float rn = SIGNS ? sqrtf(group_sum(r0 + r1)) : 0.f;
    if (live && j == 0) {
        p.norms[row] = n;
        if (p.rnorm) p.rnorm[row] = rn;
    }
}

template <int BITS>
int launch_unpacked(const ContigParams& p, cudaStream_t st) {
    const dim3 grid(static_cast<unsigned>((p.n + kItemsPerCta - 1) / kItemsPerCta)), block(kWarpsPerCta * 32);
    const uintptr_t all = reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.indices) | reinterpret_cast<uintptr_t>(p.mse) |
                          reinterpret_cast<uintptr_t>(p.signs);
    const bool wide = (all & 31) == 0;
    cudaError_t e;
    if (p.signs) e = wide ? launch_chained(compress_unpacked_kernel<BITS, true, true>, grid, block, 0, st, p)
                          : launch_chained(compress_unpacked_kernel<BITS, true, false>, grid, block, 0, st, p);
    else e = wide ? launch_chained(compress_unpacked_kernel<BITS, false, true>, grid, block, 0, st, p)
                  : launch_chained(compress_unpacked_kernel<BITS, false, false>, grid, block, 0, st, p);
    return e == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
}

// ---- packed contiguous outputs on the table-driven quantizer ------------------------------------------------------
// Persistent CTAs of 16 warps, one per SM, as the paged kernel: the table is built once per CTA, which then strides over
// groups of 128 rows, 8 per warp.  fp16 / bf16 rows that still need the rotation are staged through two buffers per
// warp, two groups ahead, and rotated on the tensor cores; fp32 and already rotated rows take plain loads.
template <int BITS, bool QJL>
__device__ __forceinline__ void store_contig_fast(const ContigParams& p, int64_t row, int quarter, const Packed& q) {
    const bool live = row < p.n;
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.idx_out + row * (16 * BITS) + quarter * (4 * BITS));
    if (live) {
        if constexpr (BITS == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(q.word[0], q.word[1], q.word[2], q.word[3]);
        else if constexpr (BITS == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(q.word[0], q.word[1]);
        else {
#pragma unroll
            for (int j = 0; j < BITS; ++j) dst[j] = q.word[j];
        }
    }
    store_contig_tail<QJL>(p, row, quarter, q.signs, q.norm, q.rnorm, live);
}

template <int BITS, bool QJL, Rows ROWS>
__global__ void __launch_bounds__(kFastWarps * 32, 1) compress_contig_fast_kernel(const __grid_constant__ ContigParams p, int64_t n_units) {
    extern __shared__ __align__(128) unsigned char tables[];
    __shared__ float csm[1 << BITS];
    __shared__ Comparisons2 comparisons[BITS == 2 ? kFastWarps : 1];
    __shared__ int bad;
    const int lane = threadIdx.x & 31, quarter = lane & 3, warp = threadIdx.x >> 5;
    constexpr bool mma = ROWS != Rows::kPlain, BF16 = ROWS == Rows::kBF16;
    const uint32_t buf = ((smem_u32(tables) + kTableBytes + 255) & ~255u) + warp * kStagePerWarp;   // two buffers of 8 rows
    const uint32_t dst = stage_at(buf, lane), src = staged_at(buf, lane);
    // units of 8 rows; as in the paged kernel the last round is spread over all SMs, and the first copies go out first
    int64_t unit = static_cast<int64_t>(warp) * gridDim.x + blockIdx.x;
    const int64_t step = static_cast<int64_t>(gridDim.x) * kFastWarps;
    auto row_of = [&](int64_t u) { return u * kItemsPerWarp + (lane >> 2); };
    pdl_wait();
    pdl_release();
    if constexpr (mma) {
        stage_row(dst, p.x, row_of(unit) * kHeadDim + 8 * quarter, row_of(unit) < p.n);
        stage_row(dst + kRowBuffer, p.x, row_of(unit + step) * kHeadDim + 8 * quarter, row_of(unit + step) < p.n);
    }
    if (threadIdx.x == 0) bad = 0;
    if (threadIdx.x < (1 << BITS)) csm[threadIdx.x] = p.c ? p.c[threadIdx.x] : 0.f;
    __syncthreads();
    if constexpr (!mma) build_table<BITS, QJL>(tables, p.b, p.c, &bad);
    else if constexpr (BITS > 2) build_table<BITS, QJL, true>(tables, p.b, p.c, &bad);
    __syncthreads();
    if (bad != 0) {   // two boundaries inside one cell: the generic quantizer
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        for (; unit < n_units; unit += step)
            compress_contig_rows<BITS, QJL ? OutMode::kPackedK : OutMode::kPackedV>(p, row_of(unit), lane, csm, [] {});
        return;
    }
    constexpr uint32_t kBias = kMagicBits * static_cast<uint32_t>(kCellStride);   // modulo 2^32
    const uint32_t tab = smem_u32(tables) + (QJL ? (lane & 7) * 16 : (lane & 15) * 8) - kBias;
    Packed q;
    if constexpr (mma) {
        const WhtFragments hf = make_wht_fragments(lane, BF16);
        Codebook2<BITS> cb;
        if constexpr (BITS == 2) cb.load(p.b, QJL ? p.c : nullptr, &comparisons[warp], lane);
        uint32_t cur = 0;   // offset of the buffer whose turn it is
        for (; unit < n_units; unit += step, cur ^= kRowBuffer) {
            const int64_t row = row_of(unit), nxt = row_of(unit + 2 * step);
            wait_staged();
            compress_row_mma<BF16, BITS, QJL, false, true>(src + cur, lane, hf, tab, cb, q, [&] {
                stage_row(dst + cur, p.x, nxt * kHeadDim + 8 * quarter, nxt < p.n);
            });
            store_contig_fast<BITS, QJL>(p, row, quarter, q);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        const bool rotate = p.rotate != 0;
        const float scale = rotate ? kWhtScale : 1.f, inv_scale = rotate ? 11.313708498984761f : 1.f;
        for (; unit < n_units; unit += step) {
            const int64_t row = row_of(unit);
            f2 y[16];
            fetch_plain(p.x, row * kHeadDim + 32 * quarter, row < p.n, p.in_dtype, rotate, lane, y);
            quantize_fast<BITS, QJL, false, true>(y, scale, inv_scale, tab, q);
            store_contig_fast<BITS, QJL>(p, row, quarter, q);
        }
    }
}

template <int BITS, bool QJL>
int launch_contig_fast(const ContigParams& p, cudaStream_t st) {
    const int64_t n_units = (p.n + kItemsPerWarp - 1) / kItemsPerWarp;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TQ_ERR_LAUNCH;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return TQ_ERR_LAUNCH;
    const unsigned grid = static_cast<unsigned>(n_units < sms ? n_units : sms);
    constexpr int kSmem = kTableBytes + kFastWarps * kStagePerWarp + 256;
    auto run = [&](auto kernel, bool (&configured)[64]) {
        if (dev < 0 || dev >= 64 || !configured[dev]) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return TQ_ERR_LAUNCH;
            if (dev >= 0 && dev < 64) configured[dev] = true;
        }
        return launch_chained(kernel, dim3(grid), dim3(kFastWarps * 32), kSmem, st, p, n_units) == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
    };
    static bool configured[3][64] = {};
    if (!p.rotate || p.in_dtype == TQ_DTYPE_F32) return run(compress_contig_fast_kernel<BITS, QJL, Rows::kPlain>, configured[0]);
    if (p.in_dtype == TQ_DTYPE_F16) return run(compress_contig_fast_kernel<BITS, QJL, Rows::kF16>, configured[1]);
    return run(compress_contig_fast_kernel<BITS, QJL, Rows::kBF16>, configured[2]);
}

template <int KB, int VB>
int launch_paged(const PagedParams& p, bool qjl, cudaStream_t st) {
    return qjl ? launch_paged_fast<KB, VB, true>(p, st) : launch_paged_fast<KB, VB, false>(p, st);
}

template <int KB>
int launch_paged_v(const PagedParams& p, int vb, bool qjl, cudaStream_t st) {
    switch (vb) {
        case 2: return launch_paged<KB, 2>(p, qjl, st);
        case 3: return launch_paged<KB, 3>(p, qjl, st);
        case 4: return launch_paged<KB, 4>(p, qjl, st);
    }
    return TQ_ERR_UNSUPPORTED;
}

template <OutMode MODE>
int launch_contig(const ContigParams& p, int bits, cudaStream_t st) {
    // Large launches: the persistent table-driven kernel.  fp16 rows with the rotation, us, binary-search kernel / persistent:
    // K 16384 rows 5.6 / 5.1, 32768 8.4 / 7.2, 65536 15.4 / 11.0; V 4.6 / 3.7, 6.6 / 5.2, 12.0 / 7.7.  The line stays above
    // the crossing: the two rotations round differently, so a lower one would change the bytes of those sizes.
    if (p.n > 2 * kSmallLaunchItems) {
        constexpr bool QJL = MODE == OutMode::kPackedK;
        switch (bits) {
            case 2: return launch_contig_fast<2, QJL>(p, st);
            case 3: return launch_contig_fast<3, QJL>(p, st);
            case 4: return launch_contig_fast<4, QJL>(p, st);
            default: return TQ_ERR_UNSUPPORTED;
        }
    }
    const dim3 grid(static_cast<unsigned>((p.n + kItemsPerCta - 1) / kItemsPerCta)), block(kWarpsPerCta * 32);
    cudaError_t e;
    switch (bits) {
        case 2: e = launch_chained(compress_contig_kernel<2, MODE>, grid, block, 0, st, p); break;
        case 3: e = launch_chained(compress_contig_kernel<3, MODE>, grid, block, 0, st, p); break;
        case 4: e = launch_chained(compress_contig_kernel<4, MODE>, grid, block, 0, st, p); break;
        default: return TQ_ERR_UNSUPPORTED;
    }
    return e == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
}

// What the index rows have to start on: a lane stores its quarter of a row as one access, or, 3-bit, as three words.
uintptr_t index_align_mask(int bits) { return bits == 4 ? 15 : bits == 2 ? 7 : 3; }

bool dtype_ok(int d) { return d == TQ_DTYPE_F16 || d == TQ_DTYPE_BF16 || d == TQ_DTYPE_F32; }
int elem_bytes(int d) { return d == TQ_DTYPE_F32 ? 4 : 2; }

}  // namespace
}  // namespace tq
using namespace tq;

extern "C" int tq_version(void) { return (0 << 16) | 1; }

extern "C" int tq_page_bytes(int k_bits, int v_bits, int use_qjl) {
    if (k_bits < 2 || k_bits > 4 || v_bits < 2 || v_bits > 4) return TQ_ERR_UNSUPPORTED;
    return page_bytes(k_bits, v_bits, use_qjl ? 1 : 0);
}

extern "C" int tq_compress_paged(const void* key, const void* value, int in_dtype, int64_t k_stride_token,
                                 int64_t k_stride_head, int64_t v_stride_token, int64_t v_stride_head, void* cache,
                                 int64_t num_blocks, int block_size, const int64_t* slot_mapping,
                                 const float* k_centroids, const float* k_boundaries, const float* v_centroids,
                                 const float* v_boundaries, int n_tokens, int n_kv_heads, int k_bits, int v_bits,
                                 int use_qjl, int prerotated, int32_t* status, tq_stream_t stream) {
    (void)v_centroids;  // V stores indices and a norm only; its centroids are not needed to compress
    if (n_tokens == 0) return TQ_OK;
    if (!key || !value || !cache || !slot_mapping || !k_centroids || !k_boundaries || !v_boundaries) return TQ_ERR_ARG;
    if (n_tokens < 0 || n_kv_heads <= 0 || num_blocks <= 0) return TQ_ERR_ARG;
    if (!dtype_ok(in_dtype)) return TQ_ERR_UNSUPPORTED;
    if (block_size <= 0 || block_size % kPageTokens) return TQ_ERR_UNSUPPORTED;
    if (k_bits < 2 || k_bits > 4 || v_bits < 2 || v_bits > 4) return TQ_ERR_UNSUPPORTED;
    const int align_elems = 16 / elem_bytes(in_dtype);  // lanes read rows with 16-byte vector loads
    if (k_stride_token % align_elems || k_stride_head % align_elems || v_stride_token % align_elems ||
        v_stride_head % align_elems)
        return TQ_ERR_ARG;
    const uintptr_t amask = 15;
    if ((reinterpret_cast<uintptr_t>(key) & amask) || (reinterpret_cast<uintptr_t>(value) & amask) ||
        (reinterpret_cast<uintptr_t>(cache) & 15))
        return TQ_ERR_ARG;
    PagedParams p;
    p.key = key;
    p.value = value;
    p.cache = static_cast<uint8_t*>(cache);
    p.slot_mapping = slot_mapping;
    p.kc = k_centroids;
    p.kb = k_boundaries;
    p.vb = v_boundaries;
    p.status = status;
    p.ks_t = k_stride_token;
    p.ks_h = k_stride_head;
    p.vs_t = v_stride_token;
    p.vs_h = v_stride_head;
    p.num_slots = num_blocks * block_size;
    p.n_items = static_cast<int64_t>(n_tokens) * n_kv_heads;
    p.n_tokens = n_tokens;
    p.Hkv = n_kv_heads;
    p.block_size = block_size;
    p.div_heads = divisor(n_kv_heads);
    p.div_block = divisor(block_size);
    p.in_dtype = in_dtype;
    p.rotate = (prerotated & 1) ? 0 : 1;
    p.use_tcgen05 = (prerotated & TQ_COMPRESS_TCGEN05) ? 1 : 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // The kernels count items in 32 bits: a launch covers at most 2^30 of them (and an even number of tokens).
    const int64_t most = n_kv_heads < (1 << 29) ? ((int64_t{1} << 30) / n_kv_heads) & ~int64_t{1} : 0;
    if (most < 2) return TQ_ERR_UNSUPPORTED;
    for (int64_t first = 0; first < n_tokens; first += most) {
        PagedParams part = p;
        part.key = static_cast<const uint8_t*>(key) + first * k_stride_token * elem_bytes(in_dtype);
        part.value = static_cast<const uint8_t*>(value) + first * v_stride_token * elem_bytes(in_dtype);
        part.slot_mapping = slot_mapping + first;
        part.n_tokens = n_tokens - first < most ? n_tokens - first : most;
        part.n_items = part.n_tokens * n_kv_heads;
        int rc = TQ_ERR_UNSUPPORTED;
        switch (k_bits) {
            case 2: rc = launch_paged_v<2>(part, v_bits, use_qjl != 0, st); break;
            case 3: rc = launch_paged_v<3>(part, v_bits, use_qjl != 0, st); break;
            case 4: rc = launch_paged_v<4>(part, v_bits, use_qjl != 0, st); break;
        }
        if (rc != TQ_OK) return rc;
    }
    return TQ_OK;
}

extern "C" int tq_compress_k(const void* K, int in_dtype, int64_t n, const float* centroids, const float* boundaries,
                             int bits, int prerotated, int permute_signs, uint8_t* k_idx, uint8_t* k_signs,
                             void* k_rnorm, void* k_norm, tq_stream_t stream) {
    if (n == 0) return TQ_OK;
    if (!K || !centroids || !boundaries || !k_idx || !k_signs || !k_rnorm || !k_norm || n < 0) return TQ_ERR_ARG;
    if (!dtype_ok(in_dtype)) return TQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(k_signs)) & 15) return TQ_ERR_ARG;
    if (reinterpret_cast<uintptr_t>(k_idx) & index_align_mask(bits)) return TQ_ERR_ARG;
    ContigParams p = {};
    p.x = K; p.c = centroids; p.b = boundaries; p.idx_out = k_idx; p.sign_out = k_signs;
    p.rnorm_h = static_cast<__half*>(k_rnorm); p.norm_h = static_cast<__half*>(k_norm);
    p.n = n; p.in_dtype = in_dtype; p.rotate = prerotated ? 0 : 1; p.permute = permute_signs;
    return launch_contig<OutMode::kPackedK>(p, bits, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tq_compress_v(const void* V, int in_dtype, int64_t n, const float* boundaries, int bits, int prerotated,
                             uint8_t* v_idx, void* v_norm, tq_stream_t stream) {
    if (n == 0) return TQ_OK;
    if (!V || !boundaries || !v_idx || !v_norm || n < 0) return TQ_ERR_ARG;
    if (!dtype_ok(in_dtype)) return TQ_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(V) & 15 || reinterpret_cast<uintptr_t>(v_idx) & index_align_mask(bits)) return TQ_ERR_ARG;
    ContigParams p = {};
    p.x = V; p.b = boundaries; p.idx_out = v_idx; p.norm_h = static_cast<__half*>(v_norm);
    p.n = n; p.in_dtype = in_dtype; p.rotate = prerotated ? 0 : 1;
    return launch_contig<OutMode::kPackedV>(p, bits, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tq_polarquant_compress(const void* x, int in_dtype, int64_t n, const float* centroids,
                                      const float* boundaries, int bits, int use_qjl, int prerotated, int64_t* indices,
                                      float* norms, float* k_mse_rot, float* signs, float* rnorm, tq_stream_t stream) {
    if (n == 0) return TQ_OK;
    if (!x || !centroids || !boundaries || !indices || !norms || !k_mse_rot || n < 0) return TQ_ERR_ARG;
    if (use_qjl && (!signs || !rnorm)) return TQ_ERR_ARG;
    if (!dtype_ok(in_dtype)) return TQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(indices) | reinterpret_cast<uintptr_t>(k_mse_rot) |
         reinterpret_cast<uintptr_t>(signs)) & 15)
        return TQ_ERR_ARG;
    ContigParams p = {};
    p.x = x; p.c = centroids; p.b = boundaries; p.indices = indices; p.norms = norms; p.mse = k_mse_rot;
    p.signs = use_qjl ? signs : nullptr; p.rnorm = use_qjl ? rnorm : nullptr;
    p.n = n; p.in_dtype = in_dtype; p.rotate = prerotated ? 0 : 1;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    switch (bits) {
        case 2: return launch_unpacked<2>(p, st);
        case 3: return launch_unpacked<3>(p, st);
        case 4: return launch_unpacked<4>(p, st);
    }
    return TQ_ERR_UNSUPPORTED;
}
