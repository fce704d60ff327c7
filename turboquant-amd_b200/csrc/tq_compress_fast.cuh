// Paged KV compression, fast path: tensor-core WHT + table-driven bucketize on the FMA pipe.
//
// Included by tq_compress.cu after the generic pieces (PagedParams, place_item, compress_items_generic).
//
// The generic path spends most of its issue slots in the half-rate integer/compare pipe (binary-search
// bucketize, select chains, shift-or packing) and in seven butterfly stages.  This path computes the same
// indices, signs and norms with far fewer, full-rate instructions:
//
//  * rotation (fp16 / bf16 inputs): the 128-point WHT is split by index bits.  Four bits are a 16-point transform
//    done by one m16n8k16 MMA against a constant +-1 matrix (the inputs go in exactly as loaded, the products
//    +-x are exact, accumulation is fp32), the other three are butterfly stages in registers; a lane group's
//    layout stays the one of the generic path (lane j of 4 owns dims 32 j .. 32 j + 31), so there is no shuffle.
//    The norm comes from MMAs too (diagonal of X X^T) and is known before the rotation.
//  * element arithmetic two at a time: sm_100 f32x2 instructions (fma / mul / add / sub on register pairs) do
//    the butterflies, the exactly rounded quotient u = x / (n + 1e-8) and the residual energy for two adjacent
//    dims per instruction.
//  * bucketize, 3- and 4-bit: u in [-1, 1] is mapped to one of 129 cells of width 1/64; no cell holds more than one
//    boundary (checked when the table is built; Lloyd-Max boundaries for 128 dims are >= 0.022 apart).  The
//    cell's table entry gives lo = #{boundaries below the cell}, and NB = -b * 2^126 for the boundary b inside
//    the cell (-inf when there is none), so  t = sat(u * 2^126 + NB)  is exactly [u > b]  (ties stay down,
//    as searchsorted(right=False)), and idx = lo + t.  The entry also carries the centroids.
//  * bucketize, 2-bit: comparisons t = sat(u * 2^126 - b * 2^126) without a table, whose shared-memory traffic was half of what
//    the data path of the SM can do.  A codebook symmetric about zero is halved twice (two comparisons, the second boundary by
//    a multiply-add), any other one takes all three; sums and centroids are two dims to an instruction.
//  * where the rotation is done here (fp16 / bf16 rows), u = y * (1 / (n + 1e-8)) is a plain product, the centroid one FMA
//    (c[lo] + t (c[lo+1] - c[lo])), and ||residual|| = n ||u - c|| is scaled once per vector.
//  * packing: the four indices of a chunk of adjacent dims are combined by three FMAs into one float (one index
//    per nibble, exact below 2^24) and converted once; residual signs are shifted in with funnel shifts.
//  * rows are staged through shared memory with cp.async one group of items ahead of their use.
//
// On an already rotated input the indices, signs and norms are those of the generic path bit for bit, except
// where u or the residual falls in the subnormal range (|.| < 2^-126).  With the rotation done here, the
// rotated values themselves differ from a butterfly or a matrix product in the last bits, as any two
// summation orders do.  A codebook with two boundaries inside one cell makes the whole grid take the generic
// path; fp32 inputs and already rotated inputs take the table-driven quantizer without the tensor-core part.
#pragma once

namespace tq {
namespace {

// What bounds it: issue (58 to 63 % of the cycles with 16 warps per SM, which is what 128 registers allow; a build at 80
// registers and 24 warps per SM spilled and measured 1.3-1.6x slower), so what counts is how many instructions an item takes: 108 with
// 2 bits (133 before indices and centroids went two to an instruction), us in a graph for 8 KV heads: 1 M tokens of turbo2
// 1505 -> 1420, and 1368 with the slots requested a key ahead of their use (single calls 1615 -> 1520); 256 K of turbo3 416 -> 381
// -> 377, of turbo4 351 -> 340 -> 336 to 346.
// One CTA of 16 warps per SM builds the tables once for all of them: 4 % faster than two CTAs of 8 warps.
#ifndef TQ_CMP_MINBLOCKS
#define TQ_CMP_MINBLOCKS 1
#endif
#ifndef TQ_CMP_WARPS
#define TQ_CMP_WARPS 16
#endif
constexpr int kCellScale = 64;   // cells per unit of u
constexpr int kCells = 2 * kCellScale + 1;
constexpr int kFastWarps = TQ_CMP_WARPS;
constexpr int kFastItemsPerCta = kFastWarps * kItemsPerWarp;
constexpr uint32_t kMagicBits = 0x4B400000u;   // 1.5 * 2^23: adding it leaves an integer in the low mantissa bits
constexpr float kMagic = 12582912.f;

__device__ __forceinline__ float big() { return __uint_as_float(0x7E800000u); }   // 2^126

__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float4 lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

__device__ __forceinline__ float2 lds64(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}

// D = A B with a zero accumulator (no register moves to clear one).
template <bool BF16>
__device__ __forceinline__ void mma_16816_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                uint32_t b0, uint32_t b1) {
    const float z = 0.f;
    if constexpr (BF16) {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(z));
    } else {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(z));
    }
}

// ---- tables ------------------------------------------------------------------------------------------
// Each cell is stored once per lane residue so that a warp's lookups never collide on a bank:
// wide entries (16 B: NB, lo, c[lo], c[lo+1]) 8 copies, narrow entries (8 B: NB, lo) 16 copies; 128 B per cell.
constexpr int kCellStride = 128;
constexpr int kTableBytes = kCells * kCellStride;

// Scans sorted boundaries for one cell.  Returns how many boundaries fall inside the cell.
template <int NB>
__device__ __forceinline__ int scan_cell(int cell, const float* __restrict__ b, int& lo, float& nbv) {
    const float center = static_cast<float>(cell - kCellScale) * (1.f / kCellScale);
    const float half = 0.5f / kCellScale + 1.f / 1048576.f;   // rounding of the cell index is absorbed by the margin
    const float lo_e = center - half, hi_e = center + half;
    int inside = 0;
    float bin = 0.f;
    lo = 0;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        const float bj = __ldg(b + j);
        lo += bj < lo_e ? 1 : 0;
        if (bj >= lo_e && bj <= hi_e) {
            ++inside;
            bin = bj;
        }
    }
    nbv = inside ? -(bin * big()) : __uint_as_float(0xff800000u);
    return inside;
}

// d with -c_lo + d == -c_hi in fp32, to within an ulp: the rounded difference, or its neighbour against the error.  There need be no
// exact one where c_hi has finer ulps than the sum; the residual then sees a centroid one ulp away.
__device__ __forceinline__ float centroid_step(float c_lo, float c_hi) {
    float d = c_lo - c_hi;
    const float off = (d - c_lo) + c_hi;
    if (off > 0.f) d = nextafterf(d, -INFINITY);
    if (off < 0.f) d = nextafterf(d, INFINITY);
    return d;
}

// Wide entries hold (NB, lo, c[lo], c[lo+1]), or, STEP, (NB, lo, -c[lo], c[lo] - c[lo+1]).  Four lanes write the 128 bytes
// of a cell.
template <int BITS, bool WIDE, bool STEP = false>
__device__ void build_table(unsigned char* tab, const float* __restrict__ b, const float* __restrict__ c, int* bad) {
    const int lane = threadIdx.x & 31;
    for (int cell = (threadIdx.x >> 5) * 8 + (lane >> 2); cell < kCells; cell += static_cast<int>(blockDim.x) / 4) {
        int lo;
        float nbv;
        const int inside = scan_cell<(1 << BITS) - 1>(cell, b, lo, nbv);
        if (inside > 1) atomicOr(bad, 1);
        float4* dst = reinterpret_cast<float4*>(tab + cell * kCellStride) + 2 * (lane & 3);
        float4 e = make_float4(nbv, static_cast<float>(lo), nbv, static_cast<float>(lo));
        if constexpr (WIDE) {
            const float c_lo = __ldg(c + lo);
            const float c_hi = lo + 1 < (1 << BITS) ? __ldg(c + lo + 1) : c_lo;
            e.z = STEP ? -c_lo : c_lo;
            e.w = STEP ? centroid_step(c_lo, c_hi) : c_hi;
        }
        dst[0] = e;
        dst[1] = e;
    }
}

// ---- packed output (bit positions: turboquant/kernels/paged_layout.py) ------------------------------------
// Both parts of a page are made of 16-bit fields of four nibbles; a chunk of four adjacent dims fills one field
// (4-bit, 3-bit) or half the bits of one (2-bit).  K: field 2 w + h is half h of index word w of the lane's
// quarter sub-record.  V: field BITS gg + j is plane j of dim group 2 quarter + gg.  3-bit indices of the last
// two chunks (K) / of every fourth chunk (V) are spread over the spare top bits of the nibbles: bit b of the
// index in nibble e goes to bit 4 e + 3 of field / word b.
struct Packed {
    uint32_t word[4];    // K: the BITS index words of the lane's quarter sub-record
    uint32_t field[8];   // V: 2 * BITS fields (only the low 16 bits of each are meaningful)
    uint32_t signs;      // bit l = 1 when the residual of local dim l is >= 0
    float norm, rnorm;
};

// ---- two fp32 per instruction (sm_100 f32x2 arithmetic on 64-bit register pairs) ----------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2pack(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2unpack(f2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2dup(float v) { return f2pack(v, v); }
__device__ __forceinline__ f2 f2fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2sub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Per-vector constants of the element loop, duplicated into both halves of a pair.
struct VecConsts {
    f2 inv, nden, inv64, n;
    uint32_t tab;
};

// One pair of adjacent dims (a = even, b = odd): returns their indices as floats; with QJL also accumulates the
// squared residuals and shifts the sign bits of the two residuals into `sacc` (1 = negative; pairs must come in
// descending order).  A residual that underflows to -0.0 is the one case that reads as negative here while the
// reference's (e >= 0) calls it positive.
// EXACT: u = y / den correctly rounded (one reciprocal multiply plus two correction FMAs), as the reference's true
// division; needed where the input is already rotated and the indices must be the reference's bit for bit.  Where the
// rotation is done here its own rounding already moves u in the last bits, so the kernels that rotate take the plain
// product y * (1 / den), at most one ulp away: a different index only for u within an ulp of a boundary (~1e-7 of
// the coordinates, inside the rotation's 1e-4 allowance).
template <bool QJL, bool EXACT = true>
__device__ __forceinline__ void quant_pair(f2 y, const VecConsts& vc, f2& rr, uint32_t& sacc, float& kfa, float& kfb) {
    const float kBig = big();
    const f2 q0 = f2mul(y, vc.inv);
    // The cell only needs the quotient to ~1e-6: take it from the first approximation so the lookup starts early.
    const f2 cellf = f2fma(y, vc.inv64, f2dup(kMagic + kCellScale));   // low mantissa bits: round(scale u) + scale
    const f2 u = EXACT ? f2fma(f2fma(q0, vc.nden, y), vc.inv, q0) : q0;   // y / den (correctly rounded when EXACT); |u| <= 1
    float ua, ub, cfa, cfb;
    f2unpack(u, ua, ub);
    f2unpack(cellf, cfa, cfb);
    const uint32_t addr_a = __float_as_uint(cfa) * static_cast<uint32_t>(kCellStride) + vc.tab;
    const uint32_t addr_b = __float_as_uint(cfb) * static_cast<uint32_t>(kCellStride) + vc.tab;
    if constexpr (QJL) {
        const float4 ea = lds128(addr_a), eb = lds128(addr_b);   // NB, lo, c[lo], c[lo+1]
        const float ta = fma_sat(ua, kBig, ea.x), tb = fma_sat(ub, kBig, eb.x);   // [u > boundary of the cell]
        const float ca = fmaf(ta, ea.w, fmaf(-ta, ea.z, ea.z));   // t is 0 or 1: exactly c[lo] or c[lo+1]
        const float cb = fmaf(tb, eb.w, fmaf(-tb, eb.z, eb.z));
        const f2 r = f2mul(f2sub(u, f2pack(ca, cb)), vc.n);
        rr = f2fma(r, r, rr);
        float ra, rb;
        f2unpack(r, ra, rb);
        // shift the two sign bits in from the right (1 = negative; the caller inverts): one funnel shift each
        sacc = __funnelshift_l(__float_as_uint(rb), sacc, 1);
        sacc = __funnelshift_l(__float_as_uint(ra), sacc, 1);
        kfa = ea.y + ta;
        kfb = eb.y + tb;
    } else {
        const float2 ea = lds64(addr_a), eb = lds64(addr_b);     // NB, lo
        kfa = ea.y + fma_sat(ua, kBig, ea.x);
        kfb = eb.y + fma_sat(ub, kBig, eb.x);
    }
}

// The same for rows rotated here: u is the plain product, residuals are not yet multiplied by the norm.
template <int BITS>
struct Codebook2 {};   // 3 and 4 bits: everything is in the table
// 2 bits by three comparisons: -b_j * 2^126; -c_0 and the steps from -c_(j-1) to -c_j.
struct Comparisons2 {
    float nb[3], nc0, nc[3];
};
// 2 bits, halving the codebook twice: t = [u > b_1], then t' = [u > b_0] or [u > b_2], idx = 2 t + t'.  The second boundary is a
// multiply-add away from the first, and the step to the second centroid of either half is the same, in a codebook symmetric about
// zero; `split` says that these sums give what the comparisons give.  Any other codebook takes the comparisons as they are, whose
// constants wait in shared memory; also one with a boundary at or near infinity (a padded codebook), as 0 times an infinite distance
// would be NaN.
template <>
struct Codebook2<2> {
    float nb_1;                          // -b_j * 2^126
    f2 nb_0, nb_0to2;
    f2 nc_0, step_01, step_12;           // -c_0, and the steps from -c_j to -c_(j+1)
    const Comparisons2* comparisons;
    bool split;
    __device__ __forceinline__ void load(const float* __restrict__ b, const float* __restrict__ c, Comparisons2* of_warp, int lane) {
        Comparisons2 k;
#pragma unroll
        for (int j = 0; j < 3; ++j) k.nb[j] = -(__ldg(b + j) * big());
        k.nc0 = c ? -__ldg(c) : 0.f;
#pragma unroll
        for (int j = 0; j < 3; ++j) k.nc[j] = c ? centroid_step(__ldg(c + j), __ldg(c + j + 1)) : 0.f;
        if (lane == 0) *of_warp = k;
        __syncwarp();
        comparisons = of_warp;
        const float db = centroid_step(-k.nb[0], -k.nb[2]), n2 = (k.nc0 + k.nc[0]) + k.nc[1];
        split = __all_sync(0xffffffffu, k.nb[0] >= k.nb[1] && k.nb[1] >= k.nb[2] && k.nb[0] + db == k.nb[2] && n2 + k.nc[0] == n2 + k.nc[2] &&
                                     fabsf(db) < INFINITY && fabsf(n2 + k.nc[0]) < INFINITY);
        nb_1 = k.nb[1];
        nb_0 = f2dup(k.nb[0]);
        nb_0to2 = f2dup(db);
        nc_0 = f2dup(k.nc0);
        step_01 = f2dup(k.nc[0]);
        step_12 = f2dup(k.nc[1]);
    }
};

struct RowConsts {
    f2 inv, inv64;
    uint32_t tab;
};

// kf: the pair's two indices.
template <int BITS, bool QJL, class Book>
__device__ __forceinline__ void quant_pair_rotated(f2 y, const RowConsts& rc, const Book& cb, f2& ee, uint32_t& sacc, f2& kf) {
    const float kBig = big();
    const f2 u = f2mul(y, rc.inv);
    float ua, ub;
    f2unpack(u, ua, ub);
    f2 nc = f2dup(0.f);   // minus the centroids
    if constexpr (BITS == 2) {
        // only the comparisons saturate and take one value at a time: the rest is two dims to an instruction
        if constexpr (std::is_same_v<Book, Codebook2<2>>) {
            const f2 t = f2pack(fma_sat(ua, kBig, cb.nb_1), fma_sat(ub, kBig, cb.nb_1));
            float na, nb;
            f2unpack(f2fma(t, cb.nb_0to2, cb.nb_0), na, nb);
            const f2 t2 = f2pack(fma_sat(ua, kBig, na), fma_sat(ub, kBig, nb));
            kf = f2fma(t, f2dup(2.f), t2);
            if constexpr (QJL) nc = f2fma(t2, cb.step_01, f2fma(t, cb.step_12, f2fma(t, cb.step_01, cb.nc_0)));
        } else {
            const f2 t0 = f2pack(fma_sat(ua, kBig, cb.nb[0]), fma_sat(ub, kBig, cb.nb[0]));
            const f2 t1 = f2pack(fma_sat(ua, kBig, cb.nb[1]), fma_sat(ub, kBig, cb.nb[1]));
            const f2 t2 = f2pack(fma_sat(ua, kBig, cb.nb[2]), fma_sat(ub, kBig, cb.nb[2]));
            kf = f2add(f2add(t0, t1), t2);
            if constexpr (QJL) nc = f2fma(t2, f2dup(cb.nc[2]), f2fma(t1, f2dup(cb.nc[1]), f2fma(t0, f2dup(cb.nc[0]), f2dup(cb.nc0))));
        }
    } else {
        const f2 cellf = f2fma(y, rc.inv64, f2dup(kMagic + kCellScale));   // low mantissa bits: round(scale u) + scale
        float cfa, cfb;
        f2unpack(cellf, cfa, cfb);
        const uint32_t addr_a = __float_as_uint(cfa) * static_cast<uint32_t>(kCellStride) + rc.tab;
        const uint32_t addr_b = __float_as_uint(cfb) * static_cast<uint32_t>(kCellStride) + rc.tab;
        if constexpr (QJL) {
            const float4 ea = lds128(addr_a), eb = lds128(addr_b);   // NB, lo, -c[lo], c[lo] - c[lo+1]
            const float ta = fma_sat(ua, kBig, ea.x), tb = fma_sat(ub, kBig, eb.x);
            nc = f2pack(fmaf(ta, ea.w, ea.z), fmaf(tb, eb.w, eb.z));
            kf = f2pack(ea.y + ta, eb.y + tb);
        } else {
            const float2 ea = lds64(addr_a), eb = lds64(addr_b);     // NB, lo
            kf = f2pack(ea.y + fma_sat(ua, kBig, ea.x), eb.y + fma_sat(ub, kBig, eb.x));
        }
    }
    if constexpr (QJL) {
        const f2 e = f2add(u, nc);
        ee = f2fma(e, e, ee);
        float e0, e1;
        f2unpack(e, e0, e1);
        sacc = __funnelshift_l(__float_as_uint(e1), sacc, 1);
        sacc = __funnelshift_l(__float_as_uint(e0), sacc, 1);
    }
}

// cv[c]: the four indices of chunk c (dims 4 c .. 4 c + 3), one per nibble, as a float.
template <int BITS, bool ISV>
__device__ __forceinline__ void assemble_indices(const float (&cv)[8], Packed& out) {
    // Adding 2^23 leaves a field's integer in the low mantissa bits; prmt 0x5410 joins two low halves.
    const float kInt = 8388608.f;
    if constexpr (ISV) {
        // V: field BITS gg + j of dim group gg (chunks 4 gg .. 4 gg + 3).
#pragma unroll
        for (int gg = 0; gg < 2; ++gg) {
            if constexpr (BITS == 4) {
#pragma unroll
                for (int j = 0; j < 4; ++j) out.field[4 * gg + j] = __float_as_uint(cv[4 * gg + j] + kInt);
            } else if constexpr (BITS == 3) {
                const uint32_t m = __float_as_uint(cv[4 * gg + 3] + kInt);   // fourth chunk: bit b of nibble e -> field b bit 4 e + 3
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    out.field[3 * gg + b] = __float_as_uint(cv[4 * gg + b] + kInt) | ((m << (3 - b)) & 0x8888u);
            } else {
                out.field[2 * gg] = __float_as_uint(fmaf(cv[4 * gg + 1], 4.f, cv[4 * gg]) + kInt);
                out.field[2 * gg + 1] = __float_as_uint(fmaf(cv[4 * gg + 3], 4.f, cv[4 * gg + 2]) + kInt);
            }
        }
    } else {
        // K: 16-bit half h of index word w.
        if constexpr (BITS == 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                out.word[j] = prmt(__float_as_uint(cv[2 * j] + kInt), __float_as_uint(cv[2 * j + 1] + kInt), 0x5410);
        } else if constexpr (BITS == 3) {
            const uint32_t m = prmt(__float_as_uint(cv[6] + kInt), __float_as_uint(cv[7] + kInt), 0x5410);
#pragma unroll
            for (int b = 0; b < 3; ++b)
                out.word[b] = prmt(__float_as_uint(cv[2 * b] + kInt), __float_as_uint(cv[2 * b + 1] + kInt), 0x5410) |
                              ((m << (3 - b)) & 0x88888888u);
        } else {
            // word w: chunks 4 w + {0, 2} in the low half (the second shifted by 2 bits), 4 w + {1, 3} in the high half
#pragma unroll
            for (int j = 0; j < 2; ++j)
                out.word[j] = prmt(__float_as_uint(fmaf(cv[4 * j + 2], 4.f, cv[4 * j]) + kInt),
                                   __float_as_uint(fmaf(cv[4 * j + 3], 4.f, cv[4 * j + 1]) + kInt), 0x5410);
        }
    }
}

// Contiguous outputs (reference byte layouts: 2-bit four per byte LSB first, 4-bit low nibble first, 3-bit a
// little-endian bit stream): cv[c] holds the four indices of chunk c densely, idx_e at bit BITS * e, so a chunk is
// 4 * BITS bits of the lane's BITS output words.
template <int BITS>
__device__ __forceinline__ void assemble_contig(const float (&cv)[8], Packed& out) {
    const float kInt = 8388608.f;
    uint32_t u[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) u[c] = __float_as_uint(cv[c] + kInt);   // 0x4B000000 | value
    if constexpr (BITS == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) out.word[j] = prmt(u[2 * j], u[2 * j + 1], 0x5410);
    } else if constexpr (BITS == 2) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
            out.word[j] = prmt(prmt(u[4 * j], u[4 * j + 1], 0x0040), prmt(u[4 * j + 2], u[4 * j + 3], 0x0040), 0x5410);
    } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) u[c] &= 0xfffu;
        out.word[0] = u[0] | (u[1] << 12) | (u[2] << 24);
        out.word[1] = (u[2] >> 8) | (u[3] << 4) | (u[4] << 16) | (u[5] << 28);
        out.word[2] = (u[5] >> 4) | (u[6] << 8) | (u[7] << 20);
    }
}

// y: this lane's 32 rotated values as 16 pairs of adjacent dims, still to be multiplied by `scale` (2^-3.5 after
// the unnormalised WHT, else 1).  tab: shared address of this lane's copy of cell 0, minus kMagicBits * 128.
// The scale is applied to the norm only: u = (scale y) / (n + 1e-8) is computed as y / ((n + 1e-8) / scale),
// which is the same number up to the rounding the rotation itself carries; with scale = 1 nothing changes.
template <int BITS, bool QJL, bool ISV, bool CONTIG = false>
__device__ __forceinline__ void quantize_fast(f2 (&y)[16], float scale, float inv_scale, uint32_t tab, Packed& out) {
    constexpr float kStep = CONTIG ? static_cast<float>(1 << BITS) : 16.f;   // spacing of a chunk's four indices
    f2 sa = f2dup(0.f), sb = f2dup(0.f);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        sa = f2fma(y[i], y[i], sa);
        sb = f2fma(y[i + 1], y[i + 1], sb);
    }
    float s0, s1, s2, s3;
    f2unpack(sa, s0, s1);
    f2unpack(sb, s2, s3);
    const float ny = sqrtf(group_sum((s0 + s1) + (s2 + s3)));
    // NaN or overflow somewhere in the vector: quantize a zero vector so that the table lookups stay in range
    // (the stored norm still shows the bad value).
    const bool finite = ny < __uint_as_float(0x7f800000u);
    if (!finite) {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = f2dup(0.f);
    }
    const float n_out = ny * scale;
    const float n = finite ? n_out : 0.f;
    const float den = (n + 1e-8f) * inv_scale;
    const float inv = __frcp_rn(den);
    VecConsts vc;
    vc.inv = f2dup(inv);
    vc.nden = f2dup(-den);
    vc.inv64 = f2dup(inv * kCellScale);
    vc.n = f2dup(n);
    vc.tab = tab;
    // Chunk c = dims 4 c .. 4 c + 3 -> one float holding its four indices, one per nibble.
    float cv[8];
    f2 rr = f2dup(0.f);
    uint32_t sg[2] = {0u, 0u};
#pragma unroll
    for (int c = 7; c >= 0; --c) {
        float k0, k1, k2, k3;
        quant_pair<QJL>(y[2 * c + 1], vc, rr, sg[c >> 2], k2, k3);
        quant_pair<QJL>(y[2 * c], vc, rr, sg[c >> 2], k0, k1);
        cv[c] = fmaf(fmaf(fmaf(k3, kStep, k2), kStep, k1), kStep, k0);
    }
    if constexpr (CONTIG) assemble_contig<BITS>(cv, out);
    else assemble_indices<BITS, ISV>(cv, out);
    if constexpr (QJL) {
        float ra, rb;
        out.signs = ~prmt(sg[0], sg[1], 0x5410);
        f2unpack(rr, ra, rb);
        out.rnorm = sqrtf(group_sum(ra + rb));
    } else {
        out.signs = 0u;
        out.rnorm = 0.f;
    }
    out.norm = n_out;
}

// ---- rotation + quantization of one fp16 / bf16 row on the tensor cores -----------------------------------------
// A lane's 64 bytes of a row are four 16-byte pieces j = 0..3 = dims 8 j .. 8 j + 7; piece j goes into an m16n8k16
// MMA exactly as loaded, as its A fragment (a0..a3 = the four words): the 8 items of the warp are rows 0..7 with
// the words whose dim bit 1 is 0, rows 8..15 the same items with dim bit 1 = 1; the 16 k-slots are dim bit 0
// (element within a word), dim bits 5,6 (lane within the group of four) and dim bit 2 (word pair).
//  * Rotation: against the constant +-1 matrix whose column n carries the same bit roles, lane (g, t) receives the
//    16-point transform over dim bits {0,2,5,6} for dim bits 5,6 = t - the 32 dims it owns - in two passes (dim bit
//    2 = nt).  The four outputs of MMA (j, nt) are the chunk of four adjacent dims 8 j + 4 nt .. + 3, as two
//    register pairs.  Dim bits {1,3,4} are three butterfly stages over the eight pairs of a pass.
//  * Norm: m16n8k8 MMAs with a word pair as A and one of its words as B accumulate <x_g, x_n> over the even
//    (rows 0..7) and the odd (rows 8..15) words; the diagonal is ||x||^2 = ||x H||^2 (H is orthonormal), so the
//    norm is known before the rotation and only half of the rotated values have to be live at a time.
struct WhtFragments {
    uint32_t b0[2], b1[2];   // B operand (16 x 8, +-1.0 in the input type) for nt = 0, 1
};

// What the rows of a launch are: already rotated or fp32 (no tensor cores), or fp16 / bf16 rows still to be rotated.  A template
// parameter: decided at run time, both kinds of every MMA were issued, one of them predicated off.
enum class Rows { kPlain, kF16, kBF16 };

__device__ __forceinline__ WhtFragments make_wht_fragments(int lane, bool bf16) {
    const int g = lane >> 2, tig = lane & 3;
    const uint32_t one = bf16 ? 0x3F80u : 0x3C00u;
    WhtFragments f;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
        const int n = g + 8 * nt;
        const uint32_t s00 = (__popc((2 * tig) & n) & 1) << 15, s01 = (__popc((2 * tig + 1) & n) & 1) << 15;
        const uint32_t s10 = (__popc((2 * tig + 8) & n) & 1) << 15, s11 = (__popc((2 * tig + 9) & n) & 1) << 15;
        f.b0[nt] = (one | s00) | ((one | s01) << 16);
        f.b1[nt] = (one | s10) | ((one | s11) << 16);
    }
    return f;
}

// D (+)= A B, m16n8k8, fp32 accumulate; ZERO starts from a zero accumulator.
template <bool BF16, bool ZERO>
__device__ __forceinline__ void mma_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    const float z = 0.f;
    if constexpr (BF16) {
        if constexpr (ZERO)
            asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                         : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "f"(z));
        else
            asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                         : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
    } else {
        if constexpr (ZERO)
            asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                         : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "f"(z));
        else
            asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                         : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
    }
}

// row: staged_at(...) of this lane (piece j is at row ^ 16 j).
__device__ __forceinline__ void read_staged(uint32_t row, uint32_t (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(w[4 * j]), "=r"(w[4 * j + 1]), "=r"(w[4 * j + 2]), "=r"(w[4 * j + 3])
                     : "r"(row ^ (16 * j)));
}

// after_read() is called once the staged row has been read for the last time (the caller requests the next row
// into the same buffer there).  Lanes past the end of the input quantize whatever their buffer holds; nobody stores it.
template <bool BF16, int BITS, bool QJL, bool ISV, bool CONTIG = false, class AfterRead>
__device__ __forceinline__ void compress_row_mma(uint32_t row, int lane, const WhtFragments& hf,
                                                 uint32_t tab, const Codebook2<BITS>& cb, Packed& out, AfterRead after_read) {
    constexpr float kStep = CONTIG ? static_cast<float>(1 << BITS) : 16.f;   // spacing of a chunk's four indices
    uint32_t w[16];
    read_staged(row, w);
    // ||x||^2: even words on the diagonal of rows 0..7 of da, odd words on that of rows 8..15 of db
    float da[4], db[4];
    mma_k8<BF16, true>(da, w[0], w[1], w[0]);
    mma_k8<BF16, true>(db, w[0], w[1], w[1]);
#pragma unroll
    for (int m = 1; m < 8; ++m) {
        mma_k8<BF16, false>(da, w[2 * m], w[2 * m + 1], w[2 * m]);
        mma_k8<BF16, false>(db, w[2 * m], w[2 * m + 1], w[2 * m + 1]);
    }
    const int g = lane >> 2;
    const float diag = (g & 1) ? da[1] + db[3] : da[0] + db[2];   // column g sits in lane (g, g >> 1)
    const float ss = __shfl_sync(0xffffffffu, diag, (lane & ~3) | (g >> 1));
    // NaN or overflow somewhere in the vector: quantize a zero vector so that the table lookups stay in range (the
    // stored norm still shows the bad value).
    const bool finite = ss < __uint_as_float(0x7f800000u);
    // (as zeros in the buffer, behind a branch: 16 predicated moves of zero a row were 4 % of the instructions)
    if (!__all_sync(0xffffffffu, finite)) {
        if (!finite) {
#pragma unroll
            for (int j = 0; j < 4; ++j) asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(row ^ (16 * j)), "r"(0) : "memory");
        }
        read_staged(row, w);
    }
    const float n_out = sqrtf(ss);                                // = ||x H / sqrt(128)||
    const float n = finite ? n_out : 0.f;
    const float den = (n + 1e-8f) * 11.313708498984761f;          // the unnormalised transform is sqrt(128) larger
    const float inv = __frcp_rn(den);
    RowConsts rc;
    rc.inv = f2dup(inv);
    rc.inv64 = f2dup(inv * kCellScale);
    rc.tab = tab;
    float cv[8];
    f2 ee = f2dup(0.f);
    uint32_t sg = 0u;   // bit l = 1 when the residual of local dim l is negative
    auto quantize = [&](const auto& book) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            if (nt == 1) {
                read_staged(row, w);
                __syncwarp();
                after_read();
            }
            f2 y[8];   // pair 2 j + r = dims 8 j + 4 nt + 2 r + {0, 1}
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float d[4];
                mma_16816_zero<BF16>(d, w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3], hf.b0[nt], hf.b1[nt]);
                y[2 * j] = f2pack(d[0], d[1]);
                y[2 * j + 1] = f2pack(d[2], d[3]);
            }
#pragma unroll
            for (int h = 1; h < 8; h <<= 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (!(i & h)) {
                        const f2 a = y[i], b = y[i + h];
                        y[i] = f2add(a, b);
                        y[i + h] = f2sub(a, b);
                    }
                }
            }
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                const int c = 2 * j + nt;   // chunk of dims 4 c .. 4 c + 3
                f2 k01, k23;
                uint32_t nib = 0u;
                quant_pair_rotated<BITS, QJL>(y[2 * j + 1], rc, book, ee, nib, k23);
                quant_pair_rotated<BITS, QJL>(y[2 * j], rc, book, ee, nib, k01);
                float a, b;
                if constexpr (BITS == 4 && QJL && CONTIG) {   // one register short for the form below: 200 us for 1 M rows of K and V instead of 197
                    float k0, k1;
                    f2unpack(k01, k0, k1);
                    f2unpack(k23, a, b);
                    cv[c] = fmaf(fmaf(fmaf(b, kStep, a), kStep, k1), kStep, k0);
                } else {
                    f2unpack(f2fma(k23, f2dup(kStep * kStep), k01), a, b);   // indices 0 and 2, 1 and 3
                    cv[c] = fmaf(b, kStep, a);
                }
                if constexpr (QJL) sg |= nib << (4 * c);
            }
        }
    };
    if constexpr (BITS == 2) {
        if (cb.split) quantize(cb);
        else quantize(Comparisons2(*cb.comparisons));
    } else {
        quantize(cb);
    }
    if constexpr (CONTIG) assemble_contig<BITS>(cv, out);
    else assemble_indices<BITS, ISV>(cv, out);
    if constexpr (QJL) {
        float ra, rb;
        out.signs = ~sg;
        f2unpack(ee, ra, rb);
        out.rnorm = n * sqrtf(group_sum(ra + rb));
    } else {
        out.signs = 0u;
        out.rnorm = 0.f;
    }
    out.norm = n_out;
}

// ---- input staging (fp16 / bf16 rows): global -> shared with cp.async, one group of items ahead --------------
// The four lanes of a row copy 64 contiguous bytes per instruction (whole sectors: with each lane copying its own 64 bytes,
// 16 at a time, every sector crossed from L2 twice) and read back 64 bytes each.  16-byte chunk c of row g sits at slot
// c ^ (c >> 2) ^ 4 (g & 1) of the row's 256 bytes, so neither the copies nor the reads of a warp collide on a bank.
constexpr int kStagePerWarp = 2 * 4 * 32 * 16;   // K and V rows of 8 items: 4 KB
constexpr int kRowBuffer = kStagePerWarp / 2;    // on a 256-byte boundary

// Chunk 4 i + quarter of this lane's row is copied to stage_at ^ 0x50 i, chunk 4 quarter + j is read from staged_at ^ 0x10 j.
__device__ __forceinline__ uint32_t stage_at(uint32_t buf, int lane) {
    const int g = lane >> 2, quarter = lane & 3;
    return buf + g * 256 + ((g & 1) << 6) + (quarter << 4);
}
__device__ __forceinline__ uint32_t staged_at(uint32_t buf, int lane) {
    const int g = lane >> 2, quarter = lane & 3;
    return buf + g * 256 + ((quarter ^ (g & 1)) << 6) + (quarter << 4);
}

// elem_off: of the row's first element plus 8 * quarter.  The lanes of the warp have read what the buffer held before.
__device__ __forceinline__ void stage_row(uint32_t dst, const void* base, int64_t elem_off, bool live) {
    if (live) {
        const uint16_t* src = static_cast<const uint16_t*>(base) + elem_off;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst ^ (0x50 * i)), "l"(src + 32 * i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Waits until at most one of the copy groups of each lane is still in flight.
__device__ __forceinline__ void wait_staged() {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
}

// Loads this lane's 32 elements of one row and returns them as fp32 pairs, rotated when asked but not yet
// scaled by 2^-3.5.  Path for fp32 inputs and for inputs that are already rotated.
__device__ __forceinline__ void fetch_plain(const void* base, int64_t elem_off, bool live, int dtype, bool rotate,
                                            int lane, f2 (&y)[16]) {
    float x[32];
    if (live) load32(base, elem_off, dtype, x);
    else {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = 0.f;
    }
    if (rotate) fwht128(x, lane);
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = f2pack(x[2 * i], x[2 * i + 1]);
}

// ---- stores ------------------------------------------------------------------------------------------------
template <int BITS, bool QJL>
__device__ __forceinline__ void store_k_fast(uint8_t* page, int t, int quarter, const Packed& q) {
    constexpr int NW = BITS + (QJL ? 1 : 0);
    constexpr int RK = 16 * NW;
    const uint32_t (&w)[4] = q.word;
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

template <int BITS>
__device__ __forceinline__ void store_v_fast(uint8_t* vpart, int t, int quarter, const Packed& q) {
    const int pair = t >> 1, half = t & 1;
#pragma unroll
    for (int gg = 0; gg < 2; ++gg) {
        const int g = 2 * quarter + gg;
#pragma unroll
        for (int j = 0; j < BITS; ++j)
            *reinterpret_cast<uint16_t*>(vpart + ((j * 8 + pair) * 8 + g) * 4 + half * 2) =
                static_cast<uint16_t>(q.field[gg * BITS + j]);
    }
    if (quarter == 0) reinterpret_cast<__half*>(vpart + 256 * BITS)[norm_slot(t)] = __float2half_rn(q.norm);
}

// The V fields of two lanes that hold neighbouring tokens of one 32-bit word (lane ^ 4, same quarter): the lane of the even
// token writes the words of dim group 2 quarter, the other one those of 2 quarter + 1, so a warp's store instruction fills
// whole 32-byte sectors (16-bit stores of single tokens cost 10 to 17 % of the kernel).
template <int BITS>
__device__ __forceinline__ void store_v_pair(uint8_t* vpart, int t, int quarter, const Packed& q, bool live) {
    const int pair = t >> 1, half = t & 1;
    uint8_t* dst = vpart + (pair * 8 + 2 * quarter + half) * 4;
#pragma unroll
    for (int j = 0; j < BITS; ++j) {
        const uint32_t keep = half ? q.field[BITS + j] : q.field[j], give = half ? q.field[j] : q.field[BITS + j];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 4);
        if (live) *reinterpret_cast<uint32_t*>(dst + j * 256) = prmt(keep, got, half ? 0x1054u : 0x5410u);
    }
    if (live && quarter == 0) reinterpret_cast<__half*>(vpart + 256 * BITS)[norm_slot(t)] = __float2half_rn(q.norm);
}

// fp32 inputs and inputs that are already rotated: plain loads, shuffle WHT, the same table-driven quantizer.
// Out of line so that its registers do not weigh on the tensor-core loop.
template <int KB, int VB, bool QJL>
__device__ __noinline__ void compress_items_plain(const void* key, const void* value, int64_t ks_t, int64_t ks_h,
                                                  int64_t vs_t, int64_t vs_h, int dtype, bool rotate, ItemPlace w, int lane,
                                                  uint32_t ktab, uint32_t vtab) {
    constexpr int KPART = k_part_bytes(KB, QJL ? 1 : 0);
    const int quarter = lane & 3;
    const float scale = rotate ? kWhtScale : 1.f, inv_scale = rotate ? 11.313708498984761f : 1.f;
    f2 x[16];
    Packed q;
    fetch_plain(key, w.tok * ks_t + w.head * ks_h + 32 * quarter, w.live, dtype, rotate, lane, x);
    quantize_fast<KB, QJL, false>(x, scale, inv_scale, ktab, q);
    if (w.live) store_k_fast<KB, QJL>(w.page, w.t, quarter, q);
    fetch_plain(value, w.tok * vs_t + w.head * vs_h + 32 * quarter, w.live, dtype, rotate, lane, x);
    quantize_fast<VB, false, true>(x, scale, inv_scale, vtab, q);
    if (w.live) store_v_fast<VB>(w.page + KPART, w.t, quarter, q);
}

// ---- kernel -----------------------------------------------------------------------------------------------
// Item order of the tensor-core loop: items 2 i and 2 i + 1 are two neighbouring tokens of one head (for store_v_pair);
// with an odd token count the last partner is not live.
__device__ __forceinline__ uint32_t paired_items(const PagedParams& p) { return static_cast<uint32_t>(p.n_tokens + 1) / 2 * 2 * p.Hkv; }
__device__ __forceinline__ ItemId identify_paired(const PagedParams& p, uint32_t item) {
    ItemId id;
    const uint32_t two = item >> 1, tp = p.div_heads(two);
    id.head = static_cast<int>(two - tp * p.Hkv);
    id.tok = 2 * tp + (item & 1);
    id.live = id.tok < p.n_tokens;
    return id;
}

// Persistent CTAs of 16 warps, one per SM: the tables are built once per CTA, then its warps stride over units of 8 (token,
// head) items, first the keys then the values of a unit.  Unit u belongs to warp u / gridDim of CTA u % gridDim: the last,
// partly filled round is spread over all SMs (3001 tokens x 8 heads: 2 rounds of 16 warps per SM on 40 SMs otherwise).
template <int KB, int VB, bool QJL, Rows ROWS>
__global__ void __launch_bounds__(kFastWarps * 32, TQ_CMP_MINBLOCKS) compress_paged_fast_kernel(const __grid_constant__ PagedParams p, uint32_t n_groups) {
    constexpr int PAGE = page_bytes(KB, VB, QJL ? 1 : 0);
    constexpr int KPART = k_part_bytes(KB, QJL ? 1 : 0);
    extern __shared__ __align__(128) unsigned char tables[];
    __shared__ float csm[1 << KB];
    __shared__ int bad;
    __shared__ Comparisons2 comparisons[KB == 2 || VB == 2 ? kFastWarps : 1][2];
    const int lane = threadIdx.x & 31, quarter = lane & 3, warp = threadIdx.x >> 5;
    constexpr uint32_t kBias = kMagicBits * static_cast<uint32_t>(kCellStride);   // modulo 2^32
    const uint32_t ktab = smem_u32(tables) + (QJL ? (lane & 7) * 16 : (lane & 15) * 8) - kBias;
    const uint32_t vtab = smem_u32(tables + kTableBytes) + (lane & 15) * 8 - kBias;
    constexpr bool mma = ROWS != Rows::kPlain, BF16 = ROWS == Rows::kBF16;

    pdl_wait();
    pdl_release();
    // Tensor-core path.  Rows are staged through shared memory one unit ahead: the key rows of the next unit are requested
    // as soon as this unit's have been consumed by the MMAs, the value rows likewise, so every copy has a whole unit's
    // arithmetic to hide behind.  The first ones are under way while the tables are built.
    const uint32_t kbuf = ((smem_u32(tables) + 2 * kTableBytes + 255) & ~255u) + warp * kStagePerWarp, vbuf = kbuf + kRowBuffer;
    const uint32_t kdst = stage_at(kbuf, lane), vdst = stage_at(vbuf, lane);
    const uint32_t units = (paired_items(p) + kItemsPerWarp - 1) / kItemsPerWarp;
    const uint32_t step = gridDim.x * kFastWarps;
    uint32_t unit = warp * gridDim.x + blockIdx.x;
    ItemId id = identify_paired(p, unit * kItemsPerWarp + (lane >> 2));
    if constexpr (mma) {
        stage_row(kdst, p.key, id.tok * p.ks_t + id.head * p.ks_h + 8 * quarter, id.live);
        stage_row(vdst, p.value, id.tok * p.vs_t + id.head * p.vs_h + 8 * quarter, id.live);
    }
    if (threadIdx.x == 0) bad = 0;
    if (threadIdx.x < (1 << KB)) csm[threadIdx.x] = p.kc[threadIdx.x];
    __syncthreads();
    if constexpr (mma) {   // 2-bit codebooks need no table here
        if constexpr (KB > 2) build_table<KB, QJL, true>(tables, p.kb, p.kc, &bad);
        if constexpr (VB > 2) build_table<VB, false, true>(tables + kTableBytes, p.vb, nullptr, &bad);
    } else {
        build_table<KB, QJL>(tables, p.kb, p.kc, &bad);
        build_table<VB, false>(tables + kTableBytes, p.vb, nullptr, &bad);
    }
    __syncthreads();
    if (bad != 0 || !mma) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        const bool generic = bad != 0;
        const uint32_t item0 = warp * kItemsPerWarp + (lane >> 2);   // + group * 128
        for (uint32_t grp = blockIdx.x; grp < n_groups; grp += gridDim.x) {
            if (generic) compress_items_generic<KB, VB, QJL>(p, grp * kFastItemsPerCta + item0, lane, csm);
            else if constexpr (!mma)
                compress_items_plain<KB, VB, QJL>(p.key, p.value, p.ks_t, p.ks_h, p.vs_t, p.vs_h, p.in_dtype, p.rotate != 0,
                                                  place_item<PAGE>(p, grp * kFastItemsPerCta + item0, quarter), lane, ktab, vtab);
        }
        return;
    }
    const uint32_t krow = staged_at(kbuf, lane), vrow = staged_at(vbuf, lane);
    const WhtFragments hf = make_wht_fragments(lane, BF16);
    Codebook2<KB> kcb;
    Codebook2<VB> vcb;
    if constexpr (KB == 2) kcb.load(p.kb, QJL ? p.kc : nullptr, &comparisons[warp][0], lane);
    if constexpr (VB == 2) vcb.load(p.vb, nullptr, &comparisons[warp][1], lane);
    Packed q;
    // Only the identity (token, head) of the next unit's item is carried across the loop body.  The current item's slot is
    // requested at its turn and waited for when its key is done.
    while (unit < units) {
        const ItemId now = id;
        const int64_t slot = now.live ? p.slot_mapping[now.tok] : 0;
        unit += step;
        id = identify_paired(p, unit * kItemsPerWarp + (lane >> 2));
        wait_staged();
        compress_row_mma<BF16, KB, QJL, false>(krow, lane, hf, ktab, kcb, q, [&] {
            stage_row(kdst, p.key, id.tok * p.ks_t + id.head * p.ks_h + 8 * quarter, id.live);
        });
        const ItemPlace w = place_item<PAGE>(p, now, slot, quarter);
        const unsigned long long at = reinterpret_cast<unsigned long long>(w.page);
        const unsigned long long at_other = __shfl_xor_sync(0xffffffffu, at, 4);
        const int t_other = __shfl_xor_sync(0xffffffffu, w.t, 4);
        // both tokens of every pair in one word of one page, or neither of them stored (no page)
        const bool pairs = __all_sync(0xffffffffu, at_other == at && (at == 0 || t_other == (w.t ^ 1)));
        if (w.live) store_k_fast<KB, QJL>(w.page, w.t, quarter, q);
        wait_staged();
        compress_row_mma<BF16, VB, false, true>(vrow, lane, hf, vtab, vcb, q, [&] {
            stage_row(vdst, p.value, id.tok * p.vs_t + id.head * p.vs_h + 8 * quarter, id.live);
        });
        if (pairs) {
            store_v_pair<VB>(w.page + KPART, w.t, quarter, q, w.live);
        } else if (w.live) {
            store_v_fast<VB>(w.page + KPART, w.t, quarter, q);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Small launches (the new tokens of one decode step): no tables to build.  Such a launch is one chain of latencies, so
// a warp takes the keys or the values of 8 items, not both one after the other, and its rows, their slots and the codebook
// are requested together (a warp of keys holds the centroids in a copy of its own: no barrier of the CTA).  Measured, us per launch in a graph of such launches,
// both in one warp / now, 8 KV heads: turbo3 64 tokens 6.1 / 3.4, 1024 tokens 9.8 / 5.6, 2048 tokens 10.1 / 8.8; turbo4 64
// tokens 6.2 / 3.4.
template <int KB, int VB, bool QJL>
__global__ void __launch_bounds__(kWarpsPerCta * 32) compress_paged_small_kernel(const __grid_constant__ PagedParams p) {
    constexpr int PAGE = page_bytes(KB, VB, QJL ? 1 : 0);
    __shared__ float csm_of[kWarpsPerCta / 2][1 << KB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quarter = lane & 3;
    const ItemId id = identify_item(p, (static_cast<int64_t>(blockIdx.x) * (kWarpsPerCta / 2) + (warp >> 1)) * kItemsPerWarp + (lane >> 2));
    pdl_wait();
    pdl_release_if_small();
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = 0.f;   // lanes past the end take part in the shuffles
    int64_t slot = 0;
    Quarter q;
    if ((warp & 1) == 0) {
        float* csm = csm_of[warp >> 1];
        Boundaries<KB> bd;
        bd.load(p.kb);
        const float centroid = QJL ? p.kc[lane & ((1 << KB) - 1)] : 0.f;
        if (id.live) {
            slot = p.slot_mapping[id.tok];
            load32(p.key, id.tok * p.ks_t + id.head * p.ks_h + 32 * quarter, p.in_dtype, x);
        }
        if (QJL && lane < (1 << KB)) csm[lane] = centroid;
        __syncwarp();
        const ItemPlace w = place_item<PAGE>(p, id, slot, quarter);
        quantize_quarter<KB, QJL>(x, p.rotate != 0, lane, bd, csm, q);
        if (w.live) store_k_paged<KB, QJL>(w.page, w.t, quarter, q);
    } else {
        Boundaries<VB> bd;
        bd.load(p.vb);
        if (id.live) {
            slot = p.slot_mapping[id.tok];
            load32(p.value, id.tok * p.vs_t + id.head * p.vs_h + 32 * quarter, p.in_dtype, x);
        }
        const ItemPlace w = place_item<PAGE>(p, id, slot, quarter);
        quantize_quarter<VB, false>(x, p.rotate != 0, lane, bd, nullptr, q);
        if (w.live) store_v_paged<VB>(w.page + k_part_bytes(KB, QJL ? 1 : 0), w.t, quarter, q);
    }
}

// Up to here launches take the small kernel, whose rotation is the plain butterfly.  The tensor-core kernel rounds its
// rotation differently, and a coordinate in a million would go to the neighbouring centroid: the line is kept for the bytes,
// not for the time.  us, small kernel / that one: turbo3 1024 tokens 5.6 / 6.0, 2048 tokens 8.8 / 7.9; turbo4 7.0 / 5.8 and
// 10.8 / 7.4; turbo2 4.9 / 4.3 and 7.3 / 6.0.
constexpr int64_t kSmallLaunchItems = 16384;

template <int KB, int VB, bool QJL>
int launch_paged_tc(const PagedParams& p, cudaStream_t st);   // tq_compress_tc.cuh

template <int KB, int VB, bool QJL>
int launch_paged_fast(const PagedParams& p, cudaStream_t st) {
    if (p.n_items <= kSmallLaunchItems) {
        constexpr int64_t kItems = kItemsPerCta / 2;   // every item has a key warp and a value warp
        const unsigned grid = static_cast<unsigned>((p.n_items + kItems - 1) / kItems);
        return launch_chained(compress_paged_small_kernel<KB, VB, QJL>, dim3(grid), dim3(kWarpsPerCta * 32), 0, st, p) == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
    }
    // on request: fp16 / bf16 rows that still need the rotation go to the tensor-memory kernel (rotation as one
    // 128 x 128 x 128 product per 128 rows, one thread per vector afterwards)
    if (p.rotate && p.in_dtype != TQ_DTYPE_F32 && p.use_tcgen05) return launch_paged_tc<KB, VB, QJL>(p, st);
    const uint32_t n_groups = static_cast<uint32_t>((p.n_items + kFastItemsPerCta - 1) / kFastItemsPerCta);
    const int64_t n_units = (p.n_items + kItemsPerWarp - 1) / kItemsPerWarp;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TQ_ERR_LAUNCH;
    static int sm_count[64] = {0};
    if (dev >= 0 && dev < 64 && sm_count[dev]) sms = sm_count[dev];
    else {
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return TQ_ERR_LAUNCH;
        if (dev >= 0 && dev < 64) sm_count[dev] = sms;
    }
    const int64_t resident = static_cast<int64_t>(sms) * TQ_CMP_MINBLOCKS;
    const unsigned grid = static_cast<unsigned>(n_units < resident ? n_units : resident);
    constexpr int kSmem = 2 * kTableBytes + kFastWarps * kStagePerWarp + 256;
    auto run = [&](auto kernel, bool (&configured)[64]) {
        if (dev < 0 || dev >= 64 || !configured[dev]) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return TQ_ERR_LAUNCH;
            if (dev >= 0 && dev < 64) configured[dev] = true;
        }
        return launch_chained(kernel, dim3(grid), dim3(kFastWarps * 32), kSmem, st, p, n_groups) == cudaSuccess ? TQ_OK : TQ_ERR_LAUNCH;
    };
    static bool configured[3][64] = {};
    if (!p.rotate || p.in_dtype == TQ_DTYPE_F32) return run(compress_paged_fast_kernel<KB, VB, QJL, Rows::kPlain>, configured[0]);
    if (p.in_dtype == TQ_DTYPE_F16) return run(compress_paged_fast_kernel<KB, VB, QJL, Rows::kF16>, configured[1]);
    return run(compress_paged_fast_kernel<KB, VB, QJL, Rows::kBF16>, configured[2]);
}

}  // namespace
}  // namespace tq
