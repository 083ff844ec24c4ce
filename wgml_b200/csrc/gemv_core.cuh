// Quantised dot products on the integer tensor-core instruction: sixteen rows of a matrix staged in shared memory against
// one input vector held in shared memory.  These are the inner loops of the fused matrix-vector kernel (gemv.cu).
//
// A warp takes a unit: sixteen rows (rows g and g + 8 belong to the lanes 4g .. 4g + 3) times UnitGeom::COLS columns.  Lane t of
// such a quad owns a quarter of the unit's columns, a run of codes that shares its sub-block scales, and reads it with
// 128-bit shared loads (row pitches are padded so that they meet no bank conflicts).
//
// Arithmetic.  x of a 32-column group is written as X * 2^e with a shared exponent and a 23-bit signed X (|X| <= 2^22, rounded to
// nearest: within one bit of f32 precision for the largest element), X is split into three bytes X = 65536 d2 + 256 d1 + d0, and
// sum_l q_l X_l is taken in integers, exact in int32:
//   mma.m16n8k32, A = codes of the sixteen rows as they come out of the mask, 32 columns per instruction: eight of every lane t's
//   quarter.  B column 2t + d holds digit d of the inputs at the k positions of lane t and zeros at those of the other lanes,
//   so one instruction keeps four groups with scales of their own apart and accumulator (row g, columns 2t, 2t + 1) is the pair
//   of sums that lane t needs for its group.  d0 and d1 go in one instruction, d2 in a second.
// Sixteen rows of 256 columns of Q4_K take 16 instructions, 10.4 clocks of a scheduler each (measured; f16 operands with K = 16 the
// same, so two 12-bit digits there would need as many and more unpacking), where dp4a took 384 and a fold of every row: a warp
// issues about 235 instructions for 4096 weights where it issued 370.
// The exact integer S enters the f32 algebra of the format:
//   Q4_K  sum_l (d*sc*q_l - dmin*m) x_l = d*sc * 2^e S  -  dmin*m * sum_l x_l
//   Q6_K  sum_l d*sc*(q_l - 32) x_l     = d*sc * (2^e S - 32 * sum_l x_l)
//   Q8_0  sum_l d*q_l x_l               = d * 2^e S
// with the sums of x (f32, from the unrounded x) computed once per thread block.  Dense f32 matrices use plain f32 FMAs.
#pragma once

#include "dequant.cuh"
#include "qmatrix.cuh"

namespace wgb {

// D = A * B + D of one warp: A 16 x 32 codes, B 32 x 8 digits, int32 sums; u / s: unsigned / signed bytes.  imma0: from zeros.
#define WGB_IMMA(NAME, AT, BT)                                                                                                   \
    __device__ __forceinline__ void NAME(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) \
    {                                                                                                                            \
        asm("mma.sync.aligned.m16n8k32.row.col.s32." AT "." BT ".s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"      \
            : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])                                                                     \
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));                                                             \
    }
#define WGB_IMMA0(NAME, AT, BT)                                                                                                  \
    __device__ __forceinline__ void NAME(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) \
    {                                                                                                                            \
        asm("mma.sync.aligned.m16n8k32.row.col.s32." AT "." BT ".s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"  \
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])                                                                     \
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));                                                     \
    }
WGB_IMMA0(imma0_uu, "u8", "u8")
WGB_IMMA0(imma0_us, "u8", "s8")
WGB_IMMA0(imma0_su, "s8", "u8")
WGB_IMMA0(imma0_ss, "s8", "s8")
#undef WGB_IMMA0
WGB_IMMA(imma_uu, "u8", "u8")
WGB_IMMA(imma_us, "u8", "s8")
WGB_IMMA(imma_su, "s8", "u8")
WGB_IMMA(imma_ss, "s8", "s8")
#undef WGB_IMMA

// Unsigned byte k of a word as f32: one byte permute drops it into the mantissa of 2^23, one FP32 subtraction removes the offset.
__device__ __forceinline__ float byte2f(uint32_t w, int k)
{
    return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440 + k)) - 8388608.0f;
}

// 65536 s2 + 256 s1 + s0 as f32 for the three digit sums of one scale group.  The two low digits are joined in
// the integer unit (|256 s1 + s0| < 2^30 for every format here) and the conversion unit is used twice.  The result is the
// correctly rounded f32 of each part and one fused multiply-add, i.e. within an ulp of the exact sum.
__device__ __forceinline__ float combine3(int s2, int s1, int s0)
{
    return fmaf(__int2float_rn(s2), 65536.0f, __int2float_rn(s1 * 256 + s0));
}

// Sign-extended byte k of a word, as f32.
__device__ __forceinline__ float s8f(uint32_t w, int k) { return __int2float_rn((int)(signed char)(w >> (8 * k))); }

__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr)
{
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
// Loads into registers that keep what they hold where `on` is 0.
__device__ __forceinline__ void lds128_if(uint32_t (&r)[4], uint32_t addr, uint32_t on)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %5, 0;\n\t"
        "@p ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3])
        : "r"(addr), "r"(on));
}

// ---------------------------------------------------------------------------------------------
// Shared-memory image of the input vector (built once per thread block by XWriter).
//   quantised formats, per unit of COLS columns:
//     pair plane   2 COLS bytes: digits d0 and d1 as 16-byte chunks of 16 columns.  Chunk (t, i) -- the i-th one of lane t's
//                  quarter -- of digit d lies at i * 128 + ((2t + d) ^ f(i)) * 16: the eight chunks that a load of the warp
//                  fetches together fill the 128 bytes of a wavefront, and so do those that half a warp of writers stores.
//     top plane    COLS bytes: digit d2, chunk (t, i) at ((4i + t) ^ 2 (i / 2)) * 16
//     factors      Q4_K: per t {2^e, 2^e / 16, sum, sum} of its two 32-column groups (high nibbles enter the sums as 16 * code)
//                  Q6_K: per (t, i) {2^e, 32 * sum} of its 16 columns        Q8_0: per t 2^e of its group
//   f32:           the values, zeros up to the end of the last unit
// ---------------------------------------------------------------------------------------------
__host__ __device__ constexpr uint32_t image_units(int qt, uint32_t K) { return (K + unit_cols(qt) - 1) / unit_cols(qt); }
__host__ __device__ constexpr uint32_t factor_bytes(int qt) { return qt == WGB_Q4_K ? 64u : qt == WGB_Q6_K ? 128u : 16u; }   // per unit
__host__ __device__ constexpr size_t ximage_bytes(int qt, uint32_t K)
{
    return (size_t)image_units(qt, K) * (qt == WGB_F32 ? 4u * unit_cols(qt) : 3u * unit_cols(qt) + factor_bytes(qt));
}
__host__ __device__ constexpr uint32_t chunk_xor(uint32_t i) { return (i & 1u) | ((i >> 1) << 2); }

// Where the planes of an image of `units` units begin (shared-memory addresses).
template <int QT>
struct XImage {
    uint32_t pair, top, factors;
    __device__ __forceinline__ XImage(uint32_t base, uint32_t units)
        : pair(base), top(base + units * 2 * unit_cols(QT)), factors(base + units * 3 * unit_cols(QT)) {}
};

// Digits of one unit's inputs in the layout of the B operand, one set of registers per lane.  Lanes whose column of B is zero at
// their k positions keep the zeros they start with.
template <int N>   // chunks per lane
struct BDigits {
    uint32_t pair[N][4], top[N][4];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
            for (int k = 0; k < 4; k++) pair[i][k] = top[i][k] = 0u;
    }
    // `u`: unit of the row.  Lane 4g + t holds column g of B at the k positions of t.
    template <int QT>
    __device__ __forceinline__ void load(const XImage<QT> &im, uint32_t u, int lane)
    {
        const uint32_t g = (uint32_t)lane >> 2, t = (uint32_t)lane & 3;
        const uint32_t on = (g >> 1) == t, on_top = on & ~g & 1u;
        const uint32_t a = im.pair + u * (2 * unit_cols(QT)) + (2 * t + (g & 1)) * 16, b = im.top + u * unit_cols(QT) + t * 16;
#pragma unroll
        for (uint32_t i = 0; i < (uint32_t)N; i++) {
            lds128_if(pair[i], (a ^ (chunk_xor(i) << 4)) + i * 128, on);
            lds128_if(top[i], (b ^ ((i >> 1) << 5)) + i * 64, on_top);
        }
    }
};

// ---------------------------------------------------------------------------------------------
// Per-format products of one unit.  `sa` / `sb`: shared-memory addresses of planes of the stage for the lane's two rows (g and
// g + 8), `w` the unit's place in the stage, `u` in the row.  eval() gives the lane's partial sums of the two rows.
// ---------------------------------------------------------------------------------------------
template <int QT>
struct Unit;

// Q4_K, raw 144-byte super-blocks: lane t owns the 64-column group t (32 bytes of qs: low nibbles = first 32 columns, high
// nibbles = next 32).
template <>
struct Unit<WGB_Q4_K> {
    using Digits = BDigits<4>;

    // d * sc, d * sc, dmin * m, dmin * m of the lane's two 32-column groups: six-bit scales and mins (get_scale_min_k4,
    // quantization.rs:381-389) as the four bytes (sc_lo, sc_hi, m_lo, m_hi) of one word, without a branch: with j = 2t, 2t+1
    //   t < 2:  sc = scales[j] & 63,                        m = scales[j+4] & 63
    //   t >= 2: sc = (scales[j+4] & 15) | (scales[j-4] >> 6) << 4,  m = (scales[j+4] >> 4) | (scales[j] >> 6) << 4
    // Both cases read bytes 2(t&1), 2(t&1)+1 of hdr.y (scales 0..3) and of hdr.z (4..7); the second also
    // those bytes of hdr.w (8..11).  The selectors and masks depend on the lane only.
    __device__ static __forceinline__ float finish(const uint4 hdr, uint32_t t, float s_lo, float s_hi, const uint4 f)
    {
        const uint32_t b0 = 2u * (t & 1u);
        const uint32_t sel_yz = (b0) | ((b0 + 1u) << 4) | ((b0 + 4u) << 8) | ((b0 + 5u) << 12);   // (y[b0], y[b0+1], z[b0], z[b0+1])
        const uint32_t yz = __byte_perm(hdr.y, hdr.z, sel_yz);
        const uint32_t t2 = __byte_perm(hdr.w, hdr.w >> 4, sel_yz);                                 // (w[b0], w[b0+1], (w>>4)[b0], (w>>4)[b0+1])
        const bool high = t >= 2;
        const uint32_t scm = ((high ? t2 : yz) & (high ? 0x0f0f0f0fu : 0x3f3f3f3fu)) | ((yz >> 2) & (high ? 0x30303030u : 0u));
        const float2 dm = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
        const float pos = fmaf(byte2f(scm, 0), s_lo * __uint_as_float(f.x), byte2f(scm, 1) * (s_hi * __uint_as_float(f.y)));
        const float neg = fmaf(byte2f(scm, 2), __uint_as_float(f.z), byte2f(scm, 3) * __uint_as_float(f.w));
        return fmaf(dm.x, pos, -(dm.y * neg));
    }
    __device__ static __forceinline__ void eval(const uint32_t (&sa)[1], const uint32_t (&sb)[1], uint32_t w, const Digits &b,
                                                const XImage<WGB_Q4_K> &im, uint32_t u, int lane, float &ya, float &yb)
    {
        const uint32_t t = (uint32_t)lane & 3;
        const uint32_t ra = sa[0] + w * 144, rb = sb[0] + w * 144;
        const uint4 a0 = lds128(ra + 16 + t * 32), a1 = lds128(ra + 32 + t * 32), b0 = lds128(rb + 16 + t * 32), b1 = lds128(rb + 32 + t * 32);
        const uint32_t qa[8] = { a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w }, qb[8] = { b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w };
        const uint4 ha = lds128(ra), hb = lds128(rb), f = lds128(im.factors + u * 64 + t * 16);
        int lo[4], lt[4], hi[4], ht[4];   // sums of (d0, d1) and of d2, low and high nibbles
        constexpr uint32_t ML = 0x0f0f0f0fu, MH = 0xf0f0f0f0u;
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const uint32_t x0 = qa[2 * p], x1 = qb[2 * p], x2 = qa[2 * p + 1], x3 = qb[2 * p + 1];
            const int i = p >> 1, k = 2 * (p & 1);
            if (p == 0) imma0_uu(lo, x0 & ML, x1 & ML, x2 & ML, x3 & ML, b.pair[i][k], b.pair[i][k + 1]);
            else imma_uu(lo, x0 & ML, x1 & ML, x2 & ML, x3 & ML, b.pair[i][k], b.pair[i][k + 1]);
            if (p == 0) imma0_us(lt, x0 & ML, x1 & ML, x2 & ML, x3 & ML, b.top[i][k], b.top[i][k + 1]);
            else imma_us(lt, x0 & ML, x1 & ML, x2 & ML, x3 & ML, b.top[i][k], b.top[i][k + 1]);
            // high nibbles stay in place (16 * code): their 2^e in the image is divided by 16
            if (p == 0) imma0_uu(hi, x0 & MH, x1 & MH, x2 & MH, x3 & MH, b.pair[2 + i][k], b.pair[2 + i][k + 1]);
            else imma_uu(hi, x0 & MH, x1 & MH, x2 & MH, x3 & MH, b.pair[2 + i][k], b.pair[2 + i][k + 1]);
            if (p == 0) imma0_us(ht, x0 & MH, x1 & MH, x2 & MH, x3 & MH, b.top[2 + i][k], b.top[2 + i][k + 1]);
            else imma_us(ht, x0 & MH, x1 & MH, x2 & MH, x3 & MH, b.top[2 + i][k], b.top[2 + i][k + 1]);
        }
        // |256 d1 sum + d0 sum| <= 257 * 32 * 15 * 255 < 2^25; the high-nibble sums are 16 times larger: < 2^29
        ya = finish(ha, t, combine3(lt[0], lo[1], lo[0]), combine3(ht[0], hi[1], hi[0]), f);
        yb = finish(hb, t, combine3(lt[2], lo[3], lo[2]), combine3(ht[2], hi[3], hi[2]), f);
    }
};

// Q6_K, planar: lane t = (h, lb) owns, in half h, the 16 positions l0 = 16*lb .. +15 of each of the four 32-column runs
// (ql[l], ql[l+32] nibbles + qh bit pairs), four scale groups.
template <>
struct Unit<WGB_Q6_K> {
    using Digits = BDigits<4>;
    __device__ static __forceinline__ void eval(const uint32_t (&sa)[4], const uint32_t (&sb)[4], uint32_t w, const Digits &b,
                                                const XImage<WGB_Q6_K> &im, uint32_t u, int lane, float &ya, float &yb)
    {
        const uint32_t t = (uint32_t)lane & 3, h = t >> 1, lb = t & 1;
        const uint32_t oql = w * 128 + h * 64 + lb * 16, oqh = w * 64 + t * 16;
        const uint4 a0 = lds128(sa[0] + oql), a1 = lds128(sa[0] + oql + 32), a2 = lds128(sa[1] + oqh);
        const uint4 b0 = lds128(sb[0] + oql), b1 = lds128(sb[0] + oql + 32), b2 = lds128(sb[1] + oqh);
        const uint32_t A0[4] = { a0.x, a0.y, a0.z, a0.w }, A1[4] = { a1.x, a1.y, a1.z, a1.w }, A2[4] = { a2.x, a2.y, a2.z, a2.w };
        const uint32_t B0[4] = { b0.x, b0.y, b0.z, b0.w }, B1[4] = { b1.x, b1.y, b1.z, b1.w }, B2[4] = { b2.x, b2.y, b2.z, b2.w };
        const uint2 sca = lds64(sa[2] + w * 16 + h * 8), scb = lds64(sb[2] + w * 16 + h * 8);
        const uint32_t da = lds16(sa[3] + w * 2), db = lds16(sb[3] + w * 2);
        auto code = [](int j, uint32_t ql0, uint32_t ql1, uint32_t qh) {
            if (j == 0) return (ql0 & 0x0f0f0f0fu) | ((qh << 4) & 0x30303030u);
            if (j == 1) return (ql1 & 0x0f0f0f0fu) | ((qh << 2) & 0x30303030u);
            if (j == 2) return ((ql0 >> 4) & 0x0f0f0f0fu) | (qh & 0x30303030u);
            return ((ql1 >> 4) & 0x0f0f0f0fu) | ((qh >> 2) & 0x30303030u);
        };
        float acca = 0.0f, accb = 0.0f;
        const uint32_t scale_at = lb * 8;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int s[4], top[4];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const int k = 2 * p;
                const uint32_t x0 = code(j, A0[k], A1[k], A2[k]), x1 = code(j, B0[k], B1[k], B2[k]);
                const uint32_t x2 = code(j, A0[k + 1], A1[k + 1], A2[k + 1]), x3 = code(j, B0[k + 1], B1[k + 1], B2[k + 1]);
                if (p == 0) {
                    imma0_uu(s, x0, x1, x2, x3, b.pair[j][k], b.pair[j][k + 1]);
                    imma0_us(top, x0, x1, x2, x3, b.top[j][k], b.top[j][k + 1]);
                } else {
                    imma_uu(s, x0, x1, x2, x3, b.pair[j][k], b.pair[j][k + 1]);
                    imma_us(top, x0, x1, x2, x3, b.top[j][k], b.top[j][k + 1]);
                }
            }
            const uint2 f = lds64(im.factors + u * 128 + t * 32 + j * 8);   // {2^e, 32 * sum}
            const float e = __uint_as_float(f.x), m = __uint_as_float(f.y);
            // int8 scales h*8 + lb + {0, 2, 4, 6}
            const float fa = s8f((j < 2 ? sca.x : sca.y) >> scale_at, 2 * (j & 1)), fb = s8f((j < 2 ? scb.x : scb.y) >> scale_at, 2 * (j & 1));
            acca = fmaf(fa, fmaf(combine3(top[0], s[1], s[0]), e, -m), acca);
            accb = fmaf(fb, fmaf(combine3(top[2], s[3], s[2]), e, -m), accb);
        }
        ya = __half2float(__ushort_as_half((uint16_t)da)) * acca;
        yb = __half2float(__ushort_as_half((uint16_t)db)) * accb;
    }
};

// Q8_0, planar: a unit is four 32-column blocks, one per lane of the quad; the codes are the operand as they are.
template <>
struct Unit<WGB_Q8_0> {
    using Digits = BDigits<2>;
    __device__ static __forceinline__ void eval(const uint32_t (&sa)[2], const uint32_t (&sb)[2], uint32_t w, const Digits &b,
                                                const XImage<WGB_Q8_0> &im, uint32_t u, int lane, float &ya, float &yb)
    {
        const uint32_t t = (uint32_t)lane & 3, o = w * 128 + t * 32;
        const uint4 a0 = lds128(sa[0] + o), a1 = lds128(sa[0] + o + 16), b0 = lds128(sb[0] + o), b1 = lds128(sb[0] + o + 16);
        const uint32_t da = lds16(sa[1] + w * 8 + t * 2), db = lds16(sb[1] + w * 8 + t * 2);
        const float e = __uint_as_float(lds32(im.factors + u * 16 + t * 4));
        int s[4], top[4];
        imma0_su(s, a0.x, b0.x, a0.y, b0.y, b.pair[0][0], b.pair[0][1]);
        imma0_ss(top, a0.x, b0.x, a0.y, b0.y, b.top[0][0], b.top[0][1]);
        imma_su(s, a0.z, b0.z, a0.w, b0.w, b.pair[0][2], b.pair[0][3]);
        imma_ss(top, a0.z, b0.z, a0.w, b0.w, b.top[0][2], b.top[0][3]);
        imma_su(s, a1.x, b1.x, a1.y, b1.y, b.pair[1][0], b.pair[1][1]);
        imma_ss(top, a1.x, b1.x, a1.y, b1.y, b.top[1][0], b.top[1][1]);
        imma_su(s, a1.z, b1.z, a1.w, b1.w, b.pair[1][2], b.pair[1][3]);
        imma_ss(top, a1.z, b1.z, a1.w, b1.w, b.top[1][2], b.top[1][3]);
        ya = __half2float(__ushort_as_half((uint16_t)da)) * (combine3(top[0], s[1], s[0]) * e);
        yb = __half2float(__ushort_as_half((uint16_t)db)) * (combine3(top[2], s[3], s[2]) * e);
    }
};

// Dense f32 (ncols a multiple of 4): 64 columns per unit.  Odd rows walk the four runs of 64 bytes in another order, so that
// neighbouring rows, whose pitch is a multiple of 128 bytes, read different banks.
template <>
struct Unit<WGB_F32> {
    struct Digits {
        __device__ __forceinline__ void clear() {}
        template <int QT>
        __device__ __forceinline__ void load(const XImage<QT> &, uint32_t, int) {}
    };
    __device__ static __forceinline__ void eval(const uint32_t (&sa)[1], const uint32_t (&sb)[1], uint32_t w, const Digits &,
                                                const XImage<WGB_F32> &im, uint32_t u, int lane, float &ya, float &yb)
    {
        const uint32_t t = (uint32_t)lane & 3, flip = ((uint32_t)lane >> 2) & 1;
        float sa4[4], sb4[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint32_t o = t * 16 + ((i ^ flip) << 6);
            const uint4 a = lds128(sa[0] + w * 256 + o), b = lds128(sb[0] + w * 256 + o), x = lds128(im.pair + u * 256 + o);
            const float x0 = __uint_as_float(x.x), x1 = __uint_as_float(x.y), x2 = __uint_as_float(x.z), x3 = __uint_as_float(x.w);
            sa4[i] = (__uint_as_float(a.x) * x0 + __uint_as_float(a.y) * x1) + (__uint_as_float(a.z) * x2 + __uint_as_float(a.w) * x3);
            sb4[i] = (__uint_as_float(b.x) * x0 + __uint_as_float(b.y) * x1) + (__uint_as_float(b.z) * x2 + __uint_as_float(b.w) * x3);
        }
        ya = (sa4[0] + sa4[1]) + (sa4[2] + sa4[3]);
        yb = (sb4[0] + sb4[1]) + (sb4[2] + sb4[3]);
    }
};

// Writer of the shared image.  put8() stores eight consecutive inputs (already normalised / transformed by the caller), 8u .. 8u + 7,
// given as two float4; it is called by whole warps (all 32 lanes, converged), lane l with u0 + l, so that four consecutive lanes
// hold one 32-column group and two hold a 16-column run; `in` is false for lanes past the end of the vector (whole groups of four
// lanes are in or out together because K is a multiple of 32 for the quantised formats), `inb` for a second float4 past it (only
// a dense f32 vector can end there).  The caller synchronises the block afterwards.
template <int QT>
struct XWriter {
    uint8_t *pair, *top;
    float *factors;

    __device__ __forceinline__ XWriter(uint8_t *image, uint32_t units)
        : pair(image), top(image + units * 2 * unit_cols(QT)), factors(reinterpret_cast<float *>(image + units * 3 * unit_cols(QT))) {}

    // What the last unit holds past the end of the vector.
    __device__ __forceinline__ void pad(uint32_t K, uint32_t units, int i, int n) const
    {
        if (QT == WGB_F32)
            for (uint32_t c = K + i; c < units * unit_cols(QT); c += n) reinterpret_cast<float *>(pair)[c] = 0.0f;
        if (QT == WGB_Q8_0)   // (the codes there are zero; so are the digits' factors)
            for (uint32_t c = K / 32 + i; c < units * 4; c += n) factors[c] = 0.0f;
    }

    __device__ __forceinline__ void put8(uint32_t u, const float4 va, const float4 vb, bool in, bool inb) const
    {
        if (QT == WGB_F32) {
            if (in) reinterpret_cast<float4 *>(pair)[2 * u] = va;
            if (in && inb) reinterpret_cast<float4 *>(pair)[2 * u + 1] = vb;
            return;
        }
        float m = fmaxf(fmaxf(fmaxf(fabsf(va.x), fabsf(va.y)), fmaxf(fabsf(va.z), fabsf(va.w))),
                        fmaxf(fmaxf(fabsf(vb.x), fabsf(vb.y)), fmaxf(fabsf(vb.z), fabsf(vb.w))));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        float sum = 0.0f;
        if (QT != WGB_Q8_0) {
            sum = ((va.x + va.y) + (va.z + va.w)) + ((vb.x + vb.y) + (vb.z + vb.w));
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            if (QT == WGB_Q4_K) sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        }
        // |v| < 2^(ex-126) for the biased exponent ex of the group maximum, so X = v * 2^(148-ex) stays
        // within +-2^22 after rounding and its third byte is a valid signed digit
        uint32_t ex = (__float_as_uint(m) >> 23) & 0xffu;
        ex = ex < 24u ? 24u : (ex > 253u ? 253u : ex);
        const float up = __uint_as_float((275u - ex) << 23);    // 2^(148 - ex)
        // round to nearest even through the 1.5 * 2^23 offset (|v * up| <= 2^22)
        auto fix = [&](float v) { return (int)(__float_as_uint(fmaf(v, up, 12582912.0f)) - 0x4b400000u); };
        const int A0 = fix(va.x), A1 = fix(va.y), A2 = fix(va.z), A3 = fix(va.w);
        const int B0 = fix(vb.x), B1 = fix(vb.y), B2 = fix(vb.z), B3 = fix(vb.w);
        if (!in) return;
        const uint32_t a01 = __byte_perm(A0, A1, 0x5410), a23 = __byte_perm(A2, A3, 0x5410);
        const uint32_t a01h = __byte_perm(A0, A1, 0x7632), a23h = __byte_perm(A2, A3, 0x7632);
        const uint32_t b01 = __byte_perm(B0, B1, 0x5410), b23 = __byte_perm(B2, B3, 0x5410);
        const uint32_t b01h = __byte_perm(B0, B1, 0x7632), b23h = __byte_perm(B2, B3, 0x7632);
        constexpr uint32_t CPU = unit_cols(QT) / 16;                     // 16-column chunks per unit
        const uint32_t c = u >> 1, unit = c / CPU, r = c % CPU;
        // the lane of a quad that owns the chunk, and which of its chunks it is
        const uint32_t t = QT == WGB_Q4_K ? r >> 2 : QT == WGB_Q6_K ? ((r >> 3) << 1) | (r & 1) : r >> 1;
        const uint32_t i = QT == WGB_Q4_K ? r & 3 : QT == WGB_Q6_K ? (r >> 1) & 3 : r & 1;
        uint8_t *p = pair + unit * (2 * unit_cols(QT)) + i * 128 + (u & 1) * 8;
        const uint32_t slot = (2 * t) ^ chunk_xor(i);
        *reinterpret_cast<uint2 *>(p + slot * 16) = make_uint2(__byte_perm(a01, a23, 0x6420), __byte_perm(b01, b23, 0x6420));
        *reinterpret_cast<uint2 *>(p + (slot ^ 1) * 16) = make_uint2(__byte_perm(a01, a23, 0x7531), __byte_perm(b01, b23, 0x7531));
        *reinterpret_cast<uint2 *>(top + unit * unit_cols(QT) + ((4 * i + t) ^ ((i >> 1) << 1)) * 16 + (u & 1) * 8) =
            make_uint2(__byte_perm(a01h, a23h, 0x6420), __byte_perm(b01h, b23h, 0x6420));
        const float e = __uint_as_float((ex - 21u) << 23);   // 2^(ex - 148)
        if (QT == WGB_Q4_K) {
            if ((u & 3) == 0) {
                float *f = factors + (unit * 4 + t) * 4 + (i >> 1);
                f[0] = i >> 1 ? e * 0.0625f : e;
                f[2] = sum;
            }
        } else if (QT == WGB_Q6_K) {
            if ((u & 1) == 0) *reinterpret_cast<float2 *>(factors + ((unit * 4 + t) * 4 + i) * 2) = make_float2(e, 32.0f * sum);
        } else {
            if ((u & 3) == 0) factors[unit * 4 + t] = e;
        }
    }
};

}  // namespace wgb
