// Wide prompt passes: up to PW_CAP prompt positions per pass through the layer stack.
//
// The passes of eight positions (prefill.cu) read every weight once per eight positions and spend their time on the
// chain unpack -> MMA -> read-back of each 256-column unit, whose tensor work is 4 % of it.  With a long prompt the
// same unpacked weights can serve up to 128 positions at a time, and the pass becomes a contraction proper: this file
// holds its matrix product on the tensor cores (tcgen05.mma kind::f16 with f32 accumulators in tensor memory), the
// activation image it reads, the element-wise kernels between the products and a causal attention over tiles of 64
// positions.  Operators as in the narrow passes: GemvQuant::dispatch (crates/wgml/src/ops/gemv_quant.rs:241-348),
// RmsNorm / LayerNorm / Silu / GELU / BatchedMultiqueryAttention of one position, for many.
//
// Arithmetic.  A unit is 256 columns.  Activations: x = X * 2^e with one exponent per position and unit, |X| <= 2048,
// written as two f16 digits X = hi + lo.  hi has eleven bits of the loudest value of its 32 columns, in steps no finer than
// 2^-PW_QUIET; lo is the rest rounded to eleven bits, so X is good to 2^-13 (loud groups) to 2^-16: 2^-24 to 2^-27 of the
// unit's loudest value.  Weights: the part of a weight that varies inside a unit, as one or two f16 numbers,
//   Q4_K  scale * code - centre  <= 520 in magnitude: one plane;  d per row and unit.  What centring takes off (codes are
//         all of one sign, and inputs of one sign would leave the accumulator's bits) comes back with the mins, which it
//         all but cancels: the group coefficients d centre - dmin min times the groups' sums of X, an MMA of their own
//   Q6_K  scale * (code - 32)    <= 4096 in magnitude: 16 a1 + a2, two planes;  d per row and unit
//   Q8_0  code * d_group / 2^E   two planes: a1 the upper nine bits, a2 the rest, exact while the group's scale is no less
//         than 1/64 of the largest of the row's eight;  2^E the row's power of two
// On even data the products of the large digits are multiples of one step (16 for Q6_K) and a unit's sum of them stays within
// about 24 bits, those of the f32 accumulator.  One accumulator takes all of a unit's products, the small ones (a2, lo)
// first: what they add below the final sum's last bit is dropped once, not per product (and towards zero: with inputs
// near a constant and codes not centred the error was 2 to 3e-6 of the result, fifteen times the eight-position product's).
// Error of a product against 64 bits (mean over rows of the 2-norm, 1024 to 11008 columns; the eight-position product in
// brackets): even data 1.3 to 1.5e-7 (2.7 to 3.4e-7), heavy tails 1.9 to 2.2e-7 (4.2e-7 to 1.3e-6), a column in 256 a hundred
// times as loud 2.2 to 2.5e-7 (5.7e-7 to 1.6e-6), inputs near a constant 1.0 to 1.2e-7 (1.2 to 1.7e-7), Q8_0 scales spread by e and
// e^2 1.5 to 1.7e-7 (2.8 to 3.4e-7).
#include "kernels.h"
#include "tc_common.cuh"

#include <algorithm>

namespace wgb {

constexpr uint32_t PW_MAXN = PW_TILE;                              // positions per tile
constexpr uint32_t PW_UNPACK_WARPS = 8;                            // build the weight operand, two groups of four
constexpr uint32_t PW_FINISH_WARPS = 8;                            // read the sums, apply scales
constexpr uint32_t PW_NT = 32 * (3 + PW_UNPACK_WARPS + PW_FINISH_WARPS);
constexpr uint32_t PW_A_COLS = 32;                                 // weight operand of 64 columns in f16, in tensor memory
constexpr uint32_t PW_A_RING = 4;                                  // one plane of a unit, in two pairs
constexpr uint32_t PW_B_STEP = 2 * PW_MAXN * 128;                  // one digit of 128 columns, largest, in shared memory
constexpr uint32_t PW_B_RING = 4;
constexpr uint32_t PW_AUX = 36 * PW_MAXN;                          // per unit: sums of the mins' product, exponents
constexpr uint32_t PW_X_RING = 3;
constexpr uint32_t PW_AMIN = 4 * TC_TILE_ROWS * 16;                // group coefficients as f16, [digit][two K-cores][row], in shared memory
// Tensor memory: two sets of sums (128 columns), the min sums (128), four weight operands (32).
constexpr uint32_t PW_TMEM_COLS = 512;
constexpr uint32_t PW_TMEM_MIN = 2 * PW_MAXN;
constexpr uint32_t PW_TMEM_A = PW_TMEM_MIN + PW_MAXN;
static_assert(PW_MAXN % 16 == 0 && PW_TMEM_A + PW_A_RING * PW_A_COLS <= PW_TMEM_COLS, "tensor memory");

// Per format: raw bytes of a unit of 128 rows (tile-major copies of prefill.cu, prefill_q6k.cu, prefill_q80.cu) and how
// many units fit.
template <int FMT> struct PwFmt;
template <> struct PwFmt<WGB_Q4_K> { static constexpr uint32_t RAW = TC_UNIT_BYTES, RAW_RING = 3, PLANES = 1, AMIN = PW_AMIN; };
template <> struct PwFmt<WGB_Q6_K> { static constexpr uint32_t RAW = TC_TILE_ROWS * 210, RAW_RING = 3, PLANES = 2, AMIN = 0; };
template <> struct PwFmt<WGB_Q8_0> { static constexpr uint32_t RAW = TC_TILE_ROWS * 272, RAW_RING = 2, PLANES = 2, AMIN = 0; };
template <int FMT> constexpr uint32_t pw_smem()
{
    return PW_B_RING * PW_B_STEP + PwFmt<FMT>::RAW_RING * PwFmt<FMT>::RAW + 2 * PwFmt<FMT>::AMIN + PW_X_RING * PW_AUX;
}
// A group of 32 columns that is quieter than the loudest of its unit takes a finer large digit, by as many bits as it is
// quieter, PW_QUIET at most: a digit finer than the accumulator's last bit (2^-2 to 2^0 in the middle of a unit's sums) is cut off
// at every MMA instead of once, and always towards zero.
constexpr uint32_t PW_QUIET = 3;
constexpr uint32_t PW_STATIC = 4 * TC_TILE_ROWS * 8 + 512;         // row scales, barriers
static_assert(pw_smem<WGB_Q4_K>() + 1024 + PW_STATIC <= 227 * 1024 && pw_smem<WGB_Q6_K>() + 1024 + PW_STATIC <= 227 * 1024 &&
                  pw_smem<WGB_Q8_0>() + 1024 + PW_STATIC <= 227 * 1024,
              "shared memory budget");
static_assert(PW_B_STEP % 1024 == 0 && PW_AUX % 16 == 0, "swizzled operands start on 1 KB boundaries");

// Activation image of a pass: [tile of np positions][unit]: the low digits of four times 64 columns, then the high ones,
// each [np rows] x 128 bytes in the 128-byte swizzle; then the sums of the eight 32-column groups as two f16 digits
// ([digit][position][group]); then one exponent (a power of two) per position.
__host__ __device__ constexpr uint32_t pw_image_unit(uint32_t np) { return (1024 + 36) * np; }

size_t prefill_wide_image_bytes(uint32_t K)
{
    // any split of PW_CAP positions into tiles of a multiple of 16 pads by less than one such multiple per tile
    return (size_t)(K / 256) * pw_image_unit(PW_CAP + 16 * ((PW_CAP + PW_MAXN - 1) / PW_MAXN + 1));
}

struct PwArgs {
    const uint8_t *w[3];
    float *out[3];            // [nsplit][slice_tok][out_stride]
    uint32_t tile0[3];
    uint32_t out_stride[3];
    uint32_t nmat, ntiles;
    const uint8_t *img;
    uint32_t nkb, nsplit, ntok, np, npt, slice_tok;
    uint32_t *err;
};

// Items of a block: blockIdx.x, blockIdx.x + gridDim.x, ...; item = ((tile, slice of the units), tile of positions),
// positions fastest, so that blocks running side by side read the same weights.
struct PwWalk {
    uint32_t tile, sp, pt, kb, kb_end;
    __device__ __forceinline__ void set(const PwArgs &a, uint32_t item)
    {
        pt = item % a.npt;
        const uint32_t r = item / a.npt;
        sp = r % a.nsplit;
        tile = r / a.nsplit;
        kb = sp * a.nkb / a.nsplit;
        kb_end = (sp + 1) * a.nkb / a.nsplit;
    }
};
__device__ __forceinline__ uint32_t pw_matrix_of(const PwArgs &a, uint32_t tile)
{
    return (a.nmat > 2 && tile >= a.tile0[2]) ? 2u : (a.nmat > 1 && tile >= a.tile0[1]) ? 1u : 0u;
}

// D (+)= A B with A in tensor memory: lane = row, a column of 32 bits = two consecutive f16 along K.
__device__ __forceinline__ void pw_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with A in shared memory.
__device__ __forceinline__ void pw_mma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// kind::f16 instruction descriptor: D f32, A and B f16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t pw_idesc(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

__device__ __forceinline__ __half2 u2h(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t h2u(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }

// A thread's 32 words into 32 columns of its lane.
__device__ __forceinline__ void pw_st32(uint32_t taddr, const uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
        "%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
        "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]),
        "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
// Two f32 at a time (the packed FMA of this architecture).
__device__ __forceinline__ uint64_t f2pack(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2unpack(uint64_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f2fma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t f2add(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b)
{
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ uint64_t f2mul(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Exponent field of the power of two above the largest of a row's eight Q8_0 scales (clamped above zero).
__device__ __forceinline__ uint32_t pw_q80_exp(uint4 sc)
{
    uint32_t m = 0;
    const uint32_t w[4] = { sc.x, sc.y, sc.z, sc.w };
#pragma unroll
    for (int i = 0; i < 4; i++) m = max(m, max(w[i] & 0x7fffu, (w[i] >> 16) & 0x7fffu));
    const uint32_t ex = __float_as_uint(__half2float(__ushort_as_half((unsigned short)m))) >> 23;
    return ex < 100u ? 100u : (ex > 142u ? 142u : ex);
}

// Exponent field of twice the unit in which a Q4_K row's group coefficients d centre - dmin min are written: they stay
// within 128 max(8 |d|, |dmin|) (centres are at most 8 * 63 + 16), 2^14 units.
__device__ __forceinline__ uint32_t pw_coef_exp(float2 dm)
{
    const uint32_t ex = (__float_as_uint(fmaxf(8.0f * fabsf(dm.x), fabsf(dm.y))) >> 23) & 0xffu;
    return (ex < 100u ? 100u : (ex > 146u ? 146u : ex)) - 5u;
}

// Two scales as f16 -> what pw_unpack takes off the low nibbles' scale * code.
__device__ __forceinline__ __half2 pw_centre(__half2 sc)
{
    return __hneg2(__hfma2(sc, __float2half2_rn(1024.0f), __hmul2(sc, __float2half2_rn(-1032.0f))));
}

// Weight operand of one step for row r: the 64 columns of chunk c of the unit at `raw`, plane 0 = the small one of a
// two-plane format, as 32 words of two f16.
// Of every four columns the words hold (0, 2) and (1, 3), which saves Q4_K a byte permutation; so does the activation image.
template <int FMT>
__device__ __forceinline__ void pw_unpack(uint32_t (&v)[32], uint32_t raw, uint32_t r, uint32_t c, bool small_plane)
{
    const uint32_t sw = r & 7;
    if constexpr (FMT == WGB_Q4_K) {
        const uint4 hdr = lds128(raw + r * 144);
        const uint32_t j0 = 2 * c;
        const uint32_t sc_lo = hdr.y & 0x3f3f3f3fu, sc_hi = (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u);
        const uint32_t scw = ((j0 & 4) ? sc_hi : sc_lo) >> (8 * (j0 & 3));
        // scale * code - centre, the centre close to 8 * scale.  Low nibbles: 1024 + code as f16, times the scale, minus 1032
        // times the scale as f16 has it (pw_centre).  High ones: 1024 + 16 code, times a sixteenth of the scale, minus 72 times
        // the scale.  The results, integers below 2^10, are exact.
        const __half2 s0 = __half2half2(__ushort2half_rn((unsigned short)(scw & 0xffu)));
        const __half2 s1 = __half2half2(__ushort2half_rn((unsigned short)((scw >> 8) & 0xffu)));
        const __half2 o0 = __hmul2(s0, __float2half2_rn(-1032.0f)), o1 = __hmul2(s1, __float2half2_rn(-72.0f)), s1s = __hmul2(s1, __float2half2_rn(0.0625f));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint4 q = lds128(raw + r * 144 + 16 + 32 * c + 16 * h);
            const uint32_t qw[4] = { q.x, q.y, q.z, q.w };
#pragma unroll
            for (int k = 0; k < 4; k++) {
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const uint32_t t = qw[k] >> (8 * p);
                    v[8 * h + 2 * k + p] = h2u(__hfma2(u2h((t & 0x000f000fu) | 0x64006400u), s0, o0));
                    v[16 + 8 * h + 2 * k + p] = h2u(__hfma2(u2h((t & 0x00f000f0u) | 0x64006400u), s1s, o1));
                }
            }
        }
    } else if constexpr (FMT == WGB_Q6_K) {
        const uint32_t H = c >> 1;   // 128-column half; 32-column groups s of it
        const uint4 scq = lds128(raw + TC_TILE_ROWS * 192 + r * 16);
        const uint32_t scw = (c & 1) ? (H ? scq.w : scq.y) : (H ? scq.z : scq.x);
        const __half2 c1056 = __float2half2_rn(1056.0f), magic = __float2half2_rn(24576.0f);
#pragma unroll
        for (uint32_t cc = 0; cc < 2; cc++) {
            const uint4 qhq = lds128(raw + TC_TILE_ROWS * 128 + (r >> 1) * 128 + (((4 * (r & 1) + 2 * H + cc) ^ ((r >> 1) & 7)) << 4));
            const uint32_t qhw[4] = { qhq.x >> (4 * (c & 1)), qhq.y >> (4 * (c & 1)), qhq.z >> (4 * (c & 1)), qhq.w >> (4 * (c & 1)) };
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {   // s = 2 (c & 1) + h
                const uint4 qlq = lds128(raw + r * 128 + (((4 * H + 2 * h + cc) ^ sw) << 4));
                const __half2 sc = __half2half2(__short2half_rn((short)(signed char)((scw >> (8 * (2 * h + cc))) & 0xffu)));
                const uint32_t qlw[4] = { qlq.x, qlq.y, qlq.z, qlq.w };
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t q = ((qlw[k] >> (4 * (c & 1))) & 0x0f0f0f0fu) | (((qhw[k] >> (2 * h)) & 0x03030303u) << 4);
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const __half2 qv = __hsub2(u2h(__byte_perm(q, 0x64646464u, p ? 0x4341 : 0x4240)), c1056);
                        const __half2 a1 = __hsub2(__hfma2(qv, sc, magic), magic);   // multiple of 16
                        v[16 * h + 8 * cc + 2 * k + p] = small_plane ? h2u(__hfma2(qv, sc, __hneg2(a1))) : h2u(a1);
                    }
                }
            }
        }
    } else {
        const uint4 scs = lds128(raw + TC_TILE_ROWS * 256 + r * 16);
        const float norm = __uint_as_float((259u - pw_q80_exp(scs)) << 23);   // 2^(6 - E): d norm < 64
        const uint32_t scw = c == 0 ? scs.x : c == 1 ? scs.y : c == 2 ? scs.z : scs.w;
        const __half2 c1152 = __float2half2_rn(1152.0f);
        const uint32_t row = raw + (c >> 1) * 16384 + r * 128;
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            const __half2 ds = __float2half2_rn(__half2float(__ushort_as_half((unsigned short)(h ? (scw >> 16) : (scw & 0xffffu)))) * norm);
            // 768 times the power of two at or below |ds| (for the largest scale in [32, 64): 768 * 32): adding it leaves the
            // product's upper nine bits, and what is left is exact in eight (a product has 18 bits)
            const __half2 magic = __hmul2(__hmax2(u2h(h2u(ds) & 0x7c007c00u), __float2half2_rn(32.0f / (1 << PW_QUIET))), __float2half2_rn(768.0f));
#pragma unroll
            for (uint32_t cc = 0; cc < 2; cc++) {
                const uint4 qq = lds128(row + (((4 * (c & 1) + 2 * h + cc) ^ sw) << 4));
                const uint32_t qw[4] = { qq.x, qq.y, qq.z, qq.w };
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t u = qw[k] ^ 0x80808080u;
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const __half2 qv = __hsub2(u2h(__byte_perm(u, 0x64646464u, p ? 0x4341 : 0x4240)), c1152);
                        const __half2 a1 = __hsub2(__hfma2(qv, ds, magic), magic);
                        v[16 * h + 8 * cc + 2 * k + p] = small_plane ? h2u(__hfma2(qv, ds, __hneg2(a1))) : h2u(a1);
                    }
                }
            }
        }
    }
}

// Roles: two producer threads (raw weights and per-unit extras; activation operand), one thread issuing MMAs, two groups
// of four warps building the weight operand (alternate chunks of 64 columns), eight warps finishing units.
// What bounds it: the turnaround of the weight operand at unit boundaries and, with two planes, its unpacking (about 1.3
// to 3 instructions per weight).  A chunk of weights therefore serves as many positions as tensor memory has room for:
// the accumulator holds both digits (low digits of the four chunks first, then the high ones over the same weight
// operands, which stay in tensor memory), so a tile is 128 positions; with an accumulator per digit it was 80.  Q4_K
// 22016x4096 times 511 positions: 227 us then, 164 us now (1.1 PFLOP/s of two-digit MMA work).  The operand goes from
// registers to tensor memory: written to and read from shared memory it cost as much of that memory's 128 bytes a
// clock as everything else together.  Raw weights are free again as soon as they are unpacked, ahead of their MMAs;
// the rows' scales travel in a small ring of their own.
template <int FMT>
__global__ void __launch_bounds__(PW_NT, 1) gemm_wide_kernel(const __grid_constant__ PwArgs a)
{
    using F = PwFmt<FMT>;
    constexpr uint32_t NA = PW_A_RING / 2, NB = PW_B_RING, NX = PW_X_RING, NR = F::RAW_RING, P = F::PLANES;
    extern __shared__ uint8_t pw_smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * NA + 2 * NB + 2 * NX + 2 * NR + 10];
    __shared__ float2 rowscale[4][TC_TILE_ROWS];
    __shared__ uint32_t tmem_base_slot;
    __shared__ uint32_t dead_flag;
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)pw_smem_raw + 1023) & ~(uintptr_t)1023);
    volatile uint32_t *dead = &dead_flag;

    pdl_launch_dependents();
    const uint32_t warp = tc_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const uint32_t nitems = a.ntiles * a.nsplit * a.npt, np = a.np;
    const uint32_t bar0 = tc_uniform(smem_addr(bars));
    auto bar = [&](uint32_t i) { return bar0 + 8 * i; };
    auto bar_a = [&](uint32_t j) { return bar(j); };                       // weight operand of chunks 2 j and 2 j + 1 is built
    auto bar_ae = [&](uint32_t j) { return bar(NA + j); };                 //   and has been read by the MMAs of both digits
    auto bar_b = [&](uint32_t s) { return bar(2 * NA + s); };              // activation operand of a step has landed
    auto bar_be = [&](uint32_t s) { return bar(2 * NA + NB + s); };        //   and has been read
    auto bar_x = [&](uint32_t s) { return bar(2 * NA + 2 * NB + s); };     // group sums and exponents of a unit have landed
    auto bar_xe = [&](uint32_t s) { return bar(2 * NA + 2 * NB + NX + s); };
    constexpr uint32_t B0 = 2 * NA + 2 * NB + 2 * NX;
    auto bar_u = [&](uint32_t i) { return bar(B0 + i); };                  // raw unit has landed
    auto bar_ue = [&](uint32_t i) { return bar(B0 + NR + i); };            //   and is unpacked
    auto bar_d = [&](uint32_t u) { return bar(B0 + 2 * NR + u); };         // the unit's sums are complete
    auto bar_t = [&](uint32_t u) { return bar(B0 + 2 * NR + 2 + u); };     //   and have been read
    auto bar_r = [&](uint32_t i) { return bar(B0 + 2 * NR + 4 + i); };     // its rows' scales are written (i = m % 4)
    const uint32_t bar_m = bar(B0 + 2 * NR + 8);                           // the min sums have been read
    const uint32_t bar_end = bar(B0 + 2 * NR + 9);                         // after an expired wait: the MMAs in flight are through
    const uint32_t sm_b = tc_uniform(smem_addr(smem)), sm_raw = sm_b + NB * PW_B_STEP, sm_min = sm_raw + NR * F::RAW, sm_aux = sm_min + 2 * F::AMIN;

    if (threadIdx.x == 0) {
        dead_flag = 0;
        for (uint32_t c = 0; c < NA; c++) {
            mbar_init(bar_a(c), PW_UNPACK_WARPS);
            mbar_init(bar_ae(c), 1);
        }
        for (uint32_t s = 0; s < NB; s++) {
            mbar_init(bar_b(s), 1);
            mbar_init(bar_be(s), 1);
        }
        for (uint32_t s = 0; s < NX; s++) {
            mbar_init(bar_x(s), 1);
            mbar_init(bar_xe(s), PW_FINISH_WARPS);
        }
        for (uint32_t s = 0; s < NR; s++) {
            mbar_init(bar_u(s), 1);
            mbar_init(bar_ue(s), PW_UNPACK_WARPS);
        }
        for (uint32_t s = 0; s < 4; s++) mbar_init(bar_r(s), PW_UNPACK_WARPS / 2);
        for (uint32_t u = 0; u < 2; u++) {
            mbar_init(bar_d(u), 1);
            mbar_init(bar_t(u), PW_FINISH_WARPS);
        }
        mbar_init(bar_m, PW_FINISH_WARPS);
        mbar_init(bar_end, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(PW_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tc_uniform(tmem_base_slot);
    pdl_wait();   // barriers and tensor memory are set up while the preceding launch (which writes the image) still runs

    // Every role walks the same items, units m, operand chunks q and steps n (numbered through over the block's life).  A
    // parity tells two phases apart, so each waiter waits on every phase of a barrier, in order, and a barrier cannot
    // run a phase ahead of any of its waiters: the next use of what it guards needs the waiter's own arrival, directly
    // (rings) or through the MMA order (scales of unit m + 4 are written when MMAs of unit m + 3 are through, which
    // takes the sums of unit m + 1 read).  A role whose wait has expired leaves its loop; the others see the flag and
    // follow.
    constexpr unsigned long long DRAIN_NS = 1000000000ull;
    if (warp == 0) {
        // ------------------------------ raw weights, group sums, exponents ------------------------------
        if (lane == 0) {
            uint32_t m = 0;
            bool ok = true;
            const uint32_t unit_bytes = pw_image_unit(np), aux = 36 * np;
            for (uint32_t item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
                PwWalk w;
                w.set(a, item);
                const uint32_t mi = pw_matrix_of(a, w.tile);
                const uint8_t *wt = a.w[mi] + (size_t)(w.tile - a.tile0[mi]) * a.nkb * F::RAW;
                for (uint32_t kb = w.kb; kb < w.kb_end; kb++, m++) {
                    const uint32_t u = m % NR, x = m % NX;
                    if (m >= NR) ok = tc_wait(bar_ue(u), (m / NR - 1) & 1, dead, a.err, 61);
                    if (ok && m >= NX) ok = tc_wait(bar_xe(x), (m / NX - 1) & 1, dead, a.err, 62);
                    if (!ok) break;
                    mbar_expect_tx(bar_u(u), F::RAW);
                    bulk_copy_g2s(sm_raw + u * F::RAW, wt + (size_t)kb * F::RAW, F::RAW, bar_u(u));
                    mbar_expect_tx(bar_x(x), aux);
                    bulk_copy_g2s(sm_aux + x * PW_AUX, a.img + ((size_t)w.pt * a.nkb + kb) * unit_bytes + 1024 * np, aux, bar_x(x));
                }
            }
            if (!ok) {   // the copies in flight land before the block gives its shared memory back
                for (uint32_t k = m > NR ? m - NR : 0; k < m; k++) mbar_wait(bar_u(k % NR), (k / NR) & 1, nullptr, 0, DRAIN_NS);
                for (uint32_t k = m > NX ? m - NX : 0; k < m; k++) mbar_wait(bar_x(k % NX), (k / NX) & 1, nullptr, 0, DRAIN_NS);
            }
        }
    } else if (warp == 2 + PW_UNPACK_WARPS + PW_FINISH_WARPS) {
        // ------------------------------ activation operand ------------------------------
        if (lane == 0) {
            uint32_t n = 0;
            bool ok = true;
            const uint32_t unit_bytes = pw_image_unit(np), bstep = 256 * np;
            for (uint32_t item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
                PwWalk w;
                w.set(a, item);
                for (uint32_t kb = w.kb; kb < w.kb_end && ok; kb++) {
                    const uint8_t *img = a.img + ((size_t)w.pt * a.nkb + kb) * unit_bytes;
                    for (uint32_t st = 0; st < 4 * P; st++, n++) {
                        const uint32_t s = n % NB;
                        if (n >= NB) ok = tc_wait(bar_be(s), (n / NB - 1) & 1, dead, a.err, 63);
                        if (!ok) break;
                        mbar_expect_tx(bar_b(s), bstep);
                        bulk_copy_g2s(sm_b + s * PW_B_STEP, img + (st & 3) * bstep, bstep, bar_b(s));
                    }
                }
            }
            if (!ok)
                for (uint32_t k = n > NB ? n - NB : 0; k < n; k++) mbar_wait(bar_b(k % NB), (k / NB) & 1, nullptr, 0, DRAIN_NS);
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issue ------------------------------
        // The whole warp walks the loop and waits, with votes, so that control flow stays uniform for the compiler.
        uint32_t m = 0, n = 0, q = 0;   // q: planes so far
        bool ok = true;
        const uint32_t idesc = pw_idesc(np);
        auto wait = [&](uint32_t b, uint32_t parity, uint32_t code) { return __all_sync(0xffffffffu, tc_wait(b, parity, dead, a.err, code)) != 0; };
        for (uint32_t item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
            PwWalk w;
            w.set(a, item);
            for (uint32_t kb = w.kb; kb < w.kb_end && ok; kb++, m++) {
                const uint32_t u = m & 1, dcol = tmem_base + u * PW_MAXN;
                // (with mins, the wait for the min sums of unit m - 2 covers this one)
                if (FMT != WGB_Q4_K && m >= 2) ok = wait(bar_t(u), ((m >> 1) - 1) & 1, 64);
                for (uint32_t pl = 0; pl < P && ok; pl++, q++) {
#pragma unroll 1
                    for (uint32_t st = 0; st < 4; st++, n++) {
                        const uint32_t j = st & 1, s = n % NB;   // low digits of the two pairs of chunks, then the high ones
                        if (st < 2) ok = wait(bar_a(j), q & 1, 66);
                        if (ok) ok = wait(bar_b(s), (n / NB) & 1, 65);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t at = tmem_base + PW_TMEM_A + 2 * j * PW_A_COLS;
                        const uint64_t bd0 = tc_smem_desc_sw128(sm_b + s * PW_B_STEP, 1024), bd1 = tc_smem_desc_sw128(sm_b + s * PW_B_STEP + 128 * np, 1024);
                        if (tc_elect()) {
#pragma unroll
                            for (uint32_t k = 0; k < 4; k++) pw_mma(dcol, at + 8 * k, bd0 + 2 * k, idesc, (pl | st | k) ? 1u : 0u);
#pragma unroll
                            for (uint32_t k = 0; k < 4; k++) pw_mma(dcol, at + PW_A_COLS + 8 * k, bd1 + 2 * k, idesc, 1u);
                            tc_commit(bar_be(s));
                            if (st >= 2) tc_commit(bar_ae(j));
                        }
                        __syncwarp();
                    }
                }
                if (FMT == WGB_Q4_K && ok && m >= 1) ok = wait(bar_m, (m - 1) & 1, 68);
                if (!ok) break;
                if (FMT == WGB_Q4_K) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (tc_elect()) {
                    // sum over the eight groups of coefficient x (sum of the group's X): both digits of the sums in one MMA, one for
                    // either digit of the coefficient, the small one first
                    if (FMT == WGB_Q4_K) {
                        const uint64_t sums = tc_smem_desc(sm_aux + (m % NX) * PW_AUX, np * 16, 128);
                        const uint32_t coef = sm_min + u * F::AMIN;
                        pw_mma_ss(tmem_base + PW_TMEM_MIN, tc_smem_desc(coef + 2 * TC_TILE_ROWS * 16, TC_TILE_ROWS * 16, 128), sums, idesc, 0u);
                        pw_mma_ss(tmem_base + PW_TMEM_MIN, tc_smem_desc(coef, TC_TILE_ROWS * 16, 128), sums, idesc, 1u);
                    }
                    tc_commit(bar_d(u));
                }
                __syncwarp();
            }
        }
        if (!ok) {   // the MMAs in flight read shared memory and write tensor memory: they end before the block gives these back
            if (tc_elect()) tc_commit(bar_end);
            __syncwarp();
            mbar_wait(bar_end, 0, nullptr, 0, DRAIN_NS);
        }
    } else if (warp < 2 + PW_UNPACK_WARPS) {
        // ------------------------------ weight operand ------------------------------
        // Group `grp` builds chunks grp and grp + 2 of a plane; a thread builds one row of 64 columns.
        const uint32_t grp = (warp - 2) >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t trow = tmem_base + (((warp & 3) * 32u) << 16);   // the quarter of tensor memory the warp may touch
        uint32_t m = 0, q = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
            PwWalk w;
            w.set(a, item);
            for (uint32_t kb = w.kb; kb < w.kb_end && ok; kb++, m++) {
                const uint32_t ur = m % NR, raw = sm_raw + ur * F::RAW;
                ok = tc_wait(bar_u(ur), (m / NR) & 1, dead, a.err, 69);
                // (on behalf of the MMA of the mins, which reads the group sums)
                if (FMT == WGB_Q4_K && grp == 1 && ok) ok = tc_wait(bar_x(m % NX), (m / NX) & 1, dead, a.err, 67);
                ok = __all_sync(0xffffffffu, ok);
#pragma unroll 1
                for (uint32_t i = 0; i < 2 * P && ok; i++) {
                    const uint32_t j = i & 1, c = 2 * j + grp;
                    // the row is built in registers before its buffer is free: only the store waits for the MMAs
                    uint32_t v[32];
                    pw_unpack<FMT>(v, raw, r, c, P == 2 && i < 2);
                    if (q) ok = __all_sync(0xffffffffu, tc_wait(bar_ae(j), (q - 1) & 1, dead, a.err, 70));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    pw_st32(trow + PW_TMEM_A + c * PW_A_COLS, v);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_a(j));
                    if (i & 1) q++;
                    if (i == 0) {
                        // Once per unit, off the path of its first MMAs.  (The MMAs of two units back are through: a chunk of
                        // the unit before has just been read.)
                        if (grp == 0) {
                            float d, coef = 0.0f;
                            if constexpr (FMT == WGB_Q4_K) {
                                uint32_t dm;
                                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(dm) : "r"(raw + r * 144));
                                const float2 f = __half22float2(u2h(dm));
                                d = f.x;
                                coef = __uint_as_float(pw_coef_exp(f) << 23);   // twice the coefficients' unit: the sums are halves
                            } else if constexpr (FMT == WGB_Q6_K) {
                                uint32_t db;
                                asm volatile("ld.shared.u16 %0, [%1];" : "=r"(db) : "r"(raw + TC_TILE_ROWS * 208 + r * 2));
                                d = __half2float(__ushort_as_half((unsigned short)db));
                            } else {
                                d = __uint_as_float((pw_q80_exp(lds128(raw + TC_TILE_ROWS * 256 + r * 16)) - 5u) << 23);   // 2^(E - 6)
                            }
                            rowscale[m & 3][r] = make_float2(d, coef);
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar_r(m & 3));
                        }
                        if constexpr (FMT == WGB_Q4_K) {
                            // Of the row's eight group coefficients d centre - dmin min (what centring took off the unit's products, and the
                            // mins) the four of this half, in two digits, each once per K-core: for either digit of the group sums.
                            const uint4 hdr = lds128(raw + r * 144);
                            const float2 f = __half22float2(u2h(hdr.x));
                            const float inv = __uint_as_float((255u - pw_coef_exp(f)) << 23);   // one over the unit
                            const float d1 = f.x * inv, dm = -f.y * inv;
                            const uint64_t d2 = f2pack(d1, 8.0f * d1), dm2 = f2pack(dm, dm), off = f2pack(-8388608.0f, -8388608.0f), one = f2pack(-1.0f, -1.0f);
                            const uint32_t sc = grp ? (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u) : hdr.y & 0x3f3f3f3fu;
                            const uint32_t mi = grp ? ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u) : hdr.z & 0x3f3f3f3fu;
                            auto two = [&](uint32_t w, uint32_t b) {   // bytes b and b + 1 as floats
                                return f2add(f2pack(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7550 + b)), __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7551 + b))), off);
                            };
                            const float2 even = __half22float2(pw_centre(__hsub2(u2h(__byte_perm(sc, 0x64646464u, 0x4240)), __float2half2_rn(1024.0f))));
                            uint32_t c1[2], c2[2];
#pragma unroll
                            for (uint32_t i = 0; i < 2; i++) {
                                const float odd = __uint_as_float(__byte_perm(sc, 0x4b000000u, 0x7551 + 2 * i)) - 8388608.0f;
                                const uint64_t w = f2fma(f2pack(i ? even.y : even.x, odd), d2, f2mul(two(mi, 2 * i), dm2));
                                float w0, w1;
                                f2unpack(w, w0, w1);
                                const __half2 hi = __floats2half2_rn(w0, w1);
                                const float2 hf = __half22float2(hi);
                                f2unpack(f2fma(f2pack(hf.x, hf.y), one, w), w0, w1);
                                c1[i] = h2u(hi);
                                c2[i] = h2u(__floats2half2_rn(w0, w1));
                            }
                            const uint32_t at = sm_min + (m & 1) * F::AMIN + r * 16 + 8 * grp;
                            sts64(at, c1[0], c1[1]);
                            sts64(at + TC_TILE_ROWS * 16, c1[0], c1[1]);
                            sts64(at + 2 * TC_TILE_ROWS * 16, c2[0], c2[1]);
                            sts64(at + 3 * TC_TILE_ROWS * 16, c2[0], c2[1]);
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_ue(ur));
            }
        }
    } else {
        // ------------------------------ finishing ------------------------------
        // Thread (quarter, lane, half): row r of the tile, groups of eight positions half, half + 2, ...
        constexpr uint32_t NG = PW_MAXN / 16;
        const uint32_t half = (warp - 2 - PW_UNPACK_WARPS) >> 2, quarter = warp & 3, r = quarter * 32 + lane, ng = np / 8;
        const uint32_t trow = tmem_base + ((quarter * 32u) << 16);
        uint64_t acc[NG][4];
        uint32_t m = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
            PwWalk w;
            w.set(a, item);
#pragma unroll
            for (uint32_t g = 0; g < NG; g++)
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) acc[g][j] = 0ull;
            for (uint32_t kb = w.kb; kb < w.kb_end && ok; kb++, m++) {
                const uint32_t u = m & 1, x = m % NX, ebase = sm_aux + x * PW_AUX + 32 * np;
                ok = tc_wait(bar_x(x), (m / NX) & 1, dead, a.err, 72) && tc_wait(bar_r(m & 3), (m >> 2) & 1, dead, a.err, 73) &&
                     tc_wait(bar_d(u), (m >> 1) & 1, dead, a.err, 74);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const float2 sc = rowscale[m & 3][r];
                const uint64_t d2 = f2pack(sc.x, sc.x), dm2 = f2pack(sc.y, sc.y);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tb = trow + u * PW_MAXN;
#pragma unroll
                for (uint32_t gi = 0; gi < NG; gi++) {
                    const uint32_t g = 2 * gi + half;
                    if (g < ng) {
                        int dv[8], mn[8];
                        tc_ld8(tb + 8 * g, dv);
                        if (FMT == WGB_Q4_K) tc_ld8(trow + PW_TMEM_MIN + 8 * g, mn);
                        const uint4 e0 = lds128(ebase + 32 * g), e1 = lds128(ebase + 32 * g + 16);
                        const uint32_t ev[8] = { e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w };
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (uint32_t j = 0; j < 4; j++) {
                            uint64_t t = f2mul(f2pack(__int_as_float(dv[2 * j]), __int_as_float(dv[2 * j + 1])), d2);
                            if (FMT == WGB_Q4_K) t = f2fma(f2pack(__int_as_float(mn[2 * j]), __int_as_float(mn[2 * j + 1])), dm2, t);
                            acc[gi][j] = f2fma(t, f2pack(__uint_as_float(ev[2 * j]), __uint_as_float(ev[2 * j + 1])), acc[gi][j]);
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bar_t(u));
                    mbar_arrive(bar_m);
                    mbar_arrive(bar_xe(x));
                }
            }
            if (!ok) break;
            const uint32_t mi = pw_matrix_of(a, w.tile), stride = a.out_stride[mi];
            const uint32_t t0 = w.pt * np;
            float *outp = a.out[mi] + ((size_t)w.sp * a.slice_tok + t0) * stride + (size_t)(w.tile - a.tile0[mi]) * TC_TILE_ROWS + r;
#pragma unroll
            for (uint32_t gi = 0; gi < NG; gi++) {
                const uint32_t g = 2 * gi + half;
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) {
                    float v0, v1;
                    f2unpack(acc[gi][j], v0, v1);
                    const uint32_t p = 8 * g + 2 * j;
                    if (p < np && t0 + p < a.ntok) outp[(size_t)p * stride] = v0;
                    if (p + 1 < np && t0 + p + 1 < a.ntok) outp[(size_t)(p + 1) * stride] = v1;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(PW_TMEM_COLS) : "memory");
    }
}

// Tiles of positions: as few as fit, of equal size (a multiple of sixteen, the step of an MMA's N).
WideTiling prefill_wide_tiling(uint32_t ntok)
{
    WideTiling t;
    t.npt = (ntok + PW_MAXN - 1) / PW_MAXN;
    t.np = ((ntok + t.npt - 1) / t.npt + 15) & ~15u;
    return t;
}

// Slices of the units: items are (row tile, tile of positions, slice); an item costs its units plus about one for
// filling the pipeline and writing its rows, and the last wave should be full.  `max_split` bounds the slices by the
// room for them.
uint32_t prefill_wide_splits(uint32_t nrows, uint32_t K, const WideTiling &t, uint32_t max_split)
{
    const uint32_t tiles = nrows / TC_TILE_ROWS * t.npt, nkb = K / 256, sms = (uint32_t)sm_count();
    uint32_t best = 1;
    float best_cost = 1e30f;
    for (uint32_t s = 1; s <= max_split && s <= PF_MAX_SPLIT && s <= nkb; s++) {
        const uint32_t waves = (tiles * s + sms - 1) / sms;
        const float cost = (float)waves * ((float)((nkb + s - 1) / s) + 1.0f) + 0.5f * (float)s;
        if (cost < best_cost - 1e-3f) { best_cost = cost; best = s; }
    }
    return best;
}

template <int FMT>
static int launch_wide(const PwArgs &a, bool *attrs, cudaStream_t stream)
{
    if (!*attrs) {
        WGB_CUDA(cudaFuncSetAttribute(gemm_wide_kernel<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(pw_smem<FMT>() + 1024)));
        *attrs = true;
    }
    const uint32_t items = a.ntiles * a.nsplit * a.npt, sms = (uint32_t)sm_count();
    WGB_CUDA(launch_pdl(gemm_wide_kernel<FMT>, dim3(items < sms ? items : sms), dim3(PW_NT), pw_smem<FMT>() + 1024, stream, a));
    return WGB_OK;
}

int launch_gemm_wide(int qtype, uint32_t nmat, const uint8_t *const *w_tiles, const uint32_t *nrows, uint32_t K, const uint8_t *image, uint32_t ntok,
                     const WideTiling &t, float *const *out, const uint32_t *out_stride, uint32_t nsplit, cudaStream_t stream)
{
    WGB_REQUIRE(nmat >= 1 && nmat <= 3 && K % 256 == 0 && ntok >= 1 && ntok <= PW_CAP && nsplit >= 1 && nsplit <= K / 256 && t.np % 16 == 0 && t.np <= PW_MAXN &&
                    t.np * t.npt >= ntok,
                "wide product: %u matrices, %u columns, %u positions, %u slices", nmat, K, ntok, nsplit);
    DeviceState *ds = device_state();
    if (!ds) return WGB_ERR_CUDA;
    PwArgs a = {};
    for (uint32_t i = 0; i < nmat; i++) {
        WGB_REQUIRE(nrows[i] > 0 && nrows[i] % TC_TILE_ROWS == 0, "wide product: %u rows", nrows[i]);
        a.w[i] = w_tiles[i];
        a.out[i] = out[i];
        a.out_stride[i] = out_stride[i];
        a.tile0[i] = a.ntiles;
        a.ntiles += nrows[i] / TC_TILE_ROWS;
    }
    a.nmat = nmat;
    a.img = image;
    a.nkb = K / 256;
    a.nsplit = nsplit;
    a.ntok = ntok;
    a.np = t.np;
    a.npt = t.npt;
    a.slice_tok = ntok;
    a.err = gemv_status_word();
    if (qtype == WGB_Q4_K) return launch_wide<WGB_Q4_K>(a, &ds->wide_attrs[0], stream);
    if (qtype == WGB_Q6_K) return launch_wide<WGB_Q6_K>(a, &ds->wide_attrs[1], stream);
    if (qtype == WGB_Q8_0) return launch_wide<WGB_Q8_0>(a, &ds->wide_attrs[2], stream);
    return fail(WGB_ERR_INVALID, "wide product of type %d", qtype);
}

// ---- activation image ---------------------------------------------------------------------------------

// One warp writes the image of 256 values of position t (lane: columns 8 lane .. 8 lane + 7 of the unit).
__device__ __forceinline__ void wide_image_unit(uint8_t *__restrict__ image, uint32_t nkb, uint32_t np, uint32_t t, uint32_t unit, uint32_t lane, const float (&v)[8])
{
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) mx = fmaxf(mx, fabsf(v[i]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const uint32_t eg = (__float_as_uint(mx) >> 23) & 0xffu;   // of the lane's group of 32 columns
    mx = warp_max(mx);
    // |v| < 2^(ex - 126), so X = v * 2^(137 - ex) lies within +-2048
    uint32_t ex = (__float_as_uint(mx) >> 23) & 0xffu;
    ex = ex < 24u ? 24u : (ex > 253u ? 253u : ex);
    const float up = __uint_as_float((264u - ex) << 23), down = __uint_as_float((ex - 10u) << 23);
    // the large digit: eleven bits of the group's largest value (1.5 * 2^23 units, added and taken away, rounds to a unit)
    const uint32_t quiet = ex > eg ? min(ex - eg, PW_QUIET) : 0u;
    const float magic = 1.5f * __uint_as_float((150u - quiet) << 23);
    uint32_t hw[4], lw[4];
    float hsum = 0.0f, lsum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float hi[2], lo[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float X = v[4 * (i >> 1) + (i & 1) + 2 * j] * up;   // (0, 2), (1, 3): see pw_unpack
            hi[j] = __fsub_rn(__fadd_rn(X, magic), magic);
            lo[j] = __half2float(__float2half_rn(X - hi[j]));
            hsum += hi[j];
            lsum += lo[j];
        }
        hw[i] = h2u(__floats2half2_rn(hi[0], hi[1]));
        lw[i] = h2u(__floats2half2_rn(lo[0], lo[1]));
    }
    hsum += __shfl_xor_sync(0xffffffffu, hsum, 1);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
    hsum += __shfl_xor_sync(0xffffffffu, hsum, 2);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
    const uint32_t pt = t / np, p = t - pt * np;
    uint8_t *base = image + ((size_t)pt * nkb + unit) * pw_image_unit(np);
    uint8_t *row = base + (lane >> 3) * (128 * np) + p * 128 + (((lane & 7) ^ (p & 7)) << 4);
    *reinterpret_cast<uint4 *>(row) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
    *reinterpret_cast<uint4 *>(row + 512 * np) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    uint8_t *aux = base + 1024 * np;
    if ((lane & 3) == 0) {
        // half the group's sum (at most 2^15), as two f16 digits
        const float l = 0.5f * lsum;
        const __half s1 = __float2half_rn(fmaf(hsum, 0.5f, l));
        __half *s = reinterpret_cast<__half *>(aux) + p * 8 + (lane >> 2);
        s[0] = s1;
        s[8 * np] = __float2half_rn(fmaf(hsum, 0.5f, -__half2float(s1)) + l);
    }
    if (lane == 0) *reinterpret_cast<float *>(aux + 32 * np + 4 * p) = down;
}

__device__ __forceinline__ void wide_load8(float (&v)[8], const float *__restrict__ p)
{
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void wide_add8(float (&v)[8], const float *__restrict__ p)
{
    float q[8];
    wide_load8(q, p);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] += q[i];
}
__device__ __forceinline__ void wide_store8(float *__restrict__ p, const float (&v)[8])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4 *>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// x (+= slices of a product and its bias, written back), then nothing, RMSNorm or LayerNorm (gain and bias), then the
// image.  One block per position; a thread owns the same eight columns of every eighth unit throughout.
constexpr uint32_t PW_NORM_NT = 256;
__global__ void __launch_bounds__(PW_NORM_NT) wide_norm_image_kernel(float *__restrict__ x, const float *__restrict__ part, uint32_t nsplit, uint32_t ntok,
                                                                     const float *__restrict__ fold_bias, const float *__restrict__ gain,
                                                                     const float *__restrict__ bias, float eps, uint32_t K, uint32_t np, uint8_t *__restrict__ image)
{
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nkb = K / 256;
    __shared__ float red[32];
    float *xr = x + (size_t)t * K;
    float s = 0.0f;
    if (part || gain) {
        for (uint32_t u = warp; u < nkb; u += PW_NORM_NT / 32) {
            const uint32_t i = u * 256 + lane * 8;
            float v[8];
            wide_load8(v, xr + i);
            if (part) {
                for (uint32_t k = 0; k < nsplit; k++) wide_add8(v, part + ((size_t)k * ntok + t) * K + i);
                if (fold_bias) wide_add8(v, fold_bias + i);
                wide_store8(xr + i, v);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) s += bias ? v[k] : v[k] * v[k];
        }
    }
    if (!image) return;
    float mean = 0.0f, scale = 1.0f;
    if (gain) {
        s = block_sum<PW_NORM_NT>(s, red);
        if (bias) {
            mean = s / (float)K;
            float ss = 0.0f;
            for (uint32_t u = warp; u < nkb; u += PW_NORM_NT / 32) {
                float v[8];
                wide_load8(v, xr + u * 256 + lane * 8);
#pragma unroll
                for (int k = 0; k < 8; k++) ss = fmaf(v[k] - mean, v[k] - mean, ss);
            }
            s = block_sum<PW_NORM_NT>(ss, red);
        }
        scale = 1.0f / sqrtf(s / (float)K + eps);
    }
    for (uint32_t u = warp; u < nkb; u += PW_NORM_NT / 32) {
        const uint32_t i = u * 256 + lane * 8;
        float v[8];
        wide_load8(v, xr + i);
        if (gain) {
            float g[8];
            wide_load8(g, gain + i);
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = ((v[k] - mean) * scale) * g[k];
            if (bias) wide_add8(v, bias + i);
        }
        wide_image_unit(image, nkb, np, t, u, lane, v);
    }
}

int launch_wide_norm_image(float *x, const float *part, uint32_t nsplit, const float *fold_bias, const float *gain, const float *bias, float eps, uint32_t K,
                           uint32_t ntok, const WideTiling &t, uint8_t *image, cudaStream_t stream)
{
    WGB_REQUIRE(K % 256 == 0, "wide image of %u columns", K);
    WGB_CUDA(launch_pdl(wide_norm_image_kernel, dim3(ntok), dim3(PW_NORM_NT), 0, stream, x, part, nsplit, ntok, fold_bias, gain, bias, eps, K, t.np, image));
    return WGB_OK;
}

// act(slices of one or two products) and its image: SiLU(gate) * up (ops/silu.wgsl:19-27) or GELU(product + bias)
// (ops/unary.wgsl:50-52).  One warp per unit and position.
template <bool GELU>
__global__ void __launch_bounds__(256) wide_act_image_kernel(const float *__restrict__ gate, uint32_t gsplit, const float *__restrict__ upv, uint32_t usplit,
                                                             const float *__restrict__ bias, uint32_t K, uint32_t ntok, uint32_t np, uint8_t *__restrict__ image)
{
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t t = blockIdx.y, lane = threadIdx.x & 31, u = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (u >= K / 256) return;
    const size_t i = (size_t)t * K + u * 256 + lane * 8;
    float v[8];
    wide_load8(v, gate + i);
    for (uint32_t k = 1; k < gsplit; k++) wide_add8(v, gate + (size_t)k * ntok * K + i);
    if constexpr (GELU) {
        if (bias) wide_add8(v, bias + u * 256 + lane * 8);
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = 0.5f * v[k] * (1.0f + tanhf(0.7978846f * v[k] * (1.0f + 0.044715f * v[k] * v[k])));
    } else {
        float b[8];
        wide_load8(b, upv + i);
        for (uint32_t k = 1; k < usplit; k++) wide_add8(b, upv + (size_t)k * ntok * K + i);
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = b[k] * (v[k] / (1.0f + expf(-v[k])));
    }
    wide_image_unit(image, K / 256, np, t, u, lane, v);
}

int launch_wide_silu_image(const float *gate, uint32_t gsplit, const float *up, uint32_t usplit, uint32_t K, uint32_t ntok, const WideTiling &t, uint8_t *image,
                           cudaStream_t stream)
{
    WGB_CUDA(launch_pdl(wide_act_image_kernel<false>, dim3((K / 256 + 7) / 8, ntok), dim3(256), 0, stream, gate, gsplit, up, usplit, nullptr, K, ntok, t.np, image));
    return WGB_OK;
}
int launch_wide_gelu_image(const float *part, uint32_t nsplit, const float *bias, uint32_t K, uint32_t ntok, const WideTiling &t, uint8_t *image, cudaStream_t stream)
{
    WGB_CUDA(launch_pdl(wide_act_image_kernel<true>, dim3((K / 256 + 7) / 8, ntok), dim3(256), 0, stream, part, nsplit, nullptr, 0u, bias, K, ntok, t.np, image));
    return WGB_OK;
}

// ---- causal attention of a wide pass --------------------------------------------------------------------

// BatchedMultiqueryAttention (ops/batched_multiquery_attention.wgsl:38-99) for positions pos0 + t, t < ntok, each
// attending to cache rows 0 .. pos0 + t.  One block per (query head, tile of 64 positions), cache rows in tiles of 64
// with a running softmax; everything in f32 on the CUDA cores.  256 threads: thread (ty, tx) owns positions 4 ty .. + 3,
// scores of rows tx + 16 j, and value columns 4 tx + 64 j.  Rows of the K and Q tiles are padded by four floats so
// that the sixteen rows a half-warp reads sit in different banks.  Longest tiles first.
// Few positions on a long context (a second turn of a conversation) are few blocks, each walking all the rows: blockIdx.z then
// shares the tiles of rows of one (head, tile of positions) among blocks, which leave their unnormalised sums, maxima and
// denominators in `scratch`; the last to arrive (a counter that wraps back to zero) merges them in the order of blockIdx.z.
template <uint32_t HD> constexpr uint32_t WA_SLOT = 4 * (HD / 64) * 256 + 32;
constexpr uint32_t WA_BLOCKS = 2;   // blocks per SM that share rows, most: as many as are resident
template <uint32_t HD, bool SHARED>   // SHARED: blocks share rows (a kernel of its own: the merge costs the other one registers)
__global__ void __launch_bounds__(256, 2) wide_attention_kernel(const float *__restrict__ q, const float *__restrict__ k_cache, const float *__restrict__ v_cache,
                                                                float *__restrict__ out, uint32_t q_dim, uint32_t kv_mul, uint32_t row_stride,
                                                                uint32_t head_stride, uint32_t pos0, uint32_t ntok, float4 *__restrict__ scratch,
                                                                uint32_t *__restrict__ counters)
{
    constexpr uint32_t LD = HD + 4, LP = 64 + 4, NC = HD / 64, NP = HD / 16;
    extern __shared__ float wa_smem[];
    float *qs = wa_smem, *ks = qs + 64 * LD, *vs = ks, *ps = ks + 64 * LD;   // K and V tiles take turns in one buffer
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t h = blockIdx.x, t0 = (gridDim.y - 1 - blockIdx.y) * 64, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const uint32_t nq = ntok - t0 < 64 ? ntok - t0 : 64;
    // the block's tiles of rows (all of them, to the last row that is attended to, where none are shared)
    uint32_t c_begin = 0, c_end = 0, nz = 1;
    if constexpr (SHARED) {
        const uint32_t ntiles = (pos0 + t0 + nq - 1) / 64 + 1;
        nz = gridDim.z < ntiles ? gridDim.z : ntiles;
        if (blockIdx.z >= nz) return;
        c_begin = 64 * (blockIdx.z * ntiles / nz);
        c_end = 64 * ((blockIdx.z + 1) * ntiles / nz);
    }
    const float *kh = k_cache + (size_t)(h / kv_mul) * head_stride, *vh = v_cache + (size_t)(h / kv_mul) * head_stride;
    const float inv_sqrt = 1.0f / sqrtf((float)HD);
    for (uint32_t i = tid; i < 64 * HD / 4; i += 256) {
        const uint32_t r = i / (HD / 4), e = 4 * (i % (HD / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nq) v = *reinterpret_cast<const float4 *>(q + (size_t)(t0 + r) * q_dim + h * HD + e);
        *reinterpret_cast<float4 *>(qs + r * LD + e) = v;
    }
    float mrun[4], lrun[4];
    float4 acc[4][NC];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        mrun[i] = -INFINITY;
        lrun[i] = 0.0f;
#pragma unroll
        for (uint32_t c = 0; c < NC; c++) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint32_t last = pos0 + t0 + nq - 1;
    // a tile travels through registers, requested one phase before it is needed
    float4 pre[NP];
    auto fetch = [&](const float *base, uint32_t c0) {
#pragma unroll
        for (uint32_t k = 0; k < NP; k++) {
            const uint32_t i = tid + 256 * k, r = i / (HD / 4), e = 4 * (i % (HD / 4));
            pre[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c0 + r <= last) pre[k] = *reinterpret_cast<const float4 *>(base + (size_t)(c0 + r) * row_stride + e);
        }
    };
    auto place = [&](bool flag) -> int {   // nonzero when any thread passes a flag
        __syncthreads();   // the tile before has been read
#pragma unroll
        for (uint32_t k = 0; k < NP; k++) {
            const uint32_t i = tid + 256 * k, r = i / (HD / 4), e = 4 * (i % (HD / 4));
            *reinterpret_cast<float4 *>(ks + r * LD + e) = pre[k];
        }
        return __syncthreads_or(flag);
    };
    auto mine = [&](uint32_t c) { return SHARED ? c < c_end : c <= last; };
    fetch(kh, c_begin);
    for (uint32_t c0 = c_begin; mine(c0); c0 += 64) {
        place(false);
        fetch(vh, c0);
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[i][j] = 0.0f;
#pragma unroll 4
        for (uint32_t e = 0; e < HD; e += 4) {
            float4 qv[4], kv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) qv[i] = *reinterpret_cast<const float4 *>(qs + (4 * ty + i) * LD + e);
#pragma unroll
            for (int j = 0; j < 4; j++) kv[j] = *reinterpret_cast<const float4 *>(ks + (tx + 16 * j) * LD + e);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    s[i][j] = fmaf(qv[i].x, kv[j].x, s[i][j]);
                    s[i][j] = fmaf(qv[i].y, kv[j].y, s[i][j]);
                    s[i][j] = fmaf(qv[i].z, kv[j].z, s[i][j]);
                    s[i][j] = fmaf(qv[i].w, kv[j].w, s[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t p = pos0 + t0 + 4 * ty + i;   // positions past the pass (zero queries) follow the same rule
            float mx = mrun[i];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t row = c0 + tx + 16 * j;
                s[i][j] = (row <= p && row <= last) ? s[i][j] * inv_sqrt : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            // -inf as long as the block has met no row that the position attends to
            const float rs = mx == -INFINITY ? 1.0f : expf(mrun[i] - mx);
            mrun[i] = mx;
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float w = s[i][j] == -INFINITY ? 0.0f : expf(s[i][j] - mx);
                ps[(4 * ty + i) * LP + tx + 16 * j] = w;
                sum += w;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            lrun[i] = lrun[i] * rs + sum;
#pragma unroll
            for (uint32_t c = 0; c < NC; c++) { acc[i][c].x *= rs; acc[i][c].y *= rs; acc[i][c].z *= rs; acc[i][c].w *= rs; }
        }
        // Where the tile holds rows that some of the block's positions do not attend to, their weight of 0 keeps a row out of
        // the sum only if the row is finite; with an infinity or NaN about, such rows are left out one by one.
        float z = 0.0f;   // 0 times every element: NaN if one is not finite
        if (c0 + 63 > pos0 + t0) {
#pragma unroll
            for (uint32_t k = 0; k < NP; k++) z = fmaf(pre[k].x, 0.0f, fmaf(pre[k].y, 0.0f, fmaf(pre[k].z, 0.0f, fmaf(pre[k].w, 0.0f, z))));
        }
        const bool one_by_one = place(z != 0.0f) != 0;
        if (mine(c0 + 64)) fetch(kh, c0 + 64);
        if (one_by_one) {
#pragma unroll 1
            for (uint32_t j = 0; j < 64; j++) {
#pragma unroll
                for (uint32_t c = 0; c < NC; c++) {
                    const float4 vv = *reinterpret_cast<const float4 *>(vs + j * LD + 64 * c + 4 * tx);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (c0 + j > pos0 + t0 + 4 * ty + i) continue;
                        const float w = ps[(4 * ty + i) * LP + j];
                        acc[i][c].x = fmaf(w, vv.x, acc[i][c].x);
                        acc[i][c].y = fmaf(w, vv.y, acc[i][c].y);
                        acc[i][c].z = fmaf(w, vv.z, acc[i][c].z);
                        acc[i][c].w = fmaf(w, vv.w, acc[i][c].w);
                    }
                }
            }
            continue;
        }
#pragma unroll 2
        for (uint32_t j = 0; j < 64; j += 4) {
            float4 pv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) pv[i] = *reinterpret_cast<const float4 *>(ps + (4 * ty + i) * LP + j);
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
#pragma unroll
                for (uint32_t c = 0; c < NC; c++) {
                    const float4 vv = *reinterpret_cast<const float4 *>(vs + (j + jj) * LD + 64 * c + 4 * tx);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float w = jj == 0 ? pv[i].x : jj == 1 ? pv[i].y : jj == 2 ? pv[i].z : pv[i].w;
                        acc[i][c].x = fmaf(w, vv.x, acc[i][c].x);
                        acc[i][c].y = fmaf(w, vv.y, acc[i][c].y);
                        acc[i][c].z = fmaf(w, vv.z, acc[i][c].z);
                        acc[i][c].w = fmaf(w, vv.w, acc[i][c].w);
                    }
                }
            }
        }
    }
    if constexpr (SHARED) {
        __shared__ uint32_t s_last;
        constexpr uint32_t SLOT = WA_SLOT<HD>;   // float4 per block: sums [register][thread], then (maximum, denominator) [row]
        const uint32_t pair = blockIdx.x * gridDim.y + blockIdx.y;
        float4 *all = scratch + (size_t)pair * gridDim.z * SLOT, *part = all + (size_t)blockIdx.z * SLOT;
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (uint32_t c = 0; c < NC; c++) part[(i * NC + c) * 256 + tid] = acc[i][c];
            if (tx == 0) reinterpret_cast<float2 *>(part + 4 * NC * 256)[4 * ty + i] = make_float2(mrun[i], lrun[i]);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicInc(counters + pair, nz - 1) == nz - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float mx = -INFINITY;
            for (uint32_t zz = 0; zz < nz; zz++) mx = fmaxf(mx, __ldcg(reinterpret_cast<const float2 *>(all + zz * SLOT + 4 * NC * 256) + 4 * ty + i).x);
            lrun[i] = 0.0f;
#pragma unroll
            for (uint32_t c = 0; c < NC; c++) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t zz = 0; zz < nz; zz++) {
                const float4 *other = all + zz * SLOT;
                const float2 ml = __ldcg(reinterpret_cast<const float2 *>(other + 4 * NC * 256) + 4 * ty + i);
                if (ml.x == -INFINITY && ml.y == 0.0f) continue;   // nothing but rows the position does not attend to
                const float w = expf(ml.x - mx);
                lrun[i] = fmaf(ml.y, w, lrun[i]);
#pragma unroll
                for (uint32_t c = 0; c < NC; c++) {
                    const float4 v = __ldcg(other + (i * NC + c) * 256 + tid);
                    acc[i][c].x = fmaf(v.x, w, acc[i][c].x);
                    acc[i][c].y = fmaf(v.y, w, acc[i][c].y);
                    acc[i][c].z = fmaf(v.z, w, acc[i][c].z);
                    acc[i][c].w = fmaf(v.w, w, acc[i][c].w);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (4 * ty + i < nq) {
#pragma unroll
            for (uint32_t c = 0; c < NC; c++) {
                const float4 v = make_float4(acc[i][c].x / lrun[i], acc[i][c].y / lrun[i], acc[i][c].z / lrun[i], acc[i][c].w / lrun[i]);
                *reinterpret_cast<float4 *>(out + (size_t)(t0 + 4 * ty + i) * q_dim + h * HD + 64 * c + 4 * tx) = v;
            }
        }
    }
}

template <uint32_t HD>
static int launch_wide_attention_hd(const float *q, const float *k_cache, const float *v_cache, float *out, uint32_t n_heads, uint32_t kv_mul, uint32_t row_stride,
                                    uint32_t head_stride, uint32_t pos0, uint32_t ntok, float *scratch, uint32_t *counters, bool *attrs, cudaStream_t stream)
{
    const size_t smem = (size_t)(2 * 64 * (HD + 4) + 64 * 68) * sizeof(float);
    if (!*attrs) {
        WGB_CUDA(cudaFuncSetAttribute(wide_attention_kernel<HD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        WGB_CUDA(cudaFuncSetAttribute(wide_attention_kernel<HD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        *attrs = true;
    }
    // Blocks for the rows of one (head, tile of positions): as many as are resident at once, with two tiles of rows or more
    // each.  Sixteen positions of a two-layer model of 7B widths (32 blocks) at position 4000: 2045 us a pass with one block
    // each, 631 with nine (eight-position passes 759); a pass with more blocks than half of what is resident is as before.
    const uint32_t pairs = n_heads * ((ntok + 63) / 64), tiles = (pos0 + ntok + 63) / 64;
    uint32_t nz = scratch && counters ? WA_BLOCKS * (uint32_t)sm_count() / pairs : 1u;
    if (nz > tiles / 2) nz = tiles / 2;
    if (nz < 1) nz = 1;
    void (*kernel)(const float *, const float *, const float *, float *, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, float4 *, uint32_t *) =
        nz > 1 ? wide_attention_kernel<HD, true> : wide_attention_kernel<HD, false>;
    WGB_CUDA(launch_pdl(kernel, dim3(n_heads, (ntok + 63) / 64, nz), dim3(256), smem, stream, q, k_cache, v_cache, out, n_heads * HD, kv_mul,
                        row_stride, head_stride, pos0, ntok, reinterpret_cast<float4 *>(scratch), counters));
    return WGB_OK;
}

// What blocks that share rows leave for one another; the counters start at zero and return to it.
size_t prefill_wide_attention_scratch_floats(uint32_t head_size)
{
    return (size_t)WA_BLOCKS * sm_count() * 4 * (head_size == 64 ? WA_SLOT<64> : WA_SLOT<128>);
}
size_t prefill_wide_attention_counters() { return (size_t)WA_BLOCKS * sm_count(); }

bool prefill_wide_attention_supported(uint32_t head_size) { return head_size == 64 || head_size == 128; }

int launch_wide_attention(const float *q, const float *k_cache, const float *v_cache, float *out, uint32_t n_heads, uint32_t head_size, uint32_t kv_mul,
                          uint32_t row_stride, uint32_t head_stride, uint32_t pos0, uint32_t ntok, float *scratch, uint32_t *counters, cudaStream_t stream)
{
    DeviceState *ds = device_state();
    if (!ds) return WGB_ERR_CUDA;
    if (head_size == 64)
        return launch_wide_attention_hd<64>(q, k_cache, v_cache, out, n_heads, kv_mul, row_stride, head_stride, pos0, ntok, scratch, counters, &ds->wide_attn_attrs[0], stream);
    WGB_REQUIRE(head_size == 128, "wide prompt attention: head size %u", head_size);
    return launch_wide_attention_hd<128>(q, k_cache, v_cache, out, n_heads, kv_mul, row_stride, head_stride, pos0, ntok, scratch, counters, &ds->wide_attn_attrs[1], stream);
}

}  // namespace wgb
