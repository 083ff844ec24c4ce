// Matrix-vector kernels: the fused, TMA-fed kernel used by the models and by GemvQuant, and the
// generic per-format fallback.
//
// Fused kernel.  One persistent block per SM with three roles: sixteen consumer warps in two groups, a producer warp and up to
// three epilogue warps.
//   * A block takes row tiles -- sixteen rows, or eight where a matrix has too few to go round -- and walks each in stages of eight
//     units of columns (gemv_core.cuh).  The producer brings stage after stage into a ring in shared memory by tensor copies (TMA,
//     one per plane and eight rows, completion on an mbarrier), as far ahead as the ring reaches.  It starts before the
//     kernel waits for its predecessor in the stream (programmatic dependent launch): weights never depend on activations.
//     (Stages of whole rows, one bulk copy each, fit two or three times into the ring where rows are long.)
//   * The consumers build the shared image of the (normalised) input vector once.  The groups alternate stages; warp w of a group
//     takes unit w of its stages: the products of the tile's rows with one unit of columns on the tensor cores, a fold over the
//     four lanes of a row, and sixteen sums to shared memory.  Consumers never wait for each other or for the epilogue.
//     (Eight consumer warps and room for the next launch's block beside this one: 19.2 us for Q4_K 32000x4096 where sixteen take
//     13.8; two warps per scheduler do not cover the latencies of a unit.)
//   * An epilogue warp waits for the eight units of a stage, adds them in a fixed order to the sums of its tile, releases the
//     stage to the producer and after the last stage of a tile applies the epilogue (bias, residual, SiLU gate, GELU,
//     RoPE + KV-cache append), one lane per output unit.  Its global loads (bias, residual) are issued a tile ahead.
//   * Tile i belongs to block i % gridDim.x.
// Bound by HBM in long launches (Q4_K 32000x4096, us: 13.8, 5.4 TB/s; Q6_K 21.4, 5.0 TB/s; Q8_0 24.1, 5.8 TB/s; the dp4a kernel
// before took 16.0, 27.9 and 27.4), in short ones by the hand-over between launches: wait 0.6, input 0.4 (under load 0.8), staging
// 0.3, first unit 0.3 to 0.7, last sums and exit 0.5.
// Every wait is bounded in time: a waiter that runs out records an error code in the launch's status word and
// carries on with whatever is in shared memory, so the kernel always terminates.
#include "async_copy.cuh"
#include "gemv_core.cuh"
#include "kernels.h"
#include "qaccess.cuh"

#include <cstdio>
#include <cstdlib>
#include <type_traits>

namespace wgb {

constexpr int GEMV_NCONS = 2 * TILE_UNITS;          // consumer warps: two groups, a warp per unit of a stage
constexpr int GEMV_CONS_THREADS = GEMV_NCONS * 32;
constexpr int GEMV_PRODUCER = GEMV_NCONS;           // warp index of the producer
constexpr int GEMV_EPILOGUE = GEMV_NCONS + 1;       // warp index of the first epilogue warp
constexpr int GEMV_NEPI = 3;                        // epilogue warps (twenty warps: five per scheduler, 96 registers a thread)
constexpr int GEMV_NT = (GEMV_EPILOGUE + GEMV_NEPI) * 32;
constexpr uint32_t GEMV_MAX_STAGES = 12;
constexpr uint32_t GEMV_ROPE_TAB = 128;             // pair indices with a precomputed rotation
constexpr uint32_t GEMV_PART_BYTES = TILE_UNITS * 16 * 4;   // partial sums of a stage: [unit][row]
constexpr size_t GEMV_SMEM_BUDGET = 224 * 1024;     // dynamic shared memory per block

__device__ __forceinline__ float4 ld_act4(const float *p)
{
    return __ldcg(reinterpret_cast<const float4 *>(p));
}

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void cons_sync() { asm volatile("bar.sync 1, %0;" ::"n"(GEMV_CONS_THREADS) : "memory"); }

// ---- tiles -------------------------------------------------------------------------------------
struct Part {
    int mat;
    uint32_t row0;
};

// n / d by a multiplication, for n * d < 2^32 and d > 1: magic = ceil(2^32 / d).  (A division is some fifty dependent instructions, and the
// epilogue warp of a q/k/v launch, which had four per tile, took longer over its tiles than the consumers.)  d = 1: magic = 0.
__device__ __forceinline__ uint32_t small_div(uint32_t n, uint32_t magic) { return magic ? __umulhi(n, magic) : n; }

// Parts of row tile `ti`: one run of up to tile_rows rows of one matrix, or two of up to eight (gate and up, the two halves of
// a Neox head) that take rows 0.. and 8.. of the tile.  `n`: rows per part.  Returns the number of parts.
__device__ __forceinline__ int tile_parts(const GemvArgs &a, const int EPI, uint32_t ti, Part (&parts)[2], uint32_t &n)
{
    if (EPI == EPI_SILU_PAIR) {
        const uint32_t r0 = ti * TILE_ROWS;
        n = min(TILE_ROWS, a.mat[0].nrows - r0);
        parts[0] = { 0, r0 };
        parts[1] = { 1, r0 };
        return 2;
    }
    int s = 0;
    if (EPI == EPI_QKV_ROPE) {
        s = ti < a.tq ? 0 : (ti < a.tq + a.tk ? 1 : 2);
        ti -= s == 0 ? 0 : (s == 1 ? a.tq : a.tq + a.tk);
        if (s < 2 && a.rope_variant == WGB_ROPE_NEOX) {
            const uint32_t half = a.head_size / 2, head = small_div(ti, a.per_head_magic), o = (ti - head * a.per_head) * TILE_ROWS;
            const uint32_t r0 = head * a.head_size + o;
            n = min(TILE_ROWS, half - o);
            parts[0] = { s, r0 };
            parts[1] = { s, r0 + half };
            return 2;
        }
    }
    const uint32_t r0 = ti * a.tile_rows;
    n = min(a.tile_rows, a.mat[s].nrows - r0);
    parts[0] = { s, r0 };
    return 1;
}

__device__ __forceinline__ float gelu_f32(float x)
{
    // UnaryOp::Gelu, crates/wgml/src/ops/unary.rs:106-110
    const float GELU_COEF_A = 0.044715f, SQRT_2_OVER_PI = 0.7978846f;
    return 0.5f * x * (1.0f + tanhf(SQRT_2_OVER_PI * x * (1.0f + GELU_COEF_A * x * x)));
}

// Output units of a tile (a unit = the tile rows that make one output: a row, or a pair) and the
// tile rows of unit u.
__device__ __forceinline__ uint32_t tile_outputs(const int EPI, const Part (&parts)[2], int nparts, uint32_t n)
{
    if (EPI == EPI_QKV_ROPE && nparts == 1 && parts[0].mat < 2) return n / 2;   // adjacent pairs
    return n;
}
__device__ __forceinline__ void output_rows(const int EPI, const Part (&parts)[2], int nparts, uint32_t u, uint32_t &ra, uint32_t &rb)
{
    if (EPI == EPI_SILU_PAIR || (EPI == EPI_QKV_ROPE && nparts == 2)) { ra = u; rb = TILE_ROWS + u; }
    else if (EPI == EPI_QKV_ROPE && parts[0].mat < 2) { ra = 2 * u; rb = 2 * u + 1; }
    else { ra = u; rb = u; }
}

// What the epilogue of one output unit needs besides the dot products; gathered before the unit's
// sums are ready so that the global loads overlap the consumers' work.
struct EpiCtx {
    bool on;            // the lane has a unit
    bool v;             // EPI_QKV_ROPE: of the value matrix (no rotation)
    uint32_t ra, rb;    // tile rows of the unit
    uint32_t r0, r1;    // output rows of the unit (matrix row indices)
    uint32_t d0, d1;    // EPI_QKV_ROPE: their offsets from `dst`
    float b0, b1;       // bias of r0 / r1, or the residual in b1 for EPI_RESIDUAL
    float sn, cs;       // RoPE rotation
    float *dst;         // EPI_QKV_*: where the rows of the unit go
};

// `pos`: the step's position (EPI_QKV_*).
__device__ __forceinline__ EpiCtx epi_prepare(const GemvArgs &a, const int EPI, uint32_t ti, uint32_t t, uint32_t pos, const float2 *rope_tab)
{
    EpiCtx c = {};
    Part parts[2];
    uint32_t n = 0;
    const int nparts = tile_parts(a, EPI, ti, parts, n);
    c.on = t < tile_outputs(EPI, parts, nparts, n);
    if (!c.on) return c;
    output_rows(EPI, parts, nparts, t, c.ra, c.rb);
    c.v = EPI == EPI_QKV_ROPE && parts[0].mat == 2;
    if (EPI == EPI_STORE || EPI == EPI_RESIDUAL || EPI == EPI_GELU) {
        c.r0 = parts[0].row0 + t;
        if (a.bias) c.b0 = a.bias[c.r0];
        if (EPI == EPI_RESIDUAL) c.b1 = a.residual[c.r0];
    } else if (EPI == EPI_SILU_PAIR) {
        c.r0 = parts[0].row0 + t;
    } else if (EPI == EPI_QKV_ROPE) {
        const int s = parts[0].mat;
        const float *bias = s == 0 ? a.bias : (s == 1 ? a.bias_k : a.bias_v);
        const uint32_t rstr = a.kv_row_stride ? a.kv_row_stride : a.kv_dim;
        c.dst = s == 0 ? a.out : ((s == 1 ? a.k_cache : a.v_cache) + (size_t)pos * rstr);
        if (s == 2) {
            c.r0 = c.r1 = parts[0].row0 + t;
        } else if (nparts == 2) {   // Neox: pairs (r0 + t, r0 + t + head_size / 2)
            c.r0 = parts[0].row0 + t;
            c.r1 = parts[1].row0 + t;
        } else {                    // Original: adjacent pairs
            c.r0 = parts[0].row0 + 2 * t;
            c.r1 = c.r0 + 1;
        }
        // where rows r0 / r1, two of one head, land: q as is, k / v by (head, element) in the cache's layout
        const uint32_t head = small_div(c.r0, a.head_magic), e0 = c.r0 - head * a.head_size;
        c.d0 = s != 0 && a.kv_row_stride ? head * a.kv_head_stride + e0 : c.r0;
        c.d1 = c.d0 + (c.r1 - c.r0);
        if (bias) {
            c.b0 = bias[c.r0];
            c.b1 = bias[c.r1];
        }
        if (s < 2) {
            // RoPE (ops/rope.wgsl:36-77): angle = pos * base^(-(2i % head_size) / head_size) for pair (r0, r1)
            const float2 r = rope_tab[a.rope_variant == WGB_ROPE_NEOX ? e0 : e0 / 2];
            c.cs = r.x;
            c.sn = r.y;
        }
    } else if (EPI == EPI_QKV_SPLIT) {
        const uint32_t row = parts[0].row0 + t, d = a.kv_dim;
        c.r0 = row;
        if (a.bias) c.b0 = a.bias[row];
        if (row < d) c.dst = a.out + row;
        else if (row < 2 * d) c.dst = a.k_cache + (size_t)pos * d + (row - d);
        else c.dst = a.v_cache + (size_t)pos * d + (row - 2 * d);
    }
    return c;
}

// ya / yb: finished dot products of the unit's first / second tile row.
template <bool PEERS>
__device__ __forceinline__ void epi_finish(const GemvArgs &a, const int EPI, const EpiCtx &c, float ya, float yb)
{
    if (!c.on) return;
    if (EPI == EPI_STORE || EPI == EPI_RESIDUAL || EPI == EPI_GELU) {
        float y = ya;
        if (a.bias) y += c.b0;
        if (EPI == EPI_RESIDUAL) y = c.b1 + y;
        if (EPI == EPI_GELU) y = gelu_f32(y);
        if (PEERS && a.peer_out.n) {
            for (uint32_t p = 0; p < a.peer_out.n; p++) a.peer_out.mail[p][c.r0] = y;   // every rank's mailbox, own included
        } else {
            a.out[c.r0] = y;
        }
    } else if (EPI == EPI_SILU_PAIR) {
        a.out[c.r0] = yb * (ya / (1.0f + expf(-ya)));
    } else if (EPI == EPI_QKV_ROPE) {
        if (c.v) {
            c.dst[c.d0] = ya + c.b0;
        } else {
            const float y0 = ya + c.b0, y1 = yb + c.b1;
            c.dst[c.d0] = c.cs * y0 - c.sn * y1;
            c.dst[c.d1] = c.sn * y0 + c.cs * y1;
        }
    } else if (EPI == EPI_QKV_SPLIT) {
        *c.dst = ya + c.b0;
    }
}

// Weights pass through L2 once per step: they are the first to go, ahead of activations, cache rows and code.
__device__ __forceinline__ uint64_t streaming_policy()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void tile_copy(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t row, uint32_t bar, uint64_t policy)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
                 "l"(map), "r"(x), "r"(row), "r"(bar), "l"(policy)
                 : "memory");
}

// Bytes of planes 0 .. pl - 1 of a tile of eight rows.
__host__ __device__ constexpr uint32_t tile_offset(int qt, int pl)
{
    uint32_t n = 0;
    for (int i = 0; i < pl; i++) n += TILE_ROWS * tile_box(qt, i);
    return n;
}
__host__ __device__ constexpr uint32_t tile_bytes(int qt) { return tile_offset(qt, tile_planes(qt)); }

// One kernel per block format, prologue and epilogue.  The launches of a decode step alternate between
// kernels and evict one another's code from the instruction caches (measured: +0.7 us per launch when two
// kernels alternate, +1.7 us with four), so what matters is how little code one launch executes: loops over the input and the tiles
// are rolled, and the exchange between tensor-parallel ranks (PEERS) is compiled apart (q/k/v of Q4_K: 57 KB of code,
// 26 without either; 68.2 and 64.4 ms for 48 steps of a 7B model, 13.9 and 12.9 for 136 of a tiny one).
template <int QT, int PRO_T, int EPI_T, bool PEERS>
__global__ void __launch_bounds__(GEMV_NT, 1) gemv_kernel(const __grid_constant__ GemvArgs a)
{
    using U = Unit<QT>;
    constexpr int PRO = PRO_T, EPI = EPI_T;
    constexpr int NPL = tile_planes(QT);
    extern __shared__ uint4 smem4[];
    __shared__ __align__(16) float red[2 * GEMV_NCONS];   // sums over the consumer warps: RMSNorm of squares, LayerNorm of values and of squared deviations
    __shared__ __align__(8) unsigned long long bars[3 * GEMV_MAX_STAGES];
    __shared__ float2 rope_tab[GEMV_ROPE_TAB];     // (cos, sin) per pair index of a head (EPI_QKV_ROPE)

    const uint32_t K = a.mat[0].ncols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nstage = a.nstage, units = a.units, nchunk = a.nchunk;
    // shared memory: image of the input, partial sums of every slot, the ring (128-byte aligned)
    const uint32_t smem0 = smem_addr(smem4), skip = ((smem0 + 127) & ~127u) - smem0;
    uint8_t *image = reinterpret_cast<uint8_t *>(smem4) + skip;
    float *part = reinterpret_cast<float *>(image + a.part_offset);      // [slot][unit][row]
    const uint32_t ring = smem0 + skip + a.ring_offset;
    const uint32_t full0 = smem_addr(&bars[0]), done0 = full0 + 8 * GEMV_MAX_STAGES, empty0 = done0 + 8 * GEMV_MAX_STAGES;

    // one thread per barrier: initialising them one after the other would cost a microsecond
    if (threadIdx.x < 3 * nstage) {
        const uint32_t kind = threadIdx.x / nstage, s = threadIdx.x - kind * nstage;
        mbar_init(full0 + 8 * (kind * GEMV_MAX_STAGES + s), kind == 1 ? TILE_UNITS : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    // Which use of a ring slot a barrier stands at is read from its parity, so a waiter must know that the use before is through.
    //   Producer (`empty`): it walks all stages.  Consumers (`full`): the slots of a group are its own (the ring is even, or not used
    //   twice), and it walks them in order.  Epilogue warps (`done`): their own tile before is through, and with it, since the
    //   groups go in order, everything up to it; plan() has no more of them than the ring allows for.
    if (warp == GEMV_PRODUCER) {
        // ------------------------------ producer ------------------------------
        const uint32_t oct = a.octets, pl = (uint32_t)lane % NPL, o = (uint32_t)lane / NPL;   // a lane per copy: plane, eight rows
        if (o >= oct) return;
        const uint32_t pmask = (1u << (NPL * oct)) - 1u;
        const uint32_t box = pl == 0 ? tile_box(QT, 0) : pl == 1 ? tile_box(QT, 1) : pl == 2 ? tile_box(QT, 2) : tile_box(QT, 3);
        const uint32_t step = (pl == 0 ? tile_step(QT, 0) : pl == 1 ? tile_step(QT, 1) : pl == 2 ? tile_step(QT, 2) : tile_step(QT, 3)) / 8;
        const uint32_t off = pl == 0 ? 0u : pl == 1 ? tile_offset(QT, 1) : pl == 2 ? tile_offset(QT, 2) : tile_offset(QT, 3);
        const uint32_t dst0 = ring + off * oct + o * TILE_ROWS * box;
        const uint64_t policy = streaming_policy();
        uint32_t s = 0, phase = 1, filled = 0;
        for (uint32_t ti = blockIdx.x; ti < a.ntiles; ti += gridDim.x) {
            Part parts[2];
            uint32_t n = 0;
            const int nparts = tile_parts(a, EPI, ti, parts, n);
            const uint32_t row = nparts == 2 ? parts[o].row0 : parts[0].row0 + o * TILE_ROWS;
            const CUtensorMap *map = &a.map[parts[0].mat + (EPI == EPI_SILU_PAIR ? o : 0)][pl];
            for (uint32_t c = 0; c < nchunk; c++) {
                if (lane == 0) {
                    if (filled >= nstage) mbar_wait(empty0 + 8 * s, phase, a.err, 2, a.wait_ns);
                    mbar_expect_tx(full0 + 8 * s, oct * tile_bytes(QT));
                }
                __syncwarp(pmask);
                tile_copy(dst0 + s * a.stage_bytes, map, c * step, row, full0 + 8 * s, policy);
                filled++;
                if (++s == nstage) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
        return;
    }
    if (warp >= GEMV_EPILOGUE) {
        // ------------------------------ epilogue ------------------------------
        // The warps take the block's tiles in turn.  (One warp needed 1.2 us per tile of a q/k/v launch, all of it latency, and ended
        // a launch of five tiles per block a microsecond after the consumers.)
        const uint32_t nepi = a.nepi, first = (uint32_t)warp - GEMV_EPILOGUE;
        if (first >= nepi || blockIdx.x + first * gridDim.x >= a.ntiles) return;
        pdl_wait();
        const uint32_t pos = EPI == EPI_QKV_ROPE || EPI == EPI_QKV_SPLIT ? __ldcg(a.pos) : 0u;
        if (EPI == EPI_QKV_ROPE) {
            // rotation of every pair index of a head at this position (ops/rope.wgsl:36-77)
#pragma unroll 1
            for (uint32_t i = lane; i < a.head_size / 2; i += 32) {
                float sn, cs;
                sincosf((float)pos * __ldg(a.rope_freq + i), &sn, &cs);
                rope_tab[i] = make_float2(cs, sn);
            }
            __syncwarp();
        }
        const uint32_t row = (uint32_t)lane & 15, half = (uint32_t)lane >> 4;   // a lane adds four units of a row
        uint32_t s = 0, phase = 0;
        auto skip_stages = [&](uint32_t n) {
            s += n;
            while (s >= nstage) {
                s -= nstage;
                phase ^= 1;
            }
        };
        skip_stages(first * nchunk);
        float rms_scale = 1.0f;
        bool have_scale = false;
        // The next tile's loads are out before this tile's sums are waited for (the first round only issues them).
        EpiCtx next = {};
#pragma unroll 1
        for (uint32_t ti = blockIdx.x + first * gridDim.x, round = 0;; ti += nepi * gridDim.x, round++) {
            const EpiCtx c = next;
            if (ti < a.ntiles) next = epi_prepare(a, EPI, ti, lane, pos, rope_tab);
            if (round == 0) continue;
            // Four sums take the stages in turn: one chain of them all rounds long rows worse than the dp4a kernel before, which spread
            // a row over up to sixteen warps (2-norm against 64 bits, that kernel, one chain, four: f32 22016 columns 1.24e-7, 1.48e-7,
            // 1.12e-7, 8192 columns 1.13e-7, 1.13e-7, 0.99e-7; Q8_0 46080 columns 2.83e-7, 2.96e-7, 2.81e-7).  Decode steps as with one
            // chain; what a sum loses, carried along exactly: 0.8 % slower.
            float acc[4] = {};
#pragma unroll 1
            for (uint32_t left = units; left; ) {
                const uint32_t in_stage = min(left, TILE_UNITS);
                mbar_wait(done0 + 8 * s, phase, a.err, 3, a.wait_ns);
                const float *p = part + s * (TILE_UNITS * 16) + half * 64 + row;
                float t[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) t[k] = half * 4 + k < in_stage ? p[k * 16] : 0.0f;
                // (t one after the other: a tenth more rounding error in a layer)
                const float sum = acc[0] + ((t[0] + t[1]) + (t[2] + t[3]));
#pragma unroll
                for (int k = 0; k < 3; k++) acc[k] = acc[k + 1];
                acc[3] = sum;
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * s);   // stage and partial sums may be overwritten
                left -= in_stage;
                skip_stages(1);
            }
            skip_stages((nepi - 1) * nchunk);
            float y = (acc[0] + acc[1]) + (acc[2] + acc[3]);
            y += __shfl_xor_sync(0xffffffffu, y, 16);
            if (PRO == PRO_RMS) {
                if (!have_scale) {
                    // every consumer warp wrote its sum of squares before its first arrival on a `done` barrier
                    float ss = 0.0f;
#pragma unroll
                    for (int w = 0; w < GEMV_NCONS; w++) ss += red[w];
                    rms_scale = 1.0f / sqrtf(ss / (float)K + a.eps);
                    have_scale = true;
                }
                y *= rms_scale;
            }
            const float ya = __shfl_sync(0xffffffffu, y, c.ra), yb = __shfl_sync(0xffffffffu, y, c.rb);
            epi_finish<PEERS>(a, EPI, c, ya, yb);
            if (ti >= a.ntiles) break;
        }
        if (PEERS && a.peer_out.n) {
            // The block's partial rows are on their way to the peers; the last block of the launch raises
            // this rank's flag everywhere once every block's stores are visible system-wide.
            __threadfence_system();
            __syncwarp();
            uint32_t last = 0;
            if (lane == 0) {
                const uint32_t t = atomicAdd(a.peer_out.ticket, 1u);
                last = (t == gridDim.x - 1);
                if (last) *a.peer_out.ticket = 0;   // ready for the next step
            }
            last = __shfl_sync(0xffffffffu, last, 0);
            if (last) {
                __threadfence_system();
                if ((uint32_t)lane < a.peer_out.n) atomicAdd_system(a.peer_out.flag[lane], 1u);
            }
        }
        if (lane == 0) stamp_end(a.stamp);
        return;
    }

    // ------------------------------ consumers ------------------------------
    // What the input does not decide is worked out while the launch before drains.
    // Task loop, further down: the warps of a group take the units of a stage, the two groups alternate stages.  The digits of the inputs
    // of a unit stay in registers as long as the unit does (one or two stages per tile).  Lane 4g + t has rows g and g + 8 of the
    // tile; in a tile of eight rows, g twice.
    const XImage<QT> im(smem0 + skip, units);
    uint32_t held = ~0u, phase = 0;
    const uint32_t w = (uint32_t)warp % TILE_UNITS, group = (uint32_t)warp / TILE_UNITS, ngroups = nstage > 1 ? 2 : 1;
    const uint32_t g = (uint32_t)lane >> 2, oct = a.octets;
    uint32_t row_at[NPL], second[NPL];   // the lane's first row within a stage, from there to the second
#pragma unroll
    for (int q = 0; q < NPL; q++) {
        row_at[q] = ring + tile_offset(QT, q) * oct + g * tile_box(QT, q);
        second[q] = (oct - 1) * TILE_ROWS * tile_box(QT, q);
    }
    const uint32_t nst = (a.per_block - (a.rem_blocks != 0 && blockIdx.x >= a.rem_blocks ? 1u : 0u)) * nchunk;   // stages of this block
    uint32_t s = group, chunk = group < nchunk ? group : 0u;
    // The input, eight consecutive values per thread and round.  The norm weights are parameters, not products of the launch
    // before: the first round's (cold, HBM-latency) loads are issued ahead of the dependency wait.  A round's loads go out a
    // round ahead.
    const uint32_t nvec = K / 4, noct = (nvec + 1) / 2;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    struct Eight { float4 a, b; };
    auto load_param = [&](const float *p, uint32_t u) {
        Eight e = { zero4, zero4 };
        if (2 * u < nvec) e.a = __ldg(reinterpret_cast<const float4 *>(p) + 2 * u);
        if (2 * u + 1 < nvec) e.b = __ldg(reinterpret_cast<const float4 *>(p) + 2 * u + 1);
        return e;
    };
    auto load_vec = [&](uint32_t c) {
        if (!PEERS || !a.peer_in.n) return ld_act4(a.x + 4 * c);
        float4 v = __ldcg(reinterpret_cast<const float4 *>(a.peer_in.mail) + c);
        for (uint32_t r = 1; r < a.peer_in.n; r++) {
            const float4 w = __ldcg(reinterpret_cast<const float4 *>(a.peer_in.mail + (size_t)r * K) + c);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        if (blockIdx.x == 0) reinterpret_cast<float4 *>(a.peer_in.x_out)[c] = v;
        return v;
    };
    auto load_x = [&](uint32_t u) {
        Eight e = { zero4, zero4 };
        if (2 * u < nvec) e.a = load_vec(2 * u);
        if (2 * u + 1 < nvec) e.b = load_vec(2 * u + 1);
        return e;
    };
    const uint32_t u0 = threadIdx.x;
    Eight gain, bias;
    if (PRO != PRO_NONE) gain = load_param(a.norm_w, u0);
    if (PRO == PRO_LN) bias = load_param(a.norm_b, u0);
    pdl_wait();
    if (PEERS && a.peer_in.n) {
        // Partial products from every rank: wait for the flags, then add in rank order.  The wait is bounded
        // in time (a.peer_wait_ns); a wait that runs out leaves code 6 in the status word, and while the word
        // is non-zero no launch waits at all, so one missing rank costs one limit, not one per exchange.
        if (threadIdx.x < a.peer_in.n) {
            const uint32_t want = __ldcg(a.peer_in.epoch);
            const uint32_t *f = a.peer_in.flag + threadIdx.x;
            bool ok = false, give_up = a.err && ld_relaxed_u32(a.err) != 0;
            unsigned long long t0 = 0;
            for (uint32_t i = 0; !ok && !give_up; i++) {
                uint32_t v;
                asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
                ok = (int32_t)(v - want) >= 0;
                if (!ok && (i & 31u) == 31u) {
                    const unsigned long long t = global_ns();
                    if (!t0) t0 = t;
                    give_up = t - t0 > a.peer_wait_ns || (a.err && ld_relaxed_u32(a.err) != 0);
                }
            }
            if (!ok && a.err) atomicCAS(a.err, 0u, 6u);
            asm volatile("fence.acq_rel.sys;" ::: "memory");
        }
        cons_sync();
    }
    Eight x = load_x(u0);
    float mean = 0.0f, scale = 1.0f;
    if (PRO == PRO_LN) {
        // Two passes, mean and deviations from it; up to 4096 columns a thread's values stay in registers.
        auto total = [&](const auto &term, float *part_sums) {
            float v = 0.0f;
            Eight e = x;
#pragma unroll 1
            for (uint32_t u = u0; u < noct;) {
                v += term(e.a);
                if (2 * u + 1 < nvec) v += term(e.b);   // (only a dense f32 vector can end in the middle of eight)
                u += GEMV_CONS_THREADS;
                if (u < noct) e = load_x(u);
            }
            v = warp_sum(v);
            if (lane == 0) part_sums[warp] = v;
            cons_sync();
            const float4 *p = reinterpret_cast<const float4 *>(part_sums);   // every thread adds the sixteen
            float4 t = p[0];
#pragma unroll
            for (int i = 1; i < GEMV_NCONS / 4; i++) { t.x += p[i].x; t.y += p[i].y; t.z += p[i].z; t.w += p[i].w; }
            return (t.x + t.y) + (t.z + t.w);
        };
        mean = total([](const float4 v) { return (v.x + v.y) + (v.z + v.w); }, red) / (float)K;
        const float m2 = total([&](const float4 v) {
            const float p = v.x - mean, q = v.y - mean, r = v.z - mean, t = v.w - mean;
            return (p * p + q * q) + (r * r + t * t);
        }, red + GEMV_NCONS);
        scale = 1.0f / sqrtf(m2 / (float)K + 1.0e-5f);
    }
    {
        const XWriter<QT> xw(image, units);
        xw.pad(K, units, threadIdx.x, GEMV_CONS_THREADS);
        // RMSNorm: the scale is one factor for the whole vector, so it commutes with the dot products.  The input is staged as x * w,
        // the warps' sums of squares go to `red`, and the epilogue multiplies every finished dot product by
        // 1 / sqrt(mean square + eps).  No block-wide reduction ahead of the staging.
        auto transform = [&](float4 v, const float4 g, const float4 b) {
            if (PRO == PRO_RMS) {
                v.x *= g.x; v.y *= g.y; v.z *= g.z; v.w *= g.w;
            } else if (PRO == PRO_LN) {
                v.x = ((v.x - mean) * scale) * g.x + b.x; v.y = ((v.y - mean) * scale) * g.y + b.y;
                v.z = ((v.z - mean) * scale) * g.z + b.z; v.w = ((v.w - mean) * scale) * g.w + b.w;
            }
            return v;
        };
        float ss = 0.0f;
        // whole warps go round together (the writer shuffles): the bound is per warp, not per lane
#pragma unroll 1
        for (uint32_t u = u0; u - lane < noct; u += GEMV_CONS_THREADS) {
            const Eight xn = x, gn = gain, bn = bias;
            if (u - lane + GEMV_CONS_THREADS < noct) {
                x = load_x(u + GEMV_CONS_THREADS);
                if (PRO != PRO_NONE) gain = load_param(a.norm_w, u + GEMV_CONS_THREADS);
                if (PRO == PRO_LN) bias = load_param(a.norm_b, u + GEMV_CONS_THREADS);
            }
            if (PRO == PRO_RMS)
                ss += ((xn.a.x * xn.a.x + xn.a.y * xn.a.y) + (xn.a.z * xn.a.z + xn.a.w * xn.a.w)) +
                      ((xn.b.x * xn.b.x + xn.b.y * xn.b.y) + (xn.b.z * xn.b.z + xn.b.w * xn.b.w));
            xw.put8(u, transform(xn.a, gn.a, bn.a), transform(xn.b, gn.b, bn.b), 2 * u < nvec, 2 * u + 1 < nvec);
        }
        if (PRO == PRO_RMS) {
            ss = warp_sum(ss);
            if (lane == 0) red[warp] = ss;
        }
    }
    cons_sync();

    if (group >= ngroups) return;
    typename U::Digits digits;
    digits.clear();
    for (uint32_t it = group; it < nst; it += ngroups) {
        const uint32_t u = chunk * TILE_UNITS + w;
        if (u < units && u != held) {
            digits.load(im, u, lane);
            held = u;
        }
        mbar_wait(full0 + 8 * s, phase, a.err, 1, a.wait_ns);
        if (u < units) {
            uint32_t sa[NPL], sb[NPL];
#pragma unroll
            for (int q = 0; q < NPL; q++) {
                sa[q] = row_at[q] + s * a.stage_bytes;
                sb[q] = sa[q] + second[q];
            }
            float ya, yb;
            U::eval(sa, sb, w, digits, im, u, lane, ya, yb);
            // fold over the quad: even lanes keep row g, odd ones row g + 8
            const float send = lane & 1 ? ya : yb;
            float y = (lane & 1 ? yb : ya) + __shfl_xor_sync(0xffffffffu, send, 1);
            y += __shfl_xor_sync(0xffffffffu, y, 2);
            if ((lane & 2) == 0) part[(s * TILE_UNITS + w) * 16 + g + 8 * (lane & 1)] = y;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(done0 + 8 * s);
        s += ngroups;
        if (s >= nstage) {
            s -= nstage;
            phase ^= 1;
        }
        chunk += ngroups;
        while (chunk >= nchunk) chunk -= nchunk;
    }
}

// One warp per row, any format and layout, x read from global memory.
template <int QT>
__global__ void __launch_bounds__(256) gemv_generic_kernel(const __grid_constant__ QMat m, const float *__restrict__ x,
                                                           float *__restrict__ out)
{
    constexpr int BL = block_len(QT), BB = block_bytes(QT);
    const int lane = threadIdx.x & 31;
    for (uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5); row < m.nrows; row += gridDim.x * 8) {
        float acc = 0.0f;
        if constexpr (BL == 1) {
            for (uint32_t c = lane; c < m.ncols; c += 32)
                acc = fmaf(dequant_one<QT>(m.p[0] + ((size_t)row * m.ncols + c) * BB, 0, 0), x[c], acc);
        } else {
            // lane <-> 32-weight group, so the scale decode is hoisted out of the inner loop
            for (uint32_t grp = lane; grp < m.ncols / 32; grp += 32) {
                constexpr uint32_t GPB = BL / 32;  // 32-weight groups per block
                const uint32_t kb = grp / GPB, g = grp % GPB;
                float s = 0.0f;
                if (m.planar) {
                    for (int l = 0; l < 32; l++) s = fmaf(qmat_weight<QT>(m, row, grp * 32 + l), x[grp * 32 + l], s);
                } else {
                    const uint8_t *b = m.p[0] + (size_t)row * m.pitch[0] + (size_t)kb * BB;
                    for (int l = 0; l < 32; l++) s = fmaf(dequant_one<QT>(b, g, l), x[grp * 32 + l], s);
                }
                acc += s;
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) out[row] = acc;
    }
}

// ---------------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------------

// Shared memory in front of the ring (the image of the input) and whether a stage of `octets` times eight rows fits behind it.
static uint32_t image_bytes(const QMat &m) { return (uint32_t)((ximage_bytes(m.qtype, m.ncols) + 127) & ~(size_t)127); }
static bool gemv_fits(const QMat &m, uint32_t octets)
{
    return (size_t)image_bytes(m) + 128 + octets * tile_bytes(m.qtype) + GEMV_PART_BYTES <= GEMV_SMEM_BUDGET;
}

bool gemv_pairs_supported(const QMat &m) { return gemv_fast_supported(m) && gemv_fits(m, 2); }

bool gemv_fast_supported(const QMat &m)
{
    if (m.qtype != WGB_Q4_K && m.qtype != WGB_Q6_K && m.qtype != WGB_Q8_0 && m.qtype != WGB_F32) return false;
    for (int i = 0; i < m.nplanes; i++)
        if (((uintptr_t)m.p[i] % 16) != 0 || m.pitch[i] % 16 != 0) return false;
    if (!gemv_fits(m, 1)) return false;   // (columns up to 67328 of Q4_K, 61184 of Q6_K, 70272 of Q8_0, 53056 of F32)
    if (m.qtype == WGB_F32) return m.ncols % 4 == 0;
    if (m.ncols % 32 != 0) return false;
    if (m.qtype == WGB_Q8_0 || m.qtype == WGB_Q6_K) return m.planar != 0;
    return true;  // Q4_K raw
}

// Device status word shared by all launches on one device: 0, or the code of the first bounded wait that
// expired (1 consumer, 2 producer, 3 epilogue, 6 flags of the tensor-parallel peers, 7 / 8 streaming attention; tensor-core
// products: 11.. single vector, 21.. / 31.. / 41.. eight vectors Q4_K / Q6_K / Q8_0, 61.. wide passes).  While it is
// non-zero the kernels do not wait for peers at all.
static bool g_trace_plan = false;   // WGML_B200_TRACE_PLAN=1 prints the plan of every launch to stderr

uint32_t *gemv_status_word()
{
    DeviceState *d = device_state();
    return d ? d->err : nullptr;
}

int gemv_report_status(uint32_t v)
{
    if (!v) return WGB_OK;
    uint32_t *w = gemv_status_word();
    if (w) cudaMemset(w, 0, sizeof(uint32_t));
    return fail(WGB_ERR_TIMEOUT, "a bounded wait inside a kernel expired (code %u%s)", v,
                v == 6 ? ": a rank of the tensor-parallel group did not deliver its partial products in time" : "");
}

int gemv_check_status()
{
    uint32_t *w = gemv_status_word();
    if (!w) return WGB_OK;
    uint32_t v = 0;
    WGB_CUDA(cudaMemcpy(&v, w, sizeof(v), cudaMemcpyDeviceToHost));
    return gemv_report_status(v);
}

int replay_with_status(cudaGraphExec_t graph, size_t total, cudaStream_t stream, uint32_t *h_slots, StatusPoll &sp)
{
    uint32_t *word = gemv_status_word();
    for (int k = 0; k < 2; k++)
        if (!sp.ev[k]) WGB_CUDA(cudaEventCreateWithFlags(&sp.ev[k], cudaEventDisableTiming));
    h_slots[0] = h_slots[1] = 0;
    uint32_t seen = 0;
    for (size_t i = 0; i < total && !seen; i++) {
        if (word && i && i % STATUS_EVERY == 0) {
            const int k = (int)((i / STATUS_EVERY) & 1);
            if (i >= 2 * STATUS_EVERY) {
                WGB_CUDA(cudaEventSynchronize(sp.ev[k]));
                seen = h_slots[k];
                if (seen) break;
            }
            WGB_CUDA(cudaMemcpyAsync(h_slots + k, word, 4, cudaMemcpyDeviceToHost, stream));
            WGB_CUDA(cudaEventRecord(sp.ev[k], stream));
        }
        WGB_CUDA(cudaGraphLaunch(graph, stream));
    }
    if (seen) {
        WGB_CUDA(cudaStreamSynchronize(stream));
        return gemv_report_status(seen);
    }
    return WGB_OK;
}

void status_poll_destroy(StatusPoll &sp)
{
    for (int k = 0; k < 2; k++) {
        if (sp.ev[k]) cudaEventDestroy(sp.ev[k]);
        sp.ev[k] = nullptr;
    }
}

int make_tile_maps(const QMat &m, TileMaps &out)
{
    using Encode = decltype(&cuTensorMapEncodeTiled);
    static Encode encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        WGB_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found));
        if (found != cudaDriverEntryPointSuccess || !fn) return fail(WGB_ERR_UNSUPPORTED, "the driver has no tensor maps");
        encode = reinterpret_cast<Encode>(fn);
    }
    for (int i = 0; i < m.nplanes; i++) {
        // rows of eight-byte elements (rows, boxes and steps are multiples of 16 bytes); past the ends of a matrix zeros are read
        const cuuint64_t dims[2] = { m.pitch[i] / 8, m.nrows }, strides[1] = { m.pitch[i] };
        const cuuint32_t box[2] = { tile_box(m.qtype, i) / 8, TILE_ROWS }, ones[2] = { 1, 1 };
        const CUresult r = encode(&out.map[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<uint8_t *>(m.p[i]), dims, strides, box, ones,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(WGB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for plane %d of %u x %u", (int)r, i, m.nrows, m.ncols);
        out.p[i] = m.p[i];
    }
    out.nrows = m.nrows;
    return WGB_OK;
}

// Chooses rows per tile, ring depth and grid; fills the plan fields of `a`.  Returns false when the image of the input leaves no
// room for a stage (pairs of rows, which take sixteen; anything else falls back to eight where sixteen do not fit).
static bool plan(GemvArgs &a, size_t &smem_bytes, uint32_t &grid)
{
    const QMat &m0 = a.mat[0];
    const int qt = m0.qtype;
    const uint32_t sms = (uint32_t)sm_count();
    const bool pairs = a.epilogue == EPI_SILU_PAIR || (a.epilogue == EPI_QKV_ROPE && a.rope_variant == WGB_ROPE_NEOX);
    uint32_t total_rows = 0;
    for (int i = 0; i < (a.epilogue == EPI_SILU_PAIR ? 1 : a.nmat); i++) total_rows += a.mat[i].nrows;
    a.octets = !pairs && ((total_rows + TILE_ROWS - 1) / TILE_ROWS <= sms || !gemv_fits(m0, 2)) ? 1 : 2;
    a.tile_rows = a.octets * TILE_ROWS;
    auto tiles = [&](const QMat &m) { return (m.nrows + a.tile_rows - 1) / a.tile_rows; };
    if (a.epilogue == EPI_SILU_PAIR) a.ntiles = (m0.nrows + TILE_ROWS - 1) / TILE_ROWS;
    else if (a.epilogue == EPI_QKV_ROPE) {
        auto magic = [](uint32_t d) { return d > 1 ? (uint32_t)((0x100000000ull + d - 1) / d) : 0u; };
        a.per_head = (a.head_size / 2 + TILE_ROWS - 1) / TILE_ROWS;
        a.per_head_magic = magic(a.per_head);
        a.head_magic = magic(a.head_size);
        if ((uint64_t)total_rows * a.head_size >> 32 || a.head_size / 2 > GEMV_ROPE_TAB) return false;   // small_div, rope_tab
        a.tq = pairs ? a.mat[0].nrows / a.head_size * a.per_head : tiles(a.mat[0]);
        a.tk = pairs ? a.mat[1].nrows / a.head_size * a.per_head : tiles(a.mat[1]);
        a.ntiles = a.tq + a.tk + tiles(a.mat[2]);
    } else a.ntiles = tiles(m0);
    grid = a.ntiles < sms ? a.ntiles : sms;
    a.per_block = (a.ntiles + grid - 1) / grid;
    a.rem_blocks = a.ntiles % grid;
    a.units = image_units(qt, m0.ncols);
    a.nchunk = (a.units + TILE_UNITS - 1) / TILE_UNITS;
    a.stage_bytes = a.octets * tile_bytes(qt);
    const uint32_t need = a.per_block * a.nchunk;   // stages of the fullest block
    a.part_offset = image_bytes(m0);
    auto stages_in = [&](size_t budget) -> uint32_t {
        if (a.part_offset + 128 > budget) return 0;
        const size_t n = (budget - a.part_offset - 128) / (a.stage_bytes + GEMV_PART_BYTES);
        return (uint32_t)(n < GEMV_MAX_STAGES ? n : GEMV_MAX_STAGES);
    };
    const uint32_t ns = stages_in(GEMV_SMEM_BUDGET);
    if (!ns) return false;
    a.nstage = ns < need ? ns : need;
    if (a.nstage < need && a.nstage > 1) a.nstage &= ~1u;   // a slot is always the same group's
    a.nepi = 1;
    while (a.nepi < (uint32_t)GEMV_NEPI && !a.peer_out.n && (a.nstage >= need || a.nstage >= (a.nepi + 1) * (a.nchunk > 1 ? a.nchunk : 2))) a.nepi++;
    a.ring_offset = a.part_offset + a.nstage * GEMV_PART_BYTES;
    smem_bytes = 128 + a.ring_offset + (size_t)a.nstage * a.stage_bytes;
    return true;
}

// The prologue / epilogue combinations the models use, each its own kernel; the last column: with the exchange between ranks.
#define WGB_GEMV_VARIANTS(F)                                                                                                        \
    F(PRO_NONE, EPI_STORE, false) F(PRO_RMS, EPI_STORE, false) F(PRO_LN, EPI_STORE, false) F(PRO_NONE, EPI_RESIDUAL, false)         \
    F(PRO_RMS, EPI_SILU_PAIR, false) F(PRO_LN, EPI_GELU, false) F(PRO_RMS, EPI_QKV_ROPE, false) F(PRO_LN, EPI_QKV_SPLIT, false)     \
    F(PRO_NONE, EPI_STORE, true) F(PRO_NONE, EPI_RESIDUAL, true) F(PRO_RMS, EPI_STORE, true) F(PRO_RMS, EPI_SILU_PAIR, true)        \
    F(PRO_RMS, EPI_QKV_ROPE, true)

template <int QT>
static int set_smem_attr()
{
#define WGB_ATTR(PRO, EPI, PEERS)                                                                                                      \
    WGB_CUDA(cudaFuncSetAttribute(gemv_kernel<QT, PRO, EPI, PEERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMV_SMEM_BUDGET));
    WGB_GEMV_VARIANTS(WGB_ATTR)
#undef WGB_ATTR
    return WGB_OK;
}

// One-time set-up of the fused kernels on the current device: the status word and the opt-in to
// large dynamic shared memory.  Must first run outside stream capture (model creation does).
int gemv_global_init()
{
    DeviceState *d = device_state();
    if (!d) return WGB_ERR_CUDA;
    if (d->gemv_attrs) return WGB_OK;
    if (!d->err) {
        WGB_CUDA(cudaMalloc((void **)&d->err, sizeof(uint32_t)));
        WGB_CUDA(cudaMemset(d->err, 0, sizeof(uint32_t)));
    }
    const char *tp = getenv("WGML_B200_TRACE_PLAN");
    g_trace_plan = tp && tp[0] == '1';
    int rc;
    if ((rc = set_smem_attr<WGB_Q4_K>()) || (rc = set_smem_attr<WGB_Q6_K>()) || (rc = set_smem_attr<WGB_Q8_0>()) ||
        (rc = set_smem_attr<WGB_F32>()))
        return rc;
    d->gemv_attrs = true;
    return WGB_OK;
}

template <int QT>
static int launch_one(GemvArgs &a, cudaStream_t stream, bool pdl)
{
    void (*kern)(const GemvArgs) = nullptr;
    const bool peers = a.peer_in.n || a.peer_out.n;
#define WGB_PICK(PRO, EPI, PEERS) if (a.prologue == PRO && a.epilogue == EPI && peers == PEERS) kern = gemv_kernel<QT, PRO, EPI, PEERS>;
    WGB_GEMV_VARIANTS(WGB_PICK)
#undef WGB_PICK
    if (!kern) return fail(WGB_ERR_UNSUPPORTED, "no fused kernel for prologue %d / epilogue %d", a.prologue, a.epilogue);
    size_t smem = 0;
    uint32_t grid = 0;
    if (!plan(a, smem, grid)) return fail(WGB_ERR_UNSUPPORTED, "matrix shape does not fit the fused kernel");
    int rc = gemv_global_init();
    if (rc) return rc;
    for (int i = 0; i < a.nmat; i++) {
        const QMat &m = a.mat[i];
        TileMaps fresh;
        const TileMaps *maps = m.maps;
        if (!maps || maps->nrows != m.nrows || maps->p[0] != m.p[0]) {   // blocks in caller memory, a run of rows of a matrix
            if ((rc = make_tile_maps(m, fresh))) return rc;
            maps = &fresh;
        }
        for (int p = 0; p < m.nplanes; p++) a.map[i][p] = maps->map[p];
    }
    a.err = gemv_status_word();
    const WaitLimits wl = wait_limits();
    a.wait_ns = wl.local_ns;
    a.peer_wait_ns = wl.peer_ns;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(GEMV_NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    if (g_trace_plan)
        fprintf(stderr, "gemv plan: qt=%d rows=%u K=%u tile rows=%u tiles=%u stages per tile=%u ring=%u x %u grid=%u smem=%zu\n", QT, a.mat[0].nrows,
                a.mat[0].ncols, a.tile_rows, a.ntiles, a.nchunk, a.nstage, a.stage_bytes, grid, smem);
    WGB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
    return WGB_OK;
}

template <int QT>
static int launch_qt(GemvArgs &a, cudaStream_t stream, bool pdl)
{
    // the combinations the kernel is written for
    bool ok = false;
    switch (a.epilogue) {
    case EPI_STORE: ok = a.prologue == PRO_NONE || a.prologue == PRO_RMS || a.prologue == PRO_LN; break;
    case EPI_RESIDUAL: ok = a.prologue == PRO_NONE; break;
    case EPI_SILU_PAIR: ok = a.prologue == PRO_RMS && a.nmat == 2; break;
    case EPI_GELU: ok = a.prologue == PRO_LN; break;
    case EPI_QKV_ROPE: ok = a.prologue == PRO_RMS && a.nmat == 3; break;
    case EPI_QKV_SPLIT: ok = a.prologue == PRO_LN; break;
    }
    if (!ok) return fail(WGB_ERR_UNSUPPORTED, "no fused kernel for prologue %d / epilogue %d", a.prologue, a.epilogue);
    return launch_one<QT>(a, stream, pdl);
}

int launch_gemv(const GemvArgs &args, cudaStream_t stream, bool pdl)
{
    GemvArgs a = args;
    for (int i = 0; i < a.nmat; i++) {
        if (!gemv_fast_supported(a.mat[i])) return fail(WGB_ERR_UNSUPPORTED, "no fast kernel for tensor type %d", a.mat[i].qtype);
        if (a.mat[i].qtype != a.mat[0].qtype || a.mat[i].ncols != a.mat[0].ncols)
            return fail(WGB_ERR_UNSUPPORTED, "fused matrices differ in format or width");
    }
    if (((uintptr_t)a.x % 16) != 0) return fail(WGB_ERR_UNSUPPORTED, "input vector is not 16-byte aligned");
    switch (a.mat[0].qtype) {
    case WGB_Q4_K: return launch_qt<WGB_Q4_K>(a, stream, pdl);
    case WGB_Q6_K: return launch_qt<WGB_Q6_K>(a, stream, pdl);
    case WGB_Q8_0: return launch_qt<WGB_Q8_0>(a, stream, pdl);
    case WGB_F32: return launch_qt<WGB_F32>(a, stream, pdl);
    }
    return fail(WGB_ERR_UNSUPPORTED, "no fast kernel for tensor type %d", a.mat[0].qtype);
}

int launch_gemv_generic(const QMat &m, const float *x, float *out, cudaStream_t stream)
{
    uint32_t grid = (m.nrows + 7) / 8;
    const uint32_t cap = (uint32_t)sm_count() * 8;
    if (grid > cap) grid = cap;
#define WGB_GENERIC_CASE(T) case T: gemv_generic_kernel<T><<<grid, 256, 0, stream>>>(m, x, out); break;
    switch (m.qtype) {
        WGB_GENERIC_CASE(WGB_F32) WGB_GENERIC_CASE(WGB_F16) WGB_GENERIC_CASE(WGB_Q4_0) WGB_GENERIC_CASE(WGB_Q4_1)
        WGB_GENERIC_CASE(WGB_Q5_0) WGB_GENERIC_CASE(WGB_Q5_1) WGB_GENERIC_CASE(WGB_Q8_0) WGB_GENERIC_CASE(WGB_Q4_K)
        WGB_GENERIC_CASE(WGB_Q5_K) WGB_GENERIC_CASE(WGB_Q6_K) WGB_GENERIC_CASE(WGB_Q8_K)
    default: return fail(WGB_ERR_UNSUPPORTED, "unsupported tensor type %d", m.qtype);
    }
#undef WGB_GENERIC_CASE
    WGB_LAUNCH_CHECK("gemv_generic_kernel");
    return WGB_OK;
}

}  // namespace wgb

using namespace wgb;

static int gemv_dispatch(const QMat &m, const float *d_v, float *d_out, cudaStream_t stream, bool early_weights)
{
    WGB_REQUIRE(d_v && d_out, "null argument");
    if (gemv_fast_supported(m) && ((uintptr_t)d_v % 16) == 0) {
        GemvArgs a = {};
        a.mat[0] = m;
        a.nmat = 1;
        a.x = d_v;
        a.prologue = PRO_NONE;
        a.epilogue = EPI_STORE;
        a.out = d_out;
        // Programmatic dependent launch: the kernel streams its first weights while the previous launch in the
        // stream is still draining, and waits for it (griddepcontrol.wait) before it reads d_v or writes d_out.
        // Only for matrices the library uploaded itself: blocks in caller memory may be the output of that
        // previous launch and must not be read before it has completed.
        return launch_gemv(a, stream, early_weights);
    }
    return launch_gemv_generic(m, d_v, d_out, stream);
}

WGB_EXPORT int wgb_gemv_quant(const wgb_quant_matrix *m, const float *d_v, float *d_out, void *stream)
{
    WGB_REQUIRE(m, "null matrix");
    return gemv_dispatch(m->view, d_v, d_out, as_stream(stream), m->storage != nullptr);
}

WGB_EXPORT int wgb_gemv_quant_raw(int qtype, const void *d_blocks, size_t nrows, size_t ncols, const float *d_v,
                                  float *d_out, void *stream)
{
    const int bl = block_len(qtype);
    if (!bl) return fail(WGB_ERR_UNSUPPORTED, "unsupported tensor type %d", qtype);
    WGB_REQUIRE(d_blocks && nrows > 0 && ncols > 0 && ncols % bl == 0, "bad matrix shape %zu x %zu", nrows, ncols);
    QMat m = {};
    m.qtype = qtype;
    m.planar = 0;
    m.nrows = (uint32_t)nrows;
    m.ncols = (uint32_t)ncols;
    m.bpr = (uint32_t)(ncols / bl);
    qmat_set_pitches(m);
    m.p[0] = (const uint8_t *)d_blocks;
    return gemv_dispatch(m, d_v, d_out, as_stream(stream), false);
}
