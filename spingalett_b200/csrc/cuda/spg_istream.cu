// spg_istream.cu -- batches of a few to a few hundred rows on integer files (INT8 / INT4 / INT2): the packed weights
// stream once per 64 rows through the 8-bit integer tensor path, for nets whose every layer qualifies.
//
//   y[n][j] = act(bias[j] + w_scale * sum_k q[j][k] * x[n][k])
//
// The 128 rows of the tcgen05.mma tile (kind::i8) are weight rows, its columns are the batch: every activation is a
// 28-bit fixed-point number V = round(x / S * (2^27-1)), S the row's largest magnitude, held as four signed base-128
// digits, one column per digit.  Products and sums are exact in int32 (tensor memory) and int64 (recombination), so a
// layer's only errors are the rounding to 28 bits (2^-28 of the row's maximum) and the final rounding to fp32.
//
// Rows of wide range.  An element below 2^-12 S keeps less than 16 bits that way, which shows in outputs whose weights on the
// large elements are zero (a quarter of the INT4 weights of a normal draw are, most of the INT2 ones).  A row in which more
// than an eighth of the non-zero elements are that small is a wide one: what the rounding left of its small elements is held
// in four more digits, with the largest such remainder as scale, so they keep 28 bits of that or 56 of S, whichever is finer.
// When a layer's input has a wide row, every k-block is multiplied with both sets of digits, into both accumulators: weights
// and unpacking are shared.  Rows of a normal draw, of pixels, or of what the hidden activations make of them are not wide
// (0.1 to 5 % of small elements; the most for a leaky rectifier, whose slope puts half of a row within 1 % of the other half).
// Looking for wide rows costs about 1 us of a layer; with one input of 1e6 beside ordinary ones, which makes every row of that net's
// layers wide, the INT4 net 8192-16384-16384-8192-1000 takes 185 us instead of 127 at 8 rows, 353 instead of 177 at 64, 1034
// instead of 492 at 256 (one batch again and again).
//
// Where the operand lies.  A product of 128 x C x 32 with both operands in shared memory takes 73 cycles at C = 32 and 172 at 256, with the
// weights in tensor memory 43 and 139 (the tensor pipe itself needs 16 and 128); and a 128 x 128 block's 16 KB of operand would go through shared memory
// twice beside its 8 KB of packed bytes and its digits.  So the unpackers store to tensor memory: 256 columns hold eight blocks, beside two
// accumulators of up to 128 columns (32 rows) or one of up to 256.  Only where a layer turns out wide and needs two of more than 128 do operand tiles
// go through shared memory.  INT8 boxes are the operand as they arrive.
//
// What bounds it.  HBM needs 41 us for the 272 MB of the INT4 net 8192-16384-16384-8192-1000, whose busiest SMs have 237 blocks: 366 cycles a
// block.  Measured in the layer 16384 x 16384: 375 cycles a block at 8 rows (6.2 TB/s; 480 with the operand in shared memory), 435 at 32 rows, 560 at 64
// (746; the tensor pipe's own 512, pairs of CTAs).  The rest of the net's time lies between the blocks, 16 us a layer at 8 rows: last
// sums 4 to 10, the staging kernel and its two boundaries 8, first digit tiles 3.
//
// Measured, large INT4 net, inputs new in every call, before and since: 8 rows 125 -> 116 us (GEMV: 201), 64 rows 172 -> 162 (16-bit streaming kernel: 577),
// 256 rows 498 -> 466 (GEMM chain: 684).  Layers of more than 32 rows a group in which a CTA has many blocks in a row run on pairs of CTAs
// (cta_group::2), each with half of the digits, of which a CTA alone would draw 32 KB a block from L2.
//
// Per CTA (one per SM, 19 warps):
//   warp 0      weight boxes by TMA (128 rows x 128 packed bytes, 128-byte swizzle), ahead of the previous layer's end:
//               weights depend on nothing
//   warp 18     digit tiles by TMA ([C] x 128 k), after the staging kernel has finished
//   warps 10-17 unpack a box into operand tiles in tensor memory (INT4: a nibble moved to the top of its byte is 16q in two's complement;
//               INT2: 64q; INT8 boxes are the operand as they arrive)
//   warp 1      issues the MMAs, four K = 32 steps per 128-wide block
//   warps 2-9   tensor memory -> int64 -> scale, bias, activation -> fp32
// The work is cut evenly: the (row tile, group of rows, box) units of a layer are numbered tile after tile and CTA c takes
// units [c U / G, (c+1) U / G), so no SM idles in a last wave (128 tiles on 148 SMs would waste 14 %).  A tile that spans
// CTAs is summed in L2 with 64-bit integer reductions, whose result does not depend on their order, and finished by the CTA
// that comes last (a counter per tile), which leaves the sums at zero for the next layer.  (Pieces written side by side and
// read back one after the other cost the last CTA 16 L2 round trips at 64 rows, 11 us of every layer.)
//
// Every mbarrier wait is bounded.  Reference: forward / batch_forward layer step, Src/Spingalett.Network.c:218-247,
// Src/Spingalett.Training.c:327-343, decode of Src/Spingalett.Serialize.c:222-294.
#include "spg_common.cuh"
#include "spg_tc.cuh"
#include <cstdio>

namespace {

using namespace spgtc;

constexpr uint32_t IS_EPI_WARPS = 8, IS_CONV_WARP0 = 2 + IS_EPI_WARPS, IS_CONV_WARPS = 8, IS_DIGIT_WARP = IS_CONV_WARP0 + IS_CONV_WARPS;
constexpr uint32_t IS_THREADS = 32 * (IS_DIGIT_WARP + 1);
constexpr uint32_t TILE_ROWS = 128;
constexpr uint32_t BOX_BYTES = 128 * TILE_ROWS;        // one box of packed weights = one operand tile = 16 KB
constexpr uint32_t GROUP_ROWS = 64;                    // batch rows per pass over the weights: 256 digit columns
constexpr uint32_t IS_PAIR_ROWS = 32, IS_PAIR_BLOCKS = 16;
constexpr uint32_t IS_EARLY_BOXES = 4;
constexpr uint32_t IS_A_COLUMN = 256, IS_A_SLOTS = 4;   // operand tiles in tensor memory: slots of two blocks, 32 columns each
constexpr uint32_t MAX_K = 131072;                     // 64 * 128 * K < 2^31
constexpr uint32_t MAX_TILES = 4096;                   // counters in the scratch head
constexpr uint32_t STAGE_THREADS = 1024;
constexpr double Q27 = 134217727.0;

struct IsParams {
    uint32_t out, groups, rpg, N, C;                   // rows per group, batch rows, columns of a tile (4 * rpg)
    uint32_t rows;                                     // groups * rpg: rows of scales, a quarter of the rows of one set of digits
    uint32_t kbr, boxes;                               // 128-wide k-blocks per box, boxes per row tile
    uint32_t RS, AS, BS, bars;                         // ring slots: boxes, operand in shared memory (G blocks each), digits (GB blocks each); barriers of operand slots
    uint32_t G, GB;
    uint32_t units;                                    // tiles * boxes (4096 * 1024 at most: times the number of CTAs still 32 bits)
    uint32_t direct; int prec, act;
    double scale; const float *bias; const double *row_scale;
    const uint8_t *wide;
    float *y; uint32_t ldy;
    unsigned long long *sums, *sums2; uint32_t *counters; int32_t *status;      // sums2: of the second set of digits
    uint32_t idesc;
};

// D[tmem] (+)= A[smem desc] * B[smem desc], signed 8-bit operands, int32 accumulate, one CTA
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
// ... over the two CTAs of a pair: 128 rows of A each, half of B's rows each
__device__ __forceinline__ void umma_i8_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// ... with A in tensor memory: 32 rows' bytes of K = 32 are eight columns
__device__ __forceinline__ void umma_i8_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void umma_i8_tmem_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// 32 columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void mbar_arrive_by(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// int32 accumulator, A and B signed 8-bit, both K-major, m x n
inline uint32_t idesc_i8(uint32_t m, uint32_t n) { return (2u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24); }

// first unit of CTA c
__host__ __device__ inline uint32_t unit_start(uint32_t units, uint32_t grid, uint32_t c) { return units * c / grid; }

// ---- staging: fp32 rows -> digit operand -------------------------------------------------------------------------------

// byte of element e (0..15) inside a group of 16 consecutive k, in the order in which the unpacking delivers the weights
template <int PREC> __host__ __device__ constexpr uint32_t is_position(uint32_t e)
{
    return PREC == SPG_P_I4 ? (e & 8u) + (e & 1u) * 4u + ((e & 7u) >> 1)
         : PREC == SPG_P_I2 ? (e & 3u) * 4u + (e >> 2) : e;
}

__device__ __forceinline__ void is_load16(float (&f)[16], const float *row, uint32_t k, uint32_t in, uint32_t vec)
{
#pragma unroll
    for (uint32_t i = 0; i < 16; i += 4) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k < in) {
            if (vec) v = *reinterpret_cast<const float4 *>(row + k + i);
            else v = make_float4(row[k + i], row[k + i + 1], row[k + i + 2], row[k + i + 3]);
        }
        f[i] = v.x; f[i + 1] = v.y; f[i + 2] = v.z; f[i + 3] = v.w;
    }
}
// largest magnitude as an integer: a NaN counts as more than an infinity
__device__ __forceinline__ uint32_t is_magnitude(const float (&f)[16])
{
    uint32_t m = 0;
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) m = max(m, __float_as_uint(f[i]) & 0x7FFFFFFFu);
    return m;
}

// The element as a fixed-point number: adding 1.5 * 2^52 leaves the product, rounded to an integer once, in the low word
__device__ __forceinline__ int is_fixed(double v, double inv) { return __double2loint(fma(v, inv, 6755399441055744.0)); }
// Elements that keep less than 16 bits: not zero and below 2^-12 of the row's maximum
constexpr int COARSE = 1 << 15;

// The four digits of 16 fixed-point numbers, at `dst` in each of four operand rows
template <int PREC> __device__ __forceinline__ void is_store16(const int (&fixed)[16], uint8_t *dst, uint32_t ld)
{
    uint32_t w[4][4] = {};
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
        int v = fixed[i];
        const uint32_t pos = is_position<PREC>(i);
#pragma unroll
        for (uint32_t d = 0; d < 4; d++) {
            const int dig = d == 3 ? v : ((v + 64) & 127) - 64;
            v = (v - dig) >> 7;
            w[d][pos >> 2] |= ((uint32_t)dig & 0xFFu) << (8 * (pos & 3u));
        }
    }
#pragma unroll
    for (uint32_t d = 0; d < 4; d++) *reinterpret_cast<uint4 *>(dst + (uint64_t)d * ld) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
}

// What the first set's rounding left of a coarse element, else 0.  Exact but for the last of 53 bits: `step` is the very
// number that V is multiplied with later.
__device__ __forceinline__ double is_left(float x, double inv, double step)
{
    const int v = is_fixed((double)x, inv);
    return x != 0.0f && abs(v) < COARSE ? fma((double)-v, step, (double)x) : 0.0;
}

// The second set of digits of a wide row: what is left of its coarse elements, with the largest of it as scale.  Returns that
// scale.  Short loops on purpose: code that ordinary rows never run costs them its way into the instruction cache (unrolled
// like the first set's it took 1 us of every layer).
template <int PREC>
__device__ __noinline__ double is_stage_second(const float *row, uint32_t in, uint32_t ld, double inv, double step, uint8_t *dst)
{
    __shared__ double s_left[32];
    const uint32_t tid = threadIdx.x;
    double left = 0.0;
#pragma unroll 1
    for (uint32_t k = tid; k < in; k += STAGE_THREADS) left = fmax(left, fabs(is_left(row[k], inv, step)));
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) left = fmax(left, __shfl_xor_sync(0xffffffffu, left, o));
    if ((tid & 31u) == 0) s_left[tid >> 5] = left;
    __syncthreads();
#pragma unroll 1
    for (uint32_t i = 0; i < 32; i++) left = fmax(left, s_left[i]);
    const double inv2 = left > 0.0 ? Q27 / left : 0.0;
#pragma unroll 1
    for (uint32_t k = tid; k < ld; k += STAGE_THREADS) {
        int v = k < in ? is_fixed(is_left(row[k], inv, step), inv2) : 0;
        uint8_t *out = dst + (k & ~15u) + is_position<PREC>(k & 15u);
#pragma unroll 1
        for (uint32_t d = 0; d < 4; d++, out += ld) {
            const int dig = d == 3 ? v : ((v + 64) & 127) - 64;
            v = (v - dig) >> 7;
            *out = (uint8_t)dig;
        }
    }
    return left * (1.0 / Q27);
}

// One CTA per batch row (rows past N and k past `in` become zero digits): the row's maximum, then four digit rows of `ld`
// bytes, 16 elements per thread and step.  64 rows of 16384: 4 MB in, 4 MB out, a few microseconds, of which the next
// layer's first weight boxes hide some.  A row with an infinity or a NaN gets a NaN scale and zero digits.
// row_scale: a scale per row, then a second one per row, which is zero unless the row is a wide one (else its second set of
// digits, 4 * gridDim.x operand rows further on, is whatever it was: finite, and multiplied with zero).
// wide: a byte per row, not zero if the row is a wide one.
template <int PREC>
__global__ void __launch_bounds__(STAGE_THREADS)
spg_is_stage_kernel(const float *__restrict__ x, uint32_t ldx, uint32_t N, uint32_t in, uint32_t ld, uint32_t vec,
                    uint8_t *__restrict__ dst, double *__restrict__ row_scale, uint8_t *__restrict__ wide)
{
    __shared__ uint32_t s_max[32];
    __shared__ int s_coarse[32];
    spg_grid_trigger();
    spg_grid_wait();
    const uint32_t n = blockIdx.x, tid = threadIdx.x;
    const bool live = n < N;
    const float *row = x + (uint64_t)(live ? n : 0) * ldx;
    float f[16];                                       // the thread's first 16 elements are read once; `in` is a multiple of 16
    is_load16(f, row, 16 * tid, live ? in : 0, vec);
    uint32_t m = is_magnitude(f);
    for (uint32_t k = 16 * (tid + STAGE_THREADS); live && k < in; k += 16 * STAGE_THREADS) {
        float g[16];
        is_load16(g, row, k, in, vec);
        m = max(m, is_magnitude(g));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((tid & 31u) == 0) s_max[tid >> 5] = m;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, s_max[tid & 31u]);
    const bool finite = m < 0x7F800000u;
    const double s = (double)__uint_as_float(m);
    const double inv = finite && m ? Q27 / s : 0.0;
    const double step = finite ? s * (1.0 / Q27) : (double)__uint_as_float(0x7FC00000u);
    const bool zero = !live || !finite;
    int coarse = 0;                                    // 8 per coarse element, -1 per element that is not zero
    for (uint32_t k = 16 * tid; k < ld; k += 16 * STAGE_THREADS) {
        if (k >= 16 * STAGE_THREADS) is_load16(f, row, k, live ? in : 0, vec);
        int fixed[16] = {};
        if (!zero) {
#pragma unroll
            for (uint32_t i = 0; i < 16; i++) {
                fixed[i] = is_fixed((double)f[i], inv);
                if (f[i] != 0.0f) coarse += abs(fixed[i]) < COARSE ? 7 : -1;
            }
        }
        is_store16<PREC>(fixed, dst + (uint64_t)(4 * n) * ld + k, ld);
    }
    coarse = __reduce_add_sync(0xffffffffu, coarse);
    double step2 = 0.0;
    if (__syncthreads_or(coarse > 0)) {                // in no warp's share: not in the row either
        if ((tid & 31u) == 0) s_coarse[tid >> 5] = coarse;
        __syncthreads();
        coarse = __reduce_add_sync(0xffffffffu, s_coarse[tid & 31u]);
        if (coarse > 0) step2 = is_stage_second<PREC>(row, in, ld, inv, step, dst + (uint64_t)4 * (gridDim.x + n) * ld);
    }
    if (tid == 0) { row_scale[n] = step; row_scale[gridDim.x + n] = step2; wide[n] = step2 != 0.0; }
}

// ---- the layer ---------------------------------------------------------------------------------------------------------

// Operand tiles go to tensor memory, beside one accumulator of up to 256 columns or two of up to 128, unless both sets of digits need more
// columns than that (or the boxes are the operand).
__device__ __forceinline__ bool is_in_tmem(const IsParams &p, bool wide) { return !p.direct && !(wide && p.C > 128); }
__device__ __forceinline__ bool is_one_accumulator(const IsParams &p, bool wide) { return wide || (!p.direct && p.C > 128); }

__device__ __forceinline__ void is_epi_sync() { asm volatile("bar.sync 2, %0;" ::"n"(32 * IS_EPI_WARPS) : "memory"); }

// `rest`: bias, and the second set's share
template <int ACT>
__device__ __forceinline__ void is_finish(const IsParams &p, uint32_t n, uint32_t row, double rest, double scale, long long sum)
{
    const float v = spg_activate((float)((double)sum * scale + rest), ACT);
    if (row < p.out && n < p.N) p.y[(uint64_t)n * p.ldy + row] = v;
}

// Segments of a CTA: the runs of its units that lie in one tile.
struct IsSegment { uint32_t u, end, tile, k0, k1; };
__device__ __forceinline__ bool is_next_segment(const IsParams &p, IsSegment &s)
{
    if (s.u >= s.end) return false;
    s.tile = s.u / p.boxes;
    s.k0 = s.u - s.tile * p.boxes;
    const uint32_t left = s.end - s.u;
    s.k1 = left < p.boxes - s.k0 ? s.k0 + left : p.boxes;
    s.u += s.k1 - s.k0;
    return true;
}

// The sum of four neighbouring columns: the digits of one batch row
__device__ __forceinline__ long long is_recombine(const uint32_t *r)
{
    return (((long long)(int)r[3] * 128 + (int)r[2]) * 128 + (int)r[1]) * 128 + (int)r[0];
}

// Whether any row of the layer's input is a wide one (a whole warp, after the staging kernel has finished)
__device__ __forceinline__ bool is_any_wide(const IsParams &p, uint32_t lane)
{
    uint32_t wide = 0;
    for (uint32_t n = 4 * lane; n < p.rows; n += 128) wide |= __ldcg(reinterpret_cast<const uint32_t *>(p.wide + n));
    return __any_sync(0xffffffffu, wide != 0);
}

// Epilogue role (warps 2..9): thread = one weight row (tensor-memory lane) of the tile; of two warps on the same lanes each
// takes every other four batch rows.  `wide`: with the second set of digits, in loops of its own (its branches and registers in
// the others took 1 to 2 us a layer).  Turning a sum into an output is a chain of some 450 cycles (two conversions of 100 and 75
// among them) and a scheduler has two of these warps: only values side by side hide it, so the activation is chosen outside and
// nothing in the chain branches (with the choice inside, the last sums of a tile took 17500 cycles at 64 rows).  `dirty`: a launch before this one failed and nobody has read its status yet, so the sums and
// counters cannot be relied on.
template <int ACT, bool PAIR>
__device__ __forceinline__ void is_epilogue(const IsParams &p, bool wide, bool dirty, IsSegment seg, uint32_t tmem_base, uint32_t tfull0, uint32_t tempty0,
                                            volatile int *abort_flag, int *s_last, double *s_scale, uint32_t warp, uint32_t lane)
{
    const uint32_t half = (warp - 2u) >> 2, et = (warp & 3u) * 32u + lane;
    const uint32_t cta = PAIR ? blockIdx.x & 1u : 0u, teams = PAIR ? gridDim.x >> 1 : gridDim.x;      // teams: pairs, or CTAs alone
    const bool one = is_one_accumulator(p, wide);      // (a wide layer's second set takes the second accumulator)
    uint32_t count = 0;
    for (; is_next_segment(p, seg); count++) {
        const uint32_t acc = one ? 0 : count & 1u, phase = (one ? count : count >> 1) & 1u, mt = seg.tile / p.groups, n0 = (seg.tile % p.groups) * p.rpg;
        const bool whole = seg.k1 - seg.k0 == p.boxes;
        const uint32_t row = (PAIR ? 2 * mt + cta : mt) * TILE_ROWS + et;
        const float bias = row < p.out ? p.bias[row] : 0.0f;
        // the group's scales, once per segment into shared memory: a global load per value would be a chain of L2 latencies
        if (half == 0 && et < p.rpg) {
            s_scale[et] = __ldcg(p.row_scale + n0 + et) * p.scale;
            if (wide) s_scale[GROUP_ROWS + et] = __ldcg(p.row_scale + p.rows + n0 + et) * p.scale;
        }
        // the sums of a tile in pieces belong to the CTA that holds its first unit: at most one tile that goes on past the end
        // of a CTA's range starts in it
        uint64_t slot = et;
        if (!whole) {
            const uint32_t t0 = seg.tile * p.boxes;
            uint32_t c = t0 * teams / p.units;
            while (c > 0 && unit_start(p.units, teams, c) > t0) c--;
            while (unit_start(p.units, teams, c + 1) <= t0) c++;
            slot += (uint64_t)(PAIR ? 2 * c + cta : c) * p.rpg * TILE_ROWS;
        }
        unsigned long long *sums = p.sums + slot, *sums2 = p.sums2 + slot;
        is_epi_sync();
        const bool ok = mbar_wait(tfull0 + 8 * acc, phase, abort_flag, p.status, 9) && !dirty;
        tc_fence_after();
        const uint32_t taddr = tmem_base + acc * p.C + ((et & ~31u) << 16);
        if (!wide) {
            for (uint32_t c0 = 16 * half; c0 < p.C; c0 += 32) {
                uint32_t r[16];
                tmem_ld16(taddr + c0, r);
                tmem_ld_wait();
                if (!ok) continue;
                if (whole) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; i++)
                        is_finish<ACT>(p, n0 + (c0 >> 2) + i, row, (double)bias, s_scale[(c0 >> 2) + i], is_recombine(r + 4 * i));
                } else {
#pragma unroll
                    for (uint32_t i = 0; i < 4; i++)
                        atomicAdd(sums + (uint64_t)((c0 >> 2) + i) * TILE_ROWS, (unsigned long long)is_recombine(r + 4 * i));
                }
            }
        } else {
#pragma unroll 1
            for (uint32_t rr = half; rr < p.rpg; rr += 2) {
                uint32_t r[4], q[4];
                tmem_ld4(taddr + 4 * rr, r);
                tmem_ld4(taddr + p.C + 4 * rr, q);
                tmem_ld_wait();
                if (!ok) continue;
                const long long v = is_recombine(r), v2 = is_recombine(q);
                if (whole) is_finish<ACT>(p, n0 + rr, row, (double)bias + (double)v2 * s_scale[GROUP_ROWS + rr], s_scale[rr], v);
                else {
                    atomicAdd(sums + (uint64_t)rr * TILE_ROWS, (unsigned long long)v);
                    atomicAdd(sums2 + (uint64_t)rr * TILE_ROWS, (unsigned long long)v2);
                }
            }
        }
        tc_fence_before();
        if (PAIR) {                                     // the accumulator may be overwritten
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(tempty0 + 8 * acc);
        } else mbar_arrive(tempty0 + 8 * acc);
        if (!whole) __threadfence();
        is_epi_sync();                                  // (also: the scales of the next segment may replace these)
        const bool failed = !ok || *abort_flag;
        if (failed) {
            // a wait gave up, here or before: nothing in the output that could pass for a result
#pragma unroll 1
            for (uint32_t rr = half; rr < p.rpg; rr += 2)
                if (row < p.out && n0 + rr < p.N) p.y[(uint64_t)(n0 + rr) * p.ldy + row] = __uint_as_float(0x7FC00000u);
        }
        if (whole) continue;
        if (warp == 2 && lane == 0) {
            const uint32_t part = seg.k1 - seg.k0;
            *s_last = !failed && atomicAdd(&p.counters[PAIR ? 2 * seg.tile + cta : seg.tile], part) + part == p.boxes;
        }
        is_epi_sync();
        if (*s_last) {
            __threadfence();
            for (uint32_t r0 = 4 * half; !wide && r0 < p.rpg; r0 += 32) {      // four groups of four rows in flight
                long long v[16];
#pragma unroll
                for (uint32_t i = 0; i < 16; i++) {
                    const uint32_t rr = r0 + (i >> 2) * 8 + (i & 3u);
                    v[i] = rr < p.rpg ? (long long)__ldcg(sums + (uint64_t)rr * TILE_ROWS) : 0;
                }
#pragma unroll
                for (uint32_t i = 0; i < 16; i++) {
                    const uint32_t rr = r0 + (i >> 2) * 8 + (i & 3u);
                    const bool live = rr < p.rpg;
                    if (live) __stcg(sums + (uint64_t)rr * TILE_ROWS, 0ull);
                    is_finish<ACT>(p, live ? n0 + rr : p.N, row, (double)bias, s_scale[live ? rr : 0], v[i]);
                }
            }
#pragma unroll 1
            for (uint32_t rr = half; wide && rr < p.rpg; rr += 2) {
                const long long v = (long long)__ldcg(sums + (uint64_t)rr * TILE_ROWS), v2 = (long long)__ldcg(sums2 + (uint64_t)rr * TILE_ROWS);
                __stcg(sums + (uint64_t)rr * TILE_ROWS, 0ull);
                __stcg(sums2 + (uint64_t)rr * TILE_ROWS, 0ull);
                is_finish<ACT>(p, n0 + rr, row, (double)bias + (double)v2 * s_scale[GROUP_ROWS + rr], s_scale[rr], v);
            }
            if (warp == 2 && lane == 0) p.counters[PAIR ? 2 * seg.tile + cta : seg.tile] = 0;
        }
        is_epi_sync();
    }
}

// Digit slots of a CTA that go out before it is known whether the layer has a wide row: the ring at most.  They are the first
// set's of consecutive blocks, which is the order of a layer without wide rows; in a wide one, where the sets alternate, they
// are thrown away.
__device__ __forceinline__ uint32_t is_early_slots(const IsParams &p, const IsSegment &seg)
{
    const uint32_t slots = (seg.end - seg.u) * p.kbr / p.GB;
    return slots < p.BS ? slots : p.BS;
}

// MMA role (warp 1): SETS sets of digits per 128-wide block of weights.  A wait costs the warp some 70 cycles even when there is nothing to wait
// for, a commit as much.  So operand tiles change hands G blocks at a time and digit tiles GB (a divisor of G), and all three are numbers
// known to the compiler (a counted loop over the sets took 3 us of the 65 that 256 rows of a 4096-4096-1024 net take).
// TMEM: the operand tiles lie in tensor memory.
struct IsBars { uint32_t rfull0, rempty0, afull0, aempty0, bfull0, bempty0, tfull0, tempty0; };
template <uint32_t SETS, uint32_t G, uint32_t GB, bool PAIR, bool TMEM>
__device__ __forceinline__ void is_mma(const IsParams &p, IsSegment seg, const IsBars &bar, uint64_t a_desc0, uint64_t b_desc0, uint32_t tmem_base,
                                       uint32_t abort_addr, volatile int *abort_flag)
{
    uint32_t as = 0, aph = 0, bs = 0, bph = 0, count = 0;      // G = 1: the boxes are the operand
    const uint32_t b_step = p.C * 128u >> (PAIR ? 5 : 4), slots = TMEM ? IS_A_SLOTS : G == 1 ? p.RS : p.AS;
    const bool one = SETS == 2 || (TMEM && p.C > 128);
    const uint32_t full0 = G == 1 ? bar.rfull0 : bar.afull0, empty0 = G == 1 ? bar.rempty0 : bar.aempty0;
    if (SETS == 2) {
        const uint32_t early = is_early_slots(p, seg);
        for (uint32_t i = 0; i < early; i++) {
            mbar_wait_uniform(bar.bfull0 + 8 * bs, bph, abort_addr, p.status, 10);
            if (*abort_flag) return;
            if (elect_one()) {
                mbar_arrive(bar.bempty0 + 8 * bs);
                if (PAIR) mbar_arrive_cluster(mapa(bar.bempty0 + 8 * bs, 1));
            }
            __syncwarp();
            if (++bs == p.BS) { bs = 0; bph ^= 1u; }
        }
    }
    for (; is_next_segment(p, seg); count++) {
        const uint32_t acc = one ? 0 : count & 1u, phase = (one ? count : count >> 1) & 1u;
        mbar_wait_uniform(bar.tempty0 + 8 * acc, phase ^ 1u, abort_addr, p.status, 3);
        if (*abort_flag) return;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * p.C;
        uint32_t accum = 0;
        const uint32_t turns = (seg.k1 - seg.k0) * p.kbr / G;  // (kbr is a multiple of G)
        for (uint32_t turn = 0; turn < turns; turn++) {
            mbar_wait_uniform(full0 + 8 * as, aph, abort_addr, p.status, G == 1 ? 4 : 5);
            const uint64_t da = a_desc0 + (uint64_t)(as * G * (BOX_BYTES >> 4));
            const uint32_t ta = tmem_base + IS_A_COLUMN + as * G * 32;
#pragma unroll
            for (uint32_t j = 0; j < G; j += GB) {
#pragma unroll
                for (uint32_t set = 0; set < SETS; set++) {
                    mbar_wait_uniform(bar.bfull0 + 8 * bs, bph, abort_addr, p.status, 6);
                    if (*abort_flag) return;
                    tc_fence_after();
                    const uint64_t db = b_desc0 + (uint64_t)(bs * GB * b_step);
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t i = 0; i < GB; i++)
#pragma unroll
                            for (uint32_t k = 0; k < 4; k++)
                                if (TMEM) PAIR ? umma_i8_tmem_pair(d_tmem + set * p.C, ta + (j + i) * 32 + 8 * k, db + i * b_step + 2 * k, p.idesc, j + i + k ? 1u : accum)
                                               : umma_i8_tmem(d_tmem + set * p.C, ta + (j + i) * 32 + 8 * k, db + i * b_step + 2 * k, p.idesc, j + i + k ? 1u : accum);
                                else PAIR ? umma_i8_pair(d_tmem + set * p.C, da + (j + i) * (BOX_BYTES >> 4) + 2 * k, db + i * b_step + 2 * k, p.idesc, j + i + k ? 1u : accum)
                                     : umma_i8(d_tmem + set * p.C, da + (j + i) * (BOX_BYTES >> 4) + 2 * k, db + i * b_step + 2 * k, p.idesc, j + i + k ? 1u : accum);
                        PAIR ? umma_commit_pair(bar.bempty0 + 8 * bs) : umma_commit(bar.bempty0 + 8 * bs);
                        if (j + GB == G && set + 1 == SETS) PAIR ? umma_commit_pair(empty0 + 8 * as) : umma_commit(empty0 + 8 * as);
                    }
                    __syncwarp();
                    if (++bs == p.BS) { bs = 0; bph ^= 1u; }
                }
            }
            accum = 1;
            if (++as == slots) { as = 0; aph ^= 1u; }
        }
        if (elect_one()) PAIR ? umma_commit_pair(bar.tfull0 + 8 * acc) : umma_commit(bar.tfull0 + 8 * acc);
        __syncwarp();
    }
}

// PAIR: clusters of two.  A pair's tiles are 256 weight rows high; each CTA has its own 128 (boxes, unpacking, accumulator, epilogue as alone) and
// half of the digit columns, and the first one's MMA warp issues for both.  The barriers it waits on live in its shared memory.
template <bool PAIR>
__global__ void __launch_bounds__(IS_THREADS, 1)
spg_istream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const IsParams p)
{
    extern __shared__ uint8_t is_smem_raw[];
    const uint32_t raw = smem_u32(is_smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *smem = is_smem_raw + (base - raw);
    // layout: box ring | operand ring (absent for INT8) | digit ring | barriers | flags | scales of a group, both sets
    const uint32_t b_bytes = p.C * (PAIR ? 64u : 128u);
    const uint32_t a_off = p.RS * BOX_BYTES;
    const uint32_t b_off = a_off + (p.direct ? 0u : p.AS * p.G * BOX_BYTES);
    const uint32_t bar_off = b_off + p.BS * p.GB * b_bytes;
    const uint32_t rfull0 = base + bar_off, rempty0 = rfull0 + 8 * p.RS;
    const uint32_t afull0 = rempty0 + 8 * p.RS, aempty0 = afull0 + 8 * p.bars;
    const uint32_t bfull0 = aempty0 + 8 * p.bars, bempty0 = bfull0 + 8 * p.BS;
    const uint32_t tfull0 = bempty0 + 8 * p.BS, tempty0 = tfull0 + 16;
    const uint32_t flag_off = bar_off + 16 * (p.RS + p.bars + p.BS) + 32;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + flag_off);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *s_last = const_cast<int *>(abort_flag) + 1;
    double *s_scale = reinterpret_cast<double *>(smem + flag_off + 16);

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t cta = PAIR ? cluster_rank() : 0u, team = PAIR ? blockIdx.x >> 1 : blockIdx.x, teams = PAIR ? gridDim.x >> 1 : gridDim.x;
    uint32_t tmem_cols = 32;
    while (tmem_cols < (p.direct ? 2 * p.C : 512u)) tmem_cols *= 2;      // two accumulators, 512 columns at most

    if (tid == 0) {
        for (uint32_t s = 0; s < p.RS; s++) { mbar_init(rfull0 + 8 * s, 1); mbar_init(rempty0 + 8 * s, p.direct ? 1 : IS_CONV_WARPS); }
        for (uint32_t s = 0; s < p.bars; s++) { mbar_init(afull0 + 8 * s, (PAIR ? 2 : 1) * IS_CONV_WARPS / 2); mbar_init(aempty0 + 8 * s, 1); }      // (half of the unpackers a slot)
        for (uint32_t s = 0; s < p.BS; s++) { mbar_init(bfull0 + 8 * s, 1); mbar_init(bempty0 + 8 * s, 1); }
        for (uint32_t a = 0; a < 2; a++) { mbar_init(tfull0 + 8 * a, 1); mbar_init(tempty0 + 8 * a, PAIR ? 2 * IS_EPI_WARPS : 32 * IS_EPI_WARPS); }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_map(&map_w);
        prefetch_map(&map_x);
    }
    if (warp == 1) PAIR ? tmem_alloc_pair(smem_u32(tmem_slot), tmem_cols) : tmem_alloc(smem_u32(tmem_slot), tmem_cols);
    tc_fence_before();
    if (PAIR) cluster_sync();                            // both CTAs' barriers exist before anyone arrives on them
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t lead_rfull0 = PAIR ? mapa(rfull0, 0) : rfull0, lead_bfull0 = PAIR ? mapa(bfull0, 0) : bfull0;
    const uint32_t lead_tempty0 = PAIR ? mapa(tempty0, 0) : tempty0;
    spg_grid_trigger();

    const uint32_t abort_addr = smem_u32(const_cast<int *>(abort_flag));
    IsSegment seg;
    seg.u = unit_start(p.units, teams, team);
    seg.end = unit_start(p.units, teams, team + 1);

    if (warp == 0) {
        // ------------------------------ weight boxes ------------------------------
        // The first boxes go out before the previous kernel of the stream has ended; every role waits for that end before its first bounded wait,
        // which would otherwise count somebody else's running time.  Not a whole ring of boxes: 24 MB of weights from HBM are in the way of the few
        // loads that the staging kernel and the first digit tiles hang on (large INT4 net at 8 and 64 rows, boxes of ten that go early: none 118.8 / 158.5
        // us, two 115.9 / 158.3, four 113.9 / 157.3, ten 114.8 / 160.1; asking L2 for up to 48 more each 121 / 169).
        uint32_t rs = 0, rph = 0, sent = 0;
        while (is_next_segment(p, seg)) {
            const int r0 = (int)((PAIR ? 2 * (seg.tile / p.groups) + cta : seg.tile / p.groups) * TILE_ROWS);
            for (uint32_t b = seg.k0; b < seg.k1; b++) {
                if (sent++ == IS_EARLY_BOXES) spg_grid_wait();
                mbar_wait_uniform(rempty0 + 8 * rs, rph ^ 1u, abort_addr, p.status, 1);
                if (*abort_flag) goto is_role_done;
                if (elect_one()) {
                    if (PAIR && p.direct) {              // the boxes are the operand: the issuer waits for both CTAs'
                        if (cta == 0) mbar_expect_tx(rfull0 + 8 * rs, 2 * BOX_BYTES);
                        tma_load_2d_pair(base + rs * BOX_BYTES, &map_w, lead_rfull0 + 8 * rs, (int)(b * 128u), r0);
                    } else {
                        mbar_expect_tx(rfull0 + 8 * rs, BOX_BYTES);
                        tma_load_2d(base + rs * BOX_BYTES, &map_w, rfull0 + 8 * rs, (int)(b * 128u), r0);
                    }
                }
                __syncwarp();
                if (++rs == p.RS) { rs = 0; rph ^= 1u; }
            }
        }
    } else if (warp == IS_DIGIT_WARP) {
        // ------------------------------ digit tiles -------------------------------
        uint32_t bs = 0, bph = 0, early = is_early_slots(p, seg);
        auto load = [&](uint32_t kb, uint32_t row) {
            mbar_wait_uniform(bempty0 + 8 * bs, bph ^ 1u, abort_addr, p.status, 2);
            if (*abort_flag) return;
            if (elect_one()) {
                if (cta == 0) mbar_expect_tx(bfull0 + 8 * bs, (PAIR ? 2 : 1) * p.GB * b_bytes);
                for (uint32_t i = 0; i < p.GB; i++) {
                    const uint32_t dst = base + b_off + (bs * p.GB + i) * b_bytes;
                    if (PAIR) tma_load_2d_pair(dst, &map_x, lead_bfull0 + 8 * bs, (int)((kb + i) * 128u), (int)(row + cta * (p.C / 2)));
                    else tma_load_2d(dst, &map_x, bfull0 + 8 * bs, (int)((kb + i) * 128u), (int)row);
                }
            }
            __syncwarp();
            if (++bs == p.BS) { bs = 0; bph ^= 1u; }
        };
        spg_grid_wait();
        IsSegment ahead = seg;
        for (uint32_t left = early; left && is_next_segment(p, ahead);)
            for (uint32_t kb = ahead.k0 * p.kbr; left && kb < ahead.k1 * p.kbr; kb += p.GB, left--) load(kb, ahead.tile % p.groups * p.C);
        const uint32_t sets = is_any_wide(p, lane) ? 2 : 1;
        if (sets == 2) early = 0;
        while (is_next_segment(p, seg)) {
            const uint32_t c0 = seg.tile % p.groups * p.C;
            for (uint32_t kb = seg.k0 * p.kbr; kb < seg.k1 * p.kbr; kb += p.GB) {
                if (early) { early--; continue; }                              // has gone out
                for (uint32_t set = 0; set < sets; set++) {
                    load(kb, c0 + set * 4 * p.rows);
                    if (*abort_flag) goto is_role_done;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------
        const IsBars bar = { rfull0, rempty0, afull0, aempty0, bfull0, bempty0, tfull0, tempty0 };
        const uint64_t a_desc0 = smem_desc_sw128(p.direct ? base : base + a_off), b_desc0 = smem_desc_sw128(base + b_off);
        spg_grid_wait();
        if (cta) goto is_role_done;                      // the first CTA issues for both
#define IS_MMA(SETSV, GV, GBV, TMEMV) is_mma<SETSV, GV, GBV, PAIR, TMEMV>(p, seg, bar, a_desc0, b_desc0, tmem_base, abort_addr, abort_flag)
        const bool wide = is_any_wide(p, lane);
        if (p.direct) { if (wide) IS_MMA(2, 1, 1, false); else IS_MMA(1, 1, 1, false); }
        else if (!is_in_tmem(p, wide)) { if (p.GB == 1) IS_MMA(2, 2, 1, false); else IS_MMA(2, 2, 2, false); }
        else if (p.GB == 1) { if (wide) IS_MMA(2, 2, 1, true); else IS_MMA(1, 2, 1, true); }
        else { if (wide) IS_MMA(2, 2, 2, true); else IS_MMA(1, 2, 2, true); }
#undef IS_MMA
    } else if (warp >= IS_CONV_WARP0) {
        // ------------------------------ unpackers ---------------------------------
        // A group of warps for each of the AS * G operand tiles that the ring holds; group g makes the tiles of the k-blocks whose
        // running number is g mod AS * G, always in place g, so that many tiles are in the making at once and the latency of one
        // (load, unpack, store, proxy fence, arrive: 600 cycles) hides behind the others.  Lanes 0-7 of a quarter warp take eight different rows of a swizzle atom: no bank
        // conflict on either side.  (Sixteen warps instead of eight: 2 to 5 % slower at every batch size.)
        if (!p.direct) spg_grid_wait();
        const bool in_tmem = !p.direct && is_in_tmem(p, p.C > 128 && is_any_wide(p, lane));
        if (in_tmem) {
            // Four warps make the two blocks of a slot, a lane a weight row; the other four make the next slot's.  A row's packed bytes are whole in
            // the box, so a lane reads them, unpacks them and stores 32 columns a block.
            const uint32_t set = (warp - IS_CONV_WARP0) >> 2, quadrant = warp & 3u, row = quadrant * 32 + lane, r7 = row & 7u;
            const bool nibbles = p.prec == SPG_P_I4;
            const uint32_t turns = nibbles ? 1 : 2;      // slots of a box
            const uint32_t tmem_a = tmem_base + IS_A_COLUMN + ((quadrant * 32) << 16);
            uint32_t rs = 0, rph = 0, as = 0, aph = 0, turn = 0;
            while (is_next_segment(p, seg)) {
                for (uint32_t b = seg.k0; b < seg.k1; b++) {
                    const uint8_t *box = smem + rs * BOX_BYTES + row * 128u;
                    bool mine = false;
                    for (uint32_t t = 0; t < turns; t++, turn++) {
                        if ((turn & 1u) == set) {
                            bool ok = mine || mbar_wait(rfull0 + 8 * rs, rph, abort_flag, p.status, 7);
                            mine = true;
                            ok = ok && mbar_wait(aempty0 + 8 * as, aph ^ 1u, abort_flag, p.status, 8);
                            __syncwarp();
                            tc_fence_after();
                            if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
                                for (uint32_t j = 0; j < 2; j++) {
                                    uint32_t r[32];
                                    if (nibbles) {
#pragma unroll
                                        for (uint32_t pc = 0; pc < 4; pc++) {
                                            const uint4 w = *reinterpret_cast<const uint4 *>(box + (((4 * j + pc) ^ r7) << 4));
                                            const uint32_t m = 0xF0F0F0F0u, ws[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
                                            for (uint32_t i = 0; i < 4; i++) { r[8 * pc + 2 * i] = (ws[i] << 4) & m; r[8 * pc + 2 * i + 1] = ws[i] & m; }
                                        }
                                    } else {
#pragma unroll
                                        for (uint32_t pc = 0; pc < 2; pc++) {
                                            const uint4 w = *reinterpret_cast<const uint4 *>(box + (((4 * t + 2 * j + pc) ^ r7) << 4));
                                            const uint32_t m = 0xC0C0C0C0u, ws[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
                                            for (uint32_t i = 0; i < 4; i++) {
                                                r[16 * pc + 4 * i] = (ws[i] << 6) & m; r[16 * pc + 4 * i + 1] = (ws[i] << 4) & m;
                                                r[16 * pc + 4 * i + 2] = (ws[i] << 2) & m; r[16 * pc + 4 * i + 3] = ws[i] & m;
                                            }
                                        }
                                    }
                                    tmem_st32(tmem_a + as * 64 + j * 32, r);
                                }
                                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                            }
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) PAIR ? mbar_arrive_cluster(mapa(afull0 + 8 * as, 0)) : mbar_arrive(afull0 + 8 * as);
                        }
                        if (++as == IS_A_SLOTS) { as = 0; aph ^= 1u; }
                    }
                    if (mine && lane == 0) mbar_arrive_by(rempty0 + 8 * rs, nibbles ? 2 : 1);      // (eight arrivals a box)
                    if (++rs == p.RS) { rs = 0; rph ^= 1u; }
                }
            }
        } else if (!p.direct) {
            const uint32_t tiles = p.AS * p.G, wpg = IS_CONV_WARPS / tiles, TG = 32u * wpg;
            const uint32_t cw = warp - IS_CONV_WARP0, grp = cw / wpg, ctg = (cw % wpg) * 32u + lane;
            const uint32_t afull = PAIR ? mapa(afull0 + 8 * (grp / p.G), 0) : afull0 + 8 * (grp / p.G), aempty = aempty0 + 8 * (grp / p.G);
            uint32_t rs = 0, rph = 0, as = 0, aph = 0;
            uint8_t *atile = smem + a_off + grp * BOX_BYTES;
            while (is_next_segment(p, seg)) {
                for (uint32_t b = seg.k0; b < seg.k1; b++) {
                    const bool okr = mbar_wait(rfull0 + 8 * rs, rph, abort_flag, p.status, 7);
                    const uint8_t *box = smem + rs * BOX_BYTES;
                    for (uint32_t j = 0; j < p.kbr; j++) {
                        if (as == grp) {
                            const bool ok = okr && mbar_wait(aempty, aph ^ 1u, abort_flag, p.status, 8);
                            if (ok && p.prec == SPG_P_I4) {
                                // a 128-wide block is pieces 4j .. 4j+3 (16 bytes, 32 nibbles) of each packed row
                                for (uint32_t u0 = ctg; u0 < 512; u0 += 4 * TG) {
                                    uint4 w[4];
#pragma unroll
                                    for (uint32_t i = 0; i < 4; i++) {
                                        const uint32_t u = u0 + i * TG, r7 = u & 7u, pc = (u >> 3) & 3u, row = (u >> 5) * 8u + r7;
                                        w[i] = *reinterpret_cast<const uint4 *>(box + row * 128u + (((4 * j + pc) ^ r7) << 4));
                                    }
#pragma unroll
                                    for (uint32_t i = 0; i < 4; i++) {
                                        const uint32_t u = u0 + i * TG, r7 = u & 7u, pc = (u >> 3) & 3u, row = (u >> 5) * 8u + r7;
                                        const uint32_t m = 0xF0F0F0F0u;
                                        uint4 lo, hi;
                                        lo.x = (w[i].x << 4) & m; lo.y = w[i].x & m; lo.z = (w[i].y << 4) & m; lo.w = w[i].y & m;
                                        hi.x = (w[i].z << 4) & m; hi.y = w[i].z & m; hi.z = (w[i].w << 4) & m; hi.w = w[i].w & m;
                                        *reinterpret_cast<uint4 *>(atile + row * 128u + (((2 * pc) ^ r7) << 4)) = lo;
                                        *reinterpret_cast<uint4 *>(atile + row * 128u + (((2 * pc + 1) ^ r7) << 4)) = hi;
                                    }
                                }
                            } else if (ok) {
                                // INT2: pieces 2j, 2j+1 (64 crumbs each), a word of 16 crumbs becomes one 16-byte chunk
                                for (uint32_t u = ctg; u < 256; u += TG) {
                                    const uint32_t r7 = u & 7u, pc = (u >> 3) & 1u, row = (u >> 4) * 8u + r7;
                                    const uint4 v = *reinterpret_cast<const uint4 *>(box + row * 128u + (((2 * j + pc) ^ r7) << 4));
                                    const uint32_t ws[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
                                    for (uint32_t i = 0; i < 4; i++) {
                                        const uint32_t m = 0xC0C0C0C0u;
                                        *reinterpret_cast<uint4 *>(atile + row * 128u + (((4 * pc + i) ^ r7) << 4)) =
                                            make_uint4((ws[i] << 6) & m, (ws[i] << 4) & m, (ws[i] << 2) & m, ws[i] & m);
                                    }
                                }
                            }
                            fence_async_smem();          // the tensor core reads the tile through the async proxy
                            __syncwarp();
                            if (lane == 0) PAIR ? mbar_arrive_cluster(afull) : mbar_arrive(afull);
                        }
                        if (++as == tiles) { as = 0; aph ^= 1u; }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(rempty0 + 8 * rs);
                    if (++rs == p.RS) { rs = 0; rph ^= 1u; }
                }
            }
        }
    } else {
        spg_grid_wait();
        if (warp == 2) {                                  // one warp looks for all eight
            const int32_t failed = __ldcg(p.status);      // by an earlier launch: its sums and counters are still about
            const bool wide = is_any_wide(p, lane);
            if (lane == 0) *s_last = (wide ? 1 : 0) | (failed ? 2 : 0);
        }
        is_epi_sync();
        const int found = *s_last;
        is_epi_sync();
#define IS_EPI(ACTV) is_epilogue<ACTV, PAIR>(p, found & 1, found & 2, seg, tmem_base, tfull0, lead_tempty0, abort_flag, s_last, s_scale, warp, lane)
        switch (p.act) {
            case SPG_ACT_RELU:    IS_EPI(SPG_ACT_RELU); break;
            case SPG_ACT_LEAKY:   IS_EPI(SPG_ACT_LEAKY); break;
            case SPG_ACT_FOO52:   IS_EPI(SPG_ACT_FOO52); break;
            case SPG_ACT_TANH:    IS_EPI(SPG_ACT_TANH); break;
            case SPG_ACT_SIGMOID: IS_EPI(SPG_ACT_SIGMOID); break;
            default:              IS_EPI(SPG_ACT_NONE); break;
        }
#undef IS_EPI
    }
is_role_done:
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // a wait gave up: give copies that may still be in flight time to land before the shared memory goes away
        if (tid == 0) for (int i = 0; i < 256; i++) __nanosleep(1000);
        __syncthreads();
    }
    if (PAIR) cluster_sync();                            // neither CTA leaves while the other's products read its shared memory or its warps arrive there
    if (warp == 1) { tc_fence_after(); PAIR ? tmem_free_pair(tmem_base, tmem_cols) : tmem_free(tmem_base, tmem_cols); }
}

// ---- host side ---------------------------------------------------------------------------------------------------------

struct IsPlan {
    uint32_t groups, rpg, C, kbr, boxes, ld, m_tiles, tiles, RS, AS, BS, bars, G, GB, grid;
    uint32_t units;
    size_t operand_bytes, smem;
    bool direct, pair, ok;
};

constexpr size_t IS_HEAD = 256 + 4 * MAX_TILES;        // status word, counters; zero between calls, like the sums behind them

// one CTA (or pair) per SM (or two), but a tile in about four pieces at most: the sum over more of them costs more than they save
uint32_t is_ctas(uint64_t tiles, uint32_t boxes, uint32_t most) { const uint64_t want = tiles * (boxes < 4 ? boxes : 4); return want < most ? (uint32_t)want : most; }

IsPlan is_plan(const spgk_layer *L, uint32_t N, uint32_t sms)
{
    IsPlan pl{};
    const int prec = L->precision;
    if (prec != SPG_P_I8 && prec != SPG_P_I4 && prec != SPG_P_I2) return pl;
    if (!L->in || !L->out || L->in > MAX_K || N == 0 || N > SPGK_ISTREAM_MAX_BATCH) return pl;
    const uint32_t bits = spg_bits_per_elem(prec);
    if ((L->in * bits) % 128 || ((uintptr_t)L->w & 15u)) return pl;       // TMA: 16-byte aligned packed rows
    pl.groups = (N + GROUP_ROWS - 1) / GROUP_ROWS;
    pl.rpg = ((N + pl.groups - 1) / pl.groups + 3u) & ~3u;
    pl.kbr = 8u / bits;
    pl.boxes = (L->in * bits + 1023u) / 1024u;
    // Pairs of CTAs where the digits are most of what an SM draws from L2 (more than 32 rows a group; up to 32 rows pairs were level or behind by 7 %)
    // and a CTA alone would have at least 16 blocks in a row.  Pairs over single CTAs in 340 layers of 2048 to 16384 inputs and 512 to 16384 outputs at
    // 40 to 256 rows, weights from HBM, by blocks in a row, INT4: 4 to 8 1.02, 8 to 16 0.99, 16 to 32 0.96, 32 to 64 0.94, beyond 0.92 (INT2 the
    // same; INT8 1.02, 1.02, 0.98, 1.00, 0.96).  INT8, which 64 rows stream at the rate of HBM, only from the second group on (40 rows: 170 against 167 us, 72
    // rows: 253 against 261).  A pair's tile has two counters.
    const uint64_t alone = (uint64_t)((L->out + TILE_ROWS - 1) / TILE_ROWS) * pl.groups, ctas = is_ctas(alone, pl.boxes, sms);
    const uint64_t paired = (uint64_t)((L->out + 2 * TILE_ROWS - 1) / (2 * TILE_ROWS)) * pl.groups;
    pl.pair = pl.rpg > IS_PAIR_ROWS && 2 * paired <= MAX_TILES && alone * pl.boxes * pl.kbr >= IS_PAIR_BLOCKS * ctas && L->out > TILE_ROWS && sms >= 2 && (prec != SPG_P_I8 || pl.groups > 1);
    if (pl.pair) pl.rpg = (pl.rpg + 7u) & ~7u;                            // (a pair's product takes multiples of 32 columns)
    pl.C = 4 * pl.rpg;
    pl.direct = prec == SPG_P_I8;
    pl.ld = pl.boxes * pl.kbr * 128u;
    const uint32_t high = pl.pair ? 2 * TILE_ROWS : TILE_ROWS;
    pl.m_tiles = (L->out + high - 1) / high;
    pl.tiles = pl.m_tiles * pl.groups;
    if (pl.tiles > MAX_TILES) return pl;
    pl.units = pl.tiles * pl.boxes;
    pl.grid = pl.pair ? 2 * is_ctas(pl.tiles, pl.boxes, sms / 2) : is_ctas(pl.tiles, pl.boxes, sms);
    // rings: operand tiles in two slots of G blocks, digit tiles up to 96 KB (in pairs up to 32 rows), boxes with the rest
    const uint32_t b_bytes = pl.C * (pl.pair ? 64u : 128u);
    pl.G = pl.direct ? 1 : 2;
    pl.AS = pl.direct ? 1 : pl.C > 128 ? 2 : 0;      // (in shared memory only for layers that turn out wide)
    pl.bars = pl.direct ? 1 : IS_A_SLOTS;
    pl.GB = pl.direct || b_bytes > 16384 ? 1 : 2;
    pl.BS = 96u * 1024 / b_bytes;
    if (pl.BS > 8) pl.BS = 8;
    pl.BS /= pl.GB;
    const uint32_t a_bytes = pl.direct ? 0 : pl.AS * pl.G * BOX_BYTES;
    pl.RS = (224u * 1024 - a_bytes - pl.BS * pl.GB * b_bytes) / BOX_BYTES;
    if (pl.RS > 10) pl.RS = 10;
    pl.smem = 1024 + (size_t)pl.RS * BOX_BYTES + a_bytes + (size_t)pl.BS * pl.GB * b_bytes + 16 * (pl.RS + pl.bars + pl.BS) + 32 + 16 + 2 * GROUP_ROWS * sizeof(double);
    pl.operand_bytes = 2 * (size_t)pl.groups * pl.C * pl.ld;              // both sets of digits
    pl.ok = pl.smem <= 227u * 1024;
    return pl;
}

typedef CUresult (*IsEncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                               const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 2-D byte map with 128-byte swizzle, box of 128 bytes x `box_rows`
int is_map(const void *ptr, uint64_t row_bytes, uint64_t rows, uint32_t box_rows, CUtensorMap *out)
{
    static IsEncodeFn fn = []() -> IsEncodeFn {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
        return reinterpret_cast<IsEncodeFn>(f);
    }();
    if (!fn) { spgk_set_error("cuTensorMapEncodeTiled", "driver entry point not available"); return SPGK_E_CUDA; }
    cuuint64_t dims[2] = { row_bytes, rows };
    cuuint64_t strides[1] = { row_bytes };
    cuuint32_t box[2] = { 128, box_rows };
    cuuint32_t estr[2] = { 1, 1 };
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char msg[64];
        snprintf(msg, sizeof msg, "CUresult %d", (int)r);
        spgk_set_error("cuTensorMapEncodeTiled (integer stream)", msg);
        return SPGK_E_CUDA;
    }
    return SPGK_OK;
}

// scratch: head | sums, one slot per CTA and set of digits, of a size that depends on the device alone (they are zero between
// calls of any batch size): 19.4 MB on 148 SMs | digit operand of the largest layer | row scales |
// a byte per row
struct IsScratch { size_t sums, sums2, operand, scales, wide, total; bool ok; };
IsScratch is_scratch(const spgk_layer *layers, uint32_t count, uint32_t N, uint32_t sms)
{
    IsScratch s{};
    size_t operand = 0, rows = 0;
    for (uint32_t l = 0; l < count; l++) {
        if (l + 1 < count && (layers[l].act == SPG_ACT_SOFTMAX || layers[l + 1].in != layers[l].out)) return s;
        const IsPlan pl = is_plan(&layers[l], N, sms);
        if (!pl.ok) return s;
        if (pl.operand_bytes > operand) operand = pl.operand_bytes;
        if ((size_t)pl.groups * pl.rpg > rows) rows = (size_t)pl.groups * pl.rpg;
    }
    if (!rows) return s;
    s.sums = IS_HEAD;
    s.sums2 = s.sums + (size_t)sms * GROUP_ROWS * TILE_ROWS * sizeof(long long);
    s.operand = s.sums2 + (s.sums2 - s.sums);
    s.scales = s.operand + ((operand + 255) & ~(size_t)255);
    s.wide = s.scales + 2 * rows * sizeof(double);
    s.total = s.wide + rows;
    s.ok = true;
    return s;
}

}  // namespace

extern "C" {

int spgk_istream_arrangement(const spgk_layer *L, uint32_t N, uint32_t sms, uint32_t out[4])
{
    SpgDeviceProps dp;
    if (!L || (!sms && spg_device_props(&dp) != SPGK_OK)) return 0;
    const IsPlan pl = is_plan(L, N, sms ? sms : (uint32_t)dp.sm_count);
    out[0] = pl.pair ? 2 : 1; out[1] = pl.rpg; out[2] = pl.tiles; out[3] = pl.grid;
    return pl.ok ? 1 : 0;
}

size_t spgk_istream_scratch_bytes(const spgk_layer *layers, uint32_t count, uint32_t N)
{
    SpgDeviceProps dp;
    if (!layers || spg_device_props(&dp) != SPGK_OK || dp.cc != 100) return 0;
    const IsScratch s = is_scratch(layers, count, N, (uint32_t)dp.sm_count);
    return s.ok ? s.total : 0;
}

int spgk_istream_forward(const spgk_layer *layers, uint32_t count, const float *x, uint32_t ldx, float *const *ys, uint32_t N,
                         void *scratch, void *stream)
{
    if (!layers || !x || !ys || !scratch) { spgk_set_error("spgk_istream_forward", "bad argument"); return SPGK_E_ARG; }
    SpgDeviceProps dp;
    int rc;
    if ((rc = spg_device_props(&dp))) return rc;
    if (dp.cc != 100) return SPGK_E_UNSUPPORTED;                         // tcgen05 / TMEM exist on sm_100 only
    const uint32_t sms = (uint32_t)dp.sm_count;
    const IsScratch sc = is_scratch(layers, count, N, sms);
    if (!sc.ok) return SPGK_E_UNSUPPORTED;
    {
        static SpgOncePerDevice once;
        int dev = 0;
        SPGK_CUDA(cudaGetDevice(&dev));
        rc = once.run(dev, [&]() -> int {
            SPGK_CUDA(cudaFuncSetAttribute(spg_istream_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            SPGK_CUDA(cudaFuncSetAttribute(spg_istream_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            return SPGK_OK;
        });
        if (rc) return rc;
    }
    cudaStream_t s = (cudaStream_t)stream;
    uint8_t *base = reinterpret_cast<uint8_t *>(scratch);
    uint8_t *operand = base + sc.operand;
    double *row_scale = reinterpret_cast<double *>(base + sc.scales);
    const float *xin = x;
    uint32_t xld = ldx;
    for (uint32_t l = 0; l < count; l++) {
        const spgk_layer *L = &layers[l];
        const IsPlan pl = is_plan(L, N, sms);
        const uint32_t vec = (((uintptr_t)xin | ((uintptr_t)xld * 4)) & 15u) == 0;
        auto stage = L->precision == SPG_P_I8 ? spg_is_stage_kernel<SPG_P_I8> : L->precision == SPG_P_I4 ? spg_is_stage_kernel<SPG_P_I4> : spg_is_stage_kernel<SPG_P_I2>;
        CUtensorMap map_w, map_x;
        if ((rc = is_map(L->w, (uint64_t)L->in * spg_bits_per_elem(L->precision) / 8, L->out, TILE_ROWS, &map_w))) return rc;
        if ((rc = is_map(operand, pl.ld, 2 * (uint64_t)pl.groups * pl.C, pl.pair ? pl.C / 2 : pl.C, &map_x))) return rc;
        SPGK_CUDA(spg_launch_chained(stage, dim3(pl.groups * pl.rpg), dim3(STAGE_THREADS), 0, s, xin, xld, N, L->in, pl.ld, vec, operand, row_scale, base + sc.wide));
        if ((rc = spgk_check_launch("spg_is_stage_kernel"))) return rc;
        IsParams p{};
        p.out = L->out; p.groups = pl.groups; p.rpg = pl.rpg; p.N = N; p.C = pl.C; p.rows = pl.groups * pl.rpg;
        p.kbr = pl.kbr; p.boxes = pl.boxes; p.units = pl.units;
        p.RS = pl.RS; p.AS = pl.AS; p.BS = pl.BS; p.bars = pl.bars; p.G = pl.G; p.GB = pl.GB;
        p.direct = pl.direct; p.prec = L->precision;
        p.act = L->act == SPG_ACT_SOFTMAX ? SPG_ACT_NONE : L->act;
        p.scale = (double)L->w_scale / (L->precision == SPG_P_I4 ? 16.0 : L->precision == SPG_P_I2 ? 64.0 : 1.0);
        p.bias = L->bias; p.row_scale = row_scale; p.wide = base + sc.wide;
        p.y = ys[l]; p.ldy = L->out;
        p.status = reinterpret_cast<int32_t *>(base);
        p.counters = reinterpret_cast<uint32_t *>(base + 256);
        p.sums = reinterpret_cast<unsigned long long *>(base + sc.sums);
        p.sums2 = reinterpret_cast<unsigned long long *>(base + sc.sums2);
        p.idesc = idesc_i8(pl.pair ? 2 * TILE_ROWS : TILE_ROWS, pl.C);
        if (pl.pair) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(pl.grid); cfg.blockDim = dim3(IS_THREADS); cfg.dynamicSmemBytes = pl.smem; cfg.stream = s;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr; cfg.numAttrs = 2;
            SPGK_CUDA(cudaLaunchKernelEx(&cfg, spg_istream_kernel<true>, map_w, map_x, p));
        } else
            SPGK_CUDA(spg_launch_chained(spg_istream_kernel<false>, dim3(pl.grid), dim3(IS_THREADS), pl.smem, s, map_w, map_x, p));
        if ((rc = spgk_check_launch("spg_istream_kernel"))) return rc;
        xin = ys[l]; xld = L->out;
    }
    return SPGK_OK;
}

int spgk_istream_status(void *scratch, void *stream)
{
    int32_t h = 0;
    SPGK_CUDA(cudaMemcpyAsync(&h, scratch, sizeof h, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    SPGK_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (h != 0) {
        char msg[96];
        snprintf(msg, sizeof msg, "bounded wait %d gave up inside the integer streaming kernel", (int)h);
        spgk_set_error("spg_istream_kernel", msg);
        SPGK_CUDA(cudaMemsetAsync(scratch, 0, sizeof h, (cudaStream_t)stream));
        return SPGK_E_TIMEOUT;
    }
    return SPGK_OK;
}

}  // extern "C"
