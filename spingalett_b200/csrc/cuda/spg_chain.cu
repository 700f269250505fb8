// spg_chain.cu -- a whole net on a batch of some ten to some thousand rows in one launch (tcgen05, clusters of up to eight CTAs).
//
// Layer by layer such a batch is all latency: 256 rows of a 784-512-1000-10 net took four launches of 5 us each whose tensor
// cores were idle nearly all of the time.  Rows do not depend on one another, so here a cluster takes a block of R rows through
// every layer and nothing ever waits for the whole grid.  Inside a cluster the outputs of a layer are shared out: CTA r computes
// its slice for all R rows, writes it to a scratch in L2 as the next layer's operand tiles, and the CTAs tell one another on an
// mbarrier.  A last layer of up to 128 outputs is cut along K instead: each CTA multiplies the outputs that it has just computed,
// from its own shared memory, and the sums of a row meet in the CTA that puts the row together (and applies a softmax).
//
// The operands are swapped: the weights are the 128-row side of the tensor core's tile and the batch rows its columns, so a
// block may have any multiple of 16 rows.  A row's high and low 16-bit terms are neighbouring columns: one product serves both.
// The input is rounded to its terms on the way into shared memory.  The weight ring runs ahead of the layers, and starts before
// the kernel in front has ended.
//
// The tensor core cuts off what of a product does not fit the sum, so what a sum loses goes by how many products follow one another in an
// accumulator.  A tile has two accumulators where there is room, and up to eight (the stages of K in turn, or one a k-block) where it takes more for all
// layers together to add no more in a row than the layer kernels do, which cut K over CTAs (`steps_allowed`); a net that does not fit with so many
// stays with those.  Error against 64 bits, positive values and weights, layer kernels / two accumulators / now: 4096-512-64 in FP16 at
// 200 rows 3.3e-6 / 11.7e-6 / 2.7e-6, 8192-512-64 in BF16 at 1000 rows 7.2e-6 / 12.7e-6 / 4.5e-6, 784-512-1000-10 in FP16 at 256 rows 2.2e-6 / 3.4e-6 /
// 1.9e-6; values of either sign half of the layer kernels'.  An accumulator more costs 250 cycles a layer and 32 rows: FP16 at 256 rows 13.7 -> 14.5 us.
//
// A row's sums depend on the size of the cluster where the last layer is cut, and on the accumulators of a tile, which go by the number of rows,
// but not on the other rows, nor on R otherwise.
//
// What bounds it: latency.  256 rows of 784-512-1000-10 in INT4, clusters of 8 on 32 rows each, in cycles: first rows of the input
// 2700, all of them in shared memory 6000, first layer multiplied 9800 (a product of 128 x 64 x 16 takes 65 cycles, 58 of them whatever
// its width, to fetch the weights from shared memory), its outputs in the other CTAs 14200 (1200 of it for the release of the stores),
// second layer 17400, last layer's sums 20000, rows put together 23500 (with sixteen epilogue warps; eight save 1200); 2 us from the end to the next launch's first load.  With
// more rows the epilogues' instructions weigh: 3001 rows of 301-777-333-129-37, clusters of 4 on 96 rows, spend half of the time there.
//
// Measured against layer by layer (us): 784-512-1000-10 at 256 rows 22.9 -> 13.9 (INT4), 22.0 -> 17.7 (fp32, three products a term), 1500 rows
// 29 -> 20; 301-777-333-129-37 in FP16 at 3001 rows 39.2 -> 32.2; 100-65-130-7 at 3000 rows 25.5 -> 13.4; 1024-256-256-256-10 at 12000 rows 76 -> 38;
// 128-128-128-128-128-128 at 256 rows 39 -> 14.  Against the 16-bit streaming kernel at 33 rows: 784-512-1000-10 in BF16 114 -> 12.
// Tried: four rows a round of the epilogue instead of eight (560 cycles a round of four, eight little more), the input's loads ahead of the
// fence that hands a tile on (the fence waits for them), one k-block a stage (waits and commits, 400 cycles a stage, twice as often).
//
// Every wait is bounded as in spg_gemm_tc.cu.  A wait that gave up in one CTA is known to its cluster, which finishes no row any more; copies
// and products under way are awaited (again with a bound) before shared and tensor memory are given back.
#include "spg_common.cuh"
#include "spg_tc.cuh"
#include "spg_gemm.cuh"
#include <cmath>

namespace {

using namespace spgtc;

constexpr uint32_t TK = 64, TM = 128;                          // of a weight tile
constexpr uint32_t KG = 2;                                     // k-blocks that change hands at once
constexpr uint32_t MAX_LAYERS = SPGK_CHAIN_MAX_LAYERS, MAX_C = 8, MAX_R = 256, MAX_RING = 12;
constexpr uint32_t threads_of(uint32_t epi) { return 128 + 32 * epi; }
constexpr uint32_t TAIL_MAX = 128, MAX_MT = 4;                 // outputs of a last layer whose sums are put together
constexpr uint32_t MAX_ACC = 8;                                // accumulators of a tile
constexpr uint32_t COUNTED_C = 4;                              // CTAs of a cluster where only the device knows the number of rows
constexpr uint32_t BAR_BYTES = 8 * (5 * MAX_RING + 6) + 32;

struct ChainLayer {
    const float *bias;
    float scale;
    int act;
    uint32_t in, out, kblocks, stages;  // stages: of KG k-blocks
    uint32_t tr, mt;                  // rows of a weight tile, tiles of a CTA
    uint32_t mains, run;              // accumulators of a tile (each of 16-bit terms times n columns), stages of one of them (0: a k-block)
    uint32_t covered;                 // outputs of all tiles together: the next layer's columns from here on are nobody's
};
struct ChainParams {
    CUtensorMap w[MAX_LAYERS];
    ChainLayer l[MAX_LAYERS];
    uint32_t layers, R, C;
    uint32_t tail, tail_rows;         // CTAs that the last layer's K is cut over (0: it is not); most rows that one of them puts together
    uint32_t SA, SW, a_slot, w_slot, tmem_cols;
    uint32_t idesc_base;
    const float *x; uint32_t ldx, vec4; const uint32_t *x_rows;
    float *y; uint32_t ldy; const uint32_t *y_rows;
    uint32_t softmax;
    float margin_theta; uint32_t *margin_idx, *margin_count;
    uint8_t *scratch; uint32_t exchange_bytes;
    uint32_t rows; const uint32_t *limit;
    int impatient;
    int ready;                        // no kernel before this one makes the weights
    int early;                        // ... and the number of rows is known before it has ended
    int32_t *status;
};

__device__ __forceinline__ void load_planes(uint32_t dst, const CUtensorMap *map, uint32_t bar, int k, int row)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(k), "r"(row), "r"(0) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void arrive_release_cluster(uint32_t addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
template <uint32_t EPI> __device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI) : "memory"); }

// (relaxed: who waits reads nothing that was written before; a release would wait for the outputs' stores, 1400 cycles)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Bounded wait on a barrier that the other CTAs of the cluster arrive on, whose writes to global memory are read afterwards
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag, int32_t *status, int code)
{
    for (uint32_t i = 0; i < 1u << 16; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity), "r"(SPG_WAIT_HINT_NS) : "memory");
        if (ok) return true;
        if ((i & 7u) == 7u && *abort_flag) return false;
    }
    *abort_flag = 1;
    atomicCAS(status, 0, code);
    return false;
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}

// the high 16-bit terms of a pair of values (a in the low half); a, b: what is left of them
template <typename T16> __device__ __forceinline__ uint32_t round2(float &a, float &b)
{
    union { uint32_t q; __half2 h; __nv_bfloat162 f; } pk;
    if constexpr (__is_same(T16, __half)) { pk.h = __floats2half2_rn(a, b); const float2 back = __half22float2(pk.h); a -= back.x; b -= back.y; }
    else { pk.f = __floats2bfloat162_rn(a, b); a -= __uint_as_float(pk.q << 16); b -= __uint_as_float(pk.q & 0xFFFF0000u); }
    return pk.q;
}

// where the 16-bit value of row r and column k of a tile of rows of 128 bytes lies (128-byte swizzle)
__device__ __forceinline__ uint32_t swizzled(uint32_t r, uint32_t k) { return r * 128 + ((((k >> 3) ^ r) & 7u) << 4) + (k & 7u) * 2; }

// a place in a ring of tiles
struct Ring {
    uint32_t slot = 0, phase = 0;
    __device__ __forceinline__ void next(uint32_t slots) { if (++slot == slots) { slot = 0; phase ^= 1u; } }
};

// What an epilogue warp needs of a layer
struct Slice {
    uint32_t tmem;                    // its lane quadrant
    uint32_t o, tiles, tr;            // the lane's output in the first tile (only lanes below tr have one), weight tiles, rows of one
    uint32_t n, mains, out;           // rows of the block
    uint32_t first, end;              // batch rows: the block's first, beyond its last
    uint32_t q, g, lane;
    int act;
    float scale, bias[MAX_MT];
};

// (not inlined: four of them side by side at every place that finishes values want more registers than there are)
__device__ __noinline__ float4 curved4(float4 v, int act)
{
    if (act == SPG_ACT_TANH) return make_float4(spg_activate(v.x, SPG_ACT_TANH), spg_activate(v.y, SPG_ACT_TANH), spg_activate(v.z, SPG_ACT_TANH), spg_activate(v.w, SPG_ACT_TANH));
    return make_float4(spg_activate(v.x, SPG_ACT_SIGMOID), spg_activate(v.y, SPG_ACT_SIGMOID), spg_activate(v.z, SPG_ACT_SIGMOID), spg_activate(v.w, SPG_ACT_SIGMOID));
}
constexpr int CURVED = -1;                                     // tanh or sigmoid
template <int ACT, int N> __device__ __forceinline__ void activate(float (&v)[N], int act)
{
    if constexpr (ACT == CURVED && N == 1) v[0] = curved4(make_float4(v[0], 0.0f, 0.0f, 0.0f), act).x;
    else if constexpr (ACT == CURVED) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float4 f = curved4(make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]), act);
            v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = spg_activate(v[i], ACT);
    }
}
constexpr int MANY = 0;
// A layer's activation is chosen once, outside the loops (a branch inside costs as much as the activation),
// and so is the number of accumulators: 1, 2, or MANY
#define SPG_CHAIN_ACCS(act, accs, call)                                                         \
    if ((accs) == 1) call(act, 1); else if ((accs) == 2) call(act, 2); else call(act, MANY)
#define SPG_CHAIN_ACTS(act, accs, call)                                                         \
    switch (act) {                                                                             \
        case SPG_ACT_RELU:  SPG_CHAIN_ACCS(SPG_ACT_RELU, accs, call); break;                     \
        case SPG_ACT_LEAKY: SPG_CHAIN_ACCS(SPG_ACT_LEAKY, accs, call); break;                    \
        case SPG_ACT_FOO52: SPG_CHAIN_ACCS(SPG_ACT_FOO52, accs, call); break;                    \
        case SPG_ACT_NONE:  SPG_CHAIN_ACCS(SPG_ACT_NONE, accs, call); break;                     \
        default:            SPG_CHAIN_ACCS(CURVED, accs, call); break;                           \
    }

// One output of eight rows: four from a place in sixteen rows on, and the four sixteen further on, or the first four again where the block has
// no more.  (A warp's instructions hang on one another: eight rows take little longer than four, 560 cycles.)  The accumulators' sums in
// their order; zeros where the output is a dead one of a warp that has some (edge: masks in every warp cost 3001 rows of 301-777-333-129-37 0.8 us of
// 31, a branch behind the wait 0.1; zeros stored afterwards 0.7 to 3.5).
template <int AP, int ACC>
__device__ __forceinline__ void sums8(const Slice &s, uint32_t taddr, uint32_t more, bool edge, bool dead, float (&v)[8])
{
    if constexpr (ACC == MANY) {
        // (two a turn; where their number is odd the last one's place is read again and left out)
        float low[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = low[i] = 0.0f;
#pragma unroll 1
        for (uint32_t a = 0; a < s.mains; a += 2) {
            const bool pair = a + 1 < s.mains;
            uint32_t hi[2][2][4], lo[2][2][4];
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t at = taddr + (a + (b && pair ? 1 : 0)) * AP * s.n + (h ? more : 0);
                    tmem_ld4(at, hi[b][h]);
                    if (AP > 1) tmem_ld4(at + s.n, lo[b][h]);
                }
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int h = i >> 2, j = i & 3;
                v[i] += __uint_as_float(hi[0][h][j]) + (pair ? __uint_as_float(hi[1][h][j]) : 0.0f);
                if (AP > 1) low[i] += __uint_as_float(lo[0][h][j]) + (pair ? __uint_as_float(lo[1][h][j]) : 0.0f);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (AP > 1) v[i] += low[i];
            if (edge && dead) v[i] = 0.0f;
        }
    } else {
        constexpr bool BOTH = ACC == 2;
        const uint32_t second = AP * s.n;
        uint32_t hi[2][4], lo[2][4], hi2[2][4], lo2[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t at = taddr + (h ? more : 0);
            tmem_ld4(at, hi[h]);
            if (AP > 1) tmem_ld4(at + s.n, lo[h]);
            if (BOTH) tmem_ld4(at + second, hi2[h]);
            if (BOTH && AP > 1) tmem_ld4(at + second + s.n, lo2[h]);
        }
        tmem_ld_wait();
        if (edge) {
            const uint32_t keep = dead ? 0u : 0xFFFFFFFFu;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int h = i >> 2, j = i & 3;
                hi[h][j] &= keep;
                if (AP > 1) lo[h][j] &= keep;
                if (BOTH) hi2[h][j] &= keep;
                if (BOTH && AP > 1) lo2[h][j] &= keep;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int h = i >> 2, j = i & 3;
            v[i] = __uint_as_float(hi[h][j]);
            if (BOTH) v[i] += __uint_as_float(hi2[h][j]);
            if (AP > 1) v[i] += BOTH ? __uint_as_float(lo[h][j]) + __uint_as_float(lo2[h][j]) : __uint_as_float(lo[h][j]);
        }
    }
}
// ... scale, bias, activation
template <int ACT, int AP, int ACC>
__device__ __forceinline__ void finish8(const Slice &s, uint32_t taddr, uint32_t more, float bias, bool edge, bool dead, float (&v)[8])
{
    sums8<AP, ACC>(s, taddr, more, edge, dead, v);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = fmaf(v[i], s.scale, bias);
    activate<ACT>(v, s.act);
}

// A layer's outputs become the next one's operand: [k-block][plane][row] of 128 bytes.  Lane pairs trade rows so that each writes
// two neighbouring values at once.  Columns beyond the layer's outputs get the activation of zero, whose weights are zeros.  Their own sums are not taken
// for it: a row with an infinity times weights of zero is NaN, and so it would be with the next layer's zeros.
template <int ACT, int ACC, typename T16, int AP, uint32_t EPI>
__device__ __forceinline__ void to_operand(const Slice &s, uint8_t *next, uint32_t k0, uint32_t next_k, uint32_t plane)
{
    const uint32_t odd = s.lane & 1u;
#pragma unroll 1
    for (uint32_t t = 0; t < s.tiles; t++) {
        const uint32_t k = ((s.o + t * s.tr) & ~1u) - k0;      // (k0: the operand's first column)
        const bool in = s.q * 32 + s.lane < s.tr && k < next_k;                               // (tr, next_k: even)
        const bool dead = s.o + t * s.tr >= s.out, edge = __any_sync(0xffffffffu, dead);
        const float bias = t == 0 ? s.bias[0] : t == 1 ? s.bias[1] : t == 2 ? s.bias[2] : s.bias[3];
        uint32_t taddr = s.tmem + t * s.mains * AP * s.n + 4 * s.g;
        uint8_t *dst = next + (k >> 6) * (AP * plane) + 4 * s.g * 128;
        // of rows c + odd and c + 2 + odd, where c is a multiple of 8; four rows on another 16 bytes
        const uint32_t at = swizzled(odd, k & 63u) ^ ((4 * s.g & 4u) << 4);
#pragma unroll 1
        for (uint32_t c = 4 * s.g; c < s.n; c += 2 * EPI, taddr += 2 * EPI, dst += 2 * EPI * 128) {
            const bool two = c + EPI < s.n;
            float v[8];
            finish8<ACT, AP, ACC>(s, taddr, two ? EPI : 0, bias, edge, dead, v);
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
                float a = odd ? got : v[i], b = odd ? v[i + 1] : got;                         // outputs k and k + 1 of a row
                uint8_t *to = dst + ((i & 2) + (i >> 2) * EPI) * 128 + (at ^ ((i & 2) << 4));
                const uint32_t hi = round2<T16>(a, b);
                if (in && (i < 4 || two)) {
                    *reinterpret_cast<uint32_t *>(to) = hi;
                    if (AP > 1) *reinterpret_cast<uint32_t *>(to + plane) = round2<T16>(a, b);
                }
            }
        }
    }
}

template <int ACT, int ACC, int AP, uint32_t EPI>
__device__ __forceinline__ void to_output(const ChainParams &p, const Slice &s)
{
#pragma unroll 1
    for (uint32_t t = 0; t < s.tiles; t++) {
        const uint32_t o = s.o + t * s.tr;
        const bool live = s.q * 32 + s.lane < s.tr && o < s.out;
        const float bias = t == 0 ? s.bias[0] : t == 1 ? s.bias[1] : t == 2 ? s.bias[2] : s.bias[3];
        const uint32_t taddr = s.tmem + t * s.mains * AP * s.n;
#pragma unroll 1
        for (uint32_t c = 4 * s.g; c < s.n; c += 2 * EPI) {
            float v[8];
            finish8<ACT, AP, ACC>(s, taddr + c, c + EPI < s.n ? EPI : 0, bias, false, false, v);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t r = c + (i & 3) + (i >> 2) * EPI, row = s.first + r;
                if (live && r < s.n && row < s.end) p.y[(uint64_t)(p.y_rows ? p.y_rows[row] : row) * p.ldy + o] = v[i];
            }
        }
    }
}

// A narrow last layer: every CTA has multiplied its own outputs of the layer before, which nobody else needs then, by their part of K.  The
// sums of a row go to the CTA that puts the row together: rows r * R / P and on are CTA r's, of P.  owners: where a row's sums begin there, and
// the barrier that counts them; part: from there to this CTA's.
template <int AP, uint32_t EPI> __device__ __forceinline__ void to_owners(const Slice &s, const uint2 *owners, uint32_t part, uint32_t bar)
{
    part += s.o * 4;
#pragma unroll 1
    for (uint32_t c = 4 * s.g; c < s.n; c += 2 * EPI) {
        const uint32_t more = c + EPI < s.n ? EPI : 0;
        float v[8];
        if (s.mains == 1) sums8<AP, 1>(s, s.tmem + c, more, false, false, v);         // (by whole warps)
        else sums8<AP, MANY>(s, s.tmem + c, more, false, false, v);
        if (s.o < s.out) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (i >= 4 && !more) break;
                const uint2 to = owners[c + (i & 3) + (i >> 2) * EPI];
                asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                             ::"r"(to.x + part), "r"(__float_as_uint(v[i])), "r"(to.y + bar) : "memory");
            }
        }
        __syncwarp();
    }
}

// ... which adds them in CTA order and finishes the rows, a warp a row; formulas and margin test of the softmax as in the epilogues of the
// layer kernels
template <int PER, uint32_t EPI>                               // PER: outputs of a lane
__device__ __forceinline__ void put_together(const ChainParams &p, int act, uint32_t out, float scale, const float (&bias)[MAX_MT], const float *parts, uint32_t first, uint32_t count,
                                             uint32_t end, uint32_t w, uint32_t lane)
{
    const uint32_t part = p.tail_rows * out;
#pragma unroll 1
    for (uint32_t r = w; r < count; r += EPI) {
        const uint32_t row = first + r;
        if (row >= end) break;
        float v[PER], mx = -FLT_MAX, second = -FLT_MAX;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const uint32_t o = i * 32 + lane;
            v[i] = 0.0f;
            if (o < out) {
                const float *at = parts + r * out + o;
                float sum = at[0];
#pragma unroll 4
                for (uint32_t c = 1; c < p.tail; c++) sum += at[c * part];
                v[i] = fmaf(sum, scale, bias[i]);
                if (v[i] > mx) { second = mx; mx = v[i]; } else if (v[i] > second) second = v[i];
            }
        }
        float *y = p.y + (uint64_t)(p.y_rows ? p.y_rows[row] : row) * p.ldy;
        if (p.softmax) {
#pragma unroll
            for (uint32_t o = 16; o > 0; o >>= 1) {
                const float m2 = __shfl_xor_sync(0xffffffffu, mx, o), s2 = __shfl_xor_sync(0xffffffffu, second, o);
                second = fmaxf(fminf(mx, m2), fmaxf(second, s2));
                mx = fmaxf(mx, m2);
            }
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < PER; i++) {
                v[i] = (uint32_t)i * 32 + lane < out ? expf(v[i] - mx) : 0.0f;
                sum += v[i];
            }
            sum = spg_warp_sum(sum);
            if (lane == 0 && p.margin_idx && out >= 2 && (!(mx - second >= p.margin_theta) || !(sum < FLT_MAX)))
                p.margin_idx[atomicAdd(p.margin_count, 1u)] = row;
            const float inv = sum > 0.0f ? 1.0f / sum : 1.0f;
#pragma unroll
            for (int i = 0; i < PER; i++) if ((uint32_t)i * 32 + lane < out) y[i * 32 + lane] = v[i] * inv;
        } else if (lane < out) {
#define SPG_CHAIN_CALL(A, B) activate<A>(v, act)
            SPG_CHAIN_ACTS(act, 1, SPG_CHAIN_CALL)
#undef SPG_CHAIN_CALL
#pragma unroll
            for (int i = 0; i < PER; i++) if ((uint32_t)i * 32 + lane < out) y[i * 32 + lane] = v[i];
        }
    }
}

// The block's rows of the input as operand tiles: a warp rounds eight rows of a stage at a time, four columns a lane, so that it waits and
// hands on once for them.  (A fence waits for the loads that are under way: none is then.)  VEC: rows lie on 16 bytes and end on a group of four.
template <typename T16, int AP, bool VEC, uint32_t EPI>
__device__ __forceinline__ bool round_input(const ChainParams &p, uint32_t block0, uint32_t rows, uint32_t in, uint32_t stages, uint32_t w, uint32_t lane, uint8_t *tiles,
                                            uint32_t a_empty, uint32_t a_conv, Ring ring, volatile int *abort_flag)
{
    const uint32_t SA = p.SA, groups = p.R / 8, plane = p.R * 128;
    uint8_t *const lane_at = tiles + (lane >> 4) * (AP * plane) + (lane & 1u) * 8;
    const uint32_t chunk = (lane >> 1) & 7u;
    uint32_t stage = 0, group = w;
    bool ok = true;
    while (group >= groups) { group -= groups; stage++; ring.next(SA); }
#pragma unroll 1
    while (stage < stages) {
        const uint32_t k = stage * (KG * TK) + 4 * lane, row0 = block0 + 8 * group;
        float4 v[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {
            const uint32_t row = row0 + j;
            const bool there = row < rows && k < in;
            const float *src = p.x + (uint64_t)(there && p.x_rows ? p.x_rows[row] : row) * p.ldx + k;
            v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (VEC) { if (there) v[j] = __ldg(reinterpret_cast<const float4 *>(src)); }
            else if (there) {
                v[j].x = __ldg(src);
                if (k + 1 < in) v[j].y = __ldg(src + 1);
                if (k + 2 < in) v[j].z = __ldg(src + 2);
                if (k + 3 < in) v[j].w = __ldg(src + 3);
            }
        }
        ok = __all_sync(0xffffffffu, ok && mbar_wait(a_empty + 8 * ring.slot, ring.phase ^ 1u, abort_flag, p.status, 69));
        if (ok) {
            uint8_t *at = lane_at + ring.slot * p.a_slot + group * 1024;
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                uint2 q;
                q.x = round2<T16>(v[j].x, v[j].y); q.y = round2<T16>(v[j].z, v[j].w);
                *reinterpret_cast<uint2 *>(at + j * 128 + ((chunk ^ j) << 4)) = q;
                if (AP > 1) {
                    q.x = round2<T16>(v[j].x, v[j].y); q.y = round2<T16>(v[j].z, v[j].w);
                    *reinterpret_cast<uint2 *>(at + plane + j * 128 + ((chunk ^ j) << 4)) = q;
                }
            }
            fence_async_smem();
        }
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(a_conv + 8 * ring.slot);
        group += EPI;
        while (group >= groups) { group -= groups; stage++; ring.next(SA); }
    }
    return ok;
}

// AP, WP: 16-bit terms of an activation and of a weight
template <typename T16, int AP, int WP, uint32_t EPI>
__global__ void __launch_bounds__(threads_of(EPI), 1)
spg_chain_kernel(const __grid_constant__ ChainParams p)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem);
    const uint32_t a_off = p.SW * p.w_slot, bar_off = a_off + p.SA * p.a_slot, owners_off = bar_off + BAR_BYTES, parts_off = owners_off + p.R * 8;
    const uint32_t w_full = base + bar_off, w_empty = w_full + 8 * MAX_RING, a_full = w_empty + 8 * MAX_RING, a_conv = a_full + 8 * MAX_RING,
                   a_empty = a_conv + 8 * MAX_RING, ready = a_empty + 8 * MAX_RING, done = ready + 8, drain = done + 8, own = drain + 8, parts_bar = own + 8;      // (two of the last)
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + bar_off + 8 * (5 * MAX_RING + 6));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1), *drain_flag = reinterpret_cast<volatile int *>(tmem_slot + 2);
    const uint32_t abort_addr = smem_u32(const_cast<int *>(abort_flag)), drain_addr = abort_addr + 4;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    const uint32_t me = cluster_rank(), C = p.C, clusters = gridDim.x / C, cluster = blockIdx.x / C;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < p.SW; i++) { mbar_init(w_full + 8 * i, 1); mbar_init(w_empty + 8 * i, 1); }
        for (uint32_t i = 0; i < p.SA; i++) { mbar_init(a_full + 8 * i, 1); mbar_init(a_conv + 8 * i, p.R / 8); mbar_init(a_empty + 8 * i, 1); }
        mbar_init(ready, C);
        mbar_init(done, 1);
        mbar_init(drain, 1);
        mbar_init(own, EPI);
        mbar_init(parts_bar, 1);
        mbar_init(parts_bar + 8, 1);
        *abort_flag = 0; *drain_flag = 0;
        mbar_fence_init();
    }
    uint2 *const owners = reinterpret_cast<uint2 *>(smem + owners_off);
    if (p.tail)
        for (uint32_t r = threadIdx.x; r < p.R; r += 128 + 32 * EPI) {
            const uint32_t owner = ((r + 1) * p.tail - 1) / p.R, first = owner * p.R / p.tail;
            owners[r] = make_uint2(mapa(base + parts_off, owner) + (r - first) * p.l[p.layers - 1].out * 4, mapa(parts_bar, owner));
        }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    if (warp == 0 && lane < p.layers) prefetch_map(&p.w[lane]);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                            // every barrier of the cluster is set up
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (!p.ready) spg_grid_wait();                             // the launch behind this one may read weights that are still being made, before its own wait
    spg_grid_trigger();
    const uint32_t last = p.layers - 1;
    // what this CTA does of layer l: tiles (0: nothing) from output o0 on; of a last layer cut along K all outputs
    const auto share = [&](uint32_t l, uint32_t &o0) -> uint32_t {
        const ChainLayer &L = p.l[l];
        o0 = 0;
        if (p.tail && l == last) return me < p.tail;
        o0 = me * L.mt * L.tr;
        if (o0 >= L.out) return 0;
        const uint32_t left = (L.out - o0 + L.tr - 1) / L.tr;
        return left < L.mt ? left : L.mt;
    };
    // its part of K there
    uint32_t tail_k0 = 0, tail_k = 0;
    if (p.tail) tail_k = share(last - 1, tail_k0) * p.l[last - 1].tr;
    // Behind the wait every first look at a parameter would be a miss of the constant cache, one after the other: they are fetched here,
    // under the kernel before.  So are weights, unless that kernel makes them.
    uint32_t seen = p.R ^ p.SA ^ p.SW ^ p.a_slot ^ p.w_slot ^ p.vec4 ^ p.ldx ^ (uint32_t)(uintptr_t)p.x ^ p.exchange_bytes ^ (uint32_t)(uintptr_t)p.scratch ^ p.softmax ^ p.ldy;
    for (uint32_t l = 0; l < p.layers; l++) seen ^= p.l[l].in ^ p.l[l].act ^ p.l[l].covered;
    if (seen == 0x5eed5eedu) __nanosleep(0);                   // (keeps them from being put off)
    if (warp > 0 || !p.early) spg_grid_wait();
    const uint32_t rows = spg_limit_rows(p.rows, p.limit), blocks = (rows + p.R - 1) / p.R;

    // What a role has sent for when a wait gives up: weight tiles; slots of the activation ring, and the parity of their next load
    uint32_t sent_w = 0, sent_a = 0, next_ph = 0;
    bool arrived = false;
    if (warp == 0) {
        // ---- weights: through all layers without a look at the activations -------------------------------------------------
        Ring ring;
        bool stop = false;
        for (uint32_t b = cluster; b < blocks && !stop; b += clusters)
            for (uint32_t l = 0; l < p.layers && !stop; l++) {
                uint32_t o0;
                const bool cut = p.tail && l == last;
                const uint32_t tiles = share(l, o0), tr = p.l[l].tr, kblocks = cut ? (tail_k + TK - 1) / TK : p.l[l].kblocks, k0 = cut ? tail_k0 : 0;
                const CUtensorMap *map = &p.w[l];
                for (uint32_t kb = 0; kb < kblocks && !stop; kb += KG)
                    for (uint32_t t = 0; t < tiles; t++) {
                        mbar_wait_uniform(w_empty + 8 * ring.slot, ring.phase ^ 1u, abort_addr, p.status, 61);
                        stop = __shfl_sync(0xffffffffu, *abort_flag, 0) != 0;
                        if (stop) break;
                        if (elect_one()) {
                            const uint32_t bytes = tr * TK * 2 * WP, at = base + ring.slot * p.w_slot, count = kblocks - kb < KG ? kblocks - kb : KG;
                            mbar_expect_tx(w_full + 8 * ring.slot, count * bytes);
                            for (uint32_t j = 0; j < count; j++) load_planes(at + j * bytes, map, w_full + 8 * ring.slot, (int)(k0 + (kb + j) * TK), (int)(o0 + t * tr));
                        }
                        __syncwarp();
                        sent_w++;
                        ring.next(p.SW);
                    }
            }
    } else if (warp == 1) {
        // ---- products (after a wait that gave up the loops run out: every later wait ends at once) ----------------------------
        Ring ra, rw;
        uint32_t conv_ph = 0, full_ph = 0, own_ph = 0;                     // a slot is filled by the epilogue warps or by copies, each with barriers of their own
        const uint32_t SA = p.SA, SW = p.SW, a_slot = p.a_slot, w_slot = p.w_slot;
        for (uint32_t b = cluster; b < blocks; b += clusters)
            for (uint32_t l = 0; l < p.layers; l++) {
                uint32_t o0;
                const uint32_t tiles = share(l, o0);
                if (!tiles) continue;
                const bool cut = p.tail && l == last;
                const uint32_t n = p.R, stages = cut ? (tail_k + KG * TK - 1) / (KG * TK) : p.l[l].stages, w_lo = p.l[l].tr * (128 >> 4), mains = p.l[l].mains;
                const uint32_t idesc = p.idesc_base | ((AP * n >> 3) << 17), idesc_lo = p.idesc_base | ((n >> 3) << 17);
                const uint32_t run = p.l[l].run, from = l == 0 ? a_conv : a_full, apart = run ? 0u : AP * n;      // (run 0: an accumulator a k-block)
                uint32_t done_stages = 0, first = tmem;                    // of an accumulator, and where it is
                uint32_t ph = l == 0 ? conv_ph : full_ph, steps = cut ? tail_k / 16 : (p.l[l].in + 15) / 16;      // of 16 values that are left
                if (cut) { mbar_wait_uniform(own, own_ph, abort_addr, p.status, 72); own_ph ^= 1u; }
                for (uint32_t st = 0; st < stages; st++) {
                    if (apart) { done_stages = 0; if (st) first += KG * apart; }
                    else if (done_stages == run) { done_stages = 0; first += AP * n; }
                    const uint32_t fresh = done_stages++ ? 1u : 0u, fresh2 = apart ? 0u : 1u;
                    uint32_t d = first;
                    const uint64_t da = smem_desc_sw128(base + a_off + (cut ? st : ra.slot) * a_slot);
                    if (!cut) {
                        mbar_wait_uniform(from + 8 * ra.slot, (ph >> ra.slot) & 1u, abort_addr, p.status, 62);
                        ph ^= 1u << ra.slot;
                    }
                    for (uint32_t t = 0; t < tiles; t++) {
                        const uint64_t dw = smem_desc_sw128(base + rw.slot * w_slot);
                        mbar_wait_uniform(w_full + 8 * rw.slot, rw.phase, abort_addr, p.status, 63);
                        tc_fence_after();
                        if (elect_one()) {
                            // the high and the low terms of the rows lie one behind the other: one product for both, side by side in tensor
                            // memory; then hi*lo of the weights on top of the corrections (lo*lo is below fp32 resolution)
                            const uint32_t a_next = AP * n * (128 >> 4), w_next = WP * w_lo;          // the second k-block of a stage
                            if (steps >= KG * TK / 16 && !apart) {
#pragma unroll
                                for (uint32_t k = 0; k < KG * TK / 16; k++) {
                                    const uint32_t j = k / (TK / 16), i = 2 * (k % (TK / 16));
                                    umma_f16(d, dw + j * w_next + i, da + j * a_next + i, idesc, k ? 1u : fresh);
                                    if (WP > 1) umma_f16(d + n, dw + j * w_next + w_lo + i, da + j * a_next + i, idesc_lo, 1u);
                                }
                            } else {
                                for (uint32_t k = 0; k < (steps < KG * TK / 16 ? steps : KG * TK / 16); k++) {
                                    const uint32_t j = k / (TK / 16), i = 2 * (k % (TK / 16));
                                    umma_f16(d + j * apart, dw + j * w_next + i, da + j * a_next + i, idesc, k == 0 ? fresh : k == TK / 16 ? fresh2 : 1u);
                                    if (WP > 1) umma_f16(d + j * apart + n, dw + j * w_next + w_lo + i, da + j * a_next + i, idesc_lo, 1u);
                                }
                            }
                            umma_commit(w_empty + 8 * rw.slot);
                            if (t + 1 == tiles) {
                                if (!cut) umma_commit(a_empty + 8 * ra.slot);
                                if (st + 1 == stages) umma_commit(done);
                            }
                        }
                        __syncwarp();
                        d += mains * AP * n;
                        rw.next(SW);
                    }
                    steps -= KG * TK / 16;
                    if (!cut) ra.next(SA);
                }
                if (l == 0) conv_ph = ph; else full_ph = ph;
            }
    } else if (warp == 2) {
        // ---- activations of the layers behind the first, as soon as the whole cluster has written them ------------------------
        // (the first layer's tiles come from the epilogue warps; both walk the ring by the same count)
        Ring ring;
        uint32_t e = 0;
        bool stop = false;
        for (uint32_t b = cluster; b < blocks && !stop; b += clusters)
            for (uint32_t l = 0; l < p.layers && !stop; l++) {
                if (p.tail && l == last) continue;
                uint32_t o0;
                const uint32_t tiles = share(l, o0), kblocks = p.l[l].kblocks;
                if (l == 0) { if (tiles) for (uint32_t st = 0; st < p.l[0].stages; st++) ring.next(p.SA); continue; }
                const bool ok = wait_cluster(ready, e & 1u, abort_flag, p.status, 64);
                stop = !__all_sync(0xffffffffu, ok);
                const uint8_t *src = p.scratch + (uint64_t)(2 * cluster + (e & 1u)) * p.exchange_bytes;
                e++;
                if (stop || !tiles) continue;
                fence_async_global();
                const uint32_t bytes = AP * p.R * 128;
                for (uint32_t kb = 0; kb < kblocks; kb += KG, src += KG * bytes) {
                    const uint32_t bar = a_full + 8 * ring.slot, at = base + a_off + ring.slot * p.a_slot;
                    mbar_wait_uniform(a_empty + 8 * ring.slot, ring.phase ^ 1u, abort_addr, p.status, 65);
                    stop = __shfl_sync(0xffffffffu, *abort_flag, 0) != 0;
                    if (stop) break;
                    if (elect_one()) {
                        const uint32_t count = kblocks - kb < KG ? kblocks - kb : KG;
                        mbar_expect_tx(bar, count * bytes);
                        bulk_load(at, src, count * bytes, bar);
                    }
                    __syncwarp();
                    next_ph ^= 1u << ring.slot;
                    sent_a |= 1u << ring.slot;
                    ring.next(p.SA);
                }
            }
    } else if (warp >= 4) {
        // ---- the input's terms, then every layer's outputs --------------------------------------------------------------------
        // (all EPI warps come to every epi_sync: one that has given up goes through the loops without doing anything)
        const uint32_t w = warp - 4;
        Ring ring;
        uint32_t e = 0, finished = 0, round = 0;
        bool ok = true;
        for (uint32_t b = cluster; b < blocks; b += clusters, round++) {
            uint32_t o0;
            uint32_t row0 = 0, row_count = 0;                  // rows that this CTA puts together
            if (me < p.tail) {
                row0 = me * p.R / p.tail; row_count = (me + 1) * p.R / p.tail - row0;
                if (w == 0 && lane == 0) mbar_expect_tx(parts_bar + 8 * (round & 1u), p.tail * row_count * p.l[last].out * 4);
            }
            if (share(0, o0) && ok) {
                if (p.vec4) ok = round_input<T16, AP, true, EPI>(p, b * p.R, rows, p.l[0].in, p.l[0].stages, w, lane, smem + a_off, a_empty, a_conv, ring, abort_flag);
                else ok = round_input<T16, AP, false, EPI>(p, b * p.R, rows, p.l[0].in, p.l[0].stages, w, lane, smem + a_off, a_empty, a_conv, ring, abort_flag);
                for (uint32_t st = 0; st < p.l[0].stages; st++) ring.next(p.SA);
            }
            for (uint32_t l = 0; l < p.layers; l++) {
                const ChainLayer &L = p.l[l];
                Slice s;
                s.q = warp & 3u; s.g = w >> 2; s.lane = lane;
                s.tiles = share(l, o0); s.o = o0 + s.q * 32 + lane; s.tr = L.tr; s.n = p.R; s.mains = L.mains; s.out = L.out; s.act = L.act; s.scale = L.scale;
                s.first = b * p.R; s.end = rows < (b + 1) * p.R ? rows : (b + 1) * p.R;
                s.tmem = tmem + ((s.q * 32) << 16);
                if (p.tail && l == last && s.mains > 1) s.mains = L.run ? ((tail_k + KG * TK - 1) / (KG * TK) + L.run - 1) / L.run : (tail_k + TK - 1) / TK;      // (those of its part of K)
                const bool idle = s.tiles == 0;
#pragma unroll
                for (uint32_t t = 0; t < MAX_MT; t++) {
                    // of the tail's rows: a lane's columns, one every 32
                    const uint32_t o = p.tail && l == last ? t * 32 + lane : s.o + t * s.tr;
                    const bool wanted = p.tail && l == last ? true : t < s.tiles && s.q * 32 + lane < s.tr;
                    s.bias[t] = wanted && o < s.out ? __ldg(L.bias + o) : 0.0f;
                }
                if (!idle) {
                    if (l && !(p.tail && l == last)) for (uint32_t st = 0; st < L.stages; st++) ring.next(p.SA);
                    if (p.impatient) { *abort_flag = 1; atomicCAS(p.status, 0, 70); }
                    ok = ok && !p.impatient && mbar_wait(done, finished & 1u, abort_flag, p.status, 70);
                    finished++;
                } else if (l && !(p.tail && l == last)) ok = ok && wait_cluster(ready, (e - 1) & 1u, abort_flag, p.status, 71);      // (nobody is ahead by two exchanges)
                ok = __all_sync(0xffffffffu, ok);
                // a wait that gave up is known to the whole cluster, which sends nothing on from here
                if (!ok && lane < C) store_remote(mapa(abort_addr, lane), 1);
                tc_fence_after();
                if (!ok || s.q * 32 >= s.tr) s.tiles = 0;
                if (p.tail && l + 1 == last) {
                    if (idle) continue;
                    // (every copy into the activation ring has been used up: its memory holds the CTA's own outputs until they are multiplied)
#define SPG_CHAIN_CALL(A, B) to_operand<A, B, T16, AP, EPI>(s, smem + a_off, o0, tail_k, p.R * 128)
                    SPG_CHAIN_ACTS(s.act, s.mains, SPG_CHAIN_CALL)
#undef SPG_CHAIN_CALL
                    fence_async_smem();
                    tc_fence_before();
                    __syncwarp();
                    if (ok && lane == 0) mbar_arrive(own);
                } else if (l < last) {
                    const uint32_t next_k = p.l[l + 1].kblocks * TK, plane = p.R * 128;
                    uint8_t *next = p.scratch + (uint64_t)(2 * cluster + (e & 1u)) * p.exchange_bytes;
#define SPG_CHAIN_CALL(A, B) to_operand<A, B, T16, AP, EPI>(s, next, 0, next_k, plane)
                    SPG_CHAIN_ACTS(s.act, s.mains, SPG_CHAIN_CALL)
#undef SPG_CHAIN_CALL
                    // columns of the last k-block that no CTA's tiles reach
                    if (ok && me == 0 && L.covered < next_k) {
                        const uint32_t pieces = (next_k - L.covered) >> 3, total = pieces * p.R * AP;
                        for (uint32_t i = threadIdx.x - 128; i < total; i += 32 * EPI) {
                            const uint32_t k = L.covered + i % pieces * 8, r = i / pieces % p.R, a = i / pieces / p.R;
                            *reinterpret_cast<uint4 *>(next + (uint64_t)((k >> 6) * AP + a) * plane + swizzled(r, k & 63u)) = make_uint4(0, 0, 0, 0);
                        }
                    }
                    __syncwarp();
                    fence_async_global();
                    tc_fence_before();
                    epi_sync<EPI>();
                    if (w == 0 && lane < C && !*abort_flag) arrive_release_cluster(mapa(ready, lane));
                    e++;
                } else if (p.tail) {
                    if (idle) continue;
                    const uint32_t part = p.tail_rows * L.out * 4, at = (round & 1u) * p.tail * part;
                    if (s.tiles) to_owners<AP, EPI>(s, owners, at + me * part, 8 * (round & 1u));
                    __syncwarp();
                    ok = ok && wait_cluster(parts_bar + 8 * (round & 1u), (round >> 1) & 1u, abort_flag, p.status, 73);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok && lane < C) store_remote(mapa(abort_addr, lane), 1);
                    __syncwarp();
                    if (b + clusters >= blocks) { cluster_arrive(); arrived = true; }       // nothing goes to another CTA any more
                    const float *parts = reinterpret_cast<const float *>(smem + parts_off + at);
                    if (ok && s.out <= 32) put_together<1, EPI>(p, s.act, s.out, s.scale, s.bias, parts, s.first + row0, row_count, s.end, w, lane);
                    else if (ok) put_together<TAIL_MAX / 32, EPI>(p, s.act, s.out, s.scale, s.bias, parts, s.first + row0, row_count, s.end, w, lane);
                    __syncwarp();
                    // (nobody sends its sums of the next block while a row of this one is still read, here or in a neighbour that waits for them)
                    tc_fence_before();
                    if (b + clusters < blocks) epi_sync<EPI>();
                } else {
#define SPG_CHAIN_CALL(A, B) to_output<A, B, AP, EPI>(p, s)
                    SPG_CHAIN_ACTS(s.act, s.mains, SPG_CHAIN_CALL)
#undef SPG_CHAIN_CALL
                    // The next block's first products take the place of these sums as soon as the first R / 8 warps have rounded a stage of its input:
                    // no warp begins with that before all of them have read theirs.
                    tc_fence_before();
                    __syncwarp();
                    if (b + clusters < blocks) epi_sync<EPI>();
                }
                __syncwarp();
                tc_fence_before();
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (*abort_flag) {
        // shared and tensor memory are given back when nothing writes to them any more
        if (warp == 0) {
            for (uint32_t i = sent_w > p.SW ? sent_w - p.SW : 0; i < sent_w; i++)
                mbar_wait_uniform(w_full + 8 * (i % p.SW), (i / p.SW) & 1u, drain_addr, p.status, 66);
        } else if (warp == 1) {
            if (elect_one()) umma_commit(drain);
            __syncwarp();
            mbar_wait_uniform(drain, 0, drain_addr, p.status, 67);
        } else if (warp == 2) {
            for (uint32_t s = 0; s < p.SA; s++)
                if ((sent_a >> s) & 1u) mbar_wait_uniform(a_full + 8 * s, ((next_ph >> s) & 1u) ^ 1u, drain_addr, p.status, 68);
        }
        __syncwarp();
        __nanosleep(20000);                                    // sums on their way to a neighbour
    }
    tc_fence_before();
    __syncthreads();
    if (!arrived) cluster_arrive();
    cluster_wait();                                            // nobody's shared memory is written any more
    if (warp == 1) { tc_fence_after(); tmem_free(tmem, p.tmem_cols); }
}

using Kernel = void (*)(const ChainParams);
template <uint32_t EPI> Kernel variant_of(int terms, int type16)
{
    if (terms > 2) return spg_chain_kernel<__nv_bfloat16, 2, 2, EPI>;
    if (terms > 1) return type16 == SPGK_T_F16 ? spg_chain_kernel<__half, 2, 1, EPI> : spg_chain_kernel<__nv_bfloat16, 2, 1, EPI>;
    return type16 == SPGK_T_F16 ? spg_chain_kernel<__half, 1, 1, EPI> : spg_chain_kernel<__nv_bfloat16, 1, 1, EPI>;
}
// terms: of an activation, and three where a weight has two as well
Kernel variant(int terms, int type16, uint32_t epi) { return epi == 8 ? variant_of<8>(terms, type16) : variant_of<16>(terms, type16); }

// clusters of 1 to 8 CTAs that the device holds at one CTA an SM (0: none)
struct AtOnce { uint32_t n[MAX_C + 1]; };
int clusters_at_once(int dev, const SpgDeviceProps &dp, AtOnce &out)
{
    static SpgOncePerDevice once;
    static AtOnce known[SPG_MAX_DEVICES];
    const int rc = once.run(dev, [&]() -> int {
        for (uint32_t terms = 0; terms < 6; terms++)
            for (uint32_t epi : { 8u, 16u })
                SPGK_CUDA(cudaFuncSetAttribute(variant((int)(terms >> 1) + 1, terms & 1u ? SPGK_T_F16 : SPGK_T_BF16, epi), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dp.smem_optin));
        for (uint32_t c = 1; c <= MAX_C; c++) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c); cfg.blockDim = dim3(threads_of(16)); cfg.dynamicSmemBytes = 160 * 1024;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr; cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, spg_chain_kernel<__nv_bfloat16, 2, 1, 16>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
            known[dev].n[c] = n > 0 ? (uint32_t)n : 0u;
        }
        return SPGK_OK;
    });
    if (rc == SPGK_OK) out = known[dev];
    return rc;
}

uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// Epilogue warps.  A warp finishes eight rows of 32 outputs in one go: sixteen warps would do every row of a block of 16 twice.  Over 2300
// arrangements of eight nets, time of eight warps against sixteen (median, 5 to 95 %): 16 rows 0.92 (0.84 to 0.96); 32 rows 0.965 (0.93 to
// 1.05), 48 rows 0.985 (0.94 to 1.02) where the epilogues are plain and the last layer is cut, else 1.03 and 1.02; 64 rows 1.07, 96 rows 1.13.
uint32_t epilogue_warps(const spgk_layer *layers, uint32_t count, uint32_t R, bool cut)
{
    if (R <= 16) return 8;
    if (R > 48 || !cut) return 16;
    for (uint32_t l = 0; l + 1 < count; l++) if (layers[l].act == SPG_ACT_TANH || layers[l].act == SPG_ACT_SIGMOID) return 16;
    return 8;
}

// How a net's layers are laid out on clusters of C CTAs with blocks of R rows (false: they do not fit), and the cycles of a block.  steps: products of K = 16
// that an accumulator may add up one after the other, all layers together (0: any number).
// The cycles come from a fit over 2037 arrangements of eight nets (40 to 12000 rows, every size of cluster, one to three products a term):
// 5 to 95 % of them within 11 %, and the arrangement that it calls the fastest 2 % behind the fastest one on average.
struct Layout { uint32_t epi, tr[MAX_LAYERS], mt[MAX_LAYERS], mains[MAX_LAYERS], run[MAX_LAYERS], SA, SW, a_slot, w_slot, tmem_cols, smem, tail, tail_rows, cycles; };
bool lay_out(const spgk_layer *layers, uint32_t count, uint32_t C, uint32_t R, uint32_t a_parts, uint32_t w_parts, bool softmax, bool counted, uint32_t steps,
             size_t smem_max, Layout &o)
{
    const uint32_t n = R * a_parts, rounds = ceil_div(R, 32), out = layers[count - 1].out;
    if (n > 256) return false;                                 // the widest product
    uint32_t cols = 0, inputs[MAX_LAYERS], tr_max = 0, kb_max = 0;
    o.tail = out <= TAIL_MAX;
    o.epi = epilogue_warps(layers, count, R, o.tail != 0);
    if (softmax && !o.tail) return false;
    // a product of K = 16: what it takes to fetch 128 rows of weights (58 cycles), or the tensor pipe's time
    const uint32_t product = (n > 144 ? n / 2 : 58 + n / 10) + (w_parts > 1 ? (R > 144 ? R / 2 : 58 + R / 10) : 0);
    o.cycles = ceil_div(ceil_div(ceil_div(layers[0].in, TK), KG) * (R / 8), 16) * 460;
    for (uint32_t l = 0; l < count; l++) {
        const spgk_layer &L = layers[l];
        const bool cut = o.tail && l + 1 == count;
        const uint32_t share = cut ? L.out : ceil_div(L.out, C), in = cut ? o.mt[l - 1] * o.tr[l - 1] : L.in, kb = ceil_div(in, TK), round = o.tail && l + 2 == count ? 16 : 8;
        o.mt[l] = ceil_div(share, TM);
        o.tr[l] = (ceil_div(share, o.mt[l]) + round - 1) / round * round;
        if (o.mt[l] > MAX_MT) return false;
        if (round == 16) o.tail = ceil_div(L.out, o.mt[l] * o.tr[l]);
        if (o.mt[l] * n > cols) cols = o.mt[l] * n;
        o.mains[l] = 1; o.run[l] = ceil_div(kb, KG); inputs[l] = in;
        if (o.tr[l] > tr_max) tr_max = o.tr[l];
        if (!cut && kb > kb_max) kb_max = kb;
        o.cycles += 2760 + ceil_div(in, 16) * o.mt[l] * product * 11 / 10;
        if (cut) o.cycles += rounds * 390;
        else o.cycles += o.mt[l] * rounds * (L.act == SPG_ACT_TANH || L.act == SPG_ACT_SIGMOID ? 1960 : 1300) + (l ? R * kb * 128 * a_parts / 44 : 0);
    }
    if (cols > 512) return false;
    // two accumulators where tensor memory has room: half as many additions in a row.  (Not where R may be another one in the next call.)
    const auto stages_of = [&](uint32_t l) { return ceil_div(ceil_div(inputs[l], TK), KG); };
    if (cols <= 256 && !counted) {
        for (uint32_t l = 0; l + (o.tail ? 1 : 0) < count; l++) if (stages_of(l) > 1) { o.run[l] = (stages_of(l) + 1) / 2; o.mains[l] = 2; }
        cols *= 2;
    }
    // more where the sums would be too long: for the layer with the longest ones that may have more, a k-block each at the most (run: 0)
    const auto longest = [&](uint32_t l) { const uint32_t all = ceil_div(inputs[l], 16), one = o.run[l] ? o.run[l] * (KG * TK / 16) : TK / 16; return all < one ? all : one; };
    for (;;) {
        uint32_t total = 0, at = count, at_mains = 0, at_run = 0;
        for (uint32_t l = 0; l < count; l++) {
            total += longest(l);
            uint32_t run = o.run[l], mains = o.mains[l];
            if (run == 0 || (at < count && longest(l) <= longest(at))) continue;
            while (mains <= o.mains[l] && run > 1) mains = ceil_div(stages_of(l), --run);
            if (run) run = ceil_div(stages_of(l), mains);       // (as even as they come)
            if (mains <= o.mains[l]) { run = 0; mains = ceil_div(inputs[l], TK); }
            if (mains <= o.mains[l] || mains > MAX_ACC || (!counted && o.mt[l] * n * mains > 512)) continue;
            at = l; at_mains = mains; at_run = run;
        }
        if (!steps || total <= steps) break;
        if (at == count) return false;
        o.mains[at] = at_mains; o.run[at] = at_run;
    }
    for (uint32_t l = 0; l < count; l++) {
        const uint32_t took = o.mt[l] * n * o.mains[l];
        if (took > cols) cols = took;
        if (o.mains[l] > 2) o.cycles += o.mt[l] * rounds * (o.mains[l] - 2) * 250;
    }
    if (cols > 512) return false;
    for (o.tmem_cols = 32; o.tmem_cols < cols; o.tmem_cols <<= 1) { }
    o.a_slot = KG * R * 128 * a_parts; o.w_slot = KG * tr_max * 128 * w_parts;
    o.tail_rows = o.tail ? ceil_div(R, o.tail) : 0;
    if (o.tail) o.cycles += ceil_div(o.tail_rows, 16) * (out <= 32 ? 780 : 1330);
    if (R <= 16) o.cycles -= 2200;                             // (the fit is of sixteen epilogue warps)
    const uint32_t parts = R * 8 + 2 * o.tail * o.tail_rows * out * 4;      // (the table of the rows' owners; sums of two blocks)
    if (parts + BAR_BYTES > smem_max) return false;
    const uint32_t room = (uint32_t)smem_max - BAR_BYTES - parts;
    // two slots of either ring at least; activations take up to half of the room, weights the rest
    uint32_t sa = room / 2 / o.a_slot;
    if (sa > ceil_div(kb_max, KG)) sa = ceil_div(kb_max, KG);
    if (sa < 2) sa = 2;
    if (sa > MAX_RING) sa = MAX_RING;
    if (o.tail && sa < ceil_div(o.mt[count - 2] * o.tr[count - 2], KG * TK)) sa = ceil_div(o.mt[count - 2] * o.tr[count - 2], KG * TK);
    if ((uint64_t)sa * o.a_slot + 2 * o.w_slot > room) return false;
    uint32_t sw = (room - sa * o.a_slot) / o.w_slot;
    if (sw > MAX_RING) sw = MAX_RING;
    o.SA = sa; o.SW = sw;
    o.smem = sw * o.w_slot + sa * o.a_slot + BAR_BYTES + parts;
    // the tensor core reads 128 rows from wherever a tile begins
    const uint32_t reach = sw * o.w_slot - tr_max * 128 + TM * 128;
    if (reach > o.smem) o.smem = reach;
    // Tensor memory is waited for without a bound, in front of the cluster's first barrier: two clusters that each held what the other wants would wait
    // for good.  Two CTAs fit an SM only where both have eight epilogue warps, one term and small rings (three never: 384 threads of 80 registers); with
    // 256 columns each at most they get them.  A CTA of more columns takes an SM to itself (its rings nearly fill the shared memory as it is).
    if (o.tmem_cols > 256) o.smem = (uint32_t)smem_max;
    return o.smem <= smem_max;
}

// Microseconds that the same rows take layer by layer (spg_split16_kernel and spgk_layer_gemm_tc), from a fit over the same nets: 10 to 90 %
// of them within 15 %
float layered_us(const spgk_layer *layers, uint32_t count, uint32_t N, uint32_t sms, uint32_t a_parts, uint32_t w_parts)
{
    const uint32_t passes = a_parts + w_parts - 1, mt = ceil_div(N, 128);
    float us = 0.8f + 6.2f * count;
    for (uint32_t l = 0; l < count; l++) {
        const float in = (float)layers[l].in, out = (float)layers[l].out;
        us += (float)N * (in * out * passes * 0.72e-9f + (in + out) * a_parts * 0.66e-6f) + in * passes * 0.54e-3f;
        us += 3.1f * (ceil_div(mt * ceil_div(layers[l].out, 192), sms) - 1);
    }
    return us;
}

// The cheapest arrangement for a number of rows (0: none): C, R and microseconds.  only: that size of cluster, no more accumulators than `steps` asks for.
float cheapest(const spgk_layer *layers, uint32_t count, uint32_t rows, uint32_t a_parts, uint32_t w_parts, bool softmax, uint32_t only, uint32_t steps, const AtOnce &at,
               const SpgDeviceProps &dp, uint32_t &best_C, uint32_t &best_R)
{
    uint64_t best = ~0ull;
    for (uint32_t C = only ? only : 1; C <= (only ? only : MAX_C); C++) {
        if (!at.n[C]) continue;
        // blocks that fill the clusters once, or a few times
        for (uint32_t waves = 1, tried = 0; waves <= 16 && tried < 3; waves++) {
            const uint32_t R = (ceil_div(rows, at.n[C] * waves) + 15) & ~15u;
            Layout o;
            if (R > MAX_R || !lay_out(layers, count, C, R, a_parts, w_parts, softmax, only != 0, steps, dp.smem_optin, o)) continue;
            tried++;
            const uint32_t blocks = ceil_div(rows, R), busy = (blocks < at.n[C] ? blocks : at.n[C]) * C;
            // (on five eighths of the chip or less the next launch's first blocks get started beside this one's last)
            const uint64_t cost = (uint64_t)o.cycles * ceil_div(blocks, at.n[C]) + (busy * 8 > (uint32_t)dp.sm_count * 5 ? 1000 : 0);
            if (cost < best) { best = cost; best_C = C; best_R = R; }
            if (R == 16) break;
        }
    }
    return best == ~0ull ? 0.0f : 3.2f + (float)best / 1965.0f;
}

// Products that may follow one another in the accumulators, all layers together: as many as in the layer kernels' (what a layer cuts off goes
// through the ones behind it, so it is their sum that counts).  Those add the products of all terms to the same
// one; of 8-bit terms and up to 1024 inputs a product's bits mostly fit the sum, and the second terms' are what is cut off: all are counted
// there, only the first terms' beyond, and of 11-bit terms.  One term of a value loses more than sixteen sums do.
// Not asked (0) of INT4 and INT2 files, whose products are short enough for the sums to hold nearly all of them.
uint32_t steps_allowed(const spgk_layer *layers, uint32_t count, uint32_t N, uint32_t a_parts, uint32_t w_parts, bool softmax, const SpgDeviceProps &dp, int dev)
{
    const int prec = layers[0].precision;
    if (prec == SPG_P_I4 || prec == SPG_P_I2) return 0;
    const uint32_t passes = a_parts + w_parts - 1;
    uint32_t total = 0;
    for (uint32_t l = 0; l < count; l++) {
        uint32_t steps = spg_gemm_steps(&layers[l], N, a_parts, w_parts, softmax && l + 1 == count, dp, dev);
        if (prec == SPG_P_F16 || layers[l].in > 1024) steps /= passes;
        total += passes == 1 && steps < 16 ? 16 : steps;
    }
    return total;
}

thread_local uint32_t tls_arrangement[2] = { 0, 0 };

}  // namespace

extern "C" {

int spgk_chain_plan(const spgk_layer *layers, uint32_t count, uint32_t N, int w_parts, int a_parts, int softmax_fused, spgk_chain *plan)
{
    if (!layers || !plan || w_parts < 1 || a_parts < w_parts || a_parts > 2) { spgk_set_error("spgk_chain_plan", "bad argument"); return SPGK_E_ARG; }
    if (count < 2 || count > MAX_LAYERS || N == 0) return SPGK_E_UNSUPPORTED;
    SpgDeviceProps dp;
    int rc = spg_device_props(&dp), dev = 0;
    if (rc) return rc;
    if (dp.cc != 100) return SPGK_E_UNSUPPORTED;
    SPGK_CUDA(cudaGetDevice(&dev));
    AtOnce at;
    if ((rc = clusters_at_once(dev, dp, at))) return rc;
    // Rows counted on the device: a guess of the count steers the rows of a block, on which no sum depends.  What sums depend on, whether
    // the net comes here and on clusters of which size, goes by 1024 rows whatever the guess.
    const bool counted = spg_tls_rows_limit != nullptr, softmax = softmax_fused != 0;
    const uint32_t a = (uint32_t)a_parts, w = (uint32_t)w_parts, rows = counted && N > 1024 ? 1024 : N;
    uint32_t steps = steps_allowed(layers, count, N, a, w, softmax, dp, dev);
    plan->layered_us = layered_us(layers, count, rows, (uint32_t)dp.sm_count, a, w);
    plan->us = cheapest(layers, count, rows, a, w, softmax, counted ? COUNTED_C : 0, steps, at, dp, plan->C, plan->R);
    if (plan->us == 0.0f && steps) {
        steps = 0;
        plan->layered_us = 0.0f;
        plan->us = cheapest(layers, count, rows, a, w, softmax, counted ? COUNTED_C : 0, steps, at, dp, plan->C, plan->R);
    }
    if (plan->us == 0.0f) return SPGK_E_UNSUPPORTED;
    if (counted) {
        const uint32_t seen = spg_tls_rows_expected ? spg_tls_rows_expected : 1024, likely = seen + 3u * (uint32_t)sqrtf((float)seen);      // (what a selection by chance varies)
        cheapest(layers, count, likely < N ? likely : N, a, w, softmax, COUNTED_C, steps, at, dp, plan->C, plan->R);
    }
    const uint32_t blocks = ceil_div(N, plan->R);
    plan->clusters = blocks < at.n[plan->C] ? blocks : at.n[plan->C];
    uint32_t kb = 0;
    for (uint32_t l = 1; l < count; l++) if (ceil_div(layers[l].in, TK) > kb) kb = ceil_div(layers[l].in, TK);
    plan->exchange_bytes = plan->R * 128 * (uint32_t)a_parts * kb;
    // What clusters * R rows take, whichever of the plans for so many rows or fewer it is: a call of another guess or of fewer rows never wants a larger
    // scratch, which would free the one that a captured call refers to.  (R rows of a block at most, and as many blocks as there are or as are at work.)
    const uint32_t most = 256 / a < MAX_R ? 256 / a : MAX_R;
    uint64_t held = 0;
    for (uint32_t C = 1; C <= MAX_C; C++) if ((!counted || C == COUNTED_C) && (uint64_t)at.n[C] * most > held) held = (uint64_t)at.n[C] * most;
    const uint64_t in_blocks = (uint64_t)N + most;
    plan->scratch_bytes = (in_blocks < held ? in_blocks : held) * 2 * 128 * a * kb;
    return SPGK_OK;
}

int spgk_chain_forward(const spgk_chain *plan, const spgk_layer *layers, uint32_t count, const void *const *w16, const uint32_t *ldw, const uint64_t *w_plane,
                       int w_parts, int type16, int a_parts, const float *x, uint32_t ldx, const uint32_t *x_rows, uint32_t N, float *y, uint32_t ldy,
                       int softmax_fused, int weights_ready, void *scratch, int32_t *status, void *stream)
{
    if (!plan || !layers || count < 2 || count > MAX_LAYERS || !w16 || !ldw || !w_plane || !x || !y || !scratch || !status || ldx < layers[0].in || ldy < layers[count - 1].out ||
        ((uintptr_t)scratch & 15u)) {
        spgk_set_error("spgk_chain_forward", "bad argument");
        return SPGK_E_ARG;
    }
    SpgDeviceProps dp;
    int rc = spg_device_props(&dp);
    if (rc) return rc;
    int dev = 0;
    SPGK_CUDA(cudaGetDevice(&dev));
    Layout o;
    const bool counted = spg_tls_rows_limit != nullptr;
    const auto fits = [&](uint32_t steps) { return lay_out(layers, count, plan->C, plan->R, (uint32_t)a_parts, (uint32_t)w_parts, softmax_fused != 0, counted, steps, dp.smem_optin, o); };
    // (as the plan was made: one that no arrangement with as many accumulators was found for has as few as there is room for)
    if (!fits(steps_allowed(layers, count, N, (uint32_t)a_parts, (uint32_t)w_parts, softmax_fused != 0, dp, dev)) && !fits(0)) { spgk_set_error("spgk_chain_forward", "plan of another net"); return SPGK_E_ARG; }
    ChainParams p{};
    for (uint32_t l = 0; l < count; l++) {
        const spgk_layer &L = layers[l];
        ChainLayer &c = p.l[l];
        c.bias = L.bias; c.scale = L.w_scale; c.act = L.act == SPG_ACT_SOFTMAX ? SPG_ACT_NONE : L.act;
        c.in = L.in; c.out = L.out; c.kblocks = ceil_div(L.in, TK); c.stages = ceil_div(c.kblocks, KG);
        c.tr = o.tr[l]; c.mt = o.mt[l];
        c.mains = o.mains[l]; c.run = o.run[l];
        c.covered = ceil_div(L.out, c.tr) * c.tr;
        if ((rc = spg_gemm_map(&p.w[l], w16[l], type16, L.in, L.out, ldw[l], w_plane[l], w_parts, c.tr, (uint32_t)w_parts))) return rc;
    }
    p.layers = count; p.R = plan->R; p.C = plan->C; p.tail = o.tail; p.tail_rows = o.tail_rows;
    p.SA = o.SA; p.SW = o.SW; p.a_slot = o.a_slot; p.w_slot = o.w_slot; p.tmem_cols = o.tmem_cols;
    p.idesc_base = idesc_f16((uint32_t)type16, (uint32_t)type16, 0);
    p.x = x; p.ldx = ldx; p.vec4 = ((ldx | layers[0].in) & 3u) == 0 && ((uintptr_t)x & 15u) == 0; p.x_rows = x_rows;
    p.y = y; p.ldy = ldy; p.y_rows = spg_tls_out_rows;
    p.softmax = softmax_fused ? 1 : 0;
    if (softmax_fused && spg_tls_margin_idx) { p.margin_theta = spg_tls_margin_theta; p.margin_idx = spg_tls_margin_idx; p.margin_count = spg_tls_margin_count; }
    p.scratch = (uint8_t *)scratch; p.exchange_bytes = plan->exchange_bytes;
    p.rows = N; p.limit = spg_tls_rows_limit;
    p.ready = weights_ready;
    p.early = weights_ready && !p.limit;
    p.impatient = spg_gemm_impatient() ? 1 : 0;
    p.status = status;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan->clusters * plan->C); cfg.blockDim = dim3(threads_of(o.epi)); cfg.dynamicSmemBytes = o.smem; cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = plan->C; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    SPGK_CUDA(cudaLaunchKernelEx(&cfg, variant(w_parts > 1 ? 3 : a_parts, type16, o.epi), p));
    tls_arrangement[0] = plan->C; tls_arrangement[1] = plan->R;
    return spgk_check_launch("spg_chain_kernel");
}

void spgk_chain_arrangement(uint32_t out[2]) { out[0] = tls_arrangement[0]; out[1] = tls_arrangement[1]; }

}  // extern "C"
