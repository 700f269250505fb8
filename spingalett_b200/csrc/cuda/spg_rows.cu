// spg_rows.cu -- one to eight rows through a small net, any precision, any width, any alignment.
//
//   y[n][j] = act(bias[j] + w_scale * sum_k q[j][k] * x[n][k])
//
// A net of a few megabytes lives in L2 and a forward pass of a sample is a chain of latencies: what a layer costs is a launch,
// the way to its input and a sum.  A warp takes an output.  Its weights depend on nothing, so the first 1024 of its row are in
// registers, decoded, before the layer before it has ended (programmatic dependent launch); then come the input (8 neighbouring
// values a lane, all loads of a round in flight), the products, four of them added in fp32 and the fours in 64 bits, and a shuffle
// tree.  (Every product in 64 bits: as accurate as the last rounding allows, and 2 to 4 us slower from six rows on, a conversion
// runs at 14 a cycle and SM.)  A warp takes 1.2 to 1.7 us for 1024 elements of a row, so rows of more than 2048 are shared by up to eight
// warps: 65536-64-10 INT8 at one row 110 -> 18 us, 4096-1000 12.9 -> 8.7.  Rows of at most 256 have a kernel that has no more than those in
// flight (30 to 61 registers instead of 56 to 70): 250-250-250-250-10 in 0.9 of the time.
//
// What bounds it: 3 us a layer of launch, two L2 latencies and the tree; beyond four rows the loads of the inputs.  Before (the
// weight-streaming GEMV, made to keep HBM busy, or the general kernel where rows are no multiple of 16 bytes) and now, us a call:
// 784-512-1000-10 at one row fp32 31.6 -> 8.0, INT8 46 -> 7.8, INT4 26 -> 7.9; at eight rows fp32 90 -> 12, INT4 118 -> 10.4;
// 301-777-333-129-37 fp32 at one row 22.6 -> 12 to 17, at eight 103 -> 19; 1024-1024-1024-1024-16 BF16 35 -> 12.5 and 117 -> 23.
// forward() of one sample 57 -> 36, and 22 since its launches are replayed as a graph and the answer is taken as it arrives.  Error against 64 bits 5e-8 to 2e-7 (before:
// 1e-7 to 5e-6).  An input that travels as a parameter of the first launch instead of through the fetch kernel: level.
//
// Reference: forward's layer step, Src/Spingalett.Network.c:218-247; decode of Src/Spingalett.Serialize.c:222-294.
#include "spg_common.cuh"
#include <type_traits>

namespace {

constexpr uint32_t GROUP = 8, TURN = 32 * GROUP, SPAN = 4 * TURN;          // neighbours a lane takes, elements that a warp takes side by side, and that it has in flight
constexpr uint32_t LONG_ROW = 2 * SPAN;                                    // inputs beyond which several warps share an output
constexpr uint32_t LAST_WARPS = 32, LAST_MAX = 128;                        // the layer whose row softmax is finished in the CTA

struct RowsParams {
    const void *w; const float *bias; double scale; uint32_t in, out; int act;
    const float *x; uint32_t ldx; float *y; uint32_t ldy; uint32_t N;
    float *copy;                           // a second place for the outputs of row 0 (page-locked host memory), or null
    uint32_t vec_w, vec_x;                 // groups of eight weights / inputs lie on their own alignment
    uint32_t parts;                        // warps that share an output: 1, 2, 4 or 8
};

// Integer weights are multiplied before their scale, which a large input times a weight of 128 would not survive in fp32: they are taken as
// multiples of 2^-9, 2^-5 and 2^-3 (INT8, INT4, INT2), so that four products add up to no more than the largest input; the scale makes up for it.
template <int PREC> constexpr int UNIT = PREC == SPG_P_I8 ? 9 : PREC == SPG_P_I4 ? 5 : PREC == SPG_P_I2 ? 3 : 0;
template <int PREC> constexpr float ONE = 1.0f / (float)(1 << UNIT<PREC>);

// weight e of the matrix in those units
template <int PREC> __device__ __forceinline__ float decode1(const void *w, uint64_t e)
{
    if constexpr (PREC == SPG_P_I4)
        return (float)(int)((uint32_t)reinterpret_cast<const uint8_t *>(w)[e >> 1] << (28 - 4 * (uint32_t)(e & 1)) & 0xF0000000u) * (ONE<PREC> / (1u << 28));
    else if constexpr (PREC == SPG_P_I2)
        return (float)(int)((uint32_t)reinterpret_cast<const uint8_t *>(w)[e >> 2] << (30 - 2 * (uint32_t)(e & 3)) & 0xC0000000u) * (ONE<PREC> / (1u << 30));
    else return spg_decode_elem(w, e, PREC) * ONE<PREC>;
}

// the weights e .. e + 7
template <int PREC> __device__ __forceinline__ void decode8(const void *w, uint64_t e, float (&q)[8])
{
    if constexpr (PREC == SPG_P_F32) {
        const float4 *p = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(w) + e);
        const float4 a = __ldg(p), b = __ldg(p + 1);
        q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w; q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
    } else if constexpr (PREC == SPG_P_F16 || PREC == SPG_P_BF16) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(w) + e));
        const uint32_t u[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t h = u[i >> 1] >> ((i & 1) * 16) & 0xFFFFu;
            q[i] = PREC == SPG_P_F16 ? __half2float(__ushort_as_half((unsigned short)h)) : __uint_as_float(h << 16);
        }
    } else if constexpr (PREC == SPG_P_I8) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const int8_t *>(w) + e));
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = (float)((int)((i < 4 ? v.x : v.y) << (24 - 8 * (i & 3))) >> 24) * ONE<PREC>;
    } else if constexpr (PREC == SPG_P_I4) {
        const uint32_t v = __ldg(reinterpret_cast<const uint32_t *>(reinterpret_cast<const uint8_t *>(w) + (e >> 1)));
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = (float)((int)(v << (28 - 4 * i)) >> 28) * ONE<PREC>;
    } else {
        const uint32_t v = __ldg(reinterpret_cast<const uint16_t *>(reinterpret_cast<const uint8_t *>(w) + (e >> 2)));
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = (float)((int)(v << (30 - 2 * i)) >> 30) * ONE<PREC>;
    }
}

// Output j for rows n0 .. n0 + NB - 1 (rows from N on read as the last one): the sums of every parts-th span from the part-th on, in every
// lane.  `wait`: the input is what the launch before this one writes, and nobody has waited for it yet.
template <int PREC, int NB, uint32_t TURNS = SPAN / TURN>
__device__ __forceinline__ void dot(const RowsParams &p, uint32_t j, uint32_t n0, uint32_t part, uint32_t parts, bool wait, uint32_t lane, double (&sum)[NB])
{
    const uint64_t row = (uint64_t)j * p.in;
    double acc[NB][2];
#pragma unroll
    for (int b = 0; b < NB; b++) acc[b][0] = acc[b][1] = 0.0;
#pragma unroll 1
    for (uint32_t k0 = part * (TURNS * TURN); k0 < p.in; k0 += parts * (TURNS * TURN)) {
        float q[TURNS][GROUP];
#pragma unroll
        for (uint32_t u = 0; u < TURNS; u++) {
            const uint32_t k = k0 + u * TURN + lane * GROUP;
            if (p.vec_w && k < p.in) decode8<PREC>(p.w, row + k, q[u]);        // (then `in` is a multiple of eight)
            else {
#pragma unroll
                for (uint32_t i = 0; i < GROUP; i++) q[u][i] = k + i < p.in ? decode1<PREC>(p.w, row + k + i) : 0.0f;
            }
        }
        if (wait) { spg_grid_wait(); wait = false; }
#pragma unroll
        for (uint32_t u = 0; u < TURNS; u++) {
            const uint32_t k = k0 + u * TURN + lane * GROUP;
            if (k0 + u * TURN >= p.in) break;                             // (the same for the whole warp)
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const float *x = p.x + (uint64_t)min(n0 + b, p.N - 1) * p.ldx + k;
                float v[GROUP];
                if (p.vec_x && k + GROUP <= p.in) {
                    const float4 lo = *reinterpret_cast<const float4 *>(x), hi = *reinterpret_cast<const float4 *>(x + 4);
                    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
                } else {
#pragma unroll
                    for (uint32_t i = 0; i < GROUP; i++) v[i] = k + i < p.in ? x[i] : 0.0f;
                }
#pragma unroll
                for (uint32_t h = 0; h < 2; h++) {
                    float four = q[u][4 * h] * v[4 * h];
#pragma unroll
                    for (uint32_t i = 4 * h + 1; i < 4 * h + 4; i++) four = fmaf(q[u][i], v[i], four);
                    acc[b][h] += (double)four;
                }
            }
        }
    }
#pragma unroll
    for (int b = 0; b < NB; b++) {
        sum[b] = acc[b][0] + acc[b][1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum[b] += __shfl_xor_sync(0xffffffffu, sum[b], o);
    }
}

__device__ __forceinline__ float value(const RowsParams &p, uint32_t j, double sum) { return (float)(sum * p.scale + (double)p.bias[j]); }

// FORM: 0 rows of any length, a warp an output; 1 rows of at most 256; 2 several warps an output
template <int PREC, int NB, int FORM>
__global__ void __launch_bounds__(256)
spg_rows_kernel(const RowsParams p)
{
    constexpr bool LONG = FORM == 2;
    __shared__ double shared[LONG ? 8 : 1][NB];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, parts = LONG ? p.parts : 1u, j = (blockIdx.x * 8 + warp) / parts, part = warp % parts;
    spg_grid_trigger();
    if (!LONG && j >= p.out) return;
    double sum[NB];
    const uint32_t n0 = blockIdx.y * NB;
    dot<PREC, NB, FORM == 1 ? 1 : SPAN / TURN>(p, LONG ? min(j, p.out - 1) : j, n0, part, parts, true, lane, sum);
    double mine = sum[0];
#pragma unroll
    for (int b = 1; b < NB; b++) if (lane == (uint32_t)b) mine = sum[b];
    if (LONG) {
        if (lane < NB) shared[warp][lane] = mine;
        __syncthreads();
        if (part || j >= p.out) return;
        if (lane < NB) for (uint32_t i = 1; i < parts; i++) mine += shared[warp + i][lane];
    }
    if (lane < NB && n0 + lane < p.N) {
        const float y = spg_activate(value(p, j, mine), p.act);
        p.y[(uint64_t)(n0 + lane) * p.ldy + j] = y;
        if (p.copy && n0 + lane == 0) p.copy[j] = y;
    }
}

// The last layer with a softmax of at most LAST_MAX outputs: one CTA a row, its warps take the outputs in turn; formulas of
// spg_softmax_rows_kernel.
template <int PREC>
__global__ void __launch_bounds__(32 * LAST_WARPS)
spg_rows_softmax_kernel(const RowsParams p)
{
    __shared__ float z[LAST_MAX];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n = blockIdx.x;
    spg_grid_trigger();
    for (uint32_t j = warp; j < p.out; j += LAST_WARPS) {
        double sum[1];
        dot<PREC, 1>(p, j, n, 0, 1, j == warp, lane, sum);
        if (lane == 0) z[j] = value(p, j, sum[0]);
    }
    __syncthreads();
    if (warp) return;
    spg_grid_wait();                       // (an output that no warp had: this row is written after the layer before has ended all the same)
    float mx = -FLT_MAX, sum = 0.0f;
    for (uint32_t j = lane; j < p.out; j += 32) if (z[j] > mx) mx = z[j];
    mx = spg_warp_max(mx);
    for (uint32_t j = lane; j < p.out; j += 32) { z[j] = expf(z[j] - mx); sum += z[j]; }
    sum = spg_warp_sum(sum);
    const float inv = sum > 0.0f ? 1.0f / sum : 1.0f;
    for (uint32_t j = lane; j < p.out; j += 32) {
        p.y[(uint64_t)n * p.ldy + j] = z[j] * inv;
        if (p.copy && n == 0) p.copy[j] = z[j] * inv;
    }
}

// a sample from page-locked host memory
__global__ void __launch_bounds__(256)
spg_rows_fetch_kernel(const float *src, float *dst, uint32_t count)
{
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    spg_grid_trigger();
    const float v = i < count ? src[i] : 0.0f;
    spg_grid_wait();                       // what is in dst may still be read
    if (i < count) dst[i] = v;
}

template <int PREC> cudaError_t launch(RowsParams p, bool softmax, cudaStream_t s)
{
    p.scale *= (double)(1 << UNIT<PREC>);
    if (softmax) return spg_launch_chained(spg_rows_softmax_kernel<PREC>, dim3(p.N), dim3(32 * LAST_WARPS), 0, s, p);
    // one row of the batch a warp up to four rows, two beyond (weights decoded once for both): 784-512-1000-10 at 4 rows 9.7 against 11.5 us,
    // at 6 rows 12.9 against 10.9
    const uint32_t each = 8 / p.parts, ctas = (p.out + each - 1) / each;
    const auto kernel = p.N <= 4 ? (p.parts > 1 ? spg_rows_kernel<PREC, 1, 2> : p.in <= TURN ? spg_rows_kernel<PREC, 1, 1> : spg_rows_kernel<PREC, 1, 0>)
                                 : (p.parts > 1 ? spg_rows_kernel<PREC, 2, 2> : p.in <= TURN ? spg_rows_kernel<PREC, 2, 1> : spg_rows_kernel<PREC, 2, 0>);
    return spg_launch_chained(kernel, dim3(ctas, p.N <= 4 ? p.N : (p.N + 1) / 2), dim3(256), 0, s, p);
}

}  // namespace

// calls f with the layer's precision as a constant
template <typename F> static cudaError_t with_precision(int precision, F f)
{
    switch (precision) {
        case SPG_P_F32:  return f(std::integral_constant<int, SPG_P_F32>());
        case SPG_P_F16:  return f(std::integral_constant<int, SPG_P_F16>());
        case SPG_P_BF16: return f(std::integral_constant<int, SPG_P_BF16>());
        case SPG_P_I8:   return f(std::integral_constant<int, SPG_P_I8>());
        case SPG_P_I4:   return f(std::integral_constant<int, SPG_P_I4>());
        default:         return f(std::integral_constant<int, SPG_P_I2>());
    }
}

// Whether the softmax is finished in one CTA a row: while a warp has at most three of the outputs and four spans.  Its time less that of all
// CTAs' products and a softmax kernel, us, by spans of a row x outputs a warp: 2 x 1 -3.9, 1 x 2 -1.4, 1 x 3 -0.9, 4 x 1 -0.1, 2 x 2 0.9, 1 x 4 1.8,
// 2 x 4 8.4, 8 x 1 7.6; for a sample, where it saves two copies, -7.7, -4.4, 1.2, -6.0, -5.6, 2.0, 1.8, 4.4.
static bool softmax_in_cta(const spgk_layer *L)
{
    const uint32_t each = (L->out + LAST_WARPS - 1) / LAST_WARPS, spans = (L->in - 1) / SPAN + 1;
    return L->act == SPG_ACT_SOFTMAX && L->out <= LAST_MAX && each <= 3 && (uint64_t)each * spans <= 4;
}

static int rows_chain(const spgk_layer *layers, uint32_t count, const float *x, uint32_t ldx, float *const *ys, float *const *copies, uint32_t N, void *stream)
{
    SpgDeviceProps dp;
    const int prc = spg_device_props(&dp);
    if (prc) return prc;
    for (uint32_t l = 0; l < count; l++) {
        const spgk_layer *L = &layers[l];
        const bool softmax = L->act == SPG_ACT_SOFTMAX, fused = softmax_in_cta(L);
        RowsParams p;
        p.w = L->w; p.bias = L->bias; p.scale = L->w_scale; p.in = L->in; p.out = L->out; p.act = softmax ? SPG_ACT_NONE : L->act;
        p.x = x; p.ldx = ldx; p.y = ys[l]; p.ldy = L->out; p.N = N; p.copy = copies ? copies[l] : nullptr;
        p.vec_w = (L->in % 8 == 0 && ((uintptr_t)L->w & 15u) == 0) ? 1u : 0u;
        // (as long as there are warps to spare: 4096-1000 FP16 at four rows 14.9 us with a warp an output, 19.0 with four)
        p.parts = 1;
        for (const uint64_t warps = (uint64_t)L->out * (N <= 4 ? N : (N + 1) / 2); L->in > LONG_ROW && p.parts < 8 && p.parts * SPAN < L->in && 2 * p.parts * warps <= 32ull * dp.sm_count;) p.parts *= 2;
        p.vec_x = (((uintptr_t)x | ((uintptr_t)ldx * 4)) & 15u) == 0 ? 1u : 0u;
        SPGK_CUDA(with_precision(L->precision, [&](auto prec) { return launch<prec.value>(p, fused, (cudaStream_t)stream); }));
        int rc = spgk_check_launch("spg_rows_kernel");
        if (rc) return rc;
        if (softmax && !fused && (rc = spgk_softmax_rows(ys[l], L->out, N, L->out, stream))) return rc;
        x = ys[l]; ldx = L->out;
    }
    return SPGK_OK;
}

static bool layers_ok(const spgk_layer *layers, uint32_t count)
{
    for (uint32_t l = 0; l < count; l++) {
        const spgk_layer *L = &layers[l];
        if (!L->w || !L->bias || L->in == 0 || L->out == 0 || (unsigned)L->precision >= SPG_P_COUNT) return false;
    }
    return true;
}

extern "C" int spgk_rows_forward(const spgk_layer *layers, uint32_t count, const float *x, uint32_t ldx, float *const *ys, uint32_t N, void *stream)
{
    if (!layers || !x || !ys || N == 0 || N > SPGK_ROWS_MAX_BATCH || !layers_ok(layers, count)) { spgk_set_error("spgk_rows_forward", "bad argument"); return SPGK_E_ARG; }
    for (uint32_t l = 0; l < count; l++) if (!ys[l]) { spgk_set_error("spgk_rows_forward", "bad argument"); return SPGK_E_ARG; }
    return rows_chain(layers, count, x, ldx, ys, nullptr, N, stream);
}

extern "C" int spgk_rows_sample(const spgk_layer *layers, uint32_t count, float *host, float *dev, void *stream)
{
    if (!layers || !host || !dev || count == 0 || count > SPGK_ROWS_MAX_LAYERS || !layers_ok(layers, count)) { spgk_set_error("spgk_rows_sample", "bad argument"); return SPGK_E_ARG; }
    float *ys[SPGK_ROWS_MAX_LAYERS], *copies[SPGK_ROWS_MAX_LAYERS];
    uint64_t at = layers[0].in;
    for (uint32_t l = 0; l < count; l++) {
        if (layers[l].act == SPG_ACT_SOFTMAX && !softmax_in_cta(&layers[l])) return SPGK_E_UNSUPPORTED;
        ys[l] = dev + at; copies[l] = host + at;
        at += layers[l].out;
    }
    // The last outputs go to the host alone: a caller that has seen every output may go on before the stream is idle, and nothing in device memory is
    // written any more then (the layers before have been read by the one behind them).
    ys[count - 1] = copies[count - 1]; copies[count - 1] = nullptr;
    SPGK_CUDA(spg_launch_chained(spg_rows_fetch_kernel, dim3((layers[0].in + 255) / 256), dim3(256), 0, (cudaStream_t)stream, host, dev, layers[0].in));
    const int rc = spgk_check_launch("spg_rows_fetch_kernel");
    return rc ? rc : rows_chain(layers, count, dev, layers[0].in, ys, copies, 1, stream);
}
