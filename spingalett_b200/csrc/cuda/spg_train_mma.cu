// spg_train_mma.cu -- the products of a training step with fewer than 148 64 x 64 tiles on the tensor cores, with fp32-level error, and the
// output end of a step.
//
// An fp32 value x is split into hi = tf32(x) and lo = tf32(x - hi); a*b is formed as a_lo*b_hi + a_hi*b_lo + a_hi*b_hi by three
// mma.m16n8k8.tf32 with fp32 accumulation (the dropped a_lo*b_lo term is below 2^-22 of the product).
//
// A 32 x 32 tile of the result is a CTA of four warps (eight when there are at most 32 tiles) that share the k range, 16 at a time in turn.
// A warp has a ring of its own for its slices of both operands (cp.async, operands as they lie in memory) and a partial sum of the whole
// tile, so warps never wait for one another before the end, and a fragment, once split, is used for two or four products.  The partial sums
// are added in warp order: results do not depend on timing, nor on where a product is launched from.  A trained network hangs on their
// last bit (ReLU corners and Adam's quotient make of 1e-7 in a gradient 1e-3 in the weights within twenty steps), so slices, their order
// and the order of the three products are kept as they are.
//
// What bounds it: issue and latency.  An mma.m16n8k8 takes 8 cycles of a warp scheduler and every other instruction one to two more on top
// (24 products alone 194 cycles, beside 16 conversions 218, beside 48 additions and masks 245); a slice of 16 is 48 products, 384 cycles,
// and takes 620 where warps fill in for one another, 790 for a warp alone; 2000 cycles go until the first slice is there, 1500 into sums,
// activation and stores.  tcgen05 would lift the first bound, but adds in another order and wants both terms of both operands written back
// to shared memory.  One launch behind another, before (register-staged tiles, one barrier of the CTA a slice) and now: 512 x 784 forward,
// 256 rows 16.5 -> 10.0 us, 1000 x 512 forward 18.0 -> 10.2, 512 x 1000 delta 16.4 -> 12.1, 1000 x 512 gradient 14.4 -> 10.7; the step of
// the 784-512-1000-10 net 98 -> 68 us (65 to 68 with the gradients of its first two layers in one launch, 15 us instead of 17).  Three and four slots: level alone, 4 us slower in the step.  A ring that the whole CTA shares, one
// barrier a stage: 0.5 to 2 us slower each, the warps then load, split and multiply in step.
#include "spg_train.cuh"

namespace {

constexpr uint32_t TILE = 32, SLICE = 16, SLOTS = 2;
constexpr uint32_t PITCH_K = SLICE + 4;      // operand kept as [row][k]: the eight rows of a block read lie on eight different 16-byte columns
constexpr uint32_t PITCH_N = TILE + 8;       // operand kept as [k][row]: lanes t, g of a fragment read bank 8t + g
constexpr uint32_t PITCH_R = TILE + 8;       // partial sums
constexpr uint32_t OPERAND = TILE * PITCH_K;                                    // floats of an operand's slice, either way
static_assert(OPERAND == SLICE * PITCH_N, "both layouts take the same room");

constexpr uint32_t ring_floats(int warps) { return warps * SLOTS * 2 * OPERAND; }
constexpr uint32_t sum_floats(int warps) { return warps * (TILE * PITCH_R + TILE); }       // partial tiles, then partial column sums

__device__ __forceinline__ uint32_t smem_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// V floats of which the first `left` are read and the others are zero
template <int V> __device__ __forceinline__ void copy_async(uint32_t dst, const float *src, uint32_t left)
{
    if constexpr (V == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(left * 4) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(dst), "l"(src), "r"(left * 4) : "memory");
}
template <int V> __device__ __forceinline__ uint32_t left_of(uint32_t first, uint32_t limit) { return first >= limit ? 0u : min((uint32_t)V, limit - first); }

// One warp's slice k0 .. k0+15 of rows r0 .. r0+31 of an operand.  Rows beyond the last are read as the last one (their results go nowhere),
// k beyond the last as zero; nothing outside the matrix is touched.
template <bool K_MAJOR, int V>
__device__ __forceinline__ void load_slice(uint32_t dst, const float *base, uint32_t ld, uint32_t r0, uint32_t rows, uint32_t k0, uint32_t K, uint32_t lane)
{
    if constexpr (K_MAJOR) {
        constexpr uint32_t pieces = SLICE / V, step = 32 / pieces;
        const uint32_t k = lane % pieces * V, row = lane / pieces, left = left_of<V>(k0 + k, K);
        const float *src = base + (left ? k0 + k : 0u);
#pragma unroll
        for (uint32_t u = 0; u < TILE; u += step)
            copy_async<V>(dst + ((row + u) * PITCH_K + k) * 4, src + (uint64_t)min(r0 + row + u, rows - 1) * ld, left);
    } else {
        constexpr uint32_t pieces = TILE / V, step = 32 / pieces;
        const uint32_t r = lane % pieces * V, k = lane / pieces, left = left_of<V>(r0 + r, rows);
        const float *src = base + (left ? r0 + r : 0u);
#pragma unroll
        for (uint32_t u = 0; u < SLICE; u += step)
            copy_async<V>(dst + ((k + u) * PITCH_N + r) * 4, src + (uint64_t)min(k0 + k + u, K - 1) * ld, k0 + k + u < K ? left : 0u);
    }
}

// hi = x rounded to 11 significant bits (to nearest, ties away), lo = the rest rounded alike.  The first by the conversion unit, the second
// by adding half a unit and cutting: each unit alone would take as long as the products.
__device__ __forceinline__ void split(float x, uint32_t &hi, uint32_t &lo)
{
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    lo = (__float_as_uint(x - __uint_as_float(hi)) + 0x1000u) & 0xFFFFE000u;
}

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// four 8 x 4 blocks of fp32 words: lane l of block q gets word l%4 of the row that lane 8q + l/4 points at
__device__ __forceinline__ void load_blocks(float (&v)[4], uint32_t row_address)
{
    uint32_t r[4];
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(row_address) : "memory");
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = __uint_as_float(r[i]);
}

template <int MODE, int V, int WARPS>
__device__ __forceinline__ void product_tile(const SpgTrainProduct &p, uint32_t tile, float *sm)
{
    constexpr bool a_k = MODE != TRAIN_GRAD, b_k = MODE == TRAIN_FWD;          // stored [M][K] / [N][K]; otherwise [K][M] / [K][N]
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t tiles_n = (p.N + TILE - 1) / TILE, m0 = tile / tiles_n * TILE, n0 = tile % tiles_n * TILE;
    const uint32_t slices = (p.K + SLICE - 1) / SLICE;
    const bool sums = MODE == TRAIN_GRAD && p.colsum && n0 == 0;
    // the outputs that this thread finishes, W neighbours of a row, and what stands beside them: asked for before the products
    constexpr uint32_t W = TILE * TILE / (WARPS * 32);
    const uint32_t mr = threadIdx.x / (TILE / W), nr = threadIdx.x % (TILE / W) * W, m = m0 + mr, n = n0 + nr;
    float beside[W];
    float *const ring = sm + warp * SLOTS * 2 * OPERAND;

    const auto load = [&](uint32_t s, uint32_t slot) {
        if (s >= slices) return;
        const uint32_t dst = smem_address(ring + slot * 2 * OPERAND);
        load_slice<b_k, V>(dst + OPERAND * 4, p.B, p.ldb, n0, p.N, s * SLICE, p.K, lane);
        load_slice<a_k, V>(dst, p.A, p.lda, m0, p.M, s * SLICE, p.K, lane);
    };

    float acc[2][4][4], bs = 0.0f;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0f;

#pragma unroll
    for (uint32_t j = 0; j < W; j++) {
        if (MODE == TRAIN_FWD) beside[j] = n + j < p.N ? p.bias[n + j] : 0.0f;
        else if (MODE == TRAIN_DELTA) beside[j] = m < p.M && n + j < p.N ? p.aux[(uint64_t)m * p.ldaux + n + j] : 0.0f;
    }
#pragma unroll 1
    for (uint32_t c = 0; c + 1 < SLOTS; c++) {
        load(warp + c * WARPS, c);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint32_t slot = 0, next = SLOTS - 1;
#pragma unroll 1
    for (uint32_t s = warp; s < slices; s += WARPS) {
        load(s + (SLOTS - 1) * WARPS, next);                    // (every lane has left that slot: the barrier at the end of the round)
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group %0;" :: "n"(SLOTS - 1) : "memory");
        __syncwarp();                                           // every lane's copies of this slice are there
        const float *As = ring + slot * 2 * OPERAND, *Bs = As + OPERAND;
#pragma unroll
        for (uint32_t k = 0; k < SLICE; k += 8) {
            float av[2][4], bv[4][2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (a_k) load_blocks(av[i], smem_address(As + (i * 16 + (lane & 15u)) * PITCH_K + k + (lane >> 4) * 4));
                else {
                    const float *q = As + (k + t) * PITCH_N + i * 16 + g;
                    av[i][0] = q[0]; av[i][1] = q[8]; av[i][2] = q[4 * PITCH_N]; av[i][3] = q[4 * PITCH_N + 8];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                if (b_k) {
                    float v[4];
                    load_blocks(v, smem_address(Bs + (j * 8 + (lane & 7u) + (lane >> 4) * 8) * PITCH_K + k + (lane >> 3 & 1u) * 4));
                    bv[j][0] = v[0]; bv[j][1] = v[1]; bv[j + 1][0] = v[2]; bv[j + 1][1] = v[3];
                } else {
                    const float *q = Bs + (k + t) * PITCH_N + j * 8 + g;
                    bv[j][0] = q[0]; bv[j][1] = q[4 * PITCH_N]; bv[j + 1][0] = q[8]; bv[j + 1][1] = q[4 * PITCH_N + 8];
                }
            }
            uint32_t ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) split(av[i][q], ah[i][q], al[i][q]);
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int q = 0; q < 2; q++) split(bv[j][q], bh[j][q], bl[j][q]);
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma(acc[i][j], al[i], bh[j]);
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma(acc[i][j], ah[i], bl[j]);
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma(acc[i][j], ah[i], bh[j]);
        }
        if (sums) {
#pragma unroll
            for (uint32_t k = 0; k < SLICE; k++) bs += As[k * PITCH_N + lane];
        }
        __syncwarp();
        next = slot;
        slot = slot + 1 == SLOTS ? 0 : slot + 1;
    }
    __syncthreads();                                            // the partial sums take the place of the rings (no copy is under way any more)
    float *mine = sm + warp * TILE * PITCH_R, *csum = sm + WARPS * TILE * PITCH_R;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float *q = mine + (i * 16 + g) * PITCH_R + j * 8 + 2 * t;
            *reinterpret_cast<float2 *>(q) = make_float2(acc[i][j][0], acc[i][j][1]);
            *reinterpret_cast<float2 *>(q + 8 * PITCH_R) = make_float2(acc[i][j][2], acc[i][j][3]);
        }
    if (sums) csum[warp * TILE + lane] = bs;
    __syncthreads();
    if (sums && threadIdx.x < TILE && m0 + threadIdx.x < p.M) {
        float s = csum[threadIdx.x];
#pragma unroll
        for (uint32_t w = 1; w < WARPS; w++) s += csum[w * TILE + threadIdx.x];
        p.colsum[m0 + threadIdx.x] = p.alpha * s;
    }
    if (m >= p.M || n >= p.N) return;
    float v[W];
#pragma unroll
    for (uint32_t j = 0; j < W; j++) v[j] = sm[mr * PITCH_R + nr + j];
#pragma unroll
    for (uint32_t w = 1; w < WARPS; w++) {
#pragma unroll
        for (uint32_t j = 0; j < W; j++) v[j] += sm[w * TILE * PITCH_R + mr * PITCH_R + nr + j];
    }
    float *c = p.C + (uint64_t)m * p.ldc + n;
#pragma unroll
    for (uint32_t j = 0; j < W; j++) {
        if (MODE == TRAIN_FWD) v[j] = spg_activate(v[j] + beside[j], p.act);
        else if (MODE == TRAIN_DELTA) v[j] *= spg_derivative(beside[j], p.act);
        else v[j] *= p.alpha;
        if (n + j < p.N) c[j] = v[j];
    }
}

template <int MODE, int V, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
spg_train_mma_kernel(const SpgTrainProduct p)
{
    extern __shared__ __align__(16) float sm[];
    spg_grid_wait();
    spg_grid_trigger();
    product_tile<MODE, V, WARPS>(p, blockIdx.x, sm);
}

// the gradients of two layers: what the second leaves idle of the GPU's last wave the first has filled already
template <int V, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
spg_train_grad2_kernel(const SpgTrainProduct a, const SpgTrainProduct b, uint32_t tiles_a)
{
    extern __shared__ __align__(16) float sm[];
    spg_grid_wait();
    spg_grid_trigger();
    const bool first = blockIdx.x < tiles_a;
    product_tile<TRAIN_GRAD, V, WARPS>(first ? a : b, first ? blockIdx.x : blockIdx.x - tiles_a, sm);
}

uint32_t tiles(const SpgTrainProduct &p) { return ((p.M + TILE - 1) / TILE) * ((p.N + TILE - 1) / TILE); }

// Launches on `count` tiles.  CTAs are started while the launch before is still running, on whatever SM has room: so that they do not pile up there,
// a CTA takes the shared memory that leaves an SM room for its even share of them (1 KB of each goes to the system).
template <typename Kernel, typename... Args>
int launch_tiles(SpgOncePerDevice &once, Kernel kernel, uint32_t count, int warps, cudaStream_t s, const Args &...args)
{
    const size_t ring = 4 * ring_floats(warps);
    int device = 0;
    SpgDeviceProps props;
    SPGK_CUDA(cudaGetDevice(&device));
    int rc = spg_device_props(&props);
    if (rc) return rc;
    rc = once.run(device, [&] {
        SPGK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)props.smem_optin));
        return SPGK_OK;
    });
    if (rc) return rc;
    const uint32_t share = (count + props.sm_count - 1) / props.sm_count;
    const size_t room = (props.smem_optin + 1024) / share - 1024 & ~(size_t)127, bytes = share < 8 && room > ring ? room : ring;
    SPGK_CUDA(spg_launch_chained(kernel, dim3(count), dim3(warps * 32), bytes, s, args...));
    return spgk_check_launch("spg_train_mma_kernel");
}

template <int MODE, int V, int WARPS>
int launch(const SpgTrainProduct &p, cudaStream_t s)
{
    static SpgOncePerDevice once;
    static_assert(sum_floats(WARPS) <= ring_floats(WARPS), "the partial sums take the place of the rings");
    return launch_tiles(once, spg_train_mma_kernel<MODE, V, WARPS>, tiles(p), WARPS, s, p);
}

template <int V, int WARPS>
int launch_grad2(const SpgTrainProduct &a, const SpgTrainProduct &b, cudaStream_t s)
{
    static SpgOncePerDevice once;
    return launch_tiles(once, spg_train_grad2_kernel<V, WARPS>, tiles(a) + tiles(b), WARPS, s, a, b, tiles(a));
}

// ---- the output end of a step, for at most 16 outputs -----------------------------------------------------------------------
// Product, softmax or sigmoid, delta and loss in one launch, two rows a CTA.  A warp has two of the outputs of both rows, its lanes striding
// over k with the loads of eight strides in flight; a shuffle tree adds them.  Then a warp a row forms the activation.  (One warp a row for
// all its outputs, one stride's loads in flight, was 12.6 us of latency for 256 rows of 1000 inputs; this is 4.)
constexpr uint32_t OUT_MAX = 16, OUT_ROWS = 2, OUT_WARPS = 8, OUT_EACH = OUT_MAX / OUT_WARPS, OUT_AHEAD = 8;

struct OutputArgs {
    const float *x; uint32_t ldx; const float *w; uint32_t ldw; const float *bias; float *y; const float *t; float *delta; float *loss;
    uint32_t rows, out, in;
};

template <bool VEC, bool SIGMOID>
__global__ void __launch_bounds__(OUT_WARPS * 32)
spg_train_output_kernel(const OutputArgs p)
{
    constexpr uint32_t V = VEC ? 4 : 1, STRIDE = 32 * V;
    __shared__ float zs[OUT_ROWS][OUT_MAX];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, m0 = blockIdx.x * OUT_ROWS;
    float sum[OUT_ROWS][OUT_EACH] = {};
    const auto load = [](float (&v)[V], const float *q, bool there) {
        if constexpr (VEC) {
            const float4 f = there ? *reinterpret_cast<const float4 *>(q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else v[0] = there ? *q : 0.0f;
    };
    spg_grid_wait();
    spg_grid_trigger();
    for (uint32_t k0 = lane * V; k0 < p.in; k0 += STRIDE * OUT_AHEAD) {
        float x[OUT_ROWS][OUT_AHEAD][V], w[OUT_EACH][OUT_AHEAD][V];
#pragma unroll
        for (uint32_t i = 0; i < OUT_AHEAD; i++) {
            const uint32_t k = k0 + i * STRIDE;
#pragma unroll
            for (uint32_t r = 0; r < OUT_ROWS; r++) load(x[r][i], p.x + (uint64_t)(m0 + r) * p.ldx + k, m0 + r < p.rows && k < p.in);
#pragma unroll
            for (uint32_t e = 0; e < OUT_EACH; e++) load(w[e][i], p.w + (uint64_t)(warp + e * OUT_WARPS) * p.ldw + k, warp + e * OUT_WARPS < p.out && k < p.in);
        }
#pragma unroll
        for (uint32_t i = 0; i < OUT_AHEAD; i++) {
            if (k0 + i * STRIDE >= p.in) break;
#pragma unroll
            for (uint32_t r = 0; r < OUT_ROWS; r++)
#pragma unroll
                for (uint32_t e = 0; e < OUT_EACH; e++)
#pragma unroll
                    for (uint32_t j = V; j-- > 0;) sum[r][e] = fmaf(x[r][i][j], w[e][i][j], sum[r][e]);
        }
    }
    __syncwarp();
#pragma unroll
    for (uint32_t r = 0; r < OUT_ROWS; r++)
#pragma unroll
        for (uint32_t e = 0; e < OUT_EACH; e++) {
            sum[r][e] = spg_warp_sum(sum[r][e]);
            if (lane == 0) zs[r][warp + e * OUT_WARPS] = sum[r][e];
        }
    __syncthreads();
    const uint32_t m = m0 + warp;
    if (warp >= OUT_ROWS || m >= p.rows) return;
    const bool mine = lane < p.out;
    const float z = mine ? zs[warp][lane] + p.bias[lane] : 0.0f;
    float o;
    if (SIGMOID) o = spg_activate(z, SPG_ACT_SIGMOID);
    else {
        const float mx = spg_warp_max(mine ? z : -FLT_MAX);
        const float e = mine ? expf(z - mx) : 0.0f;
        const float total = spg_warp_sum(e);
        o = total > 0.0f ? e * (1.0f / total) : e;
    }
    float local = 0.0f;
    if (mine) {
        const float tg = p.t[(uint64_t)m * p.out + lane];
        p.y[(uint64_t)m * p.out + lane] = o;
        p.delta[(uint64_t)m * p.out + lane] = o - tg;
        if (p.loss) {
            if (SIGMOID) {
                const float c = fminf(fmaxf(o, 1e-9f), 1.0f - 1e-9f);
                local = -(tg * logf(c) + (1.0f - tg) * logf(1.0f - c));
            } else local = -tg * logf(fmaxf(o, 1e-9f));
        }
    }
    if (p.loss) {
        local = spg_warp_sum(local);
        if (lane == 0) atomicAdd(p.loss, local);
    }
}

}  // namespace

static bool on_lines(const SpgTrainProduct &p)
{
    const auto lines = [](const void *q, uint32_t ld) { return ((uintptr_t)q & 15u) == 0 && (ld & 3u) == 0; };
    return lines(p.A, p.lda) && lines(p.B, p.ldb);
}

int spg_train_two_gradients(const SpgTrainProduct &a, const SpgTrainProduct &b, cudaStream_t s)
{
    const bool vec = on_lines(a), few = tiles(a) <= 32u;
    if (vec != on_lines(b) || few != (tiles(b) <= 32u)) return SPGK_E_UNSUPPORTED;
    return few ? (vec ? launch_grad2<4, 8>(a, b, s) : launch_grad2<1, 8>(a, b, s)) : (vec ? launch_grad2<4, 4>(a, b, s) : launch_grad2<1, 4>(a, b, s));
}

int spg_train_product(int mode, const SpgTrainProduct &p, cudaStream_t s)
{
    const bool vec = on_lines(p);
    const bool few = tiles(p) <= 32u;      // eight warps a tile instead of four: 10 x 1000 over 256 rows 4.2 against 4.8 us, 30 x 60 over 1000 9.6 against 11
#define SPG_PRODUCT(MODE) (few ? (vec ? launch<MODE, 4, 8>(p, s) : launch<MODE, 1, 8>(p, s)) : (vec ? launch<MODE, 4, 4>(p, s) : launch<MODE, 1, 4>(p, s)))
    return mode == TRAIN_FWD ? SPG_PRODUCT(TRAIN_FWD) : mode == TRAIN_DELTA ? SPG_PRODUCT(TRAIN_DELTA) : SPG_PRODUCT(TRAIN_GRAD);
#undef SPG_PRODUCT
}

extern "C" int spgk_train_output(const float *x, uint32_t ldx, const float *w, uint32_t ldw, const float *bias, float *y, const float *t,
                                 float *delta, float *loss, uint32_t rows, uint32_t out, uint32_t in, int sigmoid_output, void *stream)
{
    if (!x || !w || !bias || !y || !t || !delta || rows == 0 || in == 0 || out == 0 || out > OUT_MAX) {
        spgk_set_error("spgk_train_output", "bad argument");
        return SPGK_E_ARG;
    }
    const OutputArgs p = { x, ldx, w, ldw, bias, y, t, delta, loss, rows, out, in };
    const bool vec = ((in | ldx | ldw) & 3u) == 0 && (((uintptr_t)x | (uintptr_t)w) & 15u) == 0;
    const auto kernel = vec ? (sigmoid_output ? spg_train_output_kernel<true, true> : spg_train_output_kernel<true, false>)
                            : (sigmoid_output ? spg_train_output_kernel<false, true> : spg_train_output_kernel<false, false>);
    SPGK_CUDA(spg_launch_chained(kernel, dim3((rows + OUT_ROWS - 1) / OUT_ROWS), dim3(OUT_WARPS * 32), 0, (cudaStream_t)stream, p));
    return spgk_check_launch("spg_train_output_kernel");
}
