// spg_gemm.cuh -- what the two tensor-core layer kernels (spg_gemm_tc.cu, spg_gemm_split.cu) share on the host side.
#pragma once

#include <cuda.h>
#include "spg_common.cuh"

// one call of spgk_layer_gemm_tc, checked
struct SpgGemmArgs {
    const spgk_layer *L;
    const void *w16; uint32_t ldw; uint64_t w_plane; int w_parts, w_type16;
    const void *a16; uint32_t lda; uint64_t a_plane; int a_parts, type16;
    void *out16; uint32_t ldo16; uint64_t o_plane; int out_parts;
    float *out32; uint32_t ldo32;
    uint32_t N; int softmax_fused; int32_t *status; void *stream;
};

// what the calling thread's last product ran as (spgk_gemm_tc_arrangement)
struct SpgGemmArrangement { uint32_t few_tiles, columns, split, stages; };
extern thread_local SpgGemmArrangement spg_tls_arrangement;

// 3-D tensor map over `parts` planes of a row-major [rows][ld] 16-bit matrix whose first K columns are valid; a box is 64
// columns x box_rows x box_planes
int spg_gemm_map(CUtensorMap *map, const void *base, int type16, uint32_t K, uint32_t rows, uint32_t ld, uint64_t plane, int parts,
                 uint32_t box_rows, uint32_t box_planes);

// Launches the few-tiles kernel if it has an arrangement for this product.  SPGK_E_UNSUPPORTED: the persistent kernel is needed, for
// row counts above `served` (0: for all, nothing was launched).
int spg_gemm_split_try(const SpgGemmArgs &a, const SpgDeviceProps &dp, int dev, uint32_t &served);

// Products of K = 16 that a layer's accumulators add up one after the other, whichever kernel its product runs on
uint32_t spg_gemm_steps(const spgk_layer *L, uint32_t N, uint32_t a_parts, uint32_t w_parts, bool softmax_fused, const SpgDeviceProps &dp, int dev);

// spgk_selftest_impatient
bool spg_gemm_impatient();
