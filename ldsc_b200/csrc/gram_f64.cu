// gram_f64.cu -- FP64 plain form of the band Gram: standardised columns
// x = (g - mean) inv_std in f64, val = x_k . x_j, and the reference's fused
// unbiased-r^2 transform val^2 * r2u_a / N^2 + r2u_b (src/l2/compute.rs:1067-1077,
// 2229-2235), on the FP64 tensor path (mma.sync m8n8k4 .f64).
//
// A warp owns one block of 32 x 32 records and takes the next from a counter,
// so only blocks that hold in-band pairs are multiplied and the last wave is
// short.  The standardised columns never exist in memory: a record's values are
// four -- (2 - mean) inv_std, (1 - mean) inv_std, -mean inv_std and 0 (missing)
// -- kept as a table in shared memory, indexed by the 2-bit code of the packed
// row, and every fragment element is one table read.  Per four individuals a
// warp issues 16 MMAs (256 clocks of its quarter of the FP64 pipe, 64 FMA per
// clock and SM) for 8 table reads and about 24 integer instructions.  The
// table rows are 32 bytes, so the four rows of a half-warp cover the 32 banks
// and its reads do not conflict.
//
// Bound by the FP64 pipe.  2,490 individuals x 18,627 records, 1 cM, chunks of
// 200: 1,610 us, 31 TFLOP/s over the blocks multiplied (columns written as f64 rows and multiplied in 128 x 128 tiles on the
// SIMT pipe: decode 141 us + Gram 3,184 us).
#include <cuda_runtime.h>

#include "engine.h"
#include "epilogue.cuh"

namespace ldsc {

namespace {

constexpr int WARPS = 16;           // per CTA, one CTA per SM: 4 per quarter of the FP64 pipe
constexpr int TABLE = 2 * 32 * 4;   // doubles per warp: 64 records x 4 codes

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// The epilogue's sums for a block with an inf or NaN annotation, masked by the
// product: v[8 i + 2 j + h] is pair (k + 8 i, j0 + 8 j + h); o: 4 row sums, 8
// column sums.  Its own function, so that the usual path keeps its registers
// (with a select on every product there, the Gram and its reduction took 1,704 us
// at the size above; this way 1,620).
__device__ __noinline__ void masked_sums(const double* v, double* o, int64_t k, int64_t j0, int64_t m,
                                         const int64_t* left, const double* aeff, double r2u_a, double r2u_b) {
    for (int i = 0; i < 12; i++) o[i] = 0.0;
    for (int p = 0; p < 32; p++) {
        const int64_t kk = k + 8 * (p / 8), jj = j0 + 8 * (p / 2 % 4) + p % 2;
        if (!pair_in_band(kk, jj, m, left)) continue;
        const double r2u = v[p] * v[p] * r2u_a + r2u_b;
        o[p / 8] += r2u * aeff[jj];
        o[4 + p % 8] += r2u * aeff[kk];
    }
}

__global__ void __launch_bounds__(32 * WARPS, 1)
    k_gram_f64(PanelView p, const uint64_t* __restrict__ rec_rows, RecStats st, const GramBlock* __restrict__ blocks,
               uint32_t n_blocks, unsigned int* __restrict__ next, EpilogueArgs ep) {
    extern __shared__ __align__(16) double tables[];
    const int lane = threadIdx.x & 31;
    double* tab = tables + (threadIdx.x >> 5) * TABLE;   // [record][code 00, 01, 10, 11], left records first
    const int fr = lane >> 2, fc = lane & 3;             // fragment row (record) and column (individual)
    const char* tab_a = reinterpret_cast<const char*>(tab + 4 * fr);
    const int64_t m = ep.m;
    const uint32_t words = (uint32_t)((p.n_indiv + 15) / 16);
    const uint32_t tail = (uint32_t)(p.n_indiv & 15);    // individuals in the last word (0: sixteen)
    const uint32_t tail_mask = tail ? (1u << (2 * tail)) - 1u : 0xFFFFFFFFu;
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(next, 1u);
        u = __shfl_sync(0xFFFFFFFFu, u, 0);
        if (u >= n_blocks) return;
        const GramBlock bl = blocks[u];
        const int64_t k0 = (int64_t)bl.a * 32, j0 = (int64_t)bl.b * 32;
        __syncwarp();   // the previous block's table reads are done
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int64_t r = (h ? j0 : k0) + lane;
            const double mean = r < m ? st.mean[r] : 0.0, inv = r < m ? st.inv_std[r] : 0.0;
            double* t = tab + 4 * (32 * h + lane);
            t[0] = (2.0 - mean) * inv;
            t[1] = 0.0;
            t[2] = (1.0 - mean) * inv;
            t[3] = (0.0 - mean) * inv;
        }
        __syncwarp();
        // this lane's packed rows: left records 8 i + fr, then right ones (past the end: the last row;
        // its table is zero)
        const uint32_t* row[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            int64_t r = (i < 4 ? k0 + 8 * i : j0 + 8 * (i - 4)) + fr;
            r = r < m ? r : m - 1;
            row[i] = reinterpret_cast<const uint32_t*>(p.rows + (rec_rows ? rec_rows[r] : (uint64_t)r) * p.pitch);
        }
        double acc[4][4][2];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
        uint32_t w[8], nw[8];
#pragma unroll
        for (int i = 0; i < 8; i++) nw[i] = __ldg(row[i]);
        for (uint32_t q = 0; q < words; q++) {
            const bool last = q + 1 == words;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                // individuals past the end read as missing (code 01); this lane's four codes to bits 8 s
                w[i] = (last ? (nw[i] & tail_mask) | (0x55555555u & ~tail_mask) : nw[i]) >> (2 * fc);
                if (!last) nw[i] = __ldg(row[i] + q + 1);
            }
#pragma unroll
            for (int s = 0; s < 4; s++) {   // individuals 16 q + 4 s + fc
                double a[4], b[4];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint32_t off = (s == 0 ? w[i] << 3 : w[i] >> (8 * s - 3)) & 24u;
                    const double v = *reinterpret_cast<const double*>(tab_a + 256 * i + off);
                    if (i < 4)
                        a[i] = v;
                    else
                        b[i - 4] = v;
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
            }
        }
        // ---- epilogue: acc[i][j][h] is pair (k0 + 8 i + fr, j0 + 8 j + 2 fc + h) ----
        double* rt = ep.K == 1 ? nullptr : ep.rtiles + (size_t)bl.slot * TILE_QUARTER * TILE_RECORDS + (bl.a & 3) * 32;
        double rs[4] = {0, 0, 0, 0}, cs[4][2];
        double ak[4];
#pragma unroll
        for (int i = 0; i < 4; i++) ak[i] = ep.K == 1 && k0 + 8 * i + fr < m ? __ldg(ep.aeff + k0 + 8 * i + fr) : 0.0;
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int cj = 8 * j + 2 * fc + h;
                const int64_t jj = j0 + cj;
                const double aj = ep.K == 1 && jj < m ? __ldg(ep.aeff + jj) : 0.0;
                cs[j][h] = 0.0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int64_t k = k0 + 8 * i + fr;
                    const double v = acc[i][j][h];
                    const double r2u = pair_in_band(k, jj, m, ep.left) ? v * v * ep.n_inv_sq_r2u_a + ep.r2u_b : 0.0;
                    if (ep.K == 1) {
                        rs[i] += r2u * aj;
                        cs[j][h] += r2u * ak[i];
                    } else {
                        rt[(size_t)cj * TILE_RECORDS + 8 * i + fr] = r2u;
                    }
                }
            }
        if (ep.K == 1) {
            // inf or NaN among the block's annotations: 0 x inf of a masked pair is no part of a sum
            const bool fin = (k0 + lane >= m || isfinite(__ldg(ep.aeff + k0 + lane))) &&
                             (j0 + lane >= m || isfinite(__ldg(ep.aeff + j0 + lane)));
            if (!__all_sync(0xFFFFFFFFu, fin)) {
                double v[32], o[12];
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = acc[i / 8][i / 2 % 4][i % 2];
                masked_sums(v, o, k0 + fr, j0 + 2 * fc, m, ep.left, ep.aeff, ep.n_inv_sq_r2u_a, ep.r2u_b);
#pragma unroll
                for (int i = 0; i < 4; i++) rs[i] = o[i];
#pragma unroll
                for (int i = 0; i < 8; i++) cs[i / 2][i % 2] = o[4 + i];
            }
            // the block's row and column sums; launch_l2_reduce adds them to l2
#pragma unroll
            for (int i = 0; i < 4; i++) {
                rs[i] += __shfl_xor_sync(0xFFFFFFFFu, rs[i], 1);
                rs[i] += __shfl_xor_sync(0xFFFFFFFFu, rs[i], 2);
                if (fc == 0) ep.prow[(size_t)bl.slot * 32 + 8 * i + fr] = rs[i];
            }
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
#pragma unroll
                    for (int o = 4; o < 32; o <<= 1) cs[j][h] += __shfl_xor_sync(0xFFFFFFFFu, cs[j][h], o);
                    if (fr == 0) ep.pcol[(size_t)bl.slot * 32 + 8 * j + 2 * fc + h] = cs[j][h];
                }
        }
    }
}

constexpr size_t SMEM = sizeof(double) * WARPS * TABLE;

}  // namespace

cudaError_t launch_gram_f64(const PanelView& p, const uint64_t* rec_rows, RecStats st, const GramBlock* blocks,
                            uint32_t n_blocks, unsigned int* next, const EpilogueArgs& ep, int sms,
                            cudaStream_t stream) {
    if (n_blocks == 0) return cudaSuccess;
    if (p.n_indiv == 0 || (reinterpret_cast<uintptr_t>(p.rows) & 3) != 0 || p.pitch % 4 != 0)
        return cudaErrorInvalidValue;
    k_gram_f64<<<(unsigned)sms, 32 * WARPS, SMEM, stream>>>(p, rec_rows, st, blocks, n_blocks, next, ep);
    return cudaGetLastError();
}

cudaError_t preload_gram_f64() {
    cudaError_t e = preload_kernel(k_gram_f64);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gram_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    return e;
}

}  // namespace ldsc
