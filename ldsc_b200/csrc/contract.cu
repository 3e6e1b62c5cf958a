// contract.cu -- annotation contraction of banded r2u tiles (K > 1), in f64.
//
// The reference contracts each chunk's r2u blocks with the annotation matrix
// in both directions (src/l2/compute.rs:1869-1893, 2259-2314):
//     l2[window] += R_ab * A_chunk,   l2[chunk] += R_ab^T * A_window (+ R_bb A_chunk).
// Here the Gram kernels leave every band tile's masked r2u values in global
// memory (f64, row j of the tile = 128 values) and these passes do the two
// products per block of rows: pass "by right block" owns l2 rows j of one
// right block, pass "by left block" owns l2 rows k of one left block, so no
// row is written by two CTAs of a pass and the summation order is fixed.
// Everything is f64 -- the r2u values as the epilogue formed them, the
// effective annotations as given, the products and sums -- so each l2_jC
// carries f64 rounding only, binary and continuous columns alike.
//
// Pairs outside the band are 0 in a tile, and 0 x inf would be NaN at records
// whose windows do not hold the annotation's record.  So the passes take an inf
// or NaN annotation as 0, and a third kernel adds it to the record's partners.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "epilogue.cuh"
#include "sm100.cuh"

namespace ldsc {

namespace {

constexpr int NT = 256;  // threads of k_l2_reduce

// The contraction on the FP64 tensor path (mma.sync m8n8k4 .f64):
//   BY_RIGHT: out rows j of the right block, out[j][c] += sum_k R[j][k] A[k][c]
//   BY_LEFT:  out rows k of the left block,  out[k][c] += sum_j R[j][k] A[j][c]
// One CTA owns 64 output rows, half a block, and up to MK = 128 annotation
// columns (K > 128 runs column chunks).  The summed records of every tile of
// the block go by in steps of JS = 16; quarters that a tile leaves out, and for
// BY_RIGHT tiles without a quarter in this half, cost nothing.  A step's r2u
// values and the annotation values of its records are staged by cp.async into
// one of two buffers while
// the MMAs run on the other; the tile list is read an entry ahead.  Each of the
// 4 warps owns 16 output rows and all the chunk's columns: 2 x NF fragments of
// 8 x 8 f64 accumulators, four k-steps of four records per staged step, so the
// 2 + NF fragment loads of a k-step feed 2 NF MMAs and only about ceil(K / 8)
// fragments are multiplied.  Three CTAs share an SM: one multiplies while
// another waits for its stage, and half blocks leave less of a last wave idle.
// The FP64 pipe bounds it (64 FMA per clock and SM): 100,000 records x 97
// columns, 2,892 tiles: 379 + 350 us, 70% of the pipe (steps of 32 and two CTAs:
// 462 + 431; one CTA of 128 rows per SM and the list read in each step: 553 +
// 535).
// Fragment layouts of m8n8k4 (row.col): A element (lane / 4, lane % 4), B
// element (lane % 4, lane / 4), D elements (lane / 4, 2 (lane % 4) + {0, 1}).
// Shared rows are padded to a stride of 4 mod 16 doubles, so each half-warp's
// 16 8-byte fragment loads hit 16 distinct bank pairs.
constexpr int MK = 128;        // annotation columns per chunk
constexpr int JS = 16;         // summed records per staged step
constexpr int OB = TILE_RECORDS;
constexpr int HB = OB / 2;     // output rows of a CTA
constexpr int CTH = 128;       // threads
constexpr int SLD = JS + 4;    // staged annotation stride (annotations are [column][record])
constexpr int RLD_R = JS + 4;  // BY_RIGHT r2u stage [64 j][16 k]
constexpr int RLD_L = HB + 4;  // BY_LEFT  r2u stage [16 j][64 k]

template <int NF, bool BY_RIGHT>
struct ContractShape {
    static constexpr int R_ELEMS = BY_RIGHT ? HB * RLD_R : JS * RLD_L;
    static constexpr int STAGE = R_ELEMS + 8 * NF * SLD;   // doubles per buffer
    static constexpr size_t smem = sizeof(double) * 2 * (size_t)STAGE;
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// 8 bytes, or zeros (nothing read) when !valid
__device__ __forceinline__ void cp_async8_zfill(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src),
                 "r"(valid ? 8 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// NF: fragments of 8 columns per warp (the chunk has at most 8 NF columns;
// results past it are not stored).
template <int NF, bool BY_RIGHT>
__global__ void __launch_bounds__(CTH, 3)
    k_contract_mma(const Tile* __restrict__ tiles, const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                   int32_t nblocks, EpilogueArgs ep) {
    using S = ContractShape<NF, BY_RIGHT>;
    extern __shared__ __align__(16) double smm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = ep.K;
    const int64_t m = ep.m;
    const int nchunks = (K + MK - 1) / MK;
    const int fr = lane >> 2, fc = lane & 3;   // fragment row / column of this lane
    const bool special = *ep.special != 0;

    for (int64_t w = blockIdx.x; w < (int64_t)nblocks * nchunks * 2; w += gridDim.x) {
        const int half = (int)(w & 1);
        const int32_t blk = (int32_t)(w / 2 / nchunks);
        const int c0 = (int)(w / 2 % nchunks) * MK;
        const int kc = K - c0 < MK ? K - c0 : MK;   // columns of this chunk
        const int32_t t0 = ptr[blk], t1 = ptr[blk + 1];
        if (t0 == t1) continue;

        // the staged steps run over the block's tiles: this step's tile, and the next list entry
        struct Entry {
            Tile tl;
            uint32_t roff;
        };
        auto tile_of = [&](int32_t e) { return idx[e < t1 ? e : t1 - 1]; };
        int32_t e = t0, ahead = tile_of(t0 + 1);   // the tile after next
        Entry cur{}, next{tiles[idx[t0]], ep.roff[idx[t0]]};
        int st = 0, steps = 0;   // step of the tile, its steps
        int lo = 0, hi = 1;      // BY_RIGHT: the tile's quarters within this half's two
        bool more = true;
        auto advance = [&]() {
            if (++st < steps) return;
            do {
                more = e < t1;
                if (!more) return;
                cur = next;
                next = Entry{tiles[ahead], ep.roff[ahead]};
                ahead = tile_of(++e + 1);
                if (BY_RIGHT) {
                    lo = max((int)cur.tl.q0 - 2 * half, 0);
                    hi = min((int)(cur.tl.q0 + cur.tl.nq1) - 2 * half, 1);
                }
            } while (BY_RIGHT && lo > hi);
            st = 0;
            steps = (BY_RIGHT ? OB : ((int)cur.tl.nq1 + 1) * TILE_QUARTER) / JS;
        };
        auto issue = [&](int b) {
            const Tile tl = cur.tl;
            const double* src = ep.rtiles + (size_t)cur.roff * TILE_QUARTER * OB;
            double* Rs = smm + b * S::STAGE;
            double* As = Rs + S::R_ELEMS;
            if (BY_RIGHT) {
                // the half's rows j of the tile, values k = JS st .. JS st + JS - 1: 16-byte pieces
                const int n = (hi - lo + 1) * TILE_QUARTER;
                const double* sr = src + (size_t)(lo + 2 * half - (int)tl.q0) * TILE_QUARTER * OB + st * JS;
                double* dst = Rs + lo * TILE_QUARTER * RLD_R;
                for (int q = tid; q < n * JS / 2; q += CTH) {
                    const int r = q / (JS / 2), cc = 2 * (q % (JS / 2));
                    cp_async16(dst + r * RLD_R + cc, sr + r * OB + cc);
                }
            } else {
                // JS rows j of the tile, this half's 64 values
                const double* sr = src + (size_t)st * JS * OB + half * HB;
#pragma unroll
                for (int q = tid; q < JS * HB / 2; q += CTH) {
                    const int r = q / (HB / 2), cc = 2 * (q % (HB / 2));
                    cp_async16(Rs + r * RLD_L + cc, sr + r * OB + cc);
                }
            }
            // annotation column c0 + c of summed record s at aeff[s + (c0 + c) m]; consecutive threads
            // take consecutive records (coalesced), zeros past m or K
            const int64_t s0 = BY_RIGHT ? (int64_t)tl.a_blk * OB + st * JS
                                        : (int64_t)tl.b_blk * OB + (int)tl.q0 * TILE_QUARTER + st * JS;
            const int s = tid & (JS - 1);
            const bool in = s0 + s < m;
            const double* col = ep.aeff + (in ? s0 + s + (int64_t)(c0 + tid / JS) * m : 0);
            double* dst = As + (tid / JS) * SLD + s;
#pragma unroll 4
            for (int c = tid / JS; c < 8 * NF; c += CTH / JS, col += (CTH / JS) * m, dst += (CTH / JS) * SLD)
                cp_async8_zfill(dst, in && c < kc ? col : ep.aeff, in && c < kc);
        };

        double acc[2][NF][2];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < NF; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

        advance();
        bool staged = more;                           // something is in buffer b
        bool active = warp / 2 >= lo && warp / 2 <= hi;   // this warp's rows are in it (warp-uniform)
        if (more) issue(0);
        cp_async_commit();
        for (int b = 0; staged; b ^= 1) {
            const bool act = active;
            advance();
            staged = more;
            if (more) {
                active = warp / 2 >= lo && warp / 2 <= hi;
                issue(b ^ 1);
            }
            cp_async_commit();
            cp_async_wait1();  // the current step's copies (this thread's) have landed
            if (special) {     // inf and NaN among the annotations it copied
                double* a = smm + b * S::STAGE + S::R_ELEMS + (tid / JS) * SLD + (tid & (JS - 1));
                for (int c = tid / JS; c < 8 * NF; c += CTH / JS, a += (CTH / JS) * SLD)
                    if (!isfinite(*a)) *a = 0.0;
            }
            __syncthreads();   // ... and every thread's
            if (act) {
                const double* Rs = smm + b * S::STAGE;
                const double* As = Rs + S::R_ELEMS;
#pragma unroll 2
                for (int kk = 0; kk < JS; kk += 4) {
                    double a[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int orow = 16 * warp + 8 * i + fr;  // output row of the fragment
                        a[i] = BY_RIGHT ? Rs[orow * RLD_R + kk + fc] : Rs[(kk + fc) * RLD_L + orow];
                    }
#pragma unroll
                    for (int j = 0; j < NF; j++) {
                        const double bj = As[(8 * j + fr) * SLD + kk + fc];
#pragma unroll
                        for (int i = 0; i < 2; i++) dmma(acc[i][j][0], acc[i][j][1], a[i], bj);
                    }
                }
            }
            __syncthreads();  // this buffer is refilled by the next iteration's issue
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int64_t row = (int64_t)blk * OB + half * HB + 16 * warp + 8 * i + fr;
            if (row >= m) continue;
#pragma unroll
            for (int j = 0; j < NF; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int c = 8 * j + 2 * fc + h;
                    if (c < kc) ep.l2[row + (int64_t)(c0 + c) * m] += acc[i][j][h];
                }
        }
    }
}

// Annotations that are inf or NaN, one warp each: a r2u_rp into l2 of every
// partner p of its record r, from the tiles of r's left block (r on the left)
// and of its right block.  (Sums with inf or NaN do not depend on their order.)
__global__ void __launch_bounds__(CTH) k_contract_special(const Tile* __restrict__ tiles, const int32_t* __restrict__ ptr_r,
                                                          const int32_t* __restrict__ idx_r, const int32_t* __restrict__ ptr_l,
                                                          const int32_t* __restrict__ idx_l, EpilogueArgs ep) {
    if (*ep.special == 0) return;
    const int lane = threadIdx.x & 31;
    const int64_t m = ep.m, total = m * ep.K, warps = (int64_t)gridDim.x * (CTH / 32);
    for (int64_t e0 = 32 * ((int64_t)blockIdx.x * (CTH / 32) + (threadIdx.x >> 5)); e0 < total; e0 += 32 * warps) {
        unsigned found = __ballot_sync(0xFFFFFFFFu, e0 + lane < total && !isfinite(ep.aeff[e0 + lane]));
        for (; found; found &= found - 1) {
            const int64_t e = e0 + __ffs(found) - 1, r = e % m;
            const double a = ep.aeff[e];
            double* l2 = ep.l2 + (e - r);   // the annotation's column
            const int64_t blk = r / OB;
            const int at = (int)(r % OB);
            for (int32_t i = ptr_l[blk]; i < ptr_l[blk + 1]; i++) {
                const Tile tl = tiles[idx_l[i]];
                const double* src = ep.rtiles + (size_t)ep.roff[idx_l[i]] * TILE_QUARTER * OB + at;
                const int64_t j0 = (int64_t)tl.b_blk * OB + tl.q0 * TILE_QUARTER;
                for (int x = lane; x < ((int)tl.nq1 + 1) * TILE_QUARTER; x += 32)
                    if (pair_in_band(r, j0 + x, m, ep.left)) atomicAdd(l2 + j0 + x, src[(size_t)x * OB] * a);
            }
            for (int32_t i = ptr_r[blk]; i < ptr_r[blk + 1]; i++) {
                const Tile tl = tiles[idx_r[i]];
                const int row = at - (int)tl.q0 * TILE_QUARTER;
                if (row < 0 || row >= ((int)tl.nq1 + 1) * TILE_QUARTER) continue;
                const double* src = ep.rtiles + ((size_t)ep.roff[idx_r[i]] * TILE_QUARTER + row) * OB;
                const int64_t k0 = (int64_t)tl.a_blk * OB;
                for (int x = lane; x < OB; x += 32)
                    if (pair_in_band(k0 + x, r, m, ep.left)) atomicAdd(l2 + k0 + x, src[x] * a);
            }
        }
    }
}

// K = 1: one thread per record, the record's column sums over the tiles of its
// right block, then its row sums over the tiles of its left block, in list
// order (coalesced: consecutive records read consecutive partials of a tile).
__global__ void __launch_bounds__(NT) k_l2_reduce(int64_t m, int ta, int tb, const int32_t* __restrict__ ptr_r,
                                                  const int32_t* __restrict__ idx_r, const int32_t* __restrict__ ptr_l,
                                                  const int32_t* __restrict__ idx_l, const double* __restrict__ prow,
                                                  const double* __restrict__ pcol, double* __restrict__ l2) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    double acc = l2[j];
    const int64_t rb = j / tb, lb = j / ta;
    for (int32_t i = ptr_r[rb]; i < ptr_r[rb + 1]; i++) acc += pcol[(size_t)idx_r[i] * tb + (j - rb * tb)];
    for (int32_t i = ptr_l[lb]; i < ptr_l[lb + 1]; i++) acc += prow[(size_t)idx_l[i] * ta + (j - lb * ta)];
    l2[j] = acc;
}

}  // namespace

cudaError_t launch_l2_reduce(int64_t m, int ta, int tb, const int32_t* ptr_r, const int32_t* idx_r,
                             const int32_t* ptr_l, const int32_t* idx_l, const double* prow, const double* pcol,
                             double* l2, cudaStream_t stream) {
    if (m <= 0) return cudaSuccess;
    k_l2_reduce<<<(unsigned)((m + NT - 1) / NT), NT, 0, stream>>>(m, ta, tb, ptr_r, idx_r, ptr_l, idx_l, prow, pcol,
                                                                  l2);
    return cudaGetLastError();
}

template <int NF, bool BY_RIGHT>
static cudaError_t run_contract(const Tile* tiles, const int32_t* ptr, const int32_t* idx, int32_t nblocks,
                                const EpilogueArgs& ep, int sms, cudaStream_t stream) {
    const size_t smem = ContractShape<NF, BY_RIGHT>::smem;
    cudaError_t e =
        cudaFuncSetAttribute(k_contract_mma<NF, BY_RIGHT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t work = 2 * (int64_t)nblocks * ((ep.K + MK - 1) / MK);
    const int64_t cap = (int64_t)sms * std::min<int64_t>(3, 227 * 1024 / (int64_t)(smem + 1024));
    k_contract_mma<NF, BY_RIGHT><<<(unsigned)(work < cap ? work : cap), CTH, smem, stream>>>(tiles, ptr, idx, nblocks, ep);
    return cudaGetLastError();
}

// Fragments per warp by the columns of a chunk: every fragment is multiplied,
// so the sizes are close together (K = 97 runs 13, a 53-annotation model 7).
cudaError_t launch_contract(const Tile* tiles, const int32_t* ptr, const int32_t* idx, int32_t nblocks, bool by_right,
                            const EpilogueArgs& ep, int sms, cudaStream_t stream) {
    if (nblocks <= 0) return cudaSuccess;
#define LDSC_CONTRACT(NF_)                                                                        \
    (by_right ? run_contract<NF_, true>(tiles, ptr, idx, nblocks, ep, sms, stream)               \
              : run_contract<NF_, false>(tiles, ptr, idx, nblocks, ep, sms, stream))
    if (ep.K <= 8) return LDSC_CONTRACT(1);
    if (ep.K <= 16) return LDSC_CONTRACT(2);
    if (ep.K <= 32) return LDSC_CONTRACT(4);
    if (ep.K <= 56) return LDSC_CONTRACT(7);
    if (ep.K <= 80) return LDSC_CONTRACT(10);
    if (ep.K <= 104) return LDSC_CONTRACT(13);
    return LDSC_CONTRACT(16);
#undef LDSC_CONTRACT
}

cudaError_t launch_contract_special(const Tile* tiles, const int32_t* ptr_r, const int32_t* idx_r, const int32_t* ptr_l,
                                    const int32_t* idx_l, const EpilogueArgs& ep, int sms, cudaStream_t stream) {
    k_contract_special<<<(unsigned)(4 * sms), CTH, 0, stream>>>(tiles, ptr_r, idx_r, ptr_l, idx_l, ep);
    return cudaGetLastError();
}

cudaError_t preload_contract() {
    cudaError_t e = preload_kernel(k_contract_mma<1, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<1, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<2, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<2, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<4, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<4, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<7, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<7, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<10, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<10, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<13, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<13, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<16, true>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_mma<16, false>);
    if (e == cudaSuccess) e = preload_kernel(k_contract_special);
    if (e == cudaSuccess) e = preload_kernel(k_l2_reduce);
    return e;
}

}  // namespace ldsc
