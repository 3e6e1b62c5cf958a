// partitioned.cu -- partitioned (stratified) h2 on device-resident LD scores:
// one weighted least squares on K annotation LD-score columns plus an
// intercept, with the block jackknife.  Restates fit_h2_partitioned
// (src/regressions.rs:1121-1226): weights from the summed LD score
// (aggregate, ldsc_weights, src/h2.rs:185-218), the weighted design
// (weight_xy, src/h2.rs:60-80), jackknife_fast's per-block X'X / X'y and LU
// solves (src/h2.rs:100-183) and jackknife_se_cov (src/jackknife.rs:10-59).
//
// The design is augmented with y as its last column, Z = [x_1..x_K, 1, y],
// so one symmetric Gram per jackknife block, sum_i w_i z_i z_i', holds X'X,
// X'y and y'y.  Rows are scaled by sqrt(w_i) as in the reference, which also
// divides by sum_j sqrt(w_j): that global factor cancels in every solve.  SNPs dropped by the chi2 cut contribute nothing and the
// jackknife blocks are the reference's blocks over the kept SNPs (block starts
// mapped back to SNP indices).  Block partial sums are combined in block
// order, so results do not depend on scheduling.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <utility>

#include "engine.h"
#include "regress.h"

namespace ldsc {

namespace {

constexpr int NT = 256;
constexpr int ROWS = 32;       // SNPs staged per step of the Gram

__device__ __forceinline__ double part_n(const PartJob& jb, uint64_t i) { return jb.nv ? jb.nv[i] : jb.ns; }
__device__ __forceinline__ bool part_kept(const PartJob& jb, uint64_t i) { return jb.chi2[i] < jb.mask_max; }

template <typename T>
__device__ __forceinline__ T block_sum(T v, T* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    T t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < NT / 32; w++) t += red[w];
    __syncthreads();
    return t;
}

// x_tot[i] = sum_j l2[i, j], columns added in order (src/regressions.rs:1158-1165)
__global__ void __launch_bounds__(NT) k_p_xtot(const double* __restrict__ l2, uint64_t ld, int k, uint64_t n,
                                              double* __restrict__ xtot) {
    for (uint64_t i = (uint64_t)blockIdx.x * NT + threadIdx.x; i < n; i += (uint64_t)gridDim.x * NT) {
        double s = 0.0;
        for (int j = 0; j < k; j++) s += l2[(size_t)j * ld + i];
        xtot[i] = s;
    }
}

// Per (jackknife block, job): sum chi2, sum x_tot * N, sum N over kept SNPs.
__global__ void __launch_bounds__(NT) k_p_sums(const PartJob* __restrict__ jobs, const double* __restrict__ xtot,
                                              int nb, double* __restrict__ part) {
    __shared__ double red[NT / 32];
    const int b = blockIdx.x, j = blockIdx.y;
    const PartJob jb = jobs[j];
    const uint64_t lo = (uint64_t)jb.seps[b], hi = (uint64_t)jb.seps[b + 1];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (uint64_t i = lo + threadIdx.x; i < hi; i += NT) {
        if (!part_kept(jb, i)) continue;
        const double nn = part_n(jb, i);
        s0 += jb.chi2[i];
        s1 += xtot[i] * nn;
        s2 += nn;
    }
    double* out = part + ((size_t)j * nb + b) * 3;
    s0 = block_sum(s0, red);
    s1 = block_sum(s1, red);
    s2 = block_sum(s2, red);
    if (threadIdx.x == 0) {
        out[0] = s0;
        out[1] = s1;
        out[2] = s2;
    }
}

// nbar, mean chi2 and the aggregate h2 that seeds the weights
// (src/regressions.rs:1189-1191).  One warp per job: lane l adds blocks l, l +
// 32, ..., then a fixed-order reduction.
__global__ void k_p_aggregate(const PartJob* __restrict__ jobs, const double* __restrict__ part, int nb,
                              double m_tot, PartState* __restrict__ st, int njobs) {
    const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= njobs) return;
    double s[3] = {0.0, 0.0, 0.0};
    for (int b = lane; b < nb; b += 32)
#pragma unroll
        for (int q = 0; q < 3; q++) s[q] += part[((size_t)j * nb + b) * 3 + q];
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xFFFFFFFFu, s[q], o);
    if (lane) return;
    const double nobs = jobs[j].n_obs;
    PartState& o = st[j];
    o.n_obs = nobs;
    o.nbar = s[2] / nobs;
    o.mean_chi2 = s[0] / nobs;
    o.agg_int = jobs[j].fixed ? jobs[j].fixed_int : 1.0;
    o.hsq = m_tot * (o.mean_chi2 - o.agg_int) / (s[1] / nobs);
}

// Gram of the augmented weighted design over one jackknife block:
// G = sum_i w_i z_i z_i' with z_i = [N_i l2_i1 / nbar, ..., N_i l2_iK / nbar,
// 1 (free intercept only), chi2_i - fixed intercept] and w_i the reference's
// weight (its weighted design scales rows by sqrt(w_i) / sum_j sqrt(w_j),
// src/h2.rs:60-80; the global factor cancels in every solve), on the FP64 tensor
// path (mma.sync m8n8k4 .f64).
//
// Columns are cut into groups of 8; the upper triangle of the group grid is
// covered by units of up to 4 x 5 groups (14 on the diagonal), one per warp, so
// a k-step of 4 SNPs loads 9 fragments for up to 20 MMAs.  One matrix serves as
// both operands: it is staged once, [column][SNP], 32 SNPs per step,
// three steps in flight by cp.async, one barrier per step (raw LD scores; rows of 36 doubles, so each
// half-warp's fragment loads hit 16 distinct bank pairs).  A row is staged as
// v_i = z_i / s_i with s_i = N_i / nbar (the LD-score columns are then the raw
// values, the intercept 1 / s_i, the chi2 column y_i / s_i) and enters as
// (w_i s_i^2) v_i v_i', the factor multiplying the left fragment; a row with
// N_i = 0 is staged as z_i with factor w_i.  The warp with the
// smallest unit forms the next steps' factors meanwhile.  Few units (small K)
// split the k-steps of a stage between the warps and add their parts in order.
// Bound by the FP64 pipe: 8 traits x 300,007 SNPs x 97 annotations (99 columns,
// 91 groups): 1,287 us, 58% of the pipe (SIMT
// micro-tiles, 4 x 4 outputs per thread: 3,146 us).
constexpr int PR = 4, PC = 5;          // groups per unit
constexpr int USTRIDE = ROWS + 4;      // doubles per staged column
constexpr int GWARPS = NT / 32;
constexpr int NBUF = 3;                // staged steps
constexpr int META = 4;                // ring of row factors
__host__ __device__ inline int part_groups(int q) { return (q + 7) / 8; }
__host__ __device__ inline int part_units(int q) {
    const int nt = part_groups(q);
    int u = 0;
    for (int r = 0; r < nt; r += PR) u += (nt - r + PC - 1) / PC;
    return u;
}
// warps that share one unit's k-steps
__host__ __device__ inline int part_ksplit(int q) {
    const int u = part_units(q);
    return u == 1 ? 8 : (u == 2 ? 4 : (u <= 4 ? 2 : 1));
}
constexpr int MAX_UNITS = 16;   // q <= 161: 21 groups
struct UnitOrder {
    uint8_t u[MAX_UNITS];
};
// Units by falling number of MMAs.
inline UnitOrder part_unit_order(int q) {
    const int nt = part_groups(q), n = part_units(q);
    int cost[MAX_UNITS];
    for (int r = 0, u = 0; r < nt; r += PR)
        for (int c = r; c < nt; c += PC, u++) {
            const int nr = nt - r < PR ? nt - r : PR, nc = nt - c < PC ? nt - c : PC;
            cost[u] = 0;
            for (int i = 0; i < nr; i++) cost[u] += c == r ? (nc > i ? nc - i : 0) : nc;
        }
    UnitOrder o{};
    for (int i = 0; i < n; i++) o.u[i] = (uint8_t)i;
    std::sort(o.u, o.u + n, [&](uint8_t a, uint8_t b) { return cost[a] != cost[b] ? cost[a] > cost[b] : a < b; });
    return o;
}
__host__ __device__ inline size_t part_gram_smem(int q) {
    const size_t stage = NBUF * (size_t)8 * part_groups(q) * USTRIDE;
    const size_t parts = (size_t)(GWARPS - GWARPS / part_ksplit(q)) * PR * PC * 64;   // of the split k-steps
    return (stage > parts ? stage : parts) * sizeof(double);
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One stage's k-steps [kg, 8) by ks of a unit of NR x NC groups; DIAG: the unit's
// column groups start at its row groups (groups below the diagonal are left out).
template <bool DIAG, int NR, int NC>
__device__ __forceinline__ void gram_stage(double (&acc)[PR][PC][2], const double* left, const double* right,
                                           const double* f, int kg, int ks) {
#pragma unroll 2
    for (int kk = kg; kk < ROWS / 4; kk += ks) {
        const double fk = f[4 * kk];
        double a[NR], b[NC];
#pragma unroll
        for (int j = 0; j < NC; j++) b[j] = right[j * 8 * USTRIDE + 4 * kk];
#pragma unroll
        for (int i = 0; i < NR; i++) a[i] = left[i * 8 * USTRIDE + 4 * kk] * fk;
#pragma unroll
        for (int i = 0; i < NR; i++)
#pragma unroll
            for (int j = DIAG ? i : 0; j < NC; j++) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
}
// nr < 4 only in the last row of units, on the diagonal, where nc = nr
template <bool DIAG>
__device__ __forceinline__ void gram_stage_any(double (&acc)[PR][PC][2], const double* left, const double* right,
                                               const double* f, int nr, int nc, int kg, int ks) {
    if (nr < 4) {
        if (nr == 1) gram_stage<true, 1, 1>(acc, left, right, f, kg, ks);
        if (nr == 2) gram_stage<true, 2, 2>(acc, left, right, f, kg, ks);
        if (nr == 3) gram_stage<true, 3, 3>(acc, left, right, f, kg, ks);
        return;
    }
    if (nc == 5) gram_stage<DIAG, 4, 5>(acc, left, right, f, kg, ks);
    if (nc == 4) gram_stage<DIAG, 4, 4>(acc, left, right, f, kg, ks);
    if (!DIAG && nc == 3) gram_stage<DIAG, 4, 3>(acc, left, right, f, kg, ks);
    if (!DIAG && nc == 2) gram_stage<DIAG, 4, 2>(acc, left, right, f, kg, ks);
    if (!DIAG && nc == 1) gram_stage<DIAG, 4, 1>(acc, left, right, f, kg, ks);
}

__global__ void __launch_bounds__(NT, 2) k_p_gram(const PartJob* __restrict__ jobs, const PartState* __restrict__ st,
                                                 const double* __restrict__ l2, uint64_t ld, int k,
                                                 const double* __restrict__ xtot, const double* __restrict__ wld,
                                                 double m_tot, int nb, int q, UnitOrder order, double* __restrict__ gram) {
    extern __shared__ __align__(16) double U[];   // NBUF x 8 nt x USTRIDE, then the split k-steps' parts
    // per row: factor w s^2 (w where s = 0; 0: not kept), intercept and chi2 columns, whether s != 0
    __shared__ double mf[META][ROWS], mi[META][ROWS], my[META][ROWS];
    __shared__ bool ms[META][ROWS];
    const int b = blockIdx.x, j = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fc = lane & 3;
    const int nt = part_groups(q), ks = part_ksplit(q), upc = GWARPS / ks;   // units per CTA
    // Warps w and w + 4 share a quarter of the SM: the first four take the largest
    // units in falling order, the others the rest in rising order, and every
    // other 148 CTAs shift the quarters by two, which evens out two CTAs of an SM.
    const int turn = ks == 1 ? 2 * (((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) / 148 & 1) : 0;
    const int wt = (warp & 4) | ((warp + turn) & 3), pos = wt < 4 ? wt : GWARPS + 3 - wt;
    const int nth = blockIdx.y * upc + (ks == 1 ? pos : warp % upc), kg = warp / upc;
    const int idle = (GWARPS / 2 - turn) % 4 + 4;   // the warp with pos 7, the smallest unit if any
    // the unit's row and column groups
    int r0 = 0, left_u = nth < part_units(q) ? order.u[nth] : INT_MAX;
    while (r0 < nt && left_u >= (nt - r0 + PC - 1) / PC) {
        left_u -= (nt - r0 + PC - 1) / PC;
        r0 += PR;
    }
    const bool active = r0 < nt;
    const int c0 = r0 + left_u * PC;
    const int nr = min(PR, nt - r0), nc = min(PC, nt - c0);
    const PartJob jb = jobs[j];
    const PartState s = st[j];
    const bool free_int = !jb.fixed;
    const double yoff = jb.fixed ? jb.fixed_int : 0.0;
    const double hsq = fmin(fmax(s.hsq, 0.0), 1.0);
    const uint64_t lo = (uint64_t)jb.seps[b], hi = (uint64_t)jb.seps[b + 1];
    const int nchunks = (int)((hi - lo + ROWS - 1) / ROWS);
    const size_t bufsz = (size_t)8 * nt * USTRIDE;
    // padding columns [q, 8 nt) stay zero in every buffer
    for (int e = threadIdx.x; e < NBUF * (8 * nt - q) * ROWS; e += NT) {
        const int bb = e / ((8 * nt - q) * ROWS), c = q + (e / ROWS) % (8 * nt - q);
        U[bb * bufsz + c * USTRIDE + e % ROWS] = 0.0;
    }
    auto meta = [&](int c) {   // by one warp: row factors of stage c
        const int slot = c % META;
        const uint64_t i = lo + (uint64_t)c * ROWS + lane;
        double f = 0.0, vi = 0.0, vy = 0.0;
        bool nz = false;
        if (i < hi && part_kept(jb, i)) {
            // ldsc_weights (src/h2.rs:185-206) on x_tot with M = sum(M_k)
            const double nn = part_n(jb, i);
            const double cc = hsq * nn / m_tot;
            const double t = s.agg_int + cc * fmax(xtot[i], 1.0);
            const double w = 1.0 / (2.0 * t * t) / fmax(wld[i], 1.0);
            const double sc = nn / s.nbar, y = jb.chi2[i] - yoff;
            nz = sc != 0.0;
            f = nz ? w * sc * sc : w;
            vi = nz ? 1.0 / sc : 1.0;
            vy = nz ? y / sc : y;
        }
        mf[slot][lane] = f;
        mi[slot][lane] = vi;
        my[slot][lane] = vy;
        ms[slot][lane] = nz;
    };
    auto stage = [&](int c) {   // buffer c % NBUF: the LD scores, and the special columns from the factors
        const int slot = c % META;
        const uint64_t i0 = lo + (uint64_t)c * ROWS;
        double* buf = U + (c % NBUF) * bufsz;
        const int r = threadIdx.x % ROWS;
        const bool load = ms[slot][r];   // (row not kept, or N = 0: its LD-score columns are 0)
        for (int col = threadIdx.x / ROWS; col < k; col += NT / ROWS) {
            double* dst = buf + col * USTRIDE + r;
            if (load)
                cp_async8(dst, l2 + (size_t)col * ld + i0 + r);
            else
                *dst = 0.0;
        }
        if (threadIdx.x < ROWS) {
            if (free_int) buf[k * USTRIDE + r] = mi[slot][r];
            buf[(q - 1) * USTRIDE + r] = my[slot][r];
        }
    };
    double acc[PR][PC][2];
#pragma unroll
    for (int i = 0; i < PR; i++)
#pragma unroll
        for (int c = 0; c < PC; c++) acc[i][c][0] = acc[i][c][1] = 0.0;
    if (warp == idle && nchunks > 0) meta(0);
    if (warp == 0 && nchunks > 1) meta(1);
    if (warp == 1 && nchunks > 2) meta(2);
    __syncthreads();
    for (int c = 0; c < 2; c++) {
        if (c < nchunks) stage(c);
        cp_async_commit();
    }
    for (int c = 0; c < nchunks; c++) {
        cp_async_wait<1>();   // this thread's copies of stage c have landed
        __syncthreads();      // ... everyone's, and stage c - 1 is no longer read
        if (c + 2 < nchunks) stage(c + 2);
        cp_async_commit();
        if (warp == idle && c + 3 < nchunks) meta(c + 3);
        if (active) {
            const double* buf = U + (c % NBUF) * bufsz;
            const double* lp = buf + (8 * r0 + fr) * USTRIDE + fc;
            const double* rp = buf + (8 * c0 + fr) * USTRIDE + fc;
            const double* f = &mf[c % META][fc];
            if (c0 == r0)
                gram_stage_any<true>(acc, lp, rp, f, nr, nc, kg, ks);
            else
                gram_stage_any<false>(acc, lp, rp, f, nr, nc, kg, ks);
        }
    }
    __syncthreads();
    if (ks > 1) {   // parts of the k-steps, added in order by the unit's first warp
        if (active && kg > 0) {
            double* o = U + (size_t)((kg - 1) * upc + warp % upc) * PR * PC * 64 + lane;
#pragma unroll
            for (int i = 0; i < PR; i++)
#pragma unroll
                for (int c = 0; c < PC; c++)
#pragma unroll
                    for (int h = 0; h < 2; h++) o[((i * PC + c) * 2 + h) * 32] = acc[i][c][h];
        }
        __syncthreads();
        if (active && kg == 0)
            for (int g = 1; g < ks; g++) {
                const double* o = U + (size_t)((g - 1) * upc + warp) * PR * PC * 64 + lane;
#pragma unroll
                for (int i = 0; i < PR; i++)
#pragma unroll
                    for (int c = 0; c < PC; c++)
#pragma unroll
                        for (int h = 0; h < 2; h++) acc[i][c][h] += o[((i * PC + c) * 2 + h) * 32];
            }
    }
    if (!active || kg > 0) return;
    // write row <= col and its mirror, so the stored matrix is exactly symmetric
    double* G = gram + ((size_t)j * nb + b) * (size_t)q * q;
#pragma unroll
    for (int i = 0; i < PR; i++)
#pragma unroll
        for (int c = 0; c < PC; c++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int rr = 8 * (r0 + i) + fr, cc = 8 * (c0 + c) + 2 * fc + h;
                if (i < nr && c < nc && rr < q && cc < q && rr <= cc) {
                    G[(size_t)rr * q + cc] = acc[i][c][h];
                    G[(size_t)cc * q + rr] = acc[i][c][h];
                }
            }
}

// tot[j] = sum over blocks in order of the block Grams.
__global__ void __launch_bounds__(NT) k_p_total(const double* __restrict__ gram, int nb, int qq,
                                               double* __restrict__ tot) {
    const int j = blockIdx.y;
    const int e = blockIdx.x * NT + threadIdx.x;
    if (e >= qq) return;
    const double* g = gram + (size_t)j * nb * qq + e;
    double s = 0.0;
    for (int b = 0; b < nb; b++) s += g[(size_t)b * qq];
    tot[(size_t)j * qq + e] = s;
}

// One solve per CTA: (X'X_tot - X'X_b) beta = X'y_tot - X'y_b for b < nb
// (the delete values), the total system for b == nb, by Gauss-Jordan
// elimination with partial pivoting (largest |pivot| of the column by its upper
// word, 20 bits of mantissa, first row on ties; rows stay in place and keep
// their scale, the unknowns are divided out at the end).  The augmented p x (p + 1) system lives in
// registers, RT x CT elements per thread (row ty + 16 i, column tx + TX j); a
// step passes through shared memory only the column, its multipliers (one
// division per row, all rows at once) and the pivot row, with two barriers (elimination in shared memory had five, and two more per
// back-substituted unknown), and every warp finds the pivot for itself.  Bound
// by the latency of that chain, p steps of about 2,100 clocks for the two CTAs of an SM: 1,608 systems
// of 98: 656 us (in shared memory 1,299 us; divisions at the pivot row, 7 in
// turn per thread, 873 us).
constexpr int STY = 16;
template <typename F, int... I>
__device__ __forceinline__ void for_columns(F& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}

template <int RT, int CT, int TX>
__global__ void __launch_bounds__(STY * TX, STY * TX <= 256 ? 2 : 1) k_p_solve(const double* __restrict__ gram, const double* __restrict__ tot,
                                                      int nb, int q, double* __restrict__ sol) {
    __shared__ double col[2][STY * RT], mult[STY * RT], row[TX * CT];
    __shared__ int var_of[STY * RT];   // unknown whose pivot a row was
    __shared__ double piv[STY * RT];   // and that pivot
    const int b = blockIdx.x, j = blockIdx.y;
    const int p = q - 1;
    const size_t qq = (size_t)q * q;
    const double* T = tot + (size_t)j * qq;
    const double* G = b < nb ? gram + ((size_t)j * nb + b) * qq : nullptr;
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX, lane = threadIdx.x & 31;
    double M[RT][CT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int c = 0; c < CT; c++) {
            const int r = ty + STY * i, x = tx + TX * c;
            M[i][c] = 0.0;
            if (r < p && x <= p) {   // column p: X'y, the Gram's last column
                const size_t e = (size_t)r * q + x;
                M[i][c] = G ? T[e] - G[e] : T[e];
            }
        }
    constexpr int PER = (STY * RT + 31) / 32;   // rows per lane of the pivot search
    uint32_t used = 0;                          // bit u: row lane + 32 u has been a pivot
    // columns TX cb .. TX cb + TX - 1, whose register index is cb
    auto eliminate = [&](auto cb_c) __attribute__((always_inline)) {
        constexpr int cb = decltype(cb_c)::value;
        for (int ci = 0; ci < TX; ci++) {
            const int c = TX * cb + ci;
            if (c >= p) break;
            double* cbuf = col[c & 1];
            if (tx == ci) {
#pragma unroll
                for (int i = 0; i < RT; i++) cbuf[ty + STY * i] = M[i][cb];
            }
            __syncthreads();
            uint32_t best = 0;   // upper word of |value| + 1 (0: no free row)
            int bu = 0;
#pragma unroll
            for (int u = 0; u < PER; u++) {
                const int r = lane + 32 * u;
                if (r < p && !(used >> u & 1u)) {
                    const uint32_t v = ((uint32_t)__double2hiint(cbuf[r]) & 0x7FFFFFFFu) + 1u;
                    if (v > best) {
                        best = v;
                        bu = u;
                    }
                }
            }
            // first row among the lanes' largest: rows are lane + 32 u, so the smallest u first
            const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, best);
            const uint32_t cand = best == top ? (uint32_t)(lane + 32 * bu) : 0xFFFFu;
            const int pr = (int)__reduce_min_sync(0xFFFFFFFFu, cand);   // (a free row: c < p rows have been taken)
            if (lane == (pr & 31)) used |= 1u << (pr >> 5);
            if (ty == pr % STY) {
#pragma unroll
                for (int x = cb; x < CT; x++) {
                    double v = M[0][x];   // selects: a register array has no index
#pragma unroll
                    for (int i = 1; i < RT; i++) v = ty + STY * i == pr ? M[i][x] : v;
                    row[tx + TX * x] = v;
                }
            }
            const double d = cbuf[pr];
            if (threadIdx.x < STY * RT)
                mult[threadIdx.x] = threadIdx.x == pr ? 0.0 : cbuf[threadIdx.x] / d;
            if (threadIdx.x == 0) {
                var_of[pr] = c;
                piv[pr] = d;
            }
            __syncthreads();
            double rv[CT];
#pragma unroll
            for (int x = cb; x < CT; x++) rv[x] = row[tx + TX * x];
#pragma unroll
            for (int i = 0; i < RT; i++) {
                const double mr = mult[ty + STY * i];
#pragma unroll
                for (int x = cb; x < CT; x++) M[i][x] = fma(-mr, rv[x], M[i][x]);
            }
        }
    };
    for_columns(eliminate, std::make_integer_sequence<int, CT>{});
    double* out = sol + ((size_t)j * (nb + 1) + b) * p;
#pragma unroll
    for (int x = 0; x < CT; x++)
        if (tx + TX * x == p) {
#pragma unroll
            for (int i = 0; i < RT; i++)
                if (ty + STY * i < p) out[var_of[ty + STY * i]] = M[i][x] / piv[ty + STY * i];
        }
}

// Estimates, delete values, jackknife covariance and the h2 figures of each
// job.  res[j]: [est p][cov p x p][delete values nb x p][h2 per annotation k]
// [h2_total, h2_total_se, intercept, intercept_se, nbar, mean_chi2, n_obs].
// k_p_cov: a share of the covariance per CTA (blockIdx.y; the first also writes
// the estimates and delete values); k_p_finish: the rest.
__global__ void __launch_bounds__(NT) k_p_cov(const double* __restrict__ sol, int nb, int k, int p,
                                             double* __restrict__ res) {
    extern __shared__ double mean[];  // p pseudo-value means
    const int j = blockIdx.x, share = blockIdx.y, shares = gridDim.y;
    const double* S = sol + (size_t)j * (nb + 1) * p;
    const double* est = S + (size_t)nb * p;
    double* R = res + (size_t)j * part_result_len(nb, k, p);
    double* o_est = R;
    double* o_cov = o_est + p;
    double* o_dv = o_cov + (size_t)p * p;
    const double fnb = (double)nb;
    for (int c = threadIdx.x; c < p; c += NT) {
        if (share == 0) o_est[c] = est[c];
        double sm = 0.0;
        for (int b = 0; b < nb; b++) sm += fnb * est[c] - (fnb - 1.0) * S[(size_t)b * p + c];
        mean[c] = sm / fnb;
    }
    if (share == 0)
        for (size_t e = threadIdx.x; e < (size_t)nb * p; e += NT) o_dv[e] = S[e];
    __syncthreads();
    // jackknife_se_cov: centred pseudo-values, cov = C'C / ((nb - 1) nb)
    const double scale = (fnb - 1.0) * fnb;
    for (int e = share * NT + threadIdx.x; e < p * p; e += NT * shares) {
        const int r = e / p, c = e % p;
        if (r > c) continue;
        double acc = 0.0;
        for (int b = 0; b < nb; b++) {
            const double pr = fnb * est[r] - (fnb - 1.0) * S[(size_t)b * p + r] - mean[r];
            const double pc = fnb * est[c] - (fnb - 1.0) * S[(size_t)b * p + c] - mean[c];
            acc = fma(pr, pc, acc);
        }
        const double v = scale > 0.0 ? acc / scale : acc;
        o_cov[(size_t)r * p + c] = v;
        o_cov[(size_t)c * p + r] = v;
    }
}

__global__ void __launch_bounds__(NT) k_p_finish(const PartJob* __restrict__ jobs, const PartState* __restrict__ st,
                                                const double* __restrict__ sol, const double* __restrict__ m_vec,
                                                int nb, int k, int p, double* __restrict__ res) {
    __shared__ double red[NT / 32];
    const int j = blockIdx.x;
    const PartJob jb = jobs[j];
    const PartState s = st[j];
    const double* est = sol + ((size_t)j * (nb + 1) + nb) * p;
    double* o_cov = res + (size_t)j * part_result_len(nb, k, p) + p;
    double* o_h2 = o_cov + (size_t)p * p + (size_t)nb * p;
    double* o_sc = o_h2 + k;
    // total h2 and its SE (total_from_jknife, src/regressions.rs:1565-1610)
    double tv = 0.0;
    for (int e = threadIdx.x; e < k * k; e += NT) {
        const int r = e / k, c = e % k;
        tv += m_vec[r] * m_vec[c] * (o_cov[(size_t)r * p + c] / (s.nbar * s.nbar));
    }
    tv = block_sum(tv, red);
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int c = 0; c < k; c++) {
            const double h = est[c] / s.nbar * m_vec[c];
            o_h2[c] = h;
            tot += h;
        }
        o_sc[0] = tot;
        o_sc[1] = sqrt(fmax(tv, 0.0));
        o_sc[2] = jb.fixed ? jb.fixed_int : est[k];
        o_sc[3] = jb.fixed ? NAN : sqrt(fmax(o_cov[(size_t)k * p + k], 0.0));
        o_sc[4] = s.nbar;
        o_sc[5] = s.mean_chi2;
        o_sc[6] = s.n_obs;
    }
}

}  // namespace

cudaError_t launch_partitioned(const PartJob* jobs, PartState* st, const double* l2, uint64_t ld, int k, bool fixed,
                               const double* wld, uint64_t n, int nb, double m_tot, const double* m_vec, double* xtot,
                               bool want_xtot, double* part, double* gram, double* tot, double* sol, double* res,
                               int njobs, cudaStream_t s) {
    const int p = part_params(k, fixed), q = p + 1;
    const int upc = GWARPS / part_ksplit(q), gram_ctas = (part_units(q) + upc - 1) / upc;
    const size_t gram_smem = part_gram_smem(q);
    if (p > 160) return cudaErrorInvalidValue;
    if (want_xtot) {
        const uint64_t g = (n + NT - 1) / NT;
        k_p_xtot<<<(unsigned)(g < 148 * 8 ? g : 148 * 8), NT, 0, s>>>(l2, ld, k, n, xtot);
    }
    k_p_sums<<<dim3(nb, njobs), NT, 0, s>>>(jobs, xtot, nb, part);
    k_p_aggregate<<<(njobs + 3) / 4, 128, 0, s>>>(jobs, part, nb, m_tot, st, njobs);
    k_p_gram<<<dim3(nb, gram_ctas, njobs), NT, gram_smem, s>>>(jobs, st, l2, ld, k, xtot, wld, m_tot, nb, q,
                                                               part_unit_order(q), gram);
    k_p_total<<<dim3((q * q + NT - 1) / NT, njobs), NT, 0, s>>>(gram, nb, q * q, tot);
    const dim3 sgrid(nb + 1, njobs);
    if (p <= 31)
        k_p_solve<2, 2, 16><<<sgrid, 256, 0, s>>>(gram, tot, nb, q, sol);
    else if (p <= 63)
        k_p_solve<4, 4, 16><<<sgrid, 256, 0, s>>>(gram, tot, nb, q, sol);
    else if (p <= 111)
        k_p_solve<7, 7, 16><<<sgrid, 256, 0, s>>>(gram, tot, nb, q, sol);
    else
        k_p_solve<10, 6, 32><<<sgrid, 512, 0, s>>>(gram, tot, nb, q, sol);
    k_p_cov<<<dim3(njobs, 16), NT, (size_t)p * sizeof(double), s>>>(sol, nb, k, p, res);
    k_p_finish<<<njobs, NT, 0, s>>>(jobs, st, sol, m_vec, nb, k, p, res);
    return cudaGetLastError();
}

cudaError_t preload_partitioned() {
    cudaError_t e = preload_kernel(k_p_xtot);
    if (e == cudaSuccess) e = preload_kernel(k_p_sums);
    if (e == cudaSuccess) e = preload_kernel(k_p_aggregate);
    if (e == cudaSuccess) e = preload_kernel(k_p_gram);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_p_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)part_gram_smem(161));
    if (e == cudaSuccess) e = preload_kernel(k_p_total);
    if (e == cudaSuccess) e = preload_kernel(k_p_solve<2, 2, 16>);
    if (e == cudaSuccess) e = preload_kernel(k_p_solve<4, 4, 16>);
    if (e == cudaSuccess) e = preload_kernel(k_p_solve<7, 7, 16>);
    if (e == cudaSuccess) e = preload_kernel(k_p_solve<10, 6, 32>);
    if (e == cudaSuccess) e = preload_kernel(k_p_cov);
    if (e == cudaSuccess) e = preload_kernel(k_p_finish);
    return e;
}

}  // namespace ldsc
