// gram_tc.cu -- band Gram on the 5th-generation tensor cores (tcgen05), in
// two operand kinds that share one tile structure:
//   * INT8-exact form (kind::i8): genotype / mask rows, exact epilogue;
//   * CountSketch form (kind::tf32): each sketched f32 value v is split as
//     v = hi + lo with hi = tf32(v), lo = tf32(v - hi), stored as rows 2r (hi)
//     and 2r+1 (lo); one UMMA then yields hi.hi, hi.lo, lo.hi, lo.lo for every
//     pair, whose sum is the f32-accurate dot product (the reference's f32
//     GEMM, src/l2/compute.rs:1897-2079), followed by the quadratic bias
//     inversion (src/l2/compute.rs:947-998) in f64.
//
// INT8-exact form:
// Operands: for record r, row 2r holds its genotypes G (0/1/2, 0 at missing)
// and row 2r+1 its non-missing mask M (0/1), one byte per individual, rows of
// `ld` bytes (a multiple of 128).  A tile is 128 left records k by 128 right
// records j over K = individuals: two UMMAs per K step (A = the G rows, then
// the M rows, of the left records; B = 128 G rows and 128 M rows of the right
// ones) with INT32 accumulation in TMEM, which yields for every record pair
// the four integer products
//     GG = sum G_k G_j,  GM = sum G_k M_j,  MG = sum M_k G_j,  MM = sum M_k M_j.
// With n, s, q the per-record non-missing count, genotype sum and sum of
// squares, the reference's standardised dot product (normalize.rs:71-110
// followed by the A^T B GEMM, compute.rs:1897-2236) is recovered exactly:
//     X   = n_k (n_j GG - s_j GM) + s_k (s_j MM - n_j MG)         (int64, exact)
//     r^2 = X^2 / (n_k V_k n_j V_j),  V = n q - s^2              (f64)
//     r2u = r^2 (1 + 1/(N-2)) - 1/(N-2)                           (f64)
// N cancels from r; a monomorphic record (V = 0) gives r = 0 and
// r2u = -1/(N-2), as the reference's zero inv_std does.
//
// What bounds it and why this tile: per K step of 128 bytes an SM takes in
// A 32 KB + B 32 KB and multiplies 256 x 256 rows: 1,024 clocks of tensor
// work, 1,047 measured (50,000 individuals).  A 64 x 128 record tile (48 KB for
// 128 x 256 rows) took 776 clocks for 512 of tensor work -- the 64 bytes per
// clock an SM takes in, not the tensor pipe, set its pace; the four Gram
// launches of a 50,000 x 100,000 pass went from 13.4 to 11.6 ms.
//
// Kernel structure (persistent, one CTA per SM):
//   warp 0     TMA producer: per stage four boxes of 128 rows x 128 B (left G,
//              left M, right G, right M), 128-byte swizzle; the tensor map
//              splits the interleaved rows into (parity, record), so a box
//              holds one kind of row
//   warp 1     TMEM allocator (512 columns: two 128 x 256 accumulators, rows G
//              and M of the left records) and UMMA issuer (M=128 N=256)
//   epilogue   16 warps (8 in the fused form).  A thread owns one left record
//              and finds its pair's four products in its own TMEM lane (two
//              accumulators x two column halves), so no lane exchange forms
//              r; the right records' constants are read as broadcasts from
//              shared memory, a row's sum stays in its thread, and a column's
//              sum over the warp's 32 rows is a transposing butterfly (9 f64
//              shuffles per 8 columns).  f64 instructions and tcgen05.mma share
//              one pipe of the SM (an f64 instruction beside running MMAs waits
//              about 20 clocks), so they are kept few: five per pair in a block
//              that lies inside the band (X to double, X^2, row and column
//              terms, butterfly), with 1/(nV) of the row, the column and the
//              constant -1/(N-2) applied to the sums: about 10,000
//              clocks per tile, 13 f64 instructions per pair before (sketch: 12,000
//              with the f32 root and quotient of sqrt_nr and div_nr, 19,000 with
//              the IEEE ones and their branches; 50,000 records, d = 200: 378 -> 315
//              us per launch).
//              With K > 1 annotation columns the epilogue stores each tile's
//              masked r2u values (f64, [j][k]) for the contraction of
//              contract.cu.
// The accumulators fill TMEM, so a tile's epilogue does not overlap the next
// tile's MMAs (its loads do).  Half tiles (64 right records) with two
// accumulator buffers were slower even at 7 K steps: the epilogue's f64
// instructions then wait for the other buffer's MMAs.
//
// Fused INT8 form (the operand rows are never written to HBM): warp 0 stages
// the packed 2-bit BED rows themselves by TMA -- 32 bytes per record per 128
// individuals, 8 KB per stage for the 128 + 128 records of a tile instead of
// 64 KB of operand rows -- and eight converter warps expand each packed stage
// in shared memory into the 128-byte-swizzled G / M operand tiles the MMA warp
// reads, with a proxy fence before they hand the stage over.  The K order of
// individuals inside a 16-byte chunk is permuted (evens, then odds) the same
// way in every row, which leaves every product sum unchanged; individuals past
// N read as missing.
//
// Every mbarrier wait is bounded; on timeout the kernel records an error word,
// drains its own in-flight copies / MMAs (bounded), frees TMEM and returns.
#include <cuda.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "approx.cuh"
#include "engine.h"
#include "epilogue.cuh"
#include "expand.cuh"
#include "sm100.cuh"

namespace ldsc {

namespace {

constexpr int TA = 128;            // left records per tile
constexpr int TB = 128;            // right records per tile
constexpr int HALF = 128 * 128;    // 128 operand rows (one kind) x 128 bytes
constexpr int QROWS = TILE_QUARTER * 128;   // 32 operand rows x 128 bytes
constexpr int A_BYTES = 2 * HALF;  // one stage of A: G rows, then M rows
constexpr int B_BYTES = 2 * HALF;
// fused form: packed ring of 2-bit rows, 128 individuals (32 bytes) per record per stage
constexpr int P_STAGES = 4;
constexpr int PA_BYTES = TA * 32;
constexpr int P_BYTES = (TA + TB) * 32;
// operand stages, epilogue and converter warps of the two forms (576 threads
// either way); the fused form's packed ring leaves room for two operand stages
constexpr int STAGES_TMA = 3, EPI_TMA = 16;
// Long rows (from LONG_STEPS K steps) run 8 epilogue warps: the epilogue is a
// few percent there, and 320 threads leave the registers for three blocks of
// the decode that runs beside the Gram (576 threads: one).  At 50,000 x
// 100,000 with whole tiles a pass took 13.22 ms on the device, with 16 epilogue
// warps 13.39 ms; 15,003 kept individuals x 50,021 records (118 steps) 2.38
// against 2.50 ms.
constexpr int EPI_LONG = 8, LONG_STEPS = 100;
constexpr int STAGES_FUSED = 2, EPI_FUSED = 8, CONV_FUSED = 8;
// threads per CTA: TMA and MMA warps + ew epilogue warps + cw converter warps
__host__ __device__ constexpr int gram_threads(int ew, int cw) { return 64 + 32 * ew + 32 * cw; }
// every form is compiled for the 576 threads of the widest (112 registers at most)
constexpr int GRAM_BOUND = 576;
constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;  // 2 s per wait

// Sums over the warp's 32 lanes of 8 values per lane: lane l ends with the sum
// of value 4 (l / 16) + 2 (l / 8 % 2) + l / 4 % 2.  Each of the first three
// steps halves the values a lane holds, so 9 shuffles do what 8 butterflies
// would take 40 for.
__device__ __forceinline__ double transpose_sum8(const double (&c)[8], int lane) {
    double d[4], e[2];
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; i++)
        d[i] = (b4 ? c[4 + i] : c[i]) + __shfl_xor_sync(0xFFFFFFFFu, b4 ? c[i] : c[4 + i], 16);
#pragma unroll
    for (int i = 0; i < 2; i++)
        e[i] = (b3 ? d[2 + i] : d[i]) + __shfl_xor_sync(0xFFFFFFFFu, b3 ? d[i] : d[2 + i], 8);
    double f = (b2 ? e[1] : e[0]) + __shfl_xor_sync(0xFFFFFFFFu, b2 ? e[0] : e[1], 4);
    f += __shfl_xor_sync(0xFFFFFFFFu, f, 2);
    f += __shfl_xor_sync(0xFFFFFFFFu, f, 1);
    return f;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Whether an annotation may enter a block's sums ahead of the pair's mask and
// of r^2's other factors: 0, or of a size (2^-700 .. 2^700) that neither
// overflows nor loses bits there.  A negative exponent of p q makes it inf at a
// monomorphic record, and a column may hold inf or NaN: 0 x inf of a masked pair
// would reach records outside the window.
__device__ __forceinline__ bool plain_annot(double a) {
    return a == 0.0 || ((uint32_t)__double2hiint(a) & 0x7FFFFFFFu) - (323u << 20) < (1400u << 20);
}

// Right-record constants and partial sums of the tile being finished
// (double-buffered: a tile's sums leave while the next tile starts).
struct EpiTile {
    double2 qa[TB];        // (INT8: 1 / (n V) | sketch: kappa), effective annotation (K = 1)
    double qw[TB];         // INT8: 1 / (n V) x effective annotation
    int4 ns[TB];           // INT8: n, -s, s, -n (non-missing count, genotype sum)
    int64_t left[TB];      // left limit (m past the last record)
    double cpart[4][TB];   // column sums per TMEM lane quarter
    double rpart[4][TA];   // row sums per column group
};

// 1.5 * 2^52: an integer |x| < 2^51 plus its bits, read as a double, is this
// constant plus x exactly.
constexpr uint64_t INT_MAGIC = 0x4338000000000000ull;
// X fits that way while n^3 < 2^51 (|X| <= n_k V_k n_j V_j's root <= N^3)
constexpr double MAGIC_MAX_N = 131072.0;

// MODE 0: INT8 exact r^2; 1: TF32 sketch, quadratic correction; 2: same, MAF-aware.
// kap: kappa_k + kappa_j (MAF-aware).
template <int MODE>
__device__ __forceinline__ double sketch_r2u(float val, double kap, const EpilogueArgs& ep) {
    const double v = (double)val;
    const double tilde = v * v * ep.n_inv_sq;
    const double dm3 = ep.sketch_d - 3.0 - 2.0 * kap;
    const double disc = dm3 * dm3 + 8.0 * (ep.sketch_d * tilde - 1.0);
    const double r2 = disc >= 0.0 ? (-dm3 + sqrt(disc)) * 0.25 : 0.0;
    return r2 * ep.r2u_a + ep.r2u_b;
}

// Sketch constants in f32 for sketch_r2u_f32.
struct SketchF {
    float n_inv_sq, d, r2u_a, r2u_b;
};

// sketch_r2u in f32, for d >= 8 (then dm3 > 2 - 2 kappa > 0 and the
// discriminant is positive): the root (-dm3 + sqrt(disc)) / 4 is taken in the
// cancellation-free form 2 q / (sqrt(disc) + dm3), q = d tilde - 1 (the same
// value: disc - dm3^2 = 8 q).  Its absolute error is about ulp(d tilde) / dm3,
// 3e-10 at d = 200, against the reference's f64 evaluation; l2 sums of a
// thousand such terms move by ~1e-7 relative, far inside the sketch's own
// f32 dot-product error.  Each pair's value depends on that pair alone, so
// runs over different tile grids (slices, shards) still agree to f64
// rounding of the sums.
template <int MODE>
__device__ __forceinline__ float sketch_r2u_f32(float val, double kap2, const SketchF& cf) {
    const float kap = MODE == 2 ? (float)kap2 : 0.f;
    const float tilde = val * val * cf.n_inv_sq;
    const float dm3 = cf.d - 3.f - 2.f * kap;
    const float q = fmaf(cf.d, tilde, -1.f);
    const float disc = fmaf(dm3, dm3, 8.f * q);
    float r2;
    if (MODE == 1 || dm3 >= 4.f)   // disc >= dm3^2 - 8 >= 8 (not MAF-aware: dm3 >= 5)
        r2 = div_nr(2.f * q, sqrt_nr(disc) + dm3);
    else
        r2 = disc >= 0.f ? 2.f * q / (sqrtf(disc) + dm3) : 0.f;
    return fmaf(r2, cf.r2u_a, cf.r2u_b);
}

// CW = 0: A / B operand rows staged by TMA.  CW > 0 (INT8 only): packed 2-bit
// rows staged by TMA (the map covers the BED rows, boxes of 32 bytes x 128
// rows) and expanded by CW converter warps; n_indiv masks the last stage.
template <int STAGES, int MODE, int EW, int CW>
__global__ void __launch_bounds__(GRAM_BOUND, 1)
    k_gram_tc(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tmq, int num_kb, const Tile* __restrict__ tiles, int64_t n_tiles,
              EpilogueArgs ep, int32_t* __restrict__ dbg, int dbg_row, uint64_t n_indiv) {
    static_assert(CW == 0 || MODE == 0, "the fused form is INT8 only");
    // elements per 128-byte stage row: 128 (INT8) or 32 (TF32); TMA x is in elements
    constexpr int KSTEP = MODE == 0 ? 128 : 32;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
    uint8_t* smem = smem_raw + pad;
    uint8_t* sA = smem;
    uint8_t* sB = sA + STAGES * A_BYTES;
    uint8_t* sP = sB + STAGES * B_BYTES;   // fused form: packed ring
    uint64_t* full = reinterpret_cast<uint64_t*>(sP + (CW > 0 ? P_STAGES * P_BYTES : 0));
    uint64_t* empty = full + STAGES;
    uint64_t* pfull = empty + STAGES;   // [P_STAGES], fused form
    uint64_t* pempty = pfull + P_STAGES;
    uint64_t* tfull = pempty + P_STAGES;
    uint64_t* tempty = tfull + 1;
    uint64_t* drain = tempty + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    // 16-byte aligned: the barriers above take an even number of 8-byte words
    static_assert((2 * STAGES + 2 * P_STAGES + 4) % 2 == 0, "alignment of the epilogue arrays");
    EpiTile* epi = reinterpret_cast<EpiTile*>(drain + 2);   // [2]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], CW > 0 ? CW : 1);   // TMA transaction, or one arrival per converter warp
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < P_STAGES; s++) {
            mbar_init(&pfull[s], 1);
            mbar_init(&pempty[s], CW > 0 ? CW : 1);
        }
        mbar_init(tfull, 1);
        mbar_init(tempty, 32 * EW);
        mbar_init(drain, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (elect_one_sync()) {
            tma_prefetch_desc(&tm);
            if (CW == 0) tma_prefetch_desc(&tmq);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            uint32_t armed = 0;        // bit s: stage s has a load in flight we may need to drain
            uint32_t armed_par = 0;    // bit s: parity of that load's phase
            // the ring this warp fills: operand stages, or packed stages in the fused form
            constexpr int RING = CW > 0 ? P_STAGES : STAGES;
            uint64_t* rfull = CW > 0 ? pfull : full;
            uint64_t* rempty = CW > 0 ? pempty : empty;
            for (int64_t t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                const Tile tl = tiles[t];
                const int nq = (int)tl.nq1 + 1;
                const int32_t ra = (int32_t)tl.a_blk * TA, rb = (int32_t)(tl.b_blk * TB + tl.q0 * TILE_QUARTER);
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!mbar_wait(&rempty[stage], phase ^ 1, WAIT_LIMIT_NS)) {
                        ok = false;
                        break;
                    }
                    if constexpr (CW > 0) {
                        mbar_arrive_expect_tx(&rfull[stage], P_BYTES);
                        tma_load_2d(sP + stage * P_BYTES, &tm, &rfull[stage], kb * 32, ra);
                        tma_load_2d(sP + stage * P_BYTES + PA_BYTES, &tm, &rfull[stage], kb * 32, rb);
                    } else {
                        mbar_arrive_expect_tx(&rfull[stage], A_BYTES + nq * 2 * QROWS);
                        uint8_t* da = sA + stage * A_BYTES;
                        uint8_t* db = sB + stage * B_BYTES;
                        tma_load_3d(da, &tm, &rfull[stage], kb * KSTEP, 0, ra);
                        tma_load_3d(da + HALF, &tm, &rfull[stage], kb * KSTEP, 1, ra);
                        if (nq == 4) {
                            tma_load_3d(db, &tm, &rfull[stage], kb * KSTEP, 0, rb);
                            tma_load_3d(db + HALF, &tm, &rfull[stage], kb * KSTEP, 1, rb);
                        } else {   // the tile's quarters of the right block only
                            for (int q = 0; q < nq; q++) {
                                tma_load_3d(db + q * QROWS, &tmq, &rfull[stage], kb * KSTEP, 0, rb + q * TILE_QUARTER);
                                tma_load_3d(db + (nq + q) * QROWS, &tmq, &rfull[stage], kb * KSTEP, 1,
                                            rb + q * TILE_QUARTER);
                            }
                        }
                    }
                    armed |= 1u << stage;
                    armed_par = (armed_par & ~(1u << stage)) | (phase << stage);
                    if (++stage == RING) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) {
                atomicOr(ep.err, 1u);
                // our copies in flight must land before the CTA's smem is released
                for (int s = 0; s < RING; s++)
                    if (armed & (1u << s)) mbar_wait(&rfull[s], (armed_par >> s) & 1u, WAIT_LIMIT_NS);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ UMMA issuer
        if (elect_one_sync()) {
            int stage = 0;
            uint32_t phase = 0, aphase = 0;
            bool ok = true;
            bool issued = false;
            for (int64_t t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                if (!mbar_wait(tempty, aphase ^ 1, WAIT_LIMIT_NS)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t n2 = 64u * (tiles[t].nq1 + 1);   // the tile's right G rows and M rows
                const uint32_t idesc = MODE == 0 ? idesc_i8(128, n2) : idesc_tf32(128, n2);
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!mbar_wait(&full[stage], phase, WAIT_LIMIT_NS)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(sA + stage * A_BYTES);
                    const uint32_t b_addr = smem_u32(sB + stage * B_BYTES);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
#pragma unroll
                        for (int h = 0; h < 2; h++) {   // left G rows, left M rows
                            const uint64_t da = sdesc_k_sw128(a_addr + h * HALF + kk * 32);
                            const uint64_t db = sdesc_k_sw128(b_addr + kk * 32);
                            const uint32_t acc = (kb | kk) != 0 ? 1u : 0u;
                            const uint32_t d_tmem = tmem_base + h * 256u;
                            if (MODE == 0)
                                umma_i8(d_tmem, da, db, idesc, acc);
                            else
                                umma_tf32(d_tmem, da, db, idesc, acc);
                        }
                    }
                    issued = true;
                    umma_commit(&empty[stage]);
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit(tfull);
                aphase ^= 1;
            }
            if (!ok) atomicOr(ep.err, 2u);
            if (issued) {
                // all of this thread's MMAs complete before TMEM is freed
                umma_commit(drain);
                mbar_wait(drain, 0, WAIT_LIMIT_NS);
            }
        }
    } else if (CW > 0 && warp >= 2 + EW) {
        // ------------------------------------------------ converters (fused form)
        // Thread ct takes 16-individual word wd of the stage's packed rows for
        // records ct / 8 + RPP * i: the warp reads 128 contiguous packed bytes
        // per pass, and each 8-thread phase of a 16-byte store fills one whole
        // 128-byte operand row (no bank conflicts).
        constexpr int RPP = 32 * (CW > 0 ? CW : 1) / 8;   // records per pass
        constexpr int NPASS = (TA + TB) / RPP;
        constexpr int APASS = TA / RPP;              // passes that fill the A tile
        static_assert(CW == 0 || (RPP == TILE_QUARTER && TA % RPP == 0), "converter passes");
        const int ct = threadIdx.x - (64 + 32 * EW);
        const int wd = ct & 7;
        uint32_t offP[NPASS], offG[NPASS];
#pragma unroll
        for (int i = 0; i < NPASS; i++) {
            const int rr = (ct >> 3) + RPP * i;        // record slot: A 0..127, B 128..255
            offP[i] = (uint32_t)(rr * 32 + wd * 4);
            offG[i] = sw128_off(i < APASS ? rr : rr - TA, wd);
        }
        int os = 0, ps = 0;
        uint32_t oph = 0, pph = 0;
        bool ok = true;
        for (int64_t t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            // records past the last one read as missing (the map's zero fill would read as genotype 2)
            const Tile tl = tiles[t];
            const int nq = (int)tl.nq1 + 1;   // the right block's quarters; pass APASS + q fills quarter q
            uint32_t live = 0;
#pragma unroll
            for (int i = 0; i < NPASS; i++) {
                const int rr = (ct >> 3) + RPP * i;
                const int64_t rec = i < APASS ? (int64_t)tl.a_blk * TA + rr
                                              : (int64_t)tl.b_blk * TB + tl.q0 * TILE_QUARTER + (rr - TA);
                live |= (rec < ep.m ? 1u : 0u) << i;
            }
            for (int kb = 0; kb < num_kb; kb++) {
                // every lane waits (TMA data visible to each reader); the warp agrees on the outcome
                const bool got = mbar_wait(&pfull[ps], pph, WAIT_LIMIT_NS) &&
                                 mbar_wait(&empty[os], oph ^ 1, WAIT_LIMIT_NS);
                if (!__all_sync(0xFFFFFFFFu, got)) {
                    if (lane == 0) atomicOr(ep.err, 8u);
                    ok = false;
                    break;
                }
                const uint8_t* pk = sP + ps * P_BYTES;
                uint8_t* oa = sA + os * A_BYTES;
                uint8_t* ob = sB + os * B_BYTES;
                uint32_t w[NPASS];
#pragma unroll
                for (int i = 0; i < NPASS; i++)
                    w[i] = (live >> i) & 1u ? *reinterpret_cast<const uint32_t*>(pk + offP[i]) : 0x55555555u;
                const uint64_t i0 = (uint64_t)kb * 128 + (uint64_t)wd * 16;
                if (i0 + 16 > n_indiv) {
                    // individuals past N (and the zero fill past the row) read as missing
                    const uint32_t valid = n_indiv > i0 ? (uint32_t)(n_indiv - i0) : 0u;
                    const uint32_t keepm = (1u << (2 * valid)) - 1u;   // valid < 16 here
#pragma unroll
                    for (int i = 0; i < NPASS; i++) w[i] = (w[i] & keepm) | (0x55555555u & ~keepm);
                }
#pragma unroll
                for (int i = 0; i < NPASS; i++) {
                    if (i >= APASS + nq) break;
                    uint4 g, mk;
                    expand_chunk(w[i], g, mk);
                    uint8_t* base = i < APASS ? oa : ob;
                    *reinterpret_cast<uint4*>(base + offG[i]) = g;
                    *reinterpret_cast<uint4*>(base + (i < APASS ? HALF : nq * QROWS) + offG[i]) = mk;
                }
                // the generic-proxy stores must be visible to the tensor core's async proxy
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&full[os]);
                    mbar_arrive(&pempty[ps]);
                }
                if (++os == STAGES) {
                    os = 0;
                    oph ^= 1;
                }
                if (++ps == P_STAGES) {
                    ps = 0;
                    pph ^= 1;
                }
            }
        }
    } else {
        // ------------------------------------------------ epilogue
        constexpr int EPI_T = 32 * EW;           // epilogue threads
        constexpr int NG = 16 / EW;              // column groups (quarters of the tile's columns) per warp
        const int et = threadIdx.x - 64;         // 0..EPI_T-1
        const int ew = et >> 5;                  // epilogue warp
        const int quarter = warp & 3;            // TMEM lanes this warp may access
        const int row = quarter * 32 + lane;     // left record of the tile = TMEM lane
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const int64_t m = ep.m;
        const SketchF cf{(float)ep.n_inv_sq, (float)ep.sketch_d, (float)ep.r2u_a, (float)ep.r2u_b};
        const bool f32_corr = MODE != 0 && ep.sketch_d >= 8.0;
        const bool big = ep.n_used >= MAGIC_MAX_N;
        const uint64_t magic = big ? 0ull : INT_MAGIC;
        uint32_t aphase = 0, flip = 0;
        for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x, flip ^= 1) {
            EpiTile& E = epi[flip];
            const Tile tl = tiles[t];
            const int nq = (int)tl.nq1 + 1, ncol = nq * TILE_QUARTER;
            const int64_t k0 = (int64_t)tl.a_blk * TA, j0 = (int64_t)tl.b_blk * TB + tl.q0 * TILE_QUARTER;
            const int64_t k = k0 + row;
            const bool kval = k < m;
            const uint32_t nk = (MODE == 0 && kval) ? (uint32_t)__ldg(ep.n + k) : 0u;
            const uint32_t sk = (MODE == 0 && kval) ? (uint32_t)__ldg(ep.s + k) : 0u;
            // INT8: 1 / (n V) of the left record; MAF-aware sketch: its kappa
            double qk = !kval ? 0.0 : (MODE == 0 ? __ldg(ep.qinv + k) : (MODE == 2 ? __ldg(ep.kappa + k) : 0.0));
            if (MODE == 0) qk *= qk;
            const double ak = (kval && ep.K == 1) ? __ldg(ep.aeff + k) : 0.0;
            if (et < TB) {   // the right records' constants, while the tile's MMAs run
                const int64_t j = j0 + et;
                const bool jv = et < ncol && j < m;
                double qj = !jv ? 0.0 : (MODE == 0 ? __ldg(ep.qinv + j) : (MODE == 2 ? __ldg(ep.kappa + j) : 0.0));
                if (MODE == 0) qj *= qj;
                const double aj = (jv && ep.K == 1) ? __ldg(ep.aeff + j) : 0.0;
                E.qa[et] = make_double2(qj, aj);
                if (MODE == 0) E.qw[et] = qj * aj;
                if (MODE == 0) {
                    const int nj = jv ? __ldg(ep.n + j) : 0, sj = jv ? __ldg(ep.s + j) : 0;
                    E.ns[et] = make_int4(nj, -sj, sj, -nj);
                }
                E.left[et] = jv ? __ldg(ep.left + j) : m;
            }

            // One thread does the bounded wait; the decision is made uniform for
            // all epilogue threads through shared memory before anyone
            // continues, so no thread can be left waiting at a named barrier.
            volatile uint32_t* go = tmem_slot + 1;
            if (et == 0) *go = mbar_wait(tfull, aphase, WAIT_LIMIT_NS) ? 1u : 0u;
            named_bar_sync(2, EPI_T);
            if (*go == 0u) {
                if (et == 0) atomicOr(ep.err, 4u);
                break;
            }
            tc_fence_after();
            aphase ^= 1;
            const double a_rows = ep.K == 1 ? warp_sum(ak) : 0.0;   // annotation sum of the warp's rows
            const bool plain_rows = __all_sync(0xFFFFFFFFu, plain_annot(ak));
#pragma unroll 1
            for (int g = 0; g < NG; g++) {
                const int cg = (ew >> 2) * NG + g, c0 = cg * 8 * nq;   // columns [c0, c0 + 8 nq) of the tile
                // does the warp's 32 x 8 nq block hold any in-band pair, or only in-band pairs?
                const int64_t klo = k0 + quarter * 32;
                const int cl = c0 + (lane < 8 * nq ? lane : 0);
                const int64_t jl = j0 + cl, ll = E.left[cl];
                const int64_t lo = ll > klo ? ll : klo, hi = jl - 1 < klo + 31 ? jl - 1 : klo + 31;
                const bool any = __any_sync(0xFFFFFFFFu, jl < m && lo <= hi) || dbg != nullptr;
                const bool all = __all_sync(0xFFFFFFFFu, jl < m && ll <= klo && klo + 31 < jl);
                const bool plain = __all_sync(0xFFFFFFFFu, plain_annot(E.qa[cl].y)) && plain_rows;
                // K = 1, INT8, a block inside the band: sums of X^2 / (n V), scaled at the end
                const bool raw = MODE == 0 && all && plain && ep.K == 1 && dbg == nullptr;
                double rs[2] = {0.0, 0.0};
                double* rt = ep.K == 1 ? nullptr : ep.rtiles + ((size_t)ep.roff[t] * TILE_QUARTER + c0) * TA + row;
                if (!any) {
                    if (g == NG - 1) {
                        tc_fence_before();
                        mbar_arrive(tempty);
                    }
                    if (ep.K == 1)
                        E.cpart[quarter][cl] = 0.0;
                    else
                        for (int c = 0; c < 8 * nq; c++) rt[(size_t)c * TA] = 0.0;
                } else {
                    // WHAT 0: K = 1, raw; 1: K = 1; 2: K > 1; 3: K = 1, annotations that are not plain.
                    // F32: sketch, the f32 form of r2u
                    auto finish = [&](auto what, auto f32) {
                        constexpr int WHAT = decltype(what)::value;
                        constexpr bool F32 = decltype(f32)::value;
                        const double ck = WHAT == 0 ? qk * ak : qk * ep.r2u_a;
#pragma unroll 1
                        for (int ch = 0; ch < nq; ch++) {
                            const int cb = c0 + 8 * ch;
                            uint32_t v[4][8];   // GG, GM, MG, MM (sketch: hh, hl, lh, ll) of 8 columns
#pragma unroll
                            for (int x = 0; x < 4; x++)
                                tmem_ld_32x32b_x8(t_row + (uint32_t)((x >> 1) * 256 + (x & 1) * ncol + cb), v[x]);
                            tmem_ld_wait();
                            if (g == NG - 1 && ch == nq - 1) {
                                // this thread's part of the accumulators is read: hand them back to the MMA warp
                                tc_fence_before();
                                mbar_arrive(tempty);
                            }
                            if ((WHAT == 1 || WHAT == 3) && dbg != nullptr && row >= dbg_row && row < dbg_row + 64) {
#pragma unroll
                                for (int i = 0; i < 8; i++)
#pragma unroll
                                    for (int x = 0; x < 4; x++)
                                        dbg[(2 * (row - dbg_row) + (x >> 1)) * 256 + 2 * (cb + i) + (x & 1)] =
                                            (int32_t)v[x][i];
                            }
                            double cv[8];
#pragma unroll
                            for (int i = 0; i < 8; i++) {
                                double x2 = 0.0, r2u = 0.0;
                                if (MODE == 0) {
                                    const int4 ns = E.ns[cb + i];
                                    const int64_t pg = (int64_t)ns.x * (int32_t)v[0][i] + (int64_t)ns.y * (int32_t)v[1][i];
                                    const int64_t pm = (int64_t)ns.z * (int32_t)v[3][i] + (int64_t)ns.w * (int32_t)v[2][i];
                                    const uint64_t xb = (uint64_t)pg * nk + ((uint64_t)pm * sk + magic);
                                    const double X = big ? (double)(int64_t)xb
                                                         : __longlong_as_double((long long)xb) -
                                                               __longlong_as_double((long long)INT_MAGIC);
                                    x2 = X * X;
                                    if (WHAT != 0) r2u = fma(x2 * ck, E.qa[cb + i].x, ep.r2u_b);
                                } else {
                                    const float val = (__uint_as_float(v[0][i]) + __uint_as_float(v[1][i])) +
                                                      (__uint_as_float(v[2][i]) + __uint_as_float(v[3][i]));
                                    const double kap = MODE == 2 ? qk + E.qa[cb + i].x : 0.0;
                                    r2u = F32 ? (double)sketch_r2u_f32<MODE>(val, kap, cf)
                                              : sketch_r2u<MODE>(val, kap, ep);
                                }
                                if (WHAT == 0) {
                                    rs[i & 1] = fma(x2, E.qw[cb + i], rs[i & 1]);
                                    cv[i] = x2 * ck;
                                    continue;
                                }
                                bool in = true;
                                if (!all) {
                                    const int64_t j = j0 + cb + i;
                                    in = j < m && k < j && E.left[cb + i] <= k;
                                    if (!in) r2u = 0.0;
                                }
                                if (WHAT == 3) {   // masked pairs by the product
                                    rs[i & 1] = in ? fma(r2u, E.qa[cb + i].y, rs[i & 1]) : rs[i & 1];
                                    cv[i] = in ? r2u * ak : 0.0;
                                } else if (WHAT == 1) {
                                    rs[i & 1] = fma(r2u, E.qa[cb + i].y, rs[i & 1]);
                                    cv[i] = r2u * ak;
                                } else {
                                    // K > 1: the masked value goes to the tile's f64 slot (record j's row of
                                    // TA values) for the banded annotation contraction; a warp stores 256
                                    // contiguous bytes
                                    rt[(size_t)(8 * ch + i) * TA] = r2u;
                                }
                            }
                            if (WHAT != 2) {
                                double cs = transpose_sum8(cv, lane);
                                const int c = cb + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
                                if (WHAT == 0) cs = fma(cs * ep.r2u_a, E.qa[c].x, ep.r2u_b * a_rows);
                                if ((lane & 3) == 0) E.cpart[quarter][c] = cs;
                            }
                        }
                    };
                    auto finish_k = [&](auto f32) {
                        if (ep.K != 1)
                            finish(std::integral_constant<int, 2>{}, f32);
                        else if (MODE == 0 && raw)
                            finish(std::integral_constant<int, 0>{}, f32);
                        else if (!plain)
                            finish(std::integral_constant<int, 3>{}, f32);
                        else
                            finish(std::integral_constant<int, 1>{}, f32);
                    };
                    if (MODE != 0 && f32_corr)
                        finish_k(std::true_type{});
                    else
                        finish_k(std::false_type{});
                }
                if (ep.K == 1) {
                    double rsum = rs[0] + rs[1];
                    if (raw) {
                        const double a_cols = warp_sum(lane < 8 * nq ? E.qa[cl].y : 0.0);
                        rsum = fma(rsum * ep.r2u_a, qk, ep.r2u_b * a_cols);
                    }
                    E.rpart[cg][row] = rsum;
                }
            }
            if (ep.K == 1) {
                named_bar_sync(1, EPI_T);
                // per-tile sums in fixed order; launch_l2_reduce adds them to l2 (columns of the
                // right block that the tile leaves out are 0).  The next tile writes the other
                // buffer, and the one after it only past the barriers of the next.
                if (et < TA) {
                    const double rsum = E.rpart[0][et] + E.rpart[1][et] + E.rpart[2][et] + E.rpart[3][et];
                    if (ep.prow)
                        ep.prow[(size_t)t * TA + et] = rsum;
                    else if (k0 + et < m && rsum != 0.0)
                        atomicAdd(ep.l2 + k0 + et, rsum);
                } else if (et < TA + TB) {
                    const int cj = et - TA, c = cj - (int)tl.q0 * TILE_QUARTER;
                    const bool in = c >= 0 && c < ncol;
                    const double cs = in ? E.cpart[0][c] + E.cpart[1][c] + E.cpart[2][c] + E.cpart[3][c] : 0.0;
                    if (ep.prow)
                        ep.pcol[(size_t)t * TB + cj] = cs;
                    else if (in && j0 + c < m && cs != 0.0)
                        atomicAdd(ep.l2 + j0 + c, cs);
                }
            } else {
                // every thread has read this tile's wait decision before the next one is written
                named_bar_sync(1, EPI_T);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace

// Long rows keep whole tiles: the CTAs of a wave then walk K in step, and what
// one reads the others find in L2.  Trimmed tiles end early, the CTAs drift
// apart, and the wave's rows (about 25 blocks x 128 records x 2 rows) have to
// fit: 320 MB at 50,000 individuals, where a tile took 270 us among trimmed
// ones and 208 us among whole ones; 130 MB at sketch d = 5,000 (157 steps:
// 1,480 against 1,401 us per launch); 65 MB at 10,000 individuals (79 steps:
// 1,038 against 1,051 us).
constexpr uint64_t TRIM_STEPS = 100;
bool gram_trims(uint64_t row_bytes) { return row_bytes / 128 < TRIM_STEPS; }

using PFN_encodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                     const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                     const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                     CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode() {
    static PFN_encodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(p);
    }
    return fn;
}

// Map of the operand rows as (byte column, parity, record): row 2 r + p is
// (., p, r), so a box of records holds rows of one kind.
static bool make_map(CUtensorMap* map, const void* base, CUtensorMapDataType dt, uint64_t ld_elems,
                     uint64_t elem_bytes, uint64_t m, uint32_t box_records) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return false;
    cuuint64_t dims[3] = {ld_elems, 2, m};
    cuuint64_t strides[2] = {ld_elems * elem_bytes, 2 * ld_elems * elem_bytes};
    cuuint32_t box[3] = {(cuuint32_t)(128 / elem_bytes), 1, box_records};  // 128-byte rows
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

template <int STAGES, int MODE, int EW, int CW>
static cudaError_t run_tc(const CUtensorMap& tm, const CUtensorMap& tmq, int num_kb, const Tile* tiles, int64_t n_tiles,
                          const EpilogueArgs& ep, int32_t* dbg, int dbg_row, int sms, cudaStream_t stream,
                          uint64_t n_indiv = 0) {
    // alignment slack, operand (and packed) ring, barriers + TMEM slot words, epilogue arrays
    const size_t smem = 1024 + STAGES * (size_t)(A_BYTES + B_BYTES) + (CW > 0 ? (size_t)P_STAGES * P_BYTES : 0) +
                        8 * (2 * STAGES + 2 * P_STAGES + 4) + 2 * sizeof(EpiTile);
    cudaError_t e = cudaFuncSetAttribute(k_gram_tc<STAGES, MODE, EW, CW>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t grid = dbg ? 1 : (n_tiles < sms ? n_tiles : sms);
    k_gram_tc<STAGES, MODE, EW, CW><<<(unsigned)grid, gram_threads(EW, CW), smem, stream>>>(
        tm, tmq, num_kb, tiles, dbg ? 1 : n_tiles, ep, dbg, dbg_row, n_indiv);
    return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_tc(const void* ops, CUtensorMapDataType dt, uint64_t elem_bytes, uint64_t ld_elems,
                             int64_t m, const Tile* tiles, int64_t n_tiles, const EpilogueArgs& ep, int32_t* dbg,
                             int dbg_row, int sms, cudaStream_t stream) {
    if (n_tiles <= 0) return cudaSuccess;
    if ((ld_elems * elem_bytes) % 128 != 0 || (reinterpret_cast<uintptr_t>(ops) & 15) != 0)
        return cudaErrorInvalidValue;
    CUtensorMap tm, tmq;   // boxes of 128 records, and of 32 for a tile's quarters
    if (!make_map(&tm, ops, dt, ld_elems, elem_bytes, (uint64_t)m, 128) ||
        !make_map(&tmq, ops, dt, ld_elems, elem_bytes, (uint64_t)m, TILE_QUARTER))
        return cudaErrorInvalidValue;
    const int steps = (int)(ld_elems * elem_bytes / 128);
    if (MODE == 0 && steps >= LONG_STEPS)
        return run_tc<STAGES_TMA, 0, EPI_LONG, 0>(tm, tmq, steps, tiles, n_tiles, ep, dbg, dbg_row, sms, stream);
    return run_tc<STAGES_TMA, MODE, EPI_TMA, 0>(tm, tmq, steps, tiles, n_tiles, ep, dbg, dbg_row, sms, stream);
}

cudaError_t launch_gram_i8(const uint8_t* ops, uint64_t ld, int64_t m, const Tile* tiles, int64_t n_tiles,
                           const EpilogueArgs& ep, int32_t* dbg, int dbg_row, int sms,
                           cudaStream_t stream) {
    return launch_tc<0>(ops, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ld, m, tiles, n_tiles, ep, dbg, dbg_row, sms, stream);
}

// Map of the packed BED rows (record r at rows + r * pitch): boxes of 32 bytes
// (128 individuals) x 128 records, no swizzle (the converters read it with
// plain shared loads).  Bytes past the pitch read as zero.
static bool make_packed_map(CUtensorMap* map, const uint8_t* rows, uint64_t pitch, uint64_t m) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return false;
    cuuint64_t dims[2] = {pitch, m};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2] = {32, 128};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(rows), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

cudaError_t launch_gram_i8_packed(const uint8_t* rows, uint64_t pitch, uint64_t n_indiv, int64_t m, const Tile* tiles,
                                  int64_t n_tiles, const EpilogueArgs& ep, int32_t* dbg, int dbg_row,
                                  int sms, cudaStream_t stream) {
    if (n_tiles <= 0) return cudaSuccess;
    if (pitch % 16 != 0 || pitch < (n_indiv + 3) / 4 || n_indiv == 0 ||
        (reinterpret_cast<uintptr_t>(rows) & 15) != 0)
        return cudaErrorInvalidValue;
    CUtensorMap tm;
    if (!make_packed_map(&tm, rows, pitch, (uint64_t)m)) return cudaErrorInvalidValue;
    return run_tc<STAGES_FUSED, 0, EPI_FUSED, CONV_FUSED>(tm, tm, (int)((n_indiv + 127) / 128), tiles, n_tiles, ep, dbg,
                                                          dbg_row, sms, stream, n_indiv);
}

cudaError_t launch_gram_tf32(const float* ops, uint64_t ld, int64_t m, const Tile* tiles, int64_t n_tiles,
                             const EpilogueArgs& ep, int maf_aware, int sms, cudaStream_t stream) {
    if (maf_aware)
        return launch_tc<2>(ops, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ld, m, tiles, n_tiles, ep, nullptr, 0,
                            sms, stream);
    return launch_tc<1>(ops, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ld, m, tiles, n_tiles, ep, nullptr, 0,
                            sms, stream);
}

cudaError_t preload_gram_tc() {
    cudaError_t e = preload_kernel(k_gram_tc<STAGES_TMA, 0, EPI_TMA, 0>);
    if (e == cudaSuccess) e = preload_kernel(k_gram_tc<STAGES_TMA, 0, EPI_LONG, 0>);
    if (e == cudaSuccess) e = preload_kernel(k_gram_tc<STAGES_TMA, 1, EPI_TMA, 0>);
    if (e == cudaSuccess) e = preload_kernel(k_gram_tc<STAGES_TMA, 2, EPI_TMA, 0>);
    if (e == cudaSuccess) e = preload_kernel(k_gram_tc<STAGES_FUSED, 0, EPI_FUSED, CONV_FUSED>);
    return e;
}

}  // namespace ldsc
