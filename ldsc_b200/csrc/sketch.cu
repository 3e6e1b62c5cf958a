// sketch.cu -- CountSketch projection of BED rows (HBM-bound).
//
// Reference (src/wasm_simd.rs:1617-1784 via src/l2/compute.rs:601-770): per
// SNP, out[bucket[i]] += sign[i] * (g_i - mean) * inv_std over individuals i
// (missing -> 0), in f32, then out *= sqrt(N / sum(out^2)) with the squared
// norm accumulated in f64.
//
// Linearity gives, per bucket b,
//     out_b = inv_std * (S1_b - mean * S0_b)
//     S1_b  = sum_{i in b, present} sign_i g_i,   S0_b = sum_{i in b, present} sign_i,
// two integer sums.  The bucket/sign map is the same for every SNP, so the
// individuals are put once into bucket-major order (bucket, then sign):
// k_sketch_permute rewrites every panel row in that order (bit-plane quads of
// 64 positions, sketch_quad.cuh), after which each (bucket, sign) group is a
// contiguous run of positions.  k_sketch_row (rows too long for it:
// k_sketch_seg) then reads a permuted row once and forms the bucket sums from
// popcount prefix sums at the run boundaries; the same popcounts give the
// per-SNP moments.
//
// mean / inv_std are the reference's f32-rounded values; each bucket value is
// formed exactly and rounded to f32 once (the reference accumulates f32 in
// individual order; the two agree to f32 rounding).  The per-SNP moments
// (n, s, q, and the 3rd/4th for the MAF-aware correction) are permutation
// invariant and are produced by the same pass.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "sketch_quad.cuh"
#include "sm100.cuh"

namespace ldsc {

namespace {

constexpr int NT = 256;

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Rewrite panel rows in bucket-major individual order, as bit-plane quads
// (sketch_quad.cuh).  perm[p] = FAM index of the individual at permuted
// position p (p < n_used); positions past n_used read as missing.  One CTA per
// row, the row staged in shared memory when it fits (smem_row != 0).  A warp
// forms 32 halves (32 positions each) per step: for half h lane l reads the
// code at position 32 h + l (coalesced perm loads, eight halves' loads in
// flight), two ballots give the half's low-plane and high-plane words, and
// lane t keeps half t's pair, so the step ends in one coalesced 256-byte store.
__global__ void __launch_bounds__(NT) k_sketch_permute(PanelView p, const int32_t* __restrict__ perm,
                                                       uint64_t n_used, uint32_t* __restrict__ out,
                                                       uint64_t out_pitch_words, int smem_row) {
    extern __shared__ uint32_t srow32[];
    const uint8_t* srow = reinterpret_cast<const uint8_t*>(srow32);
    const uint64_t halves = out_pitch_words / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = NT / 32;
    for (uint64_t r = blockIdx.x; r < p.n_snp; r += gridDim.x) {
        const uint8_t* row = p.rows + r * p.pitch;
        if (smem_row) {
            const uint4* src = reinterpret_cast<const uint4*>(row);
            uint4* dst = reinterpret_cast<uint4*>(srow32);
            for (uint64_t q = threadIdx.x; q < p.pitch / 16; q += NT) dst[q] = __ldg(src + q);
            __syncthreads();
        }
        const uint8_t* from = smem_row ? srow : row;
        uint2* orow = reinterpret_cast<uint2*>(out + r * out_pitch_words);
        for (uint64_t g0 = (uint64_t)warp * 32; g0 < halves; g0 += NW * 32) {
            uint32_t my_lo = 0, my_hi = 0;
#pragma unroll 8
            for (int t = 0; t < 32; t++) {
                const uint64_t h = g0 + t;  // the same in every lane
                if (h >= halves) break;
                const uint64_t pos = h * 32 + lane;
                uint32_t code = 1u;  // missing
                if (pos < n_used) {
                    const int32_t iid = __ldg(perm + pos);
                    code = (from[iid >> 2] >> ((iid & 3) * 2)) & 3u;
                }
                const uint32_t lo = __ballot_sync(0xFFFFFFFFu, code & 1u);
                const uint32_t hi = __ballot_sync(0xFFFFFFFFu, code >> 1);
                if (lane == t) {
                    my_lo = lo;
                    my_hi = hi;
                }
            }
            if (g0 + lane < halves) orow[g0 + lane] = make_uint2(my_lo, my_hi);
        }
        __syncthreads();
    }
}

// ---- streaming form: any row length ----
//
// Bucket sums from prefix sums.  Over any span of positions (quad counts in
// sketch_quad.cuh)  sum g = 2 len - bits - missing  and  present = len -
// missing.  With the prefix (sum g, present) at every run boundary k, bucket
// b is
//     S1_b = (PF[2b+1] - PF[2b]) - (PF[2b+2] - PF[2b+1])   (g sums; S0_b with present)
// and row moments come from the totals:
//     n = present, s = sum g, q = s + 2 #2, q3 = s + 6 #2, q4 = s + 14 #2
// (#2 = number of genotype-2 codes = len - high bits - missing).
//
// Two phases per record.  (1) Streaming: each warp owns a contiguous block of
// the row's 16-byte quads and walks it 64 quads at a time, two adjacent quads
// per lane (coalesced loads, branch-free popcounts); one warp scan of the
// packed (bits, missing) counts gives the prefix at the start of every quad,
// kept in shared memory.  (2) Boundaries: after a block scan over the warps,
// thread t of T takes the buckets [d t / T, d (t+1) / T) and walks their
// boundaries in order; each prefix is the quad prefix, plus the offset of the
// warp that streamed the quad, plus popcounts inside the quad (re-read from
// L1/L2).  Thread t's boundary positions come from a thread-major table built
// once per layout (entry i * T + t = its i-th boundary, with the owning warp
// in the top bits), so their loads are coalesced.  Each bucket's value is
// formed on the spot.  No atomics, and nothing needs clearing between
// records.
template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

constexpr int SNT = 128;       // threads of the sketch kernels
constexpr int S6T = 256;       // and for large d (sketch_large_d)
constexpr int CHUNK_Q = 64;    // quads per warp step (2 per lane)

__host__ __device__ inline uint64_t sketch_quads(uint64_t n_used) { return ((n_used + 15) / 16 + 3) / 4; }

// Thread t of a T-thread CTA takes buckets [seg_b(d, t), seg_b(d, t + 1)):
// 2 (b1 - b0) + 1 boundaries; seg_rows bounds that count over t.
template <int T>
__host__ __device__ inline uint32_t seg_b(uint32_t d, uint32_t t) { return (uint32_t)((uint64_t)d * t / T); }
template <int T>
__host__ __device__ inline uint32_t seg_count(uint32_t d, uint32_t t) {
    const uint32_t b0 = seg_b<T>(d, t), b1 = seg_b<T>(d, t + 1);
    return b0 < b1 ? 2 * (b1 - b0) + 1 : 0;
}
template <int T>
__host__ __device__ inline uint32_t seg_rows(uint32_t d) { return 2 * ((d + T - 1) / T) + 1; }

// Boundary table entry of the streaming-form kernel: position | owning warp << 28.
constexpr int SEG_POS_BITS = 28;
constexpr int32_t SEG_POS_MASK = (1 << SEG_POS_BITS) - 1;

// Dynamic shared memory of the sketch kernel: per-quad prefixes (an even
// count, so the bucket values start on 16 bytes) and the d bucket values
// (+16 bytes read past d by the vector output loop).
__host__ __device__ inline size_t sketch_smem(uint64_t n_used, uint32_t d) {
    return 8 * ((sketch_quads(n_used) + 1) & ~1ull) + 4 * (size_t)d + 16;
}

// Record r's output from the bucket values ob (16-byte aligned): `ld` floats
// (zero padded past d), or with split the tensor-core operand rows
// 2r = tf32(v) and 2r+1 = tf32(v - tf32(v)), stored four at a time (ld is a
// multiple of 32 there).
template <int T>
__device__ __forceinline__ void write_sketch_row(const float* ob, uint32_t d, float scale, int split, float* orow,
                                                 uint64_t ld) {
    if (split) {
        float4* h4 = reinterpret_cast<float4*>(orow);
        float4* l4 = reinterpret_cast<float4*>(orow + ld);
        const float4* o4 = reinterpret_cast<const float4*>(ob);
        for (uint32_t v = threadIdx.x; v < (uint32_t)(ld / 4); v += T) {
            float4 x = 4 * v < d ? o4[v] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (4 * v + 4 > d) {   // past d: zero (what was read there is not a bucket)
                x.y = 4 * v + 1 < d ? x.y : 0.f;
                x.z = 4 * v + 2 < d ? x.z : 0.f;
                x.w = 0.f;
            }
            const float e[4] = {x.x, x.y, x.z, x.w};
            float hi[4], lo[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float val = e[k] * scale;
                hi[k] = to_tf32(val);
                lo[k] = to_tf32(val - hi[k]);
            }
            h4[v] = make_float4(hi[0], hi[1], hi[2], hi[3]);
            l4[v] = make_float4(lo[0], lo[1], lo[2], lo[3]);
        }
    } else {
        for (uint64_t b = threadIdx.x; b < ld; b += T) orow[b] = b < d ? ob[b] * scale : 0.f;
    }
}

// One CTA per record (grid-stride over records).  Output row r: `ld` floats
// (zero padded past d), or with split the hi/lo tensor-core rows 2r / 2r+1.
template <int T>
__global__ void __launch_bounds__(T, 1024 / T) k_sketch_seg(const uint32_t* __restrict__ pp, uint64_t pp_pitch_words,
                                                    const uint64_t* __restrict__ rec_rows, int64_t m, uint64_t n_used,
                                                    const int32_t* __restrict__ segt, uint32_t d, RecStats st,
                                                    int want_moments, int split, float* __restrict__ out,
                                                    uint64_t ld) {
    constexpr int W = T / 32;
    extern __shared__ __align__(16) int32_t sh[];
    const uint32_t quads = (uint32_t)sketch_quads(n_used);  // the permuted pitch is 4 quads' worth of words, padded
    int2* Pq = reinterpret_cast<int2*>(sh);                  // (popc, missing) before each quad, warp-relative
    float* ob = reinterpret_cast<float*>(sh + 2 * ((quads + 1) & ~1u));  // bucket values
    __shared__ int32_t wa[W], wm[W], wt[W];
    __shared__ int2 woff[W];  // (bits, missing) before each warp's block
    __shared__ double dred[W], rconst[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t wq0 = (uint32_t)((uint64_t)quads * warp / W), wq1 = (uint32_t)((uint64_t)quads * (warp + 1) / W);
    const uint32_t b0 = seg_b<T>(d, threadIdx.x), nbd = seg_count<T>(d, threadIdx.x);
    const int32_t row_len = (int32_t)(64 * quads);
    for (int64_t r = blockIdx.x; r < m; r += gridDim.x) {
        const uint64_t brow = rec_rows ? rec_rows[r] : (uint64_t)r;
        const uint4* row = reinterpret_cast<const uint4*>(pp + brow * pp_pitch_words);
        // ---- phase 1: stream the warp's quads ----
        int32_t carryA = 0, carryM = 0, HT = 0;
        uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;
        if (wq0 + 2 * lane < wq1) n0 = __ldg(row + wq0 + 2 * lane);
        if (wq0 + 2 * lane + 1 < wq1) n1 = __ldg(row + wq0 + 2 * lane + 1);
        for (uint32_t c0 = wq0; c0 < wq1; c0 += CHUNK_Q) {
            const uint32_t qa = c0 + 2 * lane;
            const bool l0 = qa < wq1, l1 = qa + 1 < wq1;
            const uint4 v0 = n0, v1 = n1;
            if (qa + CHUNK_Q < wq1) n0 = __ldg(row + qa + CHUNK_Q);
            if (qa + CHUNK_Q + 1 < wq1) n1 = __ldg(row + qa + CHUNK_Q + 1);
            int32_t a0, m0, h0, a1, m1, h1;
            quad_counts(v0, a0, m0, h0);
            quad_counts(v1, a1, m1, h1);
            const int32_t la = (l0 ? a0 : 0) + (l1 ? a1 : 0), lm = (l0 ? m0 : 0) + (l1 ? m1 : 0);
            HT += (l0 ? h0 : 0) + (l1 ? h1 : 0);
            // (bits, missing) packed in 16-bit halves: a chunk holds at most
            // 64 quads x 128 bits = 8,192, so the halves cannot carry
            const int32_t lp = la | (lm << 16);
            const int32_t ip = warp_incl_scan(lp, lane);
            const int32_t ia = ip & 0xFFFF, im = ip >> 16;
            const int32_t ea = carryA + ia - la, em = carryM + im - lm;
            if (l0) Pq[qa] = make_int2(ea, em);
            if (l1) Pq[qa + 1] = make_int2(ea + a0, em + m0);
            const int32_t tp = __shfl_sync(0xFFFFFFFFu, ip, 31);
            carryA += tp & 0xFFFF;
            carryM += tp >> 16;
        }
        const int32_t htw = warp_sum(HT);
        if (lane == 0) {
            wa[warp] = carryA;
            wm[warp] = carryM;
            wt[warp] = htw;
        }
        __syncthreads();
        // ---- block scan over the warps: offsets and row totals ----
        int32_t A = 0, MS = 0, H = 0;
#pragma unroll
        for (int w = 0; w < W; w++) {
            A += wa[w];
            MS += wm[w];
            H += wt[w];
        }
        // padding positions are missing: no effect on G and N, and TT = #2
        const int32_t G = 2 * row_len - A - MS, N = row_len - MS, TT = row_len - H - MS;
        if (threadIdx.x == 0) {
            st.n[r] = N;
            st.s[r] = G;
            st.q[r] = G + 2 * TT;
            if (want_moments && st.q3) {
                st.q3[r] = G + 6 * TT;
                st.q4[r] = G + 14 * TT;
            }
        }
        // normalize_col_f32_with_stats constants (src/l2/normalize.rs:115-154),
        // formed once and read by every thread after the barrier below
        if (threadIdx.x == 0) {
            const double dmean = N > 0 ? (double)G / (double)N : 0.0;
            const double css = (double)(G + 2 * TT) - (double)N * dmean * dmean;
            const double sd = sqrt(css / (double)n_used);
            rconst[0] = (double)(float)dmean;
            rconst[1] = sd > 0.0 ? (double)(float)(1.0 / sd) : 0.0;
        }
        if (threadIdx.x < W) {
            int32_t oa = 0, om = 0;
#pragma unroll
            for (int w = 0; w < W - 1; w++)
                if (w < (int)threadIdx.x) {
                    oa += wa[w];
                    om += wm[w];
                }
            woff[threadIdx.x] = make_int2(oa, om);
        }
        __syncthreads();
        const double mean = rconst[0], inv = rconst[1];
        // ---- phase 2: this thread's buckets ----
        // Boundaries in groups of four: the group's table entries are loaded
        // one group ahead and its four quads are loaded together.
        double part = 0.0;
        if (nbd) {
            int32_t pn[4];
#pragma unroll
            for (int u = 0; u < 4; u++) pn[u] = (uint32_t)u < nbd ? __ldg(segt + u * T + threadIdx.x) : row_len;
            int32_t g1 = 0, n1w = 0, g2 = 0, n2w = 0;  // prefixes at the previous two boundaries
            for (uint32_t i = 0; i < nbd; i += 4) {
                int32_t pc[4];
                uint4 qv[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    pc[u] = pn[u];
                    pn[u] = i + 4 + u < nbd ? __ldg(segt + (i + 4 + u) * T + threadIdx.x) : row_len;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int32_t p = pc[u] & SEG_POS_MASK;
                    qv[u] = p < row_len ? __ldg(row + (p >> 6)) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (i + u >= nbd) break;
                    const int32_t p = pc[u] & SEG_POS_MASK;
                    int32_t pg = G, pnr = N;  // at or past the row end: the totals
                    if (p < row_len) {
                        // quad prefix + offset of the warp that streamed the quad + inside the quad
                        const int2 pq = Pq[p >> 6], of = woff[(uint32_t)pc[u] >> SEG_POS_BITS];
                        int32_t ha, hm;
                        quad_head(qv[u], (uint32_t)p & 63u, ha, hm);
                        const int32_t pa = pq.x + of.x + ha, pm = pq.y + of.y + hm;
                        pg = 2 * p - pa - pm;
                        pnr = p - pm;
                    }
                    const uint32_t idx = i + u;
                    if (idx >= 2 && !(idx & 1)) {  // bucket b0 + idx/2 - 1 is complete
                        const int32_t s1 = (g1 - g2) - (pg - g1), s0 = (n1w - n2w) - (pnr - n1w);
                        const float o = (float)(inv * ((double)s1 - mean * (double)s0));
                        ob[b0 + idx / 2 - 1] = o;
                        part += (double)o * (double)o;
                    }
                    g2 = g1;
                    n2w = n1w;
                    g1 = pg;
                    n1w = pnr;
                }
            }
        }
        part = warp_sum(part);
        if (lane == 0) dred[warp] = part;
        __syncthreads();
        double nrm = 0.0;
#pragma unroll
        for (int w = 0; w < W; w++) nrm += dred[w];
        const float scale = nrm > 0.0 ? (float)sqrt((double)n_used / nrm) : 1.0f;
        write_sketch_row<T>(ob, d, scale, split, out + (uint64_t)r * (split ? 2 : 1) * ld, ld);
        __syncthreads();  // Pq, ob, wa and dred are rewritten by the next record
    }
}

// ---- row form: the row in shared memory, one stretch of it per thread ----
//
// Thread t counts quads [cq t, cq (t + 1)) of the staged row one after the
// other and leaves the counts so far before every quad (DENSE: before every
// word of 32 positions), so only the T stretch totals need a scan (the
// streaming form scans every 64 quads).  cq is odd: the stretches' shared loads
// and stores then meet no bank twice.  Counts are sum g + 65536 * present, one
// 32-bit number modulo 2^32: a bucket is a difference of prefixes, exact while
// its runs are at most SKETCH_MAX_RUN long.  A prefix is the stretch's offset
// (DENSE: added to the stored counts, there being more boundaries than words) +
// the stored count + the head of the quad (word) that holds the boundary, three
// popcounts per word.  A lane takes a bucket, neighbours share a boundary by
// shuffle, and their shared loads hit neighbouring words.  The row comes by
// 16-byte asynchronous copies, the next one once the boundaries are done, while
// other CTAs of the SM work.  The order of the norm's sum is the streaming
// form's, and so are the results, bit for bit.
// Bound by instruction issue and the popcount unit: 4,050 warp instructions per
// record of 100,000 individuals at d = 200 (streaming form 5,900), 17,300 at
// d = 5,000 (29,300 for an earlier form with the row in shared memory, prefixes
// per half quad and a thread per stretch of buckets, whose loads met banks).
// Measured: 50,000 records of 100,000 individuals, d = 200: 341 us (streaming
// form 410; reading the rows takes 190); 60,007 of 20,000, d = 1,000: 337 us
// (584); 20,011 of 100,000, d = 5,000: 513 us (the earlier form 724).
constexpr uint32_t SKETCH_MAX_RUN = 16383;

// Row length at which 256 threads stop (32 bytes per quad and 4 per bucket in 200 KB).
__host__ __device__ inline size_t sketch6_smem(uint64_t n_used, uint32_t d) {
    return 32 * sketch_quads(n_used) + 4 * (size_t)d + 16;
}
// Quads per thread: odd, and together more than the row's.
template <int T>
__host__ __device__ inline uint32_t sketch_cq(uint64_t n_used) {
    return (uint32_t)(sketch_quads(n_used) / T + 1) | 1u;
}
// Quads, stored counts, bucket values (+16 bytes read past d).
template <int T, bool DENSE>
__host__ __device__ inline size_t sketch_row_smem(uint64_t n_used, uint32_t d) {
    return (size_t)(16 + (DENSE ? 8 : 4)) * T * sketch_cq<T>(n_used) + ((4 * (size_t)d + 31) & ~(size_t)15);
}

// Boundary tables.  Streaming form, thread-major: entry i * T + t = the i-th
// boundary position of thread t (0x7FFFFFFF past its count) | owning warp << 28,
// the warp whose block holds the position's quad.
template <int T>
__global__ void k_sketch_segt(const int32_t* __restrict__ seg_off, uint32_t d, uint32_t rows, uint32_t quads,
                              int32_t* __restrict__ segt) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < rows * T; e += gridDim.x * blockDim.x) {
        const uint32_t i = e / T, t = e % T;
        int32_t v = 0x7FFFFFFF;
        if (i < seg_count<T>(d, t)) {
            v = seg_off[2 * seg_b<T>(d, t) + i];
            const uint64_t q = (uint64_t)v >> 6;
            int32_t w = 0;
            for (int o = 1; o < T / 32; o++)
                if (q >= (uint64_t)quads * o / (T / 32)) w = o;
            v |= w << SEG_POS_BITS;
        }
        segt[e] = v;
    }
}

// Row form: pair 0 = (0, 0), pair 1 + b = the run change inside bucket b and its
// end; each a position, with cq (not DENSE) | the thread that counts it << 24.
__global__ void k_sketch_rowt(const int32_t* __restrict__ seg_off, uint32_t d, uint32_t cq,
                              int32_t* __restrict__ segt) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < 2 * (d + 1); e += gridDim.x * blockDim.x) {
        const uint32_t v = e < 2 ? 0u : (uint32_t)seg_off[e - 1];
        segt[e] = (int32_t)(cq ? v | (v / 64 / cq) << 24 : v);
    }
}

// Counts of one word's positions under mask k: sum g, and #2 in two.
__device__ __forceinline__ uint32_t word_count(uint32_t lo, uint32_t hi, uint32_t k, uint32_t& twos) {
    twos = __popc(~lo & ~hi & k);
    return (__popc(~lo & k) + twos) + 65536u * __popc((~lo | hi) & k);
}

template <int T, bool DENSE>
__global__ void __launch_bounds__(T, 1024 / T) k_sketch_row(const uint32_t* __restrict__ pp, uint64_t pp_pitch_words,
                                                         const uint64_t* __restrict__ rec_rows, int64_t m,
                                                         uint64_t n_used, const int32_t* __restrict__ segt, uint32_t d,
                                                         RecStats st, int want_moments, int split,
                                                         float* __restrict__ out, uint64_t ld) {
    constexpr int W = T / 32;
    constexpr int PW = DENSE ? 2 : 1;   // stored counts per quad
    extern __shared__ __align__(16) uint4 shr[];
    const uint32_t quads = (uint32_t)sketch_quads(n_used), cq = sketch_cq<T>(n_used);
    uint32_t* P = reinterpret_cast<uint32_t*>(shr + (size_t)T * cq);
    float* ob = reinterpret_cast<float*>(P + PW * (size_t)T * cq);   // bucket values
    __shared__ uint32_t toff[DENSE ? 1 : T];                         // counts before each thread's stretch
    __shared__ uint32_t wv[W], wg[W], wn[W], wt[W];
    __shared__ double dred[W], rconst[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t b0 = seg_b<T>(d, threadIdx.x), b1 = seg_b<T>(d, threadIdx.x + 1);
    auto fetch = [&](int64_t r) {
        const uint64_t brow = rec_rows ? rec_rows[r] : (uint64_t)r;
        const uint4* row = reinterpret_cast<const uint4*>(pp + brow * pp_pitch_words) + threadIdx.x;
        uint32_t dst = smem_u32(shr + threadIdx.x);
#pragma unroll 4
        for (uint32_t q = threadIdx.x; q < quads; q += T, row += T, dst += 16 * T)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(row) : "memory");
    };
    // past the row: missing, no part of any count
    for (uint32_t q = quads + threadIdx.x; q < T * cq; q += T) shr[q] = make_uint4(~0u, 0u, ~0u, 0u);
    fetch(blockIdx.x);   // (grid <= m)
    // the warp's buckets [w0, w1), a lane each; pairs[b] opens with the bucket before it
    const uint2* pairs = reinterpret_cast<const uint2*>(segt) + 1;
    const uint32_t w0 = seg_b<W>(d, warp), w1 = seg_b<W>(d, warp + 1);
    const uint32_t first = __ldg(segt + 2 * w0 + 1);
    for (int64_t r = blockIdx.x; r < m; r += gridDim.x) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // ---- the thread's stretch ----
        uint32_t V = 0, TW = 0;
        uint32_t* pre = P + PW * threadIdx.x * cq;
        {
            const uint4* row = shr + threadIdx.x * cq;
#pragma unroll 4
            for (uint32_t i = 0; i < cq; i++) {
                const uint4 v = row[i];
                uint32_t t0, t1;
                const uint32_t v0 = V + word_count(v.x, v.y, ~0u, t0);
                if (DENSE)
                    reinterpret_cast<uint2*>(pre)[i] = make_uint2(V, v0);
                else
                    pre[i] = V;
                V = v0 + word_count(v.z, v.w, ~0u, t1);
                TW += t0 + t1;
            }
        }
        const uint32_t iv = (uint32_t)warp_incl_scan((int32_t)V, lane);
        const uint32_t rg = __reduce_add_sync(0xFFFFFFFFu, V & 0xFFFFu), rn = __reduce_add_sync(0xFFFFFFFFu, V >> 16);
        TW = __reduce_add_sync(0xFFFFFFFFu, TW);
        if (lane == 31) {
            wv[warp] = iv;
            wg[warp] = rg;
            wn[warp] = rn;
            wt[warp] = TW;
        }
        __syncthreads();
        {
            uint32_t o = iv - V;
#pragma unroll
            for (int x = 0; x < W - 1; x++)
                if (x < warp) o += wv[x];
            if (DENSE) {
                uint2* p2 = reinterpret_cast<uint2*>(pre);
#pragma unroll 4
                for (uint32_t i = 0; i < cq; i++) {
                    const uint2 v = p2[i];
                    p2[i] = make_uint2(v.x + o, v.y + o);
                }
            } else {
                toff[threadIdx.x] = o;
            }
        }
        if (threadIdx.x == 0) {
            int32_t G = 0, N = 0, TT = 0;   // sum g, present, #2
#pragma unroll
            for (int x = 0; x < W; x++) {
                G += (int32_t)wg[x];
                N += (int32_t)wn[x];
                TT += (int32_t)wt[x];
            }
            st.n[r] = N;
            st.s[r] = G;
            st.q[r] = G + 2 * TT;
            if (want_moments && st.q3) {
                st.q3[r] = G + 6 * TT;
                st.q4[r] = G + 14 * TT;
            }
            // normalize_col_f32_with_stats constants (src/l2/normalize.rs:115-154)
            const double dmean = N > 0 ? (double)G / (double)N : 0.0;
            const double css = (double)(G + 2 * TT) - (double)N * dmean * dmean;
            const double sd = sqrt(css / (double)n_used);
            rconst[0] = (double)(float)dmean;
            rconst[1] = sd > 0.0 ? (double)(float)(1.0 / sd) : 0.0;
        }
        __syncthreads();
        // ---- the warp's buckets ----
        if (w0 < w1) {
            const double mean = rconst[0], inv = rconst[1];
            auto prefix = [&](uint32_t e) {
                uint32_t t0, t1;
                if (DENSE) {   // e: the position
                    const uint2 x = reinterpret_cast<const uint2*>(shr)[e >> 5];
                    return P[e >> 5] + word_count(x.x, x.y, (1u << (e & 31u)) - 1u, t0);
                }
                const uint32_t q = (e & 0xFFFFFFu) >> 6, k = (1u << (e & 31u)) - 1u;
                const bool second = e & 32u;
                const uint4 x = shr[q];
                return P[q] + toff[e >> 24] + word_count(x.x, x.y, second ? ~0u : k, t0) +
                       word_count(x.z, x.w, second ? k : 0u, t1);
            };
            // |n| < 2^31 as a double without the conversion unit, which the popcounts keep busy
            auto to_double = [](int32_t n) {
                return __hiloint2double(0x43300000, n ^ (int32_t)0x80000000) - 4503601774854144.0;   // 2^52 + 2^31
            };
            uint2 next = w0 + lane < w1 ? __ldg(pairs + w0 + lane) : make_uint2(first, first);
            uint32_t vc = prefix(first);   // at the boundary before lane 0's bucket
            for (uint32_t bw = w0; bw < w1; bw += 32) {
                const uint32_t b = bw + lane;
                const uint2 e = next;
                if (b + 32 < w1) next = __ldg(pairs + b + 32);
                const uint32_t v1 = prefix(e.x), v2 = prefix(e.y);
                const uint32_t vu = __shfl_up_sync(0xFFFFFFFFu, v2, 1);
                const uint32_t x = 2 * v1 - (lane ? vu : vc) - v2;   // S1_b + 65536 S0_b
                vc = __shfl_sync(0xFFFFFFFFu, v2, 31);
                const int32_t s1 = (int16_t)x, s0 = (int32_t)(x - (uint32_t)s1) >> 16;
                const float o = (float)(inv * (to_double(s1) - mean * to_double(s0)));
                if (b < w1) ob[b] = o;
            }
        }
        __syncthreads();
        if (r + gridDim.x < m) fetch(r + gridDim.x);   // (the padding stays)
        // the squared norm, each thread over its own buckets
        double part = 0.0;
#pragma unroll 4
        for (uint32_t b = b0; b < b1; b++) {
            const double o = (double)ob[b];
            part += o * o;
        }
        part = warp_sum(part);
        if (lane == 0) dred[warp] = part;
        __syncthreads();
        double nrm = 0.0;
#pragma unroll
        for (int x = 0; x < W; x++) nrm += dred[x];
        const float scale = nrm > 0.0 ? (float)sqrt((double)n_used / nrm) : 1.0f;
        write_sketch_row<T>(ob, d, scale, split, out + (uint64_t)r * (split ? 2 : 1) * ld, ld);
        // (the next record writes ob, toff and the sums behind the barrier that opens it or a later one)
    }
}

}  // namespace

// 256 threads, and with them the order of the norm's sum, for large d.
static bool sketch_large_d(uint64_t n_used, uint32_t d) { return d >= 2560 && sketch6_smem(n_used, d) <= 200 * 1024; }

// Row-form CTAs of an SM by shared memory.
static int64_t sketch_ctas(size_t smem_row, int threads) {
    return std::min<int64_t>(1024 / threads, 227 * 1024 / (int64_t)(smem_row + 1024 + 4 * threads + 256));
}

// Counts before every word where there are enough boundaries to use them, unless
// the longer table leaves fewer than four CTAs.  Measured, ns per record with
// and without: N = 50,000, d = 500: 5.3, 6.0; N = 100,000, d = 1,000: 10.7, 11.6,
// d = 500: 8.8, 8.6; N = 150,000, d = 1,000: 16.4, 14.2; N = 200,000, d = 2,500:
// 37, 29.  (Large d: always, quads being at most 2.5 d there.)
static bool sketch_dense(uint64_t n_used, uint32_t d) {
    return sketch_large_d(n_used, d) ||
           (4 * (uint64_t)d > sketch_quads(n_used) && sketch_ctas(sketch_row_smem<SNT, true>(n_used, d), SNT) >= 4);
}

static size_t sketch_row_bytes(uint64_t n_used, uint32_t d) {
    return sketch_large_d(n_used, d)  ? sketch_row_smem<S6T, true>(n_used, d)
           : sketch_dense(n_used, d) ? sketch_row_smem<SNT, true>(n_used, d)
                                     : sketch_row_smem<SNT, false>(n_used, d);
}

// The row form while two CTAs fit an SM.  Measured, ns per record, row form and
// streaming form: N = 20,000, d = 200: 3.3, 4.8, d = 5,000: 22, 36; N = 100,000,
// d = 200: 7.3, 8.7, d = 5,000: 26, 40; N = 300,000, d = 500: 25.5, 29.7; with one
// CTA N = 400,000, d = 500: 47.5, 43.7; N = 300,000, d = 2,600: 51.6, 41.0.
static bool sketch_row_form(uint64_t n_used, uint32_t d, uint32_t max_run) {
    if (max_run > SKETCH_MAX_RUN) return false;
    return sketch_ctas(sketch_row_bytes(n_used, d), sketch_large_d(n_used, d) ? S6T : SNT) >= 2;
}

cudaError_t launch_sketch_permute(const PanelView& p, const int32_t* perm, uint64_t n_used, uint32_t* out,
                                  uint64_t out_pitch_words, cudaStream_t stream) {
    if (p.n_snp == 0) return cudaSuccess;
    int smem_row = p.pitch <= 160 * 1024 ? 1 : 0;
    size_t smem = smem_row ? p.pitch : 0;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sketch_permute, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    uint64_t grid = p.n_snp < 148 * 16 ? p.n_snp : 148 * 16;
    k_sketch_permute<<<(unsigned)grid, NT, smem, stream>>>(p, perm, n_used, out, out_pitch_words, smem_row);
    return cudaGetLastError();
}

cudaError_t launch_sketch_seg(const uint32_t* pp, uint64_t pp_pitch_words, const uint64_t* rec_rows, int64_t m,
                              uint64_t n_used, const int32_t* segt, uint32_t d, uint32_t max_run, RecStats st,
                              int want_moments, int split, float* out, uint64_t ld, cudaStream_t stream) {
    if (m <= 0) return cudaSuccess;
    const bool large = sketch_large_d(n_used, d);
    if (sketch_row_form(n_used, d, max_run)) {
        const bool dense = sketch_dense(n_used, d);
        const auto kernel = large ? k_sketch_row<S6T, true> : (dense ? k_sketch_row<SNT, true> : k_sketch_row<SNT, false>);
        const size_t smem_row = sketch_row_bytes(n_used, d);
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_row);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        const int t = large ? S6T : SNT;
        const int64_t fit = 148 * sketch_ctas(smem_row, t);
        kernel<<<(unsigned)(m < fit ? m : fit), t, smem_row, stream>>>(pp, pp_pitch_words, rec_rows, m, n_used, segt,
                                                                       d, st, want_moments, split, out, ld);
        return cudaGetLastError();
    }
    const size_t smem = sketch_smem(n_used, d);
    if (smem > 200 * 1024) return cudaErrorInvalidValue;  // rejected by the caller first (ldsc_sketch_supported)
    const auto kernel = large ? k_sketch_seg<S6T> : k_sketch_seg<SNT>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int64_t grid = m < 148 * 16 ? m : 148 * 16;
    kernel<<<(unsigned)grid, large ? S6T : SNT, smem, stream>>>(pp, pp_pitch_words, rec_rows, m, n_used, segt, d, st,
                                                               want_moments, split, out, ld);
    return cudaGetLastError();
}

bool sketch_supported(uint64_t n_used, uint32_t d) { return sketch_smem(n_used, d) <= 200 * 1024; }

uint64_t sketch_segt_count(uint64_t n_used, uint32_t d, uint32_t max_run) {
    return sketch_row_form(n_used, d, max_run) ? 2 * ((uint64_t)d + 1)
           : sketch_large_d(n_used, d)           ? (uint64_t)seg_rows<S6T>(d) * S6T
                                                 : (uint64_t)seg_rows<SNT>(d) * SNT;
}

cudaError_t launch_sketch_segt(const int32_t* seg_off, uint64_t n_used, uint32_t d, uint32_t max_run, int32_t* segt,
                               cudaStream_t stream) {
    const uint32_t quads = (uint32_t)sketch_quads(n_used);
    if (sketch_row_form(n_used, d, max_run))
        k_sketch_rowt<<<64, 256, 0, stream>>>(seg_off, d, sketch_dense(n_used, d) ? 0 : sketch_cq<SNT>(n_used), segt);
    else if (sketch_large_d(n_used, d))
        k_sketch_segt<S6T><<<64, 256, 0, stream>>>(seg_off, d, seg_rows<S6T>(d), quads, segt);
    else
        k_sketch_segt<SNT><<<64, 256, 0, stream>>>(seg_off, d, seg_rows<SNT>(d), quads, segt);
    return cudaGetLastError();
}

cudaError_t preload_sketch() {
    cudaError_t e = preload_kernel(k_sketch_permute);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_seg<SNT>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_seg<S6T>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_row<SNT, false>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_row<SNT, true>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_row<S6T, true>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_segt<SNT>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_segt<S6T>);
    if (e == cudaSuccess) e = preload_kernel(k_sketch_rowt);
    return e;
}

}  // namespace ldsc
