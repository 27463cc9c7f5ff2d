// Bucketed RBF-kernel attention of the HEPT layer, with the gather into LSH order and the scatter
// back fused in.
//
// Reference (models/attention/hept.py:22-33 `qkv_res`, 141-152 of HEPTAttention.forward; copies in
// models/baselines/hmamba.py:49-60 and models/attention/flatformer.py:12-23): hits are sorted per
// (round, head) by their shifted LSH key, cut into buckets of `bucket` consecutive hits, and
// inside a bucket every query i sees every key j with weight
//     p_ij = exp(min(0, q_i . k_j - |q_i|^2 / 2 - |k_j|^2 / 2))        ( = exp(-|q_i - k_j|^2 / 2) )
//     denom_i = sum_j p_ij + 1e-20,      so_i = sum_j p_ij v_j
// after which the rows go back to hit order, the rounds are summed and so / denom is the output.
//
// One CTA per (round, head, bucket), CTAs ordered head by head so that the rounds of a head find its
// rows in L2.  Keys, values and queries of the bucket are gathered into shared memory once, by
// position, with asynchronous copies (16-byte pieces when the rows are padded to whole pieces, else
// 4-byte pieces); each warp then takes tiles of 4 query rows: it computes its 4 x 128 slice of p in
// registers (thread = 4 queries x 4 keys, operands read as 16-byte shared loads: 8 loads per 64
// FMAs), keeps the slice in a private shared tile and multiplies it with V (thread = 4 queries x 4
// value columns x a share of the keys).  The CTA has as many warps as finish the bucket's tiles in
// whole rounds (7 for buckets of 100); three CTAs per SM at the layer's usual sizes, so that one
// CTA's gather overlaps the others' arithmetic.  Arithmetic is fp32 FMA: the exponent is a
// difference of large terms, which a single tensor-core operand type cannot carry.
// Measured (60 000 hits, 3 rounds x 8 heads, buckets of 100, 30 + 24 features): the gather is what
// bounds the kernel - with 4-byte pieces the copy instructions alone took 17 k of a CTA's 52 k
// cycles (in-kernel counters), with 16-byte pieces and three CTAs per SM the kernel went from
// 1.40 ms to 0.97 ms.  Rows of at most 32 features in buckets of more than 32 take the tensor-core kernel
// further down (0.47 ms).
//
// HBM traffic per (round, head, hit): the q, k, v rows once and the so row + denom once.
#include "common.cuh"
#include "split3.cuh"
#include "profile.cuh"
#include <algorithm>

namespace lampa {

constexpr int BA_MAX_WARPS = 8;
constexpr int BA_MAX_BUCKET = 128;      // keys per bucket = one pass of 32 lanes x 4 keys

struct BucketAttnArgs {
    const float* q; const float* k; const float* v;         // [rounds?][heads][n][d]
    const int64_t* q_pos; const int64_t* k_pos;             // [rounds][heads][n] or NULL (rows already in order)
    float* so; float* denom;                                // [rounds][heads][n][dv], [rounds][heads][n]
    int64_t n;
    int64_t in_round_stride_q, in_round_stride_v;           // 0: q/k/v shared by all rounds (gathered by position)
    int rounds, heads, bucket, dq, dv;
    int ldq, ldv;        // floats between consecutive rows of q / k and of v
    int vec_qk, vec_v;   // rows can be fetched as 16-byte pieces (aligned base, pitch % 4 == 0, pitch >= width rounded up to 4)
    int dq4, pk, pv, nd; // dq rounded up to 4; key pitch (floats, pk / 4 odd); value pitch; value column groups of 4 per key share (power of 2)
    int qrows;           // bucket rounded up to whole tiles
    int scatter;         // 1: row i of a bucket is written to hit q_pos[i]; 0: to its sorted place
    int vec_store;       // so rows are 16-byte aligned: dv % 4 == 0 and an aligned base
    int32_t* status;
};

// The hits at place `at` of both orders of n hits (no orders: `own`).  One that leaves the hits is reported and stands for hit 0.
// Both loads are asked for before either is looked at, and no later step asks again (a query marked as not to be written, one at
// a time: 482 instead of 474 us for 60 000 hits, 3 x 8 orders, buckets of 100).
__device__ __forceinline__ void ba_positions(const BucketAttnArgs& a, int64_t at, int64_t own, int64_t& q, int64_t& k) {
    q = k = own;
    if (!a.q_pos) return;
    q = a.q_pos[at];
    k = a.k_pos[at];
    if ((uint64_t)q < (uint64_t)a.n && (uint64_t)k < (uint64_t)a.n) return;
    set_status(a.status, LAMPA_ERR_BOUNDS, 50, (int)own);
    if ((uint64_t)q >= (uint64_t)a.n) q = 0;
    if ((uint64_t)k >= (uint64_t)a.n) k = 0;
}

__host__ __device__ inline int ba_pow2_at_least(int x) { int p = 1; while (p < x) p <<= 1; return p; }

// shared memory (floats): sK [128][pk] | sV [128][pv] | sQ [qrows][dq4] | per warp sP [4][128]
// | positions: 2 x [128] int64
__host__ __device__ inline size_t ba_smem_floats(int dq4, int pk, int pv, int qrows, int warps, int BA_QROWS) {
    return (size_t)BA_MAX_BUCKET * pk + (size_t)BA_MAX_BUCKET * pv + (size_t)qrows * dq4 +
           (size_t)warps * BA_QROWS * BA_MAX_BUCKET + 4 * BA_MAX_BUCKET;
}

// 4-byte asynchronous copy global -> shared; `live` false writes a zero without reading
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool live) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = live ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool live) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// BA_QROWS: query rows per warp tile.  4 (80 registers, up to three CTAs per SM) while at least two CTAs'
// shared memory fits an SM; 8 (fewer operand loads per FMA) for wide rows, where one CTA has the SM to itself.
// Measured at 60 000 hits, 3 x 8: dq 54 / dv 48 1.25 ms with 4 rows against 1.62 with 8; dq 102 / dv 96 3.63 against 3.40.
template <int BA_QROWS>
__global__ void __launch_bounds__(BA_MAX_WARPS * 32, BA_QROWS == 4 ? 3 : 2) bucket_rbf_attn_kernel(BucketAttnArgs a) {
    if (chain_wait()) return;
    extern __shared__ __align__(16) float ba_smem[];
    const int dq4 = a.dq4, pk = a.pk, pv = a.pv, bucket = a.bucket;
    const int nthr = blockDim.x, nwarps = nthr >> 5;
    float* sK = ba_smem;                                            // [128][pk]
    float* sV = sK + (size_t)BA_MAX_BUCKET * pk;                    // [128][pv]
    float* sQ = sV + (size_t)BA_MAX_BUCKET * pv;                    // [qrows][dq4]
    float* sPall = sQ + (size_t)a.qrows * dq4;                      // per warp [4][128]
    int64_t* sQpos = reinterpret_cast<int64_t*>(sPall + (size_t)nwarps * BA_QROWS * BA_MAX_BUCKET);
    int64_t* sKpos = sQpos + BA_MAX_BUCKET;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    const int64_t nb = a.n / bucket;
    // CTAs run head by head, the rounds of a head back to back: a head's q, k and v rows (tens of MB)
    // are fetched from DRAM by the first round and found in L2 by the others.
    const int64_t b = blockIdx.x % nb, hc = blockIdx.x / nb;
    const int h = (int)(hc / a.rounds), c = (int)(hc % a.rounds);
    const int64_t rh = (int64_t)c * a.heads + h;                    // row of the positions and outputs
    const int64_t row0 = b * bucket;
    const float* qbase = a.q + c * a.in_round_stride_q + (size_t)h * a.n * a.ldq;
    const float* kbase = a.k + c * a.in_round_stride_q + (size_t)h * a.n * a.ldq;
    const float* vbase = a.v + c * a.in_round_stride_v + (size_t)h * a.n * a.ldv;

    for (int j = tid; j < BA_MAX_BUCKET; j += nthr) {
        int64_t q = 0, k = 0;
        if (j < bucket) ba_positions(a, rh * a.n + row0 + j, row0 + j, q, k);
        sQpos[j] = q;
        sKpos[j] = k;
    }
    __syncthreads();
    // Gather by position with asynchronous copies, every piece of the bucket in flight at once; a copy
    // of size 0 writes the zero padding (value rows past the bucket meet p = 0 and must be finite, query
    // rows are padded to a whole tile).  16-byte pieces where the rows allow it, else a warp per row with
    // 4-byte pieces along the row.
    if (a.vec_qk) {
        const int c4 = dq4 >> 2;
        for (int idx = tid; idx < BA_MAX_BUCKET * c4; idx += nthr) {
            const int j = idx / c4, ch = idx - j * c4;
            cp_async16(sK + j * pk + 4 * ch, kbase + (size_t)sKpos[j] * a.ldq + 4 * ch, j < bucket);
        }
        for (int idx = tid; idx < a.qrows * c4; idx += nthr) {
            const int i = idx / c4, ch = idx - i * c4;
            cp_async16(sQ + i * dq4 + 4 * ch, qbase + (size_t)sQpos[i < bucket ? i : 0] * a.ldq + 4 * ch, i < bucket);
        }
    } else {
        for (int j = warp; j < BA_MAX_BUCKET; j += nwarps) {
            const float* src = kbase + (size_t)sKpos[j] * a.ldq;
            for (int d = lane; d < dq4; d += 32)
                cp_async4(sK + j * pk + d, src + (d < a.dq ? d : 0), j < bucket && d < a.dq);
        }
        for (int i = warp; i < a.qrows; i += nwarps) {
            const float* src = qbase + (size_t)sQpos[i < bucket ? i : 0] * a.ldq;
            for (int d = lane; d < dq4; d += 32)
                cp_async4(sQ + i * dq4 + d, src + (d < a.dq ? d : 0), i < bucket && d < a.dq);
        }
    }
    if (a.vec_v) {
        const int c4 = pv >> 2, live4 = (a.dv + 3) >> 2;
        for (int idx = tid; idx < BA_MAX_BUCKET * c4; idx += nthr) {
            const int j = idx / c4, ch = idx - j * c4;
            const bool live = j < bucket && ch < live4;
            cp_async16(sV + j * pv + 4 * ch, vbase + (size_t)sKpos[j] * a.ldv + (live ? 4 * ch : 0), live);
        }
    } else {
        for (int j = warp; j < BA_MAX_BUCKET; j += nwarps) {
            const float* src = vbase + (size_t)sKpos[j] * a.ldv;
            for (int col = lane; col < pv; col += 32)
                cp_async4(sV + j * pv + col, src + (col < a.dv ? col : 0), j < bucket && col < a.dv);
        }
    }
    cp_async_wait_all();
    __syncthreads();

    float* sP = sPall + (size_t)warp * BA_QROWS * BA_MAX_BUCKET;    // [4][128]
    const int nd = a.nd, dl = lane & (nd - 1), jl = lane / nd, js = 32 / nd;
    const int jc_end = (bucket + 3) >> 2;
    // this thread's keys: lane, lane + 32, lane + 64, lane + 96 (rows pk apart, pk / 4 odd: 16-byte loads of
    // consecutive rows fall into different bank groups); -|k|^2 / 2 of each
    const float* k0 = sK + lane * pk;
    float knv[4] = {0.f, 0.f, 0.f, 0.f};
    for (int d4 = 0; d4 < dq4; d4 += 4) {
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            const float4 x = *reinterpret_cast<const float4*>(k0 + cc * 32 * pk + d4);
            knv[cc] = fmaf(x.x, x.x, knv[cc]); knv[cc] = fmaf(x.y, x.y, knv[cc]);
            knv[cc] = fmaf(x.z, x.z, knv[cc]); knv[cc] = fmaf(x.w, x.w, knv[cc]);
        }
    }
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) knv[cc] *= -0.5f;

    for (int i0 = warp * BA_QROWS; i0 < bucket; i0 += nwarps * BA_QROWS) {
        const float* q0 = sQ + (size_t)i0 * dq4;
        float qn[BA_QROWS];
#pragma unroll
        for (int r = 0; r < BA_QROWS; ++r) qn[r] = 0.f;
        for (int d = lane; d < dq4; d += 32)
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r) { const float x = q0[r * dq4 + d]; qn[r] = fmaf(x, x, qn[r]); }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r) qn[r] += __shfl_xor_sync(0xffffffffu, qn[r], o);
#pragma unroll
        for (int r = 0; r < BA_QROWS; ++r) qn[r] *= -0.5f;

        // p = exp(min(0, q.k - |q|^2/2 - |k|^2/2)) for 4 queries x 4 keys
        float acc[BA_QROWS][4];
#pragma unroll
        for (int r = 0; r < BA_QROWS; ++r) { acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f; }
        for (int d4 = 0; d4 < dq4; d4 += 4) {
            float4 q4[BA_QROWS], k4[4];
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r) q4[r] = *reinterpret_cast<const float4*>(q0 + r * dq4 + d4);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) k4[cc] = *reinterpret_cast<const float4*>(k0 + cc * 32 * pk + d4);
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    acc[r][cc] = fmaf(q4[r].x, k4[cc].x, acc[r][cc]); acc[r][cc] = fmaf(q4[r].y, k4[cc].y, acc[r][cc]);
                    acc[r][cc] = fmaf(q4[r].z, k4[cc].z, acc[r][cc]); acc[r][cc] = fmaf(q4[r].w, k4[cc].w, acc[r][cc]);
                }
        }
        float rowsum[BA_QROWS];
#pragma unroll
        for (int r = 0; r < BA_QROWS; ++r) {
            float sum = 0.f;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const float e = __expf(fminf((acc[r][cc] + qn[r]) + knv[cc], 0.f));
                const float pe = (lane + 32 * cc < bucket) ? e : 0.f;
                sP[r * BA_MAX_BUCKET + lane + 32 * cc] = pe;
                sum += pe;
            }
            rowsum[r] = sum;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r) rowsum[r] += __shfl_xor_sync(0xffffffffu, rowsum[r], o);
        __syncwarp();

        // so = p . V for 4 queries x value columns 4*dl .. 4*dl+3, keys shared out over the js lane groups
        float o[BA_QROWS][4];
#pragma unroll
        for (int r = 0; r < BA_QROWS; ++r) { o[r][0] = o[r][1] = o[r][2] = o[r][3] = 0.f; }
        for (int jc = jl; jc < jc_end; jc += js) {
            float4 p4[BA_QROWS];
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r) p4[r] = *reinterpret_cast<const float4*>(sP + r * BA_MAX_BUCKET + 4 * jc);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const float4 v4 = *reinterpret_cast<const float4*>(sV + (size_t)(4 * jc + jj) * pv + 4 * dl);
#pragma unroll
                for (int r = 0; r < BA_QROWS; ++r) {
                    const float pj = jj == 0 ? p4[r].x : jj == 1 ? p4[r].y : jj == 2 ? p4[r].z : p4[r].w;
                    o[r][0] = fmaf(pj, v4.x, o[r][0]); o[r][1] = fmaf(pj, v4.y, o[r][1]);
                    o[r][2] = fmaf(pj, v4.z, o[r][2]); o[r][3] = fmaf(pj, v4.w, o[r][3]);
                }
            }
        }
        for (int off = nd; off < 32; off <<= 1)
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) o[r][cc] += __shfl_xor_sync(0xffffffffu, o[r][cc], off);
        if (jl == 0) {
#pragma unroll
            for (int r = 0; r < BA_QROWS; ++r) {
                const int i = i0 + r;
                if (i >= bucket) continue;
                const int64_t dst = a.scatter ? sQpos[i] : row0 + i;
                float* orow = a.so + ((size_t)rh * a.n + dst) * a.dv + 4 * dl;
                if (a.vec_store) {
                    if (4 * dl < a.dv) *reinterpret_cast<float4*>(orow) = make_float4(o[r][0], o[r][1], o[r][2], o[r][3]);
                } else {
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc)
                        if (4 * dl + cc < a.dv) orow[cc] = o[r][cc];
                }
                if (lane == 0) a.denom[(size_t)rh * a.n + dst] = rowsum[r] + 1e-20f;
            }
        }
        __syncwarp();
    }
}

// -------------------------------------------------------------------------------------------------
// Rows of at most 32 features: the same bucket on the tensor cores, at fp32 accuracy.  A float is
// carried exactly by three bf16 pieces (hi + mid + lo, 8 significant bits each); of the nine products of
// two such sums the six larger ones are issued (hi.hi, hi.mid, mid.hi, mid.mid, hi.lo, lo.hi, smallest
// first), the other three are below 2^-24 of the result, and accumulation is fp32.  The FMA kernel above
// is bound by instruction issue (64 k warp instructions per bucket, 71 % of the issue slots); this one
// spends 2 k tensor-core instructions and 10 k others.
// Warp = 16 query rows x all keys.  Keys and values are gathered, split once and kept as bf16 tiles in
// shared memory; queries go from global memory straight into operand fragments, and the weights p from
// their accumulators into the operand fragments of p V (the two layouts coincide), so that neither
// touches shared memory.  60 000 hits, 3 rounds x 8 heads, buckets of 100, 30 + 24 features: 0.97 ms -> 0.47 ms.  Buckets of
// at most 32 hits stay with the FMA kernel (two warps' worth of 16-row tiles), and so do wider rows: their fragments in
// three pieces do not fit the registers and the kernel is slower than FMA there.
// -------------------------------------------------------------------------------------------------
// c[i] += a b_i for operands in three pieces and NT column tiles (two per fragment), one piece of b in registers at a time
// (low first); `load` fetches the fragments of a piece.  Consecutive instructions go to different accumulators.
template <int NT, class Load>
__device__ __forceinline__ void mma6(float (*c)[4], const uint32_t (&ah)[4], const uint32_t (&am)[4], const uint32_t (&al)[4], Load load) {
    uint32_t b[(NT + 1) / 2][4];
    auto times = [&](const uint32_t (&x)[4]) {
#pragma unroll
        for (int i = 0; i < NT; ++i) mma16816(c[i], x, b[i / 2][2 * (i & 1)], b[i / 2][2 * (i & 1) + 1]);
    };
    load(2, b);
    times(ah);
    load(1, b);
    times(am);
    times(ah);
    load(0, b);
    times(al);
    times(am);
    times(ah);
}
__host__ __device__ inline int bam_keys(int bucket) { return (bucket + 15) & ~15; }
template <int KQ, int NV>
__host__ __device__ constexpr int bam_smem(int keys) { return 4 * 128 * 8 + keys * 3 * ((16 * KQ + 8) + (8 * ((NV + 1) & ~1) + 8)) * 2; }

template <int KQ, int NV>      // 16-wide feature steps of q / k, 8-wide value column tiles
__global__ void __launch_bounds__(256, 3) bucket_attn_mma_kernel(BucketAttnArgs a) {
    if (chain_wait()) return;
    constexpr int KP = 16 * KQ + 8, VP = 8 * ((NV + 1) & ~1) + 8;         // bf16 pitches: consecutive rows fall into different bank groups
    extern __shared__ __align__(16) float ba_smem[];
    const int bucket = a.bucket, keys = bam_keys(bucket), nthr = blockDim.x;     // nthr = 2 * keys
    int64_t* sQpos = reinterpret_cast<int64_t*>(ba_smem);
    int64_t* sKpos = sQpos + 128;
    float* sKn = reinterpret_cast<float*>(sKpos + 128);      // -|k|^2 / 2
    __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<char*>(ba_smem) + 4 * 128 * 8);   // [3][keys][KP]
    __nv_bfloat16* sV = sK + 3 * keys * KP;                  // [3][keys][VP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;

    const int64_t nb = a.n / bucket;
    const int64_t b = blockIdx.x % nb, hc = blockIdx.x / nb;
    const int h = (int)(hc / a.rounds), c = (int)(hc % a.rounds);
    const int64_t rh = (int64_t)c * a.heads + h;             // row of the positions and outputs
    const int64_t row0 = b * bucket;
    const float* qbase = a.q + c * a.in_round_stride_q + (size_t)h * a.n * a.ldq;
    const float* kbase = a.k + c * a.in_round_stride_q + (size_t)h * a.n * a.ldq;
    const float* vbase = a.v + c * a.in_round_stride_v + (size_t)h * a.n * a.ldv;

    for (int j = tid; j < bucket; j += nthr) {
        int64_t q, k;
        ba_positions(a, rh * a.n + row0 + j, row0 + j, q, k);
        sQpos[j] = q;
        sKpos[j] = k;
    }
    __syncthreads();
    // ---- keys and values: eight lanes per row, four rows per lane group, all of their loads in flight at once ----
    const int l8 = tid & 7, rstep = nthr >> 3;
    {
        float ss[4] = {0.f, 0.f, 0.f, 0.f};
        float4 x[4], y[4];
        auto fetch = [&](const float* base, int ld, int width, bool vec, int pc, float4 (&r)[4]) {
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int j = (tid >> 3) + it * rstep;
                r[it] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < bucket && 4 * pc < width) {
                    const float* src = base + (size_t)sKpos[j] * ld + 4 * pc;
                    if (vec) r[it] = __ldg(reinterpret_cast<const float4*>(src));
                    else {
                        r[it].x = __ldg(src);
                        if (4 * pc + 1 < width) r[it].y = __ldg(src + 1);
                        if (4 * pc + 2 < width) r[it].z = __ldg(src + 2);
                        if (4 * pc + 3 < width) r[it].w = __ldg(src + 3);
                    }
                }
            }
        };
        auto put = [&](__nv_bfloat16* base, int pitch, int pc, const float4 (&r)[4]) {
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int j = (tid >> 3) + it * rstep;
                const Split3 p = split3(r[it].x, r[it].y), q = split3(r[it].z, r[it].w);
                uint2* d = reinterpret_cast<uint2*>(base + j * pitch + 4 * pc);
                d[0] = make_uint2(p.h, q.h);
                d = reinterpret_cast<uint2*>(base + (keys + j) * pitch + 4 * pc);
                d[0] = make_uint2(p.m, q.m);
                d = reinterpret_cast<uint2*>(base + (2 * keys + j) * pitch + 4 * pc);
                d[0] = make_uint2(p.l, q.l);
            }
        };
        constexpr int NP = ((4 * KQ > 2 * NV ? 4 * KQ : 2 * NV) + 7) / 8;
#pragma unroll
        for (int pi = 0; pi < NP; ++pi) {
            const int pc = l8 + 8 * pi;
            if (8 * pi < 4 * KQ) fetch(kbase, a.ldq, a.dq, a.vec_qk, pc, x);
            if (8 * pi < 2 * NV) fetch(vbase, a.ldv, a.dv, a.vec_v, pc, y);
            if (8 * pi < 4 * KQ) {
                put(sK, KP, pc, x);
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    ss[it] = fmaf(x[it].x, x[it].x, ss[it]); ss[it] = fmaf(x[it].y, x[it].y, ss[it]);
                    ss[it] = fmaf(x[it].z, x[it].z, ss[it]); ss[it] = fmaf(x[it].w, x[it].w, ss[it]);
                }
            }
            if (8 * pi < 2 * NV) put(sV, VP, pc, y);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int it = 0; it < 4; ++it) ss[it] += __shfl_xor_sync(0xffffffffu, ss[it], o);
        if (l8 == 0)
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int j = (tid >> 3) + it * rstep;
                sKn[j] = j < bucket ? -0.5f * ss[it] : -INFINITY;
            }
    }
    // ---- queries: this warp's 16 rows as operand fragments ----
    const int m0 = 16 * warp;
    uint32_t qh[KQ][4], qm[KQ][4], ql[KQ][4];
    float qn[2] = {0.f, 0.f};
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int i = m0 + g + 8 * hh;
        const float* src = qbase + (size_t)(i < bucket ? sQpos[i] : 0) * a.ldq;
        float2 v[KQ][2];
#pragma unroll
        for (int kk = 0; kk < KQ; ++kk)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = 16 * kk + 8 * e + 2 * t;
                v[kk][e] = make_float2(0.f, 0.f);
                if (i < bucket && col < a.dq) {
                    if (a.vec_qk) v[kk][e] = __ldg(reinterpret_cast<const float2*>(src + col));
                    else { v[kk][e].x = __ldg(src + col); if (col + 1 < a.dq) v[kk][e].y = __ldg(src + col + 1); }
                }
            }
#pragma unroll
        for (int kk = 0; kk < KQ; ++kk)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                qn[hh] = fmaf(v[kk][e].x, v[kk][e].x, qn[hh]);
                qn[hh] = fmaf(v[kk][e].y, v[kk][e].y, qn[hh]);
                const Split3 s = split3(v[kk][e].x, v[kk][e].y);
                qh[kk][hh + 2 * e] = s.h; qm[kk][hh + 2 * e] = s.m; ql[kk][hh + 2 * e] = s.l;
            }
        qn[hh] += __shfl_xor_sync(0xffffffffu, qn[hh], 1);
        qn[hh] += __shfl_xor_sync(0xffffffffu, qn[hh], 2);
        qn[hh] *= -0.5f;
    }
    __syncthreads();

    const int mi = lane >> 3, r8 = lane & 7;
    float o[NV][4], rowsum[2] = {0.f, 0.f};
#pragma unroll
    for (int nv = 0; nv < NV; ++nv) { o[nv][0] = o[nv][1] = o[nv][2] = o[nv][3] = 0.f; }
    for (int n0 = 0; n0 < keys; n0 += 32) {                  // 32 keys: four column tiles
        float acc[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) { acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f; }
        const bool two = n0 + 16 < keys;                     // warp-uniform: the last step may hold 16 keys
#pragma unroll
        for (int kk = 0; kk < KQ; ++kk) {
            const uint32_t at = smem_u32(sK + (n0 + r8 + (mi >> 1) * 8) * KP + 16 * kk + (mi & 1) * 8);
            auto load1 = [&](int p, uint32_t (&b)[1][4]) { ldsm_x4(b[0], at + p * keys * KP * 2); };
            auto load2 = [&](int p, uint32_t (&b)[2][4]) { ldsm_x4(b[0], at + p * keys * KP * 2); ldsm_x4(b[1], at + (p * keys + 16) * KP * 2); };
            if (two) mma6<4>(acc, qh[kk], qm[kk], ql[kk], load2);
            else mma6<2>(acc, qh[kk], qm[kk], ql[kk], load1);
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
            if (ks == 0 || two) {
                uint32_t ph[4], pm[4], pl[4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = n0 + 16 * ks + 8 * e + 2 * t;
                    const float2 kn = *reinterpret_cast<const float2*>(sKn + col);      // -inf past the bucket: weight 0
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const float p0 = __expf(fminf((acc[2 * ks + e][2 * hh] + qn[hh]) + kn.x, 0.f));
                        const float p1 = __expf(fminf((acc[2 * ks + e][2 * hh + 1] + qn[hh]) + kn.y, 0.f));
                        rowsum[hh] += p0 + p1;
                        const Split3 s = split3(p0, p1);
                        ph[2 * e + hh] = s.h; pm[2 * e + hh] = s.m; pl[2 * e + hh] = s.l;
                    }
                }
                const uint32_t at = smem_u32(sV + (n0 + 16 * ks + r8 + (mi & 1) * 8) * VP + (mi >> 1) * 8);
                mma6<NV>(o, ph, pm, pl, [&](int p, uint32_t (&b)[(NV + 1) / 2][4]) {
#pragma unroll
                    for (int x = 0; x < (NV + 1) / 2; ++x) ldsm_x4_t(b[x], at + (p * keys * VP + 16 * x) * 2);
                });
            }
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        rowsum[hh] += __shfl_xor_sync(0xffffffffu, rowsum[hh], 1);
        rowsum[hh] += __shfl_xor_sync(0xffffffffu, rowsum[hh], 2);
        const int i = m0 + g + 8 * hh;
        if (i >= bucket) continue;
        const int64_t dst = a.scatter ? sQpos[i] : row0 + i;
        float* orow = a.so + ((size_t)rh * a.n + dst) * a.dv;
#pragma unroll
        for (int nv = 0; nv < NV; ++nv) {
            const int col = 8 * nv + 2 * t;
            if (a.vec_store) {                               // dv % 4 == 0: the pair is inside and 8-byte aligned
                if (col < a.dv) *reinterpret_cast<float2*>(orow + col) = make_float2(o[nv][2 * hh], o[nv][2 * hh + 1]);
            } else {
                if (col < a.dv) orow[col] = o[nv][2 * hh];
                if (col + 1 < a.dv) orow[col + 1] = o[nv][2 * hh + 1];
            }
        }
        if (t == 0) a.denom[(size_t)rh * a.n + dst] = rowsum[hh] + 1e-20f;
    }
}

// out[row][col] = (sum over rounds of so) / (sum over rounds of denom), rounds added in order; V consecutive columns per thread
template <int V>
__global__ void __launch_bounds__(256)
bucket_attn_combine_kernel(const float* __restrict__ so, const float* __restrict__ denom, int rounds,
                           int64_t rows, int dv, float* __restrict__ out) {
    if (chain_wait()) return;
    const int64_t total = rows * dv;
    for (int64_t e = ((int64_t)blockIdx.x * 256 + threadIdx.x) * V; e < total; e += (int64_t)gridDim.x * 256 * V) {
        const int64_t row = e / dv;
        float s[V], d = denom[row];
        if (V == 4) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(so + e));
            s[0] = x.x; s[1 % V] = x.y; s[2 % V] = x.z; s[3 % V] = x.w;
        } else s[0] = so[e];
        for (int c = 1; c < rounds; ++c) {
            if (V == 4) {
                const float4 x = __ldg(reinterpret_cast<const float4*>(so + (size_t)c * total + e));
                s[0] += x.x; s[1 % V] += x.y; s[2 % V] += x.z; s[3 % V] += x.w;
            } else s[0] += so[(size_t)c * total + e];
            d += denom[(size_t)c * rows + row];
        }
        if (V == 4)
            *reinterpret_cast<float4*>(out + e) = make_float4(__fdiv_rn(s[0], d), __fdiv_rn(s[1 % V], d), __fdiv_rn(s[2 % V], d), __fdiv_rn(s[3 % V], d));
        else out[e] = __fdiv_rn(s[0], d);
    }
}

// q_hat[h][i] = [query[i][h][:], scale[h][:] * coords[i][:]] (k_hat likewise), v_out[h][i] =
// value[i][h][:]; rows i >= raw_size are zero.  Token-major inputs, head-major outputs.
__global__ void __launch_bounds__(256)
hept_prep_qk_kernel(const float* __restrict__ query, const float* __restrict__ key, const float* __restrict__ value,
                    const float* __restrict__ scale, const float* __restrict__ coords, int64_t n, int heads,
                    int d, int cd, int ldq, int64_t raw_size, float* __restrict__ q_hat, float* __restrict__ k_hat,
                    float* __restrict__ v_out) {
    if (chain_wait()) return;
    const int dq = ldq;                       // columns d + cd .. ldq - 1 are zero padding
    const int64_t total = (int64_t)heads * n * dq;
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
        const int col = (int)(e % dq);
        const int64_t hi = e / dq, i = hi % n;
        const int h = (int)(hi / n);
        const bool live = i < raw_size;
        const size_t src = ((size_t)i * heads + h) * d + col;
        if (col < d) {
            q_hat[e] = live ? query[src] : 0.f;
            k_hat[e] = live ? key[src] : 0.f;
            if (v_out) v_out[(size_t)hi * d + col] = live ? value[src] : 0.f;
        } else {
            const float r = (live && col < d + cd) ? __fmul_rn(scale[h * cd + col - d], coords[(size_t)i * cd + col - d]) : 0.f;
            q_hat[e] = r;
            k_hat[e] = r;
        }
    }
}

// -------------------------------------------------------------------------------------------------
// Front of the attention layer in one pass over the tokens: prep_qk's head-major rows (as above), the
// E2LSH projections of both (operation order of lsh_hash_kernel), and per block of hits the smallest and
// largest projection of every (round, head) row.  One after the other these passes read and wrote the
// rows three times, and the generic hash walked a 128-byte row per lane (210 us for 480 000 rows); here a
// CTA stages 32 tokens with all heads in shared memory, writes whole 4 KB runs per head, and a warp hashes
// one head of its 32 hits.
// -------------------------------------------------------------------------------------------------
constexpr int HF_HITS = 32, HF_MAX_ROUNDS = 8;
__host__ __device__ inline int hf_pitch(int heads, int d) { return heads * d | 1; }      // odd: a column of hits is conflict-free
inline size_t hf_smem(int heads, int d, int cd, int rounds) {
    return ((size_t)2 * HF_HITS * hf_pitch(heads, d) + HF_HITS * cd + (size_t)heads * cd + (size_t)heads * (d + cd) * rounds) * 4;
}

template <int R, bool VEC>      // VEC: d and ldq are multiples of 4, everything 16-byte aligned
__global__ void __launch_bounds__(256)
hept_front_kernel(const float* __restrict__ query, const float* __restrict__ key, const float* __restrict__ value,
                  const float* __restrict__ scale, const float* __restrict__ coords, const float* __restrict__ alpha,
                  int64_t n, int heads, int d, int cd, int ldq, int64_t raw_size, float* __restrict__ q_hat,
                  float* __restrict__ k_hat, float* __restrict__ v_out, float* __restrict__ proj, float2* __restrict__ part) {
    if (chain_wait()) return;
    extern __shared__ __align__(16) float hf[];
    const int hd = heads * d, P = hf_pitch(heads, d), D = d + cd;
    float* sq = hf;                             // [32][P] query rows, then key rows behind them
    float* sk = sq + HF_HITS * P;
    float* sc = sk + HF_HITS * P;               // [32][cd]
    float* ss = sc + HF_HITS * cd;              // [heads][cd]
    float* sa = ss + heads * cd;                // [heads][D][R]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * HF_HITS;
    const int m = (int)max((int64_t)0, min((int64_t)HF_HITS, raw_size - i0));     // rows that hold a hit
    const int rows = (int)min((int64_t)HF_HITS, n - i0);
    if (VEC) {                                  // six 16-byte pieces of each input in flight per thread
        const int hd4 = hd >> 2, d4 = d >> 2, total = HF_HITS * hd4, dr = 256 / hd4, dc = 256 - dr * hd4;
        int r = tid / hd4, c = tid - r * hd4;
        for (int e0 = tid; e0 < total; e0 += 6 * 256) {
            float4 xq[6], xk[6], xv[6];
            int rr[6], cc[6];
#pragma unroll
            for (int x = 0; x < 6; ++x) {
                rr[x] = r; cc[x] = c;
                const bool in = e0 + 256 * x < total && r < m;
                const size_t at = (size_t)(i0 + r) * hd + 4 * c;
                xq[x] = in ? __ldg(reinterpret_cast<const float4*>(query + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
                xk[x] = in ? __ldg(reinterpret_cast<const float4*>(key + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
                xv[x] = in ? __ldg(reinterpret_cast<const float4*>(value + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
                r += dr; c += dc;
                if (c >= hd4) { c -= hd4; ++r; }
            }
#pragma unroll
            for (int x = 0; x < 6; ++x) {
                if (e0 + 256 * x >= total) break;
                float* p = sq + rr[x] * P + 4 * cc[x];
                p[0] = xq[x].x; p[1] = xq[x].y; p[2] = xq[x].z; p[3] = xq[x].w;
                p = sk + rr[x] * P + 4 * cc[x];
                p[0] = xk[x].x; p[1] = xk[x].y; p[2] = xk[x].z; p[3] = xk[x].w;
                const int h = cc[x] / d4;       // values only change their layout
                if (rr[x] < rows) *reinterpret_cast<float4*>(v_out + ((size_t)h * n + i0 + rr[x]) * d + 4 * (cc[x] - h * d4)) = xv[x];
            }
        }
    } else
        for (int r = warp; r < HF_HITS; r += 8)
            for (int c = lane; c < hd; c += 32) {
                sq[r * P + c] = r < m ? __ldg(query + (i0 + r) * hd + c) : 0.f;
                sk[r * P + c] = r < m ? __ldg(key + (i0 + r) * hd + c) : 0.f;
                if (r < rows) {
                    const int h = c / d;
                    v_out[((size_t)h * n + i0 + r) * d + c - h * d] = r < m ? __ldg(value + (i0 + r) * hd + c) : 0.f;
                }
            }
    for (int e = tid; e < HF_HITS * cd; e += 256) sc[e] = e / cd < m ? __ldg(coords + i0 * cd + e) : 0.f;
    for (int e = tid; e < heads * cd; e += 256) ss[e] = __ldg(scale + e);
    for (int e = tid; e < heads * D * R; e += 256) sa[e] = __ldg(alpha + e);
    __syncthreads();
    for (int h = warp; h < heads; h += 8) {
        if (VEC) {
            const int w4 = ldq >> 2, dr = 32 / w4, dc = 32 - dr * w4;
            int r = lane / w4, c = lane - r * w4;
            while (r < rows) {
                float x[4], y[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int col = 4 * c + e;
                    if (col < d) { x[e] = sq[r * P + h * d + col]; y[e] = sk[r * P + h * d + col]; }
                    else x[e] = y[e] = col < D && r < m ? __fmul_rn(ss[h * cd + col - d], sc[r * cd + col - d]) : 0.f;
                }
                const size_t at = ((size_t)h * n + i0 + r) * ldq + 4 * c;
                *reinterpret_cast<float4*>(q_hat + at) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(k_hat + at) = make_float4(y[0], y[1], y[2], y[3]);
                r += dr; c += dc;
                if (c >= w4) { c -= w4; ++r; }
            }
        } else
            for (int r = 0; r < rows; ++r)
                for (int c = lane; c < ldq; c += 32) {
                    float x = 0.f, y = 0.f;
                    if (c < d) { x = sq[r * P + h * d + c]; y = sk[r * P + h * d + c]; }
                    else if (c < D && r < m) x = y = __fmul_rn(ss[h * cd + c - d], sc[r * cd + c - d]);
                    q_hat[((size_t)h * n + i0 + r) * ldq + c] = x;
                    k_hat[((size_t)h * n + i0 + r) * ldq + c] = y;
                }
        float aq[R], ak[R];
        const float* al = sa + h * D * R;
        for (int c = 0; c < D; ++c) {
            float x, y;
            if (c < d) { x = sq[lane * P + h * d + c]; y = sk[lane * P + h * d + c]; }
            else x = y = lane < m ? __fmul_rn(ss[h * cd + c - d], sc[lane * cd + c - d]) : 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float w = al[c * R + r];
                aq[r] = c == 0 ? __fmul_rn(x, w) : __fadd_rn(aq[r], __fmul_rn(x, w));
                ak[r] = c == 0 ? __fmul_rn(y, w) : __fadd_rn(ak[r], __fmul_rn(y, w));
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const size_t row = (size_t)r * heads + h;
            float mn = INFINITY, mx = -INFINITY;
            if (lane < rows) {
                proj[row * n + i0 + lane] = aq[r];
                proj[((size_t)R * heads + row) * n + i0 + lane] = ak[r];
                mn = fminf(aq[r], ak[r]); mx = fmaxf(aq[r], ak[r]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if (lane == 0) part[row * gridDim.x + blockIdx.x] = make_float2(mn, mx);
        }
    }
}

}  // namespace lampa

using namespace lampa;

extern "C" int lampa_bucket_rbf_attn(const float* q, const float* k, const float* v, const int64_t* q_pos,
                                     const int64_t* k_pos, int32_t rounds, int32_t heads, int64_t n,
                                     int32_t bucket, int32_t dq, int32_t dv, int32_t ldq, int32_t ldv,
                                     int32_t inputs_per_round, int32_t scatter, float* so, float* denom,
                                     void* stream) {
    return lampa_bucket_rbf_attn_checked(q, k, v, q_pos, k_pos, rounds, heads, n, bucket, dq, dv, ldq, ldv, inputs_per_round, scatter,
                                         so, denom, nullptr, stream);
}

extern "C" int lampa_bucket_rbf_attn_checked(const float* q, const float* k, const float* v, const int64_t* q_pos,
                                             const int64_t* k_pos, int32_t rounds, int32_t heads, int64_t n,
                                             int32_t bucket, int32_t dq, int32_t dv, int32_t ldq, int32_t ldv,
                                             int32_t inputs_per_round, int32_t scatter, float* so, float* denom,
                                             int32_t* status, void* stream) {
    if (rounds <= 0 || heads <= 0 || n < 0 || bucket <= 0 || dq <= 0 || dv <= 0) return LAMPA_ERR_ARG;
    if (n % bucket != 0 || ldq < dq || ldv < dv) return LAMPA_ERR_ARG;
    if ((q_pos == nullptr) != (k_pos == nullptr)) return LAMPA_ERR_ARG;
    if (!q_pos && !inputs_per_round && rounds > 1) return LAMPA_ERR_ARG;   // nothing would tell the rounds apart
    if (n == 0) return LAMPA_OK;
    if (!q || !k || !v || !so || !denom) return LAMPA_ERR_ARG;
    if (bucket > BA_MAX_BUCKET || dv > 128 || dq > 1024) return LAMPA_ERR_UNSUPPORTED;
    BucketAttnArgs a;
    a.q = q; a.k = k; a.v = v; a.q_pos = q_pos; a.k_pos = k_pos; a.so = so; a.denom = denom; a.status = status;
    a.n = n; a.rounds = rounds; a.heads = heads; a.bucket = bucket; a.dq = dq; a.dv = dv;
    a.ldq = ldq; a.ldv = ldv;
    a.in_round_stride_q = inputs_per_round ? (int64_t)heads * n * ldq : 0;
    a.in_round_stride_v = inputs_per_round ? (int64_t)heads * n * ldv : 0;
    a.dq4 = (dq + 3) & ~3;
    a.pk = ((a.dq4 >> 2) & 1) ? a.dq4 : a.dq4 + 4;
    a.nd = ba_pow2_at_least((dv + 3) >> 2);
    a.pv = a.nd >= 8 ? 4 * a.nd : 4 * a.nd + 4;
    a.scatter = scatter ? 1 : 0;
    auto al16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    a.vec_qk = ldq % 4 == 0 && ldq >= a.dq4 && al16(q) && al16(k);
    a.vec_v = ldv % 4 == 0 && ldv >= ((dv + 3) & ~3) && al16(v);
    a.vec_store = (dv % 4 == 0) && (reinterpret_cast<uintptr_t>(so) % 16 == 0);
    // whole tiles of query rows, spread over as few warps as finish in the same number of rounds
    auto plan = [&](int qr, int& warps, size_t& smem) {
        const int tiles = (bucket + qr - 1) / qr;
        const int tile_rounds = (tiles + BA_MAX_WARPS - 1) / BA_MAX_WARPS;
        warps = (tiles + tile_rounds - 1) / tile_rounds;
        a.qrows = tiles * qr;
        smem = ba_smem_floats(a.dq4, a.pk, a.pv, a.qrows, warps, qr) * sizeof(float);
    };
    int warps; size_t smem;
    plan(4, warps, smem);
    const bool wide = smem > 113 * 1024;                   // not even two CTAs of 4-row tiles fit an SM
    if (wide) plan(8, warps, smem);
    if (smem > MAX_SMEM) return LAMPA_ERR_UNSUPPORTED;
    const int64_t units = (int64_t)rounds * heads * (n / bucket);
    if (units > 0x7fffffffLL) return LAMPA_ERR_UNSUPPORTED;
    // Rows of up to 32 features are what a warp's tile holds in registers at three CTAs per SM; with wider ones this kernel
    // measured slower than FMA (dq 54 / dv 48: 1.78 against 1.65 ms), and a bucket of fewer than 33 hits leaves it two warps.
    if (dq <= 32 && dv <= 32 && bucket > 32) {
        const int keys = bam_keys(bucket);
        auto mma = dv <= 24 ? bucket_attn_mma_kernel<2, 3> : bucket_attn_mma_kernel<2, 4>;
        const int msmem = bam_smem<2, 4>(keys);
        if (cudaFuncSetAttribute(mma, cudaFuncAttributeMaxDynamicSharedMemorySize, bam_smem<2, 4>(BA_MAX_BUCKET)) != cudaSuccess) return LAMPA_ERR_CUDA;
        ProfScope prof("bucket_rbf_attn", (cudaStream_t)stream);
        launch_chained(mma, (unsigned)units, 2 * keys, msmem, (cudaStream_t)stream, a);
        return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
    }
    auto kernel = wide ? bucket_rbf_attn_kernel<8> : bucket_rbf_attn_kernel<4>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM) != cudaSuccess) return LAMPA_ERR_CUDA;
    ProfScope prof("bucket_rbf_attn", (cudaStream_t)stream);
    launch_chained(kernel, (unsigned)units, warps * 32, smem, (cudaStream_t)stream, a);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_bucket_attn_combine(const float* so, const float* denom, int32_t rounds, int64_t rows,
                                         int32_t dv, float* out, void* stream) {
    if (rounds <= 0 || rows < 0 || dv <= 0) return LAMPA_ERR_ARG;
    if (rows == 0) return LAMPA_OK;
    if (!so || !denom || !out) return LAMPA_ERR_ARG;
    ProfScope prof("bucket_attn_combine", (cudaStream_t)stream);
    const int64_t total = rows * dv;
    const bool v4 = dv % 4 == 0 && (((uintptr_t)so | (uintptr_t)out) & 15) == 0;
    const unsigned grid = (unsigned)std::min<int64_t>((total / (v4 ? 4 : 1) + 255) / 256, 148 * 32);
    if (v4) launch_chained(bucket_attn_combine_kernel<4>, grid, 256, 0, (cudaStream_t)stream, so, denom, rounds, rows, dv, out);
    else launch_chained(bucket_attn_combine_kernel<1>, grid, 256, 0, (cudaStream_t)stream, so, denom, rounds, rows, dv, out);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_hept_prep_qk(const float* query, const float* key, const float* value, const float* scale,
                                  const float* coords, int64_t n, int32_t heads, int32_t d, int32_t cd,
                                  int32_t ldq, int64_t raw_size, float* q_hat, float* k_hat, float* v_out,
                                  void* stream) {
    if (n < 0 || heads <= 0 || d <= 0 || cd < 0 || raw_size < 0 || ldq < d + cd) return LAMPA_ERR_ARG;
    if (n == 0) return LAMPA_OK;
    if (!query || !key || !q_hat || !k_hat || (cd > 0 && (!scale || !coords)) || (v_out && !value)) return LAMPA_ERR_ARG;
    ProfScope prof("hept_prep_qk", (cudaStream_t)stream);
    const int64_t total = (int64_t)heads * n * ldq;
    const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 16);
    launch_chained(hept_prep_qk_kernel, grid, 256, 0, (cudaStream_t)stream, query, key, value, scale, coords, n, heads, d, cd,
                                                                 ldq, raw_size, q_hat, k_hat, v_out);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_hept_front_blocks(int64_t n, int64_t* blocks) {
    if (n < 0 || !blocks) return LAMPA_ERR_ARG;
    *blocks = (n + HF_HITS - 1) / HF_HITS;
    return LAMPA_OK;
}

extern "C" int lampa_hept_front(const float* query, const float* key, const float* value, const float* scale, const float* coords,
                                const float* alpha, int64_t n, int32_t heads, int32_t d, int32_t cd, int32_t rounds, int32_t ldq,
                                int64_t raw_size, float* q_hat, float* k_hat, float* v_out, float* proj, float* part, void* stream) {
    if (n < 0 || heads <= 0 || d <= 0 || cd <= 0 || rounds <= 0 || raw_size < 0 || ldq < d + cd) return LAMPA_ERR_ARG;
    if (n == 0) return LAMPA_OK;
    if (!query || !key || !value || !scale || !coords || !alpha || !q_hat || !k_hat || !v_out || !proj || !part) return LAMPA_ERR_ARG;
    const size_t smem = hf_smem(heads, d, cd, rounds);
    constexpr int most = 200 * 1024;
    if (rounds > HF_MAX_ROUNDS || smem > most) return LAMPA_ERR_UNSUPPORTED;
    using K = void (*)(const float*, const float*, const float*, const float*, const float*, const float*, int64_t, int, int, int, int, int64_t,
                       float*, float*, float*, float*, float2*);
    static const K kernels[2][HF_MAX_ROUNDS] = {
        {hept_front_kernel<1, false>, hept_front_kernel<2, false>, hept_front_kernel<3, false>, hept_front_kernel<4, false>,
         hept_front_kernel<5, false>, hept_front_kernel<6, false>, hept_front_kernel<7, false>, hept_front_kernel<8, false>},
        {hept_front_kernel<1, true>, hept_front_kernel<2, true>, hept_front_kernel<3, true>, hept_front_kernel<4, true>,
         hept_front_kernel<5, true>, hept_front_kernel<6, true>, hept_front_kernel<7, true>, hept_front_kernel<8, true>}};
    const bool vec = d % 4 == 0 && ldq % 4 == 0 && heads * d <= 1024 &&
                     (((uintptr_t)query | (uintptr_t)key | (uintptr_t)value | (uintptr_t)q_hat | (uintptr_t)k_hat | (uintptr_t)v_out) & 15) == 0;
    const K kernel = kernels[vec][rounds - 1];
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return LAMPA_ERR_CUDA;
    ProfScope prof("hept_front", (cudaStream_t)stream);
    launch_chained(kernel, (unsigned)((n + HF_HITS - 1) / HF_HITS), 256, smem, (cudaStream_t)stream, query, key, value, scale, coords, alpha, n, heads, d, cd, ldq,
                                                                                        raw_size, q_hat, k_hat, v_out, proj, (float2*)part);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}
