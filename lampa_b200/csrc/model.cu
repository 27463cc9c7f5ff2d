// The dense half of one model block around the hierarchical mixer, for d_model = 128 and bf16 layers: everything a block
// does per row besides the mixer itself, in two kernels, so that no projection, hidden layer or norm makes a round trip
// through HBM of its own.
//
//   project   gather the normed rows into the block's LSH order -> q, k, v, gate, a, b, l projections -> short causal
//             convolutions + SiLU on q, k, v; g, beta, lambda from a, b, l     (modeling_h_gated_deltanet.py:395-450)
//   update    gated norm of the mixer output -> o_proj -> residual add at the hit's row -> RMS norm -> MLP (up, GELU,
//             down) -> residual add -> the next block's RMS norm               (481-487; modeling_gated_deltaproduct.py:
//             1169-1199; the ordering around it: models/baselines/hmamba.py:428-455)
//   encode    input scaling, first Linear and the first block's norm;  head: last Linear (both fp32, on CUDA cores)
//
// As separate library calls a block moved each row about 14 KB through HBM (projections, convolutions, gates, norms,
// hidden layer, GELU, three residual passes): 5.3 ms per block for 2.05 M rows.  Here a row costs 1.4 KB in `project`
// and 1.8 KB in `update`: 1.63 + 2.0 ms.  Both run two CTAs per SM: a CTA alternates between tensor-core products and epilogues that
// cannot overlap inside one tile, and the other CTA fills the gaps.  Weights stream from L2 through a ring of 16 KB
// stages (they do not fit beside the tiles at two CTAs per SM).
#include "act.cuh"
#include "common.cuh"
#include "profile.cuh"
#include "tmap.cuh"
#include "umma.cuh"

namespace lampa {

namespace {

constexpr int MD = 128;                      // model width
constexpr int MST = 16384;                   // one weight stage: [128][64] or two [64][64] bf16 tiles, 128-byte swizzle
constexpr int MNST = 3;
constexpr int MWARPS = 16;                   // epilogue warps: the epilogues are chains of latencies, 8 warps of twice the columns took 1.5 x as long
constexpr int METHR = MWARPS * 32;

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;\n" :: "n"(METHR) : "memory"); }

// Wait of the epilogue warps: one warp polls, the others join a hardware barrier (sixteen polling warps took a third of
// the kernel's issue slots).  `also` runs in the polling warp before the barrier.
template <class F>
__device__ __forceinline__ void epi_wait(uint64_t* bar, uint32_t parity, bool& dead, int32_t* status, int where, int budget, F also) {
    if (threadIdx.x < 32) {
        mbar_wait(bar, parity, dead, status, where, budget);
        also();
    }
    epi_sync();
}

// Row r of the residual stream of n rows that position j of an ordered batch stands for (perm is local to j's event); -1 when
// the permutation leaves the event or the event's offsets, which nobody has checked before, leave the rows.
__device__ __forceinline__ int64_t ordered_row(const int64_t* __restrict__ cu, int nseq, const int64_t* __restrict__ perm,
                                               int64_t j, int64_t n, int32_t* status, bool* first = nullptr) {
    int lo = 0, hi = nseq;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(cu + mid) <= j) lo = mid; else hi = mid;
    }
    const int64_t s0 = __ldg(cu + lo), s1 = __ldg(cu + lo + 1), p = __ldg(perm + j);
    if (first) *first = j == s0;
    if (p < 0 || p >= s1 - s0 || s0 < 0 || s1 > n) {
        set_status(status, LAMPA_ERR_BOUNDS, 40, (int)j);
        return -1;
    }
    return s0 + p;
}

// bf16 element address inside a [rows][128] operand held as two swizzled [rows][64] halves of `half_bytes`
__device__ __forceinline__ uint32_t op_off(int row, int col, int half_bytes) {
    return (uint32_t)((col >> 6) * half_bytes + row * 128 + ((((col >> 3) & 7) ^ (row & 7)) << 4) + (col & 7) * 2);
}

}  // namespace

// -------------------------------------------------------------------------------------------------
// encode: x = W (hits * scale) + b, hs = rms_norm(x) w.  A lane keeps its 4 output columns of W in
// registers, a warp takes 8 rows at a time through shared memory; 864 bytes per row move.
// -------------------------------------------------------------------------------------------------
constexpr int ENC_IN = 24;

__global__ void __launch_bounds__(256) model_encode_kernel(const float* __restrict__ hits, const float* __restrict__ scale,
                                                           const float* __restrict__ W, const float* __restrict__ bias,
                                                           const float* __restrict__ nw, float eps, int64_t n,
                                                           float* __restrict__ x, __nv_bfloat16* __restrict__ hs) {
    if (chain_wait()) return;
    __shared__ __align__(16) float rows[8][8 * ENC_IN];
    __shared__ float sw[MD * (ENC_IN + 1)];                  // W through shared memory: a lane's four rows are 96 scattered words
    for (int i = threadIdx.x; i < MD * ENC_IN; i += 256) sw[i / ENC_IN * (ENC_IN + 1) + i % ENC_IN] = __ldg(W + i);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float w[4][ENC_IN], b[4], g[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int i = 0; i < ENC_IN; ++i) w[c][i] = sw[(4 * lane + c) * (ENC_IN + 1) + i];
        b[c] = bias ? __ldg(bias + 4 * lane + c) : 0.f;
        g[c] = __ldg(nw + 4 * lane + c);
    }
    float sc[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) sc[i] = __ldg(scale + (lane + 32 * i) % ENC_IN);
    const int64_t step = (int64_t)gridDim.x * 64;
    int64_t r0 = ((int64_t)blockIdx.x * 8 + warp) * 8;
    float ahead[6];                                          // the warp's next eight rows
    auto fetch = [&](int64_t r) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const int e = lane + 32 * i;
            ahead[i] = r + e / ENC_IN < n ? __ldg(hits + r * ENC_IN + e) : 0.f;
        }
    };
    fetch(r0);
    for (; r0 < n; r0 += step) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 6; ++i) rows[warp][lane + 32 * i] = ahead[i] * sc[i];
        __syncwarp();
        fetch(r0 + step);
#pragma unroll 1
        for (int q = 0; q < 8 && r0 + q < n; q += 4) {           // four rows at a time: their reductions overlap
            float y[4][4], ss[4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) y[r][c] = b[c];
#pragma unroll
            for (int i = 0; i < ENC_IN; i += 4)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float4 h = *reinterpret_cast<const float4*>(&rows[warp][(q + r) * ENC_IN + i]);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        y[r][c] = fmaf(h.w, w[c][i + 3], fmaf(h.z, w[c][i + 2], fmaf(h.y, w[c][i + 1], fmaf(h.x, w[c][i], y[r][c]))));
                }
#pragma unroll
            for (int r = 0; r < 4; ++r) ss[r] = y[r][0] * y[r][0] + y[r][1] * y[r][1] + y[r][2] * y[r][2] + y[r][3] * y[r][3];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int r = 0; r < 4; ++r) ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], o);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (r0 + q + r >= n) break;
                const float rstd = rsqrtf(ss[r] * (1.f / MD) + eps);
                *reinterpret_cast<float4*>(x + (r0 + q + r) * MD + 4 * lane) = make_float4(y[r][0], y[r][1], y[r][2], y[r][3]);
                *reinterpret_cast<uint2*>(hs + (r0 + q + r) * MD + 4 * lane) =
                    make_uint2(pack_bf16x2(y[r][0] * rstd * g[0], y[r][1] * rstd * g[1]), pack_bf16x2(y[r][2] * rstd * g[2], y[r][3] * rstd * g[3]));
            }
        }
    }
}

// -------------------------------------------------------------------------------------------------
// head: out = x W^T + b, 24 outputs.  128 rows per CTA through shared memory; thread = 2 rows x 6
// outputs, so that eight 16-byte loads feed 48 multiply-adds.  608 bytes per row move.
// -------------------------------------------------------------------------------------------------
constexpr int HEAD_OUT = 24, HEAD_PITCH = MD + 4, HEAD_ROWS = 128;
constexpr int HEAD_SMEM = (HEAD_ROWS + HEAD_OUT) * HEAD_PITCH * 4;

__global__ void __launch_bounds__(256) model_head_kernel(const float* __restrict__ x, const float* __restrict__ W,
                                                         const float* __restrict__ bias, int64_t n, float* __restrict__ out) {
    if (chain_wait()) return;
    extern __shared__ __align__(16) float head_smem[];
    float* sx = head_smem;                                   // [128][132]
    float* sw = sx + HEAD_ROWS * HEAD_PITCH;                 // [24][132]
    const int tid = threadIdx.x;
    for (int i = tid; i < HEAD_OUT * 32; i += 256)
        *reinterpret_cast<float4*>(sw + (i >> 5) * HEAD_PITCH + 4 * (i & 31)) = __ldg(reinterpret_cast<const float4*>(W) + i);
    const int og = (tid & 3) * 6, row = tid >> 2;            // rows row, row + 64
    for (int64_t r0 = (int64_t)blockIdx.x * HEAD_ROWS; r0 < n; r0 += (int64_t)gridDim.x * HEAD_ROWS) {
        __syncthreads();
        const int m = (int)min((int64_t)HEAD_ROWS, n - r0);
#pragma unroll 8
        for (int i = 0; i < 16; ++i) {
            const int r = 8 * i + (tid >> 5), c = tid & 31;
            if (r < m) *reinterpret_cast<float4*>(sx + r * HEAD_PITCH + 4 * c) = __ldg(reinterpret_cast<const float4*>(x + (r0 + r) * MD) + c);
        }
        __syncthreads();
        float y[2][6];
#pragma unroll
        for (int o = 0; o < 6; ++o) {
            const float b = bias ? __ldg(bias + og + o) : 0.f;
#pragma unroll
            for (int i = 0; i < 2; ++i) y[i][o] = b;
        }
#pragma unroll 2
        for (int c = 0; c < MD; c += 4) {
            float4 v[2], w[6];
#pragma unroll
            for (int i = 0; i < 2; ++i) v[i] = *reinterpret_cast<const float4*>(sx + (row + 64 * i) * HEAD_PITCH + c);
#pragma unroll
            for (int o = 0; o < 6; ++o) w[o] = *reinterpret_cast<const float4*>(sw + (og + o) * HEAD_PITCH + c);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int o = 0; o < 6; ++o)
                    y[i][o] = fmaf(v[i].w, w[o].w, fmaf(v[i].z, w[o].z, fmaf(v[i].y, w[o].y, fmaf(v[i].x, w[o].x, y[i][o]))));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (row + 64 * i < m)
#pragma unroll
                for (int o = 0; o < 6; o += 2)
                    *reinterpret_cast<float2*>(out + (r0 + row + 64 * i) * HEAD_OUT + og + o) = make_float2(y[i][o], y[i][o + 1]);
    }
}

// -------------------------------------------------------------------------------------------------
// project.  A tile is 112 positions of the ordered batch with the 8 before them.  The products are
// taken transposed, D[channel][position] = W x hs^T: a thread then owns one channel (tensor-memory
// lane) and 28 consecutive positions in registers, which makes the 4-tap convolution a register
// window.  Five blocks of 128 channels: q, k, v, gate, (a | b | l).  Results pass through a
// [position][channel] tile in shared memory and leave as one bulk store per block (the rows of a
// tile are contiguous in every output).
// -------------------------------------------------------------------------------------------------
constexpr int PJ_OUT = 112, PJ_ROWS = 128, PJ_HALO = 16;       // positions per tile; operand rows; the first output row
constexpr int PJ_PART = PJ_OUT / (MWARPS / 4);                 // positions of a thread
constexpr int PJ_B = 2048;                                     // two swizzled [128][64] halves
constexpr int PJ_W = PJ_B + 2 * MST;
constexpr int PJ_ST = PJ_W + MNST * MST;                       // [112][128] bf16
constexpr int PJ_SMEM = PJ_ST + PJ_OUT * MD * 2;
constexpr int PJ_THREADS = (MWARPS + 1) * 32;
constexpr int PJ_BLOCKS = 5;
constexpr int PJ_ROW_A = 112, PJ_ROW_B = 120;                  // weight rows of a and b in the last block, l from row 0: in warps of their own up to H * L = 96

struct ProjArgs {
    const __nv_bfloat16* hs; const int64_t* perm; const int64_t* cu; int nseq; int64_t n;
    const __nv_bfloat16* conv[3];            // [128][4]
    const float* A_log; const float* dt_bias; const float* Lw;
    int H, L;
    __nv_bfloat16* out[4];                   // q, k, v, gate [n][128]
    float* g; float* beta; __nv_bfloat16* lam;   // [n][H], [n][H], [n][H * L]
    int32_t* status; int budget;
};

// PARTS > 1: the blocks of a tile shared out over CTAs of their own, for batches whose tiles leave SMs idle: a tile is then one or two
// blocks long instead of five (9,001 rows, 81 tiles: 24 -> 19 us).
template <int PARTS>
__global__ void __launch_bounds__(PJ_THREADS, 2)
model_project_kernel(ProjArgs a, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                     const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mg,
                     const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                     const __grid_constant__ CUtensorMap ml) {
    if (chain_wait()) return;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);        // weight piece landed
    uint64_t* mdone = full + MNST;                             // products of a block complete, by accumulator
    uint64_t* dfree = mdone + 2;                               // accumulator read
    uint64_t* bready = dfree + 2;                              // operand rows in place
    uint64_t* drain = bready + 1;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 128);
    uint32_t* sstart = reinterpret_cast<uint32_t*>(smem + 144);   // bit p: operand row p opens an event
    int64_t* srow = reinterpret_cast<int64_t*>(smem + 1024);
    unsigned char* sB = smem + PJ_B;
    unsigned char* sW = smem + PJ_W;
    unsigned char* sST = smem + PJ_ST;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t ntiles = (a.n + PJ_OUT - 1) / PJ_OUT;
    const int cta = blockIdx.x / PARTS, ctas = gridDim.x / PARTS, piece = blockIdx.x % PARTS;
    constexpr int PER = (PJ_BLOCKS + PARTS - 1) / PARTS;            // blocks of a part; the last one has the rest
    const int m0 = PARTS == 1 ? 0 : piece * PER, m1 = PARTS == 1 ? PJ_BLOCKS : min(m0 + PER, PJ_BLOCKS), nb = m1 - m0;
    const int mine = cta < ntiles ? (int)((ntiles - cta + ctas - 1) / ctas) : 0;

    if (tid == 0) {
        for (int s = 0; s < MNST; ++s) mbar_init(full + s, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(mdone + s, 1); mbar_init(dfree + s, MWARPS); }
        mbar_init(bready, MWARPS);
        mbar_init(drain, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, 256);
    // operand rows before the halo are never written and never read back, but their products are formed: finite zeros
    for (int i = tid; i < 2 * 8 * 8; i += PJ_THREADS)
        *reinterpret_cast<uint4*>(sB + (i >> 6) * MST + (i & 63) * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *tslot;
    bool dead = false;

    if (warp == MWARPS) {
        if (lane == 0) {
            const int npieces = mine * nb * 2;
            int loaded = 0, landed = 0;
            auto load = [&](int p) {                             // piece p: block (p / 2) % 5, half p & 1 of its 128 inputs
                uint64_t* b = full + p % MNST;
                unsigned char* dst = sW + (size_t)(p % MNST) * MST;
                const int blk = m0 + (p >> 1) % nb, x = (p & 1) * 64;
                if (blk < 4) {
                    mbar_expect_tx(b, MST);
                    tma_load_2d(dst, blk == 0 ? &mq : blk == 1 ? &mk : blk == 2 ? &mv : &mg, x, 0, b);
                } else {
                    mbar_expect_tx(b, (uint32_t)(2 * a.H + a.H * a.L) * 128);
                    tma_load_2d(dst + PJ_ROW_A * 128, &ma, x, 0, b);
                    tma_load_2d(dst + PJ_ROW_B * 128, &mb, x, 0, b);
                    tma_load_2d(dst, &ml, x, 0, b);
                }
                loaded = p + 1;
            };
            for (int p = 0; p < MNST && p < npieces; ++p) load(p);
            for (int t = 0; t < mine && !dead; ++t) {
                mbar_wait(bready, (uint32_t)(t & 1), dead, a.status, 600, a.budget);
                for (int m = m0; m < m1 && !dead; ++m) {
                    const int q = t * nb + m - m0, buf = q & 1;
                    if (q >= 2) mbar_wait(dfree + buf, (uint32_t)(((q >> 1) - 1) & 1), dead, a.status, 601, a.budget);
                    for (int h = 0; h < 2 && !dead; ++h) {
                        const int p = 2 * q + h;
                        if (mbar_wait(full + p % MNST, (uint32_t)((p / MNST) & 1), dead, a.status, 602, a.budget)) landed = p + 1;
                        if (dead) break;
                        tc_fence_after();
                        const uint64_t da = umma_desc_k128(smem_u32(sW + (size_t)(p % MNST) * MST));
                        const uint64_t db = umma_desc_k128(smem_u32(sB + h * MST));
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umma_f16_ss(taddr + 128 * buf, da + 2 * kk, db + 2 * kk, umma_idesc(128, 128), h | kk ? 1u : 0u);
                    }
                    if (dead) break;
                    umma_commit(mdone + buf);
                    // the two stages of this block are free once its products are done
                    mbar_wait(mdone + buf, (uint32_t)((q >> 1) & 1), dead, a.status, 603, a.budget);
                    for (int p = 2 * q + MNST; p < 2 * q + MNST + 2 && p < npieces && !dead; ++p) load(p);
                }
            }
            for (int p = landed; p < loaded; ++p) mbar_drain(full + p % MNST, (uint32_t)((p / MNST) & 1));
            umma_commit(drain);
            mbar_drain(drain, 0u);
        }
    } else {
        const int quarter = warp & 3, part = warp >> 2;          // channels 32 quarter + lane; positions 28 part ..
        const int ch = 32 * quarter + lane;
        const uint32_t tl = taddr + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(PJ_HALO - 4 + PJ_PART * part);
        const int HL = a.H * a.L;
        // last block: the channel is a (g), b (beta), l (lambda) or nothing; g and lambda are scale * softplus(mul x + add)
        const bool is_a = ch >= PJ_ROW_A && ch < PJ_ROW_A + a.H, is_b = ch >= PJ_ROW_B && ch < PJ_ROW_B + a.H, is_l = ch < HL;
        const float sp_scale = is_a ? -__expf(__ldg(a.A_log + ch - PJ_ROW_A)) : 1.f, sp_add = is_a ? __ldg(a.dt_bias + ch - PJ_ROW_A) : 0.f;
        const float sp_mul = is_l ? __ldg(a.Lw + ch) : 1.f;

        // the rows of hs that tile t takes, in LSH order: found under the gate block of the tile before, fetched under its
        // last epilogue (both are chains of dependent loads); 2.05 M rows: 1,667 -> 1,629 us
        auto find_rows = [&](int t) {                            // warps 0..3
            const int64_t j = (cta + (int64_t)t * ctas) * PJ_OUT - PJ_HALO + tid;            // operand row tid
            bool first = false;
            int64_t r = -1;
            if (tid >= 8 && j >= 0 && j < a.n) r = ordered_row(a.cu, a.nseq, a.perm, j, a.n, a.status, &first);
            srow[tid] = r;
            const uint32_t bits = __ballot_sync(0xffffffffu, first);
            if (lane == 0) sstart[warp] = bits;
        };
        auto fetch_rows = [&] {
            for (int i = tid; i < (PJ_ROWS - 8) * 16; i += METHR) {
                const int row = 8 + (i >> 4), c = i & 15;
                const int64_t r = srow[row];
                unsigned char* dst = sB + op_off(row, 8 * c, MST);
                if (r >= 0) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(smem_u32(dst)), "l"(a.hs + r * MD + 8 * c) : "memory");
                else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        if (mine > 0) {
            if (warp < 4) find_rows(0);
            epi_sync();
            fetch_rows();
        }
        for (int t = 0; t < mine; ++t) {
            const int64_t tile = cta + (int64_t)t * ctas, j0 = tile * PJ_OUT;
            const int nv = (int)min((int64_t)PJ_OUT, a.n - j0);
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bready);
            // event starts of this thread's 28 positions and the 4 before: bit i = operand row p0 + i
            const int p0 = PJ_HALO - 4 + PJ_PART * part;
            const uint32_t starts = __funnelshift_r(sstart[p0 >> 5], (p0 >> 5) < 3 ? sstart[(p0 >> 5) + 1] : 0u, p0 & 31);
            for (int m = m0; m < m1; ++m) {
                const int q = t * nb + m - m0, buf = q & 1;
                uint2 taps = make_uint2(0u, 0u);                 // this channel's four taps
                if (m < 3) taps = __ldg(reinterpret_cast<const uint2*>(m == 0 ? a.conv[0] : m == 1 ? a.conv[1] : a.conv[2]) + ch);
                epi_wait(mdone + buf, (uint32_t)((q >> 1) & 1), dead, a.status, 610, a.budget, [] {});      // products complete
                tc_fence_after();
                if (PARTS == 1 && m == PJ_BLOCKS - 1 && t + 1 < mine) fetch_rows();        // the tile's last products: its operand is free
                float x[32];                                     // X(i) = position i - 4
                tmem_ld32(x, tl + 128 * buf);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(dfree + buf);
                uint32_t w[PJ_PART / 2];                         // the 28 results
                if (m < 3) {
                    float h1 = x[3], h2 = x[2], h3 = x[1];
                    const float2 ta = unpack_bf16x2(taps.x), tb = unpack_bf16x2(taps.y);
                    const float w0 = ta.x, w1 = ta.y, w2 = tb.x, w3 = tb.y;
                    auto tap = [&](int i) {
                        const float v = fmaf(w0, h3, fmaf(w1, h2, fmaf(w2, h1, w3 * x[4 + i])));
                        h3 = h2; h2 = h1; h1 = x[4 + i];
                        return v * sigmoid_fast(v);
                    };
                    if (starts == 0) {
#pragma unroll
                        for (int i = 0; i < PJ_PART / 2; ++i) { const float u = tap(2 * i); w[i] = pack_bf16x2(u, tap(2 * i + 1)); }
                    } else {                                     // an event opens here: its first taps are empty
                        if ((starts >> 3) & 1) h2 = h3 = 0.f;
                        if ((starts >> 2) & 1) h3 = 0.f;
#pragma unroll
                        for (int i = 0; i < PJ_PART / 2; ++i) {
                            if ((starts >> (4 + 2 * i)) & 1) h1 = h2 = h3 = 0.f;
                            const float u = tap(2 * i);
                            if ((starts >> (5 + 2 * i)) & 1) h1 = h2 = h3 = 0.f;
                            w[i] = pack_bf16x2(u, tap(2 * i + 1));
                        }
                    }
                } else if (m == 3) {
#pragma unroll
                    for (int i = 0; i < PJ_PART / 2; ++i) w[i] = pack_bf16x2(x[4 + 2 * i], x[5 + 2 * i]);
                } else if (quarter < 3 || is_l) {
#pragma unroll
                    for (int i = 0; i < PJ_PART / 2; ++i) w[i] = pack_bf16x2(softplusf_(sp_mul * x[4 + 2 * i]), softplusf_(sp_mul * x[5 + 2 * i]));
                } else if (is_a || is_b) {                       // g and beta: straight to their rows
                    float* gp = (is_a ? a.g + ch - PJ_ROW_A : a.beta + ch - PJ_ROW_B) + (j0 + PJ_PART * part) * a.H;
#pragma unroll
                    for (int i = 0; i < PJ_PART; ++i)
                        if (PJ_PART * part + i < nv) gp[i * a.H] = is_a ? sp_scale * softplusf_(x[4 + i] + sp_add) : sigmoid_fast(x[4 + i]);
                }
                if (PARTS == 1 && m == 3 && t + 1 < mine && warp < 4) find_rows(t + 1);      // (shared-out tiles: one to a CTA)
                if (tid == 0) bulk_wait_read();                  // the previous results have left the staging tile
                epi_sync();
                uint16_t* st = reinterpret_cast<uint16_t*>(sST) + ch;
                if (m < 4) {
                    st += PJ_PART * part * MD;
#pragma unroll
                    for (int i = 0; i < PJ_PART / 2; ++i) { st[2 * i * MD] = (uint16_t)w[i]; st[(2 * i + 1) * MD] = (uint16_t)(w[i] >> 16); }
                } else if (is_l) {
                    st += PJ_PART * part * HL;
#pragma unroll
                    for (int i = 0; i < PJ_PART / 2; ++i) { st[2 * i * HL] = (uint16_t)w[i]; st[(2 * i + 1) * HL] = (uint16_t)(w[i] >> 16); }
                }
                fence_async_smem();
                epi_sync();
                const uint32_t bytes = (uint32_t)nv * (m < 4 ? MD : HL) * 2;
                char* dst = m < 4 ? (char*)(m == 0 ? a.out[0] : m == 1 ? a.out[1] : m == 2 ? a.out[2] : a.out[3]) + j0 * MD * 2 : (char*)a.lam + j0 * HL * 2;
                if (bytes % 16 == 0) {
                    if (tid == 0) { bulk_s2g(dst, sST, bytes); bulk_commit(); }
                } else {                                         // last rows of lambda: not whole 16-byte pieces
                    for (int i = tid; i < nv * HL; i += METHR) a.lam[j0 * HL + i] = reinterpret_cast<const __nv_bfloat16*>(sST)[i];
                }
            }
        }
        if (tid == 0) bulk_wait_read();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(taddr, 256);
}

// -------------------------------------------------------------------------------------------------
// update.  A tile is 128 positions of the ordered batch.  Row-wise steps (gated norm, residual and
// norm) give a warp 8 rows, four columns per lane; products leave tensor memory one row per lane and
// go through the operand tile (bf16) to the row-wise layout.  The hidden layer never leaves the SM:
// eight chunks of 64 hidden units, each up product -> bias, GELU -> bf16 operand -> accumulated into
// the down product, the up product of the next chunk under the GELU of this one.
// Bound by the epilogues' instruction issue (the GELU alone is 65 k elements per tile), not by HBM.
// -------------------------------------------------------------------------------------------------
constexpr int UP_ROWS = 128, UP_WROWS = UP_ROWS / MWARPS, UP_HID = 512, UP_CH = 64, UP_NCH = UP_HID / UP_CH;
constexpr int UP_A = 1024;                                     // operand tile: two swizzled [128][64] halves
constexpr int UP_H = UP_A + 2 * MST;                           // hidden operand, two buffers of [128][64]
constexpr int UP_W = UP_H + 2 * MST;
constexpr int UP_SMEM = UP_W + MNST * MST;                     // 113 KB: two CTAs fill an SM exactly
constexpr int UP_THREADS = (MWARPS + 2) * 32;                  // + one warp issues products, one streams weights
constexpr int UP_PIECES = 2 + 2 * UP_NCH;                      // o_proj halves, then up and down of every chunk
constexpr int UT_UP = 0, UT_ACC = 128;                         // tensor-memory columns: two 64-column up accumulators; o_proj / down

struct UpdateArgs {
    const __nv_bfloat16* o; const __nv_bfloat16* gate; const __nv_bfloat16* o_norm_w; int head_dim;
    float* x; const int64_t* perm; const int64_t* cu; int nseq; int64_t n;
    const float* mlp_norm_w; const __nv_bfloat16* up_b; const __nv_bfloat16* down_b;
    const float* next_norm_w; __nv_bfloat16* hs;             // NULL: last block, no norm behind it
    float eps, next_eps, o_eps;
    int32_t* status; int budget;
};

__global__ void __launch_bounds__(UP_THREADS, 2)
model_update_kernel(UpdateArgs a, const __grid_constant__ CUtensorMap mo, const __grid_constant__ CUtensorMap mu,
                    const __grid_constant__ CUtensorMap md) {
    if (chain_wait()) return;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);        // weight piece landed
    uint64_t* wfree = full + MNST;                             // its products are done
    uint64_t* aready = wfree + MNST;                           // operand tile written
    uint64_t* macc = aready + 1;                               // o_proj / down complete
    uint64_t* mup = macc + 1;                                  // up product complete, by accumulator
    uint64_t* upfree = mup + 2;                                // up accumulator read
    uint64_t* hready = upfree + 2;                             // hidden operand written
    uint64_t* hfree = hready + 2;                              // hidden operand consumed
    uint64_t* drain = hfree + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 256);
    unsigned char* sA = smem + UP_A;
    unsigned char* sH = smem + UP_H;
    unsigned char* sW = smem + UP_W;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t ntiles = (a.n + UP_ROWS - 1) / UP_ROWS;
    const int mine = blockIdx.x < ntiles ? (int)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;

    if (tid == 0) {
        for (int s = 0; s < MNST; ++s) { mbar_init(full + s, 1); mbar_init(wfree + s, 1); }
        mbar_init(aready, MWARPS);
        mbar_init(macc, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(mup + s, 1); mbar_init(upfree + s, MWARPS); mbar_init(hready + s, MWARPS); mbar_init(hfree + s, 1); }
        mbar_init(drain, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *tslot;
    bool dead = false;
    const int npieces = mine * UP_PIECES;

    if (warp == MWARPS + 1) {
        // ---- weights: o_proj k-halves, then [64 hidden][128] of up and [128][64 hidden] of down, chunk by chunk ----
        if (lane == 0) {
            int p = 0;
            for (; p < npieces; ++p) {
                const int s = p % MNST, k = p % UP_PIECES;
                if (p >= MNST && !mbar_wait(wfree + s, (uint32_t)((p / MNST - 1) & 1), dead, a.status, 620, a.budget)) break;
                unsigned char* dst = sW + (size_t)s * MST;
                mbar_expect_tx(full + s, MST);
                if (k < 2) tma_load_2d(dst, &mo, 64 * k, 0, full + s);
                else {
                    // order of use: up 0, up 1, down 0, up 2, down 1, ..., up 7, down 6, down 7
                    const int i = k - 2;
                    const bool up = i == 0 || (i < 2 * UP_NCH - 1 && (i & 1));
                    const int c = up ? (i + 1) / 2 : (i == 2 * UP_NCH - 1 ? UP_NCH - 1 : i / 2 - 1);
                    if (up) {
                        tma_load_2d(dst, &mu, 0, UP_CH * c, full + s);
                        tma_load_2d(dst + MST / 2, &mu, 64, UP_CH * c, full + s);
                    } else {
                        tma_load_2d(dst, &md, UP_CH * c, 0, full + s);
                    }
                }
            }
            // nothing may land after the CTA has gone
            for (int i = max(0, p - MNST); i < p; ++i) mbar_drain(full + i % MNST, (uint32_t)((i / MNST) & 1));
        }
    } else if (warp == MWARPS) {
        // ---- products ----
        if (lane == 0) {
            int p = 0;
            auto piece = [&]() -> uint32_t {                     // wait for the next weight piece
                mbar_wait(full + p % MNST, (uint32_t)((p / MNST) & 1), dead, a.status, 621, a.budget);
                tc_fence_after();
                return smem_u32(sW + (size_t)(p % MNST) * MST);
            };
            for (int t = 0; t < mine && !dead; ++t) {
                mbar_wait(aready, 0u, dead, a.status, 622, a.budget);           // two phases per tile: normed mixer rows, then normed residual rows
                for (int h = 0; h < 2 && !dead; ++h) {
                    const uint64_t db = umma_desc_k128(piece()), da = umma_desc_k128(smem_u32(sA + h * MST));
                    if (dead) break;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16_ss(taddr + UT_ACC, da + 2 * kk, db + 2 * kk, umma_idesc(128, 128), h | kk ? 1u : 0u);
                    umma_commit(wfree + p % MNST);
                    ++p;
                }
                if (dead) break;
                umma_commit(macc);
                mbar_wait(aready, 1u, dead, a.status, 623, a.budget);
                auto up = [&](int c) {
                    const int q = t * UP_NCH + c, buf = q & 1;
                    if (q >= 2) mbar_wait(upfree + buf, (uint32_t)(((q >> 1) - 1) & 1), dead, a.status, 624, a.budget);
                    const uint32_t w = piece();
                    if (dead) return;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint64_t da = umma_desc_k128(smem_u32(sA + h * MST)), db = umma_desc_k128(w + h * (MST / 2));
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umma_f16_ss(taddr + UT_UP + 64 * buf, da + 2 * kk, db + 2 * kk, umma_idesc(128, 64), h | kk ? 1u : 0u);
                    }
                    umma_commit(wfree + p % MNST);
                    umma_commit(mup + buf);
                    ++p;
                };
                auto down = [&](int c) {
                    const int q = t * UP_NCH + c, buf = q & 1;
                    mbar_wait(hready + buf, (uint32_t)((q >> 1) & 1), dead, a.status, 625, a.budget);
                    const uint64_t db = umma_desc_k128(piece()), da = umma_desc_k128(smem_u32(sH + buf * MST));
                    if (dead) return;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16_ss(taddr + UT_ACC, da + 2 * kk, db + 2 * kk, umma_idesc(128, 128), c | kk ? 1u : 0u);
                    umma_commit(wfree + p % MNST);
                    umma_commit(hfree + buf);
                    ++p;
                };
                up(0);
                for (int c = 1; c < UP_NCH && !dead; ++c) { up(c); if (!dead) down(c - 1); }
                if (!dead) down(UP_NCH - 1);
                if (!dead) umma_commit(macc);
            }
            umma_commit(drain);
            mbar_drain(drain, 0u);
        }
    } else {
        const int quarter = warp & 3, part = warp >> 2;
        const uint32_t tl = taddr + ((uint32_t)(32 * quarter) << 16);
        const int trow = 32 * quarter + lane;                    // this thread's row of an accumulator
        const int lanes_per_head = a.head_dim >> 2;
        const float inv_dim = 1.f / (float)a.head_dim;
        float ow[4], mw[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            ow[c] = a.o_norm_w ? __bfloat162float(a.o_norm_w[(4 * lane + c) % a.head_dim]) : 1.f;
            mw[c] = __ldg(a.mlp_norm_w + 4 * lane + c);
        }
        // accumulator quarter-row -> bf16 -> operand tile (row-wise readers pick it up there)
        auto stage_acc = [&](const __nv_bfloat16* bias) {
            float x[32];
            tmem_ld32(x, tl + UT_ACC + 32 * part);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float* v = &x[8 * q];
                if (bias) {
                    const uint4 b = __ldg(reinterpret_cast<const uint4*>(bias + 32 * part) + q);
                    const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) { const float2 f = unpack_bf16x2(bw[e]); v[2 * e] += f.x; v[2 * e + 1] += f.y; }
                }
                *reinterpret_cast<uint4*>(sA + op_off(trow, 32 * part + 8 * q, MST)) =
                    make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
            }
        };
        auto operand_ready = [&]() {
            fence_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(aready);
        };
        for (int t = 0; t < mine; ++t) {
            const int64_t j0 = ((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * UP_ROWS + UP_WROWS * warp;   // this warp's rows
            const int nr = (int)min((int64_t)UP_WROWS, max((int64_t)0, a.n - j0));
            int64_t myrow = -1;
            if (lane < nr) myrow = ordered_row(a.cu, a.nseq, a.perm, j0 + lane, a.n, a.status);
            {   // the residual rows are wanted one product later: into L2 now (four lines each)
                const int64_t pr = __shfl_sync(0xffffffffu, myrow, lane >> 2);
                if (pr >= 0) asm volatile("prefetch.global.L2 [%0];\n" :: "l"(a.x + pr * MD + 32 * (lane & 3)));
            }
            // ---- gated norm of the mixer's rows: the operand of o_proj ----
#pragma unroll 1
            for (int r0 = 0; r0 < UP_WROWS; r0 += 4) {
                uint2 ov[4], gv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool in = r0 + i < nr;
                    ov[i] = in ? __ldg(reinterpret_cast<const uint2*>(a.o + (j0 + r0 + i) * MD) + lane) : make_uint2(0u, 0u);
                    gv[i] = in ? __ldg(reinterpret_cast<const uint2*>(a.gate + (j0 + r0 + i) * MD) + lane) : make_uint2(0u, 0u);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 o0 = unpack_bf16x2(ov[i].x), o1 = unpack_bf16x2(ov[i].y), g0 = unpack_bf16x2(gv[i].x), g1 = unpack_bf16x2(gv[i].y);
                    float ss = o0.x * o0.x + o0.y * o0.y + o1.x * o1.x + o1.y * o1.y;
                    for (int o = lanes_per_head >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    const float rstd = rsqrtf(ss * inv_dim + a.o_eps);
                    *reinterpret_cast<uint2*>(sA + op_off(UP_WROWS * warp + r0 + i, 4 * lane, MST)) =
                        make_uint2(pack_bf16x2(o0.x * rstd * ow[0] * g0.x * sigmoid_fast(g0.x), o0.y * rstd * ow[1] * g0.y * sigmoid_fast(g0.y)),
                                   pack_bf16x2(o1.x * rstd * ow[2] * g1.x * sigmoid_fast(g1.x), o1.y * rstd * ow[3] * g1.y * sigmoid_fast(g1.y)));
                }
            }
            operand_ready();
            // ---- x += o_proj at the hit's row, norm: the operand of the MLP ----
            epi_wait(macc, 0u, dead, a.status, 630, a.budget, [] {});
            tc_fence_after();
            stage_acc(nullptr);
            epi_sync();
#pragma unroll 1
            for (int r0 = 0; r0 < UP_WROWS; r0 += 4) {
                float4 v[4];
                int64_t rr[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    rr[i] = __shfl_sync(0xffffffffu, myrow, r0 + i);
                    v[i] = rr[i] >= 0 ? *reinterpret_cast<const float4*>(a.x + rr[i] * MD + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint2* op = reinterpret_cast<uint2*>(sA + op_off(UP_WROWS * warp + r0 + i, 4 * lane, MST));
                    const float2 d0 = unpack_bf16x2(op->x), d1 = unpack_bf16x2(op->y);
                    v[i].x += d0.x; v[i].y += d0.y; v[i].z += d1.x; v[i].w += d1.y;
                    if (rr[i] >= 0) *reinterpret_cast<float4*>(a.x + rr[i] * MD + 4 * lane) = v[i];
                    float ss = v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    const float rstd = rsqrtf(ss * (1.f / MD) + a.eps);
                    *op = make_uint2(pack_bf16x2(v[i].x * rstd * mw[0], v[i].y * rstd * mw[1]), pack_bf16x2(v[i].z * rstd * mw[2], v[i].w * rstd * mw[3]));
                }
            }
            operand_ready();
            // ---- hidden layer, 64 units at a time: this thread has 16 of its row ----
#pragma unroll 1
            for (int c = 0; c < UP_NCH; ++c) {
                const int q = t * UP_NCH + c, buf = q & 1;
                uint4 bias[2];
                bias[0] = bias[1] = make_uint4(0u, 0u, 0u, 0u);
                if (a.up_b) {
                    const uint4* bp = reinterpret_cast<const uint4*>(a.up_b + UP_CH * c + 16 * part);
                    bias[0] = __ldg(bp);
                    bias[1] = __ldg(bp + 1);
                }
                if (c == UP_NCH - 2 && t + 1 < mine) {           // the next tile's mixer and gate rows, on their way to L2
                    const int64_t j = j0 + (int64_t)gridDim.x * UP_ROWS + (lane >> 2);
                    const __nv_bfloat16* base = (lane & 2) ? a.gate : a.o;
                    if (j < a.n) asm volatile("prefetch.global.L2 [%0];\n" :: "l"(base + j * MD + 64 * (lane & 1)));
                }
                // up product complete, and the hidden operand of two chunks ago consumed
                epi_wait(mup + buf, (uint32_t)((q >> 1) & 1), dead, a.status, 631, a.budget, [&] {
                    if (q >= 2) mbar_wait(hfree + buf, (uint32_t)(((q >> 1) - 1) & 1), dead, a.status, 632, a.budget);
                });
                tc_fence_after();
                float x[16];
                tmem_ld16(x, tl + UT_UP + 64 * buf + 16 * part);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(upfree + buf);
                const uint32_t bw[8] = {bias[0].x, bias[0].y, bias[0].z, bias[0].w, bias[1].x, bias[1].y, bias[1].z, bias[1].w};
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 f = unpack_bf16x2(bw[e]);
                    float y0, y1;
                    gelu_pair(x[2 * e] + f.x, x[2 * e + 1] + f.y, y0, y1);
                    w[e] = pack_bf16x2(y0, y1);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<uint4*>(sH + buf * MST + op_off(trow, 16 * part + 8 * e, 0)) = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(hready + buf);
            }
            // ---- x += MLP, the next block's norm ----
            epi_wait(macc, 1u, dead, a.status, 633, a.budget, [] {});
            tc_fence_after();
            stage_acc(a.down_b);
            tc_fence_before();
            epi_sync();
#pragma unroll 1
            for (int r0 = 0; r0 < UP_WROWS; r0 += 4) {
                float4 v[4];
                int64_t rr[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    rr[i] = __shfl_sync(0xffffffffu, myrow, r0 + i);
                    v[i] = rr[i] >= 0 ? *reinterpret_cast<const float4*>(a.x + rr[i] * MD + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint2 op = *reinterpret_cast<const uint2*>(sA + op_off(UP_WROWS * warp + r0 + i, 4 * lane, MST));
                    const float2 d0 = unpack_bf16x2(op.x), d1 = unpack_bf16x2(op.y);
                    v[i].x += d0.x; v[i].y += d0.y; v[i].z += d1.x; v[i].w += d1.y;
                    if (rr[i] < 0) continue;                     // warp-uniform
                    *reinterpret_cast<float4*>(a.x + rr[i] * MD + 4 * lane) = v[i];
                    if (!a.next_norm_w) continue;
                    float ss = v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    const float rstd = rsqrtf(ss * (1.f / MD) + a.next_eps);
                    const float4 nw = __ldg(reinterpret_cast<const float4*>(a.next_norm_w) + lane);
                    *reinterpret_cast<uint2*>(a.hs + rr[i] * MD + 4 * lane) =
                        make_uint2(pack_bf16x2(v[i].x * rstd * nw.x, v[i].y * rstd * nw.y), pack_bf16x2(v[i].z * rstd * nw.z, v[i].w * rstd * nw.w));
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(taddr, 256);
}

}  // namespace lampa

using namespace lampa;

extern "C" int lampa_model_encode(const float* hits, const float* scale, const float* weight, const float* bias,
                                  const float* norm_w, float eps, int64_t n, int32_t in_dim, int32_t d_model, float* x,
                                  void* hs, void* stream) {
    if (n < 0 || !hits || !scale || !weight || !norm_w || !x || !hs) return LAMPA_ERR_ARG;
    if (in_dim != ENC_IN || d_model != MD) return LAMPA_ERR_UNSUPPORTED;
    if (n == 0) return LAMPA_OK;
    ProfScope prof("model_encode", (cudaStream_t)stream);
    const int64_t want = (n + 63) / 64, most = (int64_t)sm_count() * 4;
    launch_chained(model_encode_kernel, (unsigned)(want < most ? want : most), 256, 0, (cudaStream_t)stream,
        hits, scale, weight, bias, norm_w, eps, n, x, (__nv_bfloat16*)hs);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_model_head(const float* x, const float* weight, const float* bias, int64_t n, int32_t d_model,
                                int32_t out_dim, float* out, void* stream) {
    if (n < 0 || !x || !weight || !out) return LAMPA_ERR_ARG;
    if (out_dim != HEAD_OUT || d_model != MD) return LAMPA_ERR_UNSUPPORTED;
    if (((uintptr_t)x | (uintptr_t)weight | (uintptr_t)out) & 15) return LAMPA_ERR_UNSUPPORTED;
    if (n == 0) return LAMPA_OK;
    ProfScope prof("model_head", (cudaStream_t)stream);
    static std::atomic<uint64_t> ready{0};
    if (!allow_smem(ready, model_head_kernel, HEAD_SMEM)) return LAMPA_ERR_CUDA;
    const int64_t want = (n + HEAD_ROWS - 1) / HEAD_ROWS, most = (int64_t)sm_count() * 2;
    launch_chained(model_head_kernel, (unsigned)(want < most ? want : most), 256, HEAD_SMEM, (cudaStream_t)stream, x, weight, bias, n, out);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_model_project(const lampa_model_mixer* w, const void* hs, const int64_t* perm, const int64_t* cu, int32_t nseq,
                                   int64_t n, void* q, void* k, void* v, void* gate, float* g, float* beta, void* lam,
                                   int32_t* status, void* stream) {
    if (!w || n < 0 || nseq <= 0) return LAMPA_ERR_ARG;
    if (n == 0) return LAMPA_OK;
    if (!hs || !perm || !cu || !q || !k || !v || !gate || !g || !beta || !lam) return LAMPA_ERR_ARG;
    if (w->H <= 0 || w->H > PJ_ROW_B - PJ_ROW_A || w->L <= 0 || w->H * w->L > PJ_ROW_A || MD % w->H != 0) return LAMPA_ERR_UNSUPPORTED;
    ProjArgs a;
    a.hs = (const __nv_bfloat16*)hs; a.perm = perm; a.cu = cu; a.nseq = nseq; a.n = n;
    a.conv[0] = (const __nv_bfloat16*)w->q_conv; a.conv[1] = (const __nv_bfloat16*)w->k_conv; a.conv[2] = (const __nv_bfloat16*)w->v_conv;
    a.A_log = w->A_log; a.dt_bias = w->dt_bias; a.Lw = w->Lw; a.H = w->H; a.L = w->L;
    a.out[0] = (__nv_bfloat16*)q; a.out[1] = (__nv_bfloat16*)k; a.out[2] = (__nv_bfloat16*)v; a.out[3] = (__nv_bfloat16*)gate;
    a.g = g; a.beta = beta; a.lam = (__nv_bfloat16*)lam; a.status = status; a.budget = poll_budget();
    for (const void* p : {w->q_w, w->k_w, w->v_w, w->g_w, w->a_w, w->b_w, w->l_w, hs, (const void*)q, (const void*)k, (const void*)v, (const void*)gate, (const void*)lam})
        if (!p || ((uintptr_t)p & 15)) return LAMPA_ERR_UNSUPPORTED;
    for (const void* p : {w->q_conv, w->k_conv, w->v_conv})
        if (!p || ((uintptr_t)p & 7)) return LAMPA_ERR_UNSUPPORTED;
    const void* mats[7] = {w->q_w, w->k_w, w->v_w, w->g_w, w->a_w, w->b_w, w->l_w};
    const uint32_t rows[7] = {MD, MD, MD, MD, (uint32_t)w->H, (uint32_t)w->H, (uint32_t)(w->H * w->L)};
    CUtensorMap m[7];
    for (int i = 0; i < 7; ++i)
        if (!make_map(&m[i], mats[i], LAMPA_BF16, rows[i], MD, 64, rows[i], true)) return LAMPA_ERR_UNSUPPORTED;
    static std::atomic<uint64_t> ready[3];
    if (!allow_smem(ready[0], model_project_kernel<1>, PJ_SMEM) || !allow_smem(ready[1], model_project_kernel<2>, PJ_SMEM) ||
        !allow_smem(ready[2], model_project_kernel<3>, PJ_SMEM)) return LAMPA_ERR_CUDA;
    ProfScope prof("model_project", (cudaStream_t)stream);
    const int64_t want = (n + PJ_OUT - 1) / PJ_OUT, most = (int64_t)sm_count() * 2;
    // as many parts as all run at once, two CTAs to an SM
    if (3 * want <= most) launch_chained(model_project_kernel<3>, (unsigned)(3 * want), PJ_THREADS, PJ_SMEM, (cudaStream_t)stream, a, m[0], m[1], m[2], m[3], m[4], m[5], m[6]);
    else if (2 * want <= most) launch_chained(model_project_kernel<2>, (unsigned)(2 * want), PJ_THREADS, PJ_SMEM, (cudaStream_t)stream, a, m[0], m[1], m[2], m[3], m[4], m[5], m[6]);
    else launch_chained(model_project_kernel<1>, (unsigned)(want < most ? want : most), PJ_THREADS, PJ_SMEM, (cudaStream_t)stream, a, m[0], m[1], m[2], m[3], m[4], m[5], m[6]);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_model_update(const lampa_model_update_w* w, const void* o, const void* gate, float* x, const int64_t* perm,
                                  const int64_t* cu, int32_t nseq, int64_t n, void* hs, int32_t* status, void* stream) {
    if (!w || n < 0 || nseq <= 0) return LAMPA_ERR_ARG;
    if (n == 0) return LAMPA_OK;
    if (!o || !gate || !x || !perm || !cu || (w->next_norm_w && !hs)) return LAMPA_ERR_ARG;
    if (w->head_dim != 32 && w->head_dim != 64) return LAMPA_ERR_UNSUPPORTED;
    for (const void* p : {w->o_w, w->up_w, w->down_w, o, gate, (const void*)x})
        if (!p || ((uintptr_t)p & 15)) return LAMPA_ERR_UNSUPPORTED;
    for (const void* p : {w->up_b, w->down_b, (const void*)w->next_norm_w, (const void*)hs})
        if (p && ((uintptr_t)p & 15)) return LAMPA_ERR_UNSUPPORTED;
    UpdateArgs a;
    a.o = (const __nv_bfloat16*)o; a.gate = (const __nv_bfloat16*)gate; a.o_norm_w = (const __nv_bfloat16*)w->o_norm_w; a.head_dim = w->head_dim;
    a.x = x; a.perm = perm; a.cu = cu; a.nseq = nseq; a.n = n;
    a.mlp_norm_w = w->mlp_norm_w; a.up_b = (const __nv_bfloat16*)w->up_b; a.down_b = (const __nv_bfloat16*)w->down_b;
    a.next_norm_w = w->next_norm_w; a.hs = (__nv_bfloat16*)hs;
    a.eps = w->eps; a.next_eps = w->next_eps; a.o_eps = w->o_eps; a.status = status; a.budget = poll_budget();
    CUtensorMap mo, mu, md;
    if (!make_map(&mo, w->o_w, LAMPA_BF16, MD, MD, 64, MD, true) || !make_map(&mu, w->up_w, LAMPA_BF16, UP_HID, MD, 64, UP_CH, true) ||
        !make_map(&md, w->down_w, LAMPA_BF16, MD, UP_HID, 64, MD, true))
        return LAMPA_ERR_UNSUPPORTED;
    static std::atomic<uint64_t> ready{0};
    if (!allow_smem(ready, model_update_kernel, UP_SMEM)) return LAMPA_ERR_CUDA;
    ProfScope prof("model_update", (cudaStream_t)stream);
    const int64_t want = (n + UP_ROWS - 1) / UP_ROWS, most = (int64_t)sm_count() * 2;
    launch_chained(model_update_kernel, (unsigned)(want < most ? want : most), UP_THREADS, UP_SMEM, (cudaStream_t)stream, a, mo, mu, md);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

// Segment offsets of `rounds` copies of a packed batch behind one another: out[r * nseq + s] = r * n + cu[s], out[rounds * nseq] = rounds * n.
// An offset that leaves the batch, or falls, is moved to the highest one before it: the segments never overlap, so a bad event
// reaches neither into the events beside it nor into another copy's.  One CTA per copy.
constexpr int SEG_THREADS = 256;
static __global__ void __launch_bounds__(SEG_THREADS) model_segments_kernel(const int64_t* cu, int nseq, int64_t n, int64_t* out) {
    if (chain_wait()) return;
    __shared__ int64_t wtop[SEG_THREADS / 32];
    const int r = blockIdx.x;
    int64_t before = 0;
    for (int s0 = 0; s0 < nseq; s0 += SEG_THREADS) {
        const int s = s0 + threadIdx.x;
        const int64_t top = highest_offset<SEG_THREADS>(s < nseq ? cu[s] : 0, n, before, wtop);
        if (s < nseq) out[(int64_t)r * nseq + s] = (int64_t)r * n + top;
        __syncthreads();
    }
    if (r == gridDim.x - 1 && threadIdx.x == 0) out[(int64_t)gridDim.x * nseq] = (int64_t)gridDim.x * n;
}

extern "C" int lampa_repeat_segments(const int64_t* cu, int32_t nseq, int32_t rounds, int64_t n, int64_t* out, void* stream) {
    if (!cu || !out || nseq <= 0 || rounds <= 0) return LAMPA_ERR_ARG;
    launch_chained(model_segments_kernel, (unsigned)rounds, SEG_THREADS, 0, (cudaStream_t)stream, cu, nseq, n, out);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}
