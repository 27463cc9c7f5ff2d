// Per-chunk preparation of the gated-delta forward: one CTA of 4 warps per (chunk, head) turns
// 64 tokens of q, k, v, g, beta (and lambda) into the record {M, B^T, Q~, O_local, lambda_chunk}.
// Dense 64-wide contractions run on tensor cores (bf16 operands, fp32 accumulation); the
// 64x64 unit-lower-triangular inverse is an fp32 substitution on CUDA cores, as in the reference
// (models/hattention/solve_tril.py:54-61, 175-197), because bf16 there is where parity breaks.
#include "gdn.cuh"
#include "gdn_inv.cuh"
#include "gdn_load.cuh"
#include "profile.cuh"

namespace lampa {

// ---- plan: token / chunk / block offsets per sequence -------------------------------------------
// One CTA, a thread per sequence and a running sum over the CTA (one thread walking 64 sequences: 26 us, now 6.5).
constexpr int PLAN_THREADS = 256;
__global__ void __launch_bounds__(PLAN_THREADS) plan_kernel(PlanArgs p) {
    if (chain_wait()) return;
    __shared__ int2 wsum[PLAN_THREADS / 32];
    __shared__ int64_t wtop[PLAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t total = (int64_t)p.B * p.T;
    int c0 = 0, b0 = 0;                                     // totals of the sequences before this pass
    int64_t top0 = 0;                                       // largest offset inside the input before this pass
    if (threadIdx.x == 0) { p.chunk_off[0] = 0; p.block_off[0] = 0; }
    for (int s0 = 0; s0 < p.nseq; s0 += PLAN_THREADS) {
        const int s = s0 + threadIdx.x;
        int c = 0, b = 0;
        const int64_t t0 = s >= p.nseq ? 0 : p.cu ? p.cu[s] : (int64_t)s * p.T;
        // A sequence that begins before an earlier offset would take tokens of another one a second time: the chunks of
        // all sequences together could then outnumber the records of the workspace.
        const int64_t top = highest_offset<PLAN_THREADS>(t0, total, top0, wtop);
        if (s < p.nseq) {
            const int64_t t1 = p.cu ? p.cu[s + 1] : (int64_t)(s + 1) * p.T;
            p.tok_off[s] = t0;
            int64_t len = t1 - t0;
            if (len < 0 || t0 < 0 || t1 > total || t0 < top) { set_status(p.status, LAMPA_ERR_BOUNDS, 1, s); len = 0; }
            c = (int)((len + CHUNK - 1) / CHUNK);
            if (p.hier && c > 0 && ELL0 + ceil_log2_int(c) > p.L) set_status(p.status, LAMPA_ERR_LEVELS, 1, s);
            b = blocks_of(c);
            if (s == p.nseq - 1) p.tok_off[s + 1] = t0 + len;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int yc = __shfl_up_sync(0xffffffffu, c, o), yb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) { c += yc; b += yb; }
        }
        if (lane == 31) wsum[warp] = make_int2(c, b);
        __syncthreads();
        int tc = 0, tb = 0;
#pragma unroll
        for (int w = 0; w < PLAN_THREADS / 32; ++w) {
            if (w == warp) { c += c0 + tc; b += b0 + tb; }
            tc += wsum[w].x;
            tb += wsum[w].y;
        }
        if (s < p.nseq) { p.chunk_off[s + 1] = c; p.block_off[s + 1] = b; }
        c0 += tc;
        b0 += tb;
        __syncthreads();
    }
}

int launch_plan(const PlanArgs& p, cudaStream_t st) {
    ProfScope prof("gdn_plan", st);
    launch_chained(plan_kernel, 1, PLAN_THREADS, 0, st, p);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

// ---- shared-memory carve-up ---------------------------------------------------------------------
template <int KD, int VD>
struct PrepSmem {
    static constexpr int KP = KD + 8, VP = VD + 8, CP = CHUNK + 8;
    static constexpr int PA = CHUNK + 4;                         // fp32 pitch of the inverse's working tile (over AW and UH)
    static constexpr int Q = 0;                                  // bf16 [64][KP]   q (normalised); later W (rows are warp-private)
    static constexpr int K = Q + CHUNK * KP * 2;                 // bf16 [64][KP]   k (normalised)
    static constexpr int V = K + CHUNK * KP * 2;                 // bf16 [64][VP]   v
    static constexpr int AW = V + CHUNK * VP * 2;                // bf16 [64][CP]   Awb = (I + A0)^-1 diag(beta)
    static constexpr int UH = AW + CHUNK * CP * 2;               // bf16 [64][VP]   diag(e^{Glast-G}) U
    static constexpr int AFTER_UH = UH + CHUNK * VP * 2, AFTER_SA = AW + CHUNK * PA * 4;   // the fp32 tile covers AW and UH
    static constexpr int G = AFTER_UH > AFTER_SA ? AFTER_UH : AFTER_SA;   // fp32 [64] G, [64] beta, [64] e^G, [64] e^{Glast-G}, [64] e^{G(end of the 8-block)-G}
    static constexpr int LAM = G + 5 * CHUNK * 4;                // fp32 [64][7]: the levels inside the chunk, an odd pitch
    static constexpr int bytes(bool hier) { return LAM + (hier ? CHUNK * ELL0 * 4 : 0); }
};

// With beta folded into the columns of the inverse (Awb = (I + A0)^-1 diag(beta), Aub = Awb .* E):
//   W  = Awb K                    M   = e^{G_last} (I - K^T W)
//   U^ = diag(e^{G_last-G}) Aub V B^T = U^^T K
//   R  = tril(Q K^T) Awb          Q~  = s diag(e^G) (Q - R K)
//   O_local = s ((R .* E .* lambda[i][level(i,j)]) V)
// (s = scale and lambda = 1 for the plain rule; s = 1 for the hierarchical one).  These equal
// the definitions in gdn.cuh: every e^{G_last-G_tok} e^{G_tok} pair collapses to e^{G_last}.
// Half of a token's lambda row (levels half, half + 2, ...): NIT loads in flight, then the chunk's own levels go to
// shared memory and the others straight to the record's [level][token] table.
template <int NIT>
__device__ __forceinline__ void stage_lambda(const GdnArgs& a, size_t base, int half, bool valid, float* own, float* lamc) {
    float lv[NIT];
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int l = half + 2 * i;
        lv[i] = (valid && l < a.L) ? load_as_float(a.lam, base + l, a.lam_dt) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int l = half + 2 * i;
        if (l < ELL0) own[l] = lv[i];
        else if (l < ELL0 + a.LC) lamc[(l - ELL0) * CHUNK] = lv[i];
    }
}
// two accumulator tiles (16 x 16) as one A fragment of the next product
__device__ __forceinline__ void pack_a(uint32_t (&f)[4], const float (&c0)[4], const float (&c1)[4]) {
    f[0] = pack_bf16x2(c0[0], c0[1]);
    f[1] = pack_bf16x2(c0[2], c0[3]);
    f[2] = pack_bf16x2(c1[0], c1[1]);
    f[3] = pack_bf16x2(c1[2], c1[3]);
}

// Bound by the shared-memory pipe and issue slots at head dims up to 32 (69 and 58 % busy at K = 16, V = 32; 64 and 47 %
// at K = V = 32 with levels).  Every product is formed 16 columns at a time and products over the same fragments (K: KK^T
// and QK^T, Q~ and W; V: O_local and U^) share the pass: whole 64-wide accumulators held it at 96 registers and five CTAs
// per SM.  Four packed sequences of 12,001 to 90,001 tokens, 6 heads, K = 16, V = 32: 319 -> 246 us.
template <int KD, int VD, bool HIER>
__global__ void __launch_bounds__(128, KD == 64 ? 4 : 6) gdn_prep_kernel(GdnArgs a) {
    if (chain_wait()) return;
    using S = PrepSmem<KD, VD>;
    using R = Rec<KD, VD>;
    constexpr int KP = S::KP, VP = S::VP, CP = S::CP;
    extern __shared__ __align__(128) unsigned char smem[];
    __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(smem + S::Q);
    __nv_bfloat16* sW = sQ;
    __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(smem + S::K);
    __nv_bfloat16* sV = reinterpret_cast<__nv_bfloat16*>(smem + S::V);
    __nv_bfloat16* sAw = reinterpret_cast<__nv_bfloat16*>(smem + S::AW);
    __nv_bfloat16* sUh = reinterpret_cast<__nv_bfloat16*>(smem + S::UH);
    float* sG = reinterpret_cast<float*>(smem + S::G);
    float* sBeta = sG + CHUNK;
    float* sEG = sG + 2 * CHUNK;
    float* sEGl = sG + 3 * CHUNK;
    float* sCF = sG + 4 * CHUNK;
    float* sLam = reinterpret_cast<float*>(smem + S::LAM);

    // head is the fastest grid index: the H CTAs of one chunk run together and between them read
    // whole contiguous token rows of q, k, v (one head alone touches 128 B out of every H*128 B)
    const int h = blockIdx.x, c = blockIdx.y, H = a.H;
    ChunkLoc loc;
    if (!locate_chunk(a, c, loc)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gq = lane >> 2, tq = lane & 3;
    const int64_t t0 = loc.t0;
    const int len = loc.len;
    char* rec = a.rec + ((size_t)c * H + h) * a.rec_bytes;
    if (h == 0) check_out_perm(a, t0, len);

    // ---- stage 0: loads, l2norm, cumulative decay -------------------------------------------------
    // Every global load of the chunk is issued before any of them is consumed (one DRAM round trip
    // instead of four), and the rows of a chunk some 600 CTAs ahead are pulled into L2.
    {
        // two threads per row; at the 80-byte pitch of a 32-wide row the order 0, 1, 4, 5, 2, 3, 6, 7 puts the eight
        // 16-byte stores of a phase in different banks
        const int rl = tid >> 1, half = tid & 1;
        const int r = KD == 64 ? rl : (rl & ~6) | ((rl & 2) << 1) | ((rl & 4) >> 1);
        const bool valid = r < len;
        const size_t tok = (size_t)(t0 + r);
        const bool two_byte = a.qkv_dt != LAMPA_F32;
        uint4 rq[KD / 16], rk[KD / 16], rv[VD / 16];
        if (two_byte) {
            issue_half_row<KD>(a.q, (tok * H + h) * KD + half * (KD / 2), valid, rq);
            issue_half_row<KD>(a.k, (tok * H + h) * KD + half * (KD / 2), valid, rk);
            issue_half_row<VD>(a.v, (tok * H + h) * VD + half * (VD / 2), valid, rv);
        }
        float gv = 0.f, bv = 0.f;
        if (tid < len) {   // len <= 64: threads 0..len-1 carry g and beta of token tid
            gv = load_as_float(a.g, (size_t)(t0 + tid) * H + h, a.gb_dt);
            bv = load_as_float(a.beta, (size_t)(t0 + tid) * H + h, a.gb_dt);
        }
        if (HIER) {   // all of the row's loads in flight before the first store; the unrolled length follows L
            const size_t lam_base = (tok * H + h) * a.L;
            float* lamc = reinterpret_cast<float*>(rec + R::LAM_OFF) + r;
            if (a.L <= 18) stage_lambda<9>(a, lam_base, half, valid, sLam + r * ELL0, lamc);
            else if (a.L <= 24) stage_lambda<12>(a, lam_base, half, valid, sLam + r * ELL0, lamc);
            else stage_lambda<20>(a, lam_base, half, valid, sLam + r * ELL0, lamc);
        }
        if (h == 0) {   // L2 prefetch of the token rows (all heads) of a chunk ~80 chunks ahead
            ChunkLoc l2;
            if (locate_chunk(a, c + 80, l2) && r < l2.len) {
                const int eb = dtype_bytes(a.qkv_dt);
                const size_t rowq = (size_t)H * KD * eb, rowv = (size_t)H * VD * eb;
                const char* pq = (const char*)a.q + (size_t)(l2.t0 + r) * rowq;
                const char* pk = (const char*)a.k + (size_t)(l2.t0 + r) * rowq;
                const char* pv = (const char*)a.v + (size_t)(l2.t0 + r) * rowv;
                for (size_t off = (size_t)half * 128; off < rowq; off += 256) {
                    asm volatile("prefetch.global.L2 [%0];\n" :: "l"(pq + off));
                    asm volatile("prefetch.global.L2 [%0];\n" :: "l"(pk + off));
                }
                for (size_t off = (size_t)half * 128; off < rowv; off += 256)
                    asm volatile("prefetch.global.L2 [%0];\n" :: "l"(pv + off));
            }
        }
        float x[KD / 2];
        if (two_byte) convert_half_row<KD>(rq, a.qkv_dt, x);
        else load_half_row<KD>(a.q, a.qkv_dt, (tok * H + h) * KD + half * (KD / 2), valid, x);
        if (a.use_l2norm) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < KD / 2; ++i) ss += x[i] * x[i];
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            const float rn = rsqrtf(ss + 1e-6f);
#pragma unroll
            for (int i = 0; i < KD / 2; ++i) x[i] *= rn;
        }
        store_half_row_bf16<KD / 2>(sQ + r * KP + half * (KD / 2), x);
        if (two_byte) convert_half_row<KD>(rk, a.qkv_dt, x);
        else load_half_row<KD>(a.k, a.qkv_dt, (tok * H + h) * KD + half * (KD / 2), valid, x);
        if (a.use_l2norm) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < KD / 2; ++i) ss += x[i] * x[i];
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            const float rn = rsqrtf(ss + 1e-6f);
#pragma unroll
            for (int i = 0; i < KD / 2; ++i) x[i] *= rn;
        }
        store_half_row_bf16<KD / 2>(sK + r * KP + half * (KD / 2), x);
        if (a.qkv_dt == LAMPA_BF16) {   // v is used as it is: the raw 16-byte pieces go straight to shared memory
#pragma unroll
            for (int i = 0; i < VD / 16; ++i) reinterpret_cast<uint4*>(sV + r * VP + half * (VD / 2))[i] = rv[i];
        } else {
            float y[VD / 2];
            if (two_byte) convert_half_row<VD>(rv, a.qkv_dt, y);
            else load_half_row<VD>(a.v, a.qkv_dt, (tok * H + h) * VD + half * (VD / 2), valid, y);
            store_half_row_bf16<VD / 2>(sV + r * VP + half * (VD / 2), y);
        }

        if (tid < CHUNK) {
            float cs = gv;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float yy = __shfl_up_sync(0xffffffffu, cs, o);
                if (lane >= o) cs += yy;
            }
            if (tid == 31) sG[CHUNK - 1] = cs;      // one-float mailbox between the two warps
            sBeta[tid] = bv;
            asm volatile("bar.sync 1, 64;\n" ::: "memory");
            const float carry = (warp == 1) ? sG[CHUNK - 1] : 0.f;
            asm volatile("bar.sync 1, 64;\n" ::: "memory");
            sG[tid] = cs + carry;
        }
    }
    __syncthreads();
    if (tid < CHUNK) {
        const float Gi = sG[tid], Gl = sG[CHUNK - 1];
        sEG[tid] = __expf(Gi);
        sEGl[tid] = __expf(Gl - Gi);
        sCF[tid] = __expf(sG[tid | 7] - Gi);
    }
    const int m0 = warp * 16;
    uint32_t qk[4][4];                                       // tril(Q K^T) as A fragments
    // ---- stage 1: Awb = (I + A0)^-1 diag(beta), A0 = tril(diag(beta) K K^T, -1) ---------------------
    // Blockwise, as the reference's solve_tril does (models/hattention/solve_tril.py:221-276): warp w
    // forms rows 16w.. of A0 on the tensor cores and inverts its own 16x16 diagonal block by fp32
    // forward substitution (lane = column); the off-diagonal blocks follow as X_ba = -(X_bb A_ba) X_aa,
    // first inside the two 32x32 halves, then for the 32x32 corner, in place in one fp32 [64][68] tile
    // that lies over the Awb and U^ buffers (both written later).  These products keep fp32 accuracy
    // by splitting each operand into bf16 hi + lo and issuing hi*hi + lo*hi + hi*lo (the reference
    // asks for IEEE fp32 dots there).
    {
        constexpr int PA = S::PA;
        float* sA = reinterpret_cast<float*>(smem + S::AW);
        {
            uint32_t ak[KD / 16][4], aq[KD / 16][4];
#pragma unroll
            for (int k = 0; k < KD / 16; ++k) {
                load_a(ak[k], sK, KP, m0, 16 * k, lane);
                load_a(aq[k], sQ, KP, m0, 16 * k, lane);
            }
            const float b2[2] = {sBeta[m0 + gq], sBeta[m0 + gq + 8]};   // read before the stores below: they may alias for the compiler
#pragma unroll
            for (int np = 0; np < 4; ++np) {         // 16 columns at a time
                float acc[2][4], racc[2][4];
                zero_acc<2>(acc);
                zero_acc<2>(racc);
                if (np <= warp) {                    // tiles above the diagonal are never read
#pragma unroll
                    for (int k = 0; k < KD / 16; ++k) {
                        uint32_t b[4];
                        load_b(b, sK, KP, np * 16, 16 * k, lane);
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            mma16816(acc[x], ak[k], b[2 * x], b[2 * x + 1]);
                            mma16816(racc[x], aq[k], b[2 * x], b[2 * x + 1]);
                        }
                    }
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int hh = 0; hh < 2; ++hh) {
                            const int i = m0 + gq + hh * 8, j = np * 16 + x * 8 + 2 * tq;
                            const float bb = b2[hh];
                            *reinterpret_cast<float2*>(sA + i * PA + j) =
                                make_float2(i > j ? bb * acc[x][2 * hh] : 0.f, i > j + 1 ? bb * acc[x][2 * hh + 1] : 0.f);
                            if (np == warp) {        // only the warp's diagonal tile can hold i < j
                                if (i < j) racc[x][2 * hh] = 0.f;
                                if (i < j + 1) racc[x][2 * hh + 1] = 0.f;
                            }
                        }
                }
                pack_a(qk[np], racc[0], racc[1]);
            }
        }
        __syncwarp();
        tril_inverse_64<PA>(sA, warp, lane);
        {   // Awb = X diag(beta) as bf16, written over the front of the fp32 tile: the warp's own rows, up to the diagonal
            const int r = tid >> 1, half = tid & 1;
            uint32_t w[16];
#pragma unroll
            for (int p = 0; p < 2; ++p)
                if (2 * p + half <= warp) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {      // 16 columns per thread and step: the two halves are four bank groups apart
                        const float4 v = *reinterpret_cast<const float4*>(sA + r * PA + p * 32 + half * 16 + 4 * q);
                        const float4 b = *reinterpret_cast<const float4*>(sBeta + p * 32 + half * 16 + 4 * q);
                        w[8 * p + 2 * q] = pack_bf16x2(v.x * b.x, v.y * b.y);
                        w[8 * p + 2 * q + 1] = pack_bf16x2(v.z * b.z, v.w * b.w);
                    }
                }
            __syncthreads();
#pragma unroll
            for (int p = 0; p < 2; ++p)
                if (2 * p + half <= warp) {
                    uint4* d = reinterpret_cast<uint4*>(sAw + r * CP + p * 32 + half * 16);
                    d[0] = make_uint4(w[8 * p], w[8 * p + 1], w[8 * p + 2], w[8 * p + 3]);
                    d[1] = make_uint4(w[8 * p + 4], w[8 * p + 5], w[8 * p + 6], w[8 * p + 7]);
                }
        }
        __syncthreads();
    }
    const float osc = HIER ? 1.f : a.scale;
    // ---- per-warp part (rows m0..m0+15 of everything; nothing leaves the warp) --------------------
    {
        // R = tril(QK^T) Awb, 16 columns at a time, and Pm = R .* E .* lambda, both as A fragments.
        // level(i, j) = bit_length(i ^ j).  Off the diagonal 8x8 tile it depends on the tile only
        // (3 + bit_length(i/8 ^ j/8)): one lambda per (row, tile) serves both of the thread's columns.
        // The decay splits the same way: e^{G_i - G_end(tile)} per (row, tile) times the column's decay to the end of
        // its tile, both at most 1 - one exponential per row and tile instead of two per pair of elements.
        uint32_t ra[4][4], pa[4][4];
        const float gi2[2] = {sG[m0 + gq], sG[m0 + gq + 8]};
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            float racc[2][4];
            zero_acc<2>(racc);
#pragma unroll
            for (int kk = np; kk < 4; ++kk)              // Awb is lower-triangular too
                if (kk <= warp) {
                    uint32_t b[4];
                    load_b_t(b, sAw, CP, np * 16, kk * 16, lane);
                    mma16816(racc[0], qk[kk], b[0], b[1]);
                    mma16816(racc[1], qk[kk], b[2], b[3]);
                }
            pack_a(ra[np], racc[0], racc[1]);
            if (np <= warp) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int nt = 2 * np + x, j = nt * 8 + 2 * tq;
                    const float2 cf = *reinterpret_cast<const float2*>(sCF + j);
                    const float gend = sG[nt * 8 + 7];
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const int i = m0 + gq + hh * 8;
                        const int it = (m0 >> 3) + hh;                     // the row's 8x8 tile index (warp-uniform)
                        float p0 = 0.f, p1 = 0.f;
                        if (nt < it) {
                            p0 = __expf(gi2[hh] - gend);
                            if (HIER) p0 *= sLam[i * ELL0 + 3 + (32 - __clz(it ^ nt))];
                            p1 = p0 * cf.y;
                            p0 *= cf.x;
                        } else if (nt == it) {
                            const float2 gj = *reinterpret_cast<const float2*>(sG + j);
                            if (i >= j) p0 = __expf(gi2[hh] - gj.x);
                            if (i >= j + 1) p1 = __expf(gi2[hh] - gj.y);
                            if (HIER) {
                                p0 *= sLam[i * ELL0 + (32 - __clz(i ^ j))];
                                p1 *= sLam[i * ELL0 + (32 - __clz(i ^ (j + 1)))];
                            }
                        }
                        racc[x][2 * hh] *= p0;
                        racc[x][2 * hh + 1] *= p1;
                    }
                }
            }
            pack_a(pa[np], racc[0], racc[1]);
        }
        // Q~ = s e^G (Q - R K) and W = Awb K, 16 columns at a time over the same fragments of K.  W goes over this warp's
        // own rows of Q.
        __nv_bfloat16* gQ = reinterpret_cast<__nv_bfloat16*>(rec + R::QT_OFF);
        const float fq[2] = {osc * sEG[m0 + gq], osc * sEG[m0 + gq + 8]};
#pragma unroll
        for (int np = 0; np < KD / 16; ++np) {
            float acc[2][4], wacc[2][4];
            zero_acc<2>(acc);
            zero_acc<2>(wacc);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                if (kk <= warp) {
                    uint32_t af[4], b[4];
                    load_a(af, sAw, CP, m0, kk * 16, lane);
                    load_b_t(b, sK, KP, np * 16, kk * 16, lane);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        mma16816(acc[x], ra[kk], b[2 * x], b[2 * x + 1]);
                        mma16816(wacc[x], af, b[2 * x], b[2 * x + 1]);
                    }
                }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = m0 + gq + hh * 8, j = np * 16 + x * 8 + 2 * tq;
                    uint32_t* sq = reinterpret_cast<uint32_t*>(sQ + i * KP + j);   // read, then replaced, by this thread only
                    const float2 qv = unpack_bf16x2(*sq);
                    *sq = pack_bf16x2(wacc[x][2 * hh], wacc[x][2 * hh + 1]);
                    *reinterpret_cast<uint32_t*>(gQ + R::T::off(i, j)) =
                        pack_bf16x2(fq[hh] * (qv.x - acc[x][2 * hh]), fq[hh] * (qv.y - acc[x][2 * hh + 1]));
                }
        }
        // O_local = s Pm V and U^ = diag(e^{Glast-G}) (Awb .* E) V = (Awb diag(e^{Glast-G})) V, a column factor on the
        // A fragments in registers, over the same fragments of V
        __nv_bfloat16* gO = reinterpret_cast<__nv_bfloat16*>(rec + R::OL_OFF);
        uint32_t (&ua)[4][4] = ra;                           // R is used up
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
            if (kk <= warp) {
                load_a(ua[kk], sAw, CP, m0, kk * 16, lane);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 f = *reinterpret_cast<const float2*>(sEGl + kk * 16 + x * 8 + 2 * tq);
#pragma unroll
                    for (int y = 0; y < 2; ++y) {
                        const float2 w = unpack_bf16x2(ua[kk][2 * x + y]);
                        ua[kk][2 * x + y] = pack_bf16x2(w.x * f.x, w.y * f.y);
                    }
                }
            }
#pragma unroll
        for (int np = 0; np < VD / 16; ++np) {
            float acc[2][4], uacc[2][4];
            zero_acc<2>(acc);
            zero_acc<2>(uacc);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                if (kk <= warp) {
                    uint32_t b[4];
                    load_b_t(b, sV, VP, np * 16, kk * 16, lane);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        mma16816(acc[x], pa[kk], b[2 * x], b[2 * x + 1]);
                        mma16816(uacc[x], ua[kk], b[2 * x], b[2 * x + 1]);
                    }
                }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = m0 + gq + hh * 8, j = np * 16 + x * 8 + 2 * tq;
                    *reinterpret_cast<uint32_t*>(sUh + i * VP + j) = pack_bf16x2(uacc[x][2 * hh], uacc[x][2 * hh + 1]);
                    *reinterpret_cast<uint32_t*>(gO + R::TV::off(i, j)) = pack_bf16x2(osc * acc[x][2 * hh], osc * acc[x][2 * hh + 1]);
                }
        }
    }
    __syncthreads();

    // ---- stage 4: M[a][b] = e^{G_last} (delta_ab - sum_tok K[tok][a] W[tok][b]);  B^T = U^^T K -----
    // Both tiles are assembled in the record's layout in shared memory (over Awb and V, which are
    // dead by now) and leave as two bulk copies instead of 4-byte stores from every lane.
    __nv_bfloat16* stM = reinterpret_cast<__nv_bfloat16*>(smem + S::AW);
    __nv_bfloat16* stB = reinterpret_cast<__nv_bfloat16*>(smem + S::V);
    static_assert(R::M_BYTES <= CHUNK * CP * 2 && R::BT_BYTES <= CHUNK * VP * 2, "staging tiles must fit");
    if (m0 < KD) {
        float acc[KD / 8][4];
        zero_acc<KD / 8>(acc);
        warp_gemm<KD / 8, CHUNK, true, true>(acc, sK, KP, m0, sW, KP, 0, lane, CHUNK, KD);
        const float egl = sEG[CHUNK - 1];
#pragma unroll
        for (int nt = 0; nt < KD / 8; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = m0 + gq + hh * 8, j = nt * 8 + 2 * tq;
                const float m_0 = egl * (((i == j) ? 1.f : 0.f) - acc[nt][2 * hh]);
                const float m_1 = egl * (((i == j + 1) ? 1.f : 0.f) - acc[nt][2 * hh + 1]);
                *reinterpret_cast<uint32_t*>(stM + R::T::off(i, j)) = pack_bf16x2(m_0, m_1);
            }
    }
    const int v0 = KD <= 32 && VD <= 32 ? m0 - 32 : m0;      // two tiles of rows each: warps 0, 1 form M, warps 2, 3 form B^T
    if (v0 >= 0 && v0 < VD) {
        float acc[KD / 8][4];
        zero_acc<KD / 8>(acc);
        warp_gemm<KD / 8, CHUNK, true, true>(acc, sUh, VP, v0, sK, KP, 0, lane, CHUNK, KD);
#pragma unroll
        for (int nt = 0; nt < KD / 8; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = v0 + gq + hh * 8, j = nt * 8 + 2 * tq;
                *reinterpret_cast<uint32_t*>(stB + R::T::off(i, j)) = pack_bf16x2(acc[nt][2 * hh], acc[nt][2 * hh + 1]);
            }
    }
    fence_async_shared();
    __syncthreads();
    if (tid == 0) {
        bulk_s2g(rec + R::M_OFF, stM, R::M_BYTES);
        bulk_s2g(rec + R::BT_OFF, stB, R::BT_BYTES);
        bulk_commit();
        bulk_wait_read();
    }
}

template <int KD, int VD>
int launch_prep(const GdnArgs& a, bool hier, cudaStream_t st) {
    using S = PrepSmem<KD, VD>;
    const int smem = S::bytes(hier);
    dim3 grid(a.H, a.nc_max);
    cudaError_t e;
    ProfScope prof(hier ? "gdn_prep_hier" : "gdn_prep_plain", st);
    if (hier) {
        e = cudaFuncSetAttribute(gdn_prep_kernel<KD, VD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return LAMPA_ERR_CUDA;
        launch_chained(gdn_prep_kernel<KD, VD, true>, grid, 128, smem, st, a);
    } else {
        e = cudaFuncSetAttribute(gdn_prep_kernel<KD, VD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return LAMPA_ERR_CUDA;
        launch_chained(gdn_prep_kernel<KD, VD, false>, grid, 128, smem, st, a);
    }
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

template int launch_prep<64, 64>(const GdnArgs&, bool, cudaStream_t);
template int launch_prep<32, 32>(const GdnArgs&, bool, cudaStream_t);
template int launch_prep<16, 32>(const GdnArgs&, bool, cudaStream_t);

}  // namespace lampa
