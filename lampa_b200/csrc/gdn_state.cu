// Fenwick-state side of the hierarchical gated-delta rule: the token levels of the final state
// after a chunkwise forward, the ragged end of a prompt, and the single-token decode step.
//
// The state of one (batch row, head) is L matrices S_l [K][V] with counts[l] tokens each
// (models/hattention/recurrent.py:9-131).  Inserting token t first cascades (level l is merged
// into l + 1 while it is full, capacity 2^l), then applies the token's transition
// e^g (I - beta k k^T) to every level, then puts beta k v^T into level 0.  After T tokens level 0
// holds one token and level l >= 1 holds 2^(l-1) tokens exactly when bit l-1 of T - 1 is set.
#include "gdn.cuh"
#include "profile.cuh"
#include "split3.cuh"
#include "tmap.cuh"

#include <type_traits>

namespace lampa {

__device__ __forceinline__ float round_like(float x, int dt) {
    if (dt == LAMPA_BF16) return __bfloat162float(__float2bfloat16_rn(x));
    if (dt == LAMPA_F16) return __half2float(__float2half_rn(x));
    return x;
}

// Elements as they lie in memory, and what they stand for: the loads of a phase are all in flight before the first is looked at.
// From L2, past an L1 that may hold what an earlier kernel read there: the tail reads its inputs while the kernel in front
// of it still runs.
__device__ __forceinline__ uint32_t load_raw(const void* p, size_t i, int dt, bool live) {
    uint32_t u = 0u;
    if (live && dt == LAMPA_F32) u = __ldcg((const unsigned int*)p + i);
    if (live && dt != LAMPA_F32) u = __ldcg((const unsigned short*)p + i);
    return u;
}
__device__ __forceinline__ float raw_float(uint32_t u, int dt) {
    return dt == LAMPA_F32 ? __uint_as_float(u) : dt == LAMPA_BF16 ? __uint_as_float(u << 16) : __half2float(__ushort_as_half((unsigned short)u));
}
// eight consecutive 2-byte elements of a 16-byte aligned tensor
__device__ __forceinline__ uint4 load8_raw(const void* p, size_t i, bool live) {
    return live ? __ldcg(reinterpret_cast<const uint4*>((const uint16_t*)p + i)) : make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ void raw_floats(const uint4& u, int dt, float (&x)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 f = dt == LAMPA_BF16 ? unpack_bf16x2(w[e]) : __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
        x[2 * e] = f.x; x[2 * e + 1] = f.y;
    }
}

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// Eight consecutive elements as floats (zeros where `live` is false): 16-byte loads where the base allows them
__device__ __forceinline__ void load8_float(const void* p, size_t i, int dt, bool live, float (&x)[8]) {
    if (!live) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = 0.f;
    } else if (((uintptr_t)p & 15) != 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = raw_float(load_raw(p, i + e, dt, true), dt);
    } else if (dt == LAMPA_F32) {
        const float4 u = __ldcg(reinterpret_cast<const float4*>((const float*)p + i)), v = __ldcg(reinterpret_cast<const float4*>((const float*)p + i) + 1);
        x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    } else {
        raw_floats(load8_raw(p, i, true), dt, x);
    }
}

// -------------------------------------------------------------------------------------------------
// End of a sequence, in fp32: the token levels 0..6 after its last whole chunk (the recurrence over that
// chunk from an empty state, as the reference's postprocess_prefill_hstate_ does,
// models/hattention/kernel.py:377-466), then, for a prefill, the T mod 64 tokens behind it with all levels
// and their outputs (what the reference hands to its step function, kernel.py:470-560).
// Inside one chunk the cascade is fixed: after r tokens level l >= 1 holds 2^(l-1) tokens exactly when bit
// l-1 of r - 1 is set, the older ones higher up, and level 0 the last token.  Before the first token behind
// n0 chunks, the token levels and the trailing full chunk levels collapse into level 7 + tz(n0), after which
// the live chunk levels are the set bits of n0 and do not change any more ("slots", in bit order).
// Without a tail a ragged last chunk (cu_seqlens) is completed with null tokens (k = v = 0, beta = 0, g = 0).
// Also writes counts.
//
// This kernel is for a longer tail: it and the chunk in front of it in closed form instead of one token after the other.  With G the running sum of g and
// E_ij = e^{G_i - G_j} (j <= i), the states are independent linear recurrences with the same transitions:
//     T = (I + tril(diag(beta) K K^T .* E, -1))^-1 diag(beta)          R = (tril(Q K^T) .* E) T
//     a level that holds tokens j in J:   S = K^T diag(e^{Gl-G}) T[:, J] V[J]
//     a slot that enters with X:          X <- e^{Gl} X - K^T diag(e^{Gl-G}) T diag(e^G) K X
//     o_i = sum_j lambda[i, bit_length(i^j)] R_ij v_j + sum_slots lambda[i, slot] (e^{G_i} q_i X - (R diag(e^G) K X)_i)
// all of it at fp32 accuracy: the products on the tensor cores with every operand in three bf16 pieces (split3.cuh), the 16 x 16
// diagonal blocks of the inverse by substitution, and G summed in double, so that an exponent G_i - G_j is rounded once however long
// the sums are; E is __expf of it (two ulp and one more per unit of the exponent).  Error of the states against float64, prompts of 57
// to 121 tokens, 64 x 64 heads: 0.9e-7 with g around -2, 1.4e-7 around -0.08, 2.5e-7 around -0.004 (3.8e-7 in fp16); token by token
// 0.4e-7, 2.1e-7, 4.2e-7 to 7.5e-7.
// A CTA takes eight state columns of a (sequence, head) after the other, as many as leave one CTA to an SM (one set of eight while
// there are SMs for all); T and R do not depend on the column and are formed once by each CTA, two halves of it on the last
// chunk and the tail side by side.  A column's arithmetic is the same whichever CTA has it.
// A k, beta or e^g that is not finite enters as zero (g: as one), or the zeros above a diagonal times its row would reach outputs of
// tokens before it.  What the recurrence makes of it is filled in: with a k or beta the states that hold the token or
// older ones are NaN from then on, with a g those that hold older ones, and so are the outputs, which read them all.  (q, v and
// lambda reach only what they belong to.)
// 3,001 tokens, 8 heads, K = V = 64: 43 us token by token (0.3 - 0.4 us each) -> 33 us, 20 of which run beside the output
// pass (launch_chained): the call 95 -> 65 us.  What bounds it now is the chain of dependent phases, each a few thousand cycles for
// a few hundred products, and in them the fetching of code that a CTA passes through once (the first stall reason in ncu).  As fp32 multiply-adds it was bound by shared-memory loads (a 16-byte load of a warp returns 512 bytes, four
// cycles, for 16 multiply-adds of four) and took 34 us; one copy of the product that all phases call is slower (the call 68 us instead of 63).
// -------------------------------------------------------------------------------------------------
constexpr int TAIL_COLS = 8, TAIL_THREADS = 512, TAIL_GRP = 256, TAIL_BATCH = 4;      // states formed at a time
constexpr int TAIL_AP = CHUNK + 4, TAIL_XP = TAIL_BATCH * TAIL_COLS + 4;              // pitches of 64- and 32-wide rows

template <int KD>
struct TailSmem {                                            // offsets in floats
    static constexpr int KP = KD + 4;
    static constexpr int LOST = 2 * CHUNK + 3 * CHUNK;       // behind G (double), e^G, e^{Gl-G}, beta
    static constexpr int SCAL = LOST + 3 * CHUNK / 4;        // [3][64] bytes: whether a token's k, g or beta is not finite
    static constexpr int CH = CHUNK * KP + CHUNK * TAIL_AP + CHUNK * TAIL_COLS + SCAL;       // k, A -> T, v, scalars of one chunk
    static constexpr int K_ = 0, A_ = CHUNK * KP, V_ = A_ + CHUNK * TAIL_AP, S_ = V_ + CHUNK * TAIL_COLS;
    static constexpr int Z = CH;                             // [64][XP]
    static constexpr int B = Z + CHUNK * TAIL_XP;            // the tail's chunk
    static constexpr int Q = B + CH;                         // [64][KP]
    static constexpr int P = Q + CHUNK * KP;                 // [64][AP], then R
    static constexpr int OUT = P + CHUNK * TAIL_AP;          // [64][8]
    static constexpr int LAM = OUT + CHUNK * TAIL_COLS;      // [64][L], then the slab [KD][8][L], then [slabs][KD][8] all tokens of the last chunk
    // slots, K X, and what a batch of slots adds to the outputs, over the last chunk, which is done with by then
    static constexpr int X = 0, D = KD * TAIL_XP, Y = D + CHUNK * TAIL_XP;
    static_assert(Y + CHUNK * TAIL_XP <= CH, "slots must fit");
    static_assert(CH % 4 == 0 && Q % 4 == 0 && LAM % 4 == 0, "16-byte rows");
    __host__ __device__ static constexpr int sum(int L) { return LAM + (CHUNK * L + 3) / 4 * 4 + KD * TAIL_COLS * L; }
    __host__ __device__ static constexpr int floats(int L, int slabs) { return sum(L) + slabs * KD * TAIL_COLS; }
};

__device__ __forceinline__ void tail_meet(int grp) { asm volatile("bar.sync %0, %1;\n" :: "r"(grp + 1), "n"(TAIL_GRP) : "memory"); }

// In place: A (strictly lower triangular, fp32 [64][AP]) -> (I + A)^-1 diag(beta).  The 256 threads of a group.
__device__ __forceinline__ void tail_inverse(float* A, const float* beta, int t, int grp) {
    constexpr int AP = TAIL_AP;
    if (t < CHUNK) {                                         // diagonal blocks by substitution, a thread to a column
        const int m0 = t & ~15, cc = t & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float s0 = i == cc ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
            for (int q = 0; q < (i + 3) / 4; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(A + (m0 + i) * AP + m0 + 4 * q);
                const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (4 * q + u < i) { if (u & 1) s1 -= e[u] * x[4 * q + u]; else s0 -= e[u] * x[4 * q + u]; }
            }
            x[i] = s0 + s1;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 16; ++i) A[(m0 + i) * AP + m0 + cc] = x[i];
    }
    tail_meet(grp);
    // X_ba = -X_bb (A_ba X_aa) for blocks of W = 16, then 32; the inner product waits in the mirror image above the diagonal.  A warp
    // forms a tile of 16 x 8.
    auto corner = [&](auto width) {
        constexpr int W = decltype(width)::value, MT = W / 16, NT = W / 8;
        const int w = t >> 5, lane = t & 31, gq = lane >> 2, tq = lane & 3;
        const bool on = w < (32 / W) * MT * NT;              // (pair, row tile, column tile)
        const int p = w / (MT * NT), mt = (w / NT) % MT, n0 = (w % NT) * 8, a0 = 2 * W * p, b0 = a0 + W;
        auto product = [&](const float* left, const float* right, float* dst, float sign) {
            if (!on) return;
            float c[1][1][4] = {};
            const float* const l1[1] = {left};
            tile_product3<1, 1, false, false>(c, l1, AP, 16 * mt, right, AP, n0, 1, 0, W, lane);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
                *reinterpret_cast<float2*>(dst + (16 * mt + gq + 8 * hh) * AP + n0 + 2 * tq) = make_float2(sign * c[0][0][2 * hh], sign * c[0][0][2 * hh + 1]);
        };
        product(A + b0 * AP + a0, A + a0 * AP + a0, A + a0 * AP + b0, 1.f);
        tail_meet(grp);
        product(A + b0 * AP + b0, A + a0 * AP + b0, A + b0 * AP + a0, -1.f);
        tail_meet(grp);
        if (on)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) *reinterpret_cast<float2*>(A + (a0 + 16 * mt + gq + 8 * hh) * AP + b0 + n0 + 2 * tq) = make_float2(0.f, 0.f);
        tail_meet(grp);
    };
    corner(std::integral_constant<int, 16>{});
    corner(std::integral_constant<int, 32>{});
    for (int i = t; i < CHUNK * 16; i += TAIL_GRP) {
        float4* p = reinterpret_cast<float4*>(A + (i >> 4) * AP + 4 * (i & 15));
        const float4 b = *reinterpret_cast<const float4*>(beta + 4 * (i & 15));
        float4 v = *p;
        v.x *= b.x; v.y *= b.y; v.z *= b.z; v.w *= b.w;
        *p = v;
    }
    tail_meet(grp);
}

// ONE: one set of eight columns to a CTA, without the loop over more (code that a CTA passes through once is fetched once: 0.9 us).
template <int KD, int VD, bool ONE>
__global__ void __launch_bounds__(TAIL_THREADS) hgdn_tail_kernel(GdnArgs a, TailArgs ta) {
    const int slabs = ONE ? 1 : ta.slabs;
    // In a prefill the kernels in front let this one in early: until it waits it reads the call's inputs alone.
    if (!(ta.early && chain_seen(a.signal_word, a.signal)) && chain_wait()) return;
    using M = TailSmem<KD>;
    constexpr int KP = M::KP, AP = TAIL_AP, XP = TAIL_XP;
    extern __shared__ __align__(16) float sm[];
    const int seq = blockIdx.x, h = blockIdx.y, H = a.H, L = a.L;
    const int tid = threadIdx.x, lane = tid & 31, gq = lane >> 2, tq = lane & 3, grp = tid / TAIL_GRP, t = tid % TAIL_GRP;
    int v0 = blockIdx.z * slabs * TAIL_COLS;              // the first of the state columns that are being worked on
    const int nch = ta.n0;
    const int64_t tok0 = (int64_t)seq * a.fixed_stride;
    const int lvl0 = nch > 0 ? ELL0 + __ffs(nch) - 1 : -1;   // the slot that takes in the last chunk's tokens
    // tokens of the tail that are taken in: before token t > 0 levels 0..tz(t) move up one, which ends with the last level
    const int done = min(ta.tail, L < ELL0 ? 1 << (L - 1) : CHUNK);
    const size_t bh = (size_t)seq * H + h;
    float* st = ta.states + (bh * KD * VD + v0) * L;         // row k: VD * L floats further each
    // the chunk a thread group works on: the last whole one, or the tail
    float* ch = sm + (grp == 0 ? 0 : M::B);
    float *sK = ch + M::K_, *sA = ch + M::A_, *sV = ch + M::V_;
    double* sG = reinterpret_cast<double*>(ch + M::S_);
    float *sEg = ch + M::S_ + 2 * CHUNK, *sEl = sEg + CHUNK, *sBeta = sEl + CHUNK;
    float *sQ = sm + M::Q, *sP = sm + M::P, *sOut = sm + M::OUT, *sLam = sm + M::LAM, *slab = sLam + (CHUNK * L + 3) / 4 * 4;
    float *sZ = sm + M::Z, *sSum = sm + M::sum(L);

    // chunk levels the tail continues from: slot (tid / 8) % 4 of a batch, column tid % 8, rows tid / 32 + 16 i
    auto slot_level = [&](int s) {                           // level of slot s (bit order), or -1
        uint32_t rem = (uint32_t)nch;
        for (int i = 0; i < s; ++i) rem &= rem - 1;
        return rem ? ELL0 + __ffs(rem) - 1 : -1;
    };
    const int xs = (tid >> 3) & 3, xv = tid & 7, xk = tid >> 5;
    constexpr int XR = (KD + 15) / 16;
    float xr[XR];
    auto fetch_slots = [&](int s0) {
        const int l = slot_level(s0 + xs);
#pragma unroll
        for (int i = 0; i < XR; ++i) {
            const float* p = st + ((size_t)(xk + 16 * i) * VD + xv) * L;
            xr[i] = 0.f;
            if (l < 0) continue;
            if (l != lvl0) xr[i] = __ldcg(p + l);
            else for (int q = ELL0; q < l; ++q) xr[i] += __ldcg(p + q);
        }
    };
    // v of `len` tokens from t0 on, columns c0 .. c0 + 7, rows up to 64 null tokens; n threads
    auto stage_values = [&](float* d, int i, int n, int64_t t0, int len, int c0) {
        for (; i < CHUNK * TAIL_COLS; i += n) {
            const int r = i / TAIL_COLS;
            d[i] = raw_float(load_raw(a.v, ((size_t)(t0 + r) * H + h) * VD + c0 + i % TAIL_COLS, a.qkv_dt, r < len), a.qkv_dt);
        }
    };
    if (grp == 1 || nch > 0) {
        const bool tail = grp == 1;
        const int64_t t0 = tok0 + (int64_t)(tail ? nch : nch - 1) * CHUNK;
        const int len = tail ? done : CHUNK;
        // rows as the kernel uses them, rows up to 64 null tokens: eight elements per thread and step, KD / 8 threads per row; every
        // load is in flight before the first is used
        constexpr int PPR = KD / 8, NIT = (CHUNK * PPR + TAIL_GRP - 1) / TAIL_GRP, NV = CHUNK * TAIL_COLS / TAIL_GRP, NL = 4;
        const bool fast = a.qkv_dt != LAMPA_F32 && (((uintptr_t)a.k | (uintptr_t)a.q) & 15) == 0;
        uint4 kw[NIT], qw[NIT];
        uint32_t vv[NV], lv[NL];
        if (fast) {
#pragma unroll
            for (int it = 0; it < NIT; ++it) {
                const int p = t + it * TAIL_GRP, r = p / PPR;
                const size_t at = ((size_t)(t0 + r) * H + h) * KD + (p % PPR) * 8;
                kw[it] = load8_raw(a.k, at, r < len);
                qw[it] = load8_raw(a.q, at, r < len && tail);
            }
        }
        const uint32_t g0w = load_raw(a.g, (size_t)(t0 + 2 * t) * H + h, a.gb_dt, 2 * t < len);
        const uint32_t g1w = load_raw(a.g, (size_t)(t0 + 2 * t + 1) * H + h, a.gb_dt, 2 * t + 1 < len);
        const uint32_t btw = load_raw(a.beta, (size_t)(t0 + t) * H + h, a.gb_dt, t < len);
#pragma unroll
        for (int it = 0; it < NV; ++it) {
            const int p = t + it * TAIL_GRP, r = p / TAIL_COLS;
            vv[it] = load_raw(a.v, ((size_t)(t0 + r) * H + h) * VD + v0 + p % TAIL_COLS, a.qkv_dt, r < len);
        }
        const int nlam = tail ? len * L : 0;
        auto lam_load = [&](int p) { return load_raw(a.lam, ((size_t)(t0 + p / L) * H + h) * L + p % L, a.lam_dt, p < nlam); };
#pragma unroll
        for (int it = 0; it < NL; ++it) lv[it] = lam_load(t + it * TAIL_GRP);
        // e^g is zero far above -1e5; a g of minus infinity would make differences of G undefined
        auto decay = [&](uint32_t w, bool& bad) {
            const float g = raw_float(w, a.gb_dt);
            bad = !finite(__expf(g));
            return bad ? 0.f : g < -1e5f ? -1e5f : g;
        };
        unsigned char* bad = reinterpret_cast<unsigned char*>(ch + M::S_ + M::LOST);
        bool bad0, bad1;
        const float g0 = decay(g0w, bad0), g1 = decay(g1w, bad1), bt = raw_float(btw, a.gb_dt);
        if (t < CHUNK) {
            sBeta[t] = finite(bt) ? bt : 0.f;
            bad[2 * CHUNK + t] = !finite(bt);
        }
#pragma unroll
        for (int it = 0; it < NV; ++it) sV[t + it * TAIL_GRP] = raw_float(vv[it], a.qkv_dt);
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int p = t + it * TAIL_GRP, r = p / PPR, c = (p % PPR) * 8;
            if (p >= CHUNK * PPR) break;                     // whole warps
            float x[8], y[8];
            if (fast) {
                raw_floats(kw[it], a.qkv_dt, x);
                raw_floats(qw[it], a.qkv_dt, y);
            } else {
                const size_t at = ((size_t)(t0 + r) * H + h) * KD + c;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    x[e] = raw_float(load_raw(a.k, at + e, a.qkv_dt, r < len), a.qkv_dt);
                    y[e] = raw_float(load_raw(a.q, at + e, a.qkv_dt, r < len && tail), a.qkv_dt);
                }
            }
            float sk = 0.f, sq = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) { sk += x[e] * x[e]; sq += y[e] * y[e]; }
#pragma unroll
            for (int o = 1; o < PPR; o <<= 1) {
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
            }
            if (a.use_l2norm) {
                const float rk = rsqrtf(sk + 1e-6f), rq = rsqrtf(sq + 1e-6f);
#pragma unroll
                for (int e = 0; e < 8; ++e) { x[e] = round_like(x[e] * rk, a.qkv_dt); y[e] *= rq; }
            }
            bool any = false;
#pragma unroll
            for (int e = 0; e < 8; ++e) any |= !finite(x[e]);
            any = (__ballot_sync(0xffffffffu, any) >> (lane & ~(PPR - 1)) & ((1u << PPR) - 1u)) != 0;
            if (c == 0) bad[r] = any;
            if (any)
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = 0.f;
            float4* d = reinterpret_cast<float4*>(sK + r * KP + c);
            d[0] = make_float4(x[0], x[1], x[2], x[3]);
            d[1] = make_float4(x[4], x[5], x[6], x[7]);
            if (tail) {
                d = reinterpret_cast<float4*>(sQ + r * KP + c);
                d[0] = make_float4(y[0], y[1], y[2], y[3]);
                d[1] = make_float4(y[4], y[5], y[6], y[7]);
            }
        }
#pragma unroll
        for (int it = 0; it < NL; ++it)
            if (t + it * TAIL_GRP < nlam) sLam[t + it * TAIL_GRP] = raw_float(lv[it], a.lam_dt);
        for (int p = t + NL * TAIL_GRP; p < nlam; p += TAIL_GRP) sLam[p] = raw_float(lam_load(p), a.lam_dt);      // more than 16 levels
        if (t < 32) {
            double cs = (double)g0 + (double)g1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xffffffffu, cs, o);
                if (lane >= o) cs += u;
            }
            const double last = __shfl_sync(0xffffffffu, cs, 31);
            bad[CHUNK + 2 * t] = bad0; bad[CHUNK + 2 * t + 1] = bad1;
            sG[2 * t] = cs - (double)g1; sG[2 * t + 1] = cs;
            sEg[2 * t] = __expf((float)(cs - (double)g1)); sEg[2 * t + 1] = __expf((float)cs);
            sEl[2 * t] = __expf((float)(last - (cs - (double)g1))); sEl[2 * t + 1] = __expf((float)(last - cs));
        }
        tail_meet(grp);
        {   // A = tril(diag(beta) K K^T .* E, -1), P = tril(Q K^T .* E): warp = (16 rows, half of the column tiles up to the diagonal)
            const int mt = (t >> 5) & 3, half = t >> 7, cnt = mt + 1, n0 = 8 * half * cnt;
            float c[2][4][4];
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) { c[x][nt][0] = c[x][nt][1] = c[x][nt][2] = c[x][nt][3] = 0.f; }
            if (tail) {
                const float* const kq[2] = {sK, sQ};
                tile_product3<2, 4, false, true>(c, kq, KP, 16 * mt, sK, KP, n0, cnt, 0, KD, lane);
            } else {
                const float* const k1[1] = {sK};
                tile_product3<1, 4, false, true>(reinterpret_cast<float (&)[1][4][4]>(c), k1, KP, 16 * mt, sK, KP, n0, cnt, 0, KD, lane);
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                if (nt >= cnt) break;
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = 16 * mt + gq + 8 * hh, j = n0 + 8 * nt + 2 * tq;
                    const float f0 = j <= i ? __expf((float)(sG[i] - sG[j])) : 0.f, f1 = j + 1 <= i ? __expf((float)(sG[i] - sG[j + 1])) : 0.f;
                    const float bi = sBeta[i];
                    *reinterpret_cast<float2*>(sA + i * AP + j) = make_float2(j < i ? bi * c[0][nt][2 * hh] * f0 : 0.f, j + 1 < i ? bi * c[0][nt][2 * hh + 1] * f1 : 0.f);
                    if (tail) *reinterpret_cast<float2*>(sP + i * AP + j) = make_float2(c[1][nt][2 * hh] * f0, c[1][nt][2 * hh + 1] * f1);
                }
            }
            for (int u = 2 * cnt + half; u < 8; u += 2)      // nothing above the diagonal
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int at = (16 * mt + gq + 8 * hh) * AP + 8 * u + 2 * tq;
                    *reinterpret_cast<float2*>(sA + at) = make_float2(0.f, 0.f);
                    if (tail) *reinterpret_cast<float2*>(sP + at) = make_float2(0.f, 0.f);
                }
        }
        tail_meet(grp);
        tail_inverse(sA, sBeta, t, grp);
        for (int s = 0; s < slabs && !tail; ++s) {      // all tokens of the last chunk as one state: they join a slot
            const int w = t >> 5;
            if (s > 0) {
                tail_meet(grp);
                stage_values(sV, t, TAIL_GRP, t0, len, v0 + s * TAIL_COLS);
                tail_meet(grp);
            }
            if (w < 4) {
                float c[1][1][4] = {};
                const float* const T1[1] = {sA};
                tile_product3<1, 1, false, false>(c, T1, AP, 16 * w, sV, TAIL_COLS, 0, 1, 0, 16 * w + 16, lane);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = 16 * w + gq + 8 * hh;
                    *reinterpret_cast<float2*>(sZ + i * XP + 2 * tq) = make_float2(sEl[i] * c[0][0][2 * hh], sEl[i] * c[0][0][2 * hh + 1]);
                }
            }
            tail_meet(grp);
            if (w < KD / 16) {
                float c[1][1][4] = {};
                const float* const k1[1] = {sK};
                tile_product3<1, 1, true, false>(c, k1, KP, 16 * w, sZ, XP, 0, 1, 0, CHUNK, lane);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
                    *reinterpret_cast<float2*>(sSum + (s * KD + 16 * w + gq + 8 * hh) * TAIL_COLS + 2 * tq) = make_float2(c[0][0][2 * hh], c[0][0][2 * hh + 1]);
            }
        }
    }
    __syncthreads();
    // from here on everybody works on the tail's chunk
    const float* cs = sm + M::B;
    const float *cK = cs + M::K_, *cT = cs + M::A_, *cV = cs + M::V_, *cEg = cs + M::S_ + 2 * CHUNK, *cEl = cEg + CHUNK;
    const int row = tid >> 3, c8 = tid & 7;                  // row and column of what goes element by element
    const int warp = tid >> 5, mt = warp & 3, nt = warp >> 2;       // products: 16 rows, and eight columns: state nt of a batch
    // tokens of a chunk with a k or beta that is not finite, and with such a g, as masks; and what they take with them
    struct Lost { unsigned long long kb, g; };
    auto lost_tokens = [&](const float* c) {
        const unsigned char* f = reinterpret_cast<const unsigned char*>(c + M::S_ + M::LOST) + lane;
        Lost m;
        m.kb = (unsigned long long)__ballot_sync(0xffffffffu, f[32] | f[2 * CHUNK + 32]) << 32 | __ballot_sync(0xffffffffu, f[0] | f[2 * CHUNK]);
        m.g = (unsigned long long)__ballot_sync(0xffffffffu, f[CHUNK + 32]) << 32 | __ballot_sync(0xffffffffu, f[CHUNK]);
        return m;
    };
    const Lost lost = lost_tokens(cs), before = nch > 0 ? lost_tokens(sm) : Lost{0, 0};
    const unsigned long long lost_out = lost.kb | (nch > 0 ? lost.g : lost.g & ~1ull), lost_in = lost.kb | lost.g >> 1;
    const int first_lost = lost_out ? __ffsll((long long)lost_out) - 1 : CHUNK;      // outputs from this token on
    const int last_lost = lost_in ? 63 - __clzll((long long)lost_in) : -1;           // states with a token up to this one
    const bool lost_slots = (lost.kb | lost.g) != 0, lost_before = (before.kb | before.g >> 1) != 0;
    const float nan = __int_as_float(0x7fffffff);

    // states of the batch = e^{Gl} X (with X: the slots) -+ K^T Z, state nt to level l of the slab, or what is left of it (`gone`: nothing)
    auto kt_product = [&](const float* X, int l, bool gone) {
        if (mt >= KD / 16 || l < 0 || l >= L) return;        // (warp-uniform)
        float c[1][1][4] = {};
        const float* const k1[1] = {cK};
        tile_product3<1, 1, true, false>(c, k1, KP, 16 * mt, sZ, XP, 8 * nt, 1, 0, CHUNK, lane);
        const float egl = cEg[CHUNK - 1];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = 16 * mt + gq + 8 * (e >> 1), v = 2 * tq + (e & 1);
            slab[(k * TAIL_COLS + v) * L + l] = gone ? nan : X ? egl * X[k * XP + 8 * nt + v] - c[0][0][e] : c[0][0][e];
        }
    };

    {   // R = P T, both lower triangular: warp = (16 rows, column tiles nt and nt + 4)
        float c[2][1][1][4] = {};
        const float* const P1[1] = {sP};
#pragma unroll
        for (int x = 0; x < 2; ++x)
            if (nt + 4 * x <= 2 * mt + 1)
                tile_product3<1, 1, false, false>(c[x], P1, AP, 16 * mt, cT, AP, 8 * (nt + 4 * x), 1, (nt + 4 * x) / 2 * 16, 16 * mt + 16, lane);
        __syncthreads();
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
                *reinterpret_cast<float2*>(sP + (16 * mt + gq + 8 * hh) * AP + 8 * (nt + 4 * x) + 2 * tq) = make_float2(c[x][0][0][2 * hh], c[x][0][0][2 * hh + 1]);
        __syncthreads();
    }
    for (int s = 0; s < slabs; ++s) {                     // eight state columns at a time
        if (s > 0) {
            __syncthreads();                                 // the slab before is done with
            v0 += TAIL_COLS;
            st += TAIL_COLS * L;
            stage_values(const_cast<float*>(cV), tid, TAIL_THREADS, tok0 + (int64_t)nch * CHUNK, done, v0);
            __syncthreads();
        }
        for (int i = tid; i < KD * TAIL_COLS * L; i += TAIL_THREADS) slab[i] = 0.f;
        // outputs from the tail's own tokens: thread = (row, half of the columns, every fourth token); the tokens of level l >= 1 that
        // row i reads are the 2^(l-1) below the highest set bit they differ in
        {
            const int hf = (tid >> 2) & 1, jg = tid & 3;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < done) {
                for (int l = 0; l < ELL0 && l < L; ++l) {
                    if (l > 0 && !((row >> (l - 1)) & 1)) continue;
                    const int j0 = l == 0 ? row : (row >> l) << l, j1 = l == 0 ? row + 1 : j0 + (1 << (l - 1));
                    float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int j = j0 + jg; j < j1; j += 4) {
                        const float f = sP[row * AP + j];
                        const float4 v = *reinterpret_cast<const float4*>(cV + j * TAIL_COLS + 4 * hf);
                        u.x = fmaf(f, v.x, u.x); u.y = fmaf(f, v.y, u.y); u.z = fmaf(f, v.z, u.z); u.w = fmaf(f, v.w, u.w);
                    }
                    const float w = sLam[row * L + l];
                    o.x = fmaf(w, u.x, o.x); o.y = fmaf(w, u.y, o.y); o.z = fmaf(w, u.z, o.z); o.w = fmaf(w, u.w, o.w);
                }
            }
#pragma unroll
            for (int d = 1; d < 4; d <<= 1) {
                o.x += __shfl_xor_sync(0xffffffffu, o.x, d); o.y += __shfl_xor_sync(0xffffffffu, o.y, d);
                o.z += __shfl_xor_sync(0xffffffffu, o.z, d); o.w += __shfl_xor_sync(0xffffffffu, o.w, d);
            }
            if (jg == 0) *reinterpret_cast<float4*>(sOut + row * TAIL_COLS + 4 * hf) = o;
        }
        // token levels that hold tokens, four at a time: bit l of `held`
        const uint32_t held = (uint32_t)(done - 1) << 1 | 1u;
        auto nth = [](uint32_t m, int n) {                       // its n-th level, or -1
            for (int i = 0; i < n; ++i) m &= m - 1;
            return m ? __ffs(m) - 1 : -1;
        };
        for (int n0 = 0; n0 < __popc(held); n0 += TAIL_BATCH) {
            const int l = nth(held, n0 + nt);
            const int j0 = l < 0 ? 0 : l == 0 ? done - 1 : ((done - 1) >> l) << l, j1 = l < 0 ? 0 : l == 0 ? done : j0 + (1 << (l - 1));
            float c[1][1][4] = {};
            const float* const T1[1] = {cT};
            tile_product3<1, 1, false, false>(c, T1, AP, 16 * mt, cV, TAIL_COLS, 0, 1, j0 & ~15, min(16 * mt + 16, (j1 + 15) & ~15), lane, j0, j1);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = 16 * mt + gq + 8 * hh;
                *reinterpret_cast<float2*>(sZ + i * XP + 8 * nt + 2 * tq) = make_float2(cEl[i] * c[0][0][2 * hh], cEl[i] * c[0][0][2 * hh + 1]);
            }
            __syncthreads();
            kt_product(nullptr, l, j0 <= last_lost);
            __syncthreads();
        }
        if (s == 0 && ta.early) (void)chain_wait();        // the chunk levels are there
        float *sX = sm + M::X, *sD = sm + M::D, *sY = sm + M::Y;
        const int nslot = __popc((uint32_t)nch);
        for (int s0 = 0; s0 < nslot; s0 += TAIL_BATCH) {
            fetch_slots(s0);
#pragma unroll
            for (int i = 0; i < XR; ++i)
                sX[(xk + 16 * i) * XP + 8 * xs + xv] = xr[i] + (s0 + xs != 0 ? 0.f : lost_before ? nan : sSum[(s * KD + xk + 16 * i) * TAIL_COLS + xv]);
            __syncthreads();
            const int l = slot_level(s0 + nt);
            float y[4];
            {   // K X and Q X
                float c[2][1][4] = {};
                const float* const kq[2] = {cK, sQ};
                tile_product3<2, 1, false, false>(c, kq, KP, 16 * mt, sX, XP, 8 * nt, 1, 0, KD, lane);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = 16 * mt + gq + 8 * hh;
                    *reinterpret_cast<float2*>(sD + i * XP + 8 * nt + 2 * tq) = make_float2(cEg[i] * c[0][0][2 * hh], cEg[i] * c[0][0][2 * hh + 1]);
                    y[2 * hh] = cEg[i] * c[1][0][2 * hh];
                    y[2 * hh + 1] = cEg[i] * c[1][0][2 * hh + 1];
                }
            }
            __syncthreads();
            {   // T and R times that
                float c[2][1][4] = {};
                const float* const tr[2] = {cT, sP};
                tile_product3<2, 1, false, false>(c, tr, AP, 16 * mt, sD, XP, 8 * nt, 1, 0, 16 * mt + 16, lane);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = 16 * mt + gq + 8 * hh;
                    const float w = l >= 0 && i < done ? sLam[i * L + l] : 0.f;
                    *reinterpret_cast<float2*>(sZ + i * XP + 8 * nt + 2 * tq) = make_float2(cEl[i] * c[0][0][2 * hh], cEl[i] * c[0][0][2 * hh + 1]);
                    *reinterpret_cast<float2*>(sY + i * XP + 8 * nt + 2 * tq) = make_float2(w * (y[2 * hh] - c[1][0][2 * hh]), w * (y[2 * hh + 1] - c[1][0][2 * hh + 1]));
                }
            }
            __syncthreads();
            {
                const float* p = sY + row * XP + c8;         // the slots of the batch
                sOut[row * TAIL_COLS + c8] += (p[0] + p[8]) + (p[16] + p[24]);
            }
            kt_product(sX, l, lost_slots);
            __syncthreads();
        }
        const int64_t t0 = tok0 + (int64_t)nch * CHUNK;
        for (int i = tid; i < done * TAIL_COLS; i += TAIL_THREADS)
            store_from_float(a.o, ((size_t)(t0 + i / TAIL_COLS) * H + h) * VD + v0 + i % TAIL_COLS, i / TAIL_COLS < first_lost ? sOut[i] : nan, a.qkv_dt);
        if (((uintptr_t)ta.states & 15) == 0) {              // every level: the slab goes out as bulk copies of 8 columns x L
            fence_async_shared();
            __syncthreads();
            if (tid < KD) {
                bulk_s2g(st + (size_t)tid * VD * L, slab + tid * TAIL_COLS * L, TAIL_COLS * L * 4);
                bulk_commit();
                bulk_wait_read();
            }
        } else {
            __syncthreads();
            for (int i = tid; i < KD * TAIL_COLS * L; i += TAIL_THREADS) {
                const int k = i / (TAIL_COLS * L);
                st[(size_t)k * VD * L + (i - k * TAIL_COLS * L)] = slab[i];
            }
        }
    }
    if (done < ta.tail && tid == 0 && h == 0 && blockIdx.z == 0) set_status(a.status, LAMPA_ERR_LEVELS, 31, seq);
    if (h == 0 && blockIdx.z == 0 && tid == 0 && (!ta.one_count || seq == 0)) {
        const int64_t n = (int64_t)nch * CHUNK + done;     // tokens held
        int32_t* cn = ta.counts + (size_t)seq * L;
        int64_t rem = n > 0 ? n - 1 : 0;
        for (int l = L - 1; l >= 1; --l) {
            const int64_t cap = l - 1 < 40 ? (int64_t)1 << (l - 1) : (int64_t)1 << 40;
            const bool held = n > 0 && rem >= cap;
            cn[l] = held ? (int32_t)cap : 0;
            if (held) rem -= cap;
        }
        cn[0] = n > 0 ? 1 : 0;
        if (seq == 0 && ta.arrivals) *ta.arrivals = 0;
        if (ta.early) *a.signal_word = 0;                  // behind the wait
        if (rem != 0) set_status(a.status, LAMPA_ERR_LEVELS, 30, seq);
    }
}

// -------------------------------------------------------------------------------------------------
// The same token by token, for what the closed form is not faster at (launch_hgdn_tail).
// Before token t > 0 of a chunk, levels 0..tz(t) collapse into level tz(t) + 1 (tz = trailing zeros); the live chunk levels sit
// in HS register slots, in bit order.
//
// State columns are independent, so a half-warp owns one: lane kl has rows kl, kl + 16, ... of every
// level in registers, a level's k^T S is K / 16 FMAs and four shuffles, and the levels of a token
// are independent chains that hide each other's latency.  What bounds it is that chain, 0.3 us per
// token of the last whole chunk and 0.4 us per token behind it (8 heads, K = V = 64: 19 us at 2944
// tokens, 47 us at 3001); with one CTA per (sequence, head) and a launch per tail token (61 us for the
// token levels and 27 us per tail token) a 3001-token prompt spent 1.7 of its 1.9 ms on the device here.
// -------------------------------------------------------------------------------------------------
constexpr int STEPS_THREADS = 128;

template <int N>
__device__ __forceinline__ void half_warp_sum(float (&x)[N]) {
#pragma unroll
    for (int o = 1; o < 16; o <<= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] += __shfl_xor_sync(0xffffffffu, x[i], o);
}

// The same for many values: a butterfly that halves the number of values a lane carries at every step (15 shuffles for 16
// values instead of 64), after which lane i of the half-warp has the sum of value i, and one shuffle hands each sum to all.
template <int N>
__device__ __forceinline__ void half_warp_sum_many(float (&x)[N], int lane) {
#pragma unroll
    for (int g = 0; g < N; g += 16) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = g + i < N ? x[g + i < N ? g + i : 0] : 0.f;
#pragma unroll
        for (int h = 8; h > 0; h >>= 1) {
            const bool up = lane & h;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const float give = up ? v[i] : v[i + h];
                v[i] = (up ? v[i + h] : v[i]) + __shfl_xor_sync(0xffffffffu, give, h);
            }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (g + i < N) x[g + i < N ? g + i : 0] = __shfl_sync(0xffffffffu, v[0], (lane & 16) | i);
    }
}

template <int KD, int VD, int HS>
__global__ void __launch_bounds__(STEPS_THREADS) hgdn_tail_steps_kernel(GdnArgs a, TailArgs ta) {
    if (!(ta.early && chain_seen(a.signal_word, a.signal)) && chain_wait()) return;      // see above: only the inputs are read before the wait
    constexpr int KI = KD / 16;
    extern __shared__ __align__(16) float tail_smem[];
    float* sK = tail_smem;                       // [64][KD], normalised
    float* sQ = sK + CHUNK * KD;                 // [64][KD], normalised (tail only)
    float* sV = sQ + CHUNK * KD;                 // [64][8]
    float* sEg = sV + CHUNK * TAIL_COLS;         // [64]
    float* sBeta = sEg + CHUNK;                  // [64]
    float* sLam = sBeta + CHUNK;                 // [64][L] (tail only)
    float* sOut = sLam + CHUNK * a.L;            // [63][8][17] terms of the outputs (tail only)
    const int seq = blockIdx.x, h = blockIdx.y, H = a.H, L = a.L;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col = 2 * warp + (lane >> 4), kl = lane & 15;
    const int v0 = blockIdx.z * TAIL_COLS, vv = v0 + col;
    int nch = ta.n0;
    int64_t tok0 = (int64_t)seq * a.fixed_stride, tok_end = 0;
    if (ta.n0 < 0) {
        const SeqLoc sq = locate_seq(a, seq);
        nch = sq.nch; tok0 = sq.tok0; tok_end = sq.tok_end;
    }

    auto input = [](const void* p, size_t i, int dt) { return raw_float(load_raw(p, i, dt, true), dt); };
    // rows [t0, t0 + len) of the inputs as the kernel uses them; rows up to 64 become null tokens.  Eight elements per
    // thread and step, K / 8 threads per row, every load in flight before the first is used.
    auto stage = [&](int64_t t0, int len, bool tail) {
        constexpr int PPR = KD / 8, NIT = CHUNK * PPR / STEPS_THREADS;
        float x[NIT][8], y[NIT][8];
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int p = tid + it * STEPS_THREADS, r = p / PPR, c = (p % PPR) * 8;
            const size_t at = ((size_t)(t0 + r) * H + h) * KD + c;
            load8_float(a.k, at, a.qkv_dt, r < len, x[it]);
            load8_float(a.q, at, a.qkv_dt, r < len && tail, y[it]);
        }
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int p = tid + it * STEPS_THREADS, r = p / PPR, c = (p % PPR) * 8;
            float sk = 0.f, sq = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) { sk += x[it][e] * x[it][e]; sq += y[it][e] * y[it][e]; }
#pragma unroll
            for (int o = 1; o < PPR; o <<= 1) {
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
            }
            const float rk = rsqrtf(sk + 1e-6f), rq = rsqrtf(sq + 1e-6f);
            if (a.use_l2norm) {
#pragma unroll
                for (int e = 0; e < 8; ++e) { x[it][e] = round_like(x[it][e] * rk, a.qkv_dt); y[it][e] *= rq; }
            }
            float4* d = reinterpret_cast<float4*>(sK + r * KD + c);
            d[0] = make_float4(x[it][0], x[it][1], x[it][2], x[it][3]);
            d[1] = make_float4(x[it][4], x[it][5], x[it][6], x[it][7]);
            if (tail) {
                d = reinterpret_cast<float4*>(sQ + r * KD + c);
                d[0] = make_float4(y[it][0], y[it][1], y[it][2], y[it][3]);
                d[1] = make_float4(y[it][4], y[it][5], y[it][6], y[it][7]);
            }
        }
#pragma unroll
        for (int i = tid; i < CHUNK * TAIL_COLS; i += STEPS_THREADS) {
            const int r = i / TAIL_COLS, c = i - r * TAIL_COLS;
            sV[i] = r < len ? input(a.v, ((size_t)(t0 + r) * H + h) * VD + v0 + c, a.qkv_dt) : 0.f;
        }
        if (tid < CHUNK) {
            sEg[tid] = tid < len ? __expf(input(a.g, (size_t)(t0 + tid) * H + h, a.gb_dt)) : 1.f;
            sBeta[tid] = tid < len ? input(a.beta, (size_t)(t0 + tid) * H + h, a.gb_dt) : 0.f;
        }
        if (tail) {                             // two threads per token, up to twenty levels each
            const int r = tid >> 1;
            if (r < len) {
                float w[20];
#pragma unroll
                for (int i = 0; i < 20; ++i) w[i] = (tid & 1) + 2 * i < L ? input(a.lam, ((size_t)(t0 + r) * H + h) * L + (tid & 1) + 2 * i, a.lam_dt) : 0.f;
#pragma unroll
                for (int i = 0; i < 20; ++i)
                    if ((tid & 1) + 2 * i < L) sLam[r * L + (tid & 1) + 2 * i] = w[i];
            }
        }
        __syncthreads();
    };

    float S[ELL0][KI];
#pragma unroll
    for (int l = 0; l < ELL0; ++l)
#pragma unroll
        for (int i = 0; i < KI; ++i) S[l][i] = 0.f;
    auto cascade_low = [&](int tz) {
#pragma unroll
        for (int j = 0; j < ELL0 - 1; ++j)
            if (j <= tz) {
#pragma unroll
                for (int i = 0; i < KI; ++i) { S[j + 1][i] += S[j][i]; S[j][i] = 0.f; }
            }
    };

    float* st = ta.states + ((((size_t)seq * H + h) * KD + kl) * VD + vv) * L;     // row kl; row kl + 16 i is i * row16 further
    const size_t row16 = (size_t)16 * VD * L;
    // chunk levels the tail continues from
    float X[HS][KI];
    int lvl[HS];
    {
        uint32_t rem = (uint32_t)nch;
#pragma unroll
        for (int s = 0; s < HS; ++s) {
            lvl[s] = rem ? ELL0 + __ffs(rem) - 1 : -1;
            rem &= rem - 1;
        }
    }
    const bool room = nch == 0 || lvl[0] < L;    // the first cascade must not leave the last level
    if (nch > 0) {
        const int64_t t0 = tok0 + (int64_t)(nch - 1) * CHUNK;
        stage(t0, ta.n0 >= 0 ? CHUNK : (int)min((int64_t)CHUNK, tok_end - t0), false);
        // After a whole chunk level l >= 1 holds tokens 64 - 2^l .. 63 - 2^(l-1), carried through the rest: one running
        // state from its first token on, so that before token 32 there is one state to advance and six only at the end.
        auto advance = [&](auto first, int t0, int t1) {         // levels first .. 6 have started
            constexpr int F = decltype(first)::value, NLV = ELL0 - F;
            for (int t = t0; t < t1; ++t) {
                const float eg = sEg[t], bt = sBeta[t], bv = bt * sV[t * TAIL_COLS + col];
                float kr[KI], ek[KI], dot[NLV];
#pragma unroll
                for (int i = 0; i < KI; ++i) { kr[i] = sK[t * KD + kl + 16 * i]; ek[i] = -eg * bt * kr[i]; }
                const bool collect = t < CHUNK - (1 << (F - 1)); // the youngest of these levels is still taking tokens in
#pragma unroll
                for (int l = 0; l < NLV; ++l) {
                    dot[l] = 0.f;
#pragma unroll
                    for (int i = 0; i < KI; ++i) {
                        dot[l] += kr[i] * S[F + l][i];
                        S[F + l][i] *= eg;                       // everything but the sum's term, before the sum is there
                        if (l == 0 && collect) S[F][i] += kr[i] * bv;
                    }
                }
                half_warp_sum(dot);
#pragma unroll
                for (int l = 0; l < NLV; ++l)
#pragma unroll
                    for (int i = 0; i < KI; ++i) S[F + l][i] = fmaf(ek[i], dot[l], S[F + l][i]);
            }
        };
        advance(std::integral_constant<int, 6>{}, 0, 32);
        advance(std::integral_constant<int, 5>{}, 32, 48);
        advance(std::integral_constant<int, 4>{}, 48, 56);
        advance(std::integral_constant<int, 3>{}, 56, 60);
        advance(std::integral_constant<int, 2>{}, 60, 62);
        advance(std::integral_constant<int, 1>{}, 62, 64);
#pragma unroll
        for (int i = 0; i < KI; ++i) S[0][i] = sK[63 * KD + kl + 16 * i] * (sBeta[63] * sV[63 * TAIL_COLS + col]);
    }

    if (ta.early) (void)chain_wait();            // the chunk levels are there
#pragma unroll
    for (int s = 0; s < HS; ++s)
#pragma unroll
        for (int i = 0; i < KI; ++i) X[s][i] = ta.tail > 0 && room && lvl[s] >= 0 && s > 0 ? st[i * row16 + lvl[s]] : 0.f;
    if (ta.tail > 0 && room && nch > 0) {
#pragma unroll
        for (int i = 0; i < KI; ++i)
            for (int l = ELL0; l < lvl[0]; ++l) X[0][i] += st[i * row16 + l];
    }

    int done = 0;                                // tail tokens taken in
    if (ta.tail > 0) {
        if (room) {
            if (nch > 0) {
#pragma unroll
                for (int i = 0; i < KI; ++i)
#pragma unroll
                    for (int l = 0; l < ELL0; ++l) { X[0][i] += S[l][i]; S[l][i] = 0.f; }
            }
            __syncthreads();                               // the last chunk's rows have been read
            const int64_t t0 = tok0 + (int64_t)nch * CHUNK;
            stage(t0, ta.tail, true);
            // A token's output is a sum over the half-warp too, but nothing in the recurrence waits for it: the lanes leave
            // their terms in shared memory and all tokens are summed behind the loop.  The next token's rows are fetched
            // while this one's sums are under way.
            float kn[KI], qn[KI];
#pragma unroll
            for (int i = 0; i < KI; ++i) { kn[i] = sK[kl + 16 * i]; qn[i] = sQ[kl + 16 * i]; }
            for (int t = 0; t < ta.tail; ++t) {
                if (t > 0) {
                    const int tz = __ffs(t) - 1;
                    if (tz + 1 >= L) break;
                    cascade_low(tz);
                }
                const float eg = sEg[t], bt = sBeta[t];
                float kr[KI], ek[KI], qr[KI], dot[ELL0 - 1 + HS], acc[KI];
                const int tn = min(t + 1, CHUNK - 1);
#pragma unroll
                for (int i = 0; i < KI; ++i) {
                    kr[i] = kn[i]; qr[i] = qn[i]; acc[i] = 0.f; ek[i] = -eg * bt * kr[i];
                    kn[i] = sK[tn * KD + kl + 16 * i]; qn[i] = sQ[tn * KD + kl + 16 * i];
                }
#pragma unroll
                for (int l = 0; l < ELL0 - 1 + HS; ++l) {
                    dot[l] = 0.f;
#pragma unroll
                    for (int i = 0; i < KI; ++i) {
                        float& x = l < ELL0 - 1 ? S[l < ELL0 - 1 ? l + 1 : 0][i] : X[l < ELL0 - 1 ? 0 : l - ELL0 + 1][i];
                        dot[l] += kr[i] * x;
                        x *= eg;                                 // everything but the sum's term, before the sum is there
                    }
                }
                const float* lam = sLam + t * L;
                float lw[ELL0 + HS];
#pragma unroll
                for (int l = 0; l < ELL0; ++l) lw[l] = l < L ? lam[l] : 0.f;
#pragma unroll
                for (int s = 0; s < HS; ++s) lw[ELL0 + s] = lvl[s] >= 0 ? lam[lvl[s]] : 0.f;
                const float bv = bt * sV[t * TAIL_COLS + col];
                half_warp_sum_many(dot, lane);
#pragma unroll
                for (int l = 0; l < ELL0 - 1 + HS; ++l)
#pragma unroll
                    for (int i = 0; i < KI; ++i) {
                        float& x = l < ELL0 - 1 ? S[l < ELL0 - 1 ? l + 1 : 0][i] : X[l < ELL0 - 1 ? 0 : l - ELL0 + 1][i];
                        x = fmaf(ek[i], dot[l], x);
                        acc[i] = fmaf(lw[l + 1], x, acc[i]);
                    }
                float out = 0.f;
#pragma unroll
                for (int i = 0; i < KI; ++i) {
                    S[0][i] = kr[i] * bv;
                    out += qr[i] * (acc[i] + lw[0] * S[0][i]);
                }
                sOut[(t * TAIL_COLS + col) * 17 + kl] = out;
                done = t + 1;
            }
            __syncthreads();
            for (int i = tid; i < done * TAIL_COLS; i += STEPS_THREADS) {
                float out = 0.f;
#pragma unroll
                for (int e = 0; e < 16; ++e) out += sOut[i * 17 + e];
                store_from_float(a.o, ((size_t)(t0 + i / TAIL_COLS) * H + h) * VD + v0 + i % TAIL_COLS, out, a.qkv_dt);
            }
        }
        if (done < ta.tail && tid == 0 && h == 0 && blockIdx.z == 0) set_status(a.status, LAMPA_ERR_LEVELS, 31, seq);
    }

    if (done > 0 && ((uintptr_t)ta.states & 15) == 0) {      // every level: the slab goes out as bulk copies of 8 columns x L
        __syncthreads();
        float* slab = tail_smem;                             // [KD][8][L] over everything staged
#pragma unroll
        for (int i = 0; i < KI; ++i) {
            float* d = slab + ((kl + 16 * i) * TAIL_COLS + col) * L;
#pragma unroll
            for (int l = 0; l < ELL0; ++l)
                if (l < L) d[l] = S[l][i];
            for (int l = ELL0; l < L; ++l) d[l] = 0.f;
#pragma unroll
            for (int s = 0; s < HS; ++s)
                if (lvl[s] >= 0) d[lvl[s]] = X[s][i];
        }
        fence_async_shared();
        __syncthreads();
        if (tid < KD) {
            bulk_s2g(ta.states + ((((size_t)seq * H + h) * KD + tid) * VD + v0) * L, slab + tid * TAIL_COLS * L, TAIL_COLS * L * 4);
            bulk_commit();
            bulk_wait_read();
        }
    } else {
#pragma unroll
        for (int i = 0; i < KI; ++i) {
#pragma unroll
            for (int l = 0; l < ELL0; ++l)
                if (l < L) st[i * row16 + l] = S[l][i];      // with a refused tail: the state after the whole chunks
            if (done > 0)
                for (int l = ELL0; l < L; ++l) {
                    float x = 0.f;
#pragma unroll
                    for (int s = 0; s < HS; ++s)
                        if (lvl[s] == l) x = X[s][i];
                    st[i * row16 + l] = x;
                }
        }
    }
    if (h == 0 && blockIdx.z == 0 && tid == 0 && (ta.n0 < 0 || !ta.one_count || seq == 0)) {
        const int64_t n = (int64_t)nch * CHUNK + done;     // tokens held
        int32_t* cn = ta.counts + (size_t)seq * L;
        int64_t rem = n > 0 ? n - 1 : 0;
        for (int l = L - 1; l >= 1; --l) {
            const int64_t cap = l - 1 < 40 ? (int64_t)1 << (l - 1) : (int64_t)1 << 40;
            const bool held = n > 0 && rem >= cap;
            cn[l] = held ? (int32_t)cap : 0;
            if (held) rem -= cap;
        }
        cn[0] = n > 0 ? 1 : 0;
        if (seq == 0 && ta.arrivals) *ta.arrivals = 0;
        if (ta.early) *a.signal_word = 0;                  // behind the wait
        if (rem != 0) set_status(a.status, LAMPA_ERR_LEVELS, 30, seq);
    }
}

// Which form takes a tail follows from the tail alone (and from L, where a level is missing), because the two do not round alike: a
// prompt's state and outputs are the same bits alone and in a batch.  The steps' time grows with the tail, the closed form's does not,
// and both begin beside the output pass.  Whole calls in us, steps against closed form, 8 heads of 64: 704 tokens and 16, 24 and 63 behind
// them 56 and 56, 59 and 56, 74 and 57; 2,944 tokens 71 and 65, 75 and 65, 97 and 67; 8 behind them 53 and 56, 66 and 65 (in the form for
// several slabs, 1 to 2 slower).  Heads of 32 and 16, 2,944 tokens and 48 and 63: 54 and 51, 58 and 51 (32), 48 and 46, 52 and 46 (16); 40
// behind them 52 and 52, 47 and 47 (the same form).  In batches of more than a CTA
// to an SM a CTA of the closed form works through several slabs and gains later: 704 tokens and 16, 32, 48 and 63 in four prompts 71 and 90,
// 82 and 91, 94 and 92, 106 and 93.  Without a tail the steps are faster in every batch: 44 and 49 (704 tokens, one prompt), 55 and 65 (four),
// 155 and 169 (16).
template <int KD, int VD>
int launch_hgdn_tail(const GdnArgs& a, const TailArgs& ta, cudaStream_t st) {
    dim3 grid(a.nseq, a.H, VD / TAIL_COLS);
    ProfScope prof("hgdn_tail", st);
    const bool room = ta.n0 <= 0 || ELL0 + __builtin_ctz((unsigned)ta.n0) < a.L;      // the first cascade must not leave the last level
    if (ta.tail >= (KD == 64 ? 16 : 48) && room) {
        using M = TailSmem<KD>;
        TailArgs tc = ta;
        while ((int64_t)a.nseq * a.H * grid.z > sm_count() && grid.z > 1) { grid.z /= 2; tc.slabs *= 2; }
        const int smem = M::floats(a.L, tc.slabs) * 4;
        constexpr int most = M::floats(40, VD / TAIL_COLS) * 4;
        static_assert(most <= 227 * 1024, "shared memory of an SM");
        static std::atomic<uint64_t> ready[2];
        const bool one = tc.slabs == 1;
        const auto kernel = one ? hgdn_tail_kernel<KD, VD, true> : hgdn_tail_kernel<KD, VD, false>;
        if (!allow_smem(ready[one], kernel, most)) return LAMPA_ERR_CUDA;
        launch_chained(kernel, grid, TAIL_THREADS, smem, st, a, tc);
        return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
    }
    const int slots = ta.tail > 0 ? __builtin_popcount((unsigned)ta.n0) : 0;
    const int staged = CHUNK * (2 * KD + TAIL_COLS + 2) + (ta.tail > 0 ? CHUNK * a.L + CHUNK * TAIL_COLS * 17 : 0);
    const int slab = ta.tail > 0 ? KD * TAIL_COLS * a.L : 0;
    const size_t smem = (size_t)(staged > slab ? staged : slab) * 4;
    constexpr int most = 82 * 1024;                          // 64 x 64 heads at 40 levels
    static std::atomic<uint64_t> ready[3];
    if (!allow_smem(ready[0], hgdn_tail_steps_kernel<KD, VD, 4>, most) || !allow_smem(ready[1], hgdn_tail_steps_kernel<KD, VD, 8>, most) ||
        !allow_smem(ready[2], hgdn_tail_steps_kernel<KD, VD, 24>, most)) return LAMPA_ERR_CUDA;
    if (slots <= 4) launch_chained(hgdn_tail_steps_kernel<KD, VD, 4>, grid, STEPS_THREADS, smem, st, a, ta);
    else if (slots <= 8) launch_chained(hgdn_tail_steps_kernel<KD, VD, 8>, grid, STEPS_THREADS, smem, st, a, ta);
    else launch_chained(hgdn_tail_steps_kernel<KD, VD, 24>, grid, STEPS_THREADS, smem, st, a, ta);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

// -------------------------------------------------------------------------------------------------
// Decode step (hattention_step -> step_state / step_output, models/hattention/kernel.py:570-633,
// recurrent.py:134-166): cascade, transition, insert, then o = q^T sum_l lambda_l S_l.  The levels of
// one (k, v) element are contiguous in memory, so the cascade is a prefix sum over a thread's own
// elements.  counts is shared by the batch: the last CTA to arrive at `arrivals` advances it (every
// CTA has read it by then), or a second, single-thread kernel when the caller has no such counter.
// A CTA whose slab did not arrive in time leaves it unstepped and says so (STEP_LATE in the counter
// before it arrives, or in counts[0]): whoever advances counts then takes the mark off and leaves
// them as they were.  In the counter because the last CTA's one atomic then tells it everything: a
// mark in counts, read back behind that atomic, took a step of a single stream from 6.7 to 7.6 us.
//
// What bounds it: streaming the state tensor once in and once out.  Half of the levels are live at a
// time, but they alternate inside every 32-byte sector, so the whole tensor moves.  A thread that
// walks the levels of its own element touches 4 bytes per sector and instruction: 148 us for 64 rows
// x 8 heads of 64 x 64 x 17 levels (286 MB, 1.9 TB/s).  Here a CTA owns 8 state columns: their
// K rows of 8 * L floats (544 bytes at L = 17) enter shared memory as one tiled copy, are updated in
// place and leave the same way: 56 us (5.1 TB/s, 78 % of the measured copy).  A bulk copy per row, 64 in and
// 64 out, kept the copy unit busier than the memory: 61 us, and 7.9 instead of 6.9 for four rows.
// Eight columns keep the slab at 35 KB, so that five CTAs per SM overlap their copies with each
// other's arithmetic, and give even a single stream of 4 heads of 32 columns 16 CTAs.  Two rows per
// thread, not four: the arithmetic is a chain of shared-memory round trips, and half the warps took
// 76 us (against 65 then).  16-byte cp.async and vector stores instead of the bulk copies: 97 us.
// -------------------------------------------------------------------------------------------------
__device__ __forceinline__ int cascade_depth(const int32_t* counts, int L, int& merged, bool& overflow) {
    // levels 0 .. depth-1 move into level `depth`, which then holds `merged` tokens
    int depth = 0, carry = 0;
    overflow = false;
    merged = 0;
    for (int l = 0; l < L; ++l) {
        const int64_t cap = l < 31 ? (int64_t)1 << l : (int64_t)1 << 31;
        const int64_t cur = (int64_t)counts[l] + carry;
        if (cur == cap) {
            if (l + 1 >= L) { overflow = true; break; }
            carry = (int)cur;
            depth = l + 1;
        } else {
            if (cur > cap) overflow = true;
            merged = (int)cur;
            break;
        }
    }
    return depth;
}

constexpr int STEP_COLS = 8, STEP_MAX_L = 40, STEP_KI = 2;      // rows of a thread
constexpr uint32_t STEP_LATE = 0x80000000u;                     // some slab has not taken the token in; never left behind
template <int KD> constexpr int STEP_THREADS = KD * STEP_COLS / STEP_KI;
template <int KD> __host__ __device__ constexpr int step_smem(int L) {      // slab, partial sums, c
    return (KD * STEP_COLS + 2 * (STEP_THREADS<KD> / 32) * STEP_COLS + STEP_COLS) * L * 4;
}

template <int KD, int VD>
__global__ void __launch_bounds__(STEP_THREADS<KD>) hgdn_step_kernel(StepArgs s, const __grid_constant__ CUtensorMap map, int tiled) {
    if (chain_wait()) return;
    constexpr int NT = STEP_THREADS<KD>, NW = NT / 32, KI = STEP_KI;        // lane = (4 rows, 8 columns)
    extern __shared__ __align__(128) float slab[];              // [KD][8][L]
    float* part = slab + KD * STEP_COLS * s.L;                 // [2][warps][L][8]: k^T S and q^T S of every level
    float* sC = part + 2 * NW * STEP_COLS * s.L;               // [L][8]: beta k^T S
    __shared__ float sK[KD], sQ[KD], sLam[STEP_MAX_L], sQk;
    __shared__ int32_t sCnt[STEP_MAX_L];
    __shared__ __align__(8) uint64_t bar;
    const int b = blockIdx.x / (VD / STEP_COLS), v0 = (blockIdx.x - b * (VD / STEP_COLS)) * STEP_COLS;
    const int h = blockIdx.y, H = s.H, L = s.L;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col = lane & 7, kq = (lane >> 3) + 4 * warp;
    const size_t bh = (size_t)b * H + h;
    float* gsrc = s.states + (bh * KD * VD + v0) * L;           // row k: KD rows of 8 L floats, VD L floats apart
    const uint32_t row_bytes = STEP_COLS * L * 4;               // a multiple of 32
    const bool bulk = ((uintptr_t)s.states & 15) == 0;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        if (bulk) mbar_expect_tx(&bar, KD * row_bytes);
    }
    __syncthreads();
    if (tiled) {
        if (tid == 0) tma_load_2d(slab, &map, v0 * L, (int32_t)(bh * KD), &bar);
    } else if (bulk) {
        if (tid < KD) bulk_g2s(slab + (size_t)tid * STEP_COLS * L, gsrc + (size_t)tid * VD * L, row_bytes, &bar);
    } else {
        for (int i = tid; i < KD * STEP_COLS * L; i += NT) {
            const int r = i / (STEP_COLS * L);
            slab[i] = gsrc[(size_t)r * VD * L + (i - r * STEP_COLS * L)];
        }
    }
    if (tid >= NT - L) {
        const int l = tid - (NT - L);
        sCnt[l] = (int32_t)((uint32_t)s.counts[l] & ~STEP_LATE);
        sLam[l] = load_as_float(s.lam, bh * L + l, s.lam_dt);
    }
    const float eg = __expf(load_as_float(s.g, bh, s.gb_dt));
    const float bt = load_as_float(s.beta, bh, s.gb_dt);
    const float vt = load_as_float(s.v, bh * VD + v0 + col, s.qkv_dt);
    if (warp == 0) {
        float kx[(KD + 31) / 32], qx[(KD + 31) / 32];
        float sk = 0.f, sq = 0.f, qk = 0.f;
#pragma unroll
        for (int j = 0; j < (KD + 31) / 32; ++j) {
            const int c = lane + 32 * j;
            kx[j] = c < KD ? load_as_float(s.k, bh * KD + c, s.qkv_dt) : 0.f;
            qx[j] = c < KD ? load_as_float(s.q, bh * KD + c, s.qkv_dt) : 0.f;
            sk += kx[j] * kx[j];
            sq += qx[j] * qx[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
        }
        const float rk = rsqrtf(sk + 1e-6f), rq = rsqrtf(sq + 1e-6f);
#pragma unroll
        for (int j = 0; j < (KD + 31) / 32; ++j) {
            const int c = lane + 32 * j;
            if (s.use_l2norm) { kx[j] = round_like(kx[j] * rk, s.qkv_dt); qx[j] *= rq; }
            if (c < KD) { sK[c] = kx[j]; sQ[c] = qx[j]; }
            qk += kx[j] * qx[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) qk += __shfl_xor_sync(0xffffffffu, qk, o);
        if (lane == 0) sQk = qk;
    }
    __syncthreads();
    int merged;
    bool overflow;
    const int depth = cascade_depth(sCnt, L, merged, overflow);
    auto arrive = [&](bool late) {                 // one thread per CTA
        if (late) atomicOr(reinterpret_cast<uint32_t*>(s.arrivals ? s.arrivals : s.counts), STEP_LATE);
        if (!s.arrivals) return;
        const uint32_t n = atomicAdd(reinterpret_cast<uint32_t*>(s.arrivals), 1u);
        if ((n & ~STEP_LATE) != gridDim.x * gridDim.y - 1) return;
        *s.arrivals = 0;                           // for the next step
        if (n & STEP_LATE || overflow) return;
        for (int l = 0; l < depth; ++l) s.counts[l] = 0;
        if (depth > 0) s.counts[depth] = merged;
        s.counts[0] = 1;
    };
    bool dead = false;
    if (bulk) mbar_wait(&bar, 0u, dead, s.status, 32, s.poll_budget);
    if (overflow || __syncthreads_or(dead)) {     // nothing changes; the copies land before the CTA gives its memory back
        if (overflow && tid == 0 && bh == 0 && v0 == 0) set_status(s.status, LAMPA_ERR_LEVELS, 31, depth);
        if (bulk) mbar_drain(&bar, 0u);
        __syncthreads();
        if (tid == 0) arrive(!overflow);
        return;
    }
    uint64_t live = 0;                             // levels >= 1 that hold tokens after the cascade
    for (int l = max(depth, 1); l < L; ++l) live |= (uint64_t)(l == depth ? merged > 0 : sCnt[l] != 0) << l;

    float kr[KI], qr[KI];
    float* P[KI];
#pragma unroll
    for (int i = 0; i < KI; ++i) {
        const int r = kq + 4 * NW * i;
        kr[i] = sK[r];
        qr[i] = sQ[r];
        P[i] = slab + ((size_t)r * STEP_COLS + col) * L;
    }
    if (depth > 0) {                               // levels 0 .. depth - 1 join level `depth`
#pragma unroll
        for (int i = 0; i < KI; ++i) {
            float x = 0.f;
            for (int j = 0; j <= depth; ++j) { x += P[i][j]; P[i][j] = 0.f; }
            P[i][depth] = x;
        }
    }
    for (uint64_t m = live; m; m &= m - 1) {
        const int l = __ffsll((long long)m) - 1;
        float dk = 0.f, dq = 0.f;
#pragma unroll
        for (int i = 0; i < KI; ++i) { const float x = P[i][l]; dk += kr[i] * x; dq += qr[i] * x; }
        dk += __shfl_xor_sync(0xffffffffu, dk, 8);
        dq += __shfl_xor_sync(0xffffffffu, dq, 8);
        dk += __shfl_xor_sync(0xffffffffu, dk, 16);
        dq += __shfl_xor_sync(0xffffffffu, dq, 16);
        if (lane < 2 * STEP_COLS) part[(((lane >> 3) * NW + warp) * L + l) * STEP_COLS + col] = lane < STEP_COLS ? dk : dq;
    }
    __syncthreads();
    for (int i = tid; i < L * STEP_COLS; i += NT)
        if ((live >> (i >> 3)) & 1) {
            float c = 0.f, q = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) { c += part[w * L * STEP_COLS + i]; q += part[(NW + w) * L * STEP_COLS + i]; }
            sC[i] = bt * c;
            part[i] = q;                           // read by this thread only so far
        }
    __syncthreads();
    const float bv = bt * vt;
    for (uint64_t m = live; m; m &= m - 1) {
        const int l = __ffsll((long long)m) - 1;
        const float c = sC[l * STEP_COLS + col];
#pragma unroll
        for (int i = 0; i < KI; ++i) P[i][l] = eg * (P[i][l] - kr[i] * c);
    }
#pragma unroll
    for (int i = 0; i < KI; ++i) P[i][0] = kr[i] * bv;
    if (warp == 0) {                               // o = sum_l lambda_l e^g (q^T S_l - (q.k) c_l) + lambda_0 (q.k) beta v
        float out = 0.f;
        for (int l = 1 + (lane >> 3); l < L; l += 4)
            if ((live >> l) & 1) out += sLam[l] * (eg * (part[l * STEP_COLS + col] - sQk * sC[l * STEP_COLS + col]));
        out += __shfl_xor_sync(0xffffffffu, out, 8);
        out += __shfl_xor_sync(0xffffffffu, out, 16);
        if (lane < STEP_COLS) store_from_float(s.o, bh * VD + v0 + col, out + sLam[0] * (sQk * bv), s.qkv_dt);
    }
    if (bulk) {
        fence_async_shared();
        __syncthreads();
        if (tiled) {
            if (tid == 0) { tma_store_2d(&map, v0 * L, (int32_t)(bh * KD), slab); bulk_commit(); }
        } else if (tid < KD) {
            bulk_s2g(gsrc + (size_t)tid * VD * L, slab + (size_t)tid * STEP_COLS * L, row_bytes);
            bulk_commit();
        }
    } else {
        __syncthreads();
        for (int i = tid; i < KD * STEP_COLS * L; i += NT) {
            const int r = i / (STEP_COLS * L);
            gsrc[(size_t)r * VD * L + (i - r * STEP_COLS * L)] = slab[i];
        }
    }
    if (tid == 0) arrive(false);
    if (bulk && tid < KD) bulk_wait_read();
}

__global__ void hgdn_step_counts_kernel(int32_t* counts, int L) {
    if (chain_wait()) return;
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const uint32_t c0 = (uint32_t)counts[0];
    if (c0 & STEP_LATE) { counts[0] = (int32_t)(c0 & ~STEP_LATE); return; }
    int merged;
    bool overflow;
    const int depth = cascade_depth(counts, L, merged, overflow);
    if (overflow) return;
    for (int l = 0; l < depth; ++l) counts[l] = 0;
    if (depth > 0) counts[depth] = merged;
    counts[0] += 1;
}

template <int KD, int VD>
int launch_hgdn_step(const StepArgs& s, cudaStream_t st) {
    const int smem = step_smem<KD>(s.L);
    static std::atomic<uint64_t> ready;
    if (!allow_smem(ready, hgdn_step_kernel<KD, VD>, step_smem<KD>(STEP_MAX_L))) return LAMPA_ERR_CUDA;      // 103 KB
    // one tiled copy per slab, up to 32 levels (a box is at most 256 elements wide)
    CUtensorMap map = {};
    const int64_t rows = (int64_t)s.B * s.H * KD;
    const int tiled = ((uintptr_t)s.states & 15) == 0 && STEP_COLS * s.L <= 256 && rows <= INT32_MAX &&
                      make_map(&map, s.states, LAMPA_F32, (uint64_t)rows, (uint64_t)VD * s.L, STEP_COLS * s.L, KD, false);
    {
        ProfScope prof("hgdn_step", st);
        launch_chained(hgdn_step_kernel<KD, VD>, dim3((unsigned)s.B * (VD / STEP_COLS), s.H), STEP_THREADS<KD>, smem, st, s, map, tiled);
        if (cudaGetLastError() != cudaSuccess) return LAMPA_ERR_CUDA;
    }
    if (s.arrivals) return LAMPA_OK;
    launch_chained(hgdn_step_counts_kernel, 1, 32, 0, st, s.counts, s.L);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

#define LAMPA_INST(KD, VD)                                                                      \
    template int launch_hgdn_tail<KD, VD>(const GdnArgs&, const TailArgs&, cudaStream_t);       \
    template int launch_hgdn_step<KD, VD>(const StepArgs&, cudaStream_t);
LAMPA_INST(64, 64)
LAMPA_INST(32, 32)
LAMPA_INST(16, 32)
#undef LAMPA_INST

}  // namespace lampa
