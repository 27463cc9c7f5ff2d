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

#include <type_traits>

namespace lampa {

__device__ __forceinline__ float round_like(float x, int dt) {
    if (dt == LAMPA_BF16) return __bfloat162float(__float2bfloat16_rn(x));
    if (dt == LAMPA_F16) return __half2float(__float2half_rn(x));
    return x;
}

// Eight consecutive elements as floats (zeros where `live` is false): 16-byte loads where the base allows them
__device__ __forceinline__ void load8_as_float(const void* p, size_t i, int dt, bool live, float (&x)[8]) {
    if (!live) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = 0.f;
    } else if (((uintptr_t)p & 15) != 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = load_as_float(p, i + e, dt);
    } else if (dt == LAMPA_F32) {
        const float4 u = __ldg(reinterpret_cast<const float4*>((const float*)p + i)), v = __ldg(reinterpret_cast<const float4*>((const float*)p + i) + 1);
        x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    } else {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>((const uint16_t*)p + i));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = dt == LAMPA_BF16 ? unpack_bf16x2(w[e]) : __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
            x[2 * e] = f.x; x[2 * e + 1] = f.y;
        }
    }
}

// -------------------------------------------------------------------------------------------------
// End of a sequence, token by token in fp32: the token levels 0..6 after its last whole chunk (the
// recurrence over that chunk from an empty state, as the reference's postprocess_prefill_hstate_
// does, models/hattention/kernel.py:377-466), then, for a prefill, the T mod 64 tokens behind it with
// all levels and their outputs (what the reference hands to its step function, kernel.py:470-560).
// Inside one chunk the cascade is fixed: before token t > 0, levels 0..tz(t) collapse into level
// tz(t) + 1 (tz = trailing zeros); before the first token behind n0 chunks, the token levels and the
// trailing full chunk levels collapse into level 7 + tz(n0), after which the live chunk levels are
// the set bits of n0 and do not change any more: they sit in HS register slots, in bit order.
// Without a tail a ragged last chunk (cu_seqlens) is completed with null tokens (k = v = 0,
// beta = 0, g = 0).  Also writes counts.
//
// State columns are independent, so a half-warp owns one: lane kl has rows kl, kl + 16, ... of every
// level in registers, a level's k^T S is K / 16 FMAs and four shuffles, and the levels of a token
// are independent chains that hide each other's latency.  What bounds it is that chain, 0.3 us per
// token of the last whole chunk and 0.4 us per token behind it (8 heads, K = V = 64: 19 us at 2944
// tokens, 47 us at 3001); with one CTA per (sequence, head) and a launch per tail token (61 us for the
// token levels and 27 us per tail token) a 3001-token prompt spent 1.7 of its 1.9 ms on the device here.
// -------------------------------------------------------------------------------------------------
constexpr int TAIL_COLS = 8, TAIL_THREADS = 128;

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
__global__ void __launch_bounds__(TAIL_THREADS) hgdn_tail_kernel(GdnArgs a, TailArgs ta) {
    if (chain_wait()) return;
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

    // rows [t0, t0 + len) of the inputs as the kernel uses them; rows up to 64 become null tokens.  Eight elements per
    // thread and step, K / 8 threads per row, every load in flight before the first is used.
    auto stage = [&](int64_t t0, int len, bool tail) {
        constexpr int PPR = KD / 8, NIT = CHUNK * PPR / TAIL_THREADS;
        float x[NIT][8], y[NIT][8];
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int p = tid + it * TAIL_THREADS, r = p / PPR, c = (p % PPR) * 8;
            const size_t at = ((size_t)(t0 + r) * H + h) * KD + c;
            load8_as_float(a.k, at, a.qkv_dt, r < len, x[it]);
            load8_as_float(a.q, at, a.qkv_dt, r < len && tail, y[it]);
        }
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int p = tid + it * TAIL_THREADS, r = p / PPR, c = (p % PPR) * 8;
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
        for (int i = tid; i < CHUNK * TAIL_COLS; i += TAIL_THREADS) {
            const int r = i / TAIL_COLS, c = i - r * TAIL_COLS;
            sV[i] = r < len ? load_as_float(a.v, ((size_t)(t0 + r) * H + h) * VD + v0 + c, a.qkv_dt) : 0.f;
        }
        if (tid < CHUNK) {
            sEg[tid] = tid < len ? __expf(load_as_float(a.g, (size_t)(t0 + tid) * H + h, a.gb_dt)) : 1.f;
            sBeta[tid] = tid < len ? load_as_float(a.beta, (size_t)(t0 + tid) * H + h, a.gb_dt) : 0.f;
        }
        if (tail) {                             // two threads per token, up to twenty levels each
            const int r = tid >> 1;
            if (r < len) {
                float w[20];
#pragma unroll
                for (int i = 0; i < 20; ++i) w[i] = (tid & 1) + 2 * i < L ? load_as_float(a.lam, ((size_t)(t0 + r) * H + h) * L + (tid & 1) + 2 * i, a.lam_dt) : 0.f;
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
    // chunk levels the tail continues from, on their way while the last chunk is run
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
#pragma unroll
    for (int s = 0; s < HS; ++s)
#pragma unroll
        for (int i = 0; i < KI; ++i) X[s][i] = ta.tail > 0 && room && lvl[s] >= 0 && s > 0 ? st[i * row16 + lvl[s]] : 0.f;
    if (ta.tail > 0 && room && nch > 0) {
#pragma unroll
        for (int i = 0; i < KI; ++i)
            for (int l = ELL0; l < lvl[0]; ++l) X[0][i] += st[i * row16 + l];
    }

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
            for (int i = tid; i < done * TAIL_COLS; i += TAIL_THREADS) {
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
        if (rem != 0) set_status(a.status, LAMPA_ERR_LEVELS, 30, seq);
    }
}

template <int KD, int VD>
int launch_hgdn_tail(const GdnArgs& a, const TailArgs& ta, cudaStream_t st) {
    const int slots = ta.tail > 0 ? __builtin_popcount((unsigned)ta.n0) : 0;
    const int staged = CHUNK * (2 * KD + TAIL_COLS + 2) + (ta.tail > 0 ? CHUNK * a.L + CHUNK * TAIL_COLS * 17 : 0);
    const int slab = ta.tail > 0 ? KD * TAIL_COLS * a.L : 0;
    const size_t smem = (size_t)(staged > slab ? staged : slab) * 4;
    constexpr int most = 82 * 1024;                          // 64 x 64 heads at 40 levels
    static std::atomic<uint64_t> ready[3];
    if (!allow_smem(ready[0], hgdn_tail_kernel<KD, VD, 4>, most) || !allow_smem(ready[1], hgdn_tail_kernel<KD, VD, 8>, most) ||
        !allow_smem(ready[2], hgdn_tail_kernel<KD, VD, 24>, most)) return LAMPA_ERR_CUDA;
    const dim3 grid(a.nseq, a.H, VD / TAIL_COLS);
    ProfScope prof("hgdn_tail", st);
    if (slots <= 4) launch_chained(hgdn_tail_kernel<KD, VD, 4>, grid, TAIL_THREADS, smem, st, a, ta);
    else if (slots <= 8) launch_chained(hgdn_tail_kernel<KD, VD, 8>, grid, TAIL_THREADS, smem, st, a, ta);
    else launch_chained(hgdn_tail_kernel<KD, VD, 24>, grid, TAIL_THREADS, smem, st, a, ta);
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
// K rows of 8 * L floats (544 bytes at L = 17) enter shared memory as bulk copies, are updated in
// place and leave the same way: 65 us (4.4 TB/s).  Eight columns keep the slab at 35 KB, so that
// five CTAs per SM overlap their copies with each other's arithmetic, and give even a single stream
// of 4 heads of 32 columns 16 CTAs.  Two rows per thread, not four: the arithmetic is a chain of
// shared-memory round trips, and half the warps took 76 us.  16-byte cp.async and vector stores
// instead of the bulk copies: 97 us.
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
__global__ void __launch_bounds__(STEP_THREADS<KD>) hgdn_step_kernel(StepArgs s) {
    if (chain_wait()) return;
    constexpr int NT = STEP_THREADS<KD>, NW = NT / 32, KI = STEP_KI;        // lane = (4 rows, 8 columns)
    extern __shared__ __align__(16) float slab[];              // [KD][8][L]
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
    if (bulk) {
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
        if (tid < KD) {
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
    const int smem = step_smem<KD>(s.L);           // at most 103 KB
    if (smem > 44 * 1024 && cudaFuncSetAttribute(hgdn_step_kernel<KD, VD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return LAMPA_ERR_CUDA;
    {
        ProfScope prof("hgdn_step", st);
        launch_chained(hgdn_step_kernel<KD, VD>, dim3((unsigned)s.B * (VD / STEP_COLS), s.H), STEP_THREADS<KD>, smem, st, s);
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
