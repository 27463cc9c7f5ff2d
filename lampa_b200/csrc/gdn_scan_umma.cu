// Output pass of the hierarchical rule on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM) for K = V = 64.
//
// Per (block of up to 32 chunks, head) one CTA keeps every level state the block touches as rows of
// bf16 A operands in tensor memory: slot s holds S_l^T (64 rows v x 64 columns k), two slots
// per 128-row operand ("pair").  The first block_log slots are the chunk levels that live inside the block,
// the following ones the cross-block levels this block reads (seeded from the level pass).
// A chunk is one record {M | Q~ | B^T | O_local | lambda}; its first 16 KB, the M and Q~ tiles back to
// back, are a single 128-row K-major B operand, so ONE accumulating MMA per pair,
//     D[128 x 128] = [S_a^T ; S_b^T] (128 x 64)  x  [M ; Q~]^T (64 x 128),
// yields both the advanced states (columns 0..63: S^T M^T) and the levels' contributions to the
// output (columns 64..127: S^T Q~^T = (Q~ S)^T).  The epilogue, one thread per TMEM lane (= state
// row) and quarter of the columns, adds B^T where the level is collecting, clears it at the end of
// its period and writes the bf16 row back into the A operand for the next chunk; then it scales
// the level's contribution to its 16 tokens by lambda and accumulates it over the pairs.
// Warp-specialised: 16 epilogue warps (warp = 32 rows x 16 state columns x 16 tokens), four output warps that take the
// chunk's output from them through shared memory and store it with O_local added, and one
// control warp whose first lane streams the records in (bulk async copies, three stages) and issues
// the MMAs.  The MMAs take the accumulator buffers in turn; one is issued as soon as every epilogue warp has
// handed back the buffer it overwrites, which it does after rewriting the pair's operand and reading the
// pair's contribution (a hardware named barrier per pair that the control warp joins: no block-wide barrier
// and no polling on the state path).  MMA completion is tracked by tcgen05.commit on one mbarrier per
// pair; every mbarrier wait is bounded, and a CTA whose wait ran out stops issuing copies and MMAs, lets
// every warp walk through its remaining barriers in lockstep, waits for the copies and MMAs in flight
// and only then frees its tensor memory.
#include "act.cuh"
#include "gdn.cuh"
#include "profile.cuh"
#include "umma.cuh"

namespace lampa {

namespace {

constexpr int UKD = 64, UVD = 64;
constexpr int UNP = 5;                       // pairs of slots: up to 5 in-block levels + up to 5 cross-block levels
constexpr int UEPI_WARPS = 16;               // 4 warpgroups, each covering 16 state columns and 16 tokens of all 128 rows
constexpr int UOUT_WARPS = 4;                 // warps that store the output
constexpr int PTHREADS = (UEPI_WARPS + 2) * 32;   // with one control warp and one relay warp
constexpr int UTHREADS = PTHREADS + UOUT_WARPS * 32;
// An mbarrier poll costs the polling warp 200 - 300 cycles even when the phase is long complete, a hardware named
// barrier that everybody else has already reached about 30.  So only the relay warp polls the mbarriers the epilogue
// depends on ("record landed", "pair's MMA complete") and passes each completion on through a named barrier that the
// sixteen epilogue warps join (ids 5 + p; ids 1..4 belong to the output tile), and the epilogue hands a pair's
// accumulator back to the control warp the same way (ids 11 + p: sixteen warps arrive, the control warp waits).
// Nobody can be left waiting at a named barrier: the relay's and the control lane's own waits are bounded and both
// walk through every barrier whether or not a wait ran out, and the epilogue never waits for anything else.  Nobody
// can reach a barrier twice in one phase either: a pair's next MMA is issued only after its hand-back was joined, and
// once a wait has run out (flag in shared memory) relay and epilogue join their barriers synchronously instead of
// arriving and running on.
constexpr int UNB_PAIR = 5, UNB_DFREE = 11, UNB_COUNT = (UEPI_WARPS + 1) * 32;
// The chunk's output tile (fp32, two buffers in turn) goes to the output warps at id 1 + buffer, and
// comes back at id 3 + buffer.  Both sides wait for the other before they reuse a buffer, so neither can reach a barrier twice.
constexpr int UNB_OFULL = 1, UNB_OFREE = 3, UNB_OCOUNT = (UEPI_WARPS + UOUT_WARPS) * 32;
__device__ __forceinline__ void out_arrive(int id) { asm volatile("bar.arrive %0, %1;\n" :: "r"(id), "n"(UNB_OCOUNT) : "memory"); }
__device__ __forceinline__ void out_sync(int id) { asm volatile("bar.sync %0, %1;\n" :: "r"(id), "n"(UNB_OCOUNT) : "memory"); }
__device__ __forceinline__ void named_arrive(int id) { asm volatile("bar.arrive %0, %1;\n" :: "r"(id), "n"(UNB_COUNT) : "memory"); }
__device__ __forceinline__ void named_sync(int id) { asm volatile("bar.sync %0, %1;\n" :: "r"(id), "n"(UNB_COUNT) : "memory"); }
__device__ __forceinline__ void relay_pass(int id, bool dead) { if (dead) named_sync(id); else named_arrive(id); }
constexpr int UNST = 3;                      // record stages
using UR = Rec<UKD, UVD>;

// shared-memory map (bytes); everything that tcgen05 reads is 1024-byte aligned
constexpr int SM_BAR = 0;                    // full[UNST], mma[UNP] mbarriers, TMEM slot
constexpr int SM_OT = 1024;                  // two buffers (chunk parity) of fp32 [2][64 tokens][64 v]: output transpose / pair-half sum
// TMEM columns (512 allocated): the states as bf16 A operands, 32 columns per pair, then the
// 128-column accumulator buffers used by the MMAs in turn (three from column 128 when there are at
// most four pairs, else two from column 192)
constexpr int TM_A = 0;
constexpr int TM_D = 192;
constexpr int SM_STAGE = SM_OT + 2 * 2 * 64 * 64 * 4;
constexpr int STAGE_TILES = UR::LAM_OFF;     // M | Q~ | B^T | O_local, then the lambda rows: the whole record
__host__ __device__ constexpr int ustage_bytes(int LC) { return (STAGE_TILES + LC * CHUNK * 4 + 1023) / 1024 * 1024; }

// instruction descriptor: D fp32, A/B bf16, both K-major, M = 128, N = 128
constexpr uint32_t UMMA_IDESC = umma_idesc(128, 128);

// columns 16p .. 16p + 15 of row v of an entry state
__device__ __forceinline__ void load_state16(float (&x)[16], const float* state, int v, int p) {
    const float4* e = reinterpret_cast<const float4*>(state + UR::state_at(v, 16 * p));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 f = e[i];
        x[2 * i] = f.x; x[2 * i + 1] = f.y; x[8 + 2 * i] = f.z; x[9 + 2 * i] = f.w;
    }
}

// Launch order of the (block, head) units.  A unit's time grows with the number of level pairs it
// carries (3 to 5, from the set bits of its block index), and 240 units on 148 SMs leave the second
// round partly empty: handing the long units out first lets the short ones fill the tail.
struct UnitOrder {
    int nbs;                    // blocks per sequence when all sequences are equally long and nbs <= 64, else 0
    unsigned char order[64];    // block indices, most level pairs first
};

// A chunk's step is bound by the serial work of the epilogue warps (two tensor-memory round trips and two barriers per
// pair), so nothing else is left to them: storing the output took 1840 of a step's 5250 cycles at four pairs, most of it
// waiting for the scatter index, which four warps of their own now fetch a chunk ahead.  60,000 hits, 8 heads, 10 levels,
// scattered output: 182 -> 150 us.  (Two output warps: 158 us, and 27 instead of 25 us for a 6,000-hit event; loading both
// halves of the accumulator row at once: 166 - 217 us, the registers spill.)
__global__ void __launch_bounds__(UTHREADS, 1) gdn_out_hier_umma_kernel(GdnArgs a, UnitOrder uo) {
    if (chain_wait()) return;
    if (a.signal) chain_signal(a.signal_word, a.signal);
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM_BAR);      // record landed            (tx count)
    uint64_t* sfree = full + UNST;                                      // stage consumed           (16 + 4 warps)
    uint64_t* mdone = sfree + UNST;                                     // pair's MMA complete      (commit)
    uint64_t* drainb = mdone + UNP;                                     // every MMA issued has completed (commit at the end)
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + SM_BAR + 256);
    volatile uint32_t* sdead = reinterpret_cast<volatile uint32_t*>(smem + SM_BAR + 260);   // set once a bounded wait has run out
    float* sOT = reinterpret_cast<float*>(smem + SM_OT);

    const int H = a.H;
    int gb, h;
    if (uo.nbs > 0) {
        const int per_rank = H * a.nseq, r = blockIdx.x / per_rank, rem = blockIdx.x - r * per_rank;
        h = rem % H;
        gb = (rem / H) * uo.nbs + uo.order[r];
    } else {
        gb = blockIdx.x % a.nb_max;
        h = blockIdx.x / a.nb_max;
    }
    SeqLoc sq;
    int b;
    if (!locate_block(a, gb, sq, b)) return;
    const int nch = sq.nch;
    const int nlev = nch > 1 ? ceil_log2_int(nch) : 0;
    if (a.short_only && nlev > UMMA_LEVELS) return;
    const int bl = block_log(nch), bc = 1 << bl;
    const int nhigh = min(max(0, nlev - bl), a.nhigh_max);     // more only when the level check has already failed
    const int c0 = sq.c0 + b * bc;
    const int nsteps = min(bc, nch - b * bc);
    const int64_t tok0 = sq.tok0 + (int64_t)b * bc * CHUNK, tok_end = sq.tok_end;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wg = warp >> 2;                          // 0..3: state columns / tokens 16*wg .. 16*wg+15
    const int row = (warp & 3) * 32 + lane;            // TMEM lane = row of the pair's A operand
    const int u = row >> 6, v = row & 63;              // which slot of the pair, which state row
    const int part = wg & 3;
    const int lam_bytes = a.LC * CHUNK * 4;
    const int stage_bytes = ustage_bytes(a.LC);
    unsigned char* stage0 = smem + SM_STAGE;
    const char* rec0 = a.rec + ((size_t)c0 * H + h) * a.rec_bytes;
    const size_t rec_stride = (size_t)H * a.rec_bytes;

    // cross-block levels this block reads, compacted into slots bl, bl + 1, ...
    int nlive = 0;
    uint32_t live_pack = 0;                            // 4 bits per compact slot: the level index
    for (int lh = 0; lh < nhigh; ++lh)
        if ((b >> lh) & 1) { live_pack |= (uint32_t)lh << (4 * nlive); ++nlive; }
    const int nslots = bl + nlive;
    const int npairs = (nslots + 1) >> 1;
    // accumulator buffers of 128 columns behind the operands: three where four pairs or fewer leave room for them,
    // never more than pairs (the hand-back of MMA m - nbuf must be the latest one of its pair)
    const int nbuf = npairs <= 4 ? min(npairs, 3) : 2, tm_d = npairs <= 4 ? 128 : TM_D;

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < UNST; ++s) { mbar_init(full + s, 1); mbar_init(sfree + s, UEPI_WARPS + UOUT_WARPS); }
#pragma unroll
        for (int p = 0; p < UNP; ++p) mbar_init(mdone + p, 1);
        mbar_init(drainb, 1);
        *sdead = 0u;
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(tslot, 512);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *tslot;
    const uint32_t tlane = taddr + ((uint32_t)((warp & 3) * 32) << 16);
    // initial states: zero for the in-block levels, the block's entry state for the cross-block ones
    if (wg < 4) {
        for (int p = 0; p < npairs; ++p) {
            const int s = 2 * p + u;
            float x[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = 0.f;
            if (s >= bl && s < nslots) {
                const int lh = (live_pack >> (4 * (s - bl))) & 15;
                load_state16(x, a.entry + (((size_t)gb * a.nhigh_max + lh) * H + h) * UR::STATE_FLOATS, v, part);
            }
            tmem_st_bf16x16(tlane + TM_A + 32 * p + 8 * part, x);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    bool dead = false;
    const int budget = a.poll_budget;

    if (warp == UEPI_WARPS) {
        // ---- control warp: lane 0 streams records and issues MMAs; the whole warp joins the named barriers ----
        int loaded = 0, landed = 0;                  // records requested / records seen in shared memory (lane 0)
        auto load_record = [&](int step) {
            uint64_t* fb = full + (step % UNST);
            unsigned char* dst = stage0 + (size_t)(step % UNST) * stage_bytes;
            const char* src = rec0 + (size_t)step * rec_stride;
            mbar_expect_tx(fb, (uint32_t)(STAGE_TILES + lam_bytes));
            bulk_g2s(dst, src, (uint32_t)(STAGE_TILES + lam_bytes), fb);
            loaded = step + 1;
        };
        if (lane == 0)
            for (int s = 0; s < UNST - 1 && s < nsteps; ++s) load_record(s);
        // The MMAs are numbered through the chunks, m = i * npairs + p, and take the accumulator buffers in turn:
        // MMA m overwrites the buffer MMA m - nbuf filled, once the epilogue has handed that one back.  The epilogue hands
        // a pair's accumulator back after it has rewritten the pair's operand, and it works through chunks and pairs in
        // order, so the same hand-back also covers the operand of pair p rewritten in the previous chunk (npairs >= nbuf).
        // Every hand-back is joined exactly once and in the order it is given, whether or not anything is still issued.
        int bufi = 0;
        for (int i = 0; i < nsteps; ++i) {
            const unsigned char* st = stage0 + (size_t)(i % UNST) * stage_bytes;
            if (lane == 0 && !dead && mbar_wait(full + (i % UNST), (uint32_t)((i / UNST) & 1), dead, a.status, 200 + i, budget)) landed = i + 1;
            for (int p = 0; p < npairs; ++p) {
                __syncwarp();
                if (p >= nbuf) named_sync(UNB_DFREE + p - nbuf);
                else if (i > 0) named_sync(UNB_DFREE + npairs - nbuf + p);
                const uint32_t dcol = (uint32_t)(tm_d + bufi * 128);
                bufi = bufi + 1 == nbuf ? 0 : bufi + 1;
                if (lane == 0 && !dead) {
                    tc_fence_after();
                    const uint32_t b_base = smem_u32(st + UR::M_OFF);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16_ts(taddr + dcol, taddr + (uint32_t)(TM_A + 32 * p + 8 * kk),
                                    umma_desc_k128(b_base + kk * 32), UMMA_IDESC, kk > 0 ? 1u : 0u);
                    umma_commit(mdone + p);
                }
            }
            if (lane == 0 && !dead && i + UNST - 1 < nsteps) {       // refill the stage chunk i-1 used, once everyone is done with it
                if (i >= 1) mbar_wait(sfree + ((i - 1) % UNST), (uint32_t)(((i - 1) / UNST) & 1), dead, a.status, 500 + i, budget);
                if (!dead) load_record(i + UNST - 1);
            }
            if (lane == 0 && dead) *sdead = 1u;
        }
        __syncwarp();
        for (int p = npairs - nbuf; p < npairs; ++p) named_sync(UNB_DFREE + p);      // the last chunk's outstanding hand-backs
        if (lane == 0) {
            // nothing asynchronous may outlive the CTA: records still on their way land first, and one
            // last commit covers every MMA issued above
            for (int s = landed; s < loaded; ++s) mbar_drain(full + (s % UNST), (uint32_t)((s / UNST) & 1));
            umma_commit(drainb);
            mbar_drain(drainb, 0u);
        }
    } else if (warp == UEPI_WARPS + 1) {
        // ---- relay warp (the second warp of this group): mbarrier completions -> named barriers ----
        // "record landed" travels with the first pair of the chunk.  A pair's barrier cannot be reached a second time
        // before every epilogue warp has left it: the pair's next MMA is only issued after its accumulator came back.
        for (int i = 0; i < nsteps; ++i) {
            mbar_wait(full + (i % UNST), (uint32_t)((i / UNST) & 1), dead, a.status, 250 + i, budget);
            for (int p = 0; p < npairs; ++p) {
                mbar_wait(mdone + p, (uint32_t)(i & 1), dead, a.status, 300 + p, budget);
                if (dead) *sdead = 1u;
                relay_pass(UNB_PAIR + p, dead);
            }
        }
    } else if (warp > UEPI_WARPS + 1) {
        // ---- output warps: sum the two rows (levels) of the pairs, add O_local, store ----
        // thread = (every 16th token, 4 + 4 output columns: 4c.. and 32 + 4c..): the eight lanes of a token read 128
        // contiguous bytes of the tile per load, which is what keeps the 16-byte loads free of bank conflicts
        const int ot = tid - PTHREADS, tok = ot >> 3, col = (ot & 7) * 4;
        auto drain_tiles = [&](auto scat) {
            // a scattered row's index is asked for one chunk ahead and looked at (see out_row) when its tile is there
            int64_t next[4];
            auto ask_rows = [&](int i) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int64_t t = tok0 + (int64_t)i * CHUNK + tok + 16 * q;
                    next[q] = t >= tok_end ? -1 : t;
                    if (decltype(scat)::value && t < tok_end && t < a.out_perm_rows) next[q] = a.out_perm[t];
                }
            };
            ask_rows(0);
            for (int i = 0; i < nsteps; ++i) {
                const int64_t orow[4] = {next[0], next[1], next[2], next[3]};
                ask_rows(i + 1);
                const __nv_bfloat16* sOl = reinterpret_cast<const __nv_bfloat16*>(stage0 + (size_t)(i % UNST) * stage_bytes + UR::OL_OFF);
                const float* sOTc = sOT + (i & 1) * (2 * 64 * 64);
                out_sync(UNB_OFULL + (i & 1));
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if ((unsigned long long)orow[q] >= (unsigned long long)a.total_tokens) continue;
                    const int tk = tok + 16 * q;
                    const size_t idx = ((size_t)orow[q] * H + h) * UVD + col;
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const float4 p0 = *reinterpret_cast<const float4*>(sOTc + (0 * 64 + tk) * 64 + col + 32 * x);
                        const float4 q0 = *reinterpret_cast<const float4*>(sOTc + (1 * 64 + tk) * 64 + col + 32 * x);
                        const uint2 ol = *reinterpret_cast<const uint2*>(sOl + UR::TV::off(tk, col + 32 * x));      // 4 bf16 of O_local
                        const float2 oa = unpack_bf16x2(ol.x), ob = unpack_bf16x2(ol.y);
                        const float r0 = p0.x + q0.x + oa.x, r1 = p0.y + q0.y + oa.y, r2 = p0.z + q0.z + ob.x, r3 = p0.w + q0.w + ob.y;
                        if (a.qkv_dt == LAMPA_F32) {
                            *reinterpret_cast<float4*>((float*)a.o + idx + 32 * x) = make_float4(r0, r1, r2, r3);
                        } else {
                            uint2 w;
                            if (a.qkv_dt == LAMPA_BF16) { w.x = pack_bf16x2(r0, r1); w.y = pack_bf16x2(r2, r3); }
                            else {
                                const __half2 ha = __floats2half2_rn(r0, r1), hb = __floats2half2_rn(r2, r3);
                                w.x = *reinterpret_cast<const uint32_t*>(&ha); w.y = *reinterpret_cast<const uint32_t*>(&hb);
                            }
                            *reinterpret_cast<uint2*>((uint16_t*)a.o + idx + 32 * x) = w;
                        }
                    }
                }
                if (i + 2 < nsteps) out_arrive(UNB_OFREE + (i & 1));      // nobody waits for the last two
                __syncwarp();
                if (lane == 0) mbar_arrive(sfree + (i % UNST));           // O_local of this stage has been read
            }
        };
        if (a.out_perm_rows > 0) drain_tiles(ScatterOn{}); else drain_tiles(ScatterOff{});
    } else {
        // ---- epilogue warps: every warp advances 16 state columns and reads 16 tokens of its 32 rows ----
        // The loop over pairs is unrolled: barrier ids, bit positions and operand columns are constants in it.
        // per pair, the lambda row of this thread's slot, and the slots that exist and have a lambda row
        uint32_t lam_pack = 0, slot_ok = 0;          // 5 bits per pair: the lambda row of slot 2p + u
#pragma unroll
        for (int p = 0; p < UNP; ++p) {
            const int s = 2 * p + u;
            const int row = s < bl ? s : bl + (int)((live_pack >> (4 * max(s - bl, 0))) & 15);
            lam_pack |= (uint32_t)(row & 31) << (5 * p);
        }
        for (int s = 0; s < nslots; ++s) {
            const int row = s < bl ? s : bl + (int)((live_pack >> (4 * (s - bl))) & 15);
            if (row < a.LC) slot_ok |= 1u << s;      // a missing row is only reachable when the level check already failed
        }
        const uint32_t tpart = tlane + (uint32_t)(tm_d + 16 * part);
        uint32_t buf = 0;                            // first column of the next pair's accumulator, in step with the control warp
        for (int i = 0; i < nsteps; ++i) {
            const unsigned char* st = stage0 + (size_t)(i % UNST) * stage_bytes;
            const float* sLam = reinterpret_cast<const float*>(st + STAGE_TILES) + 16 * part;
            const unsigned char* sBt = st + UR::BT_OFF;
            const int n = b * bc + i;
            // what this chunk does to each slot, as bit masks of this thread's slots (bit 2p = slot 2p + u): in-block level
            // s is read when bit s of n is set, collects when it is not, and is cleared when its period of 2^(s+1) chunks
            // ends (all of bits 0..s set); the cross-block slots are read by every chunk
            const uint32_t low = (uint32_t)n & (bc - 1);
            const uint32_t read_mask = ((low | (~0u << bl)) & slot_ok) >> u;
            const uint32_t clear_mask = (low & ~(low + 1u) & (bc - 1)) >> u;      // trailing ones of n
            const uint32_t add_mask = (~low & (bc - 1)) >> u;
            const uint32_t step_mask = i + 1 < nsteps ? ((1u << nslots) - 1u) >> u : 0u;   // the last chunk leaves no state
            uint4 bq0, bq1;                            // this row's 16 columns of B^T, shared by every level that collects in this chunk

            F2 oacc[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) oacc[j].v = 0ull;

#pragma unroll
            for (int p = 0; p < UNP; ++p) {
                if (p >= npairs) continue;
                named_sync(UNB_PAIR + p);              // pair's MMA complete
                tc_fence_after();
                const uint32_t lockstep = *sdead;      // non-zero: a wait ran out somewhere, nobody runs ahead of anybody from here on
                if (p == 0) {                          // the record has landed too
                    bq0 = *reinterpret_cast<const uint4*>(sBt + v * 128 + (((2 * part) ^ (v & 7)) << 4));
                    bq1 = *reinterpret_cast<const uint4*>(sBt + v * 128 + (((2 * part + 1) ^ (v & 7)) << 4));
                }
                const uint32_t tcol = tpart + buf;
                buf = buf == (uint32_t)(nbuf - 1) * 128u ? 0u : buf + 128u;
                // state path first: the next chunk's MMA of this pair waits for it
                if ((step_mask >> (2 * p)) & 1u) {
                    uint32_t w[8];
                    if ((clear_mask >> (2 * p)) & 1u) {
#pragma unroll
                        for (int c = 0; c < 8; ++c) w[c] = 0u;
                    } else {
                        float x[16];
                        tmem_ld16(x, tcol);
                        if ((add_mask >> (2 * p)) & 1u) {
                            const uint32_t bw[8] = {bq0.x, bq0.y, bq0.z, bq0.w, bq1.x, bq1.y, bq1.z, bq1.w};
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                const float2 f = unpack_bf16x2(bw[c]);
                                f2_get(add2(f2(x[2 * c], x[2 * c + 1]), f2(f.x, f.y)), x[2 * c], x[2 * c + 1]);
                            }
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c) w[c] = pack_bf16x2(x[2 * c], x[2 * c + 1]);
                    }
                    tmem_st8(tlane + TM_A + 32 * p + 8 * part, w);
                }
                // read path: lambda-weighted contribution of this level to 16 tokens
                if ((read_mask >> (2 * p)) & 1u) {
                    float y[16];
                    tmem_ld16(y, tcol + 64);
                    const float4* lr = reinterpret_cast<const float4*>(sLam + ((lam_pack >> (5 * p)) & 31u) * CHUNK);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 l4 = lr[j];
                        oacc[2 * j] = fma2(f2(l4.x, l4.y), f2(y[4 * j], y[4 * j + 1]), oacc[2 * j]);
                        oacc[2 * j + 1] = fma2(f2(l4.z, l4.w), f2(y[4 * j + 2], y[4 * j + 3]), oacc[2 * j + 1]);
                    }
                }
                tc_fence_before();
                // operand rewritten, accumulator read: the control warp may go on
                if (lockstep) named_sync(UNB_DFREE + p); else named_arrive(UNB_DFREE + p);
            }
            // the output tile, [slot of the pair][token][v], goes to the output warps; its buffer was last read two chunks ago
            float* sOTc = sOT + (i & 1) * (2 * 64 * 64);
            if (i >= 2) out_sync(UNB_OFREE + (i & 1));
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float lo, hi;
                f2_get(oacc[j], lo, hi);
                sOTc[(u * 64 + 16 * part + 2 * j) * 64 + v] = lo;
                sOTc[(u * 64 + 16 * part + 2 * j + 1) * 64 + v] = hi;
            }
            out_arrive(UNB_OFULL + (i & 1));
            __syncwarp();
            if (lane == 0) mbar_arrive(sfree + (i % UNST));   // B^T and lambda of this stage have been read
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(taddr, 512);
}

}  // namespace

int launch_out_hier_umma(const GdnArgs& a, cudaStream_t st) {
    const int smem = SM_STAGE + UNST * ustage_bytes(a.LC);
    if (smem > MAX_SMEM) return LAMPA_ERR_UNSUPPORTED;
    static std::atomic<uint64_t> ready;
    if (!allow_smem(ready, gdn_out_hier_umma_kernel, MAX_SMEM)) return LAMPA_ERR_CUDA;
    UnitOrder uo;
    uo.nbs = 0;
    if (a.fixed_T > 0 && a.nseq > 0 && a.nb_max % a.nseq == 0 && a.nb_max / a.nseq <= 64) {
        uo.nbs = a.nb_max / a.nseq;
        const int bl = block_log(a.fixed_cps);
        int n = 0;
        for (int pairs = UNP; pairs >= 0; --pairs)        // stable: block order kept inside a class
            for (int b = 0; b < uo.nbs; ++b) {
                int live = 0;
                for (int lh = 0; lh < a.nhigh_max; ++lh) live += (b >> lh) & 1;
                if ((bl + live + 1) / 2 == pairs) uo.order[n++] = (unsigned char)b;
            }
        if (n != uo.nbs) uo.nbs = 0;
    }
    ProfScope prof("gdn_out_hier_umma", st);
    launch_chained(gdn_out_hier_umma_kernel, dim3((unsigned)a.nb_max * a.H), UTHREADS, smem, st, a, uo);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

}  // namespace lampa
