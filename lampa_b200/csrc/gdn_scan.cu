// Block-parallel scan of the gated-delta forward over the per-chunk records {M, B^T, Q~, O_local}.
//
// One chunk acts on a state as S <- M S + B and reads it as Q~ S, so a block of 32 chunks acts as
// S <- Mblk S + Bblk.  Three passes replace the reference's single sequential scan over all chunks
// (models/hattention/chunk_delta_h.py:35-189) and its one-scan-per-level loop
// (models/hattention/chunkwise_hgdn.py:723-789):
//   compose : per (block, head)  run [S | P] from [0 | I] through the block -> (Mblk, Bblk)
//   level   : per (sequence, head[, level])  scan the block composites -> state entering each block
//   output  : per (block, head)  re-run the block from its entry state(s) and emit the outputs
// Everything a warp owns is a 16-row slab of S^T kept in mma accumulator registers; the slab is
// re-used as the A operand (S^T M^T) and as the B operand (Q~ S) without leaving registers.
// Records stream through shared memory by bulk async copies (cp.async.bulk + mbarrier), a few
// chunks ahead of the math, issued by a warp of their own.
//
// These passes are serial chains, a product per step whose result is the next one's operand: what
// bounds them is the latency of a step.  The product itself is 373 cycles for a slab of 16 x 64 on
// an otherwise idle scheduler; a __syncthreads, a poll of a completed mbarrier by every warp, and a
// state moved in 8-byte pieces added 60, 170 - 260 and 480 (level pass: 1560 cycles per block).
// Hence one warp polls, the others meet it at a named barrier, and states and composites are laid
// out in the order of the accumulator registers.
#include "gdn.cuh"
#include "profile.cuh"

namespace lampa {

template <int KD>
__device__ __forceinline__ void zero_state(float (&C)[KD / 8][4]) {
#pragma unroll
    for (int i = 0; i < KD / 8; ++i) { C[i][0] = C[i][1] = C[i][2] = C[i][3] = 0.f; }
}

// bf16 fragments of a 16 x KD slab held as mma accumulators; sp[kk] is at once the A fragment of
// k-step kk and, pairwise, the B fragments (sp[kk][0], sp[kk][2]) / (sp[kk][1], sp[kk][3]) of the
// slab's two 8-column halves when the slab is read as S[k][v].
template <int KD>
__device__ __forceinline__ void pack_state(const float (&C)[KD / 8][4], uint32_t (&sp)[KD / 16][4]) {
#pragma unroll
    for (int kk = 0; kk < KD / 16; ++kk) {
        sp[kk][0] = pack_bf16x2(C[2 * kk][0], C[2 * kk][1]);
        sp[kk][1] = pack_bf16x2(C[2 * kk][2], C[2 * kk][3]);
        sp[kk][2] = pack_bf16x2(C[2 * kk + 1][0], C[2 * kk + 1][1]);
        sp[kk][3] = pack_bf16x2(C[2 * kk + 1][2], C[2 * kk + 1][3]);
    }
}

// C += slab * M^T for NX slabs, with the record tile sM[k_out][k_in]
template <int KD, int NX>
__device__ __forceinline__ void state_times_mt(float (&C)[NX][KD / 8][4], const uint32_t (&sp)[NX][KD / 16][4],
                                               const __nv_bfloat16* sM, int lane) {
    const int mi = lane >> 3, r = lane & 7;
#pragma unroll
    for (int kk = 0; kk < KD / 16; ++kk) {
#pragma unroll
        for (int nt = 0; nt < KD / 8; nt += 2) {
            uint32_t b[4];
            ldsm_x4(b, smem_u32(sM + Tile<KD>::off(nt * 8 + r + (mi >> 1) * 8, kk * 16 + (mi & 1) * 8)));
#pragma unroll
            for (int x = 0; x < NX; ++x) {
                mma16816(C[x][nt], sp[x][kk], b[0], b[1]);
                mma16816(C[x][nt + 1], sp[x][kk], b[2], b[3]);
            }
        }
    }
}
template <int KD>
__device__ __forceinline__ void state_times_mt(float (&C)[KD / 8][4], const uint32_t (&sp)[KD / 16][4],
                                               const __nv_bfloat16* sM, int lane) {
    state_times_mt<KD, 1>(reinterpret_cast<float (&)[1][KD / 8][4]>(C), reinterpret_cast<const uint32_t (&)[1][KD / 16][4]>(sp), sM, lane);
}
// The same with a block composite's Mblk, which is stored as the fragments themselves
template <int KD>
__device__ __forceinline__ void state_times_mblk(float (&C)[KD / 8][4], const uint32_t (&sp)[KD / 16][4], const uint4* sM, int lane) {
#pragma unroll
    for (int kk = 0; kk < KD / 16; ++kk) {
#pragma unroll
        for (int np = 0; np < KD / 16; ++np) {
            const uint4 b = sM[(kk * (KD / 16) + np) * 32 + lane];
            mma16816(C[2 * np], sp[kk], b.x, b.y);
            mma16816(C[2 * np + 1], sp[kk], b.z, b.w);
        }
    }
}
// 8 x 8 bf16 tile across the warp, transposed
__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
    return y;
}

// C = rows row0 .. row0 + 15 of a bf16 [rows][KD] record tile
template <int KD>
__device__ __forceinline__ void load_slab_bf16(float (&C)[KD / 8][4], const __nv_bfloat16* s, int row0, int lane) {
    const int mi = lane >> 3, r = lane & 7;
#pragma unroll
    for (int p = 0; p < KD / 16; ++p) {
        uint32_t w[4];
        ldsm_x4(w, smem_u32(s + Tile<KD>::off(row0 + r + (mi & 1) * 8, 16 * p + (mi >> 1) * 8)));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 f = unpack_bf16x2(w[q]);
            C[2 * p + (q >> 1)][2 * (q & 1)] = f.x;
            C[2 * p + (q >> 1)][2 * (q & 1) + 1] = f.y;
        }
    }
}
// slab `slab` of an fp32 state (Rec::state_at) in shared or global memory
template <int KD, bool GLOBAL = false>
__device__ __forceinline__ void load_slab_f32(float (&C)[KD / 8][4], const float* s, int slab, int lane) {
    const float4* p4 = reinterpret_cast<const float4*>(s) + slab * (KD / 8) * 32 + lane;
#pragma unroll
    for (int p = 0; p < KD / 16; ++p)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const float4 f = GLOBAL ? __ldcg(p4 + (2 * p + hh) * 32) : p4[(2 * p + hh) * 32];
            C[2 * p][2 * hh] = f.x; C[2 * p][2 * hh + 1] = f.y; C[2 * p + 1][2 * hh] = f.z; C[2 * p + 1][2 * hh + 1] = f.w;
        }
}
template <int KD>
__device__ __forceinline__ void store_slab_f32(const float (&C)[KD / 8][4], float* s, int slab, int lane) {
    float4* p4 = reinterpret_cast<float4*>(s) + slab * (KD / 8) * 32 + lane;
#pragma unroll
    for (int p = 0; p < KD / 16; ++p)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
            p4[(2 * p + hh) * 32] = make_float4(C[2 * p][2 * hh], C[2 * p][2 * hh + 1], C[2 * p + 1][2 * hh], C[2 * p + 1][2 * hh + 1]);
}

// tmp[x] (16 tokens x 16 state columns of this slab) = Q~[16 (mt + x) .. +16, :] * S for NM row tiles: 2 NM independent chains
// of KD / 16 dependent products
template <int KD, int NM>
__device__ __forceinline__ void read_tiles(float (&tmp)[NM][2][4], const uint32_t (&sp)[KD / 16][4],
                                           const __nv_bfloat16* sQt, int mt, int lane) {
    const int mi = lane >> 3, r = lane & 7;
#pragma unroll
    for (int x = 0; x < NM; ++x)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) { tmp[x][nt][0] = tmp[x][nt][1] = tmp[x][nt][2] = tmp[x][nt][3] = 0.f; }
#pragma unroll
    for (int kk = 0; kk < KD / 16; ++kk)
#pragma unroll
        for (int x = 0; x < NM; ++x) {
            uint32_t a[4];
            ldsm_x4(a, smem_u32(sQt + Tile<KD>::off((mt + x) * 16 + r + (mi & 1) * 8, kk * 16 + (mi >> 1) * 8)));
            mma16816(tmp[x][0], a, sp[kk][0], sp[kk][2]);
            mma16816(tmp[x][1], a, sp[kk][1], sp[kk][3]);
        }
}

// o (a row tile's 8 columns) += a level's term: its weights for the rows g and g + 8 of the tile, and Q~ S.  One rounding per level, in
// the order of the levels, in every kernel that adds them: a sequence's outputs do not depend on which one it meets.
__device__ __forceinline__ void add_level(float (&o)[4], float l0, float l1, float x, float y, float z, float w) {
    o[0] = __fmaf_rn(l0, x, o[0]); o[1] = __fmaf_rn(l0, y, o[1]);
    o[2] = __fmaf_rn(l1, z, o[2]); o[3] = __fmaf_rn(l1, w, o[3]);
}

// ---- record pipeline: thread 0 issues bulk copies NST-1 steps ahead; everyone waits on the
// stage's mbarrier.  The __syncthreads at the top of a step frees the stage consumed last step.
template <int NST>
struct Pipe {
    uint64_t* bar;
    unsigned char* stage;
    int stage_bytes;     // distance between stages in shared memory
    const char* src;     // record of step 0
    size_t src_stride;   // bytes between consecutive steps' records
    uint32_t copy_bytes;
    int nsteps;
    bool dead;
    int32_t* status;
    int budget;          // polls per wait
    int issued, landed;  // thread 0: copies started / copies seen complete

    __device__ __forceinline__ void issue(int step) {
        uint64_t* b = bar + (step % NST);
        mbar_expect_tx(b, copy_bytes);
        bulk_g2s(stage + (size_t)(step % NST) * stage_bytes, src + (size_t)step * src_stride, copy_bytes, b);
        issued = step + 1;
    }
    __device__ __forceinline__ void start() {
        issued = landed = 0;
        if (threadIdx.x == 0) {
            for (int s = 0; s < NST; ++s) mbar_init(bar + s, 1);
            fence_mbar_init();
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int s = 0; s < NST - 1 && s < nsteps; ++s) issue(s);
    }
    // returns the stage holding step i
    __device__ __forceinline__ const unsigned char* acquire(int i) {
        __syncthreads();
        if (threadIdx.x == 0 && !dead && i + NST - 1 < nsteps) issue(i + NST - 1);
        if (mbar_wait(bar + (i % NST), (uint32_t)((i / NST) & 1), dead, status, 100 + (i & 0xffff), budget) && threadIdx.x == 0)
            landed = i + 1;
        return stage + (size_t)(i % NST) * stage_bytes;
    }
    // Before the CTA exits: copies that were started but never seen complete (only after a wait
    // gave up) must land first, or they would write into shared memory that is no longer ours.
    __device__ __forceinline__ void finish() {
        if (threadIdx.x == 0)
            for (int s = landed; s < issued; ++s) mbar_drain(bar + (s % NST), (uint32_t)((s / NST) & 1));
        __syncthreads();
    }
};

// ---- the same pipeline with a warp of its own for the copies.  Steps come in groups of GRP with one mbarrier, which only that
// warp polls; a group begins with one named barrier of all NT threads, which says that its records have landed and that
// everybody is done with the group before, whose stage is refilled then.  (A poll and a copy cost the warp 170 and 150 - 350
// cycles: with one record to a group that is as long as a short step.)  A wait that runs out is recorded and everybody walks
// on to the end.
// LAG: groups that a stage stays untouched behind its own (1: until everybody has moved on; 2: one group more, for warps that
// follow a step behind).  NT = 0: every thread of the CTA.
template <int NST, int NT, int GRP, int LAG = 1>
struct Feed {
    uint64_t* bar;
    unsigned char* stage;
    int step_bytes;      // distance between steps in shared memory
    const char* src;     // record of step 0
    size_t src_stride;   // bytes between consecutive steps' records
    uint32_t copy_bytes;
    int nsteps;
    int32_t* status;
    int budget;          // polls per wait
    size_t src2;         // a second piece of every record: where it begins in the record, and its bytes (0: none).  It lands
    uint32_t copy2;      // behind the first one in the stage

    static __device__ __forceinline__ void meet() {
        if (NT == 0) asm volatile("bar.sync 1;\n" ::: "memory");
        else asm volatile("bar.sync 1, %0;\n" :: "n"(NT == 0 ? 32 : NT) : "memory");
    }
    __device__ __forceinline__ int groups() const { return (nsteps + GRP - 1) / GRP; }
    __device__ __forceinline__ void issue(int grp) const {                       // the whole warp, a lane to a step
        const int lane = threadIdx.x & 31, step = grp * GRP + lane;
        uint64_t* b = bar + (grp % NST);
        if (lane == 0) mbar_expect_tx(b, (uint32_t)min(GRP, nsteps - step) * (copy_bytes + copy2));
        __syncwarp();
        if (lane < GRP && step < nsteps) {
            unsigned char* dst = stage + (size_t)((grp % NST) * GRP + lane) * step_bytes;
            const char* from = src + (size_t)step * src_stride;
            bulk_g2s(dst, from, copy_bytes, b);
            if (copy2 > 0) bulk_g2s(dst + copy_bytes, from + src2, copy2, b);
        }
    }
    // All threads, before anything else; `producer`: the warp that goes on to produce()
    __device__ __forceinline__ void start(bool producer) const {
        if (!producer) return;
        if ((threadIdx.x & 31) == 0) {
            for (int s = 0; s < NST; ++s) mbar_init(bar + s, 1);
            fence_mbar_init();
        }
        __syncwarp();
        for (int s = 0; s < NST && s < groups(); ++s) issue(s);
    }
    // The producer warp.  `extra`: barriers behind the last step
    __device__ __forceinline__ void produce(int extra = 0) const {
        bool dead = false;
        const int ng = groups();
        int issued = ng < NST ? ng : NST, landed = 0;
        for (int i = 0; i < ng; ++i) {
            if (mbar_wait(bar + (i % NST), (uint32_t)((i / NST) & 1), dead, status, 100 + (i & 0xffff), budget)) landed = i + 1;
            dead = __any_sync(0xffffffffu, dead);
            meet();
            if (!dead && i >= LAG && i - LAG + NST < ng) { issue(i - LAG + NST); issued = i - LAG + NST + 1; }
        }
        for (int i = 0; i < extra; ++i) meet();
        // copies that were started but never seen complete (only after a wait gave up) land before the CTA's memory is given back
        for (int s = landed; s < issued; ++s) mbar_drain(bar + (s % NST), (uint32_t)((s / NST) & 1));
    }
    // Everybody else, at the top of step i: where its record is
    __device__ __forceinline__ const unsigned char* step(int i) const {
        if (GRP == 1 || i % GRP == 0) meet();
        return stage + (size_t)(GRP == 1 ? i % NST : i % (NST * GRP)) * step_bytes;
    }
};

// -------------------------------------------------------------------------------------------------
// compose: (Mblk, Bblk) of one block of chunks.  Slabs 0 .. VD / 16 - 1 run S from zero, the KD / 16 slabs behind them P from
// the identity; SPW slabs to a warp.  A slab's 32 products of a step take 290 cycles of a scheduler and its fragments of M 64
// cycles of the SM's shared-memory pipe, so with one slab to a warp the eight warps of a block spend as long on reading M
// eight times as on the products.  Two slabs to a warp share the fragments (SPLIT = 1).  SPLIT = 2: S and P in CTAs of their
// own, one slab to a warp and one warp to a scheduler: the shortest step, taken while the halves of all blocks come to at most
// two to an SM (12 blocks of 8 chunks, 8 heads: 12.2 -> 10.7 us; 4 heads, one to an SM: 11.3 -> 10.7).
// -------------------------------------------------------------------------------------------------
template <int KD, int VD, int SPLIT>
struct Compose {
    static constexpr int SLABS_S = VD / 16, SLABS_P = KD / 16;
    static constexpr int SPW = SPLIT == 1 && KD == 64 ? 2 : 1;
    static constexpr int SLABS = SPLIT == 1 ? SLABS_S + SLABS_P : (SLABS_S > SLABS_P ? SLABS_S : SLABS_P);
    static constexpr int NW = SLABS / SPW;
    static constexpr int GRP = 1, NST = 3;       // 49 KB of M and B^T at K = V = 64; registers leave room for three CTAs to an SM
    static_assert(SLABS % SPW == 0 && SLABS_S % SPW == 0, "a warp's slabs are of one kind");
};

template <int KD, int VD, int SPLIT>
__global__ void __launch_bounds__(Compose<KD, VD, SPLIT>::NW * 32 + 32) gdn_compose_kernel(GdnArgs a) {
    if (chain_wait()) return;
    using R = Rec<KD, VD>;
    using G = Compose<KD, VD, SPLIT>;
    constexpr int NW = G::NW, SPW = G::SPW, NS = G::SLABS_S;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int gb = blockIdx.x, h = blockIdx.y;
    SeqLoc sq;
    int b;
    if (!locate_block(a, gb, sq, b)) return;
    const int nch = sq.nch;
    const int bc = 1 << block_log(nch);
    const int c0 = sq.c0 + b * bc;
    const int nsteps = min(bc, nch - b * bc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const bool only_p = SPLIT == 2 && blockIdx.z == 1;

    Feed<G::NST, NW * 32 + 32, G::GRP> feed;
    feed.bar = reinterpret_cast<uint64_t*>(smem);
    feed.stage = smem + 1024;
    feed.step_bytes = R::M_BYTES + R::BT_BYTES;
    feed.src = a.rec + ((size_t)c0 * a.H + h) * a.rec_bytes;
    feed.src_stride = (size_t)a.H * a.rec_bytes;
    feed.copy_bytes = R::M_BYTES;
    feed.src2 = R::BT_OFF;
    feed.copy2 = only_p ? 0 : R::BT_BYTES;
    feed.nsteps = nsteps;
    feed.status = a.status;
    feed.budget = a.poll_budget;
    feed.start(warp == NW);
    if (warp == NW) {
        feed.produce();
        return;
    }
    const int slot = (only_p ? NS : 0) + warp * SPW;
    const bool is_s = slot < NS;
    if (slot >= (SPLIT == 2 && !only_p ? NS : NS + G::SLABS_P)) {      // a half with fewer slabs than warps
        for (int i = 0; i < nsteps; ++i) feed.step(i);
        return;
    }
    const int slab = is_s ? slot : slot - NS;
    float C[SPW][KD / 8][4];
#pragma unroll
    for (int x = 0; x < SPW; ++x) {
        zero_state<KD>(C[x]);
        if (!is_s) {
#pragma unroll
            for (int nt = 0; nt < KD / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (16 * (slab + x) + g + (e >> 1) * 8 == nt * 8 + 2 * t + (e & 1)) C[x][nt][e] = 1.f;
        }
    }
    for (int i = 0; i < nsteps; ++i) {
        const unsigned char* st = feed.step(i);
        const __nv_bfloat16* sM = reinterpret_cast<const __nv_bfloat16*>(st);
        const __nv_bfloat16* sBt = reinterpret_cast<const __nv_bfloat16*>(st + R::M_BYTES);
        uint32_t sp[SPW][KD / 16][4];
#pragma unroll
        for (int x = 0; x < SPW; ++x) {
            pack_state<KD>(C[x], sp[x]);
            if (is_s) load_slab_bf16<KD>(C[x], sBt, 16 * (slab + x), lane);
            else zero_state<KD>(C[x]);
        }
        if (i > 0 || !is_s) state_times_mt<KD, SPW>(C, sp, sM, lane);
    }
    char* blk = a.blk + ((size_t)gb * a.H + h) * R::BLK_BYTES;
#pragma unroll
    for (int x = 0; x < SPW; ++x) {
        if (is_s) {
            store_slab_f32<KD>(C[x], reinterpret_cast<float*>(blk + R::BLK_B_OFF), slab + x, lane);
        } else {
            // registers hold P^T (row = k_in, col = k_out): its 8 x 8 tiles transposed are the fragments the level pass takes
            uint4* gm = reinterpret_cast<uint4*>(blk + R::BLK_M_OFF) + (slab + x) * (KD / 16) * 32 + lane;
#pragma unroll
            for (int q = 0; q < KD / 16; ++q)
                gm[q * 32] = make_uint4(transpose8x8(pack_bf16x2(C[x][2 * q][0], C[x][2 * q][1])), transpose8x8(pack_bf16x2(C[x][2 * q][2], C[x][2 * q][3])),
                                        transpose8x8(pack_bf16x2(C[x][2 * q + 1][0], C[x][2 * q + 1][1])), transpose8x8(pack_bf16x2(C[x][2 * q + 1][2], C[x][2 * q + 1][3])));
        }
    }
}

// -------------------------------------------------------------------------------------------------
// level: scan of the block composites.  Plain rule: one state per (sequence, head), seeded by h0,
// the state entering every block is stored and the last one is the final state.  Hierarchical:
// one CTA per cross-block level lh (chunk level block_log + lh); the level collects blocks whose bit lh is
// 0, is read by blocks whose bit lh is 1 (its entry state is stored for those) and is cleared at
// the end of each period of 2^(lh+1) blocks.
//
// NW slabs of 16 state rows to a CTA.  With all four of a 64 x 64 head in one CTA the shared-memory and store pipes of the SM are
// the longest part of a step (M read four times, the state written: 640 of 1220 cycles); slabs never meet, so where that leaves
// SMs idle every slab gets a CTA.
// -------------------------------------------------------------------------------------------------
template <int KD, int NW>
struct LevelSmem {
    static constexpr int STEP = KD * KD * 2 + NW * 16 * KD * 4;      // Mblk and the slabs' rows of Bblk^T
    static constexpr int NST = KD == 64 ? 4 : 3, GRP = KD < 64 ? 4 : (NW == 1 ? 2 : 1);
    static constexpr int bytes = 1024 + NST * GRP * STEP;            // 99 KB at K = V = 64, either way: two CTAs to an SM
};

template <int KD, int VD, bool HIER, int NW>
__global__ void __launch_bounds__(NW * 32 + 32) gdn_level_kernel(GdnArgs a) {
    if (chain_wait()) return;
    using R = Rec<KD, VD>;
    using S = LevelSmem<KD, NW>;
    constexpr int PARTS = VD / 16 / NW;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int seq = blockIdx.x, h = blockIdx.y, lh = blockIdx.z / PARTS, H = a.H;
    const SeqLoc sq = locate_seq(a, seq);
    const int nblk = sq.nblk, gb0 = sq.gb0;
    if (HIER) {
        const int nch = sq.nch;
        const int nlev = nch > 1 ? ceil_log2_int(nch) : 0;
        if (lh >= nlev - block_log(nch)) return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int slab0 = (blockIdx.z - lh * PARTS) * NW, slab = slab0 + warp, row0 = slab * 16;

    Feed<S::NST, NW * 32 + 32, S::GRP> feed;
    feed.bar = reinterpret_cast<uint64_t*>(smem);
    feed.stage = smem + 1024;
    feed.step_bytes = S::STEP;
    feed.src = a.blk + ((size_t)gb0 * H + h) * R::BLK_BYTES;
    feed.src_stride = (size_t)H * R::BLK_BYTES;
    feed.copy_bytes = PARTS == 1 ? R::BLK_BYTES : R::BLK_M_BYTES;
    feed.src2 = R::BLK_B_OFF + (size_t)slab0 * 16 * KD * 4;
    feed.copy2 = PARTS == 1 ? 0 : NW * 16 * KD * 4;
    feed.nsteps = nblk;
    feed.status = a.status;
    feed.budget = a.poll_budget;
    feed.start(warp == NW);
    if (warp == NW) {
        feed.produce();
        return;
    }

    float C[KD / 8][4];
    zero_state<KD>(C);
    bool nonzero = false;
    if (!HIER && a.h0 != nullptr) {
        const float* h0 = a.h0 + ((size_t)seq * H + h) * KD * VD;   // [K][V]
#pragma unroll
        for (int nt = 0; nt < KD / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                C[nt][e] = h0[(size_t)(nt * 8 + 2 * t + (e & 1)) * VD + row0 + g + (e >> 1) * 8];
        nonzero = true;
    }
    for (int b = 0; b < nblk; ++b) {
        const unsigned char* st = feed.step(b);
        const uint4* sM = reinterpret_cast<const uint4*>(st);
        const float* sB = reinterpret_cast<const float*>(st + R::BLK_M_BYTES);
        uint32_t sp[KD / 16][4];
        if (!HIER) {
            store_slab_f32<KD>(C, a.entry + ((size_t)(gb0 + b) * H + h) * R::STATE_FLOATS, slab, lane);
            pack_state<KD>(C, sp);
            load_slab_f32<KD>(C, sB, warp, lane);
            if (nonzero) state_times_mblk<KD>(C, sp, sM, lane);
            nonzero = true;
        } else {
            const int period = 2 << lh, pos = b & (period - 1), bit = (b >> lh) & 1;
            if (bit) store_slab_f32<KD>(C, a.entry + (((size_t)(gb0 + b) * a.nhigh_max + lh) * H + h) * R::STATE_FLOATS, slab, lane);
            if (pos == period - 1) {
                zero_state<KD>(C);
            } else {
                pack_state<KD>(C, sp);
                if (bit == 0) load_slab_f32<KD>(C, sB, warp, lane);
                else zero_state<KD>(C);
                if (pos != 0) state_times_mblk<KD>(C, sp, sM, lane);
            }
        }
    }
    if (!HIER && a.ht != nullptr) {
        float* ht = a.ht + ((size_t)seq * H + h) * KD * VD;
#pragma unroll
        for (int nt = 0; nt < KD / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                ht[(size_t)(nt * 8 + 2 * t + (e & 1)) * VD + row0 + g + (e >> 1) * 8] = C[nt][e];
    }
}

// -------------------------------------------------------------------------------------------------
// final state, hierarchical rule, chunk levels.  After a sequence of NT chunks the Fenwick state
// holds chunk level l (lambda index 7 + l) exactly when bit l of NT - 1 is set: the first half of
// the level's current period, carried through every chunk up to the last one without the closing
// reset (the reference's hattention_prefill keeps the same thing, models/hattention/kernel.py:
// 377-470 and chunkwise_hgdn.py:738-739).  One CTA per (sequence, head, level) re-runs at most one
// block of chunks over the records the forward left in the workspace: levels inside a block start
// from zero at the period's first chunk, cross-block levels start from the entry state the level
// pass stored for the last block.  states is [N][H][K][V][L] fp32; unoccupied levels are zeroed.
// -------------------------------------------------------------------------------------------------
template <int KD, int VD>
__global__ void __launch_bounds__(VD * 2 + 32) hgdn_final_high_kernel(GdnArgs a, float* states) {
    // In a prefill the output pass in front lets this one in at its start: it needs nothing of that pass, only what was complete
    // before it (chain_seen), so it runs beside it and signals in turn.  One CTA waits at its end, which keeps the grid's end behind that pass's;
    // the others give their SMs to the prompt's tail.
    if (a.signal) {
        chain_signal();
        if (!chain_seen(a.signal_word, a.signal) && chain_wait()) return;
    } else if (chain_wait()) {
        return;
    }
    using R = Rec<KD, VD>;
    constexpr int NST = 3, NW = VD / 16;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int seq = blockIdx.x, h = blockIdx.y, lev = blockIdx.z, H = a.H;
    const SeqLoc sq = locate_seq(a, seq);
    const int nch = sq.nch;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int row0 = warp * 16;
    const int n = nch - 1, bl = block_log(nch);
    const bool live = nch > 0 && lev < 30 && ((n >> lev) & 1) && lev - bl < a.nhigh_max;

    float C[KD / 8][4];
    zero_state<KD>(C);
    if (live) {
        const int c_first = lev < bl ? n & ~((2 << lev) - 1) : (n >> bl) << bl;
        const int half_end = lev < bl ? c_first + (1 << lev) : c_first;
        Feed<NST, NW * 32 + 32, 1> feed;
        feed.bar = reinterpret_cast<uint64_t*>(smem);
        feed.stage = smem + 1024;
        feed.step_bytes = R::M_BYTES + R::BT_BYTES;
        feed.src = a.rec + ((size_t)(sq.c0 + c_first) * H + h) * a.rec_bytes;
        feed.src_stride = (size_t)H * a.rec_bytes;
        feed.copy_bytes = R::M_BYTES;
        feed.src2 = R::BT_OFF;
        feed.nsteps = n - c_first + 1;
        feed.status = a.status;
        feed.budget = a.poll_budget;
        feed.copy2 = R::BT_BYTES;
        feed.start(warp == NW);
        if (warp == NW) {
            feed.produce();
            return;
        }
        if (lev >= bl) {
            const int gb = sq.gb0 + (n >> bl);
            load_slab_f32<KD, true>(C, a.entry + (((size_t)gb * a.nhigh_max + (lev - bl)) * H + h) * R::STATE_FLOATS, warp, lane);
        }
        for (int i = 0; i < feed.nsteps; ++i) {
            const unsigned char* st = feed.step(i);
            const __nv_bfloat16* sM = reinterpret_cast<const __nv_bfloat16*>(st);
            const __nv_bfloat16* sBt = reinterpret_cast<const __nv_bfloat16*>(st + R::M_BYTES);
            // the state enters the tensor core as bf16 hi + bf16 lo (two products), so that re-rounding
            // it at every chunk does not accumulate in the state handed to the caller
            uint32_t sp[KD / 16][4], sl[KD / 16][4];
            pack_state<KD>(C, sp);
#pragma unroll
            for (int kk = 0; kk < KD / 16; ++kk)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 hi = unpack_bf16x2(sp[kk][e]);
                    const int nt = 2 * kk + (e >> 1), c0 = (e & 1) * 2;
                    sl[kk][e] = pack_bf16x2(C[nt][c0] - hi.x, C[nt][c0 + 1] - hi.y);
                }
            if (c_first + i < half_end) load_slab_bf16<KD>(C, sBt, row0, lane);
            else zero_state<KD>(C);
            if (i > 0 || lev >= bl) {
                state_times_mt<KD>(C, sp, sM, lane);
                state_times_mt<KD>(C, sl, sM, lane);
            }
        }
    }
    if (warp == NW) return;
    if (a.signal && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && chain_wait()) return;
    float* dst = states + ((size_t)seq * H + h) * KD * VD * a.L + ELL0 + lev;
#pragma unroll
    for (int nt = 0; nt < KD / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int kk = nt * 8 + 2 * t + (e & 1), vv = row0 + g + (e >> 1) * 8;
            dst[((size_t)kk * VD + vv) * a.L] = C[nt][e];
        }
}

// -------------------------------------------------------------------------------------------------
// output, plain rule:  O_n = O_local + Q~ S_n ;  S_{n+1} = M S_n + B
// VD / 16 slab warps, the copying warp, and one that stores: a chunk's output goes through a [token][v] tile in shared memory
// and leaves as whole rows, under the next chunk's products.  (fp32 outputs go straight from the registers.)
// Bound by streaming the records where the blocks fill the GPU (65,536 tokens, 8 heads: 56 us for 317 MB, 5.7 TB/s of the
// measured 6.5), by the step of a block elsewhere: about 1000 cycles, 64 products of a warp among them.  The same pass on
// tcgen05 (state in tensor memory, an epilogue of 16 warps around one MMA per chunk) needs two hand-overs per chunk and
// took 2800 cycles: 18.8 us against 14.7 at 6,144 tokens and 4 heads, 60.4 against 59.9 at 65,536 and 8.
// -------------------------------------------------------------------------------------------------
template <int KD, int VD>
struct OutPlainSmem {
    static constexpr int NST = 3;
    static constexpr int PITCH = VD * 2 + 16;            // output tile: 16-byte pieces, a row's pairs in banks of their own
    static constexpr int TILE = 1024, STAGE = TILE + (CHUNK * PITCH + 1023) / 1024 * 1024;
    static constexpr int bytes = STAGE + NST * Rec<KD, VD>::LAM_OFF;
};

template <int KD, int VD>
__global__ void __launch_bounds__(VD * 2 + 64) gdn_out_plain_kernel(GdnArgs a) {
    if (chain_wait()) return;
    using R = Rec<KD, VD>;
    using S = OutPlainSmem<KD, VD>;
    constexpr int NST = S::NST, NW = VD / 16;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int gb = blockIdx.x, h = blockIdx.y, H = a.H;
    SeqLoc sq;
    int b;
    if (!locate_block(a, gb, sq, b)) return;
    const int nch = sq.nch;
    const int bc = 1 << block_log(nch);
    const int c0 = sq.c0 + b * bc;
    const int nsteps = min(bc, nch - b * bc);
    const int64_t tok0 = sq.tok0 + (int64_t)b * bc * CHUNK, tok_end = sq.tok_end;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int row0 = warp * 16;
    const bool direct = a.qkv_dt == LAMPA_F32;
    unsigned char* tile = smem + S::TILE;

    Feed<NST, NW * 32 + 64, 1> feed;
    feed.bar = reinterpret_cast<uint64_t*>(smem);
    feed.stage = smem + S::STAGE;
    feed.step_bytes = R::LAM_OFF;
    feed.src = a.rec + ((size_t)c0 * H + h) * a.rec_bytes;
    feed.src_stride = (size_t)H * a.rec_bytes;
    feed.copy_bytes = R::LAM_OFF;
    feed.nsteps = nsteps;
    feed.status = a.status;
    feed.budget = a.poll_budget;
    feed.copy2 = 0;
    feed.start(warp == NW);
    auto tile_free = [] { asm volatile("bar.sync 2, %0;\n" :: "n"(NW * 32 + 32) : "memory"); };      // slab warps, joined by the storing warp
    if (warp == NW) {
        feed.produce(1);
        return;
    }
    if (warp == NW + 1) {
        for (int i = 0; i <= nsteps; ++i) {
            feed.step(i);                              // tile i - 1 is written
            if (i == 0) continue;
            if (!direct) {
                const int64_t t0 = tok0 + (int64_t)(i - 1) * CHUNK;
                constexpr int LPR = VD / 8;                // lanes to a token's row
#pragma unroll
                for (int r = 0; r < CHUNK; r += 32 / LPR) {
                    const int tk = r + lane / LPR, c = lane % LPR;
                    const uint4 w = *reinterpret_cast<const uint4*>(tile + tk * S::PITCH + 16 * c);
                    if (t0 + tk < tok_end) *reinterpret_cast<uint4*>((uint16_t*)a.o + ((size_t)(t0 + tk) * H + h) * VD + 8 * c) = w;
                }
                __syncwarp();
            }
            if (i < nsteps) asm volatile("bar.arrive 2, %0;\n" :: "n"(NW * 32 + 32) : "memory");
        }
        return;
    }
    float C[KD / 8][4];
    load_slab_f32<KD, true>(C, a.entry + ((size_t)gb * H + h) * R::STATE_FLOATS, warp, lane);
    for (int i = 0; i < nsteps; ++i) {
        const unsigned char* st = feed.step(i);
        const __nv_bfloat16* sM = reinterpret_cast<const __nv_bfloat16*>(st + R::M_OFF);
        const __nv_bfloat16* sBt = reinterpret_cast<const __nv_bfloat16*>(st + R::BT_OFF);
        const __nv_bfloat16* sQt = reinterpret_cast<const __nv_bfloat16*>(st + R::QT_OFF);
        const __nv_bfloat16* sOl = reinterpret_cast<const __nv_bfloat16*>(st + R::OL_OFF);
        uint32_t sp[KD / 16][4];
        pack_state<KD>(C, sp);
        if (i + 1 < nsteps) {                          // the state first: the next step waits for it
            load_slab_bf16<KD>(C, sBt, row0, lane);
            state_times_mt<KD>(C, sp, sM, lane);
        }
        float o[4][2][4];
        read_tiles<KD, 4>(o, sp, sQt, 0, lane);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const float2 ol = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(sOl + R::TV::off(mt * 16 + g + hh * 8, row0 + nt * 8 + 2 * t)));
                    o[mt][nt][2 * hh] += ol.x;
                    o[mt][nt][2 * hh + 1] += ol.y;
                }
        if (i > 0) tile_free();
        const int64_t t0 = tok0 + (int64_t)i * CHUNK;
        auto emit = [&](auto put) {
#pragma unroll
            for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) put(mt * 16 + g + hh * 8, row0 + nt * 8 + 2 * t, o[mt][nt][2 * hh], o[mt][nt][2 * hh + 1]);
        };
        if (a.qkv_dt == LAMPA_BF16) {
            emit([&](int r, int col, float x, float y) { *reinterpret_cast<uint32_t*>(tile + r * S::PITCH + 2 * col) = pack_bf16x2(x, y); });
        } else if (!direct) {
            emit([&](int r, int col, float x, float y) { *reinterpret_cast<__half2*>(tile + r * S::PITCH + 2 * col) = __floats2half2_rn(x, y); });
        } else {
            emit([&](int r, int col, float x, float y) {
                if (t0 + r < tok_end) *reinterpret_cast<float2*>((float*)a.o + ((size_t)(t0 + r) * H + h) * VD + col) = make_float2(x, y);
            });
        }
    }
    feed.step(nsteps);
}

// -------------------------------------------------------------------------------------------------
// output, hierarchical rule.  Warp = (level group, slab).  Group 0 carries the chunk levels that
// live and die inside the block (0 .. block_log - 1); group gi >= 1 carries cross-block levels 5*(gi-1) .. +4, seeded
// from the level pass.  A level is read by chunk n when bit l of n is set:
//     O_n += diag(lambda[:, 7 + l]) (Q~ S_l)
// and then advances: cleared at the end of its period of 2^(l+1) chunks, otherwise
//     S_l <- M S_l + [bit l of n == 0] B.
// Partial outputs of groups >= 1 are added by group 0 through shared memory, in blocks that read any.
//
// Bound by the chain of one chunk's products and their shared-memory loads, so warps in flight decide:
// at head dims up to 32 the registers are held to 168 for 12 warps per SM, whatever the split into groups
// (3 spilled words).  16 warps (128 registers, two stages) spill and are slower, 1440 us.  One model block over
// 64 events of 6,000 to 59,000 points: 2003 us with the registers unbounded and a group for every level of
// the whole batch's length -> 968 us with this bound, the level count of L, and no sum over absent groups.
// -------------------------------------------------------------------------------------------------
constexpr int HIER_TILES = 4;

template <int KD, int VD, int NG>
__global__ void __launch_bounds__(NG * VD * 2, KD == 64 ? 1 : 6 / NG) gdn_out_hier_kernel(GdnArgs a) {
    if (chain_wait()) return;
    if (a.signal) chain_signal(a.signal_word, a.signal);
    using R = Rec<KD, VD>;
    constexpr int NST = 3;
    constexpr int NS = VD / 16;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int gb = blockIdx.x, h = blockIdx.y, H = a.H;
    SeqLoc sq;
    int b;
    if (!locate_block(a, gb, sq, b)) return;
    const int nch = sq.nch;
    const int nlev = nch > 1 ? ceil_log2_int(nch) : 0;
    if (a.long_only && nlev <= UMMA_LEVELS) return;
    const int bl = block_log(nch), bc = 1 << bl;
    const int nhigh = min(max(0, nlev - bl), a.nhigh_max);     // more only when the level check has already failed
    const int c0 = sq.c0 + b * bc;
    const int nsteps = min(bc, nch - b * bc);
    const int64_t tok0 = sq.tok0 + (int64_t)b * bc * CHUNK, tok_end = sq.tok_end;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int grp = warp / NS, slab = warp - grp * NS;
    const int row0 = slab * 16;
    const int rec_copy = R::bytes(a.LC);
    const int stage_bytes = (rec_copy + 1023) / 1024 * 1024;

    Pipe<NST> pipe;
    pipe.bar = reinterpret_cast<uint64_t*>(smem);
    pipe.stage = smem + 1024;
    pipe.stage_bytes = stage_bytes;
    pipe.src = a.rec + ((size_t)c0 * H + h) * a.rec_bytes;
    pipe.src_stride = (size_t)H * a.rec_bytes;
    pipe.copy_bytes = (uint32_t)rec_copy;
    pipe.nsteps = nsteps;
    pipe.dead = false;
    pipe.status = a.status;
    pipe.budget = a.poll_budget;
    float* red = reinterpret_cast<float*>(smem + 1024 + (size_t)NST * stage_bytes);   // [NG-1][NS][32 regs][32 lanes]
    pipe.start();

    // groups of cross-block levels this block reads at all: the others have nothing to add to the sum over groups
    uint32_t groups = 0;
#pragma unroll
    for (int gi = 1; gi < NG; ++gi)
        if ((b & ((1 << min(nhigh, 30)) - 1)) >> ((gi - 1) * NLW) & ((1 << NLW) - 1)) groups |= 1u << gi;
    const bool alone = groups == 0;                    // group 0 only: no second barrier per chunk

    float C[NLW][KD / 8][4];
    uint32_t live = 0;   // bit x: level x of this warp holds a state that matters
#pragma unroll
    for (int x = 0; x < NLW; ++x) zero_state<KD>(C[x]);
    if (grp > 0) {
#pragma unroll
        for (int x = 0; x < NLW; ++x) {
            const int lh = (grp - 1) * NLW + x;
            if (lh < nhigh && ((b >> lh) & 1)) {
                live |= 1u << x;
                load_slab_f32<KD, true>(C[x], a.entry + (((size_t)gb * a.nhigh_max + lh) * H + h) * R::STATE_FLOATS, slab, lane);
            }
        }
    }

    for (int i = 0; i < nsteps; ++i) {
        const unsigned char* st = pipe.acquire(i);
        const __nv_bfloat16* sM = reinterpret_cast<const __nv_bfloat16*>(st + R::M_OFF);
        const __nv_bfloat16* sBt = reinterpret_cast<const __nv_bfloat16*>(st + R::BT_OFF);
        const __nv_bfloat16* sQt = reinterpret_cast<const __nv_bfloat16*>(st + R::QT_OFF);
        const __nv_bfloat16* sOl = reinterpret_cast<const __nv_bfloat16*>(st + R::OL_OFF);
        const float* sLam = reinterpret_cast<const float*>(st + R::LAM_OFF);
        const int n = b * bc + i;

        float O[4][2][4];
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) { O[mt][nt][0] = O[mt][nt][1] = O[mt][nt][2] = O[mt][nt][3] = 0.f; }

#pragma unroll
        for (int x = 0; x < NLW; ++x) {
            bool do_read, do_mma, add_b, clear;
            int lam_row;
            if (grp == 0 && x >= bl) continue;      // smaller blocks carry fewer levels of their own
            if (grp == 0) {
                const int per = 2 << x, pos = n & (per - 1), bit = (n >> x) & 1;
                do_read = bit != 0;
                clear = pos == per - 1;
                add_b = bit == 0;
                do_mma = !clear && pos != 0;
                lam_row = x;
            } else {
                const bool lv = (live >> x) & 1u;
                do_read = lv;
                clear = false;
                add_b = false;
                do_mma = lv && (i + 1 < nsteps);
                lam_row = bl + (grp - 1) * NLW + x;
            }
            if (lam_row >= a.LC) do_read = false;   // only reachable when the level check already failed
            uint32_t sp[KD / 16][4];
            if (do_read || do_mma) pack_state<KD>(C[x], sp);
            if (do_read) {
                const float* lr = sLam + lam_row * CHUNK;
#pragma unroll
                for (int m2 = 0; m2 < 4; m2 += HIER_TILES) {
                    float tmp[HIER_TILES][2][4];
                    read_tiles<KD, HIER_TILES>(tmp, sp, sQt, m2, lane);
#pragma unroll
                    for (int x = 0; x < HIER_TILES; ++x) {
                        const int mt = m2 + x;
                        const float l0 = lr[mt * 16 + g], l1 = lr[mt * 16 + g + 8];
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt) add_level(O[mt][nt], l0, l1, tmp[x][nt][0], tmp[x][nt][1], tmp[x][nt][2], tmp[x][nt][3]);
                    }
                }
            }
            if (grp == 0) {
                if (clear) {
                    zero_state<KD>(C[x]);
                } else {
                    if (add_b) load_slab_bf16<KD>(C[x], sBt, row0, lane);
                    else zero_state<KD>(C[x]);
                    if (do_mma) state_times_mt<KD>(C[x], sp, sM, lane);
                }
            } else if (do_mma) {
                zero_state<KD>(C[x]);
                state_times_mt<KD>(C[x], sp, sM, lane);
            }
        }

        if (NG > 1 && !alone) {
            if ((groups >> grp) & 1) {
                float* rd = red + ((size_t)(grp - 1) * NS + slab) * 1024 + lane;
#pragma unroll
                for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) rd[((mt * 2 + nt) * 4 + e) * 32] = O[mt][nt][e];
            }
            __syncthreads();
        }
        if (grp == 0) {
#pragma unroll
            for (int gi = 1; gi < NG; ++gi) {
                if (!((groups >> gi) & 1)) continue;
                const float* rd = red + ((size_t)(gi - 1) * NS + slab) * 1024 + lane;
#pragma unroll
                for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) O[mt][nt][e] += rd[((mt * 2 + nt) * 4 + e) * 32];
            }
            const int64_t t0 = tok0 + (int64_t)i * CHUNK;
            auto emit = [&](auto scat) {
#pragma unroll
                for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const int r = mt * 16 + g + hh * 8;
                        const int64_t orow = t0 + r < tok_end ? out_row<decltype(scat)::value>(a, t0 + r) : -1;
                        if (orow >= 0) {
#pragma unroll
                            for (int nt = 0; nt < 2; ++nt) {
                                const int col = row0 + nt * 8 + 2 * t;
                                const float2 ol = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(sOl + R::TV::off(r, col)));
                                store_out2(a.o, a.qkv_dt, ((size_t)orow * H + h) * VD + col,
                                           ol.x + O[mt][nt][2 * hh], ol.y + O[mt][nt][2 * hh + 1]);
                            }
                        }
                    }
            };
            if (a.out_perm_rows > 0) emit(ScatterOn{}); else emit(ScatterOff{});
        }
    }
    pipe.finish();
}

// -------------------------------------------------------------------------------------------------
// The same for head dims up to 32 with the levels spread over warps: a warp carries two levels of a 16-column slab (level
// slots p and p + pairs of those the block has: its own first, then the cross-block ones it reads), leaves their Q~ S in shared
// memory in its own register order, and eight warps a chunk behind add the terms, in the order of gdn_out_hier_kernel and so with
// its results to the bit, add O_local and store.
// A block's chunk is then two levels deep instead of five, with no barrier but the one at its top.  17 warps and 200 KB, a CTA to an
// SM: taken while the blocks of all heads are at most one to an SM (one event of 9,001 points, 72 CTAs: 25 -> 20 us; two events
// 509 -> 480 us for the whole model; three events, two rounds: 620 against 622; 64 events: 960 against 1270 us a pass).
// -------------------------------------------------------------------------------------------------
constexpr int LV_SUM = 8, LV_MAX_PAIRS = 5, LV_MAX_THREADS = (2 * LV_MAX_PAIRS + 1 + LV_SUM) * 32;

template <int KD, int VD, int STAGES>
struct LevelsSmem {
    static constexpr int NST = STAGES;
    static constexpr int PART = 1024;                        // Q~ S of the levels [2][slots][slabs][8][32 lanes][4], behind the barriers
    static int stage(int LC) { return (Rec<KD, VD>::bytes(LC) + 127) / 128 * 128; }
    static int bytes(int LC, int pairs) { return PART + 2 * 2 * pairs * 2 * 4096 + NST * stage(LC); }
};

template <int KD, int VD, int STAGES>
__global__ void __launch_bounds__(LV_MAX_THREADS) gdn_out_levels_kernel(GdnArgs a, int pairs) {
    if (chain_wait()) return;
    if (a.signal) chain_signal(a.signal_word, a.signal);
    using R = Rec<KD, VD>;
    using S = LevelsSmem<KD, VD, STAGES>;
    constexpr int NS = VD / 16;
    static_assert(NS == 2, "two slabs");
    extern __shared__ __align__(1024) unsigned char smem[];
    const int gb = blockIdx.x, h = blockIdx.y, H = a.H;
    SeqLoc sq;
    int b;
    if (!locate_block(a, gb, sq, b)) return;
    const int nch = sq.nch;
    const int nlev = nch > 1 ? ceil_log2_int(nch) : 0;
    const int bl = block_log(nch), bc = 1 << bl;
    const int nhigh = min(max(0, nlev - bl), a.nhigh_max);     // more only when the level check has already failed
    const int c0 = sq.c0 + b * bc;
    const int nsteps = min(bc, nch - b * bc);
    const int64_t tok0 = sq.tok0 + (int64_t)b * bc * CHUNK, tok_end = sq.tok_end;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    float4* part = reinterpret_cast<float4*>(smem + S::PART);
    const int buf_stride = 2 * pairs * NS * 256;                // float4 of one chunk's terms

    Feed<S::NST, 0, 1, 2> feed;
    feed.bar = reinterpret_cast<uint64_t*>(smem);
    feed.stage = smem + S::PART + 4 * pairs * NS * 4096;
    feed.step_bytes = (R::bytes(a.LC) + 127) / 128 * 128;
    feed.src = a.rec + ((size_t)c0 * H + h) * a.rec_bytes;
    feed.src_stride = (size_t)H * a.rec_bytes;
    feed.copy_bytes = R::bytes(a.LC);
    feed.nsteps = nsteps;
    feed.status = a.status;
    feed.budget = a.poll_budget;
    feed.copy2 = 0;
    const int producer = pairs * NS;
    feed.start(warp == producer);
    if (warp == producer) {
        feed.produce(1);
        return;
    }
    // the block's level slots: its own levels, then the cross-block levels it reads
    const uint32_t cross = (uint32_t)b & ((1u << min(nhigh, 30)) - 1u);
    const int nslots = bl + __popc(cross);
    auto nth_cross = [&](int k) {
        uint32_t m = cross;
        for (int i = 0; i < k; ++i) m &= m - 1;
        return __ffs(m) - 1;
    };
    // slots read in chunk n (a missing lambda row is only reachable when the level check already failed)
    auto read_slot = [&](int s, int lam_row, int n) { return s < nslots && lam_row < a.LC && (s >= bl || ((n >> s) & 1)); };
    if (warp > producer) {
        // ---- sums: warp = (slab, row tile), a chunk behind ----
        const int w = warp - producer - 1, slab = w & 1, mt = w >> 1, row0 = 16 * slab;
        const unsigned char* st = nullptr;
        for (int i = 0; i <= nsteps; ++i) {
            const unsigned char* now = feed.step(i);          // the terms of chunk i - 1 are there
            if (i > 0) {
                const int n = b * bc + i - 1;
                const float4* p0 = part + ((i - 1) & 1) * buf_stride + slab * 256 + mt * 64 + lane;
                const float* lam = reinterpret_cast<const float*>(st + R::LAM_OFF) + mt * 16 + g;
                auto add_slot = [&](float (&x)[2][4], int s, int row) {
                    const float l0 = lam[row * CHUNK], l1 = lam[row * CHUNK + 8];
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        const float4 f = p0[s * NS * 256 + nt * 32];
                        add_level(x[nt], l0, l1, f.x, f.y, f.z, f.w);
                    }
                };
                float o[2][4] = {};
                for (int s = 0; s < bl; ++s)
                    if (read_slot(s, s, n)) add_slot(o, s, s);
                // the cross-block levels by the groups of gdn_out_hier_kernel
                uint32_t m = cross;
                for (int s = bl; m != 0;) {
                    const int grp = (__ffs(m) - 1) / NLW;
                    float oc[2][4] = {};
                    for (; m != 0 && (__ffs(m) - 1) / NLW == grp; m &= m - 1, ++s) {
                        const int row = bl + __ffs(m) - 1;
                        if (read_slot(s, row, n)) add_slot(oc, s, row);
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[e >> 2][e & 3] += oc[e >> 2][e & 3];
                }
                const __nv_bfloat16* sOl = reinterpret_cast<const __nv_bfloat16*>(st + R::OL_OFF);
                const int64_t t0 = tok0 + (int64_t)(i - 1) * CHUNK;
                auto emit = [&](auto scat) {
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const int r = mt * 16 + g + hh * 8;
                        const int64_t orow = t0 + r < tok_end ? out_row<decltype(scat)::value>(a, t0 + r) : -1;
                        if (orow >= 0) {
#pragma unroll
                            for (int nt = 0; nt < 2; ++nt) {
                                const int col = row0 + nt * 8 + 2 * t;
                                const float2 ol = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(sOl + R::TV::off(r, col)));
                                store_out2(a.o, a.qkv_dt, ((size_t)orow * H + h) * VD + col, ol.x + o[nt][2 * hh], ol.y + o[nt][2 * hh + 1]);
                            }
                        }
                    }
                };
                if (a.out_perm_rows > 0) emit(ScatterOn{}); else emit(ScatterOff{});
            }
            st = now;
        }
        return;
    }
    // ---- levels: warp = (pair, slab) ----
    const int pair = warp / NS, slab = warp - pair * NS, row0 = 16 * slab;
    float C[2][KD / 8][4];
    int lam_row[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int s = pair + x * pairs;
        zero_state<KD>(C[x]);
        lam_row[x] = s;
        if (s >= bl && s < nslots) {
            const int lh = nth_cross(s - bl);
            lam_row[x] = bl + lh;
            load_slab_f32<KD, true>(C[x], a.entry + (((size_t)gb * a.nhigh_max + lh) * H + h) * R::STATE_FLOATS, slab, lane);
        }
    }
    for (int i = 0; i < nsteps; ++i) {
        const unsigned char* st = feed.step(i);
        const __nv_bfloat16* sM = reinterpret_cast<const __nv_bfloat16*>(st + R::M_OFF);
        const __nv_bfloat16* sBt = reinterpret_cast<const __nv_bfloat16*>(st + R::BT_OFF);
        const __nv_bfloat16* sQt = reinterpret_cast<const __nv_bfloat16*>(st + R::QT_OFF);
        const int n = b * bc + i;
        const bool more = i + 1 < nsteps;
        uint32_t sp[2][KD / 16][4];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int s = pair + x * pairs;
            if (s >= nslots) continue;
            pack_state<KD>(C[x], sp[x]);
            if (!more) continue;
            if (s < bl) {
                const int per = 2 << s, pos = n & (per - 1);
                if (((n >> s) & 1) == 0) load_slab_bf16<KD>(C[x], sBt, row0, lane);      // collects
                else zero_state<KD>(C[x]);
                if (pos != per - 1 && pos != 0) state_times_mt<KD>(C[x], sp[x], sM, lane);      // cleared at the end of its period
            } else {
                zero_state<KD>(C[x]);
                state_times_mt<KD>(C[x], sp[x], sM, lane);
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int s = pair + x * pairs;
            if (!read_slot(s, lam_row[x], n)) continue;
            float tmp[4][2][4];
            read_tiles<KD, 4>(tmp, sp[x], sQt, 0, lane);
            float4* d = part + (i & 1) * buf_stride + (s * NS + slab) * 256 + lane;
#pragma unroll
            for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) d[(mt * 2 + nt) * 32] = make_float4(tmp[mt][nt][0], tmp[mt][nt][1], tmp[mt][nt][2], tmp[mt][nt][3]);
        }
    }
    feed.step(nsteps);
}

// ---- launchers ------------------------------------------------------------------------------------
template <typename KernelT>
static int set_smem(KernelT kern, int bytes) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess
               ? LAMPA_OK : LAMPA_ERR_CUDA;
}
#define LAMPA_TRY(x) do { int rc_ = (x); if (rc_ != LAMPA_OK) return rc_; } while (0)
#define LAMPA_LAUNCHED() do { if (cudaGetLastError() != cudaSuccess) return LAMPA_ERR_CUDA; } while (0)

template <int KD, int VD, int SPLIT>
static int launch_compose_split(const GdnArgs& a, cudaStream_t st) {
    using R = Rec<KD, VD>;
    using G = Compose<KD, VD, SPLIT>;
    const int smem = 1024 + G::NST * G::GRP * (R::M_BYTES + R::BT_BYTES);
    LAMPA_TRY(set_smem(gdn_compose_kernel<KD, VD, SPLIT>, smem));
    ProfScope prof("gdn_compose", st);
    launch_chained(gdn_compose_kernel<KD, VD, SPLIT>, dim3(a.nb_max, a.H, SPLIT), G::NW * 32 + 32, smem, st, a);
    LAMPA_LAUNCHED();
    return LAMPA_OK;
}
template <int KD, int VD>
static int launch_compose(const GdnArgs& a, cudaStream_t st) {
    return (int64_t)a.nb_max * a.H <= sm_count() ? launch_compose_split<KD, VD, 2>(a, st) : launch_compose_split<KD, VD, 1>(a, st);
}

template <int KD, int VD, bool HIER, int NW>
static int launch_level_slabs(const GdnArgs& a, int levels, cudaStream_t st) {
    const int smem = LevelSmem<KD, NW>::bytes;
    LAMPA_TRY(set_smem(gdn_level_kernel<KD, VD, HIER, NW>, smem));
    ProfScope prof(HIER ? "gdn_level_hier" : "gdn_level_plain", st);
    launch_chained(gdn_level_kernel<KD, VD, HIER, NW>, dim3(a.nseq, a.H, levels * (VD / 16 / NW)), NW * 32 + 32, smem, st, a);
    LAMPA_LAUNCHED();
    return LAMPA_OK;
}
template <int KD, int VD, bool HIER>
static int launch_level(const GdnArgs& a, int levels, cudaStream_t st) {
    return (int64_t)a.nseq * a.H * levels * (VD / 16) <= 2 * sm_count() ? launch_level_slabs<KD, VD, HIER, 1>(a, levels, st)
                                                                       : launch_level_slabs<KD, VD, HIER, VD / 16>(a, levels, st);
}

template <int KD, int VD>
int launch_scan_plain(const GdnArgs& a, cudaStream_t st) {
    LAMPA_TRY((launch_compose<KD, VD>(a, st)));
    LAMPA_TRY((launch_level<KD, VD, false>(a, 1, st)));
    const int smem = OutPlainSmem<KD, VD>::bytes;
    LAMPA_TRY(set_smem(gdn_out_plain_kernel<KD, VD>, smem));
    ProfScope prof("gdn_out_plain", st);
    launch_chained(gdn_out_plain_kernel<KD, VD>, dim3(a.nb_max, a.H), VD * 2 + 64, smem, st, a);
    LAMPA_LAUNCHED();
    return LAMPA_OK;
}

template <int KD, int VD, int NG>
static int launch_out_hier(const GdnArgs& a, cudaStream_t st) {
    using R = Rec<KD, VD>;
    const int stage = (R::bytes(a.LC) + 1023) / 1024 * 1024;
    const int smem = 1024 + 3 * stage + (NG - 1) * (VD / 16) * 4096;
    if (smem > MAX_SMEM) return LAMPA_ERR_UNSUPPORTED;
    LAMPA_TRY(set_smem(gdn_out_hier_kernel<KD, VD, NG>, MAX_SMEM));
    ProfScope prof("gdn_out_hier", st);
    launch_chained(gdn_out_hier_kernel<KD, VD, NG>, dim3(a.nb_max, a.H), NG * VD * 2, smem, st, a);
    LAMPA_LAUNCHED();
    return LAMPA_OK;
}

template <int KD, int VD, int STAGES>
static int launch_out_levels(const GdnArgs& a, int pairs, cudaStream_t st) {
    const int smem = LevelsSmem<KD, VD, STAGES>::bytes(a.LC, pairs);
    LAMPA_TRY(set_smem(gdn_out_levels_kernel<KD, VD, STAGES>, MAX_SMEM));
    ProfScope prof("gdn_out_hier", st);
    launch_chained(gdn_out_levels_kernel<KD, VD, STAGES>, dim3(a.nb_max, a.H), (2 * pairs + 1 + LV_SUM) * 32, smem, st, a, pairs);
    LAMPA_LAUNCHED();
    return LAMPA_OK;
}

template <int KD, int VD>
int launch_scan_hier(const GdnArgs& a, cudaStream_t st) {
    const int ng = 1 + (a.nhigh_max + NLW - 1) / NLW;
    if (ng > MAX_GROUPS) return LAMPA_ERR_UNSUPPORTED;
    if (a.nhigh_max > 0) {
        LAMPA_TRY((launch_compose<KD, VD>(a, st)));
        LAMPA_TRY((launch_level<KD, VD, true>(a, a.nhigh_max, st)));
    }
    // The two passes add in different orders, so a sequence's own length decides.  A packed call knows it on the device only: where it
    // may hold sequences of more levels than the tcgen05 pass carries, both run, each on its sequences.
    GdnArgs rest = a;
    if (KD == 64 && VD == 64 && a.use_umma) {
        if (a.nlev_max <= UMMA_LEVELS) return launch_out_hier_umma(a, st);
        if (a.fixed_T == 0) {
            GdnArgs shorts = a;
            shorts.short_only = rest.long_only = 1;
            LAMPA_TRY(launch_out_hier_umma(shorts, st));
        }
    }
    if constexpr (KD <= 32) {
        const int pairs = ((a.nlev_max > MIN_BLOCK_LOG ? a.nlev_max : MIN_BLOCK_LOG) + 1) / 2;      // a block has at most a slot per level of its sequence
        if ((int64_t)a.nb_max * a.H <= sm_count() && pairs <= LV_MAX_PAIRS) {
            if (LevelsSmem<KD, VD, 4>::bytes(a.LC, pairs) <= MAX_SMEM) return launch_out_levels<KD, VD, 4>(a, pairs, st);
            if (LevelsSmem<KD, VD, 3>::bytes(a.LC, pairs) <= MAX_SMEM) return launch_out_levels<KD, VD, 3>(a, pairs, st);
        }
    }
    if (ng == 1) return launch_out_hier<KD, VD, 1>(rest, st);
    if (ng == 2) return launch_out_hier<KD, VD, 2>(rest, st);
    return launch_out_hier<KD, VD, 3>(rest, st);
}

template <int KD, int VD>
int launch_final_high(const GdnArgs& a, float* states, cudaStream_t st) {
    using R = Rec<KD, VD>;
    if (a.L <= ELL0) return LAMPA_OK;
    const int smem = 1024 + 3 * (R::M_BYTES + R::BT_BYTES);
    LAMPA_TRY(set_smem(hgdn_final_high_kernel<KD, VD>, smem));
    ProfScope prof("hgdn_final_high", st);
    launch_chained(hgdn_final_high_kernel<KD, VD>, dim3(a.nseq, a.H, a.L - ELL0), VD * 2 + 32, smem, st, a, states);
    LAMPA_LAUNCHED();
    return LAMPA_OK;
}

template int launch_final_high<64, 64>(const GdnArgs&, float*, cudaStream_t);
template int launch_final_high<32, 32>(const GdnArgs&, float*, cudaStream_t);
template int launch_final_high<16, 32>(const GdnArgs&, float*, cudaStream_t);

template int launch_scan_plain<64, 64>(const GdnArgs&, cudaStream_t);
template int launch_scan_plain<32, 32>(const GdnArgs&, cudaStream_t);
template int launch_scan_plain<16, 32>(const GdnArgs&, cudaStream_t);
template int launch_scan_hier<64, 64>(const GdnArgs&, cudaStream_t);
template int launch_scan_hier<32, 32>(const GdnArgs&, cudaStream_t);
template int launch_scan_hier<16, 32>(const GdnArgs&, cudaStream_t);

}  // namespace lampa
