// Layout of the per-chunk and per-block intermediates of the gated-delta forward, and the
// launchers shared between translation units.
//
// Algebra (per sequence and head, chunk length 64, G = inclusive cumsum of g inside the chunk,
// E_ij = exp(G_i - G_j) for i >= j):
//   Aw = (I + tril(diag(beta) K K^T, -1))^-1          W~ = diag(e^G) Aw diag(beta) K
//   U  = (Aw .* E) diag(beta) V                        K~ = diag(e^{G_last - G}) K
//   M  = e^{G_last} I - K~^T W~     B = K~^T U         Q~ = diag(e^G) Q - (tril(Q K^T) .* E) W~
// so that one chunk acts on the running state as  S <- M S + B  and reads it as  Q~ S.
// The prep kernels write one record {M, Q~, B^T, O_local, lambda} per (chunk, head); the scan
// kernels only ever multiply by those.
#pragma once
#include "common.cuh"

namespace lampa {

// Chunks per block of the block-parallel scan, as a power of two: chunk levels 0 .. block_log - 1 live inside a block.
// A block is a serial chain in the compose and output passes, the blocks of a sequence are one in the level pass, so
// the critical path of a sequence of nch chunks is about nch / blocks * (0.35 + 0.5 to 2.5 us) + blocks * 0.3 us (K = V = 64, plain
// to hierarchical output; 0.65 + 1.45 and 0.9 us when the line was drawn, and on the same side of it): 32-chunk blocks left
// 12 - 24 CTAs on the GPU for a 6000-token event (71 us at 4 heads, 30 us with 8).  The smallest block that keeps a
// sequence at 32 blocks or fewer is taken, i.e. 8 chunks up to 256 chunks, 16 up to 512, then 32:
// beyond 1024 chunks there are blocks enough to fill the GPU, and smaller ones would only add composites to move.
// The choice depends on the sequence alone, never on what else a call carries, and so does every other one that changes the order
// of a sum (which output pass a sequence meets, launch_scan_hier; which form takes a prompt's tail, launch_hgdn_tail): a sequence's
// results are the same bits alone, in a batch, packed and in a slice of its heads.
constexpr int BLOCK_LOG = 5;                         // largest block: 32 chunks
constexpr int MIN_BLOCK_LOG = 3;                     // smallest
__host__ __device__ __forceinline__ int block_log(int nch) { return nch <= 256 ? 3 : (nch <= 512 ? 4 : BLOCK_LOG); }
__host__ __device__ __forceinline__ int blocks_of(int nch) { const int bl = block_log(nch); return (nch + (1 << bl) - 1) >> bl; }
constexpr int NLW = 5;               // level states carried per warp in the hierarchical output pass
constexpr int UMMA_LEVELS = BLOCK_LOG + 5;   // chunk levels that the tcgen05 output pass carries: 1024 chunks
constexpr int MAX_GROUPS = 3;        // 1 group of in-block levels + up to 2 groups of cross-block levels

// Layout of a K-wide bf16 tile ([rows][KD]) inside a record.  For KD = 64 rows are dense 128-byte
// lines whose eight 16-byte chunks are XOR-swizzled with the row index (the 128B-swizzle pattern
// tcgen05.mma and ldmatrix both read without bank conflicts); other widths use a padded pitch.
template <int KD>
struct Tile {
    static constexpr bool SWZ = (KD == 64);
    static constexpr int PITCH = SWZ ? 64 : KD + 8;
    __host__ __device__ static constexpr int off(int r, int c) {
        return SWZ ? r * 64 + ((((c >> 3) ^ r) & 7) << 3) + (c & 7) : r * PITCH + c;
    }
    __host__ __device__ static constexpr int bytes(int rows) { return rows * PITCH * 2; }
};

template <int KD, int VD>
struct Rec {
    using T = Tile<KD>;
    using TV = Tile<VD>;                              // layout of O_local[token][v]: a V-wide bf16 tile
    static constexpr int M_OFF = 0;
    static constexpr int M_BYTES = T::bytes(KD);      // M[k_out][k_in]
    static constexpr int QT_OFF = M_OFF + M_BYTES;    // M and Q~ are adjacent: together they are one 128-row B operand
    static constexpr int QT_BYTES = T::bytes(CHUNK);  // Q~[token][k]
    static constexpr int BT_OFF = QT_OFF + QT_BYTES;
    static constexpr int BT_BYTES = T::bytes(VD);     // B^T[v][k]
    static constexpr int OL_OFF = BT_OFF + BT_BYTES;
    static constexpr int OL_BYTES = TV::bytes(CHUNK); // O_local, bf16 (added once, in fp32, by the output pass)
    static constexpr int LAM_OFF = OL_OFF + OL_BYTES; // lambda of chunk levels: [LC][64] fp32
    static constexpr int ALIGN = T::SWZ ? 1024 : 128; // records and shared-memory stages
    __host__ __device__ static constexpr int bytes(int LC) { return LAM_OFF + LC * CHUNK * 4; }
    // block composite, in the order in which the lanes of the level pass take it (16 bytes per lane, whole lines per warp):
    // Mblk as bf16 B fragments [k_in / 16][k_out / 16][lane][4 words], then Bblk^T as an fp32 state
    static constexpr int BLK_M_OFF = 0;
    static constexpr int BLK_M_BYTES = KD * KD * 2;
    static constexpr int BLK_B_OFF = BLK_M_BYTES;
    static constexpr int BLK_BYTES = BLK_M_BYTES + VD * KD * 4;
    // An fp32 state S^T[v][k] (entry states, Bblk^T) is kept as the accumulators of a warp's 16 rows hold it: element (v, k) at
    // state_at().  A warp moves its slab in KD / 8 instructions of whole 128-byte lines (row-major it was 16 instructions of 8
    // sectors each, 480 of the level pass's 1560 cycles per block), and a row's 16 columns 16p .. 16p + 15 are 64 contiguous
    // bytes: four pieces of 16, piece t holding columns 2t, 2t + 1, 8 + 2t, 9 + 2t.
    static constexpr int STATE_FLOATS = VD * KD;
    __host__ __device__ static constexpr int state_at(int v, int k) {
        return ((((v >> 4) * (KD / 16) + (k >> 4)) * 2 + ((v >> 3) & 1)) * 32 + (v & 7) * 4 + ((k >> 1) & 3)) * 4 + ((k >> 3) & 1) * 2 + (k & 1);
    }
};

struct GdnArgs {
    const void* q; const void* k; const void* v; const void* g; const void* beta; const void* lam;
    const float* h0; float* ht; void* o;
    const int64_t* out_perm; long long out_perm_rows;   // optional scatter of the output rows (lampa_hgdn_fwd_scatter)
    int qkv_dt, gb_dt, lam_dt;
    int H, L, LC;
    int use_l2norm;
    float scale;
    int nseq;
    int fixed_T;        // tokens per sequence when there is no cu_seqlens (0 otherwise)
    int fixed_stride;   // tokens from one sequence to the next in that case (fixed_T, or more when a prompt's tail is left to hgdn_tail)
    int fixed_cps;      // chunks per sequence in that case: positions follow by arithmetic, no plan loads
    int nc_max, nb_max, nhigh_max;
    int nlev_max;       // chunk levels of the longest sequence there can be
    long long total_tokens;  // B * T of the call (rows of the token-major inputs)
    const int64_t* tok_off; const int32_t* chunk_off; const int32_t* block_off;   // offset tables of a packed call (plan_kernel)
    char* rec; size_t rec_bytes;          // per (chunk, head) records
    char* blk;                            // per (block, head) composites
    float* entry;                         // entry states: plain [nb][H][V][K]; hier [nb][nhigh][H][V][K]
    int32_t* status;
    int use_umma;                         // tcgen05 kernels where they exist (K = V = 64)
    int poll_budget;                      // polls before a device wait gives up (MBAR_POLLS unless a test lowers it)
    int long_only, short_only;            // output pass: only sequences of more (of at most) UMMA_LEVELS chunk levels
    unsigned long long signal;            // a prefill's number, or 0: its output pass and chunk levels let the next kernel in (chain_signal)
    unsigned long long* signal_word;
    long long* ticks; int ticks_ctas;     // stage clocks for tuning: [ticks_ctas][16] or NULL (lampa_debug_set_tick_buffer)
};

// Stage clock of a preparation CTA: thread 0 of the first `ticks_ctas` CTAs stores clock64() in its slot.
__device__ __forceinline__ void stage_tick(const GdnArgs& a, int cta, int slot) {
    if (a.ticks != nullptr && threadIdx.x == 0 && cta < a.ticks_ctas) a.ticks[(size_t)cta * 16 + slot] = clock64();
}

struct PlanArgs {
    const int64_t* cu; int nseq; int B; int T; int L; int hier;
    int64_t* tok_off; int32_t* chunk_off; int32_t* block_off; int32_t* status;
};

int launch_plan(const PlanArgs& p, cudaStream_t st);
template <int KD, int VD> int launch_prep(const GdnArgs& a, bool hier, cudaStream_t st);
template <int KD, int VD> int launch_scan_plain(const GdnArgs& a, cudaStream_t st);
template <int KD, int VD> int launch_scan_hier(const GdnArgs& a, cudaStream_t st);

// Where chunk slot c lives: sequence, first token, number of valid tokens.  False for unused slots.
struct ChunkLoc { int seq; int64_t t0; int len; };
__device__ __forceinline__ bool locate_chunk(const GdnArgs& a, int c, ChunkLoc& loc) {
    if (a.fixed_T > 0) {
        if (c >= a.nseq * a.fixed_cps) return false;
        loc.seq = c / a.fixed_cps;
        const int local = c - loc.seq * a.fixed_cps;
        loc.t0 = (int64_t)loc.seq * a.fixed_stride + (int64_t)local * CHUNK;
        loc.len = min(CHUNK, a.fixed_T - local * CHUNK);
        return true;
    }
    if (c >= a.chunk_off[a.nseq]) return false;
    loc.seq = find_seq(a.chunk_off, a.nseq, c);
    loc.t0 = a.tok_off[loc.seq] + (int64_t)(c - a.chunk_off[loc.seq]) * CHUNK;
    loc.len = (int)min((int64_t)CHUNK, a.tok_off[loc.seq + 1] - loc.t0);
    return true;
}

// The chunks, blocks and tokens of a sequence.  Equally long sequences follow by arithmetic: the dependent loads of the offset
// tables are the first thing a CTA of the scan would wait for (about 1 us of a pass that is 10 to 20 us long).
struct SeqLoc { int nch, c0, nblk, gb0; int64_t tok0, tok_end; };
__device__ __forceinline__ SeqLoc locate_seq(const GdnArgs& a, int seq) {
    SeqLoc s;
    if (a.fixed_T > 0) {
        s.nch = a.fixed_cps;
        s.c0 = seq * a.fixed_cps;
        s.nblk = blocks_of(a.fixed_cps);
        s.gb0 = seq * s.nblk;
        s.tok0 = (int64_t)seq * a.fixed_stride;
        s.tok_end = s.tok0 + a.fixed_T;
    } else {
        s.c0 = a.chunk_off[seq];
        s.nch = a.chunk_off[seq + 1] - s.c0;
        s.gb0 = a.block_off[seq];
        s.nblk = a.block_off[seq + 1] - s.gb0;
        s.tok0 = a.tok_off[seq];
        s.tok_end = a.tok_off[seq + 1];
    }
    return s;
}
// Where block slot gb lives: its sequence and its place in it.  False for unused slots.
__device__ __forceinline__ bool locate_block(const GdnArgs& a, int gb, SeqLoc& s, int& b) {
    int seq;
    if (a.fixed_T > 0) {
        seq = gb / blocks_of(a.fixed_cps);
        if (seq >= a.nseq) return false;
    } else {
        if (gb >= a.block_off[a.nseq]) return false;
        seq = find_seq(a.block_off, a.nseq, gb);
    }
    s = locate_seq(a, seq);
    b = gb - s.gb0;
    return true;
}

// Row of o that token t of the call is written to: its own, or out_perm[t] for the first out_perm_rows tokens
// when the caller asked for the output to be scattered (the un-ordering of a sorted event folded into the store).
// -1 for an index outside the output: that row is not written (the preparation kernel has reported it, see
// check_out_perm; the output passes stay free of the reporting code).
// SCAT is a compile-time flag so that the common, unscattered store keeps its plain address arithmetic: the output
// passes test a.out_perm_rows once per chunk and run one of two copies of their store code.
template <bool SCAT>
__device__ __forceinline__ int64_t out_row(const GdnArgs& a, int64_t t) {
    if (!SCAT || t >= a.out_perm_rows) return t;
    const int64_t r = a.out_perm[t];
    return (unsigned long long)r < (unsigned long long)a.total_tokens ? r : -1;
}
struct ScatterOn { static constexpr bool value = true; };
struct ScatterOff { static constexpr bool value = false; };
// The scatter indices of one chunk's tokens, checked by the first 64 threads of one preparation CTA per chunk.
__device__ __forceinline__ void check_out_perm(const GdnArgs& a, int64_t t0, int len) {
    const int64_t t = t0 + threadIdx.x;
    if (a.out_perm_rows > 0 && (int)threadIdx.x < len && t < a.out_perm_rows &&
        (unsigned long long)a.out_perm[t] >= (unsigned long long)a.total_tokens)
        set_status(a.status, LAMPA_ERR_BOUNDS, 30, (int)t);
}

// Two output values (adjacent state columns) of one token, converted to the output type.
__device__ __forceinline__ void store_out2(void* o, int dt, size_t idx, float x, float y) {
    if (dt == LAMPA_BF16) *reinterpret_cast<uint32_t*>((__nv_bfloat16*)o + idx) = pack_bf16x2(x, y);
    else if (dt == LAMPA_F16) *reinterpret_cast<__half2*>((__half*)o + idx) = __floats2half2_rn(x, y);
    else *reinterpret_cast<float2*>((float*)o + idx) = make_float2(x, y);
}

int launch_out_hier_umma(const GdnArgs& a, cudaStream_t st);
int launch_prep_umma(const GdnArgs& a, bool hier, cudaStream_t st);   // K = V = 64, 2-byte q/k/v
template <int KD, int VD> int launch_final_high(const GdnArgs& a, float* states, cudaStream_t st);
// The end of every sequence in fp32 (gdn_state.cu): token levels of the state, and the tokens behind the last whole chunk.
struct TailArgs {
    float* states; int32_t* counts;       // [N][H][K][V][L]; [N][L], or [L] when one_count (all sequences equally long)
    int n0;                               // whole chunks of every sequence, or -1: from chunk_off, ragged chunks completed by null tokens
    int tail;                             // tokens behind them (only with n0 >= 0)
    int one_count;
    int32_t* arrivals;                    // set to zero, or NULL: the arrival counter of the decode steps to come
    int early;                            // this call's kernels in front signal early (GdnArgs::signal)
    int slabs = 1;                        // eight state columns each: what a CTA of the closed form works through
};
template <int KD, int VD> int launch_hgdn_tail(const GdnArgs& a, const TailArgs& ta, cudaStream_t st);

// One decode step of the hierarchical rule on a Fenwick state (gdn_state.cu).
struct StepArgs {
    const void* q; const void* k; const void* v; const void* g; const void* beta; const void* lam;
    float* states; int32_t* counts; void* o;
    int qkv_dt, gb_dt, lam_dt;
    int B, H, L, use_l2norm;
    int32_t* arrivals;                    // zero between steps: counts the CTAs that are done, or NULL (counts advanced by a second launch)
    int poll_budget;
    int32_t* status;
};
template <int KD, int VD> int launch_hgdn_step(const StepArgs& s, cudaStream_t st);

__host__ __device__ inline int ceil_log2_int(int x) {   // smallest e with 2^e >= x (x >= 1)
    int e = 0;
    while ((1 << e) < x) ++e;
    return e;
}

}  // namespace lampa
