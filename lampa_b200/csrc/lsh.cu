// E2LSH hashing, segmented stable radix sort, row permutation: the ordering half of the path.
// All kernels are HBM/L2-bound integer and byte work; no tensor cores here by design.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "common.cuh"
#include "profile.cuh"

namespace cg = cooperative_groups;

namespace lampa {

// -------------------------------------------------------------------------------------------------
// Hash: one thread per hit.  Reads dim floats of the hit's row (for the detector rows of this
// workload 24 B of a 96 B row: one 32 B sector) and writes rounds*heads ids, each coalesced across
// the warp.  The operation order is a contract shared with the CPU oracle (see the header).
// -------------------------------------------------------------------------------------------------
constexpr int HASH_THREADS = 256;
constexpr int HASH_MAX_PARAMS = 4096;   // heads*dim*rounds floats staged in shared memory

template <int DIMT>   // DIMT > 0: coordinates kept in registers (dim == DIMT, shared rows)
__global__ void __launch_bounds__(HASH_THREADS)
lsh_hash_kernel(const float* __restrict__ x, int64_t row_stride, int64_t head_stride,
                const float* __restrict__ alpha, const float* __restrict__ beta, float w, int64_t N,
                int heads, int rounds, int dim, int per, int32_t* __restrict__ ids, float* __restrict__ keys,
                int32_t* __restrict__ packed) {
    if (chain_wait()) return;
    __shared__ float s_alpha[HASH_MAX_PARAMS];
    __shared__ float s_beta[64];
    const int np = heads * dim * rounds;
    for (int i = threadIdx.x; i < np; i += HASH_THREADS) s_alpha[i] = alpha[i];
    for (int i = threadIdx.x; i < rounds; i += HASH_THREADS) s_beta[i] = beta[i];
    __syncthreads();
    const int64_t n = (int64_t)blockIdx.x * HASH_THREADS + threadIdx.x;
    if (n >= N) return;
    float xv[DIMT > 0 ? DIMT : 1];
    if (DIMT > 0) {
#pragma unroll
        for (int d = 0; d < DIMT; ++d) xv[d] = __ldg(x + n * row_stride + d);
    }
    const int c0 = blockIdx.y * per, c1 = min(c0 + per, rounds);
    for (int c = c0; c < c1; ++c) {
        int32_t pk = 0;
        for (int h = 0; h < heads; ++h) {
            const float* a = s_alpha + (size_t)h * dim * rounds + c;   // a[d*rounds]
            float acc;
            if (DIMT > 0) {
                acc = __fmul_rn(xv[0], a[0]);
#pragma unroll
                for (int d = 1; d < DIMT; ++d) acc = __fadd_rn(acc, __fmul_rn(xv[d], a[d * rounds]));
            } else {
                const float* xr = x + h * head_stride + n * row_stride;
                acc = __fmul_rn(__ldg(xr), a[0]);
                for (int d = 1; d < dim; ++d) acc = __fadd_rn(acc, __fmul_rn(__ldg(xr + d), a[d * rounds]));
            }
            const size_t o = ((size_t)c * heads + h) * N + n;
            if (keys) keys[o] = acc;
            if (ids || packed) {
                const int32_t id = (int32_t)floorf(__fdiv_rn(__fadd_rn(acc, s_beta[c]), w));
                if (ids) ids[o] = id;
                pk += (int32_t)((uint32_t)id << h);
            }
        }
        if (packed) packed[(size_t)c * N + n] = pk;
    }
}

// -------------------------------------------------------------------------------------------------
// Segmented stable LSD radix sort.  One thread-block cluster (up to 16 CTAs) per segment: each CTA
// owns a contiguous slice of the segment in its current order, digit histograms are exchanged
// through distributed shared memory, and the passes are separated by the hardware cluster barrier
// (no flag spinning anywhere).  The cluster size is the largest one for which the occupancy
// calculator reports all clusters resident at once: a cluster lives inside one GPC, and a size that
// merely divides the SM count left a third of the clusters waiting for a second wave (24 x 60 000
// keys: 103 us against 57 us then; 45 us with the tile as large as the slice).  Keys are reduced to
// (key - min) first, so only as many passes of 8 or 9 bits run as the key range needs: two for the
// ~15-bit bucket ids of an event.
//
// A CTA takes its slice in tiles of ITEMS * 1024 keys held in registers; a warp owns ITEMS * 32
// consecutive keys and ranks them 32 at a time with one ballot per digit bit on top of its row of
// digit counters, so the order (round, lane) is the key order and the sort is stable.  What bounds a
// pass is instruction issue and its fixed chain of barriers, so the tile is as large as the slice
// where it fits (the counters then double as the histogram: no separate sweep), the prefix over the
// 32 warps' counters is one thread per digit (a warp-wide scan per digit cost as much as the
// ranking), and the tile is grouped by digit in shared memory so that the writes are runs.
// -------------------------------------------------------------------------------------------------
constexpr int SORT_THREADS = 1024;
constexpr int SORT_MAX_CL = 16;          // beyond 8 the kernel opts in (non-portable cluster size)
constexpr int SORT_DIGITS = 512;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_MAX_ITEMS = 12;

__device__ __forceinline__ uint32_t key_xform(const void* keys, int key_type, int64_t i) {
    uint32_t u = ((const uint32_t*)keys)[i];
    if (key_type == LAMPA_KEY_I32) return u ^ 0x80000000u;
    // float: order-preserving map; -0.0 and +0.0 compare equal in torch.sort, so fold -0 onto +0
    if (u == 0x80000000u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// exclusive prefix over n values (a multiple of 32, at most 512) held by threads 0..n - 1; wtot: a word per warp of them in shared
// memory.  All threads call it.
__device__ __forceinline__ uint32_t prefix_digits(uint32_t v, uint32_t* wtot, int tid, int n) {
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t incl = v;
    if (tid < n) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wtot[warp] = incl;
    }
    __syncthreads();
    if (tid < n)
        for (int w = 0; w < warp; ++w) incl += wtot[w];
    return incl - v;
}

// INIT: a starting order is given.  Its entries are somebody else's and are held against the segment before they are followed; a
// copy of its own, since that check in a sort without one cost 24 x 60 000 keys 47.4 instead of 45.4 us (registers spilled).
template <int ITEMS, bool INIT>
__global__ void __launch_bounds__(SORT_THREADS, 1)
segsort_kernel(const void* __restrict__ keys, int key_type, int64_t n_total,
               const int64_t* __restrict__ seg, int nseg, const int64_t* __restrict__ init,
               int64_t* __restrict__ perm, uint32_t* kbuf0, uint32_t* kbuf1, uint32_t* ibuf0,
               uint32_t* ibuf1, int32_t* status) {
    if (chain_wait()) return;
    constexpr int TILE = ITEMS * SORT_THREADS;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int ncl = (int)cluster.num_blocks();
    const int s = blockIdx.x / ncl;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    int64_t s0, n;
    if (seg) { s0 = seg[s]; n = seg[s + 1] - s0; }
    else { n = n_total / nseg; s0 = (int64_t)s * n; }
    if (n < 0 || s0 < 0 || s0 + n > n_total) {   // offsets that leave the key array: sort nothing, say so
        if (tid == 0 && rank == 0) set_status(status, LAMPA_ERR_BOUNDS, 12, s);
        n = 0;
    }
    const int64_t per = (n + ncl - 1) / ncl;
    const int64_t lo = min((int64_t)rank * per, n), hi = min(lo + per, n);
    const bool one_tile = hi - lo <= TILE;

    __shared__ uint32_t hist[SORT_DIGITS], dbase[SORT_DIGITS], tstart[SORT_DIGITS], tile_tot[SORT_DIGITS];
    __shared__ uint32_t wtot[SORT_DIGITS / 32], red[2];
    __shared__ __align__(16) uint16_t wcount[SORT_WARPS][SORT_DIGITS];
    extern __shared__ uint32_t sort_dyn[];         // [TILE] keys, [TILE] indices of the tile, grouped by digit
    uint32_t* skey = sort_dyn;
    uint32_t* sidx = sort_dyn + TILE;

    uint32_t u[ITEMS], idx[ITEMS];
    const int wpos = warp * (32 * ITEMS) + lane;   // of item 0; item `it` is 32 * it further
    // an entry of the starting order that leaves the segment stands for its first element, and is reported
    bool astray = false;
    auto starting = [&](int64_t i) {
        const int64_t e = init[s0 + i];
        const bool out = (uint64_t)e >= (uint64_t)n;
        astray |= out;
        return out ? 0u : (uint32_t)e;
    };
    // keys of a tile in their current order: position i of the first pass holds element init[i]
    auto load_tile = [&](int64_t t0, int p, const uint32_t* ksrc, const uint32_t* isrc, uint32_t base) {
        if (p == 0) {
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                const int64_t i = t0 + wpos + it * 32;
                idx[it] = i < hi ? (INIT ? starting(i) : (uint32_t)i) : 0u;
            }
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) u[it] = t0 + wpos + it * 32 < hi ? key_xform(keys, key_type, s0 + idx[it]) - base : 0u;
        } else {
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                const int64_t i = t0 + wpos + it * 32;
                u[it] = i < hi ? ksrc[s0 + i] : 0u;
                idx[it] = i < hi ? isrc[s0 + i] : 0u;
            }
        }
    };

    // ---- key range over the whole segment -------------------------------------------------------
    if (tid == 0) { red[0] = 0xFFFFFFFFu; red[1] = 0u; }
    __syncthreads();
    {
        uint32_t mn = 0xFFFFFFFFu, mx = 0u;
        for (int64_t t0 = lo; t0 < hi; t0 += TILE) {
            load_tile(t0, 0, nullptr, nullptr, 0u);
#pragma unroll
            for (int it = 0; it < ITEMS; ++it)
                if (t0 + wpos + it * 32 < hi) { mn = min(mn, u[it]); mx = max(mx, u[it]); }
        }
        if (INIT && astray) set_status(status, LAMPA_ERR_BOUNDS, 14, s);
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) { atomicMin(&red[0], mn); atomicMax(&red[1], mx); }
    }
    __syncthreads();
    cluster.sync();
    uint32_t gmn = 0xFFFFFFFFu, gmx = 0u;
    for (int r = 0; r < ncl; ++r) {
        const uint32_t* rr = cluster.map_shared_rank(red, r);
        gmn = min(gmn, rr[0]); gmx = max(gmx, rr[1]);
    }
    const uint32_t range = (n > 0 && gmx >= gmn) ? (gmx - gmn) : 0u;
    const int bits = range ? (32 - __clz(range)) : 0;
    // Digits of up to eight bits, or of nine where that saves a pass (24 segments of 60,000 keys of 26 bits: 68.6 us with four
    // passes of seven bits, 57.6 with three of nine); of equal width.
    const int npass = (bits + 8) / 9 < (bits + 7) / 8 ? (bits + 8) / 9 : (bits + 7) / 8;
    const int width = npass ? (bits + npass - 1) / npass : 0;
    const int ndig = max(32, 1 << width);

    if (npass == 0) {
        for (int64_t i = lo + tid; i < hi; i += SORT_THREADS) perm[s0 + i] = INIT ? (int64_t)starting(i) : i;
    }

    for (int p = 0; p < npass; ++p) {
        const int shift = width * p;
        const uint32_t dmask = (1u << width) - 1u;
        const uint32_t* ksrc = (p & 1) ? kbuf0 : kbuf1;   // pass p reads what pass p-1 wrote
        const uint32_t* isrc = (p & 1) ? ibuf0 : ibuf1;
        uint32_t* kdst = (p & 1) ? kbuf1 : kbuf0;
        uint32_t* idst = (p & 1) ? ibuf1 : ibuf0;
        const bool last = (p == npass - 1);
        uint32_t rnk[(ITEMS + 1) / 2];                    // two 16-bit ranks (within warp and digit) per word

        // digit counters of a tile: rank of every key within its warp and digit, then the exclusive prefix over the warps
        auto rank_tile = [&](int64_t t0) {
            for (int z = lane * 8; z < ndig; z += 256) *reinterpret_cast<uint4*>(&wcount[warp][z]) = make_uint4(0u, 0u, 0u, 0u);      // the warp's own row
            __syncthreads();
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                const bool valid = t0 + wpos + it * 32 < hi;
                const uint32_t d = (u[it] >> shift) & dmask;
                uint32_t m = __ballot_sync(0xffffffffu, valid);
                if (m == 0u) { if (!(it & 1)) rnk[it >> 1] = 0u; continue; }         // warp-uniform: past the slice's end
#pragma unroll
                for (int bit = 0; bit < 8; ++bit) {
                    const bool one = (d >> bit) & 1u;
                    const uint32_t bal = __ballot_sync(0xffffffffu, one);
                    m &= one ? bal : ~bal;
                }
                if (width > 8) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, d & 256u);
                    m &= (d & 256u) ? bal : ~bal;
                }
                const uint32_t basecnt = valid ? wcount[warp][d] : 0u;
                const uint32_t r = basecnt + __popc(m & ((1u << lane) - 1u));
                if (it & 1) rnk[it >> 1] |= r << 16; else rnk[it >> 1] = r;
                __syncwarp();
                if (valid && (__ffs(m) - 1) == lane) wcount[warp][d] = (uint16_t)(basecnt + __popc(m));
                __syncwarp();
            }
            __syncthreads();
            if (tid < ndig) {
                uint32_t run = 0;
#pragma unroll 8
                for (int w = 0; w < SORT_WARPS; ++w) {
                    const uint32_t c = wcount[w][tid];
                    wcount[w][tid] = (uint16_t)run;
                    run += c;
                }
                tile_tot[tid] = run;
            }
        };

        // (a) digit histogram of this CTA's slice
        if (one_tile) {
            if (p == 0) {                                 // still in registers from the range sweep
#pragma unroll
                for (int it = 0; it < ITEMS; ++it) u[it] -= gmn;
            } else if (lo < hi) {
                load_tile(lo, p, ksrc, isrc, gmn);
            }
            rank_tile(lo);
            if (tid < ndig) hist[tid] = tile_tot[tid];
        } else {
            if (tid < ndig) hist[tid] = 0;
            __syncthreads();
            for (int64_t t0 = lo; t0 < hi; t0 += TILE) {
                load_tile(t0, p, ksrc, isrc, gmn);
#pragma unroll
                for (int it = 0; it < ITEMS; ++it)
                    if (t0 + wpos + it * 32 < hi) atomicAdd(&hist[(u[it] >> shift) & dmask], 1u);
            }
        }
        __syncthreads();
        cluster.sync();

        // (b) where each digit of this slice starts in the segment
        uint32_t tot = 0, before = 0;
        if (tid < ndig)
            for (int r = 0; r < ncl; ++r) {
                const uint32_t hv = cluster.map_shared_rank(hist, r)[tid];
                tot += hv;
                if (r < rank) before += hv;
            }
        const uint32_t ex = prefix_digits(tot, wtot, tid, ndig);
        if (tid < ndig) dbase[tid] = ex + before;
        __syncthreads();

        // (c) stable scatter, tile by tile in slice order
        for (int64_t t0 = lo; t0 < hi; t0 += TILE) {
            // A slice of several tiles reads its keys twice, for the histogram and here.  Segments that overlap (offsets that
            // fall: the segment in between reports them) rewrite each other's keys in between, and the counts no longer add
            // up: a tile whose keys would land behind the segment is not written.
            bool outside = false;
            if (!one_tile) {
                load_tile(t0, p, ksrc, isrc, gmn);
                rank_tile(t0);
                outside = __syncthreads_or(tid < ndig && (int64_t)dbase[tid] + tile_tot[tid] > n);
            }
            const uint32_t ts = prefix_digits(tid < ndig ? tile_tot[tid] : 0u, wtot, tid, ndig);
            if (tid < ndig) tstart[tid] = ts;
            __syncthreads();
            // group the tile by digit in shared memory, so that the global writes below are runs of
            // consecutive addresses (a direct scatter costs one 32-byte sector per key)
#pragma unroll
            for (int it = 0; it < ITEMS; ++it)
                if (t0 + wpos + it * 32 < hi) {
                    const uint32_t d = (u[it] >> shift) & dmask;
                    const uint32_t lp = tstart[d] + wcount[warp][d] + ((rnk[it >> 1] >> (16 * (it & 1))) & 0xffffu);
                    skey[lp] = u[it];
                    sidx[lp] = idx[it];
                }
            __syncthreads();
            const int ntile = outside ? 0 : (int)min((int64_t)TILE, hi - t0);
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                const int lp = it * SORT_THREADS + tid;
                if (lp < ntile) {
                    const uint32_t ku = skey[lp], ki = sidx[lp];
                    const uint32_t d = (ku >> shift) & dmask;
                    const int64_t pos = (int64_t)dbase[d] + (lp - tstart[d]);
                    if (last) {
                        perm[s0 + pos] = (int64_t)ki;
                    } else {
                        kdst[s0 + pos] = ku;
                        idst[s0 + pos] = ki;
                    }
                }
            }
            if (t0 + TILE < hi) {
                __syncthreads();
                if (tid < ndig) dbase[tid] += tile_tot[tid];
                __syncthreads();
            }
        }
        cluster.sync();   // release/acquire at cluster scope: scattered keys visible to the peers; histograms free again
    }
    if (npass == 0) cluster.sync();       // no CTA leaves while a peer may still read its shared memory
}

// Upper bound of the cluster size: SMs / segments (the launcher lowers it until all fit), at most 8, or 16 where eight slices would
// be longer than 4096 keys.  2 x 60,000 keys: 50 us in slices of 7,500 and 37 in slices of 3,750; 4 x 20,000 28.5 and 30, 3 x 9,001
// 14.5 and 16.9, since a cluster barrier of sixteen costs more than half a short slice.
static int sort_cluster_size(int nseg, int64_t avg_keys) {
    int cl = sm_count() / (nseg > 0 ? nseg : 1);
    const int most = avg_keys > 8 * 4096 ? SORT_MAX_CL : 8;
    if (cl > most) cl = most;
    if (cl < 1) cl = 1;
    return cl;
}

// cudaOccupancyMaxActiveClusters for a kernel, remembered per (device, cluster size, tile):
// the answer does not change and the query costs tens of microseconds of host time.
template <typename K>
static int clusters_resident(K kernel, const cudaLaunchConfig_t& cfg, int cl, int items) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, int>, int> memo;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, cl, items);
    std::lock_guard<std::mutex> lk(mu);
    const auto it = memo.find(key);
    if (it != memo.end()) return it->second;
    int resident = 0;
    if (cudaOccupancyMaxActiveClusters(&resident, kernel, &cfg) != cudaSuccess) resident = 0;
    memo[key] = resident;
    return resident;
}

static int launch_segsort(const void* keys, int key_type, int64_t n_total, const int64_t* seg, int nseg,
                          const int64_t* init, int64_t* perm, uint32_t* k0, uint32_t* k1, uint32_t* i0,
                          uint32_t* i1, int32_t* status, cudaStream_t st) {
    using Kernel = void (*)(const void*, int, int64_t, const int64_t*, int, const int64_t*, int64_t*, uint32_t*, uint32_t*, uint32_t*, uint32_t*, int32_t*);
    static const Kernel all[2][5] = {
        {segsort_kernel<1, false>, segsort_kernel<2, false>, segsort_kernel<4, false>, segsort_kernel<8, false>, segsort_kernel<SORT_MAX_ITEMS, false>},
        {segsort_kernel<1, true>, segsort_kernel<2, true>, segsort_kernel<4, true>, segsort_kernel<8, true>, segsort_kernel<SORT_MAX_ITEMS, true>}};
    const Kernel* kernels = all[init != nullptr];
    static const int item_counts[] = {1, 2, 4, 8, SORT_MAX_ITEMS};
    static std::atomic<uint64_t> ready[2][5];
    // Cluster size: the largest one for which every segment's cluster is resident at the same time.
    // A cluster has to fit inside one GPC, so the SM count alone does not tell (148 SMs hold 24
    // clusters of 6 only if every GPC has 18 usable SMs): ask the occupancy calculator.
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    int cl = sort_cluster_size(nseg, n_total / (nseg > 0 ? nseg : 1)), which = 0;
    for (;; --cl) {
        // tile: the slice of an equal split, or twice the average slice when the segments are ragged (larger slices
        // take several tiles), at most 12 keys per thread (96 KB)
        const int64_t avg = (n_total / (nseg > 0 ? nseg : 1) + cl - 1) / cl + 1;
        const int64_t want = seg ? 2 * avg : avg;
        which = 0;
        while (which < 4 && (int64_t)item_counts[which] * SORT_THREADS < want) ++which;
        if (!allow_smem(ready[init != nullptr][which], kernels[which], 2 * item_counts[which] * SORT_THREADS * 4)) return LAMPA_ERR_CUDA;
        if (cl > 8 && cudaFuncSetAttribute(kernels[which], cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return LAMPA_ERR_CUDA;
        cfg.gridDim = dim3((unsigned)nseg * cl, 1, 1);
        cfg.blockDim = dim3(SORT_THREADS, 1, 1);
        cfg.dynamicSmemBytes = (size_t)2 * item_counts[which] * SORT_THREADS * 4;
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cl;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;                    // the occupancy query knows clusters only
        if (cl == 1) break;
        if (clusters_resident(kernels[which], cfg, cl, 2 * item_counts[which] + (init != nullptr)) >= nseg) break;
    }
    attr[1] = chained_attribute();
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernels[which], keys, key_type, n_total, seg, nseg, init, perm, k0, k1, i0, i1, status);
    return e == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

// -------------------------------------------------------------------------------------------------
// Row gather/scatter and permutation inverse.
// -------------------------------------------------------------------------------------------------
__device__ __forceinline__ int find_seg64(const int64_t* off, int nseg, int64_t x) {
    int lo = 0, hi = nseg;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}

// An index outside its segment is not followed: the access is skipped and LAMPA_ERR_BOUNDS is
// recorded in the status word (a permutation that came from lampa_segsort_stable never trips it).
template <typename VEC>
__global__ void __launch_bounds__(256)
permute_rows_kernel(const VEC* __restrict__ src, const int64_t* __restrict__ perm,
                    const int64_t* __restrict__ seg, int nseg, int64_t n_rows, int64_t units_per_row,
                    int scatter, VEC* __restrict__ dst, int32_t* status) {
    if (chain_wait()) return;
    const int64_t total = n_rows * units_per_row;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = u / units_per_row, col = u - row * units_per_row;
        int64_t s0, len;
        if (seg) { const int si = find_seg64(seg, nseg, row); s0 = seg[si]; len = seg[si + 1] - s0; }
        else { len = n_rows / nseg; s0 = (row / len) * len; }
        const int64_t p = perm[row];
        if (p < 0 || p >= len || s0 < 0 || s0 + len > n_rows) {
            if (col == 0) set_status(status, LAMPA_ERR_BOUNDS, 10, (int)row);
            continue;
        }
        const int64_t other = s0 + p;
        if (scatter) dst[other * units_per_row + col] = src[u];
        else dst[u] = src[other * units_per_row + col];
    }
}

__global__ void __launch_bounds__(256)
invert_perm_kernel(const int64_t* __restrict__ perm, const int64_t* __restrict__ seg, int nseg,
                   int64_t n_total, int64_t* __restrict__ inv, int32_t* status) {
    if (chain_wait()) return;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t s0, len;
        if (seg) { const int si = find_seg64(seg, nseg, i); s0 = seg[si]; len = seg[si + 1] - s0; }
        else { len = n_total / nseg; s0 = (i / len) * len; }
        const int64_t p = perm[i];
        if (p < 0 || p >= len || s0 < 0 || s0 + len > n_total) { set_status(status, LAMPA_ERR_BOUNDS, 11, (int)i); continue; }
        inv[s0 + p] = i - s0;
    }
}

// -------------------------------------------------------------------------------------------------
// LSHOrdering: key = sum_c 2^c (coords . alpha[:, c]), rows ordered by (key, |coords|, index) — the
// norm pre-sort and the stable key sort of the reference in one order — and gathered.
//
// A point cloud of a few thousand points is all latency for a radix sort (two sorts of four passes
// each: 34 us apiece for 4 x 1500 points, beside seven small launches for keys, norms and the
// gather).  Here one launch does everything by counting: every CTA computes all keys of its segment
// (24 bytes and ~50 flops per point, from L2), takes 32 points, eight lanes to a point, and counts
// the points that come before each; the count is the point's position.  n^2 comparisons, but all in
// parallel.  The keys are half of it, and instruction issue bounds them: two points at a time, the
// coordinates in registers, and loops over coordinates and hashes known to the compiler up to 8 and
// 4.  4 x 1500 points with (coordinates, hashes) = (6, 3), (3, 3), (6, 4), (4, 6), (8, 8), (11, 3):
// 8.7, 8.1, 9.0, 9.7, 12 and 13 us; with the hash count always a loop 9.3, 8.3, 9.5, 9.6, 12 and 12;
// reading the coordinates again for every hash 11.7 for (3, 3) and 36 for (8, 8).
// -------------------------------------------------------------------------------------------------
constexpr int ORDER_THREADS = 256, ORDER_POINTS = ORDER_THREADS / 8, ORDER_MAX_N = 8192;

__device__ __forceinline__ uint32_t order_bits(float x) {          // key_xform of a float value
    uint32_t u = __float_as_uint(x);
    if (u == 0x80000000u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// Operation order of a projection as in lsh_hash_kernel; the hashes are added in four interleaved partial sums,
// which is the order torch.sum adds them in (fewer than four: simply left to right).
// DIM > 0: rows of up to ORDER_REGS coordinates, read once and kept in registers through all hashes; wider rows (DIM = 0) are read
// again for each four hashes.  NH > 0: up to four hashes, all at once (0: any number, four at a time).  alpha: [dim][nh4] in
// shared memory, nh4 the hash count rounded up to four, padded with zeros that are not added.
constexpr int ORDER_REGS = 8, ORDER_HASHES = 4;
__device__ __forceinline__ void stage_alpha(const float* __restrict__ alpha, int dim, int nh, int nh4, float* s_alpha) {
    for (int i = threadIdx.x; i < dim * nh4; i += blockDim.x) {
        const int d = i / nh4, j = i - d * nh4;
        s_alpha[i] = j < nh ? alpha[d * nh + j] : 0.f;
    }
}
__device__ __forceinline__ float hash_weight(int j) { return __int_as_float((127 + min(j, 127)) << 23); }      // 2^j
// NP points at c[0], c[1], ...: their loads and sums are independent chains.
template <int DIM, int NH, int NP>
__device__ __forceinline__ void ordering_key_norm(const float* const (&c)[NP], int dim, const float* s_alpha, int nh, int nh4, float (&key)[NP],
                                                  float (&norm)[NP]) {
    float x[NP][DIM > 0 ? DIM : 1], ss[NP], part[NP][4];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        ss[p] = part[p][0] = part[p][1] = part[p][2] = part[p][3] = 0.f;
#pragma unroll
        for (int d = 0; d < DIM; ++d) x[p][d] = __ldg(c[p] + d);
    }
    if (DIM > 0) {
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int d = 0; d < DIM; ++d) ss[p] = fmaf(x[p][d], x[p][d], ss[p]);
    } else {
        for (int d = 0; d < dim; ++d)
#pragma unroll
            for (int p = 0; p < NP; ++p) { const float v = __ldg(c[p] + d); ss[p] = fmaf(v, v, ss[p]); }
    }
    auto hashes = [&](int j0) {
        constexpr int U = NH > 0 ? NH : 4;
        float acc[NP][U];
        auto project = [&](int d, int p, float v, const float4& a) {
            const float w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int u = 0; u < U; ++u) acc[p][u] = d == 0 ? __fmul_rn(v, w[u]) : __fadd_rn(acc[p][u], __fmul_rn(v, w[u]));
        };
        const float4* ap = reinterpret_cast<const float4*>(s_alpha + j0);
        if (DIM > 0) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float4 a = ap[d * (nh4 >> 2)];
#pragma unroll
                for (int p = 0; p < NP; ++p) project(d, p, x[p][DIM > 0 ? d : 0], a);
            }
        } else {
            for (int d = 0; d < dim; ++d) {
                const float4 a = ap[d * (nh4 >> 2)];
#pragma unroll
                for (int p = 0; p < NP; ++p) project(d, p, __ldg(c[p] + d), a);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (NH > 0 || j0 + u < nh) {
                const float w = hash_weight(j0 + u);
#pragma unroll
                for (int p = 0; p < NP; ++p) part[p][u] = __fadd_rn(part[p][u], __fmul_rn(acc[p][u], w));
            }
    };
    if (NH > 0) hashes(0);
    else for (int j0 = 0; j0 < nh; j0 += 4) hashes(j0);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        norm[p] = sqrtf(ss[p]);
        key[p] = __fadd_rn(__fadd_rn(__fadd_rn(part[p][0], part[p][1]), part[p][2]), part[p][3]);
    }
}

template <int DIM, int NH>
__global__ void __launch_bounds__(ORDER_THREADS)
ordering_rank_kernel(const float* __restrict__ coords, const float* __restrict__ alpha, int dim, int nh,
                     const uint32_t* __restrict__ points, int row_words, int n, int64_t* __restrict__ idx,
                     uint32_t* __restrict__ ordered) {
    if (chain_wait()) return;
    extern __shared__ __align__(16) unsigned char order_smem[];
    const int nh4 = NH > 0 ? 4 : (nh + 3) & ~3;
    float* s_alpha = reinterpret_cast<float*>(order_smem);
    uint64_t* comp = reinterpret_cast<uint64_t*>(s_alpha + dim * nh4);      // [n]: key, norm
    __shared__ int s_pos[ORDER_POINTS];
    const int tid = threadIdx.x;
    const int64_t s0 = (int64_t)blockIdx.y * n;
    stage_alpha(alpha, dim, nh, nh4, s_alpha);
    __syncthreads();
    constexpr int NP = 2;
    for (int i0 = tid; i0 < n; i0 += NP * ORDER_THREADS) {
        const float* c[NP];
        float key[NP], norm[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) c[p] = coords + (s0 + min(i0 + p * ORDER_THREADS, n - 1)) * dim;
        ordering_key_norm<DIM, NH, NP>(c, dim, s_alpha, nh, nh4, key, norm);
#pragma unroll
        for (int p = 0; p < NP; ++p)
            if (i0 + p * ORDER_THREADS < n) comp[i0 + p * ORDER_THREADS] = ((uint64_t)order_bits(key[p]) << 32) | order_bits(norm[p]);
    }
    __syncthreads();
    const int p = blockIdx.x * ORDER_POINTS + (tid >> 3), part = tid & 7;
    const uint64_t mine = p < n ? comp[p] : 0;
    // before p an equal point counts, behind it only a smaller one does: two plain loops
    int cnt = 0;
    const int before = min(p, n);
    int j = part;
#pragma unroll 8
    for (; j < before; j += 8) cnt += comp[j] <= mine ? 1 : 0;
#pragma unroll 8
    for (; j < n; j += 8) cnt += comp[j] < mine ? 1 : 0;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (part == 0) {
        s_pos[tid >> 3] = cnt;
        if (p < n) idx[s0 + cnt] = p;
    }
    __syncthreads();
    const int first = blockIdx.x * ORDER_POINTS, m = min(ORDER_POINTS, n - first);
    for (int i = tid; i < m * row_words; i += ORDER_THREADS) {
        const int r = i / row_words, w = i - r * row_words;
        ordered[(s0 + s_pos[r]) * row_words + w] = points[(s0 + first + r) * row_words + w];
    }
}

template <int DIM>
__global__ void __launch_bounds__(256)
ordering_keys_kernel(const float* __restrict__ coords, const float* __restrict__ alpha, int dim, int nh, int64_t n,
                     float* __restrict__ keys, float* __restrict__ norms) {
    if (chain_wait()) return;
    extern __shared__ __align__(16) unsigned char order_smem[];
    float* s_alpha = reinterpret_cast<float*>(order_smem);
    const int nh4 = (nh + 3) & ~3;
    stage_alpha(alpha, dim, nh, nh4, s_alpha);
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const float* const c[1] = {coords + i * dim};
    float key[1], norm[1];
    ordering_key_norm<DIM, 0, 1>(c, dim, s_alpha, nh, nh4, key, norm);
    keys[i] = key[0];
    norms[i] = norm[0];
}

// The copy for a coordinate and a hash count: both known to the compiler up to 8 and 4, then the coordinates alone, then neither.
using OrderKernel = void (*)(const float*, const float*, int, int, const uint32_t*, int, int, int64_t*, uint32_t*);
template <int... D>
static OrderKernel order_kernel(int dim, int nh, std::integer_sequence<int, D...>) {
    static const OrderKernel some[ORDER_REGS][ORDER_HASHES + 1] = {{ordering_rank_kernel<D + 1, 0>, ordering_rank_kernel<D + 1, 1>, ordering_rank_kernel<D + 1, 2>,
                                                                    ordering_rank_kernel<D + 1, 3>, ordering_rank_kernel<D + 1, 4>}...};
    return dim <= ORDER_REGS ? some[dim - 1][nh <= ORDER_HASHES ? nh : 0] : ordering_rank_kernel<0, 0>;
}

}  // namespace lampa

using namespace lampa;

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

extern "C" int lampa_lsh_hash(const float* x, int64_t row_stride, int64_t head_stride, const float* alpha,
                              const float* beta, float w, int64_t N, int32_t heads, int32_t rounds,
                              int32_t dim, int32_t* ids, float* keys, int32_t* packed, void* stream) {
    if (!x || !alpha || !beta || N < 0 || heads <= 0 || rounds <= 0 || dim <= 0) return LAMPA_ERR_ARG;
    if (!(w > 0.f)) return LAMPA_ERR_ARG;
    if ((int64_t)heads * dim * rounds > HASH_MAX_PARAMS || rounds > 64 || heads > 31) return LAMPA_ERR_UNSUPPORTED;
    if (N == 0) return LAMPA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    // A round to a CTA where the rows alone leave the SMs short of warps (six CTAs of 256 rows each are most of what an SM holds):
    // the row is read again for each, from L2.  3 x 8 hashes of 60,000 rows: 2 us less of the event's 445.
    const int64_t rows = (N + HASH_THREADS - 1) / HASH_THREADS;
    const int per = rows < 6 * (int64_t)sm_count() ? 1 : rounds;
    const dim3 grid((unsigned)rows, (unsigned)((rounds + per - 1) / per));
    ProfScope prof("lsh_hash", st);
    if (dim == 6 && head_stride == 0)
        launch_chained(lsh_hash_kernel<6>, grid, HASH_THREADS, 0, st, x, row_stride, head_stride, alpha, beta, w, N, heads, rounds, dim, per, ids, keys, packed);
    else
        launch_chained(lsh_hash_kernel<0>, grid, HASH_THREADS, 0, st, x, row_stride, head_stride, alpha, beta, w, N, heads, rounds, dim, per, ids, keys, packed);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_segsort_workspace_bytes(int64_t n_total, size_t* bytes) {
    if (n_total < 0 || !bytes) return LAMPA_ERR_ARG;
    *bytes = 4 * align_up((size_t)n_total * 4, 256) + 256;
    return LAMPA_OK;
}

extern "C" int lampa_segsort_stable(const void* keys, int32_t key_type, int64_t n_total,
                                    const int64_t* seg_offsets, int32_t nseg, const int64_t* init,
                                    int64_t* perm, void* ws, size_t ws_bytes, int32_t* status, void* stream) {
    if (n_total < 0 || nseg <= 0 || (key_type != LAMPA_KEY_I32 && key_type != LAMPA_KEY_F32)) return LAMPA_ERR_ARG;
    if (n_total == 0) return LAMPA_OK;
    if (!keys || !perm || !ws) return LAMPA_ERR_ARG;
    if (!seg_offsets && n_total % nseg != 0) return LAMPA_ERR_ARG;
    if (n_total >= ((int64_t)1 << 32)) return LAMPA_ERR_UNSUPPORTED;
    size_t need;
    lampa_segsort_workspace_bytes(n_total, &need);
    if (ws_bytes < need || ((uintptr_t)ws & 15)) return LAMPA_ERR_WORKSPACE;
    const size_t stride = align_up((size_t)n_total * 4, 256);
    char* base = (char*)(((uintptr_t)ws + 255) / 256 * 256);
    uint32_t* k0 = (uint32_t*)base;
    uint32_t* k1 = (uint32_t*)(base + stride);
    uint32_t* i0 = (uint32_t*)(base + 2 * stride);
    uint32_t* i1 = (uint32_t*)(base + 3 * stride);
    ProfScope prof("segsort", (cudaStream_t)stream);
    return launch_segsort(keys, key_type, n_total, seg_offsets, nseg, init, perm, k0, k1, i0, i1, status, (cudaStream_t)stream);
}

// Counting costs n^2 / 2 comparisons per segment (about 0.14 us per million on this GPU), the two radix sorts 70 - 90 us
// whatever the size below some 10^5 points: up to 4 * 10^8 comparisons counting wins.
static bool ordering_counts(int32_t B, int64_t n) { return n <= ORDER_MAX_N && (double)B * n * n <= 4e8; }

extern "C" int lampa_lsh_ordering_workspace_bytes(int32_t B, int64_t n, size_t* bytes) {
    if (B <= 0 || n < 0 || !bytes) return LAMPA_ERR_ARG;
    *bytes = 256;
    if (ordering_counts(B, n)) return LAMPA_OK;
    size_t sort;
    lampa_segsort_workspace_bytes(B * n, &sort);
    *bytes = sort + 2 * align_up((size_t)B * n * 4, 256) + align_up((size_t)B * n * 8, 256) + 256;
    return LAMPA_OK;
}

extern "C" int lampa_lsh_ordering(const float* coords, const float* alpha, int32_t dim, int32_t num_hashes,
                                  const void* points, int64_t row_bytes, int32_t B, int64_t n, int64_t* idx,
                                  void* ordered, void* ws, size_t ws_bytes, int32_t* status, void* stream) {
    if (B <= 0 || n < 0 || dim <= 0 || num_hashes <= 0 || row_bytes <= 0 || (row_bytes & 3)) return LAMPA_ERR_ARG;
    if (n == 0) return LAMPA_OK;
    if (!coords || !alpha || !points || !idx || !ordered || !ws) return LAMPA_ERR_ARG;
    if ((int64_t)dim * num_hashes > HASH_MAX_PARAMS || B > 65535) return LAMPA_ERR_UNSUPPORTED;
    size_t need;
    lampa_lsh_ordering_workspace_bytes(B, n, &need);
    if (ws_bytes < need || ((uintptr_t)ws & 15)) return LAMPA_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const int params = dim * ((num_hashes + 3) & ~3) * 4;
    constexpr int params_most = 4 * HASH_MAX_PARAMS * 4;                 // one hash to a coordinate, padded to four
    if (ordering_counts(B, n) && row_bytes <= (1 << 20)) {
        const int smem = (int)n * 8 + params;
        const OrderKernel kernel = order_kernel(dim, num_hashes, std::make_integer_sequence<int, ORDER_REGS>());
        if (smem > 47 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ORDER_MAX_N * 8 + params_most) != cudaSuccess)
            return LAMPA_ERR_CUDA;
        ProfScope prof("lsh_ordering", st);
        launch_chained(kernel, dim3((unsigned)((n + ORDER_POINTS - 1) / ORDER_POINTS), (unsigned)B), ORDER_THREADS, smem, st,
            coords, alpha, dim, num_hashes, (const uint32_t*)points, (int)(row_bytes / 4), (int)n, idx, (uint32_t*)ordered);
        return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
    }
    const int64_t total = (int64_t)B * n;
    size_t sort;
    lampa_segsort_workspace_bytes(total, &sort);
    char* base = (char*)(((uintptr_t)ws + 255) / 256 * 256);
    float* keys = (float*)base;
    float* norms = (float*)(base + align_up((size_t)total * 4, 256));
    int64_t* by_norm = (int64_t*)(base + 2 * align_up((size_t)total * 4, 256));
    void* sws = (char*)by_norm + align_up((size_t)total * 8, 256);
    {
        ProfScope prof("lsh_ordering_keys", st);
        using Kernel = void (*)(const float*, const float*, int, int, int64_t, float*, float*);
        static const Kernel kernels[] = {ordering_keys_kernel<0>, ordering_keys_kernel<1>, ordering_keys_kernel<2>, ordering_keys_kernel<3>, ordering_keys_kernel<4>,
                                         ordering_keys_kernel<5>, ordering_keys_kernel<6>, ordering_keys_kernel<7>, ordering_keys_kernel<8>};
        const Kernel kernel = kernels[dim <= ORDER_REGS ? dim : 0];
        if (params > 47 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, params_most) != cudaSuccess)
            return LAMPA_ERR_CUDA;
        launch_chained(kernel, (unsigned)((total + 255) / 256), 256, params, st, coords, alpha, dim, num_hashes, total, keys, norms);
        if (cudaGetLastError() != cudaSuccess) return LAMPA_ERR_CUDA;
    }
    int rc = lampa_segsort_stable(norms, LAMPA_KEY_F32, total, nullptr, B, nullptr, by_norm, sws, sort, status, stream);
    if (rc == LAMPA_OK) rc = lampa_segsort_stable(keys, LAMPA_KEY_F32, total, nullptr, B, by_norm, idx, sws, sort, status, stream);
    if (rc != LAMPA_OK) return rc;
    return lampa_permute_rows(points, idx, nullptr, B, total, row_bytes, 0, ordered, status, stream);
}

extern "C" int lampa_permute_rows(const void* src, const int64_t* perm, const int64_t* seg_offsets,
                                  int32_t nseg, int64_t n_rows, int64_t row_bytes, int32_t scatter,
                                  void* dst, int32_t* status, void* stream) {
    if (n_rows < 0 || row_bytes <= 0 || (row_bytes & 3) || nseg <= 0) return LAMPA_ERR_ARG;
    if (n_rows == 0) return LAMPA_OK;
    if (!src || !perm || !dst) return LAMPA_ERR_ARG;
    if (!seg_offsets && n_rows % nseg != 0) return LAMPA_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const bool v16 = (row_bytes % 16 == 0) && (((uintptr_t)src | (uintptr_t)dst) % 16 == 0);
    const int64_t upr = v16 ? row_bytes / 16 : row_bytes / 4;
    const int64_t total = n_rows * upr;
    const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 32);
    ProfScope prof("permute_rows", st);
    if (v16)
        launch_chained(permute_rows_kernel<uint4>, grid, 256, 0, st, (const uint4*)src, perm, seg_offsets, nseg, n_rows, upr, scatter, (uint4*)dst, status);
    else
        launch_chained(permute_rows_kernel<uint32_t>, grid, 256, 0, st, (const uint32_t*)src, perm, seg_offsets, nseg, n_rows, upr, scatter, (uint32_t*)dst, status);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

extern "C" int lampa_invert_perm(const int64_t* perm, const int64_t* seg_offsets, int32_t nseg,
                                 int64_t n_total, int64_t* inv, int32_t* status, void* stream) {
    if (n_total < 0 || nseg <= 0) return LAMPA_ERR_ARG;
    if (n_total == 0) return LAMPA_OK;
    if (!perm || !inv) return LAMPA_ERR_ARG;
    if (!seg_offsets && n_total % nseg != 0) return LAMPA_ERR_ARG;
    const unsigned grid = (unsigned)std::min<int64_t>((n_total + 255) / 256, 148 * 32);
    ProfScope prof("invert_perm", (cudaStream_t)stream);
    launch_chained(invert_perm_kernel, grid, 256, 0, (cudaStream_t)stream, perm, seg_offsets, nseg, n_total, inv, status);
    return cudaGetLastError() == cudaSuccess ? LAMPA_OK : LAMPA_ERR_CUDA;
}

// -------------------------------------------------------------------------------------------------
// Sort without any caller- or library-side allocation: the four ping-pong buffers live in a
// fixed array that is part of the loaded module (24 MiB per GPU that loads the library, held
// until the process exits).  Host code cannot use the symbol g_sort_scratch as a pointer — on
// the host it is only a handle — so its device address is looked up once per device with
// cudaGetSymbolAddress and cached.
// -------------------------------------------------------------------------------------------------
namespace {
constexpr size_t kStaticSortStride = (size_t)LAMPA_SEGSORT_STATIC_MAX_KEYS * 4;   // bytes per buffer, multiple of 256
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
void* g_scratch_addr[kMaxDevices] = {nullptr};
}  // namespace

static __device__ __align__(256) unsigned char g_sort_scratch[4 * kStaticSortStride];

// Device address of g_sort_scratch on the CURRENT device (looked up on first use there).
static int static_sort_scratch(void** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return LAMPA_ERR_CUDA;
    if (dev < 0 || dev >= kMaxDevices) return LAMPA_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    if (g_scratch_addr[dev] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_sort_scratch) != cudaSuccess || p == nullptr) return LAMPA_ERR_CUDA;
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return LAMPA_OK;
}

extern "C" int lampa_segsort_stable_static(const void* keys, int32_t key_type, int64_t n_total,
                                           const int64_t* seg_offsets, int32_t nseg, const int64_t* init,
                                           int64_t* perm, int32_t* status, void* stream) {
    if (n_total < 0 || nseg <= 0 || (key_type != LAMPA_KEY_I32 && key_type != LAMPA_KEY_F32)) return LAMPA_ERR_ARG;
    if (n_total > (int64_t)LAMPA_SEGSORT_STATIC_MAX_KEYS) return LAMPA_ERR_TOO_LARGE;
    if (n_total == 0) return LAMPA_OK;
    if (!keys || !perm) return LAMPA_ERR_ARG;
    if (!seg_offsets && n_total % nseg != 0) return LAMPA_ERR_ARG;
    void* base_v = nullptr;
    const int rc = static_sort_scratch(&base_v);
    if (rc != LAMPA_OK) return rc;
    char* base = (char*)base_v;
    // No buffer needs clearing between calls: every pass writes positions [0, n) of its
    // destination pair before the next pass reads them, and nothing beyond n is ever read.
    ProfScope prof("segsort_static", (cudaStream_t)stream);
    return launch_segsort(keys, key_type, n_total, seg_offsets, nseg, init, perm, (uint32_t*)base,
                          (uint32_t*)(base + kStaticSortStride), (uint32_t*)(base + 2 * kStaticSortStride),
                          (uint32_t*)(base + 3 * kStaticSortStride), status, (cudaStream_t)stream);
}
