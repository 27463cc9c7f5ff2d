// Shared device/host helpers for the sm_100a kernels of the LSH + gated-delta path.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../include/lampa_b200.h"

namespace lampa {

constexpr int CHUNK = 64;          // tokens per chunk (the reference's BT, gated_delta_rule_ori.py:41)
constexpr int ELL0 = 7;            // intra-chunk levels 0..6 (get_num_levels(64, 2), base.py:37-38)

// ---- status word (device int32[4]): [0] code, [1] where, [2..3] detail -----------------------
__device__ __forceinline__ void set_status(int32_t* status, int code, int where, int detail) {
    if (status != nullptr && atomicCAS(status, 0, code) == 0) {
        status[1] = where;
        status[2] = detail;
    }
}

// ---- small numeric helpers ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);     // .x = lo (low 16 bits), .y = hi
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(v);
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// dtype codes of the C ABI
template <int DT> struct Elem;
template <> struct Elem<LAMPA_BF16> {
    using T = __nv_bfloat16;
    static __device__ __forceinline__ float ld(const void* p, size_t i) { return __bfloat162float(((const T*)p)[i]); }
    static __device__ __forceinline__ void st(void* p, size_t i, float v) { ((T*)p)[i] = __float2bfloat16_rn(v); }
};
template <> struct Elem<LAMPA_F16> {
    using T = __half;
    static __device__ __forceinline__ float ld(const void* p, size_t i) { return __half2float(((const T*)p)[i]); }
    static __device__ __forceinline__ void st(void* p, size_t i, float v) { ((T*)p)[i] = __float2half_rn(v); }
};
template <> struct Elem<LAMPA_F32> {
    using T = float;
    static __device__ __forceinline__ float ld(const void* p, size_t i) { return ((const T*)p)[i]; }
    static __device__ __forceinline__ void st(void* p, size_t i, float v) { ((T*)p)[i] = v; }
};
__device__ __forceinline__ float load_as_float(const void* p, size_t i, int dt) {
    if (dt == LAMPA_BF16) return Elem<LAMPA_BF16>::ld(p, i);
    if (dt == LAMPA_F16) return Elem<LAMPA_F16>::ld(p, i);
    return Elem<LAMPA_F32>::ld(p, i);
}
__device__ __forceinline__ void store_from_float(void* p, size_t i, float v, int dt) {
    if (dt == LAMPA_BF16) Elem<LAMPA_BF16>::st(p, i, v);
    else if (dt == LAMPA_F16) Elem<LAMPA_F16>::st(p, i, v);
    else Elem<LAMPA_F32>::st(p, i, v);
}
__host__ __device__ __forceinline__ int dtype_bytes(int dt) { return dt == LAMPA_F32 ? 4 : 2; }

// ---- warp-level tensor-core primitives (bf16 in, fp32 accumulate) ------------------------------
// D(16x8) += A(16x16, row) * B(16x8, col).  Fragment ownership (g = lane/4, t = lane%4):
//   a0:(g, 2t..2t+1) a1:(g+8, 2t..) a2:(g, 2t+8..) a3:(g+8, 2t+8..)
//   b0:(k=2t..2t+1, n=g) b1:(k=2t+8.., n=g)      c0,c1:(g, 2t..2t+1) c2,c3:(g+8, 2t..2t+1)
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// A fragment (16 rows m0.., 16 k-columns k0..) from row-major smem A[m][k] (pitch lda elements).
__device__ __forceinline__ void load_a(uint32_t (&a)[4], const __nv_bfloat16* s, int lda, int m0, int k0, int lane) {
    const int mi = lane >> 3, r = lane & 7;
    ldsm_x4(a, smem_u32(s + (size_t)(m0 + r + (mi & 1) * 8) * lda + k0 + (mi >> 1) * 8));
}
// A fragment when smem holds A transposed: At[k][m] (pitch lda).
__device__ __forceinline__ void load_a_t(uint32_t (&a)[4], const __nv_bfloat16* s, int lda, int m0, int k0, int lane) {
    const int mi = lane >> 3, r = lane & 7;
    ldsm_x4_t(a, smem_u32(s + (size_t)(k0 + r + (mi >> 1) * 8) * lda + m0 + (mi & 1) * 8));
}
// B fragments for two adjacent n-tiles (n0..n0+15) and one k-step (k0..k0+15), smem holds Bt[n][k]
// (n rows, k contiguous).  b[0],b[1] = (b0,b1) of n-tile n0; b[2],b[3] = n-tile n0+8.
__device__ __forceinline__ void load_b(uint32_t (&b)[4], const __nv_bfloat16* s, int ldb, int n0, int k0, int lane) {
    const int mi = lane >> 3, r = lane & 7;
    ldsm_x4(b, smem_u32(s + (size_t)(n0 + r + (mi >> 1) * 8) * ldb + k0 + (mi & 1) * 8));
}
// Same fragments when smem holds B[k][n] (k rows, n contiguous).
__device__ __forceinline__ void load_b_t(uint32_t (&b)[4], const __nv_bfloat16* s, int ldb, int n0, int k0, int lane) {
    const int mi = lane >> 3, r = lane & 7;
    ldsm_x4_t(b, smem_u32(s + (size_t)(k0 + r + (mi & 1) * 8) * ldb + n0 + (mi >> 1) * 8));
}

// acc[NT8][4] (16 x 8*NT8) += A[m0:m0+16, 0:k_end) * B[0:k_end, n0:n0+n_end)
// k_end / n_end (warp-uniform, multiples of 16) cut the loops short for triangular operands.
template <int NT8, int KDIM, bool A_T, bool B_T>
__device__ __forceinline__ void warp_gemm(float (&acc)[NT8][4], const __nv_bfloat16* sA, int lda, int m0,
                                          const __nv_bfloat16* sB, int ldb, int n0, int lane,
                                          int k_end = KDIM, int n_end = NT8 * 8) {
    static_assert(NT8 % 2 == 0 && KDIM % 16 == 0, "tile shape");
#pragma unroll
    for (int k0 = 0; k0 < KDIM; k0 += 16) {
        if (k0 < k_end) {
            uint32_t a[4];
            if (A_T) load_a_t(a, sA, lda, m0, k0, lane); else load_a(a, sA, lda, m0, k0, lane);
#pragma unroll
            for (int nt = 0; nt < NT8; nt += 2) {
                if (nt * 8 < n_end) {
                    uint32_t b[4];
                    if (B_T) load_b_t(b, sB, ldb, n0 + nt * 8, k0, lane); else load_b(b, sB, ldb, n0 + nt * 8, k0, lane);
                    mma16816(acc[nt], a, b[0], b[1]);
                    mma16816(acc[nt + 1], a, b[2], b[3]);
                }
            }
        }
    }
}

// ---- mbarrier + bulk async copy (TMA, untiled form) -------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" :: "r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: gives up after `budget` polls (each poll may itself block for a while in hardware;
// the default budget is 2^22), records the failure and lets the caller carry on so that no barrier
// is left unbalanced.  A thread that has given up once (`dead`) does not wait again: it runs to the
// end of its loop, issues nothing new and drains what it has in flight with mbar_drain.
constexpr int MBAR_POLLS = 1 << 22;
int poll_budget();                 // of the launches that follow (host): MBAR_POLLS unless lampa_debug_set_poll_budget lowered it
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, bool& dead, int32_t* status, int where, int budget) {
    if (dead) return false;
    for (int i = 0; i < budget; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    dead = true;
    set_status(status, LAMPA_ERR_TIMEOUT, where, (int)parity);
    return false;
}
// Wait for an asynchronous operation that was already started (a bulk copy into this CTA's shared
// memory, a committed MMA group) before the CTA gives its shared / tensor memory back; always the
// full budget, whatever made the thread give up earlier.
__device__ __forceinline__ bool mbar_drain(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < MBAR_POLLS; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// global -> shared bulk copy; dst/src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// shared -> global bulk copy (same alignment rules).  The writer threads make their shared-memory
// stores visible to the async proxy first (fence_async_shared, then a barrier); the issuing thread
// commits the group and, before the buffer is reused or the CTA exits, waits until it has been read.
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n"
                 :: "l"(dst), "r"(smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }

// ---- launches that overlap the end of the kernel before them -------------------------------------
// A call is a chain of short kernels, and between two ordinary launches of a stream the GPU drains, flushes and only then
// starts the next grid.  launch_chained() lets the next kernel's CTAs start when the last CTA of the one before has left;
// chain_wait() holds them until that kernel is complete and its results are visible.  Two rules make this the same as stream
// order for whoever reads or writes memory: a kernel touches global memory (and allocates tensor memory) only behind
// chain_wait(), and every CTA passes it.  chain_wait() returns false, from the same assembly as the wait:
// `if (chain_wait()) return;` makes all that follows depend on it, so that no load that counts as invariant
// (const __restrict__, __ldg) can be moved in front of it.
// 6,144 tokens, 4 heads: 58.4 -> 50.5 us over four launches; one 9,001-hit event through the model: 475 -> 420 over 27.
// A kernel may let the next one start before its own end (chain_signal, once all its CTAs have passed it or left).  That is
// for kernels that leave most of the GPU idle and for a next one that can do without them: everywhere else the next grid only
// fills the SMs that happen to be free, two or three CTAs to an SM beside idle ones (56 and 447 us, and 486 instead of 463 for a
// 60,000-hit event).  chain_signal comes behind chain_wait: what the kernel was waiting for is complete then.  The next one may use
// it before its own wait only where chain_seen() says so, and a CTA of it still waits before it ends, so that its end means
// theirs.  That a grid has been let in orders no memory by itself: the first thread of the signalling kernel, for which griddepcontrol.wait
// has made all of it visible, therefore leaves the call's number in a word of the call's workspace with a release, and a
// kernel that reads that number with an acquire comes behind it in the memory model's causality order.  One that does not find
// it waits as any other.  (The last kernel of the call clears the word behind its wait: a replayed call has the same number.)
__device__ __forceinline__ bool chain_wait() {
    uint32_t never;
    asm volatile("griddepcontrol.wait;\n mov.u32 %0, 0;\n" : "=r"(never) :: "memory");
    return never != 0;
}
__device__ __forceinline__ void chain_signal() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// All threads of the grid, behind chain_wait().  One thread signals for its CTA.  The word is on its way when the first one does, and
// there before the next grid's CTAs are (a fence between the two only makes everybody wait: 0.4 us of a prefill's 65).
__device__ __forceinline__ void chain_signal(unsigned long long* word, unsigned long long call) {
    if (threadIdx.x != 0) return;
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
        asm volatile("st.release.gpu.global.u64 [%0], %1;\n" :: "l"(word), "l"(call) : "memory");
    }
    chain_signal();
}
// All threads of a CTA: whether what was complete in front of the kernel that signalled with `call` may be used, by bulk copies too
__device__ __forceinline__ bool chain_seen(const unsigned long long* word, unsigned long long call) {
    unsigned long long v = 0;
    if (threadIdx.x == 0) asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(word) : "memory");
    const bool seen = __syncthreads_or(threadIdx.x == 0 && v == call) != 0;
    asm volatile("fence.proxy.async.global;\n" ::: "memory");
    return seen;
}
inline cudaLaunchAttribute chained_attribute() {
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    return at;
}
template <typename... Params, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at = chained_attribute();
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// SMs of the current device
inline int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    return n;
}

// Opt-in to `bytes` of dynamic shared memory for a kernel, once per device (`ready`: one bit per device, static at the call).
// The opt-in is the kernel's, not the launch's: where the size varies, every call opts in to the largest one that the entry point
// accepts, or a thread with a smaller size would take the opt-in of another one's launch back in front of it.
constexpr int MAX_SMEM = 227 * 1024;                     // dynamic shared memory of a kernel that has no other
template <typename K>
inline bool allow_smem(std::atomic<uint64_t>& ready, K kernel, int bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (bit && (ready.load(std::memory_order_relaxed) & bit)) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    ready.fetch_or(bit, std::memory_order_relaxed);
    return true;
}

// Largest offset up to and including this thread's, over the threads of the CTA in order and, through `before`, the passes
// before; offsets that leave [0, total] do not count.  A packed sequence in order begins at this offset.  All threads call it
// (`wtop`: one word per warp, free again behind the caller's next barrier).
template <int THREADS>
__device__ __forceinline__ int64_t highest_offset(int64_t t, int64_t total, int64_t& before, int64_t* wtop) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t top = t <= total ? t : 0;                       // (a negative one is never the largest)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) top = max(top, __shfl_up_sync(0xffffffffu, top, o));
    if (lane == 31) wtop[warp] = top;
    __syncthreads();
    top = max(top, before);
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        if (w < warp) top = max(top, wtop[w]);
        before = max(before, wtop[w]);
    }
    return top;
}

// index of the sequence whose [off[s], off[s+1]) contains x (off non-decreasing; empty ranges skipped)
__device__ __forceinline__ int find_seq(const int32_t* off, int nseq, int x) {
    int lo = 0, hi = nseq;            // invariant: off[lo] <= x < off[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}

}  // namespace lampa
