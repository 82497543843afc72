// Thread-block-cluster primitives shared by the cluster-resident solvers: rank queries,
// the hardware cluster barrier, distributed-shared-memory loads and stores, and a
// deterministic float-float reduction over the CTAs of a cluster.
#pragma once

#include "common.cuh"

namespace wcfd {

constexpr int CBS = kClusterBlock;

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_nranks() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The cluster barrier of a reduction: the first n warps (which made the remote slot stores)
// arrive with release semantics, the other warps arrive relaxed, every thread waits with
// acquire.  Everything the other warps wrote before the CTA's last __syncthreads happens
// before warp 0's release (the CTA barrier orders it, and the release is cumulative), so the
// other CTAs see it after their wait; a release by few threads instead of all.
template <int N>
__device__ __forceinline__ void cluster_sync_release() {
    if (threadIdx.x < 32 * N)
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    else
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `p` (a pointer into this CTA's shared memory) in CTA `rank`
__device__ __forceinline__ uint32_t map_rank(const void* p, unsigned rank) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// Loads stay ordered against the cluster barrier (both are volatile asm) but carry no
// memory clobber, so the compiler may keep several of them in flight.
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void st_cluster_v2f32(uint32_t addr, float a, float b) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" :: "r"(addr), "f"(a), "f"(b) : "memory");
}

// Sum NV float-float values over the CTAs of the cluster, result (float-float, the same bits
// in every CTA) in thread 0 only.  The block stage is a shared-memory tree instead of a
// butterfly in every warp, so that most warps issue one store and wait: every thread
// stores its values into sbuf [NV][CBS]; threads 0..255 merge four each ((t + t+256) +
// (t+512 + t+768), a pairwise tree so the merges overlap); warp 0 merges eight each
// (l, l+32, ..., l+224, again pairwise), then by butterfly, and stores the CTA total into
// slot `me` of every CTA (DSMEM); after the cluster barrier (release by warp 0 only)
// warp 0 merges the cs <= 16 slots in rank order (four butterfly levels).  One cluster
// barrier and two __syncthreads; slots [2][NV][16] are double-buffered by `parity`.
template <int NV>
__device__ __forceinline__ void cluster_reduce_tree(const ff (&acc)[NV], ff (&out)[NV], ff* sbuf, ff* slots,
                                                    unsigned parity, unsigned me, unsigned cs) {
    static_assert(CBS == 1024, "the tree assumes 1024 threads");
    const int t = threadIdx.x;
#pragma unroll
    for (int i = 0; i < NV; ++i) sbuf[i * CBS + t] = acc[i];
    __syncthreads();
    if (t < 256) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const ff* b = sbuf + i * CBS + t;
            ff x0 = b[0], x1 = b[256], x2 = b[512], x3 = b[768];
            ff_merge(x0, x1);
            ff_merge(x2, x3);
            ff_merge(x0, x2);
            sbuf[i * CBS + t] = x0;  // only thread t reads or writes position t in this stage
        }
    }
    __syncthreads();
    if (t < 32) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const ff* b = sbuf + i * CBS + t;
            ff y[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) y[k] = b[32 * k];
#pragma unroll
            for (int k = 0; k < 8; k += 2) ff_merge(y[k], y[k + 1]);
            ff_merge(y[0], y[2]);
            ff_merge(y[4], y[6]);
            ff_merge(y[0], y[4]);
            ff x = y[0];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ff_shfl_merge(x, o);
            if ((unsigned)t < cs) st_cluster_v2f32(map_rank(slots + (parity * NV + i) * 16 + me, t), x.hi, x.lo);
        }
    }
    cluster_sync_release<1>();
    if (t < 32) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            ff y = (unsigned)t < cs ? slots[(parity * NV + i) * 16 + t] : ff_zero();
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ff_shfl_merge(y, o);  // lanes 0..15 hold the cs <= 16 slots
            if (t == 0) out[i] = y;
        }
    }
}

// Row of thread t's u-th in a CTA of T = 256 or 512 threads, and the number of accumulators it
// adds its products to (row u to accumulator u % kClusterAcc): chosen so that merging a thread's
// accumulators (cluster_merge) and then the threads' (below) is the tree of cluster_reduce_tree
// over 1,024 threads that own the rows t, t + 1024, ... -- the same sums bit for bit whatever
// T and the rows per thread are, so a case's result does not depend on the kernel that its
// batch's largest case asks for.
template <int T>
__device__ __forceinline__ int cluster_row(int t, int u) {
    static_assert(T == 256 || T == 512, "the two block sizes");
    if constexpr (T == 256) return t + 256 * u;
    else return (t & 255) + ((t >> 8) << 9) + 256 * (u & 1) + 1024 * (u >> 1);
}
template <int T>
constexpr int kClusterAcc = T == 256 ? 4 : 2;
template <int T>
__device__ __forceinline__ ff cluster_merge(ff (&acc)[kClusterAcc<T>]) {
    ff_merge(acc[0], acc[1]);
    if constexpr (T == 256) {
        ff_merge(acc[2], acc[3]);
        ff_merge(acc[0], acc[2]);
    }
    return acc[0];
}

// Sum NV float-float values (cluster_merge of each thread's accumulators) over the CTAs of the
// cluster, the sums (normalised, the same bits) in every thread.  Warp i merges value i over
// the CTA's threads (eight or sixteen per lane, pairwise, then by butterfly) and stores the
// total into a slot of every CTA (DSMEM); the cluster barrier follows.  With eight warps every
// warp then merges the cs <= 16 slots, so that no block barrier and no broadcast follows (the
// eight warps form the scalars redundantly); with sixteen, warp i merges value i and a block
// barrier passes the sums on.  (Every warp storing its own total to every CTA, eight times the
// remote stores: 2,000-2,400 cycles a reduction on 16 CTAs against 1,900.)
// sbuf: [kClusterSums][T]; slots: [2][kClusterSums][16], double-buffered by `parity`; remote:
// the address of slots in CTA `lane`; res: [kClusterSums] (T = 512).
constexpr int kClusterSums = 3;
template <int NV, int T>
__device__ __forceinline__ void cluster_reduce_all(ff (&v)[NV], ff* sbuf, const ff* slots, ff* res, uint32_t remote,
                                                   unsigned parity, unsigned me, unsigned cs) {
    static_assert(NV <= kClusterSums, "three sums at most");
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const unsigned base = parity * (kClusterSums * 16);
#pragma unroll
    for (int i = 0; i < NV; ++i) sbuf[i * T + t] = v[i];
    __syncthreads();
    if (wid < NV) {
        ff y[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) y[k] = sbuf[wid * T + 32 * k + lane];
        if constexpr (T == 512) {
#pragma unroll
            for (int k = 0; k < 8; ++k) ff_merge(y[k], sbuf[wid * T + 256 + 32 * k + lane]);
        }
        ff_tree(y);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ff_shfl_merge(y[0], o);
        if ((unsigned)lane < cs)
            st_cluster_v2f32(remote + (base + wid * 16 + me) * (unsigned)sizeof(ff), y[0].hi, y[0].lo);
    }
    cluster_sync_release<NV>();
    if constexpr (T == 256) {
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = (unsigned)(lane & 15) < cs ? slots[base + i * 16 + (lane & 15)] : ff_zero();
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < NV; ++i) ff_shfl_merge(v[i], o);
    } else {
        if (wid < NV) {
            ff y = (unsigned)(lane & 15) < cs ? slots[base + wid * 16 + (lane & 15)] : ff_zero();
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ff_shfl_merge(y, o);
            if (lane == 0) res[wid] = y;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = res[i];
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = ff_norm(v[i]);
}

__device__ __forceinline__ float ld_shared_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 ld_shared_f32x2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 ld_cluster_f32x2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}

}  // namespace wcfd
