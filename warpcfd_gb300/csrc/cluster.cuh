// Thread-block-cluster primitives shared by the cluster-resident solvers: rank queries,
// the hardware cluster barrier, distributed-shared-memory loads and stores, and
// deterministic float-float reductions over the CTAs of a cluster (by that barrier or by messages).
#pragma once

#include "common.cuh"
#include "wait_clock.cuh"

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
// The cluster barrier of a reduction: warp 0 (which made the remote slot stores) arrives
// with release semantics, the other warps arrive relaxed, every thread waits with acquire.
// Everything the other warps wrote before the CTA's last __syncthreads happens before
// warp 0's release (the CTA barrier orders it, and the release is cumulative), so the
// other CTAs see it after their wait; a release by 32 instead of 1,024 threads.
__device__ __forceinline__ void cluster_sync_warp0_release() {
    if (threadIdx.x < 32)
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
    cluster_sync_warp0_release();
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

// ---- meetings of a cluster by messages
// A CTA tells another by an asynchronous remote store that completes bytes on the receiver's
// mbarrier, so that a reduction costs one trip of its value; the cluster's hardware barrier after
// remote stores costs their acknowledgement, the arrival and the release: 600 to 1,000 cycles
// more on 8 to 16 CTAs (per iteration of the CG, two reductions: 16 CTAs 2.71 -> 2.35 us, 8 CTAs
// 1.62 -> 1.49, 2 CTAs 1.49 -> 1.40).  What the barrier ordered follows from the values: a CTA's total leaves
// after a block barrier behind all its reads and writes of the pass, and a CTA goes on when it has
// every CTA's.  A cluster of one CTA needs block barriers only.  Waits are bounded.
constexpr int kClusterSums = 3;
constexpr unsigned kNobodyGone = ~0u;
struct ClusterFailure {
    int own;              // a wait of this CTA gave up (reductions for every thread)
    unsigned gone;        // a CTA that gave up in this reduction leaves at the next barrier of the cluster, or kNobodyGone
    unsigned gave_up[2];  // threads of this CTA that gave up on a mbarrier
};
template <int T, int SUMS>
struct ClusterShared {
    ff slots[2 * kClusterSums * 16];  // [parity][sum][CTA]
    ff sbuf[SUMS * T];
    ff res[kClusterSums];
    unsigned long long bar[2];  // by parity
    ClusterFailure failure;
};
struct ClusterMeet {
    ff *slots, *sbuf, *res;
    uint32_t bar, peer_slots, peer_bar;  // own mbarriers; slots and mbarriers of CTA `lane`
    ClusterFailure* failure;
    unsigned n, me, cs, width;           // reductions so far; width: 2^k >= cs
    uint64_t limit;                      // of a wait, ns
};

__device__ __forceinline__ bool mbarrier_try(uint32_t bar, unsigned parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Wait for the phase of one of this CTA's mbarriers, `limit` ns of polling at most.  Every thread of the CTA that
// waits for a phase gets the same answer, whichever gives up first: a thread whose time is up makes the
// mbarrier expect kGiveUpBytes that nobody sends and looks again.  Either the phase was complete before
// that, and then every thread sees it (and the next phase of this mbarrier is the one that cannot
// complete), or it never completes.  So a warp that goes on and a warp that leaves cannot part.
// The threads of a block add less than the 2^20 - 1 bytes that an mbarrier counts, and are counted in
// gave_up (null: a thread that waits alone and may just stop).
constexpr unsigned kGiveUpBytes = 512;  // more than the totals of a reduction (16 CTAs x 3 sums x 8)
__device__ __forceinline__ bool mbarrier_wait(uint32_t bar, unsigned parity, uint64_t limit, unsigned* gave_up) {
    if (mbarrier_try(bar, parity)) return true;
    WaitClock clock(global_ns());
    while (!mbarrier_try(bar, parity)) {
        if (!clock.over(global_ns(), limit)) continue;
        if (!gave_up) return false;
        atomicAdd(gave_up, 1u);
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(kGiveUpBytes) : "memory");
        return mbarrier_try(bar, parity);
    }
    return true;
}
// every thread; cluster_begin between this and the first reduction, cluster_end before leaving (no CTA
// leaves while its shared memory may be addressed)
template <int T, int SUMS>
__device__ __forceinline__ ClusterMeet cluster_meet(ClusterShared<T, SUMS>& s, uint64_t limit = kBarrierTimeoutNs) {
    ClusterMeet m;
    m.limit = limit;
    m.slots = s.slots;
    m.sbuf = s.sbuf;
    m.res = s.res;
    m.failure = &s.failure;
    m.bar = (uint32_t)__cvta_generic_to_shared(s.bar);
    m.n = 0;
    m.me = cluster_rank();
    m.cs = cluster_nranks();
    m.width = 1;
    while (m.width < m.cs) m.width *= 2;
    const unsigned peer = min((unsigned)(threadIdx.x & 31), m.cs - 1);
    m.peer_slots = map_rank(s.slots, peer);
    m.peer_bar = map_rank(s.bar, peer);
    if (threadIdx.x == 0) {
        s.failure = ClusterFailure{0, kNobodyGone, {0u, 0u}};
        for (int i = 0; i < 2; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(m.bar + 8 * i), "r"(1u) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    return m;
}
__device__ __forceinline__ void cluster_begin(const ClusterMeet& m) {
    if (m.cs > 1) cluster_sync_all();
}
// A barrier of the cluster inside a solve's loop, behind the same reduction in every CTA.  False when a
// CTA gave up in that reduction and stands in cluster_end: it leaves now, so this CTA leaves too, without
// cluster_end and without touching another CTA.  The same answer in every thread: a CTA that gives up
// later notes a later reduction.
__device__ __forceinline__ bool cluster_sync_met(const ClusterMeet& m) {
    cluster_sync_all();
    return *reinterpret_cast<volatile unsigned*>(&m.failure->gone) != m.n;
}
// Every thread, met: no wait of this CTA gave up.  Returns whether none of the cluster's did.  A CTA that
// gave up tells the others before it arrives, and goes when the totals still on their way to it have landed.
__device__ __forceinline__ bool cluster_end(const ClusterMeet& m, bool met) {
    if (m.cs == 1) return met;
    if (!met && threadIdx.x < m.cs)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_rank(&m.failure->gone, threadIdx.x)), "r"(m.n) : "memory");
    cluster_sync_all();
    if (!met && threadIdx.x == 0) {
        const unsigned p = (m.n - 1) & 1u;
        asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(m.bar + 8u * p),
                     "r"(m.failure->gave_up[p] * kGiveUpBytes)
                     : "memory");
        mbarrier_wait(m.bar + 8u * p, ((m.n - 1) >> 1) & 1u, m.limit, nullptr);
    }
    return *reinterpret_cast<volatile unsigned*>(&m.failure->gone) == kNobodyGone;
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
// cluster, the sums normalised, the same bits in every CTA: in every thread (ALL), else in warp
// 0 only.  Warp i merges value i over the CTA's threads (eight or sixteen per lane, pairwise,
// then by butterfly) and sends the total to every CTA; every warp of a small CTA (ALL, T = 256),
// warp i (ALL, T = 512) or warp 0 then merges the cs <= 16 totals.  FENCE: global memory
// written before is visible to the cluster after.  When the wait gave up: false in thread 0, which owns
// the scalars (not ALL); NaN in every sum of every thread of the CTA and cluster_gave_up true (ALL), so that
// the tests that a solver makes of its sums anyway find it.
template <int NV, int T, bool ALL, bool FENCE>
__device__ __forceinline__ bool cluster_reduce(ff (&v)[NV], ClusterMeet& m) {
    static_assert(NV <= kClusterSums, "three sums at most");
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const unsigned base = (m.n & 1u) * (kClusterSums * 16);
    const uint32_t bar = 8u * (m.n & 1u);
    const unsigned phase = (m.n >> 1) & 1u;
    ++m.n;
    const bool alone = m.cs == 1;
    if (t == 0 && !alone)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(m.bar + bar),
                     "r"(m.cs * NV * (unsigned)sizeof(ff))
                     : "memory");
#pragma unroll
    for (int i = 0; i < NV; ++i) m.sbuf[i * T + t] = v[i];
    __syncthreads();
    bool met = true;
    if (wid < NV) {
        ff y[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) y[k] = m.sbuf[wid * T + 32 * k + lane];
        if constexpr (T == 512) {
#pragma unroll
            for (int k = 0; k < 8; ++k) ff_merge(y[k], m.sbuf[wid * T + 256 + 32 * k + lane]);
        }
        ff_tree(y);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ff_shfl_merge(y[0], o);
        if (alone) {
            if (lane == 0) m.slots[base + wid * 16] = y[0];
        } else if ((unsigned)lane < m.cs) {
            if constexpr (FENCE) __threadfence();
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(
                             m.peer_slots + (base + wid * 16 + m.me) * (unsigned)sizeof(ff)),
                         "f"(y[0].hi), "f"(y[0].lo), "r"(m.peer_bar + bar)
                         : "memory");
        }
    }
    const unsigned q = lane & (m.width - 1);
    if (alone) __syncthreads();
    if constexpr (ALL && T == 512) {
        if (wid < NV) {
            ff y = ff_zero();
            if (alone || mbarrier_wait(m.bar + bar, phase, m.limit, &m.failure->gave_up[(m.n - 1) & 1u])) {
                if (q < m.cs) y = m.slots[base + wid * 16 + q];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    if ((unsigned)o < m.width) ff_shfl_merge(y, o);
            } else {
                *reinterpret_cast<volatile int*>(&m.failure->own) = 1;
                y = ff{__uint_as_float(0x7fffffffu), 0.0f};
            }
            if (lane == 0) m.res[wid] = y;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = m.res[i];
    } else if (ALL || wid == 0) {
        if (!alone && !mbarrier_wait(m.bar + bar, phase, m.limit, &m.failure->gave_up[(m.n - 1) & 1u])) {
            if constexpr (ALL) {
                *reinterpret_cast<volatile int*>(&m.failure->own) = 1;
                // this CTA's own total among them is long there and stays NaN
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    if (q < m.cs) m.slots[base + i * 16 + q] = ff{__uint_as_float(0x7fffffffu), 0.0f};
            } else {
                met = false;
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = q < m.cs ? m.slots[base + i * 16 + q] : ff_zero();
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
            if ((unsigned)o < m.width)  // the same in every CTA; merging nothing changes nothing
#pragma unroll
                for (int i = 0; i < NV; ++i) ff_shfl_merge(v[i], o);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = ff_norm(v[i]);
    return met;
}

// after a reduction for every thread (ALL) whose sums are NaN, or after the last one
__device__ __forceinline__ bool cluster_gave_up(const ClusterMeet& m) {
    return *reinterpret_cast<volatile int*>(&m.failure->own) != 0;
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
