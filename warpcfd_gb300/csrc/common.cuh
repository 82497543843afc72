// Shared device helpers for libwcfd: vector loads, block/grid reductions in fp64 and a
// bounded grid barrier for the persistent (cooperatively launched) solver kernels.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>
#include <climits>

#include "wcfd.h"

namespace wcfd {

constexpr int kBlock = 256;      // threads of the one-thread-per-face/cell kernels
constexpr int kMaxFieldBlock = 512;  // largest block of the batched field kernels (a launch parameter)
constexpr int kSolverBlock = 1024;  // threads of the barrier check, whose residency caps the Krylov grids
constexpr int kCgBlock = 512;       // threads of the persistent CG and BiCGSTAB (one block per SM)
constexpr int kMaxSlots = 6;     // faces per cell (hex)
// face reference of a null slot: a cell of a mixed mesh with fewer faces than the
// mesh's faces_per_cell (a wedge or a tetrahedron among hexes); its weights are zero
constexpr int kNullSlot = INT_MIN;
constexpr int kClusterBlock = 1024;  // threads per CTA of the cluster-resident solver

// the slot bits of a wcfd_mesh.slot_mask in use, else 0
__host__ __device__ __forceinline__ unsigned slot_bits(const wcfd_mesh& m) {
    return (m.slot_mask & 0xffff0000) == WCFD_SLOT_MASK ? (unsigned)m.slot_mask & 0xffffu : 0u;
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float comp(const float4& v, int o) {
    return o == 0 ? v.x : (o == 1 ? v.y : (o == 2 ? v.z : v.w));
}
__device__ __forceinline__ void set_comp(float4& v, int o, float x) {
    if (o == 0) v.x = x; else if (o == 1) v.y = x; else if (o == 2) v.z = x; else v.w = x;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Longest a block waits at a grid barrier before it gives up and flags
// WCFD_BARRIER_TIMEOUT (a healthy wait is one solver phase: microseconds).
constexpr uint64_t kBarrierTimeoutNs = 1500ull * 1000ull * 1000ull;

// ---------------------------------------------------------------------------------
// fp64-accurate dot products without per-element fp64 arithmetic.
//
// GB300 executes fp64 at about 1/64 of its fp32 rate, so a cast and an fp64 FMA per
// element would dominate a bandwidth-bound Krylov phase.  Instead each product is formed
// exactly as an unevaluated sum h + r (TwoProduct with an FMA) and accumulated in
// float-float arithmetic (Knuth's TwoSum), the "Dot2" scheme of Ogita, Rump and Oishi,
// "Accurate sum and dot product", SIAM J. Sci. Comput. 26 (2005): the result is as accurate
// as if it were computed in twice the working precision.  Totals are merged in float-float
// across warps, blocks and CTAs in a fixed order (TwoSum merges are exact up to the low
// word) and converted to fp64 once, by one thread: a full-warp fp64 instruction is itself
// expensive on GB300.
// __fmul_rn / __fadd_rn keep the compiler from contracting the error-free transforms.
struct ff {
    float hi, lo;
};

__device__ __forceinline__ ff ff_zero() { return ff{0.0f, 0.0f}; }

// acc += a * b
__device__ __forceinline__ void ff_fma(ff& acc, float a, float b) {
    const float h = __fmul_rn(a, b);
    const float r = fmaf(a, b, -h);
    const float s = __fadd_rn(acc.hi, h);
    const float bb = __fsub_rn(s, acc.hi);
    const float q = __fadd_rn(__fsub_rn(acc.hi, __fsub_rn(s, bb)), __fsub_rn(h, bb));
    acc.hi = s;
    acc.lo = __fadd_rn(acc.lo, __fadd_rn(q, r));
}

// a += b (symmetric: merging a into b gives the same bits, so butterfly shuffles agree)
__device__ __forceinline__ void ff_merge(ff& a, const ff& b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    const float q = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    a.hi = s;
    a.lo = __fadd_rn(__fadd_rn(a.lo, b.lo), q);
}

__device__ __forceinline__ void ff_shfl_merge(ff& v, int o) {
    ff t;
    t.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
    t.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
    ff_merge(v, t);
}

__device__ __forceinline__ double ff_to_double(const ff& v) { return (double)v.hi + (double)v.lo; }

// Scalar float-float arithmetic for the Krylov recurrences.  One dependent fp64 operation
// costs about 64 cycles on GB300 and an fp64 division about 600, against about 5 and 50
// for fp32, and the thread that forms alpha and beta holds up every other thread of the
// solve; so alpha = rz / pq, beta = rz' / rz and the stop test are evaluated on the
// float-float sums directly.

// (hi, lo) with |lo| <= ulp(hi) / 2 (Dekker's fast two-sum; the sums above keep |lo| small)
__device__ __forceinline__ ff ff_norm(const ff& a) {
    const float s = __fadd_rn(a.hi, a.lo);
    return ff{s, __fsub_rn(a.lo, __fsub_rn(s, a.hi))};
}
__device__ __forceinline__ ff ff_from_double(double d) {
    const float h = (float)d;
    return ff{h, (float)(d - (double)h)};
}
// a > b and a <= b for normalised operands (both false when either is NaN, as for fp64)
__device__ __forceinline__ bool ff_gt(const ff& a, const ff& b) {
    return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo);
}
__device__ __forceinline__ bool ff_le(const ff& a, const ff& b) {
    return a.hi < b.hi || (a.hi == b.hi && a.lo <= b.lo);
}
// a + b of two floats as a normalised float-float (TwoSum)
__device__ __forceinline__ ff ff_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return ff{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
// a * b in float-float (TwoProduct of the high words plus the cross terms)
__device__ __forceinline__ ff ff_mul(const ff& a, const ff& b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    return ff_norm(ff{p, e});
}
// a / b in float-float (see ff_div_to_float); b.hi != 0
__device__ __forceinline__ ff ff_div(const ff& an, const ff& bn) {
    const ff a = ff_norm(an), b = ff_norm(bn);
    const float q1 = __fdiv_rn(a.hi, b.hi);
    const float p = __fmul_rn(q1, b.hi);
    const float e = fmaf(q1, b.hi, -p);
    const float rh = __fsub_rn(a.hi, p);
    const float rl = __fsub_rn(__fsub_rn(a.lo, e), __fmul_rn(q1, b.lo));
    const float q2 = __fdiv_rn(__fadd_rn(rh, rl), b.hi);
    return ff_two_sum(q1, q2);
}
__device__ __forceinline__ float ff_to_float(const ff& a) { return __fadd_rn(a.hi, a.lo); }

// a / b rounded to fp32: a float quotient q1, the remainder a - q1 b formed exactly
// (TwoProduct; a.hi - q1 b.hi is exact by Sterbenz's lemma), one correction q2; q1 + q2
// agrees with a / b to about 2^-46 before the final rounding.  b.hi != 0.
__device__ __forceinline__ float ff_div_to_float(const ff& an, const ff& bn) {
    const ff a = ff_norm(an), b = ff_norm(bn);
    const float q1 = __fdiv_rn(a.hi, b.hi);
    const float p = __fmul_rn(q1, b.hi);
    const float e = fmaf(q1, b.hi, -p);
    const float rh = __fsub_rn(a.hi, p);
    const float rl = __fsub_rn(__fsub_rn(a.lo, e), __fmul_rn(q1, b.lo));
    const float q2 = __fdiv_rn(__fadd_rn(rh, rl), b.hi);
    return __fadd_rn(q1, q2);
}

// d p + sum_j o[j] g[j] of one matrix row, rounded as the compiler contracts the plain loop over
// a row whose off-diagonals stand from slot 0 on: the first product is rounded, everything
// after it is a fused multiply-add.  With the off-diagonals in place (in_place,
// wcfd_mesh.slot_mask) a row beside a boundary may have its padding (coefficient 0) before its
// first neighbour; that neighbour's product is then the rounded one, so that the layout does
// not show in the result.
template <int W>
__device__ __forceinline__ float row_product(float d, float p, const float (&o)[W > 0 ? W : 1],
                                             const float (&g)[W > 0 ? W : 1], bool in_place) {
    if constexpr (W == 0) return __fmul_rn(d, p);
    float q = fmaf(d, p, __fmul_rn(o[0], g[0]));
#pragma unroll
    for (int j = 1; j < W; ++j) q = fmaf(o[j], g[j], q);
    if (in_place && o[0] == 0.0f) {
        bool begun = false;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            q = begun ? fmaf(o[j], g[j], q) : fmaf(d, p, __fmul_rn(o[j], g[j]));
            begun = begun || o[j] != 0.0f;
        }
    }
    return q;
}

// Columns of row i, slot by slot: from the int16 offsets (wcfd_mesh.ell_dcol) when the mesh has
// them (half the bytes), else the int32 columns.  Every load is issued before the first use.
template <int W>
__device__ __forceinline__ void ell_columns(int (&c)[W > 0 ? W : 1], const int* __restrict__ col,
                                            const int16_t* __restrict__ dcol, int C, int i) {
    if (dcol) {
#pragma unroll
        for (int j = 0; j < W; ++j) c[j] = __ldcs(dcol + (size_t)j * C + i);
#pragma unroll
        for (int j = 0; j < W; ++j) c[j] += i;
    } else {
#pragma unroll
        for (int j = 0; j < W; ++j) c[j] = __ldcs(col + (size_t)j * C + i);
    }
}

// Block total of NV float-float accumulators, still as float-float (the same bits in every
// thread).  Warps merge by butterfly shuffles, then warp 0 merges the warp totals; no fp64
// instruction is issued (a full-warp fp64 instruction is expensive on GB300).
template <int NV, int BS>
__device__ __forceinline__ void block_reduce_ff(ff (&v)[NV]) {
    __shared__ ff wsum[NV][BS / 32];
    __shared__ ff res[NV];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ff_shfl_merge(v[i], o);
        if (lane == 0) wsum[i][wid] = v[i];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            ff x = lane < BS / 32 ? wsum[i][lane] : ff_zero();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ff_shfl_merge(x, o);
            if (lane == 0) res[i] = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = res[i];
    __syncthreads();
}

// Grid-wide synchronisation state living in caller-provided global memory (all of it zeroed
// before each launch): an arrival counter, the error word (WCFD_OK or WCFD_BARRIER_TIMEOUT)
// and [2 phase parities][2 sums][kMaxGrid] 16-byte words, one per block and sum: the block's
// float-float total and the phase it belongs to.
struct GridCtl {
    unsigned* ctr;
    int* err;
    char* words;
};

// most blocks of a cooperative launch that meets at grid_reduce (one per SM)
constexpr int kMaxGrid = 160;
constexpr size_t kGridCtlBytes = 256 + 2 * 2 * (size_t)kMaxGrid * 16;

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// 16-byte words that are loaded and stored whole
__device__ __forceinline__ void ld_relaxed128(const void* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st_relaxed128(void* p, unsigned long long a, unsigned long long b) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%0, %1};\n\tst.relaxed.gpu.global.b128 [%2], t;\n\t}" ::"l"(a),
                 "l"(b), "l"(p)
                 : "memory");
}

// pairwise sum of N float-float values (a tree, so that the merges overlap), result in v[0]
template <int N>
__device__ __forceinline__ void ff_tree(ff (&v)[N]) {
#pragma unroll
    for (int d = 1; d < N; d *= 2)
#pragma unroll
        for (int k = 0; k + d < N; k += 2 * d) ff_merge(v[k], v[k + d]);
}

// Barrier + reduction over all blocks of a cooperative launch, for phase number `phase`
// (1, 2, 3, ... in every block).  acc[] holds each thread's float-float sums; fin(sums) is
// called by all lanes of warp 0 with the sums over the whole grid (normalised; the same bits
// in every block on every run) and may write what the block needs to shared memory: a block
// barrier follows.  sbuf: shared memory of NV * BS/2 ff.
//
// The block stage: one butterfly level in every warp, then BS/2 values in shared memory, of
// which warp i merges sum i (BS/64 per lane as a tree, then a butterfly) and stores it as one
// 16-byte word that carries its phase.  Beside it, from the same block barrier on, warp NV
// publishes everything the block wrote so far: a release reduction on the arrival counter,
// whose fence (about 750 cycles) so overlaps the merging (about 580).  Warp 0 waits for the
// counter (acquire), then reads every block's word and merges them in one fixed order.  A
// word that is still on its way shows an older phase and is read again; words are
// double-buffered by phase parity (a block stores phase k+2 only after every block has
// arrived at k+1, and so has read k).
// Measured (152 blocks, two sums, block stage included): 2.07 us a barrier; 3.05 us for
// butterflies in every warp, partial sums ordered by the counter's own release and separate
// broadcasts.  Also tried: totals polled directly instead of a counter, in 1 / 4 / 8 / 16
// copies (6.4 / 3.9 / 3.8 / 3.5 us: 152 blocks polling 152 words), the words loaded along
// with every poll (2.3-2.7 us), a relaxed poll with a fence after it (2.5 us).
// Every wait is bounded: on timeout the block sets *err and returns false.  NV <= 2.
template <int NV, int BS, typename Fin>
__device__ __forceinline__ bool grid_reduce(const GridCtl& g, ff (&acc)[NV], ff* sbuf, unsigned phase, Fin&& fin) {
    static_assert(NV >= 1 && NV <= 2 && BS % 64 == 0, "one or two sums");
    constexpr int H = BS / 2;                 // values of one sum left in shared memory
    constexpr int PER = H / 32;               // per lane of the merging warp
    constexpr int POLL = (kMaxGrid + 31) / 32;
    __shared__ int s_fail;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_fail = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        ff_shfl_merge(acc[i], 16);
        if (lane < 16) sbuf[i * H + wid * 16 + lane] = acc[i];
    }
    __syncthreads();  // every thread's writes of the phase happen before the release below
    if (wid == NV && lane == 0) red_release_add(g.ctr, 1u);
    if (wid < NV) {
        char* words = g.words + (size_t)(phase & 1u) * (2 * kMaxGrid * 16);
        ff v[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) v[k] = sbuf[wid * H + k * 32 + lane];
        ff_tree(v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ff_shfl_merge(v[0], o);
        if (lane == 0)
            st_relaxed128(words + (size_t)(wid * kMaxGrid + blockIdx.x) * 16,
                          ((unsigned long long)__float_as_uint(v[0].lo) << 32) | __float_as_uint(v[0].hi), phase);
        if (wid == 0) {
            const int G = (int)gridDim.x;
            const unsigned target = phase * gridDim.x;
            unsigned long long w[NV][POLL];
            bool ok = true;
            unsigned spins = 0;
            uint64_t t0 = 0;
            for (;;) {
                // the warp decides as one, by lane 0's load: its lanes' loads may be served at different times.
                // (Every lane acting on its own load up to the vote below: 3 to 4% of an iteration slower.)
                if ((int)(__shfl_sync(0xffffffffu, ld_acquire(g.ctr), 0) - target) >= 0) {
                    unsigned long long tag[NV][POLL];
                    bool all = true;
#pragma unroll
                    for (int i = 0; i < NV; ++i)
#pragma unroll
                        for (int k = 0; k < POLL; ++k) {
                            const int b = k * 32 + lane;
                            w[i][k] = 0;
                            tag[i][k] = phase;
                            if (b < G) ld_relaxed128(words + (size_t)(i * kMaxGrid + b) * 16, w[i][k], tag[i][k]);
                        }
#pragma unroll
                    for (int i = 0; i < NV; ++i)
#pragma unroll
                        for (int k = 0; k < POLL; ++k) all = all && (unsigned)tag[i][k] == phase;
                    if (__all_sync(0xffffffffu, all)) break;
                }
                if ((++spins & 31u) == 0u) {
                    const uint64_t t = global_ns();
                    if (t0 == 0) t0 = t;
                    if (__any_sync(0xffffffffu, t - t0 > kBarrierTimeoutNs)) {
                        ok = false;
                        break;
                    }
                }
            }
            if (!ok) {
                if (lane == 0) {
                    s_fail = 1;
                    atomicExch(g.err, WCFD_BARRIER_TIMEOUT);
                }
            } else {
                ff sums[NV];
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    ff x[POLL];
#pragma unroll
                    for (int k = 0; k < POLL; ++k)
                        x[k] = ff{__uint_as_float((unsigned)w[i][k]), __uint_as_float((unsigned)(w[i][k] >> 32))};
                    ff_tree(x);
                    sums[i] = x[0];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < NV; ++i) ff_shfl_merge(sums[i], o);
#pragma unroll
                for (int i = 0; i < NV; ++i) sums[i] = ff_norm(sums[i]);
                fin(sums);
            }
        }
    }
    __syncthreads();
    return !s_fail;
}

// NVTX range over a host scope (a stage of a step), for Nsight Systems timelines: one
// cheap call each way when no tool is attached (NVTX v3, header-only)
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

}  // namespace wcfd
