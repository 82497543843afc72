// Cluster-resident CG: one thread-block cluster (up to 16 CTAs) holds the whole scalar
// system on chip for the length of the solve.
//
//  * CTA q of the cluster owns rows [q R, (q+1) R).  Up to 2,048 rows a CTA, eight warps keep
//    their rows' off-diagonals, neighbour addresses, x, r, q and p in registers, up to eight
//    rows a thread; beyond that sixteen warps of eight rows keep the matrix in shared memory
//    (laid out by thread) and the rest in registers.  What others gather, z and p of every row, is
//    in shared memory, as (z, p) pairs that one 8-byte load fetches.
//  * A neighbour value owned by another CTA is read through distributed shared memory
//    (mapa + ld.shared::cluster); nothing touches global memory between the set-up and
//    the final write of x.
//  * The CTAs meet in the reductions only (cluster.cuh): exact products in float-float
//    (common.cuh), merged in a fixed order, each CTA's total sent to every CTA by a store that
//    completes bytes on the receiver's mbarrier; so all CTAs (and all runs) agree bit for bit and
//    take the same branch at every test.
//  * The direction update p = z + beta p is evaluated inside the SpMV for the row and its
//    neighbours, so an iteration needs two reductions.
// Bound by latency: of its two reductions and, with many rows a CTA, of remote gathers and dependent
// arithmetic with two to four warps a scheduler (16 x 2,000 rows: an instruction in 40% of the cycles).
// Measured per iteration (1,024 threads, everything in shared memory, cluster barriers -> this
// form): 2 CTAs x 512 rows 2.68 -> 1.37 us, 8 x 512 2.87 -> 1.54, 16 x 2,000 3.77 -> 2.39, 16 x 4,096
// 4.68 -> 3.37 (the grid kernel: 4.59).
// The arithmetic is that of cg_kernel (krylov.cu): the same Jacobi-preconditioned CG with
// fp64-accurate dot products and the same stop test.
#include "bicgstab.cuh"
#include "cluster.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace wcfd {

// rows that the threads of a CTA for R rows can hold (2, 4 or 8 times 256 threads, 8 x 512),
// and its threads
int cluster_cg_capacity(int R) { return R <= 512 ? 512 : R <= 1024 ? 1024 : R <= 2048 ? 2048 : 4096; }
int cluster_cg_threads(int R) { return cluster_cg_capacity(R) > 2048 ? 512 : 256; }

// Dynamic shared memory per CTA for R rows and width W: the (z, p) pairs (8 bytes a row) and, with
// 512 threads, the off-diagonals, diag and 1/diag (4 W + 8).  16 CTAs of R <= 4096 rows hold
// 65536 rows.
size_t cluster_cg_smem_bytes(int R, int W) {
    const int cap = cluster_cg_capacity(R);
    return (size_t)cap * (8 + (cap > 2048 ? 4 * (size_t)W + 8 : 0));
}

// Largest R of a cluster solve: 4,096 up to width 4, 3,811 and 3,430 at 5 and 6, where the grid
// kernel takes over (and where the batched form's limit lies); at most what 8 x 512 threads hold.
int cluster_cg_max_rows(int W, int optin) {
    const long long r = ((long long)optin - 26624) / (6LL * W + 24);
    return r > 4096 ? 4096 : r > 0 ? (int)r : 0;
}

template <int W, int RPT, int T>
__device__ __forceinline__ void cg_cluster_body(const KrylovArgs& a, int R) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(16) ClusterShared<T, 3> meeting;
    constexpr int WA = W > 0 ? W : 1, NA = kClusterAcc<T>;
    constexpr int GR = T == 512 ? 2 : RPT < 4 ? RPT : 4;  // rows whose gathers are in flight together
    constexpr bool REG = T == 256;                        // the matrix in registers
    constexpr int RM = REG ? RPT : 1;
    const int C = a.m.n_cells;
    const unsigned me = cluster_rank();
    const int row0 = (int)me * R;
    const int nloc = max(0, min(R, C - row0));
    float2* zp = reinterpret_cast<float2*>(smem);         // [RPT T] (z, p), by row
    float* s_o = reinterpret_cast<float*>(zp + RPT * T);  // [RPT][T][W] (W = 4) or [RPT][W][T], by thread (!REG)
    float* s_d = s_o + W * RPT * T;                       // [RPT][T]
    float* s_i = s_d + RPT * T;                           // [RPT][T]
    const int t = threadIdx.x;
    const int groups = (nloc + GR * T - 1) / (GR * T);  // groups of GR rows a thread that hold any
    ClusterMeet meet = cluster_meet(meeting);
    const uint32_t zp0 = (uint32_t)__cvta_generic_to_shared(zp);

    // the matrix rows of this thread; at: where a neighbour's pair lies, here or in another CTA
    float o[RM][WA], dg[RM], iv[RM];
    uint32_t at[RPT][WA];
    unsigned local = 0;  // bit u: no row of this warp's u-th 32 has a neighbour in another CTA
    float xr[RPT], rr_[RPT], qr[RPT], pr[RPT];
    // r = b - A x (x read from global) ; z = M r ; the first direction is z (p_old = 0) ; rr ; rz ; bb
    ff arr[NA], arz[NA], abb[NA];
#pragma unroll
    for (int q = 0; q < NA; ++q) arr[q] = arz[q] = abb[q] = ff_zero();
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int l = cluster_row<T>(t, u);
        // a row past the end is a row of zeros that gathers its own pair (0, 0): the passes need
        // no test of the row, which would keep a thread's rows from overlapping
        xr[u] = rr_[u] = qr[u] = pr[u] = 0.0f;
        float d = 0.0f, di = 0.0f, zi = 0.0f, ov[WA];
#pragma unroll
        for (int j = 0; j < WA; ++j) ov[j] = 0.0f;
#pragma unroll
        for (int j = 0; j < W; ++j) at[u][j] = zp0 + 8u * l;
        bool mine = true;
        if (l < nloc) {
            const int g = row0 + l;
            d = a.A.diag[g];
            di = d != 0.0f ? 1.0f / d : 1.0f;
            float xc[WA];
#pragma unroll
            for (int j = 0; j < W; ++j) {
                ov[j] = a.A.off[(size_t)j * C + g];
                const int c = a.m.ell_col[(size_t)j * C + g];
                const int rk = c / R, lo = c - rk * R;
                xc[j] = a.x[c];
                mine = mine && rk == (int)me;
                at[u][j] = rk == (int)me ? zp0 + 8u * lo : map_rank(zp + lo, rk);
            }
            const float xi = a.x[g], bi = a.A.rhs[g];
            xr[u] = xi;
            const float ri = bi - row_product<W>(d, xi, ov, xc, false);
            zi = ri * di;
            rr_[u] = ri;
            ff_fma(arr[u % NA], ri, ri);
            ff_fma(arz[u % NA], ri, zi);
            ff_fma(abb[u % NA], bi, bi);
        }
        zp[l] = make_float2(zi, 0.0f);
        if constexpr (REG) {
            dg[u] = d;
            iv[u] = di;
#pragma unroll
            for (int j = 0; j < W; ++j) o[u][j] = ov[j];
        } else {
            s_d[u * T + t] = d;
            s_i[u * T + t] = di;
            if constexpr (W == 4) reinterpret_cast<float4*>(s_o)[u * T + t] = make_float4(ov[0], ov[1], ov[2], ov[3]);
            else
#pragma unroll
                for (int j = 0; j < W; ++j) s_o[(u * W + j) * T + t] = ov[j];
        }
        if (__all_sync(0xffffffffu, mine)) local |= 1u << u;
    }
    ff acc[3] = {cluster_merge<T>(arr), cluster_merge<T>(arz), cluster_merge<T>(abb)};
    cluster_begin(meet);
    cluster_reduce<3, T, true, false>(acc, meet);
    ff rr = acc[0], rz = acc[1];
    const ff thr2 = ff_norm(ff_from_double(fmax(a.atol2, a.rtol2 * ff_to_double(rr))));
    if (me == 0 && t == 0 && !cluster_gave_up(meet)) {
        a.stats->initial_residual = sqrt(ff_to_double(rr));
        a.stats->rhs_norm = sqrt(ff_to_double(acc[2]));
    }
    float bf = 0.0f;
    int k = 0, status = WCFD_OK;
    while (k < a.maxiter && ff_gt(rr, thr2)) {  // not with a NaN
        // p = z + beta p_old (own row and each neighbour) ; q = A p ; p.q.  The gathers of GR rows
        // are issued before the first is used.
        ff apq[NA];
#pragma unroll
        for (int q = 0; q < NA; ++q) apq[q] = ff_zero();
#pragma unroll
        for (int u0 = 0; u0 < RPT; u0 += GR) {
            if (u0 >= groups * GR) break;
            float2 v[GR][WA];
#pragma unroll
            for (int q = 0; q < GR; ++q) {
                const int u = u0 + q;
                if ((local >> u) & 1u) {  // warp-uniform: every neighbour in this CTA
#pragma unroll
                    for (int j = 0; j < W; ++j) v[q][j] = ld_shared_f32x2(at[u][j]);
                } else {
#pragma unroll
                    for (int j = 0; j < W; ++j) v[q][j] = ld_cluster_f32x2(at[u][j]);
                }
            }
#pragma unroll
            for (int q = 0; q < GR; ++q) {
                const int u = u0 + q;
                float ov[WA], d, di;
                if constexpr (REG) {
                    d = dg[u];
                    di = iv[u];
#pragma unroll
                    for (int j = 0; j < W; ++j) ov[j] = o[u][j];
                } else {
                    d = s_d[u * T + t];
                    di = s_i[u * T + t];
                    if constexpr (W == 4) {
                        const float4 c = reinterpret_cast<const float4*>(s_o)[u * T + t];
                        ov[0] = c.x; ov[1] = c.y; ov[2] = c.z; ov[3] = c.w;
                    } else {
#pragma unroll
                        for (int j = 0; j < W; ++j) ov[j] = s_o[(u * W + j) * T + t];
                    }
                }
                const float zi = __fmul_rn(rr_[u], di);  // as it was formed
                const float pi = fmaf(bf, pr[u], zi);
                float qi = __fmul_rn(d, pi);
#pragma unroll
                for (int j = 0; j < W; ++j) qi = fmaf(ov[j], fmaf(bf, v[q][j].y, v[q][j].x), qi);
                pr[u] = pi;
                qr[u] = qi;
                ff_fma(apq[u % NA], pi, qi);
            }
        }
        ff accq[1] = {cluster_merge<T>(apq)};
        cluster_reduce<1, T, true, false>(accq, meet);
        if (!(accq[0].hi < 0.0f || accq[0].hi > 0.0f)) {
            if (accq[0].hi == 0.0f) status = WCFD_KRYLOV_BREAKDOWN;
            if (accq[0].hi == 0.0f || cluster_gave_up(meet)) break;
        }
        const float af = ff_div_to_float(rz, accq[0]);
        // x += alpha p ; r -= alpha q ; z = M r ; rr ; rz
#pragma unroll
        for (int q = 0; q < NA; ++q) arr[q] = arz[q] = ff_zero();
#pragma unroll
        for (int u0 = 0; u0 < RPT; u0 += GR) {
            if (u0 >= groups * GR) break;
#pragma unroll
            for (int u = u0; u < u0 + GR; ++u) {
                float di;
                if constexpr (REG) di = iv[u];
                else di = s_i[u * T + t];
                xr[u] = fmaf(af, pr[u], xr[u]);
                const float ri = fmaf(-af, qr[u], rr_[u]);
                const float zi = __fmul_rn(ri, di);
                rr_[u] = ri;
                zp[cluster_row<T>(t, u)] = make_float2(zi, pr[u]);
                ff_fma(arr[u % NA], ri, ri);
                ff_fma(arz[u % NA], ri, zi);
            }
        }
        ff acc2[2] = {cluster_merge<T>(arr), cluster_merge<T>(arz)};
        cluster_reduce<2, T, true, false>(acc2, meet);
        rr = acc2[0];
        bf = rz.hi != 0.0f ? ff_div_to_float(acc2[1], rz) : 0.0f;
        rz = acc2[1];
        ++k;
    }
    bool met = !cluster_gave_up(meet);
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int l = cluster_row<T>(t, u);
        if (met && l < nloc) a.x[row0 + l] = xr[u];
    }
    met = cluster_end(meet, met);
    if (me == 0 && t == 0) {
        if (!met) status = WCFD_BARRIER_TIMEOUT;
        if (status == WCFD_OK && !ff_le(rr, thr2)) status = WCFD_NOT_CONVERGED;
        a.stats->iterations = k;
        a.stats->status = status;
        a.stats->residual = met ? sqrt(ff_to_double(rr)) : -1.0;
    }
}

template <int W, int RPT, int T>
__global__ void __launch_bounds__(T, 1) cg_cluster_kernel(KrylovArgs a, int R) {
    cg_cluster_body<W, RPT, T>(a, R);
}

// One cluster per case of a device case table: the pressure CG of every case
// (pres system, p_x warm start, stats[1]), cs CTAs per cluster.  refine = 1 solves a
// refinement sweep's correction instead: right-hand side p_work[0, C) (the fp64 residual
// rounded once), solution p_work[C, 2C) from zero, relative stop p_refine_rtol.
template <int W, int RPT, int T>
__global__ void __launch_bounds__(T, 1) cg_cluster_batched(const wcfd_case* __restrict__ cases, int cs, int refine) {
    const wcfd_case& c = cases[blockIdx.x / cs];
    KrylovArgs a = {};
    a.m = c.mesh;
    a.A = c.pres;
    a.x = c.p_x;
    a.atol2 = c.prm.atol_p * c.prm.atol_p;
    a.rtol2 = c.prm.rtol_p * c.prm.rtol_p;
    if (refine) {
        a.A.rhs = c.p_work;
        a.x = c.p_work + c.mesh.n_cells;
        a.atol2 = 0.0;
        a.rtol2 = c.prm.p_refine_rtol * c.prm.p_refine_rtol;
    }
    a.maxiter = c.prm.maxiter;
    a.stats = c.stats + 1;
    cg_cluster_body<W, RPT, T>(a, (c.mesh.n_cells + cs - 1) / cs);
}

// BiCGSTAB (bicgstab.cuh) over the CTAs of one cluster.  SMEM: records in the CTAs' shared memory
// with the rows' own data, up to about 1,000 rows a CTA; else records in the case's workspace.
template <int W, bool SMEM>
__device__ __forceinline__ void bicgstab_cluster_body(const BiSystem& sys, float* ws, int R, int cap) {
    constexpr int T = kBiClusterBlock;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ BiScalars sc;
    __shared__ __align__(16) ClusterShared<T, 2> meeting;
    const unsigned me = cluster_rank();
    const int row0 = (int)me * R, nloc = max(0, min(R, sys.C - row0));
    float4* records = reinterpret_cast<float4*>(smem);
    auto run = [&](auto& net, float* own) {
        net.meet = cluster_meet(meeting);
        bicgstab_body<W, T, SMEM>(sys, net, sc, own, cap, row0, nloc, me == 0);
        if (!cluster_end(net.meet, sc.status != WCFD_BARRIER_TIMEOUT) && me == 0 && threadIdx.x == 0) {
            sys.stats->status = WCFD_BARRIER_TIMEOUT;
            sys.stats->residual = -1.0;
        }
    };
    if constexpr (SMEM) {
        BiShared<T> net(records, cap, R);
        run(net, reinterpret_cast<float*>(records + 3 * (size_t)cap));
    } else {
        BiGlobal<T, true> net(ws, sys.C, row0);
        run(net, nullptr);
    }
}

template <int W>
__global__ void __launch_bounds__(kBiClusterBlock, 1) bicgstab_cluster_kernel(KrylovArgs a, int R) {
    const BiSystem sys{a.A.diag, a.A.off, a.A.rhs, a.m.ell_col, nullptr, a.x, a.m.n_cells, a.maxiter, slot_bits(a.m) != 0u, a.atol2, a.rtol2,
                       a.stats};
    bicgstab_cluster_body<W, true>(sys, nullptr, R, R);
}

// the momentum system of every case of a table, one cluster a case; cap: the most rows per CTA
template <int W, bool SMEM>
__global__ void __launch_bounds__(kBiClusterBlock, 1) bicgstab_cluster_batched(const wcfd_case* __restrict__ cases, int cs_req,
                                                                              int cap) {
    const wcfd_case& c = cases[blockIdx.x / cs_req];
    const BiSystem sys{c.mom.diag, c.mom.off, c.mom.rhs, c.mesh.ell_col, c.mesh.ell_dcol, c.hbya, c.mesh.n_cells, c.prm.maxiter, false,
                       c.prm.atol_u * c.prm.atol_u, c.prm.rtol_u * c.prm.rtol_u, c.stats + 0};
    bicgstab_cluster_body<W, SMEM>(sys, c.ws_u.vec, (c.mesh.n_cells + cs_req - 1) / cs_req, cap);
}

// Self-check of the cluster's meetings: `reductions` sums of two values against their closed form
// in every thread that gets them: in every thread (FORM 1, as the CG), in thread 0 (0, the BiCGSTAB; 2,
// the batched CG, which also meets at a barrier and gathers a word of another CTA before each reduction).
// Before reduction `at` CTA `who` sleeps delay_ns (0: nobody is late) or, with delay_ns < 0, leaves, so that
// the others' waits run out: a failure made without a fault.  status[CTA]: 0, WCFD_BARRIER_TIMEOUT when a
// CTA gave up, -1 for wrong values, -2 when this CTA's threads disagree.  Waits give up after limit_ns.
template <int T, int FORM>
__global__ void __launch_bounds__(T, 1) cluster_check_kernel(int reductions, int who, int at, long long delay_ns, long long limit_ns,
                                                            int* __restrict__ status) {
    constexpr bool ALL = FORM == 1;
    __shared__ __align__(16) ClusterShared<T, 3> meeting;
    __shared__ int s_met;
    __shared__ float s_word;
    const int t = threadIdx.x;
    ClusterMeet meet = cluster_meet(meeting, (uint64_t)limit_ns);
    const bool odd = (int)meet.me == who;
    const double n = (double)(T * meet.cs);
    bool met = true, right = true, stay = true;
    cluster_begin(meet);
    for (int i = 0; i < reductions && met; ++i) {
        if constexpr (FORM == 2) {
            if (t == 0) s_word = (float)i;
            stay = cluster_sync_met(meet);
            if (!stay) break;
            right = right && ld_cluster_f32(map_rank(&s_word, (meet.me + 1) % meet.cs)) == (float)i;
        }
        if (odd && i == at) {
            if (delay_ns < 0) break;
            const uint64_t t0 = global_ns();
            for (int s = 0; s < 10000000 && global_ns() - t0 < (uint64_t)delay_ns; ++s) __nanosleep(100);
            __syncthreads();
        }
        ff v[2] = {ff{(float)(meet.me * T + t + 1), 0.0f}, ff{(float)i, 0.0f}};
        met = cluster_reduce<2, T, ALL, false>(v, meet);
        if constexpr (ALL) met = v[0].hi == v[0].hi && v[1].hi == v[1].hi;
        right = right && (!ALL || met != cluster_gave_up(meet));
        if ((ALL || t == 0) && met) right = right && ff_to_double(v[0]) == 0.5 * n * (n + 1.0) && ff_to_double(v[1]) == n * i;
        if constexpr (!ALL) {
            if (t == 0) s_met = met;
            __syncthreads();
            met = s_met != 0;
            __syncthreads();
        }
    }
    const int went_on = __syncthreads_count(met && stay), all_right = __syncthreads_and(right);
    const bool all_met = stay && cluster_end(meet, met);
    if (t == 0)
        status[meet.me] = went_on != 0 && went_on != T ? -2 : !all_right ? -1 : all_met ? WCFD_OK : WCFD_BARRIER_TIMEOUT;
}
const void* cluster_check_kernel_for(int T, int form) {
    switch (form + (T == 512 ? 3 : 0)) {
        case 0: return (const void*)cluster_check_kernel<256, 0>;
        case 1: return (const void*)cluster_check_kernel<256, 1>;
        case 2: return (const void*)cluster_check_kernel<256, 2>;
        case 3: return (const void*)cluster_check_kernel<512, 0>;
        case 4: return (const void*)cluster_check_kernel<512, 1>;
        default: return (const void*)cluster_check_kernel<512, 2>;
    }
}

// dynamic shared memory of a CTA of R rows with everything in it, and the most rows that fit
size_t cluster_bicg_smem_bytes(int R, int W) { return (size_t)R * (48 + 4 * (size_t)(kBiPlanes + 3 * W)); }
int cluster_bicg_max_rows(int W, int optin) { return (int)(((size_t)optin - 10240) / cluster_bicg_smem_bytes(1, W)); }

// the kernel for R rows a CTA
template <int W>
const void* pick_kernel(int R, bool batched) {
    switch (cluster_cg_capacity(R)) {
        case 512: return batched ? (const void*)cg_cluster_batched<W, 2, 256> : (const void*)cg_cluster_kernel<W, 2, 256>;
        case 1024: return batched ? (const void*)cg_cluster_batched<W, 4, 256> : (const void*)cg_cluster_kernel<W, 4, 256>;
        case 2048: return batched ? (const void*)cg_cluster_batched<W, 8, 256> : (const void*)cg_cluster_kernel<W, 8, 256>;
        default: return batched ? (const void*)cg_cluster_batched<W, 8, 512> : (const void*)cg_cluster_kernel<W, 8, 512>;
    }
}

static const void* cg_cluster_pick(int W, int R, bool batched) {
    if (R > 4096) return nullptr;  // 8 rows x 512 threads
    switch (W) {
        case 0: return pick_kernel<0>(R, batched);
        case 1: return pick_kernel<1>(R, batched);
        case 2: return pick_kernel<2>(R, batched);
        case 3: return pick_kernel<3>(R, batched);
        case 4: return pick_kernel<4>(R, batched);
        case 5: return pick_kernel<5>(R, batched);
        case 6: return pick_kernel<6>(R, batched);
        default: return nullptr;
    }
}
const void* cg_cluster_kernel_for(int W, int R) { return cg_cluster_pick(W, R, false); }
const void* cg_cluster_batched_for(int W, int R) { return cg_cluster_pick(W, R, true); }
const void* bicgstab_cluster_kernel_for(int W) {
    switch (W) {
        case 0: return (const void*)bicgstab_cluster_kernel<0>;
        case 1: return (const void*)bicgstab_cluster_kernel<1>;
        case 2: return (const void*)bicgstab_cluster_kernel<2>;
        case 3: return (const void*)bicgstab_cluster_kernel<3>;
        case 4: return (const void*)bicgstab_cluster_kernel<4>;
        case 5: return (const void*)bicgstab_cluster_kernel<5>;
        case 6: return (const void*)bicgstab_cluster_kernel<6>;
        default: return nullptr;
    }
}
const void* bicgstab_cluster_batched_for(int W, bool resident) {
#define WCFD_BI(w) \
    case w: return resident ? (const void*)bicgstab_cluster_batched<w, true> : (const void*)bicgstab_cluster_batched<w, false>;
    switch (W) {
        WCFD_BI(0) WCFD_BI(1) WCFD_BI(2) WCFD_BI(3) WCFD_BI(4) WCFD_BI(5) WCFD_BI(6)
        default: return nullptr;
    }
#undef WCFD_BI
}

}  // namespace wcfd
