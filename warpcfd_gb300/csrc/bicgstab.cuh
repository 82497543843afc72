// BiCGSTAB for the momentum system (3 components a row, shared off-diagonals), one body for the
// grid, cluster and batched kernels.
//
//   phase 1   p = r + beta u            u = p_old - omega v_old, formed with r by phase 3
//             v = A (M p) ; r0.v
//   phase 2   s = r - alpha v ; t = A (M s) ; t.t ; t.s
//   phase 3   x += alpha M p + omega M s ; r = s - omega t ; u = p - omega v ; r.r ; r0.r
//
// M = 1/diag per component.  M p and M s of a neighbour are formed from what it published: the
// records R = (r, 1/d_0), U = (u, 1/d_1), V = (v, 1/d_1) of 16 bytes and 1/d_2, so that a
// phase gathers two 16-byte words and one 4-byte word per neighbour (the twelve and nine
// scalars of r, p, v and 1/d before).  s and M p are formed again where they are used instead of
// stored.  Rows are contiguous per CTA.  A resident kernel keeps a row's own data (24 floats,
// its off-diagonals and where its neighbours' records lie) in shared memory for the length of
// the solve, so that a phase touches only records; otherwise the matrix streams and r0, p and
// t are planes of the workspace.
//
// The operations per value are the same in every form.  Bound by the three reductions of an
// iteration while resident (6 us of them on the grid, about 2 in a cluster), by the bytes of the
// matrix and about 22 floats a row beyond (128^3: 350 bytes a row and iteration, 5.0 TB/s).
// Measured per iteration against the form with scalar vectors in the workspace and 1,024 threads
// of one row: 1,024 rows 14.3 -> 3.7 us, 4,096 14.8 -> 4.0 (cluster); 32,000 15.4 -> 7.3, 55,000
// tetrahedra 18.7 -> 8.3, 152,000 19.6 -> 11.8, 247,000 of width 4 25.4 -> 14.7 (grid, resident);
// 255,000 of width 6 27.9 -> 19.8, 864,000 76 -> 54, 128^3 174 -> 148 (streamed; without the prefetch 157,
// with r0, the diagonal and the records prefetched too 151 to 158).
#pragma once
#include "cluster.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace wcfd {

struct BiSystem {
    const float *diag, *off, *rhs;
    const int* col;
    const int16_t* dcol;  // column - row, or null
    float* x;
    int C, maxiter;
    bool in_place;
    double atol2, rtol2;
    wcfd_solve_stats* stats;
};
struct BiScalars {
    ff rr, rho, alpha, omega, thr2;
    float af, bf, of;
    int go, status, k;
};

// floats of a row's own data in a resident kernel: d, 1/d, r0, x, p, t, r, v, off-diagonals, handles
// (and the neighbours' 1/d_2 where that is not gathered)
constexpr int kBiPlanes = 24;

// sums of a cluster to thread 0, fin(sums) there; a wait that gave up ends the solve
template <int NV, int T, bool FENCE, class Fin>
__device__ __forceinline__ bool cluster_scalars(ff (&acc)[NV], ClusterMeet& meet, BiScalars& sc, Fin&& fin) {
    const bool met = cluster_reduce<NV, T, false, FENCE>(acc, meet);
    if (threadIdx.x == 0) {
        if (met) {
            fin(acc);
        } else {
            sc.status = WCFD_BARRIER_TIMEOUT;
            sc.go = 0;
        }
    }
    __syncthreads();
    return true;
}

// records in the workspace: 13 floats a row (R, U, V, 1/d_2), then the planes r0, p, t; 22 of 27
// floats.  CLUSTER: the CTAs of a cluster meet, else those of the grid; other CTAs' records are
// read through L2 in a cluster, whose barrier does not order the first-level caches of two SMs.
template <int T, bool CLUSTER>
struct BiGlobal {
    using Handle = int;
    static constexpr bool kOwnZ = false;
    float4 *R, *U, *V;
    float *Z, *planes;
    int row0;
    GridCtl g;          // the grid's
    ff* sbuf;
    unsigned phase;
    ClusterMeet meet;   // the cluster's
    __device__ __forceinline__ BiGlobal(float* ws, int C, int first) : row0(first), phase(0) {
        R = reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(ws) + 15) & ~(uintptr_t)15);
        U = R + C;
        V = U + C;
        Z = reinterpret_cast<float*>(V + C);
        planes = Z + C;
    }
    __device__ __forceinline__ Handle make(int c) const { return c; }
    __device__ __forceinline__ static float4 ld(const float4* p) {
        if constexpr (CLUSTER) return __ldcg(p);
        else return *p;
    }
    __device__ __forceinline__ float4 r(Handle h) const { return ld(R + h); }
    __device__ __forceinline__ float4 u(Handle h) const { return ld(U + h); }
    __device__ __forceinline__ float4 v(Handle h) const { return ld(V + h); }
    __device__ __forceinline__ float z(Handle h) const {
        if constexpr (CLUSTER) return __ldcg(Z + h);
        else return Z[h];
    }
    __device__ __forceinline__ void put_r(int l, float4 w) { R[row0 + l] = w; }
    __device__ __forceinline__ void put_u(int l, float4 w) { U[row0 + l] = w; }
    __device__ __forceinline__ void put_v(int l, float4 w) { V[row0 + l] = w; }
    __device__ __forceinline__ void put_z(int l, float w) { Z[row0 + l] = w; }
    __device__ __forceinline__ void begin() const {
        if constexpr (CLUSTER) cluster_begin(meet);
    }
    // fin(sums) in thread 0, its writes visible to the block; false when a wait gave up
    template <int NV, class Fin>
    __device__ __forceinline__ bool reduce(ff (&acc)[NV], BiScalars& sc, Fin&& fin) {
        if constexpr (CLUSTER) {
            return cluster_scalars<NV, T, true>(acc, meet, sc, fin);
        } else {
            return grid_reduce<NV, T>(g, acc, sbuf, ++phase, [&](const ff* s) {
                if (threadIdx.x == 0) fin(s);
            });
        }
    }
};

// records in the shared memory of the cluster's CTAs, gathered through DSMEM; a neighbour's
// 1/d_2, which does not change, is the row's own
template <int T>
struct BiShared {
    using Handle = uint32_t;
    static constexpr bool kOwnZ = true;
    float4* R;  // [3][cap]: R, U, V
    uint32_t us, vs;
    int rows;
    ClusterMeet meet;
    __device__ __forceinline__ BiShared(float4* records, int cap, int rows_per_cta) : R(records), rows(rows_per_cta) {
        us = 16u * cap;
        vs = 32u * cap;
    }
    __device__ __forceinline__ Handle make(int c) const {
        const int rk = c / rows;
        return map_rank(R + (c - rk * rows), rk);
    }
    __device__ __forceinline__ float4 r(Handle h) const { return ld_cluster_f32x4(h); }
    __device__ __forceinline__ float4 u(Handle h) const { return ld_cluster_f32x4(h + us); }
    __device__ __forceinline__ float4 v(Handle h) const { return ld_cluster_f32x4(h + vs); }
    __device__ __forceinline__ void put_r(int l, float4 w) { R[l] = w; }
    __device__ __forceinline__ void put_u(int l, float4 w) { R[us / 16 + l] = w; }
    __device__ __forceinline__ void put_v(int l, float4 w) { R[vs / 16 + l] = w; }
    __device__ __forceinline__ void put_z(int, float) {}
    __device__ __forceinline__ void begin() const { cluster_begin(meet); }
    template <int NV, class Fin>
    __device__ __forceinline__ bool reduce(ff (&acc)[NV], BiScalars& sc, Fin&& fin) {
        return cluster_scalars<NV, T, false>(acc, meet, sc, fin);
    }
};

// Rows [row0, row0 + nloc) of this CTA.  own: RES, [kBiPlanes + 2 W (+ W)][cap] in shared memory;
// else unused (the planes of net).  False when a wait gave up.
template <int W, int T, bool RES, class Net>
__device__ __forceinline__ bool bicgstab_body(const BiSystem& a, Net& net, BiScalars& sc, float* own, int cap, int row0, int nloc,
                                              bool first) {
    using H = typename Net::Handle;
    constexpr int WA = W > 0 ? W : 1;
    const int C = a.C, t = threadIdx.x;
    // plane k (0 d, 1 1/d, 2 r0, 3 x, 4 p, 5 t, 6 r, 7 v) of component o
    auto at = [&](int k, int o, int l) -> float& { return own[(3 * k + o) * cap + l]; };
    auto load_matrix = [&](int l, float (&ov)[WA], H (&h)[WA]) {
        if constexpr (RES) {
#pragma unroll
            for (int j = 0; j < W; ++j) {
                ov[j] = own[(kBiPlanes + j) * cap + l];
                h[j] = (H)__float_as_uint(own[(kBiPlanes + W + j) * cap + l]);
            }
        } else {
            ell_columns<W>(h, a.col, a.dcol, C, row0 + l);
#pragma unroll
            for (int j = 0; j < W; ++j) ov[j] = __ldcs(a.off + (size_t)j * C + row0 + l);
        }
    };
    // L2 prefetch of the matrix lines of the warp's next rows (lane j < W: a plane of columns, then of
    // coefficients); nothing waits on it
    auto prefetch_matrix = [&](int l) {
        if constexpr (!RES && W > 0) {
            const int lane = t & 31, rb = l - lane + T;
            if (lane < 2 * W && rb < nloc) {
                const size_t i = (size_t)(lane < W ? lane : lane - W) * C + row0 + rb;
                const void* p = lane < W ? (const void*)(a.off + i) : a.dcol ? (const void*)(a.dcol + i) : (const void*)(a.col + i);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
            }
        }
    };
    auto nbr_z = [&](int l, const H (&h)[WA], float (&z)[WA]) {
#pragma unroll
        for (int j = 0; j < W; ++j) {
            if constexpr (Net::kOwnZ) z[j] = own[(kBiPlanes + 2 * W + j) * cap + l];
            else z[j] = net.z(h[j]);
        }
    };
    if (t == 0) {
        sc.k = 0;
        sc.status = WCFD_OK;
    }
    // r = b - A x ; r0 = r ; the first direction is r itself (beta = 0) ; rr ; rho = r0.r = rr ; bb
    ff acc[2] = {ff_zero(), ff_zero()};
    for (int l = t; l < nloc; l += T) {
        const size_t g = (size_t)row0 + l;
        float ov[WA], xc[3][WA], d[3], xi[3], bi[3], ri[3], di[3];
#pragma unroll
        for (int j = 0; j < W; ++j) {
            ov[j] = a.off[(size_t)j * C + g];
            const int c = a.col[(size_t)j * C + g];
#pragma unroll
            for (int o = 0; o < 3; ++o) xc[o][j] = a.x[3 * (size_t)c + o];
            if constexpr (RES) {
                own[(kBiPlanes + j) * cap + l] = ov[j];
                own[(kBiPlanes + W + j) * cap + l] = __uint_as_float((unsigned)net.make(c));
                if constexpr (Net::kOwnZ) {
                    const float dz = a.diag[3 * (size_t)c + 2];
                    own[(kBiPlanes + 2 * W + j) * cap + l] = dz != 0.0f ? 1.0f / dz : 1.0f;
                }
            }
        }
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            d[o] = a.diag[3 * g + o];
            xi[o] = a.x[3 * g + o];
            bi[o] = a.rhs[3 * g + o];
        }
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            di[o] = d[o] != 0.0f ? 1.0f / d[o] : 1.0f;
            ri[o] = bi[o] - row_product<W>(d[o], xi[o], ov, xc[o], a.in_place);
            ff_fma(acc[0], ri[o], ri[o]);
            ff_fma(acc[1], bi[o], bi[o]);
            if constexpr (RES) {
                at(0, o, l) = d[o];
                at(1, o, l) = di[o];
                at(2, o, l) = at(4, o, l) = at(6, o, l) = ri[o];
                at(3, o, l) = xi[o];
                at(7, o, l) = 0.0f;
            } else {
                net.planes[(size_t)o * C + g] = ri[o];
            }
        }
        net.put_r(l, make_float4(ri[0], ri[1], ri[2], di[0]));
        net.put_u(l, make_float4(ri[0], ri[1], ri[2], di[1]));
        net.put_z(l, di[2]);
    }
    net.begin();
    if (!net.template reduce<2>(acc, sc, [&](const ff* v) {
            const double rr0 = ff_to_double(v[0]);
            sc.rr = sc.rho = v[0];
            sc.thr2 = ff_norm(ff_from_double(fmax(a.atol2, a.rtol2 * rr0)));
            sc.bf = sc.of = 0.0f;
            sc.go = (0 < a.maxiter && ff_gt(sc.rr, sc.thr2));
            if (first) {
                a.stats->initial_residual = sqrt(rr0);
                a.stats->rhs_norm = sqrt(ff_to_double(v[1]));
            }
        }))
        return false;
    while (sc.go) {
        const float bf = sc.bf, of0 = sc.of;
        ff accv[1] = {ff_zero()};
        for (int l = t; l < nloc; l += T) {
            float ov[WA], nz[WA], gv[3][WA], ro[3], uo[3], d[3], di[3], r0[3], vi[3], po[3];
            float4 nr[WA], nu[WA];
            H h[WA];
            prefetch_matrix(l);
            load_matrix(l, ov, h);
#pragma unroll
            for (int j = 0; j < W; ++j) nr[j] = net.r(h[j]);
#pragma unroll
            for (int j = 0; j < W; ++j) nu[j] = net.u(h[j]);
            nbr_z(l, h, nz);
            if constexpr (RES) {
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    ro[o] = at(6, o, l);
                    uo[o] = fmaf(-of0, at(7, o, l), at(4, o, l));
                    d[o] = at(0, o, l);
                    di[o] = at(1, o, l);
                    r0[o] = at(2, o, l);
                }
            } else {
                const size_t g = (size_t)row0 + l;
                const float4 r4 = net.R[g], u4 = net.U[g];
                ro[0] = r4.x; ro[1] = r4.y; ro[2] = r4.z;
                uo[0] = u4.x; uo[1] = u4.y; uo[2] = u4.z;
                di[0] = r4.w; di[1] = u4.w; di[2] = net.Z[g];
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    d[o] = a.diag[3 * g + o];
                    r0[o] = net.planes[(size_t)o * C + g];
                }
            }
#pragma unroll
            for (int j = 0; j < W; ++j) {
                gv[0][j] = fmaf(bf, nu[j].x, nr[j].x) * nr[j].w;
                gv[1][j] = fmaf(bf, nu[j].y, nr[j].y) * nu[j].w;
                gv[2][j] = fmaf(bf, nu[j].z, nr[j].z) * nz[j];
            }
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                po[o] = fmaf(bf, uo[o], ro[o]);
                vi[o] = row_product<W>(d[o], po[o] * di[o], ov, gv[o], a.in_place);
                ff_fma(accv[0], r0[o], vi[o]);
                if constexpr (RES) {
                    at(4, o, l) = po[o];
                    at(7, o, l) = vi[o];
                } else {
                    net.planes[(size_t)(3 + o) * C + row0 + l] = po[o];
                }
            }
            net.put_v(l, make_float4(vi[0], vi[1], vi[2], di[1]));
        }
        if (!net.template reduce<1>(accv, sc, [&](const ff* r0v) {
                if (r0v[0].hi == 0.0f) {
                    sc.status = WCFD_KRYLOV_BREAKDOWN;
                    sc.go = 0;
                } else {
                    sc.alpha = ff_div(sc.rho, r0v[0]);
                    sc.af = ff_to_float(sc.alpha);
                }
            }))
            return false;
        if (!sc.go) break;
        const float af = sc.af;
        ff acct[2] = {ff_zero(), ff_zero()};
        for (int l = t; l < nloc; l += T) {
            float ov[WA], nz[WA], gv[3][WA], so[3], d[3], di[3], ti[3];
            float4 nr[WA], nv[WA];
            H h[WA];
            prefetch_matrix(l);
            load_matrix(l, ov, h);
#pragma unroll
            for (int j = 0; j < W; ++j) nr[j] = net.r(h[j]);
#pragma unroll
            for (int j = 0; j < W; ++j) nv[j] = net.v(h[j]);
            nbr_z(l, h, nz);
            if constexpr (RES) {
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    so[o] = fmaf(-af, at(7, o, l), at(6, o, l));
                    d[o] = at(0, o, l);
                    di[o] = at(1, o, l);
                }
            } else {
                const size_t g = (size_t)row0 + l;
                const float4 r4 = net.R[g], v4 = net.V[g];
                so[0] = fmaf(-af, v4.x, r4.x);
                so[1] = fmaf(-af, v4.y, r4.y);
                so[2] = fmaf(-af, v4.z, r4.z);
                di[0] = r4.w; di[1] = v4.w; di[2] = net.Z[g];
#pragma unroll
                for (int o = 0; o < 3; ++o) d[o] = a.diag[3 * g + o];
            }
#pragma unroll
            for (int j = 0; j < W; ++j) {
                gv[0][j] = fmaf(-af, nv[j].x, nr[j].x) * nr[j].w;
                gv[1][j] = fmaf(-af, nv[j].y, nr[j].y) * nv[j].w;
                gv[2][j] = fmaf(-af, nv[j].z, nr[j].z) * nz[j];
            }
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                ti[o] = row_product<W>(d[o], so[o] * di[o], ov, gv[o], a.in_place);
                ff_fma(acct[0], ti[o], ti[o]);
                ff_fma(acct[1], ti[o], so[o]);
                if constexpr (RES) at(5, o, l) = ti[o];
                else net.planes[(size_t)(6 + o) * C + row0 + l] = ti[o];
            }
        }
        if (!net.template reduce<2>(acct, sc, [&](const ff* ts) {
                sc.omega = ts[0].hi != 0.0f ? ff_div(ts[1], ts[0]) : ff_zero();
                sc.of = ff_to_float(sc.omega);
            }))
            return false;
        if (!sc.go) break;  // only a wait that gave up
        const float of = sc.of;
        ff accr[2] = {ff_zero(), ff_zero()};
        for (int l = t; l < nloc; l += T) {
            const size_t g = (size_t)row0 + l;
            float ro[3], vo[3], po[3], to[3], di[3], r0[3], xo[3], uo[3];
            if constexpr (RES) {
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    ro[o] = at(6, o, l);
                    vo[o] = at(7, o, l);
                    po[o] = at(4, o, l);
                    to[o] = at(5, o, l);
                    di[o] = at(1, o, l);
                    r0[o] = at(2, o, l);
                    xo[o] = at(3, o, l);
                }
            } else {
                const float4 r4 = net.R[g], v4 = net.V[g];
                ro[0] = r4.x; ro[1] = r4.y; ro[2] = r4.z;
                vo[0] = v4.x; vo[1] = v4.y; vo[2] = v4.z;
                di[0] = r4.w; di[1] = v4.w; di[2] = net.Z[g];
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    r0[o] = net.planes[(size_t)o * C + g];
                    po[o] = net.planes[(size_t)(3 + o) * C + g];
                    to[o] = net.planes[(size_t)(6 + o) * C + g];
                    xo[o] = a.x[3 * g + o];
                }
            }
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                const float si = fmaf(-af, vo[o], ro[o]);
                const float xa = fmaf(af, po[o] * di[o], xo[o]);
                xo[o] = fmaf(of, si * di[o], xa);
                ro[o] = fmaf(-of, to[o], si);
                uo[o] = fmaf(-of, vo[o], po[o]);
                ff_fma(accr[0], ro[o], ro[o]);
                ff_fma(accr[1], r0[o], ro[o]);
                if constexpr (RES) {
                    at(3, o, l) = xo[o];
                    at(6, o, l) = ro[o];
                } else {
                    a.x[3 * g + o] = xo[o];
                }
            }
            net.put_r(l, make_float4(ro[0], ro[1], ro[2], di[0]));
            net.put_u(l, make_float4(uo[0], uo[1], uo[2], di[1]));
        }
        if (!net.template reduce<2>(accr, sc, [&](const ff* rr2) {
                sc.rr = rr2[0];
                sc.k += 1;
                if (sc.omega.hi == 0.0f || sc.rho.hi == 0.0f) {
                    sc.status = WCFD_KRYLOV_BREAKDOWN;
                    sc.go = 0;
                } else {
                    sc.bf = ff_to_float(ff_mul(ff_div(rr2[1], sc.rho), ff_div(sc.alpha, sc.omega)));
                    sc.rho = rr2[1];
                    sc.go = (sc.k < a.maxiter && ff_gt(sc.rr, sc.thr2));
                }
            }))
            return false;
    }
    if constexpr (RES) {
        for (int l = t; l < nloc; l += T)
#pragma unroll
            for (int o = 0; o < 3; ++o) a.x[3 * ((size_t)row0 + l) + o] = at(3, o, l);
    }
    if (first && t == 0) {
        int st = sc.status;
        if (st == WCFD_OK && !ff_le(sc.rr, sc.thr2)) st = WCFD_NOT_CONVERGED;
        a.stats->iterations = sc.k;
        a.stats->status = st;
        a.stats->residual = st == WCFD_BARRIER_TIMEOUT ? -1.0 : sqrt(ff_to_double(sc.rr));
    }
    return true;
}

}  // namespace wcfd
