// Persistent Krylov solvers: one cooperative launch per solve, contiguous rows per
// co-resident block, fp64-accurate dot products (exact products summed
// in float-float across threads, warps and blocks; common.cuh) reduced deterministically
// at bounded grid barriers.  They replace warp.optim.linear.cg /
// bicgstab with the diagonal (Jacobi) preconditioner as called by Equation.solve_Axb
// (warp_cfd/FV/terms/equation.py:195-200).  Stop test: ||r||_2 <= atol before an
// iteration, or maxiter iterations.
//
// Each search-direction update (CG: p = z + beta p, p double-buffered; BiCGSTAB, bicgstab.cuh:
// p = r + beta (p - omega v), s = r - alpha v) is evaluated on the fly inside the SpMV that
// consumes it, for the row itself and for every gathered neighbour.  The arithmetic is the textbook algorithm's, but a CG iteration
// needs two grid barriers instead of three and a BiCGSTAB iteration three instead of five.
//
// The scalar recurrences (alpha, beta, omega, the stop test) run on the float-float sums
// in thread 0 of each block, inside the reduction (grid_reduce), and reach the other threads
// through shared memory behind its last block barrier: GB300
// runs fp64 at about 1/64 of its fp32 rate (a dependent fp64 division costs about 600
// cycles), and every thread of the grid waits for these few operations.
#include "bicgstab.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace wcfd {

constexpr int BS = kSolverBlock;  // threads of the barrier check
constexpr int CGB = kCgBlock;     // threads of the CG and the BiCGSTAB

__device__ __forceinline__ float jacobi(float d) { return d != 0.0f ? 1.0f / d : 1.0f; }

// Krylov scalars of one block, owned by thread 0
struct KScalars {
    ff rr, rz, thr2;
    float af, bf;
    int go, status, k;
};

// On a failed barrier (timeout, or another block's error) every block leaves; block 0
// records the error word so the caller sees why the solve stopped.
__device__ void fail_stats(const KrylovArgs& a, int k) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.stats->iterations = k;
        a.stats->status = *((volatile int*)a.g.err);
        a.stats->residual = -1.0;
    }
}

// sum the float-float accumulators `acc` over the grid; fin(sums) runs in warp 0
// (grid_reduce, common.cuh), thread 0 of which owns the scalars that follow from them
#define REDUCE(NV, acc, ...)                                                  \
    do {                                                                      \
        if (!grid_reduce<NV, sizeof(sbuf) / sizeof(ff)>(a.g, acc, sbuf, ++phase, __VA_ARGS__)) { \
            fail_stats(a, sc.k);                                              \
            return;                                                           \
        }                                                                     \
    } while (0)

// set-up scalars from the initial r.r; block 0 records ||r_0||
__device__ __forceinline__ void init_scalars(const KrylovArgs& a, KScalars& sc, const ff& rr) {
    const double rr0 = ff_to_double(rr);
    sc.rr = rr;
    sc.thr2 = ff_norm(ff_from_double(fmax(a.atol2, a.rtol2 * rr0)));
    sc.go = (0 < a.maxiter && ff_gt(sc.rr, sc.thr2));
    if (blockIdx.x == 0) a.stats->initial_residual = sqrt(rr0);
}

__device__ void write_stats(const KrylovArgs& a, const KScalars& sc) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        int st = sc.status;
        if (st == WCFD_OK && !ff_le(sc.rr, sc.thr2)) st = WCFD_NOT_CONVERGED;
        a.stats->iterations = sc.k;
        a.stats->status = st;
        a.stats->residual = sqrt(ff_to_double(sc.rr));
    }
}

// Rows of the grid CG are worked on in chunks of kChunk consecutive rows by one warp, lane `lane`
// taking the rows lane, lane + 32, ... of it.  A chunk is regular when in each off-diagonal
// slot all its rows have the same column offset (or no neighbour: zero coefficient, own
// column) and every row of it exists: with the off-diagonals in place (wcfd_mesh.slot_mask)
// a structured numbering's chunks are, beside boundaries too.  The offsets are written down
// once per solve; a regular chunk then needs no column loads and one address per slot for
// all of a lane's rows.  An irregular chunk reads its columns from the mesh.
template <int W>
struct alignas(16) ChunkCols {
    int d[W > 4 ? 8 : 4];  // d[0] = kIrregular: not regular
};
constexpr int kIrregular = INT_MIN;

// Jacobi-preconditioned CG on a scalar system, W = off-diagonal width known at compile
// time so the loads of a row's coefficients and gathered values are all in flight at once.
// Workspace: r, pA, pB, q, invd, z (6 C floats; r, q and invd only of rows that do not fit
// shared memory).
//
// Block b owns the rows [b R, (b + 1) R) for the whole solve, warp w of it the chunks w,
// w + CGB / 32, ... of those.  What only the owner of a row touches stays in shared memory,
// for as many of the block's rows as fit (KrylovArgs::part rows: r, q, x; full rows: 1/diag
// too): a 128^3 system's x, r and q lie in the 152 SMs' shared memory whole.
//
// Per iteration: (1) p_new = z + beta p_old for the row and every neighbour, q = A p_new,
// p.q -- and x += alpha_prev p_old, the previous iteration's solution update, which reads
// the p_old this pass loads anyway; (2) r -= alpha q, z = r / diag, r.r and r.z.
//
// NR, the rows of a lane in a chunk: a block's rows are best covered in one pass over them (the
// loads of all are then in flight at once), so NR follows the rows per block up to 4
// (cg_kernel_for).  Measured per iteration: 1,000 rows per block (61x47x53 hexes) 5.2 us with
// NR = 2, 5.8 with 3; 1,064 (30x31x29x6 tetrahedra) 6.0 with 3, 6.7 with 2; 1,628 (cylinder)
// 6.2 with 4, 7.0 with 2; on more rows than 4 per thread 3 is the fastest (128^3: 22.4 us,
// 23.2 with 2, 26.0 with 1,024 threads of one row each).
template <int W, int NR>
__global__ void __launch_bounds__(CGB, 1) cg_kernel(KrylovArgs a) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ KScalars sc;
    __shared__ ff sbuf[2 * CGB / 2];
    constexpr int WA = W > 0 ? W : 1;  // no zero-length arrays for W = 0
    constexpr int kChunk = 32 * NR;    // rows of a warp at a time
    constexpr int STEP = CGB / 32 * kChunk;
    const int C = a.m.n_cells;
    const int t = threadIdx.x, lane = t & 31;
    const int row0 = blockIdx.x * a.rows;
    const int nloc = min(a.rows, C - row0);
    const int part = a.part, full = a.full, tab = W > 0 ? a.tab : 0;
    ChunkCols<W>* cols = reinterpret_cast<ChunkCols<W>*>(dyn);
    float* s_r = reinterpret_cast<float*>(cols + tab / kChunk);
    float* s_q = s_r + part;
    float* s_x = s_q + part;
    float* s_i = s_x + part;
    float* const r = a.ws;
    float* const pA = a.ws + (size_t)C;
    float* const pB = a.ws + 2 * (size_t)C;
    float* const q = a.ws + 3 * (size_t)C;
    float* const invd = a.ws + 4 * (size_t)C;
    float* const z = a.ws + 5 * (size_t)C;
    const float* __restrict__ b = a.A.rhs;
    const float* __restrict__ diag = a.A.diag;
    const float* __restrict__ off = a.A.off;
    const int* __restrict__ col = a.m.ell_col;
    const int16_t* __restrict__ dcol = a.m.ell_dcol;
    float* x = a.x;
    const int lw = (t >> 5) * kChunk;  // this warp's first chunk
    const bool in_place = slot_bits(a.m) != 0u;
    unsigned phase = 0;
    if (t == 0) {
        sc.k = 0;
        sc.status = WCFD_OK;
    }

    // r = b - A x ; z = M r ; p = z ; rr = r.r ; rz = r.z ; bb = b.b ; the chunks' offsets
    ff acc[2] = {ff_zero(), ff_zero()}, accb[1] = {ff_zero()};
    for (int l0 = lw; l0 < nloc; l0 += STEP) {
        int d[WA];
        unsigned seen = 0;
        bool regular = l0 + kChunk <= nloc;
#pragma unroll
        for (int j = 0; j < W; ++j) d[j] = 0;
        int c[NR][WA];
        float o[NR][WA], xc[NR][WA];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            const int i = row0 + min(l0 + 32 * k + lane, nloc - 1);
            ell_columns<W>(c[k], col, dcol, C, i);
#pragma unroll
            for (int j = 0; j < W; ++j) o[k][j] = off[(size_t)j * C + i];
        }
#pragma unroll
        for (int k = 0; k < NR; ++k)
#pragma unroll
            for (int j = 0; j < W; ++j) xc[k][j] = x[c[k][j]];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            const int l = l0 + 32 * k + lane;
            const int i = row0 + min(l, nloc - 1);
#pragma unroll
            for (int j = 0; j < W; ++j) {
                // the slot's offset: the first one seen in the chunk
                const bool real = c[k][j] != i;
                const unsigned has = __ballot_sync(0xffffffffu, real);
                if (!((seen >> j) & 1u) && has) {
                    d[j] = __shfl_sync(0xffffffffu, c[k][j] - i, __ffs(has) - 1);
                    seen |= 1u << j;
                }
                // (a caller's matrix may hold a coefficient on the own column of a padding slot)
                regular = regular && (real ? c[k][j] - i == d[j] : o[k][j] == 0.0f);
            }
            if (l >= nloc) continue;
            const float xi = x[i], di = diag[i];
            const float ax = row_product<W>(di, xi, o[k], xc[k], in_place);
            const float bi = b[i];
            const float ri = bi - ax;
            const float vi = jacobi(di);
            const float zi = ri * vi;
            if (l0 < part) {
                s_r[l] = ri;
                s_x[l] = xi;
            } else {
                r[i] = ri;
            }
            if (l0 < full) s_i[l] = vi;
            else invd[i] = vi;
            z[i] = zi;
            pA[i] = zi;
            ff_fma(acc[0], ri, ri);
            ff_fma(acc[1], ri, zi);
            ff_fma(accb[0], bi, bi);
        }
        if (l0 < tab) {
            // the rows' addresses all lie in the vectors, absent neighbours' included
#pragma unroll
            for (int j = 0; j < W; ++j)
                regular = regular && row0 + l0 + (long long)d[j] >= 0 && row0 + l0 + kChunk - 1 + (long long)d[j] < C;
            regular = __all_sync(0xffffffffu, regular);
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < W; ++j) cols[l0 / kChunk].d[j] = regular ? d[j] : kIrregular;
            }
        }
    }
    REDUCE(1, accb, [&](const ff* s) {
        if (threadIdx.x == 0 && blockIdx.x == 0) a.stats->rhs_norm = sqrt(ff_to_double(s[0]));
    });
    REDUCE(2, acc, [&](const ff* s) {
        if (threadIdx.x != 0) return;
        init_scalars(a, sc, s[0]);
        sc.rz = s[1];
        sc.bf = 0.0f;  // the first direction is z itself
    });
    int cur = 0;
    float pending = 0.0f;  // alpha of the last completed iteration, not yet added to x
    while (sc.go) {
        const float bf = sc.bf;
        const float ap = pending;
        const float* po = cur ? pB : pA;  // written by other blocks in this launch: no restrict
        float* pn = cur ? pA : pB;
        // x += alpha_prev p_old ; p_new = z + beta p_old (row and neighbours) ; q = A p_new ; p.q
        ff accq[1] = {ff_zero()};
        for (int l0 = lw; l0 < nloc; l0 += STEP) {
            const int l = l0 + lane, i = row0 + l;
            const bool inside = l0 + kChunk <= nloc;
            float o[NR][WA], zc[NR][WA], pc[NR][WA], zo[NR], poi[NR], dd[NR];
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                const int ik = row0 + min(l + 32 * k, nloc - 1);
#pragma unroll
                for (int j = 0; j < W; ++j) o[k][j] = __ldg(off + (size_t)j * C + ik);
                dd[k] = diag[ik];
            }
            if (W > 0 && l0 < tab && cols[l0 / kChunk].d[0] != kIrregular) {
                const ChunkCols<W> rec = cols[l0 / kChunk];
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const float* zj = z + i + rec.d[j];
                    const float* pj = po + i + rec.d[j];
#pragma unroll
                    for (int k = 0; k < NR; ++k) {
                        zc[k][j] = zj[32 * k];
                        pc[k][j] = pj[32 * k];
                    }
                }
            } else {
                int c[NR][WA];
#pragma unroll
                for (int k = 0; k < NR; ++k) ell_columns<W>(c[k], col, dcol, C, row0 + min(l + 32 * k, nloc - 1));
#pragma unroll
                for (int k = 0; k < NR; ++k)
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        zc[k][j] = z[c[k][j]];
                        pc[k][j] = po[c[k][j]];
                    }
            }
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                if (!inside && l + 32 * k >= nloc) continue;
                zo[k] = z[i + 32 * k];
                poi[k] = po[i + 32 * k];
            }
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                if (!inside && l + 32 * k >= nloc) continue;
                const float pi = zo[k] + bf * poi[k];
#pragma unroll
                for (int j = 0; j < W; ++j) zc[k][j] += bf * pc[k][j];
                const float qi = row_product<W>(dd[k], pi, o[k], zc[k], in_place);
                if (l0 < part) {
                    if (ap != 0.0f) s_x[l + 32 * k] += ap * poi[k];
                    s_q[l + 32 * k] = qi;
                } else {
                    if (ap != 0.0f) x[i + 32 * k] += ap * poi[k];
                    q[i + 32 * k] = qi;
                }
                pn[i + 32 * k] = pi;
                ff_fma(accq[0], pi, qi);
            }
        }
        REDUCE(1, accq, [&](const ff* pq) {
            if (threadIdx.x != 0) return;
            if (pq[0].hi == 0.0f) {
                sc.status = WCFD_KRYLOV_BREAKDOWN;
                sc.go = 0;
            } else {
                sc.af = ff_div_to_float(sc.rz, pq[0]);
            }
        });
        pending = 0.0f;  // alpha_prev p_old is in x now
        if (!sc.go) break;
        const float af = sc.af;
        // r -= alpha q ; z = M r ; rr ; rz
        ff acc2[2] = {ff_zero(), ff_zero()};
        for (int l0 = lw; l0 < nloc; l0 += STEP) {
            const int l = l0 + lane, i = row0 + l;
            const bool inside = l0 + kChunk <= nloc;
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                if (!inside && l + 32 * k >= nloc) continue;
                float ri;
                if (l0 < part) {
                    ri = s_r[l + 32 * k] - af * s_q[l + 32 * k];
                    s_r[l + 32 * k] = ri;
                } else {
                    ri = r[i + 32 * k] - af * q[i + 32 * k];
                    r[i + 32 * k] = ri;
                }
                const float zi = ri * (l0 < full ? s_i[l + 32 * k] : invd[i + 32 * k]);
                z[i + 32 * k] = zi;
                ff_fma(acc2[0], ri, ri);
                ff_fma(acc2[1], ri, zi);
            }
        }
        REDUCE(2, acc2, [&](const ff* s) {
            if (threadIdx.x != 0) return;
            sc.rr = s[0];
            sc.bf = sc.rz.hi != 0.0f ? ff_div_to_float(s[1], sc.rz) : 0.0f;
            sc.rz = s[1];
            sc.k += 1;
            sc.go = (sc.k < a.maxiter && ff_gt(sc.rr, sc.thr2));
        });
        pending = af;
        cur ^= 1;
    }
    // the last iteration's x += alpha p (its p is the current buffer's)
    const float* pl = cur ? pB : pA;
    for (int l0 = lw; l0 < nloc; l0 += STEP) {
        for (int l = l0 + lane; l < min(l0 + kChunk, nloc); l += 32) {
            const int i = row0 + l;
            if (l0 < part) x[i] = pending != 0.0f ? s_x[l] + pending * pl[i] : s_x[l];
            else if (pending != 0.0f) x[i] += pending * pl[i];
        }
    }
    write_stats(a, sc);
}

// BiCGSTAB (bicgstab.cuh) over the grid, a.rows contiguous rows a block; RES: with the rows' own
// data in shared memory.
template <int W, bool RES>
__global__ void __launch_bounds__(kCgBlock, 1) bicgstab_kernel(KrylovArgs a) {
    extern __shared__ __align__(16) float own[];
    __shared__ BiScalars sc;
    __shared__ ff sbuf[kCgBlock];
    const int C = a.m.n_cells, row0 = (int)blockIdx.x * a.rows;
    const BiSystem sys{a.A.diag, a.A.off, a.A.rhs, a.m.ell_col, a.m.ell_dcol, a.x, C, a.maxiter, slot_bits(a.m) != 0u, a.atol2, a.rtol2, a.stats};
    BiGlobal<kCgBlock, false> net(a.ws, C, row0);
    net.g = a.g;
    net.sbuf = sbuf;
    if (!bicgstab_body<W, kCgBlock, RES>(sys, net, sc, own, a.rows, row0, max(0, min(a.rows, C - row0)), blockIdx.x == 0))
        fail_stats(a, sc.k);
}
const void* bicgstab_kernel_for(int W, bool resident) {
#define WCFD_BI(w) case w: return resident ? (const void*)bicgstab_kernel<w, true> : (const void*)bicgstab_kernel<w, false>;
    switch (W) {
        WCFD_BI(0) WCFD_BI(1) WCFD_BI(2) WCFD_BI(3) WCFD_BI(4) WCFD_BI(5) WCFD_BI(6)
        default: return nullptr;
    }
#undef WCFD_BI
}
size_t bicgstab_row_bytes(int W) { return sizeof(float) * (kBiPlanes + 2 * (size_t)W); }

// ---------------------------------------------------------------------------------
// fp64 iterative refinement of a scalar solve (the precision form of the pressure solve):
// the solution is kept in fp64 and each sweep solves for a correction with the fp32 CG
// against the residual r = b - A x computed in fp64.  The few fp64 operations per row per
// sweep (not per Krylov iteration) are affordable at GB300's fp64 rate.
template <int W>
__global__ void __launch_bounds__(kBlock) residual64_kernel(wcfd_mesh m, wcfd_system A, const double* __restrict__ x,
                                                            float* __restrict__ r) {
    const int i = blockIdx.x * kBlock + threadIdx.x;
    const int C = m.n_cells;
    if (i >= C) return;
    double acc = (double)A.diag[i] * x[i];
#pragma unroll
    for (int j = 0; j < W; ++j) acc += (double)A.off[(size_t)j * C + i] * x[m.ell_col[(size_t)j * C + i]];
    r[i] = (float)((double)A.rhs[i] - acc);
}

// running total of the correction solves' iterations over the refinement sweeps; the last
// sweep writes the total into its statistics
__global__ void refine_count_kernel(wcfd_solve_stats* stats, int* acc, int first, int last) {
    const int a = (first ? 0 : *acc) + stats->iterations;
    *acc = a;
    if (last) stats->iterations = a;
}

__global__ void __launch_bounds__(kBlock) refine_update_kernel(int C, double* __restrict__ x64,
                                                               const float* __restrict__ d, float* __restrict__ x32) {
    const int i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= C) return;
    const double v = x64[i] + (double)d[i];
    x64[i] = v;
    x32[i] = (float)v;
}

const void* residual64_kernel_for(int W) {
    switch (W) {
        case 0: return (const void*)residual64_kernel<0>;
        case 1: return (const void*)residual64_kernel<1>;
        case 2: return (const void*)residual64_kernel<2>;
        case 3: return (const void*)residual64_kernel<3>;
        case 4: return (const void*)residual64_kernel<4>;
        case 5: return (const void*)residual64_kernel<5>;
        case 6: return (const void*)residual64_kernel<6>;
        default: return nullptr;
    }
}

// Self-check of the grid barrier: `phases` barriers of two sums over all blocks; every block
// checks the sums it receives against their closed form and ORs 1 into *bad on a mismatch.
// With skip >= 0 that block returns before it arrives at the first barrier, so every other
// block's wait runs out: they record WCFD_BARRIER_TIMEOUT in the error word and return (a
// failure made without a fault: nothing ever sets the count they wait for).
__global__ void __launch_bounds__(BS, 1) barrier_check_kernel(GridCtl g, int skip, int phases, int* bad) {
    if ((int)blockIdx.x == skip) return;
    __shared__ ff sbuf[2 * BS / 2];
    unsigned phase = 0;
    const float G = (float)gridDim.x;
    for (int p = 0; p < phases; ++p) {
        ff acc[2] = {ff{(float)(blockIdx.x + 1 + p), 0.0f}, ff{1.0f, 0.0f}};
        if (threadIdx.x != 0) acc[0] = acc[1] = ff_zero();
        const bool ok = grid_reduce<2, BS>(g, acc, sbuf, ++phase, [&](const ff* s) {
            const float want0 = G * (G + 1.0f) * 0.5f + G * (float)p;  // exact below 2^24
            if (threadIdx.x == 0 && (ff_to_double(s[0]) != (double)want0 || ff_to_double(s[1]) != (double)G))
                atomicOr(bad, 1);
        });
        if (!ok) return;
    }
}

const void* barrier_check_kernel_ptr() { return (const void*)barrier_check_kernel; }

template <int NR>
const void* cg_kernel_pick(int W) {
    switch (W) {
        case 0: return (const void*)cg_kernel<0, NR>;
        case 1: return (const void*)cg_kernel<1, NR>;
        case 2: return (const void*)cg_kernel<2, NR>;
        case 3: return (const void*)cg_kernel<3, NR>;
        case 4: return (const void*)cg_kernel<4, NR>;
        case 5: return (const void*)cg_kernel<5, NR>;
        case 6: return (const void*)cg_kernel<6, NR>;
        default: return nullptr;
    }
}


size_t cg_chunk_bytes(int W) { return W > 4 ? sizeof(ChunkCols<5>) : W > 0 ? sizeof(ChunkCols<4>) : 0; }

CgKernel cg_kernel_for(int W, int rows) {
    switch ((rows + CGB - 1) / CGB) {
        case 0:
        case 1: return CgKernel{cg_kernel_pick<1>(W), 32};
        case 2: return CgKernel{cg_kernel_pick<2>(W), 64};
        case 4: return CgKernel{cg_kernel_pick<4>(W), 128};
        default: return CgKernel{cg_kernel_pick<3>(W), 96};
    }
}

}  // namespace wcfd
