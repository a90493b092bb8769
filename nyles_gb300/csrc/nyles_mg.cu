// Geometric multigrid of the pressure projection, one rank (core/mgfor).
//
// Level arrays hold interior cells only. The ghost layers of the reference are implied:
// across a closed wall a ghost holds 0 and is "dry" (mask 0), in a periodic direction
// it is the periodic image of the interior (mod_halo.f90:235-262). With that, every
// operator coefficient of mgfor's setup (operators.f90:299-505) is a function of the
// cell position and is evaluated in the kernels instead of being stored:
//   diag  = number of wet face neighbours, idiag = 1/diag     (compute_diag)
//   Rcoef = 1/2 on every coarse interior cell                   (compute_Rcoef)
//   Pcoef = 1/(Wx*Wy*Wz), W = 3 + [coarse neighbour is wet]     (compute_Pcoef)
// The smoother's intermediate `y` on the ghost ring (basicoperators.f90:380-388) is 0
// across closed walls (its idiag and x are 0 there) and the periodic image otherwise.
//
// Kernel layout: blocks of 32 x 8 threads over (x, y); each thread marches over a chunk
// of z, keeping the z-1, z, z+1 values in registers. A block whose cells and stencil
// neighbours all lie inside the level takes a fast path with direct strided loads;
// only blocks touching the level's faces go through the ghost logic.
#include "nyles_internal.h"
#include "nyles_fx.cuh"
#include <cooperative_groups.h>
#include <type_traits>
#include <cstdlib>
#include <vector>
#include <cstring>

namespace nyles {

struct MgGeom {
    int n[3];          // interior extents z, y, x
    int per[3];
    double idiag[8];   // omega/diag for diag = 0..6 (0 -> 0): the damped inverse diagonal, host-computed
    double pcoef[8];   // 1/(Wx*Wy*Wz) indexed by the three "neighbour is wet" bits
    float fidiag[8];   // the same tables rounded to float: single-precision kernels read
    float fpcoef[8];   // these instead of converting (FP64 conversions use the FP64 pipe)
};
template <typename T> __device__ __forceinline__ T mg_idiag(const MgGeom& g, int k);
template <> __device__ __forceinline__ double mg_idiag<double>(const MgGeom& g, int k) { return g.idiag[k]; }
template <> __device__ __forceinline__ float mg_idiag<float>(const MgGeom& g, int k) { return g.fidiag[k]; }
template <typename T> __device__ __forceinline__ T mg_pcoef(const MgGeom& g, int k);
template <> __device__ __forceinline__ double mg_pcoef<double>(const MgGeom& g, int k) { return g.pcoef[k]; }
template <> __device__ __forceinline__ float mg_pcoef<float>(const MgGeom& g, int k) { return g.fpcoef[k]; }

// Scalars of the solve in the workspace: [0] last sum(r^2), [1] sum(b^2), [2] res,
// [3] nite of the current solve, [4] V-cycles since creation, [5] and [6] the scale of
// the mixed-precision residual sums and its inverse square.
// device scalars of the solver (SC_COUNT <= 16 doubles, zeroed when the workspace is
// bound): slots 7-12 belong to the Krylov solve; SC_NCONV counts graph-mode solves
// that stopped at maxite above tol, SC_NONFINITE graph-mode solves stopped by a
// non-finite norm
enum { SC_RR = 0, SC_NORMB = 1, SC_RES = 2, SC_NITE = 3, SC_TOTAL = 4, SC_SCALE = 5, SC_INVSCALE2 = 6,
       SC_ZQ = 7, SC_PQ = 8, SC_PR = 9, SC_BETA = 10, SC_ALPHA = 11, SC_ZMEAN = 12,
       SC_NCONV = 13, SC_NONFINITE = 14, SC_COUNT = 15 };
static_assert(SC_COUNT <= 16, "multigrid scalars exceed their 16-double slot");

constexpr int MG_BX = 32, MG_BY = 8, MG_ZC = 8;    // stencil kernels
constexpr int MG_RZC = 2;                          // restriction (coarse z per thread)
constexpr int MG_DFZC = 8;                         // float-pair residual

__device__ __forceinline__ long long mg_at(const MgGeom& g, int z, int y, int x) {
    return ((long long)z * g.n[1] + y) * g.n[2] + x;
}

// Value at (z, y, x), one cell outside the interior at most: periodic image, or 0
// across a closed wall. Branch-free on purpose: the index is folded into range, the
// load always reads an interior cell and the wall case is a select. With early
// returns before the load, the fused residual-restriction kernel built by ptxas -O3
// (CUDA 13.0, sm_103a) returned wrong sums next to closed x walls, while the same
// source was exact on the host and with -Xptxas -O0; this form is exact in both.
template <typename T>
__device__ __forceinline__ T mg_rd(const T* __restrict__ a, const MgGeom& g, int z, int y, int x) {
    bool ok = true;
    int q[3] = {z, y, x};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int n = g.n[k];
        const bool lo = q[k] < 0, hi = q[k] >= n;
        ok = ok && (g.per[k] || !(lo || hi));
        q[k] = lo ? q[k] + n : (hi ? q[k] - n : q[k]);
        q[k] = min(max(q[k], 0), n - 1);
    }
    const T v = a[((long long)q[0] * g.n[1] + q[1]) * g.n[2] + q[2]];
    return ok ? v : T(0);
}

__device__ __forceinline__ int mg_diag(const MgGeom& g, int z, int y, int x) {
    int d = 0;
    d += g.per[0] ? 2 : ((z > 0) + (z < g.n[0] - 1));
    d += g.per[1] ? 2 : ((y > 0) + (y < g.n[1] - 1));
    d += g.per[2] ? 2 : ((x > 0) + (x < g.n[2] - 1));
    return d;
}

// sum of the six face neighbours in mgfor's order: x-1, x+1, y-1, y+1, z-1, z+1
template <typename T>
__device__ __forceinline__ T mg_nsum(const T* __restrict__ a, const MgGeom& g, int z, int y, int x) {
    return ((((mg_rd(a, g, z, y, x - 1) + mg_rd(a, g, z, y, x + 1)) + mg_rd(a, g, z, y - 1, x)) +
             mg_rd(a, g, z, y + 1, x)) + mg_rd(a, g, z - 1, y, x)) + mg_rd(a, g, z + 1, y, x);
}

// residual r = msk*(b + diag*x - sum(x_nb)) (basicoperators.f90:300-323), ghost logic
template <typename T>
__device__ __forceinline__ T mg_resid(const T* __restrict__ x, const T* __restrict__ b, const MgGeom& g, int z, int y,
                                      int xx) {
    const long long c = mg_at(g, z, y, xx);
    const T dg = T(mg_diag(g, z, y, xx));
    return (b[c] + dg * x[c]) - mg_nsum(x, g, z, y, xx);
}
// ---- per-cell operators with the ghost logic (used where a kernel's chunks end)
// sum of the residuals of the 8 children of coarse cell (z, y, x)
template <typename T>
__device__ __forceinline__ T mg_restrict_cell(const MgGeom& gf, const T* __restrict__ xf, const T* __restrict__ bf,
                                              int z, int y, int x) {
    const int i = 2 * x, j = 2 * y, k = 2 * z;
    T s = mg_resid(xf, bf, gf, k, j, i);
    s = s + mg_resid(xf, bf, gf, k, j, i + 1);
    s = s + mg_resid(xf, bf, gf, k, j + 1, i);
    s = s + mg_resid(xf, bf, gf, k, j + 1, i + 1);
    s = s + mg_resid(xf, bf, gf, k + 1, j, i);
    s = s + mg_resid(xf, bf, gf, k + 1, j, i + 1);
    s = s + mg_resid(xf, bf, gf, k + 1, j + 1, i);
    s = s + mg_resid(xf, bf, gf, k + 1, j + 1, i + 1);
    return s;
}
// 9-3-3-1 prolongation increment of fine cell (z, y, x)
template <typename T>
__device__ __forceinline__ T mg_prolong_cell(const MgGeom& gf, const MgGeom& gc, const T* __restrict__ xc, int z,
                                             int y, int x) {
    const int ic = x >> 1, jc = y >> 1, kc = z >> 1;
    const int si = (x & 1) ? 1 : -1, sj = (y & 1) ? 1 : -1, sk = (z & 1) ? 1 : -1;
    auto plane = [&](int kk) -> T {
        return ((T(9) * mg_rd(xc, gc, kk, jc, ic) + T(3) * mg_rd(xc, gc, kk, jc, ic + si)) +
                T(3) * mg_rd(xc, gc, kk, jc + sj, ic)) + mg_rd(xc, gc, kk, jc + sj, ic + si);
    };
    const T bpl = plane(kc);
    const T opl = plane(kc + sk);
    auto wet = [&](int d, int v) -> int { return (gc.per[d] || (v >= 0 && v < gc.n[d])) ? 1 : 0; };
    const T pcoef = mg_pcoef<T>(gf, wet(2, ic + si) | (wet(1, jc + sj) << 1) | (wet(0, kc + sk) << 2));
    return pcoef * (T(3) * bpl + opl);
}

// ---- grid kernels: one thread per (x, y) column and chunk of z
// The neighbours of a thread's fixed coordinate along one direction: element offsets
// of the cells at c-1 and c+1 and whether they are wet. Outside the level a neighbour
// is the periodic image or, across a closed wall, dry: its offset is then 0 (the cell
// itself, a valid address) and the value read is replaced by 0 — loads are never
// skipped (see mg_rd).
struct MgNb {
    long long om, op;
    bool wm, wp;
};
__device__ __forceinline__ MgNb mg_nb(int c, int n, int per, long long stride) {
    MgNb r;
    r.wm = c > 0 || per;
    r.wp = c < n - 1 || per;
    r.om = c > 0 ? -stride : (per ? (long long)(n - 1) * stride : 0);
    r.op = c < n - 1 ? stride : (per ? -(long long)(n - 1) * stride : 0);
    return r;
}
template <typename T>
__device__ __forceinline__ T mg_ldw(const T* __restrict__ a, long long c, bool wet) {
    const T v = a[c];
    return wet ? v : T(0);
}

// per-block partial sum (one double per block, block index order); bz = the block's z
// index within its run's grid (blockIdx.z outside batched launches)
__device__ __forceinline__ void block_partial(double s, double* __restrict__ partial, int bz) {
    __shared__ double sm[MG_BX * MG_BY / 32];
    const int tid = threadIdx.y * MG_BX + threadIdx.x;
    s = warp_sum(s);
    if ((tid & 31) == 0) sm[tid >> 5] = s;
    __syncthreads();
    if (tid < 32) {
        double t = (tid < MG_BX * MG_BY / 32) ? sm[tid] : 0.0;
        t = warp_sum(t);
        if (tid == 0) partial[(bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = t;
    }
}

// two per-block partial sums at once
__device__ __forceinline__ void block_partial2(double s, double t, double* __restrict__ ps,
                                               double* __restrict__ pt, int bz) {
    __shared__ double sm[2][MG_BX * MG_BY / 32];
    const int tid = threadIdx.y * MG_BX + threadIdx.x;
    s = warp_sum(s);
    t = warp_sum(t);
    if ((tid & 31) == 0) {
        sm[0][tid >> 5] = s;
        sm[1][tid >> 5] = t;
    }
    __syncthreads();
    if (tid < 32) {
        double a = (tid < MG_BX * MG_BY / 32) ? sm[0][tid] : 0.0;
        double b = (tid < MG_BX * MG_BY / 32) ? sm[1][tid] : 0.0;
        a = warp_sum(a);
        b = warp_sum(b);
        if (tid == 0) {
            const int blk = (bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
            ps[blk] = a;
            pt[blk] = b;
        }
    }
}

// FP32 forms of block_partial and block_partial2 for kernels whose per-thread sums are
// FP32: the warp and block stages add in float and only the block total is stored as a
// double (times `scale`). On GB300 the FP64 pipe is narrow: the double shuffles, adds
// and conversions of a 256-thread reduction took a visible share of a level-0 pass.
__device__ __forceinline__ void block_partial_f(float s, double scale, double* __restrict__ partial, int bz) {
    __shared__ float smf[MG_BX * MG_BY / 32];
    const int tid = threadIdx.y * MG_BX + threadIdx.x;
    s = warp_sum(s);
    if ((tid & 31) == 0) smf[tid >> 5] = s;
    __syncthreads();
    if (tid < 32) {
        float t = (tid < MG_BX * MG_BY / 32) ? smf[tid] : 0.f;
        t = warp_sum(t);
        if (tid == 0) partial[(bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = (double)t * scale;
    }
}
__device__ __forceinline__ void block_partial2_f(float s, float t, double* __restrict__ ps, double* __restrict__ pt,
                                                 int bz) {
    __shared__ float smf[2][MG_BX * MG_BY / 32];
    const int tid = threadIdx.y * MG_BX + threadIdx.x;
    s = warp_sum(s);
    t = warp_sum(t);
    if ((tid & 31) == 0) {
        smf[0][tid >> 5] = s;
        smf[1][tid >> 5] = t;
    }
    __syncthreads();
    if (tid < 32) {
        float a = (tid < MG_BX * MG_BY / 32) ? smf[0][tid] : 0.f;
        float b = (tid < MG_BX * MG_BY / 32) ? smf[1][tid] : 0.f;
        a = warp_sum(a);
        b = warp_sum(b);
        if (tid == 0) {
            const int blk = (bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
            ps[blk] = (double)a;
            pt[blk] = (double)b;
        }
    }
}

// ---- the final sum of a reduction folded into the kernel that stores the partials
// The block that stores its partial last (a ticket from an atomic counter, taken after
// a fence that orders every block's partial store before its ticket) adds all partials
// in block order and finishes the reduction itself, instead of a separate one-block
// launch after the kernel; it resets the counter for the next launch. `ticket` lies in
// the solver's workspace (zeroed when the workspace is bound; batched launches: each
// run's own). The sum's order depends on the grid only, so results are deterministic.
struct MgFin {
    unsigned int* ticket = nullptr;   // null: the partials are summed by a later launch
    double* sc = nullptr;             // the solve's scalars (shifted to the run in batched launches)
    int k = 0;                        // Krylov iteration (-1: read sc[SC_NITE])
    double vol = 0.0;                 // level-0 cells
};
// Thread (0, 0) stored the block's partial (block_partial*): it alone fences that store
// before taking the ticket (a fence in every thread stalled every block on its way out).
__device__ __forceinline__ bool mg_last_block(unsigned int* ticket, unsigned int nblk) {
    __shared__ unsigned int s_last;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        __threadfence();
        const unsigned int t = atomicAdd(ticket, 1u);
        s_last = (t == nblk - 1) ? 1u : 0u;
        if (s_last) atomicExch(ticket, 0u);
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}
// totals of n partials of one or two sums, added in a fixed order by the threads of a
// MG_BX x MG_BY block (loads through L2: other blocks of the launch stored them); the
// result is valid in thread (0, 0)
__device__ __forceinline__ double2 mg_block_total2(const double* pa, const double* pb, int n) {
    __shared__ double sm[2][MG_BX * MG_BY / 32];
    const int tid = threadIdx.y * MG_BX + threadIdx.x;
    double a = 0.0, b = 0.0;
    for (int i = tid; i < n; i += MG_BX * MG_BY) {
        a += __ldcg(pa + i);
        if (pb) b += __ldcg(pb + i);
    }
    a = warp_sum(a);
    b = warp_sum(b);
    if ((tid & 31) == 0) {
        sm[0][tid >> 5] = a;
        sm[1][tid >> 5] = b;
    }
    __syncthreads();
    double2 r = make_double2(0.0, 0.0);
    if (tid < 32) {
        double x = (tid < MG_BX * MG_BY / 32) ? sm[0][tid] : 0.0;
        double y = (tid < MG_BX * MG_BY / 32) ? sm[1][tid] : 0.0;
        x = warp_sum(x);
        y = warp_sum(y);
        r = make_double2(x, y);
    }
    return r;
}
// the same for a kernel of one sum: the total in the last block's thread (0, 0) (false elsewhere)
__device__ __forceinline__ bool mg_fin_total(const MgFin& fin, const double* partial, unsigned int nblk, double& total) {
    if (!mg_last_block(fin.ticket, nblk)) return false;
    total = mg_block_total2(partial, nullptr, (int)nblk).x;
    return threadIdx.x == 0 && threadIdx.y == 0;
}
// beta = -(z.q)/(p.q) of the previous iteration (0 on the first: k = iteration of this
// solve, or sc[SC_NITE] when k < 0) stored as a float, and the mean of z (float)
__device__ __forceinline__ void fcg_set_beta(double zq, double zs, double vol, double* sc, int k) {
    const int it = k >= 0 ? k : (int)sc[SC_NITE];
    const double pq = sc[SC_PQ];
    double beta = (it > 0 && pq != 0.0) ? -zq / pq : 0.0;
    if (!isfinite(beta)) beta = 0.0;
    double zmean = zs / vol;
    if (!isfinite(zmean)) zmean = 0.0;
    sc[SC_ZQ] = zq;
    reinterpret_cast<float*>(sc + SC_BETA)[0] = (float)beta;
    reinterpret_cast<float*>(sc + SC_ZMEAN)[0] = (float)zmean;
}
// alpha = (p.r)/(p.q) stored as a float pair
__device__ __forceinline__ void fcg_set_alpha(double pq, double pr, double* sc) {
    double alpha = pq != 0.0 ? pr / pq : 0.0;
    if (!isfinite(alpha)) alpha = 0.0;
    sc[SC_PQ] = pq;
    sc[SC_PR] = pr;
    const float hi = (float)alpha;
    float2* a2 = reinterpret_cast<float2*>(sc + SC_ALPHA);
    *a2 = make_float2(hi, (float)(alpha - (double)hi));
}

// one damped-Jacobi half-sweep, out = (1-omega)*in + omega*(sum(in_nb) - b)*idiag
// (basicoperators.f90:379-398). MODE 0 stores it; MODE 1 adds it to the float-pair
// solution `acc` instead (mixed precision: the correction of iterative refinement,
// fused into the last half-sweep of the V-cycle); MODE 2 stores it and sums out*dot
// and out per block into `partial` and `partial2` (the Krylov solve: z.q of the new
// preconditioned residual against the previous direction's image, and the sum of z).
// BAT: batched launch over the runs of `bat` (pointers shifted to each run's memory)
template <typename T, int MODE, bool BAT = false, int ZC = MG_ZC>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_jacobi(const MgGeom g, const T* __restrict__ in,
                                                            const T* __restrict__ b, T* __restrict__ out, T omega,
                                                            float2* __restrict__ acc, const T* __restrict__ dot,
                                                            double* __restrict__ partial,
                                                            double* __restrict__ partial2, const Bat bat = Bat()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        in = bshift(in, dlt);
        b = bshift(b, dlt);
        out = bshift(out, dlt);
        acc = bshift(acc, dlt);
        dot = bshift(dot, dlt);
        partial = bshift(partial, dlt);
        partial2 = bshift(partial2, dlt);
    }
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    float sdot = 0.f, ssum = 0.f;
    if (x < g.n[2] && y < g.n[1]) {
        const int nz = g.n[0], z0 = bz * ZC;
        const long long sy = g.n[2], sz = (long long)g.n[1] * g.n[2];
        const MgNb nx = mg_nb(x, g.n[2], g.per[2], 1), ny = mg_nb(y, g.n[1], g.per[1], sy);
        const int dxy = (int)nx.wm + (int)nx.wp + (int)ny.wm + (int)ny.wp;
        const T cff1 = T(1) - omega;
        const long long c0 = mg_at(g, z0, y, x);
        // neighbour sum in mgfor's order x-1, x+1, y-1, y+1, z-1, z+1
        auto cell = [&](long long c, T zm, T x0, T zp, T idg) -> T {
            const T s = ((((mg_ldw(in, c + nx.om, nx.wm) + mg_ldw(in, c + nx.op, nx.wp)) +
                           mg_ldw(in, c + ny.om, ny.wm)) + mg_ldw(in, c + ny.op, ny.wp)) + zm) + zp;
            return cff1 * x0 + (s - b[c]) * idg;
        };
        // dv: the cell's value of `dot` (MODE 2)
        auto put = [&](long long c, T v, T dv) {
            if (MODE == 1) {
                acc[c] = df_add_f(acc[c], (float)v);
            } else {
                out[c] = v;
                if (MODE == 2) {
                    sdot = __fmaf_rn((float)v, (float)dv, sdot);
                    ssum = __fadd_rn(ssum, (float)v);
                }
            }
        };
        if (z0 + ZC <= nz) {
            // full chunk: fixed trip count, fully unrolled, so that every load of the chunk
            // is issued before the first result is needed
            const MgNb lo = mg_nb(z0, nz, g.per[0], sz), hi = mg_nb(z0 + ZC - 1, nz, g.per[0], sz);
            T col[ZC + 2];
            col[0] = mg_ldw(in, c0 + lo.om, lo.wm);
#pragma unroll
            for (int k = 1; k <= ZC; ++k) col[k] = in[c0 + (k - 1) * sz];
            col[ZC + 1] = mg_ldw(in, c0 + (ZC - 1) * sz + hi.op, hi.wp);
            const T idg = mg_idiag<T>(g, dxy + (ZC == 1 ? (int)lo.wm + (int)hi.wp : 2));
            const T idg_lo = ZC == 1 ? idg : mg_idiag<T>(g, dxy + 1 + (int)lo.wm);
            const T idg_hi = ZC == 1 ? idg : mg_idiag<T>(g, dxy + 1 + (int)hi.wp);
#pragma unroll
            for (int k = 0; k < ZC; ++k) {
                const long long c = c0 + k * sz;
                put(c, cell(c, col[k], col[k + 1], col[k + 2], k == 0 ? idg_lo : (k == ZC - 1 ? idg_hi : idg)),
                    (MODE == 2) ? dot[c] : T(0));
            }
        } else {
            for (int z = z0; z < nz; ++z) {   // last, partial chunk
                const long long c = mg_at(g, z, y, x);
                const MgNb nzb = mg_nb(z, nz, g.per[0], sz);
                const T idg = mg_idiag<T>(g, dxy + (int)nzb.wm + (int)nzb.wp);
                put(c, cell(c, mg_ldw(in, c + nzb.om, nzb.wm), in[c], mg_ldw(in, c + nzb.op, nzb.wp), idg),
                    (MODE == 2) ? dot[c] : T(0));
            }
        }
    }
    if constexpr (MODE == 2) {
        if constexpr (sizeof(T) == sizeof(float))
            block_partial2_f(sdot, ssum, partial, partial2, bz);
        else
            block_partial2((double)sdot, (double)ssum, partial, partial2, bz);
    }
}

// k_mg_jacobi for float levels with 4 consecutive x cells per thread (16-byte accesses;
// the x neighbours of a vector from the adjacent lanes, loaded at the warp's ends and at
// the level's x faces) and z-chunks of V4_ZC cells; needs nx and nz divisible by 4 and
// V4_ZC. Same per-cell arithmetic and modes as k_mg_jacobi.
constexpr int V4_ZC = 4;

// value at c, or 0 across a closed wall (mg_ldw for the float vector kernels)
__device__ __forceinline__ float mg_ldw_f(const float* __restrict__ a, long long c, bool wet) {
    const float v = a[c];
    return wet ? v : 0.f;
}

// One block of the vector half-sweep: block (bx, by, bz) of the grid grid_v4(n, ZC);
// MODE 2 accumulates the block's sums of out*dot and out into sdot and ssum.
template <int MODE, int ZC>
__device__ __forceinline__ void mg_jacobi_v4_blk(const MgGeom& g, const float* __restrict__ in,
                                                 const float* __restrict__ b, float* __restrict__ out, float omega,
                                                 float2* __restrict__ acc, const float* __restrict__ dot, int bx,
                                                 int by, int bz, float& sdot, float& ssum) {
    const int nx = g.n[2], ny = g.n[1], nz = g.n[0];
    const int nx4 = nx >> 2;
    const int lane = threadIdx.x;
    const int xv = bx * MG_BX + lane;
    const int y = by * MG_BY + threadIdx.y;
    // idle lanes shadow the last vector of the row (every lane takes part in the
    // shuffles); only active lanes store and sum
    const bool act = xv < nx4 && y < ny;
    const int x0 = min(xv, nx4 - 1) * 4, ys = min(y, ny - 1);
    const long long sy = nx, sz = (long long)ny * nx;
    const MgNb nyb = mg_nb(ys, ny, g.per[1], sy);
    const bool wl = x0 > 0 || g.per[2], wr = x0 + 4 < nx || g.per[2];
    const long long ol = x0 > 0 ? -1 : (g.per[2] ? (long long)(nx - 1) : 0);
    const long long orr = x0 + 4 < nx ? 4 : (g.per[2] ? (long long)(4 - nx) : 0);
    const bool ownl = lane == 0 || x0 == 0, ownr = lane == MG_BX - 1 || x0 + 4 >= nx;
    int dgx[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int xx = x0 + e;
        dgx[e] = (int)(xx > 0 || g.per[2]) + (int)(xx < nx - 1 || g.per[2]) + (int)nyb.wm + (int)nyb.wp;
    }
    const float cff1 = 1.f - omega;
    const int zb = bz * ZC;
    const long long c00 = (long long)ys * sy + x0;
    auto ld4 = [&](const float* a, long long c) { return *reinterpret_cast<const float4*>(a + c); };
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto zrow = [&](int zz) -> float4 {
        if (zz < 0) return g.per[0] ? ld4(in, c00 + (long long)(nz - 1) * sz) : zero4;
        if (zz >= nz) return g.per[0] ? ld4(in, c00) : zero4;
        return ld4(in, c00 + (long long)zz * sz);
    };
    float4 zm = zrow(zb - 1), zc = zrow(zb);
#pragma unroll
    for (int k = 0; k < ZC; ++k) {
        const int zz = zb + k;
        const float4 zp = zrow(zz + 1);
        const long long c = c00 + (long long)zz * sz;
        const float4 ym = nyb.wm ? ld4(in, c + nyb.om) : zero4;
        const float4 yp = nyb.wp ? ld4(in, c + nyb.op) : zero4;
        const float4 bv = ld4(b, c);
        const float4 dv = (MODE == 2) ? ld4(dot, c) : zero4;
        const float sl = __shfl_up_sync(0xffffffffu, zc.w, 1);
        const float sr = __shfl_down_sync(0xffffffffu, zc.x, 1);
        const float left = ownl ? mg_ldw_f(in, c + ol, wl) : sl;
        const float right = ownr ? mg_ldw_f(in, c + orr, wr) : sr;
        const int dzw = (int)(zz > 0 || g.per[0]) + (int)(zz < nz - 1 || g.per[0]);
        const float xc[4] = {zc.x, zc.y, zc.z, zc.w};
        const float xm[4] = {left, zc.x, zc.y, zc.z}, xp[4] = {zc.y, zc.z, zc.w, right};
        const float ymv[4] = {ym.x, ym.y, ym.z, ym.w}, ypv[4] = {yp.x, yp.y, yp.z, yp.w};
        const float zmv[4] = {zm.x, zm.y, zm.z, zm.w}, zpv[4] = {zp.x, zp.y, zp.z, zp.w};
        const float bb[4] = {bv.x, bv.y, bv.z, bv.w}, dd[4] = {dv.x, dv.y, dv.z, dv.w};
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float s = ((((xm[e] + xp[e]) + ymv[e]) + ypv[e]) + zmv[e]) + zpv[e];
            v[e] = cff1 * xc[e] + (s - bb[e]) * mg_idiag<float>(g, dgx[e] + dzw);
            if (MODE == 2 && act) {
                sdot = __fmaf_rn(v[e], dd[e], sdot);
                ssum = __fadd_rn(ssum, v[e]);
            }
        }
        if (act) {
            if (MODE == 1) {
                float4* a4 = reinterpret_cast<float4*>(acc + c);
                float4 a01 = a4[0], a23 = a4[1];
                float2 r0 = df_add_f(make_float2(a01.x, a01.y), v[0]), r1 = df_add_f(make_float2(a01.z, a01.w), v[1]);
                float2 r2 = df_add_f(make_float2(a23.x, a23.y), v[2]), r3 = df_add_f(make_float2(a23.z, a23.w), v[3]);
                a4[0] = make_float4(r0.x, r0.y, r1.x, r1.y);
                a4[1] = make_float4(r2.x, r2.y, r3.x, r3.y);
            } else {
                *reinterpret_cast<float4*>(out + c) = make_float4(v[0], v[1], v[2], v[3]);
            }
        }
        zm = zc;
        zc = zp;
    }
}

template <int MODE, bool BAT = false, int ZC = V4_ZC>
__global__ void __launch_bounds__(MG_BX * MG_BY, 5) k_mg_jacobi_v4(const MgGeom g, const float* __restrict__ in,
                                                               const float* __restrict__ b, float* __restrict__ out,
                                                               float omega, float2* __restrict__ acc,
                                                               const float* __restrict__ dot,
                                                               double* __restrict__ partial,
                                                               double* __restrict__ partial2, const Bat bat = Bat(),
                                                               const MgFin fin = MgFin()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        in = bshift(in, dlt);
        b = bshift(b, dlt);
        out = bshift(out, dlt);
        acc = bshift(acc, dlt);
        dot = bshift(dot, dlt);
        partial = bshift(partial, dlt);
        partial2 = bshift(partial2, dlt);
    }
    float sdot = 0.f, ssum = 0.f;
    mg_jacobi_v4_blk<MODE, ZC>(g, in, b, out, omega, acc, dot, blockIdx.x, blockIdx.y, bz, sdot, ssum);
    if constexpr (MODE == 2) {
        block_partial2_f(sdot, ssum, partial, partial2, bz);
        // the Krylov solve's beta and mean of z from the totals (k_fcg_final_beta's work)
        if (!BAT && fin.ticket) {
            const unsigned int nblk = gridDim.x * gridDim.y * gridDim.z;
            if (mg_last_block(fin.ticket, nblk)) {
                const double2 t = mg_block_total2(partial, partial2, (int)nblk);
                if (threadIdx.x == 0 && threadIdx.y == 0) fcg_set_beta(t.x, t.y, fin.vol, fin.sc, fin.k);
            }
        }
    }
}

// First half-sweep of a level whose solution is zero: (1-omega)*0 + omega*(0-b)*idiag
// depends on the cell's own b alone, so the kernel that produces b writes it.
template <typename T>
__device__ __forceinline__ T mg_jacobi_from_zero(T b, T omega, T idg) {
    (void)omega;   // idg = omega/diag
    return (T(0) - b) * idg;
}

// residual of the fine level restricted to the coarse right-hand side,
// bc = Rcoef*(sum of the 8 children) with Rcoef = 1/2 (basicoperators.f90:32-60,
// operators.f90:172-213). The coarse solution is zero at this point (operators.f90:209),
// so the first half-sweep of the coarse smoothing is written here, into yc.
template <typename T, bool BAT = false, int RZC = MG_RZC>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_restrict(const MgGeom gf, const T* __restrict__ xf,
                                                              const T* __restrict__ bf, const MgGeom gc,
                                                              T* __restrict__ bc, T* __restrict__ yc, T omega,
                                                              const Bat bat = Bat()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        xf = bshift(xf, dlt);
        bf = bshift(bf, dlt);
        bc = bshift(bc, dlt);
        yc = bshift(yc, dlt);
    }
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    if (x >= gc.n[2] || y >= gc.n[1]) return;
    const int nzc = gc.n[0], z0 = bz * RZC;
    auto emit = [&](int z, T s) {
        const long long c = mg_at(gc, z, y, x);
        const T bv = T(0.5) * s;
        bc[c] = bv;
        yc[c] = mg_jacobi_from_zero(bv, omega, mg_idiag<T>(gc, mg_diag(gc, z, y, x)));
    };
    if (z0 + RZC > nzc) {   // last, partial chunk
        for (int z = z0; z < nzc; ++z) emit(z, mg_restrict_cell(gf, xf, bf, z, y, x));
        return;
    }
    // Full chunk, unrolled: the 2 x 2 children of each fine plane 2*z0-1 .. 2*(z0+RZC)
    // and their x/y neighbours are loaded up front; residuals of the children in
    // mgfor's neighbour order, summed in the order (k,j,i), (k,j,i+1), (k,j+1,i),
    // (k,j+1,i+1), then the same at k+1.
    const long long sy = gf.n[2], sz = (long long)gf.n[1] * gf.n[2];
    const int i0 = 2 * x, j0 = 2 * y, k0 = 2 * z0;
    const MgNb xl = mg_nb(i0, gf.n[2], gf.per[2], 1), xh = mg_nb(i0 + 1, gf.n[2], gf.per[2], 1);
    const MgNb yl = mg_nb(j0, gf.n[1], gf.per[1], sy), yh = mg_nb(j0 + 1, gf.n[1], gf.per[1], sy);
    const MgNb zl = mg_nb(k0, gf.n[0], gf.per[0], sz), zh = mg_nb(k0 + 2 * RZC - 1, gf.n[0], gf.per[0], sz);
    // wet x/y neighbours of the children (j0,i0), (j0,i1), (j1,i0), (j1,i1)
    const int dxy[4] = {(int)xl.wm + 1 + (int)yl.wm + 1, 1 + (int)xh.wp + (int)yl.wm + 1,
                        (int)xl.wm + 1 + 1 + (int)yh.wp, 1 + (int)xh.wp + 1 + (int)yh.wp};
    const long long cb = mg_at(gf, k0, j0, i0);
    constexpr int NP = 2 * RZC + 2;   // fine planes k0-1 .. k0+2*RZC
    T v[NP][4];
    auto ld4 = [&](long long c, bool wet, T* o) {
        o[0] = mg_ldw(xf, c, wet);
        o[1] = mg_ldw(xf, c + 1, wet);
        o[2] = mg_ldw(xf, c + sy, wet);
        o[3] = mg_ldw(xf, c + sy + 1, wet);
    };
    ld4(cb + zl.om, zl.wm, v[0]);
#pragma unroll
    for (int q = 1; q < NP - 1; ++q) ld4(cb + (q - 1) * sz, true, v[q]);
    ld4(cb + (2 * RZC - 1) * sz + zh.op, zh.wp, v[NP - 1]);
    // The 8 residuals b + diag*x - sum(x_nb) summed at once: each child's 6 neighbours
    // are 3 siblings and 3 cells outside the 2 x 2 x 2 block, so the sum is
    // sum(b) + sum(w_c x_c) - sum(24 outside cells) with w_c = diag_c - 3, the child's wet
    // outside neighbours (dry ones are read as 0). Same value as the per-child sums up
    // to rounding, with 2/3 of their FP64 instructions.
    const T wxy[4] = {T(dxy[0] - 2), T(dxy[1] - 2), T(dxy[2] - 2), T(dxy[3] - 2)};
#pragma unroll
    for (int zc = 0; zc < RZC; ++zc) {
        T sb = T(0), sx = T(0), so = T(0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = 2 * zc + 1 + h;   // plane index in v
            const long long c = cb + (q - 1) * sz;
            // the plane's z-neighbour outside the block: below for the lower plane, above
            // for the upper one (dry at a closed wall)
            const bool wz = (h == 0) ? (q == 1 ? zl.wm : true) : (q == NP - 2 ? zh.wp : true);
            const T* zo = v[h == 0 ? q - 1 : q + 1];
            // x/y ring of the plane
            const T xm0 = mg_ldw(xf, c + xl.om, xl.wm), xm1 = mg_ldw(xf, c + sy + xl.om, xl.wm);
            const T xp0 = mg_ldw(xf, c + 1 + xh.op, xh.wp), xp1 = mg_ldw(xf, c + sy + 1 + xh.op, xh.wp);
            const T ym0 = mg_ldw(xf, c + yl.om, yl.wm), ym1 = mg_ldw(xf, c + 1 + yl.om, yl.wm);
            const T yp0 = mg_ldw(xf, c + sy + yh.op, yh.wp), yp1 = mg_ldw(xf, c + sy + 1 + yh.op, yh.wp);
            const T* p = v[q];
            sb = sb + ((bf[c] + bf[c + 1]) + (bf[c + sy] + bf[c + sy + 1]));
            const T pp = (p[0] + p[1]) + (p[2] + p[3]);
            sx = sx + (wxy[0] * p[0] + wxy[1] * p[1] + wxy[2] * p[2] + wxy[3] * p[3]);
            sx = wz ? sx + pp : sx;
            so = so + ((((xm0 + xm1) + (xp0 + xp1)) + ((ym0 + ym1) + (yp0 + yp1))) + ((zo[0] + zo[1]) + (zo[2] + zo[3])));
        }
        emit(z0 + zc, (sb + sx) - so);
    }
}

// trilinear 9-3-3-1 prolongation added to the fine solution (basicoperators.f90:173-231)
template <typename T, bool BAT = false>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_prolong(const MgGeom gf, T* __restrict__ xf, const MgGeom gc,
                                                             const T* __restrict__ xc, const Bat bat = Bat()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        xf = bshift(xf, dlt);
        xc = bshift(xc, dlt);
    }
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    if (x >= gf.n[2] || y >= gf.n[1]) return;
    const int nzf = gf.n[0], z0 = bz * MG_ZC;   // z0 even
    if (z0 + MG_ZC > nzf) {   // last, partial chunk
        for (int z = z0; z < nzf; ++z) {
            const long long c = mg_at(gf, z, y, x);
            xf[c] = xf[c] + mg_prolong_cell(gf, gc, xc, z, y, x);
        }
        return;
    }
    // Full chunk, unrolled: the in-plane 9-3-3-1 sums of the coarse planes z0/2-1 ..
    // z0/2+MG_ZC/2 (each used by two fine planes) are formed once; a coarse neighbour
    // outside the level is the periodic image or 0.
    const int ic = x >> 1, jc = y >> 1;
    const long long csy = gc.n[2], csz = (long long)gc.n[1] * gc.n[2];
    const MgNb cx = mg_nb(ic, gc.n[2], gc.per[2], 1), cy = mg_nb(jc, gc.n[1], gc.per[1], csy);
    const long long ox = (x & 1) ? cx.op : cx.om, oy = (y & 1) ? cy.op : cy.om;
    const bool wx = (x & 1) ? cx.wp : cx.wm, wy = (y & 1) ? cy.wp : cy.wm;
    const int kc0 = z0 >> 1;
    const MgNb zl = mg_nb(kc0, gc.n[0], gc.per[0], csz), zh = mg_nb(kc0 + MG_ZC / 2 - 1, gc.n[0], gc.per[0], csz);
    const long long cc = mg_at(gc, kc0, jc, ic);
    auto plane = [&](long long c, bool wet) -> T {
        const T a = mg_ldw(xc, c, wet), b = mg_ldw(xc, c + ox, wet && wx);
        const T d = mg_ldw(xc, c + oy, wet && wy), e = mg_ldw(xc, c + ox + oy, wet && wx && wy);
        return ((T(9) * a + T(3) * b) + T(3) * d) + e;
    };
    const long long c0 = mg_at(gf, z0, y, x), sz = (long long)gf.n[1] * gf.n[2];
    T xv[MG_ZC];   // the fine values, loaded together with the coarse ones
#pragma unroll
    for (int k = 0; k < MG_ZC; ++k) xv[k] = xf[c0 + k * sz];
    constexpr int NP = MG_ZC / 2 + 2;
    T P[NP];
    P[0] = plane(cc + zl.om, zl.wm);
#pragma unroll
    for (int q = 1; q < NP - 1; ++q) P[q] = plane(cc + (q - 1) * csz, true);
    P[NP - 1] = plane(cc + (MG_ZC / 2 - 1) * csz + zh.op, zh.wp);
    const int bxy = (int)wx | ((int)wy << 1);
    const T pc_wet = mg_pcoef<T>(gf, bxy | 4), pc_lo = mg_pcoef<T>(gf, bxy | ((int)zl.wm << 2));
    const T pc_hi = mg_pcoef<T>(gf, bxy | ((int)zh.wp << 2));
#pragma unroll
    for (int k = 0; k < MG_ZC; ++k) {
        const int m = (k >> 1) + 1;                  // plane of z>>1 in P
        const T bpl = P[m], opl = P[(k & 1) ? m + 1 : m - 1];
        const T pc = (k == 0) ? pc_lo : (k == MG_ZC - 1 ? pc_hi : pc_wet);
        xf[c0 + k * sz] = xv[k] + pc * (T(3) * bpl + opl);
    }
}

// The FP64 prolongation, one coarse column per thread: the 8 fine cells of a coarse cell share
// the x interpolations of its three coarse rows and the y interpolations of each plane, 26
// FP64 instructions for 8 cells where the per-fine-column form (k_mg_prolong) takes 40: 215 ->
// 127 us into 256^3, 28 -> 21 us into 128^3, FP64-bound. CZ coarse planes per thread, and two that it shares
// with its neighbours: 8 where the blocks still fill the chip (a 256^3 step 86.8 ms with 4, 86.3 with 8, 86.9 with 16,
// 87.6 with 2). Fine extents are twice the coarse ones (every FP64 level: only the coarsest may have odd extents).
template <int CZ>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_prolong_f64(const MgGeom gf, double* __restrict__ xf,
                                                                 const MgGeom gc, const double* __restrict__ xc) {
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    if (x >= gc.n[2] || y >= gc.n[1]) return;
    const int nzc = gc.n[0], k0 = blockIdx.z * CZ, k1 = min(k0 + CZ, nzc);
    const long long csy = gc.n[2], csz = (long long)gc.n[1] * gc.n[2];
    const MgNb cx = mg_nb(x, gc.n[2], gc.per[2], 1), cy = mg_nb(y, gc.n[1], gc.per[1], csy);
    const double* __restrict__ col = xc + mg_at(gc, 0, y, x);
    struct Plane { double v[2][2]; };   // [y low/high][x low/high]
    auto plane = [&](int k) -> Plane {
        bool wet = true;
        if (k < 0 || k >= nzc) {
            wet = gc.per[0] != 0;
            k = k < 0 ? nzc - 1 : 0;
        }
        const double* p = col + (long long)k * csz;
        double lo[3], hi[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const long long o = j == 0 ? cy.om : (j == 1 ? 0 : cy.op);
            const bool w = wet && (j == 0 ? cy.wm : (j == 1 ? true : cy.wp));
            const double a = mg_ldw(p, o, w), l = mg_ldw(p, o + cx.om, w && cx.wm), r = mg_ldw(p, o + cx.op, w && cx.wp);
            lo[j] = fma(3.0, a, l);
            hi[j] = fma(3.0, a, r);
        }
        Plane q;
        q.v[0][0] = fma(3.0, lo[1], lo[0]);
        q.v[0][1] = fma(3.0, hi[1], hi[0]);
        q.v[1][0] = fma(3.0, lo[1], lo[2]);
        q.v[1][1] = fma(3.0, hi[1], hi[2]);
        return q;
    };
    const long long fsy = gf.n[2], fsz = (long long)gf.n[1] * gf.n[2];
    double* __restrict__ f0 = xf + mg_at(gf, 0, 2 * y, 2 * x);
    Plane m = plane(k0 - 1), c = plane(k0);
#pragma unroll
    for (int kk = 0; kk < CZ; ++kk) {
        const int k = k0 + kk;
        if (k >= k1) break;
        double2 old[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                old[h][j] = *reinterpret_cast<const double2*>(f0 + (2 * k + h) * fsz + j * fsy);
        const Plane p = plane(k + 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int wz = (h == 0 ? k > 0 : k < nzc - 1) || gc.per[0] ? 4 : 0;
            const Plane& o = h == 0 ? m : p;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int wy = (j == 0 ? cy.wm : cy.wp) ? 2 : 0;
                double2 r = old[h][j];
                r.x = fma(gf.pcoef[(int)cx.wm | wy | wz], fma(3.0, c.v[j][0], o.v[j][0]), r.x);
                r.y = fma(gf.pcoef[(int)cx.wp | wy | wz], fma(3.0, c.v[j][1], o.v[j][1]), r.y);
                *reinterpret_cast<double2*>(f0 + (2 * k + h) * fsz + j * fsy) = r;
            }
        }
        m = c;
        c = p;
    }
}

// Vector forms of the two transfers (FP32): a thread owns 4 consecutive fine x cells,
// i.e. 2 coarse x cells, so that fine rows move as 16-byte and coarse pairs as 8-byte
// accesses; x neighbours come from the adjacent lanes (loaded at the warp's ends and at
// the level's x faces). Idle lanes shadow the last vector of their row so that every
// lane takes part in the shuffles; only active lanes store. Both need the fine level
// twice the coarse one in every direction and fine nx divisible by 4, and keep the
// per-cell arithmetic of the full-chunk paths above.

// k_mg_restrict: one coarse row pair of cells per thread, RZC coarse planes (needs
// coarse nz divisible by RZC); block (bx, by, bz) of the grid grid_v4_restrict(fine, coarse, RZC)
template <int RZC>
__device__ __forceinline__ void mg_restrict_v4_blk(const MgGeom& gf, const float* __restrict__ xf,
                                                   const float* __restrict__ bf, const MgGeom& gc,
                                                   float* __restrict__ bc, float* __restrict__ yc, float omega, int bx,
                                                   int by, int bz) {
    const int nx = gf.n[2], ny = gf.n[1], nz = gf.n[0];
    const int nx4 = nx >> 2;
    const int lane = threadIdx.x;
    const int xv = bx * MG_BX + lane;
    const int jc = by * MG_BY + threadIdx.y;   // coarse row
    const bool act = xv < nx4 && jc < gc.n[1];
    const int x0 = min(xv, nx4 - 1) * 4, j0 = 2 * min(jc, gc.n[1] - 1);
    const long long sy = nx, sz = (long long)ny * nx;
    const MgNb yl = mg_nb(j0, ny, gf.per[1], sy), yh = mg_nb(j0 + 1, ny, gf.per[1], sy);
    const bool wl = x0 > 0 || gf.per[2], wr = x0 + 4 < nx || gf.per[2];
    const long long ol = x0 > 0 ? -1 : (gf.per[2] ? (long long)(nx - 1) : 0);
    const long long orr = x0 + 4 < nx ? 4 : (gf.per[2] ? (long long)(4 - nx) : 0);
    const bool ownl = lane == 0 || x0 == 0, ownr = lane == MG_BX - 1 || x0 + 4 >= nx;
    // w_c = wet outside x/y neighbours of each child (j0,i), (j0,i+1), (j0+1,i), (j0+1,i+1)
    // of the coarse cells m = 0 (fine x0, x0+1) and m = 1 (x0+2, x0+3)
    const int ylw = (int)yl.wm, yhw = (int)yh.wp;
    const float wxy[2][4] = {{(float)((int)wl + ylw), (float)(1 + ylw), (float)((int)wl + yhw), (float)(1 + yhw)},
                             {(float)(1 + ylw), (float)((int)wr + ylw), (float)(1 + yhw), (float)((int)wr + yhw)}};
    const int zcb = bz * RZC, k0 = 2 * zcb;
    const long long c00 = (long long)j0 * sy + x0;
    auto ld4 = [&](const float* a, long long c) { return *reinterpret_cast<const float4*>(a + c); };
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    struct Rows { float4 r0, r1; };
    // rows j0 and j0 + 1 of fine plane k, one plane outside the level at most: periodic
    // image, or 0 across a closed wall
    auto plane = [&](int k) -> Rows {
        Rows R;
        if ((k < 0 || k >= nz) && !gf.per[0]) {
            R.r0 = zero4;
            R.r1 = zero4;
            return R;
        }
        const int kk = k < 0 ? k + nz : (k >= nz ? k - nz : k);
        const long long c = c00 + (long long)kk * sz;
        R.r0 = ld4(xf, c);
        R.r1 = ld4(xf, c + sy);
        return R;
    };
    Rows below = plane(k0 - 1), cur = plane(k0);
#pragma unroll
    for (int zc = 0; zc < RZC; ++zc) {
        const int kz = k0 + 2 * zc;
        const Rows up = plane(kz + 1), nxt = plane(kz + 2);
        float sbv[2] = {0.f, 0.f}, sxv[2] = {0.f, 0.f}, sov[2] = {0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int kf = kz + h;
            const Rows& P = h == 0 ? cur : up;
            const Rows& O = h == 0 ? below : nxt;   // the plane's z-neighbour outside the block
            const bool wz = h == 0 ? (kf > 0 || gf.per[0]) : (kf < nz - 1 || gf.per[0]);
            const long long c = c00 + (long long)kf * sz;
            const float4 ym = yl.wm ? ld4(xf, c + yl.om) : zero4;
            const float4 yp = yh.wp ? ld4(xf, c + sy + yh.op) : zero4;
            const float4 b0 = ld4(bf, c), b1 = ld4(bf, c + sy);
            const float sl0 = __shfl_up_sync(0xffffffffu, P.r0.w, 1), sl1 = __shfl_up_sync(0xffffffffu, P.r1.w, 1);
            const float sr0 = __shfl_down_sync(0xffffffffu, P.r0.x, 1), sr1 = __shfl_down_sync(0xffffffffu, P.r1.x, 1);
            const float l0 = ownl ? mg_ldw_f(xf, c + ol, wl) : sl0, l1 = ownl ? mg_ldw_f(xf, c + sy + ol, wl) : sl1;
            const float r0 = ownr ? mg_ldw_f(xf, c + orr, wr) : sr0, r1 = ownr ? mg_ldw_f(xf, c + sy + orr, wr) : sr1;
            const float x0v[4] = {P.r0.x, P.r0.y, P.r0.z, P.r0.w}, x1v[4] = {P.r1.x, P.r1.y, P.r1.z, P.r1.w};
            const float o0[4] = {O.r0.x, O.r0.y, O.r0.z, O.r0.w}, o1[4] = {O.r1.x, O.r1.y, O.r1.z, O.r1.w};
            const float ymv[4] = {ym.x, ym.y, ym.z, ym.w}, ypv[4] = {yp.x, yp.y, yp.z, yp.w};
            const float b0v[4] = {b0.x, b0.y, b0.z, b0.w}, b1v[4] = {b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int i = 2 * m;
                const float p[4] = {x0v[i], x0v[i + 1], x1v[i], x1v[i + 1]};
                const float xm0 = m == 0 ? l0 : x0v[1], xm1 = m == 0 ? l1 : x1v[1];
                const float xp0 = m == 0 ? x0v[2] : r0, xp1 = m == 0 ? x1v[2] : r1;
                sbv[m] = sbv[m] + ((b0v[i] + b0v[i + 1]) + (b1v[i] + b1v[i + 1]));
                const float pp = (p[0] + p[1]) + (p[2] + p[3]);
                sxv[m] = sxv[m] + (wxy[m][0] * p[0] + wxy[m][1] * p[1] + wxy[m][2] * p[2] + wxy[m][3] * p[3]);
                sxv[m] = wz ? sxv[m] + pp : sxv[m];
                sov[m] = sov[m] + ((((xm0 + xm1) + (xp0 + xp1)) + ((ymv[i] + ymv[i + 1]) + (ypv[i] + ypv[i + 1]))) +
                                   ((o0[i] + o0[i + 1]) + (o1[i] + o1[i + 1])));
            }
        }
        if (act) {
            const int z = zcb + zc, xc0 = x0 >> 1;
            const long long cc = mg_at(gc, z, jc, xc0);
            float bv[2], yv[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                bv[m] = 0.5f * ((sbv[m] + sxv[m]) - sov[m]);
                yv[m] = mg_jacobi_from_zero(bv[m], omega, mg_idiag<float>(gc, mg_diag(gc, z, jc, xc0 + m)));
            }
            *reinterpret_cast<float2*>(bc + cc) = make_float2(bv[0], bv[1]);
            *reinterpret_cast<float2*>(yc + cc) = make_float2(yv[0], yv[1]);
        }
        below = up;
        cur = nxt;
    }
}

template <bool BAT = false, int RZC = MG_RZC>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_restrict_v4(const MgGeom gf, const float* __restrict__ xf,
                                                                 const float* __restrict__ bf, const MgGeom gc,
                                                                 float* __restrict__ bc, float* __restrict__ yc,
                                                                 float omega, const Bat bat = Bat()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        xf = bshift(xf, dlt);
        bf = bshift(bf, dlt);
        bc = bshift(bc, dlt);
        yc = bshift(yc, dlt);
    }
    mg_restrict_v4_blk<RZC>(gf, xf, bf, gc, bc, yc, omega, blockIdx.x, blockIdx.y, bz);
}

// k_mg_prolong: one 4-cell fine row segment per thread, ZC fine planes (needs fine nz
// divisible by ZC, ZC even); block (bx, by, bz) of the grid grid_v4(fine n, ZC)
template <int ZC>
__device__ __forceinline__ void mg_prolong_v4_blk(const MgGeom& gf, float* __restrict__ xf, const MgGeom& gc,
                                                  const float* __restrict__ xc, int bx, int by, int bz) {
    const int nx = gf.n[2], ny = gf.n[1];
    const int nx4 = nx >> 2;
    const int lane = threadIdx.x;
    const int xv = bx * MG_BX + lane;
    const int y = by * MG_BY + threadIdx.y;
    const bool act = xv < nx4 && y < ny;
    const int x0 = min(xv, nx4 - 1) * 4, ys = min(y, ny - 1);
    const int ncx = gc.n[2], ic0 = x0 >> 1, jc = ys >> 1;
    const long long csy = ncx, csz = (long long)gc.n[1] * ncx;
    const MgNb cy = mg_nb(jc, gc.n[1], gc.per[1], csy);
    const long long oy = (ys & 1) ? cy.op : cy.om;
    const bool wy = (ys & 1) ? cy.wp : cy.wm;
    // coarse x neighbours of the pair ic0, ic0 + 1: ic0 - 1 (fine x0) and ic0 + 2 (x0 + 3)
    const bool cwl = ic0 > 0 || gc.per[2], cwr = ic0 + 2 < ncx || gc.per[2];
    const long long col = ic0 > 0 ? -1 : (gc.per[2] ? (long long)(ncx - 1) : 0);
    const long long cor = ic0 + 2 < ncx ? 2 : (gc.per[2] ? (long long)(2 - ncx) : 0);
    const bool ownl = lane == 0 || x0 == 0, ownr = lane == MG_BX - 1 || x0 + 4 >= nx;
    const int zb = bz * ZC, kc0 = zb >> 1;
    const MgNb zl = mg_nb(kc0, gc.n[0], gc.per[0], csz), zh = mg_nb(kc0 + ZC / 2 - 1, gc.n[0], gc.per[0], csz);
    const long long cc = mg_at(gc, kc0, jc, ic0);
    // in-plane 9-3-3-1 sums of the 4 fine cells from one coarse plane at c (0 when the
    // plane is dry): fine x0 + e takes coarse ic0 + (e >> 1) and its x neighbour on the
    // side of the fine cell
    auto plane = [&](long long c, bool wet, float* out) {
        const float2 a = wet ? *reinterpret_cast<const float2*>(xc + c) : make_float2(0.f, 0.f);
        const float2 d = (wet && wy) ? *reinterpret_cast<const float2*>(xc + c + oy) : make_float2(0.f, 0.f);
        const float sal = __shfl_up_sync(0xffffffffu, a.y, 1), sar = __shfl_down_sync(0xffffffffu, a.x, 1);
        const float sdl = __shfl_up_sync(0xffffffffu, d.y, 1), sdr = __shfl_down_sync(0xffffffffu, d.x, 1);
        const float al = ownl ? mg_ldw_f(xc, c + col, wet && cwl) : sal;
        const float ar = ownr ? mg_ldw_f(xc, c + cor, wet && cwr) : sar;
        const float dl = ownl ? mg_ldw_f(xc, c + oy + col, wet && cwl && wy) : sdl;
        const float dr = ownr ? mg_ldw_f(xc, c + oy + cor, wet && cwr && wy) : sdr;
        const float av[4] = {a.x, a.x, a.y, a.y}, bv[4] = {al, a.y, a.x, ar};
        const float dv[4] = {d.x, d.x, d.y, d.y}, ev[4] = {dl, d.y, d.x, dr};
#pragma unroll
        for (int e = 0; e < 4; ++e) out[e] = ((9.f * av[e] + 3.f * bv[e]) + 3.f * dv[e]) + ev[e];
    };
    const long long sz = (long long)ny * nx, c0 = (long long)zb * sz + (long long)ys * nx + x0;
    float4 xv4[ZC];   // the fine values, loaded together with the coarse ones
#pragma unroll
    for (int k = 0; k < ZC; ++k) xv4[k] = *reinterpret_cast<const float4*>(xf + c0 + k * sz);
    constexpr int NP = ZC / 2 + 2;
    float P[NP][4];
    plane(cc + zl.om, zl.wm, P[0]);
#pragma unroll
    for (int q = 1; q < NP - 1; ++q) plane(cc + (q - 1) * csz, true, P[q]);
    plane(cc + (ZC / 2 - 1) * csz + zh.op, zh.wp, P[NP - 1]);
    // 1/(Wx*Wy*Wz) of each fine cell: its coarse x neighbour is wet except beyond the
    // level's x faces (cells x0 and x0 + 3)
    float pc_wet[4], pc_lo[4], pc_hi[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const bool wx = e == 0 ? cwl : (e == 3 ? cwr : true);
        const int bxy = (int)wx | ((int)wy << 1);
        pc_wet[e] = mg_pcoef<float>(gf, bxy | 4);
        pc_lo[e] = mg_pcoef<float>(gf, bxy | ((int)zl.wm << 2));
        pc_hi[e] = mg_pcoef<float>(gf, bxy | ((int)zh.wp << 2));
    }
#pragma unroll
    for (int k = 0; k < ZC; ++k) {
        const int m = (k >> 1) + 1;   // plane of z >> 1 in P
        const float* bpl = P[m];
        const float* opl = P[(k & 1) ? m + 1 : m - 1];
        const float xo[4] = {xv4[k].x, xv4[k].y, xv4[k].z, xv4[k].w};
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float pc = (k == 0) ? pc_lo[e] : (k == ZC - 1 ? pc_hi[e] : pc_wet[e]);
            v[e] = xo[e] + pc * (3.f * bpl[e] + opl[e]);
        }
        if (act) *reinterpret_cast<float4*>(xf + c0 + k * sz) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

template <bool BAT = false, int ZC = V4_ZC>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_prolong_v4(const MgGeom gf, float* __restrict__ xf,
                                                                const MgGeom gc, const float* __restrict__ xc,
                                                                const Bat bat = Bat()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        xf = bshift(xf, dlt);
        xc = bshift(xc, dlt);
    }
    mg_prolong_v4_blk<ZC>(gf, xf, gc, xc, blockIdx.x, blockIdx.y, bz);
}

// ---------------------------------------------------------------- coarse levels in one cluster
// Levels l0..L-1 of a V-cycle (solvers.f90:35-55 from level l0 down and back up) run in
// one cluster of BT_CTAS thread blocks: the level arrays live in shared memory, and each
// half-sweep, restriction and prolongation is one pass followed by a barrier, instead of
// one grid launch each. Input: b of level l0 (its x is zero after the restriction that
// produced b); output: x of level l0. The per-cell arithmetic is that of the grid kernels.
// The larger of these levels are cut into slabs of z planes, one per block (MgBottomLevel::pp
// planes, an even number, so that a coarse plane's children are one block's); a pass
// writes the planes its neighbours need into their shared memory, and the cluster's barrier
// ends it. The smallest levels, where a pass is one round of loads, live in block 0, whose own
// barrier ends a pass while the others wait. Every array carries a ring of ghost cells (0 across
// walls; a pass writes a cell's periodic images with the cell), so that neighbours lie at
// offsets common to all threads, and a thread's column comes from two multiplications by
// precomputed reciprocals.
// Bound by the instructions and barriers of a pass (1.4 us each; a cluster barrier alone is 0.37 us with
// 512 threads); FP64: by the FP64 pipes of its SMs. Measured against the same levels in one block: 24^3 and
// below 53 -> 28 us per V-cycle in FP32; with the larger levels now included, a 48^3 mixed step 1464 ->
// 1224 us, ten steps of eight 64^3 runs 19.0 -> 18.4 ms, a 64 x 32 x 32 FP64 step 1521 -> 1431 us.
constexpr int MG_BOTTOM_MAXLEV = 12;
constexpr size_t MG_BOTTOM_SMEM = 200 * 1024;
// Threads of a block: 768 where that saves the first level a round of tasks (24 x 24 columns: 576 tasks in one
// round instead of two, a 48^3 mixed step 828 -> 807 us, eight batched ones 16.47 -> 16.27 ms), else 512 with
// registers for two blocks per SM: sixteen clusters of a batch do not fit side by side otherwise (sixteen 32^3
// runs 14.4 -> 16.4 ms). 1024 threads: 843 us, and 1 to 4% slower elsewhere.
constexpr int BT_CTAS = 8, BT_THREADS = 512, BT_MAXTHREADS = 768;

struct MgBottomLevel {
    int n[3];                // z, y, x
    int pp, nblk;            // z planes per block, blocks that hold planes (1: block 0 alone)
    int sy, sz, vol;         // of the padded arrays (pp + 2 planes)
    int off;                 // elements: x, then y, then b
    int zg, ng;              // cells of a column per task, tasks per column
    unsigned int mx, mcol;   // ceil(2^32 / n[2]), ceil(2^32 / (n[1] n[2]))
    int bychild;             // FP32: roundings of the smallest levels (see bottom_plan)
};
template <typename T>
struct MgBottom {
    int nlev;                // levels held, none of them empty
    int resmooth;            // the last one lies above an empty level: it is smoothed on the way up too
    int per[3];
    T idiag[8], pcoef[8];    // MgGeom's tables
    MgBottomLevel lev[MG_BOTTOM_MAXLEV];
    T* xg;                   // x of level l0 (global)
    const T* bg;             // b of level l0 (global)
};

// quotient by the n of m = ceil(2^32 / n), exact for t, n < 2^16 (n = 1: m wraps to 0)
__device__ __forceinline__ int bottom_div(int t, unsigned int m) { return m ? (int)__umulhi((unsigned int)t, m) : t; }

// a column segment of the block's slab: cells z0 <= z < z1 of the level, p = index of the first
// one in the padded arrays
struct BottomTask {
    int x, y, z0, z1, p;
};
__device__ __forceinline__ BottomTask bottom_task(const MgBottomLevel& l, int zb, int t) {
    BottomTask k;
    const int ncol = l.n[1] * l.n[2], g = bottom_div(t, l.mcol), col = t - g * ncol;
    k.y = bottom_div(col, l.mx);
    k.x = col - k.y * l.n[2];
    k.z0 = zb + g * l.zg;
    k.z1 = min(k.z0 + l.zg, min(zb + l.pp, l.n[0]));
    k.p = (k.z0 - zb + 1) * l.sz + (k.y + 1) * l.sy + k.x + 1;
    return k;
}

// A block's slab of a level
template <typename T>
struct BottomSlab {
    int zb, ze;              // planes held
    int zlo, zhi;            // the planes with an image in the slab below, above (-1: none)
    T *lo, *hi;              // shared memory there, shifted so that an element's index is its image's
};

// Offsets of a column's images across the x and y faces of a periodic level (0: none; both when n = 1)
struct BottomRing {
    int xl, xh, yl, yh;
    bool any;
};
__device__ __forceinline__ BottomRing bottom_ring(const MgBottomLevel& l, const int* per, int y, int x) {
    BottomRing r;
    r.xl = per[2] && x == 0 ? l.n[2] : 0;
    r.xh = per[2] && x == l.n[2] - 1 ? -l.n[2] : 0;
    r.yl = per[1] && y == 0 ? l.n[1] * l.sy : 0;
    r.yh = per[1] && y == l.n[1] - 1 ? -l.n[1] * l.sy : 0;
    r.any = (r.xl | r.xh | r.yl | r.yh) != 0;
    return r;
}
template <bool EDGES, typename T>
__device__ __forceinline__ void bottom_ring_put(const BottomRing& r, T* q, T v) {
    if (r.xl) q[r.xl] = v;
    if (r.xh) q[r.xh] = v;
    if (r.yl) q[r.yl] = v;
    if (r.yh) q[r.yh] = v;
    if (EDGES) {
        if (r.xl && r.yl) q[r.xl + r.yl] = v;
        if (r.xl && r.yh) q[r.xl + r.yh] = v;
        if (r.xh && r.yl) q[r.xh + r.yl] = v;
        if (r.xh && r.yh) q[r.xh + r.yh] = v;
    }
}
// element p of the array at offset o (of shared memory base `s`) = v, a cell of plane z, with its images: in
// the level's ghost columns, and of the slab's first and last plane in the neighbouring slabs. EDGES: images
// across edges and corners too (before a prolongation reads the diagonal neighbours).
template <bool EDGES, typename T>
__device__ __forceinline__ void bottom_put(const BottomSlab<T>& sl, const BottomRing& r, T* s, int o, int p, int z, T v) {
    s[o + p] = v;
    if (z == sl.zlo) sl.lo[o + p] = v;
    if (z == sl.zhi) sl.hi[o + p] = v;
    if (r.any) {
        bottom_ring_put<EDGES>(r, s + o + p, v);
        if (EDGES && z == sl.zlo) bottom_ring_put<true>(r, sl.lo + o + p, v);
        if (EDGES && z == sl.zhi) bottom_ring_put<true>(r, sl.hi + o + p, v);
    }
}
// damped inverse diagonals of a column: inside, and at the first and last plane of a closed level
template <typename T>
struct BottomDiag {
    T in, end;
    int z1;                  // last plane with a closed end (-1: periodic)
    __device__ __forceinline__ T at(int z) const { return (z == 0 || z == z1) && z1 >= 0 ? end : in; }
};

// wet x and y neighbours of a column, wet z neighbours of a cell
__device__ __forceinline__ int bottom_wet_xy(const MgBottomLevel& l, const int* per, int y, int x) {
    return (per[2] ? 2 : (x > 0) + (x < l.n[2] - 1)) + (per[1] ? 2 : (y > 0) + (y < l.n[1] - 1));
}
__device__ __forceinline__ int bottom_wet_z(const MgBottomLevel& l, const int* per, int z) {
    return per[0] ? 2 : (z > 0) + (z < l.n[0] - 1);
}
template <typename T>
__device__ __forceinline__ BottomDiag<T> bottom_diag(const MgBottomLevel& l, const int* per, const T* idiag, int y, int x) {
    BottomDiag<T> d;
    const int dxy = bottom_wet_xy(l, per, y, x);
    d.z1 = per[0] ? -1 : l.n[0] - 1;
    d.in = idiag[dxy + 2];
    d.end = idiag[dxy + (l.n[0] > 1 ? 1 : 0)];
    return d;
}

template <typename T, int THREADS>
__global__ void __cluster_dims__(BT_CTAS, 1, 1) __launch_bounds__(THREADS <= 512 ? THREADS : 1024, THREADS <= 512 ? 2 : 1)
    k_mg_bottom(const __grid_constant__ MgBottom<T> a, const Bat bat = Bat()) {
    extern __shared__ __align__(16) unsigned char mg_smem[];
    int bz;
    long long dlt;
    if (!batch_enter(bat, bz, dlt)) return;   // (one answer for the whole cluster)
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    // the arguments stay in parameter space (their level table is indexed at run time:
    // a copy of the struct would sit in every thread's local memory); only the two
    // global pointers are shifted to the block's run
    T* const xg = bshift(a.xg, dlt);
    const T* const bg = bshift(a.bg, dlt);
    T* const sm = reinterpret_cast<T*>(mg_smem);
    const T cff1 = T(1) - a.idiag[1];   // idiag[1] = omega
    const int L = a.nlev;
    // the block's slab of level l as seen from `who` (a block writes block 0's small levels
    // when it restricts into them); ghosts of the neighbouring slabs lie nz_prev planes up and
    // the block's own planes down from its first and last plane
    auto slab = [&](const MgBottomLevel& l, int who) {
        BottomSlab<T> s;
        s.zb = who * l.pp;
        s.ze = min(s.zb + l.pp, l.n[0]);
        s.zlo = s.zhi = -1;
        s.lo = s.hi = sm;
        if (who >= l.nblk) { s.ze = s.zb; return s; }
        const int prev = who > 0 ? who - 1 : (a.per[0] ? l.nblk - 1 : -1);
        const int next = who < l.nblk - 1 ? who + 1 : (a.per[0] ? 0 : -1);
        if (prev >= 0) {
            s.zlo = s.zb;
            s.lo = cluster.map_shared_rank(sm, prev) + min(l.pp, l.n[0] - prev * l.pp) * l.sz;
        }
        if (next >= 0) {
            s.zhi = s.ze - 1;
            s.hi = cluster.map_shared_rank(sm, next) - (s.ze - s.zb) * l.sz;
        }
        return s;
    };
    // ends a pass over level l (its writers and readers: the cluster, or block 0)
    auto sync = [&](const MgBottomLevel& l) {
        if (l.nblk > 1) cluster.sync();
        else if (rank == 0) __syncthreads();
    };
    auto ntasks = [&](const MgBottomLevel& l) { return rank < l.nblk ? l.n[1] * l.n[2] * l.ng : 0; };
    // offsets of a level's arrays
    enum { AX = 0, AY = 1, AB = 2 };
    auto arr = [&](const MgBottomLevel& l, int w) { return l.off + w * l.vol; };

    // ghosts across walls stay 0
    const MgBottomLevel& last = a.lev[L - 1];
    for (int q = threadIdx.x; q < last.off + 3 * last.vol; q += THREADS) sm[q] = T(0);
    cluster.sync();
    {   // level l0 starts from x = 0: its first half-sweep is y = from_zero(b)
        const MgBottomLevel& l = a.lev[0];
        const BottomSlab<T> sl = slab(l, rank);
        const int nplane = l.n[1] * l.n[2], nt = ntasks(l), ob = arr(l, AB), oy = arr(l, AY);
        for (int t = threadIdx.x; t < nt; t += THREADS) {
            const BottomTask k = bottom_task(l, sl.zb, t);
            const BottomRing ring = bottom_ring(l, a.per, k.y, k.x);
            const BottomDiag<T> dg = bottom_diag(l, a.per, a.idiag, k.y, k.x);
            const T* pb = bg + k.z0 * nplane + k.y * l.n[2] + k.x;
            int p = k.p;
            for (int z = k.z0; z < k.z1; ++z, pb += nplane, p += l.sz) {
                const T bv = *pb;
                sm[ob + p] = bv;
                bottom_put<false>(sl, ring, sm, oy, p, z, mg_jacobi_from_zero(bv, T(0), dg.at(z)));
            }
        }
        sync(l);
    }
    // one half-sweep from array wi to array wo
    auto sweep = [&](const MgBottomLevel& l, int wi, int wo, auto edges) {
        constexpr bool EDGES = decltype(edges)::value;
        const BottomSlab<T> sl = slab(l, rank);
        const int nt = ntasks(l), oo = arr(l, wo);
        const T* in = sm + arr(l, wi);
        const T* b = sm + arr(l, AB);
        for (int t = threadIdx.x; t < nt; t += THREADS) {
            const BottomTask k = bottom_task(l, sl.zb, t);
            const BottomRing ring = bottom_ring(l, a.per, k.y, k.x);
            const BottomDiag<T> dg = bottom_diag(l, a.per, a.idiag, k.y, k.x);
            int p = k.p;
            T zm = in[p - l.sz], zc = in[p];
            for (int z = k.z0; z < k.z1; ++z) {
                const T zp = in[p + l.sz];
                const T s = ((((in[p - 1] + in[p + 1]) + in[p - l.sy]) + in[p + l.sy]) + zm) + zp;
                bottom_put<EDGES>(sl, ring, sm, oo, p, z, fma(cff1, zc, mul_rn(s - b[p], dg.at(z))));
                zm = zc;
                zc = zp;
                p += l.sz;
            }
        }
        sync(l);
    };
    for (int i = 0; i < L - 1; ++i) {
        const MgBottomLevel &f = a.lev[i], &c = a.lev[i + 1];
        sweep(f, AY, AX, std::false_type());   // second half of the pre-smoothing
        // residuals of the 8 children; the coarse level starts from zero, so its first
        // half-sweep is written too
        const BottomSlab<T> fs = slab(f, rank);
        const int owner = c.nblk > 1 ? rank : 0;            // the block that holds the coarse cells
        const BottomSlab<T> cs = slab(c, owner);
        T* const smc = owner == rank ? sm : cluster.map_shared_rank(sm, owner);
        const T* xf = sm + arr(f, AX);
        const T* bf = sm + arr(f, AB);
        const int ob = arr(c, AB), oy = arr(c, AY);
        const int zc0 = fs.zb / 2, zc1 = (fs.ze + 1) / 2, ncol = c.n[1] * c.n[2];
        const int nt = rank < f.nblk ? ncol * (zc1 - zc0) : 0;
        for (int t = threadIdx.x; t < nt; t += THREADS) {
            const int g = bottom_div(t, c.mcol), col = t - g * ncol, z = zc0 + g;
            const int y = bottom_div(col, c.mx), x = col - y * c.n[2];
            const int x0 = 2 * x, y0 = 2 * y;
            const int wxl = a.per[2] || x0 > 0, wxh = a.per[2] || x0 + 2 < f.n[2];
            const int wyl = a.per[1] || y0 > 0, wyh = a.per[1] || y0 + 2 < f.n[1];
            // sum(b) + sum(w x) - sum(24 outside cells), w = wet outside neighbours (k_mg_restrict), or
            // the children's residuals one by one
            T sb = T(0), sx = T(0), so = T(0), sr = T(0);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int zf = 2 * z + h;
                const int p = (zf - fs.zb + 1) * f.sz + (y0 + 1) * f.sy + x0 + 1;
                const T *q = xf + p, *qb = bf + p, *ol = q - f.sz, *oh = q + f.sz;
                const T p0 = q[0], p1 = q[1], p2 = q[f.sy], p3 = q[f.sy + 1];
                const T xm0 = q[-1], xm1 = q[f.sy - 1], xp0 = q[2], xp1 = q[f.sy + 2];
                const T ym0 = q[-f.sy], ym1 = q[1 - f.sy], yp0 = q[2 * f.sy], yp1 = q[2 * f.sy + 1];
                if (sizeof(T) == sizeof(float) && f.bychild) {
                    const int dz = bottom_wet_z(f, a.per, zf);
                    const T r00 = (qb[0] + T(wxl + wyl + 2 + dz) * p0) - (((((xm0 + p1) + ym0) + p2) + ol[0]) + oh[0]);
                    const T r01 = (qb[1] + T(wxh + wyl + 2 + dz) * p1) - (((((p0 + xp0) + ym1) + p3) + ol[1]) + oh[1]);
                    const T r10 = (qb[f.sy] + T(wxl + wyh + 2 + dz) * p2) -
                                  (((((xm1 + p3) + p0) + yp0) + ol[f.sy]) + oh[f.sy]);
                    const T r11 = (qb[f.sy + 1] + T(wxh + wyh + 2 + dz) * p3) -
                                  (((((p2 + xp1) + p1) + yp1) + ol[f.sy + 1]) + oh[f.sy + 1]);
                    sr = (h == 0) ? r00 : sr + r00;
                    sr = sr + r01;
                    sr = sr + r10;
                    sr = sr + r11;
                } else {
                    const T* o = h == 0 ? ol : oh;
                    const bool wz = a.per[0] || (h == 0 ? zf > 0 : zf < f.n[0] - 1);
                    sb = sb + ((qb[0] + qb[1]) + (qb[f.sy] + qb[f.sy + 1]));
                    sx = sx + (T(wxl + wyl) * p0 + T(wxh + wyl) * p1 + T(wxl + wyh) * p2 + T(wxh + wyh) * p3);
                    sx = wz ? sx + ((p0 + p1) + (p2 + p3)) : sx;
                    so = so + ((((xm0 + xm1) + (xp0 + xp1)) + ((ym0 + ym1) + (yp0 + yp1))) +
                               ((o[0] + o[1]) + (o[f.sy] + o[f.sy + 1])));
                }
            }
            const T bv = T(0.5) * (sizeof(T) == sizeof(float) && f.bychild ? sr : (sb + sx) - so);
            const int p = (z - cs.zb + 1) * c.sz + (y + 1) * c.sy + x + 1;
            smc[ob + p] = bv;
            const int dg = bottom_wet_xy(c, a.per, y, x) + bottom_wet_z(c, a.per, z);
            bottom_put<false>(cs, bottom_ring(c, a.per, y, x), smc, oy, p, z, mg_jacobi_from_zero(bv, T(0), a.idiag[dg]));
        }
        sync(f);
    }
    sweep(last, AY, AX, std::true_type());
    for (int i = a.resmooth ? L - 1 : L - 2; i >= 0; --i) {
        const MgBottomLevel& f = a.lev[i];
        if (i < L - 1) {
            const MgBottomLevel& c = a.lev[i + 1];
            if (f.nblk > 1 && c.nblk == 1) cluster.sync();   // block 0's x is ready
            const BottomSlab<T> fs = slab(f, rank);
            const int owner = c.nblk > 1 ? rank : 0, czb = owner * c.pp;
            const T* xc = (owner == rank ? sm : cluster.map_shared_rank(sm, owner)) + arr(c, AX);
            const int nt = ntasks(f), ox_ = arr(f, AX);
            T* xf = sm + ox_;
            for (int t = threadIdx.x; t < nt; t += THREADS) {
                const BottomTask k = bottom_task(f, fs.zb, t);
                const int ic = k.x >> 1, jc = k.y >> 1;
                const int ox = (k.x & 1) ? 1 : -1, oy = (k.y & 1) ? c.sy : -c.sy;
                const int wx = a.per[2] || ((k.x & 1) ? ic + 1 < c.n[2] : ic > 0);
                const int wy = a.per[1] || ((k.y & 1) ? jc + 1 < c.n[1] : jc > 0);
                const T* col = xc + (jc + 1) * c.sy + ic + 1;
                // in-plane sums of a coarse plane as the cell's own and as the one beyond it (alike but
                // for the roundings of the smallest FP32 levels)
                struct Plane { T own, beyond; };
                const bool unfused = sizeof(T) == sizeof(float) && f.bychild;
                auto plane = [&](int kk) -> Plane {
                    const T* q = col + (kk - czb + 1) * c.sz;
                    const T q0 = q[0], qx = q[ox], qy = q[oy], qxy = q[ox + oy];
                    const T b3 = mul_rn(T(3), qx), d3 = mul_rn(T(3), qy), t = fma(T(9), q0, b3);
                    Plane r;
                    r.own = r.beyond = fma(T(3), qy, t) + qxy;
                    if (unfused) {
                        r.own = add_rn(add_rn(t, d3), qxy);
                        r.beyond = add_rn(add_rn(add_rn(mul_rn(T(9), q0), b3), d3), qxy);
                    }
                    return r;
                };
                const BottomRing ring = bottom_ring(f, a.per, k.y, k.x);
                const T pin = a.pcoef[wx | (wy << 1) | 4], pend = a.pcoef[wx | (wy << 1) | (a.per[0] ? 4 : 0)];
                // segments start at even z: each coarse plane is formed once
                int p = k.p, kc = k.z0 >> 1;
                Plane pm = plane(kc - 1), pc = plane(kc);
                for (int z = k.z0; z < k.z1; z += 2, ++kc) {
                    const Plane pn = plane(kc + 1);
                    bottom_put<false>(fs, ring, sm, ox_, p, z,
                                      fma(kc > 0 ? pin : pend, fma(T(3), pc.own, pm.beyond), xf[p]));
                    p += f.sz;
                    bottom_put<false>(fs, ring, sm, ox_, p, z + 1,
                                      fma(kc < c.n[0] - 1 ? pin : pend, fma(T(3), pc.own, pn.beyond), xf[p]));
                    p += f.sz;
                    pm = pc;
                    pc = pn;
                }
            }
            sync(f);
        }
        sweep(f, AX, AY, std::false_type());
        sweep(f, AY, AX, std::true_type());
    }
    const MgBottomLevel& l = a.lev[0];
    const int nplane = l.n[1] * l.n[2], nt = ntasks(l), zb = rank * l.pp, ox = arr(l, AX);
    for (int t = threadIdx.x; t < nt; t += THREADS) {
        const BottomTask k = bottom_task(l, zb, t);
        for (int z = k.z0; z < k.z1; ++z)
            xg[z * nplane + k.y * l.n[2] + k.x] = sm[ox + k.p + (z - k.z0) * l.sz];
    }
    cluster.sync();   // no block leaves while another may still write its ghosts
}

// The levels of the cluster kernel from level l0 on (n: extents; none of them empty): how each is cut, the
// arrays' places; returns the elements of shared memory per block. A level of more than `solo` cells
// is cut into an even number of planes per block, and the level under it too while half of them is even.
// FP32 keeps each level's roundings, so that solutions do not depend, to the bit, on which kernel a level
// runs in: a restriction child by child and partly unfused sums in the prolongation where this level and
// those under it hold at most 200 KB of x, b and y, as the grid kernels above.
// Returns the elements; *cost: what the first level's rounds of tasks take.
static long long bottom_plan(const int (*n)[3], int nlev, long long solo, int threads, MgBottomLevel* lev,
                             long long* cost) {
    long long off = 0;
    int half = 0;   // planes per block of the next level, from the one above (0: not cut)
    for (int k = 0; k < nlev; ++k) {
        MgBottomLevel l;
        for (int i = 0; i < 3; ++i) l.n[i] = n[k][i];
        const int nz = l.n[0], ncol = l.n[1] * l.n[2];
        const bool cut = (long long)nz * ncol > solo && nz >= 4 && (k == 0 || (half && half % 2 == 0));
        l.pp = !cut ? nz : (k == 0 ? 2 * ((nz + 2 * BT_CTAS - 1) / (2 * BT_CTAS)) : half);
        l.nblk = (nz + l.pp - 1) / l.pp;
        half = l.nblk > 1 ? l.pp / 2 : 0;
        l.sy = l.n[2] + 2;
        l.sz = l.sy * (l.n[1] + 2);
        l.vol = l.sz * (l.pp + 2);
        l.off = (int)off;
        off += 3ll * l.vol;
        // columns are cut in z (in pairs of planes, which share their coarse planes) so that the block's
        // rounds of tasks take the fewest cells, a task's start counted as two
        long long best = 1ll << 60;
        for (int zg = l.pp < 2 ? 1 : 2; zg <= 8 && (zg <= l.pp || zg <= 2); zg += zg < 2 ? 1 : 2) {
            const long long rounds = ((long long)ncol * ((l.pp + zg - 1) / zg) + threads - 1) / threads;
            if (rounds * (zg + 2) < best) {
                best = rounds * (zg + 2);
                l.zg = zg;
            }
        }
        if (k == 0 && cost) *cost = best;
        l.ng = (l.pp + l.zg - 1) / l.zg;
        l.mx = (unsigned int)(((1ull << 32) + l.n[2] - 1) / l.n[2]);
        l.mcol = (unsigned int)(((1ull << 32) + ncol - 1) / ncol);
        long long under = 0;
        for (int j = k; j < nlev; ++j) under += (long long)n[j][0] * n[j][1] * n[j][2];
        l.bychild = 3 * (long long)sizeof(float) * under <= 200 * 1024;
        if (lev) lev[k] = l;
    }
    return off;
}

// ---------------------------------------------------------------- reductions
// Deterministic sums: one partial per block of the (x, y, z-chunk) grid, then one
// block adds the partials in a fixed order.

// sum v^2
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_sumsq(const MgGeom g, const double* __restrict__ v,
                                                           double* __restrict__ partial, const MgFin fin,
                                                           double* __restrict__ out) {
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    const int nz = g.n[0], z0 = blockIdx.z * MG_ZC;
    double s = 0.0;
    if (x < g.n[2] && y < g.n[1]) {
        const long long sz = (long long)g.n[1] * g.n[2];
        const long long c0 = mg_at(g, z0, y, x);
        for (int z = z0; z < min(z0 + MG_ZC, nz); ++z) {
            const double r = v[c0 + (z - z0) * sz];
            s += r * r;
        }
    }
    block_partial(s, partial, blockIdx.z);
    double t;
    if (fin.ticket && mg_fin_total(fin, partial, gridDim.x * gridDim.y * gridDim.z, t)) *out = t;
}

// Stop-test residual of the level-1 solution together with the first half-sweep of the
// next V-cycle: both need the same neighbour sum, so one pass gives sum(r^2) (block
// partials as k_mg_sumsq's) and y = (1-omega)*x + omega*(sum - b)*idiag.
// If the solve then stops, y is simply not used.
template <typename T, int ZC = MG_ZC>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_resid_sweep(const MgGeom g, const T* __restrict__ v,
                                                                 const T* __restrict__ b, T* __restrict__ y_out,
                                                                 T omega, double* __restrict__ partial,
                                                                 const MgFin fin) {
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    const int nz = g.n[0], z0 = blockIdx.z * ZC;
    (void)omega;   // the tables hold omega/diag
    double s = 0.0;
    if (x < g.n[2] && y < g.n[1]) {
        const long long sy = g.n[2], sz = (long long)g.n[1] * g.n[2];
        const long long c0 = mg_at(g, z0, y, x);
        const MgNb nx = mg_nb(x, g.n[2], g.per[2], 1), ny = mg_nb(y, g.n[1], g.per[1], sy);
        const int dxy = (int)nx.wm + (int)nx.wp + (int)ny.wm + (int)ny.wp;
        auto cell = [&](long long c, T zm, T x0, T zp, int dg) {
            const T nsum = ((((mg_ldw(v, c + nx.om, nx.wm) + mg_ldw(v, c + nx.op, nx.wp)) + mg_ldw(v, c + ny.om, ny.wm)) +
                             mg_ldw(v, c + ny.op, ny.wp)) + zm) + zp;
            const T bv = b[c];
            const T r = (bv + T(dg) * x0) - nsum;
            s += (double)r * (double)r;
            // (1-omega)x + omega(nsum - b)/diag = x - (omega/diag) r
            y_out[c] = x0 - mg_idiag<T>(g, dg) * r;
        };
        if (z0 + ZC <= nz) {
            const MgNb lo = mg_nb(z0, nz, g.per[0], sz), hi = mg_nb(z0 + ZC - 1, nz, g.per[0], sz);
            T col[ZC + 2];
            col[0] = mg_ldw(v, c0 + lo.om, lo.wm);
#pragma unroll
            for (int k = 1; k <= ZC; ++k) col[k] = v[c0 + (k - 1) * sz];
            col[ZC + 1] = mg_ldw(v, c0 + (ZC - 1) * sz + hi.op, hi.wp);
#pragma unroll
            for (int k = 0; k < ZC; ++k)
                cell(c0 + k * sz, col[k], col[k + 1], col[k + 2],
                     dxy + (k == 0 ? (int)lo.wm : 1) + (k == ZC - 1 ? (int)hi.wp : 1));
        } else {
            for (int z = z0; z < nz; ++z) {
                const long long c = c0 + (z - z0) * sz;
                const MgNb nzb = mg_nb(z, nz, g.per[0], sz);
                cell(c, mg_ldw(v, c + nzb.om, nzb.wm), v[c], mg_ldw(v, c + nzb.op, nzb.wp),
                     dxy + (int)nzb.wm + (int)nzb.wp);
            }
        }
    }
    block_partial(s, partial, blockIdx.z);
    double t;
    if (fin.ticket && mg_fin_total(fin, partial, gridDim.x * gridDim.y * gridDim.z, t)) fin.sc[SC_RR] = t;
}

// ---------------------------------------------------------------- FP64 levels on the integer pipes
// What the V-cycle does to a level is a sum over a cell and its neighbours: a half-sweep is
// (1-omega) x + (omega/diag) (sum(x_nb) - b), the stop test and the restriction need the residual
// r = b + diag*x - sum(x_nb). In doubles the sum is 6 FP64 instructions of a half-sweep's 8, at
// 2 lanes per cycle and SM; here it is a sum of 64-bit integers (nyles_fx.cuh), about 130 instructions per cell
// with the conversions and the range tests, and 2 FP64 instructions are left. Bound by the integer
// pipe (62% busy; memory 25%). Measured against the double kernels (k_mg_jacobi,
// k_mg_resid_sweep, k_mg_restrict in 8-cell columns) per launch: 128^3 38 -> 17, 44 -> 20 and
// 37 -> 17 us (20 and 23 in a Taylor-Green step, some of whose sums are redone in doubles); 256^3 half-sweep 245 -> 95 us,
// step with the transfer below 142 -> 86.1 ms.
// A block owns 32 x 8 columns of ZC cells, one column per thread: every value of the tile
// and of the ring around it is loaded first, the block agrees on the exponent, and the
// converted columns meet in shared memory. Ghosts: 0 across a wall, else the periodic image.
// Tiles that the level cuts off, and those beyond the integers' exponents, are summed in doubles. So is, by
// itself, a sum whose operands all lie more than 64 times below the tile's largest value (a thread
// looks closer only where the cells above and below a cell, its b and itself do); in MODE 2 a
// coarse cell's, where that holds for its eight children.
// MODE 0: out = x - (omega/diag) r. MODE 1: also the block's sum of r^2. MODE 2: the coarse
// right-hand side 0.5 * (sum of r over the 8 children) and its first half-sweep (k_mg_restrict);
// fine extents are twice the coarse ones.

// one cell in doubles: r, and what the kernel stores
template <int MODE>
__device__ __forceinline__ double fx_cell_double(const MgGeom& g, const double* __restrict__ v,
                                                 const double* __restrict__ b, double* __restrict__ out, int z, int y, int x) {
    const long long c = mg_at(g, z, y, x);
    const double xc = v[c], sum = mg_nsum(v, g, z, y, x);
    const int dg = mg_diag(g, z, y, x);
    const double r = fma((double)dg, xc, b[c]) - sum;
    if (MODE == 0) out[c] = fma(g.idiag[dg], sum - b[c], (1.0 - g.idiag[1]) * xc);
    else if (MODE == 1) out[c] = fma(-g.idiag[dg], r, xc);
    return r;
}
// the cells of a warp's row that `redo` names, bit k for plane zb + k of a lane's column, shared out among
// the lanes (one round trip to memory for up to 32 of them); the sum of r^2
template <int ZC, int MODE>
__device__ __noinline__ double fx_redo_double(const MgGeom& g, const double* __restrict__ v, const double* __restrict__ b,
                                              double* __restrict__ out, int xb, int y, int zb, unsigned int redo) {
    unsigned int lanes[ZC];
    int total = 0;
#pragma unroll
    for (int k = 0; k < ZC; ++k) {
        lanes[k] = __ballot_sync(0xffffffffu, redo >> k & 1u);
        total += __popc(lanes[k]);
    }
    double s = 0.0;
    for (int j = threadIdx.x; j < total; j += 32) {
        int first = 0, pos = 0, z = 0;
        unsigned int w = 0;
#pragma unroll
        for (int k = 0; k < ZC; ++k) {
            const int n = __popc(lanes[k]);
            if (j >= first && j < first + n) {
                w = lanes[k];
                pos = j - first;
                z = zb + k;
            }
            first += n;
        }
        for (; pos; --pos) w &= w - 1;
        const double r = fx_cell_double<MODE>(g, v, b, out, z, y, xb + __ffs((int)w) - 1);
        if (MODE == 1) s = fma(r, r, s);
    }
    return s;
}
__device__ __noinline__ double fx_restrict_double(const MgGeom& g, const double* __restrict__ v,
                                                  const double* __restrict__ b, int z, int y, int x) {
    return mg_restrict_cell(g, v, b, z, y, x);
}

// the thread's column in doubles (any tile); MODE 2: the sums over the pairs in z and x
// go to `sums` [ZC/2][BY][BX/2]
template <int ZC, int MODE>
__device__ __noinline__ double fx_tile_double(const MgGeom& g, const double* __restrict__ v, const double* __restrict__ b,
                                              double* __restrict__ out, int x, int y, int zb, double* sums) {
    const bool act = x < g.n[2] && y < g.n[1];
    double s = 0.0, pair = 0.0;
    for (int k = 0; k < ZC; ++k) {
        const int z = zb + k;
        double r = 0.0;
        if (act && z < g.n[0]) r = fx_cell_double<MODE>(g, v, b, out, z, y, x);
        if (MODE == 1) s = fma(r, r, s);
        if (MODE == 2) {
            pair = (k & 1) ? pair + r : r;
            if (k & 1) {
                const double w = pair + __shfl_down_sync(0xffffffffu, pair, 1);
                if ((threadIdx.x & 1) == 0) sums[((k >> 1) * MG_BY + threadIdx.y) * (MG_BX / 2) + (threadIdx.x >> 1)] = w;
            }
        }
    }
    return s;
}

template <int ZC, int MODE>
__global__ void __launch_bounds__(MG_BX * MG_BY, 3) k_mg_fx(const MgGeom g, const double* __restrict__ v,
                                                           const double* __restrict__ b, double* __restrict__ out,
                                                           double* __restrict__ partial, const MgGeom gc,
                                                           double* __restrict__ bc) {
    constexpr int BX = MG_BX, BY = MG_BY, NT = BX * BY;
    __shared__ long long tile[ZC][BY + 2][BX + 2];
    __shared__ unsigned int swarp[BY];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * BX + tx;
    const int nx = g.n[2], ny = g.n[1], nz = g.n[0];
    const int xb = blockIdx.x * BX, yb = blockIdx.y * BY, zb = blockIdx.z * ZC;
    const int x = xb + tx, y = yb + ty;
    const long long sy = nx, sz = (long long)ny * nx;
    // MODE 2, after the tile has been read: [ZC/2][BY][BX/2] sums over the pairs in z and x
    constexpr int NS = ZC / 2 * BY * (BX / 2);
    unsigned long long* const sums_lo = reinterpret_cast<unsigned long long*>(&tile[0][0][0]);
    int* const sums_hi = reinterpret_cast<int*>(sums_lo + NS);
    unsigned char* const sums_small = reinterpret_cast<unsigned char*>(sums_hi + NS);
    double* const sums = reinterpret_cast<double*>(&tile[0][0][0]);
    double s = 0.0;
    bool fx = xb + BX <= nx && yb + BY <= ny && zb + ZC <= nz;
    int E = 0;
    if (fx) {
        const MgNb nlo = mg_nb(zb, nz, g.per[0], sz), nhi = mg_nb(zb + ZC - 1, nz, g.per[0], sz);
        const MgNb ylo = mg_nb(yb, ny, g.per[1], sy), yhi = mg_nb(yb + BY - 1, ny, g.per[1], sy);
        const MgNb xlo = mg_nb(xb, nx, g.per[2], 1), xhi = mg_nb(xb + BX - 1, nx, g.per[2], 1);
        const long long c0 = ((long long)zb * ny + y) * nx + x;
        const double* __restrict__ pv = v + c0;
        const double* __restrict__ pb = b + c0;
        double col[ZC + 2], bcol[ZC];
#pragma unroll
        for (int k = 0; k < ZC; ++k) col[k + 1] = pv[k * sz];
        col[0] = nlo.wm ? pv[nlo.om] : 0.0;
        col[ZC + 1] = nhi.wp ? pv[(ZC - 1) * sz + nhi.op] : 0.0;
#pragma unroll
        for (int k = 0; k < ZC; ++k) bcol[k] = pb[k * sz];
        // the rows below and above the tile (2 ZC row segments over BY warps) and the
        // columns beside it
        constexpr int NHY = (2 * ZC + BY - 1) / BY, NHX = (2 * ZC * BY + NT - 1) / NT;
        double hy[NHY], hx[NHX];
#pragma unroll
        for (int h = 0; h < NHY; ++h) {
            const int q = ty + h * BY, pl = q >> 1;
            const double* row = v + ((long long)(zb + pl) * ny + yb) * nx + x;
            hy[h] = 0.0;
            if (q < 2 * ZC && ((q & 1) ? yhi.wp : ylo.wm)) hy[h] = row[(q & 1) ? (BY - 1) * sy + yhi.op : ylo.om];
        }
#pragma unroll
        for (int h = 0; h < NHX; ++h) {
            const int q = tid + h * NT, pl = q / (2 * BY), yr = (q >> 1) % BY;
            const double* row = v + ((long long)(zb + pl) * ny + yb + yr) * nx + xb;
            hx[h] = 0.0;
            if (q < 2 * ZC * BY && ((q & 1) ? xhi.wp : xlo.wm)) hx[h] = row[(q & 1) ? BX - 1 + xhi.op : xlo.om];
        }
        // the tile's exponent, and the smallest one that the thread can vouch for among its sums: the largest
        // of the cells above and below a cell, its b and, where the sum has it, itself
        unsigned int all = 0, low = 0x7fffffffu;
#pragma unroll
        for (int k = 0; k < ZC; ++k) {
            unsigned int m = max(max(fx_mag(col[k]), fx_mag(col[k + 2])), fx_mag(bcol[k]));
            if (MODE != 0) m = max(m, fx_mag(col[k + 1]));
            all = max(all, m);
            low = min(low, m);
        }
#pragma unroll
        for (int h = 0; h < NHY; ++h) all = max(all, fx_mag(hy[h]));
#pragma unroll
        for (int h = 0; h < NHX; ++h) all = max(all, fx_mag(hx[h]));
        all = __reduce_max_sync(0xffffffffu, all);
        if (tx == 0) swarp[ty] = all;
        __syncthreads();
        E = (int)(__reduce_max_sync(0xffffffffu, swarp[tx % BY]) >> 20);
        fx = E >= FX_EMIN && E <= FX_EMAX;
        const bool look = (int)(low >> 20) + FX_RANGE < E;
        if (fx) {
            long long f[ZC + 2];
#pragma unroll
            for (int k = 0; k < ZC + 2; ++k) f[k] = fx_from(col[k], E);
#pragma unroll
            for (int k = 0; k < ZC; ++k) tile[k][ty + 1][tx + 1] = f[k + 1];
#pragma unroll
            for (int h = 0; h < NHY; ++h) {
                const int q = ty + h * BY;
                if (q < 2 * ZC) tile[q >> 1][(q & 1) ? BY + 1 : 0][tx + 1] = fx_from(hy[h], E);
            }
#pragma unroll
            for (int h = 0; h < NHX; ++h) {
                const int q = tid + h * NT;
                if (q < 2 * ZC * BY) tile[q / (2 * BY)][((q >> 1) % BY) + 1][(q & 1) ? BX + 1 : 0] = fx_from(hx[h], E);
            }
            __syncthreads();
            const int dxy = (int)(x > 0 || g.per[2]) + (int)(x < nx - 1 || g.per[2]) + (int)(y > 0 || g.per[1]) +
                            (int)(y < ny - 1 || g.per[1]);
            const double idg = MODE == 2 ? 0.0 : g.idiag[dxy + 2], cff1 = 1.0 - g.idiag[1];   // idiag[1] = omega
            double* __restrict__ po = MODE == 2 ? nullptr : out + c0;
            FxWide acc[MODE == 2 ? ZC / 2 : 1];
            unsigned int redo = 0;   // the sums that doubles form
            if (look) {
#pragma unroll
                for (int k = 0; k < ZC; ++k) {
                    unsigned int o = fx_fold(tile[k][ty + 1][tx]) | fx_fold(tile[k][ty + 1][tx + 2]) |
                                     fx_fold(tile[k][ty][tx + 1]) | fx_fold(tile[k][ty + 2][tx + 1]) |
                                     fx_fold(f[k]) | fx_fold(f[k + 2]) | fx_fold(fx_round(bcol[k], E));
                    if (MODE != 0) o |= fx_fold(f[k + 1]);
                    redo |= (unsigned int)(o < FX_FOLD_MIN) << k;
                }
            }
#pragma unroll
            for (int k = 0; k < ZC; ++k) {
                const unsigned int dg = dxy + (k == 0 ? (int)nlo.wm : 1) + (k == ZC - 1 ? (int)nhi.wp : 1);
                const long long sum = tile[k][ty + 1][tx] + tile[k][ty + 1][tx + 2] + tile[k][ty][tx + 1] +
                                      tile[k][ty + 2][tx + 1] + f[k] + f[k + 2];
                const long long bk = fx_round(bcol[k], E);
                if (MODE == 0) {
                    const double w = (k == 0 || k == ZC - 1) ? g.idiag[dg] : idg;
                    po[k * sz] = fma(w, fx_to_double(sum - bk, E), cff1 * col[k + 1]);
                } else {
                    const long long r = bk + fx_mul(f[k + 1], dg) - sum;
                    if (MODE == 2) {
                        if (k & 1) acc[k >> 1].add(r);
                        else acc[k >> 1].set(r);
                    } else {
                        const double rd = fx_to_double(r, E), w = (k == 0 || k == ZC - 1) ? g.idiag[dg] : idg;
                        po[k * sz] = fma(-w, rd, col[k + 1]);
                        if (!(redo >> k & 1u)) s = fma(rd, rd, s);
                    }
                }
            }
            if (MODE != 2 && __any_sync(0xffffffffu, redo)) s += fx_redo_double<ZC, MODE>(g, v, b, out, xb, y, zb, redo);
            if (MODE == 2) {
                __syncthreads();   // the tile has been read
                redo &= redo >> 1;
                redo &= __shfl_down_sync(0xffffffffu, redo, 1);
#pragma unroll
                for (int k = 0; k < ZC / 2; ++k) {
                    const unsigned long long w = acc[k].lo + __shfl_down_sync(0xffffffffu, acc[k].lo, 1);
                    const int h = acc[k].hi + __shfl_down_sync(0xffffffffu, acc[k].hi, 1);
                    if ((tx & 1) == 0) {
                        const int q = (k * BY + ty) * (BX / 2) + (tx >> 1);
                        sums_lo[q] = w;
                        sums_hi[q] = h;
                        sums_small[q] = redo >> (2 * k) & 1u;
                    }
                }
            }
        }
    }
    if (!fx) s = fx_tile_double<ZC, MODE>(g, v, b, out, x, y, zb, sums);
    if (MODE == 1) block_partial(s, partial, blockIdx.z);
    if (MODE == 2) {
        __syncthreads();
        for (int q = tid; q < (ZC / 2) * (BY / 2) * (BX / 2); q += NT) {
            const int cx = q % (BX / 2), cy = (q / (BX / 2)) % (BY / 2), cz = q / (BX / 2 * (BY / 2));
            const int X = xb / 2 + cx, Y = yb / 2 + cy, Z = zb / 2 + cz;
            if (X >= gc.n[2] || Y >= gc.n[1] || Z >= gc.n[0]) continue;
            const int q0 = (cz * BY + 2 * cy) * (BX / 2) + cx, q1 = q0 + BX / 2;
            double t;
            if (fx && sums_small[q0] & sums_small[q1]) t = fx_restrict_double(g, v, b, Z, Y, X);
            else if (fx) t = FxWide{sums_lo[q0] + sums_lo[q1], sums_hi[q0] + sums_hi[q1]}.value(E);
            else t = sums[q0] + sums[q1];
            const double bv = 0.5 * t;
            const long long c = mg_at(gc, Z, Y, X);
            bc[c] = bv;
            out[c] = mg_jacobi_from_zero(bv, 0.0, mg_idiag<double>(gc, mg_diag(gc, Z, Y, X)));
        }
    }
}

// ---------------------------------------------------------------- mixed precision
// Float-pair residual r = b + diag*p - sum(p_nb), neighbours in mgfor's order. The
// neighbour sum and the centre product are error-free (TwoSum chain, TwoProduct); the
// rounding errors and the low parts are added last, so r keeps ~2^-48 of the size of
// the cancelling terms before its final rounding to float.
__device__ __forceinline__ float df_resid(float2 bc, float2 pc, float dg, const float2* nb) {
    float s, e, t;
    two_sum(nb[0].x, nb[1].x, s, e);
#pragma unroll
    for (int k = 2; k < 6; ++k) {
        two_sum(s, nb[k].x, s, t);
        e = __fadd_rn(e, t);
    }
    float lo = nb[0].y;
#pragma unroll
    for (int k = 1; k < 6; ++k) lo = __fadd_rn(lo, nb[k].y);
    float c, ce;
    two_prod(dg, pc.x, c, ce);
    float a1, t1, a2, t2;
    two_sum(bc.x, c, a1, t1);
    two_sum(a1, -s, a2, t2);
    const float rest = __fsub_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(bc.y, ce), t1), t2), __fmul_rn(dg, pc.y)),
                                 __fadd_rn(e, lo));
    return __fadd_rn(a2, rest);
}

// float-pair neighbour read with the wet flag of mg_nb (always loads, 0 when dry)
__device__ __forceinline__ float2 mg_ldw_df(const float2* __restrict__ a, long long c, bool wet) {
    const float2 v = a[c];
    return wet ? v : make_float2(0.f, 0.f);
}

// residual of the float-pair solution: its sum of squares (for the stop test), the
// float right-hand side r32 of the next correction V-cycle, and the first half-sweep
// of that V-cycle from its zero initial correction, y32. The squares are summed in
// float per thread on r * scale, scale = sc[SC_SCALE] a power of two near 1/rms(b)
// (k_mg_sumsq_df), so that they neither underflow nor overflow; each block partial is
// unscaled in double.
template <bool BAT = false>
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_resid_df(const MgGeom g, const float2* __restrict__ p,
                                                                 const float2* __restrict__ b, float* __restrict__ r32,
                                                                 float* __restrict__ y32, float omega,
                                                                 const double* __restrict__ sc,
                                                                 double* __restrict__ partial, const Bat bat = Bat()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        p = bshift(p, dlt);
        b = bshift(b, dlt);
        r32 = bshift(r32, dlt);
        y32 = bshift(y32, dlt);
        sc = bshift(sc, dlt);
        partial = bshift(partial, dlt);
    }
    constexpr int ZC = MG_DFZC;
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    const int nz = g.n[0], z0 = bz * ZC;
    const float scale = (float)sc[SC_SCALE];
    float s = 0.f;
    if (x < g.n[2] && y < g.n[1]) {
        const long long sy = g.n[2], sz = (long long)g.n[1] * g.n[2];
        const MgNb nx = mg_nb(x, g.n[2], g.per[2], 1), ny = mg_nb(y, g.n[1], g.per[1], sy);
        const int dxy = (int)nx.wm + (int)nx.wp + (int)ny.wm + (int)ny.wp;
        const long long c0 = mg_at(g, z0, y, x);
        // bc: the cell's right-hand side (loaded ahead by the caller)
        auto cell = [&](long long c, float2 zm, float2 p0, float2 zp, int dg, float2 bc) {
            const float2 nb[6] = {mg_ldw_df(p, c + nx.om, nx.wm), mg_ldw_df(p, c + nx.op, nx.wp),
                                  mg_ldw_df(p, c + ny.om, ny.wm), mg_ldw_df(p, c + ny.op, ny.wp), zm, zp};
            const float r = df_resid(bc, p0, (float)dg, nb);
            r32[c] = r;
            y32[c] = mg_jacobi_from_zero(r, omega, mg_idiag<float>(g, dg));
            const float rs = __fmul_rn(r, scale);
            s = __fmaf_rn(rs, rs, s);
        };
        if (z0 + ZC <= nz) {
            const MgNb lo = mg_nb(z0, nz, g.per[0], sz), hi = mg_nb(z0 + ZC - 1, nz, g.per[0], sz);
            float2 col[ZC + 2];
            col[0] = mg_ldw_df(p, c0 + lo.om, lo.wm);
#pragma unroll
            for (int k = 1; k <= ZC; ++k) col[k] = p[c0 + (k - 1) * sz];
            col[ZC + 1] = mg_ldw_df(p, c0 + (ZC - 1) * sz + hi.op, hi.wp);
            float2 bcol[ZC];
#pragma unroll
            for (int k = 0; k < ZC; ++k) bcol[k] = b[c0 + k * sz];
#pragma unroll
            for (int k = 0; k < ZC; ++k)
                cell(c0 + k * sz, col[k], col[k + 1], col[k + 2],
                     dxy + (k == 0 ? 1 + (int)lo.wm : (k == ZC - 1 ? 1 + (int)hi.wp : 2)), bcol[k]);
        } else {
            for (int z = z0; z < nz; ++z) {
                const long long c = c0 + (z - z0) * sz;
                const MgNb nzb = mg_nb(z, nz, g.per[0], sz);
                cell(c, mg_ldw_df(p, c + nzb.om, nzb.wm), p[c], mg_ldw_df(p, c + nzb.op, nzb.wp),
                     dxy + (int)nzb.wm + (int)nzb.wp, b[c]);
            }
        }
    }
    block_partial_f(s, sc[SC_INVSCALE2], partial, bz);
}

// k_mg_resid_df with 4 consecutive x cells per thread: each float-pair row segment is
// two 16-byte loads, the x neighbours come from the adjacent lanes (loaded at the warp's
// ends and at the level's x faces), r32 and y32 are stored 16 bytes at a time. Needs nx
// and nz divisible by 4 and V4_ZC; same per-cell arithmetic as k_mg_resid_df.
struct DfVec4 {
    float2 v[4];
};
template <bool BAT = false>
__global__ void __launch_bounds__(MG_BX * MG_BY, 3) k_mg_resid_df_v4(const MgGeom g, const float2* __restrict__ p,
                                                                    const float2* __restrict__ b,
                                                                    float* __restrict__ r32, float* __restrict__ y32,
                                                                    float omega, const double* __restrict__ sc,
                                                                    double* __restrict__ partial,
                                                                    const Bat bat = Bat(), MgFin fin = MgFin()) {
    int bz = blockIdx.z;
    if constexpr (BAT) {
        long long dlt;
        if (!batch_enter(bat, bz, dlt)) return;
        p = bshift(p, dlt);
        b = bshift(b, dlt);
        r32 = bshift(r32, dlt);
        y32 = bshift(y32, dlt);
        sc = bshift(sc, dlt);
        partial = bshift(partial, dlt);
        fin.ticket = bshift(fin.ticket, dlt);
        fin.sc = bshift(fin.sc, dlt);
    }
    const int nx = g.n[2], ny = g.n[1], nz = g.n[0];
    const int nx4 = nx >> 2;
    const int lane = threadIdx.x;
    const int xv = blockIdx.x * MG_BX + lane;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    const float scale = (float)sc[SC_SCALE];
    float s = 0.f;
    const bool act = xv < nx4 && y < ny;
    const int x0 = min(xv, nx4 - 1) * 4, ys = min(y, ny - 1);
    const long long sy = nx, sz = (long long)ny * nx;
    const MgNb nyb = mg_nb(ys, ny, g.per[1], sy);
    const bool wl = x0 > 0 || g.per[2], wr = x0 + 4 < nx || g.per[2];
    const long long ol = x0 > 0 ? -1 : (g.per[2] ? (long long)(nx - 1) : 0);
    const long long orr = x0 + 4 < nx ? 4 : (g.per[2] ? (long long)(4 - nx) : 0);
    const bool ownl = lane == 0 || x0 == 0, ownr = lane == MG_BX - 1 || x0 + 4 >= nx;
    int dgx[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int xx = x0 + e;
        dgx[e] = (int)(xx > 0 || g.per[2]) + (int)(xx < nx - 1 || g.per[2]) + (int)nyb.wm + (int)nyb.wp;
    }
    const int zb = bz * V4_ZC;
    const long long c00 = (long long)ys * sy + x0;
    auto ld = [&](const float2* a, long long c) -> DfVec4 {
        const float4* q = reinterpret_cast<const float4*>(a + c);
        const float4 u = q[0], w = q[1];
        DfVec4 d;
        d.v[0] = make_float2(u.x, u.y);
        d.v[1] = make_float2(u.z, u.w);
        d.v[2] = make_float2(w.x, w.y);
        d.v[3] = make_float2(w.z, w.w);
        return d;
    };
    DfVec4 zero;
#pragma unroll
    for (int e = 0; e < 4; ++e) zero.v[e] = make_float2(0.f, 0.f);
    auto zrow = [&](int zz) -> DfVec4 {
        if (zz < 0) return g.per[0] ? ld(p, c00 + (long long)(nz - 1) * sz) : zero;
        if (zz >= nz) return g.per[0] ? ld(p, c00) : zero;
        return ld(p, c00 + (long long)zz * sz);
    };
    DfVec4 zm = zrow(zb - 1), zc = zrow(zb);
#pragma unroll
    for (int k = 0; k < V4_ZC; ++k) {
        const int zz = zb + k;
        const DfVec4 zp = zrow(zz + 1);
        const long long c = c00 + (long long)zz * sz;
        const DfVec4 ym = nyb.wm ? ld(p, c + nyb.om) : zero;
        const DfVec4 yp = nyb.wp ? ld(p, c + nyb.op) : zero;
        const DfVec4 bv = ld(b, c);
        const float lx = __shfl_up_sync(0xffffffffu, zc.v[3].x, 1), ly = __shfl_up_sync(0xffffffffu, zc.v[3].y, 1);
        const float rx = __shfl_down_sync(0xffffffffu, zc.v[0].x, 1), ry = __shfl_down_sync(0xffffffffu, zc.v[0].y, 1);
        const float2 left = ownl ? mg_ldw_df(p, c + ol, wl) : make_float2(lx, ly);
        const float2 right = ownr ? mg_ldw_df(p, c + orr, wr) : make_float2(rx, ry);
        const int dzw = (int)(zz > 0 || g.per[0]) + (int)(zz < nz - 1 || g.per[0]);
        float rv[4], yv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int dg = dgx[e] + dzw;
            const float2 nb[6] = {e == 0 ? left : zc.v[e - 1], e == 3 ? right : zc.v[e + 1], ym.v[e], yp.v[e],
                                  zm.v[e], zp.v[e]};
            const float r = df_resid(bv.v[e], zc.v[e], (float)dg, nb);
            rv[e] = r;
            yv[e] = mg_jacobi_from_zero(r, omega, mg_idiag<float>(g, dg));
            if (act) {
                const float rs = __fmul_rn(r, scale);
                s = __fmaf_rn(rs, rs, s);
            }
        }
        if (act) {
            *reinterpret_cast<float4*>(r32 + c) = make_float4(rv[0], rv[1], rv[2], rv[3]);
            *reinterpret_cast<float4*>(y32 + c) = make_float4(yv[0], yv[1], yv[2], yv[3]);
        }
        zm = zc;
        zc = zp;
    }
    block_partial_f(s, sc[SC_INVSCALE2], partial, bz);
    // sum(r^2) into sc[SC_RR] (k_mg_final's work)
    if (fin.ticket) {
        const unsigned int nblk = gridDim.x * gridDim.y * (gridDim.z / (BAT ? bat.nrun : 1));
        if (mg_last_block(fin.ticket, nblk)) {
            const double2 t = mg_block_total2(partial, nullptr, (int)nblk);
            if (threadIdx.x == 0 && threadIdx.y == 0) fin.sc[SC_RR] = t.x;
        }
    }
}

// ---------------------------------------------------------------- Krylov acceleration
// Mixed precision with mg_krylov: flexible conjugate gradients FCG(1) on the level-0
// equation, preconditioned by the FP32 V-cycle (zero initial guess), with the float-pair
// solution x and the float-pair true residual of iterative refinement:
//   r = b - A x (k_mg_resid_df; stop test), z = V(r), p = z + beta p with
//   beta = -(z.q)/(p.q) of the previous direction (0 on the first iteration),
//   q = A p, alpha = (p.r)/(p.q), x += alpha p.
// A x = sum(x_nb) - diag*x is the operator whose residual k_mg_resid_df forms; it is
// negative definite, which leaves alpha and beta unchanged against the positive form.
// The V-cycle is not symmetric (the restriction is not the transposed prolongation),
// hence the flexible beta. Scalars live in the solve's slots: SC_ZQ, SC_PQ, SC_PR as
// doubles, beta as a float and alpha as a float pair (so that the elementwise kernels
// do no FP64 work).


// sums of the partials of z.q and of z, then beta = -(z.q)/(p.q) of the previous
// iteration (0 on the first: k = iteration of this solve, or sc[SC_NITE] when k < 0),
// stored as a float, and the mean of z (float)
__global__ void k_fcg_final_beta(const double* __restrict__ pzq, const double* __restrict__ pz, int n, double vol,
                                 double* __restrict__ sc, int k) {
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        a += pzq[i];
        b += pz[i];
    }
    __shared__ double sm[2][32];
    a = warp_sum(a);
    b = warp_sum(b);
    if ((threadIdx.x & 31) == 0) {
        sm[0][threadIdx.x >> 5] = a;
        sm[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool in = threadIdx.x < (blockDim.x >> 5);
        double zq = in ? sm[0][threadIdx.x] : 0.0, zs = in ? sm[1][threadIdx.x] : 0.0;
        zq = warp_sum(zq);
        zs = warp_sum(zs);
        if (threadIdx.x == 0) fcg_set_beta(zq, zs, vol, sc, k);
    }
}

// New direction and its image, in place: p = (z - mean z) + beta p and
// q = A p = A z + beta q (A is linear and A 1 = 0, so only z is read at the
// neighbours), with the partial sums of p.q and p.r. A z = sum(z_nb) - diag*z.
// Walls and periodic directions leave A the constant null space: a right-hand side with
// a component along it (the reference's viscosity moves wall-face velocities) makes the
// stationary iteration stall at a residual floor, and would make the directions drift
// along the constant without the mean removal.
__global__ void __launch_bounds__(MG_BX * MG_BY) k_fcg_direction(const MgGeom g, const float* __restrict__ z,
                                                                 const float* __restrict__ r, float* __restrict__ p,
                                                                 float* __restrict__ q, const double* __restrict__ sc,
                                                                 double* __restrict__ ppq, double* __restrict__ ppr) {
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    const float beta = reinterpret_cast<const float*>(sc + SC_BETA)[0];
    const float zmean = reinterpret_cast<const float*>(sc + SC_ZMEAN)[0];
    float spq = 0.f, spr = 0.f;
    if (x < g.n[2] && y < g.n[1]) {
        const int nz = g.n[0], z0 = blockIdx.z * MG_ZC;
        const long long sy = g.n[2], sz = (long long)g.n[1] * g.n[2];
        const MgNb nx = mg_nb(x, g.n[2], g.per[2], 1), ny = mg_nb(y, g.n[1], g.per[1], sy);
        const int dxy = (int)nx.wm + (int)nx.wp + (int)ny.wm + (int)ny.wp;
        const long long c0 = mg_at(g, z0, y, x);
        auto cell = [&](long long c, float zm, float z0v, float zp, int dg) {
            const float s = ((((mg_ldw(z, c + nx.om, nx.wm) + mg_ldw(z, c + nx.op, nx.wp)) +
                               mg_ldw(z, c + ny.om, ny.wm)) + mg_ldw(z, c + ny.op, ny.wp)) + zm) + zp;
            const float az = __fmaf_rn(-(float)dg, z0v, s);
            const float pv = __fmaf_rn(beta, p[c], __fsub_rn(z0v, zmean));
            const float qv = __fmaf_rn(beta, q[c], az);
            p[c] = pv;
            q[c] = qv;
            spq = __fmaf_rn(pv, qv, spq);
            spr = __fmaf_rn(pv, r[c], spr);
        };
        if (z0 + MG_ZC <= nz) {
            const MgNb lo = mg_nb(z0, nz, g.per[0], sz), hi = mg_nb(z0 + MG_ZC - 1, nz, g.per[0], sz);
            float col[MG_ZC + 2];
            col[0] = mg_ldw(z, c0 + lo.om, lo.wm);
#pragma unroll
            for (int k = 1; k <= MG_ZC; ++k) col[k] = z[c0 + (k - 1) * sz];
            col[MG_ZC + 1] = mg_ldw(z, c0 + (MG_ZC - 1) * sz + hi.op, hi.wp);
#pragma unroll
            for (int k = 0; k < MG_ZC; ++k)
                cell(c0 + k * sz, col[k], col[k + 1], col[k + 2],
                     dxy + (k == 0 ? 1 + (int)lo.wm : (k == MG_ZC - 1 ? 1 + (int)hi.wp : 2)));
        } else {
            for (int zz = z0; zz < nz; ++zz) {
                const long long c = c0 + (zz - z0) * sz;
                const MgNb nzb = mg_nb(zz, nz, g.per[0], sz);
                cell(c, mg_ldw(z, c + nzb.om, nzb.wm), z[c], mg_ldw(z, c + nzb.op, nzb.wp),
                     dxy + (int)nzb.wm + (int)nzb.wp);
            }
        }
    }
    block_partial2_f(spq, spr, ppq, ppr, blockIdx.z);
}

// The same with 4 consecutive x cells per thread (16-byte loads and stores: the kernel
// is bound by the latency of its loads) and z-chunks of V4_ZC cells; needs nx and nz
// divisible by 4 and V4_ZC. The x neighbours of a vector come from the adjacent lanes
// of the warp (one warp = one row segment of 128 cells), and are loaded at the warp's
// ends and at the level's x faces (periodic image or dry). Same per-cell arithmetic as
// k_fcg_direction.
__global__ void __launch_bounds__(MG_BX * MG_BY, 5) k_fcg_direction_v4(const MgGeom g, const float* __restrict__ z,
                                                                    const float* __restrict__ r, float* __restrict__ p,
                                                                    float* __restrict__ q,
                                                                    const double* __restrict__ sc,
                                                                    double* __restrict__ ppq, double* __restrict__ ppr,
                                                                    const MgFin fin = MgFin()) {
    const int nx = g.n[2], ny = g.n[1], nz = g.n[0];
    const int nx4 = nx >> 2;
    const int lane = threadIdx.x;
    const int xv = blockIdx.x * MG_BX + lane;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    const float beta = reinterpret_cast<const float*>(sc + SC_BETA)[0];
    const float zmean = reinterpret_cast<const float*>(sc + SC_ZMEAN)[0];
    float spq = 0.f, spr = 0.f;
    // idle lanes shadow the last vector of the row so that every lane takes part in the
    // shuffles; only active lanes store and sum
    const bool act = xv < nx4 && y < ny;
    const int x0 = min(xv, nx4 - 1) * 4, ys = min(y, ny - 1);
    const long long sy = nx, sz = (long long)ny * nx;
    const MgNb nyb = mg_nb(ys, ny, g.per[1], sy);
    // cells x0-1 and x0+4: offsets from cell x0 and wet flags
    const bool wl = x0 > 0 || g.per[2], wr = x0 + 4 < nx || g.per[2];
    const long long ol = x0 > 0 ? -1 : (g.per[2] ? (long long)(nx - 1) : 0);
    const long long orr = x0 + 4 < nx ? 4 : (g.per[2] ? (long long)(4 - nx) : 0);
    const bool ownl = lane == 0 || x0 == 0, ownr = lane == MG_BX - 1 || x0 + 4 >= nx;
    // wet x neighbours of the four cells
    int dgx[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int xx = x0 + e;
        dgx[e] = (int)(xx > 0 || g.per[2]) + (int)(xx < nx - 1 || g.per[2]) + (int)nyb.wm + (int)nyb.wp;
    }
    const int zb = blockIdx.z * V4_ZC;
    const long long c00 = (long long)ys * sy + x0;
    auto ld4 = [&](long long c) { return *reinterpret_cast<const float4*>(z + c); };
    auto zrow = [&](int zz) -> float4 {   // z value of the vector at level row zz (periodic image or dry)
        const MgNb nzb = mg_nb(zz < 0 ? 0 : (zz >= nz ? nz - 1 : zz), nz, g.per[0], sz);
        if (zz < 0) return nzb.wm ? ld4(c00 + (long long)(nz - 1) * sz) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (zz >= nz) return nzb.wp ? ld4(c00) : make_float4(0.f, 0.f, 0.f, 0.f);
        return ld4(c00 + (long long)zz * sz);
    };
    float4 zm = zrow(zb - 1), zc = zrow(zb);
#pragma unroll
    for (int k = 0; k < V4_ZC; ++k) {
        const int zz = zb + k;
        const float4 zp = zrow(zz + 1);
        const long long c = c00 + (long long)zz * sz;
        const float4 ym = nyb.wm ? ld4(c + nyb.om) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 yp = nyb.wp ? ld4(c + nyb.op) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 pv0 = *reinterpret_cast<const float4*>(p + c);
        const float4 qv0 = *reinterpret_cast<const float4*>(q + c);
        const float4 rv = *reinterpret_cast<const float4*>(r + c);
        const float sl = __shfl_up_sync(0xffffffffu, zc.w, 1);
        const float sr = __shfl_down_sync(0xffffffffu, zc.x, 1);
        const float left = ownl ? mg_ldw(z, c + ol, wl) : sl;
        const float right = ownr ? mg_ldw(z, c + orr, wr) : sr;
        const int dzw = (int)(zz > 0 || g.per[0]) + (int)(zz < nz - 1 || g.per[0]);
        const float zv[4] = {zc.x, zc.y, zc.z, zc.w};
        const float xm[4] = {left, zc.x, zc.y, zc.z}, xp[4] = {zc.y, zc.z, zc.w, right};
        const float yv[2][4] = {{ym.x, ym.y, ym.z, ym.w}, {yp.x, yp.y, yp.z, yp.w}};
        const float zmv[4] = {zm.x, zm.y, zm.z, zm.w}, zpv[4] = {zp.x, zp.y, zp.z, zp.w};
        const float p0[4] = {pv0.x, pv0.y, pv0.z, pv0.w}, q0[4] = {qv0.x, qv0.y, qv0.z, qv0.w};
        const float rr[4] = {rv.x, rv.y, rv.z, rv.w};
        float po[4], qo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float s = ((((xm[e] + xp[e]) + yv[0][e]) + yv[1][e]) + zmv[e]) + zpv[e];
            const float az = __fmaf_rn(-(float)(dgx[e] + dzw), zv[e], s);
            po[e] = __fmaf_rn(beta, p0[e], __fsub_rn(zv[e], zmean));
            qo[e] = __fmaf_rn(beta, q0[e], az);
            if (act) {
                spq = __fmaf_rn(po[e], qo[e], spq);
                spr = __fmaf_rn(po[e], rr[e], spr);
            }
        }
        if (act) {
            *reinterpret_cast<float4*>(p + c) = make_float4(po[0], po[1], po[2], po[3]);
            *reinterpret_cast<float4*>(q + c) = make_float4(qo[0], qo[1], qo[2], qo[3]);
        }
        zm = zc;
        zc = zp;
    }
    block_partial2_f(spq, spr, ppq, ppr, blockIdx.z);
    // alpha from the totals of p.q and p.r (k_fcg_final_alpha's work)
    if (fin.ticket) {
        const unsigned int nblk = gridDim.x * gridDim.y * gridDim.z;
        if (mg_last_block(fin.ticket, nblk)) {
            const double2 t = mg_block_total2(ppq, ppr, (int)nblk);
            if (threadIdx.x == 0 && threadIdx.y == 0) fcg_set_alpha(t.x, t.y, fin.sc);
        }
    }
}

// sums of p.q and p.r, then alpha = (p.r)/(p.q) stored as a float pair
__global__ void k_fcg_final_alpha(const double* __restrict__ ppq, const double* __restrict__ ppr, int n,
                                  double* __restrict__ sc) {
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        a += ppq[i];
        b += ppr[i];
    }
    __shared__ double sm[2][32];
    a = warp_sum(a);
    b = warp_sum(b);
    if ((threadIdx.x & 31) == 0) {
        sm[0][threadIdx.x >> 5] = a;
        sm[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool in = threadIdx.x < (blockDim.x >> 5);
        double pq = in ? sm[0][threadIdx.x] : 0.0, pr = in ? sm[1][threadIdx.x] : 0.0;
        pq = warp_sum(pq);
        pr = warp_sum(pr);
        if (threadIdx.x == 0) fcg_set_alpha(pq, pr, sc);
    }
}

// x += alpha p on the float-pair solution (level 0, elementwise)
__global__ void __launch_bounds__(256) k_fcg_xupdate(float2* __restrict__ xdf, const float* __restrict__ p,
                                                     long long n, const double* __restrict__ sc) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 alpha = reinterpret_cast<const float2*>(sc + SC_ALPHA)[0];
    xdf[i] = df_add(xdf[i], df_mul_f(p[i], alpha));
}

// Extrapolated warm start of a mixed-precision solve. The solution array x(n-1) has
// MG_HIST history arrays holding x(n-2), x(n-3), ... With `order` p and at least p + 1
// solves seen (else the highest order they allow), the start becomes the polynomial
// extrapolation of the last p + 1 solutions to the next step (equal steps; binomial
// coefficients: 2, -1; 3, -3, 1; 4, -6, 4, -1), formed in float-pair arithmetic (FP64
// here ran the kernel at a fifth of the copy bandwidth: GB300's FP64 pipe, which also
// does the float-double conversions, is a small fraction of its FP32 rate). The
// history then shifts by one. Nothing changes when the right-hand side's
// norm (scalar slot SC_NORMB, set just before) is zero or not finite: the solve then
// keeps its start (a zero right-hand side) or stops at once (blow-up).
// k_mg_hist_count, launched after, counts the solve.
constexpr int MG_HIST = 3;
struct HistPtrs {
    float2* h[MG_HIST];   // x(n-2), x(n-3), x(n-4)
};
__global__ void __launch_bounds__(256) k_mg_extrapolate(float2* __restrict__ cur, HistPtrs hp, long long n,
                                                        int order, const double* __restrict__ sc,
                                                        const int* __restrict__ count, const Bat bat = Bat()) {
    int bz;
    long long dlt;
    if (!batch_enter(bat, bz, dlt)) return;
    cur = bshift(cur, dlt);
#pragma unroll
    for (int k = 0; k < MG_HIST; ++k) hp.h[k] = bshift(hp.h[k], dlt);
    sc = bshift(sc, dlt);
    count = bshift(count, dlt);
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double nb = sc[SC_NORMB];
    if (!(nb > 0.0 && nb <= 1.7976931348623157e308)) return;
    const int p = min(order, *count - 1);   // order the history allows
    float2 v[MG_HIST + 1];
    v[0] = cur[i];
#pragma unroll
    for (int k = 0; k < MG_HIST; ++k) v[k + 1] = (k < order) ? hp.h[k][i] : make_float2(0.f, 0.f);
    if (p >= 1) {
        float2 e;
        if (p == 1) e = df_add(make_float2(2.f * v[0].x, 2.f * v[0].y), df_neg(v[1]));
        else if (p == 2) e = df_add(df_mul_f(3.f, df_add(v[0], df_neg(v[1]))), v[2]);
        else e = df_add(df_add(df_mul_f(4.f, df_add(v[0], v[2])), df_mul_f(-6.f, v[1])), df_neg(v[3]));
        cur[i] = e;
    }
#pragma unroll
    for (int k = MG_HIST - 1; k >= 0; --k)
        if (k < order) hp.h[k][i] = v[k];
}

// one thread per run: the count of solves seen by the solution array (saturating at
// MG_HIST + 1)
__global__ void k_mg_hist_count(int* count, const double* sc, const Bat bat = Bat()) {
    const int r = threadIdx.x;
    if (bat.tab) {
        if (r >= bat.nrun || !bat.tab->active[r]) return;
        count = bshift(count, bat.tab->delta[r]);
        sc = bshift(sc, bat.tab->delta[r]);
    } else if (r > 0) {
        return;
    }
    const double nb = sc[SC_NORMB];
    if (nb > 0.0 && nb <= 1.7976931348623157e308 && *count < MG_HIST + 1) *count += 1;
}

// sum of squares of a float-pair array (high parts, squared and summed in double)
// |a| as a double, for normal numbers by moving its bits (the conversion instruction runs on the FP64 pipe)
__device__ __forceinline__ double exact_double(float a) {
    const unsigned int u = __float_as_uint(a) & 0x7fffffffu;
    if (u == 0u) return 0.0;
    if (u - 0x00800000u >= 0x7f000000u) return fabs((double)a);   // denormal, infinity, NaN
    return __hiloint2double((int)((u >> 3) + 0x38000000u), (int)(u << 29));
}

// Sum of the squares of the high words of the float-pair right-hand side. Bound by the FP64 pipe, which also
// does the block sums: 512 x 256 x 256 cells 169 us with a conversion per cell and 8 planes per thread (181 with the
// bits moved), 144 us with 32.
// Also the scale of the float sums of squares: 2^-e with 2^e near rms(b) = sqrt(sum(b^2)/vol),
// and its inverse square (both exact powers of two).
__global__ void __launch_bounds__(MG_BX * MG_BY) k_mg_sumsq_df(const MgGeom g, const float2* __restrict__ v,
                                                              double* __restrict__ partial, MgFin fin, const int zc,
                                                              const Bat bat = Bat()) {
    int bz;
    long long dlt;
    if (!batch_enter(bat, bz, dlt)) return;
    v = bshift(v, dlt);
    partial = bshift(partial, dlt);
    fin.ticket = bshift(fin.ticket, dlt);
    double* const sc = bshift(fin.sc, dlt);
    const int x = blockIdx.x * MG_BX + threadIdx.x;
    const int y = blockIdx.y * MG_BY + threadIdx.y;
    double s = 0.0;
    if (x < g.n[2] && y < g.n[1]) {
        const long long sz = (long long)g.n[1] * g.n[2];
        const int z1 = min((bz + 1) * zc, g.n[0]);
        for (int z = bz * zc; z < z1; z += MG_ZC) {
            const float2* q = v + mg_at(g, z, y, x);
            float h[MG_ZC];
#pragma unroll
            for (int k = 0; k < MG_ZC; ++k) h[k] = z + k < z1 ? q[k * sz].x : 0.f;
#pragma unroll
            for (int k = 0; k < MG_ZC; ++k) {
                const double d = exact_double(h[k]);
                s += d * d;
            }
        }
    }
    block_partial(s, partial, bz);
    double nb;
    if (mg_fin_total(fin, partial, gridDim.x * gridDim.y * (gridDim.z / bat.nrun), nb)) {
        int e = 0;
        if (nb > 0.0) frexp(sqrt(nb / fin.vol), &e);
        e = max(-120, min(120, e));
        sc[SC_NORMB] = nb;
        sc[SC_SCALE] = ldexp(1.0, -e);
        sc[SC_INVSCALE2] = ldexp(1.0, 2 * e);
    }
}

__global__ void k_mg_final(const double* __restrict__ partial, int n, double* __restrict__ out,
                           const Bat bat = Bat()) {
    int bz;
    long long dlt;
    if (!batch_enter(bat, bz, dlt)) return;
    partial = bshift(partial, dlt);
    out = bshift(out, dlt);
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
    __shared__ double sm[32];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = (threadIdx.x < (blockDim.x >> 5)) ? sm[threadIdx.x] : 0.0;
        t = warp_sum(t);
        if (threadIdx.x == 0) *out = t;
    }
}

// ---------------------------------------------------------------- device-side stop test
// before the loop: res = sum(r^2)/sum(b^2) (0 when b = 0), continue while res >= tol
__device__ __forceinline__ bool finite_dev(double v) { return v == v && v <= 1.7976931348623157e308; }

// One thread per run (a single thread for one run): each run's stop test, its `live`
// flag in a batched launch, and the loop condition = any run still iterating.
__global__ void k_mg_ctl_begin(double* __restrict__ sc0, cudaGraphConditionalHandle h, double tol,
                               const Bat bat = Bat()) {
    const int r = threadIdx.x;
    bool go = false;
    if (r < bat.nrun && (!bat.tab || bat.tab->active[r])) {
        double* sc = bat.tab ? bshift(sc0, bat.tab->delta[r]) : sc0;
        const double normb = sc[SC_NORMB];
        const double res = normb > 0.0 ? sc[SC_RR] / normb : 0.0;
        sc[SC_RES] = res;
        sc[SC_NITE] = 0.0;
        if (!finite_dev(normb) || !finite_dev(res))   // non-finite input: no V-cycle (host: NYLES_BLOWUP)
            sc[SC_NONFINITE] = sc[SC_NONFINITE] + 1.0;
        else
            go = !(res < tol);
    }
    if (bat.tab && r < NYLES_MAX_BATCH) bat.tab->live[r] = go ? 1 : 0;
    const int any = __syncthreads_or(go ? 1 : 0);
    if (r == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

// after each V-cycle: nite += 1; stop at maxite (res keeps its previous value, as
// solvers.f90:24-26 leaves the loop before recomputing it), else recompute res
__global__ void k_mg_ctl_step(double* __restrict__ sc0, cudaGraphConditionalHandle h, double tol, int maxite,
                              const Bat bat = Bat()) {
    const int r = threadIdx.x;
    bool go = false;
    if (r < bat.nrun && (!bat.tab || bat.tab->live[r])) {   // runs whose solve stopped keep their counters
        double* sc = bat.tab ? bshift(sc0, bat.tab->delta[r]) : sc0;
        const double nite = sc[SC_NITE] + 1.0;
        sc[SC_NITE] = nite;
        sc[SC_TOTAL] = sc[SC_TOTAL] + 1.0;
        if (nite >= (double)maxite) {
            if (sc[SC_RES] >= tol) sc[SC_NCONV] = sc[SC_NCONV] + 1.0;   // as mg_solve's count
        } else {
            const double normb = sc[SC_NORMB];
            const double res = normb > 0.0 ? sc[SC_RR] / normb : 0.0;
            sc[SC_RES] = res;
            if (!finite_dev(res))
                sc[SC_NONFINITE] = sc[SC_NONFINITE] + 1.0;
            else
                go = !(res < tol);
        }
        if (bat.tab) bat.tab->live[r] = go ? 1 : 0;
    }
    const int any = __syncthreads_or(go ? 1 : 0);
    if (r == 0) {
        if (bat.tab) bat.tab->loop_iterations += 1;
        cudaGraphSetConditional(h, any ? 1u : 0u);
    }
}

// ---------------------------------------------------------------- host side
static inline dim3 grid_zc(const int n[3], int zc) {
    return dim3((n[2] + MG_BX - 1) / MG_BX, (n[1] + MG_BY - 1) / MG_BY, (n[0] + zc - 1) / zc);
}
static inline long long blocks(dim3 g) { return (long long)g.x * g.y * g.z; }
static const dim3 kBlk(MG_BX, MG_BY, 1);
// the grid of a batched launch repeats the one-run grid along z once per run
static inline dim3 bgrid(const MgImpl* mg, dim3 g) {
    if (mg->bat.tab) g.z *= mg->bat.nrun;
    return g;
}

// FP64 levels: the integer-sum kernel where a level's 8-cell columns fill the chip; below,
// the double kernels with one cell per thread (their launches last as long as one thread's
// chain of FP64 instructions: 8 cells 9 us, 1 cell 4 us on 32^3 and 16^3). Measured with the line at
// 2^15 / 2^18 / 2^19 cells / everything in doubles: a 128^3 solve 1.364 / 1.361 / 1.387 / 2.086 ms, a
// 128 x 64 x 64 LFAM3 step 2.64 / 2.65 / 2.65 / 2.96 ms.
// A level that the 32 x 8 x 8 tiles do not divide has cut tiles, summed in doubles cell after cell; on
// small ones their latency shows, and the line lies higher. V-cycles in us, integers / doubles of one cell per
// thread / of eight: 48 x 104 x 56 173 / 147 / 198, 80 x 64 x 64 184 / 161 / 207, 48 x 96 x 96 187 / 180 / 211,
// 112 x 64 x 64 186 / 171 / 212; 80^3 191 / 194 / 224, 40 x 128 x 128 208 / 221 / 253, 48 x 192 x 96 223 / 252 / 298,
// 144^3 389 / 547 / 536.
// A level without a whole tile takes doubles: one cell per thread while that leaves few blocks (16 x 128 x 128, 2048 of
// them: 166 / 167 / 204; 24 x 128 x 128 181 / 181 / 206), else eight (8192 or more: 16 x 256 x 256 417 / 432 / 386,
// 4 x 512 x 512 961 / 1181 / 936, 512 x 4 x 512 193 / 186 / 178, 512 x 2 x 512 78 / 59 / 62).
constexpr int FX_ZC = 8;
constexpr long long FX_MINVOL = 1ll << 18, FX_MINVOL_CUT = 500000, ONE_CELL_BLOCKS = 4096;
// cells per thread of an FP64 level's double kernels, 0: the integer sums
static inline int fp64_zc(const MgImpl* mg, int l) {
    const MgLevelDesc& d = mg->lev[l];
    if (d.n[2] < MG_BX || d.n[1] < MG_BY || d.n[0] < FX_ZC) return blocks(grid_zc(d.n, 1)) <= ONE_CELL_BLOCKS ? 1 : MG_ZC;
    const bool cut = d.n[2] % MG_BX || d.n[1] % MG_BY || d.n[0] % FX_ZC;
    return d.vol >= (cut ? FX_MINVOL_CUT : FX_MINVOL) ? 0 : 1;
}

// the 4-cell vector kernels apply to a level whose x and z extents allow them; zc = the
// z cells per thread (V4_ZC for the float-pair and Krylov kernels, lvl_zc below for the others)
static inline bool use_v4(const MgImpl* mg, const int n[3], int zc = V4_ZC) {
    return mg->vec4 && n[2] % 4 == 0 && n[0] % zc == 0;
}
static inline dim3 grid_v4(const int n[3], int zc = V4_ZC) {
    return dim3((unsigned)((n[2] / 4 + MG_BX - 1) / MG_BX), (unsigned)((n[1] + MG_BY - 1) / MG_BY),
                (unsigned)(n[0] / zc));
}
// Block partials of a level-0 sum over `count` blocks (which = 0, 1: two sums of one kernel): in
// the workspace's own slots where these hold them, else in level 1's y, which holds nothing while
// the kernels that sum over level 0 run.
static inline bool partials_fit(const MgImpl* mg, long long count) {
    const long long es = mg->precision == NYLES_MIXED ? sizeof(float) : sizeof(double);
    return count <= mg->npartial || (mg->nlevels > 1 && mg->lev[1].vol * es >= 2 * count * (long long)sizeof(double));
}
static double* partials(const MgImpl* mg, int which, long long count) {
    if (count <= mg->npartial)
        return reinterpret_cast<double*>(mg->ws + (which ? mg->off_partial2 : mg->off_partial));
    return reinterpret_cast<double*>(mg->ws + mg->lev[1].off_y) + which * count;
}

// Whether the kernels that sum over level 0 (residual, Krylov) take their vector form: on narrow
// levels its blocks can be more than the workspace has slots for partials (nx <= 32 of 32 lanes x 4).
static inline bool use_v4_sums(const MgImpl* mg) {
    return use_v4(mg, mg->lev[0].n) && partials_fit(mg, blocks(grid_v4(mg->lev[0].n)));
}
// z cells per thread of the half-sweeps of level l that keep no sums (0: the scalar kernel). A large
// level 0, and one of a batch, reuses each z row from registers over V4_ZC cells; the coarser levels
// and a small level 0 are latency-bound (a few microseconds per launch whatever their size), where
// more blocks with shorter chains of dependent loads finish sooner. Mixed time steps with 4 / 1
// planes (us): 48^3 981 / 890, 64 x 64 x 32 1103 / 1008, 128 x 64 x 64 1203 / 1109, 96^3 1415 / 1379,
// 128 x 128 x 64 1555 / 1566; ten steps of four 48^3 runs 12.91 / 12.91 ms, of eight 16.64 / 17.61, of
// sixteen 32^3 runs 14.72 / 15.46. The residual stays at 4 planes: one per thread, it gains 3% of a 64 x 64 x 32
// step and loses 2% of a 64^3 one and 7% of eight batched 32^3 runs.
// Narrow levels leave lanes idle, and one plane per thread makes many blocks: 4 planes above V4_SMALL_BLOCKS of them,
// which fill the chip (V-cycles with 4 / 1 planes, us: 96^3, 1152 blocks, 1415 / 1379 a step; 16 x 128 x 128 and
// 16 x 1024 x 16, 2048 blocks, 100 / 99 and 110 / 113; 32 x 4 x 4096, 4096, 105 / 110; 4 x 256 x 256 and 8 x 256 x 256,
// 8192, 135 / 153 and 169 / 183; 4 x 4 x 16384, 208 / 243). It also keeps the planes within a grid's largest z extent.
constexpr long long V4_SMALL = 1 << 20, V4_SMALL_BLOCKS = 8 * 152;
static inline int lvl_zc(const MgImpl* mg, int l) {
    if (l) return mg->czc;
    if (!mg->bat.tab && mg->lev[0].vol < V4_SMALL && blocks(grid_v4(mg->lev[0].n, 1)) <= V4_SMALL_BLOCKS) return 1;
    return V4_ZC;
}
// coarse planes per thread of the restriction out of level l, fine planes per thread of
// the prolongation into level l (even)
static inline int lvl_rzc(const MgImpl* mg, int l) { return lvl_zc(mg, l) >= 4 ? MG_RZC : 1; }
static inline int lvl_pzc(const MgImpl* mg, int l) { return lvl_zc(mg, l) >= 4 ? V4_ZC : 2; }
static inline dim3 grid_v4_restrict(const MgGeom& gf, const MgGeom& gc, int rzc) {
    return dim3((unsigned)((gf.n[2] / 4 + MG_BX - 1) / MG_BX), (unsigned)((gc.n[1] + MG_BY - 1) / MG_BY),
                (unsigned)(gc.n[0] / rzc));
}
// ticket counter of the reductions folded into their kernels (MgFin), in a workspace
// slot zeroed when the workspace is bound
static inline unsigned int* fin_ticket(MgImpl* mg) {
    return reinterpret_cast<unsigned int*>(mg->ws + mg->off_ticket);
}
static MgFin mg_fin(MgImpl* mg) {
    MgFin fin;
    fin.ticket = fin_ticket(mg);
    fin.sc = reinterpret_cast<double*>(mg->ws + mg->off_scalars);
    fin.vol = (double)mg->lev[0].vol;
    return fin;
}

// the vector transfers between levels l and l + 1: exact halving in every direction,
// fine nx divisible by 4, and the z chunk of each kernel dividing its extent
static inline bool v4_restrict(const MgImpl* mg, const MgGeom& gf, const MgGeom& gc, int rzc) {
    if (!mg->vec4 || gf.n[2] % 4 != 0 || gc.n[0] % rzc != 0) return false;
    for (int k = 0; k < 3; ++k)
        if (gf.n[k] != 2 * gc.n[k]) return false;
    return true;
}
static inline bool v4_prolong(const MgImpl* mg, const MgGeom& gf, const MgGeom& gc, int pzc) {
    if (!mg->vec4 || gf.n[2] % 4 != 0 || gf.n[0] % pzc != 0) return false;
    for (int k = 0; k < 3; ++k)
        if (gf.n[k] != 2 * gc.n[k]) return false;
    return true;
}

// launches of the MODE-0 vector half-sweep and of the vector transfers with a z chunk
// chosen at run time
template <bool BAT>
static void launch_jacobi_v4_0(int zc, dim3 grd, cudaStream_t st, const MgGeom& g, const float* in, const float* b,
                               float* out, float om, const Bat& bt) {
    if (zc == 1)
        k_mg_jacobi_v4<0, BAT, 1><<<grd, kBlk, 0, st>>>(g, in, b, out, om, nullptr, nullptr, nullptr, nullptr, bt);
    else if (zc == 2)
        k_mg_jacobi_v4<0, BAT, 2><<<grd, kBlk, 0, st>>>(g, in, b, out, om, nullptr, nullptr, nullptr, nullptr, bt);
    else
        k_mg_jacobi_v4<0, BAT, 4><<<grd, kBlk, 0, st>>>(g, in, b, out, om, nullptr, nullptr, nullptr, nullptr, bt);
}
// the last half-sweep of the mixed V-cycle, which adds the correction to the float pairs
template <bool BAT>
static void launch_jacobi_v4_1(int zc, dim3 grd, cudaStream_t st, const MgGeom& g, const float* in, const float* b,
                               float* out, float om, float2* pdf, const Bat& bt) {
    if (zc == 1)
        k_mg_jacobi_v4<1, BAT, 1><<<grd, kBlk, 0, st>>>(g, in, b, out, om, pdf, nullptr, nullptr, nullptr, bt);
    else
        k_mg_jacobi_v4<1, BAT, V4_ZC><<<grd, kBlk, 0, st>>>(g, in, b, out, om, pdf, nullptr, nullptr, nullptr, bt);
}
template <bool BAT>
static void launch_restrict_v4(int rzc, dim3 grd, cudaStream_t st, const MgGeom& gf, const float* xf, const float* bf,
                               const MgGeom& gc, float* bc, float* yc, float om, const Bat& bt) {
    if (rzc == 1)
        k_mg_restrict_v4<BAT, 1><<<grd, kBlk, 0, st>>>(gf, xf, bf, gc, bc, yc, om, bt);
    else
        k_mg_restrict_v4<BAT, MG_RZC><<<grd, kBlk, 0, st>>>(gf, xf, bf, gc, bc, yc, om, bt);
}
template <bool BAT>
static void launch_prolong_v4(int pzc, dim3 grd, cudaStream_t st, const MgGeom& gf, float* xf, const MgGeom& gc,
                              const float* xc, const Bat& bt) {
    if (pzc == 2)
        k_mg_prolong_v4<BAT, 2><<<grd, kBlk, 0, st>>>(gf, xf, gc, xc, bt);
    else
        k_mg_prolong_v4<BAT, V4_ZC><<<grd, kBlk, 0, st>>>(gf, xf, gc, xc, bt);
}

static inline MgGeom mgg(const MgImpl* mg, int l) {
    MgGeom g;
    for (int k = 0; k < 3; ++k) { g.n[k] = mg->lev[l].n[k]; g.per[k] = mg->per[k]; }
    // compute_diag (operators.f90:454-484): idiag = 1/diag where diag > 0, times the
    // smoother's damping omega (one multiplication less per cell and half-sweep)
    g.idiag[0] = 0.0;
    for (int k = 1; k < 8; ++k) g.idiag[k] = mg->omega / (double)k;
    // compute_Pcoef (operators.f90:423-452): Pcoef = 1/(prolongation of the coarse mask)
    for (int bits = 0; bits < 8; ++bits) {
        const int W = (3 + (bits & 1)) * (3 + ((bits >> 1) & 1)) * (3 + ((bits >> 2) & 1));
        g.pcoef[bits] = 1.0 / (double)W;
    }
    for (int k = 0; k < 8; ++k) {
        g.fidiag[k] = (float)g.idiag[k];
        g.fpcoef[k] = (float)g.pcoef[k];
    }
    return g;
}
static inline bool empty(const MgImpl* mg, int l) { return mg->lev[l].vol == 0; }

template <typename T>
static T* lvp(MgImpl* mg, int l, int var) {
    size_t off = var == 1 ? mg->lev[l].off_x : (var == 2 ? mg->lev[l].off_b : mg->lev[l].off_y);
    return reinterpret_cast<T*>(mg->ws + off);
}

void* mg_level_ptr(MgImpl* mg, int lev, int var) {
    if (!mg->ws || lev < 1 || lev > mg->nlevels) return nullptr;
    if (lev == 1 && mg->precision == NYLES_MIXED) {
        if (var == 1) return reinterpret_cast<char*>(mg_pdf(mg));
        if (var == 2) return mg->ws + mg->off_bdf;
    }
    size_t off = var == 1 ? mg->lev[lev - 1].off_x : (var == 2 ? mg->lev[lev - 1].off_b : mg->lev[lev - 1].off_y);
    return mg->ws + off;
}

float2* mg_pdf(MgImpl* mg) {
    return reinterpret_cast<float2*>(mg->ws + mg->off_pdf + (size_t)mg->cur_sol * mg->sol_bytes);
}
// the solutions before the current one (history arrays, h = 1..MG_HIST) and the
// current solution's count
static float2* mg_pdf_old(MgImpl* mg, int h) {
    return reinterpret_cast<float2*>(mg->ws + mg->off_pdf + (size_t)(h * mg->nsol + mg->cur_sol) * mg->sol_bytes);
}
static int* mg_hist_count(MgImpl* mg) { return reinterpret_cast<int*>(mg->ws + mg->off_hist) + mg->cur_sol; }

// non-empty levels from l0 on, and their extents
static int bottom_extents(const MgImpl* mg, int l0, int (*n)[3]) {
    int k = 0;
    for (; l0 + k < mg->nlevels && !empty(mg, l0 + k); ++k)
        for (int i = 0; i < 3; ++i) n[k][i] = mg->lev[l0 + k].n[i];
    return k;
}
// The largest level of the cluster kernel, and the largest that block 0 holds alone. Measured (us): FP32
// up to 4096 / 14000 / 32768 cells: a 256 x 256 x 128 solve 1670 / 1665 / 1648, ten steps of eight 64^3
// runs 19300 / 19370 / 18410; block 0 alone up to 512 / 1024 / 2048 cells of a 48^3 step 1232 / 1232 / 1289.
// FP64 up to 1024 / 2048 / 4096 / 8192 cells: a 128^3 solve 1408 / 1409 / 1356 / 1304-1370, a 64 x 32 x 32
// step 1438 / 1438 / 1437 / 1599; block 0 alone up to 256 / 1024 cells 1438 / 1515.
static long long bottom_maxvol(int precision) { return precision == NYLES_MIXED ? 1 << 15 : 1 << 12; }
static long long bottom_solo(int precision) { return precision == NYLES_MIXED ? 1024 : 256; }

// mg_setup.f90:225-307 (create_hierarchy) for one rank. The reference leaves the loop
// only when x == 2 or y == 2; here coarsening also stops before an odd extent, so
// 3*2^n sizes terminate (the reference does not terminate on them).

int mg_init(MgImpl* mg, int nx, int ny, int nz, int topology, int precision, int nsol, int nhist) {
    if (nhist < 0 || nhist > MG_HIST) { set_error("multigrid: history depth out of range"); return NYLES_BAD_ARG; }
    if (nx < 2 || ny < 2 || nz < 1) { set_error("multigrid: grid too small"); return NYLES_BAD_ARG; }
    if (topology < 1 || topology > 6) { set_error("multigrid: bad topology"); return NYLES_BAD_ARG; }
    mg->precision = precision;
    mg->per[2] = (topology == NYLES_MG_XPERIO || topology == NYLES_MG_XYPERIO || topology == NYLES_MG_XYZPERIO);
    mg->per[1] = (topology == NYLES_MG_YPERIO || topology == NYLES_MG_XYPERIO || topology == NYLES_MG_XYZPERIO);
    mg->per[0] = (topology == NYLES_MG_ZPERIO || topology == NYLES_MG_XYZPERIO);
    const int nh = 3;
    int x = nx, y = ny, z = nz + 2 * nh;
    int L = 0;
    while (true) {
        if (L >= 32) { set_error("multigrid: too many levels"); return NYLES_UNSUPPORTED; }
        MgLevelDesc& d = mg->lev[L];
        d.n[0] = z - 2 * nh; d.n[1] = y; d.n[2] = x;
        if (d.n[0] < 0) d.n[0] = 0;
        d.vol = (long long)d.n[0] * d.n[1] * d.n[2];
        ++L;
        if (x == 2 || y == 2) break;
        if ((x % 2) || (y % 2) || x < 4 || y < 4) break;
        x /= 2; y /= 2; z = z / 2 + nh;
    }
    mg->nlevels = L;
    // An odd z extent above the coarsest level makes mgfor's prolongation write a ghost
    // layer (basicoperators.f90:194-229 steps k by 2 up to nz-nh); not supported.
    for (int l = 0; l + 1 < L; ++l)
        if (mg->lev[l].n[0] % 2) { set_error("multigrid: z extent must stay even above the coarsest level"); return NYLES_UNSUPPORTED; }
    if (mg->lev[0].n[0] < 1) { set_error("multigrid: empty grid"); return NYLES_BAD_ARG; }
    // workspace layout
    const size_t es = precision == NYLES_MIXED ? sizeof(float) : sizeof(double);
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
    for (int l = 0; l < L; ++l) {
        MgLevelDesc& d = mg->lev[l];
        d.off_x = take(d.vol * es);
        d.off_b = take(d.vol * es);
        d.off_y = take(d.vol * es);
    }
    if (precision == NYLES_MIXED) {
        mg->nsol = nsol < 1 ? 1 : nsol;
        mg->cur_sol = 0;
        mg->sol_bytes = (mg->lev[0].vol * sizeof(float2) + 255) & ~(size_t)255;
        mg->nhist = nhist;
        mg->extrap = 0;
        mg->off_pdf = take(mg->sol_bytes * mg->nsol * (1 + nhist));
        if (nhist) mg->off_hist = take(mg->nsol * sizeof(int));
        mg->off_bdf = take(mg->lev[0].vol * sizeof(float2));
        mg->off_fp = take(mg->lev[0].vol * sizeof(float));
        mg->off_fq = take(mg->lev[0].vol * sizeof(float));
    }
    // the coarsest levels (two at least, never level 0), up to bottom_maxvol cells, whose slabs
    // fit in a block's shared memory, run as one k_mg_bottom launch per V-cycle
    mg->bottom = L;
    mg->bottom_smem = 0;
    {
        for (int l = L - 2; l >= 1 && L - l <= MG_BOTTOM_MAXLEV; --l) {
            if (mg->lev[l].vol > bottom_maxvol(precision)) break;
            int n[MG_BOTTOM_MAXLEV][3];
            const size_t bytes = (size_t)bottom_plan(n, bottom_extents(mg, l, n), bottom_solo(precision), BT_THREADS, nullptr,
                                                     nullptr) * es;
            if (bytes > MG_BOTTOM_SMEM) break;
            mg->bottom = l;
            mg->bottom_smem = bytes;
        }
        if (mg->bottom < L) {
            auto smem = [](auto kernel) {
                return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MG_BOTTOM_SMEM);
            };
            const bool f32 = precision == NYLES_MIXED;
            cudaError_t e = f32 ? smem(k_mg_bottom<float, BT_THREADS>) : smem(k_mg_bottom<double, BT_THREADS>);
            if (e == cudaSuccess) e = f32 ? smem(k_mg_bottom<float, BT_MAXTHREADS>) : smem(k_mg_bottom<double, BT_MAXTHREADS>);
            if (e != cudaSuccess) return cuda_status(e, "multigrid coarse-level kernel attribute");
        }
    }
    // one partial per block of the largest reduction grid (the float-pair residual's)
    const dim3 g0 = grid_zc(mg->lev[0].n, MG_DFZC < MG_ZC ? MG_DFZC : MG_ZC);
    mg->npartial = (int)(g0.x * g0.y * g0.z);
    {
        const char* e = getenv("NYLES_GB300_SCALAR_KERNELS");
        mg->vec4 = !(e && e[0] == '1');
        const char* c = getenv("NYLES_GB300_COARSE_ZC");
        const int czc = c ? atoi(c) : 1;
        mg->czc = (czc == 2 || czc == 4) ? czc : 1;
    }
    mg->off_partial = take(mg->npartial * sizeof(double));
    mg->off_partial2 = take(mg->npartial * sizeof(double));
    mg->off_scalars = take(16 * sizeof(double));
    mg->off_ticket = take(64);
    mg->bytes = off;
    return NYLES_OK;
}

// smoothing of level l: half-sweeps x -> y -> x; with from_y the first one was already
// written into y by the kernel that set b from a zero solution. The last half-sweep
// runs in `last_mode` (k_mg_jacobi: 0 store, 1 add to the float-pair solution, 2 store
// and sum its dot product with the Krylov vector q).
template <typename T>
static void smooth(MgImpl* mg, int l, cudaStream_t st, int last_mode, bool from_y = false) {
    if (empty(mg, l)) return;
    MgGeom g = mgg(mg, l);
    const dim3 grd = grid_zc(g.n, MG_ZC);
    T* x = lvp<T>(mg, l, 1);
    T* b = lvp<T>(mg, l, 2);
    T* y = lvp<T>(mg, l, 3);
    const T om = T(mg->omega);
    ProfScope ps(mg->prof, 8, st);
    note_launch(from_y ? 1 : 2);
    if constexpr (sizeof(T) == sizeof(double)) {   // FP64: always stored (last_mode 0)
        const int zc = fp64_zc(mg, l);
        if (zc == 0) {
            const dim3 gx = grid_zc(g.n, FX_ZC);
            if (!from_y) k_mg_fx<FX_ZC, 0><<<gx, kBlk, 0, st>>>(g, x, b, y, nullptr, g, nullptr);
            k_mg_fx<FX_ZC, 0><<<gx, kBlk, 0, st>>>(g, y, b, x, nullptr, g, nullptr);
        } else if (zc == MG_ZC) {
            if (!from_y) k_mg_jacobi<T, 0><<<grd, kBlk, 0, st>>>(g, x, b, y, om, nullptr, nullptr, nullptr, nullptr);
            k_mg_jacobi<T, 0><<<grd, kBlk, 0, st>>>(g, y, b, x, om, nullptr, nullptr, nullptr, nullptr);
        } else {
            const dim3 gs = grid_zc(g.n, 1);
            if (!from_y) k_mg_jacobi<T, 0, false, 1><<<gs, kBlk, 0, st>>>(g, x, b, y, om, nullptr, nullptr, nullptr, nullptr);
            k_mg_jacobi<T, 0, false, 1><<<gs, kBlk, 0, st>>>(g, y, b, x, om, nullptr, nullptr, nullptr, nullptr);
        }
    } else {
        if (mg->bat.tab) {   // batched (stationary mixed refinement): modes 0 and 1
            const Bat& bt = mg->bat;
            float2* pdf = last_mode == 1 ? mg_pdf(mg) : nullptr;
            if constexpr (sizeof(T) == sizeof(float)) {
                const int zc = lvl_zc(mg, l);
                if (use_v4(mg, g.n, zc)) {
                    const dim3 gv = bgrid(mg, grid_v4(g.n, zc));
                    if (!from_y) launch_jacobi_v4_0<true>(zc, gv, st, g, x, b, y, om, bt);
                    if (last_mode == 1)
                        launch_jacobi_v4_1<true>(zc, gv, st, g, y, b, x, om, pdf, bt);
                    else
                        launch_jacobi_v4_0<true>(zc, gv, st, g, y, b, x, om, bt);
                    return;
                }
            }
            const dim3 gb = bgrid(mg, grd);
            if (!from_y) k_mg_jacobi<T, 0, true><<<gb, kBlk, 0, st>>>(g, x, b, y, om, nullptr, nullptr, nullptr, nullptr, bt);
            if (last_mode == 1)
                k_mg_jacobi<T, 1, true><<<gb, kBlk, 0, st>>>(g, y, b, x, om, pdf, nullptr, nullptr, nullptr, bt);
            else
                k_mg_jacobi<T, 0, true><<<gb, kBlk, 0, st>>>(g, y, b, x, om, nullptr, nullptr, nullptr, nullptr, bt);
            return;
        }
        if constexpr (sizeof(T) == sizeof(float)) {
            const int zc = last_mode == 2 ? V4_ZC : lvl_zc(mg, l);
            if (last_mode == 2 ? use_v4_sums(mg) : use_v4(mg, g.n, zc)) {
                const dim3 gv = grid_v4(g.n, zc);
                if (!from_y) launch_jacobi_v4_0<false>(zc, gv, st, g, x, b, y, om, Bat());
                if (last_mode == 1)
                    launch_jacobi_v4_1<false>(zc, gv, st, g, y, b, x, om, mg_pdf(mg), Bat());
                else if (last_mode == 2) {   // also beta and the mean of z for the Krylov update
                    MgFin fin;
                    fin.ticket = fin_ticket(mg);
                    fin.sc = reinterpret_cast<double*>(mg->ws + mg->off_scalars);
                    fin.k = mg->fcg_k;
                    fin.vol = (double)mg->lev[0].vol;
                    const float* q = reinterpret_cast<const float*>(mg->ws + mg->off_fq);
                    double* part = partials(mg, 0, blocks(gv));
                    double* part2 = partials(mg, 1, blocks(gv));
                    k_mg_jacobi_v4<2><<<gv, kBlk, 0, st>>>(g, y, b, x, om, nullptr, q, part, part2, Bat(), fin);
                }
                else
                    launch_jacobi_v4_0<false>(zc, gv, st, g, y, b, x, om, Bat());
                return;
            }
        }
        if (!from_y) k_mg_jacobi<T, 0><<<grd, kBlk, 0, st>>>(g, x, b, y, om, nullptr, nullptr, nullptr, nullptr);
        if (last_mode == 1)
            k_mg_jacobi<T, 1><<<grd, kBlk, 0, st>>>(g, y, b, x, om, mg_pdf(mg),
                                                    nullptr, nullptr, nullptr);
        else if (last_mode == 2)
            k_mg_jacobi<T, 2><<<grd, kBlk, 0, st>>>(g, y, b, x, om, nullptr,
                                                    reinterpret_cast<const T*>(mg->ws + mg->off_fq),
                                                    reinterpret_cast<double*>(mg->ws + mg->off_partial),
                                                    reinterpret_cast<double*>(mg->ws + mg->off_partial2));
        else
            k_mg_jacobi<T, 0><<<grd, kBlk, 0, st>>>(g, y, b, x, om, nullptr, nullptr, nullptr, nullptr);
    }
}

// solvers.f90:35-55
// levels mg->bottom..L-1 of the V-cycle in one cluster of blocks (k_mg_bottom)
template <typename T>
static void bottom(MgImpl* mg, cudaStream_t st) {
    const int l0 = mg->bottom;
    if (empty(mg, l0)) return;
    const MgGeom g0 = mgg(mg, l0);
    MgBottom<T> a;
    for (int k = 0; k < 3; ++k) a.per[k] = mg->per[k];
    for (int k = 0; k < 8; ++k) {
        a.idiag[k] = sizeof(T) == sizeof(float) ? T(g0.fidiag[k]) : T(g0.idiag[k]);
        a.pcoef[k] = sizeof(T) == sizeof(float) ? T(g0.fpcoef[k]) : T(g0.pcoef[k]);
    }
    int n[MG_BOTTOM_MAXLEV][3];
    a.nlev = bottom_extents(mg, l0, n);
    long long few = 0, many = 0;
    const long long solo = bottom_solo(mg->precision);
    bottom_plan(n, a.nlev, solo, BT_THREADS, nullptr, &few);
    bottom_plan(n, a.nlev, solo, BT_MAXTHREADS, nullptr, &many);
    const bool wide = many < few && mg->bat.nrun <= 8;
    bottom_plan(n, a.nlev, solo, wide ? BT_MAXTHREADS : BT_THREADS, a.lev, nullptr);
    a.resmooth = l0 + a.nlev < mg->nlevels;
    a.xg = lvp<T>(mg, l0, 1);
    a.bg = lvp<T>(mg, l0, 2);
    ProfScope ps(mg->prof, 8, st);
    note_launch();
    const dim3 grd = bgrid(mg, dim3(BT_CTAS, 1, 1));
    if (wide) k_mg_bottom<T, BT_MAXTHREADS><<<grd, BT_MAXTHREADS, mg->bottom_smem, st>>>(a, mg->bat);
    else k_mg_bottom<T, BT_THREADS><<<grd, BT_THREADS, mg->bottom_smem, st>>>(a, mg->bat);
}

// level0_last: mode of the last level-0 half-sweep (see smooth)
template <typename T>
static void vcycle(MgImpl* mg, cudaStream_t st, int level0_last) {
    const int L = mg->nlevels;
    const int B = mg->bottom;   // < L: levels B..L-1 in one cluster
    // The first half-sweep of level 0 was written by the stop-test residual kernel that
    // precedes every V-cycle (k_mg_resid_sweep; mixed: k_mg_resid_df, from a zero
    // correction); every restricted level gets it from the restriction.
    for (int l = 0; l < L - 1 && l < B; ++l) {
        smooth<T>(mg, l, st, 0, true);
        if (!empty(mg, l + 1)) {
            MgGeom gf = mgg(mg, l), gc = mgg(mg, l + 1);
            ProfScope ps(mg->prof, 9, st);
            note_launch();
            bool done = false;
            if constexpr (sizeof(T) == sizeof(float)) {
                const int rzc = lvl_rzc(mg, l);
                if (v4_restrict(mg, gf, gc, rzc)) {
                    const dim3 gv = grid_v4_restrict(gf, gc, rzc);
                    if (mg->bat.tab)
                        launch_restrict_v4<true>(rzc, bgrid(mg, gv), st, gf, lvp<float>(mg, l, 1), lvp<float>(mg, l, 2), gc,
                                                 lvp<float>(mg, l + 1, 2), lvp<float>(mg, l + 1, 3), (float)mg->omega,
                                                 mg->bat);
                    else
                        launch_restrict_v4<false>(rzc, gv, st, gf, lvp<float>(mg, l, 1), lvp<float>(mg, l, 2), gc,
                                                  lvp<float>(mg, l + 1, 2), lvp<float>(mg, l + 1, 3), (float)mg->omega,
                                                  Bat());
                    done = true;
                }
            }
            if constexpr (sizeof(T) == sizeof(double)) {
                const int zc = fp64_zc(mg, l);
                if (zc == 0)
                    k_mg_fx<FX_ZC, 2><<<grid_zc(gf.n, FX_ZC), kBlk, 0, st>>>(gf, lvp<T>(mg, l, 1), lvp<T>(mg, l, 2),
                                                                            lvp<T>(mg, l + 1, 3), nullptr, gc,
                                                                            lvp<T>(mg, l + 1, 2));
                else if (zc == MG_ZC)
                    k_mg_restrict<T><<<grid_zc(gc.n, MG_RZC), kBlk, 0, st>>>(
                        gf, lvp<T>(mg, l, 1), lvp<T>(mg, l, 2), gc, lvp<T>(mg, l + 1, 2), lvp<T>(mg, l + 1, 3),
                        T(mg->omega));
                else
                    k_mg_restrict<T, false, 1><<<grid_zc(gc.n, 1), kBlk, 0, st>>>(
                        gf, lvp<T>(mg, l, 1), lvp<T>(mg, l, 2), gc, lvp<T>(mg, l + 1, 2), lvp<T>(mg, l + 1, 3),
                        T(mg->omega));
            } else if (!done && mg->bat.tab)
                k_mg_restrict<T, true><<<bgrid(mg, grid_zc(gc.n, MG_RZC)), kBlk, 0, st>>>(
                    gf, lvp<T>(mg, l, 1), lvp<T>(mg, l, 2), gc, lvp<T>(mg, l + 1, 2), lvp<T>(mg, l + 1, 3),
                    T(mg->omega), mg->bat);
            else if (!done)
                k_mg_restrict<T><<<grid_zc(gc.n, MG_RZC), kBlk, 0, st>>>(gf, lvp<T>(mg, l, 1), lvp<T>(mg, l, 2), gc,
                                                                        lvp<T>(mg, l + 1, 2), lvp<T>(mg, l + 1, 3),
                                                                        T(mg->omega));
        }
    }
    if (B < L)
        bottom<T>(mg, st);
    else
        smooth<T>(mg, L - 1, st, L == 1 ? level0_last : 0, true);
    for (int l = (B < L ? B - 1 : L - 2); l >= 0; --l) {
        if (!empty(mg, l + 1)) {
            MgGeom gf = mgg(mg, l), gc = mgg(mg, l + 1);
            ProfScope ps(mg->prof, 10, st);
            note_launch();
            bool done = false;
            if constexpr (sizeof(T) == sizeof(float)) {
                const int pzc = lvl_pzc(mg, l);
                if (v4_prolong(mg, gf, gc, pzc)) {
                    if (mg->bat.tab)
                        launch_prolong_v4<true>(pzc, bgrid(mg, grid_v4(gf.n, pzc)), st, gf, lvp<float>(mg, l, 1), gc,
                                                lvp<float>(mg, l + 1, 1), mg->bat);
                    else
                        launch_prolong_v4<false>(pzc, grid_v4(gf.n, pzc), st, gf, lvp<float>(mg, l, 1), gc,
                                                 lvp<float>(mg, l + 1, 1), Bat());
                    done = true;
                }
            }
            if constexpr (sizeof(T) == sizeof(double)) {
                const int zc = fp64_zc(mg, l);
                const double* xc = lvp<T>(mg, l + 1, 1);
                double* xf = lvp<T>(mg, l, 1);
                const dim3 g8 = grid_zc(gc.n, 8);
                if (zc == 1)
                    k_mg_prolong_f64<1><<<grid_zc(gc.n, 1), kBlk, 0, st>>>(gf, xf, gc, xc);
                else if (zc == MG_ZC)   // (narrow levels: one fine column per thread)
                    k_mg_prolong<T><<<grid_zc(gf.n, MG_ZC), kBlk, 0, st>>>(gf, xf, gc, xc);
                else if (blocks(g8) >= 4 * 152)   // enough columns for 8 coarse planes per thread, or 4
                    k_mg_prolong_f64<8><<<g8, kBlk, 0, st>>>(gf, xf, gc, xc);
                else
                    k_mg_prolong_f64<4><<<grid_zc(gc.n, 4), kBlk, 0, st>>>(gf, xf, gc, xc);
            } else if (!done && mg->bat.tab)
                k_mg_prolong<T, true><<<bgrid(mg, grid_zc(gf.n, MG_ZC)), kBlk, 0, st>>>(
                    gf, lvp<T>(mg, l, 1), gc, lvp<T>(mg, l + 1, 1), mg->bat);
            else if (!done)
                k_mg_prolong<T><<<grid_zc(gf.n, MG_ZC), kBlk, 0, st>>>(gf, lvp<T>(mg, l, 1), gc, lvp<T>(mg, l + 1, 1));
        }
        smooth<T>(mg, l, st, l == 0 ? level0_last : 0);
    }
}

static int read_scalar(MgImpl* mg, double* host_out, cudaStream_t st) {
    double* out = reinterpret_cast<double*>(mg->ws + mg->off_scalars);
    cudaError_t e = cudaMemcpyAsync(host_out, out, sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return cuda_status(e, "multigrid norm");
}

static double* scalars(MgImpl* mg) { return reinterpret_cast<double*>(mg->ws + mg->off_scalars); }

// enqueue sum(v^2) of level 0 into *out
static void enqueue_sumsq(MgImpl* mg, const MgGeom& g, const double* v, double* out, cudaStream_t st) {
    double* part = reinterpret_cast<double*>(mg->ws + mg->off_partial);
    const dim3 grd = grid_zc(g.n, MG_ZC);
    ProfScope ps(mg->prof, 11, st);
    const bool few = blocks(grd) <= 1024;   // (256^3, 8192 blocks: 74 us with the ticket, 59 + 7 with the sum apart)
    note_launch(few ? 1 : 2);
    k_mg_sumsq<<<grd, kBlk, 0, st>>>(g, v, part, few ? mg_fin(mg) : MgFin(), out);
    if (!few) k_mg_final<<<1, 1024, 0, st>>>(part, (int)blocks(grd), out);
}

// mixed precision: enqueue sum(b^2) of the float-pair right-hand side into
// sc[SC_NORMB] and the scale of the residual sums
static void enqueue_normb_df(MgImpl* mg, cudaStream_t st) {
    MgGeom g = mgg(mg, 0);
    double* part = reinterpret_cast<double*>(mg->ws + mg->off_partial);
    // planes per thread: enough that the block sums (FP64 too) do not count, where the blocks still
    // fill the chip twice
    int zc = MG_ZC;
    while (zc < 64 && blocks(grid_zc(g.n, 2 * zc)) >= 2 * 8 * 152) zc *= 2;
    const dim3 grd = grid_zc(g.n, zc);
    ProfScope ps(mg->prof, 11, st);
    note_launch(1);
    k_mg_sumsq_df<<<bgrid(mg, grd), kBlk, 0, st>>>(g, reinterpret_cast<const float2*>(mg->ws + mg->off_bdf), part,
                                                   mg_fin(mg), zc, mg->bat);
}

// mixed precision: enqueue the float-pair residual (also the next correction's rhs)
// and its sum of squares into sc[SC_RR]
static void enqueue_resid_df(MgImpl* mg, cudaStream_t st) {
    MgGeom g = mgg(mg, 0);
    double* sc = reinterpret_cast<double*>(mg->ws + mg->off_scalars);
    const bool v4 = use_v4_sums(mg);
    const dim3 grd = v4 ? grid_v4(g.n) : grid_zc(g.n, MG_DFZC);
    double* part = partials(mg, 0, blocks(grd));
    ProfScope ps(mg->prof, 11, st);
    note_launch(v4 ? 1 : 2);
    const float2* pdf = mg_pdf(mg);
    const float2* bdf = reinterpret_cast<const float2*>(mg->ws + mg->off_bdf);
    MgFin fin;   // the vector kernel also adds the partials into sc[SC_RR]
    fin.ticket = fin_ticket(mg);
    fin.sc = sc;
    float* b = lvp<float>(mg, 0, 2);
    float* y = lvp<float>(mg, 0, 3);
    const float om = (float)mg->omega;
    const dim3 gb = bgrid(mg, grd);
    if (v4) {
        if (mg->bat.tab)
            k_mg_resid_df_v4<true><<<gb, kBlk, 0, st>>>(g, pdf, bdf, b, y, om, sc, part, mg->bat, fin);
        else
            k_mg_resid_df_v4<<<grd, kBlk, 0, st>>>(g, pdf, bdf, b, y, om, sc, part, Bat(), fin);
    } else if (mg->bat.tab) {
        k_mg_resid_df<true><<<gb, kBlk, 0, st>>>(g, pdf, bdf, b, y, om, sc, part, mg->bat);
    } else {
        k_mg_resid_df<<<grd, kBlk, 0, st>>>(g, pdf, bdf, b, y, om, sc, part);
    }
    if (!v4)
        k_mg_final<<<bgrid(mg, dim3(1, 1, 1)), 1024, 0, st>>>(part, (int)(grd.x * grd.y * grd.z), sc + SC_RR, mg->bat);
}

// FP64: enqueue the stop-test sum(r^2) into sc[SC_RR] together with the next V-cycle's
// first level-0 half-sweep (k_mg_resid_sweep)
static void enqueue_resid_sweep(MgImpl* mg, cudaStream_t st) {
    MgGeom g = mgg(mg, 0);
    const int zc = fp64_zc(mg, 0);
    const bool fx = zc == 0, one = zc == 1 && partials_fit(mg, blocks(grid_zc(g.n, 1)));
    const dim3 grd = grid_zc(g.n, fx ? FX_ZC : (one ? 1 : MG_ZC));
    double* part = partials(mg, 0, blocks(grd));
    ProfScope ps(mg->prof, 11, st);
    const bool apart = fx || (!one && blocks(grd) > 1024);   // the sum (as enqueue_sumsq)
    const MgFin fin = apart ? MgFin() : mg_fin(mg);
    note_launch(apart ? 2 : 1);
    const double *x = lvp<double>(mg, 0, 1), *b = lvp<double>(mg, 0, 2);
    double* y = lvp<double>(mg, 0, 3);
    if (fx)   // (many blocks: the ticket took 30 us of a 128^3 level against 20 + 4.5 with the sum apart)
        k_mg_fx<FX_ZC, 1><<<grd, kBlk, 0, st>>>(g, x, b, y, part, g, nullptr);
    else if (one)
        k_mg_resid_sweep<double, 1><<<grd, kBlk, 0, st>>>(g, x, b, y, mg->omega, part, fin);
    else
        k_mg_resid_sweep<double><<<grd, kBlk, 0, st>>>(g, x, b, y, mg->omega, part, fin);
    if (apart)
        k_mg_final<<<1, 1024, 0, st>>>(part, (int)blocks(grd), reinterpret_cast<double*>(mg->ws + mg->off_scalars) + SC_RR);
}

// mixed precision with krylov: after the V-cycle left z = V(r) in level 0's x (and the
// partial sums of z.q), one FCG(1) update of the direction p and q = A p, and
// x += alpha p on the float-pair solution (k: iteration of this solve, or -1 to read it
// on the device)
static void enqueue_fcg_update(MgImpl* mg, cudaStream_t st, int k) {
    MgGeom g = mgg(mg, 0);
    double* sc = scalars(mg);
    float* z = lvp<float>(mg, 0, 1);
    float* r = lvp<float>(mg, 0, 2);
    float* P = reinterpret_cast<float*>(mg->ws + mg->off_fp);
    float* Q = reinterpret_cast<float*>(mg->ws + mg->off_fq);
    const long long n = mg->lev[0].vol;
    const bool v4 = use_v4_sums(mg);
    const dim3 grd = v4 ? grid_v4(g.n) : grid_zc(g.n, MG_ZC);
    const int nb = (int)blocks(grd);
    double* part = partials(mg, 0, nb);
    double* part2 = partials(mg, 1, nb);
    const unsigned eb = (unsigned)((n + 255) / 256);
    ProfScope ps(mg->prof, 11, st);
    if (v4) {
        // beta came with the V-cycle's last level-0 half-sweep (k_mg_jacobi_v4<2>); the
        // direction kernel also sets alpha
        note_launch(1);
        MgFin fin;
        fin.ticket = fin_ticket(mg);
        fin.sc = sc;
        k_fcg_direction_v4<<<grd, kBlk, 0, st>>>(g, z, r, P, Q, sc, part, part2, fin);
    } else {
        // the partial sums of z.q and z were written by the V-cycle's last level-0 half-sweep
        note_launch(3);
        k_fcg_final_beta<<<1, 1024, 0, st>>>(part, part2, nb, (double)n, sc, k);
        k_fcg_direction<<<grd, kBlk, 0, st>>>(g, z, r, P, Q, sc, part, part2);
        k_fcg_final_alpha<<<1, 1024, 0, st>>>(part, part2, nb, sc);
    }
    note_launch(1);
    k_fcg_xupdate<<<eb, 256, 0, st>>>(mg_pdf(mg), P, n, sc);
}

static int sumsq(MgImpl* mg, const MgGeom& g, const double* v, double* host_out, cudaStream_t st) {
    enqueue_sumsq(mg, g, v, scalars(mg), st);
    return read_scalar(mg, host_out, st);
}

static int read_slot(MgImpl* mg, int slot, double* host_out, cudaStream_t st) {
    cudaError_t e = cudaMemcpyAsync(host_out, scalars(mg) + slot, sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return cuda_status(e, "multigrid norm");
}

// A non-finite norm means a non-finite right-hand side or solution: the solve stops
// at once with NYLES_BLOWUP (the stop rule alone would either accept it, since a NaN
// norm of b skips the iteration, or run to maxite on NaN residuals).
static bool finite_norm(double v) { return v == v && v <= 1.7976931348623157e308; }

static int blowup(MgImpl* mg, int nite, double res, const char* what) {
    mg->stats.nite = nite;
    mg->stats.res = res;
    mg->stats.solves += 1;
    mg->stats.vcycles += nite;
    mg->stats.nonfinite += 1;
    set_error(std::string("multigrid: non-finite ") + what + " (blow-up)");
    return NYLES_BLOWUP;
}

// extrapolated start of the next mixed solve (after its right-hand side norm)
static void enqueue_extrapolate(MgImpl* mg, cudaStream_t st) {
    if (!mg->extrap || mg->extrap > mg->nhist) return;
    const long long n = mg->lev[0].vol;
    const unsigned eb = (unsigned)((n + 255) / 256);
    double* sc = scalars(mg);
    note_launch(2);
    HistPtrs hp;
    for (int k = 0; k < MG_HIST; ++k) hp.h[k] = k < mg->nhist ? mg_pdf_old(mg, k + 1) : nullptr;
    k_mg_extrapolate<<<bgrid(mg, dim3(eb, 1, 1)), 256, 0, st>>>(mg_pdf(mg), hp, n, mg->extrap, sc,
                                                                 mg_hist_count(mg), mg->bat);
    k_mg_hist_count<<<1, mg->bat.tab ? NYLES_MAX_BATCH : 1, 0, st>>>(mg_hist_count(mg), sc, mg->bat);
}

// solvers.f90:8-33: stop when sum(r^2)/sum(b^2) < tol or after maxite V-cycles
int mg_solve(MgImpl* mg, cudaStream_t st) {
    if (!mg->ws) { set_error("multigrid: workspace not bound"); return NYLES_BAD_ARG; }
    MgGeom g0 = mgg(mg, 0);
    int nite = 0;
    double normb = 0.0, rr = 0.0, res = 0.0;
    int rc;
    if (mg->precision == NYLES_FP64) {
        double* b = lvp<double>(mg, 0, 2);
        if ((rc = sumsq(mg, g0, b, &normb, st))) return rc;
        if (!finite_norm(normb)) return blowup(mg, 0, normb, "right-hand side");
        if (normb > 0.0) {
            enqueue_resid_sweep(mg, st);
            if ((rc = read_slot(mg, SC_RR, &rr, st))) return rc;
            res = rr / normb;
            if (!finite_norm(res)) return blowup(mg, 0, res, "residual");
        }
        while (true) {
            if (res < mg->tol) break;
            vcycle<double>(mg, st, 0);
            ++nite;
            if (nite >= mg->maxite) break;
            if (normb > 0.0) {
                enqueue_resid_sweep(mg, st);
                if ((rc = read_slot(mg, SC_RR, &rr, st))) return rc;
                res = rr / normb;
                if (!finite_norm(res)) return blowup(mg, nite, res, "residual");
            } else {
                res = 0.0;
            }
        }
    } else {
        enqueue_normb_df(mg, st);
        enqueue_extrapolate(mg, st);
        if ((rc = read_slot(mg, SC_NORMB, &normb, st))) return rc;
        if (!finite_norm(normb)) return blowup(mg, 0, normb, "right-hand side");
        if (normb > 0.0) {
            enqueue_resid_df(mg, st);
            if ((rc = read_slot(mg, SC_RR, &rr, st))) return rc;
            res = rr / normb;
            if (!finite_norm(res)) return blowup(mg, 0, res, "residual");
        }
        while (true) {
            if (res < mg->tol) break;
            if (mg->krylov) {              // z = V(r) preconditions an FCG(1) update of p
                mg->fcg_k = nite;
                vcycle<float>(mg, st, 2);
                enqueue_fcg_update(mg, st, nite);
            } else {
                vcycle<float>(mg, st, 1);   // FP32 correction of the residual equation, added to p
            }
            ++nite;
            if (nite >= mg->maxite) break;
            if (normb > 0.0) {
                enqueue_resid_df(mg, st);
                if ((rc = read_slot(mg, SC_RR, &rr, st))) return rc;
                res = rr / normb;
                if (!finite_norm(res)) return blowup(mg, nite, res, "residual");
            } else {
                res = 0.0;
            }
        }
    }
    mg->stats.nite = nite;
    mg->stats.res = res;
    mg->stats.solves += 1;
    mg->stats.vcycles += nite;
    if (res >= mg->tol && nite >= mg->maxite) mg->stats.not_converged += 1;
    return cuda_status(cudaGetLastError(), "multigrid solve");
}

// ---------------------------------------------------------------- graph mode
void GraphBuilder::begin_segment() {
    if (error) return;
    cudaError_t e = cudaStreamBeginCaptureToGraph(st, graph, deps.empty() ? nullptr : deps.data(), nullptr,
                                                  deps.size(), cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) error = cuda_status(e, "cudaStreamBeginCaptureToGraph");
}

void GraphBuilder::end_segment() {
    if (error) return;
    cudaStreamCaptureStatus status;
    const cudaGraphNode_t* d = nullptr;
    size_t n = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(st, &status, nullptr, nullptr, &d, nullptr, &n);
    if (e == cudaSuccess) {
        std::vector<cudaGraphNode_t> frontier(d, d + n);
        cudaGraph_t g = nullptr;
        e = cudaStreamEndCapture(st, &g);
        if (e == cudaSuccess) deps.swap(frontier);
    }
    if (e != cudaSuccess) error = cuda_status(e, "graph segment capture");
}

// The same solve as mg_solve with the stop test on the device: norms and the first
// residual, then a while-node whose body is one V-cycle, the residual norm and the
// control kernel. Called with a segment of gb open; leaves a new segment open.
int mg_solve_graph(MgImpl* mg, GraphBuilder& gb) {
    if (!mg->ws) { set_error("multigrid: workspace not bound"); return NYLES_BAD_ARG; }
    cudaStream_t st = gb.st;
    MgGeom g0 = mgg(mg, 0);
    double* sc = scalars(mg);
    const bool mixed = mg->precision == NYLES_MIXED;
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, gb.graph, 0, 0);
    if (e != cudaSuccess) return gb.error = cuda_status(e, "cudaGraphConditionalHandleCreate");
    if (!mixed) {
        enqueue_sumsq(mg, g0, lvp<double>(mg, 0, 2), sc + SC_NORMB, st);
        enqueue_resid_sweep(mg, st);
    } else {
        enqueue_normb_df(mg, st);
        enqueue_extrapolate(mg, st);
        enqueue_resid_df(mg, st);
    }
    const unsigned nctl = mg->bat.tab ? NYLES_MAX_BATCH : 1;   // one thread per run
    k_mg_ctl_begin<<<1, nctl, 0, st>>>(sc, h, mg->tol, mg->bat);
    note_launch();
    gb.end_segment();
    if (gb.error) return gb.error;
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    e = cudaGraphAddNode(&node, gb.graph, gb.deps.empty() ? nullptr : gb.deps.data(), nullptr, gb.deps.size(), &p);
    if (e != cudaSuccess) return gb.error = cuda_status(e, "cudaGraphAddNode(while)");
    cudaGraph_t body = p.conditional.phGraph_out[0];
    e = cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) return gb.error = cuda_status(e, "capture of the multigrid loop body");
    const long long l0 = nyles_launch_count();
    const int gate0 = mg->bat.gate;
    mg->bat.gate = GATE_LIVE;   // batched: runs whose solve has stopped skip the loop body
    if (!mixed) {
        vcycle<double>(mg, st, 0);
        enqueue_resid_sweep(mg, st);
    } else if (mg->krylov) {
        mg->fcg_k = -1;
        vcycle<float>(mg, st, 2);
        enqueue_fcg_update(mg, st, -1);
        enqueue_resid_df(mg, st);
    } else {
        vcycle<float>(mg, st, 1);
        enqueue_resid_df(mg, st);
    }
    mg->bat.gate = gate0;
    k_mg_ctl_step<<<1, nctl, 0, st>>>(sc, h, mg->tol, mg->maxite, mg->bat);
    note_launch();
    gb.body_kernels = nyles_launch_count() - l0;
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(st, &g);
    if (e != cudaSuccess) return gb.error = cuda_status(e, "end of the multigrid loop body");
    gb.deps.assign(1, node);
    gb.begin_segment();
    return gb.error;
}

int mg_read_device_stats(MgImpl* mg, cudaStream_t st, MgDeviceStats* out) {
    double h[SC_NONFINITE + 1];
    cudaError_t e = cudaMemcpyAsync(h, scalars(mg), sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_status(e, "multigrid statistics read-back");
    out->nite = (int)h[SC_NITE];
    out->res = h[SC_RES];
    out->vcycles = (long long)h[SC_TOTAL];
    out->not_converged = (long long)h[SC_NCONV];
    out->nonfinite = (long long)h[SC_NONFINITE];
    return NYLES_OK;
}

int mg_reset_history(MgImpl* mg) {
    if (!mg->nhist || !mg->ws) return NYLES_OK;
    return cuda_status(cudaMemset(mg->ws + mg->off_hist, 0, mg->nsol * sizeof(int)), "multigrid history reset");
}

int mg_zero_scalars(MgImpl* mg) {
    cudaError_t e = cudaMemset(scalars(mg), 0, 16 * sizeof(double));
    if (e == cudaSuccess) e = cudaMemset(mg->ws + mg->off_ticket, 0, 64);
    if (e == cudaSuccess && mg->nhist) e = cudaMemset(mg->ws + mg->off_hist, 0, mg->nsol * sizeof(int));
    return cuda_status(e, "multigrid scalars reset");
}

}  // namespace nyles
