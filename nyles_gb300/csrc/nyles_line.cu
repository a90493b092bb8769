// FP64 right-hand side, one field and one direction at a time.
//
// GB300 issues FP64 at 1/64 of its FP32 rate (2 lanes per cycle and SM), so the FP64
// right-hand side costs what its FP64 instructions cost; loads, selects, integer work and
// even extra passes over memory run beside them for nothing. The kernel below is built to
// need few of them. A reconstruction has nine uses per cell: the tracer fluxes of b along x, y
// and z, and two vortex-force fluxes per direction (core/vortex_force.py:69-81). Each is
// the same operation on a line of one field, so each is a "task" of k_line: a thread marches
// along its line with everything that neighbouring faces share held in registers:
//  - the first differences D of the line, one subtraction per cell instead of the dozen
//    that the smoothness indicators and candidate values of one face take on their own;
//  - the three smoothness indicators of a stencil. The indicator of a three-point stencil
//    depends on the face's side only through its one-sided slope: right-ended, centred and
//    left-ended forms of a node serve the faces beside it for either sign of the velocity,
//    so they are formed once per node (10 FP64 instructions) and selected.
// Written in differences, the value at the face is s*q0 + (weighted sum of differences),
// with a quotient by series (nyles_div.cuh): its divisor is positive, at least 6e-46 and, with differences
// up to 1e50, within its range.
// 40 FP64 instructions per vortex-force flux and 39 per tracer flux, where one face at a time
// (weno5<double>) takes 77. The registers are read and written once per direction for it
// (33 instead of 12 words per cell), which at 256^3 is 0.7 ms of memory time under 12.6 ms
// of FP64 time.
// Measured against the march that formed every face on its own in 16-cell columns:
// 109 x 75 x 53 with a tracer and viscosity 2.22 -> 0.60 ms; 256^3 23.4 -> 12.6 ms;
// 64 x 32 x 32 (16 blocks then) 1.35 -> 0.19 ms.
#include "nyles_internal.h"
#include "nyles_div.cuh"
#include <algorithm>

namespace nyles {

// The smoothness indicators are carried as d = 4 (beta + eps): with the factor 4 the
// one-sided slopes need no scaling, and a power of two common to all of them drops out of
// the weights exactly.
struct LineK {
    static constexpr double c13 = (double)(1.0f / 3.0f), c76 = (double)(7.0f / 6.0f), c116 = (double)(11.0f / 6.0f);
    static constexpr double c16 = (double)(1.0f / 6.0f), c56 = (double)(5.0f / 6.0f);
    static constexpr double k4 = 4.0 * (double)(13.0f / 12.0f), eps4 = 4.0 * (double)1e-16f;
    // candidate values in differences (core/weno.f90:34-36 with its REAL(4) literals, whose
    // coefficient sums differ from 1 and from each other in the eighth digit): q1 = s1 q0 + ...,
    // q2 = s2 q0 + ..., q3 = s2 q0 + ...; every constant here is exact in double
    static constexpr double s1 = c13 - c76 + c116, s2 = c56 + c13 - c16, ds = s1 - s2;
    static constexpr double g10 = -c13, g11 = c76 - c13;
    static constexpr double g21 = 6.0 * c16, g22 = 6.0 * c13;                // weight 6 included
    static constexpr double g32 = 3.0 * (c56 - c16), g33 = -3.0 * c16;       // weight 3 included
};

// |d1 - d3| rounded through REAL(4) as core/weno.f90:45 does (tau5 is implicitly REAL(4)),
// to nearest even, in integer arithmetic; v carries the factor 4 of the indicators. Beyond
// the float range the result is infinite, as the reference's; below it, where a float
// would be subnormal, the weight 1 + tau/(beta + eps) is 1 either way.
__device__ __forceinline__ double line_tau(double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(fabs(v));
    b += 0x0fffffffull + ((b >> 29) & 1ull);
    b &= ~0x1fffffffull;
    if ((unsigned int)(b >> 32) >= 0x48100000u) b = 0x7ff0000000000000ull;   // 4 * 2^128
    return __longlong_as_double((long long)b);
}

// the node's indicators from the differences on its left and right: left-ended, centred and
// right-ended slope (core/weno.f90:38-43)
__device__ __forceinline__ void line_node(double dl, double dr, double& bl, double& bc, double& br) {
    const double s = dr - dl, c = dr + dl;
    const double r = fma(3.0, dr, -dl), l = fma(-3.0, dl, dr);
    const double k = fma(LineK::k4 * s, s, LineK::eps4);
    bl = fma(l, l, k);
    bc = fma(c, c, k);
    br = fma(r, r, k);
}

// |u| times the upwind WENO5 value, signed: the flux u*q of the face between q0 and q1
// (core/weno.f90:25-54). Differences d0..d4 around the face (d2 = q1 - q0); for u <= 0 the
// mirrored stencil, whose differences change sign: the sign is taken out of the sum.
struct LineFace {
    double d0, d1, d2, d3, d4;   // differences, j-2 .. j+2
    double brm, br0;             // right-ended indicators of nodes j-1, j
    double bc0, bcp;             // centred, j, j+1
    double blp, blq;             // left-ended, j+1, j+2
};
__device__ __forceinline__ double line_flux(const LineFace& f, double u, double q0, double q1) {
    typedef LineK K;
    const bool pos = u > 0.0;
    const double b1 = pos ? f.brm : f.blq, b2 = pos ? f.bc0 : f.bcp, b3 = pos ? f.blp : f.br0;
    const double e0 = pos ? f.d0 : f.d4, e1 = pos ? f.d1 : f.d3, e3 = pos ? f.d3 : f.d1;
    const double qs = pos ? q0 : -q1;
    const double tau = line_tau(b1 - b3);
    // weights w_k = g_k (1 + tau/b_k) times b1 b2 b3: positive terms only
    const double p23 = b2 * b3, p13 = b1 * b3, p12 = b1 * b2, p = p12 * b3;
    const double wa = fma(tau, p23, p), wb = fma(tau, p13, p), wc = fma(tau, p12, p);
    const double den = fma(3.0, wc, fma(6.0, wb, wa));
    const double g1 = fma(K::g11, e1, fma(K::g10, e0, K::ds * qs));
    const double g2 = fma(K::g22, f.d2, K::g21 * e1);
    const double g3 = fma(K::g32, f.d2, K::g33 * e3);
    const double num = fma(wc, g3, fma(wb, g2, wa * g1));
    return fabs(u) * fma(K::s2, qs, div_series(num, den));
}

struct LineTask {
    const double* q;      // the advected field
    const double* U;      // the contravariant velocity along the line
    double* out;
    long long sa;         // vortex force: stride of the direction the velocity is averaged along
    int vortex;           // 0: tracer (out = -(flux divergence)); 1: vortex force (out += sgn * flux)
    int assign;           // tracer: first direction (out is set, not added to)
    double sgn;
    double kd;            // tracer: diffusivity * ids2 of this direction (0: none)
    int lo[3], hi[3];     // cells (z, y, x)
};
constexpr int LINE_TASKS = NYLES_MAX_TR + 3, LINE_THREADS = 128;
struct LineArgs {
    Geom g;
    int d;                // axis of the lines: 0 = z, 1 = y, 2 = x
    int chunk;            // cells per thread
    LineTask t[LINE_TASKS];
};

// the closures near array ends, out of line (walls only)
__device__ __noinline__ double line_tr_closure(const double* __restrict__ q, double u, int i, int n, long long s) {
    auto Q = [&](int k) -> double { return __ldg(q + (long long)k * s); };
    return flux1d_at(i, n, u, Q);
}
__device__ __noinline__ double line_vf_closure(const double* __restrict__ q, double u, int i, int n, long long s) {
    auto Q = [&](int k) -> double { return k == 0 ? 0.0 : __ldg(q + (long long)(k - 1) * s); };
    return flux1d_at(i, n, u, Q);
}

// One thread per line and chunk of a task's box; blockIdx.y = chunk, blockIdx.z = task.
__global__ void __launch_bounds__(LINE_THREADS) k_line(const __grid_constant__ LineArgs a) {
    const LineTask& t = a.t[blockIdx.z];
    const int d = a.d, ax = d == 2 ? 1 : 2, bx = d == 0 ? 1 : 0;   // axes across the line, fastest first
    const int na = t.hi[ax] - t.lo[ax];
    const long long l = (long long)blockIdx.x * LINE_THREADS + threadIdx.x;
    if (l >= (long long)na * (t.hi[bx] - t.lo[bx])) return;
    const int i0 = t.lo[d] + blockIdx.y * a.chunk, i1 = min(i0 + a.chunk, t.hi[d]);
    if (i0 >= i1) return;
    const int pb = (int)(l / na), pa = (int)(l - (long long)pb * na);
    const long long s = a.g.stride(d);
    const long long base = (long long)(t.lo[ax] + pa) * a.g.stride(ax) + (long long)(t.lo[bx] + pb) * a.g.stride(bx);
    const int n = a.g.N[d];
    const double* __restrict__ q = t.q + base;
    const double* __restrict__ U = t.U + base;
    double* __restrict__ out = t.out + base;
    auto ld = [&](int k) { return __ldg(q + (long long)min(max(k, 0), n - 1) * s); };
    const bool vortex = t.vortex != 0;
    // the state of face j, between cells j and j + 1 (the vortex force's flux of cell i is
    // that of face i - 1 of the vorticity)
    int j = i0 - 1;
    LineFace f;
    double q0 = ld(j), q1 = ld(j + 1), q2 = ld(j + 2), q3 = ld(j + 3);
    double brp, brq, bcq;                  // indicators that the next faces use
    {
        const double qm = ld(j - 1), qmm = ld(j - 2);
        double x, y;
        f.d0 = qm - qmm;
        f.d1 = q0 - qm;
        f.d2 = q1 - q0;
        f.d3 = q2 - q1;
        f.d4 = q3 - q2;
        line_node(f.d0, f.d1, x, y, f.brm);
        line_node(f.d1, f.d2, x, f.bc0, f.br0);
        line_node(f.d2, f.d3, f.blp, f.bcp, brp);
        line_node(f.d3, f.d4, f.blq, bcq, brq);
    }
    // to face j + 1
    auto advance = [&](double qn) {
        f.d0 = f.d1; f.d1 = f.d2; f.d2 = f.d3; f.d3 = f.d4;
        f.d4 = qn - q3;
        q0 = q1; q1 = q2; q2 = q3; q3 = qn;
        f.brm = f.br0; f.br0 = brp; brp = brq;
        f.bc0 = f.bcp; f.bcp = bcq;
        f.blp = f.blq;
        line_node(f.d3, f.d4, f.blq, bcq, brq);
        ++j;
    };
    if (vortex) {
        const long long sa = t.sa;
        const double sgn = t.sgn;
        // velocity averaged across, at the cell behind (0 at the array's first cell)
        double um = i0 > 0 ? __ldg(U + (long long)(i0 - 1) * s) + __ldg(U + (long long)(i0 - 1) * s + sa) : 0.0;
        for (int i = i0; i < i1; ++i) {
            const long long c = (long long)i * s;
            const double qn = ld(i + 3), ua = __ldg(U + c), ub = __ldg(U + c + sa), o = out[c];
            const double uu = ua + ub;
            const double u = 0.25 * (um + uu);
            um = uu;
            const double fl = (i >= 3 && i <= n - 4) ? line_flux(f, u, q0, q1) : line_vf_closure(q, u, i, n, s);
            out[c] = fma(sgn, fl, o);
            advance(qn);
        }
    } else {
        const bool assign = t.assign != 0;
        const double kd = t.kd;
        auto face = [&](int i, double u) {
            return (i >= 2 && i <= n - 4) ? line_flux(f, u, q0, q1) : line_tr_closure(q, u, i, n, s);
        };
        double fm = 0.0;
        if (i0 > 0) {
            const double qn = ld(i0 + 3);
            fm = face(i0 - 1, __ldg(U + (long long)(i0 - 1) * s));
            advance(qn);
        } else {
            advance(ld(i0 + 3));
        }
        for (int i = i0; i < i1; ++i) {
            const long long c = (long long)i * s;
            const double qn = ld(i + 4), u = __ldg(U + c), o = assign ? 0.0 : out[c];
            const double fl = face(i, u);
            double acc = (o + fm) - fl;
            fm = fl;
            // core/tracer.py:74-76: the direction's diffusion after its advection (a wall's
            // outer difference is 0, core/fortran_dissipation.f90:18-33)
            if (kd != 0.0) acc = acc + kd * ((i < n - 1 ? f.d2 : 0.0) - (i > 0 ? f.d1 : 0.0));
            out[c] = acc;
            advance(qn);
        }
    }
}

// Cells per thread: every chunk starts with the six loads and four nodes of its first face
// (about 30 FP64 instructions, 3/4 of a flux), so chunks are long, until they leave fewer
// than 24 warps per SM, which then end unevenly. Measured, chunks of 8 / 16 / 32 / 64: the
// 109 x 75 x 53 right-hand side 614 / 644 / 706 us (16 cells: 23 warps per SM), a 128 x 64 x 64
// LFAM3 step 2.53 / 2.50 / 2.65 ms (16 cells: 29 warps per SM), a 256^3 RK3 step - / 86.7 / 85.4 /
// 85.3 ms; below 8 nothing is gained (64 x 32 x 32: 4, 6, 8, 12 cells within 3%).
static int line_chunk(long long lines, int n) {
    int chunk = 64;
    while (chunk > 8 && lines * ((n + chunk - 1) / chunk) < 152ll * 24 * 32) chunk /= 2;
    return chunk;
}

int launch_rhs_lines(const NylesDesc* d, const Geom& g, const StencilPtrs<double>& s, const ProgPtrs<double>& ds,
                     int terms, cudaStream_t st, bool interior) {
    // b and u: the interior of periodic directions (interior = true) or every stored cell
    int lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        const bool in = interior && g.per[k];
        lo[k] = in ? g.nh : 0;
        hi[k] = in ? g.nh + g.n[k] : g.N[k];
    }
    const double ids2[3] = {d->idz2, d->idy2, d->idx2};
    // vortex force along each axis: advected vorticity, register and sign, averaging axis
    // (core/vortex_force.py:69-81)
    struct Vf { int w, reg, aa; double sgn; };
    static const Vf vf[3][2] = {
        {{0, 2, 1, 1.0}, {1, 1, 2, -1.0}},     // z: u_j += U^k w_i, u_i -= U^k w_j
        {{2, 1, 2, 1.0}, {0, 3, 0, -1.0}},     // y: u_i += U^j w_k, u_k -= U^j w_i
        {{2, 2, 1, -1.0}, {1, 3, 0, 1.0}},     // x: u_j -= U^i w_k, u_k += U^i w_j
    };
    bool first = true;
    for (int ax = 2; ax >= 0; --ax) {          // x, y, z
        LineArgs a;
        a.g = g;
        a.d = ax;
        int nt = 0;
        long long lines = 0, cells = 0;
        auto add = [&](LineTask t) {
            const long long across = (long long)(t.hi[ax == 2 ? 1 : 2] - t.lo[ax == 2 ? 1 : 2]) *
                                     (t.hi[ax == 0 ? 1 : 0] - t.lo[ax == 0 ? 1 : 0]);
            if (across <= 0 || t.hi[ax] <= t.lo[ax]) return;
            lines = std::max(lines, across);
            cells = std::max(cells, (long long)(t.hi[ax] - t.lo[ax]));
            a.t[nt++] = t;
        };
        const double* U = s.f[NYLES_F_UC_I + (2 - ax)];
        if (terms & TERM_TRACER)
            for (int q = 0; q <= d->n_tracers; ++q) {
                LineTask t{};
                t.q = q == 0 ? s.f[NYLES_F_B] : s.f[NYLES_F_T0 + q - 1];
                t.out = ds.p[q == 0 ? 0 : 3 + q];
                if (!t.out) continue;
                t.U = U;
                t.assign = first;
                if ((terms & TERM_TRDIFF) && ((d->tracer_diffusion >> q) & 1))
                    t.kd = d->tracer_diffusivity[q] * ids2[ax];
                for (int k = 0; k < 3; ++k) {   // tracers t0.. cover every stored cell
                    t.lo[k] = q == 0 ? lo[k] : 0;
                    t.hi[k] = q == 0 ? hi[k] : g.N[k];
                }
                add(t);
            }
        if (terms & TERM_VF)
            for (const Vf& v : vf[ax]) {
                LineTask t{};
                t.vortex = 1;
                t.q = s.f[NYLES_F_VOR_I + v.w];
                t.U = U;
                t.out = ds.p[v.reg];
                t.sgn = v.sgn;
                t.sa = g.stride(v.aa);
                for (int k = 0; k < 3; ++k) {
                    t.lo[k] = lo[k];
                    t.hi[k] = k == v.aa ? std::min(hi[k], g.N[k] - 1) : hi[k];
                }
                add(t);
            }
        first = false;
        if (nt == 0) continue;
        a.chunk = line_chunk(lines * nt, (int)cells);
        const dim3 grd((unsigned)((lines + LINE_THREADS - 1) / LINE_THREADS),
                       (unsigned)((cells + a.chunk - 1) / a.chunk), nt);
        k_line<<<grd, LINE_THREADS, 0, st>>>(a);
        note_launch();
    }
    return cuda_status(cudaGetLastError(), "rhs line kernel");
}

}  // namespace nyles
