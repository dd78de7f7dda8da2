// Convection in (MLT, L) on every (V,K) slice, a QUICKEST pass in two stages
// over line segments: Convection_2D (src/Convection_2D.cpp:36-169) over
// Convection_1D_ULTIMATE_QUICKEST6 (QUICKEST6.cpp:22-482).  Compiled twice:
// with multiply-add contraction (stream mode), and with -fmad=false and
// -DVERB_BUILD_CONV_EXACT, which keeps the reference's operations and their
// order one by one (bit-identical to it, exp() of loss rates aside).
//
// A CTA keeps one [P][R] slice in shared memory for all of its CFL sub-steps.
// The reference's four loops over a line become two, each run by one thread
// per segment of a line (about 4 to 13 cells, threads of a warp on
// neighbouring lines):
//   stage 1  unlimited faces a .. a+own and from them the unlimited cells
//            (loops 1 and 2, :148-272), both to shared memory;
//   stage 2  the peak flags of the segment as bit masks from the unlimited
//            line, then limited faces and final cells (loops 3 and 4,
//            :277-477), in place, with the store epilogue.
// A barrier separates the stages and the sweeps.  The face between two
// segments is formed by both; what a segment reads of its neighbours' cells in
// stage 2, it keeps in registers from stage 1.
//
// What bounds it: the issue of about 240 instructions a face (a third of them
// FP64; 400 in the exact form), with 16 warps on an SM.  The streaming kernel
// (one thread a line, all four loops at once) holds some 40 values in flight,
// which limits it to 12 warps whose chains run along the whole line, so a slice
// of many sub-steps takes as long as its lines are: 24 x 25 x 31 x 31 alone 9.9
// ms, 2.7 here; 48 x 101 x 101 x 16 alone 47.4 ms, 23.2 here (one after the other
// 31.0 -> 23.1 ms).
#include "exact_div.cuh"
#include "quickest.cuh"
#include "verb_internal.cuh"

#include <algorithm>

#ifdef VERB_BUILD_CONV_EXACT
#define VERB_STAGED_NS conv_staged_exact
#define VERB_STAGED(name) name##_exact
#else
#define VERB_STAGED_NS conv_staged
#define VERB_STAGED(name) name
#endif

namespace verb {
namespace VERB_STAGED_NS {  // the two compilations keep their kernels apart
namespace {

constexpr double CG_MAX_SUBSTEPS = 1.0e6;
constexpr int CG_MAX_OWN = 25;  // cells of a segment: own + 7 flag bits in a word

// the exact form's L sweep divides by G and keeps exp(Loss dt) apart
#ifdef VERB_BUILD_CONV_EXACT
constexpr int CG_TABS = 7;
#else
constexpr int CG_TABS = 5;
#endif

// The planes carry CG_GH ghost cells around the slice, so that a window never
// needs to ask where the line ends.
constexpr int CG_GH = 5;
__host__ __device__ inline int cg_rs(int R) { return (R + 2 * CG_GH) | 1; }

// Launch shape of a [P][R] slice.
struct StagedShape {
    int threads;      // per CTA
    int own;          // most cells of a segment
    int segP, segR;   // segments of an MLT line, of an L line
};

// per CTA: c and 1/|c| of both sweeps' faces, the store epilogues (factor, and
// added term of the L sweep), line data, and room for the rows a group reads
// past a line's end
__host__ __device__ inline size_t cg_scratch(int P, int R)
{
    return 2 * (size_t)P * (R - 1) + CG_TABS * (size_t)P * R + 4 * (size_t)(R - 1) + 4 * (size_t)P +
           32 * (size_t)(P > R ? P : R);
}

__host__ __device__ inline size_t cg_plane(int P, int R)
{
    return (size_t)(P + 2 * CG_GH) * cg_rs(R);
}

// three planes and what a group reads past the last one
__host__ __device__ inline size_t cg_smem(int P, int R)
{
    return (3 * cg_plane(P, R) + 8 * (size_t)cg_rs(R) + 32) * sizeof(double) +
           (size_t)(R + P) * sizeof(int);
}

// A thread's segment of a line.
struct Seg {
    const double* E;     // cell k of the line before the pass at [k * st], with ghosts
    double* U;           // unlimited cell k, with ghosts
    double* O;           // unlimited face k + 1, replaced by cell k after the pass
    int st;
    int a, own, n;       // first cell, cells, points of the line
    int lt, ut;
    const double* ln;    // line data (lbc, ubc, dxl, dxu) at ln[i * nl]
    int nl;
    const double *cr, *rc;  // c and 1 / |c| (0 for |c| <= 1e-31) of face k at [k * nl]
    // store epilogue of cell k: times e1 (P), or: times e1 plus e2 (R); the
    // exact form divides by e3 (reciprocal e4) before, in the L sweep.  Where
    // nothing is to be added it adds -0, which leaves a -0 as it is
    const double *e1, *e2, *e3, *e4;
};

// ghost cells of the line before a pass (:89-143)
__device__ __forceinline__ void line_ghosts(double* E, int st, int n, int lt, int ut,
                                            const double* ln, int nl)
{
    if (lt == VERB_BC_PERIODIC) {
#pragma unroll
        for (int k = 1; k <= CG_GH; k++) {
            E[-k * st] = E[(n - 1 - k) * st];
            E[(n - 1 + k) * st] = E[k * st];
        }
        return;
    }
    double g = E[0], h = E[(n - 1) * st];
    const double dl = ln[0] * ln[2 * nl], du = ln[nl] * ln[3 * nl];
#pragma unroll
    for (int k = 1; k <= CG_GH; k++) {
        g = lt == VERB_BC_CONSTANT_VALUE ? ln[0] : g - dl;
        h = ut == VERB_BC_CONSTANT_VALUE ? ln[nl] : h + du;
        E[-k * st] = g;
        E[(n - 1 + k) * st] = h;
    }
}

// Stage 1 takes the faces of a segment U at a time, stage 2 three: the
// polynomials and the limiters of a group are independent of each other, and
// the window is loaded once per group instead of shifted through registers.

// NaN, infinite or above 2^300
__device__ __forceinline__ bool is_odd(double v)
{
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) >= 0x52b00000u;
}

// Unlimited value of one face from its stencil e[k * st] = E[x-5+k], the
// reference's sums as they stand
__device__ __forceinline__ double face_alone(const double* e, int st, double c)
{
    const bool pos = c >= 0;
    double a[5], b[5];  // upwind from the centre on, downwind
#pragma unroll
    for (int k = 0; k < 5; k++) {
        a[k] = e[(pos ? 4 - k : 5 + k) * st];
        b[k] = e[(pos ? 5 + k : 4 - k) * st];
    }
    return quickest_face_k(a[1], a[2], a[3], a[4], a[0], b[0], b[1], b[2], b[3], b[4], c,
                           face_coef_exact(c));
}

#ifdef VERB_BUILD_CONV_EXACT
// Unlimited values of U faces from the window d[k] = E[x-5+k], the roles of the
// stencil's points chosen by the direction (QUICKEST6.cpp:169-186)
template <int U>
__device__ __forceinline__ void faces(double (&d)[U + 9], const double (&c)[U], double (&f)[U])
{
#pragma unroll
    for (int u = 0; u < U; u++) {
        const bool pos = c[u] >= 0;
        double a[5], b[5];  // upwind from the centre on, downwind
#pragma unroll
        for (int k = 0; k < 5; k++) {
            a[k] = pos ? d[u + 4 - k] : d[u + 5 + k];
            b[k] = pos ? d[u + 5 + k] : d[u + 4 - k];
        }
        const FaceCoef k = face_coef_exact(c[u]);
        f[u] = quickest_face_k(a[1], a[2], a[3], a[4], a[0], b[0], b[1], b[2], b[3], b[4], c[u], k);
    }
}
#else
// Unlimited values of U faces from the window d[k] = E[x-5+k] (QUICKEST6.cpp:
// 162-241, in the positive orientation with the signed Courant number).  The
// differences of the stencil are built level by level for all of the group's
// faces, D^m_k = D^(m-1)_k - D^(m-1)_(k+1), shared by neighbouring faces: with
// (a, b) the two m-th differences at face u, m even, the reference's even term
// is (a + b) / 2 and its odd term a - b.  The ninth-order pair E8 + sign d9 is
// 2a or 2b: it leaves out the stencil's last point, and (a + b) of two infinities is
// not a number where the reference's sum is infinite, so slices that hold such
// values are left to a second launch (ODD), whose faces are face_alone's.
template <int U>
__device__ __forceinline__ void faces(double (&d)[U + 9], const double (&c)[U], double (&f)[U])
{
    double cs[U], p[U];
    auto level = [&](int m) {  // next difference, in place: m entries
#pragma unroll
        for (int k = 0; k < U + 8; k++)
            if (k < m) d[k] = d[k] - d[k + 1];
    };
#pragma unroll
    for (int u = 0; u < U; u++) {
        const double s0 = d[u + 4] + d[u + 5];
        const double t0 = d[u + 4] - d[u + 5];
        f[u] = 0.5 * (s0 + c[u] * t0);
        cs[u] = c[u] * c[u];
        p[u] = cs[u] - 1;
    }
    level(U + 8);
    level(U + 7);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const double x = d[u + 3], y = d[u + 4];
        f[u] += (p[u] * (1.0 / 12.0)) * ((x + y) + (c[u] * 0.5) * (x - y));
        p[u] *= cs[u] - 4;
    }
    level(U + 6);
    level(U + 5);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const double x = d[u + 2], y = d[u + 3];
        f[u] += (p[u] * (1.0 / 240.0)) * ((x + y) + (c[u] * (1.0 / 3.0)) * (x - y));
        p[u] *= cs[u] - 9;
    }
    level(U + 4);
    level(U + 3);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const double x = d[u + 1], y = d[u + 2];
        f[u] += (p[u] * (1.0 / 10080.0)) * ((x + y) + (c[u] * 0.25) * (x - y));
        p[u] *= cs[u] - 16;
    }
    level(U + 2);
    level(U + 1);
#pragma unroll
    for (int u = 0; u < U; u++)
        f[u] += (p[u] * (1.0 / 362880.0)) * (c[u] >= 0 ? d[u] : d[u + 1]);
}

#endif

// returns unlimited face a, whose slot is the neighbour's
template <int U, bool ODD>
__device__ __forceinline__ double stage1(const Seg& L)
{
    double Q = 0.0, f0 = 0.0;
    const double* cp = L.cr + L.a * L.nl;
    // faces a .. a+own, cells a .. a+own-1; what is read past the line's
    // ghosts and tables (memory of the same regions) only feeds faces past own
#pragma unroll 1
    for (int i = 0; i <= L.own; i += U) {
        const int x = L.a + i;
        double d[U + 9], c[U], f[U] = {};
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = cp[u * L.nl];
        cp += U * L.nl;
        const double* ep = L.E + (x - 5) * L.st;
#pragma unroll
        for (int k = 0; k < U + 9; k++) d[k] = ep[k * L.st];
        if constexpr (ODD) {
#pragma unroll 1
            for (int u = 0; u < U; u++) {
                const double v = face_alone(ep + u * L.st, L.st, cp[(u - U) * L.nl]);
#pragma unroll
                for (int k = 0; k < U; k++) f[k] = k == u ? v : f[k];
            }
        } else {
            faces<U>(d, c, f);
        }
        double* up = L.U + (x - 1) * L.st;
        double* fp = L.O + (x - 1) * L.st;
        if (i == 0) f0 = f[0];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const double q = c[u] * f[u];
            if ((u > 0 || i > 0) && i + u <= L.own) {
                up[u * L.st] = ep[(u + 4) * L.st] - (q - Q);
                fp[u * L.st] = f[u];
            }
            Q = q;
        }
    }
    const double* ep = L.E + L.a * L.st;
    // boundary rewrite (:257-272) and the unlimited line's ghosts (:281-330;
    // the periodic low ones come from the line before the pass)
    if (L.lt == VERB_BC_PERIODIC) {
        if (L.a == 0) {
            L.U[(L.n - 1) * L.st] = L.U[0];
#pragma unroll
            for (int k = 1; k <= 4; k++) L.U[-k * L.st] = ep[-k * L.st];
        }
        if (L.a <= 4)
            for (int k = max(1, L.a); k <= min(4, L.a + L.own - 1); k++)
                L.U[(L.n - 1 + k) * L.st] = L.U[k * L.st];
        return f0;
    }
    if (L.a == 0) {
        const double u0 = L.lt == VERB_BC_CONSTANT_VALUE ? L.ln[0] : L.U[L.st];
        const double dl = L.ln[0] * L.ln[2 * L.nl];
        double g = u0;
        L.U[0] = u0;
#pragma unroll
        for (int k = 1; k <= 4; k++) {
            g = L.lt == VERB_BC_CONSTANT_VALUE ? u0 : g - dl;
            L.U[-k * L.st] = g;
        }
    }
    if (L.a + L.own == L.n - 1) {
        double* e = L.U + (L.n - 1) * L.st;
        const double u1 = L.ut == VERB_BC_CONSTANT_VALUE ? L.ln[L.nl] : e[-L.st];
        const double du = L.ln[L.nl] * L.ln[3 * L.nl];
        double g = u1;
        e[0] = u1;
#pragma unroll
        for (int k = 1; k <= 4; k++) {
            g = L.ut == VERB_BC_CONSTANT_VALUE ? u1 : g + du;
            e[k * L.st] = g;
        }
    }
    return f0;
}

// v with its sign flipped where s is the sign bit
__device__ __forceinline__ double flip(double v, int s)
{
    return __hiloint2double(__double2hiint(v) ^ s, __double2loint(v));
}

// Limited face value (:394-447) from the unlimited value f, the Courant
// number c and 1 / |c|, cells x-2 .. x+1 and the face's peak flag.
__device__ __forceinline__ double limit(double f, double c, double rc, double em2, double em1,
                                        double e0, double ep1, bool peak)
{
    const bool pos = c >= 0;
    const double ou = pos ? em2 : ep1;
    const double oc = pos ? em1 : e0;
    const double od = pos ? e0 : em1;
    const double DEL = od - ou;
    const double CURV = od - 2 * oc + ou;
    const bool flat = fabs(CURV) >= fabs(DEL);
    const bool rise = DEL > 0, fall = DEL < 0;
    const bool useref = !peak & !flat & (__double2hiint(rc) != 0) & (rise | fall);
#ifdef VERB_BUILD_CONV_EXACT
    const double ref = ou + div_by(oc - ou, fabs(c), rc);
#else
    const double ref = ou + (oc - ou) * rc;
#endif
    // max and min as selects that keep fmax's and fmin's values where f, oc or
    // ref is not a number (ou and od are numbers here)
    const int s = rise ? 0 : (int)0x80000000;
    const double a = flip(f, s), lo = flip(oc, s), h1 = flip(ref, s), h2 = flip(od, s);
    double t = a > lo ? a : lo;
    const double hi = h1 < h2 ? h1 : h2;
    t = t < hi ? t : hi;
    double res = useref ? flip(t, s) : f;
    if (!peak & flat) res = oc;
    return res;
}

// v h1 + h2, for the exact form's L sweep (v / h3) h1 + h2 (h4 = RN(1 / h3))
__device__ __forceinline__ double epilogue(double v, double h1, double h2, double h3, double h4,
                                           bool div)
{
#ifdef VERB_BUILD_CONV_EXACT
    if (div) v = div_by(v, h3, h4);
#endif
    return v * h1 + h2;
}

// last: the line's last sub-cycle, whose cells take the store epilogue
__device__ __forceinline__ void stage2(const Seg& L, double f0, bool last)
{
    // peak flags M of positions a-4 .. : differences e_k = U[k+1] - U[k], bit
    // k - (a-4); M: rising twice, then falling twice, with a bend at both ends
    unsigned up = 0, dn = 0, bend = 0;
    {
        constexpr int W = 6;
        const double* p = L.U + (L.a - 4) * L.st;
        double v = *p, e = 0.0;
#pragma unroll 1
        for (int i = 0; i < L.own + 7; i += W) {
            double w[W];
#pragma unroll
            for (int u = 0; u < W; u++) {
                p += L.st;
                w[u] = *p;
            }
            unsigned b1 = 0, b2 = 0, b3 = 0;
#pragma unroll
            for (int u = 0; u < W; u++) {
                const double en = w[u] - v;
                if (en > 0) b1 |= 1u << u;
                if (en < 0) b2 |= 1u << u;
                if (en < e) b3 |= 1u << u;
                v = w[u];
                e = en;
            }
            up |= b1 << i;
            dn |= b2 << i;
            bend |= b3 << i;
        }
        bend >>= 1;
    }
    const unsigned M = up & up >> 1 & dn >> 2 & dn >> 3 & bend & bend >> 2;
    // face x takes positions x-4 .. x-2, or x-3 .. x-1 against the direction
    unsigned three = M | M >> 1 | M >> 2;

    constexpr int U = 3;
    double Rp = 0.0, first = 0.0, second = 0.0, end = 0.0;
    int at = L.a * L.nl;
#pragma unroll 1
    for (int i = 0; i <= L.own; i += U) {
        const int x = L.a + i;
        const double* ep = L.E + (x - 2) * L.st;
        double* op = L.O + (x - 1) * L.st;
        double c[U], rc[U], h1[U], h2[U], h3[U], h4[U], w[U + 3], f[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            c[u] = L.cr[at];
            rc[u] = L.rc[at];
            h1[u] = h3[u] = h4[u] = 1.0;
            h2[u] = -0.0;
            at += L.nl;
            // cell x + u - 1 (the first group's entry of cell a - 1, and past
            // the table's ends, is not used)
            if (last) {
                h1[u] = L.e1[at - 2 * L.nl];
                if (L.e2) h2[u] = L.e2[at - 2 * L.nl];
#ifdef VERB_BUILD_CONV_EXACT
                if (L.e2) {
                    h3[u] = L.e3[at - 2 * L.nl];
                    h4[u] = L.e4[at - 2 * L.nl];
                }
#endif
            }
        }
#pragma unroll
        for (int k = 0; k < U + 3; k++) w[k] = ep[k * L.st];
#pragma unroll
        for (int u = 0; u < U; u++) f[u] = op[u * L.st];
        if (i == 0) f[0] = f0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool peak = three >> (u + (c[u] >= 0 ? 0 : 1)) & 1u;
            const double r = c[u] * limit(f[u], c[u], rc[u], w[u], w[u + 1], w[u + 2], w[u + 3],
                                          peak);
            const double o = w[u + 1] - (r - Rp);
            if ((u > 0 || i > 0) && i + u <= L.own)
                op[u * L.st] = epilogue(o, h1[u], h2[u], h3[u], h4[u], last && L.e2);
            if (u == 1 && i == 0) first = o;
            if (u == 2 && i == 0) second = o;
            if (L.ut == VERB_BC_CONSTANT_DERIVATIVE && i + u == L.own) end = o;
            Rp = r;
        }
        three >>= U;
    }
    // boundary rewrite (:462-477): the cells at the line's ends (no source term)
    auto put = [&](int k, double v) {
#ifdef VERB_BUILD_CONV_EXACT
        if (last && L.e2) v = v / L.e3[k * L.nl];
#endif
        L.O[k * L.st] = last ? v * L.e1[k * L.nl] : v;
    };
    if (L.a == 0) {
        if (L.lt == VERB_BC_PERIODIC) put(L.n - 1, first);
        else put(0, L.lt == VERB_BC_CONSTANT_VALUE ? L.ln[0] : second);
    }
    if (L.a + L.own == L.n - 1 && L.ut != VERB_BC_PERIODIC)
        put(L.n - 1, L.ut == VERB_BC_CONSTANT_VALUE ? L.ln[L.nl] : end);
}

__device__ __forceinline__ double cg_block_max(double v, double* red)
{
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, v, o);
        v = (v < t) ? t : v;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double m = red[0];
    for (int i = 1; i < nw; i++) m = (m < red[i]) ? red[i] : m;
    __syncthreads();
    return m;
}

template <int U1, int MAXT, int MINB, bool ODD = false>
__global__ void __launch_bounds__(MAXT, MINB) convection_staged_kernel(ConvArgs a, int segP, int segR)
{
    extern __shared__ __align__(16) double sm[];
    const Dims d = a.d;
    const int P = d.P, R = d.R, V = d.V, K = d.K;
    const int PR = P * R, Rs = cg_rs(R);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x, nw = nt >> 5;
    const int plane = (int)cg_plane(P, R);
    double* S = sm + CG_GH * Rs + CG_GH;    // the slice, with ghosts
    double* F = S + plane;                  // unlimited faces, then the slice after a sweep
    double* U = F + plane;                  // unlimited cells of a sweep, with ghosts
    double* red = sm + 3 * (size_t)plane + 8 * (size_t)Rs;  // [32]
    int* nsP = (int*)(red + 32);            // [R] sub-cycles of P-line iR
    int* nsR = nsP + R;                     // [P] sub-cycles of R-line iP
    __shared__ int s_ticket, s_ns[2];

    // slice tables, line-fastest: [P faces or cells][R-1 lines], [R][P lines]
    const size_t VK = (size_t)V * K, P1 = (size_t)P * (R - 1);
    double* crP = a.scratch + (size_t)blockIdx.x * cg_scratch(P, R);
    double* rcP = crP + P1;
    double* e1P = rcP + P1;                    // G
    double* crR = e1P + (size_t)PR;
    double* rcR = crR + (size_t)PR;
    double* e1R = rcR + (size_t)PR;            // exp(Loss dt)/G, or exp(Loss dt)
    double* e2R = e1R + (size_t)PR;            // S dt, -0 at the ends
#ifdef VERB_BUILD_CONV_EXACT
    double* e3R = e2R + (size_t)PR;            // G
    double* e4R = e3R + (size_t)PR;            // 1 / G
    double* lnP = e4R + (size_t)PR;            // [4][R-1]
#else
    double *e3R = nullptr, *e4R = nullptr;
    double* lnP = e2R + (size_t)PR;            // [4][R-1]
#endif
    double* lnR = lnP + 4 * (size_t)(R - 1);   // [4][P]
    const int nslices = V * K;

    for (;;) {
        if (tid == 0) {
            if constexpr (ODD) {
                const int q = atomicAdd(a.ticket + 2, 1);
                s_ticket = q < a.ticket[1] ? a.odd[q] : nslices;
            } else {
                s_ticket = atomicAdd(a.ticket, 1);
            }
            s_ns[0] = s_ns[1] = 1;
        }
        __syncthreads();
        const int t = s_ticket;
        __syncthreads();
        if (t >= nslices) break;
        const int iV = V - 1 - t / K;
        const int iK = t - (t / K) * K;
        const size_t off = (size_t)iV * K + iK;
        auto g = [&](int iP, int iR) { return ((size_t)iP * R + iR) * VK + off; };

        // slice load and slice-level sub-step count (src/Convection_2D.cpp:57-86)
        double vpm = 0.0, vrm = 0.0;
        for (int i = tid; i < PR; i += nt) {
            const int iP = i / R, iR = i - iP * R;
            const size_t gi = g(iP, iR);
            S[iP * Rs + iR] = a.psd[gi];
            const double vp = fabs(a.VP[gi]), vr = fabs(a.VR[gi]);
            vpm = (vpm < vp) ? vp : vpm;
            vrm = (vrm < vr) ? vr : vrm;
        }
        vpm = cg_block_max(vpm, red);
        vrm = cg_block_max(vrm, red);
        double nsp, nsr;
        {
            const double dP = a.Pg[g(1, 0)] - a.Pg[g(0, 0)];
            const double x = (double)a.dt * vpm / dP / 0.25;
            nsp = x <= 1 ? 1 : ceil(x);
        }
        {
            const double dR = a.Rg[g(0, 1)] - a.Rg[g(0, 0)];
            const double x = (double)a.dt * vrm / dR / 0.25;
            nsr = x <= 1 ? 1 : ceil(x);
        }
        const double num_steps = (nsp < nsr) ? nsr : nsp;
        if (!(num_steps <= CG_MAX_SUBSTEPS)) {  // also catches inf / NaN
            if (tid == 0) {
                a.substeps[off] = -1;
                set_error(a.status, VERB_ERR_CFL);
            }
            __syncthreads();
            continue;
        }
        const double dtc = a.dt / num_steps;
        if (tid == 0) a.substeps[off] = (int)num_steps;
        bool odd = false;  // a value that is left to the second launch
        for (int i = tid; i < PR; i += nt) {
            const int iP = i / R, iR = i - iP * R;
            const size_t gi = g(iP, iR);
            const double G = a.G[gi];
            if (iR < R - 1) e1P[(size_t)iP * (R - 1) + iR] = G;
#ifdef VERB_BUILD_CONV_EXACT
            e1R[(size_t)iR * P + iP] = exp(a.loss[gi] * dtc);
            e3R[(size_t)iR * P + iP] = G;
            e4R[(size_t)iR * P + iP] = __drcp_rn(G);
#else
            const double eg = exp(a.loss[gi] * dtc) / G;
            e1R[(size_t)iR * P + iP] = eg;
            odd |= is_odd(S[iP * Rs + iR]) || is_odd(G) || is_odd(eg) || is_odd(a.S[gi]);
#endif
            e2R[(size_t)iR * P + iP] = iR && iR < R - 1 ? a.S[gi] * dtc : -0.0;
        }
        // per-line CFL sub-cycles and face Courant numbers (QUICKEST6.cpp:37-52,
        // 150-160), one warp per line; velocity vel and grid x at (line, k)
        auto line_table = [&](const double* vel, const double* x, int line, int n, bool pr,
                              double* cr, double* rc, int* nsl, double* ln, int nl) {
            auto at = [&](int k) { return pr ? g(k, line) : g(line, k); };
            double m = -INFINITY;
            for (int k = lane; k < n; k += 32) {
                const double v = fabs(vel[at(k)]);
                m = (m > v) ? m : v;
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double q = __shfl_xor_sync(0xffffffffu, m, o);
                m = (m > q) ? m : q;
            }
            const double dx = x[at(1)] - x[at(0)];
            const double sd = (double)dtc * m / dx / 1.0;
            int ns = 1;
            if (!(sd <= CG_MAX_SUBSTEPS)) set_error(a.status, VERB_ERR_CFL);
            else if (sd > 1) ns = (int)ceil(sd);
            const double dtl = dtc / ns;
            if (fabs(m / dx * dtl) > 1) set_error(a.status, VERB_ERR_CFL);
            for (int k = lane; k < n; k += 32) {
                const double c0 = vel[at(k == 0 ? n - 2 : k - 1)] / dx * dtl;
                const double c1 = vel[at(k)] / dx * dtl;
                const double c = (c0 + c1) / 2;
                cr[(size_t)k * nl + line] = c;
                rc[(size_t)k * nl + line] = fabs(c) > 1e-31 ? __drcp_rn(fabs(c)) : 0.0;
            }
            if (lane == 0) {
                nsl[line] = ns;
                if (ns > 1) atomicMax(&s_ns[pr ? 0 : 1], ns);
                ln[2 * nl + line] = dx;
                ln[3 * nl + line] = x[at(n - 1)] - x[at(n - 2)];
            }
        };
        for (int iR = warp; iR < R - 1; iR += nw) {
            line_table(a.VP, a.Pg, iR, P, true, crP, rcP, nsP, lnP, R - 1);
            if (lane == 0) {
                const size_t bo = ((size_t)iR * V + iV) * K + iK;
                const double lb = a.Pl[bo], ub = a.Pu[bo];
                lnP[iR] = lb;
                lnP[(R - 1) + iR] = ub;
                odd |= a.Pl_t != VERB_BC_PERIODIC && (is_odd(lb) || is_odd(ub));
            }
        }
        for (int iP = warp; iP < P; iP += nw) {
            line_table(a.VR, a.Rg, iP, R, false, crR, rcR, nsR, lnR, P);
            if (lane == 0) {
                const size_t bo = ((size_t)iP * V + iV) * K + iK;
                const double lb = a.Rl[bo] * a.G[g(iP, 0)], ub = a.Ru[bo] * a.G[g(iP, R - 1)];
                lnR[iP] = lb;
                lnR[P + iP] = ub;
                odd |= a.Rl_t != VERB_BC_PERIODIC && (is_odd(lb) || is_odd(ub));
            }
        }
        double steps = num_steps;
#ifdef VERB_BUILD_CONV_EXACT
        __syncthreads();
#else
        if (__syncthreads_or(odd) && !ODD) {  // (a jump out of here costs registers)
            if (tid == 0) a.odd[atomicAdd(a.ticket + 1, 1)] = t;
            steps = 0;
        }
#endif

        for (int it = 0; it < steps; it++) {
            // the MLT sweep (ph 0: P-lines iR, stored times G) and the L sweep
            // (ph 1: R-lines iP, stored as v exp(Loss dt)/G + S dt) go through
            // one copy of the stages
#pragma unroll 1
            for (int ph = 0; ph < 2; ph++) {
                const bool pr = ph == 0;
                const int nl = pr ? R - 1 : P, ns_seg = pr ? segP : segR;
                const int seg = tid / nl, line = tid - seg * nl;
                Seg L;
                L.n = pr ? P : R;
                // the n-1 cells before the last, in segments of two lengths
                const int nc = L.n - 1, len = nc / ns_seg, more = nc - len * ns_seg;
                L.own = len + (seg < more);
                L.a = seg * len + min(seg, more);
                const bool live = seg < ns_seg;
                L.st = pr ? Rs : 1;
                const int o0 = pr ? line : line * Rs;
                L.U = U + o0;
                L.lt = pr ? a.Pl_t : a.Rl_t;
                L.ut = pr ? a.Pu_t : a.Ru_t;
                L.ln = (pr ? lnP : lnR) + line;
                L.nl = nl;
                L.cr = (pr ? crP : crR) + line;
                L.rc = (pr ? rcP : rcR) + line;
                L.e1 = (pr ? e1P : e1R) + line;
                L.e2 = pr ? nullptr : e2R + line;
                L.e3 = e3R + line;
                L.e4 = e4R + line;
                const int ns = live ? (pr ? nsP : nsR)[line] : 0;
                // the line's own CFL sub-cycles (:37-52), the epilogue on the
                // last one only
                const int most = s_ns[ph];
                for (int k = 0; k < most; k++) {
                    for (int q = tid; q < nl; q += nt) {
                        double* e = S + (pr ? q : q * Rs);
                        line_ghosts(e, L.st, L.n, L.lt, L.ut, (pr ? lnP : lnR) + q, nl);
                    }
                    L.E = S + o0;
                    L.O = F + o0;
                    const bool run = k < ns, last = k == ns - 1;
                    double f0 = 0.0;
                    __syncthreads();
                    if (run) f0 = stage1<U1, ODD>(L);
                    __syncthreads();
                    if (run) {
                        stage2(L, f0, last);
                    } else if (live) {  // this line is done: carried over
                        for (int x = L.a; x < L.a + L.own + (seg == ns_seg - 1); x++)
                            L.O[x * L.st] = L.E[x * L.st];
                    }
                    // the last L row, which the MLT sweep does not touch (:104)
                    if (pr)
                        for (int iP = nt - 1 - tid; iP < P; iP += nt) {
                            const double v = S[iP * Rs + R - 1];
                            F[iP * Rs + R - 1] = k == 0 ? v * a.G[g(iP, R - 1)] : v;
                        }
                    __syncthreads();
                    double* t2 = S;
                    S = F;
                    F = t2;
                }
            }
        }
        for (int i = tid; i < PR; i += nt) {
            const int iP = i / R, iR = i - iP * R;
            a.psd[g(iP, iR)] = S[iP * Rs + iR];
        }
        __syncthreads();
    }
}

// Launch shapes: cells of a segment, longer where the lines would need more
// threads than a CTA has, and the kernel for that many threads.
//
// Contracted form.  11 cells, 512 threads (125 registers; stage 1 in groups of 6:
// 23.2 ms at 48 x 101 x 101 x 16, of 4 28.8, of 12 34.0, spilling; a window shifted
// face by face 29.8).  Below 1200 points a pass waits for the slices of the most
// sub-steps: 5 cells and two slices on an SM, 24 x 25 x 31 x 31 alone (and per
// pass of three runs at once) 2.7 (1.08) ms, against 2.8 (1.14) with four
// slices, 2.2 (2.22) with 2 cells and one slice.  Around the line, 5 cells against
// 11: 961 slices, 24 x 32 3.07 (1.77) against 4.61 (1.81), 24 x 48 3.80 (2.14) against 4.50
// (2.54), and beyond it 24 x 51 3.84 (2.11) against 5.59 (2.36), 36 x 50 5.16 (5.11)
// against 9.20 (5.25); 3721 slices, 24 x 40 7.14 (7.09) against 6.42 (6.34), 24 x 48 7.52
// (7.48) against 9.15 (9.10), and beyond it 30 x 42 14.6 (14.6) against 8.40 (7.79), 36 x 50
// 19.3 (19.2) against 18.3 (18.3): with slices as few, one run would have 5 cells
// above the line as well.
//
// Exact form, one slice on an SM at a time.  Times below are of a pass alone (and
// per pass of three runs at once).
//  * Up to 2.5 slices an SM, segments of 2 cells: the shortest chain, and there are
//    not slices enough to fill the chip otherwise.  323 slices: 24 x 25 3.32 (1.38) with
//    5 cells -> 3.23 (1.36) ms, 23 x 32 3.92 (1.66) -> 3.35 (1.41), 24 x 42 5.04 (2.37) with
//    8 cells -> 4.13 (1.75); 620 slices, 22 x 19: 3.04 (1.34) with 5 cells, 2.45 (1.72) with 2.
//  * Beyond, segments as long as they may be without the chain growing much: below
//    400 points 2 cells (12 x 13 x 31 x 31 1.18 (0.51) ms, 5 cells 1.81 (0.73)), below
//    1000 5 cells (24 x 25 x 31 x 31 3.58 (1.81), 2 cells 3.37 (3.37), 8 cells 4.80 (2.48)),
//    below 1800 8 cells (24 x 51 x 31 x 31 6.03 (3.98), 5 cells 4.52 (4.49)), larger
//    ones 5 or what 512 threads take (48 x 101 x 31 x 31, 14 cells, 25.3 (25.1)).
//    Two slices on an SM slow the ones of the most sub-steps: 12 x 13 x 31 x 20 1.04 ms
//    alone with one, 1.16 with two.
//  * Up to CG_WAVE slices an SM a pass alone waits for the slices of the most
//    sub-steps, and the kernel with the shorter sub-step is taken (cg_faster): for
//    short lines that is the line-job kernel.  961 slices, this kernel against that one: 12 x 13
//    1.18 (0.51) against 1.07 (0.70) ms, 16 x 16 1.60 (0.72) against 1.39 (0.90), 22 x 19
//    3.31 (1.57) against 3.07 (2.02), 23 x 32 4.16 (2.64) against 3.90 (2.59); but 12 x 20
//    1.23 (0.56) against 1.36 (0.90), 24 x 25 3.58 (1.81) against 3.80 (2.57), 26 x 26 4.30
//    (2.74) against 4.56 (3.10), 44 x 22 7.92 (7.91) against 11.0 (7.04); from 1000 points
//    on always this one: 24 x 51 6.03 (3.98) against 6.38 (4.28), 36 x 40 9.02 (8.98) against
//    12.4 (7.72), 48 x 101 25.3 (25.1) against 40.4 (26.6).
//  * The line-job kernel keeps what it wins so to 13 slices an SM, where it has no
//    waiting left to fill: 1891 slices, 16 x 16 1.71 (1.37) against 1.60 (1.59), 22 x 19
//    3.56 (2.45) against 3.55 (3.57); 3721, 16 x 16 2.62 (2.62) against 3.12 (3.12).
//  * Else beyond CG_WAVE the slices there are decide: small ones take one more on an
//    SM for each CG_WAVE (24 x 25 x 47 x 31 4.19 (3.66) -> 3.97 (2.71) ms with two, 5.34
//    with one; 24 x 25 x 61 x 61 8.95 (8.96) -> 6.52 (6.48) with three, 13.7 with one).
//    Where registers leave no room for three, the line-job kernel is as fast or faster and
//    runs: 24 x 51 x 61 x 61 15.4 ms against 22.9 with one slice on an SM, 24 x 51 x 47 x 31
//    6.83 (6.23) against 7.44 (6.03) with two; from 1800 points on only past 1.5 CG_WAVE:
//    36 x 76 x 45 x 30 20.6 (17.0) -> 17.1 (17.0), but 36 x 76 x 61 x 31 23.0 (23.0) against
//    24.1 (24.0), and 48 x 101 x 61 x 61 93.2 against 94.2.
constexpr int CG_MAXT = 512;

int cg_sms()
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

#ifdef VERB_BUILD_CONV_EXACT
int cg_own(int P, int R, long long slices)
{
    const int n = P * R;
    if (n < 400 || 2 * slices <= 5 * (long long)cg_sms()) return 2;
    return n >= 1000 && n < 1800 ? 8 : 5;
}
constexpr int CG_STEP = 3, CG_WAVE = 8;
#else
int cg_own(int P, int R, long long) { return P * R < 1200 ? 5 : 11; }
constexpr int CG_STEP = 6;
#endif

void cg_segments(int P, int R, int own, StagedShape& s)
{
    s.own = own;
    s.segP = (P - 1 + own - 1) / own;
    s.segR = (R - 1 + own - 1) / own;
    s.threads = (std::max((R - 1) * s.segP, P * s.segR) + 31) / 32 * 32;
}

bool cg_shape(int P, int R, long long slices, StagedShape& s)
{
    for (int own = cg_own(P, R, slices); own <= CG_MAX_OWN; own += CG_STEP) {
        cg_segments(P, R, own, s);
        if (s.threads <= CG_MAXT) return true;
    }
    return false;
}

typedef void (*StagedKernel)(ConvArgs, int, int);
StagedKernel cg_kernel(int P, int R, const StagedShape& s, bool odd = false)
{
#ifdef VERB_BUILD_CONV_EXACT
    StagedKernel fn = convection_staged_kernel<3, CG_MAXT, 1>;
    if (s.threads <= 320) fn = convection_staged_kernel<3, 320, 1>;
    if (s.threads <= 160) fn = convection_staged_kernel<3, 160, 2>;
#else
    StagedKernel fn = odd ? convection_staged_kernel<6, CG_MAXT, 1, true>
                          : convection_staged_kernel<6, CG_MAXT, 1>;
    if (P * R < 1200 && s.threads <= 160)
        fn = odd ? convection_staged_kernel<3, 160, 2, true> : convection_staged_kernel<3, 160, 2>;
#endif
    allow_max_dynamic_smem((const void*)fn);
    return fn;
}

// CTAs that an SM can hold
int cg_resident(int P, int R, long long slices)
{
    int per = 0;
    StagedShape s;
    if (!cg_shape(P, R, slices, s)) return 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, cg_kernel(P, R, s), s.threads, cg_smem(P, R));
    return std::max(per, 1);
}

#ifdef VERB_BUILD_CONV_EXACT
// us of a sub-step of one slice with segments of 2 or 5 cells: by the warps that a
// sweep puts on a scheduler.  Measured for 2 cells: 6.0 us (12 x 13: one), 6.7 (17 x 17:
// one and two), 7.4 (20 x 20), 9.1 (24 x 25: three), 11.4 (30 x 30: four); for 5: 9.1
// (20 x 24), 10.3 (26 x 26: one and two), 11.4 (30 x 30: two), 13.3 (13 x 90: three).
double cg_chain(int P, int R, const StagedShape& s)
{
    const double two[4] = {3.03, 3.7, 4.6, 5.7}, five[4] = {4.55, 5.7, 6.8, 8.0};
    double t = 0.0;
    for (int threads : {(R - 1) * s.segP, P * s.segR}) {
        const int w = ((threads + 31) / 32 + 3) / 4;  // 1 .. 4: up to CG_MAXT threads
        t += (s.own == 2 ? two : five)[w - 1];
    }
    return t;
}
#endif

// Whether this kernel is the faster one for so many slices (the contracted form
// always is: 1.2 to 4 times from 12 x 13 to 48 x 101, 961 and 3721 slices)
bool cg_faster(int P, int R, long long slices)
{
#ifdef VERB_BUILD_CONV_EXACT
    const long long n = (long long)P * R, sms = cg_sms();
    if (n >= 1000) return 2 * slices <= (n < 1800 ? 2 : 3) * CG_WAVE * sms;
    StagedShape s;
    cg_shape(P, R, slices, s);
    if (slices <= 13 * sms && conv_lines_chain(P, R) < cg_chain(P, R, s)) return false;
    return slices <= CG_WAVE * sms || cg_resident(P, R, slices) >= 3;
#else
    return true;
#endif
}

}  // namespace
}  // namespace VERB_STAGED_NS

using namespace VERB_STAGED_NS;

int VERB_STAGED(conv_staged_check)(int P, int R, long long slices)
{
    if (P < 11 || R < 11) return VERB_ERR_SIZE;
    StagedShape s;
    if (!cg_shape(P, R, slices, s) ||
        cg_smem(P, R) > allow_max_dynamic_smem((const void*)cg_kernel(P, R, s)))
        return VERB_ERR_SIZE;
    return cg_faster(P, R, slices) ? VERB_OK : VERB_ERR_SIZE;
}

size_t VERB_STAGED(conv_staged_scratch_doubles)(int P, int R) { return (cg_scratch(P, R) + 1) & ~(size_t)1; }

int VERB_STAGED(conv_staged_ctas)(int P, int R, long long slices)
{
    const int sms = cg_sms();
    long long per = cg_resident(P, R, slices);
#ifdef VERB_BUILD_CONV_EXACT
    per = std::min(per, (slices + CG_WAVE * sms - 1) / (CG_WAVE * sms));
#endif
    return (int)std::min(sms * per, slices);
}

// The contracted form's second launch finds no slice as a rule.  Three runs at once,
// without it and with it: 48 x 101 x 101 x 16 23.38 -> 23.44 ms a pass, 24 x 25 x 31 x 31 1.066
// -> 1.067, 42 x 15 x 20 x 8 1.38 -> 1.41, 12 x 13 x 31 x 31 0.436 -> 0.451 (it waits behind the
// other streams' blocks).  Its faces in the first launch, behind a branch, cost 5 % at
// 48 x 101 x 101 x 16 and 3 % at 24 x 25 x 31 x 31; a call for the whole slice there 1 to 5 %.
void VERB_STAGED(launch_convection_staged)(const ConvArgs& a, int nctas, cudaStream_t st)
{
    StagedShape s;
    cg_shape(a.d.P, a.d.R, (long long)a.d.V * a.d.K, s);
    const StagedKernel fn = cg_kernel(a.d.P, a.d.R, s);
    fn<<<nctas, s.threads, cg_smem(a.d.P, a.d.R), st>>>(a, s.segP, s.segR);
#ifndef VERB_BUILD_CONV_EXACT
    // (few blocks, of the same shape as the first launch's: another split of an SM's
    // shared memory would have to wait for other streams' blocks to leave it)
    cg_kernel(a.d.P, a.d.R, s, true)<<<std::min(nctas, 16), s.threads, cg_smem(a.d.P, a.d.R), st>>>(
        a, s.segP, s.segR);
#endif
}

}  // namespace verb
