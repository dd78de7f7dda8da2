// Radial diffusion in L: batched Thomas solves, one thread per (P,V,K) line.
//
// Compiled with -fmad=false: every operation below is the reference's
// operation in the reference's order, so results are bit-identical to
// Diffusion_1D (src/Diffusion_1D.cpp:43-184, src/MatrixSolver.cpp:353-404,
// 689-720) on the same inputs.
//
// The tridiagonal matrix depends only on L*, D_LL, G_radial, Losses_radial
// and dt, which change at most hourly; its Thomas recurrence (gam_j, bet_j and
// the sub-diagonal a_j) is cached in HBM as [R][lines] (coalesced along lines).
// radial_solve_kernel is the per-step pass: it forms RHS = B f + C, runs the
// forward sweep writing u_j into PSD in place, then the back substitution; in
// a step whose matrix changed (FACTOR) it forms the rows and the recurrence on
// the way and writes the cache.
//
// Bound by HBM (a step: f twice, a, bet, gam and twice the stores, 56 B a point;
// with FACTOR 96 B).  A thread's loads are taken RD_ROWS rows at a time before
// the recurrence uses them (one row's loads in flight at a time: 130 us for the
// kernel at 48 x 101 x 101 x 16, 60 us here; a factor kernel before it 146 us, the two
// in one 166 us here), and the quotients of a row share the reciprocals of its grid
// spacings (exact_div.cuh).  What a caller sees of a pass with new coefficients:
// 318 -> 202 us for one run, 195 -> 163 us a pass for three at once.
#include "exact_div.cuh"
#include "verb_internal.cuh"

namespace verb {

namespace {

struct Row {
    double lo, d, up;
};

// One interior row of getCalculationMatrix1DDiffusion (src/Diffusion_1D.cpp:161-178):
// A_ii = 1/dt - Loss, then SecondDerivativeApproximation_1D twice
// (src/MatrixSolver.cpp:353-404) with multiplicator -0.5, ("x_left", "x_right")
// and ("x_right", "x_left").  a = x0 - xm, b = x0 - xp and their reciprocals;
// the reference's other spacings are their negatives, and a negated divisor or
// dividend negates the quotient exactly.
__device__ __forceinline__ Row radial_interior_row(double a, double ra, double b, double rb,
                                                   double Dm, double D0, double Dp, double Gm,
                                                   double G0, double Gp, double loss, double dt)
{
    Row w;
    w.lo = 0.0;
    w.up = 0.0;
    w.d = 0.0;
    w.d += 1.0 / dt;
    w.d -= loss;
    const double c0 = div_by(-0.5, G0, recip(G0));
    {
        const double cp = div_by(c0, a, ra);
        const double q = div_by(cp, b, rb), t = div_by(cp, a, ra);
        w.d += q * D0 * G0;
        w.up += -q * D0 * G0;
        w.lo += t * Dm * Gm;
        w.d += -t * Dm * Gm;
    }
    {
        const double cp = div_by(c0, b, rb);
        const double q = div_by(cp, a, ra), t = div_by(cp, b, rb);
        w.d += q * D0 * G0;
        w.lo += -q * D0 * G0;
        w.up += t * Dp * Gp;
        w.d += -t * Dp * Gp;
    }
    return w;
}

// Rows loaded at a time, with five blocks of 128 an SM: 3 rows with FACTOR (1 row
// 267 us, 2 209, 4 at four blocks 290, 8 at three 291 for the pass below), 8 without.
constexpr int RD_ROWS = 8, RF_ROWS = 3;

template <bool FACTOR>
__global__ void __launch_bounds__(128, 5) radial_solve_kernel(RadialArgs a)
{
    constexpr int U = FACTOR ? RF_ROWS : RD_ROWS;
    const Dims d = a.d;
    const size_t nlines = (size_t)d.P * d.V * d.K;
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nlines) return;
    const size_t vk_n = (size_t)d.V * d.K;
    const size_t p = q / vk_n, vk = q - p * vk_n;
    const size_t base = p * (size_t)d.R * vk_n + vk;
    const int n = d.R;
    const double bint = 0.0 + 1.0 / a.dt;  // matr_B[0][in] += 1.0 / dt
    const double rs = (double)a.radial_sources;
    const double sc = a.dll_scale;
    double* f = a.psd + base;
    auto Dat = [&](int r) {
        const double v = a.DLL[base + (size_t)r * vk_n];
        return sc != 1.0 ? v * sc : v;
    };

    // row 0: the lower boundary (src/Diffusion_1D.cpp:66-76, 115-137)
    double bet, up_prev = 0.0, xm = 0, x0 = 0, Dm = 0, D0 = 0, Gm = 0, G0 = 0, dl = 0, rl = 0;
    if (FACTOR) {
        xm = a.L[base];
        x0 = a.L[base + vk_n];
        Dm = Dat(0);
        D0 = Dat(1);
        Gm = a.G[base];
        G0 = a.G[base + vk_n];
        const double dh = x0 - xm;
        if (a.Ll_t == VERB_BC_CONSTANT_VALUE) {
            bet = 1;
        } else if (a.Ll_t == VERB_BC_CONSTANT_DERIVATIVE) {
            bet = 1 / dh;
            up_prev = -1 / dh;
        } else {
            set_error(a.status, VERB_ERR_BC);
            return;
        }
        dl = dh;
        rl = recip(dh);
        a.fa[q] = 0.0;
        a.fbet[q] = bet;
        a.fgam[q] = 0.0;
    } else {
        bet = a.fbet[q];
    }
    double u;
    {
        double rhs = a.Ll[q];
        rhs += 0.0 * f[0];
        u = rhs / bet;
        f[0] = u;
    }
    double rbet = FACTOR ? recip(bet) : 0.0;
    for (int r0 = 1; r0 < n; r0 += U) {
        double fr[U], lo[U], be[U], xp[U], Dp[U], Gp[U], ls[U], src[U];
#pragma unroll
        for (int i = 0; i < U; i++) {
            const int r = min(r0 + i, n - 1), r1 = min(r + 1, n - 1);
            const size_t o = base + (size_t)r * vk_n, o1 = base + (size_t)r1 * vk_n;
            fr[i] = a.psd[o];
            src[i] = a.radial_sources ? a.S[o] : 0.0;
            if (FACTOR) {
                xp[i] = a.L[o1];
                Dp[i] = Dat(r1);
                Gp[i] = a.G[o1];
                ls[i] = a.loss[o];
            } else {
                const size_t fo = (size_t)r * nlines + q;
                lo[i] = a.fa[fo];
                be[i] = a.fbet[fo];
            }
        }
#pragma unroll
        for (int i = 0; i < U; i++) {
            const int r = r0 + i;
            if (r >= n) break;
            const bool end = r == n - 1;
            const size_t fo = (size_t)r * nlines + q;
            if (FACTOR) {
                Row w;
                if (end) {
                    // last row: boundary (src/Diffusion_1D.cpp:138-159)
                    const double dh = x0 - xm;
                    w.up = 0.0;
                    if (a.Lu_t == VERB_BC_CONSTANT_VALUE) {
                        w.d = 1;
                        w.lo = 0;
                    } else if (a.Lu_t == VERB_BC_CONSTANT_DERIVATIVE) {
                        w.d = 1 / dh;
                        w.lo = -1 / dh;
                    } else {
                        set_error(a.status, VERB_ERR_BC);
                        return;
                    }
                } else {
                    const double b = x0 - xp[i], rb = recip(b);
                    w = radial_interior_row(dl, rl, b, rb, Dm, D0, Dp[i], Gm, G0, Gp[i], ls[i], a.dt);
                    xm = x0;
                    x0 = xp[i];
                    dl = -b;  // of the next row
                    rl = -rb;
                    Dm = D0;
                    D0 = Dp[i];
                    Gm = G0;
                    G0 = Gp[i];
                }
                // Thomas recurrence of tridag (src/MatrixSolver.cpp:701-703)
                const double gam = div_by(up_prev, bet, rbet);
                bet = w.d - w.lo * gam;
                rbet = recip(bet);
                a.fa[fo] = w.lo;
                a.fbet[fo] = bet;
                a.fgam[fo] = gam;
                up_prev = w.up;
                lo[i] = w.lo;
                be[i] = bet;
            }
            // RHS = C + B f (src/Diffusion_1D.cpp:66-76)
            double c, b;
            if (end) {
                c = a.Lu[q];
                b = 0.0;
            } else {
                c = 0.0;
                if (a.radial_sources) c += src[i] * rs;
                b = bint;
            }
            double rhs = c;
            rhs += b * fr[i];
            const double num = rhs - lo[i] * u;
            u = FACTOR ? div_by(num, be[i], rbet) : num / be[i];
            a.psd[base + (size_t)r * vk_n] = u;
        }
    }
    for (int r0 = n - 1; r0 >= 1; r0 -= RD_ROWS) {
        double fr[RD_ROWS], ga[RD_ROWS];
#pragma unroll
        for (int i = 0; i < RD_ROWS; i++) {
            const int r = max(r0 - i, 1);
            fr[i] = a.psd[base + (size_t)(r - 1) * vk_n];
            ga[i] = a.fgam[(size_t)r * nlines + q];
        }
#pragma unroll
        for (int i = 0; i < RD_ROWS; i++) {
            const int r = r0 - i;
            if (r < 1) break;
            double um = fr[i];
            um -= ga[i] * u;
            a.psd[base + (size_t)(r - 1) * vk_n] = um;
            u = um;
        }
    }
}

// tridag (src/MatrixSolver.cpp:689-720) on one system, single thread; gam in
// global scratch after u (u must have 2n entries).
__global__ void tridag_kernel(const double* a, const double* b, const double* c, const double* r,
                              double* u, long n)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double* gam = u + n;
    double bet;
    u[0] = r[0] / (bet = b[0]);
    for (long j = 1; j <= n - 1; j++) {
        gam[j] = c[j - 1] / bet;
        bet = b[j] - a[j] * gam[j];
        u[j] = (r[j] - a[j] * u[j - 1]) / bet;
    }
    for (long j = n - 1; j >= 1; j--) u[j - 1] -= gam[j] * u[j];
}

}  // namespace

void launch_tridag(const double* a, const double* b, const double* c, const double* r, double* u,
                   long n, cudaStream_t s)
{
    tridag_kernel<<<1, 32, 0, s>>>(a, b, c, r, u, n);
}

void launch_radial_solve(const RadialArgs& a, bool factor, cudaStream_t s)
{
    const size_t nlines = (size_t)a.d.P * a.d.V * a.d.K;
    const int tb = 128;
    const unsigned g = (unsigned)((nlines + tb - 1) / tb);
    if (factor) radial_solve_kernel<true><<<g, tb, 0, s>>>(a);
    else radial_solve_kernel<false><<<g, tb, 0, s>>>(a);
}

}  // namespace verb
