// Radial Kalman-filter assimilation, batched over (P,V,K) columns.
//
// Reference: runKalmanFilterDiffusion1D (src/DataAssimilationDiffusion.cpp:151-253),
// getModelMatrixDiffusion1D (src/DataAssimilationHelper.cpp:174-198),
// convertToObservationSpace (:271-305) and runKalmanFilter
// (src/DataAssimilation.cpp:18-77).  Per column, with n = R:
//   A, B  = the radial operator with zero sources/losses (A's last-row
//           sub-diagonal is dropped by CalculationMatrix::toMatrix2D,
//           src/Matrix.cpp:6495-6575, and that is kept here)
//   F     = B A^-1          (trans_solve: X A = B)
//   Pf    = F Pa F^T + Q,   Q = model_error I,  Pa0 = 5 model_error I
//   K     = Pf H^T (H Pf H^T + R)^-1,  R = obs_error I
//   x    += K (y - H x);    Pa = Pf - K H Pf
// H selects the finite observations; with none, K = 0 (the reference's dummy
// one-row H of zeros), so x is unchanged and Pa = Pf.
//
// One persistent CTA processes one column at a time, F and T = F Pa in shared
// memory (T in a global workspace where two n x n buffers do not fit).  The two
// n^3 products run on the FP64 matrix instruction: a warp holds the right-hand
// operand of eight columns in registers and runs down the rows.  F comes from n
// tridiagonal solves with A^T (O(n^2)), the gain from an LU with partial
// pivoting of the m x m innovation covariance, and the last product takes the
// observed rows of Pf where they are.  FP64 throughout, every output one chain
// of fused multiply-adds in ascending k.
//
// Bound by the serial chains around the products (Thomas factors and the n
// substitutions, one division after another).  48 x 101 x 31 x 31 at one MLT,
// whole calls: 3.0 -> 0.81 ms (with the operands in a global workspace, scalar
// tiles, one thread forming the operator and the observation list, and the
// observations of every MLT copied to the device).
#include "dmma.cuh"
#include "verb_internal.cuh"

namespace verb {

namespace {

constexpr int KF_K4 = 32;  // k steps of four: R <= 128

// 8-row tiles of an n x n operand, and its row pitch: 4 mod 16 doubles, so that
// an 8 x 4 operand read fills the banks once
__host__ __device__ inline int kf_tiles(int n) { return (n + 7) / 8; }
__host__ __device__ inline int kf_ld(int n) { return (8 * kf_tiles(n) + 11) / 16 * 16 + 4; }
__host__ __device__ inline size_t kf_buf(int n) { return (size_t)8 * kf_tiles(n) * kf_ld(n); }

// column tile w of X = A B (A: rows x k at lda, zero padded): load(k, j) is B
template <class Load, class Store>
__device__ __forceinline__ void kf_product(int n, const double* A, int lda, int w, Load load,
                                           Store store)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, h = lane & 3;
    const int nk = (n + 3) / 4;
    double b[KF_K4];
#pragma unroll
    for (int k = 0; k < KF_K4; k++) b[k] = k < nk ? load(4 * k + h, 8 * w + g) : 0.0;
    __syncthreads();  // the operand is in registers: its buffer may be written
    for (int r = 0; r < kf_tiles(n); r++) {
        double c[2] = {0.0, 0.0};
        const double* ar = A + (size_t)(8 * r + g) * lda + h;
#pragma unroll
        for (int k = 0; k < KF_K4; k++)
            if (k < nk) dmma(c[0], c[1], ar[4 * k], b[k]);
        store(8 * r + g, 8 * w + 2 * h, c);
    }
}

__global__ void __launch_bounds__(512) kf_kernel(KFArgs a, int t_global)
{
    extern __shared__ __align__(16) double sm[];
    const Dims d = a.d;
    const int n = d.R, tid = threadIdx.x, nt = blockDim.x, w = tid >> 5;
    const size_t RR = (size_t)n * n;
    const int ld = kf_ld(n);
    const size_t buf = kf_buf(n);
    double* F = sm;                                   // F, then Pf
    double* T = t_global ? a.work + (size_t)blockIdx.x * (buf + RR) : F + buf;  // F Pa, then K
    double* Sg = a.work + (size_t)blockIdx.x * (buf + RR) + buf;  // S where T has no room for it
    double* x = t_global ? F + buf : F + 2 * buf;     // [n] forecast
    double* lo = x + n;                               // A^T Thomas: sub, diag, sup
    double* dg = lo + n;
    double* up = dg + n;
    double* bd = up + n;                              // diag of B
    double* gam = bd + n;                             // Thomas factors of A^T
    double* bet = gam + n;
    double* y = bet + n;                              // innovations [n]
    int* oidx = (int*)(y + n);                        // observed indices [n]
    __shared__ int s_col, s_m, s_any, s_nan, s_piv;
    const size_t VK = (size_t)d.V * d.K;
    const int ncols = a.p_index >= 0 ? (int)VK : (int)(d.P * VK);

    for (;;) {
        if (threadIdx.x == 0) s_col = atomicAdd(a.ticket, 1);
        __syncthreads();
        const int col = s_col;
        __syncthreads();
        if (col >= ncols) break;
        const size_t p = a.p_index >= 0 ? (size_t)a.p_index : (size_t)col / VK;
        const size_t vk = a.p_index >= 0 ? (size_t)col : (size_t)col % VK;
        const size_t cid = a.p_index >= 0 ? vk : p * VK + vk;  // Pa holds the columns in use
        double* Pa = a.Pa + cid * RR;
        auto gi = [&](int r) { return (p * d.R + r) * VK + vk; };

        // forecast, observations and the radial operator (zero sources/losses)
        if (tid == 0) s_any = 0;
        for (int r = tid; r < n; r += nt) {
            x[r] = a.psd[gi(r)];
            // rows of A (getCalculationMatrix1DDiffusion with S = Loss = 0)
            const double sc = a.dll_scale;
            double al = 0, ad = 0, au = 0, b = 0;
            if (r == 0) {
                const double dh = a.Rg[gi(1)] - a.Rg[gi(0)];
                if (a.Ll_t == VERB_BC_CONSTANT_VALUE) { ad = 1; au = 0; }
                else { ad = 1 / dh; au = -1 / dh; }
            } else if (r == n - 1) {
                const double dh = a.Rg[gi(r)] - a.Rg[gi(r - 1)];
                if (a.Lu_t == VERB_BC_CONSTANT_VALUE) { ad = 1; al = 0; }
                else { ad = 1 / dh; al = -1 / dh; }
            } else {
                const double xm = a.Rg[gi(r - 1)], x0 = a.Rg[gi(r)], xp = a.Rg[gi(r + 1)];
                double Dm = a.DLL[gi(r - 1)], D0 = a.DLL[gi(r)], Dp = a.DLL[gi(r + 1)];
                if (sc != 1.0) { Dm *= sc; D0 *= sc; Dp *= sc; }
                const double Gm = a.G[gi(r - 1)], G0 = a.G[gi(r)], Gp = a.G[gi(r + 1)];
                ad += 1.0 / a.dt;
                b += 1.0 / a.dt;
                ad -= 0.0;
                {
                    double dh1 = x0 - xm, dh21 = x0 - xp, dh22 = xm - x0;
                    double cp = -0.5 / G0 / dh1;
                    ad += +cp / dh21 * D0 * G0;
                    au += -cp / dh21 * D0 * G0;
                    al += -cp / dh22 * Dm * Gm;
                    ad += +cp / dh22 * Dm * Gm;
                }
                {
                    double dh1 = x0 - xp, dh21 = x0 - xm, dh22 = xp - x0;
                    double cp = -0.5 / G0 / dh1;
                    ad += +cp / dh21 * D0 * G0;
                    al += -cp / dh21 * D0 * G0;
                    au += -cp / dh22 * Dp * Gp;
                    ad += +cp / dh22 * Dp * Gp;
                }
            }
            if (r == n - 1) al = 0.0;  // toMatrix2D drops the last row's sub-diagonal
            // A^T: sub-diagonal of A^T row r is A[r-1][r] = up[r-1]; super is A[r+1][r]
            dg[r] = ad;
            bd[r] = b;
            up[r] = au;   // A's super-diagonal
            lo[r] = al;   // A's sub-diagonal
        }
        // the finite observations in order, by the last warp
        if (w == (nt >> 5) - 1) {
            const int lane = tid & 31;
            int m = 0;
            for (int r0 = 0; r0 < n; r0 += 32) {
                const int r = r0 + lane;
                const double o = r < n ? a.obs[gi(r)] : 0.0;
                const bool seen = r < n && isfinite(o);
                const unsigned bal = __ballot_sync(0xffffffffu, seen);
                if (seen) {
                    const int i = m + __popc(bal & ((1u << lane) - 1));
                    oidx[i] = r;
                    y[i] = o;
                }
                m += __popc(bal);
            }
            if (lane == 0) s_m = m;
        }
        for (size_t e = tid; e < buf; e += nt) F[e] = 0.0;  // padding included
        __syncthreads();
        if (tid == 0) {
            // Thomas factors of A^T: sub'[r] = up[r-1], sup'[r] = lo[r+1]
            double bt = dg[0];
            bet[0] = bt;
            gam[0] = 0;
            for (int r = 1; r < n; r++) {
                const double g = lo[r] / bt;  // sup'[r-1] = lo[r]
                bt = dg[r] - up[r - 1] * g;
                gam[r] = g;
                bet[r] = bt;
            }
        }
        // meanwhile: is Pa set (src/DataAssimilationDiffusion.cpp:213-218)
        for (size_t e = tid; e < RR; e += nt)
            if (Pa[e] != 0.0) s_any = 1;
        __syncthreads();
        const int m = s_m;

        // F = B A^-1: row i solves A^T f = b_i e_i
        for (int i = tid; i < n; i += nt) {
            double* f = F + (size_t)i * ld;
            double u = 0.0;  // and F's zeros stand above row i
            for (int r = i; r < n; r++) {
                const double rhs = (r == i) ? bd[i] : 0.0;
                u = (rhs - (r > i ? up[r - 1] * u : 0.0)) / bet[r];
                f[r] = u;
            }
            for (int r = n - 1; r >= 1; r--) {
                u = f[r - 1] - gam[r] * u;
                f[r - 1] = u;
            }
        }
        if (!s_any)
            for (int i = tid; i < n; i += nt) Pa[(size_t)i * n + i] = 5 * a.model_error;
        __syncthreads();
        // Pf = F Pa F^T + Q, Pf in F's buffer
        kf_product(
            n, F, ld, w, [&](int k, int j) { return k < n && j < n ? Pa[(size_t)k * n + j] : 0.0; },
            [&](int i, int j, const double (&c)[2]) {
                T[(size_t)i * ld + j] = c[0];
                T[(size_t)i * ld + j + 1] = c[1];
            });
        __syncthreads();
        kf_product(
            n, T, ld, w, [&](int k, int j) { return F[(size_t)j * ld + k]; },
            [&](int i, int j, const double (&c)[2]) {
                F[(size_t)i * ld + j] = i == j ? c[0] + a.model_error : c[0];
                F[(size_t)i * ld + j + 1] = i == j + 1 ? c[1] + a.model_error : c[1];
            });
        const double* Pf = F;
        __syncthreads();
        if (m == 0) {
            // no observation: x += 0 (the reference's dummy row), and the
            // NaN check still applies (src/DataAssimilation.cpp:62-67)
            bool bad = false;
            for (int i = threadIdx.x; i < n; i += blockDim.x) bad = bad || isnan(x[i]);
            if (__syncthreads_or(bad) && threadIdx.x == 0) set_error(a.status, VERB_ERR_NAN);
            for (size_t e = threadIdx.x; e < RR; e += blockDim.x) Pa[e] = Pf[e / n * ld + e % n];
            __syncthreads();
            continue;
        }
        // PfHt (n x m) and S = H Pf H^T + R (m x m)
        double* Kg = T;
        double* Sm = (size_t)n * m + (size_t)m * m <= buf ? T + (size_t)n * m : Sg;
        for (int e = threadIdx.x; e < n * m; e += blockDim.x) {
            const int i = e / m, c = e % m;
            Kg[(size_t)i * m + c] = Pf[(size_t)i * ld + oidx[c]];
        }
        for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
            const int r = e / m, c = e % m;
            // S^T, since K S = PfHt is solved as S^T K^T = PfHt^T
            Sm[(size_t)r * m + c] = Pf[(size_t)oidx[c] * ld + oidx[r]] + (r == c ? a.obs_error : 0.0);
        }
        for (int c = threadIdx.x; c < m; c += blockDim.x) y[c] = y[c] - x[oidx[c]];
        __syncthreads();
        // K S = PfHt  <=>  S^T K^T = PfHt^T: LU of S^T (held in Sm) with partial
        // pivoting; each row of Kg is one right-hand side.
        for (int k = 0; k < m; k++) {
            if (w == 0) {
                // first maximum of |column k|; a leading NaN stays, others never are
                const int lane = tid & 31;
                const double lead = fabs(Sm[(size_t)k * m + k]);
                double best = -1.0;
                int pr = m;
                for (int r = k + lane; r < m; r += 32) {
                    const double v = fabs(Sm[(size_t)r * m + k]);
                    if (v > best) { best = v; pr = r; }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    const double v = __shfl_xor_sync(0xffffffffu, best, o);
                    const int q = __shfl_xor_sync(0xffffffffu, pr, o);
                    if (v > best || (v == best && q < pr)) { best = v; pr = q; }
                }
                if (lane == 0) s_piv = lead != lead || pr >= m ? k : pr;
            }
            __syncthreads();
            const int pr = s_piv;
            if (pr != k) {
                for (int c = threadIdx.x; c < m; c += blockDim.x) {
                    const double t = Sm[(size_t)k * m + c];
                    Sm[(size_t)k * m + c] = Sm[(size_t)pr * m + c];
                    Sm[(size_t)pr * m + c] = t;
                }
                for (int i = threadIdx.x; i < n; i += blockDim.x) {
                    const double t = Kg[(size_t)i * m + k];
                    Kg[(size_t)i * m + k] = Kg[(size_t)i * m + pr];
                    Kg[(size_t)i * m + pr] = t;
                }
            }
            __syncthreads();
            const double piv = Sm[(size_t)k * m + k];
            for (int e = threadIdx.x; e < (m - k - 1) * (m - k); e += blockDim.x) {
                const int r = k + 1 + e / (m - k), c = k + e % (m - k);
                if (c == k) continue;
                const double l = Sm[(size_t)r * m + k] / piv;
                Sm[(size_t)r * m + c] -= l * Sm[(size_t)k * m + c];
            }
            for (int e = threadIdx.x; e < (m - k - 1) * n; e += blockDim.x) {
                const int r = k + 1 + e / n, i = e % n;
                const double l = Sm[(size_t)r * m + k] / piv;
                Kg[(size_t)i * m + r] -= l * Kg[(size_t)i * m + k];
            }
            __syncthreads();
            for (int r = k + 1 + threadIdx.x; r < m; r += blockDim.x)
                Sm[(size_t)r * m + k] = Sm[(size_t)r * m + k] / piv;
            __syncthreads();
        }
        // back substitution per row of Kg (each row i is one right-hand side)
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            double* kr = Kg + (size_t)i * m;
            for (int r = m - 1; r >= 0; r--) {
                double s = kr[r];
                for (int c = r + 1; c < m; c++) s -= Sm[(size_t)r * m + c] * kr[c];
                kr[r] = s / Sm[(size_t)r * m + r];
            }
        }
        __syncthreads();
        // x += K (y - H x); NaN check (src/DataAssimilation.cpp:53-67)
        if (threadIdx.x == 0) s_nan = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            double s = 0.0;
            for (int c = 0; c < m; c++) s += Kg[(size_t)i * m + c] * y[c];
            const double v = x[i] + s;
            if (isnan(v)) s_nan = 1;
            a.psd[gi(i)] = v;
        }
        __syncthreads();
        if (tid == 0 && s_nan) set_error(a.status, VERB_ERR_NAN);
        // Pa = Pf - K (H Pf): the rows of Pf at the observed indices
        for (size_t e = tid; e < RR; e += nt) {
            const int i = (int)(e / n), j = (int)(e % n);
            double v = 0.0;
            for (int c = 0; c < m; c++) v = fma(Kg[(size_t)i * m + c], Pf[(size_t)oidx[c] * ld + j], v);
            Pa[e] = Pf[(size_t)i * ld + j] - v;
        }
        __syncthreads();
    }
}

}  // namespace

namespace {

int kf_max_smem()
{
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

size_t kf_smem(int n, int bufs)
{
    return (bufs * kf_buf(n) + 8 * (size_t)n) * sizeof(double) + n * sizeof(int);
}

// T in the workspace where two buffers do not fit (R > 112)
int kf_t_global(int n) { return kf_smem(n, 2) + 1024 > (size_t)kf_max_smem(); }

}  // namespace

int kf_ctas(const Dims& d, int p_index)
{
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    allow_max_dynamic_smem((const void*)kf_kernel);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kf_kernel, 32 * kf_tiles(d.R),
                                                  kf_smem(d.R, kf_t_global(d.R) ? 1 : 2));
    const size_t cols = p_index >= 0 ? (size_t)d.V * d.K : (size_t)d.P * d.V * d.K;
    const size_t nctas = (size_t)sms * (per < 1 ? 1 : per);
    return (int)(nctas < cols ? nctas : cols);
}

size_t kf_work_doubles(int R) { return kf_buf(R) + (size_t)R * R; }

void launch_kf(const KFArgs& a, int nctas, cudaStream_t s)
{
    const int n = a.d.R, tg = kf_t_global(n);
    cudaMemsetAsync(a.ticket, 0, sizeof(int), s);
    allow_max_dynamic_smem((const void*)kf_kernel);
    kf_kernel<<<nctas, 32 * kf_tiles(n), kf_smem(n, tg ? 1 : 2), s>>>(a, tg);
}

}  // namespace verb
