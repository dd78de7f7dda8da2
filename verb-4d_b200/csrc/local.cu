// Local (V,K) diffusion: banded LU with partial pivoting, factors cached in HBM.
//
// Reference: Diffusion_2D (src/Diffusion_2D.cpp:19-153) assembles a
// 9-diagonal operator over the unknown index in = iK*V + iV
// (AddBoundaries_2D and SecondDerivativeApproximation_2D,
// src/MatrixSolver.cpp:118-213, 439-494) and Lapack
// (src/MatrixSolver.cpp:223-340) factors it with dgbtrf (kl = ku = V+1) and
// solves with dgbtrs once per diffusion sub-step.  With LU_CACHING the
// factors are kept per (P,R) system and only recomputed when the local
// coefficients change (src/VERB4D_Solver.cpp:1091-1096).
//
// Kernels:
//  * local_factor_kernel: one CTA per system, where local_factor_blk_kernel does
//    not run (V <= 7, with FP32 factors V <= 15, and grids of more than 65535
//    systems: factor_by_panels).  Rows of A are assembled on the device with the
//    reference's operation order (bit-identical matrix) and factored by the unblocked banded LU of LAPACK's xGBTF2 (partial pivoting,
//    multipliers scaled by the reciprocal pivot, rank-1 updates as fused
//    multiply-adds).
//    The active (kl+1) x (kv+1) window lives in shared memory as a circular
//    buffer over rows and columns.  Output: L multipliers (Lf, column j
//    contiguous), U columns (Uf, rows j-kv..j contiguous) and 0-based pivots.
//  * local_rows_kernel + local_factor_blk_kernel: the same factorisation by
//    panels of columns, for every other grid: the rows are assembled
//    beforehand and parked in the L columns they precede, a panel's pivot
//    chain and the update by the previous panel run side by side, and the
//    update is on the FP64 matrix instruction.
//  * local_rhs_kernel / local_store_kernel: tile transposes between the PSD
//    slab [V][K] and the unknown order, forming RHS = B o f + C.
//  * local_solve_kernel: one warp per system, the forward (L, interleaved row
//    swaps as in xGBTRS) and backward (U, column-oriented as in xTBSV)
//    substitutions.  The solution window lives in shared memory; the factor
//    columns stream through a per-warp cp.async ring so that each warp keeps
//    several columns in flight.  This kernel moves the whole factor cache
//    once per sub-step and is HBM-bound.  local_solve_rw_kernel keeps the
//    solution window in registers instead.
//
// All arithmetic follows the CPU restatement of xGBTF2/xGBTRS/xTBSV operation
// by operation without FMA contraction (the file is compiled with
// -fmad=false) except the factorisation's rank-1 update, which both compute
// as one fused multiply-add per element (fma()), so factors, pivots and
// solutions are bit-identical to it.
#include "dmma.cuh"
#include "exact_div.cuh"
#include "verb_internal.cuh"

#include <type_traits>

namespace verb {

namespace {

// slot of diagonal offset (dx,dy): offset = dy*nx + dx
__device__ __forceinline__ int dslot(int dx, int dy) { return (dy + 1) * 3 + (dx + 1); }

struct SysView {
    const double *x, *y, *Dxx, *Dyy, *Dxy, *Dyx, *G, *S, *loss;
    const double *xl, *xu, *yl, *yu;
    int nx, ny;      // logical grid of the system (ny = K - k0)
    int ld;          // stride of the V index in the [V][K] fields (K)
    bool trimmed;    // lower K edge is the loss-cone edge (ConstantValue 0)
};

__device__ __forceinline__ int sys_k0(const LocalArgs& a, int sys) { return a.k0 ? a.k0[sys] : 0; }

// first unknown of system sys in the work / pivot arrays
__device__ __forceinline__ size_t sys_uoff(const LocalArgs& a, int sys)
{
    return a.uoff ? (size_t)a.uoff[sys] : (size_t)sys * a.d.V * a.d.K;
}

__device__ __forceinline__ SysView sys_view(const LocalArgs& a, int sys)
{
    const int k0 = sys_k0(a, sys);
    const size_t base = (size_t)sys * a.d.V * a.d.K + k0;
    SysView v;
    v.x = a.Vg + base;
    v.y = a.Kg + base;
    v.Dxx = a.DVV + base;
    v.Dyy = a.DKK + base;
    v.Dxy = a.DVK + base;
    v.Dyx = a.DKV + base;
    v.G = a.G + base;
    v.S = a.S + base;
    v.loss = a.loss + base;
    v.xl = a.Vl + (size_t)sys * a.d.K + k0;
    v.xu = a.Vu + (size_t)sys * a.d.K + k0;
    v.yl = a.Kl + (size_t)sys * a.d.V;
    v.yu = a.Ku + (size_t)sys * a.d.V;
    v.nx = a.d.V;
    v.ny = a.d.K - k0;
    v.ld = a.d.K;
    v.trimmed = k0 > 0;
    return v;
}

// SecondDerivativeApproximation_2D (src/MatrixSolver.cpp:439-494) adding into
// the 9 diagonal values of row (ix,iy).
__device__ __forceinline__ void sda2(double* r, const SysView& v, int ix, int iy, int dx1, int dy1,
                                     int dx2, int dy2, const double* D, double mult)
{
    const int ld = v.ld;
#define P2(a, b) ((a) * ld + (b))
    const double x0 = v.x[P2(ix, iy)] + v.y[P2(ix, iy)];
    const double x1 = v.x[P2(ix + dx1, iy + dy1)] + v.y[P2(ix + dx1, iy + dy1)];
    const double x2 = v.x[P2(ix + dx2, iy + dy2)] + v.y[P2(ix + dx2, iy + dy2)];
    const double x12 = v.x[P2(ix + dx1 + dx2, iy + dy1 + dy2)] + v.y[P2(ix + dx1 + dx2, iy + dy1 + dy2)];
    const double dh1 = x0 - x1;
    const double dh21 = x0 - x2;
    const double dh22 = x1 - x12;
    const double G0 = v.G[P2(ix, iy)], G1 = v.G[P2(ix + dx1, iy + dy1)];
    const double D0 = D[P2(ix, iy)], D1 = D[P2(ix + dx1, iy + dy1)];
    const double cp = mult / G0 / dh1;
    r[dslot(0, 0)] += +cp / dh21 * D0 * G0;
    r[dslot(dx2, dy2)] += -cp / dh21 * D0 * G0;
    r[dslot(dx1, dy1)] += -cp / dh22 * D1 * G1;
    r[dslot(dx1 + dx2, dy1 + dy2)] += +cp / dh22 * D1 * G1;
#undef P2
}

// One row of matr_A (src/Diffusion_2D.cpp:68-130).  Returns 0 or VERB_ERR_BC.
__device__ int assemble_row(const SysView& v, int types[4], double dt, int in, double r[9])
{
    const int nx = v.nx, ny = v.ny, ld = v.ld;
    const int ix = in % nx, iy = in / nx;
    const int p = ix * ld + iy;
#pragma unroll
    for (int s = 0; s < 9; s++) r[s] = 0.0;
    int t = -1, s1 = 0;
    double dh = 0.0;
    if (ix == 0 && nx >= 3) {
        t = types[0];
        s1 = dslot(1, 0);
        dh = v.x[p + ld] - v.x[p];
    } else if (ix == nx - 1 && nx >= 3) {
        t = types[1];
        s1 = dslot(-1, 0);
        dh = v.x[p] - v.x[p - ld];
    } else if (iy == 0 && ny >= 3) {
        t = v.trimmed ? VERB_BC_CONSTANT_VALUE : types[2];
        s1 = dslot(0, 1);
        dh = v.y[p + 1] - v.y[p];
    } else if (iy == ny - 1 && ny >= 3) {
        t = types[3];
        s1 = dslot(0, -1);
        dh = v.y[p] - v.y[p - 1];
    }
    if (t >= 0) {
        if (t == VERB_BC_CONSTANT_VALUE) {
            r[4] = 1;
            r[s1] = 0;
        } else if (t == VERB_BC_CONSTANT_DERIVATIVE) {
            r[4] = 1 / dh;
            r[s1] = -1 / dh;
        } else {
            return VERB_ERR_BC;
        }
        return 0;
    }
    r[4] += 1.0 / dt;
    r[4] -= v.loss[p];
    if (nx >= 3) {
        sda2(r, v, ix, iy, -1, 0, 1, 0, v.Dxx, -0.5);
        sda2(r, v, ix, iy, 1, 0, -1, 0, v.Dxx, -0.5);
    }
    if (ny >= 3) {
        sda2(r, v, ix, iy, 0, -1, 0, 1, v.Dyy, -0.5);
        sda2(r, v, ix, iy, 0, 1, 0, -1, v.Dyy, -0.5);
    }
    if (nx >= 3 && ny >= 3) {
        sda2(r, v, ix, iy, 0, -1, 1, 0, v.Dxy, -0.25);  // y_left,  x_right
        sda2(r, v, ix, iy, 0, 1, -1, 0, v.Dxy, -0.25);  // y_right, x_left
        sda2(r, v, ix, iy, 0, -1, -1, 0, v.Dxy, -0.25); // y_left,  x_left
        sda2(r, v, ix, iy, 0, 1, 1, 0, v.Dxy, -0.25);   // y_right, x_right
        sda2(r, v, ix, iy, -1, 0, 0, 1, v.Dyx, -0.25);  // x_left,  y_right (d/dy Dyx d/dx)
        sda2(r, v, ix, iy, 1, 0, 0, -1, v.Dyx, -0.25);  // x_right, y_left
        sda2(r, v, ix, iy, -1, 0, 0, -1, v.Dyx, -0.25); // x_left,  y_left
        sda2(r, v, ix, iy, 1, 0, 0, 1, v.Dyx, -0.25);   // x_right, y_right
    }
    return 0;
}

__device__ __forceinline__ bool skip_system(const LocalArgs& a, int sys)
{
    if (a.sel && !(a.sel[sys] & a.sel_mask)) return true;
    if (a.k0 && a.d.K - a.k0[sys] < 3) return true;  // trimmed below a solvable grid
    if (a.include_boundary) return false;
    const int r = sys % a.d.R;
    return r == 0 || r == a.d.R - 1;
}

constexpr int FACT_THREADS = 512;
constexpr int FACT_COLS = 7;  // columns per lane in the rank-1 update: kv + 1 <= 224 (V <= 111)
// Assembled rows are staged in a ring of STAGE_ROWS rows, a whole ring at a
// time (one row per thread), when the window's next entering row reaches a
// multiple of STAGE_ROWS.  256 rows (18 KB) still fit beside the window at
// V = 111.
constexpr int STAGE_ROWS = 256;

// The factorisation always runs in FP64 (pivots and multipliers as LAPACK's);
// T is the storage type of the factors: double, or float for the
// mixed-precision form, whose solves are refined in FP64.
template <typename T>
__global__ void __launch_bounds__(FACT_THREADS) local_factor_kernel(LocalArgs a)
{
    extern __shared__ double sm[];
    const int sys = blockIdx.x;
    if (skip_system(a, sys)) return;
    const int nx = a.d.V;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const int kl = a.kl, ku = a.kl, kv = a.kv;
    const int RW = kl + 1;          // window rows
    const int CW = kv + 1;          // window columns (row pitch)
    double* W = sm;                 // [RW][CW]
    double* mult = W + (size_t)RW * CW;  // [RW]
    double* colj = mult + RW;       // [RW]
    double* stage = colj + RW;      // [STAGE_ROWS][9]
    __shared__ int s_jp;
    __shared__ double s_piv;
    const SysView v = sys_view(a, sys);
    int types[4] = {a.Vl_t, a.Vu_t, a.Kl_t, a.Ku_t};
    const bool f32 = sizeof(T) == sizeof(float);
    const int klp = f32 ? a.klp32 : a.klp, kvp = f32 ? a.kvp32 : a.kvp;
    T* Lf = (f32 ? (T*)a.Lf32 : (T*)a.Lf) + u0 * klp;
    T* Uf = (f32 ? (T*)a.Uf32 : (T*)a.Uf) + u0 * kvp;
    int32_t* ip = a.ipiv + u0;
    const int tid = threadIdx.x;

    auto stage_rows = [&](int q0) {
        for (int q = q0 + tid; q < q0 + STAGE_ROWS && q < n; q += blockDim.x) {
            double r[9];
            const int st = assemble_row(v, types, a.dt, q, r);
            if (st) set_error(a.status, st);
#pragma unroll
            for (int s = 0; s < 9; s++) stage[(q & (STAGE_ROWS - 1)) * 9 + s] = r[s];
        }
    };
    // value of original row q at window column slot cs, when the window's
    // first column is c0 (column of slot cs is c0 + ((cs - c0%CW) mod CW))
    auto row_value = [&](int q, int col) -> double {
        const int d = col - q;
        const int dy = (d < -1) ? -1 : (d > 1 ? 1 : 0);
        const int dx = d - dy * nx;
        if (dx < -1 || dx > 1 || col < 0 || col >= n) return 0.0;
        return stage[(q & (STAGE_ROWS - 1)) * 9 + dslot(dx, dy)];
    };

    for (int i = tid; i < RW * CW; i += blockDim.x) W[i] = 0.0;
    stage_rows(0);
    __syncthreads();
    // rows 0..kl into the window (columns 0..kv)
    for (int i = tid; i < RW * CW; i += blockDim.x) {
        const int q = i / CW, c = i - q * CW;
        if (q < n) W[q * CW + c] = row_value(q, c);
    }
    __syncthreads();

    int ju = 0;
    for (int j = 0; j < n; j++) {
        const int km = min(kl, n - 1 - j);
        const int rsj = j % RW, csj = j % CW;
        // [A] pivot: first index of max |column j| over rows j..j+km (idamax)
        if (tid < 32) {
            double best = -1.0;
            int bi = 0;
            for (int i = tid; i <= km; i += 32) {
                const double val = W[((j + i) % RW) * CW + csj];
                colj[i] = val;
                const double av = fabs(val);
                if (av > best) {
                    best = av;
                    bi = i;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) {
                    best = ob;
                    bi = oi;
                }
            }
            if (tid == 0) {
                // idamax: a NaN first element is the maximum (nothing compares
                // greater), elsewhere NaN never is
                if (colj[0] != colj[0]) bi = 0;
                s_jp = bi;
                s_piv = W[((j + bi) % RW) * CW + csj];
                ip[j] = j + bi;
            }
        }
        __syncthreads();
        const int jp = s_jp;
        const double piv = s_piv;
        const bool nz = piv != 0.0;
        if (nz) {
            ju = max(ju, min(j + ku + jp, n - 1));
            // [B] multipliers (from the pre-swap column) and the row swap
            const double rcp = 1.0 / piv;
            for (int i = 1 + tid; i <= km; i += blockDim.x) {
                const double val = (i == jp) ? colj[0] : colj[i];
                const double m = val * rcp;
                mult[i] = m;
                Lf[(size_t)j * klp + (i - 1)] = (T)m;
            }
            if (jp != 0) {
                const int rp = (j + jp) % RW;
                for (int c = j + tid; c <= ju; c += blockDim.x) {
                    const int cs = c % CW;
                    const double t = W[rsj * CW + cs];
                    W[rsj * CW + cs] = W[rp * CW + cs];
                    W[rp * CW + cs] = t;
                }
            }
        } else {
            set_error(a.status, VERB_ERR_PIVOT);
            for (int i = 1 + tid; i <= km; i += blockDim.x) Lf[(size_t)j * klp + (i - 1)] = (T)colj[i];
        }
        __syncthreads();
        // [C] U row j out; rank-1 update of rows j+1..j+km, columns j+1..ju
        for (int c = j + tid; c <= ju && c <= j + kv; c += blockDim.x)
            Uf[(size_t)c * kvp + (kv - (c - j))] = (T)W[rsj * CW + (c % CW)];
        if (nz && km > 0 && ju > j) {
            // warp w updates rows w+1, w+1+nw, ...; lane l columns j+1+l+32k.
            // The pivot row's values (negated, as xGER's temp) stay in
            // registers; window slots advance by wrap, not modulo.
            const int ncol = ju - j;  // <= kv <= 32 * FACT_COLS
            const int lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
            double ty[FACT_COLS];
            int csl[FACT_COLS];
            int cs = (j + 1 + lane) % CW;
#pragma unroll
            for (int k = 0; k < FACT_COLS; k++) {
                csl[k] = cs;
                ty[k] = (lane + 32 * k < ncol) ? -W[rsj * CW + cs] : 0.0;
                cs += 32;
                while (cs >= CW) cs -= CW;
            }
            int r = (j + 1 + wid) % RW;
            for (int i = 1 + wid; i <= km; i += nw) {
                const double m = mult[i];
                double* Wr = W + (size_t)r * CW;
#pragma unroll
                for (int k = 0; k < FACT_COLS; k++)
                    if (ty[k] != 0.0) {
                        double* w = Wr + csl[k];
                        *w = fma(m, ty[k], *w);  // xGER: A(i,k) + x(i)*temp, temp = -y(k), fused
                    }
                r += nw;
                while (r >= RW) r -= RW;
            }
        }
        __syncthreads();
        // [D] slide: row slot j <- original row j+kl+1, column slot j <- column j+kv+1
        const int q = j + kl + 1;
        if (q < n && (q & (STAGE_ROWS - 1)) == 0 && q >= STAGE_ROWS) {
            stage_rows(q);
            __syncthreads();
        }
        for (int cs = tid; cs < CW; cs += blockDim.x) {
            double val = 0.0;
            if (q < n) {
                const int c0 = j + 1;
                const int col = c0 + ((cs - (c0 % CW)) % CW + CW) % CW;
                val = row_value(q, col);
            }
            W[rsj * CW + cs] = val;
        }
        for (int rs = tid; rs < RW; rs += blockDim.x)
            if (rs != rsj) W[rs * CW + csj] = 0.0;
        __syncthreads();
    }
}

// Every row of A, assembled once before the factorisation and parked in the
// L-factor column of the same index: row q's nine diagonal values go to
// Lf[q][0..8] (as FP64, also when the factors are FP32).  local_factor_blk_kernel
// reads row q at least kl columns before it (or for the first window) and writes
// L column q only in the panel of column q, so the parked row is always read before it is overwritten.
template <typename T>
__device__ __forceinline__ double* frw_row_slot(const LocalArgs& a, size_t u)
{
    if constexpr (sizeof(T) == sizeof(float)) return (double*)(a.Lf32 + u * a.klp32);
    else return a.Lf + u * a.klp;
}

template <typename T>
__global__ void local_rows_kernel(LocalArgs a)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const SysView v = sys_view(a, sys);
    int types[4] = {a.Vl_t, a.Vu_t, a.Kl_t, a.Ku_t};
    double r[9];
    const int st = assemble_row(v, types, a.dt, q, r);
    if (st) set_error(a.status, st);
    double* dst = frw_row_slot<T>(a, sys_uoff(a, sys) + q);
#pragma unroll
    for (int s2 = 0; s2 < 9; s2++) dst[s2] = r[s2];
}

__device__ __forceinline__ void cp_async_8(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void frw_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void frw_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Blocked form of the same factorisation.  Columns are taken NB at a time: PW
// warps factor the panel (the NB columns over the kl + NB rows they reach) in
// registers, one row a thread; the other warps meanwhile
// apply the previous panel to the columns right of it, so the pivot chain of
// the next panel and the multiply-adds of this one run at the same time.  The
// (kl + NB) x (kv + NB) window lives in shared memory, circular in rows and
// columns.  The update is a product over the NB pivots on the FP64 matrix
// instruction (m8n8k4): a warp keeps the multipliers of 16 rows in registers
// and runs along the columns, so an element is loaded and stored once per NB
// columns.
//
// Every element sees the operations of local_factor_kernel (LAPACK's xGBTF2
// with the rank-1 update fused) in the same order: the update of element
// (i, c) by pivot k is fma(l_ik, -u_kc, a_ic), pivots in ascending order (the
// matrix instruction adds its four products one fused multiply-add at a time
// in that order: bit-equal to the fma chain), and a row's multipliers move
// with the row when a later pivot of the panel interchanges it.  Factors and
// pivots are therefore bit-identical to it.  xGBTF2 skips the update where
// u_kc = 0 and updates the rows within kl of the pivot only, those of zero
// multipliers included; adding a zero product leaves a finite element as it is,
// so both matter only where a panel holds a zero or tiny pivot or a value above
// 2^1000 or not finite (the slow branches below).
//
// 24 x 51 x 101 x 21 (1224 systems, factors 12.9 GB), the pass with the solve:
// 60.5 ms with the unblocked register-window kernel this replaces, 15.5 ms here;
// 24 x 25 x 31 x 31, the mixed form's pass: 4.76 -> 1.48 ms, 0.9 of it here.  The
// bound is the panel: about 1000 cycles a column of pivot search and exchange
// through shared memory, against 160-320 for the multiply-adds of the update,
// which run beside it; writing the factors at the copy bandwidth takes 2 ms.
constexpr int NB = 8;  // columns of a panel

struct FBlk {
    int RW, CW, pitch;  // window rows, columns, row pitch in doubles
};

__device__ __forceinline__ void named_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// *p = (x, y) in shared memory where c holds, as a predicated store
__device__ __forceinline__ void sts2_if(bool c, double* p, double x, double y)
{
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %0, 0;\n @q st.shared.v2.f64 [%1], {%2, %3};\n}" ::"r"(
            (int)c),
        "r"((unsigned)__cvta_generic_to_shared(p)), "d"(x), "d"(y)
        : "memory");
}

// Blocks an SM is to hold (registers up to 96, 96 and 112; the window's shared memory
// allows them for the bands that PW serves): left to itself the compiler takes 126
// registers for PW = 1 and 2, and 24 x 25 x 31 x 31 comes in two waves, 1.88 against 1.53
// ms for the pass.
constexpr int fb_min_blocks(int PW) { return PW == 1 ? 6 : PW == 2 ? 5 : PW == 3 ? 2 : 1; }

template <typename T, int PW, int NW>
__global__ void __launch_bounds__(NW * 32, fb_min_blocks(PW)) local_factor_blk_kernel(LocalArgs a, FBlk f)
{
    extern __shared__ __align__(16) double sm[];
    const int sys = blockIdx.x;
    if (skip_system(a, sys)) return;
    const int nx = a.d.V;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const int kl = a.kl, ku = a.kl, kv = a.kv;
    const int RW = f.RW, CW = f.CW, pitch = f.pitch;
    double* W = sm;                                // [RW][pitch]
    double* stage = W + (size_t)RW * pitch;        // [2][NB][10] entering rows
    double* newp = stage + 2 * NB * 10;            // [NB][NB] their part in the next panel
    double* prow = newp + NB * NB;                 // [2][PW][NB+4] pivot candidates of the warps
    double* tri = prow + 2 * PW * (NB + 4);                   // [2][NB][NB] multipliers within a panel, negated
    // a panel's interchanges as one permutation of the rows (window offsets):
    // row k <- row s_src[k], and s_no rows below the panel <- rows of it
    __shared__ int s_src[2][NB], s_od[2][NB], s_os[2][NB], s_no[2];
    // for the slow branches: row k's position before the panel, and the last such
    // position that the panel's pivot k updates (-1: it is zero and updates nothing)
    __shared__ int s_init[2][NB], s_lim[2][NB];
    __shared__ int s_ju[2];                        // last column a panel's pivot rows reach
    __shared__ int s_bad[2];                       // a non-finite multiplier in the panel
    __shared__ int s_badu;                         // a non-finite U entry
    __shared__ int s_huge;                         // a value above 2^1000 in the panel
    const bool f32 = sizeof(T) == sizeof(float);
    const int klp = f32 ? a.klp32 : a.klp, kvp = f32 ? a.kvp32 : a.kvp;
    T* Lf = (f32 ? (T*)a.Lf32 : (T*)a.Lf) + u0 * klp;
    T* Uf = (f32 ? (T*)a.Uf32 : (T*)a.Uf) + u0 * kvp;
    int32_t* ip = a.ipiv + u0;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const double* rows = frw_row_slot<T>(a, u0);
    const size_t rstride = f32 ? (size_t)a.klp32 / 2 : (size_t)a.klp;  // doubles

    // column offset of the nine stored diagonals
    auto diag_off = [&](int s) { return (s / 3 - 1) * nx + (s % 3 - 1); };
    // the rows that enter when the panel at j0 is done
    auto fetch_rows = [&](int j0, int buf, int t, int nt) {
        for (int e = t; e < NB * 9; e += nt) {
            const int r = e / 9, s = e - r * 9, q = j0 + RW + r;
            if (q < n) cp_async_8(stage + (buf * NB + r) * 10 + s, rows + q * rstride + s);
        }
        frw_commit();
    };

    // first window: rows 0 .. RW-1; the U entries above row 0 are zero
    for (int e = tid; e < RW * pitch; e += NW * 32) W[e] = 0.0;
    for (int c = wid; c < min(kv, n); c += NW)
        for (int q = lane; q < kv - c; q += 32) Uf[(size_t)c * kvp + q] = (T)0;
    if (tid == 0) s_badu = 0;
    __syncthreads();
    for (int e = tid; e < min(RW, n) * 9; e += NW * 32) {
        const int q = e / 9, s = e - q * 9, c = q + diag_off(s);
        if (c >= 0 && c < n) W[q * pitch + c] = rows[q * rstride + s];
    }
    __syncthreads();

    // One panel: columns j0 .. j0+NB-1 over rows j0 .. j0+RW-1, row tid of
    // them by each thread of the first PW warps; rj, cj: window slots of row
    // and column j0.  first: every row is in the window, else the last NB ones
    // are in newp.  Returns the new ju.  What a column costs is the chain from
    // its updated values through the pivot search to the next update, and the
    // instructions the warps fetch on the way: the loop stays rolled (column
    // jj is always R[0]; the update writes column c to R[c-1], the finished
    // column goes to the end), rows are not interchanged in the registers,
    // only their positions pos are, and there is one barrier a column.
    auto panel = [&](int j0, int rj, int cj, int par, bool first, int ju) {
        constexpr int PT = PW * 32;
        double R[NB];
        const int t = tid, nbk = min(NB, n - j0);
        int pos = t;
        auto slot = [&](int c) { return cj + c < CW ? cj + c : cj + c - CW; };
        auto off = [&](int i) { return (rj + i < RW ? rj + i : rj + i - RW) * pitch; };
        unsigned top = 0;
        {
            const bool win = first || t < kl;
            const double* src = win ? W + off(t) : newp + (t - kl) * NB;
#pragma unroll
            for (int c = 0; c < NB; c += 2) {
                double2 v = make_double2(0.0, 0.0);
                if (t < RW) v = *(const double2*)(src + (win ? slot(c) : c));
                R[c] = v.x;
                R[c + 1] = v.y;
                top = max(top, max((unsigned)__double2hiint(v.x) & 0x7fffffffu,
                                   (unsigned)__double2hiint(v.y) & 0x7fffffffu));
            }
        }
        // values up to 2^1000 stay finite over a panel (|l| <= 1); larger ones
        // and pivots whose reciprocal overflows take the slow branch
        if (tid == 0) {
            s_no[par] = 0;
            s_huge = 0;
        }
        if (tid < NB) s_lim[par][tid] = min(tid + kl, n - 1 - j0);
        named_sync(2, PT);
        if (top >= 0x7e700000u) s_huge = 1;
        int jj = 0;
        T* pl = Lf + (size_t)j0 * klp - 1;
#pragma unroll 1
        for (; jj < nbk; jj++) {
            // the warp's first maximum of |column jj| over positions jj ..
            // jj+kl, by the upper words, the lower ones only where those tie
            const int last = min(jj + kl, n - 1 - j0);
            const unsigned h =
                pos >= jj && pos <= last ? (unsigned)__double2hiint(R[0]) & 0x7fffffffu : 0u;
            const unsigned wh = __reduce_max_sync(0xffffffffu, h);
            const double rinv = recip(R[0]);
            bool own = h == wh;
            const unsigned b = __ballot_sync(0xffffffffu, own);
            if (b & (b - 1)) {
                const unsigned lo = own && wh ? (unsigned)__double2loint(R[0]) : 0u;
                const unsigned wl = __reduce_max_sync(0xffffffffu, lo);
                own = own && lo == wl;
                const unsigned p = own ? pos : 1u << 20;
                own = p == __reduce_min_sync(0xffffffffu, p);
            }
            // its row, reciprocal, |pivot| and position
            double* cand = prow + ((jj & 1) * PW + wid) * (NB + 4);
#pragma unroll
            for (int c = 0; c < NB; c += 2) sts2_if(own, cand + c, R[c], R[c + 1]);
            sts2_if(own, cand + NB, wh ? fabs(R[0]) : 0.0, __hiloint2double(0, wh ? pos : 1 << 20));
            sts2_if(own, cand + NB + 2, rinv, 0.0);
            named_sync(2, PT);
            const double* best = prow + (jj & 1) * PW * (NB + 4);
            double2 key = *(const double2*)(best + NB);
#pragma unroll
            for (int w = 1; w < PW; w++) {
                const double* o = prow + ((jj & 1) * PW + w) * (NB + 4);
                const double2 k = *(const double2*)(o + NB);
                const long long ka = __double_as_longlong(k.x), kb = __double_as_longlong(key.x);
                if (ka > kb || (ka == kb && __double2loint(k.y) < __double2loint(key.y))) {
                    key = k;
                    best = o;
                }
            }
            if (s_huge || __double2hiint(key.x) < 0x00400000) break;
            const int tp = __double2loint(key.y);
            double uc[NB];
#pragma unroll
            for (int c = 0; c < NB; c += 2) {
                const double2 v = *(const double2*)(best + c);
                // finished columns sit at the end: no update
                uc[c] = c < NB - jj ? -v.x : 0.0;
                uc[c + 1] = c + 1 < NB - jj ? -v.y : 0.0;
            }
            const double rcp = best[NB + 2];
            if (tid == 0) ip[j0 + jj] = j0 + tp;
            ju = max(ju, min(j0 + ku + tp, n - 1));
            pos = pos == tp ? jj : (pos == jj ? tp : pos);
            const double m = R[0] * rcp;
            const bool act = pos > jj && pos <= last;
            if (act) pl[pos] = (T)m;
            const double l = act ? m : 0.0, fin = act ? m : R[0];
#pragma unroll
            for (int c = 1; c < NB; c++) R[c - 1] = fma(l, uc[c], R[c]);
            R[NB - 1] = fin;
            pl += klp - 1;
        }
        // the panel back into the window, every row at its position
        const bool bad = jj < nbk;
        if (jj == NB) {
            double* row = W + off(pos);
            if (t < RW)
#pragma unroll
                for (int c = 0; c < NB; c += 2)
                    *(double2*)(row + slot(c)) = make_double2(R[c], R[c + 1]);
        } else {
            // R[c] is column jj + c, the finished ones follow from the start
#pragma unroll 1
            for (int c = 0; c < NB; c++) {
                if (t < RW) W[off(pos) + slot((jj + c) % NB)] = R[0];
#pragma unroll
                for (int k = 1; k < NB; k++) R[k - 1] = R[k];
            }
        }
        named_sync(2, PT);
        if (bad) {
            // the rest of the panel in the window, operation by operation as
            // xGBTF2 does it
            auto at = [&](int i, int c) -> double& { return W[off(i) + slot(c)]; };
#pragma unroll 1
            for (; jj < nbk; jj++) {
                const int j = j0 + jj, km = min(kl, n - 1 - j);
                int p = jj;
                double best = fabs(at(jj, jj));
#pragma unroll 1
                for (int i = jj + 1; i <= jj + km; i++) {
                    const double v = fabs(at(i, jj));
                    if (v > best) {
                        best = v;
                        p = i;
                    }
                }
                const double piv = at(p, jj);
                const bool nz = piv != 0.0;
                if (nz) ju = max(ju, min(j0 + ku + p, n - 1));
                named_sync(2, PT);
                if (nz && p != jj) {
                    if (tid < NB) {
                        const double v = at(jj, tid);
                        at(jj, tid) = at(p, tid);
                        at(p, tid) = v;
                    }
                    pos = pos == jj ? p : (pos == p ? jj : pos);
                }
                if (tid == 0) {
                    ip[j] = j0 + p;
                    if (!nz) {
                        s_lim[par][jj] = -1;
                        set_error(a.status, VERB_ERR_PIVOT);
                    }
                }
                named_sync(2, PT);
                const double rcp = 1.0 / piv;
#pragma unroll 1
                for (int i = jj + 1 + tid; i <= jj + km; i += PT) {
                    const double m = nz ? at(i, jj) * rcp : at(i, jj);
                    Lf[(size_t)j * klp + (i - jj - 1)] = (T)m;
                    at(i, jj) = nz ? m : 0.0;
#pragma unroll 1
                    for (int c = jj + 1; nz && c < NB; c++) {
                        const double u = at(jj, c);
                        if (u != 0.0) at(i, c) = fma(m, -u, at(i, c));
                    }
                }
                named_sync(2, PT);
            }
        }
        // the multipliers among the panel's rows, column by column from the
        // diagonal down (negated, zero past row NB-1), for the triangular solves
#pragma unroll
        for (int e = tid; e < NB * NB; e += PT) {
            const int m = e / NB, i = e % NB;
            tri[(par * NB + m) * NB + i] = i && m + i < NB ? -W[off(m + i) + slot(m)] : 0.0;
        }
        // the interchanges as one permutation
        if (pos < NB) {
            s_src[par][pos] = off(t);
            s_init[par][pos] = t;
        }
        if (pos >= NB && pos != t) {
            const int i = atomicAdd(&s_no[par], 1);
            s_od[par][i] = off(pos);
            s_os[par][i] = off(t);
        }
        if (tid == 0) {
            s_ju[par] = ju;
            s_bad[par] = bad;
        }
        return ju;
    };

    int ju0 = 0;  // the panel warps' running ju
    // block j0: the panel at j0 is factored; j0 = -NB only factors the first
    int rj = RW - NB, cj = CW - NB, par = 1;
    for (int j0 = -NB;; j0 += NB, par ^= 1) {
        const int jn = j0 + NB;  // next panel
        const bool head = j0 < 0;
        const int ju = head ? -1 : s_ju[par];
        auto rslot = [&](int t) {
            const int s = rj + t;
            return (s >= RW ? s - RW : s) * pitch;
        };
        auto cslot = [&](int c) {  // column j0 + c
            const int s = cj + c;
            return s >= CW ? s - CW : s;
        };
        if (!head && wid == NW - 1) {
            // U of the panel's own columns (and the padding below the diagonal)
            const int k = lane % NB;
#pragma unroll
            for (int i = 0; i < NB * NB / 32; i++) {
                const int c = lane / NB + i * (32 / NB);
                T* dst = Uf + (size_t)(j0 + c) * kvp + kv;
                if (k <= c && j0 + c < n) dst[k - c] = (T)W[rslot(k) + cslot(c)];
                if (k == c && j0 + c < n)
                    for (int z = 1; z < kvp - kv; z++) dst[z] = (T)0;
            }
        }
        if (jn >= n) break;
        // Interchanges and the triangular solve of columns c < c_hi (relative to
        // j0), one thread a column: U rows j0 .. jn-1 to the window.
        auto solve_columns = [&](int c, int step, int c_hi, bool slow) {
            const int no = s_no[par];
            const double* tr = tri + par * NB * NB;
#pragma unroll 1
            for (; c < c_hi; c += step) {
                double* col = W + cslot(c);
                double x[NB];
                unsigned top = 0;
#pragma unroll
                for (int k = 0; k < NB; k++) {
                    x[k] = col[s_src[par][k]];
                    top = max(top, (unsigned)__double2hiint(x[k]) & 0x7fffffffu);
                }
#pragma unroll 1
                for (int i = 0; i < no; i += 4) {
                    double y[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) y[e] = i + e < no ? col[s_os[par][i + e]] : 0.0;
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (i + e < no) col[s_od[par][i + e]] = y[e];
                }
                int r = rj;
                if (__builtin_expect(slow || top >= 0x7e700000u, 0)) {
                    // operation by operation as xGBTF2 does it: a pivot of the
                    // panel updates the rows it reaches, unless its u is zero
#pragma unroll
                    for (int k = 0; k < NB; k++) col[rslot(k)] = x[k];
#pragma unroll 1
                    for (int m = 0; m < NB; m++) {
                        const double u = col[rslot(m)];
                        if (((unsigned)__double2hiint(u) & 0x7fffffffu) >= 0x7ff00000u) s_badu = 1;
                        if (u == 0.0) continue;
#pragma unroll 1
                        for (int k = m + 1; k < NB; k++)
                            if (s_init[par][k] <= s_lim[par][m])
                                col[rslot(k)] = fma(tr[m * NB + k - m], u, col[rslot(k)]);
                    }
                    continue;
                }
                // row m is always x[0]: the loop stays rolled; the next
                // multipliers are loaded while these are used.  Values up to 2^1000
                // stay finite (|l| <= 1)
                double2 l[NB / 2];
#pragma unroll
                for (int k = 0; k < NB / 2; k++) l[k] = *(const double2*)(tr + 2 * k);
#pragma unroll 1
                for (int m = 0; m < NB; m++) {
                    const double u = x[0];
                    col[r * pitch] = u;
                    r = r + 1 == RW ? 0 : r + 1;
                    const double* tn = tr + min(m + 1, NB - 1) * NB;
#pragma unroll
                    for (int k = 0; k < NB / 2; k++) {
                        const double2 lk = l[k];
                        l[k] = *(const double2*)(tn + 2 * k);
                        if (k) x[2 * k - 1] = fma(lk.x, u, x[2 * k]);
                        x[2 * k] = fma(lk.y, u, x[2 * k + 1]);
                    }
                }
            }
        };
        // The update of columns c_lo .. c_hi-1 (relative to j0): warp w of nw
        // takes 16 rows at a time, whose multipliers (negated) stay in
        // registers, along all the columns, two 8-column tiles at a time.  With
        // the row pitch at 2 or 14 mod 16 doubles, the tiles' row order (bits
        // 0 and 1 of the index swapped) and columns (two pairs of a tile
        // eight apart) keep the accesses to C and U free of bank conflicts.
        auto update = [&](int c_lo, int c_hi, int w, int nw) {
            const int g = lane >> 2, h = lane & 3;
            const int gr = (g & 4) | (g & 1) << 1 | (g >> 1 & 1);
            const int hc = 2 * (h >> 1) + 8 * (h & 1);           // of C
            const int gc = 2 * (g >> 2) + 8 * (g >> 1 & 1) + (g & 1);  // of U
            int rb[NB / 4];
#pragma unroll
            for (int k = 0; k < NB / 4; k++) rb[k] = rslot(4 * k + h);
            for (int t0 = NB + 16 * w; t0 < RW; t0 += 16 * nw) {
                int ro[2];
                double l[2][NB / 4];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    ro[i] = rslot(min(t0 + 8 * i + gr, RW - 1));
#pragma unroll
                    for (int k = 0; k < NB / 4; k++) l[i][k] = -W[ro[i] + cslot(4 * k + h)];
                }
                for (int c = c_lo; c < c_hi; c += 16) {
                    double2 acc[2][2];
                    int co[2];
                    double u[2][NB / 4];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        co[e] = cslot(min(c + 4 * e + hc, CW - 2));
                        const int cb = cslot(min(c + 4 * e + gc, CW - 1));
#pragma unroll
                        for (int i = 0; i < 2; i++) acc[i][e] = *(const double2*)(W + ro[i] + co[e]);
#pragma unroll
                        for (int k = 0; k < NB / 4; k++) u[e][k] = W[rb[k] + cb];
                    }
#pragma unroll
                    for (int k = 0; k < NB / 4; k++)
#pragma unroll
                        for (int e = 0; e < 2; e++)
#pragma unroll
                            for (int i = 0; i < 2; i++) dmma(acc[i][e].x, acc[i][e].y, l[i][k], u[e][k]);
#pragma unroll
                    for (int e = 0; e < 2; e++)
#pragma unroll
                        for (int i = 0; i < 2; i++)
                            if (t0 + 8 * i + gr < RW && c + 4 * e + hc < c_hi)
                                *(double2*)(W + ro[i] + co[e]) = acc[i][e];
                }
            }
        };
        // the same update element by element as xGBTF2 does it: a pivot updates the
        // rows it reaches, those of zero multipliers included, unless its u is zero
        auto update_slow = [&](int c_lo, int c_hi, int t, int nt) {
#pragma unroll 1
            for (int e = t; e < (c_hi - c_lo) * kl; e += nt) {
                const int c = c_lo + e / kl, ro = rslot(NB + e % kl);
                int init = NB + e % kl;  // the row's position before the panel
#pragma unroll 1
                for (int i = 0; i < s_no[par]; i++)
                    if (s_od[par][i] == ro) {
                        const int q = s_os[par][i] / pitch - rj;
                        init = q < 0 ? q + RW : q;
                    }
                double v = W[ro + cslot(c)];
#pragma unroll 1
                for (int k = 0; k < NB; k++) {
                    const double u = W[rslot(k) + cslot(c)], l = W[ro + cslot(k)];
                    if (u != 0.0 && init <= s_lim[par][k]) v = fma(l, -u, v);
                }
                W[ro + cslot(c)] = v;
            }
        };

        // ---- the next panel's columns first
        const bool slow_l = !head && s_bad[par] != 0;
        const int cols_n = min(NB, n - jn);
        if (!head) {
        frw_wait_all();  // the entering rows
        if (wid == 0) solve_columns(NB + lane, 32, NB + cols_n, slow_l);
        __syncthreads();
        // U rows j0 .. jn-1 of the next panel's columns out
        for (int e = tid; e < NB * cols_n; e += NW * 32) {
            const int k = e % NB, c = NB + e / NB;
            if (c - k <= kv) Uf[(size_t)(j0 + c) * kvp + kv - (c - k)] = (T)W[rslot(k) + cslot(c)];
        }
        if (wid == NW - 1) {
            // the entering rows' part in the next panel
            for (int e = lane; e < NB * NB; e += 32) newp[e] = 0.0;
            __syncwarp();
            for (int e = lane; e < NB * 9; e += 32) {
                const int r = e / 9, s = e - r * 9, q = j0 + RW + r;
                const int c = q + diag_off(s) - jn;
                if (q < n && c >= 0 && c < NB && jn + c < n)
                    newp[r * NB + c] = stage[(par * NB + r) * 10 + s];
            }
        }
        if (!(slow_l || s_badu)) {
            update(NB, 2 * NB, wid, NW);
        } else {
            update_slow(NB, NB + cols_n, tid, NW * 32);
        }
        __syncthreads();
        }

        int rjn = rj + NB, cjn = cj + NB;
        if (rjn >= RW) rjn -= RW;
        if (cjn >= CW) cjn -= CW;
        if (wid < PW) {
            ju0 = panel(jn, rjn, cjn, par ^ 1, head, ju0);
        } else {
            // ---- the columns right of the next panel
            const int ot = tid - PW * 32;
            constexpr int ON = (NW - PW) * 32;
            const int c_hi = ju - j0 + 1;   // columns c < c_hi take the update
            solve_columns(2 * NB + ot, ON, c_hi, slow_l);
            fetch_rows(jn, par ^ 1, ot, ON);
            if (!head) {
            named_sync(1, ON);
            if (!(slow_l || s_badu)) {
                update(2 * NB, min((c_hi + 1) & ~1, CW), wid - PW, NW - PW);
            } else {
                update_slow(2 * NB, c_hi, ot, ON);
            }
            // U rows j0 .. jn-1 out (lanes along the rows: contiguous in Uf)
            {
                const int k = ot % NB, c_end = min(min(NB + kv, n - j0), kv + k + 1);
                const int rk = rslot(k);
                T* dst = Uf + (size_t)j0 * kvp + kv + k;
                constexpr int CS = ON / NB;
                for (int c = 2 * NB + ot / NB; c < c_end; c += 4 * CS) {
                    double v[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] = W[rk + cslot(min(c + i * CS, CW - 1))];
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (c + i * CS < c_end) dst[(size_t)(c + i * CS) * (kvp - 1)] = (T)v[i];
                }
            }
            named_sync(1, ON);
            // the slide: the panel's columns become columns j0 + CW .., its
            // rows become the entering rows
            const double2 z2 = make_double2(0.0, 0.0);
#pragma unroll 4
            for (int e = ot; e < (RW - NB) * (NB / 2); e += ON) {
                const int r = e / (NB / 2), c = (e - r * (NB / 2)) * 2;
                *(double2*)(W + rslot(NB + r) + cslot(c)) = z2;
            }
#pragma unroll 1
            for (int c = 2 * ot; c < CW; c += 2 * ON)
                if (c < NB || c >= 2 * NB) {
                    double* col = W + cslot(c);
#pragma unroll
                    for (int r = 0; r < NB; r++) *(double2*)(col + rslot(r)) = z2;
                }
            named_sync(1, ON);
            for (int e = ot; e < NB * 9; e += ON) {
                const int r = e / 9, s = e - r * 9, q = j0 + RW + r;
                const int c = q + diag_off(s) - j0;
                if (q < n && c >= 2 * NB && j0 + c < n) {
                    int cs = cj + c;
                    while (cs >= CW) cs -= CW;
                    W[rslot(r) + cs] = stage[(par * NB + r) * 10 + s];
                }
            }
            }
        }
        __syncthreads();
        rj = rjn;
        cj = cjn;
    }
}

// RHS = B o f + C in unknown order (src/MatrixSolver.cpp:309-320), through a
// 32x32 shared-memory tile transpose of the [V][K] slab.
__global__ void local_rhs_kernel(LocalArgs a, int from_work)
{
    __shared__ double tile[32][33];
    const int sys = blockIdx.z;
    if (skip_system(a, sys)) return;
    const int V = a.d.V, K = a.d.K;
    const int kz = sys_k0(a, sys), ny = K - kz;  // unknowns: pitch-angle indices kz..K-1
    const double* psd = a.psd + (size_t)sys * V * K;
    double* w = a.work + sys_uoff(a, sys);
    const int v0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    if (!from_work) {
        for (int r = ty; r < 32; r += 8) {
            const int iv = v0 + r, ik = k0 + tx;
            if (iv < V && ik < K) tile[r][tx] = psd[(size_t)iv * K + ik];
        }
    } else {
        for (int r = ty; r < 32; r += 8) {
            const int ik = k0 + r, iv = v0 + tx;
            if (iv < V && ik >= kz && ik < K) tile[tx][r] = w[(size_t)(ik - kz) * V + iv];
        }
    }
    __syncthreads();
    const SysView sv = sys_view(a, sys);
    const double bint = 0.0 + 1.0 / a.dt;
    const double ls = (double)a.local_sources;
    for (int r = ty; r < 32; r += 8) {
        const int ik = k0 + r, iv = v0 + tx;
        if (iv >= V || ik >= K || ik < kz) continue;
        const int ix = iv, iy = ik - kz;
        double b, c;
        if (ix == 0 && V >= 3) {
            b = 0.0;
            c = sv.xl[iy];
        } else if (ix == V - 1 && V >= 3) {
            b = 0.0;
            c = sv.xu[iy];
        } else if (iy == 0 && ny >= 3) {
            b = 0.0;
            c = sv.trimmed ? 0.0 : sv.yl[ix];
        } else if (iy == ny - 1 && ny >= 3) {
            b = 0.0;
            c = sv.yu[ix];
        } else {
            b = bint;
            c = 0.0;
            c += sv.S[(size_t)ix * K + iy] * ls;
        }
        double rhs = tile[tx][r];
        rhs *= b;
        rhs += c;
        w[(size_t)iy * V + iv] = rhs;
    }
}

__global__ void local_store_kernel(LocalArgs a)
{
    __shared__ double tile[32][33];
    const int sys = blockIdx.z;
    if (skip_system(a, sys)) return;
    const int V = a.d.V, K = a.d.K;
    const int kz = sys_k0(a, sys);
    double* psd = a.psd + (size_t)sys * V * K;
    const double* w = a.work + sys_uoff(a, sys);
    const int v0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < 32; r += 8) {
        const int ik = k0 + r, iv = v0 + tx;
        if (iv < V && ik >= kz && ik < K) tile[tx][r] = w[(size_t)(ik - kz) * V + iv];
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int iv = v0 + r, ik = k0 + tx;
        if (iv < V && ik >= kz && ik < K) psd[(size_t)iv * K + ik] = tile[r][tx];
    }
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
// cnt 16-byte chunks, cnt <= 32 * MAXT, by the 32 lanes of a warp: a fixed
// number of predicated copies instead of a loop with a run-time trip count
template <int MAXT>
__device__ __forceinline__ void warp_copy16(void* dst, const void* src, int cnt, int lane)
{
#pragma unroll
    for (int t = 0; t < MAXT; t++) {
        const int c = lane + 32 * t;
        if (c < cnt) cp_async16((char*)dst + 16 * c, (const char*)src + 16 * c);
    }
}
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Solve variants: warps (systems) per CTA, L and U factor columns in flight
// per warp.  More columns in flight hide more latency per warp but take
// shared memory that would otherwise hold more resident warps; the best
// trade depends on the grid, so the autotuner picks one per context.
// The second group keeps the right-hand-side window in registers instead of
// shared memory (local_solve_rw_kernel).
// The last group caps the registers (at least minb CTAs per SM: 36 resident
// systems per SM) so that a 48 x 101 grid's 4848 systems are resident in one
// wave instead of 32 per SM and a tail of 112.
struct SolveShape {
    int warps, fwd, bwd, rw;
    int minb = 1;
};
constexpr SolveShape SOLVE_SHAPES[] = {
    {4, 4, 2, 0},  {4, 6, 3, 0},  {2, 6, 4, 0},  {2, 8, 6, 0},  {1, 8, 6, 0},  {1, 12, 8, 0},
    {1, 12, 10, 0}, {1, 16, 12, 0}, {1, 24, 16, 0},
    {4, 4, 3, 1},  {4, 6, 4, 1},  {2, 8, 6, 1},  {2, 12, 8, 1}, {1, 12, 8, 1}, {1, 16, 12, 1},
    {4, 4, 2, 1, 9}, {2, 6, 3, 1, 18}, {4, 6, 3, 1, 9}};
constexpr int N_SOLVE_SHAPES = sizeof(SOLVE_SHAPES) / sizeof(SOLVE_SHAPES[0]);
constexpr int FWD_WIN = 128;   // >= kl + 1
constexpr int BWD_WIN = 256;   // >= kv + 1

// ring of factor columns per warp, in doubles (16-byte multiples)
__host__ __device__ constexpr size_t solve_ring_doubles(int klp, int kvp, int esize, int fd, int bd)
{
    return ((size_t)(fd * klp > bd * kvp ? fd * klp : bd * kvp) * esize + 15) / 16 * 2;
}

// T: storage type of the factors.  The substitutions run in FP64 either way
// (float factors are widened as they are used).
template <typename T, int SOLVE_WARPS, int FWD_DEPTH, int BWD_DEPTH>
__global__ void __launch_bounds__(SOLVE_WARPS * 32) local_solve_kernel(LocalArgs a, int nsys)
{
    extern __shared__ double sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sys = blockIdx.x * SOLVE_WARPS + warp;
    if (sys >= nsys || skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const bool f32 = sizeof(T) == sizeof(float);
    const int kl = a.kl, kv = a.kv, klp = f32 ? a.klp32 : a.klp, kvp = f32 ? a.kvp32 : a.kvp;
    constexpr int VEC = 16 / sizeof(T);  // elements per 16-byte cp.async
    const size_t per_warp = BWD_WIN + solve_ring_doubles(klp, kvp, sizeof(T), FWD_DEPTH, BWD_DEPTH);
    double* win = sm + (size_t)warp * per_warp;
    T* ring = (T*)(win + BWD_WIN);
    double* w = a.work + u0;
    const T* Lf = (f32 ? (const T*)a.Lf32 : (const T*)a.Lf) + u0 * klp;
    const T* Uf = (f32 ? (const T*)a.Uf32 : (const T*)a.Uf) + u0 * kvp;
    const int32_t* ip = a.ipiv + u0;

    // ---------------- forward: L with interleaved row interchanges (xGBTRS) --------
    for (int i = lane; i < FWD_WIN && i < n; i += 32) win[i] = w[i];
    auto issue_L = [&](int col) {
        if (col < n - 1) {
            T* dst = ring + (col % FWD_DEPTH) * klp;
            const T* src = Lf + (size_t)col * klp;
            warp_copy16<FWD_WIN * 8 / 16 / 32>(dst, src, klp / VEC, lane);
        }
    };
    for (int c = 0; c < FWD_DEPTH; c++) {
        issue_L(c);
        cp_commit();
    }
    int pv_cur = (lane < n) ? ip[lane] : 0;
    int pv_next = (32 + lane < n) ? ip[32 + lane] : 0;
    __syncwarp();
    for (int j = 0; j < n - 1; j++) {
        if ((j & 31) == 0 && j > 0) {
            pv_cur = pv_next;
            const int nx = j + 32 + lane;
            pv_next = (nx < n) ? ip[nx] : 0;
        }
        cp_wait<FWD_DEPTH - 1>();
        __syncwarp();
        const int lm = min(kl, n - 1 - j);
        const int l = __shfl_sync(0xffffffffu, pv_cur, j & 31);
        const double bj_old = win[j & (FWD_WIN - 1)];
        const double bl = win[l & (FWD_WIN - 1)];
        const double bj = (l != j) ? bl : bj_old;
        const T* Lc = ring + (j % FWD_DEPTH) * klp;
        const double tmp = -bj;
        const bool upd = bj != 0.0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int t = lane + 32 * k;
            const int i = j + 1 + t;
            if (t < lm) {
                double cur = (i == l) ? bj_old : win[i & (FWD_WIN - 1)];
                if (upd) cur = cur + (double)Lc[t] * tmp;  // xGER in xGBTRS
                win[i & (FWD_WIN - 1)] = cur;
            }
        }
        __syncwarp();
        if (lane == 0) {
            w[j] = bj;
            if (j + FWD_WIN < n) cp_async8(&win[j & (FWD_WIN - 1)], &w[j + FWD_WIN]);
        }
        issue_L(j + FWD_DEPTH);
        cp_commit();
    }
    cp_wait<0>();
    __syncwarp();
    if (lane == 0) w[n - 1] = win[(n - 1) & (FWD_WIN - 1)];
    __syncwarp();

    // ---------------- backward: U, column oriented (xTBSV 'U','N','N') ------------
    for (int i = n - 1 - lane; i >= 0 && i > n - 1 - BWD_WIN; i -= 32) win[i & (BWD_WIN - 1)] = w[i];
    auto issue_U = [&](int col) {
        if (col >= 0) {
            T* dst = ring + ((n - 1 - col) % BWD_DEPTH) * kvp;
            const T* src = Uf + (size_t)col * kvp;
            warp_copy16<BWD_WIN * 8 / 16 / 32>(dst, src, kvp / VEC, lane);
        }
    };
    for (int c = 0; c < BWD_DEPTH; c++) {
        issue_U(n - 1 - c);
        cp_commit();
    }
    __syncwarp();
    for (int j = n - 1; j >= 0; j--) {
        cp_wait<BWD_DEPTH - 1>();
        __syncwarp();
        const T* Uc = ring + ((n - 1 - j) % BWD_DEPTH) * kvp;
        double bj = win[j & (BWD_WIN - 1)];
        if (bj != 0.0) {
            bj = bj / (double)Uc[kv];
#pragma unroll
            for (int k = 0; k < 7; k++) {
                const int d = 1 + lane + 32 * k;
                const int i = j - d;
                if (d <= kv && i >= 0) {
                    double* x = &win[i & (BWD_WIN - 1)];
                    *x = *x - bj * (double)Uc[kv - d];  // xTBSV: X(I) - TEMP*A(L+I,J)
                }
            }
        }
        __syncwarp();
        if (lane == 0) {
            w[j] = bj;
            if (j - BWD_WIN >= 0) cp_async8(&win[j & (BWD_WIN - 1)], &w[j - BWD_WIN]);
        }
        issue_U(j - BWD_DEPTH);
        cp_commit();
    }
    cp_wait<0>();
}

// The same solve with the right-hand-side window in registers.  Forward
// (xGBTRS with interleaved row interchanges), at column j the window holds
// positions j .. j+32FS-1: lane i's slot m holds position
// j + ((i - j) & 31) + 32m, so the updates of column j (positions
// j+1 .. j+lm) touch every lane's slots in place, the pivot row l is read from
// lane l & 31, slot (l - j) >> 5, and only lane j & 31 shifts its slots down
// (position j leaves, position j + 32FS enters) when the column is done.
// Backward (xTBSV), at column j the window holds j .. j-32BS+1 the same way
// downwards.  The factor columns still stream through a per-warp cp.async
// ring in shared memory (read with rotated, conflict-free accesses), and the
// right-hand-side entries that enter the window are staged with them.  The
// operations and their order are those of local_solve_kernel, so the result is
// bit-identical; what changes is that the window no longer costs shared-memory
// loads and stores per column, which the old kernel's column chain waited on.
template <typename T, int SOLVE_WARPS, int FWD_DEPTH, int BWD_DEPTH, int FS, int BS, int MINB>
__global__ void __launch_bounds__(SOLVE_WARPS * 32, MINB) local_solve_rw_kernel(LocalArgs a, int nsys)
{
    extern __shared__ double sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sys = blockIdx.x * SOLVE_WARPS + warp;
    if (sys >= nsys || skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const bool f32 = sizeof(T) == sizeof(float);
    const int kl = a.kl, kv = a.kv, klp = f32 ? a.klp32 : a.klp, kvp = f32 ? a.kvp32 : a.kvp;
    constexpr int VEC = 16 / sizeof(T);
    constexpr int FWIN = 32 * FS, BWIN = 32 * BS;
    constexpr int STAGE = (FWD_DEPTH > BWD_DEPTH ? FWD_DEPTH : BWD_DEPTH) + 1 & ~1;
    const size_t per_warp = STAGE + solve_ring_doubles(klp, kvp, sizeof(T), FWD_DEPTH, BWD_DEPTH);
    double* stage = sm + (size_t)warp * per_warp;  // entering right-hand-side entries
    T* ring = (T*)(stage + STAGE);
    double* w = a.work + u0;
    const T* Lf = (f32 ? (const T*)a.Lf32 : (const T*)a.Lf) + u0 * klp;
    const T* Uf = (f32 ? (const T*)a.Uf32 : (const T*)a.Uf) + u0 * kvp;
    const int32_t* ip = a.ipiv + u0;

    // ---------------- forward: L with interleaved row interchanges (xGBTRS) --------
    double s[FS > BS ? FS : BS];
#pragma unroll
    for (int m = 0; m < FS; m++) {
        const int p = lane + 32 * m;
        s[m] = p < n ? w[p] : 0.0;
    }
    // column col's multipliers, and b[col + FWIN] (which enters the window
    // when column col is done)
    // (slot: col mod FWD_DEPTH, kept as a running index by the caller)
    auto issue_L = [&](int col, int slot) {
        if (col < n - 1) {
            T* dst = ring + slot * klp;
            const T* src = Lf + (size_t)col * klp;
            warp_copy16<FWD_WIN * 8 / 16 / 32>(dst, src, klp / VEC, lane);
            if (lane == 0) {
                double* st = &stage[slot];
                if (col + FWIN < n) cp_async8(st, &w[col + FWIN]);
                else *st = 0.0;
            }
        }
    };
    for (int c = 0; c < FWD_DEPTH; c++) {
        issue_L(c, c);
        cp_commit();
    }
    int fslot = 0;  // j mod FWD_DEPTH
    int pv_cur = (lane < n) ? ip[lane] : 0;
    int pv_next = (32 + lane < n) ? ip[32 + lane] : 0;
    for (int j = 0; j < n - 1; j++) {
        if ((j & 31) == 0 && j > 0) {
            pv_cur = pv_next;
            const int nx = j + 32 + lane;
            pv_next = (nx < n) ? ip[nx] : 0;
        }
        cp_wait<FWD_DEPTH - 1>();
        __syncwarp();
        const int lm = min(kl, n - 1 - j);
        const int l = __shfl_sync(0xffffffffu, pv_cur, j & 31);
        const double bj_old = __shfl_sync(0xffffffffu, s[0], j & 31);
        double bj = bj_old;
        if (l != j) {  // the same for the whole warp: an interchange
            const int sl = (l - j) >> 5;  // slot of position l in lane l & 31
            double v = s[0];
#pragma unroll
            for (int m = 1; m < FS; m++) v = (sl == m) ? s[m] : v;
            bj = __shfl_sync(0xffffffffu, v, l & 31);
            if (lane == (l & 31)) {
#pragma unroll
                for (int m = 0; m < FS; m++)
                    if (sl == m) s[m] = bj_old;
            }
        }
        if (bj != 0.0) {
            const T* Lc = ring + fslot * klp;
            const double tmp = -bj;
            const int o = (lane - j) & 31;
#pragma unroll
            for (int m = 0; m < FS; m++) {
                const int e = o + 32 * m - 1;  // position j + 1 + e; 0 <= e < lm
                if ((unsigned)e < (unsigned)lm) s[m] = s[m] + (double)Lc[e] * tmp;  // xGER in xGBTRS
            }
        }
        if (lane == (j & 31)) {
            w[j] = bj;
#pragma unroll
            for (int m = 0; m + 1 < FS; m++) s[m] = s[m + 1];
            s[FS - 1] = stage[fslot];
        }
        __syncwarp();
        issue_L(j + FWD_DEPTH, fslot);
        cp_commit();
        fslot = fslot + 1 == FWD_DEPTH ? 0 : fslot + 1;
    }
    cp_wait<0>();
    __syncwarp();
    if (lane == ((n - 1) & 31)) w[n - 1] = s[0];
    __syncwarp();

    // ---------------- backward: U, column oriented (xTBSV 'U','N','N') ------------
#pragma unroll
    for (int m = 0; m < BS; m++) {
        const int p = (n - 1) - ((n - 1 - lane) & 31) - 32 * m;
        s[m] = p >= 0 ? w[p] : 0.0;
    }
    // (slot: (n-1-col) mod BWD_DEPTH, kept as a running index by the caller)
    auto issue_U = [&](int col, int slot) {
        if (col >= 0) {
            T* dst = ring + slot * kvp;
            const T* src = Uf + (size_t)col * kvp;
            warp_copy16<BWD_WIN * 8 / 16 / 32>(dst, src, kvp / VEC, lane);
            if (lane == 0) {
                double* st = &stage[slot];
                if (col - BWIN >= 0) cp_async8(st, &w[col - BWIN]);
                else *st = 0.0;
            }
        }
    };
    for (int c = 0; c < BWD_DEPTH; c++) {
        issue_U(n - 1 - c, c);
        cp_commit();
    }
    int bslot = 0;  // (n-1-j) mod BWD_DEPTH
    for (int j = n - 1; j >= 0; j--) {
        cp_wait<BWD_DEPTH - 1>();
        __syncwarp();
        const T* Uc = ring + bslot * kvp;
        double bj = __shfl_sync(0xffffffffu, s[0], j & 31);
        if (bj != 0.0) {
            bj = bj / (double)Uc[kv];
            const int o = (j - lane) & 31;
            const unsigned dmax = (unsigned)min(kv, j);
#pragma unroll
            for (int m = 0; m < BS; m++) {
                const int d = o + 32 * m;  // position j - d; 1 <= d <= min(kv, j)
                if ((unsigned)(d - 1) < dmax)
                    s[m] = s[m] - bj * (double)Uc[kv - d];  // xTBSV: X(I) - TEMP*A(L+I,J)
            }
        }
        if (lane == (j & 31)) {
            w[j] = bj;
#pragma unroll
            for (int m = 0; m + 1 < BS; m++) s[m] = s[m + 1];
            s[BS - 1] = stage[bslot];
        }
        __syncwarp();
        issue_U(j - BWD_DEPTH, bslot);
        cp_commit();
        bslot = bslot + 1 == BWD_DEPTH ? 0 : bslot + 1;
    }
    cp_wait<0>();
}

// r = b - A x per unknown (refinement of the mixed-precision form).  A's row
// comes from assemble_row, so it is the matrix the factorisation saw; the
// 9-point product is summed in FP64.
__global__ void local_residual_kernel(LocalArgs a, const double* b, const double* x, double* r)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int nx = a.d.V;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const SysView v = sys_view(a, sys);
    int types[4] = {a.Vl_t, a.Vu_t, a.Kl_t, a.Ku_t};
    const size_t base = sys_uoff(a, sys);
    for (int in = blockIdx.x * blockDim.x + threadIdx.x; in < n; in += gridDim.x * blockDim.x) {
        double row[9];
        const int st = assemble_row(v, types, a.dt, in, row);
        if (st) set_error(a.status, st);
        double acc = b[base + in];
#pragma unroll
        for (int dy = -1; dy <= 1; dy++)
#pragma unroll
            for (int dx = -1; dx <= 1; dx++) {
                const double m = row[dslot(dx, dy)];
                const int col = in + dy * nx + dx;
                if (m != 0.0 && col >= 0 && col < n) acc -= m * x[base + col];
            }
        r[base + in] = acc;
    }
}

// x += d over every system (blockIdx.y); red[0] = max |d|, red[1] = max |x|
// as dkey values.
__global__ void local_update_kernel(LocalArgs a, double* x, const double* d, unsigned long long* red)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t base = sys_uoff(a, sys);
    double md = 0.0, mx = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = x[base + i] + d[base + i];
        x[base + i] = v;
        md = fmax(md, fabs(d[base + i]));
        mx = fmax(mx, fabs(v));
    }
    for (int o = 16; o > 0; o >>= 1) {
        md = fmax(md, __shfl_xor_sync(0xffffffffu, md, o));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&red[0], dkey(md));
        atomicMax(&red[1], dkey(mx));
    }
}

// ---------------------------------------------------------------------------
// Krylov form of the local solve (learned warm start).

__global__ void local_assemble32_kernel(LocalArgs a, float* A9)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const SysView v = sys_view(a, sys);
    int types[4] = {a.Vl_t, a.Vu_t, a.Kl_t, a.Ku_t};
    float* A = A9 + sys_uoff(a, sys) * 9;
    for (int in = blockIdx.x * blockDim.x + threadIdx.x; in < n; in += gridDim.x * blockDim.x) {
        double row[9];
        const int st = assemble_row(v, types, a.dt, in, row);
        if (st) set_error(a.status, st);
#pragma unroll
        for (int k = 0; k < 9; k++) A[(size_t)k * n + in] = (float)row[k];
    }
}

// block-wide sum of v (all threads get the result); red has 32 floats
__device__ __forceinline__ float block_sum(float v, float* red)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    float t = l < nw ? red[l] : 0.f;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

__device__ __forceinline__ float mv_row(const float* A, const float* y, int n, int nx, int i)
{
    float acc = 0.f;
#pragma unroll
    for (int dy = -1; dy <= 1; dy++)
#pragma unroll
        for (int dx = -1; dx <= 1; dx++) {
            const int col = i + dy * nx + dx;
            const float m = A[(size_t)((dy + 1) * 3 + (dx + 1)) * n + i];
            if (m != 0.f && col >= 0 && col < n) acc = fmaf(m, y[col], acc);
        }
    return acc;
}

// ---- learned preconditioner ----------------------------------------------
// M v (i) = sum over the 5 x 5 neighbourhood o of i of
//           (delta(o = 0) + C[o](i)) v(i + o) / diag(i + o)
// on the system's (V, K') grid (no wrap-around at its edges): a sparse
// approximate inverse whose 25 coefficients per unknown a CNN predicts from
// the matrix (C = 0 is the Jacobi preconditioner).  C is [sys][25][n], slot
// o = (dy + 2) * 5 + (dx + 2).
constexpr int PC_TAPS = 25;

__device__ __forceinline__ float precond_row(const float* C, const float* w, int n, int nx, int ny,
                                             int i)
{
    const int iy = i / nx, ix = i - iy * nx;
    float acc = 0.f;
#pragma unroll
    for (int dy = -2; dy <= 2; dy++) {
        const int yy = iy + dy;
        if (yy < 0 || yy >= ny) continue;
#pragma unroll
        for (int dx = -2; dx <= 2; dx++) {
            const int xx = ix + dx;
            if (xx < 0 || xx >= nx) continue;
            const int o = (dy + 2) * 5 + (dx + 2);
            const float c = C[(size_t)o * n + i] + (o == 12 ? 1.f : 0.f);
            acc = fmaf(c, w[yy * nx + xx], acc);
        }
    }
    return acc;
}

// features of the learned preconditioner, [sys][9][K'][V]: log10(|diag| dt)
// and the eight off-diagonal entries of each row over its diagonal
__global__ void precond_features_kernel(LocalArgs a, const float* A9, float* feat)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const float* A = A9 + u0 * 9;
    float* f = feat + u0 * 9;
    const float dt = (float)a.dt;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float d = A[(size_t)4 * n + i];
        f[i] = log10f(fmaxf(fabsf(d) * dt, 1e-30f));
        int c = 1;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            if (k == 4) continue;
            f[(size_t)c * n + i] = d != 0.f ? A[(size_t)k * n + i] / d : 0.f;
            c++;
        }
    }
}

// Training signal of the learned preconditioner for nprobe probe vectors z
// per system, on the Jacobi-scaled system (unit diagonal) so that every row
// counts alike whatever its scale: with A~ = D^-1 A and M~ = M D (the
// stencil of C without the division, so A M = I exactly when A~ M~ = I),
// y = M~ z, e = A~ y - z, loss += |e|^2 / cnt and
// gC[o](i) = (2 / cnt) sum_z (A^T D^-1 e)(i) z(i + o), the gradient of the
// loss with respect to C.  One CTA per system; z, y and e live in shared
// memory (3 n floats).
__global__ void precond_grad_kernel(const float* A9, const float* C, const float* Z, float* gC,
                                    float* loss, int nx, int ny, int nprobe, float inv_cnt)
{
    extern __shared__ float psm[];
    __shared__ float red[32];
    const int sys = blockIdx.x;
    const int n = nx * ny;
    const float* A = A9 + (size_t)sys * 9 * n;
    const float* dg = A + (size_t)4 * n;
    const float* Cs = C + (size_t)sys * PC_TAPS * n;
    float* g = gC + (size_t)sys * PC_TAPS * n;
    float* z = psm;
    float* y = z + n;
    float* e = y + n;
    for (size_t i = threadIdx.x; i < (size_t)PC_TAPS * n; i += blockDim.x) g[i] = 0.f;
    float lsum = 0.f;
    for (int q = 0; q < nprobe; q++) {
        const float* zq = Z + ((size_t)sys * nprobe + q) * n;
        for (int i = threadIdx.x; i < n; i += blockDim.x) z[i] = zq[i];
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            // y = M~ z: the stencil of delta + C on z
            const int iy = i / nx, ix = i - iy * nx;
            float acc = 0.f;
#pragma unroll
            for (int dy = -2; dy <= 2; dy++) {
                const int yy = iy + dy;
                if (yy < 0 || yy >= ny) continue;
#pragma unroll
                for (int dx = -2; dx <= 2; dx++) {
                    const int xx = ix + dx;
                    if (xx < 0 || xx >= nx) continue;
                    const int o = (dy + 2) * 5 + (dx + 2);
                    acc = fmaf(Cs[(size_t)o * n + i] + (o == 12 ? 1.f : 0.f), z[yy * nx + xx], acc);
                }
            }
            y[i] = acc;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float ei = mv_row(A, y, n, nx, i) / dg[i] - z[i];
            e[i] = ei / dg[i];  // D^-1 e, the operand of A^T below
            lsum = fmaf(ei, ei, lsum);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            // (A^T D^-1 e)(i): rows r = i - off with A[k](r) multiplying x(r + off)
            float gy = 0.f;
#pragma unroll
            for (int dy = -1; dy <= 1; dy++)
#pragma unroll
                for (int dx = -1; dx <= 1; dx++) {
                    const int r = i - (dy * nx + dx);
                    if (r < 0 || r >= n) continue;
                    gy = fmaf(A[(size_t)((dy + 1) * 3 + (dx + 1)) * n + r], e[r], gy);
                }
            gy *= 2.f * inv_cnt;
            const int iy = i / nx, ix = i - iy * nx;
#pragma unroll
            for (int dy = -2; dy <= 2; dy++) {
                const int yy = iy + dy;
                if (yy < 0 || yy >= ny) continue;
#pragma unroll
                for (int dx = -2; dx <= 2; dx++) {
                    const int xx = ix + dx;
                    if (xx < 0 || xx >= nx) continue;
                    g[(size_t)((dy + 2) * 5 + (dx + 2)) * n + i] += gy * z[yy * nx + xx];
                }
            }
        }
        __syncthreads();
    }
    lsum = block_sum(lsum, red);
    if (threadIdx.x == 0) atomicAdd(loss, lsum * inv_cnt);
}

// One CTA per system.  Right preconditioning with M = diag(A) (Jacobi), or
// the learned sparse approximate inverse when Cp is given:
// van der Vorst's BiCGSTAB on A M^-1 u = r, d = M^-1 u accumulated directly.
__global__ void bicgstab_kernel(LocalArgs a, const float* A9, const float* Cp, const double* rr,
                                double* dd, float* scratch, int maxit, float tol, int* iters,
                                unsigned char* ok)
{
    __shared__ float red[32];
    const int sys = blockIdx.x;
    if (skip_system(a, sys)) return;
    const int nx = a.d.V;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const float* A = A9 + u0 * 9;
    const float* dg = A + (size_t)4 * n;
    float* r = scratch + u0 * 6;
    float* rh = r + n;
    float* p = rh + n;
    float* v = p + n;
    float* y = v + n;  // y, then z
    float* t = y + n;
    double* d = dd + u0;
    const double* b = rr + u0;
    const float* Cs = Cp ? Cp + u0 * PC_TAPS : nullptr;
    const int ny = n / nx;
    float bn = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float bi = (float)b[i];
        r[i] = bi;
        rh[i] = bi;
        p[i] = 0.f;
        v[i] = 0.f;
        d[i] = 0.0;
        bn = fmaf(bi, bi, bn);
    }
    bn = sqrtf(block_sum(bn, red));
    float rho = 1.f, alpha = 1.f, omega = 1.f;
    int it = 0;
    bool conv = bn == 0.f;
    while (!conv && it < maxit) {
        it++;
        float rho1 = 0.f;
        for (int i = threadIdx.x; i < n; i += blockDim.x) rho1 = fmaf(rh[i], r[i], rho1);
        rho1 = block_sum(rho1, red);
        if (rho1 == 0.f || !isfinite(rho1)) break;
        const float beta = (rho1 / rho) * (alpha / omega);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            p[i] = r[i] + beta * (p[i] - omega * v[i]);
            if (!Cs) y[i] = p[i] / dg[i];
        }
        __syncthreads();
        if (Cs) {
            // M p = (I + C) D^-1 p: the scaled vector once (t is free here)
            for (int i = threadIdx.x; i < n; i += blockDim.x) t[i] = p[i] / dg[i];
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = precond_row(Cs, t, n, nx, ny, i);
            __syncthreads();
        }
        float rv = 0.f;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float vi = mv_row(A, y, n, nx, i);
            v[i] = vi;
            rv = fmaf(rh[i], vi, rv);
        }
        rv = block_sum(rv, red);
        if (rv == 0.f || !isfinite(rv)) break;
        alpha = rho1 / rv;
        float sn = 0.f;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            d[i] += (double)(alpha * y[i]);
            const float si = r[i] - alpha * v[i];
            r[i] = si;  // r now holds s
            sn = fmaf(si, si, sn);
        }
        sn = sqrtf(block_sum(sn, red));
        if (sn <= tol * bn) {
            conv = true;
            break;
        }
        if (Cs) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) t[i] = r[i] / dg[i];
            __syncthreads();  // every scaled s entry is written before M reads its neighbours
            for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = precond_row(Cs, t, n, nx, ny, i);
        } else {
            for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = r[i] / dg[i];  // z
        }
        __syncthreads();
        float ts = 0.f, tt = 0.f;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float ti = mv_row(A, y, n, nx, i);
            t[i] = ti;
            ts = fmaf(ti, r[i], ts);
            tt = fmaf(ti, ti, tt);
        }
        ts = block_sum(ts, red);
        tt = block_sum(tt, red);
        if (tt == 0.f || !isfinite(tt)) break;
        omega = ts / tt;
        float rn = 0.f;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            d[i] += (double)(omega * y[i]);
            const float ri = r[i] - omega * t[i];
            r[i] = ri;
            rn = fmaf(ri, ri, rn);
        }
        rn = sqrtf(block_sum(rn, red));
        if (rn <= tol * bn) conv = true;
        if (omega == 0.f) break;
        rho = rho1;
    }
    if (threadIdx.x == 0) {
        iters[sys] += it;
        if (ok) ok[sys] = conv ? 1 : 0;
    }
}

// the PSD of every system in the unknown order (the state the step starts from)
__global__ void gather_state_kernel(LocalArgs a, double* x)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int V = a.d.V, K = a.d.K, kz = sys_k0(a, sys), n = V * (K - kz);
    const size_t u0 = sys_uoff(a, sys);
    const double* f = a.psd + (size_t)sys * V * K + kz;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int iy = i / V, iv = i - iy * V;
        x[u0 + i] = f[(size_t)iv * K + iy];
    }
}

// features [sys][4][K'][V] over the system's pitch-angle rows (K' = K - k0);
// f is the state the step starts from (unknown order)
__global__ void local_features_kernel(LocalArgs a, const double* fstate, float* feat, double* scale)
{
    __shared__ float red[32];
    const int sys = blockIdx.x;
    if (skip_system(a, sys)) return;
    const int V = a.d.V, K = a.d.K, kz = sys_k0(a, sys), ny = K - kz;
    const int n = V * ny;
    const size_t u0 = sys_uoff(a, sys);
    const double* b = fstate + u0;
    float m = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, fabsf((float)b[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t = fmaxf(t, red[w]);
        red[0] = t > 0.f ? t : 1.f;
    }
    __syncthreads();
    const float sc = red[0];
    if (threadIdx.x == 0) scale[sys] = sc;
    const size_t fb = (size_t)sys * V * K;  // field slab [V][K]
    const float med = log10f(1e-5f * 86400.f);
    float* f = feat + u0 * 4;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int iy = i / V, iv = i - iy * V;
        const size_t g = fb + (size_t)iv * K + kz + iy;
        const float dvv = (float)a.DVV[g], dkk = (float)a.DKK[g], dvk = (float)a.DVK[g];
        f[i] = (log10f(dvv) - med) * 0.5f;
        f[(size_t)n + i] = (log10f(dkk) - med) * 0.5f;
        f[(size_t)2 * n + i] = dvk / sqrtf(dvv * dkk);
        f[(size_t)3 * n + i] = (float)b[i] / sc;
    }
}

__global__ void warm_start_kernel(LocalArgs a, const double* b, const float* out, const double* scale,
                                  double* x)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const double s = scale[sys];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[u0 + i] = out ? b[u0 + i] + (double)out[u0 + i] * s : b[u0 + i];
}

__global__ void local_targets_kernel(LocalArgs a, const double* b, const double* x, const double* scale,
                                     float* target)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const double s = scale[sys];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        target[u0 + i] = (float)((x[u0 + i] - b[u0 + i]) / s);
}

__global__ void residual_check_kernel(LocalArgs a, const double* b, const double* x, double tol,
                                      double stall, double* prev, unsigned char* pend,
                                      unsigned int* cnt, unsigned long long* maxkey)
{
    __shared__ double rmax[32], bmax[32];
    const int sys = blockIdx.x;
    if (skip_system(a, sys)) return;
    const int nx = a.d.V;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const SysView v = sys_view(a, sys);
    int types[4] = {a.Vl_t, a.Vu_t, a.Kl_t, a.Ku_t};
    const size_t base = sys_uoff(a, sys);
    double mr = 0.0, mb = 0.0;
    for (int in = threadIdx.x; in < n; in += blockDim.x) {
        double row[9];
        assemble_row(v, types, a.dt, in, row);
        double acc = b[base + in];
        for (int dy = -1; dy <= 1; dy++)
            for (int dx = -1; dx <= 1; dx++) {
                const double m = row[dslot(dx, dy)];
                const int col = in + dy * nx + dx;
                if (m != 0.0 && col >= 0 && col < n) acc -= m * x[base + col];
            }
        mr = fmax(mr, fabs(acc));
        mb = fmax(mb, fabs(b[base + in]));
    }
    for (int o = 16; o > 0; o >>= 1) {
        mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, o));
        mb = fmax(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    }
    if ((threadIdx.x & 31) == 0) {
        rmax[threadIdx.x >> 5] = mr;
        bmax[threadIdx.x >> 5] = mb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double R = 0, Bm = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            R = fmax(R, rmax[w]);
            Bm = fmax(Bm, bmax[w]);
        }
        const double rel = Bm > 0 ? R / Bm : R;
        const bool nan = !(rel == rel);
        unsigned char st = 0;
        if (!(rel <= tol)) {
            const double p = prev[sys];
            st = (nan || (p > 0 && rel > stall * p)) ? 2 : 1;
            atomicAdd(&cnt[st - 1], 1u);
        }
        pend[sys] = st;
        prev[sys] = nan ? 1e300 : rel;
        atomicMax(maxkey, dkey(nan ? 1e300 : rel));
    }
}

// weighted Jacobi sweep on the guess: x += omega * r / diag(A) (r = b - A x)
__global__ void jacobi_update_kernel(LocalArgs a, const float* A9, const double* r, double* x,
                                     double omega)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    const float* dg = A9 + u0 * 9 + (size_t)4 * n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[u0 + i] += omega * r[u0 + i] / (double)dg[i];
}

__global__ void masked_copy_kernel(LocalArgs a, double* x, const double* y)
{
    const int sys = blockIdx.y;
    if (skip_system(a, sys)) return;  // a.sel selects the systems to copy
    const int n = a.d.V * (a.d.K - sys_k0(a, sys));
    const size_t u0 = sys_uoff(a, sys);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[u0 + i] = y[u0 + i];
}

}  // namespace

void launch_local_residual(const LocalArgs& a, const double* b, const double* x, double* r,
                           cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    dim3 grid((n + 255) / 256, a.d.P * a.d.R);
    local_residual_kernel<<<grid, 256, 0, s>>>(a, b, x, r);
}

void launch_local_update(const LocalArgs& a, double* x, const double* d, unsigned long long* red,
                         cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    dim3 grid((n + 255) / 256, a.d.P * a.d.R);
    local_update_kernel<<<grid, 256, 0, s>>>(a, x, d, red);
}

void launch_local_assemble32(const LocalArgs& a, float* A9, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    local_assemble32_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, A9);
}

void launch_precond_features(const LocalArgs& a, const float* A9, float* feat, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    precond_features_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, A9, feat);
}

int launch_precond_grad(const float* A9, const float* C, const float* Z, float* gC, float* loss,
                        int nsys, int nx, int ny, int nprobe, cudaStream_t s)
{
    const size_t smem = (size_t)3 * nx * ny * sizeof(float);
    allow_max_dynamic_smem((const void*)precond_grad_kernel);
    int dev = 0, maxsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem + 32 * sizeof(float) > (size_t)maxsm) return VERB_ERR_SIZE;
    precond_grad_kernel<<<nsys, 256, smem, s>>>(A9, C, Z, gC, loss, nx, ny, nprobe,
                                                1.f / ((float)nsys * nprobe * nx * ny));
    return VERB_OK;
}

void launch_bicgstab(const LocalArgs& a, const float* A9, const float* Cp, const double* r, double* d,
                     float* scratch, int maxit, float tol, int* iters, unsigned char* ok,
                     cudaStream_t s)
{
    bicgstab_kernel<<<a.d.P * a.d.R, 256, 0, s>>>(a, A9, Cp, r, d, scratch, maxit, tol, iters, ok);
}

void launch_gather_state(const LocalArgs& a, double* x, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    gather_state_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, x);
}

void launch_local_features(const LocalArgs& a, const double* f, float* feat, double* scale,
                           cudaStream_t s)
{
    local_features_kernel<<<a.d.P * a.d.R, 256, 0, s>>>(a, f, feat, scale);
}

void launch_warm_start(const LocalArgs& a, const double* b, const float* out, const double* scale,
                       double* x, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    warm_start_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, b, out, scale, x);
}

void launch_local_targets(const LocalArgs& a, const double* b, const double* x, const double* scale,
                          float* target, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    local_targets_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, b, x, scale, target);
}

void launch_residual_check(const LocalArgs& a, const double* b, const double* x, double tol,
                           double stall, double* prev, unsigned char* pend, unsigned int* cnt,
                           unsigned long long* maxkey, cudaStream_t s)
{
    residual_check_kernel<<<a.d.P * a.d.R, 256, 0, s>>>(a, b, x, tol, stall, prev, pend, cnt,
                                                         maxkey);
}

void launch_jacobi_update(const LocalArgs& a, const float* A9, const double* r, double* x,
                          double omega, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    jacobi_update_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, A9, r, x, omega);
}

void launch_masked_copy(const LocalArgs& a, double* x, const double* y, cudaStream_t s)
{
    const int n = a.d.V * a.d.K;
    masked_copy_kernel<<<dim3((n + 255) / 256, a.d.P * a.d.R), 256, 0, s>>>(a, x, y);
}

size_t local_factor_smem(int V)
{
    const int kl = V + 1, kv = 2 * kl;
    return ((size_t)(kl + 1) * (kv + 1) + 2 * (kl + 1) + STAGE_ROWS * 9) * sizeof(double);
}

namespace {

template <typename T, int PW, int NW>
void launch_factor_blk(const LocalArgs& a, cudaStream_t s)
{
    const int kl = a.d.V + 1, kv = 2 * kl;
    dim3 g((a.d.V * a.d.K + 255) / 256, a.d.P * a.d.R);
    local_rows_kernel<T><<<g, 256, 0, s>>>(a);
    FBlk f{kl + NB, kv + NB, kv + NB};
    while (f.pitch % 16 != 2 && f.pitch % 16 != 14) f.pitch += 2;
    const size_t smem = ((size_t)f.RW * f.pitch + 2 * NB * 10 + NB * NB + 2 * PW * (NB + 4) + 2 * NB * NB) * sizeof(double);
    allow_max_dynamic_smem((const void*)local_factor_blk_kernel<T, PW, NW>);
    local_factor_blk_kernel<T, PW, NW><<<a.d.P * a.d.R, NW * 32, smem, s>>>(a, f);
}

// Whether the panel kernel takes the systems: a parked row needs 9 doubles of an
// L column (V >= 8, in FP32 V >= 16), and systems index grid.y of the parking launch.
bool factor_by_panels(const LocalArgs& a)
{
    return (a.factors32 ? a.klp32 >= 18 : a.klp >= 9) && a.d.P * a.d.R <= 65535;
}

template <typename T>
bool launch_factor_blk_t(const LocalArgs& a, cudaStream_t s)
{
    if (!factor_by_panels(a)) return false;
    // PW: the kl + NB rows of a panel, one a thread; the warps beside them share
    // the update.  The factorisation alone, ms by the warps in all:
    //   V = 16, 24 x 25 x 31:  2 0.451, 3 0.434, 4 0.447, 5 0.637 (FP32 0.447, 0.427, 0.440, 0.634)
    //   V = 31, 24 x 25 x 31:  3 1.116, 4 1.017, 6 1.088; V = 50: 3 2.62, 4 1.95, 6 1.76
    //   V = 60, 24 x 25 x 21:  6 2.49, 9 2.93, 12 2.87; V = 80, 24 x 25 x 15: 6 5.43, 9 4.56, 12 4.36
    //   V = 101, 24 x 51 x 21, the pass with upload and solve: 8 22.9, 12 18.9, 16 19.3 (15.5 by
    //   now with 12)
    // and panels of 16 columns instead of 8: V = 101 19.5-21.5 ms, V = 31 the pass of one run
    // 4.2 against 3.6.
    const int kl = a.d.V + 1;
    if (kl + NB <= 32) launch_factor_blk<T, 1, 3>(a, s);
    else if (kl + NB <= 64) launch_factor_blk<T, 2, 4>(a, s);
    else if (kl + NB <= 96) launch_factor_blk<T, 3, 9>(a, s);
    else launch_factor_blk<T, 4, 12>(a, s);
    return true;
}

}  // namespace

int launch_local_factor(const LocalArgs& a, cudaStream_t s)
{
    // The blocked kernel writes every entry of Uf (above row 0 and the padding
    // included) of the systems it factors; where some are skipped, and for the
    // window kernel, Uf is cleared first.
    if (!factor_by_panels(a) || !a.include_boundary || a.k0 || a.sel)
        cudaMemsetAsync(a.factors32 ? (void*)a.Uf32 : (void*)a.Uf, 0,
                        a.unknowns * (a.factors32 ? a.kvp32 * sizeof(float) : a.kvp * sizeof(double)), s);
    if (a.factors32 ? launch_factor_blk_t<float>(a, s) : launch_factor_blk_t<double>(a, s)) return 2;
    const size_t smem = local_factor_smem(a.d.V);
    if (a.factors32) {
        allow_max_dynamic_smem((const void*)local_factor_kernel<float>);
        local_factor_kernel<float><<<a.d.P * a.d.R, FACT_THREADS, smem, s>>>(a);
    } else {
        allow_max_dynamic_smem((const void*)local_factor_kernel<double>);
        local_factor_kernel<double><<<a.d.P * a.d.R, FACT_THREADS, smem, s>>>(a);
    }
    return 1;
}

void launch_local_rhs(const LocalArgs& a, bool from_work, cudaStream_t s)
{
    dim3 grid((a.d.K + 31) / 32, (a.d.V + 31) / 32, a.d.P * a.d.R);
    local_rhs_kernel<<<grid, dim3(32, 8), 0, s>>>(a, from_work ? 1 : 0);
}

void launch_local_store(const LocalArgs& a, cudaStream_t s)
{
    dim3 grid((a.d.K + 31) / 32, (a.d.V + 31) / 32, a.d.P * a.d.R);
    local_store_kernel<<<grid, dim3(32, 8), 0, s>>>(a);
}

namespace {

template <typename T, int W, int FD, int BD, int RW, int MB>
void launch_solve_t(const LocalArgs& a, const size_t kl_p, const size_t kv_p, cudaStream_t s)
{
    const int nsys = a.d.P * a.d.R;
    const int grid = (nsys + W - 1) / W;
    if (RW) {
        // slots of the register window: 32 FS > kl, 32 BS > kv
        const int fs = (a.kl + 1 + 31) / 32, bs = (a.kv + 1 + 31) / 32;
        constexpr int STAGE = (FD > BD ? FD : BD) + 1 & ~1;
        const size_t smem =
            (size_t)W * (STAGE + solve_ring_doubles((int)kl_p, (int)kv_p, sizeof(T), FD, BD)) *
            sizeof(double);
#define VERB_RW(F, B)                                                                         \
    if (fs <= F && bs <= B) {                                                                 \
        allow_max_dynamic_smem((const void*)local_solve_rw_kernel<T, W, FD, BD, F, B, MB>);   \
        local_solve_rw_kernel<T, W, FD, BD, F, B, MB><<<grid, W * 32, smem, s>>>(a, nsys);    \
        return;                                                                               \
    }
        VERB_RW(1, 1)
        VERB_RW(1, 2)
        VERB_RW(2, 3)
        VERB_RW(2, 4)
        VERB_RW(3, 5)
        VERB_RW(3, 6)
        VERB_RW(4, 7)
        VERB_RW(4, 8)
#undef VERB_RW
        // wider bands than the register window holds: the shared-memory window
    }
    const size_t smem =
        (size_t)W * (BWD_WIN + solve_ring_doubles((int)kl_p, (int)kv_p, sizeof(T), FD, BD)) *
        sizeof(double);
    allow_max_dynamic_smem((const void*)local_solve_kernel<T, W, FD, BD>);
    local_solve_kernel<T, W, FD, BD><<<grid, W * 32, smem, s>>>(a, nsys);
}

template <typename T>
void launch_solve_v(const LocalArgs& a, int v, size_t klp, size_t kvp, cudaStream_t s)
{
    switch (v) {
#define VERB_SOLVE_CASE(i)                                                                \
    case i:                                                                               \
        launch_solve_t<T, SOLVE_SHAPES[i].warps, SOLVE_SHAPES[i].fwd, SOLVE_SHAPES[i].bwd, \
                       SOLVE_SHAPES[i].rw, SOLVE_SHAPES[i].minb>(a, klp, kvp, s);         \
        break;
        VERB_SOLVE_CASE(1)
        VERB_SOLVE_CASE(2)
        VERB_SOLVE_CASE(3)
        VERB_SOLVE_CASE(4)
        VERB_SOLVE_CASE(5)
        VERB_SOLVE_CASE(6)
        VERB_SOLVE_CASE(7)
        VERB_SOLVE_CASE(8)
        VERB_SOLVE_CASE(9)
        VERB_SOLVE_CASE(10)
        VERB_SOLVE_CASE(11)
        VERB_SOLVE_CASE(12)
        VERB_SOLVE_CASE(13)
        VERB_SOLVE_CASE(14)
        VERB_SOLVE_CASE(15)
        VERB_SOLVE_CASE(16)
        VERB_SOLVE_CASE(17)
#undef VERB_SOLVE_CASE
        default:
            launch_solve_t<T, SOLVE_SHAPES[0].warps, SOLVE_SHAPES[0].fwd, SOLVE_SHAPES[0].bwd,
                           SOLVE_SHAPES[0].rw, 1>(a, klp, kvp, s);
    }
}

}  // namespace

static_assert(N_SOLVE_SHAPES == 18, "launch_solve_v lists every shape");

int local_solve_variants() { return N_SOLVE_SHAPES; }

void local_solve_variant_shape(int v, int* warps, int* fwd, int* bwd, int* rw)
{
    const SolveShape& sh = SOLVE_SHAPES[v >= 0 && v < N_SOLVE_SHAPES ? v : 0];
    *warps = sh.warps;
    *fwd = sh.fwd;
    *bwd = sh.bwd;
    if (rw) *rw = sh.rw;
}

// The shape a context takes that was not tuned.  One system per CTA with 16 L
// and 12 U columns in flight has the shortest column chain as long as the
// systems come in at most two waves (its ring leaves 11 resident on an SM at V =
// 101 in FP64): 24 x 25 x 31 x 31 0.48 ms against 0.57 for 4 x 4 x 3 and 0.77 for the
// shared-memory window 4 x 4 x 2, 24 x 51 x 101 x 21 1.39 / 1.56 / 2.48 ms, 48 x 101 x
// 61 x 12 1.07 / 1.14 / 1.44 ms.  Beyond that shallower rings with more systems
// resident: 48 x 101 x 101 x 12 2.53 ms (4 x 6 x 4) against 2.77 and 2.98 ms.
int local_solve_default(const LocalArgs& a)
{
    constexpr int deep = 14, wide = 10;
    static_assert(SOLVE_SHAPES[deep].warps == 1 && SOLVE_SHAPES[deep].fwd == 16 &&
                      SOLVE_SHAPES[wide].warps == 4 && SOLVE_SHAPES[wide].fwd == 6,
                  "the shapes the rule names");
    int dev = 0, sms = 148, smem = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    const size_t ring = a.factors32
        ? solve_ring_doubles(a.klp32, a.kvp32, sizeof(float), SOLVE_SHAPES[deep].fwd, SOLVE_SHAPES[deep].bwd)
        : solve_ring_doubles(a.klp, a.kvp, sizeof(double), SOLVE_SHAPES[deep].fwd, SOLVE_SHAPES[deep].bwd);
    const long long resident = smem / ((ring + 16) * 8 + 1024);
    return (long long)a.d.P * a.d.R <= 2 * resident * sms ? deep : wide;
}

void launch_local_solve(const LocalArgs& a, cudaStream_t s)
{
    const int v = a.solve_variant >= 0 ? a.solve_variant : local_solve_default(a);
    if (a.factors32)
        launch_solve_v<float>(a, v, a.klp32, a.kvp32, s);
    else
        launch_solve_v<double>(a, v, a.klp, a.kvp, s);
}

}  // namespace verb
