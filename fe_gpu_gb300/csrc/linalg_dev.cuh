// Device routines shared by the dense kernels of linalg.cu and the batched
// estimator (batch_est.cu): double-single products, and single-block k x k
// Cholesky solve and inverse, Jacobi eigensolver and covariance finalize (each
// run by one block of DN_THREADS threads).
#pragma once

#include "common.cuh"

namespace fegb {

constexpr int DN_THREADS = 256;

// acc_hi/acc_lo (+)= x * y in double-single arithmetic:
// (xh + xl)(yh + yl) = ph + pe + cross with ph + pe exact (TwoProd by FMA);
// TwoSum of the running high part and ph, its rounding error into the low part.
// (The _rn intrinsics are never contracted into FMAs, which TwoSum relies on.)
__device__ __forceinline__ void ds_fma(float2 x, float2 y, float& sh, float& sl) {
    const float ph = __fmul_rn(x.x, y.x);
    const float pe = fmaf(x.x, y.x, -ph);
    const float cr = fmaf(x.x, y.y, x.y * y.x);
    const float s1 = __fadd_rn(sh, ph);
    const float bb = __fsub_rn(s1, sh);
    const float err = __fadd_rn(__fsub_rn(sh, __fsub_rn(s1, bb)), __fsub_rn(ph, bb));
    sh = s1;
    sl += err + (pe + cr);
}

// Row stride and doubles of the two k x k work matrices of the dense routines:
// odd strides where they sit in shared memory (lanes walk down columns without
// bank conflicts). One block is bound by the latency of its steps: with the
// matrices in global memory and a thread per column, k = 90 took 1.08 ms and the
// eigensolver at k = 29 1.3; in shared memory, with the trailing matrix shared
// by all warps, k = 100 takes 0.50 ms and a 30-column fit of 38k rows 6.1 -> 5.6.
constexpr size_t DN_SMEM = 200 * 1024;
__host__ __device__ inline int dn_stride(int k) { return k | 1; }
__host__ __device__ inline size_t dn_work_bytes(int k) { return sizeof(double) * 2 * (size_t)k * dn_stride(k); }
__host__ __device__ inline bool dn_fits(int k) { return dn_work_bytes(k) <= DN_SMEM; }

// Upper Cholesky factor of the k x k matrix in U (row-major, stride ld, upper
// triangle used), in place: each pivot row is scaled and subtracted from the
// trailing rows, so an entry receives its terms in pivot order. Returns 0, or
// j > 0 when the leading minor j is not positive (on every thread).
__device__ inline int block_chol_factor(int k, double* U, int ld) {
    __shared__ int s_fail;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) s_fail = 0;
    __syncthreads();
    for (int j = 0; j < k; ++j) {
        double* rj = U + (size_t)j * ld;
        if (warp == 0) {
            const double d = rj[j];
            if (!(d > 0.0)) {
                if (lane == 0) s_fail = j + 1;
            } else {
                const double r = sqrt(d);
                __syncwarp();
                if (lane == 0) rj[j] = r;
                for (int c = j + 1 + lane; c < k; c += 32) rj[c] /= r;
            }
        }
        __syncthreads();
        if (s_fail) break;
        for (int r = j + 1 + warp; r < k; r += DN_THREADS / 32) {
            const double f = rj[r];
            double* row = U + (size_t)r * ld;
            for (int c = r + lane; c < k; c += 32) row[c] = fma(-f, rj[c], row[c]);
        }
        __syncthreads();
    }
    const int fail = s_fail;
    __syncthreads();
    return fail;
}

// One block of DN_THREADS threads: Q_sel = Q[idx, idx] (or the leading k x k
// block), upper Cholesky factor, solve for b_sel and the inverse. info: 0 ok,
// j > 0 when the leading minor j is not positive definite. work: 2 k ld doubles
// (global or shared), ld >= k. BY_COLUMN: a thread per column of the inverse and
// one for the back substitution, every sum over ascending indexes (stacked
// specifications, some of them so ill-conditioned that another order of these sums
// moves a standard error by 1e-7; up to 64 columns, where the longer chains cost
// some microseconds).
template <bool BY_COLUMN = false>
__device__ inline void chol_solve_inv_block(int k, const double* __restrict__ Q, int ldq, const int* __restrict__ idx,
                                     const double* __restrict__ b, double* __restrict__ beta,
                                     double* __restrict__ Qinv, int* __restrict__ info, double* work, int ld) {
    double* U = work;
    double* X = work + (size_t)k * ld;  // U^{-1}, row-major
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    for (int e = t; e < k * k; e += DN_THREADS) {
        int i = e % k, j = e / k;
        int qi = idx ? idx[i] : i, qj = idx ? idx[j] : j;
        U[(size_t)i * ld + j] = Q[qi + (long long)qj * ldq];
        X[(size_t)i * ld + j] = 0.0;
    }
    __syncthreads();
    const int fail = block_chol_factor(k, U, ld);
    if (fail) {
        if (t == 0) *info = fail;
        return;
    }
    // rows of U^{-1} from the last: X[i][j] gathers sum_p U[i][p] X[p][j] over the
    // finished rows p > i, then row i is -that / U[i][i]
    if (BY_COLUMN) {
        for (int j = t; j < k; j += DN_THREADS) {
            X[(size_t)j * ld + j] = 1.0 / U[(size_t)j * ld + j];
            for (int i = j - 1; i >= 0; --i) {
                const double* ui = U + (size_t)i * ld;
                double s = 0.0;
                for (int p = i + 1; p <= j; ++p) s = fma(ui[p], X[(size_t)p * ld + j], s);
                X[(size_t)i * ld + j] = -s / ui[i];
            }
        }
        __syncthreads();
    }
    for (int p = BY_COLUMN ? -1 : k - 1; p >= 0; --p) {
        double* xp = X + (size_t)p * ld;
        const double u = U[(size_t)p * ld + p];
        for (int j = p + t; j < k; j += DN_THREADS) xp[j] = j == p ? 1.0 / u : -xp[j] / u;
        __syncthreads();
        for (int i = warp; i < p; i += DN_THREADS / 32) {
            const double f = U[(size_t)i * ld + p];
            double* xi = X + (size_t)i * ld;
            for (int j = p + lane; j < k; j += 32) xi[j] = fma(f, xp[j], xi[j]);
        }
        __syncthreads();
    }
    // Qinv = U^{-1} U^{-T}
    for (int e = t; e < k * k; e += DN_THREADS) {
        int i = e % k, j = e / k;
        if (i > j) continue;
        double s = 0.0;
        for (int p = j; p < k; ++p) s += X[(size_t)i * ld + p] * X[(size_t)j * ld + p];
        Qinv[i + j * k] = s;
        Qinv[j + i * k] = s;
    }
    __syncthreads();
    // beta: forward then backward substitution by one warp, the right-hand side
    // in place of the first row of X
    if (warp == 0) {
        double* v = X;
        for (int i = lane; i < k; i += 32) v[i] = b[idx ? idx[i] : i];
        __syncwarp();
        for (int i = 0; i < k; ++i) {
            const double* ui = U + (size_t)i * ld;
            const double y = v[i] / ui[i];
            __syncwarp();
            if (lane == 0) v[i] = y;
            for (int c = i + 1 + lane; c < k; c += 32) v[c] = fma(-ui[c], y, v[c]);
            __syncwarp();
        }
        if (BY_COLUMN && lane == 0)
            for (int i = k - 1; i >= 0; --i) {
                const double* ui = U + (size_t)i * ld;
                double y = v[i];
                for (int p = i + 1; p < k; ++p) y = fma(-ui[p], v[p], y);
                v[i] = y / ui[i];
            }
        __syncwarp();
        for (int i = BY_COLUMN ? -1 : k - 1; i >= 0; --i) {
            const double y = v[i] / U[(size_t)i * ld + i];
            __syncwarp();
            if (lane == 0) v[i] = y;
            for (int c = lane; c < i; c += 32) v[c] = fma(-U[(size_t)c * ld + i], y, v[c]);
            __syncwarp();
        }
        for (int i = lane; i < k; i += 32) beta[i] = v[i];
        if (lane == 0) *info = 0;
    }
    __syncthreads();
}

// One block: whether the symmetric k x k matrix A (upper triangle read) has an
// upper Cholesky factor with positive pivots, i.e. is positive definite; the
// factor is formed in U (k ld doubles). The answer is the same on every thread.
__device__ inline bool block_cholesky_ok(int k, const double* __restrict__ A, double* U, int ld) {
    const int t = threadIdx.x;
    for (int e = t; e < k * k; e += DN_THREADS) U[(size_t)(e / k) * ld + e % k] = A[e / k + (long long)(e % k) * k];
    __syncthreads();
    return block_chol_factor(k, U, ld) == 0;
}

// Parallel cyclic Jacobi on a k x k symmetric matrix A (in place, stride
// ld), eigenvectors accumulated in V (stride ld); the round-robin pairing makes all
// rotations of one round touch disjoint rows/columns.
// Bound by the FP64 pipe of the one SM it runs on (the angles' divisions and
// roots, then the updates): columns and rows in one pass, half of A mirrored,
// one division, one root and one reciprocal root an angle: k = 29 887 -> 711 us.
__device__ inline void block_jacobi(int k, double* A, double* V, int ld) {
    __shared__ int sp[DN_THREADS], sq[DN_THREADS];
    __shared__ double sc[DN_THREADS], ss[DN_THREADS];
    __shared__ double s_off, s_tot;
    __shared__ double red[DN_THREADS / 32];
    const int t = threadIdx.x;
    for (int e = t; e < k * k; e += DN_THREADS) V[e % k + (size_t)(e / k) * ld] = (e % k == e / k) ? 1.0 : 0.0;
    const int kk = (k % 2) ? k + 1 : k;
    const int m = kk / 2;
    const int nup = m * (m + 1) / 2;
    __syncthreads();
    for (int sweep = 0; sweep < 60; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int e = t; e < k * k; e += DN_THREADS) {
            const double v = A[e % k + (size_t)(e / k) * ld], a = v * v;
            tot += a;
            if (e % k != e / k) off += a;
        }
        for (int pass = 0; pass < 2; ++pass) {
            double v = pass == 0 ? off : tot;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((t & 31) == 0) red[t >> 5] = v;
            __syncthreads();
            if (t == 0) {
                double s = 0.0;
                for (int w = 0; w < DN_THREADS / 32; ++w) s += red[w];
                if (pass == 0)
                    s_off = s;
                else
                    s_tot = s;
            }
            __syncthreads();
        }
        if (s_off == 0.0 || s_off <= 1e-30 * (s_tot > 0.0 ? s_tot : 1.0)) break;
        for (int round = 0; round < kk - 1; ++round) {
            for (int i = t; i < m; i += DN_THREADS) {
                int p, q;
                if (i == 0) {
                    p = round;
                    q = kk - 1;
                } else {
                    p = (round + i) % (kk - 1);
                    q = (round - i + (kk - 1)) % (kk - 1);
                }
                if (p > q) {
                    int tmp = p;
                    p = q;
                    q = tmp;
                }
                double c = 1.0, s = 0.0;
                if (q < k) {
                    double apq = A[p + q * ld];
                    if (apq != 0.0) {
                        double app = A[p + p * ld], aqq = A[q + q * ld];
                        // tan of the angle: b / (d + sign(d) hypot(d, b)), one division; scaled
                        // by b where the squares would leave the range
                        const double d = aqq - app, b = 2.0 * apq, h2 = d * d + b * b;
                        double tt;
                        if (h2 > 1e-280 && h2 < 1e280) {
                            const double h = sqrt(h2);
                            tt = b / (d >= 0.0 ? d + h : d - h);
                        } else {
                            const double theta = d / b;
                            tt = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                        }
                        c = rsqrt(tt * tt + 1.0);
                        s = tt * c;
                    }
                }
                sp[i] = p;
                sq[i] = q;
                sc[i] = c;
                ss[i] = s;
            }
            __syncthreads();
            // A <- J^T A J and V <- V J in one pass: the rotations' rows and columns are
            // disjoint, so the 2 x 2 block of rotation i's rows and rotation j's columns is
            // one thread's, columns first. Blocks i <= j are computed and mirrored: the
            // FP64 pipe of one SM is the bound.
            for (int e = t; e < nup + m * k; e += DN_THREADS) {
                if (e < nup) {
                    int i = e / (m + 1), j = e - i * (m + 1);  // rows i and m - 1 - i of the triangle, folded
                    if (j >= m - i) {
                        j -= m - i;
                        i = m - 1 - i;
                    }
                    j += i;
                    const int p = sp[i], q = sq[i], u = sp[j], w = sq[j];
                    const bool two_r = q < k, two_c = w < k;  // else the odd row out
                    const double si = ss[i], sj = ss[j];
                    if (si == 0.0 && sj == 0.0) continue;
                    const double ci = sc[i], cj = sc[j];
                    double apu = A[p + u * ld], apw = two_c ? A[p + w * ld] : 0.0;
                    double aqu = two_r ? A[q + u * ld] : 0.0, aqw = two_r && two_c ? A[q + w * ld] : 0.0;
                    if (sj != 0.0) {
                        const double xp = apu, xq = aqu;
                        apu = cj * xp - sj * apw;
                        apw = sj * xp + cj * apw;
                        aqu = cj * xq - sj * aqw;
                        aqw = sj * xq + cj * aqw;
                    }
                    if (si != 0.0) {
                        const double xu = apu, xw = apw;
                        apu = ci * xu - si * aqu;
                        aqu = si * xu + ci * aqu;
                        apw = ci * xw - si * aqw;
                        aqw = si * xw + ci * aqw;
                    }
                    A[p + u * ld] = A[u + p * ld] = apu;
                    if (two_c) A[p + w * ld] = A[w + p * ld] = apw;
                    if (two_r && i != j) A[q + u * ld] = A[u + q * ld] = aqu;
                    if (two_r && two_c) A[q + w * ld] = A[w + q * ld] = aqw;
                } else {
                    const int f = e - nup, j = f / k, r = f - j * k;
                    const int u = sp[j], w = sq[j];
                    const double s = ss[j];
                    if (w >= k || s == 0.0) continue;
                    const double c = sc[j], vu = V[r + u * ld], vw = V[r + w * ld];
                    V[r + u * ld] = c * vu - s * vw;
                    V[r + w * ld] = s * vu + c * vw;
                }
            }
            __syncthreads();
        }
    }
}

// One block: acc *= scalar, then the PSD fix (mirror, Jacobi, clamp
// negative eigenvalues, rebuild) or the CPU path's symmetrisation; se[i] =
// sqrt(max(0, acc[i, i])). work: 2 k ld doubles, ld >= k.
__device__ inline void finalize_cov_block(int k, double* __restrict__ acc, double scalar, int do_psd,
                                   double* __restrict__ se, int* __restrict__ psd_applied,
                                   double* work, int ld) {
    const int t = threadIdx.x;
    double* A = work;
    double* V = work + (size_t)k * ld;
    __shared__ int s_applied;
    if (t == 0) s_applied = 0;
    for (int e = t; e < k * k; e += DN_THREADS) acc[e] *= scalar;
    __syncthreads();
    if (!do_psd) {
        // 0.5 (A + A^T), as the CPU path does (fe_pipeline.f90:476)
        for (int e = t; e < k * k; e += DN_THREADS) {
            int i = e % k, j = e / k;
            A[i + (size_t)j * ld] = 0.5 * (acc[i + j * k] + acc[j + i * k]);
        }
        __syncthreads();
        for (int e = t; e < k * k; e += DN_THREADS) acc[e] = A[e % k + (size_t)(e / k) * ld];
        __syncthreads();
        for (int i = t; i < k; i += DN_THREADS) se[i] = sqrt(fmax(0.0, acc[i + i * k]));
        if (t == 0) *psd_applied = 0;
        return;
    }
    // mirror the upper triangle to the lower (fe_pipeline.f90:1366, 1802-1811)
    for (int e = t; e < k * k; e += DN_THREADS) {
        int i = e % k, j = e / k;
        if (i > j) acc[e] = acc[j + i * k];
    }
    __syncthreads();
    for (int e = t; e < k * k; e += DN_THREADS) A[e % k + (size_t)(e / k) * ld] = acc[e];
    __syncthreads();
    // A positive definite matrix has no negative eigenvalue to clamp, and its
    // reconstruction V diag(lambda) V' is the matrix itself up to rounding:
    // the eigensolver (0.71 ms at k = 29) runs only when the Cholesky
    // factorisation fails
    if (block_cholesky_ok(k, acc, V, ld)) {
        for (int i = t; i < k; i += DN_THREADS) se[i] = sqrt(fmax(0.0, acc[i + i * k]));
        if (t == 0) *psd_applied = 0;
        return;
    }
    block_jacobi(k, A, V, ld);
    __syncthreads();
    // lambda_j = A[j,j]; scale eigenvector columns by sqrt(max(lambda,0))
    for (int e = t; e < k * k; e += DN_THREADS) {
        int j = e / k;
        double lam = A[j + (size_t)j * ld];
        if (lam < 0.0) {
            s_applied = 1;
            lam = 0.0;
        }
        V[e % k + (size_t)j * ld] *= lam > 0.0 ? sqrt(lam) : 0.0;
    }
    __syncthreads();
    for (int e = t; e < k * k; e += DN_THREADS) {
        int i = e % k, j = e / k;
        double s = 0.0;
        for (int p = 0; p < k; ++p) s += V[i + (size_t)p * ld] * V[j + (size_t)p * ld];
        acc[e] = s;
    }
    __syncthreads();
    for (int i = t; i < k; i += DN_THREADS) se[i] = sqrt(fmax(0.0, acc[i + i * k]));
    if (t == 0) *psd_applied = s_applied;
}

}  // namespace fegb
