// Tall-skinny reductions and small dense kernels (see linalg.cuh).
#include "linalg.cuh"
#include "linalg_dev.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace fegb {

namespace {

constexpr int CP_THREADS = 256;
constexpr int CP_TR = 16;
constexpr int CP_MAXPAIRS_LAUNCH = 8192;

struct CPParams {
    const double* A;
    long long ars, acs;
    int a;
    const double* B;
    long long brs, bcs;
    int b;
    long long n;
    int gram;
    long long p0;      // first pair index of this launch
    int npairs;        // pairs in this launch
    int phases;        // row phases (PPT == 1 mode)
    long long rows_per_block;
    double* partials;  // nblocks x npairs
};

__device__ __forceinline__ void pair_ij(long long p, int gram, int a, int& i, int& j) {
    if (gram) {
        int jj = (int)((sqrt(8.0 * (double)p + 1.0) - 1.0) * 0.5);
        while ((long long)(jj + 1) * (jj + 2) / 2 <= p) ++jj;
        while ((long long)jj * (jj + 1) / 2 > p) --jj;
        j = jj;
        i = (int)(p - (long long)jj * (jj + 1) / 2);
    } else {
        i = (int)(p % a);
        j = (int)(p / a);
    }
}

__device__ __forceinline__ void load_tile(double* dst, const double* src, long long rs, long long cs, int width,
                                          long long row0, int rows) {
    const int total = rows * width;
    if (rs == 1) {
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            int r = e % rows, c = e / rows;
            dst[r * width + c] = src[(row0 + r) + (long long)c * cs];
        }
    } else {
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            int r = e / width, c = e % width;
            dst[r * width + c] = src[(row0 + r) * rs + (long long)c * cs];
        }
    }
}

template <int PPT>
__global__ void __launch_bounds__(CP_THREADS) crossprod_kernel(CPParams p) {
    extern __shared__ double sm[];
    double* sA = sm;
    double* sB = p.gram ? sm : sm + CP_TR * p.a;
    const int t = threadIdx.x;
    int pi[PPT], pj[PPT];
    bool pv[PPT];
    double acc[PPT];
    int phase = 0;
    if (PPT == 1) {
        int local = t % p.npairs;
        phase = t / p.npairs;
        pv[0] = phase < p.phases;
        pair_ij(p.p0 + local, p.gram, p.a, pi[0], pj[0]);
        acc[0] = 0.0;
    } else {
#pragma unroll
        for (int s = 0; s < PPT; ++s) {
            int local = t + s * CP_THREADS;
            pv[s] = local < p.npairs;
            pair_ij(p.p0 + (pv[s] ? local : 0), p.gram, p.a, pi[s], pj[s]);
            acc[s] = 0.0;
        }
    }
    const long long r0 = (long long)blockIdx.x * p.rows_per_block;
    const long long r1 = min(p.n, r0 + p.rows_per_block);
    for (long long tile = r0; tile < r1; tile += CP_TR) {
        const int rows = (int)min((long long)CP_TR, r1 - tile);
        load_tile(sA, p.A, p.ars, p.acs, p.a, tile, rows);
        if (!p.gram) load_tile(sB, p.B, p.brs, p.bcs, p.b, tile, rows);
        __syncthreads();
        if (PPT == 1) {
            if (pv[0])
                for (int r = phase; r < rows; r += p.phases) acc[0] += sA[r * p.a + pi[0]] * sB[r * p.b + pj[0]];
        } else {
            for (int r = 0; r < rows; ++r) {
#pragma unroll
                for (int s = 0; s < PPT; ++s)
                    if (pv[s]) acc[s] += sA[r * p.a + pi[s]] * sB[r * p.b + pj[s]];
            }
        }
        __syncthreads();
    }
    if (PPT == 1) {
        // fold row phases in a fixed order
        __shared__ double fold[CP_THREADS];
        fold[t] = pv[0] ? acc[0] : 0.0;
        __syncthreads();
        if (t < p.npairs) {
            double v = 0.0;
            for (int ph = 0; ph < p.phases; ++ph) v += fold[ph * p.npairs + t];
            p.partials[(long long)blockIdx.x * p.npairs + t] = v;
        }
    } else {
#pragma unroll
        for (int s = 0; s < PPT; ++s)
            if (pv[s]) p.partials[(long long)blockIdx.x * p.npairs + t + s * CP_THREADS] = acc[s];
    }
}

// One warp per output entry: lanes take the row blocks b = lane, lane + 32, ...
// in order, then a fixed shuffle tree.
__global__ void crossprod_reduce_kernel(const double* __restrict__ partials, int nblocks, int npairs, long long p0,
                                        int gram, int upper_only, int a, double alpha, double beta, double* out,
                                        int ldo) {
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t >= npairs) return;
    double v = 0.0;
    for (int b = lane; b < nblocks; b += 32) v += partials[(long long)b * npairs + t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane != 0) return;
    int i, j;
    pair_ij(p0 + t, gram, a, i, j);
    double* o = out + i + (long long)j * ldo;
    *o = alpha * v + (beta != 0.0 ? beta * (*o) : 0.0);
    if (gram && !upper_only && i != j) {
        double* o2 = out + j + (long long)i * ldo;
        *o2 = alpha * v + (beta != 0.0 ? beta * (*o2) : 0.0);
    }
}

inline unsigned reduce_blocks(long long npairs) { return (unsigned)((npairs * 32 + 255) / 256); }

constexpr int RS_THREADS = 256;

__global__ void __launch_bounds__(RS_THREADS)
    residual_scores_kernel(const double* __restrict__ X, int C, long long n, const double* __restrict__ beta, int k,
                           const int* __restrict__ score_cols, int n_score, double* __restrict__ S,
                           double* __restrict__ resid, double* __restrict__ partials) {
    __shared__ double red[RS_THREADS / 32];
    double local = 0.0;
    long long i = (long long)blockIdx.x * RS_THREADS + threadIdx.x;
    const long long stride = (long long)gridDim.x * RS_THREADS;
    for (; i < n; i += stride) {
        const double* row = X + i * C;
        double r = row[0];
        for (int j = 0; j < k; ++j) r -= row[1 + j] * beta[j];
        if (resid) resid[i] = r;
        if (S)
            for (int t = 0; t < n_score; ++t) S[i * n_score + t] = r * row[score_cols[t]];
        local += r * r;
    }
    // fixed-shape tree: warp then block
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < RS_THREADS / 32; ++w) v += red[w];
        partials[blockIdx.x] = v;
    }
}

// The same for wide rows (many regressors): one warp per row, lanes over the
// columns, so that reads of X and writes of S are contiguous runs (a thread
// per row made every load and store instruction touch 32 rows); the lanes'
// partial products are summed by a fixed xor tree.
__global__ void __launch_bounds__(RS_THREADS)
    residual_scores_wide_kernel(const double* __restrict__ X, int C, long long n, const double* __restrict__ beta,
                                int k, const int* __restrict__ score_cols, int n_score, double* __restrict__ S,
                                double* __restrict__ resid, double* __restrict__ partials) {
    __shared__ double red[RS_THREADS / 32];
    const int lane = threadIdx.x & 31;
    double local = 0.0;
    long long i = ((long long)blockIdx.x * RS_THREADS + threadIdx.x) >> 5;
    const long long stride = ((long long)gridDim.x * RS_THREADS) >> 5;
    for (; i < n; i += stride) {
        const double* row = X + i * C;
        double dot = 0.0;
        for (int j = lane; j < k; j += 32) dot += row[1 + j] * beta[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const double r = row[0] - dot;
        if (resid && lane == 0) resid[i] = r;
        if (S)
            for (int t = lane; t < n_score; t += 32) S[i * n_score + t] = r * row[score_cols[t]];
        if (lane == 0) local += r * r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (lane == 0) red[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < RS_THREADS / 32; ++w) v += red[w];
        partials[blockIdx.x] = v;
    }
}

// Fixed-shape tree: thread t adds elements t, t + 256, ... in order, then warps
// and the block (one thread adding 1216 partials took 60 us).
__global__ void __launch_bounds__(RS_THREADS) sum_partials_kernel(const double* __restrict__ partials, int nb, double* out) {
    __shared__ double red[RS_THREADS / 32];
    double v = 0.0;
    for (int b = threadIdx.x; b < nb; b += RS_THREADS) v += partials[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < RS_THREADS / 32; ++w) t += red[w];
        *out = t;
    }
}

// ---------------------------- dense kernels ------------------------------


__global__ void __launch_bounds__(DN_THREADS)
    chol_solve_inv_kernel(int k, const double* __restrict__ Q, int ldq, const int* __restrict__ idx,
                          const double* __restrict__ b, double* __restrict__ beta, double* __restrict__ Qinv,
                          int* __restrict__ info, double* __restrict__ work) {
    extern __shared__ __align__(16) unsigned char dn_smem[];
    if (dn_fits(k))
        chol_solve_inv_block(k, Q, ldq, idx, b, beta, Qinv, info, reinterpret_cast<double*>(dn_smem), dn_stride(k));
    else
        chol_solve_inv_block(k, Q, ldq, idx, b, beta, Qinv, info, work, k);
}

__global__ void gemm_small_kernel(int ta, int tb, int m, int n, int k, double alpha, const double* __restrict__ A,
                                  int lda, const double* __restrict__ B, int ldb, double beta, double* __restrict__ C,
                                  int ldc) {
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)m * n) return;
    int i = (int)(e % m), j = (int)(e / m);
    double s = 0.0;
    for (int p = 0; p < k; ++p) {
        double av = ta ? A[p + (long long)i * lda] : A[i + (long long)p * lda];
        double bv = tb ? B[j + (long long)p * ldb] : B[p + (long long)j * ldb];
        s += av * bv;
    }
    double* o = C + i + (long long)j * ldc;
    *o = alpha * s + (beta != 0.0 ? beta * (*o) : 0.0);
}

__global__ void select_kernel(int k, const double* __restrict__ M, int ldm, const int* __restrict__ idx,
                              double* __restrict__ out) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= k * k) return;
    int i = e % k, j = e / k;
    int mi = idx ? idx[i] : i, mj = idx ? idx[j] : j;
    out[e] = M[mi + (long long)mj * ldm];
}

__global__ void __launch_bounds__(DN_THREADS)
    finalize_cov_kernel(int k, double* __restrict__ acc, double scalar, int do_psd, double* __restrict__ se,
                        int* __restrict__ psd_applied, double* __restrict__ work) {
    extern __shared__ __align__(16) unsigned char dn_smem[];
    if (dn_fits(k))
        finalize_cov_block(k, acc, scalar, do_psd, se, psd_applied, reinterpret_cast<double*>(dn_smem), dn_stride(k));
    else
        finalize_cov_block(k, acc, scalar, do_psd, se, psd_applied, work, k);
}

}  // namespace

int crossprod(const MatView& A, const MatView& B, long long n, bool gram, bool upper_only, double alpha, double beta,
              double* out, int ldo, cudaStream_t s, Scratch& scr) {
    const int a = A.cols, b = gram ? A.cols : B.cols;
    if (a <= 0 || b <= 0) return 0;
    const long long total_pairs = gram ? (long long)a * (a + 1) / 2 : (long long)a * b;
    if (n <= 0) {
        // A^T B over zero rows is the zero matrix
        for (long long p0 = 0; p0 < total_pairs; p0 += CP_MAXPAIRS_LAUNCH) {
            int np = (int)std::min<long long>(CP_MAXPAIRS_LAUNCH, total_pairs - p0);
            double* zeros = nullptr;
            FEGB_TRY(scr.alloc(&zeros, (size_t)np, "crossprod zeros"));
            FEGB_CUDA(cudaMemsetAsync(zeros, 0, sizeof(double) * np, s), "crossprod zero");
            crossprod_reduce_kernel<<<reduce_blocks(np), 256, 0, s>>>(zeros, 1, np, p0, gram, upper_only, a, alpha,
                                                                      beta, out, ldo);
            FEGB_LAUNCH_CHECK("crossprod zero reduce");
        }
        return 0;
    }
    long long nb = std::min<long long>((n + CP_TR - 1) / CP_TR, (long long)num_sms() * 4);
    long long rpb = (n + nb - 1) / nb;
    rpb = ((rpb + CP_TR - 1) / CP_TR) * CP_TR;
    nb = (n + rpb - 1) / rpb;
    size_t smem = sizeof(double) * CP_TR * (gram ? a : a + b);
    if (smem > 200 * 1024) return set_error("crossprod: %d x %d columns exceed the shared-memory tile", a, b);
    // set once (thread-safe static initialisation) before any launch with a large tile
    static const cudaError_t attr_status = []() {
        cudaError_t e = cudaSuccess;
        const int lim = 200 * 1024;
        if (e == cudaSuccess) e = cudaFuncSetAttribute(crossprod_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(crossprod_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(crossprod_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(crossprod_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(crossprod_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        return e;
    }();
    if (attr_status != cudaSuccess) return set_cuda_error(attr_status, "crossprod attr");
    for (long long p0 = 0; p0 < total_pairs; p0 += CP_MAXPAIRS_LAUNCH) {
        const int np = (int)std::min<long long>(CP_MAXPAIRS_LAUNCH, total_pairs - p0);
        double* partials = nullptr;
        FEGB_TRY(scr.alloc(&partials, (size_t)nb * np, "crossprod partials"));
        CPParams p;
        p.A = A.ptr;
        p.ars = A.rs;
        p.acs = A.cs;
        p.a = a;
        p.B = gram ? A.ptr : B.ptr;
        p.brs = gram ? A.rs : B.rs;
        p.bcs = gram ? A.cs : B.cs;
        p.b = b;
        p.n = n;
        p.gram = gram ? 1 : 0;
        p.p0 = p0;
        p.npairs = np;
        p.phases = np <= 128 ? CP_THREADS / np : 1;
        p.rows_per_block = rpb;
        p.partials = partials;
        if (np <= 128)
            crossprod_kernel<1><<<(unsigned)nb, CP_THREADS, smem, s>>>(p);
        else if (np <= 4 * CP_THREADS)
            crossprod_kernel<4><<<(unsigned)nb, CP_THREADS, smem, s>>>(p);
        else if (np <= 8 * CP_THREADS)
            crossprod_kernel<8><<<(unsigned)nb, CP_THREADS, smem, s>>>(p);
        else if (np <= 16 * CP_THREADS)
            crossprod_kernel<16><<<(unsigned)nb, CP_THREADS, smem, s>>>(p);
        else
            crossprod_kernel<32><<<(unsigned)nb, CP_THREADS, smem, s>>>(p);
        FEGB_LAUNCH_CHECK("crossprod");
        crossprod_reduce_kernel<<<reduce_blocks(np), 256, 0, s>>>(partials, (int)nb, np, p0, gram, upper_only, a, alpha,
                                                                  beta, out, ldo);
        FEGB_LAUNCH_CHECK("crossprod reduce");
    }
    return 0;
}

// ------------------------- tensor-core Gram products -------------------------

int crossprod_split(const MatView& A, long long n, bool upper_only, double alpha, double beta, double* out, int ldo,
                    cudaStream_t s, Scratch& scr) {
    const int a = A.cols;
    if (a <= 0) return 0;
    // row-major rows whose tiles' byte offsets fit 32 bits, and a bounded number of column blocks
    if (n <= 0 || A.cs != 1 || A.rs < a || A.rs > 65536 || a > CROSSPROD_SPLIT_MAX_COLS)
        return crossprod(A, A, n, true, upper_only, alpha, beta, out, ldo, s, scr);
    int* bad = nullptr;
    FEGB_TRY(scr.alloc(&bad, 1, "gram flag"));
    FEGB_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s), "gram flag reset");
    const long long np = (long long)a * (a + 1) / 2;
    double* partials = nullptr;
    int nb = 0;
    FEGB_TRY(launch_gram_umma(A.ptr, A.rs, a, n, scr, &partials, &nb, bad, s));
    crossprod_reduce_kernel<<<reduce_blocks(np), 256, 0, s>>>(partials, nb, (int)np, 0, 1, upper_only, a, alpha, beta,
                                                              out, ldo);
    FEGB_LAUNCH_CHECK("gram reduce");
    int hbad = 0;
    FEGB_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s), "gram flag copy");
    FEGB_CUDA(cudaStreamSynchronize(s), "gram flag sync");
    if (hbad & 2) return set_error("gram: a wait of the tensor-core pass ran out of time");
    // a value that is not finite: the whole product again in FP64
    if (hbad) return crossprod(A, A, n, true, upper_only, alpha, beta, out, ldo, s, scr);
    return 0;
}

int crossprod_auto(const MatView& A, const MatView& B, long long n, bool gram, bool upper_only, double alpha,
                   double beta, double* out, int ldo, cudaStream_t s, Scratch& scr) {
    const long long pairs = gram ? (long long)A.cols * (A.cols + 1) / 2 : (long long)A.cols * B.cols;
    const long long cols = gram ? A.cols : (long long)A.cols + B.cols;
    if (gram && pairs >= (long long)tuning(TUNE_SPLIT_GRAM) * cols && n >= 4096)
        return crossprod_split(A, n, upper_only, alpha, beta, out, ldo, s, scr);
    return crossprod(A, B, n, gram, upper_only, alpha, beta, out, ldo, s, scr);
}

int residual_scores(const double* X, int C, long long n, const double* beta, int k, const int* score_cols_dev,
                    int n_score, double* S, double* resid, double* rss_dev, cudaStream_t s, Scratch& scr) {
    int nb = (int)std::min<long long>((long long)num_sms() * 8, std::max(1LL, (n + RS_THREADS - 1) / RS_THREADS));
    double* partials = nullptr;
    FEGB_TRY(scr.alloc(&partials, (size_t)nb, "rss partials"));
    if (C >= 32)
        residual_scores_wide_kernel<<<nb, RS_THREADS, 0, s>>>(X, C, n, beta, k, score_cols_dev, n_score, S, resid,
                                                              partials);
    else
        residual_scores_kernel<<<nb, RS_THREADS, 0, s>>>(X, C, n, beta, k, score_cols_dev, n_score, S, resid,
                                                         partials);
    FEGB_LAUNCH_CHECK("residual/scores");
    sum_partials_kernel<<<1, RS_THREADS, 0, s>>>(partials, nb, rss_dev);
    FEGB_LAUNCH_CHECK("rss sum");
    return 0;
}

int dense_chol_solve_inv(int k, const double* Q, int ldq, const int* idx_dev, const double* b, double* beta_out,
                         double* Qinv, int* info_dev, double* work, cudaStream_t s) {
    if (k <= 0) return 0;
    static const cudaError_t attr =
        cudaFuncSetAttribute(chol_solve_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DN_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "cholesky attr");
    chol_solve_inv_kernel<<<1, DN_THREADS, dn_fits(k) ? dn_work_bytes(k) : 0, s>>>(k, Q, ldq, idx_dev, b, beta_out, Qinv, info_dev, work);
    FEGB_LAUNCH_CHECK("cholesky");
    return 0;
}

int dense_gemm(bool ta, bool tb, int m, int n, int k, double alpha, const double* A, int lda, const double* B, int ldb,
               double beta, double* C, int ldc, cudaStream_t s) {
    long long tot = (long long)m * n;
    if (tot <= 0) return 0;
    gemm_small_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C,
                                                                     ldc);
    FEGB_LAUNCH_CHECK("small gemm");
    return 0;
}

int dense_sandwich_acc(int k, const double* Qinv, const double* M, int ldm, const int* idx_dev, double w, double* acc,
                       double* work, cudaStream_t s) {
    if (k <= 0) return 0;
    double* Ms = work;
    double* T = work + (size_t)k * k;
    select_kernel<<<(k * k + 255) / 256, 256, 0, s>>>(k, M, ldm, idx_dev, Ms);
    FEGB_LAUNCH_CHECK("meat select");
    FEGB_TRY(dense_gemm(false, false, k, k, k, 1.0, Ms, k, Qinv, k, 0.0, T, k, s));
    FEGB_TRY(dense_gemm(false, false, k, k, k, w, Qinv, k, T, k, 1.0, acc, k, s));
    return 0;
}

int dense_finalize_cov(int k, double* acc, double scalar, int do_psd, double* se_out, int* psd_applied, double* work,
                       cudaStream_t s) {
    if (k <= 0) return 0;
    static const cudaError_t attr =
        cudaFuncSetAttribute(finalize_cov_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DN_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "covariance finalize attr");
    finalize_cov_kernel<<<1, DN_THREADS, dn_fits(k) ? dn_work_bytes(k) : 0, s>>>(k, acc, scalar, do_psd, se_out, psd_applied, work);
    FEGB_LAUNCH_CHECK("covariance finalize");
    return 0;
}

}  // namespace fegb

// ---------------------------------------------------------------------------
// Allocation-free cross product (fe_gpu_syrk_noalloc, include/fe_gpu_runtime.h).
//
// fe_gpu_syrk takes the per-block partial sums of its reduction from the
// stream-ordered memory pool. Some callers cannot let a library allocate
// device memory while they run: a host that owns every device buffer through
// its own allocator and budget, or code that must not touch the allocator
// at all in a latency-critical section. For them this variant keeps the
// partials in a fixed file-scope device array of
// NOALLOC_BLOCKS x NOALLOC_MAX_PAIRS doubles (152 x 528 x 8 B = 642 KB, held
// by every GPU that loads the library until the process exits), which bounds
// the input to at most NOALLOC_MAX_COLS = 32 columns.
//
// The device address of the array is looked up with cudaGetSymbolAddress by
// the first call made while a device is current, and cached with the identity
// of that device's CUDA context (cuCtxGetId). A later call in a new context
// (after cudaDeviceReset, or a primary context that was released and created
// again) finds a different identity and looks the address up again. Make the
// first call on each device, and the first after a reset, before capturing
// any stream. Every call shares the one array: calls whose kernels overlap on
// the GPU (other host threads, or other streams) race on it. Each launch
// overwrites every partial it later reads, so nothing has to be cleared
// between calls.
// ---------------------------------------------------------------------------
namespace fegb {

namespace {

constexpr int NOALLOC_BLOCKS = 152;
constexpr int NOALLOC_MAX_COLS = 32;
constexpr int NOALLOC_MAX_PAIRS = NOALLOC_MAX_COLS * (NOALLOC_MAX_COLS + 1) / 2;

__device__ __align__(256) double g_syrk_noalloc_partials[NOALLOC_BLOCKS * NOALLOC_MAX_PAIRS];

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_partials[NOALLOC_MAX_DEVICES] = {};
unsigned long long g_noalloc_ctx_id[NOALLOC_MAX_DEVICES] = {};

// Driver entry points for the current context's identity, fetched through the
// runtime so the library needs no link against libcuda.
typedef int (*ctx_get_current_fn)(void** ctx);
typedef int (*ctx_get_id_fn)(void* ctx, unsigned long long* id);

// Identity of the calling thread's current context; *have = false when no
// context is current or its identity cannot be read (a context destroyed by a
// reset), so that the caller runs the set-up again.
int current_context_id(unsigned long long* id, bool* have) {
    static ctx_get_current_fn get_current = nullptr;
    static ctx_get_id_fn get_id = nullptr;
    *have = false;
    if (!get_current || !get_id) {
        void* f1 = nullptr;
        void* f2 = nullptr;
        cudaDriverEntryPointQueryResult q1{}, q2{};
        FEGB_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1),
                  "cudaGetDriverEntryPointByVersion (cuCtxGetCurrent)");
        FEGB_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2),
                  "cudaGetDriverEntryPointByVersion (cuCtxGetId)");
        if (q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
            return set_error("fe_gpu_syrk_noalloc: the driver does not provide cuCtxGetCurrent/cuCtxGetId");
        get_current = reinterpret_cast<ctx_get_current_fn>(f1);
        get_id = reinterpret_cast<ctx_get_id_fn>(f2);
    }
    void* ctx = nullptr;
    if (get_current(&ctx) != 0 || !ctx) return 0;
    if (get_id(ctx, id) != 0) return 0;
    *have = true;
    return 0;
}

// Device address of the partials array in the current device's context
// (looked up on the first call per device and again whenever the context
// changed since).
int noalloc_partials(double** out) {
    int dev = 0;
    FEGB_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return set_error("fe_gpu_syrk_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    unsigned long long ctx_id = 0;
    bool have = false;
    FEGB_TRY(current_context_id(&ctx_id, &have));
    if (!have || !g_noalloc_partials[dev] || g_noalloc_ctx_id[dev] != ctx_id) {
        // set-up: the lookup also makes the device's primary context current
        void* p = nullptr;
        FEGB_CUDA(cudaGetSymbolAddress(&p, g_syrk_noalloc_partials), "cudaGetSymbolAddress (syrk scratch)");
        FEGB_TRY(current_context_id(&ctx_id, &have));
        if (!have) return set_error("fe_gpu_syrk_noalloc: no current CUDA context after set-up");
        g_noalloc_partials[dev] = static_cast<double*>(p);
        g_noalloc_ctx_id[dev] = ctx_id;
    }
    *out = g_noalloc_partials[dev];
    return 0;
}

}  // namespace

}  // namespace fegb

extern "C" int fe_gpu_syrk_noalloc(int n_rows, int n_cols, double alpha, const double* W, int ldW, double beta,
                                   double* Q) {
    using namespace fegb;
    if (n_cols == 0) return set_ok();
    if (n_cols < 0 || n_rows < 0) return set_error("fe_gpu_syrk_noalloc: negative dimension");
    if (n_cols > NOALLOC_MAX_COLS)
        return set_error("fe_gpu_syrk_noalloc: n_cols=%d exceeds the %d-column limit of its fixed scratch", n_cols,
                         NOALLOC_MAX_COLS);
    if (ldW < std::max(1, n_rows))
        return set_error("fe_gpu_syrk_noalloc: ldW=%d is below max(1, n_rows=%d)", ldW, n_rows);
    double* partials = nullptr;
    FEGB_TRY(noalloc_partials(&partials));
    const cudaStream_t s = 0;  // legacy default stream, as the rest of the kernel-level ABI
    const int npairs = n_cols * (n_cols + 1) / 2;
    int nb = 0;
    if (n_rows > 0) {
        long long blocks = std::min<long long>(((long long)n_rows + CP_TR - 1) / CP_TR, NOALLOC_BLOCKS);
        long long rpb = ((long long)n_rows + blocks - 1) / blocks;
        rpb = ((rpb + CP_TR - 1) / CP_TR) * CP_TR;
        nb = (int)(((long long)n_rows + rpb - 1) / rpb);
        CPParams p;
        p.A = W;
        p.ars = 1;
        p.acs = ldW;
        p.a = n_cols;
        p.B = W;
        p.brs = 1;
        p.bcs = ldW;
        p.b = n_cols;
        p.n = n_rows;
        p.gram = 1;
        p.p0 = 0;
        p.npairs = npairs;
        p.phases = npairs <= 128 ? CP_THREADS / npairs : 1;
        p.rows_per_block = rpb;
        p.partials = partials;
        const size_t smem = sizeof(double) * CP_TR * n_cols;
        if (npairs <= 128)
            crossprod_kernel<1><<<nb, CP_THREADS, smem, s>>>(p);
        else
            crossprod_kernel<4><<<nb, CP_THREADS, smem, s>>>(p);
        FEGB_LAUNCH_CHECK("syrk noalloc");
    }
    // nb = 0 (no rows) leaves Q = beta Q on the upper triangle
    crossprod_reduce_kernel<<<reduce_blocks(npairs), 256, 0, s>>>(partials, nb, npairs, 0, 1, 1, n_cols, alpha, beta, Q,
                                                                  n_cols);
    FEGB_LAUNCH_CHECK("syrk noalloc reduce");
    FEGB_CUDA(cudaStreamSynchronize(s), "syrk noalloc sync");
    return set_ok();
}
