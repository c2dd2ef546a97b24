// Gram products X'X of FP64 columns on the 5th-generation tensor cores.
//
// Every value is written as eight digits of eight bits relative to its column's
// scale (a power of two above the largest value so far: the 53 significant bits
// lie below 2^62 of a 64-bit integer, shifted down by the difference of the
// exponents), each digit a whole number in [-128, 127] held exactly in FP16. One
// tcgen05.mma (kind::f16, FP32 accumulation) over the digits of up to 16 columns
// as M and up to 16 as N forms all 64 digit products of each column pair; a
// product is at most 2^14, so the sums of 1,024 rows are whole numbers up to
// 2^24 and therefore exact in FP32. They are then read from tensor memory, put
// together in 64-bit integers and added in FP64. A value loses what lies 2^-58
// below its column's largest; the rest is FP64 rounding of the partial sums:
// 5e-17 to 3e-16 of the columns' norms where double-single products on the FP32
// pipe left 3e-15 to 2e-14. (Against the sum of the products' magnitudes it is as
// good up to values of 2^24 in the same 1,024 rows; a value of 1e9 beside others of 1
// that no other column shares leaves 3e-13 of an entry, double-single 3e-15.)
//
// One FP64 value (one row of one column) becomes 16 bytes of digits = one row
// of a core matrix of the canonical no-swizzle MN-major operand layout, and a
// thread's eight consecutive rows of its column are one core matrix (eight K
// rows by the eight digits). Cores lie 144 bytes apart (SBO), not 128, so that
// neighbouring threads' 16-byte stores fall on different banks. A and B read the
// same tile.
//
// What bounds it: the integer instructions that make the digits (about 18 of
// them a value on the half-rate ALU pipe; 63 % of it busy at 600k x 111), next to
// the MMA (N columns x 16 rows in N / 2 cycles) and the reads. Four blocks an SM,
// each with one tile and at most 128 columns of tensor memory, overlap each
// other's phases; a block loads its next values while its MMAs run. Seven-bit
// digits in BF16 sum 4,096 rows but cost 15 shifts and masks a value where a
// byte is one permute (2 pairs of digits an instruction). Before / after: the six
// Grams of a 150M-row fit (9 and 8 columns) 14.0 -> 8.1 ms, the four of a
// 1M x 111 one 8.2 -> 4.1 ms, of 38k x 29 rows 145 -> 100 us.
#include "common.cuh"
#include "linalg.cuh"
#include "umma.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>

namespace fegb {

namespace {

constexpr int GU_THREADS = 256;
constexpr int GU_V = 8;           // values a thread converts per tile: the 8 rows of a core matrix of one column
constexpr int GU_COLS = 16;       // columns of an operand block (8 digits each: M = 128)
constexpr int GU_CORE = 144;      // bytes from one column's core matrix to the next
constexpr int GU_ROWS = 1024;     // rows summed exactly: 2^24 / (128 x 128)
constexpr int GU_BLOCKS = 4 * 152 * 4;  // blocks aimed at: four rounds of four an SM
constexpr int GU_SHIFT = 9;       // the 53 significant bits lie below 2^62
constexpr int GU_ROOM = 3;        // bits between a column's largest value and its scale
constexpr int GU_EMIN = 64;       // the scale of a column that held only zeros (exponent field 0: they shift out)
constexpr int GU_SAMPLES = 8;     // tiles looked at for the first scales

struct GramUmma {
    const double* X;  // row-major, row stride rs
    long long rs;
    long long n;
    int C;
    int bs;            // columns of a block (<= GU_COLS)
    long long rpb;     // rows per block of the grid
    double* partials;  // row blocks x C (C + 1) / 2
    int* bad;          // |= 1: a value is not finite, |= 2: a wait ran out of time
};

// groups of 8 rows that GU_THREADS threads cover, one column each (even, so that
// a tile is a whole number of 16-row MMAs)
__host__ __device__ inline int gu_groups(int cols) {
    const int g = (GU_THREADS / cols) & ~1;
    return g < GU_ROWS / GU_V ? g : GU_ROWS / GU_V;
}

// the eight bytes u of an integer as FP16 digits u - 128: 1024 + u has the
// mantissa bits u, and 1152 is subtracted
__device__ __forceinline__ uint4 gu_digits(uint32_t lo, uint32_t hi) {
    const __half2 off = __floats2half2_rn(1152.0f, 1152.0f);
    uint32_t w[4] = {__byte_perm(lo, 0x64u, 0x4140u), __byte_perm(lo, 0x64u, 0x4342u), __byte_perm(hi, 0x64u, 0x4140u),
                     __byte_perm(hi, 0x64u, 0x4342u)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&w[j]), off);
        w[j] = *reinterpret_cast<const uint32_t*>(&d);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// digits of v relative to the scale E >= its exponent field, in every digit 128
// added (the bytes of the biased integer are the digits plus 128)
__device__ __forceinline__ uint4 gu_split(double v, int E) {
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    // the 53 significant bits, the first (implicit) one at bit 61
    const uint32_t mh = (__funnelshift_l(lo, hi, GU_SHIFT) & 0x1FFFFFFFu) | 0x20000000u;
    const uint32_t ml = lo << GU_SHIFT;
    const uint32_t down = (uint32_t)E - ((hi * 2u) >> 21);
    unsigned long long mag;  // zero from a shift of 64 up
    asm("{\n.reg .b64 t;\nmov.b64 t, {%1, %2};\nshr.u64 %0, t, %3;\n}\n" : "=l"(mag) : "r"(ml), "r"(mh), "r"(down));
    const unsigned long long sg = (unsigned long long)(long long)((int)hi >> 31);
    const unsigned long long biased = (mag ^ sg) + (0x8080808080808080ull - sg);
    return gu_digits((uint32_t)biased, (uint32_t)(biased >> 32));
}

// 1.5 x 2^52 + t for a whole number |t| < 2^51, without a conversion
__device__ __forceinline__ double gu_magic(long long t) {
    return __longlong_as_double(t + 0x4338000000000000ll);
}

__global__ void __launch_bounds__(GU_THREADS, 4) gram_umma_kernel(GramUmma a) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_max[2][32], s_late;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // blocks (bi, bj), bi <= bj, of columns
    int bj = 0;
    while ((bj + 1) * (bj + 2) / 2 <= (int)blockIdx.x) ++bj;
    const int bi = (int)blockIdx.x - bj * (bj + 1) / 2;
    const bool diag = bi == bj;
    const int a0 = bi * a.bs, b0 = bj * a.bs;
    const int ca = min(a.bs, a.C - a0), cb = min(a.bs, a.C - b0);
    const int cols = diag ? ca : ca + cb;
    const int groups = gu_groups(cols);
    const int rows_tile = GU_V * groups;
    const int g = tid / cols, c = tid - g * cols;
    const bool active = g < groups;
    const int gcol = c < ca ? a0 + c : b0 + (c - ca);
    const uint32_t lbo = (uint32_t)cols * GU_CORE;
    const int N = (8 * cb + 15) / 16 * 16;
    const int tcols = N <= 32 ? 32 : (N <= 64 ? 64 : 128);
    const long long r0 = (long long)blockIdx.y * a.rpb, r1 = min(a.n, r0 + a.rpb);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                     "r"(tcols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        s_late = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 32) s_max[0][tid] = s_max[1][tid] = 0;
    // the cores past the tile that an operand of 128 rows reads (results unused)
    for (int e = tid; e < GU_COLS * GU_CORE / 16; e += GU_THREADS)
        *reinterpret_cast<uint4*>(sm + (uint32_t)groups * lbo + e * 16) = make_uint4(0, 0, 0, 0);
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_base_s;
    const uint32_t sbase = smem_u32(sm);

    // lane l of every warp: the scale of column l
    int E = GU_EMIN;
    int rows_acc = 0;
    bool bad = false;
    // this lane's output: columns ai of a (a quarter of a warp's lanes each), aj of b
    const int quad = warp & 3, p = lane & 7;
    const int ai = 4 * quad + (lane >> 3), j0 = 8 * (warp >> 2), aj = j0 + p;
    double acc = 0.0;
    // digit sums in tensor memory (row 8 i + p, column 8 j + q) -> acc. A lane
    // reads row 8 ai + p, puts together the eight digits q of each of the eight
    // columns j0 .. j0 + 7 (whole numbers below 2^49 in two halves, made FP64 by
    // placing them in the mantissa), and the eight lanes of a column add them so
    // that lane p ends with column j0 + p. FP64 instructions are what this costs
    // (35 a lane); products on the diagonal block below it are left out.
    auto drain = [&]() {
        if (4 * quad < ca && j0 < cb && !(diag && j0 + 7 < 4 * quad)) {
            const double wl = __longlong_as_double((long long)(1023 + 8 * p) << 52);
            const double wh = __longlong_as_double((long long)(1023 + 8 * p + 32) << 52);
            const double ml = -6755399441055744.0 * wl, mh = -6755399441055744.0 * wh;
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = 0.0;
                if (j0 + j < cb) {
                    float t[8];
                    tmem_ld8(tmem + ((uint32_t)(quad * 32) << 16) + 8 * (j0 + j), t);
                    tmem_wait_ld();
                    long long lo = 0, hi = 0;
#pragma unroll
                    for (int q = 3; q >= 0; --q) {
                        lo = lo * 256 + __float2int_rn(t[q]);
                        hi = hi * 256 + __float2int_rn(t[q + 4]);
                    }
                    v[j] = __fma_rn(gu_magic(hi), wh, mh) + __fma_rn(gu_magic(lo), wl, ml);
                }
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                const bool up = (p & o) != 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (j >= o) break;
                    const double mine = up ? v[j + o] : v[j], other = up ? v[j] : v[j + o];
                    v[j] = mine + __shfl_xor_sync(0xffffffffu, other, o);
                }
            }
            const int Ei = __shfl_sync(0xffffffffu, E, min(ai, ca - 1));
            const int Ej = __shfl_sync(0xffffffffu, E, diag ? min(aj, cb - 1) : ca + min(aj, cb - 1));
            acc += ldexp(v[0], Ei + Ej - 2 * (1023 + 52 + GU_SHIFT));
        }
        fence_before_sync();
    };
    double x[GU_V] = {};
    // byte offsets inside a tile (below 2^32: see the launch)
    const uint32_t row_bytes = (uint32_t)(a.rs * 8), own = (uint32_t)g * GU_V * row_bytes + (uint32_t)gcol * 8;
    auto load = [&](long long t0) {
        const long long r = t0 + (long long)g * GU_V;
        const double* src = a.X + r * a.rs + gcol;
        if (t0 + rows_tile <= r1) {
            const char* base = reinterpret_cast<const char*>(a.X + t0 * a.rs);
            if (active) {
#pragma unroll
                for (int i = 0; i < GU_V; ++i)
                    x[i] = __ldg(reinterpret_cast<const double*>(base + (own + (uint32_t)i * row_bytes)));
            }
        } else {
#pragma unroll
            for (int i = 0; i < GU_V; ++i, src += a.rs) x[i] = (active && r + i < r1) ? __ldg(src) : 0.0;
        }
    };
    auto exponent = [&]() {  // the largest of x
        uint32_t e = 0;
#pragma unroll
        for (int i = 0; i < GU_V; ++i) e = max(e, (uint32_t)__double2hiint(x[i]) * 2u);
        return (int)(e >> 21);
    };
    // first scales from tiles spread over the block's rows: a rise later costs a drain
    const long long tiles = (r1 - r0 + rows_tile - 1) / rows_tile;
    if (tiles > 2 * GU_SAMPLES) {
        int e = 0;
        for (int k = 0; k < GU_SAMPLES; ++k) {
            load(r0 + tiles * k / GU_SAMPLES * rows_tile);
            e = max(e, exponent());
        }
        if (active && e > 0) atomicMax(&s_max[1][c], e);
        __syncthreads();
        const int m = lane < cols ? s_max[1][lane] : 0;
        if (m > 0) E = max(m, GU_EMIN) + GU_ROOM;
        __syncthreads();
        if (tid < 32) s_max[1][tid] = 0;
    }
    load(r0);
    int Ec = __shfl_sync(0xffffffffu, E, c);
    uint32_t issued = 0;
    bool failed = false;
    int slot = 0;
    for (long long t0 = r0; t0 < r1; t0 += rows_tile) {
        const int e = exponent();
        bool ask = active && (e > Ec || (e > 0 && Ec == GU_EMIN));
        if (ask) atomicMax(&s_max[slot][c], e);
        bad = bad || (active && e == 0x7FF);
        // the MMAs of the tile before are done with the tile
        if (tid == 0 && issued && !mbar_wait(&bar, (issued - 1) & 1u)) {
            s_late = 1;
            ask = true;
        }
        const bool any = __syncthreads_or(ask);
        fence_after_sync();
        if (any && s_late) {
            failed = true;
            break;
        }
        int m = 0;
        bool leave = rows_acc + rows_tile > GU_ROWS;
        if (any) {
            // a column whose scale rises: what is summed so far leaves first (a column
            // of zeros has nothing to leave)
            m = lane < cols ? s_max[slot][lane] : 0;
            leave = leave || __any_sync(0xffffffffu, m > 0 && E > GU_EMIN);
        }
        if (rows_acc > 0 && leave) {
            drain();
            rows_acc = 0;
        }
        if (any) {
            if (m > 0) E = max(m, GU_EMIN) + GU_ROOM;
            if (tid < 32) s_max[slot ^ 1][tid] = 0;
            slot ^= 1;
            Ec = __shfl_sync(0xffffffffu, E, c);
        }
        if (active) {
            // core (g, c): (g cols + c) x 144 bytes = tid x 144
            uint4* dst = reinterpret_cast<uint4*>(sm + (uint32_t)tid * GU_CORE);
#pragma unroll
            for (int i = 0; i < GU_V; ++i) dst[i] = gu_split(x[i], Ec);
        }
        if (t0 + rows_tile < r1) load(t0 + rows_tile);
        fence_async_smem();
        fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            fence_after_sync();
            const uint32_t id = umma_idesc_f16(128, N, 1, 1);
            const uint32_t bofs = diag ? 0u : (uint32_t)ca * GU_CORE;
            for (int s = 0; s < rows_tile / 16; ++s) {
                const uint32_t at = sbase + (uint32_t)s * 2 * lbo;
                umma_f16(tmem, umma_desc(at, lbo, GU_CORE), umma_desc(at + bofs, lbo, GU_CORE), id,
                         rows_acc > 0 || s > 0);
            }
            umma_commit(&bar);
        }
        ++issued;
        rows_acc += rows_tile;
    }
    bool ok = true;
    if (tid == 0 && issued) ok = mbar_wait(&bar, (issued - 1) & 1u);
    if (__syncthreads_or(!ok)) failed = true;
    fence_after_sync();
    if (!failed && rows_acc > 0) drain();
    if (failed && tid == 0) atomicOr(a.bad, 2);
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.bad, 1);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols));
    const long long np = (long long)a.C * (a.C + 1) / 2;
    const long long gi = a0 + ai, gj = b0 + aj;
    if (ai < ca && aj < cb && gi <= gj) a.partials[(long long)blockIdx.y * np + gj * (gj + 1) / 2 + gi] = acc;
}

}  // namespace

int launch_gram_umma(const double* X, long long rs, int C, long long n, Scratch& scr, double** partials, int* nb,
                     int* bad, cudaStream_t s) {
    static const cudaError_t attr = [] {
        cudaError_t e = cudaFuncSetAttribute(gram_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(gram_umma_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared);
        return e;
    }();
    if (attr != cudaSuccess) return set_cuda_error(attr, "gram (tcgen05) attr");
    GramUmma a{};
    a.X = X;
    a.rs = rs;
    a.n = n;
    a.C = C;
    const int nblk = (C + GU_COLS - 1) / GU_COLS;
    a.bs = (C + nblk - 1) / nblk;
    const int pairs = nblk * (nblk + 1) / 2;
    const int widest = nblk > 1 ? 2 * a.bs : a.bs;
    // a core per thread, and the cores past the tile that an operand of 128 rows reads
    const size_t smem = (size_t)(GU_THREADS + GU_COLS) * GU_CORE;
    const int tile = GU_V * gu_groups(widest);
    const long long want = std::max<long long>(1, std::min<long long>((n + tile - 1) / tile, GU_BLOCKS / pairs));
    a.rpb = std::min<long long>(((n + want - 1) / want + tile - 1) / tile * tile, 65536 / tile * tile);
    const long long rows = (n + a.rpb - 1) / a.rpb;
    FEGB_TRY(scr.alloc(partials, (size_t)rows * ((size_t)C * (C + 1) / 2), "gram partials"));
    a.partials = *partials;
    a.bad = bad;
    gram_umma_kernel<<<dim3((unsigned)pairs, (unsigned)rows), GU_THREADS, smem, s>>>(a);
    FEGB_LAUNCH_CHECK("gram (tcgen05)");
    *nb = (int)rows;
    return 0;
}

}  // namespace fegb
