// Alternating projections on group tables (see ap_group.cuh).
#include "ap_group.cuh"
#include "umma.cuh"

#include <algorithm>
#include <cfloat>

namespace fegb {

namespace {

constexpr int AP_THREADS = 256;

// Fixed-point sums of FP64 table values. GB300 adds FP64 at 1/64 of the FP32
// rate, and converts to and from it no faster; 64-bit integers run at about 1/3.
// So counts x values are summed as integers: a value v of a column with
// max |v| < 2^(e+1) becomes round(v 2^k), k = 51 - e, 53 bits with the sign (one
// rounding of at most 2^(e-52), an ulp of the column's largest value; a small value
// beside it keeps fewer bits than FP64 would, which the bound on the tables' values
// allows for, see level_fits), in two digits hi 2^26 + lo. Products with counts add
// up in one 64-bit integer per digit: all counts of a dimension add up to n < 2^31
// rows, so neither overflows whatever the counts, and the sums are exact in any
// order.
constexpr int FIX_LO = 26;

__device__ __forceinline__ int fix_exponent(unsigned long long amax_bits) {
    const int e = (int)((amax_bits >> 52) & 0x7ff);
    return 51 - (e - 1023);  // k
}

__device__ __forceinline__ long long to_fixed(double v, int k) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    if (e == 0) return 0;
    const unsigned long long m = ((unsigned long long)b & ((1ULL << 52) - 1ULL)) | (1ULL << 52);
    const int sh = max(1, 1075 - k - e);
    const unsigned long long r = sh < 54 ? (m + (1ULL << (sh - 1))) >> sh : 0ULL;
    return b < 0 ? -(long long)r : (long long)r;
}

struct FixDigits {
    int hi;
    unsigned lo;
};
__device__ __forceinline__ FixDigits fix_digits(long long f) {
    FixDigits d;
    d.hi = (int)(f >> FIX_LO);
    d.lo = (unsigned)f & ((1u << FIX_LO) - 1u);
    return d;
}
struct FixSum {
    long long hi, lo;
};
__device__ __forceinline__ void fix_add(FixSum& s, unsigned n, const FixDigits& d) {
    s.hi += (long long)(int)n * d.hi;  // counts are below 2^31
    s.lo = (long long)((unsigned long long)s.lo + (unsigned long long)n * d.lo);
}

// Relaxation of the projection in `slot`, from the two before it.
__device__ __forceinline__ double ap_relax(const ApSlot* slots, int slot) {
    const ApSlot a = slots[(slot + AP_SLOTS - 1) % AP_SLOTS];
    const double pc = bits_dbl(slots[(slot + AP_SLOTS - 2) % AP_SLOTS].change);
    const double cd = bits_dbl(a.change);
    double r = a.relax;
    if (cd > pc * 1.05)
        r = fmax(0.4, r * 0.5);
    else if (cd < pc * 0.8)
        r = fmin(2.0, r * 1.10);
    return r;
}

__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) {
    return a > b ? a : b;
}
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL;
}
// a 2^-k, rounded to nearest, on the integer pipe (the conversion instruction
// runs at the FP64 rate)
__device__ __forceinline__ double from_fixed(long long a, int k) {
    if (a == 0) return 0.0;
    const unsigned long long u = a < 0 ? 0ULL - (unsigned long long)a : (unsigned long long)a;
    const int lz = __clzll((long long)u);
    const unsigned long long m = u << lz;  // leading bit at 63
    const int e = 63 - lz - k + 1022;      // the leading 1 of the fraction adds one to the exponent
    if (e <= 0) return 0.0;
    const unsigned long long f = (m >> 11) + ((m >> 10) & 1ULL);
    return __longlong_as_double((long long)(((unsigned long long)e << 52) + f) | (a & (long long)(1ULL << 63)));
}

// value of a fixed-point sum; a column with an infinity or NaN in its table has
// no fixed-point form, and its sums are NaN
__device__ __forceinline__ double fix_value(const FixSum& s, unsigned long long amax_bits) {
    if (amax_bits >= (0x7ffULL << 52)) return __longlong_as_double(0x7ff8LL << 48);
    const int k = fix_exponent(amax_bits);
    const long long hi = s.hi + (s.lo >> FIX_LO), lo = s.lo & ((1LL << FIX_LO) - 1);
    if (hi < (1LL << (62 - FIX_LO)) && hi > -(1LL << (62 - FIX_LO))) return from_fixed(hi * (1LL << FIX_LO) + lo, k);
    return from_fixed(hi, k - FIX_LO) + from_fixed(lo, k);
}

// float -> T; to double on the integer pipe, for the counts that weights are
// (normal numbers)
__device__ __forceinline__ void count_to(float w, float& o) { o = w; }
__device__ __forceinline__ void count_to(float w, double& o) {
    const unsigned long long b = __float_as_uint(w);
    o = __longlong_as_double((long long)(((b >> 23) + 896ULL) << 52 | (b & 0x7fffffULL) << 29));
}

// |v| for the convergence maximum, which passes over NaN as the row sweeps' does
__device__ __forceinline__ unsigned long long update_bits(double v) {
    const unsigned long long b = abs_bits(v);
    return b > (0x7ffULL << 52) ? 0ULL : b;
}

// One projection of element idx = (g, c): the new table value; mixed -> *upd.
// With t.means set, the residual's new mean instead.
template <typename T>
__device__ __forceinline__ double ap_update(const ApTables<T>& t, long long g, int c, double base, double relax,
                                            double* upd) {
    const long long idx = g * t.C + c;
    T* slot = t.tab + g * t.ld + c;
    if (t.means) {
        const double m = t.inv[g] != 0.0 ? base - (double)*slot : 0.0;
        t.means[idx] = m;
        *upd = m;
        return 0.0;
    }
    const double a = sizeof(T) == 8 ? (double)*slot : t.alpha64[idx];
    const double mean = base - a;
    const double pv = t.prev[idx];
    const double mixed = pv + relax * (mean - pv);
    t.prev[idx] = mixed;
    const double an = a + mixed;
    *slot = (T)an;
    if (sizeof(T) == 4) t.alpha64[idx] = an;
    *upd = mixed;
    return an;
}

// Block maxima of a kernel whose thread handles column c of its rows: the
// largest update into slot.change, the largest table value per column into amax.
__device__ __forceinline__ void ap_block_max(unsigned long long upd, unsigned long long av, bool active, int C,
                                             int rps, unsigned long long* red, ApSlot* slot,
                                             unsigned long long* amax) {
    __syncthreads();
    red[threadIdx.x] = active ? av : 0ULL;
    __syncthreads();
    if ((int)threadIdx.x < C) {
        unsigned long long m = 0;
        for (int j = 0; j < rps; ++j) m = umax64(m, red[j * C + threadIdx.x]);
        if (m > amax[threadIdx.x]) atomicMax(amax + threadIdx.x, m);
    }
    __syncthreads();
    red[threadIdx.x] = active ? upd : 0ULL;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long m = 0;
        for (int j = threadIdx.x; j < AP_THREADS; j += 32) m = umax64(m, red[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = umax64(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0 && m) atomicMax(&slot->change, m);
    }
}

// The slots of a launch: this projection's relaxation recorded, the next
// projection's change cleared (it was last read two projections ago).
__device__ __forceinline__ void ap_open_slot(ApSlot* slots, int slot, double relax) {
    slots[slot].relax = relax;
    slots[(slot + 1) % AP_SLOTS].change = 0ULL;
}

// The relaxation for a whole block, by one thread (the rule is eight FP64
// instructions, 128 cycles of an SM's FP64 pipe a warp), recorded by the first.
__device__ __forceinline__ double ap_block_relax(ApSlot* slots, int slot) {
    __shared__ double s_relax;
    if (threadIdx.x == 0) {
        const double r = ap_relax(slots, slot);
        s_relax = r;
        if (blockIdx.x == 0) ap_open_slot(slots, slot, r);
    }
    __syncthreads();
    return s_relax;
}

// Sums of the FP32 form: a few products in FP32, then into a pair of floats that
// keeps what an addition rounds off (six FP32 operations; an FP64 addition costs 64),
// as the row sweeps add FP32 sums of a few rows in FP64. Single floats over a lane's
// whole share would save 2 % of a mixed fit of 1.15M rows (20.2 -> 19.9 ms).
struct FloatSum {
    float hi, lo;
};
__device__ __forceinline__ void float_add(FloatSum& s, float v) {
    const float t = __fadd_rn(s.hi, v);
    const float b = __fsub_rn(t, s.hi);
    s.lo += __fadd_rn(__fsub_rn(s.hi, __fsub_rn(t, b)), __fsub_rn(v, b));
    s.hi = t;
}
// (an infinity has no remainder to speak of)
__device__ __forceinline__ double float_value(const FloatSum& s) {
    return (double)s.hi + (double)(fabsf(s.hi) <= FLT_MAX ? s.lo : 0.f);
}

// a += sum over t of N[g][t] * tab[t][c], small source, FP32 products
template <typename CT>
__device__ __forceinline__ void dense_dot(const CT* __restrict__ N, int Gs, const float* __restrict__ tab, int C, int c,
                                          FloatSum& a) {
    for (int t0 = 0; t0 < Gs; t0 += AP_PART) {
        const int t1 = min(t0 + AP_PART, Gs);
        float f = 0.f;
        int t = t0;
        for (; t + 4 <= t1; t += 4) {
            f = fmaf((float)N[t], tab[t * C + c], f);
            f = fmaf((float)N[t + 1], tab[(t + 1) * C + c], f);
            f = fmaf((float)N[t + 2], tab[(t + 2) * C + c], f);
            f = fmaf((float)N[t + 3], tab[(t + 3) * C + c], f);
        }
        for (; t < t1; ++t) f = fmaf((float)N[t], tab[t * C + c], f);
        float_add(a, f);
    }
}
// piece w (16 counts) of a row: the loads, and the counts in order
template <typename CT>
struct Piece {
    uint4 x[AP_PART * sizeof(CT) / 16];
    __device__ __forceinline__ void load(const CT* row, int w) {
        constexpr int V = AP_PART * sizeof(CT) / 16;
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = reinterpret_cast<const uint4*>(row)[w * V + i];
    }
    __device__ __forceinline__ unsigned operator[](int i) const {
        constexpr int PER = 16 / sizeof(CT), SUB = 4 / sizeof(CT);  // counts per vector, per word
        const uint4 v = x[i / PER];
        const int k = i % PER / SUB;
        const unsigned q = k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
        return sizeof(CT) == 4 ? q : (q >> (8 * (i % SUB))) & 255u;
    }
};

// the same in fixed point; tab is zero past Gs, up to a multiple of four rows
template <typename CT>
__device__ __forceinline__ void dense_dot_fixed(const void* N, long long g, int Gs, const FixDigits* __restrict__ tab,
                                                int C, int c, FixSum& a) {
    const CT* row = static_cast<const CT*>(N) + g * ap_count_pitch(Gs);
    for (int t0 = 0; t0 < Gs; t0 += AP_PART) {
        Piece<CT> n;
        n.load(row, t0 / AP_PART);
#pragma unroll
        for (int i = 0; i < AP_PART; i += 4) {
            if (t0 + i >= Gs) break;
            const FixDigits* __restrict__ q = tab + (t0 + i) * C + c;
            fix_add(a, n[i], q[0]);
            fix_add(a, n[i + 1], q[C]);
            fix_add(a, n[i + 2], q[2 * C]);
            fix_add(a, n[i + 3], q[3 * C]);
        }
    }
}

__host__ __device__ constexpr int four_rows(int Gs) { return (Gs + 3) & ~3; }

// One visit: thread (r, c) takes column c of the block's groups r, r + rps, ...
// The small sources' tables sit in shared memory, in the FP64 form as
// fixed-point digits of one scale per column, so that a group's sum over all of
// them is one pair of integers. What is left on the FP64 pipe, which bounds the
// kernel, is one FMA per swept position and the update (100k groups, 12 columns,
// 20 small groups: 37 us with FP64 sums, 19 us).
template <typename T>
__global__ void __launch_bounds__(AP_THREADS) ap_visit_kernel(ApVisit<T> p) {
    if (p.ctl->stop) return;
    extern __shared__ __align__(16) unsigned char ap_smem[];
    constexpr bool FIX = sizeof(T) == 8;
    unsigned long long* red = reinterpret_cast<unsigned long long*>(ap_smem);  // AP_THREADS
    unsigned long long* cmax = red + AP_THREADS;                               // C, to 32
    unsigned char* tabs = reinterpret_cast<unsigned char*>(cmax + 32);
    const ApTables<T>& t = p.t;
    const int C = t.C;
    const int rps = AP_THREADS / C;
    const int rr = (int)threadIdx.x / C;
    const int c = (int)threadIdx.x - rr * C;
    const bool active = rr < rps;
    const bool small = p.n_dense > 0 && !p.small_known;
    // small tables: entry (t, c) at dst[t * C + c], a multiple of four rows (zero past Gs)
    if (small) {
        if (FIX) {
            for (int i = threadIdx.x; i < C; i += AP_THREADS) {
                unsigned long long m = 0;
                for (int e = 0; e < p.n_dense; ++e) m = umax64(m, p.dense[e].amax[i]);
                cmax[i] = m;
            }
            __syncthreads();
        }
        T* dst = reinterpret_cast<T*>(tabs);
        for (int e = 0; e < p.n_dense; ++e) {
            const ApDense<T>& D = p.dense[e];
            for (int i = threadIdx.x; i < four_rows(D.Gs) * C; i += AP_THREADS) {
                const int tt = i / C, cc = i - tt * C;
                const T v = tt < D.Gs ? D.tab[tt * t.ld + cc] : T(0);
                if (FIX)
                    reinterpret_cast<FixDigits*>(dst)[i] = fix_digits(to_fixed((double)v, fix_exponent(cmax[cc])));
                else
                    dst[i] = v;
            }
            dst += four_rows(D.Gs) * C;
        }
    }
    const double relax = ap_block_relax(t.slots, p.slot);
    unsigned long long upd = 0, av = 0;
    if (active)
        for (long long g = (long long)blockIdx.x * rps + rr; g < t.G; g += (long long)gridDim.x * rps) {
            const long long idx = g * C + c;
            T acc = T(0);  // the swept sources' coupling sum (of a short group where this launch adds it up)
            if (p.sums) {
                acc = t.inv[g] != 0.0 ? -p.sums[idx] : T(0);  // sums of an empty group are not written
            } else if (p.off) {
                const int j0 = p.off[g], j1 = p.off[g + 1];
                const int32_t* __restrict__ sg0 = p.src_gid[0];
                const T* __restrict__ st0 = p.src_tab[0];
                for (int j = j0; j < j1; j += 2) {
                    const bool two = j + 1 < j1;
                    T v0 = st0[(long long)sg0[j] * t.ld + c];
                    T v1 = two ? st0[(long long)sg0[j + 1] * t.ld + c] : T(0);
                    for (int e = 1; e < p.n_src; ++e) {
                        const int32_t* __restrict__ sg = p.src_gid[e];
                        const T* __restrict__ st = p.src_tab[e];
                        v0 += st[(long long)sg[j] * t.ld + c];
                        if (two) v1 += st[(long long)sg[j + 1] * t.ld + c];
                    }
                    T w0 = T(1), w1 = T(1);
                    if (p.weight) {
                        count_to(p.weight[j], w0);
                        if (two) count_to(p.weight[j + 1], w1);
                    }
                    acc = fma(w0, v0, acc);
                    if (two) acc = fma(w1, v1, acc);
                }
            }
            double cpl;
            if constexpr (FIX) {
                cpl = acc;
                if (p.n_dense > 0) {
                    double sm;
                    if (p.small_known) {
                        sm = p.small_sums[idx];
                    } else {
                        FixSum f{0, 0};
                        const FixDigits* st = reinterpret_cast<const FixDigits*>(tabs);
                        for (int e = 0; e < p.n_dense; ++e) {
                            const ApDense<T>& D = p.dense[e];
                            if (D.wide)
                                dense_dot_fixed<uint32_t>(D.N, g, D.Gs, st, C, c, f);
                            else
                                dense_dot_fixed<uint8_t>(D.N, g, D.Gs, st, C, c, f);
                            st += four_rows(D.Gs) * C;
                        }
                        sm = fix_value(f, cmax[c]);
                        if (p.small_sums) p.small_sums[idx] = sm;
                    }
                    cpl = (p.sums || p.off) ? cpl + sm : sm;
                }
            } else {
                // what this visit adds up itself becomes FP64 once
                FloatSum facc{acc, 0.f};
                if (small) {
                    FloatSum f{0.f, 0.f};
                    const float* st = reinterpret_cast<const float*>(tabs);
                    for (int e = 0; e < p.n_dense; ++e) {
                        const ApDense<T>& D = p.dense[e];
                        const long long at = g * ap_count_pitch(D.Gs);
                        if (D.wide)
                            dense_dot(static_cast<const uint32_t*>(D.N) + at, D.Gs, st, C, c, f);
                        else
                            dense_dot(static_cast<const uint8_t*>(D.N) + at, D.Gs, st, C, c, f);
                        st += four_rows(D.Gs) * C;
                    }
                    if (p.small_sums) p.small_sums[idx] = float_value(f);
                    float_add(facc, f.hi);
                    facc.lo += f.lo;
                }
                cpl = float_value(facc);
                if (p.n_dense > 0 && !small) cpl += p.small_sums[idx];
            }
            const double base = fma(-cpl, t.inv[g], t.mu[idx]);
            if (!t.means) t.base[idx] = base;
            double u;
            const double an = ap_update(t, g, c, base, relax, &u);
            upd = umax64(upd, update_bits(u));
            av = umax64(av, abs_bits(an));
        }
    ap_block_max(upd, av, active, C, rps, red, t.slots + p.slot, t.amax);
}

template <typename T>
__global__ void __launch_bounds__(AP_THREADS) ap_repeat_kernel(ApTables<T> t, int slot, const ApCtl* ctl) {
    if (ctl->stop) return;
    __shared__ unsigned long long red[AP_THREADS];
    const int C = t.C;
    const int rps = AP_THREADS / C;
    const int rr = (int)threadIdx.x / C;
    const int c = (int)threadIdx.x - rr * C;
    const bool active = rr < rps;
    const double relax = ap_block_relax(t.slots, slot);
    unsigned long long upd = 0, av = 0;
    if (active)
        for (long long g = (long long)blockIdx.x * rps + rr; g < t.G; g += (long long)gridDim.x * rps) {
            double u;
            const double an = ap_update(t, g, c, t.base[g * C + c], relax, &u);
            upd = umax64(upd, update_bits(u));
            av = umax64(av, abs_bits(an));
        }
    ap_block_max(upd, av, active, C, rps, red, t.slots + slot, t.amax);
}

// Blocks per source of a small dimension's visit: enough that a lane has some
// AP_DEPTH groups, and no more than fit at once. The FP32 form's partials are
// folded by one block, hence their lower limit.
constexpr int AP_DEPTH = 4;
constexpr int AP_PART_BLOCKS = 152;
constexpr int AP_FIX_BLOCKS = 304;       // two an SM; one (half of them) where the sums of 24 groups fill the registers

// A block takes all groups of a small dimension of up to AP_WHOLE groups (what the
// registers hold), else one part of AP_PART of them.
constexpr int AP_WHOLE = 24;
constexpr int AP_PARTS = DENSE_SMALL_MAX_G / AP_PART;

struct ApSmallGrid {
    int first[AP_PARTS * SWEEP_MAXP + 1];  // first block of each (source, part of the small dimension)
    int parts;                            // parts of the small dimension
};

// sums over a warp's slots (lane = slot * C + c): valid in the lanes of slot 0
template <typename V>
__device__ __forceinline__ V warp_slot_sum(V v, int slot, int slots, int C, int top) {
    for (int o = top; o > 0; o >>= 1) {
        const V w = __shfl_down_sync(0xffffffffu, v, o * C);
        if (slot + o < slots) v += w;
    }
    return v;
}

// acc[t] += N[g][t] * tab[g][c] over this lane's groups, t from piece w of the rows
// on; the next group's loads are in flight while one is added (8 to 16 warps an
// SM hide little by themselves). WRITTEN: the table was written by this launch
// (read past L1).
__device__ __forceinline__ void walk_add(FixSum& s, unsigned n, const FixDigits& a) { fix_add(s, n, a); }
struct WalkF32 {
    float part;  // of up to WALK_FOLD groups
    FloatSum sum;
};
constexpr int WALK_FOLD = 8;
__device__ __forceinline__ void walk_add(WalkF32& s, unsigned n, float a) { s.part = fmaf((float)n, a, s.part); }
__device__ __forceinline__ void walk_fold(FixSum&) {}
__device__ __forceinline__ void walk_fold(WalkF32& s) {
    float_add(s.sum, s.part);
    s.part = 0.f;
}
__device__ __forceinline__ FixDigits walk_value(double v, int k, const FixSum*) { return fix_digits(to_fixed(v, k)); }
__device__ __forceinline__ float walk_value(float v, int, const WalkF32*) { return v; }

template <typename CT, int GT, bool WRITTEN = false, typename T, typename A>
__device__ __forceinline__ void small_walk(const CT* __restrict__ N, int pitch, int w, const T* tab, int ld, int c, int k,
                                           long long g, long long Ge, long long gstep, A (&acc)[GT]) {
    constexpr int NP = (GT + AP_PART - 1) / AP_PART;
    if (g >= Ge) return;
    Piece<CT> next[NP];
    T next_v = WRITTEN ? __ldcg(tab + g * ld + c) : tab[g * ld + c];
#pragma unroll
    for (int q = 0; q < NP; ++q) next[q].load(N + g * pitch, w + q);
    unsigned step = 0;
#pragma unroll 1
    while (true) {
        const auto a = walk_value(next_v, k, static_cast<const A*>(nullptr));
        Piece<CT> n[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) n[q] = next[q];
        g += gstep;
        const bool more = g < Ge;
        if (more) {
            next_v = WRITTEN ? __ldcg(tab + g * ld + c) : tab[g * ld + c];
#pragma unroll
            for (int q = 0; q < NP; ++q) next[q].load(N + g * pitch, w + q);
        }
#pragma unroll
        for (int i = 0; i < GT; ++i) walk_add(acc[i], n[i / AP_PART][i % AP_PART], a);
        if (!more || ++step % WALK_FOLD == 0) {
#pragma unroll
            for (int i = 0; i < GT; ++i) walk_fold(acc[i]);
        }
        if (!more) break;
    }
}
template <int GT, typename T, typename A>
__device__ __forceinline__ void small_walk_any(const ApDense<T>& D, int w, int ld, int c, int k, long long g,
                                               long long gstep, A (&acc)[GT]) {
    const int pitch = ap_count_pitch(D.Gs);
    if (D.wide)
        small_walk<uint32_t, GT>(static_cast<const uint32_t*>(D.N), pitch, w, D.tab, ld, c, k, g, D.Ge, gstep, acc);
    else
        small_walk<uint8_t, GT>(static_cast<const uint8_t*>(D.N), pitch, w, D.tab, ld, c, k, g, D.Ge, gstep, acc);
}

// Small dimension: sum_g N[g][t] tab[g][c] of one source for up to GT of its
// groups t and all c. A warp holds 32 / C slots of C lanes; a lane walks over
// groups g (neighbouring slots on neighbouring groups: table rows and count rows
// are read as contiguous runs, without shared memory) and keeps the sums of its
// column for its t in registers: two integer multiply-adds and the byte's
// extraction per count, or one FMA in the FP32 form. Integer sums are folded
// over the block and added to 64-bit global accumulators (exact, so the order is
// free); FP32 sums leave one FP64 partial per block, folded in block order.
// The last block to finish turns the sums into the projections.
// 100k x 20 and 12k x 20 counts, 12 columns: 81 us with FP64 sums of both
// operands in shared memory, 41 us in this form; 940k x 13, 4 columns: 75 -> 26.
template <typename T, int GT>
__global__ void __launch_bounds__(AP_THREADS, sizeof(T) == 8 && GT > AP_PART ? 1 : 2) ap_small_kernel(ApSmall<T> p, ApSmallGrid gr) {
    if (p.ctl->stop) return;
    extern __shared__ __align__(16) unsigned char ap_smem[];
    __shared__ bool s_last;
    constexpr bool FIX = sizeof(T) == 8;
    constexpr int WARPS = AP_THREADS / 32;
    const ApTables<T>& t = p.t;
    const int C = t.C, Gs = t.G;
    const int P = Gs * C;
    int part = 0;
    while (part + 1 < p.n_src * gr.parts && (int)blockIdx.x >= gr.first[part + 1]) ++part;
    const int src = part / gr.parts;
    const int t0 = (part - src * gr.parts) * AP_PART;
    const int nt = gr.parts > 1 ? min(Gs - t0, AP_PART) : Gs;
    const ApDense<T>& D = p.src[src];
    const int nb = gr.first[part + 1] - gr.first[part], b = (int)blockIdx.x - gr.first[part];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slots = 32 / C;
    const int slot = lane / C, c = lane - slot * C;
    int top = 1;
    while (top < slots) top <<= 1;
    top >>= 1;
    const long long gstep = (long long)nb * WARPS * slots;
    const long long g0 = slot < slots ? ((long long)b * WARPS + warp) * slots + slot : D.Ge;
    const int PB = nt * C;  // sums of this block
    if constexpr (FIX) {
        FixSum acc[GT];
#pragma unroll
        for (int i = 0; i < GT; ++i) acc[i] = FixSum{0, 0};
        const int k = fix_exponent(D.amax[c]);
        small_walk_any<GT>(D, t0 / AP_PART, t.ld, c, k, g0, gstep, acc);
        long long* red = reinterpret_cast<long long*>(ap_smem);  // WARPS x PB x 2
#pragma unroll
        for (int i = 0; i < GT; ++i) {
            if (i >= nt) break;
            const long long lo = warp_slot_sum(acc[i].lo, slot, slots, C, top);
            const long long hi = warp_slot_sum(acc[i].hi, slot, slots, C, top);
            if (lane < C) {
                red[2 * (warp * PB + i * C + lane)] = lo;
                red[2 * (warp * PB + i * C + lane) + 1] = hi;
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 2 * PB; i += AP_THREADS) {
            long long v = 0;
            for (int w = 0; w < WARPS; ++w) v += red[2 * w * PB + i];
            if (v) atomicAdd(p.limbs + 2 * ((size_t)src * P + t0 * C) + i, (unsigned long long)v);
        }
    } else {
        WalkF32 acc[GT];
#pragma unroll
        for (int i = 0; i < GT; ++i) acc[i] = WalkF32{0.f, {0.f, 0.f}};
        small_walk_any<GT>(D, t0 / AP_PART, t.ld, c, 0, g0, gstep, acc);
        float* red = reinterpret_cast<float*>(ap_smem);  // WARPS x PB
#pragma unroll
        for (int i = 0; i < GT; ++i) {
            if (i >= nt) break;
            const float v = warp_slot_sum(acc[i].sum.hi + acc[i].sum.lo, slot, slots, C, top);
            if (lane < C) red[warp * PB + i * C + lane] = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < PB; i += AP_THREADS) {
            double v = 0.0;
            for (int w = 0; w < WARPS; ++w) v += (double)red[w * PB + i];
            p.partials[((size_t)src * AP_PART_BLOCKS + b) * P + t0 * C + i] = v;
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(p.counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // ---- the last block: sums of all sources, then the projections ----
    double* tot = reinterpret_cast<double*>(ap_smem);            // P
    double* fold = tot + P;                                      // AP_THREADS
    unsigned long long* cmax = reinterpret_cast<unsigned long long*>(fold + AP_THREADS);  // C
    unsigned long long* wmax = cmax + C;                                                  // 8
    const int Pr = min(AP_THREADS, (P + 31) & ~31);
    for (int i = threadIdx.x; i < P; i += AP_THREADS) {
        double v = 0.0;
        for (int e = 0; e < p.n_kept; ++e) v += p.kept[e][i];
        tot[i] = v;
    }
    for (int i = threadIdx.x; i < C; i += AP_THREADS) cmax[i] = 0ULL;
    __syncthreads();
    for (int e = 0; e < p.n_src; ++e) {
        if constexpr (FIX) {
            for (int i = threadIdx.x; i < P; i += AP_THREADS) {
                unsigned long long* l = p.limbs + 2 * ((size_t)e * P + i);
                const FixSum f{(long long)__ldcg(l + 1), (long long)__ldcg(l)};
                l[0] = 0ULL;
                l[1] = 0ULL;
                const double v = fix_value(f, p.src[e].amax[i % C]);
                p.src_sums[e][i] = v;
                tot[i] += v;
            }
            __syncthreads();
            continue;
        }
        const int nparts = gr.first[e * gr.parts + 1] - gr.first[e * gr.parts];  // of every part
        const double* part = p.partials + (size_t)e * AP_PART_BLOCKS * P;
        for (int i0 = 0; i0 < P; i0 += Pr) {  // Pr pairs at a time, AP_THREADS / Pr slices of the blocks
            const int ns = AP_THREADS / Pr;
            const int sl = (int)threadIdx.x / Pr, i = i0 + (int)threadIdx.x - sl * Pr;
            double v = 0.0;
            if (sl < ns && i < P) {
#pragma unroll 8
                for (int k = sl; k < nparts; k += ns) v += __ldcg(part + (size_t)k * P + i);
            }
            fold[threadIdx.x] = v;
            __syncthreads();
            if (sl == 0 && i < P) {
                double w = 0.0;
                for (int k = 0; k < ns; ++k) w += fold[k * Pr + threadIdx.x];
                p.src_sums[e][i] = w;
                tot[i] += w;
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) *p.counter = 0u;
    for (int j = 0; j < p.projections; ++j) {
        const int slot = (p.slot + j) % AP_SLOTS;
        const double relax = ap_relax(t.slots, slot);
        unsigned long long upd = 0;
        for (int i = threadIdx.x; i < P; i += AP_THREADS) {
            const int g = i / C, c = i - g * C;
            double base;
            if (j == 0) {
                base = fma(-tot[i], t.inv[g], t.mu[i]);
                if (!t.means) t.base[i] = base;
            } else {
                base = t.base[i];
            }
            double u;
            const double an = ap_update(t, g, c, base, relax, &u);
            upd = umax64(upd, update_bits(u));
            atomicMax(cmax + c, abs_bits(an));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) upd = umax64(upd, __shfl_xor_sync(0xffffffffu, upd, o));
        __syncthreads();
        if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = upd;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long m = 0;
            for (int w = 0; w < AP_THREADS / 32; ++w) m = umax64(m, wmax[w]);
            ap_open_slot(t.slots, slot, relax);
            t.slots[slot].change = m;
            __threadfence_block();
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < C; i += AP_THREADS)
        if (cmax[i] > t.amax[i]) t.amax[i] = cmax[i];
}


// ------------------------ one large dimension, small others ------------------------

// Barrier of all blocks of a cooperative launch, the n-th one. Bounded: after
// p.wait_ns of waiting the error word is set and every block leaves.
__device__ __forceinline__ bool star_barrier(const ApStar& p, unsigned long long n, int* s_bad) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned long long target = n * gridDim.x;
        atomicAdd(p.arrived, 1ULL);
        volatile unsigned long long* a = p.arrived;
        volatile int* e = p.error;
        int bad = 0;
        unsigned long long t0 = 0;  // from the 64th poll on (a limit of zero: the first)
        for (unsigned spin = 0; *a < target; ++spin) {
            if (spin < 64 && p.wait_ns) continue;
            if (*e) {
                bad = 1;
                break;
            }
            const unsigned long long now = globaltimer();
            if (t0 == 0) t0 = now;
            if (now - t0 >= p.wait_ns) {
                *e = 1;
                bad = 1;
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
        *s_bad = bad;
    }
    __syncthreads();
    return *s_bad == 0;
}

// relaxation after a projection whose largest update was cd (fe_gpu_demean.f90:213-218)
__device__ __forceinline__ void star_relax(double& relax, double& pc, double cd) {
    if (cd > pc * 1.05)
        relax = fmax(0.4, relax * 0.5);
    else if (cd < pc * 0.8)
        relax = fmin(2.0, relax * 1.10);
    pc = cd;
}

__device__ __forceinline__ unsigned long long block_umax(unsigned long long v, unsigned long long* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = umax64(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
#pragma unroll
    for (int w = 1; w < AP_THREADS / 32; ++w) v = umax64(v, red[w]);
    return v;
}

// 28k rows over 3500/15/13 groups, 6 columns, 13 iterations, from host arrays: 3.1 ms
// with a launch per visit, 2.25 in one.
__global__ void __launch_bounds__(AP_THREADS, 2) ap_star_kernel(const __grid_constant__ ApStar p) {
    extern __shared__ __align__(16) unsigned char ap_smem[];
    __shared__ int s_bad;
    __shared__ unsigned long long s_red[AP_THREADS / 32];
    __shared__ double s_relax[SWEEP_MAXP + 1], s_pc[SWEEP_MAXP + 1];  // small dimensions, then the large one
    const int C = p.w.C, ld = p.w.ld, ns = p.n_small;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int WARPS = AP_THREADS / 32;
    // shared memory: column maxima | reduction area | per small dimension tab,
    // prev, mu, sums over w (Gs x C each), inv (Gs) | digit tables
    unsigned long long* cmax = reinterpret_cast<unsigned long long*>(ap_smem);  // 32
    long long* red = reinterpret_cast<long long*>(cmax + 32);                   // max(WARPS x AP_PART x C x 2, AP_THREADS)
    double* f = reinterpret_cast<double*>(red + max(WARPS * AP_PART * C * 2, AP_THREADS));
    double *tab[SWEEP_MAXP], *prev[SWEEP_MAXP], *mu[SWEEP_MAXP], *tw[SWEEP_MAXP], *inv[SWEEP_MAXP];
    int sum_at[SWEEP_MAXP];
    int words = 0;
    for (int i = 0; i < ns; ++i) {
        const int P = p.s[i].G * C;
        tab[i] = f;
        prev[i] = f + P;
        mu[i] = f + 2 * P;
        tw[i] = f + 3 * P;
        inv[i] = f + 4 * P;
        f += 4 * P + p.s[i].G;
        sum_at[i] = words;
        words += 2 * P;
        for (int e = threadIdx.x; e < P; e += AP_THREADS) {
            tab[i][e] = 0.0;
            prev[i][e] = p.s[i].prev[e];
            mu[i][e] = p.s[i].mu[e];
            tw[i][e] = 0.0;
        }
        for (int g = threadIdx.x; g < p.s[i].G; g += AP_THREADS) inv[i][g] = p.s[i].inv[g];
    }
    FixDigits* digits = reinterpret_cast<FixDigits*>(f);
    if (threadIdx.x <= ns) {
        s_relax[threadIdx.x] = p.relax[p.relax_at[threadIdx.x]];
        s_pc[threadIdx.x] = p.prev_change[p.relax_at[threadIdx.x]];
    }
    __syncthreads();
    // this block's groups of the large dimension
    const int G = p.w.G;
    const int gb0 = (int)((long long)G * blockIdx.x / gridDim.x), gb1 = (int)((long long)G * (blockIdx.x + 1) / gridDim.x);
    const int rps = AP_THREADS / C;
    const int rr = (int)threadIdx.x / C;
    const int c = (int)threadIdx.x - rr * C;
    const bool active = rr < rps;
    const int slots = 32 / C, slot = lane / C, sc = lane - slot * C;
    int top = 1;
    while (top < slots) top <<= 1;
    top >>= 1;
    unsigned long long it_max = 0;  // largest update of the iteration
    unsigned long long barrier = 0;
    int turn = 0;     // projections of w so far (ring of change)
    int visit = 0;    // visits of w so far (ring of sums)
    int iter = 0;
    bool stop = false, ok = true;

    // n projections in a row of small dimension i, by every block alike
    auto small_visit = [&](int i, int n) {
        const int Gi = p.s[i].G, P = Gi * C;
        for (int j = 0; j < n; ++j) {
            unsigned long long upd = 0;
            const double relax = s_relax[i];
            for (int e = threadIdx.x; e < P; e += AP_THREADS) {
                const int t = e / C, cc = e - t * C;
                double T = tw[i][e];
                for (int o = 0; o < ns; ++o) {
                    if (o == i) continue;
                    const ApDense<double>& D = p.ss[i][o];
                    const int pitch = ap_count_pitch(Gi);
                    const double* to = tab[o] + cc;
                    if (D.wide) {
                        const uint32_t* N = static_cast<const uint32_t*>(D.N) + t;
                        for (int g = 0; g < D.Ge; ++g) T = fma((double)N[g * pitch], to[g * C], T);
                    } else {
                        const uint8_t* N = static_cast<const uint8_t*>(D.N) + t;
                        for (int g = 0; g < D.Ge; ++g) T = fma((double)N[g * pitch], to[g * C], T);
                    }
                }
                const double a = tab[i][e];
                const double mean = fma(-T, inv[i][t], mu[i][e]) - a;
                const double pv = prev[i][e];
                const double mixed = pv + relax * (mean - pv);
                prev[i][e] = mixed;
                tab[i][e] = a + mixed;
                upd = umax64(upd, update_bits(mixed));
            }
            upd = block_umax(upd, s_red);
            it_max = umax64(it_max, upd);
            if (threadIdx.x == 0) star_relax(s_relax[i], s_pc[i], bits_dbl(upd));
            __syncthreads();
        }
    };
    // the largest update of the projection of w in `turn`, once all blocks are in
    auto close_projection = [&](unsigned long long upd) {
        upd = block_umax(upd, s_red);
        unsigned long long* ch = p.change + turn % AP_STAR_RING;
        if (threadIdx.x == 0) {
            if (upd) atomicMax(ch, upd);
            if (blockIdx.x == 0) p.change[(turn + 2) % AP_STAR_RING] = 0ULL;  // last read two projections ago
        }
        if (!star_barrier(p, ++barrier, &s_bad)) return false;
        const unsigned long long all = __ldcg(ch);
        it_max = umax64(it_max, all);
        if (threadIdx.x == 0) star_relax(s_relax[ns], s_pc[ns], bits_dbl(all));
        ++turn;
        __syncthreads();
        return true;
    };
    auto visit_w = [&]() {
        // digits of the small tables, one scale per column over all of them
        for (int cc = threadIdx.x; cc < C; cc += AP_THREADS) {
            unsigned long long m = 0;
            for (int i = 0; i < ns; ++i)
                for (int t = 0; t < p.s[i].G; ++t) m = umax64(m, abs_bits(tab[i][t * C + cc]));
            cmax[cc] = m;
        }
        __syncthreads();
        {
            FixDigits* d = digits;
            for (int i = 0; i < ns; ++i) {
                const int Gi = p.s[i].G;
                for (int e = threadIdx.x; e < four_rows(Gi) * C; e += AP_THREADS) {
                    const int t = e / C;
                    d[e] = fix_digits(to_fixed(t < Gi ? tab[i][e] : 0.0, fix_exponent(cmax[e - t * C])));
                }
                d += four_rows(Gi) * C;
            }
        }
        if (blockIdx.x == 0) {  // the ring entry after the next one: last read two visits ago
            unsigned long long* z = p.sums + (size_t)((visit + 2) % AP_STAR_RING) * words;
            for (int e = threadIdx.x; e < words; e += AP_THREADS) z[e] = 0ULL;
        }
        __syncthreads();
        double relax = s_relax[ns];
        unsigned long long upd = 0;
        if (active)
            for (int g = gb0 + rr; g < gb1; g += rps) {
                const long long idx = (long long)g * C + c;
                FixSum fs{0, 0};
                const FixDigits* d = digits;
                for (int i = 0; i < ns; ++i) {
                    if (p.sw[i].wide)
                        dense_dot_fixed<uint32_t>(p.sw[i].N, g, p.s[i].G, d, C, c, fs);
                    else
                        dense_dot_fixed<uint8_t>(p.sw[i].N, g, p.s[i].G, d, C, c, fs);
                    d += four_rows(p.s[i].G) * C;
                }
                const double base = fma(-fix_value(fs, cmax[c]), p.w.inv[g], p.w.mu[idx]);
                p.w.base[idx] = base;
                double* a = p.w.tab + (long long)g * ld + c;
                const double av = *a, pv = p.w.prev[idx];
                const double mixed = pv + relax * (base - av - pv);
                p.w.prev[idx] = mixed;
                *a = av + mixed;
                upd = umax64(upd, update_bits(mixed));
            }
        if (!close_projection(upd)) return false;
        relax = s_relax[ns];
        upd = 0;
        unsigned long long am = 0;
        if (active)
            for (int g = gb0 + rr; g < gb1; g += rps) {
                const long long idx = (long long)g * C + c;
                double* a = p.w.tab + (long long)g * ld + c;
                const double av = *a, pv = p.w.prev[idx];
                const double mixed = pv + relax * (p.w.base[idx] - av - pv);
                p.w.prev[idx] = mixed;
                const double an = av + mixed;
                *a = an;
                upd = umax64(upd, update_bits(mixed));
                am = umax64(am, abs_bits(an));
            }
        unsigned long long* ured = reinterpret_cast<unsigned long long*>(red);
        __syncthreads();
        ured[threadIdx.x] = active ? am : 0ULL;
        __syncthreads();
        if ((int)threadIdx.x < C) {
            unsigned long long m = 0;
            for (int j = 0; j < rps; ++j) m = umax64(m, ured[j * C + threadIdx.x]);
            if (m > __ldcg(p.w.amax + threadIdx.x)) atomicMax(p.w.amax + threadIdx.x, m);
        }
        if (!close_projection(upd)) return false;
        // sums over this block's groups for every small dimension, a piece of
        // AP_PART of its groups at a time
        unsigned long long* sums = p.sums + (size_t)(visit % AP_STAR_RING) * words;
        const int k = fix_exponent(__ldcg(p.w.amax + sc));
        const int g0 = slot < slots ? gb0 + warp * slots + slot : gb1;
        for (int i = 0; i < ns; ++i) {
            const int Gi = p.s[i].G;
            for (int t0 = 0; t0 < Gi; t0 += AP_PART) {
                FixSum acc[AP_PART];
#pragma unroll
                for (int q = 0; q < AP_PART; ++q) acc[q] = FixSum{0, 0};
                if (p.sw[i].wide)
                    small_walk<uint32_t, AP_PART, true>(static_cast<const uint32_t*>(p.sw[i].N), ap_count_pitch(Gi),
                                                  t0 / AP_PART, p.w.tab, ld, sc, k, g0, gb1, WARPS * slots, acc);
                else
                    small_walk<uint8_t, AP_PART, true>(static_cast<const uint8_t*>(p.sw[i].N), ap_count_pitch(Gi),
                                                 t0 / AP_PART, p.w.tab, ld, sc, k, g0, gb1, WARPS * slots, acc);
                const int nt = min(AP_PART, Gi - t0), PB = nt * C;
                __syncthreads();  // red of the previous piece has been read
#pragma unroll
                for (int q = 0; q < AP_PART; ++q) {
                    if (q >= nt) break;
                    const long long lo = warp_slot_sum(acc[q].lo, slot, slots, C, top);
                    const long long hi = warp_slot_sum(acc[q].hi, slot, slots, C, top);
                    if (lane < C) {
                        red[2 * (warp * PB + q * C + lane)] = lo;
                        red[2 * (warp * PB + q * C + lane) + 1] = hi;
                    }
                }
                __syncthreads();
                for (int e = threadIdx.x; e < 2 * PB; e += AP_THREADS) {
                    long long v = 0;
                    for (int w = 0; w < WARPS; ++w) v += red[2 * w * PB + e];
                    if (v) atomicAdd(sums + sum_at[i] + 2 * t0 * C + e, (unsigned long long)v);
                }
            }
        }
        if (!star_barrier(p, ++barrier, &s_bad)) return false;
        for (int i = 0; i < ns; ++i)
            for (int e = threadIdx.x; e < p.s[i].G * C; e += AP_THREADS) {
                const unsigned long long* l = sums + sum_at[i] + 2 * e;
                const FixSum fs{(long long)__ldcg(l + 1), (long long)__ldcg(l)};
                tw[i][e] = fix_value(fs, __ldcg(p.w.amax + e % C));
            }
        ++visit;
        __syncthreads();
        return true;
    };

    while (iter < p.max_iter && !stop && ok) {
        it_max = 0;
        for (int half = 0; half < 2 && ok; ++half) {
            // up through the small dimensions, the large one twice, and down again;
            // the first projection after the other half's last is of the same dimension
            for (int i = 0; i < ns; ++i) small_visit(i, 1);
            ok = visit_w();
            if (!ok) break;
            for (int i = ns - 1; i >= 0; --i) small_visit(i, 1);
        }
        ++iter;
        stop = bits_dbl(it_max) < p.ctl->tol;
    }
    if (blockIdx.x == 0) {
        for (int i = 0; i < ns; ++i)
            for (int e = threadIdx.x; e < p.s[i].G * C; e += AP_THREADS)
                p.s[i].tab[(e / C) * p.s[i].ld + e % C] = tab[i][e];
        for (int i = 0; i < ns; ++i)
            for (int cc = threadIdx.x; cc < C; cc += AP_THREADS) {
                unsigned long long m = 0;
                for (int t = 0; t < p.s[i].G; ++t) m = umax64(m, abs_bits(tab[i][t * C + cc]));
                p.s[i].amax[cc] = m;
            }
        if (threadIdx.x == 0) {
            p.ctl->iterations = iter;
            p.ctl->max_update = bits_dbl(it_max);
            p.ctl->stop = stop ? 1 : 0;
        }
    }
}

__global__ void __launch_bounds__(AP_THREADS) ap_load_kernel(const double* __restrict__ inc, long long G, int C, int ld,
                                                             double* __restrict__ tab, double* __restrict__ total,
                                                             unsigned long long* __restrict__ amax) {
    __shared__ unsigned long long red[AP_THREADS];
    const int rps = AP_THREADS / C;
    const int rr = (int)threadIdx.x / C;
    const int c = (int)threadIdx.x - rr * C;
    unsigned long long m = 0;
    if (rr < rps)
        for (long long g = (long long)blockIdx.x * rps + rr; g < G; g += (long long)gridDim.x * rps) {
            const double v = inc[g * C + c];
            tab[g * ld + c] = v;
            total[g * C + c] += v;
            m = umax64(m, abs_bits(v));
        }
    red[threadIdx.x] = m;
    __syncthreads();
    if ((int)threadIdx.x < C) {
        m = 0;
        for (int j = 0; j < rps; ++j) m = umax64(m, red[j * C + threadIdx.x]);
        if (m) atomicMax(amax + threadIdx.x, m);
    }
}

__global__ void ap_reset_kernel(ApSlot* slots, const double* relax, const double* prev_change, int n_fe, ApCtl* ctl,
                                double tol) {
    const int d = threadIdx.x;
    if (d < n_fe) {
        ApSlot* s = slots + d * AP_SLOTS;
        for (int i = 0; i < AP_SLOTS; ++i) {
            // equal changes before the first projection: the rule leaves its relaxation alone
            s[i].relax = relax[d];
            s[i].change = dbl_bits(prev_change[d]);
        }
        s[0].change = 0ULL;
    }
    if (d == 0) {
        ctl->tol = tol;
        ctl->max_update = 0.0;
        ctl->iterations = 0;
        ctl->stop = 0;
    }
}

__global__ void ap_check_kernel(const ApSlot* slots, int n_fe, int half, ApCtl* ctl) {
    if (ctl->stop) return;
    unsigned long long m = 0;
    for (int i = threadIdx.x; i < n_fe * AP_PER_ITERATION; i += 32)
        m = umax64(m, slots[i / AP_PER_ITERATION * AP_SLOTS + half * AP_PER_ITERATION + i % AP_PER_ITERATION].change);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = umax64(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) {
        const double v = bits_dbl(m);
        ctl->max_update = v;
        ctl->iterations += 1;
        if (v < ctl->tol) ctl->stop = 1;
    }
}

// Pair counts of a dimension whose rows come in group order: a block owns gpb
// consecutive groups and counts their rows in shared memory. The rows of a
// block are contiguous; nothing but the block's own table is updated, so no
// global atomics (count_pairs_kernel: 1.8 ms for 13M rows on a 13 x 12 matrix,
// every row on one of 156 addresses).
__global__ void __launch_bounds__(256) count_sorted_kernel(const int32_t* __restrict__ off, int Ge,
                                                           const int32_t* __restrict__ gid_s, int Gs, int gpb,
                                                           uint8_t* __restrict__ N8, uint32_t* __restrict__ N32,
                                                           unsigned* __restrict__ mx) {
    extern __shared__ uint32_t cnt[];  // gpb x Gs, then gpb + 1 offsets
    int32_t* so = reinterpret_cast<int32_t*>(cnt + gpb * Gs);
    const int g0 = blockIdx.x * gpb, ng = min(gpb, Ge - g0);
    for (int i = threadIdx.x; i < ng * Gs; i += blockDim.x) cnt[i] = 0u;
    for (int i = threadIdx.x; i <= ng; i += blockDim.x) so[i] = off[g0 + i];
    __syncthreads();
    const int r0 = so[0], r1 = so[ng];
    for (int r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
        int lo = 0, hi = ng - 1;  // the group of row r: last one starting at or before it
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (so[mid] <= r)
                lo = mid;
            else
                hi = mid - 1;
        }
        atomicAdd(cnt + lo * Gs + gid_s[r], 1u);
    }
    __syncthreads();
    unsigned m = 0;
    for (int i = threadIdx.x; i < ng * Gs; i += blockDim.x) {
        const uint32_t v = cnt[i];
        m = max(m, v);
        if (N32) N32[(long long)g0 * Gs + i] = v;
        if (N8) N8[(long long)g0 * Gs + i] = (uint8_t)min(v, 255u);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(mx, m);
}

template <typename CT>
__global__ void pad_counts_kernel(const CT* __restrict__ src, long long Ge, int Gs, int pitch, CT* __restrict__ dst) {
    const long long total = Ge * pitch;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long g = i / pitch;
        const int t = (int)(i - g * pitch);
        dst[i] = t < Gs ? src[g * Gs + t] : CT(0);
    }
}

// Pair counts of a small matrix: a table per block in shared memory, added to
// the global one once (integers: the order does not matter).
__global__ void __launch_bounds__(256) count_small_kernel(const int32_t* __restrict__ gid_e, int Ge,
                                                          const int32_t* __restrict__ gid_s, long long n, int Gs,
                                                          uint32_t* __restrict__ N) {
    extern __shared__ uint32_t cnt[];
    for (int i = threadIdx.x; i < Ge * Gs; i += blockDim.x) cnt[i] = 0u;
    __syncthreads();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        atomicAdd(cnt + gid_e[i] * Gs + gid_s[i], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < Ge * Gs; i += blockDim.x)
        if (cnt[i]) atomicAdd(N + i, cnt[i]);
}

// largest value the shared memory of a visit may take
constexpr int AP_SMEM = 200 * 1024;
// per-warp sums of the widest block of a small dimension (24 groups, 32 columns)
constexpr size_t AP_SMALL_SMEM = 100 * 1024;

unsigned ap_row_blocks(long long G, int C) {
    const int rps = AP_THREADS / C;
    const long long want = (G + rps - 1) / rps;
    return (unsigned)std::max(1LL, std::min(want, (long long)num_sms() * 8));
}

}  // namespace

template <typename T>
int launch_ap_visit(const ApVisit<T>& p, cudaStream_t s) {
    if (p.t.G <= 0) return 0;
    if (p.t.C > 32) return set_error("group-table projection: %d columns", p.t.C);
    size_t smem = sizeof(unsigned long long) * (AP_THREADS + 32);
    for (int e = 0; e < p.n_dense && !p.small_known; ++e) smem += sizeof(T) * (size_t)four_rows(p.dense[e].Gs) * p.t.C;
    static const cudaError_t attr =
        cudaFuncSetAttribute(ap_visit_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "group-table projection attr");
    ap_visit_kernel<T><<<ap_row_blocks(p.t.G, p.t.C), AP_THREADS, smem, s>>>(p);
    FEGB_LAUNCH_CHECK("group-table projection");
    return 0;
}
template int launch_ap_visit<float>(const ApVisit<float>&, cudaStream_t);
template int launch_ap_visit<double>(const ApVisit<double>&, cudaStream_t);

template <typename T>
int launch_ap_repeat(const ApTables<T>& t, int slot, const ApCtl* ctl, cudaStream_t s) {
    if (t.G <= 0) return 0;
    ap_repeat_kernel<T><<<ap_row_blocks(t.G, t.C), AP_THREADS, 0, s>>>(t, slot, ctl);
    FEGB_LAUNCH_CHECK("repeated group-table projection");
    return 0;
}
template int launch_ap_repeat<float>(const ApTables<float>&, int, const ApCtl*, cudaStream_t);
template int launch_ap_repeat<double>(const ApTables<double>&, int, const ApCtl*, cudaStream_t);

size_t ap_small_scratch(int Gs, int C, int n_src) { return (size_t)Gs * C * AP_PART_BLOCKS * std::max(1, n_src); }

template <typename T, int GT>
int launch_ap_small_gt(const ApSmall<T>& p, const ApSmallGrid& gr, size_t smem, cudaStream_t s) {
    static const cudaError_t attr =
        cudaFuncSetAttribute(ap_small_kernel<T, GT>, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMALL_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "small-dimension projection attr");
    ap_small_kernel<T, GT><<<gr.first[p.n_src * gr.parts], AP_THREADS, smem, s>>>(p, gr);
    FEGB_LAUNCH_CHECK("small-dimension projection");
    return 0;
}

template <typename T>
int launch_ap_small(const ApSmall<T>& p, cudaStream_t s) {
    const int C = p.t.C, Gs = p.t.G, P = Gs * C;
    if (Gs <= 0) return 0;
    if (Gs > DENSE_SMALL_MAX_G || C > 32 || p.n_src < 1) return set_error("small-dimension projection: G=%d C=%d", Gs, C);
    ApSmallGrid gr{};
    gr.parts = Gs <= AP_WHOLE ? 1 : (Gs + AP_PART - 1) / AP_PART;
    // the fold: totals, one value per thread, column and warp maxima
    const size_t per_warp = (sizeof(T) == 8 ? 2 * sizeof(long long) : sizeof(float)) * (size_t)std::min(Gs, AP_WHOLE) * C;
    const size_t smem = std::max(sizeof(double) * ((size_t)P + AP_THREADS + C + 8), per_warp * (AP_THREADS / 32));
    const long long per_block = (long long)(AP_THREADS / 32) * (32 / C) * AP_DEPTH;
    for (int e = 0; e < p.n_src; ++e) {
        const long long want = (p.src[e].Ge + per_block - 1) / per_block;
        const int limit = sizeof(T) == 4 ? AP_PART_BLOCKS : gr.parts == 1 && Gs > AP_PART ? AP_FIX_BLOCKS / 2 : AP_FIX_BLOCKS;
        const int nb = (int)std::max(1LL, std::min<long long>(want, limit));
        for (int h = 0; h < gr.parts; ++h) gr.first[e * gr.parts + h + 1] = gr.first[e * gr.parts + h] + nb;
    }
    // as many sums as the dimension has groups, nearly: a lane's registers and adds
    // (FP64 form, 940k groups, fits with two dimensions of 3 / 6 / 8 / 12 groups: 12.3
    // / 12.6 / 12.7 / 13.4 ms, all with 16 sums 12.8 / 13.0 / 13.1 / 13.5; FP32 form
    // alike within 1 %)
    if (Gs <= 4) return launch_ap_small_gt<T, 4>(p, gr, smem, s);
    if (Gs <= 8) return launch_ap_small_gt<T, 8>(p, gr, smem, s);
    if (Gs <= 12) return launch_ap_small_gt<T, 12>(p, gr, smem, s);
    if (Gs <= AP_PART || Gs > AP_WHOLE) return launch_ap_small_gt<T, AP_PART>(p, gr, smem, s);
    return launch_ap_small_gt<T, AP_WHOLE>(p, gr, smem, s);
}
template int launch_ap_small<float>(const ApSmall<float>&, cudaStream_t);
template int launch_ap_small<double>(const ApSmall<double>&, cudaStream_t);

size_t ap_star_sums(const ApStar& p) {
    size_t w = 0;
    for (int i = 0; i < p.n_small; ++i) w += 2 * (size_t)p.s[i].G * p.w.C;
    return w;
}
size_t ap_star_smem(const ApStar& p) {
    const int C = p.w.C;
    size_t b = sizeof(unsigned long long) * 32 +
               sizeof(long long) * (size_t)std::max((AP_THREADS / 32) * AP_PART * C * 2, AP_THREADS);
    for (int i = 0; i < p.n_small; ++i)
        b += sizeof(double) * ((size_t)4 * p.s[i].G * C + p.s[i].G) + sizeof(FixDigits) * (size_t)four_rows(p.s[i].G) * C;
    return b;
}

int launch_ap_star(const ApStar& p, cudaStream_t s) {
    if (p.w.G <= 0 || p.n_small < 1 || p.w.C > 32) return set_error("projections in one launch: invalid sizes");
    const size_t smem = ap_star_smem(p);
    if (smem > AP_STAR_SMEM) return set_error("projections in one launch: %zu bytes of shared memory", smem);
    static const cudaError_t attr =
        cudaFuncSetAttribute(ap_star_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AP_STAR_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "projections attr");
    int per_sm = 0;
    FEGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ap_star_kernel, AP_THREADS, smem),
              "projections occupancy");
    if (per_sm < 1) return set_error("projections in one launch: no block fits");
    // three steps of 256 / C groups a block while blocks are few (each more block
    // makes the barriers dearer), else as many as are resident
    const long long want = ((long long)p.w.G + 3 * (AP_THREADS / p.w.C) - 1) / (3 * (AP_THREADS / p.w.C));
    const unsigned blocks = (unsigned)std::max(1LL, std::min<long long>(want, (long long)per_sm * num_sms()));
    ApStar q = p;
    void* args[] = {&q};
    FEGB_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(ap_star_kernel), dim3(blocks), dim3(AP_THREADS), args,
                                          smem, s),
              "projections in one launch");
    FEGB_LAUNCH_CHECK("projections in one launch");
    return 0;
}

int launch_ap_load(const double* inc, long long G, int C, int ld, double* tab, double* total,
                   unsigned long long* amax, cudaStream_t s) {
    if (G <= 0) return 0;
    if (C > 32) return set_error("group tables: %d columns", C);
    ap_load_kernel<<<ap_row_blocks(G, C), AP_THREADS, 0, s>>>(inc, G, C, ld, tab, total, amax);
    FEGB_LAUNCH_CHECK("group tables of an increment");
    return 0;
}

int launch_ap_reset(ApSlot* slots, const double* relax, const double* prev_change, int n_fe, ApCtl* ctl, double tol,
                    cudaStream_t s) {
    ap_reset_kernel<<<1, 32, 0, s>>>(slots, relax, prev_change, n_fe, ctl, tol);
    FEGB_LAUNCH_CHECK("projection state");
    return 0;
}

int launch_ap_check(const ApSlot* slots, int n_fe, int half, ApCtl* ctl, cudaStream_t s) {
    ap_check_kernel<<<1, 32, 0, s>>>(slots, n_fe, half, ctl);
    FEGB_LAUNCH_CHECK("projection check");
    return 0;
}

int count_pairs_sorted(const int32_t* off, int Ge, const int32_t* gid_s, long long n, int Gs, uint8_t* N8,
                       uint32_t* N32, unsigned* mx, cudaStream_t s) {
    FEGB_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned), s), "count max reset");
    if (Ge <= 0 || n <= 0) return 0;
    // about 4096 rows a block, at most 32 KB of counts and 8 KB of offsets
    const long long mean = std::max(1LL, n / Ge);
    const int gpb = (int)std::max(1LL, std::min({4096 / mean, 8192LL / Gs, 2047LL}));
    const size_t smem = sizeof(uint32_t) * ((size_t)gpb * Gs + gpb + 1);
    count_sorted_kernel<<<(unsigned)((Ge + gpb - 1) / gpb), 256, smem, s>>>(off, Ge, gid_s, Gs, gpb, N8, N32, mx);
    FEGB_LAUNCH_CHECK("count pairs (sorted)");
    return 0;
}

template <typename CT>
int launch_pad_counts(const CT* src, long long Ge, int Gs, CT* dst, cudaStream_t s) {
    if (Ge <= 0) return 0;
    const int pitch = ap_count_pitch(Gs);
    pad_counts_kernel<CT><<<grid_stride_blocks(Ge * pitch, 256), 256, 0, s>>>(src, Ge, Gs, pitch, dst);
    FEGB_LAUNCH_CHECK("padded counts");
    return 0;
}
template int launch_pad_counts<uint8_t>(const uint8_t*, long long, int, uint8_t*, cudaStream_t);
template int launch_pad_counts<uint32_t>(const uint32_t*, long long, int, uint32_t*, cudaStream_t);

int count_pairs_small(const int32_t* gid_e, int Ge, const int32_t* gid_s, long long n, int Gs, uint32_t* N,
                      cudaStream_t s) {
    if ((long long)Ge * Gs > AP_COUNT_SMALL) return set_error("pair counts: %d x %d is not a small matrix", Ge, Gs);
    FEGB_CUDA(cudaMemsetAsync(N, 0, sizeof(uint32_t) * (size_t)Ge * Gs, s), "count matrix zero");
    if (n <= 0) return 0;
    const unsigned blocks = (unsigned)std::min<long long>((n + 2047) / 2048, (long long)num_sms() * 4);
    count_small_kernel<<<blocks, 256, sizeof(uint32_t) * (size_t)Ge * Gs, s>>>(gid_e, Ge, gid_s, n, Gs, N);
    FEGB_LAUNCH_CHECK("count pairs (small matrix)");
    return 0;
}

}  // namespace fegb
