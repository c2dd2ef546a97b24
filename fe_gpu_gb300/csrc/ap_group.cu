// Alternating projections on group tables (see ap_group.cuh).
#include "ap_group.cuh"

#include <algorithm>

namespace fegb {

namespace {

constexpr int AP_THREADS = 256;

// Fixed-point sums of FP64 table values. GB300 adds FP64 at 1/64 of the FP32
// rate, 64-bit integers at about 1/3 of it; so counts x values are summed as
// integers: a value v of a column with max |v| < 2^(e+1) becomes
// round(v 2^k), k = 61 - bits - e, where the counts of one sum add up to at most
// 2^bits. Such sums are exact and their order does not matter; with bits <= 9
// the one rounding of a value is at most half an ulp of the column's largest
// value, no more than an FP64 sum of such values loses.
constexpr int AP_FIX_BITS = 9;

__device__ __forceinline__ int fix_exponent(unsigned long long amax_bits, int bits) {
    const int e = (int)((amax_bits >> 52) & 0x7ff);
    return 61 - bits - (e - 1023);  // k
}

__device__ __forceinline__ long long to_fixed(double v, int k) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    if (e == 0) return 0;
    const unsigned long long m = ((unsigned long long)b & ((1ULL << 52) - 1ULL)) | (1ULL << 52);
    const int sh = e - 1075 + k;  // at most 61 - bits - 52
    unsigned long long r;
    if (sh >= 0)
        r = m << min(sh, 10);
    else if (sh > -54)
        r = (m + (1ULL << (-sh - 1))) >> (-sh);
    else
        r = 0;
    return b < 0 ? -(long long)r : (long long)r;
}

// Factor of the fixed-point sums of a column, 2^-k. A column with an infinity
// or NaN in its table has no fixed-point form: its factor is NaN, and so are its
// sums.
__device__ __forceinline__ double unfix_factor(unsigned long long amax_bits, int bits) {
    constexpr unsigned long long INF = 0x7ffULL << 52;
    if (amax_bits >= INF) return __longlong_as_double((long long)(INF | 1ULL << 51));
    const int e = max(-1022, min(1023, -fix_exponent(amax_bits, bits)));
    return __longlong_as_double((long long)(e + 1023) << 52);
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
// |v| for the convergence maximum, which passes over NaN as the row sweeps' does
__device__ __forceinline__ unsigned long long update_bits(double v) {
    const unsigned long long b = abs_bits(v);
    return b > (0x7ffULL << 52) ? 0ULL : b;
}

// One projection of element idx = (g, c): the new table value; mixed -> *upd.
template <typename T>
__device__ __forceinline__ double ap_update(const ApTables<T>& t, long long g, int c, double base, double relax,
                                            double* upd) {
    const long long idx = g * t.C + c;
    T* slot = t.tab + g * t.ld + c;
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
__device__ __forceinline__ void ap_block_max(unsigned long long upd, unsigned long long av, int c, bool active, int C,
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
    (void)c;
}

// The slots of a launch: this projection's relaxation recorded, the next
// projection's change cleared (it was last read two projections ago).
__device__ __forceinline__ void ap_open_slot(ApSlot* slots, int slot, double relax) {
    slots[slot].relax = relax;
    slots[(slot + 1) % AP_SLOTS].change = 0ULL;
}

// sum over t of N[g][t] * tab[t][c], small source, FP64/FP32 arithmetic
template <typename T, typename CT>
__device__ __forceinline__ T dense_dot(const CT* __restrict__ N, int Gs, const T* __restrict__ tab, int C, int c) {
    T a = T(0);
    int t = 0;
    for (; t + 4 <= Gs; t += 4) {
        const T n0 = (T)N[t], n1 = (T)N[t + 1], n2 = (T)N[t + 2], n3 = (T)N[t + 3];
        a = fma(n0, tab[t * C + c], a);
        a = fma(n1, tab[(t + 1) * C + c], a);
        a = fma(n2, tab[(t + 2) * C + c], a);
        a = fma(n3, tab[(t + 3) * C + c], a);
    }
    for (; t < Gs; ++t) a = fma((T)N[t], tab[t * C + c], a);
    return a;
}
__device__ __forceinline__ long long dense_dot_fixed(const uint8_t* __restrict__ N, int Gs,
                                                     const long long* __restrict__ tab, int C, int c) {
    long long a = 0;
    int t = 0;
    if ((Gs & 3) == 0) {  // rows start on 4 bytes
        for (; t < Gs; t += 4) {
            const unsigned w = *reinterpret_cast<const unsigned*>(N + t);
            a += (long long)(w & 255u) * tab[t * C + c];
            a += (long long)((w >> 8) & 255u) * tab[(t + 1) * C + c];
            a += (long long)((w >> 16) & 255u) * tab[(t + 2) * C + c];
            a += (long long)(w >> 24) * tab[(t + 3) * C + c];
        }
        return a;
    }
    for (; t < Gs; ++t) a += (long long)(unsigned)N[t] * tab[t * C + c];
    return a;
}

__device__ __forceinline__ int fix_bits(int groups, int max_count) {
    return 32 - __clz(groups * max_count);  // groups * max_count < 2^bits
}
inline bool fix_ok(int groups, int max_count) {
    return max_count > 0 && (long long)groups * max_count < (1 << AP_FIX_BITS);
}

// One visit: thread (r, c) takes column c of groups g0 + r, + rows per step...
// The small sources' tables sit in shared memory (as fixed-point integers where
// the counts allow it: FP64 form, uint8 counts).
template <typename T>
__global__ void __launch_bounds__(AP_THREADS) ap_visit_kernel(ApVisit<T> p, unsigned fixed_mask) {
    if (p.ctl->stop) return;
    extern __shared__ __align__(16) unsigned char ap_smem[];
    unsigned long long* red = reinterpret_cast<unsigned long long*>(ap_smem);
    unsigned char* tabs = ap_smem + sizeof(unsigned long long) * AP_THREADS;
    const ApTables<T>& t = p.t;
    const int C = t.C;
    const int rps = AP_THREADS / C;
    const int rr = (int)threadIdx.x / C;
    const int c = (int)threadIdx.x - rr * C;
    const bool active = rr < rps;
    // small tables: entry (t, c) at dst[t * C + c], 8 bytes per entry in the
    // FP64 form (double or fixed point), 4 in the FP32 form
    {
        T* dst = reinterpret_cast<T*>(tabs);
        for (int e = 0; e < p.n_dense; ++e) {
            const ApDense<T>& D = p.dense[e];
            const bool fx = (fixed_mask >> e) & 1u;
            const int bits = fx ? fix_bits(D.Gs, D.max_count) : 0;
            for (int i = threadIdx.x; i < D.Gs * C; i += AP_THREADS) {
                const int tt = i / C, cc = i - tt * C;
                const T v = D.tab[tt * t.ld + cc];
                if (sizeof(T) == 8 && fx)
                    reinterpret_cast<long long*>(dst)[i] = to_fixed((double)v, fix_exponent(D.amax[cc], bits));
                else
                    dst[i] = v;
            }
            dst += D.Gs * C;
        }
    }
    const double relax = ap_relax(t.slots, p.slot);
    if (blockIdx.x == 0 && threadIdx.x == 0) ap_open_slot(t.slots, p.slot, relax);
    __syncthreads();
    unsigned long long upd = 0, av = 0;
    if (active) {
        double unfix[SWEEP_MAXP];
        for (int e = 0; e < p.n_dense; ++e)
            unfix[e] = ((fixed_mask >> e) & 1u)
                           ? unfix_factor(p.dense[e].amax[c], fix_bits(p.dense[e].Gs, p.dense[e].max_count))
                           : 0.0;
        for (long long g = (long long)blockIdx.x * rps + rr; g < t.G; g += (long long)gridDim.x * rps) {
            const long long idx = g * C + c;
            T acc = T(0);  // the coupling sum
            if (p.sums) {
                acc = t.inv[g] != 0.0 ? -p.sums[idx] : T(0);  // sums of an empty group are not written
            } else if (p.off) {
                const int j0 = p.off[g], j1 = p.off[g + 1];
                int j = j0;
                for (; j + 2 <= j1; j += 2) {
                    T v0 = T(0), v1 = T(0);
                    for (int e = 0; e < p.n_src; ++e) {
                        const int32_t* __restrict__ sg = p.src_gid[e];
                        const T* __restrict__ st = p.src_tab[e];
                        v0 += st[(long long)sg[j] * t.ld + c];
                        v1 += st[(long long)sg[j + 1] * t.ld + c];
                    }
                    acc = p.weight ? fma((T)p.weight[j], v0, acc) : acc + v0;
                    acc = p.weight ? fma((T)p.weight[j + 1], v1, acc) : acc + v1;
                }
                if (j < j1) {
                    T v0 = T(0);
                    for (int e = 0; e < p.n_src; ++e) v0 += p.src_tab[e][(long long)p.src_gid[e][j] * t.ld + c];
                    acc = p.weight ? fma((T)p.weight[j], v0, acc) : acc + v0;
                }
            }
            const T* st = reinterpret_cast<const T*>(tabs);
            double cpl = (double)acc;
            for (int e = 0; e < p.n_dense; ++e) {
                const ApDense<T>& D = p.dense[e];
                if (sizeof(T) == 8 && ((fixed_mask >> e) & 1u))
                    cpl += (double)dense_dot_fixed(static_cast<const uint8_t*>(D.N) + g * D.Gs, D.Gs,
                                                   reinterpret_cast<const long long*>(st), C, c) *
                           unfix[e];
                else if (D.wide)
                    cpl += (double)dense_dot<T>(static_cast<const uint32_t*>(D.N) + g * D.Gs, D.Gs, st, C, c);
                else
                    cpl += (double)dense_dot<T>(static_cast<const uint8_t*>(D.N) + g * D.Gs, D.Gs, st, C, c);
                st += D.Gs * C;
            }
            const double base = t.mu[idx] - cpl * t.inv[g];
            t.base[idx] = base;
            double u;
            const double an = ap_update(t, g, c, base, relax, &u);
            upd = umax64(upd, update_bits(u));
            av = umax64(av, abs_bits(an));
        }
    }
    ap_block_max(upd, av, c, active, C, rps, red, t.slots + p.slot, t.amax);
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
    const double relax = ap_relax(t.slots, slot);
    if (blockIdx.x == 0 && threadIdx.x == 0) ap_open_slot(t.slots, slot, relax);
    unsigned long long upd = 0, av = 0;
    if (active)
        for (long long g = (long long)blockIdx.x * rps + rr; g < t.G; g += (long long)gridDim.x * rps) {
            double u;
            const double an = ap_update(t, g, c, t.base[g * C + c], relax, &u);
            upd = umax64(upd, update_bits(u));
            av = umax64(av, abs_bits(an));
        }
    ap_block_max(upd, av, c, active, C, rps, red, t.slots + slot, t.amax);
}

constexpr int AP_TILE = 64;       // groups of a source staged at a time
constexpr int AP_FLUSH = 32;      // groups per fixed-point run
constexpr int AP_PART_BLOCKS = 152;  // blocks per source whose partials are folded in order
constexpr int AP_FIX_BLOCKS = 608;

__device__ __forceinline__ void ap_cp16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void ap_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void ap_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// bytes of gsrc -> smem: whole 16-byte pieces asynchronously, the rest with plain stores
__device__ __forceinline__ void ap_stage(unsigned char* d, const unsigned char* g, long long bytes) {
    const long long whole = bytes & ~15LL;
    for (long long o = (long long)threadIdx.x * 16; o < whole; o += AP_THREADS * 16) ap_cp16(d + o, g + o);
    for (long long o = whole + threadIdx.x; o < bytes; o += AP_THREADS) d[o] = g[o];
}

struct ApSmallGrid {
    int first[SWEEP_MAXP + 1];  // first block of each source
    unsigned fixed_mask;        // sources summed in fixed point
};

// Small dimension (Gs groups): block b of a source reduces a range of the
// source's groups, sum_g N[g][t] tab[g][c] for all (t, c), tile by tile through
// shared memory (the next tile loads while this one is used). Thread: pairs
// (t, c) with c fastest, NP per thread, or a slice of the groups when the
// pairs are fewer than the threads. Fixed-point sums run over AP_FLUSH groups
// and are split into two 32-bit limbs added up exactly in 64-bit global
// atomics; other sums leave one FP64 partial per block, folded in block order.
// The last block to finish turns the sums into the projections.
template <typename T, int NP>
__global__ void __launch_bounds__(AP_THREADS) ap_small_kernel(ApSmall<T> p, ApSmallGrid gr) {
    if (p.ctl->stop) return;
    extern __shared__ __align__(16) unsigned char ap_smem[];
    __shared__ bool s_last;
    const ApTables<T>& t = p.t;
    const int C = t.C, Gs = t.G, ld = t.ld;
    const int P = Gs * C;
    int src = 0;
    while (src + 1 < p.n_src && (int)blockIdx.x >= gr.first[src + 1]) ++src;
    const ApDense<T>& D = p.src[src];
    const bool fx = sizeof(T) == 8 && ((gr.fixed_mask >> src) & 1u);
    const int bits = fx ? fix_bits(AP_FLUSH, D.max_count) : 0;
    const int nb = gr.first[src + 1] - gr.first[src], b = (int)blockIdx.x - gr.first[src];
    const long long tiles = (D.Ge + AP_TILE - 1) / AP_TILE;
    const long long t0 = tiles * b / nb, t1 = tiles * (b + 1) / nb;
    const size_t a_bytes = sizeof(T) * (size_t)AP_TILE * ld;
    const size_t n_bytes = (size_t)AP_TILE * Gs * (D.wide ? 4 : 1);
    const size_t buf = a_bytes + n_bytes;
    // pairs of this thread and its slice of the groups
    const int Pr = min(AP_THREADS, (P + 31) & ~31);
    const int S = NP > 1 ? 1 : AP_THREADS / Pr;
    const int slice = NP > 1 ? 0 : (int)threadIdx.x / Pr;
    const int pair0 = NP > 1 ? (int)threadIdx.x : (int)threadIdx.x - slice * Pr;
    int pt[NP], pc[NP];
    bool ok[NP];
    double sum[NP];
    long long lo[NP], hi[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int pr = pair0 + i * AP_THREADS;
        ok[i] = pr < P && slice < S;
        pt[i] = ok[i] ? pr / C : 0;
        pc[i] = ok[i] ? pr - pt[i] * C : 0;
        sum[i] = 0.0;
        lo[i] = hi[i] = 0;
    }
    auto stage = [&](long long tile, unsigned char* d) {
        const long long g0 = tile * AP_TILE;
        const int nt = (int)min((long long)AP_TILE, D.Ge - g0);
        ap_stage(d, reinterpret_cast<const unsigned char*>(D.tab + g0 * ld), (long long)nt * ld * sizeof(T));
        ap_stage(d + a_bytes, static_cast<const unsigned char*>(D.N) + g0 * Gs * (D.wide ? 4 : 1),
                 (long long)nt * Gs * (D.wide ? 4 : 1));
    };
    if (t0 < t1) stage(t0, ap_smem);
    ap_commit();
    for (long long tile = t0; tile < t1; ++tile) {
        unsigned char* cur = ap_smem + ((tile - t0) & 1 ? buf : 0);
        unsigned char* nxt = ap_smem + ((tile - t0) & 1 ? 0 : buf);
        if (tile + 1 < t1) stage(tile + 1, nxt);
        ap_commit();
        ap_wait_prev();
        __syncthreads();
        const int nt = (int)min((long long)AP_TILE, D.Ge - tile * AP_TILE);
        T* a = reinterpret_cast<T*>(cur);
        if (fx) {
            for (int i = threadIdx.x; i < nt * C; i += AP_THREADS) {
                const int gl = i / C, cc = i - gl * C;
                T* v = a + gl * ld + cc;
                *reinterpret_cast<long long*>(v) = to_fixed((double)*v, fix_exponent(D.amax[cc], bits));
            }
            __syncthreads();
            const long long* af = reinterpret_cast<const long long*>(a);
            const uint8_t* n8 = cur + a_bytes;
            for (int f = 0; f < nt; f += AP_FLUSH) {
                const int fe = min(nt, f + AP_FLUSH);
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    if (!ok[i]) continue;
                    long long acc = 0;
#pragma unroll 4
                    for (int gl = f + slice; gl < fe; gl += S)
                        acc += (long long)(unsigned)n8[gl * Gs + pt[i]] * af[gl * ld + pc[i]];
                    lo[i] += (long long)(acc & 0xffffffffLL);
                    hi[i] += acc >> 32;
                }
            }
        } else if (D.wide) {
            const uint32_t* n32 = reinterpret_cast<const uint32_t*>(cur + a_bytes);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if (!ok[i]) continue;
                T acc = T(0);
#pragma unroll 4
                for (int gl = slice; gl < nt; gl += S) acc = fma((T)n32[gl * Gs + pt[i]], a[gl * ld + pc[i]], acc);
                sum[i] += (double)acc;
            }
        } else {
            const uint8_t* n8 = cur + a_bytes;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if (!ok[i]) continue;
                T acc = T(0);
#pragma unroll 4
                for (int gl = slice; gl < nt; gl += S) acc = fma((T)n8[gl * Gs + pt[i]], a[gl * ld + pc[i]], acc);
                sum[i] += (double)acc;
            }
        }
        __syncthreads();  // this buffer is refilled by the next step
    }
    // this block's sums: limbs into the global accumulators, or its FP64 partial
    if (fx) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            if (!ok[i]) continue;
            unsigned long long* l = p.limbs + 2 * ((size_t)src * P + pair0 + i * AP_THREADS);
            if (lo[i]) atomicAdd(l, (unsigned long long)lo[i]);
            if (hi[i]) atomicAdd(l + 1, (unsigned long long)hi[i]);
        }
    } else {
        double* red = reinterpret_cast<double*>(ap_smem);
        __syncthreads();
        if (NP == 1) {
            if (slice < S) red[slice * Pr + pair0] = sum[0];
            __syncthreads();
            for (int i = threadIdx.x; i < P; i += AP_THREADS) {
                double v = 0.0;
                for (int k = 0; k < S; ++k) v += red[k * Pr + i];
                p.partials[((size_t)src * AP_PART_BLOCKS + b) * P + i] = v;
            }
        } else {
#pragma unroll
            for (int i = 0; i < NP; ++i)
                if (ok[i]) p.partials[((size_t)src * AP_PART_BLOCKS + b) * P + pair0 + i * AP_THREADS] = sum[i];
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
    for (int i = threadIdx.x; i < P; i += AP_THREADS) tot[i] = 0.0;
    for (int i = threadIdx.x; i < C; i += AP_THREADS) cmax[i] = 0ULL;
    __syncthreads();
    for (int e = 0; e < p.n_src; ++e) {
        if (sizeof(T) == 8 && ((gr.fixed_mask >> e) & 1u)) {
            const int eb = fix_bits(AP_FLUSH, p.src[e].max_count);
            for (int i = threadIdx.x; i < P; i += AP_THREADS) {
                unsigned long long* l = p.limbs + 2 * ((size_t)e * P + i);
                const long long l0 = (long long)__ldcg(l), l1 = (long long)__ldcg(l + 1);
                l[0] = 0ULL;
                l[1] = 0ULL;
                tot[i] += ((double)l1 * 4294967296.0 + (double)l0) * unfix_factor(p.src[e].amax[i % C], eb);
            }
            __syncthreads();
            continue;
        }
        const int nparts = gr.first[e + 1] - gr.first[e];  // at most AP_PART_BLOCKS
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
                base = t.mu[i] - tot[i] * t.inv[g];
                t.base[i] = base;
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
    unsigned mask = 0;
    size_t smem = sizeof(unsigned long long) * AP_THREADS;
    for (int e = 0; e < p.n_dense; ++e) {
        if (sizeof(T) == 8 && !p.dense[e].wide && fix_ok(p.dense[e].Gs, p.dense[e].max_count)) mask |= 1u << e;
        smem += sizeof(T) * (size_t)p.dense[e].Gs * p.t.C;
    }
    static const cudaError_t attr =
        cudaFuncSetAttribute(ap_visit_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "group-table projection attr");
    ap_visit_kernel<T><<<ap_row_blocks(p.t.G, p.t.C), AP_THREADS, smem, s>>>(p, mask);
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

template <typename T, int NP>
int launch_ap_small_np(const ApSmall<T>& p, const ApSmallGrid& gr, size_t smem, cudaStream_t s) {
    static const cudaError_t attr =
        cudaFuncSetAttribute(ap_small_kernel<T, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMEM);
    if (attr != cudaSuccess) return set_cuda_error(attr, "small-dimension projection attr");
    ap_small_kernel<T, NP><<<gr.first[p.n_src], AP_THREADS, smem, s>>>(p, gr);
    FEGB_LAUNCH_CHECK("small-dimension projection");
    return 0;
}

template <typename T>
int launch_ap_small(const ApSmall<T>& p, cudaStream_t s) {
    const int C = p.t.C, Gs = p.t.G, P = Gs * C;
    if (Gs <= 0) return 0;
    if (Gs > DENSE_SMALL_MAX_G || C > 32 || p.n_src < 1) return set_error("small-dimension projection: G=%d C=%d", Gs, C);
    ApSmallGrid gr{};
    size_t smem = 0;
    for (int e = 0; e < p.n_src; ++e) {
        const ApDense<T>& D = p.src[e];
        const bool fx = sizeof(T) == 8 && !D.wide && fix_ok(AP_FLUSH, D.max_count);
        if (fx) gr.fixed_mask |= 1u << e;
        const int tiles = (D.Ge + AP_TILE - 1) / AP_TILE;
        gr.first[e + 1] = gr.first[e] + std::max(1, std::min(tiles, fx ? AP_FIX_BLOCKS : AP_PART_BLOCKS));
        smem = std::max(smem, 2 * (sizeof(T) * (size_t)AP_TILE * p.t.ld + (size_t)AP_TILE * Gs * (D.wide ? 4 : 1)));
    }
    // the fold: totals, one value per thread, column and warp maxima
    smem = std::max(smem, sizeof(double) * ((size_t)P + AP_THREADS + C + 8));
    smem = std::max(smem, sizeof(double) * (size_t)AP_THREADS);
    if (P <= AP_THREADS) return launch_ap_small_np<T, 1>(p, gr, smem, s);
    if (P <= 2 * AP_THREADS) return launch_ap_small_np<T, 2>(p, gr, smem, s);
    if (P <= 4 * AP_THREADS) return launch_ap_small_np<T, 4>(p, gr, smem, s);
    return launch_ap_small_np<T, 8>(p, gr, smem, s);
}
template int launch_ap_small<float>(const ApSmall<float>&, cudaStream_t);
template int launch_ap_small<double>(const ApSmall<double>&, cudaStream_t);

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

int count_pairs_sorted(const int32_t* off, int Ge, const int32_t* gid_s, long long n, int Gs, uint8_t* N8, uint32_t* N32,
                       unsigned* mx, cudaStream_t s) {
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
