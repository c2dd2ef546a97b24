// Alternating projections on group tables.
//
// A projection of the AP scheme needs only the group means of the current
// residual r = r0 - sum_e D_e alpha_e, and those follow from group tables alone:
//
//   mean_d = mu_d - (1 / n_d) sum_{e != d} N_de alpha_e - alpha_d,
//
// with mu_d the group means of r0, n_d the group sizes, N_de = D_d'D_e the row
// counts of every (group of d, group of e) pair and alpha_e the accumulated
// updates. The rows are read once for mu and written once at the end, whatever
// the number of iterations; an iteration moves the group tables, the id tuples
// and the count matrices.
// FP64 form, whole fits, rows -> tables: 13M rows over 4142/13/12 groups, 4
// columns 72 -> 12.4 ms; 2M rows over 100k/12k/20 groups, 12 columns 180 -> 24
// ms; 5M rows over 940k/13/12, 4 columns 39 -> 15.8 ms; 800 rows 6.4 -> 1.9 ms.
//
// A visit of a dimension evaluates the coupling sum once and runs one
// projection; the symmetric order projects its end dimensions twice in a row,
// and the second projection of such a pair only repeats the table update
// (the coupling sum has not changed).
//
// Kernels by dimension:
//  * launch_ap_visit: one thread per (group, column): swept sources over the
//    group's positions or from complete sums, small sources through their count
//    matrices, and the update, in one launch.
//  * launch_ap_small: a dimension of at most DENSE_SMALL_MAX_G groups: its count
//    matrices with every other dimension are reduced over those groups; the
//    last block to finish folds the blocks' sums and runs the projections.
//  * launch_ap_repeat: one more projection on the stored coupling sums.
#pragma once

#include "sweep.cuh"

namespace fegb {

// Relaxation state of a dimension: a ring of eight slots, one per projection, the
// four of an iteration in one half. A projection reads the two before it,
// applies the reference's rule (fe_gpu_demean.f90:213-218) and records the
// relaxation it used and its largest update.
struct ApSlot {
    double relax;
    unsigned long long change;  // bits of max |update|
};
constexpr int AP_PER_ITERATION = 4;
constexpr int AP_SLOTS = 2 * AP_PER_ITERATION;

struct ApCtl {
    double tol;
    double max_update;  // largest update of the last iteration
    int iterations;
    int stop;           // set when an iteration stayed below tol: later launches return at once
};

// Count matrix of a small dimension s against a dimension e: entry (g, t) at
// N[g * ap_count_pitch(Gs) + t], zero past Gs: rows of whole 16-count pieces, one
// load each. (Rows of Gs bytes read in 4-byte pieces: three times the
// instructions of the whole walk at 700k x 30 counts.)
constexpr int AP_PART = 16;
__host__ __device__ inline int ap_count_pitch(int Gs) { return (Gs + AP_PART - 1) / AP_PART * AP_PART; }
template <typename T>
struct ApDense {
    const void* N;     // uint8, or uint32 when wide
    int wide;
    int Gs;
    const T* tab;      // visit: the small dimension's table; small: the table of e
    const unsigned long long* amax;  // per column: bits of max |tab| so far
    int Ge;            // small: groups of e
};

template <typename T>
struct ApTables {
    int G, C, ld;                // ld: row stride of the tables of T
    const double* mu;            // G x C group means of r0
    const double* inv;           // 1 / group size (0: empty)
    T* tab;                      // accumulated updates (gathered by the other dimensions)
    double* alpha64;             // FP32 form: the updates in FP64 (G x C); null: tab is FP64
    double* prev;                // G x C relaxation memory
    double* base;                // G x C: mu - coupling sum / n of the last visit
    unsigned long long* amax;    // C: bits of the running max |tab| per column
    ApSlot* slots;
    // set: no projection; the table is an increment taken out of the residual,
    // whose new means mu - coupling sum / n - tab go here, the largest of them
    // into the slot's change
    double* means;
};

template <typename T>
struct ApVisit {
    ApTables<T> t;
    int slot;
    const ApCtl* ctl;
    // the small sources' coupling sums (G x C): stored by a visit that computes
    // them, read instead by one that finds the small dimensions unchanged
    double* small_sums;
    int small_known;
    // swept sources: complete sums of -(weighted source rows) (G x C), or the
    // group's positions (off set), or neither
    const T* sums;
    const int32_t* off;
    int n_src;
    const int32_t* src_gid[SWEEP_MAXP];
    const T* src_tab[SWEEP_MAXP];
    const float* weight;
    int n_dense;
    ApDense<T> dense[SWEEP_MAXP];
};

template <typename T>
struct ApSmall {
    ApTables<T> t;
    int slot;
    int projections;  // 1 or 2 in a row
    const ApCtl* ctl;
    int n_src;                   // the sources that changed since the last visit (at least one)
    ApDense<T> src[SWEEP_MAXP];
    double* src_sums[SWEEP_MAXP];  // Gs x C: coupling sums of each source, written
    int n_kept;                  // the other sources: their sums of an earlier visit
    const double* kept[SWEEP_MAXP];
    double* partials;            // ap_small_scratch() doubles
    unsigned long long* limbs;   // 2 x Gs x C per source, zero between launches
    unsigned* counter;           // zero between launches
};

template <typename T>
int launch_ap_visit(const ApVisit<T>& p, cudaStream_t s);
template <typename T>
int launch_ap_repeat(const ApTables<T>& t, int slot, const ApCtl* ctl, cudaStream_t s);
template <typename T>
int launch_ap_small(const ApSmall<T>& p, cudaStream_t s);
// doubles of ApSmall::partials for a dimension of Gs groups with n_src sources
size_t ap_small_scratch(int Gs, int C, int n_src);

// All iterations of a problem with one large dimension and otherwise small ones
// (at most DENSE_SMALL_MAX_G groups each) in one cooperative launch, FP64: a block
// owns a range of the large dimension's groups and a copy of the small tables.
// Everything between two visits of the large dimension then happens inside
// every block alike; the blocks meet only for the largest updates of the large
// dimension and for its sums over the small groups, six times an iteration.
struct ApStar {
    ApTables<double> w;          // the large dimension (amax: running column maxima, zeroed)
    int n_small;
    ApTables<double> s[SWEEP_MAXP];        // small dimensions in sweep order (amax: of the last tables)
    ApDense<double> sw[SWEEP_MAXP];        // counts of small i against the large dimension (Ge = w.G)
    ApDense<double> ss[SWEEP_MAXP][SWEEP_MAXP];  // counts of small i against small j (Ge = groups of j)
    unsigned long long* sums;    // AP_STAR_RING x ap_star_sums() words, zeroed
    unsigned long long* change;  // AP_STAR_RING words, zeroed: largest update of a projection of w
    unsigned long long* arrived;  // zeroed: the barrier's count
    unsigned long long wait_ns;  // limit of a wait at the barrier
    int* error;                  // zeroed: a barrier ran out of time
    ApCtl* ctl;                  // tol in; iterations, max_update, stop out
    const double* relax;         // starting relaxation and last change of the small dimensions, then of w
    const double* prev_change;
    int relax_at[SWEEP_MAXP + 1];
    int max_iter;
};
// Up to this many elements of the large dimension's table: the launches of an
// iteration (eight or more, several us each) weigh less beyond, and one launch
// keeps only two blocks an SM (whole fits, 4 columns, 6 rows a group: 20k groups
// 4.05 -> 2.70 ms, 150k 5.79 -> 4.24, 400k 8.52 -> 7.29; 940k 15.0 -> 15.7).
constexpr double AP_STAR_ELEMENTS = 2.0e6;
constexpr int AP_STAR_RING = 4;
// 64-bit words of one ring entry of ApStar::sums; shared memory the kernel needs
size_t ap_star_sums(const ApStar& p);
size_t ap_star_smem(const ApStar& p);
constexpr size_t AP_STAR_SMEM = 96 * 1024;
int launch_ap_star(const ApStar& p, cudaStream_t s);

// The FP64 tables of an increment: tab (row stride ld) = inc, total += inc (G x C,
// compact) and the columns' maxima of |inc| into amax (zeroed by the caller).
int launch_ap_load(const double* inc, long long G, int C, int ld, double* tab, double* total,
                   unsigned long long* amax, cudaStream_t s);

// Slots of all dimensions for a start from relaxation `relax` and last change
// `prev_change` per dimension (device arrays of n_fe).
int launch_ap_reset(ApSlot* slots, const double* relax, const double* prev_change, int n_fe, ApCtl* ctl, double tol,
                    cudaStream_t s);
// End of an iteration whose projections used the slots of half 0 or 1: their
// largest update against the tolerance.
int launch_ap_check(const ApSlot* slots, int n_fe, int half, ApCtl* ctl, cudaStream_t s);

// Row counts of the (group of e, group of s) pairs, N[g * pitch + t], s with at
// most DENSE_SMALL_MAX_G groups (pitch >= Gs, entries past Gs zero); *mx
// (device) = the largest count.
// Sorted form: off (G_e + 1) are e's groups in the row order of gid_s, no group
// longer than AP_COUNT_LONGEST rows. N8 receives the counts, clamped to 255
// (exact when *mx < 256); N32, when set, the counts as they are.
constexpr int AP_COUNT_LONGEST = 1 << 16;
int count_pairs_sorted(const int32_t* off, int Ge, const int32_t* gid_s, long long n, int pitch, uint8_t* N8,
                       uint32_t* N32, unsigned* mx, cudaStream_t s);
// dst (pitch ap_count_pitch(Gs), zero past Gs) = src (pitch Gs)
template <typename CT>
int launch_pad_counts(const CT* src, long long Ge, int Gs, CT* dst, cudaStream_t s);
// Form for matrices of at most AP_COUNT_SMALL entries, any row order; N is
// zeroed by the call.
constexpr int AP_COUNT_SMALL = 12 * 1024;
int count_pairs_small(const int32_t* gid_e, int Ge, const int32_t* gid_s, long long n, int pitch, uint32_t* N,
                      cudaStream_t s);

}  // namespace fegb
