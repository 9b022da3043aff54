// fk_kpp.cu -- greedy k-means++ on the GPU (kmeans.rs:169-253), with the
// reference's arithmetic: every sum is the sequential left fold in F. Many
// seedings (the restarts of a fit, the fits of a batch) run together, one
// centre of each per step.
//
// The reference forms three sums per new centre, each a left fold in F from
// zero in row order: the total of the D^2 array (kmeans.rs:201), the running
// cumsum that locates each trial's candidate (:215-223), and each trial's
// potential (:225-237). A fold in F is not associative, so a tree gives other
// roundings and, at scale, other candidates. Here each fold is computed
// exactly as the sequential one, in parallel:
//
//   While the running sum p stays in one binade [2^e, 2^(e+1)), p is an
//   integer P on that binade's ulp grid, and adding v >= 0 rounds to
//   P + round(v / ulp) -- except for an exact half, where round-to-nearest-even
//   picks the even result, so the step depends on P's parity. Each element is
//   therefore a map P -> P + a[P & 1], and so is any run of elements: these
//   maps compose (associatively), and a composed map is exact whenever the
//   final P stays below the binade's top (the sum only grows, so every
//   intermediate stayed inside too). A run without an exact half is a plain
//   integer sum, in any order.
//
// Per new centre, four launches over all seedings:
//   kpp_pairs_kernel    the trials' candidates against the centres so far: a
//                       lower bound of each squared distance, as the row
//                       threshold of the next kernel.
//   kpp_trials_kernel   min(D^2, d(x, candidate)) for every trial in one pass.
//                       A row whose D^2 (its distance to its nearest centre q)
//                       is below a quarter of the bound of d(candidate, q)
//                       cannot come closer (triangle inequality, with room for
//                       every rounding): its value is copied without reading
//                       the row. The other rows are gathered, so that the
//                       arithmetic runs in full warps. Direct-form distances,
//                       no FMA; in f64 they are bounded in FP32 first and
//                       formed in FP64 only where the candidate may come
//                       closer.
//                       In f64 with many rows FP32 estimates come first and
//                       only the trials that can win are formed (kpp_contenders_kernel).
//                       Trials whose estimated potential is too far above the
//                       smallest (rounding bounds included) end here.
//   kpp_compose_kernel  per chunk of KPP_CH values the composed map for the
//                       binade of the chunk's estimated sums; where the sum may
//                       change binade inside the chunk, the maps of its groups
//                       of 32 values for both; the first chunk exactly. The
//                       estimate, an f32 prefix of partial sums, steers speed,
//                       never the result.
//   kpp_walk_kernel     one CTA per fold scans the chunk maps, 1024 at a time,
//                       with one exact F addition where the binade changes; a
//                       chunk whose maps do not apply is walked from its
//                       values. Every state it records is bit for bit the
//                       reference's running sum. The seeding's last CTA
//                       then takes the strictly smallest potential (first
//                       trial on ties: kmeans.rs:239-243), draws the next
//                       thresholds u * total in F (:213-214) and finds each
//                       trial's candidate: the first row whose running sum
//                       reaches its threshold (a 32-ary search over the chunk
//                       states, then that chunk walked exactly).
// The chosen trial's D^2 array becomes the new one without a copy (two
// buffers alternate). A non-positive total takes one uniform draw as a random
// row (:202-206).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "fk_internal.cuh"

namespace fk {
namespace {

template <typename T> __device__ __forceinline__ T kpp_mul(T a, T b);
template <> __device__ __forceinline__ float kpp_mul(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ double kpp_mul(double a, double b) { return __dmul_rn(a, b); }
template <typename T> __device__ __forceinline__ T kpp_add(T a, T b);
template <> __device__ __forceinline__ float kpp_add(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ double kpp_add(double a, double b) { return __dadd_rn(a, b); }

constexpr int KPP_CH = 1024;      // values per fold chunk
constexpr int KPP_THREADS = 256;  // every kernel's block
constexpr int KPP_WARPS = KPP_THREADS / 32;
constexpr int MAX_TRIALS = 16;
constexpr long long KPP_SPLIT_ROWS = 100000;  // f64: rows of a step from which it takes two passes
constexpr int KPP_SLAB = 32;      // features staged at a time

// ---------------------------------------------------- binade arithmetic --
template <typename T> struct Bits;
template <> struct Bits<float> {
    using U = uint32_t;
    static constexpr int MB = 23;      // stored mantissa bits
    static constexpr int EXPM = 0xFF;  // all-ones exponent (inf / NaN)
    static __device__ __forceinline__ U bits(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float from(U b) { return __uint_as_float(b); }
};
template <> struct Bits<double> {
    using U = unsigned long long;
    static constexpr int MB = 52;
    static constexpr int EXPM = 0x7FF;
    static __device__ __forceinline__ U bits(double v) { return (U)__double_as_longlong(v); }
    static __device__ __forceinline__ double from(U b) { return __longlong_as_double((long long)b); }
};

// Biased exponent of a positive normal finite value, else 0.
template <typename T>
__device__ __forceinline__ int normal_exp(T p) {
    using B = Bits<T>;
    const typename B::U b = B::bits(p);
    const int be = (int)((b >> B::MB) & (typename B::U)B::EXPM);
    const bool neg = (b >> (sizeof(typename B::U) * 8 - 1)) != 0;
    return (!neg && be >= 1 && be < B::EXPM) ? be : 0;
}

template <typename T>
__device__ __forceinline__ bool is_inf_or_nan(T p) {
    using B = Bits<T>;
    return (int)((B::bits(p) >> B::MB) & (typename B::U)B::EXPM) == B::EXPM;
}

// Significand of a normal value as an integer in [2^MB, 2^(MB+1)).
template <typename T>
__device__ __forceinline__ typename Bits<T>::U significand(T p) {
    using B = Bits<T>;
    const typename B::U m = ((typename B::U)1 << B::MB) - 1;
    return (B::bits(p) & m) | ((typename B::U)1 << B::MB);
}

template <typename T>
__device__ __forceinline__ T from_parts(int be, typename Bits<T>::U P) {
    using B = Bits<T>;
    const typename B::U m = ((typename B::U)1 << B::MB) - 1;
    return B::from(((typename B::U)be << B::MB) | (P & m));
}

// Increment of one value on the grid of binade be, and whether it is an exact
// half (then rounded down here: the sum's parity decides). Values that leave
// the binade, and negative or non-finite ones, give 2^(MB+1), which no sum in
// the binade can take.
template <typename T>
__device__ __forceinline__ typename Bits<T>::U inc_of(T v, int be, bool &tie) {
    using B = Bits<T>;
    using U = typename B::U;
    constexpr U OUT = (U)1 << (B::MB + 1);
    // without branches: neighbouring values lie in many binades
    const U b = B::bits(v);
    const int ev = (int)(b >> B::MB);  // the sign bit makes it > EXPM
    const U m = (b & (((U)1 << B::MB) - 1)) | (ev ? (U)1 << B::MB : (U)0);
    const int r = be - (ev ? ev : 1);
    const int sh = max(0, min(r, B::MB + 2));  // a shift of MB + 2 leaves nothing
    const U half = ((U)1 << sh) >> 1;
    const U s = m + half;
    const bool t = sh > 0 && (s & (((U)1 << sh) - 1)) == 0;
    const U q = (s >> sh) - (t ? (U)1 : (U)0);
    const bool out = (ev >= B::EXPM || r < 0) && (U)(b << 1) != 0;  // -0 is harmless
    tie |= t && !out;
    return out ? OUT : q;
}

// The map of 32 values, a lane each (dead lanes: increment 0), for binade be.
// A tie rounds the sum to even, so the parity after it is known and every later
// tie of the group is settled by the parities since the one before; only the
// first tie depends on the sum's parity at the start. Saturated at 2^(MB+1).
template <typename T>
struct GMap {
    typename Bits<T>::U a0, a1;
};

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) { return __reduce_add_sync(0xffffffffu, v); }
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    // values up to 2^54: two halves of 27 bits, 32 lanes
    const uint32_t lo = (uint32_t)v & ((1u << 27) - 1u), hi = (uint32_t)(v >> 27);
    return ((unsigned long long)__reduce_add_sync(0xffffffffu, hi) << 27) +
           (unsigned long long)__reduce_add_sync(0xffffffffu, lo);
}

// The parity of the increments since the last tie before this lane (from lane
// 0 if there is none), this lane's included: 1 where a tie here rounds up.
__device__ __forceinline__ unsigned tie_up(unsigned ties, unsigned odd, int lane) {
    const unsigned before = ties & ((1u << lane) - 1u);
    unsigned since = odd & (0xffffffffu >> (31 - lane));
    if (before) since &= ~(0xffffffffu >> __clz(before));
    return (unsigned)__popc(since) & 1u;
}

template <typename T>
__device__ __forceinline__ GMap<T> group_map(T v, bool live, int be) {
    using U = typename Bits<T>::U;
    constexpr U OUT = (U)1 << (Bits<T>::MB + 1);
    const int lane = threadIdx.x & 31;
    bool tie = false;
    U inc = live ? inc_of(v, be, tie) : (U)0;
    const unsigned ties = __ballot_sync(0xffffffffu, tie);
    if (!ties) {
        const U s = warp_sum(inc);
        const U a = s < OUT ? s : OUT;
        return GMap<T>{a, a};
    }
    const unsigned odd = __ballot_sync(0xffffffffu, (inc & 1) != 0);
    const int first = __ffs(ties) - 1;
    const unsigned up = tie_up(ties, odd, lane);
    if (tie && lane != first) inc += up;
    const U s = warp_sum(inc);
    const U e = (U)__shfl_sync(0xffffffffu, up, first);  // what the first tie adds to an even sum
    const U a0 = s + e, a1 = s + (1 - e);
    return GMap<T>{a0 < OUT ? a0 : OUT, a1 < OUT ? a1 : OUT};
}

// One more value at the end of a run held by one lane (at most 32 of them).
template <typename T>
__device__ __forceinline__ void run_add(GMap<T> &m, T v, int be) {
    using U = typename Bits<T>::U;
    bool tie = false;
    const U inc = inc_of(v, be, tie);
    m.a0 += inc;
    m.a1 += inc;
    m.a0 += tie ? m.a0 & 1 : (U)0;        // from an even sum: odd here rounds up
    m.a1 += tie ? 1 - (m.a1 & 1) : (U)0;  // from an odd sum
}

// f then g
template <typename T>
__device__ __forceinline__ GMap<T> gcompose(const GMap<T> &f, const GMap<T> &g) {
    return GMap<T>{f.a0 + ((f.a0 & 1) ? g.a1 : g.a0), f.a1 + ((f.a1 & 1) ? g.a0 : g.a1)};
}

// Inclusive scan over the lanes of saturated maps (at most 32 * 2^(MB+1): no overflow).
template <typename T>
__device__ __forceinline__ GMap<T> gscan(GMap<T> m) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const GMap<T> o{__shfl_up_sync(0xffffffffu, m.a0, off), __shfl_up_sync(0xffffffffu, m.a1, off)};
        if (lane >= off) m = gcompose(o, m);
    }
    return m;
}

// Up to 32 values from p (normal, binade be, significand P) on, a lane each:
// the state after each lane's value (valid up to the first that reaches 2^(MB+1)).
template <typename T>
__device__ __forceinline__ typename Bits<T>::U group_states(T v, bool live, int be, typename Bits<T>::U P) {
    using U = typename Bits<T>::U;
    const int lane = threadIdx.x & 31;
    bool tie = false;
    U inc = live ? inc_of(v, be, tie) : (U)0;
    const unsigned ties = __ballot_sync(0xffffffffu, tie);
    const unsigned odd = __ballot_sync(0xffffffffu, (inc & 1) != 0);
    if (tie) {
        unsigned up = tie_up(ties, odd, lane);
        if (!(ties & ((1u << lane) - 1u))) up ^= (unsigned)(P & 1);  // the first tie: the sum's own parity counts
        inc += up;
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const U o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += o;
    }
    return P + inc;
}

// One chunk of a fold: its map for binade elo (KIND_MAP); the exact sum at its
// end (KIND_END: the first chunk); or, where the sum may change from binade elo
// to the next inside it, the slot of its groups' maps for both (KIND_SLOT).
enum { KIND_NONE = 0, KIND_MAP = 1, KIND_END = 2, KIND_SLOT = 3 };
template <typename T>
struct CMap {
    GMap<T> s;  // KIND_END: a0 = the sum's bits
    int elo;
    short kind, slot;
};
constexpr int KPP_SLOTS = 32;  // chunks of a fold with group maps (about one per binade)

// A value as an f32 summand of the folds' estimates: F = f32 itself, F = f64
// times 2^-esc by its bits (no FP64 conversion; out of range: 0 or inf).
__device__ __forceinline__ float est_of(float v, int) { return v; }
__device__ __forceinline__ float est_of(double v, int esc) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7FFull) - 1023 - esc + 127;
    if (e <= 0) return 0.f;
    if (e >= 255) return INFINITY;
    return __uint_as_float(((uint32_t)e << 23) | (uint32_t)((b >> 29) & 0x7FFFFFull));
}
// Biased exponent in F of an estimate, else 0.
__device__ __forceinline__ int est_exp(float e, int, float) { return normal_exp(e); }
__device__ __forceinline__ int est_exp(float e, int esc, double) {
    const int be = normal_exp(e);
    const int b64 = be - 127 + esc + 1023;
    return be > 0 && b64 >= 1 && b64 < 0x7FF ? b64 : 0;
}

struct KppState {
    long long cursor;       // uniform draws consumed so far
    int direct[2];          // centre c was a uniform random row (slot c & 1): it has no trials
    int cur, cur_trial;     // buffer and trial slice of the current D^2 array
    int prev_trial;         // slice (of the other buffer) of the array before it
    int own_c;              // centre the current array was formed with (-1: the first)
    int done;               // folds of this step already walked
    int esc;                // exponent offset of the f64 estimates
    long long cand[MAX_TRIALS];
    double pot[MAX_TRIALS];  // fold of each trial's array (F, widened)
    double total;            // fold of the current D^2 array
    double est[2][MAX_TRIALS];  // estimate of each trial's fold (centre c: slot c & 1), in 2^esc
    double err[2];              // and a bound of what FP32 distances in it are off by
};

// One seeding (device copy of a KppJob and its workspace).
template <typename T>
struct KppFit {
    const T *x;
    const float *x32, *xerr;  // f32 rows (F = f32: x itself) and their rounding-error norms (F = f64)
    const double *draws;      // injected draws (n_draws of them, 0 past the end); null: the stream of seed
    T *centers;
    T *chains;                // [2][trials][n] D^2 arrays
    T *states;                // [2][trials][nch] running sum at each chunk's end
    CMap<T> *cmaps;           // [trials][nch]
    T *gstates;               // [2][trials][32] running sum after each 32 values of the first chunk
    GMap<T> *slots;           // [trials][KPP_SLOTS][2][32] group maps of the chunks that have them
    int *nslots;              // [trials]
    float *csum;              // [trials][tiles] estimates of the tiles' sums
    T *thr;                   // [k] skip threshold of each centre's rows at this step
    int32_t *own;             // [n] nearest centre so far
    unsigned short *closer;   // [n] F = f64: trials whose candidate may come closer to the row (split steps)
    int32_t *crow;            // [k] rows chosen
    KppState *st;
    long long n, nch, tiles, n_draws;
    unsigned long long seed;
    int d, k, trials, nan_direct;
};

template <typename T>
__device__ __forceinline__ double draw_at(const KppFit<T> &f, long long i) {
    if (f.draws) return i < f.n_draws ? f.draws[i] : 0.0;
    // splitmix64: draw i mixes the state after i + 1 golden-gamma steps
    unsigned long long z = f.seed + (unsigned long long)(i + 1) * 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z = z ^ (z >> 31);
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

__device__ __forceinline__ long long draw_to_range(double u, long long n) {
    long long i = (long long)floor(u * (double)n);
    if (i < 0) i = 0;
    if (i >= n) i = n - 1;
    return i;
}

// Work item: block blockIdx.x serves part y of seeding x (null table: one
// seeding, part blockIdx.x).
__device__ __forceinline__ int2 item_at(const int2 *__restrict__ items) {
    return items ? items[blockIdx.x] : make_int2(0, (int)blockIdx.x);
}

template <typename T>
__global__ void kpp_first_kernel(const KppFit<T> *__restrict__ fits) {
    const KppFit<T> f = fits[blockIdx.x];
    __shared__ long long first;
    if (threadIdx.x == 0) {
        first = draw_to_range(draw_at(f, 0), f.n);
        KppState *st = f.st;
        st->cursor = 1;
        st->direct[0] = st->direct[1] = 0;
        st->cur = st->cur_trial = st->prev_trial = 0;
        st->own_c = -1;
        st->done = 0;
        st->esc = 0;
        st->cand[0] = first;
        for (int t = 0; t < f.trials; t++) f.nslots[t] = 0;
        for (int t = 0; t < MAX_TRIALS; t++) st->est[0][t] = st->est[1][t] = 0.0;
        st->err[0] = st->err[1] = 0.0;
        f.crow[0] = (int32_t)first;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < f.d; j += blockDim.x) f.centers[j] = f.x[first * f.d + j];
}

// Squared distances of the step's candidates to the centres so far, bounded
// below (one warp per centre), as row thresholds (the smallest over the
// trials): a row whose D^2 value m is its computed distance to centre q, and
// m < thr[q], cannot come closer to any candidate. With g = (d + 4) u the relative error of a direct form, D = the
// exact distance: D(x, q) <= m (1 + 2g), thr = L (1 - rho) / 4 with L <= D(cand,
// q), so sqrt D(x, cand) >= sqrt L - sqrt D(x, q) >= sqrt D(x, q) (1 + rho - 2g)
// and the computed distance to the candidate is at least m (1 + 2 rho - 8g) > m
// for rho = (d + 8) 1e-6 (8g <= (d + 4) 4.8e-7 in f32). Bounds below 1e-30,
// where underflow would count, and NaN skip nothing.
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS) kpp_pairs_kernel(const KppFit<T> *__restrict__ fits, int c) {
    const unsigned groups = (unsigned)((c + KPP_WARPS - 1) / KPP_WARPS);
    const KppFit<T> &f = fits[blockIdx.x / groups];
    if (f.st->direct[c & 1]) return;
    const int lane = threadIdx.x & 31;
    const int q = (int)(blockIdx.x % groups) * KPP_WARPS + (threadIdx.x >> 5);
    if (q >= c) return;
    const int d = f.d;
    const long long rq = f.crow[q];
    const float *xq = f.x32 + rq * d;
    const float eq = f.xerr ? f.xerr[rq] : 0.f;
    const float rho = (float)(d + 8) * 1e-6f;
    float thmin = FLT_MAX;
#pragma unroll 4
    for (int t = 0; t < f.trials; t++) {
        const long long rc = f.st->cand[t];
        const float *xc = f.x32 + rc * d;
        float s = 0.f;
        for (int j = lane; j < d; j += 32) {
            const float v = __fsub_rn(xc[j], xq[j]);
            s = __fmaf_rn(v, v, s);
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float ec = f.xerr ? __fadd_ru(f.xerr[rc], eq) : 0.f;
        const float th = 0.25f * __fsub_rd(s, bound32(s, ec, d)) * (1.0f - rho);
        thmin = th < thmin ? th : (th >= thmin ? thmin : 0.f);  // NaN: 0
    }
    if (lane == 0) f.thr[q] = thmin > 1e-30f && thmin < FLT_MAX ? (T)thmin : T(0);
}

// d(a, b), direct form in the reference's order.
__device__ __forceinline__ double sqeuc(const double *__restrict__ a, const double *__restrict__ b, int d) {
    double v = 0.0;
#pragma unroll 8
    for (int j = 0; j < d; j++) {
        const double df = __dsub_rn(a[j], b[j]);
        v = __dadd_rn(v, __dmul_rn(df, df));
    }
    return v;
}

// m < thr for D^2 values and thresholds >= 0 (f64 by their bits: no FP64
// comparison; a NaN is never below).
__device__ __forceinline__ bool below(float m, float th) { return m < th; }
__device__ __forceinline__ bool below(double m, double th) {
    return (unsigned long long)__double_as_longlong(m) < (unsigned long long)__double_as_longlong(th);
}

// 16 or 4 bytes from global to shared memory, asynchronously; ok == false
// writes zeros (nothing is read).
__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, const float *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Row stride (floats) of a staged slab: a multiple of 4 with an odd number of
// 16-byte units, so that eight lanes reading 16 bytes of eight rows meet no
// bank conflict.
__host__ __device__ inline int slab_width(int d) { return d < KPP_SLAB ? (d + 3) / 4 * 4 : KPP_SLAB; }
__host__ __device__ inline int slab_stride(int w) { return (w / 4) & 1 ? w + 8 : w + 4; }
inline size_t trial_smem(int dmax, int tt) {
    const int w = slab_width(dmax);
    return sizeof(float) * ((size_t)KPP_THREADS * slab_stride(w) + (size_t)tt * w);
}

// Whether trial t's fold can be the smallest of the step's (by a whole warp).
// An estimate differs from the exact sum by less than 1e-5 of it (truncated to
// 24 bits, fewer than 100 f32 additions in a row) and err, and a fold in F by n u: a
// trial whose estimate is further above the smallest one than both allow has a
// strictly larger fold, which then need not be formed. Estimates that are not
// finite, or that values below the estimates' range could move, exclude no one.
// Three seedings of 1M x 64 in f64, k = 256: compose 77 -> 29 us a step, walk 54
// -> 47 (a MiniBatchKMeans fit 154 -> 142 ms); in f32 the folds' own rounding
// (n u = 6% at 1M rows) leaves more trials in.
template <typename T>
__device__ __forceinline__ bool contends(const KppFit<T> &f, int c, int t) {
    const int lane = threadIdx.x & 31;
    const float e = lane < f.trials ? (float)__ldcg(&f.st->est[c & 1][lane]) : INFINITY;
    float lo = e;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    const float eps = 1.1e-5f + 1.01f * (float)f.n * (sizeof(T) == 8 ? 1.2e-16f : 6.0e-8f);
    const float mine = __shfl_sync(0xffffffffu, e, t);
    const float err = 1.001f * (float)__ldcg(&f.st->err[c & 1]);
    if (!(lo >= 1e-18f && lo <= 1e37f) || eps > 0.2f) return true;
    return !(mine * (1.f - eps) - err > lo * (1.f + eps) + err);
}

// One CTA per tile of `scan` rows (a divisor of KPP_CH, a multiple of 256):
// every trial's min(D^2, d(x, candidate)) (INIT: d(x, first row), the first
// D^2 array; kmeans.rs:188-195, 225-233), and estimates of the tile's sums.
// First the rows' owners (nearest centre so far) are brought up to date and
// the rows that no candidate can come closer to get their values; the others
// are listed, then scored 256 at a time, a thread a row with all TT trials,
// the row read from a slab of KPP_SLAB features in shared memory.
//
// Bound at n = 1M, d = 64, 7 trials in f32: the FP32 pipe for the listed rows
// (3 d operations a pair), L2 for the values (8 bytes a pair).
//
// In f64 with many rows the step takes two passes: PASS_EST forms FP32 distances
// only, for estimates of the trials' sums with a bound of what they are off by,
// and marks the rows each candidate may come closer to; kpp_contenders_kernel
// then forms the arrays of the trials that can win, nearly always one. Three
// seedings of 1M x 64, k = 256, 7 trials: 273 us a
// step in one pass (FP64 distances and arrays of every trial), 100 + 61 in two.
enum { PASS_INIT, PASS_ALL, PASS_EST };
template <typename T, int TT, int PASS>
__global__ void __launch_bounds__(KPP_THREADS)
    kpp_trials_kernel(const KppFit<T> *__restrict__ fits, const int2 *__restrict__ items, int scan, int c) {
    constexpr bool F64 = sizeof(T) == 8, INIT = PASS == PASS_INIT, EST = PASS == PASS_EST;
    static_assert(F64 || !EST, "FP32 estimates are of FP64 distances");
    const int2 it = item_at(items);
    const KppFit<T> &f = fits[it.x];
    const KppState *st = f.st;
    if (!INIT && st->direct[c & 1]) return;
    const int d = f.d, ntr = INIT ? 1 : f.trials;
    const long long n = f.n, base = (long long)it.y * scan;
    extern __shared__ __align__(16) unsigned char kpp_smem[];
    const int W = slab_width(d), XS = slab_stride(W);
    float *const xs = reinterpret_cast<float *>(kpp_smem);  // [256][XS] rows
    float *const cs = xs + KPP_THREADS * XS;                // [TT][W] candidates
    __shared__ long long cand[TT];
    __shared__ float cerr[TT];
    __shared__ unsigned short list[KPP_CH];
    __shared__ unsigned short open_pairs[F64 ? KPP_THREADS * TT : 1];
    __shared__ int list_n, open_n;
    __shared__ float red[TT][KPP_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < TT) {
        cand[tid] = tid < ntr ? st->cand[tid] : 0;
        cerr[tid] = F64 && tid < ntr ? f.xerr[st->cand[tid]] : 0.f;
    }
    if (tid == 0) list_n = 0;
    const int cur = st->cur, esc = INIT ? 0 : st->esc;
    const T *mind = f.chains + ((long long)cur * f.trials + st->cur_trial) * n + base;
    const T *prev = f.chains + ((long long)(1 - cur) * f.trials + st->prev_trial) * n + base;
    T *out = f.chains + (long long)(INIT ? 0 : 1 - cur) * f.trials * n + base;
    const int rows = (int)min((long long)scan, n - base);
    const int own_c = st->own_c;
    // a power of two; far from 1 the estimates are not used
    const float unit = EST ? (esc >= -100 && esc <= 100 ? __int_as_float((127 - esc) << 23) : NAN) : 1.f;
    float psum[TT], skipped = 0.f, err = 0.f;
#pragma unroll
    for (int b = 0; b < TT; b++) psum[b] = 0.f;
    __syncthreads();
    if (INIT) {
        for (int i = tid; i < rows; i += KPP_THREADS) {
            list[i] = (unsigned short)i;
            f.own[base + i] = 0;
        }
        if (tid == 0) list_n = rows;
    } else {
        // at most four rows a thread, their loads issued together
        T m[KPP_CH / KPP_THREADS], pv[KPP_CH / KPP_THREADS];
        int o[KPP_CH / KPP_THREADS];
#pragma unroll
        for (int a = 0; a < KPP_CH / KPP_THREADS; a++) {
            const int i = a * KPP_THREADS + tid;
            m[a] = pv[a] = T(0);
            o[a] = 0;
            if (i < rows) {
                m[a] = mind[i];
                if (own_c >= 0) {
                    pv[a] = prev[i];
                    o[a] = f.own[base + i];
                }
            }
        }
#pragma unroll
        for (int a = 0; a < KPP_CH / KPP_THREADS; a++) {
            const int i = a * KPP_THREADS + tid;
            bool open = false;
            if (i < rows) {
                if (own_c >= 0 && m[a] < pv[a]) {
                    o[a] = own_c;
                    f.own[base + i] = own_c;
                }
                open = !below(m[a], f.thr[o[a]]);
                if (!open) {
                    skipped += est_of(m[a], esc);
                    if (EST) f.closer[base + i] = 0;
                    else
                        for (int t = 0; t < ntr; t++) out[(long long)t * n + i] = m[a];
                }
            }
            const unsigned bm = __ballot_sync(0xffffffffu, open);
            int at = 0;
            if (lane == 0 && bm) at = atomicAdd(&list_n, __popc(bm));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (open) list[at + __popc(bm & ((1u << lane) - 1u))] = (unsigned short)i;
        }
    }
    __syncthreads();
    const int nl = list_n;
    const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(f.x32) & 15) == 0;
    for (int l0 = 0; l0 < nl; l0 += KPP_THREADS) {
        const int cnt = min(KPP_THREADS, nl - l0);
        float acc[TT];
#pragma unroll
        for (int b = 0; b < TT; b++) acc[b] = 0.f;
        if (!(F64 && INIT)) {
            for (int j0 = 0; j0 < d; j0 += KPP_SLAB) {
                const int jn = min(KPP_SLAB, d - j0), j4 = (jn + 3) / 4;
                if (vec) {
                    for (int e = tid; e < cnt * (KPP_SLAB / 4); e += KPP_THREADS) {
                        const int r = e / (KPP_SLAB / 4), q = e % (KPP_SLAB / 4);
                        if (q < j4)
                            cp_async16(xs + r * XS + 4 * q, f.x32 + (base + list[l0 + r]) * d + j0 + 4 * q, true);
                    }
                } else {
                    for (int e = tid; e < cnt * KPP_SLAB; e += KPP_THREADS) {
                        const int r = e / KPP_SLAB, j = e % KPP_SLAB;
                        if (j < 4 * j4)
                            cp_async4(xs + r * XS + j, j < jn ? f.x32 + (base + list[l0 + r]) * d + j0 + j : f.x32,
                                      j < jn);
                    }
                }
                if (l0 == 0 || d > KPP_SLAB) {  // one slab: the candidates stay for every pass
                    for (int e = tid; e < TT * KPP_SLAB; e += KPP_THREADS) {
                        const int t = e / KPP_SLAB, j = e % KPP_SLAB;
                        if (j < 4 * j4) {
                            const bool ok = t < ntr && j < jn;
                            cp_async4(cs + t * W + j, ok ? f.x32 + cand[t] * d + j0 + j : f.x32, ok);
                        }
                    }
                }
                cp_async_wait_all();
                __syncthreads();
                if (tid < cnt) {
                    const float4 *xr = reinterpret_cast<const float4 *>(xs + tid * XS);
                    for (int q = 0; q < j4; q++) {
                        const float4 xv = xr[q];
#pragma unroll
                        for (int b = 0; b < TT; b++) {
                            const float4 cv = *reinterpret_cast<const float4 *>(cs + b * W + 4 * q);
                            float t0 = __fsub_rn(xv.x, cv.x), t1 = __fsub_rn(xv.y, cv.y);
                            float t2 = __fsub_rn(xv.z, cv.z), t3 = __fsub_rn(xv.w, cv.w);
                            if (F64) {
                                acc[b] = __fmaf_rn(t0, t0, acc[b]);
                                acc[b] = __fmaf_rn(t1, t1, acc[b]);
                                acc[b] = __fmaf_rn(t2, t2, acc[b]);
                                acc[b] = __fmaf_rn(t3, t3, acc[b]);
                            } else {  // a zero-padded feature adds +0: no change
                                acc[b] = __fadd_rn(acc[b], __fmul_rn(t0, t0));
                                acc[b] = __fadd_rn(acc[b], __fmul_rn(t1, t1));
                                acc[b] = __fadd_rn(acc[b], __fmul_rn(t2, t2));
                                acc[b] = __fadd_rn(acc[b], __fmul_rn(t3, t3));
                            }
                        }
                    }
                }
                __syncthreads();  // the slab is refilled
            }
        }
        if constexpr (!F64) {
            if (tid < cnt) {
                const int i = list[l0 + tid];
                const T m = INIT ? T(0) : mind[i];
#pragma unroll
                for (int b = 0; b < TT; b++)
                    if (b < ntr) {
                        const T v = acc[b];
                        const T r = INIT ? v : (v < m ? v : m);  // kmeans.rs:230-232
                        out[(long long)b * n + i] = r;
                        psum[b] += est_of(r, esc);
                    }
            }
        } else if constexpr (EST) {
            if (tid < cnt) {
                const int i = list[l0 + tid];
                const T m = mind[i];
                const float mu = __double2float_ru(m), me = est_of(m, esc), er = f.xerr[base + i];
                float worst = 0.f;
                unsigned closer = 0;
#pragma unroll
                for (int b = 0; b < TT; b++)
                    if (b < ntr) {
                        const float bnd = bound32(acc[b], __fadd_ru(er, cerr[b]), d);
                        float e = me;
                        if (!(__fsub_rd(acc[b], bnd) > mu)) {
                            closer |= 1u << b;
                            e = fminf(acc[b] * unit, me);
                            worst = bnd < FLT_MAX ? fmaxf(worst, bnd) : INFINITY;  // NaN: INFINITY
                        }
                        psum[b] += e;
                    }
                f.closer[base + i] = (unsigned short)closer;
                err = __fmaf_rn(worst, unit, err);
            }
        } else {
            // Pairs the FP32 bounds leave open -- rows the candidate may come
            // closer to, non-finite values, values beyond the f32 range --
            // are listed and formed in FP64 by the whole block, one pair a
            // thread; the others keep D^2 (d32 - bound > D^2).
            if (tid == 0) open_n = 0;
            __syncthreads();
            if (tid < cnt) {
                const int i = list[l0 + tid];
                const T m = INIT ? T(0) : mind[i];
                const float mu = INIT ? 0.f : __double2float_ru(m);
                const float er = INIT ? 0.f : f.xerr[base + i];
#pragma unroll
                for (int b = 0; b < TT; b++)
                    if (b < ntr) {
                        const float bnd = bound32(acc[b], __fadd_ru(er, cerr[b]), d);
                        if (!INIT && __fsub_rd(acc[b], bnd) > mu) {
                            out[(long long)b * n + i] = m;
                            psum[b] += est_of(m, esc);
                        } else {
                            open_pairs[atomicAdd(&open_n, 1)] = (unsigned short)((tid << 4) | b);
                        }
                    }
            }
            __syncthreads();
            const int no = open_n;
            for (int q = tid; q < no; q += KPP_THREADS) {
                const int e = open_pairs[q], b = e & 15, i = list[l0 + (e >> 4)];
                const T v = sqeuc(f.x + (base + i) * d, f.x + cand[b] * d, d);
                T r = v;
                if (!INIT) {
                    const T m = mind[i];
                    r = v < m ? v : m;
                }
                out[(long long)b * n + i] = r;
                // the summand's trial differs from thread to thread: one select per trial
#pragma unroll
                for (int t = 0; t < TT; t++) psum[t] += t == b ? est_of(r, esc) : 0.f;
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int b = 0; b < TT; b++) {
        float v = psum[b] + skipped;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[b][w] = v;
    }
    if (EST) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
        if (lane == 0 && err != 0.f) atomicAdd(&f.st->err[c & 1], (double)err);  // NaN too
    }
    __syncthreads();
    if (tid < ntr) {
        float v = 0.f;
        for (int q = 0; q < KPP_WARPS; q++) v += red[tid][q];
        if (!EST) f.csum[(long long)tid * f.tiles + it.y] = v;
        if (EST || PASS == PASS_ALL) atomicAdd(&f.st->est[c & 1][tid], (double)v);
    }
}

// The second pass of a split step: min(D^2, d(x, candidate)) of the trials that
// can win, `per` rows a CTA (2,048 or 4,096). Rows the candidate cannot come
// closer to keep their value; the others are listed and formed in FP64, a
// thread a row. Bound by the arrays' traffic (18 bytes a row) and by FP64, which
// takes a warp with one listed row as long as a full one: hence the many rows
// of a CTA (with 1,024, 104 us a step for three seedings of 1M x 64).
constexpr int CONT_ROWS = 4096;
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS)
    kpp_contenders_kernel(const KppFit<T> *__restrict__ fits, const int2 *__restrict__ items, int scan, int per, int c) {
    const int2 it = item_at(items);
    const KppFit<T> &f = fits[it.x];
    const KppState *st = f.st;
    if (st->direct[c & 1]) return;
    const long long n = f.n, base = (long long)it.y * per;
    __shared__ unsigned short list[CONT_ROWS];
    __shared__ float sums[CONT_ROWS / KPP_THREADS];  // of the tiles of `scan` rows
    __shared__ int list_n;
    const int tid = threadIdx.x, lane = tid & 31, esc = st->esc, d = f.d;
    const T *mind = f.chains + ((long long)st->cur * f.trials + st->cur_trial) * n + base;
    const int rows = (int)min((long long)per, n - base);
    for (int t = 0; t < f.trials; t++) {
        if (!contends(f, c, t)) continue;
        T *out = f.chains + ((long long)(1 - st->cur) * f.trials + t) * n + base;
        if (tid == 0) list_n = 0;
        if (tid < CONT_ROWS / KPP_THREADS) sums[tid] = 0.f;
        __syncthreads();
#pragma unroll 8
        for (int i0 = 0; i0 < rows; i0 += KPP_THREADS) {
            const int i = i0 + tid;
            const bool live = i < rows;
            const T m = live ? mind[i] : T(0);
            const bool open = live && ((f.closer[base + i] >> t) & 1u);
            if (live && !open) out[i] = m;
            float v = live && !open ? est_of(m, esc) : 0.f;
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const unsigned bm = __ballot_sync(0xffffffffu, open);
            int at = 0;
            if (lane == 0) {
                atomicAdd(&sums[i0 / scan], v);
                if (bm) at = atomicAdd(&list_n, __popc(bm));
            }
            at = __shfl_sync(0xffffffffu, at, 0);
            if (open) list[at + __popc(bm & ((1u << lane) - 1u))] = (unsigned short)i;
        }
        __syncthreads();
        const T *cand = f.x + st->cand[t] * d;
        for (int q = tid; q < list_n; q += KPP_THREADS) {
            const int i = list[q];
            const T v = sqeuc(f.x + (base + i) * d, cand, d), old = mind[i];
            const T r = v < old ? v : old;  // kmeans.rs:230-232
            out[i] = r;
            atomicAdd(&sums[i / scan], est_of(r, esc));
        }
        __syncthreads();
        if (tid * scan < rows) f.csum[(long long)t * f.tiles + base / scan + tid] = sums[tid];
        __syncthreads();
    }
}

// Rows of a staged chunk: value i at i + i / 32, so that reading a value a lane
// and reading a run of 32 a lane both spread over the banks.
__device__ __forceinline__ int staged(int i) { return i + (i >> 5); }
constexpr int KPP_STAGED = KPP_CH + 32;
template <typename T>
__device__ __forceinline__ void cp_async_one(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"((int)sizeof(T))
                 : "memory");
}

// The first chunk of a fold exactly, by one warp: f32 value by value (a
// dependent addition is four cycles); f64 (64 cycles) value by value for the
// first group, then a group at a time, by its map where its estimated sums stay
// in one binade (a run of 32 values a lane). gs[g] = the sum after group g.
template <typename T>
__device__ T first_chunk(const T *__restrict__ sv, int clen, int esc, T *__restrict__ gs) {
    using U = typename Bits<T>::U;
    constexpr U TOP = (U)1 << (Bits<T>::MB + 1);
    const int lane = threadIdx.x & 31;
    T p = T(0);
    GMap<T> run{0, 0};
    int run_be = 0;
    if (sizeof(T) == 8) {
        const int gl = max(0, min(32, clen - lane * 32));
        float es = 0.f;
#pragma unroll 4
        for (int q = 0; q < gl; q++) es += est_of(sv[lane * 33 + q], esc);
        float e = es;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const float o = __shfl_up_sync(0xffffffffu, e, off);
            if (lane >= off) e += o;
        }
        const int blo = est_exp((e - es) * 0.9990234375f, esc, T(0));
        if (blo > 0 && blo == est_exp(e * 1.0009765625f, esc, T(0))) {
            run_be = blo;
#pragma unroll 2
            for (int q = 0; q < gl; q++) run_add(run, sv[lane * 33 + q], blo);
        }
        __syncwarp();
        run = GMap<T>{min(run.a0, TOP), min(run.a1, TOP)};
    }
#pragma unroll 1
    for (int g = 0; g * 32 < clen; g++) {
        if (sizeof(T) == 8) {
            const int be = normal_exp(p);
            if (be > 0 && be == __shfl_sync(0xffffffffu, run_be, g)) {
                const U P = significand(p);
                const U Pn = P + __shfl_sync(0xffffffffu, (P & 1) ? run.a1 : run.a0, g);
                if (Pn < TOP) {
                    p = from_parts<T>(be, Pn);
                    if (lane == 0) gs[g] = p;
                    continue;
                }
            }
        }
        const int len = min(32, clen - g * 32);
        const T val = lane < len ? sv[staged(g * 32 + lane)] : T(0);
        int at = 0;
        if (sizeof(T) == 4 || g == 0) {
#pragma unroll 8
            for (; at < len; at++) p = kpp_add(p, __shfl_sync(0xffffffffu, val, at));
        }
        while (at < len) {
            const int be = normal_exp(p);
            if (be > 0) {
                const U S = group_states(val, lane >= at && lane < len, be, significand(p));
                const unsigned bad = __ballot_sync(0xffffffffu, S >= TOP);
                const int q = bad ? __ffs(bad) - 1 : 32;
                const U Sb = __shfl_sync(0xffffffffu, S, q > 0 ? q - 1 : 0);
                if (q > at) p = from_parts<T>(be, Sb);
                if (q >= len) break;
                at = q;
            }
            p = kpp_add(p, __shfl_sync(0xffffffffu, val, at));
            at++;
        }
        if (lane == 0) gs[g] = p;
    }
    return p;
}

inline size_t compose_smem(size_t elem) { return elem * KPP_WARPS * KPP_STAGED; }

// One CTA per (eight chunks, trial), one warp per chunk: the chunk's map for
// the binade its estimated sums lie in -- an integer sum over a value a lane,
// or, where exact halves occur, ordered runs of 32 a lane -- the group maps
// for both binades where the estimate says that the sum may change binade, and
// the first chunk exactly. The chunk's values are copied to shared memory
// first: read in the loops, each load's latency was exposed (700 cycles a
// value at n = 5,000).
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS)
    kpp_compose_kernel(const KppFit<T> *__restrict__ fits, const int2 *__restrict__ items, int scan, int c, bool init) {
    using U = typename Bits<T>::U;
    constexpr U OUT = (U)1 << (Bits<T>::MB + 1);
    const int2 it = item_at(items);
    const KppFit<T> &f = fits[it.x];
    const KppState *st = f.st;
    const int t = blockIdx.y;
    if (t >= (init ? 1 : f.trials) || (!init && st->direct[c & 1])) return;
    if (!init && !contends(f, c, t)) return;
    extern __shared__ __align__(16) unsigned char kpp_smem[];
    __shared__ float red[KPP_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    T *sv = reinterpret_cast<T *>(kpp_smem) + w * KPP_STAGED;
    const long long j = (long long)it.y * KPP_WARPS + w;
    const int wbuf = init ? 0 : 1 - st->cur;
    const T *v = f.chains + ((long long)wbuf * f.trials + t) * f.n + j * KPP_CH;
    const int clen = j < f.nch ? (int)min((long long)KPP_CH, f.n - j * KPP_CH) : 0;
#pragma unroll 8
    for (int i = lane; i < clen; i += 32) cp_async_one(sv + staged(i), v + i);
    const int tpc = KPP_CH / scan;  // tiles per chunk
    const float *cs = f.csum + (long long)t * f.tiles;
    const long long t0 = (long long)it.y * KPP_WARPS * tpc;  // the group's first tile
    float e = 0.f;
    for (long long q = tid; q < t0; q += KPP_THREADS) e += cs[q];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) red[w] = e;
    __syncthreads();
    if (j >= f.nch) return;
    float s = 0.f;  // this chunk's sum
    e = lane < KPP_WARPS ? red[lane] : 0.f;
    for (int q = lane; q < (w + 1) * tpc; q += 32) {
        const float x = t0 + q < f.tiles ? cs[t0 + q] : 0.f;
        if (q < w * tpc) e += x;
        else s += x;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        e += __shfl_xor_sync(0xffffffffu, e, o);
        s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    CMap<T> *cm = f.cmaps + (long long)t * f.nch + j;
    cp_async_wait_all();
    __syncwarp();
    CMap<T> m;
    m.s = GMap<T>{0, 0};
    m.elo = -1;
    m.kind = KIND_NONE;
    m.slot = 0;
    if (j == 0) {
        m.s.a0 = Bits<T>::bits(first_chunk<T>(sv, clen, init ? 0 : st->esc, f.gstates + ((long long)wbuf * f.trials + t) * 32));
        m.kind = KIND_END;
        if (lane == 0) *cm = m;
        return;
    }
    // The f32 estimate's own error and the drift of a sequential f32 fold (a
    // few 1e-5 at 10^6 values) lie inside the margins.
    const int esc = init ? 0 : st->esc;
    const int blo = est_exp(e * 0.9990234375f, esc, T(0));
    const int bhi = est_exp((e + s) * 1.0009765625f, esc, T(0));
    const int gl = max(0, min(32, clen - lane * 32));  // this lane's run
    if (blo == 0 || bhi == 0 || bhi - blo > 1) {
        if (lane == 0) *cm = m;
        return;
    }
    m.elo = blo;
    if (bhi > blo) {
        int slot = 0;
        if (lane == 0) slot = atomicAdd(f.nslots + t, 1);
        slot = __shfl_sync(0xffffffffu, slot, 0);
        if (slot < KPP_SLOTS) {
            GMap<T> g0{0, 0}, g1{0, 0};
#pragma unroll 2
            for (int q = 0; q < gl; q++) {
                const T x = sv[lane * 33 + q];
                run_add(g0, x, blo);
                run_add(g1, x, blo + 1);
            }
            GMap<T> *o = f.slots + ((long long)t * KPP_SLOTS + slot) * 64 + lane;
            o[0] = GMap<T>{min(g0.a0, OUT), min(g0.a1, OUT)};
            o[32] = GMap<T>{min(g1.a0, OUT), min(g1.a1, OUT)};
            m.kind = KIND_SLOT;
            m.slot = (short)slot;
        }
        if (lane == 0) *cm = m;
        return;
    }
    unsigned long long a = 0;  // at most 1024 increments of 2^53: no overflow
    bool tie = false;
#pragma unroll 4
    for (int i = lane; i < clen; i += 32) a += inc_of(sv[staged(i)], blo, tie);
    if (!__any_sync(0xffffffffu, tie)) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        m.s.a0 = m.s.a1 = (U)min(a, (unsigned long long)OUT);
    } else {
        GMap<T> g{0, 0};
#pragma unroll 2
        for (int q = 0; q < gl; q++) run_add(g, sv[lane * 33 + q], blo);
        __syncwarp();
        g = gscan(GMap<T>{min(g.a0, OUT), min(g.a1, OUT)});
        m.s = GMap<T>{min(g.a0, OUT), min(g.a1, OUT)};
    }
    m.kind = KIND_MAP;
    if (lane == 31) *cm = m;
}

// ------------------------------------------------- one fold by one CTA --
constexpr int KPP_ROUND = 4 * KPP_THREADS;  // chunk maps scanned at a time
static_assert(KPP_CH == 4 * KPP_THREADS && KPP_WARPS == 8, "a chunk is 32 groups, four a warp");

template <typename T>
struct WalkShared {
    unsigned long long pre[KPP_ROUND];     // prefix sums of the plain chunks' increments
    CMap<T> map[KPP_ROUND];
    unsigned long long gtot[32];
    unsigned special[32], words;           // chunks to look at one by one (words: the nonzero words)
    GMap<T> gm[32];
    T v[KPP_CH];                           // the values of a chunk walked by itself
    T pb;
    int f0, last;
};

// The values of one chunk (clen of them) added to p in order, exactly as the
// sequential fold, by the whole block: warp w holds groups 4 w .. 4 w + 3 of
// 32 values. Per pass, the groups' maps for p's binade, their scan (by every
// warp), and where the sum leaves the binade the group's own states and one
// exact F addition: two barriers a pass.
template <typename T>
__device__ T block_walk_chunk(T p, const T *__restrict__ cv, int clen, WalkShared<T> &sh) {
    using U = typename Bits<T>::U;
    constexpr U TOP = (U)1 << (Bits<T>::MB + 1);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    __syncthreads();  // the chunk before is done with sh.v
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int i = u * KPP_THREADS + tid;
        sh.v[i] = i < clen ? cv[i] : T(0);
    }
    __syncthreads();
    int start = 0;
#pragma unroll 1
    while (start < clen) {
        const int be = normal_exp(p);
        if (be == 0) {
            // a NaN sum stays; +inf stays until a NaN value; a zero sum until a
            // value other than zero; a subnormal sum takes the next value
            const bool inf = is_inf_or_nan(p);
            int first = INT32_MAX;
            if (p == p) {
#pragma unroll 1
                for (int u = 3; u >= 0; u--) {
                    const int i = (4 * w + u) * 32 + lane;
                    const T x = sh.v[i];
                    const bool hit = inf ? x != x : (p == T(0) ? !(x == T(0)) : true);
                    if (i >= start && i < clen && hit) first = i;
                }
            }
            first = __reduce_min_sync(0xffffffffu, first);
            __syncthreads();  // the pass before is done with sh.f0
            if (tid == 0) sh.f0 = INT32_MAX;
            __syncthreads();
            if (lane == 0 && first != INT32_MAX) atomicMin(&sh.f0, first);
            __syncthreads();
            const int f0 = min(sh.f0, clen);
            if (f0 == clen) return p;
            p = kpp_add(p, sh.v[f0]);
            start = f0 + 1;
            continue;
        }
#pragma unroll 2
        for (int u = 0; u < 4; u++) {
            const int i = (4 * w + u) * 32 + lane;
            const GMap<T> m = group_map(sh.v[i], i >= start && i < clen, be);
            if (lane == 0) sh.gm[4 * w + u] = m;
        }
        __syncthreads();
        const GMap<T> m = gscan(sh.gm[lane]);
        const U P = significand(p);
        const U Pl = P + ((P & 1) ? m.a1 : m.a0);  // after group `lane`
        const unsigned bad = __ballot_sync(0xffffffffu, Pl >= TOP);
        const int gf = bad ? __ffs(bad) - 1 : 32;
        if (gf == 32) return from_parts<T>(be, __shfl_sync(0xffffffffu, Pl, 31));
        const U before = __shfl_sync(0xffffffffu, Pl, gf > 0 ? gf - 1 : 0);
        const U Pg = gf > 0 ? before : P;
        if (w == gf >> 2) {
            const int i = gf * 32 + lane;
            const U S = group_states(sh.v[i], i >= start && i < clen, be, Pg);
            const int q = __ffs(__ballot_sync(0xffffffffu, S >= TOP)) - 1;  // the first value that leaves the binade
            const U Sb = __shfl_sync(0xffffffffu, S, q > 0 ? q - 1 : 0);
            if (lane == q) {
                sh.pb = from_parts<T>(be, q > 0 ? Sb : Pg);
                sh.f0 = gf * 32 + q;
            }
        }
        __syncthreads();
        p = kpp_add(sh.pb, sh.v[sh.f0]);  // the one exact addition where the binade changes
        start = sh.f0 + 1;
    }
    return p;
}

// A chunk with group maps added to p, by every warp alike (no barrier): the
// groups' maps for p's binade scanned, the group in which the sum leaves it by
// its own states and one exact F addition, the groups after it by their maps
// for the next binade. False where they do not apply.
template <typename T>
__device__ bool walk_slot_chunk(T &p, const T *__restrict__ cv, int clen, const GMap<T> *__restrict__ gm, int elo) {
    using U = typename Bits<T>::U;
    constexpr U TOP = (U)1 << (Bits<T>::MB + 1);
    const int lane = threadIdx.x & 31;
    const GMap<T> g0 = gm[lane], g1 = gm[32 + lane];
    int be = normal_exp(p);
    if (be != elo && be != elo + 1) return false;
    int done = 0;  // groups added
    T r = p;
    if (be == elo) {
        const U P = significand(r);
        const GMap<T> m = gscan(g0);
        const U Pl = P + ((P & 1) ? m.a1 : m.a0);
        const unsigned bad = __ballot_sync(0xffffffffu, Pl >= TOP);
        if (!bad) {
            p = from_parts<T>(be, __shfl_sync(0xffffffffu, Pl, 31));
            return true;
        }
        const int gf = __ffs(bad) - 1;
        const int i = gf * 32 + lane;
        const bool in = i < clen;
        const T val = in ? cv[i] : T(0);
        const U before = __shfl_sync(0xffffffffu, Pl, gf > 0 ? gf - 1 : 0);
        const U Pg = gf > 0 ? before : P;
        U S = group_states(val, in, be, Pg);
        const int q = __ffs(__ballot_sync(0xffffffffu, S >= TOP)) - 1;  // the first value that leaves the binade
        const U Sb = __shfl_sync(0xffffffffu, S, q > 0 ? q - 1 : 0);
        r = kpp_add(from_parts<T>(be, q > 0 ? Sb : Pg), __shfl_sync(0xffffffffu, val, q));
        be = normal_exp(r);
        if (be != elo + 1) return false;
        S = group_states(val, in && lane > q, be, significand(r));
        S = __shfl_sync(0xffffffffu, S, 31);
        if (S >= TOP) return false;
        r = from_parts<T>(be, S);
        done = gf + 1;
    }
    const U P = significand(r);
    const GMap<T> m = gscan(lane < done ? GMap<T>{0, 0} : g1);
    U Pl = P + ((P & 1) ? m.a1 : m.a0);
    Pl = __shfl_sync(0xffffffffu, Pl, 31);
    if (Pl >= TOP) return false;
    p = from_parts<T>(be, Pl);
    return true;
}

// The first value of a chunk whose inclusive running sum (from p) reaches thr,
// or -1, by one warp. gs: the running sums after the chunk's groups, where they
// are recorded (the first chunk): the group is found by them. Else the lanes'
// runs of 32 values give the groups' maps for p's binade.
template <typename T>
__device__ int warp_search_chunk(T p, const T *__restrict__ cv, int clen, T thr, const T *__restrict__ gs) {
    using U = typename Bits<T>::U;
    constexpr U TOP = (U)1 << (Bits<T>::MB + 1);
    const int lane = threadIdx.x & 31;
    const int ng = (clen + 31) / 32;
    int start = 0;  // the next group
    if (gs) {
        const T e = lane < ng ? __ldcg(gs + lane) : T(0);
        const unsigned m = __ballot_sync(0xffffffffu, lane < ng && !(e < thr));
        if (!m) return -1;
        start = __ffs(m) - 1;
        const T b = __shfl_sync(0xffffffffu, e, start > 0 ? start - 1 : 0);
        if (start > 0) p = b;
    }
    while (start < ng) {
        const int be = normal_exp(p);
        int gsel = start;
        if (be > 0 && !gs) {
            GMap<T> m{0, 0};
            if (lane >= start && lane < ng) {
                // this lane's run in order, from an even and from an odd sum
                const int gl = min(32, clen - lane * 32);
#pragma unroll 2
                for (int q = 0; q < gl; q++) {
                    run_add(m, cv[lane * 32 + q], be);
                }
                m.a0 = min(m.a0, TOP);
                m.a1 = min(m.a1, TOP);
            }
            __syncwarp();
            m = gscan(m);
            const U P = significand(p);
            const U Pl = P + ((P & 1) ? m.a1 : m.a0);
            const unsigned bad = __ballot_sync(0xffffffffu, lane >= start && lane < ng &&
                                                                (Pl >= TOP || from_parts<T>(be, Pl) >= thr));
            if (!bad) return -1;  // the chunk ends below thr
            gsel = __ffs(bad) - 1;
            const U Pb = __shfl_sync(0xffffffffu, Pl, gsel > 0 ? gsel - 1 : 0);
            if (gsel > start) p = from_parts<T>(be, Pb);
        }
        // group gsel value by value
        const int i0 = gsel * 32, len = min(32, clen - i0);
        const T val = lane < len ? cv[i0 + lane] : T(0);
        int at = 0;
        while (at < len) {
            const int b = normal_exp(p);
            if (b > 0) {
                const U S = group_states(val, lane >= at && lane < len, b, significand(p));
                const unsigned bad = __ballot_sync(0xffffffffu, S >= TOP);
                const int q = bad ? __ffs(bad) - 1 : len;
                const unsigned hm = __ballot_sync(0xffffffffu,
                                                  lane >= at && lane < q && from_parts<T>(b, S) >= thr);
                if (hm) return i0 + __ffs(hm) - 1;
                const U Sb = __shfl_sync(0xffffffffu, S, q > 0 ? q - 1 : 0);
                if (q > at) p = from_parts<T>(b, Sb);
                if (q >= len) break;
                at = q;
            }
            p = kpp_add(p, __shfl_sync(0xffffffffu, val, at));
            if (p >= thr) return i0 + at;
            at++;
        }
        start = gsel + 1;
    }
    return -1;
}

// The pending trials resolved into centre c (init: the first D^2 array), then
// the draws and candidates of centre c + 1 (init: 1), by one block. The folds'
// results come from this launch's other CTAs: read past L1.
template <typename T>
__device__ void kpp_select(const KppFit<T> &f, int c, bool init) {
    KppState *st = f.st;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int cn = init ? 1 : c + 1;
    const int ntr = f.trials, d = f.d;
    const long long n = f.n;
    __shared__ long long copy_row, direct_row;
    __shared__ long long draw0;
    __shared__ T stotal;
    __shared__ int scur, strial;
    if (tid < MAX_TRIALS) st->est[cn & 1][tid] = 0.0;
    if (tid == 0) st->err[cn & 1] = 0.0;
    if (tid == 0) {
        copy_row = direct_row = -1;
        if (init) {
            st->total = __ldcg(&st->pot[0]);
        } else if (!st->direct[c & 1]) {
            int best = 0;
            double bp = __ldcg(&st->pot[0]);
            for (int t = 1; t < ntr; t++) {
                const double v = __ldcg(&st->pot[t]);
                if (v < bp) {  // strictly smaller: the first trial wins ties
                    bp = v;
                    best = t;
                }
            }
            st->prev_trial = st->cur_trial;
            st->cur = 1 - st->cur;
            st->cur_trial = best;
            st->own_c = c;
            st->total = bp;
            copy_row = st->cand[best];
            f.crow[c] = (int32_t)copy_row;
        }
        scur = st->cur;
        strial = st->cur_trial;
        if (cn < f.k) {
            const T total = (T)st->total;
            stotal = total;
            long long cur = st->cursor;
            if (sizeof(T) == 8) {
                const unsigned long long b = (unsigned long long)__double_as_longlong(st->total);
                const int e = (int)((b >> 52) & 0x7FFull);
                st->esc = e > 0 && e < 0x7FF ? e - 1023 : 0;
            }
            // kmeans.rs:202-206: a uniform random row, the D^2 array unchanged
            if (f.nan_direct ? !(total > T(0)) : total <= T(0)) {
                direct_row = draw_to_range(draw_at(f, cur), n);
                f.crow[cn] = (int32_t)direct_row;
                st->direct[cn & 1] = 1;
                cur += 1;
            } else {
                st->direct[cn & 1] = 0;
                draw0 = cur;
                cur += ntr;
            }
            st->cursor = cur;
        }
    }
    __syncthreads();
    if (copy_row >= 0)
        for (int j = tid; j < d; j += KPP_THREADS) f.centers[(long long)c * d + j] = f.x[copy_row * d + j];
    if (cn >= f.k) return;
    if (direct_row >= 0) {
        for (int j = tid; j < d; j += KPP_THREADS) f.centers[(long long)cn * d + j] = f.x[direct_row * d + j];
        return;
    }
    // each trial's first row whose running sum reaches its threshold (kmeans.rs:215-223)
    const long long slice = (long long)scur * ntr + strial, nch = f.nch;
    const T *S = f.states + slice * nch;
    const T *v = f.chains + slice * n;
    for (int t = w; t < ntr; t += KPP_WARPS) {
        const T thr = kpp_mul((T)draw_at(f, draw0 + t), stotal);
        // First chunk whose end state is not below thr: a 32-ary search (the
        // states never decrease, and a NaN state stays NaN, so "not below"
        // holds from one chunk on); that chunk is then walked with the exact test.
        long long lo = 0, hi = nch;  // the answer lies in [lo, hi]; nch = none
        while (lo < hi) {
            const long long step = (hi - lo + 31) / 32;
            const long long pos = lo + (long long)lane * step;
            const unsigned m = __ballot_sync(0xffffffffu, pos < hi && !(__ldcg(S + pos) < thr));
            if (!m) {
                lo = lo + ((hi - 1 - lo) / step) * step + 1;  // past the last probe
            } else {
                const int q = __ffs(m) - 1;
                const long long pf = lo + (long long)q * step;
                if (q > 0) lo = lo + (long long)(q - 1) * step + 1;
                hi = pf;
            }
        }
        long long cand = n - 1;
        if (lo < nch) {
            const T p = lo > 0 ? __ldcg(S + lo - 1) : T(0);
            const int hit = warp_search_chunk<T>(p, v + lo * KPP_CH, (int)min((long long)KPP_CH, n - lo * KPP_CH), thr,
                                                 lo == 0 ? f.gstates + slice * 32 : nullptr);
            if (hit >= 0) cand = lo * KPP_CH + hit;
        }
        if (lane == 0) st->cand[t] = cand;
    }
}

// One CTA per (seeding, trial): the trial's fold over every chunk, the running
// sum recorded at each chunk's end; the seeding's last CTA selects.
//
// Latency bound. Per round of 1024 chunks one scan forms the prefix sums of
// the plain chunks' increments (one map, no exact half, the binade of the
// chunk before): a run of them is then one addition and one comparison. The
// others are looked at one by one: a chunk in which the sum changes binade
// (about one per binade) through its group maps; one whose maps do not apply is
// walked from its values.
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS) kpp_walk_kernel(const KppFit<T> *__restrict__ fits, int c, bool init) {
    using U = typename Bits<T>::U;
    constexpr U TOP = (U)1 << (Bits<T>::MB + 1);
    const KppFit<T> &f = fits[blockIdx.x];
    KppState *st = f.st;
    const int t = blockIdx.y, ntr = init ? 1 : f.trials;
    if (t >= ntr) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    __shared__ WalkShared<T> sh;
    if (!init && st->direct[c & 1]) {
        // no trials to fold: the next centre's draws only
        if (t == 0) kpp_select<T>(f, c, false);
        return;
    }
    const int wbuf = init ? 0 : 1 - st->cur;
    const long long slice = (long long)wbuf * f.trials + t, nch = f.nch, n = f.n;
    const T *v = f.chains + slice * n;
    const CMap<T> *cm = f.cmaps + (long long)t * nch;
    T *sout = f.states + slice * nch;
    T p = T(0);
    const bool contender = init || contends(f, c, t);
    for (long long jb = 0; contender && jb < nch; jb += KPP_ROUND) {
        const int nb = (int)min((long long)KPP_ROUND, nch - jb);
        __syncthreads();  // the round before is done with sh
#pragma unroll 2
        for (int u = 0; u < 4; u++) {
            const int i = (4 * w + u) * 32 + lane;
            CMap<T> m;
            m.elo = -1;
            m.kind = KIND_NONE;
            if (i < nb) m = cm[jb + i];
            sh.map[i] = m;
            int before = __shfl_up_sync(0xffffffffu, m.elo, 1);
            if (lane == 0) before = i > 0 && i < nb ? cm[jb + i - 1].elo : -1;
            const bool plain = m.kind == KIND_MAP && m.s.a0 == m.s.a1 && before == m.elo;
            const unsigned sp = __ballot_sync(0xffffffffu, !plain && i < nb);
            if (lane == 0) sh.special[4 * w + u] = sp;
            unsigned long long a = plain ? (unsigned long long)m.s.a0 : 0ull;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned long long o = __shfl_up_sync(0xffffffffu, a, off);
                if (lane >= off) a += o;
            }
            sh.pre[i] = a;
            if (lane == 31) sh.gtot[4 * w + u] = a;
        }
        __syncthreads();
        {
            unsigned long long g = sh.gtot[lane];
            const unsigned long long own = g;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned long long o = __shfl_up_sync(0xffffffffu, g, off);
                if (lane >= off) g += o;
            }
            g -= own;  // the groups before
#pragma unroll
            for (int u = 0; u < 4; u++) sh.pre[(4 * w + u) * 32 + lane] += __shfl_sync(0xffffffffu, g, 4 * w + u);
            const unsigned nz = __ballot_sync(0xffffffffu, sh.special[lane] != 0);
            if (tid == 0) sh.words = nz;
        }
        __syncthreads();
        int i = 0;
        while (i < nb) {  // block-uniform
            const int be = normal_exp(p);
            const U P = be > 0 ? significand(p) : (U)0;
            const int wd = i >> 5;
            unsigned rest = sh.special[wd] >> (i & 31);
            int s;  // the next chunk to look at by itself
            if (rest) {
                s = i + __ffs(rest) - 1;
            } else {
                const unsigned later = wd < 31 ? sh.words >> (wd + 1) << (wd + 1) : 0u;
                const int q = later ? __ffs(later) - 1 : 32;
                s = q < 32 ? q * 32 + __ffs(sh.special[q]) - 1 : nb;
            }
            bool slow = true;
            if (s > i) {
                if (be > 0 && sh.map[i].elo == be) {
                    const unsigned long long base = i > 0 ? sh.pre[i - 1] : 0ull;
                    int e = s;
                    if ((unsigned long long)P + (sh.pre[s - 1] - base) >= (unsigned long long)TOP) {
                        int lo = i, hi = s - 1;  // the first chunk whose end leaves the binade
                        while (lo < hi) {
                            const int mid = (lo + hi) >> 1;
                            if ((unsigned long long)P + (sh.pre[mid] - base) >= (unsigned long long)TOP) hi = mid;
                            else lo = mid + 1;
                        }
                        e = lo;
                    }
                    for (int q = i + tid; q < e; q += KPP_THREADS)
                        sout[jb + q] = from_parts<T>(be, (U)(P + (sh.pre[q] - base)));
                    if (e > i) p = from_parts<T>(be, (U)(P + (sh.pre[e - 1] - base)));
                    slow = e < s;
                    i = e;
                }
            } else {
                const CMap<T> &m = sh.map[i];
                if (m.kind == KIND_END) {
                    p = Bits<T>::from(m.s.a0);
                    slow = false;
                } else if (m.kind == KIND_MAP && be > 0 && be == m.elo) {
                    const U Pn = P + ((P & 1) ? m.s.a1 : m.s.a0);
                    if (Pn < TOP) {
                        p = from_parts<T>(be, Pn);
                        slow = false;
                    }
                } else if (m.kind == KIND_SLOT) {
                    const long long j = jb + i;
                    slow = !walk_slot_chunk<T>(p, v + j * KPP_CH, (int)min((long long)KPP_CH, n - j * KPP_CH),
                                               f.slots + ((long long)t * KPP_SLOTS + m.slot) * 64, m.elo);
                }
                if (!slow) {
                    if (tid == 0) sout[jb + i] = p;
                    i++;
                }
            }
            if (slow) {
                const long long j = jb + i;
                p = block_walk_chunk<T>(p, v + j * KPP_CH, (int)min((long long)KPP_CH, n - j * KPP_CH), sh);
                if (tid == 0) sout[j] = p;
                i++;
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        st->pot[t] = contender ? (double)p : (double)INFINITY;
        f.nslots[t] = 0;
        __threadfence();  // the block's states and the potential, before the count
        sh.last = atomicAdd(&st->done, 1) == ntr - 1;
        if (sh.last) st->done = 0;
        __threadfence();
    }
    __syncthreads();
    if (sh.last) kpp_select<T>(f, c, init);
}

// ---------------------------------------------------- small seedings --
// F = f32 with at most SMALL_N rows, SMALL_D features and SMALL_ND values: a seeding is one CTA's, its
// D^2 arrays in shared memory (slot `cur` and one for each trial), every centre in one
// launch. A fold of 1,024 f32 values is 4,096 cycles: a thread per trial walks its
// array value by value and records the running sum after every 32, which is where the
// next candidates are found. Four launches a centre took 30 to 60 us, this 3.4 (100 x 4)
// to 49 (300 seedings of 1,000 x 64, k = 40; the four 73). Above SMALL_ND values the one CTA
// is slower than the four launches where the seedings are few (1,000 x 128, k = 40 58 us
// for 45).
constexpr int SMALL_N = 1024, SMALL_D = 256, SMALL_ND = 65536;
// (4 floats past a multiple of 32: the folds of eight trials meet no bank conflict)
__host__ __device__ inline int small_stride(int n) { return (n + 31) / 32 * 32 + 4; }
inline size_t small_smem(int n, int d, int trials) {
    return sizeof(float) * ((size_t)(trials + 1) * (small_stride(n) + 32) + (size_t)trials * ((d + 3) & ~3));
}

__global__ void __launch_bounds__(KPP_THREADS) kpp_small_kernel(const KppFit<float> *__restrict__ fits) {
    const KppFit<float> f = fits[blockIdx.x];
    const int n = (int)f.n, d = f.d, ntr = f.trials, stride = small_stride(n), ng = (n + 31) / 32, dc = (d + 3) & ~3;
    const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(f.x) & 15) == 0;
    extern __shared__ __align__(16) float small_sm[];
    float *const arr = small_sm;                     // [ntr + 1][stride] D^2 arrays
    float *const gs = arr + (ntr + 1) * stride;      // [ntr + 1][32] running sums after each 32 values
    float *const crow = gs + (ntr + 1) * 32;         // [ntr][dc] candidate rows (at 16 bytes)
    __shared__ float pot[MAX_TRIALS + 1];
    __shared__ int cand[MAX_TRIALS];
    __shared__ int best_sh;
    const int tid = threadIdx.x;
    // slot of trial t beside the current array's
    auto slot = [](int t, int cur) { return t + (t >= cur ? 1 : 0); };
    auto fold = [&](int sl) {  // one thread: the sequential sum of a slot
        const float *v = arr + sl * stride;
        float p = 0.f;
        for (int g = 0; g < ng; g++) {
            const int len = min(32, n - 32 * g);
            if (len == 32) {
#pragma unroll
                for (int i = 0; i < 32; i++) p = __fadd_rn(p, v[32 * g + i]);
            } else {
                for (int i = 0; i < len; i++) p = __fadd_rn(p, v[32 * g + i]);
            }
            gs[sl * 32 + g] = p;
        }
        pot[sl] = p;
    };
    long long cursor = 1;
    int cur = 0;
    const long long first = draw_to_range(draw_at(f, 0), n);
    for (int j = tid; j < d; j += KPP_THREADS) {
        const float v = f.x[first * d + j];
        f.centers[j] = v;
        crow[j] = v;
    }
    __syncthreads();
    if (f.k > 1) {
        for (int i = tid; i < n; i += KPP_THREADS) {
            const float *xr = f.x + (int64_t)i * d;
            float acc = 0.f;
#pragma unroll 8
            for (int j = 0; j < d; j++) {
                const float t = __fsub_rn(xr[j], crow[j]);
                acc = __fadd_rn(acc, __fmul_rn(t, t));
            }
            arr[i] = acc;
        }
        __syncthreads();
        if (tid == 0) fold(0);
        __syncthreads();
    }
    for (int c = 1; c < f.k; c++) {
        const float total = pot[cur];
        if (f.nan_direct ? !(total > 0.f) : total <= 0.f) {  // kmeans.rs:202-206: a uniform random row, D^2 unchanged
            const long long r = draw_to_range(draw_at(f, cursor), n);
            cursor += 1;
            for (int j = tid; j < d; j += KPP_THREADS) f.centers[(long long)c * d + j] = f.x[r * d + j];
            continue;
        }
        if (tid < ntr) {  // the first row whose running sum reaches the threshold (kmeans.rs:213-223)
            const float thr = kpp_mul((float)draw_at(f, cursor + tid), total);
            const float *v = arr + cur * stride, *s = gs + cur * 32;
            int g = 0;
            while (g < ng && s[g] < thr) g++;  // (a NaN sum is not below: the values decide)
            int at = n - 1;
            if (g < ng) {
                float p = g > 0 ? s[g - 1] : 0.f;
                for (int i = 32 * g; i < n; i++) {
                    p = __fadd_rn(p, v[i]);
                    if (p >= thr) {
                        at = i;
                        break;
                    }
                }
            }
            cand[tid] = at;
        }
        cursor += ntr;
        __syncthreads();
        for (int e = tid; e < ntr * d; e += KPP_THREADS) crow[e / d * dc + e % d] = f.x[(int64_t)cand[e / d] * d + e % d];
        __syncthreads();
        for (int i = tid; i < n; i += KPP_THREADS) {
            const float *xr = f.x + (int64_t)i * d;
            const float m = arr[cur * stride + i];
            for (int t0 = 0; t0 < ntr; t0 += 4) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                const float *cr[4];
#pragma unroll
                for (int u = 0; u < 4; u++) cr[u] = crow + min(t0 + u, ntr - 1) * dc;
                if (vec) {
#pragma unroll 4
                    for (int q = 0; q < d / 4; q++) {
                        const float4 xv = reinterpret_cast<const float4 *>(xr)[q];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const float4 cv = *reinterpret_cast<const float4 *>(cr[u] + 4 * q);
                            const float t1 = __fsub_rn(xv.x, cv.x), t2 = __fsub_rn(xv.y, cv.y);
                            const float t3 = __fsub_rn(xv.z, cv.z), t4 = __fsub_rn(xv.w, cv.w);
                            acc[u] = __fadd_rn(acc[u], __fmul_rn(t1, t1));
                            acc[u] = __fadd_rn(acc[u], __fmul_rn(t2, t2));
                            acc[u] = __fadd_rn(acc[u], __fmul_rn(t3, t3));
                            acc[u] = __fadd_rn(acc[u], __fmul_rn(t4, t4));
                        }
                    }
                } else {
#pragma unroll 4
                    for (int j = 0; j < d; j++) {
                        const float xv = xr[j];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const float t = __fsub_rn(xv, cr[u][j]);
                            acc[u] = __fadd_rn(acc[u], __fmul_rn(t, t));
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (t0 + u < ntr) arr[slot(t0 + u, cur) * stride + i] = acc[u] < m ? acc[u] : m;  // kmeans.rs:230-232
            }
        }
        __syncthreads();
        if (tid < ntr) fold(slot(tid, cur));
        __syncthreads();
        if (tid == 0) {
            int best = 0;
            for (int t = 1; t < ntr; t++)
                if (pot[slot(t, cur)] < pot[slot(best, cur)]) best = t;  // the first trial wins ties (kmeans.rs:239-243)
            best_sh = best;
        }
        __syncthreads();
        const int best = best_sh;
        for (int j = tid; j < d; j += KPP_THREADS) f.centers[(long long)c * d + j] = crow[best * dc + j];
        cur = slot(best, cur);
        __syncthreads();  // crow and best_sh are rewritten
    }
    if (tid == 0) f.st->cursor = cursor;
}

template <typename T, int TT, int PASS>
void launch_trials(const KppFit<T> *fits, const int2 *items, unsigned grid, int scan, int c, int dmax,
                   cudaStream_t s) {
    const size_t smem = trial_smem(dmax, TT);
    FK_CUDA(cudaFuncSetAttribute((const void *)kpp_trials_kernel<T, TT, PASS>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kpp_trials_kernel<T, TT, PASS><<<grid, KPP_THREADS, smem, s>>>(fits, items, scan, c);
    FK_LAUNCH_CHECK();
}

// The trial pass with the smallest trial-slot count that holds ntr trials.
template <typename T, int PASS>
void launch_trials_any(int ntr, const KppFit<T> *fits, const int2 *items, unsigned grid, int scan, int c, int dmax,
                       cudaStream_t s) {
    switch (ntr) {
        case 1: case 2: launch_trials<T, 2, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 3: launch_trials<T, 3, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 4: launch_trials<T, 4, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 5: launch_trials<T, 5, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 6: launch_trials<T, 6, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 7: launch_trials<T, 7, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 8: launch_trials<T, 8, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 9: launch_trials<T, 9, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 10: launch_trials<T, 10, PASS>(fits, items, grid, scan, c, dmax, s); break;
        case 11: case 12: launch_trials<T, 12, PASS>(fits, items, grid, scan, c, dmax, s); break;
        default: launch_trials<T, 16, PASS>(fits, items, grid, scan, c, dmax, s); break;
    }
}

// Byte layout of one seeding's workspace (256-byte aligned parts).
struct KppLayout {
    size_t chains, states, gstates, slots, nslots, cmaps, csum, thr, own, closer, crow, st, total;
};
template <typename T>
KppLayout kpp_layout(const KppJob &j, int trials, int scan) {
    const size_t n = (size_t)j.n, nch = (n + KPP_CH - 1) / KPP_CH, tiles = (n + scan - 1) / scan;
    KppLayout L{};
    size_t at = 0;
    auto part = [&](size_t bytes) {
        const size_t p = at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    L.chains = part(sizeof(T) * 2 * trials * n);
    L.states = part(sizeof(T) * 2 * trials * nch);
    L.gstates = part(sizeof(T) * 2 * trials * 32);
    L.slots = part(sizeof(GMap<T>) * trials * KPP_SLOTS * 2 * 32);
    L.nslots = part(sizeof(int) * trials);
    L.cmaps = part(sizeof(CMap<T>) * trials * nch);
    L.csum = part(sizeof(float) * trials * tiles);
    L.thr = part(sizeof(T) * (size_t)j.k);
    L.own = part(sizeof(int32_t) * n);
    L.closer = part(sizeof(T) == 8 ? sizeof(unsigned short) * n : 0);
    L.crow = part(sizeof(int32_t) * (size_t)j.k);
    L.st = part(sizeof(KppState));
    L.total = at;
    return L;
}

// Seedings [lo, hi) of the order (largest k first) together; false when their
// workspace cannot be allocated and there are several.
template <typename T>
bool run_group(Ctx &ctx, const std::vector<KppJob> &jobs, const std::vector<int> &order, size_t lo, size_t hi, int scan,
               int64_t *draws_used) {
    cudaStream_t s = ctx.stream;
    const size_t nf = hi - lo;
    std::vector<KppFit<T>> fits(nf);
    std::vector<size_t> off(nf);
    size_t bytes = 0;
    int dmax = 0, tmax = 1;
    for (size_t q = 0; q < nf; q++) {
        const KppJob &j = jobs[(size_t)order[lo + q]];
        off[q] = bytes;
        bytes += kpp_layout<T>(j, kpp_trials_host(j.k), scan).total;
        dmax = std::max(dmax, j.d);
        tmax = std::max(tmax, kpp_trials_host(j.k));
    }
    unsigned char *ws;
    try {
        ws = (unsigned char *)ctx.get(BUF_KPP1, bytes);
    } catch (const Error &e) {
        if (e.code != FK_ERR_OOM || nf == 1) throw;
        return false;
    }
    // items of the trial pass (tiles) and of the composition (eight chunks), in
    // seeding order: the seedings still running at a step are a prefix
    std::vector<int2> items;
    std::vector<unsigned> tile_end(nf), comp_end(nf), cont_end(nf);
    unsigned nt = 0, ncg = 0, ncp = 0;
    long long rows = 0;
    for (size_t q = 0; q < nf; q++) rows += jobs[(size_t)order[lo + q]].n;
    const int per = rows >= 2ll * CONT_ROWS * ctx.num_sms ? CONT_ROWS : CONT_ROWS / 2;
    for (size_t q = 0; q < nf; q++) {
        const KppJob &j = jobs[(size_t)order[lo + q]];
        KppFit<T> &f = fits[q];
        const KppLayout L = kpp_layout<T>(j, kpp_trials_host(j.k), scan);
        unsigned char *b = ws + off[q];
        f.x = (const T *)j.x;
        f.x32 = sizeof(T) == 8 ? j.x32 : (const float *)j.x;
        f.xerr = sizeof(T) == 8 ? j.xerr : nullptr;
        f.draws = j.draws;
        f.centers = (T *)j.centers;
        f.chains = (T *)(b + L.chains);
        f.states = (T *)(b + L.states);
        f.cmaps = (CMap<T> *)(b + L.cmaps);
        f.gstates = (T *)(b + L.gstates);
        f.slots = (GMap<T> *)(b + L.slots);
        f.nslots = (int *)(b + L.nslots);
        f.csum = (float *)(b + L.csum);
        f.thr = (T *)(b + L.thr);
        f.own = (int32_t *)(b + L.own);
        f.closer = (unsigned short *)(b + L.closer);
        f.crow = (int32_t *)(b + L.crow);
        f.st = (KppState *)(b + L.st);
        f.n = j.n;
        f.nch = (j.n + KPP_CH - 1) / KPP_CH;
        f.tiles = (j.n + scan - 1) / scan;
        f.n_draws = j.n_draws;
        f.seed = j.seed;
        f.d = j.d;
        f.k = j.k;
        f.trials = kpp_trials_host(j.k);
        f.nan_direct = j.nan_direct ? 1 : 0;
        nt += (unsigned)f.tiles;
        ncg += (unsigned)((f.nch + KPP_WARPS - 1) / KPP_WARPS);
        ncp += (unsigned)((j.n + per - 1) / per);
        cont_end[q] = ncp;
        tile_end[q] = nt;
        comp_end[q] = ncg;
    }
    KppFit<T> *dfits = (KppFit<T> *)ctx.get(BUF_KPP0, sizeof(KppFit<T>) * nf);
    FK_CUDA(cudaMemcpyAsync(dfits, fits.data(), sizeof(KppFit<T>) * nf, cudaMemcpyHostToDevice, s));
    const int2 *titems = nullptr, *citems = nullptr, *pitems = nullptr;
    if (nf > 1) {
        items.reserve((size_t)nt + ncg + ncp);
        for (size_t q = 0; q < nf; q++)
            for (int t = 0; t < (int)fits[q].tiles; t++) items.push_back(make_int2((int)q, t));
        for (size_t q = 0; q < nf; q++)
            for (long long t = 0; t * KPP_WARPS < fits[q].nch; t++) items.push_back(make_int2((int)q, (int)t));
        for (size_t q = 0; q < nf; q++)
            for (long long t = 0; t * per < fits[q].n; t++) items.push_back(make_int2((int)q, (int)t));
        int2 *di = (int2 *)ctx.get(BUF_KPP2, sizeof(int2) * items.size());
        FK_CUDA(cudaMemcpyAsync(di, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, s));
        titems = di;
        citems = di + nt;
        pitems = citems + ncg;
    }
    FK_CUDA(cudaFuncSetAttribute((const void *)kpp_compose_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)compose_smem(sizeof(T))));
    kpp_first_kernel<T><<<(unsigned)nf, 128, 0, s>>>(dfits);
    FK_LAUNCH_CHECK();
    for (int c = 0;; c++) {
        // the seedings with a centre c to choose (c = 0: those with a second
        // centre form the first D^2 array)
        size_t na = 0;
        while (na < nf && fits[na].k > std::max(c, 1)) na++;
        if (na == 0) break;
        const bool init = c == 0;
        int nt_step = 1;
        for (size_t q = 0; q < na; q++) nt_step = std::max(nt_step, fits[q].trials);
        if (init) {
            launch_trials<T, 1, PASS_INIT>(dfits, titems, tile_end[na - 1], scan, c, dmax, s);
        } else {
            kpp_pairs_kernel<T><<<(unsigned)(na * ((c + KPP_WARPS - 1) / KPP_WARPS)), KPP_THREADS, 0, s>>>(dfits, c);
            FK_LAUNCH_CHECK();
            bool split = false;
            if constexpr (sizeof(T) == 8) {
                split = (long long)tile_end[na - 1] * scan >= KPP_SPLIT_ROWS;
                if (split) {
                    launch_trials_any<T, PASS_EST>(nt_step, dfits, titems, tile_end[na - 1], scan, c, dmax, s);
                    kpp_contenders_kernel<T><<<cont_end[na - 1], KPP_THREADS, 0, s>>>(dfits, pitems, scan, per, c);
                    FK_LAUNCH_CHECK();
                }
            }
            if (!split) launch_trials_any<T, PASS_ALL>(nt_step, dfits, titems, tile_end[na - 1], scan, c, dmax, s);
        }
        const unsigned gy = init ? 1u : (unsigned)nt_step;
        kpp_compose_kernel<T><<<dim3(comp_end[na - 1], gy), KPP_THREADS, compose_smem(sizeof(T)), s>>>(dfits, citems,
                                                                                                     scan, c, init);
        FK_LAUNCH_CHECK();
        kpp_walk_kernel<T><<<dim3((unsigned)na, gy), KPP_THREADS, 0, s>>>(dfits, c, init);
        FK_LAUNCH_CHECK();
    }
    // the descriptors above are host stack memory, and the draws are read back
    std::vector<long long> cur(nf);
    if (draws_used)
        for (size_t q = 0; q < nf; q++)
            FK_CUDA(cudaMemcpyAsync(&cur[q], &fits[q].st->cursor, sizeof(long long), cudaMemcpyDeviceToHost, s));
    FK_CUDA(cudaStreamSynchronize(s));
    if (draws_used)
        for (size_t q = 0; q < nf; q++) draws_used[order[lo + q]] = (int64_t)cur[q];
    return true;
}

// Every seeding in one launch.
void run_small(Ctx &ctx, const std::vector<KppJob> &jobs, int64_t *draws_used) {
    cudaStream_t s = ctx.stream;
    const size_t nf = jobs.size();
    std::vector<KppFit<float>> fits(nf);
    KppState *st = (KppState *)ctx.get(BUF_KPP1, sizeof(KppState) * nf);
    size_t smem = 0;
    for (size_t q = 0; q < nf; q++) {
        const KppJob &j = jobs[q];
        KppFit<float> &f = fits[q];
        f = KppFit<float>{};
        f.x = (const float *)j.x;
        f.draws = j.draws;
        f.centers = (float *)j.centers;
        f.st = st + q;
        f.n = j.n;
        f.n_draws = j.n_draws;
        f.seed = j.seed;
        f.d = j.d;
        f.k = j.k;
        f.trials = kpp_trials_host(j.k);
        f.nan_direct = j.nan_direct ? 1 : 0;
        smem = std::max(smem, small_smem((int)j.n, j.d, f.trials));
    }
    KppFit<float> *dfits = (KppFit<float> *)ctx.get(BUF_KPP0, sizeof(KppFit<float>) * nf);
    FK_CUDA(cudaMemcpyAsync(dfits, fits.data(), sizeof(KppFit<float>) * nf, cudaMemcpyHostToDevice, s));
    FK_CUDA(cudaFuncSetAttribute((const void *)kpp_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kpp_small_kernel<<<(unsigned)nf, KPP_THREADS, smem, s>>>(dfits);
    FK_LAUNCH_CHECK();
    std::vector<KppState> hs(draws_used ? nf : 0);
    if (draws_used) FK_CUDA(cudaMemcpyAsync(hs.data(), st, sizeof(KppState) * nf, cudaMemcpyDeviceToHost, s));
    FK_CUDA(cudaStreamSynchronize(s));
    for (size_t q = 0; q < hs.size(); q++) draws_used[q] = (int64_t)hs[q].cursor;
}

// A group that does not fit in memory runs as two halves.
template <typename T>
void run_split(Ctx &ctx, const std::vector<KppJob> &jobs, const std::vector<int> &order, size_t lo, size_t hi, int scan,
               int64_t *draws_used) {
    if (run_group<T>(ctx, jobs, order, lo, hi, scan, draws_used)) return;
    run_split<T>(ctx, jobs, order, lo, (lo + hi) / 2, scan, draws_used);
    run_split<T>(ctx, jobs, order, (lo + hi) / 2, hi, scan, draws_used);
}

}  // namespace

// Seedings run together while their workspaces stay within this many bytes
// (one larger seeding runs alone, and each one where memory is short).
constexpr size_t KPP_GROUP_BYTES = (size_t)6 << 30;

template <typename T>
void run_kmeanspp(Ctx &ctx, std::vector<KppJob> &jobs, int64_t *draws_used) {
    if (jobs.empty()) return;
    struct Seeding {
        Ctx &c;
        explicit Seeding(Ctx &ctx) : c(ctx) { c.seeding = true; }
        ~Seeding() { c.seeding = false; }
    } use(ctx);
    if (jobs.size() > 1) ctx.spared = true;
    const size_t group_bytes = ctx.lean ? 0 : KPP_GROUP_BYTES;
    long long rows = 0;
    for (const KppJob &j : jobs) {
        const int trials = kpp_trials_host(j.k);
        if (trials > MAX_TRIALS) {
            set_error("k-means++ with k=%d needs %d trials (max %d)", j.k, trials, MAX_TRIALS);
            fail(FK_ERR_UNSUPPORTED);
        }
        rows += j.n;
    }
    if constexpr (std::is_same<T, float>::value) {
        bool small = true;
        for (const KppJob &j : jobs) small = small && j.n <= SMALL_N && j.d <= SMALL_D && j.n * j.d <= SMALL_ND;
        if (small) return run_small(ctx, jobs, draws_used);
    }
    if constexpr (std::is_same<T, double>::value) {
        // f32 copies and rounding-error norms for the FP32 bounds (the f64
        // callers' seedings are restarts on one matrix)
        const KppJob &j0 = jobs[0];
        if (j0.k > 1) {
            float *x32 = (float *)ctx.get(BUF_PF_X32, sizeof(float) * (size_t)j0.n * j0.d);
            float *xerr = (float *)ctx.get(BUF_PF_XERR, sizeof(float) * (size_t)j0.n);
            launch_f32_copy(ctx, (const double *)j0.x, j0.n, j0.d, x32, xerr);
            for (KppJob &j : jobs) {
                j.x32 = x32;
                j.xerr = xerr;
            }
        }
    }
    // Rows per trial-pass tile: 1024 (most room to gather listed rows into full
    // warps), 256 while the larger tiles would leave SMs without one.
    const int scan = rows / KPP_CH >= 4 * ctx.num_sms ? KPP_CH : KPP_THREADS;
    std::vector<int> order(jobs.size());
    for (size_t q = 0; q < jobs.size(); q++) order[q] = (int)q;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return jobs[(size_t)a].k > jobs[(size_t)b].k; });
    size_t lo = 0, bytes = 0;
    for (size_t q = 0; q <= order.size(); q++) {
        const size_t add = q < order.size()
                               ? kpp_layout<T>(jobs[(size_t)order[q]], kpp_trials_host(jobs[(size_t)order[q]].k), scan).total
                               : 0;
        // (blockIdx.x counts the group's seedings too: far below its limit)
        if (q > lo && (q == order.size() || bytes + add > group_bytes)) {
            run_split<T>(ctx, jobs, order, lo, q, scan, draws_used);
            lo = q;
            bytes = 0;
        }
        bytes += add;
    }
}

template void run_kmeanspp<double>(Ctx &, std::vector<KppJob> &, int64_t *);
template void run_kmeanspp<float>(Ctx &, std::vector<KppJob> &, int64_t *);

}  // namespace fk
