// fk_prune.cu -- the plain assignment of a fit, with the centres that cannot
// win left out.
//
// The labels are nearest_center's (kmeans.rs:295-309), bit for bit: F
// direct-form distances (squared_euclidean, :159-163), strict < from F::MAX,
// the lowest index on ties. What is left out is proven to lose. Per row a fit
// keeps ub >= d(x, c_label) and lb <= d(x, c) for every other centre (true
// distances, f32 rounded outwards). In the next iteration the centres have
// moved by at most their shifts, so ub + shift(label) and lb - max shift of the
// others bound the new distances, and
//
//   prune_bound_kernel  keeps the label of a row whose bounds still separate
//                       (u (1 + 4 g) < l, g the relative rounding of a direct
//                       form: the F value to the label is then strictly the
//                       smallest) and lists the others:
//   prune_near_kernel   a row whose label's centre has at most NEAR centres
//                       within twice its distance: every other centre c has
//                       d(x, c) >= d(c_label, c) - d(x, c_label) > d(x, c_label)
//                       (triangle inequality, with room for every rounding), so
//                       the label's centre and those few are compared;
//   prune_scan_kernel   any other row, against every centre; the first
//                       iteration's pass, over all rows.
//
// Each leaves the row's new bounds. In f32 the distances are F's own. In f64
// they are formed in FP32 from f32 copies with rigorous bounds (fk_prefilter.cu)
// and rows whose intervals overlap, or are not finite, go to the FP64 direct
// form over every centre. The inertia needs each row's distance to its label
// once, for the assignment that the fit keeps.
//
// n = 1M, d = 64, k = 256 in f32, 100 iterations from k-means++: every centre
// for every row 1.92 ms an iteration, bound by the FP32 pipe; here 0.15 ms in
// the mean (62 us for every centre's pass, its first 2.0 ms included, 43 near
// centres, 26 their lists, 18 the bounds). n = 333,337, d = 50, k = 200 in f64:
// 0.81 ms with its filter and label distances, now 0.20 ms.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "fk_internal.cuh"

namespace fk {
namespace {

constexpr int NEAR = 16;          // neighbours of a centre that a row may be compared with
constexpr int NROW = NEAR + 1;    // thresholds kept per centre: the neighbours', and the first left out
constexpr int BU = 4;             // rows a thread of the bound pass takes at a time
constexpr int PT = 256;           // threads per block
constexpr float TINY = 1e-20f;    // distances below this: underflow in the squares

// Relative rounding of a direct form over d features, in f32 (F = f64 is far inside).
__device__ __forceinline__ float fold_rel(int d) { return (float)(d + 8) * 1.2e-7f; }

// Upper / lower bound of a true distance from bounds of its square.
__device__ __forceinline__ float dist_up(float sq) { return __fadd_ru(__fsqrt_ru(sq), TINY); }
__device__ __forceinline__ float dist_down(float sq) {
    return sq > 0.f ? fmaxf(__fsub_rd(__fsqrt_rd(sq), TINY), 0.f) : 0.f;
}

template <typename F>
__device__ __forceinline__ float abs_diff_up(F a, F b);
template <>
__device__ __forceinline__ float abs_diff_up(float a, float b) {
    return fmaxf(fabsf(__fsub_ru(a, b)), fabsf(__fsub_rd(a, b)));
}
template <>
__device__ __forceinline__ float abs_diff_up(double a, double b) {
    return __double2float_ru(fmax(fabs(__dsub_ru(a, b)), fabs(__dsub_rd(a, b))));
}

// Upper bound of each centre's shift (one warp per centre; +inf when not finite).
template <typename F>
__global__ void prune_shift_kernel(const F *__restrict__ c, const F *__restrict__ prev, int k, int d,
                                   float *__restrict__ shift) {
    const int lane = threadIdx.x & 31;
    const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (q >= k) return;
    float s = 0.f;
    for (int j = lane; j < d; j += 32) {
        const float t = abs_diff_up<F>(c[(int64_t)q * d + j], prev[(int64_t)q * d + j]);
        s = __fadd_ru(s, __fmul_ru(t, t));
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s = __fadd_ru(s, __shfl_xor_sync(0xffffffffu, s, o));
    if (lane == 0) {
        // an exact zero shift stays zero (TINY covers squares that underflow)
        const float t = s == 0.f ? 0.f : dist_up(s);
        shift[q] = t < INFINITY ? t : INFINITY;
    }
}

// The NROW nearest other centres of each centre (A centres per block): row
// thresholds in ascending order -- a row of this centre at computed squared
// distance m < threshold cannot be nearer to, or as near as, that neighbour --
// and the neighbours' indices. As in fk_kpp.cu: L a lower bound of D(c, q),
// threshold = L (1 - rho) / 4, rho = (d + 8) 1e-6, which exceeds every rounding
// of the two direct forms; bounds below 1e-30, where underflow would count, and
// NaN give 0 (always compared).
//
// G lanes take a centre q (one up to 16 features, else eight): each reads its
// features of q once for all A centres, and the lanes share the A thresholds.
// Every lane of a group forming each centre's threshold, and one warp selecting
// from all of them (or k ranks of k values), took 0.14 / 0.70 / 1.51 ms a launch at k
// = 1,000 / 4,000 / 8,192 and d = 300 / 64 / 8, up to twice the pass that the lists
// are to save; this takes 0.10 / 0.36 / 0.42 (256 centres of 64 features: 13 us as
// before).
template <int A, int G>
__global__ void __launch_bounds__(PT)
    prune_near_lists_kernel(const float *__restrict__ c32, const float *__restrict__ cerr, int k, int d,
                            float *__restrict__ nthr, int *__restrict__ nidx) {
    extern __shared__ __align__(16) float sm[];  // thr[A][k], then (at 16 bytes) the centres' rows [A][d]
    float *const row = sm + (((size_t)A * k + 3) & ~(size_t)3);
    const int a0 = blockIdx.x * A, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int e = tid; e < A * d; e += PT) {
        const int a = e / d;
        row[e] = c32[(int64_t)min(a0 + a, k - 1) * d + e - a * d];
    }
    __syncthreads();
    const float rho = (float)(d + 8) * 1e-6f;
    auto store = [&](int a, int q, float s) {
        const float e = cerr ? __fadd_ru(cerr[min(a0 + a, k - 1)], cerr[q]) : 0.f;
        const float th = 0.25f * __fsub_rd(s, bound32(s, e, d)) * (1.0f - rho);
        sm[(size_t)a * k + q] = q == a0 + a ? INFINITY : (th > 1e-30f && th < FLT_MAX ? th : 0.f);
    };
    const bool vec = (d & 3) == 0 && ((reinterpret_cast<uintptr_t>(c32) | reinterpret_cast<uintptr_t>(row)) & 15) == 0;
    // (one bound for every lane of a warp: the shuffles are warp-wide)
    for (int q0 = w * (32 / G); q0 < k; q0 += PT / G) {
        const int q = q0 + lane / G;
        const float *cq = c32 + (int64_t)min(q, k - 1) * d;
        float s[A];
#pragma unroll
        for (int a = 0; a < A; a++) s[a] = 0.f;
        if (vec) {
            const float4 *c4 = reinterpret_cast<const float4 *>(cq);
#pragma unroll 4
            for (int j = lane % G; j < d / 4; j += G) {
                const float4 cv = c4[j];
#pragma unroll
                for (int a = 0; a < A; a++) {
                    const float4 r = *reinterpret_cast<const float4 *>(row + a * d + 4 * j);
                    const float t0 = __fsub_rn(r.x, cv.x), t1 = __fsub_rn(r.y, cv.y), t2 = __fsub_rn(r.z, cv.z),
                                t3 = __fsub_rn(r.w, cv.w);
                    s[a] = __fmaf_rn(t3, t3, __fmaf_rn(t2, t2, __fmaf_rn(t1, t1, __fmaf_rn(t0, t0, s[a]))));
                }
            }
        } else {
#pragma unroll 8
            for (int j = lane % G; j < d; j += G) {
                const float cv = cq[j];
#pragma unroll
                for (int a = 0; a < A; a++) {
                    const float t = __fsub_rn(row[a * d + j], cv);
                    s[a] = __fmaf_rn(t, t, s[a]);
                }
            }
        }
        if (G == 1) {
            if (q < k)
#pragma unroll
                for (int a = 0; a < A; a++) store(a, q, s[a]);
        } else {
            // the lanes' sums, each lane left with those of half the centres a step
            int a = 0;
            float v = s[0];
            if constexpr (A == 4) {
                const bool hi = lane & 4, hi2 = lane & 2;
                const float k0 = (hi ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[2], 4);
                const float k1 = (hi ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, hi ? s[1] : s[3], 4);
                v = (hi2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, hi2 ? k0 : k1, 2);
                a = (hi ? 2 : 0) + (hi2 ? 1 : 0);
            } else if constexpr (A == 2) {
                const bool hi = lane & 4;
                v = (hi ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[1], 4);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                a = hi ? 1 : 0;
            } else {
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
            }
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if (q < k && (lane & (8 / A - 1)) == 0) store(a, q, v);
        }
    }
    __syncthreads();
    if (k <= PT) {
        // each centre's rank among the others, ties by index
        for (int a = 0; a < A && a0 + a < k; a++) {
            const float *thr = sm + (size_t)a * k;
            for (int q = tid; q < k; q += PT) {
                const float v = thr[q];
                int rank = 0;
#pragma unroll 8
                for (int p = 0; p < k; p++) rank += thr[p] < v || (thr[p] == v && p < q);
                if (rank < NROW) {
                    nthr[(int64_t)(a0 + a) * NROW + rank] = v;
                    if (rank < NEAR) nidx[(int64_t)(a0 + a) * NEAR + rank] = v < INFINITY ? q : -1;
                }
            }
            for (int t = k + tid; t < NROW; t += PT) {
                nthr[(int64_t)(a0 + a) * NROW + t] = INFINITY;
                if (t < NEAR) nidx[(int64_t)(a0 + a) * NEAR + t] = -1;
            }
        }
        return;
    }
    // More centres: each warp takes the smallest NROW of its part, one after the
    // other (non-negative floats order as their bits), then the ranks among the
    // parts' lists.
    constexpr int NW = PT / 32, PARTS = NW / A;  // warps per centre
    __shared__ uint32_t best_v[NW * NROW];
    __shared__ int best_q[NW * NROW];
    {
        float *thr = sm + (size_t)(w / PARTS) * k;
        for (int t = 0; t < NROW; t++) {
            uint32_t best = 0xFFFFFFFFu;
            int at = -1;
#pragma unroll 4
            for (int q = (w % PARTS) * 32 + lane; q < k; q += 32 * PARTS) {
                const uint32_t b = __float_as_uint(thr[q]);
                if (b < best) {
                    best = b;
                    at = q;
                }
            }
            const uint32_t m = __reduce_min_sync(0xffffffffu, best);
            const int src = __ffs(__ballot_sync(0xffffffffu, best == m)) - 1;
            at = __shfl_sync(0xffffffffu, at, src);
            if (lane == 0) {
                const bool any = m < 0x7F800000u;
                best_v[w * NROW + t] = any ? m : 0x7F800000u;
                best_q[w * NROW + t] = any ? at : -1;
                if (any) thr[at] = __uint_as_float(0x7F800001u);  // taken: NaN, above every float's bits
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int e = tid; e < NW * NROW; e += PT) {
        const int a = e / (PARTS * NROW), first = a * PARTS * NROW;
        const uint32_t v = best_v[e];
        int rank = 0;
        for (int p = first; p < first + PARTS * NROW; p++) rank += best_v[p] < v || (best_v[p] == v && p < e);
        if (rank < NROW && a0 + a < k) {
            nthr[(int64_t)(a0 + a) * NROW + rank] = __uint_as_float(v);
            if (rank < NEAR) nidx[(int64_t)(a0 + a) * NEAR + rank] = best_q[e];
        }
    }
}

template <int A>
void launch_near_lists(const float *c32, const float *cerr, int k, int d, float *nthr, int *nidx, cudaStream_t s) {
    const size_t smem = sizeof(float) * (A * ((size_t)k + d) + 3);
    auto run = [&](auto kernel) {
        if (smem > 48 * 1024)
            FK_CUDA(cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<(unsigned)((k + A - 1) / A), PT, smem, s>>>(c32, cerr, k, d, nthr, nidx);
        FK_LAUNCH_CHECK();
    };
    if (d <= 16) run(prune_near_lists_kernel<A, 1>);
    else run(prune_near_lists_kernel<A, 8>);
}

struct PruneLists {
    int32_t *near_rows, *scan_rows, *open_rows;
    unsigned long long *count;  // [0] near, [1] scan, [2] open
};

__device__ __forceinline__ void append(bool pred, int32_t *__restrict__ list, unsigned long long *count, int64_t v) {
    const unsigned act = __activemask();
    const unsigned m = __ballot_sync(act, pred);
    if (!m) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned long long at = 0;
    if (lane == leader) at = atomicAdd(count, (unsigned long long)__popc(m));
    at = __shfl_sync(act, at, leader);
    if (pred) list[at + __popc(m & ((1u << lane) - 1u))] = (int32_t)v;
}

// Rows whose bounds still separate keep their label; the others are listed.
// 20 bytes a row: bound by launch latency and L2.
__global__ void __launch_bounds__(PT)
    prune_bound_kernel(int64_t n, int k, int d, const int32_t *__restrict__ prev, int32_t *__restrict__ labels,
                       float *__restrict__ ub, float *__restrict__ lb, const float *__restrict__ shift,
                       const float *__restrict__ nthr, PruneLists L) {
    // the largest shift, its centre, and the largest of the others (a NaN shift is stored as +inf)
    __shared__ float m1s[PT / 32], m2s[PT / 32];
    __shared__ int a1s[PT / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    float m1 = -1.f, m2 = -1.f;
    int a1 = -1;
    auto merge = [&](float v1, int i1, float v2) {
        if (v1 > m1) {
            m2 = fmaxf(m1, v2);
            m1 = v1;
            a1 = i1;
        } else {
            m2 = fmaxf(m2, v1);
        }
    };
    for (int q = tid; q < k; q += PT) merge(shift[q], q, -1.f);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const float v1 = __shfl_xor_sync(0xffffffffu, m1, o), v2 = __shfl_xor_sync(0xffffffffu, m2, o);
        const int i1 = __shfl_xor_sync(0xffffffffu, a1, o);
        if (i1 != a1) merge(v1, i1, v2);
    }
    if (lane == 0) {
        m1s[w] = m1;
        m2s[w] = m2;
        a1s[w] = a1;
    }
    __syncthreads();
    m1 = m2 = -1.f;
    a1 = -1;
    for (int q = 0; q < PT / 32; q++)
        if (a1s[q] >= 0) merge(m1s[q], a1s[q], m2s[q]);
    m2 = fmaxf(m2, 0.f);
    const float rel = 1.f + 4.f * fold_rel(d);
    // BU rows a thread, their loads in flight together; a block reserves both
    // lists' slots once per BU * PT rows (1M rows: 10.8 us; 19.7 with a row a
    // thread and a warp's two additions to the shared counters)
    __shared__ int wn[PT / 32], ws[PT / 32];
    __shared__ unsigned long long at_near, at_scan;
    for (int64_t i0 = (int64_t)blockIdx.x * (BU * PT) + tid; i0 - tid < n; i0 += (int64_t)gridDim.x * (BU * PT)) {
        int a[BU];
        float ui[BU], li[BU];
#pragma unroll
        for (int q = 0; q < BU; q++) {
            const int64_t i = i0 + q * PT;
            a[q] = i < n ? prev[i] : -1;
            ui[q] = i < n ? ub[i] : 0.f;
            li[q] = i < n ? lb[i] : 0.f;
        }
        unsigned nearm[BU], scanm[BU];
        int cn = 0, cs = 0;
#pragma unroll
        for (int q = 0; q < BU; q++) {
            const int64_t i = i0 + q * PT;
            bool near = false, scan = false;
            if (a[q] >= 0) {
                const float u = __fadd_ru(ui[q], shift[a[q]]);
                // every other centre is at least twice the root of the nearest one's
                // threshold away from this one
                const float gap = __fmul_rd(2.f, __fsqrt_rd(nthr[(int64_t)a[q] * NROW]));
                const float l = fmaxf(__fsub_rd(li[q], a[q] == a1 ? m2 : m1), __fsub_rd(gap, u));
                if (__fmul_ru(u, rel) < l && l > 1e-15f) {
                    labels[i] = a[q];
                    ub[i] = u;
                    lb[i] = l;
                } else {
                    near = __fmul_ru(__fmul_ru(u, u), rel) < nthr[(int64_t)a[q] * NROW + NEAR];
                    scan = !near;
                }
            }
            nearm[q] = __ballot_sync(0xffffffffu, near);
            scanm[q] = __ballot_sync(0xffffffffu, scan);
            cn += __popc(nearm[q]);
            cs += __popc(scanm[q]);
        }
        if (lane == 0) {
            wn[w] = cn;
            ws[w] = cs;
        }
        __syncthreads();
        if (tid == 0) {
            int tn = 0, ts = 0;
            for (int q = 0; q < PT / 32; q++) {
                const int vn = wn[q], vs = ws[q];
                wn[q] = tn;
                ws[q] = ts;
                tn += vn;
                ts += vs;
            }
            at_near = tn ? atomicAdd(L.count, (unsigned long long)tn) : 0;
            at_scan = ts ? atomicAdd(L.count + 1, (unsigned long long)ts) : 0;
        }
        __syncthreads();
        unsigned long long pn = at_near + wn[w], ps = at_scan + ws[w];
        const unsigned before = (1u << lane) - 1u;
#pragma unroll
        for (int q = 0; q < BU; q++) {
            const int32_t i = (int32_t)(i0 + q * PT);
            if ((nearm[q] >> lane) & 1u) L.near_rows[pn + __popc(nearm[q] & before)] = i;
            if ((scanm[q] >> lane) & 1u) L.scan_rows[ps + __popc(scanm[q] & before)] = i;
            pn += __popc(nearm[q]);
            ps += __popc(scanm[q]);
        }
    }
}

// ------------------------------------------------- one row's comparison --
// F = f32: the exact minimum (lowest index on ties, below F::MAX only) and the
// smallest of the other values.
struct Best32 {
    float v, other;
    int i;
    __device__ __forceinline__ void init() {
        v = FLT_MAX;
        i = INT32_MAX;
        other = INFINITY;
    }
    __device__ __forceinline__ void add(float d32, float, int c, int) {
        if (d32 < v || (d32 == v && d32 < FLT_MAX && c < i)) {
            other = fminf(other, i == INT32_MAX ? INFINITY : v);
            v = d32;
            i = c;
        } else {
            other = fminf(other, d32);  // NaN never wins
        }
    }
    __device__ __forceinline__ void merge(const Best32 &o) {
        if (o.i == INT32_MAX) {
            other = fminf(other, o.other);
        } else if (o.v < v || (o.v == v && o.i < i)) {
            other = fminf(fminf(other, o.other), i == INT32_MAX ? INFINITY : v);
            v = o.v;
            i = o.i;
        } else {
            other = fminf(fminf(other, o.other), o.v);
        }
    }
    __device__ __forceinline__ Best32 shfl(int off) const {
        return {__shfl_xor_sync(0xffffffffu, v, off), __shfl_xor_sync(0xffffffffu, other, off),
                __shfl_xor_sync(0xffffffffu, i, off)};
    }
    __device__ __forceinline__ bool open() const { return false; }
    __device__ __forceinline__ int label() const { return i == INT32_MAX ? 0 : i; }
    __device__ __forceinline__ float up(int d) const {
        return i == INT32_MAX ? INFINITY : dist_up(__fmul_ru(v, 1.f + fold_rel(d)));
    }
    // (an F value that overflowed bounds its distance by the largest finite one only)
    __device__ __forceinline__ float down(int d) const {
        return dist_down(__fmul_rd(fminf(other, FLT_MAX), 1.f - fold_rel(d)));
    }
};

// F = f64: the centre with the smallest upper bound (ua, its lower bound la),
// and the smallest lower bound of the others; other > ua proves every other
// FP64 distance larger.
struct Best64 {
    float ua, la, other;
    int i;
    bool bad;
    __device__ __forceinline__ void init() {
        ua = la = other = INFINITY;
        i = -1;
        bad = false;
    }
    __device__ __forceinline__ void add(float d32, float err, int c, int d) {
        const float b = bound32(d32, err, d);
        const float lo = __fsub_rd(d32, b), hi = __fadd_ru(d32, b);
        if (!(lo <= hi)) bad = true;  // NaN
        if (hi < ua) {
            other = fminf(other, la);
            ua = hi;
            la = lo;
            i = c;
        } else {
            other = fminf(other, lo);
        }
    }
    __device__ __forceinline__ void merge(const Best64 &o) {
        bad = bad || o.bad;
        if (o.ua < ua) {
            other = fminf(fminf(other, o.other), la);
            ua = o.ua;
            la = o.la;
            i = o.i;
        } else {
            other = fminf(fminf(other, o.other), o.la);
        }
    }
    __device__ __forceinline__ Best64 shfl(int off) const {
        return {__shfl_xor_sync(0xffffffffu, ua, off), __shfl_xor_sync(0xffffffffu, la, off),
                __shfl_xor_sync(0xffffffffu, other, off), __shfl_xor_sync(0xffffffffu, i, off),
                __shfl_xor_sync(0xffffffffu, (int)bad, off) != 0};
    }
    __device__ __forceinline__ bool open() const { return bad || i < 0 || !(other > ua); }
    __device__ __forceinline__ int label() const { return i; }
    __device__ __forceinline__ float up(int) const { return dist_up(ua); }
    __device__ __forceinline__ float down(int) const { return dist_down(other); }
};

template <typename F> struct BestOf;
template <> struct BestOf<float> { using T = Best32; };
template <> struct BestOf<double> { using T = Best64; };

// acc + (x - c)^2: F's own rounding in f32, one rounding fewer in the FP32
// stand-in for f64 (its bound covers both).
template <typename F>
__device__ __forceinline__ float sq_step(float acc, float x, float c) {
    const float t = __fsub_rn(x, c);
    return std::is_same<F, float>::value ? __fadd_rn(acc, __fmul_rn(t, t)) : __fmaf_rn(t, t, acc);
}

template <typename F>
__device__ __forceinline__ float row_dist(const float *__restrict__ x, const float *__restrict__ c, int d, bool vec) {
    float acc = 0.f;
    if (vec) {
        const float4 *x4 = reinterpret_cast<const float4 *>(x), *c4 = reinterpret_cast<const float4 *>(c);
#pragma unroll 4
        for (int q = 0; q < d / 4; q++) {
            const float4 a = x4[q], b = c4[q];
            acc = sq_step<F>(acc, a.x, b.x);
            acc = sq_step<F>(acc, a.y, b.y);
            acc = sq_step<F>(acc, a.z, b.z);
            acc = sq_step<F>(acc, a.w, b.w);
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < d; j++) acc = sq_step<F>(acc, x[j], c[j]);
    }
    return acc;
}

template <typename F, typename B>
__device__ __forceinline__ void store_row(const B &b, int64_t i, int d, float rest, int32_t *__restrict__ labels,
                                          float *__restrict__ ub, float *__restrict__ lb, const PruneLists &L) {
    const bool open = b.open();
    labels[i] = open ? -1 : b.label();
    ub[i] = open ? INFINITY : b.up(d);
    lb[i] = open ? 0.f : fminf(b.down(d), rest);
    if (!std::is_same<F, float>::value) append(open, L.open_rows, L.count + 2, i);
}

// The rows near one centre: a thread a row, the row from shared memory (copied
// by the block, coalesced) where `staged`, the label's centre first, then its
// neighbours while they may be as near. Most rows meet none to three of them,
// so the reads of the rows are the bound.
template <typename F>
__global__ void __launch_bounds__(PT)
    prune_near_kernel(const float *__restrict__ x, const float *__restrict__ xerr, int d,
                      const float *__restrict__ c32, const float *__restrict__ cerr, const int32_t *__restrict__ prev,
                      const float *__restrict__ nthr, const int *__restrict__ nidx, int32_t *__restrict__ labels,
                      float *__restrict__ ub, float *__restrict__ lb, int tile, int xs, PruneLists L) {
    using B = typename BestOf<F>::T;
    extern __shared__ __align__(16) float rows_sm[];
    __shared__ int32_t ids[PT];
    const long long cnt = (long long)L.count[0];
    const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(c32) & 15) == 0;
    const int tid = threadIdx.x;
    for (long long t0 = (long long)blockIdx.x * tile; t0 < cnt; t0 += (long long)gridDim.x * tile) {
        const int rows = (int)min((long long)tile, cnt - t0);
        __syncthreads();
        if (tid < rows) ids[tid] = L.near_rows[t0 + tid];
        __syncthreads();
        if (xs > 0) {
            if (vec) {
                const int d4 = d / 4;
                for (int e = tid; e < rows * d4; e += PT) {
                    const int r = e / d4, q = e - r * d4;
                    *reinterpret_cast<float4 *>(rows_sm + r * xs + 4 * q) =
                        *reinterpret_cast<const float4 *>(x + (int64_t)ids[r] * d + 4 * q);
                }
            } else {
                for (int e = tid; e < rows * d; e += PT) {
                    const int r = e / d, j = e - r * d;
                    rows_sm[r * xs + j] = x[(int64_t)ids[r] * d + j];
                }
            }
            __syncthreads();
        }
        if (tid < rows) {
            const int64_t i = ids[tid];
            const float *xr = xs > 0 ? rows_sm + tid * xs : x + i * d;
            const int a = prev[i];
            const float er = std::is_same<F, float>::value ? 0.f : xerr[i];
            B b;
            b.init();
            const float ea = std::is_same<F, float>::value ? 0.f : __fadd_ru(er, cerr[a]);
            const float da = row_dist<F>(xr, c32 + (int64_t)a * d, d, vec);
            b.add(da, ea, a, d);
            // F's value of the distance to the label's centre, at most this
            const float m = std::is_same<F, float>::value ? da : __fadd_ru(da, bound32(da, ea, d));
            const float *th = nthr + (int64_t)a * NROW;
            int q = 0;
            for (; q < NEAR && !(m < th[q]); q++) {
                const int c = nidx[(int64_t)a * NEAR + q];
                if (c < 0) break;
                const float ec = std::is_same<F, float>::value ? 0.f : __fadd_ru(er, cerr[c]);
                b.add(row_dist<F>(xr, c32 + (int64_t)c * d, d, vec), ec, c, d);
            }
            // (the threshold after the last compared one bounds every centre left out)
            const float next = th[q];
            const bool all = m < next;
            if (all) {
                const float rest = next < INFINITY
                                       ? __fsub_rd(__fmul_rd(2.f, __fsqrt_rd(next)),
                                                   dist_up(__fmul_ru(m, 1.f + fold_rel(d))))
                                       : INFINITY;
                store_row<F>(b, i, d, rest, labels, ub, lb, L);
            }
            append(!all, L.scan_rows, L.count + 1, i);
        }
    }
}

constexpr int SBM = 128, SBN = 128, SDJ = 16;  // rows, centres and features of a block tile
constexpr int STM = 8, STN = 8;                // of a thread

// Every centre for the listed rows (list null: all n rows): 128 x 128 tiles,
// 8 x 8 distances a thread, 16 features staged at a time; a row's 16 threads
// merge at the end. Bound by the FP32 pipe (3 operations a feature and pair in
// f32, 2 in f64), and where there is a tile an SM at most by the loads' latency:
// FEW keeps the rows' numbers in registers then, not in shared memory before each
// load (10,000 x 1,000 against 300 centres 1.32 ms -> 0.96, 66,000 x 64 against
// 4,000 2.33 -> 2.43).
template <typename F, bool FEW>
__global__ void __launch_bounds__(PT)
    prune_scan_kernel(const float *__restrict__ x, const float *__restrict__ xerr, int64_t n, int d,
                      const float *__restrict__ c32, const float *__restrict__ cerr, int k,
                      const int32_t *__restrict__ list, int32_t *__restrict__ labels, float *__restrict__ ub,
                      float *__restrict__ lb, PruneLists L) {
    using B = typename BestOf<F>::T;
    __shared__ __align__(16) float xsm[SDJ][SBM];
    __shared__ __align__(16) float csm[SDJ][SBN];
    __shared__ int32_t ids[SBM];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t cnt = list ? (int64_t)L.count[1] : n;
    for (int64_t row0 = (int64_t)blockIdx.x * SBM; row0 < cnt; row0 += (int64_t)gridDim.x * SBM) {
        __syncthreads();  // the tile before is done with ids
        if (tid < SBM) ids[tid] = row0 + tid < cnt ? (list ? list[row0 + tid] : (int32_t)(row0 + tid)) : -1;
        __syncthreads();
        constexpr int PER = (SBM * SDJ) / PT;  // values of a tile that a thread stages, one feature of PER rows
        int32_t rid[FEW ? PER : 1];
        if constexpr (FEW) {
#pragma unroll
            for (int e = 0; e < PER; e++) rid[e] = ids[tid / SDJ + e * (PT / SDJ)];
        }
        B b[STM];
        float ex[STM];
#pragma unroll
        for (int a = 0; a < STM; a++) {
            b[a].init();
            const int id = ids[ty * STM + a];
            ex[a] = !std::is_same<F, float>::value && id >= 0 ? xerr[id] : 0.f;
        }
        for (int ct = 0; ct < k; ct += SBN) {
            float acc[STM][STN];
#pragma unroll
            for (int a = 0; a < STM; a++)
#pragma unroll
                for (int q = 0; q < STN; q++) acc[a][q] = 0.f;
            for (int j0 = 0; j0 < d; j0 += SDJ) {
#pragma unroll
                for (int e = 0; e < PER; e++) {
                    const int r = tid / SDJ + e * (PT / SDJ), jj = tid % SDJ;
                    const int gj = j0 + jj, id = FEW ? rid[FEW ? e : 0] : ids[r], gc = ct + r;
                    xsm[jj][r] = (id >= 0 && gj < d) ? x[(int64_t)id * d + gj] : 0.f;
                    csm[jj][r] = (gc < k && gj < d) ? c32[(int64_t)gc * d + gj] : 0.f;
                }
                __syncthreads();
                const int jn = min(SDJ, d - j0);
                for (int jj = 0; jj < jn; jj++) {
                    float xv[STM], cv[STN];
#pragma unroll
                    for (int a = 0; a < STM; a++) xv[a] = xsm[jj][ty * STM + a];
#pragma unroll
                    for (int q = 0; q < STN; q++) cv[q] = csm[jj][tx * STN + q];
#pragma unroll
                    for (int a = 0; a < STM; a++)
#pragma unroll
                        for (int q = 0; q < STN; q++) acc[a][q] = sq_step<F>(acc[a][q], xv[a], cv[q]);
                }
                __syncthreads();
            }
#pragma unroll
            for (int q = 0; q < STN; q++) {
                const int gc = ct + tx * STN + q;
                if (gc >= k) continue;
                const float ec = std::is_same<F, float>::value ? 0.f : cerr[gc];
#pragma unroll
                for (int a = 0; a < STM; a++) b[a].add(acc[a][q], __fadd_ru(ex[a], ec), gc, d);
            }
        }
#pragma unroll
        for (int a = 0; a < STM; a++) {
            B r = b[a];
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) r.merge(r.shfl(off));
            const int id = ids[ty * STM + a];
            if (tx == 0 && id >= 0) store_row<F>(r, id, d, INFINITY, labels, ub, lb, L);
        }
    }
}

// Each row's direct-form F distance to its label (F::MAX where it is not below:
// label 0 of a row that no centre won).
template <typename F>
__global__ void prune_dist_kernel(const F *__restrict__ x, int64_t n, int d, const F *__restrict__ c,
                                  const int32_t *__restrict__ labels, F *__restrict__ mind) {
    constexpr bool S = std::is_same<F, float>::value;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const F *xr = x + r * d, *cr = c + (int64_t)labels[r] * d;
        F acc = F(0);
#pragma unroll 4
        for (int j = 0; j < d; j++) {
            if constexpr (S) {
                const float t = __fsub_rn(xr[j], cr[j]);
                acc = __fadd_rn(acc, __fmul_rn(t, t));
            } else {
                const double t = __dsub_rn(xr[j], cr[j]);
                acc = __dadd_rn(acc, __dmul_rn(t, t));
            }
        }
        const F most = S ? (F)FLT_MAX : (F)DBL_MAX;
        mind[r] = acc < most ? acc : most;
    }
}

}  // namespace

// What the lists of near centres cost beside a pass over every centre (measured
// from k = 300, d = 1,000 to k = 8,192, d = 8: 4e-12 s a pair of centres and 3e-13 a
// feature of it, the pass 1.2e-13 s a row, centre and feature).
static double lists_cost(int64_t n, int d, int k) { return k * (32.0 + 2.6 * d) / ((double)n * d); }

bool prune_shape_ok(int64_t n, int d, int k) {
    // Below: the direct pass takes less than the lists' extra launches (about
    // 25 us). k and d: a centre's thresholds and row fill shared memory. Lists that cost
    // about half a pass pay on no data tried (66,000 x 8 against 8,192 centres,
    // 0.8 of a pass: 20 iterations 25.8-29 ms, 24.8 without).
    return k >= 32 && k <= 8192 && d >= 1 && d <= 8192 && n >= 8 * (int64_t)k && (double)n * k * d >= 1e9 &&
           lists_cost(n, d, k) <= 0.45;
}

// Whether a bounded iteration that keeps few rows is worth leaving out. 20 iterations
// on rows without structure, f32, beside the same without bounds, always bounded /
// resting: 50,000 x 32 against 2,000 centres 1.19 / 1.10, 200,000 x 64 against 8,192
// 1.09 / 1.03, 66,000 x 8 against 4,000 1.08 / 1.05 (on clusters 0.57, 0.39 and 0.97 either
// way). Below the line resting loses more where the bounds come to pay late:
// 400,000 x 80 against 32 wide clusters 0.60 / 0.66, 1M x 64 against 256 0.60 / 0.87.
bool prune_may_rest(int64_t n, int d, int k) { return lists_cost(n, d, k) > 1.0 / 16; }

template <typename F>
void launch_assign_pruned(Ctx &ctx, const F *x, int64_t n, int d, const F *c, const F *c_prev, int k,
                          const int32_t *prev, int32_t *labels, bool fresh_x, DevScalars *sc) {
    cudaStream_t s = ctx.stream;
    constexpr bool S = std::is_same<F, float>::value;
    const float *x32, *c32, *xerr = nullptr, *cerr = nullptr;
    if constexpr (S) {
        x32 = x;
        c32 = c;
    } else {
        float *xw = (float *)ctx.get(BUF_PF_X32, sizeof(float) * (size_t)n * d);
        float *xe = (float *)ctx.get(BUF_PF_XERR, sizeof(float) * (size_t)n);
        float *cw = (float *)ctx.get(BUF_PF_C32, sizeof(float) * (size_t)k * d);
        float *ce = (float *)ctx.get(BUF_PF_CERR, sizeof(float) * (size_t)k);
        if (fresh_x) launch_f32_copy(ctx, x, n, d, xw, xe);
        launch_f32_copy(ctx, c, k, d, cw, ce);
        x32 = xw;
        xerr = xe;
        c32 = cw;
        cerr = ce;
    }
    float *ub = (float *)ctx.get(BUF_PR_UB, sizeof(float) * 2 * (size_t)n), *lb = ub + n;
    float *shift = (float *)ctx.get(BUF_PR_SHIFT, sizeof(float) * (size_t)k);
    float *nthr = (float *)ctx.get(BUF_PR_NEAR, (sizeof(float) * NROW + sizeof(int) * NEAR) * (size_t)k);
    int *nidx = (int *)(nthr + (size_t)NROW * k);
    PruneLists L;
    L.near_rows = (int32_t *)ctx.get(BUF_PR_LIST, sizeof(int32_t) * 3 * (size_t)n);
    L.scan_rows = L.near_rows + n;
    L.open_rows = L.scan_rows + n;
    L.count = sc->prune;
    const int64_t tiles = (n + SBM - 1) / SBM;
    auto scan = [&](const int32_t *list, int64_t blocks) {
        if (tiles <= ctx.num_sms)
            prune_scan_kernel<F, true><<<(unsigned)blocks, PT, 0, s>>>(x32, xerr, n, d, c32, cerr, k, list, labels, ub, lb, L);
        else
            prune_scan_kernel<F, false><<<(unsigned)blocks, PT, 0, s>>>(x32, xerr, n, d, c32, cerr, k, list, labels, ub, lb, L);
        FK_LAUNCH_CHECK();
    };
    if (!c_prev) {
        scan(nullptr, tiles);
    } else {
        prune_shift_kernel<F><<<(unsigned)((k + 7) / 8), PT, 0, s>>>(c, c_prev, k, d, shift);
        FK_LAUNCH_CHECK();
        // as many centres a block as leave two blocks for every SM, and room for three on
        // it (k = 300, d = 1,000 with one: 64 us; 4,000 x 64 with one 417, with four 365)
        if (k >= 8 * ctx.num_sms && k + d <= 4608) launch_near_lists<4>(c32, cerr, k, d, nthr, nidx, s);
        else if (k >= 4 * ctx.num_sms && k + d <= 9216) launch_near_lists<2>(c32, cerr, k, d, nthr, nidx, s);
        else launch_near_lists<1>(c32, cerr, k, d, nthr, nidx, s);
        const int64_t bound_blocks = std::min<int64_t>((n + BU * PT - 1) / (BU * PT), (int64_t)ctx.num_sms * 8);
        prune_bound_kernel<<<(unsigned)bound_blocks, PT, 0, s>>>(
            n, k, d, prev, labels, ub, lb, shift, nthr, L);
        FK_LAUNCH_CHECK();
        // rows in shared memory while 64 of them fit beside other blocks; padded
        // to an odd number of 16-byte units (no bank conflicts)
        int w = (d + 3) / 4 * 4;
        w += (w / 4) & 1 ? 8 : 4;
        int tile = PT, xs = w;
        while (tile > 64 && (size_t)tile * w * sizeof(float) > 72 * 1024) tile /= 2;
        if ((size_t)tile * w * sizeof(float) > 72 * 1024) {
            tile = PT;
            xs = 0;
        }
        const size_t nsm = sizeof(float) * (size_t)tile * xs;
        if (nsm > 48 * 1024)
            FK_CUDA(cudaFuncSetAttribute((const void *)prune_near_kernel<F>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nsm));
        prune_near_kernel<F><<<(unsigned)std::min<int64_t>((n + tile - 1) / tile, (int64_t)ctx.num_sms * 8), PT, nsm,
                               s>>>(x32, xerr, d, c32, cerr, prev, nthr, nidx, labels, ub, lb, tile, xs, L);
        FK_LAUNCH_CHECK();
        scan(L.scan_rows, std::min<int64_t>(tiles, (int64_t)ctx.num_sms * 4));
    }
    if constexpr (!S) 
        launch_f64_open_rows(ctx, x, x32, xerr, d, c, c32, cerr, k, L.open_rows, L.count + 2, labels, nullptr);
}

template <typename F>
void launch_label_dist(Ctx &ctx, const F *x, int64_t n, int d, const F *c, const int32_t *labels, F *mind) {
    if (n == 0) return;
    prune_dist_kernel<F><<<(unsigned)std::min<int64_t>((n + PT - 1) / PT, (int64_t)ctx.num_sms * 8), PT, 0, ctx.stream>>>(
        x, n, d, c, labels, mind);
    FK_LAUNCH_CHECK();
}

template void launch_assign_pruned<float>(Ctx &, const float *, int64_t, int, const float *, const float *, int,
                                          const int32_t *, int32_t *, bool, DevScalars *);
template void launch_assign_pruned<double>(Ctx &, const double *, int64_t, int, const double *, const double *, int,
                                           const int32_t *, int32_t *, bool, DevScalars *);
template void launch_label_dist<float>(Ctx &, const float *, int64_t, int, const float *, const int32_t *, float *);
template void launch_label_dist<double>(Ctx &, const double *, int64_t, int, const double *, const int32_t *, double *);

}  // namespace fk
