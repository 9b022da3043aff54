// fk_batched.cu -- many independent KMeans<f32> fits (uneven n, d, k) in one
// call: kmeans.rs:417-512 once per (problem, run), all runs at once.
//
// Layout in HBM: every problem's rows packed into one f32 buffer (16-byte
// aligned starts); per fit (problem p, run r) an n_p-long int32 scratch pair
// (labels | members) and two k x d centre buffers that alternate between
// iterations.
//
// Launches:
//   k-means++            every fit's seeding together (fk_kpp.cu).
//   batch_assign_kernel  per Lloyd iteration, one persistent launch per
//                        (d, k) bucket over a queue of (fit, row range) items,
//                        largest fits first; the fit's centres in shared
//                        memory; rows that cannot have changed their label
//                        score one centre, the others every centre, rows in
//                        registers; direct-form f32 distances
//                        (no FMA), strict < from F::MAX. The tile shape (rows
//                        per thread x centres per pass) is the autotuner's
//                        choice for the bucket. Per item a fixed-tree f64
//                        inertia partial.
//   batch_near_kernel    the thresholds of that test for the next iteration.
//   batch_accum_kernel   f64 reduction: the exact (integer, order-free) sums of
//                        each (fit, row range) item added to its fit's;
//   batch_means_kernel   then per fit each sum rounded once to f64 with the mean
//                        rounded once to f32.
//   batch_update_kernel  reference reduction, one persistent launch over the
//                        fits: counting sort of the labels (stable, eight warps
//                        over contiguous row ranges), then per (cluster,
//                        feature) the row-order f32 sum exactly like
//                        recompute_centroids_into (kmeans.rs:358-401).
//                        Both end an iteration: the empty cluster rule, sqrt of
//                        the max squared shift, the tol test, n_iter and the
//                        inertia (partials in item order).
// One iteration (counter reset + bucket launches + update) is captured once
// in a CUDA graph and replayed until every fit has converged or reached
// max_iter; converged fits are skipped inside the kernels.
#include <cfloat>
#include <cmath>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "fk_internal.cuh"

namespace fk {
namespace {

struct BFit {
    int64_t x_off;  // float offset of the problem's rows in the packed X
    int64_t s_off;  // offset of this fit's n-long scratch arrays
    int64_t c_off;  // float offset of this fit's two k x d centre buffers
    int32_t n, d, k, max_iter;
    float tol;
    int32_t first_item, n_items;
    int32_t prob, pad;
    int32_t keep_sums;  // f64 reduction: the sums carry over to the next iteration
    int32_t bounded;    // rows are tested against their last label's centre first
    int64_t k_off;    // offset of this fit's k cluster counts and row thresholds
    uint64_t seed;
};

struct BState {
    double inertia;
    int32_t cur, n_iter, done;
    int32_t full;  // f64 reduction: the sums are zero, every row is to be added
};

struct BItem {
    int32_t fit, lo, hi, pad;
};

constexpr int ASSIGN_T = 128;
constexpr int UPDATE_T = 256;
constexpr int NBUCKETS = 20;  // d in {8, 16, 32, 64, other} x k in {<=16, <=32, <=64, >64}
constexpr int NVARIANTS = 5;  // (rows per thread, centres per pass): (1,1) (2,1) (1,2) (2,2) (4,1)
constexpr int BOUND_K = 128;  // clusters of a bounded fit at most
constexpr int MAX_K = 1024, MAX_D = 256, MAX_KD = 32768;

// squared_euclidean (kmeans.rs:159-163) in f32: left fold, no FMA.
__device__ __forceinline__ float sqeuc_f32(const float *__restrict__ a, const float *__restrict__ b, int d) {
    float acc = 0.f;
    for (int j = 0; j < d; j++) {
        const float t = __fsub_rn(a[j], b[j]);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
    }
    return acc;
}

// ------------------------------------------------------------ assignment --
__device__ __forceinline__ double block_sum_f64(double v, double *sh) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) r += sh[q];
    return r;
}

// Rows of an item at most, features staged at a time, stages.
constexpr int ITEM_ROWS = 1024, ROW_SLAB = 32, ROW_STAGES = 2;
__host__ __device__ constexpr int row_slab(int d) { return d < ROW_SLAB ? d : ROW_SLAB; }
// Row stride in shared memory: an odd number of 16-byte units, so that eight
// lanes reading 16 bytes of eight rows meet no bank conflict (d = 8, 16, 32, 64).
__host__ __device__ constexpr int row_stride(int d) { return d + 4; }
// Rows of up to 16 features are read straight into registers.
__host__ __device__ constexpr bool rows_staged(int d) { return d > 16; }
size_t assign_smem(int d, int k) {
    const size_t stages = rows_staged(d) ? (size_t)ROW_STAGES * ASSIGN_T * row_stride(row_slab(d)) : 0;
    return sizeof(float) * ((size_t)k * row_stride(d) + stages + ITEM_ROWS) + sizeof(uint16_t) * ITEM_ROWS;
}

__device__ __forceinline__ void copy16_async(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// acc + (a - b)^2 over four features in order, no FMA.
__device__ __forceinline__ float add_sq4(float acc, const float4 &a, const float4 &b) {
    const float t0 = __fsub_rn(a.x, b.x), t1 = __fsub_rn(a.y, b.y), t2 = __fsub_rn(a.z, b.z), t3 = __fsub_rn(a.w, b.w);
    acc = __fadd_rn(acc, __fmul_rn(t0, t0));
    acc = __fadd_rn(acc, __fmul_rn(t1, t1));
    acc = __fadd_rn(acc, __fmul_rn(t2, t2));
    return __fadd_rn(acc, __fmul_rn(t3, t3));
}

// D > 0: rows of exactly D features; D = 0: any d, one row and one centre at a
// time.
//
// From a fit's second iteration on, a row is first scored against the centre
// of its last label only: a distance below thr,
// a quarter of the centre's squared distance to its nearest other centre with
// room for every rounding (batch_near_kernel), leaves every other centre
// strictly farther, so the label stays and the distance is its term of the
// inertia. The other rows are listed and scored against every centre: rows in
// registers (TR per thread), CP centres per pass, shared-memory reads of the
// centres against 3 FP32 operations each. The inertia's terms meet in shared
// memory and are added in row order, whichever way they came.
//
// 64 problems x 10 runs (d 8 to 64, k 4 to 64, 2,000 to 200,000 rows): 108 ms in
// these kernels with every row scored against every centre, 51 ms like this
// (whole call 142 -> 115 ms). Items of 8,192 rows, as few centres and features
// once had, made a CTA's 64 passes in turn the length of an iteration (104 us at
// d = 8; 15 us with 1,024); rows of 8 or 16 features cost less read directly.
template <int D, int TR, int CP>
__global__ void __launch_bounds__(ASSIGN_T) batch_assign_kernel(const float *__restrict__ X,
                                                                const BFit *__restrict__ fits,
                                                                const BState *__restrict__ state,
                                                                const BItem *__restrict__ items, int nitems,
                                                                int *counter, const float *__restrict__ C,
                                                                const float *__restrict__ thr, int *__restrict__ lab,
                                                                double *__restrict__ partial) {
    extern __shared__ __align__(16) float cs[];
    __shared__ int it_sh, list_n;
    __shared__ double red[ASSIGN_T / 32];
    constexpr int CS = D > 0 ? row_stride(D) : 0, W = row_slab(D), XS = row_stride(W);
    const int tid = threadIdx.x;
    int loaded = -1;
    while (true) {
        if (tid == 0) it_sh = atomicAdd(counter, 1);
        __syncthreads();
        const int it = it_sh;
        __syncthreads();
        if (it >= nitems) break;
        const BItem I = items[it];
        const int f = I.fit;
        if (state[f].done) continue;
        const BFit F = fits[f];
        const int d = D > 0 ? D : F.d, k = F.k;
        if (f != loaded) {
            const float *src = C + F.c_off + (int64_t)state[f].cur * k * d;
            for (int e = tid; e < k * d; e += ASSIGN_T) cs[D > 0 ? e / D * CS + e % D : e] = src[e];
            __syncthreads();
            loaded = f;
        }
        const float *x = X + F.x_off;
        int *L = lab + F.s_off;
        double s = 0.0;
        if constexpr (D > 0) {
            float *const xs = cs + k * CS;  // [ROW_STAGES][ASSIGN_T][XS]
            float *const vals = xs + (rows_staged(D) ? ROW_STAGES * ASSIGN_T * XS : 0);  // [ITEM_ROWS] distances
            uint16_t *const list = reinterpret_cast<uint16_t *>(vals + ITEM_ROWS);       // [ITEM_ROWS] rows to score
            const bool bounded = F.bounded && state[f].n_iter > 0;
            const int rows = I.hi - I.lo;
            const float *const xi = x + (int64_t)I.lo * D;
            int nl = rows;
            if (bounded) {
                if (tid == 0) list_n = 0;
                // row i (live: it exists) at distance v from its label's centre
                auto settle = [&](int i, bool live, float v, float th) {
                    const bool open = live && !(v < th);  // NaN: open
                    if (live && !open) vals[i] = v;
                    const unsigned bm = __ballot_sync(0xffffffffu, open);
                    int at = 0;
                    if ((tid & 31) == 0 && bm) at = atomicAdd(&list_n, __popc(bm));
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (open) list[at + __popc(bm & ((1u << (tid & 31)) - 1u))] = (uint16_t)i;
                };
                if constexpr (!rows_staged(D)) {
                    __syncthreads();
                    constexpr int U = 4;  // rows a thread at a time, their loads in flight together
                    for (int st = 0; st < rows; st += U * ASSIGN_T) {
                        float4 xv[U][D / 4];
                        float th[U];
                        int l[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int i = st + u * ASSIGN_T + tid;
                            l[u] = i < rows ? L[I.lo + i] : 0;
#pragma unroll
                            for (int q = 0; q < D / 4; q++)
                                xv[u][q] = i < rows ? reinterpret_cast<const float4 *>(xi + (int64_t)i * D)[q]
                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) th[u] = thr[F.k_off + l[u]];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int i = st + u * ASSIGN_T + tid;
                            const float4 *cv = reinterpret_cast<const float4 *>(cs + l[u] * CS);
                            float acc = 0.f;
#pragma unroll
                            for (int q = 0; q < D / 4; q++) acc = add_sq4(acc, xv[u][q], cv[q]);
                            settle(i, i < rows, acc, th[u]);
                        }
                    }
                } else {
                    // slab by slab (W features of ASSIGN_T rows), the next one's copies in flight
                    constexpr int SL = D / W;
                    const int ns = (rows + ASSIGN_T - 1) / ASSIGN_T * SL;
                    auto fetch = [&](int g) {
                        const int st = g / SL * ASSIGN_T, j0 = g % SL * W, cnt = min(ASSIGN_T, rows - st);
                        float *dst = xs + g % ROW_STAGES * ASSIGN_T * XS;
                        for (int e = tid; e < cnt * (W / 4); e += ASSIGN_T) {
                            const int r = e / (W / 4), q = e % (W / 4);
                            copy16_async(dst + r * XS + 4 * q, xi + (int64_t)(st + r) * D + j0 + 4 * q);
                        }
                        asm volatile("cp.async.commit_group;" ::: "memory");
                    };
                    fetch(0);
                    float acc = 0.f, th = 0.f;
                    int l = 0;
                    for (int g = 0; g < ns; g++) {
                        const int i = g / SL * ASSIGN_T + tid;
                        if (g % SL == 0) {
                            l = i < rows ? L[I.lo + i] : 0;
                            th = thr[F.k_off + l];
                            acc = 0.f;
                        }
                        if (g + 1 < ns) {
                            fetch(g + 1);
                            asm volatile("cp.async.wait_group 1;" ::: "memory");
                        } else {
                            asm volatile("cp.async.wait_group 0;" ::: "memory");
                        }
                        __syncthreads();
                        if (i < rows) {
                            const float4 *xv = reinterpret_cast<const float4 *>(xs + (g % ROW_STAGES * ASSIGN_T + tid) * XS);
                            const float4 *cv = reinterpret_cast<const float4 *>(cs + l * CS + g % SL * W);
#pragma unroll
                            for (int q = 0; q < W / 4; q++) acc = add_sq4(acc, xv[q], cv[q]);
                        }
                        if (g % SL == SL - 1) settle(i, i < rows, acc, th);
                        __syncthreads();  // the stage is free for the fetch after next
                    }
                }
                __syncthreads();
                nl = list_n;
            }
            for (int base = 0; base < nl; base += ASSIGN_T * TR) {
                float xr[TR][D];
                int rr[TR];  // row of the item, -1: none
#pragma unroll
                for (int u = 0; u < TR; u++) {
                    const int i = base + tid + u * ASSIGN_T;
                    const bool ok = i < nl;
                    rr[u] = ok ? (bounded ? (int)list[i] : i) : -1;
#pragma unroll
                    for (int j4 = 0; j4 < D / 4; j4++) {
                        const float4 v = ok ? reinterpret_cast<const float4 *>(x + (int64_t)(I.lo + rr[u]) * D)[j4]
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
                        xr[u][4 * j4] = v.x;
                        xr[u][4 * j4 + 1] = v.y;
                        xr[u][4 * j4 + 2] = v.z;
                        xr[u][4 * j4 + 3] = v.w;
                    }
                }
                float best[TR];
                int bi[TR];
#pragma unroll
                for (int u = 0; u < TR; u++) {
                    best[u] = FLT_MAX;
                    bi[u] = 0;
                }
                for (int c = 0; c < k; c += CP) {
                    float acc[TR][CP];
#pragma unroll
                    for (int u = 0; u < TR; u++)
#pragma unroll
                        for (int p = 0; p < CP; p++) acc[u][p] = 0.f;
#pragma unroll
                    for (int j = 0; j < D; j++) {
#pragma unroll
                        for (int p = 0; p < CP; p++) {
                            const float cv = c + p < k ? cs[(c + p) * CS + j] : 0.f;
#pragma unroll
                            for (int u = 0; u < TR; u++) {
                                const float t = __fsub_rn(xr[u][j], cv);
                                acc[u][p] = __fadd_rn(acc[u][p], __fmul_rn(t, t));
                            }
                        }
                    }
#pragma unroll
                    for (int p = 0; p < CP; p++)
                        if (c + p < k)
#pragma unroll
                            for (int u = 0; u < TR; u++)
                                if (acc[u][p] < best[u]) {
                                    best[u] = acc[u][p];
                                    bi[u] = c + p;
                                }
                }
#pragma unroll
                for (int u = 0; u < TR; u++)
                    if (rr[u] >= 0) {
                        L[I.lo + rr[u]] = bi[u];
                        vals[rr[u]] = best[u];
                    }
            }
            __syncthreads();
            for (int i = tid; i < rows; i += ASSIGN_T) s += (double)vals[i];
        } else {
            for (int r = I.lo + tid; r < I.hi; r += ASSIGN_T) {
                const float *xr = x + (int64_t)r * d;
                float best = FLT_MAX;
                int bi = 0;
                for (int c = 0; c < k; c++) {
                    const float v = sqeuc_f32(xr, cs + c * d, d);
                    if (v < best) {
                        best = v;
                        bi = c;
                    }
                }
                L[r] = bi;
                s += (double)best;
            }
        }
        const double tot = block_sum_f64(s, red);
        if (tid == 0) partial[it] = tot;
        __syncthreads();
    }
}

constexpr int NEAR_T = 256, NEAR_PARTS = 4;

// Row thresholds of a bounded fit's next iteration, one per centre (CTA
// (fit, part): every NEAR_PARTS-th group of centres, a warp a centre, lanes over
// the others, all of the fit's centres in shared memory). thr[q] = (1 - rho) / 4
// of a lower bound of the smallest squared distance from centre q to another:
// a row whose computed distance m to q is below it is at least m (1 + 2 rho - 8g)
// > m from every other centre, in computed distances too, with g = (d + 4) u
// the relative error of a direct form and rho = (d + 8) 1e-6 (the triangle
// inequality: D(x, q) <= m (1 + 2g), so sqrt D(x, c) >= sqrt D(q, c) -
// sqrt D(x, q) >= sqrt D(x, q) (1 + rho - 2g)). Distances below 1e-30, where
// underflow would count, and NaN give 0: no row is below it.
__global__ void __launch_bounds__(NEAR_T)
    batch_near_kernel(const BFit *__restrict__ fits, const BState *__restrict__ state, const int *__restrict__ order,
                      const float *__restrict__ C, float *__restrict__ thr) {
    const int f = order[blockIdx.x];
    const BFit F = fits[f];
    if (!F.bounded || state[f].done) return;
    extern __shared__ __align__(16) float cs[];
    const int d = F.d, k = F.k, stride = d + 1;  // odd: lanes over rows meet no bank conflict
    const int tid = threadIdx.x, lane = tid & 31;
    if ((int)blockIdx.y * (NEAR_T / 32) >= k) return;
    const float *src = C + F.c_off + (int64_t)state[f].cur * k * d;
    for (int e = tid; e < k * d; e += NEAR_T) cs[e / d * stride + e % d] = src[e];
    __syncthreads();
    const float rho = (float)(d + 8) * 1e-6f;
    for (int q = (int)blockIdx.y * (NEAR_T / 32) + (tid >> 5); q < k; q += NEAR_PARTS * (NEAR_T / 32)) {
        float th = FLT_MAX;
        for (int c = lane; c < k; c += 32) {
            float v = 0.f;
#pragma unroll 8
            for (int j = 0; j < d; j++) {
                const float t = __fsub_rn(cs[c * stride + j], cs[q * stride + j]);
                v = __fmaf_rn(t, t, v);
            }
            const float b = 0.25f * __fsub_rd(v, bound32(v, 0.f, d)) * (1.0f - rho);
            if (c != q) th = b < th ? b : (b >= th ? th : 0.f);  // NaN: 0
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) th = fminf(th, __shfl_xor_sync(0xffffffffu, th, o));
        if (lane == 0) thr[F.k_off + q] = th > 1e-30f ? th : 0.f;
    }
}

// ---------------------------------------------------------------- update --
// Exact cluster sums for the f64 reduction: x = q1 2^(kb-23) + q2 2^(kb-46)
// + r2 with integer q1, q2 (the two-grid split: 2^ea <= max|x| < 2^(ea+1),
// kb = ea + 2, C1 = 1.5 2^kb, C2 = 1.5 2^(kb-23)); r2 is exact and zero
// unless |x| < 2^(ea-21), and then goes to a 128-bit fixed-point sum with F
// fraction bits (F = 124 - bitlen(n) - ea, so no sum can overflow; bits
// below 2^-F are truncated toward zero). Integer sums are order-free, so the
// result is the exact sum whatever the order, rounded once to f64.
__device__ __forceinline__ void add128u(uint64_t &lo, uint64_t &hi, uint64_t tlo, uint64_t thi) {
    asm("add.cc.u64 %0, %0, %2;\n\taddc.u64 %1, %1, %3;" : "+l"(lo), "+l"(hi) : "l"(tlo), "l"(thi));
}

__device__ __noinline__ void fixed_add_small(uint64_t &lo, uint64_t &hi, float x, int F) {
    const uint32_t b = __float_as_uint(x);
    const uint32_t ex = (b >> 23) & 0xFFu;
    if (ex == 0xFFu) return;
    const uint64_t m = (uint64_t)((b & 0x7FFFFFu) | (ex ? 0x800000u : 0u));
    const int s = (ex ? (int)ex : 1) - 150 + F;
    uint64_t tlo, thi;
    if (s >= 64) {
        tlo = 0;
        thi = m << (s - 64);
    } else if (s >= 0) {
        tlo = m << s;
        thi = s > 40 ? m >> (64 - s) : 0;
    } else {
        tlo = s > -32 ? m >> (-s) : 0;
        thi = 0;
    }
    if (b >> 31) {
        tlo = ~tlo;
        thi = ~thi;
        add128u(tlo, thi, 1ull, 0ull);
    }
    add128u(lo, hi, tlo, thi);
}

// Correctly rounded (nearest, ties to even) f64 value of the signed 128-bit
// fixed-point number (hi:lo) with F fraction bits.
__device__ double fixed128_to_double(uint64_t lo, uint64_t hi, int F) {
    const bool neg = (hi >> 63) != 0;
    if (neg) {
        lo = ~lo;
        hi = ~hi;
        add128u(lo, hi, 1ull, 0ull);
    }
    if (lo == 0 && hi == 0) return 0.0;
    const int msb = hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)lo);
    double r;
    if (msb <= 52) {
        r = scalbn((double)lo, -F);
    } else {
        const int sh = msb - 52;  // 1 <= sh <= 75
        uint64_t mant, rem_hi, rem_lo, half_hi, half_lo;
        if (sh < 64) {
            mant = (lo >> sh) | (sh ? (hi << (64 - sh)) : 0);
            rem_lo = lo & ((1ull << sh) - 1ull);
            rem_hi = 0;
            half_lo = 1ull << (sh - 1);
            half_hi = 0;
        } else {
            mant = hi >> (sh - 64);
            rem_lo = lo;
            rem_hi = sh > 64 ? hi & ((1ull << (sh - 64)) - 1ull) : 0;
            half_lo = sh == 64 ? (1ull << 63) : 0;
            half_hi = sh > 64 ? (1ull << (sh - 65)) : 0;
        }
        const bool above = rem_hi > half_hi || (rem_hi == half_hi && rem_lo > half_lo);
        const bool tie = rem_hi == half_hi && rem_lo == half_lo;
        if (above || (tie && (mant & 1ull))) mant += 1;
        r = scalbn((double)mant, sh - F);
    }
    return neg ? -r : r;
}

__device__ __forceinline__ int bitlen64(long long v) { return 64 - __clzll(v > 0 ? v : 1); }

// The f64 reduction's running sums: per (cluster, feature) of every fit the two
// integer sums, and the parts the grids cannot hold -- the 128-bit remainder in
// four 32-bit limbs (added limb by limb, carries resolved at the end) and what
// non-finite values occurred. Integer sums can be undone exactly: they carry
// over, and an iteration only moves the rows whose label changed. A fit with
// non-finite values, or one so long that the limbs could overflow (2^32
// additions of 32 bits), starts from zero each time instead.
struct BSums {
    unsigned long long *a1, *a2;  // two's complement
    unsigned long long *limb;     // [4] each
    uint32_t *flags;              // FLAG_*
    int *count;                   // per cluster
};
constexpr uint32_t FLAG_NAN = 1u, FLAG_PINF = 2u, FLAG_NINF = 4u, FLAG_LIMBS = 8u;

// The constants of one problem's exact sums.
struct ExactGrid {
    bool grids;
    int kb, F, b1, b2;
    float C1, C2;
    __device__ __forceinline__ ExactGrid(float amax, int n) {
        const int ea = amax > 0.f ? (int)((__float_as_uint(amax) >> 23) & 0xFFu) - 127 : -126;
        grids = ea >= -90 && ea <= 100;
        kb = ea + 2;
        F = 124 - bitlen64(n) - ea;
        C1 = grids ? ldexpf(1.5f, kb) : 0.f;
        C2 = grids ? ldexpf(1.5f, kb - 23) : 0.f;
        b1 = __float_as_int(C1);
        b2 = __float_as_int(C2);
    }
};

constexpr int ACC_T = 256;
constexpr unsigned LEAVES = 0x8000u;
constexpr int ACC_ROWS = 1024;  // rows of an item at most: with 5,000, the last fits' few items ran 130 us (1,024: 33 us)

// The f64 reduction's sums of one (fit, row range) item: the item's rows whose
// label changed, once for the cluster they join and once for the one they
// leave, grouped by cluster in shared memory; then a thread per (cluster,
// feature) over the cluster's entries (neighbouring threads read neighbouring
// features) and one addition to the fit's sums. Integer sums are order-free, so any
// number of CTAs can share a fit: 64 problems x 10 runs took 427 ms of 994
// with one CTA a fit, its largest fits' sorts and chains last; 28 of 107 with
// every row added in every iteration.
__global__ void __launch_bounds__(ACC_T) batch_accum_kernel(const float *__restrict__ X, const BFit *__restrict__ fits,
                                                            const BState *__restrict__ state,
                                                            const BItem *__restrict__ items, int nitems,
                                                            const int *__restrict__ lab, int *__restrict__ prev,
                                                            const float *__restrict__ pamax, BSums S) {
    __shared__ unsigned short ids[2 * ACC_ROWS];  // row, LEAVES: subtracted
    __shared__ int hist[MAX_K], off[MAX_K], net[MAX_K];
    __shared__ int todo[ACC_T], todo_n;
    const int tid = threadIdx.x, lane = tid & 31;
    // ACC_T of the block's items (every gridDim.x-th) looked at together: most
    // belong to converged fits (30 us an iteration one by one)
    for (int it0 = blockIdx.x; it0 < nitems; it0 += ACC_T * gridDim.x) {
        if (tid == 0) todo_n = 0;
        __syncthreads();
        const int64_t mine = it0 + (int64_t)tid * gridDim.x;
        if (mine < nitems && !state[items[mine].fit].done) todo[atomicAdd(&todo_n, 1)] = (int)mine;
        __syncthreads();
        for (int q = 0; q < todo_n; q++) {
            const BItem I = items[todo[q]];
            const BFit F = fits[I.fit];
            const int d = F.d, k = F.k, rows = I.hi - I.lo;
            const bool full = state[I.fit].full != 0;
            int nw[ACC_ROWS / ACC_T], old[ACC_ROWS / ACC_T];  // a row without a change: equal
            bool any = false;
#pragma unroll
            for (int u = 0; u < ACC_ROWS / ACC_T; u++) {
                const int r = u * ACC_T + tid;
                nw[u] = old[u] = -1;
                if (r < rows) {
                    const int64_t at = F.s_off + I.lo + r;
                    nw[u] = lab[at];
                    if (!full) old[u] = prev[at];
                    if (nw[u] != old[u]) {
                        prev[at] = nw[u];
                        any = true;
                    }
                }
            }
            if (!__syncthreads_or(any)) continue;
            for (int c = tid; c < k; c += ACC_T) hist[c] = net[c] = 0;
            __syncthreads();
#pragma unroll
            for (int u = 0; u < ACC_ROWS / ACC_T; u++) {
                if (nw[u] == old[u]) continue;
                atomicAdd(&hist[nw[u]], 1);
                atomicAdd(&net[nw[u]], 1);
                if (old[u] >= 0) {
                    atomicAdd(&hist[old[u]], 1);
                    atomicSub(&net[old[u]], 1);
                }
            }
            __syncthreads();
            if (tid < 32) {
                int base = 0;
                for (int c0 = 0; c0 < k; c0 += 32) {
                    const int v = c0 + lane < k ? hist[c0 + lane] : 0;
                    int s = v;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int u = __shfl_up_sync(0xffffffffu, s, o);
                        if (lane >= o) s += u;
                    }
                    if (c0 + lane < k) {
                        off[c0 + lane] = base + s - v;
                        if (net[c0 + lane]) atomicAdd(S.count + F.k_off + c0 + lane, net[c0 + lane]);
                    }
                    base += __shfl_sync(0xffffffffu, s, 31);
                }
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < ACC_ROWS / ACC_T; u++) {
                if (nw[u] == old[u]) continue;
                const unsigned short r = (unsigned short)(u * ACC_T + tid);
                ids[atomicAdd(&off[nw[u]], 1)] = r;
                if (old[u] >= 0) ids[atomicAdd(&off[old[u]], 1)] = (unsigned short)(r | LEAVES);
            }
            __syncthreads();  // off[c] is now the end of cluster c's entries
            const ExactGrid g(pamax[F.prob], F.n);
            const float *x = X + F.x_off + (int64_t)I.lo * d;
            const int64_t a_off = F.c_off / 2;
            // few clusters and features: several threads share one's rows
            const int kd = k * d, nsub = max(1, ACC_T / kd);
            for (int q = tid; q < kd * nsub; q += ACC_T) {
                const int sub = q / kd, pr = q - sub * kd;
                const int c = pr / d, j = pr - c * d;
                const int cnt = hist[c], o = off[c] - cnt;
                long long a1 = 0, a2 = 0;
                uint64_t slo = 0, shi = 0;
                uint32_t fl = 0;
#pragma unroll 8
                for (int m = sub; m < cnt; m += nsub) {
                    const unsigned id = ids[o + m];
                    const float xr = x[(int64_t)(id & (LEAVES - 1u)) * d + j];
                    const float xv = id & LEAVES ? -xr : xr;  // every step below is odd in xv
                    if (!(fabsf(xv) < INFINITY)) {
                        fl |= xv != xv ? FLAG_NAN : (xv > 0.f ? FLAG_PINF : FLAG_NINF);
                    } else if (g.grids) {
                        const float s1 = __fadd_rn(xv, g.C1);
                        a1 += __float_as_int(s1) - g.b1;
                        const float r = __fsub_rn(xv, __fsub_rn(s1, g.C1));
                        const float s2 = __fadd_rn(r, g.C2);
                        a2 += __float_as_int(s2) - g.b2;
                        const float r2 = __fsub_rn(r, __fsub_rn(s2, g.C2));
                        if (r2 != 0.f) fixed_add_small(slo, shi, r2, g.F);
                    } else {
                        fixed_add_small(slo, shi, xv, g.F);
                    }
                }
                const int64_t e = a_off + pr;
                if (a1) atomicAdd(S.a1 + e, (unsigned long long)a1);
                if (a2) atomicAdd(S.a2 + e, (unsigned long long)a2);
                if (slo | shi) {
                    fl |= FLAG_LIMBS;
                    atomicAdd(S.limb + 4 * e, slo & 0xFFFFFFFFull);
                    atomicAdd(S.limb + 4 * e + 1, slo >> 32);
                    atomicAdd(S.limb + 4 * e + 2, shi & 0xFFFFFFFFull);
                    atomicAdd(S.limb + 4 * e + 3, shi >> 32);
                }
                if (fl) atomicOr(S.flags + e, fl);
            }
            __syncthreads();  // ids and hist are refilled
        }
        __syncthreads();  // and todo
    }
}

// What ends an iteration of fit f, by thread 0: sqrt of the largest squared
// shift against tol, the inertia's partials in item order, the state.
__device__ __forceinline__ void finish_fit(const BFit &F, BState *state, int f, float m2,
                                           const double *__restrict__ partial, int *active) {
    const float shift = __fsqrt_rn(m2);
    BState st = state[f];
    st.n_iter += 1;
    st.cur = 1 - st.cur;
    if (shift < F.tol || st.n_iter >= F.max_iter) {
        // a serial chain of FP64 additions (10 us for 312 items): the last iteration's only
        double in = 0.0;
        for (int it = 0; it < F.n_items; it++) in += partial[F.first_item + it];
        st.inertia = in;
        st.done = 1;
        atomicSub(active, 1);
    }
    state[f] = st;
}

// The f64 reduction's new centres from the sums (kept for the next iteration,
// or left zero): each sum rounded once to f64, the mean once to f32.
__global__ void __launch_bounds__(UPDATE_T) batch_means_kernel(const BFit *__restrict__ fits, BState *__restrict__ state,
                                                               const int *__restrict__ order, int nf, int *counter,
                                                               float *__restrict__ C, const double *__restrict__ partial,
                                                               int *active, const float *__restrict__ pamax, BSums S) {
    __shared__ int q_sh;
    __shared__ float red[UPDATE_T / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    while (true) {
        if (tid == 0) q_sh = atomicAdd(counter, 1);
        __syncthreads();
        const int q = q_sh;
        __syncthreads();
        if (q >= nf) break;
        const int f = order[q];
        if (state[f].done) continue;
        const BFit F = fits[f];
        const int d = F.d, k = F.k, cur = state[f].cur;
        const float *oldc = C + F.c_off + (int64_t)cur * k * d;
        float *newc = C + F.c_off + (int64_t)(1 - cur) * k * d;
        bool full = !F.keep_sums;  // the next iteration starts from zero sums
        const ExactGrid g(pamax[F.prob], F.n);
        const int64_t a_off = F.c_off / 2;
        for (int pr = tid; pr < k * d; pr += UPDATE_T) {
            const int64_t e = a_off + pr;
            const int cnt = S.count[F.k_off + pr / d];
            if (cnt == 0) {
                newc[pr] = oldc[pr];  // empty cluster keeps its centre
                continue;
            }
            const uint32_t fl = S.flags[e];
            double sum;
            full |= (fl & (FLAG_NAN | FLAG_PINF | FLAG_NINF)) != 0;
            if (fl & (FLAG_NAN | FLAG_PINF | FLAG_NINF)) {  // IEEE f64 summation of the specials
                sum = ((fl & FLAG_NAN) || (fl & (FLAG_PINF | FLAG_NINF)) == (FLAG_PINF | FLAG_NINF))
                          ? __longlong_as_double(0x7FF8000000000000LL)
                      : (fl & FLAG_PINF) ? __longlong_as_double(0x7FF0000000000000LL)
                                         : __longlong_as_double((long long)0xFFF0000000000000ULL);
            } else {
                uint64_t slo = 0, shi = 0;
                if (fl & FLAG_LIMBS) {
                    for (int l = 0; l < 4; l++) {
                        const unsigned __int128 v = (unsigned __int128)S.limb[4 * e + l] << (32 * l);
                        add128u(slo, shi, (uint64_t)v, (uint64_t)(v >> 64));
                    }
                }
                if (g.grids) {
                    const __int128 v1 = (__int128)(long long)S.a1[e] << (g.kb - 23 + g.F);
                    const __int128 v2 = (__int128)(long long)S.a2[e] << (g.kb - 46 + g.F);
                    add128u(slo, shi, (uint64_t)v1, (uint64_t)((unsigned __int128)v1 >> 64));
                    add128u(slo, shi, (uint64_t)v2, (uint64_t)((unsigned __int128)v2 >> 64));
                }
                sum = fixed128_to_double(slo, shi, g.F);
            }
            newc[pr] = __double2float_rn(__ddiv_rn(sum, (double)cnt));
        }
        full = __syncthreads_or(full);
        if (full) {
            for (int pr = tid; pr < k * d; pr += UPDATE_T) {
                const int64_t e = a_off + pr;
                S.a1[e] = S.a2[e] = 0;
                S.flags[e] = 0;
                for (int l = 0; l < 4; l++) S.limb[4 * e + l] = 0;
            }
            for (int c = tid; c < k; c += UPDATE_T) S.count[F.k_off + c] = 0;
        }
        if (tid == 0) state[f].full = full;
        // the largest squared shift (NaN shifts never raise it)
        float ms = 0.f;
        for (int c = tid; c < k; c += UPDATE_T) {
            const float sh = sqeuc_f32(newc + (int64_t)c * d, oldc + (int64_t)c * d, d);
            if (sh > ms) ms = sh;
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) ms = fmaxf(ms, __shfl_xor_sync(0xffffffffu, ms, o));
        if (lane == 0) red[warp] = ms;
        __syncthreads();
        if (tid == 0) {
            float m2 = 0.f;
            for (int w = 0; w < UPDATE_T / 32; w++) m2 = fmaxf(m2, red[w]);
            finish_fit(F, state, f, m2, partial, active);
        }
        __syncthreads();
    }
}

// The reference reduction: row-order f32 sums, one CTA a fit.
__global__ void __launch_bounds__(UPDATE_T) batch_update_kernel(const float *__restrict__ X,
                                                                const BFit *__restrict__ fits,
                                                                BState *__restrict__ state,
                                                                const int *__restrict__ order, int nf, int *counter,
                                                                float *__restrict__ C, const int *__restrict__ lab,
                                                                int *__restrict__ mem,
                                                                const double *__restrict__ partial, int *active) {
    constexpr int NW = UPDATE_T / 32;
    __shared__ int wrun[NW][MAX_K];
    __shared__ int hist[MAX_K], off[MAX_K];
    __shared__ int q_sh;
    __shared__ float red[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned full = 0xffffffffu;
    while (true) {
        if (tid == 0) q_sh = atomicAdd(counter, 1);
        __syncthreads();
        const int q = q_sh;
        __syncthreads();
        if (q >= nf) break;
        const int f = order[q];
        if (state[f].done) continue;
        const BFit F = fits[f];
        const int n = F.n, d = F.d, k = F.k;
        const int *L = lab + F.s_off;
        int *M = mem + F.s_off;
        // counting sort, stable: warp w owns the contiguous rows [w R, (w+1) R)
        const int R = (n + NW - 1) / NW;
        const int rlo = min(n, warp * R), rhi = min(n, rlo + R);
        for (int e = tid; e < NW * k; e += UPDATE_T) wrun[e / k][e % k] = 0;
        __syncthreads();
        for (int i = rlo + lane; i < rhi; i += 32) atomicAdd(&wrun[warp][L[i]], 1);
        __syncthreads();
        for (int c = tid; c < k; c += UPDATE_T) {
            int t = 0;
            for (int w = 0; w < NW; w++) t += wrun[w][c];
            hist[c] = t;
        }
        __syncthreads();
        if (tid == 0) {
            int acc = 0;
            for (int c = 0; c < k; c++) {
                off[c] = acc;
                acc += hist[c];
            }
        }
        __syncthreads();
        for (int c = tid; c < k; c += UPDATE_T) {
            int start = off[c];
            for (int w = 0; w < NW; w++) {
                const int t = wrun[w][c];
                wrun[w][c] = start;
                start += t;
            }
        }
        __syncthreads();
        for (int base = rlo; base < rhi; base += 32) {
            const int i = base + lane;
            const int l = i < rhi ? L[i] : -1;
            const unsigned peers = __match_any_sync(full, l);
            const int leader = __ffs(peers) - 1;
            const int rank = __popc(peers & ((1u << lane) - 1u));
            int b = 0;
            if (lane == leader && l >= 0) {
                b = wrun[warp][l];
                wrun[warp][l] = b + __popc(peers);
            }
            b = __shfl_sync(full, b, leader);
            if (l >= 0) M[b + rank] = i;
        }
        __syncthreads();
        const int cur = state[f].cur;
        const float *oldc = C + F.c_off + (int64_t)cur * k * d;
        float *newc = C + F.c_off + (int64_t)(1 - cur) * k * d;
        const float *x = X + F.x_off;
        for (int pr = tid; pr < k * d; pr += UPDATE_T) {
            const int c = pr / d, j = pr - c * d;
            const int cnt = hist[c], o = off[c];
            if (cnt == 0) {
                newc[pr] = oldc[pr];  // empty cluster keeps its centre
                continue;
            }
            // values of the cluster's rows in row order, loaded 8 ahead, their rows' numbers 16
            float cur8[8], nxt8[8];
            int row8[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                cur8[u] = u < cnt ? x[(int64_t)M[o + u] * d + j] : 0.f;
                row8[u] = 8 + u < cnt ? M[o + 8 + u] : -1;
            }
            float acc = 0.f;
            for (int m = 0; m < cnt; m += 8) {
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    nxt8[u] = row8[u] >= 0 ? x[(int64_t)row8[u] * d + j] : 0.f;
                    row8[u] = m + 16 + u < cnt ? M[o + m + 16 + u] : -1;
                }
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (m + u < cnt) acc = __fadd_rn(acc, cur8[u]);
#pragma unroll
                for (int u = 0; u < 8; u++) cur8[u] = nxt8[u];
            }
            newc[pr] = __fdiv_rn(acc, (float)cnt);  // counts as F are exact below 2^24
        }
        __syncthreads();
        // sqrt of the largest squared shift (NaN shifts never raise it)
        float ms = 0.f;
        for (int c = tid; c < k; c += UPDATE_T) {
            const float sh = sqeuc_f32(newc + (int64_t)c * d, oldc + (int64_t)c * d, d);
            if (sh > ms) ms = sh;
        }
#pragma unroll
        for (int o2 = 16; o2 >= 1; o2 >>= 1) ms = fmaxf(ms, __shfl_xor_sync(full, ms, o2));
        if (lane == 0) red[warp] = ms;
        __syncthreads();
        if (tid == 0) {
            float m2 = 0.f;
            for (int w = 0; w < NW; w++) m2 = fmaxf(m2, red[w]);
            finish_fit(F, state, f, m2, partial, active);
        }
        __syncthreads();
    }
}

// max |x| over the finite values of each problem (the exact sums' scale);
// amax starts at zero, and non-negative floats order as their bits.
constexpr int AMAX_PARTS = 32;  // CTAs a problem
__global__ void batch_amax_kernel(const float *__restrict__ X, const int64_t *__restrict__ xoff,
                                  const int64_t *__restrict__ xlen, float *__restrict__ amax) {
    const int p = blockIdx.x / AMAX_PARTS, part = blockIdx.x % AMAX_PARTS;
    const float *x = X + xoff[p];
    float m = 0.f;
    for (int64_t e = (int64_t)part * blockDim.x + threadIdx.x; e < xlen[p]; e += (int64_t)AMAX_PARTS * blockDim.x) {
        const float a = fabsf(x[e]);
        if (a < INFINITY) m = fmaxf(m, a);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int *>(amax + p), __float_as_int(m));
}

__global__ void batch_labels_u64_kernel(const int *__restrict__ l, int n, uint64_t *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (uint64_t)l[i];
}

// --------------------------------------------------------------- host side --
int dbucket(int d) { return d == 8 ? 0 : d == 16 ? 1 : d == 32 ? 2 : d == 64 ? 3 : 4; }
int kbucket(int k) { return k <= 16 ? 0 : k <= 32 ? 1 : k <= 64 ? 2 : 3; }
int bucket_d(int b) { static const int v[5] = {8, 16, 32, 64, 0}; return v[b / 4]; }

using AssignFn = void (*)(const float *, const BFit *, const BState *, const BItem *, int, int *, const float *,
                          const float *, int *, double *);

template <int D>
AssignFn pick_variant(int v) {
    switch (v) {
        case 0: return batch_assign_kernel<D, 1, 1>;
        case 1: return batch_assign_kernel<D, 2, 1>;
        case 2: return batch_assign_kernel<D, 1, 2>;
        case 3: return batch_assign_kernel<D, 2, 2>;
        default: return batch_assign_kernel<D, (D <= 32 ? 4 : 2), 1>;
    }
}

AssignFn assign_fn(int bucket, int v) {
    switch (bucket_d(bucket)) {
        case 8: return pick_variant<8>(v);
        case 16: return pick_variant<16>(v);
        case 32: return pick_variant<32>(v);
        case 64: return v <= 2 ? pick_variant<64>(v) : pick_variant<64>(1);
        default: return batch_assign_kernel<0, 1, 1>;
    }
}

int n_variants(int bucket) {
    const int d = bucket_d(bucket);
    return d == 0 ? 1 : d == 64 ? 3 : NVARIANTS;
}

}  // namespace

void Branches::make() {
    if (!fork) FK_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    for (int q = 0; q < N; q++) {
        if (!stream[q]) FK_CUDA(cudaStreamCreateWithFlags(&stream[q], cudaStreamNonBlocking));
        if (!join[q]) FK_CUDA(cudaEventCreateWithFlags(&join[q], cudaEventDisableTiming));
    }
}

void Branches::release() {
    for (int q = 0; q < N; q++) {
        if (join[q]) cudaEventDestroy(join[q]);
        if (stream[q]) cudaStreamDestroy(stream[q]);
        join[q] = nullptr;
        stream[q] = nullptr;
    }
    if (fork) cudaEventDestroy(fork);
    fork = nullptr;
}

fk_status batched_fit_impl(Ctx &ctx, fk_batch_problem *P, int64_t np, int reduction, fk_batch_report *rep) {
    if (np < 0 || (np > 0 && !P)) {
        set_error("problems is NULL or n_problems is negative");
        return FK_ERR_INVALID_PARAMETER;
    }
    if (reduction != FK_REDUCE_REFERENCE && reduction != FK_REDUCE_F64) {
        set_error("unknown reduction %d", reduction);
        return FK_ERR_INVALID_PARAMETER;
    }
    // Validation of every problem first, in the order of kmeans.rs:421-449.
    for (int64_t p = 0; p < np; p++) {
        const fk_batch_problem &q = P[p];
        if (q.n_clusters <= 0) {
            set_error("problem %lld: Invalid parameter `n_clusters`: must be at least 1", (long long)p);
            return FK_ERR_INVALID_PARAMETER;
        }
        if (q.n <= 0 || q.n < q.n_clusters) {
            set_error("problem %lld: Insufficient samples: need at least %lld, got %lld", (long long)p,
                      (long long)q.n_clusters, (long long)(q.n < 0 ? 0 : q.n));
            return FK_ERR_INSUFFICIENT_SAMPLES;
        }
        if (q.n_init <= 0) {
            set_error("problem %lld: Invalid parameter `n_init`: must be at least 1", (long long)p);
            return FK_ERR_INVALID_PARAMETER;
        }
        if (q.max_iter < 0 || q.d < 1) {
            set_error("problem %lld: Invalid parameter `max_iter`/`d`", (long long)p);
            return FK_ERR_INVALID_PARAMETER;
        }
        if (!q.x || !q.centers_out || !q.labels_out || !q.inertia_out || !q.n_iter_out) {
            set_error("problem %lld: required pointer is NULL", (long long)p);
            return FK_ERR_NULL_POINTER;
        }
        if (q.n_clusters > MAX_K || q.d > MAX_D || q.n_clusters * q.d > MAX_KD || q.n > INT32_MAX / 2 ||
            q.max_iter > INT32_MAX) {
            set_error("problem %lld: batched fits support k <= %d, d <= %d, k*d <= %d (got k=%lld d=%lld)",
                      (long long)p, MAX_K, MAX_D, MAX_KD, (long long)q.n_clusters, (long long)q.d);
            return FK_ERR_UNSUPPORTED;
        }
    }
    if (rep) {
        double *fi = rep->fit_inertia;
        int64_t *fn = rep->fit_n_iter;
        memset(rep, 0, sizeof(*rep));
        rep->fit_inertia = fi;
        rep->fit_n_iter = fn;
        for (int b = 0; b < NBUCKETS; b++) rep->bucket_variant[b] = -1;
    }
    if (np == 0) return FK_OK;
    ctx.bind();
    cudaStream_t s = ctx.stream;
    Events<6> ev;
    FK_CUDA(cudaEventRecord(ev[0], s));

    // ---- layout
    std::vector<int64_t> xoff(np);
    int64_t xtot = 0;
    for (int64_t p = 0; p < np; p++) {
        xoff[p] = xtot;
        xtot += (P[p].n * P[p].d + 3) / 4 * 4;  // 16-byte aligned starts
    }
    std::vector<BFit> fits;
    std::vector<int> fit_prob, fit_run;
    int64_t soff = 0, coff = 0, koff = 0;
    bool bounds_pay = false;
    for (int64_t p = 0; p < np; p++) {
        const fk_batch_problem &q = P[p];
        for (int64_t r = 0; r < q.n_init; r++) {
            BFit F;
            memset(&F, 0, sizeof(F));
            F.x_off = xoff[p];
            F.s_off = soff;
            F.c_off = coff;
            F.k_off = koff;
            F.n = (int32_t)q.n;
            F.d = (int32_t)q.d;
            F.k = (int32_t)q.n_clusters;
            F.max_iter = (int32_t)q.max_iter;
            F.tol = (float)q.tol;
            F.seed = q.random_state + (uint64_t)r;
            F.prob = (int32_t)p;
            F.keep_sums = q.n * std::max<int64_t>(q.max_iter, 1) <= ((int64_t)1 << 30);
            // the thresholds cost k^2 d in one CTA group a fit: little beside n k d
            F.bounded = dbucket(F.d) < 4 && F.k <= BOUND_K && (int64_t)F.n >= 16 * (int64_t)F.k;
            bounds_pay = bounds_pay || (F.bounded && F.n >= 2048 && F.k >= 8);
            fits.push_back(F);
            fit_prob.push_back((int)p);
            fit_run.push_back((int)r);
            soff += q.n;
            coff += 2 * q.n_clusters * q.d;
            koff += q.n_clusters;
        }
    }
    // a call of small fits alone: the thresholds' launch is longer than what they save
    // (100 fits of 1,000 x 8, 4 clusters: 30.1 us an iteration with, 26.1 without)
    if (!bounds_pay)
        for (BFit &F : fits) F.bounded = 0;
    const int nf = (int)fits.size();
    // work items: chunks of rows, grouped by (d, k) bucket, largest fits first
    auto cost = [&](int f) { return (double)fits[f].n * fits[f].k * fits[f].d; };
    std::vector<int> byc(nf);
    std::iota(byc.begin(), byc.end(), 0);
    std::stable_sort(byc.begin(), byc.end(), [&](int a, int b) { return cost(a) > cost(b); });
    std::vector<BItem> items;
    int bstart[NBUCKETS + 1] = {0};
    for (int b = 0; b < NBUCKETS; b++) {
        bstart[b] = (int)items.size();
        for (int f : byc) {
            BFit &F = fits[f];
            if (dbucket(F.d) * 4 + kbucket(F.k) != b) continue;
            const int ch = std::max(128, std::min(ITEM_ROWS, (int)(4194304.0 / ((double)F.k * F.d * 3.0)) / 128 * 128));
            F.first_item = (int)items.size();
            for (int lo = 0; lo < F.n; lo += ch) items.push_back(BItem{f, lo, std::min(F.n, lo + ch), 0});
            F.n_items = (int)items.size() - F.first_item;
        }
    }
    bstart[NBUCKETS] = (int)items.size();
    const size_t n_assign = items.size();
    if (reduction == FK_REDUCE_F64)  // the sums' items follow the assignment's
        for (size_t i = 0; i < n_assign; i++)
            for (int lo = items[i].lo, hi = items[i].hi; lo < hi; lo += ACC_ROWS)
                items.push_back(BItem{items[i].fit, lo, std::min(hi, lo + ACC_ROWS), 0});
    const size_t n_sums = items.size() - n_assign;
    std::vector<int> kpp_order;
    for (int f : byc)
        if (!P[fit_prob[f]].init) kpp_order.push_back(f);

    // ---- device buffers
    float *X = (float *)ctx.get(BUF_BX, sizeof(float) * (size_t)xtot + 16);
    BFit *dfits = (BFit *)ctx.get(BUF_BFITS, sizeof(BFit) * (size_t)nf);
    BState *dstate = (BState *)ctx.get(BUF_BSTATE, sizeof(BState) * (size_t)nf);
    BItem *ditems = (BItem *)ctx.get(BUF_BITEMS, sizeof(BItem) * items.size() + 16);
    double *dpart = (double *)ctx.get(BUF_BPART, sizeof(double) * items.size() + 16);
    int *dorder = (int *)ctx.get(BUF_BORDER, sizeof(int) * (size_t)nf + 16);
    int *dctr = (int *)ctx.get(BUF_BCTR, sizeof(int) * 32);
    int *dlab = (int *)ctx.get(BUF_BLAB, sizeof(int) * (size_t)soff + 16);
    int *dmem = (int *)ctx.get(BUF_BMEM, sizeof(int) * (size_t)soff + 16);
    float *dthr = (float *)ctx.get(BUF_BTHR, sizeof(float) * (size_t)koff + 16);
    float *dC = (float *)ctx.get(BUF_BCEN, sizeof(float) * (size_t)coff + 16);
    int64_t *dxo = (int64_t *)ctx.get(BUF_BXOFF, sizeof(int64_t) * (size_t)(2 * np) + sizeof(float) * (size_t)np + 64);
    float *damax = (float *)(dxo + 2 * np);
    BSums sums{};
    if (reduction == FK_REDUCE_F64) {
        const size_t ne = (size_t)(coff / 2);
        unsigned char *b = (unsigned char *)ctx.get(BUF_BSUMS, ne * 52 + sizeof(int) * (size_t)koff + 16);
        sums.a1 = (unsigned long long *)b;
        sums.a2 = sums.a1 + ne;
        sums.limb = sums.a2 + ne;
        sums.flags = (uint32_t *)(sums.limb + 4 * ne);
        sums.count = (int *)(sums.flags + ne);
        FK_CUDA(cudaMemsetAsync(b, 0, ne * 52 + sizeof(int) * (size_t)koff, s));
    }
    for (int64_t p = 0; p < np; p++)
        FK_CUDA(cudaMemcpyAsync(X + xoff[p], P[p].x, sizeof(float) * (size_t)(P[p].n * P[p].d), cudaMemcpyDefault,
                                s));
    FK_CUDA(cudaMemcpyAsync(dfits, fits.data(), sizeof(BFit) * (size_t)nf, cudaMemcpyHostToDevice, s));
    {
        std::vector<int64_t> xol(2 * np);
        for (int64_t p = 0; p < np; p++) {
            xol[p] = xoff[p];
            xol[np + p] = P[p].n * P[p].d;
        }
        FK_CUDA(cudaMemcpyAsync(dxo, xol.data(), sizeof(int64_t) * xol.size(), cudaMemcpyHostToDevice, s));
        FK_CUDA(cudaStreamSynchronize(s));  // xol is host stack memory
        if (reduction == FK_REDUCE_F64) {
            FK_CUDA(cudaMemsetAsync(damax, 0, sizeof(float) * (size_t)np, s));
            batch_amax_kernel<<<(unsigned)(np * AMAX_PARTS), 256, 0, s>>>(X, dxo, dxo + np, damax);
            FK_LAUNCH_CHECK();
        }
    }
    if (!items.empty())
        FK_CUDA(cudaMemcpyAsync(ditems, items.data(), sizeof(BItem) * items.size(), cudaMemcpyHostToDevice, s));
    FK_CUDA(cudaMemcpyAsync(dorder, byc.data(), sizeof(int) * byc.size(), cudaMemcpyHostToDevice, s));
    std::vector<BState> st0(nf);
    int active = 0;
    for (int f = 0; f < nf; f++) {
        st0[f].inertia = (double)FLT_MAX;
        st0[f].cur = 0;
        st0[f].n_iter = 0;
        st0[f].done = fits[f].max_iter == 0 ? 1 : 0;
        st0[f].full = 1;
        active += st0[f].done ? 0 : 1;
    }
    FK_CUDA(cudaMemcpyAsync(dstate, st0.data(), sizeof(BState) * (size_t)nf, cudaMemcpyHostToDevice, s));
    FK_CUDA(cudaMemsetAsync(dlab, 0, sizeof(int) * (size_t)soff, s));
    FK_CUDA(cudaMemsetAsync(dctr, 0, sizeof(int) * 32, s));
    FK_CUDA(cudaMemcpyAsync(dctr + 31, &active, sizeof(int), cudaMemcpyHostToDevice, s));
    for (int f = 0; f < nf; f++) {
        const fk_batch_problem &q = P[fit_prob[f]];
        if (q.init) {
            const int64_t run = fit_run[f];
            FK_CUDA(cudaMemcpyAsync(dC + fits[f].c_off, q.init + run * q.n_clusters * q.d,
                                    sizeof(float) * (size_t)(q.n_clusters * q.d), cudaMemcpyDefault, s));
        }
    }
    FK_CUDA(cudaEventRecord(ev[1], s));

    // ---- k-means++ (fk_kpp.cu): every fit's seeding, a centre of each per step
    if (!kpp_order.empty()) {
        std::vector<KppJob> jobs;
        for (int f : kpp_order) {
            KppJob j;
            j.x = X + fits[f].x_off;
            j.n = fits[f].n;
            j.d = fits[f].d;
            j.k = fits[f].k;
            j.seed = fits[f].seed;
            j.centers = dC + fits[f].c_off;  // buffer 0
            j.nan_direct = false;
            jobs.push_back(j);
        }
        run_kmeanspp<float>(ctx, jobs, nullptr);
    }
    FK_CUDA(cudaEventRecord(ev[2], s));

    // ---- autotuner: time every variant of each new (d, k) bucket on its items
    size_t bsmem[NBUCKETS] = {0};
    size_t near_smem = 0;
    for (const BFit &F : fits) {
        const int b = dbucket(F.d) * 4 + kbucket(F.k);
        bsmem[b] = std::max(bsmem[b], bucket_d(b) ? assign_smem(F.d, F.k) : sizeof(float) * (size_t)(F.k * F.d));
        if (F.bounded) near_smem = std::max(near_smem, sizeof(float) * (size_t)F.k * (size_t)(F.d + 1));
    }
    if (near_smem)
        FK_CUDA(cudaFuncSetAttribute((const void *)batch_near_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)near_smem));
    int64_t tuned = 0;
    for (int b = 0; b < NBUCKETS; b++) {
        const int cnt = bstart[b + 1] - bstart[b];
        if (cnt == 0) continue;
        const size_t smem = bsmem[b];
        for (int v = 0; v < n_variants(b); v++)
            FK_CUDA(cudaFuncSetAttribute((const void *)assign_fn(b, v), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)std::max<size_t>(smem, 1)));
        if (ctx.batch_variant[b] >= 0) continue;
        const int grid = std::min(cnt, ctx.num_sms * 8);
        float bestms = 1e30f;
        int bestv = 0;
        for (int v = 0; v < n_variants(b); v++) {
            FK_CUDA(cudaMemsetAsync(dctr + b, 0, sizeof(int), s));
            FK_CUDA(cudaEventRecord(ev[4], s));
            assign_fn(b, v)<<<grid, ASSIGN_T, smem, s>>>(X, dfits, dstate, ditems + bstart[b], cnt, dctr + b, dC,
                                                          dthr, dlab, dpart + bstart[b]);
            FK_LAUNCH_CHECK();
            FK_CUDA(cudaEventRecord(ev[5], s));
            FK_CUDA(cudaEventSynchronize(ev[5]));
            float ms = 0.f;
            FK_CUDA(cudaEventElapsedTime(&ms, ev[4], ev[5]));
            if (ms < bestms) {
                bestms = ms;
                bestv = v;
            }
        }
        ctx.batch_variant[b] = bestv;
        tuned++;
    }
    FK_CUDA(cudaEventRecord(ev[3], s));

    // ---- Lloyd iterations: one captured iteration, replayed. The buckets'
    // assignments are independent: branches of the graph where there are several
    // (streams made for every call took 0.1 ms of a call of two 200 x 8 problems).
    int nbuckets = 0;
    for (int b = 0; b < NBUCKETS; b++) nbuckets += bstart[b + 1] > bstart[b];
    const int forks = nbuckets > 1 ? std::min(nbuckets, Branches::N) : 0;
    Branches &side = ctx.branches;
    if (forks) side.make();
    auto one_iteration = [&]() {
        FK_CUDA(cudaMemsetAsync(dctr, 0, sizeof(int) * 22, s));
        if (forks) FK_CUDA(cudaEventRecord(side.fork, s));
        for (int q = 0; q < forks; q++) FK_CUDA(cudaStreamWaitEvent(side.stream[q], side.fork, 0));
        int at = 0;
        for (int b = 0; b < NBUCKETS; b++) {
            const int cnt = bstart[b + 1] - bstart[b];
            if (cnt == 0) continue;
            const int grid = std::min(cnt, ctx.num_sms * 8);
            assign_fn(b, ctx.batch_variant[b])<<<grid, ASSIGN_T, bsmem[b], forks ? side.stream[at++ % forks] : s>>>(
                X, dfits, dstate, ditems + bstart[b], cnt, dctr + b, dC, dthr, dlab, dpart + bstart[b]);
        }
        for (int q = 0; q < forks; q++) {
            FK_CUDA(cudaEventRecord(side.join[q], side.stream[q]));
            FK_CUDA(cudaStreamWaitEvent(s, side.join[q], 0));
        }
        const int ug = std::min(nf, ctx.num_sms * 4);
        if (reduction == FK_REDUCE_F64) {
            batch_accum_kernel<<<(unsigned)std::min<size_t>(n_sums, (size_t)ctx.num_sms * 8), ACC_T, 0, s>>>(
                X, dfits, dstate, ditems + n_assign, (int)n_sums, dlab, dmem, damax, sums);
            batch_means_kernel<<<ug, UPDATE_T, 0, s>>>(dfits, dstate, dorder, nf, dctr + 20, dC, dpart, dctr + 31,
                                                       damax, sums);
        } else {
            batch_update_kernel<<<ug, UPDATE_T, 0, s>>>(X, dfits, dstate, dorder, nf, dctr + 20, dC, dlab, dmem, dpart,
                                                        dctr + 31);
        }
        if (near_smem)
            batch_near_kernel<<<dim3((unsigned)nf, NEAR_PARTS), NEAR_T, near_smem, s>>>(dfits, dstate, dorder, dC, dthr);
    };
    int max_iter = 0;
    for (const BFit &F : fits) max_iter = std::max(max_iter, F.max_iter);
    int64_t replays = 0;
    if (active > 0) {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        FK_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        try {
            one_iteration();
        } catch (...) {
            // end the capture so that the caller's stream stays usable
            cudaGraph_t partial = nullptr;
            (void)cudaStreamEndCapture(s, &partial);
            if (partial) cudaGraphDestroy(partial);
            (void)cudaGetLastError();
            throw;
        }
        cudaError_t ce = cudaStreamEndCapture(s, &graph);
        if (ce != cudaSuccess) {
            set_error("graph capture failed: %s", cudaGetErrorString(ce));
            fail(FK_ERR_CUDA);
        }
        ce = cudaGraphInstantiate(&exec, graph, 0);
        if (ce != cudaSuccess) {
            cudaGraphDestroy(graph);
            set_error("graph instantiation failed: %s", cudaGetErrorString(ce));
            fail(FK_ERR_CUDA);
        }
        int left = active;
        const int group = 4;  // replays between checks of the active count
        while (left > 0 && replays < max_iter) {
            const int g = (int)std::min<int64_t>(group, max_iter - replays);
            for (int r = 0; r < g; r++) {
                ce = cudaGraphLaunch(exec, s);
                if (ce != cudaSuccess) break;
                replays++;
            }
            if (ce == cudaSuccess) ce = cudaMemcpyAsync(&left, dctr + 31, sizeof(int), cudaMemcpyDeviceToHost, s);
            if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
            if (ce != cudaSuccess) break;
        }
        cudaGraphExecDestroy(exec);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) {
            set_error("batched Lloyd iterations failed: %s", cudaGetErrorString(ce));
            fail(FK_ERR_CUDA);
        }
    }
    FK_CUDA(cudaEventRecord(ev[4], s));

    // ---- best run per problem (strictly lowest inertia, first run on ties), outputs
    std::vector<BState> st(nf);
    FK_CUDA(cudaMemcpyAsync(st.data(), dstate, sizeof(BState) * (size_t)nf, cudaMemcpyDeviceToHost, s));
    FK_CUDA(cudaStreamSynchronize(s));
    int64_t nmax = 1;
    for (int64_t p = 0; p < np; p++) nmax = std::max(nmax, P[p].n);
    uint64_t *l64 = (uint64_t *)ctx.get(BUF_OUT, sizeof(uint64_t) * (size_t)nmax);
    int64_t iters = 0;
    for (int f = 0; f < nf; f++) iters += st[f].n_iter;
    int f0 = 0;
    for (int64_t p = 0; p < np; p++) {
        const fk_batch_problem &q = P[p];
        int best = -1;
        float bi = 0.f;
        for (int64_t r = 0; r < q.n_init; r++) {
            const float in = (float)st[f0 + r].inertia;
            if (best < 0 || in < bi) {
                best = (int)r;
                bi = in;
            }
        }
        const int f = f0 + best;
        const BFit &F = fits[f];
        FK_CUDA(cudaMemcpyAsync(q.centers_out, dC + F.c_off + (int64_t)st[f].cur * F.k * F.d,
                                sizeof(float) * (size_t)(F.k * F.d), cudaMemcpyDefault, s));
        batch_labels_u64_kernel<<<(F.n + 255) / 256, 256, 0, s>>>(dlab + F.s_off, F.n, l64);
        FK_LAUNCH_CHECK();
        FK_CUDA(cudaMemcpyAsync(q.labels_out, l64, sizeof(uint64_t) * (size_t)F.n, cudaMemcpyDefault, s));
        FK_CUDA(cudaStreamSynchronize(s));  // l64 is reused by the next problem
        *q.inertia_out = bi;
        *q.n_iter_out = st[f].n_iter;
        if (q.best_run_out) *q.best_run_out = best;
        f0 += (int)q.n_init;
    }
    FK_CUDA(cudaEventRecord(ev[5], s));
    FK_CUDA(cudaEventSynchronize(ev[5]));
    if (rep) {
        rep->fits = nf;
        rep->iterations_total = iters;
        rep->graph_launches = replays;
        rep->tuned_buckets = tuned;
        for (int b = 0; b < NBUCKETS; b++)
            rep->bucket_variant[b] = bstart[b + 1] > bstart[b] ? ctx.batch_variant[b] : -1;
        float ms = 0.f;
        FK_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
        rep->ms_upload = ms;
        FK_CUDA(cudaEventElapsedTime(&ms, ev[1], ev[2]));
        rep->ms_init = ms;
        FK_CUDA(cudaEventElapsedTime(&ms, ev[2], ev[3]));
        rep->ms_tune = ms;
        FK_CUDA(cudaEventElapsedTime(&ms, ev[3], ev[4]));
        rep->ms_lloyd = ms;
        FK_CUDA(cudaEventElapsedTime(&ms, ev[4], ev[5]));
        rep->ms_download = ms;
        FK_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[5]));
        rep->ms_total = ms;
        for (int f = 0; f < nf; f++) {
            if (rep->fit_inertia) rep->fit_inertia[f] = st[f].inertia;
            if (rep->fit_n_iter) rep->fit_n_iter[f] = st[f].n_iter;
        }
    }
    return FK_OK;
}

}  // namespace fk
