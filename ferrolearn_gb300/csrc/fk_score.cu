// fk_score.cu -- the plain f32 assignment through FMA scores.
//
// nearest_center (kmeans.rs:295-309) compares direct-form distances
// (squared_euclidean, :159-163): a subtraction, a product and an addition per
// feature, none of them fused. Half the distance less half of |x|^2 ranks the
// centres as well and takes one FMA per feature. The labels here are still
// those of the direct form:
//
//   1. Centres less m, an average of (up to 16 of) them, so that an offset
//      common to all the data costs no precision: c' = c - m, x' = x - m, and
//      per centre n2 >= |c'|^2. With T = |c'|^2 / 2 - x'c' of the exact c - m
//      and x - m, D = 2T + |x - m|^2 is the exact squared distance.
//   2. A tiled pass forms S = h - x'c' per row and centre, h = n2 / 2 - a n2. With
//      u = 2^-24, the roundings of c', x', n2 and of d FMAs, and |x'||c'| <=
//      (|x'|^2 + |c'|^2) / 2, T lies in [S - b P, S + 2 a n2 + b P], where
//      P >= |x'|^2, a = 1.1 u (2d + 12), b = 1.1 u (d/2 + 1).
//   3. A row with smallest S (centre 1) and second smallest S2 is decided if
//      S2 - S > 2 a n2[1] + 2 b P + 1.02 g D1 (1.05 times that, for the roundings
//      of the test itself), g = 1.01 (d + 2) u the relative error of a direct
//      form and D1 an upper bound of the distance to centre 1: every other
//      computed distance is then strictly larger than centre 1's.
//   4. Other rows (near ties, non-finite or huge values: no finite bound; values
//      so small that products underflow: 1e-30 is added) are listed and scored
//      in the direct form against every centre.
//
// Bound at 200,003 x 37 against 100 centres: issue slots, half of them the FMA
// per (row, centre, feature), the rest the ranking (about 5 operations a pair),
// the shared-memory reads (15 of 16 bytes per 224 FMAs of a thread) and the
// staging: 66 us in the tiled pass (FP32 pipe alone: 20), where the direct form
// took 135; 1M x 64 against 256: 1.05 ms for 1.96. The whole predict 176 ->
// 119 us.
#include <algorithm>
#include <cfloat>

#include "fk_internal.cuh"

namespace fk {
namespace {

constexpr int SBM = 128;  // rows per block tile, eight a thread
constexpr int SDJ = 64;   // features staged at a time, at most
constexpr int SNT = 256;  // 16 x 16 threads
constexpr int SMEAN = 16;  // centres that m averages, at most

// c', h, n2 (a warp per centre), m, and the centres by feature (ct, kp apart).
__global__ void __launch_bounds__(SNT)
    score_centres_kernel(const float *__restrict__ c, int k, int d, int dp, int kp, float a, float *__restrict__ cc,
                         float *__restrict__ h, float *__restrict__ n2, float *__restrict__ mean,
                         float *__restrict__ ct, unsigned long long *__restrict__ open_count) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *open_count = 0;
    extern __shared__ float m[];
    const int lane = threadIdx.x & 31, q = (int)blockIdx.x * (SNT / 32) + (threadIdx.x >> 5);
    const float *cq = c + (int64_t)min(q, k - 1) * d;
    const float first = lane < d ? cq[lane] : 0.f;  // in flight with the sum's loads
    const int ns = min(k, SMEAN), step = k / ns;
    for (int j = threadIdx.x; j < dp; j += SNT) {
        float v[SMEAN], s = 0.f;
#pragma unroll
        for (int t = 0; t < SMEAN; t++) v[t] = t < ns && j < d ? c[(int64_t)(t * step) * d + j] : 0.f;
#pragma unroll
        for (int t = 0; t < SMEAN; t++) s += v[t];
        m[j] = s / (float)ns;
        if (blockIdx.x == 0) mean[j] = m[j];
    }
    __syncthreads();
    if (q >= k) return;
    float s = 0.f;
    for (int j = lane; j < dp; j += 32) {
        const float cv = j == lane ? first : (j < d ? cq[j] : 0.f);
        const float v = j < d ? __fsub_rn(cv, m[j]) : 0.f;
        cc[(int64_t)q * dp + j] = v;
        s = __fmaf_ru(v, v, s);
        if (j < d) ct[(int64_t)j * kp + q] = cv;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s = __fadd_ru(s, __shfl_xor_sync(0xffffffffu, s, o));
    if (lane == 0) {
        n2[q] = s;
        h[q] = __fmul_rd(s, 0.5f - a);
    }
}

struct ScorePlan {
    const float *cc, *h, *n2, *mean;
    int dp;
    int w;   // features of a slab (a multiple of 4): d in as few slabs of at most SDJ as it takes, evenly
    int st;  // row stride of the stage: an odd number of 16-byte units (no bank conflict over eight rows)
    float a, b, g;
};

// The ranking's three arrays of 16 x 128 take the place of the rows; their
// stride keeps a warp's 16 x 2 writes apart.
constexpr int RST = SBM + 2;
size_t rows_smem(int bn, int st) {
    return sizeof(float) * ((size_t)bn * st + std::max<size_t>((size_t)SBM * st, (size_t)3 * 16 * RST));
}

// One CTA per 128 rows; thread (tx, ty): rows ty + 16 i, centres tx + 16 j of a
// 16 TN tile.
template <int TN>
__global__ void __launch_bounds__(SNT, 2)
    score_rows_kernel(const float *__restrict__ x, int64_t n, int d, int k, ScorePlan p, bool vec,
                      int32_t *__restrict__ labels, int32_t *__restrict__ open_list,
                      unsigned long long *__restrict__ open_count) {
    constexpr int TM = SBM / 16, BN = 16 * TN;
    extern __shared__ __align__(16) float sm[];
    const int W = p.w, SST = p.st;
    float *const cs = sm, *const xs = sm + BN * SST;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const bool resident = d <= W && k <= BN;  // one slab, one centre tile: staged once
    bool staged = false;
    for (int64_t row0 = (int64_t)blockIdx.x * SBM; row0 < n; row0 += (int64_t)gridDim.x * SBM) {
        const int rows = (int)min((int64_t)SBM, n - row0);
        const float *const xg = x + row0 * d;
        float s1[TM], s2[TM], p2 = 0.f;
        int i1[TM];
#pragma unroll
        for (int i = 0; i < TM; i++) {
            s1[i] = s2[i] = INFINITY;
            i1[i] = -1;
        }
        for (int ct = 0; ct < k; ct += BN) {
            float acc[TM][TN];
#pragma unroll
            for (int j = 0; j < TN; j++) {
                const int q = ct + tx + 16 * j;
                const float hq = q < k ? p.h[q] : INFINITY;
#pragma unroll
                for (int i = 0; i < TM; i++) acc[i][j] = hq;
            }
            for (int j0 = 0; j0 < d; j0 += W) {
                const int j4 = (min(W, d - j0) + 3) / 4;
                __syncthreads();  // the stage is free
                if (vec) {
#pragma unroll 1
                    for (int q = tid & 7; q < j4; q += 8) {
                        float4 v[4];
                        const float4 mq = *reinterpret_cast<const float4 *>(p.mean + j0 + 4 * q);
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int r = (tid >> 3) + 32 * e;
                            v[e] = r < rows ? *reinterpret_cast<const float4 *>(xg + (int64_t)r * d + j0 + 4 * q) : mq;
                        }
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            *reinterpret_cast<float4 *>(xs + ((tid >> 3) + 32 * e) * SST + 4 * q) =
                                make_float4(__fsub_rn(v[e].x, mq.x), __fsub_rn(v[e].y, mq.y), __fsub_rn(v[e].z, mq.z),
                                            __fsub_rn(v[e].w, mq.w));
                    }
                } else {
#pragma unroll 1
                    for (int j = tid & 31; j < 4 * j4; j += 32) {
                        const bool in = j0 + j < d;
                        const float mj = in ? p.mean[j0 + j] : 0.f;
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; e++) {
                            const int r = (tid >> 5) + 8 * e;
                            v[e] = r < rows && in ? xg[(int64_t)r * d + j0 + j] : mj;
                        }
#pragma unroll
                        for (int e = 0; e < 16; e++) xs[((tid >> 5) + 8 * e) * SST + j] = __fsub_rn(v[e], mj);
                    }
                }
                if (!staged)
#pragma unroll 1
                for (int r = tid >> 3; r < BN; r += SNT / 8)
#pragma unroll 2
                    for (int q = tid & 7; q < j4; q += 8)
                        *reinterpret_cast<float4 *>(cs + r * SST + 4 * q) =
                            ct + r < k ? *reinterpret_cast<const float4 *>(p.cc + (int64_t)(ct + r) * p.dp + j0 + 4 * q)
                                       : float4{};
                staged = resident;
                __syncthreads();
                if (ct == 0 && tid < SBM) {
                    for (int q = 0; q < j4; q++) {
                        const float4 v = *reinterpret_cast<const float4 *>(xs + tid * SST + 4 * q);
                        p2 = __fmaf_rn(v.x, v.x, __fmaf_rn(v.y, v.y, __fmaf_rn(v.z, v.z, __fmaf_rn(v.w, v.w, p2))));
                    }
                }
#pragma unroll 1
                for (int q = 0; q < j4; q++) {
                    float4 xv[TM];
#pragma unroll
                    for (int i = 0; i < TM; i++)
                        xv[i] = *reinterpret_cast<const float4 *>(xs + (ty + 16 * i) * SST + 4 * q);
#pragma unroll
                    for (int j = 0; j < TN; j++) {
                        const float4 cv = *reinterpret_cast<const float4 *>(cs + (tx + 16 * j) * SST + 4 * q);
#pragma unroll
                        for (int i = 0; i < TM; i++) acc[i][j] = __fmaf_rn(-xv[i].x, cv.x, acc[i][j]);
#pragma unroll
                        for (int i = 0; i < TM; i++) acc[i][j] = __fmaf_rn(-xv[i].y, cv.y, acc[i][j]);
#pragma unroll
                        for (int i = 0; i < TM; i++) acc[i][j] = __fmaf_rn(-xv[i].z, cv.z, acc[i][j]);
#pragma unroll
                        for (int i = 0; i < TM; i++) acc[i][j] = __fmaf_rn(-xv[i].w, cv.w, acc[i][j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < TN; j++)
#pragma unroll
                for (int i = 0; i < TM; i++) {
                    const float s = acc[i][j];
                    s2[i] = fminf(s2[i], fmaxf(s, s1[i]));  // NaN: s2 = s1, the row stays open
                    if (s < s1[i]) {
                        s1[i] = s;
                        i1[i] = ct + tx + 16 * j;
                    }
                }
        }
        __syncthreads();
        float *const r1 = xs, *const r2 = xs + 16 * RST;
        int *const ri = reinterpret_cast<int *>(xs + 2 * 16 * RST);
#pragma unroll
        for (int i = 0; i < TM; i++) {
            r1[tx * RST + ty + 16 * i] = s1[i];
            r2[tx * RST + ty + 16 * i] = s2[i];
            ri[tx * RST + ty + 16 * i] = i1[i];
        }
        __syncthreads();
        if (tid < SBM) {
            float b1 = INFINITY, b2 = INFINITY;
            int bi = -1;
#pragma unroll
            for (int t = 0; t < 16; t++) {
                const float v = r1[t * RST + tid];
                b2 = fminf(fminf(b2, r2[t * RST + tid]), fmaxf(v, b1));
                if (v < b1) {
                    b1 = v;
                    bi = ri[t * RST + tid];
                }
            }
            bool open = false;
            if (tid < rows) {
                bool decided = false;
                if (bi >= 0) {
                    const float P = 1.002f * p2, an = 2.0f * p.a * p.n2[bi];
                    const float d1 = fmaxf(2.0f * (b1 + an + 2.0f * p.b * P) + P, 0.f);
                    const float w = 1.05f * (an + 2.0f * p.b * P + 1.02f * p.g * d1) + 1e-30f;
                    // w bounded: no distance near F::MAX (g >= 1e-6: below 1e36)
                    decided = w < 1e30f && P < 1e36f && __fsub_rd(b2, b1) > w;
                }
                if (decided) labels[row0 + tid] = bi;
                open = !decided;
            }
            const unsigned bm = __ballot_sync(0xffffffffu, open);
            if (bm) {
                unsigned long long at = 0;
                const int lane = tid & 31;
                if (lane == 0) at = atomicAdd(open_count, (unsigned long long)__popc(bm));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (open) open_list[at + __popc(bm & ((1u << lane) - 1u))] = (int32_t)(row0 + tid);
            }
        }
    }
}

// A row against centres [c0 + 32 u, c0 + 32 u + 32) for u < U, lane by lane: the direct
// form's sums over ascending features, and of them the smallest (the lowest index of
// equals) taken into (bv, bi). 32 / U features' loads of ct, whole lines, are in flight.
template <int U>
__device__ __forceinline__ void direct_group(const float *__restrict__ xr, int d, const float *__restrict__ ct, int kp,
                                             int k, int c0, int lane, float &bv, int &bi) {
    float acc[U];
#pragma unroll
    for (int u = 0; u < U; u++) acc[u] = 0.f;
    const float *cp = ct + c0 + lane;
#pragma unroll(32 / U)
    for (int j = 0; j < d; j++) {
        const float xv = xr[j];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float t = __fsub_rn(xv, cp[(int64_t)j * kp + 32 * u]);
            acc[u] = __fadd_rn(acc[u], __fmul_rn(t, t));
        }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int cc = c0 + 32 * u + lane;
        if (cc < k && acc[u] < bv) {  // ascending index: the lowest of equals stays
            bv = acc[u];
            bi = cc;
        }
    }
}

__device__ __forceinline__ void lowest_of(float &bv, int &bi, int o) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov < bv || (ov == bv && oi < bi)) {
        bv = ov;
        bi = oi;
    }
}

// Listed rows: the direct form against every centre, lowest index among the
// smallest distances strictly below F::MAX, else 0. A row is a chain of d dependent
// sums behind d loads, so a short list is bound by latency: a CTA takes a row,
// each warp 32 centres at a time. A long one has rows enough: a warp a row, 128
// centres at a time (each feature of the row read once for four). Predict calls with
// a few hundred open rows, a warp a row / as here (us): 12,000 x 50, 400 centres
// 130 / 107, 19,000 x 100, 129: 106 / 86, 800 x 999, 300: 1,099 / 701.
__global__ void __launch_bounds__(SNT)
    score_open_rows_kernel(const float *__restrict__ x, int d, const float *__restrict__ ct, int k, int kp,
                           const int32_t *__restrict__ list, const unsigned long long *__restrict__ count,
                           int32_t *__restrict__ labels) {
    __shared__ float wv[SNT / 32];
    __shared__ int wi[SNT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long cnt = *count;
    if (cnt <= 2 * (unsigned long long)gridDim.x) {
        for (unsigned long long q = blockIdx.x; q < cnt; q += gridDim.x) {
            const int64_t r = list[q];
            float bv = FLT_MAX;
            int bi = INT32_MAX;
            for (int c0 = 32 * warp; c0 < k; c0 += SNT) direct_group<1>(x + r * d, d, ct, kp, k, c0, lane, bv, bi);
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) lowest_of(bv, bi, o);
            if (lane == 0) {
                wv[warp] = bv;
                wi[warp] = bi;
            }
            __syncthreads();
            if (warp == 0) {
                bv = wv[lane % (SNT / 32)];
                bi = wi[lane % (SNT / 32)];
#pragma unroll
                for (int o = SNT / 64; o >= 1; o >>= 1) lowest_of(bv, bi, o);
                if (lane == 0) labels[r] = bi == INT32_MAX ? 0 : bi;
            }
            __syncthreads();
        }
        return;
    }
    const unsigned long long nw = ((unsigned long long)gridDim.x * SNT) >> 5;
    for (unsigned long long q = ((unsigned long long)blockIdx.x * SNT + threadIdx.x) >> 5; q < cnt; q += nw) {
        const int64_t r = list[q];
        float bv = FLT_MAX;
        int bi = INT32_MAX;
        for (int c0 = 0; c0 < k; c0 += 128) direct_group<4>(x + r * d, d, ct, kp, k, c0, lane, bv, bi);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) lowest_of(bv, bi, o);
        if (lane == 0) labels[r] = bi == INT32_MAX ? 0 : bi;
    }
}

template <int TN>
void launch_rows(const float *x, int64_t n, int d, int k, const ScorePlan &p, bool vec, int32_t *labels, int32_t *list,
                 unsigned long long *count, int num_sms, cudaStream_t s) {
    const size_t smem = rows_smem(16 * TN, p.st);
    FK_CUDA(cudaFuncSetAttribute((const void *)score_rows_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    const unsigned grid = (unsigned)std::min<int64_t>((n + SBM - 1) / SBM, 2 * (int64_t)num_sms);
    score_rows_kernel<TN><<<grid, SNT, smem, s>>>(x, n, d, k, p, vec, labels, list, count);
    FK_LAUNCH_CHECK();
}

}  // namespace

// Below 16 features or 24 centres the ranking and the tile's padding outweigh
// the two operations saved per feature; below 2e8 products the direct pass (18 us
// at 1e8) costs little more than the two launches around the tiled one (7 us).
// Predict calls at the line, direct / scored: 1,000,000 x 16, 24 centres 382 /
// 184 us, 400,000 x 16, 32: 179 / 109, 2,000 x 256, 500: 383 / 257. Where the
// row tiles fit the SMs at once, the direct pass takes as long as one tile does,
// d k, and has the SMs full near their number: there 12,500. Direct / scored with
// no row open / with hundreds open: two waves 25,000 x 80, 100 82 / 70 / 77 us,
// 30,000 x 100, 100 96 / 74 / 86, 38,900 x 54, 100 69 / 61 / 72; one wave
// 19,000 x 110, 100 (11,000) 72 / 70 / 80, 16,000 x 126, 100 (12,600) 81 / 70 / 84,
// 19,000 x 64, 200 (12,800) 80 / 68 / 74, 10,500 x 100, 200 110 / 91 / 102.
bool f32_scores_pay(int64_t n, int d, int k, int num_sms) {
    return d >= 16 && d <= 1024 && k >= 24 && n < INT32_MAX && (double)n * d * k >= 2e8 &&
           (n > (int64_t)SBM * num_sms || (int64_t)d * k >= 12500);
}

void launch_assign_f32_scored(Ctx &ctx, const float *x, int64_t n, int d, const float *c, int k, int32_t *labels) {
    cudaStream_t s = ctx.stream;
    const int dp = (d + 3) / 4 * 4, kp = (k + 127) / 128 * 128;
    const size_t floats = (size_t)k * dp + 2 * (size_t)((k + 3) / 4 * 4) + dp + (size_t)d * kp;
    float *ws = (float *)ctx.get(BUF_SC_C, sizeof(float) * floats);
    int32_t *list = (int32_t *)ctx.get(BUF_PF_LIST, sizeof(int32_t) * (size_t)n);
    unsigned long long *count = (unsigned long long *)ctx.get(BUF_PF_CNT, sizeof(unsigned long long) * 4);
    float *cc = ws, *h = cc + (size_t)k * dp, *n2 = h + (k + 3) / 4 * 4, *mean = n2 + (k + 3) / 4 * 4, *ct = mean + dp;
    const float u = 5.9604645e-08f;
    const int slabs = (d + SDJ - 1) / SDJ, w4 = (dp / 4 + slabs - 1) / slabs;
    ScorePlan p{cc, h, n2, mean, dp, 4 * w4, 4 * (w4 | 1)};
    p.a = 1.1f * u * (2.0f * d + 12.0f);
    p.b = 1.1f * u * (0.5f * d + 1.0f);
    p.g = 1.01f * u * (d + 2.0f);
    score_centres_kernel<<<(unsigned)((k + SNT / 32 - 1) / (SNT / 32)), SNT, sizeof(float) * (size_t)dp, s>>>(
        c, k, d, dp, kp, p.a, cc, h, n2, mean, ct, count);
    FK_LAUNCH_CHECK();
    const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    // the narrowest tile that takes the centres in as few passes as 128 would
    const int passes = (k + 127) / 128, tn = (k + 16 * passes - 1) / (16 * passes);
    switch (tn) {
        case 1: case 2: launch_rows<2>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
        case 3: launch_rows<3>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
        case 4: launch_rows<4>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
        case 5: launch_rows<5>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
        case 6: launch_rows<6>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
        case 7: launch_rows<7>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
        default: launch_rows<8>(x, n, d, k, p, vec, labels, list, count, ctx.num_sms, s); break;
    }
    score_open_rows_kernel<<<ctx.num_sms * 4, SNT, 0, s>>>(x, d, ct, k, kp, list, count, labels);
    FK_LAUNCH_CHECK();
}

}  // namespace fk
