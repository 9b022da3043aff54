// fk_fold.cu -- sequential left folds in F, computed exactly in parallel.
//
// The reference sums in row order with one rounding per addition: the 2-means
// centre sums of BisectingKMeans (bisecting_kmeans.rs:264-298, and
// compute_cluster_stats :192-211) and its SSE folds (:300-309, :443-463). On
// this GPU a dependent FP64 addition takes 64 cycles, so folding 10^5 values
// one after the other costs milliseconds per chain. The folds here return the
// same bits as the sequential loop:
//
//   While the running sum p keeps its sign s and its binade [2^e, 2^(e+1)),
//   p = s * P * ulp with P an integer in [2^MB, 2^(MB+1)), and adding v
//   rounds to P + a: a = round(s * v / ulp), and for an exact half the even
//   neighbour, so a depends on P's parity. Every value is thus a map
//   P -> P + a[P & 1], and so is any run of values (the maps compose). As the
//   sum can fall as well as rise, a composed map also carries the smallest
//   and largest running increment (lo, hi); it applies exactly when the
//   whole path stays inside the binade: 2^MB < P + lo and P + hi < 2^(MB+1).
//
// fold_sums_kernel estimates the sum of each (chain, chunk of 256 values) in
// f32 and counts its values; fold_prefix_kernel turns the estimates into the
// chunks' starting sums; fold_compose_kernel forms each chunk's map for the
// sign and binade of that estimate (it steers speed, never the result);
// fold_walk_kernel walks each chain with one warp: a chunk whose map applies is
// one integer addition, any other chunk is added value by value in F.
//
// A fold whose sum stays near zero changes binade every few values, and there
// a plain addition (64 cycles) beats every map: scans of 32 maps per change and
// three binades' maps per chunk of 1,024 took 1.30 ms a fold in the mean of a
// BisectingKMeans fit (20,000 x 16, 10 runs: 320 chains), this 0.14 ms.
//
// A chain is a strided array with an optional mask: chain c folds
// base[i * stride] over i in [0, m) in order, skipping i where
// mask != null and mask[i] != mval.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "fk_internal.cuh"

namespace fk {
namespace {

constexpr int FCH = 256;               // values per chunk: eight a lane
constexpr int FWARPS = 8;              // chunks per CTA in the sums / compose passes
constexpr long long FBIG = 1LL << 60;  // a running increment no binade holds

template <typename T> struct FB;
template <> struct FB<float> {
    using U = uint32_t;
    static constexpr int MB = 23;
    static constexpr int EXPM = 0xFF;
    static __device__ __forceinline__ U bits(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float from(U b) { return __uint_as_float(b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
};
template <> struct FB<double> {
    using U = unsigned long long;
    static constexpr int MB = 52;
    static constexpr int EXPM = 0x7FF;
    static __device__ __forceinline__ U bits(double v) { return (U)__double_as_longlong(v); }
    static __device__ __forceinline__ double from(U b) { return __longlong_as_double((long long)b); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
};

// Sign (+1 / -1), biased exponent and significand of a nonzero normal finite
// value; false for zero, subnormals, inf and NaN.
template <typename T>
__device__ __forceinline__ bool split(T p, int &s, int &be, long long &P) {
    using B = FB<T>;
    const typename B::U b = B::bits(p);
    be = (int)((b >> B::MB) & (typename B::U)B::EXPM);
    if (be == 0 || be == B::EXPM) return false;
    s = (b >> (sizeof(typename B::U) * 8 - 1)) ? -1 : 1;
    P = (long long)((b & (((typename B::U)1 << B::MB) - 1)) | ((typename B::U)1 << B::MB));
    return true;
}

template <typename T>
__device__ __forceinline__ T join(int s, int be, long long P) {
    using B = FB<T>;
    typename B::U b = ((typename B::U)be << B::MB) | ((typename B::U)P & (((typename B::U)1 << B::MB) - 1));
    if (s < 0) b |= (typename B::U)1 << (sizeof(typename B::U) * 8 - 1);
    return B::from(b);
}

// A map for a running sum of sign s in binade be: the increment a0 / a1 from an
// even / odd P, and bounds lo / hi of the running increments of both (a1's
// differ from a0's by at most one per composition, which the bounds include).
struct SMap {
    long long a0, a1, lo, hi;
};

__device__ __forceinline__ SMap smap_ident() { return {0, 0, FBIG, -FBIG}; }

// One more value at the end of a run.
template <typename T>
__device__ __forceinline__ void run_add(SMap &m, T v, int be, int s) {
    using B = FB<T>;
    using U = typename B::U;
    const U b = B::bits(v);
    const int ev = (int)((b >> B::MB) & (U)B::EXPM);
    const bool neg = ((b >> (sizeof(U) * 8 - 1)) != 0) != (s < 0);
    const U mant = (b & (((U)1 << B::MB) - 1)) | (ev ? (U)1 << B::MB : (U)0);
    const int r = be - (ev ? ev : 1);
    const int sh = max(0, min(r, B::MB + 2));  // a shift of MB + 2 leaves nothing
    const U half = ((U)1 << sh) >> 1, rem = mant & (((U)1 << sh) - 1);
    const bool tie = sh > 0 && rem == half;
    const long long q = (long long)(mant >> sh) + (sh > 0 && rem > half ? 1 : 0);
    // an exact half as its floor; the sum's parity adds one or not
    const long long inc = neg ? -q - (tie ? 1 : 0) : q;
    m.a0 += inc;
    m.a1 += inc;
    m.a0 += tie ? (m.a0 & 1) : 0;
    m.a1 += tie ? 1 - (m.a1 & 1) : 0;
    const bool out = ev == B::EXPM || (r < 0 && mant != 0);  // inf, NaN, |v| >= 2^(be+1)
    m.lo = out ? -FBIG : min(m.lo, m.a0 - 1);
    m.hi = max(m.hi, m.a0 + 1);
}

// f then g (at most 256 increments of 2^53: no overflow)
__device__ __forceinline__ SMap smap_compose(const SMap &f, const SMap &g) {
    SMap o;
    o.a0 = f.a0 + ((f.a0 & 1) ? g.a1 : g.a0);
    o.a1 = f.a1 + ((f.a1 & 1) ? g.a0 : g.a1);
    const bool bad = f.lo == -FBIG || g.lo == -FBIG;
    o.lo = bad ? -FBIG : (g.lo == FBIG ? f.lo : min(f.lo, f.a0 + g.lo - 1));
    o.hi = g.hi == -FBIG ? f.hi : max(f.hi, f.a0 + g.hi + 1);
    return o;
}

__device__ __forceinline__ SMap shfl_down_smap(const SMap &m, int off) {
    return {__shfl_down_sync(0xffffffffu, m.a0, off), __shfl_down_sync(0xffffffffu, m.a1, off),
            __shfl_down_sync(0xffffffffu, m.lo, off), __shfl_down_sync(0xffffffffu, m.hi, off)};
}

// The chain descriptor (FoldChain, fk_internal.cuh) read with its values' type.
template <typename T>
struct Chain {
    const T *base;
    int64_t stride;
    const uint8_t *mask;
    int32_t mval;
    int32_t active_slot;
};
static_assert(sizeof(Chain<double>) == sizeof(FoldChain) && sizeof(Chain<float>) == sizeof(FoldChain),
              "Chain mirrors FoldChain");

template <typename T>
__device__ __forceinline__ bool takes(const Chain<T> &c, int64_t i) {
    return c.mask == nullptr || c.mask[i] == (uint8_t)c.mval;
}

// A value as an f32 summand of the estimates: F = f32 itself, F = f64 times
// 2^-esc by its bits (no FP64 conversion; out of range: 0 or inf).
__device__ __forceinline__ float est_of(float v, int) { return v; }
__device__ __forceinline__ float est_of(double v, int esc) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7FFull) - 1023 - esc + 127;
    const uint32_t sg = (uint32_t)(b >> 32) & 0x80000000u;
    if (e <= 0) return 0.f;
    if (e >= 255) return __uint_as_float(sg | 0x7F800000u);
    return __uint_as_float(sg | ((uint32_t)e << 23) | (uint32_t)((b >> 29) & 0x7FFFFFull));
}
// Biased exponent in F of an estimate, 0 where there is none.
template <typename T>
__device__ __forceinline__ int est_exp(float e, int esc) {
    const int be = (int)((__float_as_uint(e) >> 23) & 0xFFu);
    if (be == 0 || be == 0xFF) return 0;
    if (sizeof(T) == 4) return be;
    const int b64 = be - 127 + esc + 1023;
    return b64 >= 1 && b64 < 0x7FF ? b64 : 0;
}
// The scale of a chain's estimates: the exponent of its first value (f64).
template <typename T>
__device__ __forceinline__ int chain_scale(const Chain<T> &c) {
    if (sizeof(T) == 4) return 0;
    const int e = (int)((FB<T>::bits(c.base[0]) >> FB<T>::MB) & (typename FB<T>::U)FB<T>::EXPM);
    return e > 0 && e < FB<T>::EXPM ? e - 1023 : 0;
}

// Per (chain, chunk): the chain's estimated sum and its value count (CTA: FWARPS
// chunks of one chain, a warp per chunk, neighbouring lanes' values adjacent).
template <typename T>
__global__ void __launch_bounds__(FWARPS * 32)
    fold_sums_kernel(const Chain<T> *__restrict__ chains, int64_t m, const int *__restrict__ active, int64_t nch,
                     float *__restrict__ csum, int32_t *__restrict__ ccnt) {
    const int lane = threadIdx.x & 31;
    const int64_t c = blockIdx.y, j = (int64_t)blockIdx.x * FWARPS + (threadIdx.x >> 5);
    if (j >= nch) return;
    const Chain<T> ch = chains[c];
    if (ch.active_slot >= 0 && !active[ch.active_slot]) return;
    const int esc = chain_scale(ch);
    float s = 0.f;
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < FCH / 32; q++) {
        const int64_t i = j * FCH + q * 32 + lane;
        const bool live = i < m && takes(ch, i);
        const T v = live ? ch.base[i * ch.stride] : T(0);
        s += est_of(v, esc);
        cnt += live ? 1 : 0;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        csum[c * nch + j] = s;
        ccnt[c * nch + j] = cnt;
    }
}

// csum becomes each chunk's estimated starting sum (one warp per chain).
template <typename T>
__global__ void __launch_bounds__(32)
    fold_prefix_kernel(const Chain<T> *__restrict__ chains, const int *__restrict__ active, int64_t nch,
                       float *__restrict__ csum) {
    const int lane = threadIdx.x;
    const int slot = chains[blockIdx.x].active_slot;
    if (slot >= 0 && !active[slot]) return;
    float *cs = csum + (int64_t)blockIdx.x * nch;
    float run = 0.f;
    for (int64_t jb = 0; jb < nch; jb += 32) {
        const float v = jb + lane < nch ? cs[jb + lane] : 0.f;
        float s = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const float o = __shfl_up_sync(0xffffffffu, s, off);
            if (lane >= off) s += o;
        }
        const float before = __shfl_up_sync(0xffffffffu, s, 1);
        if (jb + lane < nch) cs[jb + lane] = lane > 0 ? run + before : run;
        run += __shfl_sync(0xffffffffu, s, 31);
    }
}

// One chunk's map, for running sums of one sign in one binade (be 0: none).
struct CMap {
    SMap m;
    int be, sign;
};

// Per (chain, chunk): the chunk's map (lane g composes values g*8 .. g*8+7 of
// the chunk, then an ordered warp reduction).
template <typename T>
__global__ void __launch_bounds__(FWARPS * 32)
    fold_compose_kernel(const Chain<T> *__restrict__ chains, int64_t m, const int *__restrict__ active, int64_t nch,
                        const float *__restrict__ csum, CMap *__restrict__ cmaps) {
    const int lane = threadIdx.x & 31;
    const int64_t c = blockIdx.y, j = (int64_t)blockIdx.x * FWARPS + (threadIdx.x >> 5);
    if (j >= nch) return;
    const Chain<T> ch = chains[c];
    if (ch.active_slot >= 0 && !active[ch.active_slot]) return;
    const float e = csum[c * nch + j];
    const int be = est_exp<T>(e, chain_scale(ch)), s = e < 0.f ? -1 : 1;
    CMap *out = cmaps + c * nch + j;
    if (be == 0) {
        if (lane == 0) out->be = 0;
        return;
    }
    SMap run = smap_ident();
    const int64_t g0 = j * FCH + (int64_t)lane * (FCH / 32);
    T v[FCH / 32];
    unsigned live = 0;
#pragma unroll
    for (int q = 0; q < FCH / 32; q++) {
        const bool on = g0 + q < m && takes(ch, g0 + q);
        v[q] = on ? ch.base[(g0 + q) * ch.stride] : T(0);
        live |= on ? 1u << q : 0u;
    }
#pragma unroll
    for (int q = 0; q < FCH / 32; q++)
        if (live >> q & 1u) run_add(run, v[q], be, s);
    __syncwarp();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const SMap r = shfl_down_smap(run, o);
        if ((lane & (2 * o - 1)) == 0) run = smap_compose(run, r);
    }
    if (lane == 0) {
        // a path that no binade holds: no map
        constexpr long long SPAN = 1LL << (FB<T>::MB + 1);
        const bool fits = run.lo > -SPAN && run.hi < SPAN;
        out->m = run;
        out->be = fits ? be : 0;
        out->sign = s;
    }
}

// One warp per chain: the whole fold and the count of the chain's values.
template <typename T>
__global__ void __launch_bounds__(32)
    fold_walk_kernel(const Chain<T> *__restrict__ chains, int64_t m, const int *__restrict__ active, int64_t nch,
                     const CMap *__restrict__ cmaps, const int32_t *__restrict__ ccnt, T *__restrict__ result,
                     long long *__restrict__ count) {
    using B = FB<T>;
    __shared__ T sv[FCH];
    const int64_t c = blockIdx.x;
    const int lane = threadIdx.x;
    const Chain<T> ch = chains[c];
    if (ch.active_slot >= 0 && !active[ch.active_slot]) return;
    constexpr long long LOW = (1LL << B::MB) + 1, TOP = (1LL << (B::MB + 1)) - 1;
    T p = T(0);
    int s = 1, be = 0;
    long long P = 0;
    bool normal = false;
    long long total = 0;
    for (int64_t jb = 0; jb < nch; jb += 32) {
        const int nb = (int)min((int64_t)32, nch - jb);
        CMap cm{};
        int cnt = 0;
        if (lane < nb) {
            cm = cmaps[c * nch + jb + lane];
            cnt = ccnt[c * nch + jb + lane];
        }
        for (int i = 0; i < nb; i++) {
            const int n_i = __shfl_sync(0xffffffffu, cnt, i);
            if (n_i == 0) continue;
            total += n_i;
            const int cb = __shfl_sync(0xffffffffu, cm.be, i), sg = __shfl_sync(0xffffffffu, cm.sign, i);
            if (normal && cb == be && sg == s) {
                const long long a = __shfl_sync(0xffffffffu, (P & 1) ? cm.m.a1 : cm.m.a0, i);
                const long long lo = __shfl_sync(0xffffffffu, cm.m.lo, i), hi = __shfl_sync(0xffffffffu, cm.m.hi, i);
                if (P + lo >= LOW && P + hi <= TOP) {
                    P += a;
                    p = join<T>(s, be, P);
                    continue;
                }
            }
            // the chunk's values in order, one exact addition each
            const int64_t i0 = (jb + i) * FCH;
            T v[FCH / 32];
            unsigned live = 0;
#pragma unroll
            for (int q = 0; q < FCH / 32; q++) {
                const int64_t r = i0 + q * 32 + lane;
                const bool on = r < m && takes(ch, r);
                v[q] = on ? ch.base[r * ch.stride] : T(0);
                live |= on ? 1u << q : 0u;
            }
            int at = 0;
#pragma unroll
            for (int q = 0; q < FCH / 32; q++) {
                const unsigned on = __ballot_sync(0xffffffffu, live >> q & 1u);
                if (live >> q & 1u) sv[at + __popc(on & ((1u << lane) - 1u))] = v[q];
                at += __popc(on);
            }
            __syncwarp();
            int e = 0;
            for (; e + 8 <= at; e += 8) {
#pragma unroll
                for (int u = 0; u < 8; u++) p = B::add(p, sv[e + u]);
            }
            for (; e < at; e++) p = B::add(p, sv[e]);
            __syncwarp();  // sv is refilled by the next such chunk
            normal = split(p, s, be, P);
        }
    }
    if (lane == 0) {
        result[c] = p;
        count[c] = total;
    }
}

}  // namespace

template <typename T>
void run_exact_folds(Ctx &ctx, const FoldChain *chains, int nchains, int64_t m, const int *active, T *result,
                     long long *count) {
    if (nchains <= 0) return;
    cudaStream_t s = ctx.stream;
    const int64_t nch = m > 0 ? (m + FCH - 1) / FCH : 0;
    // Chains at a time: gridDim.y holds 65,535, and their maps (48 bytes a chunk)
    // stay within 1 GB, or as many as there is room for.
    const int64_t room = (ctx.lean ? (int64_t)16 << 20 : (int64_t)1 << 30) / (48 * std::max<int64_t>(nch, 1));
    int per = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(nchains, 65535), room));
    float *csum = nullptr;
    int32_t *ccnt = nullptr;
    CMap *cmaps = nullptr;
    while (true) {
        try {
            csum = (float *)ctx.get(BUF_FOLD_SUM, sizeof(float) * (size_t)per * nch);
            ccnt = (int32_t *)ctx.get(BUF_FOLD_CNT, sizeof(int32_t) * (size_t)per * nch);
            cmaps = (CMap *)ctx.get(BUF_FOLD_MAP, sizeof(CMap) * (size_t)per * nch);
            break;
        } catch (const Error &e) {
            if (e.code != FK_ERR_OOM || per == 1) throw;
            per = (per + 1) / 2;
        }
    }
    const Chain<T> *ch = (const Chain<T> *)chains;
    for (int c0 = 0; c0 < nchains; c0 += per) {
        const unsigned nc = (unsigned)std::min(per, nchains - c0);
        if (nch > 0) {
            const dim3 grid((unsigned)((nch + FWARPS - 1) / FWARPS), nc);
            fold_sums_kernel<T><<<grid, FWARPS * 32, 0, s>>>(ch + c0, m, active, nch, csum, ccnt);
            FK_LAUNCH_CHECK();
            fold_prefix_kernel<T><<<nc, 32, 0, s>>>(ch + c0, active, nch, csum);
            FK_LAUNCH_CHECK();
            fold_compose_kernel<T><<<grid, FWARPS * 32, 0, s>>>(ch + c0, m, active, nch, csum, cmaps);
            FK_LAUNCH_CHECK();
        }
        fold_walk_kernel<T><<<nc, 32, 0, s>>>(ch + c0, m, active, nch, cmaps, ccnt, result + c0, count + c0);
        FK_LAUNCH_CHECK();
    }
}

template void run_exact_folds<double>(Ctx &, const FoldChain *, int, int64_t, const int *, double *, long long *);
template void run_exact_folds<float>(Ctx &, const FoldChain *, int, int64_t, const int *, float *, long long *);

}  // namespace fk
