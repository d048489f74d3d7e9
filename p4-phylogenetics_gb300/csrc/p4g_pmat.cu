// setPrams on the GPU: discrete-gamma rates, Q and its eigensystem, and the
// P = exp(Qt) decks of every (part, node, category), with FP64-accurate
// results.
//
// Reference: p4_setPramsPart (Pf/p4_tree.c:218-541) computes the gamma rates
// with DiscreteGamma, builds Q = R.diag(pi) and normalises it
// (Pf/util.c:44-115), takes a general real eigensystem of Q
// (Pf/eig.c:63-161) and then P(t) = V exp(lambda t) V^-1 for every node and
// category (Pf/p4_node.c:296-346, Pf/eig.c:163-223).
//
// Here Q is reversible (R symmetric, pi > 0), so the eigensystem is taken of
// the symmetric S = diag(sqrt pi) Q diag(1/sqrt pi), by FP32 Jacobi sweeps
// refined to FP64 accuracy with FP64 matrix products (eigBlock; eig4Warp for 4
// states), or by cyclic Jacobi in FP64 (round-robin pair ordering, all D/2
// disjoint rotations of a round applied together) for 2 states and spectra the
// refinement does not accept.  P(t)_ij =
// sum_k U_ik e^{lambda_k t} U_jk sqrt(pi_j/pi_i) is formed in FP32-pair
// arithmetic (k_pdeck); the FP64 decks are its values, the FP32 decks the
// pruning kernels read are the same values rounded to FP32.  This GPU's FP64
// pipe is narrow, so FP64 is used where a result needs it and FP32 elsewhere;
// the gamma rates follow the reference's iterations in FP64 step for step.
#include <cuda_runtime.h>
#include <algorithm>
#include <cfloat>
#include "p4g_internal.h"
#include "p4g_math.cuh"
#include "p4g_pmat.cuh"
#include "p4g_prune_common.cuh"
#include "p4g_tc.cuh"

namespace p4g {

// ----------------------------------------------------------------- helpers
__device__ __forceinline__ int findDesc(const int *prefix, int n, int idx)
{
    // largest d with prefix[d] <= idx
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= idx) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ----------------------------------------------------------------- gamma
// One block per (part, gdasrv).  Cut point k < K-1 is the chi-square quantile
// at (k+1)/K, then the incomplete gamma ratio of alpha+1 at it; thread 0 forms
// the bin means.
//
// What bounds it: FP64 latency (a dependent operation costs some 200 clocks on
// this GPU, a division 1.7 k), and every AS91 step needs the incomplete gamma.
// So the work goes across lanes where the method leaves it independent: a
// power series' 32 quotients are divided in one go, its terms are a prefix
// product and the partial sum up to the term that ends it a masked sum
// (gammaCoreWarp); a continued fraction's convergents are divided eight at a
// time; and the two exp/log factors of a step run on two lanes of another warp
// (of the same one where 2 (K-1) warps are more than the block has).  The
// iterations, bounds and termination tests are gm_discreteGamma's, so the
// rates agree with the serial ones to rounding; so do the start values, whose
// logarithms, lnGammas and normal quantiles several warps form at once.  With
// one lane per cut point and factor, and pow() in the start values, a new shape
// added 50 us to a setPrams of four categories, with this 26.
constexpr int GAMMA_THREADS = 320;   // ten warps: two per cut point up to 6 categories

__device__ __forceinline__ double warpSum(double v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// gm_incGammaCore with the warp's 32 lanes; every lane gets the result.
__device__ int gammaCoreWarp(double x, double p, double *ginOut)
{
    const double accurate = 1e-8, overflow = 1e30;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (x == 0.0) return 2;
    if (x < 0 || p <= 0) return -1;
    if (!(x > 1 && x >= p)) {   // power series
        double gin = 1.0, carry = 1.0;
        for (int base = 0; base < 200000; base += 32) {
            double term = x / (p + (double)(base + lane + 1));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {   // inclusive prefix product
                const double up = __shfl_up_sync(FULL, term, o);
                if (lane >= o) term *= up;
            }
            term *= carry;
            const unsigned m = __ballot_sync(FULL, !(term > accurate));
            const int last = m ? __ffs(m) - 1 : 31;
            gin += warpSum(lane <= last ? term : 0.0);
            if (m) {
                *ginOut = gin;
                return 0;
            }
            carry = __shfl_sync(FULL, term, 31);
        }
        return -1;
    }
    // continued fraction: the recurrence on every lane, lane j keeping step j
    // of a chunk, whose convergents are divided and compared together
    constexpr int CH = 8;
    double a = 1.0 - p, b = a + x + 1.0, term = 0.0;
    double p0 = 1.0, p1 = x, p2 = x + 1, p3 = x * b;
    double gin = p2 / p3;
    for (int it = 0; it < 200000; it += CH) {
        double n4 = 1.0, n5 = 1.0;
#pragma unroll
        for (int j = 0; j < CH; j++) {
            a += 1.0;
            b += 2.0;
            term += 1.0;
            const double an = a * term;
            const double p4 = b * p2 - an * p0, p5 = b * p3 - an * p1;
            if (lane == j) {
                n4 = p4;
                n5 = p5;
            }
            p0 = p2;
            p1 = p3;
            p2 = p4;
            p3 = p5;
            if (!(fabs(p4) < overflow)) {
                p0 /= overflow;
                p1 /= overflow;
                p2 /= overflow;
                p3 /= overflow;
            }
        }
        if (__any_sync(FULL, n5 == 0.0)) return gm_incGammaCore(x, p, ginOut);   // a skipped convergent
        const double rn = n4 / n5;
        double prev = __shfl_up_sync(FULL, rn, 1);
        if (lane == 0) prev = gin;
        const double dif = fabs(prev - rn);
        const unsigned m = __ballot_sync(FULL, lane < CH && !(dif > accurate) && dif <= accurate * rn);
        if (m) {
            *ginOut = __shfl_sync(FULL, prev, __ffs(m) - 1);
            return 1;
        }
        gin = __shfl_sync(FULL, rn, CH - 1);
    }
    return -1;
}

// gm_chi2Start from the logarithms and the normal quantile another warp
// formed: lp = log(prob), lpx = log(prob v / 2), z = gm_normalQuantile(prob),
// g = lnGamma(v / 2).  Powers through exp and products: a start value, and a
// quantile below 5e-7 that is returned as it is, to rounding the same.
__device__ int chi2StartFrom(double prob, double v, double g, double lp, double lpx, double z, double *chOut)
{
    const double e = 0.5e-6, aa = 0.6931471805;
    if (prob < 0.000002 || prob > 0.999998 || v <= 0.0) return -1;
    const double xx = v / 2.0, c = xx - 1.0;
    double ch;
    if (v < -1.24 * lp) {
        ch = expShort((lpx + g + xx * aa) / xx);
        if (ch - e < 0) {
            *chOut = ch;
            return 1;
        }
    } else if (v <= 0.32) {
        double lg;
        return gm_chi2Start(prob, v, chOut, &lg);
    } else {
        const double p1 = 0.222222 / v, y = z * sqrt(p1) + 1.0 - p1;
        ch = v * (y * y * y);
        if (ch > 2.2 * v + 6.0) ch = -2.0 * (log(1.0 - prob) - c * log(0.5 * ch) + g);
    }
    *chOut = ch;
    return 0;
}

// gm_chi2Step with its divisions taken off the chain: those by constants are
// products with their reciprocals, inv = 1 / *ch comes from another lane, the
// termination test is cross-multiplied.
__device__ int chi2StepFrom(double prob, double v, double t, double e2, double inv, double *ch)
{
    const double e = 0.5e-6;
    const double xx = v / 2.0, c = xx - 1.0;
    if (t < 0.0) return -1;
    const double q = *ch;
    t = (prob - t) * e2;
    const double b = t * inv;
    const double a = 0.5 * t - b * c;
    const double s1 = (210.0 + a * (140.0 + a * (105.0 + a * (84.0 + a * (70.0 + 60.0 * a))))) * (1.0 / 420.0);
    const double s2 = (420.0 + a * (735.0 + a * (966.0 + a * (1141.0 + 1278.0 * a)))) * (1.0 / 2520.0);
    const double s3 = (210.0 + a * (462.0 + a * (707.0 + 932.0 * a))) * (1.0 / 2520.0);
    const double s4 =
        (252.0 + a * (672.0 + 1182.0 * a) + c * (294.0 + a * (889.0 + 1740.0 * a))) * (1.0 / 5040.0);
    const double s5 = (84.0 + 264.0 * a + c * (175.0 + 606.0 * a)) * (1.0 / 2520.0);
    const double s6 = (120.0 + c * (346.0 + 127.0 * c)) * (1.0 / 5040.0);
    const double nch = q + t * (1 + 0.5 * t * s1 - b * c * (s1 - b * (s2 - b * (s3 - b * (s4 - b * (s5 - b * s6))))));
    *ch = nch;
    return !(fabs(q - nch) > e * fabs(nch)) ? 1 : 0;
}

// The block's threads (GAMMA_THREADS) compute one gdasrv's rates; sm:
// GAMMA_DOUBLES doubles of shared memory.
constexpr int GAMMA_DOUBLES = 10 * MAX_CAT;
__device__ void gammaBlock(const PmatPart &P, int g, int *status, double *sm)
{
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nWarps = blockDim.x >> 5;
    const int K = P.nCat;
    const double alpha = P.gval[g];
    double *cut = sm, *sF = sm + MAX_CAT, *sE2 = sF + MAX_CAT, *sCh = sE2 + MAX_CAT, *sInv = sCh + MAX_CAT;
    double *sLp = sInv + MAX_CAT, *sLpx = sLp + MAX_CAT, *sZ = sLpx + MAX_CAT, *sLg = sZ + MAX_CAT;
    int *sState = (int *)(sLg + MAX_CAT);   // per cut point: 0 iterating, 1 converged, -1 failed
    const double v = 2.0 * alpha, xx = v / 2.0;
    const double invXx = 1.0 / xx, invA1 = 1.0 / (alpha + 1);
    // what the start values need, a warp each
    if (warp == 0 && lane == 0) sLg[0] = gm_lnGamma(xx);
    if (warp == 1 % nWarps && lane == 0) sLg[1] = gm_lnGamma(alpha + 1);
    if (lane < K - 1) {
        const double prob = (lane + 1.0) / K;
        if (warp == 2 % nWarps) sLp[lane] = log(prob);
        if (warp == 3 % nWarps) sLpx[lane] = log(prob * xx);
        if (warp == 4 % nWarps) sZ[lane] = gm_normalQuantile(prob);
    }
    __syncthreads();
    const double lg = sLg[0], lga1 = sLg[1];
    if (tid < K - 1) {
        double ch = 0.0;
        sState[tid] = chi2StartFrom((tid + 1.0) / K, v, lg, sLp[tid], sLpx[tid], sZ[tid], &ch);
        sCh[tid] = ch;
    }
    __syncthreads();
    const bool two = 2 * (K - 1) <= nWarps;   // a second warp per cut point for the factors
    const int per = two ? K - 1 : nWarps;     // cut points in hand at a time
    const int role = two ? (warp >= K - 1) : 0;
    // exp(a log x - x - lnGamma(a)), x = c / 2, on lane 0 and the AS91 step's
    // factor on lane 1: one logarithm and one exponential for both
    auto factors = [&](double c, double a, double lgA, double &f, double &e2) {
        const double x = 0.5 * c, aa = 0.6931471805;
        const double l = log(lane == 0 ? x : c);
        const double arg = lane == 0 ? a * l - x - lgA : xx * aa + lg + 0.5 * c - (xx - 1.0) * l;
        const double e = expShort(arg);
        f = __shfl_sync(FULL, e, 0);
        e2 = __shfl_sync(FULL, e, 1);
    };
    // gm_incGammaFinish with 1 / a at hand
    auto finish = [](int kind, double gin, double f, double invA) {
        return kind == 2 ? 0.0 : kind < 0 ? -1.0 : kind == 0 ? gin * (f * invA) : 1.0 - f * gin;
    };
    for (int k0 = 0; k0 < K - 1; k0 += per) {
        const int k = k0 + (two ? warp % (K - 1) : warp);
        const bool mine = k < K - 1 && warp < (two ? 2 * (K - 1) : nWarps);
        const double prob = (k + 1.0) / K;
        for (int it = 0; it < 200000; it++) {
            int open = 0;
            for (int q = k0; q < min(k0 + per, K - 1); q++) open |= sState[q] == 0;
            if (!open) break;
            const bool go = mine && sState[k] == 0;
            double ch = go ? sCh[k] : 1.0;
            double gin = 0.0, f = 0.0, e2 = 0.0, inv = 0.0;
            int kind = 0;
            if (go && (role == 1 || !two)) {
                inv = 1.0 / ch;
                factors(ch, xx, lg, f, e2);
            }
            if (go && role == 0) kind = gammaCoreWarp(0.5 * ch, xx, &gin);
            if (two) {
                if (go && role == 1 && lane == 0) {
                    sF[k] = f;
                    sE2[k] = e2;
                    sInv[k] = inv;
                }
                __syncthreads();
                if (go && role == 0) {
                    f = sF[k];
                    e2 = sE2[k];
                    inv = sInv[k];
                }
            }
            int r = 0;
            if (go && role == 0) r = chi2StepFrom(prob, v, finish(kind, gin, f, invXx), e2, inv, &ch);
            __syncthreads();   // every state read before it is written
            if (go && role == 0 && lane == 0) {
                sCh[k] = ch;
                if (r != 0) sState[k] = r;
            }
            __syncthreads();
        }
        // bin means: P(alpha+1, ch/2), the factor beside the core again
        const bool good = mine && sState[k] == 1;
        const double x = good ? (sCh[k] / (2.0 * alpha)) * alpha : 0.0;
        double gin = 0.0, f = 0.0, e2 = 0.0;
        int kind = 0;
        if (good && (role == 1 || !two)) factors(2.0 * x, alpha + 1, lga1, f, e2);
        if (good && role == 0) kind = gammaCoreWarp(x, alpha + 1, &gin);
        if (two && good && role == 1 && lane == 0) sF[k] = f;
        __syncthreads();
        if (mine && role == 0 && lane == 0) cut[k] = good ? finish(kind, gin, two ? sF[k] : f, invA1) : -1.0;
        __syncthreads();
    }
    if (tid != 0) return;
    bool bad = !(alpha > 0);
    for (int k = 0; k < K - 1; k++) bad |= !(cut[k] >= 0.0);
    double *r = P.rates + g * K;
    if (bad) {
        atomicOr_system(status, 1);   // the status word may be in host memory
        for (int c = 0; c < K; c++) r[c] = 0.0;
    } else if (K == 1) {
        r[0] = 1.0;
    } else {
        const double factor = alpha / alpha * K;
        r[0] = cut[0] * factor;
        r[K - 1] = (1 - cut[K - 2]) * factor;
        for (int i = 1; i < K - 1; i++) r[i] = (cut[i] - cut[i - 1]) * factor;
    }
}

// ----------------------------------------------------------------- eig
// One block per (part, comp, rMatrix): one warp for dim <= 8, ten warps for
// larger dims (for 20 states one task of a sweep's round, and two entries of
// the refinement's products, per thread).  Latency bounds it: of the 97 k clocks
// of a 20-state eigensystem (190 k before the sweeps ran in round-robin order and
// the products took every lane) 37 k are the 95 rounds of five sweeps, 33 k the
// two refinement steps, 9 k building S, 6 k the tests between sweeps.  Shared memory: S[dim*dim], U[dim*dim], 32 rotations (c, s, p,
// q), pi, sqrt(pi), the warps' partial sums, then (larger dims) T, W and V
// [dim*dim] each for the mixed-precision start and its refinement.
constexpr int EIG_SMALL_DIM = 8;
constexpr int EIG_THREADS_LARGE = 320;
__host__ __device__ inline int eigThreads(int maxDim) { return maxDim <= EIG_SMALL_DIM ? 32 : EIG_THREADS_LARGE; }
__host__ __device__ inline size_t eigSmemDoubles(int maxDim)
{
    return (size_t)5 * maxDim * maxDim + 4 * 32 + 2 * maxDim + 64;
}

// Rotation (c, s) that zeroes S_pq of the symmetric 2x2 block [a_pp a_pq; a_pq a_qq]:
// t = sgn(d) 2 a_pq / (|d| + sqrt(d^2 + 4 a_pq^2)), d = a_qq - a_pp, the smaller
// root, as (c, s) = (u, sgn(d) 2 a_pq) / sqrt(u^2 + 4 a_pq^2) with u = |d| + sqrt(.)
// (one square root and one reciprocal square root).
__device__ __forceinline__ float absT(float x) { return fabsf(x); }
__device__ __forceinline__ double absT(double x) { return fabs(x); }
__device__ __forceinline__ float sqrtT(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrtT(double x) { return sqrt(x); }
__device__ __forceinline__ float rsqrtT(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsqrtT(double x) { return rsqrt(x); }

template <typename T>
__device__ __forceinline__ void jacobiRotation(T app, T aqq, T apq, T &c, T &s)
{
    const T dd = aqq - app;
    const T r2 = (T)2 * apq;
    const T u = absT(dd) + sqrtT(dd * dd + r2 * r2);
    const T inv = rsqrtT(u * u + r2 * r2);
    c = u * inv;
    s = (dd >= (T)0 ? r2 : -r2) * inv;
}

// Round r of the round-robin ordering over m (even) players: the tid-th pair.
__device__ __forceinline__ void rrPair(int r, int tid, int m, int &p, int &q)
{
    int a = (tid == 0) ? m - 1 : (r + tid) % (m - 1);
    int b = (r + m - 1 - tid) % (m - 1);
    if (tid == 0) b = r % (m - 1);
    p = a < b ? a : b;
    q = a < b ? b : a;
}

// The off-diagonal and diagonal squared masses of S, summed over the block
// (warps' partials through red[]).
template <typename T>
__device__ __forceinline__ void offDiagMass(const T *S, int n, double *red, double &off, double &dg)
{
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    double o = 0.0, g = 0.0;
    for (int k = tid; k < n * n; k += nt) {
        const int i = k / n, j = k % n;
        const double v = (double)S[k];
        if (i == j) g += v * v;
        else if (i < j) o += v * v;
    }
    for (int x = 16; x; x >>= 1) {
        o += __shfl_xor_sync(0xffffffffu, o, x);
        g += __shfl_xor_sync(0xffffffffu, g, x);
    }
    if (lane == 0) {
        red[2 * warp] = o;
        red[2 * warp + 1] = g;
    }
    __syncthreads();
    off = 0.0;
    dg = 0.0;
    for (int w = 0; w < nw; w++) {
        off += red[2 * w];
        dg += red[2 * w + 1];
    }
    __syncthreads();   // every thread has read the sums before they are written again
}

// One Jacobi sweep (m - 1 rounds of n/2 disjoint rotations) on S, accumulated
// into U.  rc, rs, rp, rq: the round's rotations.  classical: an element below
// the rounding of both diagonal entries is set to zero instead of rotated.
template <typename T>
__device__ void jacobiSweep(T *S, T *U, int n, T *rc, T *rs, int *rp, int *rq, bool classical)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const int m = (n + 1) & ~1, npairs = m / 2;
    for (int r = 0; r < m - 1; r++) {
        if (tid < npairs) {
            int p, q;
            rrPair(r, tid, m, p, q);
            T c = (T)1, sn = (T)0;
            if (q < n) {
                const T apq = S[p * n + q];
                const T g = (T)100 * absT(apq);
                if (classical && apq != (T)0 && absT(S[p * n + p]) + g == absT(S[p * n + p]) &&
                    absT(S[q * n + q]) + g == absT(S[q * n + q])) {
                    S[p * n + q] = (T)0;
                    S[q * n + p] = (T)0;
                } else if (apq != (T)0) {
                    jacobiRotation<T>(S[p * n + p], S[q * n + q], apq, c, sn);
                }
            }
            rp[tid] = p;
            rq[tid] = q;
            rc[tid] = c;
            rs[tid] = sn;
        }
        __syncthreads();
        // columns p, q of S and U: one (pair, row) per thread
        for (int k = tid; k < npairs * n; k += nt) {
            const int pr = k / n, row = k - pr * n;
            const int p = rp[pr], q = rq[pr];
            if (q >= n) continue;
            const T c = rc[pr], sn = rs[pr];
            const T a = S[row * n + p], b = S[row * n + q];
            S[row * n + p] = c * a - sn * b;
            S[row * n + q] = sn * a + c * b;
            const T ua = U[row * n + p], ub = U[row * n + q];
            U[row * n + p] = c * ua - sn * ub;
            U[row * n + q] = sn * ua + c * ub;
        }
        __syncthreads();
        // rows p, q of S: one (pair, column) per thread
        for (int k = tid; k < npairs * n; k += nt) {
            const int pr = k / n, col = k - pr * n;
            const int p = rp[pr], q = rq[pr];
            if (q >= n) continue;
            const T c = rc[pr], sn = rs[pr];
            const T a = S[p * n + col], b = S[q * n + col];
            S[p * n + col] = c * a - sn * b;
            S[q * n + col] = sn * a + c * b;
        }
        __syncthreads();
    }
}

// The rotation of the 2x2 block [app apq; apq aqq], as jacobiRotation with both
// roots taken by the hardware's reciprocal square root (its rounding is far
// below what the refinement corrects); the identity where nothing is to rotate.
__device__ __forceinline__ float rsqrtHw(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void pairRotation(float app, float aqq, float apq, float &c, float &s)
{
    const float dd = aqq - app, r2 = 2.f * apq;
    const float h = dd * dd + r2 * r2;
    const float u = fabsf(dd) + h * rsqrtHw(h);
    const float inv = rsqrtHw(u * u + r2 * r2);
    const bool none = r2 == 0.f || h < 1e-36f;
    c = none ? 1.f : u * inv;
    s = none ? 0.f : (dd >= 0.f ? r2 : -r2) * inv;
}

// Where the player at position p (pair p / 2) of m sits in the next round of
// the round robin: position 0 stays, the even positions move up, the odd ones
// down, one pair a round; m - 1 rounds bring everybody back.
__host__ __device__ __forceinline__ int nextPos(int p, int m)
{
    if (p == 0) return 0;
    if (p & 1) return p == 1 ? 2 : p - 2;
    return p == m - 2 ? m - 1 : p + 2;
}

// Offset in S of the element of positions a and b: pairs in order, and in order
// within a pair (the only copy of a symmetric element the sweep keeps).
__host__ __device__ __forceinline__ int symPos(int a, int b, int m)
{
    return a < b ? a * m + b : b * m + a;
}

// One Jacobi sweep in FP32 over the block on the m x m upper triangle S0 (m the
// even of n and n + 1; the extra row zero) and the n x m eigenvectors U0; the
// results, one round an odd number of times, are in S1 and U1.  The matrix is
// kept in the order of the round robin: pair k is always rows 2k and 2k + 1, and
// a round writes what it rotated to its place in the next round's order, in the
// other buffer.  So a thread's addresses are the same in every round, pairs are
// read as float2, and a round is one phase with one barrier: a thread applies
// both rotations of one 2x2 block of S (J_k^T S_kl J_l, k <= l) or the column
// rotation of one (row, pair) piece of U, and finds the rotations it needs from
// the diagonal blocks, like every other thread that needs them.  With the pairs'
// indices looked up each round, S held in both triangles, and U in place, a
// round of a 20-state matrix took 970 clocks (1,080 with rotations in a phase of
// their own); this takes 390.
template <int TASKS>
__device__ void jacobiSweepPairs(float *S0, float *S1, float *U0, float *U1, int n, int m)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const int npairs = m / 2;
    const int nS = npairs * (npairs + 1) / 2, nSw = (nS + 31) & ~31, nTask = nSw + n * npairs;
    // tasks tid + j nt, j < TASKS, the U pieces from a warp of their own on
    int kind[TASKS];   // 0 none, 1 S block, 2 U piece
    int in0[TASKS], dl[TASKS], dk[TASKS];          // block or piece; diagonal blocks l and k
    int o00[TASKS], o01[TASKS], o10[TASKS], o11[TASKS];
#pragma unroll
    for (int j = 0; j < TASKS; j++) {
        const int t = tid + j * nt;
        kind[j] = t < nS ? 1 : (t >= nSw && t < nTask) ? 2 : 0;
        in0[j] = dl[j] = dk[j] = o00[j] = o01[j] = o10[j] = o11[j] = 0;
        if (kind[j] == 1) {   // t -> (k, l), k <= l, row by row of the upper triangle
            int k = 0, rem = t;
            while (rem >= npairs - k) {
                rem -= npairs - k;
                k++;
            }
            const int l = k + rem;
            in0[j] = 2 * k * m + 2 * l;
            dk[j] = 2 * k * m + 2 * k;
            dl[j] = 2 * l * m + 2 * l;
            const int p1 = nextPos(2 * k, m), q1 = nextPos(2 * k + 1, m);
            const int p2 = nextPos(2 * l, m), q2 = nextPos(2 * l + 1, m);
            o00[j] = symPos(p1, p2, m);
            o01[j] = symPos(p1, q2, m);
            o10[j] = symPos(q1, p2, m);   // k = l: the same element as o01, with the same value
            o11[j] = symPos(q1, q2, m);
        } else if (kind[j] == 2) {
            const int a = (t - nSw) / npairs, l = (t - nSw) - a * npairs;
            in0[j] = a * m + 2 * l;
            dl[j] = 2 * l * m + 2 * l;
            o00[j] = a * m + nextPos(2 * l, m);
            o01[j] = a * m + nextPos(2 * l + 1, m);
        }
    }
    for (int r = 0; r < m - 1; r++) {
#pragma unroll
        for (int j = 0; j < TASKS; j++) {
            if (kind[j] == 0) continue;
            const float2 l0 = *(const float2 *)(S0 + dl[j]);
            float c2, s2;
            if (kind[j] == 1) {
                const bool diag = dl[j] == dk[j];
                const float2 k0 = *(const float2 *)(S0 + dk[j]);
                const float2 m0 = *(const float2 *)(S0 + in0[j]);
                const float2 m1 = *(const float2 *)(S0 + in0[j] + m);
                const float m10 = diag ? m0.y : m1.x;
                float c1, s1;
                pairRotation(l0.x, S0[dl[j] + m + 1], l0.y, c2, s2);
                pairRotation(k0.x, S0[dk[j] + m + 1], k0.y, c1, s1);
                // columns (S J_l), then rows (J_k^T .)
                const float t00 = c2 * m0.x - s2 * m0.y, t01 = s2 * m0.x + c2 * m0.y;
                const float t10 = c2 * m10 - s2 * m1.y, t11 = s2 * m10 + c2 * m1.y;
                const float n01 = c1 * t01 - s1 * t11;
                S1[o00[j]] = c1 * t00 - s1 * t10;
                S1[o01[j]] = n01;
                S1[o10[j]] = diag ? n01 : s1 * t00 + c1 * t10;
                S1[o11[j]] = s1 * t01 + c1 * t11;
            } else {
                const float2 u = *(const float2 *)(U0 + in0[j]);
                pairRotation(l0.x, S0[dl[j] + m + 1], l0.y, c2, s2);
                U1[o00[j]] = c2 * u.x - s2 * u.y;
                U1[o01[j]] = s2 * u.x + c2 * u.y;
            }
        }
        __syncthreads();
        float *x = S0;
        S0 = S1;
        S1 = x;
        x = U0;
        U0 = U1;
        U1 = x;
    }
}

// The tasks of a sweep: n <= MAX_DIM = 32 gives at most 672 for the
// EIG_THREADS_LARGE threads of a block, up to 8 states 64 for 32.  With at most
// one a thread (20 states: 264) a round has no loop over them: with that and the
// hardware's root (rsqrtHw) 515 -> 390 clocks a round.
__device__ __forceinline__ int sweepTasks(int n, int m)
{
    const int npairs = m / 2;
    return ((npairs * (npairs + 1) / 2 + 31) & ~31) + n * npairs;
}
static_assert((MAX_DIM / 2) * (MAX_DIM / 2 + 1) / 2 + 31 + MAX_DIM * (MAX_DIM / 2) <= 3 * EIG_THREADS_LARGE,
              "every task of a sweep has a thread");

// C = A^T B (transA) or A B, n x n, row-major, every thread a strided set of outputs.
__device__ __forceinline__ void matmul64(double *C, const double *A, const double *B, int n, bool transA)
{
    for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
        const int i = k / n, j = k % n;
        double acc = 0.0;
        for (int l = 0; l < n; l++) acc += (transA ? A[l * n + i] : A[i * n + l]) * B[l * n + j];
        C[k] = acc;
    }
}

// A float's exact FP64 value assembled with integer operations (normal numbers
// and zeros; the rest through the conversion instruction).
__device__ __forceinline__ double floatToDouble(float f)
{
    const unsigned u = __float_as_uint(f);
    const unsigned ex = (u >> 23) & 0xffu, man = u & 0x7fffffu;
    const unsigned long long sign = (unsigned long long)(u >> 31) << 63;
    if (ex == 0u && man == 0u) return __longlong_as_double((long long)sign);
    if (ex == 0u || ex == 0xffu) return (double)f;
    return __longlong_as_double((long long)(sign | ((unsigned long long)(ex + 896u) << 52) |
                                            ((unsigned long long)man << 29)));
}

// A double rounded toward zero to FP32 with integer operations: magnitudes
// below FP32's normal range give a signed zero, larger ones the largest float,
// NaN and infinities go through the conversion instruction.
__device__ __forceinline__ float doubleToFloatRz(double d)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const int ex11 = (int)((b >> 52) & 0x7ffu);
    if (ex11 == 0x7ff) return (float)d;
    const int ex = ex11 - 1023 + 127;
    const unsigned sign = (unsigned)(b >> 63) << 31;
    if (ex <= 0) return __uint_as_float(sign);
    if (ex >= 255) return __uint_as_float(sign | 0x7f7fffffu);
    return __uint_as_float(sign | ((unsigned)ex << 23) | (unsigned)((b >> 29) & 0x7fffffu));
}

// k / n for k < 1024 and n <= 33, with r = ceil(65536 / n).
__device__ __forceinline__ int divSmall(int k, int r) { return (k * r) >> 16; }
__device__ __forceinline__ int divRecip(int n) { return (65535 + n) / n; }

// Entry t < triCount(n) of the upper triangle (diagonal included) of an n x n
// matrix, as (i, j), i <= j; false for the filler entries of an odd n.  Rows r
// and m - 1 - r of the even m >= n make one row of m + 1 entries.
__device__ __forceinline__ int triCount(int n)
{
    const int m = (n + 1) & ~1;
    return (m / 2) * (m + 1);
}
__device__ __forceinline__ bool triIndex(int t, int n, int rm1, int &i, int &j)
{
    const int m = (n + 1) & ~1;
    const int r = divSmall(t, rm1), c = t - r * (m + 1);
    i = c > r ? r : m - 1 - r;
    j = c > r ? c - 1 : m - 1 - c;
    return j < n;
}

// sum_l a[l sa] b[l n]
template <typename T>
__device__ __forceinline__ T dotStrided(const T *a, int sa, const T *b, int n)
{
    T acc = 0;
#pragma unroll 4
    for (int l = 0; l < n; l++) acc += a[l * sa] * b[l * n];
    return acc;
}

__device__ __forceinline__ double symAt(const double *C, int n, int i, int j)
{
    return i <= j ? C[i * n + j] : C[j * n + i];
}

// Sums (MAX false) or maxima (MAX true) of two per-thread values over the
// block, returned to every thread (warps' partials through red[]).
template <bool MAX>
__device__ __forceinline__ void blockReduce2(double &a, double &b, double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int x = 16; x; x >>= 1) {
        const double oa = __shfl_xor_sync(0xffffffffu, a, x), ob = __shfl_xor_sync(0xffffffffu, b, x);
        a = MAX ? fmax(a, oa) : a + oa;
        b = MAX ? fmax(b, ob) : b + ob;
    }
    if (lane == 0) {
        red[2 * warp] = a;
        red[2 * warp + 1] = b;
    }
    __syncthreads();
    a = red[0];
    b = red[1];
    for (int w = 1; w < nw; w++) {
        a = MAX ? fmax(a, red[2 * w]) : a + red[2 * w];
        b = MAX ? fmax(b, red[2 * w + 1]) : b + red[2 * w + 1];
    }
    __syncthreads();   // every thread has read the partials before they are written again
}

// blockReduce2 in FP32.
template <bool MAX>
__device__ __forceinline__ void blockReduce2f(float &a, float &b, double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int x = 16; x; x >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, a, x), ob = __shfl_xor_sync(0xffffffffu, b, x);
        a = MAX ? fmaxf(a, oa) : a + oa;
        b = MAX ? fmaxf(b, ob) : b + ob;
    }
    float *rf = (float *)red;
    if (lane == 0) {
        rf[2 * warp] = a;
        rf[2 * warp + 1] = b;
    }
    __syncthreads();
    a = rf[0];
    b = rf[1];
    for (int w = 1; w < nw; w++) {
        a = MAX ? fmaxf(a, rf[2 * w]) : a + rf[2 * w];
        b = MAX ? fmaxf(b, rf[2 * w + 1]) : b + rf[2 * w + 1];
    }
    __syncthreads();   // every thread has read the partials before they are written again
}

// One step of the iterative refinement of a symmetric eigendecomposition by
// Ogita and Aishima (Japan J. Indust. Appl. Math. 35, 2018, Algorithm 1).
// X holds approximate eigenvectors (columns) of the symmetric A:
//   R = I - X^T X,  S = X^T A X,  lam_i = s_ii / (1 - r_ii),
//   delta = 2 (||S - diag(lam)||_F + ||A||_F ||R||_F),
//   E_ij = (s_ij + lam_j r_ij) / (lam_j - lam_i) where |lam_j - lam_i| > delta,
//   E_ij = r_ij / 2 elsewhere (the diagonal, and pairs closer than delta),
//   X <- X + X E,
// convergent quadratically for separated eigenvalues.  R and S measure the
// residual and are formed in FP64 (upper triangles: both are symmetric), and so
// are lam and, per entry of E, the numerator and the gap; E itself, its products
// X E and the threshold delta are FP32: an error of relative size 1e-7 in E
// leaves an error of 1e-7 |E| in X, far below FP64 precision after the final
// step (whose E is of the order of the error the step before left) and
// corrected by the next step otherwise.  Every FP64 instruction counts on this
// GPU (its FP64 pipe is narrow), so the rest is FP32.
// Returns, to every thread, the largest |E_ij| over the separated pairs (emax;
// the step is applied only if it is at most maxApply) and the largest |s_ij| over
// the pairs closer than delta (cmax: the coupling the step leaves unresolved).
// lam[n] receives the eigenvalue estimates.  T, W, V: n x n FP64 scratch.
__device__ void refineStep(const double *A, double *X, double *T, double *W, double *V, double *lam, int n,
                           int maxDim, double normA, double maxApply, double *red, double &emax, double &cmax)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const int nTri = triCount(n), rm1 = divRecip(((n + 1) & ~1) + 1), rn = divRecip(n);
    // G = X^T X (upper triangle; R = I - G) and A X, one entry a thread and two
    // entries in flight: FP64 throughput (2 FMAs a clock and SM) bounds these
    // products, so lanes without an entry cost as much as those with one.  In
    // strips of four outputs, 60 to 100 threads at work, the three products
    // of a 20-state step took 21 k clocks, this 6.6 k.
    for (int t = tid; t < nTri + n * n; t += 2 * nt) {
        const double *a[2], *b[2];
        double *out[2], acc[2] = {0.0, 0.0};
        int sa[2];
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const int u = t + x * nt;
            int i = 0, j = 0;
            out[x] = nullptr;
            a[x] = X;
            b[x] = X;
            sa[x] = n;
            if (u < nTri) {
                if (triIndex(u, n, rm1, i, j)) {
                    a[x] = X + i;
                    b[x] = X + j;
                    out[x] = T + i * n + j;
                }
            } else if (u < nTri + n * n) {
                i = divSmall(u - nTri, rn);
                j = u - nTri - i * n;
                a[x] = A + i * n;
                sa[x] = 1;
                b[x] = X + j;
                out[x] = W + i * n + j;
            }
        }
        if (out[1]) {
#pragma unroll 2
            for (int l = 0; l < n; l++) {
                acc[0] += a[0][l * sa[0]] * b[0][l * n];
                acc[1] += a[1][l * sa[1]] * b[1][l * n];
            }
        } else {
            acc[0] = dotStrided(a[0], sa[0], b[0], n);
        }
        if (out[0]) *out[0] = acc[0];
        if (out[1]) *out[1] = acc[1];
    }
    __syncthreads();
    for (int t = tid; t < nTri; t += nt) {         // S = X^T A X, upper triangle
        int i, j;
        if (triIndex(t, n, rm1, i, j)) V[i * n + j] = dotStrided(X + i, n, W + j, n);
    }
    __syncthreads();
    // the eigenvalue estimates in FP64; the residual norms that set delta in
    // FP32 (a threshold needs no more)
    float so = 0.f, ro = 0.f;
    for (int t = tid; t < nTri; t += nt) {
        int i, j;
        if (!triIndex(t, n, rm1, i, j)) continue;
        const double v = V[i * n + j], g = T[i * n + j];
        if (i == j) {
            // v / g; near 1, with r = g - 1, v (1 - r + r^2) to r^3 (a division is 1,700 clocks)
            const double r = g - 1.0;
            const double l = fabs(r) <= 4e-6 ? fma(v, fma(r, r, -r), v) : v / g;
            lam[i] = l;
            const float dv = doubleToFloatRz(v - l), dr = doubleToFloatRz(1.0 - g);
            so = fmaf(dv, dv, so);
            ro = fmaf(dr, dr, ro);
        } else {
            const float vf = doubleToFloatRz(v), gf = doubleToFloatRz(g);
            so = fmaf(2.f * vf, vf, so);
            ro = fmaf(2.f * gf, gf, ro);
        }
    }
    blockReduce2f<false>(so, ro, red);   // also orders the lam[] writes before their reads
    const float delta = 2.f * (sqrtf(so) + (float)normA * sqrtf(ro));
    // E in FP32 from an FP64 numerator s_ij + lam_j r_ij (r_ij = -g_ij off the
    // diagonal; one FMA, where the two terms may cancel) and an FP64 gap
    float *E32 = (float *)W;            // E, then X in FP32, in W (A X is no longer needed)
    float *X32 = E32 + maxDim * maxDim;
    float em = 0.f, cm = 0.f;
    for (int k = tid; k < n * n; k += nt) {
        const int i = divSmall(k, rn), j = k - i * n;
        float e;
        if (i == j) {
            e = 0.5f * doubleToFloatRz(1.0 - T[k]);
        } else {
            const double g = symAt(T, n, i, j), v = symAt(V, n, i, j);
            const float gap = doubleToFloatRz(lam[j] - lam[i]);
            if (fabsf(gap) > delta) {
                e = doubleToFloatRz(fma(-lam[j], g, v)) / gap;
                em = fmaxf(em, fabsf(e));
            } else {
                e = -0.5f * doubleToFloatRz(g);
                cm = fmaxf(cm, fabsf(doubleToFloatRz(v)));
            }
        }
        E32[k] = e;
        X32[k] = doubleToFloatRz(X[k]);
    }
    blockReduce2f<true>(em, cm, red);
    emax = em;
    cmax = cm;
    if (!(em <= maxApply)) return;
    for (int k = tid; k < n * n; k += nt) {   // X += X E
        const int i = divSmall(k, rn), j = k - i * n;
        X[k] += floatToDouble(dotStrided(X32 + i * n, 1, E32 + j, n));
    }
    __syncthreads();
}

__device__ void eigBlock(const PmatPart *parts, int d, int pair, int maxDim, int *status, double *eigSmem)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const PmatPart &P = parts[d];
    const int cNum = pair / P.nR, rNum = pair % P.nR;
    const int n = P.dim;
    double *S = eigSmem;
    double *U = S + maxDim * maxDim;
    double *rc = U + maxDim * maxDim;      // 32 cos
    double *rs = rc + 32;                  // 32 sin
    int *rp = (int *)(rs + 32);            // 32 p
    int *rq = rp + 32;                     // 32 q
    double *pi = (double *)(rq + 32);
    double *sq = pi + maxDim;
    double *red = sq + maxDim;             // 2 per warp (24), then the row sums (n <= 32)
    double *rowSum = red + 24;
    double *T = red + 64;                  // [n*n]  (larger dims; the FP32 S and U first)
    double *W = T + maxDim * maxDim;       // [n*n]
    double *V = W + maxDim * maxDim;       // [n*n]
    const double *comp = P.comps + (size_t)cNum * n;
    const double *R = P.R + (size_t)rNum * n * n;

    double *ri = rc;                       // 1 / sqrt(pi), until the sweeps
    for (int i = tid; i < n; i += nt) {
        const double q = sqrt(comp[i]);
        pi[i] = comp[i];
        sq[i] = q;
        ri[i] = 1.0 / q;
    }
    // Q off-diagonals R_ij pi_j (Pf/util.c:44-74)
    for (int k = tid; k < n * n; k += nt) {
        const int i = k / n, j = k - i * n;
        S[k] = i == j ? 0.0 : R[k] * comp[j];
    }
    __syncthreads();
    // row sums (the diagonal is minus them) in four chains, and each row's share
    // of the normalising sum sum_i sum_{j!=i} pi_i Q_ij = 1 (Pf/util.c:76-115)
    for (int i = tid; i < n; i += nt) {
        double c[4] = {0.0, 0.0, 0.0, 0.0};
        for (int j = 0; j < n; j++) c[j & 3] += S[i * n + j];
        const double sum = (c[0] + c[1]) + (c[2] + c[3]);
        S[i * n + i] = -sum;
        rowSum[i] = pi[i] * sum;
    }
    __syncthreads();
    if (tid < 32) {
        const double ode = warpSum(tid < n ? rowSum[tid] : 0.0);
        if (tid == 0) red[0] = 1.0 / ode;
    }
    __syncthreads();
    const double inv = red[0];
    // the symmetric form; the upper triangle's value for both halves
    for (int k = tid; k < n * n; k += nt) {
        const int i = k / n, j = k - i * n;
        if (i == j) {
            S[k] = S[k] * inv;
        } else if (i < j) {
            const double v = S[k] * inv * sq[i] * ri[j];
            S[k] = v;
            S[j * n + i] = v;
        }
        U[k] = (i == j) ? 1.0 : 0.0;
    }
    __syncthreads();

    int converged = 0;
    if (n > 2) {
        // Mixed precision (the FP64 pipe is narrow on this GPU): Jacobi sweeps
        // in FP32 find an approximate eigenbasis X, which two FP64 refinement
        // steps (refineStep) take to FP64 accuracy with matrix products alone.
        // They are accepted when the second step's correction is at most 1e-7
        // (the error left after it is of the order of its square) and every
        // pair of eigenvalues too close to separate is coupled by at most
        // 256 eps ||A||; otherwise (near-degenerate spectra) two Newton-Schulz
        // steps in FP64 (X <- X (3I - X^T X) / 2) make X orthogonal, S <- X^T S X
        // is formed in FP64, and the FP64 Jacobi sweeps below finish from the
        // nearly diagonal S, deciding convergence themselves.
        const int m = (n + 1) & ~1, rm = divRecip(m), rn = divRecip(n);
        float *S32 = (float *)T, *D32 = (float *)W;  // the sweeps' buffers, m x m
        float *U32 = (float *)V, *Y32 = (float *)U;  // and n x m, until the FP64 steps
        float a2 = 0.f, unused = 0.f;
        for (int k = tid; k < m * m; k += nt) {
            const int i = divSmall(k, rm), j = k - i * m;
            const float v = (i < n && j < n) ? (float)S[i * n + j] : 0.f;
            S32[k] = v;
            a2 = fmaf(v, v, a2);
            if (i < n) U32[k] = i == j ? 1.f : 0.f;
        }
        blockReduce2f<false>(a2, unused, red);       // also orders the writes before the sweeps
        const double normA = sqrt((double)a2);
        // The sweeps end when every |s_ij| is at most 3e-6 of its eigenvalues'
        // gap (the first step leaves about n times its square) or, for close
        // pairs, 1e-8 ||A||.  Sweeps down to FP32 rounding cost one more.
        const float tiny = 1e-8f * (float)normA;
        for (int sweep = 0; sweep < 12; sweep++) {
            bool open = false;
            for (int k = tid; k < n * n; k += nt) {
                const int i = divSmall(k, rn), j = k - i * n;
                if (i >= j) continue;
                const float v = fabsf(S32[i * m + j]);
                open |= !(v <= tiny || v <= 3e-6f * fabsf(S32[i * (m + 1)] - S32[j * (m + 1)]));
            }
            if (!__syncthreads_or(open)) break;
            if (sweepTasks(n, m) <= nt) jacobiSweepPairs<1>(S32, D32, U32, Y32, n, m);
            else jacobiSweepPairs<3>(S32, D32, U32, Y32, n, m);
            float *x = S32;
            S32 = D32;
            D32 = x;
            x = U32;
            U32 = Y32;
            Y32 = x;
        }
        if (U32 != (float *)V) {                     // out of U before it is written
            for (int k = tid; k < n * m; k += nt) Y32[k] = U32[k];
            __syncthreads();
            U32 = Y32;
        }
        for (int k = tid; k < n * n; k += nt) {
            const int i = k / n, j = k - i * n;
            U[k] = (double)U32[i * m + j];
        }
        __syncthreads();
        double *lam = rc;                            // n <= 32 eigenvalue estimates
        double emax = 0.0, cmax = 0.0;
        bool refined = true;
        for (int it = 0; it < 2 && refined; it++) {
            refineStep(S, U, T, W, V, lam, n, maxDim, normA, 1e-3, red, emax, cmax);
            refined = emax <= 1e-3;
        }
        refined = refined && emax <= 1e-7 && cmax <= 256.0 * DBL_EPSILON * normA;
        if (refined) {
            for (int i = tid; i < n; i += nt) S[i * n + i] = lam[i];
            __syncthreads();
            converged = 1;
        }
        for (int it = 0; it < 2 && !refined; it++) {
            matmul64(T, U, U, n, true);              // G = X^T X
            __syncthreads();
            for (int k = tid; k < n * n; k += nt) {   // W = X (3I - G) / 2
                const int i = k / n, j = k % n;
                double acc = 0.0;
                for (int l = 0; l < n; l++) acc += U[i * n + l] * ((l == j ? 3.0 : 0.0) - T[l * n + j]);
                W[k] = 0.5 * acc;
            }
            __syncthreads();
            for (int k = tid; k < n * n; k += nt) U[k] = W[k];
            __syncthreads();
        }
        if (!refined) {
            matmul64(T, S, U, n, false);             // S U
            __syncthreads();
            for (int k = tid; k < n * n; k += nt) {  // U^T (S U), upper triangle
                const int i = k / n, j = k % n;
                if (i > j) continue;
                double acc = 0.0;
                for (int l = 0; l < n; l++) acc += U[l * n + i] * T[l * n + j];
                S[k] = acc;
            }
            __syncthreads();
            for (int k = tid; k < n * n; k += nt) {
                const int i = k / n, j = k % n;
                if (i > j) S[k] = S[j * n + i];
            }
            __syncthreads();
        }
    }
    for (int sweep = 0; sweep < 60 && !converged; sweep++) {
        // convergence: off-diagonal mass vs diagonal mass
        double off, dg;
        offDiagMass<double>(S, n, red, off, dg);
        if (off <= 1e-32 * dg || off == 0.0) {
            converged = 1;
            break;
        }
        // after the first sweeps an element below the rounding of both
        // diagonal entries is set to zero instead of rotated (the classical
        // Jacobi rule): rounding noise cannot keep the sweeps going
        jacobiSweep<double>(S, U, n, rc, rs, rp, rq, sweep > 3);
    }
    if (!converged && tid == 0) atomicOr_system(status, 2);
    double *out = P.eig + (size_t)pair * eigRecDoubles(n);
    float *outF = (float *)(out + n * n + 2 * n);
    for (int k = tid; k < n * n; k += nt) {
        const double u = U[k];
        const float h = (float)u;
        out[k] = u;
        outF[k] = h;
        outF[n * n + k] = (float)(u - (double)h);
    }
    for (int i = tid; i < n; i += nt) {
        out[n * n + i] = S[i * n + i];
        out[n * n + n + i] = sq[i];
        const double r = 1.0 / sq[i];
        const float sh = (float)sq[i], rh = (float)r;
        outF[2 * n * n + i] = sh;
        outF[2 * n * n + n + i] = (float)(sq[i] - (double)sh);
        outF[2 * n * n + 2 * n + i] = rh;
        outF[2 * n * n + 3 * n + i] = (float)(r - (double)rh);
    }
}

// The eigensystem of a 4-state part by one warp: the method of eigBlock's
// mixed path, the FP32 Jacobi sweeps in every lane's registers (all lanes the
// same), the refinement one (i, j) entry a lane.  False, with nothing written,
// when the refinement is not accepted (eigBlock then takes the task).  Blocks
// of threads and barriers for 16 entries, or FP64 sweeps, added 24 and 36 us to
// a setPrams, this 11; FP64 latency (some 200 clocks an operation) bounds it.  sm: 64 doubles of shared
// memory.
__device__ __forceinline__ void rotate4(float (&S)[4][4], float (&U)[4][4], int p, int q)
{
    const float dd = S[q][q] - S[p][p], r2 = 2.f * S[p][q], h = dd * dd + r2 * r2;
    if (r2 == 0.f || h < 1e-36f) return;
    const float u = fabsf(dd) + h * rsqrtf(h), inv = rsqrtf(u * u + r2 * r2);
    const float c = u * inv, s = (dd >= 0.f ? r2 : -r2) * inv;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float a = S[k][p], b = S[k][q];
        S[k][p] = c * a - s * b;
        S[k][q] = s * a + c * b;
        const float ua = U[k][p], ub = U[k][q];
        U[k][p] = c * ua - s * ub;
        U[k][q] = s * ua + c * ub;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float a = S[p][k], b = S[q][k];
        S[p][k] = c * a - s * b;
        S[q][k] = s * a + c * b;
    }
    S[q][p] = S[p][q];
}

__device__ bool eig4Warp(const PmatPart &P, int pair, double *sm)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, i = (lane >> 2) & 3, j = lane & 3;   // lanes 16-31 repeat 0-15
    const bool upper = i < j;
    double *sX = sm, *sW = sm + 16, *sA = sm + 32;
    float *sE = (float *)(sm + 48), *sX32 = sE + 16;
    const double *comp = P.comps + (size_t)(pair / P.nR) * 4;
    const double rij = P.R[(size_t)(pair % P.nR) * 16 + 4 * i + j];
    const double piJ = comp[j], sqJ = sqrt(piJ), riJ = 1.0 / sqJ;
    const double piI = __shfl_sync(FULL, piJ, i), sqI = __shfl_sync(FULL, sqJ, i);   // lane i holds j = i
    // Q off-diagonals, row sums and the normalising sum, as eigBlock
    const double q = i == j ? 0.0 : rij * piJ;
    double row = q + __shfl_xor_sync(FULL, q, 1);
    row += __shfl_xor_sync(FULL, row, 2);
    double ode = piI * row;   // the same on a row's four lanes
    ode += __shfl_xor_sync(FULL, ode, 4);
    ode += __shfl_xor_sync(FULL, ode, 8);
    const double inv = 1.0 / ode;
    double a = i == j ? -row * inv : q * inv * sqI * riJ;
    const double mirror = __shfl_sync(FULL, a, 4 * j + i);
    if (i > j) a = mirror;   // the upper triangle's value for both halves
    if (lane < 16) {
        sA[lane] = a;
        sE[lane] = (float)a;
    }
    __syncwarp();
    float S[4][4], U[4][4];
#pragma unroll
    for (int x = 0; x < 4; x++)
#pragma unroll
        for (int y = 0; y < 4; y++) {
            S[x][y] = sE[4 * x + y];
            U[x][y] = x == y ? 1.f : 0.f;
        }
    float normA = 0.f;
    for (int sweep = 0; sweep < 12; sweep++) {
        float off = 0.f, dg = 0.f;
#pragma unroll
        for (int x = 0; x < 4; x++) {
            dg = fmaf(S[x][x], S[x][x], dg);
#pragma unroll
            for (int y = x + 1; y < 4; y++) off = fmaf(S[x][y], S[x][y], off);
        }
        if (sweep == 0) normA = sqrtf(dg + 2.f * off);
        if (off <= 1e-13f * dg || off == 0.f) break;
        rotate4(S, U, 0, 3);
        rotate4(S, U, 1, 2);
        rotate4(S, U, 0, 2);
        rotate4(S, U, 1, 3);
        rotate4(S, U, 0, 1);
        rotate4(S, U, 2, 3);
    }
    __syncwarp();   // sE has been read
    if (lane == 0) {
#pragma unroll
        for (int x = 0; x < 4; x++)
#pragma unroll
            for (int y = 0; y < 4; y++) sX[4 * x + y] = (double)U[x][y];
    }
    __syncwarp();
    double lam = 0.0;
    float em = 0.f, cm = 0.f;
    for (int step = 0; step < 2; step++) {   // refineStep, one entry a lane
        double g = 0.0, w = 0.0, v = 0.0;
#pragma unroll
        for (int l = 0; l < 4; l++) {
            g = fma(sX[4 * l + i], sX[4 * l + j], g);
            w = fma(sA[4 * i + l], sX[4 * l + j], w);
        }
        if (lane < 16) sW[lane] = w;
        __syncwarp();
#pragma unroll
        for (int l = 0; l < 4; l++) v = fma(sX[4 * l + i], sW[4 * l + j], v);
        const double vUp = __shfl_sync(FULL, v, 4 * j + i);
        if (i > j) v = vUp;
        lam = v / g;   // on the diagonal
        const double lamI = __shfl_sync(FULL, lam, 5 * i), lamJ = __shfl_sync(FULL, lam, 5 * j);
        float so = 0.f, ro = 0.f;
        if (i == j) {
            const float dv = doubleToFloatRz(v - lam), dr = doubleToFloatRz(1.0 - g);
            so = dv * dv;
            ro = dr * dr;
        } else if (upper) {
            const float vf = doubleToFloatRz(v), gf = doubleToFloatRz(g);
            so = 2.f * vf * vf;
            ro = 2.f * gf * gf;
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            so += __shfl_xor_sync(FULL, so, o);
            ro += __shfl_xor_sync(FULL, ro, o);
        }
        const float delta = 2.f * (sqrtf(so) + normA * sqrtf(ro));
        float e;
        em = cm = 0.f;
        if (i == j) {
            e = 0.5f * doubleToFloatRz(1.0 - g);
        } else {
            const float gap = doubleToFloatRz(lamJ - lamI);
            if (fabsf(gap) > delta) {
                e = doubleToFloatRz(fma(-lamJ, g, v)) / gap;
                em = fabsf(e);
            } else {
                e = -0.5f * doubleToFloatRz(g);
                cm = fabsf(doubleToFloatRz(v));
            }
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            em = fmaxf(em, __shfl_xor_sync(FULL, em, o));
            cm = fmaxf(cm, __shfl_xor_sync(FULL, cm, o));
        }
        if (!(em <= 1e-3f)) return false;   // the same on every lane
        const double x = sX[4 * i + j];
        if (lane < 16) {
            sE[lane] = e;
            sX32[lane] = doubleToFloatRz(x);
        }
        __syncwarp();
        float xe = 0.f;
#pragma unroll
        for (int l = 0; l < 4; l++) xe = fmaf(sX32[4 * i + l], sE[4 * l + j], xe);
        if (lane < 16) sX[lane] = x + floatToDouble(xe);
        __syncwarp();
    }
    if (!(em <= 1e-7f && cm <= 256.f * (float)DBL_EPSILON * normA)) return false;
    if (lane < 16) {
        double *out = P.eig + (size_t)pair * eigRecDoubles(4);
        float *outF = (float *)(out + 24);
        const double u = sX[lane];
        const float h = (float)u;
        out[lane] = u;
        outF[lane] = h;
        outF[16 + lane] = (float)(u - (double)h);
        if (i == j) out[16 + i] = lam;
        if (lane < 4) {   // lane = j
            const float sh = (float)sqJ, rh = (float)riJ;
            out[20 + lane] = sqJ;
            outF[32 + lane] = sh;
            outF[36 + lane] = (float)(sqJ - (double)sh);
            outF[40 + lane] = rh;
            outF[44 + lane] = (float)(riJ - (double)rh);
        }
    }
    return true;
}

// An eigensystem task: 4 states by the first warp, the rest by the block.
__device__ void eigTask(const PmatPart *parts, int2 t, int maxDim, int *status, double *sm)
{
    __shared__ int sDone;
    if (parts[t.x].dim == 4) {
        if (threadIdx.x < 32) {
            const bool done = eig4Warp(parts[t.x], t.y, sm);
            if (threadIdx.x == 0) sDone = done;
        }
        __syncthreads();
        if (sDone) return;
    }
    eigBlock(parts, t.x, t.y, maxDim, status, sm);
}

// One launch for both: blocks [0, nE) take an eigensystem each (one block,
// latency bound), blocks [nE, nE+nG) a gamma each.
// Task lists hold (descriptor, pair or gdasrv) of the inputs that changed.
__global__ void __launch_bounds__(GAMMA_THREADS)
k_gammaEig(const PmatPart *parts, const int2 *eigTasks, int nE, const int2 *gammaTasks, int nG,
           int maxDim, int *status, const int *counts)
{
    extern __shared__ double eigSmem[];
    const int b = blockIdx.x;
    const int capE = nE;
    if (counts) {   // launched over a capacity; the live task counts are in device memory
        nE = counts[0];
        nG = counts[1];
        if (b < capE) {
            if (b >= nE) return;
        } else if (b - capE >= nG) {
            return;
        } else {
            gammaBlock(parts[gammaTasks[b - capE].x], gammaTasks[b - capE].y, status, eigSmem);
            return;
        }
    }
    if (b < nE) {
        eigTask(parts, eigTasks[b], maxDim, status, eigSmem);
    } else if (b - nE < nG) {
        const int2 t = gammaTasks[b - nE];
        gammaBlock(parts[t.x], t.y, status, eigSmem);
    }
}

// ----------------------------------------------------------------- P decks
// One lane group per (node, cat): lane k computes e_k = exp(lambda_k t) once.
// For dim^2 <= 32 (DNA) the group has G = next power of two >= dim^2 lanes of
// one warp, lane i*dim + j forms the single entry P_ij and the e values go
// round by shuffle.  Larger dims take a whole block of PDECK_BLOCK threads per
// (node, cat): the eigenvectors and e values in shared memory, each thread
// some entries of the upper triangle of the symmetric form
// Ps_ij = sum_k U_ik e_k U_jk, giving P_ij = Ps_ij sqrt(pi_j/pi_i) and P_ji =
// Ps_ij sqrt(pi_i/pi_j) (half the work, every dot product 20 long instead of
// a row of 400 per lane), in FP32-pair arithmetic.  Each descriptor's task
// range is padded to a multiple of the block so groups never straddle blocks.
constexpr int PDECK_BLOCK = 128;
__host__ __device__ inline int pdeckGroup(int dim)
{
    if (dim * dim > 32) return PDECK_BLOCK;
    int g = 1;
    while (g < dim * dim) g <<= 1;
    return g;
}

// The descriptors, node tables and branch lengths come from the parameter
// image (written only by host copies) or the pinned host image, so they are
// read before the wait on the previous kernel; the Gamma rates and
// eigensystems (k_gammaEig) and the decks (which the previous evaluation's
// pruning reads) only after it.
// counts (nullable): launched over a capacity; the live task and descriptor
// counts are counts[2] and counts[3] (a batch leaves unchanged parts out).
// FP32 pairs: value = h + l with |l| <= ulp(h) / 2 (error-free transformations,
// written with the _rn intrinsics so that no product is contracted into an FMA).
struct Pair2 {
    float h, l;
};

// Knuth's TwoSum: a + b = s + e exactly.
__device__ __forceinline__ Pair2 twoSum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return Pair2{s, e};
}

// Product of two pairs, renormalised (Dekker's FastTwoSum on the FMA-exact
// product and the cross terms); relative error about 2^-46.
__device__ __forceinline__ Pair2 pairMul(Pair2 a, Pair2 b)
{
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    const float s = __fadd_rn(p, e);
    return Pair2{s, __fsub_rn(e, __fsub_rn(s, p))};
}

// Sum of two pairs (TwoSum of the high parts, the low parts added to its
// error, renormalised).
__device__ __forceinline__ Pair2 pairAdd(Pair2 a, Pair2 b)
{
    const Pair2 s = twoSum(a.h, b.h);
    const float e = __fadd_rn(s.l, __fadd_rn(a.l, b.l));
    const float h = __fadd_rn(s.h, e);
    return Pair2{h, __fsub_rn(e, __fsub_rn(h, s.h))};
}

// 1/j! as FP32 pairs, j = 0..13.
#define P4G_INV_FACT(j, f) (float)(1.0 / (f)), (float)(1.0 / (f) - (double)(float)(1.0 / (f)))
__constant__ float kInvFact[14][2] = {
    {P4G_INV_FACT(0, 1.0)}, {P4G_INV_FACT(1, 1.0)}, {P4G_INV_FACT(2, 2.0)}, {P4G_INV_FACT(3, 6.0)},
    {P4G_INV_FACT(4, 24.0)}, {P4G_INV_FACT(5, 120.0)}, {P4G_INV_FACT(6, 720.0)}, {P4G_INV_FACT(7, 5040.0)},
    {P4G_INV_FACT(8, 40320.0)}, {P4G_INV_FACT(9, 362880.0)}, {P4G_INV_FACT(10, 3628800.0)},
    {P4G_INV_FACT(11, 39916800.0)}, {P4G_INV_FACT(12, 479001600.0)}, {P4G_INV_FACT(13, 6227020800.0)}};
#undef P4G_INV_FACT

// e^x as an FP32 pair for an FP64 argument: x = k ln2 + r with one FP64 FMA
// (|r| <= ln2 / 2), e^r by its Taylor series to r^13 / 13! (truncation below
// 2e-16) in pair arithmetic (Horner), scaled by 2^k.  Relative error about
// 5e-15.  Arguments below -87 (results below FP32's normal range) give 0.
__device__ __forceinline__ Pair2 pairExp(double x)
{
    if (x != x) return Pair2{__int_as_float(0x7fc00000), 0.f};
    if (x < -87.0) return Pair2{0.f, 0.f};
    if (x > 88.0) return Pair2{__int_as_float(0x7f800000), 0.f};
    const float kf = rintf(__fmul_rn((float)x, 1.44269504088896341f));
    const double r = fma(-(double)kf, 0.69314718055994531, x);
    const float rh = (float)r;
    const Pair2 rp{rh, (float)(r - (double)rh)};
    Pair2 y{kInvFact[13][0], kInvFact[13][1]};
#pragma unroll
    for (int j = 12; j >= 0; j--) y = pairAdd(pairMul(y, rp), Pair2{kInvFact[j][0], kInvFact[j][1]});
    const float sc = __int_as_float((127 + (int)kf) << 23);   // 2^k exactly, k in [-126, 127]
    return Pair2{__fmul_rn(y.h, sc), __fmul_rn(y.l, sc)};
}

// Dot2 (see k_pdeck) of row i of the pair matrix A and row j of U; N: the
// state count at compile time (0: n at run time).
template <int N>
__device__ __forceinline__ Pair2 dot2Row(const float *ah, const float *al, const float *uh, const float *ul, int n)
{
    float ps = 0.f, es = 0.f;   // running sum and its error sum
    auto term = [&](float a, float al, float b, float bl) {
        const float h = __fmul_rn(a, b);
        float r = __fmaf_rn(a, b, -h);   // exact: a b = h + r
        r = __fmaf_rn(a, bl, r);
        r = __fmaf_rn(al, b, r);
        const Pair2 sm = twoSum(ps, h);
        ps = sm.h;
        es = __fadd_rn(es, __fadd_rn(sm.l, r));
    };
    if (N) {   // rows of a multiple of four floats, 16-byte aligned
#pragma unroll
        for (int k = 0; k < N; k += 4) {
            const float4 a = *(const float4 *)(ah + k), b = *(const float4 *)(uh + k);
            const float4 c = *(const float4 *)(al + k), d = *(const float4 *)(ul + k);
            term(a.x, c.x, b.x, d.x);
            term(a.y, c.y, b.y, d.y);
            term(a.z, c.z, b.z, d.z);
            term(a.w, c.w, b.w, d.w);
        }
    } else {
        for (int k = 0; k < n; k++) term(ah[k], al[k], uh[k], ul[k]);
    }
    return twoSum(ps, es);
}

__global__ void k_pdeck(const PmatPart *parts, const int *prefix, int nDesc, int nTasks, const int *counts)
{
    if (counts) {
        nTasks = counts[2];
        nDesc = counts[3];
        if (nTasks <= 0 || nDesc <= 0) return;
    }
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool inRange = idx < nTasks;
    const int d = findDesc(prefix, nDesc, inRange ? idx : nTasks - 1);
    const PmatPart P = parts[d];   // a copy: the wait below does not make it be read again
    const int n = P.dim;
    const int G = pdeckGroup(n);
    const int local = idx - prefix[d];
    const int unit = local / G, g = local % G;
    const bool active = inRange && unit < P.nNodes * P.nCat;
    const int node = active ? unit / P.nCat : 0;
    const int cat = active ? unit % P.nCat : 0;
    double t = 0.0, bl = 0.0;
    const double *E = P.eig;
    int cNum = 0, rNum = 0, gNum = 0;
    bool leafNode = false;
    if (active) {
        const int *ni = P.nodeIdx + ((size_t)node * P.nParts + P.partIdx) * 3;
        cNum = ni[0];
        rNum = ni[1];
        gNum = ni[2];
        bl = P.brLen[node];
        leafNode = P.isLeaf[node] != 0;
    }
    pdlEnter();
    if (active) {
        // t as p4_calculateBigPDecksPart forms it (Pf/p4_node.c:318-343)
        if (P.nG) t = bl * P.rates[gNum * P.nCat + cat] * P.relRate;
        else t = bl * P.relRate;
        if (P.pInvar != 0.0) t = t / (1.0 - P.pInvar);
        E = P.eig + (size_t)(cNum * P.nR + rNum) * eigRecDoubles(n);
    }
    const double *lam = E + n * n, *sq = lam + n;
    if (n * n <= 32) {   // one entry per lane, in FP32 pairs as the block form below
        const int base = lane - (lane % G);
        const bool elem = active && g < n * n && node != P.root;
        const int i = elem ? g / n : 0, j = elem ? g % n : 0;
        const float *F = (const float *)(E + n * n + 2 * n);   // the record's FP32 pairs
        float ps = 0.f, es = 0.f;   // Dot2 of row i of A = U diag(e) and row j of U
        auto term = [&](float uh, float ul, float eh, float el, float b, float bl) {
            const Pair2 a = pairMul(Pair2{uh, ul}, Pair2{eh, el});
            const float h = __fmul_rn(a.h, b);
            float r = __fmaf_rn(a.h, b, -h);
            r = __fmaf_rn(a.h, bl, r);
            r = __fmaf_rn(a.l, b, r);
            const Pair2 sm = twoSum(ps, h);
            ps = sm.h;
            es = __fadd_rn(es, __fadd_rn(sm.l, r));
        };
        if (n == 4) {
            // DNA: rows i and j of U loaded before e is formed (the indices are in
            // the record for every lane: i = j = 0 where there is no entry)
            float uih[4], uil[4], ujh[4], ujl[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uih[k] = F[i * 4 + k];
                uil[k] = F[16 + i * 4 + k];
                ujh[k] = F[j * 4 + k];
                ujl[k] = F[16 + j * 4 + k];
            }
            Pair2 ek{0.f, 0.f};
            if (active && g < n) ek = pairExp(lam[g] * t);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float eh = __shfl_sync(0xffffffffu, ek.h, base + k);
                const float el = __shfl_sync(0xffffffffu, ek.l, base + k);
                if (elem) term(uih[k], uil[k], eh, el, ujh[k], ujl[k]);
            }
        } else {
            Pair2 ek{0.f, 0.f};
            if (active && g < n) ek = pairExp(lam[g] * t);
            for (int k = 0; k < n; k++) {
                const float eh = __shfl_sync(0xffffffffu, ek.h, base + k);
                const float el = __shfl_sync(0xffffffffu, ek.l, base + k);
                if (elem) term(F[i * n + k], F[n * n + i * n + k], eh, el, F[j * n + k], F[n * n + j * n + k]);
            }
        }
        Pair2 v{0.f, 0.f};
        if (elem) {
            const float *sqp = F + 2 * n * n;   // sqh, sql, rqh, rql
            v = pairMul(twoSum(ps, es), pairMul(Pair2{sqp[j], sqp[n + j]}, Pair2{sqp[2 * n + i], sqp[3 * n + i]}));
        }
        const bool leaf = elem && leafNode;
        if (elem) {
            const float f = __fadd_rn(v.h, v.l);
            const int at = leaf ? j * n + i : i * n + j;   // leaves: column j contiguous
            float *d32 = P.decks32 + (size_t)node * deckFloats(n, P.nCat);
            d32[n == 4 ? deck4Offset(P.nCat, cat, at >> 2, at & 3) : cat * n * n + at] = f;   // categories in pairs
            if (P.decks64)
                P.decks64[((size_t)node * P.nCat + cat) * n * n + i * n + j] = floatToDouble(v.h) + floatToDouble(v.l);
        }
        // partial-equate sums of a leaf's rows (j order, pair sums), gathered by
        // lane (i, 0); nPartial is the same for the whole warp (one descriptor per
        // warp), and a warp that holds no leaf deck skips them (the condition is
        // warp-uniform, so the shuffles keep every lane)
        const int nPartialW = __any_sync(0xffffffffu, leaf) ? P.nPartial : 0;
        for (int q = 0; q < nPartialW; q++) {
            const uint32_t msk = P.partialMask[q];
            Pair2 sacc{0.f, 0.f};
            for (int jj = 0; jj < n; jj++) {
                const float vh = __shfl_sync(0xffffffffu, v.h, base + i * n + jj);
                const float vl = __shfl_sync(0xffffffffu, v.l, base + i * n + jj);
                if ((msk >> jj) & 1u) sacc = pairAdd(sacc, Pair2{vh, vl});
            }
            if (leaf && j == 0)
                P.eqTab[(((size_t)node * P.nPartial + q) * P.nCat + cat) * n + i] = __fadd_rn(sacc.h, sacc.l);
        }
        return;
    }
    // a whole block for this (node, cat): the block is uniform in `active`.
    // The sums run in FP32 pairs (value = hi + lo) on the FP32 pipes, which are
    // many times wider than this GPU's FP64 pipe: with A = U diag(e^{lambda t}),
    //   M_ij = sum_k A_ik U_jk    (symmetric: the upper triangle only)
    // by the compensated dot product Dot2 of Ogita, Rump and Oishi (SIAM J. Sci.
    // Comput. 26, 2005; products split exactly with an FMA, partial sums with
    // Knuth's TwoSum), the pairs' cross terms added to the error sum, then
    // P_ij = M_ij sqrt(pi_j) / sqrt(pi_i) and P_ji = M_ij sqrt(pi_i) / sqrt(pi_j)
    // as pair products.  The result carries about 2 x 24 bits (~1e-14 of the
    // terms' magnitude); the FP64 deck is hi + lo rounded once, the FP32 deck
    // hi + lo rounded to FP32.  e^{lambda t} is a pair too (pairExp); FP64 is
    // left with its argument and range reduction and that final add.
    __shared__ __align__(16) float sUh[MAX_DIM * MAX_DIM], sUl[MAX_DIM * MAX_DIM];
    __shared__ __align__(16) float sAh[MAX_DIM * MAX_DIM], sAl[MAX_DIM * MAX_DIM];
    __shared__ float sPh[MAX_DIM * MAX_DIM], sPl[MAX_DIM * MAX_DIM];   // the deck as pairs
    __shared__ float sEh[MAX_DIM], sEl[MAX_DIM], sSq[4 * MAX_DIM];   // e pairs; sqh, sql, rqh, rql
    const int tid = threadIdx.x;
    if (active) {
        const float *F = (const float *)(E + n * n + 2 * n);   // the record's FP32 pairs
        for (int k = tid; k < n * n; k += PDECK_BLOCK) {
            sUh[k] = F[k];
            sUl[k] = F[n * n + k];
        }
        for (int k = tid; k < 4 * n; k += PDECK_BLOCK) sSq[k] = F[2 * n * n + k];
        if (tid < n) {
            const Pair2 e = pairExp(lam[tid] * t);
            sEh[tid] = e.h;
            sEl[tid] = e.l;
        }
        __syncthreads();
        for (int k = tid; k < n * n; k += PDECK_BLOCK) {   // A_ik = U_ik e_k
            const int c = k % n;
            const Pair2 a = pairMul(Pair2{sUh[k], sUl[k]}, Pair2{sEh[c], sEl[c]});
            sAh[k] = a.h;
            sAl[k] = a.l;
        }
    }
    __syncthreads();
    if (!active || node == P.root) return;
    const bool leaf = leafNode;
    float *d32 = P.decks32 + ((size_t)node * P.nCat + cat) * n * n;
    double *d64 = P.decks64 ? P.decks64 + ((size_t)node * P.nCat + cat) * n * n : nullptr;
    // tensor-core image of an internal node's P (tc::imageAt; the rows 40..47
    // stay the zeros they were allocated with)
    float *tb = (P.tcB && !leaf) ? P.tcB + ((size_t)node * P.nCat + cat) * tc::IMG_FLOATS : nullptr;
    auto put = [&](int i, int j, Pair2 v) {
        const float f = __fadd_rn(v.h, v.l);
        if (leaf) d32[j * n + i] = f;   // leaves: column j contiguous
        else d32[i * n + j] = f;
        if (d64) d64[i * n + j] = floatToDouble(v.h) + floatToDouble(v.l);
        if (tb) {
            tc::imagePut(tb, i, j, f);
        }
        sPh[i * n + j] = v.h;
        sPl[i * n + j] = v.l;
    };
    const float *sqh = sSq, *sql = sSq + n, *rqh = sSq + 2 * n, *rql = sSq + 3 * n;
    // the triangle's entries without a gap: of 20 states two passes of the block,
    // where all i, j with the lower half skipped took four
    const int nTri = triCount(n), rm1 = divRecip(((n + 1) & ~1) + 1);
    for (int u = tid; u < nTri; u += PDECK_BLOCK) {
        int i, j;
        if (!triIndex(u, n, rm1, i, j)) continue;
        const Pair2 m = n == 20 ? dot2Row<20>(sAh + i * n, sAl + i * n, sUh + j * n, sUl + j * n, n)
                                : dot2Row<0>(sAh + i * n, sAl + i * n, sUh + j * n, sUl + j * n, n);
        put(i, j, pairMul(m, pairMul(Pair2{sqh[j], sql[j]}, Pair2{rqh[i], rql[i]})));
        if (j != i) put(j, i, pairMul(m, pairMul(Pair2{sqh[i], sql[i]}, Pair2{rqh[j], rql[j]})));
    }
    if (leaf && P.nPartial) {
        __syncthreads();   // leafNode is uniform over the block
        for (int w = tid; w < P.nPartial * n; w += PDECK_BLOCK) {
            const int q = w / n, i = w - q * n;
            const uint32_t msk = P.partialMask[q];
            Pair2 sacc{0.f, 0.f};
            for (int j = 0; j < n; j++)
                if ((msk >> j) & 1u) sacc = pairAdd(sacc, Pair2{sPh[i * n + j], sPl[i * n + j]});
            P.eqTab[(((size_t)node * P.nPartial + q) * P.nCat + cat) * n + i] = __fadd_rn(sacc.h, sacc.l);
        }
    }
}

// The same two launches with the eigen/gamma task counts read from device
// memory (launched over capacities capE, capG), so that the launch shape does
// not depend on which inputs changed: what a captured CUDA graph needs.
int launchPmatDev(const PmatPart *dParts, const int2 *dEigTasks, int capE, const int2 *dGammaTasks, int capG,
                  const int *dCounts, const int *dPrefixD, int nDesc, int nD, int maxDim, int *dStatus,
                  cudaStream_t s)
{
    if (capG + capE > 0) {
        size_t per = eigSmemDoubles(maxDim);
        size_t smem = std::max<size_t>(per, GAMMA_DOUBLES) * sizeof(double);
        if (smem > 48 * 1024)
            P4G_CUDA(cudaFuncSetAttribute(k_gammaEig, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_gammaEig<<<capG + capE, capG ? GAMMA_THREADS : eigThreads(maxDim), smem, s>>>(dParts, dEigTasks, capE, dGammaTasks, capG, maxDim, dStatus,
                                                  dCounts);
        P4G_CUDA(cudaGetLastError());
    }
    if (nD > 0) {
        P4G_CUDA(launchPdl(k_pdeck, dim3((nD + PDECK_BLOCK - 1) / PDECK_BLOCK), dim3(PDECK_BLOCK), 0, s, dParts,
                           dPrefixD, nDesc, nD, dCounts));
    }
    return P4G_OK;
}

int pdeckTasks(int dim, int nNodes, int nCat)
{
    int t = nNodes * nCat * pdeckGroup(dim);
    return (t + PDECK_BLOCK - 1) / PDECK_BLOCK * PDECK_BLOCK;
}

int launchPmat(const PmatPart *dParts, const int2 *dEigTasks, int nE, const int2 *dGammaTasks, int nG,
               const int *dPrefixD, int nDesc, int nD, int maxDim, int *dStatus, cudaStream_t s)
{
    if (nG + nE > 0) {
        size_t per = eigSmemDoubles(maxDim);
        size_t smem = std::max<size_t>(per, GAMMA_DOUBLES) * sizeof(double);
        if (smem > 48 * 1024)
            P4G_CUDA(cudaFuncSetAttribute(k_gammaEig, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_gammaEig<<<nG + nE, nG ? GAMMA_THREADS : eigThreads(maxDim), smem, s>>>(dParts, dEigTasks, nE, dGammaTasks, nG, maxDim, dStatus, nullptr);
        P4G_CUDA(cudaGetLastError());
    }
    if (nD > 0) {
        // one block per protein deck (several DNA decks per block): the decks spread over the SMs
        P4G_CUDA(launchPdl(k_pdeck, dim3((nD + PDECK_BLOCK - 1) / PDECK_BLOCK), dim3(PDECK_BLOCK), 0, s, dParts,
                           dPrefixD, nDesc, nD, (const int *)nullptr));
    }
    return P4G_OK;
}

}  // namespace p4g
