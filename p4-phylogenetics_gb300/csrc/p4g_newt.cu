// Newton optimisation of branch lengths (Pf/p4_treeNewt.c), FP64 on the GPU.
//
// The reference's p4_newtAround visits the non-root nodes in post-order and
// runs Newton-Raphson on each node's branch length, using the node's
// conditional likelihoods from below (cl, the FP64 pruning) and from above
// (cl2: at the parent's end of the branch, the likelihood of everything
// outside the node's subtree, Pf/p4_node.c:860-1018).  Which CLs have to be
// renewed before each branch (a node's cl when a branch below it moved, cl2
// once per round along the path from the first stale ancestor) depends on the
// tree alone, so the host writes a round down once as a schedule and one
// cooperative kernel, k_newtRound, runs it: every branch with its Newton
// steps, bounds and stopping rules, without the host.
//
// Every CL of a (pattern, category) depends on CLs of that (pattern, category)
// only, so a thread owns its pairs for the whole round and renews cl and cl2
// with no synchronisation.  Then, once per branch, it takes the two partials
// into the eigenbasis of the branch's Q,
//   A_k = (sum_f cl2_f U_fk / sqrt(pi_f)) (sum_t U_tk sqrt(pi_t) cl_t),
// after which a Newton step needs only
//   like = sum_k A_k e_k,  like' = sum_k (lambda_k r) A_k e_k,
//   like'' = sum_k (lambda_k r)^2 A_k e_k,    e_k = e^(lambda_k r t),
// 3n instead of 4n^2 FP64 operations per pair and step (P = U e U^T in the
// symmetric form k_pdeck uses; the reference's dP and d2P are the same sums).
// The blocks meet only to add up the derivatives (each block sums all blocks'
// partials in one order, so all take the same step) and once per branch for
// the moved node's P deck.
//
// What bounds it: the chain of Newton steps (exponentials, FP64 sums, a grid
// barrier of about 1.5 us each).  With a host round trip per step (two
// launches, a copy, a synchronisation) a whole optimisation of 32 taxa x 10,000
// sites took 101 ms; with the schedule on the device 24 ms.
//
// cl2 is stored for every node as [nNodes][nCat][dim][nPatPad] FP64 beside
// the FP64 path's cl of the internal nodes.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>
#include <algorithm>
#include <vector>
#include "p4g_internal.h"
#include "p4g_pmat.cuh"
#include "p4g_math.cuh"

using namespace p4g;

#define RET(call)                      \
    do {                               \
        int rc_ = (call);              \
        if (rc_ != P4G_OK) return rc_; \
    } while (0)

namespace {

constexpr int kMaxDim = 20;
constexpr int kMaxCat = 16;
constexpr int kMaxSibs = 16;    // of a branch whose cl2 is formed; a node has at most one child more
constexpr int kChunk = 64;      // patterns a block takes at a time
constexpr int kThreads = 256;   // 4 categories of a chunk
constexpr int kBlock = kThreads + 32;   // and a warp for the exponentials

// One data part: where its decks, CLs and tables live.
struct NewtPart {
    double *decks64;         // [nNodes][nCat][dim][dim], row = parent state
    const double *eig;       // eigensystems [(c * nR + r)][eigRecDoubles]: U, lambda, sqrt(pi)
    const double *rates;     // [nGdasrvs][nCat]
    const int *patterns;     // raw codes [nTax][nPat]
    const int *equates;      // [nEquates][dim]
    double *cl;              // internal nodes' CLs [nInternal][nCat][dim][nPatPad]
    double *cl2;             // [nNodes][nCat][dim][nPatPad]
    double *A;               // [nCat][dim][nPatPad] of the branch being moved
    const double *rootComp;  // [dim]
    const double *counts;    // [nPat]
    const uint32_t *invMask; // [nPat]
    double pInvar, relRate, catWeight;   // (1 - pInvar) / nCat
    int nPat, nPatPad, nCat, dim, nR, hasGamma;
};

// A node: its deck index and where its CL is (internal < 0: a leaf's code row).
struct NodeRef {
    int node, internal, seqNum, pad_;
};

// One CL to renew: a node's cl from its children (refs), or (isCl2) its cl2
// from its parent's and its siblings (refs).
struct NewtStep {
    NodeRef self;
    int isCl2, parent, parentIsRoot, nRefs;
    NodeRef refs[kMaxSibs + 1];
};

// The same with room for a binary tree's refs.
constexpr int kLocalSibs = 2, kMaxLocal = 6;
struct LocalStep {
    NodeRef self;
    int isCl2, parent, parentIsRoot, nRefs;
    NodeRef refs[kLocalSibs];
};
// One branch of a round: the moved node and the CLs to renew first, steps
// [step0, step0 + nSteps) of the round's list.  The first kMaxLocal that fit a
// LocalStep stand in the record, which a block copies to shared memory while
// the branch before runs (a grid barrier leaves nothing in L1, so every
// descriptor read from device memory costs an L2 round trip of some 700 clocks).
struct NewtBranch {
    NodeRef self;
    int step0, nSteps, pad_[2];
    LocalStep local[kMaxLocal];
};
static_assert(sizeof(NewtBranch) % 16 == 0, "copied in 16-byte words");

struct NewtRound {
    const NewtPart *parts;
    const int2 *chunks;          // (part, first pattern)
    const NewtStep *steps;
    const NewtBranch *branches;
    const int *nodeIdx;          // [nNodes][nParts][3] comp, rMatrix, gdasrv numbers
    double *brLen;               // [nNodes]
    double *hostBrLen;           // the same in host memory
    double2 *partials;           // [2][blocks] (d lnL, d2 lnL) of one step, double-buffered
    unsigned *counter;           // arrivals at the grid barrier; [1]: a wait gave up
    int *hostStatus;
    double epsilon, brMin, brMax;
    int nParts, nChunks, nBranches;
    int shareDecks;              // the blocks share a moved node's decks out (else each forms all)
};

// Grid barrier number *epoch (the launch is cooperative: all blocks are
// resident).  False in every thread of a block when the wait gave up or
// another block's did.
__device__ bool gridBarrier(unsigned *counter, unsigned &epoch)
{
    __shared__ int sOk;
    epoch++;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = epoch * gridDim.x;
        __threadfence();
        atomicAdd(counter, 1u);
        int ok = 0;
        for (int i = 0; i < (1 << 22) && !ok; i++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            ok = v >= target;
            if (!ok && (i & 1023) == 1023 && __ldcg((const int *)counter + 1)) break;
        }
        if (!ok) atomicExch(counter + 1, 1u);
        sOk = ok;
    }
    __syncthreads();
    return sOk != 0;
}

// What a branch length is multiplied by in one category: rate * relRate / (1 -
// pInvar), the reference's `temp` in p4_calculateBigPDecks_1stD / 2ndD
// (Pf/p4_node.c:442-540).
__device__ __forceinline__ double branchRate(const NewtPart &A, int gNum, int cat)
{
    double r = A.relRate;
    if (A.hasGamma) r = A.rates[gNum * A.nCat + cat] * r;
    return A.pInvar != 0.0 ? r / (1.0 - A.pInvar) : r;
}

// The tip factor of a leaf child, as p4_setCL2Down and the pruning treat
// codes (Pf/p4_node.c:948-990): P[s][code] for a state, nothing (1) for a
// gap, '?' or an all-states equate, the sum over members for other equates.
__device__ __forceinline__ double tipFactor(const double *P, int dim, int code, const int *equates, int s)
{
    if (code >= 0) return P[s * dim + code];
    if (code == GAP_CODE || code == QMARK_CODE || code == N_LIKE) return 1.0;
    const int *eq = equates + (code - EQUATES_BASE) * dim;
    bool isN = true;
    for (int j = 0; j < dim; j++)
        if (!eq[j]) isN = false;
    if (isN) return 1.0;
    double sum = 0.0;
    for (int j = 0; j < dim; j++)
        if (eq[j]) sum += P[s * dim + j];
    return sum;
}

// The step's CL for one (pattern, category).  cl: the children's transformed CLs
// or tip factors, in order (p4_setConditionalLikelihoodsOfInternalNodePart).
// cl2 (Pf/p4_treeNewt.c:597-619 with p4_initializeCL2ToRootComp, p4_setCL2Up,
// p4_setCL2Down): from the root composition when the parent is the root, else
// the parent's cl2 carried down the parent's branch (sum_from P_par[from][s]
// cl2_par[from]); times each sibling's transformed CL or tip factor, in order.
template <int n, class Step>
__device__ void renewItem(const NewtPart &A, double *cl, const Step &S, int cat, int pat)
{
    const size_t plane = (size_t)A.nPatPad;
    double w[n];
    for (int s = 0; s < n; s++) w[s] = 1.0;
    if (S.isCl2 && S.parentIsRoot) {
        for (int s = 0; s < n; s++) w[s] = A.rootComp[s];
    } else if (S.isCl2) {
        const double *P = A.decks64 + ((size_t)S.parent * A.nCat + cat) * n * n;
        const double *up = A.cl2 + ((size_t)S.parent * A.nCat + cat) * n * plane + pat;
        double u[n];
        for (int f = 0; f < n; f++) u[f] = up[f * plane];
        for (int s = 0; s < n; s++) {
            double sum = 0.0;
            for (int f = 0; f < n; f++) sum += P[f * n + s] * u[f];
            w[s] = sum;
        }
    }
    for (int k = 0; k < S.nRefs; k++) {
        const NodeRef b = S.refs[k];
        const double *P = A.decks64 + ((size_t)b.node * A.nCat + cat) * n * n;
        if (b.internal < 0) {
            const int code = A.patterns[(size_t)b.seqNum * A.nPat + pat];
            for (int s = 0; s < n; s++) w[s] *= tipFactor(P, n, code, A.equates, s);
        } else {
            const double *x = cl + ((size_t)b.internal * A.nCat + cat) * n * plane + pat;
            double xv[n];
            for (int j = 0; j < n; j++) xv[j] = x[j * plane];
            for (int s = 0; s < n; s++) {
                double sum = 0.0;
                for (int j = 0; j < n; j++) sum += P[s * n + j] * xv[j];
                w[s] *= sum;
            }
        }
    }
    double *out = S.isCl2 ? A.cl2 + ((size_t)S.self.node * A.nCat + cat) * n * plane + pat
                          : cl + ((size_t)S.self.internal * A.nCat + cat) * n * plane + pat;
    for (int s = 0; s < n; s++) out[s * plane] = w[s];
}

// A_k of one (pattern, category) of the moved node (see the head of the file):
// U, sq and 1/sq of its Q in shared memory.  A leaf's cl is its code's state
// set (all states for a gap), as p4_newtNode treats it (Pf/p4_treeNewt.c:240-520).
template <int n>
__device__ void coefItem(const NewtPart &A, const double *cl, const NodeRef self, const double *sU, const double *sSq,
                         const double *sRi, int cat, int pat)
{
    const size_t plane = (size_t)A.nPatPad;
    const double *c2 = A.cl2 + ((size_t)self.node * A.nCat + cat) * n * plane + pat;
    double a[n], b[n];
    for (int f = 0; f < n; f++) {
        const double w = c2[f * plane] * sRi[f];
        for (int k = 0; k < n; k++) a[k] = f ? fma(w, sU[f * n + k], a[k]) : w * sU[k];
    }
    if (self.internal >= 0) {
        const double *x = cl + ((size_t)self.internal * A.nCat + cat) * n * plane + pat;
        for (int t = 0; t < n; t++) {
            const double w = x[t * plane] * sSq[t];
            for (int k = 0; k < n; k++) b[k] = t ? fma(w, sU[t * n + k], b[k]) : w * sU[k];
        }
    } else {
        const int code = A.patterns[(size_t)self.seqNum * A.nPat + pat];
        if (code >= 0) {
            for (int k = 0; k < n; k++) b[k] = sSq[code] * sU[code * n + k];
        } else {
            const bool all = code == GAP_CODE || code == QMARK_CODE || code == N_LIKE;
            const int *eq = all ? nullptr : A.equates + (code - EQUATES_BASE) * n;
            for (int k = 0; k < n; k++) b[k] = 0.0;
            for (int t = 0; t < n; t++)
                if (all || eq[t])
                    for (int k = 0; k < n; k++) b[k] = fma(sSq[t], sU[t * n + k], b[k]);
        }
    }
    double *out = A.A + (size_t)cat * n * plane + pat;
    for (int k = 0; k < n; k++) out[k * plane] = a[k] * b[k];
}

// The branch's renewed CLs and A_k of a block's chunk.
template <int n>
__device__ void prepareChunk(const NewtRound &G, const NewtBranch &B, const NewtPart &A, const double *sU,
                             const double *sSq, const double *sRi, int p0)
{
    for (int i = threadIdx.x; i < kChunk * A.nCat; i += kThreads) {
        const int cat = i / kChunk, pat = p0 + i % kChunk;
        if (pat >= A.nPat) continue;
        for (int o = 0; o < B.nSteps; o++) {
            if (o < kMaxLocal && B.local[o].nRefs <= kLocalSibs) renewItem<n>(A, A.cl, B.local[o], cat, pat);
            else renewItem<n>(A, A.cl, G.steps[B.step0 + o], cat, pat);
        }
        coefItem<n>(A, A.cl, B.self, sU, sSq, sRi, cat, pat);
    }
}

// Likelihood and its derivatives of each (category, pattern) of a chunk.
template <int n>
__device__ void stepChunk(const NewtPart &A, const double *sE, double (*sLike)[kMaxCat][kChunk], int p0)
{
    const size_t plane = (size_t)A.nPatPad;
    for (int i = threadIdx.x; i < kChunk * A.nCat; i += kThreads) {
        const int cat = i / kChunk, j = i % kChunk, pat = p0 + j;
        if (pat >= A.nPat) continue;
        const double *a = A.A + (size_t)cat * n * plane + pat;
        const double *e = sE + cat * 3 * n;
        double like = 0.0, first = 0.0, second = 0.0;
        for (int k = 0; k < n; k++) {
            const double x = a[k * plane];
            like = fma(x, e[k], like);
            first = fma(x, e[n + k], first);
            second = fma(x, e[2 * n + k], second);
        }
        sLike[0][cat][j] = like;
        sLike[1][cat][j] = first;
        sLike[2][cat][j] = second;
    }
}

// BIG: parts of 20 states among them (with their code the kernel takes 168
// registers and spills 53 words, without it 96 and 37).
template <bool BIG>
__global__ void __launch_bounds__(kBlock) k_newtRound(NewtRound G)
{
    constexpr int ND = BIG ? kMaxDim : 4;
    __shared__ double sU[ND * ND], sSq[ND], sRi[ND], sLr[kMaxCat * ND];   // sLr: lambda_k r of each category
    __shared__ double sE[kMaxCat * 3 * ND];
    __shared__ double sLike[3][kMaxCat][kChunk];
    __shared__ double2 sRed[2];
    __shared__ __align__(16) NewtBranch sBranch[2];
    __shared__ double sBrLen[2];
    __shared__ int2 sQ[2];          // (comp, R) pair and gdasrv of the branch's node in a single part
    __shared__ NewtPart sPart;      // the part of the chunk in hand
    const int tid = threadIdx.x;
    unsigned epoch = 0;
    bool ok = true;
    // what sPart and sU .. sLr hold: the part, its (comp, R) pair and gdasrv
    int curPart = -1, curPair = -1, curG = -1;
    auto fetchBranch = [&](int bi) {   // into buffer bi & 1, read after later barriers
        if (bi >= G.nBranches) return;
        const int4 *src = (const int4 *)(G.branches + bi);
        for (int k = tid; k < (int)(sizeof(NewtBranch) / 16); k += kBlock) ((int4 *)&sBranch[bi & 1])[k] = __ldg(src + k);
        if (tid == kThreads) sBrLen[bi & 1] = __ldcg(G.brLen + __ldg(&G.branches[bi].self.node));
        if (tid == kThreads + 1 && G.nParts == 1) {
            const int *ni = G.nodeIdx + (size_t)__ldg(&G.branches[bi].self.node) * 3;
            const NewtPart &A = G.parts[0];
            sQ[bi & 1] = make_int2(ni[0] * A.nR + ni[1], A.hasGamma ? ni[2] : 0);
        }
    };
    const int2 chunk0 = G.chunks[blockIdx.x];
    double weight0 = 0.0;   // the first chunk's weights: one pattern a thread
    if (tid < kChunk && chunk0.y + tid < G.parts[chunk0.x].nPat) weight0 = G.parts[chunk0.x].counts[chunk0.y + tid];
    fetchBranch(0);
    __syncthreads();
    for (int bi = 0; bi < G.nBranches && ok; bi++) {
        const NewtBranch &B = sBranch[bi & 1];
        const int v = B.self.node;
        const double oldBrLen = sBrLen[bi & 1];
        fetchBranch(bi + 1);
        double cur = oldBrLen, result = oldBrLen;
        int iter = 0;
        for (int eval = 0;; eval++) {
            double d1 = 0.0, d2 = 0.0;   // threads 0 .. kChunk-1: one pattern of each chunk
            for (int ch = blockIdx.x; ch < G.nChunks; ch += gridDim.x) {
                const int2 c = ch == (int)blockIdx.x ? chunk0 : G.chunks[ch];
                if (c.x != curPart) {
                    __syncthreads();
                    static_assert(sizeof(NewtPart) % 8 == 0, "copied in 8-byte words");
                    for (int k = tid; k < (int)(sizeof(NewtPart) / 8); k += kBlock)
                        ((double *)&sPart)[k] = ((const double *)(G.parts + c.x))[k];
                    curPart = c.x;
                    curPair = curG = -1;
                    __syncthreads();
                }
                const NewtPart &A = sPart;
                const int n = A.dim;
                if (eval == 0 || G.nParts > 1) {   // the moved node's Q and rates in this part
                    int2 q = sQ[bi & 1];
                    if (G.nParts > 1) {
                        const int *ni = G.nodeIdx + ((size_t)v * G.nParts + c.x) * 3;
                        q = make_int2(ni[0] * A.nR + ni[1], A.hasGamma ? ni[2] : 0);
                    }
                    if (q.x != curPair || q.y != curG) {
                        __syncthreads();
                        const double *E = A.eig + (size_t)q.x * eigRecDoubles(n);
                        for (int k = tid; k < n * n; k += kBlock) sU[k] = E[k];
                        if (tid < n) {
                            const double sq = E[n * n + n + tid];
                            sSq[tid] = sq;
                            sRi[tid] = 1.0 / sq;
                        }
                        for (int k = tid; k < A.nCat * n; k += kBlock)
                            sLr[k] = E[n * n + k % n] * branchRate(A, q.y, k / n);
                        curPair = q.x;
                        curG = q.y;
                        __syncthreads();
                    }
                }
                for (int k = tid - kThreads; k >= 0 && k < A.nCat * n; k += 32) {   // the last warp's
                    const int cat = k / n, j = k - cat * n;
                    const double lr = sLr[k], ek = expShort(lr * cur);
                    double *e = sE + cat * 3 * n + j;
                    e[0] = ek;
                    e[n] = lr * ek;
                    e[2 * n] = (lr * lr) * ek;
                }
                if (eval == 0 && tid < kThreads) {   // a thread reads back only what it wrote
                    switch (n) {
                    case 2: prepareChunk<2>(G, B, A, sU, sSq, sRi, c.y); break;
                    case 4: prepareChunk<4>(G, B, A, sU, sSq, sRi, c.y); break;
                    default:
                        if constexpr (BIG) prepareChunk<20>(G, B, A, sU, sSq, sRi, c.y);
                        break;
                    }
                }
                __syncthreads();
                if (tid < kThreads) {
                    switch (n) {
                    case 2: stepChunk<2>(A, sE, sLike, c.y); break;
                    case 4: stepChunk<4>(A, sE, sLike, c.y); break;
                    default:
                        if constexpr (BIG) stepChunk<20>(A, sE, sLike, c.y);
                        break;
                    }
                }
                __syncthreads();
                const int pat = c.y + tid;
                if (tid < kChunk && pat < A.nPat) {
                    double like = 0.0, first = 0.0, second = 0.0;
                    for (int k = 0; k < A.nCat; k++) {
                        like += sLike[0][k][tid];
                        first += sLike[1][k][tid];
                        second += sLike[2][k][tid];
                    }
                    like *= A.catWeight;
                    first *= A.catWeight;
                    second *= A.catWeight;
                    if (A.pInvar != 0.0) {
                        const uint32_t im = A.invMask[pat];
                        for (int f = 0; f < n; f++)
                            if ((im >> f) & 1u) like += A.rootComp[f] * A.pInvar;
                    }
                    const double w = ch == (int)blockIdx.x ? weight0 : A.counts[pat];
                    if (like < 1.0e-300) {
                        d1 += w * 1000000.0;
                        d2 += w * 10000000.0;
                    } else {   // (second like - first^2) / like^2 with one division
                        const double inv = 1.0 / like, q = first * inv;
                        d1 = fma(w, q, d1);
                        d2 = fma(w, fma(second, inv, -(q * q)), d2);
                    }
                }
                if (G.nChunks > (int)gridDim.x) __syncthreads();   // sE and sLike are written again
            }
            if (tid < kChunk) {
                for (int o = 16; o; o >>= 1) {
                    d1 += __shfl_down_sync(0xffffffffu, d1, o);
                    d2 += __shfl_down_sync(0xffffffffu, d2, o);
                }
                if ((tid & 31) == 0) sRed[tid >> 5] = make_double2(d1, d2);
            }
            __syncthreads();
            double2 *part = G.partials + (size_t)(epoch & 1u) * gridDim.x;
            if (tid == 0) __stcg(part + blockIdx.x, make_double2(sRed[0].x + sRed[1].x, sRed[0].y + sRed[1].y));
            if (!(ok = gridBarrier(G.counter, epoch))) break;
            // every block adds the blocks' partials in the same order
            if (tid < 32) {
                double x = 0.0, y = 0.0;
                for (unsigned b0 = tid; b0 < gridDim.x; b0 += 32 * 5) {   // five loads in flight
                    double2 p[5];
#pragma unroll
                    for (int k = 0; k < 5; k++)
                        p[k] = b0 + 32 * k < gridDim.x ? __ldcg(part + b0 + 32 * k) : make_double2(0.0, 0.0);
                    x += ((p[0].x + p[1].x) + (p[2].x + p[3].x)) + p[4].x;
                    y += ((p[0].y + p[1].y) + (p[2].y + p[3].y)) + p[4].y;
                }
                for (int o = 16; o; o >>= 1) {
                    x += __shfl_xor_sync(0xffffffffu, x, o);
                    y += __shfl_xor_sync(0xffffffffu, y, o);
                }
                if (tid == 0) sRed[0] = make_double2(x, y);
            }
            __syncthreads();
            const double firstD = sRed[0].x, secondD = sRed[0].y;
            // p4_newtNode's step, bounds and stopping rules (Pf/p4_treeNewt.c:520-590)
            double next = cur - (firstD / secondD);
            if (secondD >= 0.0) next = cur / 5.0;
            if (next < G.brMin) {
                result = G.brMin;
                break;
            }
            if (next >= 5.0 * oldBrLen) {
                result = 5.0 * oldBrLen;
                break;
            }
            if (next > G.brMax) {
                result = G.brMax;
                break;
            }
            if (iter > 20 || fabs(firstD) < G.epsilon) {
                result = cur;
                break;
            }
            iter++;
            cur = next;
        }
        if (!ok) break;
        if (blockIdx.x == 0 && tid == 0) {
            G.brLen[v] = result;
            G.hostBrLen[v] = result;
        }
        // P of the final branch length, for the CLs that follow, P_ij =
        // (sq_j / sq_i) sum_k U_ik e_k U_jk.  Small decks: every block writes all
        // of them, the same values (no block still reads the old ones: the last
        // step's barrier is behind all of them), and goes on.  Otherwise the
        // blocks share the (part, category) pairs out and wait for one another.
        if (!G.shareDecks && G.nParts == 1) {   // Q is at hand
            const NewtPart &A = sPart;
            const int n = A.dim;
            if (result != cur) {   // the last step's exponentials are not those of the result
                for (int k = tid; k < A.nCat * n; k += kBlock)
                    sE[k / n * 3 * n + k % n] = expShort(sLr[k] * result);
                __syncthreads();
            }
            for (int k = tid; k < A.nCat * n * n; k += kBlock) {
                const int c = k / (n * n), i = (k - c * n * n) / n, j = k % n;
                double sum = 0.0;
                for (int q = 0; q < n; q++) sum += (sU[i * n + q] * sE[c * 3 * n + q]) * sU[j * n + q];
                A.decks64[(size_t)v * A.nCat * n * n + k] = sum * (sSq[j] * sRi[i]);
            }
            __syncthreads();
            continue;
        }
        int task = 0;
        for (int p = 0; p < G.nParts; p++) {
            const NewtPart &A = G.parts[p];
            const int n = A.dim;
            const int *ni = G.nodeIdx + ((size_t)v * G.nParts + p) * 3;
            const double *E = A.eig + (size_t)(ni[0] * A.nR + ni[1]) * eigRecDoubles(n);
            const int first = G.shareDecks ? (int)((blockIdx.x + gridDim.x - task % gridDim.x) % gridDim.x) : 0;
            const int step = G.shareDecks ? (int)gridDim.x : A.nCat;   // this block's categories: first, + step, ...
            task += A.nCat;
            for (int c0 = first; c0 < A.nCat; c0 += step) {
                const int nc = G.shareDecks ? 1 : A.nCat;
                __syncthreads();
                for (int k = tid; k < nc * n; k += kBlock)
                    sE[k] = expShort(E[n * n + k % n] * branchRate(A, ni[2], c0 + k / n) * result);
                __syncthreads();
                for (int k = tid; k < nc * n * n; k += kBlock) {
                    const int c = k / (n * n), i = (k - c * n * n) / n, j = k % n;
                    double sum = 0.0;
                    for (int q = 0; q < n; q++) sum += (E[i * n + q] * sE[c * n + q]) * E[j * n + q];
                    const double ri = 1.0 / E[n * n + n + i];
                    A.decks64[((size_t)v * A.nCat + c0) * n * n + k] = sum * (E[n * n + n + j] * ri);
                }
            }
        }
        if (G.shareDecks) ok = gridBarrier(G.counter, epoch);
        else __syncthreads();
    }
    if (!ok && tid == 0) atomicExch_system(G.hostStatus, 1);
}

// ------------------------------------------------------------------ host

struct Newt {
    Tree *t;
    std::vector<int> internalOf;   // node -> internal index of the FP64 path (-1: leaf)
    NewtRound G;
    int grid = 0;
    const void *kernel = nullptr;
};

NodeRef refOf(const Newt &N, int v)
{
    NodeRef r;
    r.node = v;
    r.internal = N.internalOf[v];
    r.seqNum = N.t->nodes[v]->seqNum;
    r.pad_ = 0;
    return r;
}

// The cl2 step of node v, or (isCl2 false) the step that renews its cl.
int stepOf(const Newt &N, int v, bool isCl2, NewtStep &S)
{
    Tree *t = N.t;
    const int par = t->nodes[v]->parent;
    memset(&S, 0, sizeof(S));
    S.self = refOf(N, v);
    S.isCl2 = isCl2;
    S.parent = par;
    S.parentIsRoot = (par == t->root);
    for (int c = t->nodes[isCl2 ? par : v]->leftChild; c >= 0; c = t->nodes[c]->sibling) {
        if (isCl2 && c == v) continue;
        if (S.nRefs == (isCl2 ? kMaxSibs : kMaxSibs + 1)) return setError(P4G_EUNSUPPORTED, "newtAround: more than %d siblings", kMaxSibs);
        S.refs[S.nRefs++] = refOf(N, c);
    }
    return P4G_OK;
}

// A round's schedule: for every branch in post-order the CLs that are stale
// when it is reached.
int scheduleRound(const Newt &N, const std::vector<int> &post, std::vector<NewtStep> &steps,
                  std::vector<NewtBranch> &branches)
{
    Tree *t = N.t;
    std::vector<char> clStale(t->nNodes, 0), cl2Stale(t->nNodes, 0);
    for (int v : post) cl2Stale[v] = v != t->root;
    for (int v : post) {
        if (v == t->root) continue;
        NewtBranch B;
        memset(&B, 0, sizeof(B));
        B.self = refOf(N, v);
        B.step0 = (int)steps.size();
        if (!t->nodes[v]->isLeaf && clStale[v]) {
            steps.emplace_back();
            RET(stepOf(N, v, false, steps.back()));
            clStale[v] = 0;
        }
        std::vector<int> path;
        for (int p = v; t->nodes[p]->parent >= 0 && cl2Stale[p]; p = t->nodes[p]->parent) path.push_back(p);
        for (int j = (int)path.size() - 1; j >= 0; j--) {
            steps.emplace_back();
            RET(stepOf(N, path[j], true, steps.back()));
            cl2Stale[path[j]] = 0;
        }
        B.nSteps = (int)steps.size() - B.step0;
        for (int k = 0; k < std::min(B.nSteps, kMaxLocal); k++) {
            const NewtStep &S = steps[B.step0 + k];
            LocalStep &L = B.local[k];
            L.self = S.self;
            L.isCl2 = S.isCl2;
            L.parent = S.parent;
            L.parentIsRoot = S.parentIsRoot;
            L.nRefs = S.nRefs;
            for (int i = 0; i < kLocalSibs; i++) L.refs[i] = S.refs[i];
        }
        branches.push_back(B);
        for (int p = t->nodes[v]->parent; p >= 0; p = t->nodes[p]->parent) clStale[p] = 1;
    }
    return P4G_OK;
}

std::vector<int> postOrderOf(Tree *t);

int newtSetup(Tree *t, Newt &N, double *lnL)
{
    if (t->root < 0 || !t->nodes[t->root] || t->nodes[t->root]->isLeaf)
        return setError(P4G_EUNSUPPORTED, "newtAround: the root must be an internal node");
    for (int p = 0; p < t->nParts; p++) {
        if (t->model->parts[p].dim > kMaxDim) return setError(P4G_EUNSUPPORTED, "newtAround: dim > %d", kMaxDim);
        if (t->model->parts[p].nCat > kMaxCat)
            return setError(P4G_EUNSUPPORTED, "newtAround: more than %d categories", kMaxCat);
    }
    N.t = t;
    // setPrams and every internal CL (p4_treeLogLike at the start of p4_newtAround)
    RET(fp64Evaluate(t, true, lnL));
    TreeDev &dv = t->dev;
    const int nn = t->nNodes, nP = t->nParts;
    N.internalOf.assign(nn, -1);
    for (size_t k = 0; k < dv.nodeStart64.size(); k++) N.internalOf[dv.table64[dv.nodeStart64[k]]] = (int)k;
    std::vector<NewtStep> steps;
    std::vector<NewtBranch> branches;
    RET(scheduleRound(N, postOrderOf(t), steps, branches));
    size_t nCl2 = 0, nA = 0;
    std::vector<size_t> oCl2(nP), oA(nP);
    std::vector<int2> chunks;
    for (int p = 0; p < nP; p++) {
        const ModelPart &mp = t->model->parts[p];
        const Part *dp = t->data->parts[p];
        oCl2[p] = nCl2;
        nCl2 += (size_t)nn * mp.nCat * mp.dim * dp->nPatPad;
        oA[p] = nA;
        nA += (size_t)mp.nCat * mp.dim * dp->nPatPad;
        for (int k = 0; k < dp->nPatterns; k += kChunk) chunks.push_back(make_int2(p, k));
    }
    RET(dv.dCl2.ensure(sizeof(double) * nCl2));
    RET(dv.dNewtA.ensure(sizeof(double) * nA));
    std::vector<NewtPart> parts(nP);
    bool big = false;   // parts of 20 states
    for (int p = 0; p < nP; p++) {
        const ModelPart &mp = t->model->parts[p];
        const Node64Job &J = dv.jobs64[p];
        NewtPart &A = parts[p];
        A.decks64 = dv.dDecks64.as<double>() + dv.oDecks[p];
        A.eig = dv.dEig.as<double>() + dv.oEig[p];
        A.rates = dv.dRates.as<double>() + dv.oRates[p];
        A.patterns = J.patterns;
        A.equates = J.equates;
        A.cl = J.cl;
        A.cl2 = dv.dCl2.as<double>() + oCl2[p];
        A.A = dv.dNewtA.as<double>() + oA[p];
        A.rootComp = J.rootComp;
        A.counts = J.counts;
        A.invMask = J.invMask;
        A.pInvar = mp.pInvar;
        A.relRate = mp.relRate;
        A.catWeight = (1.0 - mp.pInvar) / (double)mp.nCat;
        A.nPat = J.nPat;
        A.nPatPad = J.nPatPad;
        A.nCat = mp.nCat;
        A.dim = mp.dim;
        big |= mp.dim > 4;
        A.nR = mp.nRMatrices;
        A.hasGamma = mp.nGdasrvs > 0;
    }
    // as many blocks as chunks, up to what is resident at once
    int perSM = 0;
    N.kernel = big ? (const void *)k_newtRound<true> : (const void *)k_newtRound<false>;
    P4G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, N.kernel, kBlock, 0));
    N.grid = std::min((int)chunks.size(), std::max(perSM, 1) * ctx().nSM);
    // one buffer: the tables copied once, then what the kernel writes
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o = (o + bytes + 255) / 256 * 256;
        return at;
    };
    const size_t oParts = take(sizeof(NewtPart) * nP), oChunks = take(sizeof(int2) * chunks.size()),
                 oSteps = take(sizeof(NewtStep) * steps.size()),
                 oBranches = take(sizeof(NewtBranch) * branches.size());
    const size_t oBrLen = take(sizeof(double) * nn);
    const size_t tables = o;
    const size_t oPartials = take(sizeof(double2) * 2 * N.grid);
    const size_t oCounter = take(2 * sizeof(unsigned));
    RET(dv.dNewt.ensure(o));
    RET(dv.hNewt.ensure(sizeof(double) * nn + 16));   // branch lengths, then the status int
    std::vector<char> h(tables, 0);
    memcpy(h.data() + oParts, parts.data(), sizeof(NewtPart) * nP);
    memcpy(h.data() + oChunks, chunks.data(), sizeof(int2) * chunks.size());
    memcpy(h.data() + oSteps, steps.data(), sizeof(NewtStep) * steps.size());
    memcpy(h.data() + oBranches, branches.data(), sizeof(NewtBranch) * branches.size());
    double *br = (double *)(h.data() + oBrLen), *hBr = dv.hNewt.as<double>();
    for (int v = 0; v < nn; v++) br[v] = hBr[v] = t->nodes[v] ? t->nodes[v]->brLen : 0.0;
    memset(hBr + nn, 0, 16);
    cudaStream_t s = ctx().stream;
    P4G_CUDA(cudaMemcpyAsync(dv.dNewt.ptr, h.data(), tables, cudaMemcpyHostToDevice, s));
    P4G_CUDA(cudaStreamSynchronize(s));   // h goes out of scope
    char *d = (char *)dv.dNewt.ptr;
    void *hDev = nullptr;
    RET(dv.hNewt.device(&hDev));
    NewtRound &G = N.G;
    G.parts = (const NewtPart *)(d + oParts);
    G.chunks = (const int2 *)(d + oChunks);
    G.steps = (const NewtStep *)(d + oSteps);
    G.branches = (const NewtBranch *)(d + oBranches);
    G.nodeIdx = (const int *)((const char *)dv.dImg.ptr + dv.oNodeIdx);
    G.brLen = (double *)(d + oBrLen);
    G.hostBrLen = (double *)hDev;
    G.partials = (double2 *)(d + oPartials);
    G.counter = (unsigned *)(d + oCounter);
    G.hostStatus = (int *)((double *)hDev + nn);
    G.brMin = t->model->bounds[12] ? *t->model->bounds[12] : 1e-8;
    G.brMax = t->model->bounds[13] ? *t->model->bounds[13] : 3.0;
    G.nParts = nP;
    G.nChunks = (int)chunks.size();
    G.nBranches = (int)branches.size();
    // every block forming every deck costs sum nCat dim^3 FP64 FMAs at 2 a
    // clock, sharing them a grid barrier of about 3,000 clocks
    size_t deckWork = 0;
    for (int p = 0; p < nP; p++) deckWork += (size_t)parts[p].nCat * parts[p].dim * parts[p].dim * parts[p].dim;
    G.shareDecks = deckWork > 4096;
    return P4G_OK;
}

// The p4 post-order of the tree (the aliased postOrder array, entries < 0
// not in the tree).
std::vector<int> postOrderOf(Tree *t)
{
    std::vector<int> out;
    for (int k = 0; k < t->nNodes; k++) {
        const int v = t->postOrder ? t->postOrder[k] : -1;
        if (v >= 0 && v < t->nNodes) out.push_back(v);
    }
    if ((int)out.size() == 0) {   // no order given: children before parents from the relations
        std::vector<int> st{t->root};
        std::vector<char> seen(t->nNodes, 0);
        while (!st.empty()) {
            const int v = st.back();
            if (!seen[v]) {
                seen[v] = 1;
                std::vector<int> kids;
                for (int c = t->nodes[v]->leftChild; c >= 0; c = t->nodes[c]->sibling) kids.push_back(c);
                for (auto it = kids.rbegin(); it != kids.rend(); ++it) st.push_back(*it);
            } else {
                st.pop_back();
                out.push_back(v);
            }
        }
    }
    return out;
}

// p4_newtAround (Pf/p4_treeNewt.c:79-208).
int newtAround(Tree *t, double epsilon, double likeDelta, double *lnLOut)
{
    Newt N;
    double previousLogLike = 0.0;
    RET(newtSetup(t, N, &previousLogLike));
    N.G.epsilon = epsilon;
    double thisLogLike = previousLogLike;
    cudaStream_t s = ctx().stream;
    for (int round = 0; round < 20; round++) {
        P4G_CUDA(cudaMemsetAsync(N.G.counter, 0, 2 * sizeof(unsigned), s));
        void *args[] = {&N.G};
        P4G_CUDA(cudaLaunchCooperativeKernel(N.kernel, dim3(N.grid), dim3(kBlock), args, 0, s));
        // p4_treeLogLike on the new branch lengths (every CL recomputed)
        RET(fp64Evaluate(t, false, &thisLogLike));
        const double *out = t->dev.hNewt.as<double>();
        if (*(const int *)(out + t->nNodes))
            return setError(P4G_ETIMEOUT, "newtAround: a device-side wait gave up");
        for (int v = 0; v < t->nNodes; v++)
            if (v != t->root && t->nodes[v]) t->nodes[v]->brLen = out[v];
        const double diff = thisLogLike - previousLogLike;
        if (fabs(diff) < likeDelta) break;
        previousLogLike = thisLogLike;
    }
    if (lnLOut) *lnLOut = thisLogLike;
    return P4G_OK;
}

// ------------------------------------------------------------ model-parameter optimisation
// Tree.optLogLike(method="newtAndBrentPowell") (p4/tree.py:9467-9470 ->
// p4_newtAndBrentPowellOpt, Pf/p4_treeOpt.c:1182-1392): Newton passes over
// the branch lengths alternating with a derivative-free search over the free
// model parameters, until a pass changes lnL by less than 1e-6 (or the
// tree's pass limit is reached).  The reference searches with praxis
// (Brent's principal-axis method, Pf/brent.c); the search here is Powell's
// conjugate-direction method (M. J. D. Powell, Comput. J. 7:155, 1964) with
// Brent's line minimisation by golden section and parabolic interpolation
// (R. P. Brent, Algorithms for Minimization without Derivatives, 1973, ch. 5),
// written for this library, over an unconstrained reparameterisation:
//   a composition (dim values summing to 1) -> dim-1 logs of ratios to its last value;
//   an R matrix's dim(dim-1)/2 rates        -> logs of ratios to its last rate
//                                              (rates normalised to sum 1), or
//                                              logs of all but the last (last fixed);
//   a gamma shape                           -> its log;
//   pInvar                                  -> itself;
//   the relative rates of parts 0..n-2      -> logs; the last part's rate keeps
//                                              the site-weighted mean rate at 1;
//   (trees of fewer than 15 nodes, after the alternation, as the reference's
//   p4_allBrentPowellOptimize: also every branch length, by its log).
// Values are clamped to p4's bounds (the model's PIVEC_MIN, RATE_MIN, ...)
// when written back.  Each function value is an FP64 evaluation (setPrams +
// the plain FP64 pruning) on the GPU.
enum OptKind { O_COMP, O_RMAT, O_GAMMA, O_PINVAR, O_RELRATE, O_BRLEN };
struct OptBlock {
    int kind, part, idx, n, x0;
};

struct Opt {
    Tree *t = nullptr;
    std::vector<OptBlock> blocks;
    std::vector<double> step;   // first step of each coordinate's line search
    std::vector<double> rLast;  // per R-matrix block: the fixed last rate (not normalised to 1)
    int nX = 0, nEvals = 0;
    double fail = 0.0;          // first evaluation error (as a code), 0 if none

    double bnd(int k, double def) const { return t->model->bounds[k] ? *t->model->bounds[k] : def; }
    bool normR() const { return t->model->rMatrixNormalizeTo1 && t->model->rMatrixNormalizeTo1[0]; }
};

static void rUpper(const RMatrix &r, int dim, std::vector<double> &u)
{
    u.clear();
    for (int i = 0; i < dim - 1; i++)
        for (int j = i + 1; j < dim; j++) u.push_back(r.bigR[(size_t)i * dim + j]);
}

// The free parameters, as p4_windUpParameters counts them (Pf/p4_treeOpt.c:19-115).
static int optSpace(Opt &O, bool withBrLens)
{
    Tree *t = O.t;
    Model *m = t->model;
    O.blocks.clear();
    O.step.clear();
    O.rLast.clear();
    int n = 0, nModel = 0;
    auto add = [&](int kind, int part, int idx, int k, double st) {
        O.blocks.push_back(OptBlock{kind, part, idx, k, n});
        for (int i = 0; i < k; i++) O.step.push_back(st);
        n += k;
    };
    for (int p = 0; p < t->nParts; p++) {
        const ModelPart &mp = m->parts[p];
        for (int c = 0; c < mp.nComps; c++)
            if (mp.comps[c].free) add(O_COMP, p, c, mp.dim - 1, 0.3);
        for (int r = 0; r < mp.nRMatrices; r++)
            if (mp.rMatrices[r].free) {
                add(O_RMAT, p, r, mp.dim * (mp.dim - 1) / 2 - 1, 0.3);
                std::vector<double> u;
                rUpper(mp.rMatrices[r], mp.dim, u);
                O.rLast.push_back(u.back());
            }
        for (int g = 0; g < mp.nGdasrvs; g++)
            if (mp.gdasrvs[g]->free) add(O_GAMMA, p, g, 1, 0.3);
        if (mp.pInvarFree) add(O_PINVAR, p, 0, 1, 0.05);
    }
    if (m->relRatesAreFree)
        for (int p = 0; p < t->nParts - 1; p++) add(O_RELRATE, p, 0, 1, 0.2);
    nModel = n;
    if (withBrLens)
        for (int v = 0; v < t->nNodes; v++)
            if (v != t->root && t->nodes[v]) add(O_BRLEN, v, 0, 1, 0.3);
    O.nX = n;
    return nModel;
}

static void windUp(const Opt &O, std::vector<double> &x)
{
    Tree *t = O.t;
    Model *m = t->model;
    x.assign(O.nX, 0.0);
    int ri = 0;
    for (const OptBlock &B : O.blocks) {
        double *y = x.data() + B.x0;
        switch (B.kind) {
        case O_COMP: {
            const double *v = m->parts[B.part].comps[B.idx].val;
            const int d = m->parts[B.part].dim;
            for (int i = 0; i < d - 1; i++) y[i] = log(v[i]) - log(v[d - 1]);
            break;
        }
        case O_RMAT: {
            std::vector<double> u;
            rUpper(m->parts[B.part].rMatrices[B.idx], m->parts[B.part].dim, u);
            const size_t K = u.size();
            for (size_t k = 0; k + 1 < K; k++) y[k] = O.normR() ? log(u[k]) - log(u[K - 1]) : log(u[k]);
            ri++;
            break;
        }
        case O_GAMMA: y[0] = log(m->parts[B.part].gdasrvs[B.idx]->val[0]); break;
        case O_PINVAR: y[0] = m->parts[B.part].pInvar; break;
        case O_RELRATE: y[0] = log(m->parts[B.part].relRate); break;
        case O_BRLEN: y[0] = log(t->nodes[B.part]->brLen); break;
        }
    }
}

static double clampd(double v, double lo, double hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Positive values normalised to sum 1 with every value >= lo (and the last
// rounding put on the largest value).
static void normalise(std::vector<double> &v, double lo)
{
    for (int pass = 0; pass < 2; pass++) {
        double s = 0.0;
        for (double &a : v) {
            a = std::max(a, lo);
            s += a;
        }
        for (double &a : v) a /= s;
    }
    double s = 0.0;
    size_t big = 0;
    for (size_t i = 0; i < v.size(); i++) {
        s += v[i];
        if (v[i] > v[big]) big = i;
    }
    v[big] += 1.0 - s;
}

static void unWind(const Opt &O, const std::vector<double> &x)
{
    Tree *t = O.t;
    Model *m = t->model;
    int ri = 0;
    for (const OptBlock &B : O.blocks) {
        const double *y = x.data() + B.x0;
        switch (B.kind) {
        case O_COMP: {
            ModelPart &mp = m->parts[B.part];
            std::vector<double> v(mp.dim);
            for (int i = 0; i < mp.dim - 1; i++) v[i] = exp(clampd(y[i], -60.0, 60.0));
            v[mp.dim - 1] = 1.0;
            normalise(v, O.bnd(6, 1e-13));
            for (int i = 0; i < mp.dim; i++) mp.comps[B.idx].val[i] = v[i];
            break;
        }
        case O_RMAT: {
            ModelPart &mp = m->parts[B.part];
            const int d = mp.dim, K = d * (d - 1) / 2;
            std::vector<double> u(K);
            for (int k = 0; k < K - 1; k++) u[k] = exp(clampd(y[k], -60.0, 60.0));
            if (O.normR()) {
                u[K - 1] = 1.0;
                normalise(u, O.bnd(8, 1e-13));
            } else {
                u[K - 1] = O.rLast[ri];
            }
            int k = 0;
            for (int i = 0; i < d - 1; i++)
                for (int j = i + 1; j < d; j++) {
                    mp.rMatrices[B.idx].bigR[(size_t)i * d + j] = u[k];
                    mp.rMatrices[B.idx].bigR[(size_t)j * d + i] = u[k];
                    k++;
                }
            ri++;
            break;
        }
        case O_GAMMA:
            m->parts[B.part].gdasrvs[B.idx]->val[0] = clampd(exp(clampd(y[0], -60.0, 60.0)), O.bnd(4, 0.1), O.bnd(5, 300.0));
            break;
        case O_PINVAR: m->parts[B.part].pInvar = clampd(y[0], O.bnd(0, 0.0), O.bnd(1, 0.99)); break;
        case O_RELRATE:
            m->parts[B.part].relRate = clampd(exp(clampd(y[0], -60.0, 60.0)), O.bnd(10, 1e-8), O.bnd(11, 1e8));
            break;
        case O_BRLEN:
            t->nodes[B.part]->brLen = clampd(exp(clampd(y[0], -60.0, 60.0)), O.bnd(12, 1e-8), O.bnd(13, 3.0));
            break;
        }
    }
    if (m->relRatesAreFree && t->nParts > 1) {   // the last part keeps the site-weighted mean at 1
        double tot = 0.0, rest = 0.0;
        for (int p = 0; p < t->nParts; p++) tot += t->data->parts[p]->nChar;
        for (int p = 0; p < t->nParts - 1; p++) rest += m->parts[p].relRate * t->data->parts[p]->nChar;
        const int last = t->nParts - 1;
        m->parts[last].relRate = std::max((tot - rest) / t->data->parts[last]->nChar, O.bnd(10, 1e-8));
    }
}

// -lnL at x (FP64 setPrams + pruning); a failed or non-positive evaluation
// counts as +infinity, the first error code is kept.
static double optF(Opt &O, const std::vector<double> &x)
{
    unWind(O, x);
    O.nEvals++;
    double lnL = 0.0;
    const int rc = fp64Evaluate(O.t, true, &lnL);
    if (rc != P4G_OK) {
        if (O.fail == 0.0) O.fail = rc;
        return INFINITY;
    }
    if (!(lnL > -1.0e98)) return INFINITY;
    return -lnL;
}

// Minimise f(x + a d) over a (Brent 1973, ch. 5): bracket from a = 0 and
// a = 1 by golden-ratio expansion, then golden-section steps and parabolic
// interpolation.  x and fx move to the minimum found.
static void lineMin(Opt &O, std::vector<double> &x, const std::vector<double> &d, double &fx)
{
    const double G = 1.618033988749895, CG = 0.3819660112501051;
    const size_t n = x.size();
    std::vector<double> xt(n);
    auto g = [&](double a) {
        for (size_t i = 0; i < n; i++) xt[i] = x[i] + a * d[i];
        return optF(O, xt);
    };
    double a = 0.0, fa = fx, b = 1.0, fb = g(b);
    if (fb > fa) {
        std::swap(a, b);
        std::swap(fa, fb);
    }
    double c = b + G * (b - a), fc = g(c);
    for (int k = 0; k < 60 && fc < fb; k++) {
        a = b;
        fa = fb;
        b = c;
        fb = fc;
        c = b + G * (b - a);
        fc = g(c);
    }
    // Brent's minimiser on [lo, hi] starting from the bracket's middle point
    double lo = std::min(a, c), hi = std::max(a, c);
    double xm = b, w = b, v = b, fxm = fb, fw = fb, fv = fb, e = 0.0, dd = 0.0;
    for (int it = 0; it < 100; it++) {
        const double mid = 0.5 * (lo + hi);
        const double tol1 = 1.0e-5 * fabs(xm) + 1.0e-8, tol2 = 2.0 * tol1;
        if (fabs(xm - mid) <= tol2 - 0.5 * (hi - lo)) break;
        bool golden = true;
        if (fabs(e) > tol1) {   // try a parabola through x, w, v
            double r = (xm - w) * (fxm - fv), q = (xm - v) * (fxm - fw), p = (xm - v) * q - (xm - w) * r;
            q = 2.0 * (q - r);
            if (q > 0.0) p = -p;
            q = fabs(q);
            const double eOld = e;
            e = dd;
            if (fabs(p) < fabs(0.5 * q * eOld) && p > q * (lo - xm) && p < q * (hi - xm)) {
                dd = p / q;
                const double u = xm + dd;
                if (u - lo < tol2 || hi - u < tol2) dd = (mid >= xm) ? tol1 : -tol1;
                golden = false;
            }
        }
        if (golden) {
            e = (xm >= mid) ? lo - xm : hi - xm;
            dd = CG * e;
        }
        const double u = (fabs(dd) >= tol1) ? xm + dd : xm + (dd > 0.0 ? tol1 : -tol1);
        const double fu = g(u);
        if (fu <= fxm) {
            if (u >= xm) lo = xm;
            else hi = xm;
            v = w;
            fv = fw;
            w = xm;
            fw = fxm;
            xm = u;
            fxm = fu;
        } else {
            if (u < xm) lo = u;
            else hi = u;
            if (fu <= fw || w == xm) {
                v = w;
                fv = fw;
                w = u;
                fw = fu;
            } else if (fu <= fv || v == xm || v == w) {
                v = u;
                fv = fu;
            }
        }
    }
    if (fxm < fx) {
        for (size_t i = 0; i < n; i++) x[i] += xm * d[i];
        fx = fxm;
    }
    unWind(O, x);
}

// Powell's method from x (f(x) = fx): line searches along n directions,
// then along the pass's net displacement, which replaces the direction of
// largest decrease when Powell's test accepts it.  Returns f at the result.
static double powell(Opt &O, std::vector<double> &x, double fx)
{
    const size_t n = x.size();
    std::vector<std::vector<double>> dirs(n, std::vector<double>(n, 0.0));
    for (size_t i = 0; i < n; i++) dirs[i][i] = O.step[i];
    std::vector<double> xs(n), xe(n), dn(n);
    for (int it = 0; it < 200; it++) {
        const double fs = fx;
        xs = x;
        double big = 0.0;
        size_t ibig = 0;
        for (size_t i = 0; i < n; i++) {
            const double fp = fx;
            lineMin(O, x, dirs[i], fx);
            if (fp - fx > big) {
                big = fp - fx;
                ibig = i;
            }
        }
        if (2.0 * (fs - fx) <= 1.0e-10 * (fabs(fs) + fabs(fx)) + 1.0e-12) break;
        for (size_t i = 0; i < n; i++) {
            xe[i] = 2.0 * x[i] - xs[i];
            dn[i] = x[i] - xs[i];
        }
        const double fe = optF(O, xe);
        unWind(O, x);
        if (fe < fs) {
            const double tt = 2.0 * (fs - 2.0 * fx + fe) * (fs - fx - big) * (fs - fx - big) - big * (fs - fe) * (fs - fe);
            if (tt < 0.0) {
                lineMin(O, x, dn, fx);
                dirs[ibig] = dirs[n - 1];
                dirs[n - 1] = dn;
            }
        }
    }
    return fx;
}

int newtAndBrentPowellOpt(Tree *t)
{
    Opt O;
    O.t = t;
    double lnL = 0.0;
    // the model's nFreePrams decides, as in the reference: with none, branch
    // lengths only, whatever the free flags say
    const int nModel = t->model->nFreePrams == 0 ? 0 : optSpace(O, false);
    if (nModel != t->model->nFreePrams)
        return setError(P4G_EINVAL, "newtAndBrentPowellOpt: the model says %d free parameters, the free flags give %d",
                        t->model->nFreePrams, nModel);
    if (nModel == 0) {   // Pf/p4_treeOpt.c:1215-1224
        const double eps[4] = {1.0, 1.0e-1, 1.0e-2, 1.0e-5}, delta[4] = {10.0, 1.0, 0.1, 1.0e-7};
        for (int k = 0; k < 4; k++) RET(newtAround(t, eps[k], delta[k], &lnL));
        return P4G_OK;
    }
    const double eps[3] = {1.0, 1.0e-1, 1.0e-5}, delta[3] = {10.0, 1.0, 1.0e-7};
    for (int k = 0; k < 3; k++) RET(newtAround(t, eps[k], delta[k], &lnL));
    std::vector<double> x;
    windUp(O, x);
    double prev = -optF(O, x);
    const int limit = t->passLimit ? t->passLimit[0] : 50;
    for (int pass = 0;; pass++) {
        RET(newtAround(t, 1.0e-5, 1.0e-7, &lnL));
        windUp(O, x);
        const double cur = -powell(O, x, -lnL);
        if (O.fail != 0.0) return setError((int)O.fail, "newtAndBrentPowellOpt: an evaluation failed");
        unWind(O, x);
        if (fabs(cur - prev) < 1.0e-6 || pass >= limit) break;
        prev = cur;
    }
    if (t->nNodes < 15) {   // small trees: every branch length as well (Pf/p4_treeOpt.c:1384-1388)
        Opt A;
        A.t = t;
        optSpace(A, true);
        std::vector<double> y;
        windUp(A, y);
        double f = optF(A, y);
        for (int pass = 0; pass < 50; pass++) {
            const double f0 = f;
            f = powell(A, y, f);
            if (fabs(f - f0) < 1.0e-6) break;
        }
        unWind(A, y);
        if (A.fail != 0.0) return setError((int)A.fail, "newtAndBrentPowellOpt: an evaluation failed");
    }
    RET(fp64Evaluate(t, true, &lnL));
    return P4G_OK;
}

}  // namespace

extern "C" int p4g_newtSetup(p4g_tree *tt)
{
    Tree *t = reinterpret_cast<Tree *>(tt);
    if (!t) return setError(P4G_EINVAL, "newtSetup: null tree");
    return P4G_OK;   // the buffers are sized by each p4g_newtAround call
}

extern "C" int p4g_newtAround(p4g_tree *tt, double epsilon, double likeDelta)
{
    Tree *t = reinterpret_cast<Tree *>(tt);
    if (!t) return setError(P4G_EINVAL, "newtAround: null tree");
    double lnL = 0.0;
    RET(newtAround(t, epsilon, likeDelta, &lnL));
    t->dev.cacheValid = false;   // branch lengths moved: the next setPrams recomputes every deck
    return P4G_OK;
}

extern "C" int p4g_newtAndBrentPowellOpt(p4g_tree *tt)
{
    Tree *t = reinterpret_cast<Tree *>(tt);
    if (!t) return setError(P4G_EINVAL, "newtAndBrentPowellOpt: null tree");
    const int rc = newtAndBrentPowellOpt(t);
    t->dev.cacheValid = false;   // branch lengths and model values moved
    return rc;
}

extern "C" int p4g_getFreePrams(p4g_tree *tt, double *out, int cap, int *n)
{
    Tree *t = reinterpret_cast<Tree *>(tt);
    if (!t || !n || (cap > 0 && !out)) return setError(P4G_EINVAL, "getFreePrams: bad arguments");
    std::vector<double> v;
    const Model *m = t->model;
    for (int p = 0; p < t->nParts; p++) {   // p4_windUpParameters order (Pf/p4_treeOpt.c:19-115)
        const ModelPart &mp = m->parts[p];
        for (int c = 0; c < mp.nComps; c++)
            if (mp.comps[c].free)
                for (int i = 0; i < mp.dim - 1; i++) v.push_back(mp.comps[c].val[i]);
        for (int r = 0; r < mp.nRMatrices; r++)
            if (mp.rMatrices[r].free)
                for (int i = 0; i < mp.dim - 2; i++)
                    for (int j = i + 1; j < mp.dim; j++) v.push_back(mp.rMatrices[r].bigR[(size_t)i * mp.dim + j]);
        for (int g = 0; g < mp.nGdasrvs; g++)
            if (mp.gdasrvs[g]->free) v.push_back(mp.gdasrvs[g]->val[0]);
        if (mp.pInvarFree) v.push_back(mp.pInvar);
    }
    if (m->relRatesAreFree)
        for (int p = 0; p < t->nParts - 1; p++) v.push_back(m->parts[p].relRate);
    *n = (int)v.size();
    if ((int)v.size() > cap) return setError(P4G_EINVAL, "getFreePrams: %d values, room for %d", (int)v.size(), cap);
    for (size_t i = 0; i < v.size(); i++) out[i] = v[i];
    return P4G_OK;
}

extern "C" int p4g_getBrLens(p4g_tree *tt, double *out)
{
    Tree *t = reinterpret_cast<Tree *>(tt);
    if (!t || !out) return setError(P4G_EINVAL, "getBrLens: bad arguments");
    for (int v = 0; v < t->nNodes; v++) out[v] = t->nodes[v] ? t->nodes[v]->brLen : 0.0;
    if (t->root >= 0 && t->root < t->nNodes) out[t->root] = -1.0;   // the reference's placeholder
    return P4G_OK;
}
