// The plain FP64 GPU path: a direct restatement of the reference's pruning
// on the GPU, the FP64 evaluation mode of the library (p4g_setPrecision(tree,
// 1)), which the ML optimisation evaluates with.
//
// Same arithmetic as the reference: cl[cat][state][pattern] in FP64 from a
// node's children exactly as p4_setConditionalLikelihoodsOfInternalNodePart
// (Pf/p4_node.c:636-857) forms it -- first child assigns, later children
// multiply, leaf children look up P[s][code] (1 for gap/?/N-like, a sum over
// members for other equates), internal children sum_j P[s][j] cl[j] -- and
// no rescaling.  The root reduction follows p4_partLogLikeLoop /
// p4_partLogLikeLoopRootLeaf (Pf/p4_tree.c:1029-1378): like = sum over
// (cat, state) of pi[s] cl[cat][s][p], pInvar term, /nCat, then
// count * log(like), with the -1e99 sentinel for like <= 0.
//
// One launch for a part's whole tree: the CL of a (category, pattern) at a
// node needs those of its children at the same (category, pattern) only, so a
// thread walks all nodes in post-order for its own pair, with no barrier; the
// node before it, usually one of its children, is still in registers, and the
// two children of a binary node are formed side by side.  What bounds it is
// the FP64 pipe, 2 FMAs a clock and SM: 64 taxa x 74 k patterns x 4 categories
// need 0.6 ms.  An evaluation with a launch per node took 1.23 ms (245 us for
// 32 taxa x 7 k patterns, all launch and tail), with this kernel 0.79 ms (106 us).
#include <cuda_runtime.h>
#include <algorithm>
#include "p4g_internal.h"
#include "p4g_prune64.cuh"

namespace p4g {

// Factor of child k of the node at `node` in the table, into f: its tip
// column, or its CL (held in `last` when the child is internal node lastIdx).
template <int DIM>
__device__ __forceinline__ void childFactor(const Node64Job &J, const int *node, int k, int cat, int pat, int lastIdx,
                                            const double (&last)[DIM], double (&f)[DIM])
{
    const int child = __ldg(node + 2 + 3 * k), kind = __ldg(node + 3 + 3 * k), ref = __ldg(node + 4 + 3 * k);
    const double *P = J.decks64 + ((size_t)child * J.nCat + cat) * DIM * DIM;
    if (kind == 0) {  // leaf: raw p4 character code
        const int code = J.patterns[(size_t)ref * J.nPat + pat];
        if (code >= 0) {
#pragma unroll
            for (int s = 0; s < DIM; s++) f[s] = __ldg(P + s * DIM + code);
        } else if (code == GAP_CODE || code == QMARK_CODE || code == N_LIKE) {
#pragma unroll
            for (int s = 0; s < DIM; s++) f[s] = 1.0;
        } else {
            const int *eq = J.equates + (code - EQUATES_BASE) * DIM;
            bool isN = true;
            for (int j = 0; j < DIM; j++)
                if (!eq[j]) isN = false;
#pragma unroll
            for (int s = 0; s < DIM; s++) {
                double sum = isN ? 1.0 : 0.0;
                for (int j = 0; j < DIM && !isN; j++)
                    if (eq[j]) sum = sum + __ldg(P + s * DIM + j);
                f[s] = sum;
            }
        }
        return;
    }
    double x[DIM];   // internal child: ref = its internal index
    if (ref == lastIdx) {
#pragma unroll
        for (int j = 0; j < DIM; j++) x[j] = last[j];
    } else {
        const double *cl = J.cl + ((size_t)ref * J.nCat + cat) * DIM * J.nPatPad + pat;
#pragma unroll
        for (int j = 0; j < DIM; j++) x[j] = cl[(size_t)j * J.nPatPad];
    }
#pragma unroll
    for (int s = 0; s < DIM; s++) {
        double sum = 0.0;
#pragma unroll
        for (int j2 = 0; j2 < DIM / 2; j2++) {
            const double2 p = __ldg((const double2 *)(P + s * DIM) + j2);
            sum = sum + p.x * x[2 * j2];
            sum = sum + p.y * x[2 * j2 + 1];
        }
        f[s] = sum;
    }
}

// A block takes `chunk` patterns in every category, one thread each: thread i is
// (category i / chunk, pattern i % chunk).  At most 256 threads, 128 for 20
// states, whose 255 registers a thread leave an SM one block of 256 and the last
// of a few such blocks alone on it.  Whole warps of a category where two or more
// fit (three categories of 84 patterns instead of 64: 105 -> 125 us for 32 taxa x
// 20,000 DNA patterns; in blocks of 192 threads 114), else multiples of four patterns.  Chunks of 64 whatever
// the count, in passes of 256 threads, took 2.56 ms for 48 taxa x 10,000 protein
// patterns x 4 categories, 1.53 ms for 16 x 1,000 x 16 and 0.140 ms for 16 x 1,000
// DNA patterns x 16; these 1.99, 0.294 and 0.069 (a launch per node: 2.18, 0.431,
// 0.141).
constexpr int maxThreads64(int dim) { return dim > 4 ? 128 : 256; }
inline int chunk64(int dim, int nCat)
{
    const int n = maxThreads64(dim) / nCat;
    return n >= 64 ? n / 32 * 32 : std::max(4, n / 4 * 4);
}
static_assert(MAX_CAT * 4 <= maxThreads64(20), "a chunk of 4 patterns is one pass");

template <int DIM>
__global__ void __launch_bounds__(maxThreads64(DIM)) k_prune64(const Node64Job *__restrict__ job, int chunk)
{
    const Node64Job &J = *job;
    const int p0 = blockIdx.x * chunk;
    const int cat = threadIdx.x / chunk, pat = p0 + threadIdx.x % chunk;
    if (cat < J.nCat && pat < J.nPat) {
        double last[DIM];
#pragma unroll
        for (int s = 0; s < DIM; s++) last[s] = 0.0;
        for (int v = 0; v < J.nInternal; v++) {
            const int *node = J.table + __ldg(J.nodeStart + v);
            const int nKids = __ldg(node + 1);
            double cl[DIM], f[DIM];
            childFactor<DIM>(J, node, 0, cat, pat, v - 1, last, cl);
            int k = 1;
            if (DIM <= 4 && nKids == 2) {
                childFactor<DIM>(J, node, 1, cat, pat, v - 1, last, f);
#pragma unroll
                for (int s = 0; s < DIM; s++) cl[s] *= f[s];
                k = 2;
            }
            for (; k < nKids; k++) {
                childFactor<DIM>(J, node, k, cat, pat, v - 1, last, f);
#pragma unroll
                for (int s = 0; s < DIM; s++) cl[s] *= f[s];
            }
            double *out = J.cl + ((size_t)v * J.nCat + cat) * DIM * J.nPatPad + pat;
#pragma unroll
            for (int s = 0; s < DIM; s++) {
                out[(size_t)s * J.nPatPad] = cl[s];
                last[s] = cl[s];
            }
        }
    }
    __syncthreads();
    // root reduction, one pattern a thread, (category, state) in order
    double v = 0.0;
    int bad = 0;
    if (cat == 0 && pat < J.nPat) {
        const double *root = J.cl + (size_t)J.rootInternal * J.nCat * DIM * J.nPatPad + pat;
        double like = 0.0;
        uint32_t mask = (DIM >= 32) ? 0xffffffffu : ((1u << DIM) - 1u);
        if (J.rootLeafRow >= 0) {
            int code = J.patterns[(size_t)J.rootLeafRow * J.nPat + pat];
            if (code >= 0) mask = 1u << code;
            else if (code != GAP_CODE && code != QMARK_CODE && code != N_LIKE) {
                const int *eq = J.equates + (code - EQUATES_BASE) * DIM;
                uint32_t m = 0;
                for (int j = 0; j < DIM; j++)
                    if (eq[j]) m |= 1u << j;
                mask = m;
            }
        }
        for (int c = 0; c < J.nCat; c++)
            for (int s = 0; s < DIM; s++)
                if ((mask >> s) & 1u)
                    like = __dadd_rn(like, __dmul_rn(J.rootComp[s], root[((size_t)c * DIM + s) * J.nPatPad]));
        if (J.pInvar != 0.0) {
            like = __dmul_rn(like, J.varScale);
            uint32_t im = J.invMask[pat];
            for (int s = 0; s < DIM; s++)
                if ((im >> s) & 1u) like = __dadd_rn(like, __dmul_rn(J.rootComp[s], J.pInvar));
        } else if (J.nCat > 1) {
            like = like / (double)J.nCat;
        }
        if (!(like > 0.0)) bad = 1;
        else v = J.counts[pat] * log(like);
    }
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __shared__ double red[maxThreads64(DIM) / 32];
    __shared__ int sLast;
    const int anyBad = __syncthreads_or(bad);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = red[0];
        for (int w = 1; w < (chunk + 31) / 32; w++) s += red[w];
        J.partials[blockIdx.x] = s;
        if (anyBad) atomicOr(J.badFlag, 1);
        __threadfence();
        sLast = (atomicAdd(J.ticket, 1) == (int)gridDim.x - 1);
    }
    __syncthreads();
    if (sLast && threadIdx.x < 32) {
        __threadfence();
        double s = 0.0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) s += __ldcg(J.partials + i);
        for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) {
            *J.out = atomicExch(J.badFlag, 0) ? -1.0e99 : s;
            atomicExch(J.ticket, 0);
        }
    }
}

template <int DIM>
static int launch64(const Node64Job *dJob, const Node64Job &h, cudaStream_t s)
{
    const int chunk = chunk64(DIM, h.nCat);
    const int threads = chunk >= 64 ? maxThreads64(DIM) : (chunk * h.nCat + 31) / 32 * 32;
    k_prune64<DIM><<<(h.nPat + chunk - 1) / chunk, threads, 0, s>>>(dJob, chunk);
    P4G_CUDA(cudaGetLastError());
    return P4G_OK;
}

int launchPrune64(const Node64Job *dJob, const Node64Job &h, cudaStream_t s)
{
    switch (h.dim) {
    case 2: return launch64<2>(dJob, h, s);
    case 4: return launch64<4>(dJob, h, s);
    case 20: return launch64<20>(dJob, h, s);
    default:
        return setError(P4G_EUNSUPPORTED, "no FP64 pruning kernel for dim=%d", h.dim);
    }
}

}  // namespace p4g
