// Per-site outputs of an evaluation: the site likelihoods pf.getSiteLikes
// returns (Pf/pfmodule.c:378), expanded from the patterns' log likelihoods.
//
// One thread a site: its pattern's lnL gathered from device memory,
// exponentiated (FP64) and stored in the part's host buffer, so that neither
// the patterns' values nor the sites' are copied.  Bound by the stores to host
// memory (3.2 MB for 400,000 sites).  Copying the patterns' lnL and expanding
// them on one host core took 1.3 ms of a 1.6 ms evaluation of 61 taxa x
// 400,000 sites.
//
// The buffer holds the part's last accepted evaluation: the kernel writes
// nothing when setPrams failed or a part's lnL is not a number, the tests
// after which the host refuses the evaluation.  Those words lie in host
// memory; their loads are under way while the first site is exponentiated.
#include <cuda_runtime.h>
#include <algorithm>
#include "p4g_internal.h"

#define RET(call)                      \
    do {                               \
        int rc_ = (call);              \
        if (rc_ != P4G_OK) return rc_; \
    } while (0)

namespace p4g {

namespace {

// partLnl, status: the evaluation's nParts lnLs and setPrams status
__global__ void __launch_bounds__(1024) k_siteLikes(const double *__restrict__ lnl, const int *__restrict__ seqPos, int nChar,
                            double *__restrict__ out, const volatile double *partLnl, int nParts,
                            const volatile int *status)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int good = threadIdx.x > 0 || *status == 0;
    for (int p = threadIdx.x; p < nParts; p += blockDim.x) {
        const double x = partLnl[p];
        good &= x == x;
    }
    double v = i < nChar ? exp(lnl[seqPos[i]]) : 0.0;
    if (!__syncthreads_and(good)) return;
    while (i < nChar) {
        out[i] = v;
        i += gridDim.x * blockDim.x;
        if (i < nChar) v = exp(lnl[seqPos[i]]);
    }
}

}  // namespace

int Part::uploadSites(cudaStream_t s)
{
    std::lock_guard<std::mutex> hold(sitesLock);
    if (sitesGen == gen && dSeqPos.ptr) return P4G_OK;
    RET(dSeqPos.ensure(sizeof(int) * std::max(nChar, 1)));
    P4G_CUDA(cudaMemcpyAsync(dSeqPos.ptr, seqPosIdx.data(), sizeof(int) * nChar, cudaMemcpyHostToDevice, s));
    sitesGen = gen;
    return P4G_OK;
}

int launchSiteLikes(Part *p, const double *dLnl, const double *partLnl, int nParts, const int *status, cudaStream_t s)
{
    RET(p->uploadSites(s));
    void *out = nullptr;
    {
        std::lock_guard<std::mutex> hold(p->sitesLock);
        RET(p->hSiteLikes.ensure(sizeof(double) * std::max(p->nChar, 1)));
        RET(p->hSiteLikes.device(&out));
    }
    if (p->nChar <= 0) return P4G_OK;
    // a block per SM with an even share of the sites, since every block loads
    // the words in host memory: 400,000 sites took 433 us an evaluation with eight
    // blocks of 256 threads per SM, 411 with one of 1,024, 409 without the test
    const int nSM = ctx().nSM;
    const int threads = std::min(1024, ((p->nChar + nSM - 1) / nSM + 31) / 32 * 32);
    k_siteLikes<<<std::min((p->nChar + threads - 1) / threads, nSM), threads, 0, s>>>(
        dLnl, p->dSeqPos.as<int>(), p->nChar, (double *)out, partLnl, nParts, status);
    P4G_CUDA(cudaGetLastError());
    return P4G_OK;
}

}  // namespace p4g
