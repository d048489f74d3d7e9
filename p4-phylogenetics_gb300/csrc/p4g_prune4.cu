// Fused FP32 pruning of 4-state (DNA) parts: k_prune's method (p4g_prune.cu:
// the same host-built program, the same operations on every value, so
// per-pattern results equal the CPU mirror's bit for bit) with the
// categories of a pattern held in pairs and every product and sum formed two
// categories at a time.
//
// What bounds it: instruction issue and the latency of each node's chain of
// instructions (an alignment of 74 k patterns is 15 warps an SM).  A scalar
// kernel that took the program op by op issued 15.8 k warp instructions for
// 32 patterns of 64 taxa, 5.2 k of them the FMA pipe's own work, 62 us; this
// one 9.1 k and 49 us (no clade tables, 256 threads, caches as left by the
// evaluation before):
//   - the values of categories 2p and 2p+1 sit in one 64-bit register pair and
//     fma/mul.rn.f32x2 works on both (each half rounded as the scalar
//     instruction rounds); the P decks of 4-state parts are stored as 16-byte
//     words of two columns of a pair, [node][column half][pair][row][4], so
//     that one load gives two operand pairs and nothing is packed or moved;
//     the two pairs' words of a row lie 64 bytes apart, so that lanes that
//     hold different pairs, or codes, read different banks;
//   - the program is decoded into one entry per internal node
//     (decodeProgram4): the rescale and transform of the node before, then the
//     product its parent starts or goes on with; the three kinds that binary
//     trees are made of are straight code from the transform's registers into
//     the values (op by op the compiler moved all 16 values at each merge:
//     26 moves an entry); the next entry and its tip codes are loaded while
//     the current one runs, and REDUX leaves an entry in uniform registers,
//     which its branches and addresses then come from;
//   - the rescale test's maximum takes three operands an instruction, and the
//     usual rescale is one product.
// An odd category count's last category is alone: scalar products, its decks and
// table entries float4 rows behind the pairs'.  (Repeated in a pair's upper half it
// took two of the FMA pipe's cycles for one value's work and shared memory for
// two: evaluations of 64 taxa x 115 k patterns x 5 categories 104 us, of 500 taxa
// x 3 k x 3, whose decks no longer fitted, 490; alone 93 and 186.)
#include <cuda_runtime.h>
#include <limits.h>
#include <algorithm>
#include "p4g_internal.h"
#include "p4g_prune_common.cuh"

namespace p4g {

namespace {

typedef unsigned long long f2;   // two FP32 values: category 2p low, 2p+1 high

__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 pack2(float lo, float hi)
{
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float lo2(f2 v)
{
    return __uint_as_float((unsigned)v);
}
__device__ __forceinline__ float hi2(f2 v)
{
    return __uint_as_float((unsigned)(v >> 32));
}
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

template <bool S>
__device__ __forceinline__ ulonglong2 ldPair2(const float *p)
{
    if (S) return *(const ulonglong2 *)p;
    return __ldg((const ulonglong2 *)p);
}

// Decoded program entries.  x: flags, push slot, transform deck; y: decks of the
// product's tip (or its stack slot) and of the start's tip; z: their code rows.
// In this order: F4_XFORM rescales the values and takes them through
// the transform, F4_PUSH stacks them, F4_START replaces them by a tip's factor,
// F4_CLADE by a clade table's entry, then they are multiplied by a tip's
// factor (F4_TIP), a stack slot (F4_SLOT) or nothing.
// F4_MAIN marks the three kinds binary trees are made of: a transform, then a
// tip, a stack slot, or a push and a cherry.
constexpr int F4_XFORM = 1, F4_MAIN = 2, F4_START = 4, F4_CLADE = 8, F4_TIP = 16, F4_SLOT = 32, F4_PUSH = 64;
constexpr int SLOT4_SHIFT = 7, DECK4_SHIFT = 16;   // x: 9 bits of push slot, 16 of transform deck

struct Layout4 {
    int offProg, offDecks, offCodes, offIdx, offPi, offOnes, offSlots, offRed, total;
};

__host__ __device__ inline int align16(int x) { return (x + 15) & ~15; }

// tile = patterns per block pass; every region is sized per tile
__host__ __device__ inline Layout4 layout4(int nProg, int nDecks, int nRows, int nc, int tp, int tile, int nSlots,
                                           bool sdeck, int nClade)
{
    Layout4 L;
    int o = 0;
    L.offProg = o;
    o += nProg * 16;
    L.offDecks = o;
    if (sdeck) o += nDecks * deckFloats(4, nc) * 4;
    L.offCodes = o;
    o += align16(nRows * tile);
    L.offIdx = o;
    o += nClade * tile * 4;
    L.offPi = o;
    o += 16;
    L.offOnes = o;   // what a gap multiplies by, laid out as a deck's words of one row
    if (sdeck) o += deckFloats(4, nc) * 4;
    L.offSlots = o;
    o += nSlots * nc * 16 * tile;
    L.offRed = o;
    o += (tp / 32) * 8 + 16;
    L.total = o;
    return L;
}

// The program, decoded by one warp into entries (above), and their number to
// *count; entry [count] is a harmless one that the loop's prefetch reads.  A
// factor takes along the OP_SCALE_XFORM and OP_PUSH before it (20-state
// parts' cherry lookups, OP_CHERRY + OP_ARG, may stand between), a TIPSET the
// TIPMUL after it; the program's last op is the caller's.  Every program
// starts with a TIPSET or a clade read and ends with its last node's rescale,
// so there are fewer entries than ops.  deckOf / rowOf (nullable): staged
// deck of a node, staged row of a taxon.
__device__ void decodeProgram4(const PruneJob &J, int4 *out, int *count, const int *deckOf, const int *rowOf)
{
    constexpr int CH = 8;   // chunks of 32 ops loaded at once
    constexpr int NOP = 15;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int n = J.nProg;
    int done = 0, tail = NOP;   // tail: the ops of the chunk before, one per lane
    for (int base = 0; base < n; base += 32 * CH) {
        int r[CH + 1];
#pragma unroll
        for (int c = 0; c <= CH; c++) {   // one chunk more, for the look-ahead
            const int i = base + 32 * c + lane;
            r[c] = i < n ? __ldg(J.prog + i) : NOP;
        }
#pragma unroll
        for (int c = 0; c < CH; c++) {
            const int ins = r[c], op = ins & 15;
            int back[5];   // the ops 1 .. 4 before this lane's
#pragma unroll
            for (int k = 1; k <= 4; k++) {
                const int here = __shfl_up_sync(FULL, ins, k), past = __shfl_sync(FULL, tail, (lane + 32 - k) & 31);
                back[k] = lane < k ? past : here;
            }
            int nx = __shfl_down_sync(FULL, ins, 1);
            const int nf = __shfl_sync(FULL, r[c + 1], 0);
            if (lane == 31) nx = nf;
            const bool tipset = op == OP_TIPSET;
            const bool pair = tipset && (nx & 15) == OP_TIPMUL;
            const bool inPair = op == OP_TIPMUL && (back[1] & 15) == OP_TIPSET;
            const bool lone = op == OP_SCALE_XFORM && (back[1] & 15) == OP_SCALE_XFORM;
            const bool emit = tipset || (op == OP_TIPMUL && !inPair) || op == OP_MULSLOT || op == OP_CLADE || lone ||
                              (op == OP_SCALE && (back[1] & 15) == OP_SCALE_XFORM);
            const unsigned m = __ballot_sync(FULL, emit);
            if (emit) {
                int k = (back[1] & 15) == OP_ARG ? 3 : 1;   // past a cherry lookup
                const int push = k == 3 ? back[3] : back[1];
                const bool pushed = (push & 15) == OP_PUSH;
                const int close = !pushed ? push : (k == 3 ? back[4] : back[2]);
                const int a = (ins >> 4) & 0x3fff, b = ins >> 18;
                int4 d = make_int4(0, 0, 0, 0);
                if (tipset || op == OP_TIPMUL) {
                    const int dk = deckOf ? __ldg(deckOf + a) : a, rw = rowOf ? __ldg(rowOf + b) : b;
                    d.x = tipset ? F4_START : F4_TIP;
                    d.y = tipset ? dk << 16 : dk;
                    d.z = tipset ? rw << 16 : rw;
                    if (pair) {
                        const int a2 = (nx >> 4) & 0x3fff, b2 = nx >> 18;
                        d.x |= F4_TIP;
                        d.y |= deckOf ? __ldg(deckOf + a2) : a2;
                        d.z |= rowOf ? __ldg(rowOf + b2) : b2;
                    }
                } else if (op == OP_MULSLOT) {
                    d.x = F4_SLOT;
                    d.y = a;
                } else if (op == OP_CLADE) {
                    d.x = F4_CLADE;   // clades are numbered in the order they are read
                }
                if (pushed) d.x |= F4_PUSH | (((push >> 4) & 0x1ff) << SLOT4_SHIFT);
                if ((close & 15) == OP_SCALE_XFORM) {
                    const int v = (close >> 4) & 0x3fff;
                    d.x |= F4_XFORM | ((deckOf ? __ldg(deckOf + v) : v) << DECK4_SHIFT);
                }
                const int w = d.x & (F4_XFORM | F4_START | F4_CLADE | F4_TIP | F4_SLOT | F4_PUSH);
                if (w == (F4_XFORM | F4_TIP) || w == (F4_XFORM | F4_SLOT) ||
                    w == (F4_XFORM | F4_PUSH | F4_START | F4_TIP))
                    d.x |= F4_MAIN;
                out[done + __popc(m & ((1u << lane) - 1u))] = d;
            }
            done += __popc(m);
            tail = ins;
        }
    }
    if (lane == 0) {
        out[done] = make_int4(0, 0, 0, 0);
        *count = done;
    }
}

// One block walks tiles blockIdx.x, +gridDim.x, ...; the job's program and
// P decks are staged once per job change, the tip codes once per tile.
// A pattern is handled by G adjacent lanes, lane g holding the category pairs
// [g * CPL, (g + 1) * CPL), or where G does not divide them (shapes 14 and 15) the
// last CPL, a pair then being formed by two lanes; a thread works on PPT adjacent
// patterns, whose transforms share every P load.
// MB: resident blocks per SM the registers are held to (0: free).
template <int NC, int TP, int PPT, bool SDECK, int G, int MB>
__global__ void __launch_bounds__(TP, MB)
k_prune4(const PruneJob *__restrict__ jobs, const BlockDesc *__restrict__ blocks, int nTiles,
         const int *__restrict__ nTilesDev, int early)
{
    constexpr int CPN = NC / 2;          // category pairs
    constexpr bool ODD = NC % 2;         // and a category alone
    static_assert(CPN >= G || G == 1, "every lane has a pair of its own");
    static_assert(!ODD || G == 1, "an odd category count is not split");
    constexpr int CPL = (CPN + G - 1) / G;   // pairs per lane
    constexpr bool SHARED_PAIR = CPL * G != CPN;
    constexpr int NV = CPL * 4;          // pair values per thread and pattern
    constexpr int CL = 2 * CPL + ODD;    // categories of a lane
    constexpr int TPP = TP / G;
    constexpr int TILE = TPP * PPT;
    constexpr int DECK = NC * 16;        // floats of one node's deck: the pairs', then the last category's rows
    constexpr int ALONE = CPN * 32;      // where those begin
    constexpr int NQ = CL;               // a lane's 16-byte words of one pattern in a stack slot
    struct Vals {                        // a thread's values of one pattern
        f2 p[NV ? NV : 1];
        float s[ODD ? 4 : 1];            // the category alone
    };
    // the wait on the previous kernel comes before the first read of what it
    // may have written (PDL_EARLY_* bits: what it does not write), so the
    // staging below can run while that kernel drains
    bool waited = false;
    auto waitPrev = [&]() {
        if (!waited) {
            pdlEnter();
            waited = true;
        }
    };
    if (!(early & PDL_EARLY_JOBS)) waitPrev();
    extern __shared__ __align__(16) unsigned char smem[];
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));   // read once
    const int q = tid / G;               // thread's pattern group in the tile
    const int g = tid % G;               // lane in the group
    const int cp0 = SHARED_PAIR ? min(g * CPL, CPN - CPL) : g * CPL;   // first category pair of this lane
    // the lane's word i of its k-th pattern in a stack slot; lanes that form the same
    // pair store the same words and read only what they stored
    auto slotWord = [&](int k, int i) -> int {
        return SHARED_PAIR ? (k * NC + 2 * cp0 + i) * TPP + q : (k * NQ + i) * TP + tid;
    };
    __shared__ int sLast, sCount;
    int curJob = -1;
    Layout4 L;
    int4 *sProg = nullptr;
    float *sDecks = nullptr;
    uint8_t *sCodes = nullptr;
    uint32_t *sIdx = nullptr;
    float *sPi = nullptr;
    float4 *sSlots = nullptr;
    double *sRed = nullptr;

    if (nTilesDev) nTiles = min(nTiles, *nTilesDev);
    for (int tile = blockIdx.x; tile < nTiles; tile += gridDim.x) {
        const BlockDesc bd = blocks[tile];
        const PruneJob &J = jobs[bd.job];
        const int nTax = J.nTax;
        __syncthreads();   // previous tile is done with the shared buffers
        const bool fresh = bd.job != curJob;
        if (fresh) {
            L = layout4(J.nProg, J.deckMap ? J.nDeck : J.nNodes, J.rowMap ? J.nRow : nTax, NC, TP, TILE, J.nSlots,
                        SDECK, J.nClade);
            sProg = (int4 *)(smem + L.offProg);
            sDecks = (float *)(smem + L.offDecks);
            sCodes = smem + L.offCodes;
            sIdx = (uint32_t *)(smem + L.offIdx);
            sPi = (float *)(smem + L.offPi);
            sSlots = (float4 *)(smem + L.offSlots);
            sRed = (double *)(smem + L.offRed);
            curJob = bd.job;
        }
        {
            constexpr int V = TILE / 16;   // 16-byte chunks per taxon row
            const int *tax = J.rowMap ? J.rowMap + nTax : nullptr;
            const int total = (tax ? J.nRow : nTax) * V;
            for (int i = tid; i < total; i += TP) {
                const int row = i / V, c = i % V;
                cpAsync16(sCodes + row * TILE + 16 * c,
                          J.codes + (size_t)(tax ? __ldg(tax + row) : row) * J.nPatPad + bd.p0 + 16 * c);
            }
            const int totalIdx = J.nClade * (TILE / 4);   // table entries of each clade, this tile
            for (int i = tid; i < totalIdx; i += TP) {
                const int row = i / (TILE / 4), c = i % (TILE / 4);
                cpAsync16(sIdx + row * TILE + 4 * c, J.cladeIdx + (size_t)row * J.nPatPad + bd.p0 + 4 * c);
            }
        }
        if (fresh) {
            if (SDECK) {
                if (!(early & PDL_EARLY_DECKS)) waitPrev();
                constexpr int PER = DECK / 4;   // 16-byte words of one node's deck
                const int *node = J.deckMap ? J.deckMap + J.nNodes : nullptr;
                const int n4 = (node ? J.nDeck : J.nNodes) * PER;
                for (int i = tid; i < n4; i += TP) {
                    const int k = i / PER;
                    cpAsync16(sDecks + 4 * i,
                              J.decks + (size_t)(node ? __ldg(node + k) : k) * DECK + 4 * (i - k * PER));
                }
            }
            cpAsyncCommit();
            if (SDECK)
                for (int i = tid; i < DECK; i += TP) ((float *)(smem + L.offOnes))[i] = 1.f;
            if (tid < 32)
                decodeProgram4(J, sProg, &sCount, SDECK ? J.deckMap : nullptr, J.rowMap);
            if (tid < 4 && !J.cladeOut) sPi[tid] = (float)J.rootComp[tid];   // clade jobs have no root
        }
        int pp[PPT];
        bool valid[PPT];
        double cnt[PPT];
        uint32_t im[PPT];
#pragma unroll
        for (int k = 0; k < PPT; k++) {
            pp[k] = bd.p0 + q * PPT + k;
            valid[k] = pp[k] < J.nPat;
            const int pc = valid[k] ? pp[k] : J.nPat - 1;
            cnt[k] = J.counts[pc];
            im[k] = (J.pInvar != 0.0) ? J.invMask[pc] : 0u;
        }
        cpAsyncWaitAll();
        __syncthreads();
        waitPrev();   // the tables (and decks read through L1) of earlier kernels

        const float *decks = (SDECK ? sDecks : J.decks) + cp0 * 16;
        auto wordOf = [](int i) constexpr -> int { return (i & 1) * (CPN * 64) + (i >> 1) * 64; };
        const uint8_t *myCodes = sCodes + q * PPT;
        // the category alone: d = a * v, d = v
        auto mulAlone = [](float (&d)[ODD ? 4 : 1], const float (&a)[ODD ? 4 : 1], const float4 v) {
            if constexpr (ODD) {
                d[0] = __fmul_rn(a[0], v.x);
                d[1] = __fmul_rn(a[1], v.y);
                d[2] = __fmul_rn(a[2], v.z);
                d[3] = __fmul_rn(a[3], v.w);
            }
        };
        auto setAlone = [](float (&d)[ODD ? 4 : 1], const float4 v) {
            if constexpr (ODD) {
                d[0] = v.x;
                d[1] = v.y;
                d[2] = v.z;
                d[3] = v.w;
            }
        };
        Vals acc[PPT];
        int E[PPT];
#pragma unroll
        for (int k = 0; k < PPT; k++) {
            E[k] = 0;
#pragma unroll
            for (int i = 0; i < NV; i++) acc[k].p[i] = pack2(1.f, 1.f);
            if (ODD) setAlone(acc[k].s, make_float4(1.f, 1.f, 1.f, 1.f));
        }
        auto codesAt = [&](int row) -> int {   // the thread's codes in one row
            if (PPT == 4) return *(const int *)(myCodes + row * TILE);
            if (PPT == 2) return *(const uint16_t *)(myCodes + row * TILE);
            return myCodes[row * TILE];
        };
        // clade k's table entries are loaded one clade read ahead (clades are
        // numbered in read order), so the loads are in flight while the
        // entries before it run.  An entry index at or past the table's end
        // (which a stale or unfilled index row could hold) is not read: entry 0
        // is read instead and oob set.
        Vals pre[PPT];
        int preE[PPT];
        int oob = 0;
        auto cladeFetch = [&](int k0) {
#pragma unroll
            for (int k = 0; k < PPT; k++) {
                uint32_t u = sIdx[k0 * TILE + q * PPT + k];
                if (u >= (uint32_t)J.nCladeEntries) {
                    oob = 1;
                    u = 0;
                }
                const float *src = J.cladeTab + (size_t)u * (NC * 4) + cp0 * 8;
#pragma unroll
                for (int i = 0; i < NV / 2; i++) {
                    const ulonglong2 w = __ldg((const ulonglong2 *)src + i);
                    pre[k].p[2 * i] = w.x;
                    pre[k].p[2 * i + 1] = w.y;
                }
                if (ODD) setAlone(pre[k].s, __ldg((const float4 *)(src + CPN * 8)));
                preE[k] = __ldg(J.cladeExp + u);
            }
        };
        if (J.nClade > 0) cladeFetch(0);

        // Shared-memory offset of the words a tip's code selects in the deck at
        // index dk (word i: pair i >> 1, columns' half i & 1); a gap or an
        // ambiguity code reads ones.
        const int laneWords = cp0 * 64;
        auto tipOff = [&](int dk, int c) -> int {
            return c < 4 ? L.offDecks + dk * (DECK * 4) + laneWords + c * 16 : L.offOnes;
        };
        // the category alone: the row the code selects
        auto tipAlone = [&](int dk, int c, int off) -> float4 {
            if (SDECK) return *(const float4 *)(smem + off + ALONE * 4);
            const float4 v = __ldg((const float4 *)(J.decks + (size_t)dk * DECK + ALONE + (c < 4 ? c : 0) * 4));
            return c < 4 ? v : make_float4(1.f, 1.f, 1.f, 1.f);
        };
        // The pairs' words for decks read through L1.
        auto tipGlobal = [&](int dk, int c, int i) -> ulonglong2 {
            ulonglong2 v = __ldg((const ulonglong2 *)(J.decks + (size_t)dk * DECK + cp0 * 16 + (c < 4 ? c : 0) * 4) + wordOf(i) / 16);
            if (c >= 4) v.x = v.y = pack2(1.f, 1.f);
            return v;
        };
        auto codeOf = [](int code, int k) -> int { return PPT > 1 ? (code >> (8 * k)) & 0xff : code; };
        // the factor of a partial ambiguity code (sums over its states)
        auto equate = [&](Vals (&x)[PPT], int dk, int code) {
            const int node = (SDECK && J.deckMap) ? __ldg(J.deckMap + J.nNodes + dk) : dk;
#pragma unroll
            for (int k = 0; k < PPT; k++) {
                const int c = codeOf(code, k);
                if (c <= 4) continue;
                const float *eq = J.eqTab + (((size_t)node * J.nPartial + (c - 5)) * NC) * 4;
#pragma unroll
                for (int cp = 0; cp < CPL; cp++) {
                    const int ca = 2 * (cp0 + cp);
                    const float4 a = __ldg((const float4 *)eq + ca), b = __ldg((const float4 *)eq + ca + 1);
                    f2 *v = x[k].p + 4 * cp;
                    v[0] = mul2(v[0], pack2(a.x, b.x));
                    v[1] = mul2(v[1], pack2(a.y, b.y));
                    v[2] = mul2(v[2], pack2(a.z, b.z));
                    v[3] = mul2(v[3], pack2(a.w, b.w));
                }
                if (ODD) mulAlone(x[k].s, x[k].s, __ldg((const float4 *)eq + NC - 1));
            }
        };
        auto partialCode = [&](int code) -> bool {   // any of the thread's codes a partial ambiguity
            bool any = false;
#pragma unroll
            for (int k = 0; k < PPT; k++) any |= codeOf(code, k) > 4;
            return any;
        };
        auto times = [&](Vals &v, float f) {
#pragma unroll
            for (int i = 0; i < NV; i++) v.p[i] = mul2(v.p[i], pack2(f, f));
            if (ODD) mulAlone(v.s, v.s, make_float4(f, f, f, f));
        };
        auto rescale = [&]() {
#pragma unroll
            for (int k = 0; k < PPT; k++) {
                float mx = 0.f;
#pragma unroll
                for (int i = 0; i < NV; i++) mx = max3(mx, lo2(acc[k].p[i]), hi2(acc[k].p[i]));
                if constexpr (ODD) mx = max3(max3(mx, acc[k].s[0], acc[k].s[1]), acc[k].s[2], acc[k].s[3]);
#pragma unroll
                for (int o = 1; o < G; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                if (mx < 0x1p-32f && mx > 0.0f) {
                    const int ex = (int)(__float_as_uint(mx) >> 23);   // 2^(ex - 126) > mx >= half of it
                    if (ex >= 26) {   // one factor 2^k, k = 126 - ex <= 100
                        const float f = __uint_as_float((unsigned)(253 - ex) << 23);
                        E[k] += 126 - ex;
                        times(acc[k], f);
                    } else {
                        int e2;
                        (void)frexp32(mx, &e2);
                        int x = -e2;
                        E[k] += x;
                        while (x > 0) {
                            const int step = x > 100 ? 100 : x;
                            times(acc[k], __uint_as_float((unsigned)(127 + step) << 23));
                            x -= step;
                        }
                    }
                }
            }
        };
        auto transform = [&](int deck, Vals (&out)[PPT]) {
            const float *P = decks + deck * DECK;
#pragma unroll
            for (int cp = 0; cp < CPL; cp++)
#pragma unroll
                for (int s = 0; s < 4; s++) {   // row s: columns 0 1 and 2 3
                    const ulonglong2 a = ldPair2<SDECK>(P + wordOf(2 * cp) / 4 + s * 4),
                                     b = ldPair2<SDECK>(P + wordOf(2 * cp + 1) / 4 + s * 4);
#pragma unroll
                    for (int k = 0; k < PPT; k++) {
                        const f2 *v = acc[k].p + 4 * cp;
                        f2 t = mul2(a.x, v[0]);
                        t = fma2(a.y, v[1], t);
                        t = fma2(b.x, v[2], t);
                        out[k].p[4 * cp + s] = fma2(b.y, v[3], t);
                    }
                }
            if constexpr (ODD) {
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    const float4 *row = (const float4 *)(P + ALONE) + s;
                    const float4 a = SDECK ? *row : __ldg(row);
#pragma unroll
                    for (int k = 0; k < PPT; k++) {
                        const float *v = acc[k].s;
                        float t = __fmul_rn(a.x, v[0]);
                        t = __fmaf_rn(a.y, v[1], t);
                        t = __fmaf_rn(a.z, v[2], t);
                        out[k].s[s] = __fmaf_rn(a.w, v[3], t);
                    }
                }
            }
        };

        // acc = src * the factor of tip deck dk at the thread's codes
        auto mulTip = [&](const Vals (&src)[PPT], int dk, int code) {
#pragma unroll
            for (int k = 0; k < PPT; k++) {
                const int c = codeOf(code, k), off = SDECK ? tipOff(dk, c) : 0;
#pragma unroll
                for (int i = 0; i < NV / 2; i++) {
                    const ulonglong2 v = SDECK ? *(const ulonglong2 *)(smem + off + wordOf(i)) : tipGlobal(dk, c, i);
                    acc[k].p[2 * i] = mul2(src[k].p[2 * i], v.x);
                    acc[k].p[2 * i + 1] = mul2(src[k].p[2 * i + 1], v.y);
                }
                if (ODD) mulAlone(acc[k].s, src[k].s, tipAlone(dk, c, off));
            }
            if (partialCode(code)) equate(acc, dk, code);
        };
        auto setTip = [&](int dk, int code) {
#pragma unroll
            for (int k = 0; k < PPT; k++) {
                const int c = codeOf(code, k), off = SDECK ? tipOff(dk, c) : 0;
#pragma unroll
                for (int i = 0; i < NV / 2; i++) {
                    const ulonglong2 v = SDECK ? *(const ulonglong2 *)(smem + off + wordOf(i)) : tipGlobal(dk, c, i);
                    acc[k].p[2 * i] = v.x;
                    acc[k].p[2 * i + 1] = v.y;
                }
                if (ODD) setAlone(acc[k].s, tipAlone(dk, c, off));
            }
            if (partialCode(code)) equate(acc, dk, code);
        };
        auto mulSlot = [&](const Vals (&src)[PPT], int n) {
            const float4 *sl = sSlots + n * (NC * TILE);
#pragma unroll
            for (int k = 0; k < PPT; k++) {
#pragma unroll
                for (int i = 0; i < NV / 2; i++) {
                    const ulonglong2 v = *(const ulonglong2 *)(sl + slotWord(k, i));
                    acc[k].p[2 * i] = mul2(src[k].p[2 * i], v.x);
                    acc[k].p[2 * i + 1] = mul2(src[k].p[2 * i + 1], v.y);
                }
                if (ODD) mulAlone(acc[k].s, src[k].s, sl[slotWord(k, NQ - 1)]);
            }
        };
        auto pushSlot = [&](const Vals (&src)[PPT], int n) {
            float4 *sl = sSlots + n * (NC * TILE);
#pragma unroll
            for (int k = 0; k < PPT; k++) {
#pragma unroll
                for (int i = 0; i < NV / 2; i++)
                    *(ulonglong2 *)(sl + slotWord(k, i)) = make_ulonglong2(src[k].p[2 * i], src[k].p[2 * i + 1]);
                if constexpr (ODD)
                    sl[slotWord(k, NQ - 1)] = make_float4(src[k].s[0], src[k].s[1], src[k].s[2], src[k].s[3]);
            }
        };

        const int nEntries = sCount;
        // an entry, known to be the same in every lane (REDUX leaves it in a
        // uniform register): its branches and addresses cost the warp nothing
        auto entryAt = [&](int ip) -> int3 {
            const int4 d = sProg[ip];
            return make_int3((int)__reduce_or_sync(0xffffffffu, (unsigned)d.x),
                             (int)__reduce_or_sync(0xffffffffu, (unsigned)d.y),
                             (int)__reduce_or_sync(0xffffffffu, (unsigned)d.z));
        };
        int nextClade = 0;
        int3 I = entryAt(0);
        int code = codesAt(I.z & 0xffff), codeS = codesAt((unsigned)I.z >> 16);
        for (int ip = 0; ip < nEntries; ip++) {
            const int3 In = entryAt(ip + 1);
            const int what = I.x & 63, dk = I.y & 0xffff;
            if (what & F4_MAIN) {   // the entries of a binary tree
                Vals x[PPT];
                rescale();
                transform((unsigned)I.x >> DECK4_SHIFT, x);
                if (what & F4_TIP) {
                    if (what & F4_START) {
                        pushSlot(x, (I.x >> SLOT4_SHIFT) & 0x1ff);
                        setTip((unsigned)I.y >> 16, codeS);
                        mulTip(acc, dk, code);
                    } else {
                        mulTip(x, dk, code);
                    }
                } else {
                    mulSlot(x, dk);
                }
            } else {
                if (what & F4_XFORM) {
                    Vals x[PPT];
                    rescale();
                    transform((unsigned)I.x >> DECK4_SHIFT, x);
#pragma unroll
                    for (int k = 0; k < PPT; k++) acc[k] = x[k];
                }
                if (I.x & F4_PUSH) pushSlot(acc, (I.x >> SLOT4_SHIFT) & 0x1ff);
                if (what & F4_START) setTip((unsigned)I.y >> 16, codeS);
                if (what & F4_CLADE) {
#pragma unroll
                    for (int k = 0; k < PPT; k++) {
                        acc[k] = pre[k];
                        E[k] += preE[k];
                    }
                    if (++nextClade < J.nClade) cladeFetch(nextClade);
                }
                if (what & F4_TIP) mulTip(acc, dk, code);
                if (what & F4_SLOT) mulSlot(acc, dk);
            }
            code = codesAt(In.z & 0xffff);
            codeS = codesAt((unsigned)In.z >> 16);
            I = In;
        }
        rescale();   // the last node's; a clade's values go through its edge's transform
        if (J.cladeOut) {
            Vals out[PPT];
            transform((__ldg(J.prog + J.nProg - 1) >> 4) & 0x3fff, out);
#pragma unroll
            for (int k = 0; k < PPT; k++) acc[k] = out[k];
        }

        if (J.cladeOut) {   // clade-table job: the transformed product and its exponent
#pragma unroll
            for (int k = 0; k < PPT; k++) {
                if (!valid[k]) continue;
                float *o = J.cladeOut + (size_t)pp[k] * (NC * 4) + cp0 * 8;
#pragma unroll
                for (int i = 0; i < NV / 2; i++)
                    *((ulonglong2 *)o + i) = make_ulonglong2(acc[k].p[2 * i], acc[k].p[2 * i + 1]);
                if constexpr (ODD)
                    *(float4 *)(o + CPN * 8) = make_float4(acc[k].s[0], acc[k].s[1], acc[k].s[2], acc[k].s[3]);
                if (g == 0) J.cladeOutExp[pp[k]] = E[k];
            }
            continue;
        }

        // ---- root reduction: one fmaf chain over (category, state) in
        // category order, carried from lane to lane through the group
        double v = 0.0;
        int bad = 0;
        const int lane = tid & 31;
        const int base = lane & ~(G - 1);
        const int rootRow = (J.rootLeafRow >= 0 && J.rowMap) ? J.rowMap[J.rootLeafRow] : J.rootLeafRow;
        // category c of this lane
        auto val = [&](int k, int c, int s) -> float {
            if (ODD && c == CL - 1) return acc[k].s[ODD ? s : 0];
            const f2 w = acc[k].p[4 * (c >> 1) + s];
            return (c & 1) ? hi2(w) : lo2(w);
        };
#pragma unroll
        for (int k = 0; k < PPT; k++) {
            uint32_t rmask = 15u;
            if (rootRow >= 0) {
                const int code = sCodes[rootRow * TILE + q * PPT + k];
                if (code < 4) rmask = 1u << code;
                else if (code > 4) rmask = J.partialMask[code - 5];
            }
            float like32 = 0.0f;
#pragma unroll
            for (int j = 0; j < G; j++) {
                if (g == j) {
#pragma unroll
                    for (int c = 0; c < CL; c++) {
                        if (SHARED_PAIR && 2 * cp0 + c < 2 * CPL * j) continue;   // the lane before has it
#pragma unroll
                        for (int s = 0; s < 4; s++)
                            if ((rmask >> s) & 1u) like32 = __fmaf_rn(sPi[s], val(k, c, s), like32);
                    }
                }
                if (G > 1 && j < G - 1) {
                    const float nxt = __shfl_sync(0xffffffffu, like32, base + j);
                    if (g == j + 1) like32 = nxt;
                }
            }
            if (G > 1) like32 = __shfl_sync(0xffffffffu, like32, base + G - 1);
            if (J.rootCL && valid[k]) {   // root partials for ancestral-state draws
                float *o = J.rootCL + ((size_t)pp[k] * NC + 2 * cp0) * 4;
#pragma unroll
                for (int c = 0; c < CL; c++)
#pragma unroll
                    for (int s = 0; s < 4; s++) o[4 * c + s] = ((rmask >> s) & 1u) ? val(k, c, s) : 0.0f;
            }
            if (J.catLikes && valid[k]) {   // per-category sums for site rates
#pragma unroll
                for (int c = 0; c < CL; c++) {
                    float sc = 0.0f;
#pragma unroll
                    for (int s = 0; s < 4; s++)
                        if ((rmask >> s) & 1u) sc = __fmaf_rn(sPi[s], val(k, c, s), sc);
                    J.catLikes[(size_t)pp[k] * NC + 2 * cp0 + c] = sc;
                }
            }
            double lnl;
            bool badk;
            if (im[k]) {
                double lt = __dmul_rn(ldexp((double)like32, -E[k]), J.varScale);
                for (int s = 0; s < 4; s++)
                    if ((im[k] >> s) & 1u) lt = __dadd_rn(lt, __dmul_rn(J.rootComp[s], J.pInvar));
                badk = !(lt > 0.0);
                lnl = log(lt);
            } else {
                badk = !(like32 > 0.0f);
                int e;
                const float m = frexp32(like32, &e);
                lnl = (double)logf(m) + (double)(e - E[k]) * LN2 + J.logScale;
            }
            const bool mine = valid[k] && g == 0;
            if (mine && J.likeScaled) {
                J.likeScaled[pp[k]] = like32;
                J.exps[pp[k]] = E[k];
                J.lnl[pp[k]] = lnl;
            }
            if (mine && !badk) v += cnt[k] * lnl;
            bad |= (mine && badk);
        }
        const int anyBad = (__syncthreads_or(bad) ? 1 : 0) | (__syncthreads_or(oob) ? 4 : 0);

        // ---- tile reduction (fixed order) and last-tile-done finish per job
        for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) sRed[tid >> 5] = v;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < TP / 32; w++) s += sRed[w];
            J.partials[bd.blk] = s;
            if (anyBad) atomicOr(J.badFlag, anyBad);
            __threadfence();
            const int t = atomicAdd(J.ticket, 1);
            sLast = (t == J.nBlocks - 1);
        }
        __syncthreads();
        if (sLast && tid < 32) {
            __threadfence();
            double s = 0.0;
            for (int i = tid; i < J.nBlocks; i += 32) s += __ldcg(J.partials + i);
            for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (tid == 0) {
                const int badAny = atomicExch(J.badFlag, 0);
                *J.out = (badAny & 4) ? __longlong_as_double(0x7ff8000000000000LL) : (badAny ? -1.0e99 : s);
                atomicExch(J.ticket, 0);
            }
        }
    }
}

// Tile shapes the autotuner chooses from: threads per block, patterns per
// thread (they share every P load: shared memory's words, not its latency,
// are what large alignments wait for), P decks staged in shared memory (else
// read through L1, which leaves shared memory to the codes and the stack),
// lanes per pattern (the category pairs spread over 2 lanes, for alignments
// of few patterns; counts whose pairs do not divide take one lane and half the
// threads, so that the tile stays tp / g * ppt patterns), resident
// blocks the registers are held to, and the category counts the shape is
// offered for (a divisor, or 3 and 4 alone).
struct Shape4 {
    int tp, ppt;
    bool sdeck;
    int g, mb, div;
    bool only34;
};
// every tile holds 64 to 512 patterns; shape 13, for odd counts, is the smallest
// in shared memory, as shape 8 is for even ones; the last two are for 6 categories
constexpr Shape4 kShapes4[] = {{128, 1, true, 1, 0, 1, false},  {128, 2, true, 1, 0, 1, false},
                               {256, 1, true, 1, 0, 1, false},  {256, 1, false, 1, 0, 1, false},
                               {128, 2, false, 1, 0, 1, false}, {512, 1, false, 1, 0, 1, false},
                               {128, 1, true, 2, 0, 4, false},  {256, 1, false, 2, 0, 2, false},
                               {128, 1, false, 2, 0, 2, false}, {256, 2, true, 2, 0, 4, false},
                               {128, 2, true, 2, 0, 4, false},  {128, 4, true, 2, 0, 1, true},
                               {128, 2, true, 1, 4, 1, true},
                               {128, 1, false, 1, 0, 1, false},
                               {128, 1, false, 2, 0, 6, false}, {256, 1, false, 2, 0, 6, false}};
constexpr int kNumShapes4 = 16, kFirstShapes4 = 13;
constexpr int kSmallOdd4 = 13, kSmallEven4 = 8, kShared4 = 14;
// Shapes 14 and 15 are 8 and 7 with two lanes of two pairs for 6 categories, the
// middle pair formed by both, where those take one lane of three.  They run in
// their place for trees whose decks are more than 3/2 of a block's shared memory
// (from some 450 taxa), of which clade tables leave too many to stage: a
// chain of loads through L1 then bounds every node, and a lane's is a third
// shorter (us an evaluation, one lane and two: 500 taxa x 3,000 sites 442 and 354,
// 900 x 500 918 and 709).  Smaller trees are bound by issue, and the pair formed
// twice costs more than it gives (420 x 2,000 285 and 328, 300 x 3,000 115 and 121,
// 64 x 150,000 105 and 111).
bool sharedPair4(int nCat, int nNodes) { return nCat == 6 && nNodes * deckFloats(4, nCat) * 4 > PRUNE_SMEM_MAX / 2 * 3; }

// Where a caller may ask for a shape: (threads, tile, decks staged) as the
// numbers were first given out, 16 floats a deck and category.  The forms above
// hold more for some of them (a row of ones, decks staged where they were not); a
// tree that the first form fits and today's does not runs the smallest shape.
// (Refused instead, shapes 6 and 10 were lost from 500
// taxa on and a tree of 800 taxa and one category could not be evaluated.)
struct First4 {
    int tp, tile;
    bool sdeck;
};
constexpr First4 kFirst4[kFirstShapes4] = {{128, 128, true},  {128, 256, true},  {256, 256, true}, {256, 256, false},
                                         {128, 256, false}, {512, 512, false}, {256, 64, false}, {256, 128, false},
                                         {128, 64, false},  {256, 64, true},   {512, 128, false}, {256, 256, true},
                                         {128, 256, true}};

constexpr int lanes4(int nCat, int shape)
{
    const int g = kShapes4[shape].g;
    return (nCat % 2 == 0 && nCat / 2 % g == 0) || shape >= kShared4 ? g : 1;
}
constexpr int threads4(int nCat, int shape) { return kShapes4[shape].tp / kShapes4[shape].g * lanes4(nCat, shape); }

template <int NC, int SH>
int launchShape4(const PruneJob *dJobs, const BlockDesc *dBlocks, int nTiles, int smemBytes, cudaStream_t s,
                 const int *nTilesDev, int early)
{
    constexpr Shape4 S = kShapes4[SH];
    constexpr int TP = threads4(NC, SH);
    auto k = k_prune4<NC, TP, S.ppt, S.sdeck, lanes4(NC, SH), S.mb>;
    static int configured = 0;
    static int perSM = 0, perSMsmem = -1;
    if (smemBytes > 48 * 1024 && configured < smemBytes) {
        P4G_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes));
        configured = smemBytes;
    }
    if (perSMsmem != smemBytes) {
        P4G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k, TP, smemBytes));
        perSMsmem = smemBytes;
    }
    if (perSM < 1) return setError(P4G_EUNSUPPORTED, "pruning kernel does not fit on an SM (%d B smem)", smemBytes);
    const int grid = std::min(nTiles, perSM * ctx().nSM);
    P4G_CUDA(launchPdl(k, dim3(grid), dim3(TP), smemBytes, s, dJobs, dBlocks, nTiles, nTilesDev, early));
    return P4G_OK;
}

template <int NC>
int launchCat4(const PruneJob *dJobs, const BlockDesc *dBlocks, int nTiles, int smemBytes, int shape, cudaStream_t s,
               const int *nTilesDev, int early)
{
    switch (shape) {
#define P4G_SH(N) \
    case N: return launchShape4<NC, N>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early);
        P4G_SH(0) P4G_SH(1) P4G_SH(2) P4G_SH(3) P4G_SH(4) P4G_SH(5)
    case 6: if constexpr (NC % 4 == 0) return launchShape4<NC, 6>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case 7: if constexpr (NC % 2 == 0) return launchShape4<NC, 7>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case 8: if constexpr (NC % 2 == 0) return launchShape4<NC, 8>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case 9: if constexpr (NC % 4 == 0) return launchShape4<NC, 9>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case 10: if constexpr (NC % 4 == 0) return launchShape4<NC, 10>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case 11: if constexpr (NC == 3 || NC == 4) return launchShape4<NC, 11>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case 12: if constexpr (NC == 3 || NC == 4) return launchShape4<NC, 12>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case kShared4: if constexpr (NC == 6) return launchShape4<NC, kShared4>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case kShared4 + 1: if constexpr (NC == 6) return launchShape4<NC, kShared4 + 1>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
    case kSmallOdd4: if constexpr (NC % 2 == 1) return launchShape4<NC, kSmallOdd4>(dJobs, dBlocks, nTiles, smemBytes, s, nTilesDev, early); break;
#undef P4G_SH
    default: break;
    }
    return setError(P4G_EUNSUPPORTED, "no fused pruning kernel for dim=4 nCat=%d shape %d", NC, shape);
}

}  // namespace

int prune4NumShapes() { return kNumShapes4; }

int prune4ShapeValid(int nCat, int shape)
{
    if (shape == kSmallOdd4) return nCat % 2;
    if (shape >= kShared4 && shape < kNumShapes4) return nCat == 6;
    if (shape < 0 || shape >= kNumShapes4) return 0;
    if (kShapes4[shape].only34) return nCat == 3 || nCat == 4;
    return nCat % kShapes4[shape].div == 0;
}

int prune4KernelExists(int nCat, int shape)
{
    return prune4ShapeValid(nCat, shape) && ((nCat >= 1 && nCat <= 6) || nCat == 8);
}

int prune4Tile(int nCat, int shape) { return threads4(nCat, shape) / lanes4(nCat, shape) * kShapes4[shape].ppt; }
int prune4ShapeTimed(int nCat, int shape, int nNodes)
{
    if (!prune4ShapeValid(nCat, shape) || shape == kSmallOdd4) return 0;
    const bool two = shape >= kShared4, one = shape == 7 || shape == 8;
    return nCat != 6 || !(two || one) || two == sharedPair4(nCat, nNodes);
}

int prune4Smallest(int nCat, int nNodes)
{
    return nCat % 2 ? kSmallOdd4 : sharedPair4(nCat, nNodes) ? kShared4 : kSmallEven4;
}

// Clade tables' first shape: the combinations are few, so lane groups of 2 split the
// categories and the tables spread over more blocks; P decks are read through L1 (a
// clade touches few of them).
int prune4CladeShape(int nCat, int nNodes) { return nCat % 2 ? 3 : prune4Smallest(nCat, nNodes); }

int prune4SmemBytes(int nCat, int nProg, int nDecks, int nRows, int nSlots, int shape, int nClade)
{
    const Shape4 &S = kShapes4[shape];
    return layout4(nProg, nDecks, nRows, nCat, threads4(nCat, shape), prune4Tile(nCat, shape), nSlots, S.sdeck, nClade).total;
}

int prune4FirstBytes(int nCat, int nProg, int nDecks, int nRows, int nSlots, int shape, int nClade)
{
    if (shape >= kFirstShapes4) return INT_MAX;
    const First4 &F = kFirst4[shape];
    return layout4(nProg, 0, nRows, nCat, F.tp, F.tile, nSlots, false, nClade).total + (F.sdeck ? nDecks * nCat * 64 : 0);
}

int launchPrune4(const PruneJob *dJobs, const BlockDesc *dBlocks, int nTiles, int nCat, int smemBytes, int shape,
                 cudaStream_t s, const int *nTilesDev, int early)
{
    switch (nCat) {
#define P4G_C(N) \
    case N: return launchCat4<N>(dJobs, dBlocks, nTiles, smemBytes, shape, s, nTilesDev, early);
        P4G_C(1) P4G_C(2) P4G_C(3) P4G_C(4) P4G_C(5) P4G_C(6) P4G_C(8)
#undef P4G_C
    default: break;
    }
    return setError(P4G_EUNSUPPORTED, "no fused pruning kernel for dim=4 nCat=%d shape %d", nCat, shape);
}

}  // namespace p4g
