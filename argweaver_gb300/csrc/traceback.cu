// K4: stochastic traceback (stochastic_traceback, sample_thread.cpp:522-569;
// sample_hmm_posterior :470-503; sample_hmm_posterior_step :506-519; sample,
// common.h:272-290). Column i draws path[i] from A[j] = fw[i][j] * P(j -> path[i+1]) with the
// uniform u[i]: the first j whose running sum reaches u[i] * sum(A). Two kernels, one block
// per instance:
//   k_traceback_lots  the reference's scan, a CTA drawing or testing many columns at once: FP64,
//                     and FP32 where the decomposed draw's tables do not fit
//   k_traceback_split FP32: the draw decomposed by the structure of the transition, by one warp
//                     with two that bring its tables
//
// The scan by one warp splits the states into 32 contiguous chunks (lane t sums chunk t with
// two accumulators, even and odd states); chunk sums are scanned across lanes and the chunk
// that holds the pick is rescanned.

#include <cuda_runtime.h>

#include "async_copy.cuh"
#include "kernels.h"

namespace awg {

namespace {

template <typename F> struct TTab;
template <> struct TTab<double> {
    const double *tm, *rows, *dprob, *rrow, *crow, *fw;
    __device__ explicit TTab(const BatchDev &d)
        : tm(d.tm), rows(d.gts), dprob(d.determprob), rrow(d.recombrow), crow(d.recoalrow), fw(d.fw64) {}
    // same-node entry: get_time(a, b, c, minage, true)
    __device__ static double same(double v, double) { return v; }
};
template <> struct TTab<float> {
    const float *rstay;  // rows exclude the diagonal's stay term
    const float *tm, *rows, *dprob, *rrow, *crow, *fw;
    __device__ explicit TTab(const BatchDev &d)
        : rstay(d.rstay32), tm(d.tm32), rows(d.t2d32), dprob(d.determprob32),
          rrow(d.recombrow32), crow(d.recoalrow32), fw(d.fw32) {}
    __device__ static float same(float v, float tmab) { return v + tmab; }
};

// A hint that moves the whole 16-byte granules of [p, p + bytes) from HBM into L2.
__device__ __forceinline__ void l2_prefetch(const void *p, size_t bytes) {
    const uintptr_t a = ((uintptr_t)p + 15) & ~(uintptr_t)15, e = ((uintptr_t)p + bytes) & ~(uintptr_t)15;
    if (e > a)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a)) : "memory");
}

// Inclusive lane scan.
template <typename F>
__device__ __forceinline__ F lane_scan(F x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const F v = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += v;
    }
    return x;
}

// Given the chunk sums' inclusive scan, the pick and lane t's chunk [lo, hi): the index
// the running sum first reaches the pick at (sample(), common.h:272-290), rescanning the
// chunk that holds it 32 states at a time.
template <typename F, typename W>
__device__ __forceinline__ int finish_sample(int n, int chunk, F incl, F pick, int lo, int hi,
                                             int lane, W w) {
    F excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 0;
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= pick && hi > lo);
    if (!hit) return n - 1;
    const int src = __ffs(hit) - 1;
    const int slo = imin(src * chunk, n), shi = imin(slo + chunk, n);
    F carry = __shfl_sync(0xffffffffu, excl, src);
    int result = shi - 1;
    for (int b0 = slo; b0 < shi; b0 += 32) {
        const int jj = b0 + lane;
        const F x = lane_scan(jj < shi ? w(jj) : F(0), lane);
        const F run = carry + x;
        const unsigned got = __ballot_sync(0xffffffffu, jj < shi && run >= pick);
        if (got) {
            result = b0 + __ffs(got) - 1;
            break;
        }
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
    return result;
}

// One column on its own: weights w(j), j < n.
template <typename F, typename W>
__device__ int warp_sample(int n, double u, W w) {
    const int lane = threadIdx.x & 31;
    const int chunk = (n + 31) >> 5;
    const int lo = imin(lane * chunk, n), hi = imin(lo + chunk, n);
    F l0 = 0, l1 = 0;
    int j = lo;
    for (; j + 1 < hi; j += 2) {
        l0 += w(j);
        l1 += w(j + 1);
    }
    if (j < hi) l0 += w(j);
    const F incl = lane_scan(l0 + l1, lane);
    const F total = __shfl_sync(0xffffffffu, incl, 31);
    return finish_sample<F>(n, chunk, incl, (F)u * total, lo, hi, lane, w);
}

// G columns under one row, each as warp_sample draws it on its own (fused products), side by side:
// values cg[g][j], weights trans[j], j < n, uniforms ug.
template <typename F, int G>
__device__ void warp_sample_group(int n, const F *const (&cg)[G], const F *trans, const double (&ug)[G], int (&res)[G]) {
    const int lane = threadIdx.x & 31;
    const int chunk = (n + 31) >> 5;
    const int lo = imin(lane * chunk, n), hi = imin(lo + chunk, n);
    // every column's chunk sums under the current row, as warp_sample forms them
    F l0[G], l1[G];
#pragma unroll
    for (int g = 0; g < G; g++) l0[g] = l1[g] = F(0);
    int j = lo;
    for (; j + 1 < hi; j += 2) {
        const F t0 = trans[j], t1 = trans[j + 1];
#pragma unroll
        for (int g = 0; g < G; g++) {
            l0[g] = fma(cg[g][j], t0, l0[g]);
            l1[g] = fma(cg[g][j + 1], t1, l1[g]);
        }
    }
    if (j < hi) {
        const F t0 = trans[j];
#pragma unroll
        for (int g = 0; g < G; g++) l0[g] = fma(cg[g][j], t0, l0[g]);
    }
    F incl[G];
#pragma unroll
    for (int g = 0; g < G; g++) incl[g] = l0[g] + l1[g];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int g = 0; g < G; g++) {
            const F v = __shfl_up_sync(0xffffffffu, incl[g], o);
            if (lane >= o) incl[g] += v;
        }
    }
    // every column's draw, all G interleaved (finish_sample's steps, column-wise)
    F pick[G], carry[G];
    int slo[G], shi[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
        F excl = __shfl_up_sync(0xffffffffu, incl[g], 1);
        if (lane == 0) excl = 0;
        const F total = __shfl_sync(0xffffffffu, incl[g], 31);
        pick[g] = (F)ug[g] * total;
        const unsigned hit = __ballot_sync(0xffffffffu, incl[g] >= pick[g] && hi > lo);
        const int src = hit ? __ffs(hit) - 1 : 0;
        slo[g] = imin(src * chunk, n);
        shi[g] = hit ? imin(slo[g] + chunk, n) : slo[g];  // empty: no rescan
        carry[g] = __shfl_sync(0xffffffffu, excl, src);
        res[g] = hit ? shi[g] - 1 : n - 1;
    }
    unsigned open = 0;  // columns whose pick is not found yet
#pragma unroll
    for (int g = 0; g < G; g++)
        if (shi[g] > slo[g]) open |= 1u << g;
    if (chunk <= 16) {
        // short chunks: lane g rescans column g's chosen chunk in order, one product
        // and one add per state, the G columns side by side (a 32-lane scan per column
        // costs five warp-wide adds however few states the chunk holds: on the FP64
        // path each holds the sub-partition's FP64 pipe for about 64 cycles)
        int mine = 0;
        if (lane < G) {
            F mpick = 0, run = 0;
            int mslo = 0, mshi = 0;
            const F *mc = cg[0];
#pragma unroll
            for (int g = 0; g < G; g++)
                if (lane == g) {
                    mpick = pick[g];
                    run = carry[g];
                    mslo = slo[g];
                    mshi = (open >> g) & 1 ? shi[g] : slo[g];
                    mine = res[g];
                    mc = cg[g];
                }
            for (int jj = mslo; jj < mshi; jj++) {
                run += mc[jj] * trans[jj];
                if (run >= mpick) {
                    mine = jj;
                    break;
                }
            }
        }
#pragma unroll
        for (int g = 0; g < G; g++) res[g] = __shfl_sync(0xffffffffu, mine, g);
        open = 0;
    }
    for (int b = 0; open; b += 32) {
        F x[G];
#pragma unroll
        for (int g = 0; g < G; g++) {
            const int jj = slo[g] + b + lane;
            x[g] = ((open >> g) & 1) && jj < shi[g] ? cg[g][jj] * trans[jj] : F(0);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int g = 0; g < G; g++) {
                const F v = __shfl_up_sync(0xffffffffu, x[g], o);
                if (lane >= o) x[g] += v;
            }
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (!((open >> g) & 1)) continue;
            const int jj = slo[g] + b + lane;
            const unsigned got =
                __ballot_sync(0xffffffffu, jj < shi[g] && carry[g] + x[g] >= pick[g]);
            if (got) {
                res[g] = slo[g] + b + __ffs(got) - 1;
                open &= ~(1u << g);
            } else {
                carry[g] += __shfl_sync(0xffffffffu, x[g], 31);
                if (slo[g] + b + 32 >= shi[g]) open &= ~(1u << g);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// FP32 path: the draw decomposed by the structure of the transition.
//
// Inside a tree P(j -> k) = tm[a_j][b_k] + [node_j = node_k] tm2[a_j][k] (the structured
// step of arghmm_forward_block, sample_thread.cpp:255-290; tm2 >= 0 is the same-branch
// excess, the no-recombination stay included on the diagonal). Column i's weights
// fw[i][j] P(j -> k) thus split into the same-branch part V_y = fw[i][j1 + y] tm2[a_y][k]
// over the m states of k's node, and a background part whose total over the states of
// time bin a is W_a = bins[i][a] tm[a][b_k], bins[i] being the stored column's time-bin
// sums that the forward kernel writes. With t = u (V + W): if t <= V the draw is the first
// y whose running V sum reaches t; else the first bin whose running W sum reaches t - V,
// then the first state of that bin (states of a bin in time-sorted order) whose running
// fw sum reaches the remainder over tm[a][b_k]. This draws from exactly the distribution
// of the reference's scan over all states (sample(), common.h:272-290), mapping the
// uniform to states in another order, with O(T + m) work per column instead of O(S).
// At a tree switch only the sources with a nonzero switch probability into the drawn
// state carry weight (its gather list plus the recombination and recoalescence sources),
// so the switch draw runs over those, in state order.
//
// Speculation: the warp tests up to 32 columns at once for the common case, the draw staying at
// the current state k: four lanes take a column's V and W terms, four columns each, in whatever
// order suits the loads. All terms are >= 0, so a sum in any order is within 64 roundings of the
// one that the draw is defined by (quarters of the states and of the bins in order, then a
// tree), and a column whose pick lies within `margin` of an end of k's interval is decided by
// that one. The first column that leaves k (about one in a thousand inside an external tree, one
// in a few hundred of a cut one) is drawn exactly by the whole warp; the columns after it are
// tested again under the new state.
//
// What bounds it: latencies on one warp's path, a tree of some 28 columns (at 100 leaves) after
// the other, so per tree there is one wait for the forward table: a test reads only the states of
// k's node, straight from L2, and the switch's sources (a lane each) are loaded with the last
// test, for the state that the tree will most likely keep. Everything else is in shared memory
// by then: two producer warps copy it by TMA (cp.async.bulk) completing on mbarriers, one the
// bins and uniforms of up to 32 columns of a tree at a time into a ring (and hints the table into
// L2), the other each tree's tables into one of three buffers (two where three do not fit), with
// its same-branch rows and breakpoint factors where they fit (STAGED; else they are read from
// global memory).
// 0.085 us a column at 100 leaves; with whole columns copied in by the drawing warp itself, 8
// tested at a time, and rows and factors read when needed, 0.210. Every wait is bounded; one that
// runs out records ERR_WAIT_LIMIT and the kernel returns after its copies have landed.

constexpr float margin = 2e-5f;  // over twice 64 roundings

// Fields of a tree the traceback needs.
struct TreeRef {
    int blk, start, len, S, S1, M;
    long long cell0, state0, prev_state0, t2_0, gptr0;
};
__device__ __forceinline__ TreeRef tree_ref(const BatchDev &d, int blk) {
    const BlockDev &B = d.blocks[blk];
    return TreeRef{blk, B.start, B.len, B.S, B.S1, B.M, B.cell0, B.state0, B.prev_state0, B.t2_0, B.gptr0};
}

// The arrays of a tree buffer, each copied from the 16-byte boundary below its start.
enum { A_TM, A_RSTAY, A_BPTR, A_SINFO, A_T2OFF, A_PERM, A_GPTR, A_GIDX, A_DP, A_RROW, A_CROW, A_ROWS, ARRAYS };
// Layout of one tree buffer: array a from word at[a] on.
struct TreeBufLayout {
    int at[ARRAYS], total;
    // maxM: entries of the same-branch rows, 0: neither they nor the breakpoint's factors staged
    __host__ __device__ TreeBufLayout(int maxS, int maxM) {
        const int arr = (4 * maxS + 32 + 15) & ~15;
        const int bytes[ARRAYS] = {4 * MAXT * MAXT, 4 * MAXT, 160, 16 * maxS, arr, arr, arr, arr, arr,
                                   maxM > 0 ? arr : 0, maxM > 0 ? arr : 0,
                                   maxM > 0 ? (4 * maxM + 32 + 15) & ~15 : 0};
        total = 0;
        for (int a = 0; a < ARRAYS; a++) {
            at[a] = total / 4;
            total += bytes[a];
        }
    }
};
// A tree as its buffer holds it.
struct TreeTables {
    TreeRef ref;
    int2 src;         // the breakpoint's states
    int off[ARRAYS];  // where each array begins, in words of the buffer
};

constexpr int CC = 32;  // columns of a chunk and of a test: a tree's, from its last down
constexpr int NCH = 4;  // chunks of the ring
constexpr int CHUNK_BYTES = 4 * CC * MAXT + 8 * (CC + 4);  // bins, then uniforms (the column before too)

template <bool STAGED>
__global__ void __launch_bounds__(96) k_traceback_split(BatchDev d, int maxS, int nbuf) {
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char dyn_b[];
    unsigned char *ring = dyn_b;                            // [NCH] chunks
    unsigned char *tbuf = ring + NCH * CHUNK_BYTES;         // [nbuf] tree buffers
    __shared__ uint64_t cfull[NCH], cfree[NCH], tfull[3], tfree[3];  // copies landed; buffer read
    __shared__ int chunks_issued, trees_issued;
    __shared__ volatile int stop;
    __shared__ TreeTables trees[3];
    __shared__ __align__(16) float t2row[32], tmcol[32];    // the state's V, W factors
    __shared__ float ordw[32];
    __shared__ int ordj[32];
    const TreeBufLayout TL(maxS, STAGED ? d.maxM : 0);
    const TTab<float> tab(d);
    const int qi = cta_instance(d);
    const InstDev I = d.inst[qi];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NB = I.T - 1;
    const int L = I.seqlen;
    const double *u = d.uniforms + I.col0;

    if (threadIdx.x == 0) {
        for (int q = 0; q < NCH; q++) {
            mbar_init(&cfull[q], 1);
            mbar_init(&cfree[q], 1);
        }
        for (int q = 0; q < 3; q++) {
            mbar_init(&tfull[q], 1);
            mbar_init(&tfree[q], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        stop = chunks_issued = trees_issued = 0;
    }
    __syncthreads();
    // a producer's wait for a buffer, given up when the drawing warp has stopped
    auto wait_free = [&](uint64_t *bar, unsigned parity) -> bool {
        for (int it = 0; it < WAIT_TRIES && !stop; it++)
            if (mbar_test(bar, parity)) return true;
        return false;
    };
    int waited_chunks = 0, waited_trees = 0;  // the drawing warp's

    if (warp == 1) {
        // ---- chunks: m in slot m % NCH
        const float *bins = d.bins32 + (size_t)I.col0 * MAXT;
        int m = 0;
        bool ok = true;
        TreeRef t = tree_ref(d, I.block0 + I.ntrees - 1);
        for (int bi = I.ntrees - 1; bi >= 0 && ok; bi--) {
            TreeRef next = t;
            if (bi > 0) next = tree_ref(d, t.blk - 1);
            for (int hi = t.start + t.len - 1; hi >= t.start; hi -= CC, m++) {
                const int lo = imax(t.start, hi - CC + 1), slot = m % NCH;
                if (m >= NCH && !wait_free(&cfree[slot], (unsigned)(((m / NCH) & 1) ^ 1))) {
                    ok = false;
                    break;
                }
                if (lane == 0) {
                    // the chunk's part of the table into L2, and the column before it
                    const size_t Sm = (size_t)imax(t.S, 1), S1 = (size_t)imax(t.S1, 1);
                    const float *col = tab.fw + t.cell0 + (size_t)(lo - t.start) * Sm;
                    l2_prefetch(col, sizeof(float) * Sm * (hi - lo + 1));
                    if (lo == t.start && lo > 0) l2_prefetch(col - S1, sizeof(float) * S1);
                    unsigned char *at = ring + slot * CHUNK_BYTES;
                    const int ulo = imax(lo - 1, 0);
                    const Rounded<8> ru(u + ulo, hi - ulo + 1);
                    const unsigned bb = 4u * MAXT * (unsigned)(hi - lo + 1);
                    mbar_expect_tx(&cfull[slot], bb + ru.bytes);
                    bulk_g2s(at, bins + (size_t)lo * MAXT, bb, &cfull[slot]);
                    bulk_g2s(at + 4 * CC * MAXT, ru.a16, ru.bytes, &cfull[slot]);
                }
                __syncwarp();
            }
            t = next;
        }
        if (lane == 0) chunks_issued = m;
    } else if (warp == 2) {
        // ---- tree tables: the x-th tree from the last in buffer x % nbuf, an array a lane
        TreeRef X = tree_ref(d, I.block0 + I.ntrees - 1);
        int2 src = d.srcs[X.blk];
        int x = 0, b = 0;
        unsigned phase = 0;
        for (; x < I.ntrees; x++) {
            const bool sw = X.start > 0;  // a switch into this tree exists
            const int S = X.S, S1 = imax(X.S1, 1);
            const void *at = nullptr;
            int words = 0;
            switch (lane) {
                case A_TM: at = tab.tm + (size_t)X.blk * MAXT * MAXT; words = MAXT * NB; break;
                case A_RSTAY: at = tab.rstay + (size_t)X.blk * MAXT; words = MAXT; break;
                case A_BPTR: at = d.bt_ptr + (size_t)X.blk * (MAXT + 1); words = MAXT + 1; break;
                case A_SINFO: at = d.sinfo + X.state0; words = 4 * S; break;
                case A_T2OFF: at = d.t2off + X.state0; words = S; break;
                case A_PERM: at = d.bt_perm + X.state0; words = S; break;
                case A_ROWS: at = tab.rows + X.t2_0; words = STAGED ? X.M : 0; break;
                case A_GPTR: at = d.gptr + X.gptr0; words = imax(S, 1) + 1; break;
                case A_GIDX: at = d.gidx + X.prev_state0; words = S1; break;
                case A_DP: at = tab.dprob + X.prev_state0; words = S1; break;
                case A_RROW: at = tab.rrow + X.state0; words = STAGED ? imax(S, 1) : 0; break;
                case A_CROW: at = tab.crow + X.state0; words = STAGED ? imax(S, 1) : 0; break;
            }
            const bool of_switch = lane >= A_GPTR && lane <= A_CROW;
            if (of_switch ? !sw : S == 0) words = 0;
            const Rounded<4> r(at, words);
            if (x >= nbuf) {
                if (words > 0) l2_prefetch(r.a16, r.bytes);
                if (!wait_free(&tfree[b], phase ^ 1)) break;
            }
            const unsigned tx = __reduce_add_sync(FULL, r.bytes);
            if (lane == 0) {
                trees[b].ref = X;
                trees[b].src = src;
            }
            if (lane < ARRAYS) trees[b].off[lane] = TL.at[lane] + r.off;
            __syncwarp();
            if (lane == 0) mbar_expect_tx(&tfull[b], tx);
            __syncwarp();
            if (words > 0)
                bulk_g2s(tbuf + (size_t)b * TL.total + 4 * TL.at[lane], r.a16, r.bytes, &tfull[b]);
            if (x + 1 < I.ntrees) {
                X = tree_ref(d, X.blk - 1);
                src = d.srcs[X.blk];
            }
            if (++b == nbuf) {
                b = 0;
                phase ^= 1;
            }
        }
        if (lane == 0) trees_issued = x;
    } else {
        int *path = d.path + I.col0;
        bool failed = false;
        int state = 0, m = 0;                     // m: chunks taken
        const int g = lane >> 2, sub = lane & 3;  // a test's columns g + 8 j, by four lanes
        {
            // the last column of all (sample_thread.cpp:534-539)
            const BlockDev &B = d.blocks[I.block0 + I.ntrees - 1];
            const float *c = tab.fw + B.cell0 + (size_t)(B.len - 1) * imax(B.S, 1);
            state = warp_sample<float>(imax(B.S, 1), u[L - 1], [&](int j) { return c[j]; });
            if (lane == 0) path[L - 1] = state;
        }
        int b = 0;
        unsigned tphase = 0;
        for (int bi = I.ntrees - 1; bi >= 0 && !failed; bi--) {
            failed |= !mbar_wait(&tfull[b], tphase);
            waited_trees++;
            failed = __any_sync(FULL, failed);
            if (failed) break;
            const TreeTables &X = trees[b];
            const int S = X.ref.S, start = X.ref.start;
            const float *const fw = tab.fw + X.ref.cell0;  // the tree's table
            const int *const base = (const int *)(tbuf + (size_t)b * TL.total);
            auto floats = [&](int a) { return (const float *)base + X.off[a]; };
            const float *tmS = floats(A_TM), *rst = floats(A_RSTAY);
            const int *bptr = base + X.off[A_BPTR], *t2off = base + X.off[A_T2OFF], *perm = base + X.off[A_PERM];
            const StateInfo *sinfo = (const StateInfo *)(base + X.off[A_SINFO]);

            // The drawn state: its node's states, its V and W factors and a lane's share of them.
            int kj1 = 0, km = 0, ys = 0;
            float t2r[8];
            float4 tmr[2];
            auto set_state = [&](int k) {
                const StateInfo sk = sinfo[k];
                kj1 = sk.j1;
                km = sk.m;
                ys = k - sk.j1;
                const int row = t2off[k];
                const float stay = 1.0f - rst[sk.time];
                const float *r = STAGED ? floats(A_ROWS) + row : tab.rows + X.ref.t2_0 + row;
                __syncwarp();
                t2row[lane] = lane < km ? r[(long long)lane * km] + (lane == ys ? stay : 0.0f) : 0.0f;
                tmcol[lane] = lane < NB ? tmS[lane * MAXT + sk.time] : 0.0f;
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; i++) t2r[i] = t2row[sub + 4 * i];
#pragma unroll
                for (int q = 0; q < 2; q++) tmr[q] = ((const float4 *)tmcol)[2 * sub + ((q + g) & 1)];
            };
            // The switch into this tree (sample_hmm_posterior_step) from state k: the gather list
            // merged with the recombination and recoalescence sources, in state order; a lane's
            // source, its factor and its value of the column before. More than 30: by one lane.
            int p0 = 0, ng2 = 0, e0 = -1, e1 = -1, src_j = -1;
            float w0 = 0.0f, w1 = 0.0f, src_w = 0.0f, src_c = 0.0f;
            const float *const before = fw - imax(X.ref.S1, 1);
            const int *gi = base + X.off[A_GIDX], *gp = base + X.off[A_GPTR];
            const float *dp = floats(A_DP);
            auto sources = [&](int k) {
                p0 = gp[k];
                ng2 = gp[k + 1] - p0;
                const float rr = STAGED ? floats(A_RROW)[k] : tab.rrow[X.ref.state0 + k];
                const float cr = STAGED ? floats(A_CROW)[k] : tab.crow[X.ref.state0 + k];
                const int2 src = X.src;
                // the two extra sources in state order (get(): recoalescence wins a tie)
                e0 = e1 = -1;
                w0 = w1 = 0.0f;
                if (src.x >= 0 && src.x != src.y) { e0 = src.x; w0 = rr; }
                if (src.y >= 0) {
                    if (e0 < 0) { e0 = src.y; w0 = cr; }
                    else if (src.y < e0) { e1 = e0; w1 = w0; e0 = src.y; w0 = cr; }
                    else { e1 = src.y; w1 = cr; }
                }
                src_j = -1;
                if (ng2 <= 30) {
                    if (lane < ng2) { src_j = gi[p0 + lane]; src_w = dp[src_j]; }
                    if (lane == 30 && e0 >= 0) { src_j = e0; src_w = w0; }
                    if (lane == 31 && e1 >= 0) { src_j = e1; src_w = w1; }
                    src_c = src_j >= 0 ? before[src_j] : 0.0f;
                }
            };
            if (S > 0) set_state(state);
            bool ready = false;  // the switch's sources are loaded
            int lo = start;
            const double *uc = nullptr;  // the chunk's uniforms, by column - lo
            int slot = 0;
            for (int hi = start + X.ref.len - 1; hi >= start; hi = lo - 1) {
                lo = imax(start, hi - CC + 1);
                slot = m % NCH;
                const unsigned phase = (unsigned)((m / NCH) & 1);
                m++;
                if (lo == start && bi > 0) {
                    sources(state);
                    ready = true;
                }
                // the tree's last column is drawn already
                int c0 = hi == start + X.ref.len - 1 ? hi - 1 : hi;
                bool landed = false;
                const float *bins = (const float *)(ring + slot * CHUNK_BYTES);
                auto land = [&]() {
                    if (landed) return;
                    failed |= !mbar_wait(&cfull[slot], phase);
                    failed = __any_sync(FULL, failed);
                    waited_chunks++;
                    landed = true;
                    const int ulo = imax(lo - 1, 0);
                    uc = (const double *)(ring + slot * CHUNK_BYTES + 4 * CC * MAXT) +
                         ((uintptr_t)(u + ulo) & 15) / 8 + (lo - ulo);
                };
                if (S == 0) {
                    // fully specified tree: its single state carries over
                    if (lane <= c0 - lo) path[c0 - lane] = 0;
                    c0 = lo - 1;
                }
                while (c0 >= lo) {
                    const int ng = c0 - lo + 1;
                    // does a column's draw stay at the current state? The lane's part of V is on
                    // its way while W is summed; no branches, so that the four columns overlap
                    // (past the last one they repeat it)
                    float v[4][8], sb[4], ss[4], sr[4], uf[4];
                    const float *cp[4];
                    int col[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        col[j] = c0 - imin(g + 8 * j, ng - 1);
                        cp[j] = fw + (size_t)(col[j] - start) * S + kj1 + sub;
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (4 * i >= km) break;
#pragma unroll
                        for (int j = 0; j < 4; j++) v[j][i] = sub + 4 * i < km ? cp[j][4 * i] : 0.0f;
                    }
                    land();
                    if (failed) break;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uf[j] = (float)uc[col[j] - lo];
                        const float4 *bp = (const float4 *)(bins + (col[j] - lo) * MAXT);
                        float w[2];
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const int y = 4 * (2 * sub + ((q + g) & 1));  // no bank twice
                            const float4 bv = bp[y >> 2];
                            w[q] = ((y < NB ? bv.x * tmr[q].x : 0.0f) + (y + 1 < NB ? bv.y * tmr[q].y : 0.0f)) +
                                   ((y + 2 < NB ? bv.z * tmr[q].z : 0.0f) + (y + 3 < NB ? bv.w * tmr[q].w : 0.0f));
                        }
                        sr[j] = w[0] + w[1];
                        sb[j] = ss[j] = 0.0f;
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (4 * i >= km) break;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float w = v[j][i] * t2r[i];
                            sb[j] += sub + 4 * i < ys ? w : 0.0f;
                            ss[j] += sub + 4 * i == ys ? w : 0.0f;
                            sr[j] += sub + 4 * i > ys ? w : 0.0f;
                        }
                    }
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1) {
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            sb[j] += __shfl_xor_sync(FULL, sb[j], o);
                            ss[j] += __shfl_xor_sync(FULL, ss[j], o);
                            sr[j] += __shfl_xor_sync(FULL, sr[j], o);
                        }
                    }
                    unsigned open = 0;  // a bit per column
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float t = uf[j] * (sb[j] + ss[j] + sr[j]);
                        const bool sure = (ys == 0 || sb[j] * (1.0f + margin) < t * (1.0f - margin)) &&
                                          t * (1.0f + margin) <= (sb[j] + ss[j]) * (1.0f - margin) && t > 1e-30f;
                        open |= g + 8 * j < ng && !sure ? 1u << (g + 8 * j) : 0u;
                    }
                    open = __reduce_or_sync(FULL, open);
                    int nstay = open ? __ffs(open) - 1 : ng;
                    bool leaves = false;
                    const int cs = c0 - nstay;
                    const float *cq = fw + (size_t)(cs - start) * S, *bq = bins + (cs - lo) * MAXT;
                    if (nstay < ng) {
                        // the same for one column as the draw is defined
                        float db = 0.0f, ds = 0.0f, da = 0.0f, dw = 0.0f;
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const int y = 8 * sub + q;
                            const float w = y < km ? cq[kj1 + y] * t2row[y] : 0.0f;
                            da += w;
                            db += y < ys ? w : 0.0f;
                            ds += y == ys ? w : 0.0f;
                            dw += y < NB ? bq[y] * tmcol[y] : 0.0f;
                        }
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) {
                            db += __shfl_xor_sync(FULL, db, o);
                            ds += __shfl_xor_sync(FULL, ds, o);
                            da += __shfl_xor_sync(FULL, da, o);
                            dw += __shfl_xor_sync(FULL, dw, o);
                        }
                        const float t = (float)uc[cs - lo] * (da + dw);
                        leaves = !((ys == 0 || db < t) && t <= db + ds);
                        if (!leaves) nstay++;
                    }
                    if (lane < nstay) path[c0 - lane] = state;
                    int x = state;
                    if (leaves) {
                        // exact draw of the first column that leaves, by the whole warp
                        const float w_v = lane < km ? cq[kj1 + lane] * t2row[lane] : 0.0f;
                        const float w = lane < NB ? bq[lane] * tmcol[lane] : 0.0f;
                        const float vin = lane_scan(w_v, lane), win = lane_scan(w, lane);
                        const float vt = __shfl_sync(FULL, vin, 31), wt = __shfl_sync(FULL, win, 31);
                        const float tt = (float)uc[cs - lo] * (vt + wt);
                        if (tt <= vt) {
                            const unsigned hit = __ballot_sync(FULL, lane < km && vin >= tt);
                            x = kj1 + (hit ? __ffs(hit) - 1 : km - 1);
                        } else {
                            const float t2 = tt - vt;
                            const unsigned hit = __ballot_sync(FULL, lane < NB && win >= t2);
                            const unsigned pos = __ballot_sync(FULL, w > 0.0f);
                            const int a = hit ? __ffs(hit) - 1 : (pos ? 31 - __clz(pos) : 0);
                            const float excl = __shfl_sync(FULL, win - w, a);
                            const float rem = (t2 - excl) / tmcol[a];  // threshold on the fw scale
                            const int q0 = bptr[a], q1 = bptr[a + 1];
                            float carry = 0.0f;
                            int res = -1, last = q0;
                            for (int pb = q0; pb < q1; pb += 32) {
                                const int pp = pb + lane;
                                const float f = pp < q1 ? cq[perm[pp]] : 0.0f;
                                const float fin = lane_scan(f, lane);
                                const unsigned got = __ballot_sync(FULL, pp < q1 && carry + fin >= rem);
                                const unsigned nz = __ballot_sync(FULL, pp < q1 && f > 0.0f);
                                if (nz) last = pb + 31 - __clz(nz);
                                if (got) {
                                    res = pb + __ffs(got) - 1;
                                    break;
                                }
                                carry += __shfl_sync(FULL, fin, 31);
                            }
                            // past the bin's sum by rounding: its last state of positive weight
                            x = res >= 0 ? perm[res] : (q1 > q0 ? perm[last] : state);
                        }
                        if (lane == 0) path[cs] = x;
                    }
                    c0 -= leaves ? nstay + 1 : nstay;
                    if (x != state) {
                        state = x;
                        set_state(state);
                        ready = false;
                    }
                }
                land();
                if (failed) break;
                if (lo > start) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&cfree[slot]);
                }
            }
            if (failed) break;
            if (bi > 0) {
                if (!ready) sources(state);
                const double ub = uc[-1];
                int x = 0;
                if (ng2 <= 30) {
                    // put in state order; the sums run in that order
                    int rank = lane + (e0 >= 0 && e0 < src_j) + (e1 >= 0 && e1 < src_j);
                    const int n0 = __popc(__ballot_sync(FULL, lane < ng2 && src_j <= e0));
                    const int n1 = __popc(__ballot_sync(FULL, lane < ng2 && src_j <= e1));
                    if (lane == 30) rank = n0;
                    if (lane == 31) rank = n1 + 1;
                    if (src_j >= 0) {
                        ordw[rank] = src_c * src_w;
                        ordj[rank] = src_j;
                    }
                    __syncwarp();
                    const int cnt = ng2 + (e0 >= 0) + (e1 >= 0);
                    const float wv = lane < cnt ? ordw[lane] : 0.0f;
                    const int j = lane < cnt ? ordj[lane] : -1;
                    float tot = 0.0f, run = 0.0f;
                    for (int q = 0; q < cnt; q += 4) {  // (past the last: + 0)
                        float w[4];
#pragma unroll
                        for (int y = 0; y < 4; y++) w[y] = __shfl_sync(FULL, wv, (q + y) & 31);
#pragma unroll
                        for (int y = 0; y < 4; y++) {
                            tot += w[y];
                            if (lane == q + y) run = tot;
                        }
                    }
                    const float pick = (float)ub * tot;
                    const unsigned hit = __ballot_sync(FULL, lane < cnt && run >= pick);
                    const unsigned pos = __ballot_sync(FULL, lane < cnt && wv > 0.0f);
                    const int sel = hit ? __ffs(hit) - 1 : pos ? 31 - __clz(pos) : -1;
                    x = sel >= 0 ? __shfl_sync(FULL, j, sel) : 0;
                } else {
                    if (lane == 0) {
                        // merged walk of the gather list and the extras: pass 0 sums, pass 1 draws
                        float tot = 0.0f, run = 0.0f, pick = 0.0f;
                        int last = -1;
                        x = -1;
                        for (int pass = 0; pass < 2 && x < 0; pass++) {
                            int p = 0, q = 0;
                            while ((p < ng2 || q < 2) && x < 0) {
                                const int eq = q == 0 ? e0 : (q == 1 ? e1 : -1);
                                if (eq < 0 && q < 2) { q++; continue; }
                                int j;
                                float wv;
                                if (q < 2 && (p >= ng2 || eq < gi[p0 + p])) {
                                    j = eq;
                                    wv = before[j] * (q == 0 ? w0 : w1);
                                    q++;
                                } else {
                                    j = gi[p0 + p];
                                    wv = before[j] * dp[j];
                                    p++;
                                }
                                if (pass == 0) {
                                    tot += wv;
                                } else {
                                    run += wv;
                                    if (wv > 0.0f) last = j;
                                    if (run >= pick) x = j;
                                }
                            }
                            if (pass == 0) pick = (float)ub * tot;
                        }
                        if (x < 0) x = last >= 0 ? last : 0;
                    }
                    x = __shfl_sync(FULL, x, 0);
                }
                if (lane == 0) path[start - 1] = x;
                state = x;
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&cfree[slot]);
                mbar_arrive(&tfree[b]);
            }
            if (++b == nbuf) {
                b = 0;
                tphase ^= 1;
            }
        }
        if (failed && lane == 0) {
            stop = 1;
            report_error(d.err, ERR_WAIT_LIMIT, qi, -1, -1);
        }
    }
    __syncthreads();
    // every copy issued has landed before the CTA's shared memory is released
    if (threadIdx.x == 0) {
        for (int m = waited_chunks; m < chunks_issued; m++) mbar_wait(&cfull[m % NCH], (unsigned)((m / NCH) & 1));
        for (int m = waited_trees; m < trees_issued; m++) mbar_wait(&tfull[m % nbuf], (unsigned)((m / nbuf) & 1));
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------------------
// The reference's scan, for many columns at once by a CTA.
//
// Inside a tree the draw of column i depends on the later column only through its state k, and
// mostly stays at k: the first state whose running sum reaches u sum(A) is k when the sum before
// k is below the pick and the sum through k reaches it. Those sums do not depend on the other
// columns' draws, so the CTA tests up to 64 columns at once: four lanes take a column (8,
// 16 or 32 where the lot has fewer), lane q the states congruent to q, and butterfly steps
// combine them. The first column that
// leaves k, if any, is drawn by one warp exactly as a column on its own; the columns after it
// are tested again under the new state's row.
// In FP32 every column of a round is drawn as one on its own, up to four by a warp (the same sums
// in the same order whatever the round), and the draws are kept up to the first that leaves k:
// 0.49 us a column at 1572 states, where one warp per instance took 2.09.
//
// What bounds it in FP64: the FP64 pipe (64 cycles a warp's instruction). Four lanes a column with all
// 32 lanes at work cost S / 32 FMAs a column plus a sixteenth of an instruction for each
// butterfly step; one warp per instance (8 columns at a time, each summed in order and resolved
// by a binary search) took 980 cycles a column at 99 states and 4,100 at 483, on one
// sub-partition of the four.
//
// A tree's columns (as many as a buffer holds) and their uniforms arrive by bulk copies, the
// next lot's while this one is drawn. A tree switch has few sources of nonzero weight (the drawn
// state's gather list and the breakpoint's two states), taken in state order.
constexpr int TW = 8;  // warps of k_traceback_lots
template <int N>
struct Cols {
    static constexpr int value = N;
};
template <typename F>
constexpr int LOT = sizeof(F) == 8 ? 8 * TW : 4 * TW;  // columns of a lot and a round at most

template <typename F>
__global__ void __launch_bounds__(32 * TW) k_traceback_lots(BatchDev d, int buf_bytes) {
    constexpr bool wide = sizeof(F) == 8;
    extern __shared__ __align__(16) unsigned char dyn_b[];
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int u_bytes = 8 * LOT<F> + 32, E = sizeof(F);
    const TTab<F> tab(d);
    F *const trans = (F *)(dyn_b + 2 * buf_bytes + 2 * u_bytes);  // [maxS]
    __shared__ F tmS[MAXT * MAXT];
    __shared__ uint64_t bar[2];
    __shared__ int first, drawn, draws[LOT<F>];
    const int qi = cta_instance(d);
    const InstDev I = d.inst[qi];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int *path = d.path + I.col0;
    const double *u = d.uniforms + I.col0;
    bool failed = false;

    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();

    // lots: columns [lo, hi] of tree bi, from the last tree's last column down
    struct Lot {
        int bi, lo, hi, off, uoff;  // off, uoff: where column lo's values begin in the buffer
    };
    auto lot_at = [&](int bi, int hi) {
        const BlockDev &B = d.blocks[I.block0 + bi];
        const int Sm = imax(B.S, 1), cap = (buf_bytes - 16) / (E * Sm);
        return Lot{bi, imax(B.start, hi - imin(cap, LOT<F>) + 1), hi, 0, 0};
    };
    auto fetch = [&](Lot &t, int b) {
        const BlockDev &B = d.blocks[I.block0 + t.bi];
        const int Sm = imax(B.S, 1), n = t.hi - t.lo + 1;
        const Rounded<E> rt(tab.fw + B.cell0 + (size_t)(t.lo - B.start) * Sm, (long long)n * Sm);
        const Rounded<8> ru(u + t.lo, n);
        t.off = rt.off;
        t.uoff = ru.off;
        if (tid == 0) {
            mbar_expect_tx(&bar[b], rt.bytes + ru.bytes);
            bulk_g2s(dyn_b + (size_t)b * buf_bytes, rt.a16, rt.bytes, &bar[b]);
            bulk_g2s(dyn_b + 2 * buf_bytes + b * u_bytes, ru.a16, ru.bytes, &bar[b]);
        }
    };

    Lot cur = lot_at(I.ntrees - 1, I.seqlen - 1);
    fetch(cur, 0);
    int state = 0, n = 0;        // state of the column after; lots done
    bool pending = false;        // a lot in flight when the loop ends
    bool fresh = true;           // the state's row is to be built
    while (true) {
        const int b = n & 1;
        const BlockDev &B = d.blocks[I.block0 + cur.bi];
        const int S = B.S, Sm = imax(S, 1), start = B.start, len = B.len;
        // the next lot, into the other buffer (its last readers passed the barrier below)
        Lot next = cur;
        const bool more = cur.lo > 0;
        if (more) {
            next = cur.lo > start ? lot_at(cur.bi, cur.lo - 1) : lot_at(cur.bi - 1, cur.lo - 1);
            fetch(next, b ^ 1);
        }
        const bool top = cur.hi == start + len - 1;  // the tree's last column is in this lot
        if (top && S > 0) {
            const F *tmg = tab.tm + (size_t)(I.block0 + cur.bi) * MAXT * MAXT;
            for (int e = tid; e < (I.T - 1) * MAXT; e += 32 * TW) tmS[e] = tmg[e];
        }
        const bool landed = mbar_wait(&bar[b], (unsigned)((n >> 1) & 1));
        if (__syncthreads_or(!landed)) {
            failed = true;
            pending = more;
            break;
        }
        const F *buf = (const F *)(dyn_b + (size_t)b * buf_bytes) + cur.off;
        const double *ub = (const double *)(dyn_b + 2 * buf_bytes + b * u_bytes) + cur.uoff;
        auto column = [&](int c) { return buf + (size_t)(c - cur.lo) * Sm; };
        int c0 = cur.hi;

        if (top) {
            // the tree's last column, by warp 0; FP32: its weights through the switch by all
            if (!wide && cur.bi < I.ntrees - 1) {
                const int nb = I.block0 + cur.bi + 1;
                const BlockDev &N = d.blocks[nb];
                const int2 src = d.srcs[nb];
                const int *determ = d.determ + N.prev_state0;
                const F *c = column(c0), *dp = tab.dprob + N.prev_state0;
                const F rr = tab.rrow[N.state0 + state], cr = tab.crow[N.state0 + state];
                for (int j = tid; j < imax(N.S1, 1); j += 32 * TW) {
                    const F g = j == src.y ? cr : j == src.x ? rr : determ[j] == state ? dp[j] : F(0);
                    trans[j] = c[j] * g;
                }
                __syncthreads();
            }
            if (warp == 0) {
                const F *c = column(c0);
                const double uc = ub[c0 - cur.lo];
                int x;
                if (cur.bi == I.ntrees - 1) {
                    // the last column of all (sample_thread.cpp:534-539); a given last state
                    // (conditioned sampling) takes no draw
                    const int given = d.last_state ? d.last_state[qi] : -1;
                    x = given >= 0 ? given : warp_sample<F>(Sm, uc, [&](int j) { return c[j]; });
                } else if (!wide) {
                    x = warp_sample<F>(Sm, uc, [&](int j) { return trans[j]; });
                } else {
                    // through the switch into the next tree (sample_hmm_posterior_step)
                    const int nb = I.block0 + cur.bi + 1, k = state;
                    const BlockDev &N = d.blocks[nb];
                    const int2 src = d.srcs[nb];
                    const int *gp = d.gptr + N.gptr0 + k;
                    const int p0 = gp[0], ng = gp[1] - p0;
                    const F *dp = tab.dprob + N.prev_state0;
                    const F rr = tab.rrow[N.state0 + k], cr = tab.crow[N.state0 + k];
                    const bool hx = src.x != -1 && src.x != src.y, hy = src.y != -1;
                    if (ng + 2 <= 32) {
                        // lane e: the e-th source of the gather list, then the two states
                        int j = -1;
                        F wt = F(0);
                        if (lane < ng) {
                            j = d.gidx[N.prev_state0 + p0 + lane];
                            wt = c[j] * dp[j];
                        } else if (lane == ng && hx) {
                            j = src.x;
                            wt = c[j] * rr;
                        } else if (lane == ng + 1 && hy) {
                            j = src.y;
                            wt = c[j] * cr;
                        }
                        // their order by state, then the running sum in that order
                        int pos = 0;
                        for (int e = 0; e < ng + 2; e++) {
                            const int je = __shfl_sync(FULL, j, e);
                            pos += je >= 0 && je < j;
                        }
                        const int live = __popc(__ballot_sync(FULL, j >= 0));
                        F run = F(0), mine = F(0);
                        for (int r = 0; r < live; r++) {
                            const unsigned at = __ballot_sync(FULL, j >= 0 && pos == r);
                            run += __shfl_sync(FULL, wt, __ffs(at) - 1);
                            if (j >= 0 && pos == r) mine = run;
                        }
                        const F pick = (F)uc * run;
                        // the first state of all reaches a pick of zero
                        const unsigned hit = __ballot_sync(FULL, j >= 0 && mine >= pick);
                        if (pick <= F(0)) {
                            x = 0;
                        } else if (hit) {
                            int best = (hit >> lane & 1) ? j : 0x7fffffff;
                            best = __reduce_min_sync(FULL, best);
                            x = best;
                        } else {
                            x = imax(N.S1, 1) - 1;
                        }
                    } else {
                        const int *determ = d.determ + N.prev_state0;
                        x = warp_sample<F>(imax(N.S1, 1), uc, [&](int j) {
                            const F g = j == src.y ? cr : j == src.x ? rr : determ[j] == k ? dp[j] : F(0);
                            return c[j] * g;
                        });
                    }
                }
                if (lane == 0) {
                    path[c0] = x;
                    drawn = x;
                }
            }
            __syncthreads();
            state = drawn;
            c0--;
        }
        if (S == 0) {
            // fully specified tree: its single state carries over
            for (int c = cur.lo + tid; c <= c0; c += 32 * TW) path[c] = 0;
            state = 0;
            c0 = cur.lo - 1;
        }
        fresh |= top;
        while (c0 >= cur.lo) {
            if (fresh) {
                // trans[j] = TransMatrix::get(j, k) (trans.h:64-83)
                const StateInfo sk = d.sinfo[B.state0 + state];
                const long long row = B.t2_0 + d.t2off[B.state0 + state];
                F stay = F(0);
                if constexpr (!wide) stay = F(1) - tab.rstay[(size_t)(I.block0 + cur.bi) * MAXT + sk.time];
                for (int j = tid; j < S; j += 32 * TW) {
                    const StateInfo sj = d.sinfo[B.state0 + j];
                    const F tmab = tmS[sj.time * MAXT + sk.time];
                    F t = tmab;
                    if (sj.node == sk.node) {
                        t = TTab<F>::same(tab.rows[row + (long long)(j - sk.j1) * sk.m], tmab);
                        if (!wide && j == state) t += stay;
                    }
                    trans[j] = t;
                }
            }
            fresh = false;
            const int ncols = imin(LOT<F>, c0 - cur.lo + 1), k = state;
            if (tid == 0) first = ncols;
            __syncthreads();  // trans, first
            if constexpr (wide) {
                // lanes a column: 4, 8, 16 or 32, so that few columns still keep every warp busy
                const int lb = ncols > LOT<F> / 2 ? 2 : ncols > LOT<F> / 4 ? 3 : ncols > LOT<F> / 8 ? 4 : 5;
                const int g = tid >> lb, lanes = 1 << lb, q = tid & (lanes - 1);
                if ((tid & ~31) >> lb < ncols) {
                    const int mc = c0 - imin(g, ncols - 1);
                    const double *cp = column(mc);
                    double before = 0.0, after = 0.0;
                    int j = q;
#pragma unroll 4
                    for (; j < k; j += lanes) before = fma(cp[j], trans[j], before);
                    j += j == k ? lanes : 0;
#pragma unroll 4
                    for (; j < S; j += lanes) after = fma(cp[j], trans[j], after);
                    for (int o = 1; o < lanes; o <<= 1) {
                        before += __shfl_xor_sync(FULL, before, o);
                        after += __shfl_xor_sync(FULL, after, o);
                    }
                    const double through = fma(cp[k], trans[k], before);
                    const double pick = ub[mc - cur.lo] * (through + after);
                    const bool leave = g < ncols && !((k == 0 || before < pick) && pick <= through);
                    const unsigned l = __ballot_sync(FULL, leave);
                    if (l && lane == 0) atomicMin(&first, (tid + __ffs(l) - 1) >> lb);
                }
            } else {
                // up to 4 columns a warp, as few as keep the warps busy
                auto draw = [&](auto tag) {
                    constexpr int G = decltype(tag)::value;
                    const int g0 = G * warp;
                    if (g0 >= ncols) return;
                    const F *cg[G];
                    double ug[G];
                    int res[G];
#pragma unroll
                    for (int g = 0; g < G; g++) {
                        const int mc = c0 - imin(g0 + g, ncols - 1);
                        cg[g] = column(mc);
                        ug[g] = ub[mc - cur.lo];
                    }
                    warp_sample_group<F, G>(S, cg, trans, ug, res);
#pragma unroll
                    for (int g = G - 1; g >= 0; g--)
                        if (lane == 0 && g0 + g < ncols && res[g] != k) {
                            atomicMin(&first, g0 + g);
                            draws[g0 + g] = res[g];
                        }
                };
                if (ncols <= TW) draw(Cols<1>{});
                else if (ncols <= 2 * TW) draw(Cols<2>{});
                else draw(Cols<4>{});
            }
            __syncthreads();
            const int r = first;
            if (tid < r) path[c0 - tid] = k;
            if (r < ncols) {
                // the column that leaves, drawn as one on its own
                if (warp == 0) {
                    int x = 0;
                    if constexpr (wide) {
                        const F *cp = column(c0 - r);
                        x = warp_sample<F>(S, ub[c0 - r - cur.lo], [&](int j) { return cp[j] * trans[j]; });
                    } else {
                        x = draws[r];
                    }
                    if (lane == 0) {
                        path[c0 - r] = x;
                        drawn = x;
                    }
                }
                __syncthreads();
                fresh = drawn != state;
                state = drawn;
                c0 -= r + 1;
            } else {
                c0 -= r;
            }
            __syncthreads();  // first, drawn and trans are read
        }
        if (!more) break;
        __syncthreads();  // this lot's buffer is read
        cur = next;
        n++;
    }
    if (failed && tid == 0) {
        report_error(d.err, ERR_WAIT_LIMIT, qi, -1, -1);
        // the copies in flight, before the memory is released
        mbar_wait(&bar[n & 1], (unsigned)((n >> 1) & 1));
        if (pending) mbar_wait(&bar[(n & 1) ^ 1], (unsigned)(((n + 1) >> 1) & 1));
    }
    __syncthreads();
}

template <typename F>
void launch_lots(const BatchDev &d, cudaStream_t s) {
    // a lot of the largest tree in a buffer, where two buffers leave room for a second CTA on the
    // SM; else as many columns as two buffers hold, at least one
    const size_t col = sizeof(F) * (size_t)imax(d.maxS, 1);
    const size_t n = LOT<F> * col <= 44 * 1024 ? LOT<F> : imax(imin((int)(100 * 1024 / col), LOT<F>), 1);
    const size_t buf = (n * col + 16 + 15) & ~(size_t)15;
    const size_t smem = 2 * buf + 2 * (8 * LOT<F> + 32) + col;
    if (!raise_dynamic_smem(k_traceback_lots<F>, smem)) return;  // the launch reports it
    k_traceback_lots<F><<<d.ninst, 32 * TW, smem, s>>>(d, (int)buf);
    note_launch();
}

template <bool STAGED>
bool launch_split(const BatchDev &d, cudaStream_t s) {
    const int maxS = imax(d.maxS, 1);
    const size_t tree = TreeBufLayout(maxS, STAGED ? imax(d.maxM, 1) : 0).total;
    const int nbuf = NCH * CHUNK_BYTES + 3 * tree <= 224 * 1024 ? 3 : 2;
    const size_t smem = NCH * CHUNK_BYTES + nbuf * tree;
    if (smem > 224 * 1024) return false;
    prefer_shared(k_traceback_split<STAGED>);
    if (!raise_dynamic_smem(k_traceback_split<STAGED>, smem)) return true;  // the launch reports it
    k_traceback_split<STAGED><<<d.ninst, 96, smem, s>>>(d, maxS, nbuf);
    note_launch();
    return true;
}

// Batches drawn by the decomposed draw. It maps a uniform to another state than the scan does, so
// this line is part of the results: some 1,290 states, which two tree buffers and three times
// eight columns in 224 KB came to.
bool split_draws(const BatchDev &d) {
    const int maxS = imax(d.maxS, 1);
    const size_t columns = (4 * 8 * (size_t)maxS + 32 + 15) & ~(size_t)15;
    return d.bins32 && 3 * (columns + 4 * 8 * MAXT + 8 * (8 + 2)) + 2 * (size_t)TreeBufLayout(maxS, 0).total <= 224 * 1024;
}

}  // namespace

void launch_traceback(const BatchDev &d, bool fp32, cudaStream_t s) {
    if (!fp32) {
        launch_lots<double>(d, s);
        return;
    }
    if (split_draws(d) && (launch_split<true>(d, s) || launch_split<false>(d, s))) return;
    launch_lots<float>(d, s);
}

}  // namespace awg
