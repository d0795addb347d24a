// The column chains that need no bit-for-bit twin elsewhere: K3 in FP64 (the forward pass) and
// K5 in both precisions (the backward pass), one CTA per instance, and the parallel kernels
// that finish their tables.
//
// Forward (arghmm_forward_block, sample_thread.cpp:252-295), from column x_{i-1}:
//   bin[a] = sum of x over states of time a;  tf[b] = sum_a tm[a][b] bin[a]
//   x_i[k] = (tf[b_k] + sum over the states j of k's node of t2[a_j][k] x[j]) e_i[k]
// Backward (the reference has none), from column g_{i+1} = e_{i+1} bw_{i+1}: the transpose,
//   bw_i[j] = sum_b tm[a_j][b] G[b] + sum over the states k of j's node of t2[a_j][k] g[k]
// Both step the previous column by the same structure, so one kernel does both: bins, a small
// matrix-vector product, a dot per state over its node. At a tree boundary the column goes
// through the switch matrix (arghmm_forward_switch, sample_thread.cpp:345-389) or back.
//
// What bounds it: the chain of columns, and in FP64 the FP64 pipe, which takes 64 cycles for a
// warp's instruction whether its lanes are live or not (2 FMAs a clock an SM) and 64 for a
// dependent one. So the FP64 form counts instructions on the busiest sub-partition:
//   - no division and no normalisation in the chain: a column is scaled by a power of two from
//     the largest bin's exponent (integer work, exact), the table is written as it is scaled,
//     and parallel kernels normalise it where it is wanted. The log-likelihood telescopes to
//     log(sum of the last column) plus ln 2 times the exponents.
//   - the power is chosen a column ahead, so a column's factor is ready before its inflow and
//     ends it with one fused product: 1.22 us a column at 99 states and 2.81 at 483 when it came in, 1.27 and
//     2.90 with the power of the column's own bins (1.99 and 4.46 with a division a column).
//   - bins by a segmented scan over lanes (log2 of a bin's lanes dependent adds); the product
//     with tm split over all lanes of the four reduction warps, so the owners add one value
//     instead of four warps' shares.
//   - owners take the states in descending order of their node's length, so a warp's lanes
//     have dots of like length, and up to OWNERS / 2 states two lanes take one state's even
//     and odd terms. A dot is always (even terms) + (odd terms): results do not depend on the
//     form, the block size or the batch.
//   - a tree's set-up (13,000 cycles at 99 states, 20,000 at 483, where a tree has some 30
//     columns) waits for memory as few times as it can: rows are copied as they lie and turned
//     into moving parts by the owner of their dot, a switch's sources come two at a time.
//     10,000 columns in 221 trees at 99 states: 13.2 ms with rows gathered by state, 12.9 so.
// FP32 (backward): the stay and the emission, which carry almost all of a state's mass, on
// pairs (f2.cuh), the inflow plain.

#include <cuda_runtime.h>

#include "f2.cuh"
#include "kernels.h"

namespace awg {

namespace {

constexpr int NRW = 4;                             // reduction warps
constexpr int RBINS = (MAXT - 1 + NRW - 1) / NRW;  // time bins per reduction warp (<= 8)
constexpr int OWNERS = 384;                        // owner threads at most: 16 warps in all
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void named_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ int uniform(int v) { return (int)__reduce_max_sync(FULL, (unsigned)v); }

// Floating-point formats: biased exponents, exact powers of two.
template <typename F> struct Fmt;
template <> struct Fmt<double> {
    static constexpr int bias = 1023, top = 2047;
    __device__ static int expo(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
    __device__ static double pow2(int k) { return __hiloint2double((k + 1023) << 20, 0); }  // |k| < 1023
    // e 2^k (exact); the product is out of line: predicated, it would hold the FP64 pipe for every
    // call
    __device__ static double scaled(double e, int k) {
        const int x = expo(e) + k;
        if (expo(e) > 0 && x > 0 && x < 2047) return __hiloint2double(__double2hiint(e) + (k << 20), __double2loint(e));
        return times_pow2(e, k);
    }
    __device__ __noinline__ static double times_pow2(double e, int k) { return e * pow2(k); }
};
template <> struct Fmt<float> {
    static constexpr int bias = 127, top = 255;
    __device__ static int expo(float x) { return (__float_as_int(x) >> 23) & 0xff; }
    __device__ static float pow2(int k) { return __int_as_float((k + 127) << 23); }
};
// 1023 - E (127 - E), the power that brings the largest exponent to 0 (to 1 from the format's last
// one, whose power would not be a normal number); 0 for an empty column
template <typename F>
__device__ __forceinline__ int rescale(int E) {
    return E == 0 || E == Fmt<F>::top ? 0 : imax(imin(Fmt<F>::bias - E, Fmt<F>::bias - 1), 1 - Fmt<F>::bias);
}

template <typename F> struct Tab;
template <> struct Tab<double> {
    const double *tm, *inv, *var, *dprob, *rrow, *crow, *rows;
    const float *rstay = nullptr;
    __device__ explicit Tab(const BatchDev &d)
        : tm(d.tm), inv(d.inv_lk), var(d.varemit), dprob(d.determprob), rrow(d.recombrow),
          crow(d.recoalrow), rows(d.gts) {}
    // tmatrix2[a][k] (sample_thread.cpp:223-224)
    __device__ static double t2(double v, double tmab) { return v - tmab; }
};
template <> struct Tab<float> {
    const float *tm, *inv, *var, *dprob, *rrow, *crow, *rows, *rstay;
    __device__ explicit Tab(const BatchDev &d)
        : tm(d.tm32), inv(d.inv32), var(d.var32), dprob(d.determprob32), rrow(d.recombrow32),
          crow(d.recoalrow32), rows(d.t2d32), rstay(d.rstay32) {}
    __device__ static float t2(float v, float) { return v; }
};

template <typename F>
__device__ __forceinline__ F warp_sum(F v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// A hint that moves [p, p + bytes) (the whole 16-byte granules inside it) from HBM into L2.
__device__ __forceinline__ void l2_prefetch(const void *p, size_t bytes) {
    const uintptr_t a = ((uintptr_t)p + 15) & ~(uintptr_t)15;
    const uintptr_t e = ((uintptr_t)p + bytes) & ~(uintptr_t)15;
    if (e > a)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a))
                     : "memory");
}
// The tables of a tree's set-up and columns, prefetched while another tree runs.
template <typename F, bool FWD>
__device__ __forceinline__ void prefetch_tree(const BatchDev &d, const Tab<F> &tab, int blk) {
    const BlockDev &N = d.blocks[blk];
    const size_t S = (size_t)imax(N.S, 1), S1 = (size_t)imax(N.S1, 1);
    l2_prefetch(d.sinfo + N.state0, sizeof(StateInfo) * S);
    l2_prefetch(d.t2off + N.state0, sizeof(int) * S);
    l2_prefetch(d.bt_perm + N.state0, sizeof(int) * S);
    l2_prefetch(tab.inv + N.state0, sizeof(F) * S);
    l2_prefetch(tab.rrow + N.state0, sizeof(F) * S);
    l2_prefetch(tab.crow + N.state0, sizeof(F) * S);
    l2_prefetch(tab.tm + (size_t)blk * MAXT * MAXT, sizeof(F) * MAXT * MAXT);
    l2_prefetch(d.bt_ptr + (size_t)blk * (MAXT + 1), sizeof(int) * (MAXT + 1));
    if (FWD) {
        l2_prefetch(d.gptr + N.gptr0, sizeof(int) * (S + 1));
        l2_prefetch(d.gidx + N.prev_state0, sizeof(int) * S1);
    } else {
        l2_prefetch(d.determ + N.prev_state0, sizeof(int) * S1);
    }
    l2_prefetch(d.determprob + N.prev_state0, sizeof(double) * S1);
    if (N.M > 0) l2_prefetch(tab.rows + N.t2_0, sizeof(F) * N.M);
    if (N.nvar > 0 && N.S > 0) l2_prefetch(tab.var + N.var0, sizeof(F) * N.nvar * (size_t)N.S);
}

// The reduction warps' first time bins (bl[NRW]: NB), the bins split by their states; whole
// bins, at most RBINS a warp.
__device__ __forceinline__ void bin_split(const int *bptr, int NB, int (&bl)[NRW + 1]) {
    const int S = bptr[NB];
    bl[0] = 0;
    bl[NRW] = NB;
#pragma unroll
    for (int q = 1; q < NRW; q++) {
        const int target = (q * S + NRW - 1) / NRW;
        int b = bl[q - 1];
        while (b < NB && bptr[b] < target) b++;
        b = imax(b, NB - (NRW - q) * RBINS);
        bl[q] = imin(b, bl[q - 1] + RBINS);
    }
}

// Powers of two taken out of a tree's columns. FP64: column i is scaled by k, chosen a column
// ahead from the bins of column i - 2 and the power that column i - 1 was scaled by, so that the
// factor is there before column i - 1's bins are; a column that these show to be far off (an
// emission penalty on every state) is scaled by `extra` as well. FP32, whose range is short: by
// column i - 1's bins themselves.
template <typename F> struct Scale;
template <> struct Scale<double> {
    int k = 0, extra = 0;
    // E: the largest exponent of column i - 1's bins
    __device__ void see(int E) { extra = E < 1023 - 40 || E > 1023 + 40 ? rescale<double>(E) : 0; }
    __device__ int used() const { return k + extra; }
    __device__ void next(int E) {
        k = E == 0 || E == 2047 ? 0 : imax(imin(1023 - E - used(), 1022), -1022);
    }
};
template <> struct Scale<float> {
    static constexpr int k = 0;
    int extra = 0;
    __device__ void see(int E) { extra = rescale<float>(E); }
    __device__ int used() const { return extra; }
    __device__ void next(int) {}
};

// Shared memory of a CTA, in units of F (then ints).
template <typename F>
struct SmemPlan {
    int col, head, own, rows, lo, order, rank;
    size_t bytes;
    __host__ __device__ SmemPlan(int maxS, int rows_n) {
        const int cs = maxS + MAXT, slots = maxS + 32 * NRW;
        col = 0;                   // [2][cs] columns in state order
        head = col + 2 * cs;       // reducers' slots: the pieces that chunks begin with
        own = head + slots;        // and those that bins begin with inside a chunk
        rows = own + slots;        // the tree's same-branch rows
        lo = rows + rows_n;        // FP32: low parts of a tree's last column
        order = lo + (sizeof(F) == 4 ? maxS : 0);
        bytes = (size_t)order * sizeof(F);
        rank = (int)bytes + 4 * maxS;   // byte offsets of the int arrays: order, rank
        order = (int)bytes;
        bytes = (size_t)rank + 4 * maxS;
    }
};

template <typename F>
struct Shared {
    F tm[MAXT * MAXT], bin[MAXT], tf[MAXT];  // tmatrix; the column's bins; its moves
    F srcsum[2];                             // backward: what the states on a breakpoint get
    int bptr[MAXT + 1], hist[MAXT + 1];
    int expo[NRW], lastexp;                  // largest exponents: of a column's bins, of a
                                             // tree's last column
};

// One instance; NTC threads at work. KPT units per owner thread, SPLIT lanes per state (a unit
// is a state, or its even or odd terms). rows_n: same-branch entries that fit shared memory (0:
// read from global memory).
template <typename F, bool FWD, int KPT, int SPLIT>
__device__ __forceinline__ void run_chain(const BatchDev &d, const InstDev &I, int qi, int rows_n, int NTC, Shared<F> &sh) {
    static_assert(FWD ? sizeof(F) == 8 : true, "the FP32 forward pass is forward32.cu");
    static_assert(SPLIT == 1 || KPT == 1, "");
    constexpr bool pairs = sizeof(F) == 4;
    constexpr bool SORT = sizeof(F) == 8;
    extern __shared__ __align__(16) unsigned char dyn_b[];
    const Tab<F> tab(d);
    const int maxS = I.maxS, NB = I.T - 1;
    const int tid = threadIdx.x, lane = tid & 31, rw = tid >> 5;
    const int NTS = NTC - 32 * NRW, st = tid - 32 * NRW;
    const bool reducer = tid < 32 * NRW;
    const SmemPlan<F> P(maxS, rows_n);
    F *const base_f = (F *)dyn_b;
    const int cs = maxS + MAXT;
    F *const col = base_f + P.col, *const head = base_f + P.head, *const own = base_f + P.own;
    F *const rowsS = base_f + P.rows;
    float *const lastlo = (float *)(base_f + P.lo);
    int *const order = (int *)(dyn_b + P.order), *const rank = (int *)(dyn_b + P.rank);
    F *const tmS = sh.tm, *const binS = sh.bin, *const tfS = sh.tf, *const srcsum = sh.srcsum;
    int *const bptr = sh.bptr, *const hist = sh.hist, *const expoS = sh.expo;
    int &lastexp = sh.lastexp;

    int c = 0;                    // buffer of the current column
    long long sumk = 0;           // FWD: the powers of two taken out (thread 0)
    double lnl = 0.0;             // FWD: logs of switches into fully specified trees (thread 0)
    const uint8_t *const cls = d.colclass + I.col0;
    const int L = I.seqlen;
    // classes of 64 columns, windows aligned to 32 of the instance's columns: bit j of vm / mm:
    // column 32 (w - !FWD) + j is variant / masked; the window after them in cnext
    auto class_at = [&](int col_) { return col_ >= 0 && col_ < L ? (int)cls[col_] : 0; };
    int w = FWD ? 0 : (L - 1) >> 5;
    const int wlo = 32 * (w - (FWD ? 0 : 1));
    unsigned long long vm, mm;
    {
        const int c0 = class_at(wlo + lane), c1 = class_at(wlo + 32 + lane);
        vm = (unsigned long long)__ballot_sync(FULL, c1 == COL_VARIANT) << 32 | __ballot_sync(FULL, c0 == COL_VARIANT);
        mm = (unsigned long long)__ballot_sync(FULL, c1 == COL_MASKED) << 32 | __ballot_sync(FULL, c0 == COL_MASKED);
    }
    int cnext = class_at(FWD ? wlo + 64 + lane : wlo - 32 + lane);
    auto bit = [&](unsigned long long m, int abs) { return (m >> (abs - 32 * (FWD ? w : w - 1)) & 1) != 0; };
    auto passed = [&](int abs) {  // column abs is done with
        if (FWD ? (abs & 31) == 31 : (abs & 31) == 0) {
            const unsigned v = __ballot_sync(FULL, cnext == COL_VARIANT), x = __ballot_sync(FULL, cnext == COL_MASKED);
            if (FWD) {
                w++;
                vm = vm >> 32 | (unsigned long long)v << 32;
                mm = mm >> 32 | (unsigned long long)x << 32;
                cnext = class_at(32 * w + 64 + lane);
            } else {
                w--;
                vm = vm << 32 | v;
                mm = mm << 32 | x;
                cnext = class_at(32 * (w - 2) + lane);
            }
        }
    };
    for (int k = tid; k < 2 * cs; k += NTC) col[k] = F(0);

    for (int b0 = 0; b0 < I.ntrees; b0++) {
        const int bi = FWD ? b0 : I.ntrees - 1 - b0;
        const int blk = I.block0 + bi;
        const BlockDev &B = d.blocks[blk];
        const int S = uniform(B.S), len = uniform(B.len), start = uniform(B.start), Sm = imax(S, 1);
        const long long s0 = B.state0;
        const bool first = b0 == 0;
        // the tree that the column comes from, and the boundary's arrays (the later tree's)
        const int sblk = FWD ? blk : blk + 1;
        named_sync(4, NTC);  // T1: the last tree's column is complete
        const int ek = first ? 0 : rescale<F>(lastexp);
        if (tid == NTC - 1 && b0 + 1 < I.ntrees) prefetch_tree<F, FWD>(d, tab, FWD ? blk + 1 : blk - 1);
        F *const prev = col + c * cs;
        c ^= 1;
        F *const cur = col + c * cs;

        // ---- backward: the states that a recombination or coalescence is on take a row
        int2 src = make_int2(-1, -1);
        if (!first) src = d.srcs[sblk];
        if (!FWD && !first && rw < 2) {
            const int which = rw == 0 ? src.x : src.y;
            const int Sn = imax(d.blocks[sblk].S, 1);
            const F *row = (rw == 0 ? tab.rrow : tab.crow) + d.blocks[sblk].state0;
            F s = F(0);
            if (which != -1)
                for (int k = lane; k < Sn; k += 32)
                    if (row[k] > F(0)) s = fma(row[k], prev[k], s);
            s = warp_sum(s);
            if (lane == 0) srcsum[rw] = s;
        }

        if (S == 0) {
            // fully specified tree: one state that carries over (sample_thread.cpp:201-206)
            named_sync(4, NTC);  // sums; lastexp is read
            F v = F(1);
            if (FWD) {
                if (first) {
                    v = (F)d.fw64[B.cell0];
                    if (tid == 0) cur[0] = v;
                } else if (tid < 32) {
                    const int *gp = d.gptr + B.gptr0;
                    const int *gi = d.gidx + B.prev_state0;
                    const F *dp = tab.dprob + B.prev_state0;
                    F sum = F(0);
                    for (int p = gp[0] + lane; p < gp[1]; p += 32) sum += prev[gi[p]] * dp[gi[p]];
                    sum = warp_sum(sum);
                    if (tid == 0) {
                        const F rr = tab.rrow[s0], cr = tab.crow[s0];
                        if (src.x != -1 && rr > F(0)) sum += prev[src.x] * rr;
                        if (src.y != -1 && cr > F(0)) sum += prev[src.y] * cr;
                        lnl += log((double)sum);
                        if (!(sum > F(0))) report_error(d.err, ERR_ZERO_NORM, qi, bi, start);
                        cur[0] = F(1);
                        d.fw64[B.cell0] = 1.0;
                    }
                }
                for (int i = 1 + tid; i < len; i += NTC) d.fw64[B.cell0 + i] = (double)v;
            } else {
                F x = F(1);
                if (!first) {
                    // the single state of the earlier tree: a row or a move
                    const BlockDev &N = d.blocks[sblk];
                    const int t = d.determ[N.prev_state0];
                    if (src.y == 0) x = srcsum[1];
                    else if (src.x == 0) x = srcsum[0];
                    else if (t >= 0) {
                        if constexpr (pairs) {
                            const F2 y = f2_move(F2{prev[t], lastlo[t]}, ((const float2 *)(d.determprob + N.prev_state0))[0].x);
                            x = y.hi;
                        } else {
                            x = tab.dprob[N.prev_state0] * prev[t];
                        }
                    } else x = F(0);
                }
                for (int i = tid; i < len; i += NTC) d.post[B.cell0 + i] = (double)x;
                named_sync(4, NTC);  // lastlo is read
                if (tid == 0) {
                    cur[0] = x;
                    if (pairs) lastlo[0] = 0.0f;
                }
            }
            if (tid == 0) lastexp = Fmt<F>::bias;
            if (!FWD && tid == 0 && !first) lastexp = Fmt<F>::expo(cur[0]);
            for (int i = 0; i < len; i++) passed(FWD ? start + i : start + len - 1 - i);
            continue;
        }

        // ---- the tree's tables
        for (int e = tid; e < NB * MAXT; e += NTC) tmS[e] = tab.tm[(size_t)blk * MAXT * MAXT + e];
        for (int a = tid; a <= MAXT; a += NTC) {
            bptr[a] = d.bt_ptr[(size_t)blk * (MAXT + 1) + a];
            hist[a] = 0;
        }
        for (int p = tid; p < S; p += NTC) rank[d.bt_perm[s0 + p]] = p;
        // the rows as they lie: one wait for memory, where a thread that gathered a state's own
        // entries waited for each
        if (rows_n) {
            const F *const rows = tab.rows + B.t2_0;
            const int M = B.M;
            for (int e0 = tid; e0 < M; e0 += 8 * NTC) {
                F v[8];
#pragma unroll
                for (int x = 0; x < 8; x++) v[x] = e0 + x * NTC < M ? rows[e0 + x * NTC] : F(0);
#pragma unroll
                for (int x = 0; x < 8; x++)
                    if (e0 + x * NTC < M) rowsS[e0 + x * NTC] = v[x];
            }
        }
        named_sync(4, NTC);  // tm, bins, positions, rows, sums
        if (tid == 0) {
            if (FWD) {
                sumk -= ek;
                if (!first && (lastexp == 0 || lastexp == Fmt<F>::top))
                    report_error(d.err, ERR_ZERO_NORM, qi, bi, start - 1);
            }
            lastexp = 0;  // every thread read it before the barrier above
        }
        int plS[NRW + 1], blS[NRW + 1], ckS[NRW], sbS[NRW + 1];
        sbS[0] = 0;
        bin_split(bptr, NB, blS);
#pragma unroll
        for (int r = 0; r <= NRW; r++) plS[r] = bptr[blS[r]];
#pragma unroll
        for (int r = 0; r < NRW; r++) {
            ckS[r] = imax((plS[r + 1] - plS[r] + 31) >> 5, 1);
            sbS[r + 1] = sbS[r] + 32 * ckS[r];
        }
        for (int x = tid; x < sbS[NRW]; x += NTC) head[x] = own[x] = F(0);
        if (SORT) {
            // owners' order: descending by the node's states
            for (int k = tid; k < S; k += NTC) atomicAdd(&hist[MAXT - d.sinfo[s0 + k].m], 1);
            named_sync(4, NTC);  // counts
            if (rw == 0) {
                const int n = hist[lane];
                int incl = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += v;
                }
                __syncwarp();
                hist[lane] = incl - n;
            }
            named_sync(4, NTC);  // starts
            for (int k = tid; k < S; k += NTC) order[atomicAdd(&hist[MAXT - d.sinfo[s0 + k].m], 1)] = k;
        }
        named_sync(4, NTC);  // order, slots cleared

        if (!reducer) {
            // ================= owners
            int ks[KPT], tq[KPT], nb[KPT], cnt[KPT], ro[KPT], slot[KPT], most = 0, rst[KPT];
            bool ok[KPT];   // publishes its state
            F iv[KPT], rs[KPT], e_next[KPT];
            F2 g[KPT];      // FP32: the owned states' published pairs
            int g0[KPT], gn[KPT], gmost = 0;  // forward: the switch's gather list
            F rr[KPT], cr[KPT];               // and breakpoint factors, loaded with the rest
            const int half = SPLIT == 2 ? st & 1 : 0;
#pragma unroll
            for (int q = 0; q < KPT; q++) {
                const int u = SPLIT == 2 ? st >> 1 : st + q * NTS;
                const bool live = u < S;
                const int k = live ? (SORT ? order[u] : u) : 0;
                const StateInfo si = d.sinfo[s0 + k];
                const int off = d.t2off[s0 + k], y = k - si.j1;
                ok[q] = live && half == 0;
                ks[q] = k;
                tq[q] = si.time;
                nb[q] = si.j1 + half;
                cnt[q] = live ? (SPLIT == 2 ? (si.m - half + 1) >> 1 : si.m) : 0;
                // forward: row of target k over its sources; backward: of source k over targets
                ro[q] = FWD ? off + half * si.m : off - y + y * si.m + half;
                rst[q] = FWD ? si.m : 1;
                iv[q] = tab.inv[s0 + k];
                rs[q] = pairs ? (F)tab.rstay[(size_t)blk * MAXT + si.time] : F(0);
                e_next[q] = F(0);
                g[q] = F2{0.0f, 0.0f};
                most = imax(most, cnt[q]);
                g0[q] = gn[q] = 0;
                rr[q] = cr[q] = F(0);
                if (FWD && !first) {
                    const int *gp = d.gptr + B.gptr0 + k;
                    g0[q] = gp[0];
                    gn[q] = ok[q] ? gp[1] - g0[q] : 0;
                    rr[q] = tab.rrow[s0 + k];
                    cr[q] = tab.crow[s0 + k];
                    gmost = imax(gmost, gn[q]);
                }
                // its slot: in the first piece of a chunk, or in the bin's own piece
                const int p = rank[k], b = si.time, bs = bptr[b];
                int r = 0;
#pragma unroll
                for (int x = 1; x < NRW; x++)
                    if (b >= blS[x]) r = x;
                int plo = plS[0], ch = ckS[0], sb = sbS[0], bl = blS[0];
#pragma unroll
                for (int x = 1; x < NRW; x++)
                    if (r == x) {
                        plo = plS[x];
                        ch = ckS[x];
                        sb = sbS[x];
                        bl = blS[x];
                    }
                const int l = (p - plo) / ch, clo = plo + l * ch;
                slot[q] = clo >= bs ? P.head + sb + 32 * (p - clo) + l : P.own + sb + 32 * (p - bs) + (b - bl);
            }
            most = uniform(most);
            gmost = uniform(gmost);
            // the rows' moving parts (FP32: they are that already): an entry belongs to one dot, so
            // its owner forms them, a warp's lanes having rows of like length
            if (rows_n && !pairs) {
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    const int t0 = tq[q] - (ks[q] - (nb[q] - half)) + half;
                    F *r = rowsS + ro[q];
                    const F *tm = tmS + (FWD ? t0 * MAXT + tq[q] : tq[q] * MAXT + t0);
#pragma unroll 4
                    for (int y = 0; y < cnt[q]; y++) {
                        *r = Tab<F>::t2(*r, *tm);
                        r += SPLIT * rst[q];
                        tm += FWD ? SPLIT * MAXT : SPLIT;
                    }
                }
            }
            const F *var = tab.var + B.var0;
            int vr = FWD ? 0 : uniform(B.nvar);  // FWD: the next variant row; else one past it
            auto load_next = [&](int abs) {      // the emissions of column abs, if variant
                if (bit(vm, abs)) {
                    if (!FWD) vr--;
#pragma unroll
                    for (int q = 0; q < KPT; q++) e_next[q] = var[(size_t)vr * S + ks[q]];
                    if (FWD) vr++;
                }
            };
            // FP64: a column's emission, times 2^k
            auto factor = [&](int abs, int q, int k) -> F {
                if constexpr (!pairs) {
                    if (bit(mm, abs)) return Fmt<F>::pow2(k);
                    return Fmt<F>::scaled(bit(vm, abs) ? e_next[q] : iv[q], k);
                } else return F(0);
            };
            // FP32: times the column's emission (complements), times 2^k
            auto emit = [&](int abs, int q, F2 x, int k) -> F2 {
                if constexpr (pairs) {
                    if (bit(vm, abs)) x = e_next[q] >= 0.0f ? f2_keep(x, e_next[q]) : f2_mul(x, -e_next[q]);
                    else if (!bit(mm, abs)) x = f2_keep(x, iv[q]);
                    const float s = Fmt<float>::pow2(k);
                    return F2{x.hi * s, x.lo * s};
                } else return x;
            };
            F x_own[KPT];
#pragma unroll
            for (int q = 0; q < KPT; q++) x_own[q] = F(0);
            // the tree's last column: its largest exponent and (FP32) low parts, for the switch
            auto publish_last = [&]() {
                int E = 0;
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    if (!ok[q]) continue;
                    E = imax(E, Fmt<F>::expo(x_own[q]));
                    if (pairs) lastlo[ks[q]] = g[q].lo;
                }
                E = uniform(E);
                if (lane == 0) atomicMax(&lastexp, E);
            };
            int abs = FWD ? start : start + len - 1;  // the column being formed
            F *const outf = FWD ? (F *)d.fw64 + B.cell0 : nullptr;
            double *const outb = FWD ? nullptr : d.post + B.cell0;

            // ---- the tree's first column in the chain's direction
            load_next(abs);
            if (FWD && first) {
#pragma unroll
                for (int q = 0; q < KPT; q++)
                    if (ok[q]) cur[ks[q]] = base_f[slot[q]] = x_own[q] = outf[ks[q]];  // priors (K1)
            } else {
                F sums[KPT];
                if constexpr (FWD) {
                    const int *gi = d.gidx + B.prev_state0;
                    const F *dp = tab.dprob + B.prev_state0;
#pragma unroll
                    for (int q = 0; q < KPT; q++) sums[q] = F(0);
                    for (int t = 0; t < gmost; t += 2) {  // two sources of each state at a time
                        int j[KPT][2];
                        F p[KPT][2];
#pragma unroll
                        for (int q = 0; q < KPT; q++)
#pragma unroll
                            for (int x = 0; x < 2; x++) j[q][x] = t + x < gn[q] ? gi[g0[q] + t + x] : 0;
#pragma unroll
                        for (int q = 0; q < KPT; q++)
#pragma unroll
                            for (int x = 0; x < 2; x++) p[q][x] = t + x < gn[q] ? dp[j[q][x]] : F(0);
#pragma unroll
                        for (int q = 0; q < KPT; q++)
#pragma unroll
                            for (int x = 0; x < 2; x++)
                                if (t + x < gn[q]) sums[q] = fma(prev[j[q][x]], p[q][x], sums[q]);
                    }
                }
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    if (!ok[q]) continue;
                    const int k = ks[q];
                    if constexpr (FWD) {
                        F s = sums[q];
                        if (src.x != -1 && rr[q] > F(0)) s += prev[src.x] * rr[q];
                        if (src.y != -1 && cr[q] > F(0)) s += prev[src.y] * cr[q];
                        s = s * Fmt<F>::pow2(ek) * factor(abs, q, 0);
                        outf[k] = s;
                        cur[k] = base_f[slot[q]] = x_own[q] = s;
                    } else {
                        F x = F(1) / F(S);
                        float xlo = 0.0f;
                        if (!first) {
                            const long long p0 = d.blocks[sblk].prev_state0;
                            const int t = d.determ[p0 + k];
                            x = F(0);
                            if (k == src.y) x = srcsum[1];
                            else if (k == src.x) x = srcsum[0];
                            else if (t >= 0) {
                                if constexpr (pairs) {
                                    const F2 y = f2_move(F2{prev[t], lastlo[t]}, ((const float2 *)(d.determprob + p0))[k].x);
                                    x = y.hi;
                                    xlo = y.lo;
                                } else {
                                    x = tab.dprob[p0 + k] * prev[t];
                                }
                            }
                        }
                        outb[(size_t)(len - 1) * S + k] = (double)x;
                        if constexpr (pairs) {
                            g[q] = emit(abs, q, F2{x, xlo}, ek);
                            cur[k] = base_f[slot[q]] = x_own[q] = g[q].hi;
                        } else {
                            cur[k] = base_f[slot[q]] = x_own[q] = x * factor(abs, q, ek);
                        }
                    }
                }
            }
            passed(abs);
            const int step = FWD ? 1 : -1;
            if (len > 1) load_next(abs + step);
            if (len == 1) {
                // other owners may still read the later tree's low parts for their first column
                // (a longer tree has its columns' barriers in between)
                if (pairs) named_sync(3, NTS);
                publish_last();
            }
            Scale<F> sc;
            for (int n = 1; n < len; n++) {
                abs += step;
                const int i = abs - start;
                named_sync(1, NTC);  // A: the column before is complete
                // same-branch dots, even and odd terms
                F de[KPT], dd[KPT];
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    de[q] = dd[q] = F(0);
                    const F *x = cur + nb[q];
                    if (rows_n) {
                        const F *r = rowsS + ro[q];
                        const int rs1 = rst[q];
                        if (SPLIT == 2) {
#pragma unroll 4
                            for (int y = 0; y < most; y++) {
                                const F v = y < cnt[q] ? *r : F(0);
                                de[q] = fma(v, x[2 * y], de[q]);
                                r += 2 * rs1;
                            }
                        } else {
#pragma unroll 2
                            for (int y = 0; y < most; y += 2) {
                                const F v0 = y < cnt[q] ? r[0] : F(0), v1 = y + 1 < cnt[q] ? r[rs1] : F(0);
                                de[q] = fma(v0, x[y], de[q]);
                                dd[q] = fma(v1, x[y + 1], dd[q]);
                                r += 2 * rs1;
                            }
                        }
                    } else {
                        // rows in global memory: the same terms in the same order (a lane of
                        // a pair takes every second one)
                        const int a0 = tq[q] - (ks[q] - nb[q]);
                        const F *r = tab.rows + B.t2_0 + ro[q];
                        for (int y = 0; y < cnt[q]; y++) {
                            const int z = SPLIT * y;
                            const F tmab = FWD ? tmS[(a0 + z) * MAXT + tq[q]] : tmS[tq[q] * MAXT + a0 + z];
                            const F v = Tab<F>::t2(r[(size_t)z * rst[q]], tmab);
                            if (SPLIT == 1 && (y & 1)) dd[q] = fma(v, x[z], dd[q]);
                            else de[q] = fma(v, x[z], de[q]);
                        }
                    }
                }
                if (SPLIT == 2) dd[0] = __shfl_xor_sync(FULL, de[0], 1);
                // the power of two is the one that the last column's bins asked for: the factor is
                // there before B, and the inflow is one fused product behind it
                F fac[KPT];
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    de[q] += dd[q];
                    fac[q] = factor(abs, q, sc.k);
                    if constexpr (FWD) de[q] *= fac[q];
                }
                named_sync(2, NTC);  // B: the column's moves between times, its exponents
                const int E = imax(imax(expoS[0], expoS[1]), imax(expoS[2], expoS[3]));
                sc.see(E);
                if (!pairs && sc.extra) {  // rare
                    // (forward: on the values, as a given prior's may be too large for the factor)
                    const F x = Fmt<F>::pow2(sc.extra);
#pragma unroll
                    for (int q = 0; q < KPT; q++) {
                        if constexpr (FWD) {
                            de[q] = fma(tfS[tq[q]] * x, fac[q], de[q] * x);
                            fac[q] = F(0);
                        } else {
                            fac[q] *= x;
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    const size_t at = (size_t)i * S + ks[q];
                    const F in = FWD ? F(0) : tfS[tq[q]] + de[q];
                    if constexpr (FWD) {
                        const F v = fma(tfS[tq[q]], fac[q], de[q]);
                        if (ok[q]) {
                            cur[ks[q]] = base_f[slot[q]] = v;
                            outf[at] = v;
                        }
                        x_own[q] = v;
                    } else if constexpr (pairs) {
                        const F2 x = f2_add(f2_keep(g[q], rs[q]), in);
                        g[q] = emit(abs, q, x, sc.used());
                        if (ok[q]) {
                            cur[ks[q]] = base_f[slot[q]] = g[q].hi;
                            outb[at] = (double)x.hi;
                        }
                        x_own[q] = g[q].hi;
                    } else {
                        const F v = in * fac[q];
                        if (ok[q]) {
                            cur[ks[q]] = base_f[slot[q]] = v;
                            outb[at] = (double)in;
                        }
                        x_own[q] = v;
                    }
                }
                sc.next(E);
                passed(abs);
                if (n + 1 < len) load_next(abs + step);
                else publish_last();
            }
        } else {
            // ================= reducers
            int plo = plS[0], phi = plS[1], chunk = ckS[0], sb = sbS[0], blo = blS[0], bhi = blS[1];
#pragma unroll
            for (int x = 1; x < NRW; x++)
                if (rw == x) {
                    plo = plS[x];
                    phi = plS[x + 1];
                    chunk = ckS[x];
                    sb = sbS[x];
                    blo = blS[x];
                    bhi = blS[x + 1];
                }
            chunk = uniform(chunk);
            // the bin that the lane's chunk begins in: its lanes from seg0 on; lane b - blo: the
            // chunks lh .. lh + nh - 1 begin inside bin b
            const int clo = imin(plo + lane * chunk, phi);
            int hb = blo;
            while (hb < bhi - 1 && bptr[hb + 1] <= clo) hb++;
            const int seg0 = blo < bhi ? (bptr[hb] - plo + chunk - 1) / chunk : 0;
            int lh = 0, nh = 0, no = 0;
            const int mb = blo + lane;
            if (mb < bhi && bptr[mb + 1] > bptr[mb]) {
                lh = (bptr[mb] - plo + chunk - 1) / chunk;
                nh = (bptr[mb + 1] - 1 - plo) / chunk - lh + 1;
                no = imin(imin(plo + lh * chunk, bptr[mb + 1]) - bptr[mb], chunk);  // its own piece's positions
            }
            const int nhmax = uniform(nh), nomax = uniform(no);
            const F *const hs = head + sb + lane, *const os = own + sb + lane;
            // outputs a = oi of this warp's share, in `parts` parts of the bins
            const int o = (NB + NRW - 1) / NRW, parts = 32 / o, part = lane / o, oi = rw * o + lane % o;
            const bool outlane = part < parts && oi < NB;
            const int terms = (NB + parts - 1) / parts;
            F tmr[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int b = part + parts * t;
                tmr[t] = outlane && t < terms && b < NB ? (FWD ? tmS[b * MAXT + oi] : tmS[oi * MAXT + b]) : F(0);
            }
            Scale<F> sc;
            for (int n = 1; n < len; n++) {
                named_sync(1, NTC);  // A
                F h = hs[0], ow = F(0);
                for (int j = 1; j < chunk; j++) h += hs[32 * j];
                if (nomax) {
                    ow = os[0];
                    for (int j = 1; j < nomax; j++) ow += os[32 * j];
                }
                // running sums of a bin's chunks over its lanes
                for (int x = 1; x < nhmax; x <<= 1) {
                    const F v = __shfl_up_sync(FULL, h, x);
                    if (lane - x >= seg0) h += v;
                }
                const F t = __shfl_sync(FULL, h, (lh + nh - 1) & 31);
                F bin = nh > 0 ? t : F(0);
                if (nomax) bin = ow + bin;
                if (mb < bhi) binS[mb] = bin;
                const int E = (int)__reduce_max_sync(FULL, (unsigned)(mb < bhi ? Fmt<F>::expo(bin) : 0));
                if (lane == 0) expoS[rw] = E;
                named_sync(5, 32 * NRW);  // C: the bins
                F sum = F(0);
#pragma unroll
                for (int t2 = 0; t2 < 8; t2++)
                    if (t2 < terms) {
                        const int b = part + parts * t2;
                        const F x = b < NB ? binS[b] : F(0);
                        sum = t2 == 0 ? tmr[0] * x : fma(tmr[t2], x, sum);
                    }
                for (int wn = parts; wn > 1;) {
                    const int hf = (wn + 1) >> 1;
                    const F v = __shfl_down_sync(FULL, sum, hf * o);
                    if (part + hf < wn) sum += v;
                    wn = hf;
                }
                if (part == 0 && oi < NB) tfS[oi] = sum;
                named_sync(2, NTC);  // B
                if (FWD && tid == 0) {
                    const int Em = imax(imax(expoS[0], expoS[1]), imax(expoS[2], expoS[3]));
                    if (Em == 0 || Em == Fmt<F>::top) report_error(d.err, ERR_ZERO_NORM, qi, bi, start + n - 1);
                    sc.see(Em);
                    sumk -= sc.used();
                    sc.next(Em);
                }
            }
        }
    }
    if constexpr (FWD) {
        named_sync(4, NTC);
        if (rw == 0 && d.lnl) {
            const int Sl = imax(d.blocks[I.block0 + I.ntrees - 1].S, 1);
            const F *x = col + c * cs;
            F s = F(0);
            for (int k = lane; k < Sl; k += 32) s += x[k];
            s = warp_sum(s);
            if (lane == 0) {
                if (!(s > F(0))) report_error(d.err, ERR_ZERO_NORM, qi, I.ntrees - 1, L - 1);
                d.lnl[qi] = log((double)s) + (double)sumk * 0.69314718055994530942 + lnl;
            }
        }
    }
}

__host__ __device__ inline int owner_threads(int units, int kpt) {
    return imax(32, ((units + kpt - 1) / kpt + 31) / 32 * 32);
}

// One CTA per instance, each in the form of its own largest tree (surplus warps leave at once):
// FP64 up to OWNERS / 2 states two lanes a state, then one, two, four or eight states a thread.
template <typename F, bool FWD>
__global__ void __launch_bounds__(32 * NRW + OWNERS) k_chain(BatchDev d, int rows_n) {
    __shared__ Shared<F> sh;
    const int qi = cta_instance(d);
    const InstDev I = d.inst[qi];
    const int S = I.maxS;
    const bool split = sizeof(F) == 8 && 2 * S <= OWNERS;
    const int kpt = S <= OWNERS ? 1 : S <= 2 * OWNERS ? 2 : S <= 4 * OWNERS ? 4 : 8;
    const int ntc = 32 * NRW + owner_threads(split ? 2 * S : S, kpt);
    if ((int)threadIdx.x >= ntc) return;
    if constexpr (sizeof(F) == 8) {
        if (split) {
            run_chain<F, FWD, 1, 2>(d, I, qi, rows_n, ntc, sh);
            return;
        }
    }
    if (kpt == 1) run_chain<F, FWD, 1, 1>(d, I, qi, rows_n, ntc, sh);
    else if (kpt == 2) run_chain<F, FWD, 2, 1>(d, I, qi, rows_n, ntc, sh);
    else if (kpt == 4) run_chain<F, FWD, 4, 1>(d, I, qi, rows_n, ntc, sh);
    else run_chain<F, FWD, 8, 1>(d, I, qi, rows_n, ntc, sh);
}

// The FP64 forward table, each column divided by its sum (the instance's column 0 keeps the
// prior, as the reference's table does); a CTA per tree and share of its columns.
__global__ void __launch_bounds__(128) k_normalise(BatchDev d) {
    const BlockDev &B = d.blocks[cta_block(d)];
    const int S = B.S, lane = threadIdx.x & 31, nw = gridDim.y * 4;
    if (S == 0) return;
    for (int i = blockIdx.y * 4 + (threadIdx.x >> 5); i < B.len; i += nw) {
        if (B.b == 0 && i == 0) continue;
        double *x = d.fw64 + B.cell0 + (size_t)i * S, s = 0.0;
        for (int k = lane; k < S; k += 32) s += x[k];
        s = warp_sum(s);
        for (int k = lane; k < S; k += 32) x[k] /= s;
    }
}

// Posterior marginals fw bw / sum from the columns' forward and backward values (each on a
// scale of its own), in place of the latter; bw_out: those normalised, where it is wanted.
template <typename F>
__global__ void __launch_bounds__(128) k_posterior(BatchDev d, double *bw_out) {
    const BlockDev &B = d.blocks[cta_block(d)];
    const int S = imax(B.S, 1), lane = threadIdx.x & 31, nw = gridDim.y * 4;
    const F *fw = sizeof(F) == 4 ? (const F *)d.fw32 : (const F *)d.fw64;
    for (int i = blockIdx.y * 4 + (threadIdx.x >> 5); i < B.len; i += nw) {
        const long long c0 = B.cell0 + (long long)i * S;
        const F *f = fw + c0;
        double *b = d.post + c0;
        F z = F(0), sb = F(0);
        for (int k = lane; k < S; k += 32) {
            const F x = (F)b[k];
            z += f[k] * x;
            sb += x;
        }
        z = warp_sum(z);
        if (bw_out) sb = warp_sum(sb);
        for (int k = lane; k < S; k += 32) {
            const F x = (F)b[k];
            if (bw_out) bw_out[c0 + k] = (double)(x / sb);
            b[k] = (double)(f[k] * x / z);
        }
    }
}

// Columns' shares of a tree for the table kernels: enough CTAs for a few trees too.
int column_shares(const BatchDev &d) { return imin(64, imax(1, 4096 / imax(1, d.nblocks))); }

template <typename F, bool FWD>
bool launch(const BatchDev &d, cudaStream_t s) {
    const int maxS = imax(d.maxS, 1);
    if (maxS > 8 * OWNERS) return false;
    // the tree's same-branch rows in shared memory where they fit
    constexpr size_t LIMIT = 200 * 1024;  // beside the kernel's static shared memory
    int rows_n = imax(d.maxM, 1);
    if (SmemPlan<F>(maxS, rows_n).bytes > LIMIT) rows_n = 0;
    const size_t smem = SmemPlan<F>(maxS, rows_n).bytes;
    if (!raise_dynamic_smem(k_chain<F, FWD>, smem)) return true;  // the launch reports it
    // smaller instances of the batch may need more threads than its largest: two lanes a state
    const int units = sizeof(F) == 8 ? imin(OWNERS, 2 * maxS) : imin(OWNERS, maxS);
    k_chain<F, FWD><<<d.ninst, 32 * NRW + owner_threads(units, 1), smem, s>>>(d, rows_n);
    note_launch();
    return true;
}

}  // namespace

bool launch_forward64(const BatchDev &d, cudaStream_t s) { return launch<double, true>(d, s); }

void launch_normalise(const BatchDev &d, cudaStream_t s) {
    if (imax(d.maxS, 1) > 8 * OWNERS) return;  // the general kernel's columns are already
    k_normalise<<<dim3(d.nblocks, column_shares(d)), 128, 0, s>>>(d);
    note_launch();
}

bool launch_backward_chain(const BatchDev &d, bool fp32, cudaStream_t s) {
    return fp32 ? launch<float, false>(d, s) : launch<double, false>(d, s);
}

void launch_posterior(const BatchDev &d, bool fp32, double *bw_out, cudaStream_t s) {
    const dim3 grid(d.nblocks, column_shares(d));
    if (fp32) k_posterior<float><<<grid, 128, 0, s>>>(d, bw_out);
    else k_posterior<double><<<grid, 128, 0, s>>>(d, bw_out);
    note_launch();
}

}  // namespace awg
