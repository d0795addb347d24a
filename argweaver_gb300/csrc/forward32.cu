// K3, FP32 path: the forward pass of the threading HMM, one CTA per instance.
//
// Per column (arghmm_forward_block, sample_thread.cpp:252-295), with the FP32 path's
// complements (tables rounded once from FP64; see forward.cu's FP64 kernel for the plain
// form):
//   bin[a]  = sum of the previous column's states of time a
//   tf[b]   = sum_a tm[a][b] bin[a]
//   x_k     = ((1 - rstay[b]) x_k + sum_y t2[y][k] x_{j1 + y} + tf[b]) e_k / norm
// The stay, emission and rescaling factors, which carry almost all of a state's mass, run
// on FP32 pairs (value = hi + lo); the mass moving in from other states stays plain FP32.
//
// What bounds it: an instance's columns are one dependent chain, so its time is columns
// times one column's latency; DRAM, the FP32 pipes and shared memory are all far from their
// limits. Everything here shortens that chain.
//   - Four reduction warps and the owner warps (KPT states a thread, k = t + q * owners).
//     Two barriers a column: after A (column i-1 complete) the reduction warps form the
//     bins and their shares of tf while the owners form their same-branch dots; after B the
//     owners finish column i.
//   - A reduction warp's positions of the time-sorted column are cut into 32 chunks, one a
//     lane, and a chunk into pieces by time bin. They lie transposed in shared memory as
//     float2 slots: .x the piece that a lane's chunk begins with, .y the piece a bin begins
//     with inside a chunk, kept by the bin's own lane; unused slots hold zeros. So a lane's
//     sums are a few packed adds without masks or branches, and a bin is its own piece plus
//     the following chunks' first ones, gathered by shuffles.
//   - Two states of an owner thread share packed FP32 instructions (add / mul / fma .f32x2,
//     each half rounded as the scalar operation): the finish is issue-bound at 500 states.
//   - The owners hold their same-branch rows in registers (ROWS entries, zeros past a node's
//     states), and a node's states lie on 16 bytes in shared memory: four terms cost one
//     shared load and two packed FMAs.
//   - A tree's tables (state info, rows, gather lists, ...) arrive by bulk copies that the
//     last reduction warp (whose bins hold the fewest states) issues as soon as the tree
//     before has taken its own out of the buffer;
//     column classes are loaded a window ahead and emission rows EDEPTH columns ahead
//     (cp.async), so nothing in the chain waits for memory.
//   - The log-likelihood is a running FP64 product with its exponent split off by integer
//     operations, 32 columns' norms at a time, one a lane; one log per lane and instance.
// Every sum has an order fixed by the tree alone, so results do not depend on the block size
// or on the other problems of the batch.

#include <cuda_runtime.h>

#include <cstdlib>

#include "async_copy.cuh"
#include "f2.cuh"
#include "forward32_plan.h"
#include "kernels.h"

namespace awg {

namespace {

using namespace fwd32;

constexpr int RBINS = (MAXT - 1 + NRW - 1) / NRW;  // time bins per reduction warp (<= 8)
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void named_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void cp_async4(float *smem, const float *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// All of `threads` threads have arrived; whether any of them has v set.
__device__ __forceinline__ bool named_or(int id, int threads, bool v) {
    unsigned r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %3, 0;\n bar.red.or.pred q, %1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"(id), "r"(threads), "r"((unsigned)v)
        : "memory");
    return r != 0;
}

// A warp-wide equal value (>= 0) in a uniform register: branches on it need no reconvergence.
__device__ __forceinline__ int uniform(int v) { return (int)__reduce_max_sync(FULL, (unsigned)v); }

// Two FP32 values in one packed operand.
struct V2 {
    unsigned long long v;
};
__device__ __forceinline__ V2 pk(float a, float b) {
    V2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo(V2 a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float hi(V2 a) { return __uint_as_float((unsigned)(a.v >> 32)); }
__device__ __forceinline__ V2 operator+(V2 a, V2 b) {
    V2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 operator-(V2 a, V2 b) {
    V2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 fma2(V2 a, V2 b, V2 c) {
    V2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// f2.cuh's pair steps for two states at once: the same operations, each rounded alike.
struct P2 {
    V2 hi, lo;
};
__device__ __forceinline__ P2 p2_renorm(V2 a, V2 b) {
    const V2 s = a + b;
    return P2{s, b - (s - a)};
}
// Products are taken as fmas with nz = -0 (exact: a b + -0 = a b), a kernel argument: the
// compiler fuses a packed mul, or an fma with a -0 that it knows, with an add behind it, which
// would round once where f2.cuh rounds twice.
__device__ __forceinline__ P2 p2_keep(P2 x, V2 r, V2 nz) {
    const V2 t = fma2(x.hi, r, nz);
    const V2 h = x.hi - t;
    return p2_renorm(h, ((x.hi - h) - t) + x.lo);
}
__device__ __forceinline__ P2 p2_mul(P2 x, V2 e, V2 nz) {
    const V2 p = fma2(x.hi, e, nz);
    return p2_renorm(p, fma2(x.hi, e, V2{p.v ^ 0x8000000080000000ull}) + fma2(x.lo, e, nz));
}
__device__ __forceinline__ P2 p2_add(P2 x, V2 s) {
    const V2 h = x.hi + s;
    const V2 bb = h - x.hi;
    const V2 err = (x.hi - (h - bb)) + (s - bb);
    return p2_renorm(h, err + x.lo);
}

// sum of log(norm) as an FP64 mantissa product in [1, 2) and an integer exponent
struct LogProd {
    double prod = 1.0;
    long long e = 0;
    __device__ void mul(double v) {
        prod *= v;
        const int hi = __double2hiint(prod);
        const int ex = (hi >> 20) & 0x7ff;
        if (ex > 0 && ex < 0x7ff) {  // normal: move the exponent out
            e += ex - 1023;
            prod = __hiloint2double((hi & 0x800fffff) | (1023 << 20), __double2loint(prod));
        }
    }
    __device__ double value() const { return log(prod) + (double)e * 0.69314718055994530942; }
};

// a number as a type, for lambdas over unrolled lengths
template <int N>
struct Int {
    static constexpr int value = N;
};

// One instance. KPT states per owner thread; of their same-branch rows the first ROWS0 entries
// (a thread's first state) and ROWS (its others) in registers. TAIL: rows may be longer than
// that; the rest is read from shared memory, or from global memory where the rows do not fit.
// SORT: the owners take the states in descending order of their node's, so that a warp's dots
// are of like length, and past a thread's first state mostly short. STAGED: per-state tables staged a tree ahead
// (else read from global memory). NTC: the threads at work, reducers and owners.
template <int KPT, int ROWS0, int ROWS, bool TAIL, bool STAGED, bool SORT>
__device__ __forceinline__ void forward32(const BatchDev &d, const InstDev &I, int qi, int t2_bufs, int NTC, V2 nz) {
    extern __shared__ __align__(16) unsigned char dyn_b[];
    constexpr int NP = (KPT + 1) / 2;      // packed pairs of states
    // rows' ends, past the registers: stepped through by pointers, two states side by side where
    // a thread has four or eight, for more than 21 time points (rows of up to 31 entries) and for
    // eight states a thread (four registers a row). A column of 1,243 states with rows of 29
    // entries takes 3.7 us so and 4.9 one after another, of 2,520 with 12 5.7 and 9.2; with the
    // shorter rows of up to 21 points (1,442 states of 7) 2.6 and 2.1.
    constexpr bool LONG_ENDS = SORT || KPT == 8;
    const int maxS = I.maxS;
    const int NB = I.T - 1;
    const int tid = threadIdx.x, lane = tid & 31, rw = tid >> 5;
    const int NTS = NTC - 32 * NRW;        // owner threads
    const int st = tid - 32 * NRW;
    const bool reducer = tid < 32 * NRW, owner = !reducer, producer = tid == 32 * (NRW - 1);
    const StageLayout SL(maxS);
    const SmemPlan P(Sizes{maxS, I.maxM, I.nnodes}, t2_bufs, STAGED);
    unsigned char *const stage = dyn_b + P.stage;
    float *const t2buf = (float *)(dyn_b + P.t2);
    const int colstride = (P.red - P.col) / 8;
    // [2][colstride] columns in state order, the states of node v from (j1 + 3 v) & ~3 on (the
    // next node's start is past the last state of this one's)
    float *const col = (float *)(dyn_b + P.col);
    float *const red = (float *)(dyn_b + P.red);   // newest column, reducers' float2 slots
    float *const ring = (float *)(dyn_b + P.ring); // [EDEPTH + 1][ringstride] emission rows
    const int ringstride = (maxS + 3) & ~3;
    int *const rank = (int *)(col + colstride);    // time-sorted position of each state (until T2)
    float2 *const last = (float2 *)(dyn_b + P.last);  // a tree's last column, high and low parts
    __shared__ __align__(16) float tfp[32][NRW];   // [a][reducer] shares of tf; [31]: of the norm
    __shared__ uint64_t full;                      // the staged tree has landed
    __shared__ uint64_t rows_full;                 // the tree's rows have (unstaged forms)
    __shared__ int by_m[MAXT];                     // states by their node's, then where they begin
    __shared__ double lnl0;

    if (tid == 0) {
        mbar_init(&full, 1);
        mbar_init(&rows_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // rows read past a node's states, times 0: finite
    for (int k = tid; k < 2 * colstride; k += NTC) col[k] = 0.0f;
    named_sync(4, NTC);

    // ---- producer: one lane issues the copies of a tree (descriptor B) and of the descriptor
    // of the tree after it
    auto desc_of = [&](int b) { return (BlockDev *)(stage + SL.desc) + b % 3; };
    auto issue = [&](int blk, const BlockDev &B) {
        const bool more = B.b + 1 < I.ntrees;
        const int S = B.S, S1 = imax(B.S1, 1);
        const bool sw = B.b > 0 && S > 0;
        const Rounded<4> rb(d.bt_ptr + (size_t)blk * (MAXT + 1), MAXT + 1);
        const Rounded<4> ro(d.t2off + B.state0, S), rp(d.bt_perm + B.state0, S), ri(d.inv32 + B.state0, S);
        const Rounded<4> rg(d.gptr + B.gptr0, S + 1), rx(d.gidx + B.prev_state0, S1);
        const Rounded<8> rd(d.determprob + B.prev_state0, S1);
        const Rounded<4> rr(d.recombrow32 + B.state0, S), rc(d.recoalrow32 + B.state0, S);
        const Rounded<8> rs(d.srcs + blk, 1);
        const Rounded<4> r2(d.t2d32 + B.t2_0, B.M);
        const unsigned tmb = 4u * MAXT * (unsigned)NB;
        unsigned tx = more ? sizeof(BlockDev) : 0u;
        if (S > 0) tx += tmb + 4 * MAXT + rb.bytes;
        if (S > 0 && STAGED) tx += 16u * S + ro.bytes + rp.bytes + ri.bytes + r2.bytes;
        if (sw && STAGED) tx += rg.bytes + rx.bytes + rd.bytes + rr.bytes + rc.bytes + 16;
        mbar_expect_tx(&full, tx);
        if (more) bulk_g2s(desc_of(B.b + 1), d.blocks + blk + 1, sizeof(BlockDev), &full);
        if (S > 0) {
            bulk_g2s(stage + SL.bptr, rb.a16, rb.bytes, &full);
            bulk_g2s(stage + SL.tm, d.tm32 + (size_t)blk * MAXT * MAXT, tmb, &full);
            bulk_g2s(stage + SL.rstay, d.rstay32 + (size_t)blk * MAXT, 4 * MAXT, &full);
        }
        if (S > 0 && STAGED) {
            // rows still read by the tree before sit in the other buffer
            unsigned char *rows = dyn_b + P.t2 + (TAIL ? (B.b & 1) * P.t2_bytes : 0);
            bulk_g2s(stage + SL.sinfo, d.sinfo + B.state0, 16u * S, &full);
            bulk_g2s(stage + SL.t2off, ro.a16, ro.bytes, &full);
            bulk_g2s(rows, r2.a16, r2.bytes, &full);
            bulk_g2s(stage + SL.perm, rp.a16, rp.bytes, &full);
            bulk_g2s(stage + SL.inv, ri.a16, ri.bytes, &full);
        }
        if (sw && STAGED) {
            bulk_g2s(stage + SL.gptr, rg.a16, rg.bytes, &full);
            bulk_g2s(stage + SL.gidx, rx.a16, rx.bytes, &full);
            bulk_g2s(stage + SL.move, rd.a16, rd.bytes, &full);
            bulk_g2s(stage + SL.rrow, rr.a16, rr.bytes, &full);
            bulk_g2s(stage + SL.crow, rc.a16, rc.bytes, &full);
            bulk_g2s(stage + SL.src, rs.a16, 16, &full);
        }
    };
    // a per-state table where it was staged, or in global memory
    auto table = [&](const auto *g, int at) {
        using E = decltype(g);
        if constexpr (STAGED) return (E)(stage + at) + ((uintptr_t)g & 15) / sizeof(*g);
        else return g;
    };

    // the log-likelihood accumulates in reduction warp 1, which has little else to do between
    // barriers B and A: lane l keeps the norm of every 32nd column until 32 are there
    LogProd acc, acc0;
    double extra = 0.0;
    float mynorm = 1.0f;
    int ncols = 0;
    unsigned phase = 0, rows_phase = 0;
    bool failed = false, rows_late = false;

    // ---- owners: the coming tree's classes (lane l: columns l and 32 + l), loaded a tree
    // ahead; columns past the instance read as invariant
    const uint8_t *const cls = d.colclass + I.col0;
    auto class_at = [&](int abs_col) { return abs_col < I.seqlen ? (int)cls[abs_col] : 0; };
    int cw0 = 0, cw1 = 0;
    if (owner) {
        cw0 = class_at(lane);
        cw1 = class_at(32 + lane);
    }
    // the emission rows of a tree's first columns (classes in cw0): column i <= EDEPTH, slot i
    auto first_rows = [&](long long var0, int S, int len) {
        const float *row = d.var32 + var0;
        unsigned todo = __ballot_sync(FULL, cw0 == COL_VARIANT && lane <= EDEPTH && lane < len);
        for (; todo; todo &= todo - 1, row += S) {
            float *slot = ring + (__ffs(todo) - 1) * ringstride;
#pragma unroll
            for (int q = 0; q < KPT; q++)
                if (st + q * NTS < S) cp_async4(slot + st + q * NTS, row + st + q * NTS);
        }
#pragma unroll
        for (int i = 0; i < EDEPTH; i++) cp_commit();  // all in the first group
    };
    if (owner) first_rows(d.blocks[I.block0].var0, d.blocks[I.block0].S, d.blocks[I.block0].len);
    if (producer) {
        *desc_of(0) = d.blocks[I.block0];
        issue(I.block0, *desc_of(0));
    }

    for (int bi = 0; bi < I.ntrees; bi++) {
        const int blk = I.block0 + bi;
        const bool landed = mbar_wait(&full, phase);
        phase ^= 1u;
        // T1: the last tree's column is final, the staged tree has landed
        if (named_or(4, NTC, !landed || rows_late)) {
            failed = true;
            break;
        }
        const BlockDev *Bs = desc_of(bi);
        if (TAIL && !STAGED && producer && t2_bufs && Bs->S > 0) {
            // the last tree's rows are read: this one's by bulk copy (loaded and stored by the
            // owners, 49,000 cycles of a tree with 30,000 entries went there)
            const Rounded<4> r2(d.t2d32 + Bs->t2_0, Bs->M);
            mbar_expect_tx(&rows_full, r2.bytes);
            bulk_g2s(t2buf, r2.a16, r2.bytes, &rows_full);
        }
        const int S = uniform(Bs->S), len = uniform(Bs->len), start = uniform(Bs->start);
        float *const fw = d.fw32 + Bs->cell0;

        if (S == 0) {
            // fully specified tree: one state that carries over (sample_thread.cpp:201-206)
            float v = 1.0f;
            if (bi == 0) {
                v = fw[0];
                if (tid == 0) last[0] = make_float2(v, 0.0f);
            } else if (tid < 32) {
                const BlockDev &B = d.blocks[blk];
                const int2 src = d.srcs[blk];
                const int *gp = d.gptr + B.gptr0;
                const int *gi = d.gidx + B.prev_state0;
                const float *dp = d.determprob32 + B.prev_state0;
                const float *rr = d.recombrow32 + B.state0;
                const float *cr = d.recoalrow32 + B.state0;
                float sum = 0.0f;
                for (int p = gp[0] + lane; p < gp[1]; p += 32) sum += last[gi[p]].x * dp[gi[p]];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
                if (tid == 0) {
                    if (src.x != -1 && rr[0] > 0.0f) sum += last[src.x].x * rr[0];
                    if (src.y != -1 && cr[0] > 0.0f) sum += last[src.y].x * cr[0];
                    acc0.mul((double)sum);
                    last[0] = make_float2(1.0f, 0.0f);
                    fw[0] = 1.0f;
                }
            }
            for (int i = 1 + tid; i < len; i += NTC) fw[i] = v;
            if (owner) {
                cw0 = class_at(start + len + lane);
                cw1 = class_at(start + len + 32 + lane);
                if (bi + 1 < I.ntrees) first_rows(d.blocks[blk + 1].var0, d.blocks[blk + 1].S, d.blocks[blk + 1].len);
            }
            if (producer && bi + 1 < I.ntrees) issue(blk + 1, *desc_of(bi + 1));
            continue;
        }

        // time-sorted positions of the reducers: warp r has [pl[r], pl[r+1]), a lane a chunk of
        // ck[r] of them; its slots start at sb[r], 32 of them for each of a lane's positions
        // (rounded up to 1, 2, 4 or a multiple of 8, the lengths the sums are unrolled for)
        const int *bptr = (const int *)(stage + SL.bptr) + ((uintptr_t)(d.bt_ptr + (size_t)blk * (MAXT + 1)) & 15) / 4;
        int pl[NRW + 1], ck[NRW], cu[NRW], sb[NRW + 1];
        pl[0] = sb[0] = 0;
#pragma unroll
        for (int r = 0; r < NRW; r++) {
            pl[r + 1] = uniform(bptr[(r + 1) * NB / NRW]);
            ck[r] = imax((pl[r + 1] - pl[r] + 31) >> 5, 1);
            cu[r] = ck[r] <= 2 ? ck[r] : ck[r] <= 4 ? 4 : (ck[r] + 7) & ~7;
            sb[r + 1] = sb[r] + 32 * cu[r];
        }

        if (owner) {
            // ================= owners
            int cur = 0;  // the current column's buffer
            const long long s0 = Bs->state0, p0 = Bs->prev_state0;
            const StateInfo *sinfo = table(d.sinfo + s0, SL.sinfo);
            const int *t2off = table(d.t2off + s0, SL.t2off);
            const int *perm = table(d.bt_perm + s0, SL.perm);
            const float *inv = table(d.inv32 + s0, SL.inv);
            const float *rsv = (const float *)(stage + SL.rstay);
            const float *rows = d.t2d32 + Bs->t2_0;
            if constexpr (STAGED) {
                rows = (const float *)(dyn_b + P.t2 + (TAIL ? (bi & 1) * P.t2_bytes : 0)) + ((uintptr_t)rows & 15) / 4;
            }
            // classes: bit j of vm / mm: column i + j is variant / masked (i = 0 here)
            unsigned long long vm = (unsigned long long)__ballot_sync(FULL, cw1 == COL_VARIANT) << 32 |
                                    __ballot_sync(FULL, cw0 == COL_VARIANT);
            unsigned long long mm = (unsigned long long)__ballot_sync(FULL, cw1 == COL_MASKED) << 32 |
                                    __ballot_sync(FULL, cw0 == COL_MASKED);
            // time-sorted position of each state
            for (int p = st; p < S; p += NTS) rank[perm[p]] = p;
            bool ok[KPT];
            int ks[KPT], nbo[KPT], pos[KPT], m[KPT], roff[KPT], tq[KPT], slot[KPT], most = 0, mostq[KPT];
            V2 rs[NP], iv[NP], xh[NP], xl[NP];
            V2 row0[ROWS0 / 2], row[KPT > 1 ? KPT - 1 : 1][ROWS / 2];  // entries y and y + 1 packed
            const bool sorted = SORT && len > 3;
            int *const order = (int *)col;  // until column 0 is stored
            if (sorted) {
                if (st < MAXT) by_m[st] = 0;
                named_sync(5, NTS);
                for (int k = st; k < S; k += NTS) atomicAdd(&by_m[MAXT - sinfo[k].m], 1);
                named_sync(5, NTS);
                if (st < 32) {
                    const int c = by_m[lane];
                    int incl = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(FULL, incl, o);
                        if (lane >= o) incl += v;
                    }
                    by_m[lane] = incl - c;
                }
                named_sync(5, NTS);
                for (int k = st; k < S; k += NTS) order[atomicAdd(&by_m[MAXT - sinfo[k].m], 1)] = k;
                named_sync(5, NTS);
            }
#pragma unroll
            for (int q = 0; q < KPT; q++) {
                ok[q] = st + q * NTS < S;
                ks[q] = !ok[q] ? 0 : sorted ? order[st + q * NTS] : st + q * NTS;
                const StateInfo si = sinfo[ks[q]];
                tq[q] = si.time;
                nbo[q] = (si.j1 + 3 * si.node) & ~3;
                pos[q] = ok[q] ? nbo[q] + ks[q] - si.j1 : colstride - 1;
                m[q] = ok[q] ? si.m : 0;
                roff[q] = t2off[ks[q]];
                mostq[q] = SORT || TAIL ? uniform(m[q]) : 0;
                most = imax(most, m[q]);
            }
            // pair u: states 2 u and pair2(u), the same one where there is no second
            auto pair2 = [](int u) { return 2 * u + 1 < KPT ? 2 * u + 1 : 2 * u; };
#pragma unroll
            for (int u = 0; u < NP; u++) {
                const int q0 = 2 * u, q1 = pair2(u);
                rs[u] = pk(rsv[tq[q0]], rsv[tq[q1]]);
                iv[u] = pk(inv[ks[q0]], inv[ks[q1]]);
                xh[u] = xl[u] = pk(0.0f, 0.0f);
            }
            most = uniform(most);
            // rows: 4, 8, 12, 20 or all entries by the warp's longest, zeros past a node's states
            auto by_length = [&](auto all, int longest, auto &&fn) {
                constexpr int R = decltype(all)::value;
                if (R <= 4 || longest <= 4) fn(Int<4>{});
                else if (R <= 8 || longest <= 8) fn(Int<(R < 8 ? R : 8)>{});
                else if (R <= 12 || longest <= 12) fn(Int<(R < 12 ? R : 12)>{});
                else if (R > 20 && longest <= 20) fn(Int<(R < 20 ? R : 20)>{});
                else fn(Int<R>{});
            };
            // fn(q, its row registers, the entries to take) for each of the thread's states
            static_assert(SORT || KPT == 1 || ROWS0 == ROWS, "states in order: one length for all");
            auto each_row = [&](auto &&fn) {
                by_length(Int<ROWS0>{}, SORT ? mostq[0] : most, [&](auto n) {
                    fn(0, row0, n);
                    if constexpr (!SORT) {
#pragma unroll
                        for (int q = 1; q < KPT; q++) fn(q, row[q - 1], n);
                    }
                });
                if constexpr (SORT) {
#pragma unroll
                    for (int q = 1; q < KPT; q++)
                        by_length(Int<ROWS>{}, mostq[q], [&](auto n) { fn(q, row[q - 1], n); });
                }
            };
            // where a thread's states lie in an array of all, from `own` on
            const int own = SORT ? 0 : st;
            auto at = [&](int q) { return SORT ? ks[q] : q * NTS; };
            if (TAIL && !STAGED && t2_bufs) {
                rows_late |= !mbar_wait(&rows_full, rows_phase);
                rows_phase ^= 1u;
                rows = t2buf + ((uintptr_t)rows & 15) / 4;
            }
            each_row([&](int q, auto &into, auto n) {
                const float *r = rows + roff[q];
#pragma unroll
                for (int y = 0; y < decltype(n)::value; y += 2) {
                    const float v0 = y < m[q] ? r[0] : 0.0f, v1 = y + 1 < m[q] ? r[m[q]] : 0.0f;
                    r += 2 * m[q];
                    into[y / 2] = pk(v0, v1);
                }
            });
            cp_wait<EDEPTH - 1>();  // the first emission rows, which other threads read
            named_sync(3, NTC);  // positions stored, slots cleared
#pragma unroll
            for (int q = 0; q < KPT; q++) {
                const int p = rank[ks[q]], b = tq[q], b0 = bptr[b];
                int r = 0, plo = pl[0], ch = ck[0], base = sb[0];
#pragma unroll
                for (int x = 1; x < NRW; x++)
                    if (b >= x * NB / NRW) {
                        r = x;
                        plo = pl[x];
                        ch = ck[x];
                        base = sb[x];
                    }
                // (p - plo) / ch: both below 2^13, so the half keeps the product clear of
                // integers
                const int l = (int)(((float)(p - plo) + 0.5f) * (1.0f / (float)ch));
                const int clo = plo + l * ch;
                // in the chunk's first piece, or in the bin's own when it begins in the chunk
                const bool head = clo >= b0;
                const int j = head ? p - clo : p - b0;
                const int ln = head ? l : b - r * NB / NRW;
                slot[q] = ok[q] ? 2 * (base + 32 * j + ln) + (head ? 0 : 1) : 2 * sb[NRW];
            }
            // ---- first column
            if (bi == 0) {
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    const float v = ok[q] ? fw[ks[q]] : 0.0f;  // priors (K1)
                    col[cur + pos[q]] = v;
                    red[slot[q]] = v;
                    xh[q >> 1] = q & 1 ? pk(lo(xh[q >> 1]), v) : pk(v, 0.0f);
                }
            } else {
                const int *gp = table(d.gptr + Bs->gptr0, SL.gptr);
                const int *gi = table(d.gidx + p0, SL.gidx);
                const float2 *mv = table((const float2 *)(d.determprob + p0), SL.move);
                const float *rr = table(d.recombrow32 + s0, SL.rrow);
                const float *cr = table(d.recoalrow32 + s0, SL.crow);
                const int2 src = *table(d.srcs + blk, SL.src);
                // pairs: the previous column's values with their low parts, each deterministic
                // move by its FP64 probability (kept as a complement near 1), the
                // recombination rows (a small inflow) plain, then the emission
                int g0[KPT], gn[KPT], gmost = 0;
                F2 a[KPT];
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    g0[q] = gp[ks[q]];
                    gn[q] = ok[q] ? gp[ks[q] + 1] - g0[q] : 0;
                    a[q] = F2{0.0f, 0.0f};
                    gmost = imax(gmost, gn[q]);
                }
                gmost = uniform(gmost);
                for (int t = 0; t < gmost; t++) {
#pragma unroll
                    for (int q = 0; q < KPT; q++) {
                        const int j = t < gn[q] ? gi[g0[q] + t] : 0;
                        const float2 xj = last[j];
                        const F2 s = f2_add2(a[q], f2_move(F2{xj.x, xj.y}, mv[j].x));
                        if (t < gn[q]) a[q] = s;
                    }
                }
                const float px = src.x != -1 ? last[src.x].x : 0.0f, py = src.y != -1 ? last[src.y].x : 0.0f;
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    const float rk = rr[ks[q]], ck2 = cr[ks[q]];
                    if (src.x != -1 && rk > 0.0f) a[q] = f2_add(a[q], px * rk);
                    if (src.y != -1 && ck2 > 0.0f) a[q] = f2_add(a[q], py * ck2);
                }
                if (vm & 1) {
#pragma unroll
                    for (int q = 0; q < KPT; q++) {
                        const float e = ring[ks[q]];
                        a[q] = e >= 0.0f ? f2_keep(a[q], e) : f2_mul(a[q], -e);
                    }
                } else if (!(mm & 1)) {
#pragma unroll
                    for (int q = 0; q < KPT; q++) a[q] = f2_keep(a[q], q & 1 ? hi(iv[q >> 1]) : lo(iv[q >> 1]));
                }
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    col[cur + pos[q]] = a[q].hi;
                    red[slot[q]] = a[q].hi;
                }
#pragma unroll
                for (int u = 0; u < NP; u++) {
                    xh[u] = pk(a[2 * u].hi, a[pair2(u)].hi);
                    xl[u] = pk(a[2 * u].lo, a[pair2(u)].lo);
                }
            }
            // the variant rows: the next one to fetch (column EDEPTH + 1 on)
            const float *vrow = d.var32 + Bs->var0 + own + (size_t)__popcll(vm & ((2ull << EDEPTH) - 1)) * S;
            named_sync(4, NTC);  // T2 (barrier A of column 1): column 0 complete, the tables taken
            // the next tree's first classes and where its emission rows are
            int nS = 0, nlen = 0;
            long long nvar0 = 0;
            cw0 = class_at(start + len + lane);
            cw1 = class_at(start + len + 32 + lane);
            if (bi + 1 < I.ntrees) {
                const BlockDev *Bn = desc_of(bi + 1);
                nvar0 = Bn->var0;
                nS = Bn->S;
                nlen = Bn->len;
            }
            int cw2 = class_at(start + 64 + lane);  // the classes after the masks' 64
            float *slot_e = ring + ringstride;      // column i's emissions
            float *const ring_end = ring + EDEPTH * ringstride;

            // ---- columns; iteration i also finalises column i-1
            float *outp = fw + own;
            bool wr[KPT];  // the instance's column 0 keeps the unnormalised prior
#pragma unroll
            for (int q = 0; q < KPT; q++) wr[q] = ok[q] && bi > 0;
            V2 done[NP];  // the normalised column not yet stored (column i - 2 at the top)
            int ndone = 0;
            auto store_done = [&]() {
                if (ndone) {
#pragma unroll
                    for (int q = 0; q < KPT; q++)
                        if (wr[q]) outp[at(q)] = q & 1 ? hi(done[q >> 1]) : lo(done[q >> 1]);
#pragma unroll
                    for (int q = 0; q < KPT; q++) wr[q] = ok[q];
                    outp += S;
                }
                ndone = 1;
            };
            for (int i = 1; i < len; i++) {
                vm >>= 1;
                mm >>= 1;
                if ((i & 31) == 0) {
                    vm |= (unsigned long long)__ballot_sync(FULL, cw2 == COL_VARIANT) << 32;
                    mm |= (unsigned long long)__ballot_sync(FULL, cw2 == COL_MASKED) << 32;
                    cw2 = class_at(start + i + 64 + lane);
                }
                // same-branch dots: sum_y t2[y][k] col[j1 + y], even and odd terms in the two
                // halves of a packed sum
                V2 dot2[KPT];
                each_row([&](int q, const auto &from, auto n) {
                    const float *nb = col + cur + nbo[q];
                    V2 sum = pk(0.0f, 0.0f);
#pragma unroll
                    for (int y = 0; y < decltype(n)::value; y += 4) {
                        const float4 v = *(const float4 *)(nb + y);
                        sum = fma2(from[y / 2], pk(v.x, v.y), sum);
                        sum = fma2(from[y / 2 + 1], pk(v.z, v.w), sum);
                    }
                    dot2[q] = sum;
                });
                if (TAIL && !LONG_ENDS && most > ROWS) {
#pragma unroll
                    for (int q = 0; q < KPT; q++) {
                        for (int y = q ? ROWS : ROWS0; y < mostq[q]; y += 4) {
                            const float *r = rows + roff[q] + y * m[q];
                            float v[4];
#pragma unroll
                            for (int u = 0; u < 4; u++) v[u] = y + u < m[q] ? r[u * m[q]] : 0.0f;
                            const float4 n = *(const float4 *)(col + cur + nbo[q] + y);
                            dot2[q] = fma2(pk(v[0], v[1]), pk(n.x, n.y), dot2[q]);
                            dot2[q] = fma2(pk(v[2], v[3]), pk(n.z, n.w), dot2[q]);
                        }
                    }
                }
                if (TAIL && LONG_ENDS && most > ROWS) {
                    // W states side by side
                    constexpr int W = KPT % 4 == 0 ? 2 : 1;
#pragma unroll
                    for (int q0 = 0; q0 < KPT; q0 += W) {
                        const float *r[W], *nb[W];
                        int left[W], end = 0;
#pragma unroll
                        for (int w = 0; w < W; w++) {
                            const int q = q0 + w, y = q ? ROWS : ROWS0;
                            r[w] = rows + roff[q] + y * m[q];
                            nb[w] = col + cur + nbo[q] + y;
                            left[w] = m[q] - y;
                            end = imax(end, mostq[q] - y);
                        }
                        for (int y = 0; y < end; y += 4) {
                            float v[W][4];
                            float4 n[W];
#pragma unroll
                            for (int w = 0; w < W; w++) {
#pragma unroll
                                for (int u = 0; u < 4; u++) v[w][u] = u < left[w] ? r[w][u * m[q0 + w]] : 0.0f;
                                n[w] = *(const float4 *)(left[w] > 0 ? nb[w] : col);
                                r[w] += 4 * m[q0 + w];
                                nb[w] += 4;
                                left[w] -= 4;
                            }
#pragma unroll
                            for (int w = 0; w < W; w++) {
                                V2 &dq = dot2[q0 + w];
                                dq = fma2(pk(v[w][0], v[w][1]), pk(n[w].x, n[w].y), dq);
                                dq = fma2(pk(v[w][2], v[w][3]), pk(n[w].z, n[w].w), dq);
                            }
                        }
                    }
                }
                float dot[KPT];
#pragma unroll
                for (int q = 0; q < KPT; q++) dot[q] = lo(dot2[q]) + hi(dot2[q]);
                store_done();
                if (i > 1) {
                    // column i - 1 + EDEPTH's row into the slot before column i - 1's (column
                    // i - 2 is done); this column's class masks are one shifted on
                    if (vm >> (EDEPTH - 1) & 1) {
                        if (i - 1 + EDEPTH < len) {
                            float *slot = (slot_e == ring ? ring_end : slot_e - ringstride) + own;
#pragma unroll
                            for (int q = 0; q < KPT; q++)
                                if (ok[q]) cp_async4(slot + at(q), vrow + at(q));
                        }
                        vrow += S;
                    }
                    cp_commit();
                    slot_e = slot_e == ring_end ? ring : slot_e + ringstride;
                }
                // the emissions, complements of the largest: masked columns keep everything
                V2 e[NP];
                bool ratios = false;  // some state's emission is a ratio (stored negated)
                cp_wait<EDEPTH - 1>();
                if (vm & 1) {
                    float least = 0.0f;
#pragma unroll
                    for (int u = 0; u < NP; u++) {
                        e[u] = pk(slot_e[ks[2 * u]], slot_e[ks[pair2(u)]]);
                        least = fminf(least, fminf(lo(e[u]), hi(e[u])));
                    }
                    ratios = __any_sync(FULL, least < 0.0f);
                } else {
#pragma unroll
                    for (int u = 0; u < NP; u++) e[u] = (mm & 1) ? pk(0.0f, 0.0f) : iv[u];
                }
                // the stay, before the inflow is known
                P2 x[NP];
#pragma unroll
                for (int u = 0; u < NP; u++) x[u] = p2_keep(P2{xh[u], xl[u]}, rs[u], nz);
                named_sync(2, NTC);  // B: the shares of tf and of column i-1's norm
                const float4 n4 = *(const float4 *)tfp[MAXT - 1];
#pragma unroll
                for (int u = 0; u < NP; u++) {
                    // plus the inflow
                    const float4 t0 = *(const float4 *)tfp[tq[2 * u]], t1 = *(const float4 *)tfp[tq[pair2(u)]];
                    const V2 tf = pk(((t0.x + t0.y) + t0.z) + t0.w, ((t1.x + t1.y) + t1.z) + t1.w);
                    x[u] = p2_add(x[u], tf + pk(dot[2 * u], dot[pair2(u)]));
                }
                const float norm = ((n4.x + n4.y) + n4.z) + n4.w;
                const float inv_norm = __frcp_rn(norm);
                const V2 in2 = pk(inv_norm, inv_norm);
                // times the emission
                if (!ratios) {
#pragma unroll
                    for (int u = 0; u < NP; u++) x[u] = p2_keep(x[u], e[u], nz);
                } else {
#pragma unroll
                    for (int u = 0; u < NP; u++) {
                        const P2 a = p2_keep(x[u], e[u], nz), b = p2_mul(x[u], pk(-lo(e[u]), -hi(e[u])), nz);
                        const bool k0 = lo(e[u]) >= 0.0f, k1 = hi(e[u]) >= 0.0f;
                        x[u].hi = pk(k0 ? lo(a.hi) : lo(b.hi), k1 ? hi(a.hi) : hi(b.hi));
                        x[u].lo = pk(k0 ? lo(a.lo) : lo(b.lo), k1 ? hi(a.lo) : hi(b.lo));
                    }
                }
                cur = colstride - cur;
                // rescaled; states past the last one go to a slot of their own
#pragma unroll
                for (int u = 0; u < NP; u++) x[u] = p2_mul(x[u], in2, nz);
#pragma unroll
                for (int q = 0; q < KPT; q++) {
                    const float v = q & 1 ? hi(x[q >> 1].hi) : lo(x[q >> 1].hi);
                    col[cur + pos[q]] = v;
                    red[slot[q]] = v;
                }
                named_sync(1, NTC);  // A: column i complete
#pragma unroll
                for (int u = 0; u < NP; u++) {
                    done[u] = fma2(xh[u], in2, nz);
                    xh[u] = x[u].hi;
                    xl[u] = x[u].lo;
                }
            }
            store_done();
            // ---- the tree's last column, normalised with its low parts for the next switch
            first_rows(nvar0, nS, nlen);
            named_sync(2, NTC);  // B
            const float4 n4 = *(const float4 *)tfp[MAXT - 1];
            const float inv_norm = __frcp_rn(((n4.x + n4.y) + n4.z) + n4.w);
#pragma unroll
            for (int q = 0; q < KPT; q++) {
                const F2 x = f2_mul(q & 1 ? F2{hi(xh[q >> 1]), hi(xl[q >> 1])} : F2{lo(xh[q >> 1]), lo(xl[q >> 1])},
                                    inv_norm);
                if (ok[q]) last[ks[q]] = make_float2(x.hi, x.lo);
                if (wr[q]) outp[at(q)] = x.hi;
            }
        } else {
            // ================= reducers
            const int blo = rw * NB / NRW, bhi = (rw + 1) * NB / NRW;
            int plo = pl[0], chunk = ck[0], unrolled = cu[0], base = sb[0];
#pragma unroll
            for (int q = 1; q < NRW; q++)
                if (rw == q) {
                    plo = pl[q];
                    chunk = ck[q];
                    unrolled = cu[q];
                    base = sb[q];
                }
            unrolled = uniform(unrolled);
            float2 *const mine = (float2 *)red + base + lane;
            for (int j = 0; j < unrolled; j++) mine[32 * j] = make_float2(0.0f, 0.0f);
            named_sync(3, NTC);  // slots cleared
            // lane b - blo: the chunks lh .. lh + nh - 1 begin inside bin b
            int lh = 0, nh = 0;
            const int mb = blo + lane;
            if (mb < bhi && bptr[mb + 1] > bptr[mb]) {
                lh = (bptr[mb] - plo + chunk - 1) / chunk;
                nh = (bptr[mb + 1] - 1 - plo) / chunk - lh + 1;
            }
            const int nhmax = uniform(nh);
            float take[16];  // 1: the t-th of them is there
#pragma unroll
            for (int t = 0; t < 16; t++) take[t] = t < nh ? 1.0f : 0.0f;
            const float *tms = (const float *)(stage + SL.tm) + lane;
            float tmr[RBINS];
#pragma unroll
            for (int j = 0; j < RBINS; j++)
                tmr[j] = blo + j >= bhi ? 0.0f : lane == MAXT - 1 ? 1.0f : tms[(blo + j) * MAXT];
            const double blkx = tid == 32 ? d.blkext[blk] : 0.0;
            const bool bw = d.bins32 && mb < bhi;
            float *brow = d.bins32 ? d.bins32 + (size_t)(I.col0 + start) * MAXT + mb : nullptr;
            bool prior = bi == 0;  // the instance's column 0 is stored unnormalised
            named_sync(4, NTC);  // T2: column 0 complete, the staged tables taken
            if (producer && bi + 1 < I.ntrees) issue(blk + 1, *desc_of(bi + 1));

            for (int i = 1;; i++) {
                // the lane's pieces, their positions in order
                V2 a = pk(0.0f, 0.0f);
                auto add = [&](auto n, int j0) {
                    float2 v[decltype(n)::value];
#pragma unroll
                    for (int j = 0; j < decltype(n)::value; j++) v[j] = mine[32 * (j0 + j)];
#pragma unroll
                    for (int j = 0; j < decltype(n)::value; j++) a = a + pk(v[j].x, v[j].y);
                };
                if (unrolled == 1) add(Int<1>{}, 0);
                else if (unrolled == 2) add(Int<2>{}, 0);
                else if (unrolled == 4) add(Int<4>{}, 0);
                else
                    for (int j0 = 0; j0 < unrolled; j0 += 8) add(Int<8>{}, j0);
                // lane b - blo: bin b's own piece, then the chunks beginning inside it in order
                const float head = lo(a);
                float bin = hi(a), w[8];
                if (nhmax <= 4) {
#pragma unroll
                    for (int t = 0; t < 4; t++) w[t] = __shfl_sync(FULL, head, lh + t);
#pragma unroll
                    for (int t = 0; t < 4; t++) bin = fmaf(w[t], take[t], bin);
                } else {
#pragma unroll
                    for (int t = 0; t < 8; t++) w[t] = __shfl_sync(FULL, head, lh + t);
#pragma unroll
                    for (int t = 0; t < 8; t++) bin = fmaf(w[t], take[t], bin);
                    if (nhmax > 8) {
#pragma unroll
                        for (int t = 0; t < 8; t++) w[t] = __shfl_sync(FULL, head, lh + 8 + t);
#pragma unroll
                        for (int t = 0; t < 8; t++) bin = fmaf(w[t], take[8 + t], bin);
                        for (int t = 16; t < nhmax; t += 4) {
#pragma unroll
                            for (int u = 0; u < 4; u++) w[u] = __shfl_sync(FULL, head, lh + t + u);
#pragma unroll
                            for (int u = 0; u < 4; u++) bin += t + u < nh ? w[u] : 0.0f;
                        }
                    }
                }
                // this warp's share of tf[a] = sum_b tm[b][a] bin[b], its bins in order (past
                // the share both factors are 0)
                float tf = 0.0f;
#pragma unroll
                for (int j = 0; j < 5; j++) w[j] = __shfl_sync(FULL, bin, j);
#pragma unroll
                for (int j = 0; j < 5; j++) tf = fmaf(tmr[j], w[j], tf);
                if (NB > 5 * NRW) {
#pragma unroll
                    for (int j = 5; j < RBINS; j++) w[j] = __shfl_sync(FULL, bin, j);
#pragma unroll
                    for (int j = 5; j < RBINS; j++) tf = fmaf(tmr[j], w[j], tf);
                }
                tfp[lane][rw] = tf;
                named_sync(2, NTC);  // B
                const float4 n4 = *(const float4 *)tfp[MAXT - 1];
                const float norm = ((n4.x + n4.y) + n4.z) + n4.w;
                // the stored column's time-bin sums, on the stored column's scale
                const float stored = prior ? bin : bin * __frcp_rn(norm);
                if (bw) *brow = stored;
                brow += MAXT;
                prior = false;
                if (rw == 1) {
                    if (lane == (ncols & 31)) mynorm = norm;
                    if ((++ncols & 31) == 0) acc.mul((double)mynorm);
                    if (!(norm > 0.0f) && lane == 0) report_error(d.err, ERR_ZERO_NORM, qi, bi, start + i - 1);
                }
                if (i == len) break;
                named_sync(1, NTC);  // A
            }
            if (tid == 32) extra += blkx;
        }
    }
    if (rows_late) {
        report_error(d.err, ERR_WAIT_LIMIT, qi, -1, -1);
        mbar_wait(&rows_full, rows_phase ^ 1u);  // the copy in flight, before the memory is released
    }
    if (failed && tid == 0) {
        report_error(d.err, ERR_WAIT_LIMIT, qi, -1, -1);
        mbar_wait(&full, phase ^ 1u);  // the copies in flight, before the memory is released
    }
    if (tid == 0) lnl0 = acc0.value();
    named_sync(4, NTC);
    if (rw == 1 && d.lnl) {
        if (lane < (ncols & 31)) acc.mul((double)mynorm);
        double l = acc.value();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(FULL, l, o);
        if (lane == 0) d.lnl[qi] = l + extra + lnl0;
    }
}

// One CTA per instance, each by its own largest tree: a batch's small instances run as fast as
// alone. Warps that an instance has no use for leave at once. LONG: more than 21 time points.
// FEW: batches up to 768 states, without the form of three states a thread (in the same kernel it
// cost the smaller trees' forms 1.5%, by the registers that all of them are given: 0.91 and 0.90 us
// a column at 704 states); WIDE: more owner warps at fewer registers each.
enum Forms { FEW, MANY, WIDE };
template <bool LONG, Forms FORMS>
__global__ void __launch_bounds__(32 * NRW + (FORMS == WIDE ? WIDE_OWNERS : OWNERS)) k_forward32(BatchDev d, int smem, int least, float nzero) {
    const int qi = cta_instance(d);
    const InstDev I = d.inst[qi];
    const Form f = form_of(Sizes{I.maxS, I.maxM, I.nnodes}, smem, LONG, FORMS == WIDE, least);
    const int ntc = 32 * NRW + f.owners;
    if ((int)threadIdx.x >= ntc) return;
    const V2 nz = pk(nzero, nzero);
    // States are sorted by their node's for more than 21 time points alone: 1.69 us a column
    // unsorted and 1.40 sorted at 1138 states of 32, 0.90 and 0.90 at 704 of 20, 1.30 and 1.32 at
    // 930 (the sort and the scattered stores cost what the shorter dots give).
    constexpr int R4 = FORMS == WIDE || LONG ? 4 : 8;
    constexpr int R3 = LONG ? 20 : 8, R40 = LONG ? 12 : R4;
    if (f.kpt == 1) {
        forward32<1, LONG ? 32 : 20, 2, false, true, false>(d, I, qi, 1, ntc, nz);
    } else if (f.kpt == 2) {
        if (!LONG) forward32<2, 20, 20, false, true, false>(d, I, qi, 1, ntc, nz);
        else forward32<2, 20, 12, true, true, true>(d, I, qi, 2, ntc, nz);
    } else if (FORMS != FEW && f.kpt == 3) {
        if (f.staged) forward32<3, R3, 8, true, true, LONG>(d, I, qi, 2, ntc, nz);
        else forward32<3, R3, 8, true, false, LONG>(d, I, qi, f.bufs, ntc, nz);
    } else if (f.kpt == 4) {
        if (FORMS != WIDE && f.staged) forward32<4, R40, R4, true, true, LONG>(d, I, qi, 2, ntc, nz);
        else forward32<4, R40, R4, true, false, LONG>(d, I, qi, f.bufs, ntc, nz);
    } else {
        forward32<8, 4, 4, true, false, LONG>(d, I, qi, f.bufs, ntc, nz);
    }
}

template <bool LONG, Forms FORMS>
void launch(const BatchDev &d, cudaStream_t s, int least) {
    const int maxS = imax(d.maxS, 1);
    const int smem = launch_bytes(Sizes{maxS, imax(d.maxM, 1), d.maxnodes});
    if (!raise_dynamic_smem(k_forward32<LONG, FORMS>, smem)) return;  // the launch reports it
    // an instance with one state a thread may need every warp
    const int owners = FORMS == WIDE ? WIDE_OWNERS : OWNERS;
    const int nt = 32 * NRW + (maxS <= owners && least <= 1 ? owner_threads(maxS, 1) : owners);
    k_forward32<LONG, FORMS><<<d.ninst, nt, smem, s>>>(d, smem, least, -0.0f);
    note_launch();
}

template <Forms FORMS>
void launch(const BatchDev &d, cudaStream_t s, int least) {
    if (d.maxT <= 21) launch<false, FORMS>(d, s, least);
    else launch<true, FORMS>(d, s, least);
}

}  // namespace

bool forward_writes_bins(int maxS) { return imax(maxS, 1) <= MOST_STATES; }

bool launch_forward32(const BatchDev &d, cudaStream_t s, int want_kpt) {
    if (!forward_writes_bins(d.maxS)) return false;
    static const int env = [] {
        const char *e = getenv("AWG_FORWARD_KPT");
        return e ? atoi(e) : 0;
    }();
    auto known = [](int k) { return k == 1 || k == 2 || k == 4 || k == 8; };
    const int least = known(want_kpt) ? want_kpt : known(env) ? env : 1;
    if (d.maxS <= 2 * OWNERS) launch<FEW>(d, s, least);
    else if (d.maxS <= 4 * OWNERS) launch<MANY>(d, s, least);
    else launch<WIDE>(d, s, least);
    return true;
}

}  // namespace awg
