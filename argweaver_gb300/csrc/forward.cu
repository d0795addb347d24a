// K3: the forward pass of the threading HMM, one CTA per instance, column in shared memory: the
// dispatch, the dense test step, and the general kernel, for trees of more states (3,072) than
// the owner threads of forward32.cu (FP32) and chain.cu (FP64) hold.
//
// Per column (arghmm_forward_block, sample_thread.cpp:252-295):
//   fgroups[a] = sum of col1 over states of time a
//   tf[b]      = sum_a tmatrix[a][b] * fgroups[a]
//   col2[k]    = (tf[b_k] + sum over the states j of k's node of tmatrix2[a_j][k]*col1[j]) * e_k
//   col2      /= sum(col2)
// At a local-tree boundary the first column comes from the switch matrix
// (arghmm_forward_switch, sample_thread.cpp:345-389), gathered per target state.
//
// Schedule per column, two CTA barriers:
//   A  the previous column is complete, in state order (for same-branch neighbours) and in
//      time-sorted order (each time bin a contiguous range);
//      warps split the bins; a warp sums a bin with coalesced, conflict-free loads
//   B  every thread reads the bins: the previous column's norm and tf (lane b); then each
//      thread writes its entries of the previous column, divided by that norm, to HBM and
//      computes its entries of the new column scaled by 1/norm (the reference's
//      normalise-then-step, reordered; the normalised values are the same).
// Reductions have a fixed order, so results do not depend on the run or the batch.
// log(norm) goes into an FP64 mantissa product plus an integer exponent (one FP64 log
// every 64 columns instead of one per column).
//
// FP64 (plain path): tmatrix2 = gts - tmatrix, the reference's own subtraction, formed when
// the block's rows are staged. FP32 (chosen path): tables rounded to FP32 by the table
// kernels; columns rescaled every column; the log-likelihood accumulates in FP64. Values
// next to 1 keep their information as complements (built with expm1 in FP64):
//   stay:     x_k * norecombs[b]   ->  x_k - rstay[b] * x_k
//   emission: x_k * e_k            ->  (x_k - inv32[k] * x_k) * e_ref, e_ref into the FP64
//                                      log-likelihood once per invariant column
// so the moving probability mass and the emission contrasts, not their rounding, drive
// the chain over thousands of columns.

#include <cuda_runtime.h>

#include "kernels.h"

namespace awg {

namespace {

template <typename F> struct Tab;

template <> struct Tab<double> {
    static constexpr bool split = false;
    const double *tm, *inv, *var, *dprob, *rrow, *crow, *gts;
    const float *rstay = nullptr;
    const double *lneref = nullptr, *vref = nullptr;
    double *fw;
    __device__ explicit Tab(const BatchDev &d)
        : tm(d.tm), inv(d.inv_lk), var(d.varemit), dprob(d.determprob), rrow(d.recombrow),
          crow(d.recoalrow), gts(d.gts), fw(d.fw64) {}
    // tmatrix2[a][k] (sample_thread.cpp:223-224)
    __device__ double t2(long long idx, double tmab) const { return gts[idx] - tmab; }
};

template <> struct Tab<float> {
    static constexpr bool split = true;
    const float *tm, *inv, *var, *dprob, *rrow, *crow, *t2d;
    const float *rstay;
    const double *lneref, *vref;
    float *fw;
    __device__ explicit Tab(const BatchDev &d)
        : tm(d.tm32), inv(d.inv32), var(d.var32), dprob(d.determprob32), rrow(d.recombrow32),
          crow(d.recoalrow32), t2d(d.t2d32), rstay(d.rstay32), lneref(d.lneref), vref(d.vref),
          fw(d.fw32) {}
    __device__ float t2(long long idx, float) const { return t2d[idx]; }
};

template <typename F>
__device__ __forceinline__ F warp_sum(F v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Running sum of log(norm): mantissa product in FP64 and binary exponent in an integer.
struct LogAcc {
    double prod = 1.0;
    long long e = 0;
    int n = 0;
    double lnl = 0.0;
    double extra = 0.0;  // log(e_ref) of invariant columns (FP32 path)
    __device__ void add(double norm) {
        int ex;
        prod *= frexp(norm, &ex);
        e += ex;
        if (++n == 64) flush();
    }
    __device__ void flush() {
        lnl += extra;
        extra = 0.0;
        if (n) {
            lnl += log(prod) + (double)e * 0.69314718055994530942;
            prod = 1.0;
            e = 0;
            n = 0;
        }
    }
};

struct Meta {
    int time, j1, m, off;
};

template <typename F>
__global__ void __launch_bounds__(512) k_forward(BatchDev d, int maxS, int maxM, int t2_in_smem) {
    extern __shared__ double dyn_d[];
    const Tab<F> tab(d);
    const int qi = cta_instance(d);
    const InstDev I = d.inst[qi];
    const int T = I.T, NB = T - 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NT = blockDim.x, NW = NT >> 5;

    F *col = (F *)dyn_d;                       // [2][maxS] columns in state order
    F *colT = col + 2 * maxS;                  // [maxS] newest column, time-sorted
    F *t2s = colT + maxS;                      // [maxM] tmatrix2 entries of the block
    F *invS = t2s + maxM;                      // [maxS] invariant-site emissions
    Meta *meta = (Meta *)(((uintptr_t)(invS + maxS) + 15) & ~(uintptr_t)15);
    int *rank = (int *)(meta + maxS);          // time-sorted position of each state
    __shared__ F tmS[MAXT * MAXT];
    __shared__ F rS[MAXT];
    __shared__ F tfrow[MAXT - 1][32];          // per bin b: tm[b][lane] * sum_b, sum_b (lane 31)
    __shared__ int bptr[MAXT + 1];

    LogAcc acc;
    int c = 0;                                 // buffer holding the current column

    for (int bi = 0; bi < I.ntrees; bi++) {
        const int blk = I.block0 + bi;
        const BlockDev B = d.blocks[blk];
        const int S = B.S;
        F *fw = tab.fw + B.cell0;

        if (S == 0) {
            // fully specified tree: one state that carries over (sample_thread.cpp:201-206)
            F v;
            if (bi == 0) {
                v = fw[0];
                if (tid == 0) col[c * maxS] = v;
            } else {
                // switch into the single state: every source maps to it
                const int2 src = d.srcs[blk];
                const int *gp = d.gptr + B.gptr0;
                const int *gi = d.gidx + B.prev_state0;
                const F *dp = tab.dprob + B.prev_state0;
                const F *rr = tab.rrow + B.state0;
                const F *cr = tab.crow + B.state0;
                F part = 0;
                if (tid < 32) {
                    for (int p = gp[0] + lane; p < gp[1]; p += 32) part += col[c * maxS + gi[p]] * dp[gi[p]];
                    part = warp_sum(part);
                }
                if (tid == 0) {
                    if (src.x != -1 && rr[0] > F(0)) part += col[c * maxS + src.x] * rr[0];
                    if (src.y != -1 && cr[0] > F(0)) part += col[c * maxS + src.y] * cr[0];
                    acc.add((double)part);
                    col[c * maxS] = F(1);
                    fw[0] = F(1);
                }
                v = F(1);
            }
            for (int i = 1 + tid; i < B.len; i += NT) fw[i] = v;
            __syncthreads();
            continue;
        }

        // ---- stage the block's tables
        for (int k = tid; k < S; k += NT) {
            const StateInfo si = d.sinfo[B.state0 + k];
            meta[k] = Meta{si.time, si.j1, si.m, d.t2off[B.state0 + k]};
            rank[d.bt_perm[B.state0 + k]] = k;  // k as sorted position: rank[state] = position
            invS[k] = tab.inv[B.state0 + k];
        }
        const F *tmg = tab.tm + (size_t)blk * MAXT * MAXT;
        for (int e = tid; e < NB * MAXT; e += NT) tmS[e] = tmg[e];
        for (int a = tid; a <= MAXT; a += NT) bptr[a] = d.bt_ptr[(size_t)blk * (MAXT + 1) + a];
        if (Tab<F>::split)
            for (int a = tid; a < MAXT; a += NT) rS[a] = tab.rstay[(size_t)blk * MAXT + a];
        __syncthreads();
        if (t2_in_smem)
            for (int k = tid; k < S; k += NT) {  // same-branch entries, node blocks source-major
                const Meta mk = meta[k];
                const int a0 = mk.time - (k - mk.j1);
                for (int y = 0; y < mk.m; y++)
                    t2s[mk.off + y * mk.m] =
                        tab.t2(B.t2_0 + mk.off + y * mk.m, tmS[(a0 + y) * MAXT + mk.time]);
            }
        const uint8_t *cls = d.colclass + I.col0 + B.start;
        const int *cvar = d.colvar + I.col0 + B.start;
        const F *inv = invS;
        const F *var = tab.var + B.var0;
        // FP32: the tree's emission references, added once the tree is done
        const double blkx = Tab<F>::split && tid == 0 ? d.blkext[blk] : 0.0;
        // column classes and variant rows, 32 columns per load, read back by shuffles
        int ccache = 0, vcache = 0, cbase = -32;
        auto colinfo = [&](int i, uint8_t &ci, int &vi) {
            if (i - cbase >= 32) {
                cbase = i;
                const int q = i + lane;
                ccache = q < B.len ? cls[q] : 0;
                vcache = q < B.len ? cvar[q] : 0;
            }
            ci = (uint8_t)__shfl_sync(0xffffffffu, ccache, i - cbase);
            vi = __shfl_sync(0xffffffffu, vcache, i - cbase);
        };
        __syncthreads();  // rank[] complete

        // ---- first column of the block
        if (bi == 0) {
            for (int k = tid; k < S; k += NT) {
                const F v = fw[k];  // priors (K1)
                col[c * maxS + k] = v;
                colT[rank[k]] = v;
            }
        } else {
            // previous column is normalised in col[c] (S1 entries)
            const int2 src = d.srcs[blk];
            const int *gp = d.gptr + B.gptr0;
            const int *gi = d.gidx + B.prev_state0;
            const F *dp = tab.dprob + B.prev_state0;
            const F *rr = tab.rrow + B.state0;
            const F *cr = tab.crow + B.state0;
            uint8_t c0;
            int v0;
            colinfo(0, c0, v0);
            const F *prev = col + c * maxS;
            for (int k = tid; k < S; k += NT) {
                F s = 0;
                for (int p = gp[k]; p < gp[k + 1]; p++) {
                    const int j = gi[p];
                    s += prev[j] * dp[j];
                }
                if (src.x != -1 && rr[k] > F(0)) s += prev[src.x] * rr[k];
                if (src.y != -1 && cr[k] > F(0)) s += prev[src.y] * cr[k];
                F v;
                if (c0 == COL_MASKED) v = s;
                else if (c0 == COL_INVARIANT) v = Tab<F>::split ? s - s * inv[k] : s * inv[k];
                else {
                    const F e = var[(size_t)v0 * S + k];
                    v = !Tab<F>::split ? s * e : e >= F(0) ? s - s * e : s * -e;
                }
                col[(c ^ 1) * maxS + k] = v;
                colT[rank[k]] = v;
            }
            c ^= 1;
        }

        // ---- remaining columns; iteration i also finalises column i-1
        for (int i = 1; i <= B.len; i++) {
            __syncthreads();  // A: column i-1 complete
            // each bin's sum, and its terms of tf[a] = sum_b tm[b][a] sum_b (lane a); the
            // terms are added in bin order below, so the result does not depend on NT
            for (int b = warp; b < NB; b += NW) {
                F s = 0;
                for (int p = bptr[b] + lane; p < bptr[b + 1]; p += 32) s += colT[p];
                s = warp_sum(s);
                tfrow[b][lane] = lane == 31 ? s : (lane < NB ? tmS[b * MAXT + lane] : F(0)) * s;
            }
            __syncthreads();  // B: bin rows of column i-1
            F norm = 0, tf = 0;
            for (int b = 0; b < NB; b++) {
                tf += tfrow[b][lane];
                norm += tfrow[b][31];
            }
            const F inv_norm = F(1) / norm;
            const F *cur = col + c * maxS;
            if (tid == 0) {
                acc.add((double)norm);
                if (!(norm > F(0))) report_error(d.err, ERR_ZERO_NORM, qi, bi, B.start + i - 1);
            }
            // finalise column i-1: normalised into the table (the instance's column 0
            // keeps the unnormalised prior, as the reference's table does)
            const bool write_prev = !(bi == 0 && i == 1);
            F *outp = fw + (size_t)(i - 1) * S;
            if (i == B.len) {
                for (int k = tid; k < S; k += NT) {
                    const F v = cur[k] * inv_norm;
                    if (write_prev) outp[k] = v;
                    col[c * maxS + k] = v;  // normalised, for the next switch
                }
                break;
            }
            uint8_t ci;
            int vrow;
            colinfo(i, ci, vrow);
            F *nxt = col + (c ^ 1) * maxS;
            for (int k0 = 0; k0 < S; k0 += NT) {
                const int k = k0 + tid;
                const bool valid = k < S;
                const Meta mk = meta[valid ? k : 0];
                const F tfb = __shfl_sync(0xffffffffu, tf, mk.time);
                if (valid) {
                    const F xk = cur[k];
                    if (write_prev) outp[k] = xk * inv_norm;
                    const F *nb = cur + mk.j1;
                    F s = tfb;
                    if (t2_in_smem) {
                        const F *row = t2s + mk.off;
                        const int m = mk.m;
                        int y = 0;
                        F s1 = 0;
                        for (; y + 1 < m; y += 2) {
                            s += row[0] * nb[y];
                            s1 += row[m] * nb[y + 1];
                            row += 2 * m;
                        }
                        if (y < m) s += row[0] * nb[y];
                        s += s1;
                    } else {
                        const int a0 = mk.time - (k - mk.j1);
                        for (int y = 0; y < mk.m; y++)
                            s += tab.t2(B.t2_0 + mk.off + y * mk.m, tmS[(a0 + y) * MAXT + mk.time]) * nb[y];
                    }
                    F v;
                    if (Tab<F>::split) {
                        s = xk + (s - rS[mk.time] * xk);  // stay term apart
                        if (ci == COL_MASKED) v = s;
                        else if (ci == COL_INVARIANT) v = s - s * inv[k];
                        else {
                            const F e = var[(size_t)vrow * S + k];
                            v = e >= F(0) ? s - s * e : s * -e;
                        }
                    } else {
                        const F e = ci == COL_MASKED ? F(1)
                                  : ci == COL_INVARIANT ? inv[k] : var[(size_t)vrow * S + k];
                        v = s * e;
                    }
                    v *= inv_norm;
                    nxt[k] = v;
                    colT[rank[k]] = v;
                }
            }
            c ^= 1;
        }
        if (Tab<F>::split && tid == 0) acc.extra += blkx;
        __syncthreads();
    }
    if (tid == 0 && d.lnl) {
        acc.flush();
        d.lnl[qi] = acc.lnl;
    }
}

// ---------------------------------------------------------------------------------------
// The reference's dense test step (arghmm_forward_block_slow, sample_thread.cpp:301-337),
// FP64, one CTA per instance: every column of a local tree from the full S x S transition
// matrix, col2[k] = (sum_j col1[j] transmat[j][k]) emit[i][k], normalised by division. The
// matrix entries are TransMatrix::get (trans.h:64-83) formed where they are read from the
// table kernel's FP64 tables: the different-node entry tmatrix[a_j][b_k] for states on
// other nodes, the same-node row get_time(a, b, c, minage, true) on k's own node. Thread k
// sums over j in the reference's order. Tree switches, priors and the log-likelihood are
// the structured path's (arghmm_forward_switch, sample_thread.cpp:345-389).
__device__ double dense_block_sum(const double *v, int n, double *red) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    double s = 0.0;
    for (int k = tid; k < n; k += blockDim.x) s += v[k];
    s = warp_sum(s);
    __syncthreads();  // red free
    if (lane == 0) red[warp] = s;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < nw; w++) t += red[w];
    return t;
}

__global__ void __launch_bounds__(512) k_forward_dense(BatchDev d, int maxS) {
    extern __shared__ double dyn_d[];
    const int qi = cta_instance(d);
    const InstDev I = d.inst[qi];
    const int tid = threadIdx.x, lane = tid & 31, NT = blockDim.x;
    double *col = dyn_d;                         // [2][maxS]
    int *snode = (int *)(col + 2 * maxS);        // [maxS] node of each state
    int *stime = snode + maxS;                   // [maxS] time of each state
    __shared__ double tmS[MAXT * MAXT];
    __shared__ double red[16];
    LogAcc acc;
    int c = 0;  // buffer holding the current (normalised) column

    for (int bi = 0; bi < I.ntrees; bi++) {
        const int blk = I.block0 + bi;
        const BlockDev B = d.blocks[blk];
        const int S = B.S;
        double *fw = d.fw64 + B.cell0;
        if (S == 0) {
            // fully specified tree: one state that carries over (sample_thread.cpp:201-206)
            double v;
            if (bi == 0) {
                v = fw[0];
                if (tid == 0) col[c * maxS] = v;
            } else {
                const int2 src = d.srcs[blk];
                const int *gp = d.gptr + B.gptr0;
                const int *gi = d.gidx + B.prev_state0;
                const double *dp = d.determprob + B.prev_state0;
                const double *rr = d.recombrow + B.state0;
                const double *cr = d.recoalrow + B.state0;
                double sum = 0.0;
                if (tid < 32) {
                    for (int p = gp[0] + lane; p < gp[1]; p += 32) sum += col[c * maxS + gi[p]] * dp[gi[p]];
                    sum = warp_sum(sum);
                }
                if (tid == 0) {
                    if (src.x != -1 && rr[0] > 0.0) sum += col[c * maxS + src.x] * rr[0];
                    if (src.y != -1 && cr[0] > 0.0) sum += col[c * maxS + src.y] * cr[0];
                    acc.add(sum);
                    col[c * maxS] = 1.0;
                    fw[0] = 1.0;
                }
                v = 1.0;
            }
            for (int i = 1 + tid; i < B.len; i += NT) fw[i] = v;
            __syncthreads();
            continue;
        }
        for (int k = tid; k < S; k += NT) {
            const StateInfo si = d.sinfo[B.state0 + k];
            snode[k] = si.node;
            stime[k] = si.time;
        }
        const double *tmg = d.tm + (size_t)blk * MAXT * MAXT;
        for (int e = tid; e < MAXT * MAXT; e += NT) tmS[e] = tmg[e];
        __syncthreads();
        const uint8_t *cls = d.colclass + I.col0 + B.start;
        const int *cvar = d.colvar + I.col0 + B.start;
        auto emit = [&](int i, int k) -> double {
            const uint8_t ci = cls[i];
            if (ci == COL_MASKED) return 1.0;
            if (ci == COL_INVARIANT) return d.inv_lk[B.state0 + k];
            return d.varemit[B.var0 + (size_t)cvar[i] * S + k];
        };
        // first column: the priors, or the switch from the previous tree's last column
        double *cur = col + (c ^ 1) * maxS;
        if (bi == 0) {
            for (int k = tid; k < S; k += NT) cur[k] = fw[k];
        } else {
            const double *prev = col + c * maxS;
            const int2 src = d.srcs[blk];
            const int *gp = d.gptr + B.gptr0;
            const int *gi = d.gidx + B.prev_state0;
            const double *dp = d.determprob + B.prev_state0;
            const double *rr = d.recombrow + B.state0;
            const double *cr = d.recoalrow + B.state0;
            for (int k = tid; k < S; k += NT) {
                double s = 0.0;
                for (int p = gp[k]; p < gp[k + 1]; p++) s += prev[gi[p]] * dp[gi[p]];
                if (src.x != -1 && rr[k] > 0.0) s += prev[src.x] * rr[k];
                if (src.y != -1 && cr[k] > 0.0) s += prev[src.y] * cr[k];
                cur[k] = s * emit(0, k);
            }
            __syncthreads();
            const double norm = dense_block_sum(cur, S, red);
            if (tid == 0) {
                acc.add(norm);
                if (!(norm > 0.0)) report_error(d.err, ERR_ZERO_NORM, qi, bi, B.start);
            }
            for (int k = tid; k < S; k += NT) {
                cur[k] /= norm;
                fw[k] = cur[k];
            }
        }
        c ^= 1;
        for (int i = 1; i < B.len; i++) {
            __syncthreads();  // column i-1 complete
            const double *c1 = col + c * maxS;
            double *c2 = col + (c ^ 1) * maxS;
            for (int k = tid; k < S; k += NT) {
                const StateInfo sk = d.sinfo[B.state0 + k];
                const double *grow = d.gts + B.t2_0 + d.t2off[B.state0 + k];
                double s = 0.0;
                for (int j = 0; j < S; j++) {
                    const double p = snode[j] == sk.node ? grow[(j - sk.j1) * sk.m]
                                                         : tmS[stime[j] * MAXT + sk.time];
                    s += c1[j] * p;
                }
                c2[k] = s * emit(i, k);
            }
            __syncthreads();
            const double norm = dense_block_sum(c2, S, red);
            if (tid == 0) {
                acc.add(norm);
                if (!(norm > 0.0)) report_error(d.err, ERR_ZERO_NORM, qi, bi, B.start + i);
            }
            double *outp = fw + (size_t)i * S;
            for (int k = tid; k < S; k += NT) {
                c2[k] /= norm;
                outp[k] = c2[k];
            }
            c ^= 1;
        }
        __syncthreads();
    }
    if (tid == 0 && d.lnl) {
        acc.flush();
        d.lnl[qi] = acc.lnl;
    }
}

int forward_threads(int maxS) {
    if (maxS > 256) return 512;
    if (maxS > 128) return 256;
    return 128;
}


template <typename F>
size_t forward_smem(int maxS, int maxM) {
    return (size_t)(4 * maxS + maxM) * sizeof(F) + 16 + (size_t)maxS * (sizeof(Meta) + sizeof(int));
}

template <typename F>
void launch_old(const BatchDev &d, int maxM, cudaStream_t s) {
    const int maxS = imax(d.maxS, 1);
    maxM = imax(maxM, 1);
    // stage the same-branch rows in shared memory when they fit, else read them from L1/L2
    int t2_in_smem = forward_smem<F>(maxS, maxM) <= 200 * 1024;
    if (!t2_in_smem) maxM = 1;
    const size_t smem = forward_smem<F>(maxS, maxM);
    // opt in; static shared memory counts against 48 KB too
    if (!raise_dynamic_smem(k_forward<F>, smem)) return;
    k_forward<F><<<d.ninst, forward_threads(maxS), smem, s>>>(d, maxS, maxM, t2_in_smem);
    note_launch();
}

}  // namespace

void launch_forward_dense(const BatchDev &d, cudaStream_t s) {
    const int maxS = imax(d.maxS, 1);
    const size_t smem = 2 * (size_t)maxS * sizeof(double) + 2 * (size_t)maxS * sizeof(int);
    if (!raise_dynamic_smem(k_forward_dense, smem)) return;  // the launch reports it
    const int nt = imin(512, imax(32, (maxS + 31) / 32 * 32));
    k_forward_dense<<<d.ninst, nt, smem, s>>>(d, maxS);
    note_launch();
}

void launch_forward(const BatchDev &d, bool fp32, cudaStream_t s, int kpt) {
    if (fp32 ? launch_forward32(d, s, kpt) : launch_forward64(d, s)) return;
    if (fp32) launch_old<float>(d, d.maxM, s);
    else launch_old<double>(d, d.maxM, s);
}

}  // namespace awg
