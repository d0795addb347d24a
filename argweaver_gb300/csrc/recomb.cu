// Recombination sampling along a sampled thread (sample_recombinations, recomb.cpp:151-235)
// on the device, in recomb_sampler.cuh's expressions and order.
//
// The walk over the columns is sequential (the number of draws depends on the draws), but its
// cost was not: one thread evaluated every tree's transition terms as it reached them, some
// 140 FP64 logarithms and exponentials a tree at 64 cycles an FP64 instruction, and read the
// path a column at a time. Now a warp per tree forms the lineage counts and terms of all trees
// at once (a lane per time point; the sums and the logarithmic prefix that the reference forms
// in order stay in order), and one warp walks: 32 columns a step to the next event, a state's
// node by a scan over the nodes, a lane per candidate recombination. 2,000 columns of 44 trees
// at 23 nodes: 9.3 -> 0.6 ms a call.

#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "kernels.h"
#include "plan.h"
#include "recomb_sampler.cuh"

namespace awg {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// A tree's lineage counts and transition terms, as the walk reads them.
struct RsTables {
    int nb[MAXT], nr[MAXT], nc[MAXT];
    RsTerms terms;
};

// Tree b of the instance: root and (internal) subtree fields; false on a malformed tree.
__device__ bool tree_of(const RsInstance &in, int b, RsTree &t) {
    const int lane = threadIdx.x & 31;
    t = RsTree{in.nodes + (size_t)b * in.nnodes, in.nnodes, -1, in.internal, -1, -1, 0};
    for (int v0 = 0; v0 < t.n; v0 += 32) {
        const int v = v0 + lane;
        const unsigned r = __ballot_sync(FULL, v < t.n && t.nd[v].x == -1);
        if (r) t.root = v0 + 31 - __clz(r);  // the last one, as a walk over the nodes finds it
    }
    if (t.root < 0) return false;
    if (t.internal) {
        t.sub = t.nd[t.root].y;
        t.mainr = t.nd[t.root].z;
        if (t.sub < 0 || t.mainr < 0) return false;
        t.minage = in.minage > t.nd[t.sub].w ? in.minage : t.nd[t.sub].w;
    }
    return true;
}

// rs_lineages and rs_terms of every tree, a warp each; lane b has time point b.
__global__ void __launch_bounds__(128) k_recomb_tables(RsInstance in, RsModel m, RsTables *out) {
    const int b0 = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b0 >= in.ntrees) return;
    RsTree t;
    if (!tree_of(in, b0, t)) return;  // the walk reports it
    if (t.internal && t.nd[t.root].w < m.T) return;  // no states: not sampled
    const int T = m.T, b = lane;
    int nb = 0, nr = 0, nc = 0;
    double treelen = 0.0;
    for (int v = 0; v < t.n; v++) {
        const int4 x = t.nd[v];
        const bool top = x.x == -1 || (t.internal && x.x == t.root);
        if (!top) treelen += m.times[t.nd[x.x].w] - m.times[x.w];
        if (t.internal && (v == t.sub || v == t.root)) continue;
        const int pa = top ? T - 2 : t.nd[x.x].w;
        const int in_ = x.w <= b && b < pa, at = b == pa;
        nb += in_ + (at && top);
        nr += in_ + at;
        nc += in_ + at;
    }
    if (t.internal) {
        treelen -= m.times[t.nd[t.sub].w];
        if (b < t.nd[t.sub].w) {
            nb--;
            nr--;
            nc--;
        }
    }
    if (b == T - 1) nb = 1;
    // coalescence rates (calc_coal_rates_partial_tree, trans.cpp:13-21) and their running sums
    const bool live = b < T;
    const double r0 = live ? m.csteps[2 * b] * nb / (2.0 * m.pops[b]) : 0.0;
    const double r1 = live ? m.csteps[2 * b + 1] * nb / (2.0 * m.pops[b]) : 0.0;
    double C = 0.0, c1 = 0.0, c2 = 0.0;  // c1 = C[2b - 1], c2 = C[2b - 2]
    for (int i = 0; i < 2 * T - 1; i++) {
        if (i == 2 * b) c1 = C;
        if (i == 2 * b - 1) c2 = C;
        C += __shfl_sync(FULL, i & 1 ? r1 : r0, i >> 1);
    }
    const double rprev = __shfl_up_sync(FULL, r1, 1), before = b > 0 ? rprev : 0.0;
    RsTables &o = out[b0];
    const int ra = t.internal ? t.nd[t.mainr].w : t.nd[t.root].w;
    double term = 0.0;
    if (b < T - 1) {
        double treelen2 = treelen + m.times[b], treelen2_b;
        if (b > ra) {
            treelen2 += m.times[b] - m.times[ra];
            treelen2_b = treelen2 + m.tsteps[b];
        } else {
            treelen2_b = treelen2 + m.tsteps[ra];
        }
        term = c1 + log(m.tsteps[b] * (nb + 1.0) / (nr + 1.0));
        const double hit = b < T - 2 ? log(1 - exp(-r0 - before)) : 0.0;
        o.terms.lnE2[b] = -c2 + hit;
        o.terms.lnG4[b] = -c2 + hit;
        o.terms.G3[b] = (b < T - 2 ? 1.0 - exp(-r0) : 1.0) * m.tsteps[b] * (nb / (nr + 1.0 + int(b < ra)));
        o.terms.D[b] = (1.0 - exp(-m.rho * treelen2)) / treelen2_b;
        o.terms.E[b] = 1.0 / nc;
        o.terms.norecombs[b] = exp(-fmax(m.rho * treelen2, m.rho));
    }
    double lnB = 0.0;
    for (int i = 0; i < T - 1; i++) {
        const double x = __shfl_sync(FULL, term, i);
        lnB = i == 0 ? x : rs_logadd(lnB, x);
        if (i == b) o.terms.lnB[b] = lnB;
    }
    if (live) {
        o.nb[b] = nb;
        o.nr[b] = nr;
        o.nc[b] = nc;
    }
}

// rs_state by the warp: the node and time of state k (every lane gets them).
__device__ bool state_of(const RsTree &t, int T, int k, int &node, int &time) {
    const int lane = threadIdx.x & 31;
    if (k < 0) return false;
    for (int v0 = 0; v0 < t.n; v0 += 32) {
        int t0 = 0;
        const int n = v0 + lane < t.n ? rs_node_states(t, T, v0 + lane, t0) : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += x;
        }
        const unsigned hit = __ballot_sync(FULL, k < incl && k >= incl - n);
        if (hit) {
            const int l = __ffs(hit) - 1;
            node = v0 + l;
            time = __shfl_sync(FULL, t0 + k - (incl - n), l);
            return true;
        }
        k -= __shfl_sync(FULL, incl, 31);
    }
    return false;
}

// rs_sample by one warp over the trees' tables.
__device__ int walk(const RsInstance &in, const RsModel &m, const RsTables *tables, RsTables &tab, double *probs,
                    int *used) {
    const int lane = threadIdx.x & 31;
    int count = 0, cu = 0, end = 0;
    for (int b = 0; b < in.ntrees; b++) {
        RsTree t;
        if (!tree_of(in, b, t)) return RS_BAD_STATE;
        const int start = end;
        end = start + in.blocklens[b];
        if (t.internal) {
            bool some = false;
            for (int v0 = 0; v0 < t.n && !some; v0 += 32) {
                int t0;
                some = __any_sync(FULL, v0 + lane < t.n && rs_node_states(t, m.T, v0 + lane, t0) > 0);
            }
            if (!some) continue;  // no state space: no sampling
        }
        bool have = false;
        auto need_tables = [&]() {
            if (have) return;
            __syncwarp();
            for (int x = lane; x < (int)(sizeof(RsTables) / 4); x += 32) ((int *)&tab)[x] = ((const int *)&tables[b])[x];
            __syncwarp();
            have = true;
        };
        int next_recomb = -1;  // absolute coordinate
        // a block's first column takes no new recombination: the first block starts the
        // region, every later one begins with a switch
        for (int i = start + 1; i < end; i++) {
            if (in.path[i] == in.path[i - 1]) {
                if (in.start_coord + i > next_recomb) {  // draw the distance to the next optional one
                    int ln, lt;
                    if (!state_of(t, m.T, in.path[i - 1], ln, lt)) return RS_BAD_STATE;
                    need_tables();
                    const double self_trans =
                        rs_stay(tab.terms, lt, t.nd[ln].w, t.internal ? t.nd[t.sub].w : 0);
                    const double rate = 1.0 - (tab.terms.norecombs[lt] / self_trans);
                    if (cu >= in.nu) return RS_OUT_OF_UNIFORMS;
                    const double e = -log(in.u[cu++]) / rate;  // expovariate
                    const double endd = double(in.start_coord + end), to = in.start_coord + i + e;
                    next_recomb = int(endd < to ? endd : to);
                }
                if (in.start_coord + i < next_recomb) {
                    // on to the next change of state or the optional recombination
                    const int stop = imin(next_recomb - in.start_coord, end);
                    int j = i + 1;
                    for (; j < stop; j += 32) {
                        const int c = j + lane;
                        const unsigned ch = __ballot_sync(FULL, c < stop && in.path[c] != in.path[c - 1]);
                        if (ch) {
                            j += __ffs(ch) - 1;
                            break;
                        }
                    }
                    i = imin(j, stop);
                    if (i >= end) break;
                }
            }
            next_recomb = -1;
            int sn, st, ln, lt;
            if (!state_of(t, m.T, in.path[i], sn, st) || !state_of(t, m.T, in.path[i - 1], ln, lt))
                return RS_BAD_STATE;
            need_tables();
            // get_possible_recomb (recomb.cpp:128-148): on the state's node, then the thread's
            const int end_time = st < lt ? st : lt;
            const int a0 = t.nd[sn].w, n0 = sn == ln ? imax(end_time - a0 + 1, 0) : 0;
            const int other = t.internal ? t.sub : -1, b0 = t.internal ? t.nd[t.sub].w : 0;
            const int n = n0 + imax(end_time - b0 + 1, 0);
            auto cand = [&](int c, int &node, int &time) {
                node = c < n0 ? sn : other;
                time = c < n0 ? a0 + c : b0 + c - n0;
            };
            __syncwarp();
            for (int c = lane; c < n; c += 32) {
                int node, time;
                cand(c, node, time);
                probs[c] = rs_recomb_prob(t, m, tab.nb, tab.nr, tab.nc, ln, lt, st, node, time);
            }
            __syncwarp();
            double total = 0.0;
            for (int c = 0; c < n; c++) total += probs[c];
            // sample (common.h:272-290)
            if (cu >= in.nu) return RS_OUT_OF_UNIFORMS;
            const double pick = in.u[cu++] * total;
            int pickc = n - 1;
            double x = 0.0;
            for (int c = 0; c < n; c++) {
                x += probs[c];
                if (x >= pick) {
                    pickc = c;
                    break;
                }
            }
            if (count >= in.cap) return RS_FULL;
            if (lane == 0) {
                int node, time;
                cand(pickc, node, time);
                in.pos[count] = i;
                in.node[count] = node;
                in.time[count] = time;
            }
            count++;
        }
    }
    *used = cu;
    return count;
}

__global__ void __launch_bounds__(32) k_recomb_walk(RsInstance in, RsModel m, const RsTables *tables, int *result) {
    __shared__ RsTables tab;
    __shared__ double probs[2 * MAXT + 2];
    int used = 0;
    const int rc = walk(in, m, tables, tab, probs, &used);
    if (threadIdx.x == 0) {
        result[0] = rc;
        result[1] = used;
    }
}

}  // namespace

int sample_recombinations(const awg_problem *p, const int *path, const double *u, int nu,
                          int *pos, int *node, int *time, int cap, int *used, std::string &err) {
    if (!p || !path || (!u && nu > 0) || nu < 0 || cap < 0 || (cap > 0 && (!pos || !node || !time))) {
        err = "sample_recombinations: bad arguments";
        return -1;
    }
    HostPlan plan;
    if (!build_plan(p, 1, plan, err)) return -1;
    const int L = p->seqlen;

    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    size_t off = 0;
    const size_t o_nodes = off; off += al(sizeof(int) * plan.nodes.size());
    const size_t o_bl = off; off += al(sizeof(int) * p->ntrees);
    const size_t o_path = off; off += al(sizeof(int) * L);
    const size_t o_u = off; off += al(sizeof(double) * std::max(nu, 1));
    const size_t o_model = off; off += al(sizeof(double) * MODEL_STRIDE);
    const size_t in_bytes = off;
    const size_t o_tab = off; off += al(sizeof(RsTables) * (size_t)p->ntrees);
    const size_t o_res = off; off += al(sizeof(int) * 2);
    const size_t o_out = off; off += al(sizeof(int) * 3 * std::max(cap, 1));
    char *D = nullptr;
    cudaError_t rc = cudaMalloc(&D, off);
    if (rc != cudaSuccess) {
        err = std::string("sample_recombinations: cudaMalloc: ") + cudaGetErrorString(rc);
        return -2;
    }
    RsInstance in;
    in.nodes = (const int4 *)(D + o_nodes);
    in.blocklens = (const int *)(D + o_bl);
    in.path = (const int *)(D + o_path);
    in.u = (const double *)(D + o_u);
    in.ntrees = p->ntrees;
    in.nnodes = p->nnodes;
    in.nu = nu;
    in.start_coord = p->start_coord;
    in.internal = p->internal != 0;
    in.minage = p->minage;
    int *dout = (int *)(D + o_out);
    in.pos = dout;
    in.node = dout + std::max(cap, 1);
    in.time = dout + 2 * std::max(cap, 1);
    in.cap = cap;
    const double *dm = (const double *)(D + o_model);
    const RsModel m{p->ntimes, dm + M_TIMES, dm + M_TIMESTEPS, dm + M_COALSTEPS, dm + M_POPSIZES,
                    plan.model[M_CONST + 0]};
    int res[2] = {0, 0};
    std::vector<char> h(in_bytes);
    memcpy(h.data() + o_nodes, plan.nodes.data(), sizeof(int) * plan.nodes.size());
    memcpy(h.data() + o_bl, p->blocklens, sizeof(int) * p->ntrees);
    memcpy(h.data() + o_path, path, sizeof(int) * L);
    if (nu > 0) memcpy(h.data() + o_u, u, sizeof(double) * nu);
    memcpy(h.data() + o_model, plan.model.data(), sizeof(double) * MODEL_STRIDE);
    do {
        if ((rc = cudaMemcpy(D, h.data(), in_bytes, cudaMemcpyHostToDevice)) != cudaSuccess) break;
        RsTables *tables = (RsTables *)(D + o_tab);
        k_recomb_tables<<<(p->ntrees + 3) / 4, 128>>>(in, m, tables);
        note_launch();
        k_recomb_walk<<<1, 32>>>(in, m, tables, (int *)(D + o_res));
        note_launch();
        if ((rc = cudaGetLastError()) != cudaSuccess) break;
        if ((rc = cudaMemcpy(res, D + o_res, sizeof(res), cudaMemcpyDeviceToHost)) != cudaSuccess) break;
        if (res[0] > 0) {
            const int *dst[3] = {pos, node, time};
            const int *src[3] = {in.pos, in.node, in.time};
            for (int x = 0; x < 3 && rc == cudaSuccess; x++)
                rc = cudaMemcpy((void *)dst[x], src[x], sizeof(int) * res[0], cudaMemcpyDeviceToHost);
        }
    } while (false);
    cudaFree(D);
    if (rc != cudaSuccess) {
        err = std::string("sample_recombinations: ") + cudaGetErrorString(rc);
        return -3;
    }
    if (res[0] < 0) {
        err = res[0] == RS_BAD_STATE ? "sample_recombinations: a path entry is not a state of its tree"
            : res[0] == RS_OUT_OF_UNIFORMS ? "sample_recombinations: the uniforms ran out"
                                            : "sample_recombinations: more recombinations than cap";
        return -4;
    }
    if (used) *used = res[1];
    return res[0];
}

}  // namespace awg
