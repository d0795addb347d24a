// K2: emissions of a tree's variant columns (calc_emissions' non-invariant branch,
// emit.cpp:822-844), in FP64 as the reference forms them, or for the FP32 path in double-float,
// each as its ratio to the column's largest, rounded once.
//
// Per column: inner partials up the tree (likelihood_site_node_inner, emit.cpp:151-196), outer
// partials down it (likelihood_site_outer, emit.cpp:273-296), then calc_emit (emit.cpp:620-645)
// for the states; JC69 steps in the reference's order (FP64) or as P x = mut * sum(x) +
// (nomut - mut) * x.
//
// What bounds it: instructions at the states (about 200 each a column) and, in the tree passes,
// the chain of levels (some 15 up and 15 down at 64 leaves, few nodes on most of them) with the
// warps that an SM holds. So
//   - a warp carries several of the tree's columns up and down at once: a level's (node, column)
//     pairs are spread over the lanes, and the chain is paid once for the group;
//   - split-branch factors are read from tables per pair of time points, made once per instance
//     that a CTA serves, instead of six per state; a column's factor of the threaded leaf (or
//     cut subtree) depends on the state's time alone and is formed once per time;
//   - that leaves 12 + 32 / warps bytes of shared memory a state where there were 88 (and 8 a
//     warp), so 3 or 4 CTAs fit an SM where 1 or 2 did.
// 402,000 trees of 8 to 64 leaves, 37 columns each with 11 variant: 70.6 ms with a warp a column
// and factors by state, 47.7 ms so; 840 trees of 150 to 200 leaves at 32 time points: 6.28 and
// 1.26 ms. FP64 (the FP64 pipe, one SM a tree): 99 trees of 21 leaves 0.45 and 0.26 ms, 202 of 64
// leaves 1.55 and 1.38 ms.

#include <cuda_runtime.h>

#include <type_traits>

#include "df.cuh"
#include "emit_common.cuh"
#include "kernels.h"
#include "tree_util.cuh"

namespace awg {

namespace {

constexpr int WINDOW = 1024;  // columns whose variant ones are listed at a time
constexpr int GMAX = 8;       // columns a warp carries through the tree at once, at most
constexpr unsigned FULL = 0xffffffffu;

// JC69 factors of a branch: mut, and nomut - mut (double-float) or nomut (FP64)
template <typename R>
struct Factor;
template <>
struct Factor<df> {
    df m, d;
    __device__ Factor(df mut, df nomut) : m(mut), d(nomut - mut) {}
    __device__ explicit Factor(const float4 *t) {
        const float4 v = *t;
        m = df(v.x, v.y);
        d = df(v.z, v.w);
    }
    __device__ void store(float4 *t) const { *t = make_float4(m.hi, m.lo, d.hi, d.lo); }
};
template <>
struct Factor<double> {
    double m, d;
    __device__ Factor(double mut, double nomut) : m(mut), d(nomut) {}
    __device__ explicit Factor(const float4 *t) {
        const double2 v = *(const double2 *)t;
        m = v.x;
        d = v.y;
    }
    __device__ void store(float4 *t) const { *(double2 *)t = make_double2(m, d); }
};
__device__ __forceinline__ void load2(const float4 *p, df &a, df &b) {
    const float4 v = *p;
    a = df(v.x, v.y);
    b = df(v.z, v.w);
}
__device__ __forceinline__ void load2(const float4 *p, double &a, double &b) {
    const double2 v = *(const double2 *)p;
    a = v.x;
    b = v.y;
}
__device__ __forceinline__ void store2(float4 *p, df a, df b) { *p = make_float4(a.hi, a.lo, b.hi, b.lo); }
__device__ __forceinline__ void store2(float4 *p, double a, double b) { *(double2 *)p = make_double2(a, b); }

// An instance's branch factors by time points i <= j (entry tri(i) + j): every branch is a
// difference of two time points floored at mintime. Node branches and split branches round
// their probabilities differently, so each has its table.
__host__ __device__ inline int tri(int T, int i) { return i * (2 * T - 1 - i) / 2; }
__host__ __device__ inline int tri_size(int T) { return T * (T + 1) / 2; }

// A partial has NC components: 4 (bases) or, in a column whose observed calls all show one base
// X, 2 (X and any other: the leaves' are (1, 0) or, missing, (1, 1), and JC69 treats the other
// three alike; about 26% of all columns at 0.5% missing calls, 87% of the variant ones). Half h
// of the partials is an array of its own, so lanes on neighbouring pairs read without conflicts.
template <typename R, int NC>
struct Part {
    R x[NC];
    __device__ __forceinline__ void load(const float4 *p, int stride) {
#pragma unroll
        for (int h = 0; h < NC / 2; h++) load2(p + h * stride, x[2 * h], x[2 * h + 1]);
    }
    __device__ __forceinline__ void store(float4 *p, int stride) const {
#pragma unroll
        for (int h = 0; h < NC / 2; h++) store2(p + h * stride, x[2 * h], x[2 * h + 1]);
    }
    __device__ __forceinline__ void leaf(uint8_t ch) {
        if constexpr (NC == 2) {
            x[0] = df(1.0f, 0.0f);
            x[1] = ch == 'N' ? df(1.0f, 0.0f) : df();
        } else {
            leaf_partial<R>(ch, x);
        }
    }
    __device__ __forceinline__ void ones() {
#pragma unroll
        for (int a = 0; a < NC; a++) x[a] = R(1);
    }
    __device__ __forceinline__ Part step(const Factor<R> &f) const {
        Part y;
        if constexpr (std::is_same<R, double>::value) {
            jc_apply<false>(x, f.m, f.d, y.x);  // the reference's order
        } else {
            df sum;
            if constexpr (NC == 2) sum = df_addp(x[0], df(3.0f, 0.0f) * x[1]);
            else sum = (x[0] + x[1]) + (x[2] + x[3]);
            const df ms = f.m * sum;
#pragma unroll
            for (int a = 0; a < NC; a++) y.x[a] = df_addp(f.d * x[a], ms);
        }
        return y;
    }
    __device__ __forceinline__ Part operator*(const Part &o) const {
        Part y;
#pragma unroll
        for (int a = 0; a < NC; a++) y.x[a] = x[a] * o.x[a];
        return y;
    }
};

// A tree as the column passes see it.
struct Tree : TreeLevels {
    const float4 *nf;   // [n] a node's branch
    const float4 *st;   // split branches by time points
    const float4 *e0;   // external: the threaded leaf's branch by the state's time
    const int2 *states; // node | time << 16, table entry of the branch below | above << 16
    int S, T, age1;
};

// Bytes of a warp's area: the states' emissions, the factors by time and `cols` columns of
// partials in the four-component form.
__host__ __device__ inline int emis_bytes(int S) { return (8 * S + 15) & ~15; }
__host__ __device__ inline int warp_need(int n, int S, int T, int cols) {
    return emis_bytes(S) + 32 * T + 64 * n * cols;
}
// Bytes of the CTA's part.
__host__ __device__ inline int tables_bytes(int T) { return 16 * (2 * tri_size(T) + T); }
__host__ __device__ inline int tree_bytes(int n, int S) {
    return 32 * n + ((8 * S + 15) & ~15) + ((4 * (4 * n + 4) + 15) & ~15);
}

// G columns (window positions list[0 .. G)) of a tree by one warp.
template <typename R, int NC>
__device__ void emit_group(const BatchDev &d, const BlockDev &B, const InstDev &I, const Tree &t,
                           char *area, const uint16_t *list, int w0, int G, unsigned vword, double penalty) {
    const int lane = threadIdx.x & 31;
    const int4 *nd = t.nd;
    df *const ed = (df *)area;
    float4 *const p1s = (float4 *)(area + emis_bytes(t.S));
    const int half = t.n * G;  // distance of a partial's halves
    float4 *const in = p1s + 2 * t.T, *const out = in + (NC / 2) * half;
    const int inv = (65536 + G - 1) / G;  // x / G = x * inv >> 16 for x < 8192
    const uint8_t *seq = d.seqT + I.seq0;
    const int ns = I.nseqs, start = B.start + w0;

    for (int e = lane; e < t.inp[1] * G; e += 32) {
        const int x = e * inv >> 16, g = e - x * G, j = t.inl[x];
        Part<R, NC> p;
        p.leaf(seq[(size_t)(start + list[g]) * ns + j]);
        p.store(in + j * G + g, half);
    }
    __syncwarp();
    for (int h = 1; h < t.nlev_in; h++) {
        const int x0 = t.inp[h], m = (t.inp[h + 1] - x0) * G;
        for (int e = lane; e < m; e += 32) {
            const int x = e * inv >> 16, g = e - x * G, j = t.inl[x0 + x];
            const int c1 = nd[j].y, c2 = nd[j].z;
            Part<R, NC> a, b;
            a.load(in + c1 * G + g, half);
            b.load(in + c2 * G + g, half);
            (a.step(Factor<R>(t.nf + c1)) * b.step(Factor<R>(t.nf + c2))).store(in + j * G + g, half);
        }
        __syncwarp();
    }
    if (lane < G) {
        Part<R, NC> p;
        p.ones();
        p.store(out + t.mainr * G + lane, half);
    }
    __syncwarp();
    for (int h = 1; h < t.nlev_out; h++) {  // (level 0: the main root)
        const int x0 = t.outp[h], m = (t.outp[h + 1] - x0) * G;
        for (int e = lane; e < m; e += 32) {
            const int x = e * inv >> 16, g = e - x * G, j = t.outl[x0 + x];
            const int p = nd[j].x;
            const int4 np = nd[p];
            const int sib = np.y == j ? np.z : np.y;
            Part<R, NC> a;
            a.load(in + sib * G + g, half);
            a = a.step(Factor<R>(t.nf + sib));
            if (p != t.mainr) {
                Part<R, NC> b;
                b.load(out + p * G + g, half);
                a = a * b.step(Factor<R>(t.nf + p));
            }
            a.store(out + j * G + g, half);
        }
        __syncwarp();
    }

    for (int g = 0; g < G; g++) {
        const int col = start + list[g];
        // the threaded leaf's (or cut subtree's) factor by the state's time
        if (lane < t.T) {
            Part<R, NC> p;
            if (t.internal) p.load(in + t.node1 * G + g, half);
            else p.leaf(seq[(size_t)col * ns + t.nleaves]);
            p.step(Factor<R>(t.internal ? t.st + tri(t.T, t.age1) + imax(lane, t.age1) : t.e0 + lane))
                .store(p1s + lane, t.T);
        }
        __syncwarp();
        auto state_v = [&](int k) -> R {
            const int2 sk = t.states[k];
            const int node2 = sk.x & 0xffff;
            Part<R, NC> p1, p2, p3;
            p1.load(p1s + (sk.x >> 16), t.T);
            p2.load(in + node2 * G + g, half);
            p2 = p2.step(Factor<R>(t.st + (sk.y & 0xffff)));
            if constexpr (NC == 2) {
                if (node2 != t.mainr) {
                    p3.load(out + node2 * G + g, half);
                    p2 = p2 * p3.step(Factor<R>(t.st + (sk.y >> 16)));
                }
                return df_addp(p1.x[0] * p2.x[0], df(3.0f, 0.0f) * (p1.x[1] * p2.x[1]));
            } else {
                p1 = p1 * p2;
                if (node2 != t.mainr) {
                    p3.load(out + node2 * G + g, half);
                    p1 = p1 * p3.step(Factor<R>(t.st + (sk.y >> 16)));
                }
                if constexpr (std::is_same<R, double>::value) {
                    double v = 0;
#pragma unroll
                    for (int a = 0; a < 4; a++) v += p1.x[a] * .25;
                    return v;
                } else {
                    return ((p1.x[0] + p1.x[1]) + p1.x[2]) + p1.x[3];
                }
            }
        };
        const int vrow = d.colvar[I.col0 + col];
        if constexpr (std::is_same<R, double>::value) {
            // FP64: as they are; the states that break the infinite-sites model times the penalty
            double *row = d.varemit + B.var0 + (size_t)vrow * t.S;
            for (int kb = 0; kb < t.S; kb += 32) {
                const int k = imin(kb + lane, t.S - 1);
                double v = state_v(k);
                if (penalty < 1.0 && !state_ok(vword, t.states[k].x & 0xffff)) v *= penalty;
                if (kb + lane < t.S) row[k] = v;
            }
            __syncwarp();
        } else {
            // two states per lane at a time: independent chains the scheduler can interleave (the
            // second one repeats the first where it would run past S)
            df ref = df();
            for (int k0 = lane; k0 < t.S; k0 += 64) {
                const int k1 = k0 + 32 < t.S ? k0 + 32 : k0;
                const df v0 = state_v(k0), v1 = state_v(k1);
                ed[k0] = v0;
                ed[k1] = v1;
                ref = fmax(ref, fmax(v0, v1));
            }
            if (penalty < 1.0) {
                // states that break the infinite-sites model times the penalty (emit.cpp:847-862);
                // below FP32's range that leaves the ratio 0, written as the smallest negative
                // value below
                const df pen(penalty);
                ref = df();
                for (int kb = 0; kb < t.S; kb += 32) {
                    const int k = kb + lane;
                    const bool ok = state_ok(vword, k < t.S ? t.states[k].x & 0xffff : 0);
                    if (k < t.S) {
                        if (!ok) ed[k] = ed[k] * pen;
                        ref = fmax(ref, ed[k]);
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ref = fmax(ref, __shfl_xor_sync(FULL, ref, o));
            // 1 / (4 e_ref): the FP32 reciprocal and one Newton step in double-float
            const df one(1.0f, 0.0f);
            const df y0(1.0f / ref.hi, 0.0f);
            const df inv1 = y0 + y0 * (one - ref * y0);
            float *row = d.var32 + B.var0 + (size_t)vrow * t.S;
            for (int k = lane; k < t.S; k += 32) {
                // e_k / e_ref; the largest state's r can round a hair above 1, so its complement
                // is clamped at +0 (a negative value would read as a ratio, i.e. an emission near
                // zero)
                const df r = ed[k] * inv1;
                float v = r.hi >= 0.5f ? fmaxf((one - r).hi, 0.0f) : -r.hi;
                if (r.hi < 0.5f && v == 0.0f) v = -__int_as_float(1);  // stays a ratio
                row[k] = v;
            }
            if (lane == 0) d.vref[B.vrow0 + vrow] = .25 * (double)ref;
            __syncwarp();
        }
    }
}

// The variant columns of one tree, by the whole CTA.
template <typename R>
__device__ __forceinline__ void emit_tree(const BatchDev &d, int blk, int maxS, int smem_bytes, int &cached) {
    extern __shared__ int4 dyn[];
    __shared__ double times[MAXT];
    __shared__ int nlev_in, nlev_out, nnear, nother, taken;
    __shared__ uint16_t list[WINDOW];
    const BlockDev B = d.blocks[blk];
    const InstDev I = d.inst[B.inst];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x, nwarps = nthreads >> 5;
    constexpr bool FP32 = std::is_same<R, df>::value;  // else the plain FP64 path
    if (B.nvar == 0 || B.S == 0) {
        if (FP32 && warp == 0) block_log_offset(d, B, I, blk, lane);
        return;
    }
    const int T = I.T, n = I.nnodes, S = B.S;
    const bool internal = I.internal != 0;
    if (S > maxS || n > d.maxnodes || n < 1) {
        if (tid == 0) report_error(d.err, ERR_PLAN_MISMATCH, B.inst, B.b, B.start);
        return;
    }
    char *const base = (char *)dyn;
    float4 *const st = (float4 *)base, *const nt = st + tri_size(T), *const e0 = nt + tri_size(T);
    int4 *const nd = (int4 *)(base + tables_bytes(d.maxT));
    float4 *const nf = (float4 *)(nd + n);
    int2 *const states = (int2 *)(nf + n);
    int *const inl = (int *)((char *)states + ((8 * S + 15) & ~15)), *const outl = inl + n;
    int *const inp = outl + n, *const outp = inp + n + 2;  // [n + 2] each
    const int warps0 = tables_bytes(d.maxT) + tree_bytes(n, S);
    const int area_bytes = (smem_bytes - warps0) / nwarps & ~15;
    if (area_bytes < warp_need(n, S, T, 1)) {
        if (tid == 0) report_error(d.err, ERR_SMEM_LIMIT, B.inst, B.b, B.start);
        return;
    }
    char *const area = base + warps0 + warp * area_bytes;
    int *const hgt = (int *)(base + warps0), *const dep = hgt + n, *const cur1 = dep + n, *const cur2 = cur1 + n;

    const double *model = d.model + I.model0;
    const double mu = model[M_CONST + 1], mintime = model[M_CONST + 2];
    const double penalty = model[M_CONST + 3];  // infinite-sites penalty, 1: off
    const int root = B.root;
    // nodes, states, and the indices that the passes use as addresses
    bool bad = root < 0 || root >= n;
    for (int i = tid; i < n; i += nthreads) {
        const int4 v = d.nodes[B.nodes0 + i];
        bad |= v.x < -1 || v.x >= n || v.y < -1 || v.y >= n || v.z < -1 || v.z >= n || v.w < 0 || v.w > T + 1;
        nd[i] = v;
        hgt[i] = 0;
    }
    for (int k = tid; k < S; k += nthreads) {
        const StateInfo si = d.sinfo[B.state0 + k];
        bad |= si.node < 0 || si.node >= n || si.time < 0 || si.time >= T;
        states[k] = make_int2(si.node | si.time << 16, 0);
    }
    const bool refill = cached != B.inst;  // read by all before anyone rewrites it
    if (refill)
        for (int i = tid; i < T; i += nthreads) times[i] = model[M_TIMES + i];
    if (tid == 0) nnear = nother = taken = 0;
    if (__syncthreads_or(bad)) {
        if (tid == 0) report_error(d.err, ERR_BOUNDS, B.inst, B.b, B.start);
        return;
    }
    if (refill) {
        auto split = [&](double e, float4 *at) {  // a split branch's factors
            if constexpr (FP32) {  // branch_mut / branch_nomut in double-float
                const df quarter(0.25f, 0.0f), one(1.0f, 0.0f), three(3.0f, 0.0f), ex(e);
                Factor<df>(quarter * (one - ex), quarter * (one + three * ex)).store(at);
            } else {
                Factor<double>(branch_mut(e), branch_nomut(e)).store(at);
            }
        };
        for (int e = tid; e < T * T; e += nthreads) {
            const int i = e / T, j = e - i * T;
            if (j < i) continue;
            const double x = branch_exp(fmax(times[j] - times[i], mintime), mu);
            split(x, st + tri(T, i) + j);
            Factor<R>(R(branch_mut(x)), R(branch_nomut(x))).store(nt + tri(T, i) + j);
        }
        for (int j = tid; j < T; j += nthreads) split(branch_exp(fmax(times[j] - 0.0, mintime), mu), e0 + j);
        if (tid == 0) cached = B.inst;
    }
    // a branch's entry; ages beyond the time grid (which no branch of a valid tree has) are
    // taken at its end, as a bound on the address
    auto entry = [&](int lo, int hi) {
        lo = imin(lo, T - 1);
        return tri(T, lo) + imax(lo, imin(hi, T - 1));
    };
    const int mainr = internal ? nd[root].z : root, node1 = internal ? nd[root].y : 0;
    if (internal && (mainr < 0 || node1 < 0)) {
        if (tid == 0) report_error(d.err, ERR_BOUNDS, B.inst, B.b, B.start);
        return;
    }
    for (int k = tid; k < S; k += nthreads) {  // split branches below and above (emit.cpp:782-805)
        const int2 s = states[k];
        const int4 v = nd[s.x & 0xffff];
        const int a = s.x >> 16;
        states[k].y = entry(v.w, a) | (v.x != -1 ? entry(a, nd[v.x].w) : 0) << 16;
    }
    // level schedules: heights (longest path down to a leaf; leaves 0) and depths below the main
    // root (-1 outside its subtree), each bucketed by one warp. Walks are bounded by n steps.
    for (int i = tid; i < n; i += nthreads) {
        const bool leaf = nd[i].y == -1;
        int found = i == mainr ? 0 : -1;
        for (int v = i, dd = 1; dd <= n && nd[v].x != -1; dd++) {
            v = nd[v].x;
            if (v == mainr) found = dd;
            if (leaf) atomicMax(&hgt[v], dd);
            else if (found >= 0) break;
        }
        dep[i] = found;
    }
    __syncthreads();
    if (warp == 0) {
        const int nl = warp_levels(hgt, n, inl, inp, cur1, lane);
        if (lane == 0) nlev_in = nl;
    }
    if (warp == imin(1, nwarps - 1)) {
        const int nl = warp_levels(dep, n, outl, outp, cur2, lane);
        if (lane == 0) nlev_out = nl;
    }
    for (int i = tid; i < n; i += nthreads) {  // prob_tree_mutation (emit.cpp:97-116)
        const int pa = nd[i].x != -1 && i != root ? nd[nd[i].x].w : T + 1;
        nf[i] = pa != T + 1 ? nt[entry(nd[i].w, pa)] : make_float4(0.f, 0.f, 0.f, 0.f);
    }

    const uint8_t *cls = d.colclass + I.col0 + B.start;
    const int ns = I.nseqs;
    for (int w0 = 0; w0 < B.len; w0 += WINDOW) {
        // the window's variant columns: those whose observed calls all show one base from the
        // list's front, the others from its back
        const int len = imin(WINDOW, B.len - w0);
        int seen = 0;
        for (int b0 = 0; b0 < len; b0 += 32) {
            const int i = b0 + lane;
            unsigned mm = __ballot_sync(FULL, i < len && cls[w0 + i] == COL_VARIANT);
            for (; mm; mm &= mm - 1) {
                if (seen++ % nwarps != warp) continue;
                const int c = b0 + __ffs(mm) - 1;
                const int vrow = d.colvar[I.col0 + B.start + w0 + c];
                if (vrow < 0 || vrow >= B.nvar) {
                    if (lane == 0) report_error(d.err, ERR_BOUNDS, B.inst, B.b, B.start + w0 + c);
                    continue;
                }
                const uint8_t *chars = d.seqT + I.seq0 + (size_t)(B.start + w0 + c) * ns;
                if (!FP32) {
                    if (lane == 0) list[WINDOW - 1 - atomicAdd(&nother, 1)] = (uint16_t)c;
                    continue;
                }
                unsigned have = 0;  // bases seen: bits of the upper-case letters' low five bits
                for (int j = lane; j < ns; j += 32) {
                    const uint8_t ch = chars[j];
                    if (ch != 'N') have |= 1u << (ch & 31);
                }
                have = __reduce_or_sync(FULL, have);
                if (lane == 0) {
                    if (__popc(have) == 1) list[atomicAdd(&nnear, 1)] = (uint16_t)c;
                    else list[WINDOW - 1 - atomicAdd(&nother, 1)] = (uint16_t)c;
                }
            }
        }
        __syncthreads();
        const Tree t{{nd, inl, inp, outl, outp, nlev_in, nlev_out, mainr, node1, I.nleaves, n, internal},
                     nf, st, e0, states, S, T, imin(nd[node1].w, T - 1)};
        // groups of columns, as even as the warps' areas allow; the four-component ones first
        const int room = area_bytes - warp_need(n, S, T, 0);
        const int cap4 = penalty < 1.0 ? 1 : imin(GMAX, room / (64 * n));
        const int cap2 = penalty < 1.0 ? 1 : imin(GMAX, room / (32 * n));
        const int no = nother, nn = nnear;
        const int g4 = imax(1, imin(cap4, (no + nwarps - 1) / nwarps)), ng4 = (no + g4 - 1) / g4;
        const int g2 = imax(1, imin(cap2, (nn + nwarps - 1) / nwarps)), ng2 = (nn + g2 - 1) / g2;
        while (true) {
            int q = 0;
            if (lane == 0) q = atomicAdd(&taken, 1);
            q = __shfl_sync(FULL, q, 0);
            if (q >= ng4 + ng2) break;
            const bool near = q >= ng4;
            const int f = near ? (q - ng4) * g2 : q * g4;
            const int G = near ? imin(g2, nn - f) : imin(g4, no - f);
            const uint16_t *ls = near ? list + f : list + WINDOW - f - G;
            unsigned vword = FULL;
            if (penalty < 1.0)  // (one column a group)
                vword = infsites_nodes(t, d.seqT + I.seq0 + (size_t)(B.start + w0 + ls[0]) * ns, (uint8_t *)area,
                                       (uint8_t *)area + n);
            __syncwarp();
            if constexpr (FP32) {
                if (near) emit_group<df, 2>(d, B, I, t, area, ls, w0, G, vword, penalty);
                else emit_group<df, 4>(d, B, I, t, area, ls, w0, G, vword, penalty);
            } else {
                emit_group<double, 4>(d, B, I, t, area, ls, w0, G, vword, penalty);
            }
        }
        __syncthreads();
        if (tid == 0) nnear = nother = taken = 0;
        __syncthreads();
    }
    if (FP32 && warp == 0) block_log_offset(d, B, I, blk, lane);
}

template <typename R>
__global__ void __launch_bounds__(256, 2) k_varemit_groups(BatchDev d, int maxS, int smem_bytes, WorkQueue q) {
    __shared__ int cached;  // instance whose factor tables are in place
    if (threadIdx.x == 0) cached = -1;
    __syncthreads();
    if (!q.counter) {
        emit_tree<R>(d, cta_block(d), maxS, smem_bytes, cached);
        return;
    }
    for (int u = next_unit(q); u >= 0; u = next_unit(q)) {
        const int t1 = imin((u + 1) * q.chunk, d.nblocks);
        for (int t = u * q.chunk; t < t1; t++) {
            emit_tree<R>(d, d.blkmap ? d.blkmap[t] : t, maxS, smem_bytes, cached);
            __syncthreads();
        }
    }
}

template <typename R>
void launch(const BatchDev &d, cudaStream_t s, int *queue, int chunk) {
    const int n = imax(d.maxnodes, 1), S = imax(d.maxS, 1), T = d.maxT;
    constexpr int SM_BYTES = 227 * 1024, STATIC = 4 * 1024;
    auto need = [&](int w) { return tables_bytes(T) + tree_bytes(n, S) + w * (warp_need(n, S, T, 1) + 16); };
    // as many CTAs of four warps an SM as hold a four-component column of the largest tree each;
    // smaller trees carry more columns at once in the same room. Past two, one CTA of up to eight
    // warps (a tree's states then take most of the room, and the CTA's part is held once).
    int ctas = 4, warps = 4;
    while (ctas > 1 && need(warps) > SM_BYTES / ctas - STATIC) ctas--;
    int smem = SM_BYTES / ctas - STATIC;
    if (ctas == 1) {
        warps = 8;
        while (warps > 1 && need(warps) > smem) warps--;
    }
    smem &= ~15;
    prefer_shared(k_varemit_groups<R>);
    if (!raise_dynamic_smem(k_varemit_groups<R>, smem)) return;
    WorkQueue q{queue, d.nblocks, 1};
    int grid = d.nblocks;
    if (queue) {
        // a unit's trees are mostly one instance's, whose factor tables are then made once: up
        // to 8 trees, while the queue still holds several units a CTA
        grid = persistent_grid(k_varemit_groups<R>, 32 * warps, smem, d.nblocks);
        q.chunk = imax(imax(chunk, 1), imin(8, d.nblocks / (8 * grid)));
        q.nunits = (d.nblocks + q.chunk - 1) / q.chunk;
        grid = imin(grid, q.nunits);
    }
    k_varemit_groups<R><<<grid, 32 * warps, smem, s>>>(d, S, smem, q);
    note_launch();
}

}  // namespace

void launch_varemit_groups(const BatchDev &d, bool fp32, cudaStream_t s, int *queue, int chunk) {
    if (fp32) launch<df>(d, s, queue, chunk);
    else launch<double>(d, s, queue, chunk);
}

}  // namespace awg
