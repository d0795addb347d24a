// Host plan of a batch of threading problems.
//
// The host does only O(nodes) work per local tree and one pass over the sequences:
// validation, child arrays (the reference's set_ptree, local_tree.h:190-230), state-space
// sizes (states.cpp:53-199) for the memory layout, node mappings (make_node_mapping,
// local_tree.h:767), the model's time grid (model.h:322-333, model.cpp:9-23) and the
// column classes of the emission step (emit.cpp:30-58). Everything numeric runs on the GPU.

#include "plan.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>

namespace awg {

// An instance's model block (model.h:322-333, model.cpp:9-23): times, popsizes (zeros when
// NULL), time_steps, coal_time_steps, rho, mu, mintime and the infinite-sites penalty.
void model_arrays(const double *times, const double *popsizes, int T, double rho, double mu,
                  double penalty, double *m) {
    for (int i = 0; i < MODEL_STRIDE; i++) m[i] = 0.0;
    for (int i = 0; i < T; i++) {
        m[M_TIMES + i] = times[i];
        m[M_POPSIZES + i] = popsizes ? popsizes[i] : 0.0;
    }
    for (int i = 0; i < T - 1; i++) m[M_TIMESTEPS + i] = times[i + 1] - times[i];
    m[M_TIMESTEPS + T - 1] = INFINITY;
    std::vector<double> times2(2 * T + 1, 0.0);
    for (int i = 0; i < T - 1; i++) {
        times2[2 * i] = times[i];
        times2[2 * i + 1] = std::sqrt((times[i + 1] + 1.0) * (times[i] + 1.0));
    }
    times2[2 * T - 2] = times2[2 * T - 1] = times2[2 * T] = times[T - 1];
    for (int i = 0; i < 2 * T - 2; i++)
        m[M_COALSTEPS + i] = times2[std::min(i + 1, 2 * T)] - times2[i];
    m[M_COALSTEPS + 2 * T - 2] = INFINITY;
    m[M_COALSTEPS + 2 * T - 1] = INFINITY;
    m[M_CONST + 0] = rho;
    m[M_CONST + 1] = mu;
    m[M_CONST + 2] = times[1] * .1;
    m[M_CONST + 3] = (penalty > 0.0 && penalty < 1.0) ? penalty : 1.0;
}


namespace {

struct TreeScratch {
    int c0[MAXNODES], c1[MAXNODES];
};

// Children in index order (set_ptree), root, optional child[0] override of the root.
bool make_children(const int *parent, int n, int rc0, TreeScratch &ts, int &root) {
    for (int i = 0; i < n; i++) ts.c0[i] = ts.c1[i] = -1;
    root = -1;
    for (int i = 0; i < n; i++) {
        int p = parent[i];
        if (p < -1 || p >= n) return false;
        if (p == -1) {
            if (root != -1) return false;
            root = i;
        } else if (ts.c0[p] == -1) {
            ts.c0[p] = i;
        } else if (ts.c1[p] == -1) {
            ts.c1[p] = i;
        } else {
            return false;
        }
    }
    if (root < 0) return false;
    if (rc0 != -1 && ts.c0[root] != rc0) {
        if (ts.c1[root] != rc0) return false;
        std::swap(ts.c0[root], ts.c1[root]);
    }
    return true;
}

}  // namespace

int count_states(const int *parent, const int *age, int n, int T, bool internal, int minage,
                 int root_child0, int *M_out) {
    TreeScratch ts;
    int root;
    if (!make_children(parent, n, root_child0, ts, root)) return -1;
    long long S = 0, M = 0;
    if (!internal) {
        for (int i = 0; i < n; i++) {
            int top = parent[i] == -1 ? T - 2 : age[parent[i]];
            int m = std::max(0, top - age[i] + 1);
            S += m;
            M += (long long)m * m;
        }
    } else {
        if (age[root] < T) {
            if (M_out) *M_out = 0;
            return 0;
        }
        const int sub = ts.c0[root];
        if (sub >= 0) minage = std::max(minage, age[sub]);
        bool in_sub[MAXNODES] = {};
        int stack[MAXNODES], top_of = 0;
        if (sub >= 0) stack[top_of++] = sub;
        while (top_of > 0) {
            const int v = stack[--top_of];
            in_sub[v] = true;
            if (ts.c0[v] >= 0) stack[top_of++] = ts.c0[v];
            if (ts.c1[v] >= 0) stack[top_of++] = ts.c1[v];
        }
        for (int i = 0; i < n; i++) {
            if (i == root || in_sub[i]) continue;
            int t0 = std::max(age[i], minage);
            int top = parent[i] == root ? T - 2 : age[parent[i]];
            int m = std::max(0, top - t0 + 1);
            S += m;
            M += (long long)m * m;
        }
    }
    if (M_out) *M_out = (int)M;
    return (int)S;
}

thread_local int g_plan_threads = 0;
void set_plan_threads(int n) { g_plan_threads = std::max(0, n); }

// Threads take the tasks in order from a shared counter. A thread costs some 20 us to start, so
// there is one per 100 us of work (four problems of 3,000 columns were planned in 0.34 ms with a
// thread each, in 0.11 ms by the calling one).
void parallel_tasks(int n, double ns, const std::function<void(int)> &f) {
    const int hw = g_plan_threads > 0 ? g_plan_threads : (int)std::thread::hardware_concurrency();
    const int nthreads = std::max(1, std::min(std::min(n, hw), (int)std::min(ns / 100e3, 1e6)));
    std::atomic<int> next(0);
    auto work = [&]() {
        for (int k = next.fetch_add(1); k < n; k = next.fetch_add(1)) f(k);
    };
    std::vector<std::thread> pool;
    try {
        for (int t = 1; t < nthreads; t++) pool.emplace_back(work);
    } catch (const std::exception &) {  // fewer threads than wanted
    }
    work();
    for (auto &th : pool) th.join();
}

void parallel_copy(const std::vector<HostCopy> &copies) {
    constexpr size_t PART = 256 * 1024;
    struct Part {
        const HostCopy *c;
        size_t off;
    };
    std::vector<Part> parts;
    double bytes = 0;
    for (const HostCopy &c : copies) {
        for (size_t o = 0; o < c.bytes; o += PART) parts.push_back({&c, o});
        bytes += (double)c.bytes;
    }
    parallel_tasks((int)parts.size(), bytes * 0.2, [&](int k) {
        const HostCopy &c = *parts[k].c;
        memcpy((char *)c.dst + parts[k].off, (const char *)c.src + parts[k].off, std::min(PART, c.bytes - parts[k].off));
    });
}

namespace {

// A problem's trees [b0, b1): the work is shared out by these, so that a batch of one problem
// is planned by several threads too.
struct Unit {
    int q, b0, b1;
};
// Units of about 100 us (ns(p, b): a tree's share), and the batch's total.
template <typename Cost>
std::vector<Unit> make_units(const awg_problem *probs, int n, Cost ns, double &total) {
    std::vector<Unit> units;
    total = 0;
    for (int q = 0; q < n; q++) {
        int b0 = 0;
        double sum = 0;
        for (int b = 0; b < probs[q].ntrees; b++) {
            sum += ns(probs[q], b);
            if (sum < 100e3 && b + 1 < probs[q].ntrees) continue;
            units.push_back({q, b0, b + 1});
            total += sum;
            b0 = b + 1;
            sum = 0;
        }
    }
    return units;
}

// 1 for a byte outside A, C, G, T, N (either case of ACGT)
inline uint8_t bad_base(uint8_t c) {
    const uint8_t u = c & 0xDF;  // ACGT upper-cased; 'n' stays apart from 'N'
    return !((u == 'A') | (u == 'C') | (u == 'G') | (u == 'T') | (c == 'N'));
}

// 16 bytes at a time (GCC vectors: the same on every machine); nonzero where bad_base is 1
typedef uint8_t Bytes16 __attribute__((vector_size(16)));
inline Bytes16 load16(const uint8_t *p) {
    Bytes16 v;
    memcpy(&v, p, 16);
    return v;
}
inline Bytes16 bad_bases(Bytes16 c) {
    const Bytes16 u = c & (uint8_t)0xDF;
    return (Bytes16) ~((u == (uint8_t)'A') | (u == (uint8_t)'C') | (u == (uint8_t)'G') | (u == (uint8_t)'T') |
                       (c == (uint8_t)'N'));
}

// An 8 x 8 byte block transposed in registers: x[k] holds row k, byte j (little endian)
// column j; afterwards x[j] holds column j. Three rounds swap 4x4, 2x2 and 1x1 sub-blocks.
inline void transpose8x8(uint64_t x[8]) {
    for (int k = 0; k < 4; k++) {
        const uint64_t t = ((x[k] >> 32) ^ x[k + 4]) & 0x00000000FFFFFFFFull;
        x[k] ^= t << 32;
        x[k + 4] ^= t;
    }
    for (int a : {0, 1, 4, 5}) {
        const uint64_t t = ((x[a] >> 16) ^ x[a + 2]) & 0x0000FFFF0000FFFFull;
        x[a] ^= t << 16;
        x[a + 2] ^= t;
    }
    for (int a : {0, 2, 4, 6}) {
        const uint64_t t = ((x[a] >> 8) ^ x[a + 1]) & 0x00FF00FF00FF00FFull;
        x[a] ^= t << 8;
        x[a + 1] ^= t;
    }
}

// What a problem holds beside its trees; nullptr or what is wrong with it.
const char *check_header(const awg_problem &p, bool check_seqs) {
    if (p.ntrees < 1) return "ntrees < 1";
    if (p.nnodes < 1 || p.nnodes > MAXNODES) return "nnodes out of range [1, 1024]";
    if (p.ntimes < 3 || p.ntimes > MAXT) return "ntimes out of range [3, 32]";
    if (!p.ptrees || !p.ages || !p.sprs || !p.blocklens || !p.times || !p.popsizes || !p.seqs)
        return "missing input array";
    const int nleaves = (p.nnodes + 1) / 2;
    const int nemit = p.internal ? nleaves : nleaves + 1;
    if (p.nseqs < nemit) return "fewer sequences than leaves (+1 when external)";
    if (p.minage < 0) return "negative minage";
    long long L = 0;
    for (int b = 0; b < p.ntrees; b++) {
        if (p.blocklens[b] < 1) return "block length < 1";
        L += p.blocklens[b];
    }
    if (L != p.seqlen) return "block lengths do not add up to seqlen";
    if (p.seqlen < 1) return "seqlen < 1";
    for (int i = 0; i < p.ntimes; i++)
        if (!(p.times[i] >= 0) || !(p.popsizes[i] > 0)) return "bad times or popsizes";
    for (int i = 1; i < p.ntimes; i++)
        if (!(p.times[i] > p.times[i - 1])) return "times not increasing";
    if (check_seqs) {
        unsigned bad = 0;
        for (long long c = 0; c < (long long)nemit * p.seqlen; c++) bad |= bad_base((uint8_t)p.seqs[c]);
        if (bad) return "sequence byte outside A,C,G,T,N";
    }
    return nullptr;
}

// States (S) and same-branch row entries (M) of an external tree, its shape and ages checked in
// the same pass; nullptr or what is wrong with it.
const char *external_tree(const int *par, const int *age, int n, int T, int rc0, int &S, int &M) {
    uint8_t kids[MAXNODES];
    memset(kids, 0, n);
    int roots = 0, root = -1;
    bool bad_age = false, bad_tree = false;
    long long s = 0, mm = 0;
    for (int i = 0; i < n; i++) {
        const int p = par[i], a = age[i];
        bad_age |= a < 0 || a > T - 2;
        int top = T - 2;
        if (p >= 0 && p < n) {
            bad_tree |= kids[p] >= 2;
            kids[p] += kids[p] < 2;
            top = age[p];
        } else {
            bad_tree |= p != -1;
            roots++;
            root = i;
        }
        const long long m = top >= a ? (long long)top - a + 1 : 0;
        s += m;
        mm += m * m;
    }
    if (bad_age) return "node age out of range";
    if (bad_tree || roots != 1) return "malformed tree (parents/children)";
    if (rc0 != -1 && (rc0 < 0 || rc0 >= n || par[rc0] != root)) return "malformed tree (parents/children)";
    if (s == 0) return "external tree with no states";
    S = (int)s;
    M = (int)mm;
    return nullptr;
}

// Trees [b0, b1) of a problem whose header is sound: checks, states and row entries of each.
const char *check_trees(const awg_problem &p, int b0, int b1, int *S_of, int *M_of) {
    for (int b = b0; b < b1; b++) {
        const int *par = p.ptrees + (size_t)b * p.nnodes;
        const int *age = p.ages + (size_t)b * p.nnodes;
        const int rc0 = p.root_child0 ? p.root_child0[b] : -1;
        if (!p.internal) {
            if (const char *e = external_tree(par, age, p.nnodes, p.ntimes, rc0, S_of[b], M_of[b])) return e;
        } else {
            for (int i = 0; i < p.nnodes; i++)
                if (age[i] < 0 || age[i] > p.ntimes + 1) return "node age out of range";
            S_of[b] = count_states(par, age, p.nnodes, p.ntimes, true, p.minage, rc0, &M_of[b]);
            if (S_of[b] < 0) return "malformed tree (parents/children)";
        }
        if (b > 0) {
            const int *s = p.sprs + (size_t)b * 4;
            if (s[0] < 0 || s[0] >= p.nnodes || s[2] < 0 || s[2] >= p.nnodes) return "SPR nodes out of range";
            if (s[1] < 0 || s[1] >= p.ntimes || s[3] < 0 || s[3] >= p.ntimes) return "SPR times out of range";
            const int *prev = p.ptrees + (size_t)(b - 1) * p.nnodes;
            if (prev[s[0]] < 0) return "SPR recombines the root";
        }
    }
    return nullptr;
}

std::string problem_error(int q, const char *what) {
    char buf[256];
    snprintf(buf, sizeof(buf), "problem %d: %s", q, what);
    return std::string(buf);
}

}  // namespace

bool plan_layout(const awg_problem *probs, int n, HostPlan &plan, std::string &err,
                 bool check_seqs) {
    plan = HostPlan();
    if (n <= 0) { err = "empty batch"; return false; }
    plan.ninst = n;
    plan.inst.resize(n);

    // pass 1: validation and sizes, by units of trees, with each unit's totals. Problems before
    // the first one whose header is unsound are looked through first: theirs is the first error.
    int sound = 0;
    const char *wrong = nullptr;
    while (sound < n && !wrong)
        if (!(wrong = check_header(probs[sound], check_seqs))) sound++;
    double cost = 0;
    const std::vector<Unit> units = make_units(
        probs, sound, [](const awg_problem &p, int) { return 30.0 + (p.internal ? 8.0 : 2.5) * p.nnodes; }, cost);
    std::vector<int> tree0(sound + 1, 0);  // a problem's first tree among the batch's
    for (int q = 0; q < sound; q++) tree0[q + 1] = tree0[q] + probs[q].ntrees;
    std::vector<int> S_of(tree0[sound]), M_of(tree0[sound]);
    struct Tot {
        long long cells = 0, states = 0, t2 = 0;
        int cols = 0, maxS = 1, maxM = 1, maxlen = 1;
        const char *wrong = nullptr;
    };
    std::vector<Tot> tot(units.size());
    parallel_tasks((int)units.size(), cost, [&](int k) {
        const Unit &u = units[k];
        const awg_problem &p = probs[u.q];
        int *S = S_of.data() + tree0[u.q], *M = M_of.data() + tree0[u.q];
        Tot &t = tot[k];
        if ((t.wrong = check_trees(p, u.b0, u.b1, S, M))) return;
        for (int b = u.b0; b < u.b1; b++) {
            const int len = p.blocklens[b];
            t.cells += (long long)len * std::max(S[b], 1);
            t.states += std::max(S[b], 1);  // a zero-state space still takes one slot
            t.t2 += M[b];
            t.cols += len;
            t.maxS = std::max(t.maxS, S[b]);
            t.maxM = std::max(t.maxM, M[b]);
            t.maxlen = std::max(t.maxlen, len);
        }
    });
    for (size_t k = 0; k < units.size(); k++)
        if (tot[k].wrong) { err = problem_error(units[k].q, tot[k].wrong); return false; }
    if (wrong) { err = problem_error(sound, wrong); return false; }

    // offsets: prefixes over the units, which are in the order of the trees
    struct Off {
        long long cell, st, t2;
        int start;
    };
    std::vector<Off> off(units.size());
    long long cell = 0, col = 0, st = 0, t2 = 0, nodes = 0, map = 0, seq = 0;
    size_t k = 0;
    long long trees = 0;
    plan.model.assign((size_t)n * MODEL_STRIDE, 0.0);
    for (int q = 0; q < n; q++) {
        const awg_problem &p = probs[q];
        const int nleaves = (p.nnodes + 1) / 2;
        const int nemit = p.internal ? nleaves : nleaves + 1;
        InstDev &I = plan.inst[q];
        I.T = p.ntimes; I.internal = p.internal ? 1 : 0; I.minage = p.minage;
        I.nleaves = nleaves; I.nnodes = p.nnodes; I.nseqs = nemit; I.seqlen = p.seqlen;
        I.ntrees = p.ntrees; I.block0 = (int)trees; I.maxS = I.maxM = 1; I.pad = 0;
        I.cell0 = cell; I.col0 = col; I.seq0 = seq; I.model0 = (long long)q * MODEL_STRIDE;
        model_arrays(p.times, p.popsizes, p.ntimes, p.rho, p.mu, p.infsites_penalty,
                     &plan.model[(size_t)q * MODEL_STRIDE]);
        int start = 0;
        for (; k < units.size() && units[k].q == q; k++) {
            off[k] = Off{cell, st, t2, start};
            cell += tot[k].cells;
            st += tot[k].states;
            t2 += tot[k].t2;
            start += tot[k].cols;
            I.maxS = std::max(I.maxS, tot[k].maxS);
            I.maxM = std::max(I.maxM, tot[k].maxM);
            plan.maxlen = std::max(plan.maxlen, tot[k].maxlen);
        }
        plan.maxS = std::max(plan.maxS, I.maxS);
        plan.maxM = std::max(plan.maxM, I.maxM);
        plan.maxnodes = std::max(plan.maxnodes, p.nnodes);
        plan.maxT = std::max(plan.maxT, p.ntimes);
        nodes += (long long)p.ntrees * p.nnodes;
        map += (long long)(p.ntrees - 1) * p.nnodes;
        col += p.seqlen;
        seq += (long long)p.seqlen * nemit;
        trees += p.ntrees;
    }
    plan.nblocks = (int)trees;
    plan.blocks.resize(trees);

    // pass 2: block descriptors
    std::vector<long long> nodes0(n), map0(n);
    for (int q = 1; q < n; q++) {
        nodes0[q] = nodes0[q - 1] + (long long)probs[q - 1].ntrees * probs[q - 1].nnodes;
        map0[q] = map0[q - 1] + (long long)(probs[q - 1].ntrees - 1) * probs[q - 1].nnodes;
    }
    parallel_tasks((int)units.size(), 40.0 * trees, [&](int k) {
        const Unit &u = units[k];
        const awg_problem &p = probs[u.q];
        const int *S = S_of.data() + tree0[u.q], *M = M_of.data() + tree0[u.q];
        long long cellq = off[k].cell, stq = off[k].st, t2q = off[k].t2;
        int pos = off[k].start, blk = tree0[u.q] + u.b0;
        for (int b = u.b0; b < u.b1; b++, blk++) {
            BlockDev &B = plan.blocks[blk];
            memset(&B, 0, sizeof(B));
            B.inst = u.q; B.b = b; B.start = pos; B.len = p.blocklens[b];
            B.S = S[b];
            B.S1 = b > 0 ? S[b - 1] : 0;
            B.nodes0 = (int)(nodes0[u.q] + (long long)b * p.nnodes);
            B.prev_nodes0 = b > 0 ? B.nodes0 - p.nnodes : -1;
            const int *s = p.sprs + (size_t)b * 4;
            for (int x = 0; x < 4; x++) B.spr[x] = b > 0 ? s[x] : -1;
            B.map0 = b > 0 ? (int)(map0[u.q] + (long long)(b - 1) * p.nnodes) : -1;
            B.M = M[b];
            B.cell0 = cellq;
            B.state0 = stq;
            B.prev_state0 = b > 0 ? stq - std::max(S[b - 1], 1) : -1;
            B.gptr0 = stq + blk;
            B.t2_0 = t2q;
            cellq += (long long)B.len * std::max(B.S, 1);
            stq += std::max(B.S, 1);
            t2q += B.M;
            pos += B.len;
        }
    });
    plan.total_cells = cell; plan.total_cols = col; plan.total_states = st;
    plan.total_M = t2; plan.total_nodes = nodes; plan.total_map = map; plan.total_seq = seq;
    return true;
}

bool plan_fill(const awg_problem *probs, int n, HostPlan &plan, const PlanDst &out,
               std::string *err, const double *const *uniforms) {
    // pass 3: arrays, by units of trees, straight into the caller's buffers
    double cost = 0;
    const std::vector<Unit> units = make_units(
        probs, n,
        [&](const awg_problem &p, int b) {
            return 4.0 * p.nnodes + p.blocklens[b] * (4.0 + 0.5 * p.nseqs);
        },
        cost);
    std::vector<uint8_t> bad_seqs(n, 0);
    parallel_tasks((int)units.size(), cost, [&](int k) {
        const Unit &unit = units[k];
        const int q = unit.q;
        const awg_problem &p = probs[q];
        const InstDev &I = plan.inst[q];
        TreeScratch ts;
        int prev_root = -1;
        for (int b = std::max(unit.b0 - 1, 0); b < unit.b1; b++) {
            const int *par = p.ptrees + (size_t)b * p.nnodes;
            const int *age = p.ages + (size_t)b * p.nnodes;
            int root;
            const int rc0 = p.root_child0 ? p.root_child0[b] : -1;
            make_children(par, p.nnodes, rc0, ts, root);
            if (b >= unit.b0) {
                BlockDev &B = plan.blocks[I.block0 + b];
                B.root = root;
                int *nd = out.nodes + (size_t)B.nodes0 * 4;
                for (int i = 0; i < p.nnodes; i++) {
                    nd[4 * i + 0] = par[i];
                    nd[4 * i + 1] = ts.c0[i];
                    nd[4 * i + 2] = ts.c1[i];
                    nd[4 * i + 3] = age[i];
                }
                B.prev_root = prev_root;
                if (b > 0) {
                    int *mp = out.mapping + B.map0;
                    if (p.mapping) {
                        memcpy(mp, p.mapping + (size_t)b * p.nnodes, sizeof(int) * p.nnodes);
                    } else {
                        const int *prev = p.ptrees + (size_t)(b - 1) * p.nnodes;
                        for (int j = 0; j < p.nnodes; j++) mp[j] = j;
                        mp[prev[B.spr[0]]] = -1;
                    }
                }
            }
            prev_root = root;
        }
        // column-major sequences, column classes and byte checks, a tile of columns at a time
        const int ns = I.nseqs, L = p.seqlen;
        const int col0 = plan.blocks[I.block0 + unit.b0].start;
        const BlockDev &end = plan.blocks[I.block0 + unit.b1 - 1];
        const int col1 = end.start + end.len;
        uint8_t *dst = out.seqT + I.seq0;
        uint8_t *cls = out.colclass + I.col0;
        int *cv = out.colvar + I.col0;
        if (uniforms && uniforms[q]) memcpy(out.u + I.col0 + col0, uniforms[q] + col0, sizeof(double) * (col1 - col0));
        constexpr int TILE = 256;
        const uint8_t *src = (const uint8_t *)p.seqs;
        uint8_t diff[TILE];
        Bytes16 bad = {};
        int b = unit.b0, bend = col0 + p.blocklens[b], nv = 0;
        for (int i0 = col0; i0 < col1; i0 += TILE) {
            const int w = std::min(TILE, col1 - i0), w8 = w & ~7;
            // a column varies where some row differs from the first
            const uint8_t *row0 = src + i0;
            for (int i = 0; i + 16 <= w; i += 16) {
                const Bytes16 first = load16(row0 + i);
                Bytes16 differs = {};
                for (int r = 0; r < ns; r++) {
                    const Bytes16 x = load16(row0 + (size_t)r * L + i);
                    differs |= x ^ first;
                    bad |= bad_bases(x);
                }
                memcpy(diff + i, &differs, 16);
            }
            for (int i = w & ~15; i < w; i++) {
                diff[i] = 0;
                for (int r = 0; r < ns; r++) {
                    const uint8_t x = row0[(size_t)r * L + i];
                    diff[i] |= (uint8_t)(x ^ row0[i]);
                    bad[0] |= bad_base(x);
                }
            }
            // groups of 8 rows (the last one may repeat some of the one before): 8 x 8 blocks
            // through registers, 8-byte stores per column
            for (int r0 = 0; r0 < ns && ns >= 8; r0 += 8) {
                const int r = std::min(r0, ns - 8);
                const uint8_t *rows = src + (size_t)r * L + i0;
                for (int i = 0; i < w8; i += 8) {
                    uint64_t x[8];
                    for (int y = 0; y < 8; y++) memcpy(&x[y], rows + (size_t)y * L + i, 8);
                    transpose8x8(x);
                    for (int j = 0; j < 8; j++) memcpy(dst + (size_t)(i0 + i + j) * ns + r, &x[j], 8);
                }
            }
            for (int i = ns >= 8 ? w8 : 0; i < w; i++)
                for (int r = 0; r < ns; r++) dst[(size_t)(i0 + i) * ns + r] = src[(size_t)r * L + i0 + i];
            for (int i = i0; i < i0 + w; i++) {
                while (i >= bend) {  // the block ends: its variant count
                    plan.blocks[I.block0 + b].nvar = nv;
                    b++;
                    bend += p.blocklens[b];
                    nv = 0;
                }
                if (!diff[i - i0]) {
                    cls[i] = src[i] == 'N' ? COL_MASKED : COL_INVARIANT;
                    cv[i] = -1;
                } else {
                    cls[i] = COL_VARIANT;
                    cv[i] = nv++;
                }
            }
        }
        plan.blocks[I.block0 + b].nvar = nv;
        unsigned any = 0;
        for (int i = 0; i < 16; i++) any |= bad[i];
        if (any) {
            static std::mutex mu;
            std::lock_guard<std::mutex> lock(mu);
            bad_seqs[q] = 1;
        }
    });
    for (int q = 0; q < n; q++)
        if (bad_seqs[q]) {
            if (err) *err = problem_error(q, "sequence byte outside A,C,G,T,N");
            return false;
        }
    long long var = 0, vcols = 0;
    for (auto &B : plan.blocks) {
        B.var0 = var;
        B.vrow0 = vcols;
        var += (long long)B.nvar * std::max(B.S, 1);
        vcols += B.nvar;
    }
    plan.total_var = var;
    plan.total_vcols = vcols;
    return true;
}

bool build_plan(const awg_problem *probs, int n, HostPlan &plan, std::string &err) {
    if (!plan_layout(probs, n, plan, err, false)) return false;
    plan.nodes.assign((size_t)plan.total_nodes * 4, -1);
    plan.mapping.assign((size_t)std::max(plan.total_map, 1LL), -1);
    plan.seqT.assign((size_t)std::max(plan.total_seq, 1LL), 'N');
    plan.colclass.assign((size_t)plan.total_cols, COL_INVARIANT);
    plan.colvar.assign((size_t)plan.total_cols, -1);
    return plan_fill(probs, n, plan,
                     PlanDst{plan.nodes.data(), plan.mapping.data(), plan.seqT.data(),
                             plan.colclass.data(), plan.colvar.data(), nullptr},
                     &err);
}

}  // namespace awg
