// Shared by the emission kernels (tables.cu, emit_groups.cu): a tree's level schedules, the
// infinite-sites test, the log-likelihood's references and the persistent kernels' work queue.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "kernels.h"

namespace awg {
namespace {

// A tree with its nodes by height (children before parents) and, below the main root, by depth.
struct TreeLevels {
    const int4 *nd;
    const int *inl, *inp, *outl, *outp;
    int nlev_in, nlev_out, mainr, node1, nleaves, n;
    bool internal;
};

__device__ __forceinline__ int base_bit(uint8_t ch) {
    if (ch == 'N') return 0;
    return 1 << ((ch == 'A' || ch == 'a') ? 0 : (ch == 'C' || ch == 'c') ? 1
                 : (ch == 'G' || ch == 'g') ? 2 : 3);
}

// Infinite-sites validity of one variant column's nodes (get_infinite_sites_states,
// emit.cpp:454-589, with parsimony_ancestral_set :898-953) by one warp over the level
// schedules: Fitch sets by height, then refined from the main root down (any order with
// children first, then parents first, gives the reference's sets). A state on node j keeps
// the model when the threaded base (the cut subtree's set) meets the set of j or of its
// parent. Node j's flag is bit j / 32 of lane j % 32's word; all flags are 1 when the
// column cannot break the model. sets, anc: n bytes each of the warp's scratch.
__device__ unsigned infsites_nodes(const TreeLevels &c, const uint8_t *chars, uint8_t *sets,
                                   uint8_t *anc) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int4 *nd = c.nd;
    int all = 0, subset = 0, mainset = 0;
    for (int x = lane; x < c.inp[1]; x += 32) {
        const int j = c.inl[x];
        const int b = base_bit(chars[j]);
        sets[j] = (uint8_t)b;
        if (!c.internal) {
            all |= b;
        } else {
            int u = j;
            for (int s = 0; u != -1 && u != c.node1 && s < c.n; s++) u = nd[u].x;
            if (u == c.node1) subset |= b;
            else mainset |= b;
        }
    }
    all = __reduce_or_sync(FULL, all);
    subset = __reduce_or_sync(FULL, subset);
    mainset = __reduce_or_sync(FULL, mainset);
    __syncwarp();
    for (int h = 1; h < c.nlev_in; h++) {
        for (int x = c.inp[h] + lane; x < c.inp[h + 1]; x += 32) {
            const int j = c.inl[x];
            const int l = sets[nd[j].y], r = sets[nd[j].z];
            sets[j] = (uint8_t)((l & r) ? (l & r) : (l | r));
        }
        __syncwarp();
    }
    const int cset = c.internal ? sets[c.node1] : base_bit(chars[c.nleaves]);
    if (c.internal ? !(subset & mainset) : !(cset & all)) return FULL;
    for (int h = 0; h < c.nlev_out; h++) {
        for (int x = c.outp[h] + lane; x < c.outp[h + 1]; x += 32) {
            const int j = c.outl[x];
            if (j == c.mainr) {
                anc[j] = sets[j];
            } else {
                const int ps = anc[nd[j].x] & sets[j];
                anc[j] = (uint8_t)(ps ? ps : sets[j]);
            }
        }
        __syncwarp();
    }
    unsigned word = FULL;
    for (int w = 0; w * 32 + lane < c.n && w < 32; w++) {
        const int j = w * 32 + lane;
        int u = j;  // in the main tree (the only nodes with states)
        for (int s = 0; u != -1 && u != c.mainr && s < c.n; s++) u = nd[u].x;
        if (u != c.mainr) continue;
        const bool ok = (cset & anc[j]) || (j != c.mainr && (cset & anc[nd[j].x]));
        if (!ok) word &= ~(1u << w);
    }
    __syncwarp();
    return word;
}

// Whether state k's node keeps the infinite-sites model (all lanes call it).
__device__ __forceinline__ bool state_ok(unsigned word, int node) {
    return (__shfl_sync(0xffffffffu, word, node & 31) >> (node >> 5)) & 1;
}

// FP32 path: a tree's share of the log-likelihood's emission references, lneref per
// invariant column and log(vref) per variant column (the instance's column 0, the prior, has
// none), summed by one warp in a fixed order. The logarithms are taken here, a lane per
// variant column, not by one lane per column in the emission passes: there an FP64 log holds
// the warp's FP64 pipe for a few thousand cycles per column.
__device__ void block_log_offset(const BatchDev &d, const BlockDev &B, const InstDev &I, int blk,
                                 int lane) {
    const uint8_t *cls = d.colclass + I.col0 + B.start;
    const int first = B.b == 0 ? 1 : 0;
    double s = 0.0;
    if (B.S > 0) {
        int ninv = 0;
        for (int i = first + lane; i < B.len; i += 32) ninv += cls[i] == COL_INVARIANT;
        s = ninv * d.lneref[blk];
        for (int v = lane + (first && cls[0] == COL_VARIANT); v < B.nvar; v += 32) s += log(d.vref[B.vrow0 + v]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) d.blkext[blk] = s;
}

// Work queue of a persistent per-tree kernel: units of `chunk` consecutive trees in the
// batch's tree order (largest instances first), taken by CTAs with an atomic counter.
struct WorkQueue {
    int *counter;
    int nunits, chunk;
};

// Takes the next unit for the whole CTA; -1 when the queue is empty.
__device__ __forceinline__ int next_unit(const WorkQueue &q) {
    __shared__ int unit;
    __syncthreads();  // the previous unit's reads of `unit` are done
    if (threadIdx.x == 0) unit = atomicAdd(q.counter, 1);
    __syncthreads();
    const int u = unit;
    return u < q.nunits ? u : -1;
}

// CTAs of a persistent kernel: as many as are resident on the GPU at once, at most one per
// unit of work.
template <typename K>
int persistent_grid(K kernel, int threads, size_t smem, int nunits) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return imax(1, imin(nunits, per_sm * sms));
}

}  // namespace
}  // namespace awg
