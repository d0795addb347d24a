// The FP32 forward kernel's shared memory and the choice of its form (forward32.cu), by an
// instance's own sizes: host and device code, so that what a launch allocates and what a CTA lays
// out come from one place.
#pragma once

#include "awg_internal.h"

namespace awg {
namespace fwd32 {

constexpr int NRW = 4;     // reduction warps
constexpr int EDEPTH = 4;  // columns an emission row is loaded ahead

// The staging buffer of one tree (byte offsets; every part starts on 16 bytes and is copied
// from the 16-byte boundary below its source). The parts from sinfo on are per state.
struct StageLayout {
    int desc, tm, rstay, bptr, sinfo, t2off, perm, inv, gptr, gidx, move, rrow, crow, src, total;
    AWG_HD explicit StageLayout(int maxS) {
        const int arr = (4 * maxS + 32 + 15) & ~15;
        desc = 0;  // three descriptors: this tree's, the next one's, the one's after
        tm = desc + 3 * (int)sizeof(BlockDev);
        rstay = tm + 4 * MAXT * MAXT;
        bptr = rstay + 4 * MAXT;
        sinfo = bptr + 160;
        t2off = sinfo + 16 * maxS;
        perm = t2off + arr;
        inv = perm + arr;
        gptr = inv + arr;
        gidx = gptr + arr;
        move = gidx + arr;
        rrow = move + ((8 * maxS + 32 + 15) & ~15);
        crow = rrow + arr;
        src = crow + arr;
        total = src + 16;
    }
};
static_assert(sizeof(BlockDev) % 16 == 0, "descriptors are bulk-copied");

// An instance's largest tree (states, same-branch row entries) and its nodes; or a batch's.
struct Sizes {
    int S, M, nodes;
};

// Shared memory of one CTA (byte offsets).
struct SmemPlan {
    int stage, t2, t2_bytes, col, red, ring, last, total;
    AWG_HD SmemPlan(const Sizes &z, int t2_bufs, bool staged) {
        auto up = [](int v) { return (v + 15) & ~15; };
        stage = 0;
        t2 = stage + (staged ? StageLayout(z.S).total : StageLayout(z.S).sinfo);
        t2_bytes = up(4 * z.M + 32);
        col = t2 + t2_bufs * t2_bytes;
        // nodes on 16 bytes (up to 3 more slots each); rows end up to MAXT past a node's last
        red = col + 2 * up(4 * (z.S + 3 * z.nodes + MAXT + 8));
        // the lanes' positions in groups of up to 8, and a slot for threads without a state
        ring = red + 8 * (z.S + 32 * 9 * NRW) + 16;
        last = ring + (EDEPTH + 1) * up(4 * z.S);
        total = last + up(8 * z.S);
    }
};

// Owner threads of a CTA: 16 warps with the reducers, 4 a sub-partition, leave 128 registers
// a thread; the wide form for batches with larger trees has 20 warps at 96.
constexpr int OWNERS = 384, WIDE_OWNERS = 512;
constexpr int MOST_STATES = 8 * OWNERS;  // of a tree that the kernel takes

// Dynamic shared memory of a launch for a batch of these largest sizes: the most demanding form
// that fits beside the static part.
constexpr int LIMIT = 222 * 1024;
AWG_HD inline int launch_bytes(const Sizes &z) {
    return imin(SmemPlan(z, 2, true).total, LIMIT);
}

// States per owner thread (1, 2, 3, 4 or 8) for an instance's largest tree; at least `least`. One
// while the owners suffice: a thread's shared loads are issued one after another, so a column
// takes 0.47 us at 99 states and 0.67 at 351 with one, 0.64 and 0.78 with two; 1.24 at 789 and
// 1.30 at 930 with three, 1.48 at 930 with four.
AWG_HD inline int states_per_thread(int maxS, int least, int owners) {
    const int k = maxS <= owners ? 1 : maxS <= 2 * owners ? 2 : maxS <= 3 * owners ? 3 : maxS <= 4 * owners ? 4 : 8;
    return imax(k, least);
}
AWG_HD inline int owner_threads(int maxS, int kpt) {
    return imax(32, ((maxS + kpt - 1) / kpt + 31) / 32 * 32);
}

// How a CTA of `owners` threads runs an instance: states a thread, buffers of rows in shared memory
// (0: rows in global memory), tables staged a tree ahead or read from global memory.
struct Form {
    int kpt, bufs;
    bool staged;
    int owners;  // threads
};
// The form of an instance in a launch of `smem` bytes; LONG: more than 21 time points in the batch,
// wide: the wide CTA. Rows that the registers hold need one buffer (one state a thread; two up to
// 21 time points), longer ones two, staged with the other tables a tree ahead; where that does not
// fit, the tables stay in global memory, and so do the rows if they do not fit either.
AWG_HD inline Form form_of(const Sizes &z, int smem, bool LONG, bool wide, int least) {
    auto fits = [&](int bufs, bool staged) { return SmemPlan(z, bufs, staged).total <= smem; };
    Form f;
    f.kpt = states_per_thread(z.S, least, wide ? WIDE_OWNERS : OWNERS);
    f.owners = owner_threads(z.S, f.kpt);
    f.bufs = f.kpt == 1 || (f.kpt == 2 && !LONG) ? 1 : 2;
    f.staged = f.kpt <= 4 && !(f.kpt == 4 && wide) && fits(f.bufs, true);
    if (!f.staged) {
        if (f.kpt <= 2) f.kpt = 4;  // (there is no such form of fewer; the threads suffice)
        f.bufs = fits(1, false) ? 1 : 0;
    }
    return f;
}

}  // namespace fwd32
}  // namespace awg
