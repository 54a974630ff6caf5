// pw_plan.h -- host-side queue planning of the chained 16-bit score sweep
// (score16_chain_kernel) and of the band sweeps, and the rules of the affine
// band sweep's boundary rows.  Plain C++, no CUDA: pure functions of the items'
// shapes, so they are tested and timed without a GPU.
#pragma once
#include <algorithm>
#include <cstdint>
#include <functional>
#include <utility>
#include <vector>

#ifdef __CUDACC__
#define PW_PLAN_HD __host__ __device__
#else
#define PW_PLAN_HD
#endif

namespace pw {

// Boundary rows of the affine band sweep (pw_band_affine.cuh).  Band b hands its
// bottom row down in row b % rows of its pair's ring, in words that show the
// band's epoch (1 .. 63; 0 is a cleared word).  A row's earlier words are those
// of bands b - rows, b - 2 rows, ...; the epoch comes round again after 63 of
// them, with band b - 63 rows.  The band that reads b's row is b + 1, and it may
// look at the row long before b has run.  So band c reads only after band
// c - affine_hold(rows) = (c - 1) - 62 rows has finished: that one has then
// written over every word of band (c - 1) - 63 rows.  A row is written over
// where the band below has read it: band b + rows stores a column after the
// bands b + 1 .. b + rows - 1 have handed it down one after another.
constexpr int kAffineEpochs = 63;
PW_PLAN_HD inline uint32_t affine_epoch(int band, int rows) { return 1u + (uint32_t)(band / rows) % kAffineEpochs; }
PW_PLAN_HD inline int affine_hold(int rows) { return (kAffineEpochs - 1) * rows + 1; }

// Rows of a pair of `nbands` bands with `warps` warps in flight: as many as let
// no band be held back.  A warp has one band, a band finishes after the band
// above, so that the unfinished bands of a pair are at most `warps` consecutive
// ones; a pair with no more bands than affine_hold(2) needs two rows.
inline int affine_ring_rows(int nbands, int warps) {
    const int together = std::min(nbands, warps);
    return std::max(2, (together - 1 + kAffineEpochs - 2) / (kAffineEpochs - 1));
}

struct PlanEntry {
    int32_t item;   // index of the source item (in the order given)
    int32_t chain;  // chain index, -1 for a whole item
    int32_t strip;  // strip index in the chain, -1 for a whole item
    int32_t pred;   // queue index of the chain's previous strip, -1 if none
};

struct ChainPlan {
    std::vector<PlanEntry> queue;
    std::vector<int64_t> chain_xm4;  // per chain: its column count (ring row length / 32)
};

// Items (already ordered longest first) have nstr[k] strips of xm4[k]
// columns.  Items whose cost nstr * xm4 reaches permille/1000 of the mean
// per-warp load become chains of one-strip entries; the rest stay whole.
//
// With at least a quarter as many chains as warps the queue goes by levels, the
// chains aligned at their ends: level l holds strip l - (max strips - strips)
// of every chain that has one, longest chains first, and the whole items
// follow.  A strip's predecessor was then handed out about a level earlier and
// is well ahead, so no simulation is needed to keep the warps busy (92,000
// entries: 0.3 ms against 3.4 ms; the sweep takes the same time).
//
// With fewer chains their pipelining decides: the queue comes from a
// list-scheduling simulation of `warps` equally fast warps, time counted in
// columns of one strip.  A warp that frees up takes a strip of a ready chain
// (its predecessor started at least `lead` columns ago), the one whose chain
// has the longest way to go (strips left x lead + columns; ties go to the
// earlier chain), else the next whole item, else the strip that becomes ready
// first.  (Taking the chain that became ready first instead served all chains
// alike and left the longest ones to run by themselves at the end: 64 long DNA
// pairs, 2,368 warps: 33,900 steps against 28,500 here and 25,400 at best.)
// Every strip is queued after its predecessor.
inline void plan_chain_queue(const std::vector<int>& nstr, const std::vector<int64_t>& xm4, int warps,
                             int64_t permille, int lead, ChainPlan& out) {
    const int n = (int)nstr.size();
    out.queue.clear();
    out.chain_xm4.clear();
    warps = std::max(1, warps);
    double total = 0;
    for (int k = 0; k < n; ++k) total += (double)xm4[k] * nstr[k];
    const double thr = total / warps * (double)permille / 1000.0;
    std::vector<int32_t> chain_item, whole;
    for (int k = 0; k < n; ++k) {
        if (nstr[k] >= 2 && (double)xm4[k] * nstr[k] >= thr)
            chain_item.push_back(k);
        else
            whole.push_back(k);
    }
    const int nc = (int)chain_item.size();
    out.chain_xm4.resize(nc);
    std::vector<int32_t> next(nc, 0), last_q(nc, -1);
    size_t n_sub = whole.size();
    for (int c = 0; c < nc; ++c) {
        out.chain_xm4[c] = xm4[chain_item[c]];
        n_sub += (size_t)nstr[chain_item[c]];
    }
    out.queue.reserve(n_sub);
    if (nc > 0 && 4 * (int64_t)nc >= warps) {
        std::vector<int32_t> by_len(nc);
        for (int c = 0; c < nc; ++c) by_len[c] = c;
        std::stable_sort(by_len.begin(), by_len.end(),
                         [&](int32_t a, int32_t b) { return nstr[chain_item[a]] > nstr[chain_item[b]]; });
        const int top = nstr[chain_item[by_len[0]]];
        int active = 0;
        for (int level = 0; level < top; ++level) {
            while (active < nc && nstr[chain_item[by_len[active]]] >= top - level) ++active;
            for (int k = 0; k < active; ++k) {
                const int c = by_len[k];
                out.queue.push_back(PlanEntry{chain_item[c], c, next[c]++, last_q[c]});
                last_q[c] = (int32_t)out.queue.size() - 1;
            }
        }
        for (int32_t k : whole) out.queue.push_back(PlanEntry{k, -1, -1, -1});
        return;
    }
    // heaps: warps by free time, waiting chains by (time their next strip
    // becomes ready << 24 | chain), both smallest first; ready chains by the
    // way they have to go, longest first, then by chain; chain < 2^24
    std::vector<int64_t> freew((size_t)warps, 0);
    std::vector<int64_t> waiting;
    std::vector<std::pair<int64_t, int32_t>> ready;  // (way to go, -chain)
    waiting.reserve(nc);
    ready.reserve(nc);
    for (int c = 0; c < nc; ++c) waiting.push_back((int64_t)c);  // ready at 0, chain order
    std::make_heap(waiting.begin(), waiting.end(), std::greater<int64_t>());
    size_t wnext = 0;
    int open = nc;
    while (open > 0) {
        std::pop_heap(freew.begin(), freew.end(), std::greater<int64_t>());
        const int64_t t = freew.back();
        int64_t done;
        while (!waiting.empty() && (waiting.front() >> 24) <= t) {
            std::pop_heap(waiting.begin(), waiting.end(), std::greater<int64_t>());
            const int c = (int)(waiting.back() & 0xffffff);
            waiting.pop_back();
            ready.push_back({(int64_t)(nstr[chain_item[c]] - next[c]) * lead + out.chain_xm4[c], -c});
            std::push_heap(ready.begin(), ready.end());
        }
        if (!ready.empty() || wnext >= whole.size()) {
            int c;
            int64_t start = t;
            if (!ready.empty()) {
                std::pop_heap(ready.begin(), ready.end());
                c = -ready.back().second;
                ready.pop_back();
            } else {
                std::pop_heap(waiting.begin(), waiting.end(), std::greater<int64_t>());
                start = waiting.back() >> 24;
                c = (int)(waiting.back() & 0xffffff);
                waiting.pop_back();
            }
            out.queue.push_back(PlanEntry{chain_item[c], c, next[c], last_q[c]});
            last_q[c] = (int32_t)out.queue.size() - 1;
            done = start + out.chain_xm4[c];
            if (++next[c] < nstr[chain_item[c]]) {
                waiting.push_back(((start + lead) << 24) | c);
                std::push_heap(waiting.begin(), waiting.end(), std::greater<int64_t>());
            } else {
                --open;
            }
        } else {
            const int k = whole[wnext++];
            out.queue.push_back(PlanEntry{k, -1, -1, -1});
            done = t + xm4[k] * nstr[k];
        }
        freew.back() = done;
        std::push_heap(freew.begin(), freew.end(), std::greater<int64_t>());
    }
    // the chains are all queued: the remaining whole items follow, longest first
    for (; wnext < whole.size(); ++wnext) out.queue.push_back(PlanEntry{whole[wnext], -1, -1, -1});
}

// The queue of a band sweep: one entry per band (item: the pair, strip: the
// band), pair k of nbands[k] bands of steps[k] steps, pairs in priority order.
// Every band is queued, after the band above it.
inline void plan_band_queue(const std::vector<int>& nbands, const std::vector<int64_t>& steps, int warps, int lead,
                            std::vector<PlanEntry>& out) {
    out.clear();
    if ((int64_t)nbands.size() * 2 >= warps) {
        // many pairs: band-major order (every band 0, then every band 1, ...,
        // longest pairs first within a band); a band's predecessor was handed
        // out at least a whole band generation earlier, so nobody waits long
        int maxb = 0;
        for (int nb : nbands) maxb = std::max(maxb, nb);
        std::vector<int32_t> last(nbands.size(), -1);
        for (int b = 0; b < maxb; ++b)
            for (size_t k = 0; k < nbands.size(); ++k)
                if (b < nbands[k]) {
                    out.push_back(PlanEntry{(int32_t)k, (int32_t)k, b, last[k]});
                    last[k] = (int32_t)out.size() - 1;
                }
    } else {
        // few (long) pairs: a list-scheduling plan pipelines each pair's bands.
        // Every pair of several bands is a chain, however short beside the
        // others (no threshold): a warp takes one band, not a whole pair.
        ChainPlan plan;
        plan_chain_queue(nbands, steps, warps, 0, lead, plan);
        out.swap(plan.queue);
        for (PlanEntry& p : out) p.strip = std::max(p.strip, 0);  // pairs of one band
    }
}

}  // namespace pw
