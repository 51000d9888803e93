// One Barnes-Hut search per warp by sums over bins: the parts shared by the
// FP64 search (bh_search.cu) and the FP32 form (fp32.cu).
//
// The reference sums the weights of a descent's candidates in visiting order,
// draws r below the total and picks the first candidate whose running sum
// reaches r (ProbabilityPicker::pick_target, util/ProbabilityPicker.h:46-112).
// Which candidate that is does not need the reference's order of additions:
// sums in any order differ from its running sums by a bounded rounding error,
// so a crossing that lies further than that bound from r on both sides is the
// reference's own.  A search whose crossing lies closer is left to the ordered
// form (bh_wide.cuh; target kRedo), which repeats it in the reference's order:
// the targets are the same bits on every path.
//
// What that buys: no candidate has to be stored or put into order.  The
// cells that contain the source (its chain: root, ..., leaf) split all other
// visited nodes into the subtrees of their other children, at most 8 per
// level: the bins.  Four expanded nodes at a time (8 lanes each: one lane per
// child) come off a stack in shared memory, the lanes' accepted weights go
// to the parents' bins, and expanded children go back on the stack.  The bins
// in visiting order give the total and the bin of the crossing; only that
// bin's subtree (a few dozen nodes) is walked again, with a bin per child,
// down to the candidate.
//
#pragma once

#include <type_traits>

#include "bh_wide.cuh"

namespace rl {

constexpr uint32_t kBinCopies = 4;  // one per group of 8 lanes, so that groups never add to the same word

// What ev(node, act) returns.  Every lane evaluates (one without a node, act
// false, evaluates node 0), and the results are selected: with branches the
// lanes of a pass run the accepting, the expanding and the idle path one after
// the other (200,000 searches of 200,000 neurons, FP64 / FP32: 4.96e9 / 4.35e9
// warp instructions and 7.4 / 6.3 ms with branches, 4.43e9 / 3.51e9 and 5.6 /
// 4.2 ms selected).
struct BinsEval {
    double w;        // weight of an accepted node, else 0
    uint32_t first;  // first child (of a node that expands)
    uint32_t nch;    // and its children
    bool expand;
    bool cand;       // accepted and not the source itself
};

// Shared memory of one warp for octrees of `levels` levels below the root.
struct BinsMem {
    double* bin;            // kBinCopies x nb
    uint2* stack;           // expanded nodes: first child, bin | children << 16
    uint32_t* chain;        // cells that contain the source, root first
    uint32_t* chain_first;  // per chain level: first child
    uint32_t* chain_info;   // children | own child << 4 | own child expanded << 8 | expanded children << 16
    uint32_t nb;            // bins per copy: 8 per level
    uint32_t cap;           // stack entries
};

// The chain leaves at most 7 entries per level; on top of them a batch of four
// pops four entries and pushes as many on average (32 at most, one level
// deeper).  The room is kept small, since it comes out of the L1 cache that
// holds the octree; a search that needs more goes to the ordered form.
__host__ __device__ __forceinline__ uint32_t bins_stack_cap(uint32_t levels) {
    return 12u * levels + 96u;
}
__host__ __device__ __forceinline__ size_t bins_warp_bytes(uint32_t levels) {
    const size_t b = (size_t)kBinCopies * 8u * levels * sizeof(double) + (size_t)bins_stack_cap(levels) * sizeof(uint2) + (3u * (size_t)levels + 1u) * sizeof(uint32_t);
    return (b + 15) / 16 * 16;
}

__device__ __forceinline__ BinsMem bins_mem(unsigned char* p, uint32_t levels) {
    BinsMem M;
    M.nb = 8u * levels;
    M.cap = bins_stack_cap(levels);
    M.bin = reinterpret_cast<double*>(p);
    M.stack = reinterpret_cast<uint2*>(M.bin + kBinCopies * M.nb);
    M.chain = reinterpret_cast<uint32_t*>(M.stack + M.cap);
    M.chain_first = M.chain + levels + 1;
    M.chain_info = M.chain_first + levels;
    return M;
}

// Empties the stack of `top` entries into the bins; false if it would
// overflow or the walk visits more nodes than there are (the ordered form
// reports that).  A pass takes the evaluator's kEntries entries per group.
template <class Ev>
__device__ __forceinline__ bool bins_drain(const BinsMem& M, uint32_t top, uint32_t num_nodes, uint32_t& touched, bool& any, Ev&& ev) {
    constexpr uint32_t P = std::remove_reference_t<Ev>::kEntries;
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 3, sub = lane & 7u;
    const uint32_t below = (1u << lane) - 1u;
    double* mine = M.bin + g * M.nb;
    uint32_t guard = num_nodes;
    while (top > 0u) {
        uint2 s[P];
        BinsEval e[P];
#pragma unroll
        for (uint32_t q = 0; q < P; ++q) {
            const uint32_t at = g + 4u * q;
            s[q] = M.stack[at < top ? top - 1u - at : 0u];
            const bool act = at < top && sub < (s[q].y >> 16);
            e[q] = ev(s[q].x + sub, act);
            touched += act ? 1u : 0u;
            any = any || e[q].cand;
        }
#pragma unroll
        for (uint32_t q = 0; q < P; ++q) {
            double v = e[q].w;
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 4);
            if (sub == 0u && g + 4u * q < top) {
                mine[s[q].y & 0xFFFFu] += v;
            }
        }
        top -= top < 4u * P ? top : 4u * P;
#pragma unroll
        for (uint32_t q = 0; q < P; ++q) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, e[q].expand);
            const uint32_t at = top + (uint32_t)__popc(m & below);
            top += (uint32_t)__popc(m);
            if (top > M.cap) {
                return false;
            }
            if (e[q].expand) {
                M.stack[at] = make_uint2(e[q].first, (s[q].y & 0xFFFFu) | (e[q].nch << 16));
            }
        }
        if (guard-- == 0u) {
            return false;
        }
        __syncwarp();
    }
    return true;
}

// The candidates below each of the nch children from `first` on: lane k < 8
// returns the sum of child k (the child itself if accepted) and its
// evaluation in `mine`.
template <class Ev>
__device__ __forceinline__ bool bins_children(const BinsMem& M, uint32_t first, uint32_t nch, uint32_t num_nodes, uint32_t& touched, bool& any, Ev&& ev,
                                              BinsEval& mine, double& sum) {
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 3, sub = lane & 7u;
    mine = ev(first + lane, lane < nch);
    touched += lane < nch ? 1u : 0u;
    any = any || mine.cand;
    sum = mine.w;
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, mine.expand);
    if (m == 0u) {
        return true;
    }
    M.bin[g * M.nb + sub] = 0.0;
    if (mine.expand) {
        M.stack[__popc(m & ((1u << lane) - 1u))] = make_uint2(mine.first, lane | (mine.nch << 16));
    }
    __syncwarp();
    if (!bins_drain(M, (uint32_t)__popc(m), num_nodes, touched, any, ev)) {
        return false;
    }
    if (mine.expand) {
        sum = ((M.bin[lane] + M.bin[M.nb + lane]) + M.bin[2u * M.nb + lane]) + M.bin[3u * M.nb + lane];
    }
    __syncwarp();
    return true;
}

constexpr int64_t kPickRedo = -1;

// The crossing of r among the children of a node with running sum `start`
// before them (lane k: `sum` and `mine` of child k, from bins_children),
// followed down to the candidate; kPickRedo if r lies within `margin` of
// either side of it.
template <class Ev>
__device__ __forceinline__ int64_t bins_pick(const BinsMem& M, uint32_t first, uint32_t nch, double start, double r, double margin, uint32_t num_nodes,
                                             BinsEval mine, double sum, Ev&& ev) {
    for (int depth = 0; depth <= kMaxLevels; ++depth) {
        double run = start, pre = start, post = start;
        int hit = -1;
        for (int k = (int)nch - 1; k >= 0; --k) {  // children are visited from the last octant down
            const double next = run + __shfl_sync(0xFFFFFFFFu, sum, k);
            if (hit < 0 && next >= r) {
                hit = k;
                pre = run;
                post = next;
            }
            run = next;
        }
        if (hit < 0) {
            return kPickRedo;
        }
        if (!__shfl_sync(0xFFFFFFFFu, mine.expand ? 1 : 0, hit)) {
            return r - pre > margin && post - r > margin ? (int64_t)(first + (uint32_t)hit) : kPickRedo;
        }
        const uint32_t f = __shfl_sync(0xFFFFFFFFu, mine.first, hit);
        nch = __shfl_sync(0xFFFFFFFFu, mine.nch, hit);
        first = f;
        start = pre;
        uint32_t touched = 0;
        bool any = false;
        if (!bins_children(M, first, nch, num_nodes, touched, any, ev, mine, sum)) {
            return kPickRedo;
        }
    }
    return kPickRedo;
}

// One search by the whole warp: the target neuron, -1 when the search fails,
// kRedo when it is left to the ordered form.
//   ev(node, act)      evaluates a node (BinsEval)
//   threshold(T, d)    r of descent d for the total T
//   margin(T, visited) bound on |our running sums - the reference's| + |our r - the reference's|
//   tiny               totals below it (weights that underflow) are left to the ordered form
template <class Ev, class Threshold, class Margin>
__device__ int32_t bins_search(const BinsMem& M, const uint4* __restrict__ meta, const int32_t* __restrict__ parent, uint32_t num_nodes, uint32_t root,
                               uint32_t leaf, double tiny, uint32_t& touched, Ev&& ev, Threshold&& threshold, Margin&& margin) {
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 3, sub = lane & 7u;
    const uint32_t depth0 = topo_level(__ldg(&meta[root]).y);
    const uint32_t lv = topo_level(__ldg(&meta[leaf]).y) - depth0;
    if (8u * lv > M.nb) {
        return kRedo;
    }
    {
        uint32_t nd = leaf;
        for (uint32_t l = lv; l > 0u; --l) {
            if (lane == 0u) {
                M.chain[l] = nd;
            }
            nd = (uint32_t)__ldg(&parent[nd]);
        }
        if (lane == 0u) {
            M.chain[0] = root;
        }
    }
    for (uint32_t b = lane; b < kBinCopies * M.nb; b += 32u) {
        M.bin[b] = 0.0;
    }
    __syncwarp();
    // ---- the chain: four levels at a time
    const uint32_t before = touched;
    uint32_t seen = 0;
    bool any = false;
    uint32_t top = 0, levels = 0;
    for (uint32_t l0 = 0; l0 < lv; l0 += 4u) {
        const uint32_t l = l0 + g;
        uint32_t first = 0, nch = 0, own = 0;
        if (l < lv) {
            const uint4 ma = __ldg(&meta[M.chain[l]]);
            first = ma.x;
            nch = (uint32_t)__popc(topo_mask(ma.y));
            own = M.chain[l + 1u] - first;
        }
        const BinsEval e = ev(first + sub, sub < nch);
        const uint32_t own_exp = __ballot_sync(0xFFFFFFFFu, l < lv && sub == own && e.expand);
        // a level is visited when every own child above it was expanded
        bool visit = l < lv;
        for (uint32_t q = 0; q < g; ++q) {
            visit = visit && ((own_exp >> (8u * q)) & 0xFFu) != 0u;
        }
        const bool act = visit && sub < nch;
        seen += act ? 1u : 0u;
        any = any || (act && e.cand);
        const bool mine_exp = ((own_exp >> (8u * g)) & 0xFFu) != 0u;
        const bool push = act && e.expand && sub != own;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, push);
        const uint32_t exp_all = __ballot_sync(0xFFFFFFFFu, act && e.expand);
        if (push) {
            M.stack[top + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_uint2(e.first, (l * 8u + sub) | (e.nch << 16));
        }
        top += (uint32_t)__popc(m);
        if (act && e.cand) {
            M.bin[l * 8u + sub] = e.w;
        }
        if (visit && sub == 0u) {
            M.chain_first[l] = first;
            M.chain_info[l] = nch | (own << 4) | (mine_exp ? 256u : 0u) | (((exp_all >> (8u * g)) & 0xFFu) << 16);
        }
        levels += (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, visit && sub == 0u));
        if (own_exp == 0u || levels < l0 + 4u || ((own_exp >> 24) & 0xFFu) == 0u) {
            break;
        }
    }
    __syncwarp();
    touched += seen;
    if (!bins_drain(M, top, num_nodes, touched, any, ev)) {
        return kRedo;
    }
    // ---- the bins in visiting order: at each level the own child's later
    // octants, then (below the own child) the deeper levels, then its earlier ones
    uint32_t total_bins = 0;
    for (uint32_t l = 0; l < levels; ++l) {
        const uint32_t inf = M.chain_info[l];
        total_bins += (inf & 15u) - ((inf >> 8) & 1u);
    }
    double* seq = reinterpret_cast<double*>(M.stack);  // the stack is empty: the ordered sums
    uint32_t* seq_id = reinterpret_cast<uint32_t*>(seq + M.nb);  // and their bins
    for (uint32_t b = lane; b < 8u * levels; b += 32u) {
        const uint32_t l = b >> 3, k = b & 7u;
        const uint32_t inf = M.chain_info[l];
        const uint32_t nch = inf & 15u, own = (inf >> 4) & 15u;
        const bool through = (inf >> 8) & 1u;
        if (k < nch && !(through && k == own)) {
            uint32_t ahead = 0, behind = 0;
            for (uint32_t x = 0; x < l; ++x) {
                const uint32_t i2 = M.chain_info[x];
                const uint32_t o2 = (i2 >> 4) & 15u;
                ahead += (i2 & 15u) - 1u - o2;
                behind += o2;
            }
            const uint32_t at = !through || k > own ? ahead + (nch - 1u - k) : total_bins - 1u - (behind + k);
            seq[at] = ((M.bin[b] + M.bin[M.nb + b]) + M.bin[2u * M.nb + b]) + M.bin[3u * M.nb + b];
            seq_id[at] = b;
        }
    }
    __syncwarp();
    double total = 0.0;
    for (uint32_t base = 0; base < total_bins; base += 32u) {
        double v = base + lane < total_bins ? seq[base + lane] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double w = __shfl_up_sync(0xFFFFFFFFu, v, o);
            if (lane >= (uint32_t)o) {
                v += w;
            }
        }
        v += total;
        if (base + lane < total_bins) {
            seq[base + lane] = v;
        }
        total = __shfl_sync(0xFFFFFFFFu, v, 31);
    }
    __syncwarp();
    if (!__any_sync(0xFFFFFFFFu, any)) {
        return -1;  // no candidate but the source itself: the search fails
    }
    if (!(total >= tiny)) {
        return kRedo;
    }
    uint32_t visited = touched - before;
    for (int o = 16; o > 0; o >>= 1) {
        visited += __shfl_xor_sync(0xFFFFFFFFu, visited, o);
    }
    double r = threshold(total, 0u);
    double mg = margin(total, visited);
    uint32_t at = total_bins;
    for (uint32_t base = 0; base < total_bins; base += 32u) {
        const uint32_t hit = __ballot_sync(0xFFFFFFFFu, base + lane < total_bins && seq[base + lane] >= r);
        if (hit) {
            at = base + (uint32_t)(__ffs((int)hit) - 1);
            break;
        }
    }
    if (at >= total_bins) {
        return kRedo;
    }
    const double pre = at > 0u ? seq[at - 1u] : 0.0;
    const double post = seq[at];
    const uint32_t b = seq_id[at];
    const uint32_t inf = M.chain_info[b >> 3];
    uint32_t node = M.chain_first[b >> 3] + (b & 7u);
    __syncwarp();  // the walks below reuse the bins
    if ((inf >> (16u + (b & 7u))) & 1u) {
        const uint4 mm = __ldg(&meta[node]);
        const uint32_t nch = (uint32_t)__popc(topo_mask(mm.y));
        BinsEval mine;
        double sum;
        uint32_t t2 = 0;
        bool a2 = false;
        if (!bins_children(M, mm.x, nch, num_nodes, t2, a2, ev, mine, sum)) {
            return kRedo;
        }
        const int64_t got = bins_pick(M, mm.x, nch, pre, r, mg, num_nodes, mine, sum, ev);
        if (got < 0) {
            return kRedo;
        }
        node = (uint32_t)got;
    } else if (!(r - pre > mg && post - r > mg)) {
        return kRedo;
    }
    // ---- deeper descents from the picked node
    for (uint32_t depth = 1; depth <= (uint32_t)kMaxLevels + 2u; ++depth) {
        const uint4 sm = __ldg(&meta[node]);
        if (topo_leaf(sm.y)) {
            return (int32_t)sm.x;
        }
        const uint32_t nch = (uint32_t)__popc(topo_mask(sm.y));
        BinsEval mine;
        double sum;
        const uint32_t t0 = touched;
        any = false;
        if (!bins_children(M, sm.x, nch, num_nodes, touched, any, ev, mine, sum)) {
            return kRedo;
        }
        total = 0.0;
        for (int k = (int)nch - 1; k >= 0; --k) {
            total += __shfl_sync(0xFFFFFFFFu, sum, k);
        }
        if (!__any_sync(0xFFFFFFFFu, any)) {
            return -1;
        }
        if (!(total >= tiny)) {
            return kRedo;
        }
        uint32_t vis = touched - t0;
        for (int o = 16; o > 0; o >>= 1) {
            vis += __shfl_xor_sync(0xFFFFFFFFu, vis, o);
        }
        r = threshold(total, depth);
        mg = margin(total, vis);
        const int64_t got = bins_pick(M, sm.x, nch, 0.0, r, mg, num_nodes, mine, sum, ev);
        if (got < 0) {
            return kRedo;
        }
        node = (uint32_t)got;
    }
    return kRedo;
}

}  // namespace rl
