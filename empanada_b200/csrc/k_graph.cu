// k_graph.cu -- the unitig layer over output.bin: the downstream consumer of
// the overlap edges (the reference writes only the edge records; its GFA
// writers, overlap.cu:129-190, are dead code).
//
// Nodes are read-ends (rid = 2i read i, 2i+1 its reverse complement), edges
// the records' (from, to) pairs: the suffix of `from` equals the prefix of
// `to` over ovlp_len bases.  Under the reference's remove_used rule every
// suffix keeps only its longest overlaps, so no edge is transitive (u -> v
// and u -> w share one length) and the graph needs no reduction.  A unitig is
// a maximal path of edges u -> v with out-degree(u) = in-degree(v) = 1; a
// cycle of such edges is cut before its smallest node.  Every node belongs
// to exactly one unitig (a node on no such edge is a unitig of one).
//
//   edges     per edge, succ[from] and pred[to] by compare-and-swap; a second
//             edge at either side marks it as shared (degree above one)
//   link      per node, whether its pred (succ) is a unitig edge: the state
//             (pred, 1), or (itself, 0) at a head; tails marked
//   jump      (node, distance) states by pointer jumping, in place: every
//             node ends with its head and its distance to it, or stays undone
//             when it lies on a cycle
//   cycles    (rare) the smallest node of every cycle by doubling over pred;
//             the cycle is cut before it and jumped again
//   place     unitig sizes from the tails, starts by a scan, each node at
//             start(head) + distance
//
// Bound: random accesses of 4 and 8 bytes to arrays of V words (6.7M nodes:
// 27 and 53 MB, within L2).  Jumping takes log2(longest unitig) passes of
// one random read per unfinished node, where one thread per head used to
// walk its whole path (thousands of reads between repeats, a memory latency
// each).  Nothing of the node arrays crosses to the host but the result, and
// that only when it is asked for.  Build and unitigs of 3.3M reads' overlaps
// (6.7M read-ends, 5.6M edges, 45 MB in, 35 MB out): 48.2 -> 6.9 ms (10.4
// before the copies went through several threads), all but 1 ms host copies.
#include "kernels.h"

namespace emp {
namespace {

constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kShared = 0xfffffffeu;  // two or more edges (nodes are below 2^31)
constexpr uint64_t kDone = 1ull << 31;     // state: node << 32 | done | distance
constexpr int kGT = 256;

EMP_DEV void claim(uint32_t *p, uint32_t v) {
    if (atomicCAS(p, kNone, v) != kNone) *p = kShared;
}

__global__ void graph_edges_kernel(const uint8_t *__restrict__ out, const uint64_t *__restrict__ rec_off,
                                   const uint64_t *__restrict__ rec_e0, uint32_t nrec, uint64_t E, uint32_t nodes,
                                   uint32_t *succ, uint32_t *pred, uint32_t *err) {
    for (uint64_t e = (uint64_t)blockIdx.x * kGT + threadIdx.x; e < E; e += (uint64_t)gridDim.x * kGT) {
        uint32_t lo = 0, hi = nrec;  // last record whose first edge is <= e
        while (hi - lo > 1) {
            const uint32_t m = (lo + hi) >> 1;
            if (rec_e0[m] <= e) lo = m;
            else hi = m;
        }
        const uint64_t k = e - rec_e0[lo], n = rec_e0[lo + 1] - rec_e0[lo];
        const uint8_t *r = out + rec_off[lo] + 12;  // u64 n, i32 ovlp_len, u32 from[n], u32 to[n]: 4-byte aligned
        const uint32_t u = reinterpret_cast<const uint32_t *>(r)[k], v = reinterpret_cast<const uint32_t *>(r)[n + k];
        if (u >= nodes || v >= nodes) {
            atomicOr(err, kErrCapacity);  // an edge names a read-end beyond the reads given
            continue;
        }
        claim(succ + u, v);
        claim(pred + v, u);
    }
}

__global__ void graph_link_kernel(const uint32_t *__restrict__ succ, const uint32_t *__restrict__ pred, uint32_t nodes,
                                  uint64_t *__restrict__ state, uint8_t *__restrict__ tail) {
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) {
        const uint32_t p = pred[u], s = succ[u];
        const bool linked = p < kShared && succ[p] == u;  // neither end shared
        state[u] = linked ? (uint64_t)p << 32 | 1u : (uint64_t)u << 32 | kDone;
        tail[u] = !(s < kShared && pred[s] == u);
    }
}

// One pass of pointer jumping, up to kJumps steps per node; *more set when a
// node is left undone.  Returns at once when *go is zero.  A state is one
// 64-bit word, so a node reads a consistent (if possibly newer) state of
// another.  Distances of nodes on a cycle stop growing below `nodes`.
constexpr int kJumps = 2;
__global__ void graph_jump_kernel(uint64_t *state, uint32_t nodes, const uint32_t *go, uint32_t *more) {
    if (go && !*(const volatile uint32_t *)go) return;
    bool left = false;
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) {
        uint64_t x = __ldcg(state + u);
        if (x & kDone) continue;
        for (int k = 0; k < kJumps && !(x & kDone); ++k) {
            const uint64_t y = __ldcg(state + (x >> 32));
            const uint32_t d = ((uint32_t)x & 0x7fffffffu) + ((uint32_t)y & 0x7fffffffu);
            if (d >= nodes) break;  // on a cycle
            x = (y & (0xffffffff00000000ull | kDone)) | d;
        }
        __stcg(state + u, x);
        left |= !(x & kDone);
    }
    if (__syncthreads_or(left) && threadIdx.x == 0) *(volatile uint32_t *)more = 1u;
}

__global__ void graph_undone_kernel(const uint64_t *__restrict__ state, uint32_t nodes, uint32_t *undone) {
    uint32_t c = 0;
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) c += !(state[u] & kDone);
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(undone, c);
}

// Cycle minimum by doubling over pred: (mn, nx) in, (mn2, nx2) out, the
// undone nodes only (first: from the nodes and their pred).
__global__ void graph_cycle_min_kernel(const uint64_t *__restrict__ state, const uint32_t *__restrict__ pred,
                                       const uint32_t *__restrict__ mn, const uint32_t *__restrict__ nx,
                                       uint32_t nodes, int first, uint32_t *__restrict__ mn2,
                                       uint32_t *__restrict__ nx2) {
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) {
        if (state[u] & kDone) continue;  // on a path
        if (first) {
            mn2[u] = u;
            nx2[u] = pred[u];
        } else {
            const uint32_t x = nx[u];
            mn2[u] = min(mn[u], mn[x]);
            nx2[u] = nx[x];
        }
    }
}

// Every cycle cut before its smallest node: that node becomes a head, its
// pred a tail, the others start again from their pred.
__global__ void graph_cut_kernel(uint64_t *state, const uint32_t *__restrict__ pred, const uint32_t *__restrict__ mn,
                                 uint32_t nodes, uint8_t *tail, uint32_t *cycles) {
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) {
        if (state[u] & kDone) continue;  // on a path (or a head just made by this thread)
        const uint32_t p = pred[u];
        if (mn[u] == u) {
            state[u] = (uint64_t)u << 32 | kDone;
            tail[p] = 1;
            atomicAdd(cycles, 1u);
        } else {
            state[u] = (uint64_t)p << 32 | 1u;
        }
    }
}

__global__ void graph_size_kernel(const uint64_t *__restrict__ state, const uint8_t *__restrict__ tail, uint32_t nodes,
                                  uint32_t *__restrict__ size, uint32_t *__restrict__ is_head) {
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) {
        const uint64_t x = state[u];
        if (tail[u]) size[x >> 32] = ((uint32_t)x & 0x7fffffffu) + 1u;
        is_head[u] = (uint32_t)(x >> 32) == u;
    }
}

__global__ void graph_place_kernel(const uint64_t *__restrict__ state, const uint64_t *__restrict__ start,
                                   const uint32_t *__restrict__ size, const uint64_t *__restrict__ index,
                                   uint32_t nodes, uint32_t *__restrict__ order, uint64_t *__restrict__ starts,
                                   uint32_t *longer) {
    uint32_t c = 0;
    for (uint32_t u = blockIdx.x * kGT + threadIdx.x; u < nodes; u += gridDim.x * kGT) {
        const uint64_t x = state[u];
        const uint32_t h = (uint32_t)(x >> 32);
        const uint64_t at = start[h];
        order[at + ((uint32_t)x & 0x7fffffffu)] = u;
        if (h == u) {
            starts[index[u]] = at;
            c += size[u] >= 2;
        }
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(longer, c);
}

unsigned grid_of(uint64_t n) {
    const uint64_t g = (n + kGT - 1) / kGT;
    return (unsigned)(g < 1 ? 1 : (g > 148 * 8 ? 148 * 8 : g));
}

int jump_rounds(uint32_t nodes) {
    int r = 1;
    while ((1ull << r) < (uint64_t)nodes + 1) ++r;
    return r;
}

void jump(const GraphBufs &b, uint32_t nodes, cudaStream_t s) {
    const int rounds = jump_rounds(nodes);
    count_launch(rounds);
    cudaMemsetAsync(b.more, 0, (kGraphJumps + 1) * sizeof(uint32_t), s);
    for (int r = 0; r < rounds; ++r)  // pass r runs when pass r - 1 left a node undone
        graph_jump_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.state, nodes, r ? b.more + r - 1 : nullptr, b.more + r);
}

}  // namespace

// The paths; *b.undone = the nodes on cycles.
void graph_paths(const uint8_t *out, const uint64_t *rec_off, const uint64_t *rec_e0, uint32_t nrec, uint64_t E,
                 uint32_t nodes, const GraphBufs &b, cudaStream_t s) {
    cudaMemsetAsync(b.succ, 0xff, (size_t)nodes * 4, s);
    cudaMemsetAsync(b.pred, 0xff, (size_t)nodes * 4, s);
    count_launch(E ? 3 : 2);
    if (E)
        graph_edges_kernel<<<grid_of(E), kGT, 0, s>>>(out, rec_off, rec_e0, nrec, E, nodes, b.succ, b.pred, b.err);
    graph_link_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.succ, b.pred, nodes, b.state, b.tail);
    jump(b, nodes, s);
    graph_undone_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.state, nodes, b.undone);
}

// The cycles cut and their nodes placed on the paths (when there are any).
void graph_cycles(uint32_t nodes, const GraphBufs &b, cudaStream_t s) {
    const int rounds = jump_rounds(nodes);
    count_launch(rounds + 2);
    for (int r = 0; r <= rounds; ++r)
        graph_cycle_min_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.state, b.pred, b.mn[r & 1], b.nx[r & 1], nodes, r == 0,
                                                              b.mn[(r + 1) & 1], b.nx[(r + 1) & 1]);
    graph_cut_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.state, b.pred, b.mn[(rounds + 1) & 1], nodes, b.tail, b.cycles);
    jump(b, nodes, s);
}

// The read-ends in unitig order and the unitigs' starts; *b.total = unitigs,
// *b.longer = those of two or more.
void graph_place(uint32_t nodes, const GraphBufs &b, cudaStream_t s) {
    cudaMemsetAsync(b.size, 0, (size_t)nodes * 4, s);
    count_launch(2);
    graph_size_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.state, b.tail, nodes, b.size, b.is_head);
    launch_scan_u32_u64(b.size, b.start, nodes, b.status, b.tile_ctr, b.total + 1, b.err, s);
    launch_scan_u32_u64(b.is_head, b.index, nodes, b.status + scan_tiles(nodes), b.tile_ctr + 1, b.total, b.err, s);
    graph_place_kernel<<<grid_of(nodes), kGT, 0, s>>>(b.state, b.start, b.size, b.index, nodes, b.order, b.starts,
                                                      b.longer);
}

}  // namespace emp
