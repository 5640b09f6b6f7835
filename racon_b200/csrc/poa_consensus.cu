// Window consensus on the device with the semantics of racon's
//   src/window.cpp:65-142  Window::generate_consensus
// over spoa's partial-order graph (linear-gap NW, match/mismatch/gap from
// racon's -m/-x/-g, engine built at src/polisher.cpp:181-185).
//
// Design (B200, sm_100a). A team of one or four warps owns one window at a
// time; teams are persistent and pull windows from a size-sorted queue. Each
// team has a slot of global scratch (graph arrays first, then the DP score
// rows) and shared memory (the DP's row rings, scratch for the graph steps).
// * In-edges are kept with their node, in the order in which they were added,
//   the first eight in two 16-byte words each for sources and weights, so that
//   building a layer's rows and adding its edges are independent per node.
// * Per layer: the subgraph of a partial layer, row descriptors (predecessor
//   ranks, count, base), the DP, the end cell, the traceback and the insertion
//   of the aligned layer. Per-node and per-position steps run on the whole
//   team with four entries per thread in flight; the subgraph sweep runs on
//   one warp, 32 rows at a time, and the few serial steps (DFS, bundle scores)
//   on one lane, over shared memory.
// * The DP runs one row (graph node in a valid topological order kept
//   incrementally) at a time, the team's warps side by side on strips of its
//   columns (dp_strip), on slanted scores H - column * gap, so that the
//   in-row gap term is a plain running maximum. It keeps no decisions: the
//   walk back decides at the few hundred cells it visits from the stored
//   scores, in spoa's order (diagonal through each predecessor, then
//   vertical, then horizontal).
// * The NW end cell is the first sink in spoa's topological order with the
//   best last-column score; spoa's DFS order is built only when that cannot be
//   told from node ids (end_row).
// * After the last layer: heaviest bundle (scores in shared memory, spoa's
//   topological order only for ties), branch completion, coverages, trimming.
// Exact int32 arithmetic throughout; results are byte-identical to the CPU
// algorithm by construction.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstring>
#include <chrono>
#include <cstdlib>
#include <memory>
#include <numeric>
#include <type_traits>

#include "rb_internal.hpp"
#include "ring_queue.cuh"
#include "score_rows.hpp"

namespace rb {

// One batch of windows in the shared queue (device record, written before
// its items are published): the batch's device buffers, as PoaArgs holds
// them for a private launch.
struct PoaJobDev {
    SvcJobHead head;            // windows of the batch, generation
    const uint8_t* in;
    const PoaWinDev* wins;
    const PoaLayerDev* layers;
    char* out;
    uint32_t* out_len;
    uint8_t* flags;
    unsigned long long* cells;  // [0] DP cells, [1] edge-cells (device)
    int trim;
    uint32_t pad;
};

namespace {

// minus infinity that survives thousands of gap additions without overflow
constexpr int kNegInf = -(1 << 29);
enum PoaFlag : uint8_t {
    kPolished = 1,
    kChimeric = 2,
    kOverflow = 4,
    kFailed = 8,
};

struct PoaArgs {
    const uint8_t* in;
    const PoaWinDev* wins;
    const PoaLayerDev* layers;
    const uint32_t* order;
    uint32_t nwin;
    char* out;
    uint32_t* out_len;
    uint8_t* flags;
    uint8_t* scratch;
    size_t slot_bytes;
    int ncap, ecap, acap, lcap;  // node / edge / aligned-entry / DP-column capacities
    int match, mismatch, gap;
    int trim;
    unsigned int* counters;      // [0] window cursor, [1] status
    unsigned long long* cells;   // [0] DP cells computed, [1] edge-cells
    uint32_t per_warp_cap;       // windows a warp takes per launch (0: until the queue is empty)
    int wait_polls;              // polls of a wait between a team's warps before the window is given up
};

// Per-slot scratch view.
constexpr int kInline = 8;  // in-edges kept with their node
constexpr int kGraphArrays = 40;
struct Graph {
    // nodes
    uint8_t *code, *flag;
    uint32_t* cov;
    int *in_cnt, *out_cnt, *al_cnt;
    int4 *in_src, *in_w;    // [N][2]: the first kInline in-edges' sources and weights
    int *ov_head, *ov_tail; // list of the further ones
    int4* al4;              // the first four aligned nodes
    int *al_head, *al_tail; // list of the further ones
    int *e_src, *e_w, *e_next;  // in-edges past kInline
    int *a_node, *a_next;       // aligned entries past four
    // valid topological order kept incrementally (rank -> node, node -> rank),
    // its double buffer, per-rank shift counts
    int *ord, *ord2, *rank, *shift;
    int *dporder, *sub_rank;  // rows of a partial layer, node -> row (0: none)
    int *dfs, *dfs_rank;      // spoa's DFS order and its inverse
    int* stack;
    int4* rowdesc;            // per DP row (build_rows)
    int* pred_idx;
    uint32_t* used;           // bit r - 1: a row other than r + 1 has row r as predecessor
    int *sink_rows, *sink_h;  // sink rows and their last-column scores
    // per sequence position of the layer: row, then node on its path (0, then
    // -1 for an inserted base), node id, order slot; order slots of the new nodes
    int *path, *nid, *slot, *new_slot;
    long long* bscore;
    int *bpred, *cons;
    int* H;
    int ncap, ecap, acap, scap, lcap;
};

__host__ __device__ size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// Offsets of the slot's arrays: f(pointer to the Graph member's place, offset).
template <class F>
__host__ __device__ size_t walk_layout(int ncap, int ecap, int acap, int lcap, F&& f) {
    size_t off = 0;
    const size_t N = size_t(ncap), E = size_t(ecap), A = size_t(acap), L = size_t(lcap);
    const size_t S = N + E + A + 16;
    // graph arrays (touched by the pointer-walking steps) first, packed;
    // the DP matrix, streamed once per layer, last
    const size_t bytes[kGraphArrays] = {
        N,       N + 8,   N * 4,   N * 4,   N * 4,   N * 4,    N * 32,  N * 32,        N * 4,   N * 4,
        N * 16,  N * 4,   N * 4,   E * 4,   E * 4,   E * 4,    A * 4,   A * 4,         N * 4,   N * 4,
        N * 4,   (N + 2) * 4,      N * 4,   N * 4,   N * 4,    N * 4,   S * 4,         (N + 32) * 16,
        (N * kInline + E + 2) * 4, N / 8 + 8, N * 4, N * 4, (L + 2) * 4, (L + 2) * 4, (L + 2) * 4, N * 4, N * 8,
        N * 4,   N * 4,   (N + 1) * L * 4};
    for (int id = 0; id < kGraphArrays; ++id) {
        f(id, off);
        off += align256(bytes[id]);
    }
    // whole 2 MiB pages per slot, so that a slot's graph arrays share one page
    off = (off + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
    return off;
}

__device__ Graph make_graph(const PoaArgs& a, uint32_t slot) {
    uint8_t* base = a.scratch + size_t(slot) * a.slot_bytes;
    Graph g;
    void* p[kGraphArrays];
    walk_layout(a.ncap, a.ecap, a.acap, a.lcap, [&](int id, size_t off) { p[id] = base + off; });
    int id = 0;
    auto set = [&](auto*& m) { m = static_cast<std::remove_reference_t<decltype(m)>>(p[id++]); };
    set(g.code), set(g.flag), set(g.cov), set(g.in_cnt), set(g.out_cnt), set(g.al_cnt), set(g.in_src), set(g.in_w);
    set(g.ov_head), set(g.ov_tail), set(g.al4), set(g.al_head), set(g.al_tail);
    set(g.e_src), set(g.e_w), set(g.e_next), set(g.a_node), set(g.a_next);
    set(g.ord), set(g.ord2), set(g.rank), set(g.shift), set(g.dporder), set(g.sub_rank), set(g.dfs), set(g.dfs_rank);
    set(g.stack), set(g.rowdesc), set(g.pred_idx), set(g.used), set(g.sink_rows), set(g.sink_h);
    set(g.path), set(g.nid), set(g.slot), set(g.new_slot), set(g.bscore), set(g.bpred), set(g.cons), set(g.H);
    g.ncap = a.ncap;
    g.ecap = a.ecap;
    g.acap = a.acap;
    g.scap = a.ncap + a.ecap + a.acap + 16;
    g.lcap = a.lcap;
    return g;
}

// Shared per-team state.
struct PoaShared {
    int nnodes, nseq;
    int nedges, naligned;  // entries of the overflow pools in use
    int nnew;              // new nodes of the last insertion
    int fail;              // 0 ok, else PoaFlag
    int ndp;               // rows of the current DP
    int nsinks, nlisted;   // sink rows; entries of pred_idx in use
    int preds;             // predecessor links over the DP rows (edge-cells = |layer| x (rows + preds))
    int end_value;         // score of the NW end cell of the current layer
    int scratch_bytes;     // the team's shared memory, scratch between the DPs
    uint32_t next;         // queue position the team took
    volatile int done[4];  // per warp: rows it has finished (counting on from pass to pass)
    volatile int wait_polls;  // limit of the waits on done, 0 once one of them ran out
};

// ---------------- team memory ----------------

// the CTA's dynamic shared memory: WarpMem<NW>::bytes per warp, teams in order
extern __shared__ int4 g_poa_smem[];

// Shared memory of one warp of a team of NW: the ring of DP rows, the
// staged controls and score words of 32 rows, and the final scores at the
// right edge of the strip to its left. Between layers the whole team's
// memory is scratch for the graph steps. An SM holds 12 one-warp teams or 24
// warps of four-warp teams. (16 and 20 one-warp teams with fewer rows and
// registers each raise the throughput of the DP alone, but finish a batch's
// slowest windows later: 2001 windows at 50x 78.7 ms with 12, 83 with 16, 93
// with 20.)
constexpr int kEdgeRows = 64;
template <int NW>
struct WarpMem {
    static constexpr int ring_bytes = NW == 1 ? 17408 : 8064;
    static constexpr int ctl = ring_bytes;          // uint32_t[33]: a block's rows and 0
    static constexpr int pool = ctl + 36 * 4;       // uint32_t[32]
    static constexpr int edge = pool + 32 * 4 + 16; // int[kEdgeRows]
    static constexpr int bytes = edge + kEdgeRows * 4;
};
// rows between two looks at the neighbouring warps' progress
constexpr int kGroupRows = 8;
// Polls of a wait on another warp of the team before the window is given up as
// failed: a poll takes 75 cycles or more, so the wait at least 0.15 s, where
// the rows waited for take microseconds.
constexpr int kWaitPolls = 1 << 22;

// Waits until `done` reaches `want`. When that takes too long the window is
// given up, and the team waits no more: its warps run through their rows (whose
// scores nothing reads), every further wait a single poll. (Leaving the strip
// instead cost every row 5 %.)
__device__ __forceinline__ void wait_rows(PoaShared& sh, const volatile int& done, int want) {
    if (!__any_sync(0xffffffffu, done < want)) return;
    int left = sh.wait_polls;
    do {
        if (left-- <= 0) {
            sh.fail = kFailed;
            sh.wait_polls = 0;
            break;
        }
    } while (__any_sync(0xffffffffu, done < want));
}

// Barrier of the NW warps of one team (hardware barrier team + 1).
template <int NW>
__device__ __forceinline__ void team_sync(int team) {
    if (NW == 1) {
        __syncwarp();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(32 * NW) : "memory");
    }
}

// slanted score (row r, column j) as the layer stored it, rows of lc columns
template <bool FAST>
__device__ __forceinline__ int h_at(const uint8_t* Hb, int r, int j, int lc) {
    if (FAST) return reinterpret_cast<const int16_t*>(Hb)[size_t(r) * lc + j];
    return reinterpret_cast<const int*>(Hb)[size_t(r) * lc + j];
}

// ---------------- graph primitives ----------------

// In-edges of node v in spoa's order (the order in which they were added):
// f(source, weight); f returns false to stop.
template <class F>
__device__ __forceinline__ void for_in_edges(const Graph& g, int v, F&& f) {
    const int n = g.in_cnt[v];
    const int* s = reinterpret_cast<const int*>(g.in_src + 2 * size_t(v));
    const int* wt = reinterpret_cast<const int*>(g.in_w + 2 * size_t(v));
    for (int q = 0; q < min(n, kInline); ++q)
        if (!f(s[q], wt[q])) return;
    if (n > kInline)
        for (int e = g.ov_head[v]; e != -1; e = g.e_next[e])
            if (!f(g.e_src[e], g.e_w[e])) return;
}

// Nodes aligned to v, in the order in which they were linked: f(node) as above.
template <class F>
__device__ __forceinline__ void for_aligned(const Graph& g, int v, F&& f) {
    const int n = g.al_cnt[v];
    const int* s = reinterpret_cast<const int*>(g.al4 + v);
    for (int q = 0; q < min(n, 4); ++q)
        if (!f(s[q])) return;
    if (n > 4)
        for (int x = g.al_head[v]; x != -1; x = g.a_next[x])
            if (!f(g.a_node[x])) return;
}

// Links node y to v's aligned list. Only one thread of the team touches v's
// group during an insertion.
__device__ __forceinline__ void link_aligned(const Graph& g, PoaShared& sh, int v, int y) {
    const int n = g.al_cnt[v];
    g.al_cnt[v] = n + 1;
    if (n < 4) {
        reinterpret_cast<int*>(g.al4 + v)[n] = y;
        return;
    }
    const int x = atomicAdd(&sh.naligned, 1);
    if (x >= g.acap) {
        sh.fail = kOverflow;
        return;
    }
    g.a_node[x] = y;
    g.a_next[x] = -1;
    if (n == 4) {
        g.al_head[v] = x;
    } else {
        g.a_next[g.al_tail[v]] = x;
    }
    g.al_tail[v] = x;
}

__device__ int layer_weight(const uint8_t* qual, int k) { return qual ? int(qual[k]) - 33 : 1; }

// Warp prefix helpers: exclusive prefix of v over lanes, and the total.
__device__ __forceinline__ int warp_excl(int v, int lane, int& total) {
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// ---------------- rows of one layer's DP ----------------

// Row descriptor: word w holds the predecessor count (17 bits) and the base
// (<< 24). Up to kPacked predecessors' ranks sit in x, y, z as 16-bit halves;
// more of them, or any in a graph of 65536 rows or more (kWide), in pred_idx
// from x on.
constexpr int kPacked = 6;
constexpr int kWide = 1 << 17;
constexpr int kPrev = 1 << 18;  // a listed row's predecessors include the row before it
__device__ __forceinline__ int desc_np(int w) { return w & 0x1FFFF; }
__device__ __forceinline__ uint32_t desc_base(int w) { return uint32_t(w) >> 24; }
__device__ __forceinline__ bool desc_listed(int w) { return desc_np(w) > kPacked || (w & kWide) != 0; }
// Packed predecessor p (in in-edge order).
__device__ __forceinline__ int desc_packed(const int4& d, int p) {
    const int q = p < 2 ? d.x : p < 4 ? d.y : d.z;
    return (p & 1) ? int(unsigned(q) >> 16) : q & 0xFFFF;
}
// Predecessor p of a row: DP rank (0 = the empty prefix row when the row has
// no predecessor).
__device__ __forceinline__ int desc_pred(const int* pred_idx, const int4& d, int p) {
    if (desc_np(d.w) == 0) return 0;
    return desc_listed(d.w) ? pred_idx[d.x + p] : desc_packed(d, p);
}

// Descriptors of rows order[0 .. ndp), ranks 1 .. ndp, and the list of sink
// rows (no successor row), by the team, four rows per thread at a time so
// that one memory latency covers them. rk(v) is node v's DP rank, 0 when it
// is no row; the ranks go to shared memory as 16-bit words when they fit. With
// `partial` predecessors outside the rows are dropped and a row is a sink when
// no row lists it; otherwise a sink is a node without out-edges.
template <int NW>
__device__ void build_rows(const Graph& g, PoaShared& sh, const int* order, int ndp, bool partial, int tid, int team,
                           uint8_t* smem) {
    constexpr int NT = 32 * NW;
    const int N = sh.nnodes;
    const int* const grk = partial ? g.sub_rank : g.rank;
    const int up = partial ? 0 : 1;  // g.rank counts from 0
    const size_t rk_bytes = (2 * size_t(N) + 3) & ~size_t(3);
    const bool in_smem = N < 65535 && rk_bytes + (partial ? size_t(ndp) + 1 : 0) <= size_t(sh.scratch_bytes);
    uint16_t* const rk16 = reinterpret_cast<uint16_t*>(smem);
    uint8_t* const succ = in_smem ? smem + rk_bytes : g.flag;
    const bool wide = ndp >= 65536;
    for (int k = tid; k <= ndp / 32; k += NT) g.used[k] = 0u;
    if (in_smem)
        for (int c0 = tid; c0 < N; c0 += 4 * NT) {
            int r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) r[u] = c0 + u * NT < N ? grk[c0 + u * NT] : 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c0 + u * NT < N) rk16[c0 + u * NT] = uint16_t(r[u] + up);
        }
    if (partial)
        for (int i = tid; i <= ndp; i += NT) succ[i] = 0;
    if (tid == 0) {
        sh.nsinks = 0;
        sh.preds = 0;
        sh.nlisted = 0;
    }
    team_sync<NW>(team);
    auto rk = [&](int v) -> int { return in_smem ? int(rk16[v]) : grk[v] + up; };
    int preds = 0;
    for (int c0 = tid; c0 < ndp; c0 += 4 * NT) {
        int v[4], cnt[4], oc[4];
        uint8_t code[4];
        int4 s0[4], s1[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = c0 + u * NT < ndp ? order[c0 + u * NT] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            cnt[u] = g.in_cnt[v[u]];
            oc[u] = partial ? 1 : g.out_cnt[v[u]];
            code[u] = g.code[v[u]];
            s0[u] = g.in_src[2 * size_t(v[u])];
            s1[u] = g.in_src[2 * size_t(v[u]) + 1];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = c0 + u * NT;
            if (i >= ndp) continue;
            int np = 0;
            bool prev = false;
            int4 d = make_int4(0, 0, 0, 0);
            auto add = [&](int src) {
                const int r = rk(src);
                if (r == 0) return;
                // row i + 1's predecessor r
                if (r == i) {
                    prev = true;
                } else {
                    atomicOr(&g.used[(r - 1) >> 5], 1u << ((r - 1) & 31));
                }
                const int h = r << (16 * (np & 1));
                if (np < 2) d.x |= h;
                else if (np < 4) d.y |= h;
                else if (np < 6) d.z |= h;
                ++np;
                if (partial) succ[r] = 1;  // every writer stores the same value
            };
            const int c = cnt[u];
            if (c > 0) add(s0[u].x);
            if (c > 1) add(s0[u].y);
            if (c > 2) add(s0[u].z);
            if (c > 3) add(s0[u].w);
            if (c > 4) {
                add(s1[u].x);
                if (c > 5) add(s1[u].y);
                if (c > 6) add(s1[u].z);
                if (c > 7) add(s1[u].w);
                if (c > kInline)
                    for (int e = g.ov_head[v[u]]; e != -1; e = g.e_next[e]) add(g.e_src[e]);
            }
            if (np > kPacked || (wide && np > 0)) {
                const int off = atomicAdd(&sh.nlisted, np);
                int k = off;
                for_in_edges(g, v[u], [&](int src, int) {
                    const int r = rk(src);
                    if (r != 0) g.pred_idx[k++] = r;
                    return true;
                });
                d = make_int4(off, 0, 0, (wide ? kWide : 0) | (prev ? kPrev : 0));
            }
            d.w |= np | int(uint32_t(code[u]) << 24);
            g.rowdesc[i] = d;
            preds += np;
            if (!partial && oc[u] == 0) g.sink_rows[atomicAdd(&sh.nsinks, 1)] = i + 1;
        }
    }
    preds = __reduce_add_sync(0xffffffffu, preds);
    if ((tid & 31) == 0 && preds) atomicAdd(&sh.preds, preds);
    if (partial) {
        team_sync<NW>(team);
        for (int i = 1 + tid; i <= ndp; i += NT)
            if (!succ[i]) g.sink_rows[atomicAdd(&sh.nsinks, 1)] = i;
    }
    team_sync<NW>(team);
}

// spoa's subgraph of a partial layer: the nodes reached from end_node
// backwards over in-edges and aligned links, going on only from nodes whose id
// is not below begin_node. A sweep down the incremental order, in which every
// aligned group is contiguous and a group's successors all come after it, 32
// rows at a time, one per lane: within a chunk the reached rows grow to their
// closure over the lanes' predecessor and group masks, one warp reduction a
// step; then the chunk's rows mark their predecessors below it. A chunk ends
// at a group's edge, so that all links into a group are known when its chunk
// comes. (One lane following the links from row to row took 380 k cycles a
// layer of 24 reads against 64 k.) Leaves the rows in g.dporder (sh.ndp of them) and
// every node's DP rank (0: none) in g.sub_rank. The descriptors are those of
// the whole graph (build_rows). By the team.
template <int NW>
__device__ void mark_subgraph(const Graph& g, PoaShared& sh, int begin_node, int end_node, int lane, int w, int team,
                              uint8_t* smem) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int NT = 32 * NW;
    constexpr int kReached = 1, kInside = 2;  // flags; inside: id >= begin_node
    const int tid = 32 * w + lane;
    const int N = sh.nnodes;
    if (end_node < 0 || end_node >= N) {
        if (tid == 0) {
            sh.fail = kFailed;
            sh.ndp = 0;
        }
        team_sync<NW>(team);
        return;
    }
    // per row (by rank, from 0): flags, rows down to its group's first and up to its last
    const bool in_smem = 3 * size_t(N) <= size_t(sh.scratch_bytes);
    uint8_t* const flag = in_smem ? smem : g.flag;
    uint8_t* const down = in_smem ? smem + N : reinterpret_cast<uint8_t*>(g.shift);
    uint8_t* const upto = in_smem ? smem + 2 * size_t(N) : down + N;
    bool big = false;
    for (int c0 = tid; c0 < N; c0 += 4 * NT) {
        int v[4], ac[4];
        int4 al[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = c0 + u * NT < N ? g.ord[c0 + u * NT] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            ac[u] = g.al_cnt[v[u]];
            al[u] = g.al4[v[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = c0 + u * NT;
            if (r >= N) continue;
            int lo = r, hi = r;
            const int ys[4] = {al[u].x, al[u].y, al[u].z, al[u].w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int ry = q < ac[u] ? g.rank[ys[q]] : r;
                lo = min(lo, ry);
                hi = max(hi, ry);
            }
            if (ac[u] > 4)
                for_aligned(g, v[u], [&](int y) {
                    lo = min(lo, g.rank[y]);
                    hi = max(hi, g.rank[y]);
                    return true;
                });
            big |= hi - lo >= 32;
            flag[r] = uint8_t((v[u] == end_node ? kReached : 0) | (v[u] >= begin_node ? kInside : 0));
            down[r] = uint8_t(min(r - lo, 255));
            upto[r] = uint8_t(min(hi - r, 255));
        }
    }
    if (tid == 0) sh.nlisted = 0;
    team_sync<NW>(team);
    if (__any_sync(kFull, big) && lane == 0) sh.nlisted = 1;  // a group of more than 32 rows
    team_sync<NW>(team);
    const bool chunks = sh.nlisted == 0;
    if (w == 0) {
        if (chunks) {
            const int re = g.rank[end_node];
            int hi = re + upto[re];
            int4 next = hi - 31 + lane >= 0 ? g.rowdesc[hi - 31 + lane] : make_int4(0, 0, 0, 0);
            while (hi >= 0) {
                // rows [lo, hi]; lane l holds row base + l
                const int base = hi - 31;
                const int r = base + lane;
                const int4 d = next;
                const int first = max(base, 0);
                const int dn = down[first];
                const int lo = dn > 0 && first > 0 ? first + 1 + upto[first] : first;  // a group cut in two waits
                const int hn = lo - 1;
                const int rn = hn - 31 + lane;
                next = hn >= 0 && rn >= 0 ? g.rowdesc[rn] : make_int4(0, 0, 0, 0);
                const bool mine = r >= lo;
                const int fl = mine ? flag[r] : 0;
                const int np = mine ? desc_np(d.w) : 0;
                unsigned links = 0;
                if (mine) {
                    const int gl = lane - int(down[r]), gh = lane + int(upto[r]);
                    links = (0xffffffffu >> (31 - gh)) & (0xffffffffu << gl);
                    for (int p = 0; p < np; ++p) {
                        const int q = desc_pred(g.pred_idx, d, p) - 1 - base;
                        if (q >= lo - base) links |= 1u << q;
                    }
                }
                unsigned m = __ballot_sync(kFull, (fl & kReached) != 0);
                if (m != 0) {
                    const bool inside = (fl & kInside) != 0;
                    for (;;) {
                        const unsigned t =
                            m | __reduce_or_sync(kFull, inside && ((m >> lane) & 1u) ? links : 0u);
                        if (t == m) break;
                        m = t;
                    }
                    if ((m >> lane) & 1u) {
                        flag[r] = uint8_t(fl | kReached);
                        if (inside)
                            for (int p = 0; p < np; ++p) {
                                const int q = desc_pred(g.pred_idx, d, p) - 1;
                                if (q < lo) flag[q] = uint8_t(flag[q] | kReached);  // same value from every lane
                            }
                    }
                    __syncwarp();
                }
                hi = hn;
            }
        } else if (lane == 0) {
            // groups of more than 32 rows: follow the links
            int sp = 0;
            g.stack[sp++] = end_node;
            flag[g.rank[end_node]] &= uint8_t(~kReached);
            bool room = true;
            while (sp > 0 && room) {
                const int v = g.stack[--sp];
                const int r = g.rank[v];
                if ((flag[r] & kReached) || !(flag[r] & kInside)) continue;
                flag[r] |= kReached;
                for_in_edges(g, v, [&](int u, int) {
                    room = sp < g.scap;
                    if (room) g.stack[sp++] = u;
                    return room;
                });
                for_aligned(g, v, [&](int y) {
                    room = room && sp < g.scap;
                    if (room) g.stack[sp++] = y;
                    return room;
                });
            }
            if (!room) {
                sh.fail = kOverflow;
                for (int r = 0; r < N; ++r) flag[r] = 0;
            }
        }
        __syncwarp();
        // the rows, in order; the loads of four 32-row chunks go out together
        int cnt = 0;
        for (int c4 = 0; c4 < N; c4 += 128) {
            int vv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) vv[u] = c4 + 32 * u + lane < N ? g.ord[c4 + 32 * u + lane] : -1;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = c4 + 32 * u + lane;
                const bool in = vv[u] >= 0 && flag[r] == (kReached | kInside);
                const unsigned m = __ballot_sync(kFull, in);
                const int k = cnt + __popc(m & ((1u << lane) - 1u));
                if (vv[u] >= 0) g.sub_rank[vv[u]] = in ? k + 1 : 0;
                if (in) g.dporder[k] = vv[u];
                cnt += __popc(m);
            }
        }
        if (lane == 0) sh.ndp = cnt;
    }
    team_sync<NW>(team);
}

// ---------------- spoa's depth-first topological order ----------------

// spoa's DFS order over the nodes x with member(x), written to out; returns
// its length, -1 when the stack (cap entries) overflows. ins(v, f) and als(v,
// f) go through v's in-edge sources and aligned nodes; state(x) is a byte per
// node, cleared: bits 0-1 mark, bit 2 set once x is no primary of its group.
template <class Ins, class Als, class Mem, class Stack>
__device__ int dfs_order(int N, Ins&& ins, Als&& als, Mem&& member, uint8_t* state, Stack* stack, int cap, int* out) {
    int nr = 0, sp = 0;
    for (int i = 0; i < N; ++i) {
        if (!member(i) || (state[i] & 3) != 0) continue;
        stack[sp++] = Stack(i);
        while (sp > 0) {
            const int v = stack[sp - 1];
            const int sv = state[v];
            bool valid = true, room = true;
            if ((sv & 3) != 2) {
                ins(v, [&](int u) {
                    if (!member(u) || (state[u] & 3) == 2) return true;
                    room = sp < cap;
                    if (room) stack[sp++] = Stack(u);
                    valid = false;
                    return room;
                });
                if (!(sv & 4))
                    als(v, [&](int y) {
                        if (!member(y) || (state[y] & 3) == 2) return true;
                        room = room && sp < cap;
                        if (room) stack[sp++] = Stack(y);
                        state[y] |= 4;
                        valid = false;
                        return room;
                    });
                if (!room) return -1;
                if (valid) {
                    state[v] = uint8_t((sv & ~3) | 2);
                    if (!(sv & 4)) {
                        out[nr++] = v;
                        als(v, [&](int y) {
                            if (member(y)) out[nr++] = y;
                            return true;
                        });
                    }
                } else {
                    state[v] = uint8_t((sv & ~3) | 1);
                }
            }
            if (valid) --sp;
        }
    }
    return nr;
}

// spoa's topological order of the whole graph (g.sub_rank unused) or of the
// rows of a partial layer, into g.dfs; its inverse into g.dfs_rank. In-edge
// and aligned lists, states and the stack sit in shared memory as 16-bit
// words when they fit, else the lists are walked in global memory. Warp 0; the
// count is returned on every lane (-1: stack overflow).
__device__ int topo_sort_warp(const Graph& g, PoaShared& sh, bool partial, int lane, uint8_t* smem) {
    constexpr unsigned kFull = 0xffffffffu;
    const int N = sh.nnodes;
    auto member = [&](int x) { return !partial || g.sub_rank[x] != 0; };
    // list offsets by warp prefix of the counts
    uint16_t* const in_off = reinterpret_cast<uint16_t*>(smem);
    uint16_t* const al_off = in_off + (N + 1);
    bool fits = N < 65535 && 5 * size_t(N) + 8 <= size_t(sh.scratch_bytes);
    int E = 0, A = 0;
    if (fits) {
        for (int c4 = 0; c4 < N; c4 += 128) {
            int ci[4], ca[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int v = c4 + 32 * u + lane;
                ci[u] = v < N ? g.in_cnt[v] : 0;
                ca[u] = v < N ? g.al_cnt[v] : 0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int v = c4 + 32 * u + lane;
                int ti = 0, ta = 0;
                const int xi = warp_excl(ci[u], lane, ti), xa = warp_excl(ca[u], lane, ta);
                if (v < N) {
                    in_off[v] = uint16_t(E + xi);
                    al_off[v] = uint16_t(A + xa);
                }
                E += ti;
                A += ta;
            }
        }
        // lists, a state byte per node, and a stack of at least N + 64 entries
        fits = E < 65535 && A < 65535 &&
               2 * (size_t(N) + 1) * 2 + 2 * size_t(E) + 2 * size_t(A) + size_t(N) + 2 * (size_t(N) + 64) <=
                   size_t(sh.scratch_bytes);
    }
    int nr = -1;
    if (fits) {
        if (lane == 0) {
            in_off[N] = uint16_t(E);
            al_off[N] = uint16_t(A);
        }
        uint16_t* const in_src = al_off + (N + 1);
        uint16_t* const al_x = in_src + E;
        uint16_t* const stack = al_x + A;
        uint8_t* const end = smem + sh.scratch_bytes;
        uint8_t* const state = end - N;
        const int cap = int((state - reinterpret_cast<uint8_t*>(stack)) / 2);
        __syncwarp();
        for (int v = lane; v < N; v += 32) {
            int q = in_off[v], x = al_off[v];
            for_in_edges(g, v, [&](int s, int) {
                in_src[q++] = uint16_t(s);
                return true;
            });
            for_aligned(g, v, [&](int y) {
                al_x[x++] = uint16_t(y);
                return true;
            });
            // nodes outside the subgraph count as done and are never roots
            state[v] = member(v) ? 0 : 2;
        }
        __syncwarp();
        if (lane == 0)
            nr = dfs_order(
                N,
                [&](int v, auto&& f) {
                    for (int q = in_off[v], qe = in_off[v + 1]; q < qe; ++q)
                        if (!f(int(in_src[q]))) return;
                },
                [&](int v, auto&& f) {
                    for (int q = al_off[v], qe = al_off[v + 1]; q < qe; ++q)
                        if (!f(int(al_x[q]))) return;
                },
                [&](int) { return true; }, state, stack, cap, g.dfs);
        // members of a group outside the subgraph were listed with it
        if (partial) {
            nr = __shfl_sync(kFull, nr, 0);
            __syncwarp();  // lane 0's list (a shuffle orders no memory)
            int k = 0;
            for (int c0 = 0; c0 < nr; c0 += 32) {
                const int v = c0 + lane < nr ? g.dfs[c0 + lane] : -1;
                const bool in = v >= 0 && member(v);
                const unsigned m = __ballot_sync(kFull, in);
                __syncwarp();
                if (in) g.dfs[k + __popc(m & ((1u << lane) - 1u))] = v;
                k += __popc(m);
                __syncwarp();
            }
            nr = nr < 0 ? nr : k;
        }
        nr = __shfl_sync(kFull, nr, 0);
    }
    if (nr < 0) {
        __syncwarp();
        for (int v = lane; v < N; v += 32) g.flag[v] = 0;
        __syncwarp();
        if (lane == 0)
            nr = dfs_order(
                N,
                [&](int v, auto&& f) { for_in_edges(g, v, [&](int s, int) { return f(s); }); },
                [&](int v, auto&& f) { for_aligned(g, v, f); }, member, g.flag, g.stack, g.scap, g.dfs);
        nr = __shfl_sync(kFull, nr, 0);
    }
    __syncwarp();
    for (int r = lane; r < nr; r += 32) g.dfs_rank[g.dfs[r]] = r;
    __syncwarp();
    return nr;
}

// ---------------- NW end row ----------------

// The first sink row with the best last-column score, or, when several sinks
// share it, the first of them in spoa's topological order of the (sub)graph.
// Sets sh.end_value. Warp 0.
//
// spoa's order lists nodes by the root of the DFS that reaches them, roots in
// ascending id. Three facts order nearly all tied sinks without the DFS:
// a sink outside every aligned group is its own root (nothing else leads to
// it); a group with a backbone node x (id below B) is reached from root x,
// no earlier (every earlier root precedes x on the backbone, so the group is
// none of its ancestors; B is the backbone's length); and x, the group's
// first visited node, is listed first and then its aligned list in order. A
// group without a backbone node is reached from the smallest id among its
// members and their descendants. Only several tied sinks of one such group
// whose root lies outside it need the DFS itself. (The DFS of 9 % of the
// layers cost as much as 30 % of all DP at 50x.)
constexpr int kSweepRows = 1024;
template <bool FAST>
__device__ int end_row(const Graph& g, PoaShared& sh, const int* order, int L, int lc, bool partial, int begin_node,
                       int B, int lane, uint8_t* smem) {
    constexpr unsigned kFull = 0xffffffffu;
    const uint8_t* const Hb = reinterpret_cast<const uint8_t*>(g.H);
    const int ns = sh.nsinks;
    int best = INT_MIN, low = INT_MAX, ties = 0;
    for (int k = lane; k < ns; k += 32) {
        const int i = g.sink_rows[k];
        const int v = h_at<FAST>(Hb, i, L, lc);
        g.sink_h[k] = v;
        ties = v > best ? 1 : ties + (v == best ? 1 : 0);
        low = v > best ? i : v == best ? min(low, i) : low;
        best = max(best, v);
    }
    const int top = __reduce_max_sync(kFull, best);
    if (best != top) {
        ties = 0;
        low = INT_MAX;
    }
    int iend = __reduce_min_sync(kFull, low);
    ties = __reduce_add_sync(kFull, ties);
    if (lane == 0) sh.end_value = top;
    __syncwarp();
    if (ties <= 1) return iend;
    // key: root id, then the place in the group's listing
    bool open = false;
    unsigned root = ~0u, place = ~0u;
    int row = iend;
    for (int k = lane; k < ns; k += 32) {
        if (g.sink_h[k] != top) continue;
        const int i = g.sink_rows[k];
        const int v = order[i - 1];
        int x = v;
        for_aligned(g, v, [&](int y) {
            if (y >= begin_node) x = min(x, y);
            return true;
        });
        unsigned pl = 0;
        if (g.al_cnt[v] != 0) {
            open |= x >= B;
            if (x != v) {
                unsigned at = 1;
                for_aligned(g, x, [&](int y) {
                    if (y == v) pl = at;
                    ++at;
                    return y != v;
                });
            }
        }
        if (unsigned(x) < root || (unsigned(x) == root && pl < place)) {
            root = unsigned(x);
            place = pl;
            row = i;
        }
    }
    bool sure = !__any_sync(kFull, open);
    if (!sure && !partial) {
        // a group without a backbone node is reached from the smallest id
        // among its members and all that follow it: swept down to the lowest
        // such group, from the last row (these sinks end the graph, so the
        // sweep is short)
        int lo = INT_MAX;
        for (int k = lane; k < ns; k += 32) {
            if (g.sink_h[k] != top) continue;
            const int v = order[g.sink_rows[k] - 1];
            int x = v, first = g.rank[v];
            for_aligned(g, v, [&](int y) {
                x = min(x, y);
                first = min(first, g.rank[y]);
                return true;
            });
            if (g.al_cnt[v] != 0 && x >= B) lo = min(lo, first);
        }
        lo = __reduce_min_sync(kFull, lo);
        const int N = sh.nnodes;
        if (N - lo <= kSweepRows && 4 * (N - lo) <= sh.scratch_bytes) {
            int* const from = reinterpret_cast<int*>(smem);  // [N - lo] smallest id reached from the row
            for (int r = lane; r < N - lo; r += 32) from[r] = g.ord[lo + r];
            __syncwarp();
            if (lane == 0)
                for (int r = N - 1; r >= lo; --r) {
                    const int v = g.ord[r];
                    int first = r;
                    bool last = true;
                    for_aligned(g, v, [&](int y) {
                        first = min(first, g.rank[y]);
                        last = last && g.rank[y] < r;
                        return last;
                    });
                    if (!last) continue;  // with its group's last row
                    int id = INT_MAX;
                    for (int x = max(first, lo); x <= r; ++x) id = min(id, from[x - lo]);
                    for (int x = max(first, lo); x <= r; ++x) {
                        from[x - lo] = id;
                        for_in_edges(g, g.ord[x], [&](int u, int) {
                            const int q = g.rank[u] - lo;
                            if (q >= 0) from[q] = min(from[q], id);
                            return true;
                        });
                    }
                }
            __syncwarp();
            root = place = ~0u;
            bool lost = false;  // tied sinks whose order within their root's search is not known
            int mates = 0;
            for (int pass = 0; pass < 2; ++pass) {
                const unsigned r0 = __reduce_min_sync(kFull, root);
                for (int k = lane; k < ns; k += 32) {
                    if (g.sink_h[k] != top) continue;
                    const int i = g.sink_rows[k];
                    const int v = order[i - 1];
                    int x = v;
                    for_aligned(g, v, [&](int y) {
                        x = min(x, y);
                        return true;
                    });
                    const unsigned id = g.al_cnt[v] != 0 && x >= B ? unsigned(from[i - 1 - lo]) : unsigned(x);
                    if (pass == 0) {
                        root = min(root, id);
                        continue;
                    }
                    if (id != r0) continue;
                    ++mates;
                    lost |= id != unsigned(x);  // the root is no member of the group
                    unsigned pl = 0, at = 1;
                    if (x != v)
                        for_aligned(g, x, [&](int y) {
                            if (y == v) pl = at;
                            ++at;
                            return y != v;
                        });
                    if (pl < place) {
                        place = pl;
                        row = i;
                    }
                }
                if (pass == 1) {
                    root = place != ~0u ? r0 : ~0u;
                    sure = __reduce_add_sync(kFull, mates) == 1 || !__any_sync(kFull, lost);
                }
            }
        }
        __syncwarp();
    }
    if (sure) {
        const unsigned r0 = __reduce_min_sync(kFull, root);
        const unsigned p0 = __reduce_min_sync(kFull, root == r0 ? place : ~0u);
        return __reduce_min_sync(kFull, unsigned(root == r0 && place == p0 ? row : INT_MAX));
    }
    const int nr = topo_sort_warp(g, sh, partial, lane, smem);
    if (nr < 0) {
        if (lane == 0) sh.fail = kOverflow;
        __syncwarp();
        return iend;
    }
    int first = INT_MAX, fi = iend;
    for (int k = lane; k < ns; k += 32) {
        if (g.sink_h[k] != top) continue;
        const int i = g.sink_rows[k];
        const int rr = g.dfs_rank[order[i - 1]];
        if (rr < first) {
            first = rr;
            fi = i;
        }
    }
    const int f0 = __reduce_min_sync(kFull, first);
    return __reduce_min_sync(kFull, first == f0 ? fi : INT_MAX);
}

// ---------------- adding a layer ----------------

// Graph::add_alignment for one layer, by the team. A path visits every node
// and every aligned group at most once, so the per-position work is
// independent: classify each base (existing node, new base, new member of an
// aligned group), number the new nodes in path order, then in parallel
// create nodes, aligned-group links, edges P[k-1] -> P[k] with weight w[k-1] +
// w[k] (every sequence position k owns exactly one path node P[k]) and
// coverage. In-edges sit with their node (kInline of them in two 16-byte
// words), so that finding or adding an edge reads only its head. Leaves the
// new nodes' order slots (see order_insert) in g.new_slot.
template <int NW>
__device__ void add_layer(const Graph& g, PoaShared& sh, const int* order, const uint8_t* seq, const uint8_t* qual,
                          int len, int lane, int w, int team, uint8_t* smem) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int NT = 32 * NW;
    const int tid = 32 * w + lane;
    const int nold = sh.nnodes;
    const bool in_smem = 8 * size_t(len) <= size_t(sh.scratch_bytes);
    int* const nid = in_smem ? reinterpret_cast<int*>(smem) : g.nid;  // node of position t, -1 until numbered
    int* const slot = in_smem ? nid + len : g.slot;                   // last rank of the position's group
    int* const path = g.path;
    // 1. classify (reads only the graph as it was before this insertion); the
    //    path's rows become nodes
    for (int t4 = tid; t4 < len; t4 += 4 * NT) {
        int at[4], ac[4], rk[4];
        uint8_t cd[4], ch[4];
        int4 al[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) at[u] = t4 + u * NT < len ? path[t4 + u * NT] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) at[u] = at[u] > 0 ? order[at[u] - 1] : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int v = max(at[u], 0);
            ch[u] = t4 + u * NT < len ? seq[t4 + u * NT] : 0;
            cd[u] = g.code[v];
            ac[u] = g.al_cnt[v];
            rk[u] = g.rank[v];
            al[u] = g.al4[v];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = t4 + u * NT;
            if (t >= len) continue;
            int n = -1, sl = INT_MIN;
            if (at[u] >= 0) {
                sl = rk[u];
                if (cd[u] == ch[u]) n = at[u];
                if (ac[u] > 0) {
                    const int ys[4] = {al[u].x, al[u].y, al[u].z, al[u].w};
                    int yr[4];
                    uint8_t yc[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int y = q < ac[u] ? ys[q] : at[u];
                        yr[q] = g.rank[y];
                        yc[q] = g.code[y];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        sl = max(sl, yr[q]);
                        if (n < 0 && q < ac[u] && yc[q] == ch[u]) n = ys[q];
                    }
                    if (ac[u] > 4)
                        for_aligned(g, at[u], [&](int y) {
                            sl = max(sl, g.rank[y]);
                            if (n < 0 && g.code[y] == ch[u]) n = y;
                            return true;
                        });
                }
            }
            path[t] = at[u];
            nid[t] = n;
            slot[t] = sl;
        }
    }
    team_sync<NW>(team);
    // 2. ids and order slots of the new nodes: a new member of a group goes
    //    behind the group, an inserted base behind the last anchor before it
    //    (anchors: positions on existing groups, whose ranks rise along the
    //    path), those before the first anchor in front of its group
    if (w == 0) {
        int nnew = 0, carry = INT_MIN;
        const int room = g.ncap - nold;
        for (int c0 = 0; c0 < len; c0 += 32) {
            const int t = c0 + lane;
            const bool on = t < len;
            const int n = on ? nid[t] : 0, s = on ? slot[t] : INT_MIN;
            const unsigned ba = __ballot_sync(kFull, s != INT_MIN);
            if (carry == INT_MIN && ba != 0) {
                // the first anchor: the slot in front of its group
                const int v = path[c0 + __ffs(ba) - 1];
                int st = g.rank[v];
                for_aligned(g, v, [&](int y) {
                    st = min(st, g.rank[y]);
                    return true;
                });
                carry = st - 1;
                // bases inserted so far were given the slot "before" below,
                // as many as the slot has room for, by other lanes
                __syncwarp();
                for (int k = lane; k < min(nnew, room); k += 32) g.new_slot[k] = carry;
            }
            const unsigned bn = __ballot_sync(kFull, on && n < 0);
            const unsigned upto = ba & (0xffffffffu >> (31 - lane));
            const int sl = __shfl_sync(kFull, s, upto ? 31 - __clz(upto) : 0);
            if (on && n < 0) {
                const int k = nnew + __popc(bn & ((1u << lane) - 1u));
                if (k < room) g.new_slot[k] = upto ? sl : carry == INT_MIN ? nold - 1 : carry;
                nid[t] = nold + k;
            }
            if (ba) carry = __shfl_sync(kFull, s, 31 - __clz(ba));
            nnew += __popc(bn);
        }
        if (lane == 0) {
            const bool fits = nnew <= room;
            sh.nnew = fits ? nnew : -1;
            if (!fits) sh.fail = kOverflow;
        }
        __syncwarp();
    }
    team_sync<NW>(team);
    // (not sh.fail, which a faster thread may set below while a slower one
    // still reads it here: all threads have to take the same way)
    if (sh.nnew < 0) return;
    // 3. new nodes, and their aligned groups: a new base joining the group of
    //    `at` links to every member, then to `at` (spoa's order)
    for (int t = tid; t < len; t += NT) {
        const int G = nid[t];
        if (G < nold) continue;
        g.code[G] = seq[t];
        g.cov[G] = 0;
        g.in_cnt[G] = 0;
        g.out_cnt[G] = 0;
        g.al_cnt[G] = 0;
        const int at = path[t];
        if (at >= 0) {
            for_aligned(g, at, [&](int y) {
                link_aligned(g, sh, G, y);
                link_aligned(g, sh, y, G);
                return true;
            });
            link_aligned(g, sh, G, at);
            link_aligned(g, sh, at, G);
        }
    }
    team_sync<NW>(team);
    // 4. edges P[k-1] -> P[k]: existing ones gain weight, new ones are
    //    appended (each node is head and tail of at most one of them);
    //    coverage of every node of a path with at least two bases
    for (int k = tid; k < len; k += NT) {
        const int v = nid[k];
        if (len >= 2) g.cov[v] += 1;
        if (k == 0) continue;
        const int u = nid[k - 1];
        const int wt = layer_weight(qual, k - 1) + layer_weight(qual, k);
        const int n = g.in_cnt[v];
        const int4 a = g.in_src[2 * size_t(v)], b = g.in_src[2 * size_t(v) + 1];
        int* const wv = reinterpret_cast<int*>(g.in_w + 2 * size_t(v));
        int q = -1;
        if (n > 7 && b.w == u) q = 7;
        if (n > 6 && b.z == u) q = 6;
        if (n > 5 && b.y == u) q = 5;
        if (n > 4 && b.x == u) q = 4;
        if (n > 3 && a.w == u) q = 3;
        if (n > 2 && a.z == u) q = 2;
        if (n > 1 && a.y == u) q = 1;
        if (n > 0 && a.x == u) q = 0;
        if (q >= 0) {
            wv[q] += wt;
            continue;
        }
        if (n > kInline) {
            int e = g.ov_head[v];
            while (e != -1 && g.e_src[e] != u) e = g.e_next[e];
            if (e != -1) {
                g.e_w[e] += wt;
                continue;
            }
        }
        if (n < kInline) {
            reinterpret_cast<int*>(g.in_src + 2 * size_t(v))[n] = u;
            wv[n] = wt;
        } else {
            const int e = atomicAdd(&sh.nedges, 1);
            if (e >= g.ecap) {
                sh.fail = kOverflow;
                continue;
            }
            g.e_src[e] = u;
            g.e_w[e] = wt;
            g.e_next[e] = -1;
            if (n == kInline) {
                g.ov_head[v] = e;
            } else {
                g.e_next[g.ov_tail[v]] = e;
            }
            g.ov_tail[v] = e;
        }
        g.in_cnt[v] = n + 1;
        g.out_cnt[u] += 1;
    }
    team_sync<NW>(team);
    if (tid == 0) {
        sh.nnodes = nold + sh.nnew;
        sh.nseq += 1;
    }
}

// Splices the new nodes of the last insertion into the incremental order
// (team): an old node at rank r moves up by the number of new nodes with slot
// < r, the k-th new node (slots rise along the path) lands at slot + 1 + k.
template <int NW>
__device__ void order_insert(Graph& g, PoaShared& sh, int lane, int w, int team, uint8_t* smem) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int NT = 32 * NW;
    const int tid = 32 * w + lane;
    const int nnew = sh.nnew;
    team_sync<NW>(team);  // sh.nnodes is the new count on every thread
    const int nold = sh.nnodes - nnew;
    if (nnew == 0) return;
    int* const shift = (size_t(nold) + 1) * 4 <= size_t(sh.scratch_bytes) ? reinterpret_cast<int*>(smem) : g.shift;
    for (int r = tid; r <= nold; r += NT) shift[r] = 0;
    team_sync<NW>(team);
    for (int k = tid; k < nnew; k += NT) {
        const int at = g.new_slot[k] + 1;
        if (at < nold) atomicAdd(&shift[at], 1);
    }
    team_sync<NW>(team);
    if (w == 0) {
        // inclusive prefix, four independent 32-rank chunks at a time
        int base = 0;
        for (int c4 = 0; c4 < nold; c4 += 128) {
            int x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = c4 + 32 * u + lane < nold ? shift[c4 + 32 * u + lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int y = __shfl_up_sync(kFull, x[u], o);
                    if (lane >= o) x[u] += y;
                }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (c4 + 32 * u + lane < nold) shift[c4 + 32 * u + lane] = base + x[u];
                base += __shfl_sync(kFull, x[u], 31);
            }
        }
        __syncwarp();
    }
    team_sync<NW>(team);
    for (int c0 = tid; c0 < nold; c0 += 4 * NT) {
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = c0 + u * NT < nold ? g.ord[c0 + u * NT] : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v[u] >= 0) {
                const int r = c0 + u * NT + shift[c0 + u * NT];
                g.ord2[r] = v[u];
                g.rank[v[u]] = r;
            }
    }
    for (int k = tid; k < nnew; k += NT) {
        const int r = g.new_slot[k] + 1 + k;
        g.ord2[r] = nold + k;
        g.rank[nold + k] = r;
    }
    team_sync<NW>(team);
    if (tid == 0) {
        int* const t = g.ord;
        g.ord = g.ord2;
        g.ord2 = t;
    }
    team_sync<NW>(team);
}

// ---------------- consensus ----------------

// Heaviest bundle over the nodes in the order given (any topological order
// gives the same scores and predecessors), 64-bit, in global memory (lane 0).
__device__ void bundle_scores(const Graph& g, const int* order, int N) {
    for (int r = 0; r < N; ++r) {
        const int v = order[r];
        long long s = -1;
        int p = -1;
        for_in_edges(g, v, [&](int u, int wt) {
            const long long x = wt;
            if (s < x || (s == x && p != -1 && g.bscore[p] <= g.bscore[u])) {
                s = x;
                p = u;
            }
            return true;
        });
        g.bscore[v] = p != -1 ? s + g.bscore[p] : s;
        g.bpred[v] = p;
    }
}

// spoa's choice of the consensus' last node and its branch completion, over
// scores and predecessors by node (in shared memory where they fit): the first
// node of the best score in g.dfs, and, while that node has out-edges, the best
// of the nodes after it once the other ways into its successors are struck
// out and the scores behind it are computed again. Leaves the path back in
// g.cons and returns its length (-1: no end). Warp 0. The successors are found
// from all nodes' in-edges, four nodes a lane in flight, and the in-edges of 32
// nodes at a time are staged for the one lane that goes down the order.
// (2000 windows of 500 bases whose 12 layers all end inside the window took 28.3
// ms with one lane going through all in-edges in global memory, now 9.2; 500
// such windows 22.1, now 3.6.)
constexpr int kStagedBytes = 32 * (kInline * 8 + 8);
template <class Score, class Pred>
__device__ __noinline__ int best_path(const Graph& g, int N, Score* score, Pred* pred, int lane, uint8_t* staged) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr Pred kNone = Pred(-1);
    int* const su = reinterpret_cast<int*>(staged);  // [32][kInline] sources
    int* const sw = su + 32 * kInline;               // [32][kInline] weights
    int* const sv = sw + 32 * kInline;               // [32] node
    int* const sd = sv + 32;                         // [32] degree
    // spoa starts from node 0, whose score counts as -1 (no score is lower)
    Score top = -1;
    int rank = INT_MAX;
    for (int r = lane; r < N; r += 32) {
        const Score x = score[g.dfs[r]];
        if (x > top) {
            top = x;
            rank = r;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const Score x = __shfl_xor_sync(kFull, top, o);
        const int r = __shfl_xor_sync(kFull, rank, o);
        if (x > top || (x == top && r < rank)) {
            top = x;
            rank = r;
        }
    }
    int best = rank == INT_MAX ? 0 : g.dfs[rank];
    for (int guard = 0; g.out_cnt[best] != 0; ++guard) {
        if (guard > N + 1) return -1;
        for (int d4 = lane; d4 < N; d4 += 128) {
            int n[4];
            int4 a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int d = min(d4 + 32 * u, N - 1);
                n[u] = d4 + 32 * u < N ? g.in_cnt[d] : 0;
                a[u] = g.in_src[2 * size_t(d)];
                b[u] = g.in_src[2 * size_t(d) + 1];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q[kInline] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
                bool head = n[u] > kInline;
#pragma unroll
                for (int k = 0; k < kInline; ++k) head |= k < n[u] && q[k] == best;
                if (!head) continue;
                const int d = d4 + 32 * u;
                if (n[u] > kInline) {
                    head = false;
                    for_in_edges(g, d, [&](int x, int) {
                        head = x == best;
                        return !head;
                    });
                }
                if (head)
                    for_in_edges(g, d, [&](int x, int) {
                        if (x != best) score[x] = -1;  // every writer stores the same value
                        return true;
                    });
            }
        }
        __syncwarp();
        Score high = 0;
        int next = 0;
        for (int r0 = g.dfs_rank[best] + 1; r0 < N; r0 += 32) {
            const int r = r0 + lane;
            int deg = 0, v = 0;
            if (r < N) {
                v = g.dfs[r];
                deg = g.in_cnt[v];
                const int* s = reinterpret_cast<const int*>(g.in_src + 2 * size_t(v));
                const int* wt = reinterpret_cast<const int*>(g.in_w + 2 * size_t(v));
                for (int q = 0; q < min(deg, kInline); ++q) {
                    su[lane * kInline + q] = s[q];
                    sw[lane * kInline + q] = wt[q];
                }
            }
            sv[lane] = v;
            sd[lane] = deg;
            __syncwarp();
            if (lane == 0)
                for (int t = 0; t < min(32, N - r0); ++t) {
                    Score x = -1, xp = 0;
                    int p = -1;
                    auto consider = [&](int u, int wt) {
                        const Score at = score[u];
                        if (at == -1) return;
                        if (x < wt || (x == wt && p != -1 && xp <= at)) {
                            x = wt;
                            p = u;
                            xp = at;
                        }
                    };
                    const int n = sd[t];
                    for (int q = 0; q < min(n, kInline); ++q) consider(su[t * kInline + q], sw[t * kInline + q]);
                    if (n > kInline)
                        for (int e = g.ov_head[sv[t]]; e != -1; e = g.e_next[e]) consider(g.e_src[e], g.e_w[e]);
                    if (p != -1) x += xp;
                    score[sv[t]] = x;
                    pred[sv[t]] = p == -1 ? kNone : Pred(p);
                    if (high < x) {
                        high = x;
                        next = sv[t];
                    }
                }
            __syncwarp();
        }
        best = __shfl_sync(kFull, next, 0);
    }
    int len = 0;
    if (lane == 0) {
        int v = best;
        for (; pred[v] != kNone && len <= N; v = int(pred[v])) g.cons[len++] = v;
        if (len > N) {
            len = -1;
        } else {
            g.cons[len++] = v;
        }
    }
    len = __shfl_sync(kFull, len, 0);
    __syncwarp();
    return len;
}

// spoa's heaviest bundle: scores in topological order, the first node of the
// best score in spoa's DFS order, completed while it has out-edges, and the
// path back from it into g.cons (in reverse); returns the path length (-1 on
// failure) on every lane. Scores do not depend on which topological order
// they are computed in, so the incremental one serves, and the DFS order is
// only built when several nodes share the best score or the best has
// out-edges. Scores, predecessors and the ranks of 32 staged nodes' in-edges
// sit in shared memory when they fit (scores are bounded by sequences x 186 x
// nodes: two Phred values per sequence and edge, summed along a path). Warp 0.
__device__ int heaviest_bundle_warp(const Graph& g, PoaShared& sh, int lane, uint8_t* smem) {
    constexpr unsigned kFull = 0xffffffffu;
    const int N = sh.nnodes;
    int* const bs = reinterpret_cast<int*>(smem);                                // [N] by rank
    uint16_t* const bp = reinterpret_cast<uint16_t*>(smem + 4 * size_t(N));      // [N] by rank, 0xFFFF = none
    const size_t st_off = (6 * size_t(N) + 15) & ~size_t(15);
    int* const sw = reinterpret_cast<int*>(smem + st_off);                       // [32][kInline] weights
    uint16_t* const su = reinterpret_cast<uint16_t*>(sw + 32 * kInline);         // [32][kInline] source ranks
    int* const sd = reinterpret_cast<int*>(su + 32 * kInline);                   // [32] degree
    const size_t need = st_off + 32 * kInline * 6 + 32 * 4;
    const bool fits = N < 65535 && need <= size_t(sh.scratch_bytes) &&
                      double(sh.nseq + 1) * 186.0 * double(N + 1) < 2.0e9;
    int best_id = 0, ties = 0;
    if (fits) {
        int best = INT_MIN, best_r = 0;
        for (int r0 = 0; r0 < N; r0 += 32) {
            const int r = r0 + lane;
            int deg = 0;
            if (r < N) {
                const int v = g.ord[r];
                deg = g.in_cnt[v];
                const int* s = reinterpret_cast<const int*>(g.in_src + 2 * size_t(v));
                const int* wt = reinterpret_cast<const int*>(g.in_w + 2 * size_t(v));
                for (int q = 0; q < min(deg, kInline); ++q) {
                    su[lane * kInline + q] = uint16_t(g.rank[s[q]]);
                    sw[lane * kInline + q] = wt[q];
                }
            }
            sd[lane] = deg;
            __syncwarp();
            if (lane == 0) {
                const int cnt = min(32, N - r0);
                for (int t = 0; t < cnt; ++t) {
                    const int d = sd[t];
                    int s = -1, p = -1, sp = 0;
                    auto consider = [&](int u, int wt) {
                        const int su_ = bs[u];
                        if (s < wt || (s == wt && p != -1 && sp <= su_)) {
                            s = wt;
                            p = u;
                            sp = su_;
                        }
                    };
                    for (int q = 0; q < min(d, kInline); ++q) consider(su[t * kInline + q], sw[t * kInline + q]);
                    if (d > kInline)
                        for (int e = g.ov_head[g.ord[r0 + t]]; e != -1; e = g.e_next[e])
                            consider(g.rank[g.e_src[e]], g.e_w[e]);
                    if (p != -1) s += sp;
                    bs[r0 + t] = s;
                    bp[r0 + t] = p < 0 ? uint16_t(0xFFFF) : uint16_t(p);
                    if (s > best) {
                        best = s;
                        best_r = r0 + t;
                        ties = 1;
                    } else if (s == best) {
                        ++ties;
                    }
                }
            }
            __syncwarp();
        }
        best = __shfl_sync(kFull, best, 0);
        best_r = __shfl_sync(kFull, best_r, 0);
        ties = __shfl_sync(kFull, ties, 0);
        best_id = g.ord[best_r];
        if (ties == 1 && best > -1 && g.out_cnt[best_id] == 0) {
            int len = 0;
            if (lane == 0) {
                int r = best_r;
                for (; bp[r] != 0xFFFF; r = bp[r]) bs[len++] = r;  // in place of the scores
                bs[len++] = r;
            }
            len = __shfl_sync(kFull, len, 0);
            __syncwarp();
            for (int k = lane; k < len; k += 32) g.cons[k] = g.ord[bs[k]];
            __syncwarp();
            return len;
        }
        for (int r = lane; r < N; r += 32) {
            const int v = g.ord[r];
            g.bscore[v] = bs[r];
            g.bpred[v] = bp[r] == 0xFFFF ? -1 : g.ord[bp[r]];
        }
        __syncwarp();
    } else {
        if (lane == 0) bundle_scores(g, g.ord, N);
        __syncwarp();
    }
    // the general way: spoa's own order
    const int nr = topo_sort_warp(g, sh, false, lane, smem);
    if (nr < 0) {
        if (lane == 0) sh.fail = kOverflow;
        __syncwarp();
        return 0;
    }
    // scores and predecessors by node
    const size_t by_node = (6 * size_t(N) + 15) & ~size_t(15);
    if (!fits || by_node + kStagedBytes > size_t(sh.scratch_bytes))
        return best_path(g, N, g.bscore, g.bpred, lane, smem);
    for (int v = lane; v < N; v += 32) {
        bs[v] = int(g.bscore[v]);
        bp[v] = uint16_t(g.bpred[v]);
    }
    __syncwarp();
    return best_path(g, N, bs, bp, lane, smem + by_node);
}

// ---------------- DP of one layer (one team) ----------------

// Cells per lane for rows of wc columns: the team's NW strips of 32 * S
// columns cover the row in one pass where that fits in registers (768
// columns for one warp, 1024 for four), else in passes of the
// largest S.
__host__ __device__ inline int seg_cells(int nw, int wc) {
    if (nw == 4) return wc <= 256 ? 2 : wc <= 512 ? 4 : wc <= 768 ? 6 : 8;
    return wc <= 256 ? 8 : wc <= 512 ? 16 : wc <= 640 ? 20 : 24;
}
// Row stride of the score rows: whole passes.
__host__ __device__ inline int row_cover(int nw, int wc) {
    const int ch = 32 * nw * seg_cells(nw, wc);
    return ((wc + ch - 1) / ch) * ch;
}

// Scores are slanted (score_rows.hpp). Layers of bases A, C, G, T only whose
// scores fit (fast_scores) take the fast form, int16 rows; other layers the
// general form: int32 rows, characters compared. The DP is int32 in registers
// and in the ring either way.
__device__ __forceinline__ bool acgt_base(uint32_t c) {
    return ((0x47544341u >> (8 * ((c >> 1) & 3u))) & 0xFFu) == c;
}
// two scores in one word, lo in bits 0..15 and hi in bits 16..31
// (saturated: only columns past the layer's end can exceed 16 bits)
__device__ __forceinline__ uint32_t pack_s16(int lo, int hi) {
    uint32_t d;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(d) : "r"(hi), "r"(lo));
    return d;
}
__device__ __forceinline__ int unpack_lo(uint32_t w) { return int(w << 16) >> 16; }
__device__ __forceinline__ int unpack_hi(uint32_t w) { return int(w) >> 16; }
// Byte `sel & 7` (per nibble) of lo, sign extended by the nibble's top bit.
__device__ __forceinline__ int prmt_score(uint32_t lo, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(lo), "r"(0u), "r"(sel));
    return int(d);
}

// Scores of one row against the four bases as signed bytes, at the base's
// index (c >> 1) & 3 (A, C, T, G): match at the row's own base.
__device__ __forceinline__ uint32_t score_pool(uint32_t base, uint32_t mm4, uint32_t flip) {
    return acgt_base(base) ? mm4 ^ (flip << (8 * ((base >> 1) & 3u))) : mm4;
}

// DP of one layer against its rows (ranks 1..ndp; rank 0 = empty prefix
// row), by a team of NW warps. The columns are cut into strips of 32 * S,
// one per warp (rows longer than a pass take several); lane l owns S
// consecutive columns of its warp's strip. Each warp goes down the rows on
// its own, a few rows behind the warp to its left: the only thing it needs
// from there is each row's final score at the strips' edge, which the left
// warp leaves in a shared ring, publishing its progress every kGroupRows
// rows. A row is a chain of dependent steps, and its fixed work
// (control, in-row scan, stores) is as large as its cells' work: one warp
// over all columns spends the fewest instructions, several side by side
// finish a window sooner.
//
// Rows that other rows than the next one need (g.used) go to a shared-memory
// ring of the last R such rows, [unit][lane] and then the score left of each
// lane's segment (conflict-free, and no lane reads another's words); what has
// left the ring comes from global memory. On this chip a vote with a branch on
// it costs about 75 cycles, a warp reduction 60, a shuffle 33, so the row is
// kept nearly free of them. (Whole layers, cycles a row with one warp and with
// four: 615 and 540 for layers of 500 bases, 1500 and 690 for 1000; with every
// SM full of teams 835 and 830, 1880 and 1350.) What a row needs besides its
// scores is worked out 32 rows at a time, one row per lane: a score word, and a
// control word with the ring slots of up to 6 predecessors besides the row just
// computed, which is still in registers.
//
// Per cell: the elementwise maximum M over the predecessor rows, then
// T = max(M[j-1] + s - gap, M[j] + gap) (the substitution score comes from one
// byte permute of the row's four scores), then the running maximum along the
// row: maxima of groups of cells, a warp scan of the lanes' maxima, and one
// chain per group from what lies left of it. No decisions are kept: the walk
// visits a few cells of each row and decides there from the scores, which
// are stored anyway.
constexpr unsigned kCtlChain = 8, kCtlSlow = 7;  // control: count (7 = general way) | chain | 6 slot nibbles
template <int S, int NW, bool FAST, bool LEFT>
__device__ __noinline__ void dp_strip(const Graph& g, PoaShared& sh, int ndp_, const uint8_t* seq, int L, int mt,
                                      int mm, int gap, int lane, int w, int team, int pass) {
    static_assert(S % 2 == 0 && S >= 2 && S <= 24, "segment");
    constexpr unsigned kFull = 0xffffffffu;
    using Mem = WarpMem<NW>;
    constexpr int U = S % 4 == 0 ? 4 : 2;  // cells per ring unit
    constexpr int Q = S / U;
    constexpr int RB = S * 128 + 128;      // bytes per ring row
    constexpr int R = Mem::ring_bytes / RB < 15 ? Mem::ring_bytes / RB : 15;
    static_assert(R >= 2, "ring");
    constexpr int W = 32 * S;
    constexpr int HB = FAST ? 2 : 4;       // bytes per stored score
    // uniform registers, by way of warp votes and reductions
    const int ndp = __reduce_max_sync(kFull, ndp_);
    const int lc = row_cover(NW, L + 1);
    const int strip = pass * NW + w;
    const int tag0 = pass * (ndp + 1);
    const int c0 = strip * W;
    const int j0 = c0 + lane * S;
    uint8_t* const Hb = reinterpret_cast<uint8_t*>(g.H);
    const int4* const rowdesc = g.rowdesc;
    const int* const pred_idx = g.pred_idx;
    uint8_t* const mine = reinterpret_cast<uint8_t*>(g_poa_smem) + (team * NW + w) * Mem::bytes;
    uint8_t* const ring = mine + lane * (U * 4);              // the lane's first unit of row 0
    uint8_t* const ring_left = mine + S * 128 + lane * 4;
    uint32_t* const cblk = reinterpret_cast<uint32_t*>(mine + Mem::ctl);
    uint32_t* const pblk = reinterpret_cast<uint32_t*>(mine + Mem::pool);
    volatile int* const ein = reinterpret_cast<volatile int*>(mine + Mem::edge);
    // another warp takes this strip's edge, from the last lane
    const bool feeds = __any_sync(kFull, w + 1 < NW && c0 + W <= L);
    const bool waits = __any_sync(kFull, LEFT && w > 0);
    const bool feed_lane = feeds && lane == 31;
    const int dmt = mt - gap, dmm = mm - gap;
    const uint32_t mm4 = uint32_t(uint8_t(dmm)) * 0x01010101u;
    const uint32_t flip = uint32_t(uint8_t(dmt)) ^ uint32_t(uint8_t(dmm));
    // per cell: the permute selector of its base, or its character
    uint32_t sel[S];
#pragma unroll
    for (int k = 0; k < S; ++k) {
        const int j = j0 + k;
        const uint32_t c = (j >= 1 && j <= L) ? uint32_t(seq[j - 1]) : 0u;
        sel[k] = FAST ? ((c >> 1) & 3u) * 0x1111u + 0x8880u : c;
    }
    // row 0 (empty graph prefix) in global memory for the walk
#pragma unroll
    for (int k = 0; k < S; ++k) {
        if (FAST) {
            reinterpret_cast<int16_t*>(Hb)[j0 + k] = 0;
        } else {
            reinterpret_cast<int*>(Hb)[j0 + k] = 0;
        }
    }
    // score rows, at the lane's segment of the row being computed
    uint8_t* hrow = Hb + (size_t(lc) + j0) * HB;
    const size_t hstep = size_t(lc) * HB;
    int4 pre = lane < ndp ? rowdesc[lane] : make_int4(0, 0, 0, 0);
    // hv holds the previous row's final scores between iterations (row 0
    // first), and left that row's score left of the lane's segment
    int hv[S];
#pragma unroll
    for (int k = 0; k < S; ++k) hv[k] = 0;
    int left = j0 == 0 ? kNegInf : 0;
    int wofs = 0;             // ring offset of the next row to be kept
    unsigned kept = 0;        // rows kept before this block
    unsigned prev_used = 0;   // the previous block's used rows
    unsigned next_used = g.used[0];
    for (int i0 = 0; i0 < ndp; i0 += 32) {
        const unsigned used = next_used;
        __syncwarp();
        {
            // controls of rows i0 + 1 .. i0 + 32, one per lane. The k-th row
            // kept (from 0) is in slot k % R until R more have been kept;
            // rows of this block and the previous one are looked up.
            const int r = i0 + 1 + lane;
            const int np = desc_np(pre.w), packed = desc_listed(pre.w) ? 0 : np;
            uint32_t ctl = np == 0 || (packed != np && (pre.w & kPrev)) ? kCtlChain : 0, n = 0;
            bool slow = packed != np || (np == 0 && r > 1);
            const unsigned here = kept + __popc(used & ((1u << lane) - 1u));  // rows kept before r
            const unsigned kept1 = kept - __popc(prev_used);
#pragma unroll 1
            for (int q = 0; q < packed; ++q) {
                const int p = desc_packed(pre, q);
                if (p == r - 1) {
                    ctl |= kCtlChain;
                } else {
                    const unsigned bit = unsigned(p - 1) & 31u, below = (1u << bit) - 1u;
                    const unsigned k = p > i0 ? kept + __popc(used & below) : kept1 + __popc(prev_used & below);
                    slow |= p <= i0 - 32 || here - k > unsigned(R);
                    ctl |= (k % R) << (4 + 4 * n);
                    ++n;
                }
            }
            cblk[lane] = slow ? kCtlSlow | (r > 1 && np > 0 ? ctl & kCtlChain : 0u) : ctl | n;
            if (lane == 0) cblk[32] = 0u;  // read (as a ring slot too) after the block's last row
            pblk[lane] = FAST ? score_pool(desc_base(pre.w), mm4, flip) : desc_base(pre.w);
            if (LEFT && w == 0 && r <= ndp) {
                // the first strip of a later pass: the edge of the strip
                // to its left is in the score rows of the pass before
                ein[(r - 1) & (kEdgeRows - 1)] = h_at<FAST>(Hb, r, c0 - 1, lc);
            }
        }
        __syncwarp();
        const int nx = i0 + 32 + lane;
        pre = nx < ndp ? rowdesc[nx] : make_int4(0, 0, 0, 0);
        next_used = i0 + 32 < ndp ? g.used[(i0 >> 5) + 1] : 0u;
        const int cnt = min(32, ndp - i0);
        volatile int* const ein_b = ein + (i0 & (kEdgeRows - 1));
        // ring row at byte offset o; returns its score left of the segment
        auto ring_row = [&](int o, int (&dst)[S]) -> int {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                if constexpr (U == 4) {
                    const int4 v = *reinterpret_cast<const int4*>(ring + o + q * 512);
                    dst[4 * q] = v.x;
                    dst[4 * q + 1] = v.y;
                    dst[4 * q + 2] = v.z;
                    dst[4 * q + 3] = v.w;
                } else {
                    const int2 v = *reinterpret_cast<const int2*>(ring + o + q * 256);
                    dst[2 * q] = v.x;
                    dst[2 * q + 1] = v.y;
                }
            }
            return *reinterpret_cast<const int*>(ring_left + o);
        };
        unsigned cnext = cblk[0];
        // four-warp teams load the row's first predecessor in the ring a row
        // ahead (whatever that reads for a row without one is not used); wide
        // segments would hold too many registers over the row for it
        constexpr bool kAhead = NW > 1;
        int t[S], tleft = 0;
        if (kAhead) tleft = ring_row(((cnext >> 4) & 15u) * RB, t);
        uint32_t pnext = pblk[0];
        for (int b0 = 0; b0 < cnt; b0 += kGroupRows) {
        const int bend = min(b0 + kGroupRows, cnt);
        if (NW > 1) {
            // the left neighbour is past these rows; the right one is at
            // most the edge ring behind
            if (waits) {
                wait_rows(sh, sh.done[w - 1], tag0 + i0 + bend);
                __threadfence_block();
            }
            if (feeds) wait_rows(sh, sh.done[w + 1], tag0 + i0 + bend - kEdgeRows);
        }
#pragma unroll 1
        for (int b = b0; b < bend; ++b) {
            unsigned ctl = cnext;
            const uint32_t pool = pnext;
            // next row's
            cnext = cblk[b + 1];
            pnext = pblk[b + 1];
            int bx = kNegInf;  // final score of this row left of the strip, at lane 0
            if (LEFT) {
                const int e = ein_b[b];
                bx = lane == 0 ? e : kNegInf;
            }
            if ((ctl & 15u) != kCtlChain) {
                auto merge = [&](int lft) {
#pragma unroll
                    for (int k = 0; k < S; ++k) hv[k] = max(hv[k], t[k]);
                    left = max(left, lft);
                };
                if (!kAhead) tleft = ring_row(((ctl >> 4) & 15u) * RB, t);
                if (__builtin_expect((ctl & 15u) == (kCtlChain | 1u), 1)) {
                    merge(tleft);
                } else
                if (__builtin_expect((ctl & 7u) != kCtlSlow, 1)) {
                    if (!(ctl & kCtlChain)) {
                        // the row just computed is no predecessor
#pragma unroll
                        for (int k = 0; k < S; ++k) hv[k] = t[k];
                        left = tleft;
                    } else {
                        merge(tleft);
                    }
#pragma unroll 1
                    for (unsigned n = ctl & 7u; n > 1; --n) {
                        ctl >>= 4;
                        merge(ring_row(((ctl >> 4) & 15u) * RB, t));
                    }
                } else {
                    // general row: any number of predecessors at any distance,
                    // from the ring or from global memory
                    const int i = i0 + 1 + b;
                    const int4 d = rowdesc[i - 1];
                    const int np = desc_np(d.w);
                    const bool chain = (ctl & kCtlChain) != 0;  // in hv already
                    const unsigned here = kept + __popc(used & ((1u << b) - 1u));
                    const unsigned kept1 = kept - __popc(prev_used);
                    if (!chain) {
#pragma unroll
                        for (int k = 0; k < S; ++k) hv[k] = INT_MIN;
                        left = INT_MIN;
                    }
#pragma unroll 1
                    for (int p = 0; p < max(np, 1); ++p) {
                        const int r = desc_pred(pred_idx, d, p);
                        int lft;
                        if (chain && r == i - 1) continue;
                        const unsigned below = (1u << (unsigned(r - 1) & 31u)) - 1u;
                        const unsigned k = r > i0 ? kept + __popc(used & below) : kept1 + __popc(prev_used & below);
                        if (r > 0 && r > i0 - 32 && here - k <= unsigned(R)) {
                            lft = ring_row((k % R) * RB, t);
                        } else if (r == 0) {
                            lft = j0 == 0 ? kNegInf : 0;
#pragma unroll
                            for (int k = 0; k < S; ++k) t[k] = 0;
                        } else {
                            const uint8_t* const src = Hb + (size_t(r) * lc + j0) * HB;
                            if constexpr (FAST) {
                                uint32_t v[S / 2];
                                if constexpr (S % 8 == 0) {
#pragma unroll
                                    for (int q = 0; q < S / 8; ++q)
                                        *reinterpret_cast<uint4*>(v + 4 * q) = reinterpret_cast<const uint4*>(src)[q];
                                } else if constexpr (S % 4 == 0) {
#pragma unroll
                                    for (int q = 0; q < S / 4; ++q)
                                        *reinterpret_cast<uint2*>(v + 2 * q) = reinterpret_cast<const uint2*>(src)[q];
                                } else {
#pragma unroll
                                    for (int q = 0; q < S / 2; ++q) v[q] = reinterpret_cast<const uint32_t*>(src)[q];
                                }
#pragma unroll
                                for (int q = 0; q < S / 2; ++q) {
                                    t[2 * q] = unpack_lo(v[q]);
                                    t[2 * q + 1] = unpack_hi(v[q]);
                                }
                            } else {
#pragma unroll
                                for (int q = 0; q < S / 2; ++q) {
                                    const int2 v2 = reinterpret_cast<const int2*>(src)[q];
                                    t[2 * q] = v2.x;
                                    t[2 * q + 1] = v2.y;
                                }
                            }
                            lft = __shfl_up_sync(kFull, t[S - 1], 1);
                            int e = kNegInf;
                            if (LEFT) e = h_at<FAST>(Hb, r, c0 - 1, lc);
                            if (lane == 0) lft = e;
                        }
                        merge(lft);
                    }
                }
            }
            // T = max(M[j-1] + s - gap, M[j] + gap), in place from the right
#pragma unroll
            for (int k = S - 1; k >= 0; --k) {
                const int s = FAST ? prmt_score(pool, sel[k]) : (sel[k] == pool ? dmt : dmm);
                const int dg = (k == 0 ? left : hv[k - 1]) + s;
                hv[k] = __viaddmax_s32(hv[k], gap, dg);
            }
            // running maximum along the row: C groups of K cells
            constexpr int K = S % 4 == 0 ? 4 : S % 3 == 0 ? 3 : 2;
            constexpr int C = S / K;
            int tot[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                tot[c] = K == 2 ? max(hv[c * K], hv[c * K + 1])
                                : __vimax3_s32(hv[c * K], hv[c * K + 1], hv[c * K + 2]);
                if (K == 4) tot[c] = max(tot[c], hv[c * K + 3]);
                if (c > 0) tot[c] = max(tot[c], tot[c - 1]);
            }
            const int tnext = ((cnext >> 4) & 15u) * RB;
            // prefix maximum over the lanes by fours: three shuffles of one
            // value cost little more than one (a lane that a shuffle does not
            // reach gets its own value back)
            int x = LEFT ? max(tot[C - 1], bx) : tot[C - 1];
            {
                const int s1 = __shfl_up_sync(kFull, x, 1), s2 = __shfl_up_sync(kFull, x, 2);
                const int s3 = __shfl_up_sync(kFull, x, 3);
                x = max(__vimax3_s32(x, s1, s2), s3);
                const int t1 = __shfl_up_sync(kFull, x, 4), t2 = __shfl_up_sync(kFull, x, 8);
                const int t3 = __shfl_up_sync(kFull, x, 12);
                x = max(__vimax3_s32(x, t1, t2), t3);
                x = max(x, __shfl_up_sync(kFull, x, 16));
            }
            if (kAhead) tleft = ring_row(tnext, t);
            left = __shfl_up_sync(kFull, x, 1);  // final value left of the segment
            if (lane == 0) left = bx;
#pragma unroll
            for (int c = 0; c < C; ++c) hv[c * K] = max(hv[c * K], c == 0 ? left : max(left, tot[c - 1]));
#pragma unroll
            for (int k = 1; k < K; ++k)
#pragma unroll
                for (int c = 0; c < C; ++c) hv[c * K + k] = max(hv[c * K + k], hv[c * K + k - 1]);
            if (feed_lane)
                reinterpret_cast<volatile int*>(mine + Mem::bytes + Mem::edge)[(i0 + b) & (kEdgeRows - 1)] = hv[S - 1];
            if ((used >> b) & 1u) {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    if constexpr (U == 4) {
                        *reinterpret_cast<int4*>(ring + wofs + q * 512) =
                            make_int4(hv[4 * q], hv[4 * q + 1], hv[4 * q + 2], hv[4 * q + 3]);
                    } else {
                        *reinterpret_cast<int2*>(ring + wofs + q * 256) = make_int2(hv[2 * q], hv[2 * q + 1]);
                    }
                }
                *reinterpret_cast<int*>(ring_left + wofs) = left;
                wofs = wofs == (R - 1) * RB ? 0 : wofs + RB;
            }
            // streamed: keep the graph arrays in L2
            if constexpr (FAST) {
                uint32_t pk[S / 2];
#pragma unroll
                for (int q = 0; q < S / 2; ++q) pk[q] = pack_s16(hv[2 * q], hv[2 * q + 1]);
                if constexpr (S % 8 == 0) {
#pragma unroll
                    for (int q = 0; q < S / 8; ++q)
                        __stcs(reinterpret_cast<uint4*>(hrow) + q,
                               make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]));
                } else if constexpr (S % 4 == 0) {
#pragma unroll
                    for (int q = 0; q < S / 4; ++q)
                        __stcs(reinterpret_cast<uint2*>(hrow) + q, make_uint2(pk[2 * q], pk[2 * q + 1]));
                } else {
#pragma unroll
                    for (int q = 0; q < S / 2; ++q) __stcs(reinterpret_cast<uint32_t*>(hrow) + q, pk[q]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < S / 2; ++q)
                    __stcs(reinterpret_cast<int2*>(hrow) + q, make_int2(hv[2 * q], hv[2 * q + 1]));
            }
            hrow += hstep;
        }
            if (NW > 1) {
                // lane 31 wrote the strip's edge; its stores come before the count
                __threadfence_block();
                if (lane == 31) sh.done[w] = tag0 + i0 + bend;
            }
        }
        kept += __popc(used);
        prev_used = used;
    }
    __syncwarp();
}

// One layer's DP, all passes.
template <int S, int NW>
__device__ __forceinline__ void dp_layer(const Graph& g, PoaShared& sh, int ndp, const uint8_t* seq, int L, int mt,
                                         int mm, int gap, int lane, int w, int team, bool fast) {
    constexpr int W = 32 * S;
    const int nstrips = (L + W) / W;
    if (lane == 0) sh.done[w] = 0;
    for (int pass = 0; pass * NW < nstrips; ++pass) {
        team_sync<NW>(team);
        const int strip = pass * NW + w;
        if (strip >= nstrips) continue;
        if (fast) {
            if (strip == 0) {
                dp_strip<S, NW, true, false>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, pass);
            } else {
                dp_strip<S, NW, true, true>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, pass);
            }
        } else {
            if (strip == 0) {
                dp_strip<S, NW, false, false>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, pass);
            } else {
                dp_strip<S, NW, false, true>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, pass);
            }
        }
    }
}

template <int NW>
__device__ void dp_dispatch(const Graph& g, PoaShared& sh, int ndp, const uint8_t* seq, int L, int mt, int mm,
                            int gap, int lane, int w, int team, bool fast) {
    const int s = seg_cells(NW, L + 1);
    if constexpr (NW == 4) {
        switch (s) {
            case 2: return dp_layer<2, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
            case 4: return dp_layer<4, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
            case 6: return dp_layer<6, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
            default: return dp_layer<8, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
        }
    } else {
        switch (s) {
            case 8: return dp_layer<8, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
            case 16: return dp_layer<16, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
            case 20: return dp_layer<20, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
            default: return dp_layer<24, NW>(g, sh, ndp, seq, L, mt, mm, gap, lane, w, team, fast);
        }
    }
}

// The walk back from (iend, L) over the stored scores, by one warp. At a
// cell with slanted score h it takes spoa's first way to h: the diagonal through the
// predecessors in order, then the vertical through them, then left. The walk
// is a chain of dependent steps through nearby rows and columns, so the warp
// stages a tile of score rows, descriptors and node ids in shared memory and
// one lane walks through it, loading all candidates of a step at once and
// choosing among them without branches (votes and shuffles between lanes
// would cost more than the whole step). A predecessor above the tile is read
// from global memory; a step that leaves the tile ends the lane's run and
// the warp stages the next one, all its copies in flight at once. Writes the
// row of every sequence position (0 for an inserted base) to g.path; a
// vertical step consumes no position and adds nothing to the graph. Returns
// false on a broken walk. (The walk takes about 335
// cycles a base with its tiles, 530 where every SM is full; with one load after
// another a tile took 16 k cycles, now 2 k.)
constexpr int kTileRows = 96;
constexpr int kTilePitch = 128;  // bytes per row: 64 int16 or 32 int32 columns
constexpr int kTileBytes = 16 + kTileRows * kTilePitch;  // the walk may look one column left of the first
constexpr int kTileSmem = kTileBytes + kTileRows * 32 + 64;
static_assert(kTileSmem <= 4 * WarpMem<4>::bytes && kTileSmem <= WarpMem<1>::bytes, "the tile fits every team's memory");
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src)
                 : "memory");
}
template <bool FAST>
__device__ __noinline__ bool traceback_warp(const Graph& g, const uint8_t* seq, int L, int iend, int hend, int mt,
                                            int mm, int gap, int lane, int smem_off, int lc) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int HB = FAST ? 2 : 4;              // bytes per score
    constexpr int kCols = kTilePitch / HB;       // tile columns
    constexpr int kUnit = 16 / HB;               // columns per 16-byte chunk
    constexpr int kChunks = kTilePitch / 16;
    uint8_t* const smem = reinterpret_cast<uint8_t*>(g_poa_smem) + smem_off;
    uint8_t* const tile = smem + 16;
    // per tile row: byte offsets of the predecessors' tile rows (16-bit
    // halves of x, y, z) | base, predecessors to test (3, 6, or 0: some lie
    // outside the tile or in pred_idx) << 8
    int4* const w_desc = reinterpret_cast<int4*>(smem + kTileBytes);
    int4* const w_raw = w_desc + kTileRows;
    uint8_t* const w_seq = reinterpret_cast<uint8_t*>(w_raw + kTileRows);
    const uint8_t* const Hb = reinterpret_cast<const uint8_t*>(g.H);
    const int4* const rowdesc = g.rowdesc;
    const int* const pred_idx = g.pred_idx;
    int* const path = g.path;
    int i = iend, j = L, h = hend;
    if (iend == INT_MAX || iend < 1) return false;
    auto score = [&](const uint8_t* p) -> int {
        return FAST ? int(*reinterpret_cast<const int16_t*>(p)) : *reinterpret_cast<const int*>(p);
    };
    const int dmt = mt - gap, dmm = mm - gap;
    bool ok = true;
    while (i > 0 && ok) {
        // rows (i - kTileRows, i], columns up to j
        const int wlo = max(0, i - (kTileRows - 1));
        const int clo = max(0, (j / kUnit + 1) * kUnit - kCols);
        const int rows = i - wlo + 1;
        __syncwarp();
        // rows past i and columns past the stride repeat others and are not read
#pragma unroll
        for (int u = 0; u < kTileRows * kChunks / 32; ++u) {
            const int q = u * 32 + lane;
            const int tr = min(q / kChunks, rows - 1), tc = min(clo + q % kChunks * kUnit, lc - kUnit);
            copy16_async(tile + q * 16, Hb + (size_t(wlo + tr) * lc + tc) * HB);
        }
        int4 dd[kTileRows / 32];
#pragma unroll
        for (int u = 0; u < kTileRows / 32; ++u)
            dd[u] = rowdesc[min(max(wlo + u * 32 + lane, 1), i) - 1];
#pragma unroll
        for (int u = 0; u < kTileRows / 32; ++u) {
            const int t = u * 32 + lane;
            const int4 d = dd[u];
            const int np = desc_np(d.w);
            // absent predecessors repeat the first
            unsigned o[kPacked];
            int low = INT_MAX;
#pragma unroll
            for (int q = 0; q < kPacked; ++q) {
                const int pr = desc_packed(d, q < np ? q : 0);
                low = min(low, pr);
                o[q] = unsigned(pr - wlo) * kTilePitch;
            }
            const int n = desc_listed(d.w) || low < wlo ? 0 : np <= 3 ? 3 : 6;
            w_raw[t] = d;
            w_desc[t] = make_int4(int(o[0] | (o[1] << 16)), int(o[2] | (o[3] << 16)), int(o[4] | (o[5] << 16)),
                                  int(desc_base(d.w) | unsigned(n) << 8));
        }
        for (int c = lane; c < kCols; c += 32) w_seq[c] = (clo + c >= 1 && clo + c <= L) ? seq[clo + c - 1] : 0;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            int oi = (i - wlo) * kTilePitch, cj = j - clo;  // the cell in the tile
            const int cmin = clo > 0 ? 1 : 0;               // the walk needs column cj - 1 unless it is before the first
            const int omin = wlo == 0 ? kTilePitch : 0;     // rank 0 ends the walk
            do {
                const int4 d = w_desc[oi / kTilePitch];
                const uint8_t* const tj = tile + cj * HB;
                const int s = uint32_t(w_seq[cj]) == (uint32_t(d.w) & 0xFFu) ? dmt : dmm;
                const int hd = cj > 0 ? h - s : INT_MIN, hu = h - gap;
                int no = oi, nh = score(tj + oi - HB);  // left
                int row = 0, step = 1;
                // the first diagonal, else the first vertical, of K predecessors
                auto choose = [&](const auto& o) {
                    constexpr int K = int(sizeof(o) / sizeof(o[0]));
                    int od = -1, ou = -1;
#pragma unroll
                    for (int q = K - 1; q >= 0; --q) {
                        if (score(tj + o[q] - HB) == hd) od = o[q];
                        if (score(tj + o[q]) == hu) ou = o[q];
                    }
                    if (ou >= 0) {
                        no = ou;
                        nh = hu;
                        step = 0;
                    }
                    if (od >= 0) {
                        no = od;
                        nh = hd;
                        step = 1;
                        row = 1;
                    }
                };
                const int x0 = d.x & 0xFFFF, x1 = int(unsigned(d.x) >> 16), x2 = d.y & 0xFFFF;
                const unsigned n = (unsigned(d.w) >> 8) & 7u;
                if (n == 3) {
                    const int o[3] = {x0, x1, x2};
                    choose(o);
                } else if (n == 6) {
                    const int o[6] = {x0, x1, x2, int(unsigned(d.y) >> 16), d.z & 0xFFFF, int(unsigned(d.z) >> 16)};
                    choose(o);
                } else {
                    // long list, or a predecessor above the tile: the first
                    // diagonal, else the first vertical
                    const int4 e = w_raw[oi / kTilePitch];
                    const int np = desc_np(e.w);
                    int vr = -1, dr = -1;
                    for (int p = 0; p < max(np, 1) && dr < 0; ++p) {
                        const int r = desc_pred(pred_idx, e, p);
                        const uint8_t* const pr = r >= wlo ? tj + (r - wlo) * kTilePitch
                                                           : Hb + (size_t(r) * lc + clo + cj) * HB;  // generic address
                        if (cj > 0 && score(pr - HB) == hd) dr = r;
                        if (vr < 0 && score(pr) == hu) vr = r;
                    }
                    if (dr >= 0 || vr >= 0) {
                        no = ((dr >= 0 ? dr : vr) - wlo) * kTilePitch;
                        nh = dr >= 0 ? hd : hu;
                        row = dr >= 0 ? 1 : 0;
                        step = row;
                    }
                }
                if (step) {
                    if (cj == 0) {
                        ok = false;
                        break;
                    }
                    --cj;
                    path[clo + cj] = row ? wlo + oi / kTilePitch : 0;
                }
                oi = no;
                h = nh;
            } while (oi >= omin && cj >= cmin);
            i = wlo + (oi >= 0 ? oi / kTilePitch : -((-oi) / kTilePitch));
            j = clo + cj;
        }
        i = __shfl_sync(kFull, i, 0);
        j = __shfl_sync(kFull, j, 0);
        h = __shfl_sync(kFull, h, 0);
        ok = __shfl_sync(kFull, ok ? 1 : 0, 0) != 0;
    }
    if (ok)
        for (int k = lane; k < j; k += 32) path[k] = 0;
    __syncwarp();
    return ok;
}

// ---------------- one window (one team) ----------------

// Every thread of the team returns together.
template <int NW>
__device__ void poa_window(const PoaArgs& a, Graph& g, PoaShared& sh, uint32_t wi, int lane, int w, int team) {
    constexpr int NT = 32 * NW;
    const int tid = 32 * w + lane;
    constexpr int kTeamBytes = NW * WarpMem<NW>::bytes;
    uint8_t* const smem = reinterpret_cast<uint8_t*>(g_poa_smem) + team * kTeamBytes;
    const PoaWinDev W = a.wins[wi];
    const uint8_t* bb = a.in + W.bb_off;
    const uint8_t* bq = W.bq_off == kNoQual ? nullptr : a.in + W.bq_off;
    uint8_t* outp = reinterpret_cast<uint8_t*>(a.out) + W.out_off;
    const int B = int(W.bb_len);
    if (W.n_layers < 2) {
        for (int i = tid; i < B; i += NT) outp[i] = bb[i];
        if (tid == 0) {
            a.out_len[wi] = uint32_t(B);
            a.flags[wi] = 0;
        }
        return;
    }
    if (B > g.ncap) {
        if (tid == 0) {
            a.flags[wi] = kOverflow;
            a.out_len[wi] = 0;
        }
        return;
    }
    // backbone: chain of B nodes, edge weights from quality (0 with the dummy)
    for (int i = tid; i < B; i += NT) {
        g.code[i] = bb[i];
        g.cov[i] = B >= 2 ? 1u : 0u;
        g.in_cnt[i] = i > 0 ? 1 : 0;
        g.out_cnt[i] = i + 1 < B ? 1 : 0;
        g.al_cnt[i] = 0;
        const int wt = i > 0 && bq ? (int(bq[i - 1]) - 33) + (int(bq[i]) - 33) : 0;
        g.in_src[2 * size_t(i)] = make_int4(i - 1, 0, 0, 0);
        g.in_w[2 * size_t(i)] = make_int4(wt, 0, 0, 0);
        g.ord[i] = i;
        g.rank[i] = i;
    }
    if (tid == 0) {
        sh.nnodes = B;
        sh.nedges = 0;
        sh.naligned = 0;
        sh.nseq = 1;
        sh.fail = 0;
        sh.scratch_bytes = kTeamBytes;
        sh.wait_polls = a.wait_polls;
    }
    team_sync<NW>(team);
    unsigned long long cells = 0, edge_cells = 0;

    for (uint32_t li = 0; li < W.n_layers; ++li) {
        const PoaLayerDev Lr = a.layers[W.layer_base + li];
        const uint8_t* seq = a.in + Lr.seq_off;
        const uint8_t* qual = Lr.qual_off == kNoQual ? nullptr : a.in + Lr.qual_off;
        const int L = int(Lr.len);
        const bool full = Lr.begin < W.offset && Lr.end > uint32_t(B) - W.offset;
        const int begin = full ? 0 : int(Lr.begin);
        if (row_cover(NW, L + 1) > g.lcap) {
            if (tid == 0) sh.fail = kOverflow;
            break;
        }
        // DP rows: the incremental order, restricted to the subgraph for a
        // partial layer (any topological order gives the same DP values)
        build_rows<NW>(g, sh, g.ord, sh.nnodes, false, tid, team, smem);
        int ndp = sh.nnodes;
        const int* order = g.ord;
        if (!full) {
            mark_subgraph<NW>(g, sh, begin, int(Lr.end), lane, w, team, smem);
            ndp = sh.ndp;
            if (ndp == 0) {  // failed or overflowed
                if (tid == 0 && sh.fail == 0) sh.fail = kFailed;
                break;
            }
            order = g.dporder;
            build_rows<NW>(g, sh, order, ndp, true, tid, team, smem);
        }
        bool fast = fast_scores(a.match, a.mismatch, a.gap, ndp, L);
        for (int k = lane; k < L; k += 32) fast = fast && acgt_base(seq[k]);
        fast = __all_sync(0xffffffffu, fast);
        dp_dispatch<NW>(g, sh, ndp, seq, L, a.match, a.mismatch, a.gap, lane, w, team, fast);
        team_sync<NW>(team);
        if (w == 0 && (NW == 1 || !sh.fail)) {
            cells += (unsigned long long)ndp * (unsigned long long)L;
            edge_cells += (unsigned long long)(ndp + sh.preds) * (unsigned long long)L;
            const int lc = row_cover(NW, L + 1);
            const int iend = fast ? end_row<true>(g, sh, order, L, lc, !full, begin, B, lane, smem)
                                  : end_row<false>(g, sh, order, L, lc, !full, begin, B, lane, smem);
            if (!sh.fail) {
                const bool ok = fast ? traceback_warp<true>(g, seq, L, iend, sh.end_value, a.match, a.mismatch, a.gap,
                                                            lane, team * kTeamBytes, lc)
                                     : traceback_warp<false>(g, seq, L, iend, sh.end_value, a.match, a.mismatch, a.gap,
                                                             lane, team * kTeamBytes, lc);
                if (!ok && lane == 0) sh.fail = kFailed;
            }
        }
        team_sync<NW>(team);
        if (sh.fail) break;
        add_layer<NW>(g, sh, order, seq, qual, L, lane, w, team, smem);
        if (sh.fail) break;
        order_insert<NW>(g, sh, lane, w, team, smem);
    }
    team_sync<NW>(team);
    if (w != 0) return;
    if (lane == 0 && cells) {
        atomicAdd(a.cells, cells);
        atomicAdd(a.cells + 1, edge_cells);
    }
    const int len = sh.fail ? 0 : heaviest_bundle_warp(g, sh, lane, smem);
    if (sh.fail || len < 0) {
        if (lane == 0) {
            a.flags[wi] = uint8_t(sh.fail ? sh.fail : kFailed);
            a.out_len[wi] = 0;
        }
        __syncwarp();
        return;
    }
    // the path is in g.cons from its end
    uint8_t flags = kPolished;
    int b = 0, e = len - 1;
    if (W.tgs && a.trim) {
        const uint32_t avg = W.n_layers / 2;
        auto covered = [&](int k) {
            if (k < 0 || k >= len) return false;
            const int v = g.cons[len - 1 - k];
            uint32_t c = g.cov[v];
            for_aligned(g, v, [&](int y) {
                c += g.cov[y];
                return true;
            });
            return c >= avg;
        };
        b = len;
        e = -1;
        for (int c0 = 0; c0 < len && b == len; c0 += 32) {
            const unsigned m = __ballot_sync(0xffffffffu, covered(c0 + lane));
            if (m) b = c0 + __ffs(m) - 1;
        }
        for (int c0 = len - 1; c0 >= 0 && e < 0; c0 -= 32) {
            const unsigned m = __ballot_sync(0xffffffffu, covered(c0 - lane));
            if (m) e = c0 - (__ffs(m) - 1);
        }
        if (b >= e) {
            flags |= kChimeric;
            b = 0;
            e = len - 1;
        }
    }
    const int outl = e - b + 1;
    if (uint32_t(outl) > W.out_cap) {
        if (lane == 0) {
            a.flags[wi] = kOverflow;
            a.out_len[wi] = 0;
        }
    } else {
        for (int k = lane; k < outl; k += 32) outp[k] = g.code[g.cons[len - 1 - (b + k)]];
        if (lane == 0) {
            a.flags[wi] = flags;
            a.out_len[wi] = uint32_t(outl);
        }
    }
    __syncwarp();
}

// Warps of a full CTA (teams of NW): three CTAs fill an SM's registers and
// shared memory, with 12 one-warp teams or 24 warps of four-warp teams.
__host__ __device__ constexpr int cta_warps(int nw) { return nw == 1 ? 4 : 8; }
__host__ __device__ constexpr int warp_smem(int nw) { return nw == 1 ? WarpMem<1>::bytes : WarpMem<4>::bytes; }
constexpr int kCtasPerSm = 3;

template <int NW>
__global__ void __launch_bounds__(32 * cta_warps(NW), kCtasPerSm) poa_kernel(PoaArgs a) {
    __shared__ PoaShared sh_all[cta_warps(NW) / NW];
    // each team's view of its scratch slot lives in shared memory so the
    // ~35 array pointers are not held in registers across the DP
    __shared__ Graph g_all[cta_warps(NW) / NW];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int team = wid / NW, w = wid % NW;
    PoaShared& sh = sh_all[team];
    const uint32_t slot = blockIdx.x * (blockDim.x / (32 * NW)) + team;
    if (w == 0 && lane == 0) g_all[team] = make_graph(a, slot);
    Graph& g = g_all[team];
    // with a cap the CTA retires after that many windows per team, so other
    // streams' kernels get SMs between launches (the host launches enough)
    for (uint32_t done = 0; a.per_warp_cap == 0 || done < a.per_warp_cap; ++done) {
        if (w == 0 && lane == 0) sh.next = atomicAdd(&a.counters[0], 1u);
        team_sync<NW>(team);
        const uint32_t k = sh.next;
        if (k >= a.nwin) break;
        poa_window<NW>(a, g, sh, a.order[k], lane, w, team);
        team_sync<NW>(team);
    }
}

// Plain comparison form: one window per one-team block, block b takes window
// order[b] with scratch slot b, one launch per batch, no work queue. Same
// per-window code as poa_kernel, so results are identical.
constexpr int kPlainWarps = 1;
__global__ void __launch_bounds__(32 * cta_warps(kPlainWarps), kCtasPerSm) poa_plain_kernel(PoaArgs a) {
    __shared__ PoaShared sh;
    __shared__ Graph g;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (blockIdx.x >= a.nwin) return;
    if (threadIdx.x == 0) g = make_graph(a, blockIdx.x);
    team_sync<kPlainWarps>(0);
    poa_window<kPlainWarps>(a, g, sh, a.order[blockIdx.x], lane, w, 0);
}

// ---------------- shared queue (serving) ----------------

// The consensus service's kernel arguments: scoring, capacities and scratch
// slots, the batch records, and the queue.
struct PoaSvcArgs {
    PoaArgs base;
    const PoaJobDev* jobs;
    SvcQueueDev q;
};

// Persistent consensus over the shared queue: each team owns one scratch
// slot and takes windows of any job until the queue stays empty. Sized for
// at most kSvcCtasPerSm resident CTAs per SM, so that the rest of each SM
// stays free for the alignment and layer kernels of newly admitted jobs. Held
// to 160 registers: two of its CTAs take 10240 of an SM sub-partition's 16384,
// one of the alignment service 3072, which leaves the 3072 of a warp of
// nw_level_kernel. With 168 a job whose spans exceed the alignment service's
// scratch could not run its own levels until a service closed for lack of
// work. (Four jobs at once 91 ms either way; taking the registers from the
// alignment service instead, 80 or 88 for 96, 93 ms.)
constexpr int kSvcCtasPerSm = 3;
constexpr int kSvcTeamWarps = 1;
constexpr int kSvcWarps = cta_warps(kSvcTeamWarps);
__global__ void __maxnreg__(160) poa_service_kernel(PoaSvcArgs s) {
    constexpr int NW = kSvcTeamWarps, T = kSvcWarps / NW;
    __shared__ PoaShared sh_all[T];
    __shared__ Graph g_all[T];
    __shared__ PoaArgs a_all[T];
    __shared__ unsigned long long item_all[T];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int team = wid / NW, w = wid % NW;
    PoaShared& sh = sh_all[team];
    const uint32_t slot = blockIdx.x * T + team;
    if (w == 0 && lane == 0) g_all[team] = make_graph(s.base, slot);
    for (;;) {
        uint32_t total = 0, gen = 0;
        if (w == 0 && lane == 0) {
            const unsigned long long it = svc_claim(s.q, slot);
            item_all[team] = it;
            if (it != ~0ull) {
                // the record is rewritten for every batch that reuses the slot:
                // read it past L1
                const volatile PoaJobDev& J = s.jobs[uint32_t(it >> 32)];
                PoaArgs a = s.base;
                a.in = const_cast<const uint8_t*>(J.in);
                a.wins = const_cast<const PoaWinDev*>(J.wins);
                a.layers = const_cast<const PoaLayerDev*>(J.layers);
                a.out = const_cast<char*>(J.out);
                a.out_len = const_cast<uint32_t*>(J.out_len);
                a.flags = const_cast<uint8_t*>(J.flags);
                a.trim = J.trim;
                a.cells = const_cast<unsigned long long*>(J.cells);
                total = J.head.total;
                gen = J.head.generation;
                a.nwin = total;
                a_all[team] = a;
            }
        }
        team_sync<NW>(team);
        const unsigned long long it = item_all[team];
        if (it == ~0ull) break;
        poa_window<NW>(a_all[team], g_all[team], sh, uint32_t(it), lane, w, team);
        __threadfence();
        team_sync<NW>(team);
        if (w == 0 && lane == 0) svc_item_done(s.q, uint32_t(it >> 32), total, gen);
    }
}

}  // namespace

// Row stride that holds rows of wc columns in every team form.
static int max_cover(int wc) { return std::max(row_cover(1, wc), row_cover(4, wc)); }

size_t PoaEngine::slot_bytes_for(uint32_t max_layer_length) {
    const int ncap = 4096;
    return walk_layout(ncap, 2 * ncap, ncap, max_cover(int(max_layer_length) + 1), [](int, size_t) {});
}

PoaEngine::PoaEngine(const DeviceInfo& dev, cudaStream_t stream, int8_t m, int8_t x, int8_t g)
    : dev_(dev), stream_(stream), match_(m), mismatch_(x), gap_(g) {
    check_cuda(cudaEventCreate(&ev0_), "cudaEventCreate");
    check_cuda(cudaEventCreate(&ev1_), "cudaEventCreate");
    check_cuda(cudaEventCreate(&ev2_), "cudaEventCreate");
    check_cuda(cudaEventCreate(&ev3_), "cudaEventCreate");
    prefer_max_shared(reinterpret_cast<const void*>(poa_kernel<1>));
    prefer_max_shared(reinterpret_cast<const void*>(poa_kernel<4>));
    prefer_max_shared(reinterpret_cast<const void*>(poa_plain_kernel));
}

PoaEngine::~PoaEngine() {
    cudaEventDestroy(ev0_);
    cudaEventDestroy(ev1_);
    cudaEventDestroy(ev2_);
    cudaEventDestroy(ev3_);
}

// Phred+33 bytes '!'..'~': the window graph weights are quality - 33 in
// 0..93 (spoa's uint32 weights of other bytes are not modelled).
static bool phred_bytes(const char* q, uint32_t n) {
    uint8_t bad = 0;
    for (uint32_t k = 0; k < n; ++k) bad |= uint8_t(uint8_t(q[k] - 33) > 93);
    return bad == 0;
}

void PoaEngine::stage(const rb_window* wins, size_t n, int trim) {
    if (n > 0 && !wins) throw Error{RB_ERR_ARG, "rb_poa: windows is NULL"};
    forget();
    trim_ = trim;
    // sizes
    uint64_t in_bytes = 0, nlayers = 0, out_cap = 0;
    max_len_ = 0;
    uint32_t max_nodes = 0;
    for (size_t i = 0; i < n; ++i) {
        const rb_window& w = wins[i];
        if (!w.backbone || w.backbone_length == 0 || w.backbone_length > 65535)
            throw Error{RB_ERR_ARG, "rb_poa: backbone empty, NULL or longer than 65535"};
        if (w.n_layers > 65535) throw Error{RB_ERR_ARG, "rb_poa: more than 65535 layers"};
        if (w.n_layers && (!w.layers || !w.layer_lengths || !w.begins || !w.ends))
            throw Error{RB_ERR_ARG, "rb_poa: NULL layer arrays"};
        in_bytes += 2 * ((w.backbone_length + 15) & ~15u);
        uint64_t est = w.backbone_length;
        for (uint32_t j = 0; j < w.n_layers; ++j) {
            const uint32_t l = w.layer_lengths[j];
            if (l == 0 || l > 65535 || !w.layers[j])
                throw Error{RB_ERR_ARG, "rb_poa: empty, NULL or over-long layer"};
            // racon's layers end at a matched backbone base (end <= length - 1,
            // src/polisher.cpp:450-453); the subgraph of a partial layer is
            // rooted at backbone node `end`, so it must exist.
            if (w.begins[j] >= w.ends[j] || w.ends[j] >= w.backbone_length)
                throw Error{RB_ERR_ARG, "rb_poa: layer begin and end positions are invalid"};
            in_bytes += 2 * ((l + 15) & ~15u);
            max_len_ = std::max(max_len_, l);
            est += l;
        }
        nlayers += w.n_layers;
        out_cap += 3ull * w.backbone_length + 1024;
        max_nodes = uint32_t(std::max<uint64_t>(max_nodes, std::min<uint64_t>(est, 1u << 20)));
    }
    in_bytes_ = in_bytes;
    out_cap_ = out_cap;
    max_nodes_cap_ = max_nodes;
    h_in_.reserve(std::max<uint64_t>(in_bytes, 16));
    h_desc_.reserve(std::max<size_t>(n, 1) * sizeof(PoaWinDev));
    h_layers_.reserve(std::max<uint64_t>(nlayers, 1) * sizeof(PoaLayerDev));
    h_order_.reserve(std::max<size_t>(n, 1) * sizeof(uint32_t));
    uint8_t* in = h_in_.as<uint8_t>();
    PoaWinDev* wd = h_desc_.as<PoaWinDev>();
    PoaLayerDev* ld = h_layers_.as<PoaLayerDev>();
    uint64_t off = 0, lbase = 0, oo = 0;
    labels_.resize(n);
    std::vector<uint32_t> rank;
    for (size_t i = 0; i < n; ++i) {
        const rb_window& w = wins[i];
        labels_[i] = {w.id, w.rank};
        PoaWinDev& d = wd[i];
        d.bb_off = off;
        memcpy(in + off, w.backbone, w.backbone_length);
        off += (w.backbone_length + 15) & ~15u;
        if (w.backbone_quality) {
            if (!phred_bytes(w.backbone_quality, w.backbone_length))
                throw Error{RB_ERR_ARG, "rb_poa: quality values outside '!'..'~' (Phred+33 0..93)"};
            d.bq_off = off;
            memcpy(in + off, w.backbone_quality, w.backbone_length);
            off += (w.backbone_length + 15) & ~15u;
        } else {
            d.bq_off = kNoQual;
        }
        d.bb_len = w.backbone_length;
        d.n_layers = w.n_layers;
        d.layer_base = lbase;
        d.out_off = oo;
        d.out_cap = 3u * w.backbone_length + 1024;
        oo += d.out_cap;
        d.offset = uint32_t(0.01 * w.backbone_length);
        d.tgs = w.tgs ? 1u : 0u;
        d.pad = 0;
        // racon's layer order: std::sort by begin over entries 1.. (backbone at 0)
        // (src/window.cpp:78-85); the same call on the host keeps libstdc++'s
        // order for equal begins.
        rank.resize(size_t(w.n_layers) + 1);
        for (uint32_t j = 0; j <= w.n_layers; ++j) rank[j] = j;
        std::sort(rank.begin() + 1, rank.end(), [&](uint32_t lhs, uint32_t rhs) {
            const uint32_t a = lhs == 0 ? 0u : w.begins[lhs - 1];
            const uint32_t b = rhs == 0 ? 0u : w.begins[rhs - 1];
            return a < b;
        });
        for (uint32_t j = 1; j <= w.n_layers; ++j) {
            const uint32_t s = rank[j] - 1;
            PoaLayerDev& L = ld[lbase + j - 1];
            const uint32_t l = w.layer_lengths[s];
            L.seq_off = off;
            memcpy(in + off, w.layers[s], l);
            off += (l + 15) & ~15u;
            const char* q = w.layer_qualities ? w.layer_qualities[s] : nullptr;
            if (q) {
                if (!phred_bytes(q, l))
                    throw Error{RB_ERR_ARG, "rb_poa: quality values outside '!'..'~' (Phred+33 0..93)"};
                L.qual_off = off;
                memcpy(in + off, q, l);
                off += (l + 15) & ~15u;
            } else {
                L.qual_off = kNoQual;
            }
            L.len = l;
            L.begin = w.begins[s];
            L.end = w.ends[s];
            L.pad = 0;
        }
        lbase += w.n_layers;
    }
    // size-sorted queue: most work first
    uint32_t* order = h_order_.as<uint32_t>();
    std::iota(order, order + n, 0u);
    std::vector<uint64_t> work(n);
    for (size_t i = 0; i < n; ++i) {
        uint64_t s = 0;
        for (uint32_t j = 0; j < wd[i].n_layers; ++j) s += ld[wd[i].layer_base + j].len;
        work[i] = s * (wd[i].bb_len + s / std::max<uint32_t>(1, wd[i].n_layers));
    }
    std::sort(order, order + n, [&](uint32_t x, uint32_t y) { return work[x] != work[y] ? work[x] > work[y] : x < y; });
    d_in_.reserve(std::max<uint64_t>(off, 16));
    d_desc_.reserve(std::max<size_t>(n, 1) * sizeof(PoaWinDev));
    d_layers_.reserve(std::max<uint64_t>(nlayers, 1) * sizeof(PoaLayerDev));
    d_order_.reserve(std::max<size_t>(n, 1) * sizeof(uint32_t));
    check_cuda(cudaEventRecord(ev0_, stream_), "cudaEventRecord");
    check_cuda(cudaMemcpyAsync(d_in_.ptr, in, off, cudaMemcpyHostToDevice, stream_), "H2D windows");
    check_cuda(cudaMemcpyAsync(d_desc_.ptr, wd, n * sizeof(PoaWinDev), cudaMemcpyHostToDevice, stream_), "H2D desc");
    check_cuda(cudaMemcpyAsync(d_layers_.ptr, ld, nlayers * sizeof(PoaLayerDev), cudaMemcpyHostToDevice, stream_),
               "H2D layers");
    check_cuda(cudaMemcpyAsync(d_order_.ptr, order, n * sizeof(uint32_t), cudaMemcpyHostToDevice, stream_),
               "H2D order");
    check_cuda(cudaEventRecord(ev1_, stream_), "cudaEventRecord");
    check_cuda(cudaStreamSynchronize(stream_), "stage sync");
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0_, ev1_);
    stats_.h2d_ms = ms;
    stats_.h2d_bytes = off + n * (sizeof(PoaWinDev) + 4) + nlayers * sizeof(PoaLayerDev);
    in_bytes_ = off;
    in_ptr_ = d_in_.as<uint8_t>();
    layers_ptr_ = d_layers_.as<PoaLayerDev>();
    nwin_ = n;
}

void PoaEngine::stage_device(const uint8_t* d_in, const PoaWinDev* wins, size_t n, const PoaLayerDev* d_layers,
                             const uint64_t* sum_len, const std::vector<std::pair<uint64_t, uint32_t>>& labels,
                             uint32_t max_len, int trim) {
    forget();
    trim_ = trim;
    max_len_ = max_len;
    uint64_t out_cap = 0;
    uint32_t max_nodes = 0;
    for (size_t i = 0; i < n; ++i) {
        out_cap = std::max<uint64_t>(out_cap, wins[i].out_off + wins[i].out_cap);
        max_nodes = uint32_t(std::max<uint64_t>(max_nodes, std::min<uint64_t>(wins[i].bb_len + sum_len[i], 1u << 20)));
    }
    out_cap_ = out_cap;
    max_nodes_cap_ = max_nodes;
    labels_.assign(labels.begin(), labels.begin() + n);
    h_desc_.reserve(std::max<size_t>(n, 1) * sizeof(PoaWinDev));
    h_order_.reserve(std::max<size_t>(n, 1) * sizeof(uint32_t));
    PoaWinDev* wd = h_desc_.as<PoaWinDev>();
    if (n) memcpy(wd, wins, n * sizeof(PoaWinDev));
    // size-sorted queue, the same work estimate as stage()
    uint32_t* order = h_order_.as<uint32_t>();
    std::iota(order, order + n, 0u);
    std::vector<uint64_t> work(n);
    for (size_t i = 0; i < n; ++i) {
        const uint64_t s = sum_len[i];
        work[i] = s * (wd[i].bb_len + s / std::max<uint32_t>(1, wd[i].n_layers));
    }
    std::sort(order, order + n, [&](uint32_t x, uint32_t y) { return work[x] != work[y] ? work[x] > work[y] : x < y; });
    d_desc_.reserve(std::max<size_t>(n, 1) * sizeof(PoaWinDev));
    check_cuda(cudaEventRecord(ev0_, stream_), "cudaEventRecord");
    if (n)
        check_cuda(cudaMemcpyAsync(d_desc_.ptr, wd, n * sizeof(PoaWinDev), cudaMemcpyHostToDevice, stream_),
                   "H2D desc");
    check_cuda(cudaEventRecord(ev1_, stream_), "cudaEventRecord");
    check_cuda(cudaStreamSynchronize(stream_), "stage sync");
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0_, ev1_);
    stats_.h2d_ms = ms;
    stats_.h2d_bytes = n * sizeof(PoaWinDev);
    in_bytes_ = 0;
    in_ptr_ = d_in;
    layers_ptr_ = d_layers;
    nwin_ = n;
}

void PoaEngine::forget() {
    nwin_ = 0;
    in_ptr_ = nullptr;
    layers_ptr_ = nullptr;
}

void PoaEngine::prepare_outputs() {
    const size_t n = nwin_;
    stats_.launches = 0;
    stats_.items = n;
    stats_.cells = 0;
    stats_.edge_cells = 0;
    stats_.kernel_ms = 0;
    stats_.top_kernel_ms = 0;
    if (n == 0) return;
    d_out_.reserve(std::max<uint64_t>(out_cap_, 16));
    d_outlen_.reserve(n * 4);
    d_flags_.reserve(n);
    d_misc_.reserve(64);
}

void PoaEngine::run(bool plain) {
    prepare_outputs();
    const size_t n = nwin_;
    if (n == 0) return;
    std::vector<uint32_t> todo(n);
    const uint32_t* h_order = h_order_.as<uint32_t>();
    // batched form: size-sorted queue (heaviest first, or size buckets
    // interleaved by the device's tuning); plain form: input order
    const rb_tuning tune = tuning_get(dev_.device);
    for (size_t i = 0; i < n; ++i) todo[i] = plain ? uint32_t(i) : h_order[i];
    if (!plain && tune.consensus_order == 1)
        for (size_t i = 0, lo = 0, hi = n; i < n; ++i) todo[i] = h_order[(i & 1) ? --hi : lo++];
    // starting graph capacity; windows that outgrow it run again with four
    // times as much. RB_POA_NCAP lowers the start (tests of the retry path);
    // results do not depend on it.
    int ncap = 4096;
    if (const char* e = getenv("RB_POA_NCAP")) ncap = std::max(256, std::min(4096, atoi(e)));
    run_list(std::move(todo), ncap, plain);
}

void PoaEngine::run_list(std::vector<uint32_t> todo, int ncap, bool plain) {
    const size_t n = nwin_;
    std::vector<uint8_t> flags(n);
    float total_ms = 0;
    // DP row width: every layer's columns rounded up to whole warp passes
    const uint32_t* lens_max = &max_len_;
    const int lcap = max_cover(int(*lens_max) + 1);
    while (!todo.empty()) {
        const int ecap = 2 * ncap, acap = ncap;
        const size_t slot = walk_layout(ncap, ecap, acap, lcap, [](int, size_t) {});
        // Warps per window. Four warps side by side finish a window sooner
        // (150 windows of 1000 bases at 20x: 27 ms against 64 ms), one warp
        // spends the fewest instructions (2001 windows of 500 bases at 50x:
        // 79 ms against 109 ms). The line lies at four windows per SM, where
        // the two meet for windows of 500 bases (30x, kernel ms with one and
        // with four warps: 300 windows 24.0 / 20.4, 592 27.2 / 26.0, 600 24.8 /
        // 25.2, 888 26.3 / 30.7, 1776 31.6 / 42.9). Windows of 200 meet a
        // little before it (300: 8.7 / 8.2, 592: 9.8 / 10.0), windows of 1000
        // past the resident teams (888: 107 / 76, 1776: 162 / 115).
        const int nw = plain ? kPlainWarps : todo.size() <= 4 * size_t(dev_.sm_count) ? 4 : 1;
        const size_t teams = size_t(cta_warps(nw)) / nw;  // per full CTA
        // resident windows (one team each): enough to fill the SMs, bounded by
        // a scratch budget
        const size_t budget = scratch_budget_;
        // resident windows: the device's tuned CTAs per SM on the context's
        // share of the SMs (all by default)
        const uint32_t cps = std::min<uint32_t>(kCtasPerSm, tuning_get(dev_.device).consensus_ctas_per_sm);
        const size_t resident =
            std::max<size_t>(teams, size_t(dev_.sm_count) * teams * cps * sm_share_pct_ / 100);
        size_t slots = std::min<size_t>(todo.size(), plain ? todo.size() : resident);
        // RB_POA_SLOTS caps the resident windows (smaller scratch, e.g. for
        // profiler captures); results do not depend on it
        if (const char* e = getenv("RB_POA_SLOTS"))
            slots = std::max<size_t>(1, std::min<size_t>(slots, strtoull(e, nullptr, 10)));
        while (slots > 1 && slots * slot > budget) slots /= 2;
        // teams per CTA: one while that still leaves SMs free, so that a small
        // batch spreads over all of them
        const size_t per_cta =
            std::max<size_t>(1, std::min<size_t>(teams, slots / std::max<size_t>(1, size_t(dev_.sm_count) * sm_share_pct_ / 100)));
        if (!plain) slots = (slots + per_cta - 1) / per_cta * per_cta;
        d_graph_.reserve(slots * slot);
        DevBuf& d_todo = d_dp_;
        d_todo.reserve(todo.size() * 4);
        check_cuda(cudaMemcpyAsync(d_todo.ptr, todo.data(), todo.size() * 4, cudaMemcpyHostToDevice, stream_),
                   "H2D todo");
        PoaArgs a;
        memset(&a, 0, sizeof(a));
        a.in = in_ptr_;
        a.wins = d_desc_.as<PoaWinDev>();
        a.layers = layers_ptr_;
        a.order = d_todo.as<uint32_t>();
        a.nwin = uint32_t(todo.size());
        a.out = d_out_.as<char>();
        a.out_len = d_outlen_.as<uint32_t>();
        a.flags = d_flags_.as<uint8_t>();
        a.scratch = d_graph_.as<uint8_t>();
        a.slot_bytes = slot;
        a.ncap = ncap;
        a.ecap = ecap;
        a.acap = acap;
        a.lcap = lcap;
        a.match = match_;
        a.mismatch = mismatch_;
        a.gap = gap_;
        a.trim = trim_;
        a.counters = d_misc_.as<unsigned int>();
        a.cells = reinterpret_cast<unsigned long long*>(d_misc_.as<unsigned int>() + 8);
        // RB_POA_WAIT_POLLS shortens the limit (tests of a wait that runs out)
        a.wait_polls = kWaitPolls;
        if (const char* e = getenv("RB_POA_WAIT_POLLS")) a.wait_polls = std::max(0, std::min(kWaitPolls, atoi(e)));
        check_cuda(cudaMemsetAsync(d_misc_.ptr, 0, 64, stream_), "memset counters");
        check_cuda(cudaEventRecord(ev0_, stream_), "cudaEventRecord");
        if (plain) {
            // one launch per batch of `slots` windows
            const int smem = kPlainWarps * warp_smem(kPlainWarps);
            check_cuda(cudaFuncSetAttribute(poa_plain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "cudaFuncSetAttribute");
            for (size_t b0 = 0; b0 < todo.size(); b0 += slots) {
                PoaArgs ab = a;
                ab.order = a.order + b0;
                ab.nwin = uint32_t(std::min(slots, todo.size() - b0));
                poa_plain_kernel<<<int(ab.nwin), 32 * kPlainWarps, smem, stream_>>>(ab);
                ++stats_.launches;
            }
        } else {
            void (*const kernel)(PoaArgs) = nw == 4 ? poa_kernel<4> : poa_kernel<1>;
            const int smem = int(per_cta) * nw * warp_smem(nw);
            check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            cta_warps(nw) * warp_smem(nw)),
                       "cudaFuncSetAttribute");
            // persistent by default; with a per-warp cap, enough launches
            // back to back that every window is taken
            size_t launches = 1;
            if (yield_windows_ > 0) {
                a.per_warp_cap = yield_windows_;
                launches = (todo.size() + slots * yield_windows_ - 1) / (slots * yield_windows_);
            }
            for (size_t l = 0; l < launches; ++l) {
                kernel<<<int(slots / per_cta), int(per_cta) * nw * 32, smem, stream_>>>(a);
                ++stats_.launches;
            }
        }
        check_cuda(cudaEventRecord(ev1_, stream_), "cudaEventRecord");
        unsigned long long cells[2] = {0, 0};
        check_cuda(cudaMemcpyAsync(cells, a.cells, 16, cudaMemcpyDeviceToHost, stream_), "D2H cells");
        check_cuda(cudaMemcpyAsync(flags.data(), d_flags_.ptr, n, cudaMemcpyDeviceToHost, stream_), "D2H flags");
        check_cuda(cudaStreamSynchronize(stream_), "poa sync");
        check_cuda(cudaGetLastError(), "poa kernel");
        float ms = 0;
        cudaEventElapsedTime(&ms, ev0_, ev1_);
        total_ms += ms;
        stats_.cells += cells[0];
        stats_.edge_cells += cells[1];
        std::vector<uint32_t> again;
        for (uint32_t w : todo) {
            if (flags[w] & kFailed) throw Error{RB_ERR_DEVICE, "rb_poa: window consensus failed on the device"};
            if (flags[w] & kOverflow) again.push_back(w);
        }
        if (!again.empty()) {
            if (ncap >= (1 << 20)) throw Error{RB_ERR_DEVICE, "rb_poa: window graph exceeds 2^20 nodes"};
            ncap *= 4;
        }
        todo.swap(again);
    }
    stats_.kernel_ms += total_ms;
    stats_.top_kernel_ms += total_ms;
    stats_.max_nodes = uint32_t(ncap);
}

void PoaEngine::fetch(rb_poa_result* out) {
    const size_t n = nwin_;
    std::vector<uint32_t> lens(n);
    std::vector<uint8_t> flags(n);
    h_out_.reserve(std::max<uint64_t>(out_cap_, 16));
    check_cuda(cudaEventRecord(ev2_, stream_), "cudaEventRecord");
    if (n) {
        check_cuda(cudaMemcpyAsync(lens.data(), d_outlen_.ptr, n * 4, cudaMemcpyDeviceToHost, stream_), "D2H lens");
        check_cuda(cudaMemcpyAsync(flags.data(), d_flags_.ptr, n, cudaMemcpyDeviceToHost, stream_), "D2H flags");
        check_cuda(cudaMemcpyAsync(h_out_.ptr, d_out_.ptr, out_cap_, cudaMemcpyDeviceToHost, stream_), "D2H cons");
    }
    check_cuda(cudaEventRecord(ev3_, stream_), "cudaEventRecord");
    check_cuda(cudaStreamSynchronize(stream_), "fetch sync");
    float ms = 0;
    cudaEventElapsedTime(&ms, ev2_, ev3_);
    stats_.d2h_ms = ms;
    stats_.d2h_bytes = n * 5 + out_cap_;
    const PoaWinDev* wd = h_desc_.as<PoaWinDev>();
    const char* src = h_out_.as<char>();
    offsets_.assign(n + 1, 0);
    cons_.clear();
    polished_.assign(n, 0);
    for (size_t i = 0; i < n; ++i) {
        offsets_[i] = cons_.size();
        cons_.insert(cons_.end(), src + wd[i].out_off, src + wd[i].out_off + lens[i]);
        polished_[i] = (flags[i] & kPolished) ? 1 : 0;
        if (flags[i] & kChimeric) {
            fprintf(stderr, "[racon::Window::generate_consensus] warning: contig %lu might be chimeric in window %u!\n",
                    (unsigned long)labels_[i].first, labels_[i].second);
        }
    }
    offsets_[n] = cons_.size();
    out->consensus = cons_.data();
    out->offsets = offsets_.data();
    out->polished = polished_.data();
}

}  // namespace rb

// ---------------------------------------------------------------------------
// Shared window-consensus service (continuous batching for the serving loop)

namespace rb {

struct PoaSvcState {
    explicit PoaSvcState(int device) : ring(device, sizeof(PoaJobDev), "rb_poa service") {}
    RingService ring;
    void* d_scratch = nullptr;  // one graph slot per resident warp
    PoaSvcArgs args{};
    uint32_t slots = 0, grid = 0;
};

namespace {
cudaError_t launch_poa_service(cudaStream_t stream, void* user) {
    const PoaSvcState* S = static_cast<const PoaSvcState*>(user);
    poa_service_kernel<<<S->grid, 32 * kSvcWarps, kSvcWarps * warp_smem(kSvcTeamWarps), stream>>>(S->args);
    return cudaGetLastError();
}
}  // namespace

PoaService::PoaService(int device, int8_t m, int8_t x, int8_t g, uint32_t window_length, size_t scratch_budget,
                       uint32_t ctas_per_sm, uint32_t large_first_every)
    : st_(nullptr) {
    check_cuda(cudaSetDevice(device), "cudaSetDevice");
    int sm_count = 148;
    check_cuda(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device), "sm count");
    std::unique_ptr<PoaSvcState> S(new PoaSvcState(device));
    // slot layout for layers up to three window lengths; longer ones (and
    // graphs over 4096 nodes) overflow and run again in the job's own engine
    const int ncap = 4096, ecap = 2 * ncap, acap = ncap;
    const int lcap = row_cover(kSvcTeamWarps, int(std::max<uint32_t>(window_length, 1)) * 3 + 1);
    const size_t teams = kSvcWarps / kSvcTeamWarps;
    const size_t slot = walk_layout(ncap, ecap, acap, lcap, [](int, size_t) {});
    const uint32_t cps = std::max<uint32_t>(1, std::min<uint32_t>(ctas_per_sm, kSvcCtasPerSm));
    size_t slots = size_t(sm_count) * cps * teams;
    while (slots > teams && slots * slot > scratch_budget) slots -= teams;
    S->slots = uint32_t(slots);
    S->grid = uint32_t(slots / teams);
    check_cuda(cudaMalloc(&S->d_scratch, slots * slot), "cudaMalloc service scratch");
    PoaSvcArgs& A = S->args;
    memset(&A, 0, sizeof(A));
    A.base.scratch = static_cast<uint8_t*>(S->d_scratch);
    A.base.slot_bytes = slot;
    A.base.ncap = ncap;
    A.base.ecap = ecap;
    A.base.acap = acap;
    A.base.lcap = lcap;
    A.base.match = m;
    A.base.mismatch = x;
    A.base.gap = g;
    A.base.wait_polls = kWaitPolls;
    S->ring.set_large_first_every(large_first_every);
    A.jobs = static_cast<const PoaJobDev*>(S->ring.records());
    A.q = S->ring.queue();
    check_cuda(cudaFuncSetAttribute(poa_service_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSvcWarps * warp_smem(kSvcTeamWarps)),
               "cudaFuncSetAttribute");
    prefer_max_shared(reinterpret_cast<const void*>(poa_service_kernel));
    st_ = S.release();
    st_->ring.start(launch_poa_service, st_);
}

PoaService::~PoaService() {
    st_->ring.stop();
    cudaFree(st_->d_scratch);
    delete st_;
}

uint32_t PoaService::slots() const { return st_->slots; }
uint32_t PoaService::launches() const { return st_->ring.launches(); }

void PoaService::run_batch(const PoaJobDev& job, const uint32_t* order, size_t n, int queue) {
    st_->ring.run_batch(&job, order, n, queue);
}

void PoaEngine::run_shared(PoaService& svc, uint32_t priority_windows) {
    prepare_outputs();
    const size_t n = nwin_;
    if (n == 0) return;
    check_cuda(cudaMemsetAsync(d_misc_.ptr, 0, 64, stream_), "memset counters");
    // the batch's inputs and descriptors are complete on this engine's stream
    check_cuda(cudaStreamSynchronize(stream_), "poa stage sync");
    PoaJobDev job;
    memset(&job, 0, sizeof(job));
    job.in = in_ptr_;
    job.wins = d_desc_.as<PoaWinDev>();
    job.layers = layers_ptr_;
    job.out = d_out_.as<char>();
    job.out_len = d_outlen_.as<uint32_t>();
    job.flags = d_flags_.as<uint8_t>();
    job.cells = reinterpret_cast<unsigned long long*>(d_misc_.as<unsigned int>() + 8);
    job.trim = trim_;
    const auto t0 = std::chrono::steady_clock::now();
    // size class: ring 0 up to priority_windows windows, then x4 per ring
    const uint64_t p = std::max<uint32_t>(1, priority_windows);
    const int queue = n <= p ? 0 : n <= 4 * p ? 1 : n <= 16 * p ? 2 : 3;
    svc.run_batch(job, h_order_.as<uint32_t>(), n, queue);
    const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    std::vector<uint8_t> flags(n);
    unsigned long long cells[2] = {0, 0};
    check_cuda(cudaMemcpyAsync(flags.data(), d_flags_.ptr, n, cudaMemcpyDeviceToHost, stream_), "D2H flags");
    check_cuda(cudaMemcpyAsync(cells, job.cells, 16, cudaMemcpyDeviceToHost, stream_), "D2H cells");
    check_cuda(cudaStreamSynchronize(stream_), "poa sync");
    stats_.cells = cells[0];
    stats_.edge_cells = cells[1];
    stats_.kernel_ms = ms;
    stats_.top_kernel_ms = ms;
    std::vector<uint32_t> again;
    for (uint32_t w = 0; w < n; ++w) {
        if (flags[w] & kFailed) throw Error{RB_ERR_DEVICE, "rb_poa: window consensus failed on the device"};
        if (flags[w] & kOverflow) again.push_back(w);
    }
    // windows that outgrew the shared slots: this engine's own launch with
    // four times the graph capacity (the same path a private run takes)
    if (!again.empty()) run_list(std::move(again), 4 * 4096, false);
}

}  // namespace rb
