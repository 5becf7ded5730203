// count.cu -- exact and hybrid (exact / HyperLogLog) triangle counting.
//
// Reference semantics (ChitandaEruQ/triangle_counting_hll):
//   exact:   T = sum over oriented edges (u,v) of |N+(u) cap N+(v)|
//            src/exact.py:48-98, src/gpu_hybrid.py:96-130,332-354
//   hybrid:  edge -> HLL iff min(d+u, d+v) >= gamma and both endpoints carry a
//            sketch (src/hybrid.py:107-115, src/gpu_hybrid.py:80-89); HLL edges
//            add clamp(d+u + d+v - |N+(u) cup N+(v)|^, 0, min(d+u, d+v))
//            (src/hybrid.py:117-126, src/gpu_hybrid.py:288-302), the union
//            estimated from the register-wise max of the two sketches with the
//            reference's bias and range corrections (src/hll.py:37-54,112-120).
//
// Design
//   * Table side / probe side.  |N+(u) cap N+(v)| is symmetric, so each exact
//     edge becomes a pair (x, y) with x the endpoint of the LONGER list: the
//     members of the shorter list are looked up in the longer one, which drops
//     the look-ups from sum d+(v) to sum min(d+u, d+v) (43.4 G list elements ->
//     11.8 G on R-MAT scale 22).
//   * A first pass over the edges (pair_pass_kernel) counts pairs of short
//     lists on the spot by binary search and counts the others per table
//     side; a counting sort then groups those by x.  They are the hub pairs
//     (d+(x) > hub threshold; 98% of the look-ups on R-MAT scale 22) and, in
//     graphs of evenly long lists, the table pairs (is_table_pair).
//   * Hub pairs are counted by a CTA per group of x's pairs, all its warps
//     sharing one bitmap of N+(x) in shared memory (hub_bitmap16_kernel), in
//     the coordinates of the core, the vertices of the hub lists.
//   * Small dense graphs, per-edge outputs and fused hybrid counts take the
//     edges as given: a warp keeps N+(u) in a private hash table (count_kernel:
//     one 4-byte word per slot at load <= 1/8, a lookup is one shared load
//     with a rare walk) while it streams the N+(v) lists through it; tiny
//     pairs are merged lane-locally, lists too long for the table searched.
//   * Lists of a group are flattened into one stream of 16-byte units dealt to
//     the 32 lanes by a warp scan, so short and long lists keep every lane
//     busy.
//   * HLL edges: the warp reads both 2^p-byte register rows with 16-byte
//     loads, merges them with __vmaxu4 and accumulates sum 2^-r EXACTLY as a
//     128-bit fixed-point integer; one lane applies the FP64 corrections,
//     clamps and adds the result in 2^-32 fixed point.
//   * Every total is an integer (uint64 exact count, 128-bit fixed-point HLL
//     sum, int64 stats) added with integer atomics, so results do not depend
//     on scheduling or partitioning: they are bit-identical run to run.
#include <cub/cub.cuh>

#include <atomic>
#include <mutex>

#include "common.cuh"
#include "hll_device.cuh"

namespace tchll {

enum : int { MODE_EXACT = 0, MODE_HYBRID = 1, MODE_HYB_EXACT = 2, MODE_HYB_HLL = 3 };

enum : uint32_t {
    ST_BAD_EDGE = 1u,  // edge endpoint outside [0, n_nodes)
    ST_BAD_ROW = 2u,   // row_ptr extent outside [0, nnz] or decreasing
    ST_BAD_SLOT = 4u,  // sketch slot outside [0, n_rows)
    ST_BAD_KEY = 8u,   // neighbour id (col_idx value) outside [0, n_nodes)
};

// Pairs of one table side x, next to each other in the list of probe sides.
struct PairSeg {
    int32_t start;  // the first pair (the list holds < 2^31 entries)
    int32_t x;
    int32_t len;
    int32_t graph;  // batched counts: the graph of x (its result block); else 0
};

struct CountParams {
    const int32_t* row_ptr;
    const int2* rows;  // the row table, or null
    uint2* codes;      // per 32 edges of the first pass: {grouped pairs, those with x = u} (with rows)
    int64_t n_nodes;
    const int32_t* col_idx;
    int64_t nnz;
    const int32_t* edge_u;
    const int32_t* edge_v;
    int64_t n_edges;
    const int32_t* degrees;      // forward degree for routing (hybrid modes)
    const uint8_t* regs;         // register rows
    int64_t n_rows;              // rows available in regs
    const int64_t* slot;         // compact layout: row of v, or -1; null -> dense
    const uint8_t* has;          // dense layout: has_sketch[v] == 1 -> row v
    int p;
    int64_t gamma;
    int variant;          // HLL estimator: 0 the reference's src/hll.py, 1 cpu_exp's
    int64_t* pe_support;  // per-edge exact support (details), zeroed by host
    double* pe_s_hat;     // per-edge HLL s_hat (details)
    double* pe_s_cl;      // per-edge HLL clamped support (details)
    uint8_t* pe_method;   // per-edge 0 exact / 1 hll (details)
    tchll_count_result* result;
    unsigned long long* work;  // chunks are claimed here (null: dealt to the warps in turn)
    int check_ids;  // validate every row first
    int chunk;
    int slots_log2;  // per-warp table capacity (log2 slots)
    int tiny;        // lane-local merge when |N+x| + |N+y| <= tiny
    int sparse;      // 1: table load <= 1/4 where it fits (else <= 1/2)
    // Batched mode: work units are chunks [chunk_start[i], +chunk_len[i]) of
    // one graph each (never crossing a graph), claimed one at a time; each
    // chunk's totals go to results[chunk_graph[i]].
    const int64_t* chunk_start;
    const int32_t* chunk_len;
    const int32_t* chunk_graph;
    const int64_t* n_chunks_dev;
    const int32_t* graph_vbase;  // vertex range of graph g: [vbase[g], vbase[g+1])
    int64_t n_graphs;            // batched calls: graphs in graph_vbase (else 0)
    unsigned long long* graph_bad;  // batched calls: of them, those from the first malformed one on
    int32_t* graph_hub;          // batched calls: what the first pass left for later, GRAPH_*
    int32_t* live_flag;          // batched calls: 1 for 64 rows that touch such a graph
    int32_t* live_list;          // and those blocks of 64 rows, listed
    int32_t* n_live;             // how many
    int32_t* big_hist;           // batched calls: 512 words per slot of a big graph (core_bucket_big_kernel)
    // Table pairs (count_kernel with SEGS): their segments, the first one right
    // before segs_end, the second before that; edge_v holds the probe sides
    const PairSeg* segs_end;
    const unsigned long long* n_segs;
    unsigned long long* est;  // see Choice (null: neither hub nor table pairs)
    int hub;
    int hub_alt;
    // Hybrid with pairs: the routing pass appends HLL edges here
    int32_t* hll_u;
    int32_t* hll_v;
    unsigned long long* hll_n;
};

// Hash table of one 4-byte word per slot (per-warp tables of the pair kernel
// and the CTA tables of the hub kernel): bits 0-30 the key (0x7FFFFFFF =
// empty; vertex ids stay below INT32_MAX) and bit 31 an overflow flag.  A
// key lives in its home slot h1(k) when that was free at insertion; otherwise
// it sets the flag on h1(k) and takes the first free slot of a linear walk
// from h2(k).  A lookup reads the home slot: match -> hit; flag clear ->
// miss; flag set (about load^2 of the slots) -> walk from h2(k) to the key or
// a free slot.  At load <= 1/8 almost every lookup is ONE 4-byte shared load
// and the warp rarely diverges.
constexpr uint32_t OV_KEY = 0x7FFFFFFFu;   // key bits; this value marks an empty slot
constexpr uint32_t OV_FLAG = 0x80000000u;  // some key of this home slot lives on its h2 walk
constexpr uint32_t OV_NONE = 0x7FFFFFFEu;  // probe that matches no slot (vertex ids are below it)

__device__ __forceinline__ uint32_t ov_h1(int32_t x, int sh) { return ((uint32_t)x * 0x9E3779B1u) >> sh; }
__device__ __forceinline__ uint32_t ov_h2(int32_t x, int sh) { return ((uint32_t)x * 0x85EBCA77u) >> sh; }

// Claims slot h for key x if its key bits are empty (keeps the flag bit).
// Returns 1 placed, 0 occupied by another key, 2 already holds x.
__device__ __forceinline__ int ov_claim(uint32_t* T, uint32_t h, uint32_t x) {
    uint32_t old = *(volatile uint32_t*)(T + h);
    while ((old & OV_KEY) == OV_KEY) {
        const uint32_t prev = atomicCAS(T + h, old, (old & OV_FLAG) | x);
        if (prev == old) return 1;
        old = prev;
    }
    return (old & OV_KEY) == x ? 2 : 0;
}

// Inserts x; false only if the h2 walk finds no free slot (full table).
__device__ __forceinline__ bool ov_insert(uint32_t* T, int32_t x, int sh, uint32_t mask) {
    const uint32_t h = ov_h1(x, sh);
    if (ov_claim(T, h, (uint32_t)x)) return true;
    atomicOr(T + h, OV_FLAG);
    uint32_t g = ov_h2(x, sh);
    for (uint32_t i = 0; i <= mask; ++i) {
        if (ov_claim(T, g, (uint32_t)x)) return true;
        g = (g + 1u) & mask;
    }
    return false;
}

// The h2 walk of a lookup whose home slot was flagged: 1 at x, 0 at a free
// slot; at most mask + 1 steps.
__device__ __forceinline__ uint32_t ov_walk(const uint32_t* T, int32_t x, int sh, uint32_t mask) {
    uint32_t g = ov_h2(x, sh);
    for (uint32_t i = 0; i <= mask; ++i) {
        const uint32_t k = T[g] & OV_KEY;
        if (k == (uint32_t)x) return 1u;
        if (k == OV_KEY) return 0u;
        g = (g + 1u) & mask;
    }
    return 0u;
}

__device__ __forceinline__ int ceil_log2_i(int x) { return x <= 1 ? 0 : 32 - __clz(x - 1); }

// Loads and validates edge e; returns false (and flags status) when malformed.
__device__ __forceinline__ bool load_edge(const CountParams& P, int64_t e, int32_t& u, int32_t& v, int32_t& us,
                                          int32_t& ue, int32_t& vs, int32_t& ve, uint32_t& status) {
    // the edge arrays stream through once per pass: evict-first loads keep
    // L1 for the row_ptr entries of the high-degree endpoints, which recur
    u = __ldcs(P.edge_u + e);
    v = __ldcs(P.edge_v + e);
    const uint32_t n = (uint32_t)P.n_nodes, nnz = (uint32_t)P.nnz;  // both below 2^31
    if ((uint32_t)u >= n || (uint32_t)v >= n) {
        status |= ST_BAD_EDGE;
        return false;
    }
    us = __ldg(P.row_ptr + u);
    ue = __ldg(P.row_ptr + u + 1);
    vs = __ldg(P.row_ptr + v);
    ve = __ldg(P.row_ptr + v + 1);
    // 0 <= start <= end <= nnz
    if ((uint32_t)us > (uint32_t)ue || (uint32_t)ue > nnz || (uint32_t)vs > (uint32_t)ve || (uint32_t)ve > nnz) {
        status |= ST_BAD_ROW;
        return false;
    }
    return true;
}

// The row table (prepare_kernel): {row start, row end} per vertex, with the
// vertex's part in the routing in the sign bits: its degree reaches gamma
// (start), it has a sketch (end).  min(d+u, d+v) >= gamma iff both ends reach
// it, so one 8-byte load per endpoint replaces up to four.  Malformed entries
// have start > end.
constexpr int32_t kRowBad = 0x7FFFFFFF;   // {kRowBad, 0}: a bad extent
constexpr int32_t kSlotBad = 0x7FFFFFFE;  // {kSlotBad, 0}: a sketch slot outside the rows
__device__ __forceinline__ bool load_edge_rows(const CountParams& P, int64_t e, int32_t& u, int32_t& v, int32_t& us,
                                               int32_t& ue, int32_t& vs, int32_t& ve, bool& wants, bool& both,
                                               uint32_t& status) {
    u = __ldcs(P.edge_u + e);
    v = __ldcs(P.edge_v + e);
    const uint32_t n = (uint32_t)P.n_nodes;
    if ((uint32_t)u >= n || (uint32_t)v >= n) {
        status |= ST_BAD_EDGE;
        return false;
    }
    const int2 ru = __ldg(P.rows + u), rv = __ldg(P.rows + v);
    wants = (ru.x & rv.x) < 0;
    both = (ru.y & rv.y) < 0;
    us = ru.x & 0x7FFFFFFF;
    ue = ru.y & 0x7FFFFFFF;
    vs = rv.x & 0x7FFFFFFF;
    ve = rv.y & 0x7FFFFFFF;
    if (us > ue || vs > ve) {
        const bool slot = (us <= ue || us == kSlotBad) && (vs <= ve || vs == kSlotBad);
        status |= slot ? ST_BAD_SLOT : ST_BAD_ROW;
        return false;
    }
    return true;
}

// Every row's extent and every listed neighbour id, by the whole grid: what
// the hub core's passes check as they read the rows, for the calls that do
// not need them.  Well-formed rows cover col[row_ptr[0] .. row_ptr[n_nodes]).
__device__ __forceinline__ void validate_rows(const int32_t* __restrict__ row_ptr, int64_t n_nodes, int64_t nnz,
                                              const int32_t* __restrict__ col, uint32_t& status) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = t0; r < n_nodes; r += step) {
        const int32_t a = __ldg(row_ptr + r), b = __ldg(row_ptr + r + 1);
        if (a < 0 || b < a || (int64_t)b > nnz) status |= ST_BAD_ROW;
    }
    const int64_t lo = __ldg(row_ptr), hi = __ldg(row_ptr + n_nodes);
    if (lo < 0 || hi < lo || hi > nnz) return;
    // 16-byte loads between the first and the last 16-byte boundary: col may
    // start on any word
    const int64_t head = lo + (int64_t)((4 - (((uintptr_t)(col + lo) >> 2) & 3)) & 3);
    const int64_t l4 = min(head, hi), n4 = (hi - l4) >> 2, h4 = l4 + 4 * n4;
    const uint32_t n = (uint32_t)n_nodes;
    const uint4* __restrict__ quads = reinterpret_cast<const uint4*>(col + l4);
    bool bad = false;
    for (int64_t q = t0; q < n4; q += step) {
        const uint4 v = __ldg(quads + q);
        bad |= v.x >= n || v.y >= n || v.z >= n || v.w >= n;
    }
    if (lo + t0 < l4) bad |= (uint32_t)__ldg(col + lo + t0) >= n;
    if (h4 + t0 < hi) bad |= (uint32_t)__ldg(col + h4 + t0) >= n;
    if (bad) status |= ST_BAD_KEY;
}

// Hybrid routing (src/hybrid.py:107-115): wants = min(deg) >= gamma,
// both = both endpoints have a sketch.  Returns false on a bad slot.
__device__ __forceinline__ bool route(const CountParams& P, int32_t u, int32_t v, int32_t& du, int32_t& dv,
                                      int64_t& su, int64_t& sv, bool& wants, bool& both, uint32_t& status) {
    du = __ldg(P.degrees + u);
    dv = __ldg(P.degrees + v);
    const int64_t proxy = du < dv ? du : dv;
    wants = proxy >= P.gamma;
    if (P.slot) {
        su = __ldg(P.slot + u);
        sv = __ldg(P.slot + v);
    } else {
        su = __ldg(P.has + u) == 1 ? (int64_t)u : -1;
        sv = __ldg(P.has + v) == 1 ? (int64_t)v : -1;
    }
    if (su >= P.n_rows || sv >= P.n_rows) {
        status |= ST_BAD_SLOT;
        return false;
    }
    both = su >= 0 && sv >= 0;
    return true;
}

// ------------------------------------------------------------ pair build ----
// An exact edge is a pair of lists: the longer is its table side, the shorter
// its probe side (ties: u is the table side).
struct PairSides {
    int32_t x, y;            // table side, probe side
    int32_t xs, xl, ys, yl;  // their lists: start, length
};
__device__ __forceinline__ PairSides sides_of(int32_t u, int32_t v, int32_t us, int32_t ue, int32_t vs, int32_t ve) {
    const int32_t lu = ue - us, lv = ve - vs;
    const bool ux = lu >= lv;
    PairSides S;
    S.x = ux ? u : v;
    S.y = ux ? v : u;
    S.xs = ux ? us : vs;
    S.xl = ux ? lu : lv;
    S.ys = ux ? vs : us;
    S.yl = ux ? lv : lu;
    return S;
}
// Hub pairs: a long table side and something to probe it with.
__device__ __forceinline__ bool is_hub_pair(const PairSides& S, int hub) { return hub > 0 && S.xl > hub && S.yl > 0; }
// Table pairs, of the others: a table side and a probe side of some length.
// They are grouped by table side like hub pairs and counted with a warp's
// hash table of it (count_kernel with SEGS), where a look-up is one shared
// load instead of a search of 4 and more steps.  That takes many pairs to a
// table side, which skewed graphs do not have (R-MAT 20, 4 to a side: 272 us in
// tables, 25 in searches), so prepare_kernel estimates them, from a sample of
// the edges and the number of lists of such a length, and below kTableMin to a
// side the pairs are searched: R-MAT 16 to 22 have 4 to 17, graphs of evenly
// long lists 25 and more.  So are they where they are less than one in
// kTableShare of all pairs, which does not pay for the launch's tail (50 K
// vertices joined to 80 near ones, one in ten: 423 us in tables, 362 in
// searches).  Whole calls, us, all pairs in tables / all in searches / so: a
// million vertices joined to 20 near ones 1,493 / 1,009 / 1,024, to 30 2,088 / 2,164
// / 1,886, to 40 2,755 / 3,673 / 2,651, to 60 4,475 / 8,420 / 4,407; Erdos-Renyi, 40 M
// edges 3,808 / 4,768 / 3,480.
constexpr int kTableList = 32;
constexpr int kTableProbes = 8;
constexpr int kTableMin = 20;
constexpr int kTableShare = 5;
constexpr int kEdgeSample = 8192;
__device__ __forceinline__ bool is_table_pair(const PairSides& S, int list) {
    return list > 0 && S.xl > list && S.yl > kTableProbes;
}

// Largest core that the packed lists hold (core_lists_kernel).
constexpr int32_t kCore16Max = 131070;

// The hub threshold of a call and whether it has table pairs.  The host gives
// the threshold, and with hub_alt leaves it to the device to double it; what
// the device goes by is est: {sampled pairs with a list in (kTableList, hub]
// and more than kTableProbes probes, lists of that length, the same two for
// (hub, 2 hub], vertices of a batch's largest graph, whether a batch has a big
// graph (kBigGraph)}.  It is doubled where half
// of all pairs have lists in (kTableList, 2 hub], because evenly long lists bring
// all vertices into the core (a batch's largest graph permitting; batches of
// more than kHub64Edges edges always, when that graph's core may not fit).
// Whole calls, us, at 64 / at 128: Erdos-Renyi with 300 K vertices and 24 M edges
// 3,277 / 2,930, 300 K vertices joined to 50 near ones 1,487 / 1,129; R-MAT 20, one
// pair in ten, 1,590 / 1,800, R-MAT 22 with edge factor 2 895 / 1,013.
constexpr int kEst = 6;
constexpr int64_t kHub64Edges = 28000000;
struct Choice {
    int hub, table;
};
__host__ __device__ __forceinline__ Choice choose(const unsigned long long* est, int64_t n_edges, int hub, int hub_alt,
                                                  bool batched) {
    const unsigned long long n = (unsigned long long)n_edges, of = n < kEdgeSample ? n : kEdgeSample;
    unsigned long long pairs = est[0], lists = est[1];
    const bool even = 2 * (pairs + est[2]) >= of;
    if (hub_alt && (batched ? est[4] > (unsigned long long)kCore16Max && (even || n_edges > kHub64Edges) : even)) {
        hub *= 2;
        pairs += est[2];
        lists += est[3];
    }
    const bool table = pairs * kTableShare >= of && pairs * n >= kTableMin * lists * of;
    return Choice{hub, table ? kTableList : 0};
}

// Batched calls: the graph of vertex v, the last g with vbase[g] <= v among
// the graphs before the first malformed one (the only ones with edges).
__device__ __forceinline__ int64_t graph_of(const int32_t* vbase, int64_t n_graphs, const unsigned long long* bad,
                                            int32_t v) {
    int64_t lo = 0, hi = n_graphs - 1 - (int64_t)__ldg(bad);
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (__ldg(vbase + mid) <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Lanes whose pairs share x in a run of consecutive lanes (edges in CSR
// order share u, so the pairs with x = u come in runs): the run's first lane
// (head) and its length.  key must differ between lanes that may not merge.
// Whole warps call it (the grid-stride loops below are warp-uniform).
__device__ __forceinline__ void lane_runs(int32_t key, int lane, int& head_lane, int& run_len) {
    const int32_t prev = __shfl_up_sync(FULL, key, 1);
    const unsigned heads = __ballot_sync(FULL, lane == 0 || prev != key);
    const unsigned le = (2u << lane) - 1u;
    head_lane = 31 - __clz(heads & le);
    const unsigned after = heads & ~((2u << head_lane) - 1u);  // heads after this run's head
    run_len = (after ? __ffs(after) - 1 : 32) - head_lane;
}

// Appends the lanes' HLL-routed edges to the list, one atomic per warp.
__device__ __forceinline__ void append_hll(const CountParams& P, bool hll, int32_t u, int32_t v, int lane) {
    const unsigned bal = __ballot_sync(FULL, hll);
    if (bal) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(P.hll_n, (unsigned long long)__popc(bal));
        base = __shfl_sync(FULL, base, 0);
        if (hll) {
            const unsigned long long pos = base + __popc(bal & ((1u << lane) - 1u));
            P.hll_u[pos] = u;
            P.hll_v[pos] = v;
        }
    }
}

// The grouped pairs' probe sides, by table side: py[cursor[x] ...).  Which
// edges they are and which end is x comes from the first pass, two bits
// per edge, so no row is looked up again (R-MAT 22: 1.12 ms with the rows looked up again, 0.81 so).
__device__ __forceinline__ void scatter_step(const CountParams& P, int64_t e, uint2 code, int32_t* cursor, int32_t* py,
                                             int lane) {
    if (code.x == 0) return;  // warp-uniform
    const bool ok = (code.x >> lane) & 1u, xu = (code.y >> lane) & 1u;
    int32_t u = 0, v = 0;
    if (ok) {
        u = __ldcs(P.edge_u + e);
        v = __ldcs(P.edge_v + e);
    }
    const int32_t x = xu ? u : v;
    // a run of lanes with the same x claims its positions with one atomic
    int head, len;
    lane_runs(ok ? x : -1 - lane, lane, head, len);
    int32_t base = 0;
    if (ok && lane == head) base = atomicAdd(cursor + x, len);
    base = __shfl_sync(FULL, base, head);
    if (ok) py[base + (lane - head)] = xu ? v : u;
}

__global__ void pair_scatter_kernel(const CountParams P, int32_t* cursor, const unsigned long long* n_pairs,
                                    int32_t* py) {
    if (*n_pairs == 0) return;  // grid-uniform
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    if (P.chunk_start) {  // batched: the chunks of the graphs with grouped pairs
        const int64_t n = *P.n_chunks_dev;
        for (int64_t c = warp; c < n; c += warps) {
            if (!P.graph_hub[__ldg(P.chunk_graph + c)]) continue;
            const int64_t e0 = __ldg(P.chunk_start + c);
            const int32_t len = __ldg(P.chunk_len + c);
            for (int32_t i = 0; i < len; i += 32)
                scatter_step(P, e0 + i + lane, __ldg(P.codes + (e0 >> 5) + c + (i >> 5)), cursor, py, lane);
        }
        return;
    }
    const int64_t steps = (P.n_edges + 31) >> 5;
    for (int64_t w = warp; w < steps; w += warps)
        scatter_step(P, 32 * w + lane, __ldg(P.codes + w), cursor, py, lane);
}

// Warp-cooperative binary-search intersection count of two sorted lists in
// global memory (tables too large for a warp).  Per-lane partial counts.
__device__ __forceinline__ uint32_t warp_bsearch_count(const int32_t* a, int la, const int32_t* b, int lb, int lane) {
    if (la > lb) {
        const int32_t* t = a;
        a = b;
        b = t;
        const int tl = la;
        la = lb;
        lb = tl;
    }
    uint32_t c = 0;
    for (int i = lane; i < la; i += 32) {
        const int32_t x = __ldg(a + i);
        int lo = 0, hi = lb;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(b + mid) < x) lo = mid + 1; else hi = mid;
        }
        c += (lo < lb && __ldg(b + lo) == x);
    }
    return c;
}

__device__ __forceinline__ uint32_t lane_merge_count(const int32_t* a, int la, const int32_t* b, int lb) {
    int i = 0, j = 0;
    uint32_t c = 0;
    while (i < la && j < lb) {
        const int32_t x = __ldg(a + i), y = __ldg(b + j);
        c += (x == y);
        i += (x <= y);
        j += (y <= x);
    }
    return c;
}

// Warp-reduces the per-lane totals and adds them to *R (lane 0, integer
// atomics; order-independent).
__device__ __forceinline__ void publish(tchll_count_result* R, uint64_t acc, U128 hacc, int64_t n_approx,
                                        int64_t n_exact, int64_t n_fallback, int64_t n_clamped, uint32_t status,
                                        int lane) {
    acc = warp_sum_u64(acc);
    hacc = warp_sum_u128(hacc);  // sub-warp HLL groups each hold their own sum
    n_approx = warp_sum_i64(n_approx);
    n_exact = warp_sum_i64(n_exact);
    n_fallback = warp_sum_i64(n_fallback);
    n_clamped = warp_sum_i64(n_clamped);
    status = __reduce_or_sync(FULL, status);
    if (lane == 0) {
        if (acc) atomicAdd((unsigned long long*)&R->exact, (unsigned long long)acc);
        atomic_add_u128((unsigned long long*)&R->hll_fx_lo, hacc);
        if (n_approx) atomicAdd((unsigned long long*)&R->n_approx, (unsigned long long)n_approx);
        if (n_exact) atomicAdd((unsigned long long*)&R->n_exact, (unsigned long long)n_exact);
        if (n_fallback) atomicAdd((unsigned long long*)&R->n_fallback, (unsigned long long)n_fallback);
        if (n_clamped) atomicAdd((unsigned long long*)&R->n_clamped, (unsigned long long)n_clamped);
        if (status) atomicOr(&R->status, status);
    }
}

// What the first pass needs beforehand, in one launch: the row table
// (load_edge_rows), and everything that starts at zero.
struct Prepare {
    const int32_t* row_ptr;
    int64_t n_nodes;
    int64_t nnz;
    const int32_t* degrees;  // routing (hybrid calls, else null)
    int64_t gamma;
    const int64_t* slot;
    const uint8_t* has;
    int64_t n_rows;
    int2* rows;
    int hub;
    const int32_t* edge_u;
    const int32_t* edge_v;
    int64_t n_edges;
    unsigned long long* est;  // zeroed before
    int32_t* zero_n[2];   // n_nodes + 1 words each (or null)
    uint32_t* zero[3];    // words[i] words
    int64_t words[3];
};
__global__ void prepare_kernel(const Prepare Q) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    uint32_t est[4] = {0, 0, 0, 0};
    for (int64_t v = t0; v <= Q.n_nodes; v += step) {
        if (v < Q.n_nodes) {
            const int32_t a = __ldg(Q.row_ptr + v), b = __ldg(Q.row_ptr + v + 1);
            int2 r = make_int2(a, b);
            const bool bad = a < 0 || b < a || (int64_t)b > Q.nnz;
            if (!bad && b - a > kTableList) {
                if (Q.hub == 0 || b - a <= Q.hub) ++est[1];
                else if (b - a <= 2 * (int64_t)Q.hub) ++est[3];
            }
            if (bad) {
                r = make_int2(kRowBad, 0);
            } else if (Q.degrees) {
                const int64_t s = Q.slot ? __ldg(Q.slot + v) : (__ldg(Q.has + v) == 1 ? v : -1);
                if (s >= Q.n_rows) r = make_int2(kSlotBad, 0);
                else if (s >= 0) r.y |= (int32_t)0x80000000;
                if ((int64_t)__ldg(Q.degrees + v) >= Q.gamma) r.x |= (int32_t)0x80000000;
            }
            Q.rows[v] = r;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (Q.zero_n[i]) Q.zero_n[i][v] = 0;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        for (int64_t w = t0; w < Q.words[i]; w += step) Q.zero[i][w] = 0;
    if (t0 < kEdgeSample && t0 < Q.n_edges) {
        const int64_t e = Q.n_edges <= kEdgeSample ? t0 : t0 * Q.n_edges / kEdgeSample;
        const int32_t u = __ldg(Q.edge_u + e), v = __ldg(Q.edge_v + e);
        if ((uint32_t)u < (uint32_t)Q.n_nodes && (uint32_t)v < (uint32_t)Q.n_nodes) {
            const PairSides S = sides_of(u, v, __ldg(Q.row_ptr + u), __ldg(Q.row_ptr + u + 1), __ldg(Q.row_ptr + v),
                                         __ldg(Q.row_ptr + v + 1));
            const bool exact = !Q.degrees || min(__ldg(Q.degrees + u), __ldg(Q.degrees + v)) < Q.gamma;  // else HLL
            if (exact && is_table_pair(S, kTableList)) {
                est[0] = Q.hub == 0 || S.xl <= Q.hub;
                est[2] = Q.hub > 0 && S.xl > Q.hub && S.xl <= 2 * (int64_t)Q.hub;
            }
        }
    }
    // one atomic each per CTA
    __shared__ uint32_t sums[4][8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        est[k] = __reduce_add_sync(FULL, est[k]);
        if ((threadIdx.x & 31) == 0) sums[k][threadIdx.x >> 5] = est[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        unsigned long long t = 0;
        for (int i = 0; i < 8; ++i) t += sums[threadIdx.x][i];
        if (t) atomicAdd(Q.est + threadIdx.x, t);
    }
}

// The first pass over the edges.  Pairs with a long table side (hub pairs)
// are counted per table side in cnth, for the hub kernels, and so are table
// pairs (is_table_pair); every other pair is counted here and now, by looking
// each member of its shorter list up in the longer one by binary search.  A warp takes 32 edges at a time and deals
// their probe members to its lanes as one stream (two windows of 32 in
// flight), so lists of any length keep the lanes busy; a search touches the
// few lines of one short list, mostly in L1.  No table has to be built, so
// short-list pairs need no regrouping.  Against a per-warp hash table and
// a lane-local merge over regrouped pairs, which these replaced:
// 2,048 graphs of 88 M edges 6.1 -> 2.9 ms (exact, all launches), 49 M
// Erdos-Renyi edges 3.1 -> 1.2 ms, R-MAT 22 with its 6 M short-list pairs 1.6
// -> 1.3 ms.  Bound by instruction issue (76%, ALU 68%): no wide load or
// higher occupancy changes it.
// Edges come in chunks of P.chunk, claimed from P.work or dealt to the warps
// in turn (null), or, batched, from the chunk list (a chunk is one graph's,
// and so are its totals).
enum : int { PASS_HIST = 1, PASS_SHORT = 2 };
enum : int { GRAPH_HUB = 1, GRAPH_GROUPED = 2 };  // hub pairs; any pairs to group
constexpr int kHugeList = 1 << 25;  // 32 shorter lists of this length still add up below 2^31
// The n HLL edges of a warp's buffer go to the list.
constexpr int kHllBuf = 160;
__device__ __forceinline__ void flush_hll(const CountParams& P, const int2* buf, int n, int lane) {
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(P.hll_n, (unsigned long long)n);
    base = __shfl_sync(FULL, base, 0);
    for (int i = lane; i < n; i += 32) {
        P.hll_u[base + i] = buf[i].x;
        P.hll_v[base + i] = buf[i].y;
    }
    __syncwarp();
}

// Adds warp-uniform totals to *R.
__device__ __forceinline__ void pass_publish(tchll_count_result* R, uint64_t acc, int64_t n_exact, int64_t n_fallback,
                                             uint32_t status, int lane) {
    status = __reduce_or_sync(FULL, status);
    if (lane == 0) {
        if (acc) atomicAdd((unsigned long long*)&R->exact, (unsigned long long)acc);
        if (n_exact) atomicAdd((unsigned long long*)&R->n_exact, (unsigned long long)n_exact);
        if (n_fallback) atomicAdd((unsigned long long*)&R->n_fallback, (unsigned long long)n_fallback);
        if (status) atomicOr(&R->status, status);
    }
}

template <bool HYB, bool VEC>
__global__ void __launch_bounds__(256, 6) pair_pass_kernel(const CountParams P, int what,
                                                           int32_t* __restrict__ cnth) {
    __shared__ int4 s_list[8][32];
    __shared__ int32_t s_len[8][32];
    __shared__ int2 s_hll[HYB ? 8 : 1][HYB ? kHllBuf : 1];
    const int lane = threadIdx.x & 31;
    constexpr int UNR = 2;  // windows of 32 look-ups in flight
    int4* lst = s_list[threadIdx.x >> 5];
    int32_t* len = s_len[threadIdx.x >> 5];
    int2* hbuf = s_hll[HYB ? threadIdx.x >> 5 : 0];
    int n_hll = 0;
    const unsigned lane_le = (2u << lane) - 1u;
    const int32_t* __restrict__ col = P.col_idx;
    uint64_t acc = 0;
    int64_t n_exact = 0, n_fallback = 0;  // warp-uniform, as acc
    uint32_t status = 0;
    if (P.check_ids) validate_rows(P.row_ptr, P.n_nodes, P.nnz, col, status);
    const int32_t full_quads = (int32_t)(P.nnz >> 2);
    const Choice ch = P.est ? choose(P.est, P.n_edges, P.hub, P.hub_alt, P.graph_vbase != nullptr) : Choice{0, 0};
    const unsigned long long n_warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    unsigned long long turn = (unsigned long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    while (true) {
        uint32_t e0, e1;  // below 2^31; the loop steps up to 31 past e1
        int32_t g = -1;
        uint32_t lo_v = 0, in_v = (uint32_t)P.n_nodes;
        unsigned long long chunk;
        {
            unsigned long long c = turn;
            if (P.work) {
                if (lane == 0) c = atomicAdd(P.work, 1ull);
                c = __shfl_sync(FULL, c, 0);
            }
            turn += n_warps;
            chunk = c;
            if (P.chunk_start) {
                if ((int64_t)c >= *P.n_chunks_dev) break;
                e0 = (uint32_t)__ldg(P.chunk_start + c);
                e1 = e0 + (uint32_t)__ldg(P.chunk_len + c);
                g = __ldg(P.chunk_graph + c);
                lo_v = (uint32_t)__ldg(P.graph_vbase + g);
                in_v = (uint32_t)__ldg(P.graph_vbase + g + 1) - lo_v;
            } else {
                if ((int64_t)c * P.chunk >= P.n_edges) break;
                e0 = (uint32_t)c * (uint32_t)P.chunk;
                e1 = (uint32_t)min((int64_t)e0 + P.chunk, P.n_edges);
            }
        }
        int left = 0;  // GRAPH_*
        // the chunk's codes: no two chunks of a batch share one
        const int64_t code0 = (e0 >> 5) + (g >= 0 ? (int64_t)chunk : 0);
        for (uint32_t eb = e0; eb < e1; eb += 32) {
            const uint32_t e = eb + lane;
            int32_t u = 0, v = 0, us = 0, ue = 0, vs = 0, ve = 0;
            bool ok = e < e1, wants = false, both = false;
            if (P.rows) {
                ok = ok && load_edge_rows(P, e, u, v, us, ue, vs, ve, wants, both, status);
            } else {
                ok = ok && load_edge(P, e, u, v, us, ue, vs, ve, status);
                int32_t du, dv;
                int64_t su, sv;
                if (HYB && ok) ok = route(P, u, v, du, dv, su, sv, wants, both, status);
            }
            if (ok && ((uint32_t)u - lo_v >= in_v || (uint32_t)v - lo_v >= in_v)) {
                status |= ST_BAD_EDGE;  // an edge of another graph inside this graph's chunk
                ok = false;
            }
            if (HYB) {
                const bool hll = ok && wants && both;
                if (P.hll_u) {  // uniform; else another launch looks for the HLL edges, and counts n_fallback
                    n_fallback += __popc(__ballot_sync(FULL, ok && wants && !both));
                    // HLL edges wait in the warp's buffer: one atomic on the shared
                    // counter per 128 or so
                    const unsigned m = __ballot_sync(FULL, hll);
                    if (hll) hbuf[n_hll + __popc(m & (lane_le >> 1))] = make_int2(u, v);
                    n_hll += __popc(m);
                    if (n_hll > kHllBuf - 32) {
                        flush_hll(P, hbuf, n_hll, lane);
                        n_hll = 0;
                    }
                }
                ok = ok && !hll;
            }
            const PairSides S = sides_of(u, v, us, ue, vs, ve);
            const bool to_hub = ok && is_hub_pair(S, ch.hub);
            const bool grouped = to_hub || (ok && is_table_pair(S, ch.table));
            if (what & PASS_HIST) {
                const unsigned m = __ballot_sync(FULL, grouped), mu = __ballot_sync(FULL, S.x == u);
                if (lane == 0) P.codes[code0 + ((eb - e0) >> 5)] = make_uint2(m, mu);
                if (m) {
                    // a run of lanes with the same table side adds with one atomic
                    int head, run;
                    lane_runs(grouped ? S.x : -1 - lane, lane, head, run);
                    if (grouped && lane == head) atomicAdd(cnth + S.x, run);
                    left |= GRAPH_GROUPED | (g >= 0 && __any_sync(FULL, to_hub) ? GRAPH_HUB : 0);
                }
            }
            if (!(what & PASS_SHORT)) continue;
            const bool mine = ok && !grouped;
            n_exact += __popc(__ballot_sync(FULL, mine));
            int np = mine ? S.yl : 0;
            // lists whose lengths could overflow the stream's positions: one
            // by one (only where no hub threshold applies)
            for (unsigned huge = __ballot_sync(FULL, np > kHugeList); huge; huge &= huge - 1) {
                const int l = __ffs(huge) - 1;
                const int32_t xs = __shfl_sync(FULL, S.xs, l), xl = __shfl_sync(FULL, S.xl, l);
                const int32_t ys = __shfl_sync(FULL, S.ys, l), yl = __shfl_sync(FULL, S.yl, l);
                acc += warp_sum_u64(warp_bsearch_count(col + xs, xl, col + ys, yl, lane));
                if (lane == l) np = 0;
            }
            int incl = np;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            const int W = __shfl_sync(FULL, incl, 31);
            if (W == 0) continue;
            const int excl = incl - np;
            const unsigned ne = __ballot_sync(FULL, np > 0);
            __syncwarp();
            // {probe member of stream position 0, the table list's first unit
            // (VEC: 16-byte quad) and units, its start}, its length
            if (np > 0) {
                const int k = __popc(ne & (lane_le >> 1));
                const int q0 = VEC ? S.xs >> 2 : S.xs;
                lst[k] = make_int4(S.ys - excl, q0, VEC ? ((S.xs + S.xl - 1) >> 2) - q0 + 1 : S.xl, S.xs);
                len[k] = S.xl;
            }
            __syncwarp();
            int B = -1;  // lists that start before the window, less one
            uint32_t hits = 0;
            for (int T0 = 0; T0 < W; T0 += 32 * UNR) {
                int32_t key[UNR], at[UNR], j[UNR];
                int n[UNR], most = 0;
#pragma unroll
                for (int i = 0; i < UNR; ++i) {
                    const int Ti = T0 + 32 * i, t = Ti + lane;
                    const unsigned d = (unsigned)(excl - Ti);
                    const unsigned st = __reduce_or_sync(FULL, (np > 0 && d < 32u) ? (1u << d) : 0u);
                    j[i] = (B + __popc(st & lane_le)) & 31;
                    B += __popc(st);
                    const int4 l = lst[j[i]];
                    // lanes past the end search for their list's last member
                    key[i] = __ldg(col + l.x + min(t, W - 1));
                    at[i] = l.y;
                    n[i] = l.z;
                    most = max(most, l.z);
                }
                // at = the last unit whose first member is <= key, or the
                // first unit (a later unit's first member lies in the list)
                for (; __any_sync(FULL, most > 1); most -= most >> 1) {
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        const int half = n[i] >> 1, m = at[i] + half;
                        if (__ldg(VEC ? col + 4 * (int64_t)m : col + m) <= key[i]) at[i] = m;
                        n[i] -= half;
                    }
                }
#pragma unroll
                for (int i = 0; i < UNR; ++i) {
                    bool hit;
                    if (!VEC) {
                        hit = __ldg(col + at[i]) == key[i];
                    } else {
                        // the unit's members inside [xs, xs + length)
                        int4 q;
                        if (at[i] < full_quads) {
                            q = __ldg(reinterpret_cast<const int4*>(col) + at[i]);
                        } else {  // the array's last, partial quad
                            const int64_t m = 4 * (int64_t)at[i];
                            q.x = __ldg(col + m);
                            q.y = m + 1 < P.nnz ? __ldg(col + m + 1) : 0;
                            q.z = m + 2 < P.nnz ? __ldg(col + m + 2) : 0;
                            q.w = 0;
                        }
                        const uint32_t o = 4u * (uint32_t)at[i] - (uint32_t)lst[j[i]].w, l = (uint32_t)len[j[i]];
                        hit = (q.x == key[i] && o < l) || (q.y == key[i] && o + 1u < l) ||
                              (q.z == key[i] && o + 2u < l) || (q.w == key[i] && o + 3u < l);
                    }
                    hits += hit && T0 + 32 * i + lane < W;
                }
            }
            acc += __reduce_add_sync(FULL, hits);
        }
        if (g >= 0) {  // batched: this chunk's totals belong to its graph
            if (left && lane == 0 && (__ldcg(P.graph_hub + g) & left) != left) atomicOr(P.graph_hub + g, left);
            pass_publish(P.result + g, acc, n_exact, n_fallback, status, lane);
            acc = 0;
            n_exact = n_fallback = 0;
            status = 0;
        }
    }
    if (HYB && n_hll) flush_hll(P, hbuf, n_hll, lane);
    if (!P.chunk_start || status) pass_publish(P.result, acc, n_exact, n_fallback, status, lane);
}

// SEGS: the pairs of P's segments instead of edges, claimed kSegPart at a time:
// the first part of every segment, then the second, and so on, so that the
// last claims are short (a whole segment takes a warp tens of microseconds:
// R-MAT 17 388 us by parts, 596 by eight segments at a time).  Where there are
// many segments they are claimed whole, which builds each table once.
constexpr int kTableSeg = 256;  // pairs of a segment at most
constexpr int kSegPart = 64;
template <int MODE, bool VEC, bool DETAILS, bool SEGS = false>
__global__ void __launch_bounds__(256, 4) count_kernel(const CountParams P) {
    extern __shared__ __align__(16) int32_t smem[];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int cap_lg = P.slots_log2;
    const int cap_keys = 1 << (cap_lg - 1);  // load <= 1/2 in 2^cap_lg slots
    uint32_t* table = reinterpret_cast<uint32_t*>(smem) + ((size_t)wid << cap_lg);

    const int32_t* __restrict__ col_idx = P.col_idx;
    const int64_t n_edges = P.n_edges;

    uint64_t acc = 0;
    U128 hacc;
    int64_t n_approx = 0, n_exact = 0, n_fallback = 0, n_clamped = 0;
    uint32_t status = 0;
    int cur_u = -1;
    int cur_lg = 5;  // log2 slots of the current table
    const int m = 1 << P.p;

    if (SEGS && *P.n_segs == 0) return;  // grid-uniform
    if (P.check_ids) validate_rows(P.row_ptr, P.n_nodes, P.nnz, col_idx, status);
    const unsigned long long n_warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    unsigned long long turn = (unsigned long long)blockIdx.x * (blockDim.x >> 5) + wid;
    int32_t seg_x = 0, seg_graph = -1;
    while (true) {
        unsigned long long e0 = 0;
        int64_t e1;
        int32_t gcur = -1;
        if (SEGS) {
            const unsigned long long n = *P.n_segs;
            const int part_len = n > 16384 ? kTableSeg : kSegPart;
            unsigned long long part = 0;
            if (lane == 0) part = atomicAdd(P.work, 1ull);
            part = __shfl_sync(FULL, part, 0);
            if (part >= n * (unsigned)(kTableSeg / part_len)) break;
            const int4 s = __ldg(reinterpret_cast<const int4*>(P.segs_end) - 1 - (int64_t)(part % n));
            const int32_t first = (int32_t)(part / n) * part_len;
            if (first >= s.z) continue;
            e0 = (unsigned long long)(s.x + first);
            seg_x = s.y;
            e1 = (int64_t)e0 + min(part_len, s.z - first);
            if (P.graph_vbase && s.w != seg_graph) {  // batched: the totals so far belong to another graph
                if (seg_graph >= 0)
                    publish(P.result + seg_graph, acc, hacc, n_approx, n_exact, n_fallback, n_clamped, status, lane);
                acc = 0;
                n_exact = 0;
                seg_graph = s.w;
            }
        } else if (P.chunk_start) {
            unsigned long long ci = 0;
            if (lane == 0) ci = atomicAdd(P.work, 1ull);
            ci = __shfl_sync(FULL, ci, 0);
            if ((int64_t)ci >= *P.n_chunks_dev) break;
            e0 = (unsigned long long)__ldg(P.chunk_start + ci);
            e1 = (int64_t)e0 + __ldg(P.chunk_len + ci);
            gcur = __ldg(P.chunk_graph + ci);
        } else {
            if (P.work) {
                if (lane == 0) e0 = atomicAdd(P.work, (unsigned long long)P.chunk);
                e0 = __shfl_sync(FULL, e0, 0);
            } else {
                e0 = turn * (unsigned long long)P.chunk;
                turn += n_warps;
            }
            if (e0 >= (unsigned long long)n_edges) break;
            e1 = min((int64_t)e0 + P.chunk, n_edges);
        }
        for (int64_t eb = (int64_t)e0; eb < e1; eb += 32) {
            const int64_t e = eb + lane;
            int32_t u = 0, v = 0, us = 0, ue = 0, vs = 0, ve = 0;
            bool valid = e < e1;
            if (SEGS) {
                if (valid) {  // the first pass has checked both rows
                    u = seg_x;
                    v = __ldcs(P.edge_v + e);
                    const int2 ru = __ldg(P.rows + u), rv = __ldg(P.rows + v);
                    us = ru.x & 0x7FFFFFFF, ue = ru.y & 0x7FFFFFFF;
                    vs = rv.x & 0x7FFFFFFF, ve = rv.y & 0x7FFFFFFF;
                }
            } else {
                valid = valid && load_edge(P, e, u, v, us, ue, vs, ve, status);
            }
            if (valid && gcur >= 0) {
                // an edge of another graph inside this graph's chunk
                const int32_t lo_v = __ldg(P.graph_vbase + gcur), hi_v = __ldg(P.graph_vbase + gcur + 1);
                if (u < lo_v || u >= hi_v || v < lo_v || v >= hi_v) {
                    status |= ST_BAD_EDGE;
                    valid = false;
                }
            }
            bool is_hll = false;
            int64_t slot_u = -1, slot_v = -1;
            int32_t du = 0, dv = 0;
            if (MODE != MODE_EXACT && valid) {
                bool wants, both;
                valid = route(P, u, v, du, dv, slot_u, slot_v, wants, both, status);
                is_hll = valid && wants && both;
                // n_fallback: counted by the fused launch and, in split mode,
                // by the HLL launch (which sees every edge in both variants)
                // or, when the HLL edges are listed here, by this one
                if ((MODE != MODE_HYB_EXACT || P.hll_u) && valid && wants && !both) ++n_fallback;
            }
            if (MODE == MODE_HYB_EXACT && P.hll_u) append_hll(P, is_hll, u, v, lane);
            const bool do_exact = valid && !is_hll && MODE != MODE_HYB_HLL;
            const bool do_hll = valid && is_hll && MODE != MODE_HYB_EXACT;
            n_exact += do_exact;

            // ---------------------------------------------------- exact part
            const int lu = ue - us, lv = ve - vs;
            const bool tiny = do_exact && (lu + lv <= P.tiny || lu == 0 || lv == 0);
            if (tiny) {
                const uint32_t c = (lu && lv) ? lane_merge_count(col_idx + us, lu, col_idx + vs, lv) : 0u;
                acc += c;
                if (DETAILS) P.pe_support[e] = c;
            }
            unsigned pend = __ballot_sync(FULL, do_exact && !tiny);
            while (pend) {
                const int lead = __ffs(pend) - 1;
                const int32_t ucur = __shfl_sync(FULL, u, lead);
                const unsigned grp = __ballot_sync(FULL, ((pend >> lane) & 1u) && u == ucur);
                pend &= ~grp;
                const int32_t gus = __shfl_sync(FULL, us, lead);
                const int32_t gdu = __shfl_sync(FULL, lu, lead);
                const bool in = (grp >> lane) & 1u;
                if (gdu > cap_keys) {
                    // table side too long for a warp table: binary search per edge
                    unsigned g = grp;
                    while (g) {
                        const int j = __ffs(g) - 1;
                        g &= g - 1;
                        const int32_t jvs = __shfl_sync(FULL, vs, j);
                        const int32_t jlv = __shfl_sync(FULL, lv, j);
                        const uint32_t c = warp_bsearch_count(col_idx + gus, gdu, col_idx + jvs, jlv, lane);
                        acc += c;
                        if (DETAILS) {
                            const uint32_t tot = (uint32_t)warp_sum_u64(c);
                            const int64_t ej = __shfl_sync(FULL, e, j);
                            if (lane == 0) P.pe_support[ej] = tot;
                        }
                    }
                    continue;
                }
                if (ucur != cur_u) {
                    // (re)build the warp's table for N+(ucur): 2^lgs slots,
                    // load <= 1/8 (1/16 sparse) when the capacity allows,
                    // <= 1/2 always
                    int lgs = ceil_log2_i(gdu) + (P.sparse ? 4 : 3);
                    lgs = lgs < 5 ? 5 : (lgs > cap_lg ? cap_lg : lgs);
                    const int nslots = 1 << lgs;
                    __syncwarp();
                    for (int i = lane; i < (nslots >> 2); i += 32)
                        reinterpret_cast<uint4*>(table)[i] = make_uint4(OV_KEY, OV_KEY, OV_KEY, OV_KEY);
                    __syncwarp();
                    bool ok = true;
                    for (int i = lane; i < gdu; i += 32)
                        ok &= ov_insert(table, __ldg(col_idx + gus + i), 32 - lgs, (uint32_t)nslots - 1u);
                    __syncwarp();
                    if (!__all_sync(FULL, ok)) {
                        // no free slot (cannot happen at load <= 1/2): binary search for this group
                        cur_u = -1;
                        unsigned g = grp;
                        while (g) {
                            const int j = __ffs(g) - 1;
                            g &= g - 1;
                            const int32_t jvs = __shfl_sync(FULL, vs, j);
                            const int32_t jlv = __shfl_sync(FULL, lv, j);
                            const uint32_t c = warp_bsearch_count(col_idx + gus, gdu, col_idx + jvs, jlv, lane);
                            acc += c;
                            if (DETAILS) {
                                const uint32_t tot = (uint32_t)warp_sum_u64(c);
                                const int64_t ej = __shfl_sync(FULL, e, j);
                                if (lane == 0) P.pe_support[ej] = tot;
                            }
                        }
                        continue;
                    }
                    cur_u = ucur;
                    cur_lg = lgs;
                }
                const int sh = 32 - cur_lg;
                const uint32_t tmask = (1u << cur_lg) - 1u;
                // flatten the group's probe lists into quads
                int q0, nq;
                if (VEC) {
                    q0 = vs >> 2;
                    nq = (in && ve > vs) ? ((ve - 1) >> 2) - q0 + 1 : 0;
                } else {
                    q0 = vs;
                    nq = in ? (ve - vs) : 0;
                }
                const unsigned ne = __ballot_sync(FULL, nq > 0);
                const int k = __popc(ne);
                const int src = lane < k ? (int)__fns(ne, 0, lane + 1) : lane;
                const int c_q0 = __shfl_sync(FULL, q0, src);
                int c_nq = __shfl_sync(FULL, nq, src);
                const int32_t c_vs = __shfl_sync(FULL, vs, src);
                const int32_t c_ve = __shfl_sync(FULL, ve, src);
                int64_t c_e = 0;
                if (DETAILS) c_e = __shfl_sync(FULL, e, src);
                if (lane >= k) c_nq = 0;
                int incl = c_nq;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                const int excl = incl - c_nq;
                const int W = __shfl_sync(FULL, incl, 31);
                const int qb = c_q0 - excl;
                // Windows of 32 quads; UNR windows are mapped, loaded and then
                // probed together so each lane has UNR 16-byte loads in flight.
                constexpr int UNR = VEC ? 4 : 2;
                for (int T0 = 0; T0 < W; T0 += 32 * UNR) {
                    int qd[UNR], lo[UNR], hi[UNR];
                    int64_t my_e[UNR];
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        const int Ti = T0 + 32 * i;
                        qd[i] = -1;
                        lo[i] = hi[i] = 0;
                        my_e[i] = 0;
                        if (Ti < W) {  // warp-uniform
                            const unsigned cover = __ballot_sync(FULL, lane < k && excl <= Ti && Ti < incl);
                            const int b = __ffs(cover) - 1;
                            const unsigned bit =
                                (lane < k && excl > Ti && excl < Ti + 32) ? (1u << (excl - Ti)) : 0u;
                            const unsigned B = __reduce_or_sync(FULL, bit);
                            const int j = (b + __popc(B & ((2u << lane) - 1u))) & 31;
                            const int my_qb = __shfl_sync(FULL, qb, j);
                            const int32_t my_vs = __shfl_sync(FULL, c_vs, j);
                            const int32_t my_ve = __shfl_sync(FULL, c_ve, j);
                            if (DETAILS) my_e[i] = __shfl_sync(FULL, c_e, j);
                            if (Ti + lane < W) {
                                qd[i] = my_qb + Ti + lane;
                                const int base = VEC ? qd[i] * 4 : qd[i];
                                lo[i] = my_vs - base;  // valid elements of the quad: [lo, hi)
                                hi[i] = my_ve - base;
                            }
                        }
                    }
                    int4 val[UNR];
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        val[i] = make_int4(-1, -1, -1, -1);
                        if (qd[i] >= 0) {
                            if (VEC) {
                                const int base = qd[i] * 4;
                                if ((int64_t)base + 3 < P.nnz) {
                                    val[i] = __ldg(reinterpret_cast<const int4*>(col_idx) + qd[i]);
                                } else {
                                    val[i].x = base + 0 < P.nnz ? __ldg(col_idx + base + 0) : -1;
                                    val[i].y = base + 1 < P.nnz ? __ldg(col_idx + base + 1) : -1;
                                    val[i].z = base + 2 < P.nnz ? __ldg(col_idx + base + 2) : -1;
                                    val[i].w = base + 3 < P.nnz ? __ldg(col_idx + base + 3) : -1;
                                }
                            } else {
                                val[i].x = __ldg(col_idx + qd[i]);
                            }
                        }
                    }
                    // home slots of every key first (branch-free; elements
                    // outside the pair's list probe as OV_NONE), then the
                    // rare walks of flagged homes
                    constexpr int KPQ = VEC ? 4 : 1;  // keys per quad
                    uint32_t key[KPQ * UNR];
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        // mapped quads have lo <= KPQ - 1 and hi >= 1; unmapped: lo = hi = 0
                        key[KPQ * i + 0] = (lo[i] <= 0 && hi[i] > 0) ? (uint32_t)val[i].x : OV_NONE;
                        if (VEC) {
                            key[KPQ * i + 1] = (lo[i] <= 1 && hi[i] > 1) ? (uint32_t)val[i].y : OV_NONE;
                            key[KPQ * i + 2] = (lo[i] <= 2 && hi[i] > 2) ? (uint32_t)val[i].z : OV_NONE;
                            key[KPQ * i + 3] = (lo[i] <= 3 && hi[i] > 3) ? (uint32_t)val[i].w : OV_NONE;
                        }
                    }
                    const uint32_t* T = table;
                    uint32_t cq[UNR], pend = 0;
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        cq[i] = 0;
#pragma unroll
                        for (int j = 0; j < KPQ; ++j) {
                            const int t = KPQ * i + j;
                            const uint32_t d = T[ov_h1((int32_t)key[t], sh)] ^ key[t];
                            cq[i] += (d << 1) == 0u;
                            pend |= (d > OV_FLAG ? 1u : 0u) << t;
                        }
                    }
                    if (pend) {
#pragma unroll
                        for (int i = 0; i < UNR; ++i)
#pragma unroll
                            for (int j = 0; j < KPQ; ++j)
                                if ((pend >> (KPQ * i + j)) & 1u)
                                    cq[i] += ov_walk(T, (int32_t)key[KPQ * i + j], sh, tmask);
                    }
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        acc += cq[i];
                        if (DETAILS && cq[i])
                            atomicAdd((unsigned long long*)(P.pe_support + my_e[i]), (unsigned long long)cq[i]);
                    }
                }
            }

            // ------------------------------------------------------ HLL part
            if (MODE != MODE_EXACT && MODE != MODE_HYB_EXACT) {
                unsigned hm = __ballot_sync(FULL, do_hll);
                while (hm) {
                    const int j = __ffs(hm) - 1;
                    hm &= hm - 1;
                    const int64_t su = __shfl_sync(FULL, slot_u, j);
                    const int64_t sv = __shfl_sync(FULL, slot_v, j);
                    const int32_t jdu = __shfl_sync(FULL, du, j);
                    const int32_t jdv = __shfl_sync(FULL, dv, j);
                    const uint8_t* ra = P.regs + su * (int64_t)m;
                    const uint8_t* rb = P.regs + sv * (int64_t)m;
                    const double E = warp_union_estimate<VEC>(ra, rb, P.p, lane, P.variant);
                    if (lane == 0) {
                        const double s_hat = (double)((int64_t)jdu + (int64_t)jdv) - E;
                        const double upper = (double)(jdu < jdv ? jdu : jdv);
                        // max(0.0, min(s_hat, upper)) with Python's min/max
                        // argument order (src/hybrid.py:122)
                        double s_cl = (upper < s_hat) ? upper : s_hat;
                        s_cl = (s_cl > 0.0) ? s_cl : 0.0;
                        if (s_hat < 0.0 || s_hat > upper) ++n_clamped;
                        ++n_approx;
                        hacc.add((uint64_t)__double2ull_rn(s_cl * 4294967296.0));
                        if (DETAILS) {
                            const int64_t ej = eb + j;
                            P.pe_s_hat[ej] = s_hat;
                            P.pe_s_cl[ej] = s_cl;
                            P.pe_method[ej] = 1;
                        }
                    }
                }
            }
        }
        if (gcur >= 0) {  // batched: this chunk's totals belong to graph gcur
            publish(P.result + gcur, acc, hacc, n_approx, n_exact, n_fallback, n_clamped, status, lane);
            acc = 0;
            hacc = U128();
            n_approx = n_exact = n_fallback = n_clamped = 0;
            status = 0;
        }
    }

    // ---------------------------------------------------------- publish ----
    if (!P.chunk_start)
        publish(P.result + (SEGS && seg_graph >= 0 ? seg_graph : 0), acc, hacc, n_approx, n_exact, n_fallback, n_clamped,
                status, lane);
}

// ------------------------------------------------------------ hub pairs ----
// Pairs whose table side x has a long forward list (d+(x) > hub threshold)
// carry most of the probe work on skewed graphs (R-MAT scale 22: 90% of the
// sum of min(d+u, d+v) has d+(x) > 256).  They are counted one x at a time
// by a whole CTA: the CTA builds ONE table of N+(x) in shared memory at load
// <= 1/8 (up to 2^hub_lg slots) and its warps stream the probe lists of x's
// pairs through it (a per-warp table of 8 KB would hold N+(x) only at load
// up to 1/2, where the overflow walks of the one-load table grow).
struct HubParams {
    const int32_t* row_ptr;
    int64_t n_nodes;
    const int32_t* col_idx;
    int64_t nnz;
    const int32_t* hy;  // y of each hub pair, grouped by x
    const int32_t* pcol;  // padded lists in core coordinates (core_pad_kernel) or null: raw lists
    const int32_t* cidx;  // core index of each vertex, -1 outside the core (with pcol)
    const int32_t* n_core;  // device: core size C (with pcol)
    const int4* pl;         // packed lists per row (core_lists_kernel)
    const uint4* pool;      // their bitmap units
    int packed;             // packed 16-bit lists when C <= kCore16Max
    const PairSeg* segs;
    const unsigned long long* n_segs;
    int64_t max_segs;
    unsigned long long* seg_ctr;
    int hub_lg;    // log2 of the largest hash table (slots)
    int cap_bits;  // bitmap kernel: bits its shared buffer holds
    bool batched;  // publish per segment into result[segment graph]
    tchll_count_result* result;
};

// The hub core.  Every key that can match a hub table lies in the forward
// list of some table side x that has hub pairs; call the union of those
// lists the core (R-MAT scale 22: 108 K of 2.4 M vertices, because
// orientation by (degree, id) puts every long list's members among the
// highest-degree vertices).  The hub kernels work in core coordinates:
//   * cidx[w] = rank of w among the core vertices, the most popular first
//     (core_index_kernel), else -1;
//   * each probe list is rewritten in core indices, a member outside the
//     core becoming the sentinel C (the core size), which can never hit;
//   * a table side's list becomes a C-bit bitmap in shared memory (13.5 KB
//     on R-MAT scale 22), so a probe is one shift, one 4-byte shared load
//     and one funnel shift.
// Counts are unchanged: |N+(x) cap N+(y)| = |cidx(N+(x)) cap cidx(N+(y) cap
// core)| because N+(x) lies inside the core and cidx is one-to-one there.
//
// Padded probe lists: row y's list starts at element pad_start(y), a
// multiple of 4, and is followed by the sentinel up to the next multiple of
// 4, so every 16-byte quad holds only the list's keys or the sentinel and no
// probe needs a mask.  pad_start(y) = roundup4(row_ptr[y]) + 8 y leaves room
// for the padding of every row before y (at most 3 per row) without a scan.
__device__ __forceinline__ int64_t pad_start(int32_t rs, int32_t y) {
    return (((int64_t)rs + 3) & ~(int64_t)3) + 8 * (int64_t)y;
}

// The core, the w in N+(x) of the x with long lists (every x with hub pairs
// among them, and known before the first pass has run), and how popular its
// members are: a counted list adds to cnt[w], the others set bit w of `bits`;
// w is in the core when it has either.  In small graphs all are counted, in
// others every kMarkStep-th (by id): the counts only order the core, where a
// sample will do, and setting bits is cheaper than counting, except that with
// few lists all warps would queue to set the same words first.  A warp looks
// at four groups of 8 vertices from all over the range (long lists cluster at
// low ids in R-MAT graphs) and takes the long lists one by one, each lane with
// four members in flight.  The bits are read first, through L1 (they fit it,
// and the core's members recur; a stale 0 just repeats the atomic), and each
// list is started at another place: long lists begin with the same few popular
// members, and warps that all start there queue on the same L2 lines.  With
// an int flag per vertex and every list walked from its start: 316 us on
// R-MAT 18 (edge factor 24), 367 us on R-MAT 22; so: 64, 112 us.  Values
// outside [0, n_nodes) are reported, not stored.
constexpr int64_t kMarkAllEdges = 8000000;
constexpr int kMarkStep = 8;
__global__ void core_mark_kernel(const int32_t* __restrict__ row_ptr, int64_t n_nodes, int64_t nnz,
                                 const int32_t* __restrict__ col, const CountParams P, int count_all,
                                 const unsigned long long* __restrict__ n_segs, uint32_t* bits, int32_t* cnt,
                                 tchll_count_result* result) {
    if (n_segs && *n_segs == 0) return;  // grid-uniform: after the first pass, which found no hub pairs
    const int hub = choose(P.est, P.n_edges, P.hub, P.hub_alt, P.graph_vbase != nullptr).hub;
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t tiles = (n_nodes + 31) >> 5;
    uint32_t status = 0;
    for (int64_t tile = warp; tile < tiles; tile += nwarps) {
        const int64_t x = 8 * (tile + (lane >> 3) * tiles) + (lane & 7);
        int32_t rs = 0, re = 0;
        if (x < n_nodes) {
            rs = __ldg(row_ptr + x);
            re = __ldg(row_ptr + x + 1);
        }
        // malformed rows are reported with the lists
        unsigned todo = __ballot_sync(FULL, rs >= 0 && re >= rs && (int64_t)re <= nnz && re - rs > hub);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const int32_t s = __shfl_sync(FULL, rs, l), e = __shfl_sync(FULL, re, l);
            const uint32_t id = (uint32_t)__shfl_sync(FULL, (int32_t)x, l);
            const bool counted = count_all || id % kMarkStep == 0;
            const uint32_t parts = ((uint32_t)(e - s) + 127u) >> 7;
            uint32_t part = (id * 0x9E3779B1u >> 8) % parts;
            for (uint32_t q = 0; q < parts; ++q) {
                const int64_t i0 = (int64_t)s + 128 * (int64_t)part;
                part = part + 1 < parts ? part + 1 : 0;
                int32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int64_t i = i0 + 32 * k + lane;
                    w[k] = i < e ? __ldg(col + i) : -1;
                    if (i < e && (uint64_t)(uint32_t)w[k] >= (uint64_t)n_nodes) {
                        status |= ST_BAD_KEY;
                        w[k] = -1;
                    }
                }
                if (counted) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (w[k] >= 0) atomicAdd(cnt + w[k], 1);
                    continue;
                }
                uint32_t f[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) f[k] = w[k] >= 0 ? bits[w[k] >> 5] : ~0u;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (!((f[k] >> (w[k] & 31)) & 1u)) atomicOr(bits + (w[k] >> 5), 1u << (w[k] & 31));
            }
        }
    }
    status = __reduce_or_sync(FULL, status);
    if (lane == 0 && status) atomicOr(&result->status, status);
}

// Core indices by falling popularity: a counting sort of the core vertices
// by their count's leading four bits (256 buckets, most popular first; the
// order inside a bucket is arbitrary, and no result depends on it).  Popular
// members come first so that the low core indices, where the lists are
// dense, can be held as bitmaps (core_lists_kernel).
__device__ __forceinline__ int pop_bucket(const uint32_t* __restrict__ bits, const int32_t* cnt, int64_t w) {
    int32_t c = cnt[w];
    if (c == 0) {
        if (!((__ldg(bits + (w >> 5)) >> (w & 31)) & 1u)) return -1;  // not in the core
        c = 1;
    }
    const int e = 31 - __clz(c);
    return 255 - (8 * e + (int)((((int64_t)c << 3) >> e) & 7));
}

__global__ void __launch_bounds__(256) core_bucket_kernel(const uint32_t* __restrict__ bits,
                                                          const int32_t* __restrict__ cnt, int64_t n_nodes,
                                                          const unsigned long long* __restrict__ n_segs,
                                                          int32_t* hist) {
    __shared__ int h[256];
    if (n_segs && *n_segs == 0) return;  // grid-uniform, as core_mark_kernel
    h[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t w = blockIdx.x * 256ll + threadIdx.x; w < n_nodes; w += gridDim.x * 256ll) {
        const int b = pop_bucket(bits, cnt, w);
        if (b >= 0) atomicAdd(h + b, 1);
    }
    __syncthreads();
    if (h[threadIdx.x]) atomicAdd(hist + threadIdx.x, h[threadIdx.x]);
}

// cnt_cidx[w]: count -> core index (-1 outside the core); n_core[0] = C.
// A CTA takes a contiguous range of vertices and claims its share of every
// bucket with one atomic (cursor: 256 zeroed words).
__global__ void __launch_bounds__(256) core_index_kernel(const uint32_t* __restrict__ bits, int32_t* cnt_cidx,
                                                         int64_t n_nodes,
                                                         const int32_t* __restrict__ hist, int32_t* cursor,
                                                         const unsigned long long* __restrict__ n_segs,
                                                         int32_t* n_core) {
    __shared__ int h[256], part[8];
    if (n_segs && *n_segs == 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t per = (n_nodes + gridDim.x - 1) / gridDim.x;
    const int64_t lo = blockIdx.x * per, hi = min(n_nodes, lo + per);
    h[tid] = 0;
    __syncthreads();
    for (int64_t w = lo + tid; w < hi; w += 256) {
        const int b = pop_bucket(bits, cnt_cidx, w);
        if (b >= 0) atomicAdd(h + b, 1);
    }
    // exclusive scan of the 256 bucket sizes
    const int mine = __ldg(hist + tid);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) part[tid >> 5] = incl;
    __syncthreads();
    int before = 0;
    for (int i = 0; i < (tid >> 5); ++i) before += part[i];
    const int n_here = h[tid];
    const int base = before + incl - mine + (n_here ? atomicAdd(cursor + tid, n_here) : 0);
    if (blockIdx.x == 0 && tid == 255) n_core[0] = before + incl;
    __syncthreads();
    h[tid] = base;
    __syncthreads();
    for (int64_t w = lo + tid; w < hi; w += 256) {
        const int b = pop_bucket(bits, cnt_cidx, w);
        cnt_cidx[w] = b >= 0 ? atomicAdd(h + b, 1) : -1;
    }
}

// Batched counts: a CTA per graph numbers that graph's core on its own (two
// lists of a pair are the same graph's), so a batch's many small cores fit
// the packed lists whatever their sum; C is the largest graph's.  A CTA takes
// about 2 us per 1024 vertices, so graphs from kBigGraph on are numbered by many
// (R-MAT 22 as a batch of one: 12.6 ms by one CTA, 8.7 so).
constexpr int32_t kBigShift = 15;
constexpr int32_t kBigGraph = 1 << kBigShift;
constexpr int32_t kBigTile = 4096;
__global__ void __launch_bounds__(1024) core_index_batch_kernel(const uint32_t* __restrict__ bits, int32_t* cnt_cidx,
                                                                int64_t n_nodes, const int32_t* __restrict__ vbase,
                                                                const int32_t* __restrict__ graph_hub,
                                                                int32_t* live_flag, int32_t* live_list,
                                                                int32_t* n_live, int32_t* n_core) {
    __shared__ int h[256], part[8];
    if ((graph_hub[blockIdx.x] & GRAPH_HUB) == 0) return;  // no core
    const int tid = threadIdx.x, lane = tid & 31;
    const int32_t lo = __ldg(vbase + blockIdx.x), hi = __ldg(vbase + blockIdx.x + 1);
    if (lo < 0 || hi < lo || (int64_t)hi > n_nodes) return;  // flagged by check_vbase_kernel
    if (hi - lo >= kBigGraph) return;                        // core_index_big_kernel
    if (tid < 256) h[tid] = 0;
    __syncthreads();
    for (int32_t w = lo + tid; w < hi; w += 1024) {
        const int b = pop_bucket(bits, cnt_cidx, w);
        if (b >= 0) atomicAdd(h + b, 1);
        if (((w & 63) == 0 || w == lo) && atomicExch(live_flag + (w >> 6), 1) == 0)
            live_list[atomicAdd(n_live, 1)] = w >> 6;
    }
    __syncthreads();
    int mine = 0, incl = 0;
    if (tid < 256) {
        incl = mine = h[tid];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) part[tid >> 5] = incl;
    }
    __syncthreads();
    if (tid < 256) {
        for (int i = 0; i < (tid >> 5); ++i) incl += part[i];
        h[tid] = incl - mine;
        if (tid == 255 && incl) atomicMax(n_core, incl);
    }
    __syncthreads();
    for (int32_t w = lo + tid; w < hi; w += 1024) {
        const int b = pop_bucket(bits, cnt_cidx, w);
        cnt_cidx[w] = b >= 0 ? atomicAdd(h + b, 1) : -1;
    }
}

// The big graphs of a batch: a CTA per kBigTile vertices.  The graphs there
// that are big are those of the tile's first and last vertex at most.  A big
// graph's bucket sizes and cursors are in big_hist, at the slot that its first
// vertex gives it (no two big graphs begin within kBigGraph vertices).
template <class F>
__device__ __forceinline__ void for_big_graphs(const CountParams& P, F f) {
    const int64_t lo = blockIdx.x * (int64_t)kBigTile, hi = min(P.n_nodes, lo + kBigTile);
    const int32_t* __restrict__ vbase = P.graph_vbase;
    const int64_t good = P.n_graphs - (int64_t)*P.graph_bad;
    int64_t last = -1;
    for (int k = 0; k < 2; ++k) {  // CTA-uniform
        const int64_t g = graph_of(vbase, P.n_graphs, P.graph_bad, (int32_t)(k == 0 ? lo : hi - 1));
        if (g == last || g >= good) continue;
        last = g;
        const int64_t a = __ldg(vbase + g), b = __ldg(vbase + g + 1);
        if (b - a < kBigGraph || (P.graph_hub[g] & GRAPH_HUB) == 0) continue;
        f(max(a, lo), min(b, hi), a, P.big_hist + 512 * (a >> kBigShift));
    }
}

__global__ void __launch_bounds__(256) core_bucket_big_kernel(const uint32_t* __restrict__ bits,
                                                              const int32_t* __restrict__ cnt, const CountParams P,
                                                              const unsigned long long* __restrict__ n_segs) {
    __shared__ int h[256];
    if (*n_segs == 0 || P.est[5] == 0) return;  // grid-uniform: no big graph
    const int tid = threadIdx.x;
    for_big_graphs(P, [&](int64_t a, int64_t b, int64_t first, int32_t* hist) {
        h[tid] = 0;
        __syncthreads();
        for (int64_t w = a + tid; w < b; w += 256) {
            const int k = pop_bucket(bits, cnt, w);
            if (k >= 0) atomicAdd(h + k, 1);
            if (((w & 63) == 0 || w == first) && atomicExch(P.live_flag + (w >> 6), 1) == 0)
                P.live_list[atomicAdd(P.n_live, 1)] = (int32_t)(w >> 6);
        }
        __syncthreads();
        if (h[tid]) atomicAdd(hist + tid, h[tid]);
        __syncthreads();
    });
}

__global__ void __launch_bounds__(256) core_index_big_kernel(const uint32_t* __restrict__ bits, int32_t* cnt_cidx,
                                                             const CountParams P,
                                                             const unsigned long long* __restrict__ n_segs,
                                                             int32_t* n_core) {
    __shared__ int h[256], part[8];
    if (*n_segs == 0 || P.est[5] == 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    for_big_graphs(P, [&](int64_t a, int64_t b, int64_t first, int32_t* hist) {
        h[tid] = 0;
        __syncthreads();
        for (int64_t w = a + tid; w < b; w += 256) {
            const int k = pop_bucket(bits, cnt_cidx, w);
            if (k >= 0) atomicAdd(h + k, 1);
        }
        const int mine = __ldg(hist + tid);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) part[tid >> 5] = incl;
        __syncthreads();
        int before = 0;
        for (int i = 0; i < (tid >> 5); ++i) before += part[i];
        const int n_here = h[tid];
        const int base = before + incl - mine + (n_here ? atomicAdd(hist + 256 + tid, n_here) : 0);
        if (a == first && tid == 255) atomicMax(n_core, before + incl);
        __syncthreads();
        h[tid] = base;
        __syncthreads();
        for (int64_t w = a + tid; w < b; w += 256) {
            const int k = pop_bucket(bits, cnt_cidx, w);
            cnt_cidx[w] = k >= 0 ? atomicAdd(h + k, 1) : -1;
        }
        __syncthreads();
    });
}

// Packed probe lists (used when C <= kCore16Max; core_pad_kernel writes the
// 32-bit ones otherwise).  A row is held as
//   * a bitmap of the core indices below 128 B: B 16-byte units, unit b the
//     indices [128 b, 128 b + 128) (from a pool, units claimed with one atomic
//     per row; B = 0 when the pool is used up);
//   * its other core indices as 16-bit keys in two planes, plane 0 the
//     indices below kPlane, plane 1 the others minus kPlane, each plane padded
//     to 16-byte units of 8 keys with 0xFFFF.  In the hub kernel's bitmap,
//     core index c sits at bit c (plane 0) or c + 1 (plane 1), so bit 65535
//     (plane 0's padding) and bit 131071 (plane 1's) are never set; that
//     works while C <= kCore16Max.
// Members outside the core are dropped: they cannot match.  Row y's keys
// start at uint16 index pad16_start(y) = roundup8(row_ptr[y]) + 24 y, which
// leaves room for both planes' padding (at most 7 each) of every row before
// y; pl[y] = {pad16_start(y) / 8, plane-0 units, first bitmap unit,
// B | plane-1 units << 8}, one 16-byte record, so that the hub kernel finds a
// pair's list with one load.
//
// Why bitmaps: a key costs a random 4-byte shared load (3.8 wavefronts per
// 32), a bitmap unit one conflict-free 16-byte one for 128 columns; ordered
// by popularity, the low columns are dense enough for that on every skewed
// graph (R-MAT 22: 58 M hub pairs probe 11.5 G keys = 1.49 G key units;
// with bitmaps 0.29 G bitmap + 0.81 G key units).  B is one of a few
// sizes up to 32, chosen per row by kUnitCost per bitmap unit against kKeyCost per
// unit of 8 keys.  The L1 pipe alone would put the ratio at 0.35, but the
// list loads weigh in: hub kernel on R-MAT 22 with 8, 11, 14, 18, 24, 30 to 34:
// 6.57, 6.31, 5.65, 5.36, 5.46, 5.47 ms (keys only: 7.29 ms).
constexpr int32_t kPlane = 65535;
constexpr int kBmSteps = 8;
constexpr int kBmMax = 32;  // units of the longest bitmap
__device__ __forceinline__ constexpr int bm_units(int k) {  // the B a row chooses from (and 0)
    return k < 4 ? 1 << k : (k & 1 ? 1 << (k / 2 + 2) : 3 << (k / 2));
}
static_assert(bm_units(3) == 8 && bm_units(4) == 12 && bm_units(5) == 16 && bm_units(6) == 24 && bm_units(7) == kBmMax);
constexpr int kUnitCost = 18;   // hub kernel cost of a bitmap unit : of a key unit
constexpr int kKeyCost = 34;
constexpr int kStage = 512;     // core indices of a row staged in shared memory (longer rows gather twice)

__device__ __forceinline__ int64_t pad16_start(int32_t rs, int32_t y) {
    return (((int64_t)rs + 7) & ~(int64_t)7) + 24 * (int64_t)y;
}

// Core index of row member i, or -1 (outside the core, or not a vertex).
__device__ __forceinline__ int32_t core_of(const int32_t* __restrict__ col, const int32_t* __restrict__ cidx,
                                           int64_t n_nodes, int64_t i, uint32_t& status) {
    const int32_t w = __ldg(col + i);
    if ((uint64_t)(uint32_t)w >= (uint64_t)n_nodes) {
        status |= ST_BAD_KEY;
        return -1;
    }
    return __ldg(cidx + w);
}

// One row by a whole warp; stage and bits are the warp's shared memory.
__device__ __forceinline__ void core_list_warp(const int32_t* __restrict__ col, const int32_t* __restrict__ cidx,
                                               int64_t n_nodes, int32_t rs, int32_t d, int32_t y,
                                               uint16_t* __restrict__ pcol16, int4* __restrict__ pl,
                                               uint4* __restrict__ pool, int32_t pool_cap, int32_t* pool_used,
                                               int32_t* stage, uint32_t* bits, uint32_t& status) {
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    int lt[kBmSteps], n_all = 0, n_hi = 0;
#pragma unroll
    for (int k = 0; k < kBmSteps; ++k) lt[k] = 0;
    for (int32_t i0 = 0; i0 < d; i0 += 128) {
        int32_t c[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int32_t i = i0 + 32 * t + lane;
            c[t] = i < d ? core_of(col, cidx, n_nodes, (int64_t)rs + i, status) : -1;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int32_t i = i0 + 32 * t + lane;
            if (i < kStage) stage[i] = c[t];
            n_all += __popc(__ballot_sync(FULL, c[t] >= 0));
            n_hi += __popc(__ballot_sync(FULL, c[t] >= kPlane));
#pragma unroll
            for (int k = 0; k < kBmSteps; ++k) lt[k] += __popc(__ballot_sync(FULL, (uint32_t)c[t] < 128u * bm_units(k)));
        }
    }
    const int n_lo = n_all - n_hi, u_hi = (n_hi + 7) >> 3;
    int B = 0, in_bits = 0, best = kKeyCost * ((n_lo + 7) >> 3);
#pragma unroll
    for (int k = 0; k < kBmSteps; ++k) {
        const int cost = kUnitCost * bm_units(k) + kKeyCost * ((n_lo - lt[k] + 7) >> 3);
        if (cost < best) {
            best = cost;
            B = bm_units(k);
            in_bits = lt[k];
        }
    }
    int32_t first = 0;
    if (B) {
        if (lane == 0) first = atomicAdd(pool_used, B);
        first = __shfl_sync(FULL, first, 0);
        if (first < 0 || first > pool_cap - B) B = 0;
    }
    uint16_t* out = pcol16 + pad16_start(rs, y);
    while (true) {
        if (B == 0) in_bits = 0;
        const int keys_lo = n_lo - in_bits, u_lo = (keys_lo + 7) >> 3;
        __syncwarp();
        for (int i = lane; i < 4 * B; i += 32) bits[i] = 0u;
        __syncwarp();
        int p0 = 0, p1 = 8 * u_lo;
        for (int32_t i0 = 0; i0 < d; i0 += 32) {
            const int32_t i = i0 + lane;
            int32_t c = -1;
            if (i < d) c = i < kStage ? stage[i] : core_of(col, cidx, n_nodes, (int64_t)rs + i, status);
            const bool in = (uint32_t)c < 128u * (uint32_t)B;
            if (in) atomicOr(bits + (c >> 5), 1u << (c & 31));
            const bool lo = c >= 0 && c < kPlane && !in, hi = c >= kPlane;
            const unsigned mlo = __ballot_sync(FULL, lo), mhi = __ballot_sync(FULL, hi);
            if (lo) out[p0 + __popc(mlo & lt_mask)] = (uint16_t)c;
            if (hi) out[p1 + __popc(mhi & lt_mask)] = (uint16_t)(c - kPlane);
            p0 += __popc(mlo);
            p1 += __popc(mhi);
        }
        if (p0 + lane < 8 * u_lo) out[p0 + lane] = 0xFFFFu;
        if (p1 + lane < 8 * (u_lo + u_hi)) out[p1 + lane] = 0xFFFFu;
        __syncwarp();
        int set = 0;
        for (int i = lane; i < B; i += 32) {
            const uint4 q = reinterpret_cast<const uint4*>(bits)[i];
            pool[first + i] = q;
            set += __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w);
        }
        // a row that lists a member twice keeps both as keys
        if (B && (int)__reduce_add_sync(FULL, (unsigned)set) != in_bits) {
            B = 0;
            continue;
        }
        if (u_hi >= (1 << 23)) {  // a row of over 2^26 repeated members
            status |= ST_BAD_ROW;
            if (lane == 0) pl[y] = make_int4(0, 0, 0, 0);
        } else if (lane == 0) {
            pl[y] = make_int4((int32_t)(pad16_start(rs, y) >> 3), u_lo, first, B | (u_hi << 8));
        }
        return;
    }
}

// A warp claims eight rows at a time: rows of at least 32 members one by one
// (core_list_warp), the others four at a time, eight lanes each, as keys only.
__global__ void __launch_bounds__(256, 6) core_lists_kernel(const int32_t* __restrict__ row_ptr, int64_t n_nodes,
                                                         int64_t nnz, const int32_t* __restrict__ col,
                                                         const int32_t* __restrict__ cidx,
                                                         const int32_t* __restrict__ n_core, int packed,
                                                         uint16_t* __restrict__ pcol16, int4* __restrict__ pl,
                                                         uint4* __restrict__ pool, int32_t pool_cap,
                                                         int32_t* pool_used, unsigned long long* row_ctr,
                                                         const unsigned long long* __restrict__ n_segs,
                                                         const int32_t* __restrict__ live,
                                                         const int32_t* __restrict__ n_live, int checked,
                                                         tchll_count_result* result) {
    __shared__ int32_t s_stage[8][kStage];
    __shared__ __align__(16) uint32_t s_bits[8][4 * kBmMax];
    if (!packed || n_core[0] > kCore16Max) return;  // grid-uniform: the 32-bit lists apply
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int sub = lane & 7, grp = lane >> 3;
    uint32_t status = 0;
    // grid-uniform; else no hub pair will read a list
    const bool lists = n_segs ? *n_segs > 0 : n_core[0] > 0;
    if (!lists && !checked) validate_rows(row_ptr, n_nodes, nnz, col, status);
    // batched: only the listed blocks of 64 rows, those near a graph with hub
    // pairs, are ever read as lists; the other rows are only checked
    if (lists && live) validate_rows(row_ptr, n_nodes, nnz, col, status);
    const unsigned long long n_claim = live ? 64ull * (unsigned)*n_live : (unsigned long long)n_nodes;
    while (lists) {
        unsigned long long y0 = 0;
        if (lane == 0) y0 = atomicAdd(row_ctr, 8ull);
        y0 = __shfl_sync(FULL, y0, 0);
        if (y0 >= n_claim) break;
        if (live) y0 = 64ull * (unsigned)__ldg(live + (y0 >> 6)) + (y0 & 63);
        int32_t rs = 0, d = 0;
        if (lane < 8 && (int64_t)y0 + lane < n_nodes) {
            const int64_t y = (int64_t)y0 + lane;
            const int32_t a = __ldg(row_ptr + y), b = __ldg(row_ptr + y + 1);
            if (a < 0 || b < a || (int64_t)b > nnz) status |= ST_BAD_ROW;  // an empty list
            else rs = a, d = b - a;
        }
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            const int32_t grs = __shfl_sync(FULL, rs, h + grp), gd = __shfl_sync(FULL, d, h + grp);
            const int64_t y = (int64_t)y0 + h + grp;
            const bool mine = gd < 32 && y < n_nodes;
            int32_t c[4];
            int n_lo = 0, n_hi = 0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int32_t i = 8 * t + sub;
                c[t] = mine && i < gd ? core_of(col, cidx, n_nodes, (int64_t)grs + i, status) : -1;
            }
            unsigned mlo[4], mhi[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                mlo[t] = (__ballot_sync(FULL, c[t] >= 0 && c[t] < kPlane) >> (8 * grp)) & 0xFFu;
                mhi[t] = (__ballot_sync(FULL, c[t] >= kPlane) >> (8 * grp)) & 0xFFu;
                n_lo += __popc(mlo[t]);
                n_hi += __popc(mhi[t]);
            }
            if (!mine) continue;
            const int u_lo = (n_lo + 7) >> 3, u_hi = (n_hi + 7) >> 3;
            const int64_t ps = pad16_start(grs, (int32_t)y);
            uint16_t* out = pcol16 + ps;
            const unsigned below = (1u << sub) - 1u;
            int p0 = 0, p1 = 8 * u_lo;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if ((mlo[t] >> sub) & 1u) out[p0 + __popc(mlo[t] & below)] = (uint16_t)c[t];
                if ((mhi[t] >> sub) & 1u) out[p1 + __popc(mhi[t] & below)] = (uint16_t)(c[t] - kPlane);
                p0 += __popc(mlo[t]);
                p1 += __popc(mhi[t]);
            }
            if (p0 + sub < 8 * u_lo) out[p0 + sub] = 0xFFFFu;
            if (p1 + sub < 8 * (u_lo + u_hi)) out[p1 + sub] = 0xFFFFu;
            if (sub == 0) pl[y] = make_int4((int32_t)(ps >> 3), u_lo, 0, u_hi << 8);
        }
        unsigned big = __ballot_sync(FULL, d >= 32);
        while (big) {
            const int j = __ffs(big) - 1;
            big &= big - 1;
            core_list_warp(col, cidx, n_nodes, __shfl_sync(FULL, rs, j), __shfl_sync(FULL, d, j),
                           (int32_t)(y0 + j), pcol16, pl, pool, pool_cap, pool_used, s_stage[wid], s_bits[wid],
                           status);
        }
    }
    status = __reduce_or_sync(FULL, status);
    if (lane == 0 && status) atomicOr(&result->status, status);
}

// Probe lists in core coordinates, padded: 8 lanes per row, one 16-byte
// quad each; a member outside the core becomes the sentinel C (a bit that is
// never set: it cannot match), and so does the padding.  Rows keep their
// lengths, so a pair's probe list is [pad_start(y), + roundup4(d+(y))).
// Malformed rows are skipped with a status flag (the counting kernels flag
// them too when an edge uses them).
__global__ void core_pad_kernel(const int32_t* __restrict__ row_ptr, int64_t n_nodes, int64_t nnz,
                                const int32_t* __restrict__ col, const int32_t* __restrict__ cidx,
                                const int32_t* __restrict__ n_core, int packed, int32_t* __restrict__ pcol,
                                int checked, tchll_count_result* result) {
    const int32_t C = n_core[0];
    if (packed && C <= kCore16Max) return;  // grid-uniform: core_lists_kernel writes the lists
    const int sub = threadIdx.x & 7;
    const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
    const int64_t ng = ((int64_t)gridDim.x * blockDim.x) >> 3;
    uint32_t status = 0;
    if (C == 0 && !checked) validate_rows(row_ptr, n_nodes, nnz, col, status);  // no hub pair will read a list
    for (int64_t y = C ? g : n_nodes; y < n_nodes; y += ng) {
        const int32_t rs = __ldg(row_ptr + y), re = __ldg(row_ptr + y + 1);
        if (rs < 0 || re < rs || (int64_t)re > nnz) {
            status |= ST_BAD_ROW;
            continue;
        }
        const int32_t d = re - rs;
        const int64_t ps = pad_start(rs, (int32_t)y);  // a multiple of 4: 16-byte aligned stores
        for (int32_t i = 4 * sub; i < d; i += 32) {
            int32_t c[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c[k] = C;
                if (i + k < d) {
                    const int32_t w = __ldg(col + rs + i + k);
                    if ((uint64_t)(uint32_t)w < (uint64_t)n_nodes) {
                        const int32_t x = __ldg(cidx + w);
                        c[k] = x >= 0 ? x : C;
                    } else {
                        status |= ST_BAD_KEY;
                    }
                }
            }
            *reinterpret_cast<int4*>(pcol + ps + i) = make_int4(c[0], c[1], c[2], c[3]);
        }
    }
    status = __reduce_or_sync(FULL, status);
    if ((threadIdx.x & 31) == 0 && status) atomicOr(&result->status, status);
}

template <int UNR, bool PAD>
__global__ void __launch_bounds__(256, 5) hub_count_kernel(const HubParams H) {
    extern __shared__ __align__(16) uint32_t tbl[];
    __shared__ PairSeg s_seg;
    __shared__ int s_round;
    __shared__ int s_fail;
    if (PAD && ((H.packed && *H.n_core <= kCore16Max) || (H.cap_bits > 0 && *H.n_core + 32 <= H.cap_bits)))
        return;  // a bitmap kernel counted every segment
    const int tid = threadIdx.x, lane = tid & 31;
    const int32_t* __restrict__ col = H.col_idx;
    const int64_t nseg = min((int64_t)*H.n_segs, H.max_segs);
    uint64_t acc = 0;
    int64_t n_pairs = 0;
    while (true) {
        if (tid == 0) {
            const unsigned long long s = atomicAdd(H.seg_ctr, 1ull);
            if ((int64_t)s < nseg) {
                s_seg = H.segs[s];
            } else {
                s_seg.x = -1;
                s_seg.len = 0;
                s_seg.start = 0;
            }
            s_round = 0;
            s_fail = 0;
        }
        __syncthreads();
        const PairSeg sg = s_seg;
        if (sg.x < 0) break;
        if (tid == 0) n_pairs += sg.len;
        const int32_t xs = __ldg(H.row_ptr + sg.x);
        const int xl = __ldg(H.row_ptr + sg.x + 1) - xs;
        int lgs = ceil_log2_i(xl) + 4;  // load <= 1/16 where the cap allows
        lgs = lgs < 7 ? 7 : (lgs > H.hub_lg ? H.hub_lg : lgs);
        const uint32_t mask = (1u << lgs) - 1u;
        const int sh = 32 - lgs;
        const bool fits = 2 * (int64_t)xl <= (int64_t)(1 << lgs);  // load <= 1/2
        if (fits) {
            for (int i = tid; i < (1 << lgs) / 4; i += blockDim.x)
                reinterpret_cast<uint4*>(tbl)[i] = make_uint4(OV_KEY, OV_KEY, OV_KEY, OV_KEY);
            __syncthreads();
            for (int i = tid; i < xl; i += blockDim.x) {
                int32_t key = __ldg(col + xs + i);
                if (PAD) {  // core coordinates: every member of a hub list is in the core
                    key = (uint64_t)(uint32_t)key < (uint64_t)H.n_nodes ? __ldg(H.cidx + key) : -1;
                    if (key < 0) {
                        s_fail = 1;
                        continue;
                    }
                }
                if (!ov_insert(tbl, key, sh, mask)) s_fail = 1;
            }
            __syncthreads();
        }
        const bool table = fits && !s_fail;  // CTA-uniform
        // pairs per round: up to 32, fewer for short segments so that every
        // warp of the CTA gets about two rounds
        int rsz = (sg.len + 15) >> 4;
        rsz = rsz < 4 ? 4 : (rsz > 32 ? 32 : rsz);
        while (true) {
            int r = 0;
            if (lane == 0) r = atomicAdd(&s_round, rsz);
            r = __shfl_sync(FULL, r, 0);
            if (r >= sg.len) break;
            const int np = min(rsz, sg.len - r);
            int32_t rs = 0, re = 0, vs = 0, ve = 0;
            if (lane < np) {
                const int32_t y = __ldg(H.hy + sg.start + r + lane);
                rs = __ldg(H.row_ptr + y);
                re = __ldg(H.row_ptr + y + 1);
                if (PAD) {
                    vs = (int32_t)pad_start(rs, y);
                    ve = vs + ((re - rs + 3) & ~3);
                } else {
                    vs = rs;
                    ve = re;
                }
            }
            if (!table) {  // x's list too long for the table: binary search per pair
                for (int j = 0; j < np; ++j) {
                    const int32_t jrs = __shfl_sync(FULL, rs, j);
                    const int32_t jre = __shfl_sync(FULL, re, j);
                    acc += warp_bsearch_count(col + xs, xl, col + jrs, jre - jrs, lane);
                }
                continue;
            }
            // flatten the 32 probe lists into one stream of 16-byte quads
            const int q0 = vs >> 2;
            const int nq = (lane < np && ve > vs) ? ((ve - 1) >> 2) - q0 + 1 : 0;
            const unsigned ne = __ballot_sync(FULL, nq > 0);
            const int k = __popc(ne);
            const int src = lane < k ? (int)__fns(ne, 0, lane + 1) : lane;
            const int c_q0 = __shfl_sync(FULL, q0, src);
            int c_nq = __shfl_sync(FULL, nq, src);
            const int32_t c_vs = __shfl_sync(FULL, vs, src);
            const int32_t c_ve = __shfl_sync(FULL, ve, src);
            if (lane >= k) c_nq = 0;
            int incl = c_nq;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            const int excl = incl - c_nq;
            const int W = __shfl_sync(FULL, incl, 31);
            const int qb = c_q0 - excl;
            // a lane's list: starts before its window + starts in the window
            // up to the lane - 1 (B: the window's list starts)
            const unsigned lane_le = (2u << lane) - 1u;
            int S = 0;
            for (int T0 = 0; T0 < W; T0 += 32 * UNR) {
                int qd[UNR], lo[UNR], hi[UNR];
#pragma unroll
                for (int i = 0; i < UNR; ++i) {
                    const int Ti = T0 + 32 * i;
                    qd[i] = -1;
                    lo[i] = hi[i] = 0;
                    if (Ti < W) {  // warp-uniform
                        const unsigned d = (unsigned)(excl - Ti);
                        const unsigned B = __reduce_or_sync(FULL, (lane < k && d < 32u) ? (1u << d) : 0u);
                        const int j = (S + __popc(B & lane_le) - 1) & 31;
                        S += __popc(B);
                        const int my_qb = __shfl_sync(FULL, qb, j);
                        const int32_t my_vs = __shfl_sync(FULL, c_vs, j);
                        const int32_t my_ve = __shfl_sync(FULL, c_ve, j);
                        if (Ti + lane < W) {
                            qd[i] = my_qb + Ti + lane;
                            if (!PAD) {
                                lo[i] = my_vs - qd[i] * 4;  // valid elements of the quad: [lo, hi)
                                hi[i] = my_ve - qd[i] * 4;
                            }
                        }
                    }
                }
                // Keys of all 4 * UNR quad elements.  Elements outside the
                // pair's list (quad edges, idle lanes) probe as OV_NONE,
                // which matches no slot; padded lists need no masking.
                uint32_t key[4 * UNR];
#pragma unroll
                for (int i = 0; i < UNR; ++i) {
                    if (PAD) {
                        uint4 q = make_uint4(OV_NONE, OV_NONE, OV_NONE, OV_NONE);
                        if (qd[i] >= 0) q = __ldg(reinterpret_cast<const uint4*>(H.pcol) + qd[i]);
                        key[4 * i + 0] = q.x;
                        key[4 * i + 1] = q.y;
                        key[4 * i + 2] = q.z;
                        key[4 * i + 3] = q.w;
                    } else {
                        int4 val = make_int4(-1, -1, -1, -1);
                        if (qd[i] >= 0) {
                            const int64_t base = (int64_t)qd[i] * 4;
                            if (base + 3 < H.nnz) {
                                val = __ldg(reinterpret_cast<const int4*>(col) + qd[i]);
                            } else {
                                val.x = base + 0 < H.nnz ? __ldg(col + base + 0) : -1;
                                val.y = base + 1 < H.nnz ? __ldg(col + base + 1) : -1;
                                val.z = base + 2 < H.nnz ? __ldg(col + base + 2) : -1;
                                val.w = base + 3 < H.nnz ? __ldg(col + base + 3) : -1;
                            }
                        }
                        // lo <= 3 and hi >= 1 for every mapped quad; unmapped: lo = hi = 0
                        key[4 * i + 0] = (lo[i] <= 0 && hi[i] > 0) ? (uint32_t)val.x : OV_NONE;
                        key[4 * i + 1] = (lo[i] <= 1 && hi[i] > 1) ? (uint32_t)val.y : OV_NONE;
                        key[4 * i + 2] = (lo[i] <= 2 && hi[i] > 2) ? (uint32_t)val.z : OV_NONE;
                        key[4 * i + 3] = (lo[i] <= 3 && hi[i] > 3) ? (uint32_t)val.w : OV_NONE;
                    }
                }
                // home slots first (independent loads), then the rare walks
                // of flagged homes
                uint32_t c = 0, pend = 0, pk = 0;
#pragma unroll
                for (int t = 0; t < 4 * UNR; ++t) {
                    const uint32_t d = tbl[ov_h1((int32_t)key[t], sh)] ^ key[t];
                    c += (d << 1) == 0u;                       // key bits equal
                    const bool f = d > OV_FLAG;                // flagged home, other key
                    pend |= (f ? 1u : 0u) << t;
                    pk = f ? key[t] : pk;                      // the last such key
                }
                // each lane walks its own flagged homes: usually none, else
                // one (pk); several take the general loop
                if (pend) {
                    if ((pend & (pend - 1u)) == 0u) {
                        c += ov_walk(tbl, (int32_t)pk, sh, mask);
                    } else {
                        while (pend) {
                            const int t = __ffs(pend) - 1;
                            pend &= pend - 1u;
                            uint32_t k = key[0];
#pragma unroll
                            for (int j = 1; j < 4 * UNR; ++j) k = (t == j) ? key[j] : k;
                            c += ov_walk(tbl, (int32_t)k, sh, mask);
                        }
                    }
                }
                acc += c;
            }
        }
        if (H.batched) {  // this segment's totals belong to its graph
            acc = warp_sum_u64(acc);
            if (lane == 0 && acc) atomicAdd((unsigned long long*)&H.result[sg.graph].exact, (unsigned long long)acc);
            if (tid == 0) atomicAdd((unsigned long long*)&H.result[sg.graph].n_exact, (unsigned long long)sg.len);
            acc = 0;
            n_pairs = 0;
        }
        __syncthreads();  // every warp is done with this table
    }
    if (H.batched) return;
    acc = warp_sum_u64(acc);
    n_pairs = warp_sum_i64(n_pairs);
    if (lane == 0) {
        if (acc) atomicAdd((unsigned long long*)&H.result->exact, (unsigned long long)acc);
        if (n_pairs) atomicAdd((unsigned long long*)&H.result->n_exact, (unsigned long long)n_pairs);
    }
}

// Hub pairs over a shared-memory bitmap of N+(x) in core coordinates (see
// the hub core above).  Runs only when the core fits the shared buffer
// (C + 32 <= cap_bits, decided on the device: the host never reads C);
// otherwise it returns at once and hub_count_kernel<*, true> takes the
// segments from the same counter.
//
// A CTA claims a segment, clears ceil((C + 32) / 128) uint4 words, sets the
// bits of x's list and its warps stream the segment's probe lists through
// it, up to 32 lists per round.  The round's lists are flattened into one
// stream of 16-byte quads, 32 consecutive quads per window dealt to the 32
// lanes (coalesced loads).  A lane finds its quad's list from the bitmap B
// of list starts inside its window (one OR-reduction per window): list index
// = starts before the window + starts up to the lane - 1.  Since the probe
// lists are in core coordinates and padded with the never-set bit C, a key needs no
// mask and no bound: hit = bit key of the bitmap.
template <int UNR>
__global__ void __launch_bounds__(256, 6) hub_bitmap_kernel(const HubParams H) {
    extern __shared__ __align__(16) uint32_t bm[];
    __shared__ PairSeg s_seg;
    __shared__ int s_round;
    __shared__ int s_fail;
    const int C = *H.n_core;
    if ((H.packed && C <= kCore16Max) || C + 32 > H.cap_bits) return;  // grid-uniform: another kernel counts
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned lane_le = (2u << lane) - 1u;  // lane 31: 0 - 1 = all bits
    const uint32_t sentinel = (uint32_t)C;
    const int nw4 = (C + 32 + 127) >> 7;  // uint4 words covering bits [0, C + 32)
    const int32_t* __restrict__ col = H.col_idx;
    const uint4* __restrict__ pq = reinterpret_cast<const uint4*>(H.pcol);
    const int64_t nseg = min((int64_t)*H.n_segs, H.max_segs);
    uint64_t acc = 0;
    int64_t n_pairs = 0;
    while (true) {
        if (tid == 0) {
            const unsigned long long s = atomicAdd(H.seg_ctr, 1ull);
            if ((int64_t)s < nseg) {
                s_seg = H.segs[s];
            } else {
                s_seg.x = -1;
                s_seg.len = 0;
                s_seg.start = 0;
            }
            s_round = 0;
            s_fail = 0;
        }
        for (int i = tid; i < nw4; i += blockDim.x) reinterpret_cast<uint4*>(bm)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        const PairSeg sg = s_seg;
        if (sg.x < 0) break;
        if (tid == 0) n_pairs += sg.len;
        const int32_t xs = __ldg(H.row_ptr + sg.x);
        const int xl = __ldg(H.row_ptr + sg.x + 1) - xs;
        for (int i = tid; i < xl; i += blockDim.x) {
            const int32_t w = __ldg(col + xs + i);
            const int32_t c = (uint64_t)(uint32_t)w < (uint64_t)H.n_nodes ? __ldg(H.cidx + w) : -1;
            if (c >= 0) atomicOr(bm + (c >> 5), 1u << (c & 31));
            else s_fail = 1;  // not in the core (cannot happen for well-formed input)
        }
        __syncthreads();
        const bool table = !s_fail;  // CTA-uniform
        // pairs per round: up to 32, fewer for short segments so that every
        // warp of the CTA gets about two rounds
        int rsz = (sg.len + 15) >> 4;
        rsz = rsz < 4 ? 4 : (rsz > 32 ? 32 : rsz);
        while (true) {
            int r = 0;
            if (lane == 0) r = atomicAdd(&s_round, rsz);
            r = __shfl_sync(FULL, r, 0);
            if (r >= sg.len) break;
            const int np = min(rsz, sg.len - r);
            int32_t vs = 0, nq = 0, rs = 0, re = 0;
            if (lane < np) {
                const int32_t y = __ldg(H.hy + sg.start + r + lane);
                rs = __ldg(H.row_ptr + y);
                re = __ldg(H.row_ptr + y + 1);
                vs = (int32_t)pad_start(rs, y);
                nq = (re - rs + 3) >> 2;
            }
            if (!table) {  // binary search per pair over the raw lists
                for (int j = 0; j < np; ++j) {
                    const int32_t jrs = __shfl_sync(FULL, rs, j);
                    const int32_t jre = __shfl_sync(FULL, re, j);
                    acc += warp_bsearch_count(col + xs, xl, col + jrs, jre - jrs, lane);
                }
                continue;
            }
            // the round's non-empty lists, compacted to lanes 0..k-1, and the
            // exclusive scan of their quad counts
            const unsigned ne = __ballot_sync(FULL, nq > 0);
            const int k = __popc(ne);
            const int src = lane < k ? (int)__fns(ne, 0, lane + 1) : lane;
            const int c_q0 = __shfl_sync(FULL, vs >> 2, src);
            int c_nq = __shfl_sync(FULL, nq, src);
            if (lane >= k) c_nq = 0;
            int incl = c_nq;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            const int excl = incl - c_nq;
            const int W = __shfl_sync(FULL, incl, 31);
            const int qb = c_q0 - excl;  // quad of stream position t in list j: qb[j] + t
            const bool starts = lane < k;
            int S = 0;  // list starts before the current window
            for (int T0 = 0; T0 < W; T0 += 32 * UNR) {
                int qd[UNR];
#pragma unroll
                for (int i = 0; i < UNR; ++i) {
                    const int Ti = T0 + 32 * i;
                    qd[i] = -1;
                    if (Ti < W) {  // warp-uniform
                        const unsigned d = (unsigned)(excl - Ti);
                        const unsigned B = __reduce_or_sync(FULL, (starts && d < 32u) ? (1u << d) : 0u);
                        const int j = S + __popc(B & lane_le) - 1;
                        S += __popc(B);
                        const int my_qb = __shfl_sync(FULL, qb, j & 31);
                        if (Ti + lane < W) qd[i] = my_qb + Ti + lane;
                    }
                }
                uint32_t key[4 * UNR];
#pragma unroll
                for (int i = 0; i < UNR; ++i) {
                    uint4 q = make_uint4(sentinel, sentinel, sentinel, sentinel);
                    if (qd[i] >= 0) q = __ldg(pq + qd[i]);
                    key[4 * i + 0] = q.x;
                    key[4 * i + 1] = q.y;
                    key[4 * i + 2] = q.z;
                    key[4 * i + 3] = q.w;
                }
                uint32_t c = 0;
#pragma unroll
                for (int t = 0; t < 4 * UNR; ++t) c += __funnelshift_r(bm[key[t] >> 5], 0u, key[t]) & 1u;
                acc += c;
            }
        }
        if (H.batched) {  // this segment's totals belong to its graph
            acc = warp_sum_u64(acc);
            if (lane == 0 && acc) atomicAdd((unsigned long long*)&H.result[sg.graph].exact, (unsigned long long)acc);
            if (tid == 0) atomicAdd((unsigned long long*)&H.result[sg.graph].n_exact, (unsigned long long)sg.len);
            acc = 0;
            n_pairs = 0;
        }
        __syncthreads();  // every warp is done with this bitmap
    }
    if (H.batched) return;
    acc = warp_sum_u64(acc);
    n_pairs = warp_sum_i64(n_pairs);
    if (lane == 0) {
        if (acc) atomicAdd((unsigned long long*)&H.result->exact, (unsigned long long)acc);
        if (n_pairs) atomicAdd((unsigned long long*)&H.result->n_exact, (unsigned long long)n_pairs);
    }
}

// hub_bitmap_kernel over packed lists (core_lists_kernel; C <= kCore16Max):
// a list is B bitmap units of 128 columns and units of 8 16-bit keys.  The
// CTA's bitmap of N+(x) has 65,536 bits (C <= 65535) or 131,072 bits (16 KB of
// shared memory) and is set from x's own list (16-byte loads; x's members
// are the core's by construction, so no member can miss and there is no
// binary-search fallback).  A round's lists are walked as two flattened
// streams, so that no warp mixes the two kinds: the bitmap units (one
// 16-byte list load, one 16-byte shared load of the same columns, four
// AND + popc; consecutive lanes read consecutive units, so the shared load is
// conflict-free), then the key units (eight random 4-byte shared loads; a
// unit's plane, the bitmap's half, follows from its position in the list).
// A lane finds its unit's list as in hub_bitmap_kernel; the lists' bases sit
// in a shared-memory slot per warp.  Bound by the L1 data pipe (86% busy on
// R-MAT 21, issue 64%): R-MAT 18 / 20 / 22 249 / 1189 / 7291 us with key lists
// alone, 140 / 707 / 5094 us here.
constexpr int kHub16Threads = 128;
template <int UNR>
__global__ void __launch_bounds__(kHub16Threads, 1536 / kHub16Threads) hub_bitmap16_kernel(const HubParams H) {
    extern __shared__ __align__(16) uint32_t bm[];  // 4096 words
    __shared__ PairSeg s_seg;
    __shared__ int s_round;
    __shared__ int2 s_list[kHub16Threads / 32][32];
    const int C = H.n_core[0];
    if (!H.packed || C > kCore16Max) return;  // grid-uniform: a 32-bit kernel counts
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned lane_le = (2u << lane) - 1u;
    int2* lst = s_list[tid >> 5];
    uint4* bm4 = reinterpret_cast<uint4*>(bm);
    // uint4 words that can hold a set bit (core index c: bit c or c + 1); the
    // padding's words stay clear
    const int nw4 = (C >> 7) + 1;
    if (tid < 2) bm4[512 * tid + 511] = make_uint4(0u, 0u, 0u, 0u);
    const uint4* __restrict__ pq = reinterpret_cast<const uint4*>(H.pcol);
    const int64_t nseg = min((int64_t)*H.n_segs, H.max_segs);
    uint64_t acc = 0;
    int64_t n_pairs = 0;
    while (true) {
        if (tid == 0) {
            const unsigned long long s = atomicAdd(H.seg_ctr, 1ull);
            if ((int64_t)s < nseg) {
                s_seg = H.segs[s];
            } else {
                s_seg.x = -1;
                s_seg.len = 0;
                s_seg.start = 0;
            }
            s_round = 0;
        }
        for (int i = tid; i < nw4; i += blockDim.x) bm4[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        const PairSeg sg = s_seg;
        if (sg.x < 0) break;
        if (tid == 0) n_pairs += sg.len;
        {
            // bitmap units are whole words of their own; plane-1 key k is
            // core index k + kPlane, bit k + kPlane + 1
            const int4 xr = __ldg(H.pl + sg.x);
            const int xb = xr.w & 0xFF, xk = xr.y + (xr.w >> 8);
            for (int i = tid; i < xb; i += blockDim.x) bm4[i] = __ldg(H.pool + xr.z + i);
            for (int i = tid; i < xk; i += blockDim.x) {
                const uint4 q = __ldg(pq + xr.x + i);
                const uint32_t hb = i >= xr.y ? 65536u : 0u;
                const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const uint32_t k = (w4[t >> 1] >> (16 * (t & 1))) & 0xFFFFu;
                    if (k != 0xFFFFu) atomicOr(bm + ((k + hb) >> 5), 1u << (k & 31));
                }
            }
        }
        __syncthreads();
        constexpr int kShare = kHub16Threads / 16;  // two rounds per warp
        int rsz = (sg.len + kShare - 1) / kShare;
        rsz = rsz < 4 ? 4 : (rsz > 32 ? 32 : rsz);
        while (true) {
            int r = 0;
            if (lane == 0) r = atomicAdd(&s_round, rsz);
            r = __shfl_sync(FULL, r, 0);
            if (r >= sg.len) break;
            int4 rec = make_int4(0, 0, 0, 0);
            if (lane < min(rsz, sg.len - r)) rec = __ldg(H.pl + __ldg(H.hy + sg.start + r + lane));
#pragma unroll
            for (int kind = 0; kind < 2; ++kind) {  // 0: bitmap units, 1: key units
                const int nu = kind == 0 ? (rec.w & 0xFF) : rec.y + (rec.w >> 8);
                int incl = nu;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                const int W = __shfl_sync(FULL, incl, 31);
                if (W == 0) continue;
                const int excl = incl - nu;
                // non-empty lists, in order: {unit of stream position 0, the
                // position of its first unit / of its first plane-1 unit}
                const unsigned ne = __ballot_sync(FULL, nu > 0);
                __syncwarp();
                if (nu > 0)
                    lst[__popc(ne & (lane_le >> 1))] = make_int2((kind == 0 ? rec.z : rec.x) - excl,
                                                                 kind == 0 ? excl : excl + rec.y);
                __syncwarp();
                int S = -1;
                for (int T0 = 0; T0 < W; T0 += 32 * UNR) {
                    uint4 q[UNR];
                    int at[UNR];
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        const int Ti = T0 + 32 * i, t = Ti + lane;
                        // padding keys (bit 65535, never set) / empty bitmap units
                        q[i] = kind == 0 ? make_uint4(0u, 0u, 0u, 0u) : make_uint4(~0u, ~0u, ~0u, ~0u);
                        at[i] = 0;
                        if (Ti < W) {  // warp-uniform
                            const unsigned d = (unsigned)(excl - Ti);
                            const unsigned B = __reduce_or_sync(FULL, (nu > 0 && d < 32u) ? (1u << d) : 0u);
                            const int2 l = lst[(S + __popc(B & lane_le)) & 31];
                            S += __popc(B);
                            if (t < W) {
                                q[i] = __ldcg((kind == 0 ? H.pool : pq) + (l.x + t));  // no reuse in L1
                                // the unit's columns / plane 1: the bitmap's upper half
                                at[i] = kind == 0 ? t - l.y : (t >= l.y ? 8192 : 0);
                            }
                        }
                    }
                    uint32_t c = 0;
#pragma unroll
                    for (int i = 0; i < UNR; ++i) {
                        if (i > 0 && T0 + 32 * i >= W) break;  // warp-uniform
                        if (kind == 0) {
                            const uint4 b = bm4[at[i]];
                            c += __popc(q[i].x & b.x) + __popc(q[i].y & b.y) + __popc(q[i].z & b.z) +
                                 __popc(q[i].w & b.w);
                        } else {
                            // byte offset of the key's word: (key >> 5) * 4, plus the plane's 8 KB
                            const char* b = reinterpret_cast<const char*>(bm);
                            const uint32_t pl = (uint32_t)at[i];
                            const uint32_t w4[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                const uint32_t w = w4[t];
                                const uint32_t lo = *reinterpret_cast<const uint32_t*>(b + (((w >> 3) & 0x1FFCu) | pl));
                                const uint32_t hi = *reinterpret_cast<const uint32_t*>(b + (((w >> 19) & 0x1FFCu) | pl));
                                c += (__funnelshift_r(lo, 0u, w) & 1u) + (__funnelshift_r(hi, 0u, w >> 16) & 1u);
                            }
                        }
                    }
                    acc += c;
                }
            }
        }
        if (H.batched) {  // this segment's totals belong to its graph
            acc = warp_sum_u64(acc);
            if (lane == 0 && acc) atomicAdd((unsigned long long*)&H.result[sg.graph].exact, (unsigned long long)acc);
            if (tid == 0) atomicAdd((unsigned long long*)&H.result[sg.graph].n_exact, (unsigned long long)sg.len);
            acc = 0;
            n_pairs = 0;
        }
        __syncthreads();  // every warp is done with this bitmap
    }
    if (H.batched) return;
    acc = warp_sum_u64(acc);
    n_pairs = warp_sum_i64(n_pairs);
    if (lane == 0) {
        if (acc) atomicAdd((unsigned long long*)&H.result->exact, (unsigned long long)acc);
        if (n_pairs) atomicAdd((unsigned long long*)&H.result->n_exact, (unsigned long long)n_pairs);
    }
}

// Places of the grouped pairs, and their segments: x's cnth[x] pairs get the
// range [offh[x], + cnth[x]) of the list and are cut into segments, x's next to
// each other; those of hub pairs (x's list longer than `hub`; at most hub_seg
// pairs each) fill segs from the front, those of table pairs (at most
// kTableSeg) from the back.  The order of the ranges does not matter, so a CTA
// of 1024 vertices scans its own and claims room with one atomic each for
// pairs and segments (a scan over all vertices and one atomic per x took 94 us
// on R-MAT 22).  Batched counts (vbase != null) record the graph of x, found
// by binary search in the ascending vertex offsets vbase[0..n_graphs].
struct PairRoom {
    unsigned long long* n_pairs;
    PairSeg* segs;
    int64_t max_segs;
    unsigned long long* n_hub_segs;
    unsigned long long* n_table_segs;
};
__global__ void __launch_bounds__(256) hub_alloc_kernel(const int32_t* __restrict__ cnth,
                                                        const CountParams P, int hub_seg, int32_t* __restrict__ offh,
                                                        const PairRoom R) {
    __shared__ unsigned long long warp_sum[2][8], base[3];
    const int2* __restrict__ rows = P.rows;
    const int64_t n_nodes = P.n_nodes;
    const int32_t* __restrict__ vbase = P.graph_vbase;
    const int hub = choose(P.est, P.n_edges, P.hub, P.hub_alt, vbase != nullptr).hub;
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t x0 = blockIdx.x * 1024ll + tid;
    int32_t c[4];
    bool is_hub[4];
    unsigned long long mine[2] = {0, 0};  // pairs; hub segments + table segments << 32
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t x = x0 + 256 * i;
        c[i] = x < n_nodes ? __ldg(cnth + x) : 0;
        is_hub[i] = false;
        if (c[i] > 0) {
            const int2 r = __ldg(rows + x);
            is_hub[i] = hub > 0 && (r.y & 0x7FFFFFFF) - (r.x & 0x7FFFFFFF) > hub;
            const unsigned seg = is_hub[i] ? hub_seg : kTableSeg, n = ((unsigned)c[i] + seg - 1u) / seg;
            mine[0] += (unsigned long long)c[i];
            mine[1] += is_hub[i] ? (unsigned long long)n : (unsigned long long)n << 32;
        }
    }
    if (!__syncthreads_or(mine[0] != 0)) return;  // nothing grouped here, as in most of a batch or a road network
    unsigned long long incl[2] = {mine[0], mine[1]};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned long long t = __shfl_up_sync(FULL, incl[k], o);
            if (lane >= o) incl[k] += t;
        }
    }
    if (lane == 31) {
        warp_sum[0][tid >> 5] = incl[0];
        warp_sum[1][tid >> 5] = incl[1];
    }
    __syncthreads();
    if (tid == 0) {
        unsigned long long sum[2] = {0, 0};
        for (int k = 0; k < 2; ++k)
            for (int w = 0; w < 8; ++w) {
                const unsigned long long t = warp_sum[k][w];
                warp_sum[k][w] = sum[k];
                sum[k] += t;
            }
        if (sum[0]) {
            base[0] = atomicAdd(R.n_pairs, sum[0]);
            base[1] = sum[1] & 0xFFFFFFFFull ? atomicAdd(R.n_hub_segs, sum[1] & 0xFFFFFFFFull) : 0;
            base[2] = sum[1] >> 32 ? atomicAdd(R.n_table_segs, sum[1] >> 32) : 0;
        }
    }
    __syncthreads();
    if (mine[0] == 0) return;
    int32_t at = (int32_t)(base[0] + warp_sum[0][tid >> 5] + incl[0] - mine[0]);
    const unsigned long long before = warp_sum[1][tid >> 5] + incl[1] - mine[1];
    int64_t hs = (int64_t)(base[1] + (before & 0xFFFFFFFFull));
    int64_t ts = R.max_segs - 1 - (int64_t)(base[2] + (before >> 32));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (c[i] <= 0) continue;
        const int64_t x = x0 + 256 * i;
        const int32_t g = vbase ? (int32_t)graph_of(vbase, P.n_graphs, P.graph_bad, (int32_t)x) : 0;
        offh[x] = at;
        const int seg = is_hub[i] ? hub_seg : kTableSeg;
        for (int64_t j = 0; j < c[i]; j += seg) {
            const int64_t to = is_hub[i] ? hs++ : ts--;
            if (to < 0 || to >= R.max_segs) break;  // cannot happen: sized for the worst case
            PairSeg s;
            s.start = at + (int32_t)j;
            s.x = (int32_t)x;
            s.len = min(seg, c[i] - (int32_t)j);
            s.graph = g;
            R.segs[to] = s;
        }
        at += c[i];
    }
}

// ------------------------------------------------------ HLL edge list ------
// One group of L lanes per HLL edge (L = min(32, 2^p / 16): p = 8 runs two
// edges per warp, p >= 9 a warp per edge), the group's lanes striding over
// the two 2^p-byte rows with 16-byte loads.  Pass 1 counts the zero
// registers V of the merged row (zero bytes of row_u | row_v).  Every zero
// register adds exactly 1 to Z = sum 2^-r, so V >= lc_min (the smallest V
// with alpha*m^2/V <= 2.5m, with a 1e-9 margin for the FP64 comparison) proves
// the estimator takes its linear-counting branch: E = m * ln(m / V), the same
// expression the full estimator evaluates, and Z is not needed.  Otherwise
// pass 2 forms Z exactly (128-bit fixed point) and applies the full
// estimator.
struct HllParams {
    const int32_t* hu;
    const int32_t* hv;
    const unsigned long long* n_dev;
    const int32_t* degrees;
    const uint8_t* regs;
    const int64_t* slot;  // null: dense rows (row v at v * 2^p)
    const uint32_t* zm;   // zero masks, zst words per row (null: count zeros from the registers)
    int zst;
    const double* lc;      // with zm: linear-counting estimate by zero count
    const int32_t* vbase;  // batched: per-edge results go to result[graph of u]
    int64_t n_graphs;
    const unsigned long long* graph_bad;
    int p;
    int variant;
    uint32_t lc_min;
    tchll_count_result* result;
};

// Zero-register masks: bit j of word w of row r is set iff register 32w + j
// of the row is 0.  Rows are zst >= 4 words (16-byte aligned); bits past 2^p
// stay clear.  One warp per row; dense layouts skip rows without a sketch
// (no HLL edge reads them).  lc[z] is the linear-counting estimate of z zero
// registers: the HLL pass looks it up instead of taking an FP64 logarithm per
// edge.
__global__ void __launch_bounds__(256) zmask_kernel(const uint8_t* __restrict__ regs, int64_t n_rows,
                                                    const uint8_t* __restrict__ has, int p, int zst,
                                                    uint32_t* __restrict__ zm, double* __restrict__ lc) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int m = 1 << p;
    for (int64_t z = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; z <= m; z += (int64_t)gridDim.x * blockDim.x)
        lc[z] = z > 0 ? (double)m * log((double)m / (double)z) : 0.0;
    for (int64_t r = warp; r < n_rows; r += nwarps) {
        if (has && !__ldg(has + r)) continue;
        const uint4* row = reinterpret_cast<const uint4*>(regs + r * (int64_t)m);
        for (int w = lane; w < zst; w += 32) {
            uint32_t bits = 0;
            if (32 * w < m) {
                const uint4 a = __ldg(row + 2 * w);
                bits = (__vcmpeq4(a.x, 0u) & 0x01010101u) | ((__vcmpeq4(a.y, 0u) & 0x01010101u) << 1) |
                       ((__vcmpeq4(a.z, 0u) & 0x01010101u) << 2) | ((__vcmpeq4(a.w, 0u) & 0x01010101u) << 3);
                if (32 * w + 16 < m) {
                    const uint4 b = __ldg(row + 2 * w + 1);
                    bits |= ((__vcmpeq4(b.x, 0u) & 0x01010101u) << 4) | ((__vcmpeq4(b.y, 0u) & 0x01010101u) << 5) |
                            ((__vcmpeq4(b.z, 0u) & 0x01010101u) << 6) | ((__vcmpeq4(b.w, 0u) & 0x01010101u) << 7);
                }
            }
            zm[r * (int64_t)zst + w] = bits;  // bit order is a permutation of the registers: only popc is used
        }
    }
}

__device__ __forceinline__ uint32_t zero_bytes(uint32_t w) { return __popc(__vcmpeq4(w, 0u)) >> 3; }

template <int L>
__device__ __forceinline__ uint32_t group_sum_u32(uint32_t x, unsigned gmask) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) x += __shfl_xor_sync(gmask, x, o);
    return x;
}

template <int L>
__device__ __forceinline__ U128 group_sum_u128(U128 v, unsigned gmask) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        U128 t;
        t.lo = __shfl_xor_sync(gmask, v.lo, o);
        t.hi = __shfl_xor_sync(gmask, v.hi, o);
        v.add(t);
    }
    return v;
}

// Sum of 2^-r over the merged registers, exactly, in units of 2^-S
// (S = 65 - p, so 2^-r for every valid rank r <= S is an integer there).
// Most registers hold r <= 7: for a word w of four such registers,
//   t    = bytes 2^(7 - r_i)   (one byte permute of the table 128, 64 .. 1,
//                               selected by the four ranks packed as nibbles)
//   fast += bytes of t          (dp4a with 1,1,1,1)
//   zeros += [r_i == 0]         (a second permute of the table 1,0,..,0)
// so fast * 2^(S-7) is the words' share of the sum.  A word with a register
// >= 8 goes byte by byte: r <= 7 into fast, 8 <= r <= S into fine (units of
// 2^-S, 64 bits), r > S (only in malformed rows) into extra (FP64).
__device__ __forceinline__ void hll_word_lut(uint32_t w, int S, uint32_t& fast, uint64_t& fine, uint32_t& zeros,
                                             double& extra) {
    if ((w & 0xF8F8F8F8u) == 0u) {
        const uint32_t x = w | (w >> 4);                 // byte 0: r0 | r1 << 4, byte 2: r2 | r3 << 4
        const uint32_t sel = __byte_perm(x, 0u, 0x4420u);  // nibbles r0 r1 r2 r3
        fast = __dp4a(__byte_perm(0x10204080u, 0x01020408u, sel), 0x01010101u, fast);
        zeros = __dp4a(__byte_perm(0x00000001u, 0u, sel), 0x01010101u, zeros);
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int r = (int)((w >> (8 * k)) & 0xFFu);
        if (r <= 7) {
            fast += 128u >> r;
            zeros += (r == 0);
        } else if (r <= S) {
            fine += 1ull << (S - r);
        } else {
            extra += ldexp(1.0, S - r);
        }
    }
}

template <int L>
__device__ __forceinline__ uint64_t group_sum_u64(uint64_t x, unsigned gmask) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) x += __shfl_xor_sync(gmask, x, o);
    return x;
}

// E = the reference's estimate of the merged row from Z = ldexp(zsum, -S)
// (zsum exact, plus extra) and the zero count V (src/hll.py:37-54; variant 1:
// cpu_exp's 2^32 correction, cpu_exp/triangle_hll_experiment.py:357-366).
__device__ __forceinline__ double hll_estimate_from(U128 zsum, double extra, uint32_t zeros, int p, int S,
                                                    int variant) {
    const int m = 1 << p;
    const double Z = ldexp(u128_to_double(zsum.lo, zsum.hi) + extra, -S);
    double alpha;
    if (m == 16) alpha = 0.673;
    else if (m == 32) alpha = 0.697;
    else if (m == 64) alpha = 0.709;
    else alpha = 0.7213 / (1.0 + 1.079 / (double)m);
    double E = alpha * (double)m * (double)m / Z;
    if (variant == 1) {
        if (E <= 2.5 * (double)m && zeros > 0) E = (double)m * log((double)m / (double)zeros);
        else if (E > 4294967296.0 / 30.0) E = -4294967296.0 * log(1.0 - E / 4294967296.0);
    } else {
        if (E <= 2.5 * (double)m) {
            if (zeros > 0) E = (double)m * log((double)m / (double)zeros);
        }
        const double two64 = 18446744073709551616.0;
        if (E > two64 / 30.0) E = -two64 * log(1.0 - E / two64);
    }
    return E;
}

// One group of L lanes per HLL edge, the group's lanes striding over the two
// 2^p-byte rows with 16-byte loads.  Pass 1 counts the zero registers V of
// the merged row from the AND of the two rows' zero masks (ZM; else from the
// registers).  Every zero register adds exactly 1 to Z = sum 2^-r, so V >=
// lc_min (the smallest V with alpha*m^2/V <= 2.5m, with a 1e-9 margin for
// the FP64 comparison) proves the estimator takes its linear-counting
// branch: E = m * ln(m / V), the same expression the full estimator
// evaluates, and Z is not needed.  Otherwise pass 2 forms Z exactly and
// applies the full estimator.  For rows of at least 32 16-byte words
// (p >= 9) the whole warp runs pass 2 for one such edge at a time
// (coalesced loads, no lane idling while one group reads two whole rows),
// so narrow groups cost nothing when a few of their edges need the
// registers; smaller rows are read by the edge's own group.
// CACHE (p >= 11, or CROW): each group takes a contiguous run of the edge
// list.  The routing pass appends edges in CSR order, so consecutive HLL edges
// mostly share u, and the group keeps u's zero mask across them: in a
// shared-memory slot (ZS: p = 11 to 14 at the default widths), in registers
// where it is at most four 16-byte words per lane (wider groups, by tuning);
// at p = 15 and 16, too long for either, it is read per edge.  With CROW (rows
// of at most 8 16-byte words per lane) u's register row stays in registers too:
// an edge then reads only v's mask and row.  Otherwise the groups stride over
// the list.
// ZS:  Slots are kZsPad 16-byte words apart beyond
// their length, so that the groups that one load instruction serves in one
// phase (8 lanes) read different banks.  A variant of its own keeps the
// register form's 16 words out of it (64 registers, four CTAs per SM): with
// the padding and the table of linear-counting estimates, R-MAT 20, theta =
// 128, alone: p = 12 609 -> 339 us (L1 data pipe 67 -> 85% busy, which bounds
// it now), p = 14 1478 -> 1078.
template <int L>
constexpr int kZsPad = L < 8 ? L : 0;

template <int L, bool ZM, bool CACHE, bool CROW, bool ZS>
__global__ void __launch_bounds__(256, CROW ? 2 : (ZS ? 4 : (CACHE ? 3 : 4))) hll_edges_kernel(const HllParams H) {
    extern __shared__ __align__(16) uint4 zsm[];  // ZS: 256 / L slots of one zero mask each
    const int lane = threadIdx.x & 31;
    const int sub = lane & (L - 1);
    const unsigned gmask = (L == 32) ? FULL : (((1u << L) - 1u) << (lane & ~(L - 1)));
    const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / L;
    const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / L;
    const int64_t n = (int64_t)*H.n_dev;
    const int m = 1 << H.p;
    const int nvec = m >> 4;
    const int S = 65 - H.p;
    U128 hacc;
    int64_t n_approx = 0, n_clamped = 0;
    const int64_t per = CACHE ? (n + ngroups - 1) / ngroups : 1;
    const int64_t e_lo = CACHE ? gid * per : gid;
    const int64_t e_hi = CACHE ? min(n, e_lo + per) : n;
    const int64_t e_step = CACHE ? 1 : ngroups;
    const int64_t w_first = gid - (lane / L);  // the warp's first group
    const int nq = H.zst >> 2;
    constexpr int KA = CROW || ZS ? 1 : 4;  // mask words cached per lane (p <= 10 with a cached row: one)
    const bool cache_a = CACHE && ZM && !ZS && nq <= KA * L;
    int64_t cached = -1, cached_row = -1;
    uint4 ca[KA];
    uint4 ra[CROW ? 8 : 1];
    // warp-uniform trip count (pass 2 is warp-wide): CACHE runs `per` steps,
    // else while the warp's first group still has an edge
    for (int64_t k = 0; CACHE ? k < per : w_first + k * ngroups < n; ++k) {
        const int64_t e = e_lo + k * e_step;
        const bool act = e < e_hi;  // group-uniform
        int32_t u = 0, v = 0;
        int64_t su = 0, sv = 0;
        uint32_t zeros = 0;
        if (act) {
            u = __ldg(H.hu + e);
            v = __ldg(H.hv + e);
            su = H.slot ? __ldg(H.slot + u) : (int64_t)u;
            sv = H.slot ? __ldg(H.slot + v) : (int64_t)v;
            if (ZM) {  // registers zero in both rows: AND of the two zero masks
                const uint4* za = reinterpret_cast<const uint4*>(H.zm + su * (int64_t)H.zst);
                const uint4* zb = reinterpret_cast<const uint4*>(H.zm + sv * (int64_t)H.zst);
                if (cache_a) {
                    if (su != cached) {  // group-uniform
#pragma unroll
                        for (int kk = 0; kk < KA; ++kk) {
                            const int i = sub + kk * L;
                            ca[kk] = i < nq ? __ldg(za + i) : make_uint4(0u, 0u, 0u, 0u);
                        }
                        cached = su;
                    }
#pragma unroll
                    for (int kk = 0; kk < KA; ++kk) {
                        const int i = sub + kk * L;
                        if (i < nq) {
                            const uint4 b = __ldg(zb + i);
                            zeros += __popc(ca[kk].x & b.x) + __popc(ca[kk].y & b.y) + __popc(ca[kk].z & b.z) +
                                     __popc(ca[kk].w & b.w);
                        }
                    }
                } else if (ZS) {
                    // u's mask in the group's shared-memory slot while
                    // consecutive edges share u: each edge reads v's only
                    uint4* zs = zsm + (size_t)(threadIdx.x / L) * (nq + kZsPad<L>);
                    if (su != cached) {  // group-uniform
                        __syncwarp(gmask);  // the group is done with the previous row
                        for (int i = sub; i < nq; i += L) zs[i] = __ldg(za + i);
                        __syncwarp(gmask);
                        cached = su;
                    }
#pragma unroll 4
                    for (int i = sub; i < nq; i += L) {
                        const uint4 a = zs[i], b = __ldg(zb + i);
                        zeros += __popc(a.x & b.x) + __popc(a.y & b.y) + __popc(a.z & b.z) + __popc(a.w & b.w);
                    }
                } else {
#pragma unroll 4
                    for (int i = sub; i < nq; i += L) {
                        const uint4 a = __ldg(za + i), b = __ldg(zb + i);
                        zeros += __popc(a.x & b.x) + __popc(a.y & b.y) + __popc(a.z & b.z) + __popc(a.w & b.w);
                    }
                }
            } else {
                const uint4* a4 = reinterpret_cast<const uint4*>(H.regs + su * (int64_t)m);
                const uint4* b4 = reinterpret_cast<const uint4*>(H.regs + sv * (int64_t)m);
#pragma unroll 4
                for (int i = sub; i < nvec; i += L) {
                    const uint4 a = __ldg(a4 + i), b = __ldg(b4 + i);
                    zeros += zero_bytes(a.x | b.x) + zero_bytes(a.y | b.y) + zero_bytes(a.z | b.z) +
                             zero_bytes(a.w | b.w);
                }
            }
        }
        zeros = group_sum_u32<L>(zeros, gmask);
        const bool need = act && zeros < H.lc_min;  // group-uniform
        double E = 0.0;
        if (act && !need) E = ZM ? __ldg(H.lc + zeros) : (double)m * log((double)m / (double)zeros);
        // rows of fewer than 32 16-byte words (p <= 8) would leave most of
        // the warp idle in a warp-wide pass 2: there each group forms Z
        if (CROW || nvec < 32) {
            if (need) {  // the group forms Z itself (CROW: u's row kept in registers)
                uint32_t fast = 0, zz = 0;
                uint64_t fine = 0;
                double extra = 0.0;
                const uint4* a4 = reinterpret_cast<const uint4*>(H.regs + su * (int64_t)m);
                const uint4* b4 = reinterpret_cast<const uint4*>(H.regs + sv * (int64_t)m);
                if (CROW) {
                    if (su != cached_row) {  // group-uniform
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk) {
                            const int i = sub + kk * L;
                            ra[kk] = i < nvec ? __ldg(a4 + i) : make_uint4(0u, 0u, 0u, 0u);
                        }
                        cached_row = su;
                    }
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {
                        const int i = sub + kk * L;
                        if (i < nvec) {
                            const uint4 b = __ldg(b4 + i);
                            hll_word_lut(__vmaxu4(ra[kk].x, b.x), S, fast, fine, zz, extra);
                            hll_word_lut(__vmaxu4(ra[kk].y, b.y), S, fast, fine, zz, extra);
                            hll_word_lut(__vmaxu4(ra[kk].z, b.z), S, fast, fine, zz, extra);
                            hll_word_lut(__vmaxu4(ra[kk].w, b.w), S, fast, fine, zz, extra);
                        }
                    }
                } else {
#pragma unroll 2
                    for (int i = sub; i < nvec; i += L) {
                        const uint4 a = __ldg(a4 + i), b = __ldg(b4 + i);
                        hll_word_lut(__vmaxu4(a.x, b.x), S, fast, fine, zz, extra);
                        hll_word_lut(__vmaxu4(a.y, b.y), S, fast, fine, zz, extra);
                        hll_word_lut(__vmaxu4(a.z, b.z), S, fast, fine, zz, extra);
                        hll_word_lut(__vmaxu4(a.w, b.w), S, fast, fine, zz, extra);
                    }
                }
                fast = group_sum_u32<L>(fast, gmask);
                fine = group_sum_u64<L>(fine, gmask);
#pragma unroll
                for (int o = L / 2; o > 0; o >>= 1) extra += __shfl_xor_sync(gmask, extra, o);
                U128 z;  // fast * 2^(S-7) + fine; fast <= 2^(p+7)
                z.lo = (uint64_t)fast << (S - 7);
                z.hi = (uint64_t)fast >> (71 - S);
                z.add(fine);
                E = hll_estimate_from(z, extra, zeros, H.p, S, H.variant);
            }
        } else {
            // pass 2, warp-wide: the whole warp forms Z for one edge at a
            // time (coalesced 16-byte loads over both rows), for each group
            // whose zero count left the linear-counting branch open
            unsigned pend = __ballot_sync(FULL, need && sub == 0);
            while (pend) {
                const int f = __ffs(pend) - 1;  // the group's first lane
                pend &= pend - 1;
                const int64_t fsu = __shfl_sync(FULL, su, f), fsv = __shfl_sync(FULL, sv, f);
                const uint32_t fz = __shfl_sync(FULL, zeros, f);
                const uint4* a4 = reinterpret_cast<const uint4*>(H.regs + fsu * (int64_t)m);
                const uint4* b4 = reinterpret_cast<const uint4*>(H.regs + fsv * (int64_t)m);
                uint32_t fast = 0, zz = 0;
                uint64_t fine = 0;
                double extra = 0.0;
#pragma unroll 2
                for (int i = lane; i < nvec; i += 32) {
                    const uint4 a = __ldg(a4 + i), b = __ldg(b4 + i);
                    hll_word_lut(__vmaxu4(a.x, b.x), S, fast, fine, zz, extra);
                    hll_word_lut(__vmaxu4(a.y, b.y), S, fast, fine, zz, extra);
                    hll_word_lut(__vmaxu4(a.z, b.z), S, fast, fine, zz, extra);
                    hll_word_lut(__vmaxu4(a.w, b.w), S, fast, fine, zz, extra);
                }
                fast = group_sum_u32<32>(fast, FULL);
                // registers of rank >= 8 (fine) and > S (extra, malformed rows) are rare
                if (__any_sync(FULL, fine != 0)) fine = group_sum_u64<32>(fine, FULL);
                if (__any_sync(FULL, extra != 0.0)) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) extra += __shfl_xor_sync(FULL, extra, o);
                }
                U128 z;  // fast * 2^(S-7) + fine; fast <= 2^(p+7)
                z.lo = (uint64_t)fast << (S - 7);
                z.hi = (uint64_t)fast >> (71 - S);
                z.add(fine);
                const double Ef = hll_estimate_from(z, extra, fz, H.p, S, H.variant);
                if ((lane & ~(L - 1)) == f) E = Ef;
            }
        }
        if (act && sub == 0) {
            const int32_t du = __ldg(H.degrees + u), dv = __ldg(H.degrees + v);
            const double s_hat = (double)((int64_t)du + (int64_t)dv) - E;
            const double upper = (double)(du < dv ? du : dv);
            // max(0.0, min(s_hat, upper)) with Python's min/max argument order
            double s_cl = (upper < s_hat) ? upper : s_hat;
            s_cl = (s_cl > 0.0) ? s_cl : 0.0;
            const bool clamped = s_hat < 0.0 || s_hat > upper;
            const uint64_t fx = (uint64_t)__double2ull_rn(s_cl * 4294967296.0);
            if (H.vbase) {  // batched: straight into this edge's graph
                tchll_count_result* R = H.result + graph_of(H.vbase, H.n_graphs, H.graph_bad, u);
                U128 one;
                one.lo = fx;
                atomic_add_u128((unsigned long long*)&R->hll_fx_lo, one);
                atomicAdd((unsigned long long*)&R->n_approx, 1ull);
                if (clamped) atomicAdd((unsigned long long*)&R->n_clamped, 1ull);
            } else {
                n_clamped += clamped;
                ++n_approx;
                hacc.add(fx);
            }
        }
    }
    publish(H.result, 0, hacc, n_approx, 0, 0, n_clamped, 0u, lane);
}

// ---------------------------------------------------------------- host ------
constexpr int kHubAuto = -1;
constexpr int kHubWide = 128;
constexpr int64_t kHub64Degree = 12;
struct Tuning {
    int chunk = 256;
    int slots_log2 = 10;    // 1024 slots = 4 KB per warp: a table side of up to 128 keys at load <= 1/8
    int tiny = 16;
    int blocks_per_sm = 0;  // 0: occupancy maximum
    int warps = 8;          // warps per CTA
    int pairs = 1;          // table-side / probe-side reorientation (2: for small graphs too)
    int sparse = 0;         // table load <= 1/4 where it fits
    int hub = kHubAuto;     // pairs with d+(x) > hub go to the CTA-table kernels (0: off; kHubAuto: set_hub)
    int hub_seg = 2048;     // hub pairs per CTA work unit
    int hub_lg = 13;        // largest CTA hash table: 2^13 slots = 32 KB
    int hub_unroll = 2;     // quads per lane in flight (2 or 4)
    int bitmap_lg = 15;     // hub bitmap buffer: 2^15 bytes = 262,144 core vertices (0: hash tables only)
    int overlap = 1;        // side stream: the hub core pass (+ the hybrid HLL pass); 2 does the same as 1
    int packed = 1;         // hub probe lists as 16-bit core indices when the core allows
    int bank_sort = 0;      // kept for its setter and getter: no effect
    int hll_row_cache_p = 0;   // HLL pass: keep u's register row in registers for p <= this (0: never)
    int hll_lanes = 0;      // HLL pass: lanes per edge (0: chosen by p)
};
// Routes are chosen by the graph (nnz members in n_nodes lists), not by the
// edges asked for, which may be a part of it: each rank of a sharded count
// brings the whole graph.  Up to kDirectNnz members, and kDirectEdges edges,
// the regrouping's dozen launches cost more than it saves, and the edges are
// counted as given, with one launch.  The line is where every list still fits a
// warp's table of 512 members: a list oriented by degree has at most
// sqrt(2 nnz).  Longer lists are searched one by one there (a 1,000-clique
// with 3,000 pendant vertices, 502 K edges: 1,768 us as given, 220 regrouped);
// up to it, as given / regrouped: R-MAT 12 (48 K edges) 59 / 103 us, a
// 510-clique with 1,000 pendant vertices (131 K) 101 / 148 us; behind it, R-MAT 14
// (200 K) 107 / 114, R-MAT 15 (388 K) 146 / 134.
constexpr int64_t kDirectNnz = 1 << 17;
constexpr int64_t kDirectEdges = 1 << 19;
// Of those, graphs of at most this mean forward degree are counted by
// binary search, the others with a hash table per u: ER 100 K edges 12 / 16 us,
// R-MAT 14 (edge factor 32, mean 28) 224 / 103 us.
constexpr int64_t kSparseDegree = 8;
// Up to this mean forward degree a graph may well have no long list at all
// (road networks), though it may have a dense core too.  The hub core pass then
// follows the first pass on the caller's stream, where its kernels and the
// hub kernels return at once when there is no hub pair, instead of scanning
// the vertices beside it, and the first pass deals its chunks to the warps in
// turn, which lists as short as these allow, instead of having them claimed.
// A million-vertex lattice (mean 2.2) takes 145 us without both, 131 so.  (In
// one launch, as given, it takes 85, but a 1,200-clique inside a lattice of 2 M
// vertices then 3.6 ms against 0.45, a 4,000-clique with 10 M pendant vertices
// 95 against 2.8.)
constexpr int64_t kRoadDegree = 3;
constexpr int HUB_MIN = 64;       // smallest hub threshold (bounds the segment count)
constexpr int HUB_SEG_MIN = 256;  // smallest segment

// The launch shape is process-wide state set through tchll_set_count_*.
// Every counting call copies it once, under the lock, and uses only its
// copy, so a concurrent setter can never change a shape half-way through a
// launch sequence (e.g. a table size versus its shared-memory allocation).
static std::mutex g_tuning_mu;
static Tuning g_tuning;
static Tuning tuning_snapshot() {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    return g_tuning;
}

// Opts a kernel into `smem` bytes of dynamic shared memory once per device
// (the attribute is per device and function); `done` is that kernel's
// per-device high-water mark, guarded by its own lock.
static std::mutex g_attr_mu;
static int ensure_smem(const void* kern, size_t smem, size_t* done, const char* what, bool carveout = false) {
    const int dev = current_device();
    if (dev < 0) return cuda_status(cudaErrorInvalidDevice, "cudaGetDevice");
    std::lock_guard<std::mutex> lock(g_attr_mu);
    if (smem > done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return cuda_status(e, what);
        if (carveout) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
            if (e != cudaSuccess) return cuda_status(e, what);
        }
        done[dev] = smem;
    }
    return TCHLL_OK;
}

// Optional phase timing: CUDA events recorded on the caller's stream around
// the pair regrouping, the exact-count launch and the HLL launch.  While
// timing is on, counting calls hold g_phase_mu for their whole enqueue, so
// the events and flags belong to one call at a time.
struct PhaseTimer {
    std::atomic<bool> on{false};
    bool made = false;
    cudaEvent_t ev[4];
    cudaEvent_t hub_ev[4];  // core pass start / end, hub kernels start / end (inside phase 1)
    cudaEvent_t hll_ev[2];  // around the HLL pass when it runs on the side stream
    bool used[3] = {false, false, false};
    bool hub_used = false;
    bool core_used = false;
    bool hll_split = false;  // phase 2 (HLL) is timed by hll_ev, not ev[2..3]
};
static PhaseTimer g_phase;
static std::mutex g_phase_mu;

// Lock held by a counting call while it records phase events.
struct PhaseScope {
    std::unique_lock<std::mutex> lock;
    PhaseScope() : lock(g_phase_mu, std::defer_lock) {
        if (g_phase.on.load()) lock.lock();
    }
    bool active() const { return lock.owns_lock() && g_phase.made; }
};

static void phase_mark(const PhaseScope& ps, int i, cudaStream_t st) {
    if (ps.active()) cudaEventRecord(g_phase.ev[i], st);
}
static void phase_used(const PhaseScope& ps, int a, int b = -1, int c = -1) {
    if (!ps.active()) return;
    for (int i : {a, b, c})
        if (i >= 0) g_phase.used[i] = true;
}
static void phase_reset(const PhaseScope& ps) {
    if (!ps.active()) return;
    for (int i = 0; i < 3; ++i) g_phase.used[i] = false;
    g_phase.hub_used = false;
    g_phase.core_used = false;
    g_phase.hll_split = false;
}

template <int MODE, bool VEC, bool DETAILS, bool SEGS = false>
static int launch_mode(const CountParams& P, const Tuning& T, cudaStream_t st) {
    auto kern = count_kernel<MODE, VEC, DETAILS, SEGS>;
    const int threads = T.warps * 32;
    const size_t smem = (size_t)T.warps * ((size_t)1 << P.slots_log2) * sizeof(int32_t);
    static size_t smem_set[kMaxDevices] = {};
    int rc = ensure_smem((const void*)kern, smem, smem_set, "cudaFuncSetAttribute(count_kernel)");
    if (rc) return rc;
    int bps = T.blocks_per_sm;
    if (bps <= 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, threads, smem);
        if (e != cudaSuccess) return cuda_status(e, "occupancy(count_kernel)");
        if (bps < 1) bps = 1;
    }
    const int grid = sm_count() * bps;
    kern<<<grid, threads, smem, st>>>(P);
    TCHLL_CHECK_LAUNCH("count_kernel");
    return TCHLL_OK;
}

template <int MODE>
static int launch_count(const CountParams& P, const Tuning& T, bool details, cudaStream_t st) {
    const bool vec = ((uintptr_t)P.col_idx % 16 == 0) && (P.regs == nullptr || (uintptr_t)P.regs % 16 == 0);
    if (details) return vec ? launch_mode<MODE, true, true>(P, T, st) : launch_mode<MODE, false, true>(P, T, st);
    return vec ? launch_mode<MODE, true, false>(P, T, st) : launch_mode<MODE, false, false>(P, T, st);
}

// Edges as given (no regrouping): small chunks, so that a small graph reaches
// every warp (48 K edges, R-MAT 12: 26 us with 8 edges a warp, 40 with 32, 59
// with 64).
static int given_chunk(int64_t n_edges, int chunk) {
    int c = 8;
    while (c < 32 && n_edges >= 6144 * (int64_t)(2 * c)) c *= 2;
    return c < chunk ? c : chunk;
}

struct CountWs {
    // counters: [0] [1] chunks, [2] hub segments made, [3] hub segments
    // claimed, [4] HLL edges, [5] grouped pairs, [6] batches: the graphs from
    // the first malformed one on, [7] table segments made, [8] claimed; with
    // ncore and cbits one run of zero_words words
    unsigned long long* ctr;
    int64_t zero_words;
    int32_t* cnth;            // n_nodes + 1 (histogram of grouped pairs)
    int32_t* offh;            // n_nodes + 1 (scan, then scatter cursor)
    int32_t* py;              // n_edges (probe sides of the grouped pairs, by table side)
    int2* rows;               // n_nodes: the row table
    uint2* codes;             // n_edges / 32 + 1 (batches: their own)
    PairSeg* segs;             // max_segs
    int64_t max_segs;
    int32_t* pcol;            // padded lists in core coordinates for the hub kernels, pcap entries (null: not carved)
    int64_t pcap;
    int32_t* cflag;           // n_nodes + 1: popularity counts, then core indices (with pcol)
    uint32_t* cbits;          // (n_nodes + 31) / 32 + 1: core membership (with pcol)
    int32_t* ncore;           // kCoreWords words: see launch_core_pass (with pcol)
    int4* pl;                 // n_nodes: packed lists' records (with pcol)
    uint4* pool;              // pool_cap bitmap units (with pcol)
    int64_t pool_cap;
};

// Padded lists need nnz + 8 (n_nodes + 1) entries; the workspace holds them
// for nnz <= n_edges (every oriented edge listed once).
// int32 entries of the padded-list region: the 32-bit lists (pad_start)
// or the packed ones (pad16_start, 2 bytes a key), whichever is larger.
static int64_t pad_capacity(int64_t n_nodes, int64_t nnz) {
    const int64_t w32 = nnz + 8 * (n_nodes + 1) + 8;
    const int64_t w16 = (nnz + 24 * (n_nodes + 1) + 24 + 1) / 2 + 4;
    return w32 > w16 ? w32 : w16;
}

// The hub core pass's small arrays: [0] core size, [1] pool units claimed,
// [2..3] the list kernel's row counter (64 bits), [4 ..) popularity buckets'
// sizes and cursors (256 each), last the number of live row blocks.  Cleared
// together.
constexpr int kCoreWords = 4 + 2 * 256 + 1;
constexpr int kCounters = 10;
constexpr int kEstWords = 6;  // est (an even number), in front of the counters: cleared on its own
static_assert(kEstWords >= kEst);

static bool carve_count(void* ws, size_t bytes, int64_t n_nodes, int64_t n_edges, CountWs& W, size_t* need,
                        bool pad = true) {
    const size_t N = (size_t)(n_nodes > 0 ? n_nodes : 0) + 1;
    const size_t E = (size_t)(n_edges > 0 ? n_edges : 1);
    Carve cv(ws, bytes);
    // [counters][ncore][cbits]
    const size_t cb = pad ? N / 32 + 1 : 0, nc = pad ? kCoreWords : 0;
    W.zero_words = (int64_t)(2 * kCounters + nc + cb);
    W.ctr = reinterpret_cast<unsigned long long*>(cv.take<uint32_t>((size_t)W.zero_words + 2 * kEstWords)) + kEstWords;
    W.ncore = pad ? reinterpret_cast<int32_t*>(W.ctr + kCounters) : nullptr;
    W.cbits = pad ? reinterpret_cast<uint32_t*>(W.ncore + kCoreWords) : nullptr;
    W.cnth = cv.take<int32_t>(N);
    W.offh = cv.take<int32_t>(N);
    W.py = cv.take<int32_t>(E);
    W.rows = cv.take<int2>(N);
    W.codes = cv.take<uint2>(E / 32 + 1);
    // every hub x with pairs opens one segment, every HUB_SEG_MIN pairs at most one more
    W.max_segs = (int64_t)(N < E ? N : E) + (int64_t)(E / HUB_SEG_MIN) + 1;
    W.segs = cv.take<PairSeg>((size_t)W.max_segs);
    W.pcap = pad ? pad_capacity(n_nodes, (int64_t)E) : 0;
    W.pcol = pad ? cv.take<int32_t>((size_t)W.pcap) : nullptr;
    W.cflag = pad ? cv.take<int32_t>(N) : nullptr;
    W.pl = pad ? cv.take<int4>(N) : nullptr;
    W.pool_cap = pad ? (int64_t)(E / 16) + 64 : 0;
    W.pool = pad ? cv.take<uint4>((size_t)W.pool_cap) : nullptr;
    if (need) *need = cv.off;
    return cv.ok();
}

// Hybrid calls also hold the HLL edge list (8 bytes per edge) after the
// exact-count layout, then optionally the zero masks of the register rows
// (zmask_words(p) words per row); exact-only calls use the prefix.
struct HybridWs {
    int32_t* hll_u;
    int32_t* hll_v;
    unsigned long long* hll_n;
    uint32_t* zm;  // null when the workspace was sized without masks
    int zst;
    double* lc;    // with zm: 2^p + 1 linear-counting estimates
};

static int zmask_words(int p) {
    const int w = (1 << p) >> 5;
    return w < 4 ? 4 : w;
}

static bool carve_count_hybrid(void* ws, size_t bytes, int64_t n_nodes, int64_t n_edges, int64_t zm_rows, int p,
                               CountWs& W, HybridWs& H, size_t* need, bool pad = true) {
    size_t base = 0;
    carve_count(nullptr, 0, n_nodes, n_edges, W, &base, pad);
    const size_t E = (size_t)(n_edges > 0 ? n_edges : 1);
    Carve cv(ws, bytes);
    char* b = cv.take<char>(base);
    H.hll_u = cv.take<int32_t>(E);
    H.hll_v = cv.take<int32_t>(E);
    H.zm = nullptr;
    H.zst = 0;
    H.lc = nullptr;
    if (zm_rows > 0) {
        H.zst = zmask_words(p);
        H.zm = cv.take<uint32_t>((size_t)zm_rows * (size_t)H.zst);
        H.lc = cv.take<double>(((size_t)1 << p) + 1);
    }
    if (need) *need = cv.off;
    if (!cv.ok()) return false;
    if (!cv.dry) carve_count(b, base, n_nodes, n_edges, W, nullptr, pad);
    H.hll_n = W.ctr + 4;
    return true;
}

static uint32_t lc_min_for(int p) {
    const double m = (double)(1 << p);
    double alpha;
    if (p == 4) alpha = 0.673;
    else if (p == 5) alpha = 0.697;
    else if (p == 6) alpha = 0.709;
    else alpha = 0.7213 / (1.0 + 1.079 / m);
    return (uint32_t)ceil(alpha * m / 2.5 * (1.0 + 1e-9));
}

template <int L>
static int launch_hll_edges_L(HllParams H, bool crow, cudaStream_t st) {
    const int grid = sm_count() * 8;
    if (H.zm && crow && L * 8 >= ((1 << H.p) >> 4)) hll_edges_kernel<L, true, true, true, false><<<grid, 256, 0, st>>>(H);
    else if (H.zm && H.p >= 11) {
        // masks too large for the 4 register words per lane go to shared
        // memory, one slot per group, while that fits 104 KB per CTA
        const int nq = H.zst >> 2;
        const size_t smem = nq > 4 * L ? (size_t)(256 / L) * (nq + kZsPad<L>) * sizeof(uint4) : 0;
        if (smem > 0 && smem <= (104u << 10)) {
            static size_t set[kMaxDevices] = {0};
            auto kern = hll_edges_kernel<L, true, true, false, true>;
            const int rc = ensure_smem((const void*)kern, smem, set, "cudaFuncSetAttribute(hll_edges_kernel)");
            if (rc) return rc;
            kern<<<grid, 256, smem, st>>>(H);
        } else {
            hll_edges_kernel<L, true, true, false, false><<<grid, 256, 0, st>>>(H);
        }
    }
    else if (H.zm) hll_edges_kernel<L, true, false, false, false><<<grid, 256, 0, st>>>(H);
    else hll_edges_kernel<L, false, false, false, false><<<grid, 256, 0, st>>>(H);
    TCHLL_CHECK_LAUNCH("hll_edges_kernel");
    return TCHLL_OK;
}

// The zero masks (when the workspace holds them), before launch_hll_edges.
static int launch_zmask(const CountParams& P, const HybridWs& HW, cudaStream_t st) {
    if (HW.zm == nullptr) return TCHLL_OK;
    const int64_t rows = P.slot ? P.n_rows : P.n_nodes;
    const int64_t wgrid = (rows + 7) / 8;
    const int grid = (int)(wgrid < 1 ? 1 : (wgrid > (int64_t)sm_count() * 16 ? (int64_t)sm_count() * 16 : wgrid));
    zmask_kernel<<<grid, 256, 0, st>>>(P.regs, rows, P.slot ? nullptr : P.has, P.p, HW.zst, HW.zm, HW.lc);
    TCHLL_CHECK_LAUNCH("zmask_kernel");
    return TCHLL_OK;
}

static int launch_hll_edges(const CountParams& P, const HybridWs& HW, const Tuning& T, cudaStream_t st) {
    HllParams H;
    H.vbase = P.graph_vbase;
    H.n_graphs = P.n_graphs;
    H.graph_bad = P.graph_bad;
    H.hu = HW.hll_u;
    H.hv = HW.hll_v;
    H.n_dev = HW.hll_n;
    H.degrees = P.degrees;
    H.regs = P.regs;
    H.slot = P.slot;
    H.p = P.p;
    H.variant = P.variant;
    H.lc_min = lc_min_for(P.p);
    H.result = P.result;
    H.zm = HW.zm;
    H.zst = HW.zst;
    H.lc = HW.lc;
    // p <= row_cache_p (with zero masks): contiguous runs per group with u's
    // register row kept in registers, m / 128 lanes per edge (8 16-byte
    // words of the row per lane; off by default: at 128 registers per
    // thread too few warps hide the loads).  With zero masks the pass is
    // bound by the latency of its dependent loads and by the instructions of
    // a step, which all edges of a warp share, so narrow groups (more edges in
    // flight per warp) win until their masks no longer coalesce (R-MAT 20,
    // theta = 64 or 128, alone, us with 1 / 2 / 4 / 8 lanes: p = 10 363 / 328 /
    // 514 / 840, p = 11 459 / 259 / 293 / 518, p = 12 859 / 537 / 338 / 529,
    // p = 13 1954 / 2060 / 658 / 607, p = 14 5645 / 6165 / 3740 / 1077).
    // Without masks one 16-byte register load per lane per row.  T.hll_lanes >
    // 0 overrides the width.
    const bool crow = H.zm != nullptr && P.p <= T.hll_row_cache_p;
    int width = (1 << P.p) >> 4;
    if (crow) width = (1 << P.p) >> 7;
    else if (H.zm) width = P.p <= 9 ? 1 : P.p <= 11 ? 2 : P.p == 12 ? 4 : 8;
    if (T.hll_lanes > 0) width = T.hll_lanes;
    switch (width >= 32 ? 32 : (width < 1 ? 1 : width)) {
        case 1: return launch_hll_edges_L<1>(H, crow, st);
        case 2: return launch_hll_edges_L<2>(H, crow, st);
        case 4: return launch_hll_edges_L<4>(H, crow, st);
        case 8: return launch_hll_edges_L<8>(H, crow, st);
        case 16: return launch_hll_edges_L<16>(H, crow, st);
        default: return launch_hll_edges_L<32>(H, crow, st);
    }
}

static int grid_edges(int64_t n) {
    int64_t g = (n + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 16;
    if (g > cap) g = cap;
    return g < 1 ? 1 : (int)g;
}

// Before the first pass: the row table, and all counters, flags and results
// cleared (more: words of the caller's own).
static int pass_prepare(CountParams& P, const CountWs& W, int64_t n_results, uint32_t* more, int64_t more_words,
                        cudaStream_t st) {
    Prepare Q{};
    Q.row_ptr = P.row_ptr;
    Q.n_nodes = P.n_nodes;
    Q.rows = W.rows;
    Q.nnz = P.nnz;
    Q.degrees = P.regs || P.slot || P.has ? P.degrees : nullptr;
    Q.gamma = P.gamma;
    Q.slot = P.slot;
    Q.has = P.has;
    Q.n_rows = P.n_rows;
    Q.zero_n[0] = W.cnth;
    Q.zero_n[1] = P.hub > 0 ? W.cflag : nullptr;
    Q.zero[0] = reinterpret_cast<uint32_t*>(W.ctr);
    Q.words[0] = W.zero_words;
    Q.zero[1] = reinterpret_cast<uint32_t*>(P.result);
    Q.words[1] = n_results * (int64_t)(sizeof(tchll_count_result) / 4);
    Q.zero[2] = more;
    Q.words[2] = more_words;
    Q.hub = P.hub;
    Q.edge_u = P.edge_u;
    Q.edge_v = P.edge_v;
    Q.n_edges = P.n_edges;
    Q.est = W.ctr - kEstWords;
    TCHLL_CUDA(cudaMemsetAsync(Q.est, 0, kEstWords * sizeof(unsigned long long), st));
    const int64_t sample = P.n_edges < kEdgeSample ? P.n_edges : kEdgeSample;
    prepare_kernel<<<grid_edges(P.n_nodes + 1 > sample ? P.n_nodes + 1 : sample), 256, 0, st>>>(Q);
    TCHLL_CHECK_LAUNCH("prepare_kernel");
    P.est = Q.est;
    P.rows = W.rows;
    P.codes = W.codes;
    return TCHLL_OK;
}

// Edges per claim: a few claims per warp at least, so that the last ones
// even out.
static int pass_chunk(int64_t n_edges, int chunk) {
    while (chunk > 32 && n_edges < (int64_t)chunk * 48 * 8 * sm_count()) chunk >>= 1;
    return chunk < 32 ? 32 : chunk & ~31;
}

// The first pass: `what` of PASS_HIST (grouped pairs counted per table side) and
// PASS_SHORT (all others counted for good).
template <bool HYB>
static int pair_pass(CountParams P, const CountWs& W, const Tuning& T, int what, unsigned long long* work,
                     cudaStream_t st) {
    const bool vec = (uintptr_t)P.col_idx % 16 == 0;
    auto kern = vec ? pair_pass_kernel<HYB, true> : pair_pass_kernel<HYB, false>;
    static std::atomic<int> fit[2][kMaxDevices] = {};  // per kernel
    const int dev = current_device();
    if (dev < 0) return cuda_status(cudaErrorInvalidDevice, "cudaGetDevice");
    int bps = T.blocks_per_sm > 0 ? T.blocks_per_sm : fit[vec][dev].load();
    if (bps == 0) {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, 256, 0);
        if (e != cudaSuccess) return cuda_status(e, "occupancy(pair_pass_kernel)");
        if (bps < 1) bps = 1;
        fit[vec][dev].store(bps);
    }
    P.work = work;
    int64_t grid = (int64_t)sm_count() * bps;
    if (!P.chunk_start) {  // no more warps than chunks
        const int64_t need = (P.n_edges + 8 * (int64_t)P.chunk - 1) / (8 * (int64_t)P.chunk);
        const int64_t ids = P.check_ids ? (P.n_nodes > P.nnz / 4 ? P.n_nodes : P.nnz / 4) / 1024 + 1 : 1;
        const int64_t most = need > ids ? need : ids;
        if (grid > most) grid = most;
    }
    kern<<<(int)grid, 256, 0, st>>>(P, what, W.cnth);
    TCHLL_CHECK_LAUNCH("pair_pass_kernel");
    return TCHLL_OK;
}

// After PASS_HIST: room for the grouped pairs, and their segments (smaller
// hub segments in small graphs, so that every CTA gets a few).
static int hub_alloc(const CountParams& P, const CountWs& W, int hub_seg, cudaStream_t st) {
    while (hub_seg > HUB_SEG_MIN && P.n_edges < (int64_t)hub_seg * 24 * sm_count()) hub_seg >>= 1;
    if (hub_seg < HUB_SEG_MIN) hub_seg = HUB_SEG_MIN;
    const int grid = (int)(P.n_nodes > 0 ? (P.n_nodes + 1023) / 1024 : 1);
    const PairRoom R{W.ctr + 5, W.segs, W.max_segs, W.ctr + 2, W.ctr + 7};
    hub_alloc_kernel<<<grid, 256, 0, st>>>(W.cnth, P, hub_seg, W.offh, R);
    TCHLL_CHECK_LAUNCH("hub_alloc_kernel");
    return TCHLL_OK;
}

static int pairs_scatter(const CountParams& P, const CountWs& W, cudaStream_t st) {
    pair_scatter_kernel<<<grid_edges(P.n_edges), 256, 0, st>>>(P, W.offh, W.ctr + 5, W.py);
    TCHLL_CHECK_LAUNCH("pair_scatter_kernel");
    return TCHLL_OK;
}

// The table pairs, once scattered.
static int launch_table_pairs(const CountParams& P, const CountWs& W, const Tuning& T, cudaStream_t st) {
    CountParams Q = P;
    Q.edge_v = W.py;
    Q.segs_end = W.segs + W.max_segs;
    Q.n_segs = W.ctr + 7;
    Q.work = W.ctr + 8;
    Q.check_ids = 0;
    Q.chunk_start = nullptr;
    return (uintptr_t)P.col_idx % 16 == 0 ? launch_mode<MODE_EXACT, true, false, true>(Q, T, st)
                                          : launch_mode<MODE_EXACT, false, false, true>(Q, T, st);
}

static int grid_rows(int64_t n, int per_cta) {  // one unit of work per 256 / per_cta threads
    int64_t g = (n + per_cta - 1) / per_cta;
    const int64_t cap = (int64_t)sm_count() * 16;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

// The hub core pass and kernels use the padded lists when the workspace
// holds them and 16-byte unit indices, and steps of 128 members past the end
// of a row, fit int.
static bool hub_pad_usable(const CountParams& P, const CountWs& W) {
    const int64_t need_pad = pad_capacity(P.n_nodes, P.nnz);
    return W.pcol != nullptr && need_pad <= W.pcap && need_pad <= (int64_t)INT32_MAX - 128;
}

// The hub core pass (needs only the CSR and cleared counters, so it may run on
// a second stream from the start, beside the first pass and the scatter): core
// members, their numbering, then the lists, packed when the core allows it,
// else 32-bit (each list kernel checks the core size on the device).  Where
// hub pairs are rare (batches, road networks) it follows the first pass and
// the scatter instead (`after`), and its kernels return at once without any.
static int launch_core_pass(const CountParams& P, const CountWs& W, const Tuning& T, bool after, const PhaseScope& ps,
                            cudaStream_t st) {
    if (!hub_pad_usable(P, W)) return TCHLL_OK;
    const unsigned long long* n_segs = after ? W.ctr + 2 : nullptr;
    if (ps.active()) {
        cudaEventRecord(g_phase.hub_ev[0], st);
        g_phase.core_used = true;
    }
    core_mark_kernel<<<grid_rows(P.n_nodes, 256) < 8 * sm_count() ? grid_rows(P.n_nodes, 256) : 8 * sm_count(), 256, 0,
                       st>>>(P.row_ptr, P.n_nodes, P.nnz, P.col_idx, P, P.nnz <= kMarkAllEdges,
                             n_segs, W.cbits, W.cflag, P.result);
    TCHLL_CHECK_LAUNCH("core_mark_kernel");
    if (P.graph_vbase) {
        core_index_batch_kernel<<<(int)P.n_graphs, 1024, 0, st>>>(W.cbits, W.cflag, P.n_nodes, P.graph_vbase,
                                                                 P.graph_hub, P.live_flag, P.live_list,
                                                                 W.ncore + kCoreWords - 1, W.ncore);
        TCHLL_CHECK_LAUNCH("core_index_batch_kernel");
        if (P.n_nodes >= kBigGraph) {
            const int tiles = (int)((P.n_nodes + kBigTile - 1) / kBigTile);
            core_bucket_big_kernel<<<tiles, 256, 0, st>>>(W.cbits, W.cflag, P, n_segs);
            TCHLL_CHECK_LAUNCH("core_bucket_big_kernel");
            core_index_big_kernel<<<tiles, 256, 0, st>>>(W.cbits, W.cflag, P, n_segs, W.ncore);
            TCHLL_CHECK_LAUNCH("core_index_big_kernel");
        }
    } else {
        int64_t gv = (P.n_nodes + 1023) / 1024;
        gv = gv < 1 ? 1 : (gv > 4 * (int64_t)sm_count() ? 4 * (int64_t)sm_count() : gv);
        core_bucket_kernel<<<(int)gv, 256, 0, st>>>(W.cbits, W.cflag, P.n_nodes, n_segs, W.ncore + 4);
        TCHLL_CHECK_LAUNCH("core_bucket_kernel");
        core_index_kernel<<<(int)gv, 256, 0, st>>>(W.cbits, W.cflag, P.n_nodes, W.ncore + 4, W.ncore + 4 + 256, n_segs,
                                                   W.ncore);
        TCHLL_CHECK_LAUNCH("core_index_kernel");
    }
    int64_t gl = (P.n_nodes + 63) / 64;
    gl = gl < 1 ? 1 : (gl > 6 * (int64_t)sm_count() ? 6 * (int64_t)sm_count() : gl);
    core_lists_kernel<<<(int)gl, 256, 0, st>>>(
        P.row_ptr, P.n_nodes, P.nnz, P.col_idx, W.cflag, W.ncore, T.packed, reinterpret_cast<uint16_t*>(W.pcol), W.pl,
        W.pool, (int32_t)(W.pool_cap < INT32_MAX / 2 ? W.pool_cap : INT32_MAX / 2), W.ncore + 1,
        reinterpret_cast<unsigned long long*>(W.ncore + 2), n_segs, P.live_list, W.ncore + kCoreWords - 1, P.check_ids,
        P.result);
    TCHLL_CHECK_LAUNCH("core_lists_kernel");
    if (!T.packed || P.n_nodes > kCore16Max) {  // else the packed lists always apply
        core_pad_kernel<<<grid_rows(P.n_nodes, 32), 256, 0, st>>>(P.row_ptr, P.n_nodes, P.nnz, P.col_idx, W.cflag,
                                                                  W.ncore, T.packed, W.pcol, P.check_ids, P.result);
        TCHLL_CHECK_LAUNCH("core_pad_kernel");
    }
    if (ps.active()) cudaEventRecord(g_phase.hub_ev[1], st);
    return TCHLL_OK;
}

// The hub pairs: one CTA per segment at a time, persistent grid.  With the
// padded lists (the core pass done before, on this stream or waited for):
// the packed bitmap kernel, the 32-bit bitmap kernel, then the hash kernel;
// each but the one the core size selects returns at once.  Without them (a
// small workspace): the hash kernel over the raw lists.
static int launch_hub(const CountParams& P, const CountWs& W, const Tuning& T, const PhaseScope& ps, cudaStream_t st,
                      bool batched = false) {
    HubParams H{};
    H.batched = batched;
    H.row_ptr = P.row_ptr;
    H.n_nodes = P.n_nodes;
    H.col_idx = P.col_idx;
    H.nnz = P.nnz;
    H.hy = W.py;
    H.segs = W.segs;
    H.n_segs = W.ctr + 2;
    H.max_segs = W.max_segs;
    H.seg_ctr = W.ctr + 3;
    H.hub_lg = T.hub_lg;
    H.result = P.result;
    const bool pad = hub_pad_usable(P, W);
    if (pad) {
        H.pcol = W.pcol;
        H.cidx = W.cflag;
        H.n_core = W.ncore;
        H.pl = W.pl;
        H.pool = W.pool;
        H.packed = T.packed;
    }
    if (ps.active()) cudaEventRecord(g_phase.hub_ev[2], st);
    if (pad && T.packed) {
        const size_t smem = 16384;
        auto kern = T.hub_unroll == 4 ? hub_bitmap16_kernel<4> : hub_bitmap16_kernel<2>;
        static size_t smem_set[2][kMaxDevices] = {};
        int rc = ensure_smem((const void*)kern, smem, smem_set[T.hub_unroll == 4 ? 1 : 0],
                             "cudaFuncSetAttribute(hub_bitmap16_kernel)", true);
        if (rc) return rc;
        int bps = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, kHub16Threads, smem);
        if (e != cudaSuccess) return cuda_status(e, "occupancy(hub_bitmap16_kernel)");
        if (bps < 1) bps = 1;
        kern<<<sm_count() * bps, kHub16Threads, smem, st>>>(H);
        TCHLL_CHECK_LAUNCH("hub_bitmap16_kernel");
    }
    const bool sure = pad && T.packed && P.n_nodes <= kCore16Max;  // the packed lists apply: C <= n_nodes
    if (pad && T.bitmap_lg > 0 && !sure) {
        const size_t smem = (size_t)1 << T.bitmap_lg;
        H.cap_bits = (int)(8 * smem);
        auto kern = T.hub_unroll == 4 ? hub_bitmap_kernel<4> : hub_bitmap_kernel<2>;
        static size_t smem_set[2][kMaxDevices] = {};
        int rc = ensure_smem((const void*)kern, smem, smem_set[T.hub_unroll == 4 ? 1 : 0],
                             "cudaFuncSetAttribute(hub_bitmap_kernel)", true);
        if (rc) return rc;
        int bps = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, 256, smem);
        if (e != cudaSuccess) return cuda_status(e, "occupancy(hub_bitmap_kernel)");
        if (bps < 1) bps = 1;
        kern<<<sm_count() * bps, 256, smem, st>>>(H);
        TCHLL_CHECK_LAUNCH("hub_bitmap_kernel");
    }
    if (sure) {
        if (ps.active()) {
            cudaEventRecord(g_phase.hub_ev[3], st);
            g_phase.hub_used = true;
        }
        return TCHLL_OK;
    }
    const int vi = (T.hub_unroll == 4 ? 2 : 0) + (pad ? 1 : 0);
    auto kern = vi == 3 ? hub_count_kernel<4, true>
                        : vi == 2 ? hub_count_kernel<4, false> : vi == 1 ? hub_count_kernel<2, true> : hub_count_kernel<2, false>;
    const size_t smem = sizeof(int32_t) << T.hub_lg;
    static size_t hsmem_set[4][kMaxDevices] = {};
    int rc = ensure_smem((const void*)kern, smem, hsmem_set[vi], "cudaFuncSetAttribute(hub_count_kernel)", true);
    if (rc) return rc;
    int bps = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, 256, smem);
    if (e != cudaSuccess) return cuda_status(e, "occupancy(hub_count_kernel)");
    if (bps < 1) bps = 1;
    kern<<<sm_count() * bps, 256, smem, st>>>(H);
    TCHLL_CHECK_LAUNCH("hub_count_kernel");
    if (ps.active()) {
        cudaEventRecord(g_phase.hub_ev[3], st);
        g_phase.hub_used = true;
    }
    return TCHLL_OK;
}

// Sets P's hub threshold: 0 without the hub path, which takes the packed or
// padded lists or, for the quad loads of the raw ones, a 16-byte aligned
// col_idx.
// The automatic threshold is 64 where the lists are held and their core fits
// the packed form, else 128: bitmap lists are the faster way for pairs of 64 to
// 128 members too, but beyond kCore16Max core vertices the 32-bit kernels
// count (R-MAT 17, us, at 64 / 128: 318 / 367; R-MAT 22 has a core of 108 K vertices
// at 128, 262 K at 64).  It surely fits in graphs of so few vertices and,
// oriented by degree, of so few edges: a member of a list of over 64 has at
// least that degree.  Up to kHub64Edges edges skewed graphs' cores fit too, and
// the device chooses (choose).  Batches number each graph's core on its own,
// but need many such pairs to a table side for the core pass, which nothing
// overlaps, to pay: a mean forward degree of 12 (256 R-MAT 12, mean 23: 1,970 /
// 2,640 us; 40 R-MAT 13, mean 13: 511 / 462); the device looks at the largest
// graph.
static void set_hub(CountParams& P, const CountWs& W, const Tuning& T) {
    const bool held = hub_pad_usable(P, W);
    P.hub_alt = 0;
    P.hub = T.hub == kHubAuto ? kHubWide : T.hub;
    if (!held && (uintptr_t)P.col_idx % 16 != 0) P.hub = 0;
    if (T.hub != kHubAuto || !held) return;
    if (P.graph_vbase) {
        P.hub_alt = P.n_edges >= kHub64Degree * P.n_nodes;
        if (P.hub_alt) P.hub = kHubWide / 2;
    } else if (P.n_nodes <= kCore16Max || 2 * P.nnz < (kHubWide / 2 + 1) * (int64_t)(kCore16Max + 1)) {
        P.hub = kHubWide / 2;
    } else if (P.nnz <= kHub64Edges) {
        P.hub = kHubWide / 2;
        P.hub_alt = 1;
    }
}

// A second stream per device for work that overlaps the caller's stream: the
// HLL pass of a hybrid count runs there beside the exact pairs.  Fork = an
// event recorded on the caller's stream that the side stream waits for;
// join = an event recorded on the side stream that the caller's stream
// waits for before the call returns.  Both are recorded under the device's
// lock, held from fork to join, so concurrent calls never wait on each
// other's events; under stream capture this is the usual fork/join of a
// captured graph.  Stream and events are created on first use (outside any
// capture: the first call of a process is never captured by this package).
struct SideStream {
    cudaStream_t s = nullptr;
    cudaEvent_t fork = nullptr, mid = nullptr, join = nullptr, back = nullptr;
    std::mutex mu;
};
static SideStream g_side[kMaxDevices];
static std::mutex g_side_make_mu;

class SideFork {
  public:
    // Starts the fork (returns an error status, or TCHLL_OK with stream()
    // ready for work that may run once the caller's stream got here).
    int begin(cudaStream_t caller) {
        const int dev = current_device();
        if (dev < 0) return cuda_status(cudaErrorInvalidDevice, "cudaGetDevice");
        SideStream& S = g_side[dev];
        {
            std::lock_guard<std::mutex> mk(g_side_make_mu);
            if (S.s == nullptr) {
                TCHLL_CUDA(cudaStreamCreateWithFlags(&S.s, cudaStreamNonBlocking));
                TCHLL_CUDA(cudaEventCreateWithFlags(&S.fork, cudaEventDisableTiming));
                TCHLL_CUDA(cudaEventCreateWithFlags(&S.mid, cudaEventDisableTiming));
                TCHLL_CUDA(cudaEventCreateWithFlags(&S.join, cudaEventDisableTiming));
                TCHLL_CUDA(cudaEventCreateWithFlags(&S.back, cudaEventDisableTiming));
            }
        }
        lock_ = std::unique_lock<std::mutex>(S.mu);
        side_ = &S;
        caller_ = caller;
        TCHLL_CUDA(cudaEventRecord(S.fork, caller));
        TCHLL_CUDA(cudaStreamWaitEvent(S.s, S.fork, 0));
        return TCHLL_OK;
    }
    cudaStream_t stream() const { return side_->s; }
    // Marks the side stream's work so far; wait_mark makes the caller's
    // stream wait for it (once per fork).
    int mark() {
        TCHLL_CUDA(cudaEventRecord(side_->mid, side_->s));
        return TCHLL_OK;
    }
    int wait_mark() {
        TCHLL_CUDA(cudaStreamWaitEvent(caller_, side_->mid, 0));
        return TCHLL_OK;
    }
    // The side stream waits for the caller's work so far (once per fork).
    int side_waits_caller() {
        TCHLL_CUDA(cudaEventRecord(side_->back, caller_));
        TCHLL_CUDA(cudaStreamWaitEvent(side_->s, side_->back, 0));
        return TCHLL_OK;
    }
    // Joins: the caller's stream waits for everything enqueued on the side
    // stream so far.  Safe to call more than once.
    int end() {
        if (side_ == nullptr) return TCHLL_OK;
        SideStream* S = side_;
        side_ = nullptr;
        cudaError_t e = cudaEventRecord(S->join, S->s);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(caller_, S->join, 0);
        lock_.unlock();
        return e == cudaSuccess ? TCHLL_OK : cuda_status(e, "side stream join");
    }
    ~SideFork() { end(); }

  private:
    SideStream* side_ = nullptr;
    cudaStream_t caller_ = nullptr;
    std::unique_lock<std::mutex> lock_;
};

// col_ready (exact counts only; null = ready): an event the kernels that
// read col_idx wait for, so the grouping of hub and table pairs (row_ptr and the
// edges only) overlaps a copy of col_idx still in flight.
static int run_count(CountParams P, int mode, bool details, void* ws, size_t ws_bytes, cudaStream_t st,
                     cudaEvent_t col_ready = nullptr) {
    const Tuning T = tuning_snapshot();
    CountWs W;
    HybridWs HW{};
    size_t need = 0;
    bool ok;
    // Optional parts, used when the workspace has room (same results): the
    // core-coordinate lists of the hub kernels and, for hybrid calls, the zero
    // masks that let the HLL pass test linear counting without the registers.
    if (mode == MODE_EXACT) {
        ok = carve_count(ws, ws_bytes, P.n_nodes, P.n_edges, W, &need, true);
        if (!ok) ok = carve_count(ws, ws_bytes, P.n_nodes, P.n_edges, W, &need, false);
    } else {
        const int64_t zm_rows = P.slot ? P.n_rows : P.n_nodes;
        ok = zm_rows > 0 && carve_count_hybrid(ws, ws_bytes, P.n_nodes, P.n_edges, zm_rows, P.p, W, HW, &need);
        if (!ok) ok = carve_count_hybrid(ws, ws_bytes, P.n_nodes, P.n_edges, 0, P.p, W, HW, &need, true);
        if (!ok) ok = carve_count_hybrid(ws, ws_bytes, P.n_nodes, P.n_edges, 0, P.p, W, HW, &need, false);
    }
    if (!ok || ws == nullptr) {
        set_error("workspace too small: need %zu bytes, have %zu", need, ws_bytes);
        return TCHLL_EWORKSPACE;
    }
    const bool direct = T.pairs != 2 && P.nnz <= kDirectNnz && P.n_edges <= kDirectEdges;
    const bool direct_pass = direct && T.pairs && !details;
    const bool sparse = P.nnz <= kSparseDegree * P.n_nodes;
    const bool road = P.nnz <= kRoadDegree * P.n_nodes;
    const bool pairs = T.pairs && !details && !direct;
    const bool prepared = pairs && P.n_edges > 0 &&
                          (mode == MODE_EXACT || (mode == 2 && (uintptr_t)P.regs % 16 == 0));  // by pass_prepare
    if (!prepared) {
        if (!direct_pass || mode != MODE_EXACT)  // a direct exact count claims nothing
            TCHLL_CUDA(cudaMemsetAsync(W.ctr, 0, kCounters * sizeof(unsigned long long), st));
        TCHLL_CUDA(cudaMemsetAsync(P.result, 0, sizeof(tchll_count_result), st));
    }
    if (details && P.pe_support) TCHLL_CUDA(cudaMemsetAsync(P.pe_support, 0, sizeof(int64_t) * P.n_edges, st));
    if (details && P.pe_method) TCHLL_CUDA(cudaMemsetAsync(P.pe_method, 0, P.n_edges, st));
    P.chunk = T.chunk;
    P.slots_log2 = T.slots_log2;
    P.tiny = T.tiny;
    P.sparse = T.sparse;
    P.hll_u = nullptr;
    P.hll_v = nullptr;
    P.hll_n = nullptr;
    if (P.n_edges == 0) return TCHLL_OK;
    // small graphs, and road networks without a long list, refuse what the hub
    // core's passes refuse in others
    P.check_ids = (direct_pass ? (uintptr_t)P.col_idx % 16 == 0 : pairs && road) && T.hub != 0 && hub_pad_usable(P, W) &&
                  (mode == MODE_EXACT || (mode == 2 && (uintptr_t)P.regs % 16 == 0));
    if (T.pairs && !details && !prepared && P.n_edges <= kDirectEdges) P.chunk = given_chunk(P.n_edges, T.chunk);
    if (col_ready && !(mode == MODE_EXACT && pairs)) {
        TCHLL_CUDA(cudaStreamWaitEvent(st, col_ready, 0));
        col_ready = nullptr;
    }
    int rc;
    set_hub(P, W, T);
    const int hub = P.hub;
    PhaseScope ps;
    phase_reset(ps);
    switch (mode) {
        case MODE_EXACT:
            if (direct_pass) {
                P.work = nullptr;
                phase_mark(ps, 1, st);
                rc = sparse ? pair_pass<false>(P, W, T, PASS_SHORT, nullptr, st) : launch_count<MODE_EXACT>(P, T, false, st);
                phase_mark(ps, 2, st);
                phase_used(ps, 1);
                return rc;
            }
            if (pairs) {
                // the hub core pass runs on the side stream beside the first
                // pass and the scatter; the hub kernels wait for it.  While
                // col_idx is still being copied, the core pass and the
                // short-list pairs, which read it, wait for it, the latter
                // after the scatter.
                phase_mark(ps, 0, st);
                P.chunk = pass_chunk(P.n_edges, T.chunk);
                rc = pass_prepare(P, W, 1, nullptr, 0, st);
                if (rc) return rc;
                SideFork fork;
                const bool side = hub > 0 && T.overlap && hub_pad_usable(P, W) && !road;
                if (side) {
                    rc = fork.begin(st);
                    if (rc == TCHLL_OK && col_ready) {
                        const cudaError_t e = cudaStreamWaitEvent(fork.stream(), col_ready, 0);
                        if (e != cudaSuccess) rc = cuda_status(e, "cudaStreamWaitEvent(col_ready)");
                    }
                    if (rc == TCHLL_OK) rc = launch_core_pass(P, W, T, false, ps, fork.stream());
                    if (rc == TCHLL_OK) rc = fork.mark();
                    if (rc) return rc;
                }
                const bool split = col_ready != nullptr;
                CountParams H = P;
                if (split) H.check_ids = 0;  // col_idx is not there yet
                rc = pair_pass<false>(H, W, T, split ? PASS_HIST : PASS_HIST | PASS_SHORT, road ? nullptr : W.ctr,
                                      st);
                if (rc == TCHLL_OK) rc = hub_alloc(P, W, T.hub_seg, st);
                if (rc == TCHLL_OK) rc = pairs_scatter(P, W, st);
                if (rc) return rc;
                if (split) {
                    TCHLL_CUDA(cudaStreamWaitEvent(st, col_ready, 0));
                    rc = pair_pass<false>(P, W, T, PASS_SHORT, W.ctr + 1, st);
                    if (rc) return rc;
                }
                rc = launch_table_pairs(P, W, T, st);
                if (rc) return rc;
                phase_mark(ps, 1, st);
                if (hub > 0) {
                    rc = side ? fork.wait_mark() : launch_core_pass(P, W, T, road, ps, st);
                    if (rc == TCHLL_OK) rc = launch_hub(P, W, T, ps, st);
                }
                phase_mark(ps, 2, st);
                const int rj = fork.end();
                phase_used(ps, 0, 1);
                return rc ? rc : rj;
            }
            P.work = W.ctr;
            phase_mark(ps, 1, st);
            rc = launch_count<MODE_EXACT>(P, T, details, st);
            phase_mark(ps, 2, st);
            phase_used(ps, 1);
            return rc;
        case MODE_HYBRID:  // one fused launch over the edges as given
            P.work = W.ctr;
            phase_mark(ps, 1, st);
            rc = launch_count<MODE_HYBRID>(P, T, details, st);
            phase_mark(ps, 2, st);
            phase_used(ps, 1);
            return rc;
        case 2:  // split: exact-routed edges, then HLL-routed edges
            if (pairs && ((uintptr_t)P.regs % 16 == 0)) {
                // One first pass routes: it counts the short-list exact pairs
                // (and n_fallback), lists the hub pairs' table sides and the
                // HLL edges (estimated by hll_edges_kernel, which counts
                // n_approx / n_clamped).  The HLL pass needs only that pass
                // and runs on the side stream beside the scatter and the hub
                // kernels (all add integers into the same result block).
                P.work = W.ctr;
                P.hll_u = HW.hll_u;
                P.hll_v = HW.hll_v;
                P.hll_n = HW.hll_n;
                phase_mark(ps, 0, st);
                P.chunk = pass_chunk(P.n_edges, T.chunk);
                rc = pass_prepare(P, W, 1, nullptr, 0, st);
                if (rc) return rc;
                // side stream: the hub core pass (the hub kernels wait for
                // it) and the zero masks beside the first pass, then, once
                // that has listed the HLL edges, their pass
                SideFork fork;
                cudaStream_t hst = st;
                const bool core_side = hub > 0 && T.overlap && hub_pad_usable(P, W) && !road;
                if (T.overlap) {
                    rc = fork.begin(st);
                    if (rc) return rc;
                    hst = fork.stream();
                    if (core_side) {
                        rc = launch_core_pass(P, W, T, false, ps, hst);
                        if (rc == TCHLL_OK) rc = fork.mark();
                        if (rc) return rc;
                    }
                }
                rc = launch_zmask(P, HW, hst);
                if (rc == TCHLL_OK) rc = pair_pass<true>(P, W, T, PASS_HIST | PASS_SHORT, road ? nullptr : W.ctr, st);
                if (rc == TCHLL_OK && T.overlap) rc = fork.side_waits_caller();
                if (rc) return rc;
                if (ps.active()) cudaEventRecord(g_phase.hll_ev[0], hst);
                rc = launch_hll_edges(P, HW, T, hst);
                if (ps.active()) cudaEventRecord(g_phase.hll_ev[1], hst);
                if (rc == TCHLL_OK) rc = hub_alloc(P, W, T.hub_seg, st);
                if (rc == TCHLL_OK) rc = pairs_scatter(P, W, st);
                if (rc == TCHLL_OK) rc = launch_table_pairs(P, W, T, st);
                if (rc) return rc;
                phase_mark(ps, 1, st);
                if (hub > 0) {
                    rc = core_side ? fork.wait_mark() : launch_core_pass(P, W, T, road, ps, st);
                    if (rc == TCHLL_OK) rc = launch_hub(P, W, T, ps, st);
                    if (rc) return rc;
                }
                phase_mark(ps, 2, st);
                rc = fork.end();
                phase_used(ps, 0, 1, 2);
                if (ps.active()) g_phase.hll_split = true;
                return rc;
            }
            if (direct_pass && ((uintptr_t)P.regs % 16 == 0)) {
                // the pass lists the HLL edges for hll_edges_kernel
                P.hll_u = HW.hll_u;
                P.hll_v = HW.hll_v;
                P.hll_n = HW.hll_n;
                phase_mark(ps, 1, st);
                P.work = nullptr;
                rc = sparse ? pair_pass<true>(P, W, T, PASS_SHORT, nullptr, st)
                            : launch_count<MODE_HYB_EXACT>(P, T, false, st);
                if (rc) return rc;
                phase_mark(ps, 2, st);
                rc = launch_zmask(P, HW, st);
                if (rc == TCHLL_OK) rc = launch_hll_edges(P, HW, T, st);
                phase_mark(ps, 3, st);
                phase_used(ps, 1, 2);
                return rc;
            }
            P.work = W.ctr;
            phase_mark(ps, 1, st);
            rc = launch_count<MODE_HYB_EXACT>(P, T, details, st);
            if (rc) return rc;
            phase_mark(ps, 2, st);
            P.work = W.ctr + 1;
            rc = launch_count<MODE_HYB_HLL>(P, T, details, st);
            phase_mark(ps, 3, st);
            phase_used(ps, 1, 2);
            return rc;
        default:
            set_error("unknown count mode %d", mode);
            return TCHLL_EINVAL;
    }
}

static int check_common(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx, int64_t nnz,
                        const int32_t* eu, const int32_t* ev, int64_t n_edges, tchll_count_result* result) {
    TCHLL_ARG(n_nodes >= 0 && nnz >= 0 && n_edges >= 0, "negative size");
    TCHLL_ARG(n_nodes < (int64_t)INT32_MAX && nnz <= (int64_t)INT32_MAX && n_edges <= (int64_t)INT32_MAX,
              "int32 CSR limits exceeded");
    TCHLL_ARG(result != nullptr, "result pointer is null");
    TCHLL_ARG(n_edges == 0 || (eu && ev && row_ptr), "null edge or row_ptr pointer");
    TCHLL_ARG(nnz == 0 || col_idx, "null col_idx");
    return TCHLL_OK;
}

}  // namespace tchll

using namespace tchll;

TCHLL_EXPORT int tchll_count_workspace_bytes(int64_t n_nodes, int64_t n_edges, size_t* bytes) {
    TCHLL_ARG(bytes != nullptr && n_nodes >= 0 && n_edges >= 0, "bad arguments");
    CountWs W;
    HybridWs H;
    carve_count_hybrid(nullptr, 0, n_nodes, n_edges, 0, 4, W, H, bytes);  // covers the exact-only layout too
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_hybrid_workspace_bytes(int64_t n_nodes, int64_t n_edges, int64_t n_rows, int32_t p,
                                              size_t* bytes) {
    TCHLL_ARG(bytes != nullptr && n_nodes >= 0 && n_edges >= 0 && n_rows >= 0, "bad arguments");
    TCHLL_ARG(p >= 4 && p <= 16, "p must be in [4, 16], got %d", p);
    CountWs W;
    HybridWs H;
    carve_count_hybrid(nullptr, 0, n_nodes, n_edges, n_rows, p, W, H, bytes);
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_exact_count(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx, int64_t nnz,
                                   const int32_t* edge_u, const int32_t* edge_v, int64_t n_edges,
                                   int64_t* per_edge_support, tchll_count_result* result, void* workspace,
                                   size_t workspace_bytes, void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, result);
    if (rc) return rc;
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.pe_support = per_edge_support;
    P.result = result;
    P.p = 4;
    return run_count(P, MODE_EXACT, per_edge_support != nullptr, workspace, workspace_bytes, (cudaStream_t)stream);
}

TCHLL_EXPORT int tchll_exact_count_staged(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx,
                                          int64_t nnz, const int32_t* edge_u, const int32_t* edge_v,
                                          int64_t n_edges, tchll_count_result* result, void* workspace,
                                          size_t workspace_bytes, void* col_ready_event, void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, result);
    if (rc) return rc;
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.result = result;
    P.p = 4;
    return run_count(P, MODE_EXACT, false, workspace, workspace_bytes, (cudaStream_t)stream,
                     (cudaEvent_t)col_ready_event);
}

TCHLL_EXPORT int tchll_count_hub_threshold(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx, int64_t nnz,
                                           const int32_t* edge_u, const int32_t* edge_v, int64_t n_edges,
                                           void* workspace, size_t workspace_bytes, int32_t* out, void* stream) {
    tchll_count_result unused;
    const int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, &unused);
    if (rc) return rc;
    TCHLL_ARG(out != nullptr, "null output");
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    const Tuning T = tuning_snapshot();
    CountWs W;
    size_t need = 0;
    bool ok = carve_count(workspace, workspace_bytes, n_nodes, n_edges, W, &need, true);
    if (!ok) ok = carve_count(workspace, workspace_bytes, n_nodes, n_edges, W, &need, false);
    if (!ok || workspace == nullptr) {
        set_error("workspace too small: need %zu bytes, have %zu", need, workspace_bytes);
        return TCHLL_EWORKSPACE;
    }
    set_hub(P, W, T);
    *out = P.hub;
    if (!P.hub_alt || n_edges == 0) return TCHLL_OK;
    unsigned long long est[kEst];
    int r = pass_prepare(P, W, 0, nullptr, 0, (cudaStream_t)stream);
    if (r == TCHLL_OK) r = fetch_small(est, P.est, sizeof(est), (cudaStream_t)stream);
    if (r == TCHLL_OK) *out = choose(est, n_edges, P.hub, P.hub_alt, false).hub;
    return r;
}

static int hybrid_common(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx, int64_t nnz,
                         const int32_t* edge_u, const int32_t* edge_v, int64_t n_edges, const int32_t* degrees,
                         const uint8_t* regs, int64_t n_rows, const int64_t* slot, const uint8_t* has, int32_t p,
                         int64_t gamma, int32_t mode, int64_t* pe_support, double* pe_s_hat, double* pe_s_cl,
                         uint8_t* pe_method, tchll_count_result* result, void* ws, size_t wsb, void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, result);
    if (rc) return rc;
    TCHLL_ARG(p >= 4 && p <= 16, "p must be in [4, 16], got %d", p);
    TCHLL_ARG(n_edges == 0 || degrees, "degrees is null");
    TCHLL_ARG(n_rows == 0 || regs, "register rows are null");
    TCHLL_ARG(slot || has || n_edges == 0, "need slot (compact) or has_sketch (dense)");
    const bool details = pe_support || pe_s_hat || pe_s_cl || pe_method;
    TCHLL_ARG(!details || (pe_support && pe_s_hat && pe_s_cl && pe_method),
              "per-edge outputs must be all set or all null");
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.degrees = degrees;
    P.regs = regs;
    P.n_rows = n_rows;
    P.slot = slot;
    P.has = has;
    P.p = p;
    P.gamma = gamma;
    P.pe_support = pe_support;
    P.pe_s_hat = pe_s_hat;
    P.pe_s_cl = pe_s_cl;
    P.pe_method = pe_method;
    P.result = result;
    return run_count(P, mode, details, ws, wsb, (cudaStream_t)stream);
}

TCHLL_EXPORT int tchll_hybrid_count_dense(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx,
                                          int64_t nnz, const int32_t* edge_u, const int32_t* edge_v,
                                          int64_t n_edges, const int32_t* degrees, const uint8_t* sketch_regs,
                                          const uint8_t* has_sketch, int32_t p, int64_t gamma,
                                          int32_t split_kernels, tchll_count_result* result, void* workspace,
                                          size_t workspace_bytes, void* stream) {
    return hybrid_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, degrees, sketch_regs, n_nodes,
                         nullptr, has_sketch, p, gamma, split_kernels ? 2 : MODE_HYBRID, nullptr, nullptr, nullptr,
                         nullptr, result, workspace, workspace_bytes, stream);
}

TCHLL_EXPORT int tchll_hybrid_count_compact(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx,
                                            int64_t nnz, const int32_t* edge_u, const int32_t* edge_v,
                                            int64_t n_edges, const int32_t* degrees, const uint8_t* rows,
                                            int64_t n_rows, const int64_t* slot, int32_t p, int64_t gamma,
                                            int32_t split_kernels, int64_t* per_edge_support,
                                            double* per_edge_s_hat, double* per_edge_s_clamped,
                                            uint8_t* per_edge_method, tchll_count_result* result,
                                            void* workspace, size_t workspace_bytes, void* stream) {
    TCHLL_ARG(slot != nullptr || n_edges == 0, "slot is null");
    return hybrid_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, degrees, rows, n_rows, slot,
                         nullptr, p, gamma, split_kernels ? 2 : MODE_HYBRID, per_edge_support, per_edge_s_hat,
                         per_edge_s_clamped, per_edge_method, result, workspace, workspace_bytes, stream);
}

TCHLL_EXPORT int tchll_set_count_tuning(int32_t chunk, int32_t slots_log2, int32_t tiny, int32_t blocks_per_sm) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    TCHLL_ARG(chunk >= 32 && chunk % 32 == 0 && chunk <= (1 << 20), "chunk must be a multiple of 32 in [32, 2^20]");
    TCHLL_ARG(tiny >= 0 && tiny <= 4096, "tiny must be in [0, 4096]");
    TCHLL_ARG(blocks_per_sm >= 0 && blocks_per_sm <= 32, "blocks_per_sm must be in [0, 32]");
    TCHLL_ARG(slots_log2 >= 6 && slots_log2 <= 15 && (size_t)g_tuning.warps * ((size_t)4 << slots_log2) <= 227 * 1024,
              "slots_log2 must be in [6, 15] with warps x 2^slots_log2 x 4 bytes within 227 KB of shared memory");
    g_tuning.chunk = chunk;
    g_tuning.slots_log2 = slots_log2;
    g_tuning.tiny = tiny;
    g_tuning.blocks_per_sm = blocks_per_sm;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_set_count_shape(int32_t warps_per_cta, int32_t pairs) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    TCHLL_ARG(warps_per_cta >= 1 && warps_per_cta <= 8, "warps_per_cta must be in [1, 8]");
    TCHLL_ARG((size_t)warps_per_cta * ((size_t)4 << g_tuning.slots_log2) <= 227 * 1024,
              "warps x 2^slots_log2 x 4 bytes must fit 227 KB of shared memory");
    g_tuning.warps = warps_per_cta;
    g_tuning.pairs = pairs == 2 ? 2 : (pairs ? 1 : 0);
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_set_count_table(int32_t sparse) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    g_tuning.sparse = sparse ? 1 : 0;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_set_count_hub(int32_t threshold, int32_t seg_pairs, int32_t table_log2, int32_t unroll) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    TCHLL_ARG(threshold == kHubAuto || threshold == 0 || threshold >= HUB_MIN,
              "hub threshold must be -1 (automatic), 0 (off) or >= %d", HUB_MIN);
    TCHLL_ARG(seg_pairs >= HUB_SEG_MIN && seg_pairs <= (1 << 20), "seg_pairs must be in [%d, 2^20]", HUB_SEG_MIN);
    TCHLL_ARG(table_log2 >= 10 && table_log2 <= 15, "table_log2 must be in [10, 15]");
    TCHLL_ARG(unroll == 2 || unroll == 4, "unroll must be 2 or 4");
    g_tuning.hub = threshold;
    g_tuning.hub_seg = seg_pairs;
    g_tuning.hub_lg = table_log2;
    g_tuning.hub_unroll = unroll;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_get_count_hub(int32_t* out4) {
    TCHLL_ARG(out4 != nullptr, "null output");
    const Tuning T = tuning_snapshot();
    out4[0] = T.hub;
    out4[1] = T.hub_seg;
    out4[2] = T.hub_lg;
    out4[3] = T.hub_unroll;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_set_count_core(int32_t bitmap_log2, int32_t overlap, int32_t packed, int32_t bank_sort) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    TCHLL_ARG(bitmap_log2 == 0 || (bitmap_log2 >= 10 && bitmap_log2 <= 17),
              "bitmap_log2 must be 0 (hash tables only) or in [10, 17] (1 KB .. 128 KB of shared memory)");
    g_tuning.bitmap_lg = bitmap_log2;
    TCHLL_ARG(overlap >= 0 && overlap <= 2, "overlap must be 0, 1 or 2");
    g_tuning.overlap = overlap;
    g_tuning.packed = packed ? 1 : 0;
    g_tuning.bank_sort = bank_sort ? 1 : 0;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_get_count_core(int32_t* out4) {
    TCHLL_ARG(out4 != nullptr, "null output");
    const Tuning T = tuning_snapshot();
    out4[0] = T.bitmap_lg;
    out4[1] = T.overlap;
    out4[2] = T.packed;
    out4[3] = T.bank_sort;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_set_hll_pass(int32_t row_cache_max_p, int32_t lanes) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    TCHLL_ARG(row_cache_max_p >= 0 && row_cache_max_p <= 16, "row_cache_max_p must be in [0, 16]");
    TCHLL_ARG(lanes == 0 || (lanes >= 1 && lanes <= 32 && (lanes & (lanes - 1)) == 0),
              "lanes must be 0 (automatic) or a power of two in [1, 32]");
    g_tuning.hll_row_cache_p = row_cache_max_p;
    g_tuning.hll_lanes = lanes;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_get_hll_pass(int32_t* out2) {
    TCHLL_ARG(out2 != nullptr, "null output");
    const Tuning T = tuning_snapshot();
    out2[0] = T.hll_row_cache_p;
    out2[1] = T.hll_lanes;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_get_count_tuning(int32_t* out8) {
    TCHLL_ARG(out8 != nullptr, "out is null");
    const Tuning T = tuning_snapshot();
    out8[0] = T.chunk;
    out8[1] = T.slots_log2;
    out8[2] = T.tiny;
    out8[3] = T.blocks_per_sm;
    out8[4] = T.warps;
    out8[5] = T.pairs;
    out8[6] = T.sparse;
    out8[7] = 0;  // reserved
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_set_phase_timing(int32_t enable) {
    std::lock_guard<std::mutex> lock(g_phase_mu);
    if (enable && !g_phase.made) {
        for (int i = 0; i < 4; ++i) TCHLL_CUDA(cudaEventCreate(&g_phase.ev[i]));
        for (int i = 0; i < 4; ++i) TCHLL_CUDA(cudaEventCreate(&g_phase.hub_ev[i]));
        for (int i = 0; i < 2; ++i) TCHLL_CUDA(cudaEventCreate(&g_phase.hll_ev[i]));
        g_phase.made = true;
    }
    g_phase.on = enable != 0;
    for (int i = 0; i < 3; ++i) g_phase.used[i] = false;
    g_phase.hub_used = false;
    g_phase.core_used = false;
    g_phase.hll_split = false;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_phase_times(float* ms3) {
    TCHLL_ARG(ms3 != nullptr, "out is null");
    std::lock_guard<std::mutex> lock(g_phase_mu);
    for (int i = 0; i < 3; ++i) ms3[i] = -1.0f;
    if (!g_phase.on || !g_phase.made) return TCHLL_OK;
    for (int i = 0; i < 3; ++i) {
        if (!g_phase.used[i]) continue;
        if (i == 2 && g_phase.hll_split) {  // the HLL pass ran beside phase 1
            TCHLL_CUDA(cudaEventSynchronize(g_phase.hll_ev[1]));
            TCHLL_CUDA(cudaEventElapsedTime(&ms3[i], g_phase.hll_ev[0], g_phase.hll_ev[1]));
            continue;
        }
        TCHLL_CUDA(cudaEventSynchronize(g_phase.ev[i + 1]));
        TCHLL_CUDA(cudaEventElapsedTime(&ms3[i], g_phase.ev[i], g_phase.ev[i + 1]));
    }
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_phase_hub_ms(float* ms2) {
    TCHLL_ARG(ms2 != nullptr, "out is null");
    std::lock_guard<std::mutex> lock(g_phase_mu);
    ms2[0] = ms2[1] = -1.0f;
    if (!g_phase.on || !g_phase.made || !g_phase.hub_used) return TCHLL_OK;
    TCHLL_CUDA(cudaEventSynchronize(g_phase.hub_ev[3]));
    TCHLL_CUDA(cudaEventElapsedTime(&ms2[0], g_phase.hub_ev[2], g_phase.hub_ev[3]));
    if (g_phase.core_used) TCHLL_CUDA(cudaEventElapsedTime(&ms2[1], g_phase.hub_ev[0], g_phase.hub_ev[1]));
    return TCHLL_OK;
}

// ------------------------------------------------ allocation-free variant ---
// Some callers hold device pointers to a graph but cannot allocate device
// memory themselves: a language binding without its own CUDA allocator, or a
// service that hands all device memory to one arena up front and forbids
// allocation on the request path.  tchll_exact_count_noalloc serves them with
// the same exact count, taking its scratch (the pair list, histogram and work
// counters) from this fixed array instead of a caller workspace.  Every GPU
// that loads the library reserves the array until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[TCHLL_NOALLOC_SCRATCH_BYTES];

// Host code must not pass g_noalloc_scratch itself to a kernel (on the host
// the name stands for a host-side shadow, not the device array): the device
// address comes from cudaGetSymbolAddress, with the device current.  The
// address belongs to the module as loaded in one CUDA context, so it is
// cached per context, keyed by the context's process-unique id (cuCtxGetId,
// reached through the runtime's driver entry-point query, so the library
// needs no driver link): a non-primary context made current by a caller, or
// a primary context re-created after cudaDeviceReset, gets its own lookup.
// Where the id cannot be read, every call looks the address up again.
static std::mutex g_noalloc_mu;
struct NoallocEntry {
    unsigned long long ctx_id;
    void* ptr;
};
static NoallocEntry g_noalloc_cache[64];
static int g_noalloc_used = 0;

static int noalloc_scratch_ptr(void** out) {
    int dev = -1;
    TCHLL_CUDA(cudaGetDevice(&dev));  // also makes the runtime's context current
    unsigned long long id = 0;
    const bool have_id = current_ctx_id(&id);
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (have_id) {
        for (int i = 0; i < g_noalloc_used; ++i)
            if (g_noalloc_cache[i].ctx_id == id) {
                *out = g_noalloc_cache[i].ptr;
                return TCHLL_OK;
            }
    }
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(noalloc scratch)");
    if (have_id) {  // a full table gives up the entry the id hashes to
        const int slot = g_noalloc_used < 64 ? g_noalloc_used++ : (int)(id % 64);
        g_noalloc_cache[slot] = NoallocEntry{id, p};
    }
    *out = p;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_exact_count_noalloc(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx,
                                           int64_t nnz, const int32_t* edge_u, const int32_t* edge_v,
                                           int64_t n_edges, tchll_count_result* result, void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, result);
    if (rc) return rc;
    CountWs W;
    size_t need = 0;
    carve_count(nullptr, 0, n_nodes, n_edges, W, &need, false);  // padded lists only when they fit too
    if (need > (size_t)TCHLL_NOALLOC_SCRATCH_BYTES) {
        set_error("graph too large for tchll_exact_count_noalloc: needs %zu bytes of scratch (about 4 per edge + "
                  "32 per vertex), the fixed limit is %u bytes; use tchll_exact_count with a workspace",
                  need, (unsigned)TCHLL_NOALLOC_SCRATCH_BYTES);
        return TCHLL_EINVAL;
    }
    void* scratch = nullptr;
    rc = noalloc_scratch_ptr(&scratch);
    if (rc) return rc;
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.result = result;
    P.p = 4;
    // run_count clears the work counters, histogram and result on the stream
    // before any kernel reads them, so leftovers of the previous call are
    // harmless; calls that overlap on the GPU would share the array and race.
    return run_count(P, MODE_EXACT, false, scratch, TCHLL_NOALLOC_SCRATCH_BYTES, (cudaStream_t)stream);
}

// ------------------------------------------------------------- batched ------
// Many graphs in one launch.  The graphs share one CSR with disjoint vertex
// ranges [vbase[g], vbase[g+1]) (ids offset per graph before the CSR build:
// orientation and compaction are per vertex, so each graph's part of the CSR
// equals its own CSR shifted).  Work is a list of chunks that never cross a
// graph; each chunk adds its integer totals to results[g], so per-graph
// results are bit-identical to one graph at a time.

// Edge range of graph g; false when its vertex range or its edge range is
// malformed (no vbase entry is used as an index unchecked, and no edge outside
// [0, n_edges) is ever in a range).
__device__ __forceinline__ bool graph_range(const int32_t* row_ptr, const int32_t* vbase, int64_t g, int64_t n_nodes,
                                            int64_t n_edges, int64_t& s0, int64_t& s1) {
    const int32_t a = vbase[g], b = vbase[g + 1];
    if (a < 0 || b < a || (int64_t)b > n_nodes) return false;
    s0 = row_ptr[a];
    s1 = row_ptr[b];
    return s0 >= 0 && s1 >= s0 && s1 <= n_edges;
}

// The chunks of the graphs before the first malformed one (*bad of
// check_vbase_kernel).  Neighbouring graphs share a bound, so these ranges
// do not overlap and their chunks fit the list; behind a malformed graph
// neither is sure, so the graphs there are refused as well.
__global__ void chunk_count_kernel(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ vbase,
                                   int64_t n_graphs, int64_t n_nodes, int64_t n_edges, int chunk,
                                   const unsigned long long* __restrict__ bad, int64_t* cnt,
                                   tchll_count_result* results) {
    const int64_t good = n_graphs - (int64_t)*bad;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g <= n_graphs;
         g += (int64_t)gridDim.x * blockDim.x) {
        int64_t s0 = 0, s1 = 0;
        if (g < good) graph_range(row_ptr, vbase, g, n_nodes, n_edges, s0, s1);
        else if (g < n_graphs) results[g].status |= ST_BAD_ROW;
        cnt[g] = (s1 - s0 + chunk - 1) / chunk;
    }
}

__global__ void chunk_fill_kernel(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ vbase,
                                  int64_t n_graphs, int64_t n_nodes, int64_t n_edges, int chunk,
                                  const int64_t* __restrict__ coff, int64_t* cstart, int32_t* clen, int32_t* cgraph) {
    // one warp per graph
    const int lane = threadIdx.x & 31;
    for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < n_graphs;
         g += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t n = coff[g + 1] - coff[g];
        int64_t s0 = 0, s1 = 0;
        if (n == 0 || !graph_range(row_ptr, vbase, g, n_nodes, n_edges, s0, s1)) continue;
        for (int64_t k = lane; k < n; k += 32) {
            const int64_t st = s0 + k * chunk;
            cstart[coff[g] + k] = st;
            clen[coff[g] + k] = (int32_t)min((int64_t)chunk, s1 - st);
            cgraph[coff[g] + k] = (int32_t)g;
        }
    }
}

// *bad (zeroed before) = n_graphs less the first malformed graph, 0 when there
// is none; *largest the vertices of the largest graph, if more than the packed
// lists' core.  Without edges (row_ptr null) only the vertex ranges count.
__global__ void check_vbase_kernel(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ vbase,
                                   int64_t n_graphs, int64_t n_nodes, int64_t n_edges, unsigned long long* bad,
                                   unsigned long long* largest, tchll_count_result* results) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n_graphs;
         g += (int64_t)gridDim.x * blockDim.x) {
        int64_t s0, s1;
        bool ok;
        if (row_ptr) {
            ok = graph_range(row_ptr, vbase, g, n_nodes, n_edges, s0, s1);
        } else {
            const int32_t a = vbase[g], b = vbase[g + 1];
            ok = a >= 0 && b >= a && (int64_t)b <= n_nodes;
        }
        if (ok) {
            const int32_t n = vbase[g + 1] - vbase[g];
            if (largest && n > kCore16Max) atomicMax(largest, (unsigned long long)n);
            if (largest && n >= kBigGraph) largest[1] = 1;
            continue;
        }
        results[g].status |= ST_BAD_ROW;
        if (bad) atomicMax(bad, (unsigned long long)(n_graphs - g));
    }
}

struct BatchWs {
    CountWs cw;
    HybridWs hw;      // HLL edge list (no zero masks)
    int64_t* cnt;     // n_graphs + 1
    int64_t* coff;    // n_graphs + 1 (last entry: number of chunks)
    int64_t* cstart;  // max chunks
    int32_t* clen;
    int32_t* cgraph;
    uint2* codes;     // n_edges / 32 + max chunks + 1
    int32_t* ghub;    // n_graphs: GRAPH_*
    int32_t* rflag;   // n_nodes / 64 + 1: 64 rows touch such a graph
    int32_t* rlist;   // those blocks
    int32_t* big;     // 512 words per kBigGraph vertices
    size_t flag_bytes;  // of ghub, rflag and big, which are next to each other
    void* tmp;
    size_t tmp_bytes;
};

static int64_t max_chunks(int64_t n_edges, int64_t n_graphs, int chunk) {
    return n_edges / chunk + n_graphs + 1;
}

static bool carve_batch(void* ws, size_t bytes, int64_t n_nodes, int64_t n_edges, int64_t n_graphs, BatchWs& B,
                        size_t* need) {
    size_t cneed = 0;
    carve_count(nullptr, 0, n_nodes, n_edges, B.cw, &cneed);
    const size_t G = (size_t)n_graphs + 1;
    const size_t MC = (size_t)max_chunks(n_edges, n_graphs, 32);  // any chunk size >= 32 fits
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (int64_t*)nullptr, (int64_t*)nullptr, (int)G);
    Carve cv(ws, bytes);
    char* cbase = cv.take<char>(cneed);
    B.cnt = cv.take<int64_t>(G);
    B.coff = cv.take<int64_t>(G);
    B.cstart = cv.take<int64_t>(MC);
    B.clen = cv.take<int32_t>(MC);
    B.cgraph = cv.take<int32_t>(MC);
    B.codes = cv.take<uint2>((size_t)(n_edges > 0 ? n_edges : 1) / 32 + MC + 1);
    const size_t RL = (size_t)(n_nodes > 0 ? n_nodes : 0) / 64 + 1;
    const size_t BG = 512 * ((size_t)(n_nodes > 0 ? n_nodes : 0) / kBigGraph + 1);
    B.flag_bytes = (G + RL + BG) * sizeof(int32_t);
    B.ghub = cv.take<int32_t>(G + 2 * RL + BG);
    B.rflag = B.ghub + G;
    B.big = B.rflag + RL;
    B.rlist = B.big + BG;
    B.tmp_bytes = tb;
    B.tmp = cv.take<char>(tb);
    const size_t E = (size_t)(n_edges > 0 ? n_edges : 1);
    B.hw.hll_u = cv.take<int32_t>(E);
    B.hw.hll_v = cv.take<int32_t>(E);
    B.hw.zm = nullptr;
    B.hw.zst = 0;
    B.hw.lc = nullptr;
    if (need) *need = cv.off;
    if (!cv.ok() || cv.dry) return cv.ok();
    carve_count(cbase, cneed, n_nodes, n_edges, B.cw, nullptr);
    B.hw.hll_n = B.cw.ctr + 4;
    B.cw.codes = B.codes;
    return true;
}

// Chunk list over the graphs' edge ranges [row_ptr[vbase[g]],
// row_ptr[vbase[g+1]]), after check_vbase.
static int build_chunks(const CountParams& P, const int32_t* vbase, int64_t n_graphs, const BatchWs& B, int chunk,
                        cudaStream_t st) {
    int64_t g = (n_graphs + 256) / 256;
    if (g > (int64_t)sm_count() * 8) g = (int64_t)sm_count() * 8;
    chunk_count_kernel<<<(int)g, 256, 0, st>>>(P.row_ptr, vbase, n_graphs, P.n_nodes, P.n_edges, chunk, P.graph_bad,
                                               B.cnt, P.result);
    TCHLL_CHECK_LAUNCH("chunk_count_kernel");
    size_t tb = B.tmp_bytes;
    TCHLL_CUDA(cub::DeviceScan::ExclusiveSum(B.tmp, tb, B.cnt, B.coff, (int)(n_graphs + 1), st));
    count_launch();
    int64_t gw = (n_graphs * 32 + 255) / 256;
    if (gw > (int64_t)sm_count() * 8) gw = (int64_t)sm_count() * 8;
    if (gw < 1) gw = 1;
    chunk_fill_kernel<<<(int)gw, 256, 0, st>>>(P.row_ptr, vbase, n_graphs, P.n_nodes, P.n_edges, chunk, B.coff,
                                               B.cstart, B.clen, B.cgraph);
    TCHLL_CHECK_LAUNCH("chunk_fill_kernel");
    return TCHLL_OK;
}

static int check_vbase(const CountParams& P, const int32_t* vbase, int64_t n_graphs, cudaStream_t st) {
    int64_t g = (n_graphs + 255) / 256;
    if (g > 1024) g = 1024;
    check_vbase_kernel<<<(int)g, 256, 0, st>>>(P.n_edges > 0 ? P.row_ptr : nullptr, vbase, n_graphs, P.n_nodes,
                                               P.n_edges, P.graph_bad, P.est ? P.est + 4 : nullptr, P.result);
    TCHLL_CHECK_LAUNCH("check_vbase_kernel");
    return TCHLL_OK;
}

static int run_batch(CountParams P, bool hybrid, const int32_t* vbase, int64_t n_graphs, void* ws, size_t wsb,
                     cudaStream_t st) {
    const Tuning T = tuning_snapshot();
    BatchWs B;
    size_t need = 0;
    if (!carve_batch(ws, wsb, P.n_nodes, P.n_edges, n_graphs, B, &need) || ws == nullptr) {
        set_error("workspace too small: need %zu bytes, have %zu", need, wsb);
        return TCHLL_EWORKSPACE;
    }
    if (n_graphs == 0 || P.n_edges == 0) TCHLL_CUDA(cudaMemsetAsync(P.result, 0, sizeof(tchll_count_result) * n_graphs, st));
    if (n_graphs == 0) return TCHLL_OK;
    P.chunk = T.chunk;
    P.slots_log2 = T.slots_log2;
    P.tiny = T.tiny;
    P.sparse = T.sparse;
    P.graph_vbase = vbase;
    P.n_graphs = n_graphs;
    P.graph_bad = P.n_edges > 0 ? B.cw.ctr + 6 : nullptr;
    P.n_chunks_dev = B.coff + n_graphs;
    P.chunk_start = B.cstart;
    P.chunk_len = B.clen;
    P.chunk_graph = B.cgraph;
    P.graph_hub = B.ghub;
    P.live_flag = B.rflag;
    P.live_list = B.rlist;
    P.n_live = B.cw.ncore + kCoreWords - 1;
    P.big_hist = B.big;
    int rc;
    if (P.n_edges == 0) return check_vbase(P, vbase, n_graphs, st);
    PhaseScope ps;
    phase_reset(ps);
    // Hybrid: the routing pass also appends the HLL-routed edges to a list
    // (16-byte aligned register rows; else the HLL edges take a second pass
    // over each graph's edges below).
    const bool hll_list = hybrid && ((uintptr_t)P.regs % 16 == 0);
    P.hll_u = hll_list ? B.hw.hll_u : nullptr;
    P.hll_v = hll_list ? B.hw.hll_v : nullptr;
    P.hll_n = hll_list ? B.hw.hll_n : nullptr;
    phase_mark(ps, 0, st);
    // one pass over each graph's edges as given; pairs with a long table side
    // go to the hub kernels, which publish per segment into the graph of x
    set_hub(P, B.cw, T);
    const int hub = P.hub;
    rc = pass_prepare(P, B.cw, n_graphs, reinterpret_cast<uint32_t*>(B.ghub), (int64_t)(B.flag_bytes / 4), st);
    if (rc == TCHLL_OK) rc = check_vbase(P, vbase, n_graphs, st);
    if (rc == TCHLL_OK) rc = build_chunks(P, vbase, n_graphs, B, T.chunk, st);
    if (rc) return rc;
    if (hybrid) rc = pair_pass<true>(P, B.cw, T, PASS_HIST | PASS_SHORT, B.cw.ctr, st);
    else rc = pair_pass<false>(P, B.cw, T, PASS_HIST | PASS_SHORT, B.cw.ctr, st);
    if (rc == TCHLL_OK) rc = hub_alloc(P, B.cw, T.hub_seg, st);
    if (rc == TCHLL_OK) rc = pairs_scatter(P, B.cw, st);
    if (rc == TCHLL_OK) rc = launch_table_pairs(P, B.cw, T, st);
    if (rc) return rc;
    phase_mark(ps, 1, st);
    if (hub > 0) {
        rc = launch_core_pass(P, B.cw, T, true, ps, st);
        if (rc == TCHLL_OK) rc = launch_hub(P, B.cw, T, ps, st, true);
        if (rc) return rc;
    }
    phase_mark(ps, 2, st);
    phase_used(ps, 0, 1);
    if (!hybrid) return TCHLL_OK;
    if (hll_list) {  // per-edge estimates into each edge's graph
        rc = launch_hll_edges(P, B.hw, T, st);
        phase_mark(ps, 3, st);
        phase_used(ps, 2);
        return rc;
    }
    // HLL-routed edges: chunks over each graph's CSR edge range
    P.work = B.cw.ctr + 1;
    rc = launch_count<MODE_HYB_HLL>(P, T, false, st);
    phase_mark(ps, 3, st);
    phase_used(ps, 2);
    return rc;
}

TCHLL_EXPORT int tchll_batch_workspace_bytes(int64_t n_nodes, int64_t n_edges, int64_t n_graphs, size_t* bytes) {
    TCHLL_ARG(bytes && n_nodes >= 0 && n_edges >= 0 && n_graphs >= 0, "bad arguments");
    BatchWs B;
    carve_batch(nullptr, 0, n_nodes, n_edges, n_graphs, B, bytes);
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_batch_exact_count(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx, int64_t nnz,
                                         const int32_t* edge_u, const int32_t* edge_v, int64_t n_edges,
                                         const int32_t* graph_vbase, int64_t n_graphs, tchll_count_result* results,
                                         void* workspace, size_t workspace_bytes, void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, results);
    if (rc) return rc;
    TCHLL_ARG(n_graphs >= 0 && (n_graphs == 0 || graph_vbase), "bad graph table");
    TCHLL_ARG(n_graphs < (int64_t)INT32_MAX, "too many graphs");
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.result = results;
    P.p = 4;
    return run_batch(P, false, graph_vbase, n_graphs, workspace, workspace_bytes, (cudaStream_t)stream);
}

TCHLL_EXPORT int tchll_batch_hybrid_count(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx,
                                          int64_t nnz, const int32_t* edge_u, const int32_t* edge_v,
                                          int64_t n_edges, const int32_t* degrees, const uint8_t* rows,
                                          int64_t n_rows, const int64_t* slot, int32_t p, int64_t gamma,
                                          const int32_t* graph_vbase, int64_t n_graphs,
                                          tchll_count_result* results, void* workspace, size_t workspace_bytes,
                                          void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, results);
    if (rc) return rc;
    TCHLL_ARG(p >= 4 && p <= 16, "p must be in [4, 16], got %d", p);
    TCHLL_ARG(n_edges == 0 || (degrees && slot), "degrees / slot are null");
    TCHLL_ARG(n_rows == 0 || rows, "register rows are null");
    TCHLL_ARG(n_graphs >= 0 && (n_graphs == 0 || graph_vbase), "bad graph table");
    TCHLL_ARG(n_graphs < (int64_t)INT32_MAX, "too many graphs");
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.degrees = degrees;
    P.regs = rows;
    P.n_rows = n_rows;
    P.slot = slot;
    P.p = p;
    P.gamma = gamma;
    P.result = results;
    return run_batch(P, true, graph_vbase, n_graphs, workspace, workspace_bytes, (cudaStream_t)stream);
}

// cpu_exp estimator variant (cpu_exp/triangle_hll_experiment.py:466-498,
// 652-710): dense registers for every vertex; an edge is exact iff
// min(d+u, d+v) <= threshold (threshold < 0: every edge HLL, the pure-HLL
// count).  Same kernels as the hybrid with gamma = threshold + 1.
TCHLL_EXPORT int tchll_cx_hybrid_count(const int32_t* row_ptr, int64_t n_nodes, const int32_t* col_idx, int64_t nnz,
                                       const int32_t* edge_u, const int32_t* edge_v, int64_t n_edges,
                                       const int32_t* degrees, const uint8_t* regs, const uint8_t* has_all,
                                       int32_t p, int64_t threshold, tchll_count_result* result, void* workspace,
                                       size_t workspace_bytes, void* stream) {
    int rc = check_common(row_ptr, n_nodes, col_idx, nnz, edge_u, edge_v, n_edges, result);
    if (rc) return rc;
    TCHLL_ARG(p >= 4 && p <= 16, "p must be in [4, 16], got %d", p);
    TCHLL_ARG(n_edges == 0 || (degrees && regs && has_all), "null degrees / registers");
    CountParams P{};
    P.row_ptr = row_ptr;
    P.n_nodes = n_nodes;
    P.col_idx = col_idx;
    P.nnz = nnz;
    P.edge_u = edge_u;
    P.edge_v = edge_v;
    P.n_edges = n_edges;
    P.degrees = degrees;
    P.regs = regs;
    P.n_rows = n_nodes;
    P.has = has_all;
    P.p = p;
    P.gamma = threshold < 0 ? 0 : threshold + 1;
    P.variant = 1;
    P.result = result;
    return run_count(P, 2, false, workspace, workspace_bytes, (cudaStream_t)stream);
}
