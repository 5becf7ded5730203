// csr.cu -- device construction of the oriented CSR.
//
// Reference semantics (ChitandaEruQ/triangle_counting_hll):
//   load + dedup   src/graph.py:8-26 (canonical (min,max), self-loops dropped,
//                  set semantics), experiment/exp_gpu.py:288-303 (np.unique)
//   compaction     experiment/exp_gpu.py:317-323 (np.union1d of endpoints;
//                  ids become ranks) == src/gpu_graph.py:19-37 node_index
//   degree/orient  src/graph.py:41-54, experiment/exp_gpu.py:325-339:
//                  u -> v iff (deg u, id u) < (deg v, id v); compaction is
//                  monotone, so comparing compacted ids gives the same order
//   CSR            experiment/exp_gpu.py:350-362 (np.lexsort by (src, dst))
//
// Pipeline: largest id (one 16-byte read-back) -> pack canonical pairs into
// 2k-bit keys, k = bits of the largest id -> radix sort -> unique -> node
// table and remap -> degree histogram -> orient -> stable radix sort of the
// (src, dst) pairs by src alone -> row pointers from the sorted sources.
// The node table (compacted id = rank of the raw id among the endpoints)
// comes from a direct table when the id space fits the workspace (degrees by
// id, a scan of the ids that occur: rank[id]), else from sorting and deduplicating all endpoints and a binary
// search per endpoint.
//
// One sort by src is enough for rows sorted by dst: the pairs reach it in
// canonical (a, b) order, a < b, and compaction keeps that order.  For a
// source s, the edges it gained by flipping (b = s, dst a < s) come before
// the edges it kept (a = s, dst b > s), each group in ascending dst, so a
// stable sort by src leaves every row ascending.
//
// Sorting, unique and scans use CUB (header templates compiled into this
// library); the other passes are kernels written here.
#include <cub/cub.cuh>
#include <thrust/iterator/transform_iterator.h>

#include "common.cuh"

namespace tchll {

// Canonical keys are (a << k) | b with a < b < 2^k.  The all-ones key of 2k
// bits is never a canonical pair (it needs a == b), so it marks dropped
// self-loops and sorts after every real key.
__host__ __device__ __forceinline__ uint64_t key_sentinel(int k) { return (k >= 32) ? ~0ull : ((1ull << (2 * k)) - 1ull); }
constexpr uint32_t kEndSentinel = 0xFFFFFFFFu;

struct Occurs {
    __host__ __device__ int32_t operator()(int32_t d) const { return d != 0; }
};

struct CsrWs {
    uint64_t* k0;
    uint64_t* k1;
    uint32_t* e0;
    uint32_t* e1;
    int32_t* deg;
    // [fdeg 2 n_raw + 2][ca n_raw][cb n_raw], or, in the direct path, info of
    // up to 2 n_raw ids
    int32_t* fdeg;
    int32_t* ca;
    int32_t* cb;
    int2* info;
    int64_t* cnt;  // [0] unique keys, [1] unique endpoints, [2] negative-id flag, [3] largest id
    void* tmp;
    size_t tmp_bytes;
};

// (a build asks three times: the thread's last answer is kept, with the device
// it is for, as the sizes may depend on it, and only if all queries succeeded)
static size_t csr_cub_tmp(int64_t n_raw) {
    static thread_local int64_t last_n = -1;
    static thread_local int last_dev = -1;
    static thread_local size_t last_bytes = 0;
    const int dev = current_device();
    if (n_raw == last_n && dev == last_dev && dev >= 0) return last_bytes;
    const int R = (int)(n_raw > 0 ? n_raw : 1);
    size_t a = 0, b = 0, c = 0, d = 0, e = 0, f = 0;
    const cudaError_t rc[6] = {
        cub::DeviceRadixSort::SortKeys(nullptr, a, (uint64_t*)nullptr, (uint64_t*)nullptr, R, 0, 63),
        cub::DeviceSelect::Unique(nullptr, b, (uint64_t*)nullptr, (uint64_t*)nullptr, (int64_t*)nullptr, R),
        cub::DeviceRadixSort::SortKeys(nullptr, c, (uint32_t*)nullptr, (uint32_t*)nullptr, 2 * R, 0, 32),
        cub::DeviceSelect::Unique(nullptr, d, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t*)nullptr, 2 * R),
        cub::DeviceScan::ExclusiveSum(nullptr, e, thrust::make_transform_iterator((int32_t*)nullptr, Occurs()),
                                      (int32_t*)nullptr, 2 * R + 1),
        cub::DeviceRadixSort::SortPairs(nullptr, f, (uint32_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                        (uint32_t*)nullptr, R, 0, 32)};
    bool ok = true;
    for (const cudaError_t r : rc) ok &= r == cudaSuccess;
    size_t m = a;
    if (b > m) m = b;
    if (c > m) m = c;
    if (d > m) m = d;
    if (e > m) m = e;
    if (f > m) m = f;
    if (ok) {
        last_n = n_raw;
        last_dev = dev;
        last_bytes = m;
    }
    return m;
}

static bool carve_csr(void* ws, size_t bytes, int64_t n_raw, CsrWs& W, size_t* need) {
    const size_t R = (size_t)(n_raw > 0 ? n_raw : 1);
    Carve cv(ws, bytes);
    W.k0 = cv.take<uint64_t>(R);
    W.k1 = cv.take<uint64_t>(R);
    W.e0 = cv.take<uint32_t>(2 * R);
    W.e1 = cv.take<uint32_t>(2 * R);
    W.deg = cv.take<int32_t>(2 * R + 1);
    W.info = cv.take<int2>(2 * R + 1);
    W.fdeg = reinterpret_cast<int32_t*>(W.info);
    W.ca = W.fdeg + 2 * R + 2;
    W.cb = W.ca + R;
    W.cnt = cv.take<int64_t>(4);
    W.tmp_bytes = csr_cub_tmp(n_raw);
    W.tmp = cv.take<char>(W.tmp_bytes);
    if (need) *need = cv.off;
    return cv.ok();
}

static int grid_n(int64_t n, int threads = 256) {
    int64_t g = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 32;
    if (g > cap) g = cap;
    return g < 1 ? 1 : (int)g;
}

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// Grid-stride loop that whole warps enter and leave together (bodies with
// warp shuffles): i may reach past n in the last pass; test it in the body.
#define WARP_GRID_STRIDE(i, n)                                                               \
    for (int64_t _wb = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31u),              \
                 i = _wb + (threadIdx.x & 31u);                                              \
         _wb < (n); _wb += (int64_t)gridDim.x * blockDim.x, i = _wb + (threadIdx.x & 31u))

// Largest endpoint id (atomicMax, one per warp) and the negative-id flag.
__global__ void max_id_kernel(const int32_t* __restrict__ ru, const int32_t* __restrict__ rv, int64_t n,
                              int64_t* cnt) {
    int32_t mx = 0;
    bool neg = false;
    GRID_STRIDE(i, n) {
        const int32_t u = ru[i], v = rv[i];
        neg |= (u < 0) | (v < 0);
        mx = max(mx, max(u, v));
    }
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    neg = __any_sync(0xFFFFFFFFu, neg);
    if ((threadIdx.x & 31) == 0) {
        atomicMax((unsigned long long*)(cnt + 3), (unsigned long long)mx);
        if (neg) cnt[2] = 1;
    }
}

__global__ void canon_kernel(const int32_t* __restrict__ ru, const int32_t* __restrict__ rv, int64_t n, int k,
                             uint64_t* keys) {
    const uint64_t sent = key_sentinel(k);
    GRID_STRIDE(i, n) {
        const int32_t u = ru[i], v = rv[i];
        const uint32_t a = (uint32_t)(u < v ? u : v), b = (uint32_t)(u < v ? v : u);
        keys[i] = (u == v || u < 0 || v < 0) ? sent : (((uint64_t)a << k) | b);
    }
}

// Endpoints of the unique keys (sentinels become kEndSentinel).
__global__ void ends_kernel(const uint64_t* __restrict__ keys, int64_t cap, const int64_t* cnt, int kb,
                            uint32_t* ends) {
    const int64_t nk = cnt[0];
    const uint64_t sent = key_sentinel(kb), lo = (1ull << kb) - 1ull;
    GRID_STRIDE(i, cap) {
        uint64_t k = i < nk ? keys[i] : sent;
        if (k == sent) {
            ends[2 * i] = kEndSentinel;
            ends[2 * i + 1] = kEndSentinel;
        } else {
            ends[2 * i] = (uint32_t)(k >> kb);
            ends[2 * i + 1] = (uint32_t)(k & lo);
        }
    }
}

__device__ __forceinline__ int64_t lower_bound_u32(const uint32_t* a, int64_t n, uint32_t x) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Number of real edges / nodes: drop the trailing sentinel when present.
__device__ __forceinline__ int64_t n_real_edges(const uint64_t* keys, const int64_t* cnt, int kb) {
    const int64_t nk = cnt[0];
    return (nk > 0 && keys[nk - 1] == key_sentinel(kb)) ? nk - 1 : nk;
}
__device__ __forceinline__ int64_t n_real_nodes(const uint32_t* nodes, const int64_t* cnt) {
    const int64_t nn = cnt[1];
    return (nn > 0 && nodes[nn - 1] == kEndSentinel) ? nn - 1 : nn;
}

// deg[a] += (number of lanes with this a) from the last lane of each run of
// equal a (the keys are sorted by a, so runs are contiguous lanes); lanes
// past the end pass a = -1.
__device__ __forceinline__ void add_runs(int32_t* deg, int32_t a, int lane) {
    const unsigned FULLM = 0xFFFFFFFFu;
    const int32_t na = __shfl_down_sync(FULLM, a, 1);
    const bool tail = lane == 31 || na != a;  // the run's last lane
    const unsigned tails = __ballot_sync(FULLM, tail);
    if (a >= 0 && tail) {
        // the run starts after the previous tail
        const unsigned below = tails & ((1u << lane) - 1u);
        const int start = below ? 32 - __clz(below) : 0;
        atomicAdd(deg + a, lane - start + 1);
    }
}

// Sort path: binary search of both endpoints in the sorted node table.
__global__ void remap_kernel(const uint64_t* __restrict__ keys, int64_t cap, const uint32_t* __restrict__ nodes,
                             const int64_t* cnt, int kb, int32_t* ca, int32_t* cb, int32_t* deg) {
    const int64_t ne = n_real_edges(keys, cnt, kb);
    const int64_t nn = n_real_nodes(nodes, cnt);
    const uint64_t lo = (1ull << kb) - 1ull;
    const int lane = threadIdx.x & 31;
    WARP_GRID_STRIDE(i, cap) {
        const bool in = i < ne;
        int32_t a = -1;
        if (in) {
            const uint64_t k = keys[i];
            a = (int32_t)lower_bound_u32(nodes, nn, (uint32_t)(k >> kb));
            const int32_t b = (int32_t)lower_bound_u32(nodes, nn, (uint32_t)(k & lo));
            ca[i] = a;
            cb[i] = b;
            atomicAdd(deg + b, 1);
        }
        add_runs(deg, a, lane);
    }
}

// Direct path: undirected degrees by raw id, of every unique edge (deg zeroed
// over [0, max id + 1] before).
__global__ void id_degree_kernel(const uint64_t* __restrict__ keys, int64_t cap, const int64_t* cnt, int kb,
                                 int32_t* deg) {
    const int64_t ne = n_real_edges(keys, cnt, kb);
    const uint64_t lo = (1ull << kb) - 1ull;
    const int lane = threadIdx.x & 31;
    WARP_GRID_STRIDE(i, cap) {
        int32_t a = -1;
        if (i < ne) {
            const uint64_t k = keys[i];
            a = (int32_t)(k >> kb);
            atomicAdd(deg + (k & lo), 1);
        }
        add_runs(deg, a, lane);
    }
}

// Direct path, after rank = exclusive scan of "the id occurs" over [0, ids]
// (ids = max id + 2 entries): the node table nodes[rank[id]] = id, the number
// of nodes in cnt[1] (its sort-path meaning), and degree and rank of every id
// side by side for the orientation.
__global__ void rank_nodes_kernel(const int32_t* __restrict__ deg, const int32_t* __restrict__ rank, int64_t ids,
                                  uint32_t* nodes, int2* info, int64_t* cnt) {
    GRID_STRIDE(i, ids) {
        const int32_t r = rank[i], d = deg[i];
        if (i == ids - 1) {
            cnt[1] = r;  // deg[ids - 1] = 0: the total
        } else {
            info[i] = make_int2(d, r);
            if (d) nodes[r] = (uint32_t)i;
        }
    }
}

__global__ void sizes_kernel(const uint64_t* keys, const uint32_t* nodes, const int64_t* cnt, int kb, int direct,
                             int64_t* sizes) {
    if (cnt[2]) {
        sizes[0] = -1;
        sizes[1] = -1;
        return;
    }
    sizes[0] = direct ? cnt[1] : n_real_nodes(nodes, cnt);
    sizes[1] = n_real_edges(keys, cnt, kb);
}

// Orientation u -> v iff (deg u, u) < (deg v, v): the pair (src, dst) of
// edge i goes to okey[i] / oval[i] (canonical order kept for the stable sort).
// Direct path (as phase 1 chose it from the largest id, cnt[3]): raw ids from
// the keys, degree and rank with one 8-byte load per endpoint (a run of keys
// shares its first).  Ranks rise with the ids, so ids break ties as well.
// R-MAT 22: flagging the ids, replacing them by ranks while counting degrees
// and orienting took 0.89 + 0.82 + 0.27 ms; counting by id and this, 0.80 +
// 0.29 ms.
__global__ void orient_kernel(const uint64_t* __restrict__ keys, const int2* __restrict__ info,
                              const int64_t* __restrict__ cnt, int64_t direct_ids, const int32_t* __restrict__ ca,
                              const int32_t* __restrict__ cb, int64_t ne, const int32_t* __restrict__ deg,
                              uint32_t* okey, uint32_t* oval) {
    const int64_t max_id = cnt[3];
    const bool direct = max_id + 2 <= direct_ids;  // grid-uniform
    const int kb = max_id > 0 ? 64 - __clzll(max_id) : 1;
    const uint64_t lo = (1ull << kb) - 1ull;
    GRID_STRIDE(i, ne) {
        int32_t a, b, da, db;
        if (direct) {
            const uint64_t k = __ldcs(reinterpret_cast<const unsigned long long*>(keys) + i);
            const int2 ia = __ldg(info + (k >> kb)), ib = __ldg(info + (k & lo));
            da = ia.x, a = ia.y;
            db = ib.x, b = ib.y;
        } else {
            a = ca[i], b = cb[i];
            da = deg[a], db = deg[b];
        }
        const bool first = (da < db) || (da == db && a < b);
        okey[i] = (uint32_t)(first ? a : b);
        oval[i] = (uint32_t)(first ? b : a);
    }
}

// row_ptr from the ascending sources src[0 .. ne): entry i is the first edge
// of every row s in (src[i-1], src[i]] (src[-1] = -1, src[ne] = n_nodes),
// so each of row_ptr[0 .. n_nodes] is written exactly once.
__global__ void row_ptr_kernel(const int32_t* __restrict__ src, int64_t ne, int64_t n_nodes, int32_t* row_ptr) {
    GRID_STRIDE(i, ne + 1) {
        const int64_t lo = i > 0 ? (int64_t)src[i - 1] : -1;
        const int64_t hi = i < ne ? (int64_t)src[i] : n_nodes;
        for (int64_t r = lo + 1; r <= hi; ++r) row_ptr[r] = (int32_t)i;
    }
}

__global__ void copy_nodes_kernel(const uint32_t* __restrict__ nodes, int64_t n, const int32_t* __restrict__ row_ptr,
                                  const int32_t* __restrict__ deg, const int64_t* __restrict__ cnt, int64_t direct_ids,
                                  int32_t* node_ids, int32_t* degrees, int32_t* undirected) {
    const bool direct = cnt[3] + 2 <= direct_ids;  // deg goes by id
    GRID_STRIDE(i, n) {
        node_ids[i] = (int32_t)nodes[i];
        degrees[i] = row_ptr[i + 1] - row_ptr[i];
        if (undirected) undirected[i] = deg[direct ? (int64_t)nodes[i] : i];
    }
}

static int bits_for(int64_t maxv) {
    int b = 1;
    while (b < 63 && (maxv >> b) != 0) ++b;
    return b;
}

// ------------------------------------------------------- small builds ------
// Up to kSmallRaw raw edges the dozen sort passes cost their launches and
// little else, so the build takes another way: the canonical pairs go into a
// hash table (2 n_raw slots, in the sort's key buffers), which drops
// duplicates and counts the degrees as it goes (ids too large for direct
// tables are first replaced by their rank among the sorted endpoints); the
// oriented pairs are scattered from the table into their rows, in
// no order, and a warp sorts each row in registers or shared memory.  A
// forward list has at most sqrt(2 n_edges) members (each of the d members of
// u's list has a degree of at least u's, which is at least d), 2048 here.
// Whole builds, sorted / so: R-MAT 10, 13, 15, 16, 17 (16 K, 90 K, 524 K, 1 M, 2 M
// raw edges) 197 / 119, 236 / 138, 281 / 208, 343 / 289, 507 / 437 us; bound by
// launches and the two read-backs, then by the atomics on the popular ids.
// Lists of more than kDenseRaw edges with kDenseEnds and more to an id go by
// sorting all the same: their few counters are contended whatever the order,
// and their rows are long (clique of 1,000 / 1,400 / 2,000 vertices, by sorting / by
// table: 270 / 311, 315 / 470, 402 / 627 us; of 300: 209 / 155).
constexpr int64_t kSmallRaw = 1 << 21;
constexpr int64_t kDenseRaw = 1 << 17;
constexpr int64_t kDenseEnds = 256;
__host__ __device__ __forceinline__ bool small_route(int64_t n_raw, int64_t max_id) {
    return n_raw <= kSmallRaw && (n_raw <= kDenseRaw || n_raw < kDenseEnds * (max_id + 1));
}
constexpr int kSmallRow = 2048;
constexpr uint64_t kEmptySlot = ~0ull;

__device__ __forceinline__ uint32_t pair_slot(uint64_t key, uint32_t slots) {
    return (uint32_t)__umul64hi(splitmix64_fin(key), (uint64_t)slots);
}

// Endpoints of the raw edges; self-loops become kEndSentinel.
__global__ void small_ends_kernel(const int32_t* __restrict__ ru, const int32_t* __restrict__ rv, int64_t n,
                                  uint32_t* ends) {
    GRID_STRIDE(i, n) {
        const bool loop = ru[i] == rv[i];
        ends[2 * i] = loop ? kEndSentinel : (uint32_t)ru[i];
        ends[2 * i + 1] = loop ? kEndSentinel : (uint32_t)rv[i];
    }
}

// Whether several neighbouring lanes hold the same x (called by whole warps).
// Comparing all lanes at every step would cost R-MAT 17 several percent.
template <class T>
__device__ __forceinline__ bool lanes_repeat(T x, bool in) {
    const T other = __shfl_xor_sync(0xFFFFFFFFu, x, 1);  // every lane takes part
    return __popc(__ballot_sync(0xFFFFFFFFu, in && x == other)) >= 4;
}

// Adds 1 to deg[id] of every lane with id >= 0, lanes of one id with one atomic
// where they repeat: a popular id would queue up.
__device__ __forceinline__ void add_same(int32_t* deg, int32_t id, int lane) {
    if (!lanes_repeat(id, id >= 0)) {
        if (id >= 0) atomicAdd(deg + id, 1);
        return;
    }
    const unsigned same = __match_any_sync(0xFFFFFFFFu, id);
    if (id >= 0 && lane == __ffs(same) - 1) atomicAdd(deg + id, __popc(same));
}

// cnt[0] += unique pairs; deg[id]: undirected degrees.  With nodes (sorted,
// cnt[1] of them) an id stands for its place there.  Of a warp's lanes with
// the same pair one goes to the table (a list of few pairs repeated often
// would queue up on their slots; reading a slot before claiming it costs every
// other list a second trip: R-MAT 17 433 -> 502 us).
__global__ void small_insert_kernel(const int32_t* __restrict__ ru, const int32_t* __restrict__ rv, int64_t n,
                                    const uint32_t* __restrict__ nodes, unsigned long long* table, uint32_t slots,
                                    int32_t* deg, int64_t* cnt) {
    uint32_t fresh = 0;
    const int lane = threadIdx.x & 31;
    const int64_t nn = nodes ? n_real_nodes(nodes, cnt) : 0;
    WARP_GRID_STRIDE(i, n) {
        int32_t u = -1, v = -1;
        if (i < n) {
            u = ru[i];  // negative ids never get here
            v = rv[i];
        }
        bool mine = u != v;
        if (mine && nodes) {
            u = (int32_t)lower_bound_u32(nodes, nn, (uint32_t)u);
            v = (int32_t)lower_bound_u32(nodes, nn, (uint32_t)v);
        }
        const unsigned long long key =
            mine ? ((unsigned long long)(uint32_t)min(u, v) << 32) | (uint32_t)max(u, v) : kEmptySlot;
        if (lanes_repeat(key, mine)) {  // warp-uniform
            const unsigned same = __match_any_sync(0xFFFFFFFFu, key);
            if (lane != __ffs(same) - 1) mine = false;
        }
        if (mine) {
            uint32_t s = pair_slot(key, slots);
            for (uint32_t k = 0; k < slots; ++k) {  // at most half the slots ever fill
                const unsigned long long old = atomicCAS(table + s, kEmptySlot, key);
                mine = old == kEmptySlot;
                if (mine || old == key) break;
                s = s + 1 < slots ? s + 1 : 0;
            }
        }
        fresh += mine;
        add_same(deg, mine ? u : -1, lane);
        add_same(deg, mine ? v : -1, lane);
    }
    fresh = __reduce_add_sync(0xFFFFFFFFu, fresh);
    if (lane == 0 && fresh) atomicAdd((unsigned long long*)cnt, (unsigned long long)fresh);
}

// Tiles of 1024 entries, 256 threads: how many entries count (FLAG: 1 per
// non-zero entry, else the entry itself).
template <bool FLAG>
__global__ void __launch_bounds__(256) tile_sum_kernel(const int32_t* __restrict__ in, int64_t n, int32_t* sums) {
    __shared__ int32_t w[8];
    int32_t c = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t k = blockIdx.x * 1024ll + 256 * i + threadIdx.x;
        const int32_t x = k < n ? in[k] : 0;
        c += FLAG ? (x != 0) : x;
    }
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t t = 0;
        for (int i = 0; i < 8; ++i) t += w[i];
        sums[blockIdx.x] = t;
    }
}

// Exclusive prefix of this thread's 4 consecutive entries x[] of the tile, by
// adding up the tiles before (no tile waits for another).
__device__ __forceinline__ int32_t tile_prefix(const int32_t* __restrict__ sums, int32_t mine, int32_t* w) {
    const int tid = threadIdx.x, lane = tid & 31;
    int32_t before = 0;
    for (int64_t k = tid; k < (int64_t)blockIdx.x; k += 256) before += __ldg(sums + k);
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    int32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) w[tid >> 5] = incl;
    if (lane == 0) w[8 + (tid >> 5)] = before;
    __syncthreads();
    int32_t base = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        base += w[8 + i];
        if (i < (tid >> 5)) base += w[i];
    }
    return base + incl - mine;
}

// rank[id] among the ids that occur, nodes[rank] = id (or, when the ids stand
// for places in nodes already, left alone); the last tile writes the sizes.
__global__ void __launch_bounds__(256) small_rank_kernel(const int32_t* __restrict__ deg, int64_t ids,
                                                         const int32_t* __restrict__ sums, int32_t* rank,
                                                         uint32_t* nodes, int places, const int64_t* cnt,
                                                         int64_t* sizes) {
    __shared__ int32_t w[16];
    const int64_t k0 = blockIdx.x * 1024ll + 4 * threadIdx.x;
    int32_t f[4], c = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) c += f[i] = k0 + i < ids && deg[k0 + i] != 0;
    int32_t at = tile_prefix(sums, c, w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (f[i]) {
            rank[k0 + i] = at;
            if (!places) nodes[at] = (uint32_t)(k0 + i);
            ++at;
        }
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 255) {
        sizes[0] = at;
        sizes[1] = cnt[0];
    }
}

// The oriented pair of a table slot in ranks; false for an empty slot.
__device__ __forceinline__ bool small_pair(unsigned long long key, const int32_t* __restrict__ deg,
                                           const int32_t* __restrict__ rank, int32_t& src, int32_t& dst) {
    if (key == kEmptySlot) return false;
    const int32_t a = (int32_t)(key >> 32), b = (int32_t)(key & 0xFFFFFFFFull);  // a < b
    const int32_t da = __ldg(deg + a), db = __ldg(deg + b), ra = __ldg(rank + a), rb = __ldg(rank + b);
    const bool first = da <= db;  // ties: the lower id
    src = first ? ra : rb;
    dst = first ? rb : ra;
    return true;
}

__global__ void small_count_kernel(const unsigned long long* __restrict__ table, int64_t slots,
                                   const int32_t* __restrict__ deg, const int32_t* __restrict__ rank, int32_t* fdeg) {
    GRID_STRIDE(i, slots) {
        int32_t s, d;
        if (small_pair(table[i], deg, rank, s, d)) atomicAdd(fdeg + s, 1);
    }
}

// row_ptr, the node outputs, and fdeg turned into the rows' write cursors.
__global__ void __launch_bounds__(256) small_rows_kernel(int32_t* fdeg, int64_t n, const int32_t* __restrict__ sums,
                                                         const uint32_t* __restrict__ nodes, const int64_t* cnt,
                                                         int64_t direct_ids, const int32_t* __restrict__ deg,
                                                         int32_t* row_ptr, int32_t* degrees, int32_t* node_ids,
                                                         int32_t* undirected) {
    __shared__ int32_t w[16];
    const bool places = cnt[3] + 1 > direct_ids;  // as phase 1 decided: deg goes by place
    const int64_t k0 = blockIdx.x * 1024ll + 4 * threadIdx.x;
    int32_t f[4], c = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) c += f[i] = k0 + i < n ? fdeg[k0 + i] : 0;
    int32_t at = tile_prefix(sums, c, w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t k = k0 + i;
        if (k < n) {
            const uint32_t id = nodes[k];
            row_ptr[k] = at;
            fdeg[k] = at;
            degrees[k] = f[i];
            node_ids[k] = (int32_t)id;
            if (undirected) undirected[k] = deg[places ? k : (int64_t)id];  // id < direct_ids
            at += f[i];
            if (k == n - 1) row_ptr[n] = at;
        }
    }
}

__global__ void small_scatter_kernel(const unsigned long long* __restrict__ table, int64_t slots,
                                     const int32_t* __restrict__ deg, const int32_t* __restrict__ rank,
                                     int32_t* cursor, int32_t* out) {
    GRID_STRIDE(i, slots) {
        int32_t s, d;
        if (small_pair(table[i], deg, rank, s, d)) out[atomicAdd(cursor + s, 1)] = d;
    }
}

// Sorts the rows in[row_ptr[r] .. row_ptr[r + 1]) (distinct values) into
// col_idx and edge_v and writes edge_u; a warp takes `per` (1 or 32) rows at a
// time.  Up to 4 members: a lane sorts its row in registers; up to 64: each lane
// counts, for its two, the members below them; longer rows: a bitonic sort in
// the warp's shared memory.  (4 M rows of at most a few members: 962 us with a
// warp per row, 60 so; few and long rows want a warp each.)
__device__ __forceinline__ void order(int32_t& a, int32_t& b) {
    const int32_t lo = min(a, b);
    b = max(a, b);
    a = lo;
}
__global__ void __launch_bounds__(128) small_sort_kernel(const int32_t* __restrict__ row_ptr, int64_t n, int per,
                                                         const int32_t* __restrict__ in, int32_t* col_idx,
                                                         int32_t* edge_u, int32_t* edge_v) {
    __shared__ int32_t buf[4][kSmallRow];
    const int lane = threadIdx.x & 31;
    int32_t* b = buf[threadIdx.x >> 5];
    const int32_t none = 0x7FFFFFFF;  // above every rank
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * per; r0 < n; r0 += warps * per) {
        int32_t my_s = 0, my_d = 0;
        if (lane < per && r0 + lane < n) {
            my_s = __ldg(row_ptr + r0 + lane);
            my_d = __ldg(row_ptr + r0 + lane + 1) - my_s;
        }
        if (my_d > 0 && my_d <= 4) {
            int32_t x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = i < my_d ? __ldg(in + my_s + i) : none;
            order(x[0], x[1]);
            order(x[2], x[3]);
            order(x[0], x[2]);
            order(x[1], x[3]);
            order(x[1], x[2]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i < my_d) {
                    col_idx[my_s + i] = x[i];
                    edge_v[my_s + i] = x[i];
                    edge_u[my_s + i] = (int32_t)(r0 + lane);
                }
            }
        }
        for (unsigned todo = __ballot_sync(0xFFFFFFFFu, my_d > 4); todo; todo &= todo - 1) {
            const int k = __ffs(todo) - 1;
            const int32_t s = __shfl_sync(0xFFFFFFFFu, my_s, k), d = __shfl_sync(0xFFFFFFFFu, my_d, k);
            const int64_t r = r0 + k;
            if (d <= 64) {
                const int32_t x0 = lane < d ? __ldg(in + s + lane) : none;
                const int32_t x1 = 32 + lane < d ? __ldg(in + s + 32 + lane) : none;
                int c0 = 0, c1 = 0;
                for (int i = 0; i < d; ++i) {
                    const int32_t y = i < 32 ? __shfl_sync(0xFFFFFFFFu, x0, i) : __shfl_sync(0xFFFFFFFFu, x1, i - 32);
                    c0 += y < x0;
                    c1 += y < x1;
                }
                if (lane < d) {
                    col_idx[s + c0] = x0;
                    edge_v[s + c0] = x0;
                    edge_u[s + lane] = (int32_t)r;
                }
                if (32 + lane < d) {
                    col_idx[s + c1] = x1;
                    edge_v[s + c1] = x1;
                    edge_u[s + 32 + lane] = (int32_t)r;
                }
                continue;
            }
            int m = 128;  // the next power of two
            while (m < d) m <<= 1;
            __syncwarp();
            for (int i = lane; i < m; i += 32) b[i] = i < d ? __ldg(in + s + i) : none;
            __syncwarp();
            for (int k2 = 2; k2 <= m; k2 <<= 1) {
                for (int j = k2 >> 1; j > 0; j >>= 1) {
                    for (int t = lane; t < m / 2; t += 32) {
                        const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo | j;
                        const int32_t x = b[lo], y = b[hi];
                        if ((x > y) == ((lo & k2) == 0)) {
                            b[lo] = y;
                            b[hi] = x;
                        }
                    }
                    __syncwarp();
                }
            }
            for (int i = lane; i < d; i += 32) {
                const int32_t x = b[i];
                col_idx[s + i] = x;
                edge_v[s + i] = x;
                edge_u[s + i] = (int32_t)r;
            }
        }
    }
}

// ------------------------------------------------- forward_adj -> CSR ------
__global__ void iota_kernel(int64_t* a, int64_t n) {
    GRID_STRIDE(i, n) a[i] = i;
}

__global__ void gather_deg_kernel(const int64_t* __restrict__ lens, const int64_t* __restrict__ order, int64_t n,
                                  int32_t* degrees, int32_t* deg_scan_in) {
    GRID_STRIDE(i, n) {
        const int32_t d = (int32_t)lens[order[i]];
        degrees[i] = d;
        deg_scan_in[i] = d;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) deg_scan_in[n] = 0;
}

__device__ __forceinline__ int64_t upper_bound_i32(const int32_t* a, int64_t n, int64_t x) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((int64_t)a[mid] <= x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__global__ void adj_fill_kernel(const int64_t* __restrict__ sorted_keys, int64_t n,
                                const int64_t* __restrict__ order, const int64_t* __restrict__ dict_off,
                                const int32_t* __restrict__ row_ptr, const int64_t* __restrict__ values, int64_t nnz,
                                int32_t* col_idx, int32_t* edge_u, int32_t* edge_v, unsigned long long* missing) {
    unsigned long long miss = 0;
    GRID_STRIDE(k, nnz) {
        const int64_t row = upper_bound_i32(row_ptr, n + 1, k) - 1;
        const int64_t src = dict_off[order[row]] + (k - row_ptr[row]);
        const int64_t x = values[src];
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (sorted_keys[mid] < x) lo = mid + 1; else hi = mid;
        }
        int32_t c = (int32_t)lo;
        if (lo >= n || sorted_keys[lo] != x) {
            ++miss;
            c = -1;
        }
        col_idx[k] = c;
        edge_v[k] = c;
        edge_u[k] = (int32_t)row;
    }
    if (miss) atomicAdd(missing, miss);
}

__global__ void zero_kernel(int64_t* p) { *p = 0; }

}  // namespace tchll

using namespace tchll;

TCHLL_EXPORT int tchll_csr_workspace_bytes(int64_t n_raw, size_t* bytes) {
    TCHLL_ARG(bytes && n_raw >= 0, "bad arguments");
    TCHLL_ARG(n_raw < (int64_t)(INT32_MAX / 2), "edge list longer than 2^30 entries");
    CsrWs W;
    carve_csr(nullptr, 0, n_raw, W, bytes);
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_csr_build_phase1(const int32_t* raw_u, const int32_t* raw_v, int64_t n_raw, int64_t* sizes,
                                        void* workspace, size_t workspace_bytes, void* stream) {
    TCHLL_ARG(sizes != nullptr && n_raw >= 0, "bad arguments");
    TCHLL_ARG(n_raw == 0 || (raw_u && raw_v), "null edge arrays");
    TCHLL_ARG(n_raw < (int64_t)(INT32_MAX / 2), "edge list longer than 2^30 entries");
    CsrWs W;
    size_t need = 0;
    if (!carve_csr(workspace, workspace_bytes, n_raw, W, &need) || !workspace) {
        set_error("workspace too small: need %zu bytes, have %zu", need, workspace_bytes);
        return TCHLL_EWORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int R = (int)(n_raw > 0 ? n_raw : 1);
    TCHLL_CUDA(cudaMemsetAsync(W.cnt, 0, 4 * sizeof(int64_t), st));
    TCHLL_CUDA(cudaMemsetAsync(W.deg, 0, (2 * (size_t)R + 1) * sizeof(int32_t), st));
    if (n_raw == 0) {
        TCHLL_CUDA(cudaMemsetAsync(sizes, 0, 2 * sizeof(int64_t), st));
        return TCHLL_OK;
    }
    // the largest id sizes the keys and picks the node-table method: one
    // 16-byte read-back (the stream is waited for here)
    max_id_kernel<<<grid_n(n_raw), 256, 0, st>>>(raw_u, raw_v, n_raw, W.cnt);
    TCHLL_CHECK_LAUNCH("max_id_kernel");
    int64_t hc[2] = {0, 0};
    const int rf = fetch_small(hc, W.cnt + 2, sizeof(hc), st);
    if (rf) return rf;
    if (hc[0]) {  // a negative id: sizes -1, nothing else
        sizes_kernel<<<1, 1, 0, st>>>(W.k0, W.e0, W.cnt, 1, 0, sizes);
        TCHLL_CHECK_LAUNCH("sizes_kernel");
        return TCHLL_OK;
    }
    const int64_t max_id = hc[1];
    if (small_route(n_raw, max_id)) {
        // deg in W.deg (cleared above), rank in W.e1, nodes in W.e0, tile sums
        // in W.fdeg
        const bool places = max_id + 1 > 2 * (int64_t)R;
        const int64_t slots = 2 * (int64_t)R, ids = places ? slots : max_id + 1, tiles = (ids + 1023) / 1024;
        unsigned long long* table = reinterpret_cast<unsigned long long*>(W.k0);
        if (places) {
            small_ends_kernel<<<grid_n(n_raw), 256, 0, st>>>(raw_u, raw_v, n_raw, W.e0);
            TCHLL_CHECK_LAUNCH("small_ends_kernel");
            size_t tb = W.tmp_bytes;
            TCHLL_CUDA(cub::DeviceRadixSort::SortKeys(W.tmp, tb, W.e0, W.e1, 2 * R, 0, 32, st));
            count_launch();
            tb = W.tmp_bytes;
            TCHLL_CUDA(cub::DeviceSelect::Unique(W.tmp, tb, W.e1, W.e0, W.cnt + 1, 2 * R, st));
            count_launch();
        }
        TCHLL_CUDA(cudaMemsetAsync(table, 0xFF, (size_t)slots * sizeof(uint64_t), st));
        small_insert_kernel<<<grid_n(n_raw), 256, 0, st>>>(raw_u, raw_v, n_raw, places ? W.e0 : nullptr, table,
                                                           (uint32_t)slots, W.deg, W.cnt);
        TCHLL_CHECK_LAUNCH("small_insert_kernel");
        tile_sum_kernel<true><<<(int)tiles, 256, 0, st>>>(W.deg, ids, W.fdeg);
        TCHLL_CHECK_LAUNCH("tile_sum_kernel");
        small_rank_kernel<<<(int)tiles, 256, 0, st>>>(W.deg, ids, W.fdeg, reinterpret_cast<int32_t*>(W.e1), W.e0,
                                                      places ? 1 : 0, W.cnt, sizes);
        TCHLL_CHECK_LAUNCH("small_rank_kernel");
        return TCHLL_OK;
    }
    const int kb = bits_for(max_id);
    canon_kernel<<<grid_n(n_raw), 256, 0, st>>>(raw_u, raw_v, n_raw, kb, W.k0);
    TCHLL_CHECK_LAUNCH("canon_kernel");
    size_t tb = W.tmp_bytes;
    TCHLL_CUDA(cub::DeviceRadixSort::SortKeys(W.tmp, tb, W.k0, W.k1, R, 0, 2 * kb, st));
    count_launch();
    tb = W.tmp_bytes;
    TCHLL_CUDA(cub::DeviceSelect::Unique(W.tmp, tb, W.k1, W.k0, W.cnt + 0, R, st));
    count_launch();
    // direct rank table when ids 0 .. max_id (+ a zero flag) fit the 2R-entry
    // endpoint buffers, else sort and deduplicate the endpoints
    const int64_t ids = max_id + 2;
    const int direct = ids <= 2 * (int64_t)R ? 1 : 0;
    if (direct) {
        id_degree_kernel<<<grid_n(n_raw), 256, 0, st>>>(W.k0, n_raw, W.cnt, kb, W.deg);  // cleared above
        TCHLL_CHECK_LAUNCH("id_degree_kernel");
        int32_t* rank = reinterpret_cast<int32_t*>(W.e1);
        tb = W.tmp_bytes;
        TCHLL_CUDA(cub::DeviceScan::ExclusiveSum(W.tmp, tb, thrust::make_transform_iterator(W.deg, Occurs()), rank,
                                                 (int)ids, st));
        count_launch();
        rank_nodes_kernel<<<grid_n(ids), 256, 0, st>>>(W.deg, rank, ids, W.e0, W.info, W.cnt);
        TCHLL_CHECK_LAUNCH("rank_nodes_kernel");
    } else {
        ends_kernel<<<grid_n(n_raw), 256, 0, st>>>(W.k0, n_raw, W.cnt, kb, W.e0);
        TCHLL_CHECK_LAUNCH("ends_kernel");
        tb = W.tmp_bytes;
        TCHLL_CUDA(cub::DeviceRadixSort::SortKeys(W.tmp, tb, W.e0, W.e1, 2 * R, 0, 32, st));
        count_launch();
        tb = W.tmp_bytes;
        TCHLL_CUDA(cub::DeviceSelect::Unique(W.tmp, tb, W.e1, W.e0, W.cnt + 1, 2 * R, st));
        count_launch();
        remap_kernel<<<grid_n(n_raw), 256, 0, st>>>(W.k0, n_raw, W.e0, W.cnt, kb, W.ca, W.cb, W.deg);
        TCHLL_CHECK_LAUNCH("remap_kernel");
    }
    sizes_kernel<<<1, 1, 0, st>>>(W.k0, W.e0, W.cnt, kb, direct, sizes);
    TCHLL_CHECK_LAUNCH("sizes_kernel");
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_csr_build_phase2(int64_t n_raw, int64_t n_nodes, int64_t n_edges, int32_t* row_ptr,
                                        int32_t* col_idx, int32_t* degrees, int32_t* node_ids, int32_t* edge_u,
                                        int32_t* edge_v, int32_t* undirected_degrees, void* workspace,
                                        size_t workspace_bytes, void* stream) {
    TCHLL_ARG(n_nodes >= 0 && n_edges >= 0 && n_edges <= n_raw && n_nodes <= 2 * n_raw, "sizes out of range");
    TCHLL_ARG(row_ptr != nullptr, "row_ptr is null");
    TCHLL_ARG(n_nodes == 0 || (degrees && node_ids), "null node outputs");
    TCHLL_ARG(n_edges == 0 || (col_idx && edge_u && edge_v), "null edge outputs");
    CsrWs W;
    size_t need = 0;
    if (!carve_csr(workspace, workspace_bytes, n_raw, W, &need) || !workspace) {
        set_error("workspace too small: need %zu bytes, have %zu", need, workspace_bytes);
        return TCHLL_EWORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    bool small = n_raw <= kSmallRaw;
    if (small && n_edges > 0 && n_raw > kDenseRaw && n_raw >= kDenseEnds * n_nodes) {
        // phase 1 may have sorted (it goes by the largest id, which is at least n_nodes - 1)
        int64_t max_id = 0;
        const int rf = fetch_small(&max_id, W.cnt + 3, sizeof(max_id), st);
        if (rf) return rf;
        small = small_route(n_raw, max_id);
    }
    if (n_edges > 0 && small) {
        TCHLL_ARG(n_nodes > 1, "sizes out of range");
        const int64_t slots = 2 * n_raw, tiles = (n_nodes + 1023) / 1024;
        const unsigned long long* table = reinterpret_cast<const unsigned long long*>(W.k0);
        const int32_t* rank = reinterpret_cast<const int32_t*>(W.e1);
        TCHLL_CUDA(cudaMemsetAsync(W.fdeg, 0, (size_t)n_nodes * sizeof(int32_t), st));
        small_count_kernel<<<grid_n(slots), 256, 0, st>>>(table, slots, W.deg, rank, W.fdeg);
        TCHLL_CHECK_LAUNCH("small_count_kernel");
        tile_sum_kernel<false><<<(int)tiles, 256, 0, st>>>(W.fdeg, n_nodes, W.ca);
        TCHLL_CHECK_LAUNCH("tile_sum_kernel");
        small_rows_kernel<<<(int)tiles, 256, 0, st>>>(W.fdeg, n_nodes, W.ca, W.e0, W.cnt, slots, W.deg, row_ptr, degrees,
                                                      node_ids, undirected_degrees);
        TCHLL_CHECK_LAUNCH("small_rows_kernel");
        small_scatter_kernel<<<grid_n(slots), 256, 0, st>>>(table, slots, W.deg, rank, W.fdeg, W.cb);
        TCHLL_CHECK_LAUNCH("small_scatter_kernel");
        const int64_t warps = 4 * (int64_t)sm_count() * 7;
        const int per = n_nodes >= 32 * warps ? 32 : 1;
        const int64_t g = per == 32 ? warps / 4 : (n_nodes + 3) / 4 < warps / 4 ? (n_nodes + 3) / 4 : warps / 4;
        small_sort_kernel<<<(int)g, 128, 0, st>>>(row_ptr, n_nodes, per, W.cb, col_idx, edge_u, edge_v);
        TCHLL_CHECK_LAUNCH("small_sort_kernel");
        return TCHLL_OK;
    }
    if (n_edges > 0) {
        // the pairs in the first half of k1's bytes (2 n_raw uint32 >= 2 n_edges);
        // sorted by src straight into edge_u (src) and col_idx (dst)
        uint32_t* okey = reinterpret_cast<uint32_t*>(W.k1);
        uint32_t* oval = okey + n_edges;
        const int kn = bits_for(n_nodes > 1 ? n_nodes - 1 : 1);
        orient_kernel<<<grid_n(n_edges), 256, 0, st>>>(W.k0, W.info, W.cnt, 2 * n_raw, W.ca, W.cb, n_edges, W.deg, okey,
                                                       oval);
        TCHLL_CHECK_LAUNCH("orient_kernel");
        size_t tb = W.tmp_bytes;
        TCHLL_CUDA(cub::DeviceRadixSort::SortPairs(W.tmp, tb, okey, reinterpret_cast<uint32_t*>(edge_u), oval,
                                                   reinterpret_cast<uint32_t*>(col_idx), (int)n_edges, 0, kn, st));
        count_launch();
        TCHLL_CUDA(cudaMemcpyAsync(edge_v, col_idx, (size_t)n_edges * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    }
    row_ptr_kernel<<<grid_n(n_edges + 1), 256, 0, st>>>(edge_u, n_edges, n_nodes, row_ptr);
    TCHLL_CHECK_LAUNCH("row_ptr_kernel");
    if (n_nodes > 0) {
        copy_nodes_kernel<<<grid_n(n_nodes), 256, 0, st>>>(W.e0, n_nodes, row_ptr, W.deg, W.cnt, 2 * n_raw, node_ids,
                                                            degrees, undirected_degrees);
        TCHLL_CHECK_LAUNCH("copy_nodes_kernel");
    }
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_adj_workspace_bytes(int64_t n, int64_t nnz, size_t* bytes) {
    TCHLL_ARG(bytes && n >= 0 && nnz >= 0, "bad arguments");
    TCHLL_ARG(n < (int64_t)INT32_MAX - 1 && nnz <= (int64_t)INT32_MAX, "int32 CSR limits exceeded");
    const int N = (int)(n > 0 ? n : 1);
    size_t a = 0, b = 0, c = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, a, (int64_t*)nullptr, (int64_t*)nullptr, N + 1);
    cub::DeviceRadixSort::SortPairs(nullptr, b, (int64_t*)nullptr, (int64_t*)nullptr, (int64_t*)nullptr,
                                    (int64_t*)nullptr, N);
    cub::DeviceScan::ExclusiveSum(nullptr, c, (int32_t*)nullptr, (int32_t*)nullptr, N + 1);
    size_t m = a > b ? a : b;
    if (c > m) m = c;
    Carve cv(nullptr, 0);
    cv.take<int64_t>((size_t)N + 1);  // dict offsets
    cv.take<int64_t>((size_t)N + 1);  // lens copy with trailing 0
    cv.take<int64_t>((size_t)N);      // iota
    cv.take<int32_t>((size_t)N + 1);  // degree scan input
    cv.take<char>(m);
    *bytes = cv.off;
    return TCHLL_OK;
}

TCHLL_EXPORT int tchll_csr_from_adjacency(const int64_t* keys, const int64_t* lens, int64_t n,
                                          const int64_t* values, int64_t nnz, int64_t* node_ids, int32_t* row_ptr,
                                          int32_t* degrees, int32_t* col_idx, int32_t* edge_u, int32_t* edge_v,
                                          int64_t* order, int64_t* missing, void* workspace, size_t workspace_bytes,
                                          void* stream) {
    TCHLL_ARG(n >= 0 && nnz >= 0, "negative size");
    TCHLL_ARG(row_ptr && missing, "null output");
    TCHLL_ARG(n == 0 || (keys && lens && node_ids && degrees && order), "null node arrays");
    TCHLL_ARG(nnz == 0 || (values && col_idx && edge_u && edge_v), "null edge arrays");
    size_t need = 0;
    int rc = tchll_adj_workspace_bytes(n, nnz, &need);
    if (rc) return rc;
    TCHLL_ARG(workspace != nullptr && workspace_bytes >= need, "workspace too small: need %zu bytes", need);
    const int N = (int)(n > 0 ? n : 1);
    size_t a = 0, b = 0, c = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, a, (int64_t*)nullptr, (int64_t*)nullptr, N + 1);
    cub::DeviceRadixSort::SortPairs(nullptr, b, (int64_t*)nullptr, (int64_t*)nullptr, (int64_t*)nullptr,
                                    (int64_t*)nullptr, N);
    cub::DeviceScan::ExclusiveSum(nullptr, c, (int32_t*)nullptr, (int32_t*)nullptr, N + 1);
    size_t m = a > b ? a : b;
    if (c > m) m = c;
    Carve cv(workspace, workspace_bytes);
    int64_t* dict_off = cv.take<int64_t>((size_t)N + 1);
    int64_t* lens0 = cv.take<int64_t>((size_t)N + 1);
    int64_t* iota = cv.take<int64_t>((size_t)N);
    int32_t* dscan = cv.take<int32_t>((size_t)N + 1);
    void* tmp = cv.take<char>(m);
    cudaStream_t st = (cudaStream_t)stream;
    zero_kernel<<<1, 1, 0, st>>>(missing);
    TCHLL_CHECK_LAUNCH("zero_kernel");
    if (n == 0) {
        TCHLL_CUDA(cudaMemsetAsync(row_ptr, 0, sizeof(int32_t), st));
        return TCHLL_OK;
    }
    TCHLL_CUDA(cudaMemcpyAsync(lens0, lens, sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, st));
    TCHLL_CUDA(cudaMemsetAsync(lens0 + n, 0, sizeof(int64_t), st));
    size_t tb = m;
    TCHLL_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, lens0, dict_off, (int)(n + 1), st));
    count_launch();
    iota_kernel<<<grid_n(n), 256, 0, st>>>(iota, n);
    TCHLL_CHECK_LAUNCH("iota_kernel");
    tb = m;
    TCHLL_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, keys, node_ids, iota, order, (int)n, 0, 64, st));
    count_launch();
    gather_deg_kernel<<<grid_n(n), 256, 0, st>>>(lens, order, n, degrees, dscan);
    TCHLL_CHECK_LAUNCH("gather_deg_kernel");
    tb = m;
    TCHLL_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, dscan, row_ptr, (int)(n + 1), st));
    count_launch();
    if (nnz > 0) {
        adj_fill_kernel<<<grid_n(nnz), 256, 0, st>>>(node_ids, n, order, dict_off, row_ptr, values, nnz, col_idx,
                                                    edge_u, edge_v, (unsigned long long*)missing);
        TCHLL_CHECK_LAUNCH("adj_fill_kernel");
    }
    return TCHLL_OK;
}
