// Host orchestration of the GPU build: build_vamana (algorithms/nsw.h:547-663) and
// NSWIndex::batch_insert (nsw.h:110-286).  Kernels live in build_impl.cuh.
//
// Host-side (sequential in the reference, cheap here): the insert order
// (std::shuffle with std::mt19937(pass), nsw.h:575,620), start points per insert
// (nsw.h:566-616), the batch schedule (nsw.h:30-47, 288-295), popularity
// propagation and alpha (nsw.h:255-278, 297-324) and isolated-node repair
// (algorithms/utils/Graph/dfs.h:193-254).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <numeric>
#include <random>
#include <unordered_map>
#include <vector>

#include "build_impl.cuh"
#include "build_flag.cuh"
#include "internal.h"

namespace nbpg {

SlotLayout make_slot_layout(uint32_t Lmax, uint32_t R, bool vis_smem, uint32_t Vcap, bool hash_smem, uint32_t Scap);

enum class Popular { FixedMin = 1, FixedMax, Cal, Prune };

template <int DT, int MET, int VPL>
struct BuildKernels {
    static cudaError_t setup(size_t smem_search, size_t smem_merge)
    {
        const cudaError_t e = raise_smem_limit(build_search_prune_kernel<DT, MET, VPL>, smem_search);
        return e == cudaSuccess ? raise_smem_limit(rev_merge_kernel<DT, MET, VPL>, smem_merge) : e;
    }
    static cudaError_t occ(uint32_t threads, size_t smem, int *blocks)
    {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, build_search_prune_kernel<DT, MET, VPL>, int(threads), smem);
    }
    static void search(uint32_t grid, uint32_t threads, size_t smem, const BuildArgs &B, cudaStream_t st)
    {
        build_search_prune_kernel<DT, MET, VPL><<<grid, threads, smem, st>>>(B);
    }
    static void merge(uint32_t grid, uint32_t threads, size_t smem, const BuildArgs &B, cudaStream_t st)
    {
        rev_merge_kernel<DT, MET, VPL><<<grid, threads, smem, st>>>(B);
    }
};

struct KernelTable {
    cudaError_t (*setup)(size_t, size_t);
    cudaError_t (*occ)(uint32_t, size_t, int *);
    void (*search)(uint32_t, uint32_t, size_t, const BuildArgs &, cudaStream_t);
    void (*merge)(uint32_t, uint32_t, size_t, const BuildArgs &, cudaStream_t);
};

template <int DT, int MET, int VPL>
static KernelTable table_of()
{
    return {BuildKernels<DT, MET, VPL>::setup, BuildKernels<DT, MET, VPL>::occ, BuildKernels<DT, MET, VPL>::search,
            BuildKernels<DT, MET, VPL>::merge};
}

template <int VPL>
static bool kernel_table_v(uint32_t dtype, uint32_t metric, KernelTable &t)
{
    const bool l2 = metric == NBPG_L2;
    switch (dtype) {
    case NBPG_U8: t = l2 ? table_of<DT_U8, M_L2, VPL>() : table_of<DT_U8, M_IP, VPL>(); return true;
    case NBPG_I8: t = l2 ? table_of<DT_I8, M_L2, VPL>() : table_of<DT_I8, M_IP, VPL>(); return true;
    case NBPG_U4:
    case NBPG_I4: t = l2 ? table_of<DT_U4, M_L2, VPL>() : table_of<DT_U4, M_IP, VPL>(); return true;
    default: return false;
    }
}

static bool kernel_table(uint32_t dtype, uint32_t metric, uint32_t vpl, KernelTable &t)
{
    return vpl == 1 ? kernel_table_v<1>(dtype, metric, t) : kernel_table_v<4>(dtype, metric, t);
}

void row_geometry(uint32_t row_stride, uint32_t want, uint32_t &vecs, uint32_t &lpr, uint32_t &vpl);
SlotLayout make_flag_layout(uint32_t Lmax, uint32_t R, uint32_t row_stride, bool hash_smem, uint32_t Scap, bool drop);
cudaError_t build_flag_search(uint32_t dtype, uint32_t metric, uint32_t grid, uint32_t warps, size_t smem,
                              const BuildFlagArgs &F, int *blocks, cudaStream_t st);
cudaError_t build_flag_prune(uint32_t dtype, uint32_t metric, uint32_t grid, const BuildFlagArgs &F, const PruneLayout &lay,
                             cudaStream_t st);

// ---------------------------------------------------------------------------
// Popularity (nsw.h:255-278): the reference walks the nodes in order, sets a node's total to its own visits
// and adds them to its neighbours' totals, so a node keeps what later nodes add: its visits plus those of the
// in-neighbours with larger ids.  Visits are counts, and float sums of them are exact in any order below
// 2^24: there the device adds them, as integers.  (A total at or past 2^24 or a self-loop, and the
// host walks as the reference does; so it does where the sums do not fit.)  The host's copy of the graph and its walk took 14 of the 227 ms of a
// 250k-row build.
// ---------------------------------------------------------------------------
static __global__ void __launch_bounds__(256) popular_spread_kernel(const uint32_t *graph, uint32_t gstride, uint32_t n,
                                                                    const float *visits, unsigned long long *sum,
                                                                    uint32_t *inexact)
{
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i = blockIdx.x * 8 + (threadIdx.x >> 5); i < n; i += gridDim.x * 8) {
        const unsigned long long v = (unsigned long long)(visits[i]);
        if (!v) continue;  // (the warp's own node)
        const uint32_t *row = graph + size_t(i) * gstride;
        const uint32_t deg = row[0];
        for (uint32_t j = lane; j < deg; j += 32) {
            const uint32_t r = row[1 + j];
            if (r < i) atomicAdd(&sum[r], v);
            if (r == i) *inexact = 1;  // a self-loop doubles the total as it is being added: the host's walk
        }
    }
}

static __global__ void popular_total_kernel(uint32_t n, const float *visits, const unsigned long long *sum, float *total,
                                            uint32_t *inexact)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long t = sum[i] + (unsigned long long)(visits[i]);
    if (t >= (1ull << 24)) *inexact = 1;
    total[i] = float(t);
}

// ---------------------------------------------------------------------------
// Isolated-node repair (dfs.h:63-137, 193-215).  Reachability from the entry is a breadth-first sweep on
// the device (which nodes are reached does not depend on the order); the repair itself depends on the order
// of the nodes, so it runs on the host, over copies of the few rows it can touch.  Copying the whole graph
// to the host and walking it there took 24 ms of a 61 ms build at 100k rows, 52 of 277 ms at 250k.
// ---------------------------------------------------------------------------
constexpr uint32_t REACH_LEVELS = 16;  // levels per round of launches
constexpr uint32_t REACH_MOST = 256;   // deeper graphs (long chains of one edge per node) are walked on the host

// One level: a warp per node of [head[level], head[level + 1]) of the queue marks its neighbours and appends
// the new ones.  `head` holds the queue's end after every level (head[0] = 0, head[1] = 1: the entry).
static __global__ void __launch_bounds__(256) reach_level_kernel(const uint32_t *graph, uint32_t gstride, uint32_t *seen,
                                                                 uint32_t *queue, uint32_t *head, uint32_t level)
{
    const uint32_t lane = threadIdx.x & 31, from = head[level], to = head[level + 1];
    for (uint32_t i = from + blockIdx.x * 8 + (threadIdx.x >> 5); i < to; i += gridDim.x * 8) {
        const uint32_t *row = graph + size_t(queue[i]) * gstride;
        const uint32_t deg = row[0];
        for (uint32_t j = 0; j < deg; j += 32) {
            const uint32_t v = j + lane < deg ? row[1 + j + lane] : 0u;
            const bool fresh = j + lane < deg && !((seen[v >> 5] >> (v & 31)) & 1) &&
                               !((atomicOr(&seen[v >> 5], 1u << (v & 31)) >> (v & 31)) & 1);
            const unsigned m = __ballot_sync(kFull, fresh);
            uint32_t at = 0;
            if (m && lane == 0) at = atomicAdd(&head[level + 2], uint32_t(__popc(m)));
            at = __shfl_sync(kFull, at, 0);
            // head[level + 2] counts this level's new nodes from zero; they follow those before
            if (fresh) queue[to + at + __popc(m & lanemask_lt())] = v;
        }
    }
}

// Turns the count of the level just run into the queue's end (one thread, after the level's kernel)
static __global__ void reach_close_kernel(uint32_t *head, uint32_t level) { head[level + 2] += head[level + 1]; }

static __global__ void reach_start_kernel(uint32_t *seen, uint32_t *queue, uint32_t *head, uint32_t entry)
{
    queue[0] = entry;
    head[1] = 1;
    seen[entry >> 5] = 1u << (entry & 31);
}

static __global__ void rows_gather_kernel(const uint32_t *graph, uint32_t gstride, uint32_t words, const uint32_t *ids,
                                          uint32_t *out)
{
    for (uint32_t j = threadIdx.x; j < words; j += blockDim.x)
        out[size_t(blockIdx.x) * words + j] = graph[size_t(ids[blockIdx.x]) * gstride + j];
}

static __global__ void rows_scatter_kernel(uint32_t *graph, uint32_t gstride, uint32_t words, const uint32_t *ids,
                                           const uint32_t *in)
{
    for (uint32_t j = threadIdx.x; j < words; j += blockDim.x)
        graph[size_t(ids[blockIdx.x]) * gstride + j] = in[size_t(blockIdx.x) * words + j];
}

// Host copies of graph rows: of those asked for, through the device's gather and scatter, or of the whole graph
struct HostRows {
    nbpg_index *idx;
    bool whole = false;
    std::unordered_map<uint32_t, uint32_t> at;  // node -> row in `rows`
    std::vector<uint32_t> ids, rows;
    DevBuf d_ids, d_rows;
    ReleaseOnExit release{{&d_ids, &d_rows}};
    explicit HostRows(nbpg_index *i) : idx(i) {}
    uint32_t words() const { return idx->desc.max_degree + 1; }
    bool has(uint32_t v) const { return whole || at.find(v) != at.end(); }
    uint32_t *row(uint32_t v) { return &rows[size_t(whole ? v : at.at(v)) * words()]; }

    nbpg_status fetch_all()
    {
        rows.resize(size_t(idx->desc.n) * words());
        NBPG_CUDA_TRY(cudaMemcpy2DAsync(rows.data(), words() * 4, idx->d_graph, idx->gstride * 4, words() * 4, idx->desc.n,
                                        cudaMemcpyDeviceToHost, idx->stream));
        NBPG_CUDA_TRY(cudaStreamSynchronize(idx->stream));
        whole = true;
        return NBPG_OK;
    }
    // between the rows ids[first, ids.size()) and the device, a piece at a time: pieces shrink to the room there is
    nbpg_status move(size_t first, bool back)
    {
        size_t piece = std::min<size_t>(ids.size() - first, 65536);
        while (d_ids.ensure(piece * 4) != NBPG_OK || d_rows.ensure(piece * words() * 4) != NBPG_OK) {
            cudaGetLastError();
            if (piece <= 64) return NBPG_ERR_OOM;
            piece /= 2;
        }
        cudaStream_t st = idx->stream;
        for (size_t i = first; i < ids.size(); i += piece) {
            const uint32_t cnt = uint32_t(std::min(piece, ids.size() - i));
            uint32_t *host = rows.data() + i * words();
            const size_t bytes = size_t(cnt) * words() * 4;
            NBPG_CUDA_TRY(cudaMemcpyAsync(d_ids.ptr, ids.data() + i, size_t(cnt) * 4, cudaMemcpyHostToDevice, st));
            if (back) NBPG_CUDA_TRY(cudaMemcpyAsync(d_rows.ptr, host, bytes, cudaMemcpyHostToDevice, st));
            if (back)
                rows_scatter_kernel<<<cnt, 64, 0, st>>>(idx->d_graph, idx->gstride, words(), d_ids.as<uint32_t>(),
                                                        d_rows.as<uint32_t>());
            else
                rows_gather_kernel<<<cnt, 64, 0, st>>>(idx->d_graph, idx->gstride, words(), d_ids.as<uint32_t>(),
                                                       d_rows.as<uint32_t>());
            NBPG_CUDA_TRY(cudaGetLastError());
            if (!back) NBPG_CUDA_TRY(cudaMemcpyAsync(host, d_rows.ptr, bytes, cudaMemcpyDeviceToHost, st));
            NBPG_CUDA_TRY(cudaStreamSynchronize(st));
        }
        return NBPG_OK;
    }
    nbpg_status fetch(const std::vector<uint32_t> &want)
    {
        if (whole) return NBPG_OK;
        const size_t old = ids.size();
        for (uint32_t v : want)
            if (at.emplace(v, uint32_t(ids.size())).second) ids.push_back(v);
        rows.resize(ids.size() * words());
        return old < ids.size() ? move(old, false) : NBPG_OK;
    }
    nbpg_status write_back()
    {
        if (!whole) return move(0, true);
        NBPG_CUDA_TRY(cudaMemcpy2DAsync(idx->d_graph, idx->gstride * 4, rows.data(), words() * 4, words() * 4, idx->desc.n,
                                        cudaMemcpyHostToDevice, idx->stream));
        NBPG_CUDA_TRY(cudaStreamSynchronize(idx->stream));
        return NBPG_OK;
    }
};

// dfs.h:46-59
static bool add_edge_if_possible(uint32_t *r, uint32_t R, uint32_t to)
{
    if (r[0] >= R) return false;
    for (uint32_t k = 0; k < r[0]; ++k)
        if (r[1 + k] == to) return true;
    r[1 + r[0]] = to;
    r[0] += 1;
    return true;
}

// The nodes reachable from the entry, as bits; *swept is false where the device's sweep is too deep or has no room
static nbpg_status reach_sweep(nbpg_index *idx, uint32_t entry, std::vector<uint32_t> &seen, bool *swept)
{
    const uint32_t n = uint32_t(idx->desc.n);
    cudaStream_t st = idx->stream;
    DevBuf d_seen, d_queue, d_head;
    ReleaseOnExit release{{&d_seen, &d_queue, &d_head}};
    const size_t heads = REACH_MOST + 2;
    *swept = false;
    if (d_seen.ensure(seen.size() * 4) != NBPG_OK || d_queue.ensure(size_t(n) * 4) != NBPG_OK ||
        d_head.ensure(heads * 4) != NBPG_OK) {
        cudaGetLastError();
        return NBPG_OK;
    }
    NBPG_CUDA_TRY(cudaMemsetAsync(d_seen.ptr, 0, seen.size() * 4, st));
    NBPG_CUDA_TRY(cudaMemsetAsync(d_head.ptr, 0, heads * 4, st));
    uint32_t *head = d_head.as<uint32_t>();
    reach_start_kernel<<<1, 1, 0, st>>>(d_seen.as<uint32_t>(), d_queue.as<uint32_t>(), head, entry);
    const uint32_t grid = uint32_t(std::min<size_t>(size_t(idx->sm_count) * 8, size_t(n) / 8 + 1));
    for (uint32_t level = 0; level < REACH_MOST && !*swept; ++level) {
        reach_level_kernel<<<grid, 256, 0, st>>>(idx->d_graph, idx->gstride, d_seen.as<uint32_t>(), d_queue.as<uint32_t>(),
                                                 head, level);
        reach_close_kernel<<<1, 1, 0, st>>>(head, level);
        NBPG_CUDA_TRY(cudaGetLastError());
        if ((level + 1) % REACH_LEVELS == 0) {
            uint32_t h[2];
            NBPG_CUDA_TRY(cudaMemcpyAsync(h, head + level + 1, 8, cudaMemcpyDeviceToHost, st));
            NBPG_CUDA_TRY(cudaStreamSynchronize(st));
            *swept = h[0] == h[1];  // the last level found nothing new
        }
    }
    if (*swept) {
        NBPG_CUDA_TRY(cudaMemcpyAsync(seen.data(), d_seen.ptr, seen.size() * 4, cudaMemcpyDeviceToHost, st));
        NBPG_CUDA_TRY(cudaStreamSynchronize(st));
    }
    return NBPG_OK;
}

// Every node unreachable from the entry gets an in-edge; *count receives how many there were.
static nbpg_status repair_isolated(nbpg_index *idx, uint32_t entry, uint64_t *count)
{
    const uint32_t R = idx->desc.max_degree, n = uint32_t(idx->desc.n);
    std::vector<uint32_t> seen((size_t(n) + 31) / 32, 0u);
    auto reached = [&](uint32_t v) { return ((seen[v >> 5] >> (v & 31)) & 1) != 0; };
    HostRows rows(idx);
    bool swept = false;
    nbpg_status s = reach_sweep(idx, entry, seen, &swept);
    if (s != NBPG_OK) return s;
    if (!swept) {
        if ((s = rows.fetch_all()) != NBPG_OK) return s;
        std::vector<uint32_t> queue{entry};
        seen[entry >> 5] |= 1u << (entry & 31);
        for (size_t h = 0; h < queue.size(); ++h) {
            const uint32_t *r = rows.row(queue[h]);
            for (uint32_t j = 0; j < r[0]; ++j)
                if (!reached(r[1 + j])) {
                    seen[r[1 + j] >> 5] |= 1u << (r[1 + j] & 31);
                    queue.push_back(r[1 + j]);
                }
        }
    }
    std::vector<uint32_t> lost;
    for (uint32_t w = 0; w < seen.size(); ++w) {
        uint32_t m = ~seen[w];
        if (size_t(w) * 32 + 32 > n) m &= (1u << (n & 31)) - 1u;
        for (; m; m &= m - 1) lost.push_back(w * 32 + uint32_t(__builtin_ctz(m)));
    }
    *count = lost.size();
    if (lost.empty()) return NBPG_OK;
    // The rows the repair reads and writes: the lost nodes', their neighbours' and the entry's.  From about a 128th of
    // the graph on, one copy of it is cheaper than looking each row up (1M rows of R = 32, by rows / by the copy: one in
    // 64 lost 78 / 48 ms, one in 1,000 6 / 48, all 2,071 / 236).
    if (lost.size() > n / 128 && !rows.whole && (s = rows.fetch_all()) != NBPG_OK) return s;
    if (!rows.whole) {
        std::vector<uint32_t> want(lost);
        want.push_back(entry);
        if ((s = rows.fetch(want)) != NBPG_OK) return s;
        want.clear();
        for (uint32_t i : lost) {
            const uint32_t *r = rows.row(i);
            want.insert(want.end(), r + 1, r + 1 + r[0]);
        }
        if ((s = rows.fetch(want)) != NBPG_OK) return s;
    }
    uint32_t open = 0;  // no reached node before it has room for an edge, and none gets any
    for (uint32_t i : lost) {
        // a neighbour list of its own: adding an edge below can lengthen this node's row while it is walked
        // only by the node itself, which add_edge_if_possible refuses to repeat
        bool done = false;
        for (uint32_t j = 0; j < rows.row(i)[0] && !done; ++j) {
            const uint32_t v = rows.row(i)[1 + j];
            if (reached(v)) done = add_edge_if_possible(rows.row(v), R, i);
        }
        for (uint32_t j = 0; j < rows.row(i)[0] && !done; ++j) {
            const uint32_t v = rows.row(i)[1 + j];
            if (!rows.has(v) && (s = rows.fetch({v})) != NBPG_OK) return s;
            done = add_edge_if_possible(rows.row(v), R, i);
        }
        if (!done) done = add_edge_if_possible(rows.row(entry), R, i);
        for (; open < n && !done; ++open) {  // (a full row refuses every edge, so the place is kept between nodes)
            if (!reached(open)) continue;
            if (!rows.has(open)) {
                // the nodes from here on, a thousand at a time
                std::vector<uint32_t> next;
                for (uint32_t y = open; y < n && next.size() < 1024; ++y)
                    if (reached(y)) next.push_back(y);
                if ((s = rows.fetch(next)) != NBPG_OK) return s;
            }
            if ((done = add_edge_if_possible(rows.row(open), R, i))) break;
        }
    }
    return rows.write_back();
}

struct DevArr {
    DevBuf b;
    template <class T>
    nbpg_status make(size_t count)
    {
        return b.ensure(count * sizeof(T));
    }
};

static nbpg_status build_impl(nbpg_index *idx, const nbpg_build_params &P, nbpg_build_stats *stats, uint32_t *out_sv,
                              uint32_t *out_sd, bool fgim = false)
{
    const auto t_start = std::chrono::steady_clock::now();
    const uint64_t n = idx->desc.n;
    const uint32_t R = idx->desc.max_degree;
    const uint32_t L = P.L, VL = P.VL;
    NBPG_CHECK_ARG(L >= 1 && L <= 1024, "L must be in [1, 1024]");
    NBPG_CHECK_ARG(VL >= 1 && VL + R <= 256, "VL + R must be at most 256");
    NBPG_CHECK_ARG(P.top_degree <= R, "top_degree above R");
    NBPG_CHECK_ARG(P.num_split <= L && P.num_split <= 256, "num_split start points exceed L");
    NBPG_CHECK_ARG(n >= 1 && n < 0xFFFFFFFFull, "bad n");
    NBPG_CHECK_ARG(!fgim || P.num_split >= 1, "the FGIM build needs num_split >= 1 (with none, the reference's "
                                              "pair pass reads a stale visited list)");
    uint32_t vecs, lpr, vpl;
    row_geometry(idx->row_stride, 0, vecs, lpr, vpl);
    NBPG_CHECK_ARG(vecs <= 128, "rows above 2048 bytes are not supported");
    KernelTable kt{};
    NBPG_CHECK_ARG(kernel_table(idx->desc.dtype, idx->desc.metric, vpl, kt), "unsupported dtype");
    cudaStream_t st = idx->stream;
    nbpg_status s;

    // geometry shared with the search kernels
    SearchArgs sa{};
    sa.base = idx->d_points;
    sa.row_stride = idx->row_stride;
    sa.vecs = vecs;
    sa.lpr = lpr;
    sa.vpl = vpl;
    sa.graph = idx->d_graph;
    sa.gstride = idx->gstride;
    sa.R = R;
    sa.n = n;
    sa.limit = P.limit ? P.limit : n;
    sa.degree_limit = R;
    sa.visited_factor = 0;
    sa.prefetch = 2;
    const uint32_t S = filter_slots_for(L);
    const bool ghash = S * 4 > 32768;
    const uint32_t Lmax = std::max(std::max(L, R), VL);
    sa.lay = make_slot_layout(Lmax, R, true, VL, !ghash, S);
    NBPG_CHECK_ARG(sa.lay.bytes <= idx->smem_optin, "per-insert working set exceeds shared memory");
    const uint32_t W = std::max<uint32_t>(1, std::min<uint32_t>(16, uint32_t(idx->smem_optin / sa.lay.bytes)));
    const size_t smem_search = size_t(W) * sa.lay.bytes;
    const uint32_t MW = 8;
    const size_t smem_merge = size_t(MW) * kMergeWarpBytes;
    NBPG_CUDA_TRY(kt.setup(smem_search, smem_merge));
    int blocks = 0;
    NBPG_CUDA_TRY(kt.occ(W * 32, smem_search, &blocks));
    NBPG_CHECK_ARG(blocks >= 1, "build kernel does not fit on an SM");
    const uint32_t full_grid = uint32_t(blocks) * uint32_t(idx->sm_count);
    const size_t nslots = size_t(full_grid) * W;
    if (ghash) {
        if ((s = idx->ghash.ensure(nslots * S * 4)) != NBPG_OK) return s;
        sa.g_hash = idx->ghash.as<uint32_t>();
        sa.g_hash_slots = S;
    }

    // The search and prune kernels of build_flag.cuh where their argument holds (VL >= L); a biased candidate
    // order and FGIM's pair pass stay on the one-kernel insert.
    bool flag = VL >= L && P.dir_bias_scale <= 0;
    SlotLayout flay{};
    PruneLayout play{};
    uint32_t fw = 0, fgrid = 0, fout = 0;  // warps per CTA, CTAs, warps per CTA with a filter in global memory
    size_t fsmem = 0;
    BuildFlagArgs F{};
    F.B.s = sa;
    if (flag) {
        row_geometry(idx->row_stride, 4, F.B.s.vecs, F.B.s.lpr, F.B.s.vpl);
        flay = make_flag_layout(L, R, idx->row_stride, !ghash, S, false);
        play = make_prune_layout(VL, R, idx->row_stride);
        flag = flay.bytes <= idx->smem_optin && play.bytes <= idx->smem_optin;
    }
    if (flag) {
        // 16 warps per CTA: those whose filter fits in shared memory, the rest with theirs in global memory
        // (slower by the probes' round trips, but a batch's last inserts no longer wait for a second turn)
        F.lay_g = make_flag_layout(L, R, idx->row_stride, false, S, false);
        F.own = ghash ? 0 : std::min<uint32_t>(16, uint32_t(idx->smem_optin / flay.bytes));
        const size_t left = idx->smem_optin - F.own * size_t(flay.bytes);
        fout = std::min<uint32_t>(16 - F.own, uint32_t(left / F.lay_g.bytes));
        fw = F.own + fout;
        fsmem = F.own * size_t(flay.bytes) + fout * size_t(F.lay_g.bytes);
        int fb = 0;
        NBPG_CUDA_TRY(build_flag_search(idx->desc.dtype, idx->desc.metric, 0, fw, fsmem, F, &fb, st));
        NBPG_CUDA_TRY(build_flag_prune(idx->desc.dtype, idx->desc.metric, 0, F, play, st));
        flag = fb >= 1;
        fgrid = uint32_t(fb) * uint32_t(idx->sm_count);
    }

    // batch size (nsw.h:288-295): min(0.02 * n (through float), 1e6), at least 1
    size_t eff = std::min<size_t>(size_t(0.02 * double(float(n))), 1000000ul);
    if (eff == 0) eff = 1;
    const uint32_t nsp_max = std::max<uint32_t>(1, P.num_split);

    DevBuf d_inserts, d_sp, d_alpha, d_cos, d_pop, d_sv, d_sd, d_res_ids, d_res_d, d_res_cnt, d_rank, d_cnt, d_off,
        d_bump, d_grp, d_left, d_edges, d_bias, d_row_d, d_vis, d_near, d_info;
    ReleaseOnExit release_bufs{{&d_left, &d_row_d, &d_vis, &d_near, &d_info, &d_inserts, &d_sp, &d_alpha, &d_cos, &d_pop, &d_sv, &d_sd, &d_res_ids, &d_res_d,
                                &d_res_cnt, &d_rank, &d_cnt, &d_off, &d_bump, &d_grp, &d_edges, &d_bias}};
    auto fail_oom = [&](nbpg_status x) { return x; };
    if ((s = d_inserts.ensure(n * 4)) || (s = d_sp.ensure(n * nsp_max * 4)) || (s = d_alpha.ensure(n * 4)) ||
        (s = d_cos.ensure(n * 4)) || (s = d_pop.ensure(n * 4)) || (s = d_sv.ensure(n * 4)) ||
        (s = d_sd.ensure(n * 4)) || (s = d_res_ids.ensure(eff * R * 4)) || (s = d_res_d.ensure(eff * R * 4)) ||
        (s = d_res_cnt.ensure(eff * 4)) || (s = d_rank.ensure(eff * R * 4)) || (s = d_cnt.ensure(n * 4)) ||
        (s = d_off.ensure(n * 4)) || (s = d_bump.ensure(32)) || (s = d_grp.ensure(eff * R * 4)) ||
        (s = d_edges.ensure(eff * R * 8)))
        return fail_oom(s);
    // FGIM: the graph the pair passes write (toG), which becomes the index's graph
    DevBuf d_tog;
    ReleaseOnExit release_tog{{&d_tog}};
    if (fgim && (s = d_tog.ensure(size_t(n) * idx->gstride * 4)) != NBPG_OK) return s;
    if (P.dir_bias_scale > 0 && (s = d_bias.ensure(size_t(R + 1) * sizeof(double))) != NBPG_OK) return s;
    // What follows makes the build faster and is left out where it does not fit, so it comes after all that is needed.
    if (flag && fout) {
        if (idx->ghash.ensure(std::max(ghash ? nslots : 0, size_t(fgrid) * fout) * S * 4) != NBPG_OK) {
            cudaGetLastError();  // no room: the one-kernel insert needs less
            flag = false;
            if (ghash && (s = idx->ghash.ensure(nslots * S * 4)) != NBPG_OK) return s;
        }
        if (ghash) sa.g_hash = idx->ghash.as<uint32_t>();
    }
    NBPG_CUDA_TRY(cudaMemsetAsync(d_cnt.ptr, 0, n * 4, st));
    NBPG_CUDA_TRY(cudaMemsetAsync(d_sv.ptr, 0, n * 4, st));
    NBPG_CUDA_TRY(cudaMemsetAsync(d_sd.ptr, 0, n * 4, st));

    // The neighbours' distances beside the graph, for rev_insert_kernel.  With top_degree the merge
    // orders by interpolated distances: then, and where this does not fit, every target takes the
    // general merge.
    bool keep_d = P.top_degree == 0 || P.top_degree == R;
    if (keep_d && ((s = d_left.ensure(eff * R * 4)) || (s = d_row_d.ensure(size_t(n) * R * 4)))) {
        cudaGetLastError();
        keep_d = false;
    }

    if (flag) {
        flag = d_vis.ensure(eff * FLAG_VIS * 8) == NBPG_OK && d_near.ensure(eff * R * 8) == NBPG_OK &&
               d_info.ensure(eff * 16) == NBPG_OK;
        if (!flag) cudaGetLastError();
        F.vis = d_vis.as<uint64_t>();
        F.near = d_near.as<uint64_t>();
        F.info = d_info.as<uint4>();
    }

    BuildArgs B{};
    B.s = sa;
    B.L = L;
    B.VL = VL;
    B.R = R;
    B.top_degree = P.top_degree == 0 ? R : P.top_degree;
    B.res_ids = d_res_ids.as<uint32_t>();
    B.res_d = d_res_d.as<float>();
    B.res_cnt = d_res_cnt.as<uint32_t>();
    B.stat_vis = d_sv.as<uint32_t>();
    B.stat_dist = d_sd.as<uint32_t>();
    B.rank = d_rank.as<uint32_t>();
    B.cnt_node = d_cnt.as<uint32_t>();
    B.off_node = d_off.as<uint32_t>();
    B.bump = d_bump.as<uint32_t>();
    B.grp_target = d_grp.as<uint32_t>();
    B.edges = d_edges.as<uint64_t>();
    if (keep_d) {
        B.row_d = d_row_d.as<float>();
        B.grp_left = d_left.as<uint32_t>();
        rows_unknown_kernel<<<uint32_t((n + 255) / 256), 256, 0, st>>>(B);
        NBPG_CUDA_TRY(cudaGetLastError());
    }
    B.dir_bias = nullptr;
    std::vector<double> bias_host;
    if (P.dir_bias_scale > 0) {
        // sort_candidates' factor dir_bias_scale * log(degree + 1) + 1 in double, the float scale
        // widened as the reference's expression widens it (prune.h:59-63); a degree is at most R
        bias_host.resize(R + 1);
        for (uint32_t d = 0; d <= R; ++d) bias_host[d] = P.dir_bias_scale * std::log(double(d + 1)) + 1;
        NBPG_CUDA_TRY(cudaMemcpyAsync(d_bias.ptr, bias_host.data(), size_t(R + 1) * sizeof(double),
                                      cudaMemcpyHostToDevice, st));
        B.dir_bias = d_bias.as<double>();
    }

    const float min_alpha = float(P.min_alpha), max_alpha = float(P.max_alpha);
    const float min_cos = float(P.min_cos_angle), max_cos = float(P.max_cos_angle);
    std::vector<float> popular;  // log-popularity after a popularity pass
    float min_pop = 0.f, max_pop = 1.f;
    std::vector<uint32_t> inserts(n);
    std::iota(inserts.begin(), inserts.end(), 0u);
    std::vector<uint32_t> sp_host;
    std::mt19937 sp_engine{uint32_t(P.sp_seed)};
    uint64_t batches = 0;

    uint32_t *tog = nullptr;
    if (fgim) {
        tog = d_tog.as<uint32_t>();
        NBPG_CUDA_TRY(cudaMemsetAsync(tog, 0, size_t(n) * idx->gstride * 4, st));
    }

    // one pass of batch_insert over `inserts` with nsp start points per insert; `sg` is the
    // graph searched, `wg` the graph written (the same except in FGIM's pair passes, which
    // run pair_batch_insert's searchNghAndPrune and finish popularity without propagation)
    auto run_pass = [&](uint32_t nsp, Popular mode, uint32_t *sg, uint32_t *wg, bool pair) -> nbpg_status {
        B.s.graph = sg;
        B.pair = pair ? 1u : 0u;
        NBPG_CUDA_TRY(cudaMemcpyAsync(d_inserts.ptr, inserts.data(), n * 4, cudaMemcpyHostToDevice, st));
        NBPG_CUDA_TRY(cudaMemcpyAsync(d_sp.ptr, sp_host.data(), n * nsp * 4, cudaMemcpyHostToDevice, st));
        B.nsp_per = nsp;
        B.alpha_node = nullptr;
        B.cos_node = nullptr;
        B.popular = nullptr;
        if (mode == Popular::FixedMin) { B.alpha_all = max_alpha; B.cos_all = max_cos; }
        else if (mode == Popular::Prune) {
            // nsw.h:309-315, in float as the reference
            std::vector<float> al(n), co(n);
            for (uint64_t v = 0; v < n; ++v) {
                float cof = (popular[v] - max_pop) / (min_pop - max_pop);
                float t1 = cof * (max_alpha - min_alpha);
                al[v] = min_alpha + t1;
                float t2 = cof * (max_cos - min_cos);
                co[v] = min_cos + t2;
            }
            NBPG_CUDA_TRY(cudaMemcpyAsync(d_alpha.ptr, al.data(), n * 4, cudaMemcpyHostToDevice, st));
            NBPG_CUDA_TRY(cudaMemcpyAsync(d_cos.ptr, co.data(), n * 4, cudaMemcpyHostToDevice, st));
            NBPG_CUDA_TRY(cudaStreamSynchronize(st));
            B.alpha_node = d_alpha.as<float>();
            B.cos_node = d_cos.as<float>();
        } else { B.alpha_all = 1.0f; B.cos_all = min_cos; }
        if (mode == Popular::Cal) {
            NBPG_CUDA_TRY(cudaMemsetAsync(d_pop.ptr, 0, n * 4, st));
            B.popular = d_pop.as<float>();
        }
        size_t inc = 0, count = 0;
        while (count < n) {
            size_t lo, hi;
            if (std::pow(2.0, double(inc)) <= double(eff)) {
                lo = size_t(std::pow(2.0, double(inc))) - 1;
                hi = std::min(size_t(std::pow(2.0, double(inc + 1))) - 1, size_t(n));
                count = hi;
            } else {
                lo = count;
                hi = std::min(count + eff, size_t(n));
                count = count + (hi - lo);
            }
            ++inc;
            ++batches;
            const uint32_t bs = uint32_t(hi - lo);
            if (bs == 0) continue;
            B.inserts = d_inserts.as<uint32_t>() + lo;
            B.sp = d_sp.as<uint32_t>() + lo * nsp;
            B.bs = bs;
            B.queue = B.bump + 4;  // bump: edge allocator, groups, groups left; from 4 the work counters
            NBPG_CUDA_TRY(cudaMemsetAsync(d_bump.ptr, 0, 32, st));
            const uint32_t g1 = std::min<uint32_t>(full_grid, (bs + W - 1) / W);
            if (flag && !pair) {
                const SearchArgs geometry = F.B.s;  // this kernel's lanes per row
                F.B = B;
                F.B.s.lpr = geometry.lpr;
                F.B.s.vpl = geometry.vpl;
                F.B.s.lay = flay;
                F.B.s.g_hash = idx->ghash.as<uint32_t>();
                F.B.s.g_hash_slots = S;
                const uint32_t gf = std::min<uint32_t>(fgrid, (bs + fw - 1) / fw);
                NBPG_CUDA_TRY(build_flag_search(idx->desc.dtype, idx->desc.metric, gf, fw, fsmem, F, nullptr, st));
                NBPG_CUDA_TRY(build_flag_prune(idx->desc.dtype, idx->desc.metric, bs, F, play, st));
            } else {
                kt.search(g1, W * 32, smem_search, B, st);
            }
            BuildArgs Wr = B;
            Wr.s.graph = wg;
            forward_write_kernel<<<bs, 64, 0, st>>>(Wr);
            const uint32_t ne = bs * R;
            const uint32_t eg = (ne + 255) / 256;
            rev_count_kernel<<<eg, 256, 0, st>>>(B);
            rev_alloc_kernel<<<eg, 256, 0, st>>>(B);
            rev_scatter_kernel<<<eg, 256, 0, st>>>(B);
            BuildArgs M = Wr;
            M.queue = B.bump + 5;
            if (keep_d) {
                const uint32_t gi = std::min<uint32_t>(uint32_t(idx->sm_count) * 8, (ne + 7) / 8);
                if (R <= 32) rev_insert_kernel<1><<<gi, 256, 0, st>>>(M);
                else if (R <= 64) rev_insert_kernel<2><<<gi, 256, 0, st>>>(M);
                else rev_insert_kernel<4><<<gi, 256, 0, st>>>(M);
            }
            const uint32_t gm = std::min<uint32_t>(uint32_t(idx->sm_count) * 8, (ne + MW - 1) / MW);
            kt.merge(gm, MW * 32, smem_merge, M, st);
            NBPG_CUDA_TRY(cudaGetLastError());
        }
        NBPG_CUDA_TRY(cudaStreamSynchronize(st));
        if (mode == Popular::Cal && pair) {
            // FGIM_nsw.h:164-172: log(x + 1) of the visit counts, min/max, no propagation
            popular.resize(n);
            NBPG_CUDA_TRY(cudaMemcpyAsync(popular.data(), d_pop.ptr, n * 4, cudaMemcpyDeviceToHost, st));
            NBPG_CUDA_TRY(cudaStreamSynchronize(st));
            for (uint64_t i = 0; i < n; ++i) popular[i] = float(std::log(double(popular[i] + 1.0f)));
            auto mm = std::minmax_element(popular.begin(), popular.end());
            min_pop = *mm.first;
            max_pop = *mm.second;
        } else if (mode == Popular::Cal) {
            // nsw.h:255-278: one-hop propagation in node order, log(x + 1), min/max
            std::vector<float> tmp(n, 0.0f);
            DevBuf d_sum, d_total;
            ReleaseOnExit release_pop{{&d_sum, &d_total}};
            uint32_t inexact = 0;
            if (d_sum.ensure(n * 8 + 4) != NBPG_OK || d_total.ensure(n * 4) != NBPG_OK) {
                cudaGetLastError();
                inexact = 1;
            } else {
                auto *sum = d_sum.as<unsigned long long>();
                uint32_t *d_inexact = reinterpret_cast<uint32_t *>(sum + n);
                NBPG_CUDA_TRY(cudaMemsetAsync(sum, 0, n * 8 + 4, st));
                popular_spread_kernel<<<uint32_t(idx->sm_count) * 8, 256, 0, st>>>(wg, idx->gstride, uint32_t(n),
                                                                                  d_pop.as<float>(), sum, d_inexact);
                popular_total_kernel<<<uint32_t((n + 255) / 256), 256, 0, st>>>(uint32_t(n), d_pop.as<float>(), sum,
                                                                               d_total.as<float>(), d_inexact);
                NBPG_CUDA_TRY(cudaGetLastError());
                NBPG_CUDA_TRY(cudaMemcpyAsync(tmp.data(), d_total.ptr, n * 4, cudaMemcpyDeviceToHost, st));
                NBPG_CUDA_TRY(cudaMemcpyAsync(&inexact, d_inexact, 4, cudaMemcpyDeviceToHost, st));
                NBPG_CUDA_TRY(cudaStreamSynchronize(st));
            }
            if (inexact) {
                std::vector<float> pop(n);
                std::vector<uint32_t> G(size_t(n) * (R + 1));
                NBPG_CUDA_TRY(cudaMemcpyAsync(pop.data(), d_pop.ptr, n * 4, cudaMemcpyDeviceToHost, st));
                NBPG_CUDA_TRY(cudaMemcpy2DAsync(G.data(), (R + 1) * 4, wg, idx->gstride * 4, (R + 1) * 4, n,
                                                cudaMemcpyDeviceToHost, st));
                NBPG_CUDA_TRY(cudaStreamSynchronize(st));
                std::fill(tmp.begin(), tmp.end(), 0.0f);
                for (uint64_t i = 0; i < n; ++i) {
                    tmp[i] = pop[i];
                    const uint32_t *r = &G[i * (R + 1)];
                    for (uint32_t j = 0; j < r[0]; ++j) tmp[r[1 + j]] += tmp[i];
                }
            }
            popular.resize(n);
            for (uint64_t i = 0; i < n; ++i) popular[i] = float(std::log(double(tmp[i] + 1.0f)));
            auto mm = std::minmax_element(popular.begin(), popular.end());
            min_pop = *mm.first;
            max_pop = *mm.second;
        }
        return NBPG_OK;
    };

    Popular mode = Popular::FixedMax;
    const uint32_t ns = P.num_split;
    uint32_t *G0 = idx->d_graph;
    // split stage (nsw.h:562-575; FGIM.cpp:201-220 runs it only for num_split > 1)
    if (fgim ? ns > 1 : ns >= 1) {
        for (int i = 0; i < 2; ++i) {
            std::shuffle(inserts.begin(), inserts.end(), std::mt19937(i));
            sp_host.resize(n);
            for (uint64_t j = 0; j < n; ++j) sp_host[j] = inserts[j] % ns;
            if ((s = run_pass(1, mode, G0, G0, false)) != NBPG_OK) return s;
        }
    }
    for (int i = 0; i < int(P.num_passes); ++i) {
        std::shuffle(inserts.begin(), inserts.end(), std::mt19937(i));
        if (i == int(P.num_passes) - 2 && P.dynamic_prune) mode = Popular::Cal;
        else if (i == int(P.num_passes) - 1)
            mode = (P.dynamic_prune && P.num_passes > 1) ? Popular::Prune : Popular::FixedMin;
        else if (fgim) mode = Popular::FixedMax;
        const bool last = i == int(P.num_passes) - 1;
        if (fgim && !last) {
            // FGIM.cpp:244-249: pair pass on (G -> toG) with start points 0 .. num_split-1
            sp_host.resize(size_t(n) * ns);
            for (uint64_t j = 0; j < n; ++j)
                for (uint32_t k = 0; k < ns; ++k) sp_host[j * ns + k] = k;
            if ((s = run_pass(ns, mode, G0, tog, true)) != NBPG_OK) return s;
            continue;
        }
        uint32_t nsp = 1;
        if (!last && ns > 1) {
            nsp = ns;
            sp_host.resize(n * ns);
            std::uniform_int_distribution<uint32_t> u(0, uint32_t(n) - 1);
            for (uint64_t j = 0; j < n; ++j)
                for (uint32_t k = 0; k < ns; ++k) {
                    uint32_t rid = u(sp_engine) / ns * ns;
                    uint32_t v = rid + k;
                    if (v >= n) v -= ns;
                    sp_host[j * ns + k] = v;
                }
        } else if (last && P.rand_sp) {
            sp_host.resize(n);
            for (uint64_t j = 0; j < n; ++j) sp_host[j] = uint32_t(n - inserts[j] - 1);
        } else {
            sp_host.assign(n, 0u);
        }
        uint32_t *g = fgim ? tog : G0;  // FGIM's last pass is batch_insert on toG
        if ((s = run_pass(nsp, mode, g, g, false)) != NBPG_OK) return s;
    }
    if (fgim) {
        // toG is the FGIM result (FGIM.cpp:259-263)
        NBPG_CUDA_TRY(cudaMemcpyAsync(idx->d_graph, tog, size_t(n) * idx->gstride * 4, cudaMemcpyDeviceToDevice, st));
        NBPG_CUDA_TRY(cudaStreamSynchronize(st));
        d_tog.release();
    }

    if (out_sv) NBPG_CUDA_TRY(cudaMemcpyAsync(out_sv, d_sv.ptr, n * 4, cudaMemcpyDeviceToHost, st));
    if (out_sd) NBPG_CUDA_TRY(cudaMemcpyAsync(out_sd, d_sd.ptr, n * 4, cudaMemcpyDeviceToHost, st));
    NBPG_CUDA_TRY(cudaStreamSynchronize(st));
    uint64_t iso = 0;
    if (P.repair_isolate) {
        for (DevBuf *b : release_bufs.bufs) b->release();  // the repair's rows find room where the batches' were
        if ((s = repair_isolated(idx, 0, &iso)) != NBPG_OK) return s;
    }
    if (stats) {
        stats->isolated = iso;
        stats->batches = batches;
        stats->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
    }
    return NBPG_OK;
}

}  // namespace nbpg

using namespace nbpg;

extern "C" nbpg_status nbpg_build(nbpg_index *idx, const nbpg_build_params *params, nbpg_build_stats *stats,
                                  uint32_t *per_node_visited, uint32_t *per_node_dists)
{
    if (!idx || !params) { set_error("null argument"); return NBPG_ERR_INVALID_ARG; }
    std::lock_guard<std::mutex> g(idx->mu);
    cudaSetDevice(idx->desc.device);
    return build_impl(idx, *params, stats, per_node_visited, per_node_dists);
}

extern "C" nbpg_status nbpg_build_fgim(nbpg_index *idx, const nbpg_build_params *params, nbpg_build_stats *stats,
                                       uint32_t *per_node_visited, uint32_t *per_node_dists)
{
    if (!idx || !params) { set_error("null argument"); return NBPG_ERR_INVALID_ARG; }
    std::lock_guard<std::mutex> g(idx->mu);
    cudaSetDevice(idx->desc.device);
    return build_impl(idx, *params, stats, per_node_visited, per_node_dists, true);
}
