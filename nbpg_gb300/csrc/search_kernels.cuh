// The strict search kernels: FLAG mode first (search_core, or search_flag for beams above 32 and for inner
// product), then LIST mode for the queries it marks.
#pragma once
#include "search_flag.cuh"

namespace nbpg {

// One query of a search request: argument checks, search_core, outputs.
template <int DT, int MET, int PASS, int VPL, bool GH, bool PLAIN = false>
__device__ void search_query(const SearchArgs &a, uint32_t qi, uint8_t *slot, uint32_t gslot, int lane)
{
    constexpr bool LIST = PASS == PASS_LIST;
    const uint32_t L = a.Ls ? a.Ls[qi] : a.L_all;
    const uint32_t k = a.ks ? a.ks[qi] : a.k_all;
    const uint32_t S = filter_slots_for(L);
    const uint64_t max_visited = uint64_t(a.visited_factor) * L;
    const uint32_t *sp = a.sp;
    uint32_t nsp = a.nsp;
    if (a.sp_stride) {
        sp = a.sp + size_t(qi) * a.sp_stride;
        nsp = 1;
        while (nsp < a.sp_stride && sp[nsp] != kNoId) ++nsp;
    }
    if (L == 0 || k == 0 || k > L || L > a.lay.Lcap || nsp > L || k > a.k_stride ||
        (LIST && !a.g_vis && max_visited > a.lay.Vcap) || (!a.g_hash && S > a.lay.Scap) ||
        (a.g_hash && S > a.g_hash_slots) || (LIST && a.g_vis && max_visited > a.g_vis_cap) ||
        (PASS == PASS_WIDE && MET == M_IP && max_visited > a.vis_most)) {
        // rejected (the reference aborts on k > L, beamSearch.h:268-273): empty row + error flag
        for (uint32_t j = lane; j < a.k_stride; j += 32) {
            a.out_ids[size_t(qi) * a.k_stride + j] = kNoId;
            if (a.out_dists) a.out_dists[size_t(qi) * a.k_stride + j] = __int_as_float(0x7f800000);
        }
        if (lane == 0) {
            if (a.out_count) a.out_count[qi] = 0;
            if (a.out_visited) a.out_visited[qi] = 0;
            if (a.out_cmps) a.out_cmps[qi] = 0;
            if (a.err) atomicExch(a.err, 1u);
        }
        __syncwarp();
        return;
    }

    const uint8_t *qrow = a.queries + size_t(qi) * a.row_stride;
    const uint64_t *frb, *vis = nullptr;
    uint32_t fs, cmps, adj, vs = 0, ins = 0;
    uint64_t nvis;
    bool taint;
    if constexpr (PASS == PASS_WIDE) {
        const FlagState st = search_flag<DT, MET, VPL, false, MET == M_IP, GH>(a, qrow, L, k, max_visited, sp, nsp, a.lay, slot,
                                                                               gslot, lane, kNoId, FlagVisited{});
        frb = st.fr;
        fs = st.fs, cmps = st.cmps, adj = st.adj, nvis = st.nvis, taint = st.taint;
    } else {
        const SearchState st = search_core<DT, MET, LIST, VPL, PLAIN>(a, qrow, L, k, max_visited, sp, nsp, slot, gslot, lane, kNoId);
        frb = st.frontier();
        vis = st.vis;
        fs = st.fs, cmps = st.cmps, adj = st.adj, nvis = st.nvis, taint = st.taint;
        vs = st.vs, ins = st.ins;
    }

    // results: frontier[0:min(k, fs)] (beamSearch.h:249-254); for a re-rank, frontier[0 :
    // min(k * rerank_factor, fs)] (beamSearch.h:219-222) or, in filtering mode, the visited
    // list (beamSearch.h:236-243), whose exact distances a later pass computes
    const uint64_t *src = frb;
    uint32_t kk;
    uint32_t cmps_out = cmps;
    if (LIST && a.emit_visited) {
        src = vis;
        kk = vs < a.k_stride ? vs : a.k_stride;
        cmps_out += ins;
    } else {
        uint64_t want = uint64_t(k) * (a.emit_factor ? a.emit_factor : 1u);
        if (want > a.k_stride) want = a.k_stride;
        kk = want < fs ? uint32_t(want) : fs;
    }
    for (uint32_t j = lane; j < a.k_stride; j += 32) {
        const size_t o = size_t(qi) * a.k_stride + j;
        if (j < kk) {
            const uint64_t key = src[j];
            a.out_ids[o] = key_id(key);
            if (a.out_dists) a.out_dists[o] = output_dist<MET>(key_dist(key));
        } else {
            a.out_ids[o] = kNoId;
            if (a.out_dists) a.out_dists[o] = __int_as_float(0x7f800000);
        }
    }
    if (lane == 0) {
        if (a.out_count) a.out_count[qi] = kk;
        if (a.out_visited) a.out_visited[qi] = uint32_t(nvis);
        if (a.out_cmps) a.out_cmps[qi] = cmps_out;
        if (a.out_adj) a.out_adj[qi] = adj;
        if (a.out_fs) a.out_fs[qi] = fs;
        if constexpr (!LIST) {
            if (taint && a.taint) {
                const uint32_t t = atomicAdd(a.taint, 1u);
                a.taint[1 + t] = qi;
            }
        }
    }
    __syncwarp();
}

// Persistent form: warps pull queries from a device queue until it runs dry.  Capped at
// 80 registers (the one-warp form settles at 72 unconstrained): at the 128 that a
// 512-thread bound allows, only 16 warps fit per SM; at 80, 24 do (a few bytes spill).
template <int DT, int MET, int PASS, int VPL>
__global__ void __maxnreg__(80) search_batched_kernel(SearchArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t *slot = smem + size_t(warp) * a.lay.bytes;
    const uint32_t gslot = blockIdx.x * (blockDim.x >> 5) + warp;
    const uint32_t total = a.only ? a.only[0] : a.nq;
    while (true) {
        uint32_t w = 0;
        if (lane == 0) w = atomicAdd(a.queue, 1u);
        w = __shfl_sync(kFull, w, 0);
        if (w >= total) break;
        const uint32_t qi = a.only ? a.only[1 + w] : (a.order ? a.order[w] : w);
        if (PASS == PASS_WIDE && a.g_hash) search_query<DT, MET, PASS, VPL, true>(a, qi, slot, gslot, lane);
        else search_query<DT, MET, PASS, VPL, false>(a, qi, slot, gslot, lane);
    }
}

// Plain form: one query per thread block of one warp; everything in shared memory.  Held
// to 72 registers so that 28 blocks (warps) fit per SM.
template <int DT, int MET, int PASS, int VPL>
__global__ void __launch_bounds__(32, 28) search_plain_kernel(SearchArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t total = a.only ? a.only[0] : a.nq;
    if (blockIdx.x >= total) return;
    const uint32_t qi = a.only ? a.only[1 + blockIdx.x] : (a.order ? a.order[blockIdx.x] : blockIdx.x);
    search_query<DT, MET, PASS, VPL, false, true>(a, qi, smem, blockIdx.x, threadIdx.x);
}

}  // namespace nbpg
