// One insert of a batch as two kernels: a FLAG search per warp that leaves the expanded keys and the unseen
// neighbours' keys in global memory, and a block per insert that makes the candidate pool and prunes it
// (algorithms/nsw.h:122-175, prune.h:50-87, 159-209).  Same results as build_one (build_impl.cuh).
//
// Why the search needs no visited list: with no cut rule and the visited cap VL >= L the frontier always
// holds the L smallest keys seen.  A key that the capped list drops has VL smaller expanded ones, so it is
// not among the L smallest and is in no frontier; and a key that left the frontier lies past L others for
// good.  "In the visited list" and "expanded" then agree on every frontier entry, and the list itself is
// the VL smallest expanded keys, sorted once, by the second kernel.
//
// Why two kernels: the search is bound by the latency of its chain of expansions, in a slot whose visited
// filter (16 KB at L = 100) limits it to 12 warps per SM, so four more keep theirs in global memory; the prune
// is bound by its rounds, each a pivot against all candidates left, which four warps share, with the
// candidates' rows staged in shared memory.  RobustPrune takes one barrier per round: the survivors are a
// bitmask.
// A 2,000-insert batch of a 100k x 128 build (L = 100, VL = 140): 1.55 ms in one kernel, one warp per insert and
// LIST search; 0.38 + 0.14 ms here (the search took 0.47 with the 12 warps of the shared-memory filters alone).
#pragma once
#include "build_impl.cuh"
#include "search_flag.cuh"

namespace nbpg {

struct BuildFlagArgs {
    BuildArgs B;
    uint64_t *vis;   // [insert][FLAG_VIS] expanded keys, unsorted
    uint64_t *near;  // [insert][R] keys of the node's neighbours that the search did not see
    uint4 *info;     // [insert] expanded keys kept, neighbours, distances, expansions
    uint32_t own;    // warps of a CTA with the visited filter in shared memory; the others' is in global memory
    SlotLayout lay_g;  // and their slot
};

// Persistent warps over the batch's inserts.
template <int DT, int MET, int VPL, bool GH>
__device__ __forceinline__ void build_search_one(const BuildFlagArgs &F, uint32_t t, const SlotLayout &lay, uint8_t *slot,
                                                 uint32_t gslot, int lane)
{
    const BuildArgs &B = F.B;
    const SearchArgs &a = B.s;
    const uint32_t index = B.inserts[t];
    const uint8_t *prow = a.base + size_t(index) * a.row_stride;
    // beam search from the start points (beam_search with k = 0, cut = 0)
    const FlagState st = search_flag<DT, MET, VPL, true, false, GH>(a, prow, B.L, 0, ~uint64_t(0), B.sp + size_t(t) * B.nsp_per,
                                                             B.nsp_per, lay, slot, gslot, lane, index,
                                                             FlagVisited{F.vis + size_t(t) * FLAG_VIS, B.VL});
    // existing neighbours not seen by the search (nsw.h:150-161); has_been_seen inserts
    uint32_t *filt = reinterpret_cast<uint32_t *>(slot + lay.off_filt);
    const uint32_t *grow = a.graph + size_t(index) * a.gstride;
    const uint32_t deg = __ldg(grow);
    uint32_t nf = 0;
    for (uint32_t c = 0; c < deg; c += 32) {
        const bool act = c + lane < deg;
        const uint32_t nb = act ? __ldg(grow + 1 + c + lane) : kNoId;
        const bool seen = filter_probe<GH>(st.H, st.smask, nb, act);  // all lanes
        const bool keep = act && !seen;
        const unsigned km = __ballot_sync(kFull, keep);
        if (keep) filt[nf + __popc(km & lanemask_lt())] = nb;
        nf += __popc(km);
    }
    __syncwarp();
    flag_row_keys<DT, MET, VPL, false>(a, reinterpret_cast<const uint4 *>(slot + lay.off_q), filt, nf,
                                       F.near + size_t(t) * B.R, 0, lane);
    if (lane == 0) F.info[t] = make_uint4(st.nbuf, nf, st.cmps + nf, st.nvis);
    __syncwarp();
}

template <int DT, int MET, int VPL>
__global__ void __launch_bounds__(512) build_search_kernel(BuildFlagArgs F)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool own = uint32_t(warp) < F.own;
    const uint32_t out = uint32_t(warp) - F.own;  // index among the others
    uint8_t *slot = smem + (own ? size_t(warp) * F.B.s.lay.bytes : size_t(F.own) * F.B.s.lay.bytes + size_t(out) * F.lay_g.bytes);
    const uint32_t gslot = blockIdx.x * ((blockDim.x >> 5) - F.own) + out;
    while (true) {
        uint32_t w = 0;
        if (lane == 0) w = atomicAdd(F.B.queue, 1u);
        w = __shfl_sync(kFull, w, 0);
        if (w >= F.B.bs) break;
        if (own) build_search_one<DT, MET, VPL, false>(F, w, F.B.s.lay, slot, 0, lane);
        else build_search_one<DT, MET, VPL, true>(F, w, F.lay_g, slot, gslot, lane);
    }
}

struct PruneCtl {
    uint32_t aw[2][8];  // alive candidates (current, next)
    uint32_t pool, spare[3];
};

struct PruneLayout {
    uint32_t off_vis, off_pool, off_near;
    uint32_t off_rows;   // staged rows (over the pool), or 0: read from global memory
    uint32_t row_pitch;  // bytes between staged rows, odd in 16-byte words
    uint32_t bytes;
};

constexpr uint32_t PRUNE_THREADS = 128;

inline PruneLayout make_prune_layout(uint32_t VL, uint32_t R, uint32_t row_stride)
{
    auto up = [](uint32_t x) { return (x + 15) / 16 * 16; };
    PruneLayout l{};
    l.off_vis = up(sizeof(PruneCtl));
    l.off_pool = l.off_vis + (FLAG_VIS + 2) * 8;
    l.off_near = l.off_pool + (FLAG_VIS + 2) * 8;
    l.bytes = l.off_near + up(R * 8);
    // 16-byte reads of one word of neighbouring rows hit all banks when the pitch is odd in 16-byte words
    l.row_pitch = row_stride + (row_stride / 16 % 2 ? 0 : 16);
    if (VL * l.row_pitch <= 48 * 1024) {
        l.off_rows = l.off_pool;
        l.bytes = std::max(l.bytes, l.off_pool + up(VL * l.row_pitch));
    }
    return l;
}

// Sort the keys s[0, n), n <= 256, in place by counting (copies stay, in order).  s has room for one
// more key.  All threads; ends with a block barrier.
template <int TT>
__device__ __forceinline__ void team_sort(uint64_t *s, uint32_t n)
{
    constexpr int E = 256 / TT;  // keys per thread
    if (threadIdx.x == 0 && (n & 1)) s[n] = kKeyMax;
    __syncthreads();
    uint64_t key[E];
    uint32_t at[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = threadIdx.x + e * TT;
        key[e] = i < n ? s[i] : kKeyMax;
        at[e] = 0;
        if (e * TT < int(n))
            for (uint32_t j = 0; j < n; j += 2) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(s + j);
                at[e] += (w.x < key[e] || (w.x == key[e] && j < i)) + (w.y < key[e] || (w.y == key[e] && j + 1 < i));
            }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (threadIdx.x + e * TT < n) s[at[e]] = key[e];
    __syncthreads();
}

// alpha * d <= limit as the reference compares it in double: the product of two floats is exact
// there, and here as the rounded product and its error (FP64 issue is scarce on this part)
__device__ __forceinline__ bool scaled_le(float alpha, float d, float limit)
{
    const float p = __fmul_rn(alpha, d);
    const float e = __fmaf_rn(alpha, d, -p);
    return p < limit || (p == limit && e <= 0.0f);
}

// sort_candidates (prune.h:50-74) without a degree bias: p forced last, sorted into dst, repeats and p
// dropped.  pool has room for one more key.  Returns the count.
template <int TT>
__device__ __forceinline__ uint32_t team_sort_candidates(uint64_t *pool, uint32_t np, uint64_t *dst, uint32_t index)
{
    constexpr int E = 256 / TT;  // keys per thread
    const uint64_t pkey = (uint64_t(f2ord(3.402823466e38f)) << 32) | index;
    const uint32_t i0 = threadIdx.x;
    for (uint32_t i = i0; i < np; i += TT)
        if (key_id(pool[i]) == index) pool[i] = pkey;
    if (i0 == 0 && (np & 1)) pool[np] = kKeyMax;
    __syncthreads();
    uint32_t drops = 0;
    while (true) {
        uint64_t key[E];
        uint32_t at[E];
        bool drop[E];
        uint32_t n = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint32_t i = i0 + e * TT;
            key[e] = i < np ? pool[i] : kKeyMax;
            at[e] = 0;
            drop[e] = false;
            if (e * TT < int(np))
                for (uint32_t j = 0; j < np; j += 2) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(pool + j);
                    at[e] += (w.x < key[e]) + (w.y < key[e]);
                    drop[e] |= (w.x == key[e] && j < i) || (w.y == key[e] && j + 1 < i);
                }
            drop[e] = drop[e] && key[e] != kKeyMax;
            n += drop[e];
        }
        if (!__syncthreads_or(n != 0)) {
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (key[e] != kKeyMax) dst[at[e]] = key[e];
            break;
        }
        // repeats (a neighbour the lossy filter forgot is in the visited list too): take the later
        // copies out and count again
#pragma unroll
        for (int e = 0; e < E; ++e) {
            drops += __syncthreads_count(drop[e]);
            if (drop[e]) pool[i0 + e * TT] = kKeyMax;
        }
        __syncthreads();
    }
    __syncthreads();
    uint32_t cnt = np - drops;
    if (cnt > 0 && key_id(dst[cnt - 1]) == index) --cnt;
    return cnt;
}

template <int TT, int DT, int MET>
__global__ void __launch_bounds__(TT, 1024 / TT) build_prune_kernel(BuildFlagArgs F, PruneLayout lay)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const BuildArgs &B = F.B;
    const SearchArgs &a = B.s;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t t = blockIdx.x, index = B.inserts[t];
    const uint32_t VL = B.VL, R = B.R;
    PruneCtl *ctl = reinterpret_cast<PruneCtl *>(smem);
    uint64_t *vis = reinterpret_cast<uint64_t *>(smem + lay.off_vis);
    uint64_t *pool = reinterpret_cast<uint64_t *>(smem + lay.off_pool);
    uint64_t *tmp = reinterpret_cast<uint64_t *>(smem + lay.off_near);
    const uint4 info = F.info[t];
    const uint32_t nf = info.y;
    for (uint32_t i = tid; i < info.x; i += TT) vis[i] = F.vis[size_t(t) * FLAG_VIS + i];
    for (uint32_t i = tid; i < nf; i += TT) tmp[i] = F.near[size_t(t) * R + i];
    team_sort<TT>(vis, info.x);
    const uint32_t vs = min(info.x, VL);
    if (B.popular)
        for (uint32_t i = tid; i < vs; i += TT) atomicAdd(&B.popular[key_id(vis[i])], 1.0f);

    // merge_union of the (unsorted) neighbour list with the sorted visited list, cap VL
    // (utilities.h:128-165).  Sorting follows, so only which keys it takes matters: all of them where
    // they fit, else the sequential two-pointer walk decides.
    uint32_t np;
    if (nf + vs <= VL) {
        np = nf + vs;
        for (uint32_t i = tid; i < np; i += TT) pool[i] = i < nf ? tmp[i] : vis[i - nf];
    } else {
        if (tid == 0) {
            uint32_t i = 0, j = 0, k = 0;
            while (i < nf && j < vs && k < VL) {
                if (tmp[i] < vis[j]) pool[k++] = tmp[i++];
                else if (vis[j] < tmp[i]) pool[k++] = vis[j++];
                else { pool[k++] = tmp[i++]; ++j; }
            }
            while (i < nf && k < VL) pool[k++] = tmp[i++];
            while (j < vs && k < VL) pool[k++] = vis[j++];
            ctl->pool = k;
        }
        __syncthreads();
        np = ctl->pool;
    }
    __syncthreads();
    np = team_sort_candidates<TT>(pool, np, vis, index);
    uint64_t *cand = vis;  // sorted; the selected end in its front

    // RobustPrune (limitedSimilarityPrune, prune.h:159-209)
    const float alpha = B.alpha_node ? B.alpha_node[index] : B.alpha_all;
    const float cosa = B.cos_node ? B.cos_node[index] : B.cos_all;
    const bool by_alpha = double(alpha) > kPruneEps, by_cos = double(cosa) > kPruneEps;
    uint32_t sel = 0, rp = 0;
    if (!by_alpha && !by_cos) {
        sel = min(np, R);
    } else {
        uint8_t *rows = smem + lay.off_rows;
        const uint32_t vecs = a.vecs;
        if (lay.off_rows)
            for (uint32_t e = tid; e < np * vecs; e += TT) {
                const uint32_t i = e / vecs, c = e - i * vecs;
                *reinterpret_cast<uint4 *>(rows + size_t(i) * lay.row_pitch + c * 16) =
                    __ldg(reinterpret_cast<const uint4 *>(a.base + size_t(key_id(cand[i])) * a.row_stride) + c);
            }
        if (tid < 8) ctl->aw[0][tid] = np >= tid * 32 + 32 ? kFull : np > tid * 32 ? (1u << (np - tid * 32)) - 1u : 0u;
        __syncthreads();
        auto row_of = [&](uint32_t i) {
            return lay.off_rows ? reinterpret_cast<const uint4 *>(rows + size_t(i) * lay.row_pitch)
                                : reinterpret_cast<const uint4 *>(a.base + size_t(key_id(cand[i])) * a.row_stride);
        };
        uint32_t cur = 0, scan = 0;
        while (sel < R && scan < np) {
            // the next alive candidate is the pivot; the alive ones behind it are compared with it
            uint32_t pos = kNoId, behind = 0;
            for (uint32_t w = scan >> 5; w * 32 < np; ++w) {
                uint32_t u = ctl->aw[cur][w];
                if (w == scan >> 5) u &= ~((1u << (scan & 31)) - 1u);
                if (u && pos == kNoId) {
                    pos = w * 32 + __ffs(u) - 1;
                    u &= u - 1;
                }
                behind += __popc(u);
            }
            if (pos == kNoId) break;
            scan = pos + 1;
            const uint64_t pk = cand[pos];
            const float dps = key_dist(pk);
            const uint4 *prow = row_of(pos);
            rp += behind;
            // a warp takes every TT / 32-nd word of candidates from the pivot's on
            for (uint32_t w = warp; w * 32 < np; w += TT / 32) {
                const uint32_t alive = ctl->aw[cur][w];
                const uint32_t i = w * 32 + lane;
                bool gone = false;
                if (i > pos && ((alive >> lane) & 1)) {
                    const uint4 *crow = row_of(i);
                    uint32_t acc = 0, acc2 = 0;  // two chains
                    uint32_t c = 0;
                    for (; c + 1 < vecs; c += 2) {
                        acc = acc_vec<DT, MET>(crow[c], prow[c], acc);
                        acc2 = acc_vec<DT, MET>(crow[c + 1], prow[c + 1], acc2);
                    }
                    if (c < vecs) acc = acc_vec<DT, MET>(crow[c], prow[c], acc);
                    const float dsp = finish_dist<DT, MET>(acc + acc2), dpp = key_dist(cand[i]);
                    if (by_alpha && scaled_le(alpha, dsp, dpp)) gone = true;
                    else if (by_cos && cos_at_p(dps, dpp, dsp) > cosa) gone = true;
                }
                const unsigned g = __ballot_sync(kFull, gone);
                if (lane == 0) ctl->aw[cur ^ 1][w] = alive & ~g;
            }
            if (tid == 0) cand[sel] = pk;  // sel <= pos: what later rounds read lies behind
            ++sel;
            cur ^= 1;
            __syncthreads();
        }
        __syncthreads();
    }

    for (uint32_t j = tid; j < sel; j += TT) {
        B.res_ids[size_t(t) * R + j] = key_id(cand[j]);
        B.res_d[size_t(t) * R + j] = key_dist(cand[j]);
    }
    if (tid == 0) {
        B.res_cnt[t] = sel;
        if (B.stat_dist) B.stat_dist[index] += info.z + rp;
        if (B.stat_vis) B.stat_vis[index] += info.w;
    }
}

}  // namespace nbpg
