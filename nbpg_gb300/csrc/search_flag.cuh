// Strict greedy beam search with expanded flags instead of a visited list: FLAG mode
// (search_impl.cuh has the argument why it equals the reference's list), one warp per query.
//
// Runs the searches of beams above 32 and of inner product.  For L2 up to there the frontier is one entry per
// lane and search_core's merge is as short (10k queries at L = 19 on 1M x 128: 594 us there, 627 here; 556
// there since its filter probe is an exchange as well and its cut threshold is computed only where it matters).
//
// What bounds it: instructions.  Neither memory nor any pipe is near its limit; a warp spends 5 to 13
// cycles on each dependent instruction, so what counts is how many an expansion takes.
//   - The unexpanded entries are a bitmask over frontier positions, word w in lane w's register: finding
//     the next node is a ballot and a shuffle, and nothing is recomputed after a merge.
//   - The merge takes up to 32 candidates at a time, one per lane: a binary search gives a candidate its
//     place among the frontier entries, a count over the candidates its place among them.  The frontier
//     is updated in place, 32 positions at a time from the top down to the first one taken: a position
//     that no candidate takes gets the entry that the bit counts of the taken ones name, and the same pass
//     writes the new mask word.  No sort, no search per frontier entry, no second frontier.
//   - Inner product (DROP): the cut rule keeps next to nothing there, so expanded entries do leave the
//     frontier and can come back when the filter forgets them.  Their ids are kept, and a candidate found
//     among them enters as expanded: exactly "frontier minus visited".  More than fit, or a visited cap that
//     overflows, marks the query for LIST mode.
//   - The visited filter is probed with an exchange whose read-back shows whether two lanes met in a slot;
//     only then those lanes are sorted out (a __match_any_sync takes longer than the whole probe).
// 10k queries at L = 80 on 250k 4-bit rows: 1,196 -> 875 us; 2k re-ranked queries at L = 50: 775 -> 693 us;
// 20k inner-product queries of L = 32 .. 256 on 250k x 96 i8 (the visited lists, 16 KB a slot, are gone: 24 warps
// per SM instead of 10): 2,292 -> 1,056 us.
#pragma once
#include "search_impl.cuh"

namespace nbpg {

// What a launch of the strict kernels runs
enum SearchPass : int { PASS_FLAG = 0, PASS_LIST = 1, PASS_WIDE = 2 };

struct FlagState {
    const uint64_t *fr;  // the frontier, fs entries
    uint32_t *H;
    uint32_t fs, cmps, smask, adj, nbuf, nvis;
    bool taint;
};

// Where a build search keeps its expanded keys: room for FLAG_VIS keys in global memory, of which the
// `keep` smallest stay when it is full.
constexpr uint32_t FLAG_VIS = 256;
constexpr uint32_t FLAG_DROPS = 512;   // expanded entries that left the frontier (DROP)
constexpr uint32_t FLAG_BLOOM = 4096;  // bits that say which ids are surely not among them
__device__ __forceinline__ uint32_t drop_bit(uint32_t id) { return (id * 0x9E3779B1u) >> 20; }
struct FlagVisited {
    uint64_t *keys;
    uint32_t keep;
};

// Sort vis[0, FLAG_VIS) ascending (rare: a search that expands more nodes than fit)
static __device__ __noinline__ void flag_vis_sort(uint64_t *vis, int lane)
{
    uint64_t v[8];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = vis[r * 32 + lane];
    warp_bitonic_sort<8>(v, lane);
#pragma unroll
    for (int r = 0; r < 8; ++r) vis[r * 32 + lane] = v[r];
    __syncwarp();
}

// The query row as the distance passes read it: 16-byte words in shared memory.  Registers are what limits
// the resident warps (72 of them hold 28 per SM), and the words come back while the rows are on their way.
template <int DT, int MET, int VPL, bool FILTER>
__device__ __forceinline__ uint32_t flag_row_keys(const SearchArgs &a, const uint4 *q, const uint32_t *ids, uint32_t cnt,
                                                  uint64_t *out, uint64_t thr, int lane)
{
    const uint32_t lpr = a.lpr, rows_per = 32u / lpr;
    const uint32_t grp = uint32_t(lane) / lpr, lq = uint32_t(lane) % lpr;
    constexpr int P = VPL == 4 ? 2 : 4;  // 16 (lane width 1) or 32 rows in flight per pass group
    uint32_t stored = 0;
    for (uint32_t r0 = 0; r0 < cnt; r0 += rows_per * P) {
        uint4 bv[P][VPL];
        uint32_t id[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const uint32_t r = r0 + p * rows_per + grp;
            id[p] = r < cnt ? ids[r] : kNoId;
            const uint4 *row = reinterpret_cast<const uint4 *>(a.base + size_t(id[p]) * a.row_stride);
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                const uint32_t c = lq + v * lpr;
                bv[p][v] = (r < cnt && c < a.vecs) ? __ldg(row + c) : make_uint4(0, 0, 0, 0);
            }
        }
        uint4 qw[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            const uint32_t c = lq + v * lpr;
            qw[v] = c < a.vecs ? q[c] : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            if (r0 + p * rows_per >= cnt) break;  // warp-uniform: no rows left in this pass
            uint32_t acc = 0;
#pragma unroll
            for (int v = 0; v < VPL; ++v) acc = acc_vec<DT, MET>(bv[p][v], qw[v], acc);
            for (uint32_t o = lpr >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
            const uint32_t r = r0 + p * rows_per + grp;
            const uint64_t key = make_dist_key<MET>(finish_dist<DT, MET>(acc), id[p]);
            if constexpr (FILTER) {
                const bool keep = lq == 0 && r < cnt && key < thr;
                const unsigned m = __ballot_sync(kFull, keep);
                if (keep) out[stored + __popc(m & lanemask_lt())] = key;
                stored += __popc(m);
            } else {
                if (lq == 0 && r < cnt) out[r] = key;
            }
        }
    }
    __syncwarp();
    return FILTER ? stored : cnt;
}

// Entries of sorted s[0, n) that are < key, without branches (n <= 1024)
__device__ __forceinline__ uint32_t count_less(const uint64_t *s, uint32_t n, uint64_t key)
{
    uint32_t p = 0;
    for (uint32_t step = n ? 1u << (31 - __clz(n)) : 0; step > 0; step >>= 1) {
        const uint32_t t = p + step;
        if (t <= n && s[t - 1] < key) p = t;
    }
    return p;
}

// Shortens the frontier from fs to `to` entries; the ids of expanded ones among the rest go to drops, as many
// as fit (nd counts them all).
__device__ __forceinline__ void flag_drop(const uint64_t *fr, uint32_t &um, uint32_t to, uint32_t &fs, uint32_t *drops,
                                          uint32_t &nd, int lane)
{
    for (uint32_t b = to & ~31u; b < fs; b += 32) {
        const uint32_t i = b + lane, word = __shfl_sync(kFull, um, int(b >> 5));
        const bool d = i >= to && i < fs && !((word >> lane) & 1);
        const unsigned m = __ballot_sync(kFull, d);
        const uint32_t at = nd + __popc(m & lanemask_lt());
        if (d) {
            const uint32_t id = key_id(fr[i]), h = drop_bit(id);
            if (at < FLAG_DROPS) drops[at] = id;
            atomicOr(&drops[FLAG_DROPS + (h >> 5)], 1u << (h & 31));
        }
        nd += __popc(m);
    }
    const uint32_t b = uint32_t(lane) * 32;
    if (to < b + 32) um &= to > b ? (1u << (to - b)) - 1u : 0u;
    fs = to;
    __syncwarp();
}

// VIS: keep the expanded keys (v).  DROP: expanded entries may leave the frontier (see above).  GH: the visited filter is a global block, not shared memory (a template
// argument, so that shared-memory probes are not generic accesses).  k = 0: no cut rule.
template <int DT, int MET, int VPL, bool VIS, bool DROP, bool GH>
__device__ FlagState search_flag(const SearchArgs &a, const uint8_t *qrow_bytes, uint32_t L, uint32_t k,
                                 uint64_t max_visited, const uint32_t *sp, uint32_t nsp, const SlotLayout &lay,
                                 uint8_t *slot, uint32_t gslot, int lane, uint32_t self, FlagVisited v)
{
    const uint32_t S = filter_slots_for(L), smask = S - 1;
    uint64_t *const fr = reinterpret_cast<uint64_t *>(slot + lay.off_fr0);
    uint64_t *const cand = reinterpret_cast<uint64_t *>(slot + lay.off_cand);
    uint32_t *const filt = reinterpret_cast<uint32_t *>(slot + lay.off_filt);
    uint32_t *const H =
        GH ? a.g_hash + size_t(gslot) * a.g_hash_slots : reinterpret_cast<uint32_t *>(slot + lay.off_hash);

    uint4 *const q = reinterpret_cast<uint4 *>(slot + lay.off_q);
    for (uint32_t c = lane; c < a.vecs; c += 32) q[c] = reinterpret_cast<const uint4 *>(qrow_bytes)[c];
    // clear the visited filter (query_params.h:173-180)
    for (uint32_t i = lane; i < S / 4; i += 32) reinterpret_cast<uint4 *>(H)[i] = make_uint4(kNoId, kNoId, kNoId, kNoId);
    __syncwarp();
    // init_starting_points (query_params.h:204-221)
    flag_row_keys<DT, MET, VPL, false>(a, q, sp, nsp, fr, 0, lane);
    if (lane == 0)
        for (uint32_t s = 0; s < nsp; ++s) {
            const uint32_t id = sp[s];
            H[filter_slot(id, smask)] = id;
        }
    __syncwarp();
    sort_keys(fr, nsp, lane);

    uint32_t *const drops = reinterpret_cast<uint32_t *>(slot + lay.off_vis);
    uint32_t nd = 0;
    bool taint = false;
    if constexpr (DROP) {
        for (uint32_t i = lane; i < FLAG_BLOOM / 32; i += 32) drops[FLAG_DROPS + i] = 0;
        // repeated start points make a multiset of the frontier: LIST mode
        for (uint32_t i = lane; i + 1 < nsp; i += 32) taint |= fr[i] == fr[i + 1];
        taint = __any_sync(kFull, taint);
    }

    // lane w: unexpanded entries among positions [32 w, 32 w + 32)
    uint32_t um = nsp >= uint32_t(lane) * 32 + 32 ? kFull : nsp > uint32_t(lane) * 32 ? (1u << (nsp - lane * 32)) - 1u : 0u;
    uint32_t fs = nsp, cmps = nsp, adj = 0, cs = 0, cst = 0, nbuf = 0;
    uint32_t nvis = 0;  // no node is expanded twice, so these fit
    const uint32_t limit = uint32_t(min(a.limit, uint64_t(kNoId))), most = uint32_t(min(max_visited, uint64_t(kNoId)));
    const uint32_t nchunks = (a.R + 31) / 32;
    const float cut_low = __double2float_rd(a.cut);
    // candidates stored (cst) vs appended (cs, which drives the deferral rule): while the frontier is
    // full, a candidate at or beyond its last key can never survive the union's truncation to L, so it
    // is counted but not stored
    uint64_t tail = fs == L ? fr[L - 1] : kKeyMax;
    while (nvis < limit && !(DROP && taint)) {
        const unsigned open = __ballot_sync(kFull, um != 0);
        if (!open) break;
        const int ow = __ffs(open) - 1;
        const uint32_t oword = __shfl_sync(kFull, um, ow);
        const uint32_t pos = ow * 32 + __ffs(oword) - 1;
        const bool more = (open & (open - 1)) || (oword & (oword - 1));
        if (lane == ow) um &= um - 1;
        const uint64_t ck = fr[pos];
        const uint32_t *grow = a.graph + size_t(key_id(ck)) * a.gstride;

        // adjacency row: degree + up to 4 chunks of 32 ids, loads issued together
        uint32_t nbv[4];
        const uint32_t deg = __ldg(grow);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t e = 1 + c * 32 + lane;
            nbv[c] = (c < int(nchunks) && e < a.gstride) ? __ldg(grow + e) : kNoId;
        }
        // speculative: adjacency rows of the next unexpanded entries of this word
        if (a.prefetch && lane < int(a.prefetch) * 3 && uint32_t(lane % 3) * 32 < a.gstride) {
            uint32_t rest = oword & (oword - 1);
            for (int i = lane / 3; i > 0; --i) rest &= rest - 1;
            if (rest)
                prefetch_l2(a.graph + size_t(key_id(fr[ow * 32 + __ffs(rest) - 1])) * a.gstride + (lane % 3) * 32);
        }
        const uint32_t ne = deg < a.degree_limit ? deg : a.degree_limit;
        adj += 1 + ne;
        // visited filter, in neighbour order (beamSearch.h:71-83)
        uint32_t nf = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (uint32_t(c) * 32 >= ne) break;
            const bool act = uint32_t(c * 32 + lane) < ne;
            const bool seen = filter_probe<GH>(H, smask, nbv[c], act);
            const bool keep = act && !seen && nbv[c] != self;
            const unsigned km = __ballot_sync(kFull, keep);
            if (keep) filt[nf + __popc(km & lanemask_lt())] = nbv[c];
            nf += __popc(km);
        }
        __syncwarp();
        // distances of the new neighbours -> candidates (beamSearch.h:85-93)
        cst += flag_row_keys<DT, MET, VPL, true>(a, q, filt, nf, cand + cst, tail, lane);
        cs += nf;
        cmps += nf;
        ++nvis;
        if constexpr (VIS) {
            if (lane == 0) v.keys[nbuf] = ck;
            if (++nbuf == FLAG_VIS) {
                // keep the smallest: what the reference's sorted list, capped at v.keep, holds
                flag_vis_sort(v.keys, lane);
                nbuf = v.keep;
            }
        }
        if (nvis > most) taint = true;

        // deferred merge (beamSearch.h:119-125)
        if (cs == 0 || (limit >= 2u * L && cs < L / 8 && more)) continue;
        cs = 0;
        // Every candidate of this round lies at or past the full frontier's last key: the union truncated
        // to L is the frontier itself, and the cut rule keeps at least the old size (no taint either).
        if (cst == 0) continue;

        // set_union with the frontier, truncated to L (beamSearch.h:128-138), up to 32 candidates at a time
        // (the union of the unions is the same)
        const uint32_t fs0 = fs;
        for (uint32_t c0 = 0; c0 < cst; c0 += 32) {
            uint64_t *const cc = cand + c0;
            const uint32_t cnt = min(cst - c0, 32u);
            const bool in = uint32_t(lane) < cnt;
            const uint64_t c = in ? cc[lane] : kKeyMax;
            const uint32_t p = count_less(fr, fs, c);
            // which candidates lie below this one, and whether an earlier one is the same (equal ids are equal
            // keys).  One that the frontier holds (set_union keeps the frontier's copy, :132-135) or that is
            // stored twice (std::unique, :128-130; the filter is lossy) is struck.
            uint32_t less = 0, same = 0;
            for (uint32_t j = 0; j < cnt; j += 4) {
                const ulonglong2 w0 = *reinterpret_cast<const ulonglong2 *>(cc + j);
                const ulonglong2 w1 = *reinterpret_cast<const ulonglong2 *>(cc + j + 2);
                uint32_t l = 0, e = 0;
                if (w0.x < c) l |= 1;
                if (w0.y < c) l |= 2;
                if (w1.x < c) l |= 4;
                if (w1.y < c) l |= 8;
                if (key_id(w0.x) == key_id(c)) e |= 1;
                if (key_id(w0.y) == key_id(c)) e |= 2;
                if (key_id(w1.x) == key_id(c)) e |= 4;
                if (key_id(w1.y) == key_id(c)) e |= 8;
                less |= l << j;
                same |= e << j;
            }
            const bool keep = in && !(p < fs && fr[p] == c) && !(same & lanemask_lt());
            const unsigned km = __ballot_sync(kFull, keep);
            const uint32_t at = keep ? p + __popc(less & km) : kNoId;
            // (DROP takes the whole union, up to 32 entries past L, and drops the rest below)
            const uint32_t n0 = DROP ? fs + uint32_t(__popc(km)) : min(fs + uint32_t(__popc(km)), L);
            unsigned back = 0;  // candidates that were expanded before
            if constexpr (DROP) {
                const uint32_t h = drop_bit(key_id(c));
                bool met = keep && ((drops[FLAG_DROPS + (h >> 5)] >> (h & 31)) & 1);
                if (__any_sync(kFull, met)) {
                    const uint32_t kept = min(nd, FLAG_DROPS);
                    bool there = false;
                    for (uint32_t j = 0; j < kept; ++j) there |= drops[j] == key_id(c);
                    met = met && there;
                }
                back = __ballot_sync(kFull, met);
            }
            for (int w = int((n0 - 1) >> 5); w >= 0; --w) {
                const bool mine = (at >> 5) == uint32_t(w);
                const uint32_t taken = __reduce_or_sync(kFull, mine ? 1u << (at & 31) : 0u);
                const uint32_t below = __popc(__ballot_sync(kFull, at < uint32_t(w) * 32));
                if (!(taken | below)) break;  // nothing changes from here down
                const uint32_t x = uint32_t(w) * 32 + lane;
                const bool fresh = (taken >> lane) & 1;
                const uint32_t i = x - below - __popc(taken & lanemask_lt());
                const uint32_t ui = __shfl_sync(kFull, um, int((i >> 5) & 31));
                const bool old = !fresh && x < n0;
                const uint64_t key = old ? fr[i] : 0;
                __syncwarp();
                if (old) fr[x] = key;
                if (mine && at < n0) fr[at] = c;
                unsigned bits = __ballot_sync(kFull, x < n0 && (fresh || ((ui >> (i & 31)) & 1)));
                if (DROP && back) bits &= ~__reduce_or_sync(kFull, mine && ((back >> lane) & 1) ? 1u << (at & 31) : 0u);
                __syncwarp();
                if (lane == w) um = bits;
            }
            fs = n0;
            if constexpr (DROP)
                if (fs > L) flag_drop(fr, um, L, fs, drops, nd, lane);
        }
        cst = 0;
        // cut rule (beamSearch.h:140-149): threshold = float(cut * d_k), upper_bound of (0, thr)
        if (k > 0 && fs > k) {
            uint32_t nfs = fs;
            const float dk = key_dist(fr[k]), dlast = key_dist(fr[fs - 1]);
            // nothing to cut when the last distance lies below a product rounded down at both steps (squared
            // distances are not negative): the double product is needed only near the threshold
            if (!(MET == M_L2 && dlast < __fmul_rd(cut_low, dk))) {
                // on one lane: FP64 issue is scarce on this part
                float thr = 0.f;
                if (lane == 0) thr = __double2float_rn(a.cut * double(dk));
                thr = __shfl_sync(kFull, thr, 0);
                uint32_t ub = 0;
                for (uint32_t base = 0; base < fs; base += 32) {
                    const uint32_t i = base + lane;
                    bool pr = false;
                    if (i < fs) {
                        const uint64_t key = fr[i];
                        const float d = key_dist(key);
                        pr = d < thr || (d == thr && key_id(key) == 0);
                    }
                    ub += __popc(__ballot_sync(kFull, pr));
                }
                nfs = ub > fs0 ? ub : fs0;
                if constexpr (DROP) {
                    if (nfs < fs) flag_drop(fr, um, nfs, fs, drops, nd, lane);
                } else if (nfs < fs) {
                    const uint32_t b = uint32_t(lane) * 32;
                    if (nfs < b + 32) um &= nfs > b ? (1u << (nfs - b)) - 1u : 0u;
                    fs = nfs;
                }
            }
            if (!DROP && nfs < k + 1) taint = true;
        }
        if (DROP && nd > FLAG_DROPS) taint = true;  // some are lost
        tail = fs == L ? fr[L - 1] : kKeyMax;
    }
    FlagState st;
    st.fr = fr;
    st.H = H;
    st.fs = fs;
    st.cmps = cmps;
    st.smask = smask;
    st.adj = adj;
    st.nbuf = nbuf;
    st.nvis = nvis;
    st.taint = taint;
    return st;
}

}  // namespace nbpg
