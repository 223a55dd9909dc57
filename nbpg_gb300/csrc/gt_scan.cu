// Brute-force kNN on tcgen05 tensor cores, in stages (compute_groundtruth,
// data_tools/ANNs/data_proc/CompGT.cpp:29-134; same outputs as gt.cu).
//
// The admission rule is sequential in the row id, but only rows below the survivor bound B can be
// admitted, and B never grows (gt_tc.cu has the argument, for CompGT's replace-max rule with its
// stale read and for the exact top k).  So the base is scanned in growing stages:
// [0, 1024), [1024, 4096), [4096, 16384), ... (longer for few neighbours)  The first stage writes all distances; every later
// one records, per query, the rows below the bound that the stage before left, about 3 k of them in
// random order however long the stage; after each stage one warp per query replays its records in
// id order and publishes the new bound.  Within a stage nothing waits on anything: the (query tile,
// base tile) steps are cut into one equal range per SM.  Queries for which rows stored in some order
// fill a list are scanned again in stages too short for that (gt_scan_device).
//
// Against a scan that replays as it goes this takes the flagged candidates from 94% of the 32 x 32
// chunks to about a third, and the sequential replay out of the scan altogether.
// 10k x 1M x 128 u8, k = 100: 9.6 -> 4.2 ms (scan 3.2, of which the MMAs alone 2.2, replay 0.8, conversion
// 0.1); 1k x 50k x 96 i8 inner product, k = 10: 1.01 -> 0.135 ms; 2k x 200k x 256 u8, k = 100, which ran on
// DP4A units with 63 CTAs: 16.8 -> 0.46 ms.
//
// Exactness: u8 codes are centred by 128 (L2 does not change; the inner product is corrected with
// the rows' code sums), so that all codes are below 2^8 in magnitude, exact in bf16, and a dot
// product of up to 640 of them (the shared memory takes 576) is an integer below 2^24, exact in the fp32 accumulator.  The chunk
// test runs in fp32, widened by `slack` where its values may pass 2^24; what it flags is decided on
// the int32 distance, converted to float as the reference does (point.h:35-135).
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "tc_util.cuh"

namespace nbpg {

constexpr uint32_t SC_ROWS = 128;        // base rows per tile (MMA N) and queries per MMA tile (M)
constexpr uint32_t SC_ATOM = 128 * 128;  // bytes of one 64-code column of 128 rows
constexpr uint32_t SC_SLOTS = 4;         // TMEM accumulators of 128 columns: all 512 columns of the SM
constexpr uint32_t SC_MAX_STAGES = 8;    // shared-memory ring of base chunks (1 or 2 columns of 64 codes each)
constexpr int SC_THREADS = 352;          // warps 0-7 epilogue (4 per query tile of 128), 8 TMA, 9 MMA, 10 base values
constexpr uint32_t SC_P0 = 8;            // base tiles of the first stage
constexpr uint32_t SC_FIRST = 384;       // records in the first block of a list (one list per query and range)
constexpr uint32_t SC_BLOCK = 512;       // records in each further block, from a pool that all lists share
constexpr uint32_t SC_MORE = 31;         // most further blocks of a list
constexpr uint32_t SC_LOST = ~0u;        // length of a list that found no block
constexpr uint32_t SC_BATCH = 64;        // query tiles per batch (up to 16,384 queries)
constexpr uint32_t SC_MAX_K = 128;
constexpr uint32_t SC_MAX_ELEMS = 640;

struct ScanArgs {
    const float *qval;  // per query of the batch: |q|^2, or the inner product's correction
    const float *bval;  // per base row: the same; 3e38 past the last row
    uint64_t n;
    uint32_t nq;         // queries of the batch
    uint32_t q_row0;     // first query row of the batch in the query tensor map
    int32_t c;           // distance = (qval + bval + c * dot) * scale: c = -2 (L2) or -1 (IP)
    int32_t scale;       // 1, or 256 for 4-bit codes
    float slack;         // widens the fp32 test where its values may pass 2^24
    uint32_t katoms, mt; // K / 64; query tiles of 128 per CTA (1 or 2)
    uint32_t kps;        // columns of 64 codes per ring stage
    uint32_t T, b_first; // base tiles of the stage, and the first one
    uint64_t W, total;   // steps per range, and in all
    uint32_t stages, withhold;
    const float *bound;  // per query: B
    uint2 *lists;        // [range + query tile][query of the tile, lrows of them][cap] (ordered distance, id)
    uint32_t *list_n;    // [range + query tile][query of the tile]
    uint32_t cap, lrows;
    uint2 *pool;         // [pool_blocks][SC_BLOCK] records past the first cap of a list
    uint32_t *more;      // [range + query tile][query of the tile][SC_MORE] their blocks
    uint32_t *pool_next;
    uint32_t pool_blocks;
    float *dense;        // first stage: [query][dense_stride] distances
    uint32_t dense_stride;
    uint32_t *err;
};

struct ReplayArgs {
    ScanArgs s;
    uint32_t k, first, last;
    const uint32_t *rows;  // output row of each query, or null: its own
    uint4 *st_d, *st_i;  // [query][32 lanes] distances (ordered) and ids of the running list
    uint2 *st_top;       // [query] CompGT's topdist and toppos
    float *bound;
    uint32_t *ovf;       // per query: a record list overflowed; null: that cannot be
    uint32_t *any_ovf;
    uint32_t *out_ids;
    float *out_dists;
};

__device__ __forceinline__ void tc_ld32_start(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
// waits for the loads in flight; v is named so that no use of it moves above the wait
__device__ __forceinline__ void tc_ld32_wait(uint32_t (&v)[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]),
                   "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]),
                   "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27])
                 :
                 : "memory");
    asm volatile("" : "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31]));
}

// One lane of a converged warp.  The producer and the MMA warp run their loops with all lanes and
// issue through this: 10k x 1M x 128, k = 100 took 4.90 ms with it and 5.80 with a test of the lane.
__device__ __forceinline__ bool elect_one()
{
    uint32_t one;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}

// mbar_wait with a warp-uniform result
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, uint32_t *err)
{
    return __all_sync(kFull, mbar_wait(bar, parity, err));
}

// The low words of two 128-byte-swizzle operand descriptors (sw128_desc) of a 64-code chunk; the four
// 16-code steps of the chunk lie 32 bytes apart, two units of the address field.  The issuing thread
// is one thread, and an MMA of this size takes 64 cycles: descriptors rebuilt from the address for
// every MMA kept it from issuing fast enough.
__device__ __forceinline__ uint32_t sw128_lo(uint32_t addr) { return (addr >> 4) | (1u << 16); }
constexpr uint32_t SW128_HI = (1024u >> 4) | (1u << 14) | (2u << 29);

__device__ __forceinline__ void mma_chunk(uint32_t d, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p, t;\n .reg .b64 a, b;\n .reg .b32 x, y;\n setp.ne.b32 p, %4, 0;\n setp.eq.b32 t, %4, %4;\n"
        " mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n"
        " add.u32 x, %1, 2;\n add.u32 y, %2, 2;\n mov.b64 a, {x, %5};\n mov.b64 b, {y, %5};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n"
        " add.u32 x, %1, 4;\n add.u32 y, %2, 4;\n mov.b64 a, {x, %5};\n mov.b64 b, {y, %5};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n"
        " add.u32 x, %1, 6;\n add.u32 y, %2, 6;\n mov.b64 a, {x, %5};\n mov.b64 b, {y, %5};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n}\n" ::"r"(d),
        "r"(alo), "r"(blo), "r"(idesc), "r"(acc), "r"(SW128_HI));
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// What a thread holds of its query during a range.
struct ScanRow {
    float thr, B, qv;  // flag below thr; record below B; the query's value
    uint64_t c2;       // (c, c)
    uint2 *lst;
    uint32_t ln, end;  // records so far, and how many the list has room for (lst[ln] is the next place)
    uint32_t list;
};

// v[j] for a j known only at run time, by a tree of selects (the chunk stays in registers)
__device__ __forceinline__ uint32_t pick32(const uint32_t (&v)[32], uint32_t j)
{
    uint32_t a[16], b[8], c[4], d[2];
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = (j & 16) ? v[i + 16] : v[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) b[i] = (j & 8) ? a[i + 8] : a[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = (j & 4) ? b[i + 4] : b[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) d[i] = (j & 2) ? c[i + 2] : c[i];
    return (j & 1) ? d[1] : d[0];
}

// A further block for a list that has no room for another base tile; the rest of the present one is filled with records
// that no rule admits.  Without a block the query's records are lost (it is scanned for again later on), and nothing more
// is recorded for it in this range.  Looked at once per tile, so that the record loop itself has no limit to check
// (checked there it cost 12%: 10k x 1M, k = 100 in 4.80 ms instead of 4.21).
__device__ __forceinline__ void scan_more(const ScanArgs &a, ScanRow &row)
{
    const uint32_t x = (row.end - a.cap) / SC_BLOCK;
    const uint32_t b = x < SC_MORE && a.pool_blocks ? atomicAdd(a.pool_next, 1u) : a.pool_blocks;
    if (b < a.pool_blocks) {
        for (; row.ln < row.end; ++row.ln) row.lst[row.ln] = make_uint2(~0u, ~0u);
        a.more[size_t(row.list) * SC_MORE + x] = b;
        row.lst = a.pool + size_t(b) * SC_BLOCK - row.end;
        row.end += SC_BLOCK;
    } else {
        row.thr = row.B = -__int_as_float(0x7f800000);
        row.ln = SC_LOST;
    }
}

// One thread's query row of an accumulator chunk: 32 dot products v, the base rows' values bn (in
// shared memory) and ids id0 ..; records the rows below the bound, in id order.
// What bounds the epilogue: instruction issue, 32 x 32 pairs per warp chunk.  16 two-wide FMAs, 16
// minima and 8 vector reads decide a chunk of which no row is flagged, which hides behind the MMAs.  A
// flagged row goes through a short loop with a select tree: 32 unrolled copies of the record code missed
// the instruction cache, and reading the column again from TMEM cost a round trip per column.
__device__ __forceinline__ void scan_chunk(const ScanArgs &a, const uint32_t (&v)[32], const float *bn, uint32_t id0,
                                           ScanRow &row)
{
    float t[32];
    float m[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(bn + g * 8 + h * 4);
            const uint64_t p[2] = {w.x, w.y};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int e = g * 8 + h * 4 + j * 2;
                uint64_t x, r;
                asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[e]), "r"(v[e + 1]));
                asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(row.c2), "l"(x), "l"(p[j]));
                asm("mov.b64 {%0, %1}, %2;" : "=f"(t[e]), "=f"(t[e + 1]) : "l"(r));
            }
        }
        const float *tg = t + g * 8;
        m[g] = fminf(min3(tg[0], tg[1], tg[2]), min3(tg[3], tg[4], min3(tg[5], tg[6], tg[7])));
    }
    if (!(fminf(min3(m[0], m[1], m[2]), m[3]) < row.thr)) return;
    uint32_t mask = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g)
        if (m[g] < row.thr) {
#pragma unroll
            for (int j = 0; j < 8; ++j) mask |= t[g * 8 + j] < row.thr ? 1u << (g * 8 + j) : 0u;
        }
    while (mask) {
        const uint32_t e = __ffs(mask) - 1;
        mask &= mask - 1;
        const int32_t dot = __float2int_rn(__uint_as_float(pick32(v, e)));
        const float df = __int2float_rn((__float2int_rn(row.qv) + __float2int_rn(bn[e]) + a.c * dot) * a.scale);
        if (df < row.B) row.lst[row.ln++] = make_uint2(f2ord(df), id0 + e);
    }
}

// The first stage: all distances of the chunk, written as floats.
__device__ __forceinline__ void dense_chunk(const ScanArgs &a, const uint32_t (&v)[32], const float *bn, float qv,
                                            float *out)
{
    const int32_t q = __float2int_rn(qv);
#pragma unroll
    for (int e = 0; e < 32; e += 4) {
        float d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            d[j] = __int2float_rn((q + __float2int_rn(bn[e + j]) + a.c * __float2int_rn(__uint_as_float(v[e + j]))) *
                                  a.scale);
        *reinterpret_cast<float4 *>(out + e) = make_float4(d[0], d[1], d[2], d[3]);
    }
}

// One CTA per SM works through its range of (query tile, base tile) steps.  A query tile is mt x 128
// queries: with two, each base chunk of 64 codes x 128 rows (16 KB) feeds two MMAs, which halves the
// L2 and shared-memory traffic per flop (one 128-query tile needs 64 B per clock per SM, all that
// L2 gives).  The query tile stays in shared memory; base chunks come through a ring by TMA; four
// TMEM accumulators hold two tiles in flight (four with mt = 1).
template <bool DENSE>
__global__ void __launch_bounds__(SC_THREADS, 1)
    gt_scan_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, ScanArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *sA = smem;                                              // [mt][katoms] atoms
    uint8_t *sB = sA + a.mt * a.katoms * SC_ATOM;                    // a.stages x kps atoms
    const uint32_t stage_bytes = a.kps * SC_ATOM;
    float *nring = reinterpret_cast<float *>(sB + a.stages * stage_bytes);  // [SC_SLOTS][128] base values
    uint64_t *bars = reinterpret_cast<uint64_t *>(nring + SC_SLOTS * SC_ROWS);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 32);

    const int tid = threadIdx.x, warp = __shfl_sync(kFull, tid >> 5, 0), lane = tid & 31;
    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + SC_MAX_STAGES),
                   bar_tfull = smem_u32(bars + 2 * SC_MAX_STAGES),
                   bar_tempty = smem_u32(bars + 2 * SC_MAX_STAGES + SC_SLOTS),
                   bar_nfull = smem_u32(bars + 2 * SC_MAX_STAGES + 2 * SC_SLOTS),
                   bar_a = smem_u32(bars + 2 * SC_MAX_STAGES + 3 * SC_SLOTS), bar_aempty = bar_a + 8,
                   bar_done = bar_a + 16;
    if (tid == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (uint32_t s = 0; s < SC_SLOTS; ++s) {
            mbar_init(bar_tfull + 8 * s, 1);
            mbar_init(bar_tempty + 8 * s, 128);
            mbar_init(bar_nfull + 8 * s, 1);
        }
        mbar_init(bar_a, 1);
        mbar_init(bar_aempty, 1);
        mbar_init(bar_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(kFull, *tmem_slot, 0);
    const uint64_t p0 = uint64_t(blockIdx.x) * a.W, p1 = min(p0 + a.W, a.total);
    const uint32_t mt = a.mt, qrows = mt * SC_ROWS, T = a.T;

    if (warp == 8) {
        uint32_t s = 0, ph = 0, issued = 0, aloads = 0;
        bool ok = true;
        for (uint64_t p = p0; ok && p < p1;) {
            const uint32_t li = uint32_t(p / T), b0 = uint32_t(p % T);
            const uint32_t b1 = uint32_t(min(uint64_t(T), b0 + (p1 - p)));
            if (aloads > 0 && !warp_wait(bar_aempty, (aloads - 1) & 1, a.err)) break;
            if (elect_one()) {
                mbar_expect_tx(bar_a, mt * a.katoms * SC_ATOM);
                for (uint32_t m = 0; m < mt; ++m)
                    for (uint32_t c = 0; c < a.katoms; ++c)
                        tma_load_2d(smem_u32(sA + (m * a.katoms + c) * SC_ATOM), &tmA, int32_t(c * TC_KATOM),
                                    int32_t(a.q_row0 + li * qrows + m * SC_ROWS), bar_a);
            }
            __syncwarp();
            ++aloads;
            for (uint32_t b = b0; ok && b < (a.withhold ? b0 : b1); ++b)
                for (uint32_t c = 0; c < a.katoms; c += a.kps) {
                    ok = warp_wait(bar_empty + 8 * s, ph ^ 1, a.err);
                    if (!ok) break;
                    if (elect_one()) {
                        const uint32_t dst = smem_u32(sB + s * stage_bytes), cols = min(a.kps, a.katoms - c);
                        mbar_expect_tx(bar_full + 8 * s, cols * SC_ATOM);
                        for (uint32_t i = 0; i < cols; ++i)
                            tma_load_2d(dst + i * SC_ATOM, &tmB, int32_t((c + i) * TC_KATOM),
                                        int32_t((a.b_first + b) * SC_ROWS), bar_full + 8 * s);
                    }
                    __syncwarp();
                    ++issued;
                    if (++s == a.stages) { s = 0; ph ^= 1; }
                }
            p += b1 - b0;
        }
        // every copy of this warp has landed before the CTA may exit
        if (aloads > 0) warp_wait(bar_a, (aloads - 1) & 1, a.err);
        for (uint32_t t = issued > a.stages ? issued - a.stages : 0; t < issued; ++t)
            warp_wait(bar_full + 8 * (t % a.stages), (t / a.stages) & 1, a.err);
    } else if (warp == 9) {
        const uint32_t idesc = tc_idesc(SC_ROWS, SC_ROWS), a_base = smem_u32(sA), b_base = smem_u32(sB);
        uint32_t s = 0, ph = 0, j = 0, seg = 0;  // j: accumulator uses so far; use j takes slot j % 4
        bool ok = true;
        for (uint64_t p = p0; ok && p < p1; ++seg) {
            const uint32_t b0 = uint32_t(p % T);
            const uint32_t b1 = uint32_t(min(uint64_t(T), b0 + (p1 - p)));
            ok = warp_wait(bar_a, seg & 1, a.err);
            for (uint32_t b = b0; ok && b < b1; ++b, j += mt) {
                const uint32_t s0 = j % SC_SLOTS, s1 = (j + mt - 1) % SC_SLOTS;
                ok = warp_wait(bar_tempty + 8 * s0, ((j / SC_SLOTS) & 1) ^ 1, a.err);
                if (ok && mt == 2) ok = warp_wait(bar_tempty + 8 * s1, (((j + 1) / SC_SLOTS) & 1) ^ 1, a.err);
                if (!ok) break;
                const uint32_t d0 = tmem + s0 * SC_ROWS, d1 = tmem + s1 * SC_ROWS;
                for (uint32_t c = 0; c < a.katoms; c += a.kps) {
                    ok = warp_wait(bar_full + 8 * s, ph, a.err);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        const uint32_t cols = min(a.kps, a.katoms - c);
                        for (uint32_t i = 0; i < cols; ++i) {
                            const uint32_t blo = sw128_lo(b_base + s * stage_bytes + i * SC_ATOM);
                            mma_chunk(d0, sw128_lo(a_base + (c + i) * SC_ATOM), blo, idesc, c + i);
                            if (mt == 2) mma_chunk(d1, sw128_lo(a_base + (a.katoms + c + i) * SC_ATOM), blo, idesc, c + i);
                        }
                        tc_commit(bar_empty + 8 * s);
                        if (c + a.kps >= a.katoms) {
                            tc_commit(bar_tfull + 8 * s0);
                            if (mt == 2) tc_commit(bar_tfull + 8 * s1);
                        }
                    }
                    __syncwarp();
                    if (++s == a.stages) { s = 0; ph ^= 1; }
                }
            }
            if (elect_one()) tc_commit(bar_aempty);  // this segment's MMAs are done with the query tile
            __syncwarp();
            p += b1 - b0;
        }
        // all issued MMAs complete before teardown
        if (elect_one()) tc_commit(bar_done);
        __syncwarp();
        warp_wait(bar_done, 0, a.err);
    } else if (warp == 10) {
        // each tile's base values, beside its first accumulator, once the epilogue has released the
        // tile that had the place before
        if (lane == 0) {
            uint32_t g = 0;
            bool ok = true;
            for (uint64_t p = p0; ok && p < p1;) {
                const uint32_t b0 = uint32_t(p % T);
                const uint32_t b1 = uint32_t(min(uint64_t(T), b0 + (p1 - p)));
                for (uint32_t b = b0; b < b1; ++b, ++g) {
                    const uint32_t j0 = g * mt, ns = j0 % SC_SLOTS;
                    for (uint32_t m = 0; m < mt; ++m)
                        ok = ok && mbar_wait(bar_tempty + 8 * ((j0 + m) % SC_SLOTS), (((j0 + m) / SC_SLOTS) & 1) ^ 1, a.err);
                    if (!ok) break;
                    mbar_expect_tx(bar_nfull + 8 * ns, SC_ROWS * 4);
                    bulk_load(smem_u32(nring + ns * SC_ROWS), a.bval + size_t(a.b_first + b) * SC_ROWS, SC_ROWS * 4,
                              bar_nfull + 8 * ns);
                }
                p += b1 - b0;
            }
            // the last copies have landed before the CTA may exit
            const uint32_t ring = SC_SLOTS / mt;
            for (uint32_t t = g > ring ? g - ring : 0; t < g; ++t)
                mbar_wait(bar_nfull + 8 * (t * mt % SC_SLOTS), (t * mt / SC_SLOTS) & 1, a.err);
        }
        __syncwarp();
    } else if (uint32_t(warp >> 2) < mt) {
        const uint32_t m = warp >> 2, row = m * SC_ROWS + (warp & 3) * 32 + lane;
        const uint32_t tlane = uint32_t((warp & 3) * 32) << 16;
        const float kInf = __int_as_float(0x7f800000);
        const float cf = float(a.c);
        uint64_t c2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(c2) : "f"(cf));
        bool done = true;  // every tile consumed (false after a timed-out wait)
        uint32_t g = 0;
        for (uint64_t p = p0; done && p < p1;) {
            const uint32_t li = uint32_t(p / T), b0 = uint32_t(p % T);
            const uint32_t b1 = uint32_t(min(uint64_t(T), b0 + (p1 - p)));
            const uint32_t q = li * qrows + row;
            const bool live = q < a.nq;
            const float qv = live ? a.qval[q] : 0.0f;
            const size_t sidx = (size_t(blockIdx.x) + li) * a.lrows + row;  // (of live queries: row < lrows)
            ScanRow sr{-kInf, -kInf, qv, c2, nullptr, 0u, a.cap, uint32_t(sidx)};
            if constexpr (!DENSE) {
                if (live) {
                    sr.lst = a.lists + sidx * a.cap;
                    sr.B = a.bound[q];
                    sr.thr = __fadd_ru(__fsub_ru(__fdiv_rn(sr.B, float(a.scale)), qv), a.slack);
                }
            }
            for (uint32_t b = b0; b < b1; ++b, ++g) {
                const uint32_t j = g * mt + m, slot = j % SC_SLOTS, ns = g * mt % SC_SLOTS;
                bool ok = __all_sync(kFull, mbar_wait(bar_tfull + 8 * slot, (j / SC_SLOTS) & 1, a.err));
                ok = ok && __all_sync(kFull, mbar_wait(bar_nfull + 8 * ns, (g * mt / SC_SLOTS) & 1, a.err));
                if (!ok) {
                    done = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if constexpr (!DENSE)
                    if (sr.end - sr.ln < SC_ROWS) scan_more(a, sr);
                const float *bn = nring + ns * SC_ROWS;
                const uint32_t ta = tmem + tlane + slot * SC_ROWS;
                const uint32_t id0 = (a.b_first + b) * SC_ROWS;
                uint32_t v0[32], v1[32];  // a chunk in use, the next one on its way
                tc_ld32_start(ta, v0);
#pragma unroll 1
                for (uint32_t c = 0; c < 4; c += 2) {
                    __syncwarp();
                    tc_ld32_wait(v0);
                    tc_ld32_start(ta + (c + 1) * 32, v1);
                    if constexpr (DENSE) {
                        if (live) dense_chunk(a, v0, bn + c * 32, qv, a.dense + size_t(q) * a.dense_stride + b * SC_ROWS + c * 32);
                    } else {
                        scan_chunk(a, v0, bn + c * 32, id0 + c * 32, sr);
                    }
                    __syncwarp();
                    tc_ld32_wait(v1);
                    if (c == 0) tc_ld32_start(ta + 64, v0);
                    if constexpr (DENSE) {
                        if (live)
                            dense_chunk(a, v1, bn + (c + 1) * 32, qv,
                                        a.dense + size_t(q) * a.dense_stride + b * SC_ROWS + (c + 1) * 32);
                    } else {
                        scan_chunk(a, v1, bn + (c + 1) * 32, id0 + (c + 1) * 32, sr);
                    }
                }
                __syncwarp();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(bar_tempty + 8 * slot);
                // (with two query tiles the base values are released by both tiles' accumulators)
            }
            if constexpr (!DENSE)
                if (live) a.list_n[sidx] = sr.ln;
            p += b1 - b0;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ---------------------------------------------------------------------------
// Replay: one warp per query.  The running list lives in registers, four entries per lane.
// ---------------------------------------------------------------------------

// CompGT's list (CompGT.cpp:71-95): slot s in lane s / 4, entry s % 4; distances as ordered u32
// (0 in slots past k, below every distance).
struct CgList {
    uint32_t d[4], id[4];
    uint32_t topd, toppos, lmax;
};

// largest distance of slots 1 .. k-1 and its first slot
__device__ __forceinline__ void cg_rest_max(const CgList &L, int lane, uint32_t &M, uint32_t &pos)
{
    const uint32_t d0 = lane ? L.d[0] : 0u;
    const uint32_t m = max(max(d0, L.d[1]), max(L.d[2], L.d[3]));
    M = __reduce_max_sync(kFull, m);
    const unsigned bal = __ballot_sync(kFull, m == M);
    const uint32_t r = (lane && L.d[0] == M) ? 0u : L.d[1] == M ? 1u : L.d[2] == M ? 2u : 3u;
    pos = __shfl_sync(kFull, uint32_t(lane) * 4 + r, __ffs(bal) - 1);
}

// overwrite toppos; the rescan over slots 1 .. k-1 starts from topk[0] read before the write
__device__ __forceinline__ void cg_admit(CgList &L, uint32_t dv, uint32_t iv, int lane)
{
    const uint32_t old0 = __shfl_sync(kFull, L.d[0], 0);
    // selects, not an indexed store: the list stays in registers
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const bool here = L.toppos == uint32_t(lane) * 4 + r;
        L.d[r] = here ? dv : L.d[r];
        L.id[r] = here ? iv : L.id[r];
    }
    uint32_t M, pos;
    cg_rest_max(L, lane, M, pos);
    L.lmax = max(L.toppos == 0 ? dv : old0, M);
    L.topd = M > old0 ? M : old0;
    L.toppos = M > old0 ? pos : 0u;
}

// 32 rows in id order, one per lane
__device__ __forceinline__ void cg_batch(CgList &L, uint32_t o, uint32_t id, bool valid, int lane)
{
    unsigned mask = __ballot_sync(kFull, valid && o < max(L.lmax, L.topd));
    while (mask) {
        const int src = __ffs(mask) - 1;
        mask &= mask - 1;
        const uint32_t dv = __shfl_sync(kFull, o, src), iv = __shfl_sync(kFull, id, src);
        if (dv < L.topd) cg_admit(L, dv, iv, lane);
    }
}

// The exact rule's list: the 128 smallest (distance, id) keys, sorted, entry i in lane i % 32,
// register i / 32; rows below the k-th key gather in buf (128 keys of shared memory) and are
// merged 128 at a time.
struct ExList {
    uint64_t v[4];
    uint64_t kth;
    uint32_t fill;
};

__device__ __forceinline__ void ex_kth(ExList &L, uint32_t k)
{
    const uint32_t r = (k - 1) >> 5;
    uint64_t x = L.v[0];
    if (r == 1) x = L.v[1];
    if (r == 2) x = L.v[2];
    if (r == 3) x = L.v[3];
    L.kth = __shfl_sync(kFull, x, (k - 1) & 31);
}

__device__ __forceinline__ void ex_flush(ExList &L, uint64_t *buf, uint32_t k, int lane)
{
    uint64_t w[4];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 4; ++r) w[r] = uint32_t(r * 32 + lane) < L.fill ? buf[r * 32 + lane] : kKeyMax;
    __syncwarp();
    warp_bitonic_sort<4>(w, lane);
    // the elementwise minimum against the reversed other half holds the 128 smallest, bitonic
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint64_t o = __shfl_sync(kFull, w[3 - r], 31 - lane);
        L.v[r] = o < L.v[r] ? o : L.v[r];
    }
#pragma unroll
    for (int j = 64; j >= 32; j >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int pr = r ^ (j >> 5);
            if (pr > r) {
                const uint64_t x = L.v[r], y = L.v[pr];
                L.v[r] = x < y ? x : y;
                L.v[pr] = x < y ? y : x;
            }
        }
#pragma unroll
    for (int j = 16; j > 0; j >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint64_t o = __shfl_xor_sync(kFull, L.v[r], j);
            const bool low = (lane & j) == 0;
            L.v[r] = low == (o < L.v[r]) ? o : L.v[r];
        }
    L.fill = 0;
    ex_kth(L, k);
}

__device__ __forceinline__ void ex_batch(ExList &L, uint64_t *buf, uint32_t k, uint32_t o, uint32_t id, bool valid,
                                         int lane)
{
    const uint64_t key = (uint64_t(o) << 32) | id;
    const bool keep = valid && key < L.kth;
    const unsigned m = __ballot_sync(kFull, keep);
    if (!m) return;
    if (keep) buf[L.fill + __popc(m & lanemask_lt())] = key;
    L.fill += __popc(m);
    if (L.fill > 96) ex_flush(L, buf, k, lane);
}

template <bool EXACT, int MET>
__global__ void __launch_bounds__(128) gt_replay_kernel(ReplayArgs a)
{
    __shared__ uint64_t bufs[4][128];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t q = blockIdx.x * 4 + warp, k = a.k;
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.s.pool_next = 0;  // for the next stage
    if (q >= a.s.nq) return;
    // read together; a query whose records were lost has recorded nothing more (its bound is below every distance)
    const uint32_t err = *a.s.err, gone = a.ovf ? a.ovf[q] : 0u;
    if (err | gone) return;
    uint64_t *buf = bufs[warp];
    CgList cg{};
    ExList ex{};
    if (a.first) {
        const float *row = a.s.dense + size_t(q) * a.s.dense_stride;
        const uint32_t cnt = uint32_t(min(uint64_t(a.s.T) * SC_ROWS, a.s.n));
        uint32_t start = 0;
        if constexpr (EXACT) {
            ex.kth = kKeyMax;
#pragma unroll
            for (int r = 0; r < 4; ++r) ex.v[r] = kKeyMax;
        } else {
            // fill phase: the first k ids; topdist by a strict > scan from slot 0
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint32_t s = lane * 4 + r;
                cg.d[r] = s < k ? f2ord(row[s]) : 0u;
                cg.id[r] = s;
            }
            uint32_t M, pos;
            cg_rest_max(cg, lane, M, pos);
            const uint32_t d0 = __shfl_sync(kFull, cg.d[0], 0);
            cg.topd = cg.lmax = max(d0, M);
            cg.toppos = M > d0 ? pos : 0u;
            start = k;
        }
        for (uint32_t b = start & ~31u; b < cnt; b += 32) {
            const uint32_t i = b + lane;
            const bool valid = i >= start && i < cnt;
            const uint32_t o = valid ? f2ord(row[i]) : 0u;
            if constexpr (EXACT) ex_batch(ex, buf, k, o, i, valid, lane);
            else cg_batch(cg, o, i, valid, lane);
        }
    } else {
        const uint4 d = a.st_d[size_t(q) * 32 + lane], id = a.st_i[size_t(q) * 32 + lane];
        if constexpr (EXACT) {
            ex.v[0] = (uint64_t(d.x) << 32) | id.x;
            ex.v[1] = (uint64_t(d.y) << 32) | id.y;
            ex.v[2] = (uint64_t(d.z) << 32) | id.z;
            ex.v[3] = (uint64_t(d.w) << 32) | id.w;
            ex_kth(ex, k);
        } else {
            cg.d[0] = d.x; cg.d[1] = d.y; cg.d[2] = d.z; cg.d[3] = d.w;
            cg.id[0] = id.x; cg.id[1] = id.y; cg.id[2] = id.z; cg.id[3] = id.w;
            const uint2 t = a.st_top[q];
            cg.topd = t.x;
            cg.toppos = t.y;
            uint32_t M, pos;
            cg_rest_max(cg, lane, M, pos);
            cg.lmax = max(__shfl_sync(kFull, cg.d[0], 0), M);
        }
        // the ranges that hold a part of this query tile's scan, in id order; 32 of their lists at
        // a time are read as one sequence (a query has a record or two per range when it is alone)
        const uint32_t qrows = a.s.mt * SC_ROWS, li = q / qrows, row = q % qrows;
        const uint64_t T = a.s.T;
        const uint32_t c0 = uint32_t(li * T / a.s.W), c1 = uint32_t(((li + 1) * T - 1) / a.s.W);
        for (uint32_t s0 = c0; s0 <= c1; s0 += 32) {
            const uint32_t c = s0 + lane;
            const uint32_t cnt = c <= c1 ? a.s.list_n[size_t(c + li) * a.s.lrows + row] : 0u;
            if (__any_sync(kFull, cnt == SC_LOST)) {  // the host scans for this query again
                if (lane == 0) {
                    atomicExch(a.ovf ? a.any_ovf : a.s.err, 1u);
                    if (a.ovf) a.ovf[q] = 1;
                    a.bound[q] = -__int_as_float(0x7f800000);
                }
                return;
            }
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += x;
            }
            const uint32_t all = __shfl_sync(kFull, incl, 31), excl = incl - cnt;
            for (uint32_t e0 = 0; e0 < all; e0 += 32) {
                const uint32_t e = e0 + lane;
                uint32_t j = 0;  // lists wholly before record e
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const uint32_t x = __shfl_sync(kFull, incl, int(j) + o - 1);
                    if (x <= e) j += o;
                }
                j = min(j, 31u);
                const uint32_t off = e - __shfl_sync(kFull, excl, int(j));
                uint2 rec = make_uint2(0u, 0u);
                if (e < all) {
                    const size_t list = size_t(s0 + j + li) * a.s.lrows + row;
                    const uint32_t x = off - a.s.cap;
                    rec = off < a.s.cap ? a.s.lists[list * a.s.cap + off]
                                        : a.s.pool[size_t(a.s.more[list * SC_MORE + x / SC_BLOCK]) * SC_BLOCK + x % SC_BLOCK];
                }
                if constexpr (EXACT) ex_batch(ex, buf, k, rec.x, rec.y, e < all, lane);
                else cg_batch(cg, rec.x, rec.y, e < all, lane);
            }
        }
    }
    if constexpr (EXACT)
        if (ex.fill) ex_flush(ex, buf, k, lane);
    if (a.last) {
        // output sorted by (dist, id) (CompGT.cpp:107-124)
        const size_t out = size_t(a.rows ? a.rows[q] : q) * k;
        uint64_t key[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if constexpr (EXACT) key[r] = ex.v[r];
            else key[r] = uint32_t(lane * 4 + r) < k ? (uint64_t(cg.d[r]) << 32) | cg.id[r] : kKeyMax;
        }
        if constexpr (!EXACT) warp_bitonic_sort<4>(key, lane);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t i = r * 32 + lane;
            if (i < k) {
                a.out_ids[out + i] = key_id(key[r]);
                a.out_dists[out + i] = output_dist<MET>(key_dist(key[r]));
            }
        }
        return;
    }
    if constexpr (EXACT) {
        a.st_d[size_t(q) * 32 + lane] = make_uint4(uint32_t(ex.v[0] >> 32), uint32_t(ex.v[1] >> 32),
                                                   uint32_t(ex.v[2] >> 32), uint32_t(ex.v[3] >> 32));
        a.st_i[size_t(q) * 32 + lane] = make_uint4(uint32_t(ex.v[0]), uint32_t(ex.v[1]), uint32_t(ex.v[2]), uint32_t(ex.v[3]));
        if (lane == 0) a.bound[q] = ord2f(uint32_t(ex.kth >> 32));
    } else {
        a.st_d[size_t(q) * 32 + lane] = make_uint4(cg.d[0], cg.d[1], cg.d[2], cg.d[3]);
        a.st_i[size_t(q) * 32 + lane] = make_uint4(cg.id[0], cg.id[1], cg.id[2], cg.id[3]);
        if (lane == 0) {
            a.st_top[q] = make_uint2(cg.topd, cg.toppos);
            a.bound[q] = ord2f(max(cg.lmax, cg.topd));
        }
    }
}

// Codes -> bf16 rows of K elements (zero past the row), u8 centred by 128, and the row's value:
// squared norm (L2); for u8 inner products the correction that undoes the centring, -128 * sum(b')
// of a base row and -(128 * sum(q') + 128^2 * dims) of a query.  8 codes per thread: one 8-byte (4-bit:
// 4-byte) load and one 16-byte store.  pick: the source row of each row, or null.
template <int DT>
__global__ void __launch_bounds__(256) gt_codes_kernel(const uint8_t *src, uint32_t row_bytes, uint32_t stride, uint64_t rows,
                                                       uint64_t rows_pad, uint32_t K, uint32_t lr_log, uint32_t ip,
                                                       uint32_t query, const uint32_t *pick, __nv_bfloat16 *dst, float *val)
{
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t lr = 1u << lr_log;  // lanes per row: 8, 16 or 32
    const uint64_t r = t >> lr_log;    // rows_pad x lr is a multiple of the block: every warp is full
    const uint32_t l = uint32_t(t) & (lr - 1);
    constexpr bool nib = DT == DT_U4;
    const uint32_t codes = nib ? row_bytes * 2 : row_bytes;
    const uint8_t *const row = src + (pick && r < rows ? pick[r] : r) * stride;
    int32_t sq = 0, sum = 0;
    for (uint32_t g = l; g < K / 8; g += lr) {
        uint32_t w[2] = {0, 0};
        const bool in = r < rows && g * 8 < codes;  // whole groups lie within the padded row
        if (in) {
            if constexpr (nib) {
                w[0] = *reinterpret_cast<const uint32_t *>(row + g * 4);
            } else {
                const uint2 x = *reinterpret_cast<const uint2 *>(row + g * 8);
                w[0] = x.x;
                w[1] = x.y;
            }
        }
        uint32_t packed[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            int32_t v = 0;
            if constexpr (nib) {
                const uint32_t b = (w[0] >> (8 * (j / 2))) & 0xFFu;
                v = int32_t((j & 1) ? (b & 0x0Fu) : (b >> 4));  // nibble values; distances scaled by 256
            } else {
                const uint32_t b = (w[j / 4] >> (8 * (j % 4))) & 0xFFu;
                v = DT == DT_U8 ? int32_t(b) - 128 : int32_t(int8_t(b));
            }
            if (!in || g * 8 + j >= codes) v = 0;
            sq += v * v;
            sum += v;
            packed[j / 2] |= uint32_t(__bfloat16_as_ushort(__int2bfloat16_rn(v))) << (16 * (j & 1));
        }
        if (r < rows_pad) *reinterpret_cast<uint4 *>(dst + r * K + g * 8) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
    int32_t x = ip ? (DT == DT_U8 ? -128 * sum : 0) : sq;
    for (uint32_t o = lr / 2; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    if (ip && DT == DT_U8 && query) x -= 16384 * int32_t(row_bytes);
    if (l == 0 && r < rows_pad) val[r] = r < rows ? __int2float_rn(x) : 3e38f;
}

// Ring stages of two columns of 64 codes halve the barrier round trips per flop; one where the row has one.
static uint32_t scan_kps(uint32_t katoms) { return katoms >= 2 ? 2 : 1; }

static size_t scan_smem(uint32_t katoms, uint32_t mt, uint32_t stages)
{
    // at least 120 KB, so that one CTA holds an SM and its TMEM allocation never waits for another's
    const size_t need = 1024 + size_t(SC_ATOM) * (mt * katoms + stages * scan_kps(katoms)) + SC_SLOTS * SC_ROWS * 4 + 32 * 8 + 16;
    return std::max<size_t>(need, 120 * 1024);
}

static uint32_t scan_elems(uint32_t dtype, uint32_t dims)
{
    return (dtype == NBPG_U4 || dtype == NBPG_I4) ? 2 * dims : dims;
}

// Two query tiles per CTA while their codes fit in shared memory beside the ring (up to 256 codes).
static uint32_t scan_mt(uint32_t katoms) { return katoms <= 4 ? 2 : 1; }

static uint32_t scan_ring(uint32_t katoms, size_t smem_optin)
{
    for (uint32_t st = SC_MAX_STAGES; st >= 2; --st)
        if (scan_smem(katoms, scan_mt(katoms), st) <= smem_optin) return st;
    return 0;
}

// Whether the staged tensor scan applies: rows of up to 576 codes (query tile and ring in shared
// memory; dot products are exact up to 640), k up to 128 (the replay's registers).
bool gt_scan_supported(uint32_t dtype, uint32_t dims, uint32_t k, size_t smem_optin)
{
    if (dtype > NBPG_I4 || dims == 0 || dims > SC_MAX_ELEMS || k == 0 || k > SC_MAX_K) return false;
    const uint32_t elems = scan_elems(dtype, dims);
    return elems <= SC_MAX_ELEMS && scan_ring((elems + TC_KATOM - 1) / TC_KATOM, smem_optin) != 0;
}

// First tile of each stage and the total, in base tiles.  A stage that would leave less than half of
// itself for the next takes the rest as well.
// Growth: a stage g times as long as all before it records about k (g - 1) rows per query, and each
// stage costs two launches (25 us), so few neighbours take longer stages: 50k rows at k = 10 with
// growth 4 / 16 run in 149 / 146 us; 1M rows at k = 100 with growth 2 / 3 / 4 in 4.05 / 4.17 / 4.20 ms,
// 200k long rows in 504 / 460 / 457 us.
static std::vector<uint32_t> scan_stages(uint32_t T, uint32_t k)
{
    const uint32_t grow = k <= 16 ? 16 : k <= 48 ? 8 : 4;
    std::vector<uint32_t> at{0};
    uint32_t e = std::min(T, SC_P0);
    while (true) {
        at.push_back(e);
        if (e == T) return at;
        const uint64_t next = uint64_t(e) * grow;
        e = next * 3 >= uint64_t(T) * 2 ? T : uint32_t(next);
    }
}

struct ScanSplit {
    uint64_t total, W;
    uint32_t ctas, cap;
};

// One equal range of steps per SM; the first block of a list holds `most` records, or all rows of a range.
static ScanSplit scan_split(uint32_t qtiles, uint32_t T, uint32_t sms, uint32_t most)
{
    ScanSplit s;
    s.total = uint64_t(qtiles) * T;
    s.W = (s.total + sms - 1) / sms;
    s.ctas = uint32_t((s.total + s.W - 1) / s.W);
    s.cap = uint32_t(std::min<uint64_t>(most, std::min<uint64_t>(s.W, T) * SC_ROWS));
    return s;
}

size_t gt_tc_list_bytes(uint64_t n, uint32_t nq, uint32_t k, uint32_t sms);

struct ScanLayout {
    uint32_t K, katoms, mt, qrows, batch;  // batch: query tiles per pass
    uint32_t lrows;                        // queries of a tile that lists are kept for
    uint64_t n_pad, nq_pad;
    std::vector<uint32_t> at;
    size_t first, pool;  // records in the first blocks of all lists, and in the pool behind them
    size_t off_q, off_bval, off_qval, off_flags, off_again, off_bound, off_d, off_i, off_top, off_dense, off_listn, off_more,
        off_lists, bytes;
};

static ScanLayout scan_layout(uint32_t dtype, uint32_t dims, uint64_t n, uint32_t nq, uint32_t k, uint32_t sms)
{
    ScanLayout l;
    l.K = (scan_elems(dtype, dims) + TC_KATOM - 1) / TC_KATOM * TC_KATOM;
    l.katoms = l.K / TC_KATOM;
    l.mt = scan_mt(l.katoms);
    l.qrows = l.mt * SC_ROWS;
    l.n_pad = (n + SC_ROWS - 1) / SC_ROWS * SC_ROWS;
    l.nq_pad = (uint64_t(nq) + l.qrows - 1) / l.qrows * l.qrows;
    l.at = scan_stages(uint32_t(l.n_pad / SC_ROWS), k);
    l.batch = uint32_t(std::min<uint64_t>(SC_BATCH, l.nq_pad / l.qrows));
    l.lrows = uint32_t(std::min<uint64_t>(nq, l.qrows));
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t qb = std::min<size_t>(nq, size_t(l.batch) * l.qrows);
    l.first = l.pool = 0;
    const uint64_t qtiles = l.nq_pad / l.qrows;
    const size_t lists = l.at.size() > 2 ? size_t(sms + l.batch) * l.lrows : 0;
    uint64_t rows = 0;  // of the longest stage
    for (size_t i = 1; i + 1 < l.at.size(); ++i) {
        rows = std::max(rows, uint64_t(l.at[i + 1] - l.at[i]) * SC_ROWS);
        for (uint64_t qt : {uint64_t(l.batch), qtiles % l.batch})  // a full batch and the last one
            if (qt) {
                const ScanSplit s = scan_split(uint32_t(qt), l.at[i + 1] - l.at[i], sms, SC_FIRST);
                l.first = std::max(l.first, size_t(s.ctas + qt) * l.lrows * s.cap);
            }
    }
    // A stage records about 3 k rows of a query (15 k where k is small) over all its ranges, two at least, so most
    // lists end in their first block; the pool is for rows in an order.  It gets what is left of the memory that the
    // replaying engine takes for its lists (up to 0.32, 0.64 or 1.27 GB for k up to 25, 51 and above, on 152 SMs), or
    // 384 records per query where that is nothing, and never more than all rows of a stage.
    const size_t room = gt_tc_list_bytes(n, nq, k, sms) / 8;
    const size_t other = l.first + qb * (l.at[1] * SC_ROWS * 4 + 1036) / 8 + lists * (1 + SC_MORE) / 2;
    l.pool = std::min<size_t>(qb * rows, std::max(qb * 384, room > other ? room - other : 0));
    l.pool = (l.pool + SC_BLOCK - 1) / SC_BLOCK * SC_BLOCK;
    l.off_q = up(l.n_pad * l.K * 2);
    l.off_bval = l.off_q + up(l.nq_pad * l.K * 2);
    l.off_qval = l.off_bval + up(l.n_pad * 4);
    l.off_flags = l.off_qval + up(l.nq_pad * 4);
    l.off_again = l.off_flags + up((4 + size_t(nq)) * 4);
    l.off_bound = l.off_again + up(size_t(nq) * 4);
    l.off_d = l.off_bound + up(qb * 4);
    l.off_i = l.off_d + up(qb * 512);
    l.off_top = l.off_i + up(qb * 512);
    l.off_dense = l.off_top + up(qb * 8);
    l.off_listn = l.off_dense + up(qb * l.at[1] * SC_ROWS * 4);
    l.off_more = l.off_listn + up(lists * 4);
    l.off_lists = l.off_more + up(lists * SC_MORE * 4);
    l.bytes = l.off_lists + up((l.first + l.pool) * 8);
    return l;
}

static uint32_t scan_sms()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return 1;
    return uint32_t(sms);
}

// sms 0: the current device's
size_t gt_scan_workspace(uint32_t dtype, uint32_t dims, uint64_t n, uint32_t nq, uint32_t k, uint32_t sms)
{
    return scan_layout(dtype, dims, n, nq, k, sms ? sms : scan_sms()).bytes;
}

template <int DT>
static void launch_codes(const uint8_t *src, uint32_t dims, uint32_t stride, uint64_t rows, uint64_t rows_pad, uint32_t K,
                         uint32_t ip, uint32_t query, const uint32_t *pick, __nv_bfloat16 *dst, float *val, cudaStream_t st)
{
    const uint32_t lr_log = K == 64 ? 3 : K == 128 ? 4 : 5;
    gt_codes_kernel<DT><<<uint32_t((rows_pad << lr_log) / 256), 256, 0, st>>>(src, dims, stride, rows, rows_pad, K, lr_log, ip, query, pick,
                                                                      dst, val);
}

// Stages in which no first block can overflow, for `tiles` query tiles with lists for `lrows` queries of each: the
// blocks of all ranges (one per SM at most) have room for every row of a range.
static std::vector<uint32_t> scan_short_stages(const ScanLayout &l, uint32_t tiles, uint32_t lrows, uint32_t sms)
{
    const uint32_t T = l.at.back();
    uint32_t len = T - l.at[1];
    while (len > 1) {
        const ScanSplit s = scan_split(tiles, len, sms, ~0u);
        if (size_t(std::min<uint64_t>(sms, s.total) + tiles) * lrows * s.cap <= l.first + l.pool) break;
        len = len * 7 / 8;
    }
    std::vector<uint32_t> at{0};
    for (uint32_t b = l.at[1]; b < T; b += std::min(len, T - b)) at.push_back(b);
    at.push_back(T);
    return at;
}

template <bool EXACT>
static void launch_replay(uint32_t metric, const ReplayArgs &r, cudaStream_t st)
{
    const uint32_t grid = (r.s.nq + 3) / 4;
    if (metric == NBPG_L2) gt_replay_kernel<EXACT, M_L2><<<grid, 128, 0, st>>>(r);
    else gt_replay_kernel<EXACT, M_IP><<<grid, 128, 0, st>>>(r);
}

// Device-resident inputs (rows of dims bytes, stride bytes apart); outputs device arrays nq * k.
// ws: gt_scan_workspace() bytes, or NULL to allocate them here.  Returns after the work has finished
// on `st`.
//
// Rows in an order (a base stored by cluster, label or time) can come closer and closer to a query, more of them in
// one range than there are blocks for.  Such queries record nothing in the stages that follow; at the end they are put
// beside each other and scanned again, in stages so short that the first block of a list holds every row of a range.
// *redone receives how many queries that were.  most_blocks: no more further blocks than that (for tests).
// 10k x 1M x 128 u8 rows stored by label, k = 100 / 10: 16.5 / 19.7 ms (1,000 labels), 54 / 27 ms (64 labels, where
// most queries fill the pool); in random order 4.2 / 3.0.  With lists of 4,096 and the replaying engine for every
// query of the call behind them: 17.6 / 45 and 122 / 83.
nbpg_status gt_scan_device(uint32_t dtype, uint32_t metric, uint32_t dims, uint32_t stride, const uint8_t *d_base,
                           uint64_t n, const uint8_t *d_q, uint32_t nq, uint32_t k, uint32_t mode, uint32_t *d_ids,
                           float *d_dists, void *ws, cudaStream_t st, uint32_t *redone, uint32_t most_blocks, bool withhold)
{
    const uint32_t sms = scan_sms();
    const ScanLayout l = scan_layout(dtype, dims, n, nq, k, sms);
    if (redone) *redone = 0;
    auto fail = [](cudaError_t e) {
        set_error(std::string("nbpg_gt (tensor path): ") + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? NBPG_ERR_OOM : NBPG_ERR_CUDA;
    };
    void *owned = nullptr;
    cudaError_t e = cudaSuccess;
    if (!ws) {
        e = cudaMalloc(&owned, l.bytes);
        if (e != cudaSuccess) {
            cudaGetLastError();  // an allocation that did not fit is not a fault of later launches
            return fail(e);
        }
        ws = owned;
    }
    uint8_t *w = static_cast<uint8_t *>(ws);
    __nv_bfloat16 *bB = reinterpret_cast<__nv_bfloat16 *>(w), *bQ = reinterpret_cast<__nv_bfloat16 *>(w + l.off_q);
    float *bval = reinterpret_cast<float *>(w + l.off_bval), *qval = reinterpret_cast<float *>(w + l.off_qval);
    uint32_t *flags = reinterpret_cast<uint32_t *>(w + l.off_flags);  // [0] error, [1] any overflow, [2] pool_next; from [4] per query
    nbpg_status s = NBPG_OK;
    e = cudaMemsetAsync(flags, 0, (4 + size_t(nq)) * 4, st);
    const uint32_t ip = metric == NBPG_IP;
    auto codes = [&](const uint8_t *src, uint64_t rows, uint64_t pad, uint32_t query, const uint32_t *pick, __nv_bfloat16 *dst,
                     float *val) {
        if (dtype == NBPG_U8) launch_codes<DT_U8>(src, dims, stride, rows, pad, l.K, ip, query, pick, dst, val, st);
        else if (dtype == NBPG_I8) launch_codes<DT_I8>(src, dims, stride, rows, pad, l.K, ip, query, pick, dst, val, st);
        else launch_codes<DT_U4>(src, dims, stride, rows, pad, l.K, ip, query, pick, dst, val, st);
    };
    if (e == cudaSuccess) {
        codes(d_base, n, l.n_pad, 0, nullptr, bB, bval);
        codes(d_q, nq, l.nq_pad, 1, nullptr, bQ, qval);
        e = cudaGetLastError();
    }
    CUtensorMap mA, mB;
    if (e == cudaSuccess && (!make_map(&mA, bQ, l.nq_pad, l.K) || !make_map(&mB, bB, l.n_pad, l.K))) {
        set_error("nbpg_gt: tensor map encoding failed");
        s = NBPG_ERR_CUDA;
    }
    int dev = 0, optin = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const uint32_t ring = scan_ring(l.katoms, size_t(optin));
    if (e == cudaSuccess && s == NBPG_OK && ring == 0) {
        set_error("nbpg_gt: the tensor engine's shared memory does not fit this row length");
        s = NBPG_ERR_UNSUPPORTED;
    }
    const size_t smem = scan_smem(l.katoms, l.mt, ring ? ring : 2);
    if (e == cudaSuccess && s == NBPG_OK)
        e = raise_smem_limit(gt_scan_kernel<true>, smem);
    if (e == cudaSuccess && s == NBPG_OK)
        e = raise_smem_limit(gt_scan_kernel<false>, smem);

    ReplayArgs r{};
    r.s.bval = bval;
    r.s.n = n;
    r.s.c = ip ? -1 : -2;
    r.s.scale = (dtype == NBPG_U4 || dtype == NBPG_I4) ? 256 : 1;
    // up to 128 codes every value of the test is an integer below 2^24; past that (8-bit codes) it is
    // below 2^26, so rounding moves it by at most 2, the bound's own rounding by at most 2 more
    r.s.slack = r.s.scale == 1 && l.K > 128 ? 8.0f : 0.0f;
    r.s.katoms = l.katoms;
    r.s.mt = l.mt;
    r.s.kps = scan_kps(l.katoms);
    r.s.stages = ring;
    r.s.withhold = withhold ? 1u : 0u;
    r.s.bound = r.bound = reinterpret_cast<float *>(w + l.off_bound);
    r.s.lists = reinterpret_cast<uint2 *>(w + l.off_lists);
    r.s.list_n = reinterpret_cast<uint32_t *>(w + l.off_listn);
    r.s.dense = reinterpret_cast<float *>(w + l.off_dense);
    r.s.dense_stride = l.at[1] * SC_ROWS;
    r.s.more = reinterpret_cast<uint32_t *>(w + l.off_more);
    r.s.pool = r.s.lists + l.first;
    r.s.pool_next = flags + 2;
    r.s.err = flags;
    r.k = k;
    r.st_d = reinterpret_cast<uint4 *>(w + l.off_d);
    r.st_i = reinterpret_cast<uint4 *>(w + l.off_i);
    r.st_top = reinterpret_cast<uint2 *>(w + l.off_top);
    r.any_ovf = flags + 1;
    // all stages for the first `count` converted queries; outputs in the rows `rows`, or as they come
    auto pass = [&](uint32_t count, const uint32_t *rows) {
        const uint64_t per_batch = uint64_t(l.batch) * l.qrows;
        for (uint64_t q0 = 0; e == cudaSuccess && q0 < count; q0 += per_batch) {
            r.s.nq = uint32_t(std::min<uint64_t>(per_batch, count - q0));
            r.s.qval = qval + q0;
            r.s.q_row0 = uint32_t(q0);
            r.rows = rows ? rows + q0 : nullptr;
            r.ovf = rows ? nullptr : flags + 4 + q0;
            r.out_ids = d_ids + (rows ? 0 : q0 * k);
            r.out_dists = d_dists + (rows ? 0 : q0 * k);
            const uint32_t qtiles = (r.s.nq + l.qrows - 1) / l.qrows;
            r.s.lrows = std::min(count, l.qrows);
            r.s.pool_blocks = rows ? 0u : uint32_t(std::min<size_t>(l.pool / SC_BLOCK, most_blocks));
            const std::vector<uint32_t> at = rows ? scan_short_stages(l, qtiles, r.s.lrows, sms) : l.at;
            for (size_t i = 0; i + 1 < at.size(); ++i) {
                r.s.b_first = at[i];
                r.s.T = at[i + 1] - at[i];
                const ScanSplit sp = scan_split(qtiles, r.s.T, sms, rows ? ~0u : SC_FIRST);
                r.s.W = sp.W;
                r.s.total = sp.total;
                r.s.cap = sp.cap;
                r.first = i == 0;
                r.last = i + 2 == at.size();
                if (r.first) gt_scan_kernel<true><<<sp.ctas, SC_THREADS, smem, st>>>(mA, mB, r.s);
                else gt_scan_kernel<false><<<sp.ctas, SC_THREADS, smem, st>>>(mA, mB, r.s);
                if (mode == NBPG_GT_EXACT) launch_replay<true>(metric, r, st);
                else launch_replay<false>(metric, r, st);
            }
            e = cudaGetLastError();
        }
    };
    uint32_t h[2] = {0, 0};
    auto finish = [&](void *to, const void *from, size_t bytes) {
        if (e == cudaSuccess && s == NBPG_OK) e = cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToHost, st);
        const cudaError_t es = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = es;
    };
    if (s == NBPG_OK) pass(nq, nullptr);
    finish(h, flags, 8);
    if (e == cudaSuccess && s == NBPG_OK && !h[0] && h[1]) {
        std::vector<uint32_t> ovf(nq), rows;
        finish(ovf.data(), flags + 4, size_t(nq) * 4);
        for (uint32_t q = 0; q < nq; ++q)
            if (ovf[q]) rows.push_back(q);
        if (redone) *redone = uint32_t(rows.size());
        uint32_t *d_rows = reinterpret_cast<uint32_t *>(w + l.off_again);
        const uint32_t m = uint32_t(rows.size());
        if (e == cudaSuccess) e = cudaMemcpyAsync(d_rows, rows.data(), size_t(m) * 4, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            codes(d_q, m, (uint64_t(m) + l.qrows - 1) / l.qrows * l.qrows, 1, d_rows, bQ, qval);
            pass(m, d_rows);
        }
        finish(h, flags, 8);
    }
    if (owned) cudaFree(owned);
    if (e != cudaSuccess && s == NBPG_OK) s = fail(e);
    if (s == NBPG_OK && h[0]) {
        set_error("nbpg_gt (tensor path): a pipeline wait timed out");
        s = NBPG_ERR_TIMEOUT;
    }
    return s;
}

}  // namespace nbpg

// Test hook for the failure path: the tensor kNN on a small problem with its base tiles
// withheld, so the MMA and epilogue waits run out (nothing ever arrives on those barriers);
// the kernel must record the timeout, tear down (final commit, TMEM freed) and return, and
// the context must stay usable.  Returns NBPG_ERR_TIMEOUT on that path.
extern "C" nbpg_status nbpg_test_gt_timeout(int32_t device)
{
    using namespace nbpg;
    NBPG_CUDA_TRY(cudaSetDevice(device));
    const uint32_t n = 512, nq = 128, dims = 64, k = 10;
    uint8_t *db = nullptr, *dq = nullptr;
    uint32_t *di = nullptr;
    float *dd = nullptr;
    cudaError_t e = cudaMalloc(&db, n * dims);
    if (e == cudaSuccess) e = cudaMalloc(&dq, nq * dims);
    if (e == cudaSuccess) e = cudaMalloc(&di, nq * k * 4);
    if (e == cudaSuccess) e = cudaMalloc(&dd, nq * k * 4);
    if (e == cudaSuccess) e = cudaMemset(db, 7, n * dims);
    if (e == cudaSuccess) e = cudaMemset(dq, 3, nq * dims);
    nbpg_status s = NBPG_ERR_CUDA;
    if (e == cudaSuccess)
        s = gt_scan_device(NBPG_U8, NBPG_L2, dims, dims, db, n, dq, nq, k, NBPG_GT_COMPGT, di, dd, nullptr, nullptr,
                           nullptr, ~0u, true);
    cudaFree(db);
    cudaFree(dq);
    cudaFree(di);
    cudaFree(dd);
    if (e != cudaSuccess) {
        set_error(std::string("nbpg_test_gt_timeout: ") + cudaGetErrorString(e));
        return NBPG_ERR_CUDA;
    }
    return s;
}
