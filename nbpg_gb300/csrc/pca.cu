// PCA projection + quantisation (PCACompress, data_tools/ANNs/data_proc/PCACompress.cpp:21-83
// over data_tools/ANNs/data_proc/base/matrix.h:25-125) and the FmtConv conversions
// (data_tools/ANNs/data_proc/FmtConv.cpp:63-131) on the GPU.
//
// values[j] = bias[j] - mips_distance(mat[j], x): the dot product is summed in index order
// in fp32 with separately rounded products, which is the reference's expression as
// written (point.h:148-156); each thread keeps that order for its outputs, so the codes
// are bit-identical to a build of the reference without fast-math reassociation.  The
// work (2 x n x d_in x d_out, 16 GFLOP for 1M x 128 -> 64) is small next to the file
// I/O around it; tensor-core MMA would change the summation order and move codes that
// sit on a quantisation boundary.
//
// Quantisation (matrix.h:99-125): code = int((v + 1) * 0.5 * 255), float add then double
// products, truncated (the reference's out-of-range conversion is undefined; here it
// saturates), clamped to [0, 255], minus 128 for the signed kinds, shifted right by
// 8 - 8/chunk, masked; for 4-bit output the high nibble of byte i is element 2i+1 and the
// low nibble element 2i.
#include <algorithm>
#include <cstring>
#include <string>

#include "internal.h"

namespace nbpg {

constexpr uint32_t PCA_MAX_DIN = 576;
constexpr int PCA_THREADS = 256;  // 8 (outputs) x 32 (points)
constexpr int PCA_KC = 32;        // input elements staged per round

enum PcaIn : int { PIN_F32 = 0, PIN_U8 = 1, PIN_I8 = 2 };

template <int IN>
__device__ __forceinline__ float load_in(const void *x, uint64_t i)
{
    if constexpr (IN == PIN_F32) return static_cast<const float *>(x)[i];
    else if constexpr (IN == PIN_U8) return float(static_cast<const uint8_t *>(x)[i]);
    else return float(static_cast<const int8_t *>(x)[i]);
}

// int((v + 1) * 0.5 * 255) as matrix.h:112 evaluates it (float add, double products, truncation),
// clamped to [0, 255], without the scarce FP64 units.  s = v + 1 has 24 significant bits, so the
// double product is the exact s * 127.5; p = s * 127.5 rounded to float and its exact error e from
// an FMA hold the same value, and p's truncation is off only where p was rounded up onto an integer.
__device__ __forceinline__ int quant_code(float v)
{
    const float s = __fadd_rn(v, 1.0f);
    const float p = __fmul_rn(s, 127.5f);
    const float e = __fmaf_rn(s, 127.5f, -p);
    int t = __float2int_rz(p);  // saturates; NaN gives 0
    if (float(t) == p && e < 0.0f) --t;
    return min(max(t, 0), 255);
}

__device__ __forceinline__ uint64_t pair2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
// acc + a * b on two values at once, the product rounded before the sum.  The sum is written as
// product * one + acc, with `one` = (1, 1) from a kernel argument: the same rounding as an add, and
// nothing an optimiser may contract with the product (mul.f32x2 followed by add.f32x2 came out as
// one FMA, which rounds once and moved codes).
__device__ __forceinline__ void mul_add2(uint64_t &acc, uint64_t a, uint64_t b, uint64_t one)
{
    uint64_t t;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(a), "l"(b));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(t), "l"(one));
}

// Column of output `o` (0 .. OPT - 1) of a thread with output lane tx: four neighbours in the first
// 32 columns, the rest beside each other from column 32 on, so that a warp's 8 output lanes read
// neighbouring vectors of shared memory and a 4-bit pair stays within one thread.
template <int OPT>
__device__ __forceinline__ uint32_t pca_col(uint32_t tx, int o)
{
    return o < 4 ? tx * 4 + o : 32 + tx * (OPT - 4) + (o - 4);
}

// What a column of staged matrix row i is XORed with: the transposing stores of a warp (32 rows of one column) go to 8
// banks instead of one, and a thread's vector stays one vector (1,000 rows of 576 codes -> 128: 65 -> 53 us; 1M x 128 ->
// 64: 673 -> 620).  48 columns are 16 banks apart from row to row, and gain less from it than the address costs (200k x
// 128 -> 34: 123 us without, 131 with).
template <int OPT>
__device__ __forceinline__ uint32_t pca_swizzle(uint32_t i)
{
    return OPT == 6 ? 0 : 4 * (i & 7);
}

// One CTA: 32 * PPT points x 8 * OPT outputs; a thread owns PPT points x OPT outputs in registers
// and walks the input elements in index order, so every output keeps the reference's summation order.
// What bounds it: one multiply and one add per input element and output (two instructions, no FMA):
// 16.4 G lane operations for 1M x 128 -> 64, 0.42 ms on 152 SMs x 128 lanes at 2 GHz, against 0.08 ms
// of HBM traffic; it measures 0.62 ms (1.70 ms with one output x 8 points per thread, a whole d_in of
// both operands in shared memory and double-precision quantisation).  Hence a register tile (16 shared-memory values feed 64 multiply-adds) and
// two-wide mul / add, which leave issue slots for the loads.  xs[i][p] is stored with its point
// index XORed by 4 * ((i / 4) % 8): the transposing stores and the 16-byte reads are both free of
// bank conflicts.
// out_kind: 0 f32, 1 u8, 2 i8, 3 u4, 4 i4; vec: rows of x are 16-byte (f32) or 4-byte (codes) aligned
// and d_in is a multiple of 4; wide: d_out is a multiple of 4 and out 16-byte aligned, so four outputs
// of a thread are one store.
template <int IN, int PPT, int OPT>
__global__ void __launch_bounds__(PCA_THREADS, 2) pca_kernel(const void *x, uint64_t n, uint32_t d_in, const float *mat,
                                                            const float *bias, uint32_t d_out, uint32_t out_kind,
                                                            uint32_t vec, uint32_t wide, float one, void *out)
{
    constexpr int P = 32 * PPT, O = 8 * OPT;
    __shared__ __align__(16) float xs[PCA_KC * P];
    __shared__ __align__(16) float ms[PCA_KC * O];
    const uint32_t tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const uint32_t j0 = blockIdx.y * O;
    const uint64_t p0 = uint64_t(blockIdx.x) * P;
    const uint64_t one2 = pair2(one, one);
    uint64_t acc[PPT][OPT / 2];
#pragma unroll
    for (int q = 0; q < PPT; ++q)
#pragma unroll
        for (int o = 0; o < OPT / 2; ++o) acc[q][o] = 0;

    for (uint32_t i0 = 0; i0 < d_in; i0 += PCA_KC) {
        const uint32_t kc = min(uint32_t(PCA_KC), d_in - i0);
        if (i0) __syncthreads();
        if (vec) {
            // 8 threads per row, 4 elements each
            float4 v[PPT];
            const uint32_t i = i0 + tx * 4;
#pragma unroll
            for (int r = 0; r < PPT; ++r) {
                const uint64_t p = p0 + r * 32 + ty;
                v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p < n && i < d_in) {
                    if constexpr (IN == PIN_F32) {
                        v[r] = __ldcs(reinterpret_cast<const float4 *>(static_cast<const float *>(x) + p * d_in + i));
                    } else if constexpr (IN == PIN_U8) {
                        const uchar4 c = *reinterpret_cast<const uchar4 *>(static_cast<const uint8_t *>(x) + p * d_in + i);
                        v[r] = make_float4(c.x, c.y, c.z, c.w);
                    } else {
                        const char4 c = *reinterpret_cast<const char4 *>(static_cast<const int8_t *>(x) + p * d_in + i);
                        v[r] = make_float4(float(int8_t(c.x)), float(int8_t(c.y)), float(int8_t(c.z)), float(int8_t(c.w)));
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < PPT; ++r) {
                float *d = xs + tx * 4 * P + ((r * 32 + ty) ^ (4 * tx));
                d[0] = v[r].x;
                d[P] = v[r].y;
                d[2 * P] = v[r].z;
                d[3 * P] = v[r].w;
            }
        } else {
            for (uint32_t e = tid; e < P * PCA_KC; e += PCA_THREADS) {
                const uint32_t pl = e / PCA_KC, i = e % PCA_KC;
                const uint64_t p = p0 + pl;
                xs[i * P + (pl ^ (4 * ((i >> 2) & 7)))] = p < n && i < kc ? load_in<IN>(x, p * d_in + i0 + i) : 0.0f;
            }
        }
        for (uint32_t e = tid; e < O * PCA_KC; e += PCA_THREADS) {
            const uint32_t i = e % PCA_KC, j = e / PCA_KC;
            ms[i * O + (j ^ pca_swizzle<OPT>(i))] = i < kc && j0 + j < d_out ? __ldg(mat + size_t(j0 + j) * d_in + i0 + i) : 0.0f;
        }
        __syncthreads();
        for (uint32_t i = 0; i < kc; ++i) {
            float xv[PPT];
            const float *xr = xs + i * P;
            const uint32_t sw = 4 * ((i >> 2) & 7);
            if constexpr (PPT >= 4) {
#pragma unroll
                for (int q = 0; q < PPT; q += 4) {
                    const float4 t = *reinterpret_cast<const float4 *>(xr + ((ty * PPT + q) ^ sw));
                    xv[q] = t.x;
                    xv[q + 1] = t.y;
                    xv[q + 2] = t.z;
                    xv[q + 3] = t.w;
                }
            } else {
                const float2 t = *reinterpret_cast<const float2 *>(xr + ((ty * PPT) ^ sw));
                xv[0] = t.x;
                xv[1] = t.y;
            }
            uint64_t mv[OPT / 2];
            const float *mr = ms + i * O;
            {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(mr + ((tx * 4) ^ pca_swizzle<OPT>(i)));
                mv[0] = t.x;
                mv[1] = t.y;
            }
            if constexpr (OPT == 6) mv[2] = *reinterpret_cast<const uint64_t *>(mr + 32 + tx * 2);
            if constexpr (OPT == 8) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(mr + 32 + ((tx * 4) ^ pca_swizzle<OPT>(i)));
                mv[2] = t.x;
                mv[3] = t.y;
            }
#pragma unroll
            for (int q = 0; q < PPT; ++q) {
                const uint64_t xx = pair2(xv[q], xv[q]);
#pragma unroll
                for (int o = 0; o < OPT / 2; ++o) mul_add2(acc[q][o], mv[o], xx, one2);
            }
        }
    }

    const uint32_t chunk = out_kind >= 3 ? 2 : 1;
    const int delta = (out_kind == 2 || out_kind == 4) ? 128 : 0;
    const uint32_t width = d_out / chunk;
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
        const uint64_t p = p0 + ty * PPT + q;
        if (p >= n) break;
#pragma unroll
        for (int o = 0; o < OPT; o += 4) {
            constexpr int kMost = 4;
            const int cnt = OPT - o < kMost ? OPT - o : kMost;  // 4, or the 2 past column 32 of OPT = 6
            const uint32_t j = j0 + pca_col<OPT>(tx, o);
            float v[kMost];
#pragma unroll
            for (int c = 0; c < kMost; c += 2)
                if (c < cnt) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[c]), "=f"(v[c + 1]) : "l"(acc[q][(o + c) / 2]));
#pragma unroll
            for (int c = 0; c < kMost; ++c)
                if (c < cnt) v[c] = __fadd_rn(j + c < d_out ? __ldg(bias + j + c) : 0.0f, v[c]);  // bias - (-dot)
            if (out_kind == 0) {
                float *d = static_cast<float *>(out) + p * d_out + j;
                if (wide && j + cnt <= d_out) {
                    if (cnt == 4) __stcs(reinterpret_cast<float4 *>(d), make_float4(v[0], v[1], v[2], v[3]));
                    else __stcs(reinterpret_cast<float2 *>(d), make_float2(v[0], v[1]));
                } else {
#pragma unroll
                    for (int c = 0; c < kMost; ++c)
                        if (c < cnt && j + c < d_out) d[c] = v[c];
                }
                continue;
            }
            uint32_t code[kMost] = {0, 0, 0, 0};
#pragma unroll
            for (int c = 0; c < kMost; ++c)
                if (c < cnt) code[c] = uint32_t(quant_code(v[c]) - delta) & 0xFFu;
            uint8_t *d = static_cast<uint8_t *>(out) + p * width + j / chunk;
            if (chunk == 2) {  // high nibble = element 2i + 1 (j and d_out are even)
                const uint32_t lo = (code[1] & 0xF0u) | (code[0] >> 4), hi = (code[3] & 0xF0u) | (code[2] >> 4);
                if (wide && cnt == 4 && j + 4 <= d_out) {
                    *reinterpret_cast<uint16_t *>(d) = uint16_t(lo | (hi << 8));
                } else {
                    if (j < d_out) d[0] = uint8_t(lo);
                    if (cnt == 4 && j + 2 < d_out) d[1] = uint8_t(hi);
                }
            } else if (wide && cnt == 4 && j + 4 <= d_out) {
                *reinterpret_cast<uint32_t *>(d) = code[0] | (code[1] << 8) | (code[2] << 16) | (code[3] << 24);
            } else {
#pragma unroll
                for (int c = 0; c < kMost; ++c)
                    if (c < cnt && j + c < d_out) d[c] = uint8_t(code[c]);
            }
        }
    }
}

// FmtConv u8bin2u4bin: byte j = (row[2j+1] & 0xF0) + (row[2j] >> 4); odd last element dropped
__global__ void u8_to_u4_kernel(const uint8_t *rows, uint64_t n, uint32_t dims, uint8_t *out)
{
    const uint32_t half = dims >> 1;
    for (uint64_t e = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; e < n * half; e += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t p = e / half, j = e % half;
        out[e] = uint8_t((rows[p * dims + 2 * j + 1] & 0xF0) + (rows[p * dims + 2 * j] >> 4));
    }
}

// FmtConv fbin2u8bin: static_cast<unsigned char>(v) for 0 <= v < 256; *bad set otherwise
__global__ void f32_to_u8_kernel(const float *rows, uint64_t count, uint8_t *out, uint32_t *bad)
{
    for (uint64_t e = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; e < count; e += uint64_t(gridDim.x) * blockDim.x) {
        const float v = rows[e];
        if (!(v >= 0.0f && v < 256.0f)) {
            atomicExch(bad, 1u);
            out[e] = 0;
        } else {
            out[e] = uint8_t(__float2uint_rz(v));
        }
    }
}

static uint32_t out_width(uint32_t out_dtype, uint32_t d_out)
{
    return (out_dtype == NBPG_U4 || out_dtype == NBPG_I4) ? d_out / 2 : d_out;
}

static int out_kind_of(uint32_t out_dtype)
{
    switch (out_dtype) {
    case NBPG_F32: return 0;
    case NBPG_U8: return 1;
    case NBPG_I8: return 2;
    case NBPG_U4: return 3;
    default: return 4;
    }
}

template <int IN, int PPT>
static void launch_pca_outs(uint32_t opt, dim3 grid, cudaStream_t st, const void *x, uint64_t n, uint32_t d_in,
                            const float *mat, const float *bias, uint32_t d_out, uint32_t kind, uint32_t vec, uint32_t wide, void *out)
{
    if (opt == 4) pca_kernel<IN, PPT, 4><<<grid, PCA_THREADS, 0, st>>>(x, n, d_in, mat, bias, d_out, kind, vec, wide, 1.0f, out);
    else if (opt == 6) pca_kernel<IN, PPT, 6><<<grid, PCA_THREADS, 0, st>>>(x, n, d_in, mat, bias, d_out, kind, vec, wide, 1.0f, out);
    else pca_kernel<IN, PPT, 8><<<grid, PCA_THREADS, 0, st>>>(x, n, d_in, mat, bias, d_out, kind, vec, wide, 1.0f, out);
}

template <int IN>
static void launch_pca_in(uint32_t ppt, uint32_t opt, dim3 grid, cudaStream_t st, const void *x, uint64_t n, uint32_t d_in,
                          const float *mat, const float *bias, uint32_t d_out, uint32_t kind, uint32_t vec, uint32_t wide, void *out)
{
    if (ppt == 8) launch_pca_outs<IN, 8>(opt, grid, st, x, n, d_in, mat, bias, d_out, kind, vec, wide, out);
    else launch_pca_outs<IN, 2>(opt, grid, st, x, n, d_in, mat, bias, d_out, kind, vec, wide, out);
}

static nbpg_status launch_pca(uint32_t in_dtype, const void *d_x, uint64_t n, uint32_t d_in, const float *d_mat,
                              const float *d_bias, uint32_t d_out, uint32_t out_dtype, void *d_out_rows,
                              cudaStream_t st)
{
    // columns per CTA: 32 or 48 where they cover d_out (no columns computed for padding), else 64; 48 for many points
    // only (1,000 rows of 128 -> 34: 22.3 us with 48 columns, 21.1 with 64; 20,000: 33 and 35)
    const uint32_t opt = d_out <= 32 ? 4 : d_out <= 48 && n >= 8192 ? 6 : 8;
    // 256-point tiles once they fill every SM's two CTAs (2 x 152 x 256 = 78k points), else 64-point ones
    const uint32_t ppt = n >= 80000 ? 8 : 2;
    const uint32_t pts = 32 * ppt, outs = 8 * opt;
    const dim3 grid(uint32_t((n + pts - 1) / pts), (d_out + outs - 1) / outs);
    const uint32_t kind = uint32_t(out_kind_of(out_dtype));
    const uint32_t vec = d_in % 4 == 0 && reinterpret_cast<uintptr_t>(d_x) % (in_dtype == NBPG_F32 ? 16 : 4) == 0;
    const uint32_t wide = d_out % 4 == 0 && reinterpret_cast<uintptr_t>(d_out_rows) % 16 == 0;
    switch (in_dtype) {
    case NBPG_F32: launch_pca_in<PIN_F32>(ppt, opt, grid, st, d_x, n, d_in, d_mat, d_bias, d_out, kind, vec, wide, d_out_rows); break;
    case NBPG_U8: launch_pca_in<PIN_U8>(ppt, opt, grid, st, d_x, n, d_in, d_mat, d_bias, d_out, kind, vec, wide, d_out_rows); break;
    default: launch_pca_in<PIN_I8>(ppt, opt, grid, st, d_x, n, d_in, d_mat, d_bias, d_out, kind, vec, wide, d_out_rows);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("nbpg_pca_encode: ") + cudaGetErrorString(e));
        return NBPG_ERR_CUDA;
    }
    return NBPG_OK;
}

static nbpg_status check_pca_args(uint32_t in_dtype, uint64_t n, uint32_t d_in, uint32_t d_out, uint32_t out_dtype)
{
    NBPG_CHECK_ARG(in_dtype == NBPG_F32 || in_dtype == NBPG_U8 || in_dtype == NBPG_I8, "input rows must be f32, u8 or i8");
    NBPG_CHECK_ARG(out_dtype <= NBPG_F32, "bad output type");
    NBPG_CHECK_ARG(d_in >= 1 && d_in <= PCA_MAX_DIN, "d_in must be in [1, 576]");
    NBPG_CHECK_ARG(d_out >= 1, "d_out must be >= 1");
    NBPG_CHECK_ARG(!(out_dtype == NBPG_U4 || out_dtype == NBPG_I4) || d_out % 2 == 0,
                   "4-bit output needs an even d_out");
    NBPG_CHECK_ARG(n < (uint64_t(1) << 40), "too many rows");
    return NBPG_OK;
}

}  // namespace nbpg

using namespace nbpg;

extern "C" nbpg_status nbpg_pca_encode_device(uint32_t in_dtype, const void *d_rows, uint64_t n, uint32_t d_in,
                                              const float *d_mat, const float *d_bias, uint32_t d_out,
                                              uint32_t out_dtype, void *d_out_rows, void *stream)
{
    NBPG_CHECK_ARG(d_rows && d_mat && d_bias && d_out_rows, "null argument");
    const nbpg_status s = check_pca_args(in_dtype, n, d_in, d_out, out_dtype);
    if (s != NBPG_OK || n == 0) return s;
    return launch_pca(in_dtype, d_rows, n, d_in, d_mat, d_bias, d_out, out_dtype, d_out_rows,
                      static_cast<cudaStream_t>(stream));
}

// Host buffers; rows stream through the device in blocks of at most 4M rows.
extern "C" nbpg_status nbpg_pca_encode(uint32_t in_dtype, const void *rows, uint64_t n, uint32_t d_in,
                                       const float *mat, const float *bias, uint32_t d_out, uint32_t out_dtype,
                                       void *out, int32_t device)
{
    NBPG_CHECK_ARG(rows && mat && out, "null argument");
    nbpg_status s = check_pca_args(in_dtype, n, d_in, d_out, out_dtype);
    if (s != NBPG_OK || n == 0) return s;
    NBPG_CUDA_TRY(cudaSetDevice(device));
    const size_t in_b = in_dtype == NBPG_F32 ? 4 : 1;
    const size_t out_b = (out_dtype == NBPG_F32 ? 4 : 1) * size_t(out_width(out_dtype, d_out));
    const uint64_t blk = std::min<uint64_t>(n, uint64_t(1) << 22);
    cudaStream_t st;
    NBPG_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    void *dx = nullptr, *dy = nullptr;
    float *dm = nullptr, *db = nullptr;
    cudaError_t e = cudaMalloc(&dx, blk * d_in * in_b);
    if (e == cudaSuccess) e = cudaMalloc(&dy, blk * out_b);
    if (e == cudaSuccess) e = cudaMalloc(&dm, size_t(d_out) * d_in * 4);
    if (e == cudaSuccess) e = cudaMalloc(&db, size_t(d_out) * 4);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dm, mat, size_t(d_out) * d_in * 4, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        if (bias) e = cudaMemcpyAsync(db, bias, size_t(d_out) * 4, cudaMemcpyHostToDevice, st);
        else e = cudaMemsetAsync(db, 0, size_t(d_out) * 4, st);
    }
    for (uint64_t p = 0; e == cudaSuccess && s == NBPG_OK && p < n; p += blk) {
        const uint64_t cnt = std::min<uint64_t>(blk, n - p);
        e = cudaMemcpyAsync(dx, static_cast<const uint8_t *>(rows) + p * d_in * in_b, cnt * d_in * in_b,
                            cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) s = launch_pca(in_dtype, dx, cnt, d_in, dm, db, d_out, out_dtype, dy, st);
        if (e == cudaSuccess && s == NBPG_OK)
            e = cudaMemcpyAsync(static_cast<uint8_t *>(out) + p * out_b, dy, cnt * out_b, cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess && s == NBPG_OK) {
        set_error(std::string("nbpg_pca_encode: ") + cudaGetErrorString(e));
        s = e == cudaErrorMemoryAllocation ? NBPG_ERR_OOM : NBPG_ERR_CUDA;
    }
    cudaStreamSynchronize(st);
    cudaFree(dx);
    cudaFree(dy);
    cudaFree(dm);
    cudaFree(db);
    cudaStreamDestroy(st);
    return s;
}

extern "C" nbpg_status nbpg_u8_to_u4(const uint8_t *rows, uint64_t n, uint32_t dims, uint8_t *out, int32_t device)
{
    NBPG_CHECK_ARG(rows && out, "null argument");
    NBPG_CHECK_ARG(dims >= 2, "dims must be >= 2");
    if (n == 0) return NBPG_OK;
    NBPG_CUDA_TRY(cudaSetDevice(device));
    uint8_t *dx = nullptr, *dy = nullptr;
    const size_t half = dims >> 1;
    nbpg_status s = NBPG_OK;
    cudaError_t e = cudaMalloc(&dx, n * dims);
    if (e == cudaSuccess) e = cudaMalloc(&dy, n * half);
    if (e == cudaSuccess) e = cudaMemcpy(dx, rows, n * dims, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        u8_to_u4_kernel<<<1024, 256>>>(dx, n, dims, dy);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dy, n * half, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        set_error(std::string("nbpg_u8_to_u4: ") + cudaGetErrorString(e));
        s = e == cudaErrorMemoryAllocation ? NBPG_ERR_OOM : NBPG_ERR_CUDA;
    }
    cudaFree(dx);
    cudaFree(dy);
    return s;
}

extern "C" nbpg_status nbpg_f32_to_u8(const float *rows, uint64_t n, uint32_t dims, uint8_t *out, int32_t device)
{
    NBPG_CHECK_ARG(rows && out, "null argument");
    if (n == 0 || dims == 0) return NBPG_OK;
    NBPG_CUDA_TRY(cudaSetDevice(device));
    float *dx = nullptr;
    uint8_t *dy = nullptr;
    uint32_t *dbad = nullptr, bad = 0;
    nbpg_status s = NBPG_OK;
    const uint64_t cnt = n * dims;
    cudaError_t e = cudaMalloc(&dx, cnt * 4);
    if (e == cudaSuccess) e = cudaMalloc(&dy, cnt);
    if (e == cudaSuccess) e = cudaMalloc(&dbad, 4);
    if (e == cudaSuccess) e = cudaMemset(dbad, 0, 4);
    if (e == cudaSuccess) e = cudaMemcpy(dx, rows, cnt * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        f32_to_u8_kernel<<<1024, 256>>>(dx, cnt, dy, dbad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dy, cnt, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&bad, dbad, 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        set_error(std::string("nbpg_f32_to_u8: ") + cudaGetErrorString(e));
        s = e == cudaErrorMemoryAllocation ? NBPG_ERR_OOM : NBPG_ERR_CUDA;
    } else if (bad) {
        set_error("nbpg_f32_to_u8: a value lies outside [0, 256)");
        s = NBPG_ERR_INVALID_ARG;
    }
    cudaFree(dx);
    cudaFree(dy);
    cudaFree(dbad);
    return s;
}
