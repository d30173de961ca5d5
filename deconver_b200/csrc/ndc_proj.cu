// What stands around the update inside the layer, apart from the projection's library GEMMs: the
// weight gradient of a 1x1 projection, and the small per-parameter passes.
//
//   wgrad   gw[o, c] = sum over samples and positions of gy[b, o, p] * x[b, c, p].  A GEMM with a
//           tiny output and a huge inner dimension; both operands are read along the inner
//           dimension as they lie.  The library's convolution backward takes a kernel without
//           vector loads when the row length is not a multiple of four (1.63 ms for 192 x 48
//           channels over 2 x 88 245 positions, two reads being 0.026 ms), converts to channels-last
//           for others, and runs too few blocks for small batches.  Here the positions are split over
//           as many CTAs as fill the GPU whatever their number is; partial products are added in a
//           fixed order by a second kernel, which also converts to the parameter's type.  What
//           bounds it: one read of gy and x (at 4.1 TB/s in float32, 5.7 in bfloat16) while a tile of
//           128 x 64 outputs is enough; with more channels, or few in a tile, the rate of
//           `mma.sync` on whole tiles, 134 TFLOP/s in float32 (each warp rounds its operands to
//           TF32, three instructions a value) and 272 in bfloat16.  5 x (96 + 24) x 34916 in float32
//           takes 36 us, the read alone 13.  Where it is taken: plan_weight_grad in ndc_torch.cpp.
//   params  filter h = relu(h0) and bias as float32 for the update kernels (one launch), and the
//           parameter gradients masked and converted on the way back (one launch).
#include <cstdarg>
#include <cstdio>

#include "ndc_b200.h"
#include "ndc_common.cuh"
#include "ndc_slab.cuh"

namespace {

thread_local char g_proj_err[256] = "";

int proj_fail(int status, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_proj_err, sizeof(g_proj_err), fmt, ap);
    va_end(ap);
    return status;
}

typedef __nv_bfloat16 bf16;

// ---- weight gradient ------------------------------------------------------------------------
// One CTA: a TO x TC tile of the output over one slice of one sample's positions.  A stage holds
// TO rows of gy and TC rows of x, 32 words (32 float32 or 64 bfloat16 positions) each, in rows of
// 36 words: eight rows of 16 bytes, as ldmatrix reads them, hit 32 different banks.
// TO = 128, TC = 64: with up to 64 input channels gy, the larger operand, is read once; with more, twice.
constexpr int TO = 128, TC = 64, KW = 32, LDW = 36, STAGES = 3, WNT = 256;
constexpr size_t kWgradSmem = (size_t)STAGES * (TO + TC) * LDW * 4;

__device__ __forceinline__ void cp_async(void* dst, const void* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
// The leading 11 significant bits of v, rounded to nearest (Veltkamp's splitting by 2^13 + 1): three
// full-rate instructions, where a conversion instruction runs at a fraction of that rate.
__device__ __forceinline__ float to_tf32(float v) {
    const float c = __fmul_rn(v, 8193.0f);
    return __fsub_rn(c, __fsub_rn(c, v));
}
__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], const unsigned* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

struct WgradParams {
    const void* gy; const void* x;
    float* partial;            // [slice][Co][Ci]
    int co, ci, tiles_o, tiles_c;
    int slices_per_sample;
    long long n, slice;        // positions per sample and per slice (a multiple of 64)
};

// VEC: bytes of one copy: 16 (rows on 16-byte boundaries), 4 (float32 rows of any length, or
// bfloat16 rows of even length), 0 (element loads: bfloat16 rows of odd length).  EXACT: float32
// as the sum of two tf32 terms, three products (used where TF32 products are not allowed).  The MMA rounds its
// accumulators towards zero, which adds up along a slice, so a stage's twelve are added to sums
// that round to nearest: 3.6e-7 of the result against 64 bits where one chain was off by 3.6e-6
// (5 x (96 + 24) x 34916; the library's float32 5.8e-7).
template <typename T, int VEC, bool EXACT>
__global__ void __launch_bounds__(WNT, 2) wgrad1x1_kernel(const WgradParams P) {
    constexpr int PPW = 4 / (int)sizeof(T);    // positions per word
    constexpr int KP = KW * PPW;               // positions per stage
    extern __shared__ __align__(16) unsigned smem_w[];
    int blk = blockIdx.x;
    const int tc = blk % P.tiles_c; blk /= P.tiles_c;
    const int to = blk % P.tiles_o; blk /= P.tiles_o;
    const int slice = blk, b = slice / P.slices_per_sample;
    const long long p0 = (long long)(slice % P.slices_per_sample) * P.slice;
    const long long p1 = min(P.n, p0 + P.slice);
    const int o0 = to * TO, c0 = tc * TC;
    const T* gy = reinterpret_cast<const T*>(P.gy) + ((long long)b * P.co + o0) * P.n;
    const T* x = reinterpret_cast<const T*>(P.x) + ((long long)b * P.ci + c0) * P.n;
    const int rows_o = min(TO, P.co - o0), rows_c = min(TC, P.ci - c0);
    const int tid = threadIdx.x;
    const int steps = (int)((p1 - p0 + KP - 1) / KP);

    auto stage = [&](int s) {
        unsigned* dst = smem_w + (s % STAGES) * (TO + TC) * LDW;
        const long long p = p0 + (long long)s * KP;
        constexpr int W = VEC == 16 ? 4 : 1;   // words per copy
        constexpr int PER_ROW = KW / W;
        for (int i = tid; i < (TO + TC) * PER_ROW; i += WNT) {
            const int r = i / PER_ROW, w = (i % PER_ROW) * W;
            const bool is_o = r < TO;
            const int rr = is_o ? r : r - TO;
            unsigned* q = dst + r * LDW + w;
            const long long pos = p + (long long)w * PPW;
            const bool row_ok = rr < (is_o ? rows_o : rows_c);
            const T* src = (is_o ? gy : x) + (long long)rr * P.n + pos;
            if (VEC > 0) {
                if (row_ok && pos < p1) cp_async(q, src, VEC);   // rows hold whole copies
                else {
#pragma unroll
                    for (int k = 0; k < W; ++k) q[k] = 0u;
                }
            } else {
                unsigned v = 0u;
                const unsigned short* u = reinterpret_cast<const unsigned short*>(src);
                if (row_ok && pos < p1) v = u[0];
                if (row_ok && pos + 1 < p1) v |= (unsigned)u[1] << 16;
                q[0] = v;
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wo = (warp >> 1) * 32, wc = (warp & 1) * 32;   // 4 x 2 warps of 32 x 32 outputs
    float acc[2][4][4], sum[2][4][4];           // sum: EXACT
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = sum[i][j][k] = 0.0f;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) stage(s); else asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const bool busy = wo < rows_o && wc < rows_c;    // warps past the edge only help copying
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        if (s + STAGES - 1 < steps) stage(s + STAGES - 1); else asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (!busy) continue;
        const unsigned* base = smem_w + (s % STAGES) * (TO + TC) * LDW;
        // ldmatrix row addresses: matrices (rows 0-7, words 0-3), (8-15, 0-3), (0-7, 4-7), (8-15, 4-7)
        // for a 16-row A tile; (0-7, 0-3), (0-7, 4-7), (8-15, ...) for two 8-row B tiles
        const unsigned* A = base + (wo + (lane & 7) + ((lane >> 3) & 1) * 8) * LDW + (lane >> 4) * 4;
        const unsigned* B = base + (TO + wc + (lane & 7) + (lane >> 4) * 8) * LDW + ((lane >> 3) & 1) * 4;
#pragma unroll
        for (int k = 0; k < KW; k += 8) {
            unsigned a[2][4], bb[4][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) ldmatrix4(a[i], A + 16 * i * LDW + k);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                unsigned r[4];
                ldmatrix4(r, B + 16 * j * LDW + k);
                bb[2 * j][0] = r[0]; bb[2 * j][1] = r[1];
                bb[2 * j + 1][0] = r[2]; bb[2 * j + 1][1] = r[3];
            }
            if (sizeof(T) == 2) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], a[i], bb[j]);
            } else {
                unsigned al[2][4], bl[4][2];     // remainders (EXACT)
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float v = __uint_as_float(a[i][q]);
                        const float hi = to_tf32(v);
                        a[i][q] = __float_as_uint(hi);
                        al[i][q] = EXACT ? __float_as_uint(to_tf32(v - hi)) : 0u;
                    }
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float v = __uint_as_float(bb[j][q]);
                        const float hi = to_tf32(v);
                        bb[j][q] = __float_as_uint(hi);
                        bl[j][q] = EXACT ? __float_as_uint(to_tf32(v - hi)) : 0u;
                    }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (EXACT) {
                            mma_tf32(acc[i][j], al[i], bb[j]);
                            mma_tf32(acc[i][j], a[i], bl[j]);
                        }
                        mma_tf32(acc[i][j], a[i], bb[j]);
                    }
            }
        }
        if (EXACT) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int q = 0; q < 4; ++q) { sum[i][j][q] += acc[i][j][q]; acc[i][j][q] = 0.0f; }
        }
    }
    if (!busy) return;
    float* out = P.partial + (long long)slice * P.co * P.ci;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int o = o0 + wo + 16 * i + g + (q >> 1) * 8, c = c0 + wc + 8 * j + 2 * t + (q & 1);
                if (o < P.co && c < P.ci) out[(long long)o * P.ci + c] = EXACT ? sum[i][j][q] : acc[i][j][q];
            }
}

// gw[e] = sum of the slices' partial products in a fixed order: a warp's 32 elements are summed by
// eight warps, an eighth of the slices each, so that an output of a few thousand elements does not
// leave the GPU waiting on one long chain of loads per thread.
template <typename T>
__global__ void __launch_bounds__(256) wgrad1x1_sum_kernel(const float* __restrict__ partial, int slices,
                                                           long long n, T* __restrict__ gw) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long e = (long long)blockIdx.x * 32 + lane;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (e < n) {
        int i = w;
        for (; i + 24 < slices; i += 32)
#pragma unroll
            for (int k = 0; k < 4; ++k) s[k] += partial[(i + 8 * k) * n + e];
        for (; i < slices; i += 8) s[0] += partial[i * n + e];
    }
    part[w][lane] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    if (w == 0 && e < n) {
        float r = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) r += part[k][lane];
        gw[e] = ndc::from_f32<T>(r);
    }
}

// The same sum where there are few slices (one per sample): a thread per element.
template <typename T>
__global__ void __launch_bounds__(256) wgrad1x1_few_kernel(const float* __restrict__ partial, int slices,
                                                           long long n, T* __restrict__ gw) {
    const long long e = (long long)blockIdx.x * 256 + threadIdx.x;
    if (e >= n) return;
    float s = partial[e];
    for (int i = 1; i < slices; ++i) s += partial[i * n + e];
    gw[e] = ndc::from_f32<T>(s);
}

// Slices: enough CTAs for two rounds of two per multiprocessor, of at least 512 positions (a
// slice costs one partial product of the size of the output, written and read again).
void plan_wgrad(int batch, int co, int ci, long long n, WgradParams& P) {
    P.tiles_o = (co + TO - 1) / TO;
    P.tiles_c = (ci + TC - 1) / TC;
    const long long tiles = (long long)P.tiles_o * P.tiles_c * batch;
    long long want = (4LL * ndc::num_sms() + tiles - 1) / tiles;
    const long long most = (n + 511) / 512;
    if (want > most) want = most;
    if (want < 1) want = 1;
    P.slice = ((n + want - 1) / want + 63) / 64 * 64;
    P.slices_per_sample = (int)((n + P.slice - 1) / P.slice);
    P.co = co; P.ci = ci; P.n = n;
}

template <typename T, int VEC, bool EXACT>
cudaError_t launch_wgrad(const WgradParams& P, unsigned grid, cudaStream_t st) {
    auto kern = wgrad1x1_kernel<T, VEC, EXACT>;
    const cudaError_t e = ndc::allow_smem(kern);
    if (e != cudaSuccess) return e;
    kern<<<grid, WNT, kWgradSmem, st>>>(P);
    ndc::launched();
    return cudaGetLastError();
}

cudaError_t launch_sum(int dtype, const float* partial, int slices, long long n, void* gw, cudaStream_t st) {
    // a chain of up to 16 loads per thread is no longer than the other kernel's, as soon as the
    // elements fill the GPU (2 slices of 1 M elements: 26 us there, most warps having no slice)
    if (slices <= 16 && n >= 65536) {
        const unsigned blocks = (unsigned)((n + 255) / 256);
        if (dtype == NDC_BF16) wgrad1x1_few_kernel<bf16><<<blocks, 256, 0, st>>>(partial, slices, n, (bf16*)gw);
        else wgrad1x1_few_kernel<float><<<blocks, 256, 0, st>>>(partial, slices, n, (float*)gw);
        ndc::launched();
        return cudaGetLastError();
    }
    const unsigned blocks = (unsigned)((n + 31) / 32);
    if (dtype == NDC_BF16) wgrad1x1_sum_kernel<bf16><<<blocks, 256, 0, st>>>(partial, slices, n, (bf16*)gw);
    else wgrad1x1_sum_kernel<float><<<blocks, 256, 0, st>>>(partial, slices, n, (float*)gw);
    ndc::launched();
    return cudaGetLastError();
}

// ---- per-parameter passes ---------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) params_prepare_kernel(const T* __restrict__ h0, long long nh, float* __restrict__ h,
                                                             const T* __restrict__ bias, long long nb, float* __restrict__ b) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i < nh) {
        const float v = ndc::to_f32(h0[i]);
        h[i] = v < 0.0f ? 0.0f : v;        // relu as the library has it: a NaN stays one
    } else if (i - nh < nb) {
        b[i - nh] = ndc::to_f32(bias[i - nh]);
    }
}
template <typename T>
__global__ void __launch_bounds__(256) params_grad_kernel(const T* __restrict__ h0, const float* __restrict__ gh, long long nh,
                                                          T* __restrict__ gh0, const float* __restrict__ gb, long long nb,
                                                          T* __restrict__ gbias) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i < nh) gh0[i] = ndc::from_f32<T>(ndc::to_f32(h0[i]) <= 0.0f ? 0.0f : gh[i]);
    else if (i - nh < nb) gbias[i - nh] = ndc::from_f32<T>(gb[i - nh]);
}

// ---- row padding ------------------------------------------------------------------------------
// One thread per quad of a padded row: scalar accesses to the unpadded side (neighbouring threads
// touch neighbouring quads), one vector access to the padded one.
template <typename T> struct Quad;
template <> struct Quad<float> { typedef float4 type; };
template <> struct Quad<unsigned short> { typedef ushort4 type; };

template <typename T, bool PAD>
__global__ void __launch_bounds__(256) rows_kernel(const T* __restrict__ src, T* __restrict__ dst, long long quads, int W, int nq) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= quads) return;
    const long long row = i / nq;
    const int w = 4 * (int)(i - row * nq);
    typename Quad<T>::type q;
    T* e = reinterpret_cast<T*>(&q);
    if (PAD) {
#pragma unroll
        for (int k = 0; k < 4; ++k) e[k] = w + k < W ? src[row * W + w + k] : T(0);
        reinterpret_cast<typename Quad<T>::type*>(dst)[i] = q;
    } else {
        q = reinterpret_cast<const typename Quad<T>::type*>(src)[i];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (w + k < W) dst[row * W + w + k] = e[k];
    }
}

int launch_rows(bool pad, int64_t rows, int32_t W, int32_t pitch, int32_t dtype, const void* src, void* dst, void* stream) {
    if (!src || !dst || rows <= 0 || W <= 0 || pitch < W || pitch % 4 || (dtype != NDC_F32 && dtype != NDC_BF16))
        return proj_fail(NDC_ERR_INVALID, "row padding: invalid argument");
    if ((uintptr_t)(pad ? dst : src) % (dtype == NDC_BF16 ? 8 : 16))
        return proj_fail(NDC_ERR_ALIGNMENT, "row padding: the padded tensor is not aligned");
    const long long quads = rows * (pitch / 4);
    const unsigned blocks = (unsigned)((quads + 255) / 256);
    cudaStream_t st = (cudaStream_t)stream;
    typedef unsigned short u16;
    if (dtype == NDC_F32) {
        if (pad) rows_kernel<float, true><<<blocks, 256, 0, st>>>((const float*)src, (float*)dst, quads, W, pitch / 4);
        else rows_kernel<float, false><<<blocks, 256, 0, st>>>((const float*)src, (float*)dst, quads, W, pitch / 4);
    } else {
        if (pad) rows_kernel<u16, true><<<blocks, 256, 0, st>>>((const u16*)src, (u16*)dst, quads, W, pitch / 4);
        else rows_kernel<u16, false><<<blocks, 256, 0, st>>>((const u16*)src, (u16*)dst, quads, W, pitch / 4);
    }
    ndc::launched();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return proj_fail(NDC_ERR_CUDA, "row padding: %s", cudaGetErrorString(e));
    return NDC_OK;
}

}  // namespace

extern "C" {

const char* ndc_proj_last_error(void) { return g_proj_err; }

size_t ndc_proj_wgrad_workspace_bytes(int32_t batch, int32_t co, int32_t ci, int64_t spatial) {
    if (batch <= 0 || co <= 0 || ci <= 0 || spatial <= 0) return 0;
    WgradParams P;
    plan_wgrad(batch, co, ci, spatial, P);
    return (size_t)batch * P.slices_per_sample * co * ci * sizeof(float);
}

int ndc_proj_wgrad(int32_t batch, int32_t co, int32_t ci, int64_t spatial, int32_t dtype, int32_t tf32,
                   const void* gy, const void* x, void* gw, void* workspace, size_t workspace_bytes,
                   void* stream) {
    if (!gy || !x || !gw) return proj_fail(NDC_ERR_INVALID, "projection gradient: gy, x and gw must not be NULL");
    if (batch <= 0 || co <= 0 || ci <= 0 || spatial <= 0)
        return proj_fail(NDC_ERR_INVALID, "projection gradient: extents must be positive");
    if (dtype != NDC_F32 && dtype != NDC_BF16)
        return proj_fail(NDC_ERR_INVALID, "projection gradient: dtype must be NDC_F32 or NDC_BF16");
    const size_t need = ndc_proj_wgrad_workspace_bytes(batch, co, ci, spatial);
    if (!workspace || workspace_bytes < need)
        return proj_fail(NDC_ERR_WORKSPACE, "projection gradient: workspace of %zu bytes needed", need);
    WgradParams P;
    plan_wgrad(batch, co, ci, spatial, P);
    P.gy = gy; P.x = x; P.partial = (float*)workspace;
    const long long grid = (long long)P.tiles_o * P.tiles_c * batch * P.slices_per_sample;
    if (grid > 0x7fffffffLL) return proj_fail(NDC_ERR_UNSUPPORTED, "projection gradient: problem too large");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t row = (size_t)spatial * (dtype == NDC_BF16 ? 2 : 4);
    const uintptr_t at = (uintptr_t)gy | (uintptr_t)x | row;
    cudaError_t e;
    if (dtype == NDC_BF16)
        e = at % 16 == 0 ? launch_wgrad<bf16, 16, false>(P, (unsigned)grid, st)
          : at % 4 == 0 ? launch_wgrad<bf16, 4, false>(P, (unsigned)grid, st)
                        : launch_wgrad<bf16, 0, false>(P, (unsigned)grid, st);
    else if (tf32)
        e = at % 16 == 0 ? launch_wgrad<float, 16, false>(P, (unsigned)grid, st)
                         : launch_wgrad<float, 4, false>(P, (unsigned)grid, st);
    else
        e = at % 16 == 0 ? launch_wgrad<float, 16, true>(P, (unsigned)grid, st)
                         : launch_wgrad<float, 4, true>(P, (unsigned)grid, st);
    if (e == cudaSuccess)
        e = launch_sum(dtype, P.partial, batch * P.slices_per_sample, (long long)co * ci, gw, st);
    if (e != cudaSuccess) return proj_fail(NDC_ERR_CUDA, "projection gradient: %s", cudaGetErrorString(e));
    return NDC_OK;
}

int ndc_proj_sum(int32_t slices, int64_t n, int32_t dtype, const float* partial, void* gw, void* stream) {
    if (!partial || !gw || slices <= 0 || n <= 0 || (dtype != NDC_F32 && dtype != NDC_BF16))
        return proj_fail(NDC_ERR_INVALID, "projection gradient sum: invalid argument");
    const cudaError_t e = launch_sum(dtype, partial, slices, n, gw, (cudaStream_t)stream);
    if (e != cudaSuccess) return proj_fail(NDC_ERR_CUDA, "projection gradient sum: %s", cudaGetErrorString(e));
    return NDC_OK;
}

int ndc_pad_rows(int64_t rows, int32_t W, int32_t pitch, int32_t dtype, const void* src, void* dst, void* stream) {
    return launch_rows(true, rows, W, pitch, dtype, src, dst, stream);
}
int ndc_unpad_rows(int64_t rows, int32_t W, int32_t pitch, int32_t dtype, const void* src, void* dst, void* stream) {
    return launch_rows(false, rows, W, pitch, dtype, src, dst, stream);
}

int ndc_params_prepare(int32_t dtype, const void* h0, int64_t nh, float* h, const void* bias, int64_t nb,
                       float* b, void* stream) {
    if (nh < 0 || nb < 0 || nh + nb == 0 || (nh && (!h0 || !h)) || (nb && (!bias || !b)) || (dtype != NDC_F32 && dtype != NDC_BF16))
        return proj_fail(NDC_ERR_INVALID, "parameter preparation: invalid argument");
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)((nh + nb + 255) / 256);
    if (dtype == NDC_F32)
        params_prepare_kernel<float><<<blocks, 256, 0, st>>>((const float*)h0, nh, h, (const float*)bias, nb, b);
    else
        params_prepare_kernel<bf16><<<blocks, 256, 0, st>>>((const bf16*)h0, nh, h, (const bf16*)bias, nb, b);
    ndc::launched();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return proj_fail(NDC_ERR_CUDA, "parameter preparation: %s", cudaGetErrorString(e));
    return NDC_OK;
}

int ndc_params_grad(int32_t dtype, const void* h0, const float* gh, int64_t nh, void* gh0, const float* gb,
                    int64_t nb, void* gbias, void* stream) {
    if (nh < 0 || nb < 0 || nh + nb == 0 || (nh && (!h0 || !gh || !gh0)) || (nb && (!gb || !gbias)) ||
        (dtype != NDC_F32 && dtype != NDC_BF16))
        return proj_fail(NDC_ERR_INVALID, "parameter gradients: invalid argument");
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)((nh + nb + 255) / 256);
    if (dtype == NDC_F32)
        params_grad_kernel<float><<<blocks, 256, 0, st>>>((const float*)h0, gh, nh, (float*)gh0, gb, nb, (float*)gbias);
    else
        params_grad_kernel<bf16><<<blocks, 256, 0, st>>>((const bf16*)h0, gh, nh, (bf16*)gh0, gb, nb, (bf16*)gbias);
    ndc::launched();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return proj_fail(NDC_ERR_CUDA, "parameter gradients: %s", cudaGetErrorString(e));
    return NDC_OK;
}

}  // extern "C"
