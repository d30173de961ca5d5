// The forward update of bfloat16 tensors on the 5th-generation tensor cores (m = 1, sc = 4; 3x3x3,
// 5x5 and 3x3 kernels), where the filter and the bias are bfloat16 values too, as in a bfloat16
// module.  Two launches: tc_source_kernel (t1 = K(relu(z + b))) and tc_adjoint_kernel (out).
//
// A depthwise convolution as a matrix product.  Rows of a plane lie in shared memory one after the
// other as bfloat16, column w at place w + PW of its row, zeros between the rows; a row takes a whole
// number PB of 8-column blocks.  The MMA's A operand is not a copy of that: its row r is the window
// of 16 places that starts at block r, and in the K-major layout without swizzle (8-row groups of
// 16-byte rows) this is the memory as it lies, with 16 bytes between the two halves of the window
// and 128 bytes between groups of eight blocks.  A filter row (kd, kh) is a shift of the start
// address.  The B operand is a banded matrix of one filter row: window place k, output column o of
// the block, one copy per output channel,
//
//     A: B[k][8 j + o] = h[j][kd][kh][o + 2 PW - k]        K: B[k][o] = h[j][kd][kh][k - o]
//
// so one M = 128, K = 16 MMA computes 1024 voxels of one filter row.  With KW = 3 a third of the
// products meet a zero of the band; the tensor cores do them 30 times faster than the FMA pipe does
// the useful ones.  What bounds an MMA of so few columns is reading its A operand (4 KB of shared
// memory, 32 cycles).
//
// Precision: every product is one of two bfloat16 values, exact in float32, accumulated in float32:
// what the FMA kernels compute, in another order.  The source relu(z + b) is not a bfloat16 value, but
// relu(z + b) = max(z, -b) + b and max(z, -b) is one; b K(1) is added in float32 afterwards, from a
// table over which filter taps lie inside the volume.
#pragma once

#include <algorithm>

#include "ndc_common.cuh"
#include "ndc_dw4_common.cuh"

namespace ndc {
namespace tc {

typedef __nv_bfloat16 bf16;
constexpr int SC = 4;             // source channels
constexpr int MB = 128;           // blocks (rows of an MMA)

struct Band {
    int C, D, H, W;               // W: row pitch (a multiple of 4)
    int Wv, Wo;                   // columns of the volume, row pitch of out (see Geo)
    int NB, PB;                   // blocks that hold columns, blocks per row in shared memory
    int TH, nth, DC, ndc, MT;     // rows and bands, planes and chunks, MMA tiles per band and plane
    long long SP;
    float eps;
    int relu;
};

// ---- PTX --------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Waits for the phase to complete; gives up (false) after a second, far above any MMA's time.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned phase) {
    unsigned long long start = 0;
    for (;;) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(phase) : "memory");
        if (done) return true;
        unsigned long long now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (!start) start = now;
        if (now - start > 1000000000ull) return false;
    }
}
__device__ __forceinline__ void tmem_alloc(unsigned slot, int cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(unsigned addr, int cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Eight columns of this thread's lane; the wait is part of the statement, so that nothing that uses
// the values can move in between.
__device__ __forceinline__ void tmem_load8(unsigned addr, float (&v)[8]) {
    unsigned r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_load8x2(unsigned addr_a, unsigned addr_b, float (&a)[8], float (&b)[8]) {
    unsigned r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr_a), "r"(addr_b) : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) { a[i] = __uint_as_float(r[i]); b[i] = __uint_as_float(r[8 + i]); }
}
__device__ __forceinline__ void tmem_zero8(unsigned addr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(addr), "r"(0u) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, no swizzle; `kstep` bytes between the 16-byte halves of
// K, `rstep` bytes between groups of eight rows.
__device__ __forceinline__ unsigned long long mat_desc(unsigned addr, int kstep, int rstep) {
    return (unsigned long long)((addr >> 4) & 0x3fff) | (unsigned long long)(kstep >> 4) << 16 |
           (unsigned long long)(rstep >> 4) << 32 | 1ull << 46;
}
// Instruction descriptor: bfloat16 operands, float32 accumulators, M = 128, N columns.
__device__ __forceinline__ unsigned instr_desc(int n) { return 1u << 4 | 1u << 7 | 1u << 10 | (unsigned)(n >> 3) << 17 | (unsigned)(MB >> 4) << 24; }

// ---- staging ----------------------------------------------------------------------------------
// Set where a wait ran out; the results of that launch are then undefined.
static __device__ unsigned g_wait_expired;

// Place of a band in the volume, and of the shared-memory planes in it.
struct At {
    int bc, c, h0, TH, d0, DC;
    __device__ __forceinline__ At(const Band& b, int blk) {
        const int th = blk % b.nth; blk /= b.nth;
        const int dc = blk % b.ndc; blk /= b.ndc;
        bc = blk; c = bc % b.C;
        h0 = th * b.TH; TH = min(b.TH, b.H - h0);
        d0 = dc * b.DC; DC = min(b.DC, b.D - d0);
    }
};

// Columns w-2 .. w+7 of a global row as five words, w = 8 q; zero outside the row.
template <bool WIDE>
__device__ __forceinline__ void load_words(const bf16* row, int w, const Band& b, unsigned (&a)[5]) {
#pragma unroll
    for (int i = 0; i < 5; ++i) a[i] = 0u;
    if (w > 0 && w - 4 < b.W) a[0] = __ldg(reinterpret_cast<const unsigned*>(row + w - 2));
    if (WIDE) {
        if (w < b.W) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + w));
            a[1] = v.x; a[2] = v.y; a[3] = v.z; a[4] = v.w;
        }
    } else {
        if (w < b.W) { const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + w)); a[1] = v.x; a[2] = v.y; }
        if (w + 4 < b.W) { const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + w + 4)); a[3] = v.x; a[4] = v.y; }
    }
}
// The eight places of block q of a shared row (columns 8 q - PW .. 8 q + 7 - PW) from those words.
// SOURCE: max(value, -bias) inside the volume (`negb`: two copies of -bias), zero in the padding.
template <int PW, bool SOURCE>
__device__ __forceinline__ uint4 to_places(unsigned (&a)[5], int w, const Band& b, unsigned negb, bool relu) {
    if (SOURCE) {
        if (relu) {
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const __nv_bfloat162 v = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a[i]), *reinterpret_cast<const __nv_bfloat162*>(&negb));
                a[i] = *reinterpret_cast<const unsigned*>(&v);
            }
            if (w == 0) a[0] = 0u;
        }
        if (w + 7 >= b.Wv) {                       // the row ends here
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const int c = w - 2 + 2 * i;
                if (c >= b.Wv) a[i] = 0u;
                else if (c + 1 >= b.Wv) a[i] &= 0xffffu;
            }
        }
    }
    if (PW == 2) return make_uint4(a[0], a[1], a[2], a[3]);
    return make_uint4(__funnelshift_l(a[0], a[1], 16), __funnelshift_l(a[1], a[2], 16), __funnelshift_l(a[2], a[3], 16),
                      __funnelshift_l(a[3], a[4], 16));
}

constexpr int kStagers = 256;     // threads that stage (and then run the epilogue)

// Bands of NCH channels (`src + ch * stride`, `dst + ch * blocks`), halo included, into shared memory;
// rows outside the volume are zero.  Four blocks per thread are in flight at a time: one at a time, the
// staging of a CTA took 20 us of latency.
template <int KD, int KH, int KW, int NCH, bool SOURCE, bool WIDE>
__device__ __forceinline__ void stage(uint4* dst, int blocks, const bf16* src, long long stride, const Band& b, const At& at,
                                      const unsigned (&negb)[NCH], bool relu) {
    constexpr int U = 2;                           // times NCH channels in flight
    const int rows = b.TH + KH - 1, planes = at.DC + KD - 1;
    const int dq = kStagers % b.PB, dr = kStagers / b.PB;
    int q = threadIdx.x % b.PB, row = threadIdx.x / b.PB, pl = 0, i = threadIdx.x;
    while (row >= rows) { row -= rows; ++pl; }
    while (pl < planes) {
        unsigned a[U][NCH][5];
        int w[U], at_i[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int d = at.d0 - KD / 2 + pl, h = at.h0 - KH / 2 + row;
            at_i[u] = pl < planes ? i : -1;
            w[u] = 8 * q;
            in[u] = pl < planes && d >= 0 && d < b.D && h >= 0 && h < b.H;
            if (in[u]) {
                const bf16* p = src + ((long long)d * b.H + h) * b.W;
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) load_words<WIDE>(p + ch * stride, w[u], b, a[u][ch]);
            }
            i += kStagers; q += dq; row += dr;
            if (q >= b.PB) { q -= b.PB; ++row; }
            while (row >= rows) { row -= rows; ++pl; }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (at_i[u] < 0) continue;
#pragma unroll
            for (int ch = 0; ch < NCH; ++ch)
                dst[ch * blocks + at_i[u]] = in[u] ? to_places<KW / 2, SOURCE>(a[u][ch], w[u], b, negb[ch], relu)
                                                   : make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

// The banded matrices of a kernel by one warp: `value(t, n, kw)` is the filter tap of matrix t, column n.
// Layout of one matrix: groups of eight columns, then the two halves of K, eight 16-byte rows each.
template <int NCOL, int KW, bool ADJ, typename F>
__device__ __forceinline__ void build_bands(bf16* bmat, int mats, int lane, F value) {
    for (int e = lane; e < mats * NCOL * 2; e += 32) {
        const int n = e % 8, half = (e / 8) % 2, g = (e / 16) % (NCOL / 8), t = e / (2 * NCOL);
        unsigned words[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float v[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int k = 8 * half + 2 * i + u, kw = ADJ ? n + KW - 1 - k : k - n;
                v[u] = kw >= 0 && kw < KW ? value(t, 8 * g + n, kw) : 0.0f;
            }
            const __nv_bfloat162 p = __floats2bfloat162_rn(v[0], v[1]);
            words[i] = *reinterpret_cast<const unsigned*>(&p);
        }
        reinterpret_cast<uint4*>(bmat)[e] = make_uint4(words[0], words[1], words[2], words[3]);
    }
}

// blocks of one channel's band in shared memory
template <int KD, int KH>
__host__ __device__ inline int band_blocks(const Band& b) { return (b.DC + KD - 1) * (b.TH + KH - 1) * b.PB; }
// blocks the last MMA tile of a band may read past it
__host__ __device__ inline int slack_blocks(const Band& b) { return b.MT * MB + 1 - b.TH * b.PB > 1 ? b.MT * MB + 1 - b.TH * b.PB : 1; }

constexpr int kThreads = 288;     // eight staging / epilogue warps and the MMA warp
constexpr int kHeader = 1024;     // bytes: barriers, TMEM address (256), the filter as float32

enum Access { kWide = 0, kQuad = 1, kPaddedOut = 2 };   // 16-byte rows; 8-byte rows; 8-byte rows, out unpadded

// eight voxels of a row from column w (8-aligned), zero past the pitch
template <int AL>
__device__ __forceinline__ uint4 load8(const bf16* row, int w, int W) {
    if (AL == kWide) return __ldg(reinterpret_cast<const uint4*>(row + w));
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    const uint2 lo = __ldg(reinterpret_cast<const uint2*>(row + w));
    v.x = lo.x; v.y = lo.y;
    if (w + 4 < W) { const uint2 hi = __ldg(reinterpret_cast<const uint2*>(row + w + 4)); v.z = hi.x; v.w = hi.y; }
    return v;
}
template <int AL>
__device__ __forceinline__ void store8(bf16* row, int w, int W, uint4 v) {
    if (AL == kWide) { *reinterpret_cast<uint4*>(row + w) = v; return; }
    *reinterpret_cast<uint2*>(row + w) = make_uint2(v.x, v.y);
    if (w + 4 < W) *reinterpret_cast<uint2*>(row + w + 4) = make_uint2(v.z, v.w);
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&p);
}
__device__ __forceinline__ float word_lane(const uint4& v, int i) {      // i static
    const unsigned w = i < 2 ? v.x : i < 4 ? v.y : i < 6 ? v.z : v.w;
    return __uint_as_float(i & 1 ? w & 0xffff0000u : w << 16);
}

// ---- out = s (A(x) + eps) / (A(t1) + eps) -------------------------------------------------------
struct AdjointArgs {
    Band b;
    const bf16* x; const bf16* t1; const bf16* z; bf16* out;
    const float* h; const float* bias;
};

// Work of a CTA: a band of TH rows of a chunk of DC planes.  x and t1 are staged whole, then the MMA
// warp runs ahead of the epilogue by up to four (plane, MMA tile) items of 64 accumulator columns (A(x)
// and A(t1), four channels of eight voxels each).
template <int KD, int KH, int KW, int AL>
__global__ void __launch_bounds__(kThreads, 2) tc_adjoint_kernel(const AdjointArgs P) {
    constexpr int ROWT = KD * KH, NCOL = SC * 8, BUFS = 4, TCOLS = 256;
    extern __shared__ __align__(128) unsigned char smem_tc[];
    const Band& b = P.b;
    const At at(b, blockIdx.x);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned base = smem_u32(smem_tc);
    const unsigned full = base, empty = base + 8 * BUFS, slot = base + 16 * BUFS;
    bf16* const bmat = reinterpret_cast<bf16*>(smem_tc + kHeader);
    uint4* const xs = reinterpret_cast<uint4*>(smem_tc + kHeader + ROWT * NCOL * 32);
    const int blocks = band_blocks<KD, KH>(b), slack = slack_blocks(b);
    uint4* const ts = xs + blocks;

    if (warp == 8) tmem_alloc(slot, TCOLS);
    if (tid == 0) {
        for (int i = 0; i < BUFS; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        float* const hs = reinterpret_cast<float*>(smem_tc + 256);
        for (int e = lane; e < SC * ROWT * KW; e += 32) hs[e] = P.h[(long long)at.c * SC * ROWT * KW + e];
        __syncwarp();
        build_bands<NCOL, KW, true>(bmat, ROWT, lane, [&](int t, int n, int kw) { return hs[(n / 8) * ROWT * KW + t * KW + kw]; });
    } else {
        // x and t1 as two channels: the distance between the tensors takes the place of the stride
        const unsigned none[2] = {0u, 0u};
        const long long apart = ((long long)(uintptr_t)P.t1 - (long long)(uintptr_t)P.x) / 2;
        stage<KD, KH, KW, 2, false, AL == kWide>(xs, blocks, P.x + (long long)at.bc * b.SP, apart, b, at, none, false);
    }
    // what the windows of valid blocks may touch past the staged planes has to be a number
    for (int i = tid; i < slack; i += kThreads) ts[blocks + i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0 && at.DC < b.DC) {
        const int end = (at.DC + KD - 1) * (b.TH + KH - 1) * b.PB;
        xs[end] = make_uint4(0u, 0u, 0u, 0u);
        ts[end] = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_async_proxy();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *reinterpret_cast<volatile unsigned*>(smem_tc + 16 * BUFS);
    const int items = at.DC * b.MT, plane = (b.TH + KH - 1) * b.PB;
    bool ok = true;
    if (warp == 8) {
        const unsigned idesc = instr_desc(NCOL);
        const unsigned xa = smem_u32(xs), ta = smem_u32(ts), ba = smem_u32(bmat);
        for (int it = 0; it < items && ok; ++it) {
            const int buf = it % BUFS, pl = it / b.MT, mt = it - pl * b.MT;
            if (it >= BUFS) ok = mbar_wait(empty + 8 * buf, ((it / BUFS) - 1) & 1);
            tc_fence_after();
            if (lane == 0 && ok) {
                const unsigned d = tmem + buf * 2 * NCOL;
                for (int t = 0; t < ROWT; ++t) {
                    const int kd = t / KH, kh = t - kd * KH;
                    const unsigned off = 16 * ((pl + KD - 1 - kd) * plane + (KH - 1 - kh) * b.PB + mt * MB);
                    const unsigned long long bd = mat_desc(ba + t * NCOL * 32, 128, 256);
                    mma(d, mat_desc(xa + off, 16, 128), bd, idesc, t > 0);
                    mma(d + NCOL, mat_desc(ta + off, 16, 128), bd, idesc, t > 0);
                }
                mma_commit(full + 8 * buf);
            }
            __syncwarp();
        }
    } else {
        const int grp = warp >> 2, m = (warp & 3) * 32 + lane;
        float bj[SC];
#pragma unroll
        for (int j = 0; j < SC; ++j) bj[j] = P.bias ? P.bias[at.c * SC + j] : 0.0f;
        const bf16* const zb = P.z + (long long)at.bc * SC * b.SP;
        const long long osp = (long long)b.D * b.H * b.Wo;
        bf16* const ob = P.out + (long long)at.bc * SC * osp;
        for (int it = grp; it < items && ok; it += 2) {
            const int buf = it % BUFS, pl = it / b.MT, mt = it - pl * b.MT;
            const int blk = mt * MB + m, r = blk / b.PB, q = blk - r * b.PB, w = 8 * q;
            const bool valid = r < at.TH && q < b.NB;
            const long long line = (long long)(at.d0 + pl) * b.H + at.h0 + r;
            uint4 zr[SC];
#pragma unroll
            for (int j = 0; j < SC; ++j) {
                zr[j] = make_uint4(0u, 0u, 0u, 0u);
                if (valid) zr[j] = load8<AL>(zb + j * b.SP + line * b.W, w, b.W);
            }
            ok = mbar_wait(full + 8 * buf, (it / BUFS) & 1);
            tc_fence_after();
            const unsigned d = tmem + ((unsigned)(warp & 3) << 21) + buf * 2 * NCOL;   // lane in bits 16+: 32 lanes per warp
#pragma unroll
            for (int j = 0; j < SC; ++j) {
                float n[8], dn[8], o[8];
                __syncwarp();
                tmem_load8x2(d + 8 * j, d + NCOL + 8 * j, n, dn);
                if (j == SC - 1) {                       // the accumulators are free again
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty + 8 * buf);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float s = word_lane(zr[j], i) + bj[j];
                    if (b.relu) s = fmaxf(s, 0.0f);
                    o[i] = dw4::fast_div(s * (n[i] + b.eps), dn[i] + b.eps);
                }
                if (valid) {
                    const uint4 v = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
                    bf16* orow = ob + j * osp + line * b.Wo;
                    if (AL != kPaddedOut || b.Wo == b.W) store8<AL>(orow, w, b.W, v);
                    else {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (w + i < b.Wv) {
                                const unsigned u = i < 2 ? v.x : i < 4 ? v.y : i < 6 ? v.z : v.w;
                                reinterpret_cast<unsigned short*>(orow)[w + i] = (unsigned short)(i & 1 ? u >> 16 : u);
                            }
                    }
                }
            }
        }
    }
    if (!ok && lane == 0) atomicExch(&g_wait_expired, 1u);
    tc_fence_before();
    __syncthreads();
    if (warp == 8) tmem_free(tmem, TCOLS);
}

// ---- t1 = K(relu(z + b)) ------------------------------------------------------------------------
struct SourceArgs {
    Band b;
    const bf16* z; bf16* t1;
    const float* h; const float* bias;
};

// Accumulator columns.  Volumes: a source plane p is multiplied once per (channel, kh) by the banded
// matrices of its KD = 3 depth taps side by side (24 columns, 8 of zeros: N is a multiple of 16), onto
// the accumulators of output planes p, p - 1, p - 2 of the chunk, which lie 8 columns apart: 12 MMAs a
// plane where one per tap would be 36.  All accumulators start at zero.  Images: N = 16 with 8
// columns of zeros, one MMA per (channel, kh).
template <int KD> __host__ __device__ constexpr int source_cols(int DC) { return KD > 1 ? 8 * (DC + KD + 2) : 16; }
inline int tmem_cols(int n) { int c = 32; while (c < n) c *= 2; return c; }

template <int KD, int KH, int KW, int AL>
__global__ void __launch_bounds__(kThreads, 2) tc_source_kernel(const SourceArgs P, int tcols) {
    constexpr int PD = KD / 2, PH = KH / 2, PW = KW / 2, KT = KD * KH * KW;
    constexpr int NCOL = KD > 1 ? 32 : 16, NMAT = SC * KH, MAXSTEP = 24;
    constexpr int TABLE = (PD + 1) * (PD + 1) * (PH + 1) * (PH + 1) * (PW + 1) * (PW + 1);
    extern __shared__ __align__(128) unsigned char smem_tc[];
    const Band& b = P.b;
    const At at(b, blockIdx.x);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned base = smem_u32(smem_tc), slot = base + 8 * MAXSTEP;
    float* const table = reinterpret_cast<float*>(smem_tc + kHeader);
    bf16* const bmat = reinterpret_cast<bf16*>(smem_tc + kHeader + (TABLE * 4 + 127) / 128 * 128);
    uint4* const zs = reinterpret_cast<uint4*>(bmat + NMAT * NCOL * 16);
    const int blocks = band_blocks<KD, KH>(b), slack = slack_blocks(b);
    const int plane = (b.TH + KH - 1) * b.PB, used = (at.DC + KD - 1) * plane;
    const int steps = KD > 1 ? at.DC + KD - 1 : b.MT;
    const int mcols = source_cols<KD>(b.DC);

    if (warp == 8) tmem_alloc(slot, tcols);
    if (tid == 0) {
        for (int i = 0; i < steps; ++i) mbar_init(base + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        float* const hs = reinterpret_cast<float*>(smem_tc + 256);
        for (int e = lane; e < SC * KT; e += 32) hs[e] = P.h[(long long)at.c * SC * KT + e];
        float bj[SC];
#pragma unroll
        for (int j = 0; j < SC; ++j) bj[j] = P.bias ? P.bias[at.c * SC + j] : 0.0f;
        __syncwarp();
        // column group g: output plane p - kd, kd = KD - 1 - g
        build_bands<NCOL, KW, false>(bmat, NMAT, lane, [&](int t, int n, int kw) {
            const int j = t / KH, kh = t % KH, kd = KD - 1 - n / 8;
            return kd >= 0 ? hs[j * KT + (kd * KH + kh) * KW + kw] : 0.0f;
        });
        // sum over channels and the taps inside the volume of bias * filter, by how many taps are cut
        // off at either end of each axis
        for (int e = lane; e < TABLE; e += 32) {
            int q = e;
            const int wh = q % (PW + 1); q /= PW + 1;
            const int wl = q % (PW + 1); q /= PW + 1;
            const int hh = q % (PH + 1); q /= PH + 1;
            const int hl = q % (PH + 1); q /= PH + 1;
            const int dh = q % (PD + 1), dl = q / (PD + 1);
            float s = 0.0f;
            for (int kd = dl; kd < KD - dh; ++kd)
                for (int kh = hl; kh < KH - hh; ++kh)
                    for (int kw = wl; kw < KW - wh; ++kw) {
                        const int tau = (kd * KH + kh) * KW + kw;
#pragma unroll
                        for (int j = 0; j < SC; ++j) s = fmaf(bj[j], hs[j * KT + tau], s);
                    }
            table[e] = s;
        }
    } else {
        unsigned negb[SC];
#pragma unroll
        for (int j = 0; j < SC; ++j) {
            const __nv_bfloat162 nb = __float2bfloat162_rn(P.bias ? -P.bias[at.c * SC + j] : 0.0f);
            negb[j] = *reinterpret_cast<const unsigned*>(&nb);
        }
        stage<KD, KH, KW, SC, true, AL == kWide>(zs, blocks, P.z + (long long)at.bc * SC * b.SP, b.SP, b, at, negb, b.relu);
    }
    for (int i = tid; i < slack; i += kThreads) zs[SC * blocks + i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < SC && at.DC < b.DC) zs[tid * blocks + used] = make_uint4(0u, 0u, 0u, 0u);
    fence_async_proxy();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *reinterpret_cast<volatile unsigned*>(smem_tc + 8 * MAXSTEP);
    const unsigned lanes = (unsigned)(warp & 3) << 21;
    if (KD > 1) {
        if (warp < 8) {
            for (int c = 8 * (warp >> 2); c < b.MT * mcols; c += 16) tmem_zero8(tmem + lanes + c);
            tmem_wait_st();
            tc_fence_before();
        }
        __syncthreads();
        tc_fence_after();
    }
    bool ok = true;
    if (warp == 8) {
        if (lane == 0) {
            const unsigned idesc = instr_desc(NCOL);
            const unsigned za = smem_u32(zs), ba = smem_u32(bmat);
            for (int step = 0; step < steps; ++step) {
                const int mt0 = KD > 1 ? 0 : step, mt1 = KD > 1 ? b.MT : step + 1, p = KD > 1 ? step : 0;
                for (int mt = mt0; mt < mt1; ++mt)
                    for (int t = 0; t < NMAT; ++t) {
                        const int j = t / KH, kh = t - j * KH;
                        mma(tmem + mt * mcols + 8 * p, mat_desc(za + 16 * (j * blocks + p * plane + kh * b.PB + mt * MB), 16, 128),
                            mat_desc(ba + t * NCOL * 32, 128, 256), idesc, KD > 1 || t > 0);
                    }
                mma_commit(base + 8 * step);
            }
        }
    } else {
        const int grp = warp >> 2, m = (warp & 3) * 32 + lane;
        bf16* const tb = P.t1 + (long long)at.bc * b.SP;
        const int items = at.DC * b.MT;
        // item: output plane pl of MMA tile mt; complete after source plane pl + KD - 1 (volumes)
        for (int it = grp; it < items && ok; it += 2) {
            const int pl = it / b.MT, mt = it - pl * b.MT;
            const int blk = mt * MB + m, r = blk / b.PB, q = blk - r * b.PB, w = 8 * q;
            const bool valid = r < at.TH && q < b.NB;
            const int d = at.d0 + pl, h = at.h0 + r;
            const int dl = max(0, PD - d), dh = max(0, d + PD - (b.D - 1)), hl = max(0, PH - h), hh = min(PH, max(0, h + PH - (b.H - 1)));
            const float* tab = table + (((dl * (PD + 1) + dh) * (PH + 1) + hl) * (PH + 1) + hh) * (PW + 1) * (PW + 1);
            ok = mbar_wait(base + 8 * (KD > 1 ? pl + KD - 1 : mt), 0);
            tc_fence_after();
            __syncwarp();
            float o[8];
            tmem_load8(tmem + lanes + mt * mcols + 8 * (KD > 1 ? pl + KD - 1 : 0), o);
            if (valid) {
                const bool inner = w >= PW && w + 7 + PW < b.Wv;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    int cut = 0;
                    if (!inner) cut = max(0, PW - w - i) * (PW + 1) + min(PW, max(0, w + i + PW - (b.Wv - 1)));
                    o[i] += tab[cut];
                    if (!inner && w + i >= b.Wv) o[i] = 0.0f;
                }
                store8<AL>(tb + ((long long)d * b.H + h) * b.W, w, b.W,
                           make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7])));
            }
        }
    }
    if (!ok && lane == 0) atomicExch(&g_wait_expired, 1u);
    tc_fence_before();
    __syncthreads();
    if (warp == 8) tmem_free(tmem, tcols);
}

}  // namespace tc
}  // namespace ndc
