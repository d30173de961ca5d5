// The forward update of bfloat16 tensors on the 5th-generation tensor cores (m = 1, sc = 4; 3x3x3,
// 5x5 and 3x3 kernels), where the filter and the bias are bfloat16 values too, as in a bfloat16
// module.  Two launches: tc_source_kernel (t1 = K(relu(z + b))) and tc_adjoint_kernel (out).  The latter is
// the ratio step of the backward too (gnum, gden and the direct term, see AdjointMode).
//
// A depthwise convolution as a matrix product.  Rows of a plane lie in shared memory one after the
// other as bfloat16, in blocks of 8 columns; one M = 128, K = 16 MMA multiplies 128 blocks of a source plane
// (1024 voxels) by one filter row of every depth tap, laid out as banded matrices side by side, onto the
// accumulators of KD output planes, which lie next to each other in TMEM.  So a source plane is read
// once, when the CTA's march through the depth comes to it, and a filter row kh is a shift of the start
// address.  Batches of images march down their rows the same way (planes = image rows, plane rows =
// images, KH = 1: see SlabAddr); no filter row takes a row of their bands to another, so a band takes any of them, of
// several chunks at once (see At), and fills its 128 blocks whatever the batch.  An MMA of N columns takes 32 + N / 4
// cycles here, N / 2 from 128 on (measured; its A operand is 4 KB), and a thread whose descriptors change issues one
// every 80, hence the wide ones.  With KW = 3 most of the products meet a zero of the
// band; the tensor cores do them 30 times faster than the FMA pipe does the useful ones.  What K = 16
// holds differs:
//
//   A (tc_adjoint_kernel): the window of 16 places that starts at a block, column w at place w + PW of
//     its row, zeros between the rows.  No copy of that is made: in the K-major layout without
//     swizzle (8-row groups of 16-byte rows) it is the memory as it lies, with 16 bytes between the two halves
//     of the window and 128 bytes between groups of eight blocks; a row takes a whole number PB of blocks.
//     Window place k, output column o of the block:     B[k][8 j + o] = h[j][kd][kh][o + 2 PW - k]
//
//   K (tc_source_kernel): the source of a block as the sum of two bfloat16 terms, eight places each (next
//     paragraph).  There is no room for the neighbouring columns, so the band is wider instead: a
//     block gives 8 columns of its own and PW of either neighbour's, which the epilogue adds.
//     Place k of either term, output column o = -PW .. 7 + PW:      B[k][o] = h[j][kd][kh][k - o + PW]
//
// Precision: every product is one of two bfloat16 values, exact in float32, accumulated in float32:
// what the FMA kernels compute, in another order.  The source s = relu(z + b) is not a bfloat16 value, but
// with L = 1 where z + b > 0, else 0, s = L z + L b, two of them; where everything is rectified away
// both are zero and t1 is zero, as it is with the FMA kernels, and of nearly equal z and -b the
// products meet in one MMA.  (max(z, -b) and a table of b K(1) would be one term, but leave the rounding of
// sums that cancel: with 2 % of the sources positive t1 was off by up to 6.6 times its value, and where
// everything is rectified away it was a residue of either sign.  As it is, t1 is off by 2^-8 of itself at
// most, its rounding to bfloat16, like the FMA kernels'.)
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
    int TH, nth, DC, ndc;         // rows and bands, planes and chunks (KH = 1: bands of rows of all chunks)
    int items;                    // places of work (see Items)
    int march;                    // CTAs that have several, one after the other
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
// Waits for the phase to complete, one thread or all of a warp; gives up (false, in all of them) after
// `limit` nanoseconds.  A second is far above any MMA's time.
constexpr unsigned kWaitLimit = 1000000000u;
__device__ __forceinline__ bool mbar_wait_thread(unsigned bar, unsigned phase, unsigned limit) {
    unsigned long long start = 0;
    for (;;) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(phase), "r"(1000000u) : "memory");   // asleep for up to 1 ms
        if (done) return true;
        unsigned long long now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (!start) start = now;
        if (now - start > limit) return false;
    }
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned phase, unsigned limit = kWaitLimit) {
    return __all_sync(0xffffffffu, mbar_wait_thread(bar, phase, limit));
}
// A wait ran out: the launch's results are undefined.  `flag` is host memory that the host looks at before
// the next call (see ndc_tc.cu).
__device__ __forceinline__ void report_expired(unsigned* flag) {
    asm volatile("st.release.sys.global.u32 [%0], 1;" ::"l"(flag) : "memory");
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
// Eight columns each of two accumulators of this thread's lane; the wait is part of the statement, so that
// nothing that uses the values can move in between.
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
// Eight columns, and the N that follow them.
template <int N>
__device__ __forceinline__ void tmem_load_group(unsigned addr, float (&v)[8], float (&n)[N]) {
    static_assert(N == 2 || N == 4, "columns");
    unsigned r[8], e[4];
    if (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%10];\n\t"
                     "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%8,%9}, [%11];\n\ttcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(e[0]), "=r"(e[1])
                     : "r"(addr), "r"(addr + 8) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%12];\n\t"
                     "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%13];\n\ttcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(e[0]), "=r"(e[1]),
                       "=r"(e[2]), "=r"(e[3])
                     : "r"(addr), "r"(addr + 8) : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) n[i] = __uint_as_float(e[i]);
}
// `n` columns (a multiple of 8) of this thread's lane; eight at a time, since every column takes a register
__device__ __forceinline__ void tmem_fill(unsigned addr, float v, int n) {
#pragma unroll 4
    for (int i = 0; i < n; i += 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(addr + i), "r"(__float_as_uint(v)) : "memory");
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
// Roles of a CTA's warps: groups of four for the epilogue (they take turns, output plane by output
// plane; TMEM lane 32 i + l belongs to lane l of warp i of a group), groups that stage source planes (in
// turns as well), one warp that issues the MMAs.  The source kernel, whose epilogue is short and whose
// source planes have four channels, has one epilogue group and stages with two groups of five warps.  The
// adjoint kernel: two and two groups of two warps, two CTAs per multiprocessor; with five depth taps, whose
// accumulators leave room for one, four and four.  (Two CTAs of two channels each, 16 x 64 images of 128^2, 5x5: 203 us
// for the forward's 211, but 4 x 64 of them 78 for 71.)
constexpr int kSourceThreads = 32 * (4 + 10 + 1), kSourceStagers = 160, kSourceCtas = 2;
template <int KD> struct AdjointShape {
    static constexpr int EPI = KD > 3 ? 4 : 2, GROUPS = KD > 3 ? 4 : 2, STAGERS = 64, BLOCKS = KD > 3 ? 2 : 3;
    static constexpr int THREADS = 32 * (4 * EPI + 2 * GROUPS + 1), CTAS = KD > 3 ? 1 : 2;
};
constexpr int kSlots = 8;         // staged planes
constexpr int kSourceSlots = 4;   // of the source kernel, which stages two terms of four channels
constexpr int kHeader = 1024;     // bytes: barriers and the TMEM address (512), the filter as float32

// Place of a CTA: (sample, channel), band of rows, chunk of planes; all addresses in elements.
// ROWS: row v of the band is image v % H of chunk v / H, and its planes count from the chunk's first one; `d0` is 0.
// (Bands of the images of one chunk left blocks idle: 16 images of 128 columns fill 7 + 7 + 2 of the adjoint's
// rows, 16 of 64 columns 14 + 2.)
template <bool ROWS>
struct At {
    int bc, c, h0, TH, d0, DC;
    __device__ __forceinline__ At(const Band& b, int blk) {
        const int th = blk % b.nth; blk /= b.nth;
        const int dc = ROWS ? 0 : blk % b.ndc;
        if (!ROWS) blk /= b.ndc;
        bc = blk; c = bc % b.C;
        h0 = th * b.TH; TH = min(b.TH, (ROWS ? b.H * b.ndc : b.H) - h0);
        d0 = dc * b.DC; DC = min(b.DC, b.D - d0);
    }
};
// ROWS: the image that the 32-bit offsets of a band that begins at row h0 count from.  (Bands of several chunks jump
// back to the first image; the host sees to it that the offsets fit.)
__device__ __forceinline__ long long base_row(const Band& b, int h0) { return b.ndc == 1 ? h0 : 0; }
// The places of a CTA: its own, or (MARCH) a contiguous share of all, one after the other without emptying the pipeline
// in between; their channel (and with it the banded matrices) seldom changes.
template <bool MARCH>
struct Items {
    int first, last;               // [first, last)
    __device__ __forceinline__ Items(const Band& b) {
        first = MARCH ? (int)((long long)b.items * blockIdx.x / gridDim.x) : blockIdx.x;
        last = MARCH ? (int)((long long)b.items * (blockIdx.x + 1) / gridDim.x) : first + 1;
    }
};

// Where row h of a plane lies: its offset, and for ROWS the first plane of its chunk (else 0).
template <bool ROWS>
struct RowAt {
    long long off;
    int d;
    __device__ __forceinline__ RowAt(const Band& b, int h, long long row_stride, long long plane) {
        const int chunk = ROWS ? h / b.H : 0;
        d = chunk * b.DC;
        off = (h - chunk * b.H) * row_stride + d * plane;
    }
};

// Columns w-2 .. w+7 of a global row as five words, w = 8 q at `p[off]`; zero outside the row of W.
template <bool WIDE, typename Offset>
__device__ __forceinline__ void load_words(const bf16* p, Offset off, int w, int W, unsigned (&a)[5]) {
#pragma unroll
    for (int i = 0; i < 5; ++i) a[i] = 0u;
    if (w > 0 && w - 4 < W) a[0] = __ldg(reinterpret_cast<const unsigned*>(p + (off - (Offset)2)));
    if (WIDE) {
        if (w < W) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + off));
            a[1] = v.x; a[2] = v.y; a[3] = v.z; a[4] = v.w;
        }
    } else {
        if (w < W) { const uint2 v = __ldg(reinterpret_cast<const uint2*>(p + off)); a[1] = v.x; a[2] = v.y; }
        if (w + 4 < W) { const uint2 v = __ldg(reinterpret_cast<const uint2*>(p + (off + (Offset)4))); a[3] = v.x; a[4] = v.y; }
    }
}
// The eight places of block q of a shared row (columns 8 q - PW .. 8 q + 7 - PW) from those words.
template <int PW>
__device__ __forceinline__ uint4 to_places(const unsigned (&a)[5]) {
    if (PW == 2) return make_uint4(a[0], a[1], a[2], a[3]);
    return make_uint4(__funnelshift_l(a[0], a[1], 16), __funnelshift_l(a[1], a[2], 16), __funnelshift_l(a[2], a[3], 16),
                      __funnelshift_l(a[3], a[4], 16));
}

// A group's planes of a chunk: p counts source planes from d0 - PD, `base` those of the places before; planes
// outside the volume are passed on without data.  `S`: load, prefetch and store a plane; `again`: set where one of its
// values is not finite (see look()).
template <int SLOTS, int GROUPS, bool ROWS, typename S, typename F>
__device__ __forceinline__ bool stage_planes(S& st, F store, int D, int d0, int PD, int planes, int base, unsigned full, unsigned empty, int group,
                                             int lane, volatile unsigned* again) {
    // those inside; the stager knows which rows of several chunks are
    const int first = ROWS ? 0 : max(0, PD - d0), last = ROWS ? planes - 1 : min(planes - 1, D - 1 + PD - d0);
    const int begin = (group - base % GROUPS + GROUPS) % GROUPS;
    if (begin >= first && begin <= last) st.load(d0 - PD + begin);
    for (int p = begin; p < planes; p += GROUPS) {
        const int s = (base + p) % SLOTS, use = (base + p) / SLOTS;
        if (use && !mbar_wait(empty + 8 * s, (use - 1) & 1)) return false;
        if (p >= first && p <= last) {
            if (store(s)) *again = 1u;
            fence_async_proxy();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * s);
        if (p + GROUPS >= first && p + GROUPS <= last) st.load(d0 - PD + p + GROUPS);
        if (p + 2 * GROUPS <= last) st.prefetch(d0 - PD + p + 2 * GROUPS);
    }
    return true;
}

// Infinities and NaN.  A zero of the band times one of them is NaN, and a window reaches into its row's next block and, past
// its last one, into the next row's: what the taps never see would become NaN, in another image too.  So a CTA that has met
// one computes what became NaN once more after its march, tap by tap on the FMA pipe (adjoint_again, source_again).  The
// adjoint's stagers look at what they stage, which costs up to 2 % of it; the source kernel looks at what it stores, one
// channel for the four that it stages, which costs nothing measurable (its stagers' look 2 %).  Where no value is finite
// the forward takes 7.0 ms at 2 x 64 x 64^3, not 0.31.
// (A block of zeros between the rows would keep images apart, and NaN spread over blocks of eight columns all the same.)
// Not zero where one of the eight values is not finite.
__device__ __forceinline__ unsigned look(const uint4& v) {
    unsigned seen = 0u;
    asm("fma.rn.bf16x2 %0, %1, %5, %0;\n\tfma.rn.bf16x2 %0, %2, %5, %0;\n\tfma.rn.bf16x2 %0, %3, %5, %0;\n\tfma.rn.bf16x2 %0, %4, %5, %0;"
        : "+r"(seen) : "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(0u));
    return seen;
}

// Stages planes of NCH channels (`src + ch * stride`), halo rows included; rows outside the volume are
// zero.  A thread of a group of NTHR has up to U blocks of a plane, and the loads of its group's next plane
// are on their way in registers while it waits for a slot; the lines of the one after are asked for
// from L2.  Addresses are a base that is the same for the whole CTA and a 32-bit offset.
template <int KH, int KW, int NCH, bool WIDE, int NTHR, int U>
struct Stager {
    static constexpr bool ROWS = KH == 1;
    const Band& b;
    const bf16* src;               // row h0 - KH / 2 of plane 0 (ROWS: see base_row)
    long long stride, plane;
    int blocks;                    // per channel of a slot
    unsigned off[U];               // this thread's blocks: offset of the first column
    unsigned in;                   // bit u: inside the volume (else zero)
    int w[U], own;                 // columns; the first block
    int d0[U];                     // ROWS: first plane of the row's chunk
    unsigned a[U][NCH][5];

    __device__ __forceinline__ Stager(const Band& b_, const bf16* src_, long long stride_, long long plane_, long long row_stride, const At<ROWS>& place,
                                      int tid)
        : b(b_), src(src_ + (ROWS ? base_row(b_, place.h0) : place.h0 - KH / 2) * row_stride), stride(stride_), plane(plane_), blocks((b_.TH + KH - 1) * b_.PB),
          in(0u), own(tid) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = tid + u * NTHR, row = i / b.PB, q = i - row * b.PB, h = place.h0 - KH / 2 + row;
            w[u] = 8 * q;
            if (ROWS) {
                const RowAt<ROWS> r(b, h, row_stride, plane);
                d0[u] = r.d;
                off[u] = (unsigned)(r.off - base_row(b, place.h0) * row_stride) + w[u];
                in |= (i < blocks && row < place.TH ? 1u : 0u) << u;
            } else {
                d0[u] = 0;
                off[u] = (unsigned)(row * row_stride) + w[u];
                in |= (i < blocks && h >= 0 && h < b.H ? 1u : 0u) << u;
            }
        }
    }
    __device__ __forceinline__ bool has(int u, int d) const { return (in >> u & 1) && (!ROWS || (unsigned)(d + d0[u]) < (unsigned)b.D); }
    __device__ __forceinline__ void load(int d) {
        const bf16* p = src + d * plane;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (has(u, d)) {
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) {
                    // a pointer per block and tensor, or a base and 32-bit offsets: rows that are not whole blocks
                    // make several loads of a pointer (64 x 5 images of 203x171, 3x3, forward: 257 -> 237 us)
                    if (ROWS && !WIDE) load_words<WIDE>(p + ch * stride + off[u], 0, w[u], b.W, a[u][ch]);
                    else load_words<WIDE>(p + ch * stride, off[u], w[u], b.W, a[u][ch]);
                }
            } else if (ROWS) {
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch)
#pragma unroll
                    for (int i = 0; i < 5; ++i) a[u][ch][i] = 0u;
            }
        }
    }
    __device__ __forceinline__ void prefetch(int d) const {
        const bf16* p = src + d * plane;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (has(u, d) && (w[u] & 63) == 0 && w[u] < b.W) {
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + ch * stride + off[u]));
            }
    }
    __device__ __forceinline__ unsigned store(uint4* dst) {
        unsigned seen = 0u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = own + u * NTHR;
            if (i >= blocks) continue;
#pragma unroll
            for (int ch = 0; ch < NCH; ++ch) {
                const uint4 v = in >> u & 1 ? to_places<KW / 2>(a[u][ch]) : make_uint4(0u, 0u, 0u, 0u);
                dst[ch * blocks + i] = v;
                seen |= look(v);
            }
        }
        return seen;
    }
};

// Blocks an MMA may read past the last staged row of a slot's last channel: 128 windows of two blocks
// from the band's first row on (the source kernel: of one).
__host__ __device__ inline int slack_blocks(const Band& b) { return MB + 1 - b.TH * b.PB > 1 ? MB + 1 - b.TH * b.PB : 1; }

// ---- two-lane float32 -------------------------------------------------------------------------
using dw4::f32x2;
using dw4::pack2;
using dw4::unpack2;
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ unsigned word_of(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }  // i static

// The banded matrices of a kernel: `value(t, n, k)` is what place k of matrix t, column n is multiplied by.
// Layout of one matrix: groups of eight columns, then the two halves of K, eight 16-byte rows each.
// Done by the `threads` threads of a group of stagers, of which this is number `tid`.
template <int NCOL, typename F>
__device__ __forceinline__ void build_bands(bf16* bmat, int mats, int tid, int threads, F value) {
    for (int e = tid; e < mats * NCOL * 2; e += threads) {
        const int n = e % 8, half = (e / 8) % 2, g = (e / 16) % (NCOL / 8), t = e / (2 * NCOL);
        unsigned words[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(value(t, 8 * g + n, 8 * half + 2 * i), value(t, 8 * g + n, 8 * half + 2 * i + 1));
            words[i] = *reinterpret_cast<const unsigned*>(&p);
        }
        reinterpret_cast<uint4*>(bmat)[e] = make_uint4(words[0], words[1], words[2], words[3]);
    }
}

// whole blocks of 16 bytes (no padding); 8-byte rows; 8-byte rows, out unpadded
enum Access { kWide = 0, kQuad = 1, kPaddedOut = 2 };

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

// 32 bytes of consecutive float32 values, on a 32-byte boundary
__device__ __forceinline__ void store_f32x8(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
                 "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])) : "memory");
}

// ---- A(x) and A(t1), and what follows from them -------------------------------------------------
//   kOut       out = s (A(x) + eps) / (A(t1) + eps)                          (the forward)
//   kPairs     (gden, gnum) pairs and the direct term of the backward of volumes, see ratio_kernel
//   kPlanar    the same as two tensors, for images
enum AdjointMode { kOut = 0, kPairs = 1, kPlanar = 2 };

struct AdjointArgs {
    Band b;
    const bf16* x; const bf16* t1; const bf16* z;
    bf16* out;                        // kOut: out; else the direct term (rows of W), or NULL
    const bf16* gout; float* gnum; float* gden;
    const float* h; const float* bias;
    unsigned* expired;                // see report_expired
};

// Accumulators: per output plane 32 columns of A(x) and 32 of A(t1) (four channels of eight voxels),
// RING of them in turn, which start at eps: the epilogue leaves them so.  Three depth taps: a ring of four planes, 256
// columns, two CTAs per multiprocessor; five: eight planes, all 512.
template <int KD> __host__ __device__ constexpr int adjoint_ring() { return KD > 3 ? 8 : 4; }

// What became NaN of a place's outputs (out; gden where any of the three did) tap by tap (see look()), by all threads of the
// CTA.  A function of its own: inline, it costs the kernel's loops registers.
template <int KD, int KH, int KW, int MODE>
__device__ __noinline__ void adjoint_again(const AdjointArgs& P, int item) {
    constexpr bool ROWS = KH == 1;
    constexpr int PD = KD / 2, PH = KH / 2, PW = KW / 2, KT = KD * KH * KW;
    const Band& b = P.b;
    const At<ROWS> at(b, item);
    const dw4::SlabAddr<ROWS> addr(b.C, b.D, b.H, b.W), oaddr(b.C, b.D, b.H, b.Wo);
    const float* const hc = P.h + (long long)at.c * SC * KT;
#pragma unroll 1
    for (int o = 0; o < at.DC; ++o)
#pragma unroll 1
        for (int e = threadIdx.x; e < at.TH * b.Wv; e += blockDim.x) {
            const int r = e / b.Wv, w = e - r * b.Wv, h = at.h0 + r;
            const RowAt<ROWS> xat(b, h, addr.row_x, addr.plane), zat(b, h, addr.row_z, addr.plane), oat(b, h, oaddr.row_z, oaddr.plane);
            const int d = at.d0 + o;                 // from the row's chunk on
            if (d + xat.d >= b.D) continue;
            const long long ze0 = (long long)at.bc * SC * addr.chan + zat.off + d * addr.plane + w;
            const long long oe0 = (long long)at.bc * SC * oaddr.chan + oat.off + d * oaddr.plane + w;
            bool nan = false;
#pragma unroll
            for (int j = 0; j < SC; ++j) {
                const long long ze = ze0 + j * addr.chan;
                nan |= isnan(MODE == kOut ? to_f32(P.out[oe0 + j * oaddr.chan]) : MODE == kPairs ? P.gnum[2 * ze] : P.gden[ze]);
            }
            if (!nan) continue;
            float n[SC], dn[SC];
#pragma unroll
            for (int j = 0; j < SC; ++j) n[j] = dn[j] = b.eps;
            const long long row = (long long)at.bc * addr.chan + xat.off + w + PW;
#pragma unroll 1
            for (int t = 0; t < KT; t += KW) {
                const int kh = t / KW % KH, kd = t / (KW * KH), dd = d + PD - kd, hh = h + PH - kh;
                if ((unsigned)(dd + xat.d) >= (unsigned)b.D || (!ROWS && (unsigned)hh >= (unsigned)b.H)) continue;
                const long long off = row + dd * addr.plane + (PH - kh) * addr.row_x;
#pragma unroll
                for (int kw = 0; kw < KW; ++kw) {
                    const bool here = (unsigned)(w + PW - kw) < (unsigned)b.Wv;
                    const float xv = here ? to_f32(P.x[off - kw]) : 0.0f, tv = here ? to_f32(P.t1[off - kw]) : 0.0f;
#pragma unroll
                    for (int j = 0; j < SC; ++j) {
                        n[j] = fmaf(xv, hc[j * KT + t + kw], n[j]);
                        dn[j] = fmaf(tv, hc[j * KT + t + kw], dn[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < SC; ++j) {
                const long long ze = ze0 + j * addr.chan, oe = oe0 + j * oaddr.chan;
                float s = to_f32(P.z[ze]) + (P.bias ? P.bias[at.c * SC + j] : 0.0f);
                if (b.relu) s = fmaxf(s, 0.0f);
                const float rd = rcp(dn[j]);
                if (MODE == kOut) {
                    P.out[oe] = from_f32<bf16>(s * n[j] * rd);
                } else {
                    const float g = to_f32(P.gout[oe]) * rd, gn = g * s, gd = -(gn * n[j] * rd);
                    if (P.out) P.out[ze] = from_f32<bf16>(g * n[j]);
                    P.gnum[MODE == kPairs ? 2 * ze + 1 : ze] = gn;
                    if (MODE == kPairs) P.gnum[2 * ze] = gd; else P.gden[ze] = gd;
                }
            }
        }
}

template <int KD, int KH, int KW, int AL, int MODE, bool MARCH>
__global__ void __launch_bounds__(AdjointShape<KD>::THREADS, AdjointShape<KD>::CTAS) tc_adjoint_kernel(const __grid_constant__ AdjointArgs P) {
    constexpr bool ROWS = KH == 1;
    typedef AdjointShape<KD> Shape;
    constexpr int kThreads = Shape::THREADS, kEpilogueWarps = 4 * Shape::EPI, kMmaWarp = kThreads / 32 - 1;
    constexpr int PD = KD / 2, NC = SC * 8, RING = adjoint_ring<KD>(), TCOLS = RING * 2 * NC, KT = KD * KH * KW;
    extern __shared__ __align__(128) unsigned char smem_tc[];
    const Band& b = P.b;
    const Items<MARCH> items(b);
    const At<ROWS> first(b, items.first);
    const dw4::SlabAddr<ROWS> addr(b.C, b.D, b.H, b.W), oaddr(b.C, b.D, b.H, AL == kPaddedOut ? b.Wo : b.W);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned base = smem_u32(smem_tc);
    const unsigned sfull = base, sempty = base + 8 * kSlots, afull = base + 16 * kSlots, aempty = afull + 8 * RING;
    const unsigned bfull = aempty + 8 * RING, bfree = bfull + 8;      // the banded matrices are there; are no longer read
    constexpr int kTmemAt = 16 * kSlots + 16 * RING + 16;
    volatile unsigned* const again = reinterpret_cast<unsigned*>(smem_tc + kTmemAt + 4);      // see look()
    bf16* const bmat = reinterpret_cast<bf16*>(smem_tc + kHeader);
    uint4* const slots = reinterpret_cast<uint4*>(smem_tc + kHeader + KH * KD * NC * 32);
    const int blocks = (b.TH + KH - 1) * b.PB, slot_blocks = 2 * blocks;

    if (warp == kMmaWarp) tmem_alloc(base + kTmemAt, TCOLS);
    if (tid == 0) {
        for (int i = 0; i < kSlots; ++i) { mbar_init(sfull + 8 * i, Shape::STAGERS / 32); mbar_init(sempty + 8 * i, 1); }
        for (int i = 0; i < RING; ++i) { mbar_init(afull + 8 * i, 1); mbar_init(aempty + 8 * i, 4); }
        mbar_init(bfull, Shape::STAGERS / 32);
        mbar_init(bfree, 1);
        *again = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // windows of valid blocks may touch blocks that no plane has been staged to: those have to be numbers
    for (int i = tid; i < kSlots * slot_blocks + slack_blocks(b); i += kThreads) slots[i] = make_uint4(0u, 0u, 0u, 0u);
    // [kh][output plane p - (KD - 1) + kd: groups of 32 columns][channel, column]
    auto bands = [&](const float* h, int own, int threads) {
        build_bands<KD * NC>(bmat, KH, own, threads, [&](int kh, int n, int k) {
            const int kd = n / NC, j = n % NC / 8, kw = n % 8 + KW - 1 - k;
            return kw >= 0 && kw < KW ? h[j * KT + (kd * KH + kh) * KW + kw] : 0.0f;
        });
    };
    if (!MARCH) {
        float* const hs = reinterpret_cast<float*>(smem_tc + 512);
        for (int e = tid; e < SC * KT; e += kThreads) hs[e] = P.h[(long long)first.c * SC * KT + e];
        __syncthreads();
        bands(hs, tid, kThreads);
    }
    fence_async_proxy();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *reinterpret_cast<volatile unsigned*>(smem_tc + kTmemAt);
    if (warp < kEpilogueWarps) {
        for (int c = 32 * (warp >> 2); c < TCOLS; c += 32 * Shape::EPI) tmem_fill(tmem + ((unsigned)(warp & 3) << 21) + c, b.eps, 32);
        tmem_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    bool ok = true;
    if (warp == kMmaWarp) {
        const unsigned long long ad = mat_desc(smem_u32(slots), 16, 128), md = mat_desc(smem_u32(bmat), 128, 256);
        // base, out: planes and output planes of the places before
        auto place = [&](const At<ROWS>& at, int base, int out) {
            const int planes = at.DC + KD - 1;
            for (int p = 0; p < planes && ok && lane == 0; ++p) {
                const int s = (base + p) % kSlots, d = at.d0 - PD + p;
                ok = mbar_wait_thread(sfull + 8 * s, ((base + p) / kSlots) & 1, kWaitLimit);
                // a new output plane begins: its accumulators have been read and filled again
                const int begun = out + p;
                if (begun >= RING && p < at.DC) ok = mbar_wait_thread(aempty + 8 * (begun % RING), (begun / RING - 1) & 1, kWaitLimit) && ok;
                tc_fence_after();
                if (!ok) break;
                if (ROWS || (d >= 0 && d < b.D)) {
                    // groups g of output planes o = p - (KD - 1) + g inside the chunk
                    const int g0 = max(0, KD - 1 - p), g1 = min(KD - 1, at.DC - 1 + KD - 1 - p), o0 = p - (KD - 1) + g0;
                    const int r0 = (out + o0) % RING, n = g1 - g0 + 1, n0 = min(n, RING - r0);
                    // descriptors differ in their start address alone, in units of 16 bytes
                    const unsigned long long a0 = ad + s * slot_blocks, m0 = md + g0 * NC * 2;
                    const unsigned i0 = instr_desc(n0 * NC), i1 = instr_desc((n - n0) * NC);
#pragma unroll
                    for (int kh = 0; kh < KH; ++kh)
#pragma unroll
                        for (int a = 0; a < 2; ++a) {                            // x, t1
                            const unsigned long long ak = a0 + (KH - 1 - kh) * b.PB + a * blocks, mk = m0 + kh * KD * NC * 2;
                            mma(tmem + a * RING * NC + r0 * NC, ak, mk, i0, 1);
                            if (n > n0) mma(tmem + a * RING * NC, ak, mk + n0 * NC * 2, i1, 1);
                        }
                }
                mma_commit(sempty + 8 * s);
                const int o = p - (KD - 1);
                if (o >= 0) mma_commit(afull + 8 * ((out + o) % RING));
            }
        };
        if (MARCH) {
            int base = 0, out = 0, channel = -1, built = 0;
            for (int item = items.first; item < items.last && ok && lane == 0; ++item) {
                const At<ROWS> at(b, item);
                if (at.c != channel) {
                    if (channel >= 0) mma_commit(bfree);
                    channel = at.c;
                    ok = mbar_wait_thread(bfull, built++ & 1, kWaitLimit);
                }
                place(at, base, out);
                base += at.DC + KD - 1;
                out += at.DC;
            }
        } else {
            place(first, 0, 0);
        }
    } else if (warp >= kEpilogueWarps) {
        // x and t1 as two channels: the distance between the tensors takes the place of the stride
        const long long apart = ((long long)(uintptr_t)P.t1 - (long long)(uintptr_t)P.x) / 2;
        const int group = (tid - 32 * kEpilogueWarps) / Shape::STAGERS, own = (tid - 32 * kEpilogueWarps) % Shape::STAGERS;
        auto place = [&](const At<ROWS>& at, int base) {
            Stager<KH, KW, 2, AL == kWide, Shape::STAGERS, Shape::BLOCKS> st(b, P.x + (long long)at.bc * addr.chan, apart, addr.plane, addr.row_x, at, own);
            ok = stage_planes<kSlots, Shape::GROUPS, ROWS>(st, [&](int s) { return st.store(slots + s * slot_blocks); }, b.D, at.d0, PD, at.DC + KD - 1, base,
                                                           sfull, sempty, group, lane, again);
        };
        if (MARCH) {
            int base = 0, channel = -1, built = 0;
            for (int item = items.first; item < items.last && ok; ++item) {
                const At<ROWS> at(b, item);
                if (at.c != channel) {
                    channel = at.c;
                    if (group == 0) {      // always the same one: it sees every phase of the barrier
                        if (built) ok = mbar_wait(bfree, (built - 1) & 1);
                        bands(P.h + (long long)channel * SC * KT, own, Shape::STAGERS);
                        fence_async_proxy();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bfull);
                    }
                    ++built;
                }
                if (ok) place(at, base);
                base += at.DC + KD - 1;
            }
        } else {
            place(first, 0);
        }
    } else {
        const int m = (warp & 3) * 32 + lane, r = m / b.PB, q = m - r * b.PB, w = 8 * q;
        const unsigned lanes = tmem + ((unsigned)(warp & 3) << 21);
        auto place = [&](const At<ROWS>& at, int out) {
        const RowAt<ROWS> zat(b, at.h0 + r, addr.row_z, addr.plane), oat(b, at.h0 + r, oaddr.row_z, oaddr.plane);
        // this row's output planes in the march
        const int count = r < at.TH && q < b.NB ? (ROWS ? min(b.DC, b.D - zat.d) : at.DC) : 0;
        // as single values (as pairs for two-lane additions four registers more: forward 2.65 ms for 2.42 at 4 x 64 x 128^3); as pairs
        // in the volumes' ratio step, which spills with single ones (3 x 216 of 19x25x25: 178 us for 148)
        constexpr bool PAIRED = MODE == kPairs && KH > 1;
        float bj[SC];
        f32x2 b2[SC];
#pragma unroll
        for (int j = 0; j < SC; ++j) {
            bj[j] = P.bias ? P.bias[at.c * SC + j] : 0.0f;
            b2[j] = pack2(bj[j], bj[j]);
        }
        const long long zrow = (long long)at.bc * SC * addr.chan + zat.off;
        const long long orow = (long long)at.bc * SC * oaddr.chan + oat.off;
        const bf16* const zb = P.z + zrow;
        const bf16* const gb = MODE == kOut ? nullptr : P.gout + orow;
        for (int o = ((warp >> 2) - out % Shape::EPI + Shape::EPI) % Shape::EPI; o < at.DC && ok; o += Shape::EPI) {
            const int slot = (out + o) % RING;
            const long long d = at.d0 + o;
            const bool valid = o < count;
            // z of all channels, or z and gout of two (the registers do not hold more), are on their way
            // while the accumulators are waited for; their lines of this group's next plane come to L2
            // (one plane further ahead, in registers: 2.88 ms for 2.35 at 4 x 64 x 128^3, spills)
            constexpr int AHEAD = MODE == kOut ? SC : 2;
            uint4 zr[AHEAD], gr[AHEAD];
            auto fetch = [&](int j) {
                zr[j % AHEAD] = make_uint4(0u, 0u, 0u, 0u);
                gr[j % AHEAD] = make_uint4(0u, 0u, 0u, 0u);
                if (!valid) return;
                const bf16* zp = zb + j * addr.chan + d * addr.plane;
                const bool more = (q & 7) == 0 && o + Shape::EPI < count;
                zr[j % AHEAD] = load8<AL>(zp, w, b.W);
                if (more) asm volatile("prefetch.global.L2 [%0];" ::"l"(zp + Shape::EPI * addr.plane + w));
                if (MODE == kOut) return;
                if (more) asm volatile("prefetch.global.L2 [%0];" ::"l"(gb + j * oaddr.chan + (d + Shape::EPI) * oaddr.plane + w));
                const bf16* row = gb + j * oaddr.chan + d * oaddr.plane;
                if (AL != kPaddedOut || b.Wo == b.W) gr[j % AHEAD] = load8<AL>(row, w, b.W);
                else {
                    unsigned e[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) e[i] = w + i < b.Wv ? reinterpret_cast<const unsigned short*>(row)[w + i] : 0u;
                    gr[j % AHEAD] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
                }
            };
#pragma unroll
            for (int j = 0; j < AHEAD; ++j) fetch(j);
            ok = mbar_wait(afull + 8 * slot, ((out + o) / RING) & 1);
            tc_fence_after();
            const unsigned acc = lanes + slot * NC;
#pragma unroll
            for (int j = 0; j < SC; ++j) {
                float n[8], dn[8];
                __syncwarp();
                tmem_load8x2(acc + 8 * j, acc + RING * NC + 8 * j, n, dn);
                if (j == SC - 1) {                       // read: eps again for the plane that takes the place
                    tmem_fill(acc, b.eps, NC);
                    tmem_fill(acc + RING * NC, b.eps, NC);
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(aempty + 8 * slot);
                }
                unsigned v[4];
                float gd[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const unsigned u = word_of(zr[j % AHEAD], i);
                    float lo = __uint_as_float(u << 16), hi = __uint_as_float(u & 0xffff0000u);
                    if (PAIRED) unpack2(add2(pack2(lo, hi), b2[j]), lo, hi);
                    else { lo += bj[j]; hi += bj[j]; }
                    if (b.relu) { lo = fmaxf(lo, 0.0f); hi = fmaxf(hi, 0.0f); }
                    const f32x2 n2 = pack2(n[2 * i], n[2 * i + 1]), r2 = pack2(rcp(dn[2 * i]), rcp(dn[2 * i + 1]));
                    if (MODE == kOut) {
                        unpack2(mul2(mul2(pack2(lo, hi), n2), r2), lo, hi);
                    } else {
                        const unsigned q2 = word_of(gr[j % AHEAD], i);
                        const f32x2 g2 = mul2(pack2(__uint_as_float(q2 << 16), __uint_as_float(q2 & 0xffff0000u)), r2);
                        const f32x2 gn2 = mul2(g2, pack2(lo, hi));
                        float a, c;
                        unpack2(mul2(mul2(gn2, n2), r2), a, c);
                        gd[2 * i] = -a; gd[2 * i + 1] = -c;
                        unpack2(mul2(g2, n2), lo, hi);           // the direct term
                        unpack2(gn2, n[2 * i], n[2 * i + 1]);
                    }
                    v[i] = pack_bf16(lo, hi);
                }
                if (j + AHEAD < SC) fetch(j + AHEAD);
                if (MODE != kOut && w + 8 > b.Wv) {              // zero in the padding
#pragma unroll
                    for (int i = 0; i < 8; ++i) if (w + i >= b.Wv) { n[i] = 0.0f; gd[i] = 0.0f; }
                }
                if (valid && MODE == kOut) {
                    bf16* row = P.out + orow + j * oaddr.chan + d * oaddr.plane;
                    if (AL != kPaddedOut || b.Wo == b.W) store8<AL>(row, w, b.W, make_uint4(v[0], v[1], v[2], v[3]));
                    else {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (w + i < b.Wv) reinterpret_cast<unsigned short*>(row)[w + i] = (unsigned short)(i & 1 ? v[i / 2] >> 16 : v[i / 2]);
                    }
                } else if (valid) {
                    const long long e = zrow + j * addr.chan + d * addr.plane + w;
                    if (P.out) store8<AL>(P.out + e - w, w, b.W, make_uint4(v[0], v[1], v[2], v[3]));
                    const bool both = AL == kWide || w + 4 < b.W;
                    if (MODE == kPairs) {
                        const float lo8[8] = {gd[0], n[0], gd[1], n[1], gd[2], n[2], gd[3], n[3]};
                        const float hi8[8] = {gd[4], n[4], gd[5], n[5], gd[6], n[6], gd[7], n[7]};
                        store_f32x8(P.gnum + 2 * e, lo8);
                        if (both) store_f32x8(P.gnum + 2 * e + 8, hi8);
                    } else if (AL == kWide) {
                        store_f32x8(P.gnum + e, n);
                        store_f32x8(P.gden + e, gd);
                    } else {
                        *reinterpret_cast<float4*>(P.gnum + e) = make_float4(n[0], n[1], n[2], n[3]);
                        *reinterpret_cast<float4*>(P.gden + e) = make_float4(gd[0], gd[1], gd[2], gd[3]);
                        if (both) {
                            *reinterpret_cast<float4*>(P.gnum + e + 4) = make_float4(n[4], n[5], n[6], n[7]);
                            *reinterpret_cast<float4*>(P.gden + e + 4) = make_float4(gd[4], gd[5], gd[6], gd[7]);
                        }
                    }
                }
            }
        }
        };
        if (MARCH) {
            int out = 0;
            for (int item = items.first; item < items.last && ok; ++item) {
                const At<ROWS> at(b, item);
                place(at, out);
                out += at.DC;
            }
        } else {
            place(first, 0);
        }
    }
    if (!ok && lane == 0) report_expired(P.expired);
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == kMmaWarp) tmem_free(tmem, TCOLS);
    if (*again)
        for (int item = items.first; item < items.last; ++item) adjoint_again<KD, KH, KW, MODE>(P, item);
}

// ---- t1 = K(relu(z + b)) ------------------------------------------------------------------------
struct SourceArgs {
    Band b;
    const bf16* z; bf16* t1;
    const float* h; const float* bias;
    unsigned* expired;
};

// Accumulators: 16 columns per output plane, of which the block's own eight, PW of the left and PW of the
// right neighbour's; all 256 make a ring of P planes and KD - 1 more.  A source plane is multiplied once
// per (channel, kh), by the matrices of all depth taps at once: 12 MMAs of 48 columns for a 3x3x3 filter, 4 of
// 48 or 80 for an image filter.  Plane p of the march starts at ring place p % P and runs on over the
// ring's end, so that no MMA is split there: the sums of an output plane at one of the first KD - 1 places
// are then in two parts, P places apart, which the epilogue adds.
//
// What bounds the kernel: these MMAs, 12 x 44 cycles a plane and band at best (0.95 of 1.66 ms at 4 x 64 x 128^3), and the
// loads, of which two groups are in flight.  A block of places for each of two terms takes as many of them as a window of one
// term, and rows without zeros between them fill the 128 blocks better (16 rows of 64 columns, not 14), so
// that the exact form is the faster one too: the forward 4.66 -> 3.95 ms there, 368 -> 316 us at 2 x 64 x 64^3,
// 228 -> 181 on 16 x 64 images of 128^2, 5x5 (one term, chunks of up to 27 planes: before).
constexpr int kSourceCols = 256, kGroup = 16;
template <int KD> __host__ __device__ constexpr int source_ring() { return kSourceCols / kGroup - (KD - 1); }

// Stages the two terms of the source: per channel the blocks of L z, then those of L b.  A thread has one
// block of a plane; see Stager.
template <int KH, bool WIDE>
struct SourceStager {
    static constexpr bool ROWS = KH == 1;
    const Band& b;
    const bf16* src;
    long long stride, plane;
    int blocks;
    unsigned off;
    bool row_in, in;               // the row is the band's; and its plane is inside the volume
    int w, at, d0;
    uint4 a[SC];

    __device__ __forceinline__ SourceStager(const Band& b_, const bf16* src_, long long stride_, long long plane_, long long row_stride,
                                            const At<ROWS>& place, int i)
        : b(b_), src(src_ + (ROWS ? base_row(b_, place.h0) : place.h0 - KH / 2) * row_stride), stride(stride_), plane(plane_), blocks((b_.TH + KH - 1) * b_.NB) {
        const int row = i / b.NB, h = place.h0 - KH / 2 + row;
        at = i < blocks ? i : -1;
        w = 8 * (i - row * b.NB);
        if (ROWS) {
            const RowAt<ROWS> r(b, h, row_stride, plane);
            d0 = r.d;
            off = (unsigned)(r.off - base_row(b, place.h0) * row_stride) + w;
            row_in = i < blocks && row < place.TH;
        } else {
            d0 = 0;
            off = (unsigned)(row * row_stride) + w;
            row_in = i < blocks && h >= 0 && h < b.H;
        }
        in = row_in;
    }
    __device__ __forceinline__ void load(int d) {
        if (ROWS) in = row_in && (unsigned)(d + d0) < (unsigned)b.D;
        if (!in) return;
        const bf16* p = src + d * plane;
#pragma unroll
        for (int ch = 0; ch < SC; ++ch) a[ch] = load8<WIDE ? kWide : kQuad>(p + ch * stride + (off - w), w, b.W);
    }
    __device__ __forceinline__ void prefetch(int d) const {
        if (!row_in || (w & 63) || (ROWS && (unsigned)(d + d0) >= (unsigned)b.D)) return;
        const bf16* p = src + d * plane;
#pragma unroll
        for (int ch = 0; ch < SC; ++ch) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + ch * stride + off));
    }
    // `bias`: two copies of b per channel
    __device__ __forceinline__ void store(uint4* dst, const unsigned (&bias)[SC], bool relu) {
        if (at < 0) return;
#pragma unroll
        for (int ch = 0; ch < SC; ++ch) {
            unsigned z[4], c[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                z[i] = i == 0 ? a[ch].x : i == 1 ? a[ch].y : i == 2 ? a[ch].z : a[ch].w;
                const unsigned nb = bias[ch] ^ 0x80008000u;
                unsigned m = in ? 0xffffffffu : 0u;
                if (!WIDE) {
                    if (w + 2 * i >= b.Wv) m &= 0xffff0000u;
                    if (w + 2 * i + 1 >= b.Wv) m &= 0x0000ffffu;
                }
                if (relu) m &= __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&z[i]), *reinterpret_cast<const __nv_bfloat162*>(&nb));
                z[i] &= m;
                c[i] = bias[ch] & m;
            }
            dst[2 * ch * blocks + at] = make_uint4(z[0], z[1], z[2], z[3]);
            dst[(2 * ch + 1) * blocks + at] = make_uint4(c[0], c[1], c[2], c[3]);
        }
    }
};

// What became NaN of a place's t1 tap by tap (see look()), by all threads of the CTA.  Its arguments by value: their address,
// which a reference needs, costs the kernel 2 - 4 % (3 x 32 of 33x40x39: 34.5 us for 33.4; 2 x 64 x 64^3: 125.5 for 123.9).
template <int KD, int KH, int KW>
__device__ __noinline__ void source_again(const SourceArgs P, int item) {
    constexpr bool ROWS = KH == 1;
    constexpr int PD = KD / 2, PH = KH / 2, PW = KW / 2, KT = KD * KH * KW;
    const Band& b = P.b;
    const At<ROWS> at(b, item);
    const dw4::SlabAddr<ROWS> addr(b.C, b.D, b.H, b.W);
#pragma unroll 1
    for (int o = 0; o < at.DC; ++o)
#pragma unroll 1
        for (int e = threadIdx.x; e < at.TH * b.Wv; e += blockDim.x) {
            const int r = e / b.Wv, w = e - r * b.Wv, h = at.h0 + r;
            const RowAt<ROWS> xat(b, h, addr.row_x, addr.plane), zat(b, h, addr.row_z, addr.plane);
            const int d = at.d0 + o;                 // from the row's chunk on
            if (d + xat.d >= b.D) continue;
            bf16* const out = P.t1 + (long long)at.bc * addr.chan + xat.off + d * addr.plane + w;
            if (!isnan(to_f32(*out))) continue;
            const bf16* const zc = P.z + (long long)at.bc * SC * addr.chan + zat.off + w - PW;
            float sum = 0.0f;
#pragma unroll 1
            for (int t = 0; t < KT; t += KW) {
                const int kh = t / KW % KH, kd = t / (KW * KH), dd = d + kd - PD, hh = h + kh - PH;
                if ((unsigned)(dd + xat.d) >= (unsigned)b.D || (!ROWS && (unsigned)hh >= (unsigned)b.H)) continue;
                const long long off = dd * addr.plane + (kh - PH) * addr.row_z;
#pragma unroll
                for (int j = 0; j < SC; ++j) {
                    const float bj = P.bias ? P.bias[at.c * SC + j] : 0.0f;
#pragma unroll
                    for (int kw = 0; kw < KW; ++kw) {
                        if ((unsigned)(w + kw - PW) >= (unsigned)b.Wv) continue;
                        float s = to_f32(zc[j * addr.chan + off + kw]) + bj;
                        if (b.relu) s = fmaxf(s, 0.0f);
                        sum = fmaf(s, P.h[(long long)(at.c * SC + j) * KT + t + kw], sum);
                    }
                }
            }
            *out = from_f32<bf16>(sum);
        }
}

template <int KD, int KH, int KW, int AL>
__global__ void __launch_bounds__(kSourceThreads, kSourceCtas) tc_source_kernel(const SourceArgs P) {
    constexpr bool ROWS = KH == 1;
    constexpr int kThreads = kSourceThreads, kEpilogueWarps = 4, kMmaWarp = 14;
    constexpr int PD = KD / 2, PW = KW / 2, KT = KD * KH * KW, RING = source_ring<KD>();
    constexpr int NCOL = kGroup * KD, NMAT = SC * KH;
    extern __shared__ __align__(128) unsigned char smem_tc[];
    const Band& b = P.b;
    const At<ROWS> at(b, blockIdx.x);
    const dw4::SlabAddr<ROWS> addr(b.C, b.D, b.H, b.W);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned base = smem_u32(smem_tc);
    const unsigned sfull = base, sempty = sfull + 8 * kSourceSlots, afull = sempty + 8 * kSourceSlots, aempty = afull + 8 * RING,
                   edges = aempty + 8 * RING;
    constexpr int kEdgesAt = 320, kTmemAt = 504;
    static_assert(8 * (2 * kSourceSlots + 2 * RING + 1) <= kEdgesAt && kEdgesAt + 64 * PW <= kTmemAt, "header");
    volatile unsigned* const again = reinterpret_cast<unsigned*>(smem_tc + kTmemAt + 4);      // see look()
    float* const edge = reinterpret_cast<float*>(smem_tc + kEdgesAt);      // [parity][warp][side][PW]
    bf16* const bmat = reinterpret_cast<bf16*>(smem_tc + kHeader);
    uint4* const slots = reinterpret_cast<uint4*>(bmat + NMAT * NCOL * 16);
    const int blocks = (b.TH + KH - 1) * b.NB, slot_blocks = 2 * SC * blocks;
    const int planes = at.DC + KD - 1;

    if (warp == kMmaWarp) tmem_alloc(base + kTmemAt, kSourceCols);
    if (tid == 0) {
        for (int i = 0; i < kSourceSlots; ++i) { mbar_init(sfull + 8 * i, kSourceStagers / 32); mbar_init(sempty + 8 * i, 1); }
        for (int i = 0; i < RING; ++i) { mbar_init(afull + 8 * i, 1); mbar_init(aempty + 8 * i, kEpilogueWarps); }
        mbar_init(edges, kEpilogueWarps);
        *again = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    float* const hs = reinterpret_cast<float*>(smem_tc + 512);
    for (int e = tid; e < SC * KT; e += kThreads) hs[e] = P.h[(long long)at.c * SC * KT + e];
    __syncthreads();
    // [channel, kh][output plane p - kd, kd = KD - 1 - g: groups of 16 columns][own eight columns, left, right]
    build_bands<NCOL>(bmat, NMAT, tid, kThreads, [&](int t, int n, int k) {
        const int j = t / KH, kh = t % KH, kd = KD - 1 - n / kGroup, i = n % kGroup;
        const int o = i < 8 ? i : i < 8 + PW ? i - 8 - PW : i - PW, kw = k % 8 - o + PW;
        return i < 8 + 2 * PW && kw >= 0 && kw < KW ? hs[j * KT + (kd * KH + kh) * KW + kw] : 0.0f;
    });
    fence_async_proxy();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *reinterpret_cast<volatile unsigned*>(smem_tc + kTmemAt);
    if (warp < kEpilogueWarps) {
        for (int c = 0; c < kSourceCols; c += 32) tmem_fill(tmem + ((unsigned)(warp & 3) << 21) + c, 0.0f, 32);
        tmem_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    bool ok = true;
    if (warp == kMmaWarp) {
        const unsigned long long ad = mat_desc(smem_u32(slots), 16 * blocks, 128), md = mat_desc(smem_u32(bmat), 128, 256);
        for (int p = 0; p < planes && ok && lane == 0; ++p) {
            const int s = p % kSourceSlots, d = at.d0 - PD + p;
            ok = mbar_wait_thread(sfull + 8 * s, (p / kSourceSlots) & 1, kWaitLimit);
            // the ring place that this plane's last group begins anew has been read and zeroed
            if (p >= RING) ok = mbar_wait_thread(aempty + 8 * (p % RING), (p / RING - 1) & 1, kWaitLimit) && ok;
            tc_fence_after();
            if (ok) {
                if (ROWS || (d >= 0 && d < b.D)) {
                    const int g0 = max(0, KD - 1 - p);       // output planes of the chunk only
                    const unsigned long long a0 = ad + s * slot_blocks, m0 = md + g0 * kGroup * 2;
                    const unsigned idesc = instr_desc(NCOL - g0 * kGroup), acc = tmem + kGroup * (p % RING + g0);
#pragma unroll
                    for (int t = 0; t < NMAT; ++t)
                        mma(acc, a0 + 2 * (t / KH) * blocks + (t % KH) * b.NB, m0 + t * NCOL * 2, idesc, 1);
                }
                mma_commit(sempty + 8 * s);
                const int o = p - (KD - 1);
                if (o >= 0) mma_commit(afull + 8 * (o % RING));
            }
        }
    } else if (warp >= kEpilogueWarps) {
        unsigned bias[SC];
#pragma unroll
        for (int j = 0; j < SC; ++j) {
            const __nv_bfloat162 v = __float2bfloat162_rn(P.bias ? P.bias[at.c * SC + j] : 0.0f);
            bias[j] = *reinterpret_cast<const unsigned*>(&v);
        }
        SourceStager<KH, AL == kWide> st(b, P.z + (long long)at.bc * SC * addr.chan, addr.chan, addr.plane, addr.row_z, at,
                                         (tid - 32 * kEpilogueWarps) % kSourceStagers);
        ok = stage_planes<kSourceSlots, 2, ROWS>(st, [&](int s) { st.store(slots + s * slot_blocks, bias, b.relu); return 0u; }, b.D, at.d0, PD, planes, 0, sfull,
                                           sempty, (warp - kEpilogueWarps) / 5, lane, again);
    } else {
        const int m = warp * 32 + lane, r = m / b.NB, q = m - r * b.NB, w = 8 * q;
        const RowAt<ROWS> row(b, at.h0 + r, addr.row_x, addr.plane);
        const int count = r < at.TH ? (ROWS ? min(b.DC, b.D - row.d) : at.DC) : 0;      // this row's output planes in the march
        const bool left = q > 0, right = q + 1 < b.NB;
        const bool split = 32 % b.NB != 0;              // rows go on in another warp's lanes
        const unsigned lanes = tmem + ((unsigned)warp << 21);
        bf16* const tb = P.t1 + (long long)at.bc * addr.chan + row.off;
        for (int o = 0; o < at.DC && ok; ++o) {
            const int place = (o + KD - 1) % RING;
            ok = mbar_wait(afull + 8 * (o % RING), (o / RING) & 1);
            tc_fence_after();
            __syncwarp();
            float v[8], n[2 * PW];                       // its own columns; the left and the right neighbour's
            tmem_load_group<2 * PW>(lanes + kGroup * place, v, n);
            tmem_fill(lanes + kGroup * place, 0.0f, kGroup);
            if (place < KD - 1 && o + KD - 1 >= RING) {
                float v2[8], n2[2 * PW];
                tmem_load_group<2 * PW>(lanes + kGroup * (place + RING), v2, n2);
                tmem_fill(lanes + kGroup * (place + RING), 0.0f, kGroup);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] += v2[i];
#pragma unroll
                for (int i = 0; i < 2 * PW; ++i) n[i] += n2[i];
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(aempty + 8 * (o % RING));
            float from_right[PW], from_left[PW];
#pragma unroll
            for (int i = 0; i < PW; ++i) {
                from_right[i] = __shfl_down_sync(0xffffffffu, n[i], 1);
                from_left[i] = __shfl_up_sync(0xffffffffu, n[PW + i], 1);
            }
            if (split) {
                float* const e = edge + (o & 1) * 8 * PW;
                if (lane == 0 || lane == 31)
#pragma unroll
                    for (int i = 0; i < PW; ++i) e[(2 * warp + (lane ? 1 : 0)) * PW + i] = lane ? n[PW + i] : n[i];
                __syncwarp();
                if (lane == 0) mbar_arrive(edges);
                ok = mbar_wait(edges, o & 1) && ok;
                if (lane == 31 && warp < 3)
#pragma unroll
                    for (int i = 0; i < PW; ++i) from_right[i] = e[2 * (warp + 1) * PW + i];
                if (lane == 0 && warp > 0)
#pragma unroll
                    for (int i = 0; i < PW; ++i) from_left[i] = e[(2 * (warp - 1) + 1) * PW + i];
            }
#pragma unroll
            for (int i = 0; i < PW; ++i) {
                v[8 - PW + i] += right ? from_right[i] : 0.0f;
                v[i] += left ? from_left[i] : 0.0f;
            }
            if (o < count) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (AL != kWide && w + i >= b.Wv) v[i] = 0.0f;
                const uint4 t = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                if (look(t)) *again = 1u;
                store8<AL>(tb + (at.d0 + o) * addr.plane, w, b.W, t);
            }
        }
    }
    if (!ok && lane == 0) report_expired(P.expired);
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == kMmaWarp) tmem_free(tmem, kSourceCols);
    if (*again) source_again<KD, KH, KW>(P, blockIdx.x);
}

}  // namespace tc
}  // namespace ndc
