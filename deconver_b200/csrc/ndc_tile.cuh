// Tile kernels: any grouping with 3x3x3, 5x5 and 3x3 filters, 1 <= m, sc <= 16.  Rows and tensors of whole
// vectors go to those of ndc_pairs.cuh; these take the others: rows that are not (VEC = false), and whole ones where x or t1
// alone is off a vector address, or where a backward's scratch is within a hundredth of the built-in array's size (see use_pairs).
//
// A CTA owns a tile of one (sample, group) pair: TD planes x TH rows x TW columns of the output.
// One input channel at a time (or a few) is staged in shared memory with its halo, as float32 rows
// that start PW columns left of the tile, so that the window of a 4-voxel strip begins on a 16-byte
// quad; rows are read by consecutive lanes whatever the row length or alignment is, and what lies
// outside the volume is zero.  A thread keeps R rows x 4 voxels x up to 4 output channels in
// registers: a window loaded once feeds R filter rows and every output channel, which is what lifts
// these kernels off the one-thread-per-element form (ndc_generic.cuh, two loads per multiply-add).
// Multiply-adds are two-lane `fma.rn.f32x2` over neighbouring voxels; the filter is staged as
// duplicated (w, w) pairs.
//
// What bounds them: at 8 groups of 4 channels and 8 sources, 2 x 32x32x31 (an update and its backward, float32) they
// take 159 + 503 us, of which the multiply-adds alone are 0.13 ms; the rest is staging (a 4-byte copy and its address
// per staged element, 2.4 of them per output voxel and channel with the halo) and, in corr_kernel, one CTA of 194 - 221
// registers per thread (3x3x3) on a multiprocessor.  For depthwise ratio-4 filters the marching kernels of
// ndc_dw4_*.cuh stage each element once and are twice as fast.
//
//   adjoint_kernel   A of x and t1 (forward output, backward ratio terms) or of gt1 (source gradient)
//   k_kernel         K of the source, or of the two backward ratio tensors
//   corr_kernel      the three filter-gradient correlations, accumulated over many tiles per CTA
//   *_sum_kernel     fixed-order sums of their partial records: no atomics, bitwise reproducible
#pragma once

#include <algorithm>

#include "ndc_common.cuh"
#include "ndc_dw4_common.cuh"
#include "ndc_pairs.cuh"

namespace ndc {
namespace tile {

using dw4::f32x2;
using dw4::fma2;
using dw4::pack2;
using dw4::unpack2;

constexpr int V = 4;          // voxels per strip
constexpr int CB = 4;         // output channels per thread

struct TileGeo {
    int m, sc, G, B, D, H, W;
    long long SP;
    int NS, NP, TD;           // strips per tile row, groups of R rows, planes
    int ntw, nth, ntd;        // tiles along each axis
    int rows, planes, pitch;  // staged rows / planes (with halo), floats per row
    int plane;                // floats per staged plane
    int table;                // words of the row table
    int threads;
};

// Strips are dealt out evenly over the tiles of a row (43 strips: three tiles of 15), row groups
// likewise; CTAs of up to 256 threads.
template <int KD, int KH, int KW>
inline TileGeo plan(const Geo& g, int R, int max_threads) {
    TileGeo t;
    t.m = g.m; t.sc = g.sc; t.G = g.G; t.B = g.B; t.D = g.D; t.H = g.H; t.W = g.W; t.SP = g.SP;
    const int strips = (g.W + V - 1) / V, groups = (g.H + R - 1) / R;
    const int cap = KD > 1 ? 8 : 16;
    t.ntw = (strips + cap - 1) / cap;
    t.NS = (strips + t.ntw - 1) / t.ntw;
    t.TD = KD > 1 ? std::min(g.D, 4) : 1;
    t.ntd = (g.D + t.TD - 1) / t.TD;
    t.TD = (g.D + t.ntd - 1) / t.ntd;
    int np = std::max(1, max_threads / (t.NS * t.TD));
    t.nth = (groups + np - 1) / np;
    t.NP = (groups + t.nth - 1) / t.nth;
    t.rows = t.NP * R + (KH - 1);
    t.planes = t.TD + (KD - 1);
    int pitch = (t.NS * V + KW - 1 + 3) / 4 * 4;
    // lanes that wrap to the next row group should continue through the banks, where a few
    // more columns can bring that about
    for (int more = 0; more <= 12; more += 4)
        if ((R * (pitch + more) - V * t.NS) % 32 == 0) { pitch += more; break; }
    t.pitch = pitch;
    t.plane = t.rows * pitch;
    t.table = (t.rows * t.planes + 3) / 4 * 4;
    t.threads = (t.NS * t.NP * t.TD + 31) / 32 * 32;
    return t;
}

// Element offset of every staged row of a tile inside its channel, or -1 outside the volume:
// decoded once per tile, used for every channel.
template <int KD, int KH>
__device__ __forceinline__ void make_rows(int* tab, const TileGeo& t, int d0, int h0) {
    for (int rr = threadIdx.x; rr < t.planes * t.rows; rr += blockDim.x) {
        const int pl = rr / t.rows, row = rr - pl * t.rows;
        const int d = d0 - KD / 2 + pl, h = h0 - KH / 2 + row;
        tab[rr] = d >= 0 && d < t.D && h >= 0 && h < t.H ? (d * t.H + h) * t.W : -1;
    }
}

// One channel's tile with halo into shared memory.  Rows go to warps, columns to lanes: coalesced
// for every row length and alignment.  float32 goes by 4-byte cp.async (zero-filled outside the
// volume) and has landed after the caller's wait; bfloat16 is converted on the way, up to 12 loads
// in flight per lane.
template <int KW>
__device__ __forceinline__ void stage(float* dst, const float* __restrict__ src, const TileGeo& t, const int* tab, int w0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int wfirst = w0 - KW / 2 + lane, total = t.planes * t.rows;
    const bool in0 = wfirst >= 0 && wfirst < t.W, in1 = wfirst + 32 >= 0 && wfirst + 32 < t.W,
               in2 = wfirst + 64 >= 0 && wfirst + 64 < t.W;
    unsigned q = (unsigned)__cvta_generic_to_shared(dst + warp * t.pitch + lane);
    auto put = [&](unsigned at, const float* p, bool in) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(at), "l"(in ? p : src), "r"(in ? 4 : 0) : "memory");
    };
    for (int rr = warp; rr < total; rr += nwarp, q += nwarp * t.pitch * 4) {
        const int off = tab[rr];
        const float* p = src + off + wfirst;
        if (lane < t.pitch) put(q, p, off >= 0 && in0);
        if (lane + 32 < t.pitch) put(q + 128, p + 32, off >= 0 && in1);
        if (lane + 64 < t.pitch) put(q + 256, p + 64, off >= 0 && in2);
    }
}
template <int KW>
__device__ __forceinline__ void stage(float* dst, const __nv_bfloat16* __restrict__ src, const TileGeo& t, const int* tab, int w0) {
    constexpr int UR = 4, UC = 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int wfirst = w0 - KW / 2 + lane, total = t.planes * t.rows;
    for (int r0 = warp; r0 < total; r0 += nwarp * UR) {
        __nv_bfloat16 v[UR][UC];
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int rr = r0 + u * nwarp, off = rr < total ? tab[rr] : -1;
#pragma unroll
            for (int c = 0; c < UC; ++c) {
                const int w = wfirst + 32 * c;
                v[u][c] = __float2bfloat16_rn(0.0f);
                if (off >= 0 && w >= 0 && w < t.W && lane + 32 * c < t.pitch) v[u][c] = src[off + w];
            }
        }
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int rr = r0 + u * nwarp;
#pragma unroll
            for (int c = 0; c < UC; ++c)
                if (rr < total && lane + 32 * c < t.pitch) dst[rr * t.pitch + lane + 32 * c] = to_f32(v[u][c]);
        }
    }
}
// Bias and ReLU on the elements this thread staged (inside the volume; the halo outside stays zero).
template <int KW>
__device__ __forceinline__ void rectify(float* dst, const TileGeo& t, const int* tab, int w0, float bias, bool relu) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int wfirst = w0 - KW / 2 + lane, total = t.planes * t.rows;
    for (int rr = warp; rr < total; rr += nwarp) {
        if (tab[rr] < 0) continue;
        for (int c = lane; c < t.pitch; c += 32) {
            const int w = wfirst + (c - lane);
            if (w < 0 || w >= t.W) continue;
            float v = dst[rr * t.pitch + c] + bias;
            if (relu) v = fmaxf(v, 0.0f);
            dst[rr * t.pitch + c] = v;
        }
    }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void landed() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// 8 columns of a staged row from a quad boundary, as pairs of neighbours: even[i] = (2i, 2i+1),
// odd[i] = (2i+1, 2i+2)
struct Window {
    f32x2 even[4], odd[3];
    __device__ __forceinline__ void load(const float* p) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(p + 4);
        even[0] = a.x; even[1] = a.y; even[2] = b.x; even[3] = b.y;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            float lo, hi, lo2, hi2;
            unpack2(even[i], lo, hi);
            unpack2(even[i + 1], lo2, hi2);
            odd[i] = pack2(hi, lo2);
        }
    }
    __device__ __forceinline__ f32x2 at(int i) const { return i & 1 ? odd[i >> 1] : even[i >> 1]; }   // i static
};

__device__ __forceinline__ f32x2 dup(float v) { return pack2(v, v); }

// tile of a CTA: origin and this thread's place in it
struct Place {
    int tile, d0, h0, w0, strip, group, dz;
    bool active;
    __device__ __forceinline__ Place(const TileGeo& t, int tile_, int R) : tile(tile_) {
        const int tw = tile % t.ntw, th = (tile / t.ntw) % t.nth, td = tile / (t.ntw * t.nth);
        d0 = td * t.TD; h0 = th * t.NP * R; w0 = tw * t.NS * V;
        const int tid = threadIdx.x;
        strip = tid % t.NS;
        const int q = tid / t.NS;
        group = q % t.NP; dz = q / t.NP;
        active = dz < t.TD && d0 + dz < t.D && h0 + group * R < t.H && w0 + strip * V < t.W;
        if (!active) { dz = 0; group = 0; strip = 0; }
    }
};

template <typename T, bool VEC>
__device__ __forceinline__ void load_strip(const T* p, int n, float (&v)[V]) {
    const float4 q = dw4::load4<T, VEC>(p, n);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <typename T, bool VEC>
__device__ __forceinline__ void store_strip(T* p, int n, const float (&v)[V]) {
    dw4::store4<T, VEC>(p, n, make_float4(v[0], v[1], v[2], v[3]));
}

// ---- A: adjoint sweeps ----------------------------------------------------------------------
enum Mode { kForward = 0, kRatio = 1, kSource = 2 };

struct AdjointParams {
    TileGeo t;
    const void* x; const void* t1;       // kSource: t1 is gt1 (float32), x is not read
    const void* z; const void* gout;
    const float* h; const float* bias;
    void* out;                           // kForward: out; kRatio: direct term (or NULL); kSource: gz (in/out)
    float* gnum; float* gden;            // kRatio
    float* gb_partial;                   // kSource: [bg][block][tile][CB] bias-gradient sums, or NULL
    float eps;
    int relu, blocks;                    // blocks of CB source channels
};

template <typename T, int KD, int KH, int KW, int MODE, bool VEC>
__global__ void __launch_bounds__(256, 2) adjoint_kernel(const AdjointParams P) {
    constexpr int R = 2, KT = KD * KH * KW, NT = MODE == kSource ? 1 : 2;
    extern __shared__ __align__(16) float smem[];
    const TileGeo& t = P.t;
    const int ntiles = t.ntw * t.nth * t.ntd;
    const Place at(t, blockIdx.x % ntiles, R);
    const int cb = (blockIdx.x / ntiles) % P.blocks;
    const long long bg = blockIdx.x / ((long long)ntiles * P.blocks);
    const int g = (int)(bg % t.G), i0 = cb * CB, nch = min(CB, t.sc - i0);
    f32x2* w = reinterpret_cast<f32x2*>(smem);                  // [o][tau][CB]
    int* tab = reinterpret_cast<int*>(smem + 2 * t.m * KT * CB);
    float* const tiles0 = smem + 2 * t.m * KT * CB + t.table;
    const int tile_floats = t.planes * t.plane;
    make_rows<KD, KH>(tab, t, at.d0, at.h0);
    for (int e = threadIdx.x; e < t.m * KT * CB; e += blockDim.x) {
        const int j = e % CB, tau = (e / CB) % KT, o = e / (CB * KT);
        w[e] = dup(j < nch ? P.h[(((long long)g * t.m + o) * t.sc + i0 + j) * KT + tau] : 0.0f);
    }
    f32x2 acc[NT][R][CB][V / 2];
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int j = 0; j < CB; ++j)
#pragma unroll
                for (int v = 0; v < V / 2; ++v) acc[a][r][j][v] = dup(MODE == kSource ? 0.0f : P.eps);

    __syncthreads();
    auto request = [&](int o) {     // two buffers: the next channel lands while this one is swept
        const long long base = (bg * t.m + o) * t.SP;
        float* dst = tiles0 + (o & 1) * NT * tile_floats;
        if (MODE == kSource) {
            stage<KW>(dst, reinterpret_cast<const float*>(P.t1) + base, t, tab, at.w0);
        } else {
            stage<KW>(dst, reinterpret_cast<const T*>(P.x) + base, t, tab, at.w0);
            stage<KW>(dst + tile_floats, reinterpret_cast<const T*>(P.t1) + base, t, tab, at.w0);
        }
        commit();
    };
    request(0);
    for (int o = 0; o < t.m; ++o) {
        if (o + 1 < t.m) { request(o + 1); landed<1>(); } else landed<0>();
        __syncthreads();
        const float* tiles = tiles0 + (o & 1) * NT * tile_floats;
        // input row = output row + PH - kh: one filter row at a time (a run-time loop: unrolled, the
        // compiler keeps several rows' windows and weights alive and spills)
#pragma unroll 1
        for (int kdh = at.active ? 0 : KD * KH; kdh < KD * KH; ++kdh) {
            const int kd = kdh / KH, kh = kdh - kd * KH;
            const float* p = tiles + (at.dz + KD - 1 - kd) * t.plane + (at.group * R + KH - 1 - kh) * t.pitch + V * at.strip;
            const f32x2* wk = w + (o * KT + kdh * KW) * CB;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                asm volatile("" ::: "memory");   // the weights are read again for each row: kept, they spill
                Window win[NT];
#pragma unroll
                for (int a = 0; a < NT; ++a) win[a].load(p + a * tile_floats + r * t.pitch);
#pragma unroll
                for (int kw = 0; kw < KW; ++kw) {
                    const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(wk + kw * CB);
                    const ulonglong2 w01 = wp[0], w23 = wp[1];
                    const f32x2 wj[CB] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
                    for (int j = 0; j < CB; ++j)
#pragma unroll
                        for (int v = 0; v < V / 2; ++v)
#pragma unroll
                            for (int a = 0; a < NT; ++a)
                                fma2(acc[a][r][j][v], win[a].at(KW - 1 - kw + 2 * v), wj[j]);
                }
            }
        }
        if (o + 1 < t.m) __syncthreads();   // before this buffer is filled again
    }

    float gbs[CB] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (at.active) {
        const int wcol = at.w0 + V * at.strip, n = min(V, t.W - wcol);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int hrow = at.h0 + at.group * R + r;
            if (hrow >= t.H) continue;
            const long long off = ((long long)(at.d0 + at.dz) * t.H + hrow) * t.W + wcol;
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                if (j >= nch) continue;
                const long long e = (bg * t.sc + i0 + j) * t.SP + off;
                const float b = P.bias ? P.bias[g * t.sc + i0 + j] : 0.0f;
                float zv[V], out[V];
                load_strip<T, VEC>(reinterpret_cast<const T*>(P.z) + e, n, zv);
                if (MODE == kForward) {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float s = zv[v] + b;
                        if (P.relu) s = fmaxf(s, 0.0f);
                        out[v] = __fdiv_rn(s * dw4::lane_of(acc[0][r][j][v / 2], v & 1),
                                           dw4::lane_of(acc[NT - 1][r][j][v / 2], v & 1));
                    }
                    store_strip<T, VEC>(reinterpret_cast<T*>(P.out) + e, n, out);
                } else if (MODE == kRatio) {
                    float gv[V], gn[V], gd[V];
                    load_strip<T, VEC>(reinterpret_cast<const T*>(P.gout) + e, n, gv);
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float s = zv[v] + b;
                        if (P.relu) s = fmaxf(s, 0.0f);
                        const float nn = dw4::lane_of(acc[0][r][j][v / 2], v & 1);
                        const float dd = dw4::lane_of(acc[NT - 1][r][j][v / 2], v & 1);
                        gn[v] = __fdiv_rn(gv[v] * s, dd);
                        gd[v] = -__fdiv_rn(gn[v] * nn, dd);
                        out[v] = __fdiv_rn(gv[v] * nn, dd);
                    }
                    store_strip<float, VEC>(P.gnum + e, n, gn);
                    store_strip<float, VEC>(P.gden + e, n, gd);
                    if (P.out) store_strip<T, VEC>(reinterpret_cast<T*>(P.out) + e, n, out);
                } else {
                    float dv[V];
                    T* gz = reinterpret_cast<T*>(P.out) + e;
                    load_strip<T, VEC>(gz, n, dv);
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float q = dv[v] + dw4::lane_of(acc[0][r][j][v / 2], v & 1);
                        if (P.relu && !(zv[v] + b > 0.0f)) q = 0.0f;
                        if (v >= n) q = 0.0f;
                        out[v] = q;
                        gbs[j] += to_f32(from_f32<T>(q));      // the values as stored
                    }
                    store_strip<T, VEC>(gz, n, out);
                }
            }
        }
    }
    if (MODE == kSource && P.gb_partial) {
        __syncthreads();
        float* scratch = tiles0;
#pragma unroll
        for (int j = 0; j < CB; ++j) {
            const float s = block_sum(gbs[j], scratch);
            if (threadIdx.x == 0) P.gb_partial[(size_t)blockIdx.x * CB + j] = s;
        }
    }
}

// ---- K --------------------------------------------------------------------------------------
struct KParams {
    TileGeo t;
    const void* in[2];       // source-sized inputs (TI), one per `which`
    void* out[2];            // filter-sized outputs
    int out_f32[2];          // else T
    int count;               // inputs to convolve
    const float* h; const float* bias;
    int relu, blocks, nbuf;  // blocks of OB output channels; input channels staged at a time
};

// OB output channels per thread; R = 4 rows of one channel or 2 rows of four.
template <typename TI, typename T, int KD, int KH, int KW, int OB, bool VEC>
__global__ void __launch_bounds__(256, 2) k_kernel(const KParams P) {
    constexpr int R = OB == 1 ? 4 : 2, KT = KD * KH * KW;
    extern __shared__ __align__(16) float smem[];
    const TileGeo& t = P.t;
    const int ntiles = t.ntw * t.nth * t.ntd;
    const Place at(t, blockIdx.x % ntiles, R);
    long long q = blockIdx.x / ntiles;
    const int ob = (int)(q % P.blocks); q /= P.blocks;
    const int which = (int)(q % P.count);
    const long long bg = q / P.count;
    const int g = (int)(bg % t.G), o0 = ob * OB, nout = min(OB, t.m - o0);
    f32x2* w = reinterpret_cast<f32x2*>(smem);                  // [i][tau][OB]
    const int wfloats = (2 * t.sc * KT * OB + 3) / 4 * 4;
    int* tab = reinterpret_cast<int*>(smem + wfloats);
    float* tiles = smem + wfloats + t.table;
    const int tile_floats = t.planes * t.plane;
    make_rows<KD, KH>(tab, t, at.d0, at.h0);
    for (int e = threadIdx.x; e < t.sc * KT * OB; e += blockDim.x) {
        const int j = e % OB, tau = (e / OB) % KT, i = e / (OB * KT);
        w[e] = dup(j < nout ? P.h[(((long long)g * t.m + o0 + j) * t.sc + i) * KT + tau] : 0.0f);
    }
    const TI* in = reinterpret_cast<const TI*>(P.in[which]) + bg * t.sc * t.SP;
    f32x2 acc[R][OB][V / 2];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < OB; ++j)
#pragma unroll
            for (int v = 0; v < V / 2; ++v) acc[r][j][v] = dup(0.0f);
    __syncthreads();
    for (int i0 = 0; i0 < t.sc; i0 += P.nbuf) {
        const int ni = min(P.nbuf, t.sc - i0);
        if (i0) __syncthreads();
        for (int i = 0; i < ni; ++i) stage<KW>(tiles + i * tile_floats, in + (i0 + i) * t.SP, t, tab, at.w0);
        commit();
        landed<0>();
        if (P.bias || P.relu)
            for (int i = 0; i < ni; ++i)
                rectify<KW>(tiles + i * tile_floats, t, tab, at.w0, P.bias ? P.bias[g * t.sc + i0 + i] : 0.0f, P.relu);
        __syncthreads();
        if (!at.active) continue;
#pragma unroll 1
        for (int ik = 0; ik < ni * KD; ++ik) {
            const int i = ik / KD, kd = ik - i * KD;
            const float* p = tiles + i * tile_floats + (at.dz + kd) * t.plane + at.group * R * t.pitch + V * at.strip;
            const f32x2* wk = w + ((i0 + i) * KT + kd * KH * KW) * OB;
#pragma unroll
            for (int rr = 0; rr < R + KH - 1; ++rr) {
                Window win;
                win.load(p + rr * t.pitch);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int kh = rr - r;
                    if (kh < 0 || kh >= KH) continue;
#pragma unroll
                    for (int kw = 0; kw < KW; ++kw) {
                        f32x2 wj[OB];
                        if (OB == 4) {
                            const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(wk + (kh * KW + kw) * OB);
                            const ulonglong2 w01 = wp[0], w23 = wp[1];
                            wj[OB > 3 ? 3 : 0] = w23.y; wj[OB > 2 ? 2 : 0] = w23.x; wj[OB > 1 ? 1 : 0] = w01.y;
                            wj[0] = w01.x;
                        } else {
                            wj[0] = wk[kh * KW + kw];
                        }
#pragma unroll
                        for (int j = 0; j < OB; ++j)
#pragma unroll
                            for (int v = 0; v < V / 2; ++v) fma2(acc[r][j][v], win.at(kw + 2 * v), wj[j]);
                    }
                }
            }
        }
    }
    if (!at.active) return;
    const int wcol = at.w0 + V * at.strip, n = min(V, t.W - wcol);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int hrow = at.h0 + at.group * R + r;
        if (hrow >= t.H) continue;
        const long long off = ((long long)(at.d0 + at.dz) * t.H + hrow) * t.W + wcol;
#pragma unroll
        for (int j = 0; j < OB; ++j) {
            if (j >= nout) continue;
            const long long e = (bg * t.m + o0 + j) * t.SP + off;
            float out[V];
            unpack2(acc[r][j][0], out[0], out[1]);
            unpack2(acc[r][j][1], out[2], out[3]);
            if (P.out_f32[which]) store_strip<float, VEC>(reinterpret_cast<float*>(P.out[which]) + e, n, out);
            else store_strip<T, VEC>(reinterpret_cast<T*>(P.out[which]) + e, n, out);
        }
    }
}

// ---- filter gradient ------------------------------------------------------------------------
// gh[o, i, tau] = sum_p gden[i,p] t1[o,p+pad-tau] + gnum[i,p] x[o,..] + s[i,p] gt1[o,..]
struct CorrParams {
    TileGeo t;
    const float* gden; const float* gnum;
    const void* z; const float* bias;
    const void* t1; const void* x; const float* gt1;
    float* partial;          // [g][o][block][split][KT * CB]
    int relu, blocks, splits;
};

template <typename T, int KD, int KH, int KW, bool VEC>
__global__ void __launch_bounds__(256, 1) corr_kernel(const CorrParams P) {
    constexpr int KT = KD * KH * KW;
    extern __shared__ __align__(16) float smem[];
    const TileGeo& t = P.t;
    const int ntiles = t.ntw * t.nth * t.ntd;
    int q = blockIdx.x;
    const int split = q % P.splits; q /= P.splits;
    const int ib = q % P.blocks; q /= P.blocks;
    const int o = q % t.m, g = q / t.m;
    const int i0 = ib * CB, nch = min(CB, t.sc - i0);
    // two of each: row tables, staged tiles, and the threads' own strips of the other factor
    const int tile_floats = t.planes * t.plane;
    int* const tabs = reinterpret_cast<int*>(smem);
    float* const bufs = smem + 2 * t.table;
    float* const own = bufs + 2 * tile_floats + threadIdx.x * V;
    const int own_step = blockDim.x * V;
    f32x2 acc[KT][CB / 2];
#pragma unroll
    for (int k = 0; k < KT; ++k)
#pragma unroll
        for (int j = 0; j < CB / 2; ++j) acc[k][j] = dup(0.0f);

    // this CTA's share: every splits-th tile of the batch, three factor pairs each
    const int work = t.B * ntiles;
    const int steps = 3 * ((work - split + P.splits - 1) / P.splits);
    auto place = [&](int step) { return Place(t, (split + step / 3 * P.splits) % ntiles, 1); };
    auto sample = [&](int step) { return (long long)((split + step / 3 * P.splits) / ntiles) * t.G + g; };
    auto request = [&](int step) {
        const Place at = place(step);
        const int pair = step % 3;
        const long long bg = sample(step), base = (bg * t.m + o) * t.SP;
        float* dst = bufs + (step & 1) * tile_floats;
        const int* tab = tabs + (step / 3 & 1) * t.table;
        if (pair == 0) stage<KW>(dst, reinterpret_cast<const T*>(P.t1) + base, t, tab, at.w0);
        else if (pair == 1) stage<KW>(dst, reinterpret_cast<const T*>(P.x) + base, t, tab, at.w0);
        else stage<KW>(dst, P.gt1 + base, t, tab, at.w0);
        if (pair < 2 || sizeof(T) == 4) {
            const int wcol = at.w0 + V * at.strip, n = min(V, t.W - wcol);
            const float* src = pair == 0 ? P.gden : pair == 1 ? P.gnum : reinterpret_cast<const float*>(P.z);
            src += (bg * t.sc + i0) * t.SP + ((long long)(at.d0 + at.dz) * t.H + at.h0 + at.group) * t.W + wcol;
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                const unsigned a = (unsigned)__cvta_generic_to_shared(own + ((step & 1) * CB + j) * own_step);
                const bool ok = at.active && j < nch;
                const float* p = ok ? src + j * t.SP : P.gden;
                if (VEC) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(p), "r"(ok ? 16 : 0) : "memory");
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        const bool in = ok && v < n;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(a + 4 * v), "l"(in ? p + v : P.gden), "r"(in ? 4 : 0) : "memory");
                    }
                }
            }
        }
        commit();
    };
    if (steps > 0) {
        const Place at = place(0);
        make_rows<KD, KH>(tabs, t, at.d0, at.h0);
        __syncthreads();
        request(0);
    }
    for (int step = 0; step < steps; ++step) {
        const int pair = step % 3;
        if (pair == 2 && step + 1 < steps) {
            const Place nx = place(step + 1);
            make_rows<KD, KH>(tabs + ((step + 1) / 3 & 1) * t.table, t, nx.d0, nx.h0);
        }
        __syncthreads();       // the other buffer has been read, the next row table is written
        if (step + 1 < steps) { request(step + 1); landed<1>(); } else landed<0>();
        const Place at = place(step);
        const float* tile = bufs + (step & 1) * tile_floats;
        f32x2 a[CB / 2][V];        // channel pairs
        {
            float av[CB][V];
            const int wcol = at.w0 + V * at.strip, n = at.active ? min(V, t.W - wcol) : 0;
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                if (pair < 2 || sizeof(T) == 4) {
                    const float4 f = *reinterpret_cast<const float4*>(own + ((step & 1) * CB + j) * own_step);
                    av[j][0] = f.x; av[j][1] = f.y; av[j][2] = f.z; av[j][3] = f.w;
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) av[j][v] = 0.0f;
                    if (n > 0 && j < nch)
                        load_strip<T, VEC>(reinterpret_cast<const T*>(P.z) + (sample(step) * t.sc + i0 + j) * t.SP +
                                               ((long long)(at.d0 + at.dz) * t.H + at.h0 + at.group) * t.W + wcol, n, av[j]);
                }
                if (pair == 2) {
                    const float b = P.bias && j < nch ? P.bias[g * t.sc + i0 + j] : 0.0f;
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        av[j][v] += b;
                        if (P.relu) av[j][v] = fmaxf(av[j][v], 0.0f);
                        if (v >= n || j >= nch) av[j][v] = 0.0f;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < CB / 2; ++j)
#pragma unroll
                for (int v = 0; v < V; ++v) a[j][v] = dw4::make_pair2(av[2 * j][v], av[2 * j + 1][v]);
        }
        __syncthreads();       // everybody's part of the tile has landed
        if (!at.active) continue;
#pragma unroll
        for (int kd = 0; kd < KD; ++kd) {
            const float* p = tile + (at.dz + KD - 1 - kd) * t.plane + at.group * t.pitch + V * at.strip;
#pragma unroll
            for (int kh = 0; kh < KH; ++kh) {
                const float4 lo = *reinterpret_cast<const float4*>(p + (KH - 1 - kh) * t.pitch);
                const float4 hi = *reinterpret_cast<const float4*>(p + (KH - 1 - kh) * t.pitch + 4);
                const float c[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                f32x2 c2[V + KW - 1];
#pragma unroll
                for (int i = 0; i < V + KW - 1; ++i) c2[i] = dup(c[i]);
#pragma unroll
                for (int kw = 0; kw < KW; ++kw)
#pragma unroll
                    for (int j = 0; j < CB / 2; ++j)
#pragma unroll
                        for (int v = 0; v < V; ++v)
                            fma2(acc[(kd * KH + kh) * KW + kw][j], a[j][v], c2[KW - 1 - kw + v]);
            }
        }
    }
    // combine: shuffles inside a warp, then the warps in order
    float* rec = smem;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KT; ++k)
#pragma unroll
        for (int j = 0; j < CB / 2; ++j) {
            float lo, hi;
            unpack2(acc[k][j], lo, hi);
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                lo += __shfl_xor_sync(0xffffffffu, lo, s);
                hi += __shfl_xor_sync(0xffffffffu, hi, s);
            }
            if (lane == 0) { rec[warp * KT * CB + k * CB + 2 * j] = lo; rec[warp * KT * CB + k * CB + 2 * j + 1] = hi; }
        }
    __syncthreads();
    for (int k = threadIdx.x; k < KT * CB; k += blockDim.x) {
        float s = 0.0f;
        for (int u = 0; u < nwarp; ++u) s += rec[u * KT * CB + k];
        P.partial[(size_t)blockIdx.x * KT * CB + k] = s;
    }
}

// gb[g*sc + i] = sum over samples and tiles; one warp per channel, lanes in a fixed partition.
static __global__ void __launch_bounds__(128) gb_sum_kernel(const float* __restrict__ partial, int B, int G, int sc, int blocks,
                                                     int ntiles, float* __restrict__ gb) {
    const int ch = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (ch >= G * sc) return;
    const int g = ch / sc, i = ch % sc;
    float s = 0.0f;
    for (int b = 0; b < B; ++b) {
        const float* p = partial + (((size_t)b * G + g) * blocks + i / CB) * ntiles * CB + i % CB;
        for (int k = lane; k < ntiles; k += 32) s += p[(size_t)k * CB];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) gb[ch] = s;
}

// ---- host side ------------------------------------------------------------------------------
inline bool covers(const Geo& g) {
    if (g.m > 16 || g.sc > 16 || g.SP >= (1LL << 31)) return false;
    return (g.kD == 3 && g.kH == 3 && g.kW == 3) || (g.kD == 1 && g.kH == 5 && g.kW == 5) ||
           (g.kD == 1 && g.kH == 3 && g.kW == 3);
}

inline size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

// Scratch of the backward: gnum | gden | gt1 | bias-gradient records | correlation records.
struct BwdScratch { size_t gnum, gden, gt1, gb, corr, bytes; };

inline int source_blocks(const Geo& g) { return (g.sc + CB - 1) / CB; }

template <int KD, int KH, int KW>
inline TileGeo plan_adjoint(const Geo& g) { return plan<KD, KH, KW>(g, 2, 256); }
template <int KD, int KH, int KW>
inline TileGeo plan_corr(const Geo& g) { return plan<KD, KH, KW>(g, 1, 256); }
inline long long tiles_of(const TileGeo& t) { return (long long)t.ntw * t.nth * t.ntd; }

// CTAs per (group, output channel, block of source channels) of corr_kernel: one round of the GPU, of
// which a multiprocessor takes one CTA, but no more than there are tiles.
inline int corr_splits(const Geo& g, const TileGeo& t) {
    const long long combos = (long long)g.G * g.m * source_blocks(g), work = (long long)g.B * tiles_of(t);
    long long s = num_sms() / combos;
    if (s > work) s = work;
    return (int)std::max(1LL, s);
}

template <int KD, int KH, int KW>
inline BwdScratch scratch_shape(const Geo& g) {
    BwdScratch s;
    const size_t src = (size_t)g.B * g.G * g.sc * g.SP * sizeof(float);
    const TileGeo ta = plan_adjoint<KD, KH, KW>(g), tc = plan_corr<KD, KH, KW>(g);
    s.gnum = 0;
    s.gden = up256(src);
    s.gt1 = s.gden + up256(src);
    s.gb = s.gt1 + up256((size_t)g.B * g.G * g.m * g.SP * sizeof(float));
    s.corr = s.gb + up256((size_t)g.B * g.G * source_blocks(g) * tiles_of(ta) * CB * sizeof(float));
    s.bytes = s.corr + up256((size_t)g.G * g.m * source_blocks(g) * corr_splits(g, tc) * g.KT * CB * sizeof(float));
    return s;
}
// Whether whole vectors go to the pairs kernels, and their scratch.  Their records are larger: where they alone would take a
// backward out of what ndc_bwd_static has (its results are those of ndc_bwd), fewer of them have to do, or, where that is
// less than half, these kernels.  Seven backwards that this meets, against these
// kernels throughout: 1.00 - 1.66 times as fast (3 groups of 16 and 16, 453x64, 3x3: 373 -> 225 us).
template <int KD, int KH, int KW>
inline bool use_pairs(const Geo& g, size_t own, pairs::BwdScratch& sc) {
    return pairs::covers(g) && pairs::scratch_shape<KD, KH, KW>(g, own <= NDC_STATIC_WORKSPACE_BYTES ? NDC_STATIC_WORKSPACE_BYTES : SIZE_MAX, sc);
}
// Bytes of it for either kind of kernel: which one runs depends on the tensors' alignment too.
template <int KD, int KH, int KW>
inline size_t scratch_bytes(const Geo& g) {
    const size_t n = scratch_shape<KD, KH, KW>(g).bytes;
    pairs::BwdScratch sc;
    return use_pairs<KD, KH, KW>(g, n, sc) ? std::max(n, sc.bytes) : n;
}
inline size_t bwd_scratch(const Geo& g) {
    if (g.kD == 3) return scratch_bytes<3, 3, 3>(g);
    if (g.kH == 5) return scratch_bytes<1, 5, 5>(g);
    return scratch_bytes<1, 3, 3>(g);
}

template <typename Kern, typename P>
inline cudaError_t launch(Kern kern, long long grid, int threads, size_t smem, cudaStream_t st, const P& p) {
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    if (smem > 48 * 1024) {
        const cudaError_t e = allow_smem(kern);
        if (e != cudaSuccess) return e;
    }
    kern<<<(unsigned)grid, threads, smem, st>>>(p);
    launched();
    return cudaGetLastError();
}

template <typename T, int KD, int KH, int KW, int MODE>
cudaError_t run_adjoint(const Geo& g, AdjointParams& P, bool vec, cudaStream_t st) {
    P.t = plan_adjoint<KD, KH, KW>(g);
    P.blocks = source_blocks(g); P.eps = g.eps; P.relu = g.relu;
    const int nt = MODE == kSource ? 1 : 2;
    const size_t smem = sizeof(float) * (2 * (size_t)g.m * g.KT * CB + P.t.table +
                                        (size_t)(g.m > 1 ? 2 : 1) * nt * P.t.planes * P.t.plane);
    const long long grid = tiles_of(P.t) * P.blocks * g.B * g.G;
    return vec ? launch(adjoint_kernel<T, KD, KH, KW, MODE, true>, grid, P.t.threads, smem, st, P)
               : launch(adjoint_kernel<T, KD, KH, KW, MODE, false>, grid, P.t.threads, smem, st, P);
}

template <typename TI, typename T, int KD, int KH, int KW>
cudaError_t run_k(const Geo& g, KParams& P, bool vec, cudaStream_t st) {
    const int OB = g.m == 1 ? 1 : 4;
    P.t = plan<KD, KH, KW>(g, OB == 1 ? 4 : 2, OB == 1 ? 128 : 256);
    P.blocks = (g.m + OB - 1) / OB;
    const size_t weights = sizeof(float) * (2 * (size_t)g.sc * g.KT * OB + 4 + P.t.table);
    const size_t tile = sizeof(float) * (size_t)P.t.planes * P.t.plane;
    P.nbuf = (int)std::max((size_t)1, std::min((size_t)std::min(g.sc, 4), (64 * 1024 - weights) / tile));
    const size_t smem = weights + P.nbuf * tile;
    const long long grid = tiles_of(P.t) * P.blocks * P.count * g.B * g.G;
    if (OB == 1)
        return vec ? launch(k_kernel<TI, T, KD, KH, KW, 1, true>, grid, P.t.threads, smem, st, P)
                   : launch(k_kernel<TI, T, KD, KH, KW, 1, false>, grid, P.t.threads, smem, st, P);
    return vec ? launch(k_kernel<TI, T, KD, KH, KW, 4, true>, grid, P.t.threads, smem, st, P)
               : launch(k_kernel<TI, T, KD, KH, KW, 4, false>, grid, P.t.threads, smem, st, P);
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

template <typename T, int KD, int KH, int KW>
cudaError_t forward_shape(const Geo& g, const T* x, const T* z, const float* h, const float* bias, T* out, T* t1,
                          cudaStream_t st) {
    if (pairs::covers(g) && pairs::whole<T>({x, z, out, t1})) return pairs::forward_shape<T, KD, KH, KW>(g, x, z, h, bias, out, t1, st);
    const bool vec = g.W % V == 0 && aligned16(z) && aligned16(out) && aligned16(t1);
    KParams K{};
    K.in[0] = z; K.out[0] = t1; K.out_f32[0] = 0; K.count = 1; K.h = h; K.bias = bias; K.relu = g.relu;
    cudaError_t e = run_k<T, T, KD, KH, KW>(g, K, vec, st);
    if (e != cudaSuccess) return e;
    AdjointParams A{};
    A.x = x; A.t1 = t1; A.z = z; A.h = h; A.bias = bias; A.out = out;
    return run_adjoint<T, KD, KH, KW, kForward>(g, A, vec, st);
}

template <typename T, int KD, int KH, int KW>
cudaError_t backward_shape(const Geo& g, const T* x, const T* z, const T* t1, const float* h, const float* bias,
                           const T* gout, T* gx, T* gz, float* gh, float* gb, void* ws, cudaStream_t st) {
    const BwdScratch sc = scratch_shape<KD, KH, KW>(g);
    pairs::BwdScratch pc;
    if (pairs::whole<T>({x, z, t1, gout, gx, gz}) && use_pairs<KD, KH, KW>(g, sc.bytes, pc))
        return pairs::backward_shape<T, KD, KH, KW>(g, x, z, t1, h, bias, gout, gx, gz, gh, gb, ws, pc, st);
    float* gnum = (float*)((char*)ws + sc.gnum);
    float* gden = (float*)((char*)ws + sc.gden);
    float* gt1 = (float*)((char*)ws + sc.gt1);
    const bool vec = g.W % V == 0 && aligned16(z) && aligned16(gout) && (!gz || aligned16(gz)) && (!gx || aligned16(gx));
    AdjointParams A{};
    A.x = x; A.t1 = t1; A.z = z; A.gout = gout; A.h = h; A.bias = bias; A.out = gz; A.gnum = gnum; A.gden = gden;
    cudaError_t e = run_adjoint<T, KD, KH, KW, kRatio>(g, A, vec, st);
    if (e != cudaSuccess) return e;
    KParams K{};
    K.h = h;
    if (gz || gh) { K.in[K.count] = gden; K.out[K.count] = gt1; K.out_f32[K.count] = 1; ++K.count; }
    if (gx) { K.in[K.count] = gnum; K.out[K.count] = gx; K.out_f32[K.count] = 0; ++K.count; }
    e = run_k<float, T, KD, KH, KW>(g, K, vec, st);
    if (e != cudaSuccess) return e;
    if (gh) {
        CorrParams C{};
        C.t = plan_corr<KD, KH, KW>(g);
        C.gden = gden; C.gnum = gnum; C.z = z; C.bias = bias; C.t1 = t1; C.x = x; C.gt1 = gt1;
        C.partial = (float*)((char*)ws + sc.corr); C.relu = g.relu; C.blocks = source_blocks(g);
        C.splits = corr_splits(g, C.t);
        const size_t rec = (size_t)(C.t.threads / 32) * g.KT * CB;
        const size_t til = 2 * ((size_t)C.t.table + (size_t)C.t.planes * C.t.plane + (size_t)CB * V * C.t.threads);
        const long long grid = (long long)g.G * g.m * C.blocks * C.splits;
        e = vec ? launch(corr_kernel<T, KD, KH, KW, true>, grid, C.t.threads, sizeof(float) * std::max(rec, til), st, C)
                : launch(corr_kernel<T, KD, KH, KW, false>, grid, C.t.threads, sizeof(float) * std::max(rec, til), st, C);
        if (e != cudaSuccess) return e;
        const int n = g.G * g.m * g.sc * g.KT;
        pairs::corr_sum_kernel<<<(n + 127) / 128, 128, 0, st>>>(C.partial, g.G * g.m, g.sc, C.blocks, CB, C.splits, g.KT, gh);
        launched();
    }
    if (gz) {
        AdjointParams S{};
        S.t1 = gt1; S.z = z; S.h = h; S.bias = bias; S.out = gz;
        S.gb_partial = gb ? (float*)((char*)ws + sc.gb) : nullptr;
        e = run_adjoint<T, KD, KH, KW, kSource>(g, S, vec, st);
        if (e != cudaSuccess) return e;
        if (gb) {
            gb_sum_kernel<<<(g.G * g.sc + 3) / 4, 128, 0, st>>>(S.gb_partial, g.B, g.G, g.sc, S.blocks, (int)tiles_of(S.t), gb);
            launched();
        }
    }
    return cudaGetLastError();
}

template <typename T>
cudaError_t forward(const Geo& g, const T* x, const T* z, const float* h, const float* bias, T* out, T* t1, cudaStream_t st) {
    if (g.kD == 3) return forward_shape<T, 3, 3, 3>(g, x, z, h, bias, out, t1, st);
    if (g.kH == 5) return forward_shape<T, 1, 5, 5>(g, x, z, h, bias, out, t1, st);
    return forward_shape<T, 1, 3, 3>(g, x, z, h, bias, out, t1, st);
}
template <typename T>
cudaError_t backward(const Geo& g, const T* x, const T* z, const T* t1, const float* h, const float* bias, const T* gout,
                     T* gx, T* gz, float* gh, float* gb, void* ws, cudaStream_t st) {
    if (g.kD == 3) return backward_shape<T, 3, 3, 3>(g, x, z, t1, h, bias, gout, gx, gz, gh, gb, ws, st);
    if (g.kH == 5) return backward_shape<T, 1, 5, 5>(g, x, z, t1, h, bias, gout, gx, gz, gh, gb, ws, st);
    return backward_shape<T, 1, 3, 3>(g, x, z, t1, h, bias, gout, gx, gz, gh, gb, ws, st);
}

#define NDC_TILE_INSTANCES(PREFIX, T)                                                                            \
    PREFIX cudaError_t forward<T>(const Geo&, const T*, const T*, const float*, const float*, T*, T*, cudaStream_t); \
    PREFIX cudaError_t backward<T>(const Geo&, const T*, const T*, const T*, const float*, const float*, const T*,   \
                                   T*, T*, float*, float*, void*, cudaStream_t);
#ifdef NDC_TILE_EXTERN
NDC_TILE_INSTANCES(extern template, float)
NDC_TILE_INSTANCES(extern template, __nv_bfloat16)
#endif

}  // namespace tile
}  // namespace ndc
