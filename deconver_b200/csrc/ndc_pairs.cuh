// Tile kernels for rows of whole vectors: any grouping (m, sc <= 16) with 3x3x3, 5x5 and 3x3 filters (ndc_tile.cuh
// takes the other rows).
//
// A CTA owns a tile of one (sample, group) pair: TD planes x TH rows x TW columns of the output.  It
// stages one input channel at a time in shared memory with its halo and sweeps it with R rows x 4 voxels
// x CB output channels per thread in registers; the next channel lands meanwhile.
//
// Two streams.  Every staged element is a PAIR of float32 values, one of either stream, and every
// multiply-add a two-lane `fma.rn.f32x2` with a weight staged twice, so that what is loaded is what
// is multiplied: no lane is moved or duplicated.  The streams are two tensors that one filter is applied to
// (x and t1; gden and gnum), or two tiles of one tensor (the source, gt1).  The neighbours' voxels
// of a window lie PW places on, so that it begins on a 16-byte chunk; chunks are XOR-swizzled, so that
// the eight strips of a quarter-warp meet eight bank groups.
//
// What bounds them: the multiply-adds, at 1.2 - 1.3 instructions per two of them (a window of three or
// four 16-byte words serves all channels and up to three filter rows; weights are read by broadcast).  With
// one stream per pass, neighbouring voxels in the lanes and four channels per thread it was 2.3 - 5:
// lanes moved to make odd pairs, windows read once per filter row, and each tile staged once per four channels.
// A training step with 8 groups of 4 channels and 8 sources, 2 x 32^3, float32: 733 -> 478 us.
//
//   conv_kernel      A of x and t1 (forward output, backward ratio terms) or of gt1 (source gradient); K of the
//                    source, or of the two backward ratio tensors
//   corr_kernel      the three filter-gradient correlations, accumulated over many tiles per CTA
//   *_sum_kernel     fixed-order sums of their partial records: no atomics, bitwise reproducible
#pragma once

#include <algorithm>
#include <initializer_list>
#include <type_traits>

#include "ndc_common.cuh"
#include "ndc_dw4_common.cuh"

namespace ndc {
namespace pairs {

using dw4::f32x2;
using dw4::fma2;
using dw4::pack2;
using dw4::unpack2;

constexpr int V = 4;          // voxels per strip

struct TileGeo {
    int m, sc, G, B, D, H, W;
    long long SP;
    int NS, NP, TD;           // strips per tile row, groups of R rows, planes
    int ntw, nth, ntd;        // tiles along each axis
    int rows, planes, pitch;  // staged rows / planes (with halo), floats per row
    int plane;                // floats per staged plane
    int chunks, table;        // staged quads; words of their table
    int threads;
    __host__ __device__ int tiles() const { return ntw * nth * ntd; }
};

// Strips are dealt out evenly over the tiles of a row (43 strips: three tiles of 15), row groups
// likewise; CTAs of up to `max_threads` threads.  `lanes`: streams of a staged element.
template <int KD, int KH, int KW>
inline TileGeo plan(const Geo& g, int R, int max_threads, int lanes) {
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
    int pitch = V * (t.NS + 2);      // a quad more on either side
    if (lanes == 2) pitch = (pitch + 7) / 8 * 8;      // whole pairs of swizzled chunks
    t.pitch = lanes * pitch;
    t.plane = t.rows * t.pitch;
    t.chunks = t.rows * t.planes * (t.NS + 2);
    t.table = (t.chunks + 3) / 4 * 4;
    t.threads = (t.NS * t.NP * t.TD + 31) / 32 * 32;
    return t;
}

// The staged quads of a tile, decoded once per CTA: plane | row << 8 | quad << 24.  Columns begin one quad
// left of the tile, so that quads are whole vectors where rows are.
__device__ __forceinline__ void make_chunks(unsigned* tab, const TileGeo& t) {
    const int per_row = t.NS + 2;
    for (int e = threadIdx.x; e < t.chunks; e += blockDim.x) {
        const int rr = e / per_row, pl = rr / t.rows;
        tab[e] = (unsigned)pl | (unsigned)(rr - pl * t.rows) << 8 | (unsigned)(e - rr * per_row) << 24;
    }
}
// Offset of such a quad inside its channel, for the tile that begins at (d0, h0, w0); -1 outside the volume.
template <int KD, int KH>
__device__ __forceinline__ int quad_at(const TileGeo& t, unsigned code, int d0, int h0, int w0) {
    const int d = d0 - KD / 2 + (int)(code & 255u), h = h0 - KH / 2 + (int)((code >> 8) & 0xffffu), w = w0 - V + V * (int)(code >> 24);
    return (unsigned)d < (unsigned)t.D && (unsigned)h < (unsigned)t.H && (unsigned)w < (unsigned)t.W ? (d * t.H + h) * t.W + w : -1;
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void landed() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ f32x2 dup(float v) { return pack2(v, v); }
// Origin of a tile.
struct Origin {
    int d0, h0, w0;
    __device__ __forceinline__ Origin(const TileGeo& t, int tile, int R) {
        const int q = tile / t.ntw;
        w0 = (tile - q * t.ntw) * t.NS * V;
        d0 = q / t.nth * t.TD;
        h0 = q % t.nth * t.NP * R;
    }
};
// This thread's place in any tile.
struct Spot {
    int strip, group, dz;
    bool any;
    __device__ __forceinline__ Spot(const TileGeo& t) {
        const int q = threadIdx.x / t.NS;
        strip = threadIdx.x - q * t.NS;
        dz = q / t.NP;
        group = q - dz * t.NP;
        any = dz < t.TD;
        if (!any) { dz = 0; group = 0; strip = 0; }
    }
};

template <typename T>
__device__ __forceinline__ void load_strip(const T* p, float (&v)[V]) {
    const float4 q = dw4::load4<T, true>(p, V);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <typename T>
__device__ __forceinline__ void store_strip(T* p, const float (&v)[V]) {
    dw4::store4<T, true>(p, V, make_float4(v[0], v[1], v[2], v[3]));
}

// ---- A and K ----------------------------------------------------------------------------------
//   kForward   A of x and t1: out = (s * n) / d
//   kRatio     A of x and t1: gnum, gden and the direct term
//   kSource    A of gt1, two tiles: gz (in place on the direct term) and the bias-gradient sums
//   kTerm      K of the source, two tiles: t1
//   kBack      K of gden and gnum: gt1 and gx
enum Role { kForward = 0, kRatio = 1, kSource = 2, kTerm = 3, kBack = 4 };

struct ConvParams {
    TileGeo t;
    const void* in[2];                   // the streams' tensors (kSource, kTerm: in[0] alone; kBack: either may be NULL)
    const void* z; const void* gout;     // kForward, kRatio, kSource; kRatio
    const float* h; const float* bias;
    void* out;                           // kForward: out; kRatio: direct term (or NULL); kSource: gz (in/out); kTerm: t1; kBack: gx
    float* gnum; float* gden;            // kRatio
    float* gt1;                          // kBack
    float* gb_partial;                   // kSource: [g][block][unit][CB] bias-gradient sums, or NULL
    float eps;
    int relu, cb, blocks, units;         // CB; blocks of CB output channels; tiles (pairs of tiles) of a group, all samples
};

// A thread has R rows x CB channels: eight, 32 sums of either stream, or four where the grid is small (see plan_conv).
// Strips whose operands a thread of A loads at once (see the epilogue), as far as registers go without spilling.
template <int ROLE, int CB, int R> __host__ __device__ constexpr int conv_batch() {
    return R * CB < 8 ? R * CB : 8 / (ROLE == kForward ? (CB == 1 ? 1 : 2) : ROLE == kRatio && CB > 1 ? 4 : 2);
}
// CTAs of 128 threads a multiprocessor holds: four, of 128 registers; the compiler needs more for one instance (400 bytes
// of spills, 22.4 us for 17.6 at 32 groups of 2 channels and sources, 4 x 64^2).
template <int ROLE, int KH, int CB, int R> __host__ __device__ constexpr int conv_ctas() { return ROLE == kRatio && KH == 5 && CB == 2 && R == 4 ? 3 : 4; }

template <typename T, int KD, int KH, int KW, int ROLE, int CB, int R>
__global__ void __launch_bounds__(128, conv_ctas<ROLE, KH, CB, R>()) conv_kernel(const ConvParams P) {
    constexpr bool ADJOINT = ROLE <= kSource, TWO_TILES = ROLE == kSource || ROLE == kTerm;
    constexpr int KT = KD * KH * KW, NWC = 4;     // chunks of a window
    typedef typename std::conditional<ROLE == kSource || ROLE == kBack, float, T>::type TI;
    extern __shared__ __align__(16) float smem[];
    const TileGeo& t = P.t;
    const int ntiles = t.tiles(), nin = ADJOINT ? t.m : t.sc, nout = ADJOINT ? t.sc : t.m;
    int q = blockIdx.x;
    const int unit = q % P.units; q /= P.units;
    const int cb = q % P.blocks, g = q / P.blocks;
    const int j0 = cb * CB, nch = min(CB, nout - j0);
    // the tiles of the two streams; the second one of two may be missing
    const int index[2] = {TWO_TILES ? 2 * unit : unit, TWO_TILES ? 2 * unit + 1 : unit};
    const bool have[2] = {ROLE != kBack || P.in[0] != nullptr,
                          TWO_TILES ? index[1] < t.B * ntiles : (ROLE != kBack || P.in[1] != nullptr)};
    const Origin origin[2] = {Origin(t, index[0] % ntiles, R), Origin(t, index[1] % ntiles, R)};
    const long long bg[2] = {(long long)(index[0] / ntiles) * t.G + g, (long long)(index[1] / ntiles) * t.G + g};
    const Spot spot(t);

    f32x2* w = reinterpret_cast<f32x2*>(smem);                  // [input][tap, as the window moves][CB]
    const int wfloats = (2 * nin * KT * CB + 3) / 4 * 4;
    // of every staged quad: its place in the tile (floats) | quad of its row << 24, and its offset inside a
    // channel of either stream, -1 where there is nothing to load
    unsigned* const place = reinterpret_cast<unsigned*>(smem + wfloats);
    int* const offsets = reinterpret_cast<int*>(place + t.table);
    float* const tile = smem + wfloats + (TWO_TILES ? 3 : 2) * t.table;
    TI* const raw = reinterpret_cast<TI*>(tile + t.planes * t.plane);      // [stream][quad]
    make_chunks(place, t);
    for (int e = threadIdx.x; e < t.chunks; e += blockDim.x) {     // each thread its own
        const unsigned code = place[e];
        const int c = 2 * (int)(code >> 24);
#pragma unroll
        for (int s = 0; s < (TWO_TILES ? 2 : 1); ++s) {
            offsets[s * t.table + e] = quad_at<KD, KH>(t, code, origin[s].d0, origin[s].h0, origin[s].w0);
        }
        place[e] = ((code & 255u) * t.plane + ((code >> 8) & 0xffffu) * t.pitch + ((c ^ ((c >> 3) & 1)) << 2)) | code & 0xff000000u;
    }
    auto offset = [&](int e, int s) { return have[s] ? offsets[(TWO_TILES ? s * t.table : 0) + e] : -1; };
    f32x2 acc[R][CB][V];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < CB; ++j)
#pragma unroll
            for (int v = 0; v < V; ++v) acc[r][j][v] = dup(ROLE <= kRatio ? P.eps : 0.0f);
    int chunk[NWC];                  // places of the window's chunks in a row
#pragma unroll
    for (int i = 0; i < NWC; ++i) { const int c = 2 * spot.strip + 1 + i; chunk[i] = (c ^ ((c >> 3) & 1)) << 2; }

    // Quads come by cp.async, each thread its own, while the channel before is swept, and are then interleaved: a
    // quad of either stream makes two chunks of two pairs.
    const TI* const base[2] = {reinterpret_cast<const TI*>(P.in[0]) + bg[0] * nin * t.SP,
                               reinterpret_cast<const TI*>(P.in[TWO_TILES ? 0 : 1]) + bg[1] * nin * t.SP};
    const TI* const any = reinterpret_cast<const TI*>(P.in[0] ? P.in[0] : P.in[1]);
    auto request = [&](int i) {
        TI* q = raw + V * threadIdx.x;
        for (int e = threadIdx.x; e < t.chunks; e += blockDim.x, q += V * blockDim.x) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int off = offset(e, s);
                const unsigned a = (unsigned)__cvta_generic_to_shared(q + s * V * t.table);
                const TI* p = off >= 0 ? base[s] + i * t.SP + off : any;
                if (sizeof(TI) == 4)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(p), "r"(off >= 0 ? 16 : 0) : "memory");
                else
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(a), "l"(p), "r"(off >= 0 ? 8 : 0) : "memory");
            }
        }
        commit();
    };
    auto fill = [&](int i) {
        const float b = ROLE == kTerm && P.bias ? P.bias[g * t.sc + i] : 0.0f;
        landed<0>();
        const TI* q = raw + V * threadIdx.x;
        for (int e = threadIdx.x; e < t.chunks; e += blockDim.x, q += V * blockDim.x) {
            const unsigned code = place[e];
            float4 v[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                v[s] = dw4::to_float4(*reinterpret_cast<const dw4::Raw4<TI>*>(q + s * V * t.table));
                if (ROLE == kTerm && offset(e, s) >= 0) {    // the source: bias and ReLU on what is inside the volume
                    float q4[V] = {v[s].x, v[s].y, v[s].z, v[s].w};
#pragma unroll
                    for (int k = 0; k < V; ++k) {
                        q4[k] += b;
                        if (P.relu) q4[k] = fmaxf(q4[k], 0.0f);
                    }
                    v[s] = make_float4(q4[0], q4[1], q4[2], q4[3]);
                }
            }
            const int at = code & 0xffffffu;         // of the first chunk; the second is its neighbour
            *reinterpret_cast<float4*>(tile + at) = make_float4(v[0].x, v[1].x, v[0].y, v[1].y);
            *reinterpret_cast<float4*>(tile + (at ^ 4)) = make_float4(v[0].z, v[1].z, v[0].w, v[1].w);
        }
    };
    request(0);            // before the filter: a thread needs its own part of the tables alone
    for (int e = threadIdx.x; e < nin * KT * CB; e += blockDim.x) {
        const int j = e % CB, tau = (e / CB) % KT, i = e / (CB * KT);
        float v = 0.0f;
        if (j < nch)
            v = ADJOINT ? P.h[(((long long)g * t.m + i) * t.sc + j0 + j) * KT + KT - 1 - tau]
                        : P.h[(((long long)g * t.m + j0 + j) * t.sc + i) * KT + tau];
        w[e] = dup(v);
    }
    for (int i = 0; i < nin; ++i) {
        fill(i);
        if (i + 1 < nin) request(i + 1);
        __syncthreads();
#pragma unroll 1
        for (int kd = spot.any ? 0 : KD; kd < KD; ++kd) {
            const float* p = tile + (spot.dz + kd) * t.plane + spot.group * R * t.pitch;
            const f32x2* wk = w + (i * KT + kd * KH * KW) * CB;
#pragma unroll
            for (int rr = 0; rr < R + KH - 1; ++rr) {
                asm volatile("" ::: "memory");   // the weights are read again for each row: kept, they spill
                f32x2 win[2 * NWC];
#pragma unroll
                for (int c = 0; c < NWC; ++c) {
                    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(p + rr * t.pitch + chunk[c]);
                    win[2 * c] = u.x; win[2 * c + 1] = u.y;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int kh = rr - r;
                    if (kh < 0 || kh >= KH) continue;
#pragma unroll
                    for (int kw = 0; kw < KW; ++kw) {
                        f32x2 wj[CB];
                        if constexpr (CB == 1) {
                            wj[0] = wk[kh * KW + kw];
                        } else {
#pragma unroll
                            for (int j = 0; j < CB / 2; ++j) {
                                const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(wk + (kh * KW + kw) * CB + 2 * j);
                                wj[2 * j] = u.x; wj[2 * j + 1] = u.y;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < CB; ++j)
#pragma unroll
                            for (int v = 0; v < V; ++v) fma2(acc[r][j][v], win[v + kw + 2 - KW / 2], wj[j]);
                    }
                }
            }
        }
        if (i + 1 < nin) __syncthreads();    // the tile may be filled again
    }

    float gbs[CB];
#pragma unroll
    for (int j = 0; j < CB; ++j) gbs[j] = 0.0f;
#pragma unroll
    for (int s = 0; s < (TWO_TILES ? 2 : 1); ++s) {
        const int d = origin[s].d0 + spot.dz, wcol = origin[s].w0 + V * spot.strip, h0 = origin[s].h0 + spot.group * R;
        if (!spot.any || !have[TWO_TILES ? s : 0] && ROLE != kBack || d >= t.D || wcol >= t.W) continue;
        if constexpr (!ADJOINT) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (h0 + r >= t.H) continue;
                const long long off = ((long long)d * t.H + h0 + r) * t.W + wcol;
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    if (j >= nch) continue;
                    const long long e = (bg[s] * nout + j0 + j) * t.SP + off;
                    float lo[V], up[V];
#pragma unroll
                    for (int v = 0; v < V; ++v) unpack2(acc[r][j][v], lo[v], up[v]);
                    if (ROLE == kTerm) {
                        store_strip<T>(reinterpret_cast<T*>(P.out) + e, s ? up : lo);
                    } else {
                        if (P.gt1) store_strip<float>(P.gt1 + e, lo);
                        if (P.out) store_strip<T>(reinterpret_cast<T*>(P.out) + e, up);
                    }
                }
            }
            continue;
        }
        // Strips by rows, then channels.  What a batch of them reads is asked for ahead of its first store, or each would wait
        // for the memory in turn: at 8 groups of one channel, 4 x 20x44, 3x3, 7.5 -> 6.3 us for the forward's A and 11.3 -> 6.8
        // for the source gradient's.
        constexpr int STRIPS = R * CB, BATCH = conv_batch<ROLE, CB, R>();
        const long long e0 = (bg[s] * nout + j0) * t.SP + ((long long)d * t.H + h0) * t.W + wcol;
        auto here = [&](int i) { return h0 + i / CB < t.H && i % CB < nch; };
        auto at = [&](int i) { return e0 + (long long)(i % CB) * t.SP + (i / CB) * t.W; };
#pragma unroll
        for (int i0 = 0; i0 < STRIPS; i0 += BATCH) {
            float bj[CB];
#pragma unroll
            for (int j = 0; j < CB; ++j) bj[j] = P.bias && j < nch ? P.bias[g * t.sc + j0 + j] : 0.0f;
            dw4::Raw4<T> zr[BATCH], gr[BATCH];       // z; gout (kRatio) or the direct term (kSource)
#pragma unroll
            for (int i = i0; i < i0 + BATCH; ++i) {
                if (!here(i)) continue;
                zr[i - i0] = dw4::load4_raw<T, true>(reinterpret_cast<const T*>(P.z) + at(i), V);
                if (ROLE != kForward)
                    gr[i - i0] = dw4::load4_raw<T, true>(reinterpret_cast<const T*>(ROLE == kRatio ? P.gout : P.out) + at(i), V);
            }
#pragma unroll
            for (int i = i0; i < i0 + BATCH; ++i) {
                if (!here(i)) continue;
                const int r = i / CB, j = i % CB;
                const long long e = at(i);
                float lo[V], up[V], out[V];
#pragma unroll
                for (int v = 0; v < V; ++v) unpack2(acc[r][j][v], lo[v], up[v]);
                const float4 z4 = dw4::to_float4(zr[i - i0]), g4 = ROLE == kForward ? z4 : dw4::to_float4(gr[i - i0]);
                const float zv[V] = {z4.x, z4.y, z4.z, z4.w}, gv[V] = {g4.x, g4.y, g4.z, g4.w};
                if (ROLE == kForward) {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float sv = zv[v] + bj[j];
                        if (P.relu) sv = fmaxf(sv, 0.0f);
                        out[v] = __fdiv_rn(sv * lo[v], up[v]);
                    }
                    store_strip<T>(reinterpret_cast<T*>(P.out) + e, out);
                } else if (ROLE == kRatio) {
                    float gn[V], gd[V];
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float sv = zv[v] + bj[j];
                        if (P.relu) sv = fmaxf(sv, 0.0f);
                        gn[v] = __fdiv_rn(gv[v] * sv, up[v]);
                        gd[v] = -__fdiv_rn(gn[v] * lo[v], up[v]);
                        out[v] = __fdiv_rn(gv[v] * lo[v], up[v]);
                    }
                    store_strip<float>(P.gnum + e, gn);
                    store_strip<float>(P.gden + e, gd);
                    if (P.out) store_strip<T>(reinterpret_cast<T*>(P.out) + e, out);
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float a = gv[v] + (s ? up[v] : lo[v]);
                        if (P.relu && !(zv[v] + bj[j] > 0.0f)) a = 0.0f;
                        out[v] = a;
                        gbs[j] += to_f32(from_f32<T>(a));      // the values as stored
                    }
                    store_strip<T>(reinterpret_cast<T*>(P.out) + e, out);
                }
            }
        }
    }
    if (ROLE == kSource && P.gb_partial) {
        __syncthreads();
        float* scratch = tile;
#pragma unroll
        for (int j = 0; j < CB; ++j) {
            const float s = block_sum(gbs[j], scratch);
            if (threadIdx.x == 0) P.gb_partial[(size_t)blockIdx.x * CB + j] = s;
        }
    }
}

// One channel's tile as single values: float32 by cp.async, which has landed after the caller's wait.  Zero
// outside the volume.
template <int KD, int KH, typename T>
__device__ __forceinline__ void stage_tile(float* dst, const T* __restrict__ src, const TileGeo& t, const unsigned* tab, const Origin& at) {
    constexpr int UC = sizeof(T) == 4 ? 1 : 4;       // bfloat16: so many loads are in flight
    for (int e0 = threadIdx.x; e0 < t.chunks; e0 += UC * blockDim.x) {
        float4 v[UC];
#pragma unroll
        for (int u = 0; u < UC; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e >= t.chunks) continue;
            const int off = quad_at<KD, KH>(t, tab[e], at.d0, at.h0, at.w0);
            if (sizeof(T) == 4) {
                const unsigned q = (unsigned)__cvta_generic_to_shared(dst + V * e);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(q), "l"(off >= 0 ? src + off : src), "r"(off >= 0 ? 16 : 0) : "memory");
            } else {
                v[u] = off >= 0 ? dw4::load4<T, true>(src + off, V) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
        if (sizeof(T) == 2) {
#pragma unroll
            for (int u = 0; u < UC; ++u)
                if (e0 + u * blockDim.x < t.chunks) *reinterpret_cast<float4*>(dst + V * (e0 + u * blockDim.x)) = v[u];
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

// Rows per thread: every window is read once for both (a filter row's window of one is the next one's of
// the other).  A thread keeps the sums of CB channels, two channels to a lane pair, decodes its place once and a
// tile once per three factor pairs.  At 8 groups of 4 channels and 8 sources, 2 x 32^3: 253 -> 141 us, 142 M -> 64 M
// instructions, of which 21 M are the multiply-adds; it was integer division and, of the rest, moves that made the
// pairs anew at each use (see make_pair2).  Six warps a multiprocessor of 204 registers; what is left is their latency.
constexpr int kCorrRows = 2, kCorrThreads = 128;

template <typename T, int KD, int KH, int KW, int CB>
__global__ void __launch_bounds__(kCorrThreads, 2) corr_kernel(const CorrParams P) {
    constexpr int KT = KD * KH * KW, R = kCorrRows, NP = CB / 2;
    extern __shared__ __align__(16) float smem[];
    const TileGeo& t = P.t;
    const int ntiles = t.tiles();
    int q = blockIdx.x;
    const int split = q % P.splits; q /= P.splits;
    const int ib = q % P.blocks; q /= P.blocks;
    const int o = q % t.m, g = q / t.m;
    const int i0 = ib * CB, nch = min(CB, t.sc - i0);
    // two of each: staged tiles, and the threads' own strips of the other factor
    const int tile_floats = t.planes * t.plane;
    unsigned* const tab = reinterpret_cast<unsigned*>(smem);
    float* const bufs = smem + t.table;
    float* const own = bufs + 2 * tile_floats + threadIdx.x * V;
    const int own_step = blockDim.x * V;
    const Spot spot(t);
    f32x2 acc[KT][NP];
#pragma unroll
    for (int k = 0; k < KT; ++k)
#pragma unroll
        for (int j = 0; j < NP; ++j) acc[k][j] = dup(0.0f);
    float bj[CB];
#pragma unroll
    for (int j = 0; j < CB; ++j) bj[j] = P.bias && j < nch ? P.bias[g * t.sc + i0 + j] : 0.0f;

    // this CTA's share: every splits-th tile of the batch, three factor pairs each
    const int work = t.B * ntiles;
    auto request = [&](int unit, int pair, int parity) {        // parity: of the step; the tables' is the tile's
        const Origin at(t, unit % ntiles, R);
        const long long bg = (long long)(unit / ntiles) * t.G + g, base = (bg * t.m + o) * t.SP;
        float* dst = bufs + parity * tile_floats;
        if (pair == 2) stage_tile<KD, KH>(dst, P.gt1 + base, t, tab, at);
        else stage_tile<KD, KH>(dst, reinterpret_cast<const T*>(pair ? P.x : P.t1) + base, t, tab, at);
        if (pair < 2 || sizeof(T) == 4) {
            const int wcol = at.w0 + V * spot.strip, d = at.d0 + spot.dz;
            const float* src = pair == 0 ? P.gden : pair == 1 ? P.gnum : reinterpret_cast<const float*>(P.z);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int h = at.h0 + spot.group * R + r;
                const bool here = spot.any && d < t.D && h < t.H && wcol < t.W;
                const float* row = here ? src + (bg * t.sc + i0) * t.SP + ((long long)d * t.H + h) * t.W + wcol : P.gden;
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    const unsigned a = (unsigned)__cvta_generic_to_shared(own + ((parity * R + r) * CB + j) * own_step);
                    const bool ok = here && j < nch;
                    const float* p = ok ? row + j * t.SP : P.gden;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(p), "r"(ok ? 16 : 0) : "memory");
                }
            }
        }
        commit();
    };
    make_chunks(tab, t);
    __syncthreads();
    if (split < work) request(split, 0, 0);
    int parity = 0;
    for (int unit = split; unit < work; unit += P.splits) {
        const Origin at(t, unit % ntiles, R);
        const int wcol = at.w0 + V * spot.strip, d = at.d0 + spot.dz;
#pragma unroll 1
        for (int pair = 0; pair < 3; ++pair, parity ^= 1) {
            const int next = pair < 2 ? unit : unit + P.splits;
            __syncthreads();       // the other buffer has been read
            if (next < work) { request(next, pair < 2 ? pair + 1 : 0, parity ^ 1); landed<1>(); } else landed<0>();
            const float* tile = bufs + parity * tile_floats;
            f32x2 a[R][NP][V];         // channel pairs
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float av[CB][V];
                const int h = at.h0 + spot.group * R + r;
                const bool here = spot.any && d < t.D && h < t.H && wcol < t.W;
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    if (pair < 2 || sizeof(T) == 4) {
                        const float4 f = *reinterpret_cast<const float4*>(own + ((parity * R + r) * CB + j) * own_step);
                        av[j][0] = f.x; av[j][1] = f.y; av[j][2] = f.z; av[j][3] = f.w;
                    } else {
#pragma unroll
                        for (int v = 0; v < V; ++v) av[j][v] = 0.0f;
                        if (here && j < nch)
                            load_strip<T>(reinterpret_cast<const T*>(P.z) + (((long long)(unit / ntiles) * t.G + g) * t.sc + i0 + j) * t.SP +
                                              ((long long)d * t.H + h) * t.W + wcol, av[j]);
                    }
                    if (pair == 2) {
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            av[j][v] += bj[j];
                            if (P.relu) av[j][v] = fmaxf(av[j][v], 0.0f);
                            if (!here || j >= nch) av[j][v] = 0.0f;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < NP; ++j)
#pragma unroll
                    for (int v = 0; v < V; ++v) a[r][j][v] = dw4::make_pair2(av[2 * j][v], av[2 * j + 1][v]);
            }
            __syncthreads();       // everybody's part of the tile has landed
            if (!spot.any) continue;
#pragma unroll
            for (int kd = 0; kd < KD; ++kd) {
                const float* p = tile + (spot.dz + KD - 1 - kd) * t.plane + spot.group * R * t.pitch + V * spot.strip;
#pragma unroll
                for (int rr = 0; rr < R + KH - 1; ++rr) {
                    float c[12];
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        const float4 f = *reinterpret_cast<const float4*>(p + rr * t.pitch + 4 * i);
                        c[4 * i] = f.x; c[4 * i + 1] = f.y; c[4 * i + 2] = f.z; c[4 * i + 3] = f.w;
                    }
                    f32x2 c2[V + KW - 1];
#pragma unroll
                    for (int i = 0; i < V + KW - 1; ++i) c2[i] = dup(c[i + V - KW / 2]);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int kh = r + KH - 1 - rr;
                        if (kh < 0 || kh >= KH) continue;
#pragma unroll
                        for (int kw = 0; kw < KW; ++kw)
#pragma unroll
                            for (int j = 0; j < NP; ++j)
#pragma unroll
                                for (int v = 0; v < V; ++v)
                                    fma2(acc[(kd * KH + kh) * KW + kw][j], a[r][j][v], c2[KW - 1 - kw + v]);
                    }
                }
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
        for (int j = 0; j < NP; ++j) {
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

// gh[g*m + o][i][tau] = sum over splits; one thread per element.
static __global__ void __launch_bounds__(128) corr_sum_kernel(const float* __restrict__ partial, int GM, int sc, int blocks, int CB,
                                                       int splits, int KT, float* __restrict__ gh) {
    const int e = blockIdx.x * 128 + threadIdx.x;
    if (e >= GM * sc * KT) return;
    const int tau = e % KT, i = (e / KT) % sc, go = e / (KT * sc);
    const float* p = partial + ((size_t)(go * blocks + i / CB) * splits) * KT * CB + tau * CB + i % CB;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int k = 0;
    for (; k + 4 <= splits; k += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += p[(size_t)(k + u) * KT * CB];
    for (; k < splits; ++k) s[0] += p[(size_t)k * KT * CB];
    gh[e] = (s[0] + s[1]) + (s[2] + s[3]);
}

// gb[g*sc + i] = sum over the units of a group; one warp per channel, lanes in a fixed partition.
static __global__ void __launch_bounds__(128) gb_sum_kernel(const float* __restrict__ partial, int G, int sc, int blocks, int CB,
                                                     int units, float* __restrict__ gb) {
    const int ch = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (ch >= G * sc) return;
    const int g = ch / sc, i = ch % sc;
    const float* p = partial + ((size_t)g * blocks + i / CB) * units * CB + i % CB;
    float s = 0.0f;
    for (int k = lane; k < units; k += 32) s += p[(size_t)k * CB];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) gb[ch] = s;
}

// ---- host side ------------------------------------------------------------------------------
// Rows and tensors of whole vectors: others would come by elements, and took 1.1 - 1.4 times as long as with the
// tile kernels (5 x 37x203 and 13x25x19, one to sixteen channels a group).  On whole vectors 836 updates of 64 to 65536
// voxels, one to sixteen channels a group, take 1 / 2.27 of the tile kernels' device time forward and 1 / 1.62 backward in the
// mean; two forwards take longer, by 3 %.
inline bool covers(const Geo& g) { return g.W % V == 0; }
template <typename T> inline bool whole(std::initializer_list<const void*> tensors) {
    for (const void* p : tensors)
        if ((uintptr_t)p % (V * sizeof(T))) return false;
    return true;
}

inline size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

// Output channels per thread: eight where they fill, else four (12 channels: three blocks), two or one.
inline int block_of(int channels) { return channels > 4 && (channels % 8 == 0 || channels % 8 > 4) ? 8 : channels > 2 ? 4 : channels; }
inline int corr_block(const Geo& g) { return g.sc > 2 ? 4 : 2; }

struct ConvPlan { TileGeo t; int cb, rows, blocks, units, threads; long long grid; size_t smem; };

// `threads`: of a CTA, those of the tile or more.
// The CTA size (tiles of as many strips) of least expected time: instructions of a CTA and channel, its sweep
// and its staged quads, times the CTAs of the fullest multiprocessor, which few warps leave waiting (by 6 /
// warps; as many as fit its shared memory: counted so, the training step above took 489 us for 501).
template <int KD, int KH, int KW>
inline ConvPlan plan_conv(const Geo& g, bool adjoint, bool two_tiles) {
    const int nin = adjoint ? g.m : g.sc, nout = adjoint ? g.sc : g.m;
    auto shape = [&](int cb, int rows, int threads) {
        ConvPlan p;
        p.t = plan<KD, KH, KW>(g, rows, threads, 2);
        p.cb = cb; p.rows = rows; p.blocks = (nout + cb - 1) / cb;
        const long long tiles = (long long)p.t.tiles() * g.B;
        p.units = (int)(two_tiles ? (tiles + 1) / 2 : tiles);
        p.grid = (long long)g.G * p.blocks * (two_tiles ? (tiles + 1) / 2 : tiles);
        p.smem = sizeof(float) * ((2 * (size_t)nin * g.KT * cb + 3) / 4 * 4 + (size_t)(two_tiles ? 3 : 2) * p.t.table +
                                  (size_t)p.t.planes * p.t.plane + 2 * V * (size_t)p.t.table);
        p.threads = p.t.threads;
        return p;
    };
    ConvPlan best;
    double least = -1.0;
    const int cb = block_of(nout);
    for (int threads = cb >= 4 ? 128 : 64; threads >= 32; threads /= 2) {
        const ConvPlan p = shape(cb, 8 / cb, threads);
        if (p.smem > 220 * 1024 && threads > 32) continue;
        const int warps = p.t.threads / 32;
        const double cta = warps * 1.25 * g.KT * 8 * V + p.t.chunks / 32.0 * 30.0;
        const long long per_sm = (p.grid + num_sms() - 1) / num_sms();
        const long long fit = std::max((size_t)1, (size_t)225 * 1024 / (p.smem + 1024));
        const double resident = (double)std::min(std::min(per_sm, fit) * warps, 16LL);
        const double time = cta * (double)per_sm * (1.0 + 6.0 / resident);
        if (least < 0 || time < 0.97 * least) { least = time; best = p; }
    }
    // Where every CTA has a multiprocessor to itself, what counts is how long a thread takes.
    if (best.grid <= num_sms()) {
        // Half as much per thread: half of the rows, or of eight channels.  836 updates of 64 to 65536 voxels, most of which
        // have such grids: forward 1.23 times as fast in the mean, backward 1.18 (4 groups of 4 channels and 16 sources, 20x44,
        // 5x5, backward: 82 -> 62 us).
        const ConvPlan p = shape(std::min(cb, 4), cb == 8 ? 1 : 4 / cb, std::min(128, cb == 8 ? best.t.threads : 2 * best.t.threads));
        if (p.grid <= num_sms() && p.smem <= 220 * 1024) best = p;
        // Warps that only stage: one that stages eight rows for each of its own alone takes longer for that than for the sweep
        // (8 groups of one channel, 64^2, 3x3, forward: 18.0 -> 12.1 us, with the batches of the epilogue).  (Of several CTAs
        // the same warps sweep, and meet on the same schedulers: 16 groups of 4, 16 x 32^2, 5x5, A: 29 us for 23.)
        while (best.threads < 128 && best.t.chunks > 2 * best.threads) best.threads += 32;
    }
    return best;
}

template <int KD, int KH, int KW>
inline TileGeo plan_corr(const Geo& g) { return plan<KD, KH, KW>(g, kCorrRows, kCorrThreads, 1); }

// CTAs per (group, output channel, block of source channels) of corr_kernel: as many tiles as one of them
// walks, and its combine (about one tile's worth), times the rounds of two CTAs per multiprocessor.  Of those that
// leave a CTA as many tiles only the fewest is a candidate.
inline int corr_splits(const Geo& g, const TileGeo& t) {
    const int cb = corr_block(g);
    const long long combos = (long long)g.G * g.m * ((g.sc + cb - 1) / cb), work = (long long)g.B * t.tiles(), slots = 2LL * num_sms();
    const long long most = std::min(work, std::max(1LL, 2 * slots / combos));
    long long best = 1, least = -1;
    for (long long s = 1; s <= most;) {
        const long long walked = (work + s - 1) / s, time = (combos * s + slots - 1) / slots * (walked + 1);
        if (least < 0 || time < least) { least = time; best = s; }
        if (walked == 1) break;
        s = (work + walked - 2) / (walked - 1);
    }
    return (int)best;
}

// Scratch of the backward: gnum | gden | gt1 | bias-gradient records | correlation records, and the correlation's plan.
struct BwdScratch { size_t gnum, gden, gt1, gb, corr, bytes; TileGeo tc; int splits; };

// `limit`: bytes that there are.  The correlation makes do with fewer splits to keep to them, but with half as many as it
// wants at least: false where that does not help.
template <int KD, int KH, int KW>
inline bool scratch_shape(const Geo& g, size_t limit, BwdScratch& s) {
    const size_t src = (size_t)g.B * g.G * g.sc * g.SP * sizeof(float);
    const ConvPlan pa = plan_conv<KD, KH, KW>(g, true, true);
    const int cb = corr_block(g);
    s.tc = plan_corr<KD, KH, KW>(g);
    s.gnum = 0;
    s.gden = up256(src);
    s.gt1 = s.gden + up256(src);
    s.gb = s.gt1 + up256((size_t)g.B * g.G * g.m * g.SP * sizeof(float));
    s.corr = s.gb + up256((size_t)pa.grid * pa.cb * sizeof(float));
    const size_t split = (size_t)g.G * g.m * ((g.sc + cb - 1) / cb) * g.KT * cb * sizeof(float);
    const int wanted = corr_splits(g, s.tc);
    s.splits = wanted;
    if (s.corr + up256(wanted * split) > limit) {
        s.splits = s.corr < limit ? (int)std::min((size_t)wanted, (limit - s.corr) / 256 * 256 / split) : 0;
        if (2 * s.splits < wanted) return false;
    }
    s.bytes = s.corr + up256(s.splits * split);
    return true;
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

template <typename T, int KD, int KH, int KW, int ROLE>
cudaError_t run_conv(const Geo& g, ConvParams& P, cudaStream_t st) {
    const ConvPlan p = plan_conv<KD, KH, KW>(g, ROLE <= kSource, ROLE == kSource || ROLE == kTerm);
    P.t = p.t; P.cb = p.cb; P.blocks = p.blocks; P.units = p.units; P.eps = g.eps;
    switch (10 * p.cb + p.rows) {
        case 81: return launch(conv_kernel<T, KD, KH, KW, ROLE, 8, 1>, p.grid, p.threads, p.smem, st, P);
        case 42: return launch(conv_kernel<T, KD, KH, KW, ROLE, 4, 2>, p.grid, p.threads, p.smem, st, P);
        case 41: return launch(conv_kernel<T, KD, KH, KW, ROLE, 4, 1>, p.grid, p.threads, p.smem, st, P);
        case 24: return launch(conv_kernel<T, KD, KH, KW, ROLE, 2, 4>, p.grid, p.threads, p.smem, st, P);
        case 22: return launch(conv_kernel<T, KD, KH, KW, ROLE, 2, 2>, p.grid, p.threads, p.smem, st, P);
        case 18: return launch(conv_kernel<T, KD, KH, KW, ROLE, 1, 8>, p.grid, p.threads, p.smem, st, P);
        default: return launch(conv_kernel<T, KD, KH, KW, ROLE, 1, 4>, p.grid, p.threads, p.smem, st, P);
    }
}

template <typename T, int KD, int KH, int KW>
cudaError_t forward_shape(const Geo& g, const T* x, const T* z, const float* h, const float* bias, T* out, T* t1,
                          cudaStream_t st) {
    ConvParams K{};
    K.in[0] = z; K.out = t1; K.h = h; K.bias = bias; K.relu = g.relu;
    const cudaError_t e = run_conv<T, KD, KH, KW, kTerm>(g, K, st);
    if (e != cudaSuccess) return e;
    ConvParams A{};
    A.in[0] = x; A.in[1] = t1; A.z = z; A.h = h; A.bias = bias; A.out = out; A.relu = g.relu;
    return run_conv<T, KD, KH, KW, kForward>(g, A, st);
}

template <typename T, int KD, int KH, int KW>
cudaError_t backward_shape(const Geo& g, const T* x, const T* z, const T* t1, const float* h, const float* bias,
                           const T* gout, T* gx, T* gz, float* gh, float* gb, void* ws, const BwdScratch& sc, cudaStream_t st) {
    float* gnum = (float*)((char*)ws + sc.gnum);
    float* gden = (float*)((char*)ws + sc.gden);
    float* gt1 = (float*)((char*)ws + sc.gt1);
    ConvParams A{};
    A.in[0] = x; A.in[1] = t1; A.z = z; A.gout = gout; A.h = h; A.bias = bias; A.out = gz; A.gnum = gnum; A.gden = gden; A.relu = g.relu;
    cudaError_t e = run_conv<T, KD, KH, KW, kRatio>(g, A, st);
    if (e != cudaSuccess) return e;
    if (gz || gh || gx) {
        ConvParams K{};
        K.h = h;
        if (gz || gh) { K.in[0] = gden; K.gt1 = gt1; }
        if (gx) { K.in[1] = gnum; K.out = gx; }
        e = run_conv<T, KD, KH, KW, kBack>(g, K, st);
        if (e != cudaSuccess) return e;
    }
    if (gh) {
        CorrParams C{};
        C.t = sc.tc;
        const int cb = corr_block(g);
        C.gden = gden; C.gnum = gnum; C.z = z; C.bias = bias; C.t1 = t1; C.x = x; C.gt1 = gt1;
        C.partial = (float*)((char*)ws + sc.corr); C.relu = g.relu; C.blocks = (g.sc + cb - 1) / cb;
        C.splits = sc.splits;
        const size_t rec = (size_t)(C.t.threads / 32) * g.KT * cb;
        const size_t til = (size_t)C.t.table + 2 * ((size_t)C.t.planes * C.t.plane + (size_t)kCorrRows * cb * V * C.t.threads);
        const long long grid = (long long)g.G * g.m * C.blocks * C.splits;
        e = cb == 4 ? launch(corr_kernel<T, KD, KH, KW, 4>, grid, C.t.threads, sizeof(float) * std::max(rec, til), st, C)
                    : launch(corr_kernel<T, KD, KH, KW, 2>, grid, C.t.threads, sizeof(float) * std::max(rec, til), st, C);
        if (e != cudaSuccess) return e;
        const int n = g.G * g.m * g.sc * g.KT;
        corr_sum_kernel<<<(n + 127) / 128, 128, 0, st>>>(C.partial, g.G * g.m, g.sc, C.blocks, cb, C.splits, g.KT, gh);
        launched();
    }
    if (gz) {
        ConvParams S{};
        S.in[0] = gt1; S.z = z; S.h = h; S.bias = bias; S.out = gz; S.relu = g.relu;
        S.gb_partial = gb ? (float*)((char*)ws + sc.gb) : nullptr;
        e = run_conv<T, KD, KH, KW, kSource>(g, S, st);
        if (e != cudaSuccess) return e;
        if (gb) {
            gb_sum_kernel<<<(g.G * g.sc + 3) / 4, 128, 0, st>>>(S.gb_partial, g.G, g.sc, S.blocks, S.cb, S.units, gb);
            launched();
        }
    }
    return cudaGetLastError();
}

}  // namespace pairs
}  // namespace ndc
