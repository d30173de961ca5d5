// Host side of the tensor-core forward (ndc_tc.cuh): tiling and launches.
#include "ndc_tc.cuh"

#include "ndc_tc_host.h"

namespace ndc {
namespace tc {
namespace {

// Bands: as many rows as fill the 128 blocks of an MMA.  Chunks of planes: all of them, but for what
// the accumulators hold (`most`) and for a grid that would leave multiprocessors idle; a chunk
// stages KD - 1 planes of its neighbours.
template <int KD, int KH, int KW>
bool plan(const Geo& g, int most, Band& b) {
    b.C = g.G; b.D = g.D; b.H = g.H; b.W = g.W; b.Wv = g.Wv; b.Wo = g.Wo; b.eps = g.eps; b.relu = g.relu;
    b.NB = (g.Wv + 7) / 8;
    b.PB = (g.Wv + KW / 2 + 7) / 8;
    b.TH = std::min(g.H, std::min(MB / b.PB, kSourceStagers / b.PB - (KH - 1)));
    if (b.TH < 1) return false;
    b.nth = (g.H + b.TH - 1) / b.TH;
    b.TH = (g.H + b.nth - 1) / b.nth;
    b.nth = (g.H + b.TH - 1) / b.TH;
    // 32-bit offsets inside a band
    const long long row = KH == 1 ? (long long)g.D * g.W * g.G * SC : g.W;
    if ((b.TH + KH - 1) * row >= (1LL << 31)) return false;
    const long long per = (long long)g.B * g.G * b.nth;
    long long ndc = (g.D + most - 1) / most;
    const long long want = (4 * 148 + per - 1) / per, finest = std::max(1, g.D / (6 * (KD / 2)));
    ndc = std::max(ndc, std::min(want, finest));
    b.DC = (int)((g.D + ndc - 1) / ndc);
    b.ndc = (g.D + b.DC - 1) / b.DC;
    return true;
}

// Share of the MMAs' rows that are voxels of the volume.
double useful(const Band& b) { return (double)b.H * b.Wv / (8.0 * b.nth * MB); }

template <int KD, int KH, int KW> size_t adjoint_smem(const Band& b) {
    return kHeader + (size_t)KH * KD * SC * 8 * 32 + 16 * ((size_t)kSlots * 2 * (b.TH + KH - 1) * b.PB + slack_blocks(b));
}
template <int KD, int KH, int KW> size_t source_smem(const Band& b) {
    constexpr int PD = KD / 2, PH = KH / 2, PW = KW / 2;
    return kHeader + ((PD + 1) * (PD + 1) * (PH + 1) * (PH + 1) * (PW + 1) * (PW + 1) * 4 + 127) / 128 * 128 +
           (size_t)SC * KH * 8 * source_groups<KD>() * 32 +
           16 * ((size_t)kSlots * SC * (b.TH + KH - 1) * b.PB + slack_blocks(b));
}

template <typename K, typename P>
cudaError_t launch(K kern, int threads, const Band& b, const Geo& g, size_t smem, cudaStream_t st, const P& p) {
    const long long grid = (long long)g.B * g.G * b.nth * b.ndc;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)grid, threads, smem, st>>>(p);
    launched();
    return cudaGetLastError();
}

template <int KD, int KH, int KW>
cudaError_t run(const Geo& g, const bf16* x, const bf16* z, const float* h, const float* bias, bf16* out, bf16* t1, cudaStream_t st) {
    AdjointArgs A;
    SourceArgs S;
    if (!plan<KD, KH, KW>(g, g.D, A.b) || !plan<KD, KH, KW>(g, source_planes<KD>(), S.b)) return cudaErrorInvalidConfiguration;
    A.x = x; A.t1 = t1; A.z = z; A.out = out; A.h = h; A.bias = bias;
    S.z = z; S.t1 = t1; S.h = h; S.bias = bias;
    const size_t sa = adjoint_smem<KD, KH, KW>(A.b), ss = source_smem<KD, KH, KW>(S.b);
    auto on16 = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    const bool wide = g.W % 8 == 0 && g.Wv == g.W && on16(x) && on16(z) && on16(t1);
    cudaError_t e = wide ? launch(tc_source_kernel<KD, KH, KW, kWide>, kSourceThreads, S.b, g, ss, st, S)
                         : launch(tc_source_kernel<KD, KH, KW, kQuad>, kSourceThreads, S.b, g, ss, st, S);
    if (e != cudaSuccess) return e;
    if (g.Wo != g.W) return launch(tc_adjoint_kernel<KD, KH, KW, kPaddedOut>, AdjointShape<KD>::THREADS, A.b, g, sa, st, A);
    return wide && on16(out) ? launch(tc_adjoint_kernel<KD, KH, KW, kWide>, AdjointShape<KD>::THREADS, A.b, g, sa, st, A)
                             : launch(tc_adjoint_kernel<KD, KH, KW, kQuad>, AdjointShape<KD>::THREADS, A.b, g, sa, st, A);
}

template <int KD, int KH, int KW>
bool worth(const Geo& g) {
    Band a, s;
    return plan<KD, KH, KW>(g, g.D, a) && plan<KD, KH, KW>(g, source_planes<KD>(), s) && useful(a) >= 0.2;
}

// Image batches as volumes whose planes are the image rows and whose plane rows are the images.
Geo as_rows(const Geo& g) {
    Geo v = g;
    v.B = 1; v.D = g.H; v.H = g.B;
    v.kD = g.kH; v.kH = 1; v.pD = g.pH; v.pH = 0;
    v.SP = (long long)v.D * v.H * v.W;
    return v;
}

}  // namespace

bool covers(const Geo& g) {
    if (g.m != 1 || g.sc != SC || g.W % 4 || g.SP >= (1LL << 29)) return false;
    if (g.kD == 3 && g.kH == 3 && g.kW == 3) return worth<3, 3, 3>(g);
    if (g.kD != 1 || g.D != 1 || g.kH != g.kW) return false;
    if (g.kH == 5) return worth<5, 1, 5>(as_rows(g));
    if (g.kH == 3) return worth<3, 1, 3>(as_rows(g));
    return false;
}

cudaError_t forward(const Geo& g, const bf16* x, const bf16* z, const float* h, const float* bias, bf16* out, bf16* t1, cudaStream_t st) {
    if (g.kD == 3) return run<3, 3, 3>(g, x, z, h, bias, out, t1, st);
    if (g.kH == 5) return run<5, 1, 5>(as_rows(g), x, z, h, bias, out, t1, st);
    return run<3, 1, 3>(as_rows(g), x, z, h, bias, out, t1, st);
}

unsigned wait_expired() {
    unsigned v = 0;
    (void)cudaMemcpyFromSymbol(&v, g_wait_expired, sizeof(v));
    return v;
}

}  // namespace tc
}  // namespace ndc
