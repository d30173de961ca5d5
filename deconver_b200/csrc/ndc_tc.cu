// Host side of the tensor-core forward (ndc_tc.cuh): tiling and launches.
#include "ndc_tc.cuh"

#include "ndc_tc_host.h"

namespace ndc {
namespace tc {
namespace {

constexpr size_t kSmemPerCta = 100 * 1024;     // two CTAs share a multiprocessor

// Bands and chunks.  A band's rows fill MT MMA tiles of 128 blocks as well as they can; a chunk is as
// deep as shared memory (and, for the source kernel, TMEM) allows, but not so deep that the grid would
// leave multiprocessors idle.  Of the tile counts the one with the best product of useful MMA rows and
// of staged rows and planes that are not halo is taken.
template <int KD, int KH, int KW>
bool plan(const Geo& g, int tensors, size_t fixed, bool source, Band& b, size_t& smem) {
    constexpr int PH = KH / 2, PW = KW / 2, PD = KD / 2;
    b.C = g.G; b.D = g.D; b.H = g.H; b.W = g.W; b.Wv = g.Wv; b.Wo = g.Wo; b.SP = g.SP; b.eps = g.eps; b.relu = g.relu;
    b.NB = (g.Wv + 7) / 8;
    b.PB = (g.Wv + PW + 7) / 8;
    double best = 0.0;
    for (int most = 1; most <= (KD > 1 ? 2 : 4); ++most) {
        int th = std::min(g.H, most * MB / b.PB);
        if (th < 1) continue;
        const int nth = (g.H + th - 1) / th;
        th = (g.H + nth - 1) / nth;
        const int mt = (th * b.PB + MB - 1) / MB;
        const size_t plane = (size_t)tensors * (th + 2 * PH) * b.PB * 16, slack = 16 * (size_t)(mt * MB + 1);
        if (fixed + slack + plane * (1 + 2 * PD) > kSmemPerCta) continue;
        int dc = 1;
        if (KD > 1) {
            dc = std::min((int)((kSmemPerCta - fixed - slack) / plane) - 2 * PD, 16);
            if (source) dc = std::min(dc, 32 / mt - KD - 2);          // 256 accumulator columns
            const long long per = (long long)g.B * g.G * nth;
            while (dc > 4 && per * ((g.D + dc - 1) / dc) < 2 * 148) --dc;
            dc = std::min(dc, g.D);
            if (dc < 1) continue;
        }
        const int ndc = KD > 1 ? (g.D + dc - 1) / dc : g.D;
        if (KD > 1) dc = (g.D + ndc - 1) / ndc;
        const double use = (double)g.H * g.Wv / (8.0 * nth * mt * MB);
        const double score = use * th / (th + PH) * dc / (dc + PD);
        if (score > best * 1.02) {
            best = score;
            b.MT = mt; b.TH = th; b.nth = nth; b.DC = dc; b.ndc = ndc;
            smem = fixed + plane * (dc + 2 * PD) + 16 * (size_t)slack_blocks(b);
        }
    }
    return best > 0.0;
}

// Share of the MMAs' rows that are voxels of the volume.
double useful(const Band& b) { return (double)b.H * b.Wv / (8.0 * b.nth * b.MT * MB); }

template <int KD, int KH, int KW> constexpr size_t adjoint_fixed() { return kHeader + (size_t)KD * KH * SC * 8 * 32; }
template <int KD, int KH, int KW> constexpr size_t source_fixed() {
    constexpr int PD = KD / 2, PH = KH / 2, PW = KW / 2;
    return kHeader + ((PD + 1) * (PD + 1) * (PH + 1) * (PH + 1) * (PW + 1) * (PW + 1) * 4 + 127) / 128 * 128 +
           (size_t)SC * KH * (KD > 1 ? 32 : 16) * 32;
}

template <int KD, int KH, int KW>
bool plans(const Geo& g, Band& ba, size_t& sa, Band& bs, size_t& ss) {
    if (!plan<KD, KH, KW>(g, 2, adjoint_fixed<KD, KH, KW>(), false, ba, sa)) return false;
    return plan<KD, KH, KW>(g, SC, source_fixed<KD, KH, KW>(), true, bs, ss);
}

template <typename K, typename P, typename... More>
cudaError_t launch(K kern, const Band& b, const Geo& g, size_t smem, cudaStream_t st, const P& p, More... more) {
    const long long grid = (long long)g.B * g.G * b.nth * b.ndc;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)grid, kThreads, smem, st>>>(p, more...);
    launched();
    return cudaGetLastError();
}

template <int KD, int KH, int KW>
cudaError_t run(const Geo& g, const bf16* x, const bf16* z, const float* h, const float* bias, bf16* out, bf16* t1, cudaStream_t st) {
    AdjointArgs A;
    SourceArgs S;
    size_t sa, ss;
    if (!plans<KD, KH, KW>(g, A.b, sa, S.b, ss)) return cudaErrorInvalidConfiguration;
    A.x = x; A.t1 = t1; A.z = z; A.out = out; A.h = h; A.bias = bias;
    S.z = z; S.t1 = t1; S.h = h; S.bias = bias;
    auto on16 = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    const bool wide = g.W % 8 == 0 && on16(x) && on16(z) && on16(t1);
    const int cols = tmem_cols(S.b.MT * source_cols<KD>(S.b.DC));
    cudaError_t e = wide ? launch(tc_source_kernel<KD, KH, KW, kWide>, S.b, g, ss, st, S, cols)
                         : launch(tc_source_kernel<KD, KH, KW, kQuad>, S.b, g, ss, st, S, cols);
    if (e != cudaSuccess) return e;
    if (g.Wo != g.W) return launch(tc_adjoint_kernel<KD, KH, KW, kPaddedOut>, A.b, g, sa, st, A);
    return wide && on16(out) ? launch(tc_adjoint_kernel<KD, KH, KW, kWide>, A.b, g, sa, st, A)
                             : launch(tc_adjoint_kernel<KD, KH, KW, kQuad>, A.b, g, sa, st, A);
}

template <int KD, int KH, int KW>
bool worth(const Geo& g) {
    Band a, s;
    size_t sa, ss;
    return plans<KD, KH, KW>(g, a, sa, s, ss) && std::min(useful(a), useful(s)) >= 0.25;
}

}  // namespace

bool covers(const Geo& g) {
    if (g.m != 1 || g.sc != SC || g.W % 4 || g.SP >= (1LL << 29)) return false;
    if (g.kD == 3 && g.kH == 3 && g.kW == 3) return worth<3, 3, 3>(g);
    if (g.kD == 1 && g.kH == 5 && g.kW == 5) return worth<1, 5, 5>(g);
    if (g.kD == 1 && g.kH == 3 && g.kW == 3) return worth<1, 3, 3>(g);
    return false;
}

cudaError_t forward(const Geo& g, const bf16* x, const bf16* z, const float* h, const float* bias, bf16* out, bf16* t1, cudaStream_t st) {
    if (g.kD == 3) return run<3, 3, 3>(g, x, z, h, bias, out, t1, st);
    if (g.kH == 5) return run<1, 5, 5>(g, x, z, h, bias, out, t1, st);
    return run<1, 3, 3>(g, x, z, h, bias, out, t1, st);
}

unsigned wait_expired() {
    unsigned v = 0;
    (void)cudaMemcpyFromSymbol(&v, g_wait_expired, sizeof(v));
    return v;
}

}  // namespace tc
}  // namespace ndc
