// Host side of the tensor-core forward (ndc_tc.cuh): tiling and launches.
#include "ndc_tc.cuh"

#include <atomic>
#include <mutex>

#include "ndc_tc_host.h"

namespace ndc {
namespace tc {
namespace {

// One word per device in host memory, where a kernel whose wait ran out writes 1: a call after it reads the
// word without synchronising, reports it and writes 2.  Allocated once; a launch may be the first one under
// stream capture, which forbids allocations unless the thread says that it knows what it does.
constexpr int kMaxDevices = 64;
std::atomic<unsigned*> g_expired{nullptr};

cudaError_t expired_word(unsigned*& word) {
    static std::mutex mu;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    unsigned* all = g_expired.load(std::memory_order_acquire);
    if (!all) {
        std::lock_guard<std::mutex> lock(mu);
        all = g_expired.load(std::memory_order_acquire);
        if (!all) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            if ((e = cudaThreadExchangeStreamCaptureMode(&mode)) != cudaSuccess) return e;
            void* p = nullptr;
            e = cudaHostAlloc(&p, kMaxDevices * sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped);
            const cudaError_t back = cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) return e;
            if (back != cudaSuccess) return back;
            all = static_cast<unsigned*>(p);
            for (int i = 0; i < kMaxDevices; ++i) all[i] = 0u;
            g_expired.store(all, std::memory_order_release);
        }
    }
    word = all + dev;
    return cudaSuccess;
}

// A wait for what never comes, to see that one that runs out is reported.
__global__ void probe_wait_kernel(unsigned limit, unsigned* expired) {
    __shared__ unsigned long long bar;
    const unsigned at = smem_u32(&bar);
    if (threadIdx.x == 0) {
        mbar_init(at, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (!mbar_wait(at, 0, limit) && threadIdx.x == 0) report_expired(expired);
}

// Bands: as many rows as fill the 128 blocks of an MMA; rows of images (KH = 1) of all chunks together, so that the last
// band alone is partly filled: on 46 shapes of 1 to 20 images, forward and training step, 1.10x in the mean (16 x
// 64 of 128^2, 3x3 filter, forward: 255 -> 184 us; one of 300^2: 172 -> 97).  Chunks of planes: the cut of least
// expected time, the CTAs of the fullest multiprocessor times a chunk's planes and some more (its filling of the pipeline
// and its neighbours' planes).  Two adjoint CTAs share the tensor core and need twice the time of one (4 planes more); of the
// source's two, one alone needs 0.65 of their time (7 planes more); adjoint CTAs that are alone fill the pipeline once (12
// planes) and pay each chunk's neighbours and a plane and a half between places.  Images: any cut, the coarsest within 1 %.
// Volumes: from the cut that gives every multiprocessor four CTAs, another if it is 2 % better; the adjoint of rows that are
// not whole 8-column blocks waits for its loads instead, and keeps that one.  2 x 64 volumes of 64^3: adjoint 201 -> 188 us,
// its ratio step 428 -> 394; 12 x 128 images of 60x64, 68 -> 41.
template <int KD, int KH, int KW>
bool plan(const Geo& g, bool source, Band& b) {
    b.C = g.G; b.D = g.D; b.H = g.H; b.W = g.W; b.Wv = g.Wv; b.Wo = g.Wo; b.eps = g.eps; b.relu = g.relu;
    b.NB = (g.Wv + 7) / 8;
    b.PB = source ? b.NB : (g.Wv + KW / 2 + 7) / 8;
    // The adjoint's CTAs that are alone on their multiprocessor (five depth taps) go on from place to place where there
    // are several for each: nobody else fills their gaps (16 x 64 images of 128^2: 127 -> 105 us for three each).  With one
    // each that form is 5 % slower; and of two CTAs on a multiprocessor either fills the other's gaps.
    const bool alone = !source && AdjointShape<KD>::CTAS == 1;
    const bool waits = !(g.W % 8 == 0 && g.Wv == g.W);      // for its loads, of 8 bytes
    const long long sms = num_sms(), finest = std::max(1, g.D / (6 * (KD / 2)));
    // expected time of so many places of chunks of so many planes
    auto time = [&](int planes, long long items) {
        const long long on_one = (items + sms - 1) / sms;
        if (alone) return (float)on_one * ((float)planes + (KD - 1) + 1.5f) + 12.0f;
        const float pairs = (float)(on_one / 2) + (on_one % 2 ? 0.65f : 0.0f);
        return ((float)planes + (source ? 7.0f : 4.0f)) * (source ? pairs : (float)on_one);
    };
    b.TH = std::min(MB / b.PB, kSourceStagers / b.PB - (KH - 1));
    if (b.TH < 1) return false;
    if (KH == 1) {       // bands of rows of all chunks
        const int most = b.TH;
        const long long row = (long long)g.D * g.W * g.G * SC;      // 32-bit offsets: see base_row
        float least = -1.0f;
        for (long long n = 1; n <= std::min(finest, 32LL); ++n) {
            const int planes = (int)((g.D + n - 1) / n);
            const long long chunks = (g.D + planes - 1) / planes, rows = g.H * chunks, bands = (rows + most - 1) / most;
            const float t = time(planes, (long long)g.B * g.G * bands);
            if (rows > 0x7fffffffLL || (chunks > 1 ? g.H : std::min(g.H, most)) * row >= (1LL << 31) || (least >= 0.0f && t >= 0.99f * least)) continue;
            least = t;
            b.DC = planes; b.ndc = (int)chunks;
            b.nth = (int)bands;
            b.TH = (int)((rows + bands - 1) / bands);
        }
        if (least < 0.0f) return false;
        b.nth = (int)(((long long)g.H * b.ndc + b.TH - 1) / b.TH);
        const long long items = (long long)g.B * g.G * b.nth;
        b.items = (int)std::min(items, 0x7fffffffLL);
        b.march = alone && items > sms;
        return items <= 0x7fffffffLL;
    }
    b.TH = std::min(g.H, b.TH);
    b.nth = (g.H + b.TH - 1) / b.TH;
    b.TH = (g.H + b.nth - 1) / b.nth;
    b.nth = (g.H + b.TH - 1) / b.TH;
    // 32-bit offsets inside a band
    if ((b.TH + KH - 1) * (long long)g.W >= (1LL << 31)) return false;
    const long long per = (long long)g.B * g.G * b.nth;
    long long ndc = 1;
    const long long want = (4 * sms + per - 1) / per;
    ndc = std::max(ndc, std::min(want, finest));
    if (source || !waits) {
        auto cut = [&](long long n) {
            const int planes = (int)((g.D + n - 1) / n);
            return time(planes, per * ((g.D + planes - 1) / planes));
        };
        float least = 0.98f * cut(ndc);
        const long long last = std::min(2 * ndc + 2, (long long)finest);
        for (long long n = std::max(1LL, ndc / 6), from = ndc; n <= last; ++n)
            if (n != from && cut(n) < least) { least = cut(n); ndc = n; }
    }
    b.DC = (int)((g.D + ndc - 1) / ndc);
    b.ndc = (g.D + b.DC - 1) / b.DC;
    if (per * b.ndc > 0x7fffffffLL) return false;
    b.items = (int)(per * b.ndc);
    b.march = 0;
    return true;
}

// Share of the MMAs' rows that are voxels of the volume.
template <int KH> double useful(const Band& b) {
    return KH == 1 ? (double)b.H * b.D * b.Wv / (8.0 * b.nth * b.DC * MB) : (double)b.H * b.Wv / (8.0 * b.nth * MB);
}

template <int KD, int KH, int KW> size_t adjoint_smem(const Band& b) {
    return kHeader + (size_t)KH * KD * SC * 8 * 32 + 16 * ((size_t)kSlots * 2 * (b.TH + KH - 1) * b.PB + slack_blocks(b));
}
template <int KD, int KH, int KW> size_t source_smem(const Band& b) {
    return kHeader + (size_t)SC * KH * KD * kGroup * 32 + 16 * ((size_t)kSourceSlots * 2 * SC * (b.TH + KH - 1) * b.NB + slack_blocks(b));
}

template <typename K, typename P>
cudaError_t launch(K kern, int threads, const Band& b, size_t smem, cudaStream_t st, const P& p) {
    const cudaError_t e = allow_smem(kern);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(b.march ? num_sms() : b.items), threads, smem, st>>>(p);
    launched();
    return cudaGetLastError();
}

bool on16(const void* p) { return ((uintptr_t)p & 15) == 0; }

template <int KD, int KH, int KW, int MODE, bool MARCH>
cudaError_t launch_adjoint(const Geo& g, const AdjointArgs& A, bool wide, cudaStream_t st) {
    const size_t smem = adjoint_smem<KD, KH, KW>(A.b);
    constexpr int NT = AdjointShape<KD>::THREADS;
    if (g.Wo != g.W) return launch(tc_adjoint_kernel<KD, KH, KW, kPaddedOut, MODE, MARCH>, NT, A.b, smem, st, A);
    return wide ? launch(tc_adjoint_kernel<KD, KH, KW, kWide, MODE, MARCH>, NT, A.b, smem, st, A)
                : launch(tc_adjoint_kernel<KD, KH, KW, kQuad, MODE, MARCH>, NT, A.b, smem, st, A);
}
template <int KD, int KH, int KW, int MODE>
cudaError_t launch_adjoint(const Geo& g, const AdjointArgs& A, bool wide, cudaStream_t st) {
    if constexpr (AdjointShape<KD>::CTAS == 1) {
        if (A.b.march) return launch_adjoint<KD, KH, KW, MODE, true>(g, A, wide, st);
    }
    return launch_adjoint<KD, KH, KW, MODE, false>(g, A, wide, st);
}

template <int KD, int KH, int KW>
cudaError_t run(const Geo& g, const bf16* x, const bf16* z, const float* h, const float* bias, bf16* out, bf16* t1, cudaStream_t st) {
    AdjointArgs A{};
    SourceArgs S{};
    if (!plan<KD, KH, KW>(g, false, A.b) || !plan<KD, KH, KW>(g, true, S.b)) return cudaErrorInvalidConfiguration;
    A.x = x; A.t1 = t1; A.z = z; A.out = out; A.h = h; A.bias = bias;
    S.z = z; S.t1 = t1; S.h = h; S.bias = bias;
    const size_t ss = source_smem<KD, KH, KW>(S.b);
    cudaError_t e = expired_word(S.expired);
    if (e != cudaSuccess) return e;
    A.expired = S.expired;
    const bool wide = g.W % 8 == 0 && g.Wv == g.W && on16(x) && on16(z) && on16(t1);
    e = wide ? launch(tc_source_kernel<KD, KH, KW, kWide>, kSourceThreads, S.b, ss, st, S)
             : launch(tc_source_kernel<KD, KH, KW, kQuad>, kSourceThreads, S.b, ss, st, S);
    if (e != cudaSuccess) return e;
    return launch_adjoint<KD, KH, KW, kOut>(g, A, wide && on16(out), st);
}

template <int KD, int KH, int KW>
cudaError_t run_ratio(const Geo& g, const bf16* x, const bf16* z, const bf16* t1, const float* h, const float* bias, const bf16* gout,
                      float* gnum, float* gden, bf16* direct, bool pairs, cudaStream_t st) {
    AdjointArgs A{};
    if (!plan<KD, KH, KW>(g, false, A.b)) return cudaErrorInvalidConfiguration;
    const cudaError_t e = expired_word(A.expired);
    if (e != cudaSuccess) return e;
    A.x = x; A.t1 = t1; A.z = z; A.out = direct; A.gout = gout; A.gnum = gnum; A.gden = gden; A.h = h; A.bias = bias;
    const bool wide = g.W % 8 == 0 && g.Wv == g.W && on16(x) && on16(z) && on16(t1) && on16(gout) && (!direct || on16(direct));
    if constexpr (KH == 1) {
        if (!pairs) return launch_adjoint<KD, KH, KW, kPlanar>(g, A, wide, st);
    }
    return launch_adjoint<KD, KH, KW, kPairs>(g, A, wide, st);
}

// How large a problem has to be, and how much of the MMAs' rows it has to fill, for the tensor cores to be the faster way:
// for a forward update, or (`ratio`) for the first step of its backward, whose FMA kernel is the better one of the two, so that
// its lines lie higher.  560 shapes about the lines, in CUDA graphs over more than the L2,
// against the FMA kernels: of the 399 beyond the forward's lines none takes longer (1.61x in the mean), and a backward with
// this first step takes 0.99x - 1.5x (1.14x).  The lines that cost something:
//   volumes    0.4 M group-voxels, rows of 128 at least 30 % full (16^3 fills 25 %: forward 0.84x - 1.09x, backward 0.92x - 0.97x)
//   images     0.7 M, 45 % full, 10 rows, with 5x5 filters 20 (16 x 512 of 16^2: 0.86x, 0.93x)
//   below 3 M with rows of whole quads, which the FMA kernels take fastest:
//     3x3      forward under 2 M: few rows in bands half full stay (8 x 188 of 16x32: 0.91x); ratio from 1.2 M (8 x 172 of
//              28^2: 0.97x), from 1.6 M under 20 rows (24 x 192 of 12x28, 1.55 M: 0.98x)
//     5x5      ratio from 0.85 M (16 x 64 of 28^2, 0.80 M: 0.89x), from 1.5 M in bands half full (14 x 88 of 30x36: 0.97x),
//              unless an image has 46 rows (2 x 128 of 64^2, 1.05 M: 1.09x)
//   3x3 at the widths that the FMA kernels have compile-time instances for: from 3 M, 70 % full (1 x 64 of 128^2: 0.98x); the ratio of
//              128 and 256 columns from 5.5 M (3 x 172 of 24x256: 0.97x, 2 x 44 of 256^2: 1.02x)
template <int KD, int KH, int KW>
bool worth(const Geo& g, bool ratio) {
    Band a, s;
    if (!plan<KD, KH, KW>(g, false, a) || !plan<KD, KH, KW>(g, true, s)) return false;
    const double voxels = (double)g.B * g.G * g.D * g.H * g.Wv, use = std::min(useful<KH>(a), useful<KH>(s));
    if (KH > 1) return voxels >= 0.4e6 && use >= 0.3;
    if (KW == 3 && (g.W == 64 || g.W == 128 || g.W == 256)) return use >= 0.7 && voxels >= (ratio && g.W > 64 ? 5.5e6 : 3e6);
    if (use < 0.45 || voxels < 0.7e6) return false;
    if (voxels >= 3e6) return true;
    if (g.D < 10 * (KD / 2)) return false;                // rows of an image
    if (g.Wv != g.W) return true;
    if (KW == 3) return ratio ? voxels >= (g.D >= 20 ? 1.2e6 : 1.6e6) : voxels >= 2e6 || use >= 0.65 || g.D >= 24;
    return !ratio || voxels >= 1.5e6 || g.D >= 46 || (voxels >= 0.85e6 && use >= 0.5);
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

bool covers(const Geo& g, bool ratio) {
    if (g.m != 1 || g.sc != SC || g.W % 4 || g.SP >= (1LL << 29)) return false;
    if (g.kD == 3 && g.kH == 3 && g.kW == 3) return worth<3, 3, 3>(g, ratio);
    if (g.kD != 1 || g.D != 1 || g.kH != g.kW) return false;
    if (g.kH == 5) return worth<5, 1, 5>(as_rows(g), ratio);
    if (g.kH == 3) return worth<3, 1, 3>(as_rows(g), ratio);
    return false;
}

cudaError_t forward(const Geo& g, const bf16* x, const bf16* z, const float* h, const float* bias, bf16* out, bf16* t1, cudaStream_t st) {
    if (g.kD == 3) return run<3, 3, 3>(g, x, z, h, bias, out, t1, st);
    if (g.kH == 5) return run<5, 1, 5>(as_rows(g), x, z, h, bias, out, t1, st);
    return run<3, 1, 3>(as_rows(g), x, z, h, bias, out, t1, st);
}

cudaError_t backward_ratio(const Geo& g, const bf16* x, const bf16* z, const bf16* t1, const float* h, const float* bias,
                           const bf16* gout, float* gnum, float* gden, bf16* direct, bool pairs, cudaStream_t st) {
    if (g.kD == 3) return run_ratio<3, 3, 3>(g, x, z, t1, h, bias, gout, gnum, gden, direct, pairs, st);
    if (g.kH == 5) return run_ratio<5, 1, 5>(as_rows(g), x, z, t1, h, bias, gout, gnum, gden, direct, pairs, st);
    return run_ratio<3, 1, 3>(as_rows(g), x, z, t1, h, bias, gout, gnum, gden, direct, pairs, st);
}

unsigned wait_expired() {
    int dev = -1;
    unsigned* all = g_expired.load(std::memory_order_acquire);
    if (!all || cudaDeviceSynchronize() != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    return __atomic_load_n(all + dev, __ATOMIC_ACQUIRE);
}

bool take_expired() {
    int dev = -1;
    unsigned* all = g_expired.load(std::memory_order_acquire);
    if (!all || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
    unsigned one = 1u;
    return __atomic_load_n(all + dev, __ATOMIC_ACQUIRE) == 1u &&
           __atomic_compare_exchange_n(all + dev, &one, 2u, false, __ATOMIC_ACQ_REL, __ATOMIC_ACQUIRE);
}

cudaError_t probe_wait(unsigned limit_us, cudaStream_t st) {
    unsigned* word = nullptr;
    const cudaError_t e = expired_word(word);
    if (e != cudaSuccess) return e;
    probe_wait_kernel<<<1, 32, 0, st>>>(limit_us * 1000u, word);
    launched();
    return cudaGetLastError();
}

}  // namespace tc
}  // namespace ndc
