// Host build of csrc/bp_tile.cuh's per-(tile, pulse) arithmetic: the records
// (make_geo), the polynomial tables (write_poly_tables, 32 threads standing in
// for the warp's lanes) and a thread's phases and bins (PixelPoly,
// near_remainder), from the kernels' own source.  Compiled as plain C++; the
// paired FP32 instructions are spelled out below.
#include <algorithm>
#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

using std::isfinite;
using std::max;
using std::min;

static thread_local std::barrier<> *g_warp = nullptr;
static inline void __syncwarp(unsigned = 0xffffffffu) {
    if (g_warp) g_warp->arrive_and_wait();
}
static inline float2 __ffma2_rn(float2 a, float2 b, float2 c) {
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
}
static inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
static inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
// the device's estimates: values off by 2^-22, up or down, stand in for them
static inline float off(double v) {
    static thread_local unsigned n = 0;
    return static_cast<float>(v * (1.0 + (++n & 1 ? 0x1p-22 : -0x1p-22)));
}
static inline float rsqrtf(float x) { return off(1.0 / std::sqrt(static_cast<double>(x))); }
#define SARBP_HOST_ESTIMATES
static inline float sqrt_estimate(float x) { return off(std::sqrt(static_cast<double>(x))); }
static inline float rcp_estimate(float x) { return off(1.0 / static_cast<double>(x)); }
// off by up to 2^-20, the low word zero
static inline double rsqrt_estimate(double x) {
    static thread_local uint64_t n = 1;
    n = n * 6364136223846793005ull + 1442695040888963407ull;
    const double e = (static_cast<double>(n >> 11) * 0x1p-53 * 2.0 - 1.0) * (0x1p-20 - 0x1p-21);
    double y = 1.0 / std::sqrt(x) * (1.0 + e);
    uint64_t b;
    std::memcpy(&b, &y, 8);
    b &= ~0xffffffffull;
    std::memcpy(&y, &b, 8);
    return y;
}
static inline int __shfl_sync(unsigned, int v, int) { return v; }
static inline unsigned atomicOr(unsigned *p, unsigned v) {
    const unsigned o = *p;
    *p |= v;
    return o;
}
static inline size_t __cvta_generic_to_shared(const void *p) { return reinterpret_cast<size_t>(p); }
static inline int __double2hiint(double x) {
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return static_cast<int>(b >> 32);
}
static inline int __double2loint(double x) {
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return static_cast<int>(b);
}
static inline double __hiloint2double(int h, int l) {
    const uint64_t b = (static_cast<uint64_t>(static_cast<uint32_t>(h)) << 32) | static_cast<uint32_t>(l);
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}
struct Tid {
    unsigned x;
};
static thread_local Tid threadIdx = {0};

#include "../../uncc_sar_focusing_b200/csrc/bp_tile.cuh"

using namespace sarbp;

namespace {

// phase, bin [np][8 MX][64] (window-centred bin) of tile (0, 0), one slice;
// SPLIT: the adjoint's polynomials
template <int MX, bool SPLIT>
void run(const BpLaunch &L, bool exchanged, float *phase, float *bin, int *words) {
    using M = tile::PixelMap<MX>;
    constexpr int NQ = 4;
    const double cx = L.left + 4 * MX * L.dx, cy = L.bottom + tile::kTY / 2 * L.dy;
    for (int p0 = 0; p0 < L.np; p0 += NQ) {
        PulseGeo rec[NQ] = {};
        std::vector<float4> tabs(NQ * tile::kPolyEntries, make_float4(0.f, 0.f, 0.f, 0.f));
        const int n = std::min(NQ, L.np - p0);
        for (int q = 0; q < n; ++q) rec[q] = tile::make_geo(L, p0 + q, 0, cx, cy, L.zlow, 4 * MX, exchanged);
        std::barrier<> warp(32);
        std::vector<std::thread> lanes;
        for (int lane = 0; lane < 32; ++lane)
            lanes.emplace_back([&, lane] {
                g_warp = &warp;
                tile::write_poly_tables<MX, NQ>(tabs.data(), rec, lane, L);
            });
        for (std::thread &t : lanes) t.join();
        for (int q = 0; q < n; ++q) {
            const PulseGeo &g = rec[q];
            int *w = words + 3 * (p0 + q);
            w[0] = g.flags;
            w[1] = g.ws;
            w[2] = g.wp;
            float *P_out = phase + static_cast<size_t>(p0 + q) * 8 * MX * 64, *B_out = bin + static_cast<size_t>(p0 + q) * 8 * MX * 64;
            for (int t = 0; t < tile::kThreads; ++t) {
                const int wi = t >> 5, lane = t & 31, entry = M::entry(wi, lane), col = M::col0(wi, lane);
                const tile::PixelPoly<SPLIT> poly(g, tabs.data() + q * tile::kPolyEntries, entry, col);
                poly.template rows<MX>([&](int k, float2 P, float2 B) {
                    if (g.flags & PG_NEAR) {
                        float2 s;
                        const float2 r = tile::near_remainder(
                            g, L, static_cast<float>(M::mid_row(entry) + M::kStep * (k - M::kMid)), poly.J, s);
                        P = __ffma2_rn(tile::splat(g.kr), r, P);
                        B = __ffma2_rn(tile::splat(static_cast<float>(L.lambda)), r, B);
                    }
                    const int at = (M::row0(wi, lane) + M::kStep * k) * 64 + col;
                    P_out[at] = P.x;
                    P_out[at + 32] = P.y;
                    B_out[at] = B.x;
                    B_out[at + 32] = B.y;
                });
            }
        }
    }
}

}  // namespace

// geo: [5][np] antenna x, y, z, slant range, start frequency; the tile's first
// pixel is (left, bottom, 0).  words: [np][3] flags, ws, wp.
extern "C" int tile_probe(const double *geo, int np, int nfft, double lambda, double dx, double dy, double left,
                          double bottom, int W, double near_hd16, double near_coef, int mx, int exchanged, int split,
                          float *phase, float *bin, int *words) {
    unsigned err = 0;
    BpLaunch L{};
    L.ax = geo;
    L.ay = geo + np;
    L.az = geo + 2 * np;
    L.r0 = geo + 3 * np;
    L.f0 = geo + 4 * np;
    L.np = np;
    L.nfft = nfft;
    L.lambda = lambda;
    L.half_nfft = 0.5 * nfft;
    L.nx = 8 * mx;
    L.ny = 64;
    L.nz = 1;
    L.left = left;
    L.bottom = bottom;
    L.dx = dx;
    L.dy = dy;
    L.W = W;
    L.wsize = 2 * W + 2;
    L.near_hd16 = near_hd16;
    L.near_coef = near_coef;
    L.err = &err;
    switch (mx) {
        case 8: (split ? run<8, true> : run<8, false>)(L, exchanged != 0, phase, bin, words); break;
        case 4: (split ? run<4, true> : run<4, false>)(L, exchanged != 0, phase, bin, words); break;
        case 2: (split ? run<2, true> : run<2, false>)(L, exchanged != 0, phase, bin, words); break;
        default: (split ? run<1, true> : run<1, false>)(L, exchanged != 0, phase, bin, words); break;
    }
    return static_cast<int>(err);
}

extern "C" void sqrt_probe(const double *x, double *out, int n) {
    for (int i = 0; i < n; ++i) out[i] = sqrt_rn(x[i]);
}

extern "C" void rotation_probe(const double *x, double *cs, double *sn, int n) {
    for (int i = 0; i < n; ++i) rotation(x[i], cs[i], sn[i]);
}
