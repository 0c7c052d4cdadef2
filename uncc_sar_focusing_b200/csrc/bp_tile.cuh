// bp_tile.cuh -- the (tile, pulse) machinery shared by the mixed-precision
// forward and adjoint backprojection kernels: tile constants, the FP64
// geometry record of one pulse relative to one pixel tile, the per-warp
// producer that writes records and issues the window bulk copies, and the
// shared-memory load of one window entry.  See bp_mixed.cu for the design.
#pragma once

#include <cstdint>

#include "bp_common.cuh"
#include "sarbp_internal.h"

namespace sarbp {
namespace tile {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTY = 64;
constexpr float kRoundMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
constexpr uint32_t kRoundMagicBits = 0x4B400000u;
constexpr double kTwoPi = 6.283185307179586476925286766559;

// ---- work split over (tile, pulse-stage) units ---------------------------
//
// Tiles are numbered t = (zz * tiles_x + tx) * tiles_y + ty (zz = hypothesis
// * nz + z-slice) and unit u = t * stages + stage.  CTA c of G takes units
// [lo(c), lo(c+1)), lo(c) = floor(c U / G): with G = tiles every CTA gets
// exactly one tile; with G = the resident CTA count every SM gets the same
// number of pulse stages, whatever the tile count (no partial last wave).
struct TileGrid {
    int tiles_y, tiles_x;
    long long tiles;
    int stages;
    long long units;
};

__host__ __device__ __forceinline__ TileGrid tile_grid(const BpLaunch &L, int TX, int PB) {
    TileGrid g;
    g.tiles_y = (L.ny + kTY - 1) / kTY;
    g.tiles_x = (L.nx + TX - 1) / TX;
    g.tiles = static_cast<long long>(g.tiles_y) * g.tiles_x * L.nz * L.nhyp;
    g.stages = (L.np + PB - 1) / PB;
    g.units = g.tiles * g.stages;
    return g;
}

__host__ __device__ __forceinline__ long long sk_lo(long long c, long long units, long long G) {
    return c * units / G;
}

// The CTA whose range holds unit u: the largest c with lo(c) <= u.
__device__ __forceinline__ long long sk_owner(long long u, long long units, long long G) {
    long long c = u * G / units;
    while (c + 1 < G && sk_lo(c + 1, units, G) <= u) ++c;
    while (c > 0 && sk_lo(c, units, G) > u) --c;
    return c;
}

// Partial-sum slot of the first CTA c0 = sk_owner(first) of the tile whose
// first unit is `first`: a CTA's first segment (the one holding unit lo(c))
// uses slot 2c, a later one slot 2c + 1.  The tile's other CTAs c > c0 start
// inside it (lo(c) > first), so theirs is slot 2c.
__device__ __forceinline__ long long sk_first_slot(long long c0, long long first, long long units, long long G) {
    return sk_lo(c0, units, G) >= first ? 2 * c0 : 2 * c0 + 1;
}

// Sum of element `at` of a split tile's partial slots (`stride` elements
// each) in CTA order: slot s0, then those of CTAs c0 + 1 .. c1.  Four loads
// ahead of their additions: a tile of a small image is spread over 20 or more
// CTAs, and one load after the other took 34 us for 16 tiles x 18 slots.
template <typename V, typename ADD>
__device__ __forceinline__ V sk_sum(const V *part, long long stride, long long at, long long s0, long long c0,
                                    long long c1, ADD add) {
    V v = part[s0 * stride + at];
    long long c = c0 + 1;
    for (; c + 3 <= c1; c += 4) {
        V e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = part[2 * (c + i) * stride + at];
#pragma unroll
        for (int i = 0; i < 4; ++i) add(v, e[i]);
    }
    for (; c <= c1; ++c) add(v, part[2 * c * stride + at]);
    return v;
}

// Pixel origin (row tx0, column ty0) and hypothesis-major slice zz of tile t.
__device__ __forceinline__ void tile_origin(const TileGrid &g, long long t, int TX, int &tx0, int &ty0, int &zz) {
    const long long r = t / g.tiles_y;
    ty0 = static_cast<int>(t - r * g.tiles_y) * kTY;
    const long long q = r / g.tiles_x;
    tx0 = static_cast<int>(r - q * g.tiles_x) * TX;
    zz = static_cast<int>(q);
}

// Position of a unit, advanced one unit at a time without divisions: stage
// b of the tile at tile column ty, tile row tx, z-slice iz of hypothesis hyp.
struct UnitCursor {
    int b, ty, tx, iz, hyp;

    __device__ __forceinline__ void init(const TileGrid &g, const BpLaunch &L, long long u) {
        const long long t = u / g.stages;
        b = static_cast<int>(u - t * g.stages);
        const long long r = t / g.tiles_y;
        ty = static_cast<int>(t - r * g.tiles_y);
        const long long q = r / g.tiles_x;
        tx = static_cast<int>(r - q * g.tiles_x);
        hyp = static_cast<int>(q / L.nz);
        iz = static_cast<int>(q - static_cast<long long>(hyp) * L.nz);
    }
    __device__ __forceinline__ void advance(const TileGrid &g, const BpLaunch &L) {
        if (++b < g.stages) return;
        b = 0;
        if (++ty < g.tiles_y) return;
        ty = 0;
        if (++tx < g.tiles_x) return;
        tx = 0;
        if (++iz < L.nz) return;
        iz = 0;
        ++hyp;
    }
};

#ifndef SARBP_GEO_RSQ
#define SARBP_GEO_RSQ 1
#endif

// 1/sqrt(s) in double by Newton-Raphson for the reciprocal square root,
// y <- y (3 - s y^2) / 2, from the single-precision hardware estimate (about
// 2^-22 relative): each step squares the relative error, two reach double
// precision.  In place of a double sqrt and a double division on the
// producing lane, whose instruction sequences are several times longer.
__device__ __forceinline__ double rsqrt_newton(double s) {
    double y = static_cast<double>(rsqrtf(static_cast<float>(s)));
    const double hs = 0.5 * s;
    y = y * fma(-hs * y, y, 1.5);
    y = y * fma(-hs * y, y, 1.5);
    return y;
}

// tx_half: half the tile's rows (its columns are 64: 32 each side).  exchanged:
// the record's x (rows of the pixel map) is the image's y and the other way
// round.
__device__ __forceinline__ PulseGeo make_geo(const BpLaunch &L, int p, long long goff, double cx, double cy,
                                             double cz, int tx_half, bool exchanged = false) {
    PulseGeo g;
    g.flags = exchanged ? PG_EXCHANGED : 0;
    const double dx = exchanged ? L.dy : L.dx, dy = exchanged ? L.dx : L.dy;
    const long long gi = goff + p;  // geometry of hypothesis goff / np
    const double ax = L.ax[gi], ay = L.ay[gi], az = L.az[gi], r0 = L.r0[gi], f0 = L.f0[gi];
    const double vx = exchanged ? ay - cy : ax - cx, vy = exchanged ? ax - cx : ay - cy, vz = az - cz;
#if SARBP_GEO_RSQ
    const double s2 = vx * vx + vy * vy + vz * vz;
    const double inv = rsqrt_newton(s2);
    const double rc = s2 * inv;
    constexpr double kTwoOverC = 2.0 / kClight;
    const double k = f0 * kTwoOverC;
#else
    const double rc = sqrt(vx * vx + vy * vy + vz * vz);
    const double inv = 1.0 / rc;
    const double k = 2.0 * f0 / kClight;
#endif
    const double ux = vx * inv, uy = vy * inv;
    const double D = rc - r0;
    const double bc = D * L.lambda + L.half_nfft;
    const double kd = k * D;
    if (!(isfinite(bc) && isfinite(kd) && isfinite(ux) && isfinite(uy) && rc > 0.0 && fabs(bc) < 1.0e9 &&
          fabs(kd) < 1.0e12)) {
        atomicOr(L.err, ERRBIT_NOT_FINITE);
        return g;
    }
    const int ws = static_cast<int>(floor(bc)) - L.W;
    const double al = frac_rev(-k * ux * dx);
    const double be = frac_rev(-k * uy * dy);
    g.A = frac_rev(kd);
    g.alpha = al;
    g.beta = be;
    g.B0 = bc - static_cast<double>(ws);
    g.gam = -L.lambda * ux * dx;
    g.eta = -L.lambda * uy * dy;
    g.b32r = static_cast<float>(kTwoPi * frac_rev(32.0 * be));
    g.e32 = static_cast<float>(32.0 * g.eta);
    g.tx = static_cast<float>(ux * dx);
    g.ty = static_cast<float>(uy * dy);
    g.h = static_cast<float>(0.5 * inv);
    g.hr = static_cast<float>(0.5 * inv * inv);
    g.kr = static_cast<float>(kTwoPi * k);
    g.rc = static_cast<float>(rc);
    // validity bounds of the window-centred bin (bin - ws - W)
    g.lo = static_cast<float>(-ws - L.W);
    g.hi = static_cast<float>(L.nfft - 1 - ws - L.W);
    g.ws = ws;
    g.ux = static_cast<float>(ux);
    g.uy = static_cast<float>(uy);
    g.uz = static_cast<float>(vz * inv);
    g.rinv = static_cast<float>(inv);

    int flags = g.flags;
    // near field: the expansion would be off by 1e-7 turns, or (start frequencies
    // next to zero) 1e-4 bins.  (Bins of less than 1e-12 or more than 1e12 to the
    // metre, and 1 / Rc^2 next to the one pixel of a grid without extent, would
    // leave the polynomials' FP32 range; the exact path does without.)
    const double reach = fmax(fabs(k), 1.0e-3 * L.lambda);
    if (rc < fmax(L.near_hd16, 1.0e-9) || rc * rc * rc < reach * L.near_coef || !(L.lambda > 1.0e-12 && L.lambda < 1.0e12))
        flags |= PG_NEAR;
    // Tight window: a pixel (i, j) of the tile has bin - bc = i gam + j eta +
    // lambda g with 0 <= g <= hd^2 / (2 (Rc - hd)) (hd the tile
    // half-diagonal), |i| <= tx_half, |j| <= 32, so its floor(bin) and
    // floor(bin) + 1 lie within floor(bc) -/+ (ceil(span) + 1): wp =
    // ceil(span) + 3, at most W (the triangle-inequality bound |bin - bc| <=
    // lambda hd the full window is sized for).  Near-field pulses keep W.
    int wp = L.W;
    if (!(flags & PG_NEAR)) {
        const double hd = L.near_hd16 * (1.0 / 16.0);
        const double span = fabs(g.gam) * tx_half + fabs(g.eta) * 32.0 + L.lambda * hd * hd / (2.0 * (rc - hd));
        if (span < L.W) {
            const int w = static_cast<int>(ceil(span)) + 3;
            wp = w < L.W ? w : L.W;
        }
    }
    g.wp = wp;
    // the part of the window this pulse copies: bins [wsp, wsp + 2 wp + 2)
    const int wsp = ws + (L.W - wp), wsz = 2 * wp + 2;
    if (!(wsp + wsz - 2 <= 0 || wsp + 1 >= L.nfft - 1)) flags |= PG_ACTIVE;
    if (!(wsp >= 0 && wsp + wsz <= L.nfft)) flags |= PG_GATE;
    g.flags = flags;
    return g;
}

// ---- pixel map and polynomial tables of the mixed kernels ------------------
//
// A thread's pixels: warp w covers rows [2 MX (w >> 1), + 2 MX) and columns
// 16 (w & 1) + [0, 16) and the same 32 columns on; its lanes are 2 rows x 16
// columns, each aligned group of 8 lanes a 2 x 4 patch, and a thread steps
// MX times by two rows.  The 8 lanes of one shared-memory wavefront then look
// at bins a few entries apart whatever the look direction; as 8 columns of
// one row they spread over 7 column steps, and where the bin advances about 2
// entries a column (large workload, look direction along the columns) their
// 16-byte loads collide two to three ways.
template <int MX>
struct PixelMap {
    static constexpr int kStep = 2;                 // rows between a thread's pixels
    static constexpr int kMid = MX / 2;             // the row step the polynomials are centred on
    static constexpr int kGroupRows = kStep * MX;   // rows of a warp
    // row entry (0..7) of a thread, and the row offset of its middle pixel
    // from the tile centre
    static __host__ __device__ constexpr int entry(int warp, int lane) { return (warp >> 1) * 2 + ((lane >> 2) & 1); }
    static __host__ __device__ constexpr int mid_row(int e) {
        return (e >> 1) * kGroupRows + (e & 1) + kStep * kMid - 4 * MX;
    }
    // first row of the thread within the tile, and its first column (the second is 32 on)
    static __host__ __device__ constexpr int row0(int warp, int lane) {
        return (warp >> 1) * kGroupRows + ((lane >> 2) & 1);
    }
    static __host__ __device__ constexpr int col0(int warp, int lane) {
        return (warp & 1) * 16 + ((lane >> 3) << 2) + (lane & 3);
    }
};

// 64-row tiles can be taken with rows and columns exchanged (the map's rows run
// along the image's columns): a wavefront's 4-pixel side then lies along the
// image's rows.  The pre-pass does it, for all pulses of a tile, where the bins
// of the tile's first, middle and last pulse advance faster along the columns
// (|a - c| dx against dy per axis: the ranges are nearly one), so that the short
// side of the patch is the fast one and its 8 bins stay within 8 entries.
// 1024^2 x 2048 pulses, look direction along the columns: 1622 -> 1481 us
// (adjoint 2071 -> 1922), along the rows 1464 -> 1480 (1995 -> 1929).
__device__ __forceinline__ bool tile_exchanged(const BpLaunch &L, long long goff, double cx, double cy) {
    const int at[3] = {0, L.np >> 1, L.np - 1};
    double d = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        d += fabs(L.ay[goff + at[i]] - cy) * L.dy - fabs(L.ax[goff + at[i]] - cx) * L.dx;
    return d > 0.0;
}

// Whether tile t of a launch with pre-pass records is exchanged.
__device__ __forceinline__ bool record_exchanged(const BpLaunch &L, long long t) {
    return L.geo_tab && (static_cast<const PulseGeo *>(L.geo_tab)[t * L.np].flags & PG_EXCHANGED);
}

// Phase and bin of a tile's pixels as polynomials.  With the far-field
// remainder in bins Q(i, j) = lambda g = -lambda (t^2 - |d|^2)(h + t hr), a cubic
// in the pixel's row and column offsets i, j from the tile centre,
//     Q = i^2 (q20 + i q30) + j i (q11 + i q21) + j^2 (q02 + i q12 + j q03),
// the window-centred bin is B0 - W + i gam + j eta + Q and the phase
// 2 pi frac(A + i alpha + j beta) + tau Q, tau = kr / lambda.  (Not the phase
// and its lambda / kr: kr is zero at baseband, and a bin becomes an address.)
// Around a thread's middle row i = i_c + 2 k both are P0 + k a + k^2 b: the
// table holds the parts of P0, a, b that depend on i_c only (8 row entries of
// two float4) and the column phases (32 floats); a thread completes them with
// its two columns (13 paired operations a pulse), so phase and bin cost 22
// paired operations per 16 pixels instead of a full evaluation of t, t^2 -
// |d|^2 and the remainder for each (64).  The
// k^3 term of tau Q is carried by the lower ones (least squares): at most 10.5 of
// its 64 at the outer row is left, 2e-7 rad at 0.12 m and 8 km, 3e-7 at 0.5 m and
// 50 km, 6e-7 at 3.9 m and 800 km, the coarsest tiles of 64 rows that are far
// field there.
//   [2e]     phase, bin, x1 = i (q11 + i q21), x2 = q02 + i q12
//   [2e + 1] phase step, bin step, step's j term, k^2 term
//   [16..]   2 pi frac(j beta), j = -32..-1
// and, in the record's first two words (its FP64 steps, no longer needed):
//   [0]      2 pi frac(32 beta), eta, tau, q03
//   [1]      step's j^2 term, k^2 term's j term, lo, hi
// Near-field pulses keep the linear parts only (their remainder is evaluated
// per pixel).
constexpr int kPolyCols = 16, kPolyEntries = kPolyCols + 8;
constexpr int kRecWords = sizeof(PulseGeo) / sizeof(float4);

// The tables of NQ pulses by one warp, records in rec[0, NQ).  Lanes q < NQ
// first leave the cubic's coefficients of their pulse where its column phases
// will be, then the 8 NQ row entries and after them the 32 NQ column phases
// are spread over the 32 lanes.
template <int MX, int NQ>
__device__ __forceinline__ void write_poly_tables(float4 *tabs, PulseGeo *rec, int lane, const BpLaunch &L) {
    using M = PixelMap<MX>;
    float4 un0 = make_float4(0.f, 0.f, 0.f, 0.f), un1 = un0;
    if (lane < NQ) {
        float4 *w = reinterpret_cast<float4 *>(rec + lane);
        const float4 c0 = w[3], c1 = w[4], c2 = w[5];  // b32r, e32; tx, ty, h, hr; kr, rc, lo, hi
        const bool ex = rec[lane].flags & PG_EXCHANGED;
        const float dx = static_cast<float>(ex ? L.dy : L.dx), dy = static_cast<float>(ex ? L.dx : L.dy);
        const bool near = rec[lane].flags & PG_NEAR;
        const float lam = static_cast<float>(L.lambda);
        const float n20 = fmaf(c1.x, c1.x, -dx * dx), n11 = 2.0f * c1.x * c1.y, n02 = fmaf(c1.y, c1.y, -dy * dy);
        const float mh = near ? 0.0f : -lam * c1.z, mr = near ? 0.0f : -lam * c1.w;
        const float q21 = mr * fmaf(c1.x, n11, c1.y * n20), q12 = mr * fmaf(c1.x, n02, c1.y * n11);
        const float q03 = mr * c1.y * n02, tau = near ? 0.0f : c2.x / lam;
        float4 *coef = tabs + lane * kPolyEntries + kPolyCols;
        coef[0] = make_float4(mh * n20, mh * n11, mh * n02, mr * c1.x * n20);
        coef[1] = make_float4(q21, q12, tau, 0.0f);
        un0 = make_float4(c0.x, c0.y * (1.0f / 32.0f), tau, q03);
        un1 = make_float4(2.0f * q12, 4.0f * q21, c2.z, c2.w);
    }
    __syncwarp();
    // over the thread's rows, m = k + 1/2 = -(MX - 1)/2 .. (MX - 1)/2, m^3 ~ beta
    // m by least squares; so k^3 ~ kC0 + kC1 k - 3/2 k^2
    constexpr float kBeta = MX == 8 ? 9.25f : (MX == 4 ? 2.05f : 0.25f);
    constexpr float kC0 = 0.5f * kBeta - 0.125f, kC1 = kBeta - 0.75f;
    for (int t = lane; t < 8 * NQ; t += 32) {
        const int q = t >> 3, e = t & 7;
        const float4 *w = reinterpret_cast<const float4 *>(rec + q);
        const double2 d0 = *reinterpret_cast<const double2 *>(w);  // A, alpha
        const double B0 = rec[q].B0, gam = rec[q].gam;
        float4 *row = tabs + q * kPolyEntries + 2 * e;
        // q20, q11, q02, q30; q21, q12, tau
        const float4 qa = tabs[q * kPolyEntries + kPolyCols], qb = tabs[q * kPolyEntries + kPolyCols + 1];
        const float i = static_cast<float>(M::mid_row(e));
        const double id = static_cast<double>(i);
        const double pr = fma(id, d0.y, d0.x), ps = 2.0 * d0.y;
        const float nl = fmaf(8.0f * kC0, qa.w, i * i * fmaf(i, qa.w, qa.x));
        const float an = fmaf(8.0f * kC1, qa.w, 2.0f * i * fmaf(3.0f * i, qa.w, 2.0f * qa.x));
        row[0] = make_float4(fmaf(qb.z, nl, static_cast<float>(kTwoPi * (pr - rint(pr)))),
                             static_cast<float>(fma(id, gam, B0 - L.W)) + nl, i * fmaf(i, qb.x, qa.y),
                             fmaf(i, qb.y, qa.z));
        row[1] = make_float4(fmaf(qb.z, an, static_cast<float>(kTwoPi * (ps - rint(ps)))),
                             static_cast<float>(2.0 * gam) + an, 2.0f * fmaf(2.0f * i, qb.x, qa.y),
                             4.0f * fmaf(3.0f * (i - 1.0f), qa.w, qa.x));
    }
    __syncwarp();
    const double jd = static_cast<double>(lane - kTY / 2);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double pc = jd * rec[q].beta;
        reinterpret_cast<float *>(tabs + q * kPolyEntries + kPolyCols)[lane] =
            static_cast<float>(kTwoPi * (pc - rint(pc)));
    }
    __syncwarp();
    if (lane < NQ) {
        float4 *w = reinterpret_cast<float4 *>(rec + lane);
        w[0] = un0;
        w[1] = un1;
    }
}

// Lane 0: the window copy of pulse p (slot q) into the stage buffer, or a
// plain arrival when the tile's window misses the pulse's range bins.  The
// test hook L.drop_pulse expects that pulse's bytes without copying them.
__device__ __forceinline__ void issue_window(const BpLaunch &L, int p, int q, int flags, int wp, int ws,
                                             uint32_t win_s, uint32_t bar) {
    if (flags & PG_ACTIVE) {
        // the samples of the pulse's tight window (one more than its 2 wp + 2
        // entries), from the even sample at or before its first, to where
        // entry W - wp of the slot will be (rewrite_window)
        const long long first = static_cast<long long>(p) * L.nfft + ws + (L.W - wp);
        const int odd = static_cast<int>(first & 1);
        const uint32_t bytes = static_cast<uint32_t>((2 * wp + 3 + odd + 1) & ~1) * 8u;
        mbar_arrive_expect_tx(bar, bytes);
        if (p == L.drop_pulse) return;
        bulk_copy_g2s(win_s + (static_cast<uint32_t>(q) * static_cast<uint32_t>(L.wsize) + static_cast<uint32_t>(L.W - wp)) * 16u,
                      static_cast<const float2 *>(L.rc) + (first - odd), bytes, bar);
    } else {
        mbar_arrive(bar);
    }
}

// Producing warps of a stage of PB pulses: two, each with half the pulses (one
// warp alone, 1000 and more instructions a stage, held the accumulating ones
// up: forward 1583 against 1495 us, adjoint 2175 against 2050 us on 1024^2
// pixels x 2048 pulses).  With the 8 accumulating warps on two CTAs that is 5
// warps a scheduler, the most its registers hold at 96 a thread.
template <int PB>
struct Producers {
    static constexpr int kWarps = PB >= 2 ? 2 : 1;
    static constexpr int kPulses = PB / kWarps;  // pulses of each
};

// Pre-pass records (BpLaunch::geo_tab, [tile][pulse]) of pulses p0 .. p0 + NQ - 1
// of tile t in a producing warp's registers, 8 NQ words of 16 bytes over the
// lanes; loaded a stage before they are stored.
template <int NQ>
struct StageRecords {
    static constexpr int kPre = (kRecWords * NQ + 31) / 32;
    float4 w[kPre];

    __device__ __forceinline__ void load(const BpLaunch &L, long long t, int p0, int lane) {
        const float4 *src = reinterpret_cast<const float4 *>(static_cast<const PulseGeo *>(L.geo_tab) + t * L.np + p0);
        const int words = min(NQ, L.np - p0) * kRecWords;
#pragma unroll
        for (int r = 0; r < kPre; ++r) {
            const int k = lane + 32 * r;
            w[r] = k < words ? src[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ void store(PulseGeo *rec, int lane) const {
#pragma unroll
        for (int r = 0; r < kPre; ++r) {
            const int k = lane + 32 * r;
            if (k < kRecWords * NQ) reinterpret_cast<float4 *>(rec)[k] = w[r];
        }
    }
};

// A producing warp's part of one stage, NQ pulses from p0 of the tile at row
// tx, column ty (in tiles), slice iz: records (from the pre-pass, or computed
// by lanes q < NQ), window copies (lane q the one of pulse q) and tables.
template <int MX, int NQ>
__device__ __forceinline__ void produce_pulses(const BpLaunch &L, int p0, int tx, int ty, int iz, int hyp,
                                               const StageRecords<NQ> &pre, bool pregeo, PulseGeo *rec, float4 *tabs,
                                               uint32_t win, uint32_t bar, int lane) {
    const int p = p0 + lane;  // lane < NQ: this lane's pulse
    if (pregeo) {
        pre.store(rec, lane);
    } else if (lane < NQ) {
        const double cx = L.left + static_cast<double>(tx * 8 * MX + 4 * MX) * L.dx;
        const double cy = L.bottom + static_cast<double>(ty * kTY + kTY / 2) * L.dy;
        const double cz = L.zlow + static_cast<double>(iz) * L.dz;
        PulseGeo g = {};
        if (p < L.np) g = make_geo(L, p, static_cast<long long>(hyp) * L.np, cx, cy, cz, 4 * MX);
        rec[lane] = g;
    }
    __syncwarp();
    if (lane < NQ) issue_window(L, p, lane, rec[lane].flags, rec[lane].wp, rec[lane].ws, win, bar);
    write_poly_tables<MX, NQ>(tabs, rec, lane, L);
}

__device__ __forceinline__ float4 lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr));
    return v;
}

__device__ __forceinline__ float2 lds64(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void sts128(uint32_t addr, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

__device__ __forceinline__ float2 splat(float a) { return make_float2(a, a); }

// Phase and bin polynomials of a thread's pixel pairs for one pulse (columns
// col and col + 32 of the tile): row step k - kMid takes P0 + k Pa + k^2 Pb
// and B0 + k Ba + k^2 Bb.  SPLIT: Pb beside Bb instead of from it, for the
// adjoint, whose registers it suits (1950 against 1964 us on 1024^2 pixels x
// 2048 pulses; forward 1508 against 1484).
template <bool SPLIT>
struct PixelPoly {
    float2 J, P0, Pa, Pb, B0, Ba, Bb;
    float lo, hi;  // valid bins

    __device__ __forceinline__ PixelPoly(const PulseGeo &g, const float4 *tab, int entry, int col) {
        const float4 r0 = tab[2 * entry], r1 = tab[2 * entry + 1];
        const float4 u0 = reinterpret_cast<const float4 *>(&g)[0], u1 = reinterpret_cast<const float4 *>(&g)[1];
        const float j0 = static_cast<float>(col - kTY / 2);
        J = make_float2(j0, j0 + static_cast<float>(kTY / 2));
        const float s0 = r0.x + reinterpret_cast<const float *>(tab + kPolyCols)[col];
        const float2 w = __ffma2_rn(J, __ffma2_rn(J, splat(u0.w), splat(r0.w)), splat(r0.z));
        const float2 tJ = __fmul2_rn(J, splat(u0.z));
        P0 = __ffma2_rn(tJ, w, make_float2(s0, s0 + u0.x));
        B0 = __ffma2_rn(J, w, __ffma2_rn(J, splat(u0.y), splat(r0.y)));
        const float2 v = __ffma2_rn(J, splat(u1.x), splat(r1.z));
        Pa = __ffma2_rn(tJ, v, splat(r1.x));
        Ba = __ffma2_rn(J, v, splat(r1.y));
        Bb = __ffma2_rn(J, splat(u1.y), splat(r1.w));
        Pb = SPLIT ? __ffma2_rn(tJ, splat(u1.y), splat(r1.w * u0.z)) : __fmul2_rn(Bb, splat(u0.z));
        lo = u1.z;
        hi = u1.w;
    }

    // f(k, phase, bin) for the thread's MX pixel pairs, the middle row last
    // (first: adjoint 2085 instead of 2064 us, forward the same); rows +-k
    // share P0 + k^2 Pb.  (Without the k^2 terms, which near-field pulses do
    // not need, the batch kernel spills more: 1242 -> 1329 us on ten scenes.)
    template <int MX, typename F>
    __device__ __forceinline__ void rows(F f) const {
        using M = PixelMap<MX>;
#pragma unroll
        for (int k = M::kMid; k >= 1; --k) {
            const float x = static_cast<float>(k);
            const float2 Ps = __ffma2_rn(splat(x * x), Pb, P0), Bs = __ffma2_rn(splat(x * x), Bb, B0);
            f(M::kMid - k, __ffma2_rn(splat(-x), Pa, Ps), __ffma2_rn(splat(-x), Ba, Bs));
            if (M::kMid + k < MX) f(M::kMid + k, __ffma2_rn(splat(x), Pa, Ps), __ffma2_rn(splat(x), Ba, Bs));
        }
        f(M::kMid, P0, B0);
    }
};

// Near-field pulses: the exact remainder g = e / (s + sqrt(s^2 + e)), s = Rc - t,
// e = |d|^2 - t^2, of the pixel pair in row offset fi, columns J (and s, for
// R_q = s + g).  From the hardware's estimates of root and reciprocal r = 1 /
// (s + sqrt), g0 = e r is off by some 2^-22; one Newton step on g (2 s + g) = e,
// with 1 / (2 s + 2 g0) ~ r (1 - g0 r), leaves its own rounding: no further off
// than sqrtf() and a division, whose special cases end the block in which the
// pixels' chains are interleaved.  512^2 pixels x 1024 pulses at 0.15 m, 8 km:
// forward 674 -> 449 us, adjoint 921 -> 740.
__device__ __forceinline__ float2 near_remainder(const PulseGeo &g, const BpLaunch &L, float fi, float2 J,
                                                 float2 &s) {
    const float4 c1 = *reinterpret_cast<const float4 *>(&g.tx);  // tx, ty, h, hr
    const bool ex = g.flags & PG_EXCHANGED;
    const float di = fi * static_cast<float>(ex ? L.dy : L.dx);
    const float2 dj = __fmul2_rn(J, splat(static_cast<float>(ex ? L.dx : L.dy)));
    const float2 nt = __ffma2_rn(splat(-fi), splat(c1.x), __fmul2_rn(J, splat(-c1.y)));  // -t
    const float2 d2 = __ffma2_rn(splat(di), splat(di), __fmul2_rn(dj, dj));
    const float2 ne = __ffma2_rn(nt, nt, make_float2(-d2.x, -d2.y)), e = make_float2(-ne.x, -ne.y);
    s = __fadd2_rn(splat(g.rc), nt);
    const float2 R2 = __ffma2_rn(s, s, e);
    const float2 D = __fadd2_rn(s, make_float2(sqrt_estimate(R2.x), sqrt_estimate(R2.y)));
    const float2 r = make_float2(rcp_estimate(D.x), rcp_estimate(D.y));
    const float2 g0 = __fmul2_rn(e, r);
    const float2 f = __ffma2_rn(g0, __ffma2_rn(splat(2.0f), s, g0), ne);
    const float2 m = __fmul2_rn(g0, r);
    const float2 v = __ffma2_rn(make_float2(-m.x, -m.y), r, r);
    return __ffma2_rn(make_float2(-f.x, -f.y), v, g0);
}

// Intercept form of the windows.  A window arrives as samples v_n; entry n of
// its slot becomes {v_n - (n - W) v'_n, v'_n}, v'_n = v_(n+1) - v_n, so that a
// pixel whose window-centred bin is B = bin - ws - W (floor(B) + W = n)
// interpolates
//     v(B) = v_n + (B + W - n) v'_n = c_n + B v'_n
// with one fused multiply-add and no fraction.
// ZFORM (the adjoint, which needs only Z(B) = v'(B) + j nu v(B), nu = kr /
// lambda radians per bin): the entry becomes {Zc, Zv} with Zc = v'_n + j nu
// c_n and Zv = j nu v'_n, so that Z(B) = Zc + B Zv is again one fused
// multiply-add per component and the pixel loop neither interpolates v nor
// forms Z.
//
// In place, from the last entry to the first: the samples (8 bytes) start
// where the entries (16 bytes) do, so the entries of a group of lanes lie past
// every sample a lower group still reads; within a group all lanes read before
// any writes.  Samples instead of pair entries {v_n, v'_n} in HBM halve what
// range compression writes and the windows copy and need no pass after the
// FFT (point-target call 106 -> 94 us); the rewrite's second load and
// difference cost the 1024^2 x 2048 forward kernel 1.9% (1495 -> 1524 us).
// w: the window's first entry (W - wp); odd: its first sample is the second
// of those copied (issue_window).  kGroup: entries of a lane per round, more for
// wide windows, where the accumulating warps wait for this, fewer where the
// registers it takes cost them spills.  Forward, stages of 8 pulses (1024^2 x
// 2048): 2 1485, 3 1497, 4 1462 us; 4 pulses (windows of 474): 2 145, 4 149; 2
// (1278): 2 165, 4 151; 1 (4978): 4 823, 8 692.  Adjoint, 8: 2 1930, 4 1943; 2:
// 2 193, 4 189; 1, two CTAs an SM (2660): 3 267, 4 282, 6 255, 8 278; one CTA
// (4978): 4 1066, 8 879.
template <bool ZFORM, int kGroup>
__device__ __forceinline__ void rewrite_window(uint32_t w, int wp, uint32_t odd, int lane, float nu) {
    const int count = 2 * wp + 2;
    int n = (count - 1) / (32 * kGroup) * (32 * kGroup) + lane;  // the lane's first entry of the round
    uint32_t src = w + (static_cast<uint32_t>(n) + odd) * 8u, dst = w + static_cast<uint32_t>(n) * 16u;
    float m = static_cast<float>(n - wp);
    auto round = [&](int entries) {  // entries: those of the lane, at n, n + 32, ...
        float2 v[kGroup], vn[kGroup];
#pragma unroll
        for (int i = 0; i < kGroup; ++i)
            if (i < entries) {
                v[i] = lds64(src + 256u * i);
                vn[i] = lds64(src + 256u * i + 8u);
            }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kGroup; ++i)
            if (i < entries) {
                const float2 d = __fadd2_rn(vn[i], make_float2(-v[i].x, -v[i].y));
                const float2 c = __ffma2_rn(splat(-m - 32.0f * i), d, v[i]);
                if (ZFORM) {
                    const float2 z = __fmul2_rn(splat(nu), d);
                    sts128(dst + 512u * i, fmaf(-nu, c.y, d.x), fmaf(nu, c.x, d.y), -z.y, z.x);
                } else {
                    sts128(dst + 512u * i, c.x, c.y, d.x, d.y);
                }
            }
        __syncwarp();
    };
    round((count - n + 31) >> 5);
    for (n -= 32 * kGroup; n >= 0; n -= 32 * kGroup) {
        src -= 256u * kGroup;
        dst -= 512u * kGroup;
        m -= 32.0f * kGroup;
        round(kGroup);
    }
}

// The windows of NQ pulses, by their producing warp once the copies have landed;
// the fence orders these generic-proxy stores before the next bulk copies
// (async proxy) into the buffer, which the same warp issues.
template <int NQ, bool ZFORM, int GROUP>
__device__ __forceinline__ void rewrite_pulses(const BpLaunch &L, int p0, const PulseGeo *rec, uint32_t win_s, int lane,
                                               float inv_lam = 0.0f) {
    for (int q = 0; q < NQ; ++q) {
        if (!(rec[q].flags & PG_ACTIVE)) continue;
        const int off = L.W - rec[q].wp;
        const uint32_t odd = (static_cast<uint32_t>(p0 + q) * static_cast<uint32_t>(L.nfft) +
                              static_cast<uint32_t>(rec[q].ws + off)) & 1u;
        rewrite_window<ZFORM, GROUP>(win_s + (static_cast<uint32_t>(q) * static_cast<uint32_t>(L.wsize) + static_cast<uint32_t>(off)) * 16u,
                              rec[q].wp, odd, lane, ZFORM ? rec[q].kr * inv_lam : 0.0f);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
}

}  // namespace tile
}  // namespace sarbp
