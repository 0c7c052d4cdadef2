// bp_fp64.cu -- all-FP64 forward backprojection for sm_100a.
//
// Same tiling, shared-memory window staging (cp.async.bulk + mbarrier), pixel
// map and output layout as the mixed kernel in bp_mixed.cu, but every
// pixel-pulse is computed directly in double: |a_p - x_q| with a square root
// rounded as sqrt() rounds it (sqrt_rn), the bin index, the linear interpolation of FP64 range
// profiles and the rotation exp(+j 2 pi k dR) (k = 2 f0 / c, reduced mod one
// revolution), accumulated in double.  It is the accuracy path and the FP64
// baseline the mixed kernel is measured against; semantics as bp_mixed.cu.
//
// What bounds it is the FP64 pipe (64 lanes per SM and cycle; 66% busy) at 37
// FP64 instructions per pixel-pulse, with shared memory's data pipe at 64%.
// The common path has no branch and no library call, so a thread's eight
// pixels are independent chains the scheduler interleaves, on two CTAs per SM;
// the square root is a reciprocal-root estimate with one coupled Newton step
// and a residual correction, the rotation an entry of a table of 512 and two
// short polynomials; window entries are the range profile's samples themselves
// (the FFT output), the slope formed per pixel, so no pair rows are written
// (18-39 us a call) and a window is half the shared memory.  512^2 pixels x
// 1024 pulses: 2049 us with sqrt(), sincospi() and a gate branch per pixel at
// one CTA per SM, now 825 us.
#include <cstdint>

#include "bp_common.cuh"
#include "bp_tile.cuh"
#include "sarbp_internal.h"

namespace sarbp {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps64 = kThreads / 32;
constexpr int kTY = 64;
// four mbarriers (full, empty; two buffers each), two zero samples, and the
// table exp(+j 2 pi n / 512)
constexpr int kTurnTable = 512;
constexpr int kHdr64 = 64 + kTurnTable * 16;

__device__ __forceinline__ PulseGeo64 make_geo64(const BpLaunch &L, int p, double cx, double cy, double cz) {
    PulseGeo64 g;
    g.flags = 0;
    g.ax = L.ax[p];
    g.ay = L.ay[p];
    g.az = L.az[p];
    g.r0 = L.r0[p];
    g.k = 2.0 * L.f0[p] / kClight;
    const double vx = g.ax - cx, vy = g.ay - cy, vz = g.az - cz;
    const double rc = sqrt(vx * vx + vy * vy + vz * vz);
    const double D = rc - g.r0;
    const double bc = D * L.lambda + L.half_nfft;
    if (!(isfinite(bc) && isfinite(g.k) && fabs(bc) < 1.0e9)) {
        atomicOr(L.err, ERRBIT_NOT_FINITE);
        return g;
    }
    g.ws = static_cast<int>(floor(bc)) - L.W;
    if (!(g.ws + L.wsize - 2 <= 0 || g.ws + 1 >= L.nfft - 1)) g.flags = PG_ACTIVE;
    // the window meets an end of the range bins: test each pixel's bin
    if (g.ws < 0 || g.ws + L.wsize > L.nfft) g.flags |= PG_GATE;
    // a pixel may come close to the antenna (or the phase, of a range in the
    // thousands of kilometres, pass the reduction's range): library functions
    if (rc <= 0.125 * L.near_hd16 || !(fabs(g.k * D) < 1.0e12)) g.flags |= PG_NEAR;
    return g;
}

__device__ __forceinline__ double2 lds_d2(uint32_t addr) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr));
    return v;
}

// exp(+j 2 pi ph), |ph| < 2^42: ph = n/512 + r exactly, |r| <= 1/1024; sin
// and cos of 2 pi r as polynomials in r^2 (interpolated at the Chebyshev nodes
// of [0, 1/1024^2] in 60 digits; errors 2e-21 and 1e-17 before rounding), times
// the table's entry n mod 512.  13 FP64 instructions where quadrants
// (rotation, bp_common.cuh) take 17 and ten selects; 512^2 pixels x 1024
// pulses 915 us by quadrants, 853 with 64 entries and polynomials a degree
// longer (15 instructions), 862 with those 64 once per bank group, 825 with
// 512: the entries' bank conflicts hide behind the FP64 pipe.
__device__ __forceinline__ void rotation_table(double ph, uint32_t tab, double &cs, double &sn) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    const double t = fma(ph, static_cast<double>(kTurnTable), kMagic);
    const double2 w = lds_d2(tab + (static_cast<uint32_t>(__double2loint(t)) & (kTurnTable - 1)) * 16u);
    const double r = fma(t - kMagic, -1.0 / kTurnTable, ph);
    const double z = r * r;
    double S = fma(81.60513954752706, z, -41.34170224036052);
    double C = fma(64.93931252474451, z, -19.739208802169003);
    S = r * fma(S, z, 6.283185307179586);
    C = fma(C, z, 1.0);
    cs = fma(w.x, C, -(w.y * S));
    sn = fma(w.y, C, w.x * S);
}

// One pulse into the thread's MX x 2 pixels.  SAFE: pixels gated by the valid
// range bins, library square root and sine / cosine.
template <int MX, bool SAFE>
__device__ __forceinline__ void accumulate_pulse64(const BpLaunch &L, const PulseGeo64 &g, uint32_t w_addr,
                                                   uint32_t zero_addr, uint32_t turn_addr, const double (&xs)[MX],
                                                   const double (&ys)[2],
                                                   double z, double (&acc_re)[MX][2], double (&acc_im)[MX][2]) {
    constexpr double kMagic = 6755399441055744.0;
    const double gax = g.ax, gay = g.ay, gr0 = g.r0, gk = g.k, ez = g.az - z;
    // the squares are rounded before they are added, (x^2 + y^2) + z^2, as the
    // reference's CPU code does: a fused multiply-add rounds the range of one
    // sample in twenty the other way, 1e-10 of an image at 10 km
    const double ez2 = __dmul_rn(ez, ez);
    double ey2[2];
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const double ey = gay - ys[l];
        ey2[l] = __dmul_rn(ey, ey);
    }
    const uint32_t last = static_cast<uint32_t>(L.wsize - 2);
    // entry floor(B) - ws: low word of floor(B) + kMagic (its low 32 bits are
    // the integer itself)
    const uint32_t base = static_cast<uint32_t>(g.ws);
    int worst = 0;
#pragma unroll
    for (int k = 0; k < MX; ++k) {
        const double ex = gax - xs[k], ex2 = __dmul_rn(ex, ex);
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const double s = __dadd_rn(__dadd_rn(ex2, ey2[l]), ez2);
            const double dR = (SAFE ? sqrt(s) : sqrt_rn(s)) - gr0;
            const double B = dR * L.lambda + L.half_nfft;
            const double t = __dadd_rd(B, kMagic);
            const double a = B - (t - kMagic);
            const uint32_t idx = static_cast<uint32_t>(__double2loint(t)) - base;
            uint32_t addr = w_addr + idx * 16u;
            bool use = true;
            if (SAFE) use = B > 0.0 && B < static_cast<double>(L.nfft - 1);  // rmin < dR < rmax
            // an index outside the window cannot occur; it would read the zero
            // entry and be reported after the pulse (a branch here would end
            // the block the chains are interleaved in)
            const bool in = idx <= last;
            worst = max(worst, use && !in ? 1 : 0);
            use = use && in;
            addr = use ? addr : zero_addr;
            const double2 v = lds_d2(addr), vn = lds_d2(addr + 16u);
            const double re = fma(SAFE && !use ? 0.0 : a, vn.x - v.x, v.x);
            const double im = fma(SAFE && !use ? 0.0 : a, vn.y - v.y, v.y);
            const double ph = gk * dR;
            double sn, cs;
            if (SAFE)
                sincospi(2.0 * (ph - rint(ph)), &sn, &cs);
            else
                rotation_table(ph, turn_addr, cs, sn);
            acc_re[k][l] = fma(re, cs, fma(-im, sn, acc_re[k][l]));
            acc_im[k][l] = fma(re, sn, fma(im, cs, acc_im[k][l]));
        }
    }
    if (worst) atomicOr(L.err, ERRBIT_BOUNDS);
}

// Store (or add) a thread's pixel (k, l) of the tile at (tx0, ty0, z-slice iz).
template <int MX>
__device__ __forceinline__ void store_pixel64(const BpLaunch &L, int tx0, int ty0, int iz, int warp, int lane, int k,
                                              int l, double2 v) {
    using M = tile::PixelMap<MX>;
    double2 *img = static_cast<double2 *>(L.img);
    const int row = tx0 + M::row0(warp, lane) + M::kStep * k, col = ty0 + M::col0(warp, lane) + (kTY / 2) * l;
    if (row >= L.nx || col >= L.ny) return;
    const long long o = (static_cast<long long>(iz) * L.nx + row) * L.ny + col;
    if (L.accumulate) {
        const double2 old = img[o];
        v.x += old.x;
        v.y += old.y;
    }
    img[o] = v;
}

// Index of a thread's pixel (k, l) in a partial-sum slot of TX x 64
// complex128 values (written and read by the same threads).
__device__ __forceinline__ int slot_pixel(int k, int l) {
    return (2 * k + l) * kThreads + static_cast<int>(threadIdx.x);
}

// Units of (tile, stage) split over the CTAs as in bp_mixed.cu (tile::sk_lo).
// Two stage buffers: "full" (PB arrivals and the window bytes) and "empty"
// (one arrival per warp); warp 0 refills a buffer once every warp has
// consumed it, its lanes q < PB one pulse each.
template <int MX, int PB, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) bp_fp64_kernel(const __grid_constant__ BpLaunch L) {
    using M = tile::PixelMap<MX>;
    constexpr int TX = 8 * MX;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    double2 *zero = reinterpret_cast<double2 *>(smem + 32);
    PulseGeo64 *geo = reinterpret_cast<PulseGeo64 *>(smem + kHdr64);
    const uint32_t win_addr = smem_addr(smem + kHdr64 + 2 * PB * sizeof(PulseGeo64));
    const uint32_t pulse_bytes = static_cast<uint32_t>(L.wsize) * 16u, buf_bytes = PB * pulse_bytes;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const tile::TileGrid tg = tile::tile_grid(L, TX, PB);
    const long long G = gridDim.x;
    const long long lo = tile::sk_lo(blockIdx.x, tg.units, G);
    const int n = static_cast<int>(tile::sk_lo(blockIdx.x + 1, tg.units, G) - lo);
    if (n <= 0) return;
    const int S = tg.stages;

    double xs[MX], ys[2], z = 0.0, acc_re[MX][2], acc_im[MX][2];
#pragma unroll
    for (int k = 0; k < MX; ++k)
#pragma unroll
        for (int l = 0; l < 2; ++l) acc_re[k][l] = acc_im[k][l] = 0.0;

    const uint32_t bar_base = smem_addr(&bars[0]);  // full[s] at bar_base + 8 s, empty[s] at bar_base + 16 + 8 s
    const uint32_t zero_addr = smem_addr(zero), turn_addr = smem_addr(smem + 64);
    for (int e = threadIdx.x; e < kTurnTable; e += kThreads) {
        double2 *turn = reinterpret_cast<double2 *>(smem + 64) + e;
        sincospi(static_cast<double>(e) / (kTurnTable / 2), &turn->y, &turn->x);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(bar_base + 8u * s, PB);
            mbar_init(bar_base + 16u + 8u * s, kWarps64);
            zero[s] = make_double2(0.0, 0.0);
        }
        fence_mbar_init();
    }
    __syncthreads();

    // lane q < PB of warp 0: record and window copy of the unit's pulse q into buffer s
    auto produce = [&](const tile::UnitCursor &pc, int s) {
        if (lane >= PB) return;
        const double cx = L.left + static_cast<double>(pc.tx * TX + TX / 2) * L.dx;
        const double cy = L.bottom + static_cast<double>(pc.ty * kTY + kTY / 2) * L.dy;
        const double cz = L.zlow + static_cast<double>(pc.iz) * L.dz;
        const int p = pc.b * PB + lane;
        const uint32_t bar = bar_base + 8u * s;
        PulseGeo64 g;
        g.flags = 0;
        if (p < L.np) g = make_geo64(L, p, cx, cy, cz);
        geo[s * PB + lane] = g;
        if (g.flags & PG_ACTIVE) {
            const double2 *src = static_cast<const double2 *>(L.rc) + static_cast<long long>(p) * L.nfft + g.ws;
            mbar_arrive_expect_tx(bar, pulse_bytes);
            bulk_copy_g2s(win_addr + s * buf_bytes + lane * pulse_bytes, src, pulse_bytes, bar);
        } else {
            mbar_arrive(bar);
        }
    };

    tile::UnitCursor cc, pc;  // consumer at unit i; warp 0's producer at unit i + 1
    cc.init(tg, L, lo);
    pc = cc;
    if (warp == 0) produce(pc, 0);

    int seg = 0;
    int seg_first = cc.b;
    bool new_tile = true;
    for (int i = 0; i < n; ++i) {
        const int s = i & 1;
        bool ok = true;
        if (warp == 0 && i + 1 < n) {
            pc.advance(tg, L);
            if (i >= 1) ok = mbar_wait_bounded(bar_base + 16u + 8u * (s ^ 1), ((i - 1) >> 1) & 1, L.err);
            if (ok) produce(pc, s ^ 1);
            __syncwarp();
        }
        const int b = cc.b;
        if (new_tile) {
            const int tx0 = cc.tx * TX + M::row0(warp, lane), ty0 = cc.ty * kTY + M::col0(warp, lane);
#pragma unroll
            for (int k = 0; k < MX; ++k) xs[k] = L.left + static_cast<double>(tx0 + M::kStep * k) * L.dx;
#pragma unroll
            for (int l = 0; l < 2; ++l) ys[l] = L.bottom + static_cast<double>(ty0 + (kTY / 2) * l) * L.dy;
            z = L.zlow + static_cast<double>(cc.iz) * L.dz;
            new_tile = false;
        }
        ok = ok && mbar_wait_bounded(bar_base + 8u * s, (i >> 1) & 1, L.err);
        if (__any_sync(0xffffffffu, !ok)) {
            // a wait ran out (error bit set): the other warps end at their own;
            // warp 0's copies of the next stage land first (again bounded)
            if (warp == 0 && i + 1 < n) mbar_wait_bounded(bar_base + 8u * (s ^ 1), ((i + 1) >> 1) & 1, L.err);
            return;
        }
        const int nq = min(PB, L.np - b * PB);
#pragma unroll 1
        for (int q = 0; q < nq; ++q) {
            const PulseGeo64 &g = geo[s * PB + q];
            const uint32_t w = win_addr + s * buf_bytes + q * pulse_bytes;
            const int flags = g.flags;
            if (!(flags & PG_ACTIVE)) continue;
            if (flags & (PG_GATE | PG_NEAR))
                accumulate_pulse64<MX, true>(L, g, w, zero_addr, turn_addr, xs, ys, z, acc_re, acc_im);
            else
                accumulate_pulse64<MX, false>(L, g, w, zero_addr, turn_addr, xs, ys, z, acc_re, acc_im);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_base + 16u + 8u * s);
        if (i + 1 == n || b == S - 1) {
            if (seg_first == 0 && b == S - 1) {
#pragma unroll
                for (int k = 0; k < MX; ++k)
#pragma unroll
                    for (int l = 0; l < 2; ++l)
                        store_pixel64<MX>(L, cc.tx * TX, cc.ty * kTY, cc.iz, warp, lane, k, l,
                                          make_double2(acc_re[k][l], acc_im[k][l]));
            } else {
                double2 *slot = static_cast<double2 *>(L.sk_partial) +
                                (2 * static_cast<long long>(blockIdx.x) + (seg > 0 ? 1 : 0)) * (TX * kTY);
#pragma unroll
                for (int k = 0; k < MX; ++k)
#pragma unroll
                    for (int l = 0; l < 2; ++l) slot[slot_pixel(k, l)] = make_double2(acc_re[k][l], acc_im[k][l]);
            }
#pragma unroll
            for (int k = 0; k < MX; ++k)
#pragma unroll
                for (int l = 0; l < 2; ++l) acc_re[k][l] = acc_im[k][l] = 0.0;
            ++seg;
            seg_first = 0;
            new_tile = true;
        }
        cc.advance(tg, L);
    }
}

template <int MX>
__global__ void __launch_bounds__(kThreads) bp_sk_fixup64_kernel(const __grid_constant__ BpLaunch L, long long G, int PB) {
    constexpr int TX = 8 * MX;
    const tile::TileGrid tg = tile::tile_grid(L, TX, PB);
    const long long t = blockIdx.x;
    const long long c0 = tile::sk_owner(t * tg.stages, tg.units, G);
    const long long c1 = tile::sk_owner(t * tg.stages + tg.stages - 1, tg.units, G);
    if (c0 == c1) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.y;
    int tx0, ty0, iz;
    tile::tile_origin(tg, t, TX, tx0, ty0, iz);
    const long long s0 = tile::sk_first_slot(c0, t * tg.stages, tg.units, G);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const double2 v = tile::sk_sum(static_cast<const double2 *>(L.sk_partial), TX * kTY, slot_pixel(k, l), s0, c0,
                                       c1, [](double2 &s, const double2 &e) {
                                           s.x += e.x;
                                           s.y += e.y;
                                       });
        store_pixel64<MX>(L, tx0, ty0, iz, warp, lane, k, l, v);
    }
}

// two CTAs per SM (128 registers); one where the windows need its shared memory
constexpr size_t kTwoCtaSmem = 113u * 1024u;

template <int MX, int PB, int MINB>
cudaError_t launch64_on(const BpLaunch &L, size_t smem, cudaStream_t s) {
    constexpr int TX = 8 * MX;
    auto kern = bp_fp64_kernel<MX, PB, MINB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    const tile::TileGrid tg = tile::tile_grid(L, TX, PB);
    if (tg.units < 1) return cudaSuccess;
    long long G = tg.tiles;
    if (L.sk_partial && L.sk_resident > 0 && tg.tiles % L.sk_resident != 0) {
        const long long g = L.sk_resident < tg.units ? L.sk_resident : tg.units;
        if (2 * g * TX * kTY * static_cast<long long>(sizeof(double2)) <= L.sk_slot_bytes) G = g;
    }
    if (G > 0x7fffffffLL) return cudaErrorInvalidValue;
    kern<<<static_cast<unsigned>(G), kThreads, smem, s>>>(L);
    e = cudaGetLastError();
    if (e != cudaSuccess || G == tg.tiles) return e;
    bp_sk_fixup64_kernel<MX><<<dim3(static_cast<unsigned>(tg.tiles), MX), kThreads, 0, s>>>(L, G, PB);
    return cudaGetLastError();
}

template <int MX, int PB>
cudaError_t launch64(const BpLaunch &L, size_t smem, cudaStream_t s) {
    return smem > kTwoCtaSmem ? launch64_on<MX, PB, 1>(L, smem, s) : launch64_on<MX, PB, 2>(L, smem, s);
}

template <int MX, int PB>
int resident64(size_t smem) {
    auto kern = smem > kTwoCtaSmem ? bp_fp64_kernel<MX, PB, 1> : bp_fp64_kernel<MX, PB, 2>;
    int dev = 0, sms = 0, occ = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return occ * sms;
}

}  // namespace

size_t bp_fp64_smem_bytes(const TileConfig &tc, int wsize) {
    return kHdr64 + 2 * static_cast<size_t>(tc.pb) * sizeof(PulseGeo64) +
           2 * static_cast<size_t>(tc.pb) * static_cast<size_t>(wsize) * 16;
}

int bp_fp64_resident(const TileConfig &tc, size_t smem) {
#define SARBP_FP64_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_) return resident64<MX_, PB_>(smem);
    SARBP_FP64_CASE(4, 16)
    SARBP_FP64_CASE(4, 8)
    SARBP_FP64_CASE(4, 4)
    SARBP_FP64_CASE(4, 2)
    SARBP_FP64_CASE(4, 1)
    SARBP_FP64_CASE(2, 16)
    SARBP_FP64_CASE(2, 8)
    SARBP_FP64_CASE(2, 4)
    SARBP_FP64_CASE(2, 2)
    SARBP_FP64_CASE(2, 1)
    SARBP_FP64_CASE(1, 16)
    SARBP_FP64_CASE(1, 8)
    SARBP_FP64_CASE(1, 4)
    SARBP_FP64_CASE(1, 2)
    SARBP_FP64_CASE(1, 1)
#undef SARBP_FP64_CASE
    return 0;
}

cudaError_t launch_bp_fp64(const BpLaunch &L, const TileConfig &tc, size_t smem, cudaStream_t s) {
#define SARBP_FP64_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_) return launch64<MX_, PB_>(L, smem, s);
    SARBP_FP64_CASE(4, 16)
    SARBP_FP64_CASE(4, 8)
    SARBP_FP64_CASE(4, 4)
    SARBP_FP64_CASE(4, 2)
    SARBP_FP64_CASE(4, 1)
    SARBP_FP64_CASE(2, 16)
    SARBP_FP64_CASE(2, 8)
    SARBP_FP64_CASE(2, 4)
    SARBP_FP64_CASE(2, 2)
    SARBP_FP64_CASE(2, 1)
    SARBP_FP64_CASE(1, 16)
    SARBP_FP64_CASE(1, 8)
    SARBP_FP64_CASE(1, 4)
    SARBP_FP64_CASE(1, 2)
    SARBP_FP64_CASE(1, 1)
#undef SARBP_FP64_CASE
    return cudaErrorInvalidValue;
}

}  // namespace sarbp
