// bp_common.cuh -- shared device helpers of the sm_100a backprojection kernels.
//
// * mbarrier + cp.async.bulk (the non-tensor TMA copy, no multicast) used to
//   stage each pulse's range-bin window of a pixel tile into shared memory;
// * bounded waits: every wait gives up after a fixed wall time, sets an error
//   bit and lets the kernel return instead of hanging;
// * the per-(tile, pulse) geometry record computed in FP64 once per tile and
//   pulse and read by every thread of the tile.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sarbp {

// Device error bits (plan->d_err)
enum : unsigned {
    ERRBIT_NOT_FINITE = 1u,
    ERRBIT_TIMEOUT = 2u,
    ERRBIT_BOUNDS = 4u,
};

// speed of light, include/uncc_sar_focusing.hpp:34
constexpr double kClight = 299792458.0;

// Wall-clock limit of a bounded wait (ns).
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The warp's index as a value the compiler knows to be the same in all lanes
// (threadIdx.x >> 5 it does not): loops and addresses under a test of it stay
// on the uniform datapath.  Forward 1535 -> 1466 us, adjoint 2061 -> 1996 us on
// 1024^2 pixels x 2048 pulses.
__device__ __forceinline__ int warp_index() {
    return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
}

__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// True when phase `parity` has completed; false when it has not within about
// the suspend hint (ns): a waiting warp sleeps in the instruction that long
// instead of polling.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    constexpr uint32_t kSuspendNs = 50000;
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return ok != 0;
}

// Wait for phase `parity` of the barrier; false (and an error bit) after the
// wall-clock limit.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, unsigned *err) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_timer_ns();
    for (unsigned it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0u && global_timer_ns() - t0 > kWaitLimitNs) {
            atomicOr(err, ERRBIT_TIMEOUT);
            return false;
        }
    }
}

// Plain (non-multicast) bulk copy global -> this CTA's shared memory,
// completing transaction bytes on `bar`.  dst, src and bytes are multiples
// of 16 (FP64 windows are 16-byte samples; mixed ones 8-byte samples, an even
// number from an even one on, of rows that start on 16 bytes).
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

__device__ __forceinline__ double frac_rev(double x) { return x - rint(x); }

// The hardware's estimates of sqrt(x), 1/x (relative error about 2^-23; 0,
// infinities and NaN as the exact functions) and, in double, 1/sqrt(x) (2^-20 or
// better), one instruction each.  A host build of the kernels' arithmetic brings
// its own.
#ifndef SARBP_HOST_ESTIMATES
__device__ __forceinline__ float sqrt_estimate(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_estimate(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ double rsqrt_estimate(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
#endif

// Square root of a positive, normal s, rounded as sqrt() rounds it but for
// about one argument in 2^25, where it is the neighbour: with g ~ sqrt(s) and h
// ~ 1 / (2 sqrt(s)) from the reciprocal-root estimate (2^-20 or better), r = 1/2
// - g h corrects both to 2^-39, and the residual s - g^2 by fused multiply-add
// corrects g once more, to 2^-78 before the last rounding (Markstein's scheme,
// whose proof wants a better estimate).
__device__ __forceinline__ double sqrt_rn(double s) {
    const double y = rsqrt_estimate(s);
    double g = s * y;
    double h = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));  // y / 2
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    return fma(fma(-g, g, s), h, g);
}

// exp(+j 2 pi ph), |ph| <= 2^49: ph = n/4 + r exactly, |r| <= 1/8; sin and cos
// of 2 pi r as polynomials in r^2 (interpolated at the Chebyshev nodes of [0,
// 1/64] in 60 digits; errors 2e-17 and 5e-17 before rounding), then the
// quadrant n mod 4 by swap and sign.
__device__ __forceinline__ void rotation(double ph, double &cs, double &sn) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    const double t = fma(ph, 4.0, kMagic);
    const int q = __double2loint(t);
    const double r = fma(t - kMagic, -0.25, ph);
    const double z = r * r;
    double S = 3.7808689593022957, C = 7.810290968144191;
    S = fma(S, z, -15.093804209987114);
    C = fma(C, z, -26.42425703488269);
    S = fma(S, z, 42.058685020160894);
    C = fma(C, z, 60.24462008593029);
    S = fma(S, z, -76.70585970427454);
    C = fma(C, z, -85.45681709034115);
    S = fma(S, z, 81.60524927594804);
    C = fma(C, z, 64.93939402236538);
    S = fma(S, z, -41.341702240399634);
    C = fma(C, z, -19.73920880217842);
    S = r * fma(S, z, 6.283185307179586);
    C = fma(C, z, 1.0);
    const bool odd = q & 1;
    const double c = odd ? S : C, s = odd ? C : S;
    cs = __hiloint2double(__double2hiint(c) ^ (((q + 1) << 30) & 0x80000000), __double2loint(c));
    sn = __hiloint2double(__double2hiint(s) ^ ((q << 30) & 0x80000000), __double2loint(s));
}

// Flags of a PulseGeo record
enum : int {
    PG_ACTIVE = 1,  // the tile's window meets the valid range bins
    PG_GATE = 2,    // some pixels may fall outside (0, nfft-1): test each
    PG_NEAR = 4,    // tile too large for the far-field expansion: exact path
    PG_EXCHANGED = 8,  // x and y of the record are the image's columns and rows (tile_exchanged)
};

// Geometry of one pulse relative to one pixel tile (mixed-precision kernel).
//
// With the tile centre c on the pixel grid, pixel offset d = (i*dx, j*dy, 0)
// (integers i, j), u = (a - c)/|a - c|, Rc = |a - c|, t = u.d and
// e = |d|^2 - t^2, the differential range is exactly
//     dR = (Rc - R0) - t + g,   g = e / ((Rc - t) + sqrt((Rc - t)^2 + e))
// and g = e (h + t hr) (1 + O((|d|/Rc)^2)) with h = 1/(2Rc), hr = 1/(2Rc^2).
// Phase 2 pi k dR (k = 2 f0 / c), range bin lambda dR + nfft/2
// (lambda = nfft / max_wr).  The per-tile and per-step phase terms are
// reduced modulo one revolution in FP64, so what is left for FP32 is small.
// Field groups are 16-byte aligned so a thread reads them with vector loads.
struct __align__(16) PulseGeo {
    double A, alpha;   // frac(k (Rc - R0)); frac(-k ux dx): revolutions per x step
    double beta, B0;   // frac(-k uy dy); tile-centre bin relative to the window start
    double gam, eta;   // -lambda ux dx, -lambda uy dy: bins per x / y step
    float b32r, e32;         // 2 pi frac(32 beta) (rad), 32 eta (bins)
    float pad2, pad3;
    float tx, ty, h, hr;     // ux dx, uy dy (m); 1/(2 Rc), 1/(2 Rc^2)
    float kr, rc, lo, hi;    // 2 pi k (rad/m); Rc; valid iff lo < B_rel < hi
    int ws;                  // start bin of the tile's full window (W bins each side; may be negative)
    int flags;               // PG_*
    int wp;                  // this pulse's half-width (<= W): the bins it can reach from the tile
    int pad1;
    float ux, uy, uz, rinv;  // unit vector tile centre -> antenna, 1/Rc (adjoint kernel)
};
static_assert(sizeof(PulseGeo) == 128, "PulseGeo layout");

// Geometry of one pulse for the FP64 kernel (per-pixel exact computation).
struct __align__(16) PulseGeo64 {
    double ax, ay, az;  // antenna position
    double r0;          // slant range to scene centre
    double k;           // 2 f0 / c
    int ws;             // window start bin
    int flags;          // PG_ACTIVE
};
static_assert(sizeof(PulseGeo64) % 16 == 0, "PulseGeo64 must keep 16-byte alignment");

}  // namespace sarbp
