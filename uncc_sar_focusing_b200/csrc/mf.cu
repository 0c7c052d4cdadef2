// mf.cu -- matched-filter focusing (sarbp_matched_filter).
//
// The reference's second focusing algorithm: computeDifferentialRangeAndPhase
// CorrectionsMF / run_mf (src/cpuBackProjection/cpuBackProjection.hpp:165-228)
// and matlab/mfBasic.m:73-89:
//     img[q] = sum_p sum_k w_k ph_p[k] exp(+j 4 pi (f0_p + k dF) dR_pq / c).
// With a_p = exp(+j 4 pi f0_p dR / c) and z_p = exp(+j 4 pi dF dR / c) the
// inner sum is a_p * P_p(z_p), P_p the polynomial with coefficients w_k ph_p[k],
// evaluated by Horner's rule: K complex multiply-adds per pixel-pulse instead
// of K complex exponentials.  Both phases are reduced modulo one revolution
// in FP64; Horner and accumulation run in FP32 (MIXED) or FP64.
//
// What bounds it is the FMA pipe: four multiply-adds per sample and
// pixel-pulse.  A warp takes one pulse and 32 P pixels, P = 4 per thread (2 in
// FP64): each broadcast read of a sample feeds 4 P multiply-adds in P
// independent chains (one pixel per thread waited out every step of its
// chain), as paired FP32 instructions from samples stored twice.  The 16 warps (8
// in FP64) of a CTA take different pulses of the same pixels, the CTAs of a cluster
// too, so a small image still fills the SMs; their sums are added in warp and
// rank order through (distributed) shared memory.  96^2 pixels x 128 pulses x
// 256 samples: 461 us with one pixel a thread, 64 us now, 35 us at the measured FMA rate
// (256^2 pixels: 387 us, 256 at that rate).  Two CTAs of 16 warps an SM (64
// registers, 44 bytes spilled outside the sample loop): with 8 warps a CTA and
// 80 registers the clusters of a small image did not all fit at once, 82 us
// (256^2: 476).  FP64 keeps 8: 378 us for 128^2 x 256, 443 with 16, and no
// bound on its registers (it takes 64; 415 us when told to).  Few pulses take
// CTAs of fewer warps (launch_mf_on).
#include <cooperative_groups.h>
#include <cstdint>

#include "bp_common.cuh"
#include "sarbp_internal.h"

namespace sarbp {
namespace {

constexpr int kMfChunk = 128;  // samples a warp stages at a time

// Horner chains of a thread's pixels: FP32 in pairs, FP64 singly.
struct MfFloat {
    static constexpr int kPixels = 4, kWarps = 16;  // pixels a thread, warps a CTA
    using Sample = float4;  // re, re, im, im
    float2 hr[2], hi[2], zr[2], zi[2];

    static __device__ __forceinline__ Sample sample(double re, double im, float2 v) {
        const float wr = static_cast<float>(re * v.x - im * v.y), wi = static_cast<float>(re * v.y + im * v.x);
        return make_float4(wr, wr, wi, wi);
    }
    __device__ __forceinline__ void start(int j, double zre, double zim) {
        float *r = &zr[j >> 1].x, *i = &zi[j >> 1].x;
        r[j & 1] = static_cast<float>(zre);
        i[j & 1] = static_cast<float>(zim);
        hr[j >> 1] = hi[j >> 1] = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void step(const Sample &s) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 nr = __ffma2_rn(hr[h], zr[h], __ffma2_rn(make_float2(-hi[h].x, -hi[h].y), zi[h], make_float2(s.x, s.y)));
            const float2 ni = __ffma2_rn(hr[h], zi[h], __ffma2_rn(hi[h], zr[h], make_float2(s.z, s.w)));
            hr[h] = nr;
            hi[h] = ni;
        }
    }
    __device__ __forceinline__ void add(int j, double ca, double sa, float &re, float &im) const {
        const float r = j & 1 ? hr[j >> 1].y : hr[j >> 1].x, i = j & 1 ? hi[j >> 1].y : hi[j >> 1].x;
        const float c = static_cast<float>(ca), s = static_cast<float>(sa);
        re += r * c - i * s;
        im += r * s + i * c;
    }
};

struct MfDouble {
    static constexpr int kPixels = 2, kWarps = 8;
    using Sample = double2;
    double hr[2], hi[2], zr[2], zi[2];

    static __device__ __forceinline__ Sample sample(double re, double im, float2 v) {
        return make_double2(re * v.x - im * v.y, re * v.y + im * v.x);
    }
    __device__ __forceinline__ void start(int j, double zre, double zim) {
        zr[j] = zre;
        zi[j] = zim;
        hr[j] = hi[j] = 0.0;
    }
    __device__ __forceinline__ void step(const Sample &s) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double nr = fma(hr[h], zr[h], fma(-hi[h], zi[h], s.x));
            const double ni = fma(hr[h], zi[h], fma(hi[h], zr[h], s.y));
            hr[h] = nr;
            hi[h] = ni;
        }
    }
    __device__ __forceinline__ void add(int j, double ca, double sa, double &re, double &im) const {
        re += hr[j] * ca - hi[j] * sa;
        im += hr[j] * sa + hi[j] * ca;
    }
};

// exp(+j 2 pi ph) for any finite ph
__device__ __forceinline__ void turn(double ph, double &cs, double &sn) {
    if (fabs(ph) < 1.0e12)
        rotation(ph, cs, sn);
    else
        sincospi(2.0 * (ph - rint(ph)), &sn, &cs);
}

// Pixel block blockIdx.x / (cluster size); the cluster's rank and the warp
// choose the pulses.  T: float or double; kMfWarps: warps of the CTA.
template <typename CH, typename T, int kMfWarps>
__device__ __forceinline__ void mf_body(const float2 *__restrict__ ph, const double *__restrict__ win, const MfLaunch &M) {
    constexpr int P = CH::kPixels;
    namespace cg = cooperative_groups;
    using Sample = typename CH::Sample;
    __shared__ __align__(16) union Smem {
        Sample s[kMfWarps][kMfChunk];
        T sum[kMfWarps][P][2][32];
        __device__ Smem() {}
    } sm;
    const cg::cluster_group cluster = cg::this_cluster();
    const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const long long npix = static_cast<long long>(M.nx) * M.ny * M.nz;
    const long long q0 = static_cast<long long>(blockIdx.x / ranks) * (32 * P) + lane;

    double x[P], y[P], z[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        long long q = q0 + 32 * j;
        if (q >= npix) q = npix - 1;  // computed, not stored
        const long long r = q / M.ny;
        x[j] = M.left + static_cast<int>(r % M.nx) * M.dx;
        y[j] = M.bottom + static_cast<int>(q - r * M.ny) * M.dy;
        z[j] = M.zlow + static_cast<int>(r / M.nx) * M.dz;
    }
    T re[P], im[P];
#pragma unroll
    for (int j = 0; j < P; ++j) re[j] = im[j] = 0;
    Sample *buf = sm.s[warp];
    const double kd = 2.0 * M.df / kClight;

    for (int p = rank * kMfWarps + warp; p < M.np; p += ranks * kMfWarps) {
        const double ax = M.ax[p], ay = M.ay[p], az = M.az[p], r0 = M.r0[p], kf = 2.0 * M.f0[p] / kClight;
        CH h;
        double ph0[P];  // revolutions of the first sample
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const double ex = ax - x[j], ey = ay - y[j], ez = az - z[j];
            const double dR = sqrt(ex * ex + ey * ey + ez * ez) - r0;
            ph0[j] = kf * dR;
            double sz, cz;
            turn(kd * dR, cz, sz);
            h.start(j, cz, sz);
        }
        // P(z) = sum_k c_k z^k by Horner from the highest power, in chunks
        for (int c1 = M.K; c1 > 0; c1 -= kMfChunk) {
            const int n = c1 < kMfChunk ? c1 : kMfChunk, c0 = c1 - n;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kMfChunk / 32; ++i) {
                const int k = lane + 32 * i;
                if (k < n) {
                    const float2 v = ph[static_cast<long long>(p) * M.K + c0 + k];
                    buf[k] = CH::sample(win ? win[2 * (c0 + k)] : 1.0, win ? win[2 * (c0 + k) + 1] : 0.0, v);
                }
            }
            __syncwarp();
            int k = n - 1;
            for (; k >= 7; k -= 8) {
#pragma unroll
                for (int i = 0; i < 8; ++i) h.step(buf[k - i]);
            }
            for (; k >= 0; --k) h.step(buf[k]);
        }
#pragma unroll
        for (int j = 0; j < P; ++j) {
            double sa, ca;
            turn(ph0[j], ca, sa);
            h.add(j, ca, sa, re[j], im[j]);
        }
    }

    // the warps' sums, then the ranks', in order
    __syncthreads();
#pragma unroll
    for (int j = 0; j < P; ++j) {
        sm.sum[warp][j][0][lane] = re[j];
        sm.sum[warp][j][1][lane] = im[j];
    }
    __syncthreads();
    // component i & 1 of pixel i >> 1 of the CTA's sum: warp i mod kMfWarps
#pragma unroll
    for (int i = warp; i < 2 * P; i += kMfWarps) {
        const int j = i >> 1, c = i & 1;
        T t = 0;
        for (int w = 0; w < kMfWarps; ++w) t += sm.sum[w][j][c][lane];
        sm.sum[0][j][c][lane] = t;  // read by this thread only before now
    }
    if (ranks > 1) cluster.sync();
    if (rank == 0) {
#pragma unroll
        for (int i = warp; i < 2 * P; i += kMfWarps) {
            const int j = i >> 1, c = i & 1;
            T t = sm.sum[0][j][c][lane];
            for (int r = 1; r < ranks; ++r) t += *cluster.map_shared_rank(&sm.sum[0][j][c][lane], r);
            const long long q = q0 + 32 * j;
            if (q < npix) static_cast<T *>(M.img)[2 * q + c] = t;
        }
    }
    if (ranks > 1) cluster.sync();  // the other ranks' shared memory stays until it has been read
}

// W warps a CTA: CH::kWarps, 4 or 1.  The small CTAs take 128 registers: one
// pulse x 256 samples on 16^2 pixels 8.7 us, with 64 (44 bytes spilled, the
// sample loads not ahead) 12.2; 512^2 pixels x 12 pulses 61 against 57.
template <int W>
__global__ void __launch_bounds__(32 * W, W == MfFloat::kWarps ? 2 : MfFloat::kWarps / W)
    mf_kernel(const float2 *__restrict__ ph, const double *__restrict__ win, MfLaunch M) {
    mf_body<MfFloat, float, W>(ph, win, M);
}

template <int W>
__global__ void __launch_bounds__(32 * W)
    mf_kernel64(const float2 *__restrict__ ph, const double *__restrict__ win, MfLaunch M) {
    mf_body<MfDouble, double, W>(ph, win, M);
}

// Warps of a CTA for np pulses.  All CTAs there are running at once: the fewest
// rounds of pulses.  More than fit: fewer slots (rounds x warps) by a fifth,
// since a warp without a pulse holds its place until the others are done (512^2
// pixels x 64 samples: one pulse 49 us on CTAs of 16 warps, 9 on CTAs of one; 3
// pulses 50 / 20; 12 73, 61 on CTAs of 4; 30 140, 165 on CTAs of one; FP64 12
// pulses 123 on 8, 85 on 4).
int mf_warps(int full, int np, long long blocks, int sms) {
    if (np >= 2 * full) return full;
    if (blocks < 2LL * sms) return np == 1 ? 1 : (np <= 4 ? 4 : full);
    int best = full;
    for (const int w : {4, 1})
        if (5 * ((np + w - 1) / w * w) < 4 * ((np + best - 1) / best * best)) best = w;
    return best;
}

template <typename CH, typename F>
cudaError_t launch_mf_on(F full, F four, F one, const float2 *ph, const double *win, const MfLaunch &M, cudaStream_t s) {
    const long long npix = static_cast<long long>(M.nx) * M.ny * M.nz;
    const long long blocks = (npix + 32 * CH::kPixels - 1) / (32 * CH::kPixels);
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // CTAs that share the pulses of a pixel block: the number (up to the 8 a
    // portable cluster holds) for which the busiest SM has the fewest pulses,
    // but more of them only for a tenth less: large clusters find room on fewer
    // SMs at a time (mixed, 96^2 pixels x 128 pulses, 72 blocks: 120 / 66 / 91 /
    // 82 us with 1 / 2 / 4 / 8; 64^2 x 512 455 / 233 / 121 / 118; 256^2 x 128
    // 437 / 388 / 421 / 470; 160^2 x 100 335 / 265 / 306 / 329).  FP64's CTAs of
    // 8 warps fit more easily: the most of equals (96^2 x 128: 120 us)
    int ranks = 1;
    long long best = 0;
    for (int r = 1; r <= 8; r *= 2) {
        const long long cost = ((blocks * r + sms - 1) / sms) * ((M.np + r * CH::kWarps - 1) / (r * CH::kWarps));
        if (r == 1 || (CH::kWarps == 8 ? cost <= best : 10 * cost < 9 * best)) {
            best = cost;
            ranks = r;
        }
    }
    const int warps = mf_warps(CH::kWarps, M.np, blocks, sms);
    if (warps < CH::kWarps) ranks = 1;
    if (blocks < 1 || blocks * ranks > 0x7fffffffLL) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks * ranks));
    cfg.blockDim = dim3(32 * warps);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(ranks);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ranks > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, warps == CH::kWarps ? full : (warps == 4 ? four : one), ph, win, M);
}

}  // namespace

cudaError_t launch_mf(const void *ph, const double *win, const MfLaunch &M, bool fp64, cudaStream_t s) {
    const float2 *x = static_cast<const float2 *>(ph);
    return fp64 ? launch_mf_on<MfDouble>(mf_kernel64<MfDouble::kWarps>, mf_kernel64<4>, mf_kernel64<1>, x, win, M, s)
                : launch_mf_on<MfFloat>(mf_kernel<MfFloat::kWarps>, mf_kernel<4>, mf_kernel<1>, x, win, M, s);
}

}  // namespace sarbp
