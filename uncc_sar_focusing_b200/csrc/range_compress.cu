// range_compress.cu -- range compression kernels.
//
// The reference forms range profiles with a batched in-place cuFFT inverse
// transform of the raw phase history (no zero pad, no window), then two more
// kernels: cufftNormalize_1DBatch_kernel (x /= N) and cufftShift_1DBatch_kernel
// (swap halves) (src/gpuBackProjection/cuda_sar_focusing/cuda_sar_focusing.hpp:
// 616-620, cuda_BackProjectionKernels.cuh:95-135).  Here:
//  1. rc_prep_kernel writes the FFT input in one pass: sample k < K becomes
//     ph[k] * fac[k] with fac[k] = w_k / Nfft * exp(+j 2 pi ((k s) mod Nfft) / Nfft),
//     s = (Nfft+1)/2, and k >= K is the zero pad (matlab/bpBasic.m:82).
//     The twiddle is the fftshift (cshift by s, cpuBackProjection_fft.hpp:81-84)
//     moved to the input side: ifft(x .* e^{j 2 pi k s/N})[n] = ifft(x)[n + s].
//     The 1/Nfft scale and the taper ride along, so no normalise or shift pass.
//  2. cuFFT batched C2C (Z2Z for FP64) inverse, in place.
// The backprojection kernels copy their windows straight from these rows.
#include <cmath>
#include <complex>
#include <vector>

#include "sarbp_internal.h"

namespace sarbp {
namespace {

template <typename C>
__global__ void rc_prep_kernel(const float2 *__restrict__ ph, const C *__restrict__ fac, C *__restrict__ out, int K,
                               int nfft, long long total) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long p = i / nfft;
        const int k = static_cast<int>(i - p * nfft);
        C v;
        v.x = 0;
        v.y = 0;
        if (k < K) {
            const float2 x = ph[p * K + k];
            const C f = fac[k];
            v.x = x.x * f.x - x.y * f.y;
            v.y = x.x * f.y + x.y * f.x;
        }
        out[i] = v;
    }
}

// Batch form: scene blockIdx.y of the table, grid-stride over its elements.
__global__ void rc_prep_batch_kernel(const BatchScene *__restrict__ scenes) {
    const BatchScene &S = scenes[blockIdx.y];
    if (S.fused) return;  // range-compressed by its own fused launch
    const float2 *__restrict__ ph = static_cast<const float2 *>(S.ph);
    const float2 *__restrict__ fac = static_cast<const float2 *>(S.fac);
    float2 *__restrict__ out = static_cast<float2 *>(const_cast<void *>(S.L.rc));
    const int K = S.K, nfft = S.L.nfft;
    const long long total = static_cast<long long>(S.L.np) * nfft;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long p = i / nfft;
        const int k = static_cast<int>(i - p * nfft);
        float2 v = make_float2(0.0f, 0.0f);
        if (k < K) {
            const float2 x = ph[p * K + k];
            const float2 f = fac[k];
            v.x = x.x * f.x - x.y * f.y;
            v.y = x.x * f.y + x.y * f.x;
        }
        out[i] = v;
    }
}

// ---- fused range compression: nfft = R K, K = 32 K2 ------------------------
//
// With y[k] = fac[k] ph[k] (taper x 1/N x shift twiddle) and N = R K the
// zero-padded inverse DFT splits into R inverse DFTs of length K:
//     rc[R m + r] = sum_k (y[k] W_N^{k r}) W_K^{k m},   W_L = exp(+j 2 pi / L).
// One CTA per pulse (grid-stride), one warp per sub-transform r.  Each
// length-K transform is done in four steps with K = 32 K2, k = k1 + 32 k2,
// m = m2 + K2 m1:  lane k1 transforms its K2 samples in registers (over k2),
// multiplies by W_K^{k1 m2}, the warp transposes through shared memory, and
// lane m2 transforms the 32 values over k1 in registers.  The R results are
// read back interleaved to write the profile's samples straight to HBM: 8
// bytes read per input sample, 8 written per output sample.  Twiddles come from one table built
// in double on the host and staged into shared memory.
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

template <int L>
__host__ __device__ constexpr int log2_of() {
    int n = 0;
    for (int v = L; v > 1; v >>= 1) ++n;
    return n;
}

template <int L>
__device__ __forceinline__ constexpr int bit_reverse(int x) {
    int r = 0;
    for (int b = 1; b < L; b <<= 1) {
        r = (r << 1) | (x & 1);
        x >>= 1;
    }
    return r;
}

// exp(+j 2 pi e / 32) for e in [0, 16) as FP32 constants (correctly rounded);
// after unrolling every e is a compile-time constant
__device__ __forceinline__ float2 w32(int e) {
    constexpr float c1 = 0.980785251f, s1 = 0.195090324f, c2 = 0.923879504f, s2 = 0.382683426f;
    constexpr float c3 = 0.831469595f, s3 = 0.555570245f, h = 0.707106769f;
    switch (e) {
        case 1: return make_float2(c1, s1);
        case 2: return make_float2(c2, s2);
        case 3: return make_float2(c3, s3);
        case 4: return make_float2(h, h);
        case 5: return make_float2(s3, c3);
        case 6: return make_float2(s2, c2);
        case 7: return make_float2(s1, c1);
        case 9: return make_float2(-s1, c1);
        case 10: return make_float2(-s2, c2);
        case 11: return make_float2(-s3, c3);
        case 12: return make_float2(-h, h);
        case 13: return make_float2(-c3, s3);
        case 14: return make_float2(-c2, s2);
        case 15: return make_float2(-c1, s1);
        default: return make_float2(1.0f, 0.0f);
    }
}

// In-register inverse DFT of L points (L divides 32): radix-2 decimation in
// frequency, natural-order input, bit-reversed output.  The twiddles W_L^e =
// W_32^(e 32 / L) are constants, 1 and +j without a multiply (68.5 vs 72.2 us
// with the twiddles loaded from a shared-memory table; same results).
template <int L>
__device__ __forceinline__ void ifft_dif(float2 (&v)[L]) {
    constexpr int LOG = log2_of<L>();
#pragma unroll
    for (int st = 0; st < LOG; ++st) {
        const int half = (L >> 1) >> st;
#pragma unroll
        for (int i = 0; i < L; i += 2 * half) {
#pragma unroll
            for (int j = 0; j < half; ++j) {
                const float2 a = v[i + j], b = v[i + j + half];
                v[i + j] = make_float2(a.x + b.x, a.y + b.y);
                const float2 d = make_float2(a.x - b.x, a.y - b.y);
                const int e = j * (L / (2 * half));
                constexpr int kScale = 32 / L;
                const int e32 = e * kScale;
                v[i + j + half] = e32 == 0 ? d : (e32 == 8 ? make_float2(-d.y, d.x) : cmulf(d, w32(e32)));
            }
        }
    }
}

// Layout of the twiddle table (complex64 entries) for K = 32 K2, N = R K.
template <int K2, int R>
struct RcTable {
    static constexpr int K = 32 * K2, N = K * R, NW = N / 32;
    static constexpr int kTwk = 0;                 // W_K^{k1 m2} at m2 * 32 + k1
    static constexpr int kWn = kTwk + K;           // W_N^i, i < 32 R
    static constexpr int kWnr = kWn + 32 * R;      // W_{N/32}^i, i < N / 32
    static constexpr int kSize = kWnr + NW;
    // shared row of one sub-transform.  The row writes read element (r, m) =
    // (b mod R, b / R) for every second b: the 16 lanes of one 128-byte
    // wavefront of 8-byte reads cover the even (or odd) values of r and 32/R
    // of m, first bank 2 (r kReg + m) mod 32; kReg = 16/R mod 16 makes these
    // 16 distinct even banks for R >= 2
    static constexpr int kReg = K + 32 + 16 / R;
    static constexpr size_t kSmem = (static_cast<size_t>(K) + kSize + static_cast<size_t>(R) * kReg) * 8;
};

template <int K2, int R>
__device__ __forceinline__ void rc_fused_body(const float2 *__restrict__ ph, const float2 *__restrict__ fac,
                                              const float2 *__restrict__ tab, float2 *__restrict__ rc, int np) {
    using T = RcTable<K2, R>;
    constexpr int K = T::K, N = T::N, REG = T::kReg, LOGR = log2_of<R>();
    extern __shared__ __align__(16) float2 rc_sm[];
    float2 *y = rc_sm, *tb = y + K, *regions = tb + T::kSize;
    const int tid = threadIdx.x, r = tid >> 5, lane = tid & 31;
    for (int i = tid; i < T::kSize; i += 32 * R) tb[i] = tab[i];
    float2 *reg = regions + r * REG;
    // a pulse's input samples, loaded one pulse ahead: issued before the
    // current pulse's row writes (the long phase), consumed after the barrier
    constexpr int KPT = (K + 32 * R - 1) / (32 * R);
    float2 pre[KPT];
    auto prefetch = [&](int q) {
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const int k = tid + j * 32 * R;
            pre[j] = (q < np && k < K) ? ph[static_cast<long long>(q) * K + k] : make_float2(0.0f, 0.0f);
        }
    };
    prefetch(blockIdx.x);
    for (int p = blockIdx.x; p < np; p += gridDim.x) {
        // the factors before the barrier, all loads in flight: one after the
        // other behind the stores to y (which may alias them for all the
        // compiler knows) they cost K = 1024, R = 1 32 loads' latency, 32.8
        // against 13.1 us for 48 pulses and 45.1 against 22.5 for 2048
        float2 f[KPT];
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const int k = tid + j * 32 * R;
            f[j] = k < K ? fac[k] : make_float2(0.0f, 0.0f);
        }
        __syncthreads();  // the previous pulse's reads of the regions are done; the table is staged
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const int k = tid + j * 32 * R;
            if (k < K) y[k] = cmulf(pre[j], f[j]);
        }
        __syncthreads();
        // z[k1 + 32 k2] = y[.] W_N^{k1 r} W_{N/32}^{k2 r}, transformed over k2
        const float2 a = tb[T::kWn + lane * r];
        float2 v[K2];
#pragma unroll
        for (int k2 = 0; k2 < K2; ++k2)
            v[k2] = cmulf(y[lane + 32 * k2], cmulf(a, tb[T::kWnr + ((k2 * r) & (T::NW - 1))]));
        ifft_dif<K2>(v);
        // times W_K^{k1 m2}, transposed: element (k1, m2) at m2 * 33 + k1
#pragma unroll
        for (int m2 = 0; m2 < K2; ++m2) reg[m2 * 33 + lane] = cmulf(v[bit_reverse<K2>(m2)], tb[T::kTwk + m2 * 32 + lane]);
        // the R K2 transforms over k1 fill the first warps' lanes, K2 of one
        // sub-transform side by side (as K2 lanes of each warp they cost every
        // warp their instructions: K = 512, 2048 pulses, 34 against 28 us)
        if (K2 < 32)
            __syncthreads();
        else
            __syncwarp();
        if (tid < R * K2) {
            float2 *rg = regions + (tid / K2) * REG;
            const int m2 = tid % K2;
            constexpr unsigned group = R * K2 < 32 ? (1u << (R * K2 % 32)) - 1u : 0xffffffffu;
            float2 w[32];
#pragma unroll
            for (int k1 = 0; k1 < 32; ++k1) w[k1] = rg[m2 * 33 + k1];
            __syncwarp(group);
            ifft_dif<32>(w);
#pragma unroll
            for (int m1 = 0; m1 < 32; ++m1) rg[m2 + K2 * m1] = w[bit_reverse<32>(m1)];
        }
        __syncthreads();
        prefetch(p + gridDim.x);
        // rc[R m + r] = regions[r][m], two samples a thread (N is even)
        float4 *row = reinterpret_cast<float4 *>(rc + static_cast<long long>(p) * N);
        for (int b = 2 * tid; b < N; b += 64 * R) {
            const float2 u = regions[(b & (R - 1)) * REG + (b >> LOGR)];
            const float2 un = regions[((b + 1) & (R - 1)) * REG + ((b + 1) >> LOGR)];
            row[b >> 1] = make_float4(u.x, u.y, un.x, un.y);
        }
    }
}

// One aperture, or (scenes non-null) scenes idx[blockIdx.y] of a batch, whose
// slots of the device table hold every pointer and size (a captured graph
// replays with new buffers).  blockIdx.x: the aperture's CTAs.
struct RcArgs {
    const BatchScene *scenes;
    const float2 *ph, *fac, *tab;
    float2 *rc;
    int K, np;
    unsigned short idx[kRcGroup];
};

// The CTA's aperture.  RcArgs itself stays untouched in the parameter space:
// written to or indexed as a by-value parameter it was copied to local memory
// by every thread, 176 bytes.
struct RcJob {
    const float2 *ph, *fac;
    float2 *rc;
    int K, np;

    __device__ __forceinline__ explicit RcJob(const RcArgs &a) : ph(a.ph), fac(a.fac), rc(a.rc), K(a.K), np(a.np) {
        if (!a.scenes) return;
        const BatchScene &S = a.scenes[a.idx[blockIdx.y]];
        ph = static_cast<const float2 *>(S.ph);
        fac = static_cast<const float2 *>(S.fac);
        rc = static_cast<float2 *>(const_cast<void *>(S.L.rc));
        K = S.K;
        np = S.L.np;
    }
};

template <int K2, int R>
__global__ void __launch_bounds__(32 * R) rc_fused_kernel(const __grid_constant__ RcArgs a) {
    const RcJob j(a);
    rc_fused_body<K2, R>(j.ph, j.fac, a.tab, j.rc, j.np);
}

// ---- the same for other K <= 512: each sub-transform as a chirp convolution ----
//
// The length-K inverse DFT of sub-transform r, with c[k] = W_2K^(k^2) and
// k m = (k^2 + m^2 - (m - k)^2) / 2 (Bluestein):
//     rc[R m + r] = c[m] sum_k (y[k] W_N^{k r} c[k]) conj(c[m - k]),
// a circular convolution of length M = 32 K2 >= 2 K - 1: forward transform,
// product with the chirp's transform H (1/M included), inverse transform.  One
// warp per sub-transform; both transforms are the direct kernel's four steps,
// the first split over k = k1 + 32 k2 (K2 points in the registers of 32 lanes,
// then 32 points in K2 lanes), the second the other way round, so it starts in
// the registers where the first ends and two transposes do.  The upper half
// of the input is zero (the first butterfly of the K2 points is a twiddle) and
// the upper half of the output is not wanted.
//
// K = 424 (8 x 53) and the like went through a zero-padded buffer and cuFFT
// (radix 53, or its own chirp transform of twice nfft, on data that is 7/8
// zeros): 512 pulses of 424 samples, 8 times upsampled, 55 us with the pair
// rows of the time, 50 without, 23 us here; 777 of 501: 96 and 79 to 31 us.
template <int K2, int R>
struct CztTable {
    static_assert(K2 == 32 && (R == 4 || R == 8), "the chirp kernel's shapes");
    static constexpr int M = 32 * K2, KM = M / 2;
    static constexpr int kChirp = 0;               // c[k], k < KM
    static constexpr int kH = KM;                  // H[u], u < M
    static constexpr int kTw = kH + M;             // W_M^{k1 m2} at m2 * 32 + k1
    static constexpr int kWn = kTw + M;            // W_N^i, i < 32 R
    static constexpr int kWnk = kWn + 32 * R;      // W_N^{32 i}, i < K2 / 2 * R
    static constexpr int kSize = kWnk + K2 / 2 * R;
    // row of one sub-transform: K2 x 33 for the transposes, and 16/R mod 16 as RcTable::kReg
    static constexpr int kReg = (33 * K2 + 15) / 16 * 16 + 16 / R;
    static constexpr size_t kSmem = (static_cast<size_t>(KM) + kSize + static_cast<size_t>(R) * kReg) * 8;
};

template <int K2, int R>
__device__ __forceinline__ void rc_czt_body(const float2 *__restrict__ ph, const float2 *__restrict__ fac,
                                            const float2 *__restrict__ tab, float2 *__restrict__ rc, int K, int np) {
    using T = CztTable<K2, R>;
    constexpr int REG = T::kReg, LOGR = log2_of<R>(), H2 = K2 / 2;
    extern __shared__ __align__(16) float2 rc_sm[];
    float2 *y = rc_sm, *tb = y + T::KM, *regions = tb + T::kSize;
    const int tid = threadIdx.x, r = tid >> 5, lane = tid & 31;
    for (int i = tid; i < T::kSize; i += 32 * R) tb[i] = tab[i];
    for (int k = K + tid; k < T::KM; k += 32 * R) y[k] = make_float2(0.0f, 0.0f);
    const float2 *chirp = tb + T::kChirp;
    float2 *reg = regions + r * REG;
    const int N = R * K;
    // a pulse's input samples, loaded one pulse ahead as in rc_fused_body
    constexpr int KPT = (T::KM + 32 * R - 1) / (32 * R);
    float2 pre[KPT];
    auto prefetch = [&](int q) {
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const int k = tid + j * 32 * R;
            pre[j] = (q < np && k < K) ? ph[static_cast<long long>(q) * K + k] : make_float2(0.0f, 0.0f);
        }
    };
    prefetch(blockIdx.x);
    for (int p = blockIdx.x; p < np; p += gridDim.x) {
        // the factors before the barrier, as in rc_fused_body
        float2 f[KPT];
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const int k = tid + j * 32 * R;
            f[j] = k < K ? fac[k] : make_float2(0.0f, 0.0f);
        }
        __syncthreads();  // the previous pulse's reads of the regions are done; the table is staged
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const int k = tid + j * 32 * R;
            if (k < K) y[k] = cmulf(cmulf(pre[j], f[j]), chirp[k]);
        }
        __syncthreads();
        {
            // K2 points over k2 in lane k1, the upper half of the input zero
            const float2 a = tb[T::kWn + lane * r];
            float2 lo[H2], hi[H2];
#pragma unroll
            for (int k2 = 0; k2 < H2; ++k2) {
                lo[k2] = cmulf(y[lane + 32 * k2], cmulf(a, tb[T::kWnk + k2 * r]));
                const int e32 = k2 * (32 / K2);
                hi[k2] = e32 == 0 ? lo[k2]
                                  : (e32 == 8 ? make_float2(-lo[k2].y, lo[k2].x) : cmulf(lo[k2], w32(e32)));
            }
            ifft_dif<H2>(lo);
            ifft_dif<H2>(hi);
#pragma unroll
            for (int m2 = 0; m2 < K2; ++m2) {
                const int at = bit_reverse<K2>(m2);
                reg[m2 * 33 + lane] = cmulf(at < H2 ? lo[at < H2 ? at : 0] : hi[at < H2 ? 0 : at - H2],
                                            tb[T::kTw + m2 * 32 + lane]);
            }
        }
        __syncwarp();
        {
            float2 w[32];
#pragma unroll
            for (int k1 = 0; k1 < 32; ++k1) w[k1] = reg[lane * 33 + k1];
            __syncwarp();
            ifft_dif<32>(w);
            // times H, conjugated: the second transform runs in the same direction
            float2 z[32];
#pragma unroll
            for (int m1 = 0; m1 < 32; ++m1) {
                const float2 x = cmulf(w[bit_reverse<32>(m1)], tb[T::kH + m1 * K2 + lane]);
                z[m1] = make_float2(x.x, -x.y);
            }
            ifft_dif<32>(z);
#pragma unroll
            for (int v1 = 0; v1 < 32; ++v1)
                reg[lane * 33 + v1] = cmulf(z[bit_reverse<32>(v1)], tb[T::kTw + v1 * 32 + lane]);
        }
        __syncwarp();
        float2 q[K2];
#pragma unroll
        for (int m2 = 0; m2 < K2; ++m2) q[m2] = reg[m2 * 33 + lane];
        __syncwarp();
        ifft_dif<K2>(q);
#pragma unroll
        for (int v2 = 0; v2 < H2; ++v2) {
            const float2 x = q[bit_reverse<K2>(v2)];
            reg[lane + 32 * v2] = cmulf(make_float2(x.x, -x.y), chirp[lane + 32 * v2]);
        }
        __syncthreads();
        prefetch(p + gridDim.x);
        // rc[R m + r] = regions[r][m]
        float4 *row = reinterpret_cast<float4 *>(rc + static_cast<long long>(p) * N);
        for (int b = 2 * tid; b < N; b += 64 * R) {
            const float2 u = regions[(b & (R - 1)) * REG + (b >> LOGR)];
            const float2 un = regions[((b + 1) & (R - 1)) * REG + ((b + 1) >> LOGR)];
            row[b >> 1] = make_float4(u.x, u.y, un.x, un.y);
        }
    }
}

// registers for two CTAs of 256 threads per SM
template <int K2, int R>
__global__ void __launch_bounds__(32 * R, 2) rc_czt_kernel(const __grid_constant__ RcArgs a) {
    const RcJob j(a);
    rc_czt_body<K2, R>(j.ph, j.fac, a.tab, j.rc, j.K, j.np);
}

// x <- sum_k x[k] exp(+j 2 pi u k / M), M a power of two (double, host)
void dft_pow2(std::vector<std::complex<double>> &x) {
    const size_t M = x.size();
    for (size_t i = 1, j = 0; i < M; ++i) {
        size_t bit = M >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) std::swap(x[i], x[j]);
    }
    for (size_t len = 2; len <= M; len <<= 1)
        for (size_t k = 0; k < len / 2; ++k) {
            const std::complex<double> w = std::polar(1.0, 2.0 * M_PI * static_cast<double>(k) / static_cast<double>(len));
            for (size_t i = k; i < M; i += len) {
                const std::complex<double> a = x[i], b = x[i + len / 2] * w;
                x[i] = a + b;
                x[i + len / 2] = a - b;
            }
        }
}

template <int K2, int R>
void fill_czt_table(int K, std::vector<float> &t) {
    using T = CztTable<K2, R>;
    t.assign(2 * static_cast<size_t>(T::kSize), 0.0f);
    auto put = [&](int at, const std::complex<double> &v) {
        t[2 * static_cast<size_t>(at)] = static_cast<float>(v.real());
        t[2 * static_cast<size_t>(at) + 1] = static_cast<float>(v.imag());
    };
    auto unit = [](double num, double den) { return std::polar(1.0, 2.0 * M_PI * num / den); };
    std::vector<std::complex<double>> h(T::M);
    for (int k = 0; k < K; ++k) {
        const std::complex<double> c = unit(static_cast<double>((static_cast<long long>(k) * k) % (2 * K)), 2.0 * K);
        put(T::kChirp + k, c);
        h[k] = std::conj(c) / static_cast<double>(T::M);
        if (k > 0) h[T::M - k] = h[k];
    }
    dft_pow2(h);
    for (int u = 0; u < T::M; ++u) put(T::kH + u, h[u]);
    for (int m2 = 0; m2 < K2; ++m2)
        for (int k1 = 0; k1 < 32; ++k1)
            put(T::kTw + m2 * 32 + k1, unit(static_cast<double>(k1) * m2, T::M));
    const double N = static_cast<double>(R) * K;
    for (int i = 0; i < 32 * R; ++i) put(T::kWn + i, unit(i, N));
    for (int i = 0; i < K2 / 2 * R; ++i) put(T::kWnk + i, unit(32.0 * i, N));
}

template <int K2, int R>
void fill_rc_table(std::vector<float> &t) {
    using T = RcTable<K2, R>;
    t.assign(2 * static_cast<size_t>(T::kSize), 0.0f);
    auto put = [&](int at, double num, double den) {
        const double a = 2.0 * M_PI * num / den;
        t[2 * static_cast<size_t>(at)] = static_cast<float>(std::cos(a));
        t[2 * static_cast<size_t>(at) + 1] = static_cast<float>(std::sin(a));
    };
    for (int m2 = 0; m2 < K2; ++m2)
        for (int k1 = 0; k1 < 32; ++k1) put(T::kTwk + m2 * 32 + k1, static_cast<double>(k1) * m2, T::K);
    for (int i = 0; i < 32 * R; ++i) put(T::kWn + i, i, T::N);
    for (int i = 0; i < T::NW; ++i) put(T::kWnr + i, i, T::NW);
}

int grid_for(long long total) {
    long long blocks = (total + 255) / 256;
    const long long cap = 148LL * 16;
    return static_cast<int>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

}  // namespace

cudaError_t launch_rc_prep(int precision, const void *ph, const void *fac, void *fft_buf, int K, int nfft, int np,
                           cudaStream_t s) {
    const long long total = static_cast<long long>(np) * nfft;
    if (precision == SARBP_PRECISION_FP64)
        rc_prep_kernel<double2><<<grid_for(total), 256, 0, s>>>(static_cast<const float2 *>(ph),
                                                                 static_cast<const double2 *>(fac),
                                                                 static_cast<double2 *>(fft_buf), K, nfft, total);
    else
        rc_prep_kernel<float2><<<grid_for(total), 256, 0, s>>>(static_cast<const float2 *>(ph),
                                                               static_cast<const float2 *>(fac),
                                                               static_cast<float2 *>(fft_buf), K, nfft, total);
    return cudaGetLastError();
}

cudaError_t launch_rc_prep_batch(const BatchScene *scenes, int nscenes, cudaStream_t s) {
    if (nscenes < 1 || nscenes > 65535) return cudaErrorInvalidValue;
    rc_prep_batch_kernel<<<dim3(128, nscenes), 256, 0, s>>>(scenes);
    return cudaGetLastError();
}

// (K2, R) of the direct kernels (K = 32 K2) and of the chirp kernels (K <= 16
// K2, the upsampling factors in use).
#define SARBP_RC_SHAPES(X) \
    X(8, 1) X(8, 2) X(8, 4) X(8, 8) X(8, 16) X(16, 1) X(16, 2) X(16, 4) X(16, 8) X(16, 16) X(32, 1) X(32, 2) \
        X(32, 4) X(32, 8) X(32, 16)
#define SARBP_CZT_SHAPES(X) X(32, 4) X(32, 8)

bool rc_direct_shape(int K) { return K == 256 || K == 512 || K == 1024; }

namespace {

// Whether `pulses` pulses of K samples take the chirp kernel: where cuFFT has
// long prime factors to work through.  The chirp kernel's time hardly depends
// on K, cuFFT's on the factors (2048 pulses, 4 / 8 times upsampled, chirp 42 /
// 63 us; taper and cuFFT: K = 424 (53) 71 / 144, 244 (61) 47 / 79, 301 (43) 56 /
// 73, 319 (11 29) 55 / 61, 377 (13 29) 48 / 75; but 285 (19) 21 / 35, 276 (23)
// 21 / 31, 372 (31) 28 / 58, 260 (13) 24 / 32).  With a
// factor of 17 to 31 alone the smaller K go either way, by the number of
// pulses: K = 304, 8 times, 350 pulses 20 against 17 us, 1024 39 / 27; from 385
// on cuFFT's 8 times upsampled transforms fall behind (399 63 / 71, 460 65 /
// 73, 483 66 / 83).
bool chirp_pays(int K, int pulses) {
    if (K <= 192 || K > 512) return false;
    int prime = 1, sum = 0;  // the longest factor; the sum of those from 11 on
    for (int f = 2, left = K; left > 1; ++f) {
        if (left % f == 0 && f >= 11) sum += f;
        for (; left % f == 0; left /= f) prime = f;
    }
    if (prime >= 53) return true;
    return K > 256 && (sum >= 37 || (prime >= 17 && (K >= 385 || pulses <= 768)));
}

// Calls f(kernel, shared memory, table filler) of shape (K, R); false when
// there is none.
template <typename F>
bool with_rc_shape(int K, int R, F f) {
#define SARBP_RC_CASE(K2_, R_)                                                             \
    if (K == 32 * K2_ && R == R_) {                                                        \
        f(rc_fused_kernel<K2_, R_>, RcTable<K2_, R_>::kSmem,                               \
          [](int, std::vector<float> &t) { fill_rc_table<K2_, R_>(t); });                  \
        return true;                                                                       \
    }
    SARBP_RC_SHAPES(SARBP_RC_CASE)
#undef SARBP_RC_CASE
#define SARBP_RC_CASE(K2_, R_)                                                             \
    if (K <= 16 * K2_ && !rc_direct_shape(K) && R == R_) {                                 \
        f(rc_czt_kernel<K2_, R_>, CztTable<K2_, R_>::kSmem,                                \
          [](int k, std::vector<float> &t) { fill_czt_table<K2_, R_>(k, t); });            \
        return true;                                                                       \
    }
    SARBP_CZT_SHAPES(SARBP_RC_CASE)
#undef SARBP_RC_CASE
    return false;
}

cudaError_t launch_rc(const RcArgs &a, int K, int R, dim3 grid, cudaStream_t s) {
    cudaError_t e = cudaErrorInvalidValue;
    with_rc_shape(K, R, [&](auto kern, size_t bytes, auto) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
        if (e != cudaSuccess) return;
        kern<<<grid, 32 * R, bytes, s>>>(a);
        e = cudaGetLastError();
    });
    return e;
}

}  // namespace

bool rc_fused_shape(int K, int R, int pulses, size_t *smem, std::vector<float> *table) {
    if (!rc_direct_shape(K) && !chirp_pays(K, pulses)) return false;
    return with_rc_shape(K, R, [&](auto, size_t bytes, auto fill) {
        if (smem) *smem = bytes;
        if (table) fill(K, *table);
    });
}

int rc_fused_resident(int K, int R) {
    int occ = 0;
    with_rc_shape(K, R, [&](auto kern, size_t bytes, auto) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * R, bytes) != cudaSuccess) {
            cudaGetLastError();
            occ = 0;
        }
    });
    return occ;
}

cudaError_t launch_rc_fused(const void *ph, const void *fac, const void *table, void *rc, int K, int R, int np,
                            int grid, cudaStream_t s) {
    const RcArgs a{nullptr, static_cast<const float2 *>(ph), static_cast<const float2 *>(fac),
                   static_cast<const float2 *>(table), static_cast<float2 *>(rc), K, np, {}};
    const int g = np < grid ? np : grid;
    return launch_rc(a, K, R, dim3(static_cast<unsigned>(g > 0 ? g : 1)), s);
}

cudaError_t launch_rc_fused_scenes(const BatchScene *scenes, const unsigned short *idx, int n, const void *table, int K,
                                   int R, int grid, cudaStream_t s) {
    if (n < 1 || n > kRcGroup) return cudaErrorInvalidValue;
    RcArgs a{scenes, nullptr, nullptr, static_cast<const float2 *>(table), nullptr, 0, 0, {}};
    for (int i = 0; i < n; ++i) a.idx[i] = idx[i];
    return launch_rc(a, K, R, dim3(static_cast<unsigned>(grid > 0 ? grid : 1), static_cast<unsigned>(n)), s);
}

}  // namespace sarbp
