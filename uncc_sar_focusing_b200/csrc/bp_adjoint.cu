// bp_adjoint.cu -- gradient of an image loss with respect to the per-pulse
// geometry (antenna position and slant range), for sm_100a.
//
// The forward operator is img_q = sum_p v_p(b_pq) exp(j phi_pq) with
// b = lambda dR + nfft/2, phi = kr dR (kr = 2 pi 2 f0 / c) and
// dR = |a_p - x_q| - R0_p (bp_mixed.cu).  For a real loss with upstream
// gradient G_q = dL/dRe(img_q) + j dL/dIm(img_q):
//     dL/d(dR_pq) = s_pq = Re(conj(G_q) (lambda v'_p(b) + j kr v_p(b)) exp(j phi))
//     dL/da_p = sum_q s_pq u_pq (u_pq the unit vector pixel -> antenna),
//     dL/dR0_p = -sum_q s_pq.
// v'_p(b) is the slope of the linear interpolation, rc[b+1] - rc[b], which the
// rewritten windows hold.  Nothing per pixel-pulse is stored: the kernel
// recomputes the geometry of every (tile, pulse) exactly as the forward kernel
// does (same records, polynomial tables, shared-memory windows and FP32 per-pixel
// arithmetic).
//
// Per pixel the kernel holds G_q as |G_q| exp(j psi_q), so that with
// nu = kr / lambda and Z = v' + j nu v
//     s_pq = lambda |G_q| Re(Z exp(j (phi - psi_q))):
// the conjugate product with G becomes a phase offset folded into the sine /
// cosine argument, and lambda leaves the pixel loop.  The producing warps
// rewrite each window entry to {v' + j nu c, j nu v'} (the intercept form's
// c = v_n - (n - W) v'_n), so Z at a pixel's window-centred bin B is one
// fused multiply-add per component, Z = Zc + B Zv.  Writing d = (i dx, j dy, 0)
// for a pixel's offset from the tile centre (i, j its row and column offsets)
// and Rc/R_q = 1 + t_eff/Rc, d/R_q = d_eff/Rc (far field: t_eff = u.d =
// i ux dx + j uy dy, d_eff = d; near field: the exact ratios),
//     sum_q s u_q = u (E0 + Et/Rc) - (dx Ei, dy Ej, 0)/Rc
// with E0 = sum s, Ei = sum s i (Rc/R), Ej = sum s j (Rc/R) and Et = sum s t_eff.
// In the far field t_eff is linear in (i, j), so a thread accumulates only
// sum |G| Re(..) per column and row step * |G| Re(..) over its pixels and Et
// follows from Ei and Ej.
//
// Work split: the (tile, pulse-stage) units are divided over the resident
// CTAs in contiguous ranges (bp_tile.cuh); every unit writes the per-tile
// partial gradients of its own pulses, so no fix-up pass is needed.  As in
// the forward kernel two warps produce the stages; they also add the 8 warps'
// sums of each consumed stage and write them out.  A warp reduces the 4 sums
// of a pulse with one transposed butterfly (each step halves the values a
// lane holds), and adjoint_reduce_kernel sums the tiles per pulse in double,
// in a fixed order.
//
// What bounds it: 21.7 warp instructions per warp-pixel-pulse at 65% of issue
// slots (20.8 before, where the gathers of the 32 lanes of a row took 9.3
// shared-memory wavefronts a pixel-pulse instead of 5.8 whenever the look
// direction lay along the columns).  2048 pulses x 1024^2 pixels, look
// direction 0 / 45 / 90 degrees from the rows: 2.00 / 2.41 / 2.26 ms before,
// 1.93 / 1.95 / 1.93 ms now.  The 32 registers of the pixels' |G| and psi
// leave the 96-register budget of 20 warps short: some 3 of the instructions are
// moves that a 142-register build (10 warps, 2.39 ms) does not need.
#include <algorithm>
#include <cstdint>

#include "bp_common.cuh"
#include "bp_tile.cuh"
#include "sarbp_internal.h"

namespace sarbp {
namespace {

using namespace tile;

// s^ = |G| s~, s~ = Re(Z exp(j theta)), of the thread's MX x 2 pixels for one
// pulse.  Far field: S = sum s^ per column (x: l = 0, y: l = 1) and K = sum k
// s^ over the row steps k - kMid.
// Near field: E += (s^, s^ r i, s^ r j, s^ Rc (r - 1)), r = Rc/R.
template <int MX, bool GATE, bool NEAR>
__device__ __forceinline__ void adjoint_pulse(const PulseGeo &g, const float4 *tab, uint32_t w_addr,
                                              uint32_t zero_addr, int entry, int col, const BpLaunch &L,
                                              const float2 (&npsi)[MX], const float2 (&gm)[MX], float2 &S, float2 &K,
                                              float4 &E) {
    using M = PixelMap<MX>;
    const PixelPoly<true> poly(g, tab, entry, col);
    // B is the window-centred bin (entry floor(B) + W, Z form)
    const uint32_t w_adj = w_addr + (static_cast<uint32_t>(L.W) - kRoundMagicBits) * 16u;
    S = K = make_float2(0.0f, 0.0f);
    poly.rows<MX>([&](int k, float2 P, float2 B) {
        float2 rr = make_float2(1.0f, 1.0f);  // Rc / R_q (near field only)
        const float fi = static_cast<float>(M::mid_row(entry) + M::kStep * (k - M::kMid));
        if (NEAR) {
            float2 s;
            const float2 r = near_remainder(g, L, fi, poly.J, s);
            P = __ffma2_rn(splat(g.kr), r, P);
            B = __ffma2_rn(splat(static_cast<float>(L.lambda)), r, B);
            rr = make_float2(g.rc / (s.x + r.x), g.rc / (s.y + r.y));
        }
        // theta = phi - psi, bin B and its floor split as in the forward kernel
        const float2 TH = __fadd2_rn(P, npsi[k]);
        const float2 y = __fadd2_rd(B, splat(kRoundMagic));
        float2 ZR, NZI, CS, SN;  // the pair's Re Z, -Im Z and rotations
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const float Tl = l ? TH.y : TH.x;
            const float yl = l ? y.y : y.x;
            const float Bl = l ? B.y : B.x;
            float sn, cs;
            __sincosf(Tl, &sn, &cs);
            uint32_t addr;
            asm("mad.lo.u32 %0, %1, 16, %2;" : "=r"(addr) : "r"(__float_as_uint(yl)), "r"(w_adj));
            if (GATE) {
                const bool valid = (Bl > poly.lo) && (Bl < poly.hi);
                addr = valid ? addr : zero_addr;
            }
            // Z-form entry {Zc, Zv}: Z(B) = v' + j nu v(B) = Zc + B Zv
            const float4 v = lds128(addr);
            const float zr = fmaf(Bl, v.z, v.x);
            const float nzi = fmaf(-Bl, v.w, -v.y);
            if (l) {
                ZR.y = zr;
                NZI.y = nzi;
                CS.y = cs;
                SN.y = sn;
            } else {
                ZR.x = zr;
                NZI.x = nzi;
                CS.x = cs;
                SN.x = sn;
            }
        }
        // s~ = Re(Z exp(j theta)) of the pair as paired FP32
        const float2 st = __ffma2_rn(ZR, CS, __fmul2_rn(NZI, SN));
        if (NEAR) {
            const float2 sh = __fmul2_rn(gm[k], st);
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const float s = l ? sh.y : sh.x;
                const float r = l ? rr.y : rr.x;
                const float sr = s * r;
                E.x += s;
                E.y = fmaf(sr, fi, E.y);
                E.z = fmaf(sr, l ? poly.J.y : poly.J.x, E.z);
                E.w = fmaf(s, g.rc * (r - 1.0f), E.w);
            }
        } else if (k != M::kMid) {
            const float2 sh = __fmul2_rn(gm[k], st);
            S = __fadd2_rn(S, sh);
            K = __ffma2_rn(splat(static_cast<float>(k - M::kMid)), sh, K);
        } else {
            S = __ffma2_rn(gm[k], st, S);
        }
    });
}

// The warp sums of N values (N = 4, 8, 16 or 32) at once: each step swaps
// half of a lane's values with the partner lane and adds, so N - 1 + 5 -
// log2(N) shuffles give lane L the sum of value (L >> (5 - log2 N)).
template <int N>
__device__ __forceinline__ float warp_reduce_scatter(float (&v)[N], int lane) {
    static_assert(N == 4 || N == 8 || N == 16 || N == 32, "value count");
    int o = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float send = upper ? v[i] : v[i + h];
            const float keep = upper ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float r = v[0];
#pragma unroll
    for (; o >= 1; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}

// Entries of a lane per round of the window rewrite (tile::rewrite_window).
template <int PB, int MINB>
constexpr int kAdjRewriteGroup = PB >= 4 ? 2 : (PB == 2 ? 4 : (MINB == 1 ? 8 : 6));

// Threads of an adjoint CTA: kThreads accumulating and the producing warps.
template <int PB>
constexpr int kAdjThreads = kThreads + 32 * Producers<PB>::kWarps;
// Shared-memory header: six mbarriers (full, ready, empty; two buffers each)
// and the zero entry.
constexpr int kAdjHdr = 64;

template <int MX, int PB, int MINB>
__global__ void __launch_bounds__(kAdjThreads<PB>, MINB)
    bp_adjoint_kernel(const __grid_constant__ BpLaunch L, const float2 *__restrict__ grad,
                      float4 *__restrict__ partials) {
    using M = PixelMap<MX>;
    constexpr int TX = 8 * MX;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    float4 *zero = reinterpret_cast<float4 *>(smem + kAdjHdr - 16);
    PulseGeo *geo = reinterpret_cast<PulseGeo *>(smem + kAdjHdr);
    float4 *tabs = reinterpret_cast<float4 *>(smem + kAdjHdr + 2 * PB * sizeof(PulseGeo));
    // the warps' sums of each pulse, [buffer][pulse][sum][warp]
    float *red = reinterpret_cast<float *>(tabs + 2 * PB * kPolyEntries);
    const uint32_t win_addr = smem_addr(red + 2 * PB * 4 * kWarps);
    const uint32_t zero_addr = smem_addr(zero);
    const uint32_t pulse_bytes = static_cast<uint32_t>(L.wsize) * 16u;
    const uint32_t buf_bytes = static_cast<uint32_t>(PB) * pulse_bytes;

    const TileGrid tg = tile_grid(L, TX, PB);
    const long long G = gridDim.x;
    const long long lo = sk_lo(blockIdx.x, tg.units, G);
    const int n = static_cast<int>(sk_lo(blockIdx.x + 1, tg.units, G) - lo);
    if (n <= 0) return;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    UnitCursor cur;  // this warp's unit
    cur.init(tg, L, lo);
    auto tile_of = [&](const UnitCursor &u) {
        return ((static_cast<long long>(u.hyp) * L.nz + u.iz) * tg.tiles_x + u.tx) * tg.tiles_y + u.ty;
    };

    // full (windows landed) at bar_base + 8 s, ready (Z form) at + 16 + 8 s,
    // empty (consumed, sums written) at + 32 + 8 s
    const uint32_t bar_base = smem_addr(&bars[0]);
    auto ready_bar = [&](int b) { return bar_base + 16u + 8u * b; };
    auto empty_bar = [&](int b) { return bar_base + 32u + 8u * b; };
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_base + 8u * b, PB);
            mbar_init(ready_bar(b), Producers<PB>::kWarps);
            mbar_init(empty_bar(b), kWarps);
        }
        *zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        fence_mbar_init();
    }
    __syncthreads();

    if (warp >= kWarps) {
        // A producing warp (as in bp_mixed.cu) also finishes its pulses of
        // each consumed stage: lane q adds the 8 warps' sums of pulse q in
        // warp order and writes the tile's partial gradient, so the
        // accumulating warps meet at no barrier.
        constexpr int NQ = Producers<PB>::kPulses;
        const int q0 = (warp - kWarps) * NQ;  // this warp's pulses of each stage
        const float lam = static_cast<float>(L.lambda), inv_lam = static_cast<float>(1.0 / L.lambda);
        auto finish = [&](int s, const UnitCursor &u) {
            const int p = u.b * PB + q0 + lane;
            if (lane < NQ && p < L.np) {
                const PulseGeo &g = geo[s * PB + q0 + lane];
                float4 out = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (g.flags & PG_ACTIVE) {
                    const float4 *r = reinterpret_cast<const float4 *>(red + (s * PB + q0 + lane) * 4 * kWarps);
                    float t[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 a = r[2 * c], b = r[2 * c + 1];
                        t[c] = ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
                    }
                    // exchanged tile: the record's x, y and the sums' i, j are
                    // the image's y, x
                    const bool ex = g.flags & PG_EXCHANGED;
                    const float dx = static_cast<float>(ex ? L.dy : L.dx), dy = static_cast<float>(ex ? L.dx : L.dy);
                    // sum s u_q = u (E0 + Et/Rc) - (dx Ei, dy Ej, 0)/Rc, times
                    // lambda; dL/dR0 = -lambda E0
                    const float Et = (g.flags & PG_NEAR) ? t[3] : fmaf(g.tx, t[1], g.ty * t[2]);
                    const float c = fmaf(Et, g.rinv, t[0]);
                    out.x = lam * fmaf(g.ux, c, -dx * t[1] * g.rinv);
                    out.y = lam * fmaf(g.uy, c, -dy * t[2] * g.rinv);
                    out.z = lam * g.uz * c;
                    out.w = -lam * t[0];
                    if (ex) out = make_float4(out.y, out.x, out.z, out.w);
                }
                partials[tile_of(u) * L.np + p] = out;
            }
            __syncwarp();
        };
        const bool pregeo = L.geo_tab != nullptr;
        StageRecords<NQ> pre;
        if (pregeo) pre.load(L, tile_of(cur), cur.b * PB + q0, lane);
        UnitCursor fin = cur;  // the next stage to finish
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            if (i >= 2) {
                if (!mbar_wait_bounded(empty_bar(s), ((i - 2) >> 1) & 1, L.err)) return;
                finish(s, fin);
                fin.advance(tg, L);
            }
            PulseGeo *rec = geo + s * PB + q0;
            const uint32_t win = win_addr + s * buf_bytes + static_cast<uint32_t>(q0) * pulse_bytes;
            const int p0 = cur.b * PB + q0;
            produce_pulses<MX, NQ>(L, p0, cur.tx, cur.ty, cur.iz, cur.hyp, pre, pregeo, rec,
                                   tabs + (s * PB + q0) * kPolyEntries, win, bar_base + 8u * s, lane);
            cur.advance(tg, L);
            if (pregeo && i + 1 < n) pre.load(L, tile_of(cur), cur.b * PB + q0, lane);
            if (!mbar_wait_bounded(bar_base + 8u * s, (i >> 1) & 1, L.err)) return;
            rewrite_pulses<NQ, true, kAdjRewriteGroup<PB, MINB>>(L, p0, rec, win, lane, inv_lam);
            if (lane == 0) mbar_arrive(ready_bar(s));
        }
        for (int i = n < 2 ? 0 : n - 2; i < n; ++i) {
            if (!mbar_wait_bounded(empty_bar(i & 1), (i >> 1) & 1, L.err)) return;
            finish(i & 1, fin);
            fin.advance(tg, L);
        }
        return;
    }

    const int entry = M::entry(warp, lane), col = M::col0(warp, lane);
    const float i0f = static_cast<float>(M::mid_row(entry)), j0f = static_cast<float>(col - kTY / 2);
    // the tile's upstream gradient as -psi and |G| per pixel pair
    float2 npsi[MX], gm[MX];
    auto load_tile = [&]() {
        const bool ex = MX == 8 && record_exchanged(L, tile_of(cur));
#pragma unroll
        for (int k = 0; k < MX; ++k) {
            const int mi = M::row0(warp, lane) + M::kStep * k;
            float ps[2], mg[2];
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const int mj = col + (kTY / 2) * l;
                const int row = cur.tx * TX + (ex ? mj : mi), c = cur.ty * kTY + (ex ? mi : mj);
                const float2 q = (row < L.nx && c < L.ny)
                                     ? grad[(static_cast<long long>(cur.iz) * L.nx + row) * L.ny + c]
                                     : make_float2(0.0f, 0.0f);
                ps[l] = -atan2f(q.y, q.x);
                mg[l] = sqrtf(fmaf(q.x, q.x, q.y * q.y));
            }
            npsi[k] = make_float2(ps[0], ps[1]);
            gm[k] = make_float2(mg[0], mg[1]);
        }
    };
    load_tile();

    for (int i = 0; i < n; ++i) {
        const int s = i & 1;
        // a wait that runs out (error bit set) ends this warp; the others end at theirs
        if (!mbar_wait_bounded(ready_bar(s), (i >> 1) & 1, L.err)) return;
        const int nq = min(PB, L.np - cur.b * PB);
        const uint32_t w0 = win_addr + s * buf_bytes;
#pragma unroll 1
        for (int q = 0; q < nq; ++q) {
            const PulseGeo &g = geo[s * PB + q];
            const float4 *tq = tabs + (s * PB + q) * kPolyEntries;
            const uint32_t w = w0 + q * pulse_bytes;
            const int flags = g.flags;
            if (!(flags & PG_ACTIVE)) continue;
            float v[4];
            if (!(flags & PG_NEAR)) {
                float2 S, K;
                float4 E;
                if (flags & PG_GATE)
                    adjoint_pulse<MX, true, false>(g, tq, w, zero_addr, entry, col, L, npsi, gm, S, K, E);
                else
                    adjoint_pulse<MX, false, false>(g, tq, w, zero_addr, entry, col, L, npsi, gm, S, K, E);
                // E0, Ei = i0 E0 + 2 sum k s^, Ej = j0 E0 + 32 sum_(l=1) s^; Et follows from them
                v[0] = S.x + S.y;
                v[1] = fmaf(i0f, v[0], static_cast<float>(M::kStep) * (K.x + K.y));
                v[2] = fmaf(j0f, v[0], static_cast<float>(kTY / 2) * S.y);
                v[3] = 0.0f;
            } else {
                float2 S, K;
                float4 E = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                adjoint_pulse<MX, true, true>(g, tq, w, zero_addr, entry, col, L, npsi, gm, S, K, E);
                v[0] = E.x;
                v[1] = E.y;
                v[2] = E.z;
                v[3] = E.w;
            }
            // lane 8 c holds the warp's sum c
            const float rs = warp_reduce_scatter<4>(v, lane);
            if ((lane & 7) == 0) red[((s * PB + q) * 4 + (lane >> 3)) * kWarps + warp] = rs;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(s));
        if (i + 1 < n) {
            cur.advance(tg, L);
            if (cur.b == 0) load_tile();
        }
    }
}

// out[p] = sum over tiles of partials[t][p], in double.  Block: 32 pulses
// (the lanes) x kRedWarps warps; warp w sums tiles w, w + kRedWarps, ...,
// then warp 0 adds the warps in order (a fixed order: the result does not
// depend on scheduling).  Outputs: grad_ant [3][np] (x, y, z) and
// grad_r0 [np] (may be null).
constexpr int kRedWarps = 16;

__global__ void __launch_bounds__(32 * kRedWarps)
    adjoint_reduce_kernel(const float4 *__restrict__ partials, long long ntiles, int np, double *__restrict__ grad_ant,
                          double *__restrict__ grad_r0, int accumulate) {
    __shared__ double sums[kRedWarps][4][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    double gx = 0.0, gy = 0.0, gz = 0.0, gr = 0.0;
    if (p < np) {
        for (long long t = w; t < ntiles; t += kRedWarps) {
            const float4 v = partials[t * np + p];
            gx += v.x;
            gy += v.y;
            gz += v.z;
            gr += v.w;
        }
    }
    sums[w][0][lane] = gx;
    sums[w][1][lane] = gy;
    sums[w][2][lane] = gz;
    sums[w][3][lane] = gr;
    __syncthreads();
    if (w != 0 || p >= np) return;
    for (int u = 1; u < kRedWarps; ++u) {
        gx += sums[u][0][lane];
        gy += sums[u][1][lane];
        gz += sums[u][2][lane];
        gr += sums[u][3][lane];
    }
    if (accumulate) {
        grad_ant[p] += gx;
        grad_ant[np + p] += gy;
        grad_ant[2 * np + p] += gz;
        if (grad_r0) grad_r0[p] += gr;
    } else {
        grad_ant[p] = gx;
        grad_ant[np + p] = gy;
        grad_ant[2 * np + p] = gz;
        if (grad_r0) grad_r0[p] = gr;
    }
}

template <int MX, int PB>
cudaError_t launch_adj(const BpLaunch &L, const void *grad, void *partials, size_t smem, cudaStream_t s) {
    constexpr int TX = 8 * MX;
    // two CTAs per SM (96 registers) unless a stage of one pulse needs more
    // shared memory than two get
    auto kern = bp_adjoint_kernel<MX, PB, 2>;
    if constexpr (PB == 1) {
        if (smem > 113u * 1024u) kern = bp_adjoint_kernel<MX, PB, 1>;
    }
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    // one CTA per resident slot, each taking a contiguous range of units
    int dev = 0, sms = 0, occ = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kAdjThreads<PB>, smem);
    if (e != cudaSuccess) return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    const long long units = tile_grid(L, TX, PB).units;
    const long long ctas = std::min<long long>(units, static_cast<long long>(sms) * occ);
    if (ctas < 1 || ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
    // the (tile, pulse) records from the pre-pass when the plan holds room
    // for them, else computed by the producing lanes
    BpLaunch La = L;
    bool pregeo = false;
    e = launch_geo_records(La, MX, &pregeo, s);
    if (e != cudaSuccess) return e;
    if (!pregeo) La.geo_tab = nullptr;
    kern<<<static_cast<unsigned>(ctas), kAdjThreads<PB>, smem, s>>>(La, static_cast<const float2 *>(grad),
                                                              static_cast<float4 *>(partials));
    return cudaGetLastError();
}

}  // namespace

long long bp_tile_count(const BpLaunch &L, const TileConfig &tc) {
    const long long TX = 8 * tc.mx;
    return ((L.ny + 63) / 64) * ((L.nx + TX - 1) / TX) * static_cast<long long>(L.nz);
}

size_t bp_adjoint_smem_bytes(const TileConfig &tc, int wsize) {
    const size_t pb = static_cast<size_t>(tc.pb);
    return kAdjHdr + 2 * pb * (sizeof(PulseGeo) + kPolyEntries * sizeof(float4)) + 2 * kWarps * 4 * pb * sizeof(float) +
           2 * pb * static_cast<size_t>(wsize) * 16;
}

cudaError_t launch_bp_adjoint(const BpLaunch &L, const void *grad, void *partials, const TileConfig &tc, size_t smem,
                              cudaStream_t s) {
#define SARBP_ADJ_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_) return launch_adj<MX_, PB_>(L, grad, partials, smem, s);
    SARBP_ADJ_CASE(8, 8)
    SARBP_ADJ_CASE(8, 4)
    SARBP_ADJ_CASE(8, 2)  // wide windows: the stage depth halves below 4 at 64-row tiles too
    SARBP_ADJ_CASE(8, 1)
    SARBP_ADJ_CASE(4, 8)
    SARBP_ADJ_CASE(2, 8)
    SARBP_ADJ_CASE(1, 8)
    SARBP_ADJ_CASE(4, 4)
    SARBP_ADJ_CASE(4, 2)
    SARBP_ADJ_CASE(4, 1)
    SARBP_ADJ_CASE(2, 4)
    SARBP_ADJ_CASE(2, 2)
    SARBP_ADJ_CASE(2, 1)
    SARBP_ADJ_CASE(1, 4)
    SARBP_ADJ_CASE(1, 2)
    SARBP_ADJ_CASE(1, 1)
#undef SARBP_ADJ_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_adjoint_reduce(const void *partials, long long ntiles, int np, double *grad_ant, double *grad_r0,
                                  int accumulate, cudaStream_t s) {
    const int blocks = (np + 31) / 32;
    adjoint_reduce_kernel<<<blocks > 0 ? blocks : 1, 32 * kRedWarps, 0, s>>>(
        static_cast<const float4 *>(partials), ntiles, np, grad_ant, grad_r0, accumulate);
    return cudaGetLastError();
}

}  // namespace sarbp
