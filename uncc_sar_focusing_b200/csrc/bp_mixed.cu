// bp_mixed.cu -- mixed-precision forward backprojection for sm_100a.
//
// Replaces the reference kernel backprojection_loop
// (src/gpuBackProjection/cuda_sar_focusing/cuda_BackProjectionKernels.cuh:33-93)
// and its CPU twin computeDifferentialRangeAndPhaseCorrections
// (src/cpuBackProjection/cpuBackProjection.hpp:49-93):
//     img[q] += lerp(rc_p, bin(dR)) * exp(+j 4 pi f0_p dR / c),
//     dR = |a_p - x_q| - R0_p,  gate rmin < dR < rmax,
//     bracket [floor(bin), floor(bin)+1]  (CPU/MATLAB semantics, not the
//     GPU kernel's roundf bracket, cuda_BackProjectionKernels.cuh:68-74).
//
// Design (one CTA = one pixel tile of (8*MX) x 64 pixels of one z-slice at a
// time, 8 accumulating warps of MX x 2 pixels a thread and two producing warps):
//  * pulses go through shared memory in stages of PB pulses, two stage
//    buffers.  For each stage the producing warps write the FP64 geometry
//    records (tile-centre range, unit vector, phase and bin steps reduced mod
//    1), the polynomial tables and one cp.async.bulk copy per pulse of the
//    window of range bins any pixel of the tile can touch, rewrite the landed
//    windows to intercept form and mark the buffer ready; the accumulating
//    warps hand it back through the "empty" mbarrier, so they drift up to a
//    stage apart and meet nowhere;
//  * range profiles live in HBM as samples; in shared memory entry n of a
//    window is {rc[b] - (n - W) slope, slope}, slope = rc[b+1] - rc[b], so one
//    16-byte load and two FMAs on the window-centred bin interpolate;
//  * per pixel-pulse all arithmetic is FP32: phase and bin of a thread's
//    pixels are polynomials in the row step (write_poly_tables), the phase in
//    radians within a few multiples of pi of zero goes straight to
//    __sincosf; the floor of the bin comes from one round-down add whose
//    result bits also form the shared-memory address (near-field pulses add
//    the exact sqrt form of the remainder per pixel);
//  * the 8 lanes of a shared-memory wavefront are a 2 x 4 pixel patch
//    (PixelMap), laid across the look direction (tile_exchanged), so their
//    16-byte gathers rarely collide;
//  * MX = 8 (64 x 64-pixel tiles) by default: the per-(tile, pulse) and
//    per-(thread, pulse) work is spread over 16 pixels per thread.
//
// What bounds it (1024^2 pixels x 2048 pulses, 8 km, ncu): 16.1 warp
// instructions per warp-pixel-pulse at 65% of issue slots, shared memory's data
// pipe 83% busy (5.2 wavefronts, 4 of them the 16-byte gather's floor), MUFU
// 66%, 20 warps per SM.  With rows interleaved over the warps, a row of 32
// lanes and an evaluation of the range remainder per pixel it took 18.0
// instructions and 1.70 / 2.29 / 2.13 ms at look directions 0 / 45 / 90
// degrees from the rows, this 1.46 / 1.48 / 1.46 ms.  The 96 registers of 20
// warps are short: 24 bytes a thread are spilled and 44 loaded back (batches,
// whose accumulating warps carry the scene cursor too, 132 / 160).
#include <cstdint>

#include "bp_common.cuh"
#include "bp_tile.cuh"
#include "sarbp_internal.h"

namespace sarbp {
namespace {

using namespace tile;

// CTAs per SM the register budget is sized for when shared memory allows
// more than one (launch bounds of the default instantiation)
#ifndef SARBP_CTAS_PER_SM
#define SARBP_CTAS_PER_SM 2
#endif
constexpr int kCtasPerSm = SARBP_CTAS_PER_SM;

constexpr int kTabEntries = kPolyEntries;

// Entries of a lane per round of the window rewrite (tile::rewrite_window).
template <int PB>
constexpr int kRewriteGroup = PB == 1 ? 8 : (PB == 4 ? 2 : 4);

// Header of the shared memory: six mbarriers (full, ready and empty, two
// buffers each) and the zero entry.
constexpr int kHdr = 64;

// Threads of a forward CTA: kThreads accumulating and the producing warps.
template <int PB>
constexpr int kFwdThreads = kThreads + 32 * Producers<PB>::kWarps;

// Dynamic shared memory of the forward kernel: the header and two stage
// buffers of PB records, tables and windows.
__host__ __device__ constexpr size_t smem_bytes_of(int pb, int wsize) {
    return kHdr + 2 * static_cast<size_t>(pb) * (sizeof(PulseGeo) + kTabEntries * sizeof(float4)) +
           2 * static_cast<size_t>(pb) * static_cast<size_t>(wsize) * 16;
}

// pulse stages of split tiles walked in step across the resident CTAs
#ifndef SARBP_STAGE_ROTATION
#define SARBP_STAGE_ROTATION 1
#endif
constexpr bool kRotate = SARBP_STAGE_ROTATION != 0;


// One pulse into the thread's MX x 2 pixels (PixelMap).  The two columns
// (32 apart) of a row form a pair whose phase, bin and complex
// multiply-accumulate run as paired FP32 instructions (__ffma2_rn and
// friends); the sine/cosine, the shared-memory gather and the interpolation
// are per pixel.
template <int MX, bool GATE, bool NEAR, bool CHECKED>
__device__ __forceinline__ void accumulate_pulse(const PulseGeo &g, const float4 *tab, uint32_t w_addr,
                                                 uint32_t zero_addr, int entry, int col, const BpLaunch &L,
                                                 float (&acc_re)[MX][2], float (&acc_im)[MX][2]) {
    using M = PixelMap<MX>;
    const PixelPoly<false> poly(g, tab, entry, col);
    // B is the window-centred bin; shared address of entry floor(B) + W:
    // bits(B + 1.5*2^23, rounded down) * 16 + w_adj (mod 2^32)
    const uint32_t w_adj = w_addr + (static_cast<uint32_t>(L.W) - kRoundMagicBits) * 16u;
    poly.rows<MX>([&](int k, float2 P, float2 B) {
        if (NEAR) {
            float2 s;
            const float2 r = near_remainder(g, L, static_cast<float>(M::mid_row(entry) + M::kStep * (k - M::kMid)),
                                            poly.J, s);
            P = __ffma2_rn(splat(g.kr), r, P);
            B = __ffma2_rn(splat(static_cast<float>(L.lambda)), r, B);
        }
        const float2 y = __fadd2_rd(B, splat(kRoundMagic));
        float2 RE, IM, CS, SN;  // the pair's interpolated samples and rotations
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const float Pl = l ? P.y : P.x;
            const float Bl = l ? B.y : B.x;
            const float yl = l ? y.y : y.x;
            float sn, cs;
            __sincosf(Pl, &sn, &cs);
            // on the multiply-add pipe: as a shift-add on the ALU 1529 vs 1516 us
            uint32_t addr;
            asm("mad.lo.u32 %0, %1, 16, %2;" : "=r"(addr) : "r"(__float_as_uint(yl)), "r"(w_adj));
            if (GATE) {
                const bool valid = (Bl > poly.lo) && (Bl < poly.hi);
                addr = valid ? addr : zero_addr;
            }
            if (CHECKED) {
                // entry floor(B) + W must lie in the pulse's tight window
                // [W - wp, W + wp] (its next entry too)
                const uint32_t idx = __float_as_uint(yl) - kRoundMagicBits + static_cast<uint32_t>(g.wp);
                if (idx > static_cast<uint32_t>(2 * g.wp)) {
                    atomicOr(L.err, ERRBIT_BOUNDS);
                    addr = zero_addr;
                }
            }
            // intercept-form entry {c, v'}: v(B) = c + B v'
            const float4 e = lds128(addr);
            const float re = fmaf(Bl, e.z, e.x);
            const float im = fmaf(Bl, e.w, e.y);
            if (l) {
                RE.y = re;
                IM.y = im;
                CS.y = cs;
                SN.y = sn;
            } else {
                RE.x = re;
                IM.x = im;
                CS.x = cs;
                SN.x = sn;
            }
        }
        // complex multiply-accumulate of the pair as paired FP32 (same fused
        // operations as per pixel, half the instructions)
        float2 ar = make_float2(acc_re[k][0], acc_re[k][1]), ai = make_float2(acc_im[k][0], acc_im[k][1]);
        ar = __ffma2_rn(RE, CS, __ffma2_rn(make_float2(-IM.x, -IM.y), SN, ar));
        ai = __ffma2_rn(RE, SN, __ffma2_rn(IM, CS, ai));
        acc_re[k][0] = ar.x;
        acc_re[k][1] = ar.y;
        acc_im[k][0] = ai.x;
        acc_im[k][1] = ai.y;
    });
}

// Store (or add, L.accumulate) a thread's pixel pair k of the tile at (tx0,
// ty0, slice zz) into the complex64 image (PixelMap: every store of a warp is
// 16 consecutive pixels, 128 bytes, of each of two rows; in an exchanged tile
// 2 pixels of each of 16 rows, once per tile).  v: re, im of the
// first column, re, im of the second.
template <int MX>
__device__ __forceinline__ void store_pair(const BpLaunch &L, int tx0, int ty0, int zz, bool exchanged, int warp,
                                           int lane, int k, const float4 &v) {
    float2 *img = static_cast<float2 *>(L.img);
    const int i = PixelMap<MX>::row0(warp, lane) + PixelMap<MX>::kStep * k;
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const int j = PixelMap<MX>::col0(warp, lane) + (kTY / 2) * l;
        const int row = tx0 + (exchanged ? j : i), col = ty0 + (exchanged ? i : j);
        if (row >= L.nx || col >= L.ny) continue;
        const long long o = (static_cast<long long>(zz) * L.nx + row) * L.ny + col;
        float2 p = l ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
        if (L.accumulate) {
            const float2 old = img[o];
            p.x += old.x;
            p.y += old.y;
        }
        img[o] = p;
    }
}

// Index of a thread's pixel pair k in a partial-sum slot of TX x 64
// complex64 values (written and read by the same threads).
__device__ __forceinline__ int slot_pair(int k) { return k * kThreads + static_cast<int>(threadIdx.x); }

// Unit cursor over one launch (BATCH = false: the kernel parameter's scene)
// or over the scenes of a batch table, scene-major.
//
// Pulse-stage order within a tile (single-scene launches split over the
// resident CTAs): unit t S + b of tile t processes stage (b + rot_t) mod S
// with rot_t = t S - lo(owner of unit t S) mod S, the local step at which
// that CTA reaches the tile.  A CTA's k-th unit then works on stage k mod S,
// except on its first, partial tile, so the CTAs resident together walk the
// pulses in step and share the range profiles they stage through L2.  For
// the tiles a CTA reaches at their first stage rot_t = -lo(c) mod S, one
// value per CTA (rot_later); only the first tile has its own.  Every stage
// of a tile is still processed exactly once; only the order of the per-tile
// sums changes.
template <int TX, int PB, bool BATCH>
struct SceneCursor {
    const BpLaunch *L;
    TileGrid g;
    UnitCursor u;
    int scene;
    int rot;  // stage rotation of the current tile

    // pulse stage of the current unit
    __device__ __forceinline__ int stage() const {
        const int e = u.b + rot;
        return e >= g.stages ? e - g.stages : e;
    }

    // cursor at `unit` of U units split over the launch's G = gridDim.x CTAs
    __device__ __forceinline__ void init(const BpLaunch *L0, const BatchScene *scenes, int nscenes, long long unit,
                                         long long U) {
        scene = 0;
        L = L0;
        if constexpr (BATCH) {
            int a = 0, z = nscenes - 1;  // last scene with unit_begin <= unit
            while (a < z) {
                const int m = (a + z + 1) >> 1;
                if (scenes[m].unit_begin <= unit) a = m;
                else z = m - 1;
            }
            scene = a;
            L = &scenes[a].L;
            unit -= scenes[a].unit_begin;
        }
        g = tile_grid(*L, TX, PB);
        u.init(g, *L, unit);
        rot = 0;
        if constexpr (!BATCH && kRotate) {
            const long long G = gridDim.x;
            const long long first = unit - u.b;  // the tile's first unit
            rot = static_cast<int>((first - sk_lo(sk_owner(first, U, G), U, G)) % g.stages);
        }
    }
    // true when the cursor moved on to the next scene; rot_later: the stage
    // rotation of tiles entered at their first stage
    __device__ __forceinline__ bool advance(const BatchScene *scenes, int nscenes, int rot_later) {
        u.advance(g, *L);
        if (u.b == 0) rot = rot_later;
        if constexpr (BATCH) {
            if (u.hyp >= L->nhyp && scene + 1 < nscenes) {
                ++scene;
                L = &scenes[scene].L;
                g = tile_grid(*L, TX, PB);
                u.b = u.ty = u.tx = u.iz = u.hyp = 0;
                return true;
            }
        }
        return false;
    }
};

// BATCH = false: one scene, L0.  BATCH = true: the scenes of the table; L0
// carries only the batch-wide window size (the largest scene window: the
// stage buffers' stride) and sk_partial; each scene's image completion time
// goes to done[scene].
//
// Warps 0..7 accumulate; warps 8 and 9 produce, half of each stage's pulses
// each (Producers): per stage they wait until the buffer is empty, put its
// records, tables and window copies into it, rewrite the landed windows to
// intercept form and mark the buffer ready.  The 32 row entries of 4 pulses
// fill a warp's lanes (each accumulating warp producing its own pulse slot ran
// them with 8 of 32 lanes, the records with one), and the accumulating warps
// carry neither the production's instructions nor its latency.
template <int MX, int PB, bool CHECKED, int MINB, bool BATCH>
__global__ void __launch_bounds__(kFwdThreads<PB>, MINB)
    bp_mixed_kernel(const __grid_constant__ BpLaunch L0, const BatchScene *__restrict__ scenes, int nscenes,
                    long long batch_units, unsigned long long *__restrict__ done, int tile_mode) {
    constexpr int TX = 8 * MX;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    float4 *zero = reinterpret_cast<float4 *>(smem + kHdr - 16);
    PulseGeo *geo = reinterpret_cast<PulseGeo *>(smem + kHdr);
    float4 *tabs = reinterpret_cast<float4 *>(smem + kHdr + 2 * PB * sizeof(PulseGeo));
    const uint32_t win_addr = smem_addr(smem + kHdr + 2 * PB * (sizeof(PulseGeo) + kTabEntries * sizeof(float4)));
    const uint32_t buf_bytes = static_cast<uint32_t>(PB) * static_cast<uint32_t>(L0.wsize) * 16u;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    // this CTA's units [lo, lo + n) of the launch's (tile, stage) units
    const long long U = BATCH ? batch_units : tile_grid(L0, TX, PB).units;
    const long long G = gridDim.x;
    long long lo = sk_lo(blockIdx.x, U, G);
    int n = static_cast<int>(sk_lo(blockIdx.x + 1, U, G) - lo);
    if (BATCH && tile_mode) {
        // one CTA per tile of the batch, in scene order: CTA t takes tile t's stages
        int a = 0, z = nscenes - 1;  // last scene with tile_begin <= t
        while (a < z) {
            const int m = (a + z + 1) >> 1;
            if (scenes[m].tile_begin <= static_cast<long long>(blockIdx.x)) a = m;
            else z = m - 1;
        }
        const int S = tile_grid(scenes[a].L, TX, PB).stages;
        lo = scenes[a].unit_begin + (static_cast<long long>(blockIdx.x) - scenes[a].tile_begin) * S;
        n = S;
    }
    if (n <= 0) return;

    SceneCursor<TX, PB, BATCH> cur;  // this warp's unit
    cur.init(&L0, scenes, nscenes, lo, U);
    // stage rotation of the tiles this CTA enters at their first stage
    const int rot_later =
        (!BATCH && kRotate) ? static_cast<int>((cur.g.stages - lo % cur.g.stages) % cur.g.stages) : 0;

    // buffer s: full (windows landed: PB arrivals and their bytes) at
    // bar_base + 8 s, ready (intercept form, one arrival per producing warp) at bar_base + 16 +
    // 8 s, empty (consumed, one arrival per accumulating warp) at bar_base +
    // 32 + 8 s
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
        // Pre-pass records (single-scene launches: L0.geo_tab; batches: each
        // scene's L.geo_tab, L0.geo_tab non-null when every scene has them)
        // are loaded into the lanes' registers one stage ahead.
        constexpr int NQ = Producers<PB>::kPulses;
        const int q0 = (warp - kWarps) * NQ;  // this warp's pulses of each stage
        const bool pregeo = L0.geo_tab != nullptr;
        StageRecords<NQ> pre;
        auto load_records = [&]() {
            const BpLaunch &L = *cur.L;
            pre.load(L, ((static_cast<long long>(cur.u.hyp) * L.nz + cur.u.iz) * cur.g.tiles_x + cur.u.tx) * cur.g.tiles_y + cur.u.ty,
                     cur.stage() * PB + q0, lane);
        };
        if (pregeo) load_records();
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            const BpLaunch &L = *cur.L;
            // buffer s last held stage i - 2: every accumulating warp has consumed it
            if (i >= 2 && !mbar_wait_bounded(empty_bar(s), ((i - 2) >> 1) & 1, L.err)) return;
            PulseGeo *rec = geo + s * PB + q0;
            const uint32_t win = win_addr + s * buf_bytes + static_cast<uint32_t>(q0) * static_cast<uint32_t>(L.wsize) * 16u;
            const int p0 = cur.stage() * PB + q0;
            produce_pulses<MX, NQ>(L, p0, cur.u.tx, cur.u.ty, cur.u.iz, cur.u.hyp, pre, pregeo, rec,
                                   tabs + (s * PB + q0) * kTabEntries, win, bar_base + 8u * s, lane);
            cur.advance(scenes, nscenes, rot_later);
            if (pregeo && i + 1 < n) load_records();
            if (!mbar_wait_bounded(bar_base + 8u * s, (i >> 1) & 1, L.err)) return;
            rewrite_pulses<NQ, false, kRewriteGroup<PB>>(L, p0, rec, win, lane);
            if (lane == 0) mbar_arrive(ready_bar(s));
        }
        return;
    }

    const uint32_t zero_addr = smem_addr(zero);
    const int entry = PixelMap<MX>::entry(warp, lane), col = PixelMap<MX>::col0(warp, lane);
    float acc_re[MX][2], acc_im[MX][2];
#pragma unroll
    for (int k = 0; k < MX; ++k)
#pragma unroll
        for (int l = 0; l < 2; ++l) acc_re[k][l] = acc_im[k][l] = 0.0f;
    int seg = 0;                 // segments flushed so far
    int seg_first = cur.u.b;     // first stage of the open segment
    for (int i = 0; i < n; ++i) {
        const int s = i & 1;
        const BpLaunch &L = *cur.L;
        const int S = cur.g.stages;
        const int b = cur.u.b;  // position in the tile's stage order
        // a wait that runs out (error bit set) ends this warp; the others end at theirs
        if (!mbar_wait_bounded(ready_bar(s), (i >> 1) & 1, L.err)) return;
        const int nq = min(PB, L.np - cur.stage() * PB);
        // stage summary: all PB pulses active, none gated or near-field
        const int my_flags = lane < nq ? geo[s * PB + lane].flags : 0;
        const int any_f = __reduce_or_sync(0xffffffffu, my_flags);
        const int all_f = __reduce_and_sync(0xffffffffu, lane < nq ? my_flags : PG_ACTIVE);
        const uint32_t w0 = win_addr + s * buf_bytes;
        const uint32_t pulse_bytes = static_cast<uint32_t>(L.wsize) * 16u;
        if (nq == PB && (all_f & PG_ACTIVE) && !(any_f & (PG_GATE | PG_NEAR))) {
            // a loop of one pulse, 230 instructions, stays in the instruction
            // cache: with the stage's 8 pulses unrolled 1520-1691 us on the
            // large workload over look directions, as a loop 1511-1649
#pragma unroll 1
            for (int q = 0; q < PB; ++q)
                accumulate_pulse<MX, false, false, CHECKED>(geo[s * PB + q], tabs + (s * PB + q) * kTabEntries,
                                                            w0 + q * pulse_bytes, zero_addr, entry, col, L, acc_re,
                                                            acc_im);
        } else {
            for (int q = 0; q < nq; ++q) {
                const PulseGeo &g = geo[s * PB + q];
                const float4 *tq = tabs + (s * PB + q) * kTabEntries;
                const int flags = g.flags;
                if (!(flags & PG_ACTIVE)) continue;
                const uint32_t w = w0 + q * pulse_bytes;
                if (flags & PG_NEAR)
                    accumulate_pulse<MX, true, true, CHECKED>(g, tq, w, zero_addr, entry, col, L, acc_re, acc_im);
                else if (flags & PG_GATE)
                    accumulate_pulse<MX, true, false, CHECKED>(g, tq, w, zero_addr, entry, col, L, acc_re, acc_im);
                else
                    accumulate_pulse<MX, false, false, CHECKED>(g, tq, w, zero_addr, entry, col, L, acc_re, acc_im);
            }
        }
        const bool exchanged = MX == 8 && (geo[s * PB].flags & PG_EXCHANGED);
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(s));
        if (i + 1 == n || b == S - 1) {
            // the segment of this tile ends: whole tile -> image, else -> partial slot
            if (seg_first == 0 && b == S - 1) {
#pragma unroll
                for (int k = 0; k < MX; ++k)
                    store_pair<MX>(L, cur.u.tx * TX, cur.u.ty * kTY, cur.u.hyp * L.nz + cur.u.iz, exchanged, warp,
                                   lane, k, make_float4(acc_re[k][0], acc_im[k][0], acc_re[k][1], acc_im[k][1]));
                // completion time: the latest of the warps' stores
                if (BATCH && done) {
                    __syncwarp();
                    if (lane == 0) atomicMax(done + cur.scene, global_timer_ns());
                }
            } else {
                float4 *slot = static_cast<float4 *>(L0.sk_partial) +
                               (2 * static_cast<long long>(blockIdx.x) + (seg > 0 ? 1 : 0)) * (TX * kTY / 2);
#pragma unroll
                for (int k = 0; k < MX; ++k)
                    slot[slot_pair(k)] = make_float4(acc_re[k][0], acc_im[k][0], acc_re[k][1], acc_im[k][1]);
            }
#pragma unroll
            for (int k = 0; k < MX; ++k)
#pragma unroll
                for (int l = 0; l < 2; ++l) acc_re[k][l] = acc_im[k][l] = 0.0f;
            ++seg;
            seg_first = 0;
        }
        cur.advance(scenes, nscenes, rot_later);
    }
}

// Tiles whose stages were split over several CTAs: add the CTAs' partial
// sums in CTA order (a fixed order, so results repeat bit for bit) and store
// the tile.  One CTA per (tile of the launch, row step k of its threads), so
// the few tiles of a small image still fill the SMs; tiles held whole by one
// CTA return at once.
template <int MX, int PB, bool BATCH>
__global__ void __launch_bounds__(kThreads)
    bp_sk_fixup_kernel(const __grid_constant__ BpLaunch L0, const BatchScene *__restrict__ scenes, int nscenes,
                       long long units, long long G, unsigned long long *__restrict__ done) {
    constexpr int TX = 8 * MX;
    long long t = blockIdx.x, unit0 = 0;
    const BpLaunch *Lp = &L0;
    int scene = 0;
    if constexpr (BATCH) {
        int a = 0, z = nscenes - 1;  // last scene with tile_begin <= t
        while (a < z) {
            const int m = (a + z + 1) >> 1;
            if (scenes[m].tile_begin <= t) a = m;
            else z = m - 1;
        }
        scene = a;
        Lp = &scenes[a].L;
        t -= scenes[a].tile_begin;
        unit0 = scenes[a].unit_begin;
    }
    const BpLaunch &L = *Lp;
    const TileGrid tg = tile_grid(L, TX, PB);
    const long long first = unit0 + t * tg.stages;
    const long long c0 = sk_owner(first, units, G);
    const long long c1 = sk_owner(first + tg.stages - 1, units, G);
    if (c0 == c1) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.y;
    const float4 v = sk_sum(static_cast<const float4 *>(L0.sk_partial), TX * kTY / 2, slot_pair(k),
                            sk_first_slot(c0, first, units, G), c0, c1, [](float4 &s, const float4 &e) {
                                s.x += e.x;
                                s.y += e.y;
                                s.z += e.z;
                                s.w += e.w;
                            });
    int tx0, ty0, zz;
    tile_origin(tg, t, TX, tx0, ty0, zz);
    store_pair<MX>(L, tx0, ty0, zz, MX == 8 && record_exchanged(L, t), warp, lane, k, v);
    if (BATCH && done) {
        __syncthreads();
        if (threadIdx.x == 0) atomicMax(done + scene, global_timer_ns());
    }
}

// Geometry records of every (tile, pulse) of a launch, [tile][pulse], one
// thread each (make_geo, full warps), for the forward kernel's producers to
// load.  Each CTA computes 256 records into shared memory, then writes them
// out as consecutive 16-byte words (a warp stores 512 contiguous bytes).  In
// shared memory word k of record r sits at [k][r] with a row stride of 257
// words, so both the record-per-thread stores and the word-per-thread reads
// hit 8 distinct bank groups per quarter warp (a [r][k] layout put all 32
// lanes of each 16-byte store on the same four banks).  Indexes are 32-bit:
// the launch checks n < 2^31.
template <int MX>
__device__ __forceinline__ void geo_records_chunk(const BpLaunch &L, unsigned n, unsigned i0, float4 *words) {
    constexpr int TX = 8 * MX;
    constexpr int kWords = sizeof(PulseGeo) / sizeof(float4);
    constexpr int kStride = 257;
    const TileGrid tg = tile_grid(L, TX, 1);
    const unsigned np = static_cast<unsigned>(L.np), ty_n = static_cast<unsigned>(tg.tiles_y),
                   tx_n = static_cast<unsigned>(tg.tiles_x), nz = static_cast<unsigned>(L.nz);
    const unsigned i = i0 + threadIdx.x;
    if (i < n) {
        const unsigned t = i / np, p = i - t * np;
        const unsigned r = t / ty_n, ty = t - r * ty_n;
        const unsigned zz = r / tx_n, tx = r - zz * tx_n;
        const unsigned hyp = zz / nz, iz = zz - hyp * nz;
        const double cx = L.left + static_cast<double>(static_cast<int>(tx) * TX + TX / 2) * L.dx;
        const double cy = L.bottom + static_cast<double>(static_cast<int>(ty) * kTY + kTY / 2) * L.dy;
        const double cz = L.zlow + static_cast<double>(iz) * L.dz;
        const long long goff = static_cast<long long>(hyp) * L.np;
        const PulseGeo g = make_geo(L, static_cast<int>(p), goff, cx, cy, cz, TX / 2,
                                    MX == 8 && tile_exchanged(L, goff, cx, cy));
        const float4 *gw = reinterpret_cast<const float4 *>(&g);
#pragma unroll
        for (int k = 0; k < kWords; ++k) words[k * kStride + threadIdx.x] = gw[k];
    }
    __syncthreads();
    float4 *out = static_cast<float4 *>(L.geo_tab);
    const unsigned left = n - i0;
    const int nw = static_cast<int>((left < 256u ? left : 256u) * kWords);
    for (int w = threadIdx.x; w < nw; w += 256)
        out[static_cast<long long>(i0) * kWords + w] = words[(w % kWords) * kStride + w / kWords];
    __syncthreads();
}

template <int MX>
__global__ void __launch_bounds__(256) bp_geo_records_kernel(const __grid_constant__ BpLaunch L, int n) {
    __shared__ float4 words[(sizeof(PulseGeo) / sizeof(float4)) * 257];
    for (unsigned i0 = blockIdx.x * 256u; i0 < static_cast<unsigned>(n); i0 += gridDim.x * 256u)
        geo_records_chunk<MX>(L, static_cast<unsigned>(n), i0, words);
}

// The same for every scene of a batch (blockIdx.y = scene), into each
// scene's record rows (BatchScene::L.geo_tab).
template <int MX>
__global__ void __launch_bounds__(256) bp_geo_records_batch_kernel(const BatchScene *__restrict__ scenes) {
    __shared__ float4 words[(sizeof(PulseGeo) / sizeof(float4)) * 257];
    const BpLaunch &L = scenes[blockIdx.y].L;
    if (!L.geo_tab) return;
    const unsigned n = static_cast<unsigned>(tile_grid(L, 8 * MX, 1).tiles) * static_cast<unsigned>(L.np);
    for (unsigned i0 = blockIdx.x * 256u; i0 < n; i0 += gridDim.x * 256u) geo_records_chunk<MX>(L, n, i0, words);
}

template <int MX>
cudaError_t launch_records_mx(const BpLaunch &L, bool *ran, cudaStream_t s) {
    *ran = false;
    const long long nrec = tile_grid(L, 8 * MX, 1).tiles * L.np;
    if (!L.geo_tab || nrec < 1 || nrec > L.geo_tab_records || nrec >= 0x7fffffffLL) return cudaSuccess;
    const long long blocks = (nrec + 255) / 256;
    bp_geo_records_kernel<MX><<<static_cast<unsigned>(blocks < 148 * 64 ? blocks : 148 * 64), 256, 0, s>>>(
        L, static_cast<int>(nrec));
    const cudaError_t e = cudaGetLastError();
    *ran = e == cudaSuccess;
    return e;
}

}  // namespace

cudaError_t launch_geo_records(const BpLaunch &L, int mx, bool *ran, cudaStream_t s) {
    switch (mx) {
        case 8: return launch_records_mx<8>(L, ran, s);
        case 4: return launch_records_mx<4>(L, ran, s);
        case 2: return launch_records_mx<2>(L, ran, s);
        case 1: return launch_records_mx<1>(L, ran, s);
        default: *ran = false; return cudaSuccess;
    }
}

cudaError_t launch_geo_records_batch(const BatchScene *scenes, int nscenes, int mx, long long max_records,
                                     cudaStream_t s) {
    if (nscenes < 1 || nscenes > 65535 || max_records < 1 || max_records >= 0x7fffffffLL)
        return cudaErrorInvalidValue;
    const long long bx = (max_records + 255) / 256;
    const dim3 grid(static_cast<unsigned>(bx < 1024 ? bx : 1024), static_cast<unsigned>(nscenes));
    switch (mx) {
        case 8: bp_geo_records_batch_kernel<8><<<grid, 256, 0, s>>>(scenes); break;
        case 4: bp_geo_records_batch_kernel<4><<<grid, 256, 0, s>>>(scenes); break;
        case 2: bp_geo_records_batch_kernel<2><<<grid, 256, 0, s>>>(scenes); break;
        case 1: bp_geo_records_batch_kernel<1><<<grid, 256, 0, s>>>(scenes); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

namespace {

template <int MX, int PB, bool CHECKED, int MINB>
cudaError_t launch_kernels(const BpLaunch &L0, size_t smem, cudaStream_t s) {
    constexpr int TX = 8 * MX;
    auto kern = bp_mixed_kernel<MX, PB, CHECKED, MINB, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    const TileGrid tg = tile_grid(L0, TX, PB);
    if (tg.units < 1) return cudaSuccess;
    BpLaunch L = L0;
    bool pregeo = false;
    e = launch_geo_records(L, MX, &pregeo, s);
    if (e != cudaSuccess) return e;
    if (!pregeo) L.geo_tab = nullptr;
    // split the units over the resident CTAs unless the tiles fill whole waves
    long long G = tg.tiles;
    if (L.sk_partial && L.sk_resident > 0 && tg.tiles % L.sk_resident != 0) {
        const long long g = L.sk_resident < tg.units ? L.sk_resident : tg.units;
        if (2 * g * TX * kTY * static_cast<long long>(sizeof(float2)) <= L.sk_slot_bytes) G = g;
    }
    if (G > 0x7fffffffLL) return cudaErrorInvalidValue;
    kern<<<static_cast<unsigned>(G), kFwdThreads<PB>, smem, s>>>(L, nullptr, 0, 0, nullptr, 0);
    e = cudaGetLastError();
    if (e != cudaSuccess || G == tg.tiles) return e;
    bp_sk_fixup_kernel<MX, PB, false>
        <<<dim3(static_cast<unsigned>(tg.tiles), MX), kThreads, 0, s>>>(L, nullptr, 0, tg.units, G, nullptr);
    return cudaGetLastError();
}

template <int MX, int PB>
cudaError_t launch_mx_pb(const BpLaunch &L, bool checked, size_t smem, cudaStream_t s) {
    // two CTAs per SM (96 registers) by default; one CTA per SM (up to 200
    // registers) when the stage needs more shared memory than two CTAs get
    const bool one_cta = smem > 113u * 1024u;
    if (checked)
        return one_cta ? launch_kernels<MX, PB, true, 1>(L, smem, s) : launch_kernels<MX, PB, true, kCtasPerSm>(L, smem, s);
    return one_cta ? launch_kernels<MX, PB, false, 1>(L, smem, s) : launch_kernels<MX, PB, false, kCtasPerSm>(L, smem, s);
}

template <int PB, typename K>
int resident_of(K kern, size_t smem) {
    int dev = 0, sms = 0, occ = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kFwdThreads<PB>, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return occ * sms;
}

template <int MX, int PB>
int resident_mx_pb(size_t smem) {
    const bool one_cta = smem > 113u * 1024u;
    return one_cta ? resident_of<PB>(bp_mixed_kernel<MX, PB, false, 1, false>, smem)
                   : resident_of<PB>(bp_mixed_kernel<MX, PB, false, kCtasPerSm, false>, smem);
}

template <int MX, int PB, int MINB>
cudaError_t launch_batch_kernels(const BatchScene *scenes, int nscenes, long long units, long long tiles,
                                 size_t smem, int resident, const BpLaunch &L0, unsigned long long *done,
                                 bool per_tile, cudaStream_t s) {
    auto kern = bp_mixed_kernel<MX, PB, false, MINB, true>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    if (tiles < 1 || tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
    if (per_tile) {
        // one CTA per tile: no partial sums, scenes finish in order
        kern<<<static_cast<unsigned>(tiles), kFwdThreads<PB>, smem, s>>>(L0, scenes, nscenes, units, done, 1);
        return cudaGetLastError();
    }
    const long long G = resident < units ? resident : units;
    if (G < 1 || G > 0x7fffffffLL) return cudaErrorInvalidValue;
    kern<<<static_cast<unsigned>(G), kFwdThreads<PB>, smem, s>>>(L0, scenes, nscenes, units, done, 0);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    bp_sk_fixup_kernel<MX, PB, true>
        <<<dim3(static_cast<unsigned>(tiles), MX), kThreads, 0, s>>>(L0, scenes, nscenes, units, G, done);
    return cudaGetLastError();
}

template <int MX, int PB>
cudaError_t launch_batch_mx_pb(const BatchScene *scenes, int nscenes, long long units, long long tiles, size_t smem,
                               int resident, const BpLaunch &L0, unsigned long long *done, bool per_tile,
                               cudaStream_t s) {
    return smem > 113u * 1024u
               ? launch_batch_kernels<MX, PB, 1>(scenes, nscenes, units, tiles, smem, resident, L0, done, per_tile, s)
               : launch_batch_kernels<MX, PB, 2>(scenes, nscenes, units, tiles, smem, resident, L0, done, per_tile,
                                                 s);
}

template <int MX, int PB>
int batch_resident_mx_pb(size_t smem) {
    return smem > 113u * 1024u ? resident_of<PB>(bp_mixed_kernel<MX, PB, false, 1, true>, smem)
                               : resident_of<PB>(bp_mixed_kernel<MX, PB, false, 2, true>, smem);
}

}  // namespace

size_t bp_mixed_smem_bytes(const TileConfig &tc, int wsize) { return smem_bytes_of(tc.pb, wsize); }

int bp_mixed_resident(const TileConfig &tc, size_t smem) {
#define SARBP_MIXED_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_) return resident_mx_pb<MX_, PB_>(smem);
    SARBP_MIXED_CASE(8, 8)
    SARBP_MIXED_CASE(8, 4)
    SARBP_MIXED_CASE(4, 16)
    SARBP_MIXED_CASE(4, 8)
    SARBP_MIXED_CASE(4, 4)
    SARBP_MIXED_CASE(4, 2)
    SARBP_MIXED_CASE(4, 1)
    SARBP_MIXED_CASE(2, 16)
    SARBP_MIXED_CASE(2, 8)
    SARBP_MIXED_CASE(2, 4)
    SARBP_MIXED_CASE(2, 2)
    SARBP_MIXED_CASE(2, 1)
    SARBP_MIXED_CASE(1, 16)
    SARBP_MIXED_CASE(1, 8)
    SARBP_MIXED_CASE(1, 4)
    SARBP_MIXED_CASE(1, 2)
    SARBP_MIXED_CASE(1, 1)
#undef SARBP_MIXED_CASE
    return 0;
}

// Tile shapes instantiated for batches; the batch autotuner times these.
const TileConfig bp_batch_tiles[] = {{8, 8}, {8, 4}, {4, 8}, {4, 4}, {2, 8}, {2, 4}, {1, 8}, {1, 4}};
const int bp_batch_tile_count = static_cast<int>(sizeof(bp_batch_tiles) / sizeof(bp_batch_tiles[0]));

cudaError_t launch_bp_mixed_batch(const BatchScene *scenes, int nscenes, long long units, long long tiles,
                                  const TileConfig &tc, size_t smem, int resident, void *partial,
                                  unsigned long long *done, cudaStream_t s, int max_wsize, bool per_tile,
                                  void *records) {
    BpLaunch L0{};
    L0.wsize = max_wsize;
    L0.sk_partial = partial;
    L0.geo_tab = records;  // non-null: every scene's table slot has its record rows
#define SARBP_BATCH_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_)  \
        return launch_batch_mx_pb<MX_, PB_>(scenes, nscenes, units, tiles, smem, resident, L0, done, per_tile, s);
    SARBP_BATCH_CASE(8, 8)
    SARBP_BATCH_CASE(8, 4)
    SARBP_BATCH_CASE(4, 8)
    SARBP_BATCH_CASE(4, 4)
    SARBP_BATCH_CASE(2, 8)
    SARBP_BATCH_CASE(2, 4)
    SARBP_BATCH_CASE(1, 8)
    SARBP_BATCH_CASE(1, 4)
#undef SARBP_BATCH_CASE
    return cudaErrorInvalidValue;
}

int bp_mixed_batch_resident(const TileConfig &tc, size_t smem) {
#define SARBP_BATCH_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_) return batch_resident_mx_pb<MX_, PB_>(smem);
    SARBP_BATCH_CASE(8, 8)
    SARBP_BATCH_CASE(8, 4)
    SARBP_BATCH_CASE(4, 8)
    SARBP_BATCH_CASE(4, 4)
    SARBP_BATCH_CASE(2, 8)
    SARBP_BATCH_CASE(2, 4)
    SARBP_BATCH_CASE(1, 8)
    SARBP_BATCH_CASE(1, 4)
#undef SARBP_BATCH_CASE
    return 0;
}

cudaError_t launch_bp_mixed(const BpLaunch &L, const TileConfig &tc, bool checked, size_t smem, cudaStream_t s) {
#define SARBP_MIXED_CASE(MX_, PB_) \
    if (tc.mx == MX_ && tc.pb == PB_) return launch_mx_pb<MX_, PB_>(L, checked, smem, s);
    SARBP_MIXED_CASE(8, 8)
    SARBP_MIXED_CASE(8, 4)
    SARBP_MIXED_CASE(4, 16)
    SARBP_MIXED_CASE(4, 8)
    SARBP_MIXED_CASE(4, 4)
    SARBP_MIXED_CASE(4, 2)
    SARBP_MIXED_CASE(4, 1)
    SARBP_MIXED_CASE(2, 16)
    SARBP_MIXED_CASE(2, 8)
    SARBP_MIXED_CASE(2, 4)
    SARBP_MIXED_CASE(2, 2)
    SARBP_MIXED_CASE(2, 1)
    SARBP_MIXED_CASE(1, 16)
    SARBP_MIXED_CASE(1, 8)
    SARBP_MIXED_CASE(1, 4)
    SARBP_MIXED_CASE(1, 2)
    SARBP_MIXED_CASE(1, 1)
#undef SARBP_MIXED_CASE
    return cudaErrorInvalidValue;
}

}  // namespace sarbp
