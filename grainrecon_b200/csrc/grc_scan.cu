// grc_scan.cu -- projection-window trial scan, one trial per warp at a time.
//
// The same work as the sweep of grc_score.cu (forward_comp.m:18-90 for every trial of a round,
// every CTA walking the projections window by window so the map pixels being read stay in L2),
// organised around the warp instead of the CTA:
//   * a warp takes one trial (slot) of the window at a time and first writes that trial's FP32
//     Gw table and window thresholds for all reflections into its own shared-memory table;
//   * 32 projections at a time, each lane tests its reflections against the window, two projections
//     per packed FP32 instruction, and shifts the sign of the test into a bit mask (3 instructions
//     per pair, no ballot, no store); the set bits of a mask are runs of consecutive projections, and
//     one entry and one mark bit per run number the passing pairs, so that a batch of 32 finds its
//     pairs by a population count;
//   * batches go through the FP32 landing chain with its FP64 band (landing_row3 / landing_exact).
//     Lanes hold consecutive projections of a few reflections: their omega rows are consecutive
//     16-byte words in shared memory, their Gw words broadcasts;
//   * a selected pixel's map word is read when its batch is evaluated and counted some batches
//     later: two, in registers, for the bit mask; four, through cp.async, for the 8-bit codes, of
//     which a third miss L2;
//   * ambiguous items keep their trial in the warp's FP64 queue, drained outside the batch loop: a
//     call inside it cost 12 spill reloads per batch.
// What bounds it (FCC Al 2048^2 x 361, completeness): issue (66 % of slots, 25.3 k warp instructions
// per trial) and the shared-memory / L1 pipe (79 % of its wavefronts: 12 of a batch's 31 are its
// rows, 13 its gather) together.  64 seeds x 32,768 orientations: one ballot and one queue store per
// (projection, slot) and 64-byte rows (40.6 k instructions) 97.4 ms; bit masks and runs 73.2; the
// test two projections per instruction 70.0; landings in packed pairs, separate tables 68.8.
// Four columns (16 seeds), before the last two: 32.6 (CTA sweep) -> 25.6 ms.  Numbering the pairs
// projection-major instead (masks transposed across the warp, better shared rows) ran 82.0 ms: its
// Gw words conflict.  Four CTAs per SM (64 registers) ran 114 ms.  Rows of 10 numbers (kx and L2
// from ky and kz) ran 71.2: two wavefronts fewer do not pay for six instructions more.
// Windows: up to 128 projections within the limits of shared memory and L2 (launch_scan_t).
// The decisions are those of the sweep and of the oracle: same prefilter margins, same FP32
// algebra and band, same FP64 path.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "grc_chain.cuh"
#include "grc_internal.h"

#ifndef GRC_SCAN_BLOCKS
#define GRC_SCAN_BLOCKS 3
#endif

namespace grc {
namespace {

constexpr int kScanSlots = 96;      // most trials a CTA holds in one round
constexpr int kScanSlotsBulk = 64;  // tile of multi-round work and of explicit voxel lists
constexpr int kScanWinMin = 8;
constexpr int kHistWords = 128;     // 256 u16 bins per slot, two per word
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ int64_t scan_voxel_of(const Work &w, int64_t t) {
    if (w.trial_voxel) return (int64_t)w.trial_voxel[t];
    if (w.diag) return t;
    return t / w.n_or;
}

__device__ __forceinline__ int64_t scan_orient_of(const Work &w, int64_t t, int64_t v) {
    if (w.trial_orient) return (int64_t)w.trial_orient[t];
    return w.diag ? t : (t - v * w.n_or);
}

// Omega row of one (voxel, projection) as four float4 planes of WIN projections each, so that lanes
// on consecutive projections read consecutive 16-byte words: {kx, L2, ky, kz}, {cN, num, ay, az},
// {u0, v0, c, s} for the landing, and k_w for the window test as planes of WIN floats wx, wy, wz.
constexpr int kRowParts = 4;
// Landings of a (trial, window) awaiting their batch: fewer than 64 left over plus one run of up to
// 32 projections per lane, one mark bit each, in rings.
constexpr int kMarkRing = 64;  // words of 32 positions
constexpr int kRunRing = 128;
constexpr int kStages = 4;     // full mode: batches whose map words are in flight

struct ScanSmem {
    float4 *rows;      // [rows_cap][kRowParts][nwin] omega rows of the window
    float4 *hk;        // [nhkl] h as float
    uint32_t *hist;    // full mode: [slots * kHistWords]; completeness mode: [slots] packed counters
    float *subf;       // [slots * 12]
    double *subd;      // [slots * 9]
    int *vloc;         // [slots]
    int64_t *vglob;    // [slots]
    int64_t *vlist;    // [slots]
    unsigned char *warps;  // [kWarps] blocks of warp_block_bytes(nhkl)
};

// A warp's own block: rings, queues and the tables of its trial at fixed offsets from one base.
constexpr int kExactCap = 128;                              // ambiguous items awaiting the FP64 path
constexpr int kOffRuns = kMarkRing * 4;                     // [kRunRing]
constexpr int kOffExact = kOffRuns + kRunRing * 4;          // [kExactCap]
constexpr int kOffTable = kOffExact + kExactCap * 4;        // [nhkl] {Gw x, y, z, 1/|G|}, [nhkl] certain {lo, hi}, [nhkl] {middle, half^2}
// ... and in full mode after it [kStages * 32] map words of the batches in flight
__host__ __device__ inline size_t warp_block_bytes(int mode, int nhkl) {
    return kOffTable + sizeof(float4) * 2 * nhkl + (mode == kScanFull ? sizeof(uint32_t) * kStages * 32 : 0);
}

constexpr int kScanParts = 9;
__host__ __device__ inline size_t scan_smem_layout(int mode, int nhkl, int rows_cap, int slots, int nwin,
                                                   size_t *offs) {
    size_t o = 0, i = 0;
    auto put = [&](size_t bytes) {
        o = (o + 15) & ~size_t(15);
        offs[i++] = o;
        o += bytes;
    };
    put(sizeof(float4) * kRowParts * rows_cap * nwin);
    put(sizeof(float4) * nhkl);
    put(sizeof(uint32_t) * slots * (mode == kScanFull ? kHistWords : 1));
    put(sizeof(float) * slots * 12);
    put(sizeof(double) * slots * 9);
    put(sizeof(int) * slots);
    put(sizeof(int64_t) * slots);
    put(sizeof(int64_t) * slots);
    put(kWarps * warp_block_bytes(mode, nhkl));
    return (o + 15) & ~size_t(15);
}

__device__ __forceinline__ void cp_async4(uint32_t *dst, const uint32_t *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ ScanSmem scan_carve(unsigned char *base, int mode, int nhkl, int rows_cap, int slots,
                                               int nwin) {
    size_t offs[kScanParts];
    scan_smem_layout(mode, nhkl, rows_cap, slots, nwin, offs);
    ScanSmem m;
    m.rows = (float4 *)(base + offs[0]);
    m.hk = (float4 *)(base + offs[1]);
    m.hist = (uint32_t *)(base + offs[2]);
    m.subf = (float *)(base + offs[3]);
    m.subd = (double *)(base + offs[4]);
    m.vloc = (int *)(base + offs[5]);
    m.vglob = (int64_t *)(base + offs[6]);
    m.vlist = (int64_t *)(base + offs[7]);
    m.warps = base + offs[8];
    return m;
}

template <int MODE, int HPL, int WIN>
__global__ void __launch_bounds__(kThreads, GRC_SCAN_BLOCKS)
    scan_kernel(Geo g, ScoreBufs b, Work w, int64_t round_base, int64_t n_trials, int rows_cap, int slots,
                int parts_log2) {
    const int64_t cta_base = round_base + (int64_t)blockIdx.x * slots;
    if (cta_base >= n_trials) return;
    const int nslot = (int)min((int64_t)slots, n_trials - cta_base);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const ScanSmem sm = scan_carve(smem_raw, MODE, g.nhkl, rows_cap, slots, WIN);
    __shared__ int s_nv, s_next;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned lt = (1u << lane) - 1u, le = lt | (1u << lane);
    unsigned char *wb = sm.warps + warp * warp_block_bytes(MODE, g.nhkl);
    uint32_t *marks = (uint32_t *)wb, *runs = (uint32_t *)(wb + kOffRuns), *fq = (uint32_t *)(wb + kOffExact);
    float4 *tab = (float4 *)(wb + kOffTable);
    float2 *sure = (float2 *)(tab + g.nhkl), *span = sure + g.nhkl;
    uint32_t *stage = (uint32_t *)(span + g.nhkl) + lane;  // full mode

    // ---- set-up: per-slot S*U*B, voxels, zeroed counters
    if (tid < nslot) {
        const int64_t t = cta_base + tid;
        const int64_t v = scan_voxel_of(w, t);
        const int64_t o = scan_orient_of(w, t, v);
        double SUB[9];
        sub_matrix(g, b.U + 9 * o, SUB);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            sm.subd[9 * tid + i] = SUB[i];
            sm.subf[12 * tid + i] = (float)SUB[i];
        }
        sm.vglob[tid] = v;
        sm.vloc[tid] = in_reach(g, b.vpos + 3 * v) ? 0 : 1;
    }
    for (int i = tid; i < slots * (MODE == kScanFull ? kHistWords : 1); i += kThreads) sm.hist[i] = 0;
    for (int i = tid; i < g.nhkl; i += kThreads)
        sm.hk[i] = make_float4((float)b.hkl[3 * i], (float)b.hkl[3 * i + 1], (float)b.hkl[3 * i + 2], 0.f);
    for (int i = lane; i < kMarkRing; i += 32) marks[i] = 0;
    __syncthreads();
    if (tid == 0) {
        int nv = 0;
        for (int s = 0; s < nslot; ++s) {
            // ~voxel: out of reach of the FP32 landings
            if (s == 0 || sm.vglob[s] != sm.vglob[s - 1]) sm.vlist[nv++] = sm.vloc[s] ? ~sm.vglob[s] : sm.vglob[s];
            sm.vloc[s] = nv - 1;
        }
        s_nv = nv;
    }
    __syncthreads();
    const int nv = s_nv;
    const int64_t pw = b.plane_words;
    const uint32_t pw32 = (uint32_t)pw;

    for (int w0 = 0; w0 < g.nrot; w0 += WIN) {
        const int nw = min(WIN, g.nrot - w0);
        // ---- omega rows of this window for every voxel of the round
        for (int i = tid; i < nv * nw; i += kThreads) {
            const int vl = i / nw, wl = i - vl * nw;
            const int64_t v = sm.vlist[vl];
            const OmegaRow d = omega_row(g, b.rot_cs[w0 + wl], b.vpos + 3 * (v < 0 ? ~v : v));
            const RowF r = row_f32(g, d, v >= 0);
            float4 *o = sm.rows + vl * kRowParts * WIN + wl;
            o[0] = make_float4((float)d.kx, r.L2, r.ky, r.kz);
            o[WIN] = make_float4(r.cN, r.num, r.ay, r.az);
            o[2 * WIN] = make_float4(r.u0, r.v0, r.c, r.s);
            float *kw = (float *)(sm.rows + (vl * kRowParts + 3) * WIN) + wl;
            kw[0] = r.wx;
            kw[WIN] = r.wy;
            kw[2 * WIN] = r.wz;
        }
        if (tid == 0) s_next = 0;
        __syncthreads();

        // the window's 8-bit codes as 32-bit words; its first pixel may start inside a word, at byte wmis
        const uint8_t *wcodes = MODE == kScanFull ? b.codes8 + (int64_t)w0 * g.plane : nullptr;
        const uint32_t wmis = (uint32_t)((uintptr_t)wcodes & 3u);
        const uint32_t *wwords = (const uint32_t *)(wcodes - wmis);
        const uint32_t *wbits = MODE == kScanComp ? b.bits + (int64_t)w0 * pw : nullptr;
        // Full mode: the map word of a selected pixel is copied to shared memory when its batch is
        // evaluated and its code counted kStages batches later, whichever trials those belong
        // to, so the gather's latency (a third of the codes miss L2) overlaps their landings.  A byte
        // per batch in flight: 0x80 | bit of the code in its word, or 0; and the batch's trial.
        uint32_t pend = 0, pend_slot = 0;
        int n_batch = 0;
        auto count_oldest = [&]() {
            if (!(pend & 0x80000000u)) return;
            const uint32_t code = (stage[(n_batch & (kStages - 1)) * 32] >> ((pend >> 24) & 31u)) & 255u;
            atomicAdd(&sm.hist[(pend_slot >> 24) * kHistWords + (code >> 1)], 1u << ((code & 1u) * 16));
        };
        int fn = 0;  // ambiguous items of this warp (any of its trials), drained at the window end

        // FP64 path of one ambiguous item: counted at once (shared atomics; these items are rare)
        auto exact = [&](uint32_t item, bool valid) {
            const int s2 = (int)(item >> 16), wl = (int)((item >> 8) & 255u), ih = (int)(item & 255u);
            if (!valid) return;
            const int64_t r64 =
                landing_exact(b.geo, b.rot_cs, b.vpos + 3 * sm.vglob[s2], b.hkl, sm.subd + 9 * s2, w0 + wl, ih);
            if (r64 < 0) return;
            if (MODE == kScanComp) {
                const int64_t iw = w0 + wl, ip = r64 - iw * g.plane;
                const uint32_t word = __ldg(b.bits + iw * pw + (ip >> 5));
                atomicAdd(&sm.hist[s2], 1u + (((word >> (ip & 31)) & 1u) << 16));
            } else {
                const uint32_t code = __ldg(b.codes8 + r64);
                atomicAdd(&sm.hist[s2 * kHistWords + (code >> 1)], 1u << ((code & 1u) * 16));
            }
        };
        auto drain_exact = [&](bool all) {
            while (fn >= 32 || (all && fn > 0)) {
                const int take = fn >= 32 ? 32 : fn;
                fn -= take;
                const bool v2 = lane < take;
                const uint32_t it2 = v2 ? fq[fn + lane] : 0u;
                __syncwarp();
                exact(it2, v2);
                __syncwarp();
            }
        };

        // A slot, or one of the parts its window is cut into where a CTA holds few trials, is handed
        // out at a time, so the warps of a CTA reach the end-of-window barrier together however
        // unevenly the selected reflections fall on the slots
        const int part = WIN >> parts_log2;
        for (;;) {
            int s = 0;
            if (lane == 0) s = atomicAdd(&s_next, 1);
            s = __shfl_sync(kAll, s, 0);
            const int k0 = (s & ((1 << parts_log2) - 1)) * part, k1 = min(nw, k0 + part);
            s >>= parts_log2;
            if (s >= nslot) break;
            if (k0 >= k1) continue;
            // ---- the trial's Gw and window table
            const float *sf = sm.subf + 12 * s;
#pragma unroll
            for (int j = 0; j < HPL; ++j) {
                const int ih = lane + 32 * j;
                if (ih < g.nhkl) {
                    const float4 gv = gw_of(sf, sm.hk[ih]);
                    const float4 wv = window_f(g, gv);
                    tab[ih] = gv;
                    sure[ih] = make_float2(wv.z, wv.w);
                    span[ih] = make_float2(0.5f * (wv.x + wv.y),
                                           wv.y > wv.x ? 0.25f * (wv.y - wv.x) * (wv.y - wv.x) : -1.0f);
                }
            }
            __syncwarp();
            const float4 *vr = sm.rows + sm.vloc[s] * kRowParts * WIN;
            // completeness mode: the lane's share of this trial's counts in this window, packed as
            // the shared counter (Nr_simu low, Nr_intersect high 16 bits) and summed over the warp
            // once per trial and window
            uint32_t cnt = 0;
            // Completeness mode: a selected pixel's map word is read when its batch is evaluated and
            // counted after the next two batches have been computed, so the gather's latency overlaps
            // the landing arithmetic (pend_bit: the pixel's bit in the word)
            int pend_bit[2] = {0, 0};
            uint32_t pend_word[2] = {0, 0};
            // Positions 0, 1, 2, ... number the trial's (reflection, projection) pairs that pass the
            // window test, one run of consecutive projections of a reflection after the other.  A
            // mark bit says where a run starts, and its entry holds the reflection and the projection
            // minus the position, so a lane finds its pair from a population count.
            int end = 0, done = 0;      // positions known / evaluated (done: a multiple of 64)
            int n_run = 0, r_run = -1;  // runs known / index of the run that position `done` lies in
            // the pair at position `pos`; h: the pending pixel it takes the place of (constant)
            auto one = [&](int h, uint32_t e, int pos, bool valid) {
                const int ih = (int)(e & 255u), wl = ((int)e >> 8) + pos;
                int ip = -1;
                if (valid) {
                    const float4 gv = tab[ih];
                    const float2 wv = sure[ih];
                    const float4 *o = vr + wl;
                    ip = landing_row3(g, o[0], o[WIN], o[2 * WIN], gv, wv.x, wv.y);
                }
#ifdef GRC_AUDIT
                // audit build: every certain FP32 decision is re-decided by the FP64 path
                if (valid && ip != -2) {
                    const int64_t r64 = landing_exact(b.geo, b.rot_cs, b.vpos + 3 * sm.vglob[s], b.hkl,
                                                      sm.subd + 9 * s, w0 + wl, ih);
                    atomicAdd((unsigned long long *)(b.work_counter + 6), 1ull);
                    if ((r64 >= 0 ? (int)(r64 - (int64_t)(w0 + wl) * g.plane) : -1) != ip)
                        atomicAdd(b.work_counter + 5, 1);
                }
#endif
                const unsigned m = __ballot_sync(kAll, ip == -2);
                // offsets within the window fit 32 bits: WIN * plane < 2^31 for the codes
                // (launch_scan_t) and 8 * plane < 2^31 for the words (scan_round_trials)
                if constexpr (MODE == kScanComp) {
                    uint32_t word = 0;
                    if (ip >= 0) {
                        word = __ldg(wbits + ((uint32_t)wl * pw32 + ((uint32_t)ip >> 5)));
                        cnt += 1u;
                    }
                    cnt += ((pend_word[h] >> pend_bit[h]) & 1u) << 16;
                    pend_bit[h] = ip & 31;
                    pend_word[h] = word;
                } else {
                    cp_async_wait<kStages - 1>();
                    count_oldest();
                    uint32_t info = 0;
                    if (ip >= 0) {
                        const uint32_t off = (uint32_t)wl * (uint32_t)g.plane + (uint32_t)ip + wmis;
                        cp_async4(stage + (n_batch & (kStages - 1)) * 32, wwords + (off >> 2));
                        info = 0x80u | (off & 3u) * 8u;
                    }
                    cp_async_commit();
                    pend = (pend << 8) | info;
                    pend_slot = (pend_slot << 8) | (uint32_t)s;
                    ++n_batch;
                }
                if (m) {  // ambiguous items (rare) join the FP64 queue
                    if (ip == -2) fq[fn + __popc(m & lt)] = ((uint32_t)s << 16) | ((uint32_t)wl << 8) | (uint32_t)ih;
                    fn += __popc(m);
                }
            };
            auto two_batches = [&](bool full) {
                uint2 *mw = (uint2 *)(marks + ((done >> 5) & (kMarkRing - 1)));
                const uint2 mm = *mw;
                const int r1 = r_run + __popc(mm.x);
                const uint32_t e0 = runs[(r_run + __popc(mm.x & le)) & (kRunRing - 1)];
                const uint32_t e1 = runs[(r1 + __popc(mm.y & le)) & (kRunRing - 1)];
                r_run = r1 + __popc(mm.y);
                one(0, e0, done + lane, full || done + lane < end);
                if (full || done + 32 < end) one(1, e1, done + 32 + lane, full || done + 32 + lane < end);
                if (lane == 0) *mw = make_uint2(0, 0);  // every lane has read it: a ballot lies between
                done += 64;
            };
            // ---- 32 projections at a time: the window test of every reflection as a bit mask per
            // lane and slot, its runs of set bits numbered, full batches of 32 evaluated
            constexpr int kSpan = WIN < 32 ? WIN : 32;
            uint32_t rem[HPL];
            bool tested = false;  // rem holds what is left of the span at k
            int k = k0 & ~(kSpan - 1);
            for (;;) {
                // leaves this loop when the FP64 queue has no room for a batch, and comes back
                while (k < k1) {
                    if (!tested) {
                        tested = true;
                        uint64_t gx[HPL], gy[HPL], gz[HPL], mid[HPL], nh2[HPL];
#pragma unroll
                        for (int j = 0; j < HPL; ++j) {
                            const int ih = lane + 32 * j;
                            const bool real = ih < g.nhkl;
                            const float4 gv = tab[real ? ih : 0];
                            const float2 wv = span[real ? ih : 0];
                            gx[j] = pack2(gv.x, gv.x);
                            gy[j] = pack2(gv.y, gv.y);
                            gz[j] = pack2(gv.z, gv.z);
                            mid[j] = pack2(wv.x, wv.x);
                            const float nh = real ? -wv.y : 1.0f;
                            nh2[j] = pack2(nh, nh);
                            rem[j] = 0;
                        }
                        const float *kw = (const float *)(vr + 3 * WIN) + k;
#pragma unroll 4
                        for (int p = kSpan - 4; p >= 0; p -= 4) {
                            const ulonglong2 qx = *(const ulonglong2 *)(kw + p);
                            const ulonglong2 qy = *(const ulonglong2 *)(kw + WIN + p);
                            const ulonglong2 qz = *(const ulonglong2 *)(kw + 2 * WIN + p);
#pragma unroll
                            for (int j = 0; j < HPL; ++j) {
                                // (t - middle)^2 - half^2 is negative inside the window, t = -(k_w . Gw):
                                // the sign bits of two projections at a time join the mask from below
                                uint64_t d = fma2(qx.y, gx[j], fma2(qy.y, gy[j], fma2(qz.y, gz[j], mid[j])));
                                d = fma2(d, d, nh2[j]);
                                rem[j] = __funnelshift_l((uint32_t)(d >> 32), rem[j], 1);
                                rem[j] = __funnelshift_l((uint32_t)d, rem[j], 1);
                                d = fma2(qx.x, gx[j], fma2(qy.x, gy[j], fma2(qz.x, gz[j], mid[j])));
                                d = fma2(d, d, nh2[j]);
                                rem[j] = __funnelshift_l((uint32_t)(d >> 32), rem[j], 1);
                                rem[j] = __funnelshift_l((uint32_t)d, rem[j], 1);
                            }
                        }
                        uint32_t live = k1 - k < 32 ? (1u << (k1 - k)) - 1u : kAll;
                        if (k < k0) live &= kAll << (k0 - k);
#pragma unroll
                        for (int j = 0; j < HPL; ++j) rem[j] &= live;
                    }
                    bool spent = false;
                    for (;;) {
                        while (end - done >= 64 && fn <= kExactCap - 64) two_batches(true);
                        if (end - done >= 64) break;
                        // one run per lane: the first of its first slot that has any left
                        uint32_t x = 0;
                        int js = 0;
#pragma unroll
                        for (int j = HPL - 1; j >= 0; --j)
                            if (rem[j]) x = rem[j], js = j;
                        const unsigned any = __ballot_sync(kAll, x != 0);
                        if (!any) {
                            spent = true;
                            break;
                        }
                        const uint32_t low = x & (0u - x), rest = x & (x + low);
                        const int len = __popc(x ^ rest);
#pragma unroll
                        for (int j = 0; j < HPL; ++j)
                            if (j == js) rem[j] = rest;
                        int incl = len;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int y = __shfl_up_sync(kAll, incl, o);
                            if (lane >= o) incl += y;
                        }
                        if (x) {
                            const int pos = end + incl - len, first = k + 31 - __clz(low);
                            runs[(n_run + __popc(any & lt)) & (kRunRing - 1)] =
                                ((uint32_t)(first - pos) << 8) | (uint32_t)(lane + 32 * js);
                            atomicOr(&marks[(pos >> 5) & (kMarkRing - 1)], 1u << (pos & 31));
                        }
                        end += __shfl_sync(kAll, incl, 31);
                        n_run += __popc(any);
                        __syncwarp();
                    }
                    if (!spent) break;
                    tested = false;
                    k += kSpan;
                }
                if (k >= k1 && fn <= kExactCap - 64) break;
                __syncwarp();
                drain_exact(false);
            }
            if (end > done) two_batches(false);  // the last ones: every batch holds one trial
            __syncwarp();
            if (MODE == kScanComp) {
#pragma unroll
                for (int h = 0; h < 2; ++h) cnt += ((pend_word[h] >> pend_bit[h]) & 1u) << 16;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(kAll, cnt, o);
                if (lane == 0) atomicAdd(&sm.hist[s], cnt);
            }
        }
        if (MODE == kScanFull) {
            cp_async_wait<0>();
#pragma unroll
            for (int i = 0; i < kStages; ++i) {  // the last batches, oldest first
                count_oldest();
                pend <<= 8;
                pend_slot <<= 8;
                ++n_batch;
            }
        }
        drain_exact(true);
        __syncthreads();  // rows are rebuilt for the next window
    }

    // ---- finalize
    if constexpr (MODE == kScanFull) {
        for (int s = warp; s < nslot; s += kWarps) hist8_finish(g, b, sm.hist + s * kHistWords, cta_base + s);
        if (b.group_key) {
            __syncthreads();
            for (int base = warp * 32; base < nslot; base += kWarps * 32) {
                const bool in = base + lane < nslot;
                const TrialRes r = in ? b.res[cta_base + base + lane] : TrialRes{};
                fold_group_key(b, in, cta_base + base + lane, r.simu, r.inter);
            }
        }
    } else {
        for (int base = warp * 32; base < nslot; base += kWarps * 32) {
            const int s = base + lane;
            const bool in = s < nslot;
            const int64_t t = cta_base + s;
            int simu = 0, inter = 0;
            if (in) {
                const uint32_t c = sm.hist[s];
                simu = (int)(c & 0xffffu);
                inter = (int)(c >> 16);
                TrialRes r;
                r.simu = simu;
                r.inter = inter;
                r.median = CUDART_NAN;  // not computed in this mode
                b.res[t] = r;
            }
            if (b.group_key) fold_group_key(b, in, t, simu, inter);
        }
    }
}

// Shared memory that the CTAs of an SM may take together (1 KB reserved for each included).  Above
// some 196 KB the SM is left with 28 KB of L1, and the misses in flight each need an L1 line: full-output
// scans ran 12.9 ms with three CTAs of 24 to 40 trials and 19.4 ms with 48 to 64 (FCC Al 2048^2 x
// 361, 8 seeds x 32,768 orientations), 5.43 against 6.96 ms on BCC Fe 1024^2 x 181.
constexpr size_t kSmSmemBudget = 192 * 1024;

template <int MODE, int HPL>
cudaError_t launch_scan_t(const Geo &g, const ScoreBufs &b, const Work &w, int64_t n_trials, int num_sms,
                          cudaStream_t s, cudaEvent_t ev0, cudaEvent_t ev1, int *launches, int max_slots) {
    // An implicit seeding list meets at most two voxels per tile; explicit lists keep one row set per
    // voxel-run start of their aligned 32-trial blocks, or per trial when that bound is unknown.
    const bool explicit_voxels = w.trial_voxel || w.diag || w.n_or <= 0;
    const bool caller_tile = max_slots >= 1 && max_slots <= kScanSlots;
    if (!caller_tile) max_slots = kScanSlotsBulk;
    auto rows_for = [&](int sl) {
        int rc = (int)(w.n_or >= sl ? 2 : (w.n_or > 0 ? sl / w.n_or + 2 : sl));
        if (explicit_voxels) rc = w.starts_per_32 > 0 ? 1 + ((sl + 31) / 32 + 1) * w.starts_per_32 : sl;
        return rc > sl ? sl : rc;
    };
    size_t offs[kScanParts];
    using ScanFn = void (*)(Geo, ScoreBufs, Work, int64_t, int64_t, int, int, int);
    auto window_kernel = [](int win) -> ScanFn {
        if (win == 128) return scan_kernel<MODE, HPL, 128>;
        if (win == 64) return scan_kernel<MODE, HPL, 64>;
        if (win == 32) return scan_kernel<MODE, HPL, 32>;
        return win == 16 ? (ScanFn)scan_kernel<MODE, HPL, 16> : (ScanFn)scan_kernel<MODE, HPL, kScanWinMin>;
    };
    // The window's map stays within 3/4 of L2 (Al 2048^2 on 126 MB, bit mask: 128 projections = 67 MB,
    // fastest; 256 = 134 MB ran 30% slower), or the call touches so few of its pixels that it would
    // meet few of them again: n_trials * nhkl * window <= 4 * plane (one voxel, full output on 2048^2:
    // 64 projections against 32 0.339 and 0.348 ms for 4,096 orientations, 0.567 and 0.507 for 9,218).
    int64_t l2_budget = 0;
    int dev = 0, l2 = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) == cudaSuccess)
        l2_budget = (int64_t)l2 * 3 / 4;
    else
        cudaGetLastError();  // no L2 size: windows of at most 32 projections
    const double reads = (double)n_trials * g.nhkl;
    // Widest window first: up to 128 projections, 64 for explicit lists of completeness calls (the
    // refine's grids).  Of each, the most trials per CTA (at most the tile) that keep GRC_SCAN_BLOCKS
    // CTAs within the budget.  A full-output window above 32 projections is for calls of one round
    // (2,000 voxels with a trial each, Al 2048^2 x 361: 0.213 ms at 64, 0.225 at 32; 9,171: 0.70 and
    // 0.68) or, at 64, for scans whose window's codes stay in L2 (16 voxels x 9,218 orientations, Fe
    // 1024^2 x 181: 5.25 ms at 32, 5.00 at 64); a tile below one trial per warp, two in completeness mode, goes on to the next window
    // (30,000 voxels with 1-64 candidates, full output: 11.6 ms at 32 projections and 13 trials, 12.4 at
    // 16 and 21).
    // A completeness call that a larger tile makes one round takes it.
    if (MODE == kScanComp && !caller_tile && !explicit_voxels &&
        n_trials <= (int64_t)GRC_SCAN_BLOCKS * num_sms * kScanSlots)
        max_slots = kScanSlots;
    int win = 0, tile = 0, ctas = GRC_SCAN_BLOCKS;
    for (; ctas >= 1 && !win; --ctas)
        for (int cand : {128, 64, 32, 16, kScanWinMin}) {
            const int64_t bytes = MODE == kScanComp ? cand * b.plane_words * 4 : cand * g.plane;
            const bool sparse = reads * cand <= 4.0 * (double)g.plane;
            if (cand > 32 && bytes > l2_budget && !sparse) continue;
            if (MODE == kScanComp && explicit_voxels && cand > 64 && !sparse) continue;
            if (MODE == kScanFull && cand > kScanWinMin && bytes > 2147483647LL) continue;
            int t = max_slots;
            while (t > 0 && ctas * (scan_smem_layout(MODE, g.nhkl, rows_for(t), t, cand, offs) + 1024) > kSmSmemBudget)
                --t;
            const bool one_round = (int64_t)t * ctas * num_sms >= n_trials;
            if (caller_tile ? t < max_slots : !one_round && t < (MODE == kScanComp ? 2 : 1) * kWarps) continue;
            if (MODE == kScanFull && cand > 32 && !one_round && (cand > 64 || bytes > l2_budget || t < 2 * kWarps))
                continue;
            win = cand;
            tile = t;
            break;
        }
    if (!win) {  // one CTA per SM, of what it can hold
        win = kScanWinMin;
        tile = caller_tile ? max_slots : 2 * kWarps;
    } else {
        ++ctas;
    }
    int per_sm = 0;
    size_t smem = scan_smem_layout(MODE, g.nhkl, rows_for(tile), tile, win, offs);
    cudaError_t e = occupancy_for((const void *)window_kernel(win), smem, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    if (win && per_sm > ctas && ctas >= 1) per_sm = ctas;
    const int64_t grid = (int64_t)per_sm * num_sms;
    // A trial per warp instead of one to two, over many rounds: the lists above 11.75 -> 11.38 ms; 30,000
    // voxels with 1-64 candidates on Fe 1024^2 x 181 9.16 -> 7.88, on 2048^2 x 91 5.03 -> 4.21; 100,000
    // trials of scattered voxels on seven geometries 0-16 % faster.  On Al a voxel per trial is 1-4 %
    // slower: 30,000 voxels grown 1.69 -> 1.71 ms (2048^2 x 361), 1.68 -> 1.75 (600 x 1900 x 361), 0.655
    // -> 0.673 (1537 x 1001 x 121; candidates there 4.25 -> 4.31).
    if (MODE == kScanFull && !caller_tile && tile > kWarps && tile < 2 * kWarps && n_trials > 3 * grid * kWarps)
        tile = kWarps;
    // rounds of equal size, so that the last is not a sliver
    const int64_t rounds = (n_trials + grid * tile - 1) / (grid * tile);
    int slots = (int)((n_trials + rounds * grid - 1) / (rounds * grid));
    if (slots < 1) slots = 1;
    const int rows_cap = rows_for(slots);
    smem = scan_smem_layout(MODE, g.nhkl, rows_cap, slots, win, offs);
    const ScanFn kern = window_kernel(win);
    e = allow_smem((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    const int64_t per_round = grid * slots;
    int parts_log2 = 0;
    // A window is cut into parts of 32 projections where a CTA holds fewer than two trials per warp,
    // and of 16 where those would not go round the warps (one voxel, 8 to 256 orientations: 97-125 us
    // whole, 86-99 at 32, 84-88 at 16).
    while ((win >> parts_log2) > 32 && slots < 2 * kWarps) ++parts_log2;
    if (win >= 32 && slots * (win >> 5) < kWarps) ++parts_log2;
    e = cudaMemsetAsync(b.work_counter, 0, 8 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    if (ev0) cudaEventRecord(ev0, s);
    for (int64_t base = 0; base < n_trials; base += per_round) {
        const int64_t left = (n_trials - base + slots - 1) / slots;
        const int gr = (int)(left < grid ? left : grid);
        kern<<<gr, kThreads, smem, s>>>(g, b, w, base, n_trials, rows_cap, slots, parts_log2);
        ++*launches;
    }
    if (ev1) cudaEventRecord(ev1, s);
    if (MODE == kScanFull) {
        e = launch_refine_list(g, b, w, num_sms, s);
        if (e != cudaSuccess) return e;
        ++*launches;
    }
    return cudaGetLastError();
}

template <typename CodeT>
__global__ void pack_bits_k(const CodeT *codes, int64_t plane, int64_t nrot, uint32_t n_hit, int64_t pw,
                            uint32_t *bits) {
    // one thread per bit of the padded layout; a warp covers one 32-bit word
    const int64_t per_plane = pw * 32, total = nrot * per_plane;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;  // a multiple of 32
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int64_t iw = i / per_plane, p = i - iw * per_plane;
        const bool hit = p < plane && (uint32_t)codes[iw * plane + p] < n_hit;
        const unsigned m = __ballot_sync(kAll, hit);
        if ((threadIdx.x & 31) == 0) bits[i >> 5] = m;
    }
}

// One warp per group: the first maximum of completeness over the group's trials.
__global__ void group_argmax_k(const TrialRes *res, int64_t n_trials, int64_t gsize, unsigned long long *keys) {
    const int lane = threadIdx.x & 31;
    const int64_t n_groups = (n_trials + gsize - 1) / gsize;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t grp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); grp < n_groups; grp += warps) {
        const int64_t t0 = grp * gsize, n = min(gsize, n_trials - t0);
        unsigned long long key = 0ull;
        for (int64_t i = lane; i < n; i += 32) {
            const TrialRes r = res[t0 + i];
            const unsigned long long k = group_key_of(r.simu, r.inter, i);
            key = k > key ? k : key;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = shfl_xor_u64(key, o);
            key = y > key ? y : key;
        }
        if (lane == 0) atomicMax(keys + grp, key);
    }
}

__global__ void group_decode_k(const unsigned long long *keys, int64_t n_groups, int32_t *best, float *best_c) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_groups; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long k = keys[i];
        const uint32_t hi = (uint32_t)(k >> 32), lo = (uint32_t)k;
        if (best) best[i] = (int32_t)(0xffffffffu - lo);
        if (best_c) best_c[i] = hi == 0u ? CUDART_NAN_F : __uint_as_float(hi - 1u);
    }
}

// Spot pixels of a packed mask back to bytes: mask[iw*plane + p] = bit p of projection iw.
__global__ void unpack_bits_k(const uint32_t *bits, int64_t plane, int64_t nrot, int64_t pw, uint8_t *mask) {
    const int64_t n = nrot * plane;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t iw = i / plane, p = i - iw * plane;
        mask[i] = (uint8_t)((bits[iw * pw + (p >> 5)] >> (p & 31)) & 1u);
    }
}

}  // namespace

cudaError_t launch_unpack_bits(const uint32_t *bits, int64_t plane, int64_t nrot, int64_t plane_words, uint8_t *mask,
                               cudaStream_t s) {
    const int64_t n = nrot * plane;
    if (n <= 0) return cudaSuccess;
    const int64_t want = (n + 255) / 256;
    unpack_bits_k<<<(int)(want < 65535 * 8 ? want : 65535 * 8), 256, 0, s>>>(bits, plane, nrot, plane_words, mask);
    return cudaGetLastError();
}

cudaError_t launch_group_argmax(const TrialRes *res, int64_t n_trials, int64_t gsize, unsigned long long *keys,
                                cudaStream_t s) {
    if (n_trials <= 0 || gsize <= 0) return cudaSuccess;
    const int64_t n_groups = (n_trials + gsize - 1) / gsize;
    const int64_t want = (n_groups + 7) / 8;
    const int blocks = (int)(want < 65535 * 4 ? want : 65535 * 4);
    group_argmax_k<<<blocks, 256, 0, s>>>(res, n_trials, gsize, keys);
    return cudaGetLastError();
}

cudaError_t launch_group_decode(const unsigned long long *keys, int64_t n_groups, int32_t *best, float *best_c,
                                cudaStream_t s) {
    if (n_groups <= 0) return cudaSuccess;
    const int64_t want = (n_groups + 255) / 256;
    const int blocks = (int)(want < 65535 ? want : 65535);
    group_decode_k<<<blocks, 256, 0, s>>>(keys, n_groups, best, best_c);
    return cudaGetLastError();
}

int64_t scan_round_trials(const Geo &g, int num_sms) {
    // 16-bit histogram bins (full mode) and 13-bit items; hit codes below the saturation code
    if (g.n_hit >= 255u || g.nhkl > 128 || (int64_t)g.nrot * g.nhkl > 65535 ||
        (int64_t)kScanWinMin * g.plane > 2147483647LL)
        return 0;
    return (int64_t)num_sms * GRC_SCAN_BLOCKS * kScanSlotsBulk;
}

cudaError_t launch_scan(const Geo &g, const ScoreBufs &b, const Work &w, int64_t n_trials, int num_sms, int mode,
                        cudaStream_t s, cudaEvent_t ev0, cudaEvent_t ev1, int *launches, int max_slots) {
    const int hpl = (g.nhkl + 31) / 32;
    if (mode == kScanComp && !b.bits) return cudaErrorInvalidValue;
#define GRC_DISPATCH(H)                                                                                    \
    if (hpl == H)                                                                                          \
        return mode == kScanComp                                                                           \
                   ? launch_scan_t<kScanComp, H>(g, b, w, n_trials, num_sms, s, ev0, ev1, launches, max_slots) \
                   : launch_scan_t<kScanFull, H>(g, b, w, n_trials, num_sms, s, ev0, ev1, launches, max_slots);
    GRC_DISPATCH(1)
    GRC_DISPATCH(2)
    GRC_DISPATCH(3)
    GRC_DISPATCH(4)
#undef GRC_DISPATCH
    return cudaErrorInvalidValue;
}

cudaError_t launch_pack_bits(const void *codes, int code_bytes, int64_t plane, int64_t nrot, uint32_t n_hit,
                             int64_t plane_words, uint32_t *bits, cudaStream_t s) {
    const int64_t total = nrot * plane_words * 32;
    const int threads = 256;
    const int64_t want = (total + threads - 1) / threads;
    const int blocks = (int)(want < 65535 * 8 ? want : 65535 * 8);
    if (code_bytes == 1)
        pack_bits_k<uint8_t><<<blocks, threads, 0, s>>>((const uint8_t *)codes, plane, nrot, n_hit, plane_words, bits);
    else if (code_bytes == 2)
        pack_bits_k<uint16_t><<<blocks, threads, 0, s>>>((const uint16_t *)codes, plane, nrot, n_hit, plane_words,
                                                          bits);
    else
        pack_bits_k<uint32_t><<<blocks, threads, 0, s>>>((const uint32_t *)codes, plane, nrot, n_hit, plane_words,
                                                          bits);
    return cudaGetLastError();
}

}  // namespace grc
