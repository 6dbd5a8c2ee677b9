// grc_aux.cu -- preparation, epilogue, distance-map coding and synthetic-data kernels.
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "grc_internal.h"

#include <algorithm>
#include <mutex>
#include <vector>

namespace grc {
namespace {

constexpr int kB = 256;

inline int blocks_for(int64_t n, int per = kB) {
    int64_t b = (n + per - 1) / per;
    if (b < 1) b = 1;
    if (b > (1 << 30)) b = 1 << 30;
    return (int)b;
}

// quaternion2U.m:3-28 (no renormalisation: q is used as given).
__global__ void quat_to_u_k(const float *q, int64_t n, double *U) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double q0 = q[4 * i], q1 = q[4 * i + 1], q2 = q[4 * i + 2], q3 = q[4 * i + 3];
        double *u = U + 9 * i;
        u[0] = 2 * (q0 * q0 + q1 * q1) - 1; u[1] = 2 * (q1 * q2 - q0 * q3); u[2] = 2 * (q1 * q3 + q0 * q2);
        u[3] = 2 * (q1 * q2 + q0 * q3); u[4] = 2 * (q0 * q0 + q2 * q2) - 1; u[5] = 2 * (q2 * q3 - q0 * q1);
        u[6] = 2 * (q1 * q3 - q0 * q2); u[7] = 2 * (q2 * q3 + q0 * q1); u[8] = 2 * (q0 * q0 + q3 * q3) - 1;
    }
}

// euler2u.m:5- with angles in degrees (converted as phi*pi/180).
__global__ void euler_to_u_k(const float *e, int64_t n, double *U) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double p1 = (double)e[3 * i] * CUDART_PI / 180, P = (double)e[3 * i + 1] * CUDART_PI / 180,
                     p2 = (double)e[3 * i + 2] * CUDART_PI / 180;
        const double c1 = cos(p1), s1 = sin(p1), c = cos(P), s = sin(P), c2 = cos(p2), s2 = sin(p2);
        double *u = U + 9 * i;
        u[0] = c1 * c2 - s1 * s2 * c; u[1] = -c1 * s2 - s1 * c2 * c; u[2] = s1 * s;
        u[3] = s1 * c2 + c1 * s2 * c; u[4] = -s1 * s2 + c1 * c2 * c; u[5] = -c1 * s;
        u[6] = s2 * s; u[7] = c2 * s; u[8] = c;
    }
}

__global__ void f_to_d_k(const float *a, int64_t n, double *out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (double)a[i];
}

// grow_indexed_region_parallel.m:70-74: pos = ((idx+RVP-1)-Dim/2)*VoxSize+Center, x,y negated for simap.
__global__ void pos_rows_k(const float *rows, int stride, int64_t n, const double *p1, double *vpos) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float *r = rows + (int64_t)stride * i;
        double p[3];
        for (int k = 0; k < 3; ++k) p[k] = (((double)r[k] + p1[k] - 1) - p1[8 + k] / 2) * p1[4] + p1[5 + k];
        if (p1[3] == 1.0) {
            p[0] = -p[0];
            p[1] = -p[1];
        }
        vpos[3 * i] = p[0];
        vpos[3 * i + 1] = p[1];
        vpos[3 * i + 2] = p[2];
    }
}

__global__ void epi_forward_k(const TrialRes *res, int64_t n, float *out, int median) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const TrialRes r = res[i];
        float4 o;
        o.x = (float)r.simu;
        o.y = (float)r.inter;
        o.z = (float)((double)r.inter / (double)r.simu);  // Nr_intersect/Nr_simu, NaN for 0/0
        o.w = median ? (float)r.median : CUDART_NAN_F;    // no median in completeness-only calls
        reinterpret_cast<float4 *>(out)[i] = o;
    }
}

// Accept rule of grow_indexed_region_parallel.m:78-88 without the Ninter clause.
__global__ void epi_grow_k(const TrialRes *res, const float *rows6, int64_t m, const double *p1, float *out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const TrialRes r = res[i];
        const float *row = rows6 + 6 * i;
        const double C = (double)r.inter / (double)r.simu;
        const double I = row[3], mask = row[4], dmed = row[5];
        const double lim = fmin(dmed, p1[13]);
        const bool cand = mask > 0 && C > I && r.median <= lim;
        const bool flag = cand && C >= p1[11] * (1 - p1[12]);
        float *w = out + 7 * i;
        w[0] = row[0];
        w[1] = row[1];
        w[2] = row[2];
        w[3] = (float)r.simu;
        w[4] = (float)r.inter;
        w[5] = (float)r.median;
        w[6] = flag ? 1.0f : 0.0f;
    }
}

__global__ void csr_counts_k(const float *rows5, int64_t m, int64_t *counts) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t first = (int64_t)rows5[5 * i + 3], last = (int64_t)rows5[5 * i + 4];
        counts[i] = last >= first ? last - first + 1 : 0;
    }
}

__global__ void csr_fill_k(const float *rows5, int64_t m, const int64_t *off, const float *id_neigb, int64_t n_neigb,
                           int64_t n_grain, longlong4 *items, int32_t *trial_orient, int32_t *trial_voxel, int *bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t first = (int64_t)rows5[5 * i + 3], last = (int64_t)rows5[5 * i + 4];
        const int64_t o = off[i];
        int64_t cnt = last >= first ? last - first + 1 : 0;
        if (cnt > 0 && (first < 1 || last > n_neigb)) {
            atomicOr(bad, 1);
            cnt = 0;
        }
        for (int64_t j = 0; j < cnt; ++j) {
            int64_t gid = (int64_t)id_neigb[first - 1 + j];
            if (gid < 1 || gid > n_grain) {
                atomicOr(bad, 2);
                gid = 1;
            }
            trial_orient[o + j] = (int32_t)(gid - 1);
            trial_voxel[o + j] = (int32_t)i;
        }
        items[i] = make_longlong4(i, o, o + cnt, 0);
    }
}

// Argmax over each voxel's candidates with MATLAB max semantics (first max, NaN ignored).
__global__ void epi_compete_k(const TrialRes *res, const longlong4 *items, const int32_t *trial_orient, int64_t m,
                              const float *euler, float *out, float *trial_out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const longlong4 it = items[i];
        float *w = out + 8 * i;
        w[0] = (float)(i + 1);
        for (int k = 1; k < 8; ++k) w[k] = 0.f;
        w[7] = 2000.f;
        int64_t best = -1;
        double bestC = CUDART_NAN;
        for (int64_t t = it.y; t < it.z; ++t) {
            const TrialRes r = res[t];
            const double C = (double)r.inter / (double)r.simu;
            if (best < 0 || (!isnan(C) && (isnan(bestC) || C > bestC))) {
                best = t;
                bestC = C;
            }
            if (trial_out) {
                float4 o;
                o.x = (float)r.simu;
                o.y = (float)r.inter;
                o.z = (float)C;
                o.w = (float)r.median;
                reinterpret_cast<float4 *>(trial_out)[t] = o;
            }
        }
        if (best >= 0) {
            const int32_t gi = trial_orient[best];
            const TrialRes r = res[best];
            w[1] = euler[3 * gi];
            w[2] = euler[3 * gi + 1];
            w[3] = euler[3 * gi + 2];
            w[4] = (float)(gi + 1);
            w[5] = (float)bestC;
            w[6] = (float)r.inter;
            w[7] = (float)r.median;
        }
    }
}

// grow_unindexed_compete_comp_cuda.m:51-64 on device: write each voxel's winner into the
// sample maps (MATLAB column-major volumes, 1-based voxel indices in rows5).
__global__ void apply_compete_k(const float *out8, const float *rows5, int64_t m, int64_t d1, int64_t d2,
                                int64_t d3, float *comp, float *gid, float *dmed, float *ninter, float *visit) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t x = (int64_t)rows5[5 * i] - 1, y = (int64_t)rows5[5 * i + 1] - 1, z = (int64_t)rows5[5 * i + 2] - 1;
        if (x < 0 || y < 0 || z < 0 || x >= d1 || y >= d2 || z >= d3) continue;
        const int64_t k = x + d1 * (y + d2 * z);
        const float *o = out8 + 8 * i;
        if (comp) comp[k] = o[5];
        if (gid) gid[k] = o[4];
        if (dmed) dmed[k] = o[7];
        if (ninter) ninter[k] = o[6];
        if (visit) visit[k] = 0.5f;
    }
}

// ---- distance-map rank coding --------------------------------------------------
// Each float maps to an order-preserving 32-bit key; a presence bitmap over the keys plus a prefix
// popcount gives every value its rank among the distinct values.  A map uses few of the 65,536 upper
// halves of the keys (all distances on 1024 x 1024 pixels: 898), so the bitmap holds 65,536 bits for
// each half in use only: a first pass finds those and numbers them (slots).  The bitmap of all keys took
// 1.5 GB with its counts, allocated, cleared and read at every upload; 190 M pixels coded 2.9 -> 1.5 ms
// (three reads of the map, 0.12 ms each at the copy rate; the rest is the codes' gather of 8 bytes per
// pixel from L2, 0.72 ms), and the buffers of the map before are used again where they fit.

__device__ __forceinline__ uint32_t ordered_key(float v) {
    if (v == 0.0f) v = 0.0f;  // -0 and +0 are the same value
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ float key_value(uint32_t k) {
    const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(b);
}

constexpr int kHalfWords = 2048;  // words of 65,536 bits: of the halves in use, and of each half

// f(index, value) of the map, four values per load where its address allows.
template <typename F>
__device__ __forceinline__ void each_value(const float *map, int64_t n, F f) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t n4 = ((uintptr_t)map & 15u) ? 0 : n >> 2;
    for (int64_t i = t; i < n4; i += stride) {
        const float4 v = __ldcs(reinterpret_cast<const float4 *>(map) + i);
        f(4 * i, v.x);
        f(4 * i + 1, v.y);
        f(4 * i + 2, v.z);
        f(4 * i + 3, v.w);
    }
    for (int64_t i = 4 * n4 + t; i < n; i += stride) f(i, map[i]);
}

__global__ void mark_halves_k(const float *map, int64_t n, uint32_t *halves, int *bad) {
    __shared__ uint32_t seen[kHalfWords];
    for (int i = threadIdx.x; i < kHalfWords; i += blockDim.x) seen[i] = 0;
    __syncthreads();
    bool nan = false;
    each_value(map, n, [&](int64_t, float v) {
        nan |= isnan(v);
        const uint32_t h = ordered_key(v) >> 16, bit = 1u << (h & 31);
        if (!(seen[h >> 5] & bit)) atomicOr(&seen[h >> 5], bit);
    });
    if (nan) atomicOr(bad, 1);
    __syncthreads();
    for (int i = threadIdx.x; i < kHalfWords; i += blockDim.x)
        if (seen[i]) atomicOr(&halves[i], seen[i]);
}

// Halves in use before each word of `halves` (one block of 1024), the half of each slot, their number.
__global__ void number_halves_k(const uint32_t *halves, uint32_t *before, uint32_t *half_of, int *count) {
    __shared__ uint32_t sum[1024];
    const int t = threadIdx.x;
    const uint32_t a = halves[2 * t], b = halves[2 * t + 1];
    uint32_t incl = __popc(a) + __popc(b);
    const uint32_t own = incl;
    sum[t] = incl;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const uint32_t y = t >= o ? sum[t - o] : 0u;
        __syncthreads();
        sum[t] = incl += y;
        __syncthreads();
    }
    uint32_t slot = incl - own;
    before[2 * t] = slot;
    before[2 * t + 1] = slot + __popc(a);
    for (int w = 0; w < 2; ++w)
        for (uint32_t m = w ? b : a; m; m &= m - 1) half_of[slot++] = (uint32_t)(64 * t + 32 * w + __ffs(m) - 1);
    if (t == 1023) *count = (int)incl;
}

// Word of a key in the compact bitmap, from the CTA's copy of `halves` and `before`.
struct HalfTable {
    uint32_t bits[kHalfWords], before[kHalfWords];
    __device__ __forceinline__ void load(const uint32_t *halves, const uint32_t *b) {
        for (int i = threadIdx.x; i < kHalfWords; i += blockDim.x) {
            bits[i] = halves[i];
            before[i] = b[i];
        }
        __syncthreads();
    }
    __device__ __forceinline__ uint32_t word(uint32_t k) const {
        const uint32_t h = k >> 16, slot = before[h >> 5] + __popc(bits[h >> 5] & ((1u << (h & 31)) - 1u));
        return slot * kHalfWords + ((k & 0xffffu) >> 5);
    }
};

// Values seen lately by the CTA, so that most pixels need no word of the bitmap (0.59 -> 0.54 ms; the
// same for the codes, 8 bytes an entry, ran 1.16 ms instead of 0.72).  Key 0 is a NaN's: never stored.
constexpr int kSeen = 8192;
__device__ __forceinline__ uint32_t seen_slot(uint32_t k) { return (k * 2654435761u) >> 19; }

__global__ void mark_values_k(const float *map, int64_t n, const uint32_t *halves, const uint32_t *before,
                              uint32_t *bitmap) {
    extern __shared__ unsigned char mark_smem[];
    HalfTable &tab = *reinterpret_cast<HalfTable *>(mark_smem);
    volatile uint32_t *seen = reinterpret_cast<uint32_t *>(mark_smem + sizeof(HalfTable));
    for (int i = threadIdx.x; i < kSeen; i += blockDim.x) seen[i] = 0;
    tab.load(halves, before);
    each_value(map, n, [&](int64_t, float v) {
        const uint32_t k = ordered_key(v), at = seen_slot(k);
        if (seen[at] == k) return;
        seen[at] = k;
        const uint32_t w = tab.word(k), bit = 1u << (k & 31);
        if (!(bitmap[w] & bit)) atomicOr(&bitmap[w], bit);
    });
}

__global__ void popc_k(const uint32_t *bitmap, int64_t nw, uint32_t *cnt) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nw; i += (int64_t)gridDim.x * blockDim.x)
        cnt[i] = __popc(bitmap[i]);
}

// The value of every rank, and each word's {bits, rank of its first} side by side.
__global__ void values_k(const uint32_t *bitmap, const uint32_t *prefix, const uint32_t *half_of, int64_t nw,
                         uint2 *pairs, float *vals) {
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < nw; w += (int64_t)gridDim.x * blockDim.x) {
        uint32_t bits = bitmap[w], r = prefix[w];
        pairs[w] = make_uint2(bits, r);
        const uint32_t base = (half_of[w / kHalfWords] << 16) | ((uint32_t)(w % kHalfWords) << 5);
        for (; bits; bits &= bits - 1) vals[r++] = key_value(base | (uint32_t)(__ffs(bits) - 1));
    }
}

template <typename CodeT>
__global__ void codes_k(const float *map, int64_t n, const uint32_t *halves, const uint32_t *before,
                        const uint2 *pairs, CodeT *codes, uint8_t *codes8) {
    __shared__ HalfTable tab;
    tab.load(halves, before);
    auto code_of = [&](float v) {
        const uint32_t k = ordered_key(v);
        const uint2 p = __ldg(pairs + tab.word(k));
        return p.y + __popc(p.x & ((1u << (k & 31)) - 1u));
    };
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t n4 = ((uintptr_t)map & 15u) ? 0 : n >> 2;
    struct __align__(4 * sizeof(CodeT)) Code4 {
        CodeT x, y, z, w;
    };
    for (int64_t i = t; i < n4; i += stride) {
        const float4 v = __ldcs(reinterpret_cast<const float4 *>(map) + i);
        const uint32_t a = code_of(v.x), b = code_of(v.y), c = code_of(v.z), d = code_of(v.w);
        reinterpret_cast<Code4 *>(codes)[i] = Code4{(CodeT)a, (CodeT)b, (CodeT)c, (CodeT)d};
        reinterpret_cast<uint32_t *>(codes8)[i] =
            min(a, 255u) | min(b, 255u) << 8 | min(c, 255u) << 16 | min(d, 255u) << 24;
    }
    for (int64_t i = 4 * n4 + t; i < n; i += stride) {
        const uint32_t c = code_of(map[i]);
        codes[i] = (CodeT)c;
        codes8[i] = (uint8_t)min(c, 255u);
    }
}

// Of the pixels in the middle of the detector (35 % of its width and height, at most 64 rows of at most
// 32 projections), how many have code 255 and more.  Reflections of arbitrary orientations land there
// more often than at the edges: the share tells within 0.06 what fraction of a wrong orientation's
// landings has such a code (40 maps, 1 to 48 grains on 400 x 500 to 2048^2 pixels).
struct Middle {
    int64_t y0, z0, rows, width, row_step, rows_seen, rot_step, rots_seen;
    Middle(int64_t nz, int64_t ny, int64_t nrot) {
        rows = (ny * 35 + 99) / 100, width = (nz * 35 + 99) / 100;
        y0 = (ny - rows) / 2, z0 = (nz - width) / 2;
        row_step = (rows + 63) / 64, rows_seen = (rows + row_step - 1) / row_step;
        rot_step = (nrot + 31) / 32, rots_seen = (nrot + rot_step - 1) / rot_step;
    }
    double pixels() const { return (double)rows_seen * rots_seen * width; }
};

__global__ void far_share_k(const uint8_t *codes8, int64_t nz, int64_t ny, Middle m, int *count) {
    const int64_t y = m.y0 + (blockIdx.x % m.rows_seen) * m.row_step, iw = (blockIdx.x / m.rows_seen) * m.rot_step;
    const uint8_t *row = codes8 + (iw * ny + y) * nz + m.z0;
    int far = 0;
    for (int64_t z = threadIdx.x; z < m.width; z += blockDim.x) far += row[z] == 255;
    far = __reduce_add_sync(0xffffffffu, far);
    if ((threadIdx.x & 31) == 0 && far) atomicAdd(count, far);
}

// ---- exact EDT (bwdist semantics) ------------------------------------------------
// Along detz (contiguous) each row becomes one entry per 32 pixels: their bits, and the 1-based
// positions of the last spot pixel before and the first after them (0: none).  Across dety a CTA
// takes 32 columns of a projection, writes every row's distance g along detz to shared memory, and
// minimises g(y')^2 + (y - y')^2: an outward search for every kEdtStep-th row, and for the rows between
// two of those only over the rows between their minimisers (y' of the minimum does not decrease
// with y: for j < a, f(y, j) - f(y, a) grows with y).  Both pass over kEdtBlock rows at a time whose
// least g shows that they cannot do better: without that a warp's 32 columns, whose ranges differ,
// pay for the widest of them (3.9 ms).  Bound by issue (77 % of slots).  BCC Fe 1024^2 x 181 with 0.2 % spot
// pixels: rows 3.13 (one thread per row) -> 0.06 ms, columns 36.3 (outward in L2 for each pixel) -> 0.98 ms.
// Bit i: byte i of x is not 0.
__device__ __forceinline__ uint32_t nibble(uint32_t x) {
    const uint32_t m = ((x & 0x7f7f7f7fu) + 0x7f7f7f7fu | x) & 0x80808080u;  // 0x80 in each such byte
    return (m >> 7) * 0x10204080u >> 28;                                     // bits 0, 8, 16, 24 side by side
}

// The 32 words of a row's pixels [1024 * chunk, ...): lane l gets word l.
__device__ __forceinline__ uint32_t row_words(const uint8_t *m, int64_t nz, int chunk, bool wide, int lane) {
    const int64_t z0 = (int64_t)chunk * 1024;
    uint32_t mine = 0;
    if (wide) {
        // 16 pixels per lane and load: the half word of each, then word `lane` from two lanes
        uint32_t half[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int64_t z = z0 + j * 512 + 16 * lane;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (z < nz) v = *reinterpret_cast<const uint4 *>(m + z);
            half[j] = nibble(v.x) | nibble(v.y) << 4 | nibble(v.z) << 8 | nibble(v.w) << 12;
        }
        const int from = 2 * (lane & 15);
        const uint32_t a0 = __shfl_sync(0xffffffffu, half[0], from), a1 = __shfl_sync(0xffffffffu, half[0], from + 1);
        const uint32_t b0 = __shfl_sync(0xffffffffu, half[1], from), b1 = __shfl_sync(0xffffffffu, half[1], from + 1);
        mine = lane < 16 ? a0 | a1 << 16 : b0 | b1 << 16;
    } else {
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const int64_t z = z0 + j * 32 + lane;
            const unsigned w = __ballot_sync(0xffffffffu, z < nz && m[z]);
            if (lane == j) mine = w;
        }
    }
    return mine;
}

// A warp takes kEdtRows rows of a projection, so that a lane's entries of a word are 32 bytes side by side.
constexpr int kEdtRows = 4;
__global__ void edt_rows_k(const uint8_t *mask, int64_t nz, int64_t ny, int64_t nrot, uint2 *ent) {
    const int lane = threadIdx.x & 31;
    const int nw = (int)((nz + 31) / 32), chunks = (nw + 31) / 32;
    const bool wide = nz % 16 == 0 && ((uintptr_t)mask & 15u) == 0;  // every row starts on 16 bytes
    const int64_t groups = (ny + kEdtRows - 1) / kEdtRows, warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < nrot * groups; t += warps) {
        const int64_t iw = t / groups, y0 = (t - iw * groups) * kEdtRows;
        const uint8_t *m = mask + (iw * ny + y0) * nz;
        const int rows = (int)min((int64_t)kEdtRows, ny - y0);
        // lane c: last and first spot pixel (1-based; 0 and 0xffff: none) of chunk c of each row
        uint32_t last[kEdtRows] = {}, first[kEdtRows];
#pragma unroll
        for (int r = 0; r < kEdtRows; ++r) first[r] = 0xffffu;
        for (int c = 0; chunks > 1 && c < chunks; ++c)
            for (int r = 0; r < rows; ++r) {
                const uint32_t w = row_words(m + r * nz, nz, c, wide, lane);
                const int base = c * 1024 + lane * 32;
                const uint32_t hi = __reduce_max_sync(0xffffffffu, w ? base + 32 - __clz(w) : 0);
                const uint32_t lo = __reduce_min_sync(0xffffffffu, w ? base + __ffs(w) : 0xffff);
#pragma unroll
                for (int q = 0; q < kEdtRows; ++q)
                    if (q == r && lane == c) last[q] = hi, first[q] = lo;
            }
        for (int c = 0; c < chunks; ++c) {
            uint2 e[kEdtRows];
#pragma unroll
            for (int r = 0; r < kEdtRows; ++r) {
                const uint32_t w = r < rows ? row_words(m + r * nz, nz, c, wide, lane) : 0u;
                const uint32_t before = __reduce_max_sync(0xffffffffu, lane < c ? last[r] : 0u);
                const uint32_t after = __reduce_min_sync(0xffffffffu, lane > c ? first[r] : 0xffffu);
                const unsigned any = __ballot_sync(0xffffffffu, w != 0);
                const unsigned lower = any & ((1u << lane) - 1u), upper = any & (0xfffffffeu << lane);
                // the nearest words with spots on either side, and the words they hold
                const int from = lower ? 31 - __clz(lower) : 0, to = upper ? __ffs(upper) - 1 : 0;
                const uint32_t wl = __shfl_sync(0xffffffffu, w, from), wr = __shfl_sync(0xffffffffu, w, to);
                const uint32_t prev = lower ? (uint32_t)(c * 1024 + from * 32 + 32 - __clz(wl)) : before;
                const uint32_t next = upper ? (uint32_t)(c * 1024 + to * 32 + __ffs(wr)) : after == 0xffffu ? 0u : after;
                e[r] = make_uint2(w, prev | next << 16);
            }
            const int k = c * 32 + lane;
            if (k < nw) {
                uint2 *o = ent + (iw * nw + k) * ny + y0;
#pragma unroll
                for (int r = 0; r < kEdtRows; ++r)
                    if (r < rows) o[r] = e[r];
            }
        }
    }
}

constexpr int kEdtStep = 24;             // rows per searched row (8: 1.59, 16: 1.09, 32: 1.09 ms)
constexpr int kEdtBlock = 8;             // rows passed over at a time
constexpr int kEdtNoSpot = 0x7fff;       // distance along detz in a row without spots
constexpr int kEdtNone = kEdtNoSpot * kEdtNoSpot;
__host__ __device__ inline size_t edt_smem_bytes(int64_t ny) {
    return sizeof(uint16_t) * 32 * (ny + (ny + kEdtBlock - 1) / kEdtBlock + (ny + kEdtStep - 1) / kEdtStep + 1);
}
// Rows and columns that the strip kernel takes: 16-bit positions, squares below kEdtNone, and a
// strip's rows within a CTA's shared memory.  Larger detectors take the line and column kernels.
inline bool edt_strips(int64_t nz, int64_t ny) { return nz <= 16384 && edt_smem_bytes(ny) <= 224 * 1024; }

__global__ void edt_strip_k(const uint2 *ent, int64_t nz, int64_t ny64, float *map) {
    extern __shared__ uint16_t edt_s[];
    const int ny = (int)ny64, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int n_block = (ny + kEdtBlock - 1) / kEdtBlock, n_step = (ny + kEdtStep - 1) / kEdtStep;
    // [row * 32] distances along detz, [block * 32] the least of a block's, [step * 32] minimisers
    uint16_t *g = edt_s + lane, *gmin = g + 32 * ny, *arg = gmin + 32 * n_block;
    const int nw = (int)((nz + 31) / 32), w = blockIdx.x;
    const int64_t iw = blockIdx.y;
    const uint2 *e0 = ent + (iw * nw + w) * ny64;
    const int z = w * 32 + lane;
    for (int k = warp; k < n_block; k += warps) {
        int least = kEdtNoSpot;
#pragma unroll
        for (int i = 0; i < kEdtBlock; ++i) {
            const int y = k * kEdtBlock + i;
            if (y >= ny) break;
            const uint2 e = e0[y];
            const uint32_t lo = e.x & (0xffffffffu >> (31 - lane)), hi = e.x & (0xffffffffu << lane);
            const int prev = (int)(e.y & 0xffffu), next = (int)(e.y >> 16);
            int d = kEdtNoSpot;
            if (lo) d = lane - (31 - __clz(lo));
            else if (prev) d = z - (prev - 1);
            if (hi) d = min(d, __ffs(hi) - 1 - lane);
            else if (next) d = min(d, next - 1 - z);
            g[32 * y] = (uint16_t)d;
            least = min(least, d);
        }
        gmin[32 * k] = (uint16_t)least;
    }
    __syncthreads();
    // ---- the searched rows: the first of each step, and the last row
    for (int k = warp; k <= n_step; k += warps) {
        const int y = min(k * kEdtStep, ny - 1), kb = y / kEdtBlock;
        int best = 0x7fffffff, at = y;
        auto look = [&](int c, int gap) {  // block c, whose nearest row is `gap` rows away
            if (c < 0 || c >= n_block) return;
            const int least = gmin[32 * c];
            if (least * least + gap * gap >= best) return;
            const int y1 = c * kEdtBlock;
#pragma unroll
            for (int i = 0; i < kEdtBlock; ++i) {
                if (y1 + i >= ny) break;
                const int d = y1 + i - y, v = g[32 * (y1 + i)], f = v * v + d * d;
                if (f < best) best = f, at = y1 + i;
            }
        };
        look(kb, 0);
        for (int d = 1; d < n_block; ++d) {
            const int left = y - (kb - d) * kEdtBlock - (kEdtBlock - 1), right = (kb + d) * kEdtBlock - y;
            const int gap = min(left, right);
            if (gap * gap >= best) break;
            look(kb - d, left);
            look(kb + d, right);
        }
        arg[32 * k] = (uint16_t)at;
    }
    __syncthreads();
    // ---- every row, from its step's two minimisers and the blocks between them that could do better
    for (int k = warp; k < n_step; k += warps) {
        const int y0 = k * kEdtStep, a = arg[32 * k], b = arg[32 * (k + 1)];
        const int ga = g[32 * a], gb = g[32 * b], fa = ga * ga, fb = gb * gb;
        int best[kEdtStep], most = 0;
#pragma unroll
        for (int i = 0; i < kEdtStep; ++i) {
            best[i] = min(fa + (y0 + i - a) * (y0 + i - a), fb + (y0 + i - b) * (y0 + i - b));
            most = max(most, best[i]);
        }
        const int last = max(a, b) / kEdtBlock;
        for (int c = min(a, b) / kEdtBlock; c <= last; ++c) {
            const int least = gmin[32 * c];
            const int gap = max(0, max(c * kEdtBlock - (y0 + kEdtStep - 1), y0 - c * kEdtBlock - (kEdtBlock - 1)));
            if (least * least + gap * gap >= most) continue;
#pragma unroll
            for (int j = 0; j < kEdtBlock; ++j) {
                if (c * kEdtBlock + j >= ny) break;
                const int v = g[32 * (c * kEdtBlock + j)], s = v * v, d = y0 - c * kEdtBlock - j;
                const int near = max(0, max(-d - (kEdtStep - 1), d));
                if (s + near * near >= most) continue;
#pragma unroll
                for (int i = 0; i < kEdtStep; ++i) best[i] = min(best[i], s + (d + i) * (d + i));
            }
            most = 0;
#pragma unroll
            for (int i = 0; i < kEdtStep; ++i) most = max(most, best[i]);
        }
        float *o = map + (iw * ny64 + y0) * nz + z;
        if (z < nz) {
#pragma unroll
            for (int i = 0; i < kEdtStep; ++i)
                if (y0 + i < ny) o[i * nz] = best[i] >= kEdtNone ? CUDART_INF_F : sqrtf((float)best[i]);
        }
    }
}

// Detectors beyond the strip kernel's range.  Pass 1: along detz the squared distance to the nearest
// marked pixel of the same line (two sweeps).  Pass 2: along dety, D(y) = min_y' g(y') + (y-y')^2
// by an outward search that stops once (y-y')^2 exceeds the best value.
__global__ void edt_lines_k(const uint8_t *mask, int64_t nz, int64_t nlines, float *g) {
    for (int64_t line = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; line < nlines;
         line += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t *m = mask + line * nz;
        float *o = g + line * nz;
        int64_t last = -1;
        for (int64_t z = 0; z < nz; ++z) {
            if (m[z]) last = z;
            o[z] = last < 0 ? CUDART_INF_F : (float)((z - last) * (z - last));
        }
        last = -1;
        for (int64_t z = nz - 1; z >= 0; --z) {
            if (m[z]) last = z;
            if (last >= 0) {
                const float d = (float)((last - z) * (last - z));
                if (d < o[z]) o[z] = d;
            }
        }
    }
}

__global__ void edt_cols_k(const float *g, int64_t nz, int64_t ny, int64_t nrot, float *map) {
    const int64_t n = nz * ny * nrot;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t z = i % nz;
        const int64_t y = (i / nz) % ny;
        const int64_t base = i - y * nz;  // (iw, 0, z)
        float best = g[i];
        for (int64_t d = 1; (float)(d * d) < best && (y - d >= 0 || y + d < ny); ++d) {
            const float dd = (float)(d * d);
            if (y - d >= 0) {
                const float c = g[base + (y - d) * nz] + dd;
                if (c < best) best = c;
            }
            if (y + d < ny) {
                const float c = g[base + (y + d) * nz] + dd;
                if (c < best) best = c;
            }
        }
        map[i] = isinf(best) ? CUDART_INF_F : sqrtf(best);
        (void)z;
    }
}

}  // namespace

namespace {
struct OccEntry {
    int device;
    const void *fn;
    size_t smem;
    int per_sm;
};
struct SmemEntry {
    int device;
    const void *fn;
    size_t allowed;
};
std::mutex g_launch_mu;
std::vector<OccEntry> g_occ;
std::vector<SmemEntry> g_smem;

// caller holds g_launch_mu
cudaError_t allow_smem_locked(int dev, const void *fn, size_t smem) {
    for (SmemEntry &e : g_smem)
        if (e.device == dev && e.fn == fn) {
            if (e.allowed >= smem) return cudaSuccess;
            const cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (r == cudaSuccess) e.allowed = smem;
            return r;
        }
    const cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r == cudaSuccess) g_smem.push_back({dev, fn, smem});
    return r;
}
}  // namespace

cudaError_t allow_smem(const void *fn, size_t smem) {
    int dev = 0;
    cudaError_t r = cudaGetDevice(&dev);
    if (r != cudaSuccess) return r;
    std::lock_guard<std::mutex> g(g_launch_mu);
    return allow_smem_locked(dev, fn, smem);
}

cudaError_t occupancy_for(const void *fn, size_t smem, int *per_sm) {
    int dev = 0;
    cudaError_t r = cudaGetDevice(&dev);
    if (r != cudaSuccess) return r;
    std::lock_guard<std::mutex> g(g_launch_mu);
    for (const OccEntry &e : g_occ)
        if (e.device == dev && e.fn == fn && e.smem == smem) {
            *per_sm = e.per_sm;
            return cudaSuccess;
        }
    r = allow_smem_locked(dev, fn, smem);
    if (r != cudaSuccess) return r;
    int n = 0;
    r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kThreads, smem);
    if (r != cudaSuccess) return r;
    g_occ.push_back({dev, fn, smem, n});
    *per_sm = n;
    return cudaSuccess;
}

cudaError_t launch_quat_to_u(const float *q, int64_t n, double *U, cudaStream_t s) {
    quat_to_u_k<<<blocks_for(n), kB, 0, s>>>(q, n, U);
    return cudaGetLastError();
}
cudaError_t launch_euler_to_u(const float *e, int64_t n, double *U, cudaStream_t s) {
    euler_to_u_k<<<blocks_for(n), kB, 0, s>>>(e, n, U);
    return cudaGetLastError();
}
cudaError_t launch_f9_to_u(const float *u9, int64_t n, double *U, cudaStream_t s) {
    f_to_d_k<<<blocks_for(9 * n), kB, 0, s>>>(u9, 9 * n, U);
    return cudaGetLastError();
}
cudaError_t launch_pos_f3(const float *p, int64_t n, double *vpos, cudaStream_t s) {
    f_to_d_k<<<blocks_for(3 * n), kB, 0, s>>>(p, 3 * n, vpos);
    return cudaGetLastError();
}
cudaError_t launch_pos_rows(const float *rows, int stride, int64_t n, const double *p1, double *vpos,
                            cudaStream_t s) {
    pos_rows_k<<<blocks_for(n), kB, 0, s>>>(rows, stride, n, p1, vpos);
    return cudaGetLastError();
}
cudaError_t launch_epi_forward(const TrialRes *res, int64_t n, float *out4, bool median, cudaStream_t s) {
    epi_forward_k<<<blocks_for(n), kB, 0, s>>>(res, n, out4, median ? 1 : 0);
    return cudaGetLastError();
}
cudaError_t launch_epi_grow(const TrialRes *res, const float *rows6, int64_t m, const double *p1, float *out7,
                            cudaStream_t s) {
    epi_grow_k<<<blocks_for(m), kB, 0, s>>>(res, rows6, m, p1, out7);
    return cudaGetLastError();
}
cudaError_t launch_csr_counts(const float *rows5, int64_t m, int64_t *counts, cudaStream_t s) {
    csr_counts_k<<<blocks_for(m), kB, 0, s>>>(rows5, m, counts);
    return cudaGetLastError();
}
cudaError_t launch_csr_fill(const float *rows5, int64_t m, const int64_t *offsets, const float *id_neigb,
                            int64_t n_neigb, int64_t n_grain, longlong4 *items, int32_t *trial_orient,
                            int32_t *trial_voxel, int *bad, cudaStream_t s) {
    csr_fill_k<<<blocks_for(m), kB, 0, s>>>(rows5, m, offsets, id_neigb, n_neigb, n_grain, items, trial_orient,
                                            trial_voxel, bad);
    return cudaGetLastError();
}
cudaError_t launch_epi_compete(const TrialRes *res, const longlong4 *items, const int32_t *trial_orient, int64_t m,
                               const float *euler, float *out8, float *trial_out4, cudaStream_t s) {
    epi_compete_k<<<blocks_for(m), kB, 0, s>>>(res, items, trial_orient, m, euler, out8, trial_out4);
    return cudaGetLastError();
}

cudaError_t launch_apply_compete(const float *out8, const float *rows5, int64_t m, const int64_t *dims, float *comp,
                                 float *gid, float *dmed, float *ninter, float *visit, cudaStream_t s) {
    apply_compete_k<<<blocks_for(m), kB, 0, s>>>(out8, rows5, m, dims[0], dims[1], dims[2], comp, gid, dmed, ninter,
                                                 visit);
    return cudaGetLastError();
}

cudaError_t Scratch::get(size_t bytes, cudaStream_t s, void **out) {
    if (bytes <= cap) {
        *out = p;
        return cudaSuccess;
    }
    const bool keep = bytes <= kKeep;
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess) return e;
    if (keep) {
        if (p) {
            cudaStreamSynchronize(s);
            cudaFree(p);
        }
        p = q;
        cap = bytes;
    } else {
        once = q;
    }
    *out = q;
    return cudaSuccess;
}

void Scratch::done(cudaStream_t s) {
    if (!once) return;
    cudaStreamSynchronize(s);
    cudaFree(once);
    once = nullptr;
}

void Scratch::release() {
    cudaFree(p);
    p = nullptr;
    cap = 0;
}

void MapCodes::release() {
    cudaFree(codes);
    cudaFree(codes8);
    cudaFree(vals);
    *this = MapCodes{};
}

// A buffer of at least `bytes`: the one at hand when it is large enough and not over twice as large
// (64 MB spared), else a new one.
static cudaError_t take_buffer(void **p, size_t *cap, void *have, size_t have_cap, size_t bytes) {
    if (have && have_cap >= bytes && have_cap / 2 <= bytes + (32u << 20)) {
        *p = have;
        *cap = have_cap;
        return cudaSuccess;
    }
    *cap = bytes;
    return cudaMalloc(p, bytes);
}

cudaError_t encode_map(const float *d_map, int64_t nz, int64_t ny, int64_t nrot, cudaStream_t s, MapCodes *resident,
                       Scratch *ws, int *bad_nan) {
    const int64_t n = nz * ny * nrot;
    // [kHalfWords] halves in use, [kHalfWords] how many before, [65536] half of each slot, count, NaN flag,
    // far pixels
    constexpr size_t kMarkSmem = sizeof(HalfTable) + sizeof(uint32_t) * kSeen;
    constexpr size_t kSmall = sizeof(uint32_t) * (2 * kHalfWords + 65536 + 3);
    const int blocks = std::min(blocks_for(n, kB * 4), 148 * 8);  // each loads the 16 KB table of halves
    uint32_t *small = nullptr;
    MapCodes out{};
    void *tmp = nullptr;
    cudaError_t e;
    bool shared = false;  // buffers of the resident map are being written
    *bad_nan = 0;
    if (n <= 0) {  // no pixel, no value
        resident->n_distinct = 0;
        resident->code_bits = 0;
        resident->far_share = 0;
        return cudaSuccess;
    }
#define CK(x)                                       \
    do {                                            \
        if ((e = (x)) != cudaSuccess) goto failed;  \
    } while (0)
    CK(ws[0].get(kSmall, s, (void **)&small));
    {
        uint32_t *halves = small, *before = small + kHalfWords, *half_of = small + 2 * kHalfWords;
        int *info = (int *)(half_of + 65536), hinfo[2] = {0, 0}, far = 0;  // halves in use, NaN seen
        CK(cudaMemsetAsync(halves, 0, sizeof(uint32_t) * kHalfWords, s));
        CK(cudaMemsetAsync(info, 0, 3 * sizeof(int), s));
        mark_halves_k<<<blocks, kB, 0, s>>>(d_map, n, halves, info + 1);
        number_halves_k<<<1, 1024, 0, s>>>(halves, before, half_of, info);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(hinfo, info, sizeof hinfo, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        *bad_nan = hinfo[1];
        if (hinfo[1]) return cudaSuccess;  // the resident map stays as it is
        // bitmap, its counts, their prefix sums, and {bits, prefix} pairs
        const int64_t nw = (int64_t)hinfo[0] * kHalfWords;
        size_t tmp_bytes = 0;
        uint32_t *bitmap = nullptr;
        CK(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, bitmap, bitmap, (int)nw, s));
        const size_t head = (sizeof(uint32_t) * 5 * nw + 255) & ~size_t(255);
        CK(ws[1].get(head + tmp_bytes, s, (void **)&bitmap));
        uint32_t *cnt = bitmap + nw, *prefix = bitmap + 2 * nw, last[2] = {0, 0};
        uint2 *pairs = (uint2 *)(bitmap + (3 * nw + (nw & 1)));
        tmp = (char *)bitmap + head;
        CK(allow_smem((const void *)mark_values_k, kMarkSmem));
        CK(cudaMemsetAsync(bitmap, 0, sizeof(uint32_t) * nw, s));
        mark_values_k<<<blocks, kB, kMarkSmem, s>>>(d_map, n, halves, before, bitmap);
        popc_k<<<blocks_for(nw), kB, 0, s>>>(bitmap, nw, cnt);
        CK(cudaGetLastError());
        CK(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, cnt, prefix, (int)nw, s));
        CK(cudaMemcpyAsync(&last[0], prefix + nw - 1, 4, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(&last[1], cnt + nw - 1, 4, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        const int64_t nd = (int64_t)last[0] + last[1];
        out.n_distinct = nd;
        while (out.code_bits < 32 && (int64_t(1) << out.code_bits) < nd) ++out.code_bits;
        const bool c16 = nd <= 65536;
        CK(take_buffer((void **)&out.vals, &out.cap_vals, resident->vals, resident->cap_vals, sizeof(float) * nd));
        // 32-bit words of codes are read, so the last is whole
        CK(take_buffer((void **)&out.codes8, &out.cap_codes8, resident->codes8, resident->cap_codes8,
                       ((size_t)n + 3) & ~size_t(3)));
        CK(take_buffer(&out.codes, &out.cap_codes, resident->codes, resident->cap_codes, (size_t)n * (c16 ? 2 : 4)));
        shared = (out.codes && out.codes == resident->codes) || (out.codes8 && out.codes8 == resident->codes8) ||
                 (out.vals && out.vals == resident->vals);
        values_k<<<blocks_for(nw), kB, 0, s>>>(bitmap, prefix, half_of, nw, pairs, out.vals);
        if (c16)
            codes_k<uint16_t><<<blocks, kB, 0, s>>>(d_map, n, halves, before, pairs, (uint16_t *)out.codes, out.codes8);
        else
            codes_k<uint32_t><<<blocks, kB, 0, s>>>(d_map, n, halves, before, pairs, (uint32_t *)out.codes, out.codes8);
        const Middle mid(nz, ny, nrot);
        if (nz > 0 && ny > 0 && nrot > 0)
            far_share_k<<<(unsigned)(mid.rows_seen * mid.rots_seen), kB, 0, s>>>(out.codes8, nz, ny, mid, info + 2);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&far, info + 2, sizeof far, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        out.far_share = (float)(far / mid.pixels());
    }
    ws[1].done(s);
    if (resident->codes != out.codes) cudaFree(resident->codes);
    if (resident->codes8 != out.codes8) cudaFree(resident->codes8);
    if (resident->vals != out.vals) cudaFree(resident->vals);
    *resident = out;
    return cudaSuccess;
failed:
#undef CK
    ws[1].done(s);
    if (out.codes != resident->codes) cudaFree(out.codes);
    if (out.codes8 != resident->codes8) cudaFree(out.codes8);
    if (out.vals != resident->vals) cudaFree(out.vals);
    if (shared) resident->release();  // partly overwritten: no map is left
    return e;
}

cudaError_t launch_edt(const uint8_t *mask, int64_t nz, int64_t ny, int64_t nrot, float *map, Scratch *ws,
                       cudaStream_t s) {
    if (!edt_strips(nz, ny)) {
        float *g = nullptr;
        cudaError_t e = cudaMalloc(&g, sizeof(float) * nz * ny * nrot);
        if (e != cudaSuccess) return e;
        edt_lines_k<<<blocks_for(ny * nrot, 128), 128, 0, s>>>(mask, nz, ny * nrot, g);
        edt_cols_k<<<blocks_for(nz * ny * nrot, kB * 4), kB, 0, s>>>(g, nz, ny, nrot, map);
        e = cudaGetLastError();
        cudaError_t e2 = cudaStreamSynchronize(s);
        cudaFree(g);
        return e != cudaSuccess ? e : e2;
    }
    // as many projections at a time as keep their entries (a quarter byte per pixel) within the
    // scratch that is kept
    const int64_t nw = (nz + 31) / 32, per = (int64_t)sizeof(uint2) * nw * ny;
    int64_t step = (int64_t)Scratch::kKeep / per;
    step = step < 1 ? 1 : step > nrot ? nrot : step > 65535 ? 65535 : step;
    uint2 *ent = nullptr;
    cudaError_t e = ws->get((size_t)(per * step), s, (void **)&ent);
    if (e != cudaSuccess) return e;
    const size_t smem = edt_smem_bytes(ny);
    e = allow_smem((const void *)edt_strip_k, smem);
    if (e != cudaSuccess) return e;
    const int threads = smem > 110 * 1024 ? 1024 : smem > 72 * 1024 ? 512 : 256;  // some 24 warps per SM and more
    for (int64_t i = 0; i < nrot; i += step) {
        const int64_t c = nrot - i < step ? nrot - i : step;
        edt_rows_k<<<blocks_for(c * ((ny + kEdtRows - 1) / kEdtRows), 8), 256, 0, s>>>(mask + i * ny * nz, nz, ny, c, ent);
        edt_strip_k<<<dim3((unsigned)nw, (unsigned)c), threads, smem, s>>>(ent, nz, ny, map + i * ny * nz);
    }
    e = cudaGetLastError();
    const cudaError_t e2 = cudaStreamSynchronize(s);
    ws->done(s);
    return e != cudaSuccess ? e : e2;
}

}  // namespace grc
