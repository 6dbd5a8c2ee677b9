// grc_fit.cu -- derivatives of the continuous spot-centroid residual and the fits they drive.
//
// The reference fits grain orientation/centre (fit_grain_COM.m:5-88,
// fit_OR_fun_local.m) and the detector geometry (geo_fitting.m:5-78,
// L_shift_tilt_fitting.m:23-50) with fminsearchbnd (Nelder-Mead) on discrete
// objectives (rounded pixels, 1-completeness).  Here the residual is the continuous
// landing point (u, v) of forward_comp.m:28-59 -- no rounding -- minus the measured
// spot centroid, for a fixed set of matched (grain, omega, hkl) spots.
//
// Derivatives are propagated backwards by hand: u and v are two numbers of 6 (Rodrigues
// vector, centre) or 10 (Lsam2sou, Lsam2det, dety00, detz00, tilt_x/y/z, P0y, P0z,
// RotAxisOffset) parameters, so one backward pass for each costs about as much as the
// landing itself, whatever the number of parameters.  What does not depend on the spot
// is formed once per CTA: the detector rotation of a geometry (Beam), S*U*B of a grain.
// Everything is FP64.  Normal equations are solved per grain (6x6) or per start (10x10)
// with Levenberg-Marquardt damping.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "grc_fit.h"
#include "grc_internal.h"

namespace grc {
namespace {

// One geometry e[0..9] = Lsam2sou, Lsam2det, dety00, detz00, tilt_x, tilt_y, tilt_z [deg], P0y, P0z,
// RotAxisOffset, with RotDet = Rz*Ry*Rx (get_det_R.m:1-7).
struct Beam {
    double lss, lsd, y00, z00, p0y, p0z, rao;
    double R[9];      // row-major
    double ya, yb;    // axis of tilt_y: Rz e_y = (ya, yb, 0)
};

__device__ __noinline__ void make_beam(const double *e, Beam &b) {
    const double d2r = CUDART_PI / 180.0;
    double sx, cx, sy, cy, sz, cz;
    sincos(e[4] * d2r, &sx, &cx);
    sincos(e[5] * d2r, &sy, &cy);
    sincos(e[6] * d2r, &sz, &cz);
    b.lss = e[0], b.lsd = e[1], b.y00 = e[2], b.z00 = e[3], b.p0y = e[7], b.p0z = e[8], b.rao = e[9];
    b.R[0] = cz * cy, b.R[3] = sz * cy, b.R[6] = -sy;
    b.R[1] = cz * sy * sx - sz * cx, b.R[4] = sz * sy * sx + cz * cx, b.R[7] = cy * sx;
    b.R[2] = cz * sy * cx + sz * sx, b.R[5] = sz * sy * cx - cz * sx, b.R[8] = cy * cx;
    b.ya = -sz, b.yb = cz;
}

// U*B of a grain g[0..2] = Rodrigues vector r (U from q0 = 1/sqrt(1+|r|^2), q = r q0 via
// quaternion2U.m:3-28), g[3..5] = centre [mm].
__device__ void make_ub(const FitFixed &fx, const double *g, double *UB) {
    const double q0 = 1.0 / sqrt(1.0 + g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
    const double q1 = g[0] * q0, q2 = g[1] * q0, q3 = g[2] * q0;
    const double U[9] = {2.0 * (q0 * q0 + q1 * q1) - 1.0, 2.0 * (q1 * q2 - q0 * q3), 2.0 * (q1 * q3 + q0 * q2),
                         2.0 * (q1 * q2 + q0 * q3), 2.0 * (q0 * q0 + q2 * q2) - 1.0, 2.0 * (q2 * q3 - q0 * q1),
                         2.0 * (q1 * q3 - q0 * q2), 2.0 * (q2 * q3 + q0 * q1), 2.0 * (q0 * q0 + q3 * q3) - 1.0};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            UB[3 * i + j] = U[3 * i] * fx.B[j] + U[3 * i + 1] * fx.B[3 + j] + U[3 * i + 2] * fx.B[6 + j];
}

// y = M x, y = M^T x (row-major 3 x 3).
__device__ __forceinline__ void mul3(const double *M, double x, double y, double z, double *o) {
    o[0] = M[0] * x + M[1] * y + M[2] * z;
    o[1] = M[3] * x + M[4] * y + M[5] * z;
    o[2] = M[6] * x + M[7] * y + M[8] * z;
}
__device__ __forceinline__ void mul3t(const double *M, double x, double y, double z, double *o) {
    o[0] = M[0] * x + M[3] * y + M[6] * z;
    o[1] = M[1] * x + M[4] * y + M[7] * z;
    o[2] = M[2] * x + M[5] * y + M[8] * z;
}

enum : int { kGrain = 0, kGeometry = 1, kValue = 2 };

// Landing (u, v) of one spot -- the unrounded pixel coordinates of forward_comp.m:58-59 -- and its
// derivatives ju, jv with respect to the 6 grain (MODE kGrain) or 10 geometry parameters (kGeometry).
// UB: U*B of the grain g; (c, s) of omega; h: the reflection.  strict: false is returned when the
// reflection is outside the wavelength / Bragg-angle window or the detector (decides which spots
// exist); otherwise only for a non-finite landing (a matched spot stays in the residual during a fit).
template <int MODE>
__device__ __forceinline__ bool land_spot(const FitFixed &fx, const Beam &e, const double *g, const double *UB,
                                          double c, double s, const double *h, double &u, double &v, double *ju,
                                          double *jv, bool strict) {
    // G = Omega S U B h
    double ub[3], gw[3];
    mul3(UB, h[0], h[1], h[2], ub);
    mul3(fx.S, ub[0], ub[1], ub[2], gw);
    const double Gx = c * gw[0] - s * gw[1], Gy = s * gw[0] + c * gw[1], Gz = gw[2];
    const double k2 = Gy * Gy + Gz * Gz;
    const double rG = rsqrt(Gx * Gx + k2), rk = rsqrt(k2);
    const double gy = Gy * rk, gz = Gz * rk;
    // sample point and incident beam (forward_comp.m:17-26)
    double sp[3];
    mul3(fx.S, g[3], g[4] - e.rao, g[5], sp);
    const double swx = c * sp[0] - s * sp[1], swy = s * sp[0] + c * sp[1], swz = sp[2];
    const double px = e.lss + swx, py = swy - e.p0y + e.rao, pz = swz - e.p0z;
    const double n2 = px * px + py * py + pz * pz, rn = rsqrt(n2), ngp = n2 * rn, rx = 1.0 / px;
    const double kx = px * rn, ky = py * rn, kz = pz * rn;
    const double A = e.lsd - swx, Lrx = (e.lss + e.lsd) * rx;
    const double nrx = ngp * rx, L2 = A * nrx;
    // Bragg condition (forward_comp.m:28-37): x = cos(beta), tau = 2 theta, cph = cos(phi)
    const double x = (kx * Gx + ky * Gy + kz * Gz) * rG;
    const double lam = -4.0 * CUDART_PI * rG * x;
    if (strict && !(x < 0.0 && x > fx.cbmax && lam > fx.lmin && lam < fx.lmax)) return false;
    const double q = 1.0 - x * x, rct = rsqrt(q), ct = q == 0.0 ? 0.0 : q * rct;  // 0: straight back
    const double s2 = -2.0 * x * ct, c2 = 1.0 - 2.0 * x * x;
    const double cph = gy * ky + gz * kz, p = 1.0 - cph * cph, rsph = rsqrt(p), sph = p * rsph;
    const double rs = 1.0 / (sph * c2 - cph * s2);  // 1 / sin(phi - tau)
    const double D1 = s2 * rs, diff = L2 * D1;
    // tilted detector (forward_comp.m:49-55); K and d in the laboratory, X = f K + d on the detector
    const double Ky = py * Lrx - swy + diff * gy, Kz = pz * Lrx - swz + diff * gz;
    const double dx = swx - e.lsd, dy = swy - e.y00 + e.rao, dz = swz - e.z00;
    const double *R = e.R;
    const double rP = 1.0 / (R[0] * A + R[3] * Ky + R[6] * Kz);
    const double f = -(R[0] * dx + R[3] * dy + R[6] * dz) * rP;
    const double Xx = f * A + dx, Xy = f * Ky + dy, Xz = f * Kz + dz;
    const double y2 = R[1] * Xx + R[4] * Xy + R[7] * Xz, z2 = R[2] * Xx + R[5] * Xy + R[8] * Xz;
    const double su = -1.0 / fx.pxy, sv = -1.0 / fx.pxz;
    u = fx.dety0 + su * y2;
    v = fx.detz0 + sv * z2;
    if (MODE != kValue) {
        // diff = L2 sin(tau) / sin(phi - tau): d diff = D1 dL2 + T dx + F dcph
        const double cphy = cph * c2 + sph * s2;  // cos(phi - tau)
        const double T = (L2 * c2 + diff * cphy) * rs * (-2.0 * rct), F = diff * cphy * rs * rsph;
        const double TrG = T * rG, Arx = A * rx;
#pragma unroll
        for (int o = 1; o <= 2; ++o) {
            // y2 (or z2) = R(:,o).X with R(:,0).X = 0: its change is w.(f dK + dd) + the turn of R, with
            // w = R(:,o) - r R(:,0) and r = R(:,o).K / R(:,0).K
            const double r = (R[o] * A + R[3 + o] * Ky + R[6 + o] * Kz) * rP;
            const double wx = R[o] - r * R[0], wy = R[3 + o] - r * R[3], wz = R[6 + o] - r * R[6];
            const double lKy = f * wy, lKz = f * wz, ld = lKy * gy + lKz * gz;
            // back through k (x, cph), L2 and ay, az to the source-to-sample vector (px, py, pz)
            const double aT = ld * TrG, aF = ld * F, e1 = ld * D1;
            const double lkx = aT * Gx, lky = aT * Gy + aF * gy, lkz = aT * Gz + aF * gz;
            const double kd = e1 * Arx - rn * (kx * lkx + ky * lky + kz * lkz);
            const double lL = (lKy * py + lKz * pz) * rx;
            const double lpx = rn * lkx + kx * kd - e1 * L2 * rx - lL * Lrx;
            const double lpy = rn * lky + ky * kd + lKy * Lrx, lpz = rn * lkz + kz * kd + lKz * Lrx;
            const double lA = f * wx + e1 * nrx;
            const double lsx = lpx + wx - lA, lsy = lpy + wy - lKy, lsz = lpz + wz - lKz;  // to Omega S pos
            const double qx = c * lsx + s * lsy, qy = c * lsy - s * lsx;
            const double sc = o == 1 ? su : sv;
            double *J = o == 1 ? ju : jv;
            if (MODE == kGeometry) {
                const double d2r = CUDART_PI / 180.0;
                J[0] = sc * (lpx + lL);
                J[1] = sc * (lA + lL - wx);
                J[2] = -sc * wy;
                J[3] = -sc * wz;
                J[4] = sc * d2r * (o == 1 ? z2 : -y2);
                J[5] = sc * d2r * (Xz * (wy * e.ya - wx * e.yb) + wz * (Xx * e.yb - Xy * e.ya));
                J[6] = sc * d2r * (wx * Xy - wy * Xx);
                J[7] = -sc * lpy;
                J[8] = -sc * lpz;
                J[9] = sc * (lpy + wy - (fx.S[1] * qx + fx.S[4] * qy + fx.S[7] * lsz));
            } else {
                // centre: S^T Omega^T; orientation: dU b = omega x U b with omega = 2 (dr + r x dr) / (1 + r^2)
                double m[3];
                mul3t(fx.S, qx, qy, lsz, m);
                J[3] = sc * m[0], J[4] = sc * m[1], J[5] = sc * m[2];
                const double lpsi = (diff * (lKy * gz - lKz * gy) + aF * (ky * gz - kz * gy)) * rk;
                const double xr = x * rG;  // x = k.G / |G| (S need not keep |G|)
                const double lGx = aT * (kx - xr * Gx), lGy = aT * (ky - xr * Gy) + lpsi * gz,
                             lGz = aT * (kz - xr * Gz) - lpsi * gy;
                mul3t(fx.S, c * lGx + s * lGy, c * lGy - s * lGx, lGz, m);
                const double nx = ub[1] * m[2] - ub[2] * m[1], ny = ub[2] * m[0] - ub[0] * m[2],
                             nz = ub[0] * m[1] - ub[1] * m[0];
                const double w = 2.0 * sc / (1.0 + g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
                J[0] = w * (nx + ny * g[2] - nz * g[1]);
                J[1] = w * (ny + nz * g[0] - nx * g[2]);
                J[2] = w * (nz + nx * g[1] - ny * g[0]);
            }
        }
    }
    if (!strict) return isfinite(u) && isfinite(v);
    return u >= 0.5 && u < fx.detysize + 0.5 && v >= 0.5 && v < fx.detzsize + 0.5;
}

__device__ __forceinline__ bool spot_value(const FitFixed &fx, const Beam &e, const double *g, const double *UB, int iw,
                                           int ih, double &u, double &v, bool strict = false) {
    const double2 cs = fx.rot_cs[iw];
    return land_spot<kValue>(fx, e, g, UB, cs.x, cs.y, fx.hkl + 3 * ih, u, v, nullptr, nullptr, strict);
}

// What a thread reads of a spot, one spot ahead of the one it works on: the loads that hang on its
// indices (omega, reflection, grain) then find them at hand.
struct SpotRef {
    int64_t gi;
    int iw, ih;
    double u, v;
};
__device__ __forceinline__ SpotRef load_spot(const SpotList &sp, int64_t i, int64_t end) {
    SpotRef r{0, 0, 0, 0.0, 0.0};
    if (i < end) {
        r.gi = sp.grain[i];
        r.iw = sp.iw[i];
        r.ih = sp.ih[i];
        r.u = sp.uv[2 * i];
        r.v = sp.uv[2 * i + 1];
    }
    return r;
}

// The spot's landing against its measured centroid: the cost of forward-only fits (1e6 for a
// non-finite landing).
__device__ __forceinline__ double spot_cost(const FitFixed &fx, const Beam &e, const double *g, const double *UB,
                                            const SpotRef &r) {
    double u, v;
    if (!spot_value(fx, e, g, UB, r.iw, r.ih, u, v)) return 1e6;
    const double eu = u - r.u, ev = v - r.v;
    return eu * eu + ev * ev;
}

// ---- kernels -------------------------------------------------------------------------

// U*B (9 doubles) of every grain from 0 to kFitGrainTable that the spots name, into ub[9 * grain]: a spot
// whose predecessor belongs to another grain writes its grain's (the same values each time).  The
// entries that take it are not told how many grains there are; a spot of a later grain forms its own.
__global__ void grain_ub_k(FitFixed fx, const double *grains, SpotList sp, double *ub) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < sp.n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t gi = sp.grain[i];
        if ((i > 0 && sp.grain[i - 1] == gi) || !in_grain_table(gi)) continue;
        double M[9];
        make_ub(fx, grains + 6 * gi, M);
        for (int k = 0; k < 9; ++k) ub[9 * gi + k] = M[k];
    }
}

__device__ __forceinline__ void load_ub(const FitFixed &fx, const double *grains, const double *ub, int64_t gi,
                                        double *M) {
    if (in_grain_table(gi)) {
#pragma unroll
        for (int k = 0; k < 9; ++k) M[k] = ub[9 * gi + k];
    } else {
        make_ub(fx, grains + 6 * gi, M);
    }
}

// Per-spot residual (model - measured) and full Jacobian rows (2 x K).  A spot's 2 K derivatives are
// contiguous in the output: the CTA's go through shared memory, so that a warp writes whole lines
// (one thread per row of 80 or 160 bytes left every store to a line of its own).
constexpr int kJacThreads = 128;
template <int MODE>
__global__ void __launch_bounds__(kJacThreads) residual_jac_k(FitFixed fx, const double *grains, const double *ub,
                                                              const double *geo10, SpotList sp, double *res,
                                                              double *jac) {
    constexpr int K = MODE == kGrain ? 6 : 10;
    __shared__ Beam e;
    __shared__ double rows[kJacThreads * (2 * K + 1)];  // 2 K + 1: odd, so that lanes differ in bank
    const int t = threadIdx.x;
    if (t == 0) make_beam(geo10, e);
    __syncthreads();
    for (int64_t base = blockIdx.x * (int64_t)kJacThreads; base < sp.n; base += (int64_t)gridDim.x * kJacThreads) {
        const int64_t i = base + t;
        const int n = (int)min((int64_t)kJacThreads, sp.n - base);
        if (t < n) {
            const int64_t gi = sp.grain[i];
            double g[6], M[9], u, v, ju[K], jv[K];
#pragma unroll
            for (int k = 0; k < 6; ++k) g[k] = grains[6 * gi + k];
            load_ub(fx, grains, ub, gi, M);
            const double2 cs = fx.rot_cs[sp.iw[i]];
            const bool ok = land_spot<MODE>(fx, e, g, M, cs.x, cs.y, fx.hkl + 3 * sp.ih[i], u, v, ju, jv, false);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                rows[t * (2 * K + 1) + k] = ju[k];
                rows[t * (2 * K + 1) + K + k] = jv[k];
            }
            res[2 * i] = ok ? u - sp.uv[2 * i] : CUDART_NAN;
            res[2 * i + 1] = ok ? v - sp.uv[2 * i + 1] : CUDART_NAN;
        }
        __syncthreads();
        for (int k = t; k < n * 2 * K; k += kJacThreads) {
            const int r = k / (2 * K);
            jac[base * 2 * K + k] = rows[r * (2 * K + 1) + (k - r * 2 * K)];
        }
        __syncthreads();
    }
}

// Block reduction of n doubles per thread into out (thread 0 holds the sums).
template <int N>
__device__ __forceinline__ void block_sum(double (&a)[N], double *scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_down_sync(0xffffffffu, a[k], o);
    __syncthreads();
    if (lane == 0)
        for (int k = 0; k < N; ++k) scratch[warp * N + k] = a[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < N; ++k) {
            double t = 0;
            for (int w = 0; w < nw; ++w) t += scratch[w * N + k];
            a[k] = t;
        }
    __syncthreads();
}

// RMS distance of predicted spots between two parameter sets (fit vs ground truth), per grain.
__global__ void grain_rms_k(FitFixed fx, const double *grains, const double *truth, const double *geo10,
                            SpotList sp, const int64_t *offsets, int64_t n_grains, double *rms) {
    __shared__ double scratch[32 * 2];
    __shared__ Beam e;
    if (threadIdx.x == 0) make_beam(geo10, e);
    __syncthreads();
    for (int64_t gi = blockIdx.x; gi < n_grains; gi += gridDim.x) {
        double acc[2] = {0, 0}, UB[9], UBt[9];
        make_ub(fx, grains + 6 * gi, UB);
        make_ub(fx, truth + 6 * gi, UBt);
        for (int64_t i = offsets[gi] + threadIdx.x; i < offsets[gi + 1]; i += blockDim.x) {
            double u, v, ut, vt;
            const bool a = spot_value(fx, e, grains + 6 * gi, UB, sp.iw[i], sp.ih[i], u, v);
            const bool b = spot_value(fx, e, truth + 6 * gi, UBt, sp.iw[i], sp.ih[i], ut, vt);
            if (!(a && b)) continue;
            acc[0] += (u - ut) * (u - ut) + (v - vt) * (v - vt);
            acc[1] += 1.0;
        }
        block_sum<2>(acc, scratch);
        if (threadIdx.x == 0) rms[gi] = acc[1] > 0 ? sqrt(acc[0] / acc[1]) : CUDART_INF;
    }
}

// Cholesky solve of (A + lambda*diag(A)) x = -b for an n x n SPD matrix stored as the upper
// triangle (row-major packing); returns false when the factorisation fails.
template <int N>
__device__ __noinline__ bool lm_solve(const double *upper, const double *b, double lambda, double *x) {
    double M[N][N];
    int q = 0;
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
        for (int c = a; c < N; ++c) {
            M[a][c] = upper[q];
            M[c][a] = upper[q];
            ++q;
        }
    for (int a = 0; a < N; ++a) M[a][a] *= (1.0 + lambda);
    for (int j = 0; j < N; ++j) {
        double d = M[j][j];
        for (int k = 0; k < j; ++k) d -= M[j][k] * M[j][k];
        if (!(d > 0)) return false;
        d = sqrt(d);
        M[j][j] = d;
        for (int i = j + 1; i < N; ++i) {
            double t = M[i][j];
            for (int k = 0; k < j; ++k) t -= M[i][k] * M[j][k];
            M[i][j] = t / d;
        }
    }
    double y[N];
    for (int i = 0; i < N; ++i) {
        double t = -b[i];
        for (int k = 0; k < i; ++k) t -= M[i][k] * y[k];
        y[i] = t / M[i][i];
    }
    for (int i = N - 1; i >= 0; --i) {
        double t = y[i];
        for (int k = i + 1; k < N; ++k) t -= M[k][i] * x[k];
        x[i] = t / M[i][i];
    }
    return true;
}

// One Levenberg-Marquardt iteration of one grain per CTA: the normal equations A = J^T J (21 upper), b =
// J^T r (6), r^T r and the spot count; the damped 6x6 solve; the cost of the trial point; and its
// acceptance where it lowers the cost (lambda /= 10, else lambda *= 10).  A spot that leaves the
// detector counts 1e6 in either cost and nothing in the equations.  Bound by the FP64 chain's latency
// at 12 warps per SM: 650 FP64 instructions per spot, cost included, on accumulators in shared
// memory (in registers: 2 CTAs per SM).  Against dual numbers with 6 tangents in a kernel of their
// own, two cost kernels and the 6 sines and cosines of the tilts per spot: 5,000 grains of 3,100 spots,
// two iterations, 7.87 -> 1.95 ms (2.5 without reading the spot an iteration ahead).
constexpr int kNE6 = 21 + 6 + 2;
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? 3 : 1) grain_lm_k(FitFixed fx, double *grains, const double *geo10, SpotList sp,
                                                      const int64_t *offsets, int64_t n_grains, double *lambda,
                                                      int *improved) {
    extern __shared__ double acc_s[];  // column k of thread t at k * THREADS + t
    __shared__ double scratch[THREADS / 32], s_ne[kNE6];
    __shared__ Beam e;
    __shared__ double s_g[6], s_ub[9];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    bool moved = false;  // thread 0: the step changed a parameter
    if (t == 0) make_beam(geo10, e);
    for (int64_t gi = blockIdx.x; gi < n_grains; gi += gridDim.x) {
        __syncthreads();
        if (threadIdx.x < 6) s_g[threadIdx.x] = grains[6 * gi + threadIdx.x];
        if (threadIdx.x == 0) make_ub(fx, grains + 6 * gi, s_ub);
        __syncthreads();
        const int64_t i0 = offsets[gi], i1 = offsets[gi + 1];
        for (int k = 0; k < kNE6; ++k) acc_s[k * THREADS + t] = 0;
        SpotRef next = load_spot(sp, i0 + t, i1);
        for (int64_t i = i0 + t; i < i1; i += THREADS) {
            double u, v, ju[6], jv[6];
            const SpotRef r = next;
            const double2 cs = fx.rot_cs[r.iw];
            next = load_spot(sp, i + THREADS, i1);
            if (!land_spot<kGrain>(fx, e, s_g, s_ub, cs.x, cs.y, fx.hkl + 3 * r.ih, u, v, ju, jv, false)) continue;
            const double eu = u - r.u, ev = v - r.v;
            int q = 0;
#pragma unroll
            for (int a = 0; a < 6; ++a) {
#pragma unroll
                for (int b = a; b < 6; ++b) acc_s[(q++) * THREADS + t] += ju[a] * ju[b] + jv[a] * jv[b];
                acc_s[(21 + a) * THREADS + t] += ju[a] * eu + jv[a] * ev;
                asm volatile("" ::: "memory");  // one row's accumulators in registers at a time
            }
            acc_s[27 * THREADS + t] += eu * eu + ev * ev;
            acc_s[28 * THREADS + t] += 1.0;
        }
        __syncthreads();
        for (int k = warp; k < kNE6; k += THREADS / 32) {
            double a = 0;
#pragma unroll
            for (int w = 0; w < THREADS; w += 32) a += acc_s[k * THREADS + w + lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
            if (lane == 0) s_ne[k] = a;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double x[6] = {0, 0, 0, 0, 0, 0};
            const bool ok = s_ne[28] >= 6 && lm_solve<6>(s_ne, s_ne + 21, lambda[gi], x);
            moved = false;
            for (int k = 0; k < 6; ++k) {
                const double to = s_g[k] + (ok ? x[k] : 0.0);
                moved |= to != s_g[k];
                s_g[k] = to;
            }
            make_ub(fx, s_g, s_ub);
        }
        __syncthreads();
        const double now = s_ne[27] + 1e6 * ((double)(i1 - i0) - s_ne[28]);
        double cost[1] = {0};
        next = load_spot(sp, i0 + t, i1);
        for (int64_t i = i0 + t; i < i1; i += THREADS) {
            const SpotRef r = next;
            next = load_spot(sp, i + THREADS, i1);
            cost[0] += spot_cost(fx, e, s_g, s_ub, r);
        }
        block_sum<1>(cost, scratch);
        if (threadIdx.x == 0) {
            if (moved && cost[0] < now) {  // the two sums of one point differ by rounding
                for (int k = 0; k < 6; ++k) grains[6 * gi + k] = s_g[k];
                lambda[gi] = fmax(lambda[gi] * 0.1, 1e-9);
                if (now - cost[0] > 1e-9 * now) atomicAdd(improved, 1);
            } else {
                lambda[gi] = fmin(lambda[gi] * 10.0, 1e9);
            }
        }
    }
}

// ---- forward-only baseline: batched Nelder-Mead (fminsearchbnd) ----------------------------
// One CTA per grain.  Parameters live in the sine-transformed space of fminsearchbnd.m:263-265
// (x = lb + (ub - lb)(sin(z) + 1)/2); the simplex follows the standard Nelder-Mead moves
// (reflection 1, expansion 2, contraction 0.5, shrink 0.5; Lagarias et al. 1998 as used by
// fminsearch).  Every objective value is a cooperative sum over the grain's spots.
constexpr int kNM = 6;

__device__ double nm_objective(const FitFixed &fx, const Beam &e, const SpotList &sp, int64_t i0, int64_t i1,
                               const double *z, const double *lb, const double *ub, double *scratch) {
    double x[6], UB[9];
    for (int k = 0; k < kNM; ++k) x[k] = lb[k] + (ub[k] - lb[k]) * (sin(z[k]) + 1.0) * 0.5;
    make_ub(fx, x, UB);
    double acc[1] = {0};
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) acc[0] += spot_cost(fx, e, x, UB, load_spot(sp, i, i1));
    block_sum<1>(acc, scratch);
    __shared__ double s_out;
    if (threadIdx.x == 0) s_out = acc[0];
    __syncthreads();
    const double r = s_out;
    __syncthreads();
    return r;
}

__global__ void grain_nm_k(FitFixed fx, double *grains, const double *geo10, SpotList sp, const int64_t *offsets,
                           int64_t n_grains, const double *half_width, int max_evals, int checkpoint, double *trace,
                           int n_ck) {
    __shared__ double scratch[32];
    __shared__ double simplex[kNM + 1][kNM], fval[kNM + 1];
    __shared__ double lb[kNM], ub[kNM], zr[kNM], ze[kNM], zc[kNM], cen[kNM];
    __shared__ int s_order[kNM + 1];
    __shared__ Beam e;
    if (threadIdx.x == 0) make_beam(geo10, e);
    __syncthreads();
    for (int64_t gi = blockIdx.x; gi < n_grains; gi += gridDim.x) {
        const int64_t i0 = offsets[gi], i1 = offsets[gi + 1];
        if (threadIdx.x < kNM) {
            const double x0 = grains[6 * gi + threadIdx.x];
            lb[threadIdx.x] = x0 - half_width[threadIdx.x];
            ub[threadIdx.x] = x0 + half_width[threadIdx.x];
        }
        __syncthreads();
        // initial simplex in z-space: start at the centre (z = 0), fminsearch's 5% steps
        if (threadIdx.x == 0)
            for (int v = 0; v <= kNM; ++v)
                for (int k = 0; k < kNM; ++k) simplex[v][k] = (v == k + 1) ? 0.05 * 1.5707963267948966 : 0.0;
        __syncthreads();
        int evals = 0, ck = 0;
        for (int v = 0; v <= kNM; ++v) {
            const double f = nm_objective(fx, e, sp, i0, i1, simplex[v], lb, ub, scratch);
            if (threadIdx.x == 0) fval[v] = f;
            ++evals;
        }
        __syncthreads();
        while (evals < max_evals) {
            if (threadIdx.x == 0) {
                for (int v = 0; v <= kNM; ++v) s_order[v] = v;
                for (int a = 1; a <= kNM; ++a)
                    for (int b = a; b > 0 && fval[s_order[b]] < fval[s_order[b - 1]]; --b) {
                        const int t = s_order[b];
                        s_order[b] = s_order[b - 1];
                        s_order[b - 1] = t;
                    }
                for (int k = 0; k < kNM; ++k) {
                    double t = 0;
                    for (int v = 0; v < kNM; ++v) t += simplex[s_order[v]][k];
                    cen[k] = t / kNM;
                    zr[k] = 2.0 * cen[k] - simplex[s_order[kNM]][k];
                }
            }
            __syncthreads();
            const double fr = nm_objective(fx, e, sp, i0, i1, zr, lb, ub, scratch);
            ++evals;
            const int best = s_order[0], worst = s_order[kNM], second = s_order[kNM - 1];
            if (fr < fval[best]) {
                if (threadIdx.x == 0)
                    for (int k = 0; k < kNM; ++k) ze[k] = 3.0 * cen[k] - 2.0 * simplex[worst][k];
                __syncthreads();
                const double fe = nm_objective(fx, e, sp, i0, i1, ze, lb, ub, scratch);
                ++evals;
                if (threadIdx.x == 0) {
                    const double *src = fe < fr ? ze : zr;
                    for (int k = 0; k < kNM; ++k) simplex[worst][k] = src[k];
                    fval[worst] = fe < fr ? fe : fr;
                }
            } else if (fr < fval[second]) {
                if (threadIdx.x == 0) {
                    for (int k = 0; k < kNM; ++k) simplex[worst][k] = zr[k];
                    fval[worst] = fr;
                }
            } else {
                const bool outside = fr < fval[worst];
                if (threadIdx.x == 0)
                    for (int k = 0; k < kNM; ++k)
                        zc[k] = outside ? 1.5 * cen[k] - 0.5 * simplex[worst][k] : 0.5 * cen[k] + 0.5 * simplex[worst][k];
                __syncthreads();
                const double fc = nm_objective(fx, e, sp, i0, i1, zc, lb, ub, scratch);
                ++evals;
                if (fc < (outside ? fr : fval[worst])) {
                    if (threadIdx.x == 0) {
                        for (int k = 0; k < kNM; ++k) simplex[worst][k] = zc[k];
                        fval[worst] = fc;
                    }
                } else {
                    for (int v = 1; v <= kNM; ++v) {  // shrink towards the best vertex
                        const int vi = s_order[v];
                        if (threadIdx.x == 0)
                            for (int k = 0; k < kNM; ++k) simplex[vi][k] = simplex[best][k] + 0.5 * (simplex[vi][k] - simplex[best][k]);
                        __syncthreads();
                        const double f = nm_objective(fx, e, sp, i0, i1, simplex[vi], lb, ub, scratch);
                        ++evals;
                        if (threadIdx.x == 0) fval[vi] = f;
                    }
                }
            }
            __syncthreads();
            // checkpoint: best vertex in parameter space every `checkpoint` evaluations
            while (trace && ck < n_ck && evals >= (ck + 1) * checkpoint) {
                if (threadIdx.x == 0) {
                    int b = 0;
                    for (int v = 1; v <= kNM; ++v)
                        if (fval[v] < fval[b]) b = v;
                    for (int k = 0; k < kNM; ++k)
                        trace[((int64_t)ck * n_grains + gi) * 6 + k] =
                            lb[k] + (ub[k] - lb[k]) * (sin(simplex[b][k]) + 1.0) * 0.5;
                }
                ++ck;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            int b = 0;
            for (int v = 1; v <= kNM; ++v)
                if (fval[v] < fval[b]) b = v;
            for (int k = 0; k < kNM; ++k) grains[6 * gi + k] = lb[k] + (ub[k] - lb[k]) * (sin(simplex[b][k]) + 1.0) * 0.5;
            for (; trace && ck < n_ck; ++ck)
                for (int k = 0; k < kNM; ++k) trace[((int64_t)ck * n_grains + gi) * 6 + k] = grains[6 * gi + k];
        }
        __syncthreads();
    }
}

// ---- geometry fit: normal equations of every start ------------------------------------
// Spots are split across CTAs (blockIdx.x) for start blockIdx.y; partial sums are added
// atomically into the start's 67 accumulators (55 upper J^T J, 10 J^T r, r^T r, n).
constexpr int kNE10 = 55 + 10 + 2;
__global__ void __launch_bounds__(128, 3) geo_normal_k(FitFixed fx, const double *grains, const double *ub,
                                                    const double *starts, SpotList sp, double *ne) {
    // Each thread's 67 accumulators live in shared memory (column k of thread t at k * 128 + t), two
    // spots at a time: one spot's reads and writes of them would be 268 shared-memory cycles per
    // warp, more than its FP64 arithmetic (470 instructions, 235 cycles).  FP64 latency at 12 warps per
    // SM is what is left.  Against 10 tangents of dual numbers and the tilts' sines and cosines per
    // spot: 64 starts x 2.3 M spots 22.8 -> 6.5 ms, the cost of the trial points 4.0 -> 2.5 ms, and
    // the cost of the starts themselves (4.0 ms) comes out of the sums.
    extern __shared__ double acc_s[];
    __shared__ Beam e;
    const int st = blockIdx.y, t = threadIdx.x;
    if (t == 0) make_beam(starts + 10 * st, e);
    for (int k = 0; k < kNE10; ++k) acc_s[k * 128 + t] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    SpotRef next = load_spot(sp, i, sp.n);
    for (; i < sp.n; i += 2 * stride) {
        double ju[2][11], jv[2][11], n = 0;  // the derivatives and, last, the residual
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const SpotRef r = next;
            double u, v, M[9];
            load_ub(fx, grains, ub, r.gi, M);
            const double2 cs = fx.rot_cs[r.iw];
            next = load_spot(sp, i + (b + 1) * stride, sp.n);
            const bool ok = land_spot<kGeometry>(fx, e, grains + 6 * r.gi, M, cs.x, cs.y, fx.hkl + 3 * r.ih, u, v,
                                                 ju[b], jv[b], false) &&
                            i + b * stride < sp.n;
            ju[b][10] = u - r.u;
            jv[b][10] = v - r.v;
            if (ok) {
                n += 1.0;
            } else {
#pragma unroll
                for (int k = 0; k < 11; ++k) ju[b][k] = jv[b][k] = 0.0;
            }
        }
        int q = 0;
#pragma unroll
        for (int a = 0; a < 11; ++a) {
#pragma unroll
            for (int c = a; c < 11; ++c) {
                // rows of the 11 x 11 upper triangle: columns 0..9 are J^T J, column 10 J^T r and r^T r
                const int k = c < 10 ? q++ : a < 10 ? 55 + a : 65;
                acc_s[k * 128 + t] +=
                    ju[0][a] * ju[0][c] + jv[0][a] * jv[0][c] + ju[1][a] * ju[1][c] + jv[1][a] * jv[1][c];
            }
            asm volatile("" ::: "memory");  // one row's accumulators in registers at a time
        }
        acc_s[66 * 128 + t] += n;
    }
    __syncthreads();
    // column sums: warp w sums columns w, w + 4, ...
    const int lane = t & 31, warp = t >> 5;
    for (int k = warp; k < kNE10; k += 4) {
        double v = acc_s[k * 128 + lane] + acc_s[k * 128 + lane + 32] + acc_s[k * 128 + lane + 64] +
                   acc_s[k * 128 + lane + 96];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) atomicAdd(&ne[st * kNE10 + k], v);
    }
}

__global__ void __launch_bounds__(128) geo_cost_k(FitFixed fx, const double *grains, const double *ub,
                                                  const double *starts, SpotList sp, double *cost) {
    __shared__ double scratch[32 * 2];
    __shared__ Beam e;
    const int st = blockIdx.y;
    if (threadIdx.x == 0) make_beam(starts + 10 * st, e);
    __syncthreads();
    double acc[2] = {0, 0};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    SpotRef next = load_spot(sp, i, sp.n);
    for (; i < sp.n; i += stride) {
        const SpotRef r = next;
        double M[9];
        load_ub(fx, grains, ub, r.gi, M);
        next = load_spot(sp, i + stride, sp.n);
        acc[0] += spot_cost(fx, e, grains + 6 * r.gi, M, r);
        acc[1] += 1.0;
    }
    block_sum<2>(acc, scratch);
    if (threadIdx.x == 0) {
        atomicAdd(&cost[2 * st], acc[0]);
        atomicAdd(&cost[2 * st + 1], acc[1]);
    }
}

__global__ void geo_lm_propose_k(const double *starts, const double *ne, const double *lambda, int n,
                                 double *trial) {
    const int st = blockIdx.x * blockDim.x + threadIdx.x;
    if (st >= n) return;
    double x[10];
    for (int k = 0; k < 10; ++k) x[k] = 0;
    const double *e = ne + st * kNE10;
    const bool ok = e[66] >= 10 && lm_solve<10>(e, e + 55, lambda[st], x);
    for (int k = 0; k < 10; ++k) trial[10 * st + k] = starts[10 * st + k] + (ok ? x[k] : 0.0);
}

// Accept the trial where it lowers the cost (lambda /= 10), else keep the point (lambda *= 10).  The
// cost of the point itself is r^T r of its normal equations, and 1e6 for each spot they left out.
__global__ void geo_lm_accept_k(double *starts, const double *trial, const double *ne, int64_t n_spots,
                                const double *cost_trial, double *lambda, int n, int *improved) {
    const int st = blockIdx.x * blockDim.x + threadIdx.x;
    if (st >= n) return;
    const double now = ne[st * kNE10 + 65] + 1e6 * ((double)n_spots - ne[st * kNE10 + 66]);
    bool moved = false;  // the two sums of one point differ by rounding
    for (int k = 0; k < 10; ++k) moved |= trial[10 * st + k] != starts[10 * st + k];
    if (moved && cost_trial[2 * st] < now) {
        for (int k = 0; k < 10; ++k) starts[10 * st + k] = trial[10 * st + k];
        lambda[st] = fmax(lambda[st] * 0.1, 1e-9);
        if (now - cost_trial[2 * st] > 1e-9 * now) atomicAdd(improved, 1);
    } else {
        lambda[st] = fmin(lambda[st] * 10.0, 1e9);
    }
}

// RMS distance of predicted spots between each start's geometry and the true geometry.
__global__ void geo_rms_k(FitFixed fx, const double *grains, const double *ub, const double *starts,
                          const double *truth, SpotList sp, double *acc_out) {
    __shared__ double scratch[32 * 2];
    __shared__ Beam e, et;
    const int st = blockIdx.y;
    if (threadIdx.x == 0) make_beam(starts + 10 * st, e);
    if (threadIdx.x == 32) make_beam(truth, et);
    __syncthreads();
    double acc[2] = {0, 0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < sp.n; i += (int64_t)gridDim.x * blockDim.x) {
        double u, v, ut, vt;
        const double *g6 = grains + 6 * (int64_t)sp.grain[i];
        double M[9];
        load_ub(fx, grains, ub, sp.grain[i], M);
        const bool a = spot_value(fx, e, g6, M, sp.iw[i], sp.ih[i], u, v);
        const bool b = spot_value(fx, et, g6, M, sp.iw[i], sp.ih[i], ut, vt);
        if (!(a && b)) continue;
        acc[0] += (u - ut) * (u - ut) + (v - vt) * (v - vt);
        acc[1] += 1.0;
    }
    block_sum<2>(acc, scratch);
    if (threadIdx.x == 0) {
        atomicAdd(&acc_out[2 * st], acc[0]);
        atomicAdd(&acc_out[2 * st + 1], acc[1]);
    }
}

// ---- synthetic measured spots ---------------------------------------------------------
// Count / fill the selected (omega, hkl) landings of every grain at the given geometry.
__global__ void spots_count_k(FitFixed fx, const double *grains, const double *geo10, int64_t n_grains,
                              int64_t *counts) {
    __shared__ int s_cnt;
    __shared__ Beam e;
    if (threadIdx.x == 0) make_beam(geo10, e);
    for (int64_t gi = blockIdx.x; gi < n_grains; gi += gridDim.x) {
        if (threadIdx.x == 0) s_cnt = 0;
        __syncthreads();
        double UB[9];
        make_ub(fx, grains + 6 * gi, UB);
        int local = 0;
        for (int j = threadIdx.x; j < fx.nrot * fx.nhkl; j += blockDim.x) {
            double u, v;
            if (spot_value(fx, e, grains + 6 * gi, UB, j / fx.nhkl, j % fx.nhkl, u, v, true)) ++local;
        }
        atomicAdd(&s_cnt, local);
        __syncthreads();
        if (threadIdx.x == 0) counts[gi] = s_cnt;
        __syncthreads();
    }
}

__global__ void spots_fill_k(FitFixed fx, const double *grains, const double *geo10, int64_t n_grains,
                             const int64_t *offsets, SpotList sp) {
    __shared__ int s_pos;
    __shared__ Beam e;
    if (threadIdx.x == 0) make_beam(geo10, e);
    for (int64_t gi = blockIdx.x; gi < n_grains; gi += gridDim.x) {
        if (threadIdx.x == 0) s_pos = 0;
        __syncthreads();
        double UB[9];
        make_ub(fx, grains + 6 * gi, UB);
        // ordered fill: chunks of blockDim reflections, warp ballots + a block prefix
        for (int j0 = 0; j0 < fx.nrot * fx.nhkl; j0 += blockDim.x) {
            const int j = j0 + threadIdx.x;
            double u = 0, v = 0;
            const bool ok =
                j < fx.nrot * fx.nhkl && spot_value(fx, e, grains + 6 * gi, UB, j / fx.nhkl, j % fx.nhkl, u, v, true);
            __shared__ int s_warp[32];
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            if (lane == 0) s_warp[warp] = __popc(m);
            __syncthreads();
            int before = 0;
            for (int w = 0; w < warp; ++w) before += s_warp[w];
            if (ok) {
                const int64_t k = offsets[gi] + s_pos + before + __popc(m & ((1u << lane) - 1u));
                sp.grain[k] = (int32_t)gi;
                sp.iw[k] = j / fx.nhkl;
                sp.ih[k] = j % fx.nhkl;
                sp.uv[2 * k] = u;
                sp.uv[2 * k + 1] = v;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                int tot = 0;
                for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_warp[w];
                s_pos += tot;
            }
            __syncthreads();
        }
    }
}

inline int grid_for(int64_t n, int per) {
    int64_t b = (n + per - 1) / per;
    if (b < 1) b = 1;
    if (b > 65535LL * 16) b = 65535LL * 16;
    return (int)b;
}

// CTAs per start of the geometry kernels: every start a share of about 16 waves of 3 CTAs per SM, which
// keeps the sums that meet in one start's accumulators few.
inline int geo_ctas(int64_t n_spots, int n_starts, int num_sms, int per_thread) {
    const int64_t want = ((int64_t)num_sms * 48 + n_starts - 1) / n_starts;
    const int64_t most = grid_for(n_spots, 128 * per_thread);
    return (int)(want < most ? want : most);
}

}  // namespace

cudaError_t fit_grain_ub(const FitFixed &fx, const double *grains, const SpotList &sp, double *ub, cudaStream_t s) {
    grain_ub_k<<<grid_for(sp.n, 256), 256, 0, s>>>(fx, grains, sp, ub);
    return cudaGetLastError();
}

cudaError_t fit_residual_jacobian(const FitFixed &fx, int mode, const double *grains, const double *ub,
                                  const double *geo10, const SpotList &sp, double *res, double *jac, cudaStream_t s) {
    if (mode == 0)
        residual_jac_k<kGrain><<<grid_for(sp.n, kJacThreads), kJacThreads, 0, s>>>(fx, grains, ub, geo10, sp, res, jac);
    else
        residual_jac_k<kGeometry><<<grid_for(sp.n, kJacThreads), kJacThreads, 0, s>>>(fx, grains, ub, geo10, sp, res,
                                                                                    jac);
    return cudaGetLastError();
}

cudaError_t fit_spots_count(const FitFixed &fx, const double *grains, const double *geo10, int64_t n_grains,
                            int64_t *counts, cudaStream_t s) {
    spots_count_k<<<grid_for(n_grains, 1), 256, 0, s>>>(fx, grains, geo10, n_grains, counts);
    return cudaGetLastError();
}

cudaError_t fit_spots_fill(const FitFixed &fx, const double *grains, const double *geo10, int64_t n_grains,
                           const int64_t *offsets, const SpotList &sp, cudaStream_t s) {
    spots_fill_k<<<grid_for(n_grains, 1), 256, 0, s>>>(fx, grains, geo10, n_grains, offsets, sp);
    return cudaGetLastError();
}

cudaError_t fit_grain_lm(const FitFixed &fx, double *grains, const double *geo10, const SpotList &sp,
                         const int64_t *offsets, int64_t n_grains, double *lambda, int *improved, int num_sms,
                         cudaStream_t s) {
    // few grains: more threads each, as the chip is not filled by CTAs of 128
    const bool few = n_grains < 2 * num_sms;
    const size_t smem = sizeof(double) * kNE6 * (few ? 384 : 128);
    cudaError_t e = allow_smem(few ? (const void *)grain_lm_k<384> : (const void *)grain_lm_k<128>, smem);
    if (e != cudaSuccess) return e;
    const int grid = grid_for(n_grains, 1);
    if (few)
        grain_lm_k<384><<<grid, 384, smem, s>>>(fx, grains, geo10, sp, offsets, n_grains, lambda, improved);
    else
        grain_lm_k<128><<<grid, 128, smem, s>>>(fx, grains, geo10, sp, offsets, n_grains, lambda, improved);
    return cudaGetLastError();
}

cudaError_t fit_grain_rms(const FitFixed &fx, const double *grains, const double *truth, const double *geo10,
                          const SpotList &sp, const int64_t *offsets, int64_t n_grains, double *rms, cudaStream_t s) {
    grain_rms_k<<<grid_for(n_grains, 1), 128, 0, s>>>(fx, grains, truth, geo10, sp, offsets, n_grains, rms);
    return cudaGetLastError();
}

cudaError_t fit_grain_nm(const FitFixed &fx, double *grains, const double *geo10, const SpotList &sp,
                         const int64_t *offsets, int64_t n_grains, const double *half_width, int max_evals,
                         int checkpoint, double *trace, int n_ck, cudaStream_t s) {
    grain_nm_k<<<grid_for(n_grains, 1), 128, 0, s>>>(fx, grains, geo10, sp, offsets, n_grains, half_width, max_evals,
                                                     checkpoint, trace, n_ck);
    return cudaGetLastError();
}

cudaError_t fit_geo_normal(const FitFixed &fx, const double *grains, const double *ub, const double *starts,
                           int n_starts, const SpotList &sp, double *ne, int num_sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(ne, 0, sizeof(double) * kNE10 * n_starts, s);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(double) * kNE10 * 128;
    e = allow_smem((const void *)geo_normal_k, smem);
    if (e != cudaSuccess) return e;
    geo_normal_k<<<dim3(geo_ctas(sp.n, n_starts, num_sms, 2), n_starts), 128, smem, s>>>(fx, grains, ub, starts, sp, ne);
    return cudaGetLastError();
}

cudaError_t fit_geo_cost(const FitFixed &fx, const double *grains, const double *ub, const double *starts,
                         int n_starts, const SpotList &sp, double *cost, int num_sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(cost, 0, sizeof(double) * 2 * n_starts, s);
    if (e != cudaSuccess) return e;
    geo_cost_k<<<dim3(geo_ctas(sp.n, n_starts, num_sms, 1), n_starts), 128, 0, s>>>(fx, grains, ub, starts, sp, cost);
    return cudaGetLastError();
}

cudaError_t fit_geo_rms(const FitFixed &fx, const double *grains, const double *ub, const double *starts,
                        int n_starts, const double *truth, const SpotList &sp, double *acc, int num_sms,
                        cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(acc, 0, sizeof(double) * 2 * n_starts, s);
    if (e != cudaSuccess) return e;
    geo_rms_k<<<dim3(geo_ctas(sp.n, n_starts, num_sms, 1), n_starts), 128, 0, s>>>(fx, grains, ub, starts, truth, sp,
                                                                                   acc);
    return cudaGetLastError();
}

cudaError_t fit_geo_lm_propose(const double *starts, const double *ne, const double *lambda, int n, double *trial,
                               cudaStream_t s) {
    geo_lm_propose_k<<<(n + 63) / 64, 64, 0, s>>>(starts, ne, lambda, n, trial);
    return cudaGetLastError();
}

cudaError_t fit_geo_lm_accept(double *starts, const double *trial, const double *ne, int64_t n_spots,
                              const double *cost_trial, double *lambda, int n, int *improved, cudaStream_t s) {
    geo_lm_accept_k<<<(n + 63) / 64, 64, 0, s>>>(starts, trial, ne, n_spots, cost_trial, lambda, n, improved);
    return cudaGetLastError();
}

}  // namespace grc
