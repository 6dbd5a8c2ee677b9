// grc_band.h -- where the FP32 landing chain may decide: how far its (u, v) can lie from the FP64
// chain's, as a bound formed once per geometry.  Host code, no CUDA calls.
#pragma once
#include <algorithm>
#include <cmath>

#include "grc_internal.h"

// Narrowest band [pixel] around a half-pixel in which an FP32 landing is recomputed in FP64.
#ifndef GRC_AMBIG_PX
#define GRC_AMBIG_PX 0.004f
#endif

namespace grc {

// Limits of the FP32 chain for one geometry.  A landing further from a half-pixel than the band, from a
// voxel within `reach` of the rotation axis' origin and at a Bragg angle below sin_sure, is decided
// in FP32; any other in FP64.
struct Fp32Limits {
    float half_u, half_v;  // half a pixel less the band; -1: nothing is decided in FP32
    float sin_sure;
    double reach2;         // reach^2 [mm^2], of positions before S
};

// The FP32 error of a landing, in pixels, is a small multiple of 2^-24 times
//   T  the numbers whose difference u is: the row's offset, the ray's term (each with the cancellation in
//      its parts) and the detector's size, and
//   W  the turn of the diffracted ray by 2^-24, seen at the landing: |V|^2 / h for a landing at V from
//      the voxel on a plane at distance h, over cos(theta) (theta from its sine), the incident ray's
//      k_x twice and the sine between G and the x axis (azimuth of G); and what the offset of an
//      oblique incident ray contributes.
// 5 (T + W) 2^-24 is at least 1.1 times the largest error found by restating both FP32 chains (landing_row3,
// landing_fp32) over random geometries: 16 to 10^6 pixels a side, tilts up to 80 degrees, detectors off
// the axis, source distances of 0.25 to 8 times the detector's.  For detectors that face the source
// (audited_shape) the error stays below 0.8 of 2.8 (T + W) 2^-24: 0.0039 px on FCC Al 2048^2 and 0.0034 on BCC
// Fe 1024^2 as benchmarked, where the audit build found no disagreement at half of 0.004 px in 5.8e9
// decisions.  So 0.004 px is the narrowest band, and the one of those two; the Al detector cut into 8,192^2
// pixels takes 0.016 px, 32,768^2 0.063, and from 230,000 a side everything is decided in FP64 (Fe, with its
// larger Bragg angles: 0.007 px at 2,048^2, 0.028 at 8,192^2, all FP64 from 135,000).
inline Fp32Limits fp32_limits(const Geo &g) {
    const Fp32Limits none{-1.0f, -1.0f, 0.0f, 0.0};
    const double pi = 3.14159265358979323846;
    for (int i = 0; i < 3; ++i)  // RotDet has to be a rotation, to two figures, for what follows
        for (int j = 0; j < 3; ++j) {
            const double d = g.R[i] * g.R[j] + g.R[3 + i] * g.R[3 + j] + g.R[6 + i] * g.R[6 + j];
            if (!(std::fabs(d - (i == j)) <= 1e-2)) return none;
        }
    const double lss = std::fabs(g.lss), lsd = std::fabs(g.lsd);
    const double D0[3] = {g.lsd, g.dety00 - g.rao, g.detz00};
    const double h0 = std::fabs(g.R[0] * D0[0] + g.R[3] * D0[1] + g.R[6] * D0[2]);
    const double reach = 0.15 * std::min(std::min(lss, lsd), h0), h = h0 - reach;
    if (!(reach > 0.0)) return none;
    const double axis = std::hypot(g.p0y - g.rao, g.p0z), off = axis + reach;
    const double k0 = (lss - reach) / std::hypot(lss - reach, off), alpha = std::acos(k0);
    if (!(alpha < 70.0 / 180.0 * pi)) return none;
    // sin(theta) up to what the wavelengths reach, and at least 20 degrees between G and the x axis
    double sc = std::min(std::sin(70.0 / 180.0 * pi - alpha), 1.0001 * g.lmax * g.gmax / (4.0 * pi));
    if (g.cbmax > -1.0) sc = std::min(sc, -g.cbmax);
    if (!(sc >= 0.0)) sc = 0.0;
    const double theta = std::asin(sc);
    const double dety[2] = {0.5, g.detysize + 0.5}, detz[2] = {0.5, g.detzsize + 0.5};
    double vmax = 0, vmin = 1e300, xmax = 0, part[3] = {0, 0, 0};
    for (int c = 0; c < 4; ++c) {
        const double y = (g.dety0 - dety[c & 1]) * g.pxy, z = (g.detz0 - detz[c >> 1]) * g.pxz;
        double C[3], v2 = 0;
        for (int i = 0; i < 3; ++i) {
            C[i] = D0[i] + y * g.R[3 * i + 1] + z * g.R[3 * i + 2];
            v2 += C[i] * C[i];
        }
        vmax = std::max(vmax, std::sqrt(v2));
        vmin = std::min(vmin, std::sqrt(v2));
        xmax = std::max(xmax, std::fabs(C[0]));
        for (int o = 0; o < 3; ++o) {
            double s = 0;
            for (int i = 0; i < 3; ++i) s += std::fabs(g.R[3 * i + o]) * (std::fabs(C[i]) + reach);
            part[o] = std::max(part[o], s);
        }
    }
    const double Dy = g.detysize * g.pxy, Dz = g.detzsize * g.pxz;
    const bool audited_shape = axis <= 0.05 * lss && lss >= 0.5 * lsd && vmax <= 1.1 * vmin && Dy <= 2.0 * Dz &&
                               Dz <= 2.0 * Dy && std::max(Dy, Dz) <= 7.0 * lsd && std::fabs(g.R[0]) >= 0.999;
    vmax += reach;
    const double oblique = (xmax + reach) / (lsd - reach) * (off * (lss + lsd) / (lss - reach) + reach);
    const double turn = vmax / h * (vmax / (k0 * k0 * std::cos(theta) * std::cos(theta + alpha)) + oblique);
    double band[2];
    for (int o = 0; o < 2; ++o) {
        const double px = o ? g.pxz : g.pxy, n = o ? g.detzsize : g.detysize;
        const double c0 = o ? g.detz0 : g.dety0;
        const double at = c0 + (D0[0] * g.R[1 + o] + D0[1] * g.R[4 + o] + D0[2] * g.R[7 + o]) / px;
        const double span = std::max(std::fabs(at - 0.5), std::fabs(at - n - 0.5)) + reach / px;
        const double T = part[0] / h * span + part[1 + o] / px + std::fabs(at) + reach / px + n;
        const double e = (audited_shape ? 2.8 : 5.0) * (T + turn / px) / 16777216.0;
        band[o] = GRC_AMBIG_PX * std::max(1.0, e / 0.004);
        if (!(band[o] < 0.45)) return none;
    }
    double s2 = 0;  // of S, the largest column sum of |S^T S|: no less than its squared norm
    for (int i = 0; i < 3; ++i) {
        double sum = 0;
        for (int j = 0; j < 3; ++j) sum += std::fabs(g.S[i] * g.S[j] + g.S[3 + i] * g.S[3 + j] + g.S[6 + i] * g.S[6 + j]);
        s2 = std::max(s2, sum);
    }
    if (!(s2 > 0.0)) return none;
    return {(float)(0.5 - band[0]), (float)(0.5 - band[1]), (float)sc, reach * reach / s2};
}

}  // namespace grc
