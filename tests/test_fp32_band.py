"""The limits within which a landing is decided in FP32 (grc_band.h) against the FP32 error itself: both
chains (landing_row3 and landing_fp32) restated in numpy float32, with the reciprocals' rounding drawn at
random, over random geometries.  Every landing that the limits call certain must have the FP64
chain's pixel, and no error may exceed the band.  Landings are drawn uniformly over the detector,
forward and through the ray's extension backwards, from voxels up to the limits' distance."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from grainrecon_b200 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "grc_band.h"
extern "C" void limits(const double *p, const double *R, int ny, int nz, double *out) {
    grc::Geo g{};
    g.lss = p[0], g.lsd = p[1], g.p0y = p[2], g.p0z = p[3], g.dety00 = p[4], g.detz00 = p[5], g.pxy = p[6], g.pxz = p[7];
    g.rao = p[8], g.lmax = p[9], g.gmax = p[10], g.cbmax = p[11];
    g.detysize = ny, g.detzsize = nz, g.dety0 = ny / 2.0 + 0.5, g.detz0 = nz / 2.0 + 0.5;
    for (int i = 0; i < 9; ++i) g.R[i] = R[i], g.S[i] = i % 4 == 0;
    const grc::Fp32Limits l = grc::fp32_limits(g);
    out[0] = l.half_u, out[1] = l.half_v, out[2] = l.sin_sure, out[3] = l.reach2;
}
"""


@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    d = tmp_path_factory.mktemp("band")
    src, lib = d / "band.cpp", d / "band.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "grainrecon_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    fn = C.CDLL(str(lib)).limits

    def call(g):
        p = np.array([g["lss"], g["lsd"], *g["p0"], *g["d00"], *g["px"], g["rao"], 1.0, 4 * np.pi * g["sin"], -2.0])
        R, out = np.ascontiguousarray(g["R"], np.float64).reshape(-1), np.zeros(4)
        dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
        fn(dp(p), dp(R), C.c_int(g["n"][0]), C.c_int(g["n"][1]), dp(out))
        return out
    return call


def rotation(t):
    (cx, sx), (cy, sy), (cz, sz) = [(np.cos(np.radians(a)), np.sin(np.radians(a))) for a in t]
    return (np.array([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]]) @ np.array([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]])
            @ np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]]))


def facing(n, tilt=0.5, sin=0.82):
    """The benchmarks' detector cut into n x n pixels."""
    return dict(lss=11.0, lsd=11.0, p0=(0, 0), d00=(0, 0), n=(n, n), px=(68.8128 / n,) * 2, rao=0.0, sin=sin, R=rotation((tilt, -tilt, tilt)))


def anywhere(rng):
    n = [min(int(2 ** rng.uniform(4, 18)), 10 ** 6) for _ in (0, 1)]
    lsd = 2 ** rng.uniform(0, 8)
    lss = lsd * 2 ** rng.uniform(-2, 3)
    D = lsd * 2 ** rng.uniform(-4, 3.3, 2)
    t = rng.choice([1, 10, 40, 80])
    return dict(lss=lss, lsd=lsd, p0=lss * rng.uniform(-1, 1, 2) * rng.choice([0, 0.05, 0.5]),
                d00=D * rng.uniform(-1, 1, 2) * rng.choice([0, 0.2, 1.5, 5]), n=n, px=D / n,
                rao=rng.uniform(-0.1, 0.1) * lsd * rng.choice([0, 1]), sin=min(1.0, 2 ** rng.uniform(-2.5, 0.2)),
                R=rotation(rng.uniform(-t, t, 3)))


def draw(g, reach, count, rng):
    """Voxels, incident rays and G vectors (laboratory frame) that land uniformly on the detector."""
    R, n, px = g["R"], g["n"], g["px"]
    D0 = np.array([g["lsd"], g["d00"][0] - g["rao"], g["d00"][1]])
    d = rng.normal(size=(count, 3))
    sw = d / np.linalg.norm(d, axis=1)[:, None] * (0.999 * reach * rng.random(count) ** (1 / 3))[:, None]
    w = rng.uniform(0, 2 * np.pi, count)
    u, v = (rng.uniform(0.5, k + 0.5, count) for k in n)
    V = D0 + np.outer((n[0] / 2 + 0.5 - u) * px[0], R[:, 1]) + np.outer((n[1] / 2 + 0.5 - v) * px[1], R[:, 2]) - sw
    K = V / np.linalg.norm(V, axis=1)[:, None]
    K[rng.random(count) > 0.6] *= -1
    p = np.stack([g["lss"] + sw[:, 0], sw[:, 1] - g["p0"][0] + g["rao"], sw[:, 2] - g["p0"][1]], 1)
    k = p / np.linalg.norm(p, axis=1)[:, None]
    G = K - k
    G *= (rng.uniform(0.5, 10, count) / np.linalg.norm(G, axis=1))[:, None]
    return D0, sw, p, k, np.cos(w), np.sin(w), G


def land(g, T, form, state, rng):
    """(u, v, sin theta) of the chain in type T; form 0: landing_row3, 1: landing_fp32."""
    D0, sw, p, k, c, s, G = state
    R, n, px = g["R"], g["n"], g["px"]
    t = lambda a: np.asarray(a).astype(T)
    if T is np.float64:
        rsq, rcp, gw_err = (lambda x: 1 / np.sqrt(x)), (lambda x: 1 / x), lambda: 1.0
    else:
        near = lambda x: (x * (1 + rng.uniform(-1, 1, x.shape) * 2.0 ** -22.9)).astype(T)
        rsq = lambda x: near(1 / np.sqrt(x.astype(np.float64)))
        rcp = lambda x: near(1 / x.astype(np.float64))
        gw_err = lambda: 1 + rng.uniform(-1, 1, len(c)) * 2.0 ** -24
    gw = [t(a * gw_err()) for a in (c * G[:, 0] + s * G[:, 1], -s * G[:, 0] + c * G[:, 1], G[:, 2])]
    cc, ss, kx, ky, kz = t(c), t(s), t(k[:, 0]), t(k[:, 1]), t(k[:, 2])
    ax, L, d = g["lsd"] - sw[:, 0], g["lss"] + g["lsd"], sw - D0
    L2, ay, az = t(ax / k[:, 0]), t(p[:, 1] * L / p[:, 0] - sw[:, 1]), t(p[:, 2] * L / p[:, 0] - sw[:, 2])
    num, cN = t(-(d @ R[:, 0])), t(R[0, 0] * ax)
    at = [t(n[o] / 2 + 0.5 - (d @ R[:, 1 + o]) / px[o]) for o in (0, 1)]
    Gx, Gy, Gz = cc * gw[0] - ss * gw[1], ss * gw[0] + cc * gw[1], gw[2]
    if form == 0:
        dot = kx * Gx + ky * Gy + kz * Gz
    else:
        dot = t(c * k[:, 0] + s * k[:, 1]) * gw[0] + t(-s * k[:, 0] + c * k[:, 1]) * gw[1] + kz * gw[2]
    x = dot * rsq(gw[0] * gw[0] + gw[1] * gw[1] + gw[2] * gw[2])
    x2 = x * x
    q, c2 = 1 - x2, 1 - 2 * x2
    s2, rk = (-2 * x) * (q * rsq(q)), rsq(Gy * Gy + Gz * Gz)
    gy, gz = Gy * rk, Gz * rk
    cph = gy * ky + gz * kz
    r = 1 - cph * cph
    diff = (L2 * s2) * rcp((r * rsq(r)) * c2 - cph * s2)
    Ky, Kz = ay + diff * gy, az + diff * gz
    f = num * rcp(cN + t(R[1, 0]) * Ky + t(R[2, 0]) * Kz)
    out = []
    for o in (0, 1):
        first = t(R[0, 1 + o] / (R[0, 0] * px[o])) * cN if form == 0 else t(R[0, 1 + o] * ax / px[o])
        out.append(at[o] - f * (first + t(R[1, 1 + o] / px[o]) * Ky + t(R[2, 1 + o] / px[o]) * Kz))
    return out[0].astype(np.float64), out[1].astype(np.float64), -x


def check(g, lim, count, rng):
    """Landings compared; asserts that those called certain are right and that errors stay inside the band."""
    half, sure, reach = lim[:2], lim[2], np.sqrt(lim[3])
    state = draw(g, reach, count, rng)
    with np.errstate(all="ignore"):
        exact = land(g, np.float64, 0, state, rng)
        ok = (exact[2] > 0) & (exact[2] < sure)
        for o in (0, 1):
            ok &= (exact[o] > 0.5) & (exact[o] < g["n"][o] + 0.5)
        for form in (0, 1):
            got = land(g, np.float32, form, state, rng)
            certain = ok.copy()
            for o in (0, 1):
                certain &= np.abs(got[o] - np.rint(got[o])) <= half[o]
                assert np.abs(got[o] - exact[o])[ok].max(initial=0) < 0.5 - half[o], (g, form, o)
            for o in (0, 1):
                np.testing.assert_array_equal(np.rint(got[o][certain]), np.rint(exact[o][certain]))
    return int(ok.sum())


@pytest.mark.parametrize("n", [1024, 2048, 4096, 8192, 32768, 65536])
def test_benchmark_shape_cut_into_pixels(limits, n):
    rng = np.random.default_rng(n)
    g = facing(n)
    assert check(g, limits(g), 400000, rng) > 100000


@pytest.mark.parametrize("digits", [2, 3, 5])
def test_rotation_given_to_a_few_digits(limits, digits):
    rng = np.random.default_rng(digits)
    g = facing(2048, tilt=3.0)
    g["R"] = np.round(g["R"], digits)
    lim = limits(g)
    assert lim[0] > 0.48 and check(g, lim, 400000, rng) > 100000


@pytest.mark.parametrize("seed", range(8))
def test_random_geometries(limits, seed):
    rng = np.random.default_rng(seed)
    seen = 0
    for _ in range(60):
        g = anywhere(rng)
        lim = limits(g)
        if lim[0] > 0:
            seen += check(g, lim, 20000, rng) > 500
    assert seen > 10


def test_limits(limits):
    for kind, n in (("al400", 2048), ("fe6", 1024)):  # the benchmarks' band
        geom, _, _, hkl, *_ = synth.named_setup(kind)
        a = {"al400": 4.0495, "fe6": 2.8665}[kind]
        sin = geom.lambda_max * np.linalg.norm(hkl, axis=1).max() / a / 2
        lim = limits(dict(facing(n, sin=sin), R=geom.rot_det))
        np.testing.assert_allclose(lim[:2], 0.496, atol=1e-6)
    assert limits(facing(8192))[0] < 0.487            # a wider band on a finer grid
    assert (limits(facing(10 ** 6))[:2] == -1).all()  # nothing in FP32
    assert limits(dict(facing(1024), R=np.eye(3) * 1.1))[0] == -1   # not a rotation
    assert limits(dict(facing(1024), lss=0.0))[0] == -1
    assert limits(dict(facing(1024), d00=(0, 0), R=rotation((0, 0, 90))))[0] == -1  # plane through the sample
