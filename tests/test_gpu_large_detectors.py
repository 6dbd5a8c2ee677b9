"""Scoring and pairing on detectors of many pixels, where an FP32 landing is off by more than the narrow
band of the benchmark sizes: the 68.8 mm detector of the samples cut into 8,192 to 10^6 pixels along
dety.  The map's values differ between neighbouring pixels, so a wrong pixel shows in the counts, the
median and the pairs.  Every column equals the oracle's on each trial without a tight edge."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import seeding as S
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context
from oracle import oracle as O
from oracle import seed_oracle as SO

pytestmark = pytest.mark.gpu

WIDE = 68.8128


@pytest.fixture(scope="module", params=[(8192, 96, 24, 0.4), (32768, 48, 12, 0.4), (262144, 16, 6, 0.0),
                                        (16, 1000000, 3, 0.3)])
def scene(request):
    ny, nz, nrot, tilt = request.param
    s = synth.make_sample("fe_tiny", seed=11, rot_angles=np.linspace(3, 350, nrot), detysize=ny, detzsize=nz,
                          pxy=WIDE / ny, pxz=WIDE / nz, tilt=(tilt, -tilt, tilt / 2))
    iw, y, z = np.ogrid[:nrot, :ny, :nz]
    dmap = (((7 * y + 3 * z + iw) % 5) * 0.4).astype(np.float32)
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        ctx.upload_masks(dmap, nz, ny, nrot)
        yield s, dmap, ctx


def test_scores(scene):
    s, dmap, ctx = scene
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    q = np.concatenate([s.grain_q, G.cubic_fz_orientations(1500, 5)]).astype(np.float32)
    pos = s.vol.pos_of_index(s.voxel_indices()[7]).astype(np.float32)
    ref, _, tight = O.orientation_scan(pos, q, S9, B9, hkl, dmap, rot, R9, p, tight=True)
    ref, ok = ref.reshape(-1, 4), tight == 0
    assert ok.sum() > 0.9 * len(q) and ref[:, 0].sum() > 10000
    try:
        for path in (1, 2, 3):
            ctx.set_path(path)
            for median, cols in ((True, 4), (False, 3)):
                ctx.set_median(median)
                out = ctx.forward_comp(pos, q, S9, B9, hkl, None, rot, R9, p).reshape(-1, 4)
                np.testing.assert_array_equal(out[ok, :cols], ref[ok, :cols])
    finally:
        ctx.set_median(True)
        ctx.set_path(0)


def test_pairs(scene):
    s, dmap, ctx = scene
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    sc = SO.Scene(S9, B9, hkl, rot, R9, p, dmap)
    rng = np.random.default_rng(2)
    idx = s.voxel_indices()
    pos = s.vol.pos_of_index(idx[rng.choice(len(idx), 24)])
    q = G.cubic_fz_orientations(24, 9).astype(np.float64)
    spots = [[] for _ in rot]
    for t in range(24):  # a spot a little off every landing
        rec, _ = O.landings(G.quat_to_u(q[t]), pos[t], sc.S9, sc.B9, sc.hkl, sc.dmap, sc.rot, sc.R9, sc.param)
        for j in np.nonzero(rec["sel"])[0]:
            spots[rec["iw"][j]].append((rec["u"][j] + rng.uniform(-2, 2), rec["v"][j] + rng.uniform(-2, 2), 60.0))
    spots = [np.array(a, np.float64).reshape(-1, 3) for a in spots]
    got = S.pair_spots(ctx, pos, q, spots, s.geom.nrot)
    _, off = S.spot_arrays(spots, s.geom.nrot)
    clean = pairs = 0
    for t in range(24):
        rows, edges = SO.pair_spots(sc, G.quat_to_u(q[t]), pos[t], spots)
        if edges:
            continue
        clean += 1
        pairs += len(rows)
        mine = got[got["trial"] == t]
        assert [(a["iw"], a["ih"], a["spot"], a["dety"], a["detz"], a["dis"]) for a in mine] == \
            [(iw, ih, off[iw] + j, y, z, np.float32(d)) for iw, ih, j, y, z, _, _, _, _, d in rows]
    assert clean >= 12 and pairs > 300


def test_voxels_beyond_the_fp32_reach():
    """Voxels near the axis and 2.6 mm off it (a quarter of the distances) in turn, in one call."""
    import torch
    s = synth.make_sample("fe_small", seed=3)
    dmap = synth.distance_map(synth.simulate_mask(s, stride=3))
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    near = s.vol.pos_of_index(s.voxel_indices()[5]).reshape(3)
    vox = np.stack([near, np.array([2.0, -1.5, 0.8])]).astype(np.float32)
    q = np.concatenate([s.grain_q, G.cubic_fz_orientations(194, 3)]).astype(np.float32)
    n = 4 * len(q)
    tv, to = (np.arange(n) % 2).astype(np.int32), (np.arange(n) // 2 % len(q)).astype(np.int32)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        ctx.upload_masks(dmap, s.geom.detzsize, s.geom.detysize, s.geom.nrot)
        ref = [O.orientation_scan(v, q, S9, B9, hkl, dmap, rot, R9, p, tight=True) for v in vox]
        want = np.stack([r[0].reshape(-1, 4) for r in ref])[tv, to]
        ok = np.stack([r[2] == 0 for r in ref])[tv, to]
        assert ok.mean() > 0.9
        d = [torch.from_numpy(a).cuda() for a in (vox.astype(np.float64), q.astype(np.float64).reshape(-1), tv, to)]
        for path in (1, 2, 3):
            ctx.set_path(path)
            out = torch.empty(4 * n, dtype=torch.float32, device="cuda")
            ctx.score_trials_device(d[0], 2, d[1], len(q), d[2], d[3], n, out)
            np.testing.assert_array_equal(out.cpu().numpy().reshape(-1, 4)[ok], want[ok])
