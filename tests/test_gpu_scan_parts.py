"""Calls of fewer trials than a tile, where the warp scan cuts its projection windows into parts of 32
or 16 and widens them, and row-per-trial tiles above and below a trial per warp: one voxel with many
orientations, and a list with a voxel per trial.  Every column equals the oracle's on each trial without
a tight edge reflection, and the per-trial kernel's on all of them."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[17, 47, 48, 97, 129, 180])
def scene(request):
    s = synth.make_sample("fe_tiny", seed=7, rot_angles=np.linspace(0, 358, request.param))
    dmap = synth.distance_map(synth.simulate_mask(s, stride=3))
    with Context(0) as ctx:
        S9, B9, hkl, rot, R9, p = s.mex_arrays()
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        ctx.upload_masks(dmap, s.geom.detzsize, s.geom.detysize, s.geom.nrot)
        yield s, dmap, ctx


@pytest.mark.parametrize("n", [1, 149, 443, 445, 3000])
def test_one_voxel(scene, n):
    s, dmap, ctx = scene
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    q = np.concatenate([s.grain_q, G.cubic_fz_orientations(n, n)])[:n].astype(np.float32)
    pos = s.vol.pos_of_index(s.voxel_indices()[n % 50]).astype(np.float32)
    few = min(n, 150)
    ref, _, tight = O.orientation_scan(pos, q[:few], S9, B9, hkl, dmap, rot, R9, p, tight=True)
    ref, ok = ref.reshape(-1, 4), tight == 0
    try:
        for median, cols in ((True, 4), (False, 3)):
            ctx.set_median(median)
            out = {}
            for path in (1, 3, 0):
                ctx.set_path(path)
                out[path] = ctx.forward_comp(pos, q, S9, B9, hkl, None, rot, R9, p).reshape(-1, 4)
                if path:
                    assert ctx.last_stats()["path"] == path
            np.testing.assert_array_equal(out[3][:few][ok, :cols], ref[ok, :cols])
            np.testing.assert_array_equal(out[3], out[1])
            np.testing.assert_array_equal(out[0], out[1])
    finally:
        ctx.set_median(True)
        ctx.set_path(0)


@pytest.mark.parametrize("n", [1, 200, 900, 3600, 12000])
def test_a_voxel_per_trial(scene, n):
    import torch
    s, _, ctx = scene
    rng = np.random.default_rng(n)
    idx = s.voxel_indices()
    vox = idx[rng.integers(0, len(idx), 64)]
    pos = torch.from_numpy(np.concatenate([s.vol.pos_of_index(v) for v in vox]).astype(np.float64)).cuda()
    q = torch.from_numpy(np.concatenate([s.grain_q, G.cubic_fz_orientations(90, 3)])[:90].astype(np.float64).reshape(-1)).cuda()
    tv = torch.from_numpy(rng.integers(0, 64, n).astype(np.int32)).cuda()
    to = torch.from_numpy(rng.integers(0, 90, n).astype(np.int32)).cuda()
    try:
        for median in (True, False):
            ctx.set_median(median)
            out = {}
            for path in (1, 3, 0):
                ctx.set_path(path)
                o = torch.empty(n * 4, dtype=torch.float32, device="cuda")
                ctx.score_trials_device(pos, 64, q, 90, tv, to, n, o)
                out[path] = o.cpu().numpy()
            np.testing.assert_array_equal(out[3], out[1])
            np.testing.assert_array_equal(out[0], out[1])
    finally:
        ctx.set_median(True)
        ctx.set_path(0)
