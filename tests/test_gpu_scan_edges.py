"""The warp scan at the edges of its spans: projection counts around 32, 64 and 128, angles in any
order (runs of projections of length one), reflection counts around its slots of 32, and a detector
parallel to the beam, where every FP32 landing is undecided and the FP64 queue fills within a trial.
Every column equals the oracle's on each trial without a tight edge reflection."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(s, n_hkl, seed, min_selected=1, r00=None):
    dmap = synth.distance_map(synth.simulate_mask(s, stride=3))
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    hkl, p, R9 = hkl[:3 * n_hkl], p.copy(), R9.copy()
    if r00 is not None:
        R9[0] = r00
    p[0] = len(hkl) // 3
    idx = s.voxel_indices()
    rng = np.random.default_rng(seed)
    q = np.concatenate([s.grain_q, G.cubic_fz_orientations(300, seed)]).astype(np.float32)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        ctx.upload_masks(dmap, s.geom.detzsize, s.geom.detysize, s.geom.nrot)
        ctx.set_path(3)
        for v in idx[rng.choice(len(idx), 2, replace=False)]:
            pos = s.vol.pos_of_index(v).astype(np.float32)
            ref, _, tight = O.orientation_scan(pos, q, S9, B9, hkl, dmap, rot, R9, p, tight=True)
            ref = ref.reshape(-1, 4)
            ok = tight == 0
            assert ok.sum() > 0.9 * len(q) and ref[:, 0].sum() >= min_selected
            for median in (True, False):
                ctx.set_median(median)
                out = ctx.forward_comp(pos, q, S9, B9, hkl, None, rot, R9, p).reshape(-1, 4)
                assert ctx.last_stats()["path"] == 3
                cols = 4 if median else 3
                np.testing.assert_array_equal(out[ok, :cols], ref[ok, :cols])


@pytest.mark.parametrize("nrot,order", [(1, "up"), (7, "up"), (31, "down"), (32, "up"), (33, "mixed"), (64, "mixed"),
                                        (97, "up"), (127, "down"), (128, "mixed"), (129, "up"), (161, "mixed")])
def test_projection_counts_and_orders(nrot, order):
    a = np.linspace(0, 357.3, nrot)
    a = a if order == "up" else a[::-1].copy() if order == "down" else np.random.default_rng(nrot).permutation(a)
    _check(synth.make_sample("fe_tiny", seed=4, rot_angles=a), 86, nrot)


@pytest.mark.parametrize("n_hkl", [1, 31, 32, 33, 64, 65, 86])
def test_reflection_counts(n_hkl):
    _check(synth.make_sample("fe_tiny", seed=5, rot_angles=np.arange(0, 360, 5.0)), n_hkl, n_hkl)


def test_detector_parallel_to_the_beam():
    s = synth.make_sample("fe_tiny", seed=6, rot_angles=np.arange(0, 360, 4.0))
    s.geom.tilt = (0.0, 0.0, 90.0)
    s.geom.lsd, s.geom.dety00 = 3.0, 8.0
    _check(s, 86, 9, min_selected=1000, r00=0.0)
