"""Spot pairing where a trial's units end: geometries whose units hold one row or all of them, trials
without any pair among others, more pairs than the buffer holds, and centroids at equal distances
(the first of the list is taken).  The pairs equal the oracle's in order and values; energies agree to
1e-12 (the same FP64 formula, a few ulp)."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import seeding as S
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context
from oracle import seed_oracle as SO
from spot_fixtures import measured_spots

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_hkl,nrot", [(1, 37), (1, 300), (15, 160), (86, 24), (86, 49)])
def test_units(n_hkl, nrot):
    s = synth.make_sample("fe_tiny", seed=7, rot_angles=np.linspace(0, 357, nrot))
    s.hkl = s.hkl[-n_hkl:]
    dmap = synth.distance_map(synth.simulate_mask(s))
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    sc = SO.Scene(S9, B9, hkl, rot, R9, p, dmap)
    g = s.geom
    spots = measured_spots(s, sc, 0.4, 3, spurious=5)
    for k, sp in enumerate(spots):  # pairs of centroids mirrored about a pixel: equal distances
        if len(sp):
            m = sp[:3].copy()
            m[:, :2] = 2 * np.round(m[:, :2]) - m[:, :2]
            spots[k] = np.concatenate([sp, m, sp[:2]])
    idx = s.voxel_indices()
    rng = np.random.default_rng(nrot)
    far = np.array([[9.0, 0.0, 0.0]])  # a trial that lands nothing on the detector's spots
    pos = np.concatenate([s.vol.pos_of_index(idx[rng.choice(len(idx), 5)]), far, s.vol.pos_of_index(idx[:2])])
    q = np.concatenate([s.grain_q[:3], s.grain_q[:3], s.grain_q[:2]]).astype(np.float64)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        ctx.upload_masks(dmap, g.detzsize, g.detysize, g.nrot)
        got = S.pair_spots(ctx, pos, q, spots, g.nrot)
    _, off = S.spot_arrays(spots, g.nrot)
    key = (got["trial"].astype(np.int64) * nrot + got["iw"]) * n_hkl + got["ih"]
    assert (np.diff(key) > 0).all()
    clean = 0
    for t in range(len(pos)):
        rows, edges = SO.pair_spots(sc, G.quat_to_u(q[t]), pos[t], spots)
        mine = got[got["trial"] == t]
        if edges:
            continue
        clean += 1
        assert len(mine) == len(rows)
        for a, (iw, ih, j, dety, detz, ey, ez, area, ekev, dis) in zip(mine, rows):
            assert (a["iw"], a["ih"], a["spot"]) == (iw, ih, off[iw] + j)
            assert (a["dety"], a["detz"], a["exp_y"], a["exp_z"], a["area"]) == (dety, detz, ey, ez, area)
            assert a["dis"] == np.float32(dis)
            np.testing.assert_allclose(a["energy_kev"], ekev, rtol=1e-12)
    assert clean >= 5
