"""Spot pairing at the most reflections a geometry takes (128: the smallest units, one reflection per thread
of their set-up) and around them: the pairs equal the oracle's in order and values."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import seeding as S
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context
from oracle import seed_oracle as SO
from spot_fixtures import measured_spots

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_hkl", [120, 127, 128])
def test_most_reflections(n_hkl):
    nrot = 33
    s = synth.make_sample("fe_tiny", seed=7, rot_angles=np.linspace(0, 357, nrot))
    extra = np.array([h for h in G.gen_hkl(229, 12) if not (s.hkl == h).all(1).any()])
    s.hkl = np.concatenate([s.hkl, extra])[:n_hkl]
    assert len(s.hkl) == n_hkl
    dmap = synth.distance_map(synth.simulate_mask(s))
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    sc = SO.Scene(S9, B9, hkl, rot, R9, p, dmap)
    spots = measured_spots(s, sc, 0.4, 3, spurious=5)
    idx = s.voxel_indices()
    rng = np.random.default_rng(n_hkl)
    pos = s.vol.pos_of_index(idx[rng.choice(len(idx), 6)])
    q = np.concatenate([s.grain_q[:3], s.grain_q[:3]]).astype(np.float64)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        ctx.upload_masks(dmap, s.geom.detzsize, s.geom.detysize, nrot)
        got = S.pair_spots(ctx, pos, q, spots, nrot)
    _, off = S.spot_arrays(spots, nrot)
    clean, last = 0, 0
    for t in range(len(pos)):
        rows, edges = SO.pair_spots(sc, G.quat_to_u(q[t]), pos[t], spots)
        if edges:
            continue
        clean += 1
        mine = got[got["trial"] == t]
        assert [(a["iw"], a["ih"], a["spot"], a["dety"], a["detz"]) for a in mine] == \
            [(iw, ih, off[iw] + j, y, z) for iw, ih, j, y, z, *_ in rows]
        last += sum(ih >= n_hkl - 4 for _, ih, *_ in rows)
    assert clean >= 3 and last > 0
