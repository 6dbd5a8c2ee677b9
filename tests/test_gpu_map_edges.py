"""Distance transform and rank coding at the edges of their kernels: widths around the 32-pixel words
and the 1,024-pixel rows of a warp, heights around the searched rows, the detectors beyond the strip
kernel, projections without spots; maps with negative, infinite and very many values, device maps at
odd addresses, and uploads that reuse the buffers of another map.  Distances equal scipy's rounded
to float32 exactly (squares below 2^24 are exact in float32, the square root is correctly rounded)."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context, GrcError, GRC_EINVAL
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,ny", [(1, 1), (1, 40), (31, 9), (32, 8), (33, 7), (64, 17), (95, 1), (1000, 65), (1024, 16),
                                   (1025, 33), (2080, 24), (40, 1030), (24, 2047), (40, 4001)])
def test_distance_transform_sizes(nz, ny):
    import torch
    from scipy.ndimage import distance_transform_edt
    rng = np.random.default_rng(nz * 7 + ny)
    mask = np.zeros((6, ny, nz), np.uint8)
    mask[1] = rng.random((ny, nz)) < 0.3
    mask[2] = rng.random((ny, nz)) < 2.0 / (ny * nz)
    mask[3, ny // 2, nz - 1] = 7
    mask[4, 0, 0] = mask[4, -1, -1] = 255
    mask[5] = 1
    d_mask = torch.from_numpy(mask.reshape(-1).copy()).cuda()
    d_map = torch.empty(mask.size, dtype=torch.float32, device="cuda")
    with Context(0) as ctx:
        ctx.edt(d_mask, nz, ny, 6, d_map)
    got = d_map.cpu().numpy().reshape(mask.shape)
    for i in range(6):
        want = (np.sqrt(np.round(distance_transform_edt(mask[i] == 0) ** 2).astype(np.float32)) if mask[i].any()
                else np.full((ny, nz), np.inf, np.float32))
        np.testing.assert_array_equal(got[i], want)


def _scan(ctx, s, q, pos):
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    return ctx.forward_comp(pos, q, S9, B9, hkl, None, rot, R9, p).reshape(-1, 4)


def test_coding_of_odd_maps_and_reused_buffers():
    import torch
    s = synth.make_sample("fe_tiny", seed=4)
    g = s.geom
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    shape = (g.nrot, g.detysize, g.detzsize)
    rng = np.random.default_rng(3)
    base = synth.distance_map(synth.simulate_mask(s))
    odd = base.copy()
    odd.reshape(-1)[::97] = -0.0
    odd.reshape(-1)[5::101] = -3.5
    odd.reshape(-1)[7::103] = np.inf
    odd.reshape(-1)[9::107] = -np.inf
    many = rng.normal(size=shape).astype(np.float32) * np.float32(3.0)     # nearly all distinct: 32-bit codes
    huge = np.exp(rng.uniform(-80, 80, shape)).astype(np.float32)          # thousands of upper halves
    q = np.concatenate([s.grain_q, G.cubic_fz_orientations(60, 3)]).astype(np.float32)
    pos = s.vol.pos_of_index(s.voxel_indices()[11]).astype(np.float32)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        for path in (1, 3):
            ctx.set_path(path)
            for m in (base, many, odd, huge, base):
                for shift in (0, 1):
                    d = torch.empty(m.size + 4, dtype=torch.float32, device="cuda")[shift:shift + m.size]
                    d.copy_(torch.from_numpy(m.reshape(-1)))
                    ctx.upload_masks(d, g.detzsize, g.detysize, g.nrot)
                    assert ctx.mask_info()["n_distinct"] == len(np.unique(m))
                    ref, _, tight = O.orientation_scan(pos, q, S9, B9, hkl, m, rot, R9, p, tight=True)
                    out = _scan(ctx, s, q, pos)
                    np.testing.assert_array_equal(out[tight == 0], ref.reshape(-1, 4)[tight == 0])
        # a refused map leaves the resident one in place
        bad = base.copy()
        bad[0, 3, 4] = np.nan
        with pytest.raises(GrcError) as e:
            ctx.upload_masks(torch.from_numpy(bad.reshape(-1)).cuda(), g.detzsize, g.detysize, g.nrot)
        assert e.value.code == GRC_EINVAL
        np.testing.assert_array_equal(_scan(ctx, s, q, pos), out)
