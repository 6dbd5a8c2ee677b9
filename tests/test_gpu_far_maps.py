"""Lists on maps with far-apart spots: the share of far pixels is counted in the middle 35 % of the
detector, and decides which kernel takes a list of less than half a round; the outputs do not depend
on it."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz,nrot", [(128, 128, 13), (101, 77, 40), (70, 301, 33), (9, 5, 70), (1, 1, 600)])
def test_share_and_kernel(ny, nz, nrot):
    import torch
    s = synth.make_sample("fe_tiny", seed=4, rot_angles=np.linspace(0, 355, nrot), detysize=ny, detzsize=nz, pxy=68.8 / ny,
                          pxz=68.8 / nz)
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    rng = np.random.default_rng(ny)
    shape = (nrot, ny, nz)
    near, far = rng.integers(0, 80, shape) * 0.1, 30.0 + rng.integers(0, 400, shape) * 0.1
    y0, z0 = (ny - -(-ny * 35 // 100)) // 2, (nz - -(-nz * 35 // 100)) // 2
    middle = np.zeros(shape, bool)
    middle[:, y0:y0 + -(-ny * 35 // 100), z0:z0 + -(-nz * 35 // 100)] = True
    half = rng.random(shape)
    n = 400
    q = torch.from_numpy(np.concatenate([s.grain_q, G.cubic_fz_orientations(n, 3)])[:n].astype(np.float64).reshape(-1)).cuda()
    idx = s.voxel_indices()
    pos = torch.from_numpy(np.concatenate([s.vol.pos_of_index(v).reshape(1, 3) for v in idx[rng.integers(0, len(idx), n)]])
                           .astype(np.float64).reshape(-1)).cuda()
    cases = [(np.zeros(shape, bool), 3), (np.ones(shape, bool), 1), (middle, 1), (~middle, 3)]
    if ny > 20:
        cases += [(half < 0.3, 3), (half < 0.5, 1)]
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        for mask, path in cases:
            m = np.where(mask, far, near).astype(np.float32)
            m.reshape(-1)[:175] = -0.01 * np.arange(1, 176)  # with the 80 near ones 255 values below the far
            ctx.upload_masks(m, nz, ny, nrot)
            out = {}
            for force in (0, 1, 3):
                ctx.set_path(force)
                out[force] = torch.empty(4 * n, dtype=torch.float32, device="cuda")
                ctx.score_trials_device(pos, n, q, n, None, None, n, out[force])
                if force == 0:
                    assert ctx.last_stats()["path"] == path, (mask.mean(), path)
            assert torch.equal(out[0].nan_to_num(-1), out[1].nan_to_num(-1))
            assert torch.equal(out[0].nan_to_num(-1), out[3].nan_to_num(-1))
