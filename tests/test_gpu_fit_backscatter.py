"""A reflection straight back along the beam, cos(beta) = -1 to the last bit while G is still not parallel to
the x axis: the landing is the foot of the incident ray, a finite residual and cost."""
import numpy as np
import pytest

from grainrecon_b200 import fit as F
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_residual_straight_back(mode):
    import torch
    s = synth.make_sample("fe_tiny", seed=1)
    s.geom.lss, s.geom.tilt = 16.0, (0.0, 0.0, 0.0)
    S9, _, _, rot, R9, p = s.mex_arrays()
    p[0] = 1
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    grains = torch.tensor([0.0, 0.0, 1e-9, 0.0, 0.0, 0.0], dtype=torch.float64, device="cuda")
    uv = torch.tensor([60.0, 65.25], dtype=torch.float64, device="cuda")
    spots = F.Spots(i32([0]), i32([0]), i32([0]), uv, None)
    geo = F.geo10_of(s.geom)
    with Context(0) as ctx:
        ctx.set_geometry(S9, np.eye(3, dtype=np.float32), np.array([-1.0, 0.0, 0.0], np.float32), rot, R9, p)
        res, _ = F.residual_jacobian(ctx, mode, geo, grains, spots)
        cost = F.geometry_cost(ctx, torch.from_numpy(geo.copy()).cuda(), grains, spots)
    want = np.array([p[10] / 2 + 0.5, p[11] / 2 + 0.5]) - uv.cpu().numpy()
    np.testing.assert_allclose(res.cpu().numpy().reshape(-1), want, rtol=0, atol=1e-9)
    np.testing.assert_allclose(cost.cpu().numpy()[0], (want ** 2).sum(), rtol=1e-9)
