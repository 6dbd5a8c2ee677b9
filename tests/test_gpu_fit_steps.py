"""Levenberg-Marquardt steps that go nowhere: with fewer spots than parameters, or a step too short to change
a parameter, the trial point is the point itself.  It is never taken for an improvement: the parameters stay and lambda grows tenfold, whatever
the rounding of the two costs."""
import numpy as np
import pytest

from grainrecon_b200 import fit as F
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context

pytestmark = pytest.mark.gpu


def scene(ctx, n_grains):
    import torch
    s = synth.make_sample("fe_small", seed=3)
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    ctx.set_geometry(S9, B9, hkl, rot, R9, p)
    geo = F.geo10_of(s.geom)
    grains = torch.from_numpy(F.random_grains(n_grains, 0.05, 0.1, seed=5).reshape(-1).copy()).cuda()
    return geo, grains, F.simulate_spots(ctx, geo, grains, 2.0, 1)


@pytest.mark.parametrize("n_grains", [40, 400])
@pytest.mark.parametrize("iters", [1, 3])
def test_grains_of_few_spots(n_grains, iters):
    import torch
    with Context(0) as ctx:
        geo, grains, spots = scene(ctx, n_grains)
        off = spots.offsets.cpu().numpy()
        count = np.arange(n_grains) % 6
        pick = torch.from_numpy(np.concatenate([off[g] + np.arange(c) for g, c in enumerate(count)])).cuda()
        few = F.Spots(spots.grain[pick].contiguous(), spots.iw[pick].contiguous(), spots.ih[pick].contiguous(),
                      spots.uv.view(-1, 2)[pick].reshape(-1).contiguous(),
                      torch.from_numpy(np.concatenate([[0], np.cumsum(count)])).cuda())
        lam = torch.full((n_grains,), 1e-3, dtype=torch.float64, device="cuda")
        before = grains.clone()
        F.grains_lm(ctx, geo, grains, few, lam, iters)
        assert torch.equal(grains, before)
        assert (lam.cpu().numpy() == 1e-3 * 10.0).all()


@pytest.mark.parametrize("n_grains", [40, 400])
def test_grain_steps_too_short(n_grains):
    """At the minimum, damped by 1e9: the steps of most grains are below the parameters' resolution."""
    import torch
    with Context(0) as ctx:
        geo, grains, spots = scene(ctx, n_grains)
        lam = torch.full((n_grains,), 1e-3, dtype=torch.float64, device="cuda")
        F.grains_lm(ctx, geo, grains, spots, lam, 30)
        lam.fill_(1e9)
        before = grains.clone()
        F.grains_lm(ctx, geo, grains, spots, lam, 1)
        same = (grains == before).view(n_grains, 6).all(1)
        assert same.any()
        assert (lam[same] == 1e9).all()


def test_geometry_steps_too_short():
    import torch
    with Context(0) as ctx:
        geo, grains, spots = scene(ctx, 40)
        starts = torch.from_numpy(np.tile(geo, 64) + np.repeat(np.arange(64), 10) * 1e-3).cuda()
        lam = torch.full((64,), 1e-3, dtype=torch.float64, device="cuda")
        F.geometry_lm(ctx, starts, grains, spots, lam, 30)
        lam.fill_(1e9)
        before = starts.clone()
        F.geometry_lm(ctx, starts, grains, spots, lam, 1)
        same = (starts == before).view(64, 10).all(1)
        assert (lam[same] == 1e9).all()


@pytest.mark.parametrize("n_spots", [1, 5, 9])
def test_geometry_of_few_spots(n_spots):
    import torch
    with Context(0) as ctx:
        geo, grains, spots = scene(ctx, 40)
        few = F.Spots(*[a[:n_spots].contiguous() for a in (spots.grain, spots.iw, spots.ih)],
                      spots.uv[:2 * n_spots].contiguous(), None)
        rng = np.random.default_rng(n_spots)
        starts = torch.from_numpy((geo + rng.normal(size=(64, 10)) * [0.1, 0.1, 0.2, 0.2, 0.3, 0.3, 0.3, 0.02, 0.02, 0.01])
                                  .reshape(-1)).cuda()
        lam = torch.full((64,), 1e-3, dtype=torch.float64, device="cuda")
        before = starts.clone()
        F.geometry_lm(ctx, starts, grains, few, lam, 1)
        assert torch.equal(starts, before)
        assert (lam.cpu().numpy() == 1e-3 * 10.0).all()
