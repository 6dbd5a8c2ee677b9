"""The backward derivatives and the fits where the standard sample does not reach: a sample matrix S
that is not the identity (nor exactly orthonormal), spots in mixed grain order, grain numbers beyond
the fits' table of grains, and spot counts around a CTA's.  Against the FP64 complex-step oracle
(1e-9 relative: both are FP64 evaluations of the same derivative, 1e-12 apart at worst)."""
import numpy as np
import pytest

from grainrecon_b200 import fit as F
from grainrecon_b200 import geometry as G
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_spots", [1, 127, 129, 700])
@pytest.mark.parametrize("mode,first_grain", [(0, 0), (1, 0), (0, 24530), (1, 24530)])
def test_jacobian_general(n_spots, mode, first_grain):
    import torch
    s = synth.make_sample("fe_small", seed=3)
    s.S = G.euler_to_u(0.4, 0.7, -0.3) * 1.001
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    geo = F.geo10_of(s.geom) + np.array([0.1, -0.2, 0.3, -0.1, 2.0, -3.0, 1.5, 0.02, -0.03, 0.01])
    few = F.random_grains(80, 0.05, 0.1, seed=5)
    grains = np.zeros((first_grain + 80, 6))
    grains[first_grain:] = few
    rng = np.random.default_rng(n_spots + mode)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        sim = F.simulate_spots(ctx, geo, torch.from_numpy(few.reshape(-1).copy()).cuda(), 0.3, 1)
        pick = torch.from_numpy(rng.choice(sim.n, n_spots, replace=False)).cuda()
        spots = F.Spots((sim.grain[pick] + first_grain).int(), sim.iw[pick].contiguous(), sim.ih[pick].contiguous(),
                        sim.uv.view(-1, 2)[pick].reshape(-1).contiguous(), None)
        d = torch.from_numpy(grains.reshape(-1)).cuda()
        res, jac = (a.cpu().numpy() for a in F.residual_jacobian(ctx, mode, geo, d, spots))
        cost = F.geometry_cost(ctx, torch.from_numpy(geo.copy()).cuda(), d, spots).cpu().numpy()
    g, iw, ih = (a.cpu().numpy() for a in (spots.grain, spots.iw, spots.ih))
    uvm = spots.uv.cpu().numpy().reshape(-1, 2)
    S, B = S9.astype(np.float64), B9.astype(np.float64)
    h3, om, q = hkl.reshape(-1, 3).astype(np.float64), rot.astype(np.float64), p.astype(np.float64)
    want = np.zeros_like(res)
    for i in range(n_spots):
        uv, ju, jv = O.fit_uv_jac(mode, grains[g[i]], geo, S, B, h3[ih[i]], om[iw[i]], q[8], q[9], q[10] / 2 + 0.5,
                                  q[11] / 2 + 0.5)
        want[i] = uv - uvm[i]
        np.testing.assert_allclose(res[i], want[i], rtol=0, atol=1e-9)
        for a, b in ((jac[i, 0], ju), (jac[i, 1], jv)):
            assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max(), (i, a, b)
    np.testing.assert_allclose(cost[0], (want ** 2).sum(), rtol=1e-9)


@pytest.mark.parametrize("n_grains", [1, 5, 295, 297])
def test_grain_steps_at_both_cta_sizes(n_grains):
    """Few and many grains take CTAs of other sizes: the steps are the same and reach the noise floor."""
    import torch
    s = synth.make_sample("fe_small", seed=3)
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    geo = F.geo10_of(s.geom)
    truth = F.random_grains(n_grains, 0.05, 0.1, seed=8)
    with Context(0) as ctx:
        ctx.set_geometry(S9, B9, hkl, rot, R9, p)
        d_truth = torch.from_numpy(truth.reshape(-1).copy()).cuda()
        spots = F.simulate_spots(ctx, geo, d_truth, 0.0, 1)
        d = torch.from_numpy(F.perturb_grains(truth, 0.2, 0.002, 4).reshape(-1).copy()).cuda()
        lam = torch.full((n_grains,), 1e-3, dtype=torch.float64, device="cuda")
        first = F.grains_lm(ctx, geo, d, spots, lam, 1)
        assert first == n_grains
        F.grains_lm(ctx, geo, d, spots, lam, 8)
        rms = F.grains_rms(ctx, geo, d, d_truth, spots).cpu().numpy()
    assert (rms < 1e-6).all()
