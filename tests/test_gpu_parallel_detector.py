"""A detector exactly parallel to the beam (RotDet(1,1) = 0) against one whose 1,1 element is a rounding
error: the same landings to FP32, so the same outputs, and decided in FP32 as often: nearly as fast (2
allows for the noise of a short call; with every landing in FP64 it takes four times as long)."""
import numpy as np
import pytest

from grainrecon_b200 import geometry as G
from grainrecon_b200 import synth
from grainrecon_b200._lib import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("median", [True, False])
def test_zero_and_nearly_zero(median):
    import torch
    s = synth.make_sample("fe_tiny", seed=6, rot_angles=np.arange(0, 360, 2.0), detysize=512, detzsize=512, pxy=0.1344, pxz=0.1344)
    s.geom.tilt, s.geom.lsd, s.geom.dety00 = (0.0, 0.0, 90.0), 3.0, 8.0
    S9, B9, hkl, rot, R9, p = s.mex_arrays()
    n = 9218
    q = torch.from_numpy(G.cubic_fz_orientations(n, 3).astype(np.float32).reshape(-1)).cuda()
    pos = torch.from_numpy(s.vol.pos_of_index(s.voxel_indices()[5]).astype(np.float32).reshape(-1)).cuda()
    m = torch.sqrt((torch.arange(512 * 512 * 180, device="cuda") * 2654435761 % 97).float())
    out, ms = {}, {}
    for r00 in (0.0, 6e-17):
        R = R9.copy()
        R[0] = r00
        with Context(0) as ctx:
            ctx.set_geometry(S9, B9, hkl, rot, R, p)
            ctx.upload_masks(m, 512, 512, 180)
            ctx.set_median(median)
            out[r00] = torch.empty(4 * n, device="cuda")
            t = []
            for _ in range(10):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                ctx.forward_comp_device(pos, 1, q, n, out[r00])
                b.record()
                torch.cuda.synchronize()
                t.append(a.elapsed_time(b))
            ms[r00] = min(t)
    assert out[0.0].view(-1, 4)[:, 0].sum() > 1e6
    assert torch.equal(out[0.0].nan_to_num(-1), out[6e-17].nan_to_num(-1))
    assert ms[0.0] < 2 * ms[6e-17], ms
