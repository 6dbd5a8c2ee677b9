"""Calls at the limit of device memory: host code on the CPU, linked with a runtime that has no device."""
import pytest

from grainrecon_b200 import _lib, synth
from fake_cuda import Fake, code_map


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return Fake(tmp_path_factory.mktemp("fake"))


def scorer(fake, ctx, n):
    """A context with a map, and its forward call of n orientations of one voxel."""
    s = synth.make_sample("fe_tiny", seed=1, detysize=512, detzsize=512)
    ctx.set_geometry(*s.mex_arrays())
    code_map(fake, 3)
    ctx._dev(ctx.L.grc_upload_masks, fake.alloc(4 * 512 * 512 * s.geom.nrot), 512, 512, s.geom.nrot)
    pos, q, out = fake.alloc(12), fake.alloc(16 * n), fake.alloc(16 * n)
    return lambda: ctx.L.grc_forward_comp_device(ctx.h, pos, 1, q, n, out)


def test_a_refused_allocation_is_forgotten(fake):
    """The call after one that found no memory is not charged with its error."""
    fake.reset()
    with fake.context() as ctx:
        call = scorer(fake, ctx, 300)
        fake.limit(fake.used() + 256)
        assert call() == _lib.GRC_ECUDA
        fake.limit(1 << 40)
        assert call() == _lib.GRC_OK


@pytest.mark.parametrize("n,path", [(300, 0), (300, 3), (40000, 0)])
@pytest.mark.parametrize("median", [False, True])
def test_no_room_for_the_packed_mask(fake, n, path, median):
    """Completeness-only calls pack the map, full-output calls list trials for a refine pass; without room for
    that the per-trial kernel takes them, unless another was asked for."""
    fake.reset()
    with fake.context() as ctx:
        call = scorer(fake, ctx, n)
        ctx.set_median(median)
        ctx.set_path(1)
        assert call() == _lib.GRC_OK           # its own buffers
        ctx.set_path(path)
        fake.limit(fake.used() + 256)
        windowed = not median or path == 3 or n > 1776
        if path == 3:
            assert call() == _lib.GRC_ECUDA
        else:
            assert call() == _lib.GRC_OK
            assert ctx.last_stats()["path"] == 1
        fake.limit(1 << 40)
        assert call() == _lib.GRC_OK
        assert ctx.last_stats()["path"] == (3 if windowed else 1)
        assert fake.stray() == 0
