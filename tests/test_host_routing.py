"""Which kernel grc_set_path(ctx, 0) takes, on both sides of each line of the rule: host code on the CPU,
linked with a runtime that has no device (148 SMs: a round of the sweep is 28,416 trials, two rounds of
the warp scan 56,832)."""
import ctypes as C

import numpy as np
import pytest

from grainrecon_b200 import synth
from fake_cuda import Fake, code_map, pointer

SMS, HALF, SIXTEENTH, TWO_ROUNDS = 148, 14208, 1776, 56832


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return Fake(tmp_path_factory.mktemp("fake"))


def scorer(fake, ctx, nrot, n_hkl, far):
    """A geometry of nrot x n_hkl pairs and a map whose middle has `far` of its pixels beyond the 8-bit codes."""
    fake.reset()
    s = synth.make_sample("fe_tiny", seed=1, rot_angles=np.linspace(0, 350, nrot), detysize=100, detzsize=200)
    s.hkl = s.hkl[:n_hkl]
    ctx.set_geometry(*s.mex_arrays())
    code_map(fake, 3)
    keep = fake._keep
    seen = 35 * 70 * min(nrot, -(-nrot // -(-nrot // 32)))

    def launch(name, args):
        keep(name.encode(), args)
        if "far_share_k" in name:
            C.c_int.from_address(pointer(args, 4)).value = round(far * seen)
    fake.on_launch(launch)
    ctx._dev(ctx.L.grc_upload_masks, fake.alloc(4 * 100 * 200 * nrot), 200, 100, nrot)


def path(fake, ctx, kind, n, median):
    ctx.set_median(median)
    a, b, out = fake.alloc(24 * n), fake.alloc(32 * n), fake.alloc(32 * n)
    if kind == "voxel":
        ctx.forward_comp_device(a, 1, b, n, out)
    elif kind == "voxels":      # 100 orientations each
        ctx.forward_comp_device(a, n // 100, b, 100, out)
    elif kind == "few":         # 63 orientations each: a list
        ctx.forward_comp_device(a, n // 63, b, 63, out)
    elif kind == "grow":
        ctx.grow_device(a, n, np.eye(3), np.zeros(14), out)
    elif kind == "trials":
        ctx.score_trials_device(a, n, b, n, None, None, n, out)
    elif kind == "indexed":
        ctx.score_trials_device(a, n, b, n, fake.alloc(4 * n), fake.alloc(4 * n), n, out)
    assert ctx.last_stats()["trials"] > 0
    return ctx.last_stats()["path"]


@pytest.mark.parametrize("kind", ["grow", "trials", "indexed", "few"])
@pytest.mark.parametrize("far,start", [(0.0, SMS), (0.39, SMS), (0.42, HALF), (1.0, HALF)])
def test_lists_with_medians(fake, kind, far, start):
    with fake.context() as ctx:
        scorer(fake, ctx, 61, 86, far)
        step = 63 if kind == "few" else 1
        first = -(-start // step) * step
        assert path(fake, ctx, kind, first - step, True) == 1
        assert path(fake, ctx, kind, first, True) == 3
        assert path(fake, ctx, kind, TWO_ROUNDS + 6300, True) == 3


@pytest.mark.parametrize("far", [0.0, 1.0])
@pytest.mark.parametrize("kind,step", [("voxel", 1), ("voxels", 100)])
def test_scans_with_medians(fake, far, kind, step):
    with fake.context() as ctx:
        scorer(fake, ctx, 61, 86, far)
        first = -(-SIXTEENTH // step) * step
        assert path(fake, ctx, kind, first - step, True) == 1
        assert path(fake, ctx, kind, first, True) == 3
        assert path(fake, ctx, kind, TWO_ROUNDS + 100, True) == 3


@pytest.mark.parametrize("kind", ["voxel", "trials", "indexed"])
@pytest.mark.parametrize("far", [0.0, 1.0])
def test_completeness_only(fake, kind, far):
    with fake.context() as ctx:
        scorer(fake, ctx, 61, 86, far)
        assert [path(fake, ctx, kind, n, False) for n in (SMS - 1, SMS, TWO_ROUNDS + 1)] == [1, 3, 3]


@pytest.mark.parametrize("nrot,n_hkl,long", [(59, 84, 2), (61, 82, 3), (37, 64, 2), (100, 50, 3)])
def test_long_calls_by_pairs(fake, nrot, n_hkl, long):
    """4,956 and 5,002 pairs: the sweep for full-output calls of more than two rounds, or the scan."""
    with fake.context() as ctx:
        scorer(fake, ctx, nrot, n_hkl, 0.0)
        for kind in ("voxel", "trials"):
            assert [path(fake, ctx, kind, n, True) for n in (TWO_ROUNDS, TWO_ROUNDS + 1)] == [3, long]
            assert path(fake, ctx, kind, TWO_ROUNDS + 1, False) == 3


def test_batches(fake):
    """The batched grower without a tuned tile follows the rule of lists."""
    with fake.context() as ctx:
        for far, first in ((0.0, SMS), (1.0, HALF)):
            scorer(fake, ctx, 61, 86, far)
            base = fake._keep
            for n, kernel in ((first - 1, "score_kernel"), (first, "scan_kernel")):
                def launch(name, args, n=n):
                    base(name.encode(), args)
                    if "csr_counts_k" in name:   # one voxel of n candidates
                        C.c_int64.from_address(pointer(args, 2)).value = n
                fake.on_launch(launch)
                h = C.c_void_p()
                rows, ids, euler, out = (fake.alloc(k) for k in (20, 4 * n, 12, 32))
                p1 = np.ones(14, np.float32)
                assert ctx.L.grc_batch_create(ctx.h, rows, 1, ids, n, euler, 1, p1.ctypes.data, C.byref(h)) == 0
                before = len(fake.launched())
                assert ctx.L.grc_batch_run(h, out, None) == 0
                ran = " ".join(fake.launched()[before:])
                assert kernel in ran, (far, n, ran)
                assert ctx.L.grc_batch_destroy(h) == 0
            fake.on_launch(lambda name, args: 0)
