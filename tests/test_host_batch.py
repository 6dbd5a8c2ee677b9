"""The batched grower after the options changed: kernels get the geometry twice, by value and as the copy in
device memory that the FP64 path reads, and both have to be the present one.  Host code on the CPU, linked
with a runtime that has no device."""
import ctypes as C

import numpy as np
import pytest

from grainrecon_b200 import synth
from fake_cuda import Fake, code_map, pointer


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return Fake(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("entry", ["run", "autotune"])
@pytest.mark.parametrize("n", [100, 400])
def test_the_device_copy_follows_the_options(fake, n, entry):
    fake.reset()
    s = synth.make_sample("fe_tiny", seed=1, detysize=100, detzsize=200)
    seen = []
    with fake.context() as ctx:
        ctx.set_geometry(*s.mex_arrays())
        code_map(fake, 3)
        ctx._dev(ctx.L.grc_upload_masks, fake.alloc(4 * 100 * 200 * s.geom.nrot), 200, 100, s.geom.nrot)

        def launch(name, args):
            if "csr_counts_k" in name:   # one voxel of n candidates
                C.c_int64.from_address(pointer(args, 2)).value = n
            if "scan_kernel" in name or "score_kernel" in name or "sweep_kernel" in name:
                copy = pointer(args, 1)  # ScoreBufs begins with the copy's address
                at = 8 * 9               # dety0, detz0 after nine doubles
                seen.append(tuple((C.c_double * 2).from_address(a + at)[:] for a in (args[0], copy)))
        fake.on_launch(launch)
        h = C.c_void_p()
        rows, ids, euler, out = (fake.alloc(k) for k in (20, 4 * n, 12, 32))
        p1 = np.ones(14, np.float32)
        assert ctx.L.grc_batch_create(ctx.h, rows, 1, ids, n, euler, 1, p1.ctypes.data, C.byref(h)) == 0
        ctx.set_options(dety0=51.25, detz0=99.5)
        if entry == "run":
            assert ctx.L.grc_batch_run(h, out, None) == 0
        else:
            a, b, ms = C.c_int(), C.c_int(), C.c_double()
            assert ctx.L.grc_batch_autotune(h, out, 0, C.byref(a), C.byref(b), C.byref(ms)) == 0
        assert ctx.L.grc_batch_destroy(h) == 0
    assert len(seen) >= 1
    for by_value, copy in seen:
        assert by_value == [51.25, 99.5] and copy == by_value
