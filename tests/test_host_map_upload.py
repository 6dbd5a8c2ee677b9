"""What the context holds after a map upload that fails, is refused or is empty: host code on the CPU,
linked with a runtime that has no device."""
import ctypes as C

import pytest

from grainrecon_b200 import _lib
from fake_cuda import Fake, code_map


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return Fake(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def ctx(fake):
    fake.reset()
    code_map(fake, 3)
    with fake.context() as c:
        c._dev(c.L.grc_upload_masks, fake.alloc(4 * 64 * 32 * 2), 64, 32, 2)
        yield c


def resident(ctx):
    """(distinct values, detz, dety, projections) of the resident map, or None."""
    n, bits, d = C.c_int64(), C.c_int(), [C.c_int64() for _ in range(3)]
    rc = ctx.L.grc_mask_info(ctx.h, C.byref(n), C.byref(bits), *[C.byref(a) for a in d])
    if rc == _lib.GRC_ENOMASK:
        return None
    assert rc == _lib.GRC_OK
    return (n.value, *[a.value for a in d])


@pytest.mark.parametrize("at,left", [("mark_halves_k", True), ("mark_values_k", True), ("8values_k", False),
                                     ("codes_k", False)])
def test_a_failed_upload_leaves_a_whole_map_or_none(fake, ctx, at, left):
    """The buffers of the map before are reused: once they are written, its codes are gone."""
    assert resident(ctx) == (3, 64, 32, 2)
    fake.fail(at, 0, 719)
    d = fake.alloc(4 * 64 * 32 * 2)
    assert ctx.L.grc_upload_masks(ctx.h, d, 32, 64, 2) == _lib.GRC_ECUDA
    assert resident(ctx) == ((3, 64, 32, 2) if left else None)
    fake.reset()
    code_map(fake, 5)
    ctx._dev(ctx.L.grc_upload_masks, d, 32, 64, 2)
    assert resident(ctx) == (5, 32, 64, 2)
    assert fake.stray() == 0


@pytest.mark.parametrize("dims", [(0, 32, 2), (64, 0, 2), (64, 32, 0), (-5, 1, 1), (-1, -1, -3)])
def test_an_empty_device_map(fake, ctx, dims):
    """Accepted by grc_upload_masks as a map without values; nothing is read or copied for it."""
    fake.reset()
    d = fake.alloc(64)
    assert ctx.L.grc_upload_masks(ctx.h, d, *dims) == _lib.GRC_OK
    assert fake.stray() == 0 and fake.launched() == []
    assert resident(ctx) == (0, *dims)
    code_map(fake, 4)
    ctx._dev(ctx.L.grc_upload_masks, fake.alloc(4 * 64 * 32 * 2), 64, 32, 2)
    assert resident(ctx) == (4, 64, 32, 2)
