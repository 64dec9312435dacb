"""The serving loop admits tiles by device bytes that cover what a batch takes:
its state and the inversion's records of depth starts, 64 bytes a start and a
word a pixel up to 1 GiB a call.  No GPU needed."""
import os
import re

import pytest

from photic_gb300 import serve as S

HOST = os.path.join(os.path.dirname(os.path.abspath(S.__file__)), "csrc", "photic_host.cu")
KERNELS = os.path.join(os.path.dirname(HOST), "photic_kernels.h")


def _records(npix, starts):
    """As run_invert sizes them."""
    return min(npix, (1 << 30) // (starts * 64 + 4)) * (starts * 64 + 4)


def test_constants_are_the_library_s():
    assert re.search(r"kRecordBytesMax = 1ll << 30;", open(HOST).read())
    assert re.search(r"kStartRecordBytes = 64;", open(KERNELS).read())
    assert (S.RECORD_BYTES, S.RECORD_BYTES_MAX) == (64, 1 << 30)


@pytest.mark.parametrize("starts", [1, 8, 32])
@pytest.mark.parametrize("sides", [(48,), (256, 300, 1024), (4096,), (4096, 2048, 700)])
def test_footprints_cover_a_batch(sides, starts):
    px = [s * s for s in sides]
    need = sum(px) * S.STATE_BYTES_PER_PIXEL + _records(sum(px), starts)
    assert sum(S.tile_footprint(n, starts) for n in px) >= need


def test_executor_uses_it():
    ex = object.__new__(S.GpuTileExecutor)  # its device side needs a GPU
    ex.cfg = type("Cfg", (), {"hstarts": (40.0, 30.0, 20.0)})()
    for n in (1, 10 ** 6, 10 ** 8):
        assert ex.footprint(n) == S.tile_footprint(n, 3)
