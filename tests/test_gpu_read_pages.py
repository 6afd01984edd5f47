"""An image read into a buffer of which some pages were never touched. The
device waits for each such page (65 us of 64 KB), so the host has them provided
first: reading into a half touched buffer takes the host's faults longer (about
1 ms for 25 MB) than into one with all its pages, not 12 ms. The bytes around the
image's stay as they were, at any alignment."""
import ctypes
import mmap
import statistics
import time

import pytest

pytestmark = pytest.mark.gpu
W, H = 1920, 1080
SIZE, ROOM = W * H * 12, W * H * 12 + (1 << 20)


@pytest.fixture(scope="module")
def job(tmp_path_factory):
    from hastyrenderer_gb300 import RenderJob, scenes
    j = RenderJob(scenes.cornell_box(str(tmp_path_factory.mktemp("read")), seed=1, width=W, height=H, max_depth=4))
    j.render_passes(1, sync=True)
    yield j
    j.close()


def _read(job, offset, touched):
    """A fresh buffer with the first `touched` bytes written; (buffer, ms)."""
    from hastyrenderer_gb300 import native
    region = mmap.mmap(-1, ROOM, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    base = ctypes.addressof(ctypes.c_char.from_buffer(region))
    ctypes.memset(base, 7, touched)
    n = ctypes.c_int32()
    t = time.perf_counter()
    native.check(native.lib().hasty_job_read(job._h, 0, base + offset, W, H, ctypes.byref(n)))
    return region, (time.perf_counter() - t) * 1e3


def test_half_touched_buffer_is_no_slower(job):
    for touched in (ROOM, SIZE // 2):
        _read(job, 0, touched)
    whole = statistics.median(_read(job, 0, ROOM)[1] for _ in range(5))
    half = statistics.median(_read(job, 0, SIZE // 2)[1] for _ in range(5))
    assert half < whole + 4.0, (half, whole)


@pytest.mark.parametrize("offset", [0, 4, 12345 * 4])
def test_only_the_image_is_written(job, offset):
    want = job.compute_estimate().tobytes()
    region, _ = _read(job, offset, SIZE // 2)
    assert region[offset:offset + SIZE] == want
    assert region[:offset] == b"\7" * offset
    assert region[offset + SIZE:] == bytes(ROOM - offset - SIZE)
