"""Which batches one kernel finishes: up to the limit a batch runs without a
closest-hit launch, one row of pixels above it by the wavefront, with the same
sums; the limit grows with the depth limit; and a shallow batch just under the
size up to which deep ones are finished is not slower than the wavefront alone."""
import ctypes
import statistics
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
W = 640


def _path(tmp_path, kind, depth, h, w=W):
    from hastyrenderer_gb300 import scenes
    d = str(tmp_path / f"{kind}_{depth}_{w}x{h}")
    if kind == "cornell":
        return scenes.cornell_box(d, seed=2, width=w, height=h, spp=4, max_depth=depth)
    if kind == "room":
        return scenes.textured_room(d, seed=2, width=w, height=h, spp=4, max_depth=depth, tex_size=32)
    return scenes.sphere_field(d, seed=2, n_spheres=12, width=w, height=h, spp=4, max_depth=depth, env_size=(64, 32))


def _limits(job):
    from hastyrenderer_gb300 import native
    a, b = ctypes.c_int64(), ctypes.c_int64()
    native.check(native.lib().hasty_debug_finish_limits(job._h, ctypes.byref(a), ctypes.byref(b)))
    return a.value, b.value


@pytest.mark.parametrize("kind", ["cornell", "room", "field"])
@pytest.mark.parametrize("depth", [2, 5, 12])
def test_route_at_the_limit(tmp_path, kind, depth):
    from hastyrenderer_gb300 import Context, RenderJob
    with RenderJob(_path(tmp_path, kind, depth, 8)) as probe:
        rows = _limits(probe)[0] // W
    for h, finished in ((1, True), (rows, True), (rows + 1, False)):
        path = _path(tmp_path, kind, depth, h)
        with RenderJob(path) as job, RenderJob(path, Context(0, Context.WAVEFRONT)) as wave:
            for j in (job, wave):
                j.render_passes(1, sync=True)
            assert (job.stats()["trace_launches"] == 0) == finished, h
            assert wave.stats()["trace_launches"] == depth
            assert all(np.array_equal(job.read_sums(a)[0], wave.read_sums(a)[0]) for a in range(3)), h


def test_limit_grows_with_depth(tmp_path):
    from hastyrenderer_gb300 import RenderJob
    for kind in ("cornell", "room", "field"):
        got = []
        for depth in (1, 2, 4, 6, 8, 12, 32):
            with RenderJob(_path(tmp_path, kind, depth, 8)) as job:
                got.append(_limits(job))
        once = [a for a, _ in got]
        assert once == sorted(once) and once[0] < once[-1] and once[0] > 0
        assert len({b for _, b in got}) == 1
        assert once[-1] in (2 * got[0][1], 2 * got[0][1] + 1)


@pytest.mark.parametrize("kind,depth,w,h", [("room", 3, 512, 512), ("cornell", 4, 363, 364)])
def test_shallow_batch_is_not_slower(tmp_path, kind, depth, w, h):
    from hastyrenderer_gb300 import Context, RenderJob
    path = _path(tmp_path, kind, depth, h, w)
    times = [[], []]
    with RenderJob(path) as job, RenderJob(path, Context(0, Context.WAVEFRONT)) as wave:
        for _ in range(40):
            for k, j in enumerate((job, wave)):
                j.reset()
                j.sync()
                t = time.perf_counter()
                j.render_passes(1, sync=True)
                times[k].append(time.perf_counter() - t)
    now, wavefront = (statistics.median(t[10:]) for t in times)
    assert now < 1.1 * wavefront, (now, wavefront)       # 1.2 and 1.4 where one limit holds for all depths
