"""The two ways in which the photon gather finds a column's photons, the table of
cell starts and the search in the list of occupied cells: that each run takes the
one asked for, also for frames of a few pixels, and the same image to the bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,w,h", [("room", 17, 13), ("cornell", 1, 1), ("cornell", 33, 31), ("room", 96, 64)])
def test_each_run_takes_the_lookup_asked_for(tmp_path, kind, w, h):
    from hastyrenderer_gb300 import RenderJob, native, scenes
    if kind == "room":
        path = scenes.textured_room(str(tmp_path), seed=5, width=w, height=h, spp=4, max_depth=8, tex_size=32)
    else:
        path = scenes.cornell_box(str(tmp_path), width=w, height=h)
    used = ctypes.c_int32(-1)
    with RenderJob(path) as job:
        runs = []
        for cells, want in ((1 << 24, 1), (0, 0)):
            native.check(native.lib().hasty_debug_pm_table(job._h, cells))
            job.pm_reset()
            for _ in range(3):
                job.pm_render(1)
                bounds = job.pm_map()["cells"][:, :3]
                native.check(native.lib().hasty_debug_pm_table_used(job._h, ctypes.byref(used)))
                if len(bounds):          # no photons, no table
                    n = np.prod(bounds.max(0).astype(np.int64) - bounds.min(0) + 1)
                    assert used.value == (want if n <= 1 << 24 else 0), (cells, n)
            runs.append([job.pm_radii()] + [job.pm_read(a) for a in range(3)])
        assert all(np.array_equal(a, b) for a, b in zip(*runs))
