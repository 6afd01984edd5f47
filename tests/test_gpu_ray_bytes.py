"""The device memory that a job keeps for a caller's rays is part of the job's
device_bytes (10 words per ray of each of the two lists), and grows only to the
chunk size (2^19 rays)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CHUNK = 1 << 19


def test_ray_lists_are_counted(tmp_path):
    from hastyrenderer_gb300 import RenderJob, scenes
    with RenderJob(scenes.cornell_box(str(tmp_path), width=64, height=64)) as job:
        none = job.info.device_bytes
        rays = np.tile(np.float32([0, 1, 0, 0, 0, 1]), (2 * CHUNK + 1, 1))
        want = {1: 64, 100: 128, 50: 128, CHUNK: CHUNK, CHUNK + 1: 2 * CHUNK, 2 * CHUNK + 1: 2 * CHUNK, 3: 2 * CHUNK}
        for n, kept in want.items():
            job.intersect(rays[:n])
            assert job.info.device_bytes - none == 40 * kept, n
