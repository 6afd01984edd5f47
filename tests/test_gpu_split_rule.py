"""Into how many batches a call is cut, from the job's closest-hit launches (one
per bounce and batch): two from 1M samples of a scene with a tiny BVH; of others
up to depth 12 from 2M, or from 6M where there are area lights and the depth is 10
or more; one otherwise. The sums are those of single passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIDE = 256


@pytest.mark.parametrize("kind,depth,passes,batches", [
    ("cornell", 8, 15, 1), ("cornell", 8, 16, 2), ("cornell", 30, 17, 2),
    ("field", 12, 31, 1), ("field", 12, 32, 2), ("field", 13, 96, 1), ("room", 9, 31, 1), ("room", 9, 32, 2),
    ("room", 10, 32, 1), ("room", 12, 95, 1), ("room", 12, 96, 2)])
def test_batches_of_a_call(tmp_path, kind, depth, passes, batches):
    from hastyrenderer_gb300 import RenderJob, scenes
    if kind == "cornell":
        path = scenes.cornell_box(str(tmp_path), seed=3, width=SIDE, height=SIDE, max_depth=depth)
    elif kind == "room":
        path = scenes.textured_room(str(tmp_path), seed=3, width=SIDE, height=SIDE, max_depth=depth, tex_size=32)
    else:
        path = scenes.sphere_field(str(tmp_path), seed=3, n_spheres=20, subdiv=2, width=SIDE, height=SIDE, max_depth=depth,
                                   env_size=(256, 128))
    with RenderJob(path) as job:
        job.render_passes(passes, sync=True)
        assert job.stats()["trace_launches"] == batches * depth
        sums = [job.read_sums(a)[0] for a in range(3)]
        job.reset()
        for _ in range(passes):
            job.render_passes(1)
        assert all(np.array_equal(job.read_sums(a)[0], b) for a, b in enumerate(sums))
