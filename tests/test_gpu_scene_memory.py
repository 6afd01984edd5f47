"""Loading a scene takes no more device memory than the scene keeps: a server
whose budget is the render lanes, the scene and one request's sums takes the
scene in, for meshes that go through the upload whole and in slices (from 4,096
triangles). The shading records made on the way give the oracle's normals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIDE = 24


def _scene(tmp_path, kind):
    from hastyrenderer_gb300 import scenes
    if kind == "cornell":
        return scenes.cornell_box(str(tmp_path), seed=3, width=SIDE, height=SIDE, spp=2)
    return scenes.sphere_field(str(tmp_path), seed=3, n_spheres=kind, subdiv=2, width=SIDE, height=SIDE, spp=2,
                               env_size=(64, 32), box=4.0)


def _serve(path, budget):
    from hastyrenderer_gb300 import Server
    with Server(paths_in_flight=1 << 13, memory_budget=budget) as srv:
        rid = srv.submit(path, passes=2)
        srv.wait_idle(120000)
        res = srv.poll(wait_ms=1000)[0]
        sums = srv.read_sums(rid) if res["status"] == 0 else None
        srv.release(rid)
        return res, sums, srv.stats()


# 320 triangles a sphere and a ground of 2: one slice, one more than one, several
@pytest.mark.parametrize("kind", ["cornell", 12, 13, 100])
def test_budget_of_what_the_scene_keeps(tmp_path, kind):
    path = _scene(tmp_path, kind)
    res, want, st = _serve(path, 0)
    assert res["status"] == 0, res["error"]
    assert st["resident_scenes"] == 1
    budget = st["resident_bytes"] + SIDE * SIDE * 9 * 8     # lanes and scene, and one request's sums
    res, sums, st = _serve(path, budget)
    assert res["status"] == 0, res["error"]
    assert st["peak_resident_bytes"] <= budget
    assert np.array_equal(sums, want)


@pytest.mark.parametrize("kind", ["cornell", 12, 13, 100])
def test_records_of_every_slice(tmp_path, kind):
    from hastyrenderer_gb300 import RenderJob
    from oracle.oracle import Oracle
    path = _scene(tmp_path, kind)
    with RenderJob(path) as job:
        job.render_passes(1, sync=True)
        normal, _ = job.read_sums(1)
    ora = Oracle(path)
    _, want, _ = ora.render_samples(0, 0, 0, SIDE, SIDE)
    ora.close()
    close = np.all(np.abs(normal - want) <= 1e-3, axis=-1)
    assert np.isfinite(normal).all() and close.mean() >= 0.95, close.mean()
