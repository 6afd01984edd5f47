"""Device memory of a server's render lanes: 424 bytes a path (state 96, medium
stack 80 and its share of the overflow pool 80, rays 64, hits 32, queues 24,
outputs 48), and the path kernel's slots only in contexts whose scenes may use
that kernel. What they render is the same to the bit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "scenes")
PATHS = 1 << 16


def _serve(flags, names=("cornell", "room", "field")):
    from hastyrenderer_gb300 import Context, Server
    with Server(Context(0, flags), paths_in_flight=PATHS, lanes=2) as srv:
        ids = [srv.submit(os.path.join(GOLDEN, n, "renderJob.json"), passes=3, seed=4) for n in names]
        srv.wait_idle(120000)
        got = {}
        while len(got) < len(ids):
            for r in srv.poll(wait_ms=1000):
                assert r["status"] == 0, r["error"]
                got[r["id"]] = srv.read_sums(r["id"])
        return srv.stats()["engine_bytes"], [got[i] for i in ids]


def test_lane_bytes_and_results():
    from hastyrenderer_gb300 import Context
    plain, want = _serve(0)
    state = 2 * 424 * PATHS
    assert state <= plain <= state + (64 << 10)      # counters and 256-byte boundaries
    for flags, pools in ((Context.WAVEFRONT, False), (Context.PATH_KERNEL, True), (Context.BINARY_BVH, False)):
        size, sums = _serve(flags)
        assert (size == plain) != pools, flags
        assert all(np.array_equal(a, b) for a, b in zip(sums, want)), flags
