"""Served requests with and without the Smagorinsky closure, submitted together:
batch members share it, so they run one closure after another, and each ends as
it does alone."""
import pytest

from orrery_b200 import workloads as W
from orrery_b200.lbm3d import Smagorinsky
from orrery_b200.serve import Server

pytestmark = pytest.mark.gpu


def request(seed, closure):
    w = W.sphere3d(seed=seed, nx=64, ny=32, nz=32, diameter=8.0, reynolds=60.0)
    w.config.smagorinsky = Smagorinsky(closure, 0.1 if closure else 0.0)
    return w


def serve(workloads, kernel):
    with Server(storage="f32", chunk_steps=100, sample_every=10, kernel=kernel) as server:
        ids = [server.submit(w, window=200, tolerance=2e-3, max_steps=2000) for w in workloads]
        server.drain(timeout=600)
        return [server.poll(i) for i in ids], server.stats()


@pytest.mark.parametrize("kernel", ["auto", "staged"])
@pytest.mark.parametrize("closures", [(True, False, True), (False, False, True, True, False)])
def test_mixed_closures_end_as_alone(closures, kernel):
    requests = [request(91 + k, on) for k, on in enumerate(closures)]
    alone = [serve([w], kernel)[0][0] for w in requests]
    mixed, stats = serve(requests, kernel)
    assert stats["failed"] == 0 and stats["completed"] == len(requests)
    for got, want in zip(mixed, alone):
        for key in ("state", "steps", "cd", "cl", "cm", "delta_cd", "force", "moment"):
            assert got[key] == want[key], (key, got[key], want[key])
