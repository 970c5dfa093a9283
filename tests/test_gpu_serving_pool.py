"""The server's pool fills the budget it is given: a row holds the evaluated
directions, one of each antipodal pair."""
import numpy as np
import pytest

from pointint_gb300 import geometry as G
from pointint_gb300.kgrid import standard_kgrid
from pointint_gb300.serving import Server
from test_gpu_expansions import patch

pytestmark = pytest.mark.gpu

SMALL = dict(autotune=False, inflight_batches=1, max_batch_queries=1, max_batch_rows=8, max_batch_evals=8)
CHUNK = 32  # columns a row is padded to


@pytest.mark.parametrize("order,radii", [(9, 16), (9, 48), (29, 32)])
def test_rows_fill_the_budget(cuda, order, radii):
    kg = standard_kgrid(order, radii)
    columns = len(kg.direction_pairs()) * radii
    row_bytes = (columns + CHUNK - 1) // CHUNK * CHUNK * 8
    lib = [patch("tri", 20 + 5 * i, i) for i in range(8)]
    rng = np.random.default_rng(4)
    scenes = [(rng.integers(0, 8, 4), None, rng.normal(0, 0.3, (4, 3))) for _ in range(6)]
    rows = {}
    for extra in (0, 100, 1000):
        with Server(kg, lib, hbm_budget_bytes=256 * 1024 * 1024 + extra * row_bytes, **SMALL) as srv:
            rows[extra] = srv.stats()["pool_rows"]
            if extra == 0:
                ref = [srv.query(*s) for s in scenes]
    assert rows[100] - rows[0] == 100 and rows[1000] - rows[0] == 1000

    # a pool of five rows: evictions, and the same results
    with Server(kg, lib, hbm_budget_bytes=256 * 1024 * 1024 - (rows[0] - 5) * row_bytes, **SMALL) as srv:
        assert srv.stats()["pool_rows"] == 5
        got = [srv.query(*s) for s in scenes]
        assert srv.stats()["evictions"] > 0
    for a, b in zip(ref, got):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-12 * np.abs(a).max())
