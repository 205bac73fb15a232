"""When BatchedSolver.run captures a graph: the choice moves launches, never results."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [(40,), (200,), (209,), (210,), (40,) * 8, (220, 40), (15, 215)])
def test_capture_waits_until_it_pays(runs):
    from pycorrectedemissionct_b200 import core, engine

    n, a = 32, 24
    c = core.XrfCore(n, np.linspace(0, 2 * np.pi, a, endpoint=False))
    g = torch.Generator(device="cuda").manual_seed(3)
    maps = torch.rand((1, a, 1, n, n), device="cuda", generator=g) + 0.5
    b = torch.rand((1, 1, a, n), device="cuda", generator=g) + 0.5
    plain = engine.BatchedSolver(c, maps, b, "mlem")
    auto = engine.BatchedSolver(c, maps, b, "mlem")
    could = 0  # iterations queued eagerly after the first block of a run, in full blocks
    captured = False
    for its in runs:
        assert plain.run(its, check_every=10, use_graph=False) == its
        assert auto.run(its, check_every=10) == its
        for done in range(10, its - 9, 10):
            captured = captured or could + its - done >= engine.GRAPH_PAYS
            could += 0 if captured else 10
        assert (auto._graph is not None) == captured
    assert torch.equal(plain.x, auto.x) and torch.equal(plain.residuals, auto.residuals)
