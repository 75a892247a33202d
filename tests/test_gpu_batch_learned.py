"""The learned flux switched on between graph replays of the batch's member path."""
import numpy as np
import pytest

from test_gpu_batch import _reset, _same, _state, small_batch  # noqa: F401

pytestmark = pytest.mark.gpu


def test_learned_flux_switched_between_replays(small_batch):  # noqa: F811
    """Plain steps first, so that the member path's work arrays and graph are there; then
    the learned flux on, off and on again, each followed at once by replayed steps: the
    bits of the same calls launched directly."""
    from fesom2_tracer_dwarf_b200.learned import trained_params
    b, specs, dts, init = small_batch
    p = trained_params()

    def run(graph):
        _reset(b, init)
        b.set_path("separate")
        out = []
        for on, n in ((None, 4), (True, 3), (None, 2), (False, 5), (True, 2)):
            if on is not None:
                b.learn_set(p, on)
            b.steps(n, graph=graph)
            out.append(_state(b))
        b.learn_set(None, False)
        return out

    graph, plain = run(True), run(False)  # the replayed calls on a batch that has not had the learned flux
    assert all(_same(x, y) for x, y in zip(graph, plain))
    assert not _same(graph[0], graph[1])
