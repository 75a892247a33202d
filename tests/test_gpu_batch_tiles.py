"""The cooperative path's tiles: more blocks per SM than its register budget holds."""
import pytest

from test_gpu_batch import _reset, _same, _state, small_batch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,resident", [(256, 2), (128, 4), (64, 8)])
def test_a_tile_asks_for_more_blocks_than_fit(small_batch, threads, resident):  # noqa: F811
    """128 registers a thread leave room for 512 threads per SM: the tile reports them and
    the step gives the bits of the members' own launches."""
    b, specs, dts, init = small_batch
    b.steps_separate(3)
    want = _state(b)
    b.set_path("cooperative")
    for blocks in (3, 7, 16):
        b.set_tile(threads=threads, blocks_per_sm=blocks, wave=2)
        assert b.tile()["blocks_per_sm"] == min(blocks, resident)
        _reset(b, init)
        b.steps(3, graph=True)
        assert _same(_state(b), want)


def test_autotuner_times_each_candidate_once(small_batch):  # noqa: F811
    """No step path has a tile of cells, so each path, wave, thread and block count is
    timed once and the caller's cells per block stay; a tile outside 32..576 cells is
    still refused."""
    b, specs, dts, init = small_batch
    b.set_tile(cells_per_block=128, threads=64, blocks_per_sm=1, wave=1)
    lines = [x.rsplit(" ms_per_step=", 1)[0] for x in b.autotune(1).splitlines() if not x.startswith("best:")]
    assert len(lines) == len(set(lines)) >= 3, lines
    assert b.tile()["cells_per_block"] == 128
    for cells in (31, 577):
        with pytest.raises(RuntimeError):
            b.set_tile(cells_per_block=cells)
