"""Index generation at the edges of a word of flags, a warp's range and a tile, with
terminations at random and on those edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [32, 256, 2048]


@pytest.mark.parametrize("n", [2, 3] + [e + d for e in EDGES + [3 * 2048] for d in (-1, 0, 1, 2)] + [100003])
def test_indices_match_the_oracle(ctx, port, n):
    rng = np.random.default_rng(n)
    v = rng.normal(size=(n, 4)).astype(np.float32)
    v[:, 3] = 0.0
    term = rng.random(n) < 0.02
    for e in EDGES:
        at = np.arange(e, n, e)
        term[at[rng.random(len(at)) < 0.5]] = True
        term[at[rng.random(len(at)) < 0.5] - 1] = True
    v[term] = (-2.0, -2.0, -2.0, 0.0)
    assert np.array_equal(ctx.index_generate(v), port.index_generate(v))


@pytest.mark.parametrize("tiles", [1, 31, 33, 1023, 1025, 8191, 8192, 8193])
def test_tile_offsets_of_one_and_of_many_blocks(ctx, tiles):
    """Every vertex indexed but the last: the scan's offsets show in every index."""
    n = tiles * 2048 - 5
    v = np.ones((n, 4), np.float32)
    assert np.array_equal(ctx.index_generate(v), np.arange(n - 1, dtype=np.int32))
