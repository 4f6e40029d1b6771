"""Host copies of 32 MiB and more go through page-locked slots by several threads: images
and sinograms at the edges of that size and of its 256 KiB pieces come back bit for bit,
also when the slots are used again."""
import numpy as np
import pytest

from mlem_b200 import api

pytestmark = pytest.mark.gpu

MIB32 = (32 << 20) // 4  # floats
PIECE = (256 << 10) // 4


def long_vectors(n_rows, n_cols):
    """A matrix of one element and long vectors."""
    end = np.ones(n_rows, np.uint64)
    el = np.zeros(1, api.ELEM_DTYPE)
    el["value"] = 1.0
    return api.Context(end, el, n_rows, n_cols, flags=api.FLAG_NO_ROW_ORDER)


@pytest.mark.parametrize("n,frames", [(MIB32 - 1, 1), (MIB32, 1), (MIB32 + 1, 1), (MIB32 + 5 * PIECE - 3, 1),
                                      (MIB32 + PIECE // 2, 1), (MIB32 // 3 + 1, 3), (MIB32 // 4, 4)])
def test_images_come_back_as_they_went(n, frames):
    rng = np.random.default_rng(n)
    with long_vectors(1, n) as ctx:
        ctx.set_sinograms(np.ones((frames, 1), np.int32))
        for _ in range(2):
            x = rng.random((frames, n), dtype=np.float32)
            ctx.set_images(x)
            assert np.array_equal(ctx.get_images(), x)


@pytest.mark.parametrize("n,frames", [(MIB32, 1), (MIB32 + 1, 1), (MIB32 + 3 * PIECE + 7, 1), (MIB32 // 3 + 1, 3)])
def test_sinograms_arrive_whole(n, frames):
    """An identity matrix: an iteration from an image of ones gives the counts, exactly."""
    rng = np.random.default_rng(n)
    el = np.zeros(n, api.ELEM_DTYPE)
    el["index"] = np.arange(n)
    el["value"] = 1.0
    with api.Context(np.arange(1, n + 1, dtype=np.uint64), el, n, n, flags=api.FLAG_NO_ROW_ORDER) as ctx:
        for _ in range(2):
            s = rng.integers(0, 1 << 20, (frames, n), dtype=np.int32)
            ctx.set_sinograms(s)
            want = [np.float32(float(s[b].sum(dtype=np.int64)) / n) for b in range(frames)]
            assert np.array_equal(ctx.init_images(), want)
            ctx.set_images(np.ones((frames, n), np.float32))
            ctx.iterate(1)
            assert np.array_equal(ctx.get_images(), s)
