"""Batches of more than 2044 images, whose descriptors are uploaded: repeated
calls refill both slots while earlier calls are in flight and replay the
captured graph with new pointers, and every tile runs on that path."""
import numpy as np
import pytest

import goofy_gb300 as g
from tests.test_gpu_batch import _many, check, descriptors

pytestmark = pytest.mark.gpu

N = 2100


@pytest.fixture(scope="module")
def sets(cuda):
    """Four sets of the same shape: other pixels and other buffers."""
    out = [_many(cuda, N, 7)]
    for k in range(1, 4):
        rng = np.random.default_rng(100 + k)
        items = []
        for it in out[0]:
            rows = it["rows"].copy()
            rows[:, :4 * it["w"]] = rng.integers(0, 256, (it["h"], 4 * it["w"]), np.uint8)
            buf = np.zeros(it["src"].numel(), np.uint8)
            buf[it["offset"]:it["offset"] + rows.size] = rows.reshape(-1)
            items.append(dict(it, rows=rows, src=cuda.from_numpy(buf).cuda(), dst=cuda.full_like(it["dst"], 0x5A)))
        out.append(items)
    return out


@pytest.mark.parametrize("graphs", [True, False])
def test_slots_and_replay_with_new_pointers(cuda, sets, graphs):
    """Eight calls in a row on a stream kept busy, no synchronisation between them: each slot is filled four
    times, the set changes with every call (also from one use of a slot to the next)."""
    arrays = [g.images_array(descriptors(s)) for s in sets]
    order = [0, 1, 2, 3, 1, 0, 3, 2]
    busy = cuda.empty(64 << 20, dtype=cuda.uint8, device="cuda")
    b = g.Batch(N)
    try:
        b.set_graphs(graphs)
        for turn in range(2):
            for items in sets:
                for it in items:
                    it["dst"].fill_(0x5A)
            stream = cuda.cuda.current_stream().cuda_stream
            for _ in range(20):
                busy.random_(0, 256)
            for k in order[4 * turn:] if turn else order:
                assert b.encode(arrays[k], stream) == g.OK, g.last_error()
            for items in sets:
                check(cuda, items)
    finally:
        b.close()


def test_the_shape_changes_between_calls(cuda, sets):
    """A graph is captured again when the images' sizes, and with them the units, change."""
    other = _many(cuda, N, 8)
    b = g.Batch(N)
    try:
        stream = cuda.cuda.current_stream().cuda_stream
        for items in (sets[0], other, sets[1], sets[2], other):
            for it in items:
                it["dst"].fill_(0x5A)
            assert b.encode(descriptors(items), stream) == g.OK, g.last_error()
            check(cuda, items)
    finally:
        b.close()


@pytest.mark.parametrize("tile", [(128, 1, 64), (128, 2, 64), (256, 2, 256), (512, 2, 2048), (512, 1, 32), (256, 2, 192),
                                  (128, 1, 128, 1), (512, 2, 1024, 1)])
def test_tiles(cuda, sets, tile):
    big = _many(cuda, N, 9, big=((5, (1028, 516)), (1000, (516, 1024)), (2099, (2052, 260))))
    b = g.Batch(N)
    try:
        assert b.set_tile(*tile) == g.OK
        stream = cuda.cuda.current_stream().cuda_stream
        for items in (big, sets[3]):
            for it in items:
                it["dst"].fill_(0x5A)
            assert b.encode(descriptors(items), stream) == g.OK, g.last_error()
            check(cuda, items)
    finally:
        b.close()
