"""goofy_gpu_batch_encode_noalloc on several streams at once and captured into
a graph: calls share nothing."""
import pytest

import goofy_gb300 as g
from tests.test_gpu_batch import _many, check, descriptors

pytestmark = pytest.mark.gpu


def test_calls_overlap_on_different_streams(cuda):
    streams = [cuda.cuda.Stream() for _ in range(4)]
    sets = [_many(cuda, n, 20 + n, big=((3, (1024, 516)),)) for n in (12, 40, 256, 256)]
    arrays = [g.images_array(descriptors(s)) for s in sets]
    cuda.cuda.synchronize()
    for _ in range(10):
        for st, arr in zip(streams, arrays):
            assert g.batch_encode_noalloc(arr, st.cuda_stream) == g.OK, g.last_error()
    for items in sets:
        check(cuda, items)


@pytest.mark.parametrize("n", [5, 32, 200])
def test_captured_calls_encode_what_the_buffers_hold_at_each_replay(cuda, n):
    items = _many(cuda, n, 30 + n, big=((2, (516, 516)),))
    arr = g.images_array(descriptors(items))
    graph, stream = cuda.cuda.CUDAGraph(), cuda.cuda.Stream()
    cuda.cuda.synchronize()
    with cuda.cuda.graph(graph, stream=stream):
        assert g.batch_encode_noalloc(arr, stream.cuda_stream) == g.OK, g.last_error()
    del arr  # nothing of the caller's is read after the call
    for turn in range(2):
        for it in items:
            it["dst"].fill_(0x5A)
            if turn and it["w"]:
                rows = 255 - it["rows"]
                it["src"][it["offset"]:it["offset"] + rows.size].copy_(cuda.from_numpy(rows.reshape(-1)))
                it["rows"] = rows
        cuda.cuda.synchronize()
        graph.replay()
        check(cuda, items)
