"""Tiles recorded by a build with other image kernels are not installed."""
import pytest

import goofy_gb300 as g

pytestmark = pytest.mark.gpu


def test_entries_without_this_kernel_revision_are_left(cuda, tmp_path):
    path = str(tmp_path / "tiles.txt")
    name, sms = g.device_key(0)
    model = cuda.cuda.get_device_name(0)
    assert name.startswith(model) and name != model
    lines = ["v1|%s|%d|%s|128|1|0|40.0" % (n, sms, c) for n in (model, model + " kernels 1")
             for c in ("bc1", "etc1s", "both")]
    try:
        g.set_tile_cache_path(path)
        with open(path, "w") as f:
            f.write("\n".join(lines) + "\n")
        g.reset_tiles()
        assert g.load_tile_cache(0) == 0
        assert [g.get_tile(c) for c in range(3)] == [(512, 2, 2)] * 3
        assert g.tile_cache_store(path, name, sms, g.CODEC_BC1, (256, 1, 0), 41.0) == g.OK
        assert g.load_tile_cache(0) == 1 and g.get_tile(g.CODEC_BC1) == (256, 1, 0)  # this revision's is found
    finally:
        g.set_tile_cache_path(None)
        g.reset_tiles()
