"""The device repack's size classes (subtrees built in shared memory, ranges split a block
each, ranges split by many blocks) write the host repack's bytes at the sizes where one
class ends and the next begins."""
import pytest

import leafgen
from yune_gb300 import scenes
from yune_gb300.core import Renderer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def r():
    with Renderer(0) as rr:
        yield rr


@pytest.mark.parametrize("kind", ["random", "grid", "coincident"])
@pytest.mark.parametrize("leaves", [255, 256, 257, 16384, 16385])
def test_ends_of_the_size_classes(r, leaves, kind):
    s = leafgen.leaf_scene(leaves, kind, leaves + 1)
    lay = scenes.layout(s, 1)
    sid = r.upload(s)
    assert (r.scene_digest(sid), r.scene_depth(sid), r.scene_bytes(sid)) == (lay["digest"], lay["depth"], lay["device_bytes"])
    r.release(sid)
