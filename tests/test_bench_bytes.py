"""The bench's bytes per object are those of the records that the kernels read (csrc/vg.h), so that a
fraction of the roofline is not one of bytes that nobody moves."""
import re
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent.parent


def test_object_bytes_are_the_resident_records():
    import bench
    from helio_b200 import scene as S

    text = (ROOT / "helio_b200" / "csrc" / "vg.h").read_text()
    world = int(re.search(r"sizeof\(ObjectWorld\) == (\d+)", text).group(1))
    xform = int(re.search(r"sizeof\(InstanceXform\) == (\d+)", text).group(1))
    obj = np.zeros(6, S.DT_OBJECT)
    obj["instance_index"] = [0, 1, 1, 2, 3, 3]
    sc = S.Scene(np.zeros(1, S.DT_MESHLET), obj, np.zeros(6, S.DT_INSTANCE), np.zeros(6, S.DT_ITEM), None, None, 6, 1)
    # Objects 1, 2 and 5 are selected somewhere: two instances.
    visible = np.array([0, 1, 1, 0, 0, 1], bool)
    assert bench.object_bytes(sc, visible) == (world * 6 + (32 + 8) * 3, xform * 2)
    assert bench.object_bytes(sc, np.zeros(6, bool)) == (world * 6, 0)
