"""Scene upload: the sums that size a batch (LOD0 meshlets, 64-meshlet spans of each object's
largest LOD), taken on the device, against numpy over the same objects."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 8 * 148 * 256 + 1, 700001])
def test_upload_totals_match_host_sums(cuda, n):
    import torch
    from helio_b200 import native as N
    from helio_b200 import scene as S
    from helio_b200.passes import VgScene

    rng = np.random.default_rng(n)
    obj = np.zeros(n, S.DT_OBJECT)
    obj["instance_index"] = rng.integers(0, n + 2, n)  # some past the instances
    obj["lod_count"] = rng.integers(0, 12, n)          # none, and more than eight
    obj["lod_meshlet_counts"] = rng.integers(0, 200, (n, 8))
    obj["lod_meshlet_counts"][rng.integers(0, n)] = 0xFFFFFFFF  # the span count's u32 arithmetic wraps
    obj["local_bounds"] = (0.0, 0.0, 0.0, 1.0)
    inst = np.zeros(n, S.DT_INSTANCE)
    inst["model"] = np.eye(4, dtype=np.float32).reshape(16)
    dev = [torch.from_numpy(a.view(np.uint8).reshape(-1).copy()).cuda() for a in (obj, inst)]
    vs = VgScene()
    for version in (1, 2):  # a first upload and one into the buffers it left
        vs.upload(N.VgFrameData(dev[0].data_ptr(), dev[0].data_ptr(), dev[1].data_ptr(), dev[0].data_ptr(),
                                0, n, 0, 0, version, 1, 0, 0, N.HELIO_MEM_DEVICE, 0))
        got = vs.info()
        counts = obj["lod_meshlet_counts"].astype(np.uint64)
        used = np.arange(8)[None, :] < np.minimum(obj["lod_count"], 8)[:, None]
        largest = np.where(used, counts, 0).max(axis=1)
        spans = ((largest + 63) & 0xFFFFFFFF) // 64
        assert got.object_count == n
        assert got.lod0_meshlets == int(counts[:, 0].sum())
        assert got.max_spans == int(spans.sum())
