"""Failure detection of the single-view frame without a GPU fault: the wait of a tile for the draw
counts of the tiles before it is bounded. A tile that withholds its count makes the later tiles give
up after a short poll limit; the execute then publishes a draw count of zero (never the previous
frame's, never one that covers draws nobody wrote), the host reads HELIO_ERR_TIMEOUT, and the next
execute is bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (instances, meshlets each): 100 to 160 tiles of 8, 16 and 512 items; withheld: the first tile, one
# in the middle, the last but one, and the last (which no tile waits for).
@pytest.mark.parametrize("instances,meshlets", [(1200, 20), (2500, 20), (80000, 20)])
@pytest.mark.parametrize("withheld", ["first", "middle", "last but one", "last"])
def test_wait_that_gives_up_publishes_no_draws(cuda, instances, meshlets, withheld):
    import torch
    from helpers import assert_vg_equal, gpu_hiz, gpu_vg_view, oracle_vg_view
    from helio_b200 import native as N
    from helio_b200 import scene as S
    from helio_b200.passes import VirtualGeometryPass, camera_bytes
    from oracle import oracle as O

    sc = S.make_scene(3, instances, meshlets, 4, 0, 60.0)
    v = S.main_view(4, 320, 180, 10)
    hz, _ = gpu_hiz(v.depth)
    vg = VirtualGeometryPass(v.width, v.height)
    want = oracle_vg_view(sc, v, O.hiz_build(v.depth))
    frame = S.frame_data(sc)
    assert_vg_equal(gpu_vg_view(sc, v, hz=hz, frame=frame, vg_pass=vg), want)
    lib = N.cull_lib()
    cam = torch.from_numpy(camera_bytes(v.camera)).cuda()
    out = vg.outputs()
    items = len(sc.work_items)
    per = 512
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    while per > 8 and items < sms * per:
        per //= 2
    tiles = -(-items // per)
    assert tiles > 2
    k = {"first": 1, "middle": tiles // 2, "last but one": tiles - 1, "last": tiles}[withheld]
    before = out["counters"].cpu().numpy()
    assert before[0] > 0
    vg.set_wait_limit(2000, k)
    vg.execute(cam, hz.publish())
    torch.cuda.synchronize()
    got = out["counters"].cpu().numpy()
    if withheld == "last":
        assert lib.helio_vg_device_status(vg._h, None) == N.HELIO_OK
        np.testing.assert_array_equal(got, before)
    else:
        assert lib.helio_vg_device_status(vg._h, None) == N.HELIO_ERR_TIMEOUT
        assert got[0] == 0
        np.testing.assert_array_equal(got[2:], before[2:])  # the select does not wait
    # The same context, normal limits: exact again, and nothing more to report.
    vg.set_wait_limit()
    assert_vg_equal(gpu_vg_view(sc, v, hz=hz, frame=frame, vg_pass=vg), want)
