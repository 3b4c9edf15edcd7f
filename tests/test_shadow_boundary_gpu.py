"""Shadow cull decisions at the boundary: spheres whose signed distance to a plane of some dirty face,
in the reference's operation order and binary32 rounding, is exactly zero or one step of the radius
to either side of it. A single product that is not rounded before it is added moves many of them to
the other side."""
import numpy as np
import pytest

from helpers import u32
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def boundary_scene(seed, n):
    """Matrices, faces in use, n instances and draws: instance i lies at a random centre, with the radius
    that brings its distance to plane i % 6 of face i % faces to 0, or one ulp below or above."""
    from helio_b200 import scene as S

    mats, nf = S.shadow_faces(seed, 12, 4)
    rng = np.random.default_rng(seed)
    inst = np.zeros(n, S.DT_INSTANCE)
    m = mats[:nf].reshape(nf, 4, 4)
    c3 = m[:, 3]
    planes = np.stack([c3 + m[:, 0], c3 - m[:, 0], c3 + m[:, 1], c3 - m[:, 1], m[:, 2], c3 - m[:, 2]], axis=1)
    length = np.sqrt((planes[..., 0] * planes[..., 0] + planes[..., 1] * planes[..., 1]) + planes[..., 2] * planes[..., 2])
    assert planes.dtype == np.float32 and length.dtype == np.float32
    big = length > 1e-10
    planes = np.where(big[..., None], planes / np.where(big, length, 1)[..., None], planes)
    k = np.arange(n)
    p = planes[k % nf, (k // nf) % 6]
    c = rng.uniform(-150, 150, (n, 3)).astype(np.float32)

    def dist(c):
        return ((p[:, 0] * c[:, 0] + p[:, 1] * c[:, 1]) + p[:, 2] * c[:, 2]) + p[:, 3]

    # Centres outside the plane (a positive radius is needed): mirrored through it where they are inside.
    s = dist(c).astype(np.float64)
    c = np.where((s > -0.5)[:, None], c - ((s + 3.0) / 1.0)[:, None] * p[:, :3].astype(np.float64), c).astype(np.float32)
    s = dist(c)
    r = np.where(s < 0, -s, np.float32(1.0))
    step = k % 3
    r = np.where(step == 1, np.nextafter(r, np.float32(0)), np.where(step == 2, np.nextafter(r, np.float32(np.inf)), r))
    inst["bounds"][:, :3] = c
    inst["bounds"][:, 3] = r
    d = dist(c) + inst["bounds"][:, 3]
    assert (np.abs(d) < 1e-4).mean() > 0.9 and (d < 0).mean() > 0.2 and (d == 0).mean() > 0.2 and (d > 0).mean() > 0.2
    src = np.zeros((n, 5), np.uint32)
    src[:, 0] = 3
    src[:, 1] = 1
    src[:, 4] = np.arange(n)
    return mats, nf, inst, src


@pytest.mark.parametrize("draws", [2048, 6000, 40000])
@pytest.mark.parametrize("faces", [1, 3, 0])  # 0: all of them
@pytest.mark.parametrize("folded", [False, True])
def test_spheres_on_a_plane_match_oracle(cuda, draws, faces, folded):
    import torch
    from helio_b200 import scene as S
    from helio_b200.passes import BatchedCull, ShadowCullPass, VgScene

    mats, nf, inst, src = boundary_scene(21 + draws, draws)
    dirty = np.zeros(256, np.uint32)
    dirty[: faces or nf] = 1
    keep = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (mats, inst.view(np.uint8), src.view(np.int32), dirty.view(np.int32))]
    sh = ShadowCullPass()
    sh.prepare(*keep, nf)
    if folded:
        sc = S.make_scene(3, 500, 8, 2, 0, 40.0)
        vs, b = VgScene(), BatchedCull(1)
        vs.upload(S.frame_data(sc))
        v = S.main_view(4, 64, 64, 4)
        b.prepare(vs, [{"camera": v.camera, "depth": torch.from_numpy(v.depth).cuda()}])
        b.attach_shadow(sh)
        b.execute()
        torch.cuda.synchronize()
        b.status()
        b.attach_shadow(None)
    else:
        sh.execute()
        torch.cuda.synchronize()
    o = sh.outputs()
    got, counts = u32(o["face_indirect"]), u32(o["face_counts"])
    ref, ref_counts, ran = O.shadow_cull(mats, inst, src, dirty, nf)
    assert ran
    np.testing.assert_array_equal(counts, ref_counts)
    for f in np.nonzero(dirty)[0]:
        k = min(int(ref_counts[f]), 4096)
        np.testing.assert_array_equal(got[f * 4096:f * 4096 + k], ref[f * 4096:f * 4096 + k], err_msg=f"face {f}")
