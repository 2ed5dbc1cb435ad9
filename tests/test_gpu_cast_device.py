"""Device-resident rays (owec_cast_rays_device) at the edges of the blocks' shares: any batch gives what its rays
give in small calls, and what the host entry point gives."""
import ctypes

import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


def cast_device(c, o, d):
    import torch
    n = len(o)
    dev = [torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda() for x in (o, d)]
    b, p, t = torch.zeros(n, dtype=torch.int32).cuda(), torch.zeros(n, dtype=torch.int32).cuda(), torch.zeros(n).cuda()
    torch.cuda.synchronize()
    seconds = ctypes.c_double()
    owe_cuda._check(c.lib, c.lib.owec_cast_rays_device(c.handle, n, dev[0].data_ptr(), dev[1].data_ptr(), b.data_ptr(),
                                                       p.data_ptr(), t.data_ptr(), ctypes.byref(seconds)), "owec_cast_rays_device")
    return b.cpu().numpy().view(np.uint32), p.cpu().numpy().view(np.uint32), t.cpu().numpy()


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 148 * 3 * 128, 148 * 3 * 128 + 1, 148 * 8 * 128, 148 * 8 * 128 + 1, 400001])
def test_device_batches_match_their_rays_in_small_calls(n, full):
    sb = scenes.bvh_stress_room(16, 16, 64, 32)
    if full:
        sb.boundary(A.SHAPE_CONE, [0.1, 0.0, 0.05, 0.1], scenes.translate(0.0, 0.0, -50.0), 0, 0, sb.diffuse(0.5))
    o, d = scenes.random_rays(n, 5, (-2.5, -2.5, 0.3), (2.5, 2.5, 3.7), (-1.2, -1.2, 0.1), (1.2, 1.2, 2.4))
    with owe_cuda.Context(0) as c:
        c.upload(sb.desc())
        c.build_bvh()
        local = (o - c.scene_origin()).astype(np.float32)
        dir32 = d.astype(np.float32)
        whole = cast_device(c, local, dir32)
        parts = [cast_device(c, local[a:a + 20011], dir32[a:a + 20011]) for a in range(0, n, 20011)]
        host = c.cast_rays(local.astype(np.float64) + c.scene_origin(), dir32.astype(np.float64))
    for k in range(3):
        assert np.array_equal(whole[k], np.concatenate([p[k] for p in parts]))
    same = whole[0] == host[0]
    assert same.mean() >= 0.999
    # a distance in the room's few metres, rounded to FP32 and taken from the FP32 triangle: 1e-5 of them
    assert np.abs(whole[2] - host[2])[same].max() <= 1e-4
