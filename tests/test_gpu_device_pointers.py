"""Ray arrays in device memory at the host entry point: copies take them, so a
few rays, which otherwise go through the context's page-locked buffer by the
host's own hand, are answered (or refused) as many are."""
import ctypes

import numpy as np
import pytest

from aviatorengine2_b200 import Context, _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays_there,hits_there", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("variant", [_lib.VARIANT_FAST, _lib.VARIANT_FAST_WALK, _lib.VARIANT_QUANT])
def test_few_as_many(variant, rays_there, hits_there):
    import torch
    s = scenes.hybrid_box(width=96, height=64)
    with Context(96, 64) as ctx:
        ctx.upload(s)
        rays = ctx.camera_rays()
        want = ctx.closest_hit(rays, variant).view(np.uint8).reshape(len(rays), -1)
        d_rays = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
        outcome = []
        for n in (len(rays), 4096, 1000, 1):
            hits = np.zeros((n, want.shape[1]), np.uint8)
            d_hits = torch.zeros(hits.size, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            rc = _lib.lib().ae_closest_hit(
                ctx.handle, ctypes.c_void_p(d_rays.data_ptr() if rays_there else rays.ctypes.data), n,
                ctypes.c_void_p(d_hits.data_ptr() if hits_there else hits.ctypes.data), variant)
            outcome.append(rc)
            if rc == 0:
                got = d_hits.cpu().numpy().reshape(n, -1) if hits_there else hits
                assert np.array_equal(got, want[:n]), n
        assert len(set(outcome)) == 1, outcome
