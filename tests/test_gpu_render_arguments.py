"""NeRF.render's `chunk` is a whole number whatever the number of rays (the
reference renders whole batches of rays, base_dataset.py:853-857)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays", [0, 5, 70])
def test_chunk_is_a_whole_number(ng, cuda, rays):
    nerf = ng.NeRF(ng.make_params(N_coarse=32, N_fine=64))
    o, d, near, far = (torch.from_numpy(v).cuda() for v in ng.synthetic.sphere_rays(max(rays, 1), 1))
    batch = [v[:rays] for v in (o, d, near, far)]
    want = nerf.render(*batch, chunk=64, seed=3)
    got = nerf.render(*batch, chunk=np.int64(64), seed=3)
    assert all(torch.equal(got[k], want[k]) for k in ("rgb", "depth", "acc"))
    for chunk in (64.0, 4096.0, "64"):
        with pytest.raises(TypeError):
            nerf.render(*batch, chunk=chunk, seed=3)
    with pytest.raises(ZeroDivisionError):
        nerf.render(*batch, chunk=0, seed=3)
