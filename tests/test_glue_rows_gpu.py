"""The denoiser's element-wise kernels walk the rows of all images of a batch with a grid of at most 65535 rows: a batch
with more rows than that, and one whose levels end in single pixels, must give each image's own result."""
import numpy as np
import pytest

from sparkle_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4100, 16, 16), (3, 17, 33), (1, 1, 1)])
def test_each_image_of_a_batch_is_its_own_result(shape):
    import torch
    n, h, w = shape
    rng = np.random.default_rng(n)
    kinds = torch.from_numpy(rng.uniform(0, 1, (5, h, w, 10)).astype(np.float32)).cuda()
    pick = torch.arange(n, device="cuda") % 5
    dn = native.Denoiser(0, seed=3)
    out = dn.infer(kinds[pick].contiguous())
    alone = [dn.infer(kinds[k:k + 1].contiguous())[0] for k in range(min(n, 5))]
    for k, a in enumerate(alone):
        assert torch.equal(out[pick == k], a.expand(int((pick == k).sum()), h, w, 4))
    dn.close()
