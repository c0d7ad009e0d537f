"""aldic_load_image_raw with the image, the mask or both on the device: the same image as from host arrays, on
contexts whose scratch holds nothing else."""
import numpy as np
import pytest
import torch

import aldic_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32, np.float64])
@pytest.mark.parametrize("M,N", [(8, 8), (61, 83), (1500, 1101)])
def test_image_and_mask_on_the_device(M, N, dtype):
    rng = np.random.default_rng(M)
    img = np.asfortranarray(rng.integers(0, 250, (M, N)).astype(dtype))
    mask = np.asfortranarray((rng.random((M, N)) < 0.7).astype(np.float64))
    want = None
    for dev_img in (False, True):
        for dev_mask in (False, True):
            c = A.Context(0)  # a fresh one: nothing reserved yet
            try:
                i, m = img, mask
                if dev_img:
                    i = torch.from_numpy(img.ravel(order="F").copy()).cuda()
                if dev_mask:
                    m = torch.from_numpy(mask.ravel(order="F").copy()).cuda()
                torch.cuda.synchronize()
                for slot in (0, 1):
                    c.load_image_raw(slot, i, [1, M], [1, N], mask=m, want_stats=False, shape=(M, N))
                got = [c.get_state(slot) for slot in (0, 1)]
            finally:
                c.close()
            assert np.array_equal(got[0], got[1])
            assert np.all(got[0][mask == 0] == 0) and np.any(got[0] != 0)
            if want is None:
                want = got[0]
            assert np.array_equal(got[0], want), (dev_img, dev_mask)
