"""The reordering of an upload moves every array the same way, on both sides of the size up to which all arrays are moved
at once (65,536 slots): what was uploaded comes back to the bit, also after a second upload."""

import numpy as np
import pytest

from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1025, 65536, 65537])
def test_uploaded_arrays_come_back(n):
    rng = np.random.default_rng(n)
    shapes = {"pos": (n, 3), "mass": (n,), "vel": (n, 3), "acc": (n, 3), "density": (n,), "dstress": (n, 3, 3), "balsara": (n,)}
    with DeviceParticleBuffer(make_params(H=0.01), n, make_options()) as pb:
        for _ in range(2):
            st = {k: rng.uniform(0.5, 1.0, s).astype(np.float32) for k, s in shapes.items()}
            st["dstress"] = (st["dstress"] + st["dstress"].transpose(0, 2, 1)).astype(np.float32)
            st["dstress"][:, 2, 2] = -(st["dstress"][:, 0, 0] + st["dstress"][:, 1, 1])
            pb.upload(st)
            out = pb.download(list(shapes))
            for k in shapes:
                np.testing.assert_array_equal(out[k], st[k], err_msg=k)
