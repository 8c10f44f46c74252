"""Stage times of a call: from events in a first call, from the kernels' own time stamps in a repeated one (device
plan). Every stage that ran is positive, and together they fit into the call's device time; the two clocks are
taken to agree to 20 us (a few launch gaps and the event clock's granularity)."""
import numpy as np
import pytest

from svdimager_b200 import api
from tests.conftest import snapshot

pytestmark = pytest.mark.gpu

STAGES = ("ms_preprocess", "ms_bin", "ms_grid", "ms_fft", "ms_image")


@pytest.mark.parametrize("K", [1, 2, 5, 8, 9])
def test_stages_fit_into_the_call(cuda_device, K):
    s = snapshot("small", n_rows_limit=3000, nchan=8)
    with api.Engine(k_rule=api.KRULE_FIXED, fixed_k=K) as e:
        images = []
        for _ in range(3):
            images.append(e.image(s, 256, 4e-4))
            st = e.stats()
            t = [st[k] for k in STAGES]
            assert all(x > 0.0 for x in t), t
            assert sum(t) <= st["ms_total"] + 0.02, (t, st["ms_total"])
        # the order of FP32 reductions differs between calls
        assert np.nanmax(np.abs(images[0] - images[2])) <= 1e-5 * np.nanmax(np.abs(images[0]))


def test_stages_of_device_calls(cuda_device):
    torch = pytest.importorskip("torch")
    from tests.test_gpu_batch import _upload
    s = snapshot("small", n_rows_limit=3000, nchan=8)
    keep, (d,) = _upload([s], torch)
    out = torch.zeros(256, 256, device="cuda")
    with api.Engine() as e:
        for _ in range(3):
            e.image_device(d, 256, 4e-4, out.data_ptr())
            torch.cuda.synchronize()
            st = e.stats()
            t = [st[k] for k in STAGES]
            assert all(x > 0.0 for x in t), t
            assert sum(t) <= st["ms_total"] + 0.02, (t, st["ms_total"])
