"""A batch captured snapshot after snapshot runs on its engine's buffers. Between its launches the engine may
image anything -- the same wide field, which outside a batch goes through w planes and their larger records, a
larger snapshot, another image size -- and the next launch gives the batch's images again.

Tolerance 1e-6 relative RMS: the order of floating-point atomic adds (as in the other repeat tests)."""
import numpy as np
import pytest

from oracle import oracle as O
from svdimager_b200 import api
from tests.conftest import snapshot
from tests.test_gpu_batch import _upload

pytestmark = pytest.mark.gpu


def test_images_between_launches(cuda_device):
    import torch
    N, cell = 256, 0.3 / 256
    opt = dict(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT, max_batch_slabs=1)
    snaps = [snapshot("widefield", nchan=4, n_rows_limit=r, image_size=N, cell_size=cell) for r in (3000, 2500)]
    large = snapshot("widefield", nchan=8, n_rows_limit=20000, image_size=N, cell_size=cell)
    keep, descs = _upload(snaps + [large], torch)
    imgs = torch.zeros((2, N, N), device="cuda")
    one = torch.zeros((N, N), device="cuda")
    other = torch.zeros((2 * N, 2 * N), device="cuda")
    with api.Engine(**opt) as e, api.Engine(**opt) as free:
        free.image_device(descs[0], N, cell, one.data_ptr())
        ref = one.cpu().numpy()
        with api.Batch(e, descs[:2], N, cell, imgs.data_ptr()) as b:
            assert not b.wide and b.plan(0)["num_slabs"] > 1
            b.launch()
            b.check()
            first = imgs.cpu().numpy()
            assert O.rel_rms(first[0], ref) < 1e-5  # w planes and moments of one error target
            for _ in range(2):
                for d, n, out in ((descs[0], N, one), (descs[2], N, one), (descs[1], 2 * N, other)):
                    e.image_device(d, n, 0.3 / n, out.data_ptr())
                torch.cuda.synchronize()
                imgs.zero_()
                b.launch()
                b.check()
                assert O.rel_rms(imgs.cpu().numpy(), first) < 1e-6
        e.image_device(descs[0], N, cell, one.data_ptr())  # after the batch: through w planes again
        assert O.rel_rms(one.cpu().numpy(), ref) < 1e-6


@pytest.mark.parametrize("slabs", [0, 1])
def test_engine_closed_before_its_batch(cuda_device, slabs):
    """A batch that outlives its engine refuses to launch and can be destroyed (wide and chained)."""
    import torch
    N = 256
    opt = dict(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT, max_batch_slabs=slabs)
    snaps = [snapshot("widefield", nchan=4, n_rows_limit=r, image_size=N, cell_size=0.3 / N) for r in (3000, 2500)]
    keep, descs = _upload(snaps, torch)
    imgs = torch.zeros((2, N, N), device="cuda")
    e = api.Engine(**opt)
    b = api.Batch(e, descs, N, 0.3 / N, imgs.data_ptr())
    assert b.wide == (slabs == 0)
    e.close()
    for call in (b.launch, b.check):
        with pytest.raises(api.SvdiError) as ei:
            call()
        assert ei.value.status == 1
    b.close()
