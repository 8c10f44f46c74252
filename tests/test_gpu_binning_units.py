"""Tile binning of separable sources over both unit sizes (4 and 16 rows per warp step), channel counts below,
at and above a warp's lanes, ragged rows, one block and several blocks of the key scan: bit-exact against the
oracle, like the other binning tests."""
import pytest

from oracle import oracle as O
from svdimager_b200 import api
from tests.conftest import snapshot
from tests.test_gpu_parity import _check_binning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan,rows,N,kw", [
    (1, 37, 64, {}), (2, 5, 64, {}), (3, 101, 96, {}), (16, 8128, 256, {}), (33, 77, 512, dict(tile=64)),
    (70, 32001, 640, dict(edge_mode=api.EDGE_STRICT)), (5, 3001, 1001, dict(k_rule=api.KRULE_FIXED, fixed_k=2)),
])
def test_binning_bit_exact(cuda_device, nchan, rows, N, kw):
    s = snapshot("batching" if rows > 8128 else "small", nchan=nchan, n_rows_limit=rows, image_size=N, cell_size=0.1 / N)
    with api.Engine(**kw) as e:
        for _ in range(2):  # the second call speculates: its counters are cleared and its plan made on the device
            e.image(s)
        r = O.expand_coords(e.buffer(api.BUF_Q).reshape(-1, 3), e.buffer(api.BUF_S))
        _check_binning(e, e.stats(), r, e.buffer(api.BUF_VIS_REAL), e.buffer(api.BUF_VIS_IMAG), s.cell_size,
                       edge_mode=kw.get("edge_mode", 0))
