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


@pytest.mark.parametrize("n,N,spread", [(40, 64, 0.3), (70_000, 64, 0.3), (70_001, 64, 6.0), (300_000, 1024, 0.3),
                                        (300_000, 1024, 25.0)])
def test_chunks_of_dense_keys(cuda_device, n, N, spread):
    """Keys that hold many of the gridder's chunks beside keys of few and of none, in one block of the scan and in
    several. The planes of all records are those of 32 x 32 tiles: a chunk under a wrong key would move its records.
    Tolerance: each gridder is held to 4e-6 of the exact planes by its own tests."""
    import numpy as np
    cell, G = 2e-3, (3 * N + 1) // 2
    scale = float(np.float32(cell)) * G
    rng = np.random.default_rng(n)
    p = rng.normal(0.0, spread, (n, 2))
    p[::97] = rng.uniform(-0.45, 0.45, (len(p[::97]), 2)) * G
    b = np.concatenate([p / scale, rng.uniform(-40.0, 40.0, (n, 1))], axis=1).astype(np.float32)
    vr, vi = (rng.normal(size=n).astype(np.float32) for _ in range(2))
    planes = []
    for tile in (0, 32):
        with api.Engine(api.archive_options(keep_grid=1, k_rule=api.KRULE_FIXED, fixed_k=1, tile=tile)) as e:
            e.fipipe(vr, vi, b, np.eye(3, dtype=np.float32), N, cell)
            planes.append(e.buffer(api.BUF_GRID))
    assert np.linalg.norm(planes[0] - planes[1]) <= 8e-6 * np.linalg.norm(planes[1])


def test_dense_core_binning_time(cuda_device):
    """2 M samples of one tile are binned like 2 M samples of many: the chunks of a dense key are not written one
    after another (2.4 times as long). Twice the time is allowed: its atomics fall on one address."""
    import dataclasses
    import numpy as np
    s = snapshot("small", image_size=512, cell_size=0.1 / 512, nchan=256)

    def bin_ms(e, s):
        ms = []
        for _ in range(9):
            e.image(s)
            ms.append(e.stats()["ms_bin"])
        return float(np.median(ms))

    with api.Engine(k_rule=api.KRULE_FIXED, fixed_k=1) as e:
        spread = bin_ms(e, s)
        dense = bin_ms(e, dataclasses.replace(s, uvw=s.uvw * np.float32(1e-3)))
    assert dense <= 2 * spread, (dense, spread)


@pytest.mark.parametrize("nchan,rows", [(1, 8128), (2, 8001), (3, 5000), (16, 1000), (17, 1000)])
@pytest.mark.parametrize("scale", [1e-3, 0.02])
def test_compact_array_bit_exact(cuda_device, nchan, rows, scale):
    """Rows of a warp that share a tile without being neighbours, for one to all of a warp's lanes per row."""
    import dataclasses
    import numpy as np
    s = snapshot("small", nchan=nchan, n_rows_limit=rows, image_size=256, cell_size=0.1 / 256)
    s = dataclasses.replace(s, uvw=s.uvw * np.float32(scale))
    with api.Engine() as e:
        for _ in range(2):
            e.image(s)
        r = O.expand_coords(e.buffer(api.BUF_Q).reshape(-1, 3), e.buffer(api.BUF_S))
        _check_binning(e, e.stats(), r, e.buffer(api.BUF_VIS_REAL), e.buffer(api.BUF_VIS_IMAG), s.cell_size, edge_mode=0)


def test_few_channels_binning_time(cuda_device):
    """1 M samples of one channel, all in a few tiles, are binned in at most 1.5 times what they take spread over
    the grid (3 times where each sample is an atomic of its own on one address)."""
    import dataclasses
    import numpy as np
    s = snapshot("precision", nchan=1, image_size=512, cell_size=0.1 / 512)
    rng = np.random.default_rng(1)
    uvw = np.concatenate([s.uvw] * 8) * rng.uniform(0.9, 1.0, (8 * s.num_rows, 1)).astype(np.float32)
    many = {k: np.concatenate([v] * 8) for k, v in s.arrays().items() if k not in ("uvw", "frequencies_hz")}
    s = dataclasses.replace(s, num_rows=len(uvw), uvw=uvw, **many)

    def bin_ms(e, s):
        ms = []
        for _ in range(9):
            e.image(s)
            ms.append(e.stats()["ms_bin"])
        return float(np.median(ms))

    limit = 0.45 * 512 / 0.1 / (170e6 / 299792458.0)  # the longest baseline inside the grid
    spread = dataclasses.replace(s, uvw=s.uvw * np.float32(limit / np.abs(uvw).max()))
    with api.Engine(k_rule=api.KRULE_FIXED, fixed_k=1) as e:
        wide, dense = bin_ms(e, spread), bin_ms(e, dataclasses.replace(spread, uvw=spread.uvw * np.float32(5e-3)))
    assert dense <= 1.5 * wide, (dense, wide)
