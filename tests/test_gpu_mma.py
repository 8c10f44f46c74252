"""The matrix-instruction gridder (8 x 8 tiles, automatic tile size, support 6 and 8) against the oracle.

Positions cover what its dispatch and its edges can get wrong: tiles that the grid cuts (G not a
multiple of 8, odd G), footprints clipped at both grid edges, exactly integer positions, tiles of one
record and of many (chunks shared by several warps, a tile split over several), neighbouring and
distant tiles, and every split of the Chebyshev terms over its 4-, 2- and 1-term variants.

Tolerance: a contribution is off by at most (2 * 1.2e-7 + 3 * 2^-22) of the kernel's peak times |v|
(FP32 piecewise polynomials of both axes; FP16 hi + lo splits of both factors and the dropped lo * lo
product), about 1e-6; the planes are held to the 4e-6 relative L2 of the other gridders' tests."""
import numpy as np
import pytest

from oracle import oracle as O
from svdimager_b200 import api

pytestmark = pytest.mark.gpu

GRID_TOL = 4e-6
W_BETA = {8: O.REF_BETA, 6: O.REF_BETA * 0.75}


def _samples(rng, n, G, spread):
    """n positions in grid cells: a dense core, rows of neighbouring tiles, the whole grid and beyond its
    edges, and some exactly integer ones."""
    p = np.empty((n, 2))
    a, b, c = n // 3, n // 2, (9 * n) // 10
    p[:a] = rng.normal(0.0, spread, (a, 2))
    p[a:b, 0] = rng.uniform(-1.0, 1.0, b - a)
    p[a:b, 1] = rng.uniform(-G / 2, G / 2, b - a)
    p[b:c] = rng.uniform(-1.0, 1.0, (c - b, 2)) * (G / 2 + 3)
    p[c:] = rng.uniform(-1.0, 1.0, (n - c, 2)) * (G / 2 + 3)
    p[c::3, 0] = np.round(p[c::3, 0])
    p[c::4] = np.round(p[c::4])
    return p


def _run(n, N, W, K, seed=3, spread=3.0):
    cell, G = 2e-3, (3 * N + 1) // 2
    scale = float(np.float32(cell)) * G
    rng = np.random.default_rng(seed)
    b = np.concatenate([_samples(rng, n, G, spread) / scale, rng.uniform(-40.0, 40.0, (n, 1))], axis=1)
    b = b.astype(np.float32)
    vr, vi = (rng.normal(size=n).astype(np.float32) for _ in range(2))
    v = np.eye(3, dtype=np.float32)
    v[0], v[1] = [0.8, 0.6, 0.0], [-0.6, 0.8, 0.0]
    opt = dict(coord_mode=api.COORD_REF32, keep_grid=1, k_rule=api.KRULE_FIXED, fixed_k=K, support=W, beta=W_BETA[W])
    with api.Engine(api.archive_options(**opt)) as e:
        e.fipipe(vr, vi, b, v, N, cell)
        st = e.stats()
        grid = e.buffer(api.BUF_GRID).reshape(K, G, G)
    assert st["tile"] == 8 and st["num_terms"] == K
    sc = O.SlabConfig(st["slab_r3_min"], st["r3_max"], st["max_abs_t3"], st["alpha_max"], 1, st["slab_width"],
                      st["slab_half"], 1.0 / st["slab_half"], st["slab_alpha_max"], K)
    ref = O.grid(b.astype(np.float64), vr, vi, scale, G, sc, 1.0 / (0.8 * 0.8 + 0.6 * 0.6), W=W, beta=W_BETA[W],
                 coord_mode=1)
    return grid, ref


@pytest.mark.parametrize("n,N,W,K", [
    (1, 16, 8, 1), (33, 16, 8, 2), (700, 37, 8, 1), (5000, 100, 8, 3), (5000, 90, 6, 1), (4000, 99, 6, 2),
    (20000, 64, 8, 4), (9000, 61, 8, 5), (6000, 85, 6, 7), (300, 255, 8, 1)])
def test_planes_match_oracle(cuda_device, n, N, W, K):
    grid, ref = _run(n, N, W, K)
    for k in range(K):
        den = np.linalg.norm(ref[k])
        err = np.linalg.norm(grid[k] - ref[k])
        assert err <= GRID_TOL * den, (k, err, den)


@pytest.mark.parametrize("n", [113_663, 600_000, 2_100_000])
def test_long_runs_match_oracle(cuda_device, n):
    """The chunk sizes (32, 64 and 256 records), most tiles split over many chunks."""
    grid, ref = _run(n, 48, 8, 1, spread=12.0)
    assert np.linalg.norm(grid[0] - ref[0]) <= GRID_TOL * np.linalg.norm(ref[0])


@pytest.mark.parametrize("calls", [((200_000, 1),), ((200_000, 3), (130_003, 6), (200_000, 3))])
def test_dense_tile_rounding(cuda_device, calls):
    """Coherent samples of one tile (the sums of 32 chunks are formed apart), several shapes in turn on one
    engine. Tolerance: n / 2048 sums and at most 62 single chunks are added to a cell, 160 FP32 additions of rms
    error 0.29 * 2^-23 at up to the whole sum, 2.5e-7; the two polynomials 1.2e-7 each, the splits 2e-7, in
    squares 3.7e-7, of which 6e-7 leaves room for their all having one sign. (Added chunk by chunk: 1.1e-6.)"""
    N, cell, G = 64, 2e-3, 96
    scale = float(np.float32(cell)) * G
    v = np.eye(3, dtype=np.float32)
    v[0], v[1] = [0.8, 0.6, 0.0], [-0.6, 0.8, 0.0]
    engines = {}
    try:
        for call, (n, K) in enumerate(calls):
            rng = np.random.default_rng(call)
            p = np.clip(rng.normal(3.6, 0.7, (n, 2)), 1.0, 6.0)
            b = np.concatenate([p / scale, rng.uniform(-40.0, 40.0, (n, 1))], axis=1).astype(np.float32)
            vr, vi = ((c + 0.1 * rng.normal(size=n)).astype(np.float32) for c in (1.0, 0.3))
            if K not in engines:
                engines[K] = api.Engine(api.archive_options(coord_mode=api.COORD_REF32, keep_grid=1, fixed_k=K,
                                                            k_rule=api.KRULE_FIXED))
            e = engines[K]
            e.fipipe(vr, vi, b, v, N, cell)
            st = e.stats()
            grid = e.buffer(api.BUF_GRID).reshape(K, G, G)
            sc = O.SlabConfig(st["slab_r3_min"], st["r3_max"], st["max_abs_t3"], st["alpha_max"], 1, st["slab_width"],
                              st["slab_half"], 1.0 / st["slab_half"], st["slab_alpha_max"], K)
            ref = O.grid(b.astype(np.float64), vr, vi, scale, G, sc, 1.0, W=8, coord_mode=1)
            assert np.linalg.norm(grid[0] - ref[0]) <= 6e-7 * np.linalg.norm(ref[0])
            for k in range(1, K):  # odd terms nearly cancel over the symmetric w range
                assert np.linalg.norm(grid[k] - ref[k]) <= 6e-7 * np.linalg.norm(ref[0])
    finally:
        for e in engines.values():
            e.close()


@pytest.mark.parametrize("N,nslab", [(2048, 3), (2048, 2), (777, 3)])
def test_distant_keys(cuda_device, N, nslab):
    """A compact array in several w-slabs: a few tiles of each slab hold records, the keys between them (147,456 of
    a 3072^2 grid per slab) are empty. The planes against those of 32 x 32 tiles, each within GRID_TOL of the exact
    ones; and a slab more costs a slab's gridding, not a walk over its keys: nslab times that of one slab, and 0.1 ms
    for launches and noise."""
    import dataclasses
    from tests.conftest import snapshot
    s = snapshot("small", image_size=N, cell_size=0.1 / N)
    uvw = s.uvw * np.float32(0.01)
    uvw[:, 2] = np.random.default_rng(2).uniform(-0.2, 0.2, len(uvw)) * uvw[:, 0].std()  # records in every slab
    s = dataclasses.replace(s, uvw=uvw)
    opt = dict(k_rule=api.KRULE_FIXED, fixed_k=1)

    def grid_ms(e):
        ms = []
        for _ in range(9):
            e.image(s)
            ms.append(e.stats()["ms_grid"])
        return float(np.median(ms)), e.stats()

    with api.Engine(**opt) as e:
        one, st = grid_ms(e)
        assert st["num_slabs"] == 1
    opt["target_alpha"] = st["alpha_max"] / (nslab - 0.5)
    with api.Engine(**opt) as e:
        ms, st = grid_ms(e)
        assert st["num_slabs"] == nslab and st["tile"] == 8
    planes = []
    for tile in (0, 32):
        with api.Engine(keep_grid=1, tile=tile, **opt) as e:
            e.image(s)
            planes.append(e.buffer(api.BUF_GRID).reshape(nslab, -1))
    for a, b in zip(*planes):
        assert np.linalg.norm(a - b) <= 2 * GRID_TOL * np.linalg.norm(b) > 0
    assert ms <= nslab * one + 0.1, (ms, one)


@pytest.mark.parametrize("n,N,W,K", [(70, 48, 8, 1), (5000, 48, 8, 2), (5000, 61, 6, 3), (40_000, 64, 8, 8)])
def test_samples_at_one_position(cuda_device, n, N, W, K):
    """Many samples at the origin, among others on exact cells at the same place of neighbouring tiles and on the low
    edge, in every batch and with different w: summed where position, tile and w agree."""
    cell, G = 2e-3, (3 * N + 1) // 2
    scale = float(np.float32(cell)) * G
    rng = np.random.default_rng(n + K)
    p = rng.uniform(-1.0, 1.0, (n, 2)) * 14.0
    p[rng.random(n) < 0.5] = 0.0
    other = rng.random(n) < 0.2
    p[other] = 8.0 * rng.integers(-2, 3, (int(other.sum()), 2))
    low = rng.random(n) < 0.05
    p[low] = -(G // 2) + rng.integers(0, 3, (int(low.sum()), 2)) + 0.25
    w = np.where(rng.random(n) < 0.7, 0.0, rng.choice([-30.0, 12.5, 40.0], n))
    b = np.concatenate([p / scale, w[:, None]], axis=1).astype(np.float32)
    vr, vi = (rng.normal(size=n).astype(np.float32) for _ in range(2))
    opt = dict(coord_mode=api.COORD_REF32, keep_grid=1, k_rule=api.KRULE_FIXED, fixed_k=K, support=W, beta=W_BETA[W])
    with api.Engine(api.archive_options(**opt)) as e:
        e.fipipe(vr, vi, b, np.eye(3, dtype=np.float32), N, cell)
        st = e.stats()
        grid = e.buffer(api.BUF_GRID).reshape(K, G, G)
    sc = O.SlabConfig(st["slab_r3_min"], st["r3_max"], st["max_abs_t3"], st["alpha_max"], 1, st["slab_width"],
                      st["slab_half"], 1.0 / st["slab_half"], st["slab_alpha_max"], K)
    ref = O.grid(b.astype(np.float64), vr, vi, scale, G, sc, 1.0, W=W, beta=W_BETA[W], coord_mode=1)
    for k in range(K):
        assert np.linalg.norm(grid[k] - ref[k]) <= GRID_TOL * np.linalg.norm(ref[k]), k


@pytest.mark.parametrize("K", [1, 2, 8])
def test_autocorrelations_time(cuda_device, K):
    """A few per cent of autocorrelations (u = v = w = 0) cost a few per cent, not a chain of reductions on the origin's
    cells: twice the gridding and 0.02 ms are allowed (one after another: 3 to 7 times)."""
    import dataclasses
    from tests.conftest import snapshot
    s = snapshot("small", image_size=256, cell_size=0.1 / 256)
    uvw = s.uvw.copy()
    uvw[::32] = 0.0

    def grid_ms(e, s):
        ms = []
        for _ in range(9):
            e.image(s)
            ms.append(e.stats()["ms_grid"])
        return float(np.median(ms))

    with api.Engine(k_rule=api.KRULE_FIXED, fixed_k=K) as e:
        plain, autos = grid_ms(e, s), grid_ms(e, dataclasses.replace(s, uvw=uvw))
    assert autos <= 2 * plain + 0.02, (autos, plain)
