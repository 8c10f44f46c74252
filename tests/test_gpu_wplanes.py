"""Imaging through w planes (error-target rule, 24 and more moment planes, not too many
samples per plane cell) against the FP64 DFT of the same
samples and against the Chebyshev form of the same call (an explicit tile size keeps that form).

Tolerance: the w kernel's largest error is 2e-7 (10 planes per sample) or 7e-9 (12), below the error target
1e-6 of either form; the images are held to the 1e-5 relative RMS of the other parity tests."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from svdimager_b200 import api
from tests.conftest import snapshot

pytestmark = pytest.mark.gpu

IMG_TOL = 1e-5


def _snap(N, nchan, rows, shift=0.0):
    """A wide-field snapshot of `rows` baselines whose w range needs many moment planes; `shift` adds a
    constant w (metres), so that all r3 have one sign."""
    s = snapshot("widefield", nchan=nchan, n_rows_limit=rows, image_size=N, cell_size=0.3 / N)
    if not shift:
        return s
    uvw = s.uvw.copy()
    uvw[:, 2] += np.float32(shift)
    return dataclasses.replace(s, uvw=uvw)


def _images(s, **kw):
    opt = dict(k_rule=api.KRULE_TARGET, target_error=1e-6, presplat=1)
    opt.update(kw)
    rng = np.random.default_rng(4)
    px, py = rng.integers(0, s.image_size, 400), rng.integers(0, s.image_size, 400)
    with api.Engine(**opt) as e:
        img = e.image(s)
        st = e.stats()
        dft = e.dft_pixels(px, py)
    with api.Engine(**dict(opt, tile=32)) as e:
        ref = e.image(s)
        rst = e.stats()
    return img, st, img[py, px], dft, ref, rst


@pytest.mark.parametrize("N,nchan,rows,kw", [
    (512, 4, 6000, dict(edge_mode=api.EDGE_STRICT)),
    (512, 4, 6000, dict(edge_mode=api.EDGE_STRICT, max_batch_slabs=1)),
    (256, 33, 700, dict(edge_mode=api.EDGE_STRICT, support=6, beta=0.75 * O.REF_BETA)),
    (500, 1, 9001, dict(edge_mode=api.EDGE_STRICT, target_error=1e-7)),
    (384, 5, 5000, dict(edge_mode=api.EDGE_STRICT, support=6, beta=0.75 * O.REF_BETA, target_error=1e-7)),
    (512, 7, 3000, dict()),
    (256, 8, 30000, dict(edge_mode=api.EDGE_STRICT)),
    (500, 1, 3, dict(edge_mode=api.EDGE_STRICT)),
])
def test_matches_dft_and_chebyshev_form(cuda_device, N, nchan, rows, kw):
    s = _snap(N, nchan, rows)
    img, st, at, dft, ref, rst = _images(s, **kw)
    assert st["num_planes"] == rst["num_planes"]
    assert st["num_gridded"] == rst["num_gridded"]
    m = np.isfinite(ref)
    assert np.array_equal(m, np.isfinite(img))
    tol = IMG_TOL if kw.get("support", 8) == 8 else 2e-4  # six taps at sigma 1.5 alias at 1e-4
    assert O.rel_rms(img[m], ref[m]) < IMG_TOL
    if kw.get("edge_mode") == api.EDGE_STRICT:  # clipped footprints are no samples of the DFT
        f = np.isfinite(dft)
        assert O.rel_rms(at[f], dft[f]) < tol


def test_blocks_of_many_parts(cuda_device):
    """Nine tenths of 240 k samples in a few blocks of cells: each is shared by hundreds of CTAs, beside blocks of one
    and of none."""
    s = _snap(256, 8, 30000)
    uvw = s.uvw.copy()
    uvw[np.arange(len(uvw)) % 10 != 0] *= np.float32(0.02)
    img, st, at, dft, ref, rst = _images(dataclasses.replace(s, uvw=uvw), edge_mode=api.EDGE_STRICT)
    assert st["num_gridded"] == rst["num_gridded"]
    f = np.isfinite(dft)
    assert O.rel_rms(at[f], dft[f]) < IMG_TOL


def test_one_signed_w_range(cuda_device):
    s = _snap(512, 4, 6000, shift=400.0)
    img, st, at, dft, ref, rst = _images(s, edge_mode=api.EDGE_STRICT)
    assert st["num_planes"] >= 48
    f = np.isfinite(dft)
    assert O.rel_rms(at[f], dft[f]) < IMG_TOL


def test_exactly_integer_positions_and_both_edges(cuda_device):
    """Baselines on exact grid cells and on the outermost cells that the clip rule keeps, on both sides (the
    mirrored ones wrap from +G/2 to -G/2)."""
    N = 128
    s = _snap(N, 1, 2000)
    cell = float(np.float32(s.cell_size))
    G = (3 * N + 1) // 2
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6) as e:
        e.image(s)
        vin = np.array(e.stats()["vin"]).reshape(3, 3)
    q = s.uvw.astype(np.float64) @ vin.T
    sc = float(s.frequencies_hz[0]) / 299792458.0
    scale = cell * G * sc
    rng = np.random.default_rng(8)
    cells = rng.integers(-G // 2 - 3, G // 2 + 4, (2000, 2))
    q[:, :2] = cells / scale
    q[::2, :2] += rng.uniform(0, 1, (1000, 2)) / scale
    t = dataclasses.replace(s, uvw=(q @ vin).astype(np.float32))
    img, st, _, _, ref, rst = _images(t)
    assert st["num_gridded"] == rst["num_gridded"] and st["num_planes"] == rst["num_planes"] >= 48
    m = np.isfinite(ref)
    assert O.rel_rms(img[m], ref[m]) < IMG_TOL


def test_buffers_and_next_calls(cuda_device):
    """The records and moments of a w-plane call are those of its Chebyshev form; asking for them changes
    neither the statistics nor the calls that follow."""
    s = _snap(256, 4, 3000)
    opt = dict(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT)
    with api.Engine(**opt) as e, api.Engine(keep_grid=1, **opt) as c:
        img = e.image(s)
        st = e.stats()
        ref = c.image(s)
        assert np.array_equal(e.buffer(api.BUF_OFFSETS), c.buffer(api.BUF_OFFSETS))
        a, b = e.buffer(api.BUF_RECORDS), c.buffer(api.BUF_RECORDS)
        order = ("vim", "vre", "yq", "xq")
        assert np.array_equal(np.sort(a, order=order), np.sort(b, order=order))
        assert len(e.buffer(api.BUF_RECORDS_S)) == len(a)
        ma, mb = e.buffer(api.BUF_MOMENTS), c.buffer(api.BUF_MOMENTS)
        assert ma.shape == mb.shape and np.linalg.norm(ma - mb) < 1e-5 * np.linalg.norm(mb)
        assert e.stats() == st
        again = e.image(s)
        assert O.rel_rms(again, img) < 1e-6 and O.rel_rms(img, ref) < IMG_TOL
        flat = snapshot("small")
        assert O.rel_rms(e.image(flat), c.image(flat)) < 1e-6  # a Chebyshev call after it


def test_reading_buffers_keeps_the_route(cuda_device):
    """The calls that follow a buffer read launch the kernels of the calls before it (the moments take others)."""
    s = _snap(256, 4, 3000)
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT) as e:
        def launches():
            n0 = api.kernel_launch_count()
            e.image(s)
            return api.kernel_launch_count() - n0

        e.image(s)
        before = launches()
        e.buffer(api.BUF_RECORDS)
        assert [launches() for _ in range(3)] == [before] * 3
        with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT, keep_grid=1) as c:
            c.image(s)
            n0 = api.kernel_launch_count()
            c.image(s)
            assert api.kernel_launch_count() - n0 != before


def test_reports_its_planes(cuda_device):
    """w_planes() is the number of planes of the last call, buffers read or not; 0 for the moments."""
    s = _snap(256, 4, 3000)
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT) as e:
        assert e.w_planes() == 0
        e.image(s)
        n, st = e.w_planes(), e.stats()
        # W = 10 planes and one per 1 / (3 max|t3|) of |r3|
        hi = max(abs(st["r3_min"]), abs(st["r3_max"]))
        assert n == int(hi * 3.0 * st["max_abs_t3"] * (1 + 1e-12)) + 10 < st["num_planes"]
        e.buffer(api.BUF_RECORDS)
        assert e.w_planes() == n
        e.image(snapshot("small"))
        assert e.w_planes() == 0
        e.image(s)
        assert e.w_planes() == n


@pytest.mark.parametrize("batch", [0, 1])
def test_stage_times(cuda_device, batch):
    """Every stage of a call through w planes has its time, with the planes in one batch or several."""
    s = _snap(256, 4, 3000)
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT, max_batch_slabs=batch) as e:
        e.image(s)
        st = e.stats()
        assert e.w_planes() > 0
        stages = [st["ms_" + k] for k in ("preprocess", "bin", "grid", "fft", "image")]
        assert min(stages) > 0 and sum(stages) <= st["ms_total"] * 1.01, (stages, st["ms_total"])


def test_failed_call_after_w_planes(cuda_device):
    """A call that fails has overwritten the inputs that the last call's records and moments would be made from:
    there are none then, rather than some of other inputs, and the next call is as before."""
    s = _snap(256, 4, 3000)
    bad = dataclasses.replace(s, uvw=np.full_like(s.uvw, np.nan))
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT) as e:
        img = e.image(s)
        with pytest.raises(api.SvdiError):
            e.image(bad)
        assert all(len(e.buffer(b)) == 0 for b in (api.BUF_OFFSETS, api.BUF_RECORDS, api.BUF_RECORDS_S, api.BUF_MOMENTS))
        assert O.rel_rms(e.image(s), img) < 1e-6
        assert len(e.buffer(api.BUF_RECORDS)) == e.stats()["num_gridded"] > 0


def test_many_w_ranges_on_one_engine(cuda_device):
    """Snapshots of changing w range need another number of planes each (about 90 numbers here). The engine keeps
    the row plans of the last 32: after 40 numbers a new plan takes an old one's place, up to the fragments of a few
    2 MB allocations."""
    import torch
    s = _snap(512, 2, 4000)
    free = []
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_STRICT) as e:
        for f in np.linspace(1.0, 0.3, 96):  # all baselines shorter: the same rotation, a smaller w range
            e.image(dataclasses.replace(s, uvw=s.uvw * np.float32(f)))
            assert e.stats()["num_planes"] >= 24
            free.append(torch.cuda.mem_get_info()[0])
    assert free[39] - min(free[40:]) <= 8 << 20


def test_non_finite_visibility(cuda_device):
    s = _snap(256, 4, 3000)
    v = s.vis0_real.copy()
    row = np.argmin(np.hypot(s.uvw[:, 0], s.uvw[:, 1]) + 1e9 * (s.flag0[:s.num_rows] != 0))
    v[row] = np.nan  # channel 0 of an unflagged short baseline
    t = dataclasses.replace(s, vis0_real=v)
    with api.Engine(k_rule=api.KRULE_TARGET, target_error=1e-6, edge_mode=api.EDGE_CLIP) as e:
        img = e.image(t)
        ok = e.image(s)
    assert np.isnan(img).any() and np.array_equal(np.isnan(img), ok != 0)
