"""The two-step entry's idle engines: buffers taken over from an earlier descriptor give the images of a fresh
engine, whatever the shapes in between, with several descriptors live at once and from several threads.

Tolerance 1e-6 relative RMS: the order of floating-point atomic adds (as in the other repeat tests)."""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from svdimager_b200 import api
from tests.conftest import snapshot

pytestmark = pytest.mark.gpu

SHAPES = ((16, 8128, 256), (2, 500, 64), (16, 8128, 256), (5, 3000, 128))


def _two_step(s, want_bin=False):
    b = api.preprocess_measurement_set_gpu(s, want_bin=want_bin)
    assert bool(b.buf.d_bin) == want_bin
    img = api.FIpipeDevice(b, s.image_size, s.cell_size)
    api.free_device_preprocess_buffers(b)
    return img


@pytest.fixture(scope="module")
def cases():
    out = []
    for nchan, rows, N in SHAPES:
        s = snapshot("small", nchan=nchan, n_rows_limit=rows, image_size=N, cell_size=0.1 / N)
        with api.Engine() as e:
            out.append((s, e.image(s)))
    return out


def test_taken_over_engines_match_fresh_ones(cuda_device, cases):
    for i, (s, ref) in enumerate(cases * 2):
        assert O.rel_rms(_two_step(s, want_bin=i % 3 == 0), ref) < 1e-6, i


def test_live_descriptors_keep_their_buffers(cuda_device, cases):
    """More descriptors than idle engines, imaged after all of them were filled, twice over."""
    for _ in range(2):
        live = [(api.preprocess_measurement_set_gpu(s), s, ref) for s, ref in cases]
        assert len({b.buf.d_vis_real for b, _, _ in live}) == len(live)
        for b, s, ref in live:
            assert O.rel_rms(api.FIpipeDevice(b, s.image_size, s.cell_size), ref) < 1e-6
        for b, _, _ in live:
            b.free()


def test_threads(cuda_device, cases):
    errors = []

    def work(k):
        try:
            for i in range(6):
                s, ref = cases[(k + i) % len(cases)]
                err = O.rel_rms(_two_step(s), ref)
                if not err < 1e-6:
                    errors.append((k, i, err))
        except Exception as ex:  # noqa: BLE001
            errors.append((k, repr(ex)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_idle_memory_is_bounded_and_given_back(cuda_device, cases):
    """One descriptor imaged at many sizes with large prime factors, whose FFT plans hold work areas: what stays
    after it is freed is within the stated 1 GiB (5 % for what the driver rounds up), and nothing stays after the
    release (64 MB for what CUDA and cuFFT load once)."""
    import torch
    s, _ = cases[1]
    api.release_idle_engines()
    b = api.preprocess_measurement_set_gpu(s)
    api.FIpipeDevice(b, 64, s.cell_size)
    b.free()
    api.release_idle_engines()
    free = torch.cuda.mem_get_info()[0]
    b = api.preprocess_measurement_set_gpu(s)
    for N in range(501, 1181, 8):
        api.FIpipeDevice(b, N, 0.05 / N)
    b.free()
    assert free - torch.cuda.mem_get_info()[0] <= 1.05 * (1 << 30)
    api.release_idle_engines()
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_freeing_waits_for_the_callers_streams(cuda_device, cases):
    """Work that the caller has queued on a descriptor's arrays reads them, not the next snapshot's."""
    import dataclasses
    import torch

    class View:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3)

    s, _ = cases[0]
    other = dataclasses.replace(s, vis0_real=s.vis0_real + 1.0, vis3_real=s.vis3_real + 1.0)
    api.preprocess_measurement_set_gpu(s).free()
    b = api.preprocess_measurement_set_gpu(s)
    ref = torch.as_tensor(View(b.buf.d_vis_real, s.num_samples), device="cuda").clone()
    got = torch.zeros_like(ref)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)  # some 0.1 s
        got.copy_(torch.as_tensor(View(b.buf.d_vis_real, s.num_samples), device="cuda"))
    b.free()
    c = api.preprocess_measurement_set_gpu(other)
    torch.cuda.synchronize()
    c.free()
    assert torch.equal(got, ref)


def test_taken_over_engines_keep_no_answers(cuda_device, cases):
    """A snapshot imaged again on a taken-over engine launches what it launches on a new one."""
    s, _ = cases[0]
    counts = []
    api.release_idle_engines()
    for _ in range(3):
        n0 = api.kernel_launch_count()
        _two_step(s)
        counts.append(api.kernel_launch_count() - n0)
    assert counts[1:] == counts[:1] * 2, counts


def test_freeing_beside_a_capture(cuda_device, cases):
    """Another thread captures a CUDA graph while a descriptor is freed: the capture is not broken, and the engine
    is still kept."""
    import torch
    s, ref = cases[1]
    api.release_idle_engines()
    b = api.preprocess_measurement_set_gpu(s)
    ptr = b.buf.d_vis_real
    x = torch.zeros(16, device="cuda")
    started, freed = threading.Event(), threading.Event()
    out = []

    def capture():
        g = torch.cuda.CUDAGraph()
        try:
            with torch.cuda.graph(g, capture_error_mode="thread_local"):
                x.add_(1.0)
                started.set()
                freed.wait(20)
                x.add_(1.0)
            out.append(g)
        except Exception as ex:  # noqa: BLE001
            started.set()
            out.append(ex)

    t = threading.Thread(target=capture)
    t.start()
    started.wait(20)
    b.free()
    freed.set()
    t.join()
    assert isinstance(out[0], torch.cuda.CUDAGraph), out[0]
    out[0].replay()
    torch.cuda.synchronize()
    assert torch.equal(x, torch.full_like(x, 2.0))
    c = api.preprocess_measurement_set_gpu(s)
    assert c.buf.d_vis_real == ptr  # the kept engine's arrays
    assert O.rel_rms(api.FIpipeDevice(c, s.image_size, s.cell_size), ref) < 1e-6
    c.free()
