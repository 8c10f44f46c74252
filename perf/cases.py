"""The imaging work that the framework is timed on.

Each case is one use of the public interface on seeded synthetic snapshots: an array of stations
(baselines = all pairs), a number of channels, a point-source sky with noise, WEIGHT_SPECTRUM and
flags, imaged to image_size^2 pixels over a field of `field` radians. `kind` names the entry:

  device    Engine.image_device: the snapshot and the image stay on the GPU
  batch     Batch.launch: many snapshots of mixed channel counts, one launch
  host      Engine.image: numpy arrays in, numpy image out
  fipipe    FIpipe: the archive entry on collapsed visibilities and rotated baselines (numpy)
  two_step  preprocess_measurement_set_gpu, FIpipeDevice, free_device_preprocess_buffers (numpy)
  server    Server.submit / wait: several requests of different sizes in flight (numpy)

`rule` is the Chebyshev rule ("bucket": the default of the main path, "target": the error target
1e-6), `edge` the grid-edge rule, `support` and `sigma` the gridding kernel and the oversampling
(the kernel's beta follows from them). `layout`: "disk" (stations in a disk), "arms" (half of them
in a core, half on log-spaced radii), "wide" (arms with station heights, observed far from the
zenith: many w planes). `reach` is the longest baseline's |u| over the grid's half width: above 1 the
outermost baselines leave the grid (strict edges drop them).
"""
import math

import numpy as np
import torch

from svdimager_b200 import api

C_LIGHT = 299792458.0
ARRAY_CENTER_X = 5.1e6
LATITUDE = math.radians(-30.0)
EARTH_RADIUS = 6.371e6
REF_SUPPORT, REF_SIGMA, REF_BETA = 8, 1.5, 15.3704324328
TARGET = 1e-6


def _case(kind, stations, channels, image, field, layout="disk", reach=0.9, rule="target", edge="strict",
          flags=0.05, support=REF_SUPPORT, sigma=REF_SIGMA, snapshots=1):
    return dict(kind=kind, stations=stations, channels=channels, image=image, field=field, layout=layout,
                reach=reach, rule=rule, edge=edge, flags=flags, support=support, sigma=sigma,
                snapshots=snapshots)


def listed():
    cases = {
        # a quick look from a compact array: the smallest call, its latency is what counts
        "device_192": _case("device", 64, 12, 192, 0.08, reach=0.6, rule="bucket", edge="clip"),
        # the small configuration (128 stations, 16 channels, 256^2) with the main path's defaults
        "device_256": _case("device", 128, 16, 256, 0.1, rule="bucket", edge="clip"),
        # odd sizes: 221 stations, 47 channels, a 1001^2 image
        "device_1001": _case("device", 221, 47, 1001, 0.1, layout="arms", reach=0.95, rule="bucket", edge="clip",
                            flags=0.2),
        # one snapshot of the batching configuration (256 stations, 1024^2)
        "device_1024": _case("device", 256, 32, 1024, 0.1, layout="arms", reach=1.4, flags=0.2),
        # a kernel the autotuner offers: support 6 at oversampling 2
        "device_1024_w6": _case("device", 256, 32, 1024, 0.1, layout="arms", reach=1.4, flags=0.2, support=6,
                                sigma=2.0),
        # the precision configuration (512 stations, 64 channels, 2048^2)
        "device_2048": _case("device", 512, 64, 2048, 0.1024, layout="arms", reach=4.0),
        # wide fields: many w planes, at a moderate size and as the wide-field configuration (4096^2)
        "wide_1536": _case("device", 200, 32, 1536, 0.3, layout="wide", reach=0.9),
        "wide_4096": _case("device", 512, 64, 4096, 0.3, layout="wide", reach=6.0),
        # a stretch of the batching configuration: 32 snapshots of 16, 32 and 64 channels in one launch
        "batch_32": _case("batch", 256, 64, 1024, 0.1, layout="arms", reach=1.4, flags=0.2, snapshots=32),
        # the archive entry and the two-step entry, as callers of the reference use them
        "fipipe_1024": _case("fipipe", 200, 32, 1024, 0.1, layout="arms", reach=0.9, rule="min", edge="clip"),
        "two_step_512": _case("two_step", 128, 16, 512, 0.1, reach=0.9, rule="bucket", edge="clip"),
        # a server under a burst of requests of mixed sizes
        "server_6": _case("server", 256, 32, 1024, 0.1, layout="arms", reach=1.4, snapshots=6),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "device", "device", "wide", "batch", "host", "fipipe",
                       "two_step", "server"])
    stations = _log_int(rng, 24, 400)
    channels = _log_int(rng, 1, 64)
    image = _log_int(rng, 128, 2048)
    # most users take round sizes; the others here have an even grid ceil(1.5 image) like them (the
    # reference's indexing of an odd grid shifts the rows of the image)
    image -= image % 8 if rng.random() < 0.6 else max(0, image % 4 - 1)
    layout = rng.choice(["disk", "arms"])
    inside = kind in ("fipipe", "two_step") or rng.random() < 0.4
    # under the reference's clipping rule arrays are laid out inside the grid
    reach = rng.uniform(0.3, 0.95) if inside else math.exp(rng.uniform(math.log(0.7), math.log(4.0)))
    edge = "clip" if inside else "strict"
    rule = {"fipipe": "min", "two_step": "bucket"}.get(kind) or rng.choice(["bucket", "target", "target"])
    support, sigma, field, snapshots = REF_SUPPORT, REF_SIGMA, rng.uniform(0.04, 0.15), 1
    if kind == "device" and rng.random() < 0.3:
        support, sigma = rng.choice([(6, 2.0), (8, 1.75), (10, 1.5), (12, 1.5), (10, 1.25)])
    if kind == "wide":
        kind, layout, rule, edge = "device", "wide", "target", "strict"
        stations, image, field = min(stations, 200), min(image, 1536), rng.uniform(0.15, 0.3)
        reach = rng.uniform(0.7, 1.5)
    if kind == "batch":
        stations, image, snapshots = min(stations, 256), min(image, 1024), rng.choice([5, 12, 24])
        layout, reach, edge, rule = "arms", rng.uniform(0.7, 2.0), "strict", "target"
    if kind == "server":
        stations, image, snapshots = min(stations, 200), min(image, 1024), rng.choice([3, 6])
        edge, rule, reach = "strict", "target", min(reach, 1.4)
    return _case(kind, stations, channels, image, field, layout, reach, rule, edge, rng.uniform(0.0, 0.4), support,
                 sigma, snapshots)


# ---- inputs ------------------------------------------------------------------------------------
def _beta(case):
    w, s = case["support"], case["sigma"]
    if (w, s) == (REF_SUPPORT, REF_SIGMA):
        return REF_BETA
    return REF_BETA * (w / 8.0) * (1.0 - 1.0 / (2.0 * s)) / (1.0 - 1.0 / 3.0)


def _parts(case):
    """The snapshots of a case: (stations, channels, image size) of each."""
    n = case["snapshots"]
    if case["kind"] == "batch":  # the batching configuration mixes 16, 32 and 64 channels
        return [(case["stations"], max(1, case["channels"] >> (i % 3)), case["image"]) for i in range(n)]
    if case["kind"] == "server":  # requests of full, half and quarter size
        return [(max(8, case["stations"] >> (i % 3)), case["channels"], max(64, case["image"] >> (i % 3)))
                for i in range(n)]
    return [(case["stations"], case["channels"], case["image"])] * n


def _snapshot(case, part, seed, index):
    """One snapshot on the GPU: a dict of tensors named as in HostMeasurementSetData, plus rows and
    channels."""
    stations, nchan, image = part
    g = torch.Generator(device="cuda").manual_seed((seed * 64 + index) % (1 << 62))

    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)

    # metres of the longest baseline that `reach` times the grid's half width stands for
    f_lo, f_hi = 140e6, 170e6
    b_max = case["reach"] * 0.5 * image / case["field"] * (C_LIGHT / f_hi)
    r_max = 0.5 * b_max
    theta = 2 * math.pi * rand(stations)
    radius = r_max * torch.sqrt(rand(stations))
    if case["layout"] != "disk":
        core = stations // 2
        radius[:core] = 0.12 * r_max * torch.sqrt(rand(core))
        radius[core:] = r_max * torch.exp(torch.linspace(math.log(0.12), 0.0, stations - core, device="cuda",
                                                         dtype=torch.float64))
    east, north = radius * torch.cos(theta), radius * torch.sin(theta)
    up = torch.zeros_like(east)
    declination = -30.0
    if case["layout"] == "wide":
        up = -radius ** 2 / (2 * EARTH_RADIUS) + 10.0 * randn(stations).double()
        declination = 30.0
    sl, cl = math.sin(LATITUDE), math.cos(LATITUDE)
    xyz = torch.stack([-sl * north + cl * up, east, cl * north + sl * up], dim=1)
    i, j = torch.triu_indices(stations, stations, 1, device="cuda")
    base = xyz[j] - xyz[i]
    ha = (float(rand(1)) - 0.5) * (math.pi / 3)
    dec = math.radians(declination)
    sh, ch, sd, cd = math.sin(ha), math.cos(ha), math.sin(dec), math.cos(dec)
    uvw = torch.stack([sh * base[:, 0] + ch * base[:, 1],
                       -sd * ch * base[:, 0] + sd * sh * base[:, 1] + cd * base[:, 2],
                       cd * ch * base[:, 0] - cd * sh * base[:, 1] + sd * base[:, 2]], dim=1)
    rows = uvw.shape[0]
    freq = torch.linspace(f_lo, f_hi, nchan, device="cuda", dtype=torch.float64)
    flux = torch.exp(math.log(0.1) + math.log(100.0) * rand(12))
    lm = (rand(12, 2) - 0.5) * case["field"]
    vis = torch.zeros(2, nchan, rows, device="cuda", dtype=torch.float32)  # re, im, channel-major
    for k in range(12):
        l, m = float(lm[k, 0]), float(lm[k, 1])
        turns = torch.outer(freq / C_LIGHT, uvw[:, 0] * l + uvw[:, 1] * m
                            + uvw[:, 2] * (math.sqrt(1 - l * l - m * m) - 1))
        phase = ((turns - torch.round(turns)) * (-2 * math.pi)).float()
        vis[0] += float(flux[k]) * torch.cos(phase)
        vis[1] += float(flux[k]) * torch.sin(phase)
    sigma = 0.05 / math.sqrt(2.0)
    n = rows * nchan
    # whole rows (an antenna pair) and single samples are flagged
    flag = (rand(1, rows) < 0.25 * case["flags"]) | (rand(nchan, rows) < 0.75 * case["flags"])
    flag = flag.to(torch.uint8).reshape(n)
    out = dict(uvw=uvw.float().contiguous(), frequencies_hz=freq.float())
    for p in (0, 3):
        out[f"vis{p}_real"] = (vis[0] + sigma * randn(nchan, rows)).reshape(n)
        out[f"vis{p}_imag"] = (vis[1] + sigma * randn(nchan, rows)).reshape(n)
        out[f"flag{p}"] = flag.clone()
        out[f"weight{p}"] = (0.5 + 0.5 * rand(n)).float()
    out.update(rows=rows, channels=nchan, image=image)
    return out


def _snapshots(case, seed):
    return [_snapshot(case, part, seed, i) for i, part in enumerate(_parts(case))]


class _Host:
    """A snapshot in host memory, with the fields the library reads."""

    def __init__(self, case, snap):
        self.num_rows, self.num_channels = snap["rows"], snap["channels"]
        self.array_center_x = ARRAY_CENTER_X
        self.image_size, self.cell_size = snap["image"], case["field"] / snap["image"]
        for k, v in snap.items():
            if isinstance(v, torch.Tensor):
                setattr(self, k, v.cpu().numpy())


def _collapse(snap, dtype):
    w0 = snap["weight0"].to(dtype) * (snap["flag0"] == 0)
    w3 = snap["weight3"].to(dtype) * (snap["flag3"] == 0)
    ws = w0 + w3
    inv = torch.where(ws > 0, 1.0 / ws, torch.zeros_like(ws))
    return [(snap["vis0_" + p].to(dtype) * w0 + snap["vis3_" + p].to(dtype) * w3) * inv for p in ("real", "imag")]


def _basis(snap):
    """The rotation of a snapshot's baselines (64 bits): principal axes by descending variance, row
    0 with a non-negative u, row 1 with a v of the array centre's sign, row 2 = row 0 x row 1."""
    u = snap["uvw"].double()
    s = snap["frequencies_hz"].double() / C_LIGHT
    n = u.shape[0] * s.shape[0]
    mean = u.sum(0) * s.sum() / n
    cov = (u.T @ u) * (s * s).sum() - n * torch.outer(mean, mean)
    vec = np.linalg.eigh(cov.cpu().numpy())[1]
    a, b = vec[:, 2].copy(), vec[:, 1].copy()
    if a[0] < 0:
        a = -a
    if b[1] * ARRAY_CENTER_X < 0:
        b = -b
    c = np.cross(a, b)
    return np.stack([a, b, c / np.linalg.norm(c)])


def _quartet(case, snap):
    """The archive entry's inputs (float32) on the GPU: visibilities, rotated baselines, basis."""
    vre, vim = _collapse(snap, torch.float32)
    vin = _basis(snap).astype(np.float32)
    q = snap["uvw"].double() @ torch.as_tensor(_basis(snap), device="cuda").T
    s = snap["frequencies_hz"].double() / C_LIGHT
    coords = (s[:, None, None] * q[None]).reshape(-1, 3).float().contiguous()
    return vre.contiguous(), vim.contiguous(), coords, vin


def _options(case):
    return dict(support=case["support"], sigma=case["sigma"], beta=_beta(case),
                edge_mode=api.EDGE_CLIP if case["edge"] == "clip" else api.EDGE_STRICT,
                k_rule=api.KRULE_TARGET if case["rule"] == "target" else api.KRULE_BUCKET, target_error=TARGET)


def prepare(case, seed):
    kind = case["kind"]
    snaps = _snapshots(case, seed)
    st = dict(kind=kind, cell=case["field"] / case["image"])
    if kind in ("device", "batch"):
        N = case["image"]
        st["snaps"] = snaps
        st["ms"] = [api.device_ms(s["rows"], s["channels"], s, ARRAY_CENTER_X) for s in snaps]
        st["out"] = torch.zeros(len(snaps), N, N, device="cuda")
        torch.cuda.synchronize()
        st["engine"] = api.Engine(**_options(case))
        if kind == "batch":
            st["batch"] = api.Batch(st["engine"], st["ms"], N, st["cell"], st["out"].data_ptr())
    elif kind == "fipipe":
        vre, vim, coords, vin = _quartet(case, snaps[0])
        st["quartet"] = (vre.cpu().numpy(), vim.cpu().numpy(), coords.cpu().numpy(), vin)
        st["image"] = case["image"]
    else:
        st["host"] = [_Host(case, s) for s in snaps]
        if kind == "host":
            st["engine"] = api.Engine(**_options(case))
        elif kind == "server":
            st["server"] = api.Server(num_slots=3, hbm_budget=16 << 30, **_options(case))
    return st


def run(state):
    kind = state["kind"]
    if kind == "device":
        state["engine"].image_device(state["ms"][0], state["out"].shape[1], state["cell"], state["out"].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return state["out"][0]
    if kind == "batch":
        state["batch"].launch(torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "fipipe":
        return api.FIpipe(*state["quartet"], state["image"], state["cell"])
    if kind == "host":
        return state["engine"].image(state["host"][0])
    if kind == "two_step":
        h = state["host"][0]
        buffers = api.preprocess_measurement_set_gpu(h)
        image = api.FIpipeDevice(buffers, h.image_size, h.cell_size)
        api.free_device_preprocess_buffers(buffers)
        return image
    tickets = [state["server"].submit(h) for h in state["host"]]
    return [state["server"].wait(t)[0] for t in tickets]


def work(case):
    """Inputs read once, images written once; the gridding of one moment plane and its FFT."""
    total_bytes = flops = 0.0
    for stations, nchan, N in _parts(case):
        rows = stations * (stations - 1) // 2
        n = rows * nchan
        per_sample = 20 if case["kind"] == "fipipe" else 26
        total_bytes += per_sample * n + (0 if case["kind"] == "fipipe" else 12 * rows) + 4 * nchan + 4 * N * N
        G = case["sigma"] * N
        flops += 4.0 * case["support"] ** 2 * n + 10.0 * G * G * math.log2(G)
    return {"bytes": total_bytes, "flops": flops}


# ---- the images in 64 bits ---------------------------------------------------------------------
class _Kernel:
    """An ES kernel of 12 cells at oversampling 2 and its Fourier transform (about 1e-11)."""

    W, SIGMA = 12, 2.0
    BETA = 2.3 * 12

    def __call__(self, x):
        z = torch.clamp(1.0 - (2.0 * x / self.W) ** 2, min=0.0)
        return torch.where(z > 0, torch.exp(self.BETA * (torch.sqrt(z) - 1.0)), torch.zeros_like(z))

    def transform(self, k):
        """integral of psi(x) e^{2 pi i x k} over the support, k in cycles per cell"""
        t, w = np.polynomial.legendre.leggauss(160)
        t, w = (torch.as_tensor(v, device="cuda") for v in (t, w))
        half = self.W / 2
        psi = torch.exp(self.BETA * (torch.sqrt(1.0 - t * t) - 1.0))
        flat = k.reshape(-1)
        out = torch.cat([torch.cos(2 * math.pi * half * torch.outer(c, t)) @ (w * psi) for c in flat.split(65536)])
        return (half * out).reshape(k.shape)


def _plane(r1, r2, vre, vim, N, cell):
    """sum_k v_k e^{2 pi i (r1 t1 + r2 t2)} on the N x N pixels (t1 along rows), by one 64-bit NUFFT."""
    ker = _Kernel()
    M = 2
    while M < ker.SIGMA * N:
        M *= 2
    grid = torch.zeros(2, M * M, device="cuda", dtype=torch.float64)
    steps = torch.arange(ker.W, device="cuda")
    for a in range(0, r1.numel(), 1 << 18):
        sl = slice(a, a + (1 << 18))
        idx, wgt = [], []
        for r in (r1[sl], r2[sl]):
            x = r * (cell * M)
            first = torch.ceil(x - ker.W / 2)
            cells = first.long()[:, None] + steps
            wgt.append(ker(cells - x[:, None]))
            idx.append(torch.remainder(cells, M))
        at = (idx[0][:, :, None] * M + idx[1][:, None, :]).reshape(-1)
        w = wgt[0][:, :, None] * wgt[1][:, None, :]
        grid[0].index_add_(0, at, (w * vre[sl, None, None]).reshape(-1))
        grid[1].index_add_(0, at, (w * vim[sl, None, None]).reshape(-1))
    full = torch.fft.ifft2(torch.complex(grid[0], grid[1]).reshape(M, M), norm="forward")
    off = torch.arange(N, device="cuda") - N // 2
    img = full[torch.remainder(off, M)][:, torch.remainder(off, M)]
    corr = ker.transform(off.double() / M)
    return img / (corr[:, None] * corr[None, :])


def _bessel(x, n_max):
    """J_0 .. J_n_max at x (tensor), Miller's downward recurrence."""
    ax = torch.clamp(x.abs(), min=1e-30)
    start = 2 * ((int(float(ax.max())) + n_max + 60) // 2)
    hi, lo = torch.zeros_like(ax), torch.full_like(ax, 1e-300)
    out, norm = [None] * (n_max + 1), torch.zeros_like(ax)
    for n in range(start, 0, -1):
        if n <= n_max:
            out[n] = lo
        if n % 2 == 0:
            norm = norm + 2 * lo
        hi, lo = lo, (2.0 * n / ax) * lo - hi
        big = torch.where(lo.abs() > 1e200, torch.full_like(lo, 1e-200), torch.ones_like(lo))
        if bool((big < 1).any()):
            hi, lo, norm = hi * big, lo * big, norm * big
            out = [None if o is None else o * big for o in out]
    out[0], norm = lo, norm + lo
    tiny = x.abs() < 1e-12  # J_0 = 1, J_1 = x / 2 and nothing else there
    out = [torch.where(tiny, float(n == 0) + (0.5 * ax if n == 1 else 0.0), o / norm) for n, o in enumerate(out)]
    return [o if n % 2 == 0 else torch.where(x < 0, -o, o) for n, o in enumerate(out)]


def _order(rule, alpha):
    """The Chebyshev order of the bucket and smallest-order rules: sampled truncation error <= 1e-2."""
    na, ns = (257, 1024) if rule == "bucket" else (513, 2048)
    a = alpha * torch.arange(na, device="cuda", dtype=torch.float64) / (na - 1)
    s = -1 + 2 * torch.arange(ns, device="cuda", dtype=torch.float64) / (ns - 1)
    exact = torch.exp(1j * torch.outer(a, s))
    j = _bessel(a, 31)
    tm, t, total, first = torch.ones_like(s), s, torch.zeros_like(exact), 32
    for n in range(32):
        term = torch.outer(j[n], tm) * (1 if n == 0 else 2) * (1j ** n)
        total = total + term
        K = n + 1
        if float((exact - total).abs().max()) <= 1e-2 and (rule == "min" or K in (8, 16, 24, 32)):
            first = K
            break
        tm, t = t, 2 * s * t - tm
    return first


def _image(case, coords, vre, vim, vin, N, cell):
    """The dirty image of samples at rotated coordinates `coords` (wavelengths) in 64 bits."""
    G = math.ceil(case["sigma"] * N - 1e-9)
    if case["sigma"] != 1.5:  # the grid is the next even size with no prime factor above 7
        G += G % 2
        while True:
            r = G
            for f in (2, 3, 5, 7):
                while r % f == 0:
                    r //= f
            if r == 1:
                break
            G += 2
    count = coords.shape[0]
    r3_lo, r3_hi = float(coords[:, 2].min()), float(coords[:, 2].max())
    half_w = case["support"] // 2
    keep = torch.ones(count, dtype=torch.bool, device="cuda")
    for k in (0, 1):
        p = coords[:, k] * (cell * G)
        lo, hi = torch.ceil(p - half_w), torch.floor(p + half_w)
        if case["edge"] == "strict":
            keep &= (lo >= -(G // 2)) & (hi <= (G - 1) // 2)
        else:
            keep &= (hi >= -(G // 2)) & (lo <= (G - 1) // 2)
    r, vre, vim = coords[keep], vre[keep], vim[keep]
    off = (torch.arange(N, device="cuda", dtype=torch.float64) - N // 2) * cell
    V = [[float(v) for v in row] for row in vin]
    ra = 1.0 - (off[:, None] + V[0][2]) ** 2 - (off[None, :] + V[1][2]) ** 2
    valid = ra >= 0
    t3 = -V[2][2] + (1.0 if V[2][2] >= 0 else -1.0) * torch.sqrt(torch.clamp(ra, min=0.0))
    t3_max = float(t3[valid].abs().max()) if bool(valid.any()) else 0.0
    half = max(0.5 * (r3_hi - r3_lo), 1e-6)
    alpha = 2 * math.pi * t3_max * half
    total = torch.zeros(N, N, device="cuda", dtype=torch.float64)
    if case["rule"] == "target" and alpha > 4.0:  # w planes: a third NUFFT axis
        ker = _Kernel()
        dw = 1.0 / (2 * ker.SIGMA * t3_max)  # plane spacing in wavelengths
        w = (r[:, 2] - r3_lo) / dw
        corr = ker.transform(t3 * dw)
        for p in range(-(ker.W // 2), int(math.ceil((r3_hi - r3_lo) / dw)) + ker.W // 2 + 1):
            on = (w - p).abs() < ker.W / 2
            if not bool(on.any()):
                continue
            z = ker(w[on] - p)
            plane = _plane(r[on, 0], r[on, 1], vre[on] * z, vim[on] * z, N, cell)
            total += (plane * torch.exp(2j * math.pi * (r3_lo + p * dw) * t3)).real
        total /= corr
    else:
        slabs = 1
        if case["rule"] == "bucket":
            slabs = max(1, math.ceil(alpha / 10.0))
        width = max(r3_hi - r3_lo, 2e-6) / slabs
        h, low = max(0.5 * width, 1e-6), r3_lo
        if case["rule"] == "min":
            h, low, width = half, 0.5 * (r3_lo + r3_hi) - half, 2 * half
        arg = 2 * math.pi * t3_max * h
        K = 40 if case["rule"] == "target" else _order(case["rule"], arg)
        if case["rule"] == "target":  # the whole series
            small = _bessel(torch.tensor([arg], device="cuda", dtype=torch.float64), 40)
            K = max(n for n in range(41) if n == 0 or abs(float(small[n])) > 1e-13) + 1
        j = _bessel(2 * math.pi * t3 * h, K)
        slab = torch.clamp(torch.floor((r[:, 2] - low) / width), 0, slabs - 1)
        for m in range(slabs):
            on = slab == m
            centre = low + (m + 0.5) * width
            s = torch.clamp((r[on, 2] - centre) / h, -1.0, 1.0)
            turn = torch.exp(2j * math.pi * centre * t3)
            tm, t = torch.ones_like(s), s
            for n in range(K):
                plane = _plane(r[on, 0], r[on, 1], vre[on] * tm, vim[on] * tm, N, cell)
                total += (plane * turn * (1j ** n) * ((1 if n == 0 else 2) * j[n])).real
                tm, t = t, 2 * s * t - tm
    det = abs(V[0][0] * V[1][1] - V[0][1] * V[1][0])
    return _reproject(case, total.abs() / det / count, valid, vin, N, cell)


def _reproject(case, value, valid, vin, N, cell):
    """SIN deprojection and bilinear splat of the rotated-frame image (the archive entry's
    trigonometric form for "min", else the main path's)."""
    V = np.asarray(vin, np.float64)
    half, r0, dc = N // 2, 180.0 / math.pi, cell / math.pi * 180.0
    shift = float(half) if case["rule"] == "min" else N * 0.5
    xi, eta = V[2, 0] / V[2, 2], V[2, 1] / V[2, 2]
    iy, ix = torch.meshgrid(*[torch.arange(N, device="cuda", dtype=torch.float64) - shift] * 2, indexing="ij")
    p1 = (-V[0, 0] * ix + V[1, 0] * iy) / abs(V[2, 2]) + shift
    p2 = (-V[0, 1] * ix + V[1, 1] * iy) / abs(V[2, 2]) + shift
    x, y = -dc * (p1 - (N / 2.0 + 1.0)), dc * (p2 - (N / 2.0 + 1.0))
    s = (x * x + y * y) / (r0 * r0)
    z = r0 * s / (1.0 + torch.sqrt(torch.clamp(1.0 - s, min=0.0)))  # r0 (1 - sqrt(1 - s))
    o1, o2 = -(x + xi * z) / dc + N / 2.0 + 1.0, (y + eta * z) / dc + N / 2.0 + 1.0
    inside = s <= 1.0
    if case["rule"] == "min":
        valid = valid & inside
    else:
        o1, o2 = torch.where(inside, o1, p1), torch.where(inside, o2, p2)
    L, M = o1 - half, o2 - half
    valid = valid & (L.abs() < half - 1) & (M.abs() < half - 1)
    L, M, value = L[valid], M[valid], value[valid]
    out = torch.zeros(N * N, device="cuda", dtype=torch.float64)
    lf, mf = torch.floor(L), torch.floor(M)
    for row, wr in ((mf, 1 - M + mf), (torch.ceil(M), M - mf)):
        for col, wc in ((lf, 1 - L + lf), (torch.ceil(L), L - lf)):
            out.index_add_(0, ((row + half) * N + col + half).long(), wr * wc * value)
    return out.reshape(N, N)


def exact(case, seed):
    samples = sum(s * (s - 1) // 2 * c for s, c, _ in _parts(case))
    if case["layout"] == "wide" and samples > 1_200_000:
        return None  # its w planes take minutes in 64 bits
    images = []
    for snap in _snapshots(case, seed):
        N = snap["image"]
        cell = float(np.float32(case["field"] / N))
        if case["kind"] == "fipipe":
            vre, vim, coords, vin = _quartet(case, snap)
            coords, vre, vim = coords.double(), vre.double(), vim.double()
        else:
            vre, vim = _collapse(snap, torch.float64)
            vin = _basis(snap)
            q = snap["uvw"].double() @ torch.as_tensor(vin, device="cuda").T
            s = snap["frequencies_hz"].double() / C_LIGHT
            coords = (s[:, None, None] * q[None]).reshape(-1, 3)
        images.append(_image(case, coords, vre, vim, vin, N, cell))
    if case["kind"] == "batch":
        return torch.stack(images)
    return images if case["kind"] == "server" else images[0]
