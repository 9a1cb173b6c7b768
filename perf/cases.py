"""Performance cases of the framework: what a user has it do, through its public entry points.

A case is a dict of plain values, one of four kinds:

* "dedisp": a `Dedisperser` (MS-OSM, or classical overlap-save with `osm`) takes
  `calls` blocks of `count` x M samples per pass.  With `fold` the pass ends with
  `get_profiles()`; without, it returns the dedispersed series (on the device, or
  with `host` through `get_output()` after host input).
* "twopol": the PSRDADA driver's loop: one dedisperser per polarisation, the
  summed intensity, `Fold_GPU`; `calls` reads per pass.
* "batch": several observations of uneven size in one `DedispBatch` call.
* "cnn": the DM-proposal network, a training gradient or a forward pass.

Bands, DM ranges, FFT sizes and periods are those of the benchmark's workloads
(16 MHz at 1250 MHz, 64 MHz and 32 MHz at 1400 MHz), of the reference's drivers
(calls of 32 blocks, FFT 2^21 for two polarisations, OSM at 2^18) and of the tests.
`exact` restates the path in 64 bits with torch.
"""
import math
import random

import numpy as np
import torch

KDM = np.float32(4.15 * 1e15)
F32 = np.float32


# ---------------------------------------------------------------------------
# the listed cases
# ---------------------------------------------------------------------------

def _dedisp(name, **kw):
    c = dict(name=name, kind="dedisp", bw=16e6, f0=1242e6, dm_lo=0.0, dm_hi=100.0, trials=1, fft=4096, count=32,
             calls=1, precision="fp32", osm=False, u16=False, host=False, fold=True, bins=1024, period=0.0031,
             detect="power")
    c.update(kw)
    return c


def listed():
    return [
        # the reference driver's own call: one DM, 32 blocks of uint16 samples from pinned host memory, the
        # series copied back; the smallest call, where launches and host work count
        _dedisp("single_dm_host_u16_32blocks", dm_lo=50.0, dm_hi=50.0, u16=True, host=True, fold=False),
        # a narrow band in short transforms, a few trials, the series left on the device; an odd trial and
        # block count (the tests' small sizes)
        _dedisp("series_fft512_7trials", bw=4e6, f0=1248e6, dm_lo=0.0, dm_hi=12.0, trials=7, fft=512, count=1023,
                fold=False),
        # a search in FP32: many trials folded from device memory
        _dedisp("fp32_fft4096_128trials", trials=128, count=2048),
        # the smallest valid transform of the 16 MHz band (FP32: no tensor path at 2048), uint16 input,
        # amplitude detection
        _dedisp("fp32_fft2048_48trials_u16", trials=48, fft=2048, count=2047, u16=True, detect="amplitude"),
        # FP32 at a long transform, 64 MHz
        _dedisp("fp32_fft16384_64trials", bw=64e6, f0=1368e6, dm_hi=200.0, trials=64, fft=16384, count=512),
        # the headline: 256 trials on the tensor cores
        _dedisp("f16_fft4096_256trials", trials=256, count=4096, precision="fp16"),
        # the precision sweep's band at 8192, two calls of an odd number of blocks per pass
        _dedisp("f16_fft8192_200trials", bw=64e6, f0=1368e6, dm_hi=200.0, trials=200, fft=8192, count=511, calls=2,
                precision="fp16"),
        # the same band at 16384, where more of the chirp is coherent; bf16 operands
        _dedisp("bf16_fft16384_96trials", bw=64e6, f0=1368e6, dm_hi=200.0, trials=96, fft=16384, count=512,
                precision="bf16"),
        # classical overlap-save of one DM at 2^18 points, folded
        _dedisp("osm_fft2p18_single_dm", dm_lo=50.0, dm_hi=50.0, fft=1 << 18, count=32, osm=True, u16=True),
        # the PSRDADA pipeline: two polarisations at 2^21 points, one block per read
        dict(name="twopol_fft2p21", kind="twopol", bw=16e6, f0=1242e6, dm=750.0, fft=1 << 21, count=1, calls=4,
             bins=1024, period=0.032768),
        # observations of uneven size in one launch
        dict(name="batch_6_observations", kind="batch", obs=6, mix=3, log2_lo=18, log2_hi=21),
        # one training step's gradient of the DM-proposal network at its defaults
        dict(name="cnn_gradient_batch256", kind="cnn", batch=256, inputs=64, length=256, channels=32, train=True),
    ]


def _nd(bw, dm, f0):
    kd = KDM * F32(dm)
    fhi = F32(f0) + F32(bw)
    v = math.floor(float(kd) * (1.0 / float(F32(f0)) ** 2 - 1.0 / float(fhi) ** 2) / float(F32(1) / F32(bw)))
    return max(v, 0)


def _min_order(nd, osm):
    if osm:
        return 2 * (1 << max(0, (nd - 1).bit_length()))
    return 0 if nd == 0 else 1 << math.ceil(math.log2(2 * math.sqrt(nd)))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _folds(bw, dm, f0, samples, period):
    """Whether the pass folds some whole periods after the discarded smear."""
    return 2 * _nd(bw, dm, f0) < samples and 8 * period * bw < samples


def _unnamed(**kw):
    c = _dedisp("", **kw)
    del c["name"]
    return c


def draw(rng):
    kind = rng.choice(["dedisp"] * 8 + ["twopol", "batch", "cnn", "cnn"])
    if kind == "cnn":
        return dict(kind="cnn", batch=_log(rng, 16, 256), inputs=rng.choice([16, 32, 64]),
                    length=rng.choice([96, 128, 192, 256]), channels=rng.choice([16, 24, 32]),
                    train=rng.random() < 0.7)
    if kind == "batch":
        return dict(kind="batch", obs=rng.randint(2, 7), mix=rng.randrange(1 << 20), log2_lo=17, log2_hi=20)
    if kind == "twopol":
        c = dict(kind="twopol", bw=16e6, f0=1242e6, dm=rng.uniform(50.0, 750.0), fft=1 << rng.randint(18, 21),
                 count=rng.randint(1, 2), calls=rng.randint(2, 4), bins=rng.choice([100, 256, 500, 1024]),
                 period=rng.uniform(0.001, 0.004))
        while not _folds(c["bw"], c["dm"], c["f0"], c["fft"] // 2 * c["count"] * c["calls"], c["period"]):
            c["dm"] *= 0.7
            c["period"] = max(0.8 * c["period"], 1100.0 / c["bw"])
        return c
    bw, fc = rng.choice([(4e6, 1250e6), (16e6, 1250e6), (32e6, 1400e6), (64e6, 1400e6)])
    f0 = fc - bw / 2
    if rng.random() < 0.15:  # one DM, classical overlap-save
        dm = rng.uniform(5.0, 60.0)
        m = _min_order(_nd(bw, dm, f0), True)
        fft = max(2 * m, 1 << rng.randint(15, 18))
        return _unnamed(dm_lo=dm, dm_hi=dm, bw=bw, f0=f0, fft=fft,
                        count=max(2, _log(rng, 1 << 19, 1 << 22) // (fft // 2)), osm=True, u16=rng.random() < 0.5,
                        fold=rng.random() < 0.6)
    precision = rng.choice(["fp32", "fp32", "fp16", "fp16", "bf16"])
    fft = rng.choice([4096, 8192, 16384]) if precision != "fp32" else 1 << rng.randint(8, 14)
    dm_hi = rng.uniform(20.0, 200.0)
    while 2 * _min_order(_nd(bw, dm_hi, f0), False) > fft:
        dm_hi *= 0.7
    series = rng.random() < 0.3
    small = rng.random() < 0.35
    samples = _log(rng, 1 << 16, 1 << 18) if small else _log(rng, 1 << 19, 1 << 22)
    trials = _log(rng, 1, 24) if series or small else _log(rng, 8, min(256, (1 << 29) // samples))
    count = max(3, samples // (fft // 2))
    period = rng.uniform(0.001, 0.004)
    while not series and not _folds(bw, dm_hi, f0, count * fft // 2, period):
        dm_hi *= 0.7
        period = max(0.7 * period, 1100.0 / bw)
    return _unnamed(bw=bw, f0=f0, dm_lo=rng.uniform(0.0, 0.3) * dm_hi, dm_hi=dm_hi, trials=trials, fft=fft, count=count,
                    precision=precision, u16=rng.random() < 0.4, host=series and small and rng.random() < 0.5,
                    fold=not series, bins=rng.choice([64, 256, 500, 1024]), period=period,
                    detect=rng.choice(["power", "power", "amplitude"]))


# ---------------------------------------------------------------------------
# inputs and handles
# ---------------------------------------------------------------------------

def _dms(c):
    return np.linspace(c["dm_lo"], c["dm_hi"], c["trials"]).astype(np.float32)


def _signal(n, u16, seed, device="cuda"):
    """Receiver noise with a pulsar's slow modulation: complex64, or offset-binary uint16 pairs as int32."""
    g = torch.Generator(device=device).manual_seed(seed)
    x = torch.randn(n, 2, generator=g, device=device)
    x *= 1.0 + 0.3 * torch.sin(torch.arange(n, device=device) * (2 * math.pi / 49600.0)).square().unsqueeze(1)
    if not u16:
        return torch.view_as_complex(x.mul_(0.7071067811865476))
    v = torch.clamp(torch.round(x * 700.0) + 32768.0, 1.0, 65535.0).to(torch.int32)
    return v[:, 0] | (v[:, 1] << 16)


class _Series:
    """A handle's series buffer as an array the tensor library can wrap; the wrapper keeps the handle alive."""

    def __init__(self, handle, trials, n):
        self.handle = handle
        self.__cuda_array_interface__ = {"data": (handle.output_device_ptr(), False), "shape": (trials, n),
                                         "typestr": "<c8", "version": 3}


def _m_of(c):
    m = max(_min_order(_nd(c["bw"], d, c["f0"]), c["osm"]) for d in _dms(c))
    return max(c["fft"] // 2, m)


def _observations(c):
    """The batch's observations: (bw, f0, trial DMs, fft, count, period)."""
    r = random.Random(c["mix"])
    out = []
    for _ in range(c["obs"]):
        bw = r.choice([4e6, 16e6, 32e6, 64e6])
        f0 = r.uniform(1100e6, 1500e6) - bw / 2
        samples = int(2 ** r.uniform(c["log2_lo"], c["log2_hi"]))
        trials = int(round(math.exp(r.uniform(math.log(16), math.log(128)))))
        dm_hi = r.uniform(20.0, 120.0)
        fft = r.choice([4096, 4096, 8192])
        count, period = max(2, samples // (fft // 2)), 2000.5 / bw * r.uniform(1.0, 6.0)
        while 2 * _min_order(_nd(bw, dm_hi, f0), False) > fft or not _folds(bw, dm_hi, f0, count * fft // 2, period):
            dm_hi *= 0.7
        out.append(dict(bw=bw, f0=f0, dm_lo=0.0, dm_hi=dm_hi, trials=trials, fft=fft, osm=False, count=count,
                        period=period))
    return out


def _cnn_params(c, seed):
    g = torch.Generator().manual_seed(seed + 77)
    parts, ci, K, C = [], c["inputs"], 7, c["channels"]
    for _ in range(4):
        parts += [torch.randn(C * ci * K, generator=g) * math.sqrt(2.0 / (ci * K)), torch.randn(C, generator=g) * 0.05]
        ci = C
    for _ in range(2):
        parts += [torch.randn(C, generator=g) / math.sqrt(C), torch.randn(1, generator=g) * 0.1]
    return torch.cat(parts).numpy()


def _cnn_inputs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(c["batch"], c["inputs"], c["length"], generator=g, device="cuda")
    label = (torch.rand(c["batch"], generator=g, device="cuda") < 0.5).float()
    target = (torch.rand(c["batch"], generator=g, device="cuda") * 6 - 3) * label
    return x, label, target


def prepare(case, seed):
    from msosm_gpu_b200 import dedisp, dm_proposal, fold

    c = case
    if c["kind"] == "cnn":
        net = dm_proposal.DMProposalNet(c["inputs"], c["length"], c["channels"], max_batch=c["batch"])
        net.set_params(_cnn_params(c, seed))
        return dict(c=c, net=net, inputs=_cnn_inputs(c, seed))
    if c["kind"] == "batch":
        members, xs = [], []
        for i, o in enumerate(_observations(c)):
            d = dedisp.Dedisperser(o["bw"], _dms(o), o["f0"], o["fft"], o["count"], series=False, precision="fp16")
            d.fold_init(o["period"], o["bw"], time_bin=256, discard_Nd=int(d.Nd.max()))
            members.append(d)
            xs.append(_signal(d.block_samples, False, seed * 64 + i))
        return dict(c=c, members=members, xs=xs, batch=dedisp.DedispBatch(members))
    if c["kind"] == "twopol":
        pols = [dedisp.Dedisperser(c["bw"], [c["dm"]], c["f0"], c["fft"], c["count"]) for _ in range(2)]
        n = pols[0].block_samples
        f = fold.Fold_GPU(c["period"], c["bw"], n, time_bin=c["bins"])
        f.discard_samples(int(pols[0].Nd[0]))
        xs = [_signal(n * c["calls"], True, seed * 2 + p) for p in range(2)]
        return dict(c=c, pols=pols, fold=f, xs=[[x[i * n:(i + 1) * n] for i in range(c["calls"])] for x in xs])
    d = dedisp.Dedisperser(c["bw"], _dms(c), c["f0"], c["fft"], c["count"], osm=c["osm"], series=not c["fold"],
                           precision=c["precision"])
    n = d.block_samples
    if c["fold"]:
        d.fold_init(c["period"], c["bw"], time_bin=c["bins"], discard_Nd=0 if c["osm"] else int(d.Nd.max()),
                    detect=c["detect"])
    x = _signal(n * c["calls"], c["u16"], seed)
    s = dict(c=c, d=d)
    if c["host"]:
        pinned = torch.empty_like(x, device="cpu", pin_memory=True)
        pinned.copy_(x)
        h = pinned.numpy()
        s["keep"] = pinned
        s["xs"] = [h[i * n:(i + 1) * n].view(np.uint32) if c["u16"] else h[i * n:(i + 1) * n] for i in range(c["calls"])]
    else:
        s["xs"] = [x[i * n:(i + 1) * n] for i in range(c["calls"])]
    if not c["fold"]:
        s["out"] = torch.as_tensor(_Series(d, c["trials"], n), device="cuda")
        s["out"].handle = d  # a caller that holds the series holds the handle
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    c = state["c"]
    if c["kind"] == "cnn":
        x, label, target = state["inputs"]
        net = state["net"]
        return net.gradient(x, label, target, want_grad=True) if c["train"] else net.forward(x)
    if c["kind"] == "batch":
        state["batch"].filter_block(state["xs"])
        return [d.get_profiles() for d in state["members"]]
    if c["kind"] == "twopol":
        a, b = state["pols"]
        f = state["fold"]
        for x, y in zip(*state["xs"]):
            a.filter_block(x)
            b.filter_block(y)
            f.calculate_intensity(a, b)
            f.fold_data()
        return f.fold_data_bins()
    d = state["d"]
    for x in state["xs"]:
        d.filter_block(x)
    if c["fold"]:
        return d.get_profiles()
    return d.get_output() if c["host"] else state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _dedisp_work(c, m, fold):
    n = m * c["count"] * c.get("calls", 1)
    per_fft = 10.0 * math.log2(2 * m)  # flop per kept sample of a transform of 2 m points (5 N log2 N / m)
    last = m * c["count"]
    return dict(bytes=n * (4.0 if c.get("u16") else 8.0) + c["trials"] * (c["bins"] * 4.0 if fold else last * 8.0),
                flops=n * (per_fft + c["trials"] * (per_fft + 12.0 + (4.0 if fold else 0.0))))


def work(case):
    c = case
    if c["kind"] == "cnn":
        K, C, B, L = 7, c["channels"], c["batch"], c["length"]
        first, rest = 2.0 * B * L * C * c["inputs"] * K, 3 * 2.0 * B * L * C * C * K
        params = _cnn_params(c, 0).size
        return dict(bytes=4.0 * (B * c["inputs"] * L + (2 * params if c["train"] else 0.5 * params + 2 * B)),
                    flops=(2 * first + 3 * rest) if c["train"] else first + rest)
    if c["kind"] == "batch":
        ws = [_dedisp_work(dict(o, bins=256), _m_of(o), True) for o in _observations(c)]
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    if c["kind"] == "twopol":
        w = _dedisp_work(dict(c, trials=1, u16=True), max(c["fft"] // 2, _min_order(_nd(c["bw"], c["dm"], c["f0"]), False)), True)
        return dict(bytes=2 * w["bytes"], flops=2 * w["flops"])
    return _dedisp_work(c, _m_of(c), c["fold"])


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _filter(bw, dm, f0, m):
    """H of one trial: the chirp sampled with the float roundings that define it, M-point inverse transform
    (unnormalised), zero pad, 2M-point transform; and x 1/N^2."""
    fs, w0 = float(F32(bw)), F32(2 * math.pi * float(F32(f0)))
    step = F32(2 * math.pi * fs / m)
    j = torch.arange(m, device="cuda", dtype=torch.int64)
    i = (j + m // 2) & (m - 1)
    si = torch.tensor(step, device="cuda") * i.to(torch.float32)
    w = (-math.pi * fs + si.double()).float()
    w = (w.double() + math.pi * fs).float()
    den = (w + torch.tensor(w0, device="cuda")).double()
    ph = 4 * math.pi * math.pi * float(KDM) * float(F32(dm)) * w.double() * w.double() / den / float(w0) / float(w0)
    h = torch.polar(torch.ones_like(ph), -ph)
    p = torch.zeros(2 * m, dtype=torch.complex128, device="cuda")
    p[:m] = torch.fft.ifft(h, norm="forward")
    return torch.fft.fft(p) / float(4 * m * m)


def _delays(bw, dm, f0, m):
    """Per-bin block delay of one trial (the reference's float arithmetic)."""
    n = 2 * m
    d = np.zeros(n, np.int64)
    dc = math.ceil(float(F32(_nd(bw, dm, f0)) / F32(m)))
    if dc <= 0:
        return d
    fs, w0 = F32(bw), F32(2 * math.pi * float(F32(f0)))
    edge = [F32(-1)] + [F32(0)] * (dc - 1) + [F32(1)]
    first = 1
    c = 4 * math.pi * math.pi * float(KDM) * float(F32(dm))
    for j in range(1, dc):
        jm = F32(j * m) / fs
        s = math.sqrt(1.0 / (1.0 / float(w0) ** 2 - float(jm) / c))
        edge[j] = F32((s - float(w0) - math.pi * float(fs)) / math.pi / float(fs))
        if edge[j] < 0:
            first = j + 1
    for j in range(first):
        lo = math.floor((edge[j] + F32(2)) * F32(m))
        hi = math.floor((edge[j + 1] + F32(2)) * F32(m)) if j + 1 < first else n
        d[lo:min(hi, n)] = j
    lo = 0
    for j in range(dc - first + 1):
        hi = math.floor(edge[j + first] * F32(m))
        d[lo:min(hi, n)] = first - 1 + j
        lo = max(lo, hi)
    return d


def _decode(x, u16):
    if not u16:
        return x.to(torch.complex128)
    re, im = (x & 0xFFFF).double(), ((x >> 16) & 0xFFFF).double()
    return torch.complex(torch.where(re > 0, re - 32768.0, re), torch.where(im > 0, im - 32768.0, im))


def _spectra(x, m):
    """Spectra of the overlapping windows of a stream that begins with x."""
    p = torch.cat([torch.zeros(m, dtype=x.dtype, device=x.device), x])
    return torch.fft.fft(p.unfold(0, 2 * m, m), dim=1)


def _trial(X, bw, dm, f0, m, osm):
    """The dedispersed series of one trial from the spectra X [blocks][2m]."""
    H = _filter(bw, dm, f0, m)
    Z = X
    if not osm:
        d = _delays(bw, dm, f0, m)
        Z = torch.zeros_like(X)
        for v in np.unique(d):
            b = torch.from_numpy(np.nonzero(d == v)[0]).cuda()
            if v < X.shape[0]:
                Z[v:, b] = X[:X.shape[0] - v, b]
    return torch.fft.ifft(Z * H, dim=1, norm="forward")[:, m:].reshape(-1)


class _Fold:
    """Which samples fold into which bins, chunk by chunk (the reference's float bookkeeping)."""

    def __init__(self, period, fs, discard):
        self.psf = F32(period) * F32(fs)
        self.ps = int(self.psf)
        self.diff = F32(self.psf - F32(self.ps))
        self.discard = math.ceil(float(F32(discard) / self.psf))
        self.ready, self.seen, self.cur, self.idx, self.open = self.discard == 0, 0, F32(0), 0, False
        self.base, self.pending, self.starts = 0, None, []  # stream starts of the folded whole periods

    def _count(self):
        if not self.ready:
            self.seen += 1
            self.ready = self.seen == self.discard

    def _drift(self):
        self.cur = F32(self.cur + self.diff)

    def chunk(self, size):
        ci, cs = 0, size
        try:
            if self.cur > 1:
                self.cur = F32(self.cur - F32(1))
                ci, cs = ci + 1, cs - 1
                if cs == 0:
                    return
            if self.idx:
                n = self.ps - self.idx
                if cs < n:
                    self.pending.append((self.base + ci, cs))
                    self.idx += cs
                    return
                if self.open:
                    self.starts.append(self.pending + [(self.base + ci, n)])
                ci, cs, self.idx = ci + n, cs - n, 0
                self._drift()
                if self.cur > 1:
                    if cs == 0:
                        return
                    self.cur = F32(self.cur - F32(1))
                    ci, cs = ci + 1, cs - 1
                self._count()
            while cs >= self.ps:
                if self.ready:
                    self.starts.append([(self.base + ci, self.ps)])
                ci, cs = ci + self.ps, cs - self.ps
                self._drift()
                skip = self.cur > 1
                if skip and cs:
                    self.cur = F32(self.cur - F32(1))
                    ci, cs = ci + 1, cs - 1
                self._count()
                if skip and self.base + ci == self.base + size and cs == 0:
                    return
            if cs > 0:
                self.open, self.pending, self.idx = self.ready, [(self.base + ci, cs)], cs
        finally:
            self.base += size

    def profile(self, I, bins):
        acc = torch.zeros(self.ps, dtype=torch.float64, device="cuda")
        whole = [p[0][0] for p in self.starts if len(p) == 1]
        for s in range(0, len(whole), 256):
            at = torch.tensor(whole[s:s + 256], device="cuda")
            acc += I[at.unsqueeze(1) + torch.arange(self.ps, device="cuda")].sum(0)
        for p in self.starts:
            if len(p) > 1:
                acc += torch.cat([I[a:a + n] for a, n in p])
        if bins == self.ps:
            return acc
        per = self.ps // bins
        return acc[:per * bins].view(bins, per).sum(1) / per


def _profiles(x, o, m, bins, calls, detect, discard, osm):
    f = _Fold(o["period"], o["bw"], discard)
    for _ in range(calls):
        f.chunk(m * o["count"])
    X = _spectra(x, m)
    out = []
    for dm in _dms(o):
        y = _trial(X, o["bw"], dm, o["f0"], m, osm)
        p = y.real.square() + y.imag.square()
        out.append(f.profile(p if detect == "power" else p.sqrt(), bins))
    return torch.stack(out)


def _cnn_exact(c, seed):
    K, C, B, L = 7, c["channels"], c["batch"], c["length"]
    x, label, target = (t.double() for t in _cnn_inputs(c, seed))
    p32 = torch.from_numpy(_cnn_params(c, seed)).cuda()
    rounded, at, ci, shapes = p32.double(), 0, c["inputs"], []
    for _ in range(4):
        shapes += [("w", (C, ci, K)), ("b", (C,))]
        ci = C
    shapes += [("w", (C,)), ("b", (1,)), ("w", (C,)), ("b", (1,))]
    parts = []
    for kind, shape in shapes:
        n = math.prod(shape)
        v = p32[at:at + n]
        parts.append((v.bfloat16() if kind == "w" else v).double().view(shape).requires_grad_(True))
        at += n
    a = x
    for l in range(4):
        a = torch.cat([a[:, :, -(K // 2):], a, a[:, :, :K // 2]], 2)
        w = parts[2 * l].reshape(C, -1)
        a = torch.einsum("oc,bcl->bol", w, a.unfold(2, L, 1).reshape(B, -1, L)) + parts[2 * l + 1].view(1, -1, 1)
        a = torch.relu(a)
    h = a.mean(2)
    logit, off = h @ parts[8] + parts[9], h @ parts[10] + parts[11]
    if not c["train"]:
        return logit.detach(), off.detach()
    pos = label > 0.5
    loss = torch.nn.functional.binary_cross_entropy_with_logits(logit, label)
    loss = loss + 0.25 * ((off - target).square() * pos).sum() / pos.sum().clamp(min=1)
    loss.backward()
    return float(loss), torch.cat([q.grad.reshape(-1) for q in parts])


def exact(case, seed):
    c = case
    if c["kind"] == "cnn":
        return _cnn_exact(c, seed)
    if c["kind"] == "batch":
        out = []
        for i, o in enumerate(_observations(c)):
            m = _m_of(o)
            x = _signal(m * o["count"], False, seed * 64 + i).to(torch.complex128)
            out.append(_profiles(x, o, m, 256, 1, "power", max(_nd(o["bw"], d, o["f0"]) for d in _dms(o)), False))
        return out
    if c["kind"] == "twopol":
        nd = _nd(c["bw"], c["dm"], c["f0"])
        m = max(c["fft"] // 2, _min_order(nd, False))
        f, p = _Fold(c["period"], c["bw"], nd), 0.0
        for _ in range(c["calls"]):
            f.chunk(m * c["count"])
        for pol in range(2):
            x = _decode(_signal(m * c["count"] * c["calls"], True, seed * 2 + pol), True)
            y = _trial(_spectra(x, m), c["bw"], c["dm"], c["f0"], m, False)
            p = p + y.real.square() + y.imag.square()
        return f.profile(p.sqrt(), c["bins"])
    m = _m_of(c)
    x = _decode(_signal(m * c["count"] * c["calls"], c["u16"], seed), c["u16"])
    if c["fold"]:
        discard = 0 if c["osm"] else max(_nd(c["bw"], d, c["f0"]) for d in _dms(c))
        return _profiles(x, c, m, c["bins"], c["calls"], c["detect"], discard, c["osm"])
    X = _spectra(x, m)
    y = torch.stack([_trial(X, c["bw"], d, c["f0"], m, c["osm"])[-m * c["count"]:] for d in _dms(c)])
    return y.cpu().numpy() if c["host"] else y
