"""The transforms a user of this library runs, as cases that can be timed.

Families (a case's "family"):

- host:  one transform at a time from host arrays through the drop-in classes
         CFFT / RFFT, forward then backward: the reference's own call pattern.
- c2c:   batched complex transforms on device buffers (Plan.exec_device),
         forward then backward of the spectrum.
- r2c:   batched real transforms on device buffers; "ops" names the
         operations of one pass (forward bins, squared magnitudes, backward).
- mixed: a batch of transforms of many orders and kinds, replayed from one
         CUDA graph (MixedBatch, SCHED_GRAPH).
- stft:  framing, window and forward transform of a long signal (Plan.stft).
- istft: spectral filter, backward transform, window and overlap-add
         (Plan.istft).

"mode" is the plan's computation form: "plain" (the default; the reference's
arithmetic) or "fast" (fast-twiddle, the form the autotuner chooses for the
large orders). "pad" elements follow every transform in its buffers.
"""
import math

import numpy as np
import torch

import zldsp_fft_b200 as Z

MODES = {"plain": Z.MODE_PLAIN, "fast": Z.MODE_FAST}
LAYOUTS = {"aos": Z.AOS, "soa": Z.SOA}
# forms of the real transform's outputs: (operation, output layout)
R2C_OPS = {"fwd": (Z.FORWARD, Z.AOS), "fwd_soa": (Z.FORWARD, Z.SOA), "sqr": (Z.FORWARD_SQR_MAG, Z.AOS),
           "bwd": (Z.BACKWARD, Z.AOS), "bwd_soa": (Z.BACKWARD, Z.AOS)}


def listed():
    return [
        # one 1024-point transform from host memory and back, as a program
        # written for the reference calls it: latency only
        dict(name="host_cfft_o10", family="host", kind="c2c", order=10, dtype="f32"),
        # the same transform with its data already on the device: two launches
        dict(name="cfft_o10_single", family="c2c", order=10, batch=1, dtype="f32", mode="plain", layout="aos", pad=0),
        # many short blocks in split re/im arrays with padded rows (channel
        # banks, short-block spectra); an odd number of them
        dict(name="cfft_o8_soa_padded", family="c2c", order=8, batch=100003, dtype="f32", mode="plain", layout="soa",
             pad=8),
        # analysis of windowed audio frames, the usual frame length: bins, and
        # the power spectrum a display wants
        dict(name="rfft_o12_fwd", family="r2c", order=12, batch=8192, dtype="f32", mode="plain", ops="fwd,sqr", pad=0),
        # synthesis of such frames from edited bins; an odd number of frames
        dict(name="rfft_o12_bwd", family="r2c", order=12, batch=8191, dtype="f32", mode="plain", ops="bwd", pad=0),
        # long complex transforms that pass over memory twice, default form
        dict(name="cfft_o16_plain", family="c2c", order=16, batch=4096, dtype="f32", mode="plain", layout="aos", pad=0),
        # the longest of the usual sizes, 2 GiB of them, in the tuned form
        dict(name="cfft_o20_fast", family="c2c", order=20, batch=256, dtype="f32", mode="fast", layout="aos", pad=0),
        # long real signals, analysis and synthesis (convolution reverbs,
        # whole-file spectra)
        dict(name="rfft_o18", family="r2c", order=18, batch=1024, dtype="f32", mode="plain", ops="fwd,bwd", pad=0),
        # double precision, tuned form
        dict(name="cfft64_o16", family="c2c", order=16, batch=512, dtype="f64", mode="fast", layout="aos", pad=0),
        # 20,000 transforms of orders 6..16, half complex and half real
        dict(name="mixed_o6_16", family="mixed", count=20000, lo=6, hi=16, orders=1004, dtype="f32"),
        # spectrogram of a long signal, three quarters overlap
        dict(name="stft_o12", family="stft", order=12, hop=1024, frames=131069, dtype="f32", op="sqr"),
        # filtered resynthesis of the same signal
        dict(name="istft_o12", family="istft", order=12, hop=1024, frames=131069, dtype="f32"),
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["host", "c2c", "c2c", "c2c", "r2c", "r2c", "r2c", "mixed", "stft", "istft"])
    dtype = rng.choice(["f32", "f32", "f32", "f64"])
    size = 4 if dtype == "f32" else 8
    if family == "host":
        return dict(family=family, kind=rng.choice(["c2c", "r2c"]), order=rng.randint(6, 16), dtype=dtype)
    if family == "mixed":
        lo = rng.randint(4, 10)
        return dict(family=family, count=_loguni(rng, 50, 8000), lo=lo, hi=rng.randint(lo + 2, 16), orders=rng.randint(1, 9999),
                    dtype="f32")
    if family in ("stft", "istft"):
        order = rng.randint(10, 14 if family == "istft" or dtype == "f64" else 15)
        n = 1 << order
        if family == "istft" and dtype == "f64":
            order, n = min(order, 13), min(n, 1 << 13)
        total = _loguni(rng, 1 << 20, 1 << (26 if dtype == "f32" else 25))
        if family == "stft":
            hop = 2 * rng.randint(n // 16, n // 2)  # even, any; an eighth of the frame to all of it
            return dict(family=family, order=order, hop=hop, frames=max(1, total // hop), dtype=dtype,
                        op=rng.choice(["fwd", "sqr"]))
        hop = n >> rng.randint(1, 3)
        return dict(family=family, order=order, hop=hop, frames=max(1, total // hop), dtype=dtype)
    order = rng.randint(4, 22)
    per = (2 if family == "c2c" else 1) * size << order
    cap = 1 << 30
    batch = max(1, min(_loguni(rng, 1, max(1, cap // per)), cap // (2 * per) or 1))
    mode = rng.choice(["plain", "plain", "fast"])
    if family == "c2c":
        return dict(family=family, order=order, batch=batch, dtype=dtype, mode=mode, layout=rng.choice(["aos", "soa"]),
                    pad=rng.choice([0, 0, 4, 6]))
    return dict(family=family, order=order, batch=batch, dtype=dtype, mode=mode,
                ops=rng.choice(["fwd", "fwd_soa", "sqr", "bwd", "bwd_soa", "fwd,bwd"]), pad=rng.choice([0, 0, 2, 6]))


# ------------------------------------------------------------------ inputs
def _types(case):
    return (torch.float32, torch.complex64, np.float32) if case["dtype"] == "f32" else (
        torch.float64, torch.complex128, np.float64)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(shape, dtype, g):
    return torch.rand(shape, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _hann(n, dtype):
    t = torch.arange(n, dtype=torch.float64, device="cuda")
    return (0.5 - 0.5 * torch.cos(2 * math.pi * t / n)).to(dtype)


def _frames(batch, n, dtype, g):
    """Three sinusoids and noise under a Hann window, per frame."""
    t = torch.arange(n, dtype=dtype, device="cuda")
    x = torch.randn((batch, n), generator=g, device="cuda", dtype=dtype).mul_(0.1)
    for _ in range(3):
        f = torch.rand((batch, 1), generator=g, device="cuda", dtype=dtype) * 0.5
        a = torch.rand((batch, 1), generator=g, device="cuda", dtype=dtype) * 0.9 + 0.1
        ph = torch.rand((batch, 1), generator=g, device="cuda", dtype=dtype) * (2 * math.pi)
        x.addcmul_(a.expand_as(x), torch.sin(2 * math.pi * (f * t % 1.0) + ph))
    return x.mul_(_hann(n, dtype))


def _bins(batch, nb, dtype, g):
    x = _uniform((batch, nb, 2), dtype, g)
    x[:, 0, 1] = 0
    x[:, -1, 1] = 0
    return x


def _inputs(case, seed):
    """The input tensors of a device case, reals (complex values as pairs), on the GPU."""
    dtype = _types(case)[0]
    family, g = case["family"], _gen(seed)
    if family == "c2c":
        n, b = 1 << case["order"], case["batch"]
        if case["layout"] == "soa":
            return dict(re=_uniform((b, n + case["pad"]), dtype, g), im=_uniform((b, n + case["pad"]), dtype, g))
        return dict(x=_uniform((b, n + case["pad"], 2), dtype, g))
    if family == "r2c":
        n, b = 1 << case["order"], case["batch"]
        if case["ops"].startswith("bwd"):
            x = _bins(b, n // 2 + 1 + case["pad"], dtype, g)
            x[:, n // 2, 1] = 0
            if case["ops"] == "bwd":
                return dict(x=x)
            return dict(re=x[..., 0].contiguous(), im=x[..., 1].contiguous())
        if case["pad"]:
            x = torch.zeros((b, n + case["pad"]), dtype=dtype, device="cuda")
            x[:, :n] = _frames(b, n, dtype, g)
            return dict(x=x)
        return dict(x=_frames(b, n, dtype, g))
    if family == "stft":
        n = 1 << case["order"]
        return dict(x=_uniform(((case["frames"] - 1) * case["hop"] + n,), dtype, g), win=_hann(n, dtype))
    n = 1 << case["order"]
    nb = n // 2 + 1
    k = torch.arange(nb, dtype=torch.float64, device="cuda")
    mag, ph = 1.0 / (1.0 + (k / 256.0) ** 2), -2.0 * math.pi * 64.0 * k / n  # a low-pass with a short delay
    filt = torch.stack([mag * torch.cos(ph), mag * torch.sin(ph)], -1).to(dtype).contiguous()
    return dict(x=_bins(case["frames"], nb, dtype, g), win=_hann(n, dtype), filt=filt)


def _mixed_layout(case):
    """[(kind, order, input offset, output offset)] in reals, and the two totals
    (kinds and orders belong to the case, the data to the seed)."""
    rng = np.random.default_rng(case["orders"])
    orders = rng.integers(case["lo"], case["hi"] + 1, case["count"])
    kinds = rng.integers(0, 2, case["count"])
    items, i_off, o_off = [], 0, 0
    for kind, order in zip(kinds.tolist(), orders.tolist()):
        n = 1 << order
        items.append((kind, order, i_off, o_off))
        i_off += 2 * n if kind == 0 else n
        o_off += (2 * n if kind == 0 else n + 2) + 31 & ~31
        i_off = i_off + 31 & ~31
    return items, i_off, o_off


def _host_input(case, seed):
    rng = np.random.default_rng(seed)
    n, real = 1 << case["order"], _types(case)[2]
    if case["kind"] == "c2c":
        z = rng.uniform(-1, 1, (n, 2)).astype(real)
        return z.view(np.complex64 if real is np.float32 else np.complex128).reshape(n)
    return rng.uniform(-1, 1, n).astype(real)


def prepare(case, seed):
    family = case["family"]
    if family == "host":
        n, real = 1 << case["order"], _types(case)[2]
        cplx = np.complex64 if real is np.float32 else np.complex128
        x = _host_input(case, seed)
        if case["kind"] == "c2c":
            return dict(family=family, fft=Z.CFFT(case["order"], real), x=x, y=np.zeros(n, cplx), z=np.zeros(n, cplx))
        return dict(family=family, fft=Z.RFFT(case["order"], real), x=x, y=np.zeros(n // 2 + 1, cplx),
                    z=np.zeros(n, real))
    if family == "mixed":
        items, ni, no = _mixed_layout(case)
        x = _uniform((ni,), torch.float32, _gen(seed))
        y = torch.zeros(no, dtype=torch.float32, device="cuda")
        xp, yp = x.data_ptr(), y.data_ptr()
        descs = [(Z.C2C if kind == 0 else Z.R2C, order, Z.FORWARD, xp + 4 * i, yp + 4 * o) for kind, order, i, o in items]
        return dict(family=family, batch=Z.MixedBatch(descs, np.float32), x=x, y=y)

    s = dict(family=family, case=case, **_inputs(case, seed))
    dtype, _, real = _types(case)
    order, n = case["order"], 1 << case["order"]
    nb = n // 2 + 1

    def zeros(*shape):
        return torch.zeros(shape, dtype=dtype, device="cuda")

    if family == "c2c":
        s["plan"] = Z.Plan(Z.C2C, order, real, MODES[case["mode"]])
        b, row = case["batch"], n + case["pad"]
        if case["layout"] == "soa":
            s |= dict(yr=zeros(b, row), yi=zeros(b, row), zr=zeros(b, row), zi=zeros(b, row))
        else:
            s |= dict(y=zeros(b, row, 2), z=zeros(b, row, 2))
    elif family == "r2c":
        s["plan"] = Z.Plan(Z.R2C, order, real, MODES[case["mode"]])
        b, out = case["batch"], {}
        for op in case["ops"].split(","):
            if op.startswith("bwd"):
                out[op] = (zeros(b, n + case["pad"]),)
            elif op == "fwd":
                out[op] = (zeros(b, nb + case["pad"], 2),)
            elif op == "fwd_soa":
                out[op] = (zeros(b, nb + case["pad"]), zeros(b, nb + case["pad"]))
            else:
                out[op] = (zeros(b, nb + case["pad"]),)
        s["out"] = out
    elif family == "stft":
        s["plan"] = Z.Plan(Z.R2C, order, real)
        s["y"] = zeros(case["frames"], nb, 2) if case["op"] == "fwd" else zeros(case["frames"], nb)
    else:
        s["plan"] = Z.Plan(Z.R2C, order, real)
        s["y"] = zeros((case["frames"] - 1) * case["hop"] + n)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    family = s["family"]
    if family == "host":
        s["fft"].forward(s["x"], s["y"])
        s["fft"].backward(s["y"], s["z"])
        return dict(spectrum=s["y"], signal=s["z"])
    st = torch.cuda.current_stream().cuda_stream
    if family == "mixed":
        s["batch"].run(Z.SCHED_GRAPH, st)
        return s["y"]
    case, plan = s["case"], s["plan"]
    n = 1 << case["order"]
    if family == "c2c":
        b, row = case["batch"], n + case["pad"]
        if case["layout"] == "soa":
            plan.exec_device(Z.FORWARD, Z.SOA, Z.SOA, s["re"].data_ptr(), s["im"].data_ptr(), s["yr"].data_ptr(),
                             s["yi"].data_ptr(), b, row, row, st)
            plan.exec_device(Z.BACKWARD, Z.SOA, Z.SOA, s["yr"].data_ptr(), s["yi"].data_ptr(), s["zr"].data_ptr(),
                             s["zi"].data_ptr(), b, row, row, st)
            return dict(spectrum=(s["yr"], s["yi"]), signal=(s["zr"], s["zi"]))
        plan.exec_device(Z.FORWARD, Z.AOS, Z.AOS, s["x"].data_ptr(), None, s["y"].data_ptr(), None, b, row, row, st)
        plan.exec_device(Z.BACKWARD, Z.AOS, Z.AOS, s["y"].data_ptr(), None, s["z"].data_ptr(), None, b, row, row, st)
        return dict(spectrum=s["y"], signal=s["z"])
    if family == "r2c":
        b, pad = case["batch"], case["pad"]
        real_row, bin_row = n + pad, n // 2 + 1 + pad
        for op, out in s["out"].items():
            code, layout = R2C_OPS[op]
            o0, o1 = out[0].data_ptr(), (out[1].data_ptr() if len(out) > 1 else None)
            if code != Z.BACKWARD:
                plan.exec_device(code, Z.AOS, layout, s["x"].data_ptr(), None, o0, o1, b, real_row, bin_row, st)
            elif op == "bwd_soa":
                plan.exec_device(code, Z.SOA, Z.AOS, s["re"].data_ptr(), s["im"].data_ptr(), o0, None, b, bin_row,
                                 real_row, st)
            else:
                src = s["out"]["fwd"][0] if "fwd" in s["out"] else s["x"]
                plan.exec_device(code, Z.AOS, Z.AOS, src.data_ptr(), None, o0, None, b, bin_row, real_row, st)
        return s["out"]
    if family == "stft":
        op = Z.FORWARD if case["op"] == "fwd" else Z.FORWARD_SQR_MAG
        plan.stft(op, Z.AOS, s["x"].data_ptr(), case["hop"], s["win"].data_ptr(), s["y"].data_ptr(), None,
                  case["frames"], 0, st)
        return s["y"]
    plan.istft(Z.AOS, s["x"].data_ptr(), None, case["hop"], case["frames"], s["y"].data_ptr(),
               filter=s["filt"].data_ptr(), window=s["win"].data_ptr(), stream=st)
    return s["y"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    family = case["family"]
    if family == "mixed":
        items = _mixed_layout(case)[0]
        nbytes = sum(4 * (4 << o if kind == 0 else (2 << o) + 2) for kind, o, _, _ in items)
        flops = sum((5 if kind == 0 else 2.5) * o * (1 << o) for kind, o, _, _ in items)
        return dict(bytes=nbytes, flops=int(flops))
    size = 4 if case["dtype"] == "f32" else 8
    order, n = case["order"], 1 << case["order"]
    nb = n // 2 + 1
    if family == "host":
        both = 4 * n if case["kind"] == "c2c" else n + 2 * nb
        return dict(bytes=2 * size * both, flops=2 * int((5 if case["kind"] == "c2c" else 2.5) * n * order))
    if family == "c2c":
        return dict(bytes=2 * case["batch"] * 4 * n * size, flops=2 * case["batch"] * 5 * n * order)
    if family == "r2c":
        ops = case["ops"].split(",")
        reals = sum(n + (nb if op == "sqr" else 2 * nb) for op in ops)
        return dict(bytes=case["batch"] * reals * size, flops=int(len(ops) * case["batch"] * 2.5 * n * order))
    frames, signal = case["frames"], (case["frames"] - 1) * case["hop"] + n
    per = nb if family == "stft" and case["op"] == "sqr" else 2 * nb
    small = n if family == "stft" else n + 2 * nb  # window; filter
    return dict(bytes=size * (signal + frames * per + small), flops=int(frames * 2.5 * n * order))


# ------------------------------------------------------------------ the same in 64 bits
def _pairs(z):
    return torch.view_as_real(z)


def _padded(like, values, n):
    """64-bit tensor of like's shape, zero outside the first n entries of each row."""
    out = torch.zeros(like, dtype=torch.float64, device="cuda")
    out[:, :n] = values
    return out


def _overlap_add(frames, hop):
    """Sum of frames[f] at f * hop (hop divides the frame length)."""
    count, n = frames.shape
    k = n // hop
    out = torch.zeros((count + k - 1, hop), dtype=frames.dtype, device=frames.device)
    for j in range(k):
        out[j:j + count] += frames[:, j * hop:(j + 1) * hop]
    return out.reshape(-1)


def exact(case, seed):
    family = case["family"]
    if family == "host":
        x, n = _host_input(case, seed), 1 << case["order"]
        if case["kind"] == "c2c":
            x = x.astype(np.complex128)
            return dict(spectrum=np.fft.fft(x), signal=n * x)
        x = x.astype(np.float64)
        return dict(spectrum=np.fft.rfft(x), signal=(n // 2) * x)
    if family == "mixed":
        items, ni, no = _mixed_layout(case)
        x = _uniform((ni,), torch.float32, _gen(seed))
        y = torch.zeros(no, dtype=torch.float64, device="cuda")
        groups = {}
        for kind, order, i, o in items:
            groups.setdefault((kind, order), []).append((i, o))
        for (kind, order), places in groups.items():
            n = 1 << order
            rows = torch.stack([x[i:i + (2 * n if kind == 0 else n)] for i, _ in places]).double()
            if kind == 0:
                rows = _pairs(torch.fft.fft(torch.view_as_complex(rows.reshape(-1, n, 2)))).reshape(len(places), -1)
            else:
                rows = _pairs(torch.fft.rfft(rows)).reshape(len(places), -1)
            for row, (_, o) in zip(rows, places):
                y[o:o + row.numel()] = row
        return y
    s = _inputs(case, seed)
    n = 1 << case["order"]
    nb = n // 2 + 1
    if family == "c2c":
        b, row = case["batch"], n + case["pad"]
        if case["layout"] == "soa":
            z = torch.complex(s["re"][:, :n].double(), s["im"][:, :n].double())
            y = torch.fft.fft(z)
            return dict(spectrum=(_padded((b, row), y.real, n), _padded((b, row), y.imag, n)),
                        signal=(_padded((b, row), n * z.real, n), _padded((b, row), n * z.imag, n)))
        x = s["x"][:, :n].double()
        y = _pairs(torch.fft.fft(torch.view_as_complex(x.contiguous())))
        return dict(spectrum=_padded((b, row, 2), y, n), signal=_padded((b, row, 2), n * x, n))
    if family == "r2c":
        b, pad, out = case["batch"], case["pad"], {}
        ops = case["ops"].split(",")
        if ops[0].startswith("bwd"):
            z = s["x"] if ops[0] == "bwd" else torch.stack([s["re"], s["im"]], -1)
            z = torch.view_as_complex(z[:, :nb].double().contiguous())
            return {ops[0]: (_padded((b, n + pad), torch.fft.irfft(z, n=n) * (n // 2), n),)}
        x = s["x"][:, :n].double()
        y = torch.fft.rfft(x)
        for op in ops:
            if op == "fwd":
                out[op] = (_padded((b, nb + pad, 2), _pairs(y), nb),)
            elif op == "fwd_soa":
                out[op] = (_padded((b, nb + pad), y.real, nb), _padded((b, nb + pad), y.imag, nb))
            elif op == "sqr":
                out[op] = (_padded((b, nb + pad), y.real.square() + y.imag.square(), nb),)
            else:
                out[op] = (_padded((b, n + pad), x * (n // 2), n),)
        return out
    if family == "stft":
        frames = s["x"].unfold(0, n, case["hop"])
        y = torch.empty((case["frames"], nb) + ((2,) if case["op"] == "fwd" else ()), dtype=torch.float64, device="cuda")
        win = s["win"].double()
        step = max(1, (1 << 27) // n)
        for f in range(0, case["frames"], step):
            z = torch.fft.rfft(frames[f:f + step].double() * win)
            y[f:f + step] = _pairs(z) if case["op"] == "fwd" else z.real.square() + z.imag.square()
        return y
    filt, win = torch.view_as_complex(s["filt"].double()), s["win"].double()
    frames = torch.empty((case["frames"], n), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // n)
    for f in range(0, case["frames"], step):
        z = torch.view_as_complex(s["x"][f:f + step].double()) * filt
        frames[f:f + step] = torch.fft.irfft(z, n=n) * (n // 2) * win
    return _overlap_add(frames, case["hop"])
