"""The work a user of this framework has it do, through the package's public
entry points: whole frames (single, from host memory, in batches, with the
learned warm start) and the stages that are called by themselves, with the
sizes of the project's own configurations (256 x 4096 plain, 1024 x 8192
five-stage, 64 uneven frames, 1024 IFDS pulses of 5000 samples) and generic
ones in between, down to the smallest frame that isar_create accepts.

Inputs are seeded echoes of point scatterers (dechirped LFM, int16 counts as a
receiver delivers them), made on the GPU with torch.  exact() restates the
chain in 64 bits with torch and numpy.
"""
import functools
import math
import random

import numpy as np
import torch

import isar_imaging_cuda_gb300 as g

CUT = 512
FC, BW, FS, PRF, LIGHT = 10.0e9, 1.0e9, 100.0e6, 1000.0, 3.0e8
HPC, MTRC, HRRP, IQ16 = g.FLAG_HPC, g.FLAG_MTRC, g.FLAG_HRRP, g.FLAG_IQ16


def listed():
    return [
        # the smallest frame a context takes: latency of the whole chain
        dict(name="frame_128x512", kind="frame", M=128, N=512, flags=0, ifds=False, full=False),
        # the plain single-frame configuration
        dict(name="frame_256x4096", kind="frame", M=256, N=4096, flags=0, ifds=False, full=False),
        # IFDS data (pre-step on the echoes, its own MTRC orientation), int16 samples
        dict(name="frame_512x4096_ifds", kind="frame", M=512, N=4096, flags=MTRC | IQ16, ifds=True, full=False),
        # the five-stage single-frame configuration
        dict(name="frame_1024x8192_full", kind="frame", M=1024, N=8192, flags=HPC | MTRC, ifds=False, full=True),
        # isarMainSingle's path: echoes and image in (pageable) host memory
        dict(name="host_512x2048", kind="host", M=512, N=2048, flags=HPC | MTRC | HRRP, ifds=False, full=True),
        # 64 uneven frames in one graph launch
        dict(name="batch_uneven64", kind="batch", frames=64, lanes=16, shapes=5, flags=0, full=False),
        # large five-stage frames from sensor samples, judged learned warm start
        dict(name="learned_32x1024x8192", kind="learned", frames=32, M=1024, N=8192, flags=HPC | MTRC | IQ16,
             cluster=4, tol=1e-5),
        # IFDS ingest: one window's new pulses
        dict(name="pulses_1024x5000", kind="pulses", pulses=1024, iq_len=5000),
        # the range profiles that if_hrrp asks for
        dict(name="hrrp_1024x8192", kind="hrrp", M=1024, N=8192, ifds=False),
        # centring and cut of given profiles
        dict(name="cut_512x4096", kind="cut", M=512, N=4096),
        # autofocus of a given cut at a non-default iteration count
        dict(name="entropy_512_60", kind="entropy", M=512, iters=60),
        # one gradient step of the warm-start network, a training batch of 256-pulse frames
        dict(name="wsnet_step_64x256", kind="wsnet", frames=64, M=256),
    ]


def _log2_pick(rng, lo, hi):
    return 1 << rng.randint(int(math.log2(lo)), int(math.log2(hi)))


def _log_pick(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "host", "batch", "batch", "learned", "pulses", "hrrp", "cut",
                       "entropy", "wsnet"])
    M = _log2_pick(rng, 128, 1024)
    N = _log2_pick(rng, max(512, M), 8192)
    full = rng.random() < 0.5
    if kind in ("frame", "host"):
        ifds = rng.random() < 0.25
        flags = rng.choice([0, MTRC, HRRP, MTRC | HRRP]) | (HPC if full and not ifds else 0)
        if kind == "frame" and rng.random() < 0.3:
            flags |= IQ16
        if kind == "host":
            N = min(N, 4096)
        return dict(kind=kind, M=M, N=N, flags=flags, ifds=ifds, full=full and not ifds)
    if kind == "batch":
        return dict(kind=kind, frames=_log_pick(rng, 2, 64), lanes=rng.choice([0, 4, 16]), shapes=rng.randint(0, 999),
                    flags=rng.choice([0, HPC | MTRC]), full=full)
    if kind == "learned":
        return dict(kind=kind, frames=_log_pick(rng, 2, 24), M=M, N=N, flags=HPC | MTRC | rng.choice([0, IQ16]),
                    cluster=4, tol=1e-5)
    if kind == "pulses":
        return dict(kind=kind, pulses=_log_pick(rng, 1, 1024), iq_len=_log_pick(rng, 2048, 12000))
    if kind == "hrrp":
        return dict(kind=kind, M=M, N=N, ifds=rng.random() < 0.5)
    if kind == "cut":
        return dict(kind=kind, M=M, N=N)
    if kind == "entropy":
        return dict(kind=kind, M=M, iters=rng.randint(1, 120))
    M = _log2_pick(rng, 128, 1024)
    return dict(kind=kind, frames=_log_pick(rng, 1, 16384 // M), M=M)


# ---- inputs -----------------------------------------------------------------

def _radar(M, N, ifds=False):
    return g.radar(M, N, B=BW, fc=FC, Fs=FS, data_type=g.IFDS if ifds else g.STRETCH)


@functools.lru_cache(maxsize=2)
def _noise_free_basis(N):
    i = torch.arange(N // 64, device="cuda", dtype=torch.float64) * 64.0
    j = torch.arange(64, device="cuda", dtype=torch.float64)
    return i, j


def _echo(M, N, seed, full, drift=True):
    """int16 counts [M, N, 2] and float64 velocities [M] on the GPU: scatterers
    in a 20 m (40 m) patch, range drift, phase errors, noise at 10 dB (5 dB)."""
    gen = torch.Generator(device="cuda").manual_seed(1_000_003 * (seed % 1_000_000_007) + M + 7 * N)

    def uni(*s):
        return torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)

    def nor(*s):
        return torch.randn(*s, generator=gen, device="cuda", dtype=torch.float64)

    K, patch = (200, 40.0) if full else (50, 20.0)
    cell = LIGHT / (2.0 * BW)
    sx, sy = (uni(K) - 0.5) * patch, (uni(K) - 0.5) * min(patch, 0.5 * N * cell)
    amp, ph0 = torch.sqrt(-2.0 * torch.log(1.0 - uni(K))), 2.0 * math.pi * uni(K)
    m = torch.arange(M, device="cuda", dtype=torch.float64)
    u = (m - M / 2) / (M / 2)
    walk = torch.cumsum((0.5 if full else 0.3) * nor(M), 0) if drift else torch.zeros_like(m)
    perr = (6.0 * u * u + 0.5 * (2.0 * uni(M) - 1.0)) if full else math.pi * (2.0 * uni(M) - 1.0)
    vel = torch.round((3000.0 + 50.0 * m / PRF) * 10.0) * 0.1 if full else torch.zeros_like(m)
    th = (math.radians(4.0) / (M / PRF) if full else 0.02) * (m - M / 2) / PRF
    R = (20.0 + walk)[:, None] * cell + torch.cos(th)[:, None] * sy + torch.sin(th)[:, None] * sx
    # phase -(4 pi / c) (fc + Kr t) R: per scatterer a constant and a rate per sample
    a0 = torch.remainder(-2.0 * FC / LIGHT * R + (perr[:, None] + ph0) / (2.0 * math.pi), 1.0)
    rate = -2.0 * (BW / N) / LIGHT * R
    i, j = _noise_free_basis(N)

    def cis(cycles):
        t = 2.0 * math.pi * torch.remainder(cycles, 1.0)
        return torch.complex(torch.cos(t).float(), torch.sin(t).float())

    P = cis(a0[:, None, :] + rate[:, None, :] * i[None, :, None]) * amp.float()
    Q = cis(rate[:, None, :] * j[None, :, None])
    x = torch.matmul(P, Q.transpose(1, 2)).reshape(M, N)
    if full:
        n = torch.arange(N, device="cuda", dtype=torch.float64)
        x = x * cis(2.0 / LIGHT * (BW / N * FS) * (n / FS) ** 2 * vel[:, None])
    power = float((amp * amp).sum())
    sig = math.sqrt(power / 10.0 ** ((5.0 if full else 10.0) / 10.0) / 2.0)
    y = torch.view_as_real(x)
    y = y + sig * torch.randn(M, N, 2, generator=gen, device="cuda")
    y = torch.round(y * (1000.0 / math.sqrt(power))).clamp_(-32768, 32767)
    return y.to(torch.int16), vel


def _profiles(M, N, seed):
    """Aligned complex range profiles [M, N], as range alignment leaves them."""
    iq, _ = _echo(M, N, seed, False, drift=False)
    x = torch.view_as_complex(iq.float())
    n = torch.arange(N, device="cuda")
    return torch.fft.ifft(x * (1.0 - 2.0 * (n % 2)), dim=1).contiguous()


def _cut_of(M, seed):
    """A 512-cell cut [M, 512] of such profiles."""
    y = _profiles(M, 1024, seed)
    k = int((y[0].real.abs() + y[0].imag.abs()).argmax())
    k = min(max(k - CUT // 2, 0), 1024 - CUT)
    return y[:, k:k + CUT].contiguous()


def _chirp_pulses(pulses, iq_len, seed):
    """int16 pulses [P, 2 iq_len]: echoes of a few scatterers of the transmitted chirp, and noise."""
    gen = torch.Generator(device="cuda").manual_seed(77_003 * (seed % 1_000_000_007) + pulses + 3 * iq_len)
    S = _chirp_len(iq_len)
    n = torch.arange(iq_len, device="cuda", dtype=torch.float64)
    acc = torch.zeros(pulses, iq_len, dtype=torch.complex64, device="cuda")
    for _ in range(4):
        d = torch.rand(pulses, 1, generator=gen, device="cuda", dtype=torch.float64) * (iq_len - S) * 0.9
        a = torch.rand(pulses, 1, generator=gen, device="cuda") + 0.2
        t = (n - d) / S - 0.5
        ph = math.pi * (BW / 20.0) * (S / FS) * t * t
        on = ((t >= -0.5) & (t < 0.5)).float() * a
        acc += torch.complex(torch.cos(ph).float() * on, torch.sin(ph).float() * on)
    y = torch.view_as_real(acc) * 800.0 + 100.0 * torch.randn(pulses, iq_len, 2, generator=gen, device="cuda")
    vel = 300.0 + 10.0 * torch.rand(pulses, generator=gen, device="cuda", dtype=torch.float64)
    return torch.round(y).clamp_(-32768, 32767).to(torch.int16).reshape(pulses, 2 * iq_len), vel


def _chirp_len(iq_len):
    return int(0.8 * iq_len)


def _pulse_radar(iq_len):
    return g.radar(128, 512, B=BW / 20.0, fc=FC, Fs=FS, Tp=(_chirp_len(iq_len) + 0.5) / FS, data_type=g.IFDS)


def _net_params(seed):
    rng = np.random.default_rng(seed % (1 << 31))
    parts = []
    for r, c in [(64, 320)] * 6 + [(64, 64)]:
        parts += [(rng.standard_normal((r, c)) * math.sqrt(2.0 / c)).ravel(), np.zeros(r)]
    parts += [(rng.standard_normal((2, 64)) * 0.3).ravel(), np.array([1.0, 0.0])]
    return np.concatenate(parts).astype(np.float32)


def _net_batch(frames, M, seed):
    gen = torch.Generator(device="cuda").manual_seed(9_007 * (seed % 1_000_000_007) + frames + 5 * M)
    x0 = (0.7 * torch.randn(frames, M, 64, generator=gen, device="cuda")).to(torch.bfloat16)
    # the residual to predict follows a feature (as the Doppler increment among them does), plus noise
    t = x0[..., 0].float() + 0.3 * torch.randn(frames, M, generator=gen, device="cuda")
    return x0, t


def _batch_shapes(case):
    """Pulses uniform over 128..1024 and range cells over 2048..8192, powers of two."""
    r = random.Random(case["shapes"])
    return [(r.choice([128, 256, 512, 1024]), r.choice([2048, 4096, 8192])) for _ in range(case["frames"])]


# ---- what a program keeps: contexts, batches, the trained network ------------

@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


@functools.lru_cache(maxsize=2)
def _context(M, N, ifds):
    return g.Context(_radar(M, N, ifds), stream=_stream().cuda_stream)


@functools.lru_cache(maxsize=1)
def _batch(lanes, shapes_id):
    return g.Batch(stream=_stream().cuda_stream, lanes=lanes)


@functools.lru_cache(maxsize=1)
def _learned_batch(M, N, frames, cluster, tol):
    net = g.WSNet(M)
    net.load_params(g.WARMSTART_WEIGHTS)
    b = g.Batch(stream=_stream().cuda_stream, lanes=frames)
    b.set_tuning(_radar(M, N), g.Tuning(ra_pair_min=128, ra_rows_per_cta=4, ra_rows_final=4, af_cluster=cluster,
                                        af_tol=tol, af_iters=120, ra_rows_each_level=0))
    b.set_warmstart(net)
    return b, net


# ---- the passes ----------------------------------------------------------------

def _frame_inputs(M, N, seed, flags, full):
    iq, vel = _echo(M, N, seed, full)
    return (iq if flags & IQ16 else iq.float()), (vel if flags & HPC else None)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("frame", "host"):
        M, N = case["M"], case["N"]
        s["ctx"] = _context(M, N, case["ifds"])
        s["x"], s["v"] = _frame_inputs(M, N, seed, case["flags"], case["full"])
        if kind == "host":
            s["x"] = torch.view_as_complex(s["x"]).cpu().numpy()
            s["v"] = None if s["v"] is None else s["v"].cpu().numpy()
        else:
            s["img"] = torch.empty(M, CUT, device="cuda")
    elif kind in ("batch", "learned"):
        if kind == "batch":
            shapes = _batch_shapes(case)
            s["b"] = _batch(case["lanes"], (case["shapes"], case["frames"]))
        else:
            shapes = [(case["M"], case["N"])] * case["frames"]
            s["b"], s["net"] = _learned_batch(case["M"], case["N"], case["frames"], case["cluster"], case["tol"])
        full = case.get("full", True)
        s["in"] = [_frame_inputs(M, N, seed * 131 + k, case["flags"] & (IQ16 | (HPC if full else 0)), full)
                   for k, (M, N) in enumerate(shapes)]
        s["img"] = [torch.empty(M, CUT, device="cuda") for M, _ in shapes]
        flags = case["flags"] if full else case["flags"] & ~HPC
        s["frames"] = g.Batch.frames((_radar(M, N), x, v, flags, i)
                                     for (M, N), (x, v), i in zip(shapes, s["in"], s["img"]))
    elif kind == "pulses":
        P = case["pulses"]
        s["ctx"] = g.Context(_pulse_radar(case["iq_len"]), stream=_stream().cuda_stream)
        s["ad"], s["v"] = _chirp_pulses(P, case["iq_len"], seed)
        s["out"] = torch.empty(P, 4096, 2, device="cuda")
        s["off"] = torch.empty(P, dtype=torch.int32, device="cuda")
    elif kind == "hrrp":
        s["ctx"] = _context(case["M"], case["N"], case["ifds"])
        s["x"] = _echo(case["M"], case["N"], seed, False)[0].float()
        s["out"] = torch.empty_like(s["x"])
    elif kind == "cut":
        s["ctx"] = _context(case["M"], case["N"], False)
        s["y"] = torch.view_as_real(_profiles(case["M"], case["N"], seed))
        s["out"] = torch.empty(case["M"], CUT, 2, device="cuda")
    elif kind == "entropy":
        s["ctx"] = _context(case["M"], 1024, False)
        s["cut"] = torch.view_as_real(_cut_of(case["M"], seed))
        s["out"] = torch.empty_like(s["cut"])
    else:
        s["net"] = g.WSNet(-(-case["frames"] * case["M"] // 8) * 8, training=True, stream=_stream().cuda_stream)
        s["net"].set_params(_net_params(seed))
        s["x0"], s["t"] = _net_batch(case["frames"], case["M"], seed)
        s["out"] = torch.empty(case["frames"] * case["M"], 2, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["ctx"].image_device(s["x"], s["v"], s["img"], s["flags"])
        return s["img"]
    if kind == "host":
        return s["ctx"].image_host(s["x"], s["v"], s["flags"])
    if kind in ("batch", "learned"):
        s["b"].run(s["frames"])
        return s["img"]
    if kind == "pulses":
        s["ctx"].pulse_compress(s["ad"], s["iq_len"], s["v"], s["out"], s["off"])
        return {"out": s["out"], "offsets": s["off"]}
    if kind == "hrrp":
        s["ctx"].stage_hrrp(s["x"], s["out"])
        return s["out"]
    if kind == "cut":
        s["ctx"].stage_center_cut(s["y"], s["out"])
        return s["out"]
    if kind == "entropy":
        with torch.cuda.stream(_stream()):   # the stage works in place: on a copy
            s["out"].copy_(s["cut"])
        s["ctx"].stage_fast_entropy(s["out"], s["iters"])
        return s["out"]
    s["net"].forward(s["x0"], s["frames"], s["M"], s["out"])
    loss = s["net"].backward(s["t"], s["frames"], s["M"])
    return {"out": s["out"], "loss": loss, "grads": s["net"].grads()}


# ---- what a pass cannot do without ----------------------------------------------

def _fft_flops(n, count):
    return 5.0 * n * math.log2(n) * count


def _frame_work(M, N, flags, iters=120, bins=64):
    b = M * N * (4 if flags & IQ16 else 8) + (8 * M if flags & HPC else 0) + 4 * M * CUT
    # two transforms per row and half-cell pair, one per merge, one per row at the end
    f = _fft_flops(N, 4 * M + 3 * (M // 2 - 1) + M) + _fft_flops(M, CUT + 2 * iters * bins)
    if flags & MTRC:
        f += _fft_flops(CUT, 2 * M) + _fft_flops(2 * M, 2 * CUT)
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("frame", "host"):
        b, f = _frame_work(case["M"], case["N"], case["flags"])
    elif kind == "batch":
        b, f = map(sum, zip(*(_frame_work(M, N, case["flags"]) for M, N in _batch_shapes(case))))
    elif kind == "learned":
        b, f = _frame_work(case["M"], case["N"], case["flags"])
        b, f = b * case["frames"], f * case["frames"]
    elif kind == "pulses":
        nfft = 1 << case["iq_len"].bit_length()
        b = case["pulses"] * (4 * case["iq_len"] + 8 + 4 + 8 * 4096)
        f = _fft_flops(nfft, 3 * case["pulses"])
    elif kind == "hrrp":
        b, f = 16 * case["M"] * case["N"], _fft_flops(case["N"], case["M"])
    elif kind == "cut":
        b = 8 * min(case["M"], 256) * case["N"] + 16 * case["M"] * CUT
        f = 4.0 * case["M"] * case["N"]
    elif kind == "entropy":
        b, f = 32 * case["M"] * CUT, _fft_flops(case["M"], CUT + 2 * case["iters"] * 64)
    else:
        rows, macs = case["frames"] * case["M"], 6 * 64 * 320 + 64 * 64 + 2 * 64
        b, f = rows * (64 * 2 + 4 + 8) + 8 * (macs + 6 * 64 + 66), 6.0 * rows * macs
    return {"bytes": float(b), "flops": float(f)}


# ---- the same in 64 bits ---------------------------------------------------------
# Tables and decisions that the chain defines in 32-bit floats (windows, the
# parabolic shift, the CZT's w and a, the pulse-compression reference) are
# rounded where it rounds them; all signal arithmetic is in 64 bits.

PI32 = np.float32(3.14159265358979)


def _hamming(n):
    i = np.arange(n, dtype=np.float32)
    arg = (np.float32(2) * PI32 * i) / np.float32(n - 1)
    return np.float32(0.54) - np.float32(0.46) * np.cos(arg.astype(np.float64)).astype(np.float32)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _ramp(shift, N):
    n = torch.arange(N, device="cuda", dtype=torch.float64)
    ph = -2.0 * math.pi * torch.remainder(shift.double()[:, None] / N * n, 1.0)
    return torch.complex(torch.cos(ph), torch.sin(ph))


def _half_swap(x, dim):
    return torch.roll(x, x.shape[dim] // 2, dim)


def _exact_align(x):
    M, N = x.shape
    ham = _hamming(N)
    win = ham * np.cos((PI32 * np.arange(N, dtype=np.float32)).astype(np.float64)).astype(np.float32)
    x = x * _dev(win.astype(np.float64))
    step = 1
    while step < M:
        p = torch.fft.ifft(x, dim=1)
        env = (p.real.square() + p.imag.square()).reshape(M // step, step, N).sum(1).sqrt()
        F = torch.fft.fft(env.to(torch.complex128), dim=1)
        corr = torch.fft.ifft(F[0::2] * F[1::2].conj(), dim=1).real * N
        pos = _half_swap(corr, 1).abs().argmax(dim=1)
        at = pos + N // 2
        f1, f2, f3 = (corr.gather(1, ((at + k) % N)[:, None])[:, 0].float() for k in (-1, 0, 1))
        fa, fb = (f1 + f3 - 2.0 * f2) / 2.0, (f3 - f1) / 2.0
        shift = pos.float() + (-fb / (2.0 * fa)) - N / 2
        x = x.reshape(M // (2 * step), 2, step, N)
        x = torch.cat([x[:, :1], x[:, 1:] * _ramp(shift, N)[:, None, None, :]], 1).reshape(M, N)
        step *= 2
    return torch.fft.ifft(x, dim=1)


def _exact_center_cut(y):
    M, N = y.shape
    a = y.abs()
    arp = (a[:min(M, 256)] / a.max()).sum(0) / M
    arp = arp.cpu().numpy()
    srt = np.sort(arp)
    d = np.abs(srt[30:] - srt[:-30] - 30.0 * srt[-1] / N)
    thr = srt[int(np.argmin(d)) + 15]
    kept = []
    for i in np.nonzero(arp > thr)[0]:
        lo, hi = i - 4, i + 4
        if lo >= 0 and hi <= N - 1:
            mean = arp[lo:hi + 1].sum() / 9.0
        elif lo < 0:
            mean = arp[:hi + 1].sum() / (4.0 + i + 1)
        else:
            mean = arp[lo:].sum() / (N - i - 4.0 - 1) if N - i - 5 else math.inf
        if not mean < thr:
            kept.append(int(i))
    if kept:
        y = torch.roll(y, N // 2 - sum(kept) // len(kept), 1)
    k = int((y[0].real.abs() + y[0].imag.abs()).argmax())
    k = min(max(k - CUT // 2, 0), N - CUT)
    return y[:, k:k + CUT].clone()


def _exact_doppler(x):
    ang = torch.angle((x[:-1].conj() * x[1:]).sum(1)).cumsum(0)
    return torch.cat([torch.zeros(1, dtype=x.dtype, device=x.device), torch.exp(-1j * ang)])


def _exact_entropy(cut, iters):
    M = cut.shape[0]
    cmax = cut[:min(M, 256)].abs().amax(0)
    thr = np.float32(1.48) * (np.float32(int(cmax.to(torch.int64).sum())) / np.float32(CUT))
    tgt = int((cmax > float(thr)).sum())
    U = 1 << (tgt // 2).bit_length() if tgt // 2 else 2
    spec = torch.fft.fft(_exact_doppler(cut)[:, None] * cut, dim=0)
    q = spec.real.square() + spec.imag.square()
    energy = q.sum(0)
    q = q / energy
    ent = -(q * torch.log(q)).sum(0)
    energy, ent = energy.cpu().numpy(), ent.cpu().numpy()
    top = np.argsort(-energy, kind="stable")[:tgt]
    low = top[np.argsort(ent[top], kind="stable")][:U]
    bins = np.sort(np.concatenate([low, np.zeros(U - len(low), np.int64)])).astype(np.int64)
    x = cut[:, torch.from_numpy(bins).cuda()]
    ph = _exact_doppler(x)
    for _ in range(iters):
        t = torch.fft.fft(ph[:, None] * x, dim=0)
        s = (x.conj() * torch.fft.ifft(t * t.abs(), dim=0)).sum(1)
        ph = s / s.abs()
    return cut * ph[:, None]


def _exact_image(cut, flags, ifds):
    M = cut.shape[0]
    if flags & MTRC:
        st = _half_swap(cut, 1)
        st = torch.fft.fft(st, dim=1) if ifds else torch.fft.ifft(st, dim=1)
        rate, tp = np.float32(BW) / np.float32(_tp), np.float32(_tp)
        posa = rate * tp / (np.float32(FC) * (np.float32(CUT) - np.float32(1)))
        con = rate * tp / np.float32(2 * FC)
        base = (posa.astype(np.float64) * np.arange(CUT) + np.float64(np.float32(1) - con)).astype(np.float32)
        tw, ta = np.float32(-2) * PI32 * base / np.float32(M), np.float32(-1) * PI32 * base

        def log_of(t):   # log of the float-rounded point on the circle
            re, im = (f(t.astype(np.float64)).astype(np.float32).astype(np.float64) for f in (np.cos, np.sin))
            return 0.5 * np.log1p((re - 1.0) * (re + 1.0) + im * im) + 1j * np.arctan2(im, re)

        lw, la = _dev(log_of(tw)), _dev(log_of(ta))
        k = torch.arange(M, device="cuda", dtype=torch.float64)
        mk, out = k[:, None] * k, torch.empty_like(st)
        for c in range(0, CUT, 16):
            E = torch.exp(lw[c:c + 16, None, None] * mk - la[c:c + 16, None, None] * k)   # [c, k, m]
            out[:, c:c + 16] = torch.matmul(E, st[:, c:c + 16].T[:, :, None])[:, :, 0].T
        z = _half_swap(torch.fft.ifft(_half_swap(out, 0), dim=0), 0)
        z = _half_swap(_half_swap(torch.fft.fft(z, dim=1), 1), 0)
        cut = torch.flip(z, (1,)) if ifds else z
    cut = cut.clone()
    # the window reaches the first 512 elements only, element i by hamming[i / M]
    cut[0] *= _dev(_hamming(M)[np.arange(CUT) // M].astype(np.float64))
    img = _half_swap(torch.fft.fft(cut, dim=0), 0)
    return (torch.flip(img, (0,)) if ifds else img).abs()


_tp = 1.0


def _exact_frame(iq, vel, flags, ifds):
    global _tp
    M, N = iq.shape[:2]
    _tp = N / FS
    x = torch.view_as_complex(iq.double().contiguous())
    if ifds:
        x = _half_swap(torch.fft.ifft(_half_swap(x, 1), dim=1), 1)
    else:
        n = torch.arange(N, device="cuda", dtype=torch.float64)
        if flags & HPC:
            cyc = (-4.0 * 3.14159265358979 * (BW / _tp) / LIGHT) * ((n / FS) ** 2) * vel[:, None]
            x = x * torch.complex(torch.cos(cyc), torch.sin(cyc))
        if flags & HRRP:
            x = x * _dev(_hamming(N).astype(np.float64))
    return _exact_image(_exact_entropy(_exact_center_cut(_exact_align(x)), 120), flags, ifds)


def _exact_pulses(case, seed):
    L, S = case["iq_len"], _chirp_len(case["iq_len"])
    nfft = 1 << L.bit_length()
    ad, vel = _chirp_pulses(case["pulses"], L, seed)
    x = torch.view_as_complex(ad.reshape(-1, L, 2).double())
    f = np.float32
    tp = (S + 0.5) / FS
    v2 = f(2) * vel.cpu().numpy().astype(f)[:, None] / f(LIGHT)
    v2c = f(1) - v2
    c1 = f(-2) * PI32 * f(FC) * v2 / v2c
    c2 = f(np.float64(PI32 * f(BW / 20.0)) / tp)
    tk = v2c * (f(tp) / f(-2) + np.arange(S, dtype=f) * f(tp) / (f(S) - f(1)))
    ph = ((c1 + c2 * tk) * tk).astype(np.float64)
    ham = _hamming(S)
    ref = _dev((ham * np.cos(ph).astype(f)) + 1j * (ham * np.sin(ph).astype(f)).astype(np.float64))
    y = torch.fft.ifft(torch.fft.fft(ref, n=nfft, dim=1).conj() * torch.fft.fft(x, n=nfft, dim=1), dim=1)
    off = ((y.real.abs() + y.imag.abs()).argmax(1) - 2048).clamp(0, nfft - 4096)
    out = y.gather(1, off[:, None] + torch.arange(4096, device="cuda"))
    return {"out": torch.view_as_real(out), "offsets": off.to(torch.int32)}


def _exact_net(case, seed):
    x0, t = _net_batch(case["frames"], case["M"], seed)
    F, M = case["frames"], case["M"]
    p = torch.from_numpy(_net_params(seed)).double().cuda().requires_grad_()
    o, a = 0, x0.double()
    for li, (r, c) in enumerate([(64, 320)] * 6 + [(64, 64), (2, 64)]):
        W, b = p[o:o + r * c].reshape(r, c), p[o + r * c:o + r * c + r]
        o += r * c + r
        if c == 320:   # five taps of 64 channels, zero padding
            pad = torch.nn.functional.pad(a, (0, 0, 2, 2))
            a = torch.cat([pad[:, k:k + M] for k in range(5)], 2)
        a = a @ W.T + b
        if li < 7:
            a = torch.relu(a)
    d = torch.atan2(a[..., 1], a[..., 0]) - t.double()
    z = torch.exp(1j * d[:, :M - 1]).mean(1)
    loss = (1.0 - z.abs()).mean()
    loss.backward()
    return {"out": a.detach().reshape(F * M, 2), "loss": float(loss.detach()), "grads": p.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame", "host"):
        iq, vel = _echo(case["M"], case["N"], seed, case["full"])
        return _exact_frame(iq, vel, case["flags"], case["ifds"])
    if kind == "batch":
        flags = case["flags"] if case["full"] else case["flags"] & ~HPC
        out = []
        for k, (M, N) in enumerate(_batch_shapes(case)):
            iq, vel = _echo(M, N, seed * 131 + k, case["full"])
            out.append(_exact_frame(iq, vel, flags, False))
        return out
    if kind == "learned":
        return None   # a bf16 network proposes the start and entropies of both results decide which is kept
    if kind == "pulses":
        return _exact_pulses(case, seed)
    if kind == "hrrp":
        x = torch.view_as_complex(_echo(case["M"], case["N"], seed, False)[0].double())
        x = _half_swap(x, 1) if case["ifds"] else x * _dev(_hamming(case["N"]).astype(np.float64))
        return torch.view_as_real(_half_swap(torch.fft.fft(x, dim=1), 1))
    if kind == "cut":
        return torch.view_as_real(_exact_center_cut(_profiles(case["M"], case["N"], seed).to(torch.complex128)))
    if kind == "entropy":
        return torch.view_as_real(_exact_entropy(_cut_of(case["M"], seed).to(torch.complex128), case["iters"]))
    return _exact_net(case, seed)
