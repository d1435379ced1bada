"""The workloads whose speed is watched: the resampling stage and the entry
points around it, as a user's program calls them.

A case is a dict with a "kind":

* ``process``: one ``Resampler.process`` pass over ``frames`` B-frames of one
  packet stream.  ``thresholds``: "start" (the stream starts with this call:
  the first batch sets them), "kept" (a running stream: set by an earlier
  call, leftover snapshots carried from call to call).  ``host``: pinned host
  buffers, the copies inside the pass.  ``framed``: 8224-B VDIF frames.
* ``multi``: one ``process_multi`` pass over ``streams`` packet streams of
  ``frames_min`` to ``frames_max`` B-frames; ``window``: windowed thresholds
  on a stream with dropped and displaced packets.
* ``ingest``: one ``Resampler.ingest`` batch of ``frames`` B-frames of 8pac
  units, which completes and ships at least one 143-frame group; the
  timestamps move on from pass to pass, as received batches do.
* ``stages``: the stage's functions called one at a time on both phased sums
  of ``batches`` 143-snapshot batches, as a program does that replaces the
  reference's functions one by one.
* ``pfb``: the inverse polyphase filter bank on ``blocks`` spectra.

``precision`` is the handle's: "fp32", "tc16" or "tc16_fast".
"""
import ctypes as C
import math

import torch

from sdbe_gb300 import Resampler, _native as N, pfb
from sdbe_gb300.resampler import process_multi

PRECISIONS = {"fp32": N.PRECISION_FP32, "tc16": N.PRECISION_TC16, "tc16_fast": N.PRECISION_TC16_FAST}
GROUP = N.FRAMES_PER_GROUP
SWARM_CLK = 286_000_000   # clocks per second of the 8pac timestamps
FRAME_CLK = 262_144       # clocks per B-frame
LEGACY_STREAM = 1         # cudaStreamLegacy: the stream torch works on unless told otherwise
NA, NB, MB = 32768, 36608, 18304
SIZE_A = 2.5 * NA * math.log2(NA)                                   # nominal flops of a C2R 32768
SIZE_BC = 2.5 * (NB * math.log2(NB) + NA * math.log2(NA))           # of an R2C 36608 and a C2R 32768


def listed():
    return [
        # the smallest call that gives an output: one batch, at a stream's start (latency)
        {"name": "first_batch_2", "kind": "process", "frames": 2, "precision": "fp32", "thresholds": "start",
         "host": False, "framed": False, "trim": 150},
        # a running stream taken in small pieces, leftover snapshots carried over
        {"name": "small_calls_12", "kind": "process", "frames": 12, "precision": "fp32", "thresholds": "kept",
         "host": False, "framed": False, "trim": 150},
        # the reference's unit of work: one group of a running stream, device buffers
        {"name": "group_143", "kind": "process", "frames": 143, "precision": "fp32", "thresholds": "kept",
         "host": False, "framed": False, "trim": 150},
        # a recorded scan in one call (the benchmark's workload)
        {"name": "scan_512", "kind": "process", "frames": 512, "precision": "fp32", "thresholds": "start",
         "host": False, "framed": False, "trim": 150},
        # a group from host memory to VDIF frames in host memory, as the hashpipe threads hand it over
        {"name": "host_framed_143", "kind": "process", "frames": 143, "precision": "fp32", "thresholds": "kept",
         "host": True, "framed": True, "trim": 150},
        # several streams of uneven lengths with drops and displaced packets, windowed thresholds
        {"name": "streams_4_window", "kind": "multi", "streams": 4, "frames_min": 64, "frames_max": 158,
         "precision": "fp32", "window": True},
        # packets as received (8pac units) to a shipped group
        {"name": "ingest_8pac_143", "kind": "ingest", "frames": 143, "precision": "fp32", "first_clk": 12_345_678},
        # the fast tensor-core form on a group, and on a short recording from its start
        {"name": "fast_group_143", "kind": "process", "frames": 143, "precision": "tc16_fast", "thresholds": "kept",
         "host": False, "framed": False, "trim": 150},
        {"name": "fast_start_16", "kind": "process", "frames": 16, "precision": "tc16_fast", "thresholds": "start",
         "host": False, "framed": False, "trim": 150},
        # the accurate tensor-core form
        {"name": "tc16_start_16", "kind": "process", "frames": 16, "precision": "tc16", "thresholds": "start",
         "host": False, "framed": False, "trim": 150},
        # the reference's functions one at a time, one batch
        {"name": "stages_1", "kind": "stages", "batches": 1, "trim": 150},
        # PFB-mode spectra
        {"name": "inverse_pfb_48", "kind": "pfb", "blocks": 48, "taps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["process", "process", "process", "process", "multi", "ingest", "stages", "pfb"])
    if kind == "process":
        precision = rng.choice(["fp32", "fp32", "tc16_fast", "tc16"])
        host = rng.random() < 0.25
        return {"kind": kind, "frames": _log(rng, 2, 143 if host or precision == "tc16" else 511),
                "precision": precision, "thresholds": rng.choice(["start", "kept"]), "host": host,
                "framed": rng.random() < 0.3, "trim": rng.randrange(0, 241)}
    if kind == "multi":
        streams = rng.randrange(2, 7)
        hi = _log(rng, 3, 511 // streams)
        return {"kind": kind, "streams": streams, "frames_min": _log(rng, 2, hi), "frames_max": hi,
                "precision": rng.choice(["fp32", "tc16_fast"]), "window": rng.random() < 0.5}
    if kind == "ingest":
        return {"kind": kind, "frames": rng.randrange(143, 287), "precision": rng.choice(["fp32", "tc16_fast"]),
                "first_clk": rng.randrange(1, SWARM_CLK)}
    if kind == "stages":
        return {"kind": kind, "batches": _log(rng, 1, 12), "trim": rng.randrange(0, 241)}
    return {"kind": kind, "blocks": _log(rng, 5, 128), "taps": rng.choice([2, 3, 4, 4, 4, 6, 8])}


# -- inputs -----------------------------------------------------------------

def _byte_table(gen, shift=0.0):
    """65536 payload bytes (four 2-bit codes each) distributed as a unit
    complex Gaussian sampled at the levels {-0.98, 0, 0.98}, offset by a tone."""
    g = torch.Generator().manual_seed(gen)
    x = torch.randn(65536, 4, generator=g) + shift
    code = (x >= -0.98).int() + (x >= 0).int() + (x >= 0.98).int()
    return (code[:, 0] | (code[:, 1] << 2) | (code[:, 2] << 4) | (code[:, 3] << 6)).to(torch.uint8).cuda()


def _packets(frames, seed, b_start):
    """B-engine packets of ``frames`` B-frames on the GPU: noise and one tone."""
    n = frames * N.PKTS_PER_FRAME
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pk = torch.empty((n, N.IN_PKT_BYTES), dtype=torch.uint8, device="cuda")
    noise, tone = _byte_table(seed), _byte_table(seed + 1, 0.4)
    for lo in range(0, n, 32768):
        hi = min(n, lo + 32768)
        r = torch.randint(0, 65536, (hi - lo, 1024), device="cuda", generator=gen, dtype=torch.int32)
        pk[lo:hi, 32:] = noise[r]
    at = seed * 37 % N.PKTS_PER_FRAME  # the tone's packet within each frame, channel 3 of its eight
    r = torch.randint(0, 65536, (frames, 128), device="cuda", generator=gen, dtype=torch.int32)
    pk.view(frames, N.PKTS_PER_FRAME, N.IN_PKT_BYTES)[:, at, 32::8] = tone[r]
    w = pk.view(torch.int32).view(frames, 256, 8, 264)
    b = b_start + torch.arange(frames, device="cuda")
    c = torch.arange(256, device="cuda")
    f = torch.arange(8, device="cuda")
    w[..., 0] = 12345
    w[..., 1] = (30 << 24) + (b % 125000)[:, None, None].int()
    w[..., 2] = 1056 // 8
    w[..., 3] = (1 << 26) | (ord("S") << 8) | ord("m")
    w[..., 4] = (b >> 8)[:, None, None].int()
    w5 = c[None, :, None] | (f[None, None, :] << 16) | ((b & 0xFF) << 24)[:, None, None]
    w[..., 5] = torch.where(w5 >= 1 << 31, w5 - (1 << 32), w5).int()
    w[..., 6] = torch.arange(n, device="cuda", dtype=torch.int32).view(frames, 256, 8)
    w[..., 7] = 0
    return pk


def _impaired(pk, seed):
    """1% of the packets dropped, 0.5% displaced by up to 64 places."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 5)
    pk = pk[torch.rand(len(pk), device="cuda", generator=gen) >= 0.01]
    place = torch.arange(len(pk), device="cuda", dtype=torch.float64)
    moved = torch.rand(len(pk), device="cuda", generator=gen) < 0.005
    place += moved * torch.rand(len(pk), device="cuda", generator=gen) * 64
    return pk[torch.argsort(place)].contiguous()


def _lengths(case):
    n, lo, hi = case["streams"], case["frames_min"], max(case["frames_min"], case["frames_max"])
    return [lo + (hi - lo) * (i * 7 % n) // max(1, n - 1) for i in range(n)]


def _out(rs, frames, framed):
    """An output buffer for any leftover of earlier calls."""
    batches = (frames * N.SNAPSHOTS_PER_FRAME + N.BATCH_SNAPSHOTS - 1) // N.BATCH_SNAPSHOTS
    return 2 * batches * N.PKTS_PER_BATCH * (N.OUT_PKT_BYTES if framed else N.OUT_PKT_DATA_BYTES)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_process(case, seed):
    frames, b0 = case["frames"], 1_000_000 + seed % 1000
    rs = Resampler(trim_mhz=case["trim"], max_frames=frames, precision=PRECISIONS[case["precision"]])
    pk = _packets(frames, seed, b0)
    nbytes = _out(rs, frames, case["framed"])
    if case["host"]:
        pinned = torch.empty(pk.shape, dtype=torch.uint8, pin_memory=True)
        pk = pinned.copy_(pk).numpy()
        out = torch.zeros(nbytes, dtype=torch.uint8, pin_memory=True).numpy()
    else:
        out = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    if case["thresholds"] == "kept":
        rs.process(pk, frames, b0, out=out, framed=case["framed"])
    return {"run": _run_process, "rs": rs, "packets": pk, "out": out, "frames": frames, "b0": b0, "case": case}


def _run_process(s):
    case = s["case"]
    if case["thresholds"] == "start":
        s["rs"].reset()
    # host buffers: the call returns when the payloads are in host memory
    s["rs"].process(s["packets"], s["frames"], s["b0"], out=s["out"], framed=case["framed"], want_result=False)
    return s["out"]


def _prepare_multi(case, seed):
    lengths = _lengths(case)
    rs, items = [], []
    for i, frames in enumerate(lengths):
        mode = N.THRESH_WINDOW if case["window"] else N.THRESH_FIRST_BATCH
        r = Resampler(max_frames=frames, precision=PRECISIONS[case["precision"]], threshold_mode=mode,
                      threshold_window=32 if case["window"] else 0, wave_batches=32)
        b0 = 1_000_000 + 100_000 * i + seed % 1000
        pk = _packets(frames, 100 * seed + i, b0)
        if case["window"]:
            pk = _impaired(pk, 100 * seed + i)
        rs.append(r)
        items.append((pk, frames, b0, torch.zeros(_out(r, frames, False), dtype=torch.uint8, device="cuda")))
    torch.cuda.synchronize()
    return {"run": _run_multi, "rs": rs, "items": items}


def _run_multi(s):
    for r in s["rs"]:
        r.reset()
    return process_multi(s["rs"], s["items"])


def _prepare_ingest(case, seed):
    frames = case["frames"]
    passes = 4096  # timestamps of that many batches are laid out here
    rs = Resampler(max_frames=GROUP, precision=PRECISIONS[case["precision"]])
    units = torch.empty((frames * 256, N.PAC8_BYTES), dtype=torch.uint8, device="cuda")
    pk = _packets(frames, seed, 0).view(-1, 8, N.IN_PKT_BYTES)
    for k in range(8):
        units[:, 1064 * k:1064 * k + N.IN_PKT_BYTES] = pk[:, k]
        if k:
            units[:, 1064 * k - 8:1064 * k] = k
    w = units.view(torch.int32).view(frames, 256, 2126)
    w[..., 2] = N.PAC8_BYTES // 8
    w4, w5 = (w.as_strided((frames, 256, 8), (256 * 2126, 2126, 266), w.storage_offset() + k) for k in (4, 5))
    cf = (torch.arange(256, device="cuda")[:, None] | (torch.arange(8, device="cuda")[None, :] << 8)).int()
    t = torch.arange(1 + passes * frames, device="cuda") * FRAME_CLK + 5_000 * SWARM_CLK + case["first_clk"]
    ts = ((t // SWARM_CLK) << 29) | (t % SWARM_CLK)
    hi = (ts >> 21).int()
    lo = (ts & 0x1FFFFF) << 11
    lo = torch.where(lo >= 1 << 31, lo - (1 << 32), lo).int()
    out = torch.zeros((frames // GROUP + 1, 2, Resampler.GROUP_PACKETS_OUT, N.OUT_PKT_DATA_BYTES), dtype=torch.uint8,
                      device="cuda")
    # the stream's first frame: groups are counted from the one after it
    w4[0].copy_(hi[0].expand(256, 8))
    torch.bitwise_or(cf, lo[0], out=w5[0])
    torch.cuda.synchronize()
    rs.ingest(units[:256], out=out, pac8=True)
    return {"run": _run_ingest, "rs": rs, "units": units, "w4": w4, "w5": w5, "cf": cf, "hi": hi, "lo": lo, "at": 1,
            "frames": frames, "out": out}


def _run_ingest(s):
    at, end = s["at"], s["at"] + s["frames"]
    s["at"] = end
    # the next received batch: the same payloads under the next frames' timestamps
    s["w4"].copy_(s["hi"][at:end, None, None].expand(end - at, 256, 8))
    torch.bitwise_or(s["cf"], s["lo"][at:end, None, None], out=s["w5"])
    torch.cuda.current_stream().synchronize()  # the batch has been received before it is handed over
    out, n = s["rs"].ingest(s["units"], out=s["out"], pac8=True)
    return [out, n]


def _prepare_stages(case, seed):
    nb = case["batches"]
    frames = -(-nb * N.BATCH_SNAPSHOTS // N.SNAPSHOTS_PER_FRAME)
    snaps, chunks = nb * N.BATCH_SNAPSHOTS, nb * N.PKTS_PER_BATCH
    dev = {"device": "cuda"}
    return {"run": _run_stages, "case": case, "frames": frames, "snaps": snaps, "chunks": chunks, "b0": 1_000_000,
            "rs": Resampler(trim_mhz=case["trim"], max_frames=frames), "packets": _packets(frames, seed, 1_000_000),
            "spec": torch.zeros((2, frames * N.SNAPSHOTS_PER_FRAME, 2048), dtype=torch.int32, **dev),
            "ints": torch.zeros(frames * 65 + 1, dtype=torch.int32, **dev),
            "series": torch.zeros((2, snaps * NA), **dev),
            "bins": torch.zeros((2, chunks, MB + 1), dtype=torch.complex64, **dev),
            "res": torch.zeros((2, chunks * NA), **dev), "direct": torch.zeros((2, chunks * NA), **dev),
            "words": torch.zeros((2, chunks * NA // 16), dtype=torch.int32, **dev),
            "beng": torch.zeros((2, frames * N.SNAPSHOTS_PER_FRAME, N.CHANNELS, 2), dtype=torch.int8, **dev)}


def _run_stages(s):
    lib, h = N.lib(), s["rs"].handle
    st = C.c_void_p(LEGACY_STREAM)
    p, frames, snaps, chunks, n = s["packets"], s["frames"], s["snaps"], s["chunks"], s["packets"].shape[0]
    spec, ints = s["spec"], s["ints"]
    ints.zero_()
    bitmap, counts = ints.data_ptr(), ints.data_ptr() + frames * 256
    N.check(lib.sdbe_vdif_to_beng(p.data_ptr(), n, s["b0"], frames, N.MAP_APHIDS, s["beng"][0].data_ptr(),
                                  s["beng"][1].data_ptr(), st))
    N.check(lib.sdbe_unpack(p.data_ptr(), n, s["b0"], frames, N.MAP_APHIDS, spec.data_ptr(), spec.stride(0), 0, bitmap,
                            counts, counts + frames * 4, st))
    N.check(lib.sdbe_fill_missing(bitmap, frames, N.MAP_APHIDS, spec.data_ptr(), spec.stride(0), 0, st))
    stats = []
    for pol in range(2):
        series, bins, res, words = s["series"][pol], s["bins"][pol], s["res"][pol], s["words"][pol]
        N.check(lib.sdbe_swarm_c2r(h, spec[pol].data_ptr(), snaps, series.data_ptr(), st))
        N.check(lib.sdbe_swarm_r2c(h, series.data_ptr(), chunks, bins.data_ptr(), st))
        N.check(lib.sdbe_r2dbe_c2r(h, bins.data_ptr(), chunks, s["rs"].skip_chan, res.data_ptr(), st))
        N.check(lib.sdbe_resample_chunks(h, series.data_ptr(), chunks, s["direct"][pol].data_ptr(), st))
        two = (C.c_double * 2)()
        N.check(lib.sdbe_summary_stats(res.data_ptr(), res.numel(), two, st))
        # the threshold and the offset go back in as the reference's floats
        N.check(lib.sdbe_quantize2bit(res.data_ptr(), words.data_ptr(), res.numel(), two[1], two[0], st))
        stats += [float(two[0]), float(two[1])]
    return {"beng": s["beng"], "spec": spec, "series": s["series"], "bins": s["bins"], "res": s["res"],
            "direct": s["direct"], "words": s["words"], "std": [stats[1], stats[3]]}


def _pfb_spectra(case, seed):
    """Spectra that a forward PFB gives for a unit noise stream with a tone."""
    nb, nt = case["blocks"], case["taps"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((nb + nt - 1, NA), device="cuda", generator=gen, dtype=torch.float64)
    x += torch.cos(0.37 * torch.arange(x.numel(), device="cuda", dtype=torch.float64)).view(x.shape)
    w = _pfb_window(nt)
    y = sum(w[t] * x[t:t + nb] for t in range(nt))
    return torch.fft.rfft(y).to(torch.complex64)


def _pfb_window(nt):
    n = torch.arange(nt * NA, device="cuda", dtype=torch.float64)
    return (0.54 - 0.46 * torch.cos(2 * math.pi * n / (nt * NA - 1))).view(nt, NA)


def _prepare_pfb(case, seed):
    return {"run": _run_pfb, "rs": Resampler(max_frames=2), "spec": _pfb_spectra(case, seed), "taps": case["taps"],
            "out": torch.empty((case["blocks"] + case["taps"] - 1, NA), device="cuda")}


def _run_pfb(s):
    return pfb.inverse_pfb(s["rs"], s["spec"], s["taps"], out=s["out"], stream=LEGACY_STREAM)


# -- what a pass cannot do without --------------------------------------------

def _stage_work(frames):
    """Packets in, payloads out, and the three transforms of ``frames`` B-frames."""
    snaps = 2 * frames * N.SNAPSHOTS_PER_FRAME
    chunks = snaps * N.PKTS_PER_BATCH // N.BATCH_SNAPSHOTS
    return (frames * N.PKTS_PER_FRAME * N.IN_PKT_BYTES + chunks * N.OUT_PKT_DATA_BYTES, snaps * SIZE_A + chunks * SIZE_BC)


def work(case):
    kind = case["kind"]
    if kind == "process":
        b, f = _stage_work(case["frames"])
    elif kind == "multi":
        b, f = (sum(v) for v in zip(*(_stage_work(n) for n in _lengths(case))))
    elif kind == "ingest":
        b, f = _stage_work(case["frames"])
    elif kind == "stages":
        nb = case["batches"]
        frames = -(-nb * N.BATCH_SNAPSHOTS // N.SNAPSHOTS_PER_FRAME)
        snaps, chunks = 2 * nb * N.BATCH_SNAPSHOTS, 2 * nb * N.PKTS_PER_BATCH
        rows = 2 * frames * N.SNAPSHOTS_PER_FRAME
        packets = frames * N.PKTS_PER_FRAME * N.IN_PKT_BYTES
        b = packets + rows * N.CHANNELS * 2                       # vdif_to_beng
        b += packets + rows * 8192                                # unpack
        b += snaps * (8192 + NA * 4) + chunks * (NB * 4 + (MB + 1) * 8)   # C2R, R2C
        b += chunks * (N.CHANNELS + 1) * 8 + chunks * NA * 4      # trimmed C2R
        b += chunks * (NB * 4 + NA * 4)                           # both fused
        b += chunks * NA * 4 + chunks * NA * (4 + 0.25)           # statistics, quantizer
        f = snaps * SIZE_A + 2 * chunks * SIZE_BC
    else:
        nb, nt = case["blocks"], case["taps"]
        b = nb * 16385 * 8 + (nb + nt - 1) * NA * 4
        f = nb * SIZE_A + nb * NA * (4.0 * nt + nt * nt)
    return {"bytes": float(b), "flops": float(f)}


# -- the same in 64 bits -------------------------------------------------------

def exact(case, seed):
    if case["kind"] == "stages":
        return _exact_stages(case, seed)
    if case["kind"] == "pfb":
        return _exact_pfb(case, seed)
    return None  # bytes and 2-bit codes


def _exact_stages(case, seed):
    nb = case["batches"]
    frames = -(-nb * N.BATCH_SNAPSHOTS // N.SNAPSHOTS_PER_FRAME)
    snaps = nb * N.BATCH_SNAPSHOTS
    pk = _packets(frames, seed, 1_000_000)
    # [frame][c][f][snapshot][byte]: byte 4 j + 3 - k is channel 4 j + k of the packet's eight
    pay = pk[:, 32:].reshape(frames, 256, 8, 128, 2, 4).flip(-1).reshape(frames, 256, 8, 128, 8)
    c = torch.arange(256, device="cuda")[:, None]
    f = torch.arange(8, device="cuda")[None, :]
    base = ((c >> 1) * 16 + (c & 1) + 2 * f).reshape(-1)  # in units of 8 channels
    rows = torch.empty((frames, 128, 2048, 8), dtype=torch.uint8, device="cuda")
    rows[:, :, base] = pay.reshape(frames, 2048, 128, 8).transpose(1, 2)
    rows = rows.reshape(frames * 128, N.CHANNELS)[:snaps]
    skip = int(case["trim"] * 1e6 / (4576e6 / NB))
    series, bins, res, std = [], [], [], []
    for pol in range(2):
        im = ((rows >> (4 if pol == 0 else 0)) & 3).double() - 2
        re = ((rows >> (6 if pol == 0 else 2)) & 3).double() - 2
        spec = torch.zeros((snaps, N.CHANNELS + 1), dtype=torch.complex128, device="cuda")
        spec[:, :-1] = torch.complex(re, im)
        x = torch.fft.irfft(spec, n=NA, norm="forward")
        z = torch.fft.rfft(x.reshape(-1, NB))
        r = torch.fft.irfft(z[:, skip:skip + N.CHANNELS + 1], n=NA, norm="forward").reshape(-1)
        series.append(x.reshape(-1))
        bins.append(z)
        res.append(r)
        std.append(float(r.std(unbiased=True)))
    res = torch.stack(res)
    return {"beng": None, "spec": None, "series": torch.stack(series), "bins": torch.stack(bins), "res": res,
            "direct": res, "words": None, "std": std}


def _exact_pfb(case, seed):
    """x = P^T (P P^T)^-1 y per phase: banded Cholesky over the blocks, all phases at once."""
    nb, nt = case["blocks"], case["taps"]
    y = torch.fft.irfft(_pfb_spectra(case, seed).to(torch.complex128), n=NA)
    w = _pfb_window(nt)
    a = [sum(w[k + d] * w[k] for k in range(nt - d)) for d in range(nt)]
    rows, v = [], []  # rows[m][k]: factor entry (m, m - k); v: forward-substituted y
    for m in range(nb):
        row = [None] * nt
        for k in range(min(nt - 1, m), -1, -1):
            s = a[k].clone()
            for q in range(k + 1, min(nt - 1, m) + 1):
                s -= row[q] * rows[m - k][q - k] if k else row[q] * row[q]
            row[k] = s / rows[m - k][0] if k else torch.sqrt(s)
        rows.append(row)
        t = y[m].clone()
        for k in range(1, min(nt - 1, m) + 1):
            t -= row[k] * v[m - k]
        v.append(t / row[0])
    z = [None] * nb
    for m in range(nb - 1, -1, -1):
        t = v[m].clone()
        for k in range(1, min(nt - 1, nb - 1 - m) + 1):
            t -= rows[m + k][k] * z[m + k]
        z[m] = t / rows[m][0]
    x = torch.zeros((nb + nt - 1, NA), dtype=torch.float64, device="cuda")
    for m in range(nb):
        x[m:m + nt] += w * z[m]
    return x
