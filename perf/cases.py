"""The calls whose time matters to a user of this receive path, and how to make and check them.

Every case goes through an entry point that a receiver, a transmitter or a link simulator calls:

* the stream BP -> OSD decoder of the (128,64) code, from host memory as the link's receive loop
  drives it and on resident batches as an error-rate simulation does;
* the CSR BP decoder on medium codes and on long codes of the DVB-S2 frame sizes, in the layered and
  the flooding schedules;
* the mixed-code engine on large batches and on a serving loop's small ones;
* the OFDM receiver on batches of frames and on one frame from host memory, and the transmitter.

`listed` names the sizes; `draw` takes others from the same ranges.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sicc-baseband-proto_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from sicc_gb300 import channel, codes, engine, fec, ofdm, pipeline  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one frame's worth of short codewords through the link's receive call: host LLRs in, bits
        # out, the smallest batch the link dispatches at once (its min_batch)
        {"name": "stream_host_30", "kind": "stream_host", "batch": 30, "ebn0": 3.0, "schedule": 3},
        # error-rate simulation of the short code: one resident batch per call, layered BP then
        # order-2 OSD on the failures
        {"name": "stream_65536", "kind": "stream", "batch": 65536, "ebn0": 2.0, "schedule": 3, "osd_order": 2},
        # the same decoder in the reference's own (flooding) schedule, a ragged batch
        {"name": "stream_flooding_8191", "kind": "stream", "batch": 8191, "ebn0": 2.0, "schedule": 0, "osd_order": 2},
        # 256 OFDM frames' codewords of the (1024,512) code
        {"name": "csr_1024_7680", "kind": "csr", "code": "ofdm", "batch": 7680, "ebn0": 2.0, "schedule": 3,
         "damping": 0.0},
        # a medium rate-3/4 code in the flooding schedule with the reference's damping
        {"name": "csr_flooding_2001", "kind": "csr", "code": "mixed11", "batch": 2001, "ebn0": 3.5, "schedule": 0,
         "damping": 0.15},
        # long broadcast-size codes, four codewords per SM, coloured layers
        {"name": "long_64800_608", "kind": "csr", "code": "N64800_R1/2", "batch": 608, "ebn0": 2.0, "schedule": 2,
         "damping": 0.0},
        # the shorter broadcast frame in the node-parallel flooding schedule, a ragged batch
        {"name": "long_16200_333", "kind": "csr", "code": "N16200_R5/6", "batch": 333, "ebn0": 4.0, "schedule": 1,
         "damping": 0.0},
        # a base station's mixed batch: 15 codes, n 128..2048, three rates, OSD on failures
        {"name": "engine_20000", "kind": "engine", "count": 20000, "burst": 512, "ebn0_lo": 1.0, "ebn0_hi": 5.0,
         "protect": False},
        # one small batch of a serving loop: a few requests, half of them BP only
        {"name": "engine_500", "kind": "engine", "count": 500, "burst": 64, "ebn0_lo": 1.0, "ebn0_hi": 5.0,
         "protect": True},
        # 256 received frames on the device: search, CFO, demodulation, LLRs
        {"name": "rx_256", "kind": "rx", "phy": "wide16", "frames": 256, "snr": 14.0, "taps": 6},
        # one received frame in host memory to host LLRs (the per-frame Pipeline call)
        {"name": "rx_frame_host", "kind": "rx_host", "phy": "video", "frames": 1, "snr": 14.0, "taps": 0},
        # 256 transmitted frames from resident information bits
        {"name": "tx_256", "kind": "tx", "phy": "wide16", "frames": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stream_host", "stream", "csr", "csr", "long", "engine", "engine", "rx", "rx_host", "tx"])
    if kind == "stream_host":
        return {"kind": kind, "batch": _log(rng, 1, 8192), "ebn0": round(rng.uniform(1.5, 4.5), 2),
                "schedule": rng.choice([0, 3])}
    if kind == "stream":
        flood = rng.random() < 0.3
        return {"kind": kind, "batch": _log(rng, 64, 16384 if flood else 65536),
                "ebn0": round(rng.uniform(1.5, 4.5), 2), "schedule": rng.choice([0, 1]) if flood else rng.choice([2, 3]),
                "osd_order": rng.choice([1, 2, 2])}
    if kind == "csr":
        code = rng.choice(["short", "ofdm"] + ["mixed%d" % i for i in range(15)])
        flood = rng.random() < 0.3
        bits = _log(rng, 1 << 14, 1 << (20 if flood else 22))
        return {"kind": kind, "code": code, "batch": max(1, bits // _code(code).n),
                "ebn0": round(rng.uniform(1.5, 4.5), 2), "schedule": rng.choice([0, 1]) if flood else rng.choice([2, 3]),
                "damping": rng.choice([0.0, 0.15]) if flood else 0.0}
    if kind == "long":
        code = rng.choice(["N64800_R1/2", "N16200_R1/4", "N16200_R1/2", "N16200_R5/6"])
        flood = rng.random() < 0.3
        most = 16200 * (333 if flood else 1216)
        return {"kind": "csr", "code": code, "batch": max(1, _log(rng, 16200 * 8, most) // _code(code).n),
                "ebn0": round(rng.uniform(1.5, 4.5), 2), "schedule": rng.choice([0, 1]) if flood else 2,
                "damping": 0.0}
    if kind == "engine":
        count = _log(rng, 30, 16000)
        return {"kind": kind, "count": count, "burst": rng.choice([16, 64, 512]), "ebn0_lo": 1.0,
                "ebn0_hi": round(rng.uniform(3.0, 6.0), 2), "protect": rng.random() < 0.5}
    if kind == "rx":
        return {"kind": kind, "phy": rng.choice(list(PHYS)), "frames": _log(rng, 1, 256),
                "snr": round(rng.uniform(10.0, 22.0), 1), "taps": rng.choice([0, 3, 6])}
    if kind == "rx_host":
        return {"kind": kind, "phy": rng.choice(list(PHYS)), "frames": 1, "snr": round(rng.uniform(10.0, 22.0), 1),
                "taps": 0}
    return {"kind": "tx", "phy": rng.choice(list(PHYS)), "frames": _log(rng, 1, 256)}


# ---------------------------------------------------------------------------
# codes, codewords, LLRs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _mixed():
    return codes.mixed_codes()


@functools.lru_cache(maxsize=None)
def _code(name):
    if name == "short":
        return codes.short_code()
    if name == "ofdm":
        return codes.ofdm_code()
    if name.startswith("mixed"):
        return _mixed()[int(name[5:])]
    return codes.dvbs2_code(name)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 17)


def _encode(code, info):
    """Systematic codewords [B][n] (uint8, on the device) of info [B][k]."""
    b = info.shape[0]
    if hasattr(code, "q"):  # accumulator code: row sums of the information bits, then a prefix XOR
        rows = np.repeat(np.arange(code.m), np.diff(code.row_ptr))
        keep = code.col_ind < code.k
        r = torch.from_numpy(rows[keep]).to(DEV)
        c = torch.from_numpy(code.col_ind[keep].astype(np.int64)).to(DEV)
        s = torch.zeros((code.m, b), dtype=torch.uint8, device=DEV)
        s.index_add_(0, r, info.t().contiguous()[c])
        parity = (torch.cumsum(s & 1, dim=0, dtype=torch.int32) & 1).to(torch.uint8).t()
        return torch.cat([info, parity], dim=1).contiguous()
    z, mb, kb = code.z, code.mb, code.nb - code.mb
    u = info.view(b, kb, z)
    blocks = []
    for j in range(mb):  # dual-diagonal parity part: base row j holds parity columns j - 1 and j
        acc = torch.zeros((b, z), dtype=torch.uint8, device=DEV)
        for c in range(kb):
            acc ^= torch.roll(u[:, c], -int(code.shifts[j, c]), dims=1)
        if j > 0:
            acc ^= torch.roll(blocks[j - 1], -int(code.shifts[j, kb + j - 1]), dims=1)
        blocks.append(torch.roll(acc, int(code.shifts[j, kb + j]), dims=1))
    return torch.cat([info] + blocks, dim=1)


def _awgn(code, count, ebn0, g):
    """float32 LLRs [count][n] of random codewords over BPSK + AWGN; ebn0 in dB, a number or a tensor [count]."""
    info = torch.randint(0, 2, (count, code.k), generator=g, device=DEV, dtype=torch.uint8)
    cw = _encode(code, info)
    e = torch.as_tensor(ebn0, dtype=torch.float32, device=DEV).reshape(-1, 1)
    sigma2 = 1.0 / (2.0 * code.rate * torch.pow(10.0, e / 10.0))
    noise = torch.randn((count, code.n), generator=g, device=DEV, dtype=torch.float32)
    return ((1.0 - 2.0 * cw.float() + torch.sqrt(sigma2) * noise) * (2.0 / sigma2)).contiguous()


# ---------------------------------------------------------------------------
# OFDM frames
# ---------------------------------------------------------------------------

#: PHY profiles: the 16-QAM receive workload, the reference benchmark's long QPSK frame, a dense
#: 64-QAM variant and a narrow BPSK one.
PHYS = {
    "wide16": ofdm.OFDM_C3,
    "video": ofdm.PhyConfig(nfft=1024, cp=72, num_symbols=96, active_sc=768, pre_half_len=256, modulation="qpsk",
                            pilot_period=4),
    "dense64": ofdm.PhyConfig(nfft=2048, cp=144, num_symbols=14, active_sc=1200, pre_half_len=512,
                              modulation="64qam", pilot_period=7),
    "narrow": ofdm.PhyConfig(nfft=256, cp=20, num_symbols=12, active_sc=150, pre_half_len=128, modulation="bpsk",
                             pilot_period=6),
}
PHY_CODE = {"wide16": "ofdm", "video": "short", "dense64": "ofdm", "narrow": "short"}
MAX_OFFSET, TAIL = 200, 64


@functools.lru_cache(maxsize=None)
def _tables(phy):
    return ofdm.reference_tables(PHYS[phy])


def _blocks(phy):
    return _tables(phy).coded_bits // _code(PHY_CODE[phy]).n


def _modulate(t, coded):
    """Frames [F][frame_len] (complex128, amplitude 1 before the peak or amplitude scaling) of coded bits."""
    cfg = t.cfg
    f, bps = coded.shape[0], cfg.bits_per_symbol
    idx = torch.zeros((f, coded.shape[1] // bps), dtype=torch.int64, device=DEV)
    for b in range(bps):
        idx = idx * 2 + coded.view(f, -1, bps)[:, :, b].long()
    pts = torch.from_numpy(t.constellation).to(DEV).to(torch.complex128)
    grid = torch.zeros((f, cfg.num_symbols, cfg.nfft), dtype=torch.complex128, device=DEV)
    bins = torch.from_numpy(t.used_bins.astype(np.int64)).to(DEV)
    data = torch.from_numpy(t.data_symbols.astype(np.int64)).to(DEV)
    pil = torch.from_numpy(t.pilot_symbols.astype(np.int64)).to(DEV)
    grid[:, data[:, None], bins[None, :]] = pts[idx].view(f, len(data), cfg.active_sc)
    grid[:, pil[:, None], bins[None, :]] = torch.from_numpy(t.pilot_grid).to(DEV).to(torch.complex128)
    td = torch.fft.ifft(grid, dim=2)
    td = torch.cat([td[:, :, cfg.nfft - cfg.cp:], td], dim=2).reshape(f, -1)
    pre = torch.from_numpy(t.preamble).to(DEV).to(torch.complex128)
    return torch.cat([pre.expand(f, -1), td], dim=1)


def _received(phy, frames, snr, taps, max_offset, tail, g):
    """(IQ [frames][samples] complex64, mean noise variance per FFT bin) through fading, CFO, delay and noise."""
    t, code = _tables(phy), _code(PHY_CODE[phy])
    cfg = t.cfg
    blocks = _blocks(phy)
    info = torch.randint(0, 2, (frames * blocks, code.k), generator=g, device=DEV, dtype=torch.uint8)
    fill = torch.randint(0, 2, (frames, t.coded_bits - blocks * code.n), generator=g, device=DEV, dtype=torch.uint8)
    x = _modulate(t, torch.cat([_encode(code, info).view(frames, -1), fill], dim=1))
    x = x * (cfg.amplitude / x.abs().amax(dim=1, keepdim=True))
    body = x[:, 2 * cfg.pre_half_len:].reshape(frames, cfg.num_symbols, cfg.nfft + cfg.cp)[:, :, cfg.cp:]
    bins = torch.from_numpy(t.used_bins.astype(np.int64)).to(DEV)
    power = torch.fft.fft(body, dim=2)[:, :, bins].abs().square().mean(dim=(1, 2))
    noise_var = power / 10.0 ** (snr / 10.0)
    if taps > 0:  # exponential power-delay profile, 3 dB per tap
        p = torch.pow(10.0, -0.3 * torch.arange(taps, device=DEV, dtype=torch.float64))
        p = torch.sqrt(p / p.sum() / 2.0)
        h = torch.randn((frames, taps, 2), generator=g, device=DEV, dtype=torch.float64) * p[None, :, None]
        h = torch.view_as_complex(h)
        y = torch.zeros((frames, x.shape[1] + taps - 1), dtype=torch.complex128, device=DEV)
        for i in range(taps):
            y[:, i:i + x.shape[1]] += h[:, i:i + 1] * x
        x = y
    n = max_offset + t.frame_len + tail
    off = torch.randint(0, max_offset + 1, (frames, 1), generator=g, device=DEV)
    at = torch.arange(n, device=DEV)[None, :] - off
    y = torch.where((at >= 0) & (at < x.shape[1]), torch.gather(x, 1, at.clamp(0, x.shape[1] - 1)), 0.0)
    y = y * torch.exp(2j * math.pi * 0.1 / cfg.nfft * at)  # a tenth of a subcarrier of carrier offset
    noise = torch.view_as_complex(torch.randn((frames, n, 2), generator=g, device=DEV, dtype=torch.float64))
    y = y + noise * torch.sqrt(noise_var / cfg.nfft / 2.0)[:, None]
    return y.to(torch.complex64).contiguous(), float(noise_var.mean())


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def _engine_input(case, g):
    cs = _mixed()
    rng = np.random.default_rng([case["count"], case["burst"]])  # the requests of a case; their LLRs go by the seed
    req, sizes, left = [], [], case["count"]
    while left > 0:
        b = int(min(rng.integers(1, case["burst"] + 1), left))
        req.append(int(rng.integers(0, len(cs))))
        sizes.append(b)
        left -= b
    code_of = np.repeat(np.array(req), sizes)
    ns = np.array([c.n for c in cs], np.int64)[code_of]
    ks = np.array([c.k for c in cs], np.int64)[code_of]
    llr_off = np.concatenate([[0], np.cumsum(ns)[:-1]])
    info_off = np.concatenate([[0], np.cumsum(ks)[:-1]])
    llr = torch.empty(int(ns.sum()), dtype=torch.float32, device=DEV)
    for c in sorted(set(req)):
        rows = np.nonzero(code_of == c)[0]
        ebn0 = case["ebn0_lo"] + (case["ebn0_hi"] - case["ebn0_lo"]) * torch.rand(len(rows), generator=g, device=DEV)
        at = torch.from_numpy(llr_off[rows]).to(DEV)[:, None] + torch.arange(cs[c].n, device=DEV)
        llr[at.reshape(-1)] = _awgn(cs[c], len(rows), ebn0, g).reshape(-1)
    return code_of, ns, ks, llr_off, info_off, llr


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    s = {"case": case, "kind": kind}
    u8 = functools.partial(torch.zeros, dtype=torch.uint8, device=DEV)
    if kind in ("stream", "stream_host"):
        code, b = _code("short"), case["batch"]
        llr = _awgn(code, b, case["ebn0"], g)
        s["dec"] = fec.StreamBpOsdDecoder(code, max_batch=4096 if kind == "stream_host" else b, max_iter=20,
                                          normalization=0.75, offset=0.0, damping=0.0, min_abs_llr_accept=0.0,
                                          schedule=case["schedule"], osd_order=case.get("osd_order", 2))
        if kind == "stream_host":
            s["llr"] = llr.cpu().numpy()
        else:
            s.update(llr=llr, info=u8((b, code.k)), ok=u8(b), used=u8(b), it=u8(b))
    elif kind == "csr":
        code, b = _code(case["code"]), case["batch"]
        s["llr"] = _awgn(code, b, case["ebn0"], g)
        s["dec"] = fec.CsrBpDecoder.for_code(code, max_batch=b, max_iter=engine.iteration_cap(code.n), normalization=0.75,
                                             damping=case["damping"], schedule=case["schedule"])
        s.update(bits=u8((b, code.n)), ok=u8(b), it=u8(b))
    elif kind == "engine":
        code_of, ns, ks, llr_off, info_off, llr = _engine_input(case, g)
        n = len(code_of)
        eng = engine.Engine(n, int(ns.sum()))
        for c in _mixed():
            eng.add_code(c, max_iter=engine.iteration_cap(c.n), osd_order=engine.osd_order_for(c))
        s.update(eng=eng, n=n, llr=llr, code_of=torch.from_numpy(code_of.astype(np.uint8)).to(DEV),
                 llr_off=torch.from_numpy(llr_off).to(DEV), info_off=torch.from_numpy(info_off).to(DEV),
                 info=u8(int(ks.sum())), ok=u8(n), used=u8(n), it=u8(n), protect=None)
        if case["protect"]:
            s["protect"] = torch.randint(0, 2, (n,), generator=g, device=DEV, dtype=torch.uint8)
    elif kind in ("rx", "rx_host"):
        f, t, code = case["frames"], _tables(case["phy"]), _code(PHY_CODE[case["phy"]])
        host = kind == "rx_host"
        iq, nv = _received(case["phy"], f, case["snr"], case["taps"], 0 if host else MAX_OFFSET, 0 if host else TAIL, g)
        s["nv"] = float(np.float32(nv))
        s["pipe"] = pipeline.RxPipeline(t, code.n, code.k, _blocks(case["phy"]), s["nv"], max_batch_frames=f)
        if host:
            s["iq"] = iq[0, :t.frame_len].cpu().numpy()
        else:
            s.update(iq=iq, llr=torch.zeros((f, s["pipe"].coded_bits), dtype=torch.float32, device=DEV),
                     sync=torch.zeros((f, 6), dtype=torch.int32, device=DEV))
    else:
        f, t, code = case["frames"], _tables(case["phy"]), _code(PHY_CODE[case["phy"]])
        pipe = pipeline.RxPipeline(t, code.n, code.k, _blocks(case["phy"]), 0.1, max_batch_frames=f)
        gen = np.concatenate([np.eye(code.k, dtype=np.uint8), channel.parity_matrix(code)], axis=1)
        pipe.upload_tx_tables(generator_kn=gen)
        info = torch.randint(0, 2, (f, _blocks(case["phy"]) * code.k), generator=g, device=DEV, dtype=torch.uint8)
        s.update(pipe=pipe, info=info, out=torch.zeros((f, t.frame_len), dtype=torch.complex64, device=DEV))
    return s


def run(s):
    kind = s["kind"]
    if kind == "stream_host":
        info, used = s["dec"].decode(s["llr"])
        return {"info": info, "used": used}
    st = torch.cuda.current_stream()
    if kind == "stream":
        s["dec"].decode_device_batch(s["llr"], s["info"], s["ok"], s["used"], s["it"], stream=st)
        return {"info": s["info"], "ok": s["ok"], "used": s["used"], "it": s["it"]}
    if kind == "csr":
        s["dec"].decode_device_batch(s["llr"], s["bits"], s["ok"], None, s["it"], stream=st)
        return {"bits": s["bits"], "ok": s["ok"], "it": s["it"]}
    if kind == "engine":
        s["eng"].decode_device(s["n"], s["code_of"], s["llr"], s["llr_off"], s["info"], s["info_off"], s["ok"],
                               s["used"], s["it"], stream=st, d_protection=s["protect"])
        return {"info": s["info"], "ok": s["ok"], "used": s["used"], "it": s["it"]}
    if kind == "rx":
        n = s["iq"].shape[1]
        s["pipe"].demod_batch(s["iq"], n, n, s["iq"].shape[0], s["llr"], s["sync"], stream=st)
        sync = s["sync"]
        return {"llr": s["llr"], "found": sync[:, 0], "start": sync[:, 1],
                "metrics": sync.view(torch.float32)[:, 2:5]}  # coarse, fine, CFO
    if kind == "rx_host":
        llr, (start, fine, cfo) = s["pipe"].demod_to_host(0, s["iq"])
        return {"llr": llr, "start": int(start), "metrics": np.array([fine, cfo], np.float32)}
    s["pipe"].tx_batch(s["info"], s["info"].shape[0], s["out"], stream=st)
    return {"frames": s["out"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Inputs read once, outputs written once; per BP iteration an edge costs a subtraction, two
    comparisons, a scaling and an addition (typical mean iteration counts), an FFT 5 N log2 N, a
    frame search one multiply-add chain per candidate step.  OSD is integer work: not counted."""
    kind = case["kind"]
    if kind in ("stream", "stream_host"):
        c, b = _code("short"), case["batch"]
        return {"bytes": b * (4 * c.n + c.k + 3), "flops": 5 * c.edges * b * (6 if case["ebn0"] < 3 else 3)}
    if kind == "csr":
        c, b = _code(case["code"]), case["batch"]
        return {"bytes": b * (4 * c.n + c.n + 2), "flops": 5 * c.edges * b * (14 if c.n > 10000 else 6)}
    if kind == "engine":
        cs = _mixed()
        n, k, e = (sum(getattr(c, a) for c in cs) / len(cs) for a in ("n", "k", "edges"))
        return {"bytes": case["count"] * (4 * n + k + 20), "flops": 5 * e * 8 * case["count"]}
    t, f = _tables(case["phy"]), case["frames"]
    cfg, kept = t.cfg, _blocks(case["phy"]) * _code(PHY_CODE[case["phy"]]).n
    fft = 5 * cfg.nfft * math.log2(cfg.nfft) * cfg.num_symbols
    if kind == "tx":
        return {"bytes": f * (kept * _code(PHY_CODE[case["phy"]]).rate + 8 * t.frame_len), "flops": f * fft}
    return {"bytes": f * (8 * t.frame_len + 4 * kept), "flops": f * (fft + 30 * cfg.nfft + 20 * kept)}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------

def _exact_sync(t, x):
    """The receiver's frame search in double precision: (found, start, coarse, fine, cfo) per frame."""
    cfg = t.cfg
    f, n = x.shape
    L, pre = cfg.pre_half_len, 2 * cfg.pre_half_len
    limit = n - pre + 1
    radius = min(16, cfg.cp)

    def windows(v, length):  # sums over [d, d + length) for d < limit
        c = torch.cat([torch.zeros((f, 1), dtype=v.dtype, device=DEV), torch.cumsum(v, dim=1)], dim=1)
        return c[:, length:length + limit] - c[:, :limit]

    p = windows(x[:, :n - L].conj() * x[:, L:], L)
    e = x.abs().square()
    e1 = windows(e, L)
    e2 = windows(e[:, L:], L)
    coarse = p.abs().square() / torch.clamp(e1 * e2, min=1e-18)
    q = torch.from_numpy(t.preamble).to(DEV).to(torch.complex128)
    m = 1 << (n + pre).bit_length()
    corr = torch.fft.ifft(torch.fft.fft(x, m, dim=1) * torch.fft.fft(q, m).conj(), dim=1)[:, :limit]
    fine = corr.abs().square() / torch.clamp(windows(e, pre) * float(q.abs().square().sum()), min=1e-18)
    best = torch.nn.functional.max_pool1d(fine[:, None], 2 * radius + 1, stride=1, padding=radius)[:, 0]
    hit = (coarse >= cfg.sync_threshold) & (best >= cfg.sync_threshold)
    any_hit = hit.any(dim=1)
    cand = hit.int().argmax(dim=1)
    at = cand[:, None] + torch.arange(-radius, radius + 1, device=DEV)
    w = torch.where((at >= 0) & (at < limit), torch.gather(fine, 1, at.clamp(0, limit - 1)), -1.0)
    start = torch.gather(at, 1, w.argmax(dim=1, keepdim=True))[:, 0]
    i = start[:, None].clamp(min=0) + torch.arange(L, device=DEV)
    ac = (torch.gather(x, 1, i).conj() * torch.gather(x, 1, i + L)).sum(dim=1)
    cfo = torch.angle(ac) * cfg.sample_rate / (2.0 * math.pi * L)
    zero = torch.zeros(f, dtype=torch.float64, device=DEV)
    found = torch.where(any_hit, torch.where(start + t.frame_len > n, 2, 1), 0)
    return (found, torch.where(any_hit, start, -1),
            torch.where(any_hit, torch.gather(coarse, 1, cand[:, None])[:, 0], zero),
            torch.where(any_hit, torch.gather(fine, 1, start[:, None].clamp(min=0))[:, 0], zero),
            torch.where(any_hit, cfo, zero))


def _exact_demod(t, x, start, cfo, noise_var, kept):
    """Max-log LLRs [kept] of one frame in double precision."""
    cfg = t.cfg
    bps, L = cfg.bits_per_symbol, cfg.nfft + cfg.cp
    off = 2 * cfg.pre_half_len + torch.arange(cfg.num_symbols, device=DEV)[:, None] * L + cfg.cp + \
        torch.arange(cfg.nfft, device=DEV)
    at = start + off
    smp = torch.where(at < x.shape[0], x[at.clamp(max=x.shape[0] - 1)], 0.0)
    smp = smp * torch.exp(-2j * math.pi * (cfo / cfg.sample_rate) * off)
    grid = torch.fft.fft(smp, dim=1)[:, torch.from_numpy(t.used_bins.astype(np.int64)).to(DEV)]
    ix = lambda a: torch.from_numpy(np.asarray(a).astype(np.int64)).to(DEV)  # noqa: E731
    pil = torch.from_numpy(t.pilot_grid).to(DEV).to(torch.complex128)
    hp = grid[ix(t.pilot_symbols)] * pil.conj() / torch.clamp(pil.abs().square(), min=1e-9)
    al = torch.from_numpy(t.interp_alpha.astype(np.float64)).to(DEV)[:, None]
    h = hp[ix(t.interp_p0)] * (1.0 - al) + hp[ix(t.interp_p1)] * al
    y = grid[ix(t.data_symbols)]
    h2 = torch.clamp(h.abs().square(), min=1e-9)
    eq = y * h.conj() / (h2 + noise_var)
    sig = torch.clamp(noise_var / h2, min=1e-8)
    if bps == 1:
        return (((eq + 1.0).abs().square() - (eq - 1.0).abs().square()) / sig).reshape(-1)[:kept]
    ab = bps // 2
    lv = torch.from_numpy(t.axis_levels.astype(np.float64)).to(DEV)
    out = []
    for part in (eq.real, eq.imag):
        d = (part[..., None] - lv).square()
        for b in range(ab):
            bit = (torch.arange(len(lv), device=DEV) >> (ab - 1 - b)) & 1
            out.append((d[..., bit == 1].amin(-1) - d[..., bit == 0].amin(-1)) / sig)
    return torch.stack(out, dim=-1).reshape(-1)[:kept]


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("rx", "rx_host", "tx"):
        return None  # decoded bits and counts: no rounding
    g = _gen(seed)
    phy, f = case["phy"], case["frames"]
    t, code, blocks = _tables(phy), _code(PHY_CODE[phy]), _blocks(phy)
    kept = blocks * code.n
    if kind == "tx":
        info = torch.randint(0, 2, (f, blocks * code.k), generator=g, device=DEV, dtype=torch.uint8)
        coded = torch.zeros((f, t.coded_bits), dtype=torch.uint8, device=DEV)
        coded[:, :kept] = _encode(code, info.view(-1, code.k)).view(f, -1)
        return {"frames": _modulate(t, coded) * t.cfg.amplitude}
    host = kind == "rx_host"
    iq, nv = _received(phy, f, case["snr"], case["taps"], 0 if host else MAX_OFFSET, 0 if host else TAIL, g)
    nv = float(np.float32(nv))
    x = iq.to(torch.complex128)
    if host:
        x = x[:, :t.frame_len]
    parts = [_exact_sync(t, x[i:i + 32]) for i in range(0, f, 32)]
    found, start, coarse, fine, cfo = (torch.cat([p[i] for p in parts]) for i in range(5))
    llr = torch.zeros((f, kept), dtype=torch.float64, device=DEV)
    for i in range(f):
        if int(found[i]) == 1 or (host and int(found[i]) == 2):
            llr[i] = _exact_demod(t, x[i], int(start[i]), float(cfo[i]), nv, kept)
    if host:
        one = int(found[0]) == 1
        return {"llr": llr[0].cpu().numpy(), "start": None,
                "metrics": np.array([float(fine[0]), float(cfo[0]) if one else 0.0])}
    return {"llr": llr, "found": None, "start": None, "metrics": torch.stack([coarse, fine, cfo], dim=1)}
