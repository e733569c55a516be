"""Calls that the entry points accept, at the edges of what the fast paths take.

Arrays that start away from a 16-byte boundary, codes and grids beyond a kernel's shared memory, thresholds
equal to a metric, shapes that were tried and given up or saved for other kernels, columns and information
blocks longer than usual.  Results are compared with the same call in its ordinary form or with the oracle.
"""
import types

import numpy as np
import pytest

from sicc_gb300 import channel, codes, engine, fec, ofdm, tune

pytestmark = pytest.mark.gpu


# --- soft values away from a 16-byte boundary ---------------------------------------------------------

def _decode(torch, dec, d_llr, n):
    b = d_llr.shape[0]
    out = [torch.zeros((b, n), dtype=torch.uint8, device="cuda"), torch.zeros(b, dtype=torch.uint8, device="cuda"),
           torch.zeros((b, n), dtype=torch.float32, device="cuda"), torch.zeros(b, dtype=torch.uint8, device="cuda")]
    dec.decode_device_batch(d_llr, *out, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    return [x.cpu().numpy() for x in out]


def _offset(torch, llr, floats):
    """The rows as a view that starts `floats` floats into a buffer."""
    buf = torch.zeros(llr.size + 4, dtype=torch.float32, device="cuda")
    view = buf[floats:floats + llr.size].view(llr.shape)
    view.copy_(torch.from_numpy(llr))
    assert view.data_ptr() % 16 == 4 * floats
    return view


@pytest.mark.parametrize("floats", [1, 2, 3])
@pytest.mark.parametrize("schedule", [fec.FLOODING, fec.NODE_PARALLEL, fec.COLORED_LAYERED, fec.FLAT_LAYERED])
@pytest.mark.parametrize("base", [(4, 8, 16), (8, 16, 64), (8, 16, 128), (4, 8, 33)])
def test_unaligned_soft_values_register_kernels(cuda, base, schedule, floats):
    code = codes.qc_code(*base, seed=41)
    llr = channel.awgn_llrs(code, 37, 2.0, 3)[2].astype(np.float32)
    dec = fec.CsrBpDecoder.for_code(code, max_batch=37, max_iter=10, normalization=0.8, schedule=schedule)
    want = _decode(cuda, dec, cuda.from_numpy(llr).cuda(), code.n)
    for a, b in zip(want, _decode(cuda, dec, _offset(cuda, llr, floats), code.n)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("floats", [1, 2, 3])
@pytest.mark.parametrize("base", [(6, 12, 64), (7, 14, 96)])
def test_unaligned_soft_values_general_layered_kernel(cuda, base, floats):
    """Codes whose rows fit no register-resident shape."""
    code = codes.qc_code(*base, seed=41)
    llr = channel.awgn_llrs(code, 37, 2.0, 3)[2].astype(np.float32)
    dec = fec.CsrBpDecoder.for_code(code, max_batch=37, max_iter=10, normalization=0.8, schedule=fec.FLAT_LAYERED)
    want = _decode(cuda, dec, cuda.from_numpy(llr).cuda(), code.n)
    for a, b in zip(want, _decode(cuda, dec, _offset(cuda, llr, floats), code.n)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("schedule", [fec.NODE_PARALLEL, fec.FLAT_LAYERED])
def test_unaligned_soft_values_stream_decoder(cuda, schedule):
    """BP with its best posteriors kept for OSD."""
    torch, code = cuda, codes.short_code()
    llr = channel.awgn_llrs(code, 500, 2.0, 4)[2].astype(np.float32)
    dec = fec.StreamBpOsdDecoder(code, max_batch=500, max_iter=20, schedule=schedule)

    def run(d_llr):
        out = [torch.zeros((500, code.k), dtype=torch.uint8, device="cuda")] + \
              [torch.zeros(500, dtype=torch.uint8, device="cuda") for _ in range(3)]
        dec.decode_device_batch(d_llr, *out, stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in out]

    want = run(torch.from_numpy(llr).cuda())
    assert want[2].any()  # some went through OSD
    for a, b in zip(want, run(_offset(torch, llr, 1))):
        assert np.array_equal(a, b)


# --- codes of millions of bits ------------------------------------------------------------------------------

@pytest.mark.parametrize("damping", [0.0, 0.2])
@pytest.mark.parametrize("n", [1851360, 1851362, 2000000])  # the packed hard decisions in and past shared memory
def test_flooding_of_a_huge_code(cuda, oracle, n, damping):
    m = n // 2
    k, r = n - m, np.arange(m, dtype=np.int64)
    cols = np.stack([(3 * r) % k, (3 * r + 1 + r % 1001) % k, k + np.maximum(r - 1, 0), k + r], axis=1)
    cols.sort(axis=1)
    keep = np.ones((m, 4), bool)
    keep[0, 3] = False  # the first row has no previous parity
    row_ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    col_ind = cols[keep].astype(np.int32)
    llr = (2.0 / 0.4 * (1.0 + np.sqrt(0.4) * np.random.default_rng(n).standard_normal((2, n)))).astype(np.float32)
    dec = fec.CsrBpDecoder(n, m, row_ptr, col_ind, max_batch=2, max_iter=3, normalization=0.8, damping=damping,
                           schedule=fec.FLOODING)
    got = _decode(cuda, dec, cuda.from_numpy(llr).cuda(), n)
    oc = oracle.code(n, m, row_ptr, col_ind)
    for i, x in enumerate(llr):
        o = oc.flooding(x, 3, 0.8, 0.0, damping)
        assert got[1][i] == o[0] and got[3][i] == o[4]
        assert np.array_equal(got[0][i], o[1]) and np.array_equal(got[2][i], o[2])


# --- OFDM receiver --------------------------------------------------------------------------------------

@pytest.mark.parametrize("modulation", ["bpsk", "qpsk", "16qam", "64qam"])
def test_gather_to_unaligned_llr_rows(cuda, modulation):
    """demod_gather writes each frame's LLRs wherever the caller says, at any float."""
    from sicc_gb300.pipeline import SYNC_RECORD, RxPipeline
    torch = cuda
    cfg = ofdm.PhyConfig(nfft=128, cp=16, num_symbols=8, active_sc=64, pre_half_len=64, modulation=modulation,
                         pilot_period=4)
    t, code = ofdm.reference_tables(cfg), codes.short_code()
    b = ofdm.FrameGenerator(t, code, seed=5).batch(4, snr_db=25.0, cfo_subcarriers=0.05, max_offset=30, rayleigh_taps=0)
    p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, float(b.noise_var[0]), max_batch_frames=4)
    iq, n, st = torch.from_numpy(b.iq).cuda(), b.iq.shape[1], torch.cuda.current_stream()
    sync = torch.zeros(4 * SYNC_RECORD.itemsize, dtype=torch.uint8, device="cuda")
    want = torch.zeros((4, p.coded_bits), dtype=torch.float32, device="cuda")
    p.demod_batch(iq, n, n, 4, want, sync, st)
    rows = [f * (p.coded_bits + 4) + f for f in range(4)]  # 0 to 3 floats off
    got = torch.zeros(4 * (p.coded_bits + 5), dtype=torch.float32, device="cuda")
    p.demod_gather(iq, torch.arange(4, device="cuda") * n, n, 4, got, torch.tensor(rows, device="cuda"), sync, st)
    torch.cuda.synchronize()
    assert want.abs().sum() > 0
    for f in range(4):
        assert torch.equal(got[rows[f]:rows[f] + p.coded_bits], want[f]), f


def _large_grid(active, modulation):
    """4,096 points, every second symbol a pilot: a demodulator CTA holds four pilots of `active` subcarriers."""
    cfg = ofdm.PhyConfig(nfft=4096, cp=288, num_symbols=13, active_sc=active, pre_half_len=200, modulation=modulation,
                         pilot_period=2)
    return ofdm.reference_tables(cfg)


@pytest.mark.parametrize("frames", [1, 60])
@pytest.mark.parametrize("active,modulation", [(3168, "qpsk"), (3172, "qpsk"), (3276, "bpsk"), (3276, "16qam"),
                                               (3276, "64qam"), (3424, "qpsk")])
def test_demodulator_near_its_shared_memory_limit(cuda, oracle, active, modulation, frames):
    from sicc_gb300.pipeline import SYNC_RECORD, RxPipeline
    from test_gpu_ofdm import _llr_close
    torch = cuda
    t, code = _large_grid(active, modulation), codes.short_code()
    b = ofdm.FrameGenerator(t, code, seed=19).batch(2, snr_db=25.0, cfo_subcarriers=0.05, max_offset=60, rayleigh_taps=0)
    iq = np.tile(b.iq, ((frames + 1) // 2, 1))[:frames]
    p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, float(b.noise_var[0]), max_batch_frames=frames)
    llr = torch.zeros((frames, p.coded_bits), dtype=torch.float32, device="cuda")
    rec = torch.zeros(frames * SYNC_RECORD.itemsize, dtype=torch.uint8, device="cuda")
    p.demod_batch(torch.from_numpy(iq).cuda(), iq.shape[1], iq.shape[1], frames, llr, rec, torch.cuda.current_stream())
    torch.cuda.synchronize()
    sync, got, ph = rec.cpu().numpy().view(SYNC_RECORD), llr.cpu().numpy(), oracle.phy(t)
    for f in range(min(frames, 2)):
        r = oracle.sync_earliest(ph, iq[f])
        assert sync[f]["found"] == r[0] == 1 and sync[f]["start"] == r[1]
        ref = oracle.demod_frame(ph, iq[f][r[1]:r[1] + t.frame_len], float(sync[f]["cfo_hz"]),
                                 float(np.float32(b.noise_var[0])))
        _llr_close(got[f], ref[: p.coded_bits])
    for f in range(2, frames):
        assert np.array_equal(got[f], got[f % 2]), f


def test_demodulator_past_its_shared_memory_limit_is_refused(cuda):
    from sicc_gb300 import _lib
    from sicc_gb300.pipeline import RxPipeline
    torch = cuda
    t, code = _large_grid(3426, "qpsk"), codes.short_code()
    p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, 0.1, max_batch_frames=1)
    iq = torch.zeros((1, t.frame_len), dtype=torch.complex64, device="cuda")
    llr = torch.zeros((1, p.coded_bits), dtype=torch.float32, device="cuda")
    with pytest.raises(_lib.SiccError, match="shared memory"):
        p.demod_batch(iq, t.frame_len, t.frame_len, 1, llr, None, torch.cuda.current_stream())


@pytest.mark.parametrize("value", [0.8349244594573975 + 0.571209192276001j, 0.6395646333694458 + 0.7616397142410278j,
                                   0.5345859527587891 + 0.8649413585662842j])
@pytest.mark.parametrize("half", [24, 3968, 7936])  # no first half to stop after; long sums
def test_search_at_a_threshold_equal_to_the_metric(cuda, half, value):
    """A frame whose fine metric is exactly the threshold is found.  The preamble repeats one value whose
    square rounds the same way in every step of a sum, so long sums are off by more than 1e-5; each half
    begins and ends with three zeros, so the neighbouring positions have the same energy."""
    import dataclasses
    from sicc_gb300.pipeline import SYNC_RECORD, RxPipeline
    torch, code, at = cuda, codes.short_code(), 303

    def search(threshold):
        cfg = ofdm.PhyConfig(nfft=64, cp=16, num_symbols=6, active_sc=32, pre_half_len=half, modulation="qpsk",
                             pilot_period=3, sync_threshold=float(threshold))
        pre = np.full((2, half), value, np.complex64)
        pre[:, :3] = pre[:, -3:] = 0
        t = dataclasses.replace(ofdm.reference_tables(cfg), preamble=pre.reshape(-1))
        iq = np.zeros((1, at + t.frame_len + 50), np.complex64)
        iq[0, at:at + 2 * half] = t.preamble
        p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, 0.1, max_batch_frames=1)
        llr = torch.zeros((1, p.coded_bits), dtype=torch.float32, device="cuda")
        rec = torch.zeros(SYNC_RECORD.itemsize, dtype=torch.uint8, device="cuda")
        p.demod_batch(torch.from_numpy(iq).cuda(), iq.shape[1], iq.shape[1], 1, llr, rec, torch.cuda.current_stream())
        torch.cuda.synchronize()
        return rec.cpu().numpy().view(SYNC_RECORD)[0]

    first = search(1.0 - 0.9 / half)
    assert first["found"] == 1 and first["start"] == at
    again = search(min(first["coarse"], first["fine"], 1.0))
    assert again["found"] == 1 and again["start"] == at
    assert again["fine"] == first["fine"]


@pytest.mark.parametrize("cfo", [0.05, 0.45, -0.45])
def test_derotation_error_does_not_grow_along_the_frame(cuda, cfo):
    """LLRs of a long frame against double precision, for the carrier offset the receiver estimated.  At 0.45
    subcarriers the frame turns 46 times: an angle rounded before its reduction is off by up to 46 x 2^-24
    turns, 1.7e-5 rad.  Reduced first, a rotation is off by less than 4e-7 (angle 1e-7, sincospi 1.2e-7, a
    product 1.7e-7), the FFT by 10 x 6e-8 more, and the LLR's quotient doubles that: 2e-6."""
    from sicc_gb300.pipeline import SYNC_RECORD, RxPipeline
    torch, code = cuda, codes.short_code()
    cfg = ofdm.PhyConfig(nfft=1024, cp=72, num_symbols=96, active_sc=768, pre_half_len=256, modulation="qpsk",
                         pilot_period=4)
    t = ofdm.reference_tables(cfg)
    b = ofdm.FrameGenerator(t, code, seed=4).batch(1, snr_db=25.0, cfo_subcarriers=cfo, max_offset=40, rayleigh_taps=0)
    p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, float(b.noise_var[0]), max_batch_frames=1)
    llr = torch.zeros((1, p.coded_bits), dtype=torch.float32, device="cuda")
    rec = torch.zeros(SYNC_RECORD.itemsize, dtype=torch.uint8, device="cuda")
    p.demod_batch(torch.from_numpy(b.iq).cuda(), b.iq.shape[1], b.iq.shape[1], 1, llr, rec, torch.cuda.current_stream())
    torch.cuda.synchronize()
    sync = rec.cpu().numpy().view(SYNC_RECORD)[0]
    assert sync["found"] == 1
    nv, rate = float(np.float32(b.noise_var[0])), float(np.float32(cfg.sample_rate))
    n = 2 * cfg.pre_half_len + np.arange(cfg.num_symbols)[:, None] * (cfg.nfft + cfg.cp) + cfg.cp + np.arange(cfg.nfft)
    x = b.iq[0][int(sync["start"]) + n].astype(np.complex128) * np.exp(-2j * np.pi * float(sync["cfo_hz"]) / rate * n)
    grid = np.fft.fft(x, axis=1)[:, t.used_bins]
    pilot = t.pilot_grid.astype(np.complex128)
    hp = grid[t.pilot_symbols] * pilot.conj() / np.abs(pilot) ** 2
    al = t.interp_alpha.astype(np.float64)[:, None]
    h = hp[t.interp_p0] * (1 - al) + hp[t.interp_p1] * al
    eq = grid[t.data_symbols] * h.conj() / (np.abs(h) ** 2 + nv)
    sig, level = np.maximum(nv / np.abs(h) ** 2, 1e-8), float(t.axis_levels[0])
    want = np.stack([((v + level) ** 2 - (v - level) ** 2) / sig for v in (eq.real, eq.imag)], axis=-1).reshape(-1)
    got, want = llr.cpu().numpy()[0].astype(np.float64), want[:p.coded_bits]
    assert np.sqrt(np.mean((got - want) ** 2) / np.mean(want ** 2)) < 2e-6


# --- OFDM transmitter ------------------------------------------------------------------------------------

@pytest.mark.parametrize("aligned", [True, False])  # information bits away from a 16-byte boundary: the general encoder
@pytest.mark.parametrize("base", [(8, 16, 128), (5, 16, 128), (4, 16, 32), (4, 8, 128)])
def test_transmit_long_information_blocks(cuda, base, aligned):
    """Information blocks of one, two and three passes of 512 bits, the last one full or partial; 4 to 32 parity
    words; bytes whose low bit alone counts."""
    import tx_oracle
    from sicc_gb300.pipeline import RxPipeline
    from test_gpu_tx import _close, _gen, _kw
    torch, code = cuda, codes.qc_code(*base, seed=12)
    cfg = ofdm.PhyConfig(nfft=512, cp=36, num_symbols=9, active_sc=384, pre_half_len=64, modulation="16qam",
                         pilot_period=4)
    t = ofdm.reference_tables(cfg)
    blocks = t.coded_bits // code.n
    p = RxPipeline(t, code.n, code.k, blocks, 1e-3, slots=2)
    G = _gen(code)
    p.upload_tx_tables(generator_kn=G)
    info = np.random.default_rng(3).integers(0, 256, size=(3, blocks * code.k), dtype=np.uint8)
    buf = torch.zeros(info.size + 16, dtype=torch.uint8, device="cuda")
    view = buf[0 if aligned else 3:][:info.size].view(info.shape)
    view.copy_(torch.from_numpy(info))
    assert (view.data_ptr() % 16 == 0) == aligned
    out = torch.zeros((3, t.frame_len), dtype=torch.complex64, device="cuda")
    p.tx_batch(view, 3, out, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    coded = tx_oracle.encode_generator(info.reshape(-1, code.k), G).reshape(3, -1)
    _close(out.cpu().numpy(), tx_oracle.tx_frames(coded, **_kw(t)), base)


# --- mixed-code engine ------------------------------------------------------------------------------------

@pytest.mark.parametrize("how", ["set", "autotune"])
def test_engine_speed_survives_a_shape_given_up(cuda, how):
    """One warp for a 2,048-bit code takes the whole batch off the register-resident rows; afterwards the
    narrow codes, which have no other shape, are as fast as in an engine that never had it."""
    torch = cuda
    tune.clear()
    cs = codes.mixed_codes()
    narrow = [i for i, c in enumerate(cs) if c.n <= 256]
    wide = [i for i, c in enumerate(cs) if c.n == 2048]
    rng = np.random.default_rng(6)
    code_of = np.sort(rng.choice(narrow, 20000)).astype(np.uint8)
    rows = np.concatenate([channel.awgn_llrs(cs[c], int((code_of == c).sum()), 2.0, 9 + c)[2].reshape(-1)
                           for c in sorted(set(code_of.tolist()))]).astype(np.float32)
    ns, ks = (np.array([getattr(cs[c], a) for c in code_of], np.int64) for a in "nk")
    off = lambda v: torch.from_numpy(np.concatenate([[0], np.cumsum(v)[:-1]])).cuda()  # noqa: E731
    d = (torch.from_numpy(code_of).cuda(), torch.from_numpy(rows).cuda(), off(ns))
    io, b = off(ks), len(code_of)

    def make():
        eng = engine.Engine(max_codewords=b, max_llr_floats=rows.size)
        for c in cs:
            eng.add_code(c, engine.iteration_cap(c.n), osd_order=engine.osd_order_for(c))
        return eng

    def decode(eng):
        out = [torch.zeros(int(ks.sum()), dtype=torch.uint8, device="cuda")] + \
              [torch.zeros(b, dtype=torch.uint8, device="cuda") for _ in range(3)]
        eng.decode_device(b, *d, out[0], io, *out[1:], stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in out]

    plain, tried = make(), make()
    want = decode(plain)
    if how == "set":
        for i in wide:
            tried.set_code_warps(i, 1)
        decode(tried)
        for i in wide:
            tried.set_code_warps(i, 4)
    else:
        tried.autotune(b, *d, torch.zeros(int(ks.sum()), dtype=torch.uint8, device="cuda"), io, reps=1)
    for x, y in zip(want, decode(tried)):
        assert np.array_equal(x, y)
    ms = {}
    for _ in range(5):  # in turn; the least of each
        for name, eng in (("plain", plain), ("tried", tried)):
            decode(eng)
            ms[name] = min(ms.get(name, 1e9), eng.last_ms()[1])
    # off the register-resident rows the mixed kernel takes about twice as long
    assert ms["tried"] <= 1.25 * ms["plain"], ms
    tune.clear()


@pytest.mark.parametrize("weight", [33, 255, 256, 300, 512])
def test_long_code_osd_with_a_heavy_column(cuda, oracle, weight):
    """Columns of H of more than 32, and of more than 255, ones."""
    torch, m, k = cuda, 512, 512
    rng = np.random.default_rng(weight)
    rows = []
    for r in range(m):  # accumulator parity, three random information columns, column 0 in the first `weight` rows
        info = set(rng.choice(np.arange(1, k), 3, replace=False).tolist()) | ({0} if r < weight else set())
        rows.append(sorted(info) + ([k + r - 1] if r else []) + [k + r])
    row_ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    code = types.SimpleNamespace(n=m + k, m=m, k=k, row_ptr=row_ptr, col_ind=np.concatenate(rows).astype(np.int32))
    table = oracle.code(code.n, m, code.row_ptr, code.col_ind).systematic_parity()
    cw = np.zeros((6, code.n), np.int64)
    cw[:, :k] = rng.integers(0, 2, (6, k))
    for r in range(m):  # the row's other columns give its own parity bit
        cw[:, k + r] = cw[:, rows[r][:-1]].sum(axis=1) % 2
    llr = (4.0 * (1 - 2 * cw) + 3.0 * rng.standard_normal(cw.shape)).astype(np.float32)
    llr[:4, 0] = 0.01 * (2 * cw[:4, 0] - 1)  # the elimination meets the heavy column first; its bit is wrong
    eng = engine.Engine(max_codewords=6, max_llr_floats=llr.size)
    eng.add_code(code, 10, osd_order=1)
    info = torch.zeros(6 * k, dtype=torch.uint8, device="cuda")
    used, off = torch.zeros(6, dtype=torch.uint8, device="cuda"), torch.arange(6, device="cuda")
    metric = torch.zeros(6, dtype=torch.float32, device="cuda")
    eng.osd_device(6, torch.zeros(6, dtype=torch.uint8, device="cuda"), torch.from_numpy(llr).cuda(), off * code.n, info,
                   off * k, used, metric, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    got, gm = info.cpu().numpy().reshape(6, k), metric.cpu().numpy()
    assert used.cpu().numpy().all()
    for i in range(6):
        out, want, _, _ = oracle.osd(table, code.n, k, llr[i], 1, 64, 4096)
        assert np.array_equal(got[i], out[:k]) and gm[i] == np.float32(want), i


# --- saved shapes -----------------------------------------------------------------------------------------

def test_shapes_saved_for_other_kernels_are_not_applied(cuda, tmp_path):
    """Keys of the first kernels carry no generation; the same shapes under today's keys are applied."""
    import re
    torch, code, wide = cuda, codes.short_code(), codes.qc_code(8, 16, 128, seed=3)
    tune.clear()
    d_llr = torch.from_numpy(channel.awgn_llrs(wide, 64, 2.0, 1)[2].astype(np.float32)).cuda()

    def decoder():
        return fec.CsrBpDecoder.for_code(code, max_batch=64, max_iter=5)

    def eng():
        e = engine.Engine(max_codewords=64, max_llr_floats=64 * wide.n)
        e.add_code(wide, 5)
        return e

    decoder().autotune(torch.from_numpy(channel.awgn_llrs(code, 64, 2.0, 1)[2].astype(np.float32)).cuda(), reps=1)
    off = torch.arange(64, device="cuda")
    eng().autotune(64, torch.zeros(64, dtype=torch.uint8, device="cuda"), d_llr, off * wide.n,
                   torch.zeros(64 * wide.k, dtype=torch.uint8, device="cuda"), off * wide.k, reps=1)
    path = tmp_path / "shapes.txt"
    tune.save(str(path))
    keys = {line.split()[0].split(":")[0]: line.split()[0] for line in path.read_text().splitlines()}
    shapes = {"fec": "8 16 0 0 0", "engine-code": "1"}
    for strip in (True, False):
        tune.clear()
        path.write_text("".join("%s %s\n" % (re.sub(r"/k\d+$", "", k) if strip else k, shapes[kind])
                                for kind, k in keys.items()))
        tune.load(str(path))
        assert tune.entries() == 2
        shape = decoder().shape()
        assert (shape["lanes_per_codeword"], shape["slots_per_cta"]) == ((0, 0) if strip else (8, 16))
        assert eng().code_warps(0) == (4 if strip else 1)
    tune.clear()


# --- launch shapes ----------------------------------------------------------------------------------------

def test_osd_exchange_interval_takes_effect(cuda):
    """The warp OSD's candidate rounds between exchanges of the best metric: the same results at any interval, more
    sums (so more time, about 1.15 of the whole decode) at a long one, and an axis of the tuner's search."""
    torch, code = cuda, codes.short_code()
    llr = torch.from_numpy(channel.awgn_llrs(code, 8192, 1.0, 5)[2].astype(np.float32)).cuda()
    dec = fec.StreamBpOsdDecoder(code, max_batch=8192, max_iter=20, osd_order=3)
    out = [torch.zeros((8192, code.k), dtype=torch.uint8, device="cuda")] + \
          [torch.zeros(8192, dtype=torch.uint8, device="cuda") for _ in range(3)]
    ms, results = {}, {}
    for _ in range(6):
        for share in (0, 3, 64):
            dec.set_shape(osd_share_rounds=share)
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            dec.decode_device_batch(llr, *out, stream=torch.cuda.current_stream())
            ev[1].record()
            torch.cuda.synchronize()
            ms[share] = min(ms.get(share, 1e9), ev[0].elapsed_time(ev[1]))
            results[share] = [x.cpu().numpy() for x in out]
    for share in (3, 64):
        for a, b in zip(results[0], results[share]):
            assert np.array_equal(a, b), share
    assert ms[64] > 1.05 * ms[0], ms
    tune.clear()
    res = dec.autotune(llr, reps=1)
    assert len({shape["osd_share_rounds"] for shape, _ in res.trials}) > 2
    tune.clear()


@pytest.mark.parametrize("base,threads", [((4, 8, 16), 256), ((8, 16, 64), 128), ((8, 16, 128), 128), ((6, 12, 64), 256)])
def test_tuner_times_no_two_equal_shapes(cuda, base, threads):
    """Codewords per CTA beyond what the code's kernel runs are cut to its default: no trials of their own."""
    code = codes.qc_code(*base, seed=8)
    tune.clear()
    dec = fec.CsrBpDecoder.for_code(code, max_batch=512, max_iter=5)
    d_llr = cuda.from_numpy(channel.awgn_llrs(code, 512, 2.0, 3)[2].astype(np.float32)).cuda()
    shapes = [shape for shape, _ in dec.autotune(d_llr, reps=1).trials]
    tune.clear()
    lanes = min(base[2], 128 if threads == 128 else 32)  # of the default; the general kernel has 32 at most
    slots = [s["slots_per_cta"] for s in shapes if s["lanes_per_codeword"] == 0]
    assert all(n * lanes < threads or (base == (6, 12, 64) and n * lanes == threads) for n in slots), slots
    assert len({tuple(sorted(s.items())) for s in shapes}) == len(shapes)
