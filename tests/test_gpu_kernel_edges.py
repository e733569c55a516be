"""The kernels' size classes at their edges, against the oracle.

Row degrees and lengths around the compiled shapes of the long-code BP kernels, code sizes around the
classes of the two OSD kernels with every order and truncated test lists, soft values with ties,
zeros of both signs, subnormals, infinities and sums that overflow; FFT sizes from 16 points, every
modulation, preambles that are no multiple of a block, one to a few frames; generators that are and
are not systematic.  Bits, flags, counts and metrics are compared exactly, posteriors by value; LLRs and
samples within the bounds of the receive- and transmit-chain tests.
"""
import numpy as np
import pytest

import tx_oracle
from sicc_gb300 import channel, codes, engine, ofdm

pytestmark = pytest.mark.gpu

ODD = [0.0, -0.0, 1e-40, -1e-40, np.inf, -np.inf, 3e38, -3e38]


def _soft(code, count, ebn0, seed):
    """Noisy frames: plain, quantised (ties), with a few odd values, all equal magnitudes."""
    llr = channel.awgn_llrs(code, count, ebn0, seed)[2].astype(np.float32)
    rng = np.random.default_rng(seed)
    for f in range(count):
        if f % 4 == 1:
            llr[f] = np.round(2.0 * llr[f]) / 2.0
        elif f % 4 == 2:
            llr[f, rng.choice(code.n, 9, replace=False)] = rng.choice(ODD, 9)
        elif f % 4 == 3 and f > 4:
            llr[f] = np.copysign(np.float32(1.25), llr[f])
    return llr


# --- long-code BP -----------------------------------------------------------------------------------

# (n, k, groups): information-column degrees; row degree = edges / m + 2 at most
LONG = [
    (16200, 3240, [(4, 12), (5, 3)]),      # 4 slots, posteriors in shared memory
    (16200, 7920, [(22, 4)]),              # 6
    (32400, 16200, [(25, 5), (20, 4)]),    # 7
    (32400, 21600, [(20, 5), (40, 3)]),    # 10
    (16200, 11880, [(33, 4)]),             # 14
    (16200, 13320, [(1, 13), (36, 3)]),    # 18
    (16200, 14400, [(40, 3)]),             # 27
    (64800, 16200, [(45, 6)]),             # 4 slots, the last two beyond shared memory
    (64800, 32400, [(36, 8), (54, 3)]),    # 7
    (64800, 57600, [(160, 3)]),            # 27, information columns beyond as well
]


def _long(i):
    n, k, prof = LONG[i]
    prof = [p for p in prof if p[0]]
    have, need = sum(c for c, _ in prof), k // 360
    if have < need:
        prof.append((need - have, 2))
    return codes.ira_code(n, k, prof, seed=77 + i)


def _run_csr(torch, dec, llr, n):
    b = llr.shape[0]
    d = {"bits": torch.zeros((b, n), dtype=torch.uint8, device="cuda"),
         "ok": torch.zeros(b, dtype=torch.uint8, device="cuda"), "it": torch.zeros(b, dtype=torch.uint8, device="cuda"),
         "app": torch.zeros((b, n), dtype=torch.float32, device="cuda")}
    dec.decode_device_batch(torch.from_numpy(np.ascontiguousarray(llr)).cuda(), d["bits"], d["ok"], d["app"], d["it"],
                            stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in d.items()}


def _same(g, i, o):
    assert g["ok"][i] == o[0] and g["it"][i] == o[4], i
    assert np.array_equal(g["bits"][i], o[1]), i
    assert np.array_equal(g["app"][i], o[2], equal_nan=True), i


@pytest.mark.parametrize("beta", [0.0, 0.15])
@pytest.mark.parametrize("which", range(len(LONG)))
def test_long_layered(cuda, oracle, which, beta):
    from sicc_gb300 import fec
    code = _long(which)
    oc = oracle.code(code.n, code.m, code.row_ptr, code.col_ind)
    order, _, _ = oc.color_order()
    llr = _soft(code, 3, np.array([4.0, 2.0, 6.0]), which)
    dec = fec.CsrBpDecoder(code.n, code.m, code.row_ptr, code.col_ind, max_batch=3, max_iter=5, normalization=0.75,
                           offset=beta, schedule=fec.COLORED_LAYERED)
    g = _run_csr(cuda, dec, llr, code.n)
    for i, x in enumerate(llr):
        _same(g, i, oc.layered(x, 5, 0.75, beta, row_order=order))


@pytest.mark.parametrize("damping", [0.0, 0.2])
@pytest.mark.parametrize("which", [0, 1, 3, 5, 6, 8])
def test_long_flooding(cuda, oracle, which, damping):
    from sicc_gb300 import fec
    code = _long(which)
    oc = oracle.code(code.n, code.m, code.row_ptr, code.col_ind)
    llr = _soft(code, 3, np.array([4.0, 2.0, 6.0]), 20 + which)
    dec = fec.CsrBpDecoder(code.n, code.m, code.row_ptr, code.col_ind, max_batch=3, max_iter=5, normalization=0.8,
                           offset=0.1, damping=damping, schedule=fec.FLOODING)
    g = _run_csr(cuda, dec, llr, code.n)
    for i, x in enumerate(llr):
        _same(g, i, oc.flooding(x, 5, 0.8, 0.1, damping))


# --- OSD --------------------------------------------------------------------------------------------

TESTS = [(0, 64, 4096), (1, 64, 4096), (2, 64, 4096), (3, 24, 4096), (3, 64, 777), (2, 5, 1), (1, 1, 4096)]


@pytest.mark.parametrize("base", [(4, 8, 8), (4, 8, 9), (4, 8, 12), (4, 12, 16), (8, 16, 16), (6, 8, 16)])
def test_short_code_osd(cuda, oracle, base):
    from sicc_gb300 import _lib, fec
    torch = cuda
    code = codes.qc_code(*base, seed=5)
    oc = oracle.code(code.n, code.m, code.row_ptr, code.col_ind)
    table = oc.systematic_parity()
    llr = _soft(code, 13, 2.0, 3)
    dec = fec.StreamBpOsdDecoder(code, max_batch=64, max_iter=5)
    d_llr = torch.from_numpy(llr).cuda()
    info = torch.zeros((13, code.k), dtype=torch.uint8, device="cuda")
    cw = torch.zeros((13, code.n), dtype=torch.uint8, device="cuda")
    dist = torch.zeros(13, dtype=torch.float32, device="cuda")
    for order, flips, tests in TESTS:
        dec.set_osd_params(order, min(flips, code.k), tests)
        _lib.check(_lib.load().sicc_osd_decode_device(dec.handle, d_llr.data_ptr(), 13, info.data_ptr(), cw.data_ptr(),
                                                      dist.data_ptr(), None), "osd")
        torch.cuda.synchronize()
        g, dd = cw.cpu().numpy(), dist.cpu().numpy()
        for i, x in enumerate(llr):
            out, metric, _, _ = oracle.osd(table, code.n, code.k, x, order, min(flips, code.k), tests)
            assert np.array_equal(g[i], out), (order, flips, tests, i)
            assert np.float32(metric) == dd[i], (order, flips, tests, i)


# m at the edges of the size classes (256, 512, 640, 1024) and odd sizes; few and many columns left over
LARGE = [(4, 16, 64), (4, 18, 66), (8, 12, 64), (8, 16, 65), (8, 16, 80), (8, 12, 81), (8, 16, 128), (8, 16, 98), (5, 16, 37)]


@pytest.mark.parametrize("order,flips,tests", [t for t in TESTS if t != (3, 64, 777)])
def test_long_code_osd(cuda, oracle, order, flips, tests):
    torch = cuda
    cs = [codes.qc_code(*b, seed=9) for b in LARGE]
    eng = engine.Engine(max_codewords=64, max_llr_floats=64 * 2048)
    for c in cs:
        eng.add_code(c, 10, osd_order=order, osd_max_flip=flips, osd_max_tests=tests)
    rows, ids = [], []
    for ci, c in enumerate(cs):
        for x in _soft(c, 4, 1.5, 50 + ci):
            rows.append(x)
            ids.append(ci)
    ks = [cs[i].k for i in ids]
    lo = np.concatenate([[0], np.cumsum([r.size for r in rows])[:-1]]).astype(np.int64)
    io = np.concatenate([[0], np.cumsum(ks)[:-1]]).astype(np.int64)
    info = torch.zeros(int(np.sum(ks)), dtype=torch.uint8, device="cuda")
    used = torch.zeros(len(rows), dtype=torch.uint8, device="cuda")
    metric = torch.zeros(len(rows), dtype=torch.float32, device="cuda")
    eng.osd_device(len(rows), torch.from_numpy(np.asarray(ids, np.uint8)).cuda(),
                   torch.from_numpy(np.concatenate(rows)).cuda(), torch.from_numpy(lo).cuda(), info,
                   torch.from_numpy(io).cuda(), used, metric, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    got, gm = info.cpu().numpy(), metric.cpu().numpy()
    assert np.all(used.cpu().numpy() == 1)
    tables = {}
    for i, (ci, x) in enumerate(zip(ids, rows)):
        c = cs[ci]
        if ci not in tables:
            tables[ci] = oracle.code(c.n, c.m, c.row_ptr, c.col_ind).systematic_parity()
        out, m, _, _ = oracle.osd(tables[ci], c.n, c.k, x, order, flips, tests)
        assert np.array_equal(got[io[i]:io[i] + c.k], out[: c.k]), (LARGE[ci], i)
        assert gm[i] == np.float32(m), (LARGE[ci], i)


# --- OFDM -------------------------------------------------------------------------------------------

PHYS = [(16, 8, "16qam", 64), (32, 16, "64qam", 33), (64, 32, "qpsk", 100), (128, 64, "bpsk", 257), (512, 384, "64qam", 63),
        (2048, 1024, "16qam", 128), (4096, 2000, "qpsk", 200)]


def _tables(nfft, active, modulation, half):
    return ofdm.reference_tables(ofdm.PhyConfig(nfft=nfft, cp=nfft // 8, num_symbols=6, active_sc=active, pilot_period=3,
                                                pre_half_len=half, modulation=modulation))


@pytest.mark.parametrize("frames", [1, 2, 5])
@pytest.mark.parametrize("phy", PHYS)
def test_search_and_demodulate(cuda, oracle, phy, frames):
    from sicc_gb300.pipeline import SYNC_RECORD, RxPipeline
    from test_gpu_ofdm import _llr_close
    torch = cuda
    t, code = _tables(*phy), codes.short_code()
    b = ofdm.FrameGenerator(t, code, seed=17).batch(frames, snr_db=25.0, cfo_subcarriers=0.05, max_offset=77,
                                                    rayleigh_taps=0)
    p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, float(b.noise_var[0]), max_batch_frames=frames)
    llr = torch.zeros((frames, p.coded_bits), dtype=torch.float32, device="cuda")
    rec = torch.zeros(frames * SYNC_RECORD.itemsize, dtype=torch.uint8, device="cuda")
    p.demod_batch(torch.from_numpy(b.iq).cuda(), b.iq.shape[1], b.iq.shape[1], frames, llr, rec,
                  torch.cuda.current_stream())
    torch.cuda.synchronize()
    sync, got, ph = rec.cpu().numpy().view(SYNC_RECORD), llr.cpu().numpy(), oracle.phy(t)
    for f in range(frames):
        r = oracle.sync_earliest(ph, b.iq[f])
        assert sync[f]["found"] == r[0]
        if r[0] != 1:
            continue
        assert sync[f]["start"] == r[1]
        ref = oracle.demod_frame(ph, b.iq[f][r[1]:r[1] + t.frame_len], float(sync[f]["cfo_hz"]),
                                 float(np.float32(b.noise_var[0])))
        _llr_close(got[f], ref[: p.coded_bits])


@pytest.mark.parametrize("systematic", [True, False])
@pytest.mark.parametrize("phy", PHYS)
def test_transmit(cuda, phy, systematic):
    from sicc_gb300.pipeline import RxPipeline
    from test_gpu_tx import _close, _gen, _kw
    torch = cuda
    t, code = _tables(*phy), codes.short_code()
    blocks = t.coded_bits // code.n
    p = RxPipeline(t, code.n, code.k, blocks, 1e-3, slots=2)
    G = _gen(code)
    if not systematic:  # one bit off the identity: the general encoder
        G[3, 7] = 1
    p.upload_tx_tables(generator_kn=G)
    info = np.random.default_rng(8).integers(0, 2, size=(3, blocks * code.k), dtype=np.uint8)
    out = torch.zeros((3, t.frame_len), dtype=torch.complex64, device="cuda")
    p.tx_batch(torch.from_numpy(info).cuda(), 3, out, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    coded = tx_oracle.encode_generator(info.reshape(-1, code.k), G).reshape(3, -1)
    _close(out.cpu().numpy(), tx_oracle.tx_frames(coded, **_kw(t)), phy)


# --- mixed batches ----------------------------------------------------------------------------------

MIXED = [(4, 8, 9), (5, 16, 17), (3, 6, 20), (8, 16, 65), (8, 16, 128), (4, 8, 8), (4, 16, 32), (4, 18, 40), (5, 16, 64)]


@pytest.mark.parametrize("more", [[], [(8, 16, 256)]], ids=["small", "large"])
def test_mixed_shapes(cuda, oracle, more):
    """Codes of the register-resident and the general row arithmetic, and (large) a code whose posteriors
    take the whole batch to the general one; unaligned soft values."""
    torch = cuda
    cs = [codes.qc_code(*b, seed=13) for b in MIXED + more]
    eng = engine.Engine(max_codewords=256, max_llr_floats=1 << 18)
    for c in cs:
        eng.add_code(c, 8, alpha=0.8, beta=0.1)
    ids, rows = [], []
    for ci, c in enumerate(cs):
        for x in _soft(c, 7, 2.5, 80 + ci):
            ids.append(ci)
            rows.append(x)
    perm = np.random.default_rng(4).permutation(len(ids))
    ids, rows = [ids[i] for i in perm], [rows[i] for i in perm]
    lo, io, at, bits = [], [], 1, 0
    for ci, x in zip(ids, rows):
        lo.append(at)
        io.append(bits)
        at += x.size + 1
        bits += cs[ci].k
    llr = np.zeros(at, np.float32)
    for o, x in zip(lo, rows):
        llr[o:o + x.size] = x
    info = torch.zeros(bits, dtype=torch.uint8, device="cuda")
    ok, used, it = (torch.zeros(len(ids), dtype=torch.uint8, device="cuda") for _ in range(3))
    eng.decode_device(len(ids), torch.from_numpy(np.asarray(ids, np.uint8)).cuda(), torch.from_numpy(llr).cuda(),
                      torch.tensor(lo, dtype=torch.int64, device="cuda"), info,
                      torch.tensor(io, dtype=torch.int64, device="cuda"), ok, used, it,
                      stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    got, gok, git = info.cpu().numpy(), ok.cpu().numpy(), it.cpu().numpy()
    ocs = [oracle.code(c.n, c.m, c.row_ptr, c.col_ind) for c in cs]
    for i, (ci, x) in enumerate(zip(ids, rows)):
        o = ocs[ci].layered(x, 8, 0.8, 0.1)
        assert gok[i] == o[0] and git[i] == o[4], (ci, i)
        assert np.array_equal(got[io[i]:io[i] + cs[ci].k], o[1][: cs[ci].k]), (ci, i)


@pytest.mark.parametrize("threshold", [0.02, 0.2, 0.7, 0.93])
def test_search_thresholds(cuda, oracle, threshold):
    """Early stop of the fine metric: low and high thresholds, bursts of strong samples around the frame."""
    from sicc_gb300.pipeline import SYNC_RECORD, RxPipeline
    torch = cuda
    t, code = ofdm.reference_tables(ofdm.PhyConfig(nfft=64, cp=8, num_symbols=6, active_sc=32, pilot_period=3, pre_half_len=97,
                                                   modulation="qpsk", sync_threshold=threshold)), codes.short_code()
    b = ofdm.FrameGenerator(t, code, seed=23).batch(12, snr_db=20.0, cfo_subcarriers=0.05, max_offset=400, rayleigh_taps=0)
    rng = np.random.default_rng(5)
    for f in range(0, 12, 3):
        at = rng.integers(0, b.iq.shape[1], 20)
        b.iq[f, at] *= np.float32(50.0)
    p = RxPipeline(t, code.n, code.k, t.coded_bits // code.n, float(b.noise_var[0]), max_batch_frames=12)
    llr = torch.zeros((12, p.coded_bits), dtype=torch.float32, device="cuda")
    rec = torch.zeros(12 * SYNC_RECORD.itemsize, dtype=torch.uint8, device="cuda")
    p.demod_batch(torch.from_numpy(b.iq).cuda(), b.iq.shape[1], b.iq.shape[1], 12, llr, rec, torch.cuda.current_stream())
    torch.cuda.synchronize()
    sync, ph = rec.cpu().numpy().view(SYNC_RECORD), oracle.phy(t)
    for f in range(12):
        r = oracle.sync_earliest(ph, b.iq[f])
        assert sync[f]["found"] == r[0], f
        if r[0]:
            assert sync[f]["start"] == r[1], f
