"""Register-resident BP kernels against the oracle, bit for bit.

Codes at the edges of the compiled shapes (rows per lane, row degree, lanes per codeword 8..128, one to
four warps), ragged ones (layers narrower than their lanes, several rows of a layer per lane, n not a
multiple of 4), and frames with zeros of both signs, infinities, NaN and subnormal values among the
ordinary ones.  Posteriors are compared by value (a zero's sign and a NaN's payload carry nothing).
"""
import numpy as np
import pytest

from sicc_gb300 import channel, codes

pytestmark = pytest.mark.gpu

# (base rows, base columns, lift): layers of `lift` rows of degree columns - rows + 1 or + 2
PLAIN = [(4, 8, 16), (4, 8, 64), (4, 8, 128), (8, 16, 8), (8, 16, 32), (8, 16, 64), (8, 16, 128), (5, 16, 16), (5, 16, 64),
         (5, 16, 128), (4, 16, 32), (4, 16, 128), (4, 9, 64)]
RAGGED = [(4, 8, 9), (4, 8, 33), (5, 16, 17), (8, 16, 5), (3, 6, 20)]


def _frames(code, count, seed):
    _, _, llr = channel.awgn_llrs(code, count, np.linspace(1.0, 4.0, count), seed)
    rng = np.random.default_rng(seed)
    odd = [0.0, -0.0, np.inf, -np.inf, 1e-40, -1e-40, 3e38, -3e38, np.nan]
    for f in range(0, count, 2):  # every other frame holds special values, one NaN frame in eight
        at = rng.choice(code.n, 12, replace=False)
        llr[f, at] = rng.choice(odd if f % 8 == 0 else odd[:-1], 12)
    llr[1] = np.round(llr[1])  # ties
    return llr


def _check(torch, dec, llr, code, expect):
    b = llr.shape[0]
    d = {"bits": torch.zeros((b, code.n), dtype=torch.uint8, device="cuda"),
         "ok": torch.zeros(b, dtype=torch.uint8, device="cuda"), "it": torch.zeros(b, dtype=torch.uint8, device="cuda"),
         "app": torch.zeros((b, code.n), dtype=torch.float32, device="cuda")}
    dec.decode_device_batch(torch.from_numpy(llr).cuda(), d["bits"], d["ok"], d["app"], d["it"],
                            stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    g = {k: v.cpu().numpy() for k, v in d.items()}
    for i, x in enumerate(llr):
        o = expect(x)
        assert g["ok"][i] == o[0] and g["it"][i] == o[4], i
        assert np.array_equal(g["bits"][i], o[1]), i
        assert np.array_equal(g["app"][i], o[2], equal_nan=True), i


@pytest.mark.parametrize("beta", [0.0, 0.15])
@pytest.mark.parametrize("base", PLAIN + RAGGED)
def test_layered_register_kernel(cuda, oracle, base, beta):
    from sicc_gb300 import fec
    code = codes.qc_code(*base, seed=31)
    oc = oracle.code(code.n, code.m, code.row_ptr, code.col_ind)
    llr = _frames(code, 33, 7)
    dec = fec.CsrBpDecoder.for_code(code, max_batch=33, max_iter=12, normalization=0.8, offset=beta,
                                    schedule=fec.FLAT_LAYERED)
    _check(cuda, dec, llr, code, lambda x: oc.layered(x, 12, 0.8, beta))


@pytest.mark.parametrize("damping", [0.0, 0.15, 0.9])
@pytest.mark.parametrize("base", PLAIN)
def test_flooding_register_kernel(cuda, oracle, base, damping):
    from sicc_gb300 import fec
    code = codes.qc_code(*base, seed=32)
    oc = oracle.code(code.n, code.m, code.row_ptr, code.col_ind)
    llr = _frames(code, 33, 8)
    dec = fec.CsrBpDecoder.for_code(code, max_batch=33, max_iter=12, normalization=0.8, offset=0.15, damping=damping,
                                    schedule=fec.NODE_PARALLEL)
    _check(cuda, dec, llr, code, lambda x: oc.flooding(x, 12, 0.8, 0.15, damping))


@pytest.mark.parametrize("schedule", [0, 3])
@pytest.mark.parametrize("base", [(4, 8, 16), (8, 16, 128)])
def test_smallest_posterior_rule(cuda, oracle, base, schedule):
    """A zero syndrome is not accepted when a posterior is below min_abs_llr_accept (group minimum)."""
    from sicc_gb300 import fec
    code = codes.qc_code(*base, seed=33)
    oc = oracle.code(code.n, code.m, code.row_ptr, code.col_ind)
    _, _, llr = channel.awgn_llrs(code, 64, 3.5, 9)
    dec = fec.CsrBpDecoder.for_code(code, max_batch=64, max_iter=20, normalization=0.8, min_abs_llr_accept=1.5,
                                    schedule=schedule)
    f = oc.layered if schedule == 3 else oc.flooding
    want = [(o[0] and np.abs(o[2]).min() >= 1.5, o[1], o[2], o[3], o[4]) for o in (f(x, 20, 0.8) for x in llr)]
    assert 0 < sum(w[0] for w in want) < 64
    it = iter(want)
    _check(cuda, dec, llr, code, lambda x: next(it))
