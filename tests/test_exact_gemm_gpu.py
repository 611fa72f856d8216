"""FP64 contractions as exact digit products on the tensor cores
(csrc/exact_gemm.cu), at the edges of its tiles and of its operand range.

Bar: 1e-14 normwise on uniform inputs.  A product's error is at most ~2^-52
of the product of its rows' maxima, i.e. ~2^-50.5 of a uniform product's rms;
the sums over K are exact and the FP64 epilogue adds a few 2^-53.  Inputs
outside the split's range take the FP64 kernel, whose sums of K ~ 5000 terms
in 16-wide chunks stay within 1e-12 of max|schDt|.
"""
import numpy as np
import pytest

import workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _norm(g, o):
    return np.linalg.norm(g - o) / np.linalg.norm(o)


@pytest.mark.parametrize("case", [
    # number_bands, ncouls, ngpown, nfreq: band blocks of 40, row blocks of 128, K tiles of 32, blocks of 128
    (1, 32768, 128, 1), (39, 4099, 127, 1), (40, 4096, 64, 2), (41, 4097, 43, 3), (80, 2015, 129, 1),
    (81, 1985, 10, 26), (3, 20011, 71, 1), (200, 129, 129, 5), (513, 512, 20, 3),
], ids=lambda c: "x".join(map(str, c)))
def test_exact_contraction_edges(sigma_lib, case):
    p = W.ff_random(*case, seed=31 + case[0])
    assert case[0] * case[1] * case[2] * case[3] >= 1 << 22
    o = O.ff_schdt(p).reshape(p.number_bands, p.nfreq)
    assert _norm(sigma_lib.ff_host(p, sigma_lib.FF_MODE_FP64), o) <= 1e-14


@pytest.mark.parametrize("kind", ["coherent", "decaying", "scaled_rows", "zero_rows"])
def test_exact_contraction_value_ranges(sigma_lib, kind):
    p = W.ff_random(45, 5003, 67, 2, seed=7)
    k = np.arange(p.ncouls)
    if kind == "coherent":        # every digit sum at its largest: all elements alike, no zero digits
        p.I_epsR[:] = 0.7 + 0.9j / 1.1
        p.aqsntemp[:] = 1 / 3 - 0.8j / 1.3
    elif kind == "decaying":      # both operands fall off over 2^-20
        p.I_epsR *= 2.0 ** (-20.0 * k / p.ncouls)
        p.aqsntemp *= 2.0 ** (-20.0 * k / p.ncouls)
    elif kind == "scaled_rows":   # rows of very different size
        p.I_epsR *= (10.0 ** np.linspace(-30, 30, p.ngpown))[None, :, None]
        p.aqsntemp *= (10.0 ** np.linspace(40, -40, p.number_bands))[:, None]
    else:
        p.I_epsR[0, 5] = 0
        p.aqsntemp[7] = 0
    o = O.ff_schdt(p).reshape(p.number_bands, p.nfreq)
    g = sigma_lib.ff_host(p, sigma_lib.FF_MODE_FP64)
    if kind == "scaled_rows":
        assert max(_norm(g[n], o[n]) for n in range(p.number_bands)) <= 1e-14
    else:
        assert _norm(g, o) <= 1e-14
    if kind == "zero_rows":
        assert np.all(g[7] == 0)


@pytest.mark.parametrize("kind", ["outlier", "opposed", "huge", "nan"])
def test_out_of_range_operands_take_the_fp64_kernel(sigma_lib, kind):
    p = W.ff_random(45, 5003, 67, 2, seed=8)
    half = p.ncouls // 2
    if kind == "outlier":         # one element 2^40 above its row
        p.I_epsR[1, 3, 17] *= 2.0 ** 40
        p.aqsntemp[4, 17] = 0.0
    elif kind == "opposed":       # large elements never meet
        p.I_epsR[:, :, :half] *= 1e-9
        p.aqsntemp[:, half:] *= 1e-9
    elif kind == "huge":
        p.I_epsR *= 1e150
    else:
        p.I_epsR[0, 11, 100] = np.nan
    g = sigma_lib.ff_host(p, sigma_lib.FF_MODE_FP64)
    if kind == "nan":
        assert np.all(np.isnan(g[:, 0].real)) and np.all(np.isfinite(g[:, 1]))
        return
    o = O.ff_schdt(p).reshape(p.number_bands, p.nfreq)
    assert np.abs(g - o).max(axis=0).max() / np.abs(o).max() <= 1e-12
    assert np.linalg.norm(g[:, 0] - o[:, 0]) / np.linalg.norm(o[:, 0]) <= 1e-12


# GPP band sums (csrc/gpp_exact.cu).  Bars as the FP64 parity tests: 1e-12 per
# achtemp / asxtemp output, 1e-12 of the largest band value.
@pytest.mark.parametrize("case", [
    # number_bands, nvband, ncouls, ngpown, stress: 16-column tiles, 64- and 512-g-vector segments, padding rows
    (40, 1, 4096, 64, False), (39, 2, 1985, 43, True), (41, 0, 513, 129, False), (100, 3, 511, 85, False),
    (1, 1, 32767, 43, False), (81, 8, 2049, 17, True), (300, 2, 4000, 3, False), (512, 0, 63, 63, False),
    (24, 2, 4097, 33, False), (25, 3, 4095, 31, False), (32, 0, 4100, 31, True), (64, 5, 1991, 40, False),
    (128, 2, 1023, 41, True),
], ids=lambda c: "x".join(map(str, c[:4])) + ("s" if c[4] else ""))
def test_gpp_band_sums_edges(sigma_lib, case):
    nb, nvb, nc, ng, stress = case
    assert 3 * nb * nc * ng >= 1 << 22
    p = W.gpp_random(nb, nvb, nc, ng, 90 + nb, stress=stress)
    p.vcoul = np.abs(p.vcoul)
    o, g = O.gpp(p), sigma_lib.gpp_host(p, sigma_lib.PREC_FP64)
    assert np.all(np.abs(g[0] - o[0]) <= 1e-12 * np.abs(o[0]))
    assert np.all(np.abs(g[1] - o[1]) <= 1e-12 * np.abs(o[1]))
    assert np.abs(g[2] - o[2]).max() <= 1e-12 * np.abs(o[2]).max()


@pytest.mark.parametrize("kind", ["outlier_wtilde", "outlier_aqsn", "huge_wtilde", "all_dropped", "tiny"])
def test_gpp_band_sums_out_of_range(sigma_lib, kind):
    p = W.gpp_random(45, 2, 3001, 37, 5)
    if kind == "outlier_wtilde":
        p.wtilde_array[3, 100] = complex(2.0 ** 50, 1.0)
        p.I_eps_array[3, 100] = 2.0 ** 45
    elif kind == "outlier_aqsn":
        p.aqsntemp[7, 11] *= 2.0 ** 30
    elif kind == "huge_wtilde":
        p.wtilde_array[:] *= 1e25
    elif kind == "all_dropped":     # one column's terms all inside the guard
        p.wtilde_array[5, :] = 4.0 + 0.1j
    else:
        p.I_eps_array[:] *= 1e-60
    o, g = O.gpp(p), sigma_lib.gpp_host(p, sigma_lib.PREC_FP64)
    assert np.all(np.abs(g[0] - o[0]) <= 1e-12 * np.abs(o[0]))
    assert np.abs(g[2] - o[2]).max() <= 1e-12 * np.abs(o[2]).max()


# Real-valued sums: 80 bands per block, and the half sum: seven digits, 32
# bands per block over aqsn's and aqsm's bands, rows that end at their igp.
@pytest.mark.parametrize("case", [
    (80, 2, 4096, 43), (81, 1, 2017, 128), (159, 0, 513, 87), (5, 5, 16384, 63),
], ids=lambda c: "x".join(map(str, c)))
def test_real_band_sums_edges(sigma_lib, case):
    assert 3 * case[0] * case[2] * case[3] >= 1 << 22
    p = W.gpp_real_random(*case, seed=200 + case[0])
    o, g = O.gpp_real(p), sigma_lib.gpp_real_host(p)
    assert np.all(np.abs(g[0] - o[0]) <= 1e-12 * np.abs(o[0]))
    assert np.all(np.abs(g[1] - o[1]) <= 1e-12 * np.abs(o[1]).max())
    assert np.abs(g[2] - o[2]).max() <= 1e-12 * np.abs(o[2]).max()


@pytest.mark.parametrize("case", [
    (64, 2, 2048, 32, False), (31, 0, 4100, 96, True), (33, 3, 1025, 97, False), (129, 1, 3000, 43, True),
    (16, 16, 5121, 65, False),
], ids=lambda c: "x".join(map(str, c[:4])) + ("s" if c[4] else ""))
@pytest.mark.parametrize("static", [True, False], ids=["static", "nostatic"])
def test_halfsum_edges(sigma_lib, case, static):
    nb, nvb, nc, ng, stress = case
    assert 3 * nb * nc * ng >= 1 << 22
    p = W.gpp_random(nb, nvb, nc, ng, 300 + nb, stress=stress)
    o, g = O.gpp_halfsum(p), sigma_lib.gpp_halfsum_host(p, want_static=static)
    assert np.all(np.abs(g[0] - o[0]) <= 1e-12 * np.abs(o[0]))
    assert np.all(np.abs(g[1] - o[1]) <= 1e-12 * np.abs(o[1]))
    assert np.abs(g[2] - o[2]).max() <= 1e-12 * np.abs(o[2]).max()
    if static:
        assert abs(g[3] - o[3]) <= 1e-12 * abs(o[3])


def test_batch_mixes_exact_flagged_and_small_instances(sigma_lib):
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.float64).copy()).cuda()
    probs = [W.gpp_random(60, 2, 2048, 50, 1), W.gpp_random(9, 1, 300, 20, 2), W.gpp_random(70, 3, 3001, 33, 3)]
    probs[2].aqsntemp[3, 5] *= 2.0 ** 35   # outside the split's range
    outs, inst = [], []
    for p in probs:
        o = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in (6, 6, 2 * p.number_bands)]
        outs.append(o)
        inst.append(dict(number_bands=p.number_bands, nvband=p.nvband, ncouls=p.ncouls, ngpown=p.ngpown,
                         inv_igp_index=p.inv_igp_index, indinv=p.indinv, wx_array=dev(p.wx_array),
                         aqsmtemp=dev(p.aqsmtemp), aqsntemp=dev(p.aqsntemp), I_eps_array=dev(p.I_eps_array),
                         wtilde_array=dev(p.wtilde_array), vcoul=dev(p.vcoul), achtemp=o[0], asxtemp=o[1],
                         acht_n1_loc=o[2]))
    for k in ([0, 1, 2], [0], [0, 2]):   # with and without an instance that always takes the queue
        for o in outs:
            for t in o:
                t.zero_()
        b = sigma_lib.GppBatch([inst[i] for i in k], sigma_lib.PREC_FP64)
        b.execute()
        torch.cuda.synchronize()
        assert b.status() == 0
        b.close()
        for i in k:
            ref = O.gpp(probs[i])
            got = [t.cpu().numpy().view(np.complex128) for t in outs[i]]
            for x, y in zip(got, ref):
                assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()
