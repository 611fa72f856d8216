"""The exact contractions (csrc/exact_gemm.cu, csrc/gpp_exact.cu) on operands at
the edges of what they accept: an operand that they cannot hold has to reach
the FP64 kernels behind them, whatever its neighbours.

Bars as the FP64 parity tests: 1e-12 per achtemp / asxtemp / achstemp output
and 1e-12 of the largest band value, against the oracle.
"""
import numpy as np
import pytest

import workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _close(g, o):
    g, o = np.atleast_1d(g), np.atleast_1d(o)
    assert np.all(np.abs(g - o) <= TOL * np.abs(o)), np.abs(g - o) / np.abs(o)


def _half_close(g, o):
    _close(g[0], o[0])
    _close(g[1], o[1])
    assert np.abs(g[2] - o[2]).max() <= TOL * np.abs(o[2]).max()
    if g[3] is not None:
        _close(g[3], o[3])


# ---- half sum: a factor far above its row's others meets a zero band element
@pytest.mark.parametrize("p", [30, 40])
def test_halfsum_large_factor_meets_zero_band_element(sigma_lib, p):
    prob = W.gpp_random(64, 0, 4096, 16, 400 + p)
    assert 3 * 64 * 16 * 4096 >= 1 << 23
    for g in range(prob.ngpown):
        k = 600 + 3 * g  # below every later igp
        prob.wtilde_array[g, k] = prob.wx_array[g % 3] + 2.0 ** -p
        prob.aqsntemp[:, k] = 0
        prob.aqsmtemp[:, k] = 0
    _half_close(sigma_lib.gpp_halfsum_host(prob, want_static=False), O.gpp_halfsum(prob))


# ---- half sum, occupied bands: rows shorter than 512 g-vectors
def _short_rows(scale, seed=41):
    prob = W.gpp_random(8, 3, 4096, 128, seed)
    assert 3 * 8 * 128 * 4096 >= 1 << 23
    prob.inv_igp_index = (3 * np.arange(128) + 4).astype(np.int32)          # igp <= 385
    prob.wtilde_array.real[:] = 0.5 + (prob.wtilde_array.real - 0.5) * (1.5 / 4.5)  # none within 0.5 of a frequency
    prob.aqsntemp[:, 512:] *= scale
    prob.aqsmtemp[:, 512:] *= scale
    return prob


@pytest.mark.parametrize("p", [0, 20, 30, 40])
def test_halfsum_occupied_short_rows(sigma_lib, p):
    prob = _short_rows(2.0 ** p)
    g, o = sigma_lib.gpp_halfsum_host(prob, want_static=False), O.gpp_halfsum(prob)
    _close(g[1], o[1])
    assert np.abs(g[2] - o[2]).max() <= TOL * np.abs(o[2]).max()


# ---- half sum: no g-vector below any igp (no work for the contractions)
@pytest.mark.parametrize("static", [True, False], ids=["static", "nostatic"])
@pytest.mark.parametrize("igps", [[0], [1], [0, 1, -1], [-1, -1]], ids=str)
@pytest.mark.parametrize("nvb", [0, 2])
def test_halfsum_without_pairs(sigma_lib, igps, nvb, static):
    ng = len(igps)
    prob = W.gpp_random(512, nvb, 8192, ng, 43)
    assert 3 * 512 * ng * 8192 >= 1 << 23
    prob.inv_igp_index = np.arange(ng, dtype=np.int32)
    prob.indinv = np.arange(8192, dtype=np.int32)
    prob.indinv[:ng] = igps
    g, o = sigma_lib.gpp_halfsum_host(prob, want_static=static), O.gpp_halfsum(prob)
    scale = max(np.abs(o[0]).max(), 1e-300)
    assert np.abs(g[0] - o[0]).max() <= TOL * scale
    assert np.abs(g[1] - o[1]).max() <= TOL * max(np.abs(o[1]).max(), 1e-300)
    assert np.abs(g[2] - o[2]).max() <= TOL * max(np.abs(o[2]).max(), 1e-300)
    if static:
        assert abs(g[3] - o[3]) <= TOL * max(abs(o[3]), 1e-300)


# ---- sums over more g-vectors than the 64-bit integer sums hold
def test_ff_long_coherent_sum(sigma_lib):
    nc, x = 1 << 22, 0.96
    z = np.full((1, nc), complex(x, x))
    prob = W.FFProblem(1, nc, 1, 1, np.zeros(1, np.int32), np.arange(nc, dtype=np.int32), z.reshape(1, 1, nc),
                       np.conj(z), np.ones((1, nc), np.complex128))
    _close(sigma_lib.ff_host(prob, sigma_lib.FF_MODE_FP64), 2 * x * x * nc)


def test_gpp_long_coherent_sum(sigma_lib):
    nc = 1 << 23
    one = np.ones((1, nc), np.complex128)
    prob = W.GppProblem(1, 1, nc, 1, np.zeros(1, np.int32), np.arange(nc, dtype=np.int32), W.wx_frequencies(),
                        one, one * (0.96 - 0.96j), one * (0.96 + 0.96j), one * 1.5, np.ones(nc))
    g, o = sigma_lib.gpp_host(prob, sigma_lib.PREC_FP64), O.gpp(prob)
    assert np.abs(g[0] - o[0]).max() <= TOL * np.abs(o[0]).max()
    assert np.abs(g[1] - o[1]).max() <= TOL * np.abs(o[1]).max()


# ---- values whose squares leave the FP32 range of the row bounds
def test_halfsum_static_of_tiny_inverse_dielectric_values(sigma_lib):
    prob = W.gpp_random(64, 0, 4096, 16, 44)
    prob.I_eps_array *= 1e-30
    prob.wtilde_array.real[:] = 0.5 + (prob.wtilde_array.real - 0.5) * (1.5 / 4.5)
    _close(sigma_lib.gpp_halfsum_host(prob)[3], O.gpp_halfsum(prob)[3])


def test_gpp_tiny_inverse_dielectric_value_at_large_pole(sigma_lib):
    prob = W.gpp_random(45, 2, 3001, 37, 45)
    prob.I_eps_array[3, 100] = 1e-24
    prob.wtilde_array[3, 100] = 1e14
    g, o = sigma_lib.gpp_host(prob, sigma_lib.PREC_FP64), O.gpp(prob)
    _close(g[0], o[0])
    _close(g[1], o[1])
