"""The FFT scan through the low coefficients alone (k_scan_moments, k_scan_low,
k_scan_expand) against the oracle: every apodization that ends, padding,
pre-boxing with its deconvolution, half widths on either side of where the
whole transform takes over (M = N / 32 blocks at 512 coefficients of the
smallest transform), output limits that start and end inside a block.
Tolerance as in the repository's scan tests: 1e-11 of the largest value (the
expansion's terms are cut below 1e-16)."""
import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth
from oracle import fftscn as S

pytestmark = pytest.mark.gpu


def _spectrum(v1, n, dv, seed):
    rng = np.random.default_rng(seed)
    return 1.0 + 0.3 * np.sin(np.arange(n) * dv / 1.1) + rng.uniform(-0.5, 0.5, n)


def _check(gpu_lib, n, dv, fid, hw, a, b, fill=0.0, prebox=-1.0, deconv=0):
    v1 = 1000.0
    x = _spectrum(v1, n, dv, n)
    want, v1s, dvs = S.fftscn(x, v1, dv, fid, hw, a, b, fill=fill, prebox_hw=prebox, deconv_prebox=bool(deconv))
    h = gpu_lib.Handle(synth.line_list(1000, 600.0, 700.0, seed=0))
    try:
        got, g1, gdv = h.fftscn(T.scan_struct(fid, hw, a, b, padding=fill, prebox_hw=prebox, deconv_prebox=deconv), x,
                                v1, dv)
    finally:
        h.close()
    assert (g1, gdv, len(got)) == (v1s, dvs, len(want))
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 * np.abs(want).max())


@pytest.mark.parametrize("fid", [3, 4, 5, 6, 7, 8, 9, 10, 11])
@pytest.mark.parametrize("fill", [0.0, 1.0])
def test_every_ending_apodization(gpu_lib, fid, fill):
    _check(gpu_lib, 50001, 0.002, fid, 0.6, 1030.0011, 1070.0, fill=fill)


@pytest.mark.parametrize("hw", [0.3, 0.309, 0.3112, 0.313, 0.32, 0.7])
def test_switch_to_the_whole_transform(gpu_lib, hw):
    _check(gpu_lib, 60000, 0.002, 5, hw, 1055.0, 1062.003)


@pytest.mark.parametrize("fid", [3, 5])
def test_prebox_and_deconvolution(gpu_lib, fid):
    _check(gpu_lib, 130001, 0.001, fid, 0.75, 1060.0, 1071.0, fill=1.0, prebox=0.0026, deconv=1)


@pytest.mark.parametrize("n", [65536, 65537, 131072, 200003])
def test_data_ending_at_records_and_blocks(gpu_lib, n):
    dv = 0.0005 if n > 100000 else 0.001
    v2 = 1000.0 + dv * (n - 1)
    _check(gpu_lib, n, dv, 3, 0.8, 1000.0 + 0.3 * (v2 - 1000.0), v2)


# transforms of 4096 to 131072 points in parts (odd and even powers of two a
# part), and of 262144 points whole
@pytest.mark.parametrize("n,dv,hw", [(1000000, 5e-4, 2.6), (600000, 5e-4, 1.3), (600000, 5e-4, 0.65),
                                     (1100000, 5e-4, 0.65), (4300000, 2e-4, 0.5), (4300000, 2e-4, 0.26),
                                     (4300000, 2e-4, 0.2)])
def test_transform_sizes(gpu_lib, n, dv, hw):
    _check(gpu_lib, n, dv, 5, hw, 1000.0 + 0.4 * dv * n, 1000.0 + 0.9 * dv * n, fill=0.5)


# as many coefficients as a sixty-fourth of the points, and more: the wide form
# (24 terms, blocks of 32 points and more) and the whole transform after it
@pytest.mark.parametrize("fid", [3, 5])
@pytest.mark.parametrize("hw", [0.30, 0.12, 0.082, 0.08, 0.05])
def test_wide_form(gpu_lib, fid, hw):
    _check(gpu_lib, 60000, 0.002, fid, hw, 1055.0, 1062.003, fill=0.5)


def test_wide_form_of_many_points(gpu_lib):
    _check(gpu_lib, 700000, 0.0015, 5, 0.4, 1300.0, 1800.0)
