"""The Gaussian's apodization stops at e^-34: the coefficients past that keep
1.7e-15 of themselves.  A cosine whose path difference lies there passes the
scan with that amplitude, in both forms of the scan through the low
coefficients, pre-boxed, deconvolved, and onto the data's own buffer.  The
amplitude is taken by projection over 9000 points and more, where the roundings
of 3e-16 a point average to 1 % of it at most; held to 5 % of the oracle's."""
import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth
from oracle import fftscn as S

pytestmark = pytest.mark.gpu
FLOOR = np.exp(-34.0)


def _cosine(n, dv, period):
    return np.cos(2.0 * np.pi / period * dv * np.arange(n))


@pytest.mark.parametrize("n,dv,hw,a,b,prebox,deconv", [
    (50001, 0.002, 0.6, 1030.0011, 1070.0, -1.0, 0),   # twelve moments
    (60000, 0.002, 0.3, 1030.0, 1062.003, -1.0, 0),    # the wide form
    (130001, 0.001, 0.75, 1025.0, 1111.0, 0.0026, 0),  # means of five points
    (130001, 0.001, 0.75, 1025.0, 1111.0, 0.0026, 1),  # divided by their transform
])
def test_amplitude_past_the_floor(gpu_lib, n, dv, hw, a, b, prebox, deconv):
    v1, period = 1000.0, 0.05
    x = _cosine(n, dv, period)
    want, v1s, dvs = S.fftscn(x, v1, dv, 3, hw, a, b, prebox_hw=prebox, deconv_prebox=bool(deconv))
    h = gpu_lib.Handle(synth.line_list(1000, 600.0, 700.0, seed=0))
    try:
        got, g1, gdv = h.fftscn(T.scan_struct(3, hw, a, b, prebox_hw=prebox, deconv_prebox=deconv), x, v1, dv)
    finally:
        h.close()
    assert (g1, gdv, len(got)) == (v1s, dvs, len(want))
    c = np.cos(2.0 * np.pi / period * (v1s - v1 + dvs * np.arange(len(want))))
    assert abs(2.0 * np.mean((got - want) * c)) <= 0.05 * FLOOR


def test_output_over_the_data(gpu_lib):
    import torch

    n, dv, v1 = 50001, 0.002, 1000.0
    x = 1.0 + _cosine(n, dv, 7.0)
    sc = T.scan_struct(3, 0.6, 1030.0011, 1070.0)
    want, _, _ = S.fftscn(x, v1, dv, 3, 0.6, 1030.0011, 1070.0)
    h = gpu_lib.Handle(synth.line_list(1000, 600.0, 700.0, seed=0))
    try:
        buf = torch.from_numpy(x).cuda()
        h.fftscn_device(sc, buf.data_ptr(), n, v1, dv, buf.data_ptr() + 8 * 14000, len(want))
        torch.cuda.synchronize()
        got = buf[14000:14000 + len(want)].cpu().numpy()
    finally:
        h.close()
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 * np.abs(want).max())
