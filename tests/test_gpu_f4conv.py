"""k_f4_conv, which sums the far wings of mixed Jacobians' ODs record by record
through shared-memory stages: no stage size changes a Jacobian by a bit, and
the mirror records of lines near 0 cm-1, which follow the direct ones through
the stages, are the oracle's."""
import os

import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu

KEYS = ("rad", "dtlev", "dqlev", "dtsfc", "demis")


def _handle(gpu_lib, lines, cont, stage):
    old = os.environ.pop("CLBLM_F4_STAGE_RECORDS", None)
    if stage:
        os.environ["CLBLM_F4_STAGE_RECORDS"] = str(stage)
    try:
        return gpu_lib.Handle(lines, cont)
    finally:
        os.environ.pop("CLBLM_F4_STAGE_RECORDS", None)
        if old is not None:
            os.environ["CLBLM_F4_STAGE_RECORDS"] = old


@pytest.mark.parametrize("window", [(1000.0, 1004.0), (4.0, 40.0)])
def test_stage_size_does_not_change_a_jacobian(gpu_lib, mtckd, window):
    """Every stage size, set and chosen, on a window in the middle and on one
    whose mirror records pass through the stages."""
    lo = max(1.0, window[0] - 30.0)
    lines = synth.line_list(24000, lo, window[1] + 30.0, seed=11, mols=synth.SEVEN)
    _, col, _ = synth.config1(n_lines=10)
    c = col.sub([10, 11, 12]).with_window(*window)
    prof = synth.jac_profile(col).sub(10, 3)
    ctrl = T.rt_ctrl(precision=T.CLBLM_PREC_MIXED, grid_type=1)
    got = {}
    for stage in (0, 64, 128, 256):
        h = _handle(gpu_lib, lines, mtckd, stage)
        got[stage] = h.jac(c, ctrl, prof)
        assert h.stats()["f4_stage_records"] in ((64, 128, 256) if stage == 0 else (stage,))
        h.close()
    for stage in (64, 128, 256):
        for k in KEYS:
            np.testing.assert_array_equal(got[stage][k], got[0][k], err_msg="%s at %d records" % (k, stage))


def test_mixed_jacobian_with_mirror_records(gpu_lib, oracle_mod):
    """A mixed Jacobian below 25 cm-1, where the mirror records of the lines
    near 0 follow the direct ones through k_f4_conv's stages (hundreds of them,
    several stages): the far wings against the FP64 oracle's, at the
    repository's tolerances for Jacobians."""
    lines = synth.line_list(9000, 1.0, 70.0, seed=7, mols=synth.SEVEN)
    _, col, _ = synth.config1(n_lines=10)
    c = col.sub([20, 21]).with_window(3.0, 9.0)
    prof = synth.jac_profile(col).sub(20, 2)
    ctrl = T.rt_ctrl(precision=T.CLBLM_PREC_MIXED, grid_type=1, contnm_off=1)
    h = gpu_lib.Handle(lines, None)
    got = h.jac(c, ctrl, prof)
    h.close()
    want = oracle_mod.jac_mode2(oracle_mod.Session(), lines, c, ctrl, prof, None)
    assert len(got["rad"]) == len(want["rad"]) and got["dv"] == want["dv"]
    np.testing.assert_allclose(got["rad"], want["rad"], rtol=1e-4)
    for k in ("dtlev", "dqlev", "dtsfc", "demis"):
        scale = np.max(np.abs(want[k]), axis=-1, keepdims=True)
        assert np.max(np.abs(got[k] - want[k]) / np.where(scale > 0, scale, 1.0)) <= 2e-3, k
