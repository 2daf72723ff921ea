"""The slices of the panel kernel's line pass: layers whose panels are cut into
one, a few and the most CTAs, with shares of a tile's records that divide
evenly or not (and are empty), against the oracle.  The cut follows the lines
per 768 DV of the layer, here set by the line density: the tolerances are the
repository's for a layer OD (a slice's FP32 sums carry the same half unit in
the last place as the whole's, and they are added compensated)."""
import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(T.CLBLM_PREC_MIXED, 1e-5), (T.CLBLM_PREC_PLAIN, 1e-9)])
@pytest.mark.parametrize("n_lines,width,pave", [
    (3, 20.0, 1013.25),      # fewer records than threads, most shares empty
    (1500, 20.0, 1013.25),   # a few slices
    (3001, 61.0, 1013.25),   # odd counts, a second panel
    (30011, 15.0, 1013.25),  # the most slices
    (6000, 20.0, 60.0),      # narrow lines: one slice
])
def test_sliced_line_pass(gpu_lib, oracle_mod, n_lines, width, pave, precision, tol):
    lines = synth.line_list(n_lines, 700.0, 700.0 + width, seed=n_lines, mols=(1, 2))
    mols = np.array([1, 2], np.int32)
    w = np.array([[1.0e21, 1.0e20]]) * (pave / 1013.25)
    col = T.Column(mols, [pave], [280.0], [280.0], [280.0], w, [2.4e24 * pave / 1013.25], [4.0e24 * pave / 1013.25],
                   700.0, 700.0 + width, 280.0, 1.0)
    dn, df, _ = gpu_lib.setDV(col)
    grid = T.grid_struct(col.v1, col.v2, dn[0], df[0])
    ctrl = T.od_ctrl(precision=precision, contnm_off=1)
    h = gpu_lib.Handle(lines, None)
    od, dv = h.odlay(col.layer(0), grid, ctrl)
    h.close()
    ref, dvr, _ = oracle_mod.Session().odlay(lines, col.layer(0), grid, ctrl, None)
    assert dv == dvr and len(od) == len(ref)
    assert np.max(np.abs(od - ref) / np.abs(ref)) <= tol
