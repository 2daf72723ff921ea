"""The radiation terms formed ahead of the far-wing pass against the oracle:
panels with few segments (k_panel_segs' table), with more than it holds and
with more than shared memory holds (low wavenumbers at a coarse DV), and the
JRAD = 1 factors of far-wing blocks, one short block and several full ones.
The repository's tolerances for a layer OD."""
import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(T.CLBLM_PREC_MIXED, 1e-5), (T.CLBLM_PREC_PLAIN, 1e-9)])
@pytest.mark.parametrize("v1,v2,pave", [
    (1.5, 45.0, 1013.25),     # JRAD = 0: hundreds of segments a panel
    (40.0, 120.0, 1013.25),   # tens
    (560.0, 640.0, 1013.25),  # a few
    (800.0, 801.5, 1.0),      # one or two
    (1900.0, 1902.0, 50.0),   # JRAD = 1: one short block
    (1900.0, 2060.0, 0.3),    # full blocks of 2500 points
])
def test_radiation_terms(gpu_lib, oracle_mod, v1, v2, pave, precision, tol):
    lines = synth.line_list(int(40 * (v2 - v1 + 60)) + 500, max(0.5, v1 - 30.0), v2 + 30.0, seed=9, mols=(1,))
    mols, f = np.array([1], np.int32), pave / 1013.25
    col = T.Column(mols, [pave], [255.0], [255.0], [255.0], np.array([[1.0e21 * f]]), [2.4e24 * f], [4.0e24 * f],
                   v1, v2, 255.0, 1.0)
    dn, df, _ = gpu_lib.setDV(col)
    grid = T.grid_struct(v1, v2, dn[0], df[0])
    ctrl = T.od_ctrl(precision=precision, contnm_off=1)
    h = gpu_lib.Handle(lines, None)
    od, _ = h.odlay(col.layer(0), grid, ctrl)
    st = h.stats()
    h.close()
    ref, _, sr = oracle_mod.Session().odlay(lines, col.layer(0), grid, ctrl, None)
    assert st["jrad"] == sr["jrad"] == (1 if v1 > 886.2 else 0)  # V1 over 5 kT
    assert len(od) == len(ref)
    assert np.max(np.abs(od - ref) / np.maximum(np.abs(ref), 1e-6 * np.max(np.abs(ref)))) <= tol
