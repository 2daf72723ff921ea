"""The far wings through nodes (k_f4_far) against the oracle, where they can go
wrong: windows whose far-wing grid ends at the edges of a leaf (32 points) and
of a tile (128), thin layers whose records are far from most tiles, thick ones
without any far record, the CO2 pedestal, lines wider than the near distance,
mirror lines below 25 cm-1, windows with lines on one side alone.  The ODs are
held to the repository's tolerances (1e-5 mixed, 1e-9 FP64): the interpolation
adds below 4e-8 of a record's own term (mixed; 4e-15 FP64)."""
import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu


def _column(pave, tave, v1, v2, mols, w):
    mols = np.array(mols, np.int32)
    f = pave / 1013.25
    return T.Column(mols, [pave], [tave], [tave], [tave], np.array([[x * f for x in w]]), [2.4e24 * f], [4.0e24 * f],
                    v1, v2, tave, 1.0)


def _check(gpu_lib, oracle_mod, lines, col, precision):
    dn, df, _ = gpu_lib.setDV(col)
    grid = T.grid_struct(col.v1, col.v2, dn[0], df[0])
    ctrl = T.od_ctrl(precision=precision, contnm_off=1)
    h = gpu_lib.Handle(lines, None)
    od, dv = h.odlay(col.layer(0), grid, ctrl)
    h.close()
    ref, dvr, _ = oracle_mod.Session().odlay(lines, col.layer(0), grid, ctrl, None)
    assert dv == dvr and len(od) == len(ref)
    tol = 1e-5 if precision == T.CLBLM_PREC_MIXED else 1e-9
    err = np.abs(od - ref)
    assert np.max(err / np.maximum(np.abs(ref), 1e-6 * np.max(np.abs(ref)))) <= tol


@pytest.mark.parametrize("precision", [T.CLBLM_PREC_MIXED, T.CLBLM_PREC_PLAIN])
@pytest.mark.parametrize("points", [31, 32, 33, 127, 128, 129, 256, 258])
def test_grid_ends_at_leaf_and_tile_edges(gpu_lib, oracle_mod, points, precision):
    lines = synth.line_list(9000, 870.0, 930.0, seed=points, mols=(1, 2))
    c = _column(3.0, 230.0, 900.0, 901.0, (1, 2), (1.0e21, 1.0e20))
    dn, df, _ = gpu_lib.setDV(c)
    dv = dn[0] if abs(dn[0] - df[0]) / dn[0] > 0.2 else df[0]
    _check(gpu_lib, oracle_mod, lines, c.with_window(900.0, 900.0 + (points - 4.5) * 64.0 * dv), precision)


@pytest.mark.parametrize("precision", [T.CLBLM_PREC_MIXED, T.CLBLM_PREC_PLAIN])
@pytest.mark.parametrize("kind", ["top", "middle", "surface", "co2", "wide", "left", "right", "mirror"])
def test_far_wings(gpu_lib, oracle_mod, kind, precision):
    mols, w, v1, v2, pave, tave = (1,), (1.0e21,), 900.0, 912.0, 0.3, 230.0
    lines = synth.line_list(12000, 860.0, 952.0, seed=3, mols=mols)
    if kind == "middle":
        pave, tave = 60.0, 240.0
    elif kind == "surface":
        pave, tave = 1013.25, 290.0
    elif kind == "co2":
        mols, w = (1, 2), (1.0e20, 1.0e22)
        lines = synth.line_list(12000, 860.0, 952.0, seed=4, mols=mols)
    elif kind == "wide":  # widths of 40 times the usual: cores past the near distance
        pave = 20.0
        lines.alfa[::50] *= 40.0
        lines.hwhm[::50] *= 40.0
    elif kind == "left":
        lines = synth.line_list(6000, 860.0, 899.0, seed=5, mols=mols)
    elif kind == "right":
        lines = synth.line_list(6000, 913.0, 952.0, seed=6, mols=mols)
    elif kind == "mirror":
        v1, v2, pave = 6.0, 30.0, 20.0
        lines = synth.line_list(9000, 1.0, 70.0, seed=7, mols=mols)
    _check(gpu_lib, oracle_mod, lines, _column(pave, tave, v1, v2, mols, w), precision)
