"""The far-wing record loop in its three kernels (counts of the possible SHRINQ
calls, the record loop, the groups): line selection bit-exact against the
oracle's trace where the calls are at their edges: dense records (a call of
four records or of one), records few of whose lines are selected (calls longer
than the table holds, counted by the CTA), a call that ends the stream inside
a record, one record in all, groups longer than a call.  Whole numbers: no
tolerance; centres as in the repository's own line-selection test."""
import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu

WINDOW = (700.0, 712.0)


def _lines(kind):
    lo, hi = WINDOW[0] - 40.0, WINDOW[1] + 40.0
    if kind == "dense":       # every line selected, narrow groups
        return synth.line_list(40000, lo, hi, seed=1, mols=(1,)), 2.0
    if kind == "wide":        # a surface layer: groups of hundreds of lines
        return synth.line_list(40000, lo, hi, seed=2, mols=(1,)), 1013.25
    if kind == "sparse":      # one line in 60 selected: calls of hundreds of records
        return _one_in(60, synth.line_list(150000, lo, hi, seed=3, mols=(2,))), 2.0
    if kind == "mixed":       # one line in 7: calls of about 28 records
        return synth.line_list(60000, lo, hi, seed=4, mols=(1, 2, 3, 4, 5, 6, 8)), 30.0
    if kind == "one_record":
        return synth.line_list(200, lo, hi, seed=5, mols=(1,)), 100.0
    return synth.line_list(1260, lo, hi, seed=6, mols=(1,)), 2.0  # "five_records"


def _one_in(k, lines):
    lines.mol[::k] = 101
    return lines


@pytest.mark.parametrize("precision", [T.CLBLM_PREC_MIXED, T.CLBLM_PREC_PLAIN])
@pytest.mark.parametrize("kind", ["dense", "wide", "sparse", "mixed", "one_record", "five_records"])
def test_shrinq_calls_bit_exact(gpu_lib, oracle_mod, kind, precision):
    lines, pave = _lines(kind)
    v1, v2 = WINDOW
    mols = np.array([1], np.int32)
    f = pave / 1013.25
    col = T.Column(mols, [pave], [270.0], [270.0], [270.0], np.array([[1.0e21 * f]]), [2.4e24 * f], [4.0e24 * f],
                   v1, v2, 270.0, 1.0)
    dn, df, _ = gpu_lib.setDV(col)
    grid = T.grid_struct(v1, v2, dn[0], df[0])
    ctrl = T.od_ctrl(precision=precision, contnm_off=1)
    h = gpu_lib.Handle(lines, None)
    od, _ = h.odlay(col.layer(0), grid, ctrl)
    got = h.od_lines()
    h.close()
    ref, _, _, tr = oracle_mod.Session().odlay_trace(lines, col.layer(0), grid, ctrl, None)
    assert np.array_equal(got["shr_last"], tr["shr_last"])
    assert np.array_equal(got["shr_mol"], tr["shr_mol"])
    assert np.max(np.abs(od - ref) / np.abs(ref)) <= (1e-5 if precision == T.CLBLM_PREC_MIXED else 1e-9)
