"""Device memory of clblm_gpu_jac, whose blocks of a wide window share the OD
pipeline's launches in groups: a group keeps to its bound where one block has
many more lines than the others (the pipeline's arrays are as long as the
largest job's, times the jobs), a device with little memory left gets one block
at a time, and neither the groups nor several OD batches of a block change the
result."""
import os

import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu

KEYS = ("rad", "dtlev", "dqlev", "dtsfc", "demis")


def _column(v1, v2):
    _, col, cont = synth.config1(n_lines=10)
    first, count = 10, 6
    return col.sub(list(range(first, first + count))).with_window(v1, v2), synth.jac_profile(col).sub(first, count), cont


def _lines(v1, v2, sparse, band=None, dense=0):
    """`sparse` lines per cm-1 over the window and its wings, `dense` in `band`"""
    a = synth.line_list(int(sparse * (v2 - v1 + 60.0)), v1 - 30.0, v2 + 30.0, seed=1, mols=synth.SEVEN)
    if band is None:
        return a
    b = synth.line_list(int(dense * (band[1] - band[0])), band[0], band[1], seed=2, mols=synth.SEVEN)
    order = np.argsort(np.concatenate([a.vnu, b.vnu]), kind="stable")
    return T.Lines(**{n: np.concatenate([getattr(a, n), getattr(b, n)])[order] for n, _ in T.Lines.FIELDS})


@pytest.fixture
def budget():
    old = os.environ.pop("CLBLM_OD_BUDGET_GB", None)

    def put(gb):
        os.environ["CLBLM_OD_BUDGET_GB"] = str(gb)

    yield put
    os.environ.pop("CLBLM_OD_BUDGET_GB", None)
    if old is not None:
        os.environ["CLBLM_OD_BUDGET_GB"] = old


def test_group_with_one_dense_block_keeps_its_bound(gpu_lib, budget):
    import torch
    v1, v2 = 700.0, 1900.0
    col, prof, cont = _column(v1, v2)
    lines = _lines(v1, v2, 20.0, (1290.0, 1300.0), 6000.0)
    ctrl = T.rt_ctrl(precision=T.CLBLM_PREC_MIXED, grid_type=1)
    gb = 1.5
    budget(gb)
    h = gpu_lib.Handle(lines, cont)
    n, _ = h.jac_size(col, ctrl, prof)
    out = {k: torch.empty(((col.nlay + 1, n) if k in ("dtlev", "dqlev") else n), dtype=torch.float64, device="cuda")
           for k in KEYS}
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    h.jac_device(col, ctrl, prof, out["rad"].data_ptr(), out["dtlev"].data_ptr(), out["dqlev"].data_ptr(),
                 out["dtsfc"].data_ptr(), out["demis"].data_ptr(), n)
    torch.cuda.synchronize()
    free1, _ = torch.cuda.mem_get_info()
    h.close()
    # an eighth of each buffer for its growth, the pool of radiation-term
    # segments (0.26 GB) and the driver's local memory for the kernels
    assert free0 - free1 <= (1.25 * gb + 0.75) * 2**30, (free0 - free1) / 2**30


@pytest.mark.parametrize("precision", [T.CLBLM_PREC_MIXED, T.CLBLM_PREC_PLAIN])
def test_groups_and_batches_do_not_change_the_result(gpu_lib, budget, precision):
    v1, v2 = 1000.0, 1110.0
    col, prof, cont = _column(v1, v2)
    lines = _lines(v1, v2, 60.0, (1050.0, 1054.0), 1500.0)
    ctrl = T.rt_ctrl(precision=precision, grid_type=1)
    got = {}
    # all blocks in one group; groups of some; a batch of a few ODs at a time
    for gb in (16.0, 0.15, 0.004):
        budget(gb)
        h = gpu_lib.Handle(lines, cont)
        got[gb] = h.jac(col, ctrl, prof)
        h.close()
    for gb in (0.15, 0.004):
        for k in KEYS:
            np.testing.assert_array_equal(got[gb][k], got[16.0][k], err_msg="%s at %g GB" % (k, gb))


# the slabs and maps of all blocks still fit, then not even they
@pytest.mark.parametrize("part", [1.0, 0.5])
def test_little_memory_left(gpu_lib, budget, part):
    import torch
    v1, v2 = 700.0, 2300.0
    col, prof, cont = _column(v1, v2)
    lines = _lines(v1, v2, 2.0)
    ctrl = T.rt_ctrl(precision=T.CLBLM_PREC_MIXED, grid_type=1)
    h = gpu_lib.Handle(lines, cont)
    want = h.jac(col, ctrl, prof)  # (the kernels are loaded and have their local memory)
    h.close()
    n = len(want["rad"])
    h = gpu_lib.Handle(lines, cont)
    out = {k: torch.zeros(((col.nlay + 1, n) if k in ("dtlev", "dqlev") else n), dtype=torch.float64, device="cuda")
           for k in KEYS}
    budget(8.0)  # the least that a call plans with whatever is free
    # room for `part` of the OD slabs and maps of all blocks (16 and 32 bytes a
    # layer and point, an eighth more for growth), and 0.15 GB
    slabs = 48 * col.nlay * n * 9 // 8
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill = free - int(part * slabs) - int(0.15 * 2**30)
    assert slabs > 2**30 and fill > 0
    block = torch.empty(fill, dtype=torch.uint8, device="cuda")
    try:
        h.jac_device(col, ctrl, prof, out["rad"].data_ptr(), out["dtlev"].data_ptr(), out["dqlev"].data_ptr(),
                     out["dtsfc"].data_ptr(), out["demis"].data_ptr(), n)
        torch.cuda.synchronize()
    finally:
        del block
        torch.cuda.empty_cache()
        h.close()
    for k in KEYS:
        np.testing.assert_array_equal(out[k].cpu().numpy(), want[k], err_msg=k)


def test_call_after_an_out_of_memory_result(gpu_lib, budget):
    """A call that returns out of memory leaves no error behind: neither the
    next call of the handle nor another library's check finds it."""
    import torch
    col, prof, cont = _column(1000.0, 1004.0)
    lines = _lines(1000.0, 1004.0, 60.0)
    ctrl = T.rt_ctrl(precision=T.CLBLM_PREC_MIXED, grid_type=1)
    h = gpu_lib.Handle(lines, cont)
    want = h.jac(col, ctrl, prof)
    h.close()
    h = gpu_lib.Handle(lines, cont)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - int(0.1 * 2**30), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(gpu_lib.ClblmError) as e:
            h.jac(col, ctrl, prof)
        assert e.value.code == T.CLBLM_ERR_OOM
        torch.cuda.synchronize()
    finally:
        del block
        torch.cuda.empty_cache()
    got = h.jac(col, ctrl, prof)
    h.close()
    for k in KEYS:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
