"""Which kernel a parallel-beam call takes (CPU only: the dispatch rule itself, on the host)."""
import ctypes
import itertools

import pytest

from vamtoolbox_b200 import _lib

AUTO = dict(forward_vz=0, backward_vz=0, adjoint_vz=0, backward_batch=2, adjoint_table=1, backward_table=1,
            forward_tma=1)
ALIGNED = 1 << 20


def route(n, nz, na, op, padded=False, absorption=_lib.ABS_NONE, occlusion=0, table=0, tasks=None, src=ALIGNED,
          dst=ALIGNED, **tuning):
    """(return code, ParallelRoute) of one call."""
    t = _lib.ParallelTuning(*({**AUTO, **tuning}[k] for k, _ in _lib.ParallelTuning._fields_))
    call = _lib.ParallelCall(n, nz, na, tasks or (na + 1) // 2, absorption, occlusion, table,
                             op | (_lib.OP_PADDED if padded else 0), src, dst, t)
    out = _lib.ParallelRoute()
    return _lib.load().vam_parallel_route(ctypes.byref(call), ctypes.byref(out)), out


TUNED = [dict(backward_vz=v, backward_batch=b, backward_table=t)
         for v, b, t in itertools.product((0, 1, 4, 8), (1, 2, 4), (0, 1))]


@pytest.mark.parametrize("nz", [5, 9, 33, 63, 65, 117, 130, 191, 193, 201, 255, 257, 318])
@pytest.mark.parametrize("absorption", [_lib.ABS_NONE, _lib.ABS_MASK, _lib.ABS_RAY])
def test_padded_backprojection_steps_by_its_padded_rows(nz, absorption):
    """An input whose rows are padded goes to a body that steps by the padded rows and stores slice by slice where
    the output's rows are not whole float4s, whatever the tuning, with and without a bin table."""
    for tuned, table in itertools.product(TUNED, (0, 1)):
        rc, r = route(201, nz, 240, _lib.OP_BACKWARD_REF, padded=True, absorption=absorption, table=table, **tuned)
        assert rc == _lib.VAM_OK
        assert r.kernel in (_lib.KERNEL_BACKWARD_TABLE, _lib.KERNEL_BACKWARD_GENERIC), (tuned, table, r.kernel)
        assert r.row_stride == (nz + 3) // 4 * 4 and r.vector_loads and not r.vector_stores, (tuned, table)
        # and what the unpadded call takes is unchanged by any of this: single floats
        rc, r = route(201, nz, 240, _lib.OP_BACKWARD_REF, absorption=absorption, table=table, **tuned)
        assert (rc, r.kernel, r.slices_per_lane, r.row_stride) == (_lib.VAM_OK, _lib.KERNEL_BACKWARD_GENERIC, 1, nz)


@pytest.mark.parametrize("nz", [8, 33, 64, 67, 130, 256])
@pytest.mark.parametrize("op", [_lib.OP_FORWARD, _lib.OP_BACKWARD_REF, _lib.OP_ADJOINT])
def test_padded_rows_are_checked_for_alignment(nz, op):
    """Padded rows are read as float4s: an input off a 16-byte boundary is refused.  The output may lie anywhere
    (a multiple of four floats only): where it is off such a boundary it is stored slice by slice."""
    for off in (4, 8, 12):
        assert route(96, nz, 90, op, padded=True, table=1, src=ALIGNED + off)[0] == _lib.VAM_ERR_ARG
    for off, tuned in itertools.product((4, 8, 12), TUNED):
        rc, r = route(96, nz, 90, op, padded=True, table=1, dst=ALIGNED + off, **tuned)
        assert rc == _lib.VAM_OK or (nz == 8 and op != _lib.OP_BACKWARD_REF and rc == _lib.VAM_ERR_NOTSUP)
        assert rc != _lib.VAM_OK or not r.vector_stores, (off, tuned, r.kernel)


@pytest.mark.parametrize("n,nz,na", [(2048, 513, 8), (1300, 1301, 30), (201, 117, 240), (64, 33, 90), (3000, 31, 30000),
                                     (96, 9, 90)])
def test_rows_are_padded_only_where_the_padded_kernels_serve_the_call(n, nz, na, monkeypatch):
    """Whether a plan pads its input is the dispatch's own answer, so no padded call is refused; a padded copy has
    fewer than 2^31 elements.  A volume of 2^31 elements or more goes unpadded to the generic forward."""
    import types

    import numpy as np

    from vamtoolbox_b200.projector import Projector3DParallel as module

    forms = itertools.product((_lib.OP_FORWARD, _lib.OP_BACKWARD_REF, _lib.OP_ADJOINT),
                              (_lib.ABS_NONE, _lib.ABS_MASK, _lib.ABS_RAY), (0, 1), (0, 1),
                              (dict(), dict(forward_vz=1, adjoint_vz=1, backward_vz=1), dict(forward_vz=8, adjoint_vz=4)))
    padded = 0
    for op, absorption, occlusion, table, tuning in forms:
        form = dict(absorption=absorption, occlusion=occlusion, table=table, **tuning)
        plan = module.ParallelPlan.__new__(module.ParallelPlan)
        plan.shape_vol, plan.angles, plan._h = (n, n, nz), np.zeros(na), None
        plan.pad_from, plan.pad_backward_from = 0, 0
        serves = route(n, nz, na, op, **form)[1].pads
        monkeypatch.setattr(module._lib, "load",
                            lambda: types.SimpleNamespace(vam_parallel_serves_padded=lambda handle, code: serves))
        pads = plan._pads(op)
        monkeypatch.undo()
        rc, r = route(n, nz, na, op, padded=pads, **form)
        assert rc == _lib.VAM_OK, (op, form)
        if pads:
            padded += 1
            assert n * (n if op == _lib.OP_FORWARD else na) * ((nz + 3) // 4 * 4) < 2 ** 31, (op, form)
        elif op == _lib.OP_FORWARD and n * n * nz >= 2 ** 31:
            assert r.kernel == _lib.KERNEL_FORWARD_GENERIC, form
    assert padded or n * n * nz >= 2 ** 31 or n * na * nz >= 2 ** 31


def test_few_slices_take_the_kernel_that_is_faster_there():
    """Strips and blocks from the slice counts on at which they were measured to beat the generic kernels, which
    depend on absorption, on angles 180 degrees apart and on the slice's size; a tuning chooses either."""
    forward, adjoint = _lib.OP_FORWARD, _lib.OP_ADJOINT
    strip, block = _lib.KERNEL_FORWARD_STRIP, _lib.KERNEL_ADJOINT_BLOCK
    for n, nz, na, tasks, absorption, strips in [
            (54, 16, 636, 318, _lib.ABS_RAY, False), (256, 32, 360, 180, _lib.ABS_RAY, False),
            (256, 56, 360, 180, _lib.ABS_RAY, True), (96, 11, 90, 45, _lib.ABS_RAY, False),
            (96, 15, 90, 45, _lib.ABS_RAY, True), (96, 16, 91, 91, _lib.ABS_NONE, False),
            (96, 20, 91, 91, _lib.ABS_NONE, True), (96, 12, 90, 45, _lib.ABS_MASK, True),
            (54, 16, 90, 45, _lib.ABS_MASK, False), (54, 5, 90, 45, _lib.ABS_NONE, True),
            (96, 7, 91, 91, _lib.ABS_NONE, False), (32, 32, 90, 45, _lib.ABS_NONE, False),
            (32, 45, 90, 45, _lib.ABS_NONE, True), (32, 60, 90, 45, _lib.ABS_RAY, True),
            (64, 36, 30, 15, _lib.ABS_NONE, False), (96, 45, 8, 4, _lib.ABS_NONE, False),
            (96, 117, 8, 4, _lib.ABS_NONE, True), (96, 128, 8, 4, _lib.ABS_RAY, True),
            (12, 16, 11, 7, _lib.ABS_NONE, True)]:
        got = route(n, nz, na, forward, absorption=absorption, tasks=tasks)[1].kernel
        assert (got == strip) == strips, (n, nz, na, absorption)
    for n, nz, absorption, blocks in [(32, 12, _lib.ABS_NONE, False), (32, 16, _lib.ABS_NONE, True),
                                      (32, 24, _lib.ABS_RAY, False), (32, 28, _lib.ABS_RAY, True),
                                      (32, 6, _lib.ABS_RAY, False), (54, 12, _lib.ABS_RAY, True)]:
        assert (route(n, nz, 90, adjoint, absorption=absorption)[1].kernel == block) == blocks, (n, nz, absorption)
    for op, vz, kernel in [(forward, "forward_vz", strip), (adjoint, "adjoint_vz", block)]:
        assert route(32, 12, 90, op, **{vz: 4})[1].kernel == kernel
        assert route(128, 128, 90, op, **{vz: 1})[1].kernel == kernel + 1
    assert block + 1 == _lib.KERNEL_ADJOINT_GENERIC and strip + 1 == _lib.KERNEL_FORWARD_GENERIC
