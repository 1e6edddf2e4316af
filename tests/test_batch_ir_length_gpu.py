"""A batch query whose IR length does not fit 32 bits, or with the others' not
4 KiB, is an invalid argument."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(1 << 32,), ((1 << 32) + 3,), (1 << 31,), (4097,), (4000, 97),
                                     (16, (1 << 64) - 8)], ids=str)
def test_overlong_ir_is_refused(gpj, lengths):
    lib = gpj.load_library()
    ir = (C.c_uint8 * 4200)()
    dev = torch.zeros(256, dtype=torch.uint8, device="cuda")
    files = (gpj.BatchFile * 1)(gpj.BatchFile(0, 2, 0, 0))
    queries = (gpj.BatchQuery * len(lengths))(*[
        gpj.BatchQuery(C.addressof(ir), n, 1, 0, 2, 0) for n in lengths])
    out = C.c_void_p()
    assert lib.gpj_batch_create(None, C.c_void_p(dev.data_ptr()), 256, files, 1, queries,
                                len(lengths), 0, C.byref(out), None) == gpj.GPJ_ERR_INVALID_ARGUMENT
    assert not out.value
