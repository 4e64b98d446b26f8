"""The post-pattern stage reports a wait that fails.  The failure is the host's: a wait on a stream that
is being captured is refused, and what was enqueued has not run."""
import ctypes as C

import numpy as np
import pytest

import wukong_b200 as wk

pytestmark = pytest.mark.gpu

THREAD_LOCAL = 1   # CU_STREAM_CAPTURE_MODE_THREAD_LOCAL


@pytest.mark.parametrize("keep,distinct", [([1], 0), ([1, 0], 0)])
def test_a_refused_wait_is_no_success(built, keep, distinct):
    cuda = C.CDLL("libcuda.so.1")
    tab = np.arange(3000, dtype=np.uint32).reshape(-1, 3)
    cols = np.array(keep, np.int32)
    with wk.Context(0) as ctx:
        tin, out = ctx.table(tab), ctx.table(capacity=1 << 16)
        want = tab[:, keep]
        stream, graph = C.c_void_p(ctx.stream()), C.c_void_p()

        def final():
            return wk.lib().wk_table_final_process(ctx.h, tin.h, cols.ctypes.data_as(C.POINTER(C.c_int32)), len(keep),
                                                   distinct, 0, -1, out.h)

        assert final() == wk.SUCCESS and np.array_equal(out.download(), want)   # (the scratch has its size now)
        assert cuda.cuStreamBeginCapture_v2(stream, THREAD_LOCAL) == 0
        rc = final()
        assert cuda.cuStreamEndCapture(stream, C.byref(graph)) != 0             # the refused wait has ended it
        assert rc == wk.E_CUDA
        assert final() == wk.SUCCESS and np.array_equal(out.download(), want)
        tin.free(), out.free()
