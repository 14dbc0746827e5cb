"""A batch of more jobs than a call takes is refused before its job array is read or
anything is allocated for it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("njobs", [(1 << 19) + 1, 0xFFFFFFFF])
@pytest.mark.parametrize("flat", [False, True])
def test_too_many_jobs(gi, njobs, flat):
    from gpuintersector import meshgen as mg

    v, t = mg.icosphere(2)
    with gi.Context(0) as c:
        A = c.upload(v, t)
        arr = c._jobs([(A, None, A, None)])
        out, offsets = (ctypes.c_void_p * 1)(), np.zeros(2, dtype=np.int64)
        o = c._opts()
        if flat:
            rc = gi.lib().gi_intersect_batch_flat(c.handle, arr, njobs, ctypes.byref(o),
                                                  offsets.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), out)
        else:
            rc = gi.lib().gi_intersect_batch(c.handle, arr, njobs, ctypes.byref(o), out)
        assert rc == gi._abi.GI_ERR_INVALID_ARG and not out[0]
        assert len(c.intersect_batch_flat([(A, None, A, None)]).pairs) > 0
        A.release()
