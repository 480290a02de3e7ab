"""The tile form's second copies take memory only for the levels that can run
it (fewer than 131,072 cells): of a 352^2 hierarchy all of Q, of a 384^2 one
the quarter below its finest level.  Per byte of Q the former takes 1 - 1/4 more,
whatever else an upload holds per cell."""
import ctypes as C

import pytest

from bsam import ebOptions
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend
from cases import vardc_problem

pytestmark = pytest.mark.gpu


def _pool_bytes():
    cu, pool, n = C.CDLL('libcuda.so.1'), C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(n)) == 0      # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return n.value


def test_no_copy_of_large_levels():
    from bsam.device import DeviceBackend, DevHier
    per = {}
    for n in (352, 384):
        o = ebOptions('BaseCells', n, 'MaxLevels', 1, 'Verbose', 0)
        fl = flatten(build_hierarchy(vardc_problem(), o, OracleBackend()))
        ctx = DeviceBackend.get(0).ctx
        before = _pool_bytes()
        dh = DevHier(ctx, fl, o)
        per[n] = (_pool_bytes() - before) / (8 * fl.Q.size)
        del dh
    assert per[352] - per[384] > 0.6, per
