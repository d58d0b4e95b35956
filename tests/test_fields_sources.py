"""Fields from host arrays, device arrays and both in one call, in either layout:
the stored fields, seen through a step, are the same bits."""
import ctypes as C

import numpy as np
import pytest

from conftest import cuda_available
from helpers import STATE_KEYS, bitwise_equal, small_case
from ntlp_b200 import abi
from ntlp_b200 import generator as gen

ORDER = ("u", "v", "w", "T", "q")


@pytest.mark.parametrize("precision", [abi.NTLP_PREC_FP64, abi.NTLP_PREC_MIXED])
@pytest.mark.parametrize("layout", ["ext", "flow"])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_host_and_device_arrays_in_one_call(layout, precision):
    import torch
    import ntlp_b200
    params = dict(gen.default_params(icase=0), precision=precision)
    case = small_case(params=params, n=2000, grid_n=(9, 7, 11))
    if layout == "ext":
        fields = case.ext()
    else:
        fields = {k: np.ascontiguousarray(np.asarray(v).transpose(2, 1, 0)) for k, v in case.fields.items()}
    other = {k: np.random.default_rng(5).random(v.shape) + 300.0 for k, v in fields.items()}
    ref = None
    for where in ("hhhhh", "ddddd", "hdhdh", "dhddd", "hhhhd", "dddhh"):
        s = ntlp_b200.DropletStep(case.grid, params, capacity=2000)
        upload = s.L.ntlp_fields_upload_ext if layout == "ext" else s.L.ntlp_fields_upload
        for given in (other, fields):            # the second call replaces every value of the first
            keep = [torch.from_numpy(np.ascontiguousarray(given[k])) for k in ORDER]
            keep = [a.cuda() if w == "d" else a for a, w in zip(keep, where)]
            torch.cuda.synchronize()
            assert upload(s.h, *(C.cast(a.data_ptr(), C.POINTER(C.c_double)) for a in keep)) == 0
            s.sync()
        s.set_droplets(case.droplets)
        s.particle_update_BE(case.dt, 2)
        got = s.get_droplets()
        s.close()
        ref = ref or got
        for k in STATE_KEYS:
            assert bitwise_equal(got[k], ref[k]), (where, k)
    if layout == "flow":                          # and the two layouts agree
        s = ntlp_b200.DropletStep(case.grid, params, capacity=2000)
        s.set_fields_ext(case.ext())
        s.set_droplets(case.droplets)
        s.particle_update_BE(case.dt, 2)
        got = s.get_droplets()
        s.close()
        for k in STATE_KEYS:
            assert bitwise_equal(got[k], ref[k]), k
