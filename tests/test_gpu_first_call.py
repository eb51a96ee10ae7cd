"""A fresh engine has its streams, events and pinned memory.

They are made with the engine, not in the first call that needs them: a caller that makes an
engine per worker and scores a few regions would pay for them there (one region: 0.98 ms
for the first call, 1.38 when it made them, 0.36 now).  The CUDA runtime calls of each first
call are recorded through CUPTI's callback interface.
"""
import contextlib
import ctypes
import glob
import os
import site

import pytest

from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

RUNTIME_API = 2  # CUPTI_CB_DOMAIN_RUNTIME_API
SETUP = ("cudaStreamCreate", "cudaEventCreate", "cudaMallocHost", "cudaHostAlloc")


class _CallbackData(ctypes.Structure):
    _fields_ = [("site", ctypes.c_int), ("function_name", ctypes.c_char_p)]


def _cupti():
    places = [os.path.join(p, "nvidia", "cuda_cupti", "lib", "libcupti.so*") for p in site.getsitepackages()]
    places.append("/usr/local/cuda/extras/CUPTI/lib64/libcupti.so*")
    for pattern in places:
        for path in sorted(glob.glob(pattern)):
            with contextlib.suppress(OSError):
                return ctypes.CDLL(path)
    pytest.skip("no CUPTI library")


@contextlib.contextmanager
def runtime_calls():
    """Names of the CUDA runtime functions called inside the block."""
    lib, names = _cupti(), []
    kind = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_int, ctypes.c_uint32, ctypes.POINTER(_CallbackData))
    callback = kind(lambda user, domain, cbid, data: names.append(data.contents.function_name.decode()))
    subscriber = ctypes.c_void_p()
    if lib.cuptiSubscribe(ctypes.byref(subscriber), callback, None) != 0:
        pytest.skip("CUPTI takes no subscriber here")
    try:
        assert lib.cuptiEnableDomain(ctypes.c_uint32(1), subscriber, RUNTIME_API) == 0
        yield names
    finally:
        lib.cuptiUnsubscribe(subscriber)


def test_setup_is_done_with_the_engine():
    w = S.single_region()
    pk = native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                       region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)
    params, _ = native.make_params(w.gap, w.ext, False, native.VD_PRECISION_MIXED)
    with runtime_calls() as made:
        native.Engine(0, 1024).close()
    assert any(n.startswith(SETUP) for n in made)  # (they are seen)
    calls = {"forward": lambda e: e.forward(pk, params), "genotypes": lambda e: e.region_genotypes(pk, params),
             "plan": lambda e: e.plan(pk, params).run(), "gradient": lambda e: e.forward_backward(pk, params)}
    for name, call in calls.items():
        eng = native.Engine(0, 1024)
        with runtime_calls() as made:
            call(eng)
        assert made and not [n for n in made if n.startswith(SETUP)], name
        eng.close()
