"""A tensor-core convolution whose bounded wait ran out: every entry point of
the network reports it, the training step before its update.  The wait is not
made to run out; its flag on the device is set from here."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from ekman_bl_gb300.duct import EkError
from oracle.unet_ref import init_params

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EK_ERR_TIMEOUT = 5


class Int32At:
    def __init__(self, ptr):
        self.__cuda_array_interface__ = {"shape": (1,), "typestr": "<i4", "data": (ptr, False), "version": 2}


@pytest.fixture(scope="module")
def flag_of(tmp_path_factory):
    import torch
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no g++ or no CUDA headers")
    so = tmp_path_factory.mktemp("native") / "unet_flag.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ekman_bl_gb300", "csrc"),
                    "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "native", "unet_flag.cpp"),
                    "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.unet_timeout_flag.argtypes, lib.unet_timeout_flag.restype = [C.c_void_p], C.c_void_p
    return lambda net: torch.as_tensor(Int32At(lib.unet_timeout_flag(net.handle)), device="cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("channels", [16, 32])
def test_timeout_is_reported_before_the_update(flag_of, channels):
    import torch
    from ekman_bl_gb300.duct import UNet
    n, h, w = 2, 16, 24
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.standard_normal((n, h, w, 2)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal((n, h, w)).astype(np.float32)).cuda()
    y = torch.zeros((n, h, w), device="cuda")
    p0 = init_params(2, channels, 0).astype(np.float32)
    net = UNet(2, channels, n, h, w)
    net.set_params(p0)
    flag = flag_of(net)
    assert int(flag.item()) == 0
    net.gradient(x.data_ptr(), t.data_ptr(), n, h, w)
    flag.fill_(1)
    torch.cuda.synchronize()
    for call in (lambda: net.forward(x.data_ptr(), n, y.data_ptr()),
                 lambda: net.gradient(x.data_ptr(), t.data_ptr(), n, h, w),
                 lambda: net.train_step(x.data_ptr(), t.data_ptr(), n, h, w, 1e-2)):
        with pytest.raises(EkError) as e:
            call()
        assert e.value.code == EK_ERR_TIMEOUT
    assert np.array_equal(net.get_params(), p0)
    # without the tensor-core kernels no wait has run out
    net.set_tcgen05(False)
    net.gradient(x.data_ptr(), t.data_ptr(), n, h, w)
    net.set_tcgen05(True)
    # the first update is Adam's first: its moments and its step count are as
    # if the refused one had not been asked for (every weight with a gradient
    # moves by the rate)
    flag.fill_(0)
    torch.cuda.synchronize()
    net.train_step(x.data_ptr(), t.data_ptr(), n, h, w, 1e-2)
    d = np.abs(net.get_params() - p0)
    assert np.median(d[d > 0]) == pytest.approx(1e-2, rel=1e-3) and d.max() <= 1.001e-2
