"""A network call that runs out of device memory reports it, gives back what it had taken, and leaves the
next call alone."""
import ctypes as C

import numpy as np
import pytest
import torch

from imex_sflow2d_v2_b200.solver import ImexError, ImexMLP

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("call", ["predict", "loss_grad", "train"])
def test_out_of_memory_gives_the_first_buffer_back(call):
    net = ImexMLP(seed=2)
    x = np.random.default_rng(1).normal(size=(64, 12)).astype(np.float32)
    want = net.predict(x)
    hog = []
    while _free() > 400 * MB:                    # leave 300 to 400 MB
        hog.append(torch.empty(max(MB, min(_free() - 320 * MB, 1 << 36)), dtype=torch.uint8, device="cuda"))
    free = _free()
    # 48 bytes a row for x fit, the 8 bytes a row for y (or 8 for the order, 48, 8) no longer do
    n = int(free / 52) if call != "train" else int(free / 60)
    big = np.zeros((n, 12), np.float32)
    small = torch.zeros(64, device="cuda")
    before = _free()
    with pytest.raises(ImexError):
        if call == "predict":
            net.predict(big)
        elif call == "loss_grad":
            net.loss_grad(big, np.zeros((n, 2), np.float32))
        else:
            # fails before the pointers are used
            net.train(C.c_void_p(small.data_ptr()), C.c_void_p(small.data_ptr()), n, epochs=1)
    assert abs(_free() - before) <= 8 * MB
    np.testing.assert_array_equal(net.predict(x), want)
    del hog, small
    torch.cuda.empty_cache()
    net.close()
