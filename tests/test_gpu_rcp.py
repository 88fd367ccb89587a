"""The optimiser's reciprocal against quotients, over the exponents of normal
numbers whose reciprocals are normal."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("part", ["exponents", "near powers of two"])
def test_reciprocal_is_within_an_ulp(pkg, dev, part):
    L = C.CDLL(os.path.join(os.path.dirname(pkg.__file__), "lib", "libntgb300_probe.so"))
    L.ntgprobe_rcp.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong, C.c_void_p]
    rng, e = np.random.default_rng(5), np.arange(-1021, 1022)
    if part == "exponents":
        m = rng.uniform(1.0, 2.0, (e.size, 2000))
    else:
        k = np.arange(-500, 500)
        m = 1.0 + np.where(k < 0, k * 2.0 ** -53, k * 2.0 ** -52)[None, :] * np.ones((e.size, 1))
    x = np.ldexp(m, e[:, None]).ravel()
    x = np.concatenate([x, -x])
    x = x[(abs(x) >= 2.0 ** -1021) & (abs(x) <= 2.0 ** 1021)]
    xd = torch.from_numpy(x).to(dev)
    y = torch.empty_like(xd)
    assert L.ntgprobe_rcp(xd.data_ptr(), y.data_ptr(), x.size, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    # y x - 1: the last FMA's rounding 2^-53, the third power of an approximation within 2^-19, the
    # rounding of its correction 2^-72
    err = y.cpu().numpy().astype(np.longdouble) * x.astype(np.longdouble) - 1
    assert np.all(abs(err) <= np.longdouble(2.0) ** -53 * (1 + np.longdouble(2.0) ** -3))
