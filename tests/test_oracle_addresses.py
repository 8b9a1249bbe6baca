"""The oracle's single-step entry points on arrays anywhere in the address space."""

import ctypes
import mmap

import numpy as np

N = 1024


def _mapped(value, dtype=np.float32):
    """An array in a mapping of its own, far above 4 GB."""
    a = np.frombuffer(mmap.mmap(-1, 4 * N), dtype=dtype)
    a[:] = value
    return a


def test_single_steps_take_high_addresses(oracle_mod):
    L = oracle_mod.lib()
    p, m, v, bias = (_mapped(0.0) for _ in range(4))
    g, d = _mapped(1.0), _mapped(1, np.int32)
    assert min(a.ctypes.data for a in (p, m, v, g, d, bias)) >= 1 << 32
    n = ctypes.c_int64(N)
    L.oracle_sgd_f32(p.ctypes.data, g.ctypes.data, n, ctypes.c_float(2.0), ctypes.c_int64(4))
    assert np.all(p == -0.5)
    L.oracle_adam_f32(p.ctypes.data, g.ctypes.data, m.ctypes.data, v.ctypes.data, n, ctypes.c_int64(1),
                      ctypes.c_float(1.0), ctypes.c_int64(1))
    assert np.all(m > 0.09) and np.all(v > 0.0009) and np.all(p < -1.4)
    p[:] = 2.0  # past one: the delay rolls on
    L.oracle_roll_delays_f32(p.ctypes.data, d.ctypes.data, n)
    assert np.all(d == d[0])
    L.oracle_adam_bias_f32(ctypes.c_int64(1), bias.ctypes.data)
    assert abs(bias[0] - 0.1) < 1e-6 and abs(bias[1] - 0.001) < 1e-6
