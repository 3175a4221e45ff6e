"""The binding's pointers hold the arrays they point into."""
import gc
import weakref

import numpy as np

from ib_parallel_gb300 import ibgpu as G


def test_a_pointer_keeps_its_array():
    x = np.arange(24.0).reshape(4, 6)
    copy = np.ascontiguousarray(x[:, ::2])   # what a strided argument becomes
    alive, p = weakref.ref(copy), G._ptr(copy)
    del copy
    gc.collect()
    assert alive() is not None and p.value == alive().ctypes.data
    del p
    gc.collect()
    assert alive() is None
