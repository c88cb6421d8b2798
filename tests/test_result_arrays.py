"""The result's arrays in Python (native._Copies, native._Block): copies in parts over several
arrays of odd sizes, blocks given back only when the last view of them goes, and an array kept
through a fork and in another thread."""

import gc
import os
import threading

import numpy as np
import pytest

from unround import native


def _pointer(array):
    return array.ctypes.data_as(native.ctypes.POINTER(native.ctypes.c_double))


@pytest.mark.parametrize("shapes", [[(1,)], [(3, 5), (0, 4), (257, 1025)], [(7,), (1, 2, 3), (3, 700, 1001), (131072,)]])
def test_copies(shapes):
    library = native._library()
    rng = np.random.default_rng(0)
    sources = [rng.normal(size=shape) for shape in shapes]
    copies = native._Copies(library)
    made = [copies.of(_pointer(s), s.shape) for s in sources]
    copies.run()
    for a, b in zip(made, sources):
        np.testing.assert_array_equal(a, b)
        assert a.flags.writeable and a.flags.c_contiguous


def test_a_block_lives_as_long_as_a_view_of_it():
    library = native._library()
    whole = native._empty(library, (300, 1000))
    whole[:] = 1.0
    part, at = whole[10:20], whole.ctypes.data
    del whole
    gc.collect()
    other = native._empty(library, (300, 1000))
    other[:] = 2.0
    assert other.ctypes.data != at
    assert (part == 1.0).all()
    worker = threading.Thread(target=lambda: native._empty(library, (200, 1000)).fill(0.0))
    worker.start()
    worker.join()
    child = os.fork()
    if child == 0:
        os._exit(0 if (part == 1.0).all() and (other == 2.0).all() else 1)
    assert os.waitpid(child, 0)[1] == 0


def test_missing_values_are_refused():
    copies = native._Copies(native._library())
    with pytest.raises(RuntimeError):
        copies.of(native.ctypes.POINTER(native.ctypes.c_double)(), (2, 2))
