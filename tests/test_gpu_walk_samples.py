"""The walk of pictures of rounded samples (walk_samples.cu: an iteration as one launch) against the
dual sweep and the primal kernel apart (UNROUND_B200_KERNELS=split): the same operations on the same
operands, so the canvases are equal bit for bit, and so are the records, which both take by the same
kernels. Pictures of odd rows and columns at the edges of its strips (32 columns, 64 with one
channel) and chunks (8 rows), of one row and of one column, of one and several strips of rows; 16
bits; and with records on the way and a tolerance that stops it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _levels(rows, columns, channels, bits):
    rng = np.random.default_rng(rows + columns)
    y, x = np.mgrid[0:rows, 0:columns].astype(np.float64)
    planes = [120 + 60 * np.sin(x / 17 + c) * np.cos(y / 23) + 30 * (x > columns // 2) + rng.normal(0, 2, x.shape)
              for c in range(channels)]
    return np.rint(np.clip(np.stack(planes, -1), 0, 255) * (2**bits - 1) / 255).astype(np.uint16)


def _compare(monkeypatch, levels, bits, options):
    from unround import native

    monkeypatch.delenv("UNROUND_B200_KERNELS", raising=False)
    assert native.measure_samples(levels, bits, options, warmup=1, iterations=3).launches_per_iteration == 1
    walk = native.solve_samples(levels, bits, options)
    monkeypatch.setenv("UNROUND_B200_KERNELS", "split")
    split = native.solve_samples(levels, bits, options)
    np.testing.assert_array_equal(walk.canvas, split.canvas)
    assert walk.result.iterations == split.result.iterations
    np.testing.assert_array_equal(walk.result.history.gap, split.result.history.gap)


@pytest.mark.parametrize("method", ["tv", "tgv"])
@pytest.mark.parametrize("rows,columns,bits", [(128, 257, 8), (65, 511, 16), (1, 32769, 8), (32769, 1, 8), (9, 4095, 8),
                                               (1031, 777, 8), (600, 64, 8)])
def test_grey(monkeypatch, rows, columns, bits, method):
    _compare(monkeypatch, _levels(rows, columns, 1, bits), bits, ["--method", method, "--iterations", "41", "--tolerance", "0"])


@pytest.mark.parametrize("options", [[], ["--channels", "apart", "--channel-weights", "1,0.5,0.75"], ["--mu", "0.05"]])
@pytest.mark.parametrize("method", ["tv", "tgv"])
@pytest.mark.parametrize("rows,columns", [(104, 107), (65, 171), (1, 10925), (10925, 1), (515, 1027), (32, 352)])
def test_colour(monkeypatch, rows, columns, method, options):
    _compare(monkeypatch, _levels(rows, columns, 3, 8), 8,
             ["--method", method, "--iterations", "41", "--tolerance", "0", *options])


@pytest.mark.parametrize("method", ["tv", "tgv"])
def test_records_and_stop(monkeypatch, method):
    levels = _levels(131, 99, 3, 8)
    _compare(monkeypatch, levels, 8, ["--method", method, "--iterations", "50", "--tolerance", "0", "--record-every", "7"])
    _compare(monkeypatch, levels, 8, ["--method", method, "--iterations", "400", "--tolerance", "3", "--record-every", "10"])
