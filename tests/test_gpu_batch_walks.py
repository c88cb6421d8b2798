"""A batch's larger pictures, which iterate by walks of their own (batch.cpp): each result is the one
solve() gives the picture alone, bit for bit where that iterates by the same kernels, beside smaller
and one-channel TV pictures that stay batched; more walking pictures than lanes, none batched, and
few iterations."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Rows, columns, colour, method: 2^17 samples or more walk (but one channel of TV).
MIXED = [(384, 352, False, "tgv"), (48, 72, True, "tgv"), (209, 217, True, "tv"), (512, 500, False, "tv"),
         (300, 400, True, "tgv"), (61, 45, False, "tv"), (640, 333, True, "tgv"), (256, 256, True, "tv"),
         (363, 363, False, "tgv")]


def _compare(pictures, iterations):
    from unround import native, synthetic

    images, options = [], []
    for k, (rows, columns, colour, method) in enumerate(pictures):
        make = synthetic.colour if colour else synthetic.grey
        images.append(make(rows, columns, quality=50, seed=k, noise=2).image)
        options.append(["--method", method, "--iterations", str(iterations), "--tolerance", "0", "--record-every", "0"])
    decoded, timing = native.solve_batch(images, options)
    assert timing.iterations == max(iterations - 1, 0)
    for k, (rows, columns, colour, method) in enumerate(pictures):
        alone, made = native.solve(images[k], options[k]), decoded[k]
        if colour or method == "tgv":
            np.testing.assert_array_equal(made.canvas, alone.canvas)
            np.testing.assert_array_equal(made.coefficients[0], alone.coefficients[0])
        else:
            assert np.linalg.norm(made.canvas - alone.canvas) <= 1e-5 * np.linalg.norm(alone.canvas)
        mine, its = made.result.history, alone.result.history
        np.testing.assert_allclose(mine.primal, its.primal, rtol=1e-5)
        np.testing.assert_allclose(mine.dual, its.dual, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("iterations", [1, 2, 3, 60])
def test_mixed(iterations):
    _compare(MIXED, iterations)


@pytest.mark.parametrize("count", [1, 3, 5])
def test_walks_only(count):
    _compare([p for p in MIXED if p[2] and p[0] > 100][:1] * count, 40)
