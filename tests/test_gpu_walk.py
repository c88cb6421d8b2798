"""The walk (walk.cuh: an iteration as one launch, keeping nothing or one of its steps' values)
against the dual sweep and the primal kernels apart (UNROUND_B200_KERNELS=split): the same
operations on the same operands, so the canvases and coefficients are equal bit for bit; the
records' sums are of the same terms in another order (binary64: within 1e-12). Sizes at the edges of its strips (32
columns, 64 with one channel), chunks (8 rows), bands (8 or 16) and of one and several strips of
rows; every cell layout it takes and one it leaves to the others; radii whose projections go by
its packed square root and quotient, and by the library's (far from 1)."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(image, options, split):
    from unround import native

    if split:
        os.environ["UNROUND_B200_KERNELS"] = "split"
    try:
        return native.solve(image, options)
    finally:
        os.environ.pop("UNROUND_B200_KERNELS", None)


GREY = [(8, 8), (8, 64), (16, 72), (24, 56), (61, 45), (600, 136), (72, 1000), (1031, 777)]
COLOUR = [(16, 16), (17, 33), (32, 32), (61, 77), (560, 112), (515, 1027)]
RADII = [("1", "2"), ("0.3", "0.7"), ("3", "5.5"), ("1e-14", "1e13")]


@pytest.mark.parametrize("method", ["tv", "tgv"])
@pytest.mark.parametrize("rows,columns", GREY)
def test_grey(rows, columns, method):
    from unround import synthetic

    _compare(synthetic.grey(rows, columns, quality=40, seed=rows, noise=2).image, ["--method", method])


@pytest.mark.parametrize("coupling", ["coupled", "apart"])
@pytest.mark.parametrize("sampling", [(1, 1), (1, 2), (2, 1), (2, 2), (4, 1)])
@pytest.mark.parametrize("method", ["tv", "tgv"])
def test_cells(method, sampling, coupling):
    from unround import synthetic

    image = synthetic.colour(61, 77, quality=75, seed=8, noise=3, sampling=sampling).image
    _compare(image, ["--method", method, "--channels", coupling, "--channel-weights", "1,0.5,0.75"])


@pytest.mark.parametrize("method", ["tv", "tgv"])
@pytest.mark.parametrize("rows,columns", COLOUR)
def test_colour(rows, columns, method):
    from unround import synthetic

    _compare(synthetic.colour(rows, columns, quality=60, seed=columns, noise=3).image, ["--method", method])


@pytest.mark.parametrize("alpha1,alpha0", RADII)
def test_radii_and_general_map(alpha1, alpha0):
    from unround import synthetic

    image = synthetic.colour(48, 80, quality=50, seed=5, noise=3).image
    given = ["--method", "tgv", "--alpha1", alpha1, "--alpha0", alpha0]
    _compare(image, given)
    _compare(image, [*given, "--centres", "mmse", "--slack", "0.5", "--slack-cost", "3"])


@pytest.mark.parametrize("method", ["tv", "tgv"])
def test_flat_fields(method):
    # Around a detail in a flat picture the duals fall off into the subnormal range.
    from unround import jpegio, synthetic

    for made in (synthetic.grey(256, 512, quality=50, seed=1), synthetic.colour(256, 512, quality=50, seed=1)):
        parts = []
        for c in made.image.components:
            levels = np.zeros_like(c.coefficients)
            levels[3:5, 3:6] = c.coefficients[3:5, 3:6]
            parts.append((levels, c.quant_table, c.h_samp_factor, c.v_samp_factor))
        image = jpegio.image_of(256, 512, made.image.color_space, parts)
        _compare(image, ["--method", method], 200)


def _compare(image, options, iterations=60):
    # 24 iterations between records: eager ones, graphs of eight, and the kept ones between; or none
    # between, one and a few, where a record's two launches meet the next one's.
    for every, count in ((25, iterations), (1, 4), (2, 7), (3, 11)):
        _compare_every(image, [*options, "--iterations", str(count), "--tolerance", "0", "--record-every", str(every)])


def _compare_every(image, options):
    walk, split = _solve(image, options, False), _solve(image, options, True)
    np.testing.assert_array_equal(walk.canvas, split.canvas)
    for a, b in zip(walk.coefficients, split.coefficients):
        np.testing.assert_array_equal(a, b)
    a, b = walk.result.history, split.result.history
    np.testing.assert_array_equal(a.iterations, b.iterations)
    np.testing.assert_array_equal(a.scaling, b.scaling)
    scale = np.abs(b.primal).max() + np.abs(b.dual).max()
    for name in ("primal", "dual", "partial_gap"):
        np.testing.assert_allclose(getattr(a, name), getattr(b, name), rtol=1e-12, atol=1e-12 * scale)


def test_partial_gap():
    from unround import synthetic

    image = synthetic.colour(61, 77, quality=75, seed=8, noise=3).image
    _compare(image, ["--method", "tgv", "--partial-radius", "3"])


@pytest.mark.parametrize("every", ["1", "2", "7", "10"])
@pytest.mark.parametrize("method,tolerance", [("tv", "0.02"), ("tgv", "0.2"), ("tgv", "1e9")])
def test_a_stop(method, tolerance, every):
    # The iterations that follow a record on the stream before it is looked at leave the result alone.
    from unround import synthetic

    image = synthetic.colour(96, 80, quality=75, seed=4, noise=2).image
    options = ["--method", method, "--tolerance", tolerance, "--iterations", "400", "--record-every", every]
    walk, split = _solve(image, options, False), _solve(image, options, True)
    assert walk.result.iterations == split.result.iterations < 400
    assert walk.result.stop == split.result.stop
    assert len(walk.result.history.iterations) == len(split.result.history.iterations)
    np.testing.assert_array_equal(walk.canvas, split.canvas)
    assert (np.diff(walk.result.history.seconds) >= 0).all()
