"""The device memory of a solve is no more than it was with one buffer of x~: 28 binary32 planes for
TGV (two states of 8, their tilde duals 7, x~ twice, v, and div_2 of r~ twice) and 11 for TV (two states
of 3, the duals 2, x~ twice, v), the canvas and the coefficients in binary64, zeta in binary32 and the
levels of 16 bits. Of samples: no coefficients and zeta, levels twice. 2% more for the sums and tables."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["grey", "colour"])
@pytest.mark.parametrize("method,planes", [("tgv", 28), ("tv", 11)])
def test_of_a_jpeg_file(kind, method, planes):
    from unround import native, synthetic

    image = getattr(synthetic, kind)(1024, 1024, quality=60, seed=2).image
    timing = native.measure(image, ["--method", method], warmup=1, iterations=3)
    timing = timing[0] if isinstance(timing, tuple) else timing
    coefficients = sum(c.coefficients.size for c in image.components)
    assert timing.launches_per_iteration == 1
    assert timing.device_bytes <= 1.02 * (timing.samples * (4 * planes + 8) + 14 * coefficients)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("method,planes", [("tgv", 28), ("tv", 11)])
def test_of_samples(channels, method, planes):
    from unround import native

    levels = np.random.default_rng(1).integers(0, 256, (1024, 1024, channels), dtype=np.uint16)
    timing = native.measure_samples(levels if channels > 1 else levels[..., 0], 8, ["--method", method], warmup=1,
                                    iterations=3)
    assert timing.launches_per_iteration == 1
    assert timing.device_bytes <= 1.02 * timing.samples * (4 * planes + 8 + 4)
