"""Solves of different pictures on several threads at once, each on its own stream, iterating by
walks long enough to run beside one another: their results are those of the same solves one after
another, bit for bit."""

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [4, 12])
def test_threads(threads):
    from unround import native, synthetic

    jobs = []
    for k, (rows, columns) in enumerate([(160, 120), (435, 298), (386, 856), (996, 376), (512, 512), (662, 959)]):
        for method in ("tv", "tgv"):
            options = ["--method", method, "--iterations", "600", "--tolerance", "0", "--record-every", "0"]
            grey = k % 2 == 0
            made = (synthetic.grey if grey else synthetic.colour)(rows, columns, quality=50, seed=k, noise=2)
            jobs.append(lambda image=made.image, o=options: native.solve(image, o).canvas)
            if not grey:
                levels = np.rint(np.clip(made.samples, 0, 255)).astype(np.uint16)
                jobs.append(lambda levels=levels, o=options: native.solve_samples(levels, 8, o).canvas)
    alone = [job() for job in jobs]
    with ThreadPoolExecutor(threads) as pool:
        together = list(pool.map(lambda job: job(), [*jobs, *jobs]))
    for k, canvas in enumerate(together):
        np.testing.assert_array_equal(canvas, alone[k % len(alone)])
