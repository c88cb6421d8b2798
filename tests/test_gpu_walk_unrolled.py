"""The unrolled solve's walk (walk_unrolled.cu) against the FP64 reference of the same map at the
sizes where it can go wrong: one block, a strip of 64 columns and one more block, several pictures
whose parameters differ, one and several strips of rows, checkpoints that fall on and beside the last
iterate. Six iterations in binary32 move a picture of 0..255 by a few units in the last place of its
samples each: 2e-6 relative."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pictures,rows,columns,every", [(1, 8, 8, 1), (2, 16, 64, 2), (3, 72, 72, 5), (2, 600, 136, 10),
                                                         (5, 40, 1000, 3)])
def test_forward(pictures, rows, columns, every):
    import torch

    from oracle.unrolled_torch import Reference
    from unround import synthetic, unrolled

    images = [synthetic.grey(rows, columns, quality=30, seed=s, noise=2).image for s in range(pictures)]
    problem = unrolled.UnrolledProblem(images, ["--method", "tgv"], iterations=6, checkpoint_every=every)
    values = [torch.linspace(a, b, pictures) for a, b in ((2.0, 0.5), (1.0, 0.3), (problem.tau, 0.8 * problem.tau),
                                                          (problem.sigma, 0.9 * problem.sigma))]
    x, _, _ = problem.forward(*(v.cuda() for v in values))
    expected = Reference(problem).run(*(v.double() for v in values), 6).numpy()
    got = x.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - expected) <= 2e-6 * np.linalg.norm(expected)
