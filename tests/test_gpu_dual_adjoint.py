"""The dual step's adjoint's tiles (unrolled.cu: 14 rows x 32 columns, what a phase makes put where
the state was) against the FP64 reference's gradients: pictures of less than a tile, of whole tiles,
of whole tiles and a block more, each way, with inner tiles and without.

The tolerance is the other gradient tests' one: the branches of clip and ball at ties within binary32
rounding move a gradient by up to 2e-3 of the parameter's largest."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pictures,rows,columns", [(1, 8, 8), (2, 16, 32), (2, 56, 96), (1, 64, 40), (2, 112, 136),
                                                   (1, 120, 264)])
def test_gradients(pictures, rows, columns):
    import torch

    from oracle.unrolled_torch import Reference
    from unround import synthetic, unrolled

    made = [synthetic.grey(rows, columns, quality=30, seed=s, noise=2) for s in range(pictures)]
    clean = torch.tensor(np.stack([m.samples for m in made]))
    problem = unrolled.UnrolledProblem([m.image for m in made], ["--method", "tgv"], iterations=5, checkpoint_every=2)
    base = [np.linspace(a, b, pictures) for a, b in ((2.0, 0.5), (1.0, 0.3), (problem.tau, 0.8 * problem.tau),
                                                     (problem.sigma, 0.9 * problem.sigma))]
    ours = [torch.tensor(b, dtype=torch.float32, device="cuda", requires_grad=True) for b in base]
    torch.mean((unrolled.unrolled_tgv(problem, *ours).double() - clean.cuda()) ** 2).backward()
    exact = [torch.tensor(b, dtype=torch.float64, requires_grad=True) for b in base]
    torch.mean((Reference(problem).run(*exact, 5) - clean) ** 2).backward()
    for got, expected in zip(ours, exact):
        g, e = got.grad.double().cpu().numpy(), expected.grad.numpy()
        assert np.abs(g - e).max() <= 2e-3 * np.abs(e).max() + 1e-6
