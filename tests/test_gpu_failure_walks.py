"""The failure path of the bounded waits in the walks of the unrolled solve and of pictures of samples,
made to run as in test_gpu_failure.py: the dual step's warps are given 0 tries, each CTA gives up at its
first chunk, its copies in flight are waited for, and nothing faults or hangs. Every picture of an unrolled
solve's output, and its gradient of sigma, then has a NaN, wherever in the pass it happened; with the full
limit back both are as before."""

import threading
import time

import numpy as np
import pytest
from test_gpu_failure import _setter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pictures,rows,columns,iterations", [(1, 8, 8, 2), (2, 24, 136, 2), (2, 24, 136, 7), (3, 600, 72, 9)])
def test_the_unrolled_solve_says_so(pictures, rows, columns, iterations):
    import torch

    from unround import synthetic, unrolled

    images = [synthetic.grey(rows, columns, quality=30, seed=s, noise=2).image for s in range(pictures)]
    problem = unrolled.UnrolledProblem(images, ["--method", "tgv"], iterations=iterations, checkpoint_every=4)
    values = [torch.full((pictures,), v, device="cuda") for v in (2.0, 1.0, problem.tau, problem.sigma)]

    def run():
        x, checkpoints, workspace = problem.forward(*values)
        return x.clone(), problem.backward(*values, checkpoints, workspace, 2.0 * (x - 128.0))

    before, grads = run()
    assert torch.isfinite(before).all() and torch.isfinite(grads).all()
    _, checkpoints, workspace = problem.forward(*values)
    set_limit = _setter()
    set_limit(0)
    try:
        failed, _, _ = problem.forward(*values)
        # A forward pass that was whole, and a backward pass whose recomputed walks fail (from two
        # iterations of a segment on: the first is the checkpoint's).
        back = problem.backward(*values, checkpoints, workspace, 2.0 * (before - 128.0))
        torch.cuda.synchronize()
    finally:
        set_limit(-1)
    assert torch.isnan(failed).flatten(1).any(1).all()
    assert torch.isnan(back[3]).all()
    after, again = run()
    assert torch.equal(after, before)
    torch.testing.assert_close(again, grads, rtol=1e-6, atol=0.0)


def test_a_failure_of_the_first_walks_reaches_the_output():
    """The limit is 0 while the first of 40,000 walks are launched and full again for the others: the
    NaN lasts to the output."""
    import torch

    from unround import synthetic, unrolled

    image = synthetic.grey(8, 8, quality=30, seed=5, noise=2).image
    problem = unrolled.UnrolledProblem([image], ["--method", "tgv"], iterations=40000, checkpoint_every=40000)
    values = [torch.full((1,), v, device="cuda") for v in (2.0, 1.0, problem.tau, problem.sigma)]
    before, _, _ = problem.forward(*values)
    torch.cuda.synchronize()
    set_limit = _setter()
    made, ready = [], threading.Event()

    def work():
        problem.forward(*values)  # the thread's first calls take their time
        torch.cuda.synchronize()
        set_limit(0)
        ready.set()
        made.append(problem.forward(*values)[0])

    worker = threading.Thread(target=work)
    try:
        worker.start()
        ready.wait()
        time.sleep(0.02)
        launching = worker.is_alive()
    finally:
        set_limit(-1)
    worker.join()
    assert launching, "every walk was launched within the limit of 0"
    assert torch.isnan(made[0]).any()
    assert torch.equal(problem.forward(*values)[0], before)


@pytest.mark.parametrize("channels,method", [(1, "tv"), (1, "tgv"), (3, "tv"), (3, "tgv")])
def test_a_picture_of_samples_is_an_internal_error(channels, method):
    from unround import native

    rng = np.random.default_rng(3)
    levels = rng.integers(0, 256, (131, 203 if channels == 3 else 301) + ((3,) if channels == 3 else ()), dtype=np.uint8)
    options = ["--method", method, "--iterations", "6", "--tolerance", "0", "--record-every", "0"]
    before = native.solve_samples(levels, 8, options)
    set_limit = _setter()
    set_limit(0)
    try:
        with pytest.raises(native.UnroundError) as raised:
            native.solve_samples(levels, 8, options)
    finally:
        set_limit(-1)
    assert raised.value.status == native.Status.INTERNAL
    np.testing.assert_array_equal(native.solve_samples(levels, 8, options).canvas, before.canvas)
