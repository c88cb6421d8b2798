"""A solve that stops at a record ends with it: the iterations launched behind a record before the host
has looked at it are few, however far the next record is. Here the start's record stops it and the next
lies 20,000 iterations on, which take 150 ms and more on the device; making them would be as long as
the solve that does not stop."""

import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,rows,columns", [("tgv", 512, 512), ("tv", 120, 160)])
def test_a_stop_is_not_waited_for(method, rows, columns):
    from unround import native, synthetic

    image = synthetic.grey(rows, columns, quality=40, seed=4).image
    options = ["--method", method, "--iterations", "20000", "--record-every", "20000"]

    def seconds(tolerance: str) -> float:
        took = []
        for _ in range(3):
            at = time.perf_counter()
            out = native.solve(image, [*options, "--tolerance", tolerance])
            took.append(time.perf_counter() - at)
        assert out.result.iterations == (20000 if tolerance == "0" else 0)
        return min(took)

    native.solve(image, [*options, "--tolerance", "1e9"])
    # Unstopped: 20,000 iterations of 3.7 us and more. Stopped: the set-up and the result, 1 to 3 ms.
    assert seconds("1e9") < 0.3 * seconds("0")
