"""The balls' scale of the walk (csrc/walk.cuh: ball, and ball2 for pairs of samples by fused
multiply-adds) equals sqrtf and the division, bit for bit: on every float of six octaves above the
radius's square for 600 radii, and at radii and squares far from 1, where the norm decides. Compiled
here from the kernels' own header (tests/ball_check.cu).

The unrolled solve takes negative radii too, as its FP64 reference does: beyond the square alpha / |q|,
within it 1."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest
from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    library = tmp_path_factory.mktemp("ball") / "ball_check.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++20", "--expt-relaxed-constexpr",
                    "-Xcompiler", "-fPIC", "-shared", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "jpeg-unround_b200" / "csrc"), str(ROOT / "tests" / "ball_check.cu"), "-o",
                    str(library)], check=True)
    function = ctypes.CDLL(str(library)).ball_check
    function.restype = ctypes.c_longlong
    function.argtypes = [ctypes.c_float, ctypes.c_int, ctypes.c_uint, ctypes.c_uint, ctypes.c_uint]
    return function


def _bits(x: float) -> int:
    return int(np.float32(x).view(np.uint32))


def test_six_octaves_above_600_radii(check):
    rng = np.random.default_rng(7)
    radii = np.exp(rng.uniform(np.log(1e-3), np.log(1e3), 596)).astype(np.float32)
    for radius in [*radii, 1.0, 2.0, 0.5, 255.0]:
        assert check(radius, 0, _bits(np.float32(radius) ** 2 * np.float32(0.99999)), 1, 6 << 23) == 0


@pytest.mark.parametrize("radius", [0.0, 1e-45, 3e-23, 1e-22, 1.1e-20, 3e-19, 9e-13, 1.1e-12, 9e11, 1.1e12, 2e19, 3e38,
                                    float("inf"), float("nan")])
def test_every_square_at_radii_far_from_one(check, radius):
    # 0 to infinity and NaNs, every 127th float; and each subnormal square of the smallest.
    for any_radius in (0, 1) if 1e-12 < radius < 1e12 else (1,):
        assert check(radius, any_radius, 0, 127, 0x7f800100 // 127) == 0
    if radius < 1e-18:
        assert check(radius, 1, 0, 1, 1 << 20) == 0


@pytest.mark.parametrize("method,alpha", [("tv", "3e-23"), ("tgv", "1e-13"), ("tv", "1e13")])
def test_a_solve_at_unusual_radii_takes_the_split_kernels(monkeypatch, method, alpha):
    from unround import native, synthetic

    image = synthetic.grey(64, 160, quality=40, seed=8).image
    options = ["--method", method, "--iterations", "12", "--tolerance", "0"]
    options += ["--alpha", alpha] if method == "tv" else ["--alpha1", alpha, "--alpha0", "1"]
    monkeypatch.delenv("UNROUND_B200_KERNELS", raising=False)
    assert native.measure(image, options, warmup=1, iterations=3)[0].launches_per_iteration == 2
    ours = native.solve(image, options)
    monkeypatch.setenv("UNROUND_B200_KERNELS", "split")
    np.testing.assert_array_equal(ours.canvas, native.solve(image, options).canvas)


def test_the_unrolled_solve_at_negative_radii():
    import torch

    from oracle.unrolled_torch import Reference
    from unround import synthetic, unrolled

    images = [synthetic.grey(24, 72, quality=30, seed=s, noise=2).image for s in range(2)]
    problem = unrolled.UnrolledProblem(images, ["--method", "tgv"], iterations=6, checkpoint_every=3)
    values = [torch.tensor(v) for v in ([-2.0, 1.5], [1.0, -0.7], [problem.tau] * 2, [problem.sigma] * 2)]
    x, _, _ = problem.forward(*(v.cuda() for v in values))
    expected = Reference(problem).run(*(v.double() for v in values), 6).numpy()
    got = x.cpu().numpy().astype(np.float64)
    # As test_gpu_walk_unrolled's: six iterations in binary32.
    assert np.linalg.norm(got - expected) <= 2e-6 * np.linalg.norm(expected)
