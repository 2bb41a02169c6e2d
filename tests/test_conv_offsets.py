"""Where the convolution GEMMs' operands lie, on the host: offsets of tensors
with fewer and with more than 2^31 elements against exact integers."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def offsets(tmp_path_factory):
    cc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cc):
        pytest.skip("nvcc is missing")
    exe = str(tmp_path_factory.mktemp("conv") / "conv_offsets")
    subprocess.run([cc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "gpuvmem_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "conv_offsets.cu"), "-o", exe], check=True)

    def run(cases):
        text = "\n".join(" ".join(map(str, c)) for c in cases)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


@pytest.mark.parametrize("B,C,c0,H,W", [
    (3, 5, 2, 24, 40),
    (11, 48, 32, 2048, 2048),    # 2^31 elements within the eleventh image
    (43, 48, 32, 1024, 1024),
    (33, 64, 0, 1024, 1024),
    (1, 600, 599, 2048, 2048),   # within one image
    (2040, 256, 255, 1024, 1024),
])
def test_pixels_and_rows(offsets, B, C, c0, H, W):
    pixels = [0, 1, W, H * W - 1, H * W, B * H * W // 2 + 7, B * H * W - W - 1, B * H * W - 1]
    pixels = [m for m in pixels if 0 <= m < B * H * W]
    cases = [(op, C, c0, H, W, m) for op in "xyzw" for m in pixels]
    want = []
    for _, _, _, _, _, m in cases:
        b, r = divmod(m, H * W)
        want.append((((b * C + c0) * H + r // W) * W + r % W, r // W, r % W, b))
    assert offsets(cases) == want
