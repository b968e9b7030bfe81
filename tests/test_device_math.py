"""Shading helpers on the CPU (a host build of the device headers): sincos()
gives the bits of sin() and cos(), the texture fetch wraps its texels as the
remainder of each texel's coordinates does, and the tile order names every
pixel once."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "wavefront-path-tracer_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    compiler = shutil.which("g++")
    if compiler is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    out = tmp_path_factory.mktemp("math") / "libmath.so"
    subprocess.run([compiler, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-w", f"-I{CSRC}",
                    f"-I{CUDA_INCLUDE}", "-o", str(out), str(ROOT / "tests" / "device_math_host.cpp")], check=True)
    lib = C.CDLL(str(out))
    lib.sincos_differences.restype = C.c_uint64
    return lib


def test_sincos_is_sin_and_cos(lib):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-10, 10, 200_000), rng.uniform(-8e5, 8e5, 200_000),
                        np.arange(-64, 65) * (np.pi / 4), [0.0, -0.0, 1e-300, np.inf, -np.inf, np.nan]])
    x = np.ascontiguousarray(x, np.float64)
    assert lib.sincos_differences(C.c_void_p(x.ctypes.data), C.c_uint64(len(x))) == 0


@pytest.mark.parametrize("size", [(1, 1), (1, 7), (2, 3), (5, 1), (64, 33)])
def test_texture_fetch_wraps(lib, size):
    """Against the bilinear filter with every texel's own remainder, in the
    same float operations (rows, then columns)."""
    w, h = size
    f = np.float32
    rng = np.random.default_rng(w * 100 + h)
    texels = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    edge = np.linspace(-2, 2, 4 * max(w, h) * 2 + 1)
    uv = np.concatenate([rng.uniform(-3, 3, (500, 2)), rng.uniform(-900, 900, (200, 2)),
                         np.stack([edge, edge[::-1]], 1), [[0, 0], [1, 1], [-1, 1]]]).astype(f)
    got = np.zeros((len(uv), 4), f)
    lib.fetch_texture(C.c_void_p(texels.ctypes.data), C.c_uint32(w), C.c_uint32(h), C.c_void_p(uv.ctypes.data),
                      C.c_uint64(len(uv)), C.c_void_p(got.ctypes.data))
    tx, ty = uv[:, 0] * f(w) - f(0.5), uv[:, 1] * f(h) - f(0.5)
    x, y = np.floor(tx).astype(np.int64), np.floor(ty).astype(np.int64)
    fx, fy = tx - x.astype(f), ty - y.astype(f)
    want = np.zeros_like(got)
    for j in range(2):
        for i in range(2):
            weight = (fx if i else f(1) - fx) * (fy if j else f(1) - fy)
            p = texels[(y + j) % h, (x + i) % w].astype(f) * f(1.0 / 255.0)
            want += weight[:, None] * p
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (8, 4), (9, 5), (3, 40), (40, 3), (64, 32), (65, 33), (250, 131)])
def test_tile_order_names_every_pixel_once(lib, size):
    w, h = size
    xy = np.zeros((w * h, 2), np.uint32)
    lib.tile_pixels(C.c_uint32(w), C.c_uint32(h), C.c_void_p(xy.ctypes.data))
    assert (xy[:, 0] < w).all() and (xy[:, 1] < h).all()
    assert len(np.unique(xy[:, 1].astype(np.int64) * w + xy[:, 0])) == w * h
    for k in range(0, (w // 8 * 8) * (h // 4 * 4), 32):  # whole blocks are 8 x 4
        block = xy[k:k + 32]
        assert (np.ptp(block, axis=0) == (7, 3)).all() and (block[0] % (8, 4) == 0).all()
