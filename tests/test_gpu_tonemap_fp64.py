"""The tonemap of the reference's arithmetic (precise=False) against the same kernel
text with every pixel's power in FP64, bit for bit: every density magnitude, zero,
negative and non-finite channels, gammas on both sides of the pair's range, and images
with more open pixels than a block sets aside."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import build
from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu

FORMATS = {lr.HALF3: (3, torch.float16), lr.HALF4: (4, torch.float16), lr.FLOAT3: (3, torch.float32), lr.FLOAT4: (4, torch.float32)}


@pytest.fixture(scope="module")
def fp64(tmp_path_factory):
    so = tmp_path_factory.mktemp("tonemap") / "fp64.so"
    subprocess.run([str(build.CUDA / "bin" / "nvcc"), build.ARCH, "-O3", "-std=c++17", *build.CUDA_SOURCES["tonemap_fast.cu"],
                    "-DRFK_TONEMAP_FP64", "-Xcompiler", "-fPIC", "-shared", "-cudart", "shared", str(build.CSRC / "kernels" / "tonemap_fast.cu"),
                    "-o", str(so)], check=True)
    f = C.CDLL(str(so)).rfk_launch_tonemap_fast
    f.argtypes = [C.c_void_p, C.c_uint, C.c_void_p, C.c_int] + [C.c_float] * 5 + [C.c_void_p] * 3 + [C.c_double, C.c_uint, C.c_uint,
                                                                                                     C.c_void_p]
    return f


def _bins(w, h, kind):
    rng = np.random.default_rng(w)
    d = np.exp2(rng.uniform(-40.0, 40.0, size=(h, w))).astype(np.float32)
    if kind == "counts":
        d = rng.poisson(30.0, size=(h, w)).astype(np.float32)
    if kind == "faint":
        d[:] = 1e-30  # log(1 + x) is 0 in FP32: the power of 0
    bins = np.concatenate([rng.uniform(0, 1, size=(h, w, 3)) * d[..., None], d[..., None]], -1).astype(np.float32)
    if kind == "odd":
        flat = bins.reshape(-1)
        flat[rng.integers(0, flat.size, 400)] = np.inf
        flat[rng.integers(0, flat.size, 400)] = np.nan
        flat[rng.integers(0, flat.size, 400)] = 0.0
        flat[rng.integers(0, flat.size, 400)] = -0.0
        flat[rng.integers(0, flat.size, 400)] *= -1.0
        flat[rng.integers(0, flat.size, 400)] = 1e-42
    return bins


@pytest.mark.parametrize("kind,w,h", [("all", 61, 67), ("counts", 640, 360), ("odd", 67, 61), ("faint", 1100, 1000)])
@pytest.mark.parametrize("gamma", [0.3, 0.5, 1.0, 2.2, 4.0])
def test_fast_variant_is_the_fp64_one_bit_for_bit(fp64, kind, w, h, gamma):
    bins = torch.from_numpy(_bins(w, h, kind)).cuda()
    quality, brightness = 64.0, 4.0
    libm = C.CDLL("libm.so.6")  # the host's constant, in single precision
    libm.powf.argtypes, libm.log10f.argtypes = [C.c_float] * 2, [C.c_float]
    libm.powf.restype = libm.log10f.restype = C.c_float
    scale = libm.powf(10.0, float(np.float32(-libm.log10f(quality)) - np.float32(0.5)))
    for fmt, (c, dt) in FORMATS.items():
        for vib, hp in ((1.0, -1.0), (0.4, 1.0)):
            out, want = (torch.full((h, w, c), 7.0, device="cuda", dtype=dt) for _ in range(2))
            hist, whist = (torch.zeros(lr.HISTOGRAM_BINS, device="cuda", dtype=torch.int64) for _ in range(2))
            top, wtop = (torch.zeros(1, device="cuda", dtype=torch.int64) for _ in range(2))
            lr.tonemapper().run(bins, out, (w, h), quality, gamma, brightness, vib, highlight_power=hp, fmt=fmt, precise=False,
                                histogram=hist, max_density_out=top)
            assert fp64(bins.data_ptr(), w * h, want.data_ptr(), fmt, gamma, scale, brightness, vib, hp, whist.data_ptr(),
                        wtop.data_ptr(), None, 0.0, (w * h + 255) // 256, 152, None) == 0
            torch.cuda.synchronize()
            bits = torch.int16 if dt == torch.float16 else torch.int32
            assert torch.equal(out.view(bits), want.view(bits)), (fmt, vib)
            assert torch.equal(hist, whist) and torch.equal(top, wtop)
