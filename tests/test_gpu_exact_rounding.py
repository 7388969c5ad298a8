"""Values that the reference evaluates in double and the kernels in pairs of
floats: bit for bit the double expression's, over every float that the pairs
take (ACES, the sRGB power) and every random number of a camera ray.  The
device functions are called directly, from a test kernel built over them."""
import ctypes as C
import subprocess

import pytest

from eleven import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "post.cu"
#include "shade.cuh"
using namespace er;
template <typename F>
__global__ void k_differ(uint64_t lo, uint64_t hi, unsigned long long* n, F differs) {
  unsigned c = 0;
  for (uint64_t i = lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < hi; i += (uint64_t)gridDim.x * blockDim.x)
    c += differs((uint32_t)i);
  if (c) atomicAdd(n, (unsigned long long)c);
}
template <typename F>
static long long count(uint64_t lo, uint64_t hi, F differs) {
  unsigned long long* n = nullptr;
  unsigned long long h = 0;
  if (cudaMalloc(&n, 8) != cudaSuccess) return -1;
  cudaMemset(n, 0, 8);
  k_differ<<<1216, 256>>>(lo, hi, n, differs);
  const cudaError_t e = cudaMemcpy(&h, n, 8, cudaMemcpyDeviceToHost);
  cudaFree(n);
  return e == cudaSuccess ? (long long)h : -1;
}
struct Root {
  __device__ unsigned operator()(uint32_t i) const {
    const float x = __uint_as_float(i);
    return __float_as_uint(root22(x)) != __float_as_uint(root22_exact(x));
  }
};
struct Aces {
  __device__ unsigned operator()(uint32_t i) const {
    const float x = __uint_as_float(i);
    return __float_as_uint(aces(x)) != __float_as_uint(aces_exact(x));
  }
};
struct Offset {
  int32_t res;
  float h, l, size;
  __device__ unsigned operator()(uint32_t i) const {
    const float r = (float)i * 0x1p-24f;
    return __float_as_uint(pixel_offset(r, res, h, l, size)) != __float_as_uint(pixel_offset_exact(r, res, size));
  }
};
extern "C" long long differ_root22(uint64_t lo, uint64_t hi) { return count(lo, hi, Root{}); }
extern "C" long long differ_aces(uint64_t lo, uint64_t hi) { return count(lo, hi, Aces{}); }
extern "C" long long differ_offset(int32_t res, float size) {
  er_camera c{};
  c.x_res = c.y_res = res;
  const DevCamera d = make_dev_camera(c);
  return count(0, 1u << 24, Offset{res, d.px_h, d.px_l, size});
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    build.build_product()
    d = tmp_path_factory.mktemp("rounding")
    (d / "r.cu").write_text(SRC)
    subprocess.run([build.NVCC, *build.CU_FLAGS, *build.ARCH, "-shared", str(d / "r.cu"), "-o", str(d / "r.so"),
                    "-L" + build.PKG_ROOT, "-leleven", "-lcudart", "-Xlinker", "-rpath", "-Xlinker", build.PKG_ROOT],
                   check=True)
    L = C.CDLL(str(d / "r.so"))
    L.differ_root22.argtypes = L.differ_aces.argtypes = [C.c_uint64, C.c_uint64]
    L.differ_offset.argtypes = [C.c_int32, C.c_float]
    L.differ_root22.restype = L.differ_aces.restype = L.differ_offset.restype = C.c_longlong
    return L


def _bits(e):
    return (e + 127) << 23


def test_srgb_power_of_every_float(lib):
    """The pairs' range 2^-60 .. 2^16 and two powers of two beyond, negatives included."""
    assert lib.differ_root22(_bits(-62), _bits(18)) == 0
    assert lib.differ_root22(0x80000000, 0x80000000 + (1 << 22)) == 0


def test_aces_of_every_float(lib):
    assert lib.differ_aces(_bits(-32), _bits(32)) == 0


SIZES = [0.035, 0.0196875, 36.0, 24.0, -0.035, 1e-20, 2.0 ** -78, 1e-30, 0.0, 3e20, 1e37]


@pytest.mark.parametrize("res", [1, 2, 3, 7, 320, 479, 641, 1080, 1920, 4095, 16_777_217, 1 << 28])
def test_camera_offsets_of_every_random_number(lib, res):
    assert [lib.differ_offset(res, s) for s in SIZES] == [0] * len(SIZES)
