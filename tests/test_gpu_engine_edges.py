"""The N4 engine on grids, masks and options at the edges of its range, against
the FP64 oracle at the parity bound of the other N4 tests (1e-4 relative,
max|gpu - ref| / max|ref|)."""
import ctypes
import subprocess

import numpy as np
import pytest

import n4_oracle as O
from n4b200.build import nvcc
from n4b200.phantom import make_phantom
from test_gpu_row_ranges import TOL, nrel, run

pytestmark = pytest.mark.gpu

# every word of the shared memory of all SMs, by ordinary stores
FILL = r"""
__global__ void k_fill(int words) {
  extern __shared__ unsigned sm[];
  volatile unsigned *s = sm;
  for (int i = threadIdx.x; i < words; i += blockDim.x) s[i] = 0x7fc00000u;   // NaN
}
extern "C" int fill(int blocks) {
  const int bytes = 227 << 10;
  cudaError_t e = cudaFuncSetAttribute(k_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return (int)e;
  k_fill<<<blocks, 1024, bytes>>>(bytes / 4);
  e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
"""


@pytest.fixture(scope="module")
def fill_shared_memory(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("fill")
    (d / "fill.cu").write_text(FILL)
    so = str(d / "fill.so")
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-shared", "-cudart",
                    "shared", "-o", so, str(d / "fill.cu")], check=True)
    lib = ctypes.CDLL(so)
    blocks = 4 * cuda.cuda.get_device_properties(0).multi_processor_count

    def fill():
        assert lib.fill(blocks) == 0
    return fill


@pytest.mark.parametrize("force", [0, 0x8])
@pytest.mark.parametrize("shape", [(64, 64, 16), (32, 32, 24), (16, 16, 10), (90, 80, 2), (40, 40, 3)])
def test_leftovers_in_shared_memory_do_not_matter(cuda, fill_shared_memory, shape, force):
    """Short rows: the contractions' steps reach past the row's weights.  After
    a kernel that left NaNs in all shared memory, the same bits as before it; the
    first level's denominators come before any histogram, so one iteration of
    one level is compared with the oracle where the volume is large enough for
    that (one voxel in the top bin moves a lattice by about 0.5 / voxels)."""
    im = (np.abs(make_phantom(shape, seed=5, sigma=0.03, grid=4, coeff_std=0.15).im) + 0.3).astype(np.float32)
    fill_shared_memory()
    a = run(cuda, im, None, 3, [2] * 3, flags=force)
    assert a.report["status"] == "N4_OK" and bool(cuda.isfinite(a.lattice).all())
    b = run(cuda, im, None, 3, [2] * 3, flags=force)
    assert cuda.equal(a.lattice, b.lattice) and cuda.equal(a.im_normalized, b.im_normalized)
    if im.size >= 12_000:
        fill_shared_memory()
        c = run(cuda, im, None, 1, [1], flags=force)
        out, lat = O.N4(im, np.ones(shape, np.float32), low_value=0, maximumNumberOfLevels=1,
                        maximumNumberOfIterations=[1], ConvergenceThreshold=0.0)
        assert nrel(c.lattice, lat) < TOL and nrel(c.im_normalized, out) < TOL
