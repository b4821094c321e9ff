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


def log_volume(shape, seed):
    return (np.abs(make_phantom(shape, seed=seed, sigma=0.03, grid=4, coeff_std=0.15).im) + 0.3).astype(np.float32)


def thin_rows_and_solid_planes(shape):
    """Rows of two voxels, and two x-planes of whole rows in one CTA's share:
    one CTA of the whole-GPU path has a third of the volume's voxels."""
    m = np.zeros(shape, np.float32)
    m[:, :, 0] = m[:, :, -1] = 1
    m[shape[0] // 2:shape[0] // 2 + 2] = 1
    return m


def hollow_box(shape):
    m = np.zeros(shape, np.float32)
    m[[0, -1]] = 1
    m[:, [0, -1]] = 1
    m[:, :, [0, -1]] = 1
    return m


def one_row(shape, n):
    m = np.zeros(shape, np.float32)
    m[shape[0] // 2, 10:10 + n] = 1
    return m


@pytest.mark.parametrize("shape,mask,levels", [
    ((256, 256, 160), thin_rows_and_solid_planes, 2),
    ((100, 400, 400), hollow_box, 1),
    ((24, 24, 1000), lambda s: one_row(s, 10), 1),
])
def test_masks_that_leave_most_voxels_to_one_cta(cuda, shape, mask, levels):
    """The lattice sums of the whole-GPU path hold the whole volume's terms in
    any one CTA.  (Of 10,000 voxels one more or less in the top bin moves the
    lattice by 5e-5 a step: one iteration there, two on the large masks.)"""
    im, m = log_volume(shape, 5), mask(shape)
    iters = [2] * levels if m.sum() > 20_000 else [1]
    p = run(cuda, im, m, levels, iters, flags=0x8)
    out, lat = O.N4(im, m, low_value=0, maximumNumberOfLevels=levels, maximumNumberOfIterations=iters,
                    ConvergenceThreshold=0.0)
    assert p.report["status"] == "N4_OK" and p.report["path"] == "grid"
    assert nrel(p.lattice, lat) < TOL and nrel(p.im_normalized, out) < TOL


@pytest.mark.parametrize("force", [0x8, 0])
@pytest.mark.parametrize("flags,eps", [(0x2, 1e-3), (0, 0.0), (0, 1e-9)])
def test_control_points_almost_without_voxels(cuda, flags, eps, force):
    """A mask in one corner of one span: the denominators of the far control
    points are 1e-8 to 1e-24 of the largest, and without an epsilon the lattice
    there is a quotient of such sums.  Bound 1e-5: the sums along z are plain
    FP32 over at most 52 voxels of a row, 52 * 2^-24 = 3e-6 for numerator and
    denominator each, the other sums compensated, and one voxel in the top bin
    (174720 voxels) 3e-6."""
    import n4b200
    shape = (128, 120, 112)
    im = log_volume(shape, 5)
    m = np.zeros(shape, np.float32)
    m[2:62, 2:58, 2:54] = 1
    p = n4b200.N4Param(NumberOfFittingLevels=1, MaximumNumberOfIterations=[2], ConvergenceThreshold=0.0, low_value=0.0,
                       flags=flags | force, FitEpsilon=eps)
    res = n4b200.N4(cuda.tensor(im, device="cuda"), cuda.tensor(m, device="cuda"), p)
    out, lat = O.N4(im, m, low_value=0, maximumNumberOfLevels=1, maximumNumberOfIterations=[2],
                    ConvergenceThreshold=0.0, fit_eps=eps, fit_zero_den=bool(flags & 2))
    assert res.report["status"] == "N4_OK"
    assert nrel(res.lattice, lat) < 1e-5 and nrel(res.im_normalized, out) < 1e-5


@pytest.mark.parametrize("shape,nc,levels,bins", [
    ((117, 27, 18), (22, 20, 20), 1, 200),   # 176 KB of lattices in shared memory
    ((90, 60, 24), (7, 6, 4), 4, 32),        # 35 x 27 x 11 control points, 208 KB
])
def test_lattices_that_fill_the_shared_memory(cuda, shape, nc, levels, bins):
    """A lattice beside which the whole-GPU path has no room for its row and
    plane buffers in shared memory runs with them in global memory."""
    import n4b200
    im = log_volume(shape, 5)
    p = n4b200.N4Param(NumberOfFittingLevels=levels, MaximumNumberOfIterations=[2] * levels, ConvergenceThreshold=0.0,
                       low_value=0.0, flags=0x8, NumberOfControlPoints_x=nc[0], NumberOfControlPoints_y=nc[1],
                       NumberOfControlPoints_z=nc[2], NumberOfHistogramBins=bins)
    res = n4b200.N4(cuda.tensor(im, device="cuda"), None, p)
    out, lat = O.N4(im, np.ones(shape, np.float32), low_value=0, maximumNumberOfLevels=levels,
                    maximumNumberOfIterations=[2] * levels, ConvergenceThreshold=0.0, numberOfControlPoints=nc,
                    numberOfHistogramBins=bins)
    assert res.report["status"] == "N4_OK" and res.report["path"] == "grid"
    assert nrel(res.lattice, lat) < TOL and nrel(res.im_normalized, out) < TOL


@pytest.mark.parametrize("shape,levels,k", [((28, 152, 17), 2, 2), ((220, 220, 6), 3, 16), ((320, 320, 1), 1, 16)])
@pytest.mark.parametrize("kind", ["full", "holes"])
def test_forced_clusters_of_short_rows(cuda, shape, levels, k, kind):
    """Volumes of short rows that fit a cluster of the requested size only
    without the list of their rows."""
    im = log_volume(shape, 5)
    m = np.ones(shape, np.float32)
    if kind == "holes":
        m = (np.random.default_rng(7).random(shape) < 0.5).astype(np.float32)
        m[:, 20:25] = 0
        m[3] = 0
    for flags in (k << 8, 0x10) if k == 16 else (k << 8,):
        res = run(cuda, im, m, levels, [2] * levels, flags=flags)
        out, lat = O.N4(im, m, low_value=0, maximumNumberOfLevels=levels, maximumNumberOfIterations=[2] * levels,
                        ConvergenceThreshold=0.0)
        assert res.report["status"] == "N4_OK" and res.report["path"] == "cluster" and res.report["cluster_size"] == k
        assert nrel(res.lattice, lat) < TOL and nrel(res.im_normalized, out) < TOL


@pytest.mark.parametrize("seed", [6, 7])
@pytest.mark.parametrize("force", [0, 0x8])
def test_a_bright_voxel_leaves_the_sums_their_digits(cuda, seed, force):
    """One voxel of 1e12: all others lie in a few of the histogram's bins, and
    the map's values in the bins between, quotients of rounding errors, must not
    set the scale of the whole-GPU path's lattice sums.  Bound 1e-5: FP32 sums
    over at most 56 voxels of a row, 56 * 2^-24 = 3e-6, and one of 98,000 voxels
    in the top bin, 5e-6."""
    shape = (72, 64, 56)
    ph = make_phantom(shape, seed=seed, sigma=0.03, grid=4, coeff_std=0.15)
    im, m = (np.abs(ph.im) + 0.3).astype(np.float32), ph.mask.astype(np.float32)
    im[20, 20, 15] = 1e12
    res = run(cuda, im, m, 1, [1], flags=force)
    _, lat = O.N4(im, m, low_value=0, maximumNumberOfLevels=1, maximumNumberOfIterations=[1], ConvergenceThreshold=0.0)
    assert res.report["status"] == "N4_OK" and nrel(res.lattice, lat) < 1e-5
