"""Edges of the row-range engine and of the component kernels that choose
their path by size and alignment, against the FP64 oracle.

Tolerances: 1e-4 relative (max|gpu - ref| / max|ref|) for N4 runs, the bound of
the other parity tests.  The volumes hold at least 30,000 masked voxels where
iterations are compared: one voxel more or less in the histogram's top bin
(where an ulp decides) moves a lattice by about 0.5 / voxels.  1e-5 for fits and
1e-6 for sharpened values, as in the component tests; kernels that differ only
in how they load agree bitwise.
"""
import numpy as np
import pytest

import n4_oracle as O
from n4b200.phantom import make_phantom

TOL = 1e-4


def nrel(a, b):
    a = a.detach().cpu().numpy() if hasattr(a, "detach") else np.asarray(a)
    return float(np.abs(a.astype(np.float64) - b).max() / max(np.abs(b).max(), 1e-30))


# ------------------------------------------------------------------ the partition of the whole-GPU path, on the CPU
def partition(lens, K, Z):
    """Rows of each CTA as the whole-GPU path deals them out: even shares'
    weights first, then the first row whose preceding weight reaches the
    CTA's part of the total."""
    c = max(Z // 8, 16)
    w = np.where(lens > 0, lens + c, 0).astype(np.int64)
    n = w.size
    cut = [n * k // K for k in range(K + 1)]
    prefix = [0]
    for k in range(K):
        prefix.append(prefix[-1] + int(w[cut[k]:cut[k + 1]].sum()))

    def boundary(target):
        k = max(q for q in range(K) if prefix[q] <= target)
        run = prefix[k]
        for i in range(cut[k], cut[k + 1]):
            if run >= target:
                return i
            run += int(w[i])
        return cut[k + 1]

    b = [boundary(prefix[K] * r // K) for r in range(K)] + [n]
    rows_bound = (n * (Z + c) // K + Z + c) // (1 + c) + 2
    voxels_bound = n * (Z + c) // K + 2 * (Z + c)
    return b, w, c, rows_bound, voxels_bound


@pytest.mark.parametrize("seed", range(6))
def test_partition_covers_every_row_once_within_its_buffers(seed):
    rng = np.random.default_rng(seed)
    Z = int(rng.choice([1, 5, 60, 181, 700]))
    n, K = int(rng.integers(3, 4000)), 148
    lens = rng.integers(0, Z + 1, n)
    if seed % 3 == 1:
        lens[rng.random(n) < 0.95] = 0
    if seed % 3 == 2:
        lens = np.where(rng.random(n) < 0.5, 1, Z)   # short rows beside full ones
    b, w, c, rows_bound, voxels_bound = partition(lens, K, Z)
    assert b[0] == 0 or not w[:b[0]].any()
    assert all(x <= y for x, y in zip(b, b[1:]))
    for r in range(K):
        part = lens[b[r]:b[r + 1]]
        assert (part > 0).sum() <= rows_bound and part.sum() <= voxels_bound


# ------------------------------------------------------------------ the engine
def run(cuda, im, mask, levels, iters, nc=(4, 4, 4), flags=0):
    import n4b200
    p = n4b200.N4Param(NumberOfFittingLevels=levels, MaximumNumberOfIterations=list(iters), ConvergenceThreshold=0.0,
                       low_value=0.0, flags=flags, NumberOfControlPoints_x=nc[0], NumberOfControlPoints_y=nc[1],
                       NumberOfControlPoints_z=nc[2])
    return n4b200.N4(cuda.tensor(im, device="cuda"), None if mask is None else cuda.tensor(mask, device="cuda"), p)


def check(cuda, im, mask, levels, iters, nc=(4, 4, 4), flags=0):
    res = run(cuda, im, mask, levels, iters, nc, flags)
    ones = np.ones(im.shape, np.float32)
    out, lat = O.N4(im, ones if mask is None else mask, low_value=0, maximumNumberOfLevels=levels,
                    maximumNumberOfIterations=list(iters), ConvergenceThreshold=0.0, numberOfControlPoints=nc)
    assert res.report["status"] == "N4_OK"
    assert nrel(res.lattice, lat) < TOL
    assert nrel(res.im_normalized, out) < TOL
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("force", [0, 0x8])
@pytest.mark.parametrize("shape,nc,levels", [
    ((96, 88, 9), (4, 4, 4), 2),      # rows shorter than the lanes that share one
    ((60, 40, 64), (4, 4, 4), 3),     # 8 lanes per row in the histogram, 4 spans
    ((60, 40, 65), (4, 5, 6), 2),     # 16 lanes per row, 6 spans
    ((44, 30, 257), (4, 4, 12), 1),   # 32 lanes per row, 9 spans: two span rounds of 8 lanes do not do
    ((50, 30, 90), (4, 4, 41), 1),    # 38 spans: more than a warp
])
def test_row_lengths_and_spans(cuda, shape, nc, levels, force):
    ph = make_phantom(shape, seed=21, sigma=0.03, grid=4, coeff_std=0.15)
    check(cuda, ph.im, np.ones(shape, np.float32) if shape[2] == 9 else ph.mask, levels, [2] * levels, nc, force)


@pytest.mark.gpu
@pytest.mark.parametrize("force", [0, 0x8])
@pytest.mark.parametrize("kind", ["holes", "stripes", "sparse", "one_row_planes", "none"])
def test_masks(cuda, kind, force):
    """Rows with holes, empty rows between others, single voxels, planes of one
    row, no mask."""
    shape = (72, 64, 56)
    ph = make_phantom(shape, seed=22, sigma=0.03, grid=4, coeff_std=0.15)
    rng = np.random.default_rng(22)
    im = np.abs(ph.im) + 0.3
    m = np.ones(shape, np.float32)
    if kind == "holes":
        m = (rng.random(shape) < 0.3).astype(np.float32)
    elif kind == "stripes":
        m[:, 10:30] = 0
        m[:, 33] = 0
        m[::5] = 0
        m[:, :, 20:24] = 0
    elif kind == "sparse":
        m = (rng.random(shape) < 0.13).astype(np.float32)
        m[:, rng.random(64) < 0.3] = 0
        m[40:] = (rng.random((32, 64, 56)) < 0.3)
    elif kind == "one_row_planes":
        m[:48, :50] = 0
        m[:48, 51:] = 0
    check(cuda, im.astype(np.float32), None if kind == "none" else m, 2, [2, 2], (4, 4, 4), force)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,nc", [
    ((168, 170, 168), (4, 4, 4)),    # more voxels per CTA than its shared memory holds
    ((560, 540, 8), (4, 4, 4)),      # row list and row sums beyond their shared memory
    ((900, 6, 60), (5, 11, 11)),     # a CTA's planes in several rounds of T2
    ((60, 70, 150), (4, 40, 40)),    # a plane's sums beyond T2's shared memory
])
def test_whole_gpu_path_beyond_shared_memory(cuda, shape, nc):
    ph = make_phantom(shape, seed=23, sigma=0.03, grid=4, coeff_std=0.15)
    res = check(cuda, (np.abs(ph.im) + 0.2).astype(np.float32), None, 1, [2], nc, 0x8)
    assert res.report["path"] == "grid"


@pytest.mark.gpu
def test_threads_do_not_change_the_result(cuda):
    """512 and more threads per CTA take the rows in other groups, the sums in
    the same order."""
    ph = make_phantom((64, 60, 50), seed=24, sigma=0.03, grid=4, coeff_std=0.15)
    a = run(cuda, ph.im, ph.mask, 3, [6] * 3, flags=0x8)
    b = run(cuda, ph.im, ph.mask, 3, [6] * 3, flags=0x8 | 0x2000)
    assert cuda.equal(a.lattice, b.lattice)


# ------------------------------------------------------------------ components
@pytest.mark.gpu
@pytest.mark.parametrize("shape,nc", [((40, 30, 181), (6, 5, 7)), ((33, 21, 7), (5, 4, 4)), ((21, 17, 1), (4, 4, 4)),
                                      ((12, 9, 1023), (4, 5, 12)), ((16, 12, 30), (5, 6, 40))])
def test_fit_rows_at_any_alignment(cuda, shape, nc):
    """Rows that start anywhere: register steps from the boundary before them
    (field and mask off it alike), or the staged kernel (off it differently),
    bitwise the same, with and without a mask."""
    import n4b200
    rng = np.random.default_rng(31)
    n = int(np.prod(shape))
    f = rng.normal(0, 0.3, n).astype(np.float32)
    m = (rng.random(n) < 0.6).astype(np.float32)
    f[(m == 0) & (rng.random(n) < 0.05)] = np.nan
    lats = []
    for fo, mo in ((0, 0), (3, 3), (7, 7), (1, 2)):
        fb, mb = cuda.full((n + 8,), float("nan"), device="cuda"), cuda.ones(n + 8, device="cuda")
        fb[fo:fo + n] = cuda.tensor(f, device="cuda")
        mb[mo:mo + n] = cuda.tensor(m, device="cuda")
        lats.append(n4b200.FitBspline3D(fb[fo:fo + n].view(shape), mb[mo:mo + n].view(shape), nc))
    for lat in lats[1:]:
        assert cuda.equal(lats[0], lat)
    ref = O.FitBspline3D(np.where(m == 0, 0.0, f).reshape(shape).astype(np.float64), m.reshape(shape), nc)
    assert nrel(lats[0], ref) < 1e-5
    f = np.nan_to_num(f)
    full = n4b200.FitBspline3D(cuda.tensor(f, device="cuda").view(shape), None, nc)
    assert nrel(full, O.FitBspline3D(f.reshape(shape).astype(np.float64), np.ones(shape), nc)) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("n,bins", [(1, 200), (3, 64), (4099, 2), (30_001, 1024), (700_003, 200)])
@pytest.mark.parametrize("off", [0, 1])
def test_sharpen_sizes_and_alignment(cuda, n, bins, off):
    """Voxel counts that leave a remainder, pointers off the 16-byte boundary,
    the fewest and the most bins; NaNs outside the mask are not read."""
    import n4b200
    rng = np.random.default_rng(n + bins)
    x = (rng.choice([-1.0, -0.35, 0.0], n) + rng.normal(0, 0.06, n)).astype(np.float32)
    m = (rng.random(n) < 0.5).astype(np.float32)
    m[0] = 1.0
    xb, mb = cuda.empty(n + 4, device="cuda"), cuda.empty(n + 4, device="cuda")
    xb[off:off + n] = cuda.tensor(np.where(m != 0, x, np.nan).astype(np.float32), device="cuda")
    mb[off:off + n] = cuda.tensor(m, device="cuda")
    out = n4b200.sharpenImage(xb[off:off + n], mb[off:off + n], bins, 0.01, 0.15).cpu().numpy()
    assert np.all(out[m == 0] == 0.0)
    if n == 1:
        assert out[0] == x[0]
        return
    if (m != 0).sum() < 2:
        pytest.skip("one masked voxel has no bin range")
    ref = O.sharpenImage(x.astype(np.float64), m, bins, 0.01, 0.15)
    assert nrel(out, ref) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 3, 11])
def test_encoder_gradients_of_ragged_batches(cuda, batch):
    """Batches whose rows do not fill the tiles of the data gradient's parity
    classes, against the FP64 reference at the bound of the encoder tests."""
    import encoder_ref as R
    from n4b200.encoder import Encoder
    rng = np.random.default_rng(batch)
    enc = Encoder(max_batch=batch, seed=5)
    x = R.bf16(rng.normal(-0.5, 0.4, (batch, 32, 32, 24)))
    t = rng.normal(0, 0.2, (batch, 64)).astype(np.float32)
    enc.train_step(cuda.tensor(x, dtype=cuda.bfloat16, device="cuda"), cuda.tensor(t, device="cuda"), 0.0)
    got = enc.grads().astype(np.float64)
    ref, _ = R.backward(enc.params(), x, t)
    at = 0
    from n4b200.encoder import layer_shapes
    for name, shape in layer_shapes():
        k = int(np.prod(shape))
        g, r = got[at:at + k], ref[at:at + k]
        assert np.abs(g - r).max() <= 2e-2 * np.abs(r).max(), name
        at += k


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(40, 30, 4), (40, 30, 44), (20, 30, 92), (20, 30, 108), (12, 9, 1020)])
def test_fit_rows_on_16_byte_boundaries(cuda, shape):
    """Rows of 4 k voxels, k odd: steps of 4 voxels or of 8 from any offset, by
    their length; bitwise the same as off the boundary, and the oracle's."""
    import n4b200
    rng = np.random.default_rng(33)
    n, nc = int(np.prod(shape)), (5, 4, 6)
    f, m = rng.normal(0, 0.3, n).astype(np.float32), (rng.random(n) < 0.6).astype(np.float32)
    lats = []
    for off in (0, 4, 1):
        fb, mb = cuda.zeros(n + 8, device="cuda"), cuda.zeros(n + 8, device="cuda")
        fb[off:off + n], mb[off:off + n] = cuda.tensor(f, device="cuda"), cuda.tensor(m, device="cuda")
        lats.append(n4b200.FitBspline3D(fb[off:off + n].view(shape), mb[off:off + n].view(shape), nc))
    assert cuda.equal(lats[0], lats[1]) and cuda.equal(lats[0], lats[2])
    assert nrel(lats[0], O.FitBspline3D(f.reshape(shape).astype(np.float64), m.reshape(shape), nc)) < 1e-5
