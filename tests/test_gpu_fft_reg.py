"""The register-pencil FFT passes at every kind of extent they are compiled
for (axes of one to four threads, whole and partial blocks, radices 2 to 7),
against numpy's transform in 64 bits; the conjugate-gradient sums that the
inverse xy passes take, against the oracle; the FP32 passes against the FP64
ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from glu_b200 import gfix  # noqa: E402


def _accelerate(f, dims, nd):
    """FFT, times maxp / p^2, FFT back, of f (4, V)."""
    d = dims[:nd]
    k = sum(np.cos(2 * np.pi * np.arange(n) / n).reshape([-1 if a == nd - 1 - i else 1
                                                          for a in range(nd)])
            for i, n in enumerate(d))
    p2 = np.where(np.abs(nd - k) < 1e-14, 1.0, 2 * (nd - k))
    g = f.reshape((4,) + d[::-1])
    ax = tuple(range(1, nd + 1))
    # the library's transforms are unnormalised both ways
    out = np.fft.ifftn(np.fft.fftn(g, axes=ax) * (4.0 * nd / np.prod(d) / p2), axes=ax)
    return (out * np.prod(d)).reshape(4, -1)


@pytest.mark.parametrize("dims", [
    (4, 4, 4, 4), (4, 4, 4, 8), (6, 6, 6, 12), (8, 8, 8, 16), (10, 10, 10, 20), (12, 12, 12, 24),
    (14, 14, 14, 28), (16, 16, 16, 32), (18, 18, 18, 36), (20, 20, 20, 40), (24, 24, 24, 48),
    (28, 28, 28, 28), (28, 28, 28, 56), (30, 30, 30, 60), (32, 32, 32, 32), (32, 32, 32, 64),
    (6, 6, 32, 64), (5, 5, 32, 64), (8, 4, 48, 96), (5, 6, 48, 96),
    (8, 4, 36, 72), (8, 4, 40, 80), (36, 36, 4, 4), (40, 40, 6, 3), (64, 64, 3, 2), (10, 10, 5, 3)])
def test_landau_transform(dims):
    rng = np.random.default_rng(1)
    V = int(np.prod(dims))
    f = rng.normal(size=(4, V)) + 1j * rng.normal(size=(4, V))
    got = gfix.fourier_accelerate(f, dims, 4)
    ref = _accelerate(f, dims, 4)
    # two transforms of log2 V stages, each rounding at 1e-16 of the largest
    assert np.abs(got - ref).max() < 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("dims", [(4, 4, 6), (6, 6, 4), (10, 10, 10), (20, 20, 20), (14, 14, 18),
                                  (24, 24, 10), (28, 28, 30), (32, 32, 21), (32, 32, 32),
                                  (30, 30, 24), (18, 18, 28), (48, 48, 48), (64, 64, 64)])
def test_coulomb_transform(dims):
    rng = np.random.default_rng(2)
    V = int(np.prod(dims))
    f = rng.normal(size=(4, V)) + 1j * rng.normal(size=(4, V))
    got = gfix.fourier_accelerate(f, dims + (2,), 3)
    ref = _accelerate(f, dims, 3)
    assert np.abs(got - ref).max() < 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("dims", [(6, 6, 6, 12), (10, 10, 10, 10), (18, 18, 18, 36),
                                  (20, 20, 20, 40), (36, 36, 36, 36), (40, 40, 40, 80),
                                  (48, 48, 48, 48), (4, 4, 48, 96), (8, 8, 32, 64), (5, 5, 48, 96),
                                  (8, 8, 36, 72), (64, 64, 2, 2)])
def test_fp32_passes_follow_fp64(dims):
    """One steepest-descent step in each phase of a mixed fix (FP32 fields in
    both) against two FP64 ones: links to FP32 rounding of the directions."""
    rng = np.random.default_rng(3)
    V = int(np.prod(dims))
    z = np.eye(3)[None, None, :, :2] + 0.3 * (rng.normal(size=(V, 4, 3, 2))
                                              + 1j * rng.normal(size=(V, 4, 3, 2)))
    c0 = z[..., 0] / np.linalg.norm(z[..., 0], axis=-1, keepdims=True)
    c1 = z[..., 1] - np.sum(np.conj(c0) * z[..., 1], axis=-1, keepdims=True) * c0
    c1 /= np.linalg.norm(c1, axis=-1, keepdims=True)
    U = np.stack([c0, c1, np.conj(np.cross(c0, c1))], axis=-1)
    m = gfix.landau_fix(U, dims, 0.08, 1e-30, 1, "FASD", precision="MIXED").links
    w = gfix.landau_fix(U, dims, 0.08, 1e-30, 2, "FASD").links
    # a step moves the links by O(1); FP32 fields and links round at 6e-8
    # and the transforms multiply that by their log2 V stages
    assert np.abs(m - w).max() < 2e-5
    assert np.linalg.norm(m - w) < 2e-6 * np.linalg.norm(w)


def _links(dims, seed):
    from glu_b200.workload import random_su3
    V = int(np.prod(dims))
    return random_su3(4 * V, np.random.default_rng(seed)).reshape(V, 4, 3, 3)


# planes of every compiled width, in runs of four, two and one to a block, and
# blocks whose last warp is not whole
PLANES = [(n, n, z, t) for n in (4, 6, 10, 14, 18, 20, 28, 30, 32, 36, 40, 48, 64)
          for z, t in ((2, 2), (3, 2), (3, 3))]


@pytest.mark.parametrize("dims", PLANES)
def test_conjugate_gradient_sums(oracle, dims):
    """Three iterations of conjugate gradients: beta comes from the sums that
    the inverse xy passes take of the new and the previous fields, theta and the
    links after them show it."""
    U = _links(dims, 5)
    w = oracle.landau(U, dims, 0.08, 1e-30, 3, "FACG", traj_cap=8)
    r = gfix.landau_fix(U, dims, 0.08, 1e-30, 3, "FACG", traj_cap=8)
    n = len(w["traj_theta"])
    assert n >= 4
    # rounding of the sums and transforms, through four line searches
    assert np.abs(r.traj_theta[:n] / w["traj_theta"] - 1).max() < 1e-11
    assert np.abs(r.links.ravel() - np.asarray(w["links"]).ravel()).max() < 1e-9
    m = gfix.landau_fix(U, dims, 0.08, 1e-30, 3, "FACG", precision="MIXED", traj_cap=8)
    # the same in FP32: 6e-8 of the fields in each of the four
    assert np.abs(m.traj_theta[:n] / w["traj_theta"] - 1).max() < 1e-4


@pytest.mark.parametrize("dims", [(n, n, n, 2) for n in (6, 10, 14, 18, 20, 28, 30, 36, 40, 48)]
                         + [(64, 64, 4, 2), (36, 36, 5, 3), (40, 40, 10, 2), (10, 10, 30, 3)])
def test_coulomb_sums_and_fp32_passes(dims):
    """Smooth slices come to theta < 1e-6 in as many steps by the FP32 passes
    and sums as by the FP64 ones, whose z passes are others (fft_reg.cuh,
    fft_ct.cuh or generic by the extent)."""
    rng = np.random.default_rng(6)
    V = int(np.prod(dims))
    z = 4 * np.eye(3)[:, :2] + rng.normal(size=(V, 4, 3, 2)) + 1j * rng.normal(size=(V, 4, 3, 2))
    c0 = z[..., 0] / np.linalg.norm(z[..., 0], axis=-1, keepdims=True)
    c1 = z[..., 1] - np.sum(np.conj(c0) * z[..., 1], axis=-1, keepdims=True) * c0
    c1 /= np.linalg.norm(c1, axis=-1, keepdims=True)
    U = np.stack([c0, c1, np.conj(np.cross(c0, c1))], axis=-1)
    a = gfix.coulomb_fix(U, dims, 0.08, 1e-6, 200, "FACG")
    b = gfix.coulomb_fix(U, dims, 0.08, 1e-6, 200, "FACG", precision="MIXED", switch_theta=1e-6)
    assert np.all(a.slice_theta < 1e-6) and np.all(b.slice_theta < 1e-6)
    assert 3 * dims[3] < a.iters < 60 * dims[3]
    # rounding moves a theta near the mark past it: a step for each slice
    assert abs(b.iters_fp32 - a.iters) <= dims[3]
