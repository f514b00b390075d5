"""The register-pencil FFT passes at every kind of extent they are compiled
for (axes of one to four threads, whole and partial blocks, radices 2 to 7),
against numpy's transform in 64 bits."""
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
