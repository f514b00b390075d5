"""Configuration generation on the GPU (gfix_heatbath, gfix_overrelax)
against GLU: the over-relaxation value for value (GLU's OR_lattice on the
same links, committed in lat400.npz), the heatbath in distribution (GLU's
average plaquette at beta 6.0 and 5.7, tests/golden/heatbath_glu.json),
plus unitarity, reproducibility and continuation."""
import json
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from glu_b200 import gfix, update  # noqa: E402

GOLD = Path(__file__).resolve().parent / "golden"


def _dims(g):
    return tuple(int(d) for d in g["dims"])


def test_overrelax_matches_glu(lat400):
    U = update.overrelax(lat400["links"], _dims(lat400), 2)
    ref = lat400["or2_links"]
    assert np.abs(U - ref).max() < 1e-12


def test_overrelax_matches_glu_on_heatbath_config(reference, hb8):
    dims = _dims(hb8)
    reference.setup(dims)
    reference.put_links(hb8["links"])
    reference.overrelax(3)
    U = update.overrelax(hb8["links"], dims, 3)
    assert np.abs(U - reference.get_links()).max() < 1e-11


def test_overrelax_keeps_the_action(hb8):
    dims = _dims(hb8)
    p0 = gfix.av_plaquette(hb8["links"], dims)
    U = update.overrelax(hb8["links"], dims, 5)
    assert abs(gfix.av_plaquette(U, dims) - p0) < 1e-13
    assert np.abs(U - hb8["links"]).max() > 0.1  # the links did move


def _binned(x, b):
    n = len(x) // b
    m = np.asarray(x[: n * b]).reshape(n, b).mean(axis=1)
    return m.mean(), m.std(ddof=1) / np.sqrt(n)


@pytest.mark.parametrize("run", json.loads((GOLD / "heatbath_glu.json").read_text())["runs"],
                         ids=lambda r: "beta%.1f" % r["beta"])
def test_heatbath_plaquette_matches_glu(run):
    dims = (8, 8, 8, 8)
    _, p = update.heatbath(update.unit_config(dims), dims, run["beta"],
                           run["therm"] + run["iterations"], run["n_or"], seed=2024)
    mean, err = _binned(p[run["therm"]:], run["bin"])
    sigma = np.hypot(err, run["err"])
    assert abs(mean - run["mean"]) < 5 * sigma, (mean, err, run["mean"], run["err"])


def test_links_stay_in_su3():
    dims = (8, 8, 8, 16)
    U, _ = update.heatbath(update.unit_config(dims), dims, 5.9, 20, 2, seed=3)
    eye = np.eye(3)
    assert np.abs(U @ np.conj(np.swapaxes(U, -1, -2)) - eye).max() < 1e-13
    assert np.abs(np.linalg.det(U) - 1).max() < 1e-13


def test_reproducible_and_continuable():
    dims = (8, 8, 8, 8)
    U0 = update.unit_config(dims)
    a, pa = update.heatbath(U0, dims, 6.0, 10, 1, seed=99)
    b, _ = update.heatbath(U0, dims, 6.0, 6, 1, seed=99)
    b, pb = update.heatbath(b, dims, 6.0, 4, 1, seed=99, first_iteration=6)
    assert np.array_equal(a, b)
    assert pa[-1] == pb[-1]
    c, _ = update.heatbath(U0, dims, 6.0, 10, 1, seed=100)
    assert not np.array_equal(a, c)


def test_device_entry_matches_host_entry():
    dims = (8, 8, 8, 8)
    U0 = update.unit_config(dims)
    a, pa = update.heatbath(U0, dims, 5.8, 5, 2, seed=5)
    d = torch.from_numpy(U0.view(np.float64).reshape(-1).copy()).cuda()
    pd = update.heatbath_device(d, dims, 5.8, 5, 2, seed=5)
    assert np.array_equal(d.cpu().numpy().view(np.complex128).reshape(a.shape), a)
    assert np.array_equal(pa, pd)


def test_odd_extents_are_rejected():
    with pytest.raises(update.UpdateError):
        update.heatbath(update.unit_config((4, 4, 4, 5)), (4, 4, 4, 5), 6.0, 1)


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 4, 2, 2), (10, 6, 4, 6), (8, 8, 8, 16)])
def test_links_outside_su3_keep_all_columns(dims):
    """Links times a common phase are no longer the cross product of their
    first two columns and are kept whole; U S^dag is unchanged by the phase,
    so the over-relaxed links are those of the SU(3) links times the phase."""
    V = int(np.prod(dims))
    rng = np.random.default_rng(5)
    z = 8 * np.eye(3)[:, :2] + rng.normal(size=(V, 4, 3, 2)) + 1j * rng.normal(size=(V, 4, 3, 2))
    c0 = z[..., 0] / np.linalg.norm(z[..., 0], axis=-1, keepdims=True)
    c1 = z[..., 1] - np.sum(np.conj(c0) * z[..., 1], axis=-1, keepdims=True) * c0
    c1 /= np.linalg.norm(c1, axis=-1, keepdims=True)
    U = np.stack([c0, c1, np.conj(np.cross(c0, c1))], axis=-1)
    ph = np.exp(0.3j)
    a = update.overrelax(U, dims, 2)
    b = update.overrelax(ph * U, dims, 2)
    # two sweeps of products and rotations, rounding at 1e-16 each over the
    # size of the subgroups they normalise (links with a common mean keep
    # those of order one; on independent links some are near zero)
    assert np.abs(b - ph * a).max() < 1e-12
    assert np.abs(np.linalg.det(a) - 1).max() < 1e-12


@pytest.mark.parametrize("off", [1e-12, 1e-8, 1e-6, 1e-3])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 4, 2, 2), (8, 8, 8, 8)])
def test_links_off_unitarity_keep_all_columns(dims, off):
    """Links whose first two columns are off unitarity by `off` and whose
    third is the conjugate cross product of these (what a long fix, or a
    reader of 12 rounded reals, leaves): the third column of a product of such
    links is not that of its first two, nor is it after a common phase, which
    U S^dag does not see."""
    V = int(np.prod(dims))
    rng = np.random.default_rng(7)
    z = 8 * np.eye(3)[:, :2] + rng.normal(size=(V, 4, 3, 2)) + 1j * rng.normal(size=(V, 4, 3, 2))
    c0 = z[..., 0] / np.linalg.norm(z[..., 0], axis=-1, keepdims=True)
    c1 = z[..., 1] - np.sum(np.conj(c0) * z[..., 1], axis=-1, keepdims=True) * c0
    c1 /= np.linalg.norm(c1, axis=-1, keepdims=True)
    e = off * rng.normal(size=(3, V, 4, 1))
    c0, c1 = (1 + e[0]) * c0, (1 + e[1]) * c1 + e[2] * c0
    U = np.stack([c0, c1, np.conj(np.cross(c0, c1))], axis=-1)
    ph = np.exp(0.3j)
    a = update.overrelax(U, dims, 2)
    b = update.overrelax(ph * U, dims, 2)
    # rounding at 1e-16 each over the size of the subgroups normalised, as
    # for SU(3) links; products completed from two columns are off by `off`
    assert np.abs(b - ph * a).max() < 1e-13


def test_runs_from_links_outside_su3_continue():
    """A run from links that no column completes goes on where it was left,
    bit for bit, as from SU(3) links."""
    dims = (8, 4, 4, 6)
    U0 = np.exp(0.4j) * update.unit_config(dims)
    a, pa = update.heatbath(U0, dims, 6.0, 4, 1, seed=9)
    b, _ = update.heatbath(U0, dims, 6.0, 1, 1, seed=9)
    b, pb = update.heatbath(b, dims, 6.0, 3, 1, seed=9, first_iteration=1)
    assert np.array_equal(a, b) and pa[-1] == pb[-1]
