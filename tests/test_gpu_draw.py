"""Shots drawn by a warp each: every search depth over the tiles, states with one, few and all
amplitudes non-zero (also far from normalised), uniforms at random and on the edges between
outcomes (where float32 sums cannot tell them apart); and the means over the shots of Z-type
strings.

An outcome is right if the target lies in its interval of the float64 running sums, up to 1e-12
of the total (their own rounding), and its amplitude is not zero."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bsz,shots", [(1, 1, 5), (7, 3, 33), (8, 2, 64), (9, 1, 1), (13, 2, 257), (14, 1, 500),
                                         (18, 2, 300)])
@pytest.mark.parametrize("kind", ["dense", "few", "one", "tiny", "skewed"])
def test_draws_lie_in_their_intervals(n, bsz, shots, kind):
    from torchquantum_gb300 import _lib

    rng = np.random.default_rng(n + shots)
    dim = 1 << n
    amp = rng.normal(size=(bsz, dim)) + 1j * rng.normal(size=(bsz, dim))
    if kind == "one":
        amp *= np.arange(dim) == rng.integers(dim)
    elif kind == "few":
        amp *= rng.random((bsz, dim)) < 3.0 / dim
        amp[:, rng.integers(dim)] = 1.0
    elif kind == "tiny":
        amp *= 1e-21
    elif kind == "skewed":
        amp *= 10.0 ** rng.uniform(-12, 0, size=(1, dim))
    amp = amp.astype(np.complex64)
    prob = amp.real.astype(np.float64) ** 2 + amp.imag.astype(np.float64) ** 2
    cum = prob.cumsum(axis=1)
    u = rng.random((bsz, shots))
    if dim > 2:  # a third on the edges
        edge = rng.integers(dim, size=(bsz, shots))
        u = np.where(rng.random((bsz, shots)) < 0.33, np.take_along_axis(cum / cum[:, -1:], edge, 1), u)
    u = np.minimum(u, 1.0 - 2.0 ** -53)
    got = _lib.sample(torch.tensor(amp, device="cuda"), n, torch.tensor(u, device="cuda")).cpu().numpy()
    assert got.min() >= 0 and got.max() < dim
    assert (np.take_along_axis(prob, got, 1) > 0).all()
    target, tol = u * cum[:, -1:], 1e-12 * cum[:, -1:]
    assert (np.take_along_axis(cum, got, 1) > target - tol).all()
    assert (np.take_along_axis(cum - prob, got, 1) <= target + tol).all()


@pytest.mark.parametrize("bsz,shots,m", [(1, 1, 1), (3, 255, 5), (2, 1000, 33)])
def test_parity_means(bsz, shots, m):
    from torchquantum_gb300 import _lib

    rng = np.random.default_rng(m)
    idx, masks = rng.integers(1 << 30, size=(bsz, shots)), [int(v) for v in rng.integers(1 << 30, size=m)]
    got = _lib.sample_parity(torch.tensor(idx, device="cuda"), masks).cpu().numpy()
    for j, mask in enumerate(masks):
        odd = np.array([[bin(int(v) & mask).count("1") & 1 for v in row] for row in idx])
        want = torch.tensor(1.0 - 2.0 * odd, dtype=torch.float64, device="cuda").mean(dim=1).to(torch.float32)
        assert (got[j] == want.cpu().numpy()).all()
