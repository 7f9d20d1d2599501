"""Shots from rows of less than one tile (1 to 7 qubits) are those of the float64 walk over the row, whole
number by whole number: shot counts around a block's, many rows, amplitudes that are zero, targets on and past
the running sums, and rows with infinities and NaN (which end the walk at the last amplitude not zero)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1), (1, 70, 300), (2, 3, 255), (3, 5, 256), (4, 33, 257), (5, 2, 5000), (6, 9, 1000), (7, 4, 40000), (7, 1300, 20)]


@pytest.mark.parametrize("kind", ["dense", "few", "nan", "inf"])
@pytest.mark.parametrize("n,bsz,shots", CASES)
def test_outcomes_are_the_walks(n, bsz, shots, kind):
    from torchquantum_gb300 import _lib

    rng = np.random.default_rng(10 * n + shots)
    dim = 1 << n
    # whole numbers: squares and their sums are exact, so every order of additions gives the same sums
    amp = (rng.integers(-9, 10, size=(bsz, dim)) + 1j * rng.integers(-9, 10, size=(bsz, dim))).astype(np.complex64)
    if kind == "few":
        amp *= rng.random((bsz, dim)) < 2.0 / dim
        amp[:, dim // 2] = 3
    else:
        amp[:, 0] = 1
    prob = amp.real.astype(np.float64) ** 2 + amp.imag.astype(np.float64) ** 2
    if kind in ("nan", "inf"):
        at = int(rng.integers(dim))
        amp[::2, at] = np.nan if kind == "nan" else np.inf
        prob[::2, at] = np.nan if kind == "nan" else np.inf
    cum = prob.cumsum(axis=1)
    u = rng.random((bsz, shots))
    with np.errstate(invalid="ignore"):
        edge = np.take_along_axis(cum, rng.integers(dim, size=(bsz, shots)), 1) / np.where(cum[:, -1:] > 0, cum[:, -1:], 1)
    u = np.where(rng.random((bsz, shots)) < 0.3, np.nan_to_num(edge, nan=0.5, posinf=0.5), u)
    u[:, 0] = 0.0
    u[:, -1] = np.nextafter(1.0, 0.0)
    with np.errstate(invalid="ignore"):
        target = u * cum[:, -1:]
        over = cum[:, None, :] > target[:, :, None] if bsz * shots * dim < 1 << 23 else None
        want = np.empty((bsz, shots), dtype=np.int64)
        for b in range(bsz):
            hit = over[b] if over is not None else cum[b][None, :] > target[b][:, None]
            some = np.flatnonzero(prob[b] > 0)
            want[b] = np.where(hit.any(1), hit.argmax(1), some[-1] if len(some) else 0)
    got = _lib.sample(torch.tensor(amp, device="cuda"), n, torch.tensor(u, device="cuda")).cpu().numpy()
    assert np.array_equal(got, want)
