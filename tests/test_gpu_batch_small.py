"""Batches of many small circuits: the launch shapes with 8 CTAs an SM against numpy (tolerance of
test_gpu_batch_sweeps.py), far more circuits than CTAs, and the autotuner offers those shapes where every
circuit is small."""
import numpy as np
import pytest
import torch

from tests import test_gpu_batch_sweeps as sweeps


def test_small_circuits_may_run_in_many_ctas():
    from torchquantum_gb300 import autotune as A

    for n in (1, 5, 9, 11):
        assert max(c.ctas_per_sm for c in A.batch_candidates(n)) == 8
    assert all(c.tile_bits <= 11 for c in A.batch_candidates(11))


@pytest.mark.gpu
@pytest.mark.parametrize("config", [(10, 128, 8), (11, 128, 8), (10, 128, 4), (11, 128, 5)])
def test_every_width(config):
    sweeps.test_sweeps_match_numpy(config)


@pytest.mark.gpu
@pytest.mark.parametrize("config", [(10, 128, 8), (11, 128, 8), "auto"])
def test_many_circuits(config, tmp_path, monkeypatch):
    from torchquantum_gb300 import autotune as A
    from torchquantum_gb300 import batch as B

    monkeypatch.setenv("TQ_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    A.clear()
    rng = np.random.default_rng(3)
    kinds = [sweeps._random_ir(rng, n, count) for n, count in ((1, 3), (3, 20), (4, 41), (5, 9), (7, 30), (9, 25), (10, 60))]
    widths = [1, 3, 4, 5, 7, 9, 10]
    want = [sweeps._simulate(n, *ir) for n, ir in zip(widths, kinds)]
    cb = B.CircuitBatch()
    for i in range(2100):
        cb.add_ops(widths[i % 7], *kinds[i % 7])
    res = cb.run(torch.device("cuda", 0), return_states=True, config=config if config == "auto" else B.BatchConfig(*config))
    for i in list(range(14)) + list(range(1000, 1014)) + list(range(2086, 2100)):
        assert np.linalg.norm(res.states[i].cpu().numpy() - want[i % 7]) <= 4 * 2.0 ** -24 * max(1, len(kinds[i % 7][0]))
    z = np.array([[(abs(s[:len(s) // 2]) ** 2).sum() - (abs(s[len(s) // 2:]) ** 2).sum()] for s in want])[:, 0]
    assert np.abs(np.asarray(res.z) - z[np.arange(2100) % 7]).max() <= 8 * 2.0 ** -24 * 60
