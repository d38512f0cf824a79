"""The fast kernels (a sweep by a cluster of blocks per row, a finishing kernel) against the CPU oracle
at the sizes where their decomposition changes: units of 512 logits, blocks of 16 and 32 units,
one to sixteen blocks per row, rows that start on any address, and rows whose sum behaves badly
(masked, constant, sorted, powers of two, far from zero)."""
import numpy as np
import pytest
import torch

from executorch_b200 import Sampler, seeds_to_states
from executorch_b200 import workloads as W

from parity import THREADS, to_device

pytestmark = pytest.mark.gpu


def _payload(x, dtype):
    if dtype == "fp32":
        return x.astype(np.float32)
    return W.f32_to_bf16_bits(x) if dtype == "bf16" else x.astype(np.float16).view(np.uint16)


def _check(restatement, x, dtype, device, settings):
    rows, vocab = x.shape
    seeds = np.arange(rows, dtype=np.uint64) * 7919 + 3
    t = to_device(x, dtype, device)
    for temperature, topp, topk in settings:
        s = Sampler(vocab, temperature, topp, 0, device=device)
        try:
            s.set_topk(topk)
            states = seeds_to_states(seeds, device)
            got = s.sample_rows(t, states).cpu().numpy()
            assert s.status == 0
        finally:
            s.close()
        want, want_states = restatement.sample_rows(x, temperature, topp, seeds, dtype=dtype, topk=topk,
                                                    threads=THREADS, return_states=True)
        assert np.array_equal(got, want), (dtype, vocab, temperature, topp, topk, np.nonzero(got != want)[0][:8])
        assert np.array_equal(states.cpu().numpy().view(np.uint64), want_states)


@pytest.mark.parametrize("dtype", ["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("vocab", [256, 511, 513, 8191, 8193, 16385, 32769, 131073, 200001, 262137, 262138])
def test_sizes(cuda_device, restatement, dtype, vocab):
    rng = np.random.default_rng(vocab)
    x = _payload(3.0 * rng.standard_normal((5, vocab)), dtype)  # an odd vocabulary: rows on any address
    _check(restatement, x, dtype, cuda_device, [(0.8, 0.9, 0), (0.7, 1.0, 0), (1.0, 0.5, 20)])


@pytest.mark.parametrize("dtype", ["bf16", "fp16", "fp32"])
def test_sums_that_behave_badly(cuda_device, restatement, dtype):
    rng = np.random.default_rng(5)
    vocab = 30011
    base = 3.0 * rng.standard_normal(vocab)
    masked = np.where(np.arange(vocab) < vocab // 2, -np.inf, base)
    rows = [masked, np.where(rng.random(vocab) < 0.99, -np.inf, base), np.zeros(vocab), np.sort(base), -np.sort(-base),
            base + 100.0, base - 3000.0, 20.0 * base, 0.6931472 * rng.integers(0, 12, vocab), np.round(2.0 * base)]
    _check(restatement, _payload(np.stack(rows), dtype), dtype, cuda_device,
           [(1.0, 0.9, 0), (0.8, 1.0, 0), (0.9, 0.7, 50)])
