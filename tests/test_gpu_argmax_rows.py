"""Greedy rows shared by a cluster of blocks: sizes around the vectors and slices, rows that start off
16-byte boundaries, equal maxima, and the edge rules of a sequential scan (sampler.cpp:44-56)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def scan(x):
    """Lowest index of the maximum; a NaN never replaces, and is never replaced in element 0."""
    if np.isnan(x[0]):
        return 0
    return int(np.argmax(np.where(np.isnan(x), -np.inf, x)))


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("rows,vocab", [(1, 1), (3, 7), (5, 17), (2, 4097), (9, 16384), (1, 65537), (3, 131071),
                                        (64, 50257), (300, 33001), (700, 8191), (1300, 4100)])
def test_argmax_rows(dtype, rows, vocab):
    from executorch_b200 import Sampler
    rng = np.random.default_rng(rows * vocab)
    x = torch.from_numpy(np.round(rng.standard_normal((rows, vocab)), 1).astype(np.float32)).to(DTYPES[dtype])
    x[0, :] = -float("inf")
    if rows > 2:
        x[1, 0] = float("nan")
        x[2, vocab // 2] = float("nan")
        x[2, vocab - 1] = 30.0
    want = [scan(r) for r in x.float().numpy()]
    s = Sampler(vocab, 0.0, 0.9, 0, device=torch.device("cuda", 0))
    flat = torch.empty(rows * vocab + 1, dtype=x.dtype, device="cuda")
    for offset in (0, 1):  # with and without rows on 16-byte boundaries
        dev = flat[offset:offset + rows * vocab].view(rows, vocab)
        dev.copy_(x)
        got = s.sample_rows(dev, None if rows == 1 else torch.ones(rows, dtype=torch.int64, device="cuda"))
        assert got.cpu().tolist() == want
    s.close()
