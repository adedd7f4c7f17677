"""The radix sort at the edges of its tiles, digits and tile sizes, against a stable argsort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDE = 148 * 4 * 2048   # keys from which tiles hold 4096 keys instead of 2048


def keys_of(kind, n, bits, rng):
    hi = (1 << bits) - 1
    if kind == "random":
        return rng.integers(0, hi, n, endpoint=True, dtype=np.uint64).astype(np.uint32)
    if kind == "equal":
        return np.full(n, hi, np.uint32)
    run = np.repeat(rng.integers(0, hi, n // 9 + 1, endpoint=True, dtype=np.uint64), 9)[:n]   # runs of equal keys
    return run.astype(np.uint32)


@pytest.mark.parametrize("kind", ["random", "equal", "runs"])
@pytest.mark.parametrize("n,bits", [(1, 1), (31, 4), (2047, 5), (2048, 8), (2049, 9), (6145, 13), (70_001, 17),
                                    (WIDE - 1, 23), (WIDE, 18), (WIDE + 4097, 32), (7_000_003, 24)])
def test_radix_sort_edges(engine, kind, n, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    k = keys_of(kind, n, bits, rng)
    v = rng.permutation(n).astype(np.uint32)
    dk, dv = torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
    torch.cuda.synchronize()
    engine.radix_sort_pairs_device(dk, dv, n, bits)
    engine.sync()
    o = np.argsort(k, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), k[o])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), v[o])
