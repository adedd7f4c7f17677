"""hr_trace_rays with its arrays in other memory than pageable host memory, at sizes that pass
through the context's staging and above."""
import itertools

import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, Engine
from happyray_b200 import scenes as S

pytestmark = pytest.mark.gpu


def setup(stream=None):
    v, f = S.heightfield(33, seed=1)
    e = Engine(0, stream)
    e.upload(v, v, f, 1.0)
    e.build(GRID_TWO_LEVEL)
    return e


def rays(n, seed):
    rng = np.random.default_rng(seed)
    o = np.concatenate([rng.uniform(0.1, 0.9, (n, 2)), np.ones((n, 1))], 1)
    d = np.concatenate([rng.uniform(0.1, 0.9, (n, 2)), np.zeros((n, 1))], 1) - o
    return o.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def call(e, arrays, n):
    e._chk(e.L.hr_trace_rays(e.ctx, arrays[0].data_ptr(), arrays[1].data_ptr(), n, *[x.data_ptr() for x in arrays[2:]]),
           "trace_rays")


@pytest.mark.parametrize("n", [64, 7000])
@pytest.mark.parametrize("where", [p for p in itertools.product(("pageable", "locked", "device"), repeat=2)])
def test_arrays_in_any_memory(hrlib, n, where):
    """Rays and hits each in pageable, page-locked or device memory."""
    import torch
    e = setup()
    org, d = rays(n, n)
    want = e.trace_rays(org, d)

    def put(a, w):
        t = torch.from_numpy(a.copy())
        return t if w == "pageable" else t.pin_memory() if w == "locked" else t.cuda()
    arrays = [put(org, where[0]), put(d, where[0])] + [put(np.zeros_like(x), where[1]) for x in want]
    torch.cuda.synchronize()
    call(e, arrays, n)
    for got, x in zip(arrays[2:], want):
        assert np.array_equal(got.cpu().numpy(), x)
    e.close()


@pytest.mark.parametrize("n", [64, 7000])
def test_locked_rays_written_by_earlier_work_of_the_stream(hrlib, n):
    """The query's copies follow what its stream does before: here a copy into its ray arrays,
    behind a wait of some milliseconds."""
    import torch
    st = torch.cuda.Stream()
    e = setup(st.cuda_stream)
    org, d = rays(n, n + 1)
    want = e.trace_rays(org, d)
    dev = [torch.from_numpy(x).cuda() for x in (org, d)]
    old = rays(n, n + 2)
    arrays = ([torch.from_numpy(x.copy()).pin_memory() for x in old]
              + [torch.from_numpy(np.zeros_like(x)).pin_memory() for x in want])
    call(e, arrays, n)
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        torch.cuda._sleep(20_000_000)
        for a, x in zip(arrays, dev):
            a.copy_(x, non_blocking=True)
    call(e, arrays, n)
    for got, x in zip(arrays[2:], want):
        assert np.array_equal(got.numpy(), x)
    e.close()
