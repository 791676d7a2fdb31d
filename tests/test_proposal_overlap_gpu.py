"""Training kernels that start while the one before them ends: a run of many steps gives the parameters, bit for bit, of
single steps with a wait after each."""

import numpy as np
import pytest

from raspa3_b200 import native

pytestmark = pytest.mark.gpu


# one tile, tiles that leave SMs free for the next kernel's start, and more tiles than SMs
@pytest.mark.parametrize("batch,steps", [(32, 400), (1024, 300), (4096, 200), (16384, 60)])
def test_overlapped_steps(batch, steps):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(batch)
    s = torch.from_numpy(rng.random((20000, 3)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(size=20000).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    ctx = native.Context(0)
    one, many = native.Mlp(ctx, seed=2), native.Mlp(ctx, seed=2)
    loss = many.train(s.data_ptr(), t.data_ptr(), 20000, steps, batch=batch, seed=7)
    for _ in range(steps):
        last = one.train(s.data_ptr(), t.data_ptr(), 20000, 1, batch=batch, seed=7)
    assert loss == last
    assert np.array_equal(one.params(), many.params())
    ctx.close()
