"""The proposal's kernels at the edges of their 32-sample tiles and of the table's 256-cell blocks.

Tolerance 2e-5 of the norm: two layers of sums of 96 and 64 products, each rounded at 6e-8, and the activations' few ulp
give at most 2 (96 + 64) 6e-8."""

import importlib

import numpy as np
import pytest

from raspa3_b200 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


# 32,768 and 32,769 samples are 1,024 and 1,025 tiles: partial sums in shared scratch and in the network's own
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 4097, 32768, 32769])
def test_batches_against_fp64(ctx, n):
    torch = pytest.importorskip("torch")
    mo = importlib.import_module("oracle.mlp")
    m = native.Mlp(ctx, seed=n)
    theta = m.params().astype(np.float64)
    rng = np.random.default_rng(n)
    s = rng.random((n, 3)).astype(np.float32)
    t = (3.0 * rng.normal(size=n)).astype(np.float32)
    ds, dt = torch.from_numpy(s).cuda(), torch.from_numpy(t).cuda()
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    m.evaluate(ds.data_ptr(), n, out.data_ptr())
    loss, grad = m.loss_and_gradient(ds.data_ptr(), dt.data_ptr(), n)
    f = mo.forward(theta, s.astype(np.float64))
    assert np.linalg.norm(out.cpu().numpy() - f) <= 2e-5 * max(1.0, np.linalg.norm(f))
    ref, g = mo.loss_and_grad(theta, s.astype(np.float64), t.astype(np.float64))
    assert abs(loss - ref) <= 2e-5 * ref
    assert np.linalg.norm(grad - g) <= 2e-5 * np.linalg.norm(g)


@pytest.mark.parametrize("cells", [1, 2, 7, 33])
def test_table_against_fp64(ctx, cells):
    mo = importlib.import_module("oracle.mlp")
    m = native.Mlp(ctx, seed=cells)
    p = native.Proposal(m, cells_per_axis=cells, eps_uniform=0.2)
    g = (np.arange(cells) + 0.5) / cells
    k, j, i = np.meshgrid(g, g, g, indexing="ij")
    s = np.stack([i, j, k], -1).reshape(-1, 3)
    f = mo.forward(m.params().astype(np.float64), s.astype(np.float32).astype(np.float64))
    w = np.exp(f - f.max())
    ref = 0.8 * len(w) * w / w.sum() + 0.2
    q = p.density(s)
    # the density is a normalised exponential of f: its relative error is f's absolute error
    assert np.max(np.abs(q / ref - 1.0)) <= 4e-5 * max(1.0, np.abs(f).max())
    assert abs(q.mean() - 1.0) <= 1e-12
    p.close()
