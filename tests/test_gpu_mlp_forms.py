"""The warm start's kernels at the edges of their row tiles (GPU).

loss_grad: batches of one tile, batches that 512 does not divide (one split of the rows, its
last piece shorter), and one large enough for 128 rows per CTA (64 below 19,456 rows), against the
FP64 restatement with the same bfloat16 rounding; what is left is FP32 accumulation order, the
2e-3 of test_gpu_mlp.py.  infer: cell counts that no tile divides, below and above that size.
"""
import numpy as np
import pytest

from bes_gb300 import lib, meshgen
from oracle import mlp_oracle as M
from tests.test_gpu_mlp import _blocks, _ctx

pytestmark = pytest.mark.gpu


def _net(ctx, seed):
    net = lib.WarmStart(ctx, seed=seed)
    rng = np.random.default_rng(seed)
    blocks = _blocks(net.params().astype(np.float64))
    for l in range(4):
        blocks[f"F{l}"][:] = rng.normal(size=blocks[f"F{l}"].size) * 0.2
        blocks[f"g{l}"][:] = rng.normal(size=blocks[f"g{l}"].size) * 0.1
        blocks[f"b{l}"][:] = rng.normal(size=blocks[f"b{l}"].size) * 0.05
    p = np.concatenate([blocks[n] for n, _ in M.layout()]).astype(np.float32)
    net.set_params(p)
    return net, p.astype(np.float64)


@pytest.mark.parametrize("B", [128, 640, 1152, 19456])
def test_gradient_at_tile_edges(B):
    ctx = _ctx(meshgen.bump_channel(7, 3, 3, 0.08))
    net, p = _net(ctx, B)
    rng = np.random.default_rng(B + 1)
    cells = rng.integers(0, ctx.n_cells, B)
    cond = rng.normal(size=(B, 3))
    tgt = rng.normal(size=(B, 5)) * 0.5
    loss, g, out = net.loss_grad(cells, cond, tgt)
    X = M.encode(net.features().astype(np.float64)[cells])
    lo, go, oo = M.loss_and_grad(p, X, cond, tgt, rounded=True)
    assert loss == pytest.approx(lo, rel=2e-3)
    assert np.abs(out - oo).max() <= 2e-3 * np.abs(oo).max()
    gb, gob = _blocks(g.astype(np.float64)), _blocks(go)
    for name, _ in M.layout():
        err = np.linalg.norm(gb[name] - gob[name]) / max(np.linalg.norm(gob[name]), 1e-30)
        assert err <= 2e-3, (name, err)
    net.close()
    ctx.close()


@pytest.mark.parametrize("shape", [(5, 3, 1), (13, 11, 9), (31, 26, 25)])
def test_inference_equals_the_forward_pass(shape):
    """The same arithmetic on the same rows: U - U_inf is the forward pass's output, up to four
    roundings of values below 4 (U_inf is formed on the host in either case)."""
    ctx = _ctx(meshgen.bump_channel(*shape, 0.08))
    net, _ = _net(ctx, 3)
    n = ctx.n_cells
    cells = np.arange(-(-n // 128) * 128) % n
    mach = np.array([[0.5, 0.02, -0.01], [0.7, 0.0, 0.1]])
    U = net.infer(mach)
    for q, c in enumerate(mach):  # untrained: conditions and outputs are not scaled
        _, _, o = net.loss_grad(cells, np.broadcast_to(c, (len(cells), 3)).copy(), np.zeros((len(cells), 5)))
        Uinf = np.array([1.0, *c, 1.0 / (1.4 * 0.4) + (c @ c) / 2])
        assert np.abs(U[q] - (Uinf + o[:n])).max() <= 4 * 2.0 ** -51
    net.close()
    ctx.close()
