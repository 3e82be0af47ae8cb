"""A batch whose buffers do not fit (GPU): the call says so, and the handle stays usable."""
import numpy as np
import pytest

from bes_gb300 import lib, meshgen
from tests.test_gpu_mlp import _ctx

pytestmark = pytest.mark.gpu


def test_batch_that_does_not_fit():
    torch = pytest.importorskip("torch")
    ctx = _ctx(meshgen.bump_channel(7, 3, 3, 0.08))
    net = lib.WarmStart(ctx, seed=1)
    rng = np.random.default_rng(0)
    rows = [rng.integers(0, ctx.n_cells, 256), rng.normal(size=(256, 3)), rng.normal(size=(256, 5))]
    before = net.loss_grad(*rows)
    # all but 6 GB taken: a batch of a million rows needs 12
    free, _ = torch.cuda.mem_get_info()
    try:
        hog = torch.empty(max(0, free - (6 << 30)), dtype=torch.uint8, device="cuda")
    except torch.cuda.OutOfMemoryError:
        pytest.skip("the rest of the memory is in use")
    try:
        U = np.tile(np.array([1.0, 0.5, 0.0, 0.0, 1.9]), (1, ctx.n_cells, 1))
        with pytest.raises(lib.BesError):
            net.train(np.array([[0.5, 0.0, 0.0]]), U, steps=0, batch=1 << 20)
        after = net.loss_grad(*rows)
    finally:
        del hog
        torch.cuda.empty_cache()
    for a, b in zip(before, after):
        assert np.array_equal(a, b)
    net.close()
    ctx.close()
