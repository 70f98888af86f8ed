"""A batch under little free memory is cut to what its buffers really take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GB = 10 ** 9


@pytest.mark.parametrize("precision", [0, 1])
def test_a_batch_fits_the_memory_that_is_free(libpath, precision):
    import torch
    from gpu_hdbscan_b200 import Context
    ctx = Context(0)
    n, count = 5400, 100
    rng = np.random.default_rng(0)
    Xs = [torch.from_numpy(rng.normal(size=(n, 4)).astype(np.float32)).cuda() for _ in range(count)]
    run = lambda X: ctx.hdbscan_batched(X, k=8, mpts=8, sample_num=4, precision=precision, strict=False)
    run(Xs[:2])  # the kernels are loaded
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - 3 * GB // 2, dtype=torch.uint8, device="cuda")
    try:
        labels, ncl, _ = run(Xs)[:3]
    finally:
        del filler
        torch.cuda.empty_cache()
    assert len(labels) == count and all(len(x) == n for x in labels)
    ctx.close()
