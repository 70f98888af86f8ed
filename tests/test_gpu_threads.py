"""Calls of different sizes at the same time, one context a thread: a kernel's attributes are the
whole process's, so what one call sets must do for every other."""
import threading

import pytest

from conftest import blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,precision", [((128, 12), 0), ((400, 260), 1)])
def test_widths_side_by_side(libpath, dims, precision):
    from gpu_hdbscan_b200 import Context
    errors = []

    def work(d):
        try:
            ctx = Context(0)
            X = ctx._dev(blobs(300, d, d), ctx._torch.float32)
            for _ in range(400):
                ctx.NNDescent(X, k=8, sample_num=4, iterations=1, precision=precision)
            ctx.close()
        except Exception as e:  # to the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(d,)) for d in dims for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
