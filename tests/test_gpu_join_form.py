"""The run statistics name the FP32 join's form that ran: 1 by rows, 2 in tiles."""
import pytest

from conftest import blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,setting,form", [(12, 0, 1), (28, 0, 1), (29, 0, 2), (64, 0, 2), (12, 1, 1),
                                            (28, 1, 1), (29, 1, 2), (12, 2, 2), (29, 2, 2)])
def test_join_config_names_the_form(ctx, d, setting, form):
    X = blobs(600, d, seed=d)
    ctx.set_join_tiles(setting)
    try:  # not strict: a run whose graph falls apart has its statistics all the same
        _, _, st, *_ = ctx.hdbscan_batched([X, X], k=8, mpts=8, sample_num=4, strict=False)
    finally:
        ctx.set_join_tiles(0)
    assert st["join_config"] == form
