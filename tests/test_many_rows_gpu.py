"""Row reductions with more threads than 32 bits count: 8 lanes to a row from 2^29 rows on, a warp from 2^27."""
import pytest

from test_kernels_gpu import ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n", [(2 ** 29 + 1000, 1), (2 ** 27 + 1000, 33)])
def test_rows_beyond_2_to_32_threads(ctx, rows, n):  # noqa: F811
    import torch
    z = torch.zeros(rows, n, device="cuda")                  # one plane for both parts: 18 GB at 33 columns
    loss = torch.full((rows,), -1.0, device="cuda")
    at = [0, 7, rows // 2, rows - 1001, rows - 1]
    for k, r in enumerate(at):
        z[r] = k + 1
    rc = ctx.lib.cnb_l2out_fwd_bwd(ctx.h, z.data_ptr(), z.data_ptr(), loss.data_ptr(), None, None, rows, n, ctx._stream())
    assert rc == 0
    assert loss.amin().item() == 0 and loss.count_nonzero().item() == len(at)
    assert [loss[r].item() for r in at] == [2.0 * n * (k + 1) ** 2 for k in range(len(at))]
    del z, loss
    torch.cuda.empty_cache()
