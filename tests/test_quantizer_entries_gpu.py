"""What the quantizer's C entry points do with lists and sizes that they refuse: a status, before anything is launched."""
import pytest
import torch

import nanochat_cpp_b200 as nc

pytestmark = pytest.mark.gpu
lib, capi = nc.capi.lib, nc.capi


def test_a_list_is_read_in_place():
    """A count beyond any memory with a first member that is refused: nothing is copied on the way there."""
    jobs, items = (capi.QuantizeJob * 1)(), (capi.QuantizeItem * 1)()
    for n in (1, 2 ** 31 - 1):
        assert lib.mxb200_quantize_mx_batch(jobs, n, 1, 0, None) == capi.ERR_NULL
        assert lib.mxb200_quantize_mx_items(items, n, 0, None) == capi.ERR_NULL
    for call in (lambda n: lib.mxb200_quantize_mx_batch(None, n, 1, 0, None), lambda n: lib.mxb200_quantize_mx_items(None, n, 0, None)):
        assert call(1) == call(-1) == capi.ERR_NULL and call(0) == capi.OK


@pytest.mark.parametrize("bf16,tiles", [(0, 2 ** 30), (1, 2 ** 31)])
def test_a_tensor_of_more_units_than_a_launch_counts_is_refused(bf16, tiles):
    x = torch.empty(16, device="cuda")  # only its address is looked at
    out = capi.MxOut(x.data_ptr(), 128 * tiles, x.data_ptr(), tiles)
    assert lib.mxb200_quantize_mx(x.data_ptr(), bf16, 128, 128 * tiles, out, capi.MxOut(), 0, 0, None) == capi.ERR_SHAPE
