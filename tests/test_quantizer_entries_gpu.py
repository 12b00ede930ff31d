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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(256, 384), (6144, 1664)])  # a CTA per tile, streamed
@pytest.mark.parametrize("pad,shift", [(16, 0), (0, 16), (16, 16)])
def test_layouts_off_their_32_bytes(dtype, rows, cols, pad, shift):
    """Row strides and addresses of an odd multiple of 16 bytes take two 16-byte stores where 32 would go: the same bytes,
    and none beside them."""
    x = torch.randn(rows, cols, generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda").to(dtype)
    want = nc.quantize_mx(x)

    def placed(R, C):
        flat = torch.full((shift + R * (C + pad) + 16,), 0x5a, dtype=torch.uint8, device="cuda")
        return flat, flat[shift:shift + R * (C + pad)].view(R, C + pad)
    (flat, data), (flat_t, data_t) = placed(rows, cols), placed(cols, rows)
    scale, scale_t = (torch.empty(rows * cols // 32, dtype=torch.uint8, device="cuda") for _ in range(2))
    out = capi.MxOut(data.data_ptr(), cols + pad, scale.data_ptr(), cols // 128)
    out_t = capi.MxOut(data_t.data_ptr(), rows + pad, scale_t.data_ptr(), rows // 128)
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.mxb200_quantize_mx(x.data_ptr(), int(dtype == torch.bfloat16), rows, cols, out, out_t, 0, 0, stream) == capi.OK
    byte = torch.uint8
    assert torch.equal(data[:, :cols], want.data.view(byte)) and torch.equal(data_t[:, :rows], want.data_t.view(byte))
    assert torch.equal(scale, want.inv_scale.view(byte)) and torch.equal(scale_t, want.inv_scale_t.view(byte))
    for whole, inside, n in ((flat, data, cols), (flat_t, data_t, rows)):
        assert (inside[:, n:] == 0x5a).all() and (whole[:shift] == 0x5a).all() and (whole[-16:] == 0x5a).all()
