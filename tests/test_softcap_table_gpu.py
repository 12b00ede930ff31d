"""The table paths of the softcap kernels: lookups give the bits of the direct evaluation, and logits outside the tables
take the direct path beside them."""
import pytest
import torch

import nanochat_cpp_b200 as nc

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, -0.0, 2 ** -16, -(2 ** -16), 2 ** -17, 2 ** -25, 2 ** -26, 127.5, -127.5, 128.0, -1e30, 1e-40]


def _inputs(rows, padded, vocab, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = (torch.randn(rows, padded, generator=g, device="cuda") * 2).to(torch.bfloat16)
    for v in SPECIAL:
        z.view(-1)[torch.randint(0, z.numel(), (16,), generator=g, device="cuda")] = v
    t = torch.randint(-1, vocab, (rows,), generator=g, device="cuda")
    t[:3] = torch.tensor([-1, 0, vocab - 1])
    return z, t


@pytest.mark.parametrize("rows,padded,vocab", [(256, 24448, 24321), (640, 8192, 8192), (1280, 4096, 4090)])
def test_loss_rows_together_equal_rows_alone(rows, padded, vocab):
    """Many rows go through the table, a single row of these lengths does not."""
    z, t = _inputs(rows, padded, vocab, rows)
    loss, lse = nc.softcap_ce_loss(z, t, vocab, 15.0)
    for r in list(range(0, rows, 37)) + [1, 2, rows - 1]:
        one_loss, one_lse = nc.softcap_ce_loss(z[r:r + 1], t[r:r + 1], vocab, 15.0)
        assert torch.equal(one_loss, loss[r:r + 1])
        if t[r] >= 0:
            assert torch.equal(one_lse, lse[r:r + 1])


@pytest.mark.parametrize("rows,padded,vocab", [(128, 128, 128), (128, 256, 129), (384, 1152, 1100), (1024, 8192, 8191)])
def test_gradient_against_torch(rows, padded, vocab):
    z, t = _inputs(rows, padded, vocab, padded)
    _, lse = nc.softcap_ce_loss(z, t, vocab, 15.0)
    scale = torch.rand(rows, device="cuda") + 0.5
    q = nc.empty_mx(rows, padded, z.device)
    nc.softcap_ce_grad_mx(z, t, lse, vocab, 15.0, *nc.mx_outs(q), scale)
    th = torch.tanh(z.double() / 15)
    onehot = torch.nn.functional.one_hot(t.clamp(min=0), padded)
    g = (torch.exp(15 * th - lse[:, None].double()) - onehot) * (1 - th * th) * scale[:, None]
    g[t < 0] = 0
    g[:, vocab:] = 0
    want = nc.quantize_mx(g.to(torch.bfloat16))
    # fp32 with device tanh and exp (a few ulp) against float64: a value lands on another bf16 with the chance of a few
    # 2^-24 in 2^-9, and on another e4m3 byte more rarely still; a changed block maximum changes up to 32 bytes
    for got, ref in ((q.data, want.data), (q.data_t, want.data_t), (q.inv_scale, want.inv_scale), (q.inv_scale_t, want.inv_scale_t)):
        assert (got.view(torch.uint8) != ref.view(torch.uint8)).float().mean().item() < 2e-3
    assert nc.capi.device_status() == 0
