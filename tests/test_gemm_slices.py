"""How many K slices a GEMM is cut into follows from its shape alone: not from the GEMMs that share its launch, the type of
its output or whether it accumulates. So a GEMM has the same bits by itself and in any group."""
import ctypes

import pytest
import torch

import nanochat_cpp_b200 as nc

lib, capi = nc.capi.lib, nc.capi


def workspace(*gemms):
    arr = (capi.GemmDesc * len(gemms))()
    for d, (M, N, K, kind, accumulate) in zip(arr, gemms):
        d.M, d.N, d.K, d.out_kind, d.accumulate = M, N, K, kind, accumulate
    return lib.mxb200_gemm_group_workspace_bytes(arr, len(gemms))


@pytest.mark.parametrize("tokens,embd", [(256, 768), (4096, 256), (8192, 256), (16384, 256), (16384, 512), (32768, 128)])
def test_slices_follow_from_the_shape(tokens, embd):
    """The three GEMMs of an MLP's backward, together and alone (the queries need no GPU)."""
    hidden = 4 * embd
    fc, proj, dx = (hidden, embd, tokens), (embd, hidden, tokens), (tokens, embd, hidden)
    forms = [(capi.OUT_F32, 0), (capi.OUT_F32, 1), (capi.OUT_BF16, 0)]
    alone = [{workspace((*shape, *form)) for form in forms} for shape in (fc, proj, dx)]
    assert all(len(sizes) == 1 for sizes in alone)
    for form in forms:
        assert workspace((*fc, *form), (*proj, *form), (*dx, capi.OUT_BF16, 0)) == sum(s for sizes in alone for s in sizes)


@pytest.mark.parametrize("M,N,K,slices", [
    (128, 1536, 6144, 4), (384, 1536, 6144, 4), (512, 1536, 6144, 2), (1024, 1536, 6144, 1), (128, 768, 3968, 1), (128, 768, 4096, 4),
    (256, 256, 8064, 4), (256, 256, 8192, 2), (256, 256, 16384, 4), (768, 1152, 16384, 4), (768, 1280, 16384, 1), (128, 9472, 16384, 4),
    (128, 9600, 16384, 1)])
def test_slices_at_the_rules_lines(M, N, K, slices):
    """On 148 SMs, by the workspace asked for."""
    assert workspace((M, N, K, capi.OUT_BF16, 0)) == (M * N * 4 * slices if slices > 1 else 0)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (128, 128, 0), (0, 256, 8192), (-128, 256, 8192), (256, 256, -128)])
def test_queries_take_any_shape(M, N, K):
    """A shape that no GEMM accepts needs no workspace; the refusal is the call's."""
    assert workspace((M, N, K, capi.OUT_F32, 0)) == 0
    assert lib.mxb200_gemm_splits(M, N, K) == 1


def test_gemms_that_touch_one_output_do_not_share_a_launch():
    """By the workspace that the launches need together (256 x 256 x 8192 is cut into two slices): nothing is launched."""
    M = N = 256
    K, slices = 8192, 2 * 256 * 256 * 4

    def need(**second):
        arr = (capi.GemmDesc * 2)()
        for d, base in zip(arr, (1 << 32, 1 << 33)):
            d.a, d.b, d.a_scale, d.b_scale, d.d = (base + (i << 24) for i in range(5))
            d.M, d.N, d.K, d.out_kind, d.accumulate = M, N, K, capi.OUT_F32, 1
        for name, value in second.items():
            setattr(arr[1], name, value)
        return lib.mxb200_gemm_group_workspace_bytes(arr, 2)

    first = (1 << 32) + (4 << 24)  # the first one's output, M * N * 4 bytes
    assert need() == 2 * slices and need(d=first + M * N * 4) == 2 * slices and need(d=first - M * N * 4) == 2 * slices
    for name in ("d", "a", "b", "a_scale", "b_scale", "resid", "alpha"):
        assert need(**{name: first + M * N * 4 - 4}) == slices, name
    assert need(d=(1 << 32) + 16) == slices  # writes into the first one's operand


def operand(rows, k, seed):
    x = torch.randn(rows, k, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
    return nc.quantize_mx(x.to(torch.bfloat16), True, False)


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(256, 256, 8192), (640, 256, 256)], [(512, 384, 8192), (128, 768, 16384), (896, 128, 128)],
                                    [(256, 640, 384), (384, 384, 16384)]], ids=len)
def test_group_has_the_bits_of_separate_calls(shapes):
    """Sliced and unsliced members, fp32 (+= with alpha) and bf16 in turn."""
    arr, held = (capi.GemmDesc * len(shapes))(), []
    stream = torch.cuda.current_stream().cuda_stream
    alpha = torch.tensor([0.75], device="cuda")
    for i, (d, (M, N, K)) in enumerate(zip(arr, shapes)):
        qa, qb = operand(M, K, 2 * i), operand(N, K, 2 * i + 1)
        f32 = i % 2 == 0
        got = torch.randn(M, N, device="cuda").to(torch.float32 if f32 else torch.bfloat16)
        want = got.clone()
        d.a, d.a_scale, d.b, d.b_scale = qa.data.data_ptr(), qa.inv_scale.data_ptr(), qb.data.data_ptr(), qb.inv_scale.data_ptr()
        d.d, d.alpha, d.M, d.N, d.K = got.data_ptr(), alpha.data_ptr() if f32 else None, M, N, K
        d.out_kind, d.accumulate = (capi.OUT_F32, 1) if f32 else (capi.OUT_BF16, 0)
        if f32:
            nc.mx_gemm_f32(qa.data, qa.inv_scale, qb.data, qb.inv_scale, want, True, alpha)
        else:
            nc.mx_gemm_out(want, qa.data, qa.inv_scale, qb.data, qb.inv_scale)
        held.append((qa, qb, got, want))
    need = lib.mxb200_gemm_group_workspace_bytes(arr, len(shapes))
    assert need > 0
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert lib.mxb200_gemm_group(arr, len(shapes), ws.data_ptr(), need, stream) == capi.OK
    assert all(torch.equal(got, want) for _, _, got, want in held)
    assert capi.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,embd", [(256, 768), (4096, 256), (16384, 256)])
@pytest.mark.parametrize("input_grad", [True, False])
def test_mlp_equals_two_linears_over_micro_batches(tokens, embd, input_grad):
    """Outputs and every gradient, bit for bit, where the weight gradients (K = tokens) are deep enough to be sliced; the
    second micro-batch accumulates."""
    g = torch.Generator(device="cuda").manual_seed(tokens + embd)
    fc = torch.randn(4 * embd, embd, generator=g, device="cuda") * embd ** -0.5
    proj = torch.randn(embd, 4 * embd, generator=g, device="cuda") * embd ** -0.5
    fc, proj, fc2, proj2 = (w.clone().requires_grad_() for w in (fc, proj, fc, proj))
    for _ in range(2):
        x = torch.randn(tokens, embd, generator=g, device="cuda").to(torch.bfloat16)
        dy = (torch.randn(tokens, embd, generator=g, device="cuda") * 1e-3).to(torch.bfloat16)
        x, x2 = x.clone().requires_grad_(input_grad), x.clone().requires_grad_(input_grad)
        y = nc.fp8_relu_square_mlp(x, fc, proj)
        y2 = nc.fp8_matmul(torch.relu(nc.fp8_matmul(x2, fc2)).square(), proj2)
        y.backward(dy)
        y2.backward(dy)
        assert torch.equal(y, y2)
        assert not input_grad or torch.equal(x.grad, x2.grad)
    assert torch.equal(fc.grad, fc2.grad) and torch.equal(proj.grad, proj2.grad)


@pytest.mark.gpu
def test_mlp_with_one_weight_for_both_projections():
    """Two weight gradients into one .grad, over micro-batches: as two Linears on that weight."""
    g = torch.Generator(device="cuda").manual_seed(5)
    w = torch.randn(768, 768, generator=g, device="cuda") * 768 ** -0.5
    w, w2 = w.clone().requires_grad_(), w.clone().requires_grad_()
    for _ in range(3):
        x = torch.randn(512, 768, generator=g, device="cuda").to(torch.bfloat16)
        dy = torch.randn(512, 768, generator=g, device="cuda").to(torch.bfloat16)
        nc.fp8_relu_square_mlp(x, w, w).backward(dy)
        nc.fp8_matmul(torch.relu(nc.fp8_matmul(x, w2)).square(), w2).backward(dy)
        assert torch.equal(w.grad, w2.grad)
