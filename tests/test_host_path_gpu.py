"""The native host path (csrc/torch_engine.cpp) and the small kernels it launches, against torch on the same inputs."""
import pytest
import torch

import nanochat_cpp_b200 as nc

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 16384])
def test_loss_reductions(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    targets = torch.randint(-1, 4, (n,), generator=g, device="cuda")
    losses = torch.rand(n, generator=g, device="cuda") * (targets >= 0)
    count = torch.empty((), dtype=torch.int64, device="cuda")
    assert nc.capi.lib.mxb200_count_valid(targets.data_ptr(), n, count.data_ptr(), _stream()) == 0
    assert count.item() == (targets >= 0).sum().item()
    total = torch.empty((), device="cuda")
    assert nc.capi.lib.mxb200_reduce_losses(losses.data_ptr(), n, None, total.data_ptr(), _stream()) == 0
    # fp32 sum of n non-negative values: n / 1024 terms per thread, then 10 butterfly steps, half an ulp each
    bound = (n / 1024 + 11) * 2 ** -24 * losses.double().sum().item()
    assert abs(total.double() - losses.double().sum()).item() <= bound
    if count.item():
        mean = torch.empty((), device="cuda")
        assert nc.capi.lib.mxb200_reduce_losses(losses.data_ptr(), n, count.data_ptr(), mean.data_ptr(), _stream()) == 0
        assert torch.equal(mean, total / count)


@pytest.mark.parametrize("n", [8, 8 * 257, 128 * 1664, 16384 * 1536])
def test_scale_bf16_matches_torch(n):
    x = torch.randn(n, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda").to(torch.bfloat16)
    x[:3] = torch.tensor([float("nan"), float("inf"), -0.0])
    scale = torch.tensor(0.7312, device="cuda")
    y = torch.empty_like(x)
    assert nc.capi.lib.mxb200_scale_bf16(x.data_ptr(), scale.data_ptr(), y.data_ptr(), n, _stream()) == 0
    assert torch.equal(y.nan_to_num(7.0), (x * scale).nan_to_num(7.0))


@pytest.mark.parametrize("cached", [False, True])
def test_no_grad_forward_equals_training_forward(cached):
    """Without grad only the row-wise layouts are made; the output is the same, and a cache is filled or left alone."""
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(384, 256, generator=g, device="cuda").to(torch.bfloat16)
    ws = [torch.randn(n, 256, generator=g, device="cuda").requires_grad_() for n in (256, 128, 128)]
    caches = [nc.Fp8WeightCache(cached) for _ in range(3)]
    with torch.no_grad():
        y = nc.fp8_matmul(x, ws[0], caches[0])
        qkv = nc.fp8_qkv(x, *ws, cache=caches[1])
        mlp = nc.fp8_relu_square_mlp(x, ws[0], torch.eye(256, device="cuda"), caches[2])
        again = nc.fp8_matmul(x, ws[0], caches[0])
    assert not y.requires_grad and torch.equal(y, again)
    assert torch.equal(y, nc.fp8_matmul(x, ws[0]).detach())
    assert torch.equal(y, nc.fp8_matmul(x, ws[0], caches[0]).detach())
    assert all(torch.equal(a, b.detach()) for a, b in zip(qkv, nc.fp8_qkv(x, *ws, cache=caches[1])))
    assert torch.equal(mlp, nc.fp8_relu_square_mlp(x, ws[0], torch.eye(256, device="cuda")).detach())


def test_per_token_loss_with_cache_matches_without():
    """Reduction none holds its cache in the graph node and uses it again in backward."""
    g = torch.Generator(device="cuda").manual_seed(4)
    x0 = torch.randn(256, 128, generator=g, device="cuda").to(torch.bfloat16)
    w0 = torch.randn(384, 128, generator=g, device="cuda") * 0.1
    t = torch.randint(-1, 380, (256,), generator=g, device="cuda")
    up = torch.rand(256, generator=g, device="cuda")
    got = []
    for cache in (None, nc.Fp8WeightCache(True)):
        x, w = x0.clone().requires_grad_(), w0.clone().requires_grad_()
        loss = nc.softcap_cross_entropy(x, w, t, 380, 15.0, 128, "none", cache)
        del cache
        loss.backward(up)
        got.append((loss.detach(), x.grad, w.grad))
    assert all(torch.equal(a, b) for a, b in zip(*got))


def test_backward_twice_needs_retain_graph():
    x = torch.randn(128, 128, device="cuda").to(torch.bfloat16).requires_grad_()
    w = torch.randn(128, 128, device="cuda").requires_grad_()
    y = nc.fp8_matmul(x, w)
    y.backward(torch.ones_like(y), retain_graph=True)
    first = w.grad.clone()
    y.backward(torch.ones_like(y))
    assert torch.equal(w.grad, 2 * first)
    with pytest.raises(RuntimeError):
        y.backward(torch.ones_like(y))


def test_first_call_of_a_fresh_thread_may_be_a_gemm():
    """A thread without a CUDA context of its own yet (an autograd worker) can start with a launch that encodes tensor
    maps: its buffers come out of the allocator's cache without a CUDA call."""
    import threading
    q = nc.quantize_mx(torch.randn(256, 256, device="cuda"))
    want, got = torch.empty(256, 256, device="cuda"), torch.zeros(256, 256, device="cuda")
    args = (q.data.data_ptr(), q.inv_scale.data_ptr()) * 2
    stream, status = _stream(), []
    lib = nc.capi.lib
    assert lib.mxb200_gemm_f32(*args, want.data_ptr(), 256, 256, 256, None, 0, stream) == 0
    torch.cuda.synchronize()
    t = threading.Thread(target=lambda: status.append(
        lib.mxb200_gemm_f32(*args, got.data_ptr(), 256, 256, 256, None, 0, stream)))
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert status == [0] and torch.equal(got, want)


def _x_mx_users(x, x_mx):
    w = [torch.randn(n, x.size(1), device="cuda").requires_grad_() for n in (256, 128, 128)]
    proj = torch.randn(128, 256, device="cuda").requires_grad_()
    return [lambda: nc.fp8_qkv(x, *w, x_mx=x_mx), lambda: nc.fp8_relu_square_mlp(x, w[0], proj, x_mx=x_mx)]


BAD_X_MX = {
    "host data": lambda q: setattr(q, "data", q.data.cpu()),
    "host scale": lambda q: setattr(q, "inv_scale", q.inv_scale.cpu()),
    "host data_t": lambda q: setattr(q, "data_t", q.data_t.cpu()),
    "host scale_t": lambda q: setattr(q, "inv_scale_t", q.inv_scale_t.cpu()),
    "data_t of data's shape": lambda q: setattr(q, "data_t", q.data_t.view(q.data.shape)),
    "data_t of another type": lambda q: setattr(q, "data_t", q.data_t.view(torch.uint8)),
    "data_t transposed view": lambda q: setattr(q, "data_t", q.data.t()),
    "short scale": lambda q: setattr(q, "inv_scale", q.inv_scale[:-1]),
    "short scale_t": lambda q: setattr(q, "inv_scale_t", q.inv_scale_t[:-1]),
    "wide scale_t": lambda q: setattr(q, "inv_scale_t", q.inv_scale_t.to(torch.float32)),
}


@pytest.mark.parametrize("bad", BAD_X_MX)
def test_x_mx_is_checked_before_anything_is_launched(bad):
    """Host checks only: nothing is launched on the operands that are refused."""
    x = torch.randn(256, 384, device="cuda").to(torch.bfloat16).requires_grad_()
    q = nc.quantize_mx(x.detach())
    BAD_X_MX[bad](q)
    launches = nc.capi.launch_count()
    for call in _x_mx_users(x, q):
        with pytest.raises(RuntimeError):
            call()
    assert nc.capi.launch_count() == launches


def test_x_mx_scales_may_be_bytes_and_no_grad_reads_rows_only():
    x = torch.randn(256, 384, device="cuda").to(torch.bfloat16).requires_grad_()
    q = nc.quantize_mx(x.detach())
    raw = nc.Fp8Tensor(q.data, q.data_t, q.inv_scale.view(torch.uint8), q.inv_scale_t.view(torch.uint8))
    rows = nc.Fp8Tensor(q.data, q.data.t(), q.inv_scale, q.inv_scale[:1])
    for call in _x_mx_users(x, raw):
        out = call()
        out = out if isinstance(out, tuple) else (out,)
        torch.autograd.backward(out, [torch.ones_like(t) for t in out])
    assert x.grad is not None
    with torch.no_grad():
        for call in _x_mx_users(x, rows):
            call()


@pytest.mark.parametrize("which", ["x", "w"])
@pytest.mark.parametrize("no_grad", [False, True])
def test_forward_mode_is_refused(which, no_grad):
    """Without a node a tangent would be dropped, which reads as a derivative of zero."""
    import torch.autograd.forward_ad as fwd
    x, w = torch.randn(128, 256, device="cuda").to(torch.bfloat16), torch.randn(256, 256, device="cuda")
    t = torch.zeros(128, dtype=torch.int64, device="cuda")
    with fwd.dual_level(), torch.set_grad_enabled(not no_grad):
        if which == "x":
            x = fwd.make_dual(x, torch.ones_like(x))
        else:
            w = fwd.make_dual(w, torch.ones_like(w))
        for call in (lambda: nc.fp8_matmul(x, w), lambda: nc.fp8_qkv(x, w, w, w), lambda: nc.fp8_relu_square_mlp(x, w, w),
                     lambda: nc.softcap_cross_entropy(x, w, t, 256, 15.0, 128)):
            with pytest.raises(NotImplementedError):
                call()


def test_function_transforms_are_refused():
    x, w = torch.randn(2, 128, 256, device="cuda").to(torch.bfloat16), torch.randn(256, 256, device="cuda")
    q = nc.quantize_mx(x[0])
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda a: nc.fp8_matmul(a, w))(x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda a: nc.fp8_relu_square_mlp(a, w, w, x_mx=q))(x)
    with pytest.raises(RuntimeError):
        torch.func.jvp(lambda a: nc.fp8_relu_square_mlp(a, w, w, x_mx=q), (x[0],), (x[0],))


def test_gate_gradient_of_an_fp32_input_is_rounded_once():
    """The gate's columns of an fp32 x carry an fp32 gradient: dx = bf16(dx of the projections + that gradient)."""
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(256, 256, generator=g, device="cuda").requires_grad_()
    w = [(torch.randn(128, 256, generator=g, device="cuda") * 0.06).requires_grad_() for _ in range(3)]
    dy = [torch.randn(256, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]
    gate = torch.randn(256, 12, generator=g, device="cuda")
    grads = []
    for gate_grad in (torch.zeros_like(gate), gate):
        x.grad = None
        torch.autograd.backward(nc.fp8_qkv(x, *w, gate_cols=12), [*dy, gate_grad])
        grads.append(x.grad)
    assert torch.equal(grads[1][:, :12], (grads[0][:, :12] + gate).to(torch.bfloat16).float())
    assert torch.equal(grads[1][:, 12:], grads[0][:, 12:])


def test_whether_a_weight_gets_a_gradient_is_decided_in_forward():
    """Frozen for the forward and thawed before the backward, as the discriminator of a generator's step: no gradient."""
    x = torch.randn(128, 128, device="cuda").to(torch.bfloat16).requires_grad_()
    w = [torch.randn(128, 128, device="cuda") for _ in range(3)]
    for call, used in ((lambda: (nc.fp8_matmul(x, w[0]),), w[:1]), (lambda: nc.fp8_qkv(x, *w), w)):
        for frozen in (True, False):
            for t in used:
                t.requires_grad_(not frozen)
                t.grad = None
            out = call()
            for t in used:
                t.requires_grad_(frozen)
            torch.autograd.backward(out, [torch.ones_like(t) for t in out])
            assert all((t.grad is None) == frozen for t in used)


class _Counting(nc.Fp8WeightCache):
    def __init__(self, enabled=False):
        super().__init__(enabled)
        self.asked = []

    def get(self, kind, weights, make):
        self.asked.append((kind, len(weights)))
        return super().get(kind, weights, make)


class _Plain:
    """A cache that is none of the library's classes."""

    def __init__(self):
        self.value, self.asked = None, []

    def get(self, kind, weights, make):
        self.asked.append((kind, len(weights)))
        self.value = make() if self.value is None else self.value
        return self.value


@pytest.mark.parametrize("cls", [lambda: _Counting(True), _Plain])
def test_any_cache_is_asked_through_its_get(cls):
    g = torch.Generator(device="cuda").manual_seed(8)
    x = torch.randn(128, 256, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(256, 256, generator=g, device="cuda")
    t = torch.randint(0, 256, (128,), generator=g, device="cuda")
    calls = {
        "matmul": (lambda x, w, c: nc.fp8_matmul(x, w, c), [(1, 1)]),
        "qkv": (lambda x, w, c: torch.cat(nc.fp8_qkv(x, w, w[:128], w[128:], cache=c), 1), [(1, 3)]),
        "mlp": (lambda x, w, c: nc.fp8_relu_square_mlp(x, w, w, c, None), [(1, 1)]),
        "loss": (lambda x, w, c: nc.softcap_cross_entropy(x, w, t, 256, 15.0, 128, "none", c), [(1, 1)]),
    }
    for name, (call, asked) in calls.items():
        got = []
        for cache in (None, cls()):
            a, b = x.clone().requires_grad_(), w.clone().requires_grad_()
            out = call(a, b, cache)
            out.backward(torch.ones_like(out))
            got.append((out, a.grad, b.grad))
        assert cache.asked[:1] == asked, name
        assert all(torch.equal(u, v) for u, v in zip(*got)), name


def test_a_copied_cache_is_empty_and_of_its_class():
    import copy
    cache = _Counting(True)
    cache.get(1, [torch.zeros(1)], lambda: [1])
    other = copy.deepcopy(cache)
    assert type(other) is _Counting and other.enabled and other.asked == [(1, 1)]


def test_calls_let_other_python_threads_run():
    """Nothing else hands the interpreter over for 100 seconds: the other thread runs when a call gives it up."""
    import sys
    import threading
    x = torch.randn(128, 128, device="cuda").to(torch.bfloat16)
    w = torch.randn(128, 128, device="cuda")
    t = torch.zeros(128, dtype=torch.int64, device="cuda")
    q = nc.quantize_mx(w)
    outs = nc.mx_outs(q)
    calls = [lambda: nc.fp8_matmul(x, w), lambda: nc.fp8_qkv(x, w, w, w), lambda: nc.fp8_relu_square_mlp(x, w, w),
             lambda: nc.softcap_cross_entropy(x, w, t, 128, 15.0, 128), lambda: nc.residual_norm_mx(x),
             lambda: nc.quantize_mx_batch_into([(w, *outs)])]
    interval = sys.getswitchinterval()
    for call in calls:
        call()
        torch.cuda.synchronize()
        ran, start = [], threading.Event()
        thread = threading.Thread(target=lambda: (start.wait(), ran.append(True)))
        thread.start()
        sys.setswitchinterval(100.0)
        try:
            start.set()
            for _ in range(500):
                call()
                if ran:
                    break
        finally:
            sys.setswitchinterval(interval)
        seen = bool(ran)
        thread.join()
        assert seen


def test_a_refusal_is_the_librarys_error_in_forward_and_backward():
    """An operand off its 16 bytes is refused on the host; its status is the error's, also from autograd's worker."""
    def off(t):  # contiguous, two bytes past an aligned address
        return torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)
    x = torch.randn(128, 128, device="cuda").to(torch.bfloat16)
    w = torch.randn(128, 128, device="cuda").requires_grad_()
    for call in (lambda a: nc.fp8_matmul(a, w), lambda a: nc.fp8_relu_square_mlp(a, w, w), lambda a: nc.fp8_qkv(a, w, w, w)[0]):
        with pytest.raises(nc.capi.Mxb200Error) as forward:
            call(off(x))
        y = call(x)
        with pytest.raises(nc.capi.Mxb200Error) as backward:
            y.backward(off(torch.ones_like(y)))
        assert forward.value.status == backward.value.status == nc.capi.ERR_ALIGNMENT
        assert "quantize_mx" in str(backward.value)
