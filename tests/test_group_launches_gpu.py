"""Launches that carry several problems: mxb200_gemm_group and mxb200_quantize_mx_items, against the CPU oracle and the
separate calls, at the edges of their tiles, groups and routes."""
import ctypes

import numpy as np
import pytest
import torch

import nanochat_cpp_b200 as nc
from helpers import np_f32, np_u8
from oracle import mx_oracle as mo

pytestmark = pytest.mark.gpu
lib, capi = nc.capi.lib, nc.capi

TOL_BF16 = 2e-3  # one bf16 rounding per value: 2^-9 at most, relative to the value
TOL_F32 = 1e-5   # fp32 sums of up to 16384 products in another order


@pytest.fixture(autouse=True)
def _default_config():
    lib.mxb200_set_gemm_config(0, 0)
    yield
    lib.mxb200_set_gemm_config(0, 0)
    assert capi.device_status() == 0


def _stream():
    return torch.cuda.current_stream().cuda_stream


def rel(got, want):
    got, want = got.double().cpu(), want.double().cpu()
    return ((got - want).norm() / (want.norm() + 1e-30)).item()


def operand(rows, k, seed):
    x = torch.randn(rows, k, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16)
    return nc.quantize_mx(x.cuda(), True, False)


def gemm_group(problems):
    """problems: (qa, qb, out, resid, alpha, accumulate); returns the workspace bytes asked for."""
    arr = (capi.GemmDesc * len(problems))()
    p = lambda t: None if t is None else t.data_ptr()
    for d, (qa, qb, out, resid, alpha, acc) in zip(arr, problems):
        kind = capi.OUT_BF16 if out.dtype == torch.bfloat16 else capi.OUT_F32
        d.a, d.a_scale, d.b, d.b_scale = p(qa.data), p(qa.inv_scale), p(qb.data), p(qb.inv_scale)
        d.d, d.resid, d.alpha = p(out), p(resid), p(alpha)
        d.M, d.N, d.K, d.out_kind, d.accumulate = out.size(0), out.size(1), qa.data.size(1), kind, acc
    need = lib.mxb200_gemm_group_workspace_bytes(arr, len(problems))
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert lib.mxb200_gemm_group(arr, len(problems), ws.data_ptr() if need else None, need, _stream()) == capi.OK
    return need


# tiles of 128 and 256 rows that are half empty, one 128-row matrix in a group, K of one tile beside a K that is cut into
# slices (from 4096 on), lists of one to four (a fourth takes a launch of its own)
GROUPS = [
    [(128, 128, 128)],
    [(256, 384, 512), (640, 256, 128)],
    [(128, 768, 4096), (384, 256, 256)],
    [(256, 256, 4096), (256, 384, 2048), (896, 640, 384)],
    [(384, 128, 256), (256, 256, 128), (128, 512, 384), (640, 384, 256)],
    [(256, 384, 8192), (384, 256, 128), (128, 256, 16384)],
]


@pytest.mark.parametrize("shapes", GROUPS, ids=len)
@pytest.mark.parametrize("tile_n", [0, 128, 256, 384, 512, 640])
@pytest.mark.parametrize("max_ctas", [0, 4])  # 4: a CTA (or pair) goes from one member to the next, several times
def test_gemm_group(shapes, tile_n, max_ctas):
    lib.mxb200_set_gemm_config(tile_n, max_ctas)
    problems, wants = [], []
    for i, (M, N, K) in enumerate(shapes):
        qa, qb = operand(M, K, 2 * i), operand(N, K, 2 * i + 1)
        want = torch.from_numpy(mo.mx_gemm_ref(np_u8(qa.data), np_u8(qa.inv_scale), np_u8(qb.data), np_u8(qb.inv_scale))).cuda()
        if i % 3 == 0:  # fp32, += alpha * product
            alpha = torch.tensor([0.5], device="cuda")
            out = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda")
            wants.append((out + 0.5 * want, TOL_F32))
            problems.append((qa, qb, out, None, alpha, 1))
        elif i % 3 == 1:
            wants.append((want, TOL_BF16))
            problems.append((qa, qb, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), None, None, 0))
        else:
            r = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda").to(torch.bfloat16)
            wants.append((want + r.float(), 2 * TOL_BF16))  # rounded twice
            problems.append((qa, qb, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), r, None, 0))
    gemm_group(problems)
    for (_, _, out, *_), (want, tol) in zip(problems, wants):
        assert rel(out, want) < tol


def test_group_refuses_a_short_workspace_and_bad_members():
    qa, qb = operand(256, 8192, 0), operand(256, 8192, 1)
    out = torch.empty(256, 256, device="cuda")
    d = capi.GemmDesc(qa.data.data_ptr(), qa.inv_scale.data_ptr(), qb.data.data_ptr(), qb.inv_scale.data_ptr(),
                      out.data_ptr(), None, None, 256, 256, 8192, capi.OUT_F32, 0)
    need = lib.mxb200_gemm_group_workspace_bytes(ctypes.byref(d), 1)
    assert need > 0  # few tiles and a deep K: cut into slices
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert lib.mxb200_gemm_group(ctypes.byref(d), 1, None, 0, _stream()) == capi.ERR_WORKSPACE
    assert lib.mxb200_gemm_group(ctypes.byref(d), 1, ws.data_ptr(), need - 1, _stream()) == capi.ERR_WORKSPACE
    bad = (capi.GemmDesc * 2)(d, d)
    bad[1].N = 100
    out.fill_(7.0)
    assert lib.mxb200_gemm_group(bad, 2, ws.data_ptr(), need, _stream()) == capi.ERR_SHAPE
    assert (out == 7.0).all()  # checked before anything is launched
    assert lib.mxb200_gemm_group(None, 0, None, 0, _stream()) == capi.OK


@pytest.mark.parametrize("M,N,K", [(128, 256, 16384), (768, 768, 16384), (3072, 768, 16384), (1536, 6144, 16384), (512, 6144, 6144)])
def test_chosen_slices_fit_the_built_in_scratch(M, N, K):
    """mxb200_gemm_splits' own choice is always accepted by mxb200_gemm_splitk_static."""
    splits = lib.mxb200_gemm_splits(M, N, K)
    assert splits >= 1 and lib.mxb200_gemm_workspace_bytes(M, N, K, splits) <= capi.STATIC_SCRATCH_BYTES


# (rows, cols, bf16): fewer units than the machine holds go a CTA per tile, more stream (592 stages on 148 SMs); a list of
# up to 4 and of up to 64 tensors stream through different kernels
LISTS = [
    [(128, 128, True), (128, 256, False)],
    [(256, 384, False), (128, 128, False), (384, 128, True), (640, 256, True), (128, 128, False)],
    [(16384, 640, True), (128, 128, False)],
    [(6144, 896, False), (128, 1024, True), (256, 128, False)],
    [(2048, 640, True), (1024, 768, False)] * 4 + [(128, 128, True)],
]


@pytest.mark.parametrize("shapes", LISTS, ids=len)
@pytest.mark.parametrize("layouts", ["both", "rows", "columns"])
def test_quantizer_list_of_both_types(shapes, layouts):
    items = (capi.QuantizeItem * len(shapes))()
    held = []
    for i, (rows, cols, bf16) in enumerate(shapes):
        g = torch.Generator(device="cuda").manual_seed(i)
        x = torch.randn(rows, cols, generator=g, device="cuda") * torch.logspace(-6, 6, cols, device="cuda")
        x[0, :32] = 0
        x[1, 3], x[2, 40], x[5, 64] = float("nan"), float("inf"), 448 * 1.8
        x[64:96, 7] = float("nan")  # a whole column block
        x = x.to(torch.bfloat16) if bf16 else x
        got = nc.empty_mx(rows, cols, x.device)
        for t in (got.data, got.inv_scale, got.data_t, got.inv_scale_t):
            t.view(torch.uint8).fill_(0x5a)
        job = items[i].job
        job.x, job.rows, job.cols = x.data_ptr(), rows, cols
        if layouts != "columns":
            job.out = nc.mx_out(got.data, got.inv_scale)
        if layouts != "rows":
            job.out_t = nc.mx_out(got.data_t, got.inv_scale_t)
        items[i].x_bf16 = int(bf16)
        held.append((x, got))
    assert lib.mxb200_quantize_mx_items(items, len(shapes), capi.SCALE_REFERENCE, _stream()) == capi.OK
    for x, got in held:
        if x.numel() <= 640 * 256:
            want = mo.quantize_mx(np_f32(x))
            pairs = [(got.data, want["data"]), (got.inv_scale, want["scale"]), (got.data_t, want["data_t"]), (got.inv_scale_t, want["scale_t"])]
        else:
            # 640-row strips are small enough for the kernel with a CTA per tile, which the oracle tests cover; a strip's
            # row-wise layout is a run of rows of the whole one
            pairs = []
            for r in (0, x.size(0) // 256 * 128, x.size(0) - 128):
                strip = nc.quantize_mx(x[r:r + 128].contiguous())
                c = x.size(1)
                pairs += [(got.data[r:r + 128], strip.data), (got.inv_scale.view(-1)[r * c // 32:(r + 128) * c // 32], strip.inv_scale),
                          (got.data_t[:, r:r + 128], strip.data_t)]
                tiles = got.inv_scale_t.view(torch.uint8).view(c // 128, x.size(0) // 128, 512)
                pairs.append((tiles[:, r // 128], strip.inv_scale_t))
            pairs = [(a, np_u8(b.contiguous())) for a, b in pairs]
        for i, (a, w) in enumerate(pairs):
            a = np_u8(a.contiguous()).reshape(-1)
            column = i % 4 >= 2
            if (layouts == "rows" and column) or (layouts == "columns" and not column):
                assert (a == 0x5a).all()
            else:
                assert np.array_equal(a, np.asarray(w).reshape(-1))
