"""llaisysSelfAttention against the oracle: the reference's own cases and tolerances
(reference: test/ops/self_attention.py:71-81), the golden vectors, and benchmark configuration 1."""
import pytest
import torch

import llaisys_b200 as llaisys
from oracle import attention, workloads
from tests import helpers

REF_SHAPES = [(2, 2, 1, 1, 4), (5, 11, 4, 2, 8)]
MORE_SHAPES = [(1, 1, 12, 2, 128), (1, 513, 12, 2, 128), (16, 16, 12, 2, 128), (40, 100, 12, 2, 128),
               (3, 35, 8, 8, 64), (7, 7, 6, 1, 32)]


def check_reference_case(device, shape, dname):
    qlen, kvlen, nh, nkvh, hd = shape
    dt = helpers.TORCH_DTYPE[dname]
    g = torch.Generator().manual_seed(hash(shape) % 1000)
    # U[0, 1) like the reference's random_tensor (test/test_utils.py:8-12)
    q = torch.rand((qlen, nh, hd), generator=g).to(dt)
    k = torch.rand((kvlen, nkvh, hd), generator=g).to(dt)
    v = torch.rand((kvlen, nkvh, hd), generator=g).to(dt)
    scale = 1.0 / hd ** 0.5
    expect = attention.self_attention(q, k, v, scale)
    got = helpers.run_self_attention(q, k, v, scale, device, dname)
    tol = helpers.REF_TOL[dname]
    assert got.shape == expect.shape and got.dtype == expect.dtype
    assert torch.allclose(got.float(), expect.float(), atol=tol, rtol=tol), helpers.max_abs(got, expect)


def check_golden(device, name):
    dname, q, k, v, scale, expect, _ = helpers.load_golden(name)
    if q is None:
        q, k, v, scale = workloads.config1()
    got = helpers.run_self_attention(q, k, v, scale, device, dname)
    assert helpers.max_abs(got, expect) <= helpers.MAX_ABS[dname]
    # tighter: an f32-accumulating kernel sits within about one output ulp of the float64 result
    f64 = attention.self_attention_f64(q, k, v, scale)
    ulp = {"f32": 1e-6, "f16": 1e-3, "bf16": 8e-3}[dname]
    assert helpers.max_abs(got, f64) <= ulp * max(1.0, f64.abs().max().item())


@pytest.mark.parametrize("dname", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("shape", REF_SHAPES + MORE_SHAPES)
def test_reference_cases_cpu(shape, dname):
    check_reference_case(llaisys.DeviceType.CPU, shape, dname)


@pytest.mark.parametrize("name", helpers.golden_cases())
def test_golden_cpu(name):
    check_golden(llaisys.DeviceType.CPU, name)


@pytest.mark.gpu
@pytest.mark.parametrize("dname", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("shape", REF_SHAPES + MORE_SHAPES)
def test_reference_cases_nvidia(cuda_device, shape, dname):
    check_reference_case(llaisys.DeviceType.NVIDIA, shape, dname)


@pytest.mark.gpu
@pytest.mark.parametrize("name", helpers.golden_cases())
def test_golden_nvidia(cuda_device, name):
    check_golden(llaisys.DeviceType.NVIDIA, name)


@pytest.mark.gpu
@pytest.mark.parametrize("kvlen", [1, 15, 16, 17, 255, 256, 257, 4096, 5000])
def test_decode_lengths_around_page_and_split_boundaries_nvidia(cuda_device, kvlen):
    """qlen 1 over contiguous bf16 K/V takes the split-KV kernel: lengths on both sides of the page size (16)
    and of the split size."""
    g = torch.Generator().manual_seed(kvlen)
    q = workloads.randn((1, 12, 128), torch.bfloat16, g)
    k = workloads.randn((kvlen, 2, 128), torch.bfloat16, g)
    v = workloads.randn((kvlen, 2, 128), torch.bfloat16, g)
    scale = 1.0 / 128 ** 0.5
    got = helpers.run_self_attention(q, k, v, scale, llaisys.DeviceType.NVIDIA, "bf16")
    assert helpers.max_abs(got, attention.self_attention(q, k, v, scale)) <= helpers.MAX_ABS["bf16"]
    f64 = attention.self_attention_f64(q, k, v, scale)
    assert helpers.max_abs(got, f64) <= 8e-3 * max(1.0, f64.abs().max().item())


@pytest.mark.gpu
@pytest.mark.parametrize("dname", ["bf16", "f16"])
@pytest.mark.parametrize("qlen,kvlen", [(16, 16), (100, 100), (130, 131), (512, 1024), (300, 2049), (2048, 2048)])
def test_multi_token_queries_over_plain_tensors_nvidia(cuda_device, qlen, kvlen, dname):
    """From 16 query rows on, 16-bit contiguous K/V with head_dim 128 take the tensor-core (tcgen05) kernel through
    tensor maps made over the caller's tensors: lengths that end inside a 16-token tile, inside a 64-key block and
    inside a 128-row query tile, and a square causal case with several query tiles."""
    dt = helpers.TORCH_DTYPE[dname]
    g = torch.Generator().manual_seed(qlen * 7 + kvlen)
    q = workloads.randn((qlen, 12, 128), dt, g)
    k = workloads.randn((kvlen, 2, 128), dt, g)
    v = workloads.randn((kvlen, 2, 128), dt, g)
    scale = 1.0 / 128 ** 0.5
    got = helpers.run_self_attention(q, k, v, scale, llaisys.DeviceType.NVIDIA, dname)
    assert helpers.max_abs(got, attention.self_attention(q, k, v, scale)) <= helpers.MAX_ABS[dname]
    f64 = attention.self_attention_f64(q, k, v, scale)
    ulp = {"f16": 1e-3, "bf16": 8e-3}[dname]
    assert helpers.max_abs(got, f64) <= ulp * max(1.0, f64.abs().max().item())


@pytest.mark.gpu
@pytest.mark.parametrize("dname", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("qlen,kvlen,nh,nkvh,d", [
    (1, 1, 12, 2, 64), (5, 16, 12, 2, 64), (5, 17, 12, 2, 64), (1, 129, 12, 2, 128), (2, 128, 12, 2, 128), (15, 127, 5, 1, 128), (15, 900, 18, 2, 128),  # tiles of 16 rows
    (65, 65, 32, 8, 64), (86, 300, 12, 2, 64), (96, 777, 12, 2, 128), (300, 301, 12, 2, 64), (257, 513, 33, 3, 128)])  # tiles of 64 rows
def test_tiles_over_plain_tensors_nvidia(cuda_device, qlen, kvlen, nh, nkvh, d, dname):
    """Calls that neither 16-bit kernel takes: tiles that end inside the rows, key blocks that end inside a split, groups that do not
    divide a tile, CTAs of a cluster without keys. A sum of n products in f32 is off by at most n rounding errors of its terms' magnitudes;
    a softmax row's weights sum to one, so 2 (d + kvlen) x 2^-24 of the largest value bounds scores and outputs."""
    g = torch.Generator().manual_seed(qlen * kvlen)
    q, k, v = (workloads.randn((n, h, d), helpers.TORCH_DTYPE[dname], g) for n, h in ((qlen, nh), (kvlen, nkvh), (kvlen, nkvh)))
    got = helpers.run_self_attention(q, k, v, d ** -0.5, llaisys.DeviceType.NVIDIA, dname)
    f64 = attention.self_attention_f64(q, k, v, d ** -0.5)
    rounding = {"f32": 0.0, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dname]
    assert helpers.max_abs(got, f64) <= 2 * (d + kvlen) * 2.0 ** -24 * v.abs().max().item() + rounding * f64.abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("qlen,kvlen,nh,nkvh", [(16, 64, 12, 2), (64, 64, 32, 8), (128, 1000, 12, 2), (512, 1000, 12, 2), (129, 4096, 16, 2),
                                                (129, 4097, 16, 2), (128, 1000, 32, 32)])
def test_chunk_kernels_over_plain_tensors_nvidia(cuda_device, qlen, kvlen, nh, nkvh):
    """16-bit calls on both sides of the rule between the two chunk kernels. Rounding of the weights and of the result to bf16."""
    g = torch.Generator().manual_seed(qlen + kvlen)
    q, k, v = (workloads.randn((n, h, 128), torch.bfloat16, g) for n, h in ((qlen, nh), (kvlen, nkvh), (kvlen, nkvh)))
    got = helpers.run_self_attention(q, k, v, 128 ** -0.5, llaisys.DeviceType.NVIDIA, "bf16")
    f64 = attention.self_attention_f64(q, k, v, 128 ** -0.5)
    assert helpers.max_abs(got, f64) <= 8e-3 * max(1.0, f64.abs().max().item())


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("qlen", [3, 96])
def test_values_behind_the_mask_stay_out_nvidia(cuda_device, qlen, bad):
    """The last key's V row is not finite: only the last query sees it."""
    g = torch.Generator().manual_seed(qlen)
    q, k, v = (workloads.randn((n, h, 128), torch.float32, g) for n, h in ((qlen, 12), (200, 2), (200, 2)))
    v[-1] = bad
    got = helpers.run_self_attention(q, k, v, 128 ** -0.5, llaisys.DeviceType.NVIDIA, "f32")
    assert torch.isfinite(got[:-1]).all() and not torch.isfinite(got[-1]).any()
    assert helpers.max_abs(got[:-1], attention.self_attention_f64(q[:-1], k[:-1], v[:-1], 128 ** -0.5)) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("qlen,kvlen,d", [(1, 1, 128), (2, 20, 64), (3, 200, 128), (8, 700, 64), (40, 40, 128), (96, 97, 64), (96, 777, 128),
                                          (1, 1, 96), (2, 20, 96), (3, 200, 96)])  # tiles of 16 rows, of 64, one CTA per row
def test_scores_that_are_not_finite_show_nvidia(cuda_device, qlen, kvlen, d, bad):
    """A query row, a key in the middle and the first half of the keys that are not finite: in f32 the rows that see one come out as in
    float64 (NaN, or without the keys of weight zero) and the others untouched. Tolerance: see test_tiles_over_plain_tensors_nvidia."""
    g = torch.Generator().manual_seed(qlen * kvlen)
    q, k, v = (workloads.randn((n, h, d), torch.float32, g) for n, h in ((qlen, 12), (kvlen, 2), (kvlen, 2)))
    tol = 2 * (d + kvlen) * 2.0 ** -24 * v.abs().max().item()
    sees = torch.arange(kvlen)[None, :] <= torch.arange(qlen)[:, None] + kvlen - qlen
    for where in ("q", "middle", "half"):
        q_bad, k_bad = q.clone(), k.clone()
        if where == "q":
            q_bad[qlen // 2, 5, 3] = bad
            rows = torch.arange(qlen) == qlen // 2
        else:
            keys = slice(kvlen // 2, kvlen // 2 + 1) if where == "middle" else slice(0, (kvlen + 1) // 2)
            k_bad[keys, 1, 3] = bad
            rows = sees[:, keys].any(1)
        got = helpers.run_self_attention(q_bad, k_bad, v, d ** -0.5, llaisys.DeviceType.NVIDIA, "f32")
        want = torch.where(rows[:, None, None], attention.self_attention_f64(q_bad, k_bad, v, d ** -0.5),
                           attention.self_attention_f64(q, k, v, d ** -0.5))
        # (rows whose only scores are -inf have no weights at all: 0 by this operator's definition, 0 / 0 in the float64 statement)
        scores = torch.einsum("qhd,khd->qhk", q_bad.double(), k_bad.double().repeat_interleave(6, dim=1))
        empty = (scores.masked_fill(~sees[:, None, :], -float("inf")) == -float("inf")).all(2)
        want[empty] = 0
        assert torch.equal(torch.isnan(got), torch.isnan(want)), (where, torch.isnan(got).any(2).sum(), torch.isnan(want).any(2).sum())
        assert helpers.max_abs(got.nan_to_num(0), want.nan_to_num(0)) <= tol, where
