"""Integer group quantisation and optimizer-state packing kernels against their PyTorch references."""
import pytest
import torch

from atorch_b200.ops import lowbit, quantizer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("sym", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_quantize_dequantize(bits, sym, dtype):
    torch.manual_seed(0)
    x = torch.randn(64 * 2048, device="cuda").to(dtype)
    q, p = quantizer.quantize(x, 64, bits, sym)
    qr, pr = quantizer.quantize_reference(x, 64, bits, sym)
    assert torch.allclose(p, pr.to(p.device), rtol=1e-5, atol=1e-7)
    assert (q != qr).float().mean() < 2e-3
    d = quantizer.dequantize(q, p, 64, bits, sym, torch.float32)
    dr = quantizer.dequantize_reference(q, p, 64, bits, sym, torch.float32)
    assert torch.allclose(d, dr, rtol=1e-5, atol=1e-6)
    assert (d - x.float()).abs().max() < (0.03 if bits == 8 else 0.5)


def test_swizzle_and_reduce():
    torch.manual_seed(1)
    x = torch.randn(32 * 256, device="cuda", dtype=torch.bfloat16)
    q, p = quantizer.swizzle_quant(x, 32, 8, True, 2, 2, 4)
    gm = quantizer.swizzle_group_map(32, 2, 2, 4, "cuda").long()
    q0, p0 = quantizer.quantize(x, 32, 8, True)
    assert torch.equal(q.view(32, -1)[gm], q0.view(32, -1)) and torch.equal(p[gm], p0)
    parts = [torch.randn(8 * 512, device="cuda", dtype=torch.bfloat16) for _ in range(8)]
    qs, ps = zip(*(quantizer.quantize(t, 8, 8, True) for t in parts))
    qo, po = quantizer.quantized_reduction(torch.cat(qs), torch.cat(ps), 64, 8, 8, True, 8)
    got = quantizer.dequantize(qo, po, 8, 8, True, torch.float32)
    ref = sum(quantizer.dequantize(a, b, 8, 8, True, torch.float32) for a, b in zip(qs, ps))
    assert (got - ref).abs().max() < 0.05 * ref.abs().max()


def test_state_packing():
    torch.manual_seed(2)
    x = torch.randn(100000, device="cuda")
    for bits in (8, 16):
        c, am = lowbit.pack_absmax_linear(x, bits, 2048)
        back = lowbit.unpack_absmax_linear(c, am, bits, 2048)
        assert (back - x).abs().max() < (0.03 if bits == 8 else 2e-4)
    for bits, gs in ((4, 128), (8, 2048)):
        qm = lowbit.create_dynamic_map(True, bits).cuda()
        c, am = lowbit.pack_nonlinear(x, qm, bits, gs)
        back = lowbit.unpack_nonlinear(c, am, qm, x.numel(), bits, gs)
        cpu_c, cpu_am = lowbit.pack_nonlinear(x.cpu(), qm.cpu(), bits, gs)
        ref = lowbit.unpack_nonlinear(cpu_c, cpu_am, qm.cpu(), x.numel(), bits, gs)
        assert (back.cpu() - ref).abs().max() < 1e-5
        s1, _ = lowbit.pack_nonlinear(x, qm, bits, gs, stochastic=True, seed=1)
        s2, _ = lowbit.pack_nonlinear(x, qm, bits, gs, stochastic=True, seed=1)
        s3, _ = lowbit.pack_nonlinear(x, qm, bits, gs, stochastic=True, seed=7)
        assert torch.equal(s1, s2) and not torch.equal(s1, s3)
        mean_err = (lowbit.unpack_nonlinear(s1, am, qm, x.numel(), bits, gs) - x).mean().abs()
        assert mean_err < 5e-3            # stochastic rounding is unbiased


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("group", [8, 248, 256, 520, 1024, 2040, 2056, 4096, 8192, 8200, 30])
def test_quantize_group_lengths(group, dtype):
    """Every split of a group over lanes and warps, the lengths at its edges, and the general kernel beyond it."""
    torch.manual_seed(group)
    groups = 37
    x = (torch.randn(groups, group, device="cuda") * torch.rand(groups, 1, device="cuda")).to(dtype)
    x[3] = 0
    for bits in (8, 4):
        for sym in (True, False):
            q, p = quantizer.quantize(x.reshape(-1), groups, bits, sym)
            qr, pr = quantizer.quantize_reference(x.reshape(-1), groups, bits, sym)
            assert torch.allclose(p, pr, rtol=1e-6, atol=0)
            # the kernel multiplies by the rounded reciprocal of the scale, the reference divides: x / s differs by
            # 2^-23 |x / s| <= 2^-15, so an element may differ only if its exact quotient is that close to a tie. Of a
            # 16-bit input many lie exactly on one (the scale is absmax / 127 of the same grid), hence no fixed share
            lo = 0.0 if sym else pr.double()[:, 1:2]
            v = (x.double() - lo) / pr.double()[:, :1]
            near = ((v - v.floor() - 0.5).abs() < 2 ** -14).reshape(-1)
            if bits == 8:
                assert not bool(((q != qr) & ~near).any()) and (q.int() - qr.int()).abs().max() <= 1
            else:
                assert not bool(((q != qr) & ~(near[0::2] | near[1::2])).any())
            for out in (torch.float32, dtype):
                d = quantizer.dequantize(q, p, groups, bits, sym, out)
                dr = quantizer.dequantize_reference(q, p, groups, bits, sym, out)     # one rounding to `out`
                assert torch.equal(d, dr) or torch.allclose(d.float(), dr.float(), rtol=2 ** -7, atol=1e-6)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("group", [8, 64, 72, 128, 256, 264, 512, 1024, 2048, 4104])
def test_quantize_special_values_like_the_general_kernel(group, dtype):
    """NaN, infinities, zeros and values whose scale has no finite reciprocal, for every split of a group over lanes: the same
    codes and parameters as the general kernel, which inputs off a 16-byte boundary take. Odd numbers of groups leave lanes
    without one."""
    torch.manual_seed(group)
    groups = 37
    x = torch.randn(groups, group, device="cuda").to(dtype)
    x[1, 3], x[2, 0], x[4, 7] = float("nan"), float("inf"), -float("inf")
    x[5], x[6], x[7] = float("nan"), 0, float("inf")
    x[8] = torch.where(torch.arange(group, device="cuda") % 2 == 0, 1e-45, -0.0).to(dtype)
    x[36, group - 1] = 1e4
    flat = x.reshape(-1)
    shifted = torch.empty(flat.numel() + 1, device="cuda", dtype=dtype)[1:]
    shifted.copy_(flat)
    for bits in (8, 4):
        for sym in (True, False):
            (q, p), (qg, pg) = (quantizer.quantize(t, groups, bits, sym) for t in (flat, shifted))
            assert torch.equal(q, qg) and torch.equal(p.nan_to_num(7.0), pg.nan_to_num(7.0))
