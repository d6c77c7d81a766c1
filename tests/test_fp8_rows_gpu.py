"""The block-scaled fp8 product of prompts against the same sums in 64 bits."""
import pytest
import torch

from vllm_b200.ops import ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(129, 256, 128), (1, 8, 128), (300, 392, 384), (1000, 2112, 1280), (1153, 5000, 640)])
def test_prompt_rows(M, N, K, dtype):
    from vllm_b200.ops import cuda as cu
    torch.manual_seed(3)
    x = (torch.randn(M, K, device="cuda") * (1 + 3 * torch.rand(M, 1, device="cuda"))).to(dtype)
    wq, ws = ref.block_quant_weight_fp8(torch.randn(N, K, device="cuda") * 0.05, 128)
    ws, bias = ws.contiguous(), torch.randn(N, device="cuda", dtype=dtype)
    xq, xs = cu.per_token_group_quant_fp8(x, 128, col_major=True)
    want = (xq.double() * xs.double().repeat_interleave(128, 1)) @ (wq.double() * ws.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)).t()
    y = torch.full((M + 1, N), 7.0, device="cuda", dtype=dtype)
    cu.gemm_fp8_rows(xq, xs, wq, ws, bias, y[:M])
    cu.check_kernel_error(x.device)
    # the result's own rounding (at most 2^-8 of it in bf16, 2^-11 in fp16: 8 and 11 bits of significand) and fp32 sums of K products,
    # K 2^-24 of their magnitudes in each of the two levels
    size = (xq.double().abs() * xs.double().repeat_interleave(128, 1)) @ (wq.double().abs() * ws.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)).t()
    half = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    want = want + bias.double()
    assert ((y[:M].double() - want).abs() <= want.abs() * half + size * K * 2.0 ** -23 + 2.0 ** -24).all()
    assert bool((y[M] == 7).all())
