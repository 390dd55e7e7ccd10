"""Products with a second output: what is refused, and the product without terms."""
import pytest
import torch

from maco_b200 import ops

pytestmark = pytest.mark.gpu


def test_gelu_dual_without_terms_writes_both_outputs():
    a, b = torch.empty(16, 0, device="cuda", dtype=torch.bfloat16), torch.empty(32, 0, device="cuda", dtype=torch.bfloat16)
    z, act = torch.ones(16, 32, device="cuda", dtype=torch.bfloat16), torch.ones(16, 32, device="cuda", dtype=torch.bfloat16)
    ops.gemm(a, b, out=z, aux=act, epilogue="gelu_dual")
    assert not z.any() and not act.any()             # gelu(0) is 0
    with pytest.raises(ValueError):
        ops.gemm(a, b, out=z, epilogue="gelu_dual")
    with pytest.raises(ValueError):
        ops.gemm(a, b, out=z, aux=act[:8], epilogue="gelu_dual")


@pytest.mark.parametrize("k", [0, 64])
def test_gelu_dual_refuses_a_second_output_on_the_host(k):
    a, b = torch.zeros(16, k, device="cuda", dtype=torch.bfloat16), torch.zeros(32, k, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="device"):
        ops.gemm(a, b, aux=torch.zeros(16, 32, dtype=torch.bfloat16), epilogue="gelu_dual")
