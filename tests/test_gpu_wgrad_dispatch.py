"""Weight-gradient GEMM around the lines of its dispatch (one CTA or two per tile, split or not, one buffer or two per
epilogue warp) and with tiles in both orders. Small whole numbers: every product and every partial sum is exact."""
import pytest
import torch

from switchml_b200.ops.wgrad import wgrad_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [192, 193, 384, 385, 512, 513, 896, 897])
@pytest.mark.parametrize("m, n", [(1024, 1024), (1032, 1024),      # 16 tiles of 256 x 256, 20
                                  (8, 8448), (8704, 8),            # 33 and 34, ragged
                                  (512, 9472), (520, 9472),        # 74, and 111 in three rows
                                  (18944, 264), (2304, 2304)])     # 148 in two columns, 81 square
def test_exact_products(k, m, n):
    g = torch.Generator(device="cuda").manual_seed(k + m)
    dy = torch.randint(-2, 3, (k, m), generator=g, device="cuda").bfloat16()
    x = torch.randint(-2, 3, (k, n), generator=g, device="cuda").bfloat16()
    want = dy.float().t() @ x.float()  # exact in any order: at most 4 * 897
    out = torch.full((m, n), float("nan"), device="cuda")
    assert torch.equal(wgrad_gemm(dy, x, out=out), want)
