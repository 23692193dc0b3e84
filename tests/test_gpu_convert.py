"""convert_weight on CUDA tensors (csrc/sal_pack.cu: bit transpose and scales in one launch) against its CPU code, value for value: word rows
shorter and longer than the 32 words a CTA stages, every plane count, scales that fill several CTAs or none of one."""
import pytest
import torch

from shiftaddllm_b200.kernel import convert_weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,words,q,groups", [(32, 1, 1, 1), (64, 31, 2, 4), (96, 32, 3, 62), (32, 33, 4, 66), (64, 65, 5, 130), (32, 5, 6, 1),
                                              (32, 40, 7, 80), (64, 70, 8, 35), (1024, 128, 3, 256)])
def test_convert_against_cpu(k, words, q, groups):
    gen = torch.Generator().manual_seed(words)
    planes = torch.randint(-2 ** 31, 2 ** 31, (k, words, q), dtype=torch.int32, generator=gen)
    alpha = torch.randn(k // 8, groups, q, generator=gen)
    alpha[0, 0, 0] = float("nan")
    want = convert_weight(planes, alpha)
    for a in (alpha.cuda(), alpha.half().cuda(), alpha, alpha.cuda().transpose(0, 1).contiguous().transpose(0, 1)):   # fused, and the general path
        got = convert_weight(planes.cuda(), a)
        assert torch.equal(got[0].cpu(), want[0])
        ref = a.cpu().transpose(1, 2).float().contiguous()
        assert got[1].is_contiguous() and torch.allclose(got[1].cpu(), ref, rtol=0, atol=0, equal_nan=True)
