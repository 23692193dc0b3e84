"""A launch sequence whose launches do not feed one another computes ahead of the launch in front (`LaunchSequence`): same bits as one
launch after the other, eagerly, repeated and as a CUDA graph; a sequence that does feed itself is not run that way."""
import pytest
import torch

from shiftaddllm_b200 import _lib, lutgemm

pytestmark = pytest.mark.gpu


def _problem(k, n, q, seed, x=None, y=None):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    bits = torch.randint(-2 ** 31, 2 ** 31, (k // 32, q, n), dtype=torch.int32, device="cuda", generator=gen)
    alpha = torch.exp2(-torch.randint(2, 9, (k // 128, q, n), device="cuda", generator=gen).float()).half()
    x = torch.randn(1, k, device="cuda", generator=gen).half() if x is None else x
    y = torch.empty(1, n, dtype=torch.float16, device="cuda") if y is None else y
    return dict(output=y, bWeight=bits, alpha=alpha, bias=None, d_input=x, mSize=n, kSize=k, nb=q, num_groups=k // 128)


@pytest.mark.parametrize("q", [2, 3, 4])
def test_overlapped_sequence_is_bit_identical(q):
    blocks = [[_problem(k, n, q, 10 * i + j) for j, (k, n) in enumerate(((4096, 4096), (512, 264), (1024, 4096)))] for i in range(6)]
    launches = [lutgemm.prepare_grouped(b, pdl=True) for b in blocks]
    outs = [p["output"] for b in blocks for p in b]
    ins = [p["d_input"] for b in blocks for p in b]
    seq = lutgemm.LaunchSequence(launches)
    assert seq._overlap
    for rep in range(4):   # new activations written by the kernel right in front of the sequence
        for x in ins:
            x.mul_(-1.5 if rep % 2 else 0.5)
        for o in outs:
            o.fill_(float("nan"))
        seq()
        got = [o.clone() for o in outs]
        for l in launches:
            torch.cuda.synchronize()
            l()
        assert all(torch.equal(a, b) for a, b in zip(got, outs)), rep
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        seq()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            seq()
            seq()
    for o in outs:
        o.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, outs))


def test_dependent_sequences_wait():
    a = _problem(1024, 512, 3, 1)
    b = _problem(512, 1024, 3, 2, x=a["output"])
    own = _problem(512, 512, 3, 3)
    own["output"] = own["d_input"]
    plain = [lutgemm.prepare_grouped([p], pdl=True) for p in (a, b)]
    assert not lutgemm.LaunchSequence(plain)._overlap and not lutgemm.LaunchSequence(plain[::-1])._overlap
    assert not lutgemm.LaunchSequence([lutgemm.prepare_grouped([own], pdl=True)])._overlap
    assert not lutgemm.LaunchSequence([lutgemm.prepare_grouped([_problem(512, 512, 3, 4)])])._overlap     # no programmatic launch
    lutgemm.LaunchSequence(plain)()
    got = b["output"].clone()
    for l in plain:
        torch.cuda.synchronize()
        l()
    assert torch.equal(got, b["output"])
    assert _lib.load().sal_sequence_independent(None, 1) == 0
