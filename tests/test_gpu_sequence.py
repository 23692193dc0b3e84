"""A launch sequence whose launches do not feed one another computes ahead of the launch in front (`LaunchSequence`): same bits as one
launch after the other, eagerly, repeated and as a CUDA graph; a sequence that does feed itself is not run that way."""
import ctypes

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


@pytest.mark.parametrize("rows,form", [(1, "plain"), (2, "plain"), (6, "plain"), (1, "swiglu"), (3, "swiglu"), (1, "fixed"), (1, "swiglu_fixed")])
def test_later_launches_see_what_the_stream_wrote_before_the_sequence(rows, form):
    """A first launch on two CTAs and later ones on all SMs.  Every pass rewrites all operands right in front of the sequence, at the
    addresses that the pass before read."""
    flags = dict(atomic_fixed=form in ("fixed", "swiglu_fixed"), swiglu_fixed=form == "swiglu_fixed")
    gen = torch.Generator(device="cuda").manual_seed(5)
    swiglu = form.startswith("swiglu")
    operands = []

    def operand(k):
        x = torch.zeros(rows, k, dtype=torch.int64 if flags["swiglu_fixed"] else torch.float16, device="cuda")
        operands.append(x)
        return x

    blocks = []
    for i, shapes in enumerate([((256, 8),)] + 5 * [((4096, 4096), (2048, 6144))]):
        block = [_problem(k, n, 3, 10 * i + j, x=operand(k), y=torch.empty(rows, n, dtype=torch.float16, device="cuda"))
                 for j, (k, n) in enumerate(shapes)]
        for p in block:
            if swiglu:
                p["d_input_mul"] = operand(p["kSize"])
            if flags["atomic_fixed"]:
                p["output"] = torch.empty(rows, p["mSize"], dtype=torch.int64, device="cuda")
        blocks.append(block)
    launches = [lutgemm.prepare_grouped(b, pdl=True, **flags) for b in blocks]
    outs = [p["output"] for b in blocks for p in b]
    seq = lutgemm.LaunchSequence(launches)
    assert seq._overlap
    for rep in range(6):
        fresh = [torch.randn(x.shape, device="cuda", generator=gen) for x in operands]
        fresh = [f.half() if x.dtype == torch.float16 else (f.half().double() * lutgemm.FIXED_ONE).long() for f, x in zip(fresh, operands)]
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for x, f in zip(operands, fresh):
            x.copy_(f)
        seq()
        got = [o.clone() for o in outs]
        for o in outs:
            o.zero_()
        for l in launches:
            torch.cuda.synchronize()
            l()
        assert all(torch.equal(a, b) for a, b in zip(got, outs)), rep


def graph_of(fn):
    """Kernel launches, dependencies and programmatic dependencies of what `fn` enqueues, from a graph captured of it."""
    rt = ctypes.CDLL("libcudart.so.12")
    stream, graph, nodes, edges = torch.cuda.Stream(), ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_size_t()
    with torch.cuda.stream(stream):
        fn()   # scratch and the library's probe, not under capture
        torch.cuda.synchronize()
        assert rt.cudaStreamBeginCapture(ctypes.c_void_p(stream.cuda_stream), 1) == 0
        fn()
        assert rt.cudaStreamEndCapture(ctypes.c_void_p(stream.cuda_stream), ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(nodes)) == 0
    assert rt.cudaGraphGetEdges_v2(graph, None, None, None, ctypes.byref(edges)) == 0
    ends, data = ((ctypes.c_void_p * edges.value)(), (ctypes.c_void_p * edges.value)()), (ctypes.c_uint8 * (8 * edges.value))()
    assert rt.cudaGraphGetEdges_v2(graph, *ends, data, ctypes.byref(edges)) == 0
    programmatic = sum(data[8 * i + 2] == 1 for i in range(edges.value))   # cudaGraphEdgeData: from port, to port, type
    assert rt.cudaGraphDestroy(graph) == 0
    return nodes.value, edges.value, programmatic


def test_head_of_a_sequence_is_an_ordinary_launch():
    """Behind another programmatic launch, only the launches after the first of the sequence depend programmatically on the one in front."""
    front = lutgemm.prepare_grouped([_problem(512, 512, 3, 1)], pdl=True)
    seq = lutgemm.LaunchSequence([lutgemm.prepare_grouped([_problem(512, 512, 3, s)], pdl=True) for s in (2, 3, 4)])
    assert seq._overlap

    def both():
        front()
        seq()

    assert graph_of(both) == (4, 3, 2)
    assert graph_of(lambda: (front(), front())) == (2, 1, 1)
