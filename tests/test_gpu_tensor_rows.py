"""Several activation rows on the tensor cores (csrc/sal_mma.cu) where the kernel's edges are: column tiles of 128, row tiles of up to
256 padded to 16, units of 128 and steps of 64 features, groups that straddle a unit, planes fetched by TMA or by 4-byte copies, a tile
shared by many CTAs or none, and the scratch limits that change the split.

Reference: the same product in float64.  Bound per element: the output's fp16 rounding (2**-11 of the value, or half the smallest
subnormal) plus one fp32 rounding (2**-23, which also covers truncation) per accumulation step, of which a tile has K * q / 16 and the
sum over CTAs at most 64, each of at most the sum of the magnitudes."""
import ctypes

import pytest
import torch

from shiftaddllm_b200 import _lib, lutgemm
from shiftaddllm_b200.quant import LutLinear
from test_gpu_sequence import graph_of

pytestmark = pytest.mark.gpu


def _case(layout, m, k, n, q, g, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    bits = torch.randint(-2 ** 31, 2 ** 31, (k // 32, q, n), dtype=torch.int32, device="cuda", generator=gen)
    shape = (k // g, q, n) if layout == 0 else (k // 8, q, n // g)
    if layout == 2:
        alpha = torch.randint(0, 512, shape, device="cuda", generator=gen).to(torch.int16)
        mult = sum(torch.exp2(((alpha >> s) & 7).double()) for s in (0, 3, 6))
    else:
        alpha = (torch.exp2(-torch.randint(2, 9, shape, device="cuda", generator=gen).float())
                 * (0.5 + 0.5 * torch.rand(shape, device="cuda", generator=gen))).half()
        mult = alpha.double()
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    bias = (0.1 * torch.randn(n, device="cuda", generator=gen)).half()
    return bits, alpha, mult, x, bias


def _reference(bits, mult, x, bias):
    words, q, n = bits.shape
    signs = ((bits[:, None] >> torch.arange(32, device="cuda", dtype=torch.int32).view(1, 32, 1, 1)) & 1).reshape(32 * words, q, n).double() * 2 - 1
    scale = mult.repeat_interleave(32 * words // mult.shape[0], 0).repeat_interleave(n // mult.shape[2], 2)
    y = x.double() @ (signs * scale).sum(1) + bias.double()
    size = x.double().abs() @ scale.sum(1) + bias.double().abs()
    bound = 2.0 ** -11 * y.abs() + 2.0 ** -25 + (32 * words * q / 16 + 64) * 2.0 ** -23 * size
    return y, bound


def _call(layout, bits, alpha, x, bias, y, groups, ws, ws_bytes, flags=0):
    return _lib.load().sal_lutgemm_rows(layout, bits.data_ptr(), alpha.data_ptr(), bias.data_ptr(), x.data_ptr(), y.data_ptr(), x.shape[0],
                                        x.shape[1], bits.shape[2], bits.shape[1], groups, flags, ws.data_ptr() if ws_bytes else None, ws_bytes,
                                        torch.cuda.current_stream().cuda_stream)


# layout, rows, K, N, q, group; scratch bytes (None: what the header asks for)
CASES = [
    (0, 2, 32, 8, 1, 32, None), (0, 16, 64, 128, 2, 64, None), (0, 17, 96, 132, 3, 96, None), (0, 3, 2080, 1378, 3, 32, None),
    (0, 64, 1024, 1000, 4, 128, None), (0, 65, 128, 127, 3, 128, None), (0, 255, 512, 256, 3, 256, None), (0, 257, 384, 260, 2, 128, None),
    (0, 600, 256, 64, 3, 256, None), (0, 8, 160, 130, 3, 160, None), (0, 5, 11008, 16, 3, 128, None), (0, 1, 256, 256, 3, 128, None),
    (1, 2, 64, 16, 3, 16, None), (1, 33, 288, 96, 4, 32, None), (1, 9, 256, 144, 2, 48, None), (1, 130, 512, 512, 3, 256, None),
    (1, 1, 32, 128, 1, 128, None), (2, 12, 256, 256, 3, 16, None), (2, 70, 96, 80, 2, 16, None),
    (0, 16, 4096, 512, 3, 128, 0), (0, 16, 4096, 512, 3, 128, 16384 + 3 * 1024 * 16), (1, 40, 2048, 384, 2, 16, 0),
]


@pytest.mark.parametrize("layout,m,k,n,q,g,scratch", CASES)
def test_rows_against_float64(layout, m, k, n, q, g, scratch):
    bits, alpha, mult, x, bias = _case(layout, m, k, n, q, g)
    groups = k // g if layout == 0 else n // g
    ref, bound = _reference(bits, mult, x, bias)
    need = _lib.load().sal_lutgemm_rows_workspace_bytes(m) if scratch is None else scratch
    ws = torch.zeros(max(need, 256), dtype=torch.uint8, device="cuda")
    y = torch.full((m, n), float("nan"), dtype=torch.float16, device="cuda")
    for rep in range(2):   # the second call finds the scratch buffer as the first one left it
        assert _call(layout, bits, alpha, x, bias, y, groups, ws, need) == 0
        assert ((y.double() - ref).abs() <= bound).all(), rep
    first = y.clone()
    assert _call(layout, bits, alpha, x, bias, y, groups, ws, need, _lib.SAL_ACCUMULATE) == 0
    assert ((y.double() - ref - first.double()).abs() <= bound + 2.0 ** -11 * (ref + first.double()).abs()).all()
    if need >= 256:
        assert _lib.load().sal_workspace_status(ws.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0


def test_layer_of_many_rows_and_its_limits():
    """LutLinear takes any number of rows; rows beyond one call's limit go in further calls, and what the tensor-core product does not
    take (more than four planes) still runs 64 rows at a time."""
    for q, rows in ((3, 4100), (5, 130)):
        bits, alpha, mult, x, bias = _case(0, rows, 256, 64, q, 128, seed=q)
        lin = LutLinear(256, 64, 128, q, bias=bias)
        lin.binaryWeight = bits
        lin.set_row_alpha(alpha)
        ref, bound = _reference(bits, mult, x, bias)
        assert ((lin(x).double() - ref).abs() <= bound).all()
        wide = lin(x.float().view(2, rows // 2, 256))
        assert wide.dtype == torch.float32 and wide.shape == (2, rows // 2, 64)
    lib, y = _lib.load(), torch.empty(64, 64, dtype=torch.float16, device="cuda")
    ws = torch.zeros(lutgemm.workspace_for(y.device, 64, 64).numel(), dtype=torch.uint8, device="cuda")
    args = (_case(0, 64, 256, 64, 5, 128))
    assert _call(0, args[0], args[1], args[3], args[4], y, 2, ws, ws.numel()) == _lib.SAL_E_UNSUPPORTED
    assert lib.sal_lutgemm_rows(0, args[0].data_ptr(), args[1].data_ptr(), None, args[3].data_ptr(), y.data_ptr(), 4097, 256, 64, 4, 2, 0,
                                None, 0, None) == _lib.SAL_E_SHAPE


@pytest.mark.parametrize("m", [7, 64, 300])   # from 7 rows on
def test_grouped_rows_with_swiglu(m):
    """Problems of different widths in one launch, and the activation silu(x) * x_mul of a down projection."""
    probs, refs = [], []
    for i, (k, n) in enumerate(((256, 264), (512, 128), (256, 1000))):
        bits, alpha, mult, x, bias = _case(0, m, k, n, 3, 128, seed=i)
        y = torch.empty(m, n, dtype=torch.float16, device="cuda")
        probs.append(dict(output=y, bWeight=bits, alpha=alpha, bias=bias, d_input=x, mSize=n, kSize=k, nb=3, num_groups=k // 128))
        refs.append(_reference(bits, mult, x, bias))
    lutgemm.lutgemv_grouped(probs, pdl=True, many_rows=m > 64)
    for p, (ref, bound) in zip(probs, refs):
        assert ((p["output"].double() - ref).abs() <= bound).all()
    if m > 64:
        with pytest.raises(RuntimeError):
            lutgemm.lutgemv_grouped(probs)
    p = probs[1]
    p["d_input_mul"] = torch.randn(m, 512, device="cuda", generator=torch.Generator(device="cuda").manual_seed(9)).half()
    lutgemm.lutgemv_grouped([p], pdl=True, many_rows=m > 64)
    act = torch.nn.functional.silu(p["d_input"]) * p["d_input_mul"]
    bits, alpha, mult, _, bias = _case(0, m, 512, 128, 3, 128, seed=1)
    ref, bound = _reference(bits, mult, act, bias)
    # silu is rounded to fp16 before the product here and in torch; a last-bit difference of its exponential moves an activation by 2**-10
    assert ((p["output"].double() - ref).abs() <= bound + 2.0 ** -10 * (act.double().abs() @ mult.sum(1).repeat_interleave(128, 0))).all()


@pytest.mark.parametrize("pdl", [False, True])
def test_programmatic_launch_only_where_it_was_asked_for(pdl):
    """The two launches of a SwiGLU product: the second one may read planes and scales ahead of its dependencies only with `pdl`."""
    bits, alpha, _, x, _ = _case(0, 8, 512, 128, 3, 128)
    p = dict(output=torch.empty(8, 128, dtype=torch.float16, device="cuda"), bWeight=bits, alpha=alpha, bias=None, d_input=x, d_input_mul=x,
             mSize=128, kSize=512, nb=3, num_groups=4)
    assert graph_of(lutgemm.prepare_grouped([p], pdl=pdl)) == (2, 1, int(pdl))


@pytest.mark.parametrize("m", [16, 1])   # tensor-core and table kernel
def test_a_long_kernel_in_front_does_not_run_the_waits_out(m):
    """Programmatic launches start while the ones in front still run, and their waits are limited to about a second each.  Four products of one
    CTA and some tenths of a second each in front: the time of those must not count."""
    k, lib = 1 << 27, _lib.load()
    long_bits = torch.zeros(k // 32, 4, 8, dtype=torch.int32, device="cuda")
    long_alpha, long_x = torch.ones(1, 4, 8, dtype=torch.float16, device="cuda"), torch.zeros(2, k, dtype=torch.float16, device="cuda")
    long_y = torch.empty(2, 8, dtype=torch.float16, device="cuda")
    bits, alpha, _, x, bias = _case(0, m, 8192, 512, 3, 128)
    ws = torch.zeros(lib.sal_lutgemm_rows_workspace_bytes(64), dtype=torch.uint8, device="cuda")
    y = torch.empty(m, 512, dtype=torch.float16, device="cuda")

    def product():
        assert lib.sal_lutgemv_shift_scale(bits.data_ptr(), alpha.data_ptr(), bias.data_ptr(), x.data_ptr(), y.data_ptr(), m, 8192, 512, 3, 64,
                                           _lib.SAL_PDL, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream) == 0

    product()
    want = y.clone()
    y.zero_()
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record()
    for _ in range(4):
        assert lib.sal_lutgemm_rows(0, long_bits.data_ptr(), long_alpha.data_ptr(), None, long_x.data_ptr(), long_y.data_ptr(), 2, k, 8, 4, 1,
                                    _lib.SAL_PDL, ws.data_ptr(), 256, torch.cuda.current_stream().cuda_stream) == 0
    product()
    end.record()
    torch.cuda.synchronize()
    assert begin.elapsed_time(end) > 1500   # otherwise this shows nothing
    assert torch.equal(y, want)
    assert lib.sal_workspace_status(ws.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("layout,m,k,n,q,g", [(0, 8, 20480, 256, 3, 128), (0, 3, 2080, 130, 3, 32), (0, 64, 4096, 264, 2, 64), (1, 16, 4096, 384, 3, 32),
                                              (2, 9, 8192, 96, 2, 16)])
def test_the_same_call_has_the_same_bits_whatever_the_scratch_grew_to(layout, m, k, n, q, g):
    """Through a layer, a first call on a stream against the same call after a larger one, and through the C interface with the scratch that
    the header asks for against more of it.  The split over CTAs decides the last bits."""
    bits, alpha, _, x, bias = _case(layout, m, k, n, q, g)
    lin = LutLinear(k, n, g if layout == 0 else 8 * g, q, bias=bias)
    lin.binaryWeight, lin.alpha, lin.alpha_layout = bits, alpha, "row" if layout == 0 else "block"
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        first = lin(x)
        lin(x.repeat(200, 1)[:300])
        assert torch.equal(lin(x), first)
    torch.cuda.synchronize()
    asked = _lib.load().sal_workspace_bytes(m, n)
    ys = []
    for size in (asked, 2 * asked, 1 << 28):
        ws, y = torch.zeros(size, dtype=torch.uint8, device="cuda"), torch.empty(m, n, dtype=torch.float16, device="cuda")
        assert _call(layout, bits, alpha, x, bias, y, k // g if layout == 0 else n // g, ws, size) == 0
        ys.append(y)
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])


def test_little_scratch_and_more_tiles_than_sms():
    """Scratch for three CTAs where 150 column tiles have to be done: one CTA per tile."""
    bits, alpha, mult, x, bias = _case(0, 16, 256, 150 * 128, 2, 128)
    ref, bound = _reference(bits, mult, x, bias)
    y = torch.empty(16, 150 * 128, dtype=torch.float16, device="cuda")
    size = 16384 + 3 * 1024 * 16
    ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
    assert _call(0, bits, alpha, x, bias, y, 2, ws, size) == 0
    assert ((y.double() - ref).abs() <= bound).all() and not ws[256:].any()


@pytest.mark.parametrize("layout,m,k,n,q,g", [(0, 8, 2048, 264, 3, 128), (0, 40, 512, 128, 2, 512), (0, 5, 2080, 130, 3, 32), (0, 300, 512, 64, 4, 256),
                                              (1, 9, 1024, 144, 3, 16), (1, 70, 288, 768, 2, 48)])
def test_infinite_and_nan_operands_as_in_the_tables(layout, m, k, n, q, g):
    """Infinite scales, alone and several in a column, NaN scales, and infinite and NaN activations: where a row of one gives an infinity (of
    which sign) or NaN, so do many; everywhere else the elements stay within the bound.  `m` rows are tensor-core work, one row is the tables'."""
    bits, alpha, mult, x, bias = _case(layout, m, k, n, q, g)
    ref, bound = _reference(bits, mult, x, bias)
    inf, nan = float("inf"), float("nan")
    alpha[0, 0, 1], alpha[-1, q - 1, 2], alpha[0, q - 1, 3], alpha[-1, 0, 3], alpha[0, 0, 5] = inf, -inf, inf, inf, nan
    x[1, 7], x[2, k - 1], x[3, 11] = inf, -inf, nan
    lin = LutLinear(k, n, g if layout == 0 else 8 * g, q, bias=bias)
    lin.binaryWeight, lin.alpha, lin.alpha_layout = bits, alpha, "row" if layout == 0 else "block"
    got, want = lin(x), torch.cat([lin(x[i:i + 1]) for i in range(m)])
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(torch.where(got.isinf(), got, 0), torch.where(want.isinf(), want, 0))
    finite = got.isfinite()
    assert finite.sum() >= (m - 3) * n // 2 and got.isinf().any() and got.isnan().any()
    assert ((got.double() - ref).abs() <= bound)[finite].all()


def _block_sizes(fn):
    """Threads per block of the kernels that `fn` enqueues."""
    drv, stream, graph, count = ctypes.CDLL("libcuda.so.1"), torch.cuda.Stream(), ctypes.c_void_p(), ctypes.c_size_t()
    with torch.cuda.stream(stream):
        fn()
        torch.cuda.synchronize()
        assert drv.cuStreamBeginCapture_v2(ctypes.c_void_p(stream.cuda_stream), 1) == 0
        fn()
        assert drv.cuStreamEndCapture(ctypes.c_void_p(stream.cuda_stream), ctypes.byref(graph)) == 0
    assert drv.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert drv.cuGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    sizes = []
    for node in nodes:
        params = (ctypes.c_uint32 * 32)()   # CUDA_KERNEL_NODE_PARAMS: function, grid x y z, block x y z, ..
        assert drv.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), params) == 0
        sizes.append(params[5])
    assert drv.cuGraphDestroy(graph) == 0
    return sizes


@pytest.mark.parametrize("layout,m,k,n,q,g,tensor", [(1, 4, 768, 768, 3, 16, False), (1, 4, 2048, 512, 3, 16, False), (1, 32, 768, 768, 3, 16, False),
                                                     (1, 6, 2048, 2048, 3, 16, True), (1, 6, 2048, 2048, 3, 128, False), (1, 4, 11008, 4096, 3, 16, True),
                                                     (2, 4, 4096, 4096, 2, 128, False), (1, 3, 4096, 4096, 4, 16, False), (1, 64, 512, 2048, 2, 16, True)])
def test_block_layouts_run_where_they_are_faster(layout, m, k, n, q, g, tensor):
    """The table kernel has 288 threads, the tensor-core kernel 736; both within the bound on either side of the line."""
    bits, alpha, mult, x, bias = _case(layout, m, k, n, q, g)
    ref, bound = _reference(bits, mult, x, bias)
    y = torch.empty(m, n, dtype=torch.float16, device="cuda")

    def call():
        lutgemm.lutgemm_block_fused(y, bits, alpha, bias, x, n, k, q, n // g)

    assert _block_sizes(call) == [736 if tensor else 288]
    call()
    assert ((y.double() - ref).abs() <= bound).all()
