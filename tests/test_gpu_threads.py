"""Host threads that enqueue on one stream, and so share its scratch buffer: every product has the bits it has alone."""
import threading

import pytest
import torch

from shiftaddllm_b200 import lutgemm

pytestmark = pytest.mark.gpu


def _problem(k, n, m, q, seed, swiglu=False):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    bits = torch.randint(-2 ** 31, 2 ** 31, (k // 32, q, n), dtype=torch.int32, device="cuda", generator=gen)
    alpha = torch.exp2(-torch.randint(2, 9, (k // 128, q, n), device="cuda", generator=gen).float()).half()
    p = dict(output=torch.zeros(m, n, dtype=torch.float16, device="cuda"), bWeight=bits, alpha=alpha, bias=None,
             d_input=torch.randn(m, k, device="cuda", generator=gen).half(), mSize=n, kSize=k, nb=q, num_groups=k // 128)
    if swiglu:
        p["d_input_mul"] = torch.randn(m, k, device="cuda", generator=gen).half()
    return p


def _run(work):
    """One thread per list of launches, all on one stream, started together."""
    stream, start, errors = torch.cuda.Stream(), threading.Barrier(len(work)), []
    torch.cuda.synchronize()

    def thread(launches):
        try:
            with torch.cuda.stream(stream):
                start.wait()
                for launch in launches:
                    launch()
        except Exception as e:   # noqa: BLE001 - reported by the test
            errors.append(e)

    threads = [threading.Thread(target=thread, args=(w,)) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors


def test_swiglu_rows_and_split_products_from_two_threads():
    """silu(x) * x_mul of several rows passes through the scratch buffer from one launch to the next; so do the partial sums of the
    others, inside one launch."""
    shapes = [(512, 256, 8, True), (2048, 512, 16, True), (1024, 4096, 1, False), (1024, 1024, 8, False)]
    problems = [[_problem(k, n, m, 3, 100 * t + i, sw) for i, (k, n, m, sw) in enumerate(24 * shapes)] for t in range(2)]
    work = [[lutgemm.prepare_grouped([p], pdl=bool(i & 1)) for i, p in enumerate(ps)] for ps in problems]
    for launches in work:   # alone
        for launch in launches:
            launch()
    torch.cuda.synchronize()
    alone = [[p["output"].clone() for p in ps] for ps in problems]
    for rep in range(4):
        for ps in problems:
            for p in ps:
                p["output"].zero_()
        _run(work)
        for t, ps in enumerate(problems):
            assert all(torch.equal(p["output"], a) for p, a in zip(ps, alone[t])), (rep, t)


def test_launches_of_different_shared_memory_from_several_threads():
    """Products whose plans ask the same kernel for different amounts of shared memory (rows, small groups, plain copies): every launch goes
    through, whichever thread was there first."""
    shapes = [(512, 256, 300, 128), (512, 264, 7, 128), (512, 512, 130, 128), (512, 128, 17, 128)]
    work, problems = [], []
    for t in range(4):
        ps = [_problem(*shapes[(i + t) % 4][:3], 1, 10 * t + i) for i in range(8)]
        problems += ps
        work.append(200 * [lutgemm.prepare_grouped([p], many_rows=True) for p in ps])
    for launches in work:
        for launch in launches[:8]:
            launch()
    torch.cuda.synchronize()
    alone = [p["output"].clone() for p in problems]
    _run(work)
    assert all(torch.equal(p["output"], a) for p, a in zip(problems, alone))
