"""Calls that return numbers (norms, inner products) come back when the numbers
are there, not when the stream is idle: by then everything the call has written
can be read on any stream, and a call that waits long returns the same numbers."""
import pytest

gpu = pytest.mark.gpu


def _need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _field(g, dims, prec, n_rhs, seed):
    import torch

    lay = g.layout.get(g.grid(dims, prec), 1, n_rhs, five_d=False)
    x = g.lattice(lay, g.full)
    gen = torch.Generator("cuda").manual_seed(seed)
    n = x.tensor.numel() * 24 // prec.nbytes  # reals
    v = torch.randn(n, dtype=torch.float64 if prec is g.double else torch.float32, device="cuda", generator=gen)
    x.tensor.copy_(v.view(torch.uint8))
    return x


# (one-warp blocks: one right-hand side on small fields; 24 threads and more per block: packed ones)
@gpu
@pytest.mark.parametrize("dims,n_rhs", [((4, 4, 4, 4), 1), ((8, 8, 8, 8), 1), ((8, 8, 8, 8), 3), ((12, 12, 12, 16), 1)])
@pytest.mark.parametrize("prec", ["double", "single"])
def test_axpy_norm2_output_is_complete_for_a_second_stream(dims, n_rhs, prec):
    _need_gpu()
    import torch

    import gpt_gb300 as g

    pr = getattr(g, prec)
    x, y = _field(g, list(dims), pr, n_rhs, 1), _field(g, list(dims), pr, n_rhs, 2)
    dt = torch.float64 if prec == "double" else torch.float32
    xs, ys = x.tensor.view(dt), y.tensor.view(dt)
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    for i in range(50):
        out = x.new()
        a = 0.25 + i
        got = torch.empty_like(xs)
        torch.cuda.synchronize()
        with torch.cuda.stream(first):
            g.axpy_norm2(out, a, x, y)
        with torch.cuda.stream(second):  # no event, no synchronisation between the two streams
            got.copy_(out.tensor.view(dt))
        torch.cuda.synchronize()
        want = torch.addcmul(ys, xs, torch.full_like(xs, a))
        assert torch.allclose(got, want, rtol=1e-12 if prec == "double" else 1e-5, atol=1e-12 if prec == "double" else 1e-4), i


@gpu
def test_results_behind_long_queued_work():
    """The call comes milliseconds before its own launch can start."""
    _need_gpu()
    import torch

    import gpt_gb300 as g

    x = _field(g, [8, 8, 8, 8], g.double, 1, 3)
    ref = float((x.tensor.view(torch.float64) ** 2).sum())
    ref_ip = g.inner_product(x, x)
    a = torch.randn(8192, 8192, device="cuda")
    b = torch.empty_like(a)
    torch.mm(a, a, out=b)
    torch.cuda.synchronize()
    for _ in range(3):
        for _ in range(4):
            torch.mm(a, a, out=b)
        assert abs(g.norm2(x) - ref) < 1e-12 * ref
        for _ in range(4):
            torch.mm(a, a, out=b)
        assert g.inner_product(x, x) == ref_ip
    torch.cuda.synchronize()


@gpu
@pytest.mark.parametrize("call", ["norm2", "inner_product", "axpy_norm2"])
def test_work_queued_before_the_call_has_completed(call):
    _need_gpu()
    import torch

    import gpt_gb300 as g

    x, y = _field(g, [8, 8, 8, 8], g.double, 1, 4), _field(g, [8, 8, 8, 8], g.double, 1, 5)
    out = x.new()
    a = torch.randn(4096, 4096, device="cuda")
    b = torch.mm(a, a)
    run = {"norm2": lambda: g.norm2(x), "inner_product": lambda: g.inner_product(x, y),
           "axpy_norm2": lambda: g.axpy_norm2(out, 0.5, x, y)}[call]
    run()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for n in (0, 1, 8):
            for _ in range(n):
                torch.mm(a, a, out=b)
            before = torch.cuda.Event()
            before.record()
            run()
            assert before.query(), n
    torch.cuda.synchronize()
