"""The operator's place in torch's machinery: its graph node, traces, function transforms, forward mode."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _make(kind, precision="exact"):
    """(callable, its tensor arguments as leaves that want gradients)"""
    import deform_conv3d_pytorch_op_b200 as dcn
    g = torch.Generator(device="cuda").manual_seed(7)

    def leaf(*shape, std=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * std).requires_grad_(True)

    x, w, b = leaf(2, 16, 13, 12), leaf(24, 16, 3, 3, std=0.1), leaf(24)
    if kind == "deform":
        return (lambda x, off, w, b: dcn.ConvOffset2dFunction.apply(x, off, w, b, 1, 1, 1, 16, 1, precision),
                [x, leaf(2, 18, 13, 12), w, b])
    if kind == "plain":
        return lambda x, w, b: dcn.Conv2dFunction.apply(x, w, b, 1, 1, 1, 1, precision), [x, w, b]
    return (lambda x, ow, ob, w, b: dcn.DeformLayerFunction.apply(x, ow, ob, w, b, 1, 1, 1, 16, 1, precision),
            [x, leaf(18, 16, 3, 3, std=0.05), leaf(18, std=0.1), w, b])


def _close(a, b):
    # exact precision: the same sums of at most 16 * 9 products, the gradients' in another order
    return torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max()))


KINDS = ["deform", "plain", "layer"]


@pytest.mark.parametrize("kind", KINDS)
def test_a_trace_records_the_operation(kind):
    fn, args = _make(kind)
    traced = torch.jit.trace(fn, tuple(a.detach() for a in args), check_trace=False)
    other = [(a.detach() * 0.5 + 0.1).requires_grad_(True) for a in args]
    y, want = traced(*other), fn(*other)
    assert _close(y, want)
    dy = torch.randn_like(y)
    for a, b in zip(torch.autograd.grad(y, other, dy), torch.autograd.grad(want, other, dy)):
        assert _close(a, b)


@pytest.mark.parametrize("kind", KINDS)
def test_transforms_and_forward_mode_are_refused_by_torch(kind):
    import torch.autograd.forward_ad as fw
    fn, args = _make(kind)
    args = [a.detach() for a in args]
    for i in (0, len(args) - 1):
        def of(v):
            return fn(*args[:i], v, *args[i + 1:])
        with pytest.raises(RuntimeError, match="setup_context"):
            torch.func.grad(lambda v: of(v).sum())(args[i])
        with pytest.raises(RuntimeError, match="setup_context"):
            torch.vmap(of)(torch.stack([args[i]] * 2))
        with pytest.raises(RuntimeError, match="setup_context"):
            torch.func.functionalize(of)(args[i])
        with fw.dual_level(), pytest.raises(NotImplementedError):
            of(fw.make_dual(args[i], torch.ones_like(args[i])))
    assert torch.isfinite(fn(*args)).all()


def test_compiled_callers_keep_the_operation():
    fn, args = _make("deform")
    compiled = torch.compile(lambda x, *rest: fn(x * 2, *rest).relu(), backend="aot_eager")
    y, want = compiled(*args), fn(args[0] * 2, *args[1:]).relu()
    assert _close(y, want)
    for a, b in zip(torch.autograd.grad(y.sum(), args), torch.autograd.grad(want.sum(), args)):
        assert _close(a, b)


def _held(fn, args, base):
    """Bytes that a forward pass leaves allocated beside its output (and, for a layer, the offsets it saves)."""
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    y = fn(*args)
    return torch.cuda.memory_allocated() - before - base, y


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("precision", ["exact", "bf16"])
def test_what_stays_allocated_until_the_backward_pass(kind, precision):
    fn, args = _make(kind, precision)
    fn(*args)                                                        # (module loading)
    pages = lambda n: (n + 511) // 512 * 512
    base = pages(2 * 24 * 13 * 12 * 4) + (pages(2 * 18 * 13 * 12 * 4) if kind == "layer" else 0)
    held, y = _held(fn, args, base)
    assert held <= (pages(args[0].numel() * 2 + 255) if precision == "bf16" else 0)     # at most the bf16 input copy
    want = torch.autograd.grad(y.square().sum(), args)
    del y
    # with hooks on saved tensors nothing stays beside the tensors that the hooks were given
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda v: (seen.append(v.shape), v.cpu())[1], lambda v: v.cuda()):
        held, y = _held(fn, args, pages(2 * 24 * 13 * 12 * 4))
    assert held <= 0 and len(seen) == {"deform": 3, "plain": 2, "layer": 4}[kind]
    tol = 1e-4 if precision == "exact" else 2e-2
    for a, b in zip(torch.autograd.grad(y.square().sum(), args), want):
        assert torch.allclose(a, b, rtol=tol, atol=tol * float(b.abs().max()))


@pytest.mark.parametrize("precision", ["exact", "bf16"])
def test_tensors_that_do_not_match_are_refused_alike(precision):
    import deform_conv3d_pytorch_op_b200 as dcn
    x, w, off = torch.zeros(2, 16, 9, 9).cuda(), torch.zeros(16, 16, 3, 3).cuda(), torch.zeros(2, 18, 9, 9).cuda()
    for fmt in (torch.contiguous_format, torch.channels_last):
        xf = x.contiguous(memory_format=fmt)
        op = dcn.Op(xf, w, 1, 1, 1, 16, 1, precision=precision)
        for o, u in ((off.double(), w), (off.cpu(), w), (off[:, :9], w), (off, w.double()), (off, w.cpu())):
            texts = []
            for call in (lambda: op.forward(xf, o, u),
                         lambda: dcn.ConvOffset2dFunction.apply(xf, o, u, None, 1, 1, 1, 16, 1, precision)):
                with pytest.raises(dcn.DcnError) as e:
                    call()
                texts.append(str(e.value))
            assert texts[0] == texts[1]


def test_a_second_backward_pass():
    for kind in KINDS:
        fn, args = _make(kind)
        y = fn(*args)
        dy = torch.randn_like(y)
        first = torch.autograd.grad(y, args, dy, retain_graph=True)
        for a, b in zip(torch.autograd.grad(y, args, dy), first):
            assert _close(a, b)
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(y, args, dy)


@pytest.mark.parametrize("kind", KINDS)
def test_gradients_of_gradients_are_refused(kind):
    fn, args = _make(kind)
    y = fn(*args)
    dy = torch.ones_like(y, requires_grad=True)
    g = torch.autograd.grad(y, args, dy, create_graph=True)
    assert all(v.requires_grad for v in g)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        sum(v.sum() for v in g).backward()


@pytest.mark.parametrize("kind", KINDS)
def test_a_change_in_place_before_the_backward_pass_is_refused(kind):
    for i in range(len(_make(kind)[1]) - 1):                         # the last is the bias, which the gradients do not read
        fn, args = _make(kind)
        if kind == "layer" and i == 2:                               # (so is the offset-producing convolution's)
            continue
        y = fn(*args)
        with torch.no_grad():
            args[i].mul_(2)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            y.sum().backward()


@pytest.mark.parametrize("precision", ["exact", "bf16"])
@pytest.mark.parametrize("kind", KINDS)
def test_gradients_for_some_inputs_only(kind, precision):
    fn, args = _make(kind, precision)
    y = fn(*args)
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, args, dy)
    tol = 1e-4 if precision == "exact" else 2e-2
    for mask in range(1, 2 ** len(args)):
        some = [a.detach().requires_grad_(bool(mask >> i & 1)) for i, a in enumerate(args)]
        got = torch.autograd.grad(fn(*some), [a for a in some if a.requires_grad], dy)
        for a, b in zip(got, [b for i, b in enumerate(want) if mask >> i & 1]):
            assert torch.allclose(a, b, rtol=tol, atol=tol * float(b.abs().max())), mask
    with torch.no_grad():
        assert fn(*args).grad_fn is None


@pytest.mark.parametrize("precision", ["exact", "bf16"])
def test_threads_with_streams_of_their_own(precision):
    """Four threads, each on its own stream, run steps of a layer and of the operator at the same time."""
    import threading
    made = [_make(kind, precision) for kind in ("deform", "layer", "plain", "deform")]
    want = []
    for fn, args in made:
        y = fn(*args)
        want.append((y.detach(),) + torch.autograd.grad(y, args, torch.ones_like(y)))
    torch.cuda.synchronize()
    got, errors = [None] * len(made), []

    def work(i):
        try:
            fn, args = made[i]
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    y = fn(*args)
                    g = torch.autograd.grad(y, args, torch.ones_like(y))
                torch.cuda.current_stream().synchronize()
                got[i] = (y.detach(),) + g
        except Exception as e:                                       # handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(made))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    tol = 1e-4 if precision == "exact" else 2e-2
    for a, b in zip(sum(got, ()), sum(want, ())):
        assert torch.allclose(a, b, rtol=tol, atol=tol * float(b.abs().max()))
