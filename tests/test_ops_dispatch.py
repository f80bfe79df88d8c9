"""ops.call runs an operator's implementation directly only for plain calls: everything that has to
see the operator (autograd, tracing, modes, transforms, profilers) still goes through it."""
import pytest
import torch


def _seen(run):
    """What ops._plain says of one tensor argument inside ``run``."""
    from hellblast_b200 import ops
    got = []
    run(lambda t: got.append(ops._plain((t, 3, None))))
    return got[-1]


def _vmap(f):
    def g(t):
        f(t)
        return t
    torch.func.vmap(g)(torch.ones(2, 3))


def _forward_ad(f):
    with torch.autograd.forward_ad.dual_level():
        f(torch.ones(2))


def _fake(f):
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        f(torch.ones(2))


def _function_mode(f):
    class M(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with M():
        f(torch.ones(2))


def _trace(f):
    def g(t):
        f(t)
        return t + 1
    torch.jit.trace(g, torch.ones(2), check_trace=False)


def _profile(f):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        f(torch.ones(2))


def test_plain_calls_only():
    assert _seen(lambda f: f(torch.ones(2)))
    leaf = torch.ones(2, requires_grad=True)
    assert not _seen(lambda f: f(leaf))
    with torch.no_grad():
        assert _seen(lambda f: f(leaf))
        assert not _seen(lambda f: f(torch.nn.Parameter(torch.ones(2))))


@pytest.mark.parametrize("run", [_vmap, _forward_ad, _fake, _function_mode, _trace, _profile], ids=lambda r: r.__name__)
def test_contexts_use_the_operator(run):
    assert not _seen(run)


@pytest.mark.gpu
def test_same_result_and_same_autograd_behaviour():
    import hellblast_b200 as hb
    m = torch.randn(2, 12 * 64, device="cuda")
    direct = hb.hp_compat.map2alm(m, lmax=20)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        through = hb.hp_compat.map2alm(m, lmax=20)
    assert torch.equal(direct, through)
    a = hb.hp_compat.map2alm(m.requires_grad_(True), lmax=20)
    assert a.requires_grad
    with pytest.raises(RuntimeError):  # no gradient formula on this entry point: an error, not zeros
        a.abs().sum().backward()


def _lazy(t):
    """Tensors whose storage is not their value: still to be conjugated or negated."""
    z = torch.complex(t, t + 1)
    return {"conj": z.conj(), "neg": torch._neg_view(t)}


@pytest.mark.parametrize("kind", ["conj", "neg"])
def test_lazy_tensors_use_the_operator(kind):
    from hellblast_b200 import ops
    x = _lazy(torch.ones(2, 3))[kind]
    assert not ops._plain((x, 3, None))
    assert not ops._plain((torch.ones(2), 3, x))


@pytest.mark.gpu
def test_conjugated_inputs():
    import hellblast_b200 as hb
    gen = torch.Generator(device="cuda").manual_seed(1)
    lmax, nside = 40, 16
    a, b = (torch.randn(2, hb.alm_ops.alm_size(lmax), dtype=torch.complex128, device="cuda", generator=gen) for _ in range(2))
    for dt in (torch.complex128, torch.complex64):
        x, y = a.to(dt), b.to(dt)
        xc, yc = x.conj().resolve_conj(), y.conj().resolve_conj()
        assert torch.equal(hb.hp_compat.alm2map(x.conj(), nside), hb.hp_compat.alm2map(xc, nside))
        for got, want in zip(hb.hp_compat.alm2map_spin(x.conj(), y.conj(), 2, nside), hb.hp_compat.alm2map_spin(xc, yc, 2, nside)):
            assert torch.equal(got, want)
        want = hb.hp_compat.alm2cl(xc, y)
        assert not torch.equal(want, hb.hp_compat.alm2cl(x, y))
        assert torch.equal(hb.hp_compat.alm2cl(x.conj(), y), want)
        assert torch.equal(hb.hp_compat.alm2cl(xc, yc.conj()), want)


@pytest.mark.gpu
def test_gradients_that_arrive_conjugated():
    """autograd hands a backward pass lazily conjugated gradients: against a dense transform whose rows are the
    transforms of the unit maps (1e-12 relative: FP64 sums of 48 terms)."""
    import hellblast_b200 as hb
    nside, lmax = 2, 4
    npix = 12 * nside * nside
    gen = torch.Generator(device="cuda").manual_seed(2)
    n = hb.alm_ops.alm_size(lmax)
    w, v = (torch.randn(1, n, dtype=torch.complex128, device="cuda", generator=gen) for _ in range(2))
    eye, none = torch.eye(npix, dtype=torch.float64, device="cuda"), torch.zeros(npix, npix, dtype=torch.float64, device="cuda")

    def check(x, transform, dense, loss):
        grads = []
        for f in (transform, dense):
            y = [t.clone().requires_grad_(True) for t in x]
            loss(f(*y)).backward()
            grads.append([t.grad for t in y])
        for g, want in zip(*grads):
            assert torch.linalg.norm(g - want) < 1e-12 * torch.linalg.norm(want)

    def loss(alms):
        return sum((a.conj() * k).sum().abs() for a, k in zip(alms, (w, v)))

    m = torch.randn(2, 1, npix, dtype=torch.float64, device="cuda", generator=gen)
    Y = hb.autograd.map2alm(eye, nside, lmax)
    check([m[0]], lambda t: [hb.autograd.map2alm(t, nside, lmax)], lambda t: [t.to(Y.dtype) @ Y], loss)
    (EQ, BQ), (EU, BU) = hb.autograd.map2alm_spin(eye, none, nside, lmax), hb.autograd.map2alm_spin(none, eye, nside, lmax)
    check([m[0], m[1]], lambda q, u: hb.autograd.map2alm_spin(q, u, nside, lmax),
          lambda q, u: (q.to(EQ.dtype) @ EQ + u.to(EU.dtype) @ EU, q.to(BQ.dtype) @ BQ + u.to(BU.dtype) @ BU), loss)


@pytest.mark.parametrize("kind", ["meta", "zero"])
def test_tensors_without_storage_use_the_operator(kind):
    from hellblast_b200 import ops
    x = torch.ones(2, 3, device="meta") if kind == "meta" else torch._efficientzerotensor((2, 3))
    assert not ops._plain((x, 3, None))
    assert not ops._plain((torch.ones(2), 3, x))


@pytest.mark.gpu
def test_meta_tensors_give_shapes():
    import hellblast_b200 as hb
    a = hb.hp_compat.map2alm(torch.empty(3, 12 * 16 * 16, device="meta"), lmax=20)
    assert a.is_meta and a.shape == (3, hb.alm_ops.alm_size(20)) and a.dtype == torch.complex64


@pytest.mark.parametrize("owner,name", [
    (torch._C, "_len_torch_dispatch_stack"), (torch._C, "_len_torch_function_stack"), (torch._C._functorch, "peek_interpreter_stack"),
    (torch._C, "_get_tracing_state"), (torch.autograd.forward_ad, "_current_level"), (torch.autograd, "_profiler_enabled")],
    ids=lambda v: v if isinstance(v, str) else "")
def test_a_torch_without_an_internal_query_uses_the_operator(monkeypatch, owner, name):
    from hellblast_b200 import ops
    t = torch.ones(2)
    assert ops._plain((t,))
    with monkeypatch.context() as m:
        m.delattr(owner, name)
        plain = ops._plain((t,))
    assert not plain


@pytest.mark.gpu
def test_stream_without_the_shortcut(monkeypatch):
    from hellblast_b200 import ops
    dev = torch.device("cuda", 0)
    with torch.cuda.stream(torch.cuda.Stream(dev)):
        want = torch.cuda.current_stream(dev).cuda_stream
        assert ops._stream(dev) == want
        with monkeypatch.context() as m:
            m.delattr(torch._C, "_cuda_getCurrentRawStream")
            got = ops._stream(dev)
    assert got == want
