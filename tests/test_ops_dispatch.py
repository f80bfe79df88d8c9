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
