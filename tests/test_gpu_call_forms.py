"""Forms in which a program calls the differentiable entry points: traced,
checkpointed, from several streams and threads, from a restored module, out of
memory, and under the transforms that they refuse."""
import copy
import threading

import pytest
import torch
from torch.utils.checkpoint import checkpoint

from dmgs_gb300.texture import MLPTexture3D
from test_gpu_native_nodes import D, OPS, _gen, _run, _same

pytestmark = pytest.mark.gpu


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("op", ["loss", "sh", "bind2", "bind3", "texture", "raster-sh", "flexicubes-none"])
def test_a_traced_call_follows_its_input(op):
    """torch.jit.trace records the call: another input gives that input's result."""
    tensors, fn = OPS[op]()
    name = next(iter(tensors))
    rest = {k: v.detach() for k, v in tensors.items() if k != name}
    for v in tensors.values():  # a module's parameters: constants of the trace
        v.requires_grad_(False)
    x0 = tensors[name].detach()
    x1 = x0 * 0.9 + 0.01

    def call(x):
        return fn(**{name: x}, **rest)[0]
    traced = torch.jit.trace(call, (x0,), check_trace=False)
    assert torch.equal(traced(x0), call(x0))
    assert torch.equal(traced(x1), call(x1))
    assert not torch.equal(traced(x1), traced(x0))


@pytest.mark.parametrize("op", list(OPS))
def test_checkpointed_calls_have_the_same_gradients(op):
    def wrapped():
        tensors, fn = OPS[op]()
        names = list(tensors)
        return tensors, lambda **k: checkpoint(lambda *a: fn(**dict(zip(names, a))), *[k[n] for n in names], use_reentrant=False)
    a, b = _run(wrapped), _run(OPS[op])
    a = (a[0], a[1], a[2])
    _same(a, b)


@pytest.mark.parametrize("op", list(OPS))
def test_streams_and_threads(op):
    """Each of four threads on its own stream, twice over."""
    want = _run(OPS[op])
    got, errors = [None] * 4, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(2):
                    got[i] = _run(OPS[op])
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    torch.cuda.synchronize()
    if op == "texture":  # its inputs are made with the process's one CPU generator
        threads = threads[:1]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for r in got[:len(threads)]:
        _same(r, want)


@pytest.mark.parametrize("op", ["loss", "sh", "bind2", "bind3", "texture", "raster-sh", "flexicubes-none"])
def test_transforms_are_refused(op):
    tensors, fn = OPS[op]()
    name = next(iter(tensors))
    rest = {k: v.detach() for k, v in tensors.items() if k != name}
    x = tensors[name].detach()

    def total(x):
        return fn(**{name: x}, **rest)[0].sum()
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.grad(total)(x)
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.vmap(total)(torch.stack([x, x]))
    with torch.autograd.forward_ad.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError)):
            total(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))


def test_out_of_memory_keeps_its_type():
    """An allocation that the process's memory limit refuses is torch's OutOfMemoryError, from any entry."""
    x = torch.rand(3, 1500, 1500, device=D)
    y = torch.rand(3, 1500, 1500, device=D)
    from dmgs_gb300.loss import l1_ssim_loss
    l1_ssim_loss(x[:, :8, :8].contiguous(), y[:, :8, :8].contiguous())
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    try:
        torch.cuda.set_per_process_memory_fraction(2e-4)
        with pytest.raises(torch.OutOfMemoryError):
            l1_ssim_loss(x, y)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert bool(torch.isfinite(l1_ssim_loss(x, y)))


def test_restored_texture_module():
    """A module whose host copy of the box was made by an earlier version (or
    is not there) is used like a new one."""
    m = MLPTexture3D(torch.tensor([[-1.0] * 3, [1.0] * 3]), channels=3, device=D)
    x = 2 * torch.rand(50, 3, device=D, generator=_gen(3)) - 1
    want = m.sample_noact(x)
    assert "_aabb_cache" in m.__dict__
    r = copy.deepcopy(m)
    for k in [k for k in r.__dict__ if k.startswith("_aabb") and k not in ("_aabb_src", "_aabb_ver", "_aabb_cache")]:
        del r.__dict__[k]
    r._aabb_src, r._aabb_ver = r.AABB, r.AABB._version  # as a whole-module pickle restores them
    assert torch.equal(r.sample_noact(x), want)
    r.AABB = torch.tensor([[-2.0] * 3, [2.0] * 3])
    assert not torch.equal(r.sample_noact(x), want)
