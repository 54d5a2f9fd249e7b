"""Calls under tracers, dispatch modes and autocast: the custom kernels must leave them to operations that these see."""
import io

import pytest
import torch
import torch.nn.functional as F
from torch._subclasses import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx
from torch.utils.flop_counter import FlopCounterMode

import aussm_b200
from aussm_b200 import models, ops, stages
from tests.helpers import NAMES, model_like_inputs


def _eager_inside(run):
    seen = []

    def f(x):
        seen.append(ops._eager())
        return x * 2

    run(f)
    return seen[0]


def test_a_plain_call_is_eager():
    assert _eager_inside(lambda f: f(torch.ones(2)))
    with torch.device("cpu"):
        assert _eager_inside(lambda f: f(torch.ones(2)))


@pytest.mark.parametrize("mode", ["real", "fake", "symbolic"])
def test_make_fx_is_not_eager(mode):
    assert not _eager_inside(lambda f: make_fx(f, tracing_mode=mode)(torch.ones(2)))
    assert not _eager_inside(lambda f: make_fx(f, tracing_mode=mode, pre_dispatch=True)(torch.ones(2)))


def test_jit_trace_and_dispatch_modes_are_not_eager():
    assert not _eager_inside(lambda f: torch.jit.trace(f, torch.ones(2)))
    for mode in (FakeTensorMode(), FlopCounterMode(display=False)):
        with mode:
            assert not _eager_inside(lambda f: f(torch.ones(2)))
    assert ops._eager()


def test_shapes_propagate_with_fake_tensors():
    """No kernel may be launched on a tensor without memory: the shapes come from the operators' fake implementations."""
    with FakeTensorMode(), torch.no_grad():
        inp = {k: torch.empty(t.shape, dtype=t.dtype, device="cuda") for k, t in model_like_inputs(1, 2, 8, 4, 40).items()
               if k in NAMES}
        assert aussm_b200.ssm_adaptive_interface(**inp).shape == (2, 8, 40)
        x, w = torch.empty(3, 5, 16, device="cuda"), torch.empty(16, device="cuda")
        assert stages.rms_norm(x, w).shape == x.shape
        assert [t.shape for t in stages.rms_norm_residual(x, w)] == [x.shape, x.shape]


@pytest.mark.parametrize("convert", [torch.fx.symbolic_trace, torch.jit.script])
def test_rms_norm_can_be_converted(convert):
    norm = models.RMSNorm(8)
    x = torch.randn(3, 8)
    assert torch.equal(convert(norm)(x), norm(x))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["real", "fake", "symbolic"])
def test_a_traced_norm_computes_on_new_inputs(mode):
    x, other, w = torch.randn(6, 16, device="cuda"), torch.randn(6, 16, device="cuda"), torch.randn(16, device="cuda")
    for fn in (lambda t, v: stages.rms_norm(t, v), lambda t, v: stages.rms_norm_residual(t, v)[0]):
        graph = make_fx(fn, tracing_mode=mode)(x, w)
        expected = F.rms_norm(other.double(), (16,), w.double(), 1e-5)
        # a mean of 16 squares and five roundings
        assert (graph(other, w).double() - expected).abs().max() < 1e-6 * expected.abs().max()


@pytest.mark.gpu
def test_a_traced_operator_computes_on_new_inputs():
    first, second = ({k: t.cuda() for k, t in model_like_inputs(seed, 2, 8, 4, 48).items() if k in NAMES} for seed in (5, 6))
    with torch.no_grad():
        graph = make_fx(lambda *a: aussm_b200.ssm_adaptive_interface(*a))(*(first[k] for k in NAMES))
        got, expected = graph(*(second[k] for k in NAMES)), aussm_b200.ssm_adaptive_interface(**second)
    # the radii of B and C from another softplus: a few ulp of the 4 states' sum
    assert (got - expected).abs().max() < 2e-6 * expected.abs().max()


@pytest.mark.gpu
def test_a_jit_traced_norm_can_be_saved():
    norm = models.RMSNorm(16).cuda()
    x = torch.randn(6, 16, device="cuda")
    buffer = io.BytesIO()
    torch.jit.save(torch.jit.trace(norm, x), buffer)
    buffer.seek(0)
    assert (torch.jit.load(buffer)(x) - norm(x)).abs().max() < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("name,shape,product", [
    ("project_tokens", (2, 24, 8), lambda W, x: torch.matmul(W, x.transpose(1, 2))),
    ("project_channels", (2, 8, 24), lambda W, x: torch.matmul(W, x)),
    ("project_back", (2, 8, 24), lambda W, x: torch.matmul(x.transpose(1, 2), W.t()))])
def test_small_projections_under_autocast(name, shape, product):
    """Forward and backward, as torch.matmul does them; the backward pass runs outside of the context, as is usual."""
    W, x = (torch.randn(s, device="cuda", requires_grad=True) for s in ((12, 8), shape))
    results = []
    for fn in (getattr(stages, name), product):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = fn(W, x)
        results.append((y, *torch.autograd.grad(y.float().square().sum(), (W, x))))
    for got, expected in zip(*results):
        assert got.dtype == expected.dtype
        # products of up to 48 bf16 values in another order, rounded to bf16
        assert (got.float() - expected.float()).abs().max() < 2.0 ** -7 * expected.float().abs().max()
