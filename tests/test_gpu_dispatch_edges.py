"""Kernel variants and dispatch rules at the sizes where they can go wrong, against the float64 oracle."""
import math

import pytest
import torch
import torch.nn.functional as F

import aussm_b200
from aussm_b200 import _lib, ops, stages, variants
from aussm_b200.s6 import selective_scan_fn
from oracle import unitary as O
from oracle.s6 import selective_scan_ref
from oracle.variants import scan_complex_ref
from tests.helpers import NAMES, model_like_inputs, scaled_error, scan_core_inputs

pytestmark = pytest.mark.gpu

SCAN_KEYS = ["theta", "u", "dt", "z", "B_r", "B_theta", "C_r", "C_theta", "D", "h0_re", "h0_im"]


def scan_errors(b, d, n, l, seed):
    """Largest error of every output and gradient of the scan core, relative to the tensor's largest magnitude."""
    inp = scan_core_inputs(seed, b, d, n, l)
    results = []
    for dev, dtype, fn in (("cpu", torch.float64, O.scan_unitary_recurrence), ("cuda", torch.float32, aussm_b200.scan_unitary)):
        a = [inp[k].to(dev, dtype).clone().requires_grad_(True) for k in SCAN_KEYS]
        out = fn(*a)
        loss = sum((o * inp[k].to(dev, dtype)).sum() for o, k in zip(out, ("gy", "gh_re", "gh_im")))
        loss.backward()
        results.append(dict(zip(("y", "h_re", "h_im"), out)) | {"grad_" + k: t.grad for k, t in zip(SCAN_KEYS, a)})
    truth, got = results
    return {k: scaled_error(got[k].detach().cpu(), truth[k].detach()) for k in truth}


# A step costs at most two roundings (2^-24 each) of the rotated state and 1e-7 from the sine and cosine, 2.2e-7 of
# its magnitude; the adjoint the same.  The steps' errors are independent: a deviation of 2.2e-7 sqrt(l) at most after l
# steps, of which the largest of some thousand values takes 4.5; the activations and the sums over the states another
# 1e-6.  (Largest seen: 0.45e-6 sqrt(l), at one step; 0.2e-6 sqrt(l) from 1000 steps on.)
def scan_bound(l):
    return 1e-6 * (math.sqrt(l) + 1.0)


# The gradients of B, C and D are sums of b d l signed terms, whose rounding errors are relative to the terms: in a
# tensor of n values (one at the smallest) the terms of the largest sum may cancel to a tenth of their magnitude.
def check_scan(errors, l):
    bound = scan_bound(l)
    for k, e in errors.items():
        assert e < (10 * bound if k[5:] in ("B_r", "B_theta", "C_r", "C_theta", "D") else bound), (k, e, bound)


@pytest.mark.parametrize("n", [1, 3, 4, 7, 8, 10, 16, 17, 32, 40, 64, 128])
@pytest.mark.parametrize("l", [1, 3, 31, 33, 63, 65, 129])
def test_scan_rows_that_start_anywhere(n, l):
    """Lengths that are no multiple of 4: rows shift against the 16-byte grid, tiles end inside a group of 4 steps."""
    b, d = 2, 3
    errors = scan_errors(b, d, n, l, 1000 + 10 * n + l)
    assert aussm_b200.device_status() == 0
    check_scan(errors, l)


@pytest.mark.parametrize("n", [1, 4, 5, 8, 9, 16, 20, 32, 33, 64, 100, 128])
@pytest.mark.parametrize("l", [4, 28, 32, 36, 132])
def test_scan_whole_launches_of_aligned_rows(n, l):
    """Every tile shape in the form that whole launches take: warps with missing channels and states, short last tiles."""
    b, d = 2, 5
    errors = scan_errors(b, d, n, l, 1500 + 10 * n + l)
    assert aussm_b200.device_status() == 0
    check_scan(errors, l)


@pytest.mark.parametrize("shape", [(1, 3, 16, 1024), (1, 2, 5, 1029), (2, 5, 4, 1533), (1, 2, 33, 1280),
                                   (1, 1, 128, 1100), (1, 1, 1, 2047), (3, 7, 10, 1027)])
def test_scan_cut_into_unequal_segments(shape):
    """Few channels: as many segments as a wave holds, the last one what is left, at any length and alignment."""
    assert _lib.load().aussm_b200_scan_unitary_fwd_workspace_bytes(*shape) > 0, "this shape should be split"
    errors = scan_errors(*shape, 2000 + sum(shape))
    assert aussm_b200.device_status() == 0
    check_scan(errors, shape[-1])


@pytest.mark.parametrize("shape", [(1, 8, 16, 20001), (1, 4, 4, 20000), (2, 3, 40, 8192)])
def test_segments_are_as_accurate_as_the_whole_scan(shape):
    """What a split adds (rotation products of thousands of steps, chains over the segments, sums per segment) must stay
    below the rounding of the sequential scan, in the gradients of B above all, whose boundary terms cancel."""
    results = []
    try:
        for split in (1, 0):
            _lib.set_option("time_split", split)
            results.append(scan_errors(*shape, 9))
    finally:
        _lib.set_option("time_split", 1)
    for k, whole in results[1].items():
        assert results[0][k] < 1.5 * whole + 1e-6, (k, results[0][k], whole)


# The phases come from a product over d terms held to 2^-22 each, 2.4e-7 of a phase: a deviation of 3.3e-7 sqrt(l)
# together with the scan's own.  (Largest seen: 0.25e-6 sqrt(l).)
def operator_bound(l):
    return 1e-6 * (1.5 * math.sqrt(l) + 1.0)


def operator_errors(b, d, n, l, seed, gain=1.0):
    inp = model_like_inputs(seed, b, d, n, l)
    inp["gy"] = inp["gy"] * gain
    results = []
    for dev, real, cplx, fn in (("cpu", torch.float64, torch.complex128, O.interface_unitary),
                                ("cuda", torch.float32, torch.complex64, aussm_b200.ssm_adaptive_interface)):
        a = [inp[k].to(dev, cplx if inp[k].is_complex() else real).clone().requires_grad_(True) for k in NAMES]
        y = fn(*a)
        (y * inp["gy"].to(dev, real)).sum().backward()
        results.append({"y": y.detach()} | {"grad_" + k: t.grad for k, t in zip(NAMES, a)})
    truth, got = results
    view = lambda t: torch.view_as_real(t.cpu()) if t.is_complex() else t.cpu()
    return {k: scaled_error(view(got[k]), view(truth[k])) for k in truth}


# One output tile and a long contraction (many runs), runs that do not divide the K blocks, tiles that do not divide
# the output, d that is no multiple of 4 (scalar stores of the partial outputs), no split at all.
@pytest.mark.parametrize("shape", [(8, 16, 4, 256), (3, 37, 9, 200), (2, 130, 10, 500), (1, 65, 32, 96), (1, 8, 1, 16)])
def test_operator_adjoints_summed_in_runs(shape):
    errors = operator_errors(*shape, 3000 + sum(shape))
    assert aussm_b200.device_status() == 0
    bound = operator_bound(shape[-1])
    assert max(errors.values()) < bound, (errors, bound)


# The phase gradients are split into FP16 parts scaled by their maximum: any magnitude of the incoming gradient.
@pytest.mark.parametrize("gain", [1e-25, 1e-6, 1.0, 1e18])
@pytest.mark.parametrize("shape", [(1, 9, 5, 1500), (2, 20, 16, 130)])
def test_operator_gradients_of_any_magnitude(shape, gain):
    errors = operator_errors(*shape, 3200 + sum(shape), gain)
    assert aussm_b200.device_status() == 0
    assert max(errors.values()) < operator_bound(shape[-1]), errors


# Channels far apart in magnitude: every row of dx has to be right on its own scale.  The FP16 parts resolve 2^-50 of the
# largest |dtheta|, so a channel 2^-s below it (its rows' norm up to 8 times below its maximum) has its values to 2^(s-47);
# the scan itself is held to four times the 4e-7 sqrt(l) measured for the operator.
@pytest.mark.parametrize("l", [300, 4096])
@pytest.mark.parametrize("how", ["gradient", "large step"])
def test_operator_rows_of_small_channels(l, how):
    b, d, n = 1, 6, 4
    inp = model_like_inputs(3250 + l, b, d, n, l)
    below = torch.zeros(d)
    if how == "gradient":
        below = torch.tensor([0.0, 12.0, 20.0, 26.0, 30.0, 34.0])
        inp["gy"] = inp["gy"] * (0.5 ** below)[:, None]
    else:                                            # one step of one channel drives its state and dtheta far up
        inp["dt"][0, 0, l // 2] *= 1e7
        below[1:] = 24.0
    dx = []
    for dev, real, cplx, fn in (("cpu", torch.float64, torch.complex128, O.interface_unitary),
                                ("cuda", torch.float32, torch.complex64, aussm_b200.ssm_adaptive_interface)):
        a = {k: inp[k].to(dev, cplx if inp[k].is_complex() else real).requires_grad_(k == "x") for k in NAMES}
        dx.append(torch.autograd.grad(fn(*(a[k] for k in NAMES)), a["x"], inp["gy"].to(dev, real))[0].double().cpu())
    truth, got = dx
    assert aussm_b200.device_status() == 0
    error = (got - truth).flatten(1).norm(dim=1) / truth.flatten(1).norm(dim=1)
    bound = 1.6e-6 * math.sqrt(l) + 2.0 ** (below.double() - 47)
    assert (error < bound).all(), (error, bound)


def test_a_nan_spoils_its_own_channel_only():
    """A NaN in one channel's incoming gradient must not reach the other channels' rows of dx nor other batch entries."""
    b, d, n, l = 2, 6, 4, 200
    inp = model_like_inputs(3300, b, d, n, l)
    results = []
    for bad in (0.0, float("nan")):
        a = {k: inp[k].cuda().requires_grad_(True) for k in NAMES}
        gy = inp["gy"].cuda()
        gy[0, 2, 77] = bad
        results.append(torch.autograd.grad(aussm_b200.ssm_adaptive_interface(**a), (a["x"], a["u"]), gy))
    (dx, du), (dx_nan, du_nan) = results
    others = [i for i in range(d) if i != 2]
    assert torch.isnan(dx_nan[2]).any() and torch.isnan(du_nan[0]).any()
    assert scaled_error(dx_nan[others], dx[others]) < operator_bound(l)
    assert scaled_error(du_nan[1], du[1]) < operator_bound(l)


@pytest.mark.parametrize("bad", [float("inf"), float("-inf")])
@pytest.mark.parametrize("l", [200, 1100])
def test_an_infinity_does_not_reach_the_scale_of_the_others(bad, l):
    """In one channel's incoming gradient: the other channels' rows of dx, the other batch entries' du.  In one batch
    entry's u: the other entries' outputs and du."""
    b, d, n = 2, 6, 4
    inp = model_like_inputs(3350, b, d, n, l)
    results = []
    for which in (None, "gy", "u"):
        a = {k: inp[k].cuda() for k in NAMES}
        gy = inp["gy"].cuda()
        if which == "gy":
            gy[0, 2, 77] = bad
        elif which == "u":
            a["u"][0, 2, 77] = bad
        a = {k: t.requires_grad_(True) for k, t in a.items()}
        y = aussm_b200.ssm_adaptive_interface(**a)
        results.append((y.detach(), *torch.autograd.grad(y, (a["x"], a["u"]), gy)))
    (y, dx, du), (_, dx_gy, du_gy), (y_u, _, du_u) = results
    others = [i for i in range(d) if i != 2]
    bound = operator_bound(l)
    assert not torch.isfinite(dx_gy[2]).all() and not torch.isfinite(y_u[0]).all()
    assert scaled_error(dx_gy[others], dx[others]) < bound and scaled_error(du_gy[1], du[1]) < bound
    assert scaled_error(y_u[1], y[1]) < bound and scaled_error(du_u[1], du[1]) < bound


@pytest.mark.parametrize("steps", [576, 640, 2000])
def test_operator_windows_of_unequal_length_split_in_time(steps):
    """2000 steps in windows of 576 (the last one shorter than a segment), 640 and one: same result."""
    b, d, n, l = 1, 5, 6, 2000
    try:
        _lib.set_option("window_steps", steps)
        errors = operator_errors(b, d, n, l, 3100)
    finally:
        _lib.set_option("window_steps", 0)
    assert aussm_b200.device_status() == 0
    assert max(errors.values()) < operator_bound(l), errors


S6_KEYS = ["u", "delta", "A", "B", "C", "D", "z", "delta_bias"]


# A step of the contracting recurrence costs two roundings and the exponential's 2^-22, and earlier errors decay: the
# length does not enter.  dA sums terms of both signs and is the worst: 3.2e-6 seen, four times that allowed.
@pytest.mark.parametrize("shape", [(1, 5, 16, 512), (2, 33, 4, 516), (1, 16, 7, 1028), (3, 40, 12, 516), (1, 1, 1, 4096),
                                   (1, 9, 17, 520), (2, 3, 32, 1000), (40, 7, 24, 64)])
@pytest.mark.parametrize("full", [True, False])
def test_selective_scan_cut_into_segments(shape, full):
    b, d, n, l = shape
    g = torch.Generator().manual_seed(4000 + sum(shape))
    r = lambda *s: torch.randn(*s, generator=g)
    inp = dict(u=r(b, d, l), delta=r(b, d, l) * 0.5 - 1.0, A=-torch.exp(r(d, n)), B=r(b, n, l) / math.sqrt(n),
               C=r(b, n, l) / math.sqrt(n), D=r(d), z=r(b, d, l), delta_bias=r(d) * 0.5)
    gy = r(b, d, l)
    if not full:
        inp["z"] = inp["D"] = inp["delta_bias"] = None
        inp["delta"] = torch.nn.functional.softplus(inp["delta"])
    results = []
    for dev, dtype, fn in (("cpu", torch.float64, selective_scan_ref), ("cuda", torch.float32, selective_scan_fn)):
        a = [None if inp[k] is None else inp[k].to(dev, dtype).clone().requires_grad_(True) for k in S6_KEYS]
        y, last = fn(*a, delta_softplus=full, return_last_state=True)
        (y * gy.to(dev, dtype)).sum().backward()
        results.append({"y": y.detach(), "last": last.detach()} |
                       {k: t.grad for k, t in zip(S6_KEYS, a) if t is not None})
    assert aussm_b200.device_status() == 0
    truth, got = results
    for k in truth:
        assert scaled_error(got[k].cpu(), truth[k]) < 1.3e-5, k


# Channels that do not fill a warp, states that do not fill their lanes, whole and cut into segments (from 768 steps).
# Per step the multiplier (exponential, sine, cosine) and the products cost 4e-7 of the magnitude; errors decay within a
# few steps.  4.6e-7 seen, four times that allowed.
DECAY_BOUND = 2e-6
DECAY_SHAPES = [(2, 3, 4, 40), (1, 5, 8, 36), (1, 3, 10, 52), (2, 1, 16, 16), (1, 3, 20, 44), (1, 3, 16, 768),
                (2, 5, 3, 900), (1, 1, 32, 1028), (1, 7, 9, 2048)]


def decay_inputs(shape, angle, seed):
    b, d, n, l = shape
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g)
    return dict(rho=-F.softplus(r(b, d, n, l)), theta=3 * r(b, d, n, l) if angle else None, u=r(b, d, l),
                dt=F.softplus(r(b, d, l)), z=r(b, d, l), B_re=r(b, n, l), B_im=r(b, n, l) if angle else None,
                C_re=r(b, n, l), C_im=r(b, n, l) if angle else None, D=r(d)), r(b, d, l)


@pytest.mark.parametrize("shape", DECAY_SHAPES)
@pytest.mark.parametrize("angle", [True, False])
def test_decaying_scan_partial_warps_and_segments(shape, angle):
    b, d, n, l = shape
    inp, gy = decay_inputs(shape, angle, 7000 + sum(shape))
    results = []
    for dev, dtype in (("cpu", torch.float64), ("cuda", torch.float32)):
        a = {k: None if t is None else t.to(dev, dtype).requires_grad_(True) for k, t in inp.items()}
        if dev == "cpu":
            pair = (lambda x, y: torch.complex(x, y)) if angle else (lambda x, y: x)
            y = scan_complex_ref(a["rho"], a["theta"], a["u"], a["dt"], a["z"], pair(a["B_re"], a["B_im"]),
                                 pair(a["C_re"], a["C_im"]), a["D"])
        else:
            y = variants.scan_complex(**a)
        (y * gy.to(dev, dtype)).sum().backward()
        results.append({"y": y.detach()} | {k: t.grad for k, t in a.items() if t is not None})
    assert aussm_b200.device_status() == 0
    for k, t in results[0].items():
        assert scaled_error(results[1][k].cpu(), t) < DECAY_BOUND, k


@pytest.mark.parametrize("shape", [(1, 3, 16, 768), (1, 2, 5, 1040)])
@pytest.mark.parametrize("angle", [True, False])
def test_decaying_scan_state_record_does_not_depend_on_the_segments(shape, angle):
    """The record of the states and gradients that arrive through it, cut into segments and whole."""
    inp, gy = decay_inputs(shape, angle, 7100 + sum(shape))
    results = []
    try:
        for split in (1, 0):
            _lib.set_option("time_split", split)
            a = {k: None if t is None else t.cuda().requires_grad_(True) for k, t in inp.items()}
            y, states = variants.scan_complex(**a, return_states=True)
            weight = torch.linspace(-1, 1, states.numel(), device="cuda").view_as(states)
            ((y * gy.cuda()).sum() + (states * weight).sum()).backward()
            results.append({"y": y.detach(), "states": states.detach()} | {k: t.grad for k, t in a.items() if t is not None})
    finally:
        _lib.set_option("time_split", 1)
    for k, t in results[1].items():
        assert scaled_error(results[0][k], t) < DECAY_BOUND, k


# A row's mean square sums d products (a lane d / 32 of them in a chain, then five additions), the rest is a handful
# of roundings; the weight's gradient sums over the rows.
@pytest.mark.parametrize("rows,d", [(1, 4), (3, 128), (9, 132), (7, 252), (1300, 516), (5000, 1024), (2, 1028), (4, 30)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rms_norm_and_its_residual(rows, d, shift):
    g = torch.Generator().manual_seed(5000 + rows + d)
    r = lambda *s: torch.randn(*s, generator=g)
    x, w, gy, gr = r(rows, d) * 3, r(d), r(rows, d), r(rows, d)
    results = []
    for dev, dtype in (("cpu", torch.float64), ("cuda", torch.float32)):
        flat = torch.zeros(rows * d + shift, device=dev, dtype=dtype)      # shift: rows that are not 16-byte aligned
        flat[shift:] = x.to(dev, dtype).reshape(-1)
        xs = flat[shift:].view(rows, d).requires_grad_(True)
        ws = w.to(dev, dtype).requires_grad_(True)
        if dev == "cpu":
            y, res = xs * torch.rsqrt(xs.pow(2).mean(-1, keepdim=True) + 1e-5) * ws, xs
        else:
            y, res = stages.rms_norm_residual(xs, ws)
        loss = (y * gy.to(dev, dtype)).sum() + (res * gr.to(dev, dtype)).sum()
        dx, dw = torch.autograd.grad(loss, (xs, ws), create_graph=True)
        (ddx,) = torch.autograd.grad((dx * gy.to(dev, dtype)).sum(), xs)
        plain = torch.autograd.grad((stages.rms_norm(xs, ws) * gy.to(dev, dtype)).sum(), (xs, ws))
        results.append([y, dx, dw, ddx, *plain])
    for t, o in zip(*results):
        assert scaled_error(o.detach().cpu(), t.detach()) < 1.2e-7 * (16 + d / 16 + (rows if t.dim() == 1 else 0))


# exp, log1p and the quotient to a few ulp each
@pytest.mark.parametrize("n", [1, 5, 64, 128])
def test_polar_parameters(n):
    g = torch.Generator().manual_seed(6000 + n)
    B, C = (torch.complex(torch.randn(n, generator=g) * s, torch.randn(n, generator=g)) for s in (1.0, 30.0))
    weights = [torch.randn(n, generator=g) for _ in range(4)]
    results = []
    for dev, cplx, real in (("cpu", torch.complex128, torch.float64), ("cuda", torch.complex64, torch.float32)):
        b, c = B.to(dev, cplx).requires_grad_(True), C.conj().to(dev, cplx).requires_grad_(True)
        if dev == "cpu":
            out = (F.softplus(b.real), b.imag, F.softplus(c.conj().real), c.conj().imag)
        else:
            out = ops._polar_params(b, c.conj())
        loss = sum((o * w.to(dev, real)).sum() for o, w in zip(out, weights))
        results.append([*out, *(torch.stack([t.real, t.imag]) for t in torch.autograd.grad(loss, (b, c)))])
    for t, o in zip(*results):
        assert scaled_error(o.detach().cpu(), t.detach()) < 1e-6


# Small products of the blocks, batched (one sequence: its weight gradient in pieces).  Sums of k or m products, the
# weight's of b l products, half an ulp each and independent.
@pytest.mark.parametrize("b,l,m,k", [(1, 4096, 16, 24), (1, 1000, 8, 40), (3, 96, 40, 20), (64, 33, 12, 12), (2, 8, 300, 200)])
def test_small_projections(b, l, m, k):
    g = torch.Generator().manual_seed(8000 + b + l)
    r = lambda *s: torch.randn(*s, generator=g)
    cases = [(stages.project_tokens, r(b, l, k), "mk,blk->bml"), (stages.project_channels, r(b, k, l), "mk,bkl->bml"),
             (stages.project_back, r(b, k, l), "mk,bkl->blm")]
    for fn, x, formula in cases:
        W, results = r(m, k), []
        for dev, dtype in (("cpu", torch.float64), ("cuda", torch.float32)):
            a = [t.to(dev, dtype).requires_grad_(True) for t in (W, x)]
            y = torch.einsum(formula, *a) if dev == "cpu" else fn(*a)
            grads = torch.autograd.grad(y.square().sum(), a, create_graph=True)
            (second,) = torch.autograd.grad(grads[0].sum(), a[1])
            results.append([y, *grads, second])
        for t, o in zip(*results):
            assert o.shape == t.shape and scaled_error(o.detach().cpu(), t.detach()) < 1.2e-7 * (4 + math.sqrt(m + k + b * l)), fn.__name__


# Rows in chunks, several rows in a block, lengths that end inside a quad.  A gradient of the weight or the bias sums
# b l terms.
@pytest.mark.parametrize("b,d,l,taps", [(1, 3, 9001, 4), (1, 2, 4096, 2), (3, 5, 130, 3), (2, 9, 515, 4), (1, 1, 3, 4), (40, 70, 20, 1)])
def test_conv_and_step_size_row_plans(b, d, l, taps):
    g = torch.Generator().manual_seed(9000 + l)
    r = lambda *s: torch.randn(*s, generator=g)
    x, w, bias, gy = r(b, d, l), r(d, 1, taps), r(d), r(b, d, l)
    results = []
    for dev, dtype in (("cpu", torch.float64), ("cuda", torch.float32)):
        a = [t.to(dev, dtype).requires_grad_(True) for t in (x, w, bias)]
        if dev == "cpu":
            u = F.conv1d(a[0], a[1], a[2], padding=taps - 1, groups=d)[..., :l]
            dt = F.softplus(a[0] + 2.0 * a[2][:, None])
        else:
            u, dt = stages.causal_conv_bias(*a), stages.softplus_bias(a[0], a[2], 2.0)
        gu = torch.autograd.grad((u * gy.to(dev, dtype)).sum(), a)
        gd = torch.autograd.grad((dt * gy.to(dev, dtype)).sum(), (a[0], a[2]))
        results.append([u, dt, *gu, *gd])
    for t, o in zip(*results):
        assert scaled_error(o.detach().cpu(), t.detach()) < 1e-6 + (1.2e-7 * b * l if t.numel() <= d * taps else 0.0)
