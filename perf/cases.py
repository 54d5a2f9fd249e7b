"""The workloads this package's speed is measured on: what a training or inference program calls, with the sizes of
the repository's own benchmark configurations, of its tests, and of generic ragged batches between them.

Kinds of work (``case["kind"]``), each through the public entry point that a user's program calls:

``operator``    ``aussm_b200.ops.ssm_adaptive_interface``: the AUSSM block's operator with its phase projection
``scan``        ``aussm_b200.ops.scan_unitary``: the unitary scan on a phase tensor the caller made
``mamba``       ``aussm_b200.s6.selective_scan_fn``: the Mamba block's scan
``decay``       ``aussm_b200.variants.scan_complex``: the scan with decaying eigenvalues, complex (``angle``) or
                positive real
``timeseries``  ``aussm_b200.models.SSMTS``: training pass of the time-series model
``classifier``  ``aussm_b200.models.SSMSequenceClassifier``: training pass of the token classifier

``train`` asks for the forward and the backward pass, otherwise the call runs without gradients.  All data is
float32 (complex64 for B and C): the only type the operators take.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from aussm_b200 import models, ops, s6, variants


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The operator at the size of its unit fixture: the smallest call, where launches and host work are all.
        dict(name="operator_small", kind="operator", b=8, d=16, n=4, l=256, train=True),
        # A training call of a small model on ragged data: no size a multiple of anything.
        dict(name="operator_ragged", kind="operator", b=5, d=181, n=12, l=1003, train=True),
        # One micro-batch of the benchmark's width (d_inner 1024): where training spends its time.
        dict(name="operator_wide", kind="operator", b=4, d=1024, n=16, l=4096, train=True),
        # Evaluating two long sequences through one block of the classifier's width: forward only.
        dict(name="operator_forward", kind="operator", b=2, d=512, n=16, l=8192, train=False),
        # The benchmark's scan: batch 16, d_inner 1024, 16384 steps.
        dict(name="scan_large", kind="scan", b=16, d=1024, n=16, l=16384, train=True),
        # The shortest sequence of the benchmark's length sweep.
        dict(name="scan_short", kind="scan", b=16, d=1024, n=16, l=256, train=True),
        # Ragged lengths: rows that do not start on 16-byte boundaries, states that do not fill their lanes.
        dict(name="scan_ragged", kind="scan", b=6, d=300, n=10, l=1021, train=True),
        # One very long sequence: few channels, all parallelism has to come from the time axis.
        dict(name="scan_long", kind="scan", b=1, d=512, n=16, l=65536, train=True),
        # The Mamba scan of the three-variant comparison.
        dict(name="mamba_wide", kind="mamba", b=8, d=2048, n=16, l=4096, train=True),
        # The complex scan of the same comparison.
        dict(name="decay_wide", kind="decay", b=8, d=2048, n=16, l=4096, train=True, angle=True),
        # A training pass of the hybrid time-series model (720 steps of 21 variables, batch 64): many small kernels.
        dict(name="timeseries_train", kind="timeseries", b=64, d=128, n=16, l=720, layers="a|m|a|m", train=True),
        # A training pass of the token classifier on one sequence of 65536 tokens.
        dict(name="classifier_train", kind="classifier", b=1, d=512, n=16, l=65536, layers="a|a|a|a", train=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length: mostly what data sets have (multiples of 16), often enough any number."""
    l = _log_int(rng, lo, hi)
    return max(16, l // 16 * 16) if rng.random() < 0.5 else l


def draw(rng):
    """One more case of the ranges above: same kinds, sizes spread over their logarithm, no costlier than the largest."""
    kind = rng.choice(["operator", "operator", "operator", "scan", "scan", "scan", "mamba", "mamba", "decay", "decay",
                       "timeseries", "classifier"])
    n = rng.choice([4, 8, 16, 16, 16, 32, rng.randint(2, 64)])
    b = _log_int(rng, 1, 16)
    train = rng.random() < 0.8
    if kind == "operator":
        d = rng.choice([16, 64, 128, 256, 512, 1024, rng.randint(16, 1024)])
        l = _length(rng, 14, 16384)
        while b * l * d * d * n > 1 << 38:                  # twice the products of operator_wide
            b, l = max(1, b // 2), max(14, l * 2 // 3)
        return dict(kind=kind, b=b, d=d, n=n, l=l, train=train)
    if kind == "scan":
        d = rng.choice([64, 256, 512, 1024, rng.randint(16, 1024)])
        l = _length(rng, 16, 65536)
        while b * d * n * l > 1 << 31:                      # half of scan_large
            b, l = max(1, b // 2), max(16, l * 2 // 3)
        return dict(kind=kind, b=b, d=d, n=n, l=l, train=train)
    if kind == "mamba":
        d = rng.choice([256, 512, 1024, 2048, rng.randint(32, 2048)])
        n = min(n, 32)
        l = _length(rng, 64, 16384)
        while b * d * l > 1 << 26:                          # mamba_wide
            b, l = max(1, b // 2), max(64, l * 2 // 3)
        return dict(kind=kind, b=b, d=d, n=n, l=l, train=train)
    if kind == "decay":
        d = rng.choice([256, 512, 1024, 2048, rng.randint(32, 2048)])
        n = min(n, 32)
        l = _length(rng, 64, 16384)
        while b * d * n * l > 1 << 30:                      # decay_wide
            b, l = max(1, b // 2), max(64, l * 2 // 3)
        return dict(kind=kind, b=b, d=d, n=n, l=l, train=train, angle=rng.random() < 0.6)
    if kind == "timeseries":
        return dict(kind=kind, b=_log_int(rng, 8, 64), d=rng.choice([64, 128, 128, 256]), n=16,
                    l=rng.choice([96, 192, 336, 720, rng.randint(96, 720)]), layers=rng.choice(["a|m|a|m", "a|m", "m|a", "a|a"]),
                    train=True)
    return dict(kind=kind, b=rng.choice([1, 1, 2]), d=rng.choice([256, 512]), n=16, l=_length(rng, 1024, 32768),
                layers=rng.choice(["a|a|a|a", "a|a", "a|m|a"]), train=True)


# ---------------------------------------------------------------------------
# inputs, a pass
# ---------------------------------------------------------------------------
INPUT_DIM = 21          # variables of the time series
VOCAB, CLASSES = 256, 10


def prepare(case, seed):
    kind, b, d, n, l, train = (case[k] for k in ("kind", "b", "d", "n", "l", "train"))
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)

    def randn(*s):
        return torch.randn(*s, generator=g, device=dev)

    def angles(*s):
        return (torch.rand(*s, generator=g, device=dev).mul_(2.0).sub_(1.0)).mul_(math.pi)

    def pair(*s):
        return torch.complex(randn(*s) / math.sqrt(n), randn(*s) / math.sqrt(n))

    state = {"case": dict(case)}
    if kind in ("timeseries", "classifier"):
        with torch.random.fork_rng(devices=[dev]):
            torch.manual_seed(seed)
            if kind == "timeseries":
                model = models.SSMTS(d_model=d, input_dim=INPUT_DIM, output_dim=INPUT_DIM, layers=case["layers"], d_state=n)
            else:
                model = models.SSMSequenceClassifier(d_model=d, vocab_size=VOCAB, output_dim=CLASSES,
                                                     layers=case["layers"], d_state=n)
        state["model"] = model.to(dev)
        if kind == "timeseries":
            t = torch.arange(l, dtype=torch.float32, device=dev)[None, :, None]
            period = torch.randint(4, 169, (b, 1, INPUT_DIM), generator=g, device=dev).float()
            state["x"] = randn(b, l, INPUT_DIM) + torch.sin(2 * math.pi * t / period)
            state["target"] = randn(b, l, INPUT_DIM)
        else:
            state["x"] = torch.randint(0, VOCAB, (b, l), generator=g, device=dev)
            state["target"] = torch.randint(0, CLASSES, (b,), generator=g, device=dev)
        return state

    if kind == "operator":
        inputs = dict(u=randn(b, d, l), dt=F.softplus(randn(b, d, l)), x=randn(d, n, d) / math.sqrt(d), x_bias=angles(d, n),
                      B=pair(n), C=pair(n), D=randn(d), z=randn(b, d, l))
    elif kind == "scan":
        inputs = dict(theta=angles(b, d, n, l), u=randn(b, d, l), dt=F.softplus(randn(b, d, l)), z=randn(b, d, l),
                      B_r=F.softplus(randn(n) / math.sqrt(n)), B_theta=randn(n) / math.sqrt(n),
                      C_r=F.softplus(randn(n) / math.sqrt(n)), C_theta=randn(n) / math.sqrt(n), D=randn(d))
    elif kind == "mamba":
        inputs = dict(u=randn(b, d, l), delta=randn(b, d, l), A=-torch.exp(randn(d, n)), B=randn(b, n, l), C=randn(b, n, l),
                      D=randn(d), z=randn(b, d, l), delta_bias=0.5 * randn(d))
    elif kind == "decay":
        sc = 1.0 / math.sqrt(n)
        angle = case["angle"]
        inputs = dict(rho=F.softplus(randn(b, d, n, l)).neg_(), theta=angles(b, d, n, l) if angle else None,
                      u=randn(b, d, l), dt=F.softplus(randn(b, d, l)), z=randn(b, d, l),
                      B_re=randn(b, n, l) * sc, B_im=randn(b, n, l) * sc if angle else None,
                      C_re=randn(b, n, l) * sc, C_im=randn(b, n, l) * sc if angle else None, D=randn(d))
    else:
        raise ValueError(kind)
    state["inputs"] = inputs
    if train:
        for t in inputs.values():
            if t is not None:
                t.requires_grad_(True)
        state["grad_y"] = randn(b, d, l)
    return state


def _forward(kind, inputs):
    if kind == "operator":
        return ops.ssm_adaptive_interface(**inputs)
    if kind == "scan":
        return ops.scan_unitary(**inputs)
    if kind == "mamba":
        return s6.selective_scan_fn(**inputs, delta_softplus=True)
    return variants.scan_complex(**inputs)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("timeseries", "classifier"):
        model, x, target = state["model"], state["x"], state["target"]
        model.zero_grad(set_to_none=True)
        out = model(x)
        loss = F.mse_loss(out, target) if kind == "timeseries" else F.cross_entropy(out, target)
        loss.backward()
        return {"out": out.detach(), "loss": loss.detach(), "grads": {k: p.grad for k, p in model.named_parameters()}}
    inputs = state["inputs"]
    if not case["train"]:
        with torch.no_grad():
            out = _forward(kind, inputs)
        return out if kind != "scan" else dict(zip(("y", "h_re", "h_im"), out))
    out = _forward(kind, inputs)
    y = out[0] if kind == "scan" else out
    wanted = {k: t for k, t in inputs.items() if t is not None}
    grads = torch.autograd.grad(y, list(wanted.values()), state["grad_y"])
    result = {"y": y.detach(), "grads": dict(zip(wanted, grads))}
    if kind == "scan":
        result["h_re"], result["h_im"] = out[1].detach(), out[2].detach()
    return result


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _block_work(kind, b, d, n, l):
    """Multiply-adds of the matrix products of one block's forward pass, and its parameters."""
    if kind == "a":
        weights = 2 * d * d + d * n + n * d + d * n * d + d * d           # in, x, dt, phase projection, out
        return b * l * weights, weights
    di, r = 2 * d, math.ceil(d / 16)
    weights = 2 * di * d + di * (r + 2 * n) + r * di + di * d
    return b * l * weights, weights


def work(case):
    kind, b, d, n, l, train = (case[k] for k in ("kind", "b", "d", "n", "l", "train"))
    rows, states = b * d * l, b * d * n * l
    if kind == "operator":
        # u, dt, z and the weights in, y out; backward: y's gradient in, the four gradients out.  The phase
        # projection forward, its two adjoint products backward; about 25 operations per state and step each way.
        w = d * n * d
        if train:
            return {"bytes": 4.0 * (8 * rows + 2 * w), "flops": 6.0 * states * d + 75.0 * states}
        return {"bytes": 4.0 * (4 * rows + w), "flops": 2.0 * states * d + 25.0 * states}
    if kind == "scan":
        # the backward pass reads the inputs again: no card holds them on chip
        if train:
            return {"bytes": 4.0 * (3 * states + 11 * rows), "flops": 75.0 * states}
        return {"bytes": 4.0 * (states + 4 * rows), "flops": 25.0 * states}
    if kind == "mamba":
        bc = b * n * l
        if train:
            return {"bytes": 4.0 * (11 * rows + 6 * bc), "flops": 30.0 * states}
        return {"bytes": 4.0 * (4 * rows + 2 * bc), "flops": 8.0 * states}
    if kind == "decay":
        streams = 2 if case["angle"] else 1
        bc = 2 * streams * b * n * l
        if train:
            return {"bytes": 4.0 * (3 * streams * states + 11 * rows + 3 * bc), "flops": (90.0 if streams == 2 else 40.0) * states}
        return {"bytes": 4.0 * (streams * states + 4 * rows + bc), "flops": (35.0 if streams == 2 else 10.0) * states}
    macs = params = elem = 0
    for k in case["layers"].split("|"):
        m, w = _block_work(k, b, d, n, l)
        macs, params = macs + m, params + w
        elem += states * (75 if k == "a" else 60)
    # each layer's input is kept for the backward pass: written once, read once
    layers = len(case["layers"].split("|"))
    return {"bytes": 4.0 * (2 * layers * rows + 2 * params), "flops": 6.0 * macs + elem}


def tolerance(case):
    """About four times the largest relative error (2-norm, over all outputs) of the float32 path against float64.
    A unitary recurrence never forgets a rounding error, so there it grows with the root of the length (measured:
    4e-7 sqrt(l) with the phases projected, 1.5e-7 sqrt(l) with the phases given); decaying recurrences forget
    (2e-6 for sums over batch and time in the Mamba scan, 5e-7 otherwise).  The models stack layers of the former:
    6e-6 for 720 steps; for the classifier 2e-5 at 2048 and 1e-4 at 8192 tokens, and two orders of the same sums
    differ by 9e-4 at 65536."""
    kind, l = case["kind"], case["l"]
    if kind == "operator":
        return {"rel": max(1e-5, 1.6e-6 * math.sqrt(l))}
    if kind == "scan":
        return {"rel": max(4e-6, 6e-7 * math.sqrt(l))}
    if kind == "mamba":
        return {"rel": 1e-5}
    if kind == "decay":
        return {"rel": 4e-6}
    if kind == "timeseries":
        return {"rel": 4e-5}
    return {"rel": max(1e-4, 5.5e-8 * l)}


# ---------------------------------------------------------------------------
# the same passes in 64 bits, in plain torch
# ---------------------------------------------------------------------------
class _LinearRecurrence(torch.autograd.Function):
    """h_t = a_t h_{t-1} + x_t over the first axis, from zero."""

    @staticmethod
    def forward(ctx, a, x):
        h = torch.empty_like(x)
        h[0] = x[0]
        for p, q, ai, xi in zip(h[:-1].unbind(0), h[1:].unbind(0), a[1:].unbind(0), x[1:].unbind(0)):
            torch.addcmul(xi, ai, p, out=q)
        ctx.save_for_backward(a, h)
        return h

    @staticmethod
    def backward(ctx, g):
        a, h = ctx.saved_tensors
        e, ac = g.clone(), a.conj().resolve_conj()
        rows, mult = e.unbind(0), ac.unbind(0)
        for t in range(len(rows) - 2, -1, -1):
            rows[t].addcmul_(mult[t + 1], rows[t + 1])
        ga = torch.zeros_like(a)
        torch.mul(e[1:], h[:-1].conj(), out=ga[1:])
        return ga, e


def _unitary(theta, drive, coef):
    """sum_j Re(coef_j h_j) and the last state of h_t = exp(i theta_t) h_{t-1} + drive_t, theta (c, n, l)."""
    turn = torch.polar(torch.ones_like(theta), torch.cumsum(theta, -1))
    h = turn * torch.cumsum(turn.conj() * drive, -1)
    return (coef[:, None] * h).real.sum(-2), h[..., -1]


def _polar(r, angle):
    return torch.polar(r, torch.zeros_like(r)) * torch.polar(torch.ones_like(angle), angle)


def _exact_scan(theta_of, u, dt, z, Bc, Cc, D, part):
    """The unitary operator, `part` channels of one batch entry at a time; theta_of(b, i0, i1) is their phases."""
    ys, hs = [], []
    for b in range(u.shape[0]):
        for i in range(0, u.shape[1], part):
            def piece(ub, dtb, zb, Db, *own, b=b, i=i):
                v = F.silu(ub)
                y, h = _unitary(theta_of(b, i, *own), Bc[:, None] * (dtb * v)[:, None], Cc)
                return F.silu(zb) * (Db[:, None] * v + y), h
            own = theta_of.own(b, i, i + part)
            cut = (u[b, i:i + part], dt[b, i:i + part], z[b, i:i + part], D[i:i + part]) + own
            y, h = checkpoint(piece, *cut, use_reentrant=False)
            ys.append(y)
            hs.append(h)
    shape = u.shape[:2]
    return torch.cat(ys).view(*shape, -1), torch.cat(hs).view(*shape, -1)


class _Projected:
    def __init__(self, x, bias, u):
        self.x, self.bias, self.u = x, bias, u

    def own(self, b, i0, i1):
        return self.x[i0:i1], self.bias[i0:i1], self.u[b]

    def __call__(self, b, i, x, bias, u):
        return torch.matmul(x, u) + bias[..., None]


class _Given:
    def __init__(self, theta):
        self.theta = theta

    def own(self, b, i0, i1):
        return (self.theta[b, i0:i1],)

    def __call__(self, b, i, theta):
        return theta


def _part(n, l):
    return max(1, (1 << 26) // (n * l))


def _exact_operator(u, dt, x, x_bias, B, C, D, z):
    Bc, Cc = _polar(F.softplus(B.real), B.imag), _polar(F.softplus(C.real), C.imag)
    return _exact_scan(_Projected(x, x_bias, u), u, dt, z, Bc, Cc, D, _part(x.shape[1], u.shape[2]))[0]


def _exact_decaying(u, a_of, x_of, C, part):
    """sum_j Re(C_j h_j) of h_t = a_t h_{t-1} + x_t; a_of and x_of give (channels, n, l) from a channel's own rows."""
    rows = []
    for b in range(u.shape[0]):
        for i in range(0, u.shape[1], part):
            def piece(b=b, i=i):
                a, x = a_of(b, slice(i, i + part)), x_of(b, slice(i, i + part))
                h = _LinearRecurrence.apply(a.movedim(-1, 0).contiguous(), x.movedim(-1, 0).contiguous())
                y = C[b].movedim(-1, 0)[:, None] * h
                return (y.real if y.is_complex() else y).sum(-1).t()
            rows.append(checkpoint(piece, use_reentrant=False))
    return torch.cat(rows).view(u.shape)


def _exact_mamba(u, delta, A, B, C, D, z, delta_bias):
    dl = F.softplus(delta + delta_bias[:, None])
    y = _exact_decaying(u, lambda b, i: torch.exp(dl[b, i, None] * A[i, :, None]),
                        lambda b, i: (dl[b, i] * u[b, i])[:, None] * B[b], C, 8 * _part(A.shape[1], u.shape[2]))
    return F.silu(z) * (y + D[:, None] * u)


def _exact_decay(rho, theta, u, dt, z, B_re, B_im, C_re, C_im, D):
    B, C = (B_re, C_re) if theta is None else (torch.complex(B_re, B_im), torch.complex(C_re, C_im))
    s = dt * F.silu(u)

    def multiplier(b, i):
        r = torch.exp(rho[b, i])
        return r if theta is None else torch.polar(torch.ones_like(r), theta[b, i]) * r
    y = _exact_decaying(u, multiplier, lambda b, i: s[b, i, None] * B[b], C, 4 * _part(rho.shape[2], u.shape[2]))
    return F.silu(z) * (D[:, None] * F.silu(u) + y)


def _exact_block(kind, p, x):
    """One mixer; p: its parameters by name; x (b, l, d)."""
    d = x.shape[-1]
    inner = p["conv1d.weight"].shape[0]
    xs, z = (x @ p["in_proj.weight"].t()).transpose(1, 2).split([inner, inner], dim=1)
    l = x.shape[1]
    xs = F.conv1d(xs, p["conv1d.weight"], p["conv1d.bias"], padding=p["conv1d.weight"].shape[-1] - 1,
                  groups=inner)[..., :l]
    low = p["x_proj.weight"] @ xs
    rank = p["dt_proj.weight"].shape[1]
    pre = p["dt_proj.weight"] @ low[:, :rank] + p["dt_proj.bias"][:, None]
    if kind == "a":
        n = p["B"].shape[0]
        y = _exact_operator(xs, F.softplus(pre + p["dt_proj.bias"][:, None]),
                            p["xA_proj.weight"].view(n, d, d).transpose(0, 1) / math.sqrt(d),
                            p["xA_proj.bias"].view(n, d).t(), p["B"], p["C"], p["D"], z)
    else:
        n = p["A_log"].shape[1]
        y = _exact_mamba(F.silu(xs), pre, -torch.exp(p["A_log"]), low[:, rank:rank + n], low[:, rank + n:], p["D"], z,
                         p["dt_proj.bias"])
    return y.transpose(1, 2) @ p["out_proj.weight"].t()


def _exact_model(case, state):
    def norm(x, w):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * w

    double = {torch.float32: torch.float64, torch.complex64: torch.complex128}
    p = {k: v.detach().to(double[v.dtype]).requires_grad_(True) for k, v in state["model"].named_parameters()}
    if case["kind"] == "timeseries":
        x = state["x"].double() @ p["embedding.weight"].t() + p["embedding.bias"]
    else:
        x = p["embedding.weight"][state["x"]]
    for k, kind in enumerate(case["layers"].split("|")):
        pre = "layers.%d." % k
        mixer = {name[len(pre) + 6:]: t for name, t in p.items() if name.startswith(pre + "mixer.")}
        x = x + _exact_block(kind, mixer, norm(x, p[pre + "norm.weight"]))
    if case["kind"] == "classifier":
        x = x.mean(1)
    out = norm(x, p["norm_f.weight"]) @ p["output.weight"].t()
    target = state["target"]
    loss = F.mse_loss(out, target.double()) if case["kind"] == "timeseries" else F.cross_entropy(out, target)
    return {"out": out.detach(), "loss": loss.detach(), "grads": dict(zip(p, torch.autograd.grad(loss, list(p.values()))))}


def exact(case, seed):
    """What `run` returns, in 64 bits; None for the largest cases, whose 64-bit gradients alone fill much of a card,
    and for Mamba layers in a very long model (a step by step loop)."""
    kind, states = case["kind"], case["b"] * case["d"] * case["n"] * case["l"]
    if states > 1 << 30 or (kind == "classifier" and "m" in case["layers"] and case["l"] > 8192):
        return None
    state = prepare(case, seed)
    if kind in ("timeseries", "classifier"):
        return _exact_model(case, state)
    double = {torch.float32: torch.float64, torch.complex64: torch.complex128}
    inputs = {k: None if t is None else t.detach().to(double[t.dtype]).requires_grad_(case["train"])
              for k, t in state["inputs"].items()}
    with torch.set_grad_enabled(case["train"]):
        h = None
        if kind == "operator":
            y = _exact_operator(**inputs)
        elif kind == "scan":
            i = inputs
            y, h = _exact_scan(_Given(i["theta"]), i["u"], i["dt"], i["z"], _polar(i["B_r"], i["B_theta"]),
                               _polar(i["C_r"], i["C_theta"]), i["D"], _part(case["n"], case["l"]))
        else:
            y = (_exact_mamba if kind == "mamba" else _exact_decay)(**inputs)
    result = {"y": y.detach()}
    if h is not None:
        result["h_re"], result["h_im"] = h.detach().real, h.detach().imag
    if not case["train"]:
        return result if h is not None else result["y"]
    wanted = {k: t for k, t in inputs.items() if t is not None}
    grads = torch.autograd.grad(y, list(wanted.values()), state["grad_y"].double())
    result["grads"] = dict(zip(wanted, grads))
    return result
