"""Kernel variants and dispatch rules at the sizes where they can go wrong, against the float64 oracle."""
import math

import pytest
import torch

import aussm_b200
from oracle import unitary as O
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
# its magnitude; the adjoint the same; sums over n states and l steps add an ulp each at worst.
def scan_bound(b, d, n, l):
    return 4.5e-7 * l + 1.2e-7 * (n + b * d)


# The gradients of B, C and D are sums of b d l signed terms, whose rounding errors are relative to the terms: in a
# tensor of n values (one at the smallest) the terms of the largest sum may cancel to a tenth of their magnitude.
def check_scan(errors, b, d, n, l):
    bound = scan_bound(b, d, n, l)
    for k, e in errors.items():
        assert e < (10 * bound if k[5:] in ("B_r", "B_theta", "C_r", "C_theta", "D") else bound), (k, e, bound)


@pytest.mark.parametrize("n", [1, 3, 4, 7, 8, 10, 16, 17, 32, 40, 64, 128])
@pytest.mark.parametrize("l", [1, 3, 31, 33, 63, 65, 129])
def test_scan_rows_that_start_anywhere(n, l):
    """Lengths that are no multiple of 4: rows shift against the 16-byte grid, tiles end inside a group of 4 steps."""
    b, d = 2, 3
    errors = scan_errors(b, d, n, l, 1000 + 10 * n + l)
    assert aussm_b200.device_status() == 0
    check_scan(errors, b, d, n, l)


# The phases come from a product over d terms held to 2^-22 each: another 2.4e-7 sqrt(d) per step at worst.
def operator_bound(b, d, n, l):
    return scan_bound(b, d, n, l) + 2.4e-7 * math.sqrt(d) * l


def operator_errors(b, d, n, l, seed):
    inp = model_like_inputs(seed, b, d, n, l)
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
    bound = operator_bound(*shape)
    assert max(errors.values()) < 10 * bound, (errors, bound)
