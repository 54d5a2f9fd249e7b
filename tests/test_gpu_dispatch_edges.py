"""Kernel variants and dispatch rules at the sizes where they can go wrong, against the float64 oracle."""
import pytest
import torch

import aussm_b200
from oracle import unitary as O
from tests.helpers import scaled_error, scan_core_inputs

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
