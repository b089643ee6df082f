"""Shared helpers of the GPU parity tests."""
import contextlib

import numpy as np


def rel_l2(a, b, J):
    """J-weighted relative L2 difference (vec_math_mod.f90:50-90 weighting)."""
    num = np.sqrt(np.sum(J * (a - b) ** 2))
    den = np.sqrt(np.sum(J * b ** 2))
    return float(num / den) if den > 0 else float(num)


def fmt7(x):
    return "%.6E" % x


@contextlib.contextmanager
def busy_default_stream():
    """Some 100 ms of work queued on the legacy default stream (another
    library's, say), so that nothing else put there runs before it."""
    import torch
    a = torch.ones(1 << 28, device="cuda")
    torch.cuda.synchronize()
    for _ in range(300):
        a.mul_(1.0)
    try:
        yield
    finally:
        torch.cuda.synchronize()
