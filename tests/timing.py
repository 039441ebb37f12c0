"""Comparing the times of two calls on the GPU: in turn, each waited for, the
shortest of many, measured again before a difference counts."""
import time


def _best(call, runs):
    import torch
    best = float("inf")
    for _ in range(runs):
        t = time.perf_counter()
        call()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


def ratio(call, other, bound, runs=30, tries=4):
    """Seconds of `call` over those of `other`: the first ratio below `bound`, or the
    smallest of `tries`."""
    import torch
    for f in (call, other):
        f()
        torch.cuda.synchronize()
    least = float("inf")
    for _ in range(tries):
        a, b = _best(call, runs), _best(other, runs)
        a, b = min(a, _best(call, runs)), min(b, _best(other, runs))
        least = min(least, a / b)
        if least < bound:
            break
    return least
