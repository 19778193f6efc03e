"""Which implementation a product gets (CPU): what the two sides are that are timed, and how a near tie is settled.  The kernels are replaced by torch arithmetic."""
import sys

import pytest
import torch

import pico_engine.ops                                       # noqa: F401  (the package's attribute `linear` is the function)
import pico_engine.ops.kernels as kernels

L = sys.modules["pico_engine.ops.linear"]


@pytest.fixture
def timed(monkeypatch):
    """A stand-in for the device: every kernel adds its name to the call under way; times come from ``cost``."""
    seen, cost = [], {}
    monkeypatch.setattr(L.Choice, "table", {})
    monkeypatch.setattr(L.Choice, "timings", {})
    monkeypatch.setattr(L, "_FORCED", "auto")
    monkeypatch.setattr(L, "_takes_tcgen05", lambda a, w: True)
    monkeypatch.setattr(kernels, "fused_takes", lambda *a: False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)

    def note(name, fn):
        def run(*args, **more):
            seen.append(name)
            return fn(*args, **more)
        return run

    monkeypatch.setattr(kernels, "gemm_tcgen05", note("own", lambda a, w, accumulate_into: accumulate_into.add_(a.float() @ w.float().T)))
    monkeypatch.setattr(kernels, "residual_add", note("sum", lambda x, y: x.add_(y.float())))
    monkeypatch.setattr(kernels, "rmsnorm", note("norm", lambda x, w, eps, dtype: x.to(dtype)))
    monkeypatch.setattr(kernels, "add_rmsnorm", note("sum and norm", lambda x, y, w, eps, dtype: x.add_(y.float()).to(dtype)))

    def device_times(*fns):
        out = []
        for fn in fns:
            seen.clear()
            fn()
            out.append(cost[tuple(seen)])
        return out

    monkeypatch.setattr(L, "_device_times", device_times)
    return cost


A, W = torch.ones(300, 8, dtype=torch.bfloat16), torch.ones(16, 8, dtype=torch.bfloat16)


def test_a_sum_that_may_wait_is_timed_with_the_norm_behind_it(timed):
    timed.update({("own",): 7.7, ("sum",): 8.4, ("own", "norm"): 11.4, ("sum and norm",): 10.1})
    x, waiting = torch.zeros(300, 16), []
    L.linear(A, W, accumulate_into=x, defer_add=waiting.append)
    assert len(waiting) == 1 and not x.any()                  # the library's product, whose sum waits
    L.linear(A, W, accumulate_into=x)
    assert len(waiting) == 1 and (x == 8).all()               # without a norm behind it: this library's kernel
    assert L.Choice.timings == {("accumulate_normed", 512, 16, 8): (11.4, 10.1), ("accumulate", 512, 16, 8): (7.7, 8.4)}


@pytest.mark.parametrize("own,taken", [(100.0, "library"), (99.0, "library"), (98.0, "library"), (95.0, "tcgen05"), (104.0, "library")])
def test_a_near_tie_is_the_librarys(timed, own, taken):
    timed.update({("own",): own, ("sum",): 100.0})
    L.linear(A, W, accumulate_into=torch.zeros(300, 16))
    assert L.Choice.table == {("accumulate", 512, 16, 8): taken}
