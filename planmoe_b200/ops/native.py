"""Loader for the in-tree native extension ``planmoe_b200/_C*.so``.

The extension holds every sm_100a kernel, the symmetric-heap runtime and the CPU C++
reference ops.  It is built in-tree by ``planmoe_b200.utils.build`` (never pip-installed),
so the shared object travels with the source tree.

``lib()`` returns the module or raises with the build command; ``available()`` probes.
GPU code paths call ``lib()`` so that a missing extension is a loud error, never a silent
fallback to eager PyTorch.
"""

import functools
import importlib
import os

_LIB = None
_ERR = None


def _try_load():
    global _LIB, _ERR
    if _LIB is not None or _ERR is not None:
        return
    try:
        import torch  # noqa: F401  (libtorch must be loaded before the extension)
        _LIB = importlib.import_module("planmoe_b200._C")
    except Exception as ex:  # ImportError or a loader error
        _ERR = ex


def available():
    _try_load()
    return _LIB is not None


def lib():
    _try_load()
    if _LIB is None:
        raise RuntimeError(
            "planmoe_b200 native extension is not built or failed to load (%r). "
            "Build it with:  python -m planmoe_b200.utils.build" % (_ERR,))
    return _LIB


def maybe_lib():
    """The module, or None when it is absent (CPU-only fallbacks may use this)."""
    _try_load()
    return _LIB


def aligned(t):
    """``t`` contiguous with its first element on a 16-byte boundary: what kernels that move rows as 16-byte vectors take.  A
    contiguous view may start anywhere in its storage."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def first_order(backward):
    """For the backward of an autograd function that runs kernels and has no gradient of its own.  Under create_graph its results
    are the same and raise when they are differentiated, by whatever they depend on: the incoming gradients, the saved inputs and
    those that the forward names in ``ctx.also``.  (``torch.autograd.function.once_differentiable`` looks at the incoming
    gradients alone, and an engine that is asked for certain inputs does not come by its error.)"""
    @functools.wraps(backward)
    def run(ctx, *grads):
        import torch
        if not torch.is_grad_enabled():
            return backward(ctx, *grads)
        with torch.no_grad():
            found = backward(ctx, *grads)
        found = found if isinstance(found, tuple) else (found,)
        values = [t.detach() for t in found if t is not None]
        on = [t for t in (*grads, *ctx.saved_tensors, *getattr(ctx, 'also', ())) if t is not None and t.requires_grad]
        if not values or not on:
            return found
        made = iter(torch._C._functions.DelayedError(SECOND_ORDER, len(values) + len(on))(*values, *on))
        return tuple(None if t is None else next(made) for t in found)
    return run


SECOND_ORDER = ("the gradient was computed by kernels and cannot be differentiated twice; PLANMOE_GEMM=cublas makes a layer of "
                "operations that can")


def force_python_fallback():
    """True when env PLANMOE_NO_NATIVE=1 asks CPU paths to avoid the extension."""
    return os.environ.get("PLANMOE_NO_NATIVE", "0") == "1"
