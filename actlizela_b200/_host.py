"""The native host path of the entry points (``csrc/backends/sm100/torch_host.cpp``).

Each function does a whole pass (checks, allocation, launch) and returns None for anything it does not take; the caller
then runs its Python checks, which raise or go on.  Until the native library has been loaded, every function is
``decline``.  Callers look the functions up in this module at every call (``_host.forward(...)``).
"""
from __future__ import annotations

NAMES = ("forward", "varlen", "projections", "prepare_inputs", "decode_step", "verify_step", "commit_step",
         "rmsnorm_gated", "out_proj_gemm")
# C-ABI entries in the order the extension binds them
ENTRIES = ("select", "workspace_bytes", "forward_prepared", "varlen_workspace_bytes", "forward_varlen",
           "forward_varlen_device", "projections_workspace_bytes", "forward_projections", "last_failure", "prepare_inputs",
           "decode_step", "verify_step", "commit_step", "rmsnorm_gated", "out_proj")
_module = None


def decline(*_):
    return None


for _name in NAMES:
    globals()[_name] = decline


def bind(lib, path, override):
    """Bind the extension to the entries of a loaded native library (``lib``: its ctypes view)."""
    global _module
    import ctypes
    import importlib.util
    if _module is None:
        import torch  # noqa: F401  (the extension resolves its symbols from torch's libraries)
        spec = importlib.util.spec_from_file_location("actlize_la_sm100_host", path)
        _module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(_module)
    _module.bind(tuple(ctypes.cast(getattr(lib, "actlize_la_sm100_" + name), ctypes.c_void_p).value for name in ENTRIES), override)
    for name in NAMES:
        globals()[name] = getattr(_module, name)


def configured(device_index):
    """The bound library is set up on this device."""
    if _module is not None:
        _module.configured(device_index)
