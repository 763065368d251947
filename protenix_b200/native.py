"""Access to ``_C.so``, the native host path (``csrc/torch_ext.cpp``), and the parameter look-ups it keeps per module."""
from __future__ import annotations

import importlib
import os
from typing import Sequence, Tuple

from . import _lib

_ext = None


def load():
    """The extension module, bound to the kernel library; raises if it has not been built."""
    global _ext
    if _ext is None:
        path = os.path.join(_lib.HERE, "_C.so")
        if not os.path.exists(path):
            raise RuntimeError(f"{path} is missing: build it with `python -m protenix_b200.build`. "
                               "This package has no fallback path.")
        ext = importlib.import_module("protenix_b200._C")
        ext.bind_library(_lib.load()._handle)
        _ext = ext
    return _ext


def params(root, group: str, spec: Sequence[Tuple[str, str, Tuple[int, ...]]], scalars: Sequence[str]):
    """A ``Params`` object of a ``group`` over ``root``: spec lists (path of a parameter, kind, shape), scalars the paths of plain
    attributes.  The path's last part is the name, the parts before it submodules, which are checked for identity."""
    checks, places = [], []

    def owner(path):
        module = root
        *subs, name = path.split(".")
        for sub in subs:
            checks.append((module._modules, sub))
            module = module._modules[sub]
        return module, name

    for path, kind, shape in spec:
        module, name = owner(path)
        places.append((module._parameters, name, kind, list(shape), module))
    attributes = [owner(path) for path in scalars]
    return load().Params(group, root, list(dict(((id(d), n), (d, n)) for d, n in checks).values()), places, attributes)


def kept(module, make, name: str = "_px_params"):
    """``make()``, kept in the module's __dict__ until one of the submodules it looked through is replaced.  A module that has
    taken over the __dict__ of another one (a replica, a shallow copy) makes its own."""
    held = module.__dict__.get(name)
    if held is None or not held.current(module):
        held = make()
        module.__dict__[name] = held
    return held


def under(prefix: str, group: str, spec, scalars):
    """The same description seen from a parent module."""
    return group, [(f"{prefix}.{p}", k, s) for p, k, s in spec], [f"{prefix}.{p}" for p in scalars]
