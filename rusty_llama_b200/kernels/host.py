"""What a launch costs the host: calling the kernel libraries' launchers, checking their tensors, and the few tensor operations in between.

`csrc/host_calls.cpp` does this natively (an `add_rmsnorm` with the tensor of its result: 6.2 us instead of 10.9, of which the driver has 3; a
sublayer of nine kernels: 92 us a pass instead of 165, which is the host's time); the classes and functions below are the same in Python,
used until a library is first asked for if that module is not built yet, where it cannot be built (no Python or PyTorch headers) and where there is no GPU to launch on.
Results and errors are the same.
"""

from __future__ import annotations

import ctypes
import operator
import os
import re
import threading
from typing import Dict, List, Optional, Tuple

import torch

from ..errors import KernelError
from . import build


_MOST_FLOATS, _MOST_INTS = 8, 56
_TOO_MANY = f"a launcher takes {_MOST_FLOATS} floats and {_MOST_INTS} integers and tensors at most"


class PythonLauncher:
    """A launcher called with tensors, numbers and None as they are.  kinds: of every argument 'p' (a pointer: a tensor, an address or
    None), 'i' (a whole number) or 'f' (a float); calls are checked against it.  Without kinds each argument goes by its own type."""

    def __init__(self, address: int, wide: bool, kinds: Optional[str] = None):
        if kinds is not None and (kinds.count("f") > _MOST_FLOATS or len(kinds) - kinds.count("f") > _MOST_INTS):
            raise TypeError(_TOO_MANY)
        self.fn = ctypes.CFUNCTYPE(ctypes.c_longlong if wide else ctypes.c_int)(address)
        self.kinds = kinds

    def __call__(self, *args):
        kinds = self.kinds
        if kinds is None:
            kinds = ["f" if isinstance(a, float) else "p" if a is None or isinstance(a, torch.Tensor) else "i" for a in args]
        elif len(kinds) != len(args):
            raise TypeError(f"this launcher takes {len(kinds)} arguments, not {len(args)}")
        if kinds is not self.kinds and (sum(k == "f" for k in kinds) > _MOST_FLOATS or sum(k != "f" for k in kinds) > _MOST_INTS):
            raise TypeError(_TOO_MANY)
        given = []
        for n, (kind, a) in enumerate(zip(kinds, args)):
            if kind == "f":
                given.append(ctypes.c_float(a))
            elif isinstance(a, int):
                given.append(ctypes.c_longlong(a))
            elif kind == "i":
                given.append(ctypes.c_longlong(operator.index(a)))  # (refuses floats and None)
            elif isinstance(a, torch.Tensor):
                given.append(ctypes.c_void_p(a.data_ptr()))
            elif a is None:
                given.append(ctypes.c_void_p(0))
            else:
                raise TypeError(f"argument {n + 1} of a launcher is a tensor, an address or None, not {type(a).__name__}")
        return self.fn(*given)


def python_cuda(t: torch.Tensor, what: str, dtype=None, contiguous=True) -> torch.Tensor:
    if not isinstance(t, torch.Tensor):
        raise KernelError(f"{what}: not a tensor")
    if not t.is_cuda:
        raise KernelError(f"{what}: tensor is on {t.device}, the kernels run on CUDA only")
    if dtype is not None and not isinstance(dtype, torch.dtype):
        raise TypeError("cuda: dtype is not a torch.dtype")
    if dtype is not None and t.dtype != dtype:
        raise KernelError(f"{what}: dtype {t.dtype}, expected {dtype}")
    if contiguous and not t.is_contiguous():
        raise KernelError(f"{what}: tensor is not contiguous")
    return t


def python_rows(t: torch.Tensor, what: str) -> int:
    """Row stride of a 2-D tensor whose rows are dense."""
    if not isinstance(t, torch.Tensor):
        raise TypeError("rows(tensor, what)")
    if t.dim() != 2 or t.stride(1) != 1:
        raise KernelError(f"{what}: expected a 2-D tensor with dense rows")
    return t.stride(0)


def python_matrices(t: torch.Tensor, other: Optional[torch.Tensor], like: torch.Tensor, what: str) -> Tuple[int, int, int, int, int]:
    """(matrices, rows, columns, row stride, matrix stride) of a 3-D tensor of like's type and device whose rows are dense; other: None or one
    that has to lie in the same way."""
    if not (isinstance(t, torch.Tensor) and isinstance(like, torch.Tensor) and (other is None or isinstance(other, torch.Tensor))):
        raise TypeError("matrices(tensor, tensor or None, tensor, what)")
    if t.dim() != 3 or t.stride(2) != 1 or t.dtype != like.dtype or t.device != like.device:
        raise KernelError(f"{what}: expected a 3-D tensor with dense rows beside the others")
    if other is not None and (other.shape != t.shape or other.stride() != t.stride() or other.dtype != t.dtype or other.device != t.device):
        raise KernelError(f"{what}: two tensors that do not lie in the same way")
    return (*t.shape, t.stride(1), t.stride(0))


def python_odd(x: torch.Tensor, w: torch.Tensor) -> bool:
    """Whether rows of the two cannot be moved in 16-byte pieces (eight 16-bit numbers)."""
    if not (isinstance(x, torch.Tensor) and isinstance(w, torch.Tensor)):
        raise TypeError("odd(x, w)")
    if x.dim() != 2 or w.dim() < 1:
        raise IndexError("odd: rows expected")
    return bool(x.shape[1] % 8 or x.stride(0) % 8 or w.stride(0) % 8 or x.data_ptr() % 16 or w.data_ptr() % 16)


def python_stream() -> int:
    # (without making a Stream object: 0.3 us a launch, `torch.cuda.current_stream().cuda_stream` takes 3.3)
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def python_empty(like: torch.Tensor, dtype, *sizes: int) -> torch.Tensor:
    if not (isinstance(like, torch.Tensor) and isinstance(dtype, torch.dtype) and 1 <= len(sizes) <= 4):
        raise TypeError("empty(like, dtype, one to four sizes)")
    return torch.empty(sizes, dtype=dtype, device=like.device)


def python_columns(t: torch.Tensor, first: int, end: int) -> torch.Tensor:
    if not isinstance(t, torch.Tensor):
        raise TypeError("columns(tensor, first, end)")
    return t.narrow(1, first, end - first)  # (what is not there is refused, not left out)


cuda, rows, matrices, odd, stream = python_cuda, python_rows, python_matrices, python_odd, python_stream
empty, columns, launcher = python_empty, python_columns, PythonLauncher

_lock = threading.Lock()
_bound: List[Tuple[dict, Dict[str, str]]] = []


def bind(namespace: dict, **names: str) -> None:
    """Puts this module's functions into another's namespace, under names of its own, and puts the native ones there once they are loaded."""
    with _lock:
        _bound.append((namespace, names))
        namespace.update((own, globals()[name]) for own, name in names.items())


def _find_native(importing: bool = False) -> None:
    """Takes the native module up: at import where it is built, which touches neither CUDA nor a compiler (functions that change under code that
    has run already cost its calls 1 to 3 us a sublayer), else with the first library.  It is built where a process that uses a GPU finds it
    missing; a run of shapes alone stays with Python."""
    with _lock:
        if "_module" in globals():
            return
        try:
            module = build.built_host_calls() if importing else build.load_host_calls(torch.cuda.is_initialized())
            if module is None and (importing or not torch.cuda.is_initialized()):
                return  # (asked again by the next library)
        except Exception as e:  # whatever is missing on this machine: the Python side does the same
            build._say(f"host_calls.cpp is not used: {str(e).strip().splitlines()[-1][:200] if str(e).strip() else type(e).__name__}")
            module = None
        globals()["_module"] = module
        if module is None:
            return
        module.set_error(KernelError)
        for name in ("cuda", "rows", "matrices", "odd", "stream", "empty", "columns", "launcher"):
            globals()[name] = getattr(module, name)
        for namespace, names in _bound:
            namespace.update((own, globals()[name]) for own, name in names.items())


_find_native(importing=True)


def __getattr__(name: str):
    if name == "_module":  # the native module, or None
        _find_native()
        return globals().get("_module")
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


_RETURNS = {"int": False, "long long": True}


def launcher_kinds(source: str) -> Dict[str, Tuple[bool, str]]:
    """The launchers that a source exports: whether each returns 64 bits, and the kinds of its arguments as `PythonLauncher` takes them."""
    found = {}
    for returns, name, declared in re.findall(r"^RL_API\s+([\w ]+?)\s+(rl_\w+)\(([^)]*)\)", source, re.M):
        kinds = ""
        for argument in filter(None, (a.strip() for a in declared.split(","))):
            kind = " ".join(w for w in argument.split()[:-1] if w != "const")
            if "*" in argument or kind == "cudaStream_t":
                kinds += "p"
            elif kind in ("int", "long long", "unsigned", "unsigned int"):
                kinds += "i"
            elif kind == "float":
                kinds += "f"
            else:
                raise KernelError(f"{name}: no way to pass '{argument}'")
        found[name] = (_RETURNS[returns], kinds)
    return found


class Library:
    """A kernel library's launchers as attributes, made when first asked for."""

    def __init__(self, name: str):
        _find_native()
        self._cdll = build.load(name)
        with open(os.path.join(build.CSRC_DIR, name + ".cu")) as f:
            self._kinds = launcher_kinds(f.read())

    def __getattr__(self, name: str):
        if name not in self._kinds:
            raise AttributeError(name)
        wide, kinds = self._kinds[name]
        fn = launcher(ctypes.cast(getattr(self._cdll, name), ctypes.c_void_p).value, wide, kinds)
        setattr(self, name, fn)
        return fn

    def rl_error_text(self) -> bytes:
        return self._cdll.rl_error_text()


_libraries: Dict[str, Library] = {}


def library(name: str) -> Library:
    """The library of `csrc/<name>.cu`, built first if need be."""
    lib = _libraries.get(name)
    if lib is None:
        lib = _libraries[name] = Library(name)
    return lib
