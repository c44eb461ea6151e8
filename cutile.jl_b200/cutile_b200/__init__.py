"""Python mirror of the Julia call surface kept by libcutile_b200.

Each module carries the name of the reference example whose entry points it
mirrors (examples/<name>.jl) and exposes functions with the same names and
argument order; tensors are torch CUDA tensors laid out like the Julia arrays
(so torch shapes are the Julia shapes reversed).  All arithmetic happens in the
CUDA library; nothing here computes on the host.
"""
import torch  # noqa: F401  (its libraries are loaded before the extension that is linked against them)

from . import _lib  # noqa: F401  (fails loudly when the shared library is missing)
from . import _host

if _host.TORCH_VERSION != torch.__version__:  # it reads tensors by the layout of the torch that it was compiled against
    raise ImportError(f"_host.so was built for torch {_host.TORCH_VERSION}, this is torch {torch.__version__}: "
                      "build it again with `python cutile.jl_b200/csrc/build.py`")
from ._lib import CtbError, version_info, check_device_status  # noqa: F401
from . import softmax, layernorm, matmul, batchmatmul, fmha, moe, multi, vadd, transpose, fft, tiled  # noqa: F401
