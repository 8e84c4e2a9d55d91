"""Where the PyTorch extension (csrc/torch/ext.cpp) lies.  Kept apart from the build, which a process that finds the
file does not need."""
from __future__ import annotations

import hashlib
import importlib.machinery
import importlib.util
import re
from pathlib import Path

DIR = Path(__file__).resolve().parent
CSRC, INCLUDE = DIR.parent / "csrc", DIR.parent / "include"


def torch_dir() -> Path | None:
    """Where the PyTorch is that the extension can be built against: one with CUDA."""
    spec = importlib.util.find_spec("torch")
    if spec is None or not spec.submodule_search_locations:
        return None
    d = Path(spec.submodule_search_locations[0])
    return d if (d / "lib" / "libc10_cuda.so").exists() else None


def torch_ext_path() -> Path | None:
    """The extension's file for the installed PyTorch and this Python, or None where there is none with CUDA.  Its
    name holds both versions and a hash of the source: a file made for another PyTorch, another Python or from
    another source is never taken for it."""
    at = torch_dir()
    if at is None:
        return None
    version = re.search(r"^__version__ = '([^']+)'", (at / "version.py").read_text(), re.M).group(1)
    suffix = importlib.machinery.EXTENSION_SUFFIXES[0]
    sources = [CSRC / "torch" / "ext.cpp", *sorted(INCLUDE.glob("*.h"))]
    if not sources[0].exists():    # a tree without sources: what was built for these versions
        built = sorted(DIR.glob(f"_torch_ext-{version}-*{suffix}"))
        return built[-1] if built else None
    digest = hashlib.sha1(b"".join(p.read_bytes() for p in sources)).hexdigest()[:8]
    return DIR / f"_torch_ext-{version}-{digest}{suffix}"
