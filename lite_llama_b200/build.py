"""Build the in-tree C-ABI shared library ``libb200lite.so`` with nvcc for sm_100a.

nvcc cross-compiles without a GPU, so this runs in the GPU-less build container; the ``.so``
then travels with the repo snapshot to the B200 box. No torch headers are involved: the
library only depends on the (statically linked) CUDA runtime.

Usage:
    python -m lite_llama_b200.build            # incremental
    python -m lite_llama_b200.build --force

``build(sources=...)`` compiles and links only the named sources (plus the library plumbing): a first run that
serves one model family does not wait for the kernels of the others.  A library that already holds the wanted
sources (a fuller build) is left alone; a later full build relinks.
"""

from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

CSRC = Path(__file__).resolve().parent / "csrc"
OUT = Path(__file__).resolve().parent / "libb200lite.so"
HEADER = CSRC.parents[1] / "include" / "b200_lite_kernels.h"
FAST_SRC = CSRC / "host" / "fast_calls.cpp"
FAST_OUT = Path(__file__).resolve().parent / "_fast.so"
OBJ_DIR = CSRC / "build"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stamp(src: Path) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    h.update(src.read_bytes())
    for hdr in sorted(CSRC.glob("*.cuh")):
        h.update(hdr.read_bytes())
    return h.hexdigest()


def _compile(src: Path, force: bool) -> Path:
    obj = OBJ_DIR / (src.stem + ".o")
    stamp_file = OBJ_DIR / (src.stem + ".stamp")
    stamp = _stamp(src)
    if not force and obj.exists() and stamp_file.exists() and stamp_file.read_text() == stamp:
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    stamp_file.write_text(stamp)
    return obj


# plumbing every subset needs (error strings, launch counter, TMA descriptors)
BASE_SOURCES = ("core", "tma_desc")
# what the layer-list decoders launch between them: dense tcgen05 GEMM, fp32 / odd-shape / per-head / grouped GEMM,
# residual streams (sequential and parallel blocks), state-space and gated recurrences, attention, rotary and
# latent-attention kernels, expert routing, argmax and expert sum.  Each
# registered architecture names its own subset (executor.registry.Architecture.sources).
LAYERED_SOURCES = ("gemm_dense", "gemm_pair", "gemm_simt", "gemm_rows_mma", "residual_stream", "parallel_stream", "ssm_scan",
                   "decay_attention_mma", "gated_recurrence", "gated_linear_attention", "mlstm", "hyper_stream", "tanh_norm_stream",
                   "attention_sink",
                   "rotary_heads", "latent_attention", "moe_routing", "elementwise")
LINK_STAMP = OBJ_DIR / "link.stamp"


def linked_sources() -> set[str]:
    """Source stems the current library was linked from (empty when there is none)."""
    if not OUT.exists() or not LINK_STAMP.exists():
        return set()
    return set(LINK_STAMP.read_text().split())


def fast_tag(torch_version: str) -> str:
    """What a build of the extension is good for.  It calls the library through bare function pointers, so one of another
    header, source, interpreter or torch must not be used: the header and the source by their contents."""
    h = hashlib.sha256(FAST_SRC.read_bytes() + HEADER.read_bytes())
    return f"{torch_version} {sys.version_info.major}.{sys.version_info.minor} {h.hexdigest()}"


def build_fast(force: bool = False) -> str | None:
    """The native form of the hot shims, built against this interpreter and this torch.  None, or why it could not be built:
    the shims then run in Python, slower on the host and otherwise the same (an earlier extension does not stay)."""
    stamp_file = OBJ_DIR / "fast_calls.stamp"
    try:
        import torch
    except ImportError as e:
        FAST_OUT.unlink(missing_ok=True)
        return str(e)
    root = Path(torch.__file__).resolve().parent
    include = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"],
               Path(_nvcc()).resolve().parent.parent / "include"]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DBUILT_FOR="{fast_tag(torch.__version__)}"',
           *(f"-I{d}" for d in include), str(FAST_SRC), "-o", str(FAST_OUT), f"-L{root / 'lib'}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    stamp = hashlib.sha256((" ".join(cmd) + sys.version).encode() + FAST_SRC.read_bytes()).hexdigest()
    if not force and FAST_OUT.exists() and stamp_file.exists() and stamp_file.read_text() == stamp:
        return None
    FAST_OUT.unlink(missing_ok=True)
    stamp_file.unlink(missing_ok=True)
    try:
        res = subprocess.run(cmd, capture_output=True, text=True)
    except OSError as e:
        return str(e)
    if res.returncode != 0:
        FAST_OUT.unlink(missing_ok=True)
        return res.stderr or f"{cmd[0]} returned {res.returncode}"
    stamp_file.write_text(stamp)
    return None


def build(force: bool = False, verbose: bool = True, sources: tuple[str, ...] | None = None) -> Path:
    OBJ_DIR.mkdir(exist_ok=True)
    every = sorted(CSRC.glob("*.cu"))
    if not every:
        raise RuntimeError(f"no CUDA sources under {CSRC}")
    if sources is not None:
        wanted = set(BASE_SOURCES) | set(sources)
        have = linked_sources()
        if wanted <= have and not force:
            wanted = have                     # a fuller library is kept (and refreshed if its sources changed)
        every = [s for s in every if s.stem in wanted]
    with ThreadPoolExecutor(max_workers=min(8, len(every)) + 1) as pool:
        fast = pool.submit(build_fast, force)
        objs = list(pool.map(lambda s: _compile(s, force), every))
    why = fast.result()
    if why and verbose:
        print(f"[b200lite] {FAST_OUT.name} was not built, the shims run in Python: {why}")
    newest = max(o.stat().st_mtime for o in objs)
    stems = sorted(s.stem for s in every)
    if force or not OUT.exists() or OUT.stat().st_mtime < newest or linked_sources() != set(stems):
        cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
               "-o", str(OUT), *map(str, objs)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
        LINK_STAMP.write_text(" ".join(stems))
        if verbose:
            print(f"[b200lite] linked {OUT} from {len(objs)} objects")
    elif verbose:
        print(f"[b200lite] {OUT.name} is up to date")
    return OUT


if __name__ == "__main__":
    build(force="--force" in sys.argv)
