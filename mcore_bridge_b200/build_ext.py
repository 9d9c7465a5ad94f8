"""Builds the sources under ``csrc/``, in-tree: one shared library of CUDA kernels for sm_100a and one CPython module.

The kernels expose a plain C ABI and are loaded through ``ctypes`` (see ``ops/_lib.py``): a handful of ``nvcc``
invocations with no dependency on the torch headers, which work on a machine without a GPU (nvcc cross-compiles).  The
module (``csrc/host``, the host side of the most frequent calls) is compiled against one Python and one torch, which its
file name carries: after an upgrade of either it is missing rather than stale.

Run as ``python -m mcore_bridge_b200.build_ext`` or call :func:`build`.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
REPO_DIR = PKG_DIR.parent
CSRC = REPO_DIR / 'csrc'
LIB_DIR = PKG_DIR / 'lib'
LIB_NAME = 'libmcb200.so'
OBJ_DIR = REPO_DIR / 'build' / 'obj'

NVCC_FLAGS = [
    '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17', '--use_fast_math',
    '-Xcompiler', '-fPIC', '-Xptxas', '-v', '--expt-relaxed-constexpr',
]
# sources whose fp32 results are computed with the full-precision math functions and divisions (denormals are flushed in
# them as everywhere else)
PRECISE_SOURCES = {'attention/attn_sink_grad.cu', 'elementwise/ce_combine.cu', 'elementwise/token_tables.cu',
                   'linear_attention/gdn_inputs.cu', 'linear_attention/gated_delta_rule.cu', 'moe/router_terms.cu'}


def _flags(src: Path) -> list[str]:
    precise = src.relative_to(CSRC).as_posix() in PRECISE_SOURCES
    return ['-ftz=true' if precise and f == '--use_fast_math' else f for f in NVCC_FLAGS]


def _nvcc() -> str:
    cand = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(cand):
        raise RuntimeError('nvcc not found; the CUDA kernels of mcore_bridge_b200 cannot be built')
    return cand


def sources() -> list[Path]:
    return sorted(p for p in CSRC.rglob('*.cu'))


def _deps_hash(src: Path) -> str:
    h = hashlib.sha1()
    h.update(' '.join(_flags(src)).encode())
    h.update(src.read_bytes())
    for hdr in sorted(CSRC.rglob('*.cuh')) + sorted(CSRC.rglob('*.h')):
        h.update(hdr.read_bytes())
    return h.hexdigest()


def _compile_one(src: Path, verbose: bool) -> Path:
    rel = src.relative_to(CSRC)
    obj = OBJ_DIR / rel.with_suffix('.o')
    stamp = obj.with_suffix('.sha1')
    digest = _deps_hash(src)
    if obj.exists() and stamp.exists() and stamp.read_text() == digest:
        return obj
    obj.parent.mkdir(parents=True, exist_ok=True)
    cmd = [_nvcc(), *_flags(src), '-I', str(CSRC), '-c', str(src), '-o', str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    log = obj.with_suffix('.log')
    log.write_text(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f'nvcc failed for {src}:\n{res.stdout}\n{res.stderr}')
    if verbose:
        sys.stderr.write(f'[build_ext] compiled {rel}\n')
    stamp.write_text(digest)
    return obj


def host_name() -> str:
    """File name of the CPython module for the running Python and torch."""
    import re
    import sysconfig

    import torch
    version = re.sub('[^0-9A-Za-z.]', '_', torch.__version__)
    return f'_mcb200_host.torch-{version}.{sysconfig.get_config_var("SOABI")}.so'


def _host_command(out: Path) -> list[str]:
    import sysconfig

    import torch
    inc = Path(torch.__file__).resolve().parent / 'include'
    cuda = Path(_nvcc()).resolve().parent.parent / 'include'
    dirs = [inc, inc / 'torch' / 'csrc' / 'api' / 'include', Path(sysconfig.get_paths()['include']), cuda]
    return ['g++', '-O2', '-std=c++17', '-fPIC', '-shared',
            f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}',
            *(f'-I{d}' for d in dirs), *map(str, sorted((CSRC / 'host').glob('*.cpp'))), '-o', str(out),
            f'-L{inc.parent / "lib"}', '-ltorch_python', '-ltorch_cpu', '-lc10', '-lc10_cuda', '-ldl']


def build_host(verbose: bool = True, force: bool = False) -> Path:
    """Compile the CPython module ``lib/_mcb200_host.*.so`` against this interpreter and its torch. Returns its path."""
    out = LIB_DIR / host_name()
    stamp = OBJ_DIR / f'{out.name}.sha1'
    h = hashlib.sha1()
    for src in sorted(p for e in ('cpp', 'h') for p in (CSRC / 'host').glob(f'*.{e}')):
        h.update(src.read_bytes())
    if out.exists() and stamp.exists() and stamp.read_text() == h.hexdigest() and not force:
        return out
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    tmp = out.with_name(out.name + f'.tmp{os.getpid()}')
    res = subprocess.run(_host_command(tmp), capture_output=True, text=True)
    if res.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f'g++ failed for csrc/host:\n{res.stdout}\n{res.stderr}')
    os.replace(tmp, out)
    stamp.write_text(h.hexdigest())
    if verbose:
        sys.stderr.write(f'[build_ext] linked {out}\n')
    return out


def build(verbose: bool = True, force: bool = False) -> Path:
    """Compile every ``.cu`` under ``csrc/`` and link ``lib/libmcb200.so``, and the host module beside it. Returns the
    library path."""
    if force and OBJ_DIR.exists():
        shutil.rmtree(OBJ_DIR)
    srcs = sources()
    if not srcs:
        raise RuntimeError(f'no CUDA sources under {CSRC}')
    with ThreadPoolExecutor(max_workers=min(8, len(srcs) + 1)) as ex:
        host = ex.submit(build_host, verbose, force)
        objs = list(ex.map(lambda s: _compile_one(s, verbose), srcs))
        host.result()
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    out = LIB_DIR / LIB_NAME
    newest = max(o.stat().st_mtime for o in objs)
    if out.exists() and out.stat().st_mtime >= newest and not force:
        return out
    # link next to the target and rename: a process (or a copy of the tree) never sees a half-written library
    tmp = out.with_name(out.name + f'.tmp{os.getpid()}')
    cmd = [_nvcc(), '-shared', '-o', str(tmp), *map(str, objs), '-gencode', 'arch=compute_100a,code=sm_100a']
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f'link failed:\n{res.stdout}\n{res.stderr}')
    os.replace(tmp, out)
    if verbose:
        sys.stderr.write(f'[build_ext] linked {out}\n')
    return out


if __name__ == '__main__':
    build(force='--force' in sys.argv)
