"""Builds ``libunit_b200.so`` (nvcc, sm_100a) and the CPython extension ``_host.*.so`` (g++, torch's headers) in-tree
(no JIT cache)."""
from __future__ import annotations

import importlib.metadata
import os
import shutil
import subprocess
import sys
import sysconfig

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, 'libunit_b200.so')
_SOURCES = [os.path.join(_HERE, 'csrc', 'unit_abi.cu')]
_DEPS = _SOURCES + [os.path.join(_HERE, 'csrc', 'igemm_sm100.cuh'), os.path.join(_HERE, 'csrc', 'layout.cuh'),
                    os.path.join(_HERE, 'csrc', 'tensor_peak.cuh'),
                    os.path.join(os.path.dirname(_HERE), 'include', 'unit_b200.h')]

_HOST_SOURCE = os.path.join(_HERE, 'csrc', 'host_ext.cpp')
_HOST_DEPS = [_HOST_SOURCE, os.path.join(os.path.dirname(_HERE), 'include', 'unit_b200.h')]


def host_path() -> str:
    """The extension's file.  It is compiled against the C++ headers of one torch and one Python, so its name carries
    both: after an upgrade of either the old file is neither fresh nor found."""
    try:
        torch_version = importlib.metadata.version('torch')
    except importlib.metadata.PackageNotFoundError:
        torch_version = 'none'
    return os.path.join(_HERE, f'_host.{sys.implementation.cache_tag}-torch{torch_version}.so')


def _nvcc() -> str:
    for cand in (shutil.which('nvcc'), '/usr/local/cuda/bin/nvcc'):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError('nvcc not found: unit_b200 needs the CUDA toolkit to build its kernels')


def _newer(target: str, deps) -> bool:
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(s) <= t for s in deps)


def is_fresh() -> bool:
    return _newer(LIB_PATH, _DEPS)


def build_host(force: bool = False) -> str:
    """The extension sees torch's tensors directly, so it is built against the installed torch."""
    path = host_path()
    if _newer(path, _HOST_DEPS) and not force:
        return path
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [shutil.which('g++') or 'g++', '-O2', '-std=c++17', '-shared', '-fPIC', '-fvisibility=hidden',
           f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}', '-o', path, _HOST_SOURCE]
    cmd += ['-isystem', os.path.join(root, 'include'), '-isystem', os.path.join(root, 'include', 'torch', 'csrc', 'api', 'include'),
            '-isystem', os.path.join(cuda, 'include'), '-I', sysconfig.get_paths()['include']]
    cmd += ['-L', os.path.join(root, 'lib'), '-lc10', '-lc10_cuda', '-ltorch_cpu', '-ltorch_cuda', '-ltorch_python']
    subprocess.run(cmd, check=True)
    return path


def build(force: bool = False, verbose: bool = False) -> str:
    build_host(force)
    if is_fresh() and not force:
        return LIB_PATH
    cmd = [_nvcc(), '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
           '-shared', '-Xcompiler', '-fPIC', '-o', LIB_PATH] + _SOURCES
    if verbose:
        cmd.insert(1, '-Xptxas')
        cmd.insert(2, '-v')
    subprocess.run(cmd, check=True)
    return LIB_PATH


if __name__ == '__main__':
    print(build(force=True, verbose=True))
