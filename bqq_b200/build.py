"""Build libbqq_b200.so (sm_100a) and the Python module's native side in-tree.

Each .cu under csrc/ is compiled to an object file in parallel with nvcc, then linked
into bqq_b200/libbqq_b200.so; csrc/bqq_torch.cpp becomes the extension module
bqq_b200/_bqq_torch.so with g++ against the installed torch.  Objects are rebuilt only when
a source or header is newer.  Usable as `python -m bqq_b200.build [--force]`.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, 'csrc')
OBJ = os.path.join(PKG, 'build')
LIB = os.path.join(PKG, 'libbqq_b200.so')
EXT = os.path.join(PKG, '_bqq_torch.so')

NVCC_FLAGS = ['-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
              '-Xcompiler', '-fPIC', '-I' + os.path.join(ROOT, 'include'), '-I' + CSRC]


def nvcc_path() -> str:
    exe = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(exe):
        raise RuntimeError('nvcc not found; the bqq_b200 CUDA library cannot be built')
    return exe


def _torch_command(src: str) -> list:
    """g++ command of the extension module: linked against torch and, by its own folder, libbqq_b200.so."""
    import sysconfig

    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(nvcc_path())), 'include')
    inc = [os.path.join(base, 'include'), os.path.join(base, 'include', 'torch', 'csrc', 'api', 'include'), cuda,
           sysconfig.get_paths()['include'], os.path.join(ROOT, 'include')]
    return ['g++', '-O2', '-std=c++17', '-fPIC', '-shared', '-fvisibility=hidden', '-w',
            f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}', *('-I' + i for i in inc), src, '-o', EXT,
            '-L' + os.path.join(base, 'lib'), '-L' + PKG, '-ltorch_python', '-ltorch', '-ltorch_cpu', '-ltorch_cuda',
            '-lc10', '-lc10_cuda', '-l:libbqq_b200.so', '-Wl,-rpath,$ORIGIN']


def _newest_header() -> float:
    hdrs = glob.glob(os.path.join(CSRC, '*.cuh')) + glob.glob(os.path.join(ROOT, 'include', '*.h'))
    return max(os.path.getmtime(h) for h in hdrs)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = nvcc_path()
    srcs = sorted(glob.glob(os.path.join(CSRC, '*.cu')))
    hdr_time = _newest_header()
    jobs = []
    objs = []
    for src in srcs:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + '.o')
        objs.append(obj)
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time)
        if stale:
            jobs.append([nvcc, *NVCC_FLAGS, *(['-Xptxas', '-v'] if verbose else []), '-c', src, '-o', obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose:
                    sys.stderr.write(r.stderr)
                if r.returncode != 0:
                    raise RuntimeError('nvcc failed: ' + ' '.join(cmd) + '\n' + r.stdout + r.stderr)
    if jobs or not os.path.exists(LIB) or force:
        r = subprocess.run([nvcc, '-shared', '-o', LIB, *objs], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError('link failed:\n' + r.stdout + r.stderr)
    src = os.path.join(CSRC, 'bqq_torch.cpp')
    if force or not os.path.exists(EXT) or os.path.getmtime(EXT) < max(os.path.getmtime(src), os.path.getmtime(__file__),
                                                                       _newest_header()):
        cmd, r = run(_torch_command(src))
        if r.returncode != 0:
            raise RuntimeError('g++ failed: ' + ' '.join(cmd) + '\n' + r.stdout + r.stderr)
    return LIB


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='-v' in sys.argv))
