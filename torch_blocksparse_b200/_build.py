"""Compiles the native code in-tree: the library (CUDA kernels + host table builders) and the
torch module around it.

    python -m torch_blocksparse_b200._build [--force] [--verbose]

The results are torch_blocksparse_b200/libbsp_b200.so, built with nvcc for
sm_100a only, and torch_blocksparse_b200/_ops.so (csrc/torch/, host code: what
a call does around its kernels, against the installed torch).  Object files are
cached under torch_blocksparse_b200/build/ and recompiled when a source or
header is newer.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
SRC_DIR = os.path.join(PKG_DIR, 'csrc')
OBJ_DIR = os.path.join(PKG_DIR, 'build')
LIB_PATH = os.path.join(PKG_DIR, 'libbsp_b200.so')
OPS_SRC = os.path.join(SRC_DIR, 'torch', 'ops.cpp')
OPS_PATH = os.path.join(PKG_DIR, '_ops.so')
INCLUDE_DIR = os.path.join(os.path.dirname(PKG_DIR), 'include')

NVCC_FLAGS = ['-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
              '-Xcompiler', '-fPIC', '-Xcompiler', '-O3',
              '--expt-relaxed-constexpr', '-I', INCLUDE_DIR]


def _nvcc():
    for cand in (os.environ.get('NVCC'), '/usr/local/cuda/bin/nvcc', 'nvcc'):
        if cand and (os.path.isfile(cand) or cand == 'nvcc'):
            return cand
    return 'nvcc'


def _sources():
    return sorted(os.path.join(SRC_DIR, f) for f in os.listdir(SRC_DIR) if f.endswith(('.cu', '.cpp')))


def _headers():
    hs = [os.path.join(SRC_DIR, f) for f in os.listdir(SRC_DIR) if f.endswith(('.h', '.cuh'))]
    hs += [os.path.join(INCLUDE_DIR, f) for f in os.listdir(INCLUDE_DIR) if f.endswith('.h')]
    return hs


def _mtime(p):
    return os.path.getmtime(p) if os.path.exists(p) else 0.0


def needs_build():
    newest_src = max(_mtime(p) for p in _sources() + _headers())
    return _mtime(LIB_PATH) < newest_src


def _ops_need_build():
    return _mtime(OPS_PATH) < max(_mtime(OPS_SRC), _mtime(os.path.join(INCLUDE_DIR, 'bsp.h')))


def _run(cmd, verbose):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(' '.join(cmd) + '\n' + r.stdout + r.stderr)
    return r.returncode == 0


def _build_ops(verbose=False):
    """Compile the torch module; it finds libbsp_b200.so next to itself."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else '/usr/local/cuda'
    inc = [os.path.join(root, 'include'), os.path.join(root, 'include', 'torch', 'csrc', 'api', 'include'),
           os.path.join(cuda, 'include'), sysconfig.get_paths()['include'], INCLUDE_DIR]
    tmp = OPS_PATH + '.%d' % os.getpid()
    cmd = (['g++', '-O3', '-std=c++17', '-fPIC', '-shared', '-fvisibility=hidden',
            '-D_GLIBCXX_USE_CXX11_ABI=%d' % torch.compiled_with_cxx11_abi(), '-DTORCH_EXTENSION_NAME=_ops']
           + [x for d in inc for x in ('-isystem' if d != INCLUDE_DIR else '-I', d)] + [OPS_SRC, '-o', tmp]
           + ['-L' + os.path.join(root, 'lib'), '-lc10', '-lc10_cuda', '-ltorch_cpu', '-ltorch_python', '-ltorch',
              '-L' + os.path.join(cuda, 'lib64'), '-lcudart_static', '-ldl', '-lrt', '-lpthread',
              '-L' + PKG_DIR, '-l:' + os.path.basename(LIB_PATH), '-Wl,-rpath,$ORIGIN'])
    if not _run(cmd, verbose):
        raise RuntimeError('compiling %s failed' % OPS_SRC)
    os.replace(tmp, OPS_PATH)


def build(force=False, verbose=False):
    """Compile every source for sm_100a, link libbsp_b200.so and build the torch module around it.
    Returns the library's path."""
    if force or needs_build():
        _build_lib(force, verbose)
    if force or _ops_need_build():
        _build_ops(verbose)
    return LIB_PATH


def _build_lib(force, verbose):
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()
    newest_hdr = max(_mtime(p) for p in _headers())
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src) + '.o')
        objs.append(obj)
        if force or _mtime(obj) < max(_mtime(src), newest_hdr):
            cmd = [nvcc] + NVCC_FLAGS + (['-Xptxas', '-v'] if verbose else []) + ['-x', 'cu', '-c', src, '-o', obj]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(' '.join(cmd) + '\n' + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError('nvcc failed for ' + cmd[-3])
    link = [nvcc, '-shared', '-o', LIB_PATH] + objs + ['-Xcompiler', '-fPIC', '-lpthread']
    r = subprocess.run(link, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError('link failed')


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='--verbose' in sys.argv))
