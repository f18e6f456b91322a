"""Compile the sm_100a CUDA engine into lens_sensor_b200/_lib/liblens_fdtd.so.

The library is built in-tree with nvcc (no JIT cache), so the file travels with
the source tree to the machine that runs it.  Usage:

    python -m lens_sensor_b200.build          # or lens_sensor_b200.build.build()
"""
import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, 'csrc')
LIBDIR = os.path.join(HERE, '_lib')
LIB = os.path.join(LIBDIR, 'liblens_fdtd.so')
# (source, definitions): each compiled on its own, side by side
UNITS = [(f, ()) for f in ('fdtd2d_resident.cu', 'fdtd3d.cu', 'fdtd2d_batch.cu', 'fdtd2d_tb.cu', 'fdtd3d_tb.cu',
                           'fdtd2d.cu')] + \
        [('grid2d_resident.cu', ())] + \
        [('grid2d_resident_k.cu', (f'-DRS_RM={rm}', f'-DRS_GEN={min(2, rm // 2)}')) for rm in range(20, 0, -2)]
ARCH = ['-gencode', 'arch=compute_100a,code=sm_100a']


def nvcc():
    for c in (os.environ.get('NVCC'), '/usr/local/cuda/bin/nvcc', 'nvcc'):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return 'nvcc'


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(ROOT, 'include', 'lens_fdtd.h'))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False, extra=()):
    """Compile the shared library if any source is newer than it."""
    if not force and not _stale():
        return LIB
    os.makedirs(LIBDIR, exist_ok=True)
    flags = ['-O3', '-std=c++17', '-lineinfo', *ARCH, '-Xcompiler', '-fPIC', '-I', os.path.join(ROOT, 'include'),
             '-I', CSRC, '--expt-relaxed-constexpr', *extra]
    work = tempfile.mkdtemp(prefix='build_', dir=LIBDIR)

    def run(cmd):
        if verbose:
            print(' '.join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError('nvcc failed:\n' + r.stdout + r.stderr)
        if verbose and (r.stdout or r.stderr):
            print(r.stdout + r.stderr, flush=True)

    def unit(k):
        src, defs = UNITS[k]
        obj = os.path.join(work, f'{k}.o')
        run([nvcc(), *flags, *defs, '-c', os.path.join(CSRC, src), '-o', obj])
        return obj
    try:
        with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
            objs = list(pool.map(unit, range(len(UNITS))))
        run([nvcc(), *ARCH, '-shared', '-Xcompiler', '-fPIC', '-o', LIB + '.tmp', *objs])
    finally:
        shutil.rmtree(work, ignore_errors=True)
    os.replace(LIB + '.tmp', LIB)
    return LIB


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose=True,
                extra=(['-Xptxas', '-v'] if '--ptxas' in sys.argv else [])))
