"""
Build the in-tree native library ``macromax_b200/libmacromax_b200.so`` for sm_100a with nvcc.

    python -m macromax_b200.build            # rebuild if a source changed
    python -m macromax_b200.build --force    # always rebuild
"""
from __future__ import annotations

import hashlib
import os
import re
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, 'csrc')
INCLUDE = os.path.join(ROOT, 'include')
LIB_NAME = 'libmacromax_b200.so'
LIB_PATH = os.path.join(PKG, LIB_NAME)
STAMP = LIB_PATH + '.srchash'

OBJ_DIR = os.path.join(PKG, '_build')
# Translation units (source, definitions), compiled side by side and linked into one library; a unit whose sources did not
# change keeps its object.  The longest first.
UNITS = [('mmx_capi.cu', ())]
UNITS += [('mmx_len.cu', (f'-DMMX_LEN_PART={part}', f'-DMMX_LEN_DOUBLE={double}')) for double in (1, 0)
          for part in (0, 2, 1, 3)]
UNITS += [(name, ()) for name in ('mmx_loop.cu', 'mmx_loop_f64.cu', 'mmx_gen.cu', 'mmx_gen_f64.cu')]
NVCC_FLAGS = ['-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
              '-Xcompiler', '-fPIC', '-Xcompiler', '-O2', '-Xfatbin', '-compress-all']


def _nvcc() -> str:
    for cand in (os.environ.get('NVCC'), shutil.which('nvcc'), '/usr/local/cuda/bin/nvcc'):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError('nvcc not found: set NVCC or put the CUDA toolkit on PATH')


def _source_hash() -> str:
    h = hashlib.sha256()
    for d in (CSRC, INCLUDE):
        for name in sorted(os.listdir(d)):
            if name.endswith(('.cu', '.cuh', '.h')):
                with open(os.path.join(d, name), 'rb') as f:
                    h.update(name.encode())
                    h.update(f.read())
    h.update(' '.join(NVCC_FLAGS).encode())
    return h.hexdigest()


def up_to_date() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(STAMP):
        return False
    with open(STAMP) as f:
        return f.read().strip() == _source_hash()


def _unit_hash(source: str, defs) -> str:
    """Of one translation unit: its source, the files of this tree that it includes, and the flags."""
    seen, todo = set(), [os.path.join(CSRC, source)]
    h = hashlib.sha256(' '.join([*NVCC_FLAGS, *defs]).encode())
    while todo:
        path = os.path.normpath(todo.pop())
        if path in seen or not os.path.exists(path):
            continue
        seen.add(path)
        with open(path, 'rb') as f:
            text = f.read()
        h.update(os.path.basename(path).encode() + text)
        todo += sorted(os.path.join(os.path.dirname(path), m) for m in re.findall(r'#include "([^"]+)"', text.decode()))
    return h.hexdigest()


def _compile(unit, force: bool, verbose: bool) -> str:
    source, defs = unit
    obj = os.path.join(OBJ_DIR, source + ''.join(defs).replace('=', '') + '.o')
    stamp = obj + '.srchash'
    digest = _unit_hash(source, defs)
    if not force and os.path.exists(obj) and os.path.exists(stamp):
        with open(stamp) as f:
            if f.read().strip() == digest:
                return obj
    cmd = [_nvcc(), *NVCC_FLAGS, *defs, '-I', INCLUDE, '-c', '-o', obj + '.tmp', os.path.join(CSRC, source)]
    if verbose:
        print(' '.join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(obj + '.tmp', obj)
    with open(stamp, 'w') as f:
        f.write(digest)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    with ThreadPoolExecutor(max_workers=min(len(UNITS), os.cpu_count() or 1)) as pool:
        objs = list(pool.map(lambda unit: _compile(unit, force, verbose), UNITS))
    tmp = LIB_PATH + '.tmp'
    cmd = [_nvcc(), *NVCC_FLAGS[:2], '-shared', '-o', tmp, *objs]
    if verbose:
        print(' '.join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(tmp, LIB_PATH)
    with open(STAMP, 'w') as f:
        f.write(_source_hash())
    return LIB_PATH


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose=True))
