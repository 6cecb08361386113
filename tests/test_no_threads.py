"""The plan check runs with the threads it can get: where the system creates none, it still answers
instead of ending the process (pthread_create is interposed and refuses)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
int refuse_threads = 0, refused_threads = 0;
int pthread_create( pthread_t * t, const pthread_attr_t * a, void * (*f)( void * ), void * p )
{
    if( refuse_threads ) { ++refused_threads; return EAGAIN; }
    int (*next)( pthread_t *, const pthread_attr_t *, void * (*)( void * ), void * ) = dlsym( RTLD_NEXT, "pthread_create" );
    return next( t, a, f, p );
}
"""

CHILD = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
from tensors_b200 import matrices as M, ordering as O
from tensors_b200.cholesky import CholeskyDecomposition
A = M.grid_laplacian_3d(int(sys.argv[3]), 1, 1e-2)
c = CholeskyDecomposition(A.outer, A.inner, O.nested_dissection(A), thread_count=4)
c.SymbolicFactorization()
shim = ctypes.CDLL(sys.argv[2])
ctypes.c_int.in_dll(shim, "refuse_threads").value = 1
c.CheckPlan()
print("refused", ctypes.c_int.in_dll(shim, "refused_threads").value)
"""


@pytest.mark.parametrize("size", [24, 40])       # a second thread for the check; threads of its loops too
def test_plan_check_without_threads(tmp_path, size):
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    run = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(lib), str(size)], capture_output=True, text=True,
                         env=dict(os.environ, LD_PRELOAD=str(lib)))
    assert run.returncode == 0, run.stderr
    assert int(run.stdout.split()[1]) > 0
