"""GPU: a complex64 batch whose tile programs cannot have their memory runs on the
engine, and reports an error only when that cannot have its own either.

The library's objects are linked once more with cudaMalloc wrapped
(tests/cpp/failing_malloc.cpp): requests above a limit are refused on the host.
A child process runs a copy of the package with that library.
"""
import ctypes as C
import glob
import os
import shutil
import subprocess
import sys

import pytest

from conftest import PKG_DIR, ROOT

pytestmark = pytest.mark.gpu

CASES = ("refused", [13] * 8 + [8, 10, 12], 60)
STATES = sum(2 * 8 << n for n in CASES[1]) # bytes of the tile path's state buffer


@pytest.fixture(scope="module")
def package(tmp_path_factory):
    d = tmp_path_factory.mktemp("refused")
    pkg = d / "pennylane_lightning_kokkos"
    shutil.copytree(os.path.join(PKG_DIR, "pennylane_lightning_kokkos"), pkg, ignore=shutil.ignore_patterns("*.so", "__pycache__"))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-shared", "-Xcompiler", "-fPIC", "-o", str(pkg / "libplk_gb300.so"), "-gencode",
                    "arch=compute_103a,code=sm_103a", os.path.join(ROOT, "tests", "cpp", "failing_malloc.cpp")]
                   + sorted(glob.glob(os.path.join(PKG_DIR, "_build", "*.o")))
                   + ["-Xlinker", "--wrap=cudaMalloc", "-lcudart_static", "-lrt", "-ldl", "-lpthread"], check=True)
    return str(d)


def child(package, what):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), package, what], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("what", ["states", "everything"])
def test_refused_memory(package, what):
    assert "done" in child(package, what)


def main(package, what):
    sys.path[:0] = [package, os.path.dirname(os.path.abspath(__file__)), ROOT, os.path.join(ROOT, "oracle")]
    from pennylane_lightning_kokkos import _native as N
    assert os.path.dirname(N.LIB_PATH).startswith(package)
    from pennylane_lightning_kokkos.batch import CircuitBatch
    from test_gpu_batch import check_against_oracle, make_cases

    limit = N.lib.malloc_limit
    limit.argtypes = [C.c_size_t]
    cases = make_cases(*CASES)
    b = CircuitBatch("c64")
    for c in cases:
        b.add(*c)
    if what == "states": # all but the buffer of the states
        limit(STATES - 1)
        ev, jac = b.run()
        assert N.lib.malloc_refused() == 1
        assert b.last_time()[1] <= 2 # the engine's launches
        check_against_oracle(cases, ev, b.gradients(jac), 1e-4)
        ev2, jac2 = b.run()
        assert (ev2 == ev).all() and (jac2 == jac).all()
    else:
        limit(16)
        try:
            b.run()
        except N.NativeError as e:
            assert "OUT_OF_MEMORY" in str(e) or "out of memory" in str(e), e
        else:
            raise AssertionError("no error")
    limit((1 << 64) - 1) # with memory again, a batch that grows goes back to tiles
    extra = make_cases("one more", [7], 30)
    b.add(*extra[0])
    ev, jac = b.run()
    assert b.last_time()[1] > 2
    check_against_oracle(cases + extra, ev, b.gradients(jac), 1e-4)
    b.close()
    print("done")


if __name__ == "__main__":
    main(*sys.argv[1:])
