"""Fields of a live context that tests set and no caller can: a small library built
from the context's own header."""
import ctypes as C
import functools
import subprocess
import tempfile
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include "mg_internal.cuh"
#include "tc.cuh"
__global__ void k_report(int* status) { mg::tc::report_timeout(status); }
extern "C" {
// the waits for the Coulomb CG's sums give up after so many clocks, from an iteration on
void poke_cg_sum_wait(mg_ctx* c, long long clocks, int from) {
    c->cg_sum_wait = clocks;
    c->cg_sum_wait_from = from;
}
// a kernel on the context's stream that reports what a tensor-core kernel reports whose
// wait has run out
int poke_tc_timeout(mg_ctx* c) {
    k_report<<<1, 1, 0, c->stream>>>(c->tc_status);
    return (int)cudaGetLastError();
}
}
"""


@functools.cache
def load():
    from mocca_gb300.build import CSRC, nvcc
    d = Path(tempfile.mkdtemp())
    (d / "poke.cu").write_text(SOURCE)
    subprocess.run([nvcc(), "-std=c++17", "-shared", "-cudart", "shared", "-Xcompiler", "-fPIC",
                    "-gencode", "arch=compute_103a,code=sm_103a", "-I", str(CSRC), "-o",
                    str(d / "poke.so"), str(d / "poke.cu")], check=True)
    lib = C.CDLL(str(d / "poke.so"))
    lib.poke_cg_sum_wait.argtypes = [C.c_void_p, C.c_longlong, C.c_int]
    lib.poke_cg_sum_wait.restype = None
    lib.poke_tc_timeout.argtypes = [C.c_void_p]
    lib.poke_tc_timeout.restype = C.c_int
    return lib
