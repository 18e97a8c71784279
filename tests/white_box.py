"""Access to a context's internal state, for tests of what the C ABI cannot
bring about: a few lines of C++ over the library's own headers."""
import ctypes as C
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "satin-computerasteriser_b200")

SOURCE = r"""
#include "cr_internal.h"
#include "cr_pack.h"
extern "C" {
void set_sort_wait_limit(cr_context *c, uint32_t polls) { c->sort_wait_limit = polls; }
uint32_t get_sort_wait_limit(const cr_context *c) { return c->sort_wait_limit; }
void *sort_indices(const cr_context *c, int k) { return c->pack->idx[k]; }
void *sort_ties(const cr_context *c) { return c->pack->radix.ties; }
}
"""


def build(tmp_path, cr):
    """The helper library, compiled into tmp_path."""
    nvcc = os.path.realpath(__import__("importlib").import_module(f"{cr.__name__}.build").nvcc())
    cuda = os.path.dirname(os.path.dirname(nvcc))
    src, so = os.path.join(tmp_path, "white_box.cpp"), os.path.join(tmp_path, "white_box.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-w", "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"), "-I",
                    os.path.join(cuda, "include"), src, "-o", so], check=True)
    lib = C.CDLL(so)
    lib.set_sort_wait_limit.argtypes = [C.c_void_p, C.c_uint32]
    lib.get_sort_wait_limit.argtypes = [C.c_void_p]
    lib.get_sort_wait_limit.restype = C.c_uint32
    lib.sort_indices.argtypes = [C.c_void_p, C.c_int]
    lib.sort_indices.restype = C.c_void_p
    lib.sort_ties.argtypes = [C.c_void_p]
    lib.sort_ties.restype = C.c_void_p
    return lib
