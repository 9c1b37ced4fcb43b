"""The C interface as ctypes sees it: every function of kernels.h gets its
argument and return types from the header's own text."""
import ctypes
import os
import re

import pytest

from janas_b200.csrc import ops

HEADER = os.path.join(os.path.dirname(os.path.abspath(ops.__file__)), "kernels.h")


class _Fn:
    argtypes = None
    restype = None


class _Lib:
    def __init__(self):
        self.fns = {}

    def __getattr__(self, name):
        if not name.startswith("jb_"):
            raise AttributeError(name)
        return self.fns.setdefault(name, _Fn())


def test_every_declaration_is_read():
    text = open(HEADER).read()
    lib = _Lib()
    n = ops.declare(lib, text)
    names = set(re.findall(r"\b(jb_\w+)\s*\(", re.sub(r"//[^\n]*", "", text)))
    assert n == len(names) == len(lib.fns) and n >= 20
    f = lib.fns["jb_rmsnorm"]
    assert f.restype is ctypes.c_int
    assert f.argtypes == [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong,
                          ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                          ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_float, ctypes.c_void_p]
    assert lib.fns["jb_attention_scratch"].restype is ctypes.c_longlong
    assert lib.fns["jb_attention_chunk"].argtypes == []
    assert lib.fns["jb_sample"].argtypes[11] is ctypes.c_longlong        # big_cap
    assert lib.fns["jb_sample"].argtypes[8] is ctypes.c_void_p           # unsigned long long *rng


def test_small_headers():
    lib = _Lib()
    assert ops.declare(lib, """
        // int jb_commented_out(int a);
        int jb_one(const float *x, unsigned long long *y, long long n,
                   cudaStream_t st);
        long long jb_two(void);
        unsigned long long jb_three(size_t n, double d, unsigned u, const int32_t *p, int32_t v);
    """) == 3
    assert lib.fns["jb_one"].argtypes == [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong,
                                          ctypes.c_void_p]
    assert lib.fns["jb_two"].argtypes == [] and lib.fns["jb_two"].restype is ctypes.c_longlong
    assert lib.fns["jb_three"].restype is ctypes.c_ulonglong
    assert lib.fns["jb_three"].argtypes == [ctypes.c_size_t, ctypes.c_double, ctypes.c_uint,
                                            ctypes.c_void_p, ctypes.c_int32]
    with pytest.raises(KeyError):
        ops.declare(_Lib(), "int jb_bad(short s);")      # a type the table does not know


def test_which_float_products_go_in_parts():
    """By the weight alone: features and k from a size on, rows that TMA takes, and no k so long that a tile without a
    finite sum could outlast the kernel's waits."""
    ok = ops.lib().jb_gemm_f32_tc_ok
    assert ok(0, 512, 1024) and ok(0, 513, 1028) and ok(0, 151936, 2560) and ok(0, 512, 1 << 17)
    assert not ok(0, 511, 1024) and not ok(0, 512, 1020) and not ok(0, 512, 1026) and not ok(4, 512, 1024)
    assert not ok(0, 512, (1 << 17) + 4)


@pytest.mark.parametrize("m,k", [(6144, 2560), (2560, 9728), (151936, 2560), (512, 32768), (18944, 65536), (513, 1028)])
def test_scratch_of_float_products_is_bounded(m, k):
    """At most 72 MiB whatever the rows (host code; asked without a GPU too), and a plan for less, down to none."""
    L = ops.lib()
    for n in (1, 16, 17, 33, 60, 161, 300, 1000, 2048, 5001, 40000):
        need = L.jb_gemm_f32_tc_scratch(n, m, k)
        assert 0 <= need * 4 <= 72 << 20, (n, need)
        few, many = L.jb_gemm_f32_tc_launches(n, m, k, need), L.jb_gemm_f32_tc_launches(n, m, k, 0)
        assert 1 <= few and many == -(-n // 32), (n, few, many)
