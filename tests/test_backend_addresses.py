"""Addresses given to the Backend operations: integers, or None for the null
address; host data and other objects are refused before the library is called."""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("bad", [b"0123456789abcdef", "0123456789abcdef", np.zeros(4), np.zeros(4).ctypes,
                                 (ctypes.c_double * 4)(), ctypes.c_void_p(64), 1.5, [64]],
                         ids=["bytes", "str", "array", "array-ctypes", "c-array", "c_void_p", "float", "list"])
def test_what_is_no_address_is_refused(gs, bad):
    calls = {
        "dot": [lambda p: gs.dot(4, p, 64, 64, gs.F64), lambda p: gs.dot(4, 64, 64, 64, gs.F64, p)],
        "dot_noalloc": [lambda p: gs.dot_noalloc(4, 64, p, 64, gs.F64)],
        "vector_op": [lambda p: gs.vector_op(gs.VEC_AXPY, 4, p, 64), lambda p: gs.vector_op(gs.VEC_AXPY, 4, 64, 64, alpha_ptr=p)],
        "scalar_op": [lambda p: gs.scalar_op(0, p, 64, 64), lambda p: gs.scalar_op(0, None, None, p)],
        "apply_block_inverses3x3": [lambda p: gs.apply_block_inverses3x3(3, p, 64, 64, gs.F64)],
    }

    class Matrix:  # no device here: the address is refused before the handle is used
        _h = ctypes.c_void_p(0)

    calls["spmv"] = [lambda p: gs.spmv(Matrix, p, 64), lambda p: gs.spmv(Matrix, 64, p)]
    calls["gauss_seidel_color"] = [lambda p: gs.gauss_seidel_color(Matrix, p, 0, 4, 64, 64, 1.0)]
    calls["block_gauss_seidel_color3x3"] = [lambda p: gs.block_gauss_seidel_color3x3(Matrix, 64, 0, 4, p, 64, 64, 1.0)]
    for name, fs in calls.items():
        for f in fs:
            with pytest.raises(TypeError):
                f(bad)


def test_null_addresses_reach_the_librarys_own_check(gs):
    for f in (lambda: gs.dot(4, None, None, None, gs.F64), lambda: gs.vector_op(gs.VEC_AXPY, 4, None, 0),
              lambda: gs.scalar_op(0, None, None, None)):
        with pytest.raises(gs.SolverError):
            f()
