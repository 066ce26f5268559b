"""The CPython calls' handling of their arguments, as far as it goes without a GPU: a NULL context is refused by the
library after the arguments have been read."""
import ctypes
import os
import subprocess
import sys
import types

import pytest

from colormlm_b200 import _lib as L
from colormlm_b200.s14 import S14Error, S14NumericPipelines

STREAM = 1  # a handle that is only passed on


@pytest.fixture
def pipelines(cuda_lib):
    return S14NumericPipelines(types.SimpleNamespace(_hv=None, handle=None, _calls=L.pycall()))


RECORDS = {"mxfp4_matvec": L.Mxfp4Dispatch, "fp8_matvec": L.Fp8Dispatch, "swiglu_limit": L.SwigluLimitDispatch,
           "route_mix": L.RouteMixDispatch, "moe_accumulate": L.MoeAccumulateDispatch}


@pytest.mark.parametrize("operator", sorted(RECORDS))
def test_a_bound_operator_takes_its_own_record_alone(pipelines, operator):
    call = getattr(pipelines, "cmd_" + operator)
    for name, kind in RECORDS.items():
        if name == operator:
            with pytest.raises(S14Error) as e:
                call(kind(), STREAM)
            assert e.value.code == L.ERR_CONTRACT
        else:
            with pytest.raises(TypeError):
                call(kind(), STREAM)
    for other in (bytes(64), bytearray(24), None, 7):
        with pytest.raises(TypeError):
            call(other, STREAM)


class NamesItsPointer:
    """As torch.cuda.Stream does."""

    def __init__(self, p):
        self._as_parameter_ = p


@pytest.mark.parametrize("handle", [0, 1, 2 ** 63, ctypes.c_void_p(1), ctypes.c_void_p(None), NamesItsPointer(ctypes.c_void_p(5)),
                                    NamesItsPointer(5)])
def test_what_ctypes_takes_as_a_handle_is_taken(pipelines, handle):
    with pytest.raises(S14Error) as e:   # read, then the NULL context is refused
        pipelines.cmd_route_mix(L.RouteMixDispatch(), handle)
    assert e.value.code == L.ERR_CONTRACT


@pytest.mark.parametrize("handle", ["1", 1.0, object(), ctypes.c_uint64(1), NamesItsPointer(1.5), NamesItsPointer(NamesItsPointer("x"))])
def test_what_is_no_handle_is_refused(pipelines, handle):
    with pytest.raises(TypeError):
        pipelines.cmd_route_mix(L.RouteMixDispatch(), handle)


def test_calls_that_need_no_torch_do_not_import_it(cuda_lib):
    """A program with streams and buffers of its own: the module loads and a call runs up to the library without torch."""
    program = """
import sys
from colormlm_b200 import _lib as L, s14
calls = L.pycall()
assert calls.route_mix(None, 1, L.RouteMixDispatch()) == L.ERR_CONTRACT
assert "torch" not in sys.modules
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", program], check=True, cwd=root)
