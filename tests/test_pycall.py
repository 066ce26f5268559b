"""The CPython calls' handling of their arguments, as far as it goes without a GPU: a NULL context is refused by the
library after the arguments have been read."""
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
