"""A result whose copy to the host fails is reported."""
import pytest


def test_failed_result_copy_raises(tp):
    """A result whose copy to the host fails is an error, not arrays of what the memory held."""
    destroyed = []

    class Lib:
        tp_result_info = staticmethod(lambda *a: tp._abi.TP_OK)
        tp_result_copy = staticmethod(lambda *a: tp._abi.TP_E_CUDA)
        tp_result_elapsed_ms = staticmethod(lambda *a: tp._abi.TP_OK)
        tp_result_destroy = staticmethod(destroyed.append)
        tp_last_error = staticmethod(lambda ctx: b"result copy: out of memory")

    ctx = object.__new__(tp.Context)
    ctx.lib, ctx.handle = Lib, 1
    with pytest.raises(RuntimeError, match="out of memory"):
        ctx._collect("result")
    assert destroyed == ["result"]
