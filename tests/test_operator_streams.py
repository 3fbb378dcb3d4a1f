"""CPU: what the Python operators take for a stream."""
import ctypes as C

import pytest


def test_a_stream_is_a_whole_number():
    from lmdeploy_b200 import turbomind as tm
    assert C.c_void_p.from_param(tm._stream(0)) is not None and tm._stream(1 << 40).value == 1 << 40
    for wrong in (b"stream", "stream", 1.0, [0]):
        with pytest.raises(TypeError):
            tm._stream(wrong)
