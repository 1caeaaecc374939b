"""What an error word of the device is reported as."""
import ctypes

import pytest


# the words kernels set: indices out of range, a quicksort's corrupted
# partition, a grid barrier that was given up
@pytest.mark.parametrize("bits,says,says_not", [
    (1, ["out-of-range index"], ["barrier", "partition"]), (8, ["out-of-range index"], ["barrier", "partition"]),
    (128, ["out-of-range index"], ["barrier", "partition"]),
    (64, ["partition in a quicksort"], ["barrier", "out-of-range"]),
    (256, ["barrier"], ["partition", "out-of-range"]),
    (256 | 8, ["barrier", "out-of-range index"], ["partition"]),
    (256 | 64, ["barrier", "partition in a quicksort"], ["out-of-range"])])
def test_error_words_tell_their_causes_apart(cuda_lib, bits, says, says_not):
    buf = ctypes.create_string_buffer(512)
    assert cuda_lib.orqcu_device_error_text(bits, buf, ctypes.c_size_t(512)) == 0
    text = buf.value.decode()
    assert f"(code {bits})" in text
    assert all(s in text for s in says) and not any(s in text for s in says_not)


def test_error_text_keeps_to_its_buffer(cuda_lib):
    buf = ctypes.create_string_buffer(b"x" * 16, 16)
    assert cuda_lib.orqcu_device_error_text(256, buf, ctypes.c_size_t(8)) == 0
    assert len(buf.value) == 7 and buf.raw[8:15] == b"x" * 7
    assert cuda_lib.orqcu_device_error_text(256, None, ctypes.c_size_t(8)) != 0
