"""The library's device code is stored as it is (unpacking it would be part of a process's first solve)."""
import build


def test_device_code_is_not_packed():
    with open(build.build(), "rb") as f:
        code = f.read()
    assert code.count(b".text._ZN8rgbdflow") > 100  # names of the kernels' sections
