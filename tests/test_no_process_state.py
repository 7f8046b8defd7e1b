"""The library keeps no state of a device or a problem in function-local statics: a flag or a value cached there would be
one for the whole process, where a kernel's attributes and a GPU's properties are per device and threads may share it."""
import re

from conftest import PKG

# the driver's entry point for encoding tensor maps: one function for every device
ALLOWED = {"encode"}
LOCAL_STATIC = re.compile(r"^\s+static\s+(?!constexpr|const\b|inline|__global__|__device__|__host__)[\w:<>*&\s]*?(\w+)\s*(?:=|;|\{|\[)")


def test_no_function_local_static_state():
    found = []
    for f in sorted((PKG / "csrc").glob("*.cu*")):
        for n, line in enumerate(f.read_text().splitlines(), 1):
            m = LOCAL_STATIC.match(line)
            if m and m.group(1) not in ALLOWED:
                found.append(f"{f.name}:{n}: {line.strip()}")
    assert not found, found
