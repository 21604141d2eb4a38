"""Arrays in shared memory that are read or written 16 bytes at a time are declared on 16 bytes: where the compiler puts one without is its own affair."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "krasis_b200", "csrc")
WIDE = r"(?:float4|uint4|int4|ulonglong2|double2|longlong2)"


def _shared(body):
    """{name: declared on 16 bytes} of the arrays that a kernel's body declares in shared memory."""
    out = {}
    for m in re.finditer(r"__shared__\s+(__align__\((\d+)\)\s+)?([\w ]+?)\s+((?:\w+(?:\s*\[[^;\]]*\])+(?:\s*,\s*)?)+);", body):
        for name in re.findall(r"(\w+)\s*\[", re.sub(r"\[[^\]]*\]", "[", m.group(4))):
            out[name] = int(m.group(2) or 0) >= 16 or re.fullmatch(WIDE, m.group(3).split()[-1]) is not None
    return out


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in re.split(r"(?=__global__|__device__ __forceinline__)", text):
            yield os.path.basename(path), part


def test_arrays_read_16_bytes_at_a_time():
    seen, bad = 0, []
    for path, body in _kernels():
        for name, aligned in _shared(body).items():
            if re.search(r"reinterpret_cast<(?:const )?%s\s*\*>\(\s*&?\s*%s\b" % (WIDE, name), body):
                seen += 1
                bad += [] if aligned else [(path, name)]
    assert seen >= 10 and not bad, (seen, bad)
