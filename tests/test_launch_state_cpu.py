"""State of a kernel that outlasts a launch, read from the sources.  The largest dynamic shared memory of a launch is such: threads that call one kernel
with sizes of their own must not lower it for one another between setting it and launching."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "sparseswin3d_b200" / "csrc"


def test_every_caller_allows_the_same_shared_memory():
    allowed = []
    for f in sorted(CSRC.glob("*.cu*")):
        code = re.sub(r"//[^\n]*", "", f.read_text())
        constants = set(re.findall(r"constexpr (?:int|size_t) (\w+) =", code))
        for call in re.findall(r"(?:allow_smem\(|cudaFuncSetAttribute\()([^;]*)\);", code):
            most = call.rstrip(")").split(",")[-1].strip()
            if "," in call and most != "most":   # (`most`: in allow_smem itself, a constant by default)
                assert most in constants, f"{f.name}: {call}"
            allowed.append(f.name)
    assert len(allowed) >= 12 and "ssw_common.cuh" in allowed
