"""Order of tensor-memory accesses in the tcgen05 kernels, read from their sources: an access that follows a wait on
an mbarrier comes after a tcgen05.fence::after_thread_sync.  Without it the hardware may move the access above the
wait, which no run is sure to show."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "sparseswin3d_b200" / "csrc"
FENCE = "tc_fence_after()"
USE = r"tmem_(?:ld|st)(?!_wait)\w*\(|umma_(?:ss|ts)\("
WAIT = r"mbar_(?:wait_bounded|wait_asleep|test|try_wait)\("


def _block(code, at):
    """End of the braces that open at or after `at`."""
    depth = 0
    for i in range(code.index("{", at), len(code)):
        depth += (code[i] == "{") - (code[i] == "}")
        if depth == 0:
            return i + 1


def _source(name):
    """The code without comments, and patterns of what waits and what accesses, the lambdas that do so in it included: such a lambda is taken out where it
    is defined and counts where it is called.  One that waits and accesses stays (its calls have the fence in it)."""
    code = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    wait, use = WAIT, USE
    while True:
        for m in re.finditer(r"auto (\w+) = \[&\]", code):
            end = _block(code, m.end())
            body = code[m.start():end]
            waits, uses = bool(re.search(wait, body)), bool(re.search(use, body))
            if waits != uses:
                if waits:
                    wait += rf"|\b{m[1]}\("
                else:
                    use += rf"|\b{m[1]}\("
                code = code[:m.start()] + code[end:]
                break
        else:
            return code, wait, use


def _unfenced(code, wait, use):
    """The accesses in front of which the last wait was not followed by a fence, and how many there are."""
    fenced, uses, bad = False, 0, []
    for m in re.finditer(rf"(?P<wait>{wait})|(?P<fence>tc_fence_after\(\))|(?P<use>{use})", code):
        if m["use"]:
            uses += 1
            if not fenced:
                bad.append(code[m.start():m.start() + 80])
        else:
            fenced = m["fence"] is not None
    return bad, uses


@pytest.mark.parametrize("name, least", [("attn_dense.cu", 12), ("gemm_f32.cu", 20), ("gemm_gelu.cu", 2)])
def test_every_access_behind_a_wait_is_fenced(name, least):
    bad, uses = _unfenced(*_source(name))
    assert not bad and uses >= least, (bad, uses)


@pytest.mark.parametrize("name, least", [("attn_dense.cu", 5), ("gemm_f32.cu", 6), ("gemm_gelu.cu", 2)])
def test_every_fence_is_missed(name, least):
    """Each fence behind a wait taken out in turn."""
    code, wait, use = _source(name)
    tried = 0
    for m in re.finditer(re.escape(FENCE), code):
        if code[:m.start()].rstrip().endswith("__syncthreads();"):   # (where a kernel reads its tensor-memory address)
            continue
        tried += 1
        assert _unfenced(code[:m.start()] + code[m.end():], wait, use)[0], code[m.start() - 200:m.end()]
    assert tried >= least, tried
