"""Properties of the kernel sources that cannot be provoked on a GPU without faulting or hanging it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "csrc"


def code_of(name):
    return "\n".join(line.split("//")[0] for line in (CSRC / name).read_text().splitlines())


@pytest.mark.parametrize("name", ["gdn.cu", "gdn_chain.cu"])
def test_bounded_waits_are_voted_before_warp_instructions(name):
    """Every lane of a scan's warp polls the barrier for itself.  Where the verdict decides whether the warp goes on to ldmatrix / mma.sync, it must
    be the warp's, not the lane's: lanes that disagree at the limit would leave those instructions and the block barrier behind them half attended."""
    code = code_of(name)
    used = [m for m in re.finditer(r"(?:=|\|\||&&|if \(!)\s*ptx::mbar_wait(_warp)?\(", code)]
    assert used, "no waits found"
    for m in used:
        product = code.find("mma64<", m.end())
        voted = m.group(1) or "__all_sync(" in code[m.end():product]
        assert voted, code[m.start():m.start() + 120]


@pytest.mark.parametrize("op", ["gemm2d", "gemm2d_out", "gdn_rule_fwd", "gdn_rule_bwd", "gdn_chain_bwd", "gdn_scan_fwd"])
def test_error_word_is_declared_as_written(op):
    """These kernels store into the device's error word when a wait runs out, so their schemas say that the argument is mutated."""
    schema = re.search(r'm\.def\("' + op + r"\(([^\"]*)\) ->", code_of("bindings.cpp")).group(1)
    assert re.search(r"Tensor\([a-z]!\)\??\s+err\b", schema), schema
