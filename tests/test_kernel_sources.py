"""Properties of the kernel sources that cannot be provoked on a GPU without faulting or hanging it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "csrc"


def code_of(name):
    return "\n".join(line.split("//")[0] for line in (CSRC / name).read_text().splitlines())


@pytest.mark.parametrize("name", ["gdn.cu", "gdn_chain.cu"])
def test_no_lane_leaves_its_warp_between_a_wait_and_a_product(name):
    """Every lane of a scan's warp polls the barrier for itself.  Lanes that disagree at the limit must not part before ldmatrix / mma.sync, which
    would run half attended: the warp votes or a block barrier exchanges the verdict before anything branches on it."""
    code = code_of(name)
    used = [m for m in re.finditer(r"(?:=|\|\||&&|if \()\s*!?ptx::mbar_wait(_warp)?\(", code)]
    assert used, "no waits found"
    for m in used:
        product = code.find("mma64<", m.end())
        if product < 0:                                        # the wait ends a loop whose next round begins with the product
            loop = code.rfind("\n  for (", 0, m.start())
            between = code[m.end():code.find("\n}", m.end())] + code[loop:code.find("mma64<", loop)]
        else:
            between = code[m.end():product]
        vote = re.search(r"__all_sync\(|__syncthreads_or\(", between)
        parted = re.search(r"if \(!?(?:dead|late|ok)\b|break;|return;", between)
        assert m.group(1) or vote and not (parted and parted.start() < vote.start()), code[m.start():m.start() + 120]


def enclosing_headers(code, at):
    """Text in front of every brace that is open at position `at`."""
    heads, start = [], 0
    for i, ch in enumerate(code[:at]):
        if ch == "{":
            heads.append(code[start:i])
            start = i + 1
        elif ch == "}":
            heads.pop()
            start = i + 1
        elif ch == ";":
            start = i + 1
    return heads


@pytest.mark.parametrize("name", ["gemm.cu", "gemm_pair.cu", "gemm_persistent.cu", "moe.cu", "moe_persistent.cu", "mxfp8.cu", "qsa_tc.cu"])
def test_waits_of_whole_warps_are_voted(name):
    """The same for the warps that read accumulators (tcgen05.ld needs all lanes): a wait whose verdict belongs to one lane stands in a part
    that one elected lane executes; everywhere else the warp votes."""
    code = code_of(name)
    for m in re.finditer(r"ptx::mbar_wait\(", code):
        assert any("elect_one()" in head for head in enclosing_headers(code, m.start())), code[m.start():m.start() + 100]


@pytest.mark.parametrize("op", ["gemm2d", "gemm2d_out", "gdn_rule_fwd", "gdn_rule_bwd", "gdn_chain_bwd", "gdn_scan_fwd"])
def test_error_word_is_declared_as_written(op):
    """These kernels store into the device's error word when a wait runs out, so their schemas say that the argument is mutated."""
    schema = re.search(r'm\.def\("' + op + r"\(([^\"]*)\) ->", code_of("bindings.cpp")).group(1)
    assert re.search(r"Tensor\([a-z]!\)\??\s+err\b", schema), schema


# kernels that set up their barriers and tensor memory while the kernel before them ends
SETS_UP_FIRST = ("gemm_persistent.cu", "gemm_pair.cu")


def test_kernels_wait_for_the_kernels_before_them():
    """A kernel started by `launch` (programmatic dependent launch) may begin before its predecessor's writes are visible: each waits, and none
    releases its successor early, whose blocks could hold tensor memory that the running kernel's blocks have yet to allocate."""
    for path in sorted(CSRC.glob("*.cu")):
        code = code_of(path.name)
        assert "launch_dependents" not in code, path.name
        if '#include "launch.cuh"' not in code:
            continue
        bodies = re.split(r"\n(?:template[^\n]*\n)?(?:static )?__global__", code)[1:]
        assert bodies, path.name
        for body in bodies:
            name = re.search(r"(\w+)\s*\((?!\d)", re.sub(r"__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\)", "", body)).group(1)
            body = body[body.index("{") + 1:body.find("\n}")]
            before, wait, _ = body.partition("grid_wait();")
            assert wait, (path.name, name)
            if path.name in SETS_UP_FIRST:
                # barriers, tensor memory and addresses only: every block reaches the wait, and no operand is touched before it
                assert before.count("{") == before.count("}") and not re.search(r"\breturn\b|tma_(load|store|reduce)|\bp\.C(in)?\b|\bp\.err\b", before), (path.name, name)
            else:
                assert not before.strip(), (path.name, name)
        assert "<<<" not in code, path.name


def test_c_entry_points_report_launch_errors():
    """`launch` throws; an exception that crosses a C boundary ends the caller's process.  Functions with C linkage use `try_launch`, and nothing
    else that throws."""
    found = 0
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp")):
        code = code_of(path.name)
        for m in re.finditer(r'extern "C"[^{;]*\)\s*(?:noexcept\s*)?\{', code):
            body = code[m.start():code.find("\n}", m.start())]
            found += 1
            assert not re.search(r"\blaunch\(|C10_CUDA_|TORCH_CHECK|\bat::", body), path.name
    assert found


# conditions of a `continue` that whole warps agree on
WARP_UNIFORM = r"k\.num_kb == 0|EPI == \w+|TMA_OUT|jb > row0 / 64 \+ \(quarter >> 1\)"


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu") if "tmem_ld" in p.read_text()))
def test_no_lane_skips_ahead_of_a_tensor_memory_read(name):
    """tcgen05.ld and tcgen05.st need all lanes of a warp.  Lanes that leave a round of a loop early (`continue` under a condition of their own) meet
    the others at a __syncwarp() before the next round's read."""
    code = code_of(name)
    for m in re.finditer(r"\bcontinue;", code):
        heads, opened = [], []
        for i, ch in enumerate(code[:m.start()]):
            if ch == "{":
                heads.append(code[code.rfind("\n", 0, i) + 1:i])
                opened.append(i)
            elif ch == "}":
                heads.pop()
                opened.pop()
        loop = max(k for k, head in enumerate(heads) if re.search(r"\b(for|while) \(", head))
        depth, end = 1, opened[loop] + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(code[end], 0)
            end += 1
        body = code[opened[loop] + 1:end]
        condition = code[code.rfind("\n", 0, m.start()) + 1:m.start()] + " ".join(heads[loop + 1:])
        if re.search(r"tmem_(ld|st)_32", body) and not re.search(WARP_UNIFORM, condition):
            assert body.lstrip().startswith("__syncwarp();"), (name, condition)
